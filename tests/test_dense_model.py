"""CPU model of the dense tcgen05 kernels: their constant tables, read back from
the K-major core-matrix layout, the operand bytes their unpacking makes and
their reductions, against the oracle.  No GPU needed."""
import os
import subprocess

import numpy as np
import pytest

from conftest import rng
from py_oracle import Q, canon

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tensorkyber_b200", "csrc")


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    """table(expr, size): the bytes that a C++ statement fills `out` with."""
    d = tmp_path_factory.mktemp("tables")

    def get(statement, size):
        src, exe = d / "t.cpp", d / "t"
        src.write_text('#include <stdio.h>\n#include "tk_tables.h"\nusing namespace tk;\n'
                       f"static unsigned char out[{size}];\n"
                       f"int main() {{ {statement} fwrite(out, 1, {size}, stdout); return 0; }}\n")
        subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src),
                        os.path.join(CSRC, "tk_tables.cpp"), "-o", str(exe)], check=True)
        return np.frombuffer(subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE).stdout,
                             dtype=np.uint8)
    return get


def decode(tile: np.ndarray, rows: int) -> np.ndarray:
    """B[n][k] of one K step (rows x 32 bytes) from the K-major layout."""
    n, k = np.arange(rows)[:, None], np.arange(32)[None, :]
    off = (n >> 3) * 256 + (k >> 4) * 128 + (n & 7) * 16 + (k & 15)
    assert sorted(off.ravel().tolist()) == list(range(32 * rows))
    return tile[off]


def reduce_pair(s0, s1):
    """tk_pack.cu's reduce_pair on arrays: the packed pair as uint32."""
    m, half = 1290168, 645083
    q0, q1 = (s0 * m + half) >> 32, (s1 * m + half) >> 32
    return ((s0 + (s1 << 16)) - (q0 + (q1 << 16)) * Q) & 0xffffffff


def test_reduce_pair_is_exact_over_its_range():
    s = np.arange(-128 * 4 * 1664, 128 * 4 * 1664 + 1, dtype=np.int64)
    for other in (s[::-1], np.full_like(s, s[0]), np.full_like(s, s[-1])):
        assert (reduce_pair(s, other) == (s % Q) + ((other % Q) << 16)).all()
        assert (reduce_pair(other, s) == (other % Q) + ((s % Q) << 16)).all()


def operand(bits, packed):
    """The even and odd operand rows (signed bytes, [n][256]) of packed rows."""
    w = packed.reshape(packed.shape[0], -1).view(np.uint32)
    out = []
    for parity in (0, 1):
        if bits == 2:
            f = (w >> np.uint32(2 * parity)) & np.uint32(0x33333333)
            x, top = np.array([0, 1, -2, -1], np.int8), np.array([0, 64, -128, -64], np.int8)
            nib = np.stack([(f >> np.uint32(4 * i)) & np.uint32(3) for i in range(8)], axis=2)
            row = np.concatenate([x[nib], top[nib]], axis=2)        # [n][word][16]
        else:
            f = (w >> np.uint32(3 * parity)) & np.uint32(0x07070707)
            x = f + (f & np.uint32(0x04040404)) * np.uint32(62)
            row = np.stack([x, f << np.uint32(5)], axis=2).view(np.int8)
        out.append(row.reshape(w.shape[0], 256).astype(np.int64))
    return out


@pytest.mark.parametrize("bits,lo,hi", [(2, -2, 1), (3, -4, 3)])
def test_packed_forward_model(table, oracle, bits, lo, hi):
    raw = table(f"build_pack_tables({bits}, out);", 2 * 8 * 2048)
    B = np.concatenate([np.concatenate([decode(raw[2048 * (8 * h + i):][:2048], 64)
                                        for i in range(8)], axis=1) for h in (0, 1)])
    B = B.view(np.int8).astype(np.int64)                               # [128 outputs][256]
    r = rng(bits)
    x = r.integers(lo, hi + 1, size=(96, 256)).astype(np.int16)
    x[0], x[1] = lo, hi
    ev, od = operand(bits, oracle.pack_small(bits, x))
    s0, s1 = ev @ B.T, od @ B.T
    assert max(np.abs(s0).max(), np.abs(s1).max()) <= 128 * -lo * 1664
    pair = reduce_pair(s0, s1)
    got = np.stack([pair & 0xffff, pair >> 16], axis=2).reshape(-1, 256)
    assert (got == canon(oracle.ntt(x))).all()
