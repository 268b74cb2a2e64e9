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
    s = np.arange(-(1 << 20), (1 << 20) + 1, dtype=np.int64)
    for other in (s[::-1], np.full_like(s, s[0]), np.full_like(s, s[-1])):
        assert (reduce_pair(s, other) == (s % Q) + ((other % Q) << 16)).all()
        assert (reduce_pair(other, s) == (other % Q) + ((s % Q) << 16)).all()


def operand(bits, packed):
    """The operand rows (signed bytes, [n][128]) of packed rows, [parity][part]."""
    w = packed.reshape(packed.shape[0], -1).view(np.uint32)
    mask, sign = (0x03030303, 0x02020202) if bits == 2 else (0x07070707, 0x04040404)
    if bits == 2:
        fields = [[w, w >> np.uint32(4)], [w >> np.uint32(2), w >> np.uint32(6)]]
    else:
        by = packed.reshape(packed.shape[0], -1, 8)           # bytes of a word pair
        halves = [np.ascontiguousarray(by[:, :, h::2]).view(np.uint32)[..., 0] for h in (0, 1)]
        fields = [halves, [v >> np.uint32(3) for v in halves]]
    out = []
    for per_part in fields:
        out.append([])
        for f in per_part:
            f = f & np.uint32(mask)
            row = np.stack([f ^ np.uint32(sign), f << np.uint32(8 - bits)], axis=2)
            out[-1].append(row.view(np.int8).reshape(w.shape[0], 128).astype(np.int64))
    return out


@pytest.mark.parametrize("bits,lo,hi", [(2, -2, 1), (3, -4, 3)])
def test_packed_forward_model(table, oracle, bits, lo, hi):
    raw = table(f"build_pack_tables({bits}, out);", 2 * 4 * 2048)
    B = [np.concatenate([decode(raw[2048 * (4 * h + i):][:2048], 64) for i in range(4)],
                        axis=1).view(np.int8).astype(np.int64) for h in (0, 1)]
    for b in B:                            # words alternate: constants of x - lo, of 2^s x
        c0, c1 = b.reshape(64, 32, 4)[:, 0::2], b.reshape(64, 32, 4)[:, 1::2]
        assert (c0.sum((1, 2)) == 0).all()                     # the offset drops out
    # |P +- M| over every input: the reduction's exact range
    worst = sum(np.abs(b.reshape(64, 32, 4)[:, 0::2] + (1 << (8 - bits)) *
                       b.reshape(64, 32, 4)[:, 1::2]).sum((1, 2)) for b in B) * -lo
    assert worst.max() < 1 << 20
    r = rng(bits)
    x = r.integers(lo, hi + 1, size=(96, 256)).astype(np.int16)
    x[0], x[1] = lo, hi
    sums = [[part @ b.T for part, b in zip(parts, B)]
            for parts in operand(bits, oracle.pack_small(bits, x))]
    got = np.zeros((96, 256), dtype=np.int64)
    for sign, at in ((1, 0), (-1, 2)):
        s0, s1 = (p + sign * m for p, m in sums)
        pair = reduce_pair(s0, s1)
        got[:, at::4], got[:, at + 1::4] = pair & 0xffff, pair >> 16
    assert (got == canon(oracle.ntt(x))).all()


def test_tc5_signed_first_stage_sums(table, oracle):
    """The tcgen05 inverse and forward on signed first-stage sums: below 2^24 for
    every input, their top byte (0 or 255) weighted by the kernels' own tiles."""
    from test_tc5_model import as_s8, as_u8, decode as decode_tiles
    t = decode_tiles(table("static Matrices M; build_matrices(&M); build_tc5_tables(M, out, true);",
                           68 * 1024))
    x = rng(77).integers(-32768, 32768, size=(64, 256)).astype(np.int16)
    x[0], x[1], x[2] = -32768, 32767, np.where(np.arange(256) % 2, -32768, 32767)
    raw = x.view(np.uint8).reshape(64, 256, 2)

    def first(by, lo, hi):
        d = as_u8(by) @ lo.T + as_s8(by) @ hi.T
        return d[:, :16] + 128 * d[:, 16:]

    def second(s, tiles):
        by = np.ascontiguousarray(s.astype(np.int32)).view(np.uint8).reshape(-1, 64).astype(np.int64)
        d = by[:, :32] @ tiles[0].T + by[:, 32:] @ tiles[1].T
        v = d[:, :16] + 128 * d[:, 16:]
        assert v.min() >= 0 and v.max() + 1664 < 1 << 26
        return v % Q
    # the bound of the sums over all inputs: low bytes 0..255, high bytes -128..127
    for lo, hi in [(t[2 * m], t[2 * m + 1]) for m in range(16)] + [(t[34], t[35])]:
        top = (255 * lo.sum(1) + 127 * hi.sum(1)).reshape(2, 16)
        low = (-128 * hi.sum(1)).reshape(2, 16)
        assert (top[0] + 128 * top[1]).max() < 1 << 24 and (low[0] + 128 * low[1]).min() > -(1 << 24)
    inv = np.zeros((64, 16, 16), dtype=np.int64)
    Y = np.stack([first(raw[:, 16 * m:16 * m + 16].reshape(64, 32), t[2 * m], t[2 * m + 1])
                  for m in range(16)], axis=1)                        # [p][m][c]
    fwd = np.zeros((64, 16, 16), dtype=np.int64)
    Z = np.stack([first(np.ascontiguousarray(raw.reshape(64, 16, 16, 2)[:, :, c]).reshape(64, 32),
                        t[34], t[35]) for c in range(16)], axis=2)    # [p][i][c]
    for n in range(16):
        inv[:, :, n] = second(Y[:, :, n], t[32:34])
        fwd[:, n] = second(Z[:, n], t[36 + 2 * n:38 + 2 * n])
    c = canon(x).astype(np.int16)
    assert (inv.reshape(64, 256) == canon(oracle.invntt(c))).all()
    assert (fwd.reshape(64, 256) == canon(oracle.ntt(c))).all()
