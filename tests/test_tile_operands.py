"""The tiled matrix-vector kernel's basemul operands and stage-A tables, on the
CPU: dp2a sums over operand bytes against the plain sums at the bounds of ntt(s)
and A, and the stage-A fragments (parity halves in coefficient order) against
the batch inverse's (interleaved slots)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import rng
from py_oracle import Q
from test_basemul_model import pair_roots

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tensorkyber_b200", "csrc")
SUM_BIAS_Z = 3329 << 19


def red_wide(x):
    return x - ((x * 1290167) >> 32) * Q


def dp2a(a0, a1, w, hi):
    return a0 * w[..., 2 * hi] + a1 * w[..., 2 * hi + 1]


@pytest.mark.parametrize("k", [2, 3, 4])
@pytest.mark.parametrize("extreme", [None, -32768, 32767])
def test_dp2a_sums(k, extreme):
    r = rng(k)
    a = r.integers(-32768, 32768, size=(k, 128, 2))
    b = r.integers(0, Q + 22, size=(k, 128, 2))
    if extreme is not None:
        a[:], b[:] = extreme, Q + 21
    z = pair_roots()
    zb = red_wide(b[..., 1] * z)
    assert zb.min() >= 0 and zb.max() < Q + 4
    lo = lambda v: v & 255          # noqa: E731
    hi = lambda v: v >> 8           # noqa: E731
    w0 = np.stack([lo(b[..., 0]), lo(zb), hi(b[..., 0]), hi(zb)], axis=-1)
    w1 = np.stack([lo(b[..., 1]), lo(b[..., 0]), hi(b[..., 1]), hi(b[..., 0])], axis=-1)
    for w, want in ((w0, a[..., 0] * b[..., 0] + a[..., 1] * zb),
                    (w1, a[..., 0] * b[..., 1] + a[..., 1] * b[..., 0])):
        t = SUM_BIAS_Z + dp2a(a[..., 0], a[..., 1], w, 0).sum(0) \
            + 256 * dp2a(a[..., 0], a[..., 1], w, 1).sum(0)
        assert (t == SUM_BIAS_Z + want.sum(0)).all()
        assert t.min() >= 0 and t.max() < 1 << 32
        assert red_wide(t).max() < 4682


def test_forward_lazy_reduction_bound():
    """stage_c<lazy> on forward sums below 2^26: [0, q + 22)."""
    s = np.concatenate([np.arange(1 << 20), np.arange((1 << 26) - (1 << 20), 1 << 26),
                        Q * np.arange(1, (1 << 26) // Q) - 1]).astype(np.int64)
    y = red_wide(s)
    assert (y % Q == s % Q).all() and y.min() >= 0 and y.max() < Q + 22


def test_stage_a_fragments(tk, tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <stdio.h>\n#include "tk_tables.h"\nusing namespace tk;\n'
                   "static Matrices M; static TileFrags F;\n"
                   "int main() { build_matrices(&M); build_tile_frags(M, &F);\n"
                   "fwrite(&F, sizeof(F), 1, stdout); return 0; }\n")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(src),
                    os.path.join(CSRC, "tk_tables.cpp"), "-o", str(exe)], check=True)
    raw = subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE).stdout

    def rows(words):                 # [16][2][32 lanes][2 regs] -> [16][2][16 rows][16 k]
        by = np.ascontiguousarray(words).view(np.uint8).reshape(16, 2, 32, 2, 4)
        out = np.zeros((16, 2, 16, 16), dtype=np.uint8)
        for lane in range(32):
            for j in range(2):
                out[:, :, lane // 4 + 8 * j, 4 * (lane % 4):4 * (lane % 4) + 4] = by[:, :, lane, j]
        return out
    tile = rows(np.frombuffer(raw, dtype=np.uint32).reshape(16, 2, 32, 2))
    batch = rows(tk.get_table(5)[:2048].reshape(16, 2, 32, 2))
    slot = [(j >> 1) + 4 * (j & 1) for j in range(8)]        # batch slot j: c' = 2 slot[j] + s
    for j in range(8):
        assert (tile[..., 2 * slot[j]:2 * slot[j] + 2] == batch[..., 2 * j:2 * j + 2]).all()
