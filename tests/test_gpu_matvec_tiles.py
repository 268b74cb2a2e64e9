"""Tile kinds of the tiled matrix-vector kernel: job counts at the edges of a tile
and of the dispatch between one, two and four units, each k alone and mixed, out
of place and in place, against the three-kernel pipeline and the oracle."""
import numpy as np
import pytest

from conftest import rng
from py_oracle import Q, canon

pytestmark = pytest.mark.gpu

CASES = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (3, 3, 3), (4, 2, 2), (5, 7, 3), (0, 24, 0), (0, 25, 0),
         (0, 0, 37), (0, 1184, 0), (0, 1185, 0), (0, 0, 1184), (0, 0, 1185), (2368, 0, 0),
         (2369, 0, 0), (0, 0, 2369), (450, 449, 451), (500, 499, 501), (900, 901, 899),
         (1100, 1101, 1099), (4736, 0, 0), (4737, 5, 0)]


@pytest.mark.parametrize("jobs", CASES)
@pytest.mark.parametrize("with_e", [True, False])
def test_tile_kinds(tk, cuda, oracle, jobs, with_e):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(sum(j << (8 * i) for i, j in enumerate(jobs)))

    def rand(shape, lo, hi):
        return torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=torch.int16)
    batches = []
    for k, n in zip((2, 3, 4), jobs):
        if n:
            batches.append((k, rand((n, k, k, 256), -32768, 32767), rand((n, k, 256), -32768, 32767),
                            rand((n, k, 256), -32768, 32767) if with_e else None))

    def run(mode, in_place):
        outs, call = [], []
        for k, A, s, e in batches:
            if in_place:
                v = s.clone()
                call.append((k, A, v, e, v))
                outs.append(v)
            else:
                v = torch.full((s.shape[0] + 1, k, 256), 99, dtype=torch.int16, device="cuda")
                call.append((k, A, s, e, v[:-1]))
                outs.append(v)
        tk.set_option(tk.OPT_MATVEC_MODE, mode)
        try:
            tk.matvec(call)
        finally:
            tk.set_option(tk.OPT_MATVEC_MODE, tk.MATVEC_TILED)
        if not in_place:
            assert all((v[-1] == 99).all() for v in outs)      # nothing past the batch
            outs = [v[:-1] for v in outs]
        return outs
    want = run(tk.MATVEC_PIPELINE, False)
    for in_place in (False, True):
        for got, ref in zip(run(tk.MATVEC_TILED, in_place), want):
            assert torch.equal(got, ref), in_place
    assert tk.device_status(0) == 0
    # the sums of products are exact mod q: small operands for the oracle's int16 path
    for k, n in zip((2, 3, 4), jobs):
        if not n:
            continue
        r = rng(n)
        A = r.integers(0, Q, size=(n, k, k, 256)).astype(np.int16)
        s = r.integers(-3, 4, size=(n, k, 256)).astype(np.int16)
        e = r.integers(-3, 4, size=(n, k, 256)).astype(np.int16)
        dA, ds, de = (torch.from_numpy(v).cuda() for v in (A, s, e))
        out = torch.empty_like(ds)
        tk.matvec([(k, dA, ds, de, out)])
        got = out.cpu().numpy()
        for j in sorted({0, n // 2, n - 1}):
            want_j = oracle.matvec_job(k, A[j].reshape(k * k, 256), s[j], e[j])
            assert (canon(got[j]) == canon(want_j)).all(), (k, j)
