"""A CTA's last tile with one, two or three quarters of its units (mma.sync
kernels): every variant and input form at sizes that leave each, and one
unit per CTA, against the tcgen05 kernel byte for byte and the oracle."""
import numpy as np
import pytest

from conftest import rng
from py_oracle import canon

pytestmark = pytest.mark.gpu

# units of 8 polynomials over 444, 592, 888 or 296 CTAs: fewer units than CTAs,
# then 1 to 9 per CTA, ragged by one polynomial on either side of a unit
SIZES = [1, 8, 9, 23, 1000, 3552, 4737, 7104, 7113, 8 * 444 * 3 - 7, 8 * 592 * 3 + 1,
         8 * 444 * 5 + 1, 8 * 592 * 6, 8 * 888 * 7 - 1, 8 * 296 * 15 + 3]


def dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("n", SIZES)
def test_every_variant_short_last_tile(tk, cuda, oracle, n):
    import torch
    x = rng(n).integers(-32768, 32768, size=(n, 256), dtype=np.int16)
    d = dev(x)
    pick = np.r_[0:min(n, 24), max(0, n - 24):n]
    want = {tk.FORWARD: oracle.ntt(canon(x[pick]).astype(np.int16)),
            tk.INVERSE: oracle.invntt(canon(x[pick]).astype(np.int16))}
    for direction, f in ((tk.FORWARD, tk.ntt), (tk.INVERSE, tk.invntt)):
        ref = None
        try:
            for v in (4, 0, 1, 2, 3):
                tk.set_variant(direction, v)
                out = torch.full((n + 8, 256), 777, dtype=torch.int16, device="cuda")
                f(d, out=out[:n])
                assert (out[n:] == 777).all(), v
                ref = out[:n] if ref is None else ref
                assert torch.equal(out[:n], ref), (direction, v)
        finally:
            tk.set_variant(direction, -1)
        assert (canon(ref.cpu().numpy()[pick]) == canon(want[direction])).all()
    assert tk.device_status(0) == 0


@pytest.mark.parametrize("n", SIZES)
def test_forms_short_last_tile(tk, cuda, oracle, n):
    import torch
    for bits, lo, hi in ((2, -2, 2), (3, -4, 4)):
        x = rng(n + bits).integers(lo, hi, size=(n, 256)).astype(np.int16)
        full = tk.ntt(dev(x))
        assert torch.equal(tk.ntt_packed(dev(oracle.pack_small(bits, x)), bits), full)
        assert torch.equal(tk.ntt_small(dev(x)), full)
    assert tk.device_status(0) == 0
