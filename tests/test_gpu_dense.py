"""GPU parity of the dense tcgen05 kernels at the sizes where their tiling can
go wrong.  Integer work: bit-exact."""
import numpy as np
import pytest

from conftest import rng
from py_oracle import canon

pytestmark = pytest.mark.gpu


def dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


# both sides of the dispatch line (two waves of 3 x 148 CTAs of 32), a tile of
# one row, two to several 128-polynomial tiles per CTA with and without a remainder
@pytest.mark.parametrize("npoly", [28416, 28417, 128 * 223 + 1, 128 * 148 * 2 - 127,
                                   128 * 148 * 2 + 1, 128 * 148 * 4 + 77, 128 * 148 * 7])
@pytest.mark.parametrize("bits,lo,hi", [(2, -2, 2), (3, -4, 4)])
def test_packed_dense(tk, cuda, oracle, bits, lo, hi, npoly):
    import torch
    x = rng(bits + npoly).integers(lo, hi, size=(npoly, 256)).astype(np.int16)
    x[0], x[-1] = lo, hi - 1
    pk = dev(oracle.pack_small(bits, x))
    out = torch.full((npoly + 1, 256), 12345, dtype=torch.int16, device="cuda")
    tk.ntt_packed(pk, bits, out=out[:npoly])
    full = dev(x)
    tk.ntt(full)
    assert torch.equal(out[:npoly], full)
    assert (out[npoly] == 12345).all()                # nothing past the batch
    pick = np.r_[0:64, npoly - 64:npoly]
    assert (out[:npoly].cpu().numpy()[pick] == canon(oracle.ntt(x[pick]))).all()
    assert tk.device_status(0) == 0
