"""Which buffers tk_matvec_host uses in place, and that a call above the size limit
is staged (in place, its kernel would hold the GPU for the length of the
transfer): every page-locked layout, the sizes around the limit, and large calls
of each tile kind, each with the outputs of a pageable arena."""
import numpy as np
import pytest

from conftest import rng
from test_gpu_matvec_host import layout, pinned, run

pytestmark = pytest.mark.gpu

ONE, TWO = ((3, 20),), ((4, 9), (2, 16))
LAYOUTS = [("packed", ONE, 2), ("packed", TWO, 2), ("apart", TWO, 2), ("in_place", TWO, 2),
           ("no_addend", ONE, 2), ("out_is_e", ONE, 1), ("out_in_A", ONE, 1),
           ("out_half_over_s", ONE, 1), ("out_is_next_s", TWO, 1), ("outs_overlap", TWO, 0),
           ("misaligned", ONE, 0), ("packed", ((2, 1),) * 4, 2), ("packed", ((2, 1),) * 5, 0)]
# 5,120, 9,216 and 14,336 bytes a job; the limit is 1 MiB
SIZES = [("packed", ((2, 204),), 2), ("packed", ((2, 205),), 0), ("packed", ((3, 113),), 2),
         ("packed", ((3, 114),), 0), ("packed", ((4, 73),), 2), ("packed", ((4, 74),), 0),
         ("packed", ((4, 36), (3, 57)), 2), ("packed", ((4, 37), (3, 57)), 0),
         ("out_is_e", ((4, 73),), 1), ("out_is_e", ((4, 74),), 0), ("packed", ((4, 1500),), 0),
         ("packed", ((2, 8000),), 0), ("packed", ((3, 6000),), 0)]


@pytest.mark.parametrize("kind,specs,in_place", LAYOUTS + SIZES)
def test_buffers_used_in_place(tk, cuda, kind, specs, in_place):
    lay, size = layout(kind, specs)
    locked = pinned(size)
    for turn in range(2):          # the host rewrites the buffers between calls
        data = rng(turn + size).integers(-32768, 32768, size=size).astype(np.int16)
        want = data.copy()
        run(tk, want, lay)
        assert tk.get_option(tk.OPT_MATVEC_HOST_IN_PLACE) == 0     # pageable
        locked[:] = data
        run(tk, locked, lay)
        assert tk.get_option(tk.OPT_MATVEC_HOST_IN_PLACE) == in_place
        assert np.array_equal(locked, want), turn
    assert tk.device_status(0) == 0


def test_other_modes_are_staged(tk, cuda):
    lay, size = layout("packed", ONE)
    locked = pinned(size)
    for mode in (tk.MATVEC_PIPELINE, tk.MATVEC_FUSED):
        tk.set_option(tk.OPT_MATVEC_MODE, mode)
        try:
            run(tk, locked, lay)
            assert tk.get_option(tk.OPT_MATVEC_HOST_IN_PLACE) == 0
        finally:
            tk.set_option(tk.OPT_MATVEC_MODE, tk.MATVEC_TILED)
