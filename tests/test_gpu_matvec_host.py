"""tk_matvec_host on page-locked buffers, which the kernel uses in place: every
layout of one arena (back to back, apart, in place, misaligned, overlapping in the
ways the host form accepts) leaves a page-locked arena exactly as a pageable one,
whose buffers are copied to the device and back."""
import numpy as np
import pytest

from conftest import rng

pytestmark = pytest.mark.gpu

P = 256  # int16 per polynomial


def layout(kind, specs):
    """[(k, jobs, A, s, e, out offsets)] and the arena's size, in coefficients."""
    at, out = 0, []
    for k, n in specs:
        a, v = n * k * k * P, n * k * P
        gap = {"apart": 8, "misaligned": 1}.get(kind, 0)
        A = at + gap
        s = A + a + gap
        e = s + v + gap
        o = e + v + gap
        at = o + v
        if kind == "in_place":
            o = s
        elif kind == "no_addend":
            e = None
        elif kind == "out_is_e":
            o = e
        elif kind == "out_in_A":
            o = A
        elif kind == "out_half_over_s":
            o = s + v // 2 // 8 * 8
        out.append([k, n, A, s, e, o])
    if kind == "out_is_next_s" and len(out) > 1:
        out[0][5] = out[1][3]
    if kind == "outs_overlap" and len(out) > 1:
        out[1][5] = out[0][5]
    return out, at + 4096 + max(n * k * P for k, n in specs)


KINDS = ["packed", "apart", "in_place", "no_addend", "misaligned", "out_is_e", "out_in_A",
         "out_half_over_s", "out_is_next_s", "outs_overlap"]
SPECS = [((3, 1),), ((4, 36),), ((4, 37),), ((2, 5), (3, 3), (4, 2)),
         ((2, 1), (3, 2), (4, 3), (2, 4), (3, 5)), ((3, 700), (2, 9))]


def run(tk, arena, lay, outs=None):
    items = []
    for i, (k, n, A, s, e, o) in enumerate(lay):
        def view(at, *shape, of=arena):
            return None if at is None else of[at:at + int(np.prod(shape))].reshape(shape)
        items.append((k, view(A, n, k, k, P), view(s, n, k, P), view(e, n, k, P),
                      view(o, n, k, P) if outs is None else outs[i]))
    tk.matvec_host(items)


def pinned(size):
    import torch
    return torch.empty(size, dtype=torch.int16, pin_memory=True).numpy()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("specs", SPECS)
def test_page_locked_arena_as_pageable(tk, cuda, kind, specs):
    lay, size = layout(kind, specs)
    locked = pinned(size)
    for turn in range(3):          # the host rewrites the buffers between calls
        data = rng(turn + size).integers(-32768, 32768, size=size).astype(np.int16)
        want = data.copy()
        run(tk, want, lay)
        locked[:] = data
        run(tk, locked, lay)
        assert np.array_equal(locked, want), turn
    assert tk.device_status(0) == 0


@pytest.mark.parametrize("locked_inputs", [True, False])
def test_one_side_page_locked(tk, cuda, locked_inputs):
    lay, size = layout("packed", SPECS[3])
    data = rng(5).integers(-32768, 32768, size=size).astype(np.int16)
    want = data.copy()
    run(tk, want, lay)
    inputs = pinned(size) if locked_inputs else np.empty(size, np.int16)
    inputs[:] = data
    outs = [(np.empty(n * k * P, np.int16) if locked_inputs else pinned(n * k * P))
            .reshape(n, k, P) for k, n, *_ in lay]
    run(tk, inputs, lay, outs)
    for (k, n, _, _, _, o), got in zip(lay, outs):
        assert np.array_equal(got.ravel(), want[o:o + n * k * P])
    assert np.array_equal(inputs, data)


def test_many_rewrites_are_seen(tk, cuda):
    lay, size = layout("packed", ((4, 37),))
    locked, want = pinned(size), np.empty(size, np.int16)
    gen = rng(9)
    for _ in range(100):
        want[:] = gen.integers(-32768, 32768, size=size).astype(np.int16)
        locked[:] = want
        run(tk, want, lay)
        run(tk, locked, lay)
        assert np.array_equal(locked, want)
