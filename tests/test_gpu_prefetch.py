"""Kernels fetch their first tile's lines into L2 before they wait for the previous
kernel in the stream: chains in which every kernel reads what the one before it
wrote, at sizes on both sides of the line from which they do, give what the same
calls give with a synchronisation after each."""
import pytest

pytestmark = pytest.mark.gpu

# 148 SMs x 3 (forward) or 4 (inverse) CTAs x 8 polynomials, and x 32 x 1.5 tiles
SIZES = [3552, 3553, 4736, 4737, 16411, 21304, 21305, 21313, 28408, 28409, 28417, 60000, 262145]


def ints(gen, shape, lo, hi, dtype):
    import torch
    return torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=torch.int16).to(dtype)


@pytest.mark.parametrize("n", SIZES)
def test_chain_of_transforms(tk, cuda, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = ints(gen, (n, 256), -32768, 32767, torch.int16)
    small = ints(gen, (n, 256), -2, 2, torch.int16)
    packed = ints(gen, (n, 64), 0, 256, torch.uint8)
    buf, y = torch.empty_like(x), torch.empty_like(x)

    def chain(sync):
        out = []
        for src in (x, small):
            for step in (lambda: buf.copy_(src), lambda: tk.ntt(buf), lambda: tk.ntt(buf, out=y),
                         lambda: tk.invntt(y), lambda: tk.invntt(y, out=buf),
                         lambda: tk.ntt_small(small, out=y), lambda: tk.invntt(y),
                         lambda: tk.ntt(y), lambda: tk.ntt_packed(packed, 2, out=buf),
                         lambda: tk.invntt(buf), lambda: tk.ntt(buf, out=y)):
                step()
                if sync:
                    torch.cuda.synchronize()
            out += [buf.clone(), y.clone()]
        return out
    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(chain(False), want))
    # an input rewritten by a small kernel just before the launch
    for turn in range(5):
        buf.fill_(turn)
        tk.ntt(buf, out=y)
        ref = tk.ntt(torch.full((1, 256), turn, dtype=torch.int16, device="cuda"))
        assert (y == ref).all(), turn
    assert tk.device_status(0) == 0


@pytest.mark.parametrize("jobs", [(11824, 0, 0), (11825, 0, 0), (0, 5912, 0), (0, 5913, 0),
                                  (0, 0, 5920), (3000, 3000, 3000)])
def test_chain_of_matvecs(tk, cuda, jobs):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(sum(jobs))
    batches = [(k, ints(gen, (n, k, k, 256), -32768, 32767, torch.int16),
                ints(gen, (n, k, 256), -32768, 32767, torch.int16),
                ints(gen, (n, k, 256), -32768, 32767, torch.int16))
               for k, n in zip((2, 3, 4), jobs) if n]

    def chain(sync):
        v = [s.clone() for _, _, s, _ in batches]
        w = [torch.empty_like(s) for s in v]
        for _ in range(4):      # v -> w -> v, the second time with e
            for src, dst, add in ((v, w, None), (w, v, batches)):
                tk.matvec([(k, A, a, e if add else None, b)
                           for (k, A, _, e), a, b in zip(batches, src, dst)])
                if sync:
                    torch.cuda.synchronize()
        return v
    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(chain(False), want))
    assert tk.device_status(0) == 0
