"""tk_ntt_small's range check at every size of a CTA's last tile: a coefficient
outside [-128, 127] raises the flag wherever it lies, and a launch on clean inputs
right after, whose CTAs find the other's rows in shared memory, raises none."""
import pytest

pytestmark = pytest.mark.gpu


# units of 8 polynomials per SM: 1 to 4 and 5 to 8 per CTA at two to four CTAs per SM
@pytest.mark.parametrize("per_sm", [1, 2, 3, 5, 6, 8, 9, 12, 13, 15, 18, 21, 24])
def test_range_flag(tk, cuda, per_sm):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 8 * sms * per_sm - 3
    gen = torch.Generator(device="cuda").manual_seed(n)
    clean = torch.randint(-128, 128, (n, 256), generator=gen, device="cuda", dtype=torch.int16)
    want = tk.ntt(clean.clone())
    out = torch.empty_like(clean)
    dirty = torch.full_like(clean, 32767)
    tk.ntt_small(clean, out)
    assert tk.device_status(0) == 0 and torch.equal(out, want)
    for at in (0, n // 3, n // 2, n - 1):
        x = clean.clone()
        x[at, (7 * at) % 256] = 128 if at % 2 else -129
        tk.ntt_small(x, out)
        assert tk.device_status(0) == tk.FLAG_SMALL_RANGE, at
        tk.ntt_small(dirty, out)
        assert tk.device_status(0) == tk.FLAG_SMALL_RANGE
        tk.ntt_small(clean, out)
        assert tk.device_status(0) == 0 and torch.equal(out, want)
