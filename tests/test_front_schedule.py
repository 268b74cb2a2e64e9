"""CPU model of the batch kernels' work split (k_ntt_mma in tk_ntt_mma.cu): whole
tiles of W units round robin, the units left over split evenly into a last,
short tile per CTA, the inverse mirrored.  Every unit is computed exactly once,
CTAs differ by at most one unit, and the launch moves as one front."""
import pytest


def tiles(nunits, G, W, cta, inverse):
    """[(first unit, units)] of a CTA, in order."""
    whole = nunits // (G * W)
    left = nunits - whole * G * W
    left0, left1 = cta * left // G, (cta + 1) * left // G
    out = []
    for k in range(whole + (left1 > left0)):
        n = W if k < whole else left1 - left0
        i = (k * G + cta) * W if k < whole else whole * G * W + left0
        out.append((nunits - i - n if inverse else i, n))
    return out


@pytest.mark.parametrize("W", [4, 8])
@pytest.mark.parametrize("G", [1, 5, 296, 444, 592, 888])
@pytest.mark.parametrize("npoly", [1, 8, 9, 1000, 4737, 100003, 262144, (1 << 20) + 3])
def test_units_once_even_and_one_front(W, G, npoly):
    nunits = (npoly + 7) // 8
    G = min(G, nunits)
    for inverse in (False, True):
        seen, counts, lo = [0] * nunits, [], {}
        for cta in range(G):
            mine = tiles(nunits, G, W, cta, inverse)
            counts.append(sum(n for _, n in mine))
            for k, (u, n) in enumerate(mine):
                assert 0 < n <= W and 0 <= u and u + n <= nunits
                for i in range(u, u + n):
                    seen[i] += 1
                lo.setdefault(k, []).append((u, u + n))
        assert all(c == 1 for c in seen) and max(counts) - min(counts) <= 1
        # every tile k lies past every tile k - 1 of the launch
        for k in range(1, len(lo)):
            if inverse:
                assert max(b for _, b in lo[k]) <= min(a for a, _ in lo[k - 1])
            else:
                assert min(a for a, _ in lo[k]) >= max(b for _, b in lo[k - 1])
