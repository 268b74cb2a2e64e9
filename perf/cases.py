"""Performance cases of the batched ML-KEM NTT engine: the calls that programs
make through the Python entry points, at the sizes they make them.

A case is a dict of plain values.  ``kind`` names the call:

  ntt, invntt   one transform of n polynomials, out of place
  roundtrip     ntt out of place, then invntt in place on its output (the
                headline benchmark's step)
  small         ntt_small: coefficients in [-3, 3] (ML-KEM secrets and noise)
  packed        ntt_packed: 2- or 3-bit packed secrets
  matvec        matrix-vector jobs on device buffers, jobs2 / jobs3 / jobs4 of
                k = 2 / 3 / 4 (ML-KEM-512 / 768 / 1024) in one call
  matvec_host   one request of jobs on page-locked host buffers, inputs back
                to back, as a service without the server would run it

``values`` says what the int16 coefficients are: "canonical" [0, q), "centred"
[-(q-1)/2, (q-1)/2] or "int16" (the full accepted range).
"""
import functools

import torch

import tensorkyber_b200 as tk

Q = 3329
N = 256


def listed():
    return [
        # one ML-KEM-768 vector: the latency of a single call
        {"name": "ntt_3", "kind": "ntt", "n": 3, "values": "canonical"},
        # a service's small batch on the way back from the NTT domain
        {"name": "invntt_1021", "kind": "invntt", "n": 1021, "values": "canonical"},
        # ordinary ragged batches, each direction
        {"name": "ntt_16411", "kind": "ntt", "n": 16411, "values": "centred"},
        {"name": "invntt_100003", "kind": "invntt", "n": 100003, "values": "canonical"},
        # the headline workload: forward and inverse of 262,144 polynomials
        {"name": "roundtrip_262144", "kind": "roundtrip", "n": 262144, "values": "canonical"},
        # offline bulk work, at the full accepted input range
        {"name": "ntt_1048575", "kind": "ntt", "n": 1048575, "values": "int16"},
        # noise polynomials of a key-generation batch
        {"name": "small_40009", "kind": "small", "n": 40009},
        # packed secrets: a bulk batch of ternary ones and an ordinary 3-bit one
        {"name": "packed2_1048576", "kind": "packed", "n": 1048576, "bits": 2},
        {"name": "packed3_20011", "kind": "packed", "n": 20011, "bits": 3},
        # A s + e: a handful of ML-KEM-768 jobs, and a bulk mix of all three sets
        {"name": "matvec_24", "kind": "matvec", "jobs2": 0, "jobs3": 24, "jobs4": 0, "e": True},
        {"name": "matvec_65536", "kind": "matvec", "jobs2": 21846, "jobs3": 21845,
         "jobs4": 21845, "e": True},
        # one request from host memory and back
        {"name": "matvec_host_37", "kind": "matvec_host", "jobs2": 0, "jobs3": 0, "jobs4": 37,
         "e": True},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["ntt", "invntt", "ntt", "invntt", "roundtrip", "small", "packed",
                       "matvec", "matvec", "matvec_host"])
    case = {"kind": kind}
    if kind in ("ntt", "invntt", "roundtrip"):
        case["n"] = _log_int(rng, 1, 262144 if kind == "roundtrip" else 1048576)
        case["values"] = rng.choice(["canonical", "centred", "int16"])
    elif kind in ("small", "packed"):
        case["n"] = _log_int(rng, 1, 1048576)
        if kind == "packed":
            case["bits"] = rng.choice([2, 3])
    else:
        jobs = _log_int(rng, 1, 64 if kind == "matvec_host" else 65536)
        split = {"jobs2": 0, "jobs3": 0, "jobs4": 0}
        if jobs >= 3 and rng.random() < 0.5:  # a mix of the three sets
            # at most a third of the jobs at k = 4: no dearer than the listed mix
            split["jobs4"] = rng.randint(0, jobs // 3)
            split["jobs3"] = rng.randint(0, jobs // 3)
            split["jobs2"] = jobs - split["jobs4"] - split["jobs3"]
        else:
            k = rng.choice([2, 3, 4])
            split[f"jobs{k}"] = jobs if k < 4 else max(1, jobs * 2 // 3)
        case.update(split)
        case["e"] = rng.random() < 0.75
    return case


def _batches(case):
    return [(k, case[f"jobs{k}"]) for k in (2, 3, 4) if case[f"jobs{k}"]]


def _uniform(shape, lo, hi, gen):
    """int16 uniform in [lo, hi] on the GPU."""
    return torch.randint(lo, hi + 1, shape, generator=gen, device="cuda", dtype=torch.int16)


def _inputs(case, seed):
    """The call's input tensors on the GPU, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("ntt", "invntt", "roundtrip"):
        lo, hi = {"canonical": (0, Q - 1), "centred": (-(Q - 1) // 2, (Q - 1) // 2),
                  "int16": (-32768, 32767)}[case["values"]]
        return _uniform((case["n"], N), lo, hi, gen)
    if kind == "small":
        return _uniform((case["n"], N), -3, 3, gen)
    if kind == "packed":
        # fields of every value the format has: random bytes are 4 fields of
        # 2 bits, or 2 fields of 3 bits with the top two bits clear
        row, top = (64, 255) if case["bits"] == 2 else (128, 63)
        return _uniform((case["n"], row), 0, top, gen).to(torch.uint8)
    out = []
    for k, jobs in _batches(case):
        A = _uniform((jobs, k, k, N), 0, Q - 1, gen)  # NTT-domain, uniform
        s = _uniform((jobs, k, N), -3, 3, gen)
        e = _uniform((jobs, k, N), -3, 3, gen) if case["e"] else None
        out.append((k, A, s, e))
    return out


def _pinned(jobs, k, A, s, e):
    """A | s | e back to back in one page-locked buffer, and a page-locked out."""
    parts = [A, s] + ([e] if e is not None else [])
    buf = torch.empty(sum(t.numel() for t in parts), dtype=torch.int16, pin_memory=True)
    views, at = [], 0
    for t in parts:
        view = buf[at:at + t.numel()].view(t.shape)
        view.copy_(t)
        views.append(view.numpy())
        at += t.numel()
    out = torch.empty((jobs, k, N), dtype=torch.int16, pin_memory=True)
    return (k, views[0], views[1], views[2] if e is not None else None, out.numpy())


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "matvec":
        return kind, [(k, A, s, e, torch.empty_like(s)) for k, A, s, e in x]
    if kind == "matvec_host":
        return kind, [_pinned(s.shape[0], k, A, s, e) for k, A, s, e in x]
    out = torch.empty((case["n"], N), dtype=torch.int16, device="cuda")
    return kind, x, out, case.get("bits")


def run(state):
    kind = state[0]
    if kind == "matvec":
        tk.matvec(state[1])
        return [batch[4] for batch in state[1]]
    if kind == "matvec_host":
        tk.matvec_host(state[1])
        return [batch[4] for batch in state[1]]
    _, x, out, bits = state
    if kind == "ntt":
        return tk.ntt(x, out=out)
    if kind == "invntt":
        return tk.invntt(x, out=out)
    if kind == "small":
        return tk.ntt_small(x, out=out)
    if kind == "packed":
        return tk.ntt_packed(x, bits, out=out)
    tk.ntt(x, out=out)
    return tk.invntt(out)


def work(case):
    """Bytes: each input read once and each output written once.  Operations:
    7 layers of 128 butterflies (a product, a sum and a difference) per
    transform, and 128 degree-1 products per pair of polynomials."""
    kind = case["kind"]
    ntt_ops, mul_ops, poly = 7 * 128 * 3, 128 * 8, 2 * N
    if kind in ("matvec", "matvec_host"):
        nbytes = flops = 0
        for k, jobs in _batches(case):
            nbytes += jobs * (k * k + k * (3 if case["e"] else 2)) * poly
            flops += jobs * (2 * k * ntt_ops + k * k * mul_ops + (k * N if case["e"] else 0))
        return {"bytes": nbytes, "flops": flops}
    n = case["n"]
    if kind == "roundtrip":  # two calls, each with its input and its output
        return {"bytes": n * 4 * poly, "flops": n * 2 * ntt_ops}
    row = {"packed": 32 * 2 if case.get("bits") == 2 else 128}.get(kind, poly)
    return {"bytes": n * (row + poly), "flops": n * ntt_ops}


# ------------------------------------------------------------------ exact ----
@functools.lru_cache(maxsize=None)
def _constants():
    """The 128-point transform of the even (and of the odd) coefficients, its
    inverse times 2^16, and the pair roots, as float64 / int64 on the GPU."""
    def brv7(i):
        return int(f"{i:07b}"[::-1], 2)
    exps = [2 * brv7(i) + 1 for i in range(128)]
    fwd = [[pow(17, e * j, Q) for j in range(128)] for e in exps]
    scale = 2 ** 16 * pow(128, -1, Q) % Q
    inv = [[scale * pow(17, -e * j, Q) % Q for e in exps] for j in range(128)]
    roots = [pow(17, e, Q) for e in exps]
    return (torch.tensor(fwd, dtype=torch.float64, device="cuda"),
            torch.tensor(inv, dtype=torch.float64, device="cuda"),
            torch.tensor(roots, dtype=torch.int64, device="cuda"))


def _transform(matrix, x):
    """matrix applied to the even and to the odd coefficients, mod q in
    [0, q); exact in float64 (sums below 2^53)."""
    out = torch.empty(x.shape, dtype=torch.int64, device="cuda")
    flat_in, flat_out = x.reshape(-1, 128, 2), out.view(-1, 128, 2)
    for at in range(0, flat_in.shape[0], 131072):
        v = flat_in[at:at + 131072].to(torch.float64)
        for parity in (0, 1):
            y = v[:, :, parity] @ matrix.T
            flat_out[at:at + 131072, :, parity] = y.to(torch.int64).remainder_(Q)
    return out


def _centred(x):
    return torch.where(x > (Q - 1) // 2, x - Q, x)


def _unpacked(packed, bits):
    per = 8 // bits
    fields = [(packed >> (bits * i)) & ((1 << bits) - 1) for i in range(per)]
    v = torch.stack(fields, dim=-1).to(torch.int16).reshape(packed.shape[0], N)
    return torch.where(v >= 1 << (bits - 1), v - (1 << bits), v)


def exact(case, seed):
    x = _inputs(case, seed)
    fwd, inv, roots = _constants()
    kind = case["kind"]
    if kind in ("matvec", "matvec_host"):
        outs = []
        for k, A, s, e in x:
            b = _transform(fwd, s)
            b0, b1 = b[..., 0::2], b[..., 1::2]
            acc = torch.empty_like(b)
            for i in range(k):
                a = A[:, i].to(torch.int64)
                a0, a1 = a[..., 0::2], a[..., 1::2]
                acc[:, i, 0::2] = (a0 * b0 + a1 * b1 % Q * roots).sum(1)
                acc[:, i, 1::2] = (a0 * b1 + a1 * b0).sum(1)
            acc = acc.remainder_(Q) * pow(2, -16, Q) % Q
            y = _centred(_transform(inv, acc))
            if e is not None:
                y = y + e
            y = y.to(torch.int16)
            outs.append(y.cpu().numpy() if kind == "matvec_host" else y)
        return outs
    if kind == "packed":
        x = _unpacked(x, case["bits"])
    if kind == "invntt":
        return _centred(_transform(inv, x)).to(torch.int16)
    y = _transform(fwd, x)
    if kind == "roundtrip":
        y = _centred(_transform(inv, y))
    return y.to(torch.int16)
