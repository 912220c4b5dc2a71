"""Workloads that the performance of this framework is measured on, each through its public entry
points: base-2 nets (one fused call, the plain calls, a batched plan), rank-1 lattices, Halton points
(the fused plan, the plain calls on digits, the qrng form), nested uniform scrambling, and the fast
transforms.  A case is a dict: "kind" names the path, the rest are its sizes and options."""
import math

import numpy as np
import torch

import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import batch, halton, tc_fft
from qmctoolscl_gb300.c_funcs import halton_qrng_c

DEV = "cuda"
U = np.uint64


def listed():
    return [
        # one small point set inside a user's loop (an integrand evaluated a thousand points at a time):
        # generation, digital shift and float in one call, where the call itself is the cost
        dict(name="net_call", kind="net_call", r=1, n=1000, d=5, m=16),
        # the plain calls one after the other, as a program written for the reference makes them
        dict(name="net_chain", kind="net_chain", r=8, n=100003, d=21, m=17, order="gray"),
        # a batch of uneven requests in a plan (LMS, order-2 interlacing, digital shift), new matrices each pass
        dict(name="net_plan", kind="net_plan", requests=48, log2n_lo=12, log2n_hi=17, d_lo=8, d_hi=64, r=3),
        # the large shifted lattice of the benchmark
        dict(name="lattice", kind="lattice", r=16, n=1 << 20, d=64, order="gray"),
        # randomised Halton points in the first 100 primes, the benchmark's, new randomisation each pass
        dict(name="halton", kind="halton", r=32, n=1 << 18, d=100, perms=True, shifts=True),
        # the plain calls on base-b digits: matrix scramble, generation, digital shift, float
        dict(name="gdn_chain", kind="gdn_chain", r=16, n=65536, d=4, tmax=32, step="shift"),
        # qrng's generalized Halton sequence
        dict(name="qrng", kind="qrng", n=1 << 20, d=100, n0=0, generalized=1),
        # long FP64 transforms (the eigenvalues of a large lattice kernel matrix, several right-hand sides)
        dict(name="fft_long", kind="fft", d1=4, d2=8, m=20),
        # many short inverse transforms
        dict(name="ifft_short", kind="ifft", d1=37, d2=3, m=10),
        # FP64 Walsh-Hadamard transforms of middling length
        dict(name="fwht", kind="fwht", d1=300, d2=1, m=16),
        # the fast kernel matrix-vector product on the tensor cores, the operand kept
        dict(name="kernel_product", kind="product", d1=100, d2=1, m=16, form="tc", divide=False),
        # nested uniform (Owen) scrambling of net points
        dict(name="owen", kind="owen", r=4, n=200000, d=8, m=18),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["net_call", "net_chain", "net_plan", "lattice", "halton", "gdn_chain", "qrng", "fft", "ifft",
                       "fwht", "product", "owen"])
    if kind == "net_call":
        return dict(kind=kind, r=rng.randint(1, 4), n=_log(rng, 100, 1 << 16), d=_log(rng, 1, 64), m=16)
    if kind == "net_chain":
        order = rng.choice(["natural", "gray"])
        n = 1 << rng.randint(10, 17) if order == "natural" else _log(rng, 1000, 1 << 17)
        return dict(kind=kind, r=_log(rng, 1, 16), n=n, d=_log(rng, 1, 64), m=17, order=order)
    if kind == "net_plan":
        lo = rng.randint(9, 13)
        return dict(kind=kind, requests=_log(rng, 1, 60), log2n_lo=lo, log2n_hi=lo + rng.randint(1, 4),
                    d_lo=rng.randint(1, 16), d_hi=rng.randint(17, 64), r=rng.randint(1, 3))
    if kind == "lattice":
        order = rng.choice(["natural", "gray"])
        n = 1 << rng.randint(8, 20) if order == "natural" else _log(rng, 200, 1 << 20)
        return dict(kind=kind, r=_log(rng, 1, 16), n=n, d=_log(rng, 1, 64), order=order)
    if kind == "halton":
        perms = rng.random() < 0.6
        return dict(kind=kind, r=_log(rng, 1, 32), n=_log(rng, 1000, 1 << 18), d=_log(rng, 1, 100), perms=perms,
                    shifts=(not perms) or rng.random() < 0.5)
    if kind == "gdn_chain":
        return dict(kind=kind, r=_log(rng, 1, 16), n=_log(rng, 1000, 65536), d=rng.randint(1, 4),
                    tmax=rng.randint(16, 32), step=rng.choice(["shift", "perm"]))
    if kind == "qrng":
        return dict(kind=kind, n=_log(rng, 1000, 1 << 20), d=_log(rng, 1, 100), n0=rng.choice([0, 1, 12345]),
                    generalized=rng.randint(0, 1))
    if kind == "owen":
        return dict(kind=kind, r=rng.randint(1, 4), n=_log(rng, 2000, 200000), d=rng.randint(1, 8), m=18)
    m = rng.randint(8, 20)
    most = (1 << 24) >> m  # vectors: at most 2^24 values in all, every length alike
    vectors = _log(rng, 1, min(most, 3000))
    d2 = rng.randint(1, 3) if vectors >= 6 else 1
    case = dict(kind=kind, d1=max(1, vectors // d2), d2=d2, m=m)
    if kind == "product":
        case.update(form=rng.choice(["tc", "fp64", "walsh"]), divide=rng.random() < 0.4)
    return case


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2 + 1)


def _primes(k):
    out, v = [], 2
    while len(out) < k:
        if all(v % p for p in out if p * p <= v):
            out.append(v)
        v += 1
    return out


def _bits(g, shape, bits):
    """Uniform integers of `bits` bits (up to 64) as int64 words."""
    hi = torch.randint(0, 1 << 32, shape, generator=g, device=DEV)
    lo = torch.randint(0, 1 << 32, shape, generator=g, device=DEV)
    w = (hi << 32) | lo
    return w if bits == 64 else w & ((1 << bits) - 1)


def _net_matrices(g, lead, m, bits):
    """Upper-unit-triangular random generating matrices: column k is a word whose bit k from the top is
    set, the bits above it random, those below zero."""
    k = torch.arange(m, device=DEV)
    diag = torch.ones(m, dtype=torch.int64, device=DEV) << (bits - 1 - k)
    above = _bits(g, lead + (m,), bits) & ~(diag - 1) & ~diag
    return (above | diag).contiguous()


def _halton_dims(case, g, bases):
    r, n = case["r"], case["n"]
    dims = []
    for b in bases:
        tmax = math.ceil(64 / math.log2(b))
        mmax, v = 0, n - 1
        while v:
            v //= b
            mmax += 1
        mmax = max(1, mmax)
        C = torch.zeros((mmax, tmax), dtype=torch.int64, device=DEV)
        C[torch.arange(mmax), torch.arange(mmax)] = 1
        S = torch.tril(torch.randint(0, b, (r, tmax, tmax), generator=g, device=DEV), -1)
        S += torch.eye(tmax, dtype=torch.int64, device=DEV)
        dim = dict(b=b, tmax=tmax, mmax=mmax, C=C, S=S)
        if case["perms"]:
            dim["perms"] = torch.rand((r, tmax, b), generator=g, device=DEV).argsort(dim=2).contiguous()
        if case["shifts"]:
            dim["shifts"] = torch.randint(0, b, (r, tmax), generator=g, device=DEV)
        dims.append(dim)
    return dims


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case=case)
    f64, i64 = torch.float64, torch.int64
    if kind in ("net_call", "net_chain"):
        r, n, d, m = case["r"], case["n"], case["d"], case["m"]
        s.update(C=_net_matrices(g, (r, d), m, 63), shifts=_bits(g, (r, d), 63),
                 lshifts=torch.zeros(r, dtype=i64, device=DEV), tmaxes=torch.full((r,), 63, dtype=i64, device=DEV),
                 x=torch.empty((r, n, d), dtype=f64, device=DEV))
        if kind == "net_chain":
            s.update(xb=torch.empty((r, n, d), dtype=i64, device=DEV), xrb=torch.empty((r, n, d), dtype=i64, device=DEV))
    elif kind == "net_plan":
        shape = np.random.default_rng(1)  # the requests' sizes are the program's, the same whatever the inputs
        reqs = []
        for _ in range(case["requests"]):
            log2n = int(shape.integers(case["log2n_lo"], case["log2n_hi"] + 1))
            n = (1 << log2n) - int(shape.integers(0, 2)) * int(shape.integers(0, 1 << (log2n - 1)))
            d, r = int(shape.integers(case["d_lo"], case["d_hi"] + 1)), int(shape.integers(1, case["r"] + 1))
            low = torch.tensor([1 << (63 - t) if t else -(1 << 63) for t in range(64)], dtype=i64, device=DEV)
            S = (_bits(g, (r, 2 * d, 64), 64) & ~(low - 1) & ~low) | low
            reqs.append(dict(r=r, n=n, d=d, n_start=0, mmax=log2n, d_pre=2 * d, alpha=2, tmax=64, tmax_new=64,
                             tmax_alpha=64, r_C=1, order=("gray", "natural")[int(shape.integers(0, 2))] if
                             n == 1 << log2n else "gray", C=_net_matrices(g, (1, 2 * d), log2n, 63) << 1, S=S,
                             lshifts=torch.zeros(r, dtype=i64, device=DEV), shifts=_bits(g, (r, d), 64),
                             xb=torch.empty((r, n, d), dtype=i64, device=DEV)))
        s.update(plan=batch.NetPlan(reqs), reqs=reqs)
    elif kind == "lattice":
        r, n, d = case["r"], case["n"], case["d"]
        s.update(g=torch.randint(0, 1 << 19, (r, d), generator=g, device=DEV) * 2 + 1,
                 shifts=torch.rand((r, d), generator=g, device=DEV, dtype=f64),
                 x=torch.empty((r, n, d), dtype=f64, device=DEV))
    elif kind == "halton":
        dims = _halton_dims(case, g, _primes(case["d"]))
        x = torch.empty((case["r"], case["n"], case["d"]), dtype=f64, device=DEV)
        s.update(dims=dims, x=x, plan=halton.HaltonPlan(case["r"], case["n"], 0, dims, x))
    elif kind == "gdn_chain":
        r, n, d, tmax = case["r"], case["n"], case["d"], case["tmax"]
        bases = torch.tensor(_primes(d), dtype=i64, device=DEV)
        mmax = min(17, tmax)
        bv = bases.view(1, d, 1, 1)
        S = torch.tril(_bits(g, (r, d, tmax, tmax), 40) % bv, -1) + torch.eye(tmax, dtype=i64, device=DEV)
        C = torch.zeros((1, d, mmax, tmax), dtype=i64, device=DEV)
        C[:, :, torch.arange(mmax), torch.arange(mmax)] = 1
        bmax = int(bases.max())
        order = torch.rand((r, d, tmax, bmax), generator=g, device=DEV) + \
            (torch.arange(bmax, device=DEV) >= bv) * 2.0
        s.update(bases=bases, bmax=bmax, mmax=mmax, S=S, C=C, C_lms=torch.empty((r, d, mmax, tmax), dtype=i64, device=DEV),
                 perms=order.argsort(dim=3).contiguous(), shifts=(_bits(g, (r, d, tmax), 40) % bases.view(1, d, 1)).contiguous(),
                 xdig=torch.empty((r, n, d, tmax), dtype=i64, device=DEV),
                 xnew=torch.empty((r, n, d, tmax), dtype=i64, device=DEV), x=torch.empty((r, n, d), dtype=f64, device=DEV))
    elif kind == "qrng":
        n, d = case["n"], case["d"]
        s.update(res=torch.empty(d * n, dtype=f64, device=DEV), randu=torch.rand(d * 32, generator=g, device=DEV, dtype=f64),
                 dvec=torch.arange(d, dtype=torch.int32, device=DEV))
    elif kind == "owen":
        r, n, d, m = case["r"], case["n"], case["d"], case["m"]
        xb = torch.empty((1, n, d), dtype=i64, device=DEV)
        C = _net_matrices(g, (1, d), m, 63) << 1
        q.dnb2_gen_natural(U(1), U(1 << m), U(d), U(0), U(m), C,
                           full := torch.empty((1, 1 << m, d), dtype=i64, device=DEV))
        xb.copy_(full[:, :n])
        s.update(xb=xb, xrb=torch.empty((r, n, d), dtype=i64, device=DEV), seed=int(seed))
    else:
        n, nv = 1 << case["m"], case["d1"] * case["d2"]
        shape = (case["d1"], case["d2"], n)
        form = case.get("form")
        s["xr"] = torch.randn(shape, generator=g, device=DEV, dtype=f64)
        if kind != "fwht" and form != "walsh":
            s["xi"] = torch.randn(shape, generator=g, device=DEV, dtype=f64)
        if kind in ("fft", "ifft"):
            s.update(twr=torch.empty(n, dtype=f64, device=DEV), twi=torch.empty(n, dtype=f64, device=DEV))
        if kind == "product":
            # eigenvalues of a kernel matrix: positive, decaying, a nugget below them
            k = torch.arange(n, dtype=f64, device=DEV)
            lam = 1e-3 + (1 + torch.rand(n, generator=g, device=DEV, dtype=f64)) / (1 + torch.minimum(k, n - k)) ** 1.5
            s.update(lam_r=lam, lam_i=torch.randn(n, generator=g, device=DEV, dtype=f64) * 1e-4,
                     yr=torch.empty_like(s["xr"]), yi=torch.empty_like(s["xr"]) if "xi" in s else None)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "net_call":
        batch.dnb2_gen_fused(c["r"], c["n"], c["d"], 0, c["m"], s["C"], order="gray", lshifts=s["lshifts"],
                             shiftsb=s["shifts"], tmaxes=s["tmaxes"], x=s["x"])
        return s["x"]
    if kind == "net_chain":
        r, n, d, m = U(c["r"]), U(c["n"]), U(c["d"]), U(c["m"])
        gen = q.dnb2_gen_gray if c["order"] == "gray" else q.dnb2_gen_natural
        gen(r, n, d, U(0), m, s["C"], s["xb"], wait=False)
        q.dnb2_digital_shift(r, n, d, r, s["lshifts"], s["xb"], s["shifts"], s["xrb"], wait=False)
        q.dnb2_integer_to_float(r, n, d, s["tmaxes"], s["xrb"], s["x"], wait=False)
        return s["xrb"], s["x"]
    if kind == "net_plan":
        s["plan"].run()
        return [p["xb"] for p in s["reqs"]]
    if kind == "lattice":
        batch.lattice_gen_shift(c["r"], c["n"], c["d"], 0, s["g"], s["shifts"], s["x"], order=c["order"])
        return s["x"]
    if kind == "halton":
        s["plan"].prepare()
        s["plan"].run()
        return s["x"]
    if kind == "gdn_chain":
        r, n, d, tmax, mmax = U(c["r"]), U(c["n"]), U(c["d"]), U(c["tmax"]), U(s["mmax"])
        q.gdn_linear_matrix_scramble(r, d, mmax, U(1), U(1), tmax, tmax, s["bases"], s["S"], s["C"], s["C_lms"],
                                     wait=False)
        q.gdn_gen_natural(r, n, d, U(1), mmax, tmax, U(0), s["bases"], s["C_lms"], s["xdig"], wait=False)
        if c["step"] == "shift":
            q.gdn_digital_shift(r, n, d, r, U(1), tmax, tmax, s["bases"], s["shifts"], s["xdig"], s["xnew"], wait=False)
        else:
            q.gdn_digital_permutation(r, n, d, r, U(1), tmax, tmax, U(s["bmax"]), s["perms"], s["xdig"], s["xnew"],
                                      wait=False)
        q.gdn_integer_to_float(r, n, d, U(1), tmax, s["bases"], s["xnew"], s["x"], wait=False)
        return s["xnew"], s["x"]
    if kind == "qrng":
        halton_qrng_c(c["n"], c["d"], c["n0"], c["generalized"], s["res"], s["randu"], s["dvec"])
        return s["res"]
    if kind == "owen":
        r, n, d = c["r"], c["n"], c["d"]
        rngs = [np.random.Generator(np.random.SFC64(k)) for k in np.random.SeedSequence(s["seed"]).spawn(r * d)]
        roots = [q.NUSNode_dnb2() for _ in range(r * d)]
        q.dnb2_nested_uniform_scramble(r, n, d, 1, 64, 64, rngs, roots, s["xb"], s["xrb"])
        return s["xrb"]
    d1, d2, nh = c["d1"], c["d2"], (1 << c["m"]) // 2
    if kind in ("fft", "ifft"):
        f = q.fft_bro_1d_radix2 if kind == "fft" else q.ifft_bro_1d_radix2
        f(U(d1), U(d2), U(nh), s["twr"], s["twi"], s["xr"], s["xi"], wait=False)
        return s["twr"], s["twi"], s["xr"], s["xi"]
    if kind == "fwht":
        q.fwht_1d_radix2(U(d1), U(d2), U(nh), s["xr"], wait=False)
        return s["xr"]
    s["yr"].copy_(s["xr"])  # a solver keeps its direction vector
    if c["form"] == "walsh":
        tc_fft.fwht_mul_fwht(d1, d2, nh, s["lam_r"], s["yr"], divide=c["divide"])
        return s["yr"]
    s["yi"].copy_(s["xi"])
    f = tc_fft.fft_mul_ifft_tc if c["form"] == "tc" else tc_fft.fft_mul_ifft
    f(d1, d2, nh, s["lam_r"], s["lam_i"], s["yr"], s["yi"], divide=c["divide"])
    return s["yr"], s["yi"]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    c, kind = case, case["kind"]
    if kind in ("net_call", "net_chain", "lattice", "halton", "qrng", "owen", "gdn_chain"):
        pts = c.get("r", 1) * c["n"] * c["d"]
    if kind == "net_call":
        return dict(bytes=8 * pts + 8 * c["r"] * c["d"] * (c["m"] + 1), flops=0)
    if kind == "net_chain":
        return dict(bytes=16 * pts, flops=0)
    if kind == "net_plan":
        shape, total = np.random.default_rng(1), 0
        for _ in range(c["requests"]):
            log2n = int(shape.integers(c["log2n_lo"], c["log2n_hi"] + 1))
            n = (1 << log2n) - int(shape.integers(0, 2)) * int(shape.integers(0, 1 << (log2n - 1)))
            d, r = int(shape.integers(c["d_lo"], c["d_hi"] + 1)), int(shape.integers(1, c["r"] + 1))
            if n == 1 << log2n:
                shape.integers(0, 2)
            total += 8 * r * n * d + 8 * 2 * d * (log2n + 64 * r)
        return dict(bytes=total, flops=0)
    if kind == "lattice":
        return dict(bytes=8 * pts, flops=2 * pts)
    if kind == "halton":
        digits = sum(math.ceil(64 / math.log2(b)) for b in _primes(c["d"]))
        return dict(bytes=8 * pts, flops=c["r"] * c["n"] * digits)
    if kind == "gdn_chain":
        return dict(bytes=8 * pts * (c["tmax"] + 1), flops=pts * c["tmax"])
    if kind == "qrng":
        return dict(bytes=8 * pts, flops=sum(2 * c["n"] * math.ceil(math.log(max(2, c["n"])) / math.log(b))
                                             for b in _primes(c["d"])))
    if kind == "owen":
        return dict(bytes=8 * pts + 8 * c["n"] * c["d"], flops=0)
    n = 1 << c["m"]
    values = c["d1"] * c["d2"] * n
    if kind in ("fft", "ifft"):
        return dict(bytes=32 * values + 16 * n, flops=5 * values * c["m"])
    if kind == "fwht":
        return dict(bytes=16 * values, flops=values * c["m"])
    if c["form"] == "walsh":
        return dict(bytes=16 * values + 8 * n, flops=2 * values * c["m"] + values)
    return dict(bytes=32 * values + 16 * n, flops=10 * values * c["m"] + 6 * values)


# ---------------------------------------------------------------- the same in plain torch, 64 bits

def _index_digits(n, b, count, start=0):
    """Base-b digits of start .. start+n-1, least significant first: (n, count) float64."""
    i = torch.arange(start, start + n, device=DEV)
    out = torch.empty((n, count), dtype=torch.float64, device=DEV)
    for k in range(count):
        out[:, k] = (i % b).to(torch.float64)
        i = i // b
    return out


def _digit_points(n, b, mmax, tmax, S, perms, shifts):
    """(digits, floats) of one randomisation and dimension: S is tmax x tmax, the matrix identity."""
    dig = (_index_digits(n, b, mmax) @ S[:, :mmax].to(torch.float64).T) % b  # whole numbers below 2^53
    dig = dig.to(torch.int64)
    if perms is not None:
        dig = torch.gather(perms, 1, dig.T.contiguous()).T
    if shifts is not None:
        dig = (dig + shifts) % b
    w = torch.tensor([float(b) ** -(t + 1) for t in range(tmax)], dtype=torch.float64, device=DEV)
    return dig, (dig.to(torch.float64) * w).sum(1)


def _net_points(C, m, n, order):
    """Integer points of base-2 matrices C (lead..., m): (lead..., n), from index 0."""
    i = torch.arange(n, device=DEV)
    if order == "gray":
        i = i ^ (i >> 1)
    out = torch.zeros(C.shape[:-1] + (n,), dtype=torch.int64, device=DEV)
    for k in range(m):
        out ^= C[..., k:k + 1] * ((i >> k) & 1)
    return out


def _bit_reverse(m):
    i = torch.arange(1 << m, device=DEV)
    out = torch.zeros_like(i)
    for k in range(m):
        out |= ((i >> k) & 1) << (m - 1 - k)
    return out


def _walsh(x):
    """Orthonormal Walsh-Hadamard transform along the last axis."""
    shape, n, h = x.shape, x.shape[-1], 1
    while h < n:
        v = x.reshape(-1, n // (2 * h), 2, h)
        x = torch.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), dim=2)
        h *= 2
    return x.reshape(shape) * n ** -0.5


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("net_plan", "owen"):
        return None  # whole numbers
    if kind == "qrng" and c["generalized"]:
        return None  # the multipliers' table is not plain arithmetic
    s = prepare(case, seed)
    if kind in ("net_call", "net_chain"):
        pts = _net_points(s["C"], c["m"], c["n"], c.get("order", "gray")) ^ s["shifts"][..., None]
        x = (pts.to(torch.float64) * 2.0 ** -63).transpose(1, 2).contiguous()
        return x if kind == "net_call" else [None, x]
    if kind == "lattice":
        i = torch.arange(c["n"], device=DEV)
        if c["order"] == "gray":
            i = i ^ (i >> 1)
        v = torch.zeros(c["n"], dtype=torch.float64, device=DEV)
        for k in range(21):
            v += ((i >> k) & 1).to(torch.float64) * 2.0 ** -(k + 1)
        return torch.stack([((s["g"][l].to(torch.float64) * v[:, None]) % 1.0 + s["shifts"][l]) % 1.0
                            for l in range(c["r"])])
    if kind == "halton":
        x = torch.empty((c["r"], c["n"], c["d"]), dtype=torch.float64, device=DEV)
        for j, dm in enumerate(s["dims"]):
            for l in range(c["r"]):
                x[l, :, j] = _digit_points(c["n"], dm["b"], dm["mmax"], dm["tmax"], dm["S"][l],
                                           dm["perms"][l] if c["perms"] else None,
                                           dm["shifts"][l] if c["shifts"] else None)[1]
        return x
    if kind == "gdn_chain":
        x = torch.empty((c["r"], c["n"], c["d"]), dtype=torch.float64, device=DEV)
        for j, b in enumerate(_primes(c["d"])):
            for l in range(c["r"]):
                x[l, :, j] = _digit_points(c["n"], b, s["mmax"], c["tmax"], s["S"][l, j],
                                           s["perms"][l, j] if c["step"] == "perm" else None,
                                           s["shifts"][l, j] if c["step"] == "shift" else None)[1]
        return [None, x]
    if kind == "qrng":
        n, d = c["n"], c["d"]
        u = s["randu"].reshape(d, 32)
        out = torch.empty((d, n), dtype=torch.float64, device=DEV)
        for j, b in enumerate(_primes(d)):
            dig = _index_digits(n, b, 32, c["n0"])
            v = torch.zeros(n, dtype=torch.float64, device=DEV)
            for k in range(31, -1, -1):
                v = (v + (dig[:, k] + torch.floor(u[j, k] * b)) % b) / b
            out[j] = v
        return out.reshape(-1)
    m, n = c["m"], 1 << c["m"]
    if kind == "fwht":
        return _walsh(s["xr"])
    if kind == "product" and c["form"] == "walsh":
        y = _walsh(s["xr"])
        return _walsh(y / s["lam_r"] if c["divide"] else y * s["lam_r"])
    rev = _bit_reverse(m)
    z = torch.complex(s["xr"], s["xi"])
    if kind == "fft":
        y = torch.fft.fft(z[..., rev], norm="ortho")
    elif kind == "ifft":
        y = torch.fft.ifft(z, norm="ortho")[..., rev]
    else:
        lam = torch.complex(s["lam_r"], s["lam_i"])
        y = torch.fft.fft(z[..., rev], norm="ortho")
        y = torch.fft.ifft(y / lam if c["divide"] else y * lam, norm="ortho")[..., rev]
        return y.real.contiguous(), y.imag.contiguous()
    a = torch.arange(n, dtype=torch.float64, device=DEV) * (2 * math.pi / n)
    return torch.cos(a), torch.sin(a) * (-1.0 if kind == "fft" else 1.0), y.real.contiguous(), y.imag.contiguous()
