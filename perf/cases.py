"""The work a user has this framework do, as timed cases.

Each case is one call (or one plan replay) through the public Python entry
points, with device-resident float32 inputs made from a seed. The families
and their ranges are the benchmark's own configurations and the options the
entry points take:

  sgemm        the benchmark's launch: niter independent n x n products
  gemm         one general product in a chosen arithmetic form, row-major or
               transposed operands, round and odd sizes, uniform or wide-range
               values (the scaled forms exist for the latter)
  grouped      a planned batch of uneven products, replayed
  jacobi       one 7-point step on an nx x ny x nz grid
  bs_records   Black-Scholes pricing of option records in place
  bs_arrays    the same on separate arrays
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hb_hammerbench_b200 as hb
from hb_hammerbench_b200 import blackscholes as bs

PRODUCTS = {"ffma": 1, "bf16x3": 3, "bf16x6": 6, "bf16x3_scaled": 3, "bf16x6_scaled": 6}


def _gemm(name, m, n, k, variant, ta=False, tb=False, dist="uniform"):
    c = {"family": "gemm", "m": m, "n": n, "k": k, "variant": variant, "ta": ta, "tb": tb,
         "dist": dist}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the benchmark's registered launch N_512__NITER_2 in plain FP32: a
        # small batch, a few microseconds of arithmetic
        {"name": "sgemm_512x2", "family": "sgemm", "n": 512, "niter": 2},
        # the square sweep of the plain FP32 kernel at an ordinary size
        {"name": "sgemm_4096", "family": "sgemm", "n": 4096, "niter": 1},
        # plain FP32 with a transposed A and odd sizes: the rectangular
        # interface, where no row starts on a 16-byte boundary
        _gemm("ffma_ragged_ta", 1531, 1009, 2047, "ffma", ta=True),
        # a small square in the 6-product form: several short launches
        _gemm("x6_1024", 1024, 1024, 1024, "bf16x6"),
        # the headline product
        _gemm("x6_8192", 8192, 8192, 8192, "bf16x6"),
        # wide-range values through the scaled 3-product form at odd sizes
        _gemm("x3_scaled_ragged", 3001, 2503, 3607, "bf16x3_scaled", dist="wide"),
        # small output, very long K (accumulation of a long reduction)
        _gemm("x6_long_k", 256, 256, 1048576, "bf16x6"),
        # tall, narrow output
        _gemm("x6_tall", 65536, 64, 4096, "bf16x6"),
        # the uneven batch of 512 products, planned once and replayed
        {"name": "grouped_x6_512", "family": "grouped", "count": 512, "shape_seed": 0,
         "variant": "bf16x6"},
        # a stencil step on a grid well beyond L2
        {"name": "jacobi_512", "family": "jacobi", "nx": 512, "ny": 512, "nz": 512},
        # the option benchmark's whole input file, records in place
        {"name": "bs_records_10m", "family": "bs_records", "n": 10000000},
        # a mid-sized book held as separate arrays, an odd count
        {"name": "bs_arrays_1m", "family": "bs_arrays", "n": 1000003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Log-uniform size; two in five are taken as they fall (mostly odd or
    ragged), the others rounded to a multiple of 32 as users tend to choose."""
    x = _log(rng, lo, hi)
    if rng.random() < 0.6:
        x = max(32, (x + 16) // 32 * 32)
    return max(lo, min(hi, x))


def draw(rng):
    kind = rng.choice(["sgemm", "ffma", "split", "split", "long_k", "tall", "grouped", "jacobi",
                       "bs"])
    if kind == "sgemm":
        n = _size(rng, 64, 4096)
        niter = rng.randint(1, 4) if n <= 2048 else 1
        return {"family": "sgemm", "n": n, "niter": niter}
    if kind == "ffma":
        return _gemm(None, _size(rng, 64, 3000), _size(rng, 64, 3000), _size(rng, 64, 4096),
                     "ffma", ta=rng.random() < 0.3, tb=rng.random() < 0.3)
    if kind == "split":
        variant = rng.choice(["bf16x3", "bf16x6", "bf16x3_scaled", "bf16x6_scaled"])
        return _gemm(None, _size(rng, 128, 8192), _size(rng, 128, 8192), _size(rng, 128, 8192),
                     variant, ta=rng.random() < 0.2, tb=rng.random() < 0.2,
                     dist="wide" if variant.endswith("scaled") else "uniform")
    if kind == "long_k":
        return _gemm(None, _size(rng, 64, 512), _size(rng, 64, 256), _size(rng, 32768, 1048576),
                     rng.choice(["bf16x3", "bf16x6"]))
    if kind == "tall":
        return _gemm(None, _size(rng, 8192, 65536), _size(rng, 32, 128), _size(rng, 512, 4096),
                     rng.choice(["bf16x3", "bf16x6"]))
    if kind == "grouped":
        variant = rng.choice(["ffma", "bf16x3", "bf16x6", "bf16x6_scaled"])
        return {"family": "grouped", "count": _log(rng, 8, 128 if variant == "ffma" else 512),
                "shape_seed": rng.randint(1, 1 << 20), "variant": variant}
    if kind == "jacobi":
        return {"family": "jacobi", "nx": _size(rng, 8, 512), "ny": _size(rng, 8, 512),
                "nz": _size(rng, 32, 512)}
    return {"family": rng.choice(["bs_records", "bs_arrays"]), "n": _log(rng, 1000, 10000000)}


def _grouped_dims(case):
    """M, N, K of each product: multiples of 32 in [64, 2048]."""
    rng = np.random.Generator(np.random.PCG64(case["shape_seed"]))
    d = rng.integers(2, 65, size=(case["count"], 3)) * 32
    return [tuple(int(x) for x in row) for row in d]


def _values(count, seed, dist="uniform"):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(count, device="cuda", generator=g) * 2 - 1
    if dist == "wide":
        u = torch.rand(count, device="cuda", generator=g) * 40 - 20
        x = torch.sign(x) * torch.exp2(u)
    return x


def _operands(case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    buf = _values(m * k + k * n, seed, case["dist"])
    a, b = buf[:m * k].clone(), buf[m * k:].clone()  # each on its own allocation
    return (a.view(k, m) if case["ta"] else a.view(m, k),
            b.view(n, k) if case["tb"] else b.view(k, n))


def _grouped_operands(case, seed):
    dims = _grouped_dims(case)
    buf = _values(sum(m * k + k * n for m, n, k in dims), seed)
    As, Bs, off = [], [], 0
    for m, n, k in dims:
        As.append(buf[off:off + m * k].view(m, k))
        off += m * k
        Bs.append(buf[off:off + k * n].view(k, n))
        off += k * n
    return As, Bs


def _options(n, seed):
    """Option fields over the benchmark input's ranges: spot 40-100, spot /
    strike 0.82-1.22 with one in eight at the money, rate 0.0275-0.1,
    volatility 0.05-0.65, maturity 0.05-1 year."""
    u = _values(6 * n, seed).view(6, n) * 0.5 + 0.5
    s = 40 + 60 * u[0]
    strike = torch.where(u[5] < 0.125, s, s / (0.82 + 0.40 * u[1]))
    return [s.contiguous(), strike.contiguous(), 0.0275 + 0.0725 * u[2], 0.05 + 0.60 * u[3],
            0.05 + 0.95 * u[4]]


def prepare(case, seed):
    f = case["family"]
    st = {"case": case}
    if f == "sgemm":
        n, niter = case["n"], case["niter"]
        buf = _values(2 * niter * n * n, seed).view(2, niter, n, n)
        st.update(a=buf[0].clone(), b=buf[1].clone(),
                  c=torch.empty((niter, n, n), device="cuda"))
    elif f == "gemm":
        a, b = _operands(case, seed)
        st.update(a=a, b=b, c=torch.empty((case["m"], case["n"]), device="cuda"))
    elif f == "grouped":
        As, Bs = _grouped_operands(case, seed)
        # the outputs lie one after another in one buffer
        out = torch.empty(sum(a.shape[0] * b.shape[1] for a, b in zip(As, Bs)), device="cuda")
        Cs, off = [], 0
        for a, b in zip(As, Bs):
            size = a.shape[0] * b.shape[1]
            Cs.append(out[off:off + size].view(a.shape[0], b.shape[1]))
            off += size
        st.update(plan=hb.GroupedPlan(As, Bs, Cs, variant=case["variant"]), out=out)
    elif f == "jacobi":
        n = case["nx"] * case["ny"] * case["nz"]
        st.update(grid=_values(n, seed), out=torch.empty(n, device="cuda"))
    elif f == "bs_records":
        rec = torch.zeros((case["n"], bs.RECORD_FLOATS), device="cuda")
        for i, x in enumerate(_options(case["n"], seed)):
            rec[:, i] = x
        st["records"] = rec
    else:
        st["fields"] = _options(case["n"], seed)
        st["call"] = torch.empty(case["n"], device="cuda")
        st["put"] = torch.empty(case["n"], device="cuda")
    return st


def run(st):
    case = st["case"]
    f = case["family"]
    if f == "sgemm":
        return hb.sgemm(st["a"], st["b"], st["c"])
    if f == "gemm":
        return hb.gemm(st["a"], st["b"], st["c"], variant=case["variant"], trans_a=case["ta"],
                       trans_b=case["tb"])
    if f == "grouped":
        st["plan"].run()
        return st["out"]
    if f == "jacobi":
        return hb.jacobi(st["grid"], case["nx"], case["ny"], case["nz"], out=st["out"])
    if f == "bs_records":
        return bs.price(st["records"])
    return bs.price_arrays(*st["fields"], call=st["call"], put=st["put"])


def work(case):
    """Bytes: inputs read once, outputs written once. Operations: for products
    2*M*N*K for each product of the arithmetic form (1, 3 or 6)."""
    f = case["family"]
    if f == "sgemm":
        n, niter = case["n"], case["niter"]
        return {"bytes": 12 * niter * n * n, "flops": 2 * niter * n ** 3}
    if f == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + k * n + m * n),
                "flops": 2 * m * n * k * PRODUCTS[case["variant"]]}
    if f == "grouped":
        d = _grouped_dims(case)
        return {"bytes": sum(4 * (m * k + k * n + m * n) for m, n, k in d),
                "flops": sum(2 * m * n * k for m, n, k in d) * PRODUCTS[case["variant"]]}
    if f == "jacobi":
        pts = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8 * pts, "flops": 8 * pts}
    if f == "bs_records":  # the 32-byte record is the unit of memory traffic each way
        return {"bytes": 64 * case["n"], "flops": 100 * case["n"]}
    return {"bytes": 28 * case["n"], "flops": 100 * case["n"]}


def _price64(s, strike, r, v, t):
    s, strike, r, v, t = (x.double() for x in (s, strike, r, v, t))
    den = v * torch.sqrt(t)
    d1 = (torch.log(s / strike) + (r + 0.5 * v * v) * t) / den
    n1 = 0.5 * torch.special.erfc(-d1 / math.sqrt(2.0))
    n2 = 0.5 * torch.special.erfc(-(d1 - den) / math.sqrt(2.0))
    fv = strike * torch.exp(-r * t)
    return s * n1 - fv * n2, fv * (1.0 - n2) - s * (1.0 - n1)


def exact(case, seed):
    f = case["family"]
    if f == "sgemm":
        n, niter = case["n"], case["niter"]
        buf = _values(2 * niter * n * n, seed).view(2, niter, n, n)
        return torch.bmm(buf[0].double(), buf[1].double())
    if f == "gemm":
        a, b = _operands(case, seed)
        a, b = a.double(), b.double()
        return (a.t() if case["ta"] else a) @ (b.t() if case["tb"] else b)
    if f == "grouped":
        As, Bs = _grouped_operands(case, seed)
        return torch.cat([(a.double() @ b.double()).reshape(-1) for a, b in zip(As, Bs)])
    if f == "jacobi":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        g = torch.zeros((ny + 2, nx + 2, nz + 2), dtype=torch.float64, device="cuda")
        g[1:-1, 1:-1, 1:-1] = _values(nx * ny * nz, seed).view(ny, nx, nz)
        nb = g[1:-1, :-2, 1:-1] + g[1:-1, 2:, 1:-1] + g[:-2, 1:-1, 1:-1] + g[2:, 1:-1, 1:-1]
        nb = nb + g[1:-1, 1:-1, :-2] + g[1:-1, 1:-1, 2:]
        return (4.0 * nb - 2.0 * g[1:-1, 1:-1, 1:-1]).reshape(-1)
    fields = _options(case["n"], seed)
    call, put = _price64(*fields)
    if f == "bs_arrays":
        return call, put
    out = torch.zeros((case["n"], bs.RECORD_FLOATS), dtype=torch.float64, device="cuda")
    for i, x in enumerate(fields):
        out[:, i] = x
    out[:, 5], out[:, 6] = call, put
    return out
