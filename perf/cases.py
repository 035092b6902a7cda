"""The workloads this library is timed on, through its public Python entry points.

Every family below is one call (or one forward and backward pair) of
`magma_gb300`.  The listed sizes are those of the repository's benchmark and
tests, with small, odd and few-but-large ones beside them; `draw` spreads over
the same ranges.  Matrices are column-major storage (batch, ncols, ld), so
S[k, j, i] is A_k(i, j).  Routines that overwrite their operands work on copies
made in the pass, as a program does that still needs its matrices afterwards.
"""
from __future__ import annotations

import math

import torch

import magma_gb300 as mg
from magma_gb300 import autograd as mg_autograd

DTYPES = {"f64": torch.float64, "f32": torch.float32}


def listed():
    return [
        # a handful of very small systems: the latency of one call (a control loop, one element)
        {"name": "gesv_f64_tiny", "kind": "gesv", "dtype": "f64", "n": 8, "nrhs": 1, "batch": 16, "pad": 0},
        # many small systems at once: one per grid point or per finite element
        {"name": "gesv_f64_n32", "kind": "gesv", "dtype": "f64", "n": 32, "nrhs": 1, "batch": 10000, "pad": 0},
        # an odd order and a padded leading dimension, a few right-hand sides
        {"name": "gesv_f64_n100", "kind": "gesv", "dtype": "f64", "n": 100, "nrhs": 3, "batch": 1000, "pad": 4},
        # the largest: plain FP64 solves, which mixed precision is compared with
        {"name": "gesv_f64_n512", "kind": "gesv", "dtype": "f64", "n": 512, "nrhs": 4, "batch": 512, "pad": 0},
        # single precision, medium order
        {"name": "gesv_f32_n200", "kind": "gesv", "dtype": "f32", "n": 200, "nrhs": 8, "batch": 1000, "pad": 0},
        # a few large systems: fewer matrices than the GPU has SMs
        {"name": "gesv_f32_few_n1000", "kind": "gesv", "dtype": "f32", "n": 1000, "nrhs": 1, "batch": 6, "pad": 0},
        # factors kept by the program, new right-hand sides in each pass, both directions
        {"name": "getrs_f64_n150", "kind": "getrs", "dtype": "f64", "n": 150, "nrhs": 16, "batch": 500, "pad": 0},
        # matrices of mixed sizes in one call (fronts of a sparse factorisation)
        {"name": "vbatched_f64_4096", "kind": "vbatched", "dtype": "f64", "nmin": 8, "nmax": 256, "rmax": 16, "batch": 4096, "mix": 7},
        # mixed-precision refinement, the benchmark's workload
        {"name": "refine_n512", "kind": "refine", "n": 512, "nrhs": 4, "batch": 512, "pad": 0},
        # a differentiable layer that solves linear systems: forward and backward
        {"name": "solve_grad_f64_n64", "kind": "solve_grad", "dtype": "f64", "n": 64, "nrhs": 4, "batch": 2048},
        # a serving batch of mixed sizes with its gradients, refined from FP32 factors
        {"name": "refine_var_grad_256", "kind": "refine_var_grad", "nmin": 128, "nmax": 1024, "nrhs": 8, "batch": 256, "mix": 3},
        # symmetric positive definite systems (covariances, normal equations), refined
        {"name": "spd_refine_n256", "kind": "spd_refine", "n": 256, "nrhs": 2, "batch": 256, "pad": 0},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gesv", "gesv", "gesv", "getrs", "vbatched", "refine", "solve_grad",
                       "refine_var_grad", "spd_refine"])
    dtype = rng.choice(["f64", "f64", "f32"])
    while True:
        if kind == "gesv":
            c = {"kind": kind, "dtype": dtype, "n": _log(rng, 4, 1000), "nrhs": _log(rng, 1, 16),
                 "batch": _log(rng, 1, 20000), "pad": rng.choice([0, 0, 1, 4])}
            cost, most = c["batch"] * c["n"] ** 3, 512 * 512 ** 3
        elif kind == "getrs":
            c = {"kind": kind, "dtype": dtype, "n": _log(rng, 8, 600), "nrhs": _log(rng, 1, 64),
                 "batch": _log(rng, 1, 2000), "pad": rng.choice([0, 0, 1, 4])}
            cost, most = c["batch"] * c["n"] ** 2 * max(c["nrhs"], 8), 4 * 500 * 150 ** 2 * 16
        elif kind == "vbatched":
            hi = _log(rng, 24, 256)
            c = {"kind": kind, "dtype": dtype, "nmin": rng.randint(4, max(4, hi // 3)), "nmax": hi,
                 "rmax": rng.randint(1, 16), "batch": _log(rng, 64, 4096),
                 "mix": rng.randint(0, 999)}
            cost, most = 0, 1
        elif kind == "refine":
            c = {"kind": kind, "n": _log(rng, 40, 640), "nrhs": rng.randint(1, 8),
                 "batch": _log(rng, 4, 1000), "pad": rng.choice([0, 0, 3])}
            cost, most = c["batch"] * c["n"] ** 3, 512 * 512 ** 3
        elif kind == "solve_grad":
            c = {"kind": kind, "dtype": dtype, "n": _log(rng, 8, 200), "nrhs": rng.randint(1, 16),
                 "batch": _log(rng, 8, 4096)}
            cost, most = c["batch"] * c["n"] ** 3, 16 * 2048 * 64 ** 3
        elif kind == "refine_var_grad":
            hi = _log(rng, 128, 1024)
            c = {"kind": kind, "nmin": rng.randint(hi // 10, hi // 2), "nmax": hi,
                 "nrhs": rng.randint(1, 8), "batch": _log(rng, 8, 256), "mix": rng.randint(0, 999)}
            cost, most = 0, 1
        else:
            c = {"kind": kind, "n": _log(rng, 24, 512), "nrhs": rng.randint(1, 8),
                 "batch": _log(rng, 4, 600), "pad": rng.choice([0, 0, 3])}
            cost, most = c["batch"] * c["n"] ** 3, 4 * 256 * 256 ** 3
        if cost <= most:
            return c


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, shape, dtype=torch.float64):
    """uniform(-1, 1), as the reference's tester fills its matrices."""
    return torch.empty(shape, dtype=dtype, device="cuda").uniform_(-1.0, 1.0, generator=g)


def _padded(A, pad):
    """(batch, m, n) -> column-major storage with pad unused rows (zero) under every matrix."""
    S = torch.zeros((A.shape[0], A.shape[2], A.shape[1] + pad), dtype=A.dtype, device=A.device)
    S[:, :, :A.shape[1]] = A.transpose(1, 2)
    return S


def _cosines(n):
    """The orthogonal matrix of the type-2 cosine transform."""
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    C = torch.cos(math.pi / n * torch.outer(i, i + 0.5)) * math.sqrt(2.0 / n)
    C[0] *= math.sqrt(0.5)
    return C


def _signs(g, shape):
    return torch.randint(0, 2, shape, device="cuda", generator=g, dtype=torch.int64).double() * 2 - 1


def _svd_type(g, n, kappas):
    """A_k = U_k diag(s) V_k^T (batch, n, n), s geometric from 1 to 1/kappa_k, U_k and V_k
    orthogonal: sign changes, cosine transforms and a permutation of the singular values."""
    b = len(kappas)
    C = _cosines(n)
    K1, K2 = C @ (_signs(g, (n, 1)) * C.T), C @ (_signs(g, (n, 1)) * C.T)
    order = torch.rand((b, n), device="cuda", generator=g).argsort(1).double()
    lk = torch.tensor([math.log(k) for k in kappas], dtype=torch.float64, device="cuda")
    s = torch.exp(-order / max(n - 1, 1) * lk[:, None])
    A = (K1 * _signs(g, (b, n, 1)) * s[:, None, :]) @ K2
    return A * _signs(g, (b, 1, n))


def _general(g, c):
    """Uniform matrices; in single precision rows of a well-conditioned matrix in random
    order, so that a solution has correct digits whatever the batch."""
    n, b, dt = c["n"], c["batch"], DTYPES[c["dtype"]]
    A = _uniform(g, (b, n, n), dt)
    if dt == torch.float32:
        A += torch.eye(n, dtype=dt, device="cuda") * (2.0 * math.sqrt(n / 3.0))
        A = A[:, torch.randperm(n, device="cuda", generator=g), :]
    return A


def _sizes(c):
    """The orders of a variable-size batch: part of the case, the same for every seed."""
    g = torch.Generator().manual_seed(c["mix"])
    return torch.randint(c["nmin"], c["nmax"] + 1, (c["batch"],), generator=g).tolist()


def _nrhs_of(c):
    if "rmax" not in c:
        return [c["nrhs"]] * c["batch"]
    g = torch.Generator().manual_seed(c["mix"] + 1)
    return torch.randint(1, c["rmax"] + 1, (c["batch"],), generator=g).tolist()


def _gradient_inputs(c, seed):
    g = _gen(seed)
    n, b, r, dt = c["n"], c["batch"], c["nrhs"], DTYPES[c["dtype"]]
    A = _uniform(g, (b, n, n), dt) + torch.eye(n, dtype=dt, device="cuda") * max(4.0, 0.5 * math.sqrt(n))
    B = _uniform(g, (b, n, r), dt)
    G = torch.randn((b, n, r), dtype=dt, device="cuda", generator=g)
    return A, B, G


def _fixed_inputs(c, seed):
    """(A, B) in math orientation of the fixed-size families."""
    g = _gen(seed)
    n, b, r = c["n"], c["batch"], c["nrhs"]
    if c["kind"] == "refine":
        A = _svd_type(g, n, [(1e2, 1e4, 1e6)[k % 3] for k in range(b)])
    elif c["kind"] == "spd_refine":
        M = _uniform(g, (b, n, n))
        A = M @ M.transpose(1, 2) / n + 0.05 * torch.eye(n, dtype=torch.float64, device="cuda")
    else:
        A = _general(g, c)
    return A, _uniform(g, (b, n, r), A.dtype)


def _variable_inputs(c, seed):
    """VBatches (A, B, G); G only for the family with gradients."""
    g = _gen(seed)
    ns, rs = _sizes(c), _nrhs_of(c)
    dt = DTYPES[c.get("dtype", "f64")]
    dev = torch.device("cuda")
    A = mg.VBatch([(n, n) for n in ns], ns, dt, dev)
    B = mg.VBatch([(r, n) for n, r in zip(ns, rs)], ns, dt, dev)
    B.buf.uniform_(-1.0, 1.0, generator=g)
    if c["kind"] == "vbatched":
        A.buf.uniform_(-1.0, 1.0, generator=g)
        if dt == torch.float32:
            for k, n in enumerate(ns):
                A.view(k).diagonal().add_(2.0 * math.sqrt(n / 3.0))
        return A, B, None
    kg = torch.Generator().manual_seed(int(seed) + 1)
    lk = torch.rand((len(ns),), generator=kg).tolist()
    for k, n in enumerate(ns):
        A.view(k).copy_(_svd_type(g, n, [10.0 ** (4.0 * lk[k])])[0].T)
    B.buf.normal_(generator=g)
    G = mg.VBatch(B.shapes, ns, dt, dev)
    G.buf.normal_(generator=g)
    return A, B, G


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve_grad":
        A, B, G = _gradient_inputs(c, seed)
        return {"kind": kind, "A": A.requires_grad_(), "B": B.requires_grad_(), "G": G}
    if kind in ("vbatched", "refine_var_grad"):
        A, B, G = _variable_inputs(c, seed)
        s = {"kind": kind, "A": A, "B": B, "G": G, "A0": A.buf.clone(), "B0": B.buf.clone(), "work": None}
        if kind == "refine_var_grad":
            s["X"] = mg.VBatch(B.shapes, B.nrows, torch.float64, B.buf.device)
        return s
    A, B = _fixed_inputs(c, seed)
    S, Bs = _padded(A, c["pad"]), _padded(B, c["pad"])
    s = {"kind": kind, "S0": S, "B0": Bs}
    if kind == "gesv":
        s |= {"S": torch.empty_like(S), "X": torch.empty_like(Bs)}
    elif kind == "getrs":
        s["ipiv"], _ = mg.getrf_batched(S, m=c["n"])
        s |= {"X": torch.empty_like(Bs), "Y": torch.empty_like(Bs)}
    else:
        s["X"] = torch.zeros_like(Bs)
    if kind == "refine":
        s["work"] = torch.empty((mg.dsgesv_workspace_bytes(c["n"], c["nrhs"], c["batch"]),),
                                dtype=torch.uint8, device="cuda")
    return s


# ---------------------------------------------------------------------------
# one pass

def run(s):
    kind = s["kind"]
    if kind == "gesv":
        s["S"].copy_(s["S0"])
        s["X"].copy_(s["B0"])
        ipiv, info = mg.gesv_batched(s["S"], s["X"])
        return {"x": s["X"], "lu": s["S"], "ipiv": ipiv, "info": info}
    if kind == "getrs":
        s["X"].copy_(s["B0"])
        s["Y"].copy_(s["B0"])
        mg.getrs_batched(s["S0"], s["ipiv"], s["X"])
        mg.getrs_batched(s["S0"], s["ipiv"], s["Y"], trans=True)
        return {"x": s["X"], "y": s["Y"]}
    if kind == "vbatched":
        s["A"].buf.copy_(s["A0"])
        s["B"].buf.copy_(s["B0"])
        ipiv, _, info = mg.gesv_vbatched(s["A"], s["B"])
        return {"x": s["B"].buf, "lu": s["A"].buf, "ipiv": ipiv, "info": info}
    if kind == "refine":
        x, ipiv, info, iters = mg.dsgesv_batched(s["S0"], s["B0"], X=s["X"], work=s["work"])
        return {"x": x, "ipiv": ipiv, "info": info, "iters": iters}
    if kind == "solve_grad":
        x = mg_autograd.solve(s["A"], s["B"])
        ga, gb = torch.autograd.grad(x, (s["A"], s["B"]), s["G"])
        return {"x": x.detach(), "ga": ga, "gb": gb}
    if kind == "refine_var_grad":
        x, ipiv, offs, info, iters, s["work"] = mg.dxgesv_vbatched(s["A"], s["B"], X=s["X"], work=s["work"])
        gb, ga, back = mg.dxgesv_adjoint_vbatched(s["A"], ipiv, offs, x, s["G"], iters, info, s["work"])
        return {"x": x.buf, "gb": gb.buf, "ga": ga.buf, "ipiv": ipiv, "info": info, "iters": iters, "back": back}
    x, info, iters = mg.dsposv_batched(s["S0"], s["B0"], X=s["X"])
    return {"x": x, "info": info, "iters": iters}


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _lu_flops(n):
    return 2.0 * n ** 3 / 3.0


def work(case):
    c, kind = case, case["kind"]
    if kind in ("vbatched", "refine_var_grad"):
        # the expected sums over sizes uniform in [nmin, nmax]
        ns = range(c["nmin"], c["nmax"] + 1)
        m1, m2, m3 = (sum(n ** p for n in ns) / len(ns) * c["batch"] for p in (1, 2, 3))
        r = (1 + c["rmax"]) / 2 if "rmax" in c else c["nrhs"]
        if kind == "vbatched":
            el = 4 if c["dtype"] == "f32" else 8
            return {"bytes": el * (2 * m2 + 2 * r * m1) + 4 * m1, "flops": 2 / 3 * m3 + 2 * r * m2}
        # A read, gA written, b and the upstream gradient read, x and gb written; one
        # factorisation, and in each direction a solve, a correction and a residual
        return {"bytes": 8 * (2 * m2 + 4 * r * m1) + 4 * m1, "flops": 2 / 3 * m3 + 2 * r * m2 * (2 * 4 + 0.5)}
    n, b, r = c["n"], c["batch"], c["nrhs"]
    el = 4 if c.get("dtype") == "f32" else 8
    if kind == "gesv":
        return {"bytes": b * (el * (2 * n * n + 2 * n * r) + 4 * n), "flops": b * (_lu_flops(n) + 2.0 * n * n * r)}
    if kind == "getrs":
        return {"bytes": b * (el * (2 * n * n + 3 * n * r) + 4 * n), "flops": b * 4.0 * n * n * r}
    if kind == "solve_grad":
        return {"bytes": b * el * (2 * n * n + 5 * n * r), "flops": b * (_lu_flops(n) + 5.0 * n * n * r)}
    # refinement: one factorisation, two solves, two residuals
    half = 0.5 if kind == "spd_refine" else 1.0
    return {"bytes": b * 8 * (half * n * n + 2 * n * r), "flops": b * (half * _lu_flops(n) + 8.0 * n * n * r)}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch

def _solve(A, B):
    return torch.linalg.solve(A, B)


def _by_order(A, B, transposed=False):
    """Solutions of a variable-size batch as B's packed buffer, matrices of one order together."""
    out = B.buf.double()
    groups = {}
    for k, (n, _) in enumerate(A.shapes):
        groups.setdefault(n, []).append(k)
    for n, ks in groups.items():
        As = torch.stack([A.view(k) for k in ks]).double()
        r = max(B.shapes[k][0] for k in ks)
        Bs = torch.zeros((len(ks), n, r), dtype=torch.float64, device=out.device)
        for i, k in enumerate(ks):
            Bs[i, :, :B.shapes[k][0]] = B.view(k).T
        X = _solve(As if transposed else As.transpose(1, 2), Bs)
        for i, k in enumerate(ks):
            nc, ld = B.shapes[k]
            out[B.offsets[k]:B.offsets[k] + nc * ld].view(nc, ld).copy_(X[i, :, :nc].T)
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve_grad":
        A, B, G = (t.double() for t in _gradient_inputs(c, seed))
        x = _solve(A, B)
        gb = _solve(A.transpose(1, 2), G)
        return {"x": x, "ga": -gb @ x.transpose(1, 2), "gb": gb}
    if kind == "vbatched":
        A, B, _ = _variable_inputs(c, seed)
        return {"x": _by_order(A, B), "lu": None, "ipiv": None, "info": torch.zeros(c["batch"], dtype=torch.int32)}
    if kind == "refine_var_grad":
        A, B, G = _variable_inputs(c, seed)
        xs, gs = _by_order(A, B), _by_order(A, G, transposed=True)
        x, gb, ga = torch.zeros_like(xs), torch.zeros_like(gs), torch.zeros_like(A.buf)
        for (r, n), o, oa in zip(B.shapes, B.offsets, A.offsets):
            x[o:o + r * n], gb[o:o + r * n] = xs[o:o + r * n], gs[o:o + r * n]
            ga[oa:oa + n * n] = -(xs[o:o + r * n].view(r, n).T @ gs[o:o + r * n].view(r, n)).reshape(-1)
        return {"x": x, "gb": gb, "ga": ga, "ipiv": None, "info": None, "iters": None, "back": None}
    A, B = (t.double() for t in _fixed_inputs(c, seed))
    x = _padded(_solve(A, B), c["pad"])
    if kind == "getrs":
        return {"x": x, "y": _padded(_solve(A.transpose(1, 2), B), c["pad"])}
    if kind == "gesv":
        return {"x": x, "lu": None, "ipiv": None, "info": torch.zeros(c["batch"], dtype=torch.int32)}
    if kind == "refine":
        return {"x": x, "ipiv": None, "info": None, "iters": None}
    return {"x": x, "info": None, "iters": None}
