"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the Python mirror of the C ABI (first-project_b200/
cudecompose.py): device buffers in, device buffers out, column-major data in
flat tensors.  The tensors are sums of rank-1 terms with uniform [0, 1)
factors (or Tucker models with a decaying multilinear spectrum) plus 1e-3
relative Gaussian noise, like the benchmark's workloads, made with plain torch
from the seed alone.
"""
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "first-project_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cudecompose as cd  # noqa: E402

NOISE = 1e-3


def listed():
    return [
        # The MTTKRP of every mode, the step that CP programs spend their time
        # in.  The smallest: the sizes of the library's smoke test, where the
        # launches count.
        {"name": "mttkrp-small", "kind": "mttkrp", "dims": "48x40x36", "R": 8, "precision": "default"},
        # The headline: a 512 MiB tensor, rank 64, default (BF16x3) precision.
        {"name": "mttkrp-512-r64", "kind": "mttkrp", "dims": "512x512x512", "R": 64, "precision": "default"},
        # The benchmark's 4th-order tensor.
        {"name": "mttkrp-96p4-r32", "kind": "mttkrp", "dims": "96x96x96x96", "R": 32, "precision": "default"},
        # Measured data seldom has round extents: no extent is a multiple of 4.
        {"name": "mttkrp-odd", "kind": "mttkrp", "dims": "253x211x187", "R": 20, "precision": "default"},
        # Plain FP32, for a caller that wants no 16-bit operands.
        {"name": "mttkrp-fp32", "kind": "mttkrp", "dims": "256x256x256", "R": 32, "precision": "fp32"},
        # The double-precision programs.
        {"name": "mttkrp-f64", "kind": "mttkrp", "dims": "160x144x120", "R": 16, "precision": "f64"},
        # Whole call: ten CP-ALS sweeps of the benchmark's small configuration
        # through a plan that the program keeps, and the fit.
        {"name": "cp-sweeps-128", "kind": "sweeps", "dims": "128x128x128", "R": 16, "precision": "default", "sweeps": 10},
        # The exact reconstruction error of a CP model, which every checked
        # CP-ALS run computes.
        {"name": "residual-384-r64", "kind": "residual", "dims": "384x384x384", "R": 64},
        # Many small tensors of uneven shape and rank at once, as in the
        # benchmark (dims 16 to 96, ranks 4 to 16).
        {"name": "batched-256", "kind": "batched", "tensors": 256, "sweeps": 3},
        # Whole call: HOSVD in the entry point's default precision (FP32) ...
        {"name": "hosvd-fp32", "kind": "tucker", "dims": "96x80x72", "r": 12, "precision": "fp32", "sweeps": -1},
        # ... and on the tensor cores.
        {"name": "hosvd-256-r16", "kind": "tucker", "dims": "256x256x256", "r": 16, "precision": "bf16x3", "sweeps": -1},
        # Tensor times matrix in every mode: a projection onto factors.
        {"name": "ttm-fp32", "kind": "ttm", "dims": "256x240x224", "J": 32},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, most, order=None, steps=(32, 8, 1)):
    """Extents uniform in their logarithm, each a multiple of 32 or 8 or any."""
    order = order or rng.choice((3, 3, 4))
    while True:
        dims = []
        for _ in range(order):
            m = rng.choice(steps)
            dims.append(max(m, _log_uniform(rng, lo, hi) // m * m))
        if lo ** 3 <= math.prod(dims) <= most:
            return "x".join(map(str, dims))


def draw(rng):
    kind = rng.choice(("mttkrp", "mttkrp", "mttkrp", "mttkrp", "sweeps", "residual", "batched", "tucker", "ttm"))
    if kind == "mttkrp":
        precision = rng.choice(("default", "default", "default", "fp32", "bf16", "fp16", "f64"))
        return {"kind": kind, "dims": _shape(rng, 24, 512, 1 << 23 if precision == "f64" else 1 << 25),
                "R": _log_uniform(rng, 4, 64), "precision": precision}
    if kind == "sweeps":
        return {"kind": kind, "dims": _shape(rng, 64, 256, 1 << 23, 3), "R": rng.randint(4, 16),
                "precision": rng.choice(("default", "fp32")), "sweeps": rng.choice((5, 10))}
    if kind == "residual":
        return {"kind": kind, "dims": _shape(rng, 48, 512, 1 << 25), "R": rng.randint(8, 64)}
    if kind == "batched":
        return {"kind": kind, "tensors": _log_uniform(rng, 32, 256), "sweeps": rng.choice((2, 3))}
    if kind == "tucker":
        # HOSVD (-1) or a HOOI sweep; the tensor cores take extents that are
        # multiples of 8
        sweeps = rng.choice((-1, 1))
        if rng.random() < 0.5:
            return {"kind": kind, "dims": _shape(rng, 40, 96 if sweeps < 0 else 64, 1 << 20, 3), "r": rng.randint(6, 16),
                    "precision": "fp32", "sweeps": sweeps}
        return {"kind": kind, "dims": _shape(rng, 40, 256, 1 << 23, 3, (32, 8)), "r": rng.randint(6, 16),
                "precision": "bf16x3", "sweeps": sweeps}
    return {"kind": kind, "dims": _shape(rng, 24, 512, 1 << 24), "J": rng.randint(8, 64)}


def _dims(case):
    return [int(x) for x in case["dims"].split("x")]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape, dtype=torch.float32):
    return torch.rand(*shape, generator=g, device="cuda", dtype=dtype)


def _noisy(X, g):
    E = torch.randn(X.numel(), generator=g, device="cuda", dtype=X.dtype)
    return X.add_(E, alpha=float(NOISE * torch.linalg.norm(X) / math.sqrt(X.numel())))


def _khatri_rao(factors):
    """Rows of the Khatri-Rao product of (R x d) factors, the first fastest."""
    kr = factors[0].t()
    for f in factors[1:]:
        kr = (f.t()[:, None, :] * kr[None, :, :]).reshape(-1, kr.shape[1])
    return kr


def _cp_tensor(dims, factors, g):
    """The flat column-major tensor of the (R x d) factors, and noise."""
    return _noisy((_khatri_rao(factors[1:]) @ factors[0]).reshape(-1), g)


def _cp_data(dims, R, seed, dtype=torch.float32):
    """X, its generating factors and a random start, all (R x d) factors."""
    g = _generator(seed)
    true = [_rand(g, R, d, dtype=dtype) for d in dims]
    X = _cp_tensor(dims, true, g)
    return X, true, [_rand(g, R, d, dtype=dtype) for d in dims]


def _tucker_data(dims, r, seed):
    """X = core x_1 Q_1 x_2 Q_2 ...: the rows of a Gaussian core decay from 1
    to 0.4 in every mode, the Q_n have orthonormal columns."""
    g = _generator(seed)
    X = torch.randn([r] * len(dims), generator=g, device="cuda", dtype=torch.float64)
    w = torch.linspace(1.0, 0.4, r, device="cuda", dtype=torch.float64)
    for m, d in enumerate(reversed(dims)):  # X's axes run slowest mode first
        Q = torch.linalg.qr(torch.randn(d, r, generator=g, device="cuda", dtype=torch.float64))[0]
        X = torch.movedim(torch.tensordot(Q * w, X, dims=([1], [m])), 0, m)
    return _noisy(X.float().contiguous().reshape(-1), g)


def _batch_data(case, seed):
    """A packed batch: tensors of uneven shape and rank, and their starts."""
    n = case["tensors"]
    pick = torch.Generator().manual_seed(7)  # the shapes are the case's, the values the seed's
    dims = torch.randint(16, 97, (n, 3), generator=pick).tolist()
    ranks = torch.randint(4, 17, (n,), generator=pick).tolist()
    g = _generator(seed)
    b = cd.Batch(dims, ranks)
    for t, (d, r) in enumerate(zip(dims, ranks)):
        true = [_rand(g, r, x) for x in d]
        b.x_view(t).copy_(_cp_tensor(d, true, g))
        for m in range(3):
            b.u_view(t, m).copy_(_rand(g, r, d[m]).reshape(-1))
    return b


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batched":
        b = _batch_data(case, seed)
        return {"case": case, "batch": b, "start": b.U.clone()}
    dims = _dims(case)
    if kind == "mttkrp":
        dtype = torch.float64 if case["precision"] == "f64" else torch.float32
        X, _, U = _cp_data(dims, case["R"], seed, dtype)
        return {"case": case, "dims": dims, "X": X, "U": [u.reshape(-1) for u in U],
                "out": [torch.empty(d * case["R"], device="cuda", dtype=dtype) for d in dims]}
    if kind == "sweeps":
        X, _, U = _cp_data(dims, case["R"], seed)
        start = [u.reshape(-1) for u in U]
        U = [u.clone() for u in start]
        plan = cd.CpPlan(X, dims, case["R"], U, precision=cd.PRECISIONS[case["precision"]])
        return {"case": case, "X": X, "U": U, "start": start, "plan": plan}
    if kind == "residual":
        X, true, _ = _cp_data(dims, case["R"], seed)
        g = _generator(seed + 1000003)  # a model on its way to the solution
        U = [(u * (1 + 0.02 * torch.randn(u.shape, generator=g, device="cuda"))).reshape(-1) for u in true]
        return {"case": case, "dims": dims, "X": X, "U": U}
    if kind == "tucker":
        r = case["r"]
        return {"case": case, "dims": dims, "X": _tucker_data(dims, r, seed),
                "core": torch.empty(r ** len(dims), device="cuda"),
                "U": [torch.empty(d * r, device="cuda") for d in dims]}
    g = _generator(seed)
    J = case["J"]
    W = [torch.randn(J * d, generator=g, device="cuda") / math.sqrt(d) for d in dims]
    X = _rand(g, math.prod(dims))
    return {"case": case, "dims": dims, "X": X, "W": W,
            "out": [torch.empty(X.numel() // d * J, device="cuda") for d in dims]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mttkrp":
        for mode, out in enumerate(state["out"]):
            if case["precision"] == "f64":
                cd.mttkrp_f64(state["X"], state["dims"], state["U"], mode, case["R"], out)
            else:
                cd.mttkrp(state["X"], state["dims"], state["U"], mode, case["R"], out, cd.PRECISIONS[case["precision"]])
        return state["out"]
    if kind == "sweeps":
        for u, s in zip(state["U"], state["start"]):
            u.copy_(s)
        state["plan"].run(case["sweeps"])
        fit, _ = state["plan"].fit()
        return [state["U"], fit]
    if kind == "residual":
        return list(cd.cp_residual(state["X"], state["dims"], state["U"], case["R"]))
    if kind == "batched":
        b = state["batch"]
        b.U.copy_(state["start"])
        fits, _, _ = cd.cp_als_batched(b, max_sweeps=case["sweeps"], tol=0.0)
        return [b.U, torch.tensor(fits)]
    if kind == "tucker":
        ranks = [case["r"]] * len(state["dims"])
        precision = cd.PRECISIONS[case["precision"]]
        if case["sweeps"] < 0:
            cd.tucker_hosvd(state["X"], state["dims"], ranks, state["core"], state["U"], precision)
        else:
            cd.tucker_hooi(state["X"], state["dims"], ranks, state["core"], state["U"], case["sweeps"], precision)
        return [state["core"], state["U"]]
    for mode, (W, out) in enumerate(zip(state["W"], state["out"])):
        cd.mode_product(state["X"], state["dims"], mode, W, case["J"], out)
    return state["out"]


def work(case):
    """Bytes: the tensor once per MTTKRP / product / sweep mode, the factors
    once, the outputs once.  Flops: the contraction's multiply-adds."""
    kind = case["kind"]
    if kind == "batched":
        pick = torch.Generator().manual_seed(7)
        n = case["tensors"]
        dims = torch.randint(16, 97, (n, 3), generator=pick).tolist()
        ranks = torch.randint(4, 17, (n,), generator=pick).tolist()
        byts = sum(4 * (3 * math.prod(d) + 2 * r * sum(d)) for d, r in zip(dims, ranks)) * case["sweeps"]
        return {"bytes": byts, "flops": sum(6 * math.prod(d) * r for d, r in zip(dims, ranks)) * case["sweeps"]}
    dims = _dims(case)
    N, n = len(dims), math.prod(dims)
    if kind in ("mttkrp", "sweeps"):
        R, times = case["R"], case.get("sweeps", 1)
        size = 8 if case["precision"] == "f64" else 4
        return {"bytes": N * size * (n + R * sum(dims)) * times, "flops": N * 2 * n * R * times}
    if kind == "residual":
        return {"bytes": 4 * (n + case["R"] * sum(dims)), "flops": 2 * n * case["R"]}
    if kind == "tucker":
        # a Gram per mode and the projection; HOOI: a projection and the Gram
        # of what it leaves per mode and sweep
        r, s = case["r"], max(0, case["sweeps"])
        grams = (N - 1 if s else N)
        flops = grams * n * sum(dims) / N + 2 * n * r + s * N * 2 * n * r
        return {"bytes": 4 * n * (grams + 1 + s * N) + 4 * r * sum(dims) + 4 * r ** N, "flops": flops}
    J = case["J"]
    return {"bytes": 4 * sum(n + J * d + n // d * J for d in dims), "flops": N * 2 * n * J}


def _mttkrp64(X, dims, U, mode):
    """(d_mode x R) in 64 bits; U: (R x d) float64 factors."""
    P, Q, S = math.prod(dims[:mode]), dims[mode], math.prod(dims[mode + 1:])
    after = _khatri_rao(U[mode + 1:]) if mode + 1 < len(dims) else None
    if mode == 0:
        return X.reshape(S, Q).t() @ after
    Y = (X.reshape(S * Q, P) @ _khatri_rao(U[:mode])).reshape(S, Q, -1)
    return (Y * after[:, None, :]).sum(0) if after is not None else Y[0]


def _als64(X, dims, U, sweeps):
    """`sweeps` ALS sweeps from U (R x d, float64): the factors and the fit."""
    U = list(U)
    for _ in range(sweeps):
        for mode in range(len(dims)):
            V = torch.ones_like(U[0] @ U[0].t())
            for m, u in enumerate(U):
                if m != mode:
                    V = V * (u @ u.t())
            M = _mttkrp64(X, dims, U, mode)
            U[mode] = torch.linalg.solve(V, M.t()).contiguous()
    norm = torch.linalg.norm(X)
    full = V * (U[-1] @ U[-1].t())
    res2 = norm * norm - 2 * (M.t() * U[-1]).sum() + full.sum()
    return U, 1 - torch.sqrt(res2.clamp_min(0)) / norm


def exact(case, seed):
    kind = case["kind"]
    if kind == "batched":
        b = _batch_data(case, seed)
        U, fits = b.U.double(), []
        for t, (d, r) in enumerate(zip(b.dims, b.ranks)):
            got, fit = _als64(b.x_view(t).double(), d, [b.u_view(t, m).double().reshape(r, -1) for m in range(3)], case["sweeps"])
            for m in range(3):
                o = b.u_offsets[3 * t + m]
                U[o: o + d[m] * r] = got[m].reshape(-1)
            fits.append(fit)
        return [U, torch.stack(fits)]
    dims = _dims(case)
    if kind == "mttkrp":
        X, _, U = _cp_data(dims, case["R"], seed, torch.float64 if case["precision"] == "f64" else torch.float32)
        X, U = X.double(), [u.double() for u in U]
        return [_mttkrp64(X, dims, U, m).t().contiguous().reshape(-1) for m in range(len(dims))]
    if kind == "sweeps":
        X, _, U = _cp_data(dims, case["R"], seed)
        U, fit = _als64(X.double(), dims, [u.double() for u in U], case["sweeps"])
        return [[u.reshape(-1) for u in U], fit]
    s = prepare(case, seed)
    X = s["X"].double()
    if kind == "residual":
        U = [u.double().reshape(case["R"], -1) for u in s["U"]]
        rec = (_khatri_rao(U[1:]) @ U[0]).reshape(-1)
        return [(X - rec).square().sum(), X.square().sum()]
    if kind == "tucker":
        return None  # eigenvectors up to their signs: held to the start's outputs alone
    out = []
    for mode, (d, W) in enumerate(zip(dims, s["W"])):
        P, S = math.prod(dims[:mode]), math.prod(dims[mode + 1:])
        Wm = W.double().reshape(d, case["J"])  # J x d, column-major
        out.append(torch.einsum("sqp,qj->sjp", X.reshape(S, d, P), Wm).reshape(-1))
    return out
