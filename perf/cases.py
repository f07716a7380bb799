"""Measured workloads of the library: the calls that its users make, over the sizes that they make them at.

Every case is a dict of plain values whose ``kind`` names one use:

* ``chain``:   n <= 32, many matrices: getrf, getrs and (``inverse``) getri on the same factors;
* ``solve``:   32 < n <= 512: getrf and getrs, trans N or T;
* ``inverse``: 32 < n <= 256: getrf and getri;
* ``grouped``: a plan over instances of mixed order, factored and solved in one call;
* ``refine``:  mixed-precision factor, solve and FP64-residual refinement;
* ``grad``:    the differentiable solve, forward and backward;
* ``geqrf`` / ``gels``: Householder QR, least squares;
* ``gemm``:    GemmBatchedEx (BF16, FP16, FP32 in TF32);
* ``cgemm``:   complex GEMM with complex alpha and beta.

The LU calls work in place, so a program that keeps its matrices copies them first; that copy is part
of the pass. Pointer arrays, pivot and info buffers, plans and handles are made once.

LU inputs are G + 2 sqrt(n) I with G ~ N(0, 1) and the rows of every matrix shuffled: well conditioned
(so that the results can be compared), every column pivots to another row, and no pivot is a near tie.
"""
import importlib.util
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_DEV = "cuda:0"


def _package():
    name = "ops_blas_b200"
    if name not in sys.modules:
        path = os.path.join(_ROOT, "ops-blas_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path, submodule_search_locations=[os.path.dirname(path)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


ob = _package()
_handles = {}


def _handle():
    """One handle on the current stream, kept as a program keeps it."""
    if "h" not in _handles:
        _handles["h"] = ob.Handle()
    return _handles["h"]


def listed():
    return [
        # the parity workload of the benchmark: one small batch, where launches and latency count
        {"name": "chain_n16_b1024", "kind": "chain", "n": 16, "pad": 0, "batch": 1024, "nrhs": 1, "inverse": False},
        # the benchmark's headline: a large batch of small systems, solved and inverted
        {"name": "chain_n32_b131072", "kind": "chain", "n": 32, "pad": 0, "batch": 131072, "nrhs": 4, "inverse": True},
        # instances of mixed order in one launch, as a batched solver of irregular blocks meets them
        {"name": "grouped_50000_n4_128", "kind": "grouped", "lo": 4, "hi": 128, "count": 50000, "nrhs": 1},
        # an ordinary mid-size batch with an odd leading dimension
        {"name": "solve_n100_b4096", "kind": "solve", "n": 100, "pad": 1, "batch": 4096, "nrhs": 1, "trans": "N"},
        # the largest plain factorisation of the benchmark
        {"name": "solve_n512_b256", "kind": "solve", "n": 512, "pad": 0, "batch": 256, "nrhs": 16, "trans": "N"},
        # mixed precision with refinement, condition 1e4, as the benchmark runs it
        {"name": "refine_tf32_n256_b2048", "kind": "refine", "n": 256, "batch": 2048, "nrhs": 16, "compute": "tf32"},
        # the differentiable solve of the benchmark, forward and backward
        {"name": "grad_n64_b65536", "kind": "grad", "n": 64, "batch": 65536, "nrhs": 8},
        # explicit inverses of a mid-size batch (covariances, preconditioner blocks)
        {"name": "inverse_n128_b2048", "kind": "inverse", "n": 128, "pad": 0, "batch": 2048},
        # QR above the warp-sized blocks
        {"name": "geqrf_64x48_b4096", "kind": "geqrf", "m": 64, "n": 48, "batch": 4096},
        # many small least-squares fits, as the benchmark runs them
        {"name": "gels_32x16_b65536", "kind": "gels", "m": 32, "n": 16, "batch": 65536, "nrhs": 2},
        # the benchmark's tensor-core GEMM
        {"name": "gemm_bf16_256_b2048", "kind": "gemm", "dtype": "bf16", "ta": "N", "tb": "N", "m": 256, "n": 256, "k": 256, "batch": 2048},
        # the benchmark's complex GEMM
        {"name": "cgemm_64_b16384", "kind": "cgemm", "ta": "N", "tb": "N", "m": 64, "n": 64, "k": 64, "batch": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "solve", "inverse", "grouped", "refine", "grad", "geqrf", "gels", "gemm", "cgemm"])
    if kind == "chain":
        return {"kind": kind, "n": rng.randint(4, 32), "pad": rng.choice([0, 0, 0, 1, 4]), "batch": _log(rng, 1024, 131072),
                "nrhs": rng.choice([1, 1, 2, 4, 8]), "inverse": rng.random() < 0.5}
    if kind == "solve":
        n = _log(rng, 33, 512)
        return {"kind": kind, "n": n, "pad": rng.choice([0, 0, 0, 1, 4]), "batch": _log(rng, 64, max(128, min(16384, (1 << 26) // (n * n)))),
                "nrhs": rng.choice([1, 2, 4, 8, 16]), "trans": rng.choice(["N", "N", "T"])}
    if kind == "inverse":
        n = _log(rng, 33, 256)
        return {"kind": kind, "n": n, "pad": rng.choice([0, 0, 0, 1, 4]), "batch": _log(rng, 64, min(8192, (1 << 25) // (n * n)))}
    if kind == "grouped":
        return {"kind": kind, "lo": rng.choice([4, 8, 16, 33]), "hi": rng.randint(40, 128), "count": _log(rng, 1000, 50000), "nrhs": rng.choice([1, 1, 2])}
    if kind == "refine":
        n = _log(rng, 64, 512)
        return {"kind": kind, "n": n, "batch": _log(rng, 64, min(4096, (1 << 26) // (n * n))), "nrhs": rng.choice([1, 4, 16]),
                "compute": rng.choice(["tf32", "tf32", "f32"])}
    if kind == "grad":
        n = _log(rng, 8, 96)
        return {"kind": kind, "n": n, "batch": _log(rng, 1024, min(65536, (1 << 27) // (n * n))), "nrhs": rng.choice([1, 2, 4, 8])}
    if kind == "geqrf":
        m = rng.randint(12, 64)
        return {"kind": kind, "m": m, "n": rng.randint(max(4, m // 2), m), "batch": _log(rng, 512, (1 << 24) // (m * m))}
    if kind == "gels":
        m = rng.randint(12, 48)
        return {"kind": kind, "m": m, "n": rng.randint(4, 3 * m // 4), "batch": _log(rng, 512, (1 << 24) // (m * m)), "nrhs": rng.choice([1, 2, 4])}
    if kind == "gemm":
        m, n, k = _log(rng, 48, 512), _log(rng, 48, 512), _log(rng, 48, 512)
        if rng.random() < 0.6:  # rows that tensor maps take; the rest stay ragged
            m, n, k = (-(-v // 8) * 8 for v in (m, n, k))
        return {"kind": kind, "dtype": rng.choice(["bf16", "f16", "tf32"]), "ta": rng.choice(["N", "T"]), "tb": rng.choice(["N", "N", "T"]),
                "m": m, "n": n, "k": k, "batch": _log(rng, 64, max(128, min(4096, (1 << 26) // max(m * n, m * k, n * k))))}
    m, n, k = rng.randint(16, 128), rng.randint(16, 128), rng.randint(16, 128)
    return {"kind": kind, "ta": rng.choice(["N", "T", "C"]), "tb": rng.choice(["N", "T", "C"]), "m": m, "n": n, "k": k,
            "batch": _log(rng, 128, (1 << 25) // max(m * n, m * k, n * k))}


# ------------------------------------------------------------------------------------- inputs --


def _generator(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, device=_DEV, generator=g, dtype=dtype)


def _matrices(g, batch, n, ld=None):
    """(batch, n, ld) column-major matrices: rows of G + 2 sqrt(n) I in a random order."""
    A = _randn(g, batch, n, ld or n)
    perm = torch.rand(batch, n, device=_DEV, generator=g).argsort(1)  # column j's large entry sits in row perm[j]
    A.scatter_add_(2, perm.unsqueeze(2), torch.full((batch, n, 1), 2.0 * math.sqrt(n), device=_DEV))
    return A


def _conditioned(g, batch, n):
    """(batch, n, n) matrices Q1 diag(s) Q2^T, s log-spaced from 1 to 1e4 in another order for every matrix."""
    q1 = torch.linalg.qr(_randn(g, n, n, dtype=torch.float64))[0].float()
    q2 = torch.linalg.qr(_randn(g, n, n, dtype=torch.float64))[0].float()
    s = torch.logspace(0, 4, n, device=_DEV)[torch.rand(batch, n, device=_DEV, generator=g).argsort(1)]
    return torch.matmul(q1.unsqueeze(0) * s.unsqueeze(1), q2.t())


def _orders(case):
    """The orders of a grouped batch: the structure of the problem, the same for all its values."""
    g = torch.Generator().manual_seed(case["count"])
    n = torch.randint(case["lo"], case["hi"] + 1, (case["count"],), generator=g).tolist()
    orders = sorted(set(n), reverse=True)
    counts = {}
    for v in n:
        counts[v] = counts.get(v, 0) + 1
    return orders, [counts[v] for v in orders]


_GEMM = {"bf16": (torch.bfloat16, ob.ACL_BF16, ob.COMPUTE_32F), "f16": (torch.float16, ob.ACL_FLOAT16, ob.COMPUTE_32F),
         "tf32": (torch.float32, ob.ACL_FLOAT, ob.COMPUTE_32F_FAST_TF32)}
_ALPHA, _BETA = 1.5 + 0.3j, 0.3 - 0.1j


def _int(*shape):
    return torch.empty(shape, dtype=torch.int32, device=_DEV)


def _inputs(case, seed):
    """The numbers a case starts from; the same for prepare() and exact()."""
    g, kind = _generator(seed), case["kind"]
    if kind in ("chain", "solve", "inverse"):
        n = case["n"]
        d = {"A": _matrices(g, case["batch"], n, n + case["pad"])}
        if kind != "inverse":
            d["B"] = torch.rand(case["batch"], case["nrhs"], n, device=_DEV, generator=g) * 2 - 1
    elif kind == "grouped":
        orders, counts = _orders(case)
        d = {"orders": orders, "counts": counts, "A": [_matrices(g, c, n) for n, c in zip(orders, counts)],
             "B": [_randn(g, c, case["nrhs"], n) for n, c in zip(orders, counts)]}
    elif kind == "refine":
        d = {"A": _conditioned(g, case["batch"], case["n"]), "B": _randn(g, case["batch"], case["nrhs"], case["n"])}
    elif kind == "grad":
        n = case["n"]
        d = {"A": _matrices(g, case["batch"], n), "B": _randn(g, case["batch"], case["nrhs"], n), "dX": _randn(g, case["batch"], case["nrhs"], n)}
    elif kind == "geqrf":
        d = {"A": _randn(g, case["batch"], case["n"], case["m"])}
    elif kind == "gels":
        d = {"A": _randn(g, case["batch"], case["n"], case["m"]), "C": _randn(g, case["batch"], case["nrhs"], case["m"])}
    else:
        dt = torch.complex64 if kind == "cgemm" else _GEMM[case["dtype"]][0]
        m, n, k = case["m"], case["n"], case["k"]
        base = dt if kind == "cgemm" else torch.float32
        a = (case["batch"], k, m) if case["ta"] == "N" else (case["batch"], m, k)
        b = (case["batch"], n, k) if case["tb"] == "N" else (case["batch"], k, n)
        d = {"A": _randn(g, *a, dtype=base).to(dt), "B": _randn(g, *b, dtype=base).to(dt)}
        if kind == "cgemm":
            d["C"] = _randn(g, case["batch"], n, m, dtype=dt)
    return d


def prepare(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    s["case"], s["h"] = case, _handle()
    if kind in ("chain", "solve", "inverse"):
        b, n = case["batch"], case["n"]
        s["LU"], s["piv"], s["info"] = torch.empty_like(s["A"]), _int(b, n), _int(b)
        s["pa"] = ob.ptr_array(s["LU"])
        if "B" in s:
            s["X"] = torch.empty_like(s["B"])
            s["px"] = ob.ptr_array(s["X"])
        if kind == "inverse" or case.get("inverse"):
            s["C"], s["cinfo"] = torch.empty(b, n, n, device=_DEV), _int(b)
            s["pc"] = ob.ptr_array(s["C"])
    elif kind == "grouped":
        orders, counts, r = s["orders"], s["counts"], case["nrhs"]
        a_off, a_len = ob.grouped_offsets(orders, orders, orders, counts)
        b_off, b_len = ob.grouped_offsets(orders, [r] * len(orders), orders, counts)
        s["A0"], s["B0"] = torch.zeros(a_len, device=_DEV), torch.zeros(b_len, device=_DEV)
        at = 0
        for n, c, A, B in zip(orders, counts, s.pop("A"), s.pop("B")):
            for dst, off, src in ((s["A0"], a_off, A), (s["B0"], b_off, B)):
                step = off[at + 1] - off[at] if c > 1 else src[0].numel()
                dst.as_strided((c, src[0].numel()), (step, 1), off[at]).copy_(src.reshape(c, -1))
            at += c
        s["A"], s["B"] = torch.empty_like(s["A0"]), torch.empty_like(s["B0"])
        s["pa"], s["pb"] = ob.slab_ptrs(s["A"], a_off), ob.slab_ptrs(s["B"], b_off)
        s["piv"], s["info"] = _int(sum(n * c for n, c in zip(orders, counts))), _int(sum(counts))
        s["plan"] = ob.GroupedPlan(s["h"], orders, [r] * len(orders), counts)
    elif kind == "grad":
        s["A"].requires_grad_(True)
        s["B"].requires_grad_(True)
    elif kind == "geqrf":
        s["Q"], s["tau"] = torch.empty_like(s["A"]), torch.empty(case["batch"], case["n"], device=_DEV)
        s["pa"], s["pt"] = ob.ptr_array(s["Q"]), ob.ptr_array(s["tau"])
    elif kind == "gels":
        s["Q"], s["X"], s["info"] = torch.empty_like(s["A"]), torch.empty_like(s["C"]), _int(case["batch"])
        s["pa"], s["pc"] = ob.ptr_array(s["Q"]), ob.ptr_array(s["X"])
    elif kind == "gemm":
        s["C"] = torch.empty(case["batch"], case["n"], case["m"], device=_DEV, dtype=s["A"].dtype)
        s["pa"], s["pb"], s["pc"] = (ob.ptr_array(s[k]) for k in "ABC")
    elif kind == "cgemm":
        s["R"] = torch.empty_like(s["C"])
        s["pa"], s["pb"], s["pc"] = ob.ptr_array(s["A"]), ob.ptr_array(s["B"]), ob.ptr_array(s["R"])
    return s


def run(s):
    case, h = s["case"], s["h"]
    kind = case["kind"]
    if kind in ("chain", "solve", "inverse"):
        n, ld = case["n"], case["n"] + case["pad"]
        LU = s["LU"]
        LU.copy_(s["A"])
        h.getrf(LU, n, ld, piv=s["piv"], info=s["info"], aptr=s["pa"])
        out = [LU, s["piv"], s["info"]]
        if "X" in s:
            s["X"].copy_(s["B"])
            h.getrs(case.get("trans", "N"), LU, n, ld, s["piv"], s["X"], case["nrhs"], n, aptr=s["pa"], bptr=s["px"])
            out.append(s["X"])
        if "C" in s:
            h.getri(LU, n, ld, s["piv"], s["C"], n, info=s["cinfo"], aptr=s["pa"], cptr=s["pc"])
            out += [s["C"], s["cinfo"]]
        return out
    if kind == "grouped":
        s["A"].copy_(s["A0"])
        s["B"].copy_(s["B0"])
        s["plan"].run(h, s["pa"], s["piv"], s["info"], s["pb"])
        return [s["A"], s["piv"], s["info"], s["B"]]
    if kind == "refine":
        # the solution; the factors are its by-product, and a pivot among near equals is the rounding's choice
        X, _, _, info, _, iters = h.refine(s["A"], s["B"], case["n"], case["nrhs"], tol=1e-6,
                                           compute=ob.COMPUTE_32F_FAST_TF32 if case["compute"] == "tf32" else ob.COMPUTE_32F)
        return [X, info, iters]
    if kind == "grad":
        X = ob.batched_solve(s["A"], s["B"])
        dA, dB = torch.autograd.grad(X, (s["A"], s["B"]), s["dX"])
        return [X, dA, dB]
    if kind == "geqrf":
        s["Q"].copy_(s["A"])
        h.geqrf(s["Q"], case["m"], case["n"], case["m"], tau=s["tau"], aptr=s["pa"], tptr=s["pt"])
        return [s["Q"], s["tau"]]
    if kind == "gels":
        s["Q"].copy_(s["A"])
        s["X"].copy_(s["C"])
        h.gels("N", s["Q"], case["m"], case["n"], case["nrhs"], case["m"], s["X"], case["m"], info=s["info"], aptr=s["pa"], cptr=s["pc"])
        return [s["Q"], s["X"], s["info"]]
    m, n, k = case["m"], case["n"], case["k"]
    lda, ldb = (m if case["ta"] == "N" else k), (k if case["tb"] == "N" else n)
    if kind == "gemm":
        t, compute = _GEMM[case["dtype"]][1:]
        h.gemm_batched_ex(case["ta"], case["tb"], m, n, k, 1.0, s["A"], t, lda, s["B"], t, ldb, 0.0, s["C"], t, m, compute=compute,
                          aptr=s["pa"], bptr=s["pb"], cptr=s["pc"])
        return s["C"]
    s["R"].copy_(s["C"])
    h.cgemm(case["ta"], case["tb"], m, n, k, _ALPHA, s["A"], lda, s["B"], ldb, _BETA, s["R"], m, aptr=s["pa"], bptr=s["pb"], cptr=s["pc"])
    return s["R"]


# ------------------------------------------------------------------------------ cost and errors --


def work(case):
    """Each input read once, each output written once; the operations of the textbook algorithm."""
    kind, b = case["kind"], case.get("batch", 0)
    if kind in ("chain", "solve", "inverse"):
        n, r = case["n"], case.get("nrhs", 0)
        inv = kind == "inverse" or case.get("inverse", False)
        return {"bytes": b * (8 * n * n + 8 * n * r + 4 * n + 4 + (4 * n * n + 4 if inv else 0)),
                "flops": b * (2 * n ** 3 / 3 + 2 * n * n * r + (4 * n ** 3 / 3 if inv else 0))}
    if kind == "grouped":
        r, groups = case["nrhs"], list(zip(*_orders(case)))
        return {"bytes": sum(c * (8 * n * n + 8 * n * r + 4 * n + 4) for n, c in groups), "flops": sum(c * (2 * n ** 3 / 3 + 2 * n * n * r) for n, c in groups)}
    if kind == "refine":  # factor and solve, and the residual of one check in FP64
        n, r = case["n"], case["nrhs"]
        return {"bytes": b * (8 * n * n + 8 * n * r + 4 * n + 16), "flops": b * (2 * n ** 3 / 3 + 4 * n * n * r)}
    if kind == "grad":  # A, B and dX in; X, dA and dB out
        n, r = case["n"], case["nrhs"]
        return {"bytes": b * (8 * n * n + 16 * n * r), "flops": b * (2 * n ** 3 / 3 + 6 * n * n * r)}
    if kind == "geqrf":
        m, n = case["m"], case["n"]
        return {"bytes": b * (8 * m * n + 4 * n), "flops": b * (2 * m * n * n - 2 * n ** 3 / 3)}
    if kind == "gels":
        m, n, r = case["m"], case["n"], case["nrhs"]
        return {"bytes": b * (8 * m * n + 8 * m * r + 4), "flops": b * (2 * m * n * n - 2 * n ** 3 / 3 + (4 * m * n - n * n) * r)}
    m, n, k = case["m"], case["n"], case["k"]
    if kind == "gemm":
        es = 4 if case["dtype"] == "tf32" else 2
        return {"bytes": b * es * (m * k + k * n + m * n), "flops": b * 2 * m * n * k}
    return {"bytes": b * 8 * (m * k + k * n + 2 * m * n), "flops": b * 8 * m * n * k}


def tolerance(case):
    """About four times the error that the calls show against exact()."""
    kind = case["kind"]
    if kind == "gemm":  # one rounding of the result (BF16, FP16) or of the operands (TF32)
        return {"bf16": {"rel": 7e-3, "max": 4e-2}, "f16": {"rel": 1e-3, "max": 5e-3}, "tf32": {"rel": 1e-3, "max": 8e-3}}[case["dtype"]]
    if kind == "cgemm":  # 1.6e-7 measured
        return {"rel": 1e-6}
    if kind == "refine":  # condition 1e4: 1.5e-4 measured; a step more or less of refinement for a few
        return {"rel": 1e-3, "differ": 1e-2}
    if kind in ("geqrf", "gels"):  # 3e-7 measured
        return {"rel": 2e-6}
    return {"rel": 4e-6}  # 8e-7 measured at n = 512


def _lu64(A):
    """LU, 1-based pivots of column-major batches in 64 bits, laid out as getrf leaves them."""
    lu, piv = torch.linalg.lu_factor(A.double().transpose(1, 2))
    return lu.transpose(1, 2).contiguous(), piv.int()


def _solve64(A, B, trans="N"):
    M = A.double().transpose(1, 2)
    return torch.linalg.solve(M.transpose(1, 2) if trans != "N" else M, B.double().transpose(1, 2)).transpose(1, 2).contiguous()


def _householder64(A, n, keep_positive):
    """Householder QR of the first n rows of A (batch, columns, m): every row is a column of a matrix. With
    keep_positive a column that is zero below a diagonal >= 0 is left alone (else: zero below any diagonal)."""
    A = A.double().clone()
    tau = torch.zeros(A.shape[0], n, device=A.device, dtype=torch.float64)
    for i in range(n):
        x1, tail = A[:, i, i].clone(), A[:, i, i + 1:]
        sigma = tail.square().sum(1)
        skip = (sigma == 0) & (x1 >= 0) if keep_positive else sigma == 0
        norm = (sigma + x1 * x1).sqrt()
        alpha = torch.where(x1 >= 0, -norm, norm)
        t = torch.where(skip, torch.zeros_like(x1), (alpha - x1) / alpha)
        v = torch.where(skip.unsqueeze(1), torch.zeros_like(tail), tail / (x1 - alpha).unsqueeze(1))
        later = A[:, i + 1:, :]
        w = t.unsqueeze(1) * (later[:, :, i] + torch.einsum("bcr,br->bc", later[:, :, i + 1:], v))
        later[:, :, i] -= w
        later[:, :, i + 1:] -= w.unsqueeze(2) * v.unsqueeze(1)
        A[:, i, i] = torch.where(skip, x1, alpha)
        A[:, i, i + 1:] = torch.where(skip.unsqueeze(1), tail, v)
        tau[:, i] = t
    return A, tau


def exact(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    if kind in ("chain", "solve", "inverse"):
        n, b = case["n"], case["batch"]
        A = d["A"][:, :, :n]
        lu, piv = _lu64(A)
        LU = torch.cat([lu, d["A"][:, :, n:].double()], 2)
        out = [LU, piv, torch.zeros(b, dtype=torch.int32, device=_DEV)]
        if "B" in d:
            out.append(_solve64(A, d["B"], case.get("trans", "N")))
        if kind == "inverse" or case.get("inverse"):
            out += [torch.linalg.inv(A.double().transpose(1, 2)).transpose(1, 2).contiguous(), torch.zeros(b, dtype=torch.int32, device=_DEV)]
        return out
    if kind == "grouped":
        LU, X, piv = [], [], []
        for n, A, B in zip(d["orders"], d["A"], d["B"]):
            lu, p = _lu64(A)
            x = _solve64(A, B)
            for out, v in ((LU, lu), (X, x)):  # every instance starts at a multiple of 64 floats
                flat = v.reshape(v.shape[0], -1)
                out.append(torch.nn.functional.pad(flat, (0, -flat.shape[1] % 64)).reshape(-1))
            piv.append(p.reshape(-1))
        return [torch.cat(LU), torch.cat(piv), torch.zeros(case["count"], dtype=torch.int32, device=_DEV), torch.cat(X)]
    if kind == "refine":
        return [_solve64(d["A"], d["B"]), torch.zeros(case["batch"], dtype=torch.int32, device=_DEV), None]
    if kind == "grad":
        X, dB = _solve64(d["A"], d["B"]), _solve64(d["A"], d["dX"], "T")
        return [X, -torch.einsum("bri,brj->bji", dB, X), dB]
    if kind == "geqrf":
        return list(_householder64(d["A"], case["n"], False))
    if kind == "gels":
        n = case["n"]
        Q = _householder64(torch.cat([d["A"], d["C"]], 1), n, True)[0]
        Q, X = Q[:, :n].contiguous(), Q[:, n:].contiguous()
        R = Q[:, :, :n].transpose(1, 2).triu()
        X[:, :, :n] = torch.linalg.solve_triangular(R, X[:, :, :n].transpose(1, 2), upper=True).transpose(1, 2)
        return [Q, X, torch.zeros(case["batch"], dtype=torch.int32, device=_DEV)]
    dt = torch.complex128 if kind == "cgemm" else torch.float64

    def op(X, t):  # column-major storage holds the transpose
        X = X.to(dt)
        return X.transpose(1, 2) if t == "N" else (X.conj() if t == "C" else X)

    P = torch.matmul(op(d["A"], case["ta"]), op(d["B"], case["tb"])).transpose(1, 2)
    return (P if kind == "gemm" else _ALPHA * P + _BETA * d["C"].to(dt)).contiguous()
