"""Performance cases of the embedding pipeline: what a program built on this
package has it do, stage by stage, over the range of sizes it is used at.

The stages are the pipeline's own entry points: the NetSMF sparsifier
(generate_trunc_log_matrix_v2), the SpMM of the C ABI (lne_spmm), the
randomized SVD (randsvd), the spectral propagation (chebyshev_expansion) and
its gradient (ChebyshevPropagation), the dense embedding
(get_embedding_dense), and the four of them in a row.  Graphs are Chung-Lu
power-law graphs (exponent 2.1), the family of this repository's benchmark,
drawn on the GPU; "BlogCatalog-sized" is n = 10,312 and m = 333,983 edges,
"YouTube-sized" n = 1,138,499 and m = 2,990,443.
"""
import ctypes
import math

import numpy as np
import torch

from lightne_gb300 import _lib
from lightne_gb300.api import (CSR, ChebyshevPropagation, Context, Graph, chebyshev_expansion, generate_trunc_log_matrix_v2,
                               get_embedding_dense, randsvd)

DEV = "cuda:0"
BLOG = {"n": 10312, "m": 333983}
YOUTUBE = {"n": 1138499, "m": 2990443}
SVD_SEED = 777
MU, S_ARG = 0.2, 0.5
X_TYPES = {"fp32": (_lib.LNE_PREC_FP32, torch.float32), "bf16": (_lib.LNE_PREC_BF16, torch.bfloat16),
           "fp16": (_lib.LNE_PREC_FP16, torch.float16)}


def listed():
    return [
        # the smallest graphs (a test graph, a subgraph, a parameter search):
        # one call is mostly launches, allocations and waits
        {"name": "sparsify small", "kind": "sparsify", "n": 1000, "m": 8000, "walk_len": 10, "per_edge": 20.0,
         "negative": 1, "upper": False},
        # a dense social graph at the usual 20 T m samples
        {"name": "sparsify BlogCatalog", "kind": "sparsify", **BLOG, "walk_len": 10, "per_edge": 100.0, "negative": 1,
         "upper": False},
        # the benchmark's sparsifier: 299M samples, a 351M-entry matrix
        {"name": "sparsify YouTube", "kind": "sparsify", **YOUTUBE, "walk_len": 10, "per_edge": 50.0, "negative": 1,
         "upper": False},
        # the product of a sparse matrix and a thin dense block through the C
        # ABI, 16-bit operand, ragged width (one power iteration)
        {"name": "spmm fp16", "kind": "spmm", "n": 200003, "avg": 120, "d": 138, "x": "fp16"},
        # the command line's defaults: rank 256, dim 128, FP32
        {"name": "randsvd BlogCatalog rank 256", "kind": "randsvd", **BLOG, "walk_len": 10, "per_edge": 100.0,
         "rank": 256, "dim": 128, "precision": "fp32"},
        # the benchmark's randomized SVD in its 16-bit form
        {"name": "randsvd YouTube fp16", "kind": "randsvd", **YOUTUBE, "walk_len": 10, "per_edge": 50.0, "rank": 138,
         "dim": 128, "precision": "fp16"},
        # propagation of a small embedding, odd sizes
        {"name": "propagate small fp32", "kind": "propagate", "n": 2001, "m": 15000, "dim": 33, "order": 10,
         "precision": "fp32"},
        # propagation of an ordinary graph
        {"name": "propagate BlogCatalog fp32", "kind": "propagate", **BLOG, "dim": 128, "order": 10,
         "precision": "fp32"},
        # the benchmark's propagation
        {"name": "propagate YouTube fp16", "kind": "propagate", **YOUTUBE, "dim": 128, "order": 10,
         "precision": "fp16"},
        # a training step through the propagation: forward, gradients of the
        # embedding and of both filter parameters
        {"name": "train step YouTube fp32", "kind": "train", **YOUTUBE, "dim": 128, "order": 10, "precision": "fp32"},
        # the dense SVD embedding of a propagated embedding
        {"name": "dense embedding YouTube", "kind": "dense", "n": YOUTUBE["n"], "dim": 128},
        # a whole embedding of a small graph, end to end
        {"name": "pipeline small", "kind": "pipeline", "n": 3001, "m": 30000, "walk_len": 10, "per_edge": 50.0,
         "rank": 42, "dim": 32, "order": 10, "precision": "fp32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sparsify", "sparsify", "spmm", "randsvd", "propagate", "propagate", "train", "dense",
                       "pipeline"])
    if kind == "spmm":
        n = _log_int(rng, 1000, 400000)
        avg = min(n // 4, _log_int(rng, 4, min(200, 24000000 // n)))
        return {"kind": kind, "n": n, "avg": avg, "d": _log_int(rng, 16, 160), "x": rng.choice(["fp32", "bf16", "fp16"])}
    if kind == "dense":
        return {"kind": kind, "n": _log_int(rng, 1000, 1100000), "dim": rng.choice([16, 32, 50, 64, 100, 128])}
    n = _log_int(rng, 700, 1000000)
    m = int(n * rng.uniform(2.5, min(12.0, 2900000.0 / n if n > 260000 else 12.0)))
    case = {"kind": kind, "n": n, "m": m}
    if kind in ("sparsify", "randsvd", "pipeline"):
        case["walk_len"] = rng.choice([2, 5, 10])
        # at most 250M samples in all
        case["per_edge"] = round(rng.uniform(5.0, min(60.0, 2.5e8 / (2.0 * m))), 2)
    if kind == "sparsify":
        case["negative"] = rng.choice([1, 1, 5])
        case["upper"] = rng.random() < 0.25
    if kind in ("randsvd", "pipeline"):
        case["dim"] = rng.choice([32, 64, 100, 128])
        case["rank"] = case["dim"] + rng.choice([10, 28])
    if kind in ("propagate", "train"):
        case["dim"] = rng.choice([16, 32, 50, 64, 100, 128])
    if kind in ("propagate", "train", "pipeline"):
        case["order"] = rng.choice([3, 6, 10])
    if kind != "sparsify":
        case["precision"] = rng.choice(["fp32", "fp16", "fp16", "bf16"]) if kind != "train" else rng.choice(["fp32", "fp16"])
    return case


# --- inputs -----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)


def _power_law_ids(n, count, g, exponent=2.1):
    """Vertex ids drawn in proportion to (i + 1)^(-1 / (exponent - 1))."""
    w = torch.arange(1, n + 1, dtype=torch.float64, device=DEV).pow(-1.0 / (exponent - 1.0))
    cdf = torch.cumsum(w, 0)
    u = torch.rand(count, dtype=torch.float64, device=DEV, generator=g) * cdf[-1]
    return torch.searchsorted(cdf, u, right=True).clamp_(max=n - 1)


def _graph(n, m, seed):
    """Chung-Lu graph with about m undirected edges: (offsets, neighbours),
    symmetric, rows sorted (vertices without edges occur, as in real files)."""
    g = _gen(seed)
    have = torch.empty(0, dtype=torch.int64, device=DEV)
    for _ in range(12):
        want = int((m - have.numel()) * 1.6) + 4096
        a, b = _power_law_ids(n, want, g), _power_law_ids(n, want, g)
        keep = a != b
        lo, hi = torch.minimum(a, b)[keep], torch.maximum(a, b)[keep]
        have = torch.unique(torch.cat([have, lo * n + hi]))
        if have.numel() >= m:
            have = have[torch.randperm(have.numel(), device=DEV, generator=g)[:m]]
            break
    lo, hi = have // n, have % n
    keys = torch.sort(torch.cat([lo * n + hi, hi * n + lo]))[0]
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    return off, (keys % n).to(torch.int32)


def _sparse_matrix(n, avg, seed):
    """CSR of the sparsifier's kind: power-law rows and columns, rows sorted,
    positive log-like values."""
    g = _gen(seed)
    count = int(n) * int(avg)
    keys = torch.unique(_power_law_ids(n, count, g, 2.6) * n + _power_law_ids(n, count, g, 2.6))
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row_ptr[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    val = torch.rand(keys.numel(), dtype=torch.float32, device=DEV, generator=g).mul_(6.0).add_(0.01)
    return row_ptr, (keys % n).to(torch.int32), val


def _embedding(n, dim, seed):
    """What the SVD stage hands on: U sqrt(S) with a decaying spectrum, in
    a rotated basis."""
    g = _gen(seed)
    x = torch.randn(n, dim, dtype=torch.float32, device=DEV, generator=g)
    s = torch.arange(1, dim + 1, dtype=torch.float32, device=DEV).pow(-0.75)
    v = torch.linalg.qr(torch.randn(dim, dim, dtype=torch.float64, device=DEV, generator=g))[0].float()
    return ((x * s) @ v).mul_(1.0 / math.sqrt(n)).contiguous()


def _sample_args(case):
    """sample_ratio and table size for about per_edge samples per directed entry."""
    total = case["per_edge"] * 2.0 * case["m"]
    t_n_logn = case["walk_len"] * case["n"] * math.log(case["n"])
    return {"walk_len": case["walk_len"], "sample_ratio": total / t_n_logn, "table_size": int(total) + 1000}


def _sparsify(st, seed, negative=1, upper=False):
    return generate_trunc_log_matrix_v2(st["ctx"], st["graph"], seed=seed, upper=upper, negative=negative, **st["args"])[0]


def prepare(case, seed):
    st = {"case": case, "kind": case["kind"], "seed": int(seed), "ctx": Context(0)}
    kind, n = case["kind"], case["n"]
    if kind == "spmm":
        d, (_, dtype) = case["d"], X_TYPES[case["x"]]
        ld = (d + 7) // 8 * 8
        st["arrays"] = _sparse_matrix(n, case["avg"], seed)
        rp, col, val = st["arrays"]
        st["csr"] = CSR.wrap_device(st["ctx"], n, col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr())
        X = torch.zeros(n, ld, dtype=torch.float32, device=DEV)
        X[:, :d] = torch.randn(n, d, dtype=torch.float32, device=DEV, generator=_gen(seed + 1))
        st["X"], st["ld"] = X.to(dtype), ld
        st["Y"] = torch.empty(n, d, dtype=torch.float32, device=DEV)
        return st
    if kind == "dense":
        st["x"] = _embedding(n, case["dim"], seed)
        return st
    off, nbrs = _graph(n, case["m"], seed)
    torch.cuda.synchronize()
    st["graph"] = Graph.from_device(st["ctx"], n, off.data_ptr(), nbrs.data_ptr(), nbrs.numel())
    if kind in ("sparsify", "randsvd", "pipeline"):
        st["args"] = _sample_args(case)
    if kind == "sparsify":
        st["out"] = _empty_csr(case)
    if kind == "randsvd":
        st["csr"] = _sparsify(st, seed)
    if kind in ("propagate", "train"):
        st["a"] = _embedding(n, case["dim"], seed + 1)
    if kind == "train":
        st["a"].requires_grad_(True)
        st["mu"] = torch.tensor(MU, device=DEV, requires_grad=True)
        st["s"] = torch.tensor(S_ARG, device=DEV, requires_grad=True)
        # the gradient of a linear read-out loss
        st["gy"] = torch.randn(n, case["dim"], dtype=torch.float32, device=DEV, generator=_gen(seed + 2))
    return st


# --- one pass ---------------------------------------------------------------

def _empty_csr(case, val_type=torch.float32):
    """The program's own arrays for a matrix: as large as it can get, zero
    past its entries."""
    cap = min(case["n"] ** 2, 2 * (int(_samples(case)) + case["m"]))
    return {"row_ptr": torch.zeros(case["n"] + 1, dtype=torch.int64, device=DEV),
            "col": torch.zeros(cap, dtype=torch.int32, device=DEV), "val": torch.zeros(cap, dtype=val_type, device=DEV)}


class _View:
    """A device array of the library, for torch.as_tensor: the tensor holds
    this object, which holds the array's owner."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _take(csr, out):
    """The matrix in the program's arrays; the library's copy is freed."""
    rp, col, val = csr.device_ptrs()
    out["row_ptr"].copy_(torch.as_tensor(_View(csr, rp, csr.n + 1, "<i8"), device=DEV))
    out["col"][:csr.nnz].copy_(torch.as_tensor(_View(csr, col, csr.nnz, "<i4"), device=DEV))
    out["val"][:csr.nnz].copy_(torch.as_tensor(_View(csr, val, csr.nnz, "<f4"), device=DEV))
    csr.free()
    return out


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = st["kind"]
    if kind == "sparsify":
        return _take(_sparsify(st, st["seed"], case["negative"], case["upper"]), st["out"])
    if kind == "spmm":
        _lib.check(_lib.load().lne_spmm(ctx.handle, st["csr"].handle, X_TYPES[case["x"]][0],
                                        ctypes.c_void_p(st["X"].data_ptr()), st["ld"], case["d"], 1.0, 0.0,
                                        ctypes.c_void_p(st["Y"].data_ptr()), case["d"]))
        return st["Y"]
    if kind == "randsvd":
        emb, S, _ = randsvd(ctx, st["csr"], case["rank"], case["dim"], precision=case["precision"], seed=SVD_SEED)
        return {"emb": emb, "S": S}
    if kind == "propagate":
        y, a_out, _ = chebyshev_expansion(ctx, st["graph"], st["a"], case["dim"], order=case["order"], mu=MU, s=S_ARG,
                                          precision=case["precision"], return_a=True)
        return {"y": y, "a": a_out}
    if kind == "train":
        y = ChebyshevPropagation(st["a"], st["mu"], st["s"], ctx, st["graph"], order=case["order"],
                                 precision=case["precision"])
        ga, gmu, gs = torch.autograd.grad(y, (st["a"], st["mu"], st["s"]), st["gy"])
        return {"y": y, "ga": ga, "gmu": gmu, "gs": gs}
    if kind == "dense":
        emb, S = get_embedding_dense(ctx, st["x"], case["dim"])
        return {"emb": emb, "S": S}
    # the whole pipeline, as the command line runs it
    csr = _sparsify(st, st["seed"])
    emb, S, _ = randsvd(ctx, csr, case["rank"], case["dim"], precision=case["precision"], seed=SVD_SEED)
    csr.free()
    y, _ = chebyshev_expansion(ctx, st["graph"], emb, case["dim"], order=case["order"], mu=MU, s=S_ARG,
                               precision=case["precision"])
    pro, S2 = get_embedding_dense(ctx, y, case["dim"])
    return {"emb": emb, "S": S, "pro": pro, "S_pro": S2}


# --- the least a pass has to do ------------------------------------------------

def _samples(case):
    return case["per_edge"] * 2.0 * case["m"]


def _graph_bytes(case):
    return 8.0 * (case["n"] + 1) + 8.0 * case["m"]


def _nnz(case):
    """Entries of the sparsifier's matrix, about: two per distinct pair; on
    these graphs some 0.6 distinct pairs per sample, at most all pairs."""
    return min(0.9 * case["n"] ** 2, 1.2 * _samples(case))


def _prop_flops(case):
    # 2 (K - 1) products with the graph's operator and one with A + I
    return (2.0 * max(case["order"] - 1, 1) + 1.0) * 2.0 * (2.0 * case["m"] + case["n"]) * case["dim"]


def work(case):
    kind, n = case["kind"], float(case["n"])
    if kind == "sparsify":
        out = _nnz(case) * (0.5 if case["upper"] else 1.0)
        return {"bytes": _graph_bytes(case) + 8.0 * (n + 1) + 8.0 * out, "flops": 0}
    if kind == "spmm":
        nnz, d = 0.8 * n * case["avg"], case["d"]
        return {"bytes": 8.0 * (n + 1) + 8.0 * nnz + n * d * (4.0 if case["x"] == "fp32" else 2.0) + 4.0 * n * d,
                "flops": 2.0 * nnz * d}
    if kind == "dense":
        return {"bytes": 8.0 * n * case["dim"], "flops": 8.0 * n * case["dim"] ** 2}
    if kind == "propagate":
        return {"bytes": _graph_bytes(case) + 12.0 * n * case["dim"], "flops": _prop_flops(case)}
    if kind == "train":
        # forward; adjoint; the recursion again with its tangent
        return {"bytes": _graph_bytes(case) + 16.0 * n * case["dim"], "flops": 4.0 * _prop_flops(case)}
    nnz, r, d = _nnz(case), case["rank"], case["dim"]
    svd = {"bytes": 16.0 * nnz + 4.0 * n * d, "flops": 4.0 * nnz * r + 12.0 * n * r * r + 2.0 * n * r * d}
    if kind == "randsvd":
        return svd
    return {"bytes": _graph_bytes(case) + svd["bytes"] + 8.0 * n * d,
            "flops": svd["flops"] + _prop_flops(case) + 8.0 * n * d * d}


# --- 64-bit values ---------------------------------------------------------------

_M1, _M2 = -4658895280553007687, -7723592293110705685  # 0xbf58476d1ce4e5b9, 0x94d049bb133111eb


def _shr(x, s):
    return (x >> s) & ((1 << (64 - s)) - 1)


def _hash64(x):
    x = (x ^ _shr(x, 30)) * _M1
    x = (x ^ _shr(x, 27)) * _M2
    return x ^ _shr(x, 31)


def _umod(x, d):
    """x mod d for x as an unsigned 64-bit word, 1 <= d < 2^31."""
    hi, lo = _shr(x, 32), x & 0xFFFFFFFF
    return ((hi % d) * ((1 << 32) % d) + lo % d) % d


def _exact_sparsify(case, seed):
    """The path sampler of every directed entry in 64-bit integers, the pair
    counts, and the truncated logarithm in doubles."""
    n, T, args = case["n"], case["walk_len"], _sample_args(case)
    off, nbrs = _graph(n, case["m"], seed)
    deg = off[1:] - off[:-1]
    m_dir = nbrs.numel()
    ratio = float(np.float32(args["sample_ratio"]))
    total = float(T * n) * math.log(float(n)) * ratio
    inv_lambda = total / float(m_dir)
    exp_rv = int(inv_lambda)
    frac = inv_lambda - exp_rv
    u = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
    v = nbrs.to(torch.int64)
    s = _hash64(_hash64(((u << 32) | v) + int(seed)))
    todo = torch.full((m_dir,), exp_rv, dtype=torch.int64, device=DEV)

    def advance(state):
        x = _hash64(state)
        return x, _hash64(x)

    if frac > 1e-10:
        x, s = advance(s)
        # the word as a double, scaled by 2^-64
        as_double = (_shr(x, 32).double() * 4294967296.0 + (x & 0xFFFFFFFF).double()) * 2.0 ** -64
        todo += (as_double < frac).to(torch.int64)
    keys = []
    for i in range(exp_rv + 1):
        live = (todo > i).nonzero().flatten()
        if live.numel() == 0:
            break
        su, sv, ss = u[live], v[live], s[live]
        x, ss = advance(ss)
        r = _umod(x, torch.full_like(x, T)) + 1
        x, ss = advance(ss)
        k = _umod(x, r) + 1
        a, b, left_a, left_b = su.clone(), sv.clone(), k - 1, r - k
        for _ in range(T - 1):
            step_a = left_a > 0
            on = (step_a | (left_b > 0)).nonzero().flatten()
            if on.numel() == 0:
                break
            fa = step_a[on]
            cur = torch.where(fa, a[on], b[on])
            x, nxt = advance(ss[on])
            ss[on] = nxt
            to = v[off[cur] + _umod(x, deg[cur])]
            a[on] = torch.where(fa, to, a[on])
            b[on] = torch.where(fa, b[on], to)
            left_a[on] -= fa.to(torch.int64)
            left_b[on] -= (~fa).to(torch.int64)
        s[live] = ss
        keys.append((torch.minimum(a, b) << 32) | torch.maximum(a, b))
    keys, count = torch.unique(torch.cat(keys), return_counts=True)
    lo, hi = keys >> 32, keys & 0xFFFFFFFF
    factor = float(m_dir) * float(m_dir) / float(int(count.sum())) / 2 / float(case["negative"])
    w = count.double() * torch.where(lo == hi, 2.0, 1.0).double()
    logw = torch.log(w * factor / deg[lo].double() / deg[hi].double())
    keep = logw > 0
    lo, hi, logw = lo[keep], hi[keep], logw[keep]
    if not case["upper"]:
        offd = lo != hi
        lo, hi, logw = torch.cat([lo, hi[offd]]), torch.cat([hi, lo[offd]]), torch.cat([logw, logw[offd]])
    order = torch.sort(lo * n + hi)[1]
    out = _empty_csr(case, torch.float64)
    out["row_ptr"][1:] = torch.cumsum(torch.bincount(lo, minlength=n), 0)
    out["col"][:hi.numel()] = hi[order].to(torch.int32)
    out["val"][:hi.numel()] = logw[order]
    return out


def _bessel(k, x):
    """I_k(x) by its power series (x: a 64-bit tensor)."""
    h = x / 2
    term = torch.ones_like(x)
    for i in range(1, k + 1):
        term = term * h / i
    out = term
    for j in range(1, 40):
        term = term * h * h / (j * (j + k))
        out = out + term
    return out


def _propagate64(case, off, nbrs, a, mu, s):
    """(A + I)(a - sum_k c_k T_k a) and a - sum_k c_k T_k a in 64 bits."""
    n, order = case["n"], case["order"]
    A = torch.sparse_csr_tensor(off, nbrs.to(torch.int64), torch.ones(nbrs.numel(), dtype=torch.float64, device=DEV),
                                size=(n, n))
    inv = (1.0 / (off[1:] - off[:-1] + 1).double())[:, None]

    class Product(torch.autograd.Function):  # A is symmetric
        @staticmethod
        def forward(fctx, x):
            return A @ x

        @staticmethod
        def backward(fctx, g):
            return A @ g

    def M(x):
        return (1.0 - mu) * x - inv * (Product.apply(x) + x)

    t0, t1 = a, 0.5 * M(M(a)) - a
    conv = _bessel(0, s) * t0 - 2.0 * _bessel(1, s) * t1
    for k in range(2, order):
        t0, t1 = t1, M(M(t1)) - 2.0 * t1 - t0
        conv = conv + (-2.0 if k % 2 else 2.0) * _bessel(k, s) * t1
    out = a - conv
    return Product.apply(out) + out, out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sparsify":
        # 64-bit torch takes too long above this many draws in a row
        return _exact_sparsify(case, seed) if case["per_edge"] * case["m"] <= 1.6e8 else None
    if kind == "spmm":
        n, d = case["n"], case["d"]
        rp, col, val = _sparse_matrix(n, case["avg"], seed)
        X = torch.randn(n, d, dtype=torch.float32, device=DEV, generator=_gen(seed + 1)).to(X_TYPES[case["x"]][1])
        A = torch.sparse_csr_tensor(rp, col.to(torch.int64), val.double(), size=(n, n))
        return A @ X.double()
    if kind == "dense":
        # the embedding's columns are fixed up to their signs only
        x = _embedding(case["n"], case["dim"], seed).double()
        return {"emb": None, "S": torch.linalg.svdvals(torch.linalg.qr(x)[1])}
    if kind in ("propagate", "train"):
        off, nbrs = _graph(case["n"], case["m"], seed)
        a = _embedding(case["n"], case["dim"], seed + 1).double()
        mu = torch.tensor(float(np.float32(MU)), dtype=torch.float64, device=DEV)
        s = torch.tensor(float(np.float32(S_ARG)), dtype=torch.float64, device=DEV)
        if kind == "propagate":
            y, out = _propagate64(case, off, nbrs, a, mu, s)
            return {"y": y, "a": out}
        for t in (a, mu, s):
            t.requires_grad_(True)
        gy = torch.randn(case["n"], case["dim"], dtype=torch.float32, device=DEV, generator=_gen(seed + 2)).double()
        y, _ = _propagate64(case, off, nbrs, a, mu, s)
        ga, gmu, gs = torch.autograd.grad(y, (a, mu, s), gy)
        return {"y": y.detach(), "ga": ga, "gmu": gmu, "gs": gs}
    # the randomized SVD depends on its own random sketch
    return None
