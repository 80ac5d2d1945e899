"""The calls this engine is timed on, with their inputs and their results in
64 bits: single solves from the tutorial's size to an atlas slice, in FP64 and
in the split-bf16 form, with a fixed length and with the stationary stop; the
consensus workflow (batched restarts, consensus matrices and their summaries);
sparse inputs; and ranks above 32.

V has the structure of log-normalised single-cell counts (gamma programs, 70 %
of their entries zero, Dirichlet usages, log-normal library sizes, Poisson
counts, columns scaled to 1e4, log1p), drawn on the GPU from the seed.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rust-nmf_b200"))
import nmf_rs  # noqa: E402
from nmf_rs import _native, consensus  # noqa: E402

F64 = torch.float64
EPS = 1e-9                        # nmf()'s default eps
DEPS = float(np.finfo(np.float64).eps)  # brunet's clamp


def listed():
    return [
        # The tutorial's call: nmf() on host arrays of 200 x 60, brunet (the
        # default method), 200 iterations.  All latency.
        dict(name="host_brunet_200x60", kind="host", method="brunet", n=200, p=60, rank=5,
             iters=200),
        # A gene-selected subset of a data set: V (36 MB) stays in L2.
        dict(name="lee_1500x3000", kind="solve", method="lee", n=1500, p=3000, rank=8, iters=100),
        # The pbmc8k shape, brunet, fixed length.
        dict(name="brunet_2000x7750", kind="solve", method="brunet", n=2000, p=7750, rank=10,
             iters=100),
        # The same with the stationary stop, which records the objective of
        # every iteration (deviances).
        dict(name="stationary_brunet_2000x7750", kind="stationary", method="brunet", n=2000,
             p=7750, rank=10, iters=60),
        # Slices of an atlas in the reference's precision: V is far above L2.
        dict(name="lee_f64_20000x40000", kind="atlas", method="lee", n=20000, p=40000, rank=20,
             iters=10),
        dict(name="brunet_f64_20000x20000", kind="atlas", method="brunet", n=20000, p=20000,
             rank=20, iters=10),
        # The same kind of slice in the precision form (25 iterations, the
        # last two in FP64).
        dict(name="lee_bf16x3_20000x60000", kind="mixed", method="lee", n=20000, p=60000, rank=20,
             iters=25),
        dict(name="brunet_bf16x3_20000x60000", kind="mixed", method="brunet", n=20000, p=60000,
             rank=20, iters=25),
        # Consensus clustering: restarts of every rank 2..10 as one batch.
        dict(name="consensus_solves_2000x5000", kind="batch", n=2000, p=5000, rank_lo=2,
             rank_hi=10, runs=8, iters=40),
        # ... and the consensus matrices, cophenetic correlation and
        # dispersion of its ranks.
        dict(name="consensus_matrices_5000", kind="stats", p=5000, rank_lo=2, rank_hi=10, runs=64),
        # A sparse atlas slice (CSR, 10 % stored).
        dict(name="sparse_brunet_20000x50000", kind="sparse", method="brunet", n=20000, p=50000,
             rank=20, density=0.10, iters=5),
        # Many programs: a rank above 32.
        dict(name="wide_lee_5000x20000_r50", kind="wide", method="lee", n=5000, p=20000, rank=50,
             iters=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "solve", "solve", "stationary", "atlas", "atlas", "mixed", "mixed",
                       "batch", "stats", "sparse", "wide"])
    if kind == "host":
        return dict(kind=kind, method=rng.choice(["brunet", "brunet", "lee"]),
                    n=_log(rng, 40, 1000), p=_log(rng, 30, 2000), rank=rng.randint(2, 12),
                    iters=rng.randint(100, 200))
    if kind == "solve":
        return dict(kind=kind, method=rng.choice(["lee", "brunet", "hals", "dnmf"]),
                    n=_log(rng, 500, 5000), p=_log(rng, 1000, 50000), rank=rng.randint(5, 30),
                    iters=rng.randint(25, 100))
    if kind == "stationary":
        return dict(kind=kind, method=rng.choice(["brunet", "lee"]), n=_log(rng, 500, 4000),
                    p=_log(rng, 1000, 20000), rank=rng.randint(4, 20), iters=rng.randint(40, 80))
    if kind == "atlas":
        return dict(kind=kind, method=rng.choice(["lee", "brunet"]), n=_log(rng, 8000, 20000),
                    p=_log(rng, 10000, 40000), rank=rng.randint(10, 30), iters=rng.randint(5, 10))
    if kind == "mixed":
        return dict(kind=kind, method=rng.choice(["lee", "brunet"]), n=_log(rng, 8000, 20000),
                    p=_log(rng, 15000, 60000), rank=rng.randint(10, 30), iters=25)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 1000, 2000), p=_log(rng, 2000, 5000), rank_lo=2,
                    rank_hi=rng.randint(5, 12), runs=rng.randint(6, 10), iters=rng.randint(25, 40))
    if kind == "stats":
        lo = rng.randint(2, 6)
        return dict(kind=kind, p=_log(rng, 800, 5000), rank_lo=lo, rank_hi=lo + rng.randint(0, 8),
                    runs=rng.randint(16, 64))
    if kind == "sparse":
        return dict(kind=kind, method=rng.choice(["brunet", "lee", "hals"]),
                    n=_log(rng, 5000, 20000), p=_log(rng, 8000, 50000), rank=rng.randint(8, 30),
                    density=round(rng.uniform(0.03, 0.12), 3), iters=5)
    return dict(kind=kind, method=rng.choice(["lee", "brunet", "hals"]), n=_log(rng, 1500, 5000),
                p=_log(rng, 4000, 20000), rank=rng.randint(33, 96), iters=rng.randint(5, 10))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _counts(g, n, p, k, ld):
    """V (n x ld f64, columns past p zero), its programs W_true and usages H_true."""
    w = torch._standard_gamma(torch.full((n, k), 0.5, dtype=F64, device="cuda"), generator=g)
    w[torch.rand((n, k), generator=g, device="cuda", dtype=F64) < 0.7] = 0.0
    V = torch.zeros((n, ld), dtype=F64, device="cuda")
    H = torch.empty((k, p), dtype=F64, device="cuda")
    for c0 in range(0, p, 8192):
        c = min(8192, p - c0)
        h = torch._standard_gamma(torch.full((k, c), 0.2, dtype=F64, device="cuda"), generator=g)
        h /= h.sum(0, keepdim=True).clamp_min(1e-300)
        lib = torch.empty(c, dtype=F64, device="cuda").log_normal_(7.0, 0.5, generator=g)
        counts = torch.poisson((w @ h) * lib[None, :], generator=g)
        col = counts.sum(0, keepdim=True)
        V[:, c0:c0 + c] = torch.log1p(counts * torch.where(col > 0, 1e4 / col.clamp_min(1e-300),
                                                           torch.zeros_like(col)))
        H[:, c0:c0 + c] = h
    return V, w, H


def _truth(rank):
    return max(2, min(20, rank))


def _dense_inputs(case, seed):
    g = _gen(seed)
    n, p, r = case["n"], case["p"], case["rank"]
    ld = (p + 15) // 16 * 16
    # The HALS family starts near programs of the data, as from an NNDSVD
    # start (a uniform start makes its sweeps ill conditioned).
    near = case["method"] in ("hals", "dnmf")
    V, w, h = _counts(g, n, p, r if near else _truth(r), ld)
    top = float(V.max())
    W0 = torch.rand((n, r), generator=g, device="cuda", dtype=F64)
    H0 = torch.rand((r, p), generator=g, device="cuda", dtype=F64)
    if near:
        W0 = w + 0.1 * W0
        H0 = top * (h + 0.1 * H0)
    else:
        W0 = W0 * top
        H0 = H0 * top
    return V, ld, W0, H0


def _csr(V, density, g):
    """V's stored entries thinned or filled to about `density` of all, as CSR."""
    n, p = V.shape
    indptr = [torch.zeros(1, dtype=torch.int64, device="cuda")]
    cols, vals = [], []
    for i0 in range(0, n, 1024):
        blk = V[i0:i0 + 1024]
        keep = torch.rand(blk.shape, generator=g, device="cuda") < density
        # a kept entry without a count holds a small one
        blk = torch.where(keep, blk.clamp_min(0.5), torch.zeros((), dtype=F64, device="cuda"))
        csr = blk.to_sparse_csr()
        indptr.append(csr.crow_indices().diff())
        cols.append(csr.col_indices().to(torch.int32))
        vals.append(csr.values())
    return torch.cat(indptr).cumsum(0), torch.cat(cols), torch.cat(vals)


def _sparse_inputs(case, seed):
    g = _gen(seed)
    n, p, r = case["n"], case["p"], case["rank"]
    V, w, h = _counts(g, n, p, r, p)
    indptr, indices, data = _csr(V, case["density"], g)
    W0 = torch.rand((n, r), generator=g, device="cuda", dtype=F64)
    H0 = torch.rand((r, p), generator=g, device="cuda", dtype=F64)
    if case["method"] == "hals":
        W0, H0 = w + 0.1 * W0, h + 0.1 * H0
    return indptr, indices, data, W0, H0


def _batch_inputs(case, seed):
    g = _gen(seed)
    n, p = case["n"], case["p"]
    V, _, _ = _counts(g, n, p, 6, p)
    mean = float(V.mean())
    ranks, W, H = [], [], []
    for k in range(case["rank_lo"], case["rank_hi"] + 1):
        for _ in range(case["runs"]):
            s = math.sqrt(mean / k)
            ranks.append(k)
            W.append(torch.rand((n, k), generator=g, device="cuda", dtype=F64) * s)
            H.append(torch.rand((k, p), generator=g, device="cuda", dtype=F64) * s)
    return V, np.array(ranks, dtype=np.int32), torch.cat(W, 1).contiguous(), torch.cat(H, 0)


def _stats_inputs(case, seed):
    """The stacked H of every run: most columns keep their cluster, some
    waver between two of them (so the consensus has intermediate values)."""
    g = _gen(seed)
    p = case["p"]
    ranks, H = [], []
    for k in range(case["rank_lo"], case["rank_hi"] + 1):
        home = torch.randint(0, k, (p,), generator=g, device="cuda")
        away = torch.randint(0, k, (p,), generator=g, device="cuda")
        waver = 0.5 * torch.rand(p, generator=g, device="cuda") ** 3
        for _ in range(case["runs"]):
            lab = torch.where(torch.rand(p, generator=g, device="cuda") < waver, away, home)
            h = torch.rand((k, p), generator=g, device="cuda", dtype=F64)
            h[lab, torch.arange(p, device="cuda")] += 1.0
            perm = torch.randperm(k, generator=g, device="cuda")
            ranks.append(k)
            H.append(h[perm])
    return np.array(ranks, dtype=np.int32), torch.cat(H, 0).contiguous()


_kept = {}


def _context():
    """The engine context and the stream a program keeps for its device calls."""
    if not _kept:
        _kept["ctx"] = _native.Context(0)
        _kept["stream"] = torch.cuda.Stream()
    return _kept["ctx"], _kept["stream"]


def _options(case):
    o = _native.default_options()
    o.method = _native.parse_method(case["method"])
    o.max_iter = case["iters"]
    if case["kind"] == "stationary":
        o.stop = _native.parse_stop("stationary")
    if case["kind"] == "mixed":
        o.precision = _native.PRECISIONS["bf16x3"]
    return o


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "host":
        V, _, W0, H0 = _dense_inputs(case, seed)
        st.update(V=np.ascontiguousarray(V[:, :case["p"]].cpu().numpy()), W0=W0.cpu().numpy(),
                  H0=H0.cpu().numpy())
        return st
    st["ctx"], st["stream"] = _context()
    if kind == "batch":
        V, ranks, W0, H0 = _batch_inputs(case, seed)
        st.update(V=V, ranks=ranks, W0=W0, H0=H0)
    elif kind == "stats":
        ranks, H = _stats_inputs(case, seed)
        st.update(ranks=ranks, H=H)
    elif kind == "sparse":
        indptr, indices, data, W0, H0 = _sparse_inputs(case, seed)
        st.update(indptr=indptr, indices=indices, data=data, W0=W0, H0=H0, opts=_options(case))
    else:
        V, ld, W0, H0 = _dense_inputs(case, seed)
        st.update(V=V, ld=ld, W0=W0, H0=H0, opts=_options(case))
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "host":
        res = nmf_rs.nmf(st["V"], case["rank"], case["method"], W0=st["W0"], H0=st["H0"],
                         max_iter=case["iters"])
        return {"W": res.W, "H": res.H}
    ctx, stream = st["ctx"], st["stream"]
    lib = _native.load()
    with torch.cuda.stream(stream):
        if kind == "stats":
            return _run_stats(st, ctx, stream, lib)
        W, H = st["W0"].clone(), st["H0"].clone()
        s = stream.cuda_stream
        if kind == "batch":
            n, p = case["n"], case["p"]
            _native.check(lib.nmfcu_run_batch_device(
                ctx.handle, _native.parse_method("brunet"), _native.PRECISIONS["fp32"],
                case["iters"], n, p, _ptr(st["V"]), p, len(st["ranks"]),
                consensus._ranks_ptr(st["ranks"]), _ptr(W), _ptr(H), ctypes.c_void_p(s)))
            # computed in f32 from an f32 V, and handed on as such
            return {"W": W.float(), "H": H.float()}
        if kind == "sparse":
            nd, ni = ctypes.c_int64(0), ctypes.c_int64(0)
            _native.check(lib.nmfcu_run_csr_device(
                ctx.handle, ctypes.byref(st["opts"]), case["n"], case["p"], case["rank"],
                st["data"].numel(), _ptr(st["indptr"]), _ptr(st["indices"]), _ptr(st["data"]),
                _ptr(W), _ptr(H), None, ctypes.byref(nd), ctypes.byref(ni), ctypes.c_void_p(s)))
            return {"W": W, "H": H}
        dev = None
        if kind == "stationary":
            dev = torch.empty(case["iters"] + 1, dtype=F64, device="cuda")
        n_iter, n_dev = ctx.run(st["opts"], case["n"], case["p"], case["rank"],
                                st["V"].data_ptr(), _native.F64, st["ld"], W.data_ptr(),
                                H.data_ptr(), dev_ptr=dev.data_ptr() if dev is not None else 0,
                                stream=s)
        if kind == "mixed":  # the precision form's factors, handed on in f32
            return {"W": W.float(), "H": H.float()}
        if dev is not None:
            return {"W": W, "H": H, "deviances": dev[:n_dev], "n_iter": n_iter}
        return {"W": W, "H": H}


def _run_stats(st, ctx, stream, lib):
    case = st["case"]
    p, runs = case["p"], case["runs"]
    count = case["rank_hi"] - case["rank_lo"] + 1
    C = torch.empty((count, p, p), dtype=torch.float32, device="cuda")
    for m in range(count):
        sel = np.arange(m * runs, (m + 1) * runs, dtype=np.int32)
        _native.check(lib.nmfcu_consensus_device(
            ctx.handle, p, len(st["ranks"]), consensus._ranks_ptr(st["ranks"]), _ptr(st["H"]),
            runs, consensus._ranks_ptr(sel), _ptr(C[m]), ctypes.c_void_p(stream.cuda_stream)))
    stats = consensus.consensus_stats_batch(C, ctx)
    return {"consensus": C, "cophenetic": torch.tensor([s[0] for s in stats], dtype=F64),
            "dispersion": torch.tensor([s[1] for s in stats], dtype=F64)}


# ---------------------------------------------------------------------------
# Work and results in 64 bits
# ---------------------------------------------------------------------------

def work(case):
    """Bytes and flops a pass cannot do without.  An iteration reads V twice
    (the W update needs the new H) and does a contraction each time; brunet
    also forms W H each time.  V counts in the precision that the form streams
    it in."""
    kind = case["kind"]
    if kind == "stats":
        p, count = case["p"], case["rank_hi"] - case["rank_lo"] + 1
        hbytes = 8 * p * case["runs"] * sum(range(case["rank_lo"], case["rank_hi"] + 1))
        # consensus matrices written and read once for the trees, whose
        # average-linkage updates touch every pair of clusters once.
        return {"bytes": hbytes + count * p * p * (4 + 4), "flops": count * p * p * 3}
    n, p, it = case["n"], case["p"], case["iters"]
    if kind == "batch":
        R = case["runs"] * sum(range(case["rank_lo"], case["rank_hi"] + 1))
        return {"bytes": it * 2 * 4 * n * p + 16 * R * (n + p), "flops": it * 8 * n * p * R}
    r = case["rank"]
    fl = 8 if case["method"] == "brunet" else 4
    factors = 16 * r * (n + p)
    if kind == "sparse":
        nnz = case["density"] * n * p
        return {"bytes": it * 2 * 12 * nnz + factors, "flops": it * fl * nnz * r}
    per = 4 if kind == "mixed" else 8
    passes = it * (3 if kind == "stationary" else 2)
    return {"bytes": passes * per * n * p + factors, "flops": it * fl * n * p * r}


def _lee(V, W, H):
    H = torch.clamp_min(H * (W.T @ V), EPS) / ((W.T @ W) @ H + EPS)
    W = torch.clamp_min(W * (V @ H.T), EPS) / (W @ (H @ H.T) + EPS)
    s = W.sum(0, keepdim=True)
    return torch.where(s > 0, W / s, W), H


def _ratio(V, W, H):
    """V / (W H) (0 where W H is 0), of a dense V or of a V given by its
    stored entries (rows, columns, values), then as a dense or sparse matrix."""
    wh = W @ H
    return torch.where(wh != 0, V / wh, torch.zeros((), dtype=F64, device="cuda"))


def _brunet(V, W, H, it):
    H = H * (W.T @ _ratio(V, W, H)) / W.sum(0)[:, None]
    W = W * (_ratio(V, W, H) @ H.T) / H.sum(1)[None, :]
    if it % 10 == 0:
        W, H = W.clamp_min(DEPS), H.clamp_min(DEPS)
    return W, H


def _sweep(X, N, G):
    """Gauss-Seidel over the rows of X (r x m): numerators N, Gram G."""
    X = X.clone()
    for k in range(X.shape[0]):
        g = G[k].clone()
        g[k] = 0.0
        X[k] = torch.clamp_min((N[k] - g @ X) / G[k, k].clamp_min(EPS), EPS)
    return X


def _hals(V, W, H, diag):
    H = _sweep(H, W.T @ V, W.T @ W)
    G = H @ H.T
    W = _sweep(W.T.contiguous(), H @ V.T if not V.is_sparse_csr else (V @ H.T).T, G).T.contiguous()
    if diag:  # dnmf: unit columns and rows, the scales on H
        nw, nh = (W * W).sum(0).sqrt(), G.diagonal().sqrt()
        W = torch.where(nw > 0, W / nw, W)
        H = torch.where(nh[:, None] > 0, H / nh[:, None], H) * (nw * nh)[:, None]
    return W, H


def _kl(V, W, H):
    wh = W @ H
    t = torch.where((V > 0) & (wh > 0), V * torch.log(V / wh) - V + wh,
                    torch.zeros((), dtype=F64, device="cuda"))
    return float(torch.where(V > 0, t, wh).sum())


def _exact_dense(V, W, H, case):
    method, dev = case["method"], []

    def record():
        if case["kind"] == "stationary":
            dev.append(_kl(V, W, H) if method == "brunet"
                       else 0.5 * float(((V - W @ H) ** 2).sum()))

    record()
    for it in range(1, case["iters"] + 1):
        if method == "lee":
            W, H = _lee(V, W, H)
        elif method == "brunet":
            W, H = _brunet(V, W, H, it)
        else:
            W, H = _hals(V, W, H, method == "dnmf")
        record()
    return W, H, dev


def _exact_sparse(case, seed):
    indptr, indices, data, W, H = _sparse_inputs(case, seed)
    n, p = case["n"], case["p"]
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), indptr.diff())
    cols = indices.long()
    V = torch.zeros((n, p), dtype=F64, device="cuda")
    V[rows, cols] = data
    del rows, cols
    for it in range(1, case["iters"] + 1):
        if case["method"] == "lee":
            W, H = _lee(V, W, H)
        elif case["method"] == "brunet":
            W, H = _brunet(V, W, H, it)
        else:
            W, H = _hals(V, W, H, False)
    return {"W": W, "H": H}


def exact(case, seed):
    """What run() computes, in plain 64-bit torch.  The cophenetic correlation
    (an average-linkage tree) has no such value here."""
    kind = case["kind"]
    if kind == "sparse":
        return _exact_sparse(case, seed)
    if kind == "stats":
        ranks, H = _stats_inputs(case, seed)
        p, runs = case["p"], case["runs"]
        cons, disp, row = [], [], 0
        for k in range(case["rank_lo"], case["rank_hi"] + 1):
            C = torch.zeros((p, p), dtype=F64, device="cuda")
            for _ in range(runs):
                hot = torch.zeros((k, p), dtype=F64, device="cuda")
                hot[H[row:row + k].argmax(0), torch.arange(p, device="cuda")] = 1.0
                C += hot.T @ hot
                row += k
            C /= runs
            cons.append(C.float())
            disp.append(float((4.0 * (C - 0.5) ** 2).mean()))
        return {"consensus": torch.stack(cons).double(), "cophenetic": None,
                "dispersion": torch.tensor(disp, dtype=F64)}
    if kind == "batch":
        V, ranks, W0, H0 = _batch_inputs(case, seed)
        Ws, Hs, off = [], [], 0
        for r in ranks:
            r = int(r)
            W, H = W0[:, off:off + r].contiguous(), H0[off:off + r].contiguous()
            for it in range(1, case["iters"] + 1):
                W, H = _brunet(V, W, H, it)
            Ws.append(W)
            Hs.append(H)
            off += r
        return {"W": torch.cat(Ws, 1), "H": torch.cat(Hs, 0)}
    V, _, W0, H0 = _dense_inputs(case, seed)
    W, H, dev = _exact_dense(V[:, :case["p"]], W0, H0, case)
    if kind == "stationary":
        return {"W": W, "H": H, "deviances": torch.tensor(dev, dtype=F64), "n_iter": None}
    return {"W": W, "H": H}
