"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values.  ``kind`` says which public entry point it goes
through:

* ``id64``    ``Handle.column_id`` on an FP64 matrix: the plain form (the reference
  driver's and the notebook's own runs).
* ``id32``    ``Handle.column_id`` on an FP32 matrix: the mixed-precision form.
* ``batch``   ``Batch.run`` + ``Batch.results``: many uneven FP32 blocks in one launch,
  in device memory or (``host``) in pinned host memory.
* ``adjoint`` forward and backward of ``fixed_skeleton_id_loss``.
* ``cpqr``    ``sketch_ids.cpqr_id``: deterministic column-pivoted QR ID.
* ``lupp``    ``sketch_ids.rand_lupp_os``: the sketched LU comparison ID.

All inputs come from a ``torch.Generator`` on the GPU seeded by ``seed``.
"""
import math

import numpy as np
import torch

from robust_blockwise_random_pivoting_gb300.adjoint import fixed_skeleton_id_loss
from robust_blockwise_random_pivoting_gb300.rbrp import Batch, Handle, packed_offsets
from robust_blockwise_random_pivoting_gb300.sketch_ids import cpqr_id, rand_lupp_os

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # The seeded 1000 x 1000 workload with an exponential spectrum, to 1e-6 relative error: a
        # skeleton alone is asked for (column subset selection).  A small call: latency counts.
        dict(name="id64_exp1000", kind="id64", gen="exp", m=1000, n=1000, b=40, tol=1e-12, kmax=0, T=False),
        # The notebook's Gaussian-mixture run: 2000 points in R^500, b = 30, to rank 270, with T.
        dict(name="id64_gmm500x2000", kind="id64", gen="gmm", m=500, n=2000, b=30, tol=0.0, kmax=270, T=True),
        # The reference driver's run: its Gaussian mixture, 64-column blocks, 10 of them, with T.
        dict(name="id64_driver8k", kind="id64", gen="driver", m=8192, n=8192, b=64, tol=0.0, kmax=640, T=True),
        # An ordinary single matrix in FP32: sparse non-negative low rank plus tail, most of its rank.
        dict(name="id32_snn1000", kind="id32", gen="snn", m=1000, n=1200, b=64, tol=1e-12, kmax=900, T=True),
        # The large single matrix: 16384 x 16384, 2000 rank-one terms, at their number.
        dict(name="id32_snn16k", kind="id32", gen="snn", m=16384, n=16384, b=64, tol=1e-12, kmax=2000, T=True),
        # A data set: 65536 points of an imbalanced Gaussian mixture in R^1024, b = 32.
        dict(name="id32_gmm65k", kind="id32", gen="gmm", m=1024, n=65536, b=32, tol=1e-4, kmax=1000, T=True),
        # A few small off-diagonal kernel blocks, as one level of a small hierarchical matrix.
        dict(name="batch_32", kind="batch", host=False, count=32, lo=64, hi=512, b=16, tol=1e-8),
        # 4096 uneven kernel blocks, sides 64 to 2048, in device memory: the largest batch.
        dict(name="batch_4096", kind="batch", host=False, count=4096, lo=64, hi=2048, b=16, tol=1e-8),
        # The same kind of blocks in pinned host memory, read in place.
        dict(name="batch_host_512", kind="batch", host=True, count=512, lo=64, hi=2048, b=16, tol=1e-8),
        # A training step through the fixed-skeleton ID of an 8192 x 8192 Gaussian kernel matrix.
        dict(name="adjoint_8k", kind="adjoint", n=8192, k=4096, b=64),
        # The deterministic comparison ID of the reference's driver, at rank 192.
        dict(name="cpqr_8k", kind="cpqr", m=8192, n=8192, k=192),
        # The sketched comparison ID of the reference's driver on a ragged matrix.
        dict(name="lupp_6000", kind="lupp", m=6001, n=5003, k=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["id64", "id64", "id32", "id32", "batch", "batch", "adjoint", "cpqr", "lupp"])
    if kind == "id64":
        gen = rng.choice(["exp", "gmm", "driver"])
        if gen == "exp":
            return dict(kind=kind, gen=gen, m=_log(rng, 200, 2000), n=_log(rng, 200, 2000), b=rng.choice([7, 16, 32, 40, 64]),
                        tol=10.0 ** -rng.uniform(4, 12), kmax=0, T=False)
        if gen == "gmm":
            m, b = _log(rng, 200, 1500), rng.choice([10, 20, 30, 48])
            return dict(kind=kind, gen=gen, m=m, n=_log(rng, 500, 16000), b=b, tol=0.0, kmax=int(m * rng.uniform(0.2, 0.6)), T=True)
        n = _log(rng, 800, 8192)
        b = rng.choice([32, 64])
        return dict(kind=kind, gen=gen, m=_log(rng, 800, 8192), n=n, b=b, tol=0.0, kmax=min(640, n // 4), T=True)
    if kind == "id32":
        if rng.random() < 0.5:
            m, n = _log(rng, 400, 12000), _log(rng, 400, 12000)
            return dict(kind=kind, gen="snn", m=m, n=n, b=rng.choice([32, 48, 64]), tol=1e-12,
                        kmax=int(min(2000, m, n) * rng.uniform(0.2, 0.95)), T=True)
        m = _log(rng, 100, 1024)
        return dict(kind=kind, gen="gmm", m=m, n=_log(rng, 1000, 65536), b=rng.choice([20, 32, 64]), tol=1e-6,
                    kmax=int(m * rng.uniform(0.2, 0.9)), T=True)
    if kind == "batch":
        lo = _log(rng, 16, 128)
        return dict(kind=kind, host=rng.random() < 0.4, count=_log(rng, 8, 1024), lo=lo, hi=_log(rng, 4 * lo, 2048),
                    b=rng.choice([8, 16, 16, 24, 32]), tol=10.0 ** -rng.uniform(4, 12))
    if kind == "adjoint":
        n = _log(rng, 500, 8000)
        return dict(kind=kind, n=n, k=int(n * rng.uniform(0.1, 0.5)), b=rng.choice([32, 64]))
    if kind == "cpqr":
        return dict(kind=kind, m=_log(rng, 400, 8192), n=_log(rng, 400, 8192), k=_log(rng, 16, 192))
    return dict(kind=kind, m=_log(rng, 1000, 8192), n=_log(rng, 1000, 8192), k=_log(rng, 16, 256))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _colmajor(A, dtype):
    return A.to(dtype).t().contiguous().t()


def _haar(g, n, r):
    q, t = torch.linalg.qr(torch.randn(n, r, generator=g, device=DEV, dtype=F64))
    return q * torch.sign(t.diagonal())


def _matrix(gen, m, n, seed):
    """One FP64 test matrix (columns are the items)."""
    g = _gen(seed)
    if gen == "exp":          # Haar singular vectors, singular values exp(-i / 20)
        r = min(m, n)
        s = torch.exp(-torch.arange(r, device=DEV, dtype=F64) / 20.0)
        return (_haar(g, m, r) * s) @ _haar(g, n, r).t()
    if gen == "snn":          # sparse non-negative: 10/j for the first 100 terms, 1/j up to 2000, density 0.02
        r = min(2000, m, n)
        j = torch.arange(1, r + 1, device=DEV, dtype=F64)
        w = torch.where(j <= 100, 10.0 / j, 1.0 / j)
        X, Y = (torch.where(torch.rand(d, r, generator=g, device=DEV, dtype=F64) < 0.02,
                            torch.rand(d, r, generator=g, device=DEV, dtype=F64), 0.0) for d in (m, n))
        return (X * w) @ Y.t()
    if gen == "gmm":          # 20 imbalanced clusters, weights 2^-c, spreads U[0.1, 1], means N(0, 4 I)
        wts = 2.0 ** -np.arange(20)
        sizes = np.maximum(1, np.round(n * wts / wts.sum())).astype(np.int64)
        sizes[0] = n - sizes[1:].sum()
        label = torch.from_numpy(np.repeat(np.arange(20), sizes)).to(DEV)
        means = 2.0 * torch.randn(m, 20, generator=g, device=DEV, dtype=F64)
        sig = 0.1 + 0.9 * torch.rand(20, generator=g, device=DEV, dtype=F64)
        return means[:, label] + torch.randn(m, n, generator=g, device=DEV, dtype=F64) * sig[label]
    # driver: N(0, 1) entries, 10 (c + 1) added to coordinate c of the points of cluster c
    A = torch.randn(m, n, generator=g, device=DEV, dtype=F64)
    c = torch.arange(n, device=DEV) // -(-n // 100)
    A[c, torch.arange(n, device=DEV)] += 10.0 * (c + 1)
    return A


def _shapes(case):
    """Block shapes, log-uniform; the same for every seed, as a hierarchical matrix's blocks are."""
    r = np.random.default_rng(case["count"] * 7919 + case["hi"])
    return np.round(np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), (case["count"], 2)))).astype(np.int64)


def _blocks(case, seed):
    """Gaussian-kernel blocks between point clusters in unit cubes 2 to 8 apart, each divided by
    its largest entry, packed column major on 16-byte boundaries in one FP32 buffer."""
    g = _gen(seed)
    shapes = _shapes(case)
    offs, _ = packed_offsets(shapes)
    pack = torch.zeros(int(offs[-1]), dtype=torch.float32, device=DEV)
    pts = torch.rand(int(shapes.sum()), 3, generator=g, device=DEV)
    to = torch.randn(case["count"], 3, generator=g, device=DEV)
    to *= (2.0 + 6.0 * torch.rand(case["count"], 1, generator=g, device=DEV)) / to.norm(dim=1, keepdim=True)
    views, at = [], 0
    for q, (m, n) in enumerate(shapes.tolist()):
        d2 = torch.cdist(pts[at + m: at + m + n] + to[q], pts[at: at + m],
                         compute_mode="donot_use_mm_for_euclid_dist").square_()      # n x m: column major m x n
        v = pack[int(offs[q]): int(offs[q]) + m * n].view(n, m)
        torch.exp((d2.min() - d2).mul_(2.0), out=v)                                  # length scale 0.5
        views.append(v.t())
        at += m + n
    return shapes, offs, pack, views


def _kernel_points(case, seed):
    return torch.randn(case["n"], 8, generator=_gen(seed), device=DEV, dtype=F64)


def _kernel(x, ls=1.5):
    return torch.exp(-torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist").square_() / (2.0 * ls * ls))


def _skeleton(K, k, seed):
    """k columns of the kernel matrix by randomly pivoted block Cholesky."""
    g = _gen(seed + 1)
    n = K.shape[0]
    F = torch.zeros(n, k, dtype=F64, device=DEV)
    d = K.diagonal().clone()
    S, i = [], 0
    while i < k:
        s = torch.multinomial(d.clamp_min(0.0), min(64, k - i), generator=g)
        G = K[:, s] - F[:, :i] @ F[s, :i].t()
        H = G[s]
        C = torch.linalg.cholesky(H + 1e-13 * H.diagonal().sum() * torch.eye(len(s), dtype=F64, device=DEV))
        F[:, i: i + len(s)] = torch.linalg.solve_triangular(C, G.t(), upper=False).t()
        d = d - F[:, i: i + len(s)].square().sum(1)
        d[s] = 0.0
        S.append(s)
        i += len(s)
    return torch.cat(S).to(torch.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("id64", "id32"):
        A = _colmajor(_matrix(case["gen"], case["m"], case["n"], seed), F64 if kind == "id64" else torch.float32)
        return dict(case=case, A=A, h=Handle(0))
    if kind == "batch":
        shapes, offs, pack, views = _blocks(case, seed)
        if case["host"]:
            pack = pack.cpu().pin_memory()
            views = [pack[int(offs[q]): int(offs[q]) + m * n].view(n, m).t() for q, (m, n) in enumerate(shapes.tolist())]
        h = Handle(0)
        bt = Batch(h, views, b=case["b"], tol=case["tol"], t_rank_cap=64)
        bt.T_buf.zero_()      # the room behind each problem's own T stays as it is from here on
        return dict(case=case, h=h, pack=pack, bt=bt)
    if kind == "adjoint":
        x = _kernel_points(case, seed)
        K = _kernel(x)
        w = torch.randn(case["n"], generator=_gen(seed + 2), device=DEV)
        return dict(case=case, A=_colmajor(K, torch.float32).requires_grad_(), S=_skeleton(K, case["k"], seed), w=w, h=Handle(0))
    if kind == "cpqr":
        return dict(case=case, A=_colmajor(_matrix("driver", case["m"], case["n"], seed), F64), h=Handle(0))
    return dict(case=case, A=_colmajor(_matrix("driver", case["m"], case["n"], seed), torch.float32), h=Handle(0))


def _trace(x, cap):
    """A per-block trace in an array of the longest one's length."""
    out = np.zeros(cap, x.dtype)
    out[: len(x)] = x[:cap]
    return out


def run(state):
    case, h = state["case"], state["h"]
    kind = case["kind"]
    if kind in ("id64", "id32"):
        r = h.column_id(state["A"], b=case["b"], tol=case["tol"] or None, kmax=case["kmax"] or None, compute_T=case["T"])
        cap = 4 * (case["kmax"] or min(case["m"], case["n"])) // case["b"] + 64
        return dict(perm=r.perm, ranks=_trace(r.ranks, cap), residuals=_trace(r.residuals, cap), T=r.T)
    if kind == "batch":
        bt = state["bt"]
        bt.run()
        r = bt.results()
        return dict(perm=bt.perm_buf, T=bt.T_buf, k=r.k, status=r.status, err_est=r.err_est)
    if kind == "adjoint":
        state["A"].grad = None
        loss = fixed_skeleton_id_loss(state["A"], state["S"], state["w"], case["b"], h)
        loss.backward()
        return dict(loss=loss.detach(), grad=state["A"].grad)
    if kind == "cpqr":
        sk, rd, T = cpqr_id(state["A"], case["k"], handle=h)
    else:
        sk, rd, T = rand_lupp_os(state["A"], case["k"], seed=0, handle=h)
    return dict(sk=sk, rd=rd, T=T)


# --------------------------------------------------------------------------
# what one pass cannot do without
# --------------------------------------------------------------------------
def _rank(case):
    """The rank a run ends at: the cap, or about where the tolerance is met."""
    r = min(case["m"], case["n"])
    if case["kmax"]:
        return min(r, case["kmax"])
    return min(r, int(10.0 * math.log(1.0 / case["tol"]) + 30))     # the exponential spectrum


def work(case):
    kind = case["kind"]
    if kind in ("id64", "id32"):
        m, n, k, e = case["m"], case["n"], _rank(case), 8 if kind == "id64" else 4
        t = 8.0 * k * (n - k) if case["T"] else 0.0
        flops = 2.0 * m * k * (2 * n - k) / 2 * (1 if kind == "id64" else 2) + (k * k * (n - k) if case["T"] else 0)
        return dict(bytes=float(e) * m * n + t + 4.0 * n, flops=float(flops))
    if kind == "batch":
        s = _shapes(case).astype(float)
        k = 12.0 + 1.5 * math.log10(1.0 / case["tol"])
        mn = float((s[:, 0] * s[:, 1]).sum())
        return dict(bytes=4.0 * mn + (8.0 * k + 4.0) * float(s[:, 1].sum()), flops=4.0 * mn * k)
    if kind == "adjoint":
        n, k = float(case["n"]), float(case["k"])
        # factor and T forward, E = B - C T, and E T^T backward
        return dict(bytes=8.0 * n * n, flops=2 * n * k * (2 * n - k) + k * k * (n - k) + 4 * n * k * (n - k))
    m, n, k = float(case["m"]), float(case["n"]), float(case["k"])
    if kind == "cpqr":
        return dict(bytes=8.0 * m * n + 8.0 * k * (n - k), flops=2 * m * n * k + k * k * (n - k))
    return dict(bytes=4.0 * m * n + 8.0 * k * (n - k), flops=4 * k * m * n + n * k * k + 4 * k * n * k)


# --------------------------------------------------------------------------
# the same in plain 64-bit torch and numpy
# --------------------------------------------------------------------------
def _lstsq(A, perm, k):
    perm = torch.as_tensor(perm, device=DEV)
    Q, R = torch.linalg.qr(A[:, perm[:k]])
    return torch.linalg.solve_triangular(R, Q.t() @ A[:, perm[k:]], upper=True)


def _panel(V, tol_loc):
    """Pivoted QR of a panel by orthogonalisation of what is left, each direction twice, and the
    number of pivots that the block filter keeps."""
    V, bs = V.clone(), V.shape[1]
    Q, piv, tail = torch.zeros_like(V), list(range(bs)), []
    for t in range(bs):
        d = V[:, t:].square().sum(0)
        tail.append(float(d.sum()))
        p = t + int(d.argmax())
        V[:, [t, p]] = V[:, [p, t]]
        piv[t], piv[p] = piv[p], piv[t]
        q = V[:, t].clone()
        q -= Q[:, :t] @ (Q[:, :t].t() @ q)
        Q[:, t] = q / q.norm()
        V[:, t + 1:] -= torch.outer(Q[:, t], Q[:, t] @ V[:, t + 1:])
    keep = next((t for t in range(bs) if not tail[t] >= tol_loc * tail[0]), bs)
    return Q[:, :keep], piv[:keep]


def _rbrp(A, b, tol, kmax):
    """Adaptive block random pivoting with numpy's sampler (Philox key 0), in 64 bits."""
    m, n = A.shape
    rng = np.random.Generator(np.random.Philox(key=0))
    perm, d = np.arange(n), A.square().sum(0)
    Q = torch.zeros(m, kmax, dtype=F64, device=DEV)
    res0, i, ranks, res = float(d.sum()), 0, [], []
    while i < kmax:
        w = d[torch.from_numpy(perm[i:]).to(DEV)].cpu().numpy()
        rel = rng.choice(n - i, size=min(kmax - i, b, np.count_nonzero(w)), p=w / w.sum(), replace=False)
        V = A[:, torch.from_numpy(perm[i + rel]).to(DEV)]
        V = V - Q[:, :i] @ (Q[:, :i].t() @ V)
        q, piv = _panel(V, 1.0 / b)
        bs = len(piv)
        at = i + rel[piv]
        cols, own = perm[at].copy(), set(at.tolist())
        free = [p for p in range(i, i + bs) if p not in own]
        perm[at[(at < i) | (at >= i + bs)]] = perm[free]
        perm[i: i + bs] = cols
        Q[:, i: i + bs] = q
        d = (d - (q.t() @ A).square().sum(0)).clamp_min(0.0)
        i += bs
        left = float(d[torch.from_numpy(perm[i:]).to(DEV)].sum())
        ranks.append(i)
        res.append(left / res0)
        if tol and left < res0 * tol:
            break
    return perm, i, np.array(ranks), np.array(res)


def _cpqr(A, k):
    """Skeleton and remaining columns of the column-pivoted QR, by rank-one updates of the residual."""
    R = A.clone()
    perm = torch.arange(A.shape[1], device=DEV)
    for t in range(k):
        d = R.square().sum(0)[perm[t:]]
        p = t + int(d.argmax())
        perm[[t, p]] = perm[[p, t]]
        q = R[:, perm[t]] / R[:, perm[t]].norm()
        R -= torch.outer(q, q @ R)
    return perm


def exact(case, seed):
    kind = case["kind"]
    if kind == "id64":
        A = _matrix(case["gen"], case["m"], case["n"], seed)
        kmax = case["kmax"] or min(case["m"], case["n"])
        perm, k, _, res = _rbrp(A, case["b"], case["tol"], kmax)
        cap = 4 * kmax // case["b"] + 64
        return dict(perm=None, ranks=None, residuals=_trace(res, cap), T=_lstsq(A, perm, k) if case["T"] else None)
    if kind == "cpqr":
        A = _matrix("driver", case["m"], case["n"], seed)
        return dict(sk=None, rd=None, T=_lstsq(A, _cpqr(A, case["k"]), case["k"]))
    if kind == "adjoint":
        K = _kernel(_kernel_points(case, seed))
        S = _skeleton(K, case["k"], seed).long()
        A = K.to(torch.float32).to(F64)
        w = torch.randn(case["n"], generator=_gen(seed + 2), device=DEV).to(F64)
        rest = torch.ones(case["n"], dtype=torch.bool, device=DEV)
        rest[S] = False
        C, B, w = A[:, S], A[:, rest], w[rest]
        Q, R = torch.linalg.qr(C)
        T = torch.linalg.solve_triangular(R, Q.t() @ B, upper=True)
        E, u = B - C @ T, T @ w
        z = torch.linalg.solve_triangular(R.t(), u[:, None], upper=False)
        z = torch.linalg.solve_triangular(R, z, upper=True)[:, 0]
        Cz, G = C @ z, torch.empty_like(A)
        G[:, rest] = 2 * E + 2 * torch.outer(Cz, w)
        G[:, S] = -2 * E @ T.t() - 2 * torch.outer(Cz, u) + 2 * torch.outer(E @ w, z)
        return dict(loss=E.square().sum() + u.square().sum(), grad=G)
    # id32 and batch: which column is drawn last depends on the 32-bit residual; lupp: on the sketch
    return None
