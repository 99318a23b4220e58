"""Performance cases of the package: the work its users have it do, through
its public entry points.

A barrier or maximum-likelihood program factors a chordal matrix and takes
the projected inverse of the factor (value and gradient of log det), applies
the Hessian of the barrier, completes partial matrices, and solves with the
factor; a batched program does the first of these for many matrices, or many
value sets of one pattern, at once.  The patterns are the seeded grids of
`chompack_b200.grids` (2-D 5-point, 3-D 7-point, and 2-D with random extra
neighbours), ordered by AMD, with and without the merging of supernodes, at
the sizes of the benchmark and the tests and the odd sizes between them.

Every case keeps what such a program keeps: the symbolic factorisation (and
with it the compiled plan and workspace), which depends on the pattern only.
New values arrive with every seed.
"""
import functools
import math

import numpy as np
import torch

import chompack_b200 as cp
from chompack_b200 import autograd, grids, mixed


def listed():
    return [
        # value and gradient of log det on the smallest grid of the tests: a
        # call's latency counts (an outer loop over many small matrices)
        {"name": "step_grid2d_30", "kind": "step", "pattern": "grid2d", "side": 30, "merge": 16},
        # one matrix of the batched workload alone, unmerged, many small fronts
        {"name": "step_extra_97", "kind": "step", "pattern": "extra", "side": 97, "merge": 0},
        # the benchmark's headline: a 3-D problem with large separators
        {"name": "step_grid3d_40", "kind": "step", "pattern": "grid3d", "side": 40, "merge": 32},
        # the largest order (n = 10^6): a wide tree of moderate fronts
        {"name": "step_grid2d_1000", "kind": "step", "pattern": "grid2d", "side": 1000, "merge": 64},
        # the benchmark's batch of uneven grids, one launch per sweep
        {"name": "batch_extra_256", "kind": "batch", "pattern": "extra", "side": 120, "merge": 0, "count": 256},
        # training on log det: forward and backward of 16 value sets
        {"name": "autograd_grid3d_32x16", "kind": "autograd", "pattern": "grid3d", "side": 32, "merge": 32,
         "count": 16},
        # maximum-determinant completion, both forms of its updates (the
        # factored one is the default)
        {"name": "completion_grid3d_40", "kind": "completion", "pattern": "grid3d", "side": 40, "merge": 32,
         "factored": True},
        {"name": "completion_plain_grid3d_40", "kind": "completion", "pattern": "grid3d", "side": 40, "merge": 32,
         "factored": False},
        # the barrier's Hessian applied to one direction (default options but
        # adj=None, the whole operator), as the autograd tests use it
        {"name": "hessian_grid3d_32", "kind": "hessian", "pattern": "grid3d", "side": 32, "merge": 32,
         "factored": True},
        # solves with a factor in hand, 8 right-hand sides, both triangles
        {"name": "solve_grid3d_40", "kind": "solve", "pattern": "grid3d", "side": 40, "merge": 32, "nrhs": 8},
        # the product L L^T and a trace inner product
        {"name": "llt_grid3d_40", "kind": "llt", "pattern": "grid3d", "side": 40, "merge": 32},
        # factor in TF32, solve refined to FP64 accuracy
        {"name": "mixed_grid3d_48", "kind": "mixed", "pattern": "grid3d", "side": 48, "merge": 64, "nrhs": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "autograd", "completion", "hessian", "solve", "llt",
                       "mixed"])
    if kind == "batch":
        return {"kind": kind, "pattern": "extra", "side": rng.randint(40, 120), "merge": rng.choice([0, 0, 16]),
                "count": _log_int(rng, 4, 128)}
    pattern = rng.choice(["grid2d", "grid3d", "grid3d", "extra"])
    top = {"step": (700, 44, 119), "autograd": (160, 28, 80), "completion": (500, 38, 119),
           "hessian": (300, 31, 100), "solve": (600, 44, 119), "llt": (600, 42, 119), "mixed": (600, 46, 119)}[kind]
    if pattern == "grid2d":
        side = _log_int(rng, 20, top[0])
    elif pattern == "grid3d":
        side = rng.randint(8, top[1])
    else:
        side = rng.randint(20, top[2])
    case = {"kind": kind, "pattern": pattern, "side": side, "merge": rng.choice([0, 16, 32, 32, 64])}
    if kind == "autograd":
        case["count"] = _log_int(rng, 1, 16)
    if kind in ("completion", "hessian"):
        case["factored"] = rng.random() < 0.6
    if kind in ("solve", "mixed"):
        case["nrhs"] = rng.choice([1, 1, 3, 8, 17, 40])
    return case


# --------------------------------------------------------------- patterns
class _Pattern(object):
    """A symbolic factorisation and where the entries of a matrix on its
    pattern go: id[k] is the entry (of the lower triangle in A's order) that
    lies at position pos[k] of the block values."""

    def __init__(self, A, merge):
        self.n = A.size[0]
        self.I, self.J = np.asarray(A._I), np.asarray(A._J)
        self.off = np.flatnonzero(self.I != self.J)
        self.dia = np.flatnonzero(self.I == self.J)
        self.symb = cp.symbolic(A, p=cp.amd.order(A),
                                merge_function=cp.merge_size_fill(merge, merge) if merge else None)
        tags = cp.spmatrix(np.arange(1.0, self.I.size + 1.0), self.I, self.J, A.size)
        host = (cp.cspmatrix(self.symb, device="cpu") + tags).blkval
        self.pos = torch.nonzero(host).reshape(-1)
        self.id = host[self.pos].to(torch.int64) - 1
        self.size = int(self.symb.blkptr[-1])

    def entries(self, rng):
        """Random entries by the recipe of `grids`: N(0, 1) below the
        diagonal, and a diagonal that dominates its row by 1."""
        V = np.empty(self.I.size)
        v = rng.standard_normal(self.off.size)
        V[self.off] = v
        a, i, j = np.abs(v), self.I[self.off], self.J[self.off]
        d = np.bincount(i, a, self.n) + np.bincount(j, a, self.n) + 1.0
        V[self.dia] = d[self.I[self.dia]]
        return V

    def place(self, V, out):
        """V's entries at their places in the values `out` (zeros before)."""
        out[self.pos.to(out.device)] = torch.from_numpy(V).to(out.device)[self.id.to(out.device)]
        return out


def _grid(pattern, side, seed=3):
    if pattern == "grid2d":
        return grids.grid2d(side)
    if pattern == "grid3d":
        return grids.grid3d(side)
    return grids.grid2d_extra(side, seed=seed)


@functools.lru_cache(maxsize=2)
def _pattern(pattern, side, merge):
    return _Pattern(_grid(pattern, side), merge)


@functools.lru_cache(maxsize=1)
def _batch(side, merge, count):
    """count uneven grids with sides from 20 to `side`, and their batch."""
    ps = [_Pattern(grids.grid2d_extra(sd, seed=s), merge) for sd, s in grids.uneven_batch_specs(count, hi=side)]
    return ps, cp.batch([p.symb for p in ps])


def _values(P, rng):
    return P.place(P.entries(rng), torch.zeros(P.size, dtype=torch.float64, device="cuda"))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = dict(case)
    kind = case["kind"]
    if kind == "batch":
        ps, s["batch"] = _batch(case["side"], case["merge"], case["count"])
        host = torch.zeros(s["batch"].size, dtype=torch.float64)
        at = 0
        for P in ps:
            P.place(P.entries(rng), host[at:at + P.size])
            at += P.size
        s["x"] = host.to("cuda")
        return s
    P = _pattern(case["pattern"], case["side"], case["merge"])
    s["symb"] = P.symb
    if kind == "autograd":
        x = torch.stack([_values(P, rng) for _ in range(case["count"])])
        s["x"] = (x[0] if case["count"] == 1 else x).requires_grad_()
        return s
    X = cp.cspmatrix(P.symb, blkval=_values(P, rng))
    s["X"] = X
    if kind in ("completion", "hessian", "solve", "llt"):
        L = X.copy()
        cp.cholesky(L)
        s["L"] = L
    if kind in ("completion", "hessian", "llt"):
        Y = s["L"].copy()
        cp.projected_inverse(Y)
        s["Y"] = Y
    if kind == "hessian":
        V = P.entries(rng)
        V[P.dia] = rng.standard_normal(P.dia.size)
        s["U"] = cp.cspmatrix(P.symb, blkval=P.place(V, torch.zeros(P.size, dtype=torch.float64, device="cuda")))
    if kind in ("solve", "mixed"):
        # column-major, as the solves take it
        s["B"] = torch.from_numpy(rng.standard_normal((case["nrhs"], P.n))).to("cuda").t()
    return s


def run(s):
    kind = s["kind"]
    if kind == "step":
        L = s["X"].copy()
        cp.cholesky(L)
        Y = L.copy()
        cp.projected_inverse(Y)
        return {"L": L.blkval, "Y": Y.blkval}
    if kind == "batch":
        B = s["batch"]
        v = s["x"].clone()
        B.cholesky(v)
        f = B.logdet(v)
        B.projected_inverse(v)
        return {"f": f, "Y": v}
    if kind == "autograd":
        f = autograd.logdet_values(s["x"], s["symb"])
        g, = torch.autograd.grad(f.sum(), s["x"])
        return {"f": f.detach(), "g": g}
    if kind == "completion":
        L = s["Y"].copy()
        cp.completion(L, factored_updates=s["factored"])
        return {"L": L.blkval}
    if kind == "hessian":
        U = s["U"].copy()
        cp.hessian(s["L"], s["Y"], U, adj=None, factored_updates=s["factored"])
        return {"U": U.blkval}
    if kind == "solve":
        B = s["B"].clone()
        cp.trsm(s["L"], B, trans="N")
        Z = B.clone()
        cp.trsm(s["L"], B, trans="T")
        return {"Z": Z, "X": B}
    if kind == "llt":
        X = s["L"].copy()
        cp.llt(X)
        return {"X": X.blkval, "d": cp.dot(X, s["Y"])}
    L = s["X"].copy()
    cp.cholesky(L, precision="tf32")
    x, _ = mixed.solve(s["X"], L, s["B"])
    return {"x": x}


# ------------------------------------------------------------- least work
def _flops(symb):
    """Floating-point operations of each sweep, summed over the supernodes
    (nn columns, na rows below them)."""
    nn = np.diff(np.asarray(symb.snptr)).astype(np.float64)
    na = np.diff(np.asarray(symb.relptr)).astype(np.float64)
    nj = nn + na
    chol = nn ** 3 / 3 + 2 * nn ** 2 * na + nn * na ** 2
    pinv = 4 * nn ** 3 / 3 + 2 * na ** 2 * nn + 2 * nn ** 2 * na
    llt = na * nn ** 2 + nn * nj ** 2
    comp = na ** 3 / 3 + 2 * na ** 2 * nn + nn ** 2 * na + 2 * nn ** 3 / 3
    hess = 2 * (4 * na ** 2 * nn + 2 * na * nn ** 2 + nj * nn ** 2 + nn ** 3 + na ** 2 * nn)
    rhs = 2 * (nn ** 2 + 2 * na * nn)
    return {k: float(v.sum()) for k, v in
            dict(chol=chol, pinv=pinv, llt=llt, comp=comp, hess=hess, rhs=rhs).items()}


def work(case):
    """Bytes: the values of the inputs read and of the outputs written once
    each; flops: the sweeps' own formulas."""
    kind = case["kind"]
    if kind == "batch":
        ps, _ = _batch(case["side"], case["merge"], case["count"])
        fl = [_flops(P.symb) for P in ps]
        return {"bytes": 16.0 * sum(P.size for P in ps), "flops": sum(f["chol"] + f["pinv"] for f in fl)}
    P = _pattern(case["pattern"], case["side"], case["merge"])
    f, v, n = _flops(P.symb), 8.0 * P.size, 8.0 * P.n * case.get("nrhs", 0)
    c = case.get("count", 1)
    return {"step": {"bytes": 3 * v, "flops": f["chol"] + f["pinv"]},
            "autograd": {"bytes": 2 * c * v, "flops": c * (f["chol"] + f["pinv"])},
            "completion": {"bytes": 2 * v, "flops": f["comp"]},
            "hessian": {"bytes": 4 * v, "flops": f["hess"]},
            "solve": {"bytes": v + 3 * n, "flops": 2 * f["rhs"] * case.get("nrhs", 0)},
            "llt": {"bytes": 3 * v, "flops": f["llt"]},
            "mixed": {"bytes": v + 2 * n, "flops": f["chol"] + 2 * f["rhs"] * case.get("nrhs", 0)}}[kind]


# ---------------------------------------------------------- 64-bit results
DENSE_MAX = 33000  # order up to which the dense result takes a few seconds


def _dense(P, V):
    """The symmetric matrix of entries V, rows and columns in the order of
    the factorisation."""
    ip = torch.as_tensor(np.argsort(np.asarray(P.symb.p)), device="cuda")
    I, J = (ip[torch.from_numpy(np.asarray(a)).cuda()] for a in (P.I, P.J))
    A = torch.zeros(P.n, P.n, dtype=torch.float64, device="cuda")
    v = torch.from_numpy(V).cuda()
    A[I, J] = v
    A[J, I] = v
    return A


def _blocks(P, M, conventional=False):
    """The lower trapezoids of M's supernode blocks in the layout of the
    block values; for a factor (conventional=True: M is one) the
    rows below a diagonal block are multiplied by its inverse."""
    s = P.symb
    sp, cpt, rows, bp = (np.asarray(a) for a in (s.snptr, s.sncolptr, s.snrowidx, s.blkptr))
    nn, nj = np.diff(sp), np.diff(cpt)
    col = np.repeat(np.arange(P.n), np.repeat(nj, nn))
    start = np.repeat(bp[:-1], nn * nj)
    r = (np.arange(P.size) - start) % np.repeat(nj, nn * nj)
    row = rows[np.repeat(cpt[:-1], nn * nj) + r]
    out = M[torch.from_numpy(row).cuda(), torch.from_numpy(col).cuda()]
    out[torch.from_numpy(np.flatnonzero(row < col)).cuda()] = 0.0
    if conventional:
        for k in range(s.Nsn):
            b = out[int(bp[k]):int(bp[k + 1])].view(int(nn[k]), int(nj[k])).t()
            if nj[k] > nn[k]:
                b[int(nn[k]):] = torch.linalg.solve_triangular(b[:int(nn[k])].clone(), b[int(nn[k]):].clone(),
                                                               upper=False, left=False)
    return out


def _conjugate_gradients(P, V, B):
    """A^{-1} B in 64 bits by conjugate gradients with a diagonal
    preconditioner on the sparse matrix, restarted once on the residual."""
    I, J = np.concatenate([P.I, P.J[P.off]]), np.concatenate([P.J, P.I[P.off]])
    A = torch.sparse_coo_tensor(np.stack([I, J]), np.concatenate([V, V[P.off]]), (P.n, P.n)).coalesce()
    A = A.to_sparse_csr().cuda()
    d = torch.empty(P.n, dtype=torch.float64)
    d[torch.from_numpy(np.array(P.I[P.dia]))] = torch.from_numpy(V[P.dia])
    w = (1.0 / d.cuda())[:, None]
    x = torch.zeros_like(B).contiguous()
    for _ in range(3):
        r = B - A @ x
        top = r.norm(dim=0)
        z = w * r
        p, rz, dx = z.clone(), (r * z).sum(0), torch.zeros_like(x)
        for it in range(3000):
            q = A @ p
            a = rz / (p * q).sum(0).clamp_min(1e-300)
            dx += a * p
            r -= a * q
            if it % 20 == 0 and float((r.norm(dim=0) / top.clamp_min(1e-300)).max()) < 1e-13:
                break
            z = w * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        x += dx
    return x


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "batch":
        if case["count"] * case["side"] ** 6 > 2e14:  # too long for one dense inverse a matrix
            return None
        ps, _ = _batch(case["side"], case["merge"], case["count"])
        f, Y = [], []
        for P in ps:
            L = torch.linalg.cholesky(_dense(P, P.entries(rng)))
            f.append(2.0 * L.diagonal().log().sum())
            Y.append(_blocks(P, torch.cholesky_inverse(L)))
        return {"f": torch.stack(f), "Y": torch.cat(Y)}
    P = _pattern(case["pattern"], case["side"], case["merge"])
    if kind == "autograd":
        if P.n > DENSE_MAX or case["count"] * float(P.n) ** 3 > 4e13:
            return None
        f, g = [], []
        for _ in range(case["count"]):
            L = torch.linalg.cholesky(_dense(P, P.entries(rng)))
            f.append(2.0 * L.diagonal().log().sum())
            Z = torch.cholesky_inverse(L)
            D = Z.diagonal().clone()
            Z *= 2.0
            Z.diagonal().copy_(D)
            g.append(_blocks(P, Z))
        if case["count"] == 1:
            return {"f": f[0], "g": g[0]}
        return {"f": torch.stack(f), "g": torch.stack(g)}
    V = P.entries(rng)
    if kind == "mixed":
        B = torch.from_numpy(rng.standard_normal((case["nrhs"], P.n))).cuda().t()
        return {"x": _conjugate_gradients(P, V, B)}
    if kind == "llt":
        # L L^T is the matrix again; <A, P(A^{-1})> is the trace of the identity
        X = torch.zeros(P.size, dtype=torch.float64, device="cuda")
        return {"X": P.place(V, X), "d": float(P.n)}
    if kind == "solve":
        B = torch.from_numpy(rng.standard_normal((case["nrhs"], P.n))).cuda().t()
        if P.n > DENSE_MAX:
            return {"Z": None, "X": _conjugate_gradients(P, V, B)}
        p = torch.as_tensor(np.asarray(P.symb.p), device="cuda")
        L = torch.linalg.cholesky(_dense(P, V))
        z = torch.linalg.solve_triangular(L, B[p], upper=False)
        x = torch.linalg.solve_triangular(L.t(), z, upper=True)
        Z, X = torch.empty_like(z), torch.empty_like(x)
        Z[p], X[p] = z, x
        return {"Z": Z, "X": X}
    if P.n > DENSE_MAX:
        return None
    L = torch.linalg.cholesky(_dense(P, V))
    if kind == "completion":
        return {"L": _blocks(P, L, conventional=True)}
    if kind == "step":
        return {"L": _blocks(P, L, conventional=True), "Y": _blocks(P, torch.cholesky_inverse(L))}
    V2 = P.entries(rng)
    V2[P.dia] = rng.standard_normal(P.dia.size)
    return {"U": _blocks(P, torch.cholesky_solve(torch.cholesky_solve(_dense(P, V2), L).t().contiguous(), L))}
