"""The work that programs have this library do, as measurable cases.

A case is one call (or one batch of calls) through the public C entry points, as the Python binding
exposes them.  ``listed()`` gives the named ones, ``draw(rng)`` more of the same ranges; ``prepare``
makes what a program holds before the call, ``run`` makes one pass, ``work`` counts the bytes and
operations a pass cannot do without, and ``exact`` restates the results in 64 bits.

Kinds (a case's ``"kind"``):

  solve    one isvd_?Isvd_ex solve (x: "s" / "d"; mixed: the precision mode; host: A and the results
           in pageable host memory, as a C program that malloc'ed them holds them, else in GPU memory;
           order: row- or column-major A; algs: the stage selectors)
  stages   a program that keeps A and calls the sketch and the tall-skinny QR stages itself
  batch    many uneven matrices through isvd_sBatchIsvd
  adjoint  isvd_sSvdAdjoint of a truncated SVD (the backward pass of a differentiated solve)

Singular vectors are defined up to a sign per pair; every pass ends as programs that keep, average or
compare factors end it: the pairs are turned so that each column of U has a non-negative sum.

Matrices are a factor model: A = X diag(d) Y' + noise, with Gaussian X and Y of l strong factors (d
falling from 1 to 0.3) and 3 l weak ones (0.1 to 1e-3), and noise of spectral norm 0.02.
"""
import ctypes
import math
import weakref

import numpy as np
import torch

import isvd_b200
from isvd_b200.capi import c_int_t, ptr

DEV = "cuda:0"
F64 = torch.float64


def listed():
    solve = dict(kind="solve", algs="GP/GR/KN/GR", mixed=False, host=False, order="R")
    return [
        # the reference demo's use: a matrix read from a file, a few vectors, host arrays, FP64 (the
        # sizes of the reference's own data files)
        dict(solve, name="d_host_101x1001", x="d", m=101, n=1001, k=10, p=1, N=12, host=True),
        # the plain FP64 workload of the benchmark configurations
        dict(solve, name="d_2000x1000", x="d", m=2000, n=1000, k=20, p=12, N=16),
        # a large FP64 solve
        dict(solve, name="d_40000x6000", x="d", m=40000, n=6000, k=64, p=32, N=16),
        # an ordinary FP32 data matrix of odd sizes, column-major as Fortran, R and MATLAB programs hold it
        dict(solve, name="s_30011x2003_col", x="s", m=30011, n=2003, k=50, p=15, N=16, order="C"),
        # a large FP32 solve in the default precision
        dict(solve, name="s_100000x10000", x="s", m=100000, n=10000, k=100, p=28, N=16),
        # the headline workload: MIXED, 200000 x 20000, k = 100, p = 28, N = 32, A on the GPU
        dict(solve, name="mixed_200000x20000", x="s", m=200000, n=20000, k=100, p=28, N=32, mixed=True),
        # the forward pass of the differentiated workload
        dict(solve, name="mixed_16384x4096", x="s", m=16384, n=4096, k=64, p=32, N=16, mixed=True),
        # FP32 data in host memory, results wanted in host memory, MIXED
        dict(solve, name="mixed_host_12007x3001", x="s", m=12007, n=3001, k=40, p=24, N=16, mixed=True, host=True),
        # a symmetric matrix (a kernel or covariance matrix): hierarchical reduction and symmetric
        # postprocessing, eigenpairs wanted
        dict(solve, name="s_sym_5003_hr_sy", x="s", m=5003, n=5003, k=32, p=16, N=8, algs="GP/TS/HR/SY"),
        # a program with its own pipeline: sketch and orthonormal bases of the N sketches, FP64
        dict(kind="stages", name="d_stages_20011x1501", x="d", m=20011, n=1501, k=30, p=18, N=8, mixed=False,
             order="R"),
        # 64 uneven matrices in one batch (the sizes of the batched workload, N = 8)
        dict(kind="batch", name="batch_64_uneven", count=64, mlo=512, mhi=8192, nlo=256, nhi=4096, N=8, noise=1e-4),
        # the backward pass of the differentiated workload, MIXED
        dict(kind="adjoint", name="adjoint_16384x4096", m=16384, n=4096, k=64, r=512, mixed=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["d", "d", "s", "s", "mixed", "mixed", "sym", "stages", "batch", "adjoint"])
    base = dict(kind="solve", algs="GP/GR/KN/GR", mixed=False, host=False, order="R")
    if kind == "d":  # between the demo's size and the large FP64 solve
        l = _log(rng, 11, 96)
        p = max(1, l // 3)
        return dict(base, x="d", m=_log(rng, 6 * l, 40000), n=_log(rng, 6 * l, 6000), k=l - p, p=p,
                    N=rng.choice([8, 12, 16]), host=rng.random() < 0.25, order=rng.choice("RC"))
    if kind == "s":
        l = _log(rng, 24, 128)
        p = max(1, l // 4)
        return dict(base, x="s", m=_log(rng, 2000, 100000), n=_log(rng, 8 * l, 10000), k=l - p, p=p,
                    N=rng.choice([8, 12, 16]), host=rng.random() < 0.25, order=rng.choice("RC"))
    if kind == "mixed":
        l = rng.choice([32, 48, 64, 96, 128])
        p = max(1, l // 4)
        return dict(base, x="s", m=_log(rng, 4000, 120000), n=_log(rng, 8 * l, 16000), k=l - p, p=p,
                    N=rng.choice([8, 16, 32]), mixed=True, host=rng.random() < 0.25, order=rng.choice("RC"))
    if kind == "sym":
        l = rng.choice([20, 32, 48, 64])
        m = _log(rng, 1000, 8000)
        return dict(base, x=rng.choice("sd"), m=m, n=m, k=l - l // 4, p=l // 4, N=rng.choice([4, 8]),
                    algs=rng.choice(["GP/TS/HR/SY", "GP/GR/HR/SY", "GP/TS/KN/SY"]), order=rng.choice("RC"))
    if kind == "stages":
        l = _log(rng, 16, 96)
        return dict(kind="stages", x=rng.choice("sd"), m=_log(rng, 8 * l, 40000), n=_log(rng, 8 * l, 5000),
                    k=l - l // 4, p=l // 4, N=rng.choice([4, 8, 16]), mixed=False, order=rng.choice("RC"))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(12, 64), mlo=rng.choice([300, 512, 1000]), mhi=rng.choice([2000, 8192]),
                    nlo=256, nhi=rng.choice([1000, 4096]), N=8, noise=1e-4)
    k = rng.choice([16, 32, 48, 64])
    return dict(kind="adjoint", m=_log(rng, 2000, 16384), n=_log(rng, 1000, 4096), k=k, r=4 * k,
                mixed=rng.random() < 0.7)


# ---------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _dtype(x):
    return torch.float32 if x == "s" else F64


def _strengths(l, r):
    d = np.concatenate([np.linspace(1.0, 0.3, l), np.geomspace(0.1, 1e-3, max(r - l, 0))])[:r]
    return torch.as_tensor(d, device=DEV, dtype=F64)


def _matrix(case, seed):
    """The m x n factor-model matrix, as stored: m x n row-major, or n x m (the columns) for order 'C'."""
    g = _gen(seed)
    m, n, l = case["m"], case["n"], case["k"] + case["p"]
    dt = _dtype(case["x"])
    r = min(4 * l, n, m)
    noise = 0.02 / (math.sqrt(m) + math.sqrt(n))
    d = _strengths(l, r).to(dt)
    x = torch.randn(m, r, device=DEV, dtype=dt, generator=g).mul_(1.0 / math.sqrt(m))
    if case.get("algs", "").endswith("SY"):
        a = torch.randn(m, m, device=DEV, dtype=dt, generator=g).mul_(noise * 0.5)
        a = a + a.t()
        return a.addmm_(x * d, x.t())
    y = torch.randn(n, r, device=DEV, dtype=dt, generator=g).mul_(1.0 / math.sqrt(n))
    if case["order"] == "R":
        return torch.randn(m, n, device=DEV, dtype=dt, generator=g).mul_(noise).addmm_(x * d, y.t())
    return torch.randn(n, m, device=DEV, dtype=dt, generator=g).mul_(noise).addmm_(y, (x * d).t())


def _as_mn(case, a):
    return a if case["order"] == "R" else a.t()


class _Batch:
    """A batch handle and what it solves, as a program that solves the same shapes again keeps them."""

    def __init__(self, lib, mats, N):
        vp = ctypes.c_void_p
        self.lib, self.mats = lib, mats
        count = len(mats)
        arr = lambda vals, ct=c_int_t: (ct * len(vals))(*vals)  # noqa: E731
        create = lib.lib.isvd_sBatchCreate
        create.argtypes, create.restype = [c_int_t, vp, vp, vp, vp, c_int_t], vp
        self.solve = lib.lib.isvd_sBatchIsvd
        self.solve.argtypes, self.solve.restype = [vp] * 10 + [c_int_t, vp, vp], ctypes.c_int
        self.handle = create(count, arr([d["m"] for d in mats]), arr([d["n"] for d in mats]),
                             arr([d["k"] for d in mats]), arr([d["p"] for d in mats]), N)
        if not self.handle:
            raise RuntimeError("isvd_sBatchCreate: %s" % (lib.last_error(),))
        destroy = lib.lib.isvd_gpu_batch_destroy
        destroy.argtypes = [vp]
        weakref.finalize(self, destroy, self.handle)
        p = lambda key: arr([d[key].data_ptr() for d in mats], vp)  # noqa: E731
        # the results of all matrices as row blocks of one U and one V
        self.lmax = max(d["k"] + d["p"] for d in mats)
        rows = lambda key: torch.cat([torch.full((d[key],), i, device=DEV) for i, d in enumerate(mats)])  # noqa: E731
        self.useg, self.vseg = rows("m"), rows("n")
        self.u, self.v = (torch.zeros(len(seg), self.lmax, device=DEV) for seg in (self.useg, self.vseg))
        self.kept = torch.zeros(count, self.lmax, device=DEV)
        um = vm = 0
        for i, d in enumerate(mats):
            d["ut"], d["vt"] = self.u[um:], self.v[vm:]
            um, vm = um + d["m"], vm + d["n"]
            self.kept[i, :d["k"]] = 1.0
        torch.cuda.synchronize()
        ls = arr([self.lmax] * count)
        self.argv = np.asarray([256, 1e-4], dtype=np.float32)
        self.its = arr([0] * count)
        self.args = (self.handle, p("a"), arr([d["n"] for d in mats]), p("s"), p("ut"), ls, p("vt"), ls,
                     arr([11 + i for i in range(count)]), self.argv.ctypes.data, 2, self.its, None)

    def __call__(self):
        if self.solve(*self.args):
            raise RuntimeError("isvd_sBatchIsvd: %s" % (self.lib.last_error(),))
        total = torch.zeros(len(self.mats), self.lmax, device=DEV).index_add_(0, self.useg, self.u)
        turn = torch.where(total < 0, -self.kept, self.kept)  # the k kept columns of each matrix, the others 0
        return {"u": self.u * turn[self.useg], "v": self.v * turn[self.vseg]}


def _batch_shapes(case, seed):
    rng = np.random.default_rng(1000 + case["count"])  # the shapes are the case's; the values the seed's
    out = []
    for _ in range(case["count"]):
        m = int(np.exp(rng.uniform(np.log(case["mlo"]), np.log(case["mhi"]))))
        n = int(np.exp(rng.uniform(np.log(case["nlo"]), np.log(min(m, case["nhi"]) + 1))))
        k = int(rng.choice([8, 16, 32, 64]))
        out.append((m, n, k, k // 2))
    return out


def prepare(case, seed):
    lib = isvd_b200.load()
    st = dict(case=case, lib=lib, seed=int(seed) % 100000)
    if case["kind"] == "batch":
        mats = []
        for i, (m, n, k, p) in enumerate(_batch_shapes(case, seed)):
            c = dict(x="s", m=m, n=n, k=k, p=p, order="R")
            mats.append(dict(m=m, n=n, k=k, p=p, a=_matrix(c, seed * 1000 + i), s=torch.zeros(k + p, device=DEV)))
        st["batch"] = _Batch(lib, mats, case["N"])
        return st
    if case["kind"] == "adjoint":
        g = _gen(seed)
        m, n, k, r = case["m"], case["n"], case["k"], min(case["r"], case["n"], case["m"])
        u = torch.linalg.qr(torch.randn(m, r, device=DEV, dtype=F64, generator=g))[0]
        v = torch.linalg.qr(torch.randn(n, r, device=DEV, dtype=F64, generator=g))[0]
        sig = torch.logspace(0, -2, r, device=DEV, dtype=F64)
        f = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
        u0 = u[:, :k]
        xx = torch.randn(m, 32, device=DEV, dtype=F64, generator=g)
        st.update(a=f((u * sig) @ v.t()), s=f(sig[:k]), u=f(u0), v=f(v[:, :k]),
                  ds=torch.randn(k, device=DEV, generator=g), du=f(2.0 * xx @ (xx.t() @ u0)),
                  dv=torch.randn(n, k, device=DEV, generator=g))
        st["da"] = torch.zeros_like(st["a"])
        return st
    m, n, k, p, N = (case[q] for q in ("m", "n", "k", "p", "N"))
    l, dt = k + p, _dtype(case["x"])
    a = _matrix(case, seed)
    st["prm"] = lib.create_param(m, n, k, p, N)
    if case["kind"] == "stages":
        st["a"], st["yst"] = a, torch.zeros(m, N * l, device=DEV, dtype=dt)
        return st
    if case["host"]:
        npdt = np.float32 if case["x"] == "s" else np.float64
        st["a"] = a.cpu().numpy()
        st["s"], st["ut"], st["vt"] = np.zeros(l, npdt), np.zeros((m, l), npdt), np.zeros((n, l), npdt)
    else:
        st["a"] = a
        st["s"] = torch.zeros(l, device=DEV, dtype=dt)
        st["ut"], st["vt"] = torch.zeros(m, l, device=DEV, dtype=dt), torch.zeros(n, l, device=DEV, dtype=dt)
    return st


# ------------------------------------------------------------------------------------ pass
def _lda(case):
    return case["n"] if case["order"] == "R" else case["m"]


def _turned(u, v):
    """u and v with the pairs turned so that each column of u has a non-negative sum."""
    neg = u.sum(0) < 0
    turn = np.where(neg, -1, 1).astype(u.dtype) if isinstance(u, np.ndarray) else torch.where(neg, -1.0, 1.0).to(u.dtype)
    return u * turn, None if v is None else v * turn


def _run_adjoint(st):
    case, lib = st["case"], st["lib"]
    m, n, k = case["m"], case["n"], case["k"]
    vp = ctypes.c_void_p
    fn = lib.lib.isvd_sSvdAdjoint
    fn.argtypes = [c_int_t, c_int_t, c_int_t, ctypes.c_char, vp, c_int_t, vp, vp, c_int_t, vp, c_int_t, vp, vp,
                   c_int_t, vp, c_int_t, vp, c_int_t, ctypes.c_int, ctypes.c_double, ctypes.POINTER(ctypes.c_int)]
    fn.restype = ctypes.c_int
    lib.lib.isvd_gpu_set_precision(1 if case["mixed"] else 0)
    try:
        status = fn(m, n, k, b"R", ptr(st["a"]), n, ptr(st["s"]), ptr(st["u"]), k, ptr(st["v"]), k, ptr(st["ds"]),
                    ptr(st["du"]), k, ptr(st["dv"]), k, ptr(st["da"]), n, 400, 1e-7, None)
    finally:
        lib.lib.isvd_gpu_set_precision(0)
    if status:
        raise RuntimeError("isvd_sSvdAdjoint: %s" % (lib.last_error(),))
    return {"da": st["da"]}


def run(state):
    case, lib = state["case"], state["lib"]
    if case["kind"] == "batch":
        out = state["batch"]()
        out["iterations"] = np.array(state["batch"].its, dtype=np.int64)
        out["s"] = torch.cat([d["s"] for d in state["batch"].mats])
        return out
    if case["kind"] == "adjoint":
        return _run_adjoint(state)
    l = case["k"] + case["p"]
    prm, x, order = state["prm"], case["x"], case["order"].encode()
    if case["kind"] == "stages":
        y = state["yst"]
        lib.sketch(x, prm, state["a"], _lda(case), y, case["N"] * l, state["seed"], ordera=order)
        lib.orthogonalize(x, "TS", prm, y, case["N"] * l)
        if lib.last_error()[0]:
            raise RuntimeError("stages: %s" % (lib.last_error(),))
        return {"q": y}
    algs = tuple(case["algs"].split("/"))
    sym = algs[3] == "SY"
    kn = algs[2] == "KN"
    retv, _, status = lib.isvd(x, prm, algs, state["a"], _lda(case), state["s"], state["ut"], l, state["vt"], l,
                               seed=state["seed"], ordera=order, argv=[None, None, [256, 1e-4], None] if kn else None,
                               retc=(0, 0, 2 if kn else 0, 0), vt_root=-2 if sym else -1,
                               precision=1 if case["mixed"] else 0)
    if status:
        raise RuntimeError("isvd_%sIsvd_ex: %s" % (x, lib.last_error()))
    out = {"s": state["s"]}
    out["u"], v = _turned(state["ut"][:, :case["k"]], None if sym else state["vt"][:, :case["k"]])
    if not sym:
        out["v"] = v
    if kn:
        out["iterations"] = int(retv[2][0])
    return out


# ------------------------------------------------------------------------------------ work
def work(case):
    """One pass: inputs read once, results written once, and the multiplications of the stages (the
    integration's iterations apart: their number depends on the values)."""
    if case["kind"] == "batch":
        b = f = 0.0
        for m, n, k, p in _batch_shapes(case, 0):
            l, N = k + p, case["N"]
            b += 4.0 * (m * n + (m + n) * k + l)
            f += 2.0 * m * n * N * l + 1.0 * m * (N * l) ** 2 + 2.0 * m * n * l
        return {"bytes": b, "flops": f}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "adjoint":  # dA = U Q1' + P2 V', and one application of A to either side
        return {"bytes": 4.0 * (2 * m * n + 2 * (m + n) * k), "flops": 8.0 * m * n * k}
    e = 4.0 if case["x"] == "s" else 8.0
    l, N = k + case["p"], case["N"]
    if case["kind"] == "stages":
        return {"bytes": e * (m * n + m * N * l), "flops": 2.0 * m * n * N * l + 4.0 * m * N * l * l}
    sym = case["algs"].endswith("SY")
    flops = 2.0 * m * n * N * l + 4.0 * m * N * l * l + 1.0 * m * (N * l) ** 2 + 2.0 * m * n * l
    return {"bytes": e * (m * n + m * k + (0 if sym else n * k) + l), "flops": flops}


# --------------------------------------------------------------------------- 64-bit results
def _omega(n, nl, seed):
    """The Gaussian test matrix of a seed (n x nl): Philox4x32-10 blocks, Box-Muller, rounded to bf16."""
    pairs = (n * nl + 1) // 2
    out = torch.empty(2 * pairs, device=DEV, dtype=F64)
    lo32 = 0xFFFFFFFF
    for b in range(0, pairs, 1 << 24):
        c = torch.arange(b, min(b + (1 << 24), pairs), device=DEV, dtype=torch.int64)
        x = [c & lo32, (c >> 32) & lo32, torch.zeros_like(c), torch.zeros_like(c)]
        k0, k1 = seed & lo32, 0
        for _ in range(10):
            p0, p1 = x[0] * 0xD2511F53, x[2] * 0xCD9E8D57
            x = [((p1 >> 32) & lo32) ^ x[1] ^ k0, p1 & lo32, ((p0 >> 32) & lo32) ^ x[3] ^ k1, p0 & lo32]
            k0, k1 = (k0 + 0x9E3779B9) & lo32, (k1 + 0xBB67AE85) & lo32
        u1 = (((x[0] << 21) | (x[1] >> 11)) + 1).to(F64) * 2.0 ** -53
        u2 = ((x[2] << 21) | (x[3] >> 11)).to(F64) * 2.0 ** -53
        rad = torch.sqrt(-2.0 * torch.log(u1))
        out[2 * b:2 * b + 2 * len(c):2] = rad * torch.cos(2.0 * math.pi * u2)
        out[2 * b + 1:2 * b + 2 * len(c):2] = rad * torch.sin(2.0 * math.pi * u2)
    frac, expo = torch.frexp(out[:n * nl])  # to 8 significant bits at once (not through FP32)
    return torch.ldexp(torch.round(frac * 256.0), expo - 8).view(n, nl)


def _householder_q(y):
    """The orthonormal factor of a block with LAPACK's column signs: by Cholesky twice, then the signs
    from the modified LU of the leading block (the diagonal of Householder's R)."""
    q = y
    for _ in range(3):
        r = torch.linalg.cholesky(q.t() @ q).t()
        q = torch.linalg.solve_triangular(r, q, upper=True, left=False)
    l = q.shape[1]
    t = q[:l].clone().cpu().numpy()
    sign = np.ones(l)
    for j in range(l):
        sign[j] = -1.0 if t[j, j] >= 0 else 1.0
        t[j, j] -= sign[j]
        t[j + 1:, j] /= t[j, j]
        t[j + 1:, j + 1:] -= np.outer(t[j + 1:, j], t[j, j + 1:])
    return q * torch.as_tensor(sign, device=q.device)


def _kn(qs, l, N, tol, maxit):
    G = qs.t() @ qs
    M = torch.zeros(N * l, l, device=DEV, dtype=F64)
    M[:l] = torch.eye(l, device=DEV, dtype=F64)
    eye = torch.eye(l, device=DEV, dtype=F64)
    it = 0
    while True:
        it += 1
        B = G @ M
        Dc, Dg = B.t() @ B / N, B.t() @ (G @ B) / N ** 2
        z, w = torch.linalg.eigh(Dg - Dc @ Dc)
        c = torch.sqrt(0.5 + torch.sqrt(0.25 - z.clamp(0, 0.25)))
        C, Ci = (w * c) @ w.t(), (w / c) @ w.t()
        M = M @ (C - Dc @ Ci) + (B / N) @ Ci
        if float(torch.linalg.matrix_norm(C - eye)) <= tol:
            return qs @ M, it
        if it == maxit:
            return qs @ M, it + 1


def _hr(qs, l, N):
    q = [qs[:, i * l:(i + 1) * l] for i in range(N)]
    while len(q) > 1:
        h = len(q) // 2
        for i in range(h):
            w, s, t = torch.linalg.svd(q[i].t() @ q[i + h])
            q[i] = (q[i] @ w + q[i + h] @ t.t()) / torch.sqrt(2.0 * (1.0 + s))
        q = q[:h] if len(q) % 2 == 0 else q[:h] + [q[-1]]
    return q[0]


def _exact_adjoint(st):
    a, s, u, v = (st[q].double() for q in ("a", "s", "u", "v"))
    ds, du, dv = (st[q].double() for q in ("ds", "du", "dv"))
    s2 = s * s
    b = a - u @ (u.t() @ a)
    b = b - (b @ v) @ v.t()
    lam, w = torch.linalg.eigh(b.t() @ b)
    solve = lambda rhs: w @ ((w.t() @ rhs) / (s2[None, :] - lam[:, None]))  # noqa: E731
    ru = du - u @ (u.t() @ du)
    rv = dv - v @ (v.t() @ dv)
    gam = solve(rv)
    lmb = (ru + b @ solve(b.t() @ ru)) / s2
    f = 1.0 / (s2[None, :] - s2[:, None] + torch.eye(len(s), device=s.device, dtype=F64))
    f.fill_diagonal_(0.0)
    ju, jv = u.t() @ du, v.t() @ dv
    j = torch.diag(ds) + (f * (ju - ju.t())) * s[None, :] + s[:, None] * (f * (jv - jv.t()))
    da = u @ j @ v.t() + (lmb * s) @ v.t() + u @ (lmb.t() @ b) + (u * s) @ gam.t() + (b @ gam) @ v.t()
    return {"da": da}


def _exact_solve(case, a, seed):
    m, n, N, l = case["m"], case["n"], case["N"], case["k"] + case["p"]
    y = torch.empty(m, N * l, device=DEV, dtype=F64)
    om = _omega(n, N * l, seed)
    rows = max(1, (1 << 28) // n)
    for r0 in range(0, m, rows):
        y[r0:r0 + rows] = a[r0:r0 + rows].double() @ om
    del om
    for i in range(N):
        blk = y[:, i * l:(i + 1) * l]
        if case["kind"] == "stages":
            y[:, i * l:(i + 1) * l] = _householder_q(blk)
        else:
            y[:, i * l:(i + 1) * l] = torch.linalg.qr(blk)[0] if m < 50000 else _householder_q(blk)
    if case["kind"] == "stages":
        return {"q": y}
    algs = case["algs"].split("/")
    out, k = {}, case["k"]
    if algs[2] == "KN":
        q, out["iterations"] = _kn(y, l, N, 1e-4, 256)
    else:
        q = _hr(y, l, N)
    del y
    z = torch.zeros(n, l, device=DEV, dtype=F64)
    for r0 in range(0, m, rows):
        z += a[r0:r0 + rows].double().t() @ q[r0:r0 + rows]
    if algs[3] == "SY":
        out["s"], w = torch.linalg.eigh((z.t() @ q + q.t() @ z) * 0.5)
        out["u"], _ = _turned(q @ w[:, :k], None)
        return out
    lam, w = (t.flip(-1) for t in torch.linalg.eigh(z.t() @ z))
    out["s"] = lam.clamp_min(0).sqrt()
    out["u"], out["v"] = _turned(q @ w[:, :k], z @ (w[:, :k] / out["s"][:k]))
    return out


def exact(case, seed):
    if case["kind"] == "adjoint":
        st = prepare(case, seed)
        return _exact_adjoint(st)
    if case["kind"] == "batch":
        shapes = _batch_shapes(case, seed)
        lmax = max(k + p for _, _, k, p in shapes)
        parts = []
        for i, (m, n, k, p) in enumerate(shapes):
            c = dict(kind="solve", x="s", m=m, n=n, k=k, p=p, N=case["N"], order="R", algs="GP/GR/KN/GR")
            e = _exact_solve(c, _matrix(c, seed * 1000 + i), 11 + i)
            for q in "uv":
                e[q] = torch.nn.functional.pad(e[q], (0, lmax - k))
            parts.append(e)
        return {"s": torch.cat([e["s"] for e in parts]), "u": torch.cat([e["u"] for e in parts]),
                "v": torch.cat([e["v"] for e in parts]),
                "iterations": np.array([e["iterations"] for e in parts], dtype=np.int64)}
    return _exact_solve(case, _as_mn(case, _matrix(case, seed)), int(seed) % 100000)
