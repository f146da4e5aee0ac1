"""Performance cases of the low-rank factorizations.

Each case is one call (or one burst of calls) that a program makes through the
public API, over the range of sizes, element types and options the package is
used at.  The randomness of a single call is injected (a RandStream the
program draws once), so that the same case gives the same factorization every
time; the batch and the serving loop restart their generators per matrix by
themselves.

Singular and eigenvectors are returned scaled by their values (the principal
coordinates U S and S Vt that a PCA program goes on with on the GPU, signs
fixed as usual by the largest entry of U): an unscaled vector of a tiny
singular value is defined only up to rounding of the matrix over its gap.
Interpolation matrices go to the GPU, where a program applies them, each at
the start of a slot sized for the largest rank its caller allows for.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "lowrankapprox.jl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import lowrankapprox as lra  # noqa: E402

DTYPES = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}
NP_REAL = {"f32": np.float32, "f64": np.float64, "c64": np.float32, "c128": np.float64}


def listed():
    return [
        # one small interaction block of a hierarchical-matrix code: latency
        dict(name="id_kernel_256", kind="id", matrix="kernel", m=256, n=192, dtype="f64", precision="mixed",
             sketch="randn", rtol=1e-10, r=0.0),
        # a call that leaves precision at its default (plain FP64)
        dict(name="id_native_2001", kind="id", matrix="geom", m=2001, n=1501, dtype="f64", precision="native",
             sketch="randn", rtol=1e-6, r=20.3),
        # complex samples of a Fourier kernel, rank about 100 (default precision)
        dict(name="id_complex_1024", kind="id", matrix="fourier", m=1024, n=768, dtype="c128", precision="native",
             sketch="randn", rtol=1e-6, r=0.0),
        # the tall Float32 workload of the benchmark, SRFT and Gaussian sketch
        dict(name="id_tall_srft", kind="id", matrix="geom", m=65536, n=4096, dtype="f32", precision="mixed",
             sketch="srft", rtol=1e-6, r=138.2),
        dict(name="id_tall_randn", kind="id", matrix="geom", m=65536, n=4096, dtype="f32", precision="mixed",
             sketch="randn", rtol=1e-6, r=138.2),
        # many independent kernel blocks of uneven sizes (128 to 2048) in one call
        dict(name="batch_160", kind="batch", count=160, lo=128, hi=2048, rtol=1e-10),
        # the benchmark's headline: psvdfact of a dense 8192 x 8192 matrix
        dict(name="psvd_8192", kind="psvd", matrix="geom", m=8192, n=8192, dtype="f64", precision="mixed",
             sketch="randn", rtol=1e-10, r=40.3),
        # a slowly decaying spectrum (rank about 1800): the serving mix's heavy end
        dict(name="psvd_rank1800", kind="psvd", matrix="geom", m=3001, n=2203, dtype="f64", precision="mixed",
             sketch="randn", rtol=1e-10, r=200.3),
        # a Float32 matrix of ordinary size from the serving mix, odd sides
        dict(name="psvd_f32_1501", kind="psvd", matrix="geom", m=1501, n=1103, dtype="f32", precision="mixed",
             sketch="randn", rtol=1e-6, r=60.3),
        # eigendecomposition of a symmetric matrix with eigenvalues of both signs
        dict(name="pheig_1500", kind="pheig", m=1500, n=1500, dtype="f64", precision="mixed", sketch="randn",
             rtol=1e-8, r=30.3),
        # a burst of mixed idfact / psvdfact requests to the serving loop
        dict(name="serve_16", kind="serve", count=16, lo=256, hi=4096, slots=2),
        # the spectral norm of a dense matrix larger than the L2 cache
        dict(name="snorm_6000", kind="snorm", matrix="geom", m=6000, n=5003, dtype="f64", rtol=1e-6, r=40.3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _decay(rng, m, n, lo, hi):
    """Values per decade: at most a sixteenth of the smaller side, so that
    the matrix has low rank."""
    return round(min(rng.uniform(lo, hi), max(4.0, min(m, n) / 16.0)), 1) + 0.03


def draw(rng):
    kind = rng.choice(["id", "id", "id", "psvd", "psvd", "pheig", "batch", "serve", "snorm"])
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 8, 160), lo=128, hi=rng.randint(256, 2048), rtol=1e-10)
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(4, 12), lo=256, hi=rng.randint(512, 3000), slots=2)
    if kind == "snorm":
        return dict(kind="snorm", matrix="geom", m=_log_int(rng, 256, 8000), n=_log_int(rng, 256, 8000),
                    dtype=rng.choice(["f64", "f32"]), rtol=1e-6, r=round(rng.uniform(20, 60), 1) + 0.03)
    if kind == "pheig":
        n = _log_int(rng, 256, 3000)
        return dict(kind="pheig", m=n, n=n, dtype="f64", precision="mixed", sketch="randn", rtol=1e-8,
                    r=_decay(rng, n, n, 10, 40))
    if kind == "psvd":
        dtype = rng.choice(["f64", "f32"])
        m, n = _log_int(rng, 256, 8000), _log_int(rng, 256, 8000)
        return dict(kind="psvd", matrix="geom", m=m, n=n, dtype=dtype, precision="mixed", sketch="randn",
                    rtol=1e-10 if dtype == "f64" else 1e-6, r=_decay(rng, m, n, 20, 120))
    form = rng.choice(["kernel", "geom64", "tall32", "native", "complex"])
    if form == "kernel":
        return dict(kind="id", matrix="kernel", m=_log_int(rng, 128, 2048), n=_log_int(rng, 128, 2048), dtype="f64",
                    precision="mixed", sketch="randn", rtol=1e-10, r=0.0)
    if form == "geom64":
        m, n = _log_int(rng, 256, 8000), _log_int(rng, 256, 8000)
        return dict(kind="id", matrix="geom", m=m, n=n, dtype="f64", precision="mixed", sketch="randn", rtol=1e-10,
                    r=_decay(rng, m, n, 20, 100))
    if form == "tall32":
        m, n = _log_int(rng, 4096, 65536), _log_int(rng, 256, 4096)
        return dict(kind="id", matrix="geom", m=m, n=n, dtype="f32", precision="mixed",
                    sketch=rng.choice(["srft", "randn"]), rtol=1e-6, r=_decay(rng, m, n, 20, 138))
    if form == "native":
        m, n = _log_int(rng, 256, 4096), _log_int(rng, 256, 4096)
        return dict(kind="id", matrix="geom", m=m, n=n, dtype=rng.choice(["f64", "f32"]), precision="native",
                    sketch="randn", rtol=1e-6, r=_decay(rng, m, n, 10, 40))
    return dict(kind="id", matrix="fourier", m=_log_int(rng, 128, 2048), n=_log_int(rng, 128, 1536),
                dtype=rng.choice(["c128", "c64"]), precision="native", sketch="randn",
                rtol=1e-6 if rng.random() < 0.5 else 1e-5, r=0.0)


# ---- inputs --------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _colmajor(A):
    return A.t().contiguous().t()


def _geom_rank(m, n, r, rtol):
    return max(1, min(m, n, int((-math.log10(rtol) - 1.0) * r) + 1))


def _geom_factors(m, n, r, rtol, seed, dtype):
    """U, s, V of A = U diag(s) V' of numerical rank k: U and V orthonormal
    (QR of Gaussians), s_i = 10^(-i/r) down to ten times the tolerance."""
    k = _geom_rank(m, n, r, rtol)
    g = _gen(seed)
    facs = []
    for rows in (m, n):
        G = _randn(g, rows, k)
        if dtype == "f32" and rows > 8192:
            G = G.float()
        facs.append(torch.linalg.qr(G).Q)
    s = torch.pow(10.0, -torch.arange(k, dtype=torch.float64, device="cuda") / r)
    return facs[0], s, facs[1]


def _kernel(m, n, g):
    """1 / (1 + |x - y|^2) between points of [0,1]^2 and of a square 0.5 away."""
    x = torch.rand(m, 2, generator=g, device="cuda", dtype=torch.float64)
    y = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    y[:, 0] += 1.5
    d2 = (x[:, None, 0] - y[None, :, 0]) ** 2 + (x[:, None, 1] - y[None, :, 1]) ** 2
    return _colmajor(1.0 / (1.0 + d2))


def _matrix(c, seed):
    if c["matrix"] == "kernel":
        return _kernel(c["m"], c["n"], _gen(seed))
    if c["matrix"] == "fourier":
        # exp(-2 pi i x y), x in [0, m/16), y in [0, 1): rank about m/16
        g = _gen(seed)
        x = torch.rand(c["m"], generator=g, device="cuda", dtype=torch.float64) * (c["m"] / 16.0)
        y = torch.rand(c["n"], generator=g, device="cuda", dtype=torch.float64)
        ph = -2.0 * math.pi * torch.outer(x, y)
        return _colmajor(torch.polar(torch.ones_like(ph), ph).to(DTYPES[c["dtype"]]))
    U, s, V = _geom_factors(c["m"], c["n"], c["r"], c["rtol"], seed, c["dtype"])
    dt = U.dtype if U.dtype == V.dtype else torch.float32
    return _colmajor(((U * s.to(U.dtype)).to(dt) @ V.T.to(dt)).to(DTYPES[c["dtype"]]))


def _herm_factors(c, seed):
    """Eigenvalues 10^(-i/r), every third negative, and orthonormal vectors."""
    n = c["n"]
    k = _geom_rank(n, n, c["r"], c["rtol"])
    V = torch.linalg.qr(_randn(_gen(seed), n, k)).Q
    i = torch.arange(k, dtype=torch.float64, device="cuda")
    w = torch.pow(10.0, -i / c["r"]) * torch.where(i % 3 == 2, -1.0, 1.0)
    return V, w


def _rank(c):
    """About the rank the call finds (the length of the streams, the work)."""
    top = min(c["m"], c["n"])
    if c.get("matrix") == "kernel":
        return min(top, 48)
    if c.get("matrix") == "fourier":
        return min(top, c["m"] // 16 + 40)
    return _geom_rank(c["m"], c["n"], c["r"], c["rtol"])


def _orders(rank):
    """The adaptive loop's sketch orders up to the one that reveals `rank`."""
    out, nt = [], 32
    while True:
        out.append(nt + 8)
        if rank < nt:
            return out
        nt *= 2


def _stream(c, seed):
    """Draws for one step more than the call should need."""
    orders = _orders(2 * _rank(c) + 64)
    g = _gen(seed + 7919)
    if c["sketch"] == "srft":
        gauss = _randn(g, c["m"] * len(orders))
        ints = np.random.default_rng(seed).integers(1, c["m"] + 1, sum(orders))
        return lra.RandStream(gauss=gauss, ints=ints)
    per = 2 if c["dtype"] in ("c64", "c128") else 1
    side = max(c["m"], c["n"]) if c["kind"] == "psvd" else c["m"]  # psvdfact sketches the longer side
    gauss = _randn(g, side * sum(orders) * per)
    gauss.mul_(32.0).round_().clamp_(-127.0, 127.0).div_(32.0)
    return lra.RandStream(gauss=gauss)


def _options(c):
    return lra.LRAOptions(NP_REAL[c["dtype"]], rtol=c["rtol"], sketch=c["sketch"], precision=c["precision"])


def _requests(c, seed):
    """70 % idfact / 30 % psvdfact, sides log-uniform, Float32 / Float64 half
    and half, s_i = 10^(-i/r) with r from 20 to 200 (at most a sixteenth of
    the smaller side, so that every matrix has low rank)."""
    shapes = np.random.default_rng(5)  # the mix itself is the case's, the entries are the seed's
    out = []
    for i in range(c["count"]):
        m, n = (int(round(math.exp(shapes.uniform(math.log(c["lo"]), math.log(c["hi"]))))) for _ in range(2))
        dtype = "f64" if i % 2 == 0 else "f32"
        kind = "psvdfact" if i % 10 in (2, 5, 8) else "idfact"
        r = round(min(float(shapes.uniform(20, 200)), max(8.0, min(m, n) / 16.0)), 1) + 0.03
        rtol = 1e-10 if dtype == "f64" else 1e-6
        U, s, V = _geom_factors(m, n, r, rtol, seed * 1000 + i, dtype)
        A = _colmajor(((U * s) @ V.T).to(DTYPES[dtype]))
        o = lra.LRAOptions(NP_REAL[dtype], rtol=rtol, precision="mixed", seed=11 + i)
        out.append((kind, A, o, (U, s, V)))
    return out


def prepare(case, seed):
    c = case
    state = {"case": c}
    if c["kind"] == "batch":
        sizes = np.random.default_rng(4).integers(c["lo"], c["hi"] + 1, (c["count"], 2))
        g = _gen(seed)
        state["mats"] = [_kernel(int(m), int(n), g) for m, n in sizes]
        state["opts"] = lra.LRAOptions(rtol=c["rtol"], precision="mixed", seed=3)
    elif c["kind"] == "serve":
        state["requests"] = [(kind, A, o) for kind, A, o, _ in _requests(c, seed)]
        state["server"] = lra.Server(slots=c["slots"], hbm_budget_bytes=64 << 30)
    elif c["kind"] == "pheig":
        V, w = _herm_factors(c, seed)
        A = (V * w) @ V.T
        state["A"] = _colmajor(0.5 * (A + A.T))
        state["rand"], state["opts"] = _stream(c, seed), _options(c)
    elif c["kind"] == "snorm":
        state["A"] = _matrix(c, seed)
        state["rand"] = lra.RandStream(gauss=_randn(_gen(seed + 7919), c["n"]))
    else:
        state["A"] = _matrix(c, seed)
        state["rand"], state["opts"] = _stream(c, seed), _options(c)
        state["top"] = _orders(_rank(c))[-1]
    torch.cuda.synchronize()
    return state


# ---- one pass ------------------------------------------------------------------------


def _coords(U, S, Vt):
    """S, U S and S Vt, the sign of each pair fixed by U's largest entry."""
    S = S.to(U.dtype)
    if Vt is None:
        lead = U.gather(0, U.abs().argmax(0, keepdim=True)).sign()
        return U * (S * lead)
    lead = U.gather(0, U.abs().argmax(0, keepdim=True)).sign()
    w = S * lead[0]
    return [S, U * w, w[:, None] * Vt]


def _to_gpu(a):
    """A column-major host factor on the GPU, layout kept."""
    return torch.from_numpy(a.T).cuda().t()


def _svd_out(F):
    return _coords(_to_gpu(F.U), torch.from_numpy(F.S).cuda(), _to_gpu(F.Vt))


def _id_out(Vs, ns, top):
    """Permutations, ranks, and the interpolation matrices back to back on
    the GPU, each in a slot for rank min(top, n)."""
    pack = torch.zeros(sum(min(top, n) * n for n in ns), dtype=torch.from_numpy(Vs[0].T).dtype, device="cuda")
    at = 0
    for V, n in zip(Vs, ns):
        pack[at:at + V.T.size].copy_(torch.from_numpy(V.T.reshape(-1, order="F")), non_blocking=True)
        at += min(top, n) * n
    torch.cuda.current_stream().synchronize()  # before the host copies are given back
    return {"p": np.concatenate([x for V in Vs for x in (V.sk, V.rd)]), "k": np.array([V.k for V in Vs]), "T": pack}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "id":
        V = lra.idfact(state["A"], state["opts"], rand=state["rand"])
        return _id_out([V], [c["n"]], state["top"])
    if kind == "psvd":
        return _svd_out(lra.psvdfact(state["A"], state["opts"], rand=state["rand"]))
    if kind == "pheig":
        F = lra.pheigfact(state["A"], state["opts"], rand=state["rand"])
        w = torch.from_numpy(F.values).cuda()
        return [w, _coords(_to_gpu(F.vectors), w, None)]
    if kind == "snorm":
        return lra.snorm(state["A"], rand=state["rand"])
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(k, A, o) for k, A, o in state["requests"]]
        out = []
        for (k, _, _), t in zip(state["requests"], tickets):
            F = srv.result(t)
            out.append(_id_out([F], [F.k + len(F.rd)], 2056) if k == "idfact" else _svd_out(F))
        return out
    Vs = lra.idfact_batched(state["mats"], state["opts"])
    return _id_out(Vs, [V.k + len(V.rd) for V in Vs], 96)


# ---- what a pass cannot do without ---------------------------------------------------


def _work_one(kind, m, n, k, size, cplx=False):
    """The matrix read once, the factors written once; one sketch of the
    final order, its pivoted QR to k, the solve, and for psvdfact the QR of
    the skeleton, the k x k SVD's products and U and Vt."""
    l = _orders(k)[-1]
    fl = 2.0 * l * m * n + 4.0 * l * n * k - 2.0 * k * k * (l + n) + 4.0 / 3.0 * k ** 3 + k * k * max(0, n - k)
    by = size * (m * n + k * max(0, n - k)) + 8 * n
    if kind in ("psvd", "psvdfact"):
        fl += 2.0 * m * k * k + k * k * max(0, n - k) + 12.0 * k ** 3 + 2.0 * (m + n) * k * k
        by = size * (m * n + (m + n) * k + k)
    elif kind == "pheig":
        fl += k * k * max(0, n - k) + 12.0 * k ** 3 + 2.0 * n * k * k
        by = size * (m * n + n * k + k)
    return by, fl * (4.0 if cplx else 1.0)


def work(case):
    c = case
    if c["kind"] == "batch":
        sizes = np.random.default_rng(4).integers(c["lo"], c["hi"] + 1, (c["count"], 2))
        parts = [_work_one("id", int(m), int(n), min(41, int(m), int(n)), 8) for m, n in sizes]
    elif c["kind"] == "serve":
        shapes, parts = np.random.default_rng(5), []
        for i in range(c["count"]):
            m, n = (int(round(math.exp(shapes.uniform(math.log(c["lo"]), math.log(c["hi"]))))) for _ in range(2))
            r = min(float(shapes.uniform(20, 200)), max(8.0, min(m, n) / 16.0))
            k = min(m, n, int(r * (9 if i % 2 == 0 else 5)))
            parts.append(_work_one("psvd" if i % 10 in (2, 5, 8) else "id", m, n, k, 8 if i % 2 == 0 else 4))
    elif c["kind"] == "snorm":
        size = 8 if c["dtype"] == "f64" else 4
        # 32 power iterations, each reading the matrix twice where it does not
        # stay in the cache between the two
        return {"bytes": float(size * c["m"] * c["n"]), "flops": 32.0 * 4.0 * c["m"] * c["n"]}
    else:
        size = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}[c["dtype"]]
        parts = [_work_one(c["kind"], c["m"], c["n"], _rank(c), size, c["dtype"] in ("c64", "c128"))]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ---- the same in 64 bits without the package -----------------------------------------


def _exact_svd(U, s, V):
    return _coords(U.double(), s, V.double().t())


def exact(case, seed):
    """Singular and eigenvalues and principal coordinates from the factors the
    matrix was made of; the norm by the same power iteration.  The skeleton
    and T of an ID follow from the random sketch and have no value of their
    own: None."""
    c = case
    if c["kind"] == "psvd":
        U, s, V = _geom_factors(c["m"], c["n"], c["r"], c["rtol"], seed, c["dtype"])
        return _exact_svd(U, s, V)
    if c["kind"] == "pheig":
        V, w = _herm_factors(c, seed)
        w, at = w.sort()
        return [w, _coords(V[:, at], w, None)]
    if c["kind"] == "serve":
        return [None if kind == "idfact" else _exact_svd(*f)
                for kind, _, _, f in _requests(c, seed)]
    if c["kind"] == "snorm":
        A = _matrix(c, seed).double()
        x = _randn(_gen(seed + 7919), c["n"])
        nrm, s, t, it = x.norm(), 1.0, 0.0, 0
        tol = 5 * float(np.finfo(NP_REAL[c["dtype"]]).eps)
        while s > 0 and abs(s - t) > t * tol and it < 32:
            x = A.t() @ (A @ (x / nrm))
            nrm = x.norm()
            s, t, it = math.sqrt(float(nrm)), s, it + 1
        return float(s)
    return None
