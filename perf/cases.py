"""The calls this framework is timed on, through its public functions.

Every case is one user-level call (``logdet``, ``traceinv``, ``trace``,
``trexp`` with ``method="slq", gpu=True``, or ``BatchPlan.run``) on a seeded
synthetic matrix of the kinds the test-suite, the benchmark script and the
reference's own speed benchmark use:

* ``toeplitz``: Gram form of the upper bidiagonal Toeplitz matrix, float64,
  with the adaptive stopping rule;
* ``corr``: sparse exponential-kernel correlation matrices with the points in
  no particular order -- one estimate on a kept operator, a call on a host
  matrix (set-up included), or a sweep of t in A + t I;
* ``grid``: shifted five-point Laplacians (the finite-element matrices of the
  reference's speed benchmark have 7 to 14 entries a row), no
  reorthogonalisation;
* ``dense``: dense float32 correlation matrices;
* ``design``: X^T X + t I of a sparse rectangular X;
* ``batch``: many correlation matrices of different sizes in one plan.
"""

import math

import numpy as np
import torch

import imate_b200 as ib
from imate_b200.batch import BatchPlan
from imate_b200.sample_matrices import correlation_matrix_device

CSR = type(ib.toeplitz(2.0, 1.0, 2))
CSC = type(ib.toeplitz(2.0, 1.0, 2, format="csc"))
FUNCS = {"logdet": ib.logdet, "traceinv": ib.traceinv, "trace": ib.trace,
         "trexp": ib.trexp}


def listed():
    return [
        # the smallest call: a small matrix, every option at its default
        # (degree 20, 10 to 50 samples, no reorthogonalisation)
        dict(name="small default f64", kind="corr", n=500, row=20,
             dtype="float64", func="logdet", degree=20, lo=10, hi=50,
             rtol=1e-2, orth=0, sweep=0, one_shot=False, csc=False),
        # the first benchmark configuration: Golub-Kahan with full
        # reorthogonalisation, stopped by the relative error of the estimate
        dict(name="toeplitz gram f64", kind="toeplitz", n=16384,
             func="logdet", degree=30, lo=50, hi=200, rtol=1e-3, orth=-1),
        # the headline configuration: 256 probes, 50 steps, full
        # reorthogonalisation on 48 million entries
        dict(name="corr logdet f32", kind="corr", n=262144, row=185,
             dtype="float32", func="logdet", degree=50, lo=256, hi=256,
             rtol=0.0, orth=-1, sweep=0, one_shot=False, csc=False),
        # the drop-in call on a host matrix: upload, orders and formats are
        # part of every call
        dict(name="corr one shot f32", kind="corr", n=100003, row=90,
             dtype="float32", func="logdet", degree=30, lo=128, hi=128,
             rtol=0.0, orth=-1, sweep=0, one_shot=True, csc=False),
        # plain double precision on a matrix of a size that is no round number
        dict(name="corr traceinv f64", kind="corr", n=40009, row=60,
             dtype="float64", func="traceinv", degree=40, lo=64, hi=64,
             rtol=0.0, orth=-1, sweep=0, one_shot=False, csc=False),
        # a sweep of 512 t by the eigenvalue shift of one Krylov run a probe
        dict(name="sweep logdet f32", kind="corr", n=32768, row=100,
             dtype="float32", func="logdet", degree=50, lo=64, hi=64,
             rtol=0.0, orth=-1, sweep=512, one_shot=False, csc=False),
        # a window of reorthogonalisation, CSC input, a probe count that is
        # no power of two
        dict(name="corr trexp window f32", kind="corr", n=30011, row=40,
             dtype="float32", func="trexp", degree=30, lo=100, hi=100,
             rtol=0.0, orth=5, sweep=0, one_shot=False, csc=True),
        # the reference's speed benchmark: traceinv, 200 probes, degree 80, no
        # reorthogonalisation, half a million rows of a mesh matrix
        dict(name="grid traceinv f32", kind="grid", nx=725, ny=723,
             dtype="float32", func="traceinv", degree=80, probes=200),
        dict(name="grid traceinv f64", kind="grid", nx=301, ny=299,
             dtype="float64", func="traceinv", degree=80, probes=100),
        # a dense kernel matrix
        dict(name="dense logdet f32", kind="dense", n=8192, func="logdet",
             degree=50, probes=256, orth=-1),
        # regularised normal equations of a tall sparse matrix
        dict(name="design logdet f32", kind="design", rows=524288,
             cols=131072, row=16, func="logdet", degree=30, probes=128,
             orth=0),
        # a plan over matrices of different sizes, launched as one graph
        dict(name="batch logdet f32", kind="batch", count=16, log2_lo=10.0,
             log2_hi=15.0, func="logdet", degree=40, probes=256, orth=0),
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["corr", "corr", "corr", "toeplitz", "grid", "dense",
                       "design", "batch"])
    if kind == "toeplitz":
        return dict(kind=kind, n=_log(rng, 2000, 60000), func="logdet",
                    degree=rng.randint(20, 40), lo=50,
                    hi=rng.randint(100, 200), rtol=1e-3,
                    orth=rng.choice([0, -1, -1]))
    if kind == "corr":
        f64 = rng.random() < 0.4
        n = _log(rng, 500, 50000 if f64 else 200000)
        probes = rng.choice([32, 64, 100] if f64 else [64, 100, 128, 256])
        sweep = rng.choice([0, 0, 0, 16, 512]) if n < 50000 else 0
        return dict(kind=kind, n=n, row=rng.randint(15, 60 if f64 else 150),
                    dtype="float64" if f64 else "float32",
                    func="logdet" if sweep else
                    rng.choice(["logdet", "traceinv", "trexp"]),
                    degree=rng.randint(20, 50), lo=probes, hi=probes,
                    rtol=0.0, orth=rng.choice([0, -1, -1, 6]), sweep=sweep,
                    one_shot=not sweep and rng.random() < 0.25,
                    csc=not sweep and rng.random() < 0.2)
    if kind == "grid":
        f64 = rng.random() < 0.5
        side = _log(rng, 80, 350 if f64 else 720)
        return dict(kind=kind, nx=side, ny=side + rng.randint(-7, 7),
                    dtype="float64" if f64 else "float32",
                    func=rng.choice(["traceinv", "logdet"]),
                    degree=rng.randint(30, 80),
                    probes=rng.choice([50, 100, 200]))
    if kind == "dense":
        return dict(kind=kind, n=_log(rng, 1000, 9000),
                    func=rng.choice(["logdet", "traceinv"]),
                    degree=rng.randint(20, 50),
                    probes=rng.choice([64, 100, 256]),
                    orth=rng.choice([0, -1, -1]))
    if kind == "design":
        cols = _log(rng, 10000, 150000)
        return dict(kind=kind, rows=int(cols * rng.uniform(1.5, 4.5)),
                    cols=cols, row=rng.randint(6, 18), func="logdet",
                    degree=rng.randint(20, 40),
                    probes=rng.choice([64, 128, 200]),
                    orth=rng.choice([0, 0, -1]))
    return dict(kind="batch", count=rng.randint(5, 20), log2_lo=10.0,
                log2_hi=rng.uniform(12.0, 15.0), func="logdet",
                degree=rng.randint(20, 40), probes=rng.choice([100, 128, 256]),
                orth=rng.choice([0, 0, -1]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _corr_scale(n, row):
    """The length scale at which a row of the correlation matrix of n points
    in the unit square holds about ``row`` entries (cut at 0.05)."""
    return math.sqrt(row / (math.pi * n)) / -math.log(0.05)


def _correlation(n, row, dtype, seed, csc=False):
    """Host CSR (or CSC) of the correlation matrix of n random points, rows
    in the points' own order, shifted to be positive definite."""
    pts = np.random.default_rng(seed).random((n, 2))
    ptr, ind, val, perm = correlation_matrix_device(
        n, scale=_corr_scale(n, row), threshold=0.05, shift=0.2, points=pts,
        dtype=dtype)
    # undo the builder's cell order
    perm = perm.long()
    r = perm[torch.repeat_interleave(torch.arange(n, device=perm.device),
                                     (ptr[1:] - ptr[:-1]).long())]
    key, at = torch.sort(r * n + perm[ind.long()])
    ptr = torch.zeros(n + 1, dtype=torch.long, device=r.device)
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    return (CSC if csc else CSR)(
        (val[at].cpu().numpy(), (key % n).int().cpu().numpy(),
         ptr.int().cpu().numpy()), shape=(n, n))


def _grid(nx, ny, dtype, seed):
    """Five-point diffusion operator on an nx x ny grid with edge weights
    that vary by a quarter, plus 0.5 I."""
    g = np.random.default_rng(seed)
    n = nx * ny
    at = np.arange(n).reshape(ny, nx)
    wx = g.uniform(0.75, 1.0, (ny, nx - 1))
    wy = g.uniform(0.75, 1.0, (ny - 1, nx))
    # neighbours of every cell in column order: up, left, self, right, down
    val = np.zeros((n, 5))
    v = val.reshape(ny, nx, 5)
    v[1:, :, 0] = -wy
    v[:, 1:, 1] = -wx
    v[:, :-1, 3] = -wx
    v[:-1, :, 4] = -wy
    val[:, 2] = 0.5 - val[:, [0, 1, 3, 4]].sum(1)
    col = at.reshape(-1, 1) + np.array([-nx, -1, 0, 1, nx])
    keep = val != 0.0
    ptr = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(keep.sum(1), out=ptr[1:])
    return CSR((val[keep].astype(dtype), col[keep].astype(np.int32), ptr),
               shape=(n, n))


def _dense(n, seed):
    """Dense float32 kernel matrix of n points in the unit square."""
    p = torch.from_numpy(np.random.default_rng(seed).random((n, 2))).cuda()
    k = torch.exp(-torch.cdist(p, p) / 0.02)
    k.diagonal().fill_(1.1)
    return k.float().cpu().numpy()


def _design(rows, cols, per_col, seed):
    """Sparse X in CSC: per column, ``per_col`` rows one in each of equally
    many strata, values N(0, 1)."""
    g = np.random.default_rng(seed)
    step = rows // per_col
    ind = (g.integers(0, step, (cols, per_col)) +
           step * np.arange(per_col)).astype(np.int32)
    ptr = np.arange(0, cols * per_col + 1, per_col, dtype=np.int32)
    val = g.standard_normal(cols * per_col).astype(np.float32)
    return CSC((val, ind.reshape(-1), ptr), shape=(rows, cols))


def _batch_arrays(case, seed):
    """(n, indptr, indices, data) on the GPU of each matrix of a batch."""
    g = np.random.default_rng(seed)
    # the largest size of the range is always there, so that the work of a
    # batch does not hang on its seed
    x = np.linspace(case["log2_lo"], case["log2_hi"], case["count"])
    out = []
    for i, e in enumerate(x):
        n = int(round(2.0 ** e)) + int(g.integers(0, 9))
        ptr, ind, val, _ = correlation_matrix_device(
            n, scale=_corr_scale(n, 60), threshold=0.05, shift=0.2,
            seed=seed * 1000 + i, dtype="float32")
        out.append((n, ptr, ind, val))
    return out


def _sweep(case):
    return np.logspace(-4, 2, case["sweep"]) if case.get("sweep") else None


def _options(case, seed):
    """Keyword arguments of one estimate."""
    lo = case.get("lo", case.get("probes"))
    return dict(min_num_samples=lo, max_num_samples=case.get("hi", lo),
                error_rtol=case.get("rtol", 0.0),
                lanczos_degree=case["degree"],
                orthogonalize=case.get("orth", 0), seed=seed % 1000003)


def prepare(case, seed):
    kind = case["kind"]
    opts = _options(case, seed)
    if kind == "batch":
        plan = BatchPlan([dict(opts, func=case["func"],
                               A=ib.DeviceMatrix(p, i, v, (n, n)))
                          for n, p, i, v in _batch_arrays(case, seed)])
        return {"plan": plan}
    if kind == "toeplitz":
        # seeded coefficients near the a = 2, b = 1 of the benchmark
        a, b = 2.0 + np.random.default_rng(seed).uniform(0.0, 0.1, 2)
        A, opts["gram"] = ib.Matrix(ib.toeplitz(a, b - 1.0, case["n"])), True
    elif kind == "corr":
        A = _correlation(case["n"], case["row"], case["dtype"], seed,
                         case["csc"])
        if case["sweep"]:
            A = ib.AffineMatrixFunction(A)
            opts["parameters"] = _sweep(case)
        elif not case["one_shot"]:
            A = ib.Matrix(A)
    elif kind == "grid":
        A = ib.Matrix(_grid(case["nx"], case["ny"], case["dtype"], seed))
    elif kind == "dense":
        A = ib.Matrix(_dense(case["n"], seed))
    else:
        A = ib.GramAffineMatrixFunction(_design(case["rows"], case["cols"],
                                                case["row"], seed))
        opts["parameters"] = 0.5
    if hasattr(A, "get_device_operator"):
        A.get_device_operator(need_transpose=kind in ("toeplitz", "design"))
    return {"A": A, "func": FUNCS[case["func"]], "opts": opts}


# ---------------------------------------------------------------------------
# the call
# ---------------------------------------------------------------------------


def _outputs(value, info):
    c = info["convergence"]
    return {"value": value, "error": info["error"]["absolute_error"],
            "samples": c["samples"], "used": c["num_samples_used"]}


def run(state):
    if "plan" in state:
        got = [_outputs(v, info) for v, info in state["plan"].run()]
        return {"value": np.array([g["value"] for g in got]),
                "error": np.array([g["error"] for g in got]),
                "samples": np.stack([g["samples"] for g in got]),
                "used": np.array([g["used"] for g in got])}
    value, info = state["func"](state["A"], method="slq", gpu=True,
                                num_gpu_devices=1, return_info=True,
                                **state["opts"])
    return _outputs(value, info)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------


def _krylov_work(n, entries, entry_bytes, width, b, m, orth, sides=1):
    """Bytes and operations of b Lanczos runs of m steps on n rows: every
    step reads the matrix once and the basis vectors it orthogonalises
    against once, and writes one new vector (``sides`` = 2: left and right
    vectors, two products).  A dense basis of a large matrix fits no cache;
    one that would is counted as written and read once all the same."""
    by = fl = 0.0
    for j in range(m):
        window = j + 1 if orth < 0 else min(j + 1, max(orth, 2))
        by += sides * (entries * entry_bytes + (window + 1.0) * n * b * width)
        fl += sides * b * (2.0 * entries + 6.0 * n +
                           (4.0 * n * window if orth else 0.0))
    return by, fl


def work(case):
    kind, m = case["kind"], case["degree"]
    b = case.get("hi", case.get("probes"))
    orth = case.get("orth", 0)
    if kind == "batch":
        by = fl = 0.0
        for e in np.linspace(case["log2_lo"], case["log2_hi"], case["count"]):
            n = 2.0 ** e
            x, y = _krylov_work(n, 60.0 * n, 8, 4, b, m, orth)
            by, fl = by + x, fl + y
    elif kind == "toeplitz":
        n = case["n"]
        by, fl = _krylov_work(n, 2.0 * n, 12, 8, b, m, orth, sides=2)
    elif kind == "corr":
        w = 8 if case["dtype"] == "float64" else 4
        by, fl = _krylov_work(case["n"], float(case["n"]) * case["row"],
                              w + 4, w, b, m, orth)
        fl += 30.0 * b * m * case["sweep"]
    elif kind == "grid":
        n = float(case["nx"]) * case["ny"]
        w = 8 if case["dtype"] == "float64" else 4
        by, fl = _krylov_work(n, 5.0 * n, w + 4, w, b, m, 0)
    elif kind == "dense":
        n = float(case["n"])
        by, fl = _krylov_work(n, n * n, 4, 4, b, m, orth)
    else:
        n, z = float(case["cols"]), float(case["cols"]) * case["row"]
        by, fl = _krylov_work(n, 2.0 * z, 8, 4, b, m, orth)
        by += 2.0 * m * case["rows"] * b * 4
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# the same estimates in 64 bits with plain torch
# ---------------------------------------------------------------------------

_M64 = (1 << 64) - 1


def _draw64(s):
    """One xoshiro256** draw of the state list s (Blackman and Vigna)."""
    x = (s[1] * 5) & _M64
    r = ((((x << 7) | (x >> 57)) & _M64) * 9) & _M64
    t = (s[1] << 17) & _M64
    s[2] ^= s[0]
    s[3] ^= s[1]
    s[1] ^= s[2]
    s[0] ^= s[3]
    s[2] ^= t
    s[3] = ((s[3] << 45) | (s[3] >> 19)) & _M64
    return r


def _probes(seed, n, count):
    """The documented probe stream: Rademacher vectors from the words of one
    xoshiro256** stream (SplitMix64 seeding, one jump), n // 64 + 1 words to
    a probe, least significant bit first.  [count, n] of +-1."""
    z, s = (seed << 32) | seed, []
    for _ in range(4):
        z = (z + 0x9e3779b97f4a7c15) & _M64
        x = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & _M64
        x = ((x ^ (x >> 27)) * 0x94d049bb133111eb) & _M64
        s.append(x ^ (x >> 31))
    acc = [0, 0, 0, 0]
    for w in (0x180ec6d33cfd0aba, 0xd5a61266f0c9392c, 0xa9582618e03fc9aa,
              0x39abdc4529b1661c):
        for i in range(64):
            if (w >> i) & 1:
                acc = [a ^ b for a, b in zip(acc, s)]
            _draw64(s)
    words = n // 64 + 1
    w = np.array([_draw64(acc) for _ in range(count * words)], np.uint64)
    bits = np.unpackbits(w.view(np.uint8), bitorder="little")
    bits = bits.reshape(count, words * 64)[:, :n]
    return torch.from_numpy(bits).cuda().double() * 2.0 - 1.0


def _to_torch(A):
    """A host CSR or CSC matrix as a float64 CSR tensor on the GPU (a CSC
    matrix as the CSR of its transpose)."""
    shape = A.shape if A.format == "csr" else A.shape[::-1]
    return torch.sparse_csr_tensor(
        torch.from_numpy(A.indptr).cuda(), torch.from_numpy(A.indices).cuda(),
        torch.from_numpy(A.data).cuda().double(), size=shape)


def _lanczos_samples(mul, n, case, seed, params, shift=0.0):
    """[probes, params] samples n * e1^T f(T + t I) e1 of Lanczos runs with
    full reorthogonalisation in float64 (none where the case asks for none:
    the matrices of those cases lose no orthogonality in these steps)."""
    opts = _options(case, seed)
    m, count = opts["lanczos_degree"], opts["max_num_samples"]
    keep = m if opts["orthogonalize"] else 2
    Z = _probes(opts["seed"], n, count)
    width = max(1, min(count, int(24e9 / (8.0 * n * keep))))
    out = []
    for c0 in range(0, count, width):
        v = Z[c0:c0 + width].T.contiguous() / math.sqrt(n)
        w = v.shape[1]
        V = torch.zeros((keep, n, w), dtype=torch.float64, device="cuda")
        T = torch.zeros((w, m, m), dtype=torch.float64, device="cuda")
        beta, prev = None, None
        for j in range(m):
            V[j % keep] = v
            u = mul(v)
            if prev is not None:
                u = u - beta * prev
            a = (v * u).sum(0)
            u = u - a * v
            if keep == m:
                for _ in range(2):
                    h = torch.einsum("jnw,nw->jw", V[:j + 1], u)
                    u = u - torch.einsum("jnw,jw->nw", V[:j + 1], h)
            T[:, j, j] = a
            beta = u.norm(dim=0)
            if j + 1 < m:
                T[:, j, j + 1] = T[:, j + 1, j] = beta
            prev, v = v, u / beta
        theta, Q = torch.linalg.eigh(T)
        x = theta[:, :, None] + torch.as_tensor(params, device="cuda") + shift
        f = {"logdet": torch.log, "traceinv": torch.reciprocal,
             "trace": torch.clone, "trexp": torch.exp}[case["func"]](x)
        out.append(n * (Q[:, 0, :, None] ** 2 * f).sum(1))
        del V, T
    return torch.cat(out).cpu().numpy()


def _used(samples, opts):
    """Samples the sequential stopping rule takes (the first count from
    min_num_samples on whose 95 % error is below rtol times the mean)."""
    lo, hi, rtol = (opts[k] for k in ("min_num_samples", "max_num_samples",
                                      "error_rtol"))
    z = math.sqrt(2.0) * float(torch.erfinv(torch.tensor(0.95).double()))
    for k in range(lo, hi):
        x = samples[:k]
        if k > 1 and z * x.std(ddof=1) / math.sqrt(k) < rtol * x.mean():
            return k
    return hi


def exact(case, seed):
    kind, opts = case["kind"], _options(case, seed)
    cost = work(case)
    if max(cost["bytes"] / 2e12, cost["flops"] / 2e13) > 8.0:
        return None
    t, shift = np.zeros(1), 0.0
    if kind == "batch":
        rows = []
        for n, ptr, ind, val in _batch_arrays(case, seed):
            M = torch.sparse_csr_tensor(ptr, ind, val.double(), size=(n, n))
            rows.append(_lanczos_samples(lambda x: M @ x, n, case, seed, t)
                        [:, 0])
        return {"value": None, "error": None, "samples": np.stack(rows),
                "used": None}
    if kind == "dense":
        K = torch.from_numpy(_dense(case["n"], seed)).cuda().double()
        n, mul = case["n"], lambda x: K @ x
    elif kind == "toeplitz":
        a, b = 2.0 + np.random.default_rng(seed).uniform(0.0, 0.1, 2)
        b -= 1.0
        n = case["n"]

        def mul(x):
            y = a * x
            y[:-1] += b * x[1:]
            z = a * y
            z[1:] += b * y[:-1]
            return z
    elif kind == "design":
        Xt = _to_torch(_design(case["rows"], case["cols"], case["row"], seed))
        X = Xt.to_sparse_coo().T.coalesce().to_sparse_csr()
        n, shift, mul = case["cols"], 0.5, lambda x: Xt @ (X @ x)
    else:
        A = _grid(case["nx"], case["ny"], case["dtype"], seed) \
            if kind == "grid" else \
            _correlation(case["n"], case["row"], case["dtype"], seed)
        M = _to_torch(A)
        n, mul = A.shape[0], lambda x: M @ x
        if case.get("sweep"):
            t = _sweep(case).astype(case["dtype"]).astype(np.float64)
    s = _lanczos_samples(mul, n, case, seed, t, shift)
    used = _used(s[:, 0], opts) if opts["error_rtol"] else len(s)
    s[used:] = np.nan
    return {"value": None, "error": None,
            "samples": s if case.get("sweep") else s[:, 0], "used": None}
