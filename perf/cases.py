"""The library's work, as programs that use it call it: what each case stands for, its inputs, one pass
through the public entry points, and the same result in 64 bits.

Every LP is in the standard form of ``lpgen.StdLP``: A x (<= | =) b, l <= x <= u.  Solves run to a cap
on the iterations (a full solve takes thousands to a hundred thousand of the same iterations); the caps
are multiples of the check cadence, so a pass ends on a restart check as a full solve does.  An answer
of a mixed-precision solve is kept in single precision, one of an FP64 solve in double.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

b2p = importlib.import_module("mangalore-refinery-and-petrochemicals-limited_b200")

PARAM_SEED = 7
_family = None


def family():
    """The parametric refinery planning LP (2000 x 8000, one fixed structure)."""
    global _family
    if _family is None:
        _family = b2p.lpgen.RefineryPlanningFamily()
    return _family


def listed():
    return [
        # the GpuBackend primitives on one small LP's data: A x, A^T y, axpy, dot, norm (a host
        # program that uses the GPU for single operations)
        dict(name="backend_small", kind="backend", m=300, n=1000, k=5),
        # the drop-in's default: the reference PDHG, iterate for iterate, on an LP that arrives with
        # the call (upload and solve)
        dict(name="reference_small", kind="reference", m=300, n=1000, k=5, iterations=2000),
        # the same on a larger LP of odd size
        dict(name="reference_mid", kind="reference", m=20011, n=60013, k=8, iterations=1000),
        # one small LP through the Halpern engine, upload and solve
        dict(name="single_small_fp64", kind="single", shape="random", m=300, n=1000, k=5, precision="fp64",
             iterations=4096, upload=True),
        # the multi-period blending LP at its full size, mixed precision
        dict(name="single_block_mixed", kind="single", shape="block", periods=50, rows=4000, cols=20000, k=8,
             link=4000, precision="fp32", iterations=2048, upload=False),
        # a large LP without structure, plain FP64
        dict(name="single_random_fp64", kind="single", shape="random", m=100003, n=400009, k=10, precision="fp64",
             iterations=1024, upload=False),
        # branch-and-bound: the relaxations of the open nodes, one matrix, the bounds differ
        dict(name="nodes_fp64", kind="nodes", m=100, n=251, k=4, count=48, precision="fp64", iterations=8192),
        # independent LPs of uneven size, each with its own matrix
        dict(name="uneven_mixed", kind="uneven", count=1024, m_lo=50, m_hi=2000, precision="fp32", iterations=1024),
        # the planning family: a thousand scenarios of one matrix, mixed precision
        dict(name="planning_mixed", kind="planning", count=1024, precision="fp32", iterations=2048, check_every=256),
        # the same in plain FP64 (the comparison the benchmark makes)
        dict(name="planning_fp64", kind="planning", count=500, precision="fp64", iterations=1024, check_every=256),
        # new scenarios from the host: upload, predicted warm start, mixed solve, answers
        dict(name="planning_learned", kind="learned", count=400, iterations=512, check_every=256),
        # training of the warm-start network on the labels of a solved batch
        dict(name="mlp_train", kind="train", count=2000, batch=1024, epochs=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["backend", "reference", "small", "block", "random", "nodes", "uneven", "planning", "learned",
                       "train"])
    if kind == "backend":
        m = _log(rng, 40, 4000)
        return dict(kind="backend", m=m, n=int(m * rng.uniform(2, 5)), k=rng.randint(4, 10))
    if kind == "reference":
        m = _log(rng, 60, 20000)
        return dict(kind="reference", m=m, n=int(m * rng.uniform(2, 3)), k=rng.randint(4, 8),
                    iterations=rng.choice([300, 500, 1000]))
    if kind == "small":
        m = _log(rng, 60, 3000)
        return dict(kind="single", shape="random", m=m, n=int(m * rng.uniform(2, 5)), k=rng.randint(4, 8),
                    precision=rng.choice(["fp64", "fp32"]), iterations=64 * rng.randint(8, 32), upload=True)
    if kind == "block":
        p = rng.randint(5, 50)
        return dict(kind="single", shape="block", periods=p, rows=rng.randint(1000, 4000),
                    cols=rng.randint(5000, 20000), k=rng.randint(4, 8), link=p * rng.randint(4, 80),
                    precision=rng.choice(["fp32", "fp32", "fp64"]), iterations=64 * rng.randint(8, 16), upload=False)
    if kind == "random":
        m = _log(rng, 4000, 100000)
        return dict(kind="single", shape="random", m=m, n=int(m * rng.uniform(2, 4)), k=rng.randint(4, 10),
                    precision=rng.choice(["fp64", "fp32"]), iterations=64 * rng.randint(8, 16), upload=False)
    if kind == "nodes":
        m = _log(rng, 30, 300)
        return dict(kind="nodes", m=m, n=int(m * rng.uniform(2, 4)), k=rng.randint(3, 6), count=_log(rng, 4, 300),
                    precision=rng.choice(["fp64", "fp32"]), iterations=64 * rng.randint(8, 64))
    if kind == "uneven":
        return dict(kind="uneven", count=_log(rng, 64, 1024), m_lo=50, m_hi=_log(rng, 200, 2000),
                    precision=rng.choice(["fp32", "fp64"]), iterations=64 * rng.randint(4, 16))
    if kind == "planning":
        return dict(kind="planning", count=_log(rng, 60, 1024), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    iterations=256 * rng.randint(1, 4), check_every=rng.choice([64, 256]))
    if kind == "learned":
        return dict(kind="learned", count=_log(rng, 60, 400), iterations=256 * rng.randint(1, 2),
                    check_every=rng.choice([64, 256]))
    return dict(kind="train", count=_log(rng, 250, 2000), batch=rng.choice([256, 512, 1024]), epochs=rng.randint(2, 8))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _signs(g, n):
    return torch.randint(0, 2, (n,), generator=g, device="cuda").double() * 2 - 1


def _csr(m, n, rows, cols):
    """Sorted distinct entries of a pattern: row pointers, rows and columns."""
    key = torch.unique(rows.long() * n + cols.long())
    r, c = key // n, key % n
    ptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=m), 0)
    return ptr, r, c


def _lp(g, m, n, ptr, r, c, vals, lb, ub, cost, eq):
    """Feasible by construction: b = A x0, plus slack on the <= rows."""
    x0 = lb + (ub - lb) * _uniform(g, n, 0.0, 1.0) * 0.1
    ax0 = np.bincount(r.cpu().numpy(), weights=(vals * x0[c]).cpu().numpy(), minlength=m)  # one fixed order
    b = torch.from_numpy(ax0).cuda()
    b += torch.where(eq, torch.zeros_like(b), _uniform(g, m, 0.0, 1.0))
    h = lambda t, d: np.ascontiguousarray(t.cpu().numpy().astype(d))  # noqa: E731
    return b2p.lpgen.StdLP(m, n, h(ptr, np.int32), h(c, np.int32), h(vals, np.float64), h(b, np.float64),
                           h(cost, np.float64), h(lb, np.float64), h(ub, np.float64), h(eq, np.uint8))


def _random_lp(g, m, n, k):
    """About k entries per column at uniform rows, values +-U(0.1, 10), half the rows equalities."""
    rows = torch.randint(0, m, (n * k,), generator=g, device="cuda")
    cols = torch.arange(n, device="cuda").repeat_interleave(k)
    ptr, r, c = _csr(m, n, rows, cols)
    vals = _uniform(g, r.numel(), 0.1, 10.0) * _signs(g, r.numel())
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    return _lp(g, m, n, ptr, r, c, vals, zero, zero + 10.0, _uniform(g, n, -1.0, 1.0),
               torch.arange(m, device="cuda") % 2 == 0)


def _block_lp(g, periods, rows, cols, k, link):
    """Period blocks, linked by inventory balances x_t - x_{t-1} + flows = d_t."""
    m, n, items = periods * rows + link, periods * cols, link // periods
    col = torch.arange(n, device="cuda").repeat_interleave(k)
    row = torch.randint(0, rows, (n * k,), generator=g, device="cuda") + (col // cols) * rows
    i = torch.arange(link, device="cuda")
    item, t = i % items, (i // items).clamp(max=periods - 1)
    flow = t[:, None] * cols + items + torch.randint(0, cols - items, (link, 3), generator=g, device="cuda")
    lr = periods * rows + i
    back = t > 0
    r = torch.cat([row, lr, lr[back], lr.repeat_interleave(3)])
    c = torch.cat([col, t * cols + item, ((t - 1) * cols + item)[back], flow.reshape(-1)])
    ptr, r, c = _csr(m, n, r, c)
    vals = torch.exp(torch.randn(r.numel(), generator=g, device="cuda", dtype=torch.float64)) * _signs(g, r.numel())
    ub = _uniform(g, n, 1.0, 100.0)
    eq = (torch.arange(m, device="cuda") % 3 == 2) | (torch.arange(m, device="cuda") >= periods * rows)
    cost = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return _lp(g, m, n, ptr, r, c, vals, torch.zeros_like(ub), ub, cost, eq)


def _uneven(g, count, m_lo, m_hi):
    """Independent LPs, m ~ logU(m_lo, m_hi), n = m U(2, 5), 4-10 entries per column, made in one go."""
    rng = np.random.default_rng(count)  # the sizes belong to the case, the data to the seed
    ms = np.exp(rng.uniform(math.log(m_lo), math.log(m_hi), count)).astype(np.int64)
    ns = (ms * rng.uniform(2.0, 5.0, count)).astype(np.int64)
    ro, co = np.concatenate([[0], np.cumsum(ms)]), np.concatenate([[0], np.cumsum(ns)])
    M, N = int(ro[-1]), int(co[-1])
    inst = torch.from_numpy(np.repeat(np.arange(count), ns)).cuda()
    kc = torch.randint(4, 11, (N,), generator=g, device="cuda")
    col = torch.arange(N, device="cuda").repeat_interleave(kc)
    dm, dro = torch.from_numpy(ms).cuda(), torch.from_numpy(ro).cuda()
    who = inst[col]
    row = dro[who] + (_uniform(g, col.numel(), 0.0, 1.0) * dm[who]).long()
    ptr, r, c = _csr(M, N, row, col)
    vals = _uniform(g, r.numel(), 0.1, 10.0) * _signs(g, r.numel())
    zero = torch.zeros(N, dtype=torch.float64, device="cuda")
    eq = torch.from_numpy(np.concatenate([np.arange(v) % 2 == 0 for v in ms])).cuda()
    return _lp(g, M, N, ptr, r, c, vals, zero, zero + 10.0, _uniform(g, N, -1.0, 1.0), eq), ro, co


def _batch_inputs(case, seed):
    """(mats, inst_mat, b, c, lb, ub, is_eq) of batch_upload."""
    kind = case["kind"]
    if kind == "uneven":
        lp, ro, co = _uneven(_gen(seed), case["count"], case["m_lo"], case["m_hi"])
        mats = []
        for i in range(case["count"]):
            e0, e1 = lp.rowptr[ro[i]], lp.rowptr[ro[i + 1]]
            mats.append((int(ro[i + 1] - ro[i]), int(co[i + 1] - co[i]), lp.rowptr[ro[i]:ro[i + 1] + 1] - e0,
                         lp.colidx[e0:e1] - np.int32(co[i]), lp.vals[e0:e1]))
        return mats, np.arange(case["count"], dtype=np.int32), lp.b, lp.c, lp.lb, lp.ub, lp.is_eq
    cnt = case["count"]
    if kind == "nodes":
        lp = _random_lp(_gen(seed), case["m"], case["n"], case["k"])
        rng = np.random.default_rng(seed)
        lb, ub = np.tile(lp.lb, (cnt, 1)), np.tile(lp.ub, (cnt, 1))
        for i in range(1, cnt):  # a node has up to four branched columns, each within a unit of x0's range
            j = rng.integers(0, lp.n, 4)
            ub[i, j] = rng.integers(2, 10, 4)
        return ([(lp.m, lp.n, lp.rowptr, lp.colidx, lp.vals)], np.zeros(cnt, np.int32), np.tile(lp.b, cnt),
                np.tile(lp.c, cnt), lb.ravel(), ub.ravel(), np.tile(lp.is_eq, cnt))
    P = family().sample_params(cnt, 1000 + seed)
    s0, B, C, LB, UB, EQ = family().standard_batch(P)
    return ([(s0.m, s0.n, s0.rowptr, s0.colidx, s0.vals)], np.zeros(cnt, np.int32), B.ravel(), C.ravel(), LB.ravel(),
            UB.ravel(), EQ.ravel().astype(np.uint8))


def _weights(g, hidden, out):
    """Parameters of the 256 -> hidden -> hidden -> out network, as b2p_mlp_set_params takes them."""
    parts = []
    for fan_in, rows in ((256, hidden), (hidden, hidden), (hidden, out)):
        a = 1.0 / math.sqrt(fan_in)
        parts += [_uniform(g, rows * fan_in, -a, a), _uniform(g, rows, -a, a)]
    return torch.cat(parts).float().cpu().numpy()


def _single_lp(case, seed):
    g = _gen(seed)
    if case.get("shape") == "block":
        return _block_lp(g, case["periods"], case["rows"], case["cols"], case["k"], case["link"])
    return _random_lp(g, case["m"], case["n"], case["k"])


def prepare(case, seed):
    kind = case["kind"]
    ctx = b2p.Context(0)
    s = dict(case=case, ctx=ctx)
    if kind in ("backend", "reference", "single"):
        s["lp"] = lp = _single_lp(case, seed)
        if kind == "backend":
            rng = np.random.default_rng(seed)
            s["x"], s["x2"], s["y"] = rng.standard_normal(lp.n), rng.standard_normal(lp.n), rng.standard_normal(lp.m)
        elif not case.get("upload", True):
            ctx.upload(lp)
        return s
    s["inputs"] = _batch_inputs(dict(case, kind="planning") if kind in ("learned", "train") else case, seed)
    if kind in ("learned", "train"):
        f = family()
        s["features"] = f.sample_params(case["count"], 1000 + seed).astype(np.float32)
        ctx.mlp_create(256, 1024, f.n + f.m + 1, seed=PARAM_SEED)
    if kind == "learned":  # a trained model: weights and normalisation of its data set
        ctx.mlp_set_params(_weights(_gen(PARAM_SEED), 1024, f.n + f.m + 1))
        mid = np.concatenate([0.02 * f.ub, np.zeros(f.m), [0.0]]).astype(np.float32)
        std = np.concatenate([np.full(f.n, 2.0), np.full(f.m, 10.0), [0.2]]).astype(np.float32)
        ctx.mlp_set_normalization(np.ones(256, np.float32), np.full(256, 0.15, np.float32), mid, std)
    if kind in ("uneven", "planning", "train"):
        ctx.batch_upload(*s["inputs"])
    if kind == "train":  # labels: the answers of a solved batch, kept on the device
        ctx.batch_solve(precision="fp32", max_iterations=256, check_every=256, outputs=False)
        ctx.mlp_dataset_from_batch(s["features"])
    return s


# ------------------------------------------------------------------ one pass
def _answers(case, x, y, iterations):
    if case.get("precision", "fp32") == "fp32":
        x, y = x.astype(np.float32), y.astype(np.float32)
    return dict(x=x, y=y, iterations=iterations)


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "backend":
        lp = s["lp"]
        ax, _ = ctx.spmv(lp.m, lp.n, lp.rowptr, lp.colidx, lp.vals, s["x"])
        aty, _ = ctx.spmv(lp.m, lp.n, lp.rowptr, lp.colidx, lp.vals, s["y"], transpose=True)
        return dict(ax=ax, aty=aty, axpy=ctx.vector_op("axpy", s["x"], s["x2"], alpha=0.37),
                    dot=ctx.dot(s["x"], s["x2"]), norm=ctx.norm2(s["y"]))
    if kind == "reference":
        ctx.upload(s["lp"])
        r, x, y = ctx.solve(engine="reference", max_iterations=case["iterations"])
        return dict(x=x, y=y, iterations=r["iterations"], used_average=r["used_average"])
    if kind == "single":
        if case["upload"]:
            ctx.upload(s["lp"])
        r, x, y = ctx.solve(engine="halpern", precision=case["precision"], eps=1e-6,
                            max_iterations=case["iterations"])
        return _answers(case, x, y, r["iterations"])
    if kind == "nodes":
        ctx.batch_upload(*s["inputs"])
        _, per, x, y = ctx.batch_solve(precision=case["precision"], eps=1e-6, max_iterations=case["iterations"])
        return _answers(case, x, y, per["iterations"])
    if kind in ("uneven", "planning"):
        _, per, x, y = ctx.batch_solve(precision=case["precision"], eps=1e-6, eps_objective=1e-6,
                                       check_every=case.get("check_every", 64), max_iterations=case["iterations"])
        return _answers(case, x, y, per["iterations"])
    if kind == "learned":
        ctx.batch_upload(*s["inputs"])
        _, per, x, y = ctx.batch_solve_learned(s["features"], eps=1e-6, eps_objective=1e-6,
                                               check_every=case["check_every"], max_iterations=case["iterations"])
        return _answers(case, x, y, per["iterations"])
    loss = ctx.mlp_train(case["epochs"], batch=case["batch"], lr_start=2e-3, lr_end=2e-5, seed=3)
    return dict(loss=np.float32(loss), params=ctx.mlp_get_params())


# ------------------------------------------------------------------ what one pass cannot do without
def _sizes(case):
    """(rows, columns, nonzeros, matrix entries) over all LPs of the case; expected values where drawn."""
    kind = case["kind"]
    if kind in ("learned", "planning", "train"):
        c = case["count"]
        return 2000 * c, 8000 * c, 47984 * c, 47984
    if kind == "nodes":
        return case["m"] * case["count"], case["n"] * case["count"], case["n"] * case["k"] * case["count"], case["n"] * case["k"]
    if kind == "uneven":
        mean = (case["m_hi"] - case["m_lo"]) / math.log(case["m_hi"] / case["m_lo"])
        m, n = mean * case["count"], 3.5 * mean * case["count"]
        return m, n, 7 * n, 7 * n
    if case.get("shape") == "block":
        n = case["periods"] * case["cols"]
        return case["periods"] * case["rows"] + case["link"], n, n * case["k"] + 5 * case["link"], n * case["k"] + 5 * case["link"]
    return case["m"], case["n"], case["n"] * case["k"], case["n"] * case["k"]


def work(case):
    m, n, nnz, own = _sizes(case)
    if case["kind"] == "backend":
        return dict(bytes=12.0 * 2 * nnz + 8.0 * (4 * n + 3 * m), flops=4.0 * nnz + 4 * n + 2 * m)
    if case["kind"] == "train":
        steps = case["epochs"] * case["count"]
        params = 256 * 1024 + 1024 * 1024 + 1024 * 10001
        per_epoch = -(-case["count"] // case["batch"])
        return dict(bytes=4.0 * steps * (256 + 10001) + 32.0 * params * case["epochs"] * per_epoch,
                    flops=6.0 * steps * params)
    # every input and answer once; the iterations' multiply-adds and vector updates
    return dict(bytes=12.0 * own + 8.0 * (4 * n + 2 * m), flops=case["iterations"] * (4.0 * nnz + 14.0 * n + 9.0 * m))


# ------------------------------------------------------------------ the same in 64 bits
def _sparse(m, n, rowptr, colidx, vals):
    A = torch.sparse_csr_tensor(torch.as_tensor(rowptr).long(), torch.as_tensor(colidx).long(),
                                torch.as_tensor(vals), (m, n), device="cuda")
    return A, A.to_sparse_coo().t().coalesce().to_sparse_csr()


def _exact_reference(lp, iterations):
    A, At = _sparse(lp.m, lp.n, lp.rowptr, lp.colidx, lp.vals)
    b, c, lb, ub = (torch.from_numpy(v).cuda() for v in (lp.b, lp.c, lp.lb, lp.ub))
    eq = torch.from_numpy(lp.is_eq).cuda().bool()
    absA, absAt = _sparse(lp.m, lp.n, lp.rowptr, lp.colidx, np.abs(lp.vals))
    step = lambda s: torch.where(s > 1e-12, 0.95 / s, torch.ones_like(s))  # noqa: E731
    tau, sigma = step(absAt @ torch.ones_like(b)), step(absA @ torch.ones_like(c))
    x, y, total = 0.5 * (lb + ub), torch.zeros_like(b), torch.zeros_like(c)
    for _ in range(iterations):
        xn = torch.minimum(torch.maximum(x - tau * (c + At @ y), lb), ub)
        y = y + sigma * (A @ (2 * xn - x) - b)
        y = torch.where(eq, y, y.clamp(min=0.0))
        x = xn
        total += x
    avg = torch.minimum(torch.maximum(total / iterations, lb), ub)
    viol = lambda v: float(torch.where(eq, (A @ v - b).abs(), (A @ v - b).clamp(min=0.0)).max())  # noqa: E731
    used = viol(avg) <= viol(x)
    return dict(x=(avg if used else x).cpu().numpy(), y=y.cpu().numpy(), iterations=None, used_average=None)


def _start_vector(n):
    """Entries in (0.5, 1.5) from a splitmix64 stream, the power iteration's start."""
    with np.errstate(over="ignore"):
        z = np.arange(n, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0x1234567)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return 0.5 + (z >> np.uint64(11)).astype(np.float64) / 9007199254740992.0


def _exact_halpern(mats, inst_mat, b, c, lb, ub, is_eq, iterations, K, window, eps=1e-6, eps_obj=0.0):
    """Restarted Halpern PDHG of every instance in 64 bits: vectors are [dimension, instances] over one
    matrix, or [all dimensions, 1] over the block-diagonal matrix of several.  window: 0 for a batch
    (columns numbered by length, power iteration stopped at every step), else the length-sort window of
    the single-LP engine (power iteration looked at every 16 steps)."""
    cuda = lambda v, d=torch.float64: torch.as_tensor(np.asarray(v)).cuda().to(d)  # noqa: E731
    nm, cnt = len(mats), len(inst_mat)
    shared = nm == 1
    ms, ns = np.array([q[0] for q in mats]), np.array([q[1] for q in mats])
    ro, co = np.concatenate([[0], np.cumsum(ms)]), np.concatenate([[0], np.cumsum(ns)])
    M, N = int(ro[-1]), int(co[-1])
    nnz = np.concatenate([[0], np.cumsum([len(q[4]) for q in mats])])
    ptr = np.concatenate([np.asarray(q[2][:-1], np.int64) + nnz[i] for i, q in enumerate(mats)] + [nnz[-1:]])
    idx = np.concatenate([np.asarray(q[3], np.int64) + co[i] for i, q in enumerate(mats)])
    val = cuda(np.concatenate([q[4] for q in mats]))
    rowid, colid = cuda(np.repeat(np.arange(M), np.diff(ptr)), torch.int64), cuda(idx, torch.int64)
    cmat, rmat = cuda(np.repeat(np.arange(nm), ns), torch.int64), cuda(np.repeat(np.arange(nm), ms), torch.int64)
    # Ruiz and Pock-Chambolle scaling
    dr, dc = torch.ones(M, device="cuda", dtype=torch.float64), torch.ones(N, device="cuda", dtype=torch.float64)
    for p in range(11):
        a = val.abs() * dr[rowid] * dc[colid]
        how = "amax" if p < 10 else "sum"
        r = torch.zeros_like(dr).scatter_reduce_(0, rowid, a, how)
        q = torch.zeros_like(dc).scatter_reduce_(0, colid, a, how)
        dr, dc = torch.where(r > 0, dr / r.sqrt(), dr), torch.where(q > 0, dc / q.sqrt(), dc)
    A, At = _sparse(M, N, ptr, idx, val * dr[rowid] * dc[colid])
    # largest singular value of every matrix, from the same start and with the same stop
    clen = np.bincount(idx, minlength=N)
    start = np.empty(N)
    for k in range(nm):
        cl, n = clen[co[k]:co[k + 1]], int(ns[k])
        order = np.lexsort((np.arange(n), -cl, np.arange(n) // window if window else np.zeros(n)))
        start[co[k] + order] = _start_vector(n)
    v = cuda(start)
    per_mat = lambda w: torch.zeros(nm, device="cuda", dtype=torch.float64).index_add_(0, cmat, w)  # noqa: E731
    norm, sig2 = per_mat(v * v).sqrt(), torch.zeros(nm, device="cuda", dtype=torch.float64)
    open_ = torch.ones(nm, device="cuda", dtype=torch.bool)
    for t in range(512 if window else 1000):
        w = At @ ((A @ v) / norm[rmat])
        nn = per_mat(w * w).sqrt()
        settled = (nn - sig2).abs() <= 1e-7 * nn
        v, norm = torch.where(open_[cmat], w, v), torch.where(open_, nn, norm)
        sig2 = torch.where(open_, nn, sig2)
        if not window or t % 16 == 15:
            open_ &= ~settled
            if not bool(open_.any()):
                break
    eta = 0.998 / sig2.sqrt()
    # vectors and per-instance scalars
    if shared:
        col = lambda v: cuda(v).reshape(cnt, N).t().contiguous()  # noqa: E731
        row = lambda v, d=torch.float64: cuda(v, d).reshape(cnt, M).t().contiguous()  # noqa: E731
        dcol, drow = dc[:, None], dr[:, None]
        tot_c = tot_r = lambda w: w.sum(0)  # noqa: E731
        on_c = on_r = lambda w: w[None, :]  # noqa: E731
        eta = eta.expand(cnt)
    else:
        col = lambda v: cuda(v)[:, None]  # noqa: E731
        row = lambda v, d=torch.float64: cuda(v, d)[:, None]  # noqa: E731
        dcol, drow = dc[:, None], dr[:, None]
        tot_c = lambda w: torch.zeros(cnt, device="cuda", dtype=torch.float64).index_add_(0, cmat, w[:, 0])  # noqa: E731
        tot_r = lambda w: torch.zeros(cnt, device="cuda", dtype=torch.float64).index_add_(0, rmat, w[:, 0])  # noqa: E731
        on_c, on_r = lambda w: w[cmat][:, None], lambda w: w[rmat][:, None]  # noqa: E731
    ob, oc, ol, ou, eq = row(b), col(c), col(lb), col(ub), row(is_eq, torch.bool)
    sb, sc, sl, su = ob * drow, oc * dcol, ol / dcol, ou / dcol
    low = torch.where(eq, -torch.inf, 0.0).double()
    bn, cn = tot_r(ob * ob).sqrt(), tot_c(oc * oc).sqrt()
    om = tot_c(sc * sc).sqrt() / tot_r(sb * sb).sqrt()
    x = torch.minimum(torch.maximum(torch.zeros_like(sl), sl), su)
    y = torch.zeros_like(sb)
    xa, ya, xr, yr = x, y, x, y
    kk = torch.zeros(cnt, device="cuda", dtype=torch.float64)
    r0, rprev, its = torch.zeros_like(kk), torch.zeros_like(kk), torch.zeros_like(kk)
    first, done = torch.ones_like(kk, dtype=torch.bool), torch.zeros_like(kk, dtype=torch.bool)
    for it in range(iterations):
        tau, sigma = on_c(eta / om), on_r(eta * om)
        xt = torch.minimum(torch.maximum(x - tau * (sc + At @ y), sl), su)
        yt = torch.maximum(y + sigma * (A @ (2 * xt - x) - sb), low)
        if it % K == 0 or it % K == K - 1:
            res = (om * tot_c((x - xt) ** 2) + tot_r((y - yt) ** 2) / om).sqrt()
            r0, rprev = torch.where(first, res, r0), torch.where(first, res, rprev)
            first = torch.zeros_like(first)
        wk, wa = (kk + 1) / (kk + 2), 1 / (kk + 2)
        x = on_c(wk) * (2 * xt - x) + on_c(wa) * xa
        y = on_r(wk) * (2 * yt - y) + on_r(wa) * ya
        kk = kk + 1
        if it % K != K - 1:
            continue
        live = ~done
        lc, lr = on_c(live), on_r(live)
        xr, yr = torch.where(lc, xt, xr), torch.where(lr, yt, yr)
        its = torch.where(live, torch.full_like(its, it + 1), its)
        # relative KKT and the objective-error bound on the original LP
        px, py = dcol * xt, drow * yt
        rp = (A @ xt) / drow - ob
        rp = torch.where(eq, rp, rp.clamp(min=0.0))
        g = oc + (At @ yt) / dcol
        p, d = tot_c(oc * px), -tot_r(ob * py) + tot_c(torch.where(g > 0, g * ol, g * ou))
        ok = (tot_r(rp * rp).sqrt() <= eps * (1 + bn)) & ((p - d).abs() <= eps * (1 + p.abs() + d.abs()))
        if eps_obj > 0:
            err = torch.maximum((p - d).clamp(min=0.0), tot_r(py.abs() * rp.abs()))
            ok &= err <= eps_obj * p.abs().clamp(min=1.0)
        done |= ok
        again = ((res <= 0.2 * r0) | ((res <= 0.8 * r0) & (res > rprev)) | (kk >= 0.36 * (it + 1))) & ~done
        rprev = res
        dx, dy = tot_c((xt - xa) ** 2).sqrt(), tot_r((yt - ya) ** 2).sqrt()
        nw = torch.exp(0.5 * torch.log(dy / dx) + 0.5 * torch.log(om))
        om = torch.where(again & (dx > 1e-10) & (dy > 1e-10) & torch.isfinite(nw), nw, om)
        x, xa = torch.where(on_c(again), xt, x), torch.where(on_c(again), xt, xa)
        y, ya = torch.where(on_r(again), yt, y), torch.where(on_r(again), yt, ya)
        kk = torch.where(again, torch.zeros_like(kk), kk)
        first = again
        if bool(done.all()):
            break
    flat = lambda t: t.t().reshape(-1).cpu().numpy()  # noqa: E731
    return dict(x=flat(dcol * xr), y=flat(drow * yr), iterations=None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "backend":
        lp = _single_lp(case, seed)
        rng = np.random.default_rng(seed)
        x, x2, y = rng.standard_normal(lp.n), rng.standard_normal(lp.n), rng.standard_normal(lp.m)
        return dict(ax=lp.spmv(x), aty=lp.spmv_t(y), axpy=0.37 * x + x2, dot=float(x @ x2), norm=float(np.sqrt(y @ y)))
    if kind == "reference":
        return _exact_reference(_single_lp(case, seed), case["iterations"])
    if kind == "single":
        lp = _single_lp(case, seed)
        return _exact_halpern([(lp.m, lp.n, lp.rowptr, lp.colidx, lp.vals)], [0], lp.b, lp.c, lp.lb, lp.ub, lp.is_eq,
                              case["iterations"], 64, 4096)
    if kind in ("nodes", "uneven", "planning"):
        return _exact_halpern(*_batch_inputs(case, seed), case["iterations"], case.get("check_every", 64), 0,
                              eps_obj=0.0 if kind == "nodes" else 1e-6)
    return None  # a 16-bit network: what follows from it has no value of its own in 64 bits
