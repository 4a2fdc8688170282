"""Workloads the framework's speed is measured on: what its users have it do, through its public entry points.

A case is a dict of plain values. `kind` names the entry point and `lp` the family of the model:

  spmv    SpmvPlan.run                y = A x on a matrix resident on the device (FP32 and FP64)
  solve   pdhg.solve                  one LP from host arrays to its answer, within an iteration budget
  engine  Engine.solve                the same on a resident context: the driver's power iteration, iterations,
                                      evaluations, restarts and the download of the point
  steps   Engine.start / iterate / eval_pair / restart / download: a caller's own driver on a resident context
  batch   Batch.solve                 many LPs together, per-instance restarts on the device
  predict Mlp.forward                 the warm start's network, host arrays in and out
  train   Mlp.set_params / train      Adam steps of that network; returns the loss and the updated weights

Model families (lpgen): planted (uniform-random rows), zipf (power-law row lengths), general (every row and bound
kind), packing, refinery (multi-period, rows of 40-110 nonzeros). Points of FP32 contexts are returned as float32, the
precision the context holds them in (and the one the network is trained on).
"""
import dataclasses
import functools
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parents[1] / "taral-lp_b200"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))
import lpgen  # noqa: E402
import pdhg  # noqa: E402

FREQ = 64  # iterations between evaluations, the solver's default
ZIPF = dict(zipf=1.2, cap=2000, floor=5)


def listed():
    return [
        # the smallest call: one product with the small planted LP's matrix, where a launch is all there is
        dict(name="spmv_small_fp64", kind="spmv", lp="planted", m=2000, n=5000, per_col=5, fp32=False),
        # the benchmark LP's matrix: 5M nonzeros, power-law rows, random gathers
        dict(name="spmv_zipf_fp32", kind="spmv", lp="zipf", m=200_000, n=500_000, per_col=10, fp32=True),
        # medium rows (40-110 nonzeros) in double: a multi-period model of 12 periods
        dict(name="spmv_refinery_fp64", kind="spmv", lp="refinery", periods=12, fp32=False),
        # one small LP from host arrays, as a caller with a stream of LPs sends them
        dict(name="solve_small_fp64", kind="solve", lp="planted", m=2000, n=5000, per_col=5, fp32=False, iters=1024),
        # a small mixed LP with every row and bound kind, odd sizes
        dict(name="solve_general_fp32", kind="solve", lp="general", m=307, n=701, per_col=4, fp32=True, iters=1024),
        # a medium multi-period LP on a resident context
        dict(name="engine_refinery8_fp32", kind="engine", lp="refinery", periods=8, fp32=True, iters=1024),
        # the benchmark LP, driven block by block
        dict(name="steps_zipf_fp32", kind="steps", lp="zipf", m=200_000, n=500_000, per_col=10, fp32=True, iters=512),
        # the largest multi-period LP in double precision
        dict(name="engine_refinery48_fp64", kind="engine", lp="refinery", periods=48, fp32=False, iters=256),
        # a scenario family of uneven sizes, matrices shared by the scenarios of one length
        dict(name="batch_family_fp32", kind="batch", lp="refinery", periods=12, count=48, fp32=True, iters=256),
        # many small LPs, every matrix its own
        dict(name="batch_small_fp64", kind="batch", lp="general", m=151, n=347, per_col=4, count=40, fp32=False,
             iters=320),
        # the warm start's prediction for a chunk of scenarios of 24 periods (36,000 rows + 96,000 columns + 1)
        dict(name="predict_24_periods", kind="predict", in_dim=256, hidden=512, depth=3, out=132_001, batch=128),
        # its training step, 64 scenarios a batch
        dict(name="train_24_periods", kind="train", in_dim=256, hidden=512, depth=3, out=132_001, batch=64, count=64,
             steps=48),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_lp(rng, lo, hi, periods):
    fam = rng.choice(["planted", "zipf", "general", "packing", "refinery", "refinery"])
    if fam == "refinery":
        return dict(lp=fam, periods=rng.randint(1, periods))
    n = _log(rng, lo, hi)
    if fam == "packing":
        return dict(lp=fam, n=n)
    return dict(lp=fam, m=max(20, int(n * rng.uniform(0.3, 0.6))), n=n, per_col=rng.randint(3, 10))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "solve", "engine", "steps", "batch", "batch", "predict", "train"])
    fp32 = rng.random() < 0.5
    if kind == "spmv":
        return dict(kind=kind, fp32=fp32, **_draw_lp(rng, 300, 500_000, 24))
    if kind == "solve":
        return dict(kind=kind, fp32=fp32, iters=FREQ * rng.randint(4, 16), **_draw_lp(rng, 300, 60_000, 4))
    if kind in ("engine", "steps"):
        return dict(kind=kind, fp32=fp32, iters=FREQ * rng.randint(2, 8), **_draw_lp(rng, 700, 400_000, 40))
    if kind == "batch":
        if rng.random() < 0.5:
            return dict(kind=kind, lp="refinery", periods=rng.randint(1, 12), count=rng.randint(3, 48), fp32=fp32,
                        iters=FREQ * rng.randint(1, 4))
        n = _log(rng, 120, 4000)
        return dict(kind=kind, lp=rng.choice(["general", "planted"]), m=int(n * rng.uniform(0.3, 0.6)), n=n,
                    per_col=rng.randint(3, 8), count=rng.randint(3, 40), fp32=fp32, iters=FREQ * rng.randint(1, 5))
    size = dict(in_dim=256, hidden=64 * rng.randint(2, 8), depth=rng.randint(1, 3), out=_log(rng, 900, 132_001))
    if kind == "predict":
        return dict(kind=kind, batch=_log(rng, 1, 256), **size)
    batch = 8 * rng.randint(2, 8)
    return dict(kind=kind, batch=batch, count=batch * rng.choice([1, 1, 2]), steps=rng.randint(16, 48), **size)


# ------------------------------------------------------------------------------------------------ models
@functools.lru_cache(maxsize=4)
def _structure(lp, m, n, per_col):
    """The sparsity of a random family's model (drawn once; values and vectors come from the seed)."""
    return lpgen.planted(m, n, per_col, seed=m + n, **(ZIPF if lp == "zipf" else {}))


@functools.lru_cache(maxsize=4)
def _refinery(periods):
    return lpgen.RefineryBase(periods, seed=7)


def _planted(lp, m, n, per_col, seed):
    """lpgen.planted's construction on a cached sparsity: values, planted optimum and costs from the seed."""
    if n <= 20_000 and lp == "planted":
        return lpgen.planted(m, n, per_col, seed=seed)
    base = _structure(lp, m, n, per_col)
    rng = np.random.default_rng(seed)
    val = rng.standard_normal(len(base.val))
    cols = np.repeat(np.arange(n), np.diff(base.col_ptr))
    u = rng.random(n)
    x = np.where(u < 0.4, 0.0, np.where(u < 0.5, 10.0, rng.uniform(0.5, 9.5, n)))
    y, mag = rng.standard_normal(m), rng.uniform(0.1, 1.0, n)
    b = np.bincount(base.row_idx, weights=val * x[cols], minlength=m)
    c = np.bincount(cols, weights=val * y[base.row_idx], minlength=n)
    c += np.where(u < 0.4, mag, np.where(u < 0.5, -mag, 0.0))
    return dataclasses.replace(base, val=val, cost=c, row_lo=b, row_up=b.copy())


def _model(case, seed):
    lp = case["lp"]
    if lp == "refinery":
        return _refinery(case["periods"]).instance(case["periods"], lpgen.perturbations(1, seed)[0])
    if lp == "packing":
        return lpgen.packing(case["n"], seed=seed)
    if lp == "general":
        return lpgen.general(case["m"], case["n"], case["per_col"], seed=seed)
    return _planted(lp, case["m"], case["n"], case["per_col"], seed)


def _models(case, seed):
    """The LPs of a batch: refinery scenarios of 1 .. periods periods, or random LPs of about one size."""
    k = case["count"]
    if case["lp"] == "refinery":
        base, p = _refinery(case["periods"]), lpgen.perturbations(k, seed)
        return [base.instance(1 + (5 * i + 2) % case["periods"], p[i]) for i in range(k)]
    return [_model(dict(case, m=case["m"] + i % 7, n=case["n"] + 3 * (i % 11)), 1000 * seed + i) for i in range(k)]


def _values(case, lp, seed):
    """The matrix values of a product: a family's one matrix gets values of this seed."""
    if case["lp"] != "refinery":
        return lp.val
    return lp.val * np.random.default_rng(seed).uniform(0.5, 1.5, len(lp.val))


def _rows(lp, val):
    """The row-wise copy of a column-wise model: row pointers on the host, indices and values on the device."""
    ptr = torch.zeros(lp.m + 1, dtype=torch.int64)
    rows = torch.from_numpy(np.array(lp.row_idx)).cuda()
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=lp.m), 0).cpu()
    order = torch.sort(rows, stable=True).indices
    cols = torch.from_numpy(np.repeat(np.arange(lp.n, dtype=np.int32), np.diff(lp.col_ptr))).cuda()
    return ptr, cols[order].contiguous(), torch.from_numpy(np.array(val)).cuda()[order].contiguous()


def _sizes(case):
    """(rows, columns, nonzeros) of a case's model or, for a batch, of all its models together."""
    if case["kind"] == "batch" and case["lp"] == "refinery":
        per = [1 + (5 * i + 2) % case["periods"] for i in range(case["count"])]
    else:
        per = [case["periods"]] if case["lp"] == "refinery" else []
    if per:
        return 1500 * sum(per), 4000 * sum(per), 70_800 * sum(per)
    n = case["n"]
    m, nnz = (n // 2, 5 * n) if case["lp"] == "packing" else (case["m"], case["per_col"] * n)
    k = case.get("count", 1)
    return k * m, k * n, k * nnz


def _precision(case):
    return pdhg.FP32 if case["fp32"] else pdhg.FP64


# ------------------------------------------------------------------------------------------------ network
def _net_data(case, seed, rows):
    """A chunk of normalised perturbations and normalised targets, uniform and normal like the family's."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (rows, case["in_dim"])).astype(np.float32) * np.float32(3.0 ** 0.5)
    return x, rng


def _net_params(case, seed):
    """He-initialised weights, small random biases: per layer W (in x out), then b."""
    rng = np.random.default_rng(seed + 1)
    dims = [case["in_dim"]] + [case["hidden"]] * case["depth"] + [case["out"]]
    parts = []
    for i, o in zip(dims[:-1], dims[1:]):
        w = rng.standard_normal(i * o, dtype=np.float32)
        w *= np.float32((2.0 / i) ** 0.5)
        parts += [w, 0.01 * rng.standard_normal(o, dtype=np.float32)]
    return dims, np.concatenate(parts)


# ------------------------------------------------------------------------------------------------ measured calls
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        dims, p = _net_params(case, seed)
        net = pdhg.Mlp(case["in_dim"], case["hidden"], case["depth"], case["out"], max_batch=case["batch"])
        net.set_params(p)
        rows = case["batch"] if kind == "predict" else case["count"]
        x, rng = _net_data(case, seed, rows)
        if kind == "train":
            net.set_dataset(x, rng.standard_normal((rows, case["out"]), dtype=np.float32))
        return dict(case=case, net=net, x=x, seed=seed)
    if kind == "batch":
        b = pdhg.Batch(_models(case, seed), tol=1e-9, max_iter=case["iters"], eval_freq=FREQ,
                       precision=_precision(case))
        return dict(case=case, batch=b)
    lp = _model(case, seed)
    if kind == "spmv":
        dt = torch.float32 if case["fp32"] else torch.float64
        ptr, idx, val = _rows(lp, _values(case, lp, seed))
        g = torch.Generator().manual_seed(seed)
        x = torch.randn(lp.n, dtype=dt, generator=g).cuda()
        plan = pdhg.SpmvPlan(ptr.numpy(), lp.n, _precision(case))
        return dict(case=case, plan=plan, x=x, y=torch.empty(lp.m, dtype=dt, device="cuda"),
                    ptr=ptr.to(torch.int32).cuda(), idx=idx, val=val.to(dt))
    if kind == "solve":
        return dict(case=case, lp=lp)
    e = pdhg.Engine.from_model(lp, precision=_precision(case), eval_freq=FREQ)
    if kind == "steps":  # steps of the size the driver takes, from the operator norm
        tau = 0.95 / e.power_norm(200)
        e.set_steps(tau, tau)
    return dict(case=case, engine=e)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "spmv":
        y = state["y"]
        state["plan"].run(state["ptr"].data_ptr(), state["idx"].data_ptr(), state["val"].data_ptr(),
                          state["x"].data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return y
    if kind == "predict":
        return state["net"].forward(state["x"])
    if kind == "train":
        net = state["net"]
        epochs = max(1, case["steps"] * case["batch"] // case["count"])
        loss = net.train(epochs=epochs, batch=case["batch"], lr=1e-4, seed=state["seed"])
        return [loss, net.get_params()]
    if kind == "batch":
        res, xs, ys = state["batch"].solve()
        return _out(case, [np.concatenate(xs), np.concatenate(ys), np.array([r["objective"] for r in res]),
                           np.array([r["rel_primal"] for r in res])])
    if kind == "solve":
        r, x, y = pdhg.solve(state["lp"], tol=1e-9, max_iter=case["iters"], eval_freq=FREQ,
                             precision=_precision(case))
        return _out(case, [x, y, r["objective"], r["rel_primal"], r["rel_dual"]])
    e = state["engine"]
    if kind == "engine":
        r, x, z = e.solve(e.bnorm, e.cnorm, tol=1e-9, max_iter=case["iters"], eval_freq=FREQ)
        return _out(case, [x, z, r["rel_primal"], r["rel_dual"], r["norm_a"]])
    e.start()
    half = max(1, case["iters"] // FREQ // 2)
    for block in range(1, case["iters"] // FREQ + 1):
        e.iterate(FREQ)
        since = FREQ * (block if block <= half else block - half)
        cur, avg = e.eval_pair(1.0 / since)
        if block == half:  # the driver's restart to the average
            e.restart(True, 1.0 / since)
    x, z = e.download(False, 1.0)
    return _out(case, [x, z, cur, avg])


def _out(case, values):
    """A context's results in the precision it holds its points in."""
    return [np.asarray(v, np.float32) for v in values] if case["fp32"] else values


def work(case):
    """Bytes and operations of a pass. An iteration reads the indices and values of A and of its transpose once and
    reads or writes each state vector once (44 bytes a row and column in FP32, 72 in FP64, running sums in FP64)."""
    kind = case["kind"]
    if kind in ("predict", "train"):
        dims = [case["in_dim"]] + [case["hidden"]] * case["depth"] + [case["out"]]
        weights = sum(i * o for i, o in zip(dims[:-1], dims[1:]))
        rows = case["batch"]
        if kind == "predict":
            return {"bytes": 2 * weights + 4 * rows * (dims[0] + dims[-1]), "flops": 2 * rows * weights}
        steps = max(1, case["steps"] * rows // case["count"]) * (case["count"] // rows)
        # per step the masters and both moments read and written, the operands' bf16 copy written and read twice
        return {"bytes": steps * (30 * weights + 4 * rows * dims[-1]) + 4 * weights, "flops": 6 * steps * rows * weights}
    m, n, nnz = _sizes(case)
    t = 4 if case["fp32"] else 8
    if kind == "spmv":
        return {"bytes": (4 + t) * nnz + 4 * (m + 1) + t * (m + n), "flops": 2 * nnz}
    per = 2 * (4 + t) * nnz + 4 * (m + n + 2) + (44 if case["fp32"] else 72) * (m + n)
    return {"bytes": case["iters"] * per, "flops": case["iters"] * 4 * nnz}


# ------------------------------------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        return _exact_spmv(case, seed)
    if kind == "predict":
        dims, p = _net_params(case, seed)
        return _forward64(dims, _split64(dims, p), torch.from_numpy(_net_data(case, seed, case["batch"])[0]))[0][-1].cpu()
    if kind == "train":  # with one batch an epoch the order of the shuffled rows does not matter
        return _exact_train(case, seed) if case["count"] == case["batch"] else None
    if kind == "batch":
        got = [_Pdhg(lp).solve(case["iters"]) for lp in _models(case, seed)]
        return [torch.cat([g["x"] for g in got]), torch.cat([g["y"] for g in got]),
                np.array([g["objective"] for g in got]), np.array([g["best"][0] for g in got])]
    p = _Pdhg(_model(case, seed))
    if kind == "solve":
        g = p.solve(case["iters"])
        return [g["x"], g["y"], g["objective"], g["best"][0], g["best"][1]]
    if kind == "engine":
        g = p.solve(case["iters"])
        return [g["xs"], g["zs"], g["best"][0], g["best"][1], g["norm"]]
    return p.steps(case["iters"])


def _exact_spmv(case, seed):
    lp = _model(case, seed)
    t = np.float32 if case["fp32"] else np.float64
    x = torch.randn(lp.n, dtype=torch.float32 if case["fp32"] else torch.float64,
                    generator=torch.Generator().manual_seed(seed)).numpy().astype(np.float64)
    val = _values(case, lp, seed).astype(t).astype(np.float64)
    cols = np.repeat(np.arange(lp.n), np.diff(lp.col_ptr))
    return np.bincount(lp.row_idx, weights=val * x[cols], minlength=lp.m)


def _split64(dims, p):
    out, at = [], 0
    p = torch.from_numpy(p).cuda().double()
    for i, o in zip(dims[:-1], dims[1:]):
        out.append([p[at:at + i * o].reshape(i, o).clone(), p[at + i * o:at + i * o + o].clone()])
        at += i * o + o
    return out


def _forward64(dims, layers, x):
    h, z = [x.cuda().double()], []
    for k, (w, b) in enumerate(layers):
        z.append(h[-1] @ w + b)
        h.append(torch.nn.functional.gelu(z[-1]) if k + 1 < len(layers) else z[-1])
    return h, z


def _exact_train(case, seed):
    dims, p = _net_params(case, seed)
    layers = _split64(dims, p)
    x, rng = _net_data(case, seed, case["count"])
    target = torch.from_numpy(rng.standard_normal((case["count"], case["out"]), dtype=np.float32)).cuda().double()
    x = torch.from_numpy(x)
    m = [[torch.zeros_like(t) for t in l] for l in layers]
    v = [[torch.zeros_like(t) for t in l] for l in layers]
    loss = 0.0
    for step in range(1, max(1, case["steps"] * case["batch"] // case["count"]) + 1):
        h, z = _forward64(dims, layers, x)
        r = h[-1] - target
        loss = float((r * r).mean())
        d = 2.0 * r / r.numel()
        for k in range(len(layers) - 1, -1, -1):
            w = layers[k][0]
            grads = [h[k].T @ d, d.sum(0)]
            if k:
                zz = z[k - 1]
                cdf = 0.5 * (1 + torch.erf(zz / 2 ** 0.5))
                d = (d @ w.T) * (cdf + zz * torch.exp(-0.5 * zz * zz) / (2 * np.pi) ** 0.5)
            for q, g in enumerate(grads):
                m[k][q].mul_(0.9).add_(g, alpha=0.1)
                v[k][q].mul_(0.999).addcmul_(g, g, value=0.001)
                layers[k][q] -= 1e-4 * (m[k][q] / (1 - 0.9 ** step)) / ((v[k][q] / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return [loss, torch.cat([t.reshape(-1) for l in layers for t in l]).cpu()]


class _Pdhg:
    """The restarted-average PDHG in 64 bits with torch's sparse products: Ruiz (10 passes) and Pock-Chambolle scaling,
    power iteration, iteration blocks, KKT evaluation and the restart rules, as the solver documents them."""

    def __init__(self, lp):
        dev, f = "cuda", torch.float64
        t = lambda a: torch.as_tensor(np.array(a, np.float64), dtype=f, device=dev)  # noqa: E731
        self.lp, m, n = lp, lp.m, lp.n
        cols = torch.from_numpy(np.repeat(np.arange(n), np.diff(lp.col_ptr))).to(dev)
        rows = torch.from_numpy(np.array(lp.row_idx, np.int64)).to(dev)
        v, dr, dc = t(lp.val), torch.ones(m, dtype=f, device=dev), torch.ones(n, dtype=f, device=dev)
        for k in range(11):
            how = "amax" if k < 10 else "sum"
            r = torch.zeros(m, dtype=f, device=dev).scatter_reduce(0, rows, v.abs(), how)
            c = torch.zeros(n, dtype=f, device=dev).scatter_reduce(0, cols, v.abs(), how)
            r, c = (torch.where(q > 0, q.sqrt(), torch.ones_like(q)) for q in (r, c))
            dr, dc = dr / r, dc / c
            v = v / (r[rows] * c[cols])
        at = lambda i, j, a, b: torch.sparse_coo_tensor(torch.stack([i, j]), v, (a, b)).coalesce().to_sparse_csr()  # noqa: E731
        self.A, self.AT, self.dr, self.dc = at(rows, cols, m, n), at(cols, rows, n, m), dr, dc
        sign = -1.0 if lp.maximize else 1.0
        lo, up = t(lp.row_lo), t(lp.row_up)
        self.c, self.l, self.u = sign * t(lp.cost) * dc, t(lp.col_lo) / dc, t(lp.col_up) / dc
        self.rl, self.ru = lo * dr, up * dr
        self.bnorm, self.cnorm = float(self._size(lo, up).norm()), float(t(lp.cost).norm())

    @staticmethod
    def _size(lo, up):
        z = torch.zeros_like(lo)
        return torch.maximum(torch.where(lo.isfinite(), lo.abs(), z), torch.where(up.isfinite(), up.abs(), z))

    def power(self):
        j = np.arange(self.lp.n, dtype=np.uint64)
        h = 0.5 + ((j * 2654435761 % 2 ** 32) % 1000) / 1000.0
        v = torch.from_numpy(h / np.sqrt((h * h).sum())).cuda()
        est = 0.0
        for it in range(200):
            v = self.AT @ (self.A @ v)
            s = float(v @ v)
            if s <= 0:
                return 0.0
            prev, est = est, s ** 0.25
            v = v / s ** 0.5
            if it >= 10 and abs(est - prev) <= 1e-7 * est:
                break
        return est

    def start(self):
        zero = torch.zeros_like(self.c)
        self.x = torch.minimum(torch.maximum(zero, self.l), self.u)
        self.z = torch.zeros_like(self.rl)
        self.anchor(self.x, self.z)

    def anchor(self, x, z):
        self.x, self.z, self.xl, self.zl = x, z, x, z
        self.xs, self.zs = torch.zeros_like(x), torch.zeros_like(z)
        self.ax, self.atz = self.A @ x, self.AT @ z

    def iterate(self, tau, sigma):
        for _ in range(FREQ):
            self.x = torch.minimum(torch.maximum(self.x - tau * (self.c + self.atz), self.l), self.u)
            ax = self.A @ self.x
            v = self.z + sigma * (2 * ax - self.ax)
            q = v / sigma
            self.z = torch.where(q < self.rl, v - sigma * self.rl, torch.where(q > self.ru, v - sigma * self.ru, 0.0))
            self.ax, self.atz = ax, self.AT @ self.z
            self.xs, self.zs = self.xs + self.x, self.zs + self.z

    def kkt(self, x, z, ax, atz):
        r = torch.clamp(torch.maximum(self.rl - ax, ax - self.ru), min=0.0)
        ro = r / self.dr
        rr = ro / (1 + self._size(self.rl, self.ru) / self.dr)
        drow = -torch.where((z > 0) & self.ru.isfinite(), z * self.ru, 0.0).sum() \
            - torch.where((z < 0) & self.rl.isfinite(), z * self.rl, 0.0).sum()
        d = self.c + atz
        edge = torch.where(d > 0, self.l, self.u)
        dcol = torch.where(edge.isfinite() & (d != 0), d * edge, 0.0).sum()
        res = torch.where(edge.isfinite(), 0.0, d.abs())
        sq = lambda q: float(q @ q)  # noqa: E731
        return np.array([sq(r), sq(ro), sq(rr), float(drow), sq(z - self.zl), sq(res), sq(res / self.dc),
                         float(self.c @ x), float(dcol), sq(x - self.xl)])

    def pair(self, f):
        xa, za = self.xs * f, self.zs * f
        return (self.kkt(self.x, self.z, self.ax, self.atz), self.kkt(xa, za, self.A @ xa, self.AT @ za), xa, za)

    def steps(self, iters):
        tau = 0.95 / self.power()
        self.start()
        half = max(1, iters // FREQ // 2)
        for block in range(1, iters // FREQ + 1):
            self.iterate(tau, tau)
            cur, avg, xa, za = self.pair(1.0 / (FREQ * (block if block <= half else block - half)))
            x, z = self.x, self.z
            if block == half:
                self.anchor(xa, za)
                x, z = xa, za
        return [x.cpu(), z.cpu(), cur, avg]

    def solve(self, iters):
        norm = self.power()
        cn, bn = float(self.c.norm()), float(self._size(self.rl, self.ru).norm())
        eta, w = 0.95 / norm if norm > 0 else 1.0, cn / bn if cn > 1e-10 and bn > 1e-10 else 1.0
        tau, sigma = eta / w, eta * w

        def error(k, w):
            return np.sqrt(w * k[0] + k[5] / w + (k[7] - k[3] - k[8]) ** 2)

        def rel(k):
            dual = k[3] + k[8]
            return [np.sqrt(k[1]) / (1 + self.bnorm), np.sqrt(k[6]) / (1 + self.cnorm),
                    abs(k[7] - dual) / (1 + abs(k[7]) + abs(dual))]
        self.start()
        ref, prev, it, since = error(self.kkt(self.x, self.z, self.ax, self.atz), w), np.inf, 0, 0
        while True:
            self.iterate(tau, sigma)
            it, since = it + FREQ, since + FREQ
            cur, avg, xa, za = self.pair(1.0 / since)
            use_avg = max(rel(avg)) < max(rel(cur))
            best = rel(avg) if use_avg else rel(cur)
            if max(best) <= 1e-9 or it >= iters:
                break
            wc, wa = error(cur, w), error(avg, w)
            cand, last = min(wa, wc), prev
            prev = cand
            if since >= 0.36 * it or cand <= 0.2 * ref or (cand <= 0.8 * ref and cand > last):
                to = avg if wa < wc else cur
                dx, dz = np.sqrt(to[9]), np.sqrt(to[4])
                if dx > 1e-10 and dz > 1e-10:
                    w = np.exp(0.5 * np.log(dz / dx) + 0.5 * np.log(w))
                    tau, sigma = eta / w, eta * w
                self.anchor(xa, za) if wa < wc else self.anchor(self.x, self.z)
                ref, prev, since = error(to, w), np.inf, 0
        xs, zs = (xa, za) if use_avg else (self.x, self.z)
        x, y = xs * self.dc, zs * self.dr
        obj = float(x @ torch.as_tensor(np.array(self.lp.cost, np.float64), device=x.device)) + self.lp.obj_const
        return dict(x=x.cpu(), y=y.cpu(), xs=xs.cpu(), zs=zs.cpu(), best=best, norm=norm, objective=obj)
