"""The forms in which a context or a batch runs its iterations (clusters, a cooperative grid, panels, a launch per phase)
beside one another, at the limits of what they accept and where one of them gives up."""
import dataclasses
import threading

import numpy as np
import pytest

import lpgen
import pdhg

pytestmark = pytest.mark.gpu


def _drive(eng, reps, out, errors):
    try:
        norm = eng.power_norm(20)
        eng.set_steps(0.7 / norm, 0.9 / norm)
        eng.start()
        for k in range(reps):
            eng.iterate(1)  # a launch or two per call: as many chances as possible to meet the other thread's
            if k % 16 == 15:
                eng.eval_pair(1.0 / (k + 1))
        out += [np.array([norm])] + list(eng.eval_pair(1.0 / reps)) + list(eng.download(0, 1.0))
    except Exception as e:  # noqa: BLE001 -- reported by the test's own thread
        errors.append(e)


@pytest.mark.parametrize("form,small,large", [
    ("one_cta", lambda: lpgen.general(30, 70, seed=1), lambda: lpgen.general(300, 700, seed=3)),
    ("cluster", lambda: lpgen.planted(900, 2300, 5, seed=2), lambda: lpgen.planted(2000, 5000, 5, seed=2)),
    ("grid", lambda: lpgen.general(30, 70, seed=1), lambda: lpgen.planted(60_000, 150_000, 6, seed=2)),
    ("panels", lambda: lpgen.RefineryBase(1, seed=5).instance(1), lambda: lpgen.RefineryBase(3, seed=5).instance(3)),
    ("grid_beside_panels", lambda: lpgen.planted(10_000, 25_000, 5, seed=2), lambda: lpgen.RefineryBase(3, seed=5).instance(3)),
], ids=["one_cta", "cluster", "grid", "panels", "grid_beside_panels"])
def test_contexts_of_two_threads(engine_lib, monkeypatch, form, small, large):
    """Contexts are independent of each other: two threads, each with its own context of another size, get the bits that
    they get one after the other."""
    monkeypatch.setenv("TARAL_TUNE", "0")
    if form == "grid":
        monkeypatch.setenv("TARAL_RESIDENT", "1")
    if "panels" in form:
        monkeypatch.setenv("TARAL_PANELS", "1")
    lps = [small(), large()]
    alone = []
    for lp in lps:
        eng, out, errors = pdhg.Engine.from_model(lp), [], []
        _drive(eng, 400, out, errors)
        eng.close()
        assert not errors, errors
        alone.append(out)
    for _ in range(3):
        engines = [pdhg.Engine.from_model(lp) for lp in lps]
        outs, errors = [[], []], []
        threads = [threading.Thread(target=_drive, args=(e, 400, o, errors)) for e, o in zip(engines, outs)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for e in engines:
            e.close()
        assert not errors, errors
        for a, b in zip(alone, outs):
            assert len(a) == len(b) and all(np.array_equal(p, q) for p, q in zip(a, b))


def test_batch_of_more_matrices_than_a_grid_dimension(engine_lib):
    """65,537 LPs of a matrix each, beyond the 65,535 CTAs of a grid's second dimension: every one gets the answer that it
    gets in a batch of a few."""
    count = (1 << 16) + 1
    ptr, idx = np.array([0, 1, 2], np.int64), np.array([0, 0], np.int32)
    cost, lo, up, rhs = np.array([1.0, 2.0]), np.zeros(2), np.full(2, 5.0), np.array([3.0])

    def lp(k):  # min x0 + 2 x1, (1 + k / count) x0 + x1 = 3
        return lpgen.LP(f"two_{k}", 1, 2, ptr, idx, np.array([1.0 + k / count, 1.0]), cost, lo, up, rhs, rhs)
    picked = [0, 1, 40_000, 65_534, 65_535, 65_536]
    few = pdhg.Batch([lp(k) for k in picked], tol=1e-8, max_iter=128)
    r0, x0, y0 = few.solve()
    few.close()
    many = pdhg.Batch([lp(k) for k in range(count)], tol=1e-8, max_iter=128)
    assert many.info()["distinct_matrices"] == count
    r1, x1, y1 = many.solve()
    many.close()
    for i, k in enumerate(picked):
        assert (r0[i]["status"], r0[i]["iterations"], r0[i]["norm_a"]) == (r1[k]["status"], r1[k]["iterations"], r1[k]["norm_a"])
        assert np.array_equal(x0[i], x1[k]) and np.array_equal(y0[i], y1[k])


@pytest.mark.parametrize("call", ["eval_current", "eval_average", "eval_pair", "download", "restart_then_eval", "power_norm"])
def test_barrier_that_gives_up_is_reported(engine_lib, monkeypatch, call):
    """A block of iterations whose grid barrier gives up its wait (here: at once) leaves a half-done iterate. The first
    call that would return numbers of it fails, so do the others, and a new start makes the context usable again."""
    lp = lpgen.planted(4000, 10_000, 5, seed=2)  # several CTAs
    monkeypatch.setenv("TARAL_RESIDENT", "1")
    good = pdhg.Engine.from_model(lp)
    good.set_steps(0.1, 0.1)
    good.start()
    expected, point = good.eval(0, 1.0), good.download(0, 1.0)
    good.close()
    monkeypatch.setenv("TARAL_BARRIER_POLLS", "0")
    eng = pdhg.Engine.from_model(lp)
    eng.set_steps(0.1, 0.1)
    calls = {"eval_current": lambda: eng.eval(0, 1.0), "eval_average": lambda: eng.eval(1, 1.0 / 8),
             "eval_pair": lambda: eng.eval_pair(1.0 / 8), "download": lambda: eng.download(0, 1.0),
             "restart_then_eval": lambda: (eng.restart(False, 1.0), eng.eval(0, 1.0)),
             "power_norm": lambda: eng.power_norm(20)}
    for _ in range(2):
        eng.start()
        assert np.array_equal(eng.eval(0, 1.0), expected)
        assert all(np.array_equal(a, b) for a, b in zip(eng.download(0, 1.0), point))
        eng.iterate(8)
        with pytest.raises(pdhg.TaralError) as e:
            calls[call]()
        assert "timed out" in str(e.value)
        for other in calls.values():
            with pytest.raises(pdhg.TaralError):
                other()
        with pytest.raises(pdhg.TaralError):
            eng.iterate(8)
    with pytest.raises(pdhg.TaralError):
        eng.solve(eng.bnorm, eng.cnorm, tol=1e-4, max_iter=64)
    eng.start()
    assert np.array_equal(eng.eval(0, 1.0), expected)
    eng.close()


@pytest.mark.parametrize("resident,block,pair", [("0", 1 + 2 * 64, 6), ("1", 1, 1), ("2", 1, 1)], ids=["phases", "grid", "cluster"])
def test_launches_are_counted(engine_lib, monkeypatch, resident, block, pair):
    """device_launches and a solve's kernel_launches are what the device was given; kernel_launches of a context counts the
    phases, the same in every form."""
    monkeypatch.setenv("TARAL_RESIDENT", resident)
    eng = pdhg.Engine.from_model(lpgen.packing(2000, seed=3))
    eng.set_steps(0.5, 0.5)
    eng.start()

    def counted(call):
        before = eng.device_launches, eng.kernel_launches
        call()
        return eng.device_launches - before[0], eng.kernel_launches - before[1]
    assert counted(lambda: eng.iterate(64)) == (block, 129)
    assert counted(lambda: eng.iterate(1)) == (1 + 2 if resident == "0" else 1, 3)
    assert counted(lambda: eng.eval_pair(1 / 64)) == (pair, 6)
    launched, _ = counted(lambda: eng.power_norm(50))
    # the start vector, and chunks of 8 steps of 4 launches or all steps in one
    assert launched >= 1 + 8 * 4 if resident == "0" else launched == 2
    before = eng.device_launches
    r, _, _ = eng.solve(eng.bnorm, eng.cnorm, tol=1e-12, max_iter=128)
    assert r["kernel_launches"] == eng.device_launches - before
    eng.close()


@pytest.mark.parametrize("precision,tiles,long,resident", [
    (pdhg.FP32, 640, 0, True), (pdhg.FP32, 900, 0, True), (pdhg.FP32, 1000, 0, False), (pdhg.FP64, 1000, 0, True), (pdhg.FP64, 2300, 0, True),
    (pdhg.FP64, 2450, 0, False), (pdhg.FP64, 560, 33_000, False), (pdhg.FP32, 100, 25_600, True),
])
def test_power_iteration_form(engine_lib, monkeypatch, precision, tiles, long, resident):
    """One launch for the whole power iteration up to the sizes where it is the faster one, a launch per phase beyond and
    where a row is many tiles long; the same norm bit for bit."""
    monkeypatch.setenv("TARAL_TUNE", "0")
    n = 256 * tiles  # columns of 5: a tile of A^T holds 256 of them
    lp = lpgen.planted(max(n // 3, 100), n, 5, seed=1)
    if long:  # one row more, over the first columns: longer than 16 tiles of 2,044 nonzeros or not
        rows = np.split(lp.row_idx, lp.col_ptr[1:-1])
        vals = np.split(lp.val, lp.col_ptr[1:-1])
        rows = [np.append(r, lp.m) if j < long else r for j, r in enumerate(rows)]
        vals = [np.append(v, 0.01) if j < long else v for j, v in enumerate(vals)]
        ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64)
        lp = dataclasses.replace(lp, m=lp.m + 1, col_ptr=ptr, row_idx=np.concatenate(rows).astype(np.int32), val=np.concatenate(vals),
                                 row_lo=np.append(lp.row_lo, -np.inf), row_up=np.append(lp.row_up, np.inf))
    norms = {}
    for mode in (None, "0"):
        if mode is not None:
            monkeypatch.setenv("TARAL_RESIDENT", mode)
        eng = pdhg.Engine.from_model(lp, precision=precision)
        before = eng.device_launches
        norms[mode] = eng.power_norm(24)
        if mode is None:
            assert (eng.device_launches - before == 2) == resident
        eng.close()
    assert norms[None] == norms["0"]


def _blocks(count, rows, cols, seed=0):
    """A block-diagonal LP of dense blocks."""
    rng = np.random.default_rng(seed)
    m, n = count * rows, count * cols
    idx = ((np.arange(n) // cols * rows)[:, None] + np.arange(rows)).ravel().astype(np.int32)
    val, x = rng.standard_normal(n * rows), rng.uniform(0, 1, n)
    b = np.zeros(m)
    np.add.at(b, idx, val * np.repeat(x, rows))
    return lpgen.LP(f"blocks_{count}", m, n, np.arange(n + 1, dtype=np.int64) * rows, idx, val, rng.standard_normal(n), np.zeros(n),
                    np.full(n, 10.0), b, b.copy())


@pytest.mark.parametrize("lp,precision,cluster", [
    (lambda: lpgen.planted(2000, 5000, 5, seed=1), pdhg.FP64, True), (lambda: lpgen.general(307, 701, seed=1), pdhg.FP32, True),
    (lambda: lpgen.planted(1996, 3338, 7, seed=1, zipf=1.2, cap=2000, floor=5), pdhg.FP64, True),  # the grid is slower still
    (lambda: _blocks(4, 100, 100), pdhg.FP32, False), (lambda: _blocks(12, 70, 80), pdhg.FP32, False),
], ids=["planted", "general", "a_very_long_row", "long_rows", "many_long_rows"])
def test_cluster_choice(engine_lib, monkeypatch, lp, precision, cluster):
    """One LP runs on a cluster where the plan's estimate is below the grid's time, not where a warp would take many long
    rows one after another."""
    lp, mem = lp(), {}
    for mode in ("1", "2"):  # 1: never a cluster
        monkeypatch.setenv("TARAL_RESIDENT", mode)
        eng = pdhg.Engine.from_model(lp, precision=precision)
        mem[mode] = eng.info()[1]
        eng.close()
    assert (mem["2"] > mem["1"]) == cluster


@pytest.mark.parametrize("lps,precision,cluster", [
    (lambda: [lpgen.general(151, 347, seed=k) for k in range(40)], pdhg.FP64, True),
    (lambda: [lpgen.general(1500, 3500, seed=1)] * 14, pdhg.FP32, True),
    (lambda: [lpgen.general(1500, 3500, seed=1)] * 128, pdhg.FP32, False),   # more waves of clusters than they are worth
    (lambda: [_blocks(4, 150, 200)] * 16, pdhg.FP32, False),                 # long rows
    (lambda: [_blocks(2, 100, 100)] * 100, pdhg.FP32, False),
], ids=["small", "a_wave", "many_waves", "large", "long_rows"])
def test_batch_cluster_choice(engine_lib, monkeypatch, lps, precision, cluster):
    lps, mem = lps(), {}
    for mode in ("0", "2"):
        monkeypatch.setenv("TARAL_RESIDENT", mode)
        b = pdhg.Batch(lps, precision=precision)
        mem[mode] = b.info()["device_mem_bytes"]
        b.close()
    assert (mem["2"] > mem["0"]) == cluster


def _engine_numbers(lp, precision):
    eng = pdhg.Engine.from_model(lp, precision=precision)
    norm = eng.power_norm(30)
    eng.set_steps(0.7 / norm, 0.9 / norm)
    eng.start()
    eng.iterate(64)
    out = [np.array([norm])] + list(eng.eval_pair(1 / 64)) + list(eng.download(0, 1.0))
    mem = eng.info()[1]
    eng.close()
    return mem, out


def _batch_numbers(lps, precision):
    b = pdhg.Batch(lps, tol=1e-12, max_iter=128, precision=precision)
    res, xs, ys = b.solve()
    mem = b.info()["device_mem_bytes"]
    b.close()
    return mem, [np.array([r["norm_a"], r["rel_primal"], r["rel_dual"]]) for r in res] + xs + ys


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("form", ["panels", "batch_panels", "cluster", "batch_cluster"])
def test_forms_give_way_where_memory_is_short(engine_lib, monkeypatch, form, precision):
    """What panels and clusters hold on the device is extra: a context or a batch for whose plain form the memory suffices
    is created all the same, and gives the same numbers."""
    monkeypatch.setenv("TARAL_TUNE", "0")
    monkeypatch.setenv("TARAL_ROWORDER", "0")
    base = lpgen.RefineryBase(2, seed=5)
    pert = lpgen.perturbations(6, seed=8)
    small = lpgen.general(200, 450, seed=5)
    if form.startswith("batch"):
        lps = [base.instance(2, p) for p in pert] if form == "batch_panels" else [
            dataclasses.replace(small, cost=small.cost * (1 + k / 10)) for k in range(4)]
        numbers = lambda: _batch_numbers(lps, precision)  # noqa: E731
    else:
        lp = base.instance(2, pert[0]) if form == "panels" else small
        numbers = lambda: _engine_numbers(lp, precision)  # noqa: E731
    switch, off, on = ("TARAL_PANELS", "0", "1") if "panels" in form else ("TARAL_RESIDENT", "0", "2")
    monkeypatch.setenv(switch, off)
    plain, expected = numbers()
    monkeypatch.setenv(switch, on)
    full, got = numbers()
    assert full > plain  # the form is there
    for a, b in zip(expected, got):
        assert np.array_equal(a, b)
    try:
        for limit in (plain, plain + (full - plain) // 3, plain + 2 * (full - plain) // 3, full - 1, full):
            pdhg.set_device_alloc_limit(limit)
            mem, got = numbers()
            assert mem <= limit and (mem == full) == (limit == full)
            for a, b in zip(expected, got):
                assert np.array_equal(a, b)
    finally:
        pdhg.set_device_alloc_limit(0)


def _band(rows, k, extra=0, seed=0):
    """A square LP whose column j has the rows j .. j + k - 1, with `extra` empty rows and columns at the end."""
    rng = np.random.default_rng(seed)
    m = n = rows + k - 1 + extra
    lens = np.where(np.arange(n) < rows, k, 0)
    idx = np.concatenate([np.arange(j, j + k) for j in range(rows)]).astype(np.int32)
    val, x = rng.standard_normal(idx.size), rng.uniform(0, 1, n)
    b = np.zeros(m)
    np.add.at(b, idx, val * np.repeat(x, lens))
    return lpgen.LP(f"band_{rows}_{k}", m, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.int64), idx, val, rng.standard_normal(n),
                    np.zeros(n), np.full(n, 10.0), b, b.copy())


def _column_limit():
    """A band of 24 and, at its end, rows of 10 with columns of their own: more than 6,144 columns in one panel's nonzeros, so
    that its rows are halved. Those columns lie where the plan does not look first."""
    base, rows, per, at = _band(24_000, 24), 700, 10, 8200
    rng = np.random.default_rng(5)
    cut = base.col_ptr[at]
    idx = np.concatenate([base.row_idx[:cut], np.repeat(base.m + np.arange(rows), per), base.row_idx[cut:]]).astype(np.int32)
    val = np.concatenate([base.val[:cut], rng.uniform(0.5, 1.5, rows * per), base.val[cut:]])
    ptr = np.concatenate([base.col_ptr[:at], cut + np.arange(rows * per), base.col_ptr[at:] + rows * per])
    n, pad = base.n + rows * per, np.full(rows, 3.0)
    return lpgen.LP("column_limit", base.m + rows, n, ptr.astype(np.int64), idx, val, rng.standard_normal(n), np.zeros(n), np.full(n, 10.0),
                    np.concatenate([base.row_lo, pad]), np.concatenate([base.row_up, pad]))


PANELS = {
    "full_panels_of_1024_rows": lambda: _band(3000, 8),
    "empty_rows": lambda: _band(2500, 12, extra=300),
    "long_rows_only": lambda: _band(1500, 60),
    "blocks": lambda: _blocks(6, 70, 90),
    "column_limit": _column_limit,
    "refinery": lambda: lpgen.RefineryBase(3, seed=5).instance(3, lpgen.perturbations(1, 3)[0]),
}


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(PANELS))
def test_panels_and_one_launch_evaluations(engine_lib, monkeypatch, case, precision):
    """Panels as they run (with the one-launch evaluation) against a launch per phase on row blocks, both in the model's row
    order: the same bits, also for points that are not finite."""
    lp = PANELS[case]()
    monkeypatch.setenv("TARAL_TUNE", "0")
    monkeypatch.setenv("TARAL_ROWORDER", "0")
    got, mem = [], []
    for panels, resident in (("0", "0"), ("1", None)):
        monkeypatch.setenv("TARAL_PANELS", panels)
        if resident is None:
            monkeypatch.delenv("TARAL_RESIDENT")
        else:
            monkeypatch.setenv("TARAL_RESIDENT", resident)
        eng = pdhg.Engine.from_model(lp, precision=precision)
        mem.append(eng.info()[1])
        out = [np.array([eng.power_norm(40)])]
        eng.set_steps(0.02, 0.03)
        for x0 in (None, np.where(np.arange(lp.n) % 97 == 5, np.inf, 0.25), np.where(np.arange(lp.n) % 89 == 3, np.nan, -1.0)):
            eng.start(x0, None if x0 is None else np.linspace(-1, 1, lp.m))
            for steps in (64, 64, 3):
                eng.iterate(steps)
                out += list(eng.eval_pair(1.0 / steps))
                eng.restart(steps == 64, 1.0 / steps)
            out += [eng.eval(0, 1.0)] + [v for avg in (0, 1) for v in eng.download(avg, 0.5)]
        got.append(out)
        if resident is None:  # a launch per phase, so these are the panels
            before = eng.device_launches
            eng.iterate(5)
            assert eng.device_launches - before == 11
        eng.close()
    size = 8 if precision == pdhg.FP64 else 4
    assert mem[1] - mem[0] >= 2 * lp.nnz * (size + 2)  # both matrices' values and positions once more
    for k, (a, b) in enumerate(zip(*got)):
        assert np.array_equal(a, b, equal_nan=True), (k, a, b)
