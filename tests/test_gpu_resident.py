"""Launches that take a whole block of iterations, an evaluation or the power iteration (csrc/resident.cuh: a
cooperative grid; csrc/cluster.cuh: one thread-block cluster, the LP in its shared memory) against the phase kernels they
stand for: the same products summed in the same order, so every number is the same bit for bit. TARAL_RESIDENT forces
a form: 0 phase kernels, 1 the grid; TARAL_CLUSTER the smallest cluster (the LP's data may ask for a larger one)."""
import dataclasses

import numpy as np
import pytest

import lpgen
import pdhg

pytestmark = pytest.mark.gpu

CASES = {
    "one_row": lambda: lpgen.packing(2, seed=1),                     # one row block each, mostly idle teams
    "general_300x700": lambda: lpgen.general(300, 700, seed=3),      # every row and bound kind, empty rows
    "packing_2000": lambda: lpgen.packing(2000, seed=3),             # several blocks, short rows
    "zipf_rows_over_a_tile": lambda: lpgen.planted(3000, 8000, 8, seed=5, zipf=1.1, cap=3000, floor=1),
    "refinery_2": lambda: lpgen.RefineryBase(2, seed=5).instance(2, lpgen.perturbations(1, 3)[0]),  # rows of 49-112
    "planted_90k": lambda: lpgen.planted(30_000, 90_000, 12, seed=2),  # more blocks than teams: several tiles a team
}


PANEL_CASES = {
    "refinery_2": CASES["refinery_2"],      # long rows and slices, panels over several periods
    "dense_columns": lambda: lpgen.planted(40, 900, 5, seed=3),   # A: 40 rows of ~112 on 900 columns; A^T: 900 rows of 5 on 40
    "transport_9x30": lambda: lpgen.transport(9, 30, seed=4),
}


def _record(lp, precision):
    e = pdhg.Engine.from_model(lp, precision=precision)
    norm = e.power_norm(200)
    e.set_steps(0.7 / norm, 0.9 / norm)
    e.start()
    out = [np.array([norm])]
    for steps, restart in ((64, True), (64, False), (7, None)):  # the last block is not of the evaluation length
        e.iterate(steps)
        out += list(e.eval_pair(1.0 / steps))
        if restart is not None:
            e.restart(restart, 1.0 / steps)
    out += [v for avg in (0, 1) for v in e.download(avg, 1.0 / 7)]
    r, x, z = e.solve(e.bnorm, e.cnorm, tol=1e-6, max_iter=640)
    e.close()
    return out + [x, z, np.array([r["iterations"], r["restarts"], r["rel_primal"], r["rel_dual"], r["rel_gap"]])]


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_resident_launches_change_nothing(engine_lib, monkeypatch, case, precision):
    lp = CASES[case]()
    monkeypatch.setenv("TARAL_TUNE", "0")  # both sides on the default row split
    got = {}
    for mode, cluster in (("0", "1"), ("1", "1"), ("2", "1"), ("2", "4"), ("2", "16")):
        monkeypatch.setenv("TARAL_RESIDENT", mode)
        monkeypatch.setenv("TARAL_CLUSTER", cluster)
        got[mode + cluster] = _record(lp, precision)
    for mode in got:
        for k, (a, b) in enumerate(zip(got["01"], got[mode])):
            assert np.array_equal(a, b, equal_nan=True), (mode, k, np.max(np.abs(a - b)))


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("case", sorted(PANEL_CASES))
def test_panels_change_nothing(engine_lib, monkeypatch, case, precision):
    """Products by panels (csrc/panels.cuh; TARAL_PANELS=1 takes them at any size where the columns are shared) against
    the row blocks in the same row order."""
    lp = PANEL_CASES[case]()
    monkeypatch.setenv("TARAL_TUNE", "0")
    monkeypatch.setenv("TARAL_ROWORDER", "0")
    monkeypatch.setenv("TARAL_RESIDENT", "0")
    got = []
    for flag in ("0", "1"):
        monkeypatch.setenv("TARAL_PANELS", flag)
        got.append(_record(lp, precision))
    for k, (a, b) in enumerate(zip(*got)):
        assert np.array_equal(a, b, equal_nan=True), (k, np.max(np.abs(a - b)))


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", ["one_cta", "several_ctas", "shared_matrix"])
def test_batch_clusters_change_nothing(engine_lib, monkeypatch, shape, precision):
    """A batch of small LPs on one cluster each against the batch's phase kernels: the same norms, iterations and points,
    bit for bit, through restarts, instances that stop at different blocks and a final partial block."""
    if shape == "shared_matrix":  # instances of one matrix with their own costs and bounds
        base = lpgen.general(200, 450, seed=5)
        rng = np.random.default_rng(1)
        lps = [dataclasses.replace(base, cost=base.cost * rng.uniform(0.8, 1.2, base.n)) for _ in range(5)]
    else:
        m, n = (120, 300) if shape == "one_cta" else (900, 2100)
        lps = [lpgen.general(m + 7 * k, n + 11 * k, seed=k) for k in range(5)] + [lpgen.transport(12, 17, seed=2)]
    got = []
    for mode in ("0", "2"):
        monkeypatch.setenv("TARAL_RESIDENT", mode)
        b = pdhg.Batch(lps, tol=1e-5, max_iter=1000, precision=precision)
        got.append(b.solve() + b.solve())  # the second solve replays the captured launches
        b.close()
    for (r0, x0, y0), (r1, x1, y1) in zip((got[0][:3], got[0][3:]), (got[1][:3], got[1][3:])):
        for a, c in zip(r0, r1):
            assert (a["status"], a["iterations"], a["restarts"], a["norm_a"]) == (c["status"], c["iterations"], c["restarts"], c["norm_a"])
        assert all(np.array_equal(p, q) for p, q in zip(x0 + y0, x1 + y1))


@pytest.mark.parametrize("precision", [pdhg.FP64, pdhg.FP32], ids=["fp64", "fp32"])
def test_batch_panels_change_nothing(engine_lib, monkeypatch, precision):
    """A batch's phases on panels, several instances to a CTA (7 and 2 of two matrices: full and partly used groups),
    against the row blocks; instances stop at different blocks, so the lists are rebuilt on the way."""
    base = lpgen.RefineryBase(2, seed=5)
    pert = lpgen.perturbations(9, seed=8)
    lps = [base.instance(2, p) for p in pert[:7]] + [base.instance(1, p) for p in pert[7:]]
    monkeypatch.setenv("TARAL_TUNE", "0")
    got = []
    for flag in ("0", "1"):
        monkeypatch.setenv("TARAL_PANELS", flag)
        b = pdhg.Batch(lps, tol=1e-4, max_iter=20_000, precision=precision, time_limit=120)
        got.append((b.solve(), b.solve()))  # the second solve restores the full lists
        b.close()
    assert len({r["iterations"] for r in got[0][0][0]}) > 2
    for (r0, x0, y0), (r1, x1, y1) in zip(*got):
        for a, c in zip(r0, r1):
            assert (a["status"], a["iterations"], a["restarts"], a["norm_a"]) == (c["status"], c["iterations"], c["restarts"], c["norm_a"])
        assert all(np.array_equal(p, q) for p, q in zip(x0 + y0, x1 + y1))
