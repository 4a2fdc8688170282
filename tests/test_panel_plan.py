"""The plan of a matrix's panels (taral-lp_b200/csrc/panels.cuh, host side) on the CPU: every row once, its entries in the
column list, the limits of columns and rows kept, the same plan for every number of host threads, no panels (and no
exception) where memory runs out; and the rule that says which LPs' products run on panels."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

import lpgen

ROOT = Path(__file__).resolve().parents[1]
I64, I32, F64 = C.POINTER(C.c_int64), C.POINTER(C.c_int32), C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("panels") / "libpanel_plan.so"
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I", str(ROOT / "include"), "-I", str(ROOT / "taral-lp_b200" / "csrc"),
                    "-Xlinker", "-Bsymbolic", *(str(ROOT / "tests" / "native" / f) for f in ("panel_plan.cu", "failing_new.cpp")),
                    "-o", str(out)], check=True)
    L = C.CDLL(str(out))
    L.panel_product.argtypes = [C.c_int, C.c_int, I64, I32, F64, F64, C.c_int, C.c_int, C.c_int, C.c_int64, F64, I64]
    L.panels_suit_sizes.argtypes = [C.c_int64] * 5 + [C.c_int, C.c_int]
    L.least_panels_of.argtypes, L.least_panels_of.restype = [C.c_int64, C.c_int64, C.c_int], C.c_int64
    return L


def rows_to_csr(rows):
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return ptr, np.concatenate([np.asarray(r, np.int32) for r in rows] + [np.zeros(0, np.int32)])


def band(rows, k, cols=None):
    cols = cols or rows + k
    return [np.arange(r, r + k) for r in range(rows)], cols


def _mixed():  # short, long and empty rows over shared columns, in no order of length; column indices not ascending
    rng = np.random.default_rng(3)
    rows = []
    for r in range(900):
        k = int(rng.choice([0, 1, 4, 8, 20, 47, 48, 49, 64, 200]))
        rows.append(rng.permutation(400)[:k] + 300 * (r // 300))
    return rows, 1000


CASES = {
    "full_rows": lambda: band(3000, 8),                    # panels of 1,024 rows of 8
    "one_more_than_full": lambda: band(1025, 8),
    "mixed_long_short_empty": _mixed,
    # a stretch of rows whose columns are all different (more than 6,144 in a panel's nonzeros: its rows are halved)
    "column_limit": lambda: (band(6000, 12)[0] + [np.arange(7000 + 8 * r, 7008 + 8 * r) for r in range(1000)], 15_000),
    "all_long": lambda: band(700, 60),
    "empty_first_last": lambda: ([[]] * 40 + band(1200, 8)[0] + [[]] * 40, 1208),
}
REFUSED = {
    "no_shared_columns": lambda: ([np.arange(8 * r, 8 * r + 8) for r in range(2000)], 16_000),
    "padding": lambda: band(3000, 5),                      # rows of 5 stored as 8
    "row_of_more_columns_than_fit": lambda: (band(3000, 8)[0] + [np.arange(0, 2000)], 3008),  # with max_cols 1,500 below
    "row_longer_than_a_block": lambda: (band(3000, 8)[0] + [np.arange(2045)], 3008),
    # shared columns in the rows that are looked at first, none in most of the others: refused with the plan half done
    "late": lambda: ([np.arange(16) + 16 * (r // 600) if r % 5000 < 1100 else np.arange(16 * r, 16 * r + 16) for r in range(20_000)], 320_016),
    "few_rows": lambda: ([np.arange(40)] * 16, 40),        # a slice holds 32
    "empty": lambda: ([[]] * 10, 5),
}


def product(lib, rows, cols, threads=1, target=8192, max_cols=6144, allocs=-1):
    ptr, idx = rows_to_csr(rows)
    rng = np.random.default_rng(1)
    val, x = rng.integers(-8, 9, idx.size).astype(np.float64), rng.integers(-8, 9, cols).astype(np.float64)
    y, sizes = np.zeros(len(rows)), np.zeros(6, np.int64)
    rc = lib.panel_product(len(rows), cols, ptr.ctypes.data_as(I64), idx.ctypes.data_as(I32), val.ctypes.data_as(F64), x.ctypes.data_as(F64),
                           target, max_cols, threads, allocs, y.ctypes.data_as(F64), sizes.ctypes.data_as(I64))
    if rc == 1:  # whole numbers: exact in any order
        expected = np.array([val[a:b] @ x[idx[a:b]] for a, b in zip(ptr[:-1], ptr[1:])])
        assert np.array_equal(y, expected)
    return rc, dict(zip(("panels", "cols", "rows", "long", "listed", "padded"), sizes.tolist()))


@pytest.mark.parametrize("case", sorted(CASES))
def test_plan_covers_the_matrix(lib, case):
    rows, cols = CASES[case]()
    plans = [product(lib, rows, cols, threads) for threads in (1, 3, 16)]
    assert all(rc == 1 for rc, _ in plans) and all(p == plans[0] for p in plans)
    sizes = plans[0][1]
    if case.startswith(("full", "one_more")):
        assert sizes["rows"] == 1024
    if case == "column_limit":
        free = product(lib, rows, cols, max_cols=15_000)[1]
        assert free["cols"] > 6144 >= sizes["cols"] and sizes["panels"] > free["panels"]
    if case == "mixed_long_short_empty":
        assert sizes["long"] > 0


@pytest.mark.parametrize("case", sorted(REFUSED))
def test_plan_refuses(lib, case):
    rows, cols = REFUSED[case]()
    assert product(lib, rows, cols, max_cols=1500 if case == "row_of_more_columns_than_fit" else 6144)[0] == 0


@pytest.mark.parametrize("threads", [1, 8])
def test_plan_without_memory(lib, threads):
    rows, cols = band(6000, 12)  # four parts
    complete = product(lib, rows, cols, threads, target=2048)
    assert complete[0] == 1
    outcomes = [product(lib, rows, cols, threads, target=2048, allocs=k)[0] for k in (0, 1, 2, 5, 10, 20, 40, 80, 100, 150, 200, 300, 1000, 1_000_000)]
    assert set(outcomes) == {0, 1} and outcomes[0] == 0 and outcomes[-1] == 1


def test_rule(lib):
    """Which single LPs run on panels, at sizes measured on both sides."""
    def decide(nnz, m, n, fp64, panels=None):
        target = min(16384, max(8192, nnz // 296 * 21 // 20))
        a, t = (lib.least_panels_of(nnz, r, target) for r in (m, n)) if panels is None else panels
        return bool(lib.panels_suit_sizes(nnz, m, n, a, t, 148, fp64))
    for fp64 in (0, 1):
        assert decide(3_398_000, 72_000, 192_000, fp64)        # refinery of 48 periods
        assert decide(2_240_000, 280_000, 280_000, fp64)       # band of 8
        assert not decide(2_100_000, 350_000, 350_000, fp64)   # band of 6: short rows, more than a wave
        assert not decide(4_000_000, 400_000, 400_000, fp64)   # band of 10: panels filled by their rows
    assert not decide(6_796_540, 144_000, 384_000, 0) and decide(6_796_540, 144_000, 384_000, 1)  # refinery of 96
    assert not decide(9_000_000, 90_000, 90_000, 0) and decide(9_000_000, 90_000, 90_000, 1)      # band of 100
    assert decide(4_530_000, 96_000, 256_000, 0, (288, 325)) and not decide(4_530_000, 96_000, 256_000, 0, (288, 326))


def test_refinery_panels_are_one_wave(lib):
    """Multi-period LPs: one wave of 2 x 148 panels each way, on any host."""
    for periods in (32, 48):
        lp = lpgen.RefineryBase(periods, seed=7).instance(periods)
        target = min(16384, max(8192, lp.nnz // 296 * 21 // 20))
        ptr, idx, _ = lp.csr()
        for p, i, rows, cols in ((ptr, idx, lp.m, lp.n), (lp.col_ptr, lp.row_idx, lp.n, lp.m)):
            p, i, v, x = p.astype(np.int64), i.astype(np.int32), np.ones(lp.nnz), np.ones(cols)
            y, sizes = np.zeros(rows), np.zeros(6, np.int64)
            rc = lib.panel_product(rows, cols, p.ctypes.data_as(I64), i.ctypes.data_as(I32), v.ctypes.data_as(F64), x.ctypes.data_as(F64),
                                   target, 6144, 4, -1, y.ctypes.data_as(F64), sizes.ctypes.data_as(I64))
            assert rc == 1 and np.array_equal(y, np.diff(p)) and sizes[0] <= 296
