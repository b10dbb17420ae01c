"""The cell list's one-launch scan at both sides of its limit, the correction's
lanes per particle at each change, and slab lists over more cell rows than a
warp has lanes, against the oracle; counters that are left zero for the next
solve are exercised by solving twice."""
import numpy as np
import pytest

from gpu_helpers import both, kw_of, rel_l2

import ffcm_oracle as O

pytestmark = pytest.mark.gpu
TOL = {np.float32: 1e-5, np.float64: 1e-10}   # the suite's end-to-end bounds


def _solve_twice(ffcm, T, kw, seed):
    prod, ora = both(ffcm, T, **kw)
    rng = np.random.default_rng(seed)
    for _ in range(2):
        Y = (rng.random((kw["N"], 3)) * np.array(kw["L"])).astype(T)
        F = rng.standard_normal((kw["N"], 3)).astype(T)
        V = ffcm.mobility(np.empty_like(Y), prod, Y, F)
        ref = O.apply(ora, Y, F)
        assert rel_l2(V, ref) < TOL[np.dtype(T).type]
    return prod, ora, V, ref, Y, F


@pytest.mark.parametrize("cells", [(3, 3, 3), (16, 16, 8), (32, 32, 32), (33, 32, 32), (40, 41, 42)])
def test_cell_list_scan(ffcm, cells):
    fine = 3 if min(cells) < 8 else 1
    kw = kw_of(tuple(float(c) for c in cells), 4000, tuple(fine * c for c in cells), M_G=4, R_c=1.0)
    prod, ora, V, ref, Y, F = _solve_twice(ffcm, np.float64, kw, sum(cells))
    assert np.array_equal(prod.original_index, ora.original_index)
    assert np.array_equal(prod.cell_start, ora.cell_start) and np.array_equal(prod.cell_end, ora.cell_end)
    # the step API counts for itself
    ffcm.wrap_positions(prod, Y)
    ffcm.assign_cells(prod)
    ffcm.sort_particles_by_cell(prod, F)
    assert np.array_equal(prod.original_index, ora.original_index)


@pytest.mark.parametrize("T,N", [(T, N) for T in (np.float32, np.float64) for N in (16000, 16001, 50000, 50001)])
def test_correction_lanes(ffcm, T, N):
    # 5% by volume: pairs closer than a diameter are rare
    L = (N * 4.0 / 3.0 * np.pi / 0.05) ** (1.0 / 3.0)
    _, _, V, ref, _, _ = _solve_twice(ffcm, T, kw_of(L, N, 64, R_c=3.0), N)
    assert rel_l2(V, ref) < TOL[T]


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_slab_lists_over_many_cell_rows(ffcm, T):
    # 12 x 10 cell rows reach a slab of 4 x 2 grid rows
    _, _, V, ref, _, _ = _solve_twice(ffcm, T, kw_of(64.0, 3000, 64, R_c=1.0), 7)
    assert rel_l2(V, ref) < TOL[T]


@pytest.mark.parametrize("cells", [(64, 32, 32), (41, 40, 40)])
def test_cell_list_scan_limit(ffcm, cells):
    """65,536 cells (one launch) and 65,600 (three)."""
    kw = kw_of(tuple(float(c) for c in cells), 4000, cells, M_G=4, R_c=1.0)
    prod, ora, V, ref, Y, F = _solve_twice(ffcm, np.float64, kw, sum(cells))
    assert np.array_equal(prod.original_index, ora.original_index)
    assert np.array_equal(prod.cell_start, ora.cell_start) and np.array_equal(prod.cell_end, ora.cell_end)
    assert rel_l2(V, ref) < TOL[np.float64]
