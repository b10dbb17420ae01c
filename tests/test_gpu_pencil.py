"""Pencil spread and interpolation (csrc/pencil.cuh), forced on with FFCM_PENCIL=1,
against the oracle: grids whose sides are no multiple of a pencil or of a
segment, stencils of every instance width and as wide as the grid, particles
on one spot, at the box edges and alone; and the paths that keep the lists
(operator, conjugate gradients, adjoint, batch capture)."""
import numpy as np
import pytest

from gpu_helpers import both, kw_of, rel_l2

import ffcm_oracle as O

pytestmark = pytest.mark.gpu
# the end-to-end parity bounds of the whole suite (test_gpu_mobility.py)
TOL = {np.float32: 1e-5, np.float64: 1e-10}


def _inputs(T, L, N, layout, seed):
    rng = np.random.default_rng(seed)
    L = np.broadcast_to(np.asarray(L, np.float64), (3,))
    Y = rng.random((N, 3)) * L
    if layout == "spot":          # more than one batch of entries with one first x point
        Y = 0.3 * L + 0.05 * rng.standard_normal((N, 3))
    elif layout == "edges":       # half of them within a tenth of the box of a face, no two alike
        Y[::2] = np.mod(0.2 * (Y[::2] - 0.5 * L), L)
    return Y.astype(T), rng.standard_normal((N, 3)).astype(T)


@pytest.fixture
def forced(monkeypatch):
    monkeypatch.setenv("FFCM_PENCIL", "1")
    return monkeypatch


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M,MG,N,layout", [
    ((10, 12, 14), 6, 40, "uniform"), ((10, 12, 14), 10, 40, "edges"), ((7, 9, 8), 7, 30, "uniform"),
    ((33, 17, 9), 9, 300, "edges"), ((24, 8, 4), 4, 60, "uniform"), ((12, 12, 12), 12, 50, "edges"),
    ((40, 30, 50), 7, 900, "uniform"), ((100, 31, 29), 11, 700, "edges"), ((96, 40, 36), 12, 500, "uniform"),
    ((130, 24, 20), 5, 400, "edges"), ((64, 64, 64), 10, 1500, "uniform"), ((45, 33, 30), 8, 200, "spot"),
    ((20, 18, 22), 2, 100, "uniform"), ((60, 60, 60), 9, 1, "uniform"),
])
def test_pencil_solve_matches_oracle(ffcm, forced, T, M, MG, N, layout):
    L = tuple(0.6 * m for m in M)
    prod, ora = both(ffcm, T, **kw_of(L, N, M, M_G=MG, R_c=0.4 * min(L)))
    Y, F = _inputs(T, L, N, layout, N + MG)
    if layout == "spot":
        # the pair terms of overlapping spheres cancel badly in Float32, in the
        # oracle as here: compare with the same pair terms beside the
        # warp-per-particle grid steps
        forced.setenv("FFCM_PENCIL", "0")
        ref = ffcm.mobility(np.empty_like(Y), ffcm.FFCMConfig(T, **kw_of(L, N, M, M_G=MG, R_c=0.4 * min(L))), Y, F)
    else:
        ref = O.apply(ora, Y, F)
    for _ in range(2):            # the second solve reuses the list buffers
        assert rel_l2(ffcm.mobility(np.empty_like(Y), prod, Y, F), ref) < TOL[T]


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_pencil_lists_are_kept(ffcm, forced, T):
    """Operator, conjugate gradients and adjoint on kept lists: the same as
    without the pencils, in either stencil mode."""
    M, N, L = (50, 36, 42), 600, tuple(0.55 * m for m in (50, 36, 42))
    kw = kw_of(L, N, M, M_G=9, R_c=3.0)
    Y, F = _inputs(T, L, N, "uniform", 3)
    lam = F[::-1].copy()
    got = []
    for mode in "10":
        forced.setenv("FFCM_PENCIL", mode)
        cfg = ffcm.FFCMConfig(T, **kw)
        res = []
        for stencil in ("reference", "float64"):
            cfg.stencil = stencil
            A = ffcm.FFCMMobility(cfg, Y)
            res += [A @ F, A @ lam, ffcm.cg(A, F, reltol=0.0, maxiter=5)]
            V, pull = ffcm.rrule_mobility(cfg, Y, F)
            res += [V, *pull(lam)]
        got.append(res)
    for a, b in zip(*got):
        assert rel_l2(a, b) < 10 * TOL[T]   # five iterations and the gradient's cancellation


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_stencil_switch_on_fixed_positions(ffcm, forced, T):
    """The lists follow a stencil mode changed after the positions were fixed
    (positions half way between grid points, whose anchors depend on the mode)."""
    M, N = (50, 36, 42), 400
    L = tuple(0.537 * m for m in M)
    cfg = ffcm.FFCMConfig(T, **kw_of(L, N, M, M_G=9, R_c=3.0))
    rng = np.random.default_rng(8)
    Y = ((rng.integers(0, np.array(M), (N, 3)) + 0.5) * np.array(L) / np.array(M)
         + 1e-9 * rng.standard_normal((N, 3))).astype(T)
    Y = Y[np.unique(Y, axis=0, return_index=True)[1]]
    Y = np.concatenate([Y, (rng.random((N - len(Y), 3)) * np.array(L)).astype(T)])
    F = rng.standard_normal((N, 3)).astype(T)
    A = ffcm.FFCMMobility(cfg, Y)
    A @ F
    for mode in ("float64", "reference"):
        cfg.stencil = mode
        got = A @ F
        assert rel_l2(got, ffcm.mobility(np.empty_like(F), cfg, Y, F)) < TOL[T]
        A = ffcm.FFCMMobility(cfg, Y)
        A @ F


def test_pencil_batch_under_capture(ffcm, forced):
    T = np.float32
    systems = [dict(L=(27.0,) * 3, R_c=3.0, N=400, num_grid_points=(48, 48, 48)),
               dict(L=(30.0, 15.0, 20.0), R_c=3.0, N=200, num_grid_points=(60, 30, 40))]
    b = ffcm.FFCMBatch(T, systems=systems, kernel_widths_ratio=2.0, M_G=9, viscosity=1.0, nrhs=2)
    rng = np.random.default_rng(0)
    Ys = [(rng.random((s["N"], 3)) * np.array(s["L"])).astype(T) for s in systems]
    Fs = [[rng.standard_normal((s["N"], 3)).astype(T) for _ in range(2)] for s in systems]
    Yp, Fp = b.pack(Ys, Fs)
    V = np.empty_like(Fp)
    b.mobility(V, Yp, Fp)
    for s, Y, fs, vs in zip(systems, Ys, Fs, b.unpack(V)):
        ora = O.OracleConfig(T, kernel_widths_ratio=2.0, M_G=9, viscosity=1.0, **s)
        for f, v in zip(fs, vs):
            assert rel_l2(v, O.apply(ora, Y, f)) < TOL[T]


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M,MG,N", [((40, 30, 50), 7, 3000), ((96, 40, 36), 12, 4000), ((130, 24, 20), 5, 2500),
                                    ((33, 17, 9), 9, 1500)])
def test_pencils_shared_by_several_warps(ffcm, forced, T, M, MG, N):
    """Clusters whose segments hold more entries than one warp walks:
    every solve of a configuration, on new and on kept lists and in the adjoint,
    against the warp-per-particle grid steps."""
    L = tuple(0.6 * m for m in M)
    rng = np.random.default_rng(N)
    Y = np.concatenate([np.array(c) * np.array(L) + 1.2 * rng.standard_normal((N // 2, 3))
                        for c in ((0.4, 0.5, 0.3), (0.98, 0.02, 0.97))]).astype(T)
    F, lam = (rng.standard_normal((N, 3)).astype(T) for _ in range(2))
    got = []
    for mode in "10":
        forced.setenv("FFCM_PENCIL", mode)
        cfg = ffcm.FFCMConfig(T, **kw_of(L, N, M, M_G=MG, R_c=0.3 * min(L)))
        res = [ffcm.mobility(np.empty_like(Y), cfg, Y, F) for _ in range(2)]
        A = ffcm.FFCMMobility(cfg, Y)
        res += [A @ F, A @ lam]
        V, pull = ffcm.rrule_mobility(cfg, Y, F)
        res += [V, *pull(lam)]
        got.append(res)
    for i, (a, b) in enumerate(zip(*got)):
        assert rel_l2(a, b) < TOL[T] * (10 if i > 4 else 1)   # (gradients cancel, as above)


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("overlap", ["0", "1"])
def test_pencil_solve_with_the_correction_beside_it(ffcm, forced, T, overlap):
    """Both orders of the pair correction, from host arrays and from device
    arrays on a caller's stream, the first solve of a configuration included."""
    import torch
    forced.setenv("FFCM_OVERLAP_PAIRS", overlap)
    M, N = (50, 36, 42), 700
    L = tuple(0.55 * m for m in M)
    kw = kw_of(L, N, M, M_G=9, R_c=3.0)
    prod, ora = both(ffcm, T, **kw)
    Y, F = _inputs(T, L, N, "uniform", 17)
    ref = O.apply(ora, Y, F)
    for _ in range(3):
        assert rel_l2(ffcm.mobility(np.empty_like(Y), prod, Y, F), ref) < TOL[T]
    cfg, s = ffcm.FFCMConfig(T, **kw), torch.cuda.Stream()
    with torch.cuda.stream(s):
        Yd, Fd = torch.from_numpy(Y).cuda(), torch.from_numpy(F).cuda()
        for _ in range(3):
            V = ffcm.mobility(torch.empty_like(Fd), cfg, Yd, Fd)
            s.synchronize()
            assert rel_l2(V.cpu().numpy(), ref) < TOL[T]
