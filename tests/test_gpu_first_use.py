"""A configuration's first calls, which allocate and zero buffers, while other
work keeps the legacy default stream busy: the zeroing must come before the
call's own writes, whatever that stream does."""
import numpy as np
import pytest

from gpu_helpers import both, kw_of, rel_l2

import ffcm_oracle as O

pytestmark = pytest.mark.gpu
TOL = {np.float32: 1e-5, np.float64: 1e-10}   # the suite's end-to-end bounds


@pytest.fixture
def busy():
    """Queues some 60 ms of work on the legacy stream."""
    import torch
    x = torch.zeros(1 << 28, device="cuda")

    def queue():
        for _ in range(200):
            x.add_(1.0)

    torch.cuda.synchronize()
    yield queue
    torch.cuda.synchronize()


def _inputs(T, L, N):
    rng = np.random.default_rng(N)
    return (rng.random((N, 3)) * np.array(L)).astype(T), rng.standard_normal((N, 3)).astype(T)


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("pencil", ["0", "1"])
@pytest.mark.parametrize("arrays", ["host", "device"])
def test_first_solve_on_the_real_grids(ffcm, busy, monkeypatch, T, pencil, arrays):
    import torch
    monkeypatch.setenv("FFCM_PENCIL", pencil)
    M = (90, 80, 96)
    L = tuple(0.55 * m for m in M)
    prod, ora = both(ffcm, T, **kw_of(L, 500, M, M_G=9, R_c=3.0))
    Y, F = _inputs(T, L, 500)
    ref = O.apply(ora, Y, F)
    if arrays == "host":
        busy()
        V = ffcm.mobility(np.empty_like(Y), prod, Y, F)
    else:
        s = torch.cuda.Stream()
        Yd, Fd = torch.from_numpy(Y).cuda(), torch.from_numpy(F).cuda()
        Vd = torch.empty_like(Fd)
        torch.cuda.synchronize()
        busy()
        with torch.cuda.stream(s):
            ffcm.mobility(Vd, prod, Yd, Fd)
        s.synchronize()
        V = Vd.cpu().numpy()
    assert rel_l2(V, ref) < TOL[T]


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M,MG", [((64, 64, 64), 8), ((90, 80, 96), 9)])
def test_first_gradient_and_cg(ffcm, busy, T, M, MG):
    L = tuple(0.55 * m for m in M)
    kw = kw_of(L, 400, M, M_G=MG, R_c=3.0)
    Y, F = _inputs(T, L, 400)
    cfg = ffcm.FFCMConfig(T, **kw)
    target = (0.5 * F).astype(T)
    busy()
    first = ffcm.objective_gradient(cfg, Y, F, target)
    again = ffcm.objective_gradient(cfg, Y, F, target)
    for a, b in zip(first, again):
        assert rel_l2(a, b) < TOL[T]
    cfg = ffcm.FFCMConfig(T, **kw)
    A = ffcm.FFCMMobility(cfg, Y)
    busy()
    first = ffcm.cg(A, F, reltol=0.0, maxiter=4)
    again = ffcm.cg(A, F, reltol=0.0, maxiter=4)
    assert rel_l2(first, again) < TOL[T]


def test_overlapped_solve_allocates_nothing(ffcm, monkeypatch):
    """The first solve with the correction on the side stream, which a
    configuration takes some solves after its first, works in memory from the
    configuration's creation."""
    import torch
    monkeypatch.setenv("FFCM_OVERLAP_PAIRS", "1")
    N, M = 1_000_000, 256
    L = (0.9 * M,) * 3
    g = torch.Generator("cuda")
    g.manual_seed(4)
    Y = torch.rand(N, 3, generator=g, device="cuda") * L[0]
    F = torch.randn(N, 3, generator=g, device="cuda")
    V = torch.empty_like(F)
    kw = kw_of(L, N, M, R_c=3.0)
    warm = ffcm.FFCMConfig(np.float32, **kw)      # loads the kernels
    ffcm.mobility(V, warm, Y, F)
    cfg = ffcm.FFCMConfig(np.float32, **kw)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ffcm.mobility(V, cfg, Y, F)
    torch.cuda.synchronize()
    # (the pair terms of N particles are 12 MB; streams and events take some room)
    assert before - torch.cuda.mem_get_info()[0] < 8 << 20
