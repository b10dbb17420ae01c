"""A call that fails leaves the configurations that exist as they were: the next
solve on them neither reports the earlier error nor meets counters that a call
given up half way has left behind."""
import numpy as np
import pytest

from gpu_helpers import both, kw_of, rel_l2

import ffcm_oracle as O

pytestmark = pytest.mark.gpu
TOL = {np.float32: 1e-5, np.float64: 1e-10}   # the suite's end-to-end bounds


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M,MG", [((64, 64, 64), 8), ((90, 80, 96), 9)])
def test_solve_after_a_configuration_that_did_not_fit(ffcm, monkeypatch, T, M, MG):
    monkeypatch.setenv("FFCM_PENCIL", "1")
    L = tuple(0.55 * m for m in M)
    prod, ora = both(ffcm, T, **kw_of(L, 300, M, M_G=MG, R_c=3.0))
    rng = np.random.default_rng(5)
    for _ in range(3):
        # a spectrum of 209 GB and more, refused by its one allocation
        huge = (2048, 2048, 4096 if T == np.float32 else 2048)
        with pytest.raises(MemoryError):
            ffcm.FFCMConfig(T, **kw_of(tuple(float(m) for m in huge), 4, huge, M_G=MG, R_c=900.0))
        Y = (rng.random((300, 3)) * np.array(L)).astype(T)
        F = rng.standard_normal((300, 3)).astype(T)
        assert rel_l2(ffcm.mobility(np.empty_like(Y), prod, Y, F), O.apply(ora, Y, F)) < TOL[T]
