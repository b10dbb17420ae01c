"""Mixed-radix transforms of the spectral Stokes solve against the oracle, at
line lengths that reach every butterfly, one to four stages, the odd x rows
(two rows a line, the last one alone), the primes beyond the register
butterflies, blocks with one and with two shared-memory buffers, and lines
whose twiddle table stays in global memory."""
import numpy as np
import pytest

from gpu_helpers import both, kw_of, rel_l2

import ffcm_oracle as O

pytestmark = pytest.mark.gpu

# an unnormalised transform of n points accumulates a relative error of about
# log2(n) rounding units in each direction (n <= 2^25 here), and the projector
# a few more
UNITS = 2 * 25 + 10


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M", [
    (4, 3, 5), (6, 9, 7), (36, 20, 25), (50, 18, 24), (22, 13, 11), (28, 15, 14), (33, 21, 35),
    (62, 17, 34), (61, 19, 23), (122, 61, 37), (27, 200, 12), (40, 12, 160), (30, 324, 10), (20, 14, 300),
    (480, 6, 10), (405, 5, 7), (1000, 4, 6), (6, 1000, 4), (4, 6, 1000), (8, 2100, 6), (6, 8, 2100),
    (64, 48, 32), (48, 64, 40), (3, 5, 3), (9000, 4, 6), (16000, 4, 4), (4, 6000, 6), (4, 10000, 4), (4, 4, 4200),
])
def test_stokes_solve_of_any_grid(ffcm, T, M):
    values = max(M[0] // 2 if M[0] % 2 == 0 else M[0], M[1], 3 * M[2])
    if 2 * values * 2 * np.dtype(T).itemsize > 200 * 1024:
        pytest.skip("two buffers of such a line need more shared memory than there is")
    kw = kw_of(tuple(float(m) for m in M), 1, M, M_G=2, R_c=min(M) / 2)
    prod, ora = both(ffcm, T, **kw)
    rng = np.random.default_rng(sum(M))
    f = rng.standard_normal(ora.force_density.shape).astype(T) + T(0.3)
    prod.set("FORCE_DENSITY", f)
    ora.force_density[:] = f
    ffcm.stokes_solve(prod)
    O.stokes_solve(ora)
    assert rel_l2(prod.fluid_velocity, ora.fluid_velocity) < UNITS * np.finfo(T).eps


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("M", [(64, 136, 32), (64, 32, 136), (60, 190, 24), (48, 24, 228), (96, 204, 30), (96, 30, 114)])
def test_prime_first_stage_of_many_warps(ffcm, T, M):
    """Lines whose first stage is a prime beyond the register butterflies (it
    reads the shared twiddle table at once), in blocks of several warps; a grid
    of other line lengths is solved before each solve, so that shared memory
    does not hold the right table from the solve before."""
    rng = np.random.default_rng(sum(M))
    grids = []
    for m in ((60, 150, 126), M):
        prod, ora = both(ffcm, T, **kw_of(tuple(float(n) for n in m), 1, m, M_G=2, R_c=min(m) / 2))
        f = rng.standard_normal(ora.force_density.shape).astype(T) + T(0.3)
        ora.force_density[:] = f
        O.stokes_solve(ora)
        grids.append((prod, f, ora.fluid_velocity))
    for _ in range(3):
        for prod, f, u in grids:
            prod.set("FORCE_DENSITY", f)
            ffcm.stokes_solve(prod)
            assert rel_l2(prod.fluid_velocity, u) < UNITS * np.finfo(T).eps
