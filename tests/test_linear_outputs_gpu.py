"""The output-parallel linear stage (variant 0) over the sizes where its kernels change."""
import numpy as np
import pytest

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu

# from three outputs (one warp, partly filled) over grids of a few warps (lists split over four warps)
# to ones with an output per thread and, mixed, k + 1 outputs per thread; each degree, one to six dimensions
SIZES = [(1, 0, 2), (1, 1, 1), (1, 7, 3), (2, 3, 1), (2, 6, 2), (2, 5, 3), (3, 3, 2), (3, 6, 3), (4, 3, 3), (4, 4, 2),
         (5, 4, 1), (4, 6, 3), (5, 4, 3), (5, 6, 2), (6, 3, 2), (6, 2, 1)]


@pytest.mark.parametrize("dim,nmax,k", SIZES)
@pytest.mark.parametrize("prec,tol", [(amdg.FP64, 1e-12), (amdg.MIXED, 1e-6)])
def test_output_parallel_steps_match_the_oracle(ctx, dim, nmax, k, prec, tol):
    """Two SSP-RK3 steps against the oracle: FP64 sums of at most a few hundred terms of both signs
    (1e-12 of the largest entry, the bar of the linear path), mixed 1e-6 (its bar for steps)."""
    g = amdg.Grid(ctx, dim, nmax, k)
    rng = np.random.default_rng(100 * dim + 10 * nmax + k)
    vel = (rng.uniform(0.3, 1.0, dim) * rng.choice([-1.0, 1.0], dim)).tolist()
    u0 = rng.standard_normal((g.num_elements, g.block))
    g.set_coefficients(u0)
    op = amdg.LinearOperator(g, vel)
    op.set_variant(prec, 0)
    dt = 0.1 / (2.0 ** nmax * sum(abs(v) for v in vel))
    op.rk3_steps(dt, 2, prec)
    ctx.synchronize()
    lv, sp = g.elements()
    ref = O.linear_rk3(dim, nmax, k, lv, sp, vel, u0, dt, 2)
    assert np.abs(g.coefficients() - ref).max() <= tol * np.abs(ref).max()
    op.close()
    g.close()
