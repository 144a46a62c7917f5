"""The mixed stage state's FP32 (hi, lo) pairs: split from and merged into FP64."""
import numpy as np
import pytest

import amdg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nmax,k", [(1, 0, 1), (1, 0, 2), (2, 0, 2), (1, 3, 2), (2, 3, 1), (3, 2, 2), (2, 5, 3)])
def test_mixed_step_of_length_zero_returns_the_state(ctx, dim, nmax, k):
    """dt = 0: a step only splits, combines (3/4 u + 1/4 u, 1/3 u + 2/3 u) and merges.  Entries from
    1e-30 to 1e30, zeros of both signs and parts below the FP32 normal range among them, sizes that
    leave one to three entries after the last group of four: each comes back to a few units of the
    pairs' 2^-48 (six roundings of the combinations; 2^-44 is asserted), or within the smallest
    normal float where its low part has no normal float."""
    g = amdg.Grid(ctx, dim, nmax, k)
    rng = np.random.default_rng(dim * 100 + nmax * 10 + k)
    u = rng.standard_normal(g.dof) * 10.0 ** rng.uniform(-30, 30, g.dof)
    u[::5] = np.resize([0.0, -0.0, 2.0 ** -140, 1.0 + 2.0 ** -25, -1.0], u[::5].shape)
    g.set_coefficients(u)
    op = amdg.LinearOperator(g, [0.0] * dim)
    op.rk3_steps(0.0, 1, amdg.MIXED)
    ctx.synchronize()
    got = g.coefficients().reshape(-1)
    assert (np.abs(got - u) <= 2.0 ** -44 * np.abs(u) + 2.0 ** -126).all()
    op.close()
    g.close()
