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


# grids with k + 1 outputs per thread in mixed precision (at least 1,280 threads per multiprocessor so), both
# degrees that have the form: two to six dimensions, element counts that leave the last CTA partly filled
LARGE = [(2, 8, 2, "full"), (2, 8, 3, "full"), (3, 5, 2, "full"), (3, 5, 3, "full"), (4, 8, 2, "sparse"),
         (4, 7, 3, "sparse"), (5, 5, 3, "sparse"), (6, 5, 2, "sparse"), (6, 4, 3, "sparse")]


@pytest.mark.parametrize("dim,nmax,k,shape", LARGE)
def test_outputs_per_thread_match_the_oracle(ctx, dim, nmax, k, shape):
    """Two mixed steps on random coefficients against the oracle and the column kernel (1e-6, the bar of
    mixed steps)."""
    import torch

    g = amdg.Grid(ctx, dim, nmax, k, sparse=shape == "sparse")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert g.dof // (k + 1) >= 1280 * sms
    rng = np.random.default_rng(1000 * dim + 10 * nmax + k)
    vel = (rng.uniform(0.3, 1.0, dim) * rng.choice([-1.0, 1.0], dim)).tolist()
    u0 = rng.standard_normal((g.num_elements, g.block))
    op = amdg.LinearOperator(g, vel)
    dt = 0.1 / (2.0 ** nmax * sum(abs(v) for v in vel))
    out = []
    for variant in (0, 1) if (k + 1) ** (dim - 1) <= 256 else (0,):  # the column kernel takes columns of one CTA
        op.set_variant(amdg.MIXED, variant)
        g.set_coefficients(u0)
        op.rk3_steps(dt, 2, amdg.MIXED)
        ctx.synchronize()
        out.append(g.coefficients().copy())
    lv, sp = g.elements()
    ref = O.linear_rk3(dim, nmax, k, lv, sp, vel, u0, dt, 2)
    assert np.abs(out[0] - ref).max() <= 1e-6 * np.abs(ref).max()
    assert np.abs(out[0] - out[-1]).max() <= 1e-6 * np.abs(ref).max()
    op.close()
    g.close()
