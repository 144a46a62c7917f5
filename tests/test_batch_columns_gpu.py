"""Batches on both sides of the line between one and np columns per thread (FP32 column kernels,
k = 2): a solve of a batch large enough for np columns equals, bit for bit, the same solve in a batch
too small for them -- the operations of an output and their order are the same."""
import numpy as np
import pytest

import amdg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nmax,level,k", [(3, 5, 5, 2), (4, 4, 4, 2), (5, 3, 3, 2), (6, 3, 2, 2), (3, 5, 5, 1),
                                              (2, 6, 6, 2)])
def test_columns_per_thread_agree(ctx, dim, nmax, level, k):
    np1 = k + 1
    g = amdg.Grid(ctx, dim, nmax, k, level_init=level)
    rng = np.random.default_rng(10 * dim + k)
    u0 = rng.standard_normal((g.num_elements, np1**dim))
    per_element = max(1, np1 ** (dim - 2))  # threads per element with np columns each
    n = -(-1300 * 152 // (per_element * g.num_elements))
    vel = [list(rng.uniform(-1.0, 1.0, dim)) for _ in range(n)]
    dts = list(rng.uniform(0.5e-3, 1e-3, n))
    kernels = [2, amdg.Batch.DF_COLUMN_FIRST + 2]
    if dim <= 3:
        kernels += [0, 4, amdg.Batch.DF_COLUMN_FIRST, amdg.Batch.PERSIST_FIRST, amdg.Batch.PERSIST_FIRST + 2]
    picks = [0, n - 1]

    def run(solves, kernel):
        g.set_coefficients(u0)
        b = amdg.Batch(ctx, [g] * len(solves), [vel[i] for i in solves])
        b.set_dt([dts[i] for i in solves])
        b.set_kernel(amdg.MIXED, kernel)
        b.rk3_steps(2, amdg.MIXED, use_graph=False)
        ctx.synchronize()
        out = []
        for i in picks:
            b.store(solves.index(i))
            out.append(g.coefficients().copy())
        b.close()
        return out

    for kernel in kernels:
        big, small = run(list(range(n)), kernel), run(picks, kernel)
        for a, b in zip(big, small):
            assert np.array_equal(a, b), kernel
    g.close()
