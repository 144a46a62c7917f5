"""Failure detection without a GPU fault: a bounded device-side wait made to give up at once must
come back as AMDG_ERR_TIMEOUT with the state left as it was, and device allocations made to fail
must come back as AMDG_ERR_NOMEM, with the library usable afterwards."""
import numpy as np
import pytest
import torch

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu

TIMEOUT, NOMEM = 4, 7


def test_bulk_copy_wait_timeout_reports_and_leaves_the_state(ctx):
    """The bulk-copy linear kernel with a wait limit of 0 polls: every warp's first wait gives up,
    the kernel drains the copies it issued (their own bound) and returns without writing; the call
    fails with AMDG_ERR_TIMEOUT and the coefficients are bitwise unchanged.  With the default
    limit restored the same step succeeds and equals a step of a fresh operator."""
    g = amdg.Grid(ctx, 3, 6, 2)
    g.init_separable(O.sin_sum_terms(3))
    u0 = g.coefficients().copy()
    op = amdg.LinearOperator(g, [1.0, -0.5, 0.25])
    op.set_variant(amdg.MIXED, 2)
    op.set_wait_limit(0)
    with pytest.raises(amdg.AmdgError) as ei:
        op.rk3_steps(1e-3, 1, amdg.MIXED)
    assert ei.value.status == TIMEOUT
    ctx.synchronize()
    assert np.array_equal(g.coefficients(), u0)
    op.set_wait_limit(1 << 22)
    op.rk3_steps(1e-3, 1, amdg.MIXED)
    ctx.synchronize()
    stepped = g.coefficients().copy()
    g.set_coefficients(u0)
    op2 = amdg.LinearOperator(g, [1.0, -0.5, 0.25])
    op2.set_variant(amdg.MIXED, 2)
    op2.rk3_steps(1e-3, 1, amdg.MIXED)
    ctx.synchronize()
    assert np.array_equal(g.coefficients(), stepped)
    op.close()
    op2.close()
    g.close()


def test_device_allocation_failure_reports_nomem(ctx):
    """Every device allocation made to fail: grid, operator and classifier creation report
    AMDG_ERR_NOMEM (not a CUDA error, not a crash); after some successful allocations the failure
    surfaces from a later call the same way; with the hook off the library works again."""
    lib = amdg.load()
    try:
        lib.amdg_debug_fail_device_allocations(0)
        with pytest.raises(amdg.AmdgError) as ei:
            amdg.Grid(ctx, 2, 5, 2)
        assert ei.value.status == NOMEM
        with pytest.raises(amdg.AmdgError) as ei:
            amdg.MLP(ctx, 45, 64, 3, 3, seed=1)
        assert ei.value.status == NOMEM
        lib.amdg_debug_fail_device_allocations(-1)
        g = amdg.Grid(ctx, 2, 5, 2, level_init=3)
        g.init_separable_adaptive(O.burgers_ic_terms(2), 1e-4)
        # the operator's own allocations fail part-way
        for after in (0, 3, 9):
            lib.amdg_debug_fail_device_allocations(after)
            with pytest.raises(amdg.AmdgError) as ei:
                amdg.BurgersOperator(g, 0.825)
            assert ei.value.status == NOMEM, after
        lib.amdg_debug_fail_device_allocations(-1)
        op = amdg.BurgersOperator(g, 0.825)
        op.adaptive_step(0.1, 0.75, 1e-4, 1e-5)
        ctx.synchronize()
        assert np.all(np.isfinite(g.coefficients()))
        op.close()
        g.close()
    finally:
        lib.amdg_debug_fail_device_allocations(-1)


def _rhs(ctx, op, u):
    du = torch.from_numpy(u.reshape(-1).copy()).cuda()
    out = torch.zeros_like(du)
    torch.cuda.synchronize()
    op.rhs_device(du.data_ptr(), out.data_ptr())
    ctx.synchronize()
    return out.cpu().numpy()


def test_sweep_lists_that_could_not_be_stored_are_stored_by_the_next_call(ctx):
    """The sweep trees of a variant and the sweep plans of the term groups are built on first use.  With
    no device memory left for them the call fails with AMDG_ERR_NOMEM, and a later call stores them:
    the same results as of an operator that never failed."""
    lib = amdg.load()
    g = amdg.Grid(ctx, 3, 3, 2)
    g.init_separable(O.wave_ic_terms(3))
    u = g.coefficients()
    op, fresh = amdg.WaveOperator(g, 10.0), amdg.WaveOperator(g, 10.0)
    want = _rhs(ctx, fresh, u)
    fresh.set_sweep_variant(0)
    want0 = _rhs(ctx, fresh, u)

    def by_groups():
        g.set_rhs_zero()
        for call, arg in ((op.interpolate, op.INTERP_GRADU), (op.rhs_add, op.RHS_FLX_GRADU), (op.rhs_add, op.RHS_VOL),
                          (op.interpolate, op.INTERP_U), (op.rhs_add, op.RHS_FLX_U), (op.rhs_add, op.RHS_IPDG)):
            call(arg)
        ctx.synchronize()
        return g.rhs().reshape(-1)

    g.set_rhs_zero()
    try:
        lib.amdg_debug_fail_device_allocations(0)
        with pytest.raises(amdg.AmdgError) as ei:
            by_groups()
        assert ei.value.status == NOMEM
        lib.amdg_debug_fail_device_allocations(-1)
        assert np.array_equal(by_groups(), want)
        assert np.array_equal(_rhs(ctx, op, u), want)
        op.set_sweep_variant(0)
        lib.amdg_debug_fail_device_allocations(0)
        with pytest.raises(amdg.AmdgError) as ei:
            _rhs(ctx, op, u)
        assert ei.value.status == NOMEM
        lib.amdg_debug_fail_device_allocations(-1)
        assert np.array_equal(_rhs(ctx, op, u), want0)
    finally:
        lib.amdg_debug_fail_device_allocations(-1)
    op.close()
    fresh.close()
    g.close()


def test_refinement_that_ran_out_of_memory_can_be_repeated(ctx):
    """A refinement whose allocations fail after its marks leaves the element set as it was, and the same
    call with memory adds the same elements as on a grid that never failed."""
    lib = amdg.load()
    grids = []
    for _ in range(2):
        g = amdg.Grid(ctx, 3, 6, 2, level_init=3)
        g.init_separable_adaptive(O.burgers_ic_terms(3), 1e-3)
        grids.append(g)
    want, g = grids
    n = g.num_elements
    try:
        after, failed = 0, 0
        while True:
            lib.amdg_debug_fail_device_allocations(after)
            try:
                g.refine(1e-6)
                break
            except amdg.AmdgError as err:
                assert err.status == NOMEM
                failed += 1
                after += 1
        assert failed > 1
    finally:
        lib.amdg_debug_fail_device_allocations(-1)
    want.refine(1e-6)
    assert g.num_elements > n
    assert all(np.array_equal(a, b) for a, b in zip(g.elements(), want.elements()))
    assert np.array_equal(g.coefficients(), want.coefficients())
    g.close()
    want.close()
