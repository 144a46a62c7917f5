"""Values that are not finite in the planned sweeps: they reach the entries that they reach term by term."""
import numpy as np
import pytest
import torch

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dim,nmax", [("burgers", 2, 8), ("burgers", 3, 5), ("hermite", 2, 7), ("wave", 2, 7),
                                           ("wave", 3, 4)])
@pytest.mark.parametrize("prec", [amdg.FP64, amdg.MIXED])
def test_non_finite_entries_are_those_of_the_sweeps_term_by_term(ctx, kind, dim, nmax, prec):
    """One coefficient of a fine element NaN, infinite, or (FP64) so large that the first sweep overflows:
    the same entries of the right-hand side and of the point values are not finite.  Then a finite state
    again: the same bits as before."""
    g = amdg.Grid(ctx, dim, nmax, 2)
    op = amdg.WaveOperator(g, 10.0) if kind == "wave" else amdg.BurgersOperator(g, 0.825, hermite=kind == "hermite")
    levels, _ = g.elements()
    u0 = np.random.default_rng(dim).standard_normal((g.num_elements, g.block))
    fine = np.flatnonzero(np.asarray(levels).reshape(g.num_elements, dim)[:, 0] == nmax - 1)[3]

    def results(u, variant):
        op.set_sweep_variant(variant)
        du = torch.from_numpy(u.reshape(-1).copy()).cuda()
        outs = [torch.zeros_like(du)]
        torch.cuda.synchronize()
        op.rhs_device(du.data_ptr(), outs[0].data_ptr(), prec)
        if kind != "wave":
            outs.append(torch.zeros(g.num_elements * 4 ** dim, dtype=torch.float64, device="cuda"))
            torch.cuda.synchronize()
            op.point_values_device(du.data_ptr(), outs[1].data_ptr(), prec)
        ctx.synchronize()
        return [o.cpu().numpy() for o in outs]

    before = results(u0, -1)
    values = [np.nan, np.inf, -np.inf] + ([1e308] if prec == amdg.FP64 else [])
    for value in values:
        u = u0.copy()
        u[fine, 1] = value
        for got, want in zip(results(u, -1), results(u, 0)):
            assert not np.isfinite(want).all()
            assert np.array_equal(np.isfinite(got), np.isfinite(want)), value
    for got, want in zip(results(u0, -1), before):
        assert np.array_equal(got, want)
    op.close()
    g.close()


@pytest.mark.parametrize("kind,dim,nmax", [("burgers", 2, 7), ("hermite", 2, 6), ("wave", 2, 6)])
@pytest.mark.parametrize("prec", [amdg.FP64, amdg.MIXED])
def test_steps_spread_them_alike(ctx, kind, dim, nmax, prec):
    """Three steps in one call (stages that read what another stage wrote, a step replayed as a graph) from
    a state with one infinite coefficient; then a finite state again, whose steps keep their bits."""
    g = amdg.Grid(ctx, dim, nmax, 2)
    u0 = np.random.default_rng(7).standard_normal((g.num_elements, g.block))
    levels, _ = g.elements()
    fine = np.flatnonzero(np.asarray(levels).reshape(g.num_elements, dim)[:, 0] == nmax - 1)[1]
    bad = u0.copy()
    bad[fine, 1] = np.inf
    outs = {}
    for variant in (-1, 0):
        op = amdg.WaveOperator(g, 10.0) if kind == "wave" else amdg.BurgersOperator(g, 0.825, hermite=kind == "hermite")
        op.set_sweep_variant(variant)
        for name, u in (("first", u0), ("bad", bad), ("again", u0)):
            g.set_coefficients(u)
            if kind == "wave":
                g.set_velocity(np.zeros_like(u))
                op.rk4_steps(1e-6, 3, prec)
            else:
                op.rk3_steps(1e-6, 3, prec)
            ctx.synchronize()
            outs[variant, name] = g.coefficients().copy()
        op.close()
    assert not np.isfinite(outs[0, "bad"]).all()
    assert np.array_equal(np.isfinite(outs[-1, "bad"]), np.isfinite(outs[0, "bad"]))
    assert np.isfinite(outs[-1, "first"]).all()
    assert np.array_equal(outs[-1, "first"], outs[-1, "again"])
    g.close()


@pytest.mark.parametrize("hermite", [False, True])
def test_stages_that_overflow_spread_alike(ctx, hermite):
    """One FP64 step from a finite state with one coefficient so large that its square is near the largest
    double: the stages overflow, and the later ones read what the earlier ones wrote (the look at the state
    found nothing).  The same entries are not finite as with the sweeps term by term."""
    g = amdg.Grid(ctx, 2, 6, 2)
    u = np.random.default_rng(9).standard_normal((g.num_elements, g.block))
    levels, _ = g.elements()
    fine = np.flatnonzero(np.asarray(levels).reshape(g.num_elements, 2)[:, 0] == 5)[2]
    outs = []
    for variant in (-1, 0):
        v = u.copy()
        v[fine, 1] = 1e153
        g.set_coefficients(v)
        op = amdg.BurgersOperator(g, 0.825, hermite=hermite)
        op.set_sweep_variant(variant)
        op.rk3_steps(1e-3, 1)
        ctx.synchronize()
        outs.append(g.coefficients().copy())
        op.close()
    assert not np.isfinite(outs[1]).all()
    assert np.array_equal(np.isfinite(outs[0]), np.isfinite(outs[1]))
    g.close()
