"""The term groups of a right-hand side called one by one against the fused call: equal bitwise."""
import numpy as np
import pytest
import torch

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu

# (operator, dim, finest level, grid): rows long enough to be shared out (2^6 and more neighbours) in one
# dimension and not in another; grids whose terms go in several pieces; and, in five and six dimensions,
# blocks whose parts fit the column form of the last FP32 sweep for one group but not for all (35 x 243
# and 30 x 729 entries against 8,192), on grids refined along one dimension: more outputs than those that
# four lanes share, few enough elements for all terms at once, rows of more than four neighbours
CASES = [("burgers", 2, 8, "sparse"), ("burgers", 3, 7, "sparse"), ("burgers", 2, 7, "adaptive"),
         ("hermite", 2, 8, "sparse"), ("wave", 2, 7, "full"), ("wave", 2, 8, "adaptive"),
         ("burgers", 4, 3, "sparse"), ("burgers", 5, 3, "sparse"), ("wave", 3, 5, "full"),
         ("burgers", 4, 4, "full"), ("wave", 5, 5, "line"), ("burgers", 6, 4, "line")]


@pytest.mark.parametrize("kind,dim,nmax,shape", CASES)
@pytest.mark.parametrize("prec", [amdg.FP64, amdg.MIXED])
def test_groups_one_by_one_equal_the_fused_call(ctx, kind, dim, nmax, shape, prec):
    """Random coefficients, the same terms in the same order: no bit differs."""
    if shape == "adaptive":
        g = amdg.Grid(ctx, dim, nmax, 2, level_init=3)
        g.init_separable_adaptive(O.wave_ic_terms(dim) if kind == "wave" else O.burgers_ic_terms(dim), 1e-4)
    else:
        g = amdg.Grid(ctx, dim, nmax, 2, sparse=shape != "full")
    if shape == "line":  # every level of the last dimension, its coarse ones also at the first of the first
        levels, _ = g.elements()
        lv = np.asarray(levels).reshape(g.num_elements, dim)
        keep = (lv[:, :-1].sum(1) == 0) | ((lv[:, 0] == 1) & (lv[:, 1:-1].sum(1) == 0) & (lv[:, -1] <= 2))
        g.set_coefficients(np.ones((g.num_elements, g.block)) * keep[:, None])
        g.coarsen(0.5)
        assert g.num_elements == keep.sum()
    rng = np.random.default_rng(dim)
    g.set_coefficients(rng.standard_normal((g.num_elements, g.block)))
    du = torch.from_numpy(g.coefficients().reshape(-1).copy()).cuda()
    fused = torch.zeros_like(du)
    if kind == "wave":
        op = amdg.WaveOperator(g, 10.0)
        calls = [(op.interpolate, op.INTERP_GRADU), (op.rhs_add, op.RHS_FLX_GRADU), (op.rhs_add, op.RHS_VOL),
                 (op.interpolate, op.INTERP_U), (op.rhs_add, op.RHS_FLX_U), (op.rhs_add, op.RHS_IPDG)]
    else:
        op = amdg.BurgersOperator(g, 0.825, hermite=kind == "hermite")
        calls = [(lambda _, prec: op.interpolate(prec), None)]
        calls += [(op.rhs_add, group) for group in (op.RHS_VOL, op.RHS_FLX, op.RHS_PENALTY)]
    torch.cuda.synchronize()
    op.rhs_device(du.data_ptr(), fused.data_ptr(), prec)
    g.set_rhs_zero()
    for call, arg in calls:
        call(arg, prec=prec)
    ctx.synchronize()
    assert np.array_equal(g.rhs().reshape(-1), fused.cpu().numpy())
    op.close()
    g.close()
