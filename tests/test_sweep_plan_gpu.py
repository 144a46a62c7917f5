"""The planned transform sweeps (the default) against the sweeps term by term (sweep variant 0)."""
import numpy as np
import pytest
import torch

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu

# (operator, dim, finest level, grid): two to six dimensions, levels below and above the length
# from which a row's neighbours are shared out (2^6 and more), blocks larger than one window of the
# last sweep (5 and 6 dimensions), element counts that leave CTAs partly filled, the empty level
CASES = [("burgers", 2, 0, "sparse"), ("burgers", 2, 1, "sparse"),
         ("burgers", 2, 8, "sparse"), ("burgers", 2, 7, "adaptive"), ("burgers", 2, 6, "full"),
         ("burgers", 3, 6, "sparse"), ("burgers", 3, 7, "adaptive"), ("burgers", 4, 3, "sparse"),
         ("burgers", 5, 2, "sparse"), ("burgers", 6, 1, "sparse"), ("hermite", 2, 7, "sparse"),
         ("hermite", 2, 8, "adaptive"), ("wave", 2, 6, "full"),
         ("wave", 2, 8, "adaptive"), ("wave", 3, 4, "sparse"), ("wave", 4, 2, "sparse")]


@pytest.mark.parametrize("kind,dim,nmax,shape", CASES)
@pytest.mark.parametrize("prec,tol", [(amdg.FP64, 1e-12), (amdg.MIXED, 1e-4)])
def test_planned_sweeps_match_the_sweeps_term_by_term(ctx, kind, dim, nmax, shape, prec, tol):
    """Same transforms, sums in another order: equal to rounding (FP64: 1e-12 of the largest entry;
    mixed: the 1e-4 of the mixed right-hand side, whose FP32 terms cancel), and the same from one
    evaluation to the next."""
    if shape == "adaptive":
        g = amdg.Grid(ctx, dim, nmax, 2, level_init=min(3, nmax))
        g.init_separable_adaptive(O.wave_ic_terms(dim) if kind == "wave" else O.burgers_ic_terms(dim), 1e-4)
    else:
        g = amdg.Grid(ctx, dim, nmax, 2, sparse=shape == "sparse")
        g.init_separable(O.burgers_ic_terms(dim))
    if kind == "wave":
        op = amdg.WaveOperator(g, 10.0)
    else:
        op = amdg.BurgersOperator(g, 0.825, hermite=kind == "hermite")
    du = torch.from_numpy(g.coefficients().reshape(-1).copy()).cuda()
    outs = []
    for variant in (-1, 0, -1):
        op.set_sweep_variant(variant)
        out = torch.zeros_like(du)
        torch.cuda.synchronize()
        op.rhs_device(du.data_ptr(), out.data_ptr(), prec)
        ctx.synchronize()
        outs.append(out.cpu().numpy())
    assert np.isfinite(outs[0]).all()
    assert np.abs(outs[0] - outs[1]).max() <= tol * np.abs(outs[1]).max()
    assert np.array_equal(outs[0], outs[2])
    op.close()
    g.close()
