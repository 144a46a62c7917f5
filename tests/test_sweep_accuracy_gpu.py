"""Accuracy of the planned transform sweeps on random coefficients: element by element, where a wrong or
missing neighbour of one element shows, and on average against the sweeps term by term."""
import numpy as np
import pytest
import torch

import amdg
import amdg_oracle as O

pytestmark = pytest.mark.gpu


def make(ctx, kind, dim, nmax, shape):
    if shape == "adaptive":
        g = amdg.Grid(ctx, dim, nmax, 2, level_init=3)
        g.init_separable_adaptive(O.wave_ic_terms(dim) if kind == "wave" else O.burgers_ic_terms(dim), 2e-6)
    else:
        g = amdg.Grid(ctx, dim, nmax, 2, sparse=shape == "sparse")
    op = amdg.WaveOperator(g, 10.0) if kind == "wave" else amdg.BurgersOperator(g, 0.825, hermite=kind == "hermite")
    return g, op


def randomise(g, seed, decay):
    """Normal coefficients, an element's scaled by 2^(-decay times its level sum)."""
    levels, _ = g.elements()
    scale = 2.0 ** (-decay * np.asarray(levels).reshape(g.num_elements, -1).sum(1))
    u = np.random.default_rng(seed).standard_normal((g.num_elements, g.block)) * scale[:, None]
    g.set_coefficients(u)
    return u


def rhs(ctx, g, op, prec):
    du = torch.from_numpy(g.coefficients().reshape(-1).copy()).cuda()
    out = torch.zeros_like(du)
    torch.cuda.synchronize()
    op.rhs_device(du.data_ptr(), out.data_ptr(), prec)
    ctx.synchronize()
    return out.cpu().numpy().reshape(g.num_elements, g.block)


def per_element(err, ref):
    return (np.linalg.norm(err, axis=1) / np.linalg.norm(ref, axis=1)).max()


# both sides of the size up to which lanes share an entry, rows to share out, FP32 columns with one and
# several dimensions in a node, odd lengths of rows, blocks in windows
SHAPES = [("burgers", 3, 4, "sparse"), ("burgers", 3, 7, "sparse"), ("burgers", 2, 8, "sparse"),
          ("burgers", 3, 7, "adaptive"), ("burgers", 4, 5, "sparse"), ("burgers", 5, 4, "sparse"),
          ("burgers", 6, 3, "sparse"), ("hermite", 2, 6, "sparse"), ("hermite", 2, 8, "sparse"),
          ("wave", 2, 5, "full"), ("wave", 2, 7, "full"), ("wave", 3, 5, "sparse"), ("wave", 4, 4, "sparse")]


@pytest.mark.parametrize("kind,dim,nmax,shape", SHAPES)
def test_mixed_right_hand_side_element_by_element(ctx, kind, dim, nmax, shape):
    """The largest relative error of an element's block against FP64 stays within four times that of the
    sweeps term by term (FP32 roundings of the same sums in another order); a neighbour left out or a
    wrong block would make it some 1e-2."""
    g, op = make(ctx, kind, dim, nmax, shape)
    randomise(g, 3, 1.0)
    errs = []
    for variant in (-1, 0):
        op.set_sweep_variant(variant)
        exact = rhs(ctx, g, op, amdg.FP64)
        errs.append(per_element(rhs(ctx, g, op, amdg.MIXED) - exact, exact))
    assert errs[0] <= 4.0 * errs[1], errs
    op.close()
    g.close()


@pytest.mark.parametrize("kind,dim,nmax", [("burgers", 2, 7), ("burgers", 3, 5), ("burgers", 4, 3), ("wave", 2, 6)])
def test_right_hand_side_element_by_element_against_the_oracle(ctx, kind, dim, nmax):
    """FP64: every element's block to 1e-10 of its norm (a block is up to some 1e2 smaller than the terms
    that it is the sum of; the terms agree to the 1e-12 of the whole field)."""
    g, op = make(ctx, kind, dim, nmax, "sparse")
    u = randomise(g, 4, 1.0)
    levels, support = g.elements()
    if kind == "wave":
        ref = O.wave_rhs(dim, nmax, 2, levels, support, u, 10.0)
    else:
        ref = O.burgers_rhs(dim, nmax, 2, levels, support, u, 0.825)[0]
    ref = np.asarray(ref).reshape(g.num_elements, g.block)
    assert per_element(rhs(ctx, g, op, amdg.FP64) - ref, ref) <= 1e-10
    op.close()
    g.close()


@pytest.mark.parametrize("kind,dim,nmax,shape", [("hermite", 2, 6, "sparse"), ("hermite", 2, 7, "adaptive"),
                                                 ("burgers", 2, 5, "sparse"), ("burgers", 3, 5, "sparse"),
                                                 ("wave", 2, 4, "full"), ("wave", 2, 5, "sparse")])
def test_mixed_error_is_no_larger_than_term_by_term(ctx, kind, dim, nmax, shape):
    """The L2 error of the mixed right-hand side against FP64, geometric mean over 40 states with the
    coefficients of a smooth function (2^-3 per level): no larger than that of the sweeps term by term
    with a warp per element."""
    g, op = make(ctx, kind, dim, nmax, shape)
    logs = []
    for seed in range(40):
        randomise(g, seed, 3.0)
        errs = []
        for variant in (-1, 2):
            op.set_sweep_variant(variant)
            exact = rhs(ctx, g, op, amdg.FP64)
            errs.append(np.linalg.norm(rhs(ctx, g, op, amdg.MIXED) - exact))
        logs.append(np.log(errs[0] / errs[1]))
    assert np.exp(np.mean(logs)) <= 1.0
    op.close()
    g.close()


# grids on which not all terms fit one launch sequence: the fields of the wave one by one and its groups in
# pieces; four and eight pieces of the transforms to point values, groups term by term
PIECES = [("wave", 3, 5), ("burgers", 4, 4), ("burgers", 5, 3)]


@pytest.mark.parametrize("kind,dim,nmax", PIECES)
def test_terms_in_pieces_element_by_element(ctx, kind, dim, nmax):
    """FP64 against the sweeps term by term to 1e-10 of an element's norm, mixed as above."""
    g, op = make(ctx, kind, dim, nmax, "full")
    randomise(g, 5, 1.0)
    exact, errs = [], []
    for variant in (-1, 0):
        op.set_sweep_variant(variant)
        exact.append(rhs(ctx, g, op, amdg.FP64))
        errs.append(per_element(rhs(ctx, g, op, amdg.MIXED) - exact[-1], exact[-1]))
    assert per_element(exact[0] - exact[1], exact[1]) <= 1e-10
    assert errs[0] <= 4.0 * errs[1], errs
    op.close()
    g.close()


@pytest.mark.parametrize("prec", [amdg.FP64, amdg.MIXED])
def test_sums_do_not_depend_on_an_earlier_larger_grid(ctx, prec):
    """A wave operator whose grid shrank from 32,768 elements, where its groups go in pieces, to the
    coarse levels: the same bits as of a new operator on that grid."""
    g, op = make(ctx, "wave", 3, 5, "full")
    levels, _ = g.elements()
    keep = np.asarray(levels).reshape(g.num_elements, -1).sum(1) <= 6
    u = np.random.default_rng(6).standard_normal((g.num_elements, g.block)) * keep[:, None]
    g.set_coefficients(u)
    rhs(ctx, g, op, prec)
    g.coarsen(1e-6)
    assert g.num_elements == keep.sum()
    got = rhs(ctx, g, op, prec)
    new = amdg.WaveOperator(g, 10.0)
    assert np.array_equal(got, rhs(ctx, g, new, prec))
    new.close()
    op.close()
    g.close()


def test_slices_of_the_terms_are_allocated_for_the_sweeps_term_by_term_only(ctx):
    """The planned sweeps write no slice per term: their operator holds that memory only after a variant
    that does was chosen (32,768 elements x 64 points, some 20 terms: hundreds of MB)."""
    g = amdg.Grid(ctx, 3, 5, 2, sparse=False)
    op = amdg.BurgersOperator(g, 0.825)
    randomise(g, 8, 1.0)
    exact = rhs(ctx, g, op, amdg.FP64)
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(rhs(ctx, g, op, amdg.FP64), exact)
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    op.set_sweep_variant(0)
    rhs(ctx, g, op, amdg.FP64)
    assert free - torch.cuda.mem_get_info()[0] > 128 << 20
    op.close()
    g.close()
