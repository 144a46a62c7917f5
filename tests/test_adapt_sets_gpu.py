"""Device element-set changes and neighbour lists at the edges of their kernels, against the host
implementation: every number of lanes an element takes in the refinement (1 to 6 dimensions),
sets on both sides of the one-CTA coarsening (8,192 elements) and of the one-CTA scan of the row
counts, rows of one and of several dozen candidates, coarsenings that remove nothing and all but the
root.  The results are element sets, copied coefficients and right-hand sides over equal lists in equal
order: everything is compared bit for bit."""
import numpy as np
import pytest

import amdg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,nmax,k,level", [(1, 12, 2, 9), (1, 4, 1, 0), (2, 8, 1, 6), (2, 8, 2, 7), (3, 6, 2, 4),
                                              (4, 4, 1, 2), (5, 3, 1, 1), (6, 3, 1, 1)])
def test_set_changes_device_matches_host(dim, nmax, k, level):
    rng = np.random.default_rng(17 * dim + nmax)
    dev, host = amdg.Context(0), amdg.Context(0)
    host.set_adapt_mode(amdg.Context.ADAPT_HOST)
    grids = [amdg.Grid(c, dim, nmax, k, level_init=level) for c in (dev, host)]
    block = (k + 1) ** dim

    def same(what):
        (la, sa), (lb, sb) = grids[0].elements(), grids[1].elements()
        assert np.array_equal(la, lb) and np.array_equal(sa, sb), what
        assert np.array_equal(grids[0].coefficients(), grids[1].coefficients()), what

    for rnd, (eps, eta) in enumerate([(0.5, 0.3), (1.2, 0.9), (-1.0, 0.0), (0.9, 1e300)]):
        ne = grids[0].num_elements
        ind = rng.standard_normal((ne, block)) * rng.uniform(0, 2.0 / np.sqrt(block), (ne, 1))
        added = []
        for g in grids:
            d = torch.from_numpy(ind.reshape(-1).copy()).cuda()
            torch.cuda.synchronize()
            added.append(g.refine(eps, d.data_ptr()))
            g.ctx.synchronize()
            del d
        assert added[0] == added[1]
        ne = grids[0].num_elements
        u = rng.standard_normal((ne, block)) * rng.uniform(0, 2.0 / np.sqrt(block), (ne, 1))
        for g in grids:
            g.set_coefficients(u)
        same(f"refine {rnd}")
        if dim in (2, 3) and k == 2 and rnd < 2:
            outs = []
            for g in grids:
                op = amdg.BurgersOperator(g, 0.825)
                du = torch.from_numpy(u.reshape(-1).copy()).cuda()
                out = torch.zeros_like(du)
                torch.cuda.synchronize()
                op.rhs_device(du.data_ptr(), out.data_ptr())
                g.ctx.synchronize()
                outs.append(out.cpu().numpy())
                op.close()
            assert np.array_equal(outs[0], outs[1]), rnd
        removed = [g.coarsen(eta) for g in grids]
        assert removed[0] == removed[1]
        same(f"coarsen {rnd}")
    for g in grids:
        g.close()
