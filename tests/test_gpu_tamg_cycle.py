"""phmg's tree-AMG cycle as one launch, at the sizes and settings where its
loops change: several vertices a thread, one Chebyshev step, two cycles, two
levels only, and a last level that is not the vertex level (separate
launches).  One application against the oracle with the bound of
test_gpu_phmg.py."""
import numpy as np
import pytest
import torch

from test_gpu_phmg import _cuda, _np, _pair, _rel, nb  # noqa: F401

pytestmark = pytest.mark.gpu

CASES = [((21, 20, 22), 4, dict(schedule=(1,))),
         ((6, 5, 4), 4, dict(schedule=(1,), cheby_degree=1, coarse_iterations=2)),
         ((7, 6, 5), 5, dict(schedule=(1,), coarse_levels=2)),
         ((2, 2, 2), 5, dict()),
         ((4, 3, 5), 5, dict(schedule=(2,)))]


@pytest.mark.parametrize("nel,lx,kw", CASES)
def test_cycle_matches_oracle(nb, oracle, nel, lx, kw):  # noqa: F811
    P, O = _pair(nb, oracle, nel, lx, amp=0.05)
    H = oracle.OraclePhmg(O, **kw)
    M = nb.Phmg(**kw)
    r = O.bc_apply(O.gs_add(O.f64("B") * np.random.default_rng(5).standard_normal(O.n)))
    z = P.zeros()
    M.solve(z, _cuda(r), P)
    torch.cuda.synchronize()
    assert _rel(_np(z), H.apply(r)) < 1e-9
    H.close()
