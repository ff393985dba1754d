"""phmg's tree-AMG cycle on both sides of the vertex count up to which it is
one launch (8192, one vertex a thread of a cluster of 16 blocks): a resident
cycle, a cycle whose elements are more than the cluster's threads, and the
separate launches beyond, with and without a mask and with two cycles.  One
application against the oracle with the bound of test_gpu_phmg.py, and the
form by the kernels an application launches: the separate cycle alone is more
than 60."""
import numpy as np
import pytest
import torch

from test_gpu_phmg import _cuda, _np, _pair, _rel, nb  # noqa: F401

pytestmark = pytest.mark.gpu

#        elements, periodic, one launch, settings
CASES = [((20, 19, 21), False, True, dict()),                       # 6840 vertices
         ((20, 20, 20), True, True, dict()),                        # 8000
         ((21, 20, 22), False, True, dict(coarse_iterations=2)),    # 7980, 9240 elements
         ((22, 21, 21), False, False, dict()),                      # 8400
         ((21, 20, 20), True, False, dict(coarse_iterations=2)),    # 8400
         ((27, 26, 28), False, False, dict(coarse_iterations=2))]   # 17550


@pytest.mark.parametrize("nel,per,one,kw", CASES)
def test_form_and_result(nb, oracle, nel, per, one, kw):  # noqa: F811
    P, O = _pair(nb, oracle, nel, 4, per=(per,) * 3, amp=0.05, hi=2 * np.pi if per else 1.0,
                 dirichlet=not per)
    H = oracle.OraclePhmg(O, schedule=(1,), **kw)
    M = nb.Phmg(schedule=(1,), **kw)
    r = O.gs_add(O.f64("B") * np.random.default_rng(5).standard_normal(O.n))
    if per:
        r = r - r.mean()
    else:
        r = O.bc_apply(r)
    z = P.zeros()
    M.solve(z, _cuda(r), P)
    torch.cuda.synchronize()
    assert (M.describe(P, 10) < 60) == one
    assert _rel(_np(z), H.apply(r)) < 1e-9
    H.close()
