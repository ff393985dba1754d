"""The hsmg coarse solve at the sizes where its launch changes form: no
unmasked vertex at all, one block, clusters with the vectors and the matrix
resident in every block, the matrix in global memory, and the element-local
grid of larger meshes, with its vectors in registers and in memory.  One
application against the CPU oracle with the bounds of test_gpu_hsmg.py (lx 4
keeps the other levels small)."""
import numpy as np
import pytest
import torch

from test_gpu_hsmg import _cuda, _np, _pair, _residual, nb  # noqa: F401

pytestmark = pytest.mark.gpu

#        elements       periodic              vertices
NODES = [((1, 1, 1), (False,) * 3),         # 0
         ((2, 2, 2), (False,) * 3),         # 1
         ((9, 7, 8), (False,) * 3),         # 336: four blocks
         ((17, 16, 18), (False,) * 3),      # 4080: sixteen blocks
         ((21, 20, 21), (False,) * 3),      # 7600: matrix in global memory
         ((21, 20, 22), (True, False, True)),   # 8400: element-local
         ((26, 25, 27), (False,) * 3),      # 15600
         ((28, 28, 27), (True, False, False)),  # 19656
         ((33, 33, 34), (True, False, False)),  # 34848
         ((34, 34, 33), (True, False, False))]  # vectors in memory


@pytest.mark.parametrize("nel,per", NODES)
def test_coarse_sizes_match_oracle(nb, oracle, nel, per):  # noqa: F811
    P, O = _pair(nb, oracle, nel, 4, per, 0.05, 2 * np.pi)
    H = oracle.OracleHsmg(O)
    r = _residual(O, np.random.default_rng(nel[0]), False)
    ref = H.apply(r)
    z = P.zeros()
    nb.Hsmg().solve(z, _cuda(r), P)
    torch.cuda.synchronize()
    err = np.abs(_np(z) - ref).max() / np.abs(ref).max()
    assert err < 1e-10, err


@pytest.mark.parametrize("nel,per", NODES[1:4])
def test_coarse_follows_coefficients(nb, oracle, nel, per):  # noqa: F811
    """After set_coefficients the coarse matrix is rebuilt: a problem whose
    coefficients change equals one that had them before its set-up."""
    P, O = _pair(nb, oracle, nel, 6, per, 0.05, 2 * np.pi)
    r = _cuda(_residual(O, np.random.default_rng(3), False))
    h1 = (1.5 + torch.sin(P.field("x")) * torch.cos(P.field("y"))).contiguous()
    z0, z1 = P.zeros(), P.zeros()
    nb.Hsmg().solve(z0, r, P)
    P.set_coefficients(h1)
    nb.Hsmg().solve(z0, r, P)
    Q, _ = _pair(nb, oracle, nel, 6, per, 0.05, 2 * np.pi)
    Q.set_coefficients(h1)
    nb.Hsmg().solve(z1, r, Q)
    torch.cuda.synchronize()
    assert torch.equal(z0, z1)
