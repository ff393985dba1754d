"""The fused direction/operator/curvature step where its ring wraps at every
streamed order: more pairs of elements than the grid has blocks at odd orders,
with a lone last element, and the h2 forms, whose work planes at lx 9 lie over the
stage that is refilled.  The separate steps are the reference: 1e-12 of the
largest value for the operator, 1e-12 of the sum of magnitudes for the
curvature."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(4, (21, 21, 21)), (5, (17, 19, 19)), (5, (3, 1, 1)), (6, (17, 17, 17)),
         (7, (13, 13, 15)), (7, (1, 1, 1)), (8, (13, 13, 13)), (9, (11, 11, 13)), (9, (3, 3, 1)),
         (10, (11, 11, 11))]


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


@pytest.mark.parametrize("lx,nel", SIZES)
@pytest.mark.parametrize("h2", [False, True])
def test_step(nb, lx, nel, h2):
    P = nb.Problem(nel, lx, deform=0.05)
    h1 = 1.0 + 0.5 * torch.sin(3 * P.field("x")) * torch.cos(P.field("y"))
    P.set_coefficients(h1.contiguous(), 20.0 + P.field("z") if h2 else None)
    g = torch.Generator(device="cuda").manual_seed(lx)
    p, z = (torch.randn(P.n, generator=g, dtype=torch.float64, device="cuda") for _ in range(2))
    w, ref, pap = P.zeros(), P.zeros(), torch.zeros(1, dtype=torch.float64, device="cuda")
    want = z - 0.5 * p
    nb.AxHelm().compute(ref, want, P)
    nb.AxHelm().update_p_compute(w, p, z, -0.5, P, pap=pap)
    P.sync()
    assert torch.allclose(p, want, rtol=1e-15, atol=1e-15)
    assert float((w - ref).abs().max() / ref.abs().max()) < 1e-12
    t = want * ref
    assert abs(float(pap) - float(t.sum())) < 1e-12 * float(t.abs().sum())
