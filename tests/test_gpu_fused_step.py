"""The fused direction/operator/curvature step (nb_ax_update_p, the step of
every CG iteration) against the separate steps, over what selects its
kernels: streaming (lx 4, 6, 8, 10, aligned) and general (the other orders,
operands 8 bytes off a 16-byte boundary), with and without the h2 term, on
masked problems, and on more elements than the streaming grid has blocks, so
that each block's ring wraps.

The step does the operator's own sums, so w agrees to the operator's 1e-12;
the curvature is a sum of n products, whose rounding is far below 1e-12 of the
sum of their magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


def _vec(n, seed, offset):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.empty(n + offset, dtype=torch.float64, device="cuda")
    v[offset:] = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    return v[offset:]


SIZES = [(lx, (2, 3, 1)) for lx in range(2, 17)] + \
    [(4, (16, 15, 17)), (6, (12, 11, 13)), (8, (10, 11, 9)), (10, (8, 9, 8)), (7, (13, 17, 19)),
     (3, (33, 32, 33))]


@pytest.mark.parametrize("lx,nel", SIZES)
@pytest.mark.parametrize("h2", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_fused_step(nb, lx, nel, h2, offset):
    P = nb.Problem(nel, lx, deform=0.05)
    h1 = 1.0 + 0.5 * torch.sin(P.field("x"))
    P.set_coefficients(h1.contiguous(), torch.full_like(h1, 7.0) if h2 else None)
    p, z = _vec(P.n, 1, offset), _vec(P.n, 2, offset)
    w = torch.empty(P.n + offset, dtype=torch.float64, device="cuda")[offset:]
    pap = torch.zeros(1, dtype=torch.float64, device="cuda")
    want = z + 0.75 * p
    ref = P.zeros()
    nb.AxHelm().compute(ref, want, P)
    nb.AxHelm().update_p_compute(w, p, z, 0.75, P, pap=pap)
    P.sync()
    assert torch.allclose(p, want, rtol=1e-15, atol=1e-15)
    assert float((w - ref).abs().max() / ref.abs().max()) < 1e-12
    t = want * ref
    assert abs(float(pap) - float(t.sum())) < 1e-12 * float(t.abs().sum())
