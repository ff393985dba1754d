"""The streaming operator at the orders it takes (4 to 10): fewer elements
than blocks, more than two a stage of every block (the ring wraps), and odd
counts, whose last element odd orders stream alone.  The general kernel
(taken for an operand 8 bytes off a 16-byte boundary) is the reference.

The two differ in the order of sums of at most 3 lx + 1 terms: 1e-12 of the
largest value."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(lx, nel) for lx in range(4, 11) for nel in ((1, 1, 1), (3, 1, 1), (2, 5, 2))] + \
    [(4, (21, 21, 21)), (5, (17, 19, 19)), (6, (17, 17, 17)), (7, (13, 13, 15)),
     (8, (13, 13, 13)), (9, (11, 11, 13)), (10, (11, 11, 11))]


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


@pytest.mark.parametrize("lx,nel", SIZES)
@pytest.mark.parametrize("h2", [False, True])
def test_matches_general(nb, lx, nel, h2):
    P = nb.Problem(nel, lx, deform=0.05)
    h1 = 1.0 + 0.5 * torch.sin(3 * P.field("x")) * torch.cos(P.field("y"))
    P.set_coefficients(h1.contiguous(), 20.0 + P.field("z") if h2 else None)
    g = torch.Generator(device="cuda").manual_seed(lx)
    b = torch.empty(P.n + 1, dtype=torch.float64, device="cuda")
    b[1:] = torch.randn(P.n, generator=g, dtype=torch.float64, device="cuda")
    out, ref = P.zeros(), P.zeros()
    nb.AxHelm().compute(out, b[1:].clone(), P)
    nb.AxHelm().compute(ref, b[1:], P)
    P.sync()
    assert float((out - ref).abs().max() / ref.abs().max()) < 1e-12
