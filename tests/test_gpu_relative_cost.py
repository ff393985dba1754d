"""Calls whose cost is bounded by that of a related one: a form of an operator
with more operands, or an operand off a 16-byte boundary, takes little longer
than the plain one.  Both times are taken in one process, best of several
groups of launches on the same problem, with data larger than the L2 cache.

A bound is the ratio of the bytes the two calls move, and a quarter more for a
form whose registers or order of loads are less favourable."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


def _best(*calls):
    """Best time of each call, in groups of 20 launches taken in turn."""
    out = [float("inf")] * len(calls)
    for c in calls:
        c()
    for _ in range(5):
        for k, c in enumerate(calls):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                c()
            b.record()
            torch.cuda.synchronize()
            out[k] = min(out[k], a.elapsed_time(b))
    return out


def _problem(nb, nel, lx, h2):
    P = nb.Problem(nel, lx, deform=0.05)
    one = torch.ones_like(P.field("x"))
    P.set_coefficients(one, 20.0 * one if h2 else None)
    return P


def _rand(n, offset=0):
    return torch.randn(n + offset, dtype=torch.float64, device="cuda")[offset:]


@pytest.mark.parametrize("lx,nel", [(11, (13, 12, 11)), (12, (13, 12, 11)), (13, (12, 11, 10)),
                                    (16, (10, 9, 8))])
def test_mass_term_scalar(nb, lx, nel):
    """w = A u with and without h2 B u: 11 arrays against 9."""
    A, P, Q = nb.AxHelm(), _problem(nb, nel, lx, False), _problem(nb, nel, lx, True)
    u, w = _rand(P.n), P.zeros()
    plain, mass = _best(lambda: A.compute(w, u, P), lambda: A.compute(w, u, Q))
    assert mass < 1.25 * 11 / 9 * plain


@pytest.mark.parametrize("lx,nel", [(12, (13, 12, 11)), (13, (12, 11, 10))])
@pytest.mark.parametrize("h2", [False, True])
def test_fused_step(nb, lx, nel, h2):
    """The fused step moves 11 arrays where the operator alone moves 9 (13 and
    11 with h2)."""
    A, P = nb.AxHelm(), _problem(nb, nel, lx, h2)
    p, z, w = P.zeros(), _rand(P.n), P.zeros()
    pap = torch.zeros(1, dtype=torch.float64, device="cuda")
    op, step = _best(lambda: A.compute(w, z, P),
                     lambda: A.update_p_compute(w, p, z, 0.5, P, pap=pap))
    assert step < 1.25 * (13 / 11 if h2 else 11 / 9) * op


@pytest.mark.parametrize("h2", [False, True])
def test_stress_outputs_off_a_boundary(nb, h2):
    """lx 8: results that start 8 bytes off a 16-byte boundary move the same
    bytes as others and take the same sums."""
    A, P = nb.AxHelmFull(), _problem(nb, (17, 16, 15), 8, h2)
    u = [_rand(P.n) for _ in range(3)]
    w = [[_rand(P.n, k) for _ in range(3)] for k in (0, 1)]
    on, off = _best(lambda: A.compute_vector(*w[0], *u, P), lambda: A.compute_vector(*w[1], *u, P))
    assert off < 1.25 * on
    for a, b in zip(*w):
        assert float((a - b).abs().max() / a.abs().max()) < 1e-14
