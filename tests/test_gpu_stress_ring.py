"""The streaming full-stress operator where its ring wraps: more elements
than the grid has blocks, so every block refills each of its stages.  The
general kernel (taken for operands 8 bytes off a 16-byte boundary) is the
reference for the operator, plain CG steps around that operator for the
coupled solve, whose iterations take the fused form of the kernel and the
three-component gather-scatter.

The two operators differ in the order of a few sums of at most 3 lx terms:
1e-12 of the largest value.  Five CG steps keep their iterates to the same
order times the few digits the inner products lose: 1e-10."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        lx, elements: at least three a block
SIZES = [(4, (16, 15, 16)), (6, (12, 13, 12)), (8, (10, 9, 11)), (10, (8, 8, 9))]


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


def _problem(nb, lx, nel, h2):
    P = nb.Problem(nel, lx, deform=0.05)
    h1 = 1.0 + 0.5 * torch.sin(3 * P.field("x")) * torch.cos(P.field("y"))
    P.set_coefficients(h1.contiguous(), torch.full_like(h1, 20.0) if h2 else None)
    return P


def _rand(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("lx,nel", SIZES)
@pytest.mark.parametrize("h2", [False, True])
def test_ring_wraps(nb, lx, nel, h2):
    P = _problem(nb, lx, nel, h2)
    u = [_rand(P.n, c) for c in range(3)]
    off = []
    for v in u:
        b = torch.empty(P.n + 1, dtype=torch.float64, device="cuda")
        b[1:] = v
        off.append(b[1:])
    out, ref = [P.zeros() for _ in u], [P.zeros() for _ in u]
    nb.AxHelmFull().compute_vector(*out, *u, P)
    nb.AxHelmFull().compute_vector(*ref, *off, P)
    P.sync()
    for a, b in zip(out, ref):
        assert float((a - b).abs().max() / b.abs().max()) < 1e-12


@pytest.mark.parametrize("lx,nel", SIZES)
@pytest.mark.parametrize("h2", [False, True])
def test_coupled_steps(nb, lx, nel, h2):
    P = _problem(nb, lx, nel, h2)
    f = []
    for c in range(3):
        v = (P.field("B") * _rand(P.n, 10 + c)).contiguous()
        P.gs.op(v)
        P.bclst.apply(v)
        f.append(v)
    xs = [P.zeros() for _ in f]
    nb.CoupledCG(abs_tol=0.0, M=nb.Jacobi()).solve_coupled(nb.AxHelmFull(), *xs, *f, P.n, P,
                                                           niter=5)
    mult, d = P.field("mult"), P.field("jacobi")
    dot = lambda a, b: sum((u * mult * v).sum() for u, v in zip(a, b))  # noqa: E731
    x, r = [torch.zeros_like(v) for v in f], [v.clone() for v in f]
    z = [d * v for v in r]
    p, rz = [v.clone() for v in z], dot(r, z)
    w = [P.zeros() for _ in f]
    for _ in range(5):
        nb.AxHelmFull().compute_vector(*w, *p, P)
        for v in w:
            P.gs.op(v)
            P.bclst.apply(v)
        a = rz / dot(p, w)
        for k in range(3):
            x[k] += a * p[k]
            r[k] -= a * w[k]
        z = [d * v for v in r]
        rz, old = dot(r, z), rz
        p = [v + (rz / old) * q for v, q in zip(z, p)]
    torch.cuda.synchronize()
    for a, b in zip(xs, x):
        assert float((a - b).abs().max() / b.abs().max()) < 1e-10
