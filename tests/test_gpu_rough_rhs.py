"""CG on right-hand sides that are not assembled and masked: the inner products
that the fused kernels form before the gather-scatter are then not the
reference's, and the solve takes the reference's own.  A few steps of CG,
flexible CG and coupled CG against the same steps in plain torch around the
operator, gather-scatter and mask (cg_device.f90:162-238 and
cg_cpld_device.f90:292-417), over the orders and problems whose kernels differ;
an assembled f beside them as the control, and f within rounding of one.

Operators and sums differ in order only; a few steps keep the iterates to the
operators' 1e-12 times the digits the inner products lose: 1e-10."""
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = 4


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


def _problem(nb, lx, h2, masked):
    hi = 1.0 if masked else 6.283185307179586
    P = nb.Problem((4, 3, 5), lx, hi=(hi,) * 3, periodic=(not masked,) * 3, deform=0.05,
                   dirichlet=masked)
    one = torch.ones_like(P.field("x"))
    P.set_coefficients(one, 7.0 * one if h2 else None)
    return P


def _rhs(P, kind, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = (P.field("B") * torch.randn(P.n, generator=g, dtype=torch.float64, device="cuda"))
    f = f.contiguous()
    if kind != "local":
        P.gs.op(f)
    if kind in ("assembled", "rounded"):
        P.bclst.apply(f)
    if kind == "rounded":
        f *= 1.0 + 1e-15 * torch.randn(P.n, generator=g, dtype=torch.float64, device="cuda")
    return f


def _apply(P, A, us):
    ws = [P.zeros() for _ in us]
    if len(us) == 1:
        A.compute(ws[0], us[0], P)
    else:
        A.compute_vector(*ws, *us, P)
    for w in ws:
        P.gs.op(w)
        P.bclst.apply(w)
    return ws


def _steps(P, A, fs, precond, flexible=False):
    mult = P.field("mult")
    dot = lambda a, b: sum((u * mult * v).sum() for u, v in zip(a, b))  # noqa: E731
    x, r = [torch.zeros_like(f) for f in fs], [f.clone() for f in fs]
    p, w, alpha, rz = None, None, None, None
    for _ in range(STEPS):
        z = precond(r)
        old, rz = rz, dot(r, z)
        if p is None:
            p = z
        else:
            beta = -alpha * dot(w, z) / old if flexible else rz / old
            p = [u + beta * v for u, v in zip(z, p)]
        w = _apply(P, A, p)
        alpha = rz / dot(p, w)
        x = [u + alpha * v for u, v in zip(x, p)]
        r = [u - alpha * v for u, v in zip(r, w)]
    return x


def _close(xs, ys):
    torch.cuda.synchronize()
    for a, b in zip(xs, ys):
        assert float((a - b).abs().max() / b.abs().max()) < 1e-10


@pytest.mark.parametrize("lx", [3, 4, 5, 7, 8, 10, 11])
@pytest.mark.parametrize("h2,masked", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("kind", ["assembled", "rounded", "unmasked", "local"])
def test_cg(nb, lx, h2, masked, kind):
    P = _problem(nb, lx, h2, masked)
    f, x, d = _rhs(P, kind, lx), P.zeros(), P.field("jacobi")
    S = nb.CG(abs_tol=0.0, M=nb.Jacobi())
    for _ in range(2):  # the captured iterations are kept between solves
        S.solve(nb.AxHelm(), x, f, P.n, P, niter=STEPS)
        _close([x], _steps(P, nb.AxHelm(), [f], lambda r: [d * r[0]]))
        f = _rhs(P, "assembled", 9)


@pytest.mark.parametrize("lx", [5, 8])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind", ["assembled", "unmasked", "local"])
def test_flexible_hsmg(nb, lx, mixed, kind):
    """The preconditioner is the device's own, so FP32 smoothing differs by
    nothing but its input's rounding: 1e-6."""
    P = _problem(nb, lx, False, True)
    f, x = _rhs(P, kind, lx), P.zeros()
    M = nb.Hsmg(mixed=mixed)

    def precond(r):
        z = P.zeros()
        M.solve(z, r[0], P)
        torch.cuda.synchronize()
        return [z]

    nb.FCG(abs_tol=0.0, M=M).solve(nb.AxHelm(), x, f, P.n, P, niter=STEPS)
    y = _steps(P, nb.AxHelm(), [f], precond, flexible=True)
    torch.cuda.synchronize()
    bound = 1e-6 if mixed else 1e-9
    assert float((x - y[0]).abs().max() / y[0].abs().max()) < bound


@pytest.mark.parametrize("lx", [4, 7, 8, 10])
@pytest.mark.parametrize("kind", ["assembled", "unmasked", "local"])
def test_coupled_stress(nb, lx, kind):
    P = _problem(nb, lx, True, True)
    fs, d = [_rhs(P, kind, c) for c in range(3)], P.field("jacobi")
    xs = [P.zeros() for _ in fs]
    nb.CoupledCG(abs_tol=0.0, M=nb.Jacobi()).solve_coupled(nb.AxHelmFull(), *xs, *fs, P.n, P,
                                                           niter=STEPS)
    _close(xs, _steps(P, nb.AxHelmFull(), fs, lambda r: [d * v for v in r]))
