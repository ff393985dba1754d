"""Direct launches chain through programmatic dependent launch: calls between a
caller's own kernels, on a stream of the caller's, and inside a caller's capture.
Small problems, where every launch is chained.  The same calls with a wait
between them are the reference: the kernels and their sums are the same, so the
results are equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(8, (6, 5, 4), False), (7, (5, 4, 3), True), (11, (3, 3, 2), True)]


@pytest.fixture(scope="module")
def nb():
    import neko_b200
    neko_b200.load()
    return neko_b200


def _problem(nb, lx, nel, h2):
    P = nb.Problem(nel, lx, deform=0.05)
    one = torch.ones_like(P.field("x"))
    P.set_coefficients(one, 3.0 * one if h2 else None)
    return P


def _rand(P, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(P.n, generator=g, dtype=torch.float64, device="cuda")


def _run(nb, P, M, u, wait):
    """Twenty rounds in which torch kernels write what the next call reads and
    overwrite what the last one has read."""
    A, w, z = nb.AxHelm(), P.zeros(), P.zeros()
    x = u.clone()
    for _ in range(20):
        for call in (lambda: A.compute(w, x, P), lambda: P.gs.op(w), lambda: P.bclst.apply(w),
                     lambda: x.mul_(0.5), lambda: M.solve(z, w, P), lambda: x.add_(z),
                     lambda: w.fill_(float("nan")), lambda: z.div_(z.abs().max() + 1.0),
                     lambda: x.div_(x.abs().max())):
            call()
            if wait:
                torch.cuda.synchronize()
    torch.cuda.synchronize()
    return x, z


@pytest.mark.parametrize("lx,nel,h2", CASES)
@pytest.mark.parametrize("own_stream", [False, True])
def test_between_a_callers_kernels(nb, lx, nel, h2, own_stream):
    P = _problem(nb, lx, nel, h2)
    M = nb.Hsmg()
    M.init(P)
    u = _rand(P, lx)
    ref = _run(nb, P, M, u, wait=True)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.current_stream()):
        out = _run(nb, P, M, u, wait=False)
    for a, b in zip(out, ref):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lx,nel,h2", CASES)
def test_inside_a_callers_capture(nb, lx, nel, h2):
    P = _problem(nb, lx, nel, h2)
    A, F = nb.AxHelm(), nb.AxHelmFull()
    u = _rand(P, 1)
    w, vs = P.zeros(), [P.zeros() for _ in range(3)]

    def calls():
        u.mul_(2.0)
        A.compute(w, u, P)
        P.gs.op(w)
        P.bclst.apply(w)
        F.compute_vector(*vs, w, u, w, P)
        vs[0].add_(w)

    calls()  # first uses, outside the capture
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        calls()
    for seed in (2, 3):
        u.copy_(_rand(P, seed))
        g.replay()
        torch.cuda.synchronize()
        out = [w.clone()] + [v.clone() for v in vs]
        u.copy_(_rand(P, seed))
        calls()
        torch.cuda.synchronize()
        for a, b in zip(out, [w] + vs):
            assert torch.equal(a, b)
