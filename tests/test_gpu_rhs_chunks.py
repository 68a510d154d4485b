"""cf_rhs on both sides of its planes-per-CTA limits (N = 128 for the 13-point stencil, 144 for the
7-point one) and with a shorter last chunk, against the stencil written with rolls."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


def laplacian(f, stencil):
    """(sum of the terms, sum of their absolute values) of the FD Laplacian, h = 1."""
    def near(d):
        return [torch.roll(f, s * d, a) for a in range(3) for s in (1, -1)]
    if stencil == 7:
        return sum(near(1)) - 6 * f, sum(x.abs() for x in near(1)) + 6 * f.abs()
    a, b = near(1), near(2)
    return ((16 * sum(a) - sum(b) - 90 * f) / 12,
            (16 * sum(x.abs() for x in a) + sum(x.abs() for x in b) + 90 * f.abs()) / 12)


@pytest.mark.parametrize("stencil,N", [(7, 8), (7, 72), (7, 136), (7, 144), (7, 200), (13, 8), (13, 72), (13, 120),
                                       (13, 128), (13, 136)])
def test_rhs(stencil, N):
    m, a1, H1, t1, t = 1.3, 1.1, 0.5, 1.0, 1.5
    c = cfb200.Context(N, float(N), m=m, equation=cfb200.EQ_KG_FRW, stencil=stencil, a1=a1, H1=H1, t1=t1)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    x = torch.randn((2, N, N, N), generator=g, device="cuda", dtype=torch.float64)
    out = torch.empty_like(x)
    c.rhs(x, out, t)
    a2, hubble = a1 ** 2 * (1 + 2 * H1 * (t - t1)), H1 / (1 + 2 * H1 * (t - t1))
    lap, size = laplacian(x[0], stencil)
    want = lap / a2 - 3 * hubble * x[1] - m * m * x[0]
    # under 24 roundings of terms no larger than their absolute sum, on either side
    bound = 48 * 2.0 ** -53 * (size / a2 + 3 * hubble * x[1].abs() + m * m * x[0].abs())
    assert torch.equal(out[0], x[1])
    assert bool(((out[1] - want).abs() <= bound).all())
    c.close()
