"""cf_density_slices on both sides of its route limits (one march over all planes, with 3 or 4 CTAs per
SM, or the density and a pass over it): every route sums a column in increasing a and divides by N,
so the mean equals, bit for bit, the same sum over cf_energy_density's output."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 200, 224, 312, 320, 328, 336, 448, 464, 512])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
@pytest.mark.parametrize("eq", [cfb200.EQ_KG_FRW, cfb200.EQ_FIXED_CURVATURE_FRW])
def test_slices(N, prec, eq):
    c = cfb200.Context(N, float(N), m=1.1, equation=eq, precision=prec, a1=1.0, H1=0.5, t1=1.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    x = torch.randn(2 * N ** 3, generator=g, device="cuda", dtype=torch.float64)
    if eq == cfb200.EQ_FIXED_CURVATURE_FRW:
        c.set_psi((1e-2 * x[: N ** 3]).contiguous(), on_device=True)
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.import_f64(st, x)
    rho = torch.empty((N, N * N), dtype=torch.float64, device="cuda")
    c.energy_density(st, 1.7, rho)
    want = torch.zeros(N * N, dtype=torch.float64, device="cuda")
    for a in range(N):
        want += rho[a]
    want = want / torch.full_like(want, N)  # by a tensor: torch takes a scalar divisor's reciprocal
    sl, av, sl1, av1 = (torch.full((N * N,), -1.0, dtype=torch.float64, device="cuda") for _ in range(4))
    c.density_slices(st, 1.7, sl, av)
    c.density_slices(st, 1.7, sl1, None)
    c.density_slices(st, 1.7, None, av1)
    c.density_slices(st, 1.7)
    assert torch.equal(sl, rho[0]) and torch.equal(av, want)
    assert torch.equal(sl1, sl) and torch.equal(av1, av)
    c.close()
