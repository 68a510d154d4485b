"""The resolution of the spectra's fixed point: its scale follows the sum over the lattice
(Parseval), so a mode far below the total keeps its digits also where the field is a few sites.

Two sites, 0 and (N/2, N/2, N/2), hold values r and r - d with d ~ 2^-40 r: the modes of odd s^2
are d, those of even s^2 2 r - d, and the transform forms both without rounding (every line
holds values at 0 and N/2 only).  The bound B = N^3 (r^2 + (r - d)^2) gives a step of at most
2 B 2^-126 per mode, so a bin of odd s^2 is off by at most 4 N^3 r^2 2^-126 / d^2 of itself, less than
2^-21 at N = 128."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu

N = 128
FRW = dict(a1=1.0, H1=0.5, t1=1.0)


def check(c, out, r, d):
    counts = torch.empty(c.info.s2_bins, dtype=torch.int64, device="cuda")
    c.s2_counts(counts)
    s2 = torch.arange(counts.numel(), device="cuda")
    want = torch.where(s2 % 2 == 1, d * d, (2 * r - d) ** 2) * counts
    some = counts > 0
    assert 4 * N ** 3 * r * r * 2.0 ** -126 <= 2.0 ** -21 * d * d
    assert float(((out - want).abs() / want)[some].max()) <= 2.0 ** -21


def sites(c, component, first, second):
    x = torch.zeros((2, N, N, N), dtype=torch.float64, device="cuda")
    x[component, 0, 0, 0] = first
    x[component, N // 2, N // 2, N // 2] = second
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.import_f64(st, x)
    return st


@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
def test_density_spectrum(prec):
    c = cfb200.Context(N, float(N), m=1.1, equation=cfb200.EQ_KG_FRW, precision=prec, **FRW)
    st = sites(c, 1, 1.5, 1.5 - 1.2345678 * 2.0 ** -40)
    rho = torch.empty(N ** 3, dtype=torch.float64, device="cuda")
    c.energy_density(st, 1.0, rho)
    r, far = float(rho[0]), float(rho.reshape(N, N, N)[N // 2, N // 2, N // 2])
    out = torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda")
    c.density_spectrum_s2(st, 1.0, out)
    check(c, out, r, r - far)
    c.close()


@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
def test_mode_spectrum(prec):
    c = cfb200.Context(N, float(N), m=1.1, equation=cfb200.EQ_KG_FRW, precision=prec, **FRW)
    st = sites(c, 0, 1.5, 1.5 - 1.2345678 * 2.0 ** -40)
    x = torch.empty((2, N, N, N), dtype=torch.float64, device="cuda")
    c.export_f64(x, st)
    r, far = float(x[0, 0, 0, 0]), float(x[0, N // 2, N // 2, N // 2])
    out = torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda")
    c.mode_power_spectrum_s2(st, 1.0, out)
    check(c, out, r, r - far)
    c.close()
