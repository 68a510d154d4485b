"""Observers at the edges of the energy pass's tiles (64 sites of a row, chunks along a, one
chunk of all planes for the slices of larger lattices) and of the scale bounds, against torch FP64.

Energy density: about 20 FP64 roundings per site, relative to its own terms: 1e-13 of its norm.
Spectra: 1e-12 norm-wise (the transform's rounding); FP32_COMP states are widened exactly."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu

FRW = dict(a1=1.0, H1=0.5, t1=1.0)


def setup(N, prec, m=1.1, eq=cfb200.EQ_KG_FRW):
    c = cfb200.Context(N, float(N), m=m, equation=eq, precision=prec, lam=0.8, f_a=0.7, **FRW)
    x = np.random.default_rng(N).standard_normal(2 * N ** 3)
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.upload(st, x)
    c.download(x, st)  # what the state holds (FP32_COMP: 48 bits)
    return c, st, torch.from_numpy(x).cuda().reshape(2, N, N, N)


def density(x, t, m, eq):
    f, p = x[0], x[1]
    grad = sum((f.roll(-1, k) - f.roll(1, k)).square() for k in range(3)) / (4 * t)
    rho = 0.5 * (p * p + grad)
    if eq == cfb200.EQ_SQRT_FRW:
        return rho + m * m * f * f / (torch.sqrt(1 + f * f / 0.49) + 1)
    rho = rho + 0.5 * m * m * f * f
    return rho + 0.2 * f ** 4 if eq == cfb200.EQ_LAMBDA_FRW else rho


def bins(N, v):
    i = torch.arange(N, device="cuda")
    i = torch.minimum(i, N - i)
    k = torch.arange(N // 2 + 1, device="cuda")
    s2 = (i * i)[:, None, None] + (i * i)[None, :, None] + (k * k)[None, None, :]
    w = torch.full((N // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    w[0] = w[-1] = 1.0
    out = torch.zeros(3 * (N // 2) ** 2 + 1, device="cuda", dtype=torch.float64)
    return out.index_add(0, s2.reshape(-1), (v * w).reshape(-1)), s2


def close(a, b, tol):
    return float((a - b).norm()) <= tol * float(b.norm())


@pytest.mark.parametrize("N", [8, 56, 64, 72, 136, 328])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
@pytest.mark.parametrize("eq", [cfb200.EQ_KG_FRW, cfb200.EQ_LAMBDA_FRW, cfb200.EQ_SQRT_FRW])
def test_density_outputs(N, prec, eq):
    t, m = 1.7, 1.1
    c, st, x = setup(N, prec, m, eq)
    want = density(x, t, m, eq)
    for offset in (0, 1):  # 16- and 8-byte aligned output
        buf = torch.empty(N ** 3 + 1, dtype=torch.float64, device="cuda")[offset:offset + N ** 3]
        c.energy_density(st, t, buf)
        assert close(buf.reshape(N, N, N), want, 1e-13)
        sl, av = (torch.empty(N * N + 1, dtype=torch.float64, device="cuda")[offset:offset + N * N] for _ in range(2))
        c.density_slices(st, t, sl, av)
        assert close(sl.reshape(N, N), want[0], 1e-13) and close(av.reshape(N, N), want.mean(0), 1e-13)
    rho = torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda")
    shells = torch.empty(c.info.shells, dtype=torch.float64, device="cuda")
    c.density_spectrum_s2(st, t, rho)
    c.s2_to_shells(shells)
    f = torch.fft.rfftn(want)
    b, _ = bins(N, f.real ** 2 + f.imag ** 2)
    assert close(rho, b, 1e-12)
    idx = torch.tensor([math.isqrt(s) for s in range(b.numel())], device="cuda")
    assert close(shells, torch.zeros_like(shells).index_add(0, idx, rho), 1e-14)
    c.close()


# a mass for which the state's sums bound the modes, one for which they do not (max pass)
@pytest.mark.parametrize("m", [1.1, 1e-4])
@pytest.mark.parametrize("N", [8, 40, 72])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
def test_mode_spectrum(N, prec, m):
    a = 1.3
    c, st, x = setup(N, prec, m)
    out = torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda")
    c.mode_power_spectrum_s2(st, a, out)
    f, p = torch.fft.rfftn(x[0]), torch.fft.rfftn(x[1])
    _, s2 = bins(N, f.real)
    w2 = m * m + (2 * math.pi / N) ** 2 * s2.double() / a ** 2
    want, _ = bins(N, f.real ** 2 + f.imag ** 2 + (p.real ** 2 + p.imag ** 2) / w2)
    assert close(out, want, 1e-12)
    big = want >= 1e-9 * want.max()
    assert float(((out - want).abs() / want)[big].max()) <= 1e-11
    c.close()
