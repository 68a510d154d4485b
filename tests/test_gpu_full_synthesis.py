"""The FP64 full Psi synthesis by three passes of its own, at every lattice it is built for (and
one beside, which takes the library transforms), against torch FP64: every mode of R_fft non-zero,
the real-valued modes with an imaginary part that a C2R ignores.

The sums run over N^3 modes in three passes of at most three radix passes each, every value
rounded about 30 times with random signs: 1e-14 of the field's norm."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu

FRW = dict(a1=1.0, H1=0.5, t1=1.0)


@pytest.mark.parametrize("N", [56, 64, 96, 128, 192, 256, 384, 512])
def test_full_synthesis(N):
    t, L = 1.7, float(N)
    c = cfb200.Context(N, L, equation=cfb200.EQ_COMOVING_FRW, **FRW)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    w = torch.randn((N, N, N), generator=g, device="cuda", dtype=torch.float64)
    i = torch.arange(N, device="cuda")
    i = torch.minimum(i, N - i).double()
    s2 = i[:, None, None] ** 2 + i[None, :, None] ** 2 + torch.arange(N // 2 + 1, device="cuda").double()[None, None, :] ** 2
    R = torch.fft.rfftn(w) * 1e-3
    junk = R.clone()
    for a in (0, N // 2):  # the modes that stand for themselves: real in the transform of a real field
        for b in (0, N // 2):
            for k in (0, N // 2):
                junk[a, b, k] += 0.1j
    c.set_R_fft(torch.view_as_real(junk).reshape(-1).contiguous(), on_device=True)
    assert c.info.psi_route == cfb200.PSI_FULL
    out = torch.empty(2 * N ** 3, dtype=torch.float64, device="cuda")
    c.psi_fields(t, out)
    x = torch.sqrt(s2) * (2 * math.pi / L * 2 * math.sqrt(t) / math.sqrt(3))
    x[0, 0, 0] = 1.0
    common = 2 / x ** 3
    common[0, 0, 0] = 0.0
    sn, cs = torch.sin(x), torch.cos(x)
    want = [torch.fft.irfftn(R * f, s=(N, N, N)) for f in
            ((sn - x * cs) * common, (0.5 / t) * (3 * x * cs + (x * x - 3) * sn) * common)]
    for k in range(2):
        got = out[k * N ** 3:(k + 1) * N ** 3].reshape(N, N, N)
        assert float((got - want[k]).norm()) <= 1e-14 * float(want[k].norm())
    c.close()
