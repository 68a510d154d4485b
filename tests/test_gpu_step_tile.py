"""The whole-step passes (7- and 13-point) at the edges of its tiles and chunks: bit-identical to the
paired-stage passes, which form every value from another layout."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402
from cfb200 import fields  # noqa: E402

pytestmark = pytest.mark.gpu

FRW = dict(a1=1.0, H1=0.5, t1=1.0)


def run(N, eq, prec, flags, nsteps, stencil):
    L = float(N)
    c = cfb200.Context(N, L, m=1.0, equation=eq, precision=prec, flags=flags, stencil=stencil, lam=0.8, f_a=0.7, M=8, **FRW)
    x = fields.initial_state(N, L, 0.5, seed=5)
    x[N ** 3:] = 0.1 * x[: N ** 3][::-1]
    if eq in (cfb200.EQ_COMOVING_FRW, cfb200.EQ_APPROX_COMOVING_FRW):
        c.set_R_fft(fields.curvature_R_fft(N, L, 2.0, 1e-2, 0.5, seed=6), on_device=False)
    if eq == cfb200.EQ_FIXED_CURVATURE_FRW:
        c.set_psi(np.ascontiguousarray(1e-2 * x[: N ** 3]), on_device=False)
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.upload(st, x)
    c.rk4_steps(st, 1.0, 0.05, nsteps)
    torch.cuda.synchronize()
    out = st.view(torch.int64).clone()
    c.close()
    return out


# one tile smaller than the CTA's, partial tiles along b and c, a last chunk shorter than the
# others, whole tiles; every equation that has a form of its own for what a thread keeps
@pytest.mark.parametrize("stencil", [7, 13])
@pytest.mark.parametrize("N", [8, 40, 72, 104, 128, 136])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
@pytest.mark.parametrize("eq", [cfb200.EQ_KG_FRW, cfb200.EQ_SQRT_FRW, cfb200.EQ_COMOVING_FRW,
                                cfb200.EQ_FIXED_CURVATURE_FRW, cfb200.EQ_APPROX_COMOVING_FRW])
def test_step_pass_equals_paired_passes(N, prec, eq, stencil):
    a = run(N, eq, prec, 0, 3, stencil)
    b = run(N, eq, prec, cfb200.FLAG_PAIR_KERNELS, 3, stencil)
    assert torch.equal(a, b)
