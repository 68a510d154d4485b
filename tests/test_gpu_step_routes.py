"""Which passes cf_rk4_steps takes where the choice depends on the lattice and the call (a curvature
input), and that each route gives the bits of the four single-stage passes, which
share neither tiles nor chunks with them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402
from cfb200 import fields  # noqa: E402

pytestmark = pytest.mark.gpu

COMOVING, FIXED, APPROX = cfb200.EQ_COMOVING_FRW, cfb200.EQ_FIXED_CURVATURE_FRW, cfb200.EQ_APPROX_COMOVING_FRW


def run(N, eq, prec, flags, nsteps, stencil):
    """The state after nsteps, and how many whole-step and first paired passes ran."""
    L = float(N)
    c = cfb200.Context(N, L, m=1.0, equation=eq, precision=prec, flags=flags, stencil=stencil, lam=0.8, f_a=0.7, M=8,
                       a1=1.0, H1=0.5, t1=1.0)
    x = fields.initial_state(N, L, 0.5, seed=5)
    x[N ** 3:] = 0.1 * x[: N ** 3][::-1]
    if eq in (COMOVING, APPROX):
        c.set_R_fft(fields.curvature_R_fft(N, L, 2.0, 1e-2, 0.5, seed=6), on_device=False)
    if eq == FIXED:
        c.set_psi(np.ascontiguousarray(1e-2 * x[: N ** 3]), on_device=False)
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.upload(st, x)
    c.profile()
    c.rk4_steps(st, 1.0, 0.05, nsteps)
    torch.cuda.synchronize()
    prof = c.profile_read()
    out = st.view(torch.int64).clone()
    c.close()
    return out, prof["step"][0], prof["pair_a"][0]


FP64, COMP = cfb200.FP64, cfb200.FP32_COMP

# (precision, stencil, equation, N, steps, whole-step passes)
ROUTES = [(COMP, 13, FIXED, 72, 2, True), (COMP, 13, FIXED, 80, 1, True), (COMP, 13, FIXED, 88, 2, False),
          (COMP, 13, FIXED, 96, 1, False), (COMP, 13, FIXED, 104, 2, True), (COMP, 13, APPROX, 72, 2, True),
          (COMP, 13, APPROX, 96, 2, False), (COMP, 13, APPROX, 104, 1, True), (COMP, 13, COMOVING, 72, 1, True),
          (COMP, 13, COMOVING, 72, 3, False), (COMP, 13, COMOVING, 88, 1, False), (COMP, 13, COMOVING, 104, 1, True),
          (COMP, 13, COMOVING, 120, 3, False), (COMP, 13, COMOVING, 128, 2, True), (COMP, 13, COMOVING, 136, 1, True),
          (COMP, 13, COMOVING, 200, 3, True)]
ROUTES += [(p, s, COMOVING, N, n, whole) for p in (FP64, COMP) for s in (7, 13)
           for N, n, whole in ((32, 2, True), (40, 1, True), (40, 2, False), (64, 3, False))]
ROUTES += [(FP64, 13, FIXED, 88, 2, True), (FP64, 7, COMOVING, 72, 2, True), (FP64, 13, COMOVING, 72, 2, True),
           (COMP, 7, COMOVING, 72, 2, True)]


@pytest.mark.parametrize("prec,stencil,eq,N,nsteps,whole", ROUTES)
def test_route_and_bits(prec, stencil, eq, N, nsteps, whole):
    out, step, pair = run(N, eq, prec, 0, nsteps, stencil)
    assert (step, pair) == ((nsteps, 0) if whole else (0, nsteps))
    want, step, pair = run(N, eq, prec, cfb200.FLAG_STAGE_KERNELS, nsteps, stencil)
    assert (step, pair) == (0, 0)
    assert torch.equal(out, want)


# the serial Psi refreshes leave the step alone: the route of a one-step call
def test_serial_refreshes():
    out, step, pair = run(72, COMOVING, cfb200.FP32_COMP, cfb200.FLAG_PSI_SERIAL, 2, 13)
    assert (step, pair) == (2, 0)
    assert torch.equal(out, run(72, COMOVING, cfb200.FP32_COMP, cfb200.FLAG_STAGE_KERNELS, 2, 13)[0])


# the self-interacting field has forms of its own
@pytest.mark.parametrize("stencil", [7, 13])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
@pytest.mark.parametrize("N", [8, 72, 128])
def test_lambda(N, prec, stencil):
    out, step, _ = run(N, cfb200.EQ_LAMBDA_FRW, prec, 0, 3, stencil)
    assert step == 3
    assert torch.equal(out, run(N, cfb200.EQ_LAMBDA_FRW, prec, cfb200.FLAG_STAGE_KERNELS, 3, stencil)[0])
