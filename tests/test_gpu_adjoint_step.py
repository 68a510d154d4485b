"""The whole reverse step (7-point) at the edges of its tiles and chunks against the reverse
sweep in numpy FP64 (the transpose of each RK4 stage, stage by stage).

lambda_0 is FP64 in both precisions: a few hundred roundings per step, 1e-12 of its norm.
dL/dm sums products of lambda with the forward stage inputs, which are FP32 in FP32_COMP
(relative error 2^-24 each, unbiased): 1e-12 and 1e-5 of the sum of their magnitudes' norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu

FRW = dict(a1=1.0, H1=0.5, t1=1.0)


def lap(f):
    return sum(np.roll(f, s, ax) for ax in range(3) for s in (1, -1)) - 6 * f


def coefs(t):
    return 1.0 / (1 + (t - 1.0)), 3 * 0.5 / (1 + (t - 1.0))  # h^-2 a^-2, 3H (h = 1)


def forward_op(x, t, m):
    inv, rub = coefs(t)
    return np.stack([x[1], inv * lap(x[0]) - m * m * x[0] - rub * x[1]])


def adjoint_op(k, t, m):
    inv, rub = coefs(t)
    return np.stack([inv * lap(k[1]) - m * m * k[1], k[0] - rub * k[1]])


def reference(x0, lam, t0, dt, nsteps, m):
    states, x = [], x0
    for j in range(nsteps):
        t = t0 + j * dt
        y1 = x
        k1 = forward_op(y1, t, m)
        y2 = x + dt / 2 * k1
        k2 = forward_op(y2, t + dt / 2, m)
        y3 = x + dt / 2 * k2
        k3 = forward_op(y3, t + dt / 2, m)
        y4 = x + dt * k3
        k4 = forward_op(y4, t + dt, m)
        states.append((t, y1, y2, y3, y4))
        x = x + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    dm = 0.0
    for t, y1, y2, y3, y4 in reversed(states):
        k4 = dt / 6 * lam
        a4 = adjoint_op(k4, t + dt, m)
        k3 = dt / 3 * lam + dt * a4
        a3 = adjoint_op(k3, t + dt / 2, m)
        k2 = dt / 3 * lam + dt / 2 * a3
        a2 = adjoint_op(k2, t + dt / 2, m)
        k1 = dt / 6 * lam + dt / 2 * a2
        a1 = adjoint_op(k1, t, m)
        dm += sum(np.sum(k[1] * y[0]) for k, y in ((k4, y4), (k3, y3), (k2, y2), (k1, y1))) * (-2 * m)
        lam = lam + a4 + a3 + a2 + a1
    return lam, dm


@pytest.mark.parametrize("N", [8, 32, 40, 72, 104])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
def test_reverse_step(N, prec):
    m, t0, dt, nsteps = 1.1, 1.0, 0.05, 5
    rng = np.random.default_rng(N)
    x0 = rng.standard_normal((2, N, N, N))
    lam = rng.standard_normal((2, N, N, N))
    want, dm_want = reference(x0, lam, t0, dt, nsteps, m)
    c = cfb200.Context(N, float(N), m=m, equation=cfb200.EQ_KG_FRW, precision=prec, **FRW)
    st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
    c.upload(st, np.ascontiguousarray(x0.reshape(-1)))
    adj = cfb200.Adjoint(c, nsteps, 2)
    adj.forward(st, t0, dt)
    adj.set_lambda(torch.from_numpy(lam.reshape(-1)).cuda())
    out = torch.empty(2 * N ** 3, dtype=torch.float64, device="cuda")
    dm = adj.backward(out)
    got = out.cpu().numpy().reshape(want.shape)
    adj.close()
    c.close()
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
    scale = nsteps * dt * 2 * m * np.linalg.norm(lam[1]) * np.linalg.norm(x0[0])
    assert abs(dm - dm_want) <= (1e-12 if prec == cfb200.FP64 else 1e-5) * scale
