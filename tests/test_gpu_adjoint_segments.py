"""The adjoint's kept states: a checkpoint at every step (no kept states), in the middle of a run and
beyond its end give the same gradient, bit for bit, and so does a second reverse sweep."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stencil", [7, 13])
@pytest.mark.parametrize("prec", [cfb200.FP64, cfb200.FP32_COMP])
def test_checkpoint_distances(prec, stencil):
    N, steps = 24, 5
    c = cfb200.Context(N, float(N), m=1.1, equation=cfb200.EQ_KG_FRW, precision=prec, stencil=stencil, a1=1.0, H1=0.5, t1=1.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.randn(2 * N ** 3, generator=g, device="cuda", dtype=torch.float64)
    lam = torch.randn(2 * N ** 3, generator=g, device="cuda", dtype=torch.float64)
    seen = []
    for every in (1, 2, 5, 7):
        adj = cfb200.Adjoint(c, steps, every)
        st = torch.empty(c.info.state_bytes // 8, dtype=torch.float64, device="cuda")
        c.import_f64(st, x)
        adj.forward(st, 1.0, 0.05)
        for _ in range(2):
            out = torch.empty_like(lam)
            adj.set_lambda(lam)
            seen.append((adj.backward(out), out))
        adj.close()
    for dm, out in seen[1:]:
        assert dm == seen[0][0] and torch.equal(out, seen[0][1])
    c.close()
