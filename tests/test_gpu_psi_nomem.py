"""A step that finds no room for all three Psi slots reports it, as often as it is asked; with room it
takes the missing ones and gives the bits of a context that always had them."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402
from cfb200 import fields  # noqa: E402

pytestmark = pytest.mark.gpu


def test_no_room_then_room():
    N = 256  # 268 MB a slot
    R = torch.from_numpy(fields.curvature_R_fft(N, float(N), 2.0, 1e-2, 0.2, seed=6)).cuda()
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(2 * N ** 3, generator=g, device="cuda", dtype=torch.float64)

    def context():
        c = cfb200.Context(N, float(N), equation=cfb200.EQ_COMOVING_FRW, a1=1.0, H1=0.5, t1=1.0)
        c.set_R_fft(R, on_device=True)
        return c

    full = context()
    want = x.clone()
    full.rk4_steps(want, 1.0, 0.05, 1)
    torch.cuda.synchronize()
    full.close()
    c = context()
    got = x.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")  # room for one slot
    for _ in range(2):
        with pytest.raises(cfb200.CfError, match="NOMEM"):
            c.energy_density(got, 1.0, filler[: 8 * N ** 3].view(torch.float64))
    del filler
    torch.cuda.empty_cache()
    c.rk4_steps(got, 1.0, 0.05, 1)
    assert torch.equal(got, want)
    c.close()
