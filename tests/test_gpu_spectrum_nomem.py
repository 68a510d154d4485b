"""A spectrum call that finds no room for its scratch leaves none of it behind: it reports the lack of
memory, and the next call with room takes a whole one.  The slices do without."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


def test_no_room_then_room():
    N = 256  # the half-complex fields 270 MB, the fields 268 MB, and transforms
    c = cfb200.Context(N, float(N), equation=cfb200.EQ_KG_FRW, a1=1.0, H1=0.5, t1=1.0)
    full = cfb200.Context(N, float(N), equation=cfb200.EQ_KG_FRW, a1=1.0, H1=0.5, t1=1.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(2 * N ** 3, generator=g, device="cuda", dtype=torch.float64)
    out, want = (torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda") for _ in range(2))
    mean, mean_want = (torch.empty(N * N, dtype=torch.float64, device="cuda") for _ in range(2))
    full.density_spectrum_s2(x, 1.0, want)
    full.density_slices(x, 1.0, None, mean_want)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")  # room for the first piece only
    for _ in range(2):
        with pytest.raises(cfb200.CfError, match="NOMEM"):
            c.density_spectrum_s2(x, 1.0, out)
    c.density_slices(x, 1.0, None, mean)
    assert torch.equal(mean, mean_want)
    del filler
    torch.cuda.empty_cache()
    c.density_spectrum_s2(x, 1.0, out)
    assert torch.equal(out, want)
    c.close()
    full.close()
