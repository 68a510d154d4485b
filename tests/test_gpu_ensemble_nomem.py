"""Ensemble spectra that find no room leave nothing half made: the call reports it each time and works
once there is room."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


def test_no_room_then_room():
    spec = [dict(N=N, L=float(N), m=1.0, equation=cfb200.EQ_KG_FRW, precision=cfb200.FP64, stencil=7, a1=1.0, H1=0.5,
                 t1=1.0) for N in (32, 256)]  # the larger class: 134 MB of density, 135 of half-complex field

    def ensemble():
        e = cfb200.Ensemble(spec)
        for i, d in enumerate(spec):
            e.upload(i, np.random.default_rng(i).standard_normal(2 * d["N"] ** 3))
        torch.cuda.synchronize()
        return e

    full = ensemble()
    want = torch.empty(full.spectra_total, dtype=torch.float64, device="cuda")
    full.density_spectra_s2(1.0, want)
    torch.cuda.synchronize()
    full.close()
    e = ensemble()
    got = torch.empty_like(want)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")  # the density of the larger class only
    for _ in range(2):
        with pytest.raises(cfb200.CfError):
            e.density_spectra_s2(1.0, got)
    del filler
    torch.cuda.empty_cache()
    e.density_spectra_s2(1.0, got)
    assert torch.equal(got, want)
    e.close()
