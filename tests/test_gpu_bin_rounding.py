"""The bins' last step, 128-bit fixed point to double, rounds once.

A field of one site A has every mode equal to A; with A of 26 bits the mode values A^2 and the bins,
A^2 times the modes they hold, are exact in the fixed point, so a bin is that product rounded once."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 16, 32])
@pytest.mark.parametrize("A", [67108859 / 2 ** 26, 40265327 / 2 ** 26, 53687089 / 2 ** 20, 33554467 / 2 ** 40])
def test_one_site(N, A):
    c = cfb200.Context(N, float(N))
    f = torch.zeros(N ** 3, dtype=torch.float64, device="cuda")
    f[0] = A
    out = torch.empty(c.info.s2_bins, dtype=torch.float64, device="cuda")
    shells = torch.empty(c.info.shells, dtype=torch.float64, device="cuda")
    counts = torch.empty(c.info.s2_bins, dtype=torch.int64, device="cuda")
    in_shell = torch.empty(c.info.shells, dtype=torch.int64, device="cuda")
    c.power_spectrum_s2(f, out)
    c.s2_counts(counts)
    c.s2_to_shells(shells, in_shell)
    assert torch.equal(out, counts.double() * (A * A))
    assert torch.equal(shells, in_shell.double() * (A * A))
    c.close()
