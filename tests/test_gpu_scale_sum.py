"""cf_scale_sum: the vector form (16-byte aligned arrays, an even length, up to six inputs) and the
general one give the same bits: the same products and sums in the same order."""
import pytest

torch = pytest.importorskip("torch")

import cfb200  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 14])
@pytest.mark.parametrize("length", [1, 2, 1023, 1024, 2 * 40 ** 3])
def test_vector_form(n, length):
    c = cfb200.Context(8, 8.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    room = [torch.randn(length + 1, generator=g, device="cuda", dtype=torch.float64) for _ in range(n)]
    alpha = [1.0, 0.025, -0.3, 1 / 3, 0.7, 1e-3, 2.0, 3.0, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6][:n]
    aligned = [r[:length] for r in room]
    shifted = [r.clone()[1:] for r in [torch.cat([r[:1], r[:length]]) for r in room]]  # 8-byte aligned
    a, b = torch.empty(length, device="cuda", dtype=torch.float64), torch.empty(length + 1, device="cuda", dtype=torch.float64)[1:]
    c.scale_sum(a, aligned, alpha, length)
    c.scale_sum(b, shifted, alpha, length)
    assert torch.equal(a, b)
    c.scale_sum(aligned[0], aligned, alpha, length)  # in place
    assert torch.equal(aligned[0], a)
    c.close()
