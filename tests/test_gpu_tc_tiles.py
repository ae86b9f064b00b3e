"""tcgen05 GEMM tiles: launches of few tiles (cut to 64 or 32 columns, more
pipeline stages) and operand loads trimmed to ragged rows give the same bits
as the 128-column tiles of a large launch, and lie within the split's error.

Split BF16 keeps 16 bits of each operand: |err| <= 2^-15 |a||b| summed, plus
FP32 accumulation; TF32 keeps 11: 2^-10."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from tenax_b200 import dense  # noqa: E402

BIG = 128 * 160  # more 128-row tiles than the GPU has SMs


@pytest.mark.parametrize("precision,eps", [("bf16x3", 2.0 ** -15), ("tf32", 2.0 ** -10)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (7, 16, 31), (8, 17, 64), (9, 33, 65), (100, 64, 300), (128, 65, 33),
                                   (129, 100, 129), (200, 128, 257), (64, 129, 64), (130, 200, 1000)])
def test_few_tiles_equal_many(precision, eps, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + 31 * n + 7 * k)
    a = torch.randn(BIG, k, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(n, k, generator=g, dtype=torch.float64, device="cuda")
    big = dense.einsum("mk,nk->mn", a, b, precision=precision)
    few = dense.einsum("mk,nk->mn", a[:m].contiguous(), b, precision=precision)
    assert torch.equal(few, big[:m])
    ref, mag = a[:m] @ b.T, a[:m].abs() @ b.abs().T
    assert bool(((few - ref).abs() <= (eps + (k + 4) * 2.0 ** -24) * mag).all())


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
def test_plan_buffers_hold_nothing_of_the_last_call(precision):
    """A plan's operand images are cleared once and refilled by every call: a
    call after one with NaN and other values equals a fresh plan's."""
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(37, 5, 9, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(9, 21, 5, generator=g, dtype=torch.float64, device="cuda")
    dense._PLANS.clear()
    fresh = dense.einsum("mak,kna->nm", a, b, precision=precision)
    dense._PLANS.clear()
    dense.einsum("mak,kna->nm", torch.full_like(a, float("nan")), b * 1e30, precision=precision)
    assert torch.equal(dense.einsum("mak,kna->nm", a, b, precision=precision), fresh)


@pytest.mark.parametrize("precision", ["bf16x3", "tf32"])
@pytest.mark.parametrize("n,k", [(129, 31), (200, 64), (256, 130), (300, 65), (513, 33)])
def test_wide_tiles_equal_narrow(precision, n, k):
    """Launches of many tiles take 256 columns at a time: the same bits as one
    row tile alone (32 or 64 columns)."""
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a = torch.randn(128 * 620, k, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(n, k, generator=g, dtype=torch.float64, device="cuda")
    big = dense.einsum("mk,nk->mn", a, b, precision=precision)
    for r0 in (0, 128 * 333):
        rows = a[r0:r0 + 100].contiguous()
        assert torch.equal(dense.einsum("mk,nk->mn", rows, b, precision=precision), big[r0:r0 + 100])
