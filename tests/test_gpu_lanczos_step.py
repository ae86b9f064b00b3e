"""One Lanczos step and the dot/norm primitives on both sides of the
one-launch limit (65536 elements) and of the cluster sizes, against host
sums.  A sum of n products in any order is within n u of the sum of their
magnitudes (u = 2^-53)."""

import math

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from tenax_b200 import _capi, vector  # noqa: E402

U = 2.0 ** -53


def _step(w, v, vp, vn, n, alpha, beta, k, tol, tol_rel, done):
    _capi.check(_capi.LIB.tnx_lanczos_step(w.data_ptr(), v.data_ptr(), 0 if vp is None else vp.data_ptr(),
                                           vn.data_ptr(), n, alpha.data_ptr(), beta.data_ptr(), k, tol, tol_rel,
                                           done.data_ptr(), vector.scratch(w.device).data_ptr(),
                                           torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 16385, 65535, 65536, 65537, 300001])
@pytest.mark.parametrize("k", [0, 1])
def test_step(n, k):
    g = torch.Generator().manual_seed(n)
    w0, v, vp = (torch.randn(n, generator=g, dtype=torch.float64) for _ in range(3))
    d = [x.cuda() for x in (w0, v, vp)]
    alpha = torch.zeros(3, dtype=torch.float64, device="cuda")
    beta = torch.full((4,), 0.75, dtype=torch.float64, device="cuda")
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    vn = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    _step(d[0], d[1], d[2] if k else None, vn, n, alpha, beta, k, 0.0, 0.0, done)
    a = float(alpha[k])
    assert abs(a - math.fsum((v * w0).tolist())) <= (n + 2) * U * math.fsum((v * w0).abs().tolist())
    x = w0 - v * a - (vp * 0.75 if k else 0.0)  # the recurrence with the device's alpha
    tol = 4 * U * (w0.abs() + (v * a).abs() + (vp * 0.75).abs() * k)
    assert bool(((d[0].cpu() - x).abs() <= tol).all())
    b2 = math.fsum((d[0].cpu() ** 2).tolist())
    assert abs(float(beta[k + 1]) ** 2 - b2) <= (n + 4) * U * b2
    if b2 > 0:
        ref = d[0].cpu() / float(beta[k + 1])
        assert bool(((vn.cpu() - ref).abs() <= 4 * U * ref.abs()).all())
    assert int(done) == 0


@pytest.mark.parametrize("n", [5, 4096, 65537])
def test_stop_and_skip(n):
    w, v = torch.ones(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    alpha = torch.zeros(2, dtype=torch.float64, device="cuda")
    beta = torch.zeros(3, dtype=torch.float64, device="cuda")
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    vn = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    _step(w, v, None, vn, n, alpha, beta, 0, 1e300, 0.0, done)  # beta below tol: stop, next vector not written
    assert int(done) == 1 and bool((vn == 7.0).all())
    assert float(alpha[0]) == float(n)
    before = [t.clone() for t in (w, alpha, beta, vn)]
    _step(w, v, v, vn, n, alpha, beta, 1, 0.0, 0.0, done)  # done: nothing changes
    assert all(torch.equal(x, y) for x, y in zip(before, (w, alpha, beta, vn)))


@pytest.mark.parametrize("n", [0, 1, 2048, 2049, 65536, 65537])
def test_dot_and_norm(n):
    g = torch.Generator().manual_seed(n + 1)
    x, y = (torch.randn(n, generator=g, dtype=torch.float64) for _ in range(2))
    d = float(vector.dot(x.cuda(), y.cuda()))
    assert abs(d - math.fsum((x * y).tolist())) <= (n + 2) * U * math.fsum((x * y).abs().tolist())
    nn = float(vector.nrm2(x.cuda()))
    assert abs(nn - math.sqrt(math.fsum((x * x).tolist()))) <= (n + 4) * U * max(nn, 1e-300)


@pytest.mark.parametrize("n", [65537, 300001, 2000003])
def test_no_block_writes_the_next_vector_on_a_stop(n):
    """The three-launch step stops in the launch that would write v_next, while
    its blocks start: none of them may write, in any of many steps."""
    w, v = torch.ones(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    alpha = torch.zeros(2, dtype=torch.float64, device="cuda")
    beta = torch.zeros(3, dtype=torch.float64, device="cuda")
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    vn = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    for _ in range(200):
        w.fill_(1.0)
        done.zero_()
        _step(w, v, None, vn, n, alpha, beta, 0, 1e300, 0.0, done)
    assert int(done) == 1 and bool((vn == 7.0).all())
