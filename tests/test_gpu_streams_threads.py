"""The overlapping launch chains on a side stream, and two threads with plans
and operators of their own: the bits of the same calls one after another on the
default stream."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import tenax_b200 as tb  # noqa: E402
from tenax_b200 import dense  # noqa: E402
from tenax_b200.dmrg import lanczos  # noqa: E402
from tenax_b200.tensor import embed_in_keys  # noqa: E402
from tenax_b200.workloads import chain_bulk_w, make_heff_problem  # noqa: E402


def _chains(seed):
    """Calls of several launches each, all tensors their own: a three-operand
    contraction, one with its K in parts, and an operator's applies and solve."""
    g = torch.Generator().manual_seed(seed)
    t = [torch.randn(s, generator=g, dtype=torch.float64).cuda() for s in ((70, 90), (90, 110), (110, 50), (5, 9000), (9000, 7))]
    p3 = dense._DensePlan(["ab", "bc", "cd"], "da", [tuple(x.shape) for x in t[:3]], "fp64")
    pk = dense._DensePlan(["ak", "kb"], "ab", [tuple(x.shape) for x in t[3:]], "fp64")
    px = dense._DensePlan(["ab", "bc"], "ca", [tuple(x.shape) for x in t[:2]], "bf16x3")
    Wl, Wr = chain_bulk_w()
    p = make_heff_problem(48, 48, Wl, Wr, np.random.default_rng(seed), n_sectors=7, hi=14, lo=1)
    ops = [tb.HeffOperator(p.L, p.Wl, p.Wr, p.R, p.theta.indices, p.theta.keys, prec) for prec in ("fp64", "tf32")]
    x = embed_in_keys(p.theta, ops[0].keys)

    def run(n):
        out = []
        for _ in range(n):
            y = ops[0].apply(ops[0].apply(x.data))
            out = [p3(*t[:3]), pk(*t[3:]), px(*t[:2]), y, ops[1].apply(x.data)]
            e, v, _ = lanczos(ops[0], x, 6, 1e-10)[:3]
            out += [torch.tensor(e), v.data]
        return out

    return run


def test_side_stream():
    run = _chains(1)
    ref = run(1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = run(8)
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(ref, got))


def test_two_threads():
    runs = [_chains(2), _chains(3)]
    refs = [r(1) for r in runs]
    torch.cuda.synchronize()
    got, errors = [None, None], []

    def work(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                got[i] = runs[i](20)
            s.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors
    for ref, g in zip(refs, got):
        assert all(torch.equal(a, b) for a, b in zip(ref, g))
