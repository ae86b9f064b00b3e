"""The one-launch FP64 contraction: tile edges, remainders, leg orders, K
splits, against plain torch on the host and against the packed path.

Both sides sum K products in some order, each rounding within u = 2^-53 of
the exact sum of |a||b|, so they differ by at most 2 (K + 2) u (|A| |B|)
entry by entry.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import tenax_b200 as tb  # noqa: E402
from tenax_b200 import _capi, dense  # noqa: E402
from tenax_b200.contraction import get_plan  # noqa: E402

IN, OUT = tb.FlowDirection.IN, tb.FlowDirection.OUT


def _check(subs, sa, sb, seed=0):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn(sa, generator=g, dtype=torch.float64)
    b = torch.randn(sb, generator=g, dtype=torch.float64)
    got = dense.einsum(subs, a.cuda(), b.cuda()).cpu()
    ref = torch.einsum(subs, a, b)
    mag = torch.einsum(subs, a.abs(), b.abs())
    lhs, so = subs.split("->")
    dims = dict(zip(lhs.replace(",", ""), (*sa, *sb)))
    k = int(np.prod([n for c, n in dims.items() if c not in so]))
    assert got.shape == ref.shape
    assert bool(((got - ref).abs() <= 2.0 * (k + 2) * 2.0 ** -53 * mag).all()), (subs, sa, sb)


# every pair of fast axes (K or free, in A and in B) and of output orders
ORDERS = ["mk,kn->mn", "km,kn->mn", "mk,nk->mn", "km,nk->nm"]


@pytest.mark.parametrize("subs", ORDERS)
@pytest.mark.parametrize("m,n,k", [
    (1, 1, 1), (1, 9, 3), (8, 8, 4), (7, 33, 5), (31, 17, 16), (32, 32, 15), (33, 65, 17), (64, 64, 64),
    (65, 63, 63), (127, 16, 31), (128, 17, 32), (129, 15, 33), (500, 8, 26), (16, 16, 1280), (80, 80, 1280),
    (80, 80, 1279), (640, 640, 37), (1500, 9, 3),
])
def test_matrix_edges(subs, m, n, k):
    d = {"m": m, "n": n, "k": k}
    lhs = subs.split("->")[0].split(",")
    _check(subs, tuple(d[c] for c in lhs[0]), tuple(d[c] for c in lhs[1]), seed=m * 7 + n * 3 + k)


@pytest.mark.parametrize("subs,sa,sb", [
    ("axby,xcyd->dbca", (5, 3, 7, 11), (3, 6, 11, 9)),    # interleaved legs on both sides
    ("yaxb,dxcy->acbd", (11, 5, 3, 7), (9, 3, 6, 11)),
    ("pxq,qwB->pxwB", (20, 9, 20), (20, 9, 20)),
    ("pxwB,swxt->pBst", (20, 9, 9, 20), (9, 9, 9, 9)),
    ("psA,pBst->AtB", (20, 9, 20), (20, 20, 9, 9)),
    ("a,b->ab", (70,), (130,)),                            # no contracted leg
    ("ab,ab->", (40, 50), (40, 50)),                       # no free leg: K = 2000 in one output
    ("abc,b->ca", (6, 1, 9), (1,)),                        # extent-1 contracted leg
])
def test_leg_orders(subs, sa, sb):
    _check(subs, sa, sb)


@pytest.mark.parametrize("sym,n", [(tb.U1Symmetry(), None), (tb.ZnSymmetry(3), 3)])
@pytest.mark.parametrize("sizes", [(1, 2, 1), (3, 17, 8), (40, 70, 33)])
def test_blocks_match_packed_path(sym, n, sizes):
    """Ragged sectors, several contracted legs and several K blocks of one
    output block, on odd offsets: the one-launch result against the packed
    path of the allocation-free entry point."""
    q = np.repeat(np.array([-1, 0, 1] if n is None else [0, 1, 2]), sizes).astype(np.int32)
    p = np.array([0, 1, 1], np.int32)
    ia = (tb.TensorIndex(sym, q, IN, "a"), tb.TensorIndex(sym, p, IN, "x"), tb.TensorIndex(sym, q[::-1].copy(), OUT, "m"),
          tb.TensorIndex(sym, p, OUT, "b"))
    ib = (tb.TensorIndex(sym, p, OUT, "x"), tb.TensorIndex(sym, q, OUT, "c"), tb.TensorIndex(sym, q[::-1].copy(), IN, "m"))
    a, b = tb.SymmetricTensor.random_normal(ia, key=1), tb.SymmetricTensor.random_normal(ib, key=2)
    for out in ("abc", "cab", "bca"):
        idx = {"a": ia[0], "b": ia[3], "c": ib[1]}
        plan = get_plan([a, b], ["axmb", "xcm"], out, _capi.MATCH_UNFILTERED, tuple(idx[ch] for ch in out))
        got = plan.execute([a, b], "fp64")
        ref = torch.full((plan.total,), float("nan"), dtype=torch.float64, device="cuda")
        ptrs = (C.c_void_p * 2)(a.data.data_ptr(), b.data.data_ptr())
        _capi.check(_capi.LIB.tnx_plan_execute_static(plan.handle, ptrs, ref.data_ptr(),
                                                     torch.cuda.current_stream().cuda_stream))
        k = 3 * sum(sizes)
        scale = float(a.data.abs().max()) * float(b.data.abs().max())
        assert float((got - ref).abs().max()) <= 2.0 * (k + 2) * 2.0 ** -53 * k * scale


def test_non_finite_values_stay_in_their_row():
    """A row of A with an infinity and a NaN: only that row of C is touched."""
    a = torch.ones(70, 37, dtype=torch.float64)
    a[5, 3], a[5, 30] = float("inf"), float("nan")
    b = torch.ones(37, 66, dtype=torch.float64)
    got = dense.einsum("mk,kn->mn", a.cuda(), b.cuda()).cpu()
    assert bool(torch.isnan(got[5]).all())
    keep = [i for i in range(70) if i != 5]
    assert bool((got[keep] == 37.0).all())


# K shared out over several clusters of one output tile, whose parts a second
# launch adds: 16 to 32 parts of these shapes
@pytest.mark.parametrize("subs", ORDERS)
@pytest.mark.parametrize("m,n,k", [(16, 16, 8000), (4, 4, 102400), (5, 13, 20001), (13, 5, 20000), (33, 70, 20011),
                                   (70, 33, 20011), (129, 9, 30000)])
def test_long_k_in_parts(subs, m, n, k):
    d = {"m": m, "n": n, "k": k}
    lhs = subs.split("->")[0].split(",")
    _check(subs, tuple(d[c] for c in lhs[0]), tuple(d[c] for c in lhs[1]), seed=m * 7 + n * 3 + k)


@pytest.mark.parametrize("subs,sa,sb", [
    ("aklx,ylkb->bxya", (3, 150, 140, 5), (7, 140, 150, 4)),   # output legs of both operands interleaved
    ("kalx,ylbk->xyab", (150, 3, 140, 9), (7, 140, 4, 150)),
])
def test_long_k_in_parts_leg_orders(subs, sa, sb):
    _check(subs, sa, sb)


@pytest.mark.parametrize("order", ["ab", "ba"])
def test_long_k_in_parts_of_blocks(order):
    """Three sectors of different K, so shares of different lengths in one
    launch; ragged rows and columns; the output in both orders."""
    u1 = tb.U1Symmetry()
    rows = np.repeat(np.array([-1, 0, 1], np.int32), (5, 9, 13))
    cols = np.repeat(np.array([-1, 0, 1], np.int32), (11, 3, 8))
    k = np.repeat(np.array([-1, 0, 1], np.int32), (20011, 7000, 12345))
    a = tb.SymmetricTensor.random_normal((tb.TensorIndex(u1, rows, IN, "a"), tb.TensorIndex(u1, k, OUT, "k")), key=1)
    b = tb.SymmetricTensor.random_normal((tb.TensorIndex(u1, k, IN, "k"), tb.TensorIndex(u1, cols, OUT, "b")), key=2)
    idx = {"a": a.indices[0], "b": b.indices[1]}
    plan = get_plan([a, b], ["ak", "kb"], order, _capi.MATCH_UNFILTERED, tuple(idx[c] for c in order))
    got = plan.wrap(tuple(idx[c] for c in order), plan.execute([a, b], "fp64")).todense()
    da, db = a.todense(), b.todense()
    ref, mag = torch.einsum(f"ak,kb->{order}", da, db), torch.einsum(f"ak,kb->{order}", da.abs(), db.abs())
    assert bool(((got - ref).abs() <= 2.0 * (20011 + 2) * 2.0 ** -53 * mag).all())
