"""The FP64 H_eff on plain blocks: term sums by products or by their own
kernel, weights beyond the kept copies of R, odd extents, and operators of
different K splits in one batch.  Tolerance against the oracle: the FP64 bar of
the parity tests (1e-12 in the 2-norm)."""

import numpy as np
import pytest

from oracle.blocksparse import Leg, OTensor, blockwise_contract

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import tenax_b200 as tb  # noqa: E402
from tenax_b200.auto_mpo import build_auto_mpo_sites, to_symmetric  # noqa: E402
from tenax_b200.tensor import SymmetricTensor, embed_in_keys  # noqa: E402
from tenax_b200.tensor import restrict_to_keys  # noqa: E402
from tenax_b200.workloads import chain_bulk_w, cylinder_bulk_w, make_heff_problem  # noqa: E402


def _random_couplings(L=10, reach=4, seed=0):
    """XXZ couplings of every pair up to ``reach`` apart, all different: more
    distinct W_l W_r weights than R copies are kept."""
    rng = np.random.default_rng(seed)
    terms = []
    for i in range(L):
        for j in range(i + 1, min(L, i + reach + 1)):
            a, b = rng.standard_normal(2)
            terms += [(a, "Sz", i, "Sz", j), (b, "Sp", i, "Sm", j), (b, "Sm", i, "Sp", j)]
    sites = build_auto_mpo_sites(terms, L)
    return to_symmetric(sites[4]), to_symmetric(sites[5])


MPOS = {"chain": chain_bulk_w, "cylinder": cylinder_bulk_w, "random": _random_couplings}


def _op(mpo, chi, seed, **kw):
    Wl, Wr = MPOS[mpo]()
    p = make_heff_problem(chi, chi, Wl, Wr, np.random.default_rng(seed), **kw)
    return p, tb.HeffOperator(p.L, p.Wl, p.Wr, p.R, p.theta.indices, p.theta.keys, "fp64")


def _host(t):
    return OTensor(tuple(Leg(i.charges, int(i.flow), i.label) for i in t.indices), t.numpy_blocks())


@pytest.mark.parametrize("mpo,chi,kw", [
    ("chain", 23, dict(n_sectors=5, hi=9, lo=1)),
    ("chain", 64, dict(n_sectors=9, hi=17, lo=1)),
    ("cylinder", 41, dict(n_sectors=7, hi=13, lo=1)),      # every term a product
    ("cylinder", 420, dict(n_sectors=6, hi=131, lo=3)),    # multi-term slots summed first
    ("random", 37, dict(n_sectors=7, hi=11, lo=1)),        # weights without a copy of R
    ("random", 200, dict(n_sectors=5, hi=65, lo=3)),
])
def test_matches_oracle(mpo, chi, kw):
    p, op = _op(mpo, chi, chi, **kw)
    x = embed_in_keys(p.theta, op.keys)
    out = torch.full_like(x.data, float("nan"))  # every element must be written
    op.apply(x.data, out)
    got = SymmetricTensor.from_flat(p.theta.indices, op.keys, out).numpy_blocks()
    ref = blockwise_contract([_host(t) for t in (p.L, x, p.Wl, p.Wr, p.R)], "abc,apqd,bpse,eqtf,dfg->cstg").blocks
    num = sum(float(np.sum((got[k] - ref.get(k, 0.0)) ** 2)) for k in got)
    den = sum(float(np.sum(v ** 2)) for v in ref.values())
    assert set(ref) <= set(got)
    assert (num / den) ** 0.5 < 1e-12


def test_batch_of_different_splits_equals_single_applies():
    probs = [_op("chain", 30, 1, n_sectors=5, hi=9, lo=1), _op("cylinder", 300, 2, n_sectors=12, hi=64),
             _op("random", 90, 3, n_sectors=5, hi=31, lo=1), _op("cylinder", 700, 4, n_sectors=8, hi=160)]
    ops = [o for _, o in probs]
    xs = [embed_in_keys(p.theta, o.keys).data for p, o in probs]
    singles = [o.apply(x) for o, x in zip(ops, xs)]
    batch = tb.HeffBatch(ops)
    outs = [o.out_like() for o in ops]
    batch.apply([x * 3.0 for x in xs], outs)  # other values in every intermediate first
    batch.apply(xs, outs)
    for a, b in zip(singles, outs):
        assert torch.equal(a, b)


def test_extreme_ranges_of_the_environments():
    """L near 1e-180 and R near 1e180: the powers of two divided out of both keep
    every intermediate in range, and the result is that of L and R near 1."""
    p, op = _op("chain", 40, 5, n_sectors=6, hi=12, lo=1)
    x = embed_in_keys(p.theta, op.keys).data
    y = op.apply(x)
    sc = 2.0 ** 600
    L = SymmetricTensor.from_flat(p.L.indices, p.L.keys, p.L.data / sc)
    R = SymmetricTensor.from_flat(p.R.indices, p.R.keys, p.R.data * sc)
    op2 = tb.HeffOperator(L, p.Wl, p.Wr, R, p.theta.indices, p.theta.keys, "fp64")
    assert torch.equal(op2.apply(x), y)


def test_long_block_strides():
    """theta[a, p, q, d] of 32 x 32 x 16384: its K stride is 2^24 elements, which
    in-tile offsets of 128 rows would not reach.  W_l W_r is the identity, so
    the result is L . theta . R; each of the two sums rounds within
    (K + 2) u of the sum of its magnitudes."""
    u1 = tb.U1Symmetry()
    IN, OUT = tb.FlowDirection.IN, tb.FlowDirection.OUT
    a, p, d = 2, 32, 16384

    def leg(n, flow, label):
        return tb.TensorIndex(u1, np.zeros(n, np.int32), flow, label)

    def tensor(*legs, data):
        return SymmetricTensor.from_flat(legs, [(0,) * len(legs)], data)

    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda n: torch.randn(n, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    eye = torch.eye(p, dtype=torch.float64, device="cuda").reshape(-1)
    L = tensor(leg(a, OUT, "a"), leg(1, IN, "b"), leg(a, IN, "c"), data=rnd(a * a))
    th = tensor(leg(a, IN, "a"), leg(p, IN, "p"), leg(p, IN, "q"), leg(d, OUT, "d"), data=rnd(a * p * p * d))
    W = [tensor(leg(1, OUT, "l"), leg(p, OUT, "i"), leg(p, IN, "o"), leg(1, IN, "r"), data=eye.clone()) for _ in range(2)]
    R = tensor(leg(d, IN, "d"), leg(1, OUT, "f"), leg(d, OUT, "g"), data=rnd(d * d))
    op = tb.HeffOperator(L, W[0], W[1], R, th.indices, th.keys, "fp64")
    got = op.apply(th.data).view(a, p * p, d)
    Lm, Rm, t = L.data.view(a, a), R.data.view(d, d), th.data.view(a, p * p * d)
    ref = ((Lm.T @ t).view(a * p * p, d) @ Rm).view(a, p * p, d)
    mag = ((Lm.abs().T @ t.abs()).view(a * p * p, d) @ Rm.abs()).view(a, p * p, d)
    assert bool(((got - ref).abs() <= 2.0 * (a + d + 4) * 2.0 ** -53 * mag).all())


def test_unreached_blocks_are_zero_when_the_scale_overflows():
    """L and R near 2^600: the factor that undoes their scaling is infinite, and
    theta blocks that no product reaches are still cleared."""
    p, op = _op("chain", 40, 6, n_sectors=6, hi=12, lo=1)
    x = embed_in_keys(p.theta, op.keys)
    qc = sorted({k[2] for k in p.L.keys})[2]
    keys = [k for k in p.L.keys if k[2] != qc]
    L = SymmetricTensor.from_flat(p.L.indices, keys, restrict_to_keys(p.L, keys).data * 2.0 ** 600)
    R = SymmetricTensor.from_flat(p.R.indices, p.R.keys, p.R.data * 2.0 ** 600)
    op2 = tb.HeffOperator(L, p.Wl, p.Wr, R, p.theta.indices, op.keys, "fp64")
    out = op2.apply(embed_in_keys(x, op2.keys).data, torch.full((op2.size,), 7.0, dtype=torch.float64, device="cuda"))
    got = SymmetricTensor.from_flat(p.theta.indices, op2.keys, out).numpy_blocks()
    unreached = [k for k in got if k[0] == qc]
    assert unreached and all(np.array_equal(got[k], np.zeros_like(got[k])) for k in unreached)


def test_large_weights_with_a_tiny_environment():
    """|R| in [2^-1021, 2^-1020) and W_l W_r weights above 2^5: R's share is
    scaled up before a weight multiplies it (2^1021 times the weight is out of
    range).  All factors are powers of two, so the bits are those of R near 1."""
    Wl, Wr = chain_bulk_w()
    Wl = SymmetricTensor.from_flat(Wl.indices, Wl.keys, Wl.data * 64.0)
    p = make_heff_problem(40, 40, Wl, Wr, np.random.default_rng(7), n_sectors=6, hi=12, lo=1)
    r = torch.sign(p.R.data) * (1.0 + p.R.data.abs().frac())
    ops = []
    for sL, sR in ((1.0, 1.0), (2.0 ** 600, 2.0 ** -1021)):
        L = SymmetricTensor.from_flat(p.L.indices, p.L.keys, p.L.data * sL)
        R = SymmetricTensor.from_flat(p.R.indices, p.R.keys, r * sR)
        ops.append(tb.HeffOperator(L, Wl, Wr, R, p.theta.indices, p.theta.keys, "fp64"))
    x = embed_in_keys(p.theta, ops[0].keys).data
    y, tiny = (op.apply(x) for op in ops)
    assert bool(torch.isfinite(y).all()) and torch.equal(tiny * 2.0 ** 421, y)
