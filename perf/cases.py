"""The calls whose speed is followed, from the smallest to the largest.

Each case is one call (or one short chain of calls) of the package's public
entry points on seeded synthetic inputs, over the sizes of the spin-1/2
Heisenberg chain (L = 20, chi = 64) and of the width-6 Heisenberg cylinder
(MPO bond 26, about 30 U(1) sectors a bond, chi up to 2048), and of CTM
environments of iPEPS with D = 2 to 5.

Kinds of case:

``contract``  theta = A . B, the two-site tensor that every DMRG step forms
              from two neighbouring MPS sites; ``precision`` as the caller of
              ``contract`` chooses it.
``grad``      ``contract_ad``: the same product and the gradients of both
              operands, as a variational optimisation calls it.
``env``       ``update_left_env`` / ``update_right_env``: the four-operand
              environment update after each DMRG step.
``heff``      one application of the two-site effective Hamiltonian, for one
              problem (``HeffOperator.apply``) or a batch (``HeffBatch``).
``lanczos``   a whole eigensolve of one site pair: Krylov loop, the read-back
              and the Ritz vector.
``ctm``       dense CTM sweeps with given projectors, the energy and its
              gradient in the site tensor: one optimisation step of an iPEPS
              whose projectors are held fixed.
``fuse``      ``fuse_indices`` of a grown CTM corner or edge (pure data
              movement).
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import tenax_b200 as tb
from tenax_b200.dmrg import lanczos, update_left_env, update_right_env
from tenax_b200.ipeps import CTMConfig, compute_energy_ctm, ctm, heisenberg_gate
from tenax_b200.tensor_utils import fuse_indices
from tenax_b200.workloads import chain_bulk_w, cylinder_bulk_w

IN, OUT = tb.FlowDirection.IN, tb.FlowDirection.OUT
U1 = tb.U1Symmetry()


def listed() -> list:
    return [
        # theta of the L=20 chain at chi=64: a call dominated by latency
        {"name": "theta_chain_chi64", "kind": "contract", "chi": 64, "sectors": 9, "precision": "fp64"},
        # theta of the cylinder at the headline bond dimension, DMRG's default precision
        {"name": "theta_cylinder_chi2048", "kind": "contract", "chi": 2048, "sectors": 30, "precision": "fp64"},
        # the same product with split-BF16 GEMMs, as a mixed-precision caller asks for it
        {"name": "theta_bf16x3_chi1024", "kind": "contract", "chi": 1024, "sectors": 30, "precision": "bf16x3"},
        # forward and both gradients; odd, ragged sectors
        {"name": "contract_grad_chi333", "kind": "grad", "chi": 333, "sectors": 11, "precision": "fp64"},
        # environment update of the cylinder (MPO bond 26), always FP64 in DMRG
        {"name": "env_left_cylinder_chi512", "kind": "env", "side": "left", "mpo": "cylinder", "chi": 512,
         "sectors": 30, "precision": "fp64"},
        # H_eff of the L=20 chain at chi=64: the launch-bound matvec
        {"name": "heff_chain_chi64_fp64", "kind": "heff", "mpo": "chain", "chis": "64", "sectors": 9,
         "precision": "fp64"},
        # H_eff of the cylinder in FP64: the matvec of a default DMRG run
        {"name": "heff_cylinder_chi1024_fp64", "kind": "heff", "mpo": "cylinder", "chis": "1024", "sectors": 30,
         "precision": "fp64"},
        # H_eff of the cylinder in TF32, one problem: small sectors
        {"name": "heff_cylinder_chi512_tf32", "kind": "heff", "mpo": "cylinder", "chis": "512", "sectors": 30,
         "precision": "tf32"},
        # a quarter of the 64-problem batch of mixed bond dimensions, split-BF16
        {"name": "heff_batch16_bf16x3", "kind": "heff", "mpo": "cylinder",
         "chis": "2048 1024 1024 512 256 256 256 256 256 2048 1024 2048 1024 1024 2048 1024", "sectors": 30,
         "precision": "bf16x3"},
        # the eigensolve of one site pair of the L=20 chain (10 Lanczos steps)
        {"name": "lanczos_chain_chi64", "kind": "lanczos", "mpo": "chain", "chis": "64", "sectors": 9,
         "precision": "fp64", "steps": 10},
        # one optimisation step of a D=4, chi=80 iPEPS: two CTM sweeps, energy, gradient
        {"name": "ctm_grad_D4_chi80", "kind": "ctm", "D": 4, "chi": 80, "sweeps": 2},
        # the leg fusion of a grown D=5, chi=150 edge with U(1) legs
        {"name": "fuse_D5_chi150", "kind": "fuse", "D": 5, "chi": 150, "adjacent": True},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["contract", "contract", "grad", "env", "heff", "heff", "lanczos", "ctm", "fuse"])
    sectors = rng.choice([5, 9, 11, 17, 24, 30])
    mpo = rng.choice(["chain", "cylinder"])
    if kind == "contract":
        return {"kind": kind, "chi": _log_int(rng, 48, 2048), "sectors": sectors,
                "precision": rng.choice(["fp64", "fp64", "bf16x3", "tf32"])}
    if kind == "grad":
        return {"kind": kind, "chi": _log_int(rng, 48, 1100), "sectors": sectors, "precision": "fp64"}
    if kind == "env":
        return {"kind": kind, "side": rng.choice(["left", "right"]), "mpo": mpo, "chi": _log_int(rng, 48, 700),
                "sectors": sectors, "precision": rng.choice(["fp64", "fp64", "bf16x3"])}
    if kind == "heff":
        n = rng.choice([1, 1, 2, 5])
        return {"kind": kind, "mpo": mpo, "chis": " ".join(str(_log_int(rng, 64, 1400)) for _ in range(n)),
                "sectors": sectors, "precision": rng.choice(["fp64", "bf16x3", "tf32"])}
    if kind == "lanczos":
        return {"kind": kind, "mpo": mpo, "chis": str(_log_int(rng, 48, 700)), "sectors": sectors,
                "precision": "fp64", "steps": rng.randint(4, 12)}
    if kind == "ctm":
        return {"kind": kind, "D": rng.choice([2, 3, 4]), "chi": rng.randint(12, 90), "sweeps": rng.choice([1, 2])}
    return {"kind": kind, "D": rng.choice([3, 4, 5]), "chi": rng.randint(30, 160), "adjacent": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _bond(chi: int, sectors: int, parity: int) -> np.ndarray:
    """Charges of one bond: ``sectors`` charges of one parity, sizes
    proportional to exp(-q^2 / 18), at least 1 and at most 256 (more only
    where ``sectors`` of 256 cannot hold chi), summing to chi."""
    q = (parity % 2) + 2 * (np.arange(sectors) - sectors // 2)
    g = np.exp(-(q.astype(np.float64) ** 2) / 18.0)
    cap = max(256, -(-chi // sectors))
    lo, hi = 0.0, 1e9 * chi
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if np.clip(np.floor(mid * g), 1, cap).sum() < chi else (lo, mid)
    size = np.clip(np.floor(lo * g), 1, cap).astype(np.int64)
    order = np.argsort(-g, kind="stable")
    i = 0
    while size.sum() != chi:
        j = order[i % sectors]
        i += 1
        if size.sum() < chi:
            size[j] += size[j] < cap
        elif size[j] > 1:
            size[j] -= 1
    return np.repeat(q, size).astype(np.int32)


def _tensor(legs, gen) -> tb.SymmetricTensor:
    """N(0,1) blocks on every charge-conserving key of ``legs`` =
    [(charges, flow, label), ...], scaled to a Frobenius norm of about 1."""
    idx = tuple(tb.TensorIndex(U1, c, f, lab) for c, f, lab in legs)
    dims = [dict(zip(*(x.tolist() for x in np.unique(c, return_counts=True)))) for c, _, _ in legs]
    keys = [()]
    for d in dims[:-1]:
        keys = [k + (q,) for k in keys for q in d]
    full = []
    for k in keys:
        last = -int(legs[-1][1]) * sum(int(f) * q for (_, f, _), q in zip(legs, k))
        if last in dims[-1]:
            full.append(k + (last,))
    full.sort()
    n = sum(math.prod(d[q] for d, q in zip(dims, k)) for k in full)
    data = torch.randn(n, generator=gen, dtype=torch.float64, device="cuda") / math.sqrt(max(1, n))
    return tb.SymmetricTensor.from_flat(idx, full, data)


@functools.lru_cache(maxsize=None)
def _mpo(name: str):
    return cylinder_bulk_w() if name == "cylinder" else chain_bulk_w()


PHYS = np.array([1, -1], np.int32)


def _site(vl, vr, names, gen):
    return _tensor([(vl, IN, names[0]), (PHYS, IN, names[1]), (vr, OUT, names[2])], gen)


def _generator(seed: int) -> torch.Generator:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _inputs(case: dict, seed: int) -> dict:
    gen = _generator(seed)
    kind = case["kind"]
    if kind in ("contract", "grad"):
        chi, ns = case["chi"], case["sectors"]
        v0, v1 = _bond(chi, ns, 1), _bond(chi, ns, 0)
        s = {"A": _site(v0, v1, ("vl", "p0", "vm"), gen), "B": _site(v1, v0, ("vm", "p1", "vr"), gen)}
        if kind == "grad":
            # on the blocks the product writes
            C, _ = _pair_shapes("apm", _of(s["A"]), "mqb", _of(s["B"]), "apqb")
            n = _elems(C)
            s["cotangent"] = tb.SymmetricTensor.from_flat(
                s["A"].indices[:2] + s["B"].indices[1:], sorted(C),
                torch.randn(n, generator=gen, dtype=torch.float64, device="cuda") / math.sqrt(n))
        return s
    if kind == "env":
        wl, _ = _mpo(case["mpo"])
        vl, vr = _bond(case["chi"], case["sectors"], 1), _bond(case["chi"], case["sectors"], 0)
        s = {"A": _site(vl, vr, ("v0", "p", "v1"), gen), "W": wl}
        if case["side"] == "left":
            v, w, f = vl, wl.indices[0].charges, IN
        else:
            v, w, f = vr, wl.indices[3].charges, OUT
        # q_ket = q_mpo + q_bra
        s["env"] = _tensor([(v, OUT if f is IN else IN, "k"), (w, f, "w"), (v, f, "b")], gen)
        return s
    if kind in ("heff", "lanczos"):
        wl, wr = _mpo(case["mpo"])
        problems = []
        for chi in (int(x) for x in case["chis"].split()):
            v = _bond(chi, case["sectors"], 1)
            L = _tensor([(v, OUT, "k"), (wl.indices[0].charges, IN, "w"), (v, IN, "b")], gen)
            th = _tensor([(v, IN, "vl"), (PHYS, IN, "p1"), (PHYS, IN, "p2"), (v, OUT, "vr")], gen)
            R = _tensor([(v, OUT, "k"), (wr.indices[3].charges, IN, "w"), (v, IN, "b")], gen)
            problems.append((L, wl, wr, R, th))
        return {"problems": problems}
    if kind == "ctm":
        D, chi = case["D"], case["chi"]
        A = torch.randn(D, D, D, D, 2, generator=gen, dtype=torch.float64, device="cuda") / math.sqrt(2 * D ** 4)
        n = chi * D * D
        P = []
        for _ in range(4 * case["sweeps"]):
            q, _r = torch.linalg.qr(torch.randn(n, chi, generator=gen, dtype=torch.float64, device="cuda"))
            P.append(q.contiguous())
        return {"A": A, "P": P}
    D, chi = case["D"], case["chi"]
    d2 = np.add.outer(np.arange(D) - D // 2, -(np.arange(D) - D // 2)).reshape(-1).astype(np.int32)
    qs = np.arange(-3, 4)
    x = np.sort(np.resize(qs, chi)).astype(np.int32)
    t = _tensor([(x, IN, "x"), (d2, IN, "u"), (d2, OUT, "r"), (x, OUT, "y")], gen)
    return {"t": t}


def prepare(case: dict, seed: int) -> dict:
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "heff":
        ops = [tb.HeffOperator(L, wl, wr, R, th.indices, th.keys, case["precision"])
               for L, wl, wr, R, th in s["problems"]]
        s["ops"] = ops
        s["x"] = [p[4].data for p in s["problems"]]
        s["y"] = [torch.empty_like(x) for x in s["x"]]
        if len(ops) > 1:
            s["batch"] = tb.HeffBatch(ops)
        del s["problems"]  # the operators hold what they need
    elif case["kind"] == "lanczos":
        (L, wl, wr, R, th), = s.pop("problems")
        s["op"] = tb.HeffOperator(L, wl, wr, R, th.indices, th.keys, case["precision"])
        s["theta"] = th
    elif case["kind"] == "ctm":
        s["A"].requires_grad_(True)
        s["gate"] = heisenberg_gate()
        s["config"] = CTMConfig(chi=case["chi"], max_iter=case["sweeps"], conv_tol=0.0)
    elif case["kind"] == "grad":
        s["A"].data.requires_grad_(True)
        s["B"].data.requires_grad_(True)
    return s


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "contract":
        return tb.contract(s["A"], s["B"], precision=case["precision"]).data
    if kind == "grad":
        out = tb.contract_ad(s["A"], s["B"], precision=case["precision"])
        ga, gb = torch.autograd.grad(out.data, (s["A"].data, s["B"].data), s["cotangent"].data)
        return {"theta": out.data.detach(), "grad_A": ga, "grad_B": gb}
    if kind == "env":
        update = update_left_env if case["side"] == "left" else update_right_env
        return update(s["env"], s["A"], s["W"], case["precision"]).data
    if kind == "heff":
        if "batch" in s:
            s["batch"].apply(s["x"], s["y"])
        else:
            s["ops"][0].apply(s["x"][0], s["y"][0])
        return s["y"]
    if kind == "lanczos":
        energy, vec, _ = lanczos(s["op"], s["theta"], case["steps"], 1e-12)
        return {"energy": float(energy), "vector": vec.data}
    if kind == "ctm":
        env = ctm(s["A"], s["config"], projectors=s["P"])
        energy = compute_energy_ctm(s["A"], env, s["gate"], 2)
        (g,) = torch.autograd.grad(energy, s["A"])
        return {"energy": energy.detach(), "grad": g, "env": [t.detach() for t in env]}
    a, b = (0, 1) if case["adjacent"] else (0, 2)
    return fuse_indices(s["t"], a, b, "xu", IN).data


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _sizes(charges) -> dict:
    return dict(zip(*(x.tolist() for x in np.unique(charges, return_counts=True))))


def _structure(subs_legs):
    """Key -> shape of every charge-conserving block of [(charges, flow), ...]."""
    dims = [_sizes(c) for c, _ in subs_legs]
    keys = [()]
    for d in dims[:-1]:
        keys = [k + (q,) for k in keys for q in d]
    out = {}
    for k in keys:
        last = -int(subs_legs[-1][1]) * sum(int(f) * q for (_, f), q in zip(subs_legs, k))
        if last in dims[-1]:
            k = k + (last,)
            out[k] = tuple(d[q] for d, q in zip(dims, k))
    return out


def _pair_shapes(sa, A, sb, B, so):
    """Output shapes and FLOPs of one pairwise contraction of key -> shape maps."""
    shared = [c for c in sa if c in sb]
    by = {}
    for k, shp in B.items():
        by.setdefault(tuple(k[sb.index(c)] for c in shared), []).append((k, shp))
    out, flops = {}, 0.0
    for ka, xa in A.items():
        for kb, xb in by.get(tuple(ka[sa.index(c)] for c in shared), ()):
            q = {**dict(zip(sa, ka)), **dict(zip(sb, kb))}
            n = {**dict(zip(sa, xa)), **dict(zip(sb, xb))}
            out[tuple(q[c] for c in so)] = tuple(n[c] for c in so)
            flops += 2.0 * math.prod(n.values())
    return out, flops


def _elems(shapes) -> int:
    return sum(math.prod(s) for s in shapes.values())


def _of(t) -> dict:
    return {tuple(k): tuple(s) for k, s in t.block_shapes().items()}


def _heff_work(chi, sectors, mpo):
    wl, wr = _mpo(mpo)
    v = _bond(chi, sectors, 1)
    L = _structure([(v, OUT), (wl.indices[0].charges, IN), (v, IN)])
    th = _structure([(v, IN), (PHYS, IN), (PHYS, IN), (v, OUT)])
    R = _structure([(v, OUT), (wr.indices[3].charges, IN), (v, IN)])
    x, f1 = _pair_shapes("abc", L, "apqd", th, "bcpqd")
    x, f2 = _pair_shapes("bcpqd", x, "bpse", _of(wl), "cseqd")
    x, f3 = _pair_shapes("cseqd", x, "eqtf", _of(wr), "cstfd")
    _, f4 = _pair_shapes("cstfd", x, "dfg", R, "cstg")
    return 8 * (_elems(L) + _elems(R) + 2 * _elems(th)), f1 + f2 + f3 + f4, _elems(th)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("contract", "grad"):
        v0, v1 = _bond(case["chi"], case["sectors"], 1), _bond(case["chi"], case["sectors"], 0)
        A = _structure([(v0, IN), (PHYS, IN), (v1, OUT)])
        B = _structure([(v1, IN), (PHYS, IN), (v0, OUT)])
        C, flops = _pair_shapes("apm", A, "mqb", B, "apqb")
        b = 8 * (_elems(A) + _elems(B) + _elems(C))
        # forward reads A, B, writes C; the gradients read the cotangent too and write two more
        return ({"bytes": b, "flops": flops} if kind == "contract"
                else {"bytes": b + 8 * (_elems(A) + _elems(B) + _elems(C)), "flops": 3 * flops})
    if kind == "env":
        wl, _ = _mpo(case["mpo"])
        vl, vr = _bond(case["chi"], case["sectors"], 1), _bond(case["chi"], case["sectors"], 0)
        A = _structure([(vl, IN), (PHYS, IN), (vr, OUT)])
        if case["side"] == "left":
            E = _structure([(vl, OUT), (wl.indices[0].charges, IN), (vl, IN)])
            x, f1 = _pair_shapes("abc", E, "apd", A, "bcpd")
            x, f2 = _pair_shapes("bcpd", x, "bpxe", _of(wl), "cdxe")
            x, f3 = _pair_shapes("cdxe", x, "cxf", A, "def")
        else:
            E = _structure([(vr, IN), (wl.indices[3].charges, OUT), (vr, OUT)])
            x, f1 = _pair_shapes("abc", E, "dpa", A, "bcdp")
            x, f2 = _pair_shapes("bcdp", x, "epxb", _of(wl), "cdex")
            x, f3 = _pair_shapes("cdex", x, "fxc", A, "def")
        return {"bytes": 8 * (_elems(E) + _elems(A) + _elems(x)), "flops": f1 + f2 + f3}
    if kind in ("heff", "lanczos"):
        total = {"bytes": 0, "flops": 0.0}
        for chi in (int(c) for c in case["chis"].split()):
            b, f, n = _heff_work(chi, case["sectors"], case["mpo"])
            if kind == "lanczos":
                # each step reads the operator and writes one Krylov vector; the Ritz vector reads them all
                m = case["steps"]
                b, f = m * b + 8 * n * (m + 1), m * f + 12.0 * n * m
            total["bytes"] += b
            total["flops"] += f
        return total
    if kind == "ctm":
        D, chi, n = case["D"], case["chi"], case["sweeps"]
        d2 = D * D
        corner = 2.0 * chi * chi * d2 * chi * 2          # grow and project one corner
        edge = 2.0 * (2 * chi ** 3 * d2 ** 2 + chi ** 2 * d2 ** 4)
        moves = 4 * n * (2 * corner + edge)
        rdm = 2 * 2.0 * 2 * (chi ** 3 * d2 ** 2 + chi ** 2 * d2 ** 4 * 4 + chi ** 3 * d2 ** 2 * 4)
        elems = 4 * n * (2 * chi * chi + chi * chi * d2 + chi * d2 * chi)  # environments and projectors
        return {"bytes": 8 * 3 * elems, "flops": 3 * (moves + rdm)}
    D, chi = case["D"], case["chi"]
    d2 = np.add.outer(np.arange(D) - D // 2, -(np.arange(D) - D // 2)).reshape(-1)
    x = np.sort(np.resize(np.arange(-3, 4), chi))
    return {"bytes": 16 * _elems(_structure([(x, IN), (d2, IN), (d2, OUT), (x, OUT)])), "flops": 0}


# ---------------------------------------------------------------------------
# the same results in 64 bits with plain torch
# ---------------------------------------------------------------------------

def _blocks(t) -> dict:
    """Key -> block view of a tensor's flat buffer."""
    counts = [_sizes(i.charges) for i in t.indices]
    out, off = {}, 0
    flat = t.data.detach()
    for k in t.keys:
        shp = tuple(c[q] for c, q in zip(counts, k))
        n = math.prod(shp)
        out[tuple(k)] = flat[off:off + n].view(shp)
        off += n
    return out


def _pair(sa, A, sb, B, so) -> dict:
    shared = [c for c in sa if c in sb]
    by = {}
    for k, x in B.items():
        by.setdefault(tuple(k[sb.index(c)] for c in shared), []).append((k, x))
    out = {}
    for ka, xa in A.items():
        for kb, xb in by.get(tuple(ka[sa.index(c)] for c in shared), ()):
            q = {**dict(zip(sa, ka)), **dict(zip(sb, kb))}
            y = torch.einsum(f"{sa},{sb}->{so}", xa, xb)
            k = tuple(q[c] for c in so)
            out[k] = out[k] + y if k in out else y
    return out


def _flat(blocks: dict, keys=None) -> torch.Tensor:
    return torch.cat([blocks[k].reshape(-1) for k in (sorted(blocks) if keys is None else keys)])


def _heff_exact(L, wl, wr, R, x: dict) -> dict:
    y = _pair("abc", L, "apqd", x, "bcpqd")
    y = _pair("bcpqd", y, "bpse", wl, "cseqd")
    y = _pair("cseqd", y, "eqtf", wr, "cstfd")
    y = _pair("cstfd", y, "dfg", R, "cstg")
    return {k: y[k] if k in y else torch.zeros_like(v) for k, v in x.items()}


def _split(flat, like: dict) -> dict:
    out, off = {}, 0
    for k in sorted(like):
        n = like[k].numel()
        out[k] = flat[off:off + n].view(like[k].shape)
        off += n
    return out


def _lanczos_exact(apply, x0, steps):
    """Three-term recurrence without reorthogonalisation, Ritz pair of the lowest value."""
    v = [x0 / x0.norm()]
    alpha, beta = [], []
    for k in range(steps):
        w = apply(v[k])
        alpha.append(float(v[k] @ w))
        w = w - alpha[-1] * v[k] - (beta[-1] * v[k - 1] if k else 0.0)
        beta.append(float(w.norm()))
        v.append(w / beta[-1])
    T = np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1)
    ev, vecs = np.linalg.eigh(T)
    i = int(np.argmin(ev))
    y = sum(float(vecs[k, i]) * v[k] for k in range(steps))
    return float(ev[i]), y / y.norm()


_MOVES = (  # corner growths, order of the double layer's legs, inputs and outputs of each move
    ("ab,buc->auc", "gh,hdi->gdi", "swxt", (0, 4, 3, 6, 7), (0, 3, 7)),
    ("ce,buc->eub", "im,hdi->mdh", "swtx", (1, 4, 2, 6, 5), (1, 2, 5)),
    ("ab,alg->blg", "ce,erm->crm", "xtsw", (0, 7, 1, 5, 4), (0, 1, 4)),
    ("gh,alg->hla", "im,erm->ire", "txsw", (3, 7, 2, 5, 6), (3, 2, 6)),
)


def _ctm_exact(A, P, chi, sweeps, gate):
    E = torch.einsum
    A = A.detach().clone().requires_grad_(True)
    D = A.shape[0]
    d2 = D * D
    a = E("udlrs,UDLRs->uUdDlLrR", A, A).reshape(d2, d2, d2, d2)
    ao = E("udlrs,UDLRt->uUdDlLrRst", A, A).reshape(d2, d2, d2, d2, 2, 2)
    m = min(chi, d2)
    C = torch.zeros(chi, chi, dtype=A.dtype, device=A.device)
    C[:m, :m] = torch.eye(m, dtype=A.dtype, device=A.device)
    T = torch.zeros(chi, d2, chi, dtype=A.dtype, device=A.device)
    i = torch.arange(m, device=A.device)
    T[i, :, i] = 1.0
    env = [C, C, C, C, T, T, T, T]
    for sweep in range(sweeps):
        for mv, (c1, c2, asub, ins, outs) in enumerate(_MOVES):
            X, Ex, Y, Ey, Ed = (env[k] for k in ins)
            p = P[4 * sweep + mv].view(chi, d2, chi)
            g1, g2 = E(c1, X, Ex), E(c2, Y, Ey)
            u = E("pxq,qwB->pxwB", Ed, p)
            w = E(f"pxwB,{asub}->pBst", u, a)
            for k, t in zip(outs, (E("psA,psq->Aq", p, g1), E("psA,psq->Aq", p, g2), E("psA,pBst->AtB", p, w))):
                env[k] = t
        env = [t / (t.abs().amax() + 1e-15) for t in env]
    C1, C2, C3, C4, T1, T2, T3, T4 = env

    def close(rdm):
        r = rdm.permute(0, 2, 1, 3).reshape(4, 4)
        r = 0.5 * (r + r.T)
        return (r / (torch.trace(r) + 1e-15)).reshape(2, 2, 2, 2)

    x = E("ucxg,udxrst->cgdrst", E("auc,axg->ucxg", E("ab,buc->auc", C1, T1), T4), ao)
    left = E("cgdrst,gdj->crjst", x, E("gi,idj->gdj", C4, T3))
    y = E("curm,udlrtv->cmdltv", E("cuf,frm->curm", E("cuf,fg->cug", T1, C2), T2), ao)
    right = E("cmdltv,jdm->cjltv", y, E("jdk,mk->jdm", T3, C3))
    h = close(E("crjst,cjruv->stuv", left, right))
    top = E("auc,ce->aue", E("ab,buc->auc", C1, T1), C2)
    z = E("uelf,udlrst->efdrst", E("aue,alf->uelf", top, T4), ao)
    up = E("efdrst,erg->dfgst", z, T2)
    bot = E("hqk,ik->hqi", E("hj,jqk->hqk", C4, T3), C3)
    w = E("fmqi,pqmnwx->fipnwx", E("fmh,hqi->fmqi", T4, bot), ao)
    down = E("fipnwx,gni->fgpwx", w, T2)
    v = close(E("dfgst,fgdwx->stwx", up, down))
    energy = (h * gate).sum() + (v * gate).sum()
    (g,) = torch.autograd.grad(energy, A)
    return {"energy": energy.detach(), "grad": g, "env": [t.detach() for t in env]}


def _fuse_exact(t, a: int, b: int) -> torch.Tensor:
    """Fused sectors: the (q_a, q_b) pairs of one fused charge stacked in sorted order."""
    qa, qb = _sizes(t.indices[a].charges), _sizes(t.indices[b].charges)
    fa, fb = int(t.indices[a].flow), int(t.indices[b].flow)
    pairs: dict = {}
    for x in sorted(qa):
        for y in sorted(qb):
            pairs.setdefault(fa * x + fb * y, []).append((x, y))
    parts: dict = {}
    for k, blk in _blocks(t).items():
        rest = tuple(q for i, q in enumerate(k) if i not in (a, b))
        q = fa * k[a] + fb * k[b]
        order = [a] + [b] + [i for i in range(blk.ndim) if i not in (a, b)]
        y = blk.permute(order).reshape(blk.shape[a] * blk.shape[b], *(blk.shape[i] for i in order[2:]))
        parts.setdefault((rest, q), {})[(k[a], k[b])] = y
    out = {}
    for (rest, q), by in parts.items():
        shape = next(iter(by.values())).shape[1:]
        rows = [by[p] if p in by else torch.zeros(qa[p[0]] * qb[p[1]], *shape, dtype=torch.float64, device="cuda")
                for p in pairs[q]]
        f = torch.cat(rows)
        # the fused leg goes where the first of the two was
        perm = list(range(1, a + 1)) + [0] + list(range(a + 1, f.ndim))
        out[rest[:a] + (q,) + rest[a:]] = f.permute(perm)
    return _flat(out)


def exact(case: dict, seed: int):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("contract", "grad"):
        A, B = _blocks(s["A"]), _blocks(s["B"])
        C = _pair("apm", A, "mqb", B, "apqb")
        if kind == "contract":
            return _flat(C)
        G = _blocks(s["cotangent"])
        ga, gb = _pair("apqb", G, "mqb", B, "apm"), _pair("apm", A, "apqb", G, "mqb")
        return {"theta": _flat(C), "grad_A": _flat(ga, sorted(A)), "grad_B": _flat(gb, sorted(B))}
    if kind == "env":
        E, A, W = _blocks(s["env"]), _blocks(s["A"]), _blocks(s["W"])
        if case["side"] == "left":
            x = _pair("bcpd", _pair("abc", E, "apd", A, "bcpd"), "bpxe", W, "cdxe")
            return _flat(_pair("cdxe", x, "cxf", A, "def"))
        x = _pair("bcdp", _pair("abc", E, "dpa", A, "bcdp"), "epxb", W, "cdex")
        return _flat(_pair("cdex", x, "fxc", A, "def"))
    if kind in ("heff", "lanczos"):
        ys = []
        for L, wl, wr, R, th in s["problems"]:
            L, wl, wr, R, x = (_blocks(t) for t in (L, wl, wr, R, th))
            if kind == "lanczos":
                e, y = _lanczos_exact(lambda v: _flat(_heff_exact(L, wl, wr, R, _split(v, x))), _flat(x),
                                      case["steps"])
                return {"energy": e, "vector": y}
            ys.append(_flat(_heff_exact(L, wl, wr, R, x)))
        return ys
    if kind == "ctm":
        return _ctm_exact(s["A"], s["P"], case["chi"], case["sweeps"], heisenberg_gate())
    return _fuse_exact(s["t"], *((0, 1) if case["adjacent"] else (0, 2)))
