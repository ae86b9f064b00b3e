"""Block layouts counted once per leg, and the conservation check of all blocks at once."""

import copy
import itertools
import math
import pickle

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from tenax_b200.core import (FermionicU1, FermionParity, FlowDirection, TensorIndex, U1Symmetry,  # noqa: E402
                             ZnSymmetry)
from tenax_b200.tensor import SymmetricTensor, block_shape, make_layout  # noqa: E402
from tenax_b200.tensor_utils import fuse_indices  # noqa: E402

SYMS = [U1Symmetry(), ZnSymmetry(2), ZnSymmetry(3), FermionParity(), FermionicU1()]


def _legs(sym, n):
    rng = np.random.default_rng(n)
    hi = sym.n_values() or 3
    return tuple(TensorIndex(sym, rng.integers(0, hi, 3 + 2 * i).astype(np.int32),
                             FlowDirection.IN if i % 2 else FlowDirection.OUT, f"l{i}") for i in range(n))


@pytest.mark.parametrize("sym", SYMS, ids=repr)
@pytest.mark.parametrize("n", [0, 1, 2, 4])
def test_layout_matches_block_shapes(sym, n):
    idx = _legs(sym, n)
    keys = list(itertools.product(range(-1, 3), repeat=n))  # charges that no state carries among them
    lay = make_layout(idx, keys)
    assert lay.shapes == [block_shape(idx, k) for k in keys]
    assert lay.offsets.tolist() == np.concatenate([[0], np.cumsum([math.prod(s) for s in lay.shapes])]).tolist()
    assert [lay.key_pos[k] for k in keys] == list(range(len(keys)))


@pytest.mark.parametrize("sym", SYMS, ids=repr)
@pytest.mark.parametrize("n", [1, 2, 3])
def test_validate_agrees_with_fuse_many(sym, n):
    idx = _legs(sym, n)
    for key in itertools.product(range(3), repeat=n):
        t = SymmetricTensor.from_flat(idx, [key], torch.zeros(math.prod(block_shape(idx, key)), dtype=torch.float64))
        fused = sym.fuse_many([int(i.flow) * q for i, q in zip(idx, key)])
        if fused == sym.identity():
            t._validate()
        else:
            with pytest.raises(ValueError, match="charge conservation"):
                t._validate()


def test_pickles_with_and_without_a_layout():
    idx = _legs(U1Symmetry(), 2)
    keys = [(q, q) for q in range(3) if math.prod(block_shape(idx, (q, q)))]
    n = sum(math.prod(block_shape(idx, k)) for k in keys)
    t = SymmetricTensor.from_flat(idx, keys, torch.arange(n, dtype=torch.float64))
    state = {s: getattr(t, s) for s in SymmetricTensor.__slots__ if s != "_layout"}
    old = object.__new__(SymmetricTensor)
    old.__setstate__((None, state))  # as a tensor written before layouts were kept comes back
    for u in (pickle.loads(pickle.dumps(t)), copy.deepcopy(t), old):
        assert u._layout.keys == tuple(keys) and u._layout.shapes == t._layout.shapes
        assert u._layout.offsets.tolist() == t._layout.offsets.tolist() and u._layout.key_pos == t._layout.key_pos
        assert torch.equal(u.data if hasattr(u, "data") else u._data, t._data)


def test_validate_reads_only_the_charges_a_leg_has():
    idx = _legs(U1Symmetry(), 2)
    t = SymmetricTensor.from_flat(idx, [(0, 0)], torch.zeros(math.prod(block_shape(idx, (0, 0))), dtype=torch.float64))
    t._keys = [(0, 0, 5), (1, 1, 7)]
    t._validate()


class _Annotated(SymmetricTensor):
    """A subclass with attributes of its own (no slots)."""


def test_pickles_of_a_subclass_keep_its_attributes():
    idx = _legs(U1Symmetry(), 2)
    n = math.prod(block_shape(idx, (0, 0)))
    t = _Annotated.from_flat(idx, [(0, 0)], torch.arange(n, dtype=torch.float64))
    t.note = "left"
    for u in (pickle.loads(pickle.dumps(t)), copy.deepcopy(t), copy.copy(t)):
        assert type(u) is _Annotated and u.note == "left" and u._keys == [(0, 0)] and torch.equal(u._data, t._data)


def test_fusing_a_tensor_on_the_host_is_a_value_error():
    idx = _legs(U1Symmetry(), 2)
    t = SymmetricTensor.from_flat(idx, [(0, 0)], torch.zeros(math.prod(block_shape(idx, (0, 0))), dtype=torch.float64))
    with pytest.raises(ValueError, match="cuda device"):
        fuse_indices(t, 0, 1, "f", FlowDirection.IN)
