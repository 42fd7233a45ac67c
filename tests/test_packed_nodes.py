"""The C structure that a dispatch keeps on its node."""
import copy
import pickle
from types import SimpleNamespace

import numpy as np
import pytest

from oxionnx_b200 import _ffi
from oxionnx_b200.graph import Node

FIELDS = {"op": "Conv", "name": "c", "inputs": ["x", "w"], "outputs": ["y"], "attrs": {"pads": [1, 1, 1, 1], "alpha": 1.5}}


@pytest.mark.parametrize("kind", [Node, SimpleNamespace])
@pytest.mark.parametrize("duplicate", [copy.copy, copy.deepcopy, lambda n: pickle.loads(pickle.dumps(n))])
def test_a_dispatched_node_can_be_copied_and_pickled(kind, duplicate):
    node = kind(**copy.deepcopy(FIELDS))
    _ffi.packed_node(node)
    twin = duplicate(node)
    assert twin == node and twin == kind(**FIELDS)
    _, cnode, _ = _ffi.packed_node(twin)
    assert cnode.op_type == b"Conv" and cnode.n_inputs == 2 and cnode.n_attrs == 2


@pytest.mark.parametrize("before,after,kind", [(2, 2.0, 1), (2.0, 2, 0), ([2, 2], [2, 2.0], 4), ([2.0, 2.0], (2, 2), 3)])
def test_the_kept_structure_follows_an_attribute_type(before, after, kind):
    node = Node("Gemm", "g", ["a", "b"], ["y"], {"alpha": before})
    _ffi.packed_node(node)
    node.attrs["alpha"] = after
    assert _ffi.packed_node(node)[1].attrs[0].kind == kind


def test_an_array_attribute_is_packed_anew():
    node = Node("Conv", "c", ["x", "w"], ["y"], {"pads": np.array([1, 1, 1, 1])})
    _ffi.packed_node(node)
    node.attrs["pads"][0] = 2
    assert _ffi.packed_node(node)[1].attrs[0].ints[0] == 2


def test_the_kept_structure_follows_the_fields():
    node = Node(**copy.deepcopy(FIELDS))
    first = _ffi.packed_node(node)
    assert _ffi.packed_node(node) is first
    node.attrs["pads"][0] = 2
    cnode = _ffi.packed_node(node)[1]
    assert cnode.attrs[0].ints[0] == 2


def test_empty_and_absent_attributes():
    for attrs in ({"axes": []}, {}, None):
        node = Node("Pad", "p", ["x"], ["y"], attrs)
        assert _ffi.packed_node(node)[1].n_attrs == len(attrs or {})
        assert _ffi.packed_node(node) is _ffi.packed_node(node)
