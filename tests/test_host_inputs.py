"""Edges and weights as they come: what is no whole number is refused as before
the arguments were read in fewer passes, and the result is the caller's own."""
import numpy as np
import pytest

from forceatlas2_rc_gb300.layout import _edges, edge_weights


@pytest.mark.parametrize("edges,error", [
    ([[0j, 1]], TypeError),
    ([[1 + 2j, 1]], TypeError),
    ([[float("nan"), 1]], ValueError),
    ([[float("inf"), 1]], OverflowError),
    ([[None, 1]], TypeError),
    ([["a", 1]], ValueError),
])
def test_edges_that_are_no_numbers_are_refused(edges, error):
    with pytest.raises(error):
        _edges(3, edges)


@pytest.mark.parametrize("edges", [
    [[0, 1], [1, 2]], [[0.0, 1.9], [1.0, 2.0]], [["0", "1"], ["1", "2"]],
    np.array([[0, 1], [1, 2]], np.uint8), np.array([[0, 1], [1, 2]], np.uint64),
    np.array([[0, 1], [1, 2]], np.float32), np.array([[0, 1], [1, 2]], object),
    np.asfortranarray(np.array([[0, 1], [1, 2]], np.int32)),
])
def test_edges_of_every_kind(edges):
    frm, to = _edges(3, edges)
    assert frm.dtype == to.dtype == np.int32
    assert frm.tolist() == [0, 1] and to.tolist() == [1, 2]


def test_weights_are_not_the_argument():
    w = np.array([1.0, 2.0, 3.0])
    out = edge_weights(3, w)
    assert not np.shares_memory(out, w)
    assert out.tolist() == [1.0, 2.0, 3.0]


@pytest.mark.parametrize("influence", ["a", None])
def test_bad_influence_is_refused_without_weights(influence):
    with pytest.raises(TypeError):
        edge_weights(3, None, edge_weight_influence=influence)
    with pytest.raises(TypeError):
        edge_weights(3, np.ones(3), edge_weight_influence=influence)
