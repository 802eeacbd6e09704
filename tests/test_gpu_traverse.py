"""Candidate search: the warp-per-probe walk (few probes) and the thread walk (many) give every pair of meeting boxes once."""
import numpy as np
import pytest

import pyoracle as O
from shapes import S, make_set, square

pytestmark = pytest.mark.gpu


def boxes(n, seed, side, size):
    r = np.random.default_rng(seed)
    return make_set([[square(x, y, s)] for x, y, s in zip(r.uniform(0, side, n), r.uniform(0, side, n), r.uniform(0.2 * size, size, n))])


def nested(n, side, f):
    """Small boxes at distances side * f^k from a corner: the tree is a chain, then ids alone tell its leaves apart."""
    k = np.arange(n)
    return make_set([[square(side * f ** i, side * f ** i, 0.1 * side * f ** i + 1e-12)] for i in k])


CASES = {
    "chain": (boxes(5, 11, 400 * S, 400 * S), nested(3000, 400 * S, 0.97)),
    "chain_2": (boxes(5, 11, 400 * S, 400 * S), nested(64, 400 * S, 0.5)),
    "one_leaf": (boxes(5, 1, S, S), make_set([[square(0, 0, S)]])),
    "one_probe": (make_set([[square(0, 0, 100 * S)]]), boxes(9000, 2, 100 * S, S)),      # the probe meets every leaf
    "same_boxes": (boxes(3, 3, S, S), make_set([[square(0, 0, S)]] * 3000)),             # leaves told apart by their ids alone
    "warps_5": (boxes(5, 4, 50 * S, 20 * S), boxes(9000, 5, 50 * S, S)),
    "line_8192": (boxes(8192, 6, 50 * S, S), boxes(300, 7, 50 * S, S)),
    "line_8193": (boxes(8193, 6, 50 * S, S), boxes(300, 7, 50 * S, S)),
    "line_24576": (boxes(24576, 8, 200 * S, S), boxes(8192, 9, 200 * S, S)),
    "line_24577": (boxes(24577, 8, 200 * S, S), boxes(8192, 9, 200 * S, S)),
    "apart": (boxes(10, 10, S, S), make_set([[square(50 * S, 0, S)], [square(60 * S, 0, S)]])),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("upper", [False, True])
def test_candidates(engine, name, upper):
    A, B = CASES[name]
    want = O.candidates(O.OSet(A), O.OSet(B), upper=upper)
    got = engine.candidates(engine.upload_polygons(A), engine.upload_polygons(B), upper=upper)
    key = lambda p: np.sort(p[:, 0].astype(np.int64) << 32 | p[:, 1])
    assert np.array_equal(key(got), key(np.asarray(want)))
