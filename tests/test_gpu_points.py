"""Distance and point kernels at the sizes where their lane groups and marks end: rings around multiples of 8, 32 and 256 edges, points on
vertices, on edges and at the search distance give or take its band. Every variant gives the oracle's rows."""
import numpy as np
import pytest

import gsj
import pyoracle as O
from shapes import S, X0, Y0, cw, make_set, square
from test_gpu_bins import comb, ngon

pytestmark = pytest.mark.gpu
MODES = [gsj.GSJ_REFINE_PLAIN, gsj.GSJ_REFINE_FILTERED, gsj.GSJ_REFINE_FILTERED_FP32]
SIZES = [3, 7, 8, 9, 31, 32, 33, 64, 255, 256, 257, 300]
D = 5.0


def layer():
    """A polygon of each size, every other one with a hole, and points around them."""
    geoms, pts = [], []
    rng = np.random.default_rng(3)
    for k, n in enumerate(SIZES):
        cx, cy, r = 4 * S * k, 0.0, S
        ring = ngon(n, r, cx, cy)
        geoms.append([ring, cw(ngon(5, 0.3 * r, cx, cy))] if k % 2 else [ring])
        ring = np.array(ring)
        a, b = ring[:-1], ring[1:]
        out = (0.5 * (a + b) - [cx, cy])
        out /= np.linalg.norm(out, axis=1, keepdims=True)
        at = D / 111000.0
        pts += [a, 0.5 * (a + b), 0.25 * a + 0.75 * b, np.column_stack([rng.uniform(cx - 1.5 * r, cx + 1.5 * r, 200), np.repeat(a[:1, 1], 200)])]
        pts += [0.5 * (a + b) + out * at * f for f in (0.5, 0.99, 0.9999, 1.0, 1.0001, 1.003, 1.01, 1.2)]
        pts += [rng.uniform([cx - 2 * r, -2 * r], [cx + 2 * r, 2 * r], (200, 2))]
    return make_set(geoms), np.concatenate(pts) + [X0, Y0]


@pytest.fixture(scope="module")
def both(engine):
    g, p = layer()
    return g, p, engine.upload_polygons(g), engine.upload_points(p)


@pytest.mark.parametrize("mode", MODES)
def test_points_in_polygons(engine, both, mode):
    g, p, lg, lp = both
    op, ow, _ = O.pip(p, O.OSet(g))
    gp, gw, _ = engine.join_points(lp, lg, refine_mode=mode)
    assert np.array_equal(gp, op) and np.array_equal(gw, ow)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("d", [0.5, D, 2 * D])
def test_points_within(engine, both, mode, d):
    g, p, lg, lp = both
    assert np.array_equal(engine.points_dwithin(lp, lg, d, refine_mode=mode)[0], O.pt_dwithin(p, O.OSet(g), d))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("d", [0.5, D, 2 * D])
def test_polygons_within(engine, mode, d):
    """Polygons of 3 to 129 edges (the lists hold 128) side by side at gaps around d, one inside another, and apart."""
    sizes = [3, 31, 32, 33, 64, 127, 128, 129]
    m = 1.0 / (111320.0 * np.cos(np.radians(Y0)))   # about a metre of longitude
    A, B = [], []
    for k, n in enumerate(sizes):
        for q, f in enumerate((0.5, 0.99, 0.9999, 1.0001, 1.01, 1.5)):
            cx, cy = 8 * S * k, 4 * S * q
            A.append([ngon(n, S, cx, cy)])
            B.append([ngon(sizes[(k + q) % len(sizes)], S, cx + 2 * S + f * d * m, cy)])
        A.append([ngon(n, 0.2 * S, 8 * S * k, -4 * S)])
        B.append([ngon(9, S, 8 * S * k, -4 * S)])
    a, b = make_set(A), make_set(B)
    la, lb = engine.upload_polygons(a), engine.upload_polygons(b)
    for lr, rs, same in ((lb, b, False), (la, a, True)):
        got, want = engine.dwithin(la, lr, d, same=same, refine_mode=mode)[0], O.dwithin(O.OSet(a), O.OSet(rs), d, same=same)[0]
        assert set(map(tuple, got.tolist())) == set(map(tuple, want.tolist()))


def fine_square(n, x0, y0, w, h):
    """A rectangle of n edges, its sides divided evenly."""
    c = [(x0, y0), (x0 + w, y0), (x0 + w, y0 + h), (x0, y0 + h), (x0, y0)]
    pts = []
    for k in range(4):
        m = n // 4 + (k < n % 4)
        pts += [(c[k][0] + (c[k + 1][0] - c[k][0]) * t / m, c[k][1] + (c[k + 1][1] - c[k][1]) * t / m) for t in range(m)]
    return pts + pts[:1]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,m", [(7, 128), (128, 128), (128, 129), (129, 7), (255, 255), (255, 256), (256, 256), (256, 257), (257, 5), (5, 257), (300, 600)])
def test_polygons_within_lists(engine, n, m, mode):
    """Lists around the sizes of the two forms (128 and 256 edges a side): a polygon of n edges in a hole of m, all of them
    within reach up to the distance, gaps from half of it to just in and out of the band around it."""
    w = np.sqrt(1 - 0.0066943799901413165 * np.sin(np.radians(Y0)) ** 2)
    mx, my = 1.0 / (np.radians(6378137.0) / w * np.cos(np.radians(Y0))), 1.0 / (np.radians(6378137.0) * (1 - 0.0066943799901413165) / w ** 3)   # a metre
    F = [0.5, 0.9, 0.999] + [1 + k * 2e-5 for k in range(-6, 7)] + [1.001]
    A, B = [], []
    for k, f in enumerate(F):
        x, y, g, h = 8 * S * k, 0.0, f * D * mx, f * D * my
        A.append([fine_square(n, x, y, S, S)])
        B.append([square(x - S, y - S, 3 * S), cw(fine_square(m, x - g, y - h, S + 2 * g, S + 2 * h))])
    a, b = make_set(A), make_set(B)
    pairs, st = engine.dwithin(engine.upload_polygons(a), engine.upload_polygons(b), D, refine_mode=mode)
    want = O.dwithin(O.OSet(a), O.OSet(b), D)[0]
    assert set(map(tuple, pairs.tolist())) == set(map(tuple, want.tolist()))
    assert 3 < len(want) < len(F)
    if mode != gsj.GSJ_REFINE_PLAIN:   # to the kernel with the geodesic: pairs in the band, or all whose lists are too long
        assert st["heavy"] >= sum(f < 1 for f in F) if max(n, m) > 256 else 0 < st["heavy"] < 13


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("r", [1.0, 4.0, 20.0])
def test_eroded(engine, mode, r):
    """Eroded polygons of 3 to 130 edges (the lists hold 64 edges and 128 elements), convex and with reflex corners,
    each with itself and with shifted copies whose eroded forms just meet or just do not."""
    sizes = [3, 31, 32, 33, 63, 64, 65, 130]
    m = 1.0 / (111320.0 * np.cos(np.radians(Y0)))
    A, B = [], []
    for k, n in enumerate(sizes):
        for q, f in enumerate((0.0, 0.3, 1.9, 1.99, 2.01, 2.1)):
            cx, cy = 8 * S * k, 4 * S * q
            A.append([ngon(n, S, cx, cy)])
            B.append([ngon(n, S, cx + 2 * S - f * r * m if f else cx, cy)])
        A.append([comb(max(2, n // 5), 2 * S, 2 * S, 8 * S * k, -4 * S)])
        B.append([comb(max(2, n // 5), 2 * S, 2 * S, 8 * S * k + 0.1 * S, -4 * S - 0.2 * S)])
    a, b = make_set(A), make_set(B)
    la, lb = engine.upload_polygons(a), engine.upload_polygons(b)
    for lr, rs, same in ((lb, b, False), (la, a, True)):
        got, want = engine.erode(la, lr, r, r, same=same, refine_mode=mode)[0], O.erode(O.OSet(a), O.OSet(rs), r, r, same=same)
        want = want[0] if isinstance(want, tuple) else want
        assert set(map(tuple, got.tolist())) == set(map(tuple, want.tolist()))
