"""The bins of the refinement at the sizes where they hand pairs on (a warp's bin, a block's, global scratch): an edge cut
more often than its split list holds, more cuts than there is room for, edge lists around the bins' sizes, an
overlap box of no height, tolerances of zero. Every variant has to give the oracle's rows bit for bit."""
import ctypes

import numpy as np
import pytest

import gsj
import pyoracle as O
from shapes import S, cw, make_set, square

pytestmark = pytest.mark.gpu
MODES = [gsj.GSJ_REFINE_PLAIN, gsj.GSJ_REFINE_FILTERED, gsj.GSJ_REFINE_FILTERED_FP32]


def comb(teeth, w, h, x0=0.0, y0=0.0, flip=False):
    """A comb of upright teeth on a bar: 4 teeth + 3 edges; flip: lying on its side."""
    pts = [(x0, y0), (x0 + w, y0)]
    for t in reversed(range(teeth)):
        a, b = x0 + w * (t + 0.25) / teeth, x0 + w * (t + 0.75) / teeth
        pts += [(b, y0 + 0.1 * h), (b, y0 + h), (a, y0 + h), (a, y0 + 0.1 * h)]
    pts += [(x0, y0 + 0.1 * h), (x0, y0)]
    return [(y, x) for x, y in reversed(pts)] if flip else pts


def ngon(n, r, cx=0.0, cy=0.0):
    a = 2 * np.pi * np.arange(n) / n
    p = [(cx + r * np.cos(t), cy + r * np.sin(t)) for t in a]
    return p + p[:1]


def fine(n):
    """A square whose lower side is divided into n edges."""
    return [(S * k / n, 0.0) for k in range(n)] + [(S, 0.0), (S, S), (0.0, S), (0.0, 0.0)]


SHAPES = {
    # a bar across every tooth: 2 x teeth splits on its long edges (an edge keeps 22 beside its ends)
    **{f"bar_{n}": ([[comb(n, 40 * S, 4 * S)]], [[[(-S, 2 * S), (41 * S, 2 * S), (41 * S, 2.5 * S), (-S, 2.5 * S), (-S, 2 * S)]]]) for n in (10, 11, 12, 28, 100, 200)},
    # crossed combs: more split points than the lists hold
    "combs_9": ([[comb(9, 10 * S, 10 * S)]], [[comb(9, 10 * S, 10 * S, flip=True)]]),
    "combs_28": ([[comb(28, 10 * S, 10 * S)]], [[comb(28, 10 * S, 10 * S, flip=True)]]),
    "combs_60": ([[comb(60, 10 * S, 10 * S)]], [[comb(60, 10 * S, 10 * S, flip=True)]]),
    # a whole side against one divided into n: coincident edges beyond the 8 that an edge keeps, and 2 (n - 1) splits
    **{f"fine_{n}": ([[fine(n)]], [[square(0, -S, S)], [square(0, -0.5 * S, S)]]) for n in (7, 8, 9, 11, 12, 13, 40, 120, 300, 700)},
    # more cuts than the block bins' lists hold
    "combs_130": ([[comb(130, 10 * S, 10 * S)]], [[comb(130, 10 * S, 10 * S, flip=True)]]),
    # holes and several parts, more than 1024 edges in all: global scratch
    "parts_1200": ([[ngon(600, S), cw(ngon(300, 0.3 * S, 0.4 * S)), cw(ngon(300, 0.3 * S, -0.4 * S, 0.1 * S)), ngon(60, 0.1 * S, 0.4 * S)]],
                   [[ngon(600, S, 0.3 * S, 0.2 * S), cw(ngon(500, 0.5 * S, 0.3 * S, 0.2 * S))], [ngon(700, 0.4 * S, 0.1 * S), ngon(400, 0.2 * S, S)]]),
    # level neighbours: the overlap box is as thin as its pad
    "touch": ([[square(0, 0, S)]], [[square(0, S, S)], [square(S, S, S)]]),
    "twins": ([[square(0, 0, S)], [comb(9, S, S)]], [[square(0, 0, S)], [comb(9, S, S)]]),
}
for _n in (31, 32, 33, 64, 96, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025):
    SHAPES[f"ngon_{_n}"] = ([[ngon(_n, S)]], [[ngon(_n, S, 0.3 * S, 0.2 * S)], [ngon(7, 0.2 * S)]])


def rows(r):
    i = np.lexsort((r.pairs[:, 1], r.pairs[:, 0]))
    return r.pairs[i], None if r.area is None else r.area[i], None if r.code is None else r.code[i]


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("area,relate", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_handed_on_pairs(engine, name, area, relate):
    A, B = (make_set(g) for g in SHAPES[name])
    both = make_set([*SHAPES[name][0], *SHAPES[name][1]])
    for P, R, up in ((A, B, False), (B, A, False), (both, both, True)):
        p, oa, oc, _ = O.join(O.OSet(P), O.OSet(R), O.params(area, relate), upper=up)
        lp = engine.upload_polygons(P)
        lr = lp if R is P else engine.upload_polygons(R)
        for m in MODES:
            gp, ga, gc = rows(engine.join(lp, lr, want_area=bool(area), want_relate=bool(relate), upper=up, refine_mode=m))
            assert np.array_equal(gp, p)
            assert not area or np.array_equal(ga, oa)
            assert not relate or np.array_equal(gc, oc)


@pytest.mark.parametrize("name", [k for k in sorted(SHAPES) if k[:4] in ("bar_", "fine") and int(k.split("_")[1]) < 29])
@pytest.mark.parametrize("area,relate", [(1, 0), (0, 1), (1, 1)])
def test_many_cuts_stay(engine, name, area, relate):
    """However often an edge is cut: pairs whose lists fit are not handed to the bins for larger ones."""
    lp, lr = (engine.upload_polygons(make_set(g)) for g in SHAPES[name])
    for a, b in ((lp, lr), (lr, lp)):
        for m in MODES[1:]:
            assert engine.join(a, b, want_area=bool(area), want_relate=bool(relate), refine_mode=m).stats["heavy"] == 0


@pytest.mark.parametrize("area,relate", [(1, 0), (0, 1), (1, 1)])
def test_large_pieces(engine, area, relate):
    """Pieces of more than 1024 edges with cut edges among them: global scratch, folded."""
    def wavy(n, cx):
        t = 2 * np.pi * np.arange(n) / n
        r = S * (1 + 0.05 * np.sin(40 * t))
        return [*zip(cx + r * np.cos(t), r * np.sin(t)), (cx + r[0], 0.0)]

    P, R = (engine.subdivide(make_set([[wavy(6000, x + dx)] for x in (0.0, 1.7 * S)]), 2400) for dx in (0.0, 0.4 * S))
    assert np.diff(P.rvo.astype(np.int64)).max() > 1025 and P.n > 2 and P.syn.any()
    for m in MODES:
        for A, B, up in ((P, R, False), (P, P, True)):
            la = engine.upload_polygons(A)
            lb = la if B is A else engine.upload_polygons(B)
            r = engine.join(la, lb, want_area=bool(area), want_relate=bool(relate), upper=up, refine_mode=m)
            gp, ga, gc = rows(r)
            p, oa, oc, _ = O.join(O.OSet(A), O.OSet(B), O.params(area, relate), upper=up)
            assert r.stats["heavy"] > 0 and np.array_equal(gp, p)
            assert not area or np.array_equal(ga, oa)
            assert not relate or np.array_equal(gc, oc)


@pytest.mark.parametrize("tol", [0.0, 1e-11, 1e-7])
def test_own_tolerances(engine, tol):
    """Tolerances of zero turn the shared inside tests off, wide ones make whole edges candidates: as the plain kernels."""
    from gsj import gen
    P, R = gen.layer_parcels(1500, (-118.30, 33.95, -118.25, 34.00), seed=5), gen.layer_parcels(900, (-118.30, 33.95, -118.25, 34.00), seed=6)
    lp, lr = engine.upload_polygons(P), engine.upload_polygons(R)
    for a, b in ((lp, lr), (lp, lp)):
        pairs = np.ascontiguousarray(engine.candidates(a, b))
        got = []
        for m in MODES:
            n = len(pairs)
            out = [np.zeros(n, np.uint8), np.zeros(n), np.zeros((n, 4)), np.zeros(n, np.uint32)]
            rp = gsj.refine_params(True, True)
            rp.tol_abs, rp.tol_rel = tol, 0.0
            engine._check(gsj.lib().gsj_refine_pairs(engine.ctx, a.h, b.h, pairs.ctypes.data, n, ctypes.byref(rp), m, *[x.ctypes.data for x in out]))
            got.append(out)
        for out in got[1:]:
            assert all(np.array_equal(x, y) for x, y in zip(got[0], out))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 1023, 1024, 1025, 4097])
def test_every_row_arrives(engine, n):
    """Rows are appended 1024 candidates a block: n squares apart give n rows, whatever the count."""
    side = int(np.ceil(np.sqrt(n)))
    g = make_set([[square(3 * S * (k % side), 3 * S * (k // side), S)] for k in range(n)])
    la = engine.upload_polygons(g)
    lp = engine.upload_points(g.xy[g.rvo[:-1].astype(np.int64)] + 0.5 * S)
    same = np.repeat(np.arange(n, dtype=np.uint32)[:, None], 2, axis=1)
    p, area, code = rows(engine.join(la, la, want_area=True, want_relate=True, upper=True))
    assert np.array_equal(p, same) and np.allclose(area, S * S, rtol=1e-9) and (code == code[0]).all()
    pp, where, _ = engine.join_points(lp, la)
    assert np.array_equal(pp, same) and (where == 1).all()
    assert np.array_equal(engine.dwithin(la, la, 5.0, same=True)[0], same)
    assert np.array_equal(engine.points_dwithin(lp, la, 5.0)[0], same)
    assert np.array_equal(engine.erode(la, la, 1.0, 1.0, same=True)[0], same)
    assert np.array_equal(engine.cluster(la)[0], np.arange(n, dtype=np.uint32))


def de9im(ev, bits, la, lb):
    """DE-9IM codes from boundary evidence (lengths of A inside / on B, of B inside / on A) and the whole lengths."""
    a_in, a_out = ev[:, 0] > 1e-9 * la, la - ev[:, 0] - ev[:, 1] > 1e-9 * la
    b_in, b_out = ev[:, 2] > 1e-9 * lb, lb - ev[:, 2] - ev[:, 3] > 1e-9 * lb
    same, opp, touch = (bits & 1) != 0, (bits & 2) != 0, (bits & 4) != 0
    cells = [3 * (a_in | b_in | same), 2 * b_in, 3 * (a_out | b_in | opp),
             2 * a_in, np.where(same | opp, 2, touch), 2 * a_out,
             3 * (b_out | a_in | opp), 2 * b_out, 3]
    return sum(np.asarray(c, np.uint32) << (2 * k) for k, c in enumerate(cells))


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("maxv,differ", [(12, 4), (64, 92)])
def test_unfolded_pieces_relate(engine, maxv, differ, mode):
    """no_agg on subdivided layers: piece pairs, whose boundary lengths are their parents' (kept per parent, not per piece)."""
    from gsj import gen
    P = engine.subdivide(gen.layer_parcels(300, (-118.30, 33.95, -118.29, 33.96), seed=5), maxv)
    lp, op = engine.upload_polygons(P), O.OSet(P)
    p, _, code = rows(engine.join(lp, lp, want_area=False, want_relate=True, no_agg=True, refine_mode=mode))
    cand = O.candidates(op, op)
    flag, _, ev, bits = O.refine_pairs(op, op, cand, O.params(0, 1))
    i = np.lexsort((cand[:, 1], cand[:, 0]))
    i = i[flag[i] == 1]
    ev, bits = ev[i], bits[i]
    assert P.n > P.parent.max() + 1 and np.array_equal(p, cand[i])
    # boundary lengths: the real edges of all pieces of a parent
    d = np.hypot(*np.diff(P.xy, axis=0).T) * (P.syn[:-1] == 0)
    d[P.rvo[1:-1].astype(np.int64) - 1] = 0   # from one ring's end to the next one's start: no edge
    v0 = P.rvo[P.gro.astype(np.int64)].astype(np.int64)
    length = np.bincount(P.parent, [d[a:b - 1].sum() for a, b in zip(v0, v0[1:])])
    assert np.array_equal(code, de9im(ev, bits, length[P.parent[p[:, 0]]], length[P.parent[p[:, 1]]]))
    # ... which lengths taken by piece would not give
    by_piece = np.resize(length, P.n)
    assert (code != de9im(ev, bits, by_piece[p[:, 0]], by_piece[p[:, 1]])).sum() == differ
