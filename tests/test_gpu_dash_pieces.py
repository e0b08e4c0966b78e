"""Dashed pieces as they leave the lanes: contours that end at every place of a full set of lanes (32
points: lines of 2, quadratics of 3, cubics of 4), and pieces that are not pushed (a segment whose length
overflows splits into points that are not finite), against the oracle's outline bit for bit (a NaN's sign
and payload, which differ between processors, aside)."""
import numpy as np
import pytest

import scenes as S
from conftest import OUTLINE_KEYS

pytestmark = pytest.mark.gpu


def paths(contours, kinds, pattern):
    """One path per entry of contours: a list of segment counts, one per contour, or -k for k segments
    whose second to last point is far away."""
    pts, flags, starts, first = [], [], [0], [0]
    for p, counts in enumerate(contours):
        for c, n in enumerate(counts):
            f = [0]
            for i in range(abs(n)):
                f += [[0], [1, 0], [1, 2, 0]][kinds[i % len(kinds)] - 1]
            q = S.Rng(100 * p + c, 25).uniform(2 * len(f)).reshape(-1, 2) * 40.0 + 20.0
            if n < 0:
                q[-2] = (3e38, -3e38)
                q[-1] = (-3e38, 3e38)
            pts.append(q.astype(np.float32))
            flags += f
            starts.append(starts[-1] + len(f))
        first.append(first[-1] + len(counts))
    n = len(contours)
    st = np.zeros(n, S.STROKE_DTYPE)
    st["line_width"], st["miter_limit"], st["dash_count"] = 1.0, 4.0, len(pattern)
    sc = S.Scene(points=np.concatenate(pts), flags=np.asarray(flags, np.uint8), contour_start=np.asarray(starts, np.uint32),
                 path_start=np.asarray(first, np.uint32), fill_rule=np.zeros(n, np.uint8),
                 color=np.full(n, 0xff2040f0, np.uint32), width=128.0, height=128.0)
    sc.path_stroke, sc.dashes = st, np.asarray(pattern, np.float32)
    sc.contour_closed = np.zeros(len(starts) - 1, np.uint8)
    return sc


WHOLE = [[1 + i % 17, 3, 1 + i % 5] for i in range(40)]
SHORT = [[2 + i % 3] for i in range(40)]
FAR = [[4, -3, 5], [3, 2], [-1, 6], [-2, -2]]


@pytest.mark.parametrize("contours,kinds,pattern", [
    *((WHOLE, k, (1e6, 1.0)) for k in ([1], [2], [3], [1, 3, 2])),  # whole segments, gaps never reached
    *((SHORT, k, (3.0, 0.5)) for k in ([1], [2], [3], [1, 3, 2])),
    *(([[9, 9]], k, (0.25, 0.125, 2.0)) for k in ([1], [2], [3], [1, 3, 2])),
    (FAR, [2], (1e6, 1.0)), (FAR[:3], [2], (11.0, 2.0))])
def test_pieces_match_oracle(pf, oracle_mod, contours, kinds, pattern):
    sc = paths(contours, kinds, pattern)
    want = oracle_mod.stroke_scene(sc)
    with pf.Renderer() as r:
        r.upload(sc)
        got = r.outline()
        for k in OUTLINE_KEYS:
            g, w = got[k], getattr(want, k)
            if g.dtype == np.float32:
                g, w = (np.where(np.isnan(x), np.float32(np.nan), x) for x in (g, w))
            assert g.shape == w.shape and np.array_equal(g.view(np.uint8), w.view(np.uint8)), k
