"""Stroke jobs by a lane per path and by its warp: paths of one contour among paths of 31, 32, 33 and hundreds,
few contours a path on average and many, filled, open, closed and dashed, with empty contours; against the
oracle's outline bit for bit."""
import numpy as np
import pytest

import scenes as S
from conftest import OUTLINE_KEYS


def _scene(counts, seed, dash):
    """Paths of the given numbers of contours, of 0 to 4 points each."""
    rng = S.Rng(seed, 31)
    n, c = len(counts), int(sum(counts))
    size = rng.integers(0, 4, c)
    pts = (rng.uniform(2 * int(size.sum())).reshape(-1, 2) * 200.0).astype(np.float32)
    st = np.zeros(n, S.STROKE_DTYPE)
    st["line_width"] = np.where(np.arange(n) % 4 == 3, 0.0, 2.0)  # every fourth path is filled
    st["miter_limit"] = 4.0
    st["dash_count"] = np.where(np.arange(n) % 3 == 0, dash, 0)
    sc = S.Scene(points=pts, flags=np.zeros(len(pts), np.uint8),
                 contour_start=np.concatenate([[0], np.cumsum(size)]).astype(np.uint32),
                 path_start=np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32),
                 fill_rule=np.zeros(n, np.uint8), color=np.full(n, 0xff2040f0, np.uint32), width=200.0, height=200.0)
    sc.path_stroke = st
    sc.contour_closed = (np.arange(c) % 3 == 0).astype(np.uint8)
    sc.dashes = np.array([9.0, 5.0], np.float32)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[1] * 70, [1, 0, 2, 1] * 40 + [31, 32, 33, 64, 65], [1] * 300 + [400] + [1] * 31,
                                    [40, 5, 33, 6] * 12, [700]])
@pytest.mark.parametrize("dash", [0, 2])
def test_jobs_match_oracle(pf, oracle_mod, counts, dash):
    sc = _scene(counts, len(counts) + dash, dash)
    want = oracle_mod.stroke_scene(sc)
    with pf.Renderer() as r:
        r.upload(sc)
        got = r.outline()
    for k in OUTLINE_KEYS:
        w = getattr(want, k)
        assert got[k].shape == w.shape and np.array_equal(got[k].view(np.uint8), w.view(np.uint8)), k
