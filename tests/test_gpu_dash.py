"""Dashed contours through the chunk pool and past it, against the oracle's outline bit for bit:
paths of a point to many chunks, dashes that run on across contours and over curves, a first upload
whose pool is too small (walked again) and a second one whose pool fits (gathered)."""
import numpy as np
import pytest

import scenes as S
from conftest import OUTLINE_KEYS


def dashed(seed, n_paths, pattern, length, kinds):
    """Stroked paths of two contours each, `kinds` the points per segment in turn (1 line, 2
    quadratic, 3 cubic), about `length` px across, with one dash pattern."""
    rng = S.Rng(seed, 23)
    flags = np.concatenate([[0]] + [[[0], [1, 0], [1, 2, 0]][k - 1] for k in kinds]).astype(np.uint8)
    n = len(flags)
    pts = ((rng.uniform(4 * n_paths * n).reshape(-1, 2) - 0.25) * length).astype(np.float32)
    st = np.zeros(n_paths, S.STROKE_DTYPE)
    st["line_width"] = 1.5
    st["miter_limit"] = 4.0
    st["dash_count"] = len(pattern)
    st["dash_offset"] = np.linspace(0.0, 0.9 * sum(pattern), n_paths)
    sc = S.Scene(points=pts, flags=np.tile(flags, 2 * n_paths), contour_start=np.arange(2 * n_paths + 1, dtype=np.uint32) * n,
                 path_start=np.arange(n_paths + 1, dtype=np.uint32) * 2, fill_rule=np.zeros(n_paths, np.uint8),
                 color=np.full(n_paths, 0xff2040f0, np.uint32), width=256.0, height=256.0)
    sc.path_stroke = st
    sc.contour_closed = (np.arange(2 * n_paths) % 3 == 0).astype(np.uint8)
    sc.dashes = np.asarray(pattern, np.float32)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("n_paths,pattern,length,kinds", [
    (1, (4.0, 2.0), 10.0, [1]), (1, (0.5, 0.25), 900.0, [1]), (3, (1.0, 0.0, 2.0, 1.0), 600.0, [1, 2, 3, 3]),
    (200, (7.0, 3.0, 1.0), 120.0, [3, 1, 2]), (70, (1e4, 5.0), 50.0, [2, 3])])
def test_dashed_outline_matches_oracle(pf, oracle_mod, n_paths, pattern, length, kinds):
    sc = dashed(n_paths, n_paths, pattern, length, kinds)
    want = oracle_mod.stroke_scene(sc)
    with pf.Renderer() as r:
        for _ in range(2):
            r.upload(sc)
            got = r.outline()
            for k in OUTLINE_KEYS:
                w = getattr(want, k)
                assert got[k].shape == w.shape and np.array_equal(got[k].view(np.uint8), w.view(np.uint8)), k
