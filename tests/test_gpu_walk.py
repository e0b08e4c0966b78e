"""The binning walk's forms of one line, against the oracle bit for bit: lines on tile corners and
boundaries, of one to hundreds of tiles (walked by a lane or by the whole warp, wherever
long_line draws the line), coordinates too small or too far out for the lane form, tiles outside
the path's rect, and paths of 1 to 3000 lines (a part of a warp, several warps, a full stage)."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS
from test_gpu_edges import LIST_KEYS


def lines(paths, side):
    """One closed path per list of points, opaque colours."""
    n = [len(p) for p in paths]
    first = np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)
    return S.Scene(points=np.concatenate(paths), flags=np.zeros(sum(n), np.uint8), contour_start=first,
                   path_start=np.arange(len(n) + 1, dtype=np.uint32), fill_rule=np.zeros(len(n), np.uint8),
                   color=np.arange(len(n), dtype=np.uint32) * 977 | np.uint32(0xff000000), width=side, height=side)


def _snapped(rng, n, lo, hi, grid):
    """Points on multiples of `grid`, some of them nudged to a neighbouring float."""
    p = (np.round(rng.uniform(n).reshape(-1, 2) * (hi - lo) / grid + lo / grid) * grid).astype(np.float32)
    nudge = rng.integers(-1, 1, n).reshape(-1, 2)
    return np.where(nudge == 0, p, np.nextafter(p, np.where(nudge > 0, 1e9, -1e9).astype(np.float32)))


def scene(seed, side=300.0):
    rng = S.Rng(seed, 21)
    paths = [_snapped(rng, 4, -48.0, side + 48.0, g) for g in (16.0, 8.0, 0.5) for _ in range(60)]
    # short lines: a walk from point to point, up to about a tile a step, with repeated points
    for n, step in ((31, 3.0), (200, 12.0), (3000, 9.0), (900, 40.0)):
        d = (rng.uniform(2 * n).reshape(-1, 2) - 0.5) * 2.0 * step * (rng.uniform(n) < 0.9)[:, None]
        walk = np.cumsum(d, axis=0) + 0.5 * side
        paths.append((np.abs((walk + side) % (2 * side) - side) - 10.0).astype(np.float32))
    # around the axes: zeros, subnormal and tiny coordinates on both sides of them
    tiny = np.array([0.0, 1e-44, -1e-44, 1e-38, -3e-37, 2.0 ** -122, -2.0 ** -30, 17.0, -17.0], np.float32)
    k = rng.integers(0, len(tiny) - 1, 60).reshape(-1, 2)
    paths.append(tiny[k])
    # far above the view box (the walk's top is open), and far to the sides and below (clipped)
    far = np.array([-3e6, -2e5, -500.0, 20.0, 150.0, 290.0, 400.0, 9e5], np.float32)
    paths.append(np.stack([far[rng.integers(2, 7, 40)], far[rng.integers(1, 7, 40)]], axis=1))
    return paths


def walkable(oracle_mod, paths, side, view_box):
    """The paths whose walk ends: a line through a tile corner may, by rounding, miss its end tile,
    which the reference never returns from and the library reports as an error."""
    out = []
    for p in paths:
        sc = lines([p], side)
        sc.view_box = view_box
        try:
            oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11)
            out.append(p)
        except RuntimeError:
            pass
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("view_box", [None, (-37.0, -20.5, 250.0, 260.0), (33.0, 17.0, 280.0, 301.0)])
@pytest.mark.parametrize("long_line", [1.0, 8.0, 4096.0])
def test_walk_matches_oracle(renderer, oracle_mod, view_box, long_line):
    start = renderer.tuning()
    try:
        renderer.set_tuning({**start, "long_line": long_line})
        for seed in (1, 2):
            vb = None if view_box is None else np.asarray(view_box, np.float32)
            paths = walkable(oracle_mod, scene(seed), 300.0, vb)
            assert len(paths) > 120
            sc = lines(paths, 300.0)
            sc.view_box = vb
            want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11)
            renderer.upload(sc)
            renderer.render()
            got = renderer.canon()
            for key in TILE_KEYS + LIST_KEYS:
                assert np.array_equal(got[key], want[key]), (seed, key)
    finally:
        renderer.set_tuning(start)
