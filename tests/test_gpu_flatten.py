"""Flattening by the lanes of a warp, and the kernel picked for shallow segments, against the
oracle's tiles: from one segment (a group of one) to more than every resident warp's group, shallow
and deep ones, curves that fill the warp's pool, and contours that stop at a malformed pattern."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS

pytestmark = pytest.mark.gpu


def curves(seed, n_paths, segs, span, side=512.0):
    """Paths of `segs` segments (cubics, quadratics and lines in turn), each path in a box of `span`
    px; a third of them open, some with point flags that end the contour early."""
    rng = S.Rng(seed, 22)
    kinds = np.resize([3, 2, 3, 1], segs)
    flags1 = np.concatenate([[0]] + [[[0], [1, 0], [1, 2, 0]][k - 1] for k in kinds]).astype(np.uint8)
    n = len(flags1)
    flags = np.tile(flags1, (n_paths, 1))
    origin = rng.uniform(2 * n_paths).reshape(n_paths, 1, 2) * side - 0.5 * span + 0.25 * side
    pts = (origin + rng.uniform(2 * n_paths * n).reshape(n_paths, n, 2) * span).astype(np.float32)
    closed = np.arange(n_paths) % 3 != 0
    pts[closed, -1] = pts[closed, 0]
    for p in range(5, n_paths, 11):  # a pattern the iterator stops at
        flags[p, min(n - 1, p % n)] = 2
    first = (np.arange(n_paths + 1) * n).astype(np.uint32)
    return S.Scene(points=pts.reshape(-1, 2), flags=flags.reshape(-1), contour_start=first,
                   path_start=np.arange(n_paths + 1, dtype=np.uint32), fill_rule=np.zeros(n_paths, np.uint8),
                   color=np.full(n_paths, 0xff3080c0, np.uint32), width=side, height=side)


@pytest.mark.parametrize("n_paths,segs,span", [
    (1, 1, 300.0), (3, 33, 2.0), (3, 33, 400.0), (40, 70, 30.0), (700, 50, 8.0), (1500, 40, 60.0),
    (30000, 17, 12.0), (2, 40, 60000.0)])
def test_flatten_matches_oracle(renderer, oracle_mod, n_paths, segs, span):
    sc = curves(n_paths + segs, n_paths, segs, span)
    want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11)
    renderer.upload(sc)
    for _ in range(2):  # a second frame over the buffers the first one left
        renderer.render()
        got = renderer.canon()
        for key in TILE_KEYS:
            assert np.array_equal(got[key], want[key]), key
    renderer.sizer_load()
    renderer.render_learned()
    got = renderer.canon()
    for key in TILE_KEYS:
        assert np.array_equal(got[key], want[key]), key
