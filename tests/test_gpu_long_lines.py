"""Paths of long lines, against the oracle bit for bit: a few, which the warps of a CTA or cluster share out, and
hatchings, whose warps walk their lines in step; by class (a warp's rect, a CTA's, a cluster's, one of the
global passes), on either side of the lines where each begins."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS
from test_gpu_edges import LIST_KEYS
from test_gpu_walk import lines, walkable

pytestmark = pytest.mark.gpu


def _path(rng, side, n, zigzag):
    """n lines across side px: from edge to edge, or to anywhere; a short one now and then."""
    p = rng.uniform(2 * n).reshape(-1, 2) * (side - 4.0) + 2.0
    if zigzag:
        p[:, 0] = np.where(np.arange(n) % 2, side - 3.0, 2.0) + rng.uniform(n) * 0.9
    short = rng.uniform(n) < 0.2
    p[1:] = np.where(short[1:, None], p[:-1] + 5.0, p[1:])
    return np.clip(p, 1.0, side - 1.0).astype(np.float32)


# canvas side: rects of at most 128, 1,088, 4,352, 16,896 words, a cluster's, and more columns than it takes
@pytest.mark.parametrize("side", [150.0, 500.0, 1000.0, 2000.0, 3500.0, 8300.0])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 49, 100, 400])
@pytest.mark.parametrize("zigzag", [False, True])
def test_long_lines_match_oracle(renderer, oracle_mod, side, n, zigzag):
    rng = S.Rng(int(side) + n, 23)
    paths = walkable(oracle_mod, [_path(rng, side, n, zigzag) for _ in range(3)], side, None)
    if not paths:
        pytest.skip("every path has a line that the reference does not return from")
    sc = lines(paths, side)
    want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11)
    renderer.upload(sc)
    renderer.render()
    got = renderer.canon()
    for key in TILE_KEYS + LIST_KEYS:
        assert np.array_equal(got[key], want[key]), key
