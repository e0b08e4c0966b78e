"""Which grid the composite takes by itself - a warp per tile, or resident warps in frames of many tiles with
gradients or clip paths - never shows in the pixels: scenes in a batch on either side of the line equal
the scene alone, whose few tiles are always a warp each."""
import numpy as np
import pytest

import scenes as S

pytestmark = pytest.mark.gpu

SMS = 152


def _clipped(side):
    return S.clipped(4, 40, side)


def _gradients(side):
    return S.gradient_scene(4, 40, side)


def _both(side):
    return S.with_gradients(_clipped(side), 9, 0.5)


# tiles per resident warp at the line, and the resident warps per SM
@pytest.mark.parametrize("make,line,warps,side", [(_gradients, 4, 20, 512), (_both, 4, 20, 512),
                                                  (_clipped, 64, 24, 1024)])
@pytest.mark.parametrize("past", [-1, 0, 1])
@pytest.mark.parametrize("load", [0, 1])
def test_batch_on_either_side_of_the_line_equals_alone(pf, make, line, warps, side, past, load):
    sc = make(side)
    sc.load_action = load
    n = -(-line * warps * SMS // (side // 16) ** 2) + past  # from past = 0 on, resident warps
    dest = np.random.default_rng(1).integers(0, 256, (side, side, 4), dtype=np.uint8)
    with pf.Renderer() as r:
        r.upload(sc)
        r.write_image(0, dest)
        r.render()
        want = r.image()
        r.upload([sc] * n)
        for i in range(n):
            r.write_image(i, dest)
        r.render()
        for i in range(n):
            assert np.array_equal(r.image(i), want), i
