"""The framebuffer rows' path lists, against the oracle's composite lists: path counts around a
chunk of the list kernel (256), canvas heights around its window of 64 tile rows, alone and as a
range of a batch."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS
from test_gpu_edges import LIST_KEYS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_paths", [1, 255, 256, 257, 700])
@pytest.mark.parametrize("height", [1, 1008, 1024, 1041, 2100])
def test_row_lists(renderer, oracle_mod, n_paths, height):
    sc = S.glyphs(seed=n_paths + height, n_paths=n_paths, side=max(height, 300))
    sc.width, sc.height = 80.0, float(height)
    # translucent, so that lists are long
    sc.color = np.full(n_paths, 0x80402010, np.uint32)
    other = S.plain_small(seed=5, n_paths=9, side=100)
    want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11)
    for batch, first in (([sc], 0), ([other, sc, other], 1)):
        renderer.upload(batch)
        renderer.render(first, 1)
        got = renderer.canon(first)
        for key in TILE_KEYS + LIST_KEYS:
            assert np.array_equal(got[key], want[key]), (first, key)
