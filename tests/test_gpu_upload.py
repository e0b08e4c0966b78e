"""What an upload stages and what it copies by itself: arrays around the staged size (128 KB: 16,384
points, 32,768 starts or colours), odd lengths that leave every array of the next scene unaligned, and
more ranges than one spreading kernel takes (32: every other scene has gradients), against the oracle."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS

pytestmark = pytest.mark.gpu


def polygons(seed, sizes, side=256):
    """A closed polygon per size, around points of the canvas."""
    rng = np.random.default_rng(seed)
    pts = [(rng.uniform(8, side - 8, 2) + rng.uniform(-7, 7, (n, 2))).astype(np.float32) for n in sizes]
    n = len(sizes)
    return S.Scene(points=np.concatenate(pts), flags=np.zeros(sum(sizes), np.uint8),
                   contour_start=np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32),
                   path_start=np.arange(n + 1, dtype=np.uint32), fill_rule=(np.arange(n) % 2).astype(np.uint8),
                   color=rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32), width=float(side), height=float(side))


def check(renderer, oracle_mod, batch):
    renderer.upload(batch)
    renderer.render()
    for i, sc in enumerate(batch):
        got, want = renderer.canon(i), oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11, threads=8)
        for key in TILE_KEYS:
            assert np.array_equal(got[key], want[key]), (i, key)


@pytest.mark.parametrize("n", [16383, 16384, 16385])
def test_points_around_the_staged_size(renderer, oracle_mod, n):
    check(renderer, oracle_mod, [polygons(1, [7, 5]), polygons(n, [n - 100, 97, 3]), polygons(3, [11])])


@pytest.mark.parametrize("n", [32766, 32767, 32768])
def test_paths_around_the_staged_size(renderer, oracle_mod, n):
    check(renderer, oracle_mod, [polygons(4, [3] * n), polygons(5, [5, 3])])


@pytest.mark.parametrize("n", [1, 33, 70])
def test_many_ranges(renderer, oracle_mod, n):
    batch = [polygons(10 + i, [3 + i % 9, 4, 5 + i % 4][:1 + i % 3]) for i in range(n)]
    for i in range(0, n, 2):
        batch[i] = S.with_gradients(batch[i], seed=i, share=0.7)
    check(renderer, oracle_mod, batch)
    images = [renderer.image(i) for i in range(n)]
    for i, sc in enumerate(batch):
        renderer.upload(sc)
        renderer.render()
        assert np.array_equal(renderer.image(0), images[i]), i
