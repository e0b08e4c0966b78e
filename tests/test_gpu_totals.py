"""Frame totals past 2^32.

A frame's tiles, columns, row entries and leaf lines are numbered in 32 bits.  A frame that needs more is
refused with PF_ERR_OVERFLOW before anything is sized or written by those numbers; leaf budgets past
2^32 (a learned frame's, with a wide margin) send the frame to the exact method instead.
"""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS

pytestmark = pytest.mark.gpu

OVERFLOW = 4


def _triangles(n, view_box=None):
    pts = np.tile(np.array([[-70000, -70000], [70000, -70000], [0, 70000]], np.float32), (n, 1))
    return S.Scene(points=pts, flags=np.zeros(3 * n, np.uint8), contour_start=np.arange(n + 1, dtype=np.uint32) * 3,
                   path_start=np.arange(n + 1, dtype=np.uint32), fill_rule=np.zeros(n, np.uint8),
                   color=np.full(n, 0x80402010, np.uint32), width=64.0, height=64.0, clear=0xffffffff,
                   view_box=view_box)


def _cubics(contours):
    """Contours of 64 cubics that each bisect into thousands of lines."""
    one = np.concatenate([np.array([[40, 30]], np.float32),
                          np.tile(np.array([[1.0e6, -1.0e6], [-1.0e6, 1.0e6], [40, 30]], np.float32), (64, 1))])
    flags = np.concatenate([np.zeros(1, np.uint8), np.tile(np.array([1, 2, 0], np.uint8), 64)])
    return S.Scene(points=np.tile(one, (contours, 1)), flags=np.tile(flags, contours),
                   contour_start=np.arange(contours + 1, dtype=np.uint32) * 193,
                   path_start=np.array([0, contours], np.uint32), fill_rule=np.zeros(1, np.uint8),
                   color=np.full(1, 0xff402010, np.uint32), width=64.0, height=64.0, clear=0xffffffff)


def _usable(pf, r):
    sc = S.plain_small(seed=5, n_paths=20, side=256)
    r.upload(sc)
    r.render()
    with pf.Renderer() as fresh:
        fresh.upload(sc)
        fresh.render()
        assert np.array_equal(r.image(), fresh.image())


@pytest.mark.parametrize("n", [64, 65, 130])  # 2^26 tiles each: totals that wrap to 0, 2^26 and 2 * 2^26
def test_tiles(pf, n):
    box = np.array([-65536, -65536, 65536, 65536], np.float32)
    with pf.Renderer() as r:
        r.sizer_load()
        r.upload(_triangles(n, box))
        for frame in (r.render, r.render_learned, r.render_auto):
            with pytest.raises(pf.PfError) as e:
                frame()
            assert e.value.status == OVERFLOW
        _usable(pf, r)


def test_leaf_lines(pf):
    with pf.Renderer() as r:
        r.upload(_cubics(1))
        per = r.render()["microlines"]
        assert per >= 64 * 1024
        r.upload(_cubics(2 ** 32 // per + 2))
        with pytest.raises(pf.PfError) as e:
            r.render()
        assert e.value.status == OVERFLOW
        _usable(pf, r)


@pytest.mark.parametrize("n", [5, 9, 40])  # 1e9 lines each: 5e9, 9e9 and 4e10
def test_leaf_budgets(pf, n):
    sc = S.plain_small(seed=6, n_paths=n, side=256)
    with pf.Renderer() as r:
        r.sizer_load()
        r.upload(sc)
        r.render()
        want, img = r.canon(), r.image()
        r.sizer_margin(1.0e9, 1.0e9)
        for _ in range(3):
            r.render_learned()
            got = r.canon()
            for k in TILE_KEYS:
                assert np.array_equal(got[k], want[k]), k
            assert np.array_equal(r.image(), img)
