"""The binning's size classes at their borders, against the oracle: rects of 127 to 130 words (a warp
or a CTA), lines per path around the most a warp bins and stages, the CTA classes' 1088, 4352 and
16896 words and past them (a cluster of CTAs, up to 512 columns and 16384 tiles a band; the global
passes), in frames large enough that a path's lines do not move it to a larger class and in small
ones where they do."""
import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS


def paths(seed, sizes, n_lines, side):
    """A closed polyline per (w, h) tiles rect and line count, over all of its rect."""
    rng = S.Rng(seed, 24)
    out = []
    for (w, h), n in zip(sizes, n_lines):
        lo = np.floor(rng.uniform(2) * (side / 16 - np.array([w, h]))) * 16
        step = (rng.uniform(2 * n).reshape(n, 2) - 0.5) * np.array([w, h]) * 16 * min(1.0, 40.0 / max(w, h))
        walk = np.abs((np.cumsum(step, axis=0) + 5.0) % (2 * 16 * np.array([w, h])) - 16 * np.array([w, h]))
        walk[:2] = [[0.5, 0.5], [16 * w - 0.5, 16 * h - 0.5]]  # the rect's corners
        out.append((lo + np.clip(walk, 0.25, 16 * np.array([w, h]) - 0.25)).astype(np.float32))
    n = [len(p) for p in out]
    return S.Scene(points=np.concatenate(out), flags=np.zeros(sum(n), np.uint8),
                   contour_start=np.concatenate([[0], np.cumsum(n)]).astype(np.uint32),
                   path_start=np.arange(len(n) + 1, dtype=np.uint32), fill_rule=np.zeros(len(n), np.uint8),
                   color=np.full(len(n), 0xff6080a0, np.uint32), width=float(side), height=float(side))


SMALL = [(1, 127), (1, 126), (7, 17), (8, 15), (8, 16), (12, 9), (12, 10), (31, 3), (63, 1), (64, 1), (65, 1), (2, 2)]
LARGE = [(32, 33), (33, 32), (33, 33), (64, 67), (65, 66), (66, 66), (128, 131), (129, 130), (130, 130), (2, 140)]


HUGE = [(512, 34), (513, 34), (256, 256), (257, 257), (560, 31), (130, 501), (2, 9), (512, 128), (511, 129)]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,n,lines,side", [(SMALL, 6000, (383, 384, 385, 400), 2304), (SMALL, 60, (3, 64, 65, 383, 385, 3000), 2304),
                                                (LARGE, 40, (5, 700, 1025, 5000), 2304), (HUGE, 18, (40, 9000), 9100)])
def test_classes_match_oracle(renderer, oracle_mod, sizes, n, lines, side):
    sc = paths(n, [sizes[i % len(sizes)] for i in range(n)], [lines[i // len(sizes) % len(lines)] for i in range(n)], side)
    want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11, threads=8)
    renderer.upload(sc)
    renderer.render()
    got = renderer.canon()
    for key in TILE_KEYS:
        assert np.array_equal(got[key], want[key]), key


@pytest.mark.gpu
@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 4095, 4096, 4097, 8200])
def test_lists_by_path_count(pf, oracle_mod, n, learned):
    """Around one block's threads (1024) and the paths one block lists (4096); every class present."""
    sizes = [SMALL[i % 12] for i in range(n)]
    for k, s in enumerate([(33, 33), (66, 66), (130, 130), (513, 34), (256, 2)]):
        sizes[(k * 997 + 5) % n] = s
    sc = paths(n, sizes, [3 + i % 9 for i in range(n)], 8400)
    want = oracle_mod.tile_scene(sc, oracle_mod.Z_D3D11, threads=8)
    with pf.Renderer() as r:
        r.sizer_load(pf.DEFAULT_WEIGHTS)
        r.upload(sc)
        r.render_learned() if learned else r.render()
        got = r.canon()
    for key in TILE_KEYS:
        assert np.array_equal(got[key], want[key]), key
