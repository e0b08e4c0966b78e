"""Many dashed paths, of which the short ones are dashed by a lane each and the rest by warps, against the oracle's
outline bit for bit: on either side of the number of paths from which on that is so, with the border
between them at different numbers of steps, with lines and curves, and with a pool of chunks that the long
ones overrun at first."""
import numpy as np
import pytest

import scenes as S
from conftest import OUTLINE_KEYS

MANY, STEPS = 16384, 64  # paths from which on lanes dash, and a number of steps


def _scene(n, long, lengths, quads):
    """n paths of one contour each; `long` of them, spread out, of the longest of the lengths."""
    rng = S.Rng(n + long, 29)
    a = rng.uniform(2 * n).reshape(-1, 2) * 400.0
    turn = rng.uniform(n) * 6.2831853
    size = np.asarray(lengths[:-1])[rng.integers(0, len(lengths) - 2, n)] * (0.5 + rng.uniform(n))
    size[np.linspace(0, n - 1, long).astype(int)] = lengths[-1]
    d = np.stack([np.cos(turn), np.sin(turn)], 1) * size[:, None]
    mid = a + 0.5 * d + np.stack([-d[:, 1], d[:, 0]], 1) * 0.2
    pts = np.stack([a, mid, a + d], 1)
    st = np.zeros(n, S.STROKE_DTYPE)
    st["line_width"] = 1.5
    st["miter_limit"] = 4.0
    st["dash_count"] = 2
    st["dash_first"] = (np.arange(n) % 2) * 2
    st["dash_offset"] = np.linspace(0.0, 2.9, n)
    sc = S.Scene(points=pts.astype(np.float32).reshape(-1, 2), flags=np.tile(np.array([0, 1 if quads else 0, 0], np.uint8), n),
                 contour_start=np.arange(n + 1, dtype=np.uint32) * 3, path_start=np.arange(n + 1, dtype=np.uint32),
                 fill_rule=np.zeros(n, np.uint8), color=np.full(n, 0xff2040f0, np.uint32), width=400.0, height=400.0)
    sc.path_stroke = st
    sc.contour_closed = (np.arange(n) % 3 == 0).astype(np.uint8)
    sc.dashes = np.array([2.0, 1.0, 1.0, 2.5], np.float32)
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("n", [MANY - 1, MANY, 20000])
@pytest.mark.parametrize("long,lengths", [
    (0, (0.0, 1.0, 12.0, 40.0)),           # every path by a lane
    (40, (3.0, 20.0, 20000.0)),            # chains of thousands of steps among them
    (5000, (3.0, 1.5 * STEPS, 2.0 * STEPS)),  # two lengths, near each other
    (MANY - 1, (5.0, 300.0))])             # nearly all of one length, past the first pool
@pytest.mark.parametrize("quads", [False, True])
def test_many_dashed_paths_match_oracle(pf, oracle_mod, n, long, lengths, quads):
    sc = _scene(n, long, lengths, quads)
    want = oracle_mod.stroke_scene(sc)
    with pf.Renderer() as r:
        for _ in range(2):
            r.upload(sc)
            got = r.outline()
            for k in OUTLINE_KEYS:
                w = getattr(want, k)
                assert got[k].shape == w.shape and np.array_equal(got[k].view(np.uint8), w.view(np.uint8)), k
