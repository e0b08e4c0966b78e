"""Lines whose walk, by rounding, passes its end tile by: the reference never returns from them, the library
reports the walk bound.  Both forms of the walk find them, in every binning class, also where a path's
visits do not fit the stage; the context stays usable."""
import numpy as np
import pytest

from conftest import TILE_KEYS
from test_gpu_walk import lines, scene

pytestmark = pytest.mark.gpu

KERNEL_LIMIT = 5
# canvas side (0: the line's own box), points around the line: a warp's class, those of a CTA, and a
# cluster's; few enough visits for the stage, and more
PATHS = [(0.0, 0), (0.0, 60), (300.0, 30), (300.0, 200), (300.0, 3500), (2400.0, 20), (2400.0, 900)]


def _lost(oracle_mod):
    """Lines (a, b) that the oracle does not come to the end of, there or back, within 300 px."""
    out = []
    for seed in (1, 2):
        for p in scene(seed)[:180]:
            if (p < 0).any() or (p > 300).any():
                continue
            for a, b in zip(p, np.roll(p, -1, axis=0)):
                try:
                    oracle_mod.tile_scene(lines([np.stack([a, b])], 300.0), oracle_mod.Z_D3D11)
                except RuntimeError as e:
                    assert "status 5" in str(e)
                    out.append((a, b))
    return out


@pytest.fixture(scope="module")
def lost(oracle_mod):
    found = _lost(oracle_mod)
    assert len(found) >= 4
    return found


@pytest.mark.parametrize("long_line", [1.0, 8.0, 4096.0])
@pytest.mark.parametrize("side,around", PATHS)
def test_lost_line_is_an_error(pf, oracle_mod, lost, long_line, side, around):
    rng = np.random.default_rng(9)
    good = lines([np.array([[10, 10], [200, 40], [90, 260]], np.float32)], 300.0)
    want = oracle_mod.tile_scene(good, oracle_mod.Z_D3D11)
    with pf.Renderer() as r:
        r.sizer_load()
        r.set_tuning({**r.tuning(), "long_line": long_line})
        for a, b in lost[::4]:
            if side:
                more = rng.random((around, 2)) * (side - 8.0) + 4.0
            else:  # from end to end of the line's box
                t = rng.random((around, 2)) * 0.05
                more = a + (b - a) * np.where(np.arange(around)[:, None] % 2, t, 1.0 - t)
            more = more.astype(np.float32)
            r.upload(lines([np.concatenate([np.stack([a, b, a]), more])], side or 300.0))
            for frame in (r.render, r.render_learned):
                with pytest.raises(pf.PfError) as e:
                    frame()
                assert e.value.status == KERNEL_LIMIT
        r.upload(good)
        r.render()
        got = r.canon()
        for key in TILE_KEYS:
            assert np.array_equal(got[key], want[key]), key
