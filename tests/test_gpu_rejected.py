"""An upload that fails: a rejected batch leaves the one before as it was, a batch that does not fit leaves none."""
import dataclasses

import numpy as np
import pytest

import scenes as S

pytestmark = pytest.mark.gpu

INVALID, OUT_OF_MEMORY, NOT_READY = 1, 3, 6


def _batch(n):
    return [S.plain_small(seed=40 + i, n_paths=30 + i, side=192) for i in range(n)]


@pytest.mark.parametrize("n", [1, 2, 4, 7])  # scenes of the rejected batch: fewer, as many, more
@pytest.mark.parametrize("at", ["first", "last"])
def test_rejected_batch_leaves_the_one_before(pf, n, at):
    good = _batch(4)
    bad = _batch(n)
    k = 0 if at == "first" else n - 1
    bad[k] = dataclasses.replace(bad[k], load_action=2)
    with pf.Renderer() as r:
        r.sizer_load()
        r.upload(good)
        r.render()
        want = [r.image(i) for i in range(4)]
        for frame in (r.render, r.render_learned, r.render_learned, r.render_auto):
            with pytest.raises(pf.PfError) as e:
                r.upload(bad)
            assert e.value.status == INVALID
            assert all(np.array_equal(r.image(i), want[i]) for i in range(4))
            frame()
            assert all(np.array_equal(r.image(i), want[i]) for i in range(4))


def test_batch_that_does_not_fit_leaves_none(pf):
    good = _batch(4)
    # 25 images of 17 GB: the allocation fails at once
    huge = [dataclasses.replace(S.plain_small(seed=3, n_paths=2, side=64), width=65536.0, height=65536.0)] * 25
    with pf.Renderer() as r:
        r.sizer_load()
        r.upload(good)
        r.render()
        with pytest.raises(pf.PfError) as e:
            r.upload(huge)
        assert e.value.status == OUT_OF_MEMORY
        for call in (r.render, r.render_learned, r.render_auto, r.image):
            with pytest.raises(pf.PfError) as e:
                call()
            assert e.value.status == NOT_READY


def test_failed_allocation_does_not_fail_the_next_call(pf):
    good = _batch(4)
    huge = [dataclasses.replace(S.plain_small(seed=3, n_paths=2, side=64), width=65536.0, height=65536.0)] * 25
    with pf.Renderer() as r:
        r.upload(good)
        r.render()
        want = r.image(2)
        with pytest.raises(pf.PfError) as e:
            r.upload(huge)
        assert e.value.status == OUT_OF_MEMORY
        r.upload(good)
        r.render()
        assert np.array_equal(r.image(2), want)
