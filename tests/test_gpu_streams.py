"""Frames whose binning classes run at once, on side streams: on a caller's own stream, and in two contexts that
two threads draw with at the same time."""
import threading

import numpy as np
import pytest

import scenes as S
from conftest import TILE_KEYS

pytestmark = pytest.mark.gpu


def _scenes(seed):
    return [S.mixed(seed, 1500, 4096), S.clipped(seed, 60, 512), S.gradient_scene(seed, 60, 512)]


def _frames(r, scs):
    out = []
    r.upload(scs)
    for frame in (r.render, r.render_learned, r.render_learned, r.render_learned, r.render):
        frame()
        out.append([r.image(i) for i in range(len(scs))])
    return out, [r.canon(i) for i in range(len(scs))]


def _same(got, want):
    for a, b in zip(got[0], want[0]):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    for a, b in zip(got[1], want[1]):
        assert all(np.array_equal(a[k], b[k]) for k in TILE_KEYS)


def test_callers_stream(pf):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    scs = _scenes(3)
    with pf.Renderer() as r, pf.Renderer(stream=stream.cuda_stream) as own:
        r.sizer_load()
        own.sizer_load()
        _same(_frames(own, scs), _frames(r, scs))


def test_two_threads(pf):
    work = [_scenes(4), _scenes(5)]
    want = []
    for scs in work:
        with pf.Renderer() as r:
            r.sizer_load()
            want.append(_frames(r, scs))
    got = [[], []]

    def draw(k):
        with pf.Renderer() as r:
            r.sizer_load()
            for _ in range(3):
                got[k].append(_frames(r, work[k]))

    threads = [threading.Thread(target=draw, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(got[k]) == 3
        for g in got[k]:
            _same(g, want[k])
