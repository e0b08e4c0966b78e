"""The work a user of the renderer has it do, as cases for timing and for comparing outputs.

Two forms of use are covered.  A program that shows a new picture each time hands host arrays (or
SVG text) to the renderer and takes the image back: ``draw`` cases, where the upload, the frame
and the read-back all count.  A program that keeps its scenes on the device renders them frame
after frame: ``frame`` and ``learned`` cases, whose image stays on the device.  The sizer's
training step is the one path that computes real numbers.

Every frame also returns its integer totals (leaf lines, tiles, fills), which are exact.
"""
from __future__ import annotations

import dataclasses
import math
import os
import sys

import numpy as np
import torch

for _p in (os.path.join(os.getcwd(), "pathfinder-cpp_gb300"),):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import pfcuda  # noqa: E402
import scenes as S  # noqa: E402
import svg_docs  # noqa: E402


def listed():
    return [
        # one icon, host arrays in, pixels out: a UI that redraws small artwork; nothing but latency
        {"name": "draw_icon", "use": "draw", "family": "plain", "paths": 24, "side": 201},
        # the plain scene of 240 cubic paths, drawn whole from host arrays
        {"name": "draw_plain", "use": "draw", "family": "plain", "paths": 240, "side": 1024},
        # a page of text as it is typed: a few thousand small glyphs, drawn whole
        {"name": "draw_page", "use": "draw", "family": "glyphs", "paths": 3000, "side": 765},
        # SVG artwork: parse, upload (strokes, dashes and gradients on the device), frame, pixels
        {"name": "draw_svg", "use": "svg", "family": "svg", "scenes": 8, "paths": 96},
        # an animation's small frame over resident data, on a canvas that is no multiple of a tile
        {"name": "frame_plain", "use": "frame", "family": "plain", "paths": 240, "side": 1000},
        # a map or a drawing: 20,000 paths of every size, both fill rules, translucent ones, 4096 x 4096
        {"name": "frame_large", "use": "frame", "family": "large", "paths": 20000, "side": 4096},
        # a text-heavy screen: 150,000 glyph outlines
        {"name": "frame_glyphs", "use": "frame", "family": "glyphs", "paths": 150000, "side": 2048},
        # a mixture of the path families by the one-pass frame, whose buffers the sizer predicts
        {"name": "learned_mixed", "use": "learned", "family": "mixed", "paths": 8192, "side": 4095},
        # a server's batch: independent scenes of 16-4096 paths on canvases of 256-2048, one replayed frame
        {"name": "learned_batch", "use": "learned", "family": "batch", "scenes": 256, "paths": 4096},
        # the same kind of batch with clip paths, by the exact two-pass frame
        {"name": "frame_clips", "use": "frame", "family": "clips", "scenes": 24, "paths": 2048},
        # a batch of stroked and dashed drawings that changes each time: upload with the stroke pass, frame
        {"name": "frame_strokes", "use": "upload", "family": "strokes", "scenes": 48, "paths": 2048},
        # the sizer's training step on a mini-batch: loss, the gradients of all weights, and its predictions
        {"name": "sizer_step", "use": "sizer", "family": "sizer", "rows": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(["draw_plain", "draw_page", "svg", "plain", "large", "glyphs", "mixed", "batch", "clips",
                       "strokes", "gradients", "sizer"])
    if pick == "draw_plain":
        return {"use": "draw", "family": "plain", "paths": _log(rng, 8, 400), "side": _log(rng, 100, 1024)}
    if pick == "draw_page":
        return {"use": "draw", "family": "glyphs", "paths": _log(rng, 200, 8000), "side": _log(rng, 300, 1024)}
    if pick == "svg":
        return {"use": "svg", "family": "svg", "scenes": _log(rng, 1, 12), "paths": _log(rng, 16, 128)}
    if pick == "plain":
        return {"use": rng.choice(["frame", "learned"]), "family": "plain", "paths": _log(rng, 16, 1000),
                "side": _log(rng, 250, 2048)}
    if pick == "large":
        return {"use": rng.choice(["frame", "learned"]), "family": "large", "paths": _log(rng, 1000, 20000),
                "side": _log(rng, 2048, 4096)}
    if pick == "glyphs":
        return {"use": rng.choice(["frame", "learned"]), "family": "glyphs", "paths": _log(rng, 5000, 150000),
                "side": _log(rng, 1024, 2500)}
    if pick == "mixed":
        return {"use": rng.choice(["frame", "learned"]), "family": "mixed", "paths": _log(rng, 800, 12000),
                "side": _log(rng, 2048, 4096)}
    if pick == "batch":
        return {"use": rng.choice(["frame", "learned"]), "family": "batch", "scenes": _log(rng, 8, 200),
                "paths": rng.choice([1024, 2048, 4096])}
    if pick == "clips":
        return {"use": rng.choice(["frame", "learned"]), "family": "clips", "scenes": _log(rng, 2, 32),
                "paths": rng.choice([512, 1024, 2048])}
    if pick == "strokes":
        return {"use": "upload", "family": "strokes", "scenes": _log(rng, 2, 64), "paths": rng.choice([512, 1024, 2048])}
    if pick == "gradients":
        return {"use": rng.choice(["frame", "upload"]), "family": "gradients", "scenes": _log(rng, 1, 12),
                "paths": rng.choice([256, 512, 1024])}
    return {"use": "sizer", "family": "sizer", "rows": _log(rng, 1000, 65536) | 1}


def _scenes(case, seed):
    """The case's scenes, from its seed alone."""
    f = case["family"]
    first, seed = 1000 * (seed % 16001), seed % 500009  # the generators take seeds below 2^24
    if f == "plain":
        return [S.plain_small(seed=seed, n_paths=case["paths"], side=case["side"])]
    if f == "large":
        return [S.large_single(seed=seed, n_paths=case["paths"], side=case["side"])]
    if f == "glyphs":
        return [S.glyphs(seed=seed, n_paths=case["paths"], side=case["side"])]
    if f == "mixed":
        return [S.mixed(seed=seed, n_paths=case["paths"], side=case["side"])]
    out = []
    for i in range(case["scenes"]):
        # canvas and path count of scene i: the same for every seed, so that images have one layout
        u = S.Rng(i, 11).uniform(2)
        n = int(16 * (case["paths"] / 16) ** u[0])
        side = (256, 512, 1024, 2048)[int(4 * u[1])] if f == "batch" else (250, 512, 999, 1500)[int(4 * u[1])]
        if f == "strokes":
            out.append(S.stroked(seed=first + i, n_paths=n, side=side))
            continue
        sc = S.plain_small(seed=first + i, n_paths=n, side=side)
        if f == "gradients":
            sc = S.with_gradients(sc, first + i)
        elif f == "clips":
            sc = S.add_clips(sc, first + i)
            # every third path translucent, so that what lies below counts
            alpha = np.where(np.arange(sc.n_paths) % 3 == 0, 0x90000000, 0xFF000000).astype(np.uint32)
            sc = dataclasses.replace(sc, color=(sc.color & np.uint32(0xFFFFFF)) | alpha)
        out.append(sc)
    return out


def _svg_texts(case, seed):
    # the generator's documents, each on a page of a fixed size
    out = []
    for i in range(case["scenes"]):
        text = svg_docs.random_document(100 * seed + i, n_shapes=case["paths"])
        out.append('<svg xmlns="http://www.w3.org/2000/svg" xmlns:xlink="http://www.w3.org/1999/xlink" '
                   'width="%d" height="%d">' % (300 - 7 * (i % 8), 200 + 9 * (i % 8)) + text[text.index(">") + 1:])
    return out


def _sizer_inputs(case, seed):
    """Weights, features and labels of a training step: log1p counts and lengths, as the sizer sees them."""
    r = np.random.default_rng([seed, case["rows"]])
    n = case["rows"]
    top = np.array([5, 4, 4, 4, 1.2, 7, 7, 13, 9, 5, 8, 1], np.float64)  # the features' usual largest values
    feat = (r.random((n, 12)) * top).astype(np.float32)
    feat[:, 11] = np.where(feat[:, 11] < 0.5, 0.0, np.float32(np.log(2.0)))
    size = 0.5 * feat[:, 8] + 0.5 * feat[:, 0] + 0.3 * r.standard_normal(n)
    target = np.stack([size, size + 0.8], axis=1).astype(np.float32)
    bound = [np.sqrt(6 / 12), np.sqrt(6 / 64), np.sqrt(3 / 64)]
    parts = []
    for (rows, cols), b in zip(((64, 12), (64, 64), (2, 64)), bound):
        parts.append((r.random(rows * cols) * 2 - 1) * b)
        parts.append((r.random(rows) * 2 - 1) * 0.1)
    return np.concatenate(parts).astype(np.float32), feat, target


class _DeviceBytes:
    """The renderer's image buffer for torch.as_tensor, without a copy; the tensor keeps this
    object, and so the renderer that owns the memory."""

    def __init__(self, renderer, ptr, nbytes):
        self.renderer = renderer
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _images(r):
    """Every image of the last frame, where it lies on the device."""
    ptr = pfcuda.C.c_void_p()
    r._check(r.lib.pf_image_device_ptr(r.ctx, pfcuda.C.byref(ptr), None, None), r.ctx)
    return torch.as_tensor(_DeviceBytes(r, ptr.value, r.image_bytes()), device="cuda")


def _frame(r, stats):
    return {"image": _images(r),
            "totals": np.array([stats[k] for k in ("paths", "segments", "microlines", "tiles", "fills")], np.int64)}


def prepare(case, seed):
    use = case["use"]
    r = pfcuda.Renderer()
    if use == "svg":
        return {"use": use, "r": r, "texts": _svg_texts(case, seed)}
    if use == "sizer":
        w, feat, target = _sizer_inputs(case, seed)
        r.set_sizer_params(w)
        return {"use": use, "r": r, "feat": feat, "target": target}
    sc = _scenes(case, seed)
    st = {"use": use, "r": r, "scenes": sc}
    if use == "draw":
        return st
    if use == "upload":
        # the arrays as one program-owned copy, described once: what changes is their content
        pairs = [pfcuda.scene_view(s) for s in sc]
        st["views"], st["keep"] = [p[0] for p in pairs], [p[1] for p in pairs]
        return st
    if use == "learned":
        r.sizer_load()
    r.upload(sc)
    return st


def run(state):
    r, use = state["r"], state["use"]
    if use == "draw":
        return r.draw(state["scenes"][0])
    if use == "svg":
        docs = [pfcuda.SvgDocument(t) for t in state["texts"]]
        r.upload_views([d.view for d in docs])
        r.render()
        return [r.image(i) for i in range(len(docs))]
    if use == "sizer":
        grad, loss = r.sizer_gradient(state["feat"], state["target"])
        return {"grad": grad, "loss": np.array([loss], np.float32), "pred": r.sizer_predict(state["feat"])}
    if use == "upload":
        r.upload_views(state["views"])
    return _frame(r, r.render_learned() if use == "learned" else r.render())


def _points(case):
    """Points of the case's outlines, on average."""
    f = case["family"]
    if f in ("batch", "clips", "gradients", "strokes"):
        # paths per scene: log-uniform from 16 to case["paths"]
        n = case["scenes"] * (case["paths"] - 16) / math.log(case["paths"] / 16)
        return n, n * (28 if f == "strokes" else 49), case["scenes"] * (1.39e6 if f == "batch" else 0.89e6)
    if f == "svg":
        n = case["scenes"] * case["paths"]
        return n, n * 16, case["scenes"] * 5.4e4
    per = {"plain": 49, "large": 90, "glyphs": 52, "mixed": 66}[f]
    return case["paths"], case["paths"] * per, case["side"] ** 2


def work(case):
    if case["family"] == "sizer":
        n = case["rows"]
        return {"bytes": n * (12 + 2 + 2) * 4 + 5122 * 4 * 2, "flops": 3 * 2 * 4992 * n}
    paths, points, pixels = _points(case)
    # coordinates, point kinds, offsets, rule and colour in; RGBA8 out.  What is computed are
    # the crossings of curves with tiles and pixels, which a count of operations does not describe.
    return {"bytes": int(points * 9 + paths * 13 + pixels * 4), "flops": int(points * 100)}


def exact(case, seed):
    if case["family"] != "sizer":
        return None  # bytes and whole numbers
    w, feat, target = _sizer_inputs(case, seed)
    # the forward pass takes the weights rounded to bfloat16, the biases among them
    bits = w.view(np.uint32).astype(np.uint64)
    w = ((bits + 0x7FFF + ((bits >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)
    shapes, parts, at = ((64, 12), (64,), (64, 64), (64,), (2, 64), (2,)), [], 0
    for s in shapes:
        n = int(np.prod(s))
        parts.append(w[at:at + n].reshape(s))
        at += n
    w1, b1, w2, b2, w3, b3 = parts
    x, t = feat.astype(np.float64), target.astype(np.float64)
    z1 = x @ w1.T + b1
    h1 = np.maximum(z1, 0)
    z2 = h1 @ w2.T + b2
    h2 = np.maximum(z2, 0)
    pred = h2 @ w3.T + b3
    e = pred - t
    n = e.size
    dy = 2.0 * e / n
    d2 = (dy @ w3) * (z2 > 0)
    d1 = (d2 @ w2) * (z1 > 0)
    grad = [d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0)]
    return {"grad": np.concatenate([g.reshape(-1) for g in grad]), "loss": np.array([(e * e).sum() / n]),
            "pred": pred}
