"""The blend's per-cell record lists against the oracle, where they can go
wrong: batches of 128 records one short, full and one over, images that end
inside a tile or a 4x4 cell, long thin splats at every angle (the ellipse
test decides which cells walk them), splats far larger than the image, and
records whose colour is not finite (a pixel they do not touch must not see
them). Images are equal bit for bit, as everywhere on the forward path."""
from __future__ import annotations

import numpy as np
import pytest

import lucabrtrender_b200 as L
import helpers as H

pytestmark = pytest.mark.gpu


def cloud(n, seed, spread, log_scale, sigma, opacity=-1.0):
    rng = np.random.default_rng(seed)
    raw = np.zeros((n, 14), np.float32)
    raw[:, 0:3] = rng.standard_normal((n, 3)) * spread
    raw[:, 3] = opacity + 0.5 * rng.standard_normal(n)
    raw[:, 4:7] = log_scale + sigma * rng.standard_normal((n, 3))
    raw[:, 7:11] = rng.standard_normal((n, 4))
    raw[:, 11:14] = rng.standard_normal((n, 3))
    return L.pack_splats(raw, 0, 0)


def check(rasterizer, packed, width, height, **kw):
    scene = H.Scene("cells", [(packed, np.eye(4), None)], H.camera((0.3, 0.4, 4.0), focal=30.0),
                    H.settings(width, height, **kw))
    ref = scene.oracle_render()
    targets = L.RenderTargets()
    rasterizer.render(scene.camera, scene.gpu_instances(), scene.settings, targets)
    for got, want in ((targets.colour, ref["colour"]), (targets.depth, ref["depth"])):
        got = got.cpu().numpy()
        same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want)) | (got == want)
        assert same.all(), int((~same).sum())


@pytest.mark.parametrize("depth", [0, 1], ids=["mean", "threshold"])
@pytest.mark.parametrize("size", [(1, 1), (3, 5), (16, 16), (17, 15), (19, 35)], ids=str)
@pytest.mark.parametrize("n", [1, 127, 128, 129, 400])
def test_batches_and_ragged_tiles(rasterizer, n, size, depth):
    check(rasterizer, cloud(n, n, 0.3, -2.0, 0.3, opacity=-3.5), *size, depth=depth)


@pytest.mark.parametrize("log_scale,sigma", [(-3.0, 1.5), (-5.5, 0.2), (1.0, 1.0)], ids=["thin", "tiny", "huge"])
def test_shapes(rasterizer, log_scale, sigma):
    check(rasterizer, cloud(4000, 11, 1.0, log_scale, sigma), 203, 157)


@pytest.mark.parametrize("value", [0x7C00, 0xFC00, 0x7E00], ids=["inf", "-inf", "nan"])
def test_colours_that_are_not_finite(rasterizer, value):
    packed = cloud(3000, 5, 0.8, -3.2, 0.4)
    packed.shape[::41, 3] = (packed.shape[::41, 3] & 0xFFFF0000) | value   # the base colour's green
    check(rasterizer, packed, 130, 97)
