"""The per-splat backward writes a warp's gradients as one piece, through the
warp's rows in shared memory: at counts where the last warp or block is part
full, the gradients equal, bit for bit, those of the same splats followed by
splats behind the camera (which fill the last rows and get zeros)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import lucabrtrender_b200 as L

import train_fixtures as TF

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 32, 33, 127, 128, 129, 1000]
NAMES = ("means", "log_scales", "quats", "logits", "sh")
SIZE = 64


def parameters(count, extra):
    """`count` splats, then `extra` far behind the camera that draws them."""
    p = {k: np.ascontiguousarray(v[:count]) for k, v in TF.make_params(1000, 41).items()}
    cam, settings = TF.frame(SIZE, SIZE)
    if extra:
        projection = L.projection_for(cam, SIZE, SIZE)
        forward = np.asarray(projection.world_to_view, np.float64)[2, :3]
        behind = (np.asarray(projection.eye_world, np.float64) - 50.0 * forward).astype(np.float32)
        for k, v in TF.make_params(extra, 42).items():
            if k == "means":
                v = np.tile(behind, (extra, 1))
            p[k] = np.concatenate([p[k], v.astype(p[k].dtype)])
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in p.items()}, cam, settings


def target():
    return torch.from_numpy(np.random.default_rng(7).uniform(0, 1, (SIZE, SIZE, 3)).astype(np.float32)).cuda()


def single(rasterizer, count, extra):
    p, cam, settings = parameters(count, extra)
    for t in p.values():
        t.requires_grad_(True)
    colour, _ = L.rasterize(*(p[k] for k in NAMES), cam, settings, rasterizer)
    L.l1_loss(colour, target(), rasterizer).backward()
    return {k: t.grad.cpu().numpy() for k, t in p.items()}


def batch(rasterizer, count, extra):
    p, cam, settings = parameters(count, extra)
    views = [(cam, target()), (cam, 1.0 - target())]
    grads = L.train_batch(*(p[k] for k in NAMES), views, settings, rasterizer)[3]
    return {k: grads["opacity_logits" if k == "logits" else k].cpu().numpy() for k in NAMES}


@pytest.mark.parametrize("step", [single, batch], ids=["one-view", "batch"])
@pytest.mark.parametrize("count", COUNTS)
def test_part_full_rows_hold_the_same_gradients(rasterizer, step, count):
    plain, padded = step(rasterizer, count, 0), step(rasterizer, count, 200)
    for name in NAMES:
        a, b = plain[name].reshape(count, -1), padded[name].reshape(count + 200, -1)
        assert np.array_equal(a, b[:count]), name
        assert not b[count:].any(), name
    assert plain["sh"].any() or count == 1
