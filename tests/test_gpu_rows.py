"""A frame's pairs made from runs of tiles (frames of at most 256 tiles a side
whose last counts were at least 2^21 pairs and six a splat), against the
oracle bit for bit: the widest and tallest frames that take this form and the
first ones past it, splats from a few tiles (tile masks) to the whole frame
(kept rows, and rows planned again where the first frame's table is too
small), a tile row's runs around the number one block sorts or spreads
(2048), training frames, and frames that outgrow their buffers."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import lucabrtrender_b200 as L
from lucabrtrender_b200 import _abi
import helpers as H
import oracle as ora
import train_fixtures as TF
from test_gpu_blend_cells import cloud
from test_gpu_parity import check_parity

pytestmark = pytest.mark.gpu

MIN_PAIRS, MIN_PER_SPLAT = 1 << 21, 6


def scene(n, width, height, log_scale, sigma=0.5, spread=1.0, eye=(0.2, 0.3, 4.0), opacity=-1.0, focal=24.0):
    return H.Scene("rows", [(cloud(n, n + width, spread, log_scale, sigma, opacity), np.eye(4), None)],
                   H.camera(eye, focal=focal), H.settings(width, height))


def check(sc, rasterizer=None):
    """Twice: the first frame's counts choose the form of the second."""
    r = rasterizer or L.TileRasterizer.create(0)
    try:
        ref = sc.oracle_render()
        assert ref["pairs"] >= MIN_PAIRS and ref["pairs"] >= MIN_PER_SPLAT * ref["slots"], ref["pairs"]
        for _ in range(2):
            check_parity(r, sc, ref)
    finally:
        if rasterizer is None:
            r.close()


@pytest.mark.parametrize("n,width,height", [(4000, 4096, 48), (4000, 4097, 48), (24000, 48, 4096), (24000, 48, 4097),
                                            (1200, 250, 4090)], ids=str)
def test_frame_shapes(n, width, height):
    check(scene(n, width, height, 2.0, 0.3, spread=0.3))


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4097])
def test_runs_in_a_row(n):
    check(scene(n, 1040, 272, 2.0, 0.3, spread=0.3, opacity=-3.0))   # every splat over nearly every tile


@pytest.mark.parametrize("n,log_scale,sigma", [(120000, -3.4, 0.3), (20000, -2.6, 1.2), (3000, 0.0, 1.0)],
                         ids=["masks", "thin", "large"])
def test_splat_sizes(n, log_scale, sigma):
    check(scene(n, 1500, 1100, log_scale, sigma))


def test_training_frames():
    """The forward bit for bit, and the same gradients as the frame made from sorted words."""
    n, width, height = 30000, 800, 640
    p = TF.make_params(n, 3, log_scale_mean=-1.7, log_scale_sigma=0.8)
    cam, settings = TF.frame(width, height)
    target = torch.rand(height, width, 3, generator=torch.Generator().manual_seed(1)).cuda()
    ref = ora.train_render(L.projection_for(cam, width, height).struct(), TF.raw_cloud(p), settings.struct())
    r = L.TileRasterizer.create(0)
    try:
        grads = []
        for _ in range(2):
            t = {k: torch.from_numpy(v).cuda().requires_grad_(True) for k, v in p.items()}
            colour, depth = L.rasterize(t["means"], t["log_scales"], t["quats"], t["logits"], t["sh"], cam, settings, r)
            dbg = r.debug_arrays()
            assert dbg["pairs"].numel() >= max(MIN_PAIRS, MIN_PER_SPLAT * n)
            assert np.array_equal(dbg["ranges"].cpu().numpy().view(np.uint32), ref["ranges"])
            assert np.abs(colour.detach().cpu().numpy() - ref["colour"]).max() <= 1e-5
            assert np.abs(depth.cpu().numpy() - ref["depth"]).max() <= 1e-5
            L.l1_loss(colour, target, r).backward()
            grads.append([v.grad.clone() for v in t.values()])
        # A splat's partials stand in the same order either way, so its sums are the same.
        for a, b in zip(*grads):
            assert torch.equal(a, b)
    finally:
        r.close()


def test_enqueued_frames_that_outgrow_their_buffers():
    """Reported, and the redraw is exact: a far view sizes the buffers, a near one has several times the pairs."""
    far = scene(30000, 1200, 900, -1.9, 0.4, eye=(0.2, 0.3, 6.0))
    near = scene(30000, 1200, 900, -1.9, 0.4, eye=(0.1, 0.2, 2.2))
    r = L.TileRasterizer.create(0)
    try:
        instances, targets = far.gpu_instances(), L.RenderTargets()
        first = r.render(far.camera, instances, far.settings, targets)
        r.render_async(far.camera, instances, far.settings, targets)   # leaves a quarter of the buffers free
        r.settle()
        want = near.oracle_render()
        assert first.pairs >= max(MIN_PAIRS, MIN_PER_SPLAT * first.splats) and want["pairs"] > 2 * first.pairs
        r.render_async(near.camera, instances, near.settings, targets)
        with pytest.raises(L.LrtError):
            r.settle()
        r.render(near.camera, instances, near.settings, targets)
        assert np.array_equal(targets.colour.cpu().numpy().view(np.uint32), want["colour"].view(np.uint32))
    finally:
        r.close()


def test_an_enqueued_training_step_that_outgrows_its_buffer():
    """The step's backward is enqueued over the frame before its counts are
    read: it reports OVERFLOW, and the step run again has the image and the
    gradients of a handle that never overflowed, bit for bit. (A frame cut at
    the buffer's end in tile order would hold emit indices past it.)"""
    n, width, height = 30000, 800, 640
    p = TF.make_params(n, 3, log_scale_mean=-1.7, log_scale_sigma=0.8)
    far, settings = TF.frame(width, height, eye=(0.0, 0.0, 6.0))    # 2.6M pairs
    near, _ = TF.frame(width, height, eye=(0.0, 0.0, 3.0))          # 8.2M
    target = torch.rand(height, width, 3, generator=torch.Generator().manual_seed(2)).cuda()

    def step(r, cam):
        t = {k: torch.from_numpy(v).cuda().requires_grad_(True) for k, v in p.items()}
        colour, _ = L.rasterize(t["means"], t["log_scales"], t["quats"], t["logits"], t["sh"], cam, settings, r)
        L.l1_loss(colour, target, r).backward()
        return [colour.detach()] + [v.grad for v in t.values()]

    r, fresh = L.TileRasterizer.create(0), L.TileRasterizer.create(0)
    try:
        for _ in range(3):   # the first sizes the buffers, the second leaves a quarter free, the third is enqueued
            step(r, far)
        assert r.debug_arrays()["pairs"].numel() >= max(MIN_PAIRS, MIN_PER_SPLAT * n)
        with pytest.raises(L.LrtError) as info:
            step(r, near)
        assert info.value.code == _abi.OVERFLOW
        for a, b in zip(step(r, near), step(fresh, near)):
            assert torch.equal(a, b)
    finally:
        r.close()
        fresh.close()
