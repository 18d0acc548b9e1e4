"""A frame's pairs made from runs of tiles (frames of at most 256 tiles a side
whose last counts were at least 2^21 pairs and six a splat), against the
oracle bit for bit: the widest and tallest frames that take this form and the
first ones past it, splats from a few tiles (tile masks) to the whole frame
(kept rows, and rows planned again where the first frame's table is too
small), a tile row's runs around the number one block sorts or spreads
(2048), training frames, frames that outgrow their buffers or have more runs
than pairs, and every kind of frame that takes this form."""
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
from test_gpu_points import check_frame

pytestmark = pytest.mark.gpu

MIN_PAIRS, MIN_PER_SPLAT, MAX_SIDE = 1 << 21, 6, 4096


def scene(n, width, height, log_scale, sigma=0.5, spread=1.0, eye=(0.2, 0.3, 4.0), opacity=-1.0, focal=24.0):
    return H.Scene("rows", [(cloud(n, n + width, spread, log_scale, sigma, opacity), np.eye(4), None)],
                   H.camera(eye, focal=focal), H.settings(width, height))


def check(sc):
    """Twice: the first frame's pairs do not fit the buffer of a fresh handle,
    and it is drawn again in the form its counts choose; the second's form is
    known before it starts."""
    r = L.TileRasterizer.create(0)
    try:
        ref = sc.oracle_render()
        assert ref["pairs"] >= MIN_PAIRS and ref["pairs"] >= MIN_PER_SPLAT * ref["slots"], ref["pairs"]
        for _ in range(2):
            dbg = check_parity(r, sc, ref)[2]
            assert dbg["from_runs"] == (max(sc.settings.width, sc.settings.height) <= MAX_SIDE)
    finally:
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


def words_handle(n, pairs, width, height):
    """A handle whose next frame of n splats is made from sorted words: its
    buffer holds as many pairs, and the last frame it read was of fewer splats."""
    tiles = -(-width // 16) * -(-height // 16)
    k = -(-pairs // tiles) + 1
    assert k != n
    r = L.TileRasterizer.create(0)
    sc = scene(k, width, height, 3.0, 0.1, spread=0.1)   # every splat over every tile
    assert r.render(sc.camera, sc.gpu_instances(), sc.settings, L.RenderTargets()).pairs >= pairs
    return r


def test_training_frames():
    """The forward against the oracle from both forms, and the same gradients."""
    n, width, height = 30000, 800, 640
    p = TF.make_params(n, 3, log_scale_mean=-1.7, log_scale_sigma=0.8)
    cam, settings = TF.frame(width, height)
    target = torch.rand(height, width, 3, generator=torch.Generator().manual_seed(1)).cuda()
    ref = ora.train_render(L.projection_for(cam, width, height).struct(), TF.raw_cloud(p), settings.struct())
    r = words_handle(n, 8_000_000, width, height)
    try:
        grads = []
        for from_runs in (False, False, True):   # words; words, their runs counted; runs
            t = {k: torch.from_numpy(v).cuda().requires_grad_(True) for k, v in p.items()}
            colour, depth = L.rasterize(t["means"], t["log_scales"], t["quats"], t["logits"], t["sh"], cam, settings, r)
            dbg = r.debug_arrays()
            assert dbg["pairs"].numel() >= max(MIN_PAIRS, MIN_PER_SPLAT * n) and dbg["from_runs"] == from_runs
            assert np.array_equal(dbg["ranges"].cpu().numpy().view(np.uint32), ref["ranges"])
            assert np.abs(colour.detach().cpu().numpy() - ref["colour"]).max() <= 1e-5
            assert np.abs(depth.cpu().numpy() - ref["depth"]).max() <= 1e-5
            L.l1_loss(colour, target, r).backward()
            grads.append([v.grad.clone() for v in t.values()])
        # A splat's partials stand in the same order either way, so its sums are the same.
        for a, *others in zip(*grads):
            assert all(torch.equal(a, b) for b in others)
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
        assert r.debug_view().from_runs
        r.render_async(near.camera, instances, near.settings, targets)
        with pytest.raises(L.LrtError):
            r.settle()
        r.render(near.camera, instances, near.settings, targets)
        assert r.debug_view().from_runs
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
        dbg = r.debug_arrays()
        assert dbg["pairs"].numel() >= max(MIN_PAIRS, MIN_PER_SPLAT * n) and dbg["from_runs"]
        with pytest.raises(L.LrtError) as info:
            step(r, near)
        assert info.value.code == _abi.OVERFLOW
        for a, b in zip(step(r, near), step(fresh, near)):
            assert torch.equal(a, b)
    finally:
        r.close()
        fresh.close()


# Faint needles thousands of pixels long. A row of tiles of which such a splat
# touches some with a gap between them makes it a run for every tile of its
# rectangle: these have 2.3M pairs or more, and several runs for each.
NEEDLES, NEEDLE_PAIRS, NEEDLE_SIZE = 100_000, 6_000_000, (3840, 2160)


def needle_arrays(n=NEEDLES):
    rng = np.random.default_rng(1)
    log_scales = np.full((n, 3), -9.0, np.float32)
    log_scales[:, 0] = 2.0 + 0.3 * rng.standard_normal(n)
    return (0.5 * rng.standard_normal((n, 3))).astype(np.float32), log_scales, \
        rng.standard_normal((n, 4)).astype(np.float32), rng.uniform(-5.5, -5.4, n).astype(np.float32)


def needles():
    means, log_scales, quats, logits = needle_arrays()
    raw = np.zeros((NEEDLES, 14), np.float32)
    raw[:, 0:3], raw[:, 3], raw[:, 4:7], raw[:, 7:11], raw[:, 11:14] = means, logits, log_scales, quats, means
    return H.Scene("needles", [(L.pack_splats(raw, 0, 0), np.eye(4), None)], H.camera((0.2, 0.3, 2.5), focal=24.0),
                   H.settings(*NEEDLE_SIZE))


def blobs():
    """As many splats, of 2^21 pairs and six a splat too, but fewer runs than pairs."""
    return scene(NEEDLES, *NEEDLE_SIZE, -4.2, 0.3)


def draw(r, sc):
    t = L.RenderTargets()
    stats = r.render(sc.camera, sc.gpu_instances(), sc.settings, t)
    assert stats.pairs >= max(MIN_PAIRS, MIN_PER_SPLAT * NEEDLES) and stats.pairs <= NEEDLE_PAIRS, stats.pairs
    return t.colour.clone(), t.depth.clone(), bool(r.debug_view().from_runs)


def test_frames_of_more_runs_than_pairs():
    """Drawn from sorted words, whether the runs are met with a wait (they do
    not fit, on the second attempt) or in an enqueued frame that counts them
    first; one enqueued after a frame that fitted is reported, and drawn again."""
    sc, fits = needles(), blobs()
    r, words = L.TileRasterizer.create(0), words_handle(NEEDLES, NEEDLE_PAIRS, *NEEDLE_SIZE)
    other = L.TileRasterizer.create(0)
    try:
        want_colour, want_depth, from_runs = draw(words, sc)
        assert not from_runs and float(want_colour.abs().max()) > 0.0
        for _ in range(2):   # runs unknown, then known
            colour, depth, from_runs = draw(r, sc)
            assert not from_runs
            assert torch.equal(colour, want_colour) and torch.equal(depth, want_depth)
        assert draw(other, fits)[2]
        for handle, overflows in ((words, False), (other, True)):   # both forms' counts of the frame before
            t = L.RenderTargets(*NEEDLE_SIZE)
            instances = sc.gpu_instances()
            if overflows:
                fit_instances = fits.gpu_instances()
                handle.render_async(fits.camera, fit_instances, fits.settings, t)
                handle.settle()
                handle.render_async(sc.camera, instances, sc.settings, t)
                with pytest.raises(L.LrtError) as info:
                    handle.settle()
                assert info.value.code == _abi.OVERFLOW
            for _ in range(3):
                handle.render_async(sc.camera, instances, sc.settings, t)
                handle.settle()
                assert torch.equal(t.colour, want_colour) and torch.equal(t.depth, want_depth)
    finally:
        for handle in (r, words, other):
            handle.close()


def test_training_steps_of_more_runs_than_pairs():
    """The same in training steps: a waited one, and one enqueued after a step
    whose runs fitted, which is reported by its backward."""
    means, log_scales, quats, logits = needle_arrays()
    sh = np.random.default_rng(2).uniform(-0.5, 0.5, (NEEDLES, 16, 3)).astype(np.float16).astype(np.float32)
    thin = dict(means=means, log_scales=log_scales, quats=quats, logits=logits, sh=sh)
    wide = dict(thin, log_scales=np.full_like(log_scales, -4.4), logits=np.full_like(logits, -1.0))
    cam, settings = TF.frame(*NEEDLE_SIZE, eye=(0.2, 0.3, 1.6))
    target = torch.rand(NEEDLE_SIZE[1], NEEDLE_SIZE[0], 3, generator=torch.Generator().manual_seed(3)).cuda()

    def step(r, p):
        t = {k: torch.from_numpy(v).cuda().requires_grad_(True) for k, v in p.items()}
        colour, _ = L.rasterize(t["means"], t["log_scales"], t["quats"], t["logits"], t["sh"], cam, settings, r)
        L.l1_loss(colour, target, r).backward()
        return [colour.detach()] + [v.grad for v in t.values()], bool(r.debug_view().from_runs)

    r, words = L.TileRasterizer.create(0), words_handle(NEEDLES, NEEDLE_PAIRS, *NEEDLE_SIZE)
    waited = L.TileRasterizer.create(0)
    try:
        want, from_runs = step(words, thin)
        assert not from_runs and float(want[0].abs().max()) > 0.0
        for _ in range(2):
            got, from_runs = step(waited, thin)
            assert not from_runs
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        for _ in range(3):
            assert step(r, wide)[1]
        with pytest.raises(L.LrtError) as info:
            step(r, thin)
        assert info.value.code == _abi.OVERFLOW
        got, from_runs = step(r, thin)
        assert not from_runs
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    finally:
        for handle in (r, words, waited):
            handle.close()


@pytest.mark.parametrize("kind", ["instances", "edit", "threshold", "orthographic", "discs", "discs-under"])
def test_other_frames(kind):
    """What a frame may hold besides one cloud seen in perspective, against the
    oracle, bit for bit: instances, an edit, the threshold depth, a parallel
    projection, discs, and a layer under the splats."""
    sc = scene(20000, 1200, 900, -2.5, 0.8)
    packed = sc.clouds[0][0]
    if kind == "instances":
        sc.clouds.append((cloud(7000, 3, 0.7, -2.0, 0.5), H.translation((0.4, -0.2, 0.5)) @ H.rotation_y(35.0), None))
    elif kind == "edit":
        edit = L.SplatEdit(active=True, centre=(0.1, 0.0, 0.2), size=(1.5, 1.2, 1.4), tint=(1.0, 0.6, 0.3),
                           opacity=0.7, brightness=1.2)
        sc.clouds[0] = (packed, np.eye(4), edit)
    elif kind == "threshold":
        sc.settings.depth = L.Depth(1)
    elif kind == "orthographic":
        sc.camera = H.camera((0.2, 0.3, 4.0), focal=7.0, orthographic=True)
    pr, style = sc.projection(), L.PointStyle(size_mode=1, size=40.0)
    packed_points = L.pack_points(ora.random_points(2000, 6), 2)
    points = [L.PointInstance(L.points_to_device(packed_points), np.eye(4), style)] if "discs" in kind else []
    host_points = [(ora.HostPoints(packed_points.positions, packed_points.colours), np.eye(4),
                    H.point_style(1, 40.0))] if points else []
    under = under_host = None
    if "under" in kind:
        under = L.RenderTargets(sc.settings.width, sc.settings.height)
        gen = torch.Generator().manual_seed(4)
        shape = (sc.settings.height, sc.settings.width)
        under.colour.copy_(torch.rand((*shape, 4), generator=gen))
        depth = 2.0 + 4.0 * torch.rand(shape, generator=gen)
        under.depth.copy_(torch.where(torch.rand(shape, generator=gen) < 0.3, torch.zeros(shape), depth))
        under_host = (under.colour.cpu().numpy(), under.depth.cpu().numpy())
    ref = ora.render(pr.struct(), sc.oracle_instances(), sc.settings.struct(), points=host_points, under=under_host)
    assert ref["pairs"] >= MIN_PAIRS and ref["pairs"] >= MIN_PER_SPLAT * ref["slots"], (ref["pairs"], ref["slots"])
    r, targets, instances = L.TileRasterizer.create(0), L.RenderTargets(), sc.gpu_instances()
    try:
        for _ in range(2):
            out = r.render(pr, instances, sc.settings, targets, points=points, under=under)
            check_frame(r, out, ref, targets)
            assert r.debug_view().from_runs
    finally:
        r.close()


def test_frames_of_more_than_a_run_for_two_pairs():
    """Upright needles, nearly a run a pair: a fresh handle's first frame meets
    their runs as it is drawn again, and the frames after it take words."""
    n, rng = 120000, np.random.default_rng(8)
    raw = np.zeros((n, 14), np.float32)
    raw[:, 0:3] = 0.7 * rng.standard_normal((n, 3))
    raw[:, 4:7] = -6.5
    raw[:, 4] = -2.0 + 0.3 * rng.standard_normal(n)
    half = 0.5 * (np.pi / 2 + 0.03 * rng.standard_normal(n))
    raw[:, 7], raw[:, 10] = np.cos(half), np.sin(half)
    raw[:, 11:14] = rng.standard_normal((n, 3))
    sc = H.Scene("upright", [(L.pack_splats(raw, 0, 0), np.eye(4), None)], H.camera((0.2, 0.3, 4.0), focal=24.0),
                 H.settings(1500, 1100))
    ref = sc.oracle_render()
    assert ref["pairs"] >= MIN_PAIRS and ref["pairs"] >= MIN_PER_SPLAT * ref["slots"], ref["pairs"]
    r = L.TileRasterizer.create(0)
    try:
        for from_runs in (True, False, False):
            assert check_parity(r, sc, ref)[2]["from_runs"] == from_runs
    finally:
        r.close()
