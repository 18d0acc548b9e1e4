"""Launches whose shared memory goes past the limit a kernel has unasked. The
limit belongs to the process: frames of different widths on two threads, rows
of harmonics from the usual 23 words to far longer, padded ones, and records
from the usual 59 floats to more than a block stages."""
from __future__ import annotations

import dataclasses
import threading

import pytest
import torch

import lucabrtrender_b200 as L
import helpers as H
from test_gpu_rows import scene

pytestmark = pytest.mark.gpu


def test_two_handles_of_different_widths_on_two_threads():
    """Each draws what it draws alone: the shared memory a launch may take is
    the process's, and one thread's frame is six times as wide as the other's."""
    scenes = [scene(20000, 640, 480, 0.5, 0.3), scene(4000, 3840, 96, 2.0, 0.3, spread=0.3)]
    handles = [L.TileRasterizer.create(0) for _ in scenes]
    streams = [torch.cuda.Stream() for _ in scenes]
    frames = [(sc.gpu_instances(), L.RenderTargets()) for sc in scenes]
    try:
        want = []
        for r, sc, (instances, t) in zip(handles, scenes, frames):
            for _ in range(2):
                r.render(sc.camera, instances, sc.settings, t)
            assert r.debug_view().from_runs
            want.append((t.colour.clone(), t.depth.clone()))
        torch.cuda.synchronize()
        start, failures = threading.Barrier(len(scenes)), []

        def work(k):
            try:
                start.wait()
                for _ in range(200):
                    handles[k].render(scenes[k].camera, frames[k][0], scenes[k].settings, frames[k][1], streams[k])
            except Exception as e:   # noqa: BLE001  (shown below)
                failures.append(e)

        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(scenes))]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        torch.cuda.synchronize()
        assert not failures, failures
        for (_, t), (colour, depth) in zip(frames, want):
            assert torch.equal(t.colour, colour) and torch.equal(t.depth, depth)
    finally:
        for r in handles:
            r.close()


@pytest.mark.parametrize("words", [24, 25, 64, 200])
def test_padded_rows_of_harmonics(rasterizer, words):
    """sh_words past what the degree needs: staged whole, the image the same."""
    sc = H.synthetic_scene(3000, 200, 120, seed=5)
    (instance,) = sc.gpu_instances()
    assert instance.splats.sh.shape[1] == 23
    sh = torch.full((instance.splats.count, words), -1, dtype=instance.splats.sh.dtype, device="cuda")
    sh[:, :23] = instance.splats.sh
    padded = dataclasses.replace(instance, splats=dataclasses.replace(instance.splats, sh=sh))
    images = []
    for one in (instance, padded):
        t = L.RenderTargets()
        rasterizer.render(sc.camera, [one], sc.settings, t)
        images.append((t.colour.clone(), t.depth.clone()))
    assert torch.equal(images[0][0], images[1][0]) and torch.equal(images[0][1], images[1][1])
    assert float(images[0][0].abs().max()) > 0.0


@pytest.mark.parametrize("floats", [60, 93, 94, 95, 96, 320, 321])
def test_padded_records(rasterizer, floats):
    """Records decoded on the device: 128 of them are staged up to 160 KB (320 floats each)."""
    raw = torch.from_numpy(L.synthetic_records(1000, 6)).cuda()
    assert raw.shape[1] == 59
    padded = torch.full((raw.shape[0], floats), 1e30, device="cuda")
    padded[:, :59] = raw
    encoding = L.ply_encoding(15)
    want = rasterizer.decode_splats(raw, encoding, 15)
    encoding.floats_per_record = floats
    got = rasterizer.decode_splats(padded, encoding, 15)
    for name in ("positions", "shape", "sh"):
        assert torch.equal(getattr(got, name).view(torch.int32), getattr(want, name).view(torch.int32)), name
