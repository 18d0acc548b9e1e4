"""The work a user of the rasteriser has it do, as cases that can be timed.

Scenes have the distributions of the repository's benchmark (`bench.py`,
`oracle/bench_workload.py`): means N(0, spread) per axis, log-scales
N(log_scale, log_scale_sigma), rotations uniform, opacity sigmoid(N(0, 1)),
base colour and harmonics N(0, 0.5) and N(0, 0.05) stored as fp16. Cameras
look at the origin with a 60 degree vertical field of view.

`exact` restates the image formation in 64-bit torch on the device: the
splats' projections, the (24-bit depth key, slot) order, and per pixel the
front-to-back loop with its cuts and its stop, differentiated by autograd for
the training cases.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lucabrtrender_b200 as L
from lucabrtrender_b200.replicas import GradientBucket

REST = {0: 0, 1: 3, 2: 8, 3: 15}   # harmonics per colour above the base, by degree
TILE = 16
# Image sizes of the views of a batch (the benchmark's batched configuration and odd ones).
VIEW_SIZES = [(256, 256), (640, 480), (1280, 720), (1920, 1080), (333, 517), (1001, 563)]


# ---- the cases --------------------------------------------------------------------------

def _frame(name, splats, width, height, **more):
    case = {"name": name, "kind": "frame", "splats": splats, "width": width, "height": height, "degree": 3,
            "spread": 1.0, "log_scale": -4.5, "log_scale_sigma": 0.5, "antialias": True, "linearise": True,
            "threshold_depth": False, "edit": False}
    case.update(more)
    return case


def listed():
    return [
        # The render tests' cloud: a thumbnail or a probe, all launches and waits.
        _frame("frame_3k_250x190", 3000, 250, 190, log_scale=-3.2),
        # A small captured object in a square viewport (the CPU-runnable configuration).
        _frame("frame_100k_512", 100_000, 512, 512),
        # The headline: one frame of a captured scene in full HD.
        _frame("frame_1m_1080p", 1_000_000, 1920, 1080),
        # A close, dense scene at 4K: some 256 million (tile, splat) pairs.
        _frame("frame_6m_4k", 6_000_000, 3840, 2160, spread=2.0, log_scale=-3.5, log_scale_sigma=0.7),
        # A viewer's loop: frames enqueued from a moving camera, settled once; a lower degree, an odd window.
        _frame("enqueued_500k_1279x719", 500_000, 1279, 719, kind="enqueued", degree=2, frames=4,
               linearise=False),
        # Splats, a point cloud's discs and an under layer in one picture, with an edit on the cloud.
        _frame("composite_300k_1366x768", 300_000, 1366, 768, kind="composite", degree=1, points=200_000,
               threshold_depth=True, edit=True),
        # Many cameras of one scene in one call (dataset previews, evaluation).
        _frame("views_1m_x12", 1_000_000, 0, 0, kind="views", views=12),
        # The first steps of a small training run: few splats, an odd image.
        _frame("train_20k_333x217", 20_000, 333, 217, kind="train", storage=False, log_scale=-3.6),
        # A training step at the size captured scenes reach: forward, L1 loss, backward.
        _frame("train_1m_1080p", 1_000_000, 1920, 1080, kind="train", storage=True),
        # A training step over a handful of views in one call.
        _frame("train_views_400k_x6", 400_000, 0, 0, kind="train_views", views=6),
        # Loading a scene: raw PLY records to the packed layout.
        {"name": "decode_1m", "kind": "decode", "splats": 1_000_000, "degree": 3},
        # A far view of a large scene: this frame's cut of the levels of detail, and the frame drawn from it.
        _frame("lod_1m_1080p", 1_000_000, 1920, 1080, kind="lod", threshold=10.0, distance=30.0),
    ]


def _spread_out(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, n):
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "enqueued", "composite", "views", "train", "train", "train_views",
                       "decode", "lod"])
    if kind == "decode":
        return {"kind": kind, "splats": _odd(rng, _spread_out(rng, 1000, 2_000_000)), "degree": rng.randrange(4)}
    many = kind in ("views", "train_views")
    dense = rng.random() < 0.25
    most = 600_000 if many or dense else 2_000_000
    height = _odd(rng, _spread_out(rng, 96, 1440))
    width = _odd(rng, max(64, int(height * rng.uniform(0.7, 2.0))))
    case = _frame("", _odd(rng, _spread_out(rng, 2000, most)), 0 if many else width, 0 if many else height, kind=kind)
    del case["name"]
    case["degree"] = 3 if kind in ("train", "train_views") else rng.randrange(4)
    case["antialias"] = rng.random() < 0.8
    case["linearise"] = rng.random() < 0.8
    case["threshold_depth"] = rng.random() < 0.25
    if dense:
        case.update(spread=2.0, log_scale=-3.6, log_scale_sigma=0.7)
    if kind == "lod":
        case["threshold"], case["distance"] = round(rng.uniform(0.0, 40.0), 2), round(rng.uniform(6.0, 40.0), 2)
    if kind == "enqueued":
        case["frames"] = rng.randrange(2, 6)
    if kind == "composite":
        case["points"] = _spread_out(rng, 1000, 500_000)
    if kind in ("frame", "composite"):
        case["edit"] = rng.random() < 0.2
    if many:
        case["views"] = rng.randrange(2, 9)
    if kind == "train":
        case["storage"] = rng.random() < 0.5
    return case


# ---- inputs ------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (int(seed) + 1))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _parameters(case, g):
    """fp32 splat parameters: means, log-scales, quaternions (w, x, y, z), opacity logits, harmonics [N, 16, 3]."""
    n = case["splats"]
    sh = _normal(g, n, 16, 3) * 0.05
    sh[:, 0] *= 10.0
    return {"means": _normal(g, n, 3) * case.get("spread", 1.0),
            "log_scales": _normal(g, n, 3) * case.get("log_scale_sigma", 0.5) + case.get("log_scale", -4.5),
            "quats": _normal(g, n, 4), "logits": _normal(g, n), "sh": sh}


def _halves(low, high):
    """Two float tensors as the fp16 halves of an int32 word, the first in the low half."""
    lo = low.half().view(torch.int16).int() & 0xFFFF
    hi = high.half().view(torch.int16).int() & 0xFFFF
    return lo | (hi << 16)


def _pack(p, degree):
    """The packed cloud: positions (x, y, z, opacity); four words (rotation as the smallest three of the quaternion in
    10 bits each and the largest's index; fp16 log-scales and base colour); fp16 harmonics."""
    n = p["means"].shape[0]
    q = p["quats"][:, [1, 2, 3, 0]]
    q = q / q.norm(dim=1, keepdim=True)
    largest = q.abs().argmax(dim=1)
    q = q * torch.sign(q.gather(1, largest[:, None]))
    others = torch.tensor([[1, 2, 3], [0, 2, 3], [0, 1, 3], [0, 1, 2]], device="cuda")[largest]
    small = (q.gather(1, others) * math.sqrt(0.5) + 0.5).clamp(0, 1).mul(1023.0).round().int()
    rotation = (small[:, 0] << 22) | (small[:, 1] << 12) | (small[:, 2] << 2) | largest.int()
    ls, base = p["log_scales"], 0.5 + 0.28209479177387814 * p["sh"][:, 0]
    shape = torch.stack([rotation, _halves(ls[:, 0], ls[:, 1]), _halves(ls[:, 2], base[:, 0]),
                         _halves(base[:, 1], base[:, 2])], dim=1).contiguous()
    rest = p["sh"][:, 1:1 + REST[degree]].reshape(n, -1)
    if rest.shape[1] % 2 or rest.shape[1] == 0:
        rest = torch.cat([rest, rest.new_zeros(n, 2 if rest.shape[1] == 0 else 1)], dim=1)
    sh = _halves(rest[:, 0::2], rest[:, 1::2]).contiguous()
    positions = torch.cat([p["means"], torch.sigmoid(p["logits"])[:, None]], dim=1).contiguous()
    return positions, shape, sh


def _camera(eye, width, height):
    """A pinhole Projection looking at the origin: view x right, y up, z forward."""
    eye = np.asarray(eye, np.float64)
    forward = -eye / np.linalg.norm(eye)
    right = np.cross(forward, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, forward)
    m = np.eye(4)
    for row, axis in enumerate((right, up, forward)):
        m[row, :3], m[row, 3] = axis, -axis @ eye
    focal = height / 2.0 / math.tan(math.radians(30.0))
    return L.Projection(m, focal, focal, width / 2.0, height / 2.0, 0.01, 10000.0, False, eye)


def _eye(seed, k=0, radius=4.0):
    a = 0.7 * seed + 0.31 * k
    return (radius * math.sin(a), 0.35 * radius * math.sin(1.3 * a + k), radius * math.cos(a))


def _edit(case):
    if not case.get("edit"):
        return L.SplatEdit()
    return L.SplatEdit(active=True, shape=L.EditShape.SPHERE, mode=L.EditMode.GRADE, size=(1.0, 1.0, 1.0),
                       tint=(1.0, 0.8, 0.6), saturation=0.5, brightness=1.2, opacity=0.7)


def _settings(case, width, height):
    return L.RenderSettings(width=width, height=height, antialias=case["antialias"], linearise=case["linearise"],
                            depth=L.Depth.THRESHOLD if case["threshold_depth"] else L.Depth.MEAN)


def _views(case, seed):
    sizes = [VIEW_SIZES[(3 + 5 * k + k // 6) % len(VIEW_SIZES)] for k in range(case["views"])]
    return [(_camera(_eye(seed, k, 3.0 + (k % 4)), w, h), w, h) for k, (w, h) in enumerate(sizes)]


def _under_layer(g, width, height):
    """An opaque layer behind part of the picture: colour, and depth (0 where there is none)."""
    x = torch.linspace(0, 1, width, device="cuda").expand(height, width)
    y = torch.linspace(0, 1, height, device="cuda")[:, None].expand(height, width)
    shift = float(torch.rand((), generator=g, device="cuda"))
    depth = torch.where((x + shift) % 1.0 < 0.5, 3.5 + y, torch.zeros_like(x)).contiguous()
    colour = torch.stack([x, y, 1.0 - x, torch.ones_like(x)], dim=2).contiguous()
    return colour, depth


def _raw_records(case, g):
    """3DGS PLY records: x y z, logit, 3 log-scales, quaternion w x y z, base triple, harmonics red, green, blue."""
    p = _parameters(case, g)
    rest = p["sh"][:, 1:1 + REST[case["degree"]]].transpose(1, 2).reshape(case["splats"], -1)
    return torch.cat([p["means"], p["logits"][:, None], p["log_scales"], p["quats"], p["sh"][:, 0], rest],
                     dim=1).contiguous()


class State:
    """What a program holds: its handle, its scene on the device, its cameras, its targets."""


def prepare(case, seed):
    g = _generator(seed)
    s = State()
    s.case, s.raster, kind = case, L.TileRasterizer.create(0), case["kind"]
    if kind == "decode":
        s.raw = _raw_records(case, g)
        s.encoding = L.ply_encoding(REST[case["degree"]])
        return s
    p = _parameters(case, g)
    if kind in ("train", "train_views"):
        s.params = {k: v.requires_grad_(kind == "train") for k, v in p.items()}
        s.bucket = GradientBucket(case["splats"], torch.device("cuda", 0))
        s.storage = p["sh"].detach().reshape(case["splats"], 48).half().contiguous() \
            if kind == "train_views" or case["storage"] else None
    else:
        s.cloud = L.GpuSplats(*_pack(p, case["degree"]), REST[case["degree"]])
        s.instances = [L.SplatInstance(s.cloud, edit=_edit(case))]
    if kind == "lod":
        s.lod = L.LodBuilder.create(s.raster).build(s.cloud)
        s.selector = L.CutSelector.create(s.raster)
    if kind in ("views", "train_views"):
        s.views = _views(case, seed)
        s.settings = _settings(case, 16, 16)
        if kind == "train_views":
            s.steps = [(pr, torch.rand(h, w, 3, generator=g, device="cuda")) for pr, w, h in s.views]
        else:
            s.targets = [L.RenderTargets(w, h) for _, w, h in s.views]
        return s
    w, h = case["width"], case["height"]
    s.settings = _settings(case, w, h)
    frames = case.get("frames", 1)
    s.projections = [_camera(_eye(seed, k, case.get("distance", 4.0)), w, h) for k in range(frames)]
    if kind == "train":
        s.target = torch.rand(h, w, 3, generator=g, device="cuda")
        return s
    s.targets = [L.RenderTargets(w, h) for _ in range(frames)]
    if kind == "composite":
        at = torch.cat([_normal(g, case["points"], 3), torch.ones(case["points"], 1, device="cuda")], dim=1)
        rgb = torch.rand(case["points"], 4, generator=g, device="cuda")
        words = torch.stack([_halves(rgb[:, 0], rgb[:, 1]), _halves(rgb[:, 2], torch.ones_like(rgb[:, 3]))], dim=1)
        s.points = [L.PointInstance(L.GpuPoints(at.contiguous(), words.contiguous()),
                                    style=L.PointStyle(size_mode=0, size=0.01))]
        s.under = L.RenderTargets(w, h)
        colour, depth = _under_layer(g, w, h)
        s.under.colour.copy_(colour)
        s.under.depth.copy_(depth)
    return s


# ---- one pass ----------------------------------------------------------------------------

def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "frame":
        stats = s.raster.render(s.projections[0], s.instances, s.settings, s.targets[0])
        return {"colour": s.targets[0].colour, "depth": s.targets[0].depth, "pairs": stats.pairs,
                "visible": stats.visible}
    if kind == "enqueued":
        for projection, targets in zip(s.projections, s.targets):
            s.raster.render_async(projection, s.instances, s.settings, targets)
        stats = s.raster.settle()
        return {"frames": [{"colour": t.colour, "depth": t.depth} for t in s.targets], "pairs": stats.pairs}
    if kind == "composite":
        stats = s.raster.render(s.projections[0], s.instances, s.settings, s.targets[0], points=s.points,
                                under=s.under)
        return {"colour": s.targets[0].colour, "depth": s.targets[0].depth, "pairs": stats.pairs}
    if kind == "views":
        s.raster.render_batch(s.views, s.instances, s.settings, s.targets)
        return {"frames": [{"colour": t.colour, "depth": t.depth} for t in s.targets]}
    if kind == "train":
        p = s.params
        for t in p.values():
            t.grad = None
        colour, depth = L.rasterize(p["means"], p["log_scales"], p["quats"], p["logits"], p["sh"], s.projections[0],
                                    s.settings, s.raster, grad_bucket=s.bucket, sh_storage=s.storage)
        loss = L.l1_loss(colour, s.target, s.raster)
        loss.backward()
        return {"colour": colour.detach(), "depth": depth, "loss": loss.detach(),
                "grads": {k: t.grad for k, t in p.items()}}
    if kind == "train_views":
        p = s.params
        colours, depths, losses, grads, _ = L.train_batch(
            p["means"], p["log_scales"], p["quats"], p["logits"], p["sh"], s.steps, s.settings, s.raster,
            sh_storage=s.storage, grad_bucket=s.bucket)
        grads["logits"] = grads.pop("opacity_logits")
        return {"frames": [{"colour": c, "depth": d} for c, d in zip(colours, depths)], "losses": losses,
                "grads": grads}
    if kind == "decode":
        cloud = s.raster.decode_splats(s.raw, s.encoding, REST[case["degree"]])
        return {"positions": cloud.positions, "shape": cloud.shape, "sh": cloud.sh}
    cut = s.selector.select(s.projections[0], [L.LodInstance(s.lod)], case["threshold"])
    stats = s.raster.render(s.projections[0], cut, s.settings, s.targets[0])
    return {"colour": s.targets[0].colour, "depth": s.targets[0].depth, "drawn": stats.splats, "pairs": stats.pairs}


# ---- what a pass cannot do without ---------------------------------------------------------

def work(case):
    n, kind = case["splats"], case["kind"]
    words = max((REST[case["degree"]] * 3 + 1) // 2, 1)
    packed = n * (32 + 4 * words)
    if kind == "decode":
        return {"bytes": n * 4 * (14 + 3 * REST[case["degree"]]) + packed, "flops": 60 * n}
    if kind in ("views", "train_views"):
        sizes = [(w, h) for _, w, h in _views(case, 0)]
    else:
        sizes = [(case["width"], case["height"])] * case.get("frames", 1)
    pixels = sum(w * h for w, h in sizes)
    train = kind in ("train", "train_views")
    read = n * (44 + 96) if train else packed * (1 if kind == "views" else len(sizes))
    moved = read + 20 * pixels + (n * 236 + 12 * pixels if train else 0)
    if kind == "lod":   # the cells' codes too
        moved += 4 * n
    if kind == "composite":
        moved += 24 * case["points"] + 20 * pixels
    # Per splat and view about 350 operations of projection and colour (three times that with the backward); per
    # pixel some tens of contributing splats of about 40 operations (again three times).
    return {"bytes": moved, "flops": (3 if train else 1) * (350 * n * len(sizes) + 800 * pixels)}


# ---- tolerances ----------------------------------------------------------------------------

def tolerance(case):
    kind = case["kind"]
    if kind == "decode":
        return "exact"   # packed words
    if kind in ("train", "train_views"):
        # Sums over pixels and tiles in fp32 in another order, through the projection's conditioning.
        return {"rel": 3e-5}
    # Images: fp32 sums of some tens of terms; a cut or a stop decided the other way moves a pixel by up to 1/255
    # of a splat's colour.
    return {"rel": 2e-5, "differ": 0.0}


# ---- the same in 64 bits -------------------------------------------------------------------

def _words_to_halves(words):
    lo = (words & 0xFFFF).to(torch.int16).view(torch.float16)
    hi = ((words >> 16) & 0xFFFF).to(torch.int16).view(torch.float16)
    return lo.double(), hi.double()


def _unpack(positions, shape, sh, degree):
    """The packed cloud's parameters in 64 bits: position, opacity, scale, quaternion (x, y, z, w), base, harmonics."""
    word = shape[:, 0].long() & 0xFFFFFFFF
    small = torch.stack([(word >> 22) & 1023, (word >> 12) & 1023, (word >> 2) & 1023], dim=1).double()
    small = (small / 1023.0 * 2.0 - 1.0) * 0.70710678
    rest = (1.0 - small.square().sum(1)).clamp(min=0).sqrt()
    q = torch.empty(len(word), 4, device="cuda", dtype=torch.float64)
    others = torch.tensor([[1, 2, 3], [0, 2, 3], [0, 1, 3], [0, 1, 2]], device="cuda")[word & 3]
    q.scatter_(1, others, small)
    q.scatter_(1, (word & 3)[:, None], rest[:, None])
    a, b = _words_to_halves(shape[:, 1:])
    scale = torch.exp(torch.stack([a[:, 0], b[:, 0], a[:, 1]], dim=1))
    base = torch.stack([b[:, 1], a[:, 2], b[:, 2]], dim=1)
    lo, hi = _words_to_halves(sh)
    k = REST[degree]
    harmonics = torch.stack([lo, hi], dim=2).reshape(len(word), -1)[:, :3 * k].reshape(len(word), k, 3)
    return positions[:, :3], positions[:, 3].double(), scale, q, base, harmonics


def _harmonics(rest, d):
    """The sum of the rest basis functions at unit directions d."""
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    xx, yy, zz = x * x, y * y, z * z
    basis = [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x,
             1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
             -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy),
             -0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
             -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
             -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
             -0.5900435899266435 * x * (xx - 3 * yy)][:rest.shape[1]]
    return (torch.stack(basis, dim=1)[:, :, None] * rest).sum(1) if basis else rest.new_zeros(len(x), 3)


def _to_view(m, p):
    """View coordinates, the depth rounded as 32-bit arithmetic rounds it (the depth key is its bits)."""
    f = torch.tensor(m[:3], device="cuda", dtype=torch.float64).float()
    p32 = p.detach().float()
    z32 = f[2, 0] * p32[:, 0] + f[2, 1] * p32[:, 1] + f[2, 2] * p32[:, 2] + f[2, 3]
    t = p.double() @ f[:, :3].double().T + f[:, 3].double()
    return f.double(), t, z32


def _project(pr, width, height, antialias, p, opacity, scale, q, colour_of):
    """Per splat: centre, depth, conic, alpha, cut, colour; which are visible; the order's key."""
    f, t, z32 = _to_view(pr.world_to_view, p)
    x, y, z, w = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).reshape(-1, 3, 3)
    M = R * scale[:, None, :]
    alive = (z32 > pr.near_z) & (z32 <= pr.far_z)
    fx, fy = float(np.float32(pr.focal_x)), float(np.float32(pr.focal_y))
    tz = torch.where(alive, t[:, 2], torch.ones_like(t[:, 2]))
    u, v = t[:, 0] / tz, t[:, 1] / tz
    cu = u.clamp((-0.15 * width - pr.centre_x) / fx, (1.15 * width - pr.centre_x) / fx)
    cv = v.clamp((-0.15 * height - pr.centre_y) / fy, (1.15 * height - pr.centre_y) / fy)
    zero = torch.zeros_like(tz)
    J = torch.stack([fx / tz, zero, -fx * cu / tz, zero, fy / tz, -fy * cv / tz], dim=1).reshape(-1, 2, 3)
    A = (J @ f[:, :3]) @ M
    S = A @ A.transpose(1, 2)
    before = S[:, 0, 0] * S[:, 1, 1] - S[:, 0, 1] ** 2
    a, b, c = S[:, 0, 0] + 0.3, S[:, 0, 1], S[:, 1, 1] + 0.3
    det = a * c - b * b
    alpha = opacity * (before.clamp(min=0) / det).sqrt() if antialias else opacity
    alive = alive & (det > 1e-12) & (alpha >= 1.0 / 255.0)
    cut = (2 * (255 * alpha).clamp(min=1.0001).log()).clamp(max=9.0)
    d = p.double() - torch.tensor(pr.eye_world, device="cuda").float().double()
    colour = colour_of(d / d.norm(dim=1, keepdim=True)).clamp(min=0)
    rec = torch.stack([fx * u + pr.centre_x, fy * v + pr.centre_y, t[:, 2], c / det, -b / det, a / det, alpha,
                       cut.detach()], dim=1)
    key = z32.contiguous().view(torch.int32).long() >> 7
    return torch.cat([rec, colour], dim=1), alive, key


def _tile_lists(rec, alive, key, width, height):
    """(tile, splat) pairs by tile, then key, then slot, over every tile of each splat's bounding rectangle."""
    with torch.no_grad():
        cx, cy, a, b, c, cut = (rec[:, k] for k in (0, 1, 3, 4, 5, 7))
        det = a * c - b * b
        ex, ey = (cut * c / det).sqrt() + 0.01, (cut * a / det).sqrt() + 0.01
        tx, ty = -(-width // TILE), -(-height // TILE)
        x0, x1 = ((cx - ex) / TILE).floor().clamp(0, tx), ((cx + ex) / TILE).floor().clamp(-1, tx - 1)
        y0, y1 = ((cy - ey) / TILE).floor().clamp(0, ty), ((cy + ey) / TILE).floor().clamp(-1, ty - 1)
        w, h = (x1 - x0 + 1).clamp(min=0), (y1 - y0 + 1).clamp(min=0)
        area = torch.where(alive, w * h, torch.zeros_like(w)).nan_to_num(0).long()
        order = torch.argsort(key, stable=True)
        order = order[area[order] > 0]
        reps = area[order]
        total = int(reps.sum())
        if total > 120_000_000:
            return None
        who = torch.repeat_interleave(order, reps)
        k = torch.arange(total, device="cuda") - torch.repeat_interleave(reps.cumsum(0) - reps, reps)
        ww = w.long()[who]
        tile = (y0.long()[who] + k // ww) * tx + x0.long()[who] + k % ww
        tile, at = torch.sort(tile, stable=True)
        counts = torch.bincount(tile, minlength=tx * ty)
        return who[at], counts, counts.cumsum(0) - counts, tx, ty


def _linear(c):
    c = c.clamp(min=0)
    return torch.where(c <= 0.04045, c / 12.92, ((c.clamp(min=0.04045) + 0.055) / 1.055) ** 2.4)


def _blend(case, rec, disc, lists, width, height, under=None, target=None, order_z=None):
    """Every pixel of every tile in 64 bits: colour, depth, and (with a target) the gradient of the mean absolute
    error with respect to `rec`. Tiles of similar length go together."""
    who, counts, starts, tx, ty = lists
    colour = torch.zeros(ty * TILE, tx * TILE, 4, device="cuda", dtype=torch.float64)
    depth = torch.zeros(ty * TILE, tx * TILE, device="cuda", dtype=torch.float64)
    grad, loss = torch.zeros_like(rec), 0.0
    by_length = torch.argsort(counts).tolist()
    length = counts.tolist()
    px = torch.arange(TILE, device="cuda").repeat(TILE)
    py = torch.arange(TILE, device="cuda").repeat_interleave(TILE)
    at = 0
    budget = 1 << (24 if target is None else 22)
    while at < len(by_length):
        end = at + 1
        while end < len(by_length) and (end + 1 - at) * max(length[by_length[end]], 1) * 256 <= budget:
            end += 1
        tiles = torch.tensor(by_length[at:end], device="cuda")
        most = max(length[by_length[end - 1]], 1)
        at = end
        k = torch.arange(most, device="cuda")
        has = k[None] < counts[tiles][:, None]
        pick = who[(starts[tiles][:, None] + k).clamp(max=max(len(who) - 1, 0))] if len(who) else torch.zeros_like(has).long()
        r = (rec.detach()[pick]).requires_grad_(target is not None)          # [T, K, 11]
        X, Y = (tiles % tx)[:, None] * TILE + px, (tiles // tx)[:, None] * TILE + py
        dx = (X + 0.5)[:, None, :] - r[:, :, 0:1]
        dy = (Y + 0.5)[:, None, :] - r[:, :, 1:2]
        power = r[:, :, 3:4] * dx * dx + 2 * r[:, :, 4:5] * dx * dy + r[:, :, 5:6] * dy * dy
        take = has[:, :, None] & ~(power > r[:, :, 7:8])
        uz = None
        if under is not None:
            ux, uy = X.clamp(max=width - 1), Y.clamp(max=height - 1)
            uz = under[1][uy, ux].double()
            z32 = torch.where(has, order_z[pick], torch.full_like(order_z[pick], -3.0e38)).cummax(1).values
            take = take & ~((uz > 0)[:, None] & (z32.double()[:, :, None] >= uz[:, None]))
        is_disc = take & disc[pick][:, :, None]
        alpha = (r[:, :, 6:7] * torch.exp(-0.5 * power)).clamp(max=0.99)
        part = torch.where(take & ~is_disc & (alpha >= 1.0 / 255.0), alpha, torch.zeros_like(alpha))
        T = torch.cumprod(1 - part, dim=1)
        before = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], dim=1)
        on = before >= 1e-4
        past_disc = torch.cumsum(is_disc.int(), dim=1) - is_disc.int() > 0
        on = on & ~past_disc
        part = torch.where(on & ~is_disc, part, torch.zeros_like(part))
        weight = torch.where(on, before, torch.zeros_like(before)) * part
        final = torch.prod(torch.where(part > 0, 1 - part, torch.ones_like(part)), dim=1)
        rgb = (weight[:, :, :, None] * r[:, :, None, 8:11]).sum(1)
        cover = 1 - final
        if case["linearise"]:
            some = cover > 1e-6
            safe = torch.where(some, cover, torch.ones_like(cover))[..., None]
            rgb = torch.where(some[..., None], _linear(rgb / safe) * safe, rgb)
        behind = torch.zeros(*cover.shape, 4, device="cuda", dtype=torch.float64)
        z = r[:, :, 2:3]
        d_sum = (weight * z).sum(1)
        after = torch.cumprod(1 - part, dim=1)
        reached = (weight > 0) & (1 - after >= 0.5)
        first = torch.where(reached.any(1), reached.int().argmax(1), torch.full_like(tiles, -1)[:, None])
        d_at = torch.where(first >= 0, z[..., 0].gather(1, first.clamp(min=0)), torch.full_like(cover, -1.0))
        hit = (is_disc & on).any(1)
        opaque_z = torch.zeros_like(cover)
        if disc.any():
            h = (is_disc & on).int().argmax(1)
            behind = torch.where(hit[..., None], torch.cat([r[:, :, 8:11], torch.ones_like(z)], dim=2).gather(
                1, h[..., None].expand(-1, -1, 4)), behind)
            opaque_z = torch.where(hit, z[..., 0].gather(1, h), opaque_z)
        if uz is not None:
            layer = ~hit & (uz > 0)
            behind = torch.where(layer[..., None], under[0][uy, ux].double(), behind)
            opaque_z = torch.where(layer, uz, opaque_z)
            hit = hit | layer
        total = torch.where(hit, torch.ones_like(cover), cover)
        d_sum = d_sum + torch.where(hit, final * opaque_z, torch.zeros_like(cover))
        d_at = torch.where(hit & (d_at < 0), opaque_z, d_at)
        out = torch.cat([rgb, cover[..., None]], dim=2) + final[..., None] * behind
        d = d_at.clamp(min=0) if case["threshold_depth"] else torch.where(
            total > 1e-6, d_sum / total.clamp(min=1e-6), torch.zeros_like(total))
        if target is not None:
            inside = ((X < width) & (Y < height))[..., None]
            want = target[Y.clamp(max=height - 1), X.clamp(max=width - 1)].double()
            part_loss = (torch.where(inside, (out[..., :3] - want).abs(), torch.zeros_like(want))).sum() / (
                3.0 * width * height)
            part_loss.backward()
            grad.index_add_(0, pick.reshape(-1), torch.where(has[..., None], r.grad, torch.zeros_like(r)).reshape(-1, rec.shape[1]))
            loss += float(part_loss)
        colour[Y, X], depth[Y, X] = out.detach(), d.detach()
    return colour[:height, :width], depth[:height, :width], loss, grad


def _edited(case, p, opacity, colour):
    """The grade inside the edit's sphere: opacity and colour as the edit makes them, and who it removes."""
    if not case["edit"]:
        return opacity, colour, torch.zeros(len(p), device="cuda", dtype=torch.bool)
    inside = p.float().square().sum(1) <= 1.0
    tint = torch.tensor([1.0, 0.8, 0.6], device="cuda", dtype=torch.float32).double()
    bright = float(np.float32(1.2))

    def graded(d):
        c = colour(d).clamp(min=0)
        t = c * tint * bright
        luma = t @ torch.tensor([0.2126, 0.7152, 0.0722], device="cuda", dtype=torch.float64)
        return torch.where(inside[:, None], (luma[:, None] + (t - luma[:, None]) * 0.5).clamp(min=0), c)

    faded = opacity * float(np.float32(0.7))
    return torch.where(inside, faded, opacity), graded, inside & (faded < 1.0 / 255.0)


def _points_records(g, case, pr, width, height):
    at = _normal(g, case["points"], 3)
    rgb = torch.rand(case["points"], 4, generator=g, device="cuda")[:, :3].half().double()
    _, t, z32 = _to_view(pr.world_to_view, at)
    alive = (z32 > pr.near_z) & (z32 <= pr.far_z)
    tz = torch.where(alive, t[:, 2], torch.ones_like(t[:, 2]))
    radius = (0.005 * pr.focal_x / tz).clamp(min=0.5)
    one = torch.ones_like(tz)
    rec = torch.stack([pr.focal_x * t[:, 0] / tz + pr.centre_x, pr.focal_y * t[:, 1] / tz + pr.centre_y, t[:, 2],
                       1 / radius ** 2, 0 * one, 1 / radius ** 2, one, one], dim=1)
    return torch.cat([rec, rgb], dim=1), alive, z32.contiguous().view(torch.int32).long() >> 7, z32


def _exact_frame(case, cloud, pr, width, height, g=None):
    p, opacity, scale, q, base, rest = cloud
    opacity, colour, removed = _edited(case, p, opacity, lambda d: base + _harmonics(rest, d))
    rec, alive, key = _project(pr, width, height, case["antialias"], p, opacity, scale, q, colour)
    alive = alive & ~removed
    disc = torch.zeros(len(rec), device="cuda", dtype=torch.bool)
    under = order_z = None
    if g is not None:
        more, more_alive, more_key, more_z = _points_records(g, case, pr, width, height)
        order_z = torch.cat([_to_view(pr.world_to_view, p)[2], more_z])
        rec, alive, key = torch.cat([rec, more]), torch.cat([alive, more_alive]), torch.cat([key, more_key])
        disc = torch.cat([disc, torch.ones(len(more), device="cuda", dtype=torch.bool)])
        under = _under_layer(g, width, height)
    lists = _tile_lists(rec, alive, key, width, height)
    if lists is None:
        return None
    image, depth, _, _ = _blend(case, rec, disc, lists, width, height, under, None, order_z)
    return {"colour": image, "depth": depth}


def _exact_train(case, leaves, views):
    """Colours, depths, losses and the gradients of their sum; `views`: (projection, target)."""
    p64 = {k: (v.half().double() if k == "sh" else v.double()).requires_grad_(True) for k, v in leaves.items()}
    q = p64["quats"] / p64["quats"].norm(dim=1, keepdim=True)
    frames, losses = [], []
    for pr, target in views:
        h, w = target.shape[:2]
        rec, alive, key = _project(pr, w, h, case["antialias"], p64["means"], torch.sigmoid(p64["logits"]),
                                   p64["log_scales"].exp(), q[:, [1, 2, 3, 0]],
                                   lambda d: 0.5 + 0.28209479177387814 * p64["sh"][:, 0] + _harmonics(p64["sh"][:, 1:], d))
        lists = _tile_lists(rec, alive, key, w, h)
        if lists is None:
            return None
        disc = torch.zeros(len(rec), device="cuda", dtype=torch.bool)
        image, depth, loss, grad = _blend(case, rec, disc, lists, w, h, None, target)
        good = alive[:, None] & torch.isfinite(grad)
        torch.where(good, rec * grad.detach().nan_to_num(0.0), torch.zeros_like(rec)).sum().backward(retain_graph=True)
        frames.append({"colour": image, "depth": depth})
        losses.append(loss)
    return frames, losses, {k: v.grad for k, v in p64.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        return None   # packed words: no computed sums
    if kind == "lod":
        return None   # a million splats' moments, cell by cell down ten levels, takes minutes
    if kind in ("train", "train_views") and case["splats"] > 250_000:
        return None   # autograd over every (pixel, splat) pair would take minutes
    g = _generator(seed)
    p = _parameters(case, g)
    if kind == "train":
        w, h = case["width"], case["height"]
        got = _exact_train(case, p, [(_camera(_eye(seed), w, h), torch.rand(h, w, 3, generator=g, device="cuda"))])
        return got and {"colour": got[0][0]["colour"], "depth": got[0][0]["depth"],
                        "loss": torch.tensor(got[1][0], dtype=torch.float64), "grads": got[2]}
    if kind == "train_views":
        got = _exact_train(case, p, [(pr, torch.rand(h, w, 3, generator=g, device="cuda"))
                                     for pr, w, h in _views(case, seed)])
        return got and {"frames": got[0], "losses": torch.tensor(got[1], dtype=torch.float64), "grads": got[2]}
    cloud = _unpack(*_pack(p, case["degree"]), case["degree"])
    if kind == "views":
        frames = [_exact_frame(case, cloud, pr, w, h) for pr, w, h in _views(case, seed)]
        return None if any(f is None for f in frames) else {"frames": frames}
    w, h = case["width"], case["height"]
    frames = [_exact_frame(case, cloud, _camera(_eye(seed, k), w, h), w, h, g if kind == "composite" else None)
              for k in range(case.get("frames", 1))]
    if any(f is None for f in frames):
        return None
    if kind == "enqueued":
        return {"frames": frames, "pairs": None}
    return {**frames[0], "pairs": None, "visible": None} if kind == "frame" else {**frames[0], "pairs": None}
