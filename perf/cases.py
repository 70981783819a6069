"""The work a program gives this library, as cases to time.

Every case is one pass through the public entry points of `voxelg_b200`: a
primary frame, a frame delivered to host memory, a batch of generic rays, the
mixed ray queue, picking, an edited and gated frame, a streamed window, the
learned form of a frame, a training step of its network.  Sizes are those of
the benchmark workloads (the c1 and c2 worlds, 640x360 and 1920x1080 frames,
requests of 1 to 50,000 rays, batches of 16,384 samples) and odd ones beside
them.

Records and masks come back as 32-bit words: hit records are exact, so they are
compared bit for bit.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import voxelg_b200 as vg
from voxelg_b200 import _lib as L
from voxelg_b200 import learned, queue

DEVICE = torch.device("cuda", 0)

PLAIN = L.VX_F_L4
LUT_LOD = L.VX_F_L4 | L.VX_F_LUT | L.VX_F_LOD
FULL = L.VX_F_METHOD | L.VX_F_SHADOW

# an MLP gradient's floats, by tensor: (name, first, shape)
MLP_TENSORS = (("w1", (64, 80)), ("b1", (64,)), ("w2", (64, 64)), ("b2", (64,)),
               ("w3", (64, 64)), ("b3", (64,)), ("wo", (64,)), ("bo", (1,)))


def listed():
    return [
        # the smallest frame that is in use: the c1 workload, plain hierarchical DDA
        {"name": "frame 640x360 plain", "op": "frame", "bx": 128, "bz": 128, "width": 640,
         "height": 360, "flags": PLAIN, "origin_x": 0, "origin_z": 0, "jitter": False},
        # the c2 workload, the library's headline: beam, LUT, LOD and a shadow ray per hit
        {"name": "frame 1080p full", "op": "frame", "bx": 512, "bz": 512, "width": 1920,
         "height": 1080, "flags": FULL, "origin_x": 0, "origin_z": 0, "jitter": False},
        # a large frame of odd size over a window that is no power of two and has been
        # streamed away from the origin, with temporal jitter
        {"name": "frame 3839x2157 streamed", "op": "frame", "bx": 320, "bz": 192, "width": 3839,
         "height": 2157, "flags": FULL, "origin_x": 416, "origin_z": -1184, "jitter": True},
        # the c2 frame for a program that reads its records on the host
        {"name": "host frame 1080p", "op": "host_frame", "bx": 512, "bz": 512, "width": 1920,
         "height": 1080, "flags": FULL},
        # one request of the serving load at its upper size: first-hit, line-of-sight and
        # physics rays of 8 to 512 voxels
        {"name": "trace 50000 rays", "op": "trace", "rays": 50000},
        # the mixed queue: a 1080p frame's primaries and shadows, GI probes and picks, shuffled
        {"name": "queue 1080p mixed", "op": "queue", "width": 1920, "height": 1080,
         "probe_radius": 256, "picks": 10000},
        # the drop-in raycast() call of the editor: one ray under the cursor
        {"name": "pick 1", "op": "pick_one"},
        # picking rays of many agents at once, as the picking benchmark has them
        {"name": "pick 200000", "op": "pick", "rays": 200000},
        # a game loop's frame after an edit: 1% of the c1 world's bricks per second at 60 Hz,
        # only the screen tiles that they touch (and the rotating refresh) traced again
        {"name": "edited frame 175 bricks", "op": "edit", "bricks": 175, "width": 1920,
         "height": 1080},
        # the loaded window following the player: chunks generated, then a frame of them
        {"name": "streamed window 8x3 chunks", "op": "stream", "bx": 512, "bz": 512, "dx": 8,
         "dz": 3, "width": 1280, "height": 720},
        # the learned form of the plain 1080p frame
        {"name": "learned frame 1080p", "op": "learned", "width": 1920, "height": 1080},
        # a training step of the proposal network: loss and gradient of one default batch
        {"name": "gradient 16384", "op": "grad", "batch": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["frame", "frame", "frame", "host_frame", "trace", "queue", "pick", "edit",
                     "stream", "learned", "grad"])
    if op == "frame":
        # any size from the smallest listed to the largest, any method in use
        bx, bz = rng.choice([64, 128, 192, 320, 512]), rng.choice([64, 128, 192, 320, 512])
        height = _log(rng, 360, 2100)
        return {"op": op, "bx": bx, "bz": bz, "width": int(height * rng.uniform(1.25, 1.8)),
                "height": height, "flags": rng.choice([PLAIN, LUT_LOD, LUT_LOD | L.VX_F_BEAM,
                                                       FULL, FULL]),
                "origin_x": 32 * rng.randint(-50, 50), "origin_z": 32 * rng.randint(-50, 50),
                "jitter": rng.random() < 0.5}
    if op == "host_frame":
        height = _log(rng, 360, 1080)
        return {"op": op, "bx": rng.choice([128, 320, 512]), "bz": rng.choice([128, 192, 512]),
                "width": int(height * rng.uniform(1.25, 1.78)), "height": height,
                "flags": rng.choice([LUT_LOD, FULL])}
    if op == "trace":
        return {"op": op, "rays": _log(rng, 1000, 2000000)}
    if op == "queue":
        height = _log(rng, 120, 1080)
        return {"op": op, "width": int(height * rng.uniform(1.25, 1.77)), "height": height,
                "probe_radius": 16 * rng.randint(2, 16), "picks": _log(rng, 100, 10000)}
    if op == "pick":
        return {"op": op, "rays": _log(rng, 1000, 200000)}
    if op == "edit":
        height = _log(rng, 360, 1080)
        return {"op": op, "bricks": _log(rng, 1, 3000),
                "width": int(height * rng.uniform(1.25, 1.77)), "height": height}
    if op == "stream":
        height = _log(rng, 360, 720)
        return {"op": op, "bx": rng.choice([128, 192, 256, 512]),
                "bz": rng.choice([128, 192, 256, 512]), "dx": rng.randint(0, 8),
                "dz": rng.randint(-3, 3) or 1, "width": int(height * rng.uniform(1.25, 1.77)),
                "height": height}
    if op == "learned":
        height = _log(rng, 360, 1080)
        return {"op": op, "width": int(height * rng.uniform(1.25, 1.77)), "height": height}
    return {"op": op, "batch": _log(rng, 500, 16384)}


# ------------------------------------------------------------------ inputs
def _world(bx, bz, seed):
    """A world of the benchmark's terrain: 256 voxels high, its own seed."""
    world = vg.DeviceWorld(bx, 64, bz)
    world.generate(vg.TerrainParams(seed=(seed * 0x9E3779B97F4A7C15 + 0xC0FFEE) % 2**64))
    return world


def _camera(world, rng, width, height, origin=(0, 0, 0), jitter=False):
    """A pose near the window's centre, over the terrain, looking ahead and a little down."""
    vx, _, vz = world.voxels
    pos = (origin[0] + vx / 2 + rng.uniform(-30, 30), rng.uniform(135, 165),
           origin[2] + vz / 2 + rng.uniform(-30, 30))
    cam = vg.camera_from_pose(pos, rng.uniform(0, 2 * math.pi),
                              math.radians(rng.uniform(-20, -10)), math.radians(70.0), width,
                              height, origin)
    if jitter:
        cam.jitter_x, cam.jitter_y = rng.uniform(-0.5, 0.5), rng.uniform(-0.5, 0.5)
    return cam


def _directions(n, gen):
    d = torch.randn((n, 3), generator=gen, device=DEVICE)
    return d / d.norm(dim=1, keepdim=True)


def _rays(org, direction, tmax, kind):
    """RAY_DTYPE rows on the device."""
    r = torch.empty((len(org), 8), dtype=torch.float32, device=DEVICE)
    r[:, 0:3], r[:, 3:6], r[:, 6] = org, direction, tmax
    r.view(torch.int32)[:, 7] = kind
    return r.view(torch.uint8).reshape(-1)


def _trace_rays(world, n, gen):
    """A client's request: origins in the window's air and ground, every direction, lengths
    log-uniform in 8 to 512 voxels; half first hits, the rest line of sight and no-water."""
    size = torch.tensor([float(v) for v in world.voxels], device=DEVICE)
    org = torch.rand((n, 3), generator=gen, device=DEVICE) * size
    length = torch.exp(torch.rand(n, generator=gen, device=DEVICE) * math.log(64.0)) * 8.0
    kind = torch.randint(0, 4, (n,), generator=gen, device=DEVICE, dtype=torch.int32)
    return _rays(org, _directions(n, gen), length, torch.where(kind == 3, 0, kind))


def _queue_rays(world, cam, case, gen):
    """The mixed queue: every primary ray with its shadow, GI probes of 64 directions on a
    16-voxel grid around the camera, picks of 8 voxels, shuffled."""
    w, h = case["width"], case["height"]
    vec = lambda v: torch.tensor(list(v), dtype=torch.float32, device=DEVICE)  # noqa: E731
    x = ((torch.arange(w, device=DEVICE) + 0.5) / w * 2 - 1) * (cam.tan_half_fov * w / h)
    y = (1 - (torch.arange(h, device=DEVICE) + 0.5) / h * 2) * cam.tan_half_fov
    d = (vec(cam.forward) + vec(cam.right) * x[None, :, None]) + vec(cam.up) * y[:, None, None]
    d = (d / d.norm(dim=2, keepdim=True)).reshape(-1, 3)
    eye = vec(cam.origin)
    primary = _rays(eye.expand(len(d), 3), d, 700.0, L.VX_RAY_SPAWN_SHADOW)
    vx, vy, vz = world.voxels
    r = case["probe_radius"]

    def axis(c, n):
        a = torch.arange(int(c) - r, int(c) + r, 16, device=DEVICE)
        return a[(a >= 0) & (a < n)].float() + 8.0

    sites = torch.cartesian_prod(axis(cam.origin[0], vx),
                                 torch.arange(0, vy, 16, device=DEVICE).float() + 8.0,
                                 axis(cam.origin[2], vz))
    fib = torch.from_numpy(queue.fibonacci_dirs(64)).to(DEVICE)
    probes = _rays(sites.repeat_interleave(64, 0), fib.repeat(len(sites), 1), 256.0, 0)
    n = case["picks"]
    size = torch.tensor([float(v) for v in world.voxels], device=DEVICE)
    picks = _rays(torch.rand((n, 3), generator=gen, device=DEVICE) * size, _directions(n, gen),
                  8.0, 0)
    rays = torch.cat([primary, probes, picks]).reshape(-1, 32)
    order = torch.randperm(len(rays), generator=gen, device=DEVICE)
    return rays[order].reshape(-1).contiguous()


def _picks(n, rng):
    """Picking rays of the reference's bench: eyes over the terrain, looking down ahead."""
    cams = np.stack([rng.uniform(60, 450, n), rng.uniform(85, 130, n),
                     rng.uniform(60, 450, n)], 1).astype(np.float32)
    a = rng.uniform(0, 2 * math.pi, n)
    dirs = np.stack([np.sin(a), np.full(n, -0.5), np.cos(a)], 1)
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    return cams, dirs.astype(np.float32)


def _bricks(n, world, cam, rng):
    """n bricks re-randomised near the camera: occupancy exactly where the material is set."""
    bx, by, bz = world.dims
    x, z = rng.integers(0, bx, n), rng.integers(0, bz, n)
    y = rng.integers(16, 32, n)
    b = np.zeros(n, L.BRICK_DTYPE)
    mat = np.where(rng.random((n, 64)) < 0.5, rng.integers(1, 5, (n, 1)), 0).astype(np.uint8)
    b["materials"] = mat
    b["occupancy"] = np.packbits(mat != 0, axis=1, bitorder="little").view(np.uint64)[:, 0]
    return (x + y * bx + z * bx * by).astype(np.uint32), b


def _samples(n, seed):
    """Network inputs and targets, with the distribution that labelled camera rays have:
    an origin inside its chunk, a direction, the chunk's tile bits (solid below some
    height, ragged at it) and the log of a first-hit distance."""
    gen = torch.Generator(DEVICE).manual_seed(seed)
    x = torch.zeros((n, L.MLP_FEATURES), dtype=torch.float32, device=DEVICE)
    x[:, 0:3] = torch.rand((n, 3), generator=gen, device=DEVICE)
    x[:, 3:6] = _directions(n, gen)
    layer = torch.arange(64, device=DEVICE) // 16        # bit x + z*4 + y*16
    fill = torch.rand((n, 1), generator=gen, device=DEVICE) * 4.0
    p = (fill - layer).clamp(0.0, 1.0)
    x[:, 6:70] = (torch.rand((n, 64), generator=gen, device=DEVICE) < p).float()
    t = torch.rand(n, generator=gen, device=DEVICE) * math.log(700.0)
    return x, t


def _parameters(seed):
    """Parameters of the size that training starts from and keeps."""
    gen = torch.Generator().manual_seed(seed + 1)
    out = []
    for name, shape in MLP_TENSORS:
        v = torch.randn(shape, generator=gen)
        if name == "w1":
            v = v / math.sqrt(70.0)
            v[:, 70:] = 0.0
        elif name.startswith("w"):
            v = v / 8.0
        else:
            v = v * 0.1 + (math.log(150.0) if name == "bo" else 0.0)
        out.append(v.reshape(-1))
    return torch.cat(out).numpy()


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.turn = case, 0
    op = case["op"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(DEVICE).manual_seed(seed)
    if op in ("frame", "host_frame"):
        s.world = _world(case["bx"], case["bz"], seed)
        origin = (case.get("origin_x", 0), 0, case.get("origin_z", 0))
        n = case["width"] * case["height"]
        s.cam = _camera(s.world, rng, case["width"], case["height"], origin,
                        case.get("jitter", False))
        s.params = vg.default_params(case["flags"], frame=float(rng.integers(0, 64)))
        if op == "frame":
            s.rec = torch.empty(n * 24, dtype=torch.uint8, device=DEVICE)
            s.shadow = torch.empty(n * 8, dtype=torch.uint8, device=DEVICE) \
                if case["flags"] & L.VX_F_SHADOW else None
        else:
            s.host = torch.empty(n * 12, dtype=torch.uint8, pin_memory=True)
            s.out = s.host.numpy().view(L.COMPACT_DTYPE).reshape(-1)
    elif op == "trace":
        s.world = _world(128, 128, seed)
        s.params = vg.default_params(LUT_LOD)
        s.rays = _trace_rays(s.world, case["rays"], gen)
        s.out = torch.empty(case["rays"] * 24, dtype=torch.uint8, device=DEVICE)
    elif op == "queue":
        s.world = _world(128, 128, seed)
        s.params = vg.default_params(LUT_LOD)
        s.cam = _camera(s.world, rng, case["width"], case["height"])
        s.rays = _queue_rays(s.world, s.cam, case, gen)
        n = s.rays.numel() // 32
        s.out = torch.empty(n * 24, dtype=torch.uint8, device=DEVICE)
        s.shadow = torch.empty(n * 8, dtype=torch.uint8, device=DEVICE)
    elif op in ("pick", "pick_one"):
        s.world = vg.DeviceWorld(128, 64, 128)
        s.world.fill_window(seed, 0, 0)
        s.cams, s.dirs = _picks(case.get("rays", 1), rng)
    elif op == "edit":
        s.world = _world(128, 128, seed)
        w, h = case["width"], case["height"]
        s.params = vg.default_params(FULL)
        s.cam = _camera(s.world, rng, w, h)
        s.sets = [_bricks(case["bricks"], s.world, s.cam, rng) for _ in range(2)]
        s.rec, s.shadow = vg.render_primary(s.world, s.cam, s.params)
        s.mask = torch.zeros(vg.tile_mask_words(w, h), dtype=torch.int32, device=DEVICE)
        torch.cuda.synchronize()
        s.stream = torch.cuda.Stream()
    elif op == "stream":
        s.world = vg.DeviceWorld(case["bx"], 64, case["bz"])
        s.seed = seed
        s.at = [int(rng.integers(-1000, 1000)), int(rng.integers(-1000, 1000))]
        s.pose = [float(rng.uniform(135, 165)), float(rng.uniform(0, 2 * math.pi)),
                  math.radians(float(rng.uniform(-20, -10)))]
        s.world.fill_window(seed, *s.at)
        s.params = vg.default_params(FULL)
        n = case["width"] * case["height"]
        s.rec = torch.empty(n * 24, dtype=torch.uint8, device=DEVICE)
        s.shadow = torch.empty(n * 8, dtype=torch.uint8, device=DEVICE)
    elif op == "learned":
        s.world = _world(128, 128, seed)
        s.params = vg.default_params(LUT_LOD)
        s.cam = _camera(s.world, rng, case["width"], case["height"])
        s.net = learned.Proposal(s.world, seed)
        s.rec = torch.empty(case["width"] * case["height"] * 24, dtype=torch.uint8, device=DEVICE)
    elif op == "grad":
        s.world = vg.DeviceWorld(64, 16, 64)
        s.net = learned.Proposal(s.world, seed)
        s.net.set_params(_parameters(seed))
        s.x, s.t = _samples(case["batch"], seed)
    else:
        raise ValueError(op)
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- passes
def _words(t):
    return t.view(torch.int32)


def run(s):
    case, op = s.case, s.case["op"]
    turn, s.turn = s.turn, s.turn + 1
    if op == "frame":
        vg.render_primary(s.world, s.cam, s.params, s.rec, s.shadow)
        return [_words(s.rec)] + ([] if s.shadow is None else [_words(s.shadow)])
    if op == "host_frame":
        vg.render_primary_host_compact(s.world, s.cam, s.params, s.out)
        return s.out.view(np.int32)
    if op == "trace":
        return _words(vg.trace(s.world, s.rays, s.params, out=s.out))
    if op == "queue":
        queue.run(s.world, s.rays, s.params, out=s.out, shadow=s.shadow)
        return [_words(s.out), _words(s.shadow)]
    if op == "pick_one":
        hit = vg.raycast(s.cams[0], s.dirs[0], s.world)
        return [-1] if hit is None else [*hit.voxel, *hit.normal]
    if op == "pick":
        hits, found = vg.raycast_batch(s.world, s.cams, s.dirs)
        return [hits.view(np.int32), found]
    if op == "edit":
        idx, bricks = s.sets[turn % 2]
        with torch.cuda.stream(s.stream):
            st = s.stream.cuda_stream
            s.world.apply_dirty(idx, bricks, st)
            s.mask.zero_()
            vg.project_dirty(s.world, s.cam, idx, s.mask, st)
            vg.tile_refresh(case["width"], case["height"], 16, turn % 16, s.mask, st)
            vg.render_primary_gated(s.world, s.cam, s.params, s.mask, s.rec, s.shadow, st)
        return [s.mask, _words(s.rec), _words(s.shadow)]
    if op == "stream":
        s.at[0] += case["dx"]
        s.at[1] += case["dz"]
        n = s.world.shift_origin(*s.at)
        origin = (32 * s.at[0], 0, 32 * s.at[1])
        vx, _, vz = s.world.voxels
        y, yaw, pitch = s.pose
        cam = vg.camera_from_pose((origin[0] + vx / 2 + 0.3, y, origin[2] + vz / 2 + 0.7), yaw,
                                  pitch, math.radians(70.0), case["width"], case["height"], origin)
        vg.render_primary(s.world, cam, s.params, s.rec, s.shadow)
        return [n, _words(s.rec), _words(s.shadow)]
    if op == "learned":
        learned.render_learned(s.world, s.net, s.cam, s.params, s.rec, stats=False)
        return _words(s.rec)
    loss, grad = s.net.grad(s.x, s.t)
    out, at = {"loss": loss}, 0
    for name, shape in MLP_TENSORS:
        n = math.prod(shape)
        out[name] = grad[at:at + n].reshape(shape)
        at += n
    return out


def work(case):
    op = case["op"]
    pixels = case.get("width", 0) * case.get("height", 0)
    shadow = 32 if case.get("flags", FULL) & L.VX_F_SHADOW else 24
    if op == "frame":        # records written; the world's masks read once
        return {"bytes": pixels * shadow + case["bx"] * case["bz"] * 10.0, "flops": 0}
    if op == "host_frame":
        return {"bytes": pixels * 12 + case["bx"] * case["bz"] * 10.0, "flops": 0}
    if op == "trace":
        return {"bytes": case["rays"] * 56.0, "flops": 0}
    if op == "queue":
        probes = (2 * case["probe_radius"] // 16) ** 2 * 16 * 64
        return {"bytes": (pixels + probes + case["picks"]) * 64.0, "flops": 0}
    if op == "pick_one":
        return {"bytes": 52.0, "flops": 0}
    if op == "pick":
        return {"bytes": case["rays"] * 52.0, "flops": 0}
    if op == "edit":         # the bricks, and the sixteenth of the frame that is refreshed
        return {"bytes": case["bricks"] * 152.0 + pixels * 2.0, "flops": 0}
    if op == "stream":       # the new chunks' 512 bricks of 73 bytes, and the frame
        sx, sz = case["bx"] // 8, case["bz"] // 8
        kept = max(0, sx - abs(case["dx"])) * max(0, sz - abs(case["dz"]))
        return {"bytes": (sx * sz - kept) * 8 * 512 * 73.0 + pixels * 32.0, "flops": 0}
    if op == "learned":
        return {"bytes": pixels * 24.0, "flops": 0}
    b = case["batch"]        # forward, and the gradients of weights and activations
    return {"bytes": b * 324.0, "flops": b * (2.0 * 2 * 64 * 70 + 3 * 2.0 * (2 * 64 * 64 + 64))}


def exact(case, seed):
    """The training step in 64 bits; the other outputs are whole numbers and bytes."""
    if case["op"] != "grad":
        return None
    x, t = (v.double() for v in _samples(case["batch"], seed))
    flat, at, p = torch.from_numpy(_parameters(seed)).to(DEVICE).double(), 0, {}
    for name, shape in MLP_TENSORS:
        n = math.prod(shape)
        p[name] = flat[at:at + n].reshape(shape).clone().requires_grad_(True)
        at += n

    def gelu(z):             # the tanh form, with the constants that the library states
        return 0.5 * z * (1.0 + torch.tanh(0.7978845608 * (z + 0.044715 * z * z * z)))

    h = gelu(x @ p["w1"].T + p["b1"])
    h = gelu(h @ p["w2"].T + p["b2"])
    h = gelu(h @ p["w3"].T + p["b3"])
    loss = ((h @ p["wo"] + p["bo"] - t) ** 2).mean()
    loss.backward()
    out = {k: v.grad for k, v in p.items()}
    out["loss"] = float(loss.detach())
    return out
