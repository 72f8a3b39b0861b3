"""The work that users of the render-and-encode library have it do, as cases
that can be timed and checked: renders over the wire, to YUV420P on the host
and to device buffers, batched serving, scene refits and the frame glue.

Each case goes through the public Python binding (nes.py), as a caller's
program does.  listed() are named cases; draw() gives others of the same
ranges; exact() restates the renderer's and the trainer's math in 64 bits.
"""
import math
import os
import struct
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "ngp-encode-server_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import nes  # noqa: E402

RES = (16, 22, 30, 42, 58, 80, 111, 153, 212, 294, 406, 561, 776, 1072, 1482, 2048)
DT = float(np.float32(math.sqrt(3.0) / 1024.0))
P1, P2 = 2654435761, 805459861
FLOPS_PER_SAMPLE = 2 * 9344  # the two MLPs' multiply-adds
SERVE_SIZES = ((640, 360, 1), (1280, 720, 1), (1920, 1080, 1), (1920, 1832, 2))  # the serving configuration's mix


def listed():
    return [
        # One small frame over neserver's renderer protocol: FrameRequest bytes in, RenderedFrame bytes
        # (RGB24 + GRAY8 depth) out.  Latency and launches are the whole cost.
        {"name": "wire_64x48", "kind": "wire", "precision": "tc", "w": 64, "h": 48, "scene": "seeded", "log2T": 19},
        # The smallest view of the serving mix, pose -> YUV420P and uint16 depth in host memory for the encoder.
        {"name": "yuv_360p", "kind": "yuv", "precision": "tc", "w": 640, "h": 360, "n": 1, "fov": 90.0,
         "radius": 1.5, "scene": "seeded", "log2T": 19},
        # The headline drop-in frame on the tensor cores, left on the device.
        {"name": "views_1080p", "kind": "views", "precision": "tc", "w": 1920, "h": 1080, "n": 1, "fov": 90.0,
         "radius": 1.5, "scene": "seeded", "log2T": 19},
        # The precision form's headset pair, both eyes in one batch, planes on the host: the largest request.
        {"name": "yuv_stereo_1832", "kind": "yuv", "precision": "tc", "w": 1920, "h": 1832, "n": 2, "fov": 100.0,
         "radius": 1.6, "scene": "seeded", "log2T": 19},
        # Odd-sized views in one batch over an opaque, mostly empty field, as a fitted scene has: the
        # occupancy grid and early termination set the samples.
        {"name": "views_surface_odd", "kind": "views", "precision": "tc", "w": 853, "h": 481, "n": 3, "fov": 90.0,
         "radius": 1.4, "scene": "surface", "log2T": 19},
        # The plain FP32 path: the CPU pipeline's 256 x 256 view, and the drop-in frame.
        {"name": "views_fp32_256", "kind": "views", "precision": "fp32", "w": 256, "h": 256, "n": 1, "fov": 90.0,
         "radius": 1.5, "scene": "seeded", "log2T": 19},
        {"name": "views_fp32_1080p", "kind": "views", "precision": "fp32", "w": 1920, "h": 1080, "n": 1, "fov": 90.0,
         "radius": 1.5, "scene": "seeded", "log2T": 19},
        # Eight requests of the serving mix submitted at once, batched by the server, fetched for the host encoder.
        {"name": "serve_mix_8", "kind": "serve", "requests": 8, "first": 0, "fov": 90.0, "radius": 1.6, "log2T": 19},
        # One step of the refit configuration: 2^18 rays, gradients and Adam; the scene read back afterwards.
        {"name": "refit_step_256k", "kind": "step", "rays": 1 << 18, "exact_grads": 0, "log2T": 19},
        # Loss and gradient of a small batch in the default mode and in the strict FP32 mode (gradient checks,
        # callers with an optimizer of their own).
        {"name": "grad_16k", "kind": "grad", "rays": 16384, "exact_grads": 0, "log2T": 17},
        {"name": "grad_strict_4k", "kind": "grad", "rays": 4001, "exact_grads": 1, "log2T": 16},
        # The frame glue alone: a second of 720p frames in one launch per plane kind.
        {"name": "glue_720p_x30", "kind": "glue", "w": 1280, "h": 720, "frames": 30, "batched": True, "pad": True},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["wire", "yuv", "yuv", "views", "views", "views_fp32", "serve", "step", "grad", "glue"])
    scene = rng.choice(["seeded", "seeded", "surface"])
    log2T = rng.choice([14, 17, 19, 19, 19, 22])
    fov = float(rng.choice([70, 90, 100]))
    radius = round(rng.uniform(1.35, 2.0), 3)
    if kind == "wire":
        w = log_int(32, 960)
        return {"kind": "wire", "precision": rng.choice(["tc", "fp32"]) if w < 300 else "tc", "w": w,
                "h": max(1, int(w * rng.uniform(0.4, 0.8))), "scene": scene, "log2T": log2T}
    if kind == "yuv":
        n = rng.choice([1, 2])
        w = log_int(96, 1920)
        return {"kind": "yuv", "precision": "tc", "w": w, "h": max(2, int(w * rng.uniform(0.5, 0.9))), "n": n,
                "fov": fov, "radius": max(radius, 1.6), "scene": scene, "log2T": log2T}
    if kind == "views":
        n = rng.choice([1, 1, 2, 4])
        w = log_int(48, 1920 // n)
        return {"kind": "views", "precision": "tc", "w": w, "h": max(1, int(w * rng.uniform(0.4, 0.9))), "n": n,
                "fov": fov, "radius": radius, "scene": scene, "log2T": log2T}
    if kind == "views_fp32":
        w = log_int(48, 960)
        return {"kind": "views", "precision": "fp32", "w": w, "h": max(1, int(w * rng.uniform(0.4, 0.8))), "n": 1,
                "fov": fov, "radius": radius, "scene": scene, "log2T": log2T}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randrange(1, 9), "first": rng.randrange(4), "fov": 90.0,
                "radius": max(radius, 1.6), "log2T": 19}
    if kind == "step":
        return {"kind": "step", "rays": log_int(1 << 11, 1 << 18), "exact_grads": 0, "log2T": rng.choice([15, 17, 19])}
    if kind == "grad":
        e = rng.choice([0, 0, 1])
        return {"kind": "grad", "rays": log_int(256, 8192 if e else 32768), "exact_grads": e,
                "log2T": rng.choice([14, 16, 19])}
    w = log_int(64, 3840)
    return {"kind": "glue", "w": w, "h": max(1, int(w * rng.uniform(0.4, 0.8))),
            "frames": rng.choice([1, 1, 4, 30]) if w <= 1280 else 1, "batched": rng.choice([True, False]),
            "pad": rng.choice([True, False])}


# ---------------------------------------------------------------- scenes


class Scene:
    """A hash-grid field's parameters as a caller loads them into a context: tables U(-0.5, 0.5) and
    Xavier-uniform weights (the seeded scene's distributions).  "surface": the density logit spread as a fitted
    scene's is (empty space, opaque walls), its occupancy threshold at density 1."""

    def __init__(self, seed, log2T, kind):
        rng = np.random.default_rng([seed, 77])
        self.log2T, self.T = log2T, 1 << log2T
        self.table = rng.random(16 * self.T * 2, dtype=np.float32) - np.float32(0.5)

        def xavier(o, i, fan=None):
            a = math.sqrt(6.0 / (o + (fan or i)))
            return ((rng.random((o, i), dtype=np.float32) * 2 - 1) * np.float32(a)).astype(np.float32)

        self.w = [xavier(64, 32), xavier(16, 64), xavier(64, 32, 31), xavier(64, 64), xavier(3, 64)]
        self.w[2][:, 31] = 0.0
        self.threshold = 0.01
        if kind == "surface":
            self.threshold = 1.0
            x = torch.from_numpy(rng.random((4096, 3), dtype=np.float32)).cuda()
            h = torch.relu(_encode64(self.table64(), self.T, x) @ torch.from_numpy(self.w[0]).cuda().double().T)
            row = torch.from_numpy(self.w[1][0]).cuda().double()
            lg = h @ row
            row = row - lg.mean() / h.sum(1).mean()
            lg = h @ row
            row = row * (5.5 / lg.std())
            row = row + (-2.3 - (h @ row).mean()) / h.sum(1).mean()
            self.w[1][0] = row.float().cpu().numpy()

    def table64(self):
        return torch.from_numpy(self.table).cuda().double().view(-1, 2)

    def load(self, renderer):
        renderer.set_scene_param(0, self.table)
        for k, w in enumerate(self.w):
            renderer.set_scene_param(k + 1, w)
        renderer.rebuild_occupancy(self.threshold)


def _renderer(scene, precision, max_pixels):
    r = nes.Renderer(precision=nes.PREC_FP32 if precision == "fp32" else nes.PREC_FP16_TC, log2_table_size=scene.log2T,
                     max_pixels=max_pixels)
    scene.load(r)
    return r


def _poses(case, seed):
    """The poses of a case's views: a stereo pair for a two-view host request, else one pose each."""
    n = case["n"]
    r = case["radius"]
    base = nes.shell_poses(seed, n, r, r)
    return nes.stereo_pair(base[0], 0.063) if case["kind"] == "yuv" and n == 2 else base


def _wire_request(matrix, w, h, index):
    def varint(v):
        out = b""
        while v > 127:
            out += bytes([v & 127 | 128])
            v >>= 7
        return out + bytes([v])

    m = struct.pack("<12f", *matrix)
    # Camera{is_left = 2, width = 3, height = 4, matrix = 12}, FrameRequest{index = 1, camera = 2, is_left = 3}
    cam = b"\x10\x01" + b"\x18" + varint(w) + b"\x20" + varint(h) + b"\x62" + varint(len(m)) + m
    return b"\x08" + varint(index) + b"\x12" + varint(len(cam)) + cam + b"\x18\x01"


class _Serving:
    """A server and the context it serves, closed in that order."""

    def __init__(self, renderer):
        self.renderer = renderer
        self.server = nes.Server(renderer, max_queue_ms=0.0)

    def __del__(self):
        self.server.close()
        self.renderer.close()


class _Training:
    def __init__(self, renderer, trainer):
        self.renderer, self.trainer = renderer, trainer

    def __del__(self):
        self.trainer.close()
        self.renderer.close()


TRAIN_VIEWS, TRAIN_SIDE, TRAIN_FOV = 16, 400, 40.0


def _targets(seed):
    """Images to refit to, as photographs are: smooth colour and depth with a little noise, views one after another."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = TRAIN_SIDE * TRAIN_SIDE
    y, x = torch.meshgrid(*[torch.arange(TRAIN_SIDE, device="cuda") / TRAIN_SIDE] * 2, indexing="ij")
    k = 2 + 6 * torch.rand(TRAIN_VIEWS, 4, 3, device="cuda", generator=g)
    wave = torch.sin(k[:, 0, :, None, None] * x + k[:, 1, :, None, None]) \
        * torch.cos(k[:, 2, :, None, None] * y + k[:, 3, :, None, None])
    rgb = 0.5 + 0.2 * wave.permute(0, 2, 3, 1).reshape(TRAIN_VIEWS * n, 3)
    dep = 1.1 + 0.2 * wave.mean(1).reshape(-1)
    rgb = rgb + 0.02 * torch.randn(rgb.shape, device="cuda", generator=g)
    return rgb.contiguous(), dep.contiguous()


def _train_poses(seed):
    return nes.shell_poses(seed, TRAIN_VIEWS, 1.2, 2.0)


def _pairs(case, seed):
    rng = np.random.default_rng([seed, 3])
    return np.stack([rng.integers(0, TRAIN_VIEWS, case["rays"]),
                     rng.integers(0, TRAIN_SIDE * TRAIN_SIDE, case["rays"])], 1).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "glue":
        g = torch.Generator(device="cuda").manual_seed(seed)
        w, h, nf = case["w"], case["h"], case["frames"]
        rls = (3 * w + 31) // 32 * 32 if case["pad"] else 3 * w
        gls = (w + 31) // 32 * 32 if case["pad"] else w
        ls = nes.linesizes(w)
        ch = (h + 1) // 2

        def planes():  # the frames' planes, one array per plane kind
            return [torch.zeros(nf, k, dtype=torch.uint8, device="cuda") for k in (ls[0] * h, ls[1] * ch, ls[2] * ch)]

        def at(t):
            return [t.data_ptr() + i * t[0].numel() * t.element_size() for i in range(nf)]

        ramp = (torch.arange(rls, device="cuda") * 255 // max(1, rls - 1)).to(torch.int32)
        rgb = ((torch.randint(0, 256, (nf, h, rls), device="cuda", generator=g, dtype=torch.int32) + ramp) // 2)
        rgb = rgb.to(torch.uint8)
        gray = torch.randint(0, 256, (nf, h, gls), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
        dep = torch.rand(nf, h * w, device="cuda", generator=g) * 9.9 + 0.1
        mm = torch.zeros(nf, h * w, dtype=torch.int16, device="cuda")
        s = {"case": case, "rls": rls, "gls": gls, "ls": ls, "rgb": rgb, "gray": gray, "dep": dep, "mm": mm,
             "scene": planes(), "depth": planes()}
        for k in ("rgb", "gray", "dep", "mm"):
            s[k + "_p"] = at(s[k])
        for k in ("scene", "depth"):
            s[k + "_p"] = [at(p) for p in s[k]]
        return s
    if kind in ("step", "grad"):
        scene = Scene(seed, case["log2T"], "seeded")
        r = _renderer(scene, "fp32", 4096)
        # Adam's common epsilon: updated parameters then vary smoothly with a gradient near zero, where a smaller
        # one turns the order of the atomic additions into the sign of the step.
        t = nes.Trainer(r, batch_rays=case["rays"], exact_weight_grads=case["exact_grads"], eps=1e-8)
        rgb, dep = _targets(seed)
        f = nes.focal_from_fov(TRAIN_SIDE, TRAIN_FOV)
        t.set_targets([nes.make_view(m, TRAIN_SIDE, TRAIN_SIDE, f) for m in _train_poses(seed)], rgb.data_ptr(),
                      dep.data_ptr())
        return {"case": case, "train": _Training(r, t), "rgb": rgb, "dep": dep, "seed": seed * 1000,
                "pairs": _pairs(case, seed), "floats": 16 * scene.T * 2}
    if kind == "serve":
        scene = Scene(seed, case["log2T"], "seeded")
        reqs = []
        for k in range(case["requests"]):
            w, h, n = SERVE_SIZES[(case["first"] + k) % 4]
            pose = nes.shell_poses(seed * 16 + k, 1, case["radius"], case["radius"])[0]
            f = nes.focal_from_fov(w, case["fov"])
            reqs.append([nes.make_view(m, w, h, f) for m in ([pose] if n == 1 else nes.stereo_pair(pose, 0.063))])
        return {"case": case, "serving": _Serving(_renderer(scene, "tc", 4096)), "reqs": reqs}
    scene = Scene(seed, case["log2T"], case["scene"])
    w, h = case["w"], case["h"]
    if kind == "wire":
        m = nes.shell_poses(seed, 1, 1.5, 1.5)[0]
        return {"case": case, "r": _renderer(scene, case["precision"], w * h),
                "request": _wire_request(m, w, h, 1 + seed % 1000)}
    n = case["n"]
    f = nes.focal_from_fov(w, case["fov"])
    views = [nes.make_view(m, w, h, f) for m in _poses(case, seed)]
    s = {"case": case, "r": _renderer(scene, case["precision"], n * w * h), "views": views}
    if kind == "views":
        s["rgb"] = [torch.zeros(h, w, 3, device="cuda") for _ in range(n)]
        s["depth"] = [torch.zeros(h, w, device="cuda") for _ in range(n)]
    else:
        ls, ch = nes.linesizes(w), (h + 1) // 2
        s["ls"] = ls
        s["planes"] = [[torch.zeros(k, dtype=torch.uint8, pin_memory=True) for _ in range(n)]
                       for k in (ls[0] * h, ls[1] * ch, ls[2] * ch)]
        s["mm"] = [torch.zeros(h * w, dtype=torch.uint16, pin_memory=True) for _ in range(n)]
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "wire":
        return np.frombuffer(state["r"].render(state["request"]), np.uint8)
    if kind == "views":
        stream = torch.cuda.current_stream().cuda_stream
        state["r"].render_views(state["views"], [t.data_ptr() for t in state["rgb"]],
                                [t.data_ptr() for t in state["depth"]], stream)
        return {"rgb": state["rgb"], "depth": state["depth"]}
    if kind == "yuv":
        y, u, v = ([t.data_ptr() for t in p] for p in state["planes"])
        state["r"].render_yuv_views(state["views"], y, u, v, state["ls"], [t.data_ptr() for t in state["mm"]])
        return {"planes": state["planes"], "mm": state["mm"]}
    if kind == "serve":
        srv = state["serving"].server
        tickets = [srv.submit(v) for v in state["reqs"]]
        out = []
        for t, views in zip(tickets, state["reqs"]):
            res = srv.wait(t)
            out.append([srv.fetch(res, k) for k in range(len(views))])
            srv.release(t)
        return out
    if kind == "step":
        state["seed"] += 1
        loss = state["train"].trainer.step(state["seed"])
        r = state["train"].renderer
        sizes = (state["floats"], 64 * 32, 16 * 64, 64 * 32, 64 * 64, 3 * 64)
        return {"loss": loss, "params": [r.scene_param(k, n) for k, n in enumerate(sizes)]}
    if kind == "grad":
        loss, gt, gw = state["train"].trainer.grad(state["pairs"], state["floats"])
        return {"loss": loss, "table": gt, "weights": gw}
    w, h, ls, s = case["w"], case["h"], state["ls"], state
    if case["batched"]:
        nes.yuv420p_batch(s["rgb_p"], w, h, s["rls"], *s["scene_p"], ls)
        nes.yuv420p_batch(s["gray_p"], w, h, s["gls"], *s["depth_p"], ls, gray=True)
        nes.depth_pack_u16mm_batch(s["dep_p"], w * h, s["mm_p"])
    else:
        for i in range(case["frames"]):
            nes.rgb24_to_yuv420p(s["rgb_p"][i], w, h, s["rls"], *[p[i] for p in s["scene_p"]], ls)
            nes.gray8_to_yuv420p(s["gray_p"][i], w, h, s["gls"], *[p[i] for p in s["depth_p"]], ls)
            nes.depth_pack_u16mm(s["dep_p"][i], w * h, s["mm_p"][i])
    return {"scene": s["scene"], "depth": s["depth"], "mm": s["mm"]}


# ---------------------------------------------------------------- what a pass cannot do without


def _steps(pose, w, h, focal):
    """Mean march steps per pixel of a view, from a 48 x 48 grid of its rays."""
    m = np.asarray(pose, np.float64).reshape(3, 4)
    g = (np.arange(48) + 0.5) / 48
    u, v = np.meshgrid((g * w - 0.5 * w) / focal, (g * h - 0.5 * h) / focal)
    d = m[:, 0, None, None] * u + m[:, 1, None, None] * v + m[:, 2, None, None]
    d /= np.sqrt((d * d).sum(0))
    with np.errstate(divide="ignore"):
        t = np.stack([(0.0 - m[:, 3, None, None]) / d, (1.0 - m[:, 3, None, None]) / d])
    near, far = np.maximum(t.min(0).max(0), 0.0), t.max(0).min(0)
    return float(np.where(far > near, np.minimum(1024, np.floor((far - near) / DT)), 0).mean())


#: Share of the march steps that are evaluated in a "surface" scene (occupied and before the ray ends).
SURFACE_SHARE = 0.1


def _mean_steps(w, h, fov, radius):
    f = 0.5 * w / math.tan(math.radians(fov) / 2)
    return sum(_steps(p, w, h, f) for p in nes.shell_poses(1, 6, radius, radius)) / 6


def work(case):
    kind = case["kind"]
    if kind == "glue":
        px, c = case["w"] * case["h"], ((case["w"] + 1) // 2) * ((case["h"] + 1) // 2)
        per = 3 * px + px + 2 * c + px + px + 2 * c + 4 * px + 2 * px
        return {"bytes": per * case["frames"], "flops": 15 * px * case["frames"]}
    params = 16 * (1 << case["log2T"]) * 2
    if kind in ("step", "grad"):
        f = 0.5 * TRAIN_SIDE / math.tan(math.radians(TRAIN_FOV) / 2)
        m = sum(_steps(p, TRAIN_SIDE, TRAIN_SIDE, f) for p in nes.shell_poses(1, 8, 1.2, 2.0)) / 8
        samples = case["rays"] * m
        # table read, its gradient written; a step also reads and writes both moments and the parameters.
        per = 4 * params * (8 if kind == "step" else 2)
        return {"bytes": per + 16 * case["rays"], "flops": 3 * FLOPS_PER_SAMPLE * samples}
    size = 2 if case.get("precision", "tc") == "tc" else 4
    if kind == "serve":
        px = samples = 0.0
        for k in range(case["requests"]):
            w, h, n = SERVE_SIZES[(case["first"] + k) % 4]
            px += n * w * h
            samples += n * w * h * _mean_steps(w, h, case["fov"], case["radius"])
        return {"bytes": size * params + 3.5 * px, "flops": FLOPS_PER_SAMPLE * samples}
    w, h, n = case["w"], case["h"], case.get("n", 1)
    samples = n * w * h * _mean_steps(w, h, case.get("fov", 90.0), case.get("radius", 1.5))
    samples *= SURFACE_SHARE if case["scene"] == "surface" else 1.0
    per_px = {"wire": 4.0, "views": 16.0, "yuv": 3.5}[kind]
    return {"bytes": size * params + per_px * n * w * h, "flops": FLOPS_PER_SAMPLE * samples}


# ---------------------------------------------------------------- the same in 64 bits


def _cells(x, level):
    n = RES[level]
    p = x.double() * n
    i = p.floor().clamp(0, n - 1)
    return i.long(), p - i


def _corner(i, level, T, k):
    n = RES[level]
    x, y, z = i[:, 0] + (k & 1), i[:, 1] + (k >> 1 & 1), i[:, 2] + (k >> 2 & 1)
    if (n + 1) ** 3 <= T:
        return level * T + x + (n + 1) * (y + (n + 1) * z)
    return level * T + ((x ^ (y * P1) ^ (z * P2)) & (T - 1))


def _weight(f, k):
    w = (f[:, 0] if k & 1 else 1 - f[:, 0]) * (f[:, 1] if k & 2 else 1 - f[:, 1])
    return w * (f[:, 2] if k & 4 else 1 - f[:, 2])


def _encode64(table, T, x):
    out = torch.empty(x.shape[0], 32, dtype=torch.float64, device=x.device)
    for level in range(16):
        i, f = _cells(x, level)
        a = 0
        for k in range(8):
            a = a + _weight(f, k)[:, None] * table[_corner(i, level, T, k)]
        out[:, 2 * level:2 * level + 2] = a
    return out


def _sh64(d):
    x, y, z = d.double().unbind(1)
    pi = math.pi
    c1, c2 = math.sqrt(3 / (4 * pi)), 0.5 * math.sqrt(15 / pi)
    c3a, c3c = 0.25 * math.sqrt(35 / (2 * pi)), 0.25 * math.sqrt(21 / (2 * pi))
    return torch.stack([
        torch.full_like(x, 0.5 / math.sqrt(pi)), c1 * y, c1 * z, c1 * x, c2 * x * y, c2 * y * z,
        0.25 * math.sqrt(5 / pi) * (3 * z * z - 1), c2 * x * z, 0.5 * c2 * (x * x - y * y),
        c3a * y * (3 * x * x - y * y), 0.5 * math.sqrt(105 / pi) * x * y * z, c3c * y * (5 * z * z - 1),
        0.25 * math.sqrt(7 / pi) * z * (5 * z * z - 3), c3c * x * (5 * z * z - 1),
        0.25 * math.sqrt(105 / pi) * z * (x * x - y * y), c3a * x * (x * x - 3 * y * y)], 1)


def _mlp64(enc, sh, w):
    out = torch.relu(enc @ w[0].T) @ w[1].T
    cin = torch.cat([sh, out[:, 1:], torch.zeros_like(out[:, :1])], 1)
    rgb = torch.sigmoid(torch.relu(torch.relu(cin @ w[2].T) @ w[3].T) @ w[4].T)
    return torch.exp(out[:, 0] - 1), rgb


def _occupancy(scene, table, w):
    g = (torch.arange(128, device="cuda", dtype=torch.float32) + 0.5) / 128
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    x = torch.stack([x, y, z], -1).view(-1, 3)
    occ = torch.empty(x.shape[0], dtype=torch.bool, device="cuda")
    for a in range(0, x.shape[0], 1 << 19):
        out = torch.relu(_encode64(table, scene.T, x[a:a + (1 << 19)]) @ w[0].T) @ w[1][0]
        occ[a:a + (1 << 19)] = torch.exp(out - 1) > scene.threshold
    return occ


def _rays(matrix, w, h, focal, pix):
    """The ray set-up, in FP32 as it is defined: direction, start, whole number of steps."""
    m = torch.tensor(matrix, dtype=torch.float32, device="cuda").view(3, 4)
    f = torch.tensor(focal, dtype=torch.float32, device="cuda")
    u = ((pix % w).float() + 0.5 - 0.5 * w) / f
    v = ((pix // w).float() + 0.5 - 0.5 * h) / f
    dv = [m[a, 0] * u + m[a, 1] * v + m[a, 2] for a in range(3)]
    nrm = torch.sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2])
    d = torch.stack([a / nrm for a in dv], 1)
    o = m[:, 3].expand(pix.shape[0], 3)
    inv = torch.ones_like(d) / d
    t0, t1 = (torch.zeros_like(o) - o) * inv, (torch.ones_like(o) - o) * inv
    ts = torch.minimum(t0, t1).amax(1).clamp(min=0)
    tf = torch.maximum(t0, t1).amin(1)
    n = torch.where(tf > ts, torch.floor((tf - ts) / torch.tensor(DT, dtype=torch.float32, device="cuda")),
                    torch.zeros_like(tf)).clamp(0, 1024).long()
    return o, d, ts, n


def _chunks(n, limit):
    """Ranges of rays whose padded steps stay within `limit`."""
    n = n.cpu().numpy()
    a = 0
    while a < len(n):
        b, most = a, 0
        while b < len(n) and max(most, int(n[b])) * (b + 1 - a) <= limit:
            most = max(most, int(n[b]))
            b += 1
        yield a, max(b, a + 1), max(most, 1)
        a = max(b, a + 1)


def _march(rays, most):
    """t and positions of a range of rays' steps (FP32 values, as the steps are defined) and which exist."""
    o, d, ts, n = rays
    i = torch.arange(most, device="cuda", dtype=torch.float64) + 0.5
    t = (i[None] * DT + ts.double()[:, None]).float()
    x = (t.double()[..., None] * d.double()[:, None] + o.double()[:, None]).float().clamp(0, 1)
    return t, x, torch.arange(most, device="cuda")[None] < n[:, None]


def _occupied(occ, x):
    c = (x * 128).floor().clamp(0, 127).long()
    return occ[c[..., 0] + 128 * (c[..., 1] + 128 * c[..., 2])]


def _composite(alpha, rgb, t):
    trans = torch.cumprod(1 - alpha, 1)
    before = torch.cat([torch.ones_like(trans[:, :1]), trans[:, :-1]], 1)
    wgt = torch.where(before >= 1e-4, before * alpha, torch.zeros_like(alpha))
    return (wgt[..., None] * rgb).sum(1), (wgt * t).sum(1)


def _render64(scene, matrix, w, h, focal):
    table, wt = scene.table64(), [torch.from_numpy(a).cuda().double() for a in scene.w]
    occ = _occupancy(scene, table, wt)
    order = torch.arange(w * h, device="cuda")
    rays = _rays(matrix, w, h, focal, order)
    order = torch.argsort(rays[3])
    rays = [a[order] for a in rays]
    rgb = torch.zeros(w * h, 3, dtype=torch.float64, device="cuda")
    dep = torch.zeros(w * h, dtype=torch.float64, device="cuda")
    for a, b, most in _chunks(rays[3], 2_000_000):
        part = [v[a:b] for v in rays]
        t, x, ok = _march(part, most)
        ok &= _occupied(occ, x)
        sh = _sh64(part[1])[:, None].expand(-1, most, -1)[ok]
        sigma, c = _mlp64(_encode64(table, scene.T, x[ok]), sh, wt)
        al = torch.zeros(ok.shape, dtype=torch.float64, device="cuda")
        cc = torch.zeros(*ok.shape, 3, dtype=torch.float64, device="cuda")
        al[ok] = -torch.expm1(-sigma * DT)
        cc[ok] = c
        rgb[order[a:b]], dep[order[a:b]] = _composite(al, cc, t.double())
    return rgb.view(h, w, 3), dep.view(h, w)


def _grad64(case, seed):
    scene = Scene(seed, case["log2T"], "seeded")
    table, wt = scene.table64(), [torch.from_numpy(a).cuda().double().requires_grad_() for a in scene.w]
    occ = _occupancy(scene, table, [a.detach() for a in wt])
    rgb, dep = _targets(seed)
    pairs = torch.from_numpy(_pairs(case, seed)).cuda().long()
    f = 0.5 * TRAIN_SIDE / math.tan(0.5 * TRAIN_FOV * math.pi / 180)
    parts = []
    for v, m in enumerate(_train_poses(seed)):
        at = torch.nonzero(pairs[:, 0] == v).flatten()
        if at.numel():
            parts.append([*_rays(m, TRAIN_SIDE, TRAIN_SIDE, f, pairs[at, 1]), at])
    rays = [torch.cat([p[k] for p in parts]) for k in range(5)]
    order = torch.argsort(rays[3])
    rays = [a[order] for a in rays]
    q = (pairs[:, 0] * TRAIN_SIDE * TRAIN_SIDE + pairs[:, 1])[rays.pop()]
    gt, total = torch.zeros_like(table), 0.0
    for a, b, most in _chunks(rays[3], 700_000):
        part = [v[a:b] for v in rays]
        t, x, ok = _march(part, most)
        ok &= _occupied(occ, x)
        enc = _encode64(table, scene.T, x[ok]).requires_grad_()
        sigma, c = _mlp64(enc, _sh64(part[1])[:, None].expand(-1, most, -1)[ok], wt)
        al = torch.zeros(ok.shape, dtype=torch.float64, device="cuda").masked_scatter(ok, -torch.expm1(-sigma * DT))
        cc = torch.zeros(*ok.shape, 3, dtype=torch.float64, device="cuda").masked_scatter(
            ok[..., None].expand(-1, -1, 3), c)
        C, D = _composite(al, cc, t.double())
        e, ed = C - rgb[q[a:b]].double(), D - dep[q[a:b]].double()
        loss = ((e * e).sum() + 0.1 * (ed * ed).sum()) / case["rays"]
        loss.backward()
        total += float(loss.detach())
        for level in range(16):
            i, fr = _cells(x[ok], level)
            for k in range(8):
                gt.index_add_(0, _corner(i, level, scene.T, k),
                              _weight(fr, k)[:, None] * enc.grad[:, 2 * level:2 * level + 2])
    return {"loss": total, "table": gt.view(-1),
            "weights": torch.cat([torch.zeros_like(a).view(-1) if a.grad is None else a.grad.view(-1) for a in wt])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "views" and case["n"] * case["w"] * case["h"] <= 2_100_000:
        scene = Scene(seed, case["log2T"], case["scene"])
        w, h = case["w"], case["h"]
        f = float(np.float32(0.5 * w / math.tan(0.5 * case["fov"] * math.pi / 180)))
        out = [_render64(scene, m, w, h, f) for m in _poses(case, seed)]
        return {"rgb": [o[0] for o in out], "depth": [o[1] for o in out]}
    if kind == "grad":
        return _grad64(case, seed)
    return None
