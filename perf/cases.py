"""The work that programs have this library do, as measurable cases.

A case names one call a user's program makes -- a batch of ray queries, a BVH rebuild, a
rendered frame, a batch of small renders, a film denoise, a training step's gradients, one
of the NLM filters, a tonemap -- with its sizes and options.  `listed` holds the cases that
are measured, `draw` gives more of the same ranges, `prepare` makes a case's inputs from a
seed, `run` makes the call once through the public API, `work` counts the bytes and
operations the call cannot do without, and `exact` gives the result in 64 bits where the
result is a plain formula of the inputs.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

import salty_gb300 as sg
from salty_gb300 import scenes
from salty_gb300.denoiser import DEFAULT_WEIGHTS, load_weights


def listed():
    return [
        # a picking or visibility query of an interactive program: few rays, small scene
        {"name": "trace_4k_rays", "kind": "trace", "tris": 30000, "rays": 4096, "watertight": False, "host": False},
        # the traversal microbenchmark on device arrays, at a quarter of its rays
        {"name": "trace_4m_rays", "kind": "trace", "tris": 1000000, "rays": 1 << 22, "watertight": False,
         "host": False},
        # the same scene end to end from pinned host arrays, a ragged count, watertight test
        {"name": "trace_host_2m_rays", "kind": "trace", "tris": 1000000, "rays": 2500003, "watertight": True,
         "host": True},
        # a changed scene: rebuild its BVH, then trace a first set of rays
        {"name": "rebuild_1m_tris", "kind": "rebuild", "tris": 1000000, "rays": 1 << 18},
        # the Cornell box preview: 256 x 256 at 16 samples per pixel, depth 8
        {"name": "render_cornell_256", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "compat": False},
        # one progressive pass of a full-size heightfield frame
        {"name": "render_terrain_1080p", "kind": "render", "scene": "terrain", "grid": 1024, "spheres": 1024,
         "width": 1920, "height": 1080, "spp": 8, "depth": 12, "compat": False},
        # many uneven scenes in one call (data generation, thumbnails)
        {"name": "render_batch_12", "kind": "batch", "scenes": 12, "tris": 300000},
        # the learned denoiser on a film, averaged over the 8 symmetries (Denoiser's default)
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080, "mirrors": 8},
        # the denoiser's training batch
        {"name": "train_16x256", "kind": "train", "n": 16, "h": 256, "w": 256},
        # the variance-scaled NLM at its default window, the denoiser without weights
        {"name": "nlm_1080p", "kind": "nlm", "width": 1920, "height": 1080, "search": 10, "patch": 3},
        # the reference's NLM filter on an odd-sized frame
        {"name": "nlm_ref_odd_720p", "kind": "nlm_ref", "width": 1279, "height": 719},
        # the tonemap and sRGB8 step of a displayed frame
        {"name": "tonemap_1080p", "kind": "tonemap", "width": 1920, "height": 1080, "type": sg.TM_ACES},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "rebuild", "render", "render", "batch", "denoise", "train", "nlm", "nlm_ref",
                       "tonemap"])
    if kind == "trace":
        return {"kind": kind, "tris": _log_int(rng, 1000, 1000000), "rays": _log_int(rng, 1000, 1 << 22),
                "watertight": rng.random() < 0.5, "host": rng.random() < 0.3}
    if kind == "rebuild":
        n = _log_int(rng, 1000, 1000000)
        return {"kind": kind, "tris": n, "rays": max(1, n // 4)}
    if kind == "render":
        if rng.random() < 0.5:
            return {"kind": kind, "scene": "cornell", "width": _log_int(rng, 48, 512),
                    "height": _log_int(rng, 48, 512), "spp": rng.choice([1, 4, 16]), "depth": rng.choice([5, 8, 12]),
                    "compat": rng.random() < 0.4}
        return {"kind": kind, "scene": "terrain", "grid": _log_int(rng, 64, 1024), "spheres": _log_int(rng, 16, 1024),
                "width": _log_int(rng, 128, 1920), "height": _log_int(rng, 128, 1080), "spp": rng.choice([1, 4, 8]),
                "depth": rng.choice([5, 8, 12]), "compat": False}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 12), "tris": _log_int(rng, 3000, 300000)}
    if kind == "denoise":
        return {"kind": kind, "width": _log_int(rng, 32, 1920), "height": _log_int(rng, 32, 1080),
                "mirrors": rng.choice([1, 2, 4, 8])}
    if kind == "train":
        return {"kind": kind, "n": rng.choice([1, 2, 4, 8, 16]), "h": 16 * rng.randint(1, 16),
                "w": 16 * rng.randint(1, 16)}
    w, h = _log_int(rng, 17, 1920), _log_int(rng, 17, 1080)
    if kind == "nlm":
        return {"kind": kind, "width": w, "height": h, "search": rng.randint(2, 10), "patch": rng.randint(1, 3)}
    if kind == "nlm_ref":
        return {"kind": kind, "width": min(w, 1279), "height": min(h, 719)}
    return {"kind": kind, "width": w, "height": h,
            "type": rng.choice([sg.TM_REINHARD, sg.TM_UNCHARTED2, sg.TM_ACES])}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _smooth(g, n, c, h, w, cells=12):
    """n smooth random images of c channels in [0, 1] (N, C, H, W)."""
    low = torch.rand((n, c, cells, cells), device="cuda", generator=g)
    return F.interpolate(low, size=(h, w), mode="bilinear", align_corners=True)


def _picture(g, n, h, w):
    """A noisy low-sample render: smooth radiance with a few bright regions, its noise and
    its variance, (N, H, W, 3) each."""
    clean = torch.exp(3.0 * _smooth(g, n, 3, h, w) - 2.0).permute(0, 2, 3, 1)
    var = (0.15 * clean) ** 2 * torch.exp(0.5 * torch.randn(clean.shape, device="cuda", generator=g))
    noisy = (clean + var.sqrt() * torch.randn(clean.shape, device="cuda", generator=g)).clamp_min(0.0)
    return clean.contiguous(), noisy.contiguous(), var.contiguous()


def _features(g, n, h, w):
    """First-hit features (N, H, W, 7): albedo, unit normal, 1 / (1 + distance)."""
    albedo = _smooth(g, n, 3, h, w, 24)
    normal = F.normalize(_smooth(g, n, 3, h, w, 16) - 0.5, dim=1)
    depth = _smooth(g, n, 1, h, w, 8)
    return torch.cat([albedo, normal, depth], 1).permute(0, 2, 3, 1).contiguous()


def _terrain(ctx, grid, spheres, seed):
    s = scenes.upload(ctx, scenes.heightfield(grid=grid, n_spheres=spheres, seed=seed, subdiv=3 if grid >= 512 else 2))
    s.build()
    return s


def _outputs(w, h):
    return {"mean": torch.empty((h, w, 3), device="cuda"), "var": torch.empty((h, w, 3), device="cuda"),
            "srgb": torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")}


def _batch_opts(case):
    """Triangle count, side and samples per pixel of each scene of a batch."""
    k = case["scenes"]
    for i in range(k):
        tris = int(1000 * (case["tris"] / 1000.0) ** (((5 * i) % k) / max(1, k - 1)))
        yield tris, (64, 256, 128, 512)[i % 4], (16, 4, 64)[i % 3]


def _film(case, seed):
    """A film's state (sums over 16 samples) as a checkpoint holds it."""
    g, n = _gen(seed), 16
    h, w = case["height"], case["width"]
    _, noisy, var = _picture(g, 1, h, w)
    s = (noisy[0] * n).double()
    m = s / n
    q = ((m * m + var[0].double() * (n - 1)) * n).float().double()
    aov = _features(g, 1, h, w)[0] * n
    return {"sum": s.cpu().numpy(), "sumsq": q.cpu().numpy(), "comp": np.zeros((h, w, 3), np.float32),
            "aov": aov.cpu().numpy(), "samples": n}


def _train_batch(case, seed):
    g = _gen(seed)
    n, h, w = case["n"], case["h"], case["w"]
    clean, noisy, var = _picture(g, n, h, w)
    noise = (var.sqrt() / (1.0 + noisy)).mean(-1, keepdim=True)
    return torch.cat([noisy, _features(g, n, h, w), noise], -1).contiguous(), clean


def _initial_params(seed):
    """A network at the start of its training: He-uniform weights, a small last layer, no
    biases; layer by layer the weights [9][cout][cin], then the biases."""
    rng, parts = np.random.default_rng(seed), []
    for i, (cin, cout, relu) in enumerate(sg.UNET_LAYERS):
        real = sg.UNET_FEATURES if i == 0 else cin
        w = rng.uniform(-1.0, 1.0, (9, cout, cin)) * math.sqrt(6.0 / (9 * real)) * (1.0 if relu else 0.1)
        w[:, :, real:] = 0.0
        parts += [w.reshape(-1), np.zeros(cout)]
    return np.concatenate(parts).astype(np.float32)


def _nlm_image(case, seed):
    _, noisy, var = _picture(_gen(seed), 1, case["height"], case["width"])
    return noisy[0].contiguous(), var[0].contiguous()


def _rgba_image(case, seed):
    rgb = _nlm_image(case, seed)[0]
    return torch.cat([rgb / (1.0 + rgb), torch.ones_like(rgb[..., :1])], -1).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    ctx = sg.Context(0)
    st = {"case": case, "ctx": ctx, "kind": kind}
    if kind in ("trace", "rebuild"):
        st["scene"] = ctx.upload_scene(sg.microbench_soup(seed, case["tris"]))
        st["scene"].build()
        n = case["rays"]
        if case.get("host"):
            st["rays"] = torch.from_numpy(sg.microbench_rays(seed + 1, n)).pin_memory()
            st["hits"] = torch.empty((n, 4), pin_memory=True)
        else:
            st["rays"] = torch.from_numpy(sg.microbench_rays(seed + 1, n)).cuda()
            st["hits"] = torch.empty((n, 4), device="cuda")
    elif kind == "render":
        if case["scene"] == "cornell":
            d = scenes.cornell("specular" if case["compat"] else "mixed")
            d["camera"]["pos"] = (0.5 + 0.01 * ((seed % 17) / 17.0 - 0.5), 0.5, -1.4)
            st["scene"] = scenes.upload(ctx, d)
            st["scene"].build()
        else:
            st["scene"] = _terrain(ctx, case["grid"], case["spheres"], seed)
        st["out"] = _outputs(case["width"], case["height"])
        st["opts"] = {"width": case["width"], "height": case["height"], "spp": case["spp"],
                      "max_depth": case["depth"], "seed": seed,
                      "profile": sg.PROFILE_COMPAT if case["compat"] else sg.PROFILE_PHYSICAL}
    elif kind == "batch":
        st["scenes"], st["opts"], st["outs"] = [], [], []
        for i, (tris, side, spp) in enumerate(_batch_opts(case)):
            if i % 2:
                grid = max(8, int(math.sqrt(0.3 * tris)))
                s = _terrain(ctx, grid, max(1, (tris - 2 * grid * grid) // 320), seed + i)
            else:
                s = scenes.upload(ctx, scenes.soup(tris, seed=seed + i))
                s.build()
            st["scenes"].append(s)
            st["opts"].append({"width": side, "height": side, "spp": spp, "max_depth": 8, "seed": seed + i})
            st["outs"].append({k: v for k, v in _outputs(side, side).items() if k != "srgb"})
    elif kind == "denoise":
        st["net"] = sg.Unet(ctx)
        load_weights(st["net"], DEFAULT_WEIGHTS)
        st["scene"] = scenes.upload(ctx, scenes.cornell())
        st["scene"].build()
        st["scene"].restore(_film(case, seed), case["width"], case["height"])
        st["out"] = torch.empty((case["height"], case["width"], 3), device="cuda")
    elif kind == "train":
        st["net"] = sg.Unet(ctx)
        st["net"].set_params(_initial_params(seed))
        st["features"], st["target"] = _train_batch(case, seed)
        st["grads"] = torch.empty(st["net"].n_params, device="cuda")
    elif kind == "nlm":
        st["rgb"], st["var"] = _nlm_image(case, seed)
        st["out"] = torch.empty_like(st["rgb"])
    elif kind == "nlm_ref":
        st["rgba"] = _rgba_image(case, seed)
        st["out"] = torch.empty_like(st["rgba"])
    elif kind == "tonemap":
        st["rgb"] = _nlm_image(case, seed)[0]
        st["out"] = torch.empty_like(st["rgb"])
        st["srgb"] = torch.empty(st["rgb"].shape, dtype=torch.uint8, device="cuda")
        st["ave"], st["max"] = ctypes.c_float(), ctypes.c_float()
    return st


# ---------------------------------------------------------------- one pass
def _hits(hits):
    """Hit records (t, id, u, v) as their columns, the ids as integers."""
    return {"t": hits[:, 0], "id": hits.view(torch.int32)[:, 1], "uv": hits[:, 2:]}


def run(st):
    case, ctx, kind = st["case"], st["ctx"], st["kind"]
    if kind == "trace":
        st["scene"].trace_raw(st["rays"], st["hits"], watertight=case["watertight"])
        return _hits(st["hits"])
    if kind == "rebuild":
        st["scene"].build()
        st["scene"].trace_raw(st["rays"], st["hits"])
        return _hits(st["hits"])
    if kind == "render":
        st["scene"].render(out=st["out"], **st["opts"])
        return st["out"]
    if kind == "batch":
        ctx.render_batch(st["scenes"], st["opts"])
        for s, o, d in zip(st["scenes"], st["opts"], st["outs"]):
            s.read(o["width"], o["height"], want=("mean", "var"), out=d)
        return st["outs"]
    if kind == "denoise":
        return st["net"].denoise_film(st["scene"], out=st["out"], mirrors=case["mirrors"])
    if kind == "train":
        # lr = 0: the loss and the gradients alone (gradient accumulation, an optimiser of the
        # caller's own); with an update one pass's rounding would enter the next pass's weights
        loss = st["net"].train_step(st["features"], st["target"], lr=0.0)
        ctx.check(sg.lib().salty_unet_get_params(ctx.h, st["net"].h, 0, st["grads"].data_ptr()), "get_params")
        return {"loss": np.float32(loss), "grads": st["grads"]}
    if kind == "nlm":
        return ctx.nlm(st["rgb"], st["var"], case["search"], case["patch"], out=st["out"])
    if kind == "nlm_ref":
        # the C entry point: device arrays stay on the device
        ctx.check(sg.lib().salty_denoise_nlm_ref(ctx.h, case["width"], case["height"], 0.1, st["rgba"].data_ptr(),
                                                 st["out"].data_ptr()), "nlm_ref")
        return st["out"]
    ctx.check(sg.lib().salty_tonemap(ctx.h, case["type"], case["width"], case["height"], st["rgb"].data_ptr(),
                                     st["out"].data_ptr(), st["srgb"].data_ptr(), 1, ctypes.byref(st["ave"]),
                                     ctypes.byref(st["max"])), "tonemap")
    return {"rgb": st["out"], "srgb": st["srgb"], "max": np.float32(st["max"].value)}


# ---------------------------------------------------------------- what a pass cannot do without
_UNET_MACS = sum(9 * cin * cout / 4.0 ** lv for (cin, cout, _), lv in
                 zip(sg.UNET_LAYERS, (0, 0, 1, 1, 2, 2, 3, 3, 4, 3, 2, 1, 0, 0)))  # per full-resolution pixel


def work(case):
    kind = case["kind"]
    if kind in ("trace", "rebuild"):
        # rays in, hits out, the triangles once (a rebuild also writes them in leaf order)
        return {"bytes": case["rays"] * 48 + case["tris"] * (36 + (48 if kind == "rebuild" else 0)), "flops": 0}
    if kind == "render":
        tris = 36 if case["scene"] == "cornell" else 2 * case["grid"] ** 2 + 1280 * case["spheres"]
        return {"bytes": case["width"] * case["height"] * (12 + 12 + 3) + tris * 36, "flops": 0}
    if kind == "batch":
        return {"bytes": sum(t * 36 + r * r * 24 for t, r, _ in _batch_opts(case)), "flops": 0}
    if kind == "denoise":
        px = case["width"] * case["height"]
        return {"bytes": px * (24 + 28 + 12), "flops": 2 * _UNET_MACS * px * case["mirrors"]}
    if kind == "train":
        px = case["n"] * case["h"] * case["w"]
        first = 9 * 16 * 32  # the first layer has no input gradient
        return {"bytes": px * 4 * (sg.UNET_FEATURES + 3), "flops": 2 * px * (3 * _UNET_MACS - first)}
    px = case["width"] * case["height"]
    if kind == "nlm":
        # per offset and pixel: the normalised squared difference of three channels (about 8
        # operations each), a separable box sum, the weight and three weighted sums
        return {"bytes": px * 36, "flops": px * (2 * case["search"] + 1) ** 2 * (24 + 4 * case["patch"] + 10)}
    if kind == "nlm_ref":
        return {"bytes": px * 32, "flops": px * 169 * (11 + 8 + 11)}
    return {"bytes": px * (12 + 12 + 3), "flops": 0}


# ---------------------------------------------------------------- 64-bit results
def _double(p):
    return torch.from_numpy(p.astype(np.float64)).cuda()


def _net(p, x):
    """The U-Net's correction for inputs x (N, 16, H, W) in 64 bits; p: the parameters."""
    layers, off = [], 0
    for cin, cout, relu in sg.UNET_LAYERS:
        w = p[off:off + 9 * cin * cout].reshape(3, 3, cout, cin).permute(2, 3, 0, 1)
        off += 9 * cin * cout
        layers.append((w, p[off:off + cout], relu))
        off += cout

    def conv(i, t):
        w, b, relu = layers[i]
        t = F.conv2d(t, w, b, padding=1)
        return F.relu(t) if relu else t

    def up(t):
        return t.repeat_interleave(2, -1).repeat_interleave(2, -2)

    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.max_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.max_pool2d(e1, 2)))
    e3 = conv(7, conv(6, F.max_pool2d(e2, 2)))
    d = conv(8, F.max_pool2d(e3, 2))
    for i, skip in ((9, e3), (10, e2), (11, e1), (12, e0)):
        d = conv(i, torch.cat([up(d), skip], 1))
    return conv(13, d)[:, :3]


def _net_input(f):
    """(N, H, W, 11) features -> (N, 16, H, W): log colour first, zero padding last."""
    f = f.double().permute(0, 3, 1, 2)
    return torch.cat([torch.log1p(f[:, :3].clamp_min(0.0)), f[:, 3:], torch.zeros_like(f[:, :5])], 1)


def _exact_denoise(case, seed):
    film, p = _film(case, seed), _double(np.load(DEFAULT_WEIGHTS)["params"])
    h, w, n = case["height"], case["width"], film["samples"]
    s, q = (torch.from_numpy(film[k]).cuda() for k in ("sum", "sumsq"))
    mean = s / n
    var = ((q / n - mean * mean) / (n - 1.0)).clamp_min(0.0)
    noise = (var.sqrt() / (1.0 + mean.clamp_min(0.0))).mean(-1, keepdim=True)
    frame = torch.cat([mean, torch.from_numpy(film["aov"]).cuda().double() / n, noise], -1)
    ph, pw = (-h) % 16, (-w) % 16
    total = torch.zeros_like(mean)
    for k in range(case["mirrors"]):
        flips = ([1] if k & 1 else []) + ([0] if k & 2 else [])
        f = frame.flip(flips) if flips else frame
        ys = [y if y < h else max(2 * h - 2 - y, 0) for y in range(h + ph)]
        xs = [x if x < w else max(2 * w - 2 - x, 0) for x in range(w + pw)]
        f = f[torch.tensor(ys, device="cuda")][:, torch.tensor(xs, device="cuda")]
        if k & 4:
            f = f.transpose(0, 1)
        x = _net_input(f[None].contiguous())
        y = torch.expm1(x[:, :3] + _net(p, x))[0].permute(1, 2, 0).clamp_min(0.0)
        if k & 4:
            y = y.transpose(0, 1)
        y = y[:h, :w]
        total += (y.flip(flips) if flips else y) / case["mirrors"]
    return total


def _exact_train(case, seed):
    feat, target = _train_batch(case, seed)
    p = _double(_initial_params(seed)).requires_grad_(True)
    total, loss = case["n"] * case["h"] * case["w"] * 3, 0.0
    for i in range(case["n"]):  # one image at a time: the graph of all of them is large
        x = _net_input(feat[i:i + 1])
        t = torch.log1p(target[i:i + 1].double().permute(0, 3, 1, 2).clamp_min(0.0))
        part = (x[:, :3] + _net(p, x) - t).abs().sum() / total
        part.backward()
        loss += float(part.detach())
    return {"loss": loss, "grads": p.grad}


def _shift(a, ys, xs):
    return a[ys][:, xs]


def _exact_nlm(case, seed):
    rgb, var = (t.double() for t in _nlm_image(case, seed))
    h, w, R, P, k = case["height"], case["width"], case["search"], case["patch"], 0.45
    ay = torch.arange(-P, h + P, device="cuda")
    ax = torch.arange(-P, w + P, device="cuda")
    cy, cx = ay.clamp(0, h - 1), ax.clamp(0, w - 1)
    a, va = _shift(rgb, cy, cx), _shift(var, cy, cx)
    y, x = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    out, tot = torch.zeros_like(rgb), torch.zeros((h, w, 1), dtype=torch.float64, device="cuda")
    for dy in range(-R, R + 1):
        for dx in range(-R, R + 1):
            qy, qx = (ay + dy).clamp(0, h - 1), (ax + dx).clamp(0, w - 1)
            b, vb = _shift(rgb, qy, qx), _shift(var, qy, qx)
            d = (((a - b) ** 2 - (va + torch.minimum(va, vb))) / (1e-10 + k * k * (va + vb))).sum(-1)
            d = F.avg_pool2d(d[None, None], 2 * P + 1, stride=1)[0, 0] / 3.0
            wt = torch.exp(-d.clamp_min(0.0))[..., None]
            out += wt * _shift(rgb, (y + dy).clamp(0, h - 1), (x + dx).clamp(0, w - 1))
            tot += wt
    return out / tot


def _exact_nlm_ref(case, seed):
    img = _rgba_image(case, seed).double()
    h, w, c = case["height"], case["width"], float(np.float32(0.1))
    ay, ax = torch.arange(-2, h + 2, device="cuda"), torch.arange(-2, w + 2, device="cuda")
    a = _shift(img, ay.clamp(0, h - 1), ax.clamp(0, w - 1))
    y, x = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    out, tot = torch.zeros_like(img), torch.zeros((h, w, 1), dtype=torch.float64, device="cuda")
    for dy in range(-6, 7):
        for dx in range(-6, 7):
            b = _shift(img, (ay + dy).clamp(0, h - 1), (ax + dx).clamp(0, w - 1))
            d = F.avg_pool2d(((a - b) ** 2).sum(-1)[None, None], 5, stride=1)[0, 0] * 25.0
            wt = torch.exp(-(d - 2.0 * c * c).clamp_min(0.0) / (c * c))[..., None]
            out += wt * _shift(img, (y + dy).clamp(0, h - 1), (x + dx).clamp(0, w - 1))
            tot += wt
    return out / tot


def _exact_tonemap(case, seed):
    x = _nlm_image(case, seed)[0].double()
    lw = (x * torch.tensor([0.299, 0.587, 0.114], dtype=torch.float64, device="cuda")).sum(-1)
    lw = torch.where(lw < float(np.finfo(np.float32).eps), torch.full_like(lw, 1e-5), lw)
    ave, top = math.exp(float(torch.log(lw + 1e-5).mean())), float(lw.max())
    key = (0.27 if case["type"] == sg.TM_ACES else 0.18) / ave

    def filmic(v):
        return (v * (0.15 * v + 0.05) + 0.002) / (v * (0.15 * v + 0.5) + 0.06) - 0.01 / 0.3

    v = x * key
    if case["type"] == sg.TM_ACES:
        a = v * 0.665406
        y = (v * (2.51 * a / 12.0 + 0.03)
             / (a / 12.0 * (2.43 * a + 0.59) + 0.14)).clamp(0.0, 1.0)
    elif case["type"] == sg.TM_UNCHARTED2:
        y = filmic(2.0 * v) / filmic(torch.tensor(11.2, dtype=torch.float64, device="cuda"))
    else:
        y = v * (1.0 + v / (top * key) ** 2) / (1.0 + v)
    return {"rgb": y, "srgb": None, "max": top}


def exact(case, seed):
    kind = case["kind"]
    if kind == "denoise":
        return _exact_denoise(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "nlm":
        return _exact_nlm(case, seed)
    if kind == "nlm_ref":
        return _exact_nlm_ref(case, seed)
    if kind == "tonemap":
        return _exact_tonemap(case, seed)
    return None  # hits and renders: walks and random paths, not a formula of the inputs
