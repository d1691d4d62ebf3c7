"""The workloads whose speed is tracked: calls of the public entry points as a user's program makes them.

Every case names its kind and its sizes:
  stereo    PMHuberStereo.disparity_map (levels > 1: the coarse-to-fine loop; fused: the contracted arithmetic)
  depth     PMHuberStereo.depth_map
  batch     PMHuberStereo.disparity_map_batch, uneven pairs in one call
  learned   PlaneProposal.propose for both views, then disparity_map from the two proposals
  vpm       VPMStereoCL.disparity_simple
  flow      SVPMFlowCL.flow
  gradients PlaneProposal.gradients: forward pass, loss and all gradients of one training batch

`radius` is the half-width of the matching window, `dispmax` the disparity (flow) range, `iters` the iteration
(pass) count that the caller asks for.  host: numpy images in, numpy maps out; otherwise CUDA tensors.

Images are procedural: slanted planar patches with four octaves of noise texture, the second view warped by the
patches' motion plus noise of standard deviation 2, RGBA8.  PatchMatch takes discrete decisions along the way, so
its maps have no value in exact arithmetic; the network's gradients have one.
"""
import math

import numpy as np
import torch

from cvt_b200 import learn
from cvt_b200.learn import PlaneProposal
from cvt_b200.stereo import PMHuberStereo
from cvt_b200.svpm import SVPMFlowCL
from cvt_b200.vpm import VPMStereoCL

# operations per pixel, window position and executed pass: the candidates' costs and the Gauss-Newton steps
# that a pass evaluates (early exits left out), measured once at 1280x720 with a 21x21 (flow: 7x7) window
OPS_STEREO, OPS_VPM, OPS_FLOW = 1007.0, 1118.0, 965.0


def listed():
    return [
        # a thumbnail-size pair: one small call, where the latency of a thread's own work counts
        dict(name="stereo_thumb", kind="stereo", width=64, height=48, radius=5, dispmax=16.0, iters=4, views=2, pp=1,
             levels=1, fused=False, host=False, planes=False),
        # QVGA, left view only, host images in and out: an interactive preview
        dict(name="stereo_qvga", kind="stereo", width=320, height=240, radius=7, dispmax=32.0, iters=4, views=1, pp=0,
             levels=1, fused=False, host=True, planes=False),
        # the headline: 1280x720, both views, left-right check
        dict(name="stereo_hd", kind="stereo", width=1280, height=720, radius=10, dispmax=128.0, iters=8, views=2, pp=1,
             levels=1, fused=False, host=False, planes=False),
        # a large image with the largest window in use (35x35), few iterations
        dict(name="stereo_wide", kind="stereo", width=1920, height=1080, radius=17, dispmax=192.0, iters=1, views=2,
             pp=1, levels=1, fused=False, host=False, planes=False),
        # odd sizes, coarse to fine over three levels, filled result
        dict(name="stereo_pyramid", kind="stereo", width=517, height=389, radius=6, dispmax=48.0, iters=3, views=2,
             pp=2, levels=3, fused=False, host=False, planes=False),
        # the training targets' recipe: 512x384, 11x11, fused arithmetic, both views' planes returned
        dict(name="stereo_fused", kind="stereo", width=512, height=384, radius=5, dispmax=64.0, iters=8, views=2, pp=1,
             levels=1, fused=True, host=False, planes=True),
        # depthMap at a ragged size
        dict(name="depth", kind="depth", width=643, height=361, radius=10, dispmax=64.0, iters=5, views=2, pp=1),
        # uneven pairs in one call, as a dataset sweep issues them
        dict(name="batch", kind="batch", pairs=6, size_seed=5, wmin=320, wmax=960, hmin=240, hmax=540, radius=10,
             iters=1),
        # a learned start and two iterations, 1280x720
        dict(name="learned_hd", kind="learned", width=1280, height=720, radius=10, dispmax=128.0, iters=2),
        # the one-view sibling, VGA
        dict(name="vpm_vga", kind="vpm", width=640, height=480, radius=10, dispmax=64.0, iters=8),
        # optical flow, VGA, the reference's 200 passes of a 7x7 window
        dict(name="flow_vga", kind="flow", width=640, height=480, radius=3, dispmax=64.0, iters=200),
        # one batch of the proposal network's training recipe: 32 maps of 96x128
        dict(name="gradients", kind="gradients", maps=32, rows=96, cols=128),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        kind = rng.choice(["stereo", "stereo", "stereo", "stereo", "depth", "batch", "learned", "vpm", "flow", "gradients"])
        W, H = size(48, 1920), size(32, 1080)
        dm = float(max(16, round(W * rng.uniform(0.05, 0.12))))
        c = dict(kind=kind, width=W, height=H, radius=rng.randint(2, 17), dispmax=dm, iters=rng.randint(1, 9))
        if kind == "stereo":
            views = rng.choice([2, 2, 1])
            levels = rng.choice([1, 1, 1, 2, 3]) if min(W, H) >= 96 else 1
            c.update(views=views, pp=rng.randint(0, 2) if views == 2 else 0, levels=levels,
                     fused=rng.random() < 0.25, host=rng.random() < 0.25, planes=rng.random() < 0.3)
        elif kind == "depth":
            c.update(views=2, pp=rng.randint(0, 2))
        elif kind == "batch":
            c = dict(kind=kind, pairs=rng.randint(2, 12), size_seed=rng.randint(0, 9999), wmin=96, wmax=max(128, W),
                     hmin=64, hmax=max(96, H), radius=rng.randint(3, 10), iters=rng.randint(1, 4))
        elif kind == "learned":
            c.update(width=max(W, 128), height=max(H, 96), iters=rng.randint(1, 4))
            c["dispmax"] = float(max(32, round(c["width"] * 0.1)))
        elif kind == "flow":
            c.update(radius=rng.randint(1, 5), iters=size(20, 200))
        elif kind == "gradients":
            c = dict(kind=kind, maps=size(1, 32), rows=rng.randint(24, 96), cols=rng.randint(32, 128))
        if work(c)["flops"] <= work(listed()[2])["flops"]:
            return c


def batch_sizes(c):
    g = np.random.default_rng(c["size_seed"])
    return [(int(g.integers(c["wmin"], c["wmax"] + 1)), int(g.integers(c["hmin"], c["hmax"] + 1)))
            for _ in range(c["pairs"])]


def work(c):
    if c["kind"] == "gradients":
        px = c["maps"] * c["rows"] * c["cols"]
        macs = sum(9 * ci * co for ci, co, _ in learn.layer_shapes())
        first = 9 * learn.layer_shapes()[0][0] * learn.layer_shapes()[0][1]
        # forward, weight gradient, and the data gradient of all layers but the first
        return {"bytes": px * (16 * 2 + 16) + 4 * 2 * macs, "flops": 2.0 * px * (3 * macs - first)}
    if c["kind"] == "batch":
        px = sum(w * h for w, h in batch_sizes(c))
    else:
        px = c["width"] * c["height"]
    win = (2 * c["radius"] + 1) ** 2
    if c["kind"] == "vpm":
        return {"bytes": 12 * px, "flops": px * win * c["iters"] * OPS_VPM}
    if c["kind"] == "flow":
        return {"bytes": 16 * px, "flops": px * win * c["iters"] * OPS_FLOW}
    done = c["iters"] if c["kind"] == "depth" else c["iters"] | 1
    out = 4 + (32 if c.get("planes") else 0)
    return {"bytes": (8 + out) * px, "flops": px * win * done * c.get("views", 2) * OPS_STEREO}


def _noise(g, H, W, period):
    """RGB value noise of one octave: a random grid of the given period, interpolated"""
    gh, gw = int(H / period) + 3, int(W / period) + 3
    t = torch.from_numpy(g.random((1, 3, gh, gw), dtype=np.float32)).cuda()
    ys = torch.arange(H, device="cuda") / period
    xs = torch.arange(W, device="cuda") / period
    yy, xx = torch.meshgrid(ys * 2 / (gh - 1) - 1, xs * 2 / (gw - 1) - 1, indexing="ij")
    return torch.nn.functional.grid_sample(t, torch.stack([xx, yy], -1)[None], align_corners=True)[0]


def _scene(seed, W, H, lo, hi, vertical=False):
    """two (H, W, 4) uint8 CUDA images and the (3, H, W) motion (d, slope in x, slope in y) of the second"""
    g = np.random.default_rng(seed)
    pad = int(hi) + 2
    tex = sum(_noise(g, H + 2 * pad, W + 2 * pad, 24.0 / 2 ** o) * 0.5 ** o for o in range(4)) * (255.0 / 1.875)
    k = int(g.integers(8, 40))
    py, px = torch.from_numpy(g.random(k) * H).cuda(), torch.from_numpy(g.random(k) * W).cuda()
    y, x = torch.meshgrid(torch.arange(H, device="cuda", dtype=torch.float64),
                          torch.arange(W, device="cuda", dtype=torch.float64), indexing="ij")
    best = torch.full((H, W), 1e30, device="cuda", dtype=torch.float64)
    d = torch.zeros_like(best)
    v = torch.zeros_like(best)
    sx, sy = torch.zeros_like(best), torch.zeros_like(best)
    p = g.random((k, 4))
    for i in range(k):
        r2 = (x - px[i]) ** 2 + (y - py[i]) ** 2
        m = r2 < best
        best = torch.where(m, r2, best)
        gx, gy = 0.4 * p[i, 1] - 0.2, 0.4 * p[i, 2] - 0.2
        di = (lo + (hi - lo) * p[i, 0] + gx * (x - px[i]) + gy * (y - py[i])).clamp(lo, hi)
        d, v = torch.where(m, di, d), torch.where(m, torch.full_like(v, (p[i, 3] - 0.5) * 0.5 * hi), v)
        sx, sy = torch.where(m, torch.full_like(sx, gx), sx), torch.where(m, torch.full_like(sy, gy), sy)
    if not vertical:
        v = torch.zeros_like(v)
    gw, gh = W + 2 * pad - 1, H + 2 * pad - 1
    at = torch.stack([(x + pad + d) * 2 / gw - 1, (y + pad + v) * 2 / gh - 1], -1).float()[None]
    second = torch.nn.functional.grid_sample(tex[None], at, align_corners=True)[0]
    first = tex[:, pad:pad + H, pad:pad + W]
    noise = torch.Generator(device="cuda").manual_seed(int(seed))
    second = second + 2.0 * torch.randn(second.shape, generator=noise, device="cuda")
    out = []
    for im in (first, second):
        a = torch.full((H, W, 4), 255, dtype=torch.uint8, device="cuda")
        a[..., :3] = im.permute(1, 2, 0).round().clamp(0, 255).to(torch.uint8)
        out.append(a)
    return out[0], out[1], torch.stack([d, sx, sy]).float()


def prepare(c, seed):
    s = {"case": c}
    if c["kind"] == "batch":
        s["sizes"] = batch_sizes(c)
        s["dmax"] = [float(max(32, w // 10)) for w, _ in s["sizes"]]
        im = [_scene(seed * 1000 + i, w, h, 2.0, 0.9 * dm)[:2] for i, ((w, h), dm) in enumerate(zip(s["sizes"], s["dmax"]))]
        s["left"], s["right"] = [a for a, _ in im], [b for _, b in im]
        s["pm"] = PMHuberStereo()
        return s
    if c["kind"] == "gradients":
        s["net"] = PlaneProposal.load(learn.default_weights())
        xs, ts = [], []
        g = np.random.default_rng(seed)
        for i in range(0, c["maps"], 8):   # eight crops of each scene
            n = min(8, c["maps"] - i)
            a, b, m = _scene(seed * 1000 + i, 4 * c["cols"] + 64, 4 * c["rows"] + 64, 2.0, 58.0)
            for _ in range(n):
                oy, ox = int(g.integers(0, 65)), int(g.integers(0, 65))
                cut = (slice(oy, oy + 4 * c["rows"]), slice(ox, ox + 4 * c["cols"]))
                xs.append(s["net"].net_input(a[cut].contiguous(), b[cut].contiguous(), 4))
                t = torch.nn.functional.avg_pool2d(m[(slice(None),) + cut][None], 4)[0]
                nz = 1.0 / torch.sqrt(1.0 + t[1] ** 2 + t[2] ** 2)
                ok = torch.from_numpy((g.random((c["rows"], c["cols"])) < 0.8).astype(np.float32)).cuda()
                ts.append(torch.stack([t[0] / 4 * ok, -t[1] * nz * ok, -t[2] * nz * ok, ok], -1)[None])
        s["x"], s["t"] = torch.cat(xs), torch.cat(ts)
        s["count"] = int((s["t"][..., 3] > 0).sum())
        return s
    W, H, dm = c["width"], c["height"], c["dispmax"]
    s["left"], s["right"], _ = _scene(seed, W, H, 2.0 if dm > 16 else 1.0, 0.9 * dm if c["kind"] != "flow" else 0.2 * dm,
                                      vertical=c["kind"] == "flow")
    if c["kind"] == "vpm":
        s["vpm"] = VPMStereoCL(c["radius"], c["iters"], dm)
    elif c["kind"] == "flow":
        s["flow"] = SVPMFlowCL()
    elif c["kind"] == "learned":
        s["net"] = PlaneProposal.load(learn.default_weights())
        s["pm"] = PMHuberStereo()
    else:
        s["pm"] = PMHuberStereo(views=c["views"], fused=c.get("fused", False), levels=c.get("levels", 1))
        if c.get("host"):
            s["left"], s["right"] = s["left"].cpu().numpy(), s["right"].cpu().numpy()
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "stereo":
        return s["pm"].disparity_map(s["left"], s["right"], c["radius"], c["dispmax"], c["iters"], pp=c["pp"],
                                     planes=c["planes"])
    if c["kind"] == "depth":
        return s["pm"].depth_map(s["left"], s["right"], c["radius"], c["dispmax"], c["iters"], pp=c["pp"],
                                 normalmap=True)
    if c["kind"] == "batch":
        n = len(s["left"])
        return s["pm"].disparity_map_batch(s["left"], s["right"], [c["radius"]] * n, s["dmax"], c["iters"])
    if c["kind"] == "learned":
        dl, nl = s["net"].propose(s["left"], s["right"], c["dispmax"], view=0)
        dr, nr = s["net"].propose(s["left"], s["right"], c["dispmax"], view=1)
        d = s["pm"].disparity_map(s["left"], s["right"], c["radius"], c["dispmax"], c["iters"], initdisparity=dl,
                                  initnormalmap=nl, initdisparity_right=dr, initnormalmap_right=nr)
        return {"dmap": d, "proposal": dl, "normal": nl}
    if c["kind"] == "vpm":
        return s["vpm"].disparity_simple(s["left"], s["right"])
    if c["kind"] == "flow":
        return s["flow"].flow(s["left"], s["right"], c["radius"], c["dispmax"], iterations=c["iters"])
    loss, grads = s["net"].gradients(s["x"], s["t"], s["count"])
    return {"loss": loss, "grads": grads}


def exact(c, seed):
    """the gradients in 64-bit arithmetic from the BF16 weights that the forward pass multiplies by"""
    if c["kind"] != "gradients":
        return None
    s = prepare(c, seed)
    h = s["x"].double().permute(0, 3, 1, 2)
    params = []
    for l, (ci, co, dil) in enumerate(learn.layer_shapes()):
        p = s["net"].p[l]
        w = p[:co * 9 * ci].to(torch.bfloat16).double().reshape(co, 3, 3, ci).requires_grad_()
        b = p[co * 9 * ci:].double().requires_grad_()
        params.append((w, b))
        h = torch.nn.functional.conv2d(h, w.permute(0, 3, 1, 2), b, padding=dil, dilation=dil)
        if l < learn.NL - 1:
            h = torch.relu(h)
    e = (h.permute(0, 2, 3, 1)[..., :3] - s["t"][..., :3].double()).abs()
    weight = torch.tensor([1.0, learn.WN, learn.WN], device=e.device, dtype=torch.float64)
    loss = ((e * weight).sum(-1) * (s["t"][..., 3] > 0)).sum() / s["count"]
    g = torch.autograd.grad(loss, [t for p in params for t in p])
    return {"loss": loss.detach(), "grads": [torch.cat([g[2 * l].flatten(), g[2 * l + 1]]) for l in range(learn.NL)]}
