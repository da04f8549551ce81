"""The work that users of gbpt have it do, as timed cases.

Rendering is most of it: one progressive pass of an interactive view, whole
images at a few samples per pixel, every renderer mode, small, ordinary and
large frames, round and ragged sizes, on the three procedural scenes (36 to
332,180 triangles).  Beside it stand the library's other entry points: rays
traced for a caller, the bilateral filter on the caller's planes, the
learned allocator's training and inference, and a batch of requests served
at once.

A case is a dict of plain values; its "kind" names the family:

  render  RTRenderer: `passes` progressive passes, restarted first when
          `restart` is set; mode 0 "BDPTSC", 1 "Adap Bilat PLL", 2 "Adap
          Bilat Binary", 3 "Bilaterial" (filter-only), 4 "PTSC"
  rays    gbpt_trace_rays on device arrays, or RTScene.trace_rays on host ones
  filter  gbpt_bilateral on device planes
  mlp     MLP.gradients of a batch and MLP.forward of an image's tiles
  serve   a Server's batch of requests of mixed size
"""
import ctypes
import math

import numpy as np
import torch

import cudapt_gb300 as gb
from cudapt_gb300 import _native, mlp, scenes, serving

# scene name -> generator, its arguments, triangles
SCENES = {
    "cornell": (scenes.cornell, {}, 36),
    "interior": (scenes.interior, {"level": 2}, 57_614),
    "interior_fine": (scenes.interior, {"level": 3}, 230_414),
    "hall": (scenes.hall, {}, 332_180),
}
_arrays = {}


def _scene_arrays(name):
    """Geometry, materials and camera of a scene: read once, as a program loads its model file once."""
    if name not in _arrays:
        make, kw, _ = SCENES[name]
        _arrays[name] = make(**kw)
    return _arrays[name]


def _build(name):
    (v, t, m), _ = _scene_arrays(name)
    return gb.RTScene(v, t, m).build_bvh()


def _view(name, rng):
    """The scene's camera moved a little: a view of its own for every seed."""
    _, cam = _scene_arrays(name)
    size = 0.02 if name == "cornell" else 0.4
    pos = np.array(cam["pos"], np.float64) + size * (rng.random(3) - 0.5)
    d = np.array(cam["dir"], np.float64) + 0.06 * (rng.random(3) - 0.5)
    return dict(pos=tuple(pos), dir=tuple(d / np.linalg.norm(d)), up=cam["up"], fov=cam["fov"])


def listed():
    return [
        # the smallest call: one pass of a thumbnail view, the image on the host; launches and latency count
        dict(name="cornell_64_pass", kind="render", scene="cornell", width=64, height=64, mode=0, depth=8, env=0.0,
             passes=1, restart=False, radius=5),
        # a small whole image: 16 samples per pixel of the Cornell box from a new start
        dict(name="cornell_256_image", kind="render", scene="cornell", width=256, height=256, mode=0, depth=8, env=0.0,
             passes=16, restart=True, radius=5),
        # an interactive view of a large interior: one deep progressive pass with an environment
        dict(name="interior_768p_pass", kind="render", scene="interior_fine", width=1024, height=768, mode=0, depth=10,
             env=0.1, passes=1, restart=False, radius=5),
        # the headline view: one pass of the largest scene at 720p
        dict(name="hall_720p_pass", kind="render", scene="hall", width=1280, height=720, mode=0, depth=5, env=0.0,
             passes=1, restart=False, radius=5),
        # an adaptive image: 8 uniform then 4 budgeted passes, the guide filter at radius 4
        dict(name="hall_720p_adaptive", kind="render", scene="hall", width=1280, height=720, mode=1, depth=5, env=0.0,
             passes=12, restart=True, radius=4),
        # the binary allocator at a ragged size: 5 uniform then 3 budgeted passes
        dict(name="interior_500_binary", kind="render", scene="interior", width=500, height=375, mode=2, depth=6,
             env=0.0, passes=8, restart=True, radius=5),
        # the filter-only mode: 5 traced passes, each filtered, at a ragged size
        dict(name="interior_641_bilat", kind="render", scene="interior", width=641, height=359, mode=3, depth=5,
             env=0.0, passes=5, restart=True, radius=5),
        # the unidirectional mode at an odd size
        dict(name="interior_333_ptsc", kind="render", scene="interior", width=333, height=217, mode=4, depth=10,
             env=0.0, passes=8, restart=True, radius=5),
        # rays of the caller's own (picking, baking, visibility): a million in device arrays
        dict(name="hall_rays_device", kind="rays", scene="hall", rays=1_000_003, device=True),
        # the bilateral filter on the caller's planes: four features, a wide window, a ragged image
        dict(name="filter_1003_r9", kind="filter", width=1003, height=617, radius=9, emit=True),
        # the learned allocator: a training batch's gradients, then every 8x8 tile of a 720p image
        dict(name="mlp_4096", kind="mlp", batch=4096, tiles=14_400),
        # requests of mixed size served at once, two of each of four sizes
        dict(name="serve_mixed", kind="serve", requests=8, frames=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 8 + ["rays"] * 2 + ["filter"] * 2 + ["mlp", "serve"])
    if kind == "render":
        mode = rng.choice([0, 0, 0, 1, 2, 3, 4])
        width = _log_int(rng, 48, 1280)
        height = max(32, min(1024, int(width * rng.uniform(0.5, 1.1))))
        restart = mode != 0 or rng.random() < 0.5
        passes = rng.randint(6, 10) if mode in (1, 2) else rng.randint(2, 6) if mode == 3 else rng.randint(1, 8)
        while passes > 1 and width * height * passes > 6_000_000:
            passes -= 1
        return dict(kind="render", scene=rng.choice(sorted(SCENES)), width=width, height=height, mode=mode,
                    depth=rng.randint(3, 10) if mode != 1 else rng.randint(3, 6), env=rng.choice([0.0, 0.1]),
                    passes=passes, restart=restart, radius=rng.randint(2, 6))
    if kind == "rays":
        device = rng.random() < 0.7
        return dict(kind="rays", scene=rng.choice(sorted(SCENES)), device=device,
                    rays=_log_int(rng, 1000, 1_500_000 if device else 300_000))
    if kind == "filter":
        radius = rng.randint(1, 12)
        width = _log_int(rng, 64, 1280)
        return dict(kind="filter", width=width, height=max(48, min(900, int(width * rng.uniform(0.5, 1.0)))),
                    radius=radius, emit=rng.random() < 0.5)
    if kind == "mlp":
        return dict(kind="mlp", batch=_log_int(rng, 256, 8192), tiles=_log_int(rng, 100, 20_000))
    return dict(kind="serve", requests=rng.randint(4, 12), frames=rng.randint(2, 4))


# --- render -----------------------------------------------------------------


def _params(case, seed):
    # the adaptive modes trace this many uniform passes first
    warm = 8 if case["passes"] > 8 else 5
    return gb.default_params(seed=seed & 0x7FFFFFFF, eye_depth_max=case["depth"], light_depth_max=case["depth"],
                             pt_depth_max=case["depth"], env=(case["env"],) * 3, warmup_frames=warm,
                             filter_radius=case["radius"], bilat_radius=case["radius"], render_iterations=0)


def _prepare_render(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    cam = _view(case["scene"], rng)
    cam = gb.camera(cam["pos"], cam["dir"], cam["up"], cam["fov"])
    renderer = gb.RTRenderer(case["width"], case["height"], case["mode"], _params(case, seed))
    return dict(renderer=renderer, scene=_build(case["scene"]), cam=cam)


def _run_render(case, s):
    r = s["renderer"]
    if case["restart"]:
        r.reset()
    if case["passes"] > 1:
        r.render_frames(s["scene"], s["cam"], case["passes"] - 1, stats=False)
    return r.render(s["scene"], s["cam"], stats=case["passes"] == 1)


def _render_work(scene, pixels, passes, depth):
    """A path walks at most `depth` extension rays and as many connections; half of them are a fair floor.  A walk
    cannot do with fewer than about two box tests a level (24 operations each) and two triangle tests (50); a
    vertex is about 300 operations.  The scene (boxes, triangles, shading records) is read once, the image and its
    sample counts are read and written once a pass."""
    tris = SCENES[scene][2]
    rays = pixels * passes * max(2, depth)
    flops = rays * (2 * 24 * math.log2(max(tris, 2)) + 100) + 0.5 * rays * 300
    return flops, tris * (2 * 32 + 48 + 80) + pixels * passes * 2 * 16


# --- rays ---------------------------------------------------------------------


def _prepare_rays(case, seed):
    """Origins in the scene's box, directions over the sphere."""
    (v, _, _), _ = _scene_arrays(case["scene"])
    lo, hi = v["pos"].min(0).astype(np.float64), v["pos"].max(0).astype(np.float64)
    g = torch.Generator("cuda").manual_seed(seed)
    n = case["rays"]
    lo, hi = (torch.tensor(x, device="cuda") for x in (lo, hi))
    o = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g, dtype=torch.float64)
    d = torch.randn(n, 3, device="cuda", generator=g, dtype=torch.float64)
    rays = torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).float().contiguous()
    state = dict(scene=_build(case["scene"]))
    if case["device"]:
        state["rays"] = rays
        state["out"] = {k: torch.zeros(n, device="cuda") for k in ("t", "w", "u", "v")}
        state["out"]["tri"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    else:
        state["rays"] = rays.cpu().numpy()
    return state


def _run_rays(case, s):
    if not case["device"]:
        return s["scene"].trace_rays(s["rays"], eps=1e-4)
    o = s["out"]
    _native.check(_native.load().gbpt_trace_rays(
        s["scene"].handle, s["rays"].data_ptr(), case["rays"], 1e20, 1e-4, 0, o["t"].data_ptr(), o["tri"].data_ptr(),
        o["w"].data_ptr(), o["u"].data_ptr(), o["v"].data_ptr(), None, None, 1))
    return o


def _exact_rays(case, seed):
    """The closest hit's distance by testing every triangle in 64 bits (barycentrics of a shared edge may belong to
    either neighbour, so only the distance has one value)."""
    (v, t, _), _ = _scene_arrays(case["scene"])
    if case["rays"] * len(t) > 6e10:
        return None
    rays = _prepare_rays(case, seed)["rays"]
    rays = torch.as_tensor(rays, device="cuda").double()
    pos = torch.tensor(v["pos"], device="cuda").double()
    idx = torch.tensor(np.stack([t["v0"], t["v1"], t["v2"]], 1).astype(np.int64), device="cuda")
    p0 = pos[idx[:, 0]]
    e0, e1 = (pos[idx[:, 1]] - p0), (pos[idx[:, 2]] - p0)
    push = float(np.float32(1e-4))
    out = torch.empty(len(rays), dtype=torch.float64, device="cuda")
    step = max(1, int(1.5e7 // len(t)))
    # u, v and t of Moeller and Trumbore as triple products, each a matrix product of ray and triangle terms
    nrm = torch.linalg.cross(e0, e1)
    for i in range(0, len(rays), step):
        o, d = rays[i:i + step, :3] + push * rays[i:i + step, 3:], rays[i:i + step, 3:]
        m = torch.linalg.cross(o, d)  # moment of the ray's line
        div = -d @ nrm.T
        div = torch.where(div.abs() < 1e-9, torch.full_like(div, math.nan), div)
        dist = (o @ nrm.T - (p0 * nrm).sum(1)) / div
        a0, a1 = torch.linalg.cross(p0, e0), torch.linalg.cross(p0, e1)
        u = (m @ e1.T + d @ a1.T) / div
        w = -(m @ e0.T + d @ a0.T) / div
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (dist >= 0)
        best = torch.where(ok, dist, torch.full_like(dist, math.inf)).min(dim=1).values
        out[i:i + step] = torch.where(torch.isinf(best), torch.full_like(best, -1.0), best)
    t_out = out if case["device"] else out.cpu().numpy()
    return dict(t=t_out, tri=None, w=None, u=None, v=None)


# --- filter -------------------------------------------------------------------

DELTAS = dict(color=50.0, pos=1.0, norm=0.25, emit=0.5)


def _planes(case, seed):
    """Planes such as a noisy pass writes: surfaces of blocks with their own depth and normal, colours with a few
    very bright pixels, emission on a few blocks."""
    W, H = case["width"], case["height"]
    g = torch.Generator("cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(*shape, device="cuda", generator=g)

    by, bx = H // 37 + 1, W // 53 + 1
    y = (torch.arange(H, device="cuda") // 37)[:, None].expand(H, W)
    x = (torch.arange(W, device="cuda") // 53)[None, :].expand(H, W)
    n = torch.randn(by, bx, 3, device="cuda", generator=g)
    norm = (n / n.norm(dim=2, keepdim=True))[y, x]
    gy, gx = torch.meshgrid(torch.linspace(0, 8, H, device="cuda"), torch.linspace(0, 20, W, device="cuda"),
                            indexing="ij")
    depth = (10 * rand(by, bx))[y, x] + 0.02 * rand(H, W)
    pos = torch.stack([gx, gy, depth], 2)
    color = (rand(by, bx, 3))[y, x] * (0.2 - torch.log(rand(H, W, 1) + 1e-7))
    color = torch.where(rand(H, W, 1) > 0.999, color * 60, color)
    emit = torch.where(rand(by, bx, 1) > 0.95, 10 * rand(by, bx, 3), torch.zeros(by, bx, 3, device="cuda"))[y, x]
    return [p.float().contiguous() for p in (color, pos, norm, emit)]


def _prepare_filter(case, seed):
    planes = _planes(case, seed)
    g = np.zeros(2 * case["radius"] + 1, np.float32)
    _native.check(_native.load().gbpt_gaussian_table(ctypes.c_float(_sigma(case)), case["radius"], g.ctypes.data))
    torch.cuda.synchronize()
    return dict(planes=planes, g=g, out=torch.zeros_like(planes[0]))


def _sigma(case):
    return 0.5 * case["radius"]


def _run_filter(case, s):
    c, p, n, e = s["planes"]
    _native.check(_native.load().gbpt_bilateral(
        c.data_ptr(), p.data_ptr(), n.data_ptr(), e.data_ptr() if case["emit"] else None, case["width"],
        case["height"], DELTAS["color"], DELTAS["pos"], DELTAS["norm"], DELTAS["emit"], case["radius"],
        s["g"].ctypes.data, s["out"].data_ptr(), 1))
    return s["out"]


def _exact_filter(case, seed):
    W, H, R = case["width"], case["height"], case["radius"]
    c, p, n, e = (x.double() for x in _planes(case, seed))
    feats = [(c, DELTAS["color"]), (p, DELTAS["pos"]), (n, DELTAS["norm"])] + ([(e, DELTAS["emit"])] * case["emit"])
    ys, xs = torch.arange(H, device="cuda"), torch.arange(W, device="cuda")

    def wrap(k, size):  # taps outside the image read its last row or column, on either side
        return torch.where((k < 0) | (k >= size), torch.full_like(k, size - 1), k)

    total = torch.zeros(H, W, 1, dtype=torch.float64, device="cuda")
    acc = torch.zeros_like(c)
    s2 = 2 * _sigma(case) ** 2
    for i in range(-R, R + 1):
        yi = wrap(ys + i, H)
        for j in range(-R, R + 1):
            xj = wrap(xs + j, W)
            a = torch.full((H, W, 1), -(i * i + j * j) / s2, dtype=torch.float64, device="cuda")
            for f, delta in feats:
                a = a - ((f - f[yi][:, xj]) ** 2).sum(2, keepdim=True) / (2 * delta * delta)
            k = torch.exp(a)
            acc += k * c[yi][:, xj]
            total += k
    return acc / total


# --- mlp ----------------------------------------------------------------------


def _mlp_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    F = mlp.N_FEATURES
    x = (np.abs(rng.normal(size=(case["batch"], F))) * rng.random((1, F)) * 2).astype(np.float32)
    t = (np.tanh(x[:, :6].sum(1) - 3) + 0.1 * rng.normal(size=len(x))).astype(np.float32)
    tiles = (np.abs(rng.normal(size=(case["tiles"], F))) * rng.random((1, F)) * 2).astype(np.float32)
    return x, t, tiles


def _mlp_params(seed):
    """He-uniform weights and small biases, in the library's flat layout W1, b1, W2, b2, w3, b3."""
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    F = mlp.N_FEATURES
    parts = []
    for shape, fan in (((64, F), F), ((64,), 0), ((64, 64), 64), ((64,), 0), ((64,), 64), ((1,), 0)):
        lim = math.sqrt(6.0 / fan) if fan else 0.05
        parts.append(((2 * rng.random(shape) - 1) * lim).astype(np.float32).reshape(-1))
    return np.concatenate(parts)


def _prepare_mlp(case, seed):
    x, t, tiles = _mlp_inputs(case, seed)
    return dict(net=mlp.MLP(params=_mlp_params(seed)), x=x, t=t, tiles=tiles)


def _run_mlp(case, s):
    grad, loss = s["net"].gradients(s["x"], s["t"])
    return dict(grad=grad, loss=float(loss), pred=s["net"].forward(s["tiles"]))


def _exact_mlp(case, seed):
    x, t, tiles = (torch.tensor(a, dtype=torch.float64) for a in _mlp_inputs(case, seed))
    w = torch.tensor(_mlp_params(seed), dtype=torch.float64, requires_grad=True)
    F = mlp.N_FEATURES
    W1, b1, W2, b2, w3, b3 = w.split([64 * F, 64, 64 * 64, 64, 64, 1])

    def net(a):
        h = torch.nn.functional.gelu(a @ W1.view(64, F).T + b1)
        h = torch.nn.functional.gelu(h @ W2.view(64, 64).T + b2)
        return h @ w3 + b3

    loss = ((net(x) - t) ** 2).mean()
    (grad,) = torch.autograd.grad(loss, w)
    with torch.no_grad():
        pred = net(tiles)
    return dict(grad=grad.numpy(), loss=float(loss.detach()), pred=pred.numpy())


# --- serve --------------------------------------------------------------------

SERVE_SIZES = ((128, 128), (256, 256), (200, 150), (512, 384))


def _serve_plan(case):
    names = ("cornell", "interior")
    return [(names[k % 2],) + SERVE_SIZES[(k // 2) % 4] + ((6, 8, 10)[k % 3],) for k in range(case["requests"])]


def _prepare_serve(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    built = {n: _build(n) for n in ("cornell", "interior")}
    plan = []
    for k, (name, w, h, depth) in enumerate(_serve_plan(case)):
        # the scheduling knob is given, as by a program that has tuned its classes
        p = gb.default_params(seed=(seed + k) & 0x7FFFFFFF, eye_depth_max=depth, light_depth_max=depth, walk_refill=2)
        plan.append((built[name], _view(name, rng), w, h, p, np.zeros(w * h * 3, np.float32)))
    return dict(server=serving.Server(workers=4), plan=plan)


def _run_serve(case, s):
    ids = [s["server"].submit(sc, cam, w, h, case["frames"], params=p, out=out)
           for sc, cam, w, h, p, out in s["plan"]]
    for i in ids:
        s["server"].wait(i)
    return [q[5] for q in s["plan"]]


# --- the interface ------------------------------------------------------------

_PREPARE = dict(render=_prepare_render, rays=_prepare_rays, filter=_prepare_filter, mlp=_prepare_mlp,
                serve=_prepare_serve)
_RUN = dict(render=_run_render, rays=_run_rays, filter=_run_filter, mlp=_run_mlp, serve=_run_serve)
_EXACT = dict(rays=_exact_rays, filter=_exact_filter, mlp=_exact_mlp)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["case"] = case
    return state


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def work(case):
    kind = case["kind"]
    if kind == "render":
        pixels = case["width"] * case["height"]
        flops, data = _render_work(case["scene"], pixels, case["passes"], case["depth"])
        if case["mode"] in (1, 2, 3):  # the filter passes: a pixel's window over three or four planes
            filtered = case["passes"] if case["mode"] == 3 else max(0, case["passes"] - (8 if case["passes"] > 8 else 5))
            flops += filtered * pixels * (2 * case["radius"] + 1) ** 2 * 3 * 28
            data += filtered * pixels * 5 * 12
    elif kind == "rays":
        tris = SCENES[case["scene"]][2]
        flops = case["rays"] * (2 * 24 * math.log2(tris) + 100)
        data = case["rays"] * 44 + tris * (2 * 32 + 48)
    elif kind == "filter":
        n = 3 + case["emit"]
        pixels = case["width"] * case["height"]
        flops = pixels * (2 * case["radius"] + 1) ** 2 * (n * 28 + 8)
        data = pixels * 12 * (n + 1)
    elif kind == "mlp":
        per = 2 * (mlp.N_FEATURES * 64 + 64 * 64 + 64)
        flops = per * (3 * case["batch"] + case["tiles"])
        data = (case["batch"] + case["tiles"]) * 4 * (mlp.N_FEATURES + 1) + 3 * 4 * 5825
    else:
        flops, data = 0.0, 0.0
        for name, w, h, depth in _serve_plan(case):
            f, d = _render_work(name, w * h, case["frames"], depth)
            flops, data = flops + f, data + d
    return dict(bytes=float(data), flops=float(flops))


def exact(case, seed):
    """64-bit values where a computation has them: a path's image is one draw of an estimator whose every branch
    follows single-precision comparisons, so renders have none."""
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None
