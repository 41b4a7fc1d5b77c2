"""What this framework is measured on: calls that a user's program makes through the Python API.

The sizes are those of the benchmark configurations (Cornell box, dense mesh, moving spheres under a sky, interior),
of the evaluation tools and of the tests; `draw` spreads over the ranges between them, odd sizes among them.
"""
import ctypes as C
import math

import numpy as np
import torch

import azimuth_b200 as az
from azimuth_b200.tiles_eval import camera_copy

SCENES = {"cornell": az.SCENE_CORNELL, "dense_mesh": az.SCENE_DENSE_MESH, "motion_env": az.SCENE_MOTION_ENV,
          "interior": az.SCENE_INTERIOR, "features": az.SCENE_FEATURES, "env_spheres": az.SCENE_ENV_SPHERES}
MESH_SCENES = ("dense_mesh", "interior")       # their meshes come as vertices and faces, as a file's do
SHARED_NET = (4, 64, 64)
LEVELS, TABLE = 16, 1 << 19


def _render(name, scene, width, height, spp, depth=0, detail=0, film="device", filter=-1, watertight=False,
            env_importance=False):
    c = {"kind": "render", "scene": scene, "width": width, "height": height, "spp": spp, "depth": depth,
         "detail": detail, "film": film, "filter": filter, "watertight": watertight, "env_importance": env_importance}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a preview tile while a scene is edited: every material, light and texture kind, a host film, 23,668 samples
        _render("preview", "features", 97, 61, 4, film="host"),
        # a small frame of a light scene, where launches and tails count
        _render("cornell frame", "cornell", 256, 256, 16, 5),
        # the benchmark's frame: 1.3 M displaced triangles, seven reflection models, 67 M camera samples
        _render("dense mesh frame", "dense_mesh", 1024, 1024, 64, 8),
        # motion blur, dielectrics and a sky map: 10,000 moving spheres at full HD
        _render("moving spheres frame", "motion_env", 1920, 1080, 25, 12),
        # indirect light through doorways: 4 M triangles, ten levels, full HD
        _render("interior frame", "interior", 1920, 1080, 16, 10),
        # picking and baking: nearest hits of a list of rays from the host
        {"name": "ray queries", "kind": "hits", "scene": "dense_mesh", "detail": 8, "rays": 200003, "watertight": False},
        # one progressive pass of a guided render with the weights of an earlier session
        {"name": "guided pass", "kind": "guided", "detail": 49, "width": 1280, "height": 720, "spp": 4, "depth": 10},
        # fitting the guide to recorded vertices: the rows of a wave, four steps
        {"name": "guide training", "kind": "train", "rows": 100003, "steps": 4},
        # a render server's queue: small jobs of three scenes in shared waves
        {"name": "job batch", "kind": "tiles", "jobs": 24, "side": 192, "spp": 16, "detail": 6},
        # the drop-in call of a batch renderer: scene in, host film out, nothing kept
        {"name": "one-shot image", "kind": "oneshot", "scene": "interior", "detail": 12, "width": 320, "height": 180,
         "spp": 4, "depth": 6},
        # loading a mesh: normals, areas, hierarchy, and a first probe of it
        {"name": "mesh load", "kind": "load", "scene": "dense_mesh", "detail": 8, "rays": 4099},
        # tone mapping and 8-bit output of a full-HD film
        {"name": "tone mapping", "kind": "post", "width": 1920, "height": 1080, "photographic": True, "srgb": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["guided", "train", "tiles", "oneshot", "load", "hits", "post"])
    if kind == "render":
        scene = rng.choice(["cornell", "dense_mesh", "dense_mesh", "motion_env", "interior", "features",
                            "env_spheres"])
        spp = rng.choice([4, 9, 16, 25, 64])
        top = {"cornell": 2.0e7, "dense_mesh": 3.0e7, "motion_env": 2.0e7, "interior": 1.6e7, "features": 4.0e6,
               "env_spheres": 8.0e6}[scene]
        samples = _log(rng, 6000, top)
        aspect = rng.choice([1.0, 1.5, 16 / 9, 0.6])
        h = max(8, int(math.sqrt(samples / spp / aspect)) | rng.randint(0, 1))
        w = max(8, int(aspect * h) | rng.randint(0, 1))
        detail = {"dense_mesh": rng.randint(5, 8), "interior": rng.randint(8, 49),
                  "motion_env": _log(rng, 500, 10000)}.get(scene, 0)
        depth = {"cornell": rng.randint(2, 6), "features": rng.randint(2, 5)}.get(scene, rng.randint(3, 10))
        return _render("", scene, w, h, spp, depth, detail, rng.choice(["device", "device", "host"]),
                       rng.choice([-1, 0, 1]), rng.random() < 0.15,
                       scene in ("motion_env", "env_spheres") and rng.random() < 0.3)
    if kind == "guided":
        h = _log(rng, 90, 600)
        return {"kind": "guided", "detail": rng.randint(8, 49), "width": int(h * 16 / 9), "height": h,
                "spp": rng.choice([1, 4]), "depth": rng.randint(4, 10)}
    if kind == "train":
        return {"kind": "train", "rows": _log(rng, 500, 250000), "steps": rng.randint(1, 8)}
    if kind == "tiles":
        return {"kind": "tiles", "jobs": rng.randint(3, 40), "side": _log(rng, 40, 256),
                "spp": rng.choice([4, 9, 16]), "detail": rng.randint(4, 7)}
    if kind == "oneshot":
        scene = rng.choice(["cornell", "features", "interior", "dense_mesh"])
        h = _log(rng, 30, 300)
        return {"kind": "oneshot", "scene": scene, "detail": {"interior": rng.randint(6, 16),
                                                              "dense_mesh": rng.randint(3, 6)}.get(scene, 0),
                "width": int(h * rng.choice([1.0, 1.5, 1.78])) | 1, "height": h, "spp": rng.choice([1, 4, 9]),
                "depth": rng.randint(3, 6)}
    if kind == "load":
        scene = rng.choice(MESH_SCENES)
        return {"kind": "load", "scene": scene, "detail": rng.randint(4, 8) if scene == "dense_mesh" else
                rng.randint(6, 40), "rays": _log(rng, 100, 5000)}
    if kind == "hits":
        return {"kind": "hits", "scene": rng.choice(["cornell", "dense_mesh", "interior", "motion_env"]),
                "detail": rng.randint(4, 8), "rays": _log(rng, 300, 300000), "watertight": rng.random() < 0.3}
    h = _log(rng, 60, 2160)
    return {"kind": "post", "width": int(h * rng.choice([1.0, 1.5, 1.78])) | 1, "height": h,
            "photographic": rng.random() < 0.7, "srgb": rng.random() < 0.6}


# ---- what a program has in hand before the call ----

def _scene(case, seed, soup=None):
    """The host scene; mesh scenes as the importer's arrays unless finished structs are asked for."""
    name = case["scene"]
    soup = name in MESH_SCENES if soup is None else soup
    detail = case.get("detail", 0)
    if name == "motion_env" and detail < 100:
        detail = 0
    if name in ("cornell", "features", "env_spheres"):
        detail = 0
    return az.generate_scene(SCENES[name], seed=seed, width=case.get("width", 0), height=case.get("height", 0),
                             spp=case.get("spp", 0), max_depth=case.get("depth", 0), detail=detail,
                             filter=case.get("filter", -1), soup_only=soup)


def _rays(seed, n, lo, hi):
    """Rays inside the box lo..hi toward all directions: origin, direction, shutter time 0."""
    r = np.random.default_rng(seed)
    rays = np.zeros((n, 7), np.float32)
    rays[:, 0:3] = lo + (hi - lo) * (0.02 + 0.96 * r.random((n, 3)))
    d = r.normal(size=(n, 3))
    rays[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return rays


def _box(scene):
    """Bounds of the scene's vertices (every mesh lies where its vertices say), or of the moving spheres' field."""
    v = scene.soup_arrays()[0]
    return (v.min(axis=0), v.max(axis=0)) if len(v) else (np.full(3, -1.0), np.full(3, 1.0))


def _rows(seed, n, lo, hi):
    """Training vertices: positions in the box, normals, directions, and light arriving mostly from above."""
    r = np.random.default_rng(seed)
    rows = np.zeros((n, 16), np.float32)
    rows[:, 0:3] = lo + (hi - lo) * r.random((n, 3))
    rows[:, 3] = r.exponential(1.0, n)
    unit = r.normal(size=(3, n, 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    unit[2] += np.array([0.0, 1.0, 0.0])
    unit[2] /= np.linalg.norm(unit[2], axis=1, keepdims=True)
    rows[:, 4:7], rows[:, 8:11], rows[:, 12:15] = unit[0], unit[1], unit[2]
    return rows


def _weights(seed):
    """A guide's parameters as an earlier session left them: mixtures of moderate width, chosen about half the time."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    mlp = (torch.rand(SHARED_NET, generator=g, device="cuda") - 0.5) * 0.45
    bias = torch.zeros(64, device="cuda")
    bias[3:40:5] = 1.0
    grid = (torch.rand((LEVELS, TABLE, 2), generator=g, device="cuda") - 0.5) * 0.2
    return [x.cpu().numpy() for x in (mlp, bias, grid)]


def _film(seed, w, h):
    """A film of 16 samples a pixel: log-normal light over a smooth picture, a few dark pixels."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    y, x = torch.meshgrid(torch.linspace(0, 6.0, h, device="cuda"), torch.linspace(0, 9.0, w, device="cuda"),
                          indexing="ij")
    f = torch.empty((h, w, 4), device="cuda")
    base = 0.3 + 0.25 * torch.sin(x) * torch.cos(y)
    noise = torch.randn((h, w, 3), generator=g, device="cuda")
    f[..., :3] = 16.0 * base[..., None] * torch.exp(0.8 * noise)
    f[..., :3] *= (torch.rand((h, w, 1), generator=g, device="cuda") > 0.01)
    f[..., 3] = 16.0
    return f


def prepare(case, seed):
    kind = case["kind"]
    if kind == "post":
        w, h = case["width"], case["height"]
        return {"kind": kind, "case": case, "film": _film(seed, w, h),
                "rgb": torch.empty((h, w, 3), device="cuda"),
                "rgb8": torch.empty((h, w, 3), dtype=torch.uint8, device="cuda")}
    if kind == "oneshot":
        return {"kind": kind, "scene": _scene(case, seed, soup=False), "seed": seed}
    if kind == "load":
        sc = _scene(case, seed)
        return {"kind": kind, "scene": sc, "rays": _rays(seed, case["rays"], *_box(sc))}
    if kind == "hits":
        sc = _scene(case, seed)
        gs = az.GpuScene(sc, from_soup=case["scene"] in MESH_SCENES)
        return {"kind": kind, "scene": sc, "gpu": gs, "rays": _rays(seed, case["rays"], *_box(sc)),
                "flags": az.FLAG_WATERTIGHT if case["watertight"] else 0}
    if kind == "tiles":
        return _prepare_tiles(case, seed)
    if kind == "train":
        sc = az.generate_scene(az.SCENE_CORNELL, seed=seed, width=8, height=8, spp=1)
        gs = az.GpuScene(sc)
        guide = az.Guide(gs, seed=seed)
        guide.set_params(*_weights(seed))
        info = guide.info()
        lo = info["lo"].astype(np.float64)
        rows = _rows(seed, case["rows"], lo, lo + 1.0 / info["inv_ext"].astype(np.float64))
        return {"kind": kind, "scene": sc, "gpu": gs, "guide": guide, "rows": rows, "steps": case["steps"],
                "box": (info["lo"], info["inv_ext"])}
    if kind == "guided":
        sc = _scene(dict(case, scene="interior"), seed)
        gs = az.GpuScene(sc, from_soup=True)
        guide = az.Guide(gs, seed=seed)
        guide.set_params(*_weights(seed))
        w, h = sc.resolution()
        return {"kind": kind, "scene": sc, "gpu": gs, "guide": guide, "film": torch.zeros((h, w, 4), device="cuda"),
                "seed": seed}
    sc = _scene(case, seed)
    gs = az.GpuScene(sc, from_soup=case["scene"] in MESH_SCENES)
    w, h = sc.resolution()
    flags = (az.FLAG_WATERTIGHT if case["watertight"] else 0) | \
        (az.FLAG_ENV_IMPORTANCE if case["env_importance"] else 0)
    if case["film"] == "host":
        film = torch.zeros((h, w, 4), pin_memory=True).numpy()
    else:
        film = torch.zeros((h, w, 4), device="cuda")
    return {"kind": kind, "scene": sc, "gpu": gs, "film": film, "flags": flags, "seed": seed,
            "host": case["film"] == "host"}


def _prepare_tiles(case, seed):
    r = np.random.default_rng(seed)
    parts = [("cornell", 0), ("dense_mesh", case["detail"]), ("motion_env", 1500)]
    scenes = [_scene({"scene": n, "detail": d, "depth": 6}, seed + k) for k, (n, d) in enumerate(parts)]
    gpu = [az.GpuScene(s, from_soup=n in MESH_SCENES) for s, (n, _) in zip(scenes, parts)]
    sizes = np.random.default_rng(1000 + case["jobs"])      # the jobs' sizes are the case's, their seeds the inputs'
    jobs, films, cams = [], [], []
    for j in range(case["jobs"]):
        side = max(8, int(case["side"] * math.exp(sizes.uniform(-1.0, 0.5))))
        spp = case["spp"] if j % 3 else 4
        cam = camera_copy(scenes[j % 3], side, side, spp)
        film = torch.zeros((side, side, 4), device="cuda")
        jobs.append({"gpu_scene": gpu[j % 3], "film_ptr": film.data_ptr(), "camera_ptr": C.addressof(cam),
                     "scissor": az.Scissor(az.Vec2u(side, side), az.Vec2u(0, 0)), "seed": int(r.integers(1 << 30))})
        films.append(film)
        cams.append(cam)
    return {"kind": "tiles", "scenes": scenes, "gpu": gpu, "jobs": jobs, "films": films, "cams": cams}


# ---- one call ----

def run(state):
    kind = state["kind"]
    if kind == "render":
        film = state["film"]
        if state["host"]:
            film[:] = 0.0
            state["gpu"].render_host(film, seed=state["seed"], flags=state["flags"])
        else:
            film.zero_()
            state["gpu"].render_device(film.data_ptr(), seed=state["seed"], flags=state["flags"])
        return film
    if kind == "guided":
        state["film"].zero_()
        state["guide"].render(state["film"].data_ptr(), train=False, seed=state["seed"], stats=False)
        return state["film"]
    if kind == "train":
        losses = state["guide"].train(state["rows"], state["steps"])
        mlp, bias, _ = state["guide"].params(grid=False)
        return {"losses": losses, "mlp": mlp, "bias": bias}
    if kind == "tiles":
        for f in state["films"]:
            f.zero_()
        az.render_tiles(state["jobs"])
        return state["films"]
    if kind == "oneshot":
        return az.produce_image(state["scene"], seed=state["seed"])
    if kind == "load":
        with az.GpuScene(state["scene"], from_soup=True) as gs:
            hit, uid, face, t = gs.closest_hit(state["rays"])
        return {"hit": hit, "uid": uid, "face": face, "t": t}
    if kind == "hits":
        hit, uid, face, t = state["gpu"].closest_hit(state["rays"], flags=state["flags"])
        return {"hit": hit, "uid": uid, "face": face, "t": t}
    c = state["case"]
    az.postprocess(state["film"].data_ptr(), c["width"], c["height"], burnout=1.0, photographic=c["photographic"],
                   srgb=c["srgb"], rgb_ptr=state["rgb"].data_ptr(), rgb8_ptr=state["rgb8"].data_ptr())
    return {"rgb": state["rgb"], "rgb8": state["rgb8"]}


# ---- what a call cannot do without ----

TRIANGLES = {"cornell": 12, "features": 24, "env_spheres": 2, "motion_env": 0}


def _triangles(scene, detail):
    if scene == "dense_mesh":
        return 20 * 4 ** (detail or 8) + 12
    if scene == "interior":
        return 1650 * (detail or 49) ** 2
    return TRIANGLES[scene]


def work(case):
    """Bytes: inputs read and outputs written once.  Operations: for renders and ray queries one pass down a
    balanced 8-wide hierarchy and one triangle per query, at the scene's mean number of path segments per sample."""
    kind = case["kind"]
    if kind == "post":
        n = case["width"] * case["height"]
        return {"bytes": n * (16 + 12 + 3), "flops": n * 60}
    if kind == "train":
        n = case["rows"] * case["steps"]
        return {"bytes": case["rows"] * 64 + case["steps"] * 4 * 4 * 64 * 64, "flops": n * 6 * 4 * 64 * 64}
    if kind in ("load", "hits"):
        tri = _triangles(case["scene"], case["detail"])
        levels = 1 + math.log(max(tri, 8), 8)
        return {"bytes": (tri * 18 if kind == "load" else 0) + case["rays"] * 44,
                "flops": case["rays"] * (levels * 8 * 20 + 60) + (tri * 200 if kind == "load" else 0)}
    segments = {"cornell": 4.0, "dense_mesh": 5.0, "motion_env": 5.0, "interior": 10.0, "features": 8.0,
                "env_spheres": 4.0}
    if kind == "tiles":
        samples, tri, seg, pixels = case["jobs"] * case["side"] ** 2 * case["spp"], 20 * 4 ** case["detail"], 4.5, \
            case["jobs"] * case["side"] ** 2
    else:
        name = case.get("scene", "interior")
        pixels = case["width"] * case["height"]
        samples = pixels * case["spp"]
        seg = min(segments[name], 1.0 + (case["depth"] or 5))
        tri = 10000 if name == "motion_env" else _triangles(name, case["detail"])
    levels = 1 + math.log(max(tri, 8), 8)
    flops = samples * seg * 2 * (levels * 8 * 20 + 60)
    if kind == "guided":
        flops += samples * seg * 2 * 4 * 64 * 64
    return {"bytes": pixels * 16 + tri * 48, "flops": flops}


# ---- the same in 64 bits ----

def _exact_hits(scene, rays):
    """t of the nearest triangle of the scene's meshes (azimuth's tolerance of -1e-6 on the barycentrics), 0: none."""
    v, f, _, _ = scene.soup_arrays()      # the meshes of these scenes are placed as they are
    v = torch.from_numpy(v).cuda().double()
    f = torch.from_numpy(f.astype(np.int64)).cuda()
    p0, p1, p2 = (v[f[:, k]] for k in range(3))
    e1, e2 = p1 - p0, p2 - p0
    r = torch.from_numpy(rays).cuda().double()
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // max(1, len(f)))
    for a in range(0, len(rays), step):
        o, d = r[a:a + step, None, 0:3], r[a:a + step, None, 3:6]
        h = torch.linalg.cross(d, e2[None])
        det = (e1[None] * h).sum(-1)
        s = o - p0[None]
        u = (s * h).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        w = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (u > -1e-6) & (w > -1e-6) & (1.0 - u - w > -1e-6) & (t > 0.0)
        best[a:a + step] = torch.where(ok, t, math.inf).min(dim=1).values
    return torch.where(torch.isfinite(best), best, 0.0).cpu().numpy()


def _exact_train(state, seed):
    """The steps in float64: hash-grid encoding, three hidden layers, the mixture's loss, Adam."""
    dev = "cuda"
    mlp, bias, grid = (torch.from_numpy(x).to(dev).double() for x in _weights(seed))
    rows = torch.from_numpy(state["rows"]).to(dev).double()
    lo, inv = (torch.from_numpy(x).to(dev).double() for x in state["box"])
    p = ((rows[:, 0:3] - lo) * inv).clamp(0.0, 1.0)
    weight, n, wo, wi = rows[:, 3], rows[:, 4:7], rows[:, 8:11], rows[:, 12:15]
    cells = []
    for level in range(LEVELS):
        res = int(math.floor(16.0 * 2.0 ** (7.0 * level / 15.0)))
        x = p * res
        i = torch.minimum(x.floor().long(), torch.tensor(res - 1, device=dev))
        fr = x - i
        idx, wt = [], []
        for k in range(8):
            d = torch.tensor([k & 1, k >> 1 & 1, k >> 2 & 1], device=dev)
            c = i + d
            if (res + 1) ** 3 <= TABLE:
                e = c[:, 0] + (res + 1) * (c[:, 1] + (res + 1) * c[:, 2])
            else:
                e = (c[:, 0] ^ (c[:, 1] * 2654435761) ^ (c[:, 2] * 805459861)) & (TABLE - 1)
            idx.append(e)
            wt.append(torch.where(d == 1, fr, 1.0 - fr).prod(dim=1))
        cells.append((torch.stack(idx, 1), torch.stack(wt, 1)))
    ws = [x.clone().requires_grad_() for x in (mlp, bias, grid)]
    m = [torch.zeros_like(x) for x in ws]
    s = [torch.zeros_like(x) for x in ws]
    losses = []
    for step in range(1, state["steps"] + 1):
        feats = [(ws[2][lv][idx] * wt[..., None]).sum(1) for lv, (idx, wt) in enumerate(cells)]
        a = torch.cat(feats + [n, wo, torch.ones_like(n[:, :1]), torch.zeros((len(n), 25), device=dev,
                                                                           dtype=torch.float64)], 1)
        for layer in range(3):
            a = (a @ ws[0][layer]).relu()
        o = a @ ws[0][3] + ws[1]
        lobes = o[:, :40].reshape(-1, 8, 5)
        mu = lobes[..., 0:3] / (lobes[..., 0:3].square().sum(-1, keepdim=True) + 1e-12).sqrt()
        kap = lobes[..., 3].clamp(-3.0, 5.0).exp()
        pi = lobes[..., 4].softmax(dim=1)
        cos = (mu * wi[:, None]).sum(-1)
        vmf = kap / (2.0 * math.pi * -torch.expm1(-2.0 * kap)) * torch.exp(kap * (cos - 1.0))
        alpha = 0.05 + 0.75 * torch.sigmoid(o[:, 40])
        q = alpha * (pi * vmf).sum(1) + (1.0 - alpha) * (n * wi).sum(1).clamp(min=0.0) / math.pi
        loss = (-weight * q.clamp(min=1e-30).log()).sum()
        losses.append(float(loss.detach()))
        grads = torch.autograd.grad(loss, ws)
        with torch.no_grad():
            for x, g, mm, ss in zip(ws, grads, m, s):
                mm.mul_(0.9).add_(g, alpha=0.1)
                ss.mul_(0.99).addcmul_(g, g, value=0.01)
                x -= 0.01 * (mm / (1 - 0.9 ** step)) / ((ss / (1 - 0.99 ** step)).sqrt() + 1e-8)
    return {"losses": np.array(losses), "mlp": ws[0].detach().cpu().numpy(), "bias": ws[1].detach().cpu().numpy()}


def _exact_post(state):
    c = state["case"]
    f = state["film"].double()
    rgb = f[..., :3] / f[..., 3:]
    lum = rgb @ torch.tensor([0.27, 0.67, 0.06], dtype=torch.float64, device="cuda")
    if c["photographic"]:
        flat = lum.reshape(-1)
        factor = 0.18 / flat.add(1e-5).log().mean().exp()
        at = int((1.0 - 0.01) * (flat.numel() - 1) + 0.5)
        white = flat.sort().values[at] * factor
        ls = lum * factor
        ld = ls * (1.0 + ls / white.square()) / (1.0 + ls)
        mapped = (rgb / lum[..., None] * ld[..., None]).clamp(0.0, 1.0)
        rgb = torch.where(lum[..., None] != 0.0, mapped, rgb)
    if c["srgb"]:
        out = torch.where(rgb > 0.0031308, 1.055 * rgb.clamp(min=0.0) ** (1.0 / 2.2) - 0.055, rgb * 12.92)
    else:
        out = rgb ** (1.0 / 2.2)
    return {"rgb": out, "rgb8": None}


def exact(case, seed):
    if case["kind"] == "post":
        return _exact_post(prepare(case, seed))
    if case["kind"] == "train":
        return _exact_train(prepare(case, seed), seed)
    if case["kind"] in ("load", "hits") and case["scene"] in MESH_SCENES and \
            case["rays"] * _triangles(case["scene"], case["detail"]) < 1e10:
        sc = _scene(case, seed)
        return {"hit": None, "uid": None, "face": None, "t": _exact_hits(sc, _rays(seed, case["rays"], *_box(sc)))}
    return None      # films: a path tracer in 64 bits takes other branches, and hours
