"""Performance cases: what a program does with this library, each through the public Python entry
points (api.Scene / api.Device / api.render_batch / the filters / denoiser.Denoiser).

  listed()             the fixed cases
  draw(rng)            another case of the same ranges
  prepare(case, seed)  inputs, scene, plan and output buffers, as the program holds them
  run(state)           one pass
  work(case)           bytes and floating-point operations a pass cannot do without
  exact(case, seed)    the pass's results in 64 bits from plain torch, where they can be had
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cudapathtracing_gb300 import abi, api, procedural as P, training
from cudapathtracing_gb300.denoiser import SPECS, Denoiser, layer_slices

LAYOUTS = {"bvh2": (2, False), "bvh2q": (2, True), "bvh8": (8, False)}
INTEGRATORS = {"megakernel": abi.INTEGRATOR_MEGAKERNEL, "wavefront": abi.INTEGRATOR_WAVEFRONT}
PATH = dict(max_depth=16, rr_depth=3, rr_prob=0.8)   # the config estimator's depth settings


def listed():
    return [
        # picking, probes and light-map points: a few rays from host memory, an answer at once
        dict(name="probe_rays_1k", kind="probe", freq=32, rays=1000, layout="bvh2"),
        # cloth and skinned meshes: the tree of a small mesh rebuilt every frame, ragged count
        dict(name="build_12k", kind="build", triangles=12305),
        # a large mesh's tree, from vertices that are already on the device
        dict(name="build_1M", kind="build", triangles=1310720),
        # bulk visibility queries against a resident scene (default layout)
        dict(name="trace_10M", kind="trace", freq=256, rays=10_000_000, layout="bvh2", rebuild=False),
        # an animated mesh: rebuild into the 8-wide layout, then this frame's queries (odd count)
        dict(name="rebuild_trace_wide", kind="trace", freq=256, rays=2_000_003, layout="bvh8", rebuild=True),
        # the reference's estimator as it ships: the 512 x 512 Cornell box at 16 spp
        dict(name="cornell_reference", kind="render", scene="cornell", width=512, spp=16, estimator="reference",
             integrator="megakernel", layout="bvh2", slots=1 << 21, gbuffer=False),
        # an editor's preview: one small frame at few samples, with its G-buffer for the denoiser
        dict(name="preview_256", kind="render", scene="random", width=256, spp=4, estimator="config",
             integrator="wavefront", layout="bvh2", slots=1 << 21, gbuffer=True),
        # production frame: 4.1M triangles, 1920 x 1080, 64 spp, the knobs that the autotuner picks
        dict(name="frame_1080p_64spp", kind="render", scene="spheres", width=1920, spp=64, estimator="config",
             integrator="wavefront", layout="bvh8", slots=1 << 24, gbuffer=False),
        # the serving loop's batch: small jobs of several scenes in one wavefront
        dict(name="serve_batch", kind="batch", jobs="256x16 512x4 256x1 512x16 256x64 512x1", layout="bvh2",
             slots=1 << 21),
        # learned denoiser: one 1080p frame; and its training step on a batch of 256 x 256 crops
        dict(name="denoise_1080p", kind="denoise", width=1920, height=1080),
        dict(name="train_16x256", kind="train", batch=16, size=256),
        # the real-time loop's filters on a 1080p frame while the camera moves
        dict(name="filter_1080p", kind="filter", width=1920, height=1080, moving=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["probe", "build", "build", "trace", "trace", "render", "render", "render", "batch", "denoise",
                       "train", "filter"])
    layout = rng.choice(sorted(LAYOUTS))
    if kind == "probe":
        return dict(kind=kind, freq=_log(rng, 4, 64), rays=_log(rng, 1, 20000), layout=layout)
    if kind == "build":
        return dict(kind=kind, triangles=_log(rng, 2, 1310720))
    if kind == "trace":
        return dict(kind=kind, freq=_log(rng, 8, 256), rays=_log(rng, 1000, 10_000_000), layout=layout,
                    rebuild=rng.random() < 0.5)
    if kind == "render":
        scene = rng.choice(["cornell", "random", "random", "spheres"])
        reference = rng.random() < 0.25
        width = _log(rng, 97, 1920 if scene == "spheres" else 1024)
        return dict(kind=kind, scene=scene, width=width, spp=_log(rng, 1, 32 if scene == "spheres" else 16),
                    estimator="reference" if reference else "config",
                    integrator="megakernel" if reference else rng.choice(["megakernel", "wavefront", "wavefront"]),
                    layout=layout, slots=1 << rng.randint(19, 24), gbuffer=rng.random() < 0.5)
    if kind == "batch":
        jobs = ["%dx%d" % (rng.choice([128, 256, 400, 512]), rng.choice([1, 4, 16, 64]))
                for _ in range(rng.randint(2, 8))]
        return dict(kind=kind, jobs=" ".join(jobs), layout=layout, slots=1 << rng.randint(19, 22))
    if kind == "denoise":
        return dict(kind=kind, width=_log(rng, 65, 1920), height=_log(rng, 65, 1080))
    if kind == "train":
        return dict(kind=kind, batch=rng.randint(1, 16), size=16 * rng.randint(4, 16))
    return dict(kind="filter", width=_log(rng, 65, 1920), height=_log(rng, 65, 1080), moving=rng.random() < 0.5)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _geodesic(freq):
    """(20 freq^2, 3, 3) unit vectors: the icosahedron's faces cut into freq^2 triangles each."""
    v, f = P.icosphere(0)
    v = torch.tensor(v, dtype=torch.float64, device="cuda")
    f = torch.tensor(f, device="cuda")
    k = torch.arange(freq, device="cuda")
    i, j = torch.meshgrid(k, k, indexing="ij")
    i, j = i.reshape(-1), j.reshape(-1)
    up, down = i + j <= freq - 1, i + j <= freq - 2
    iu, ju, idn, jdn = i[up], j[up], i[down], j[down]
    a = torch.cat([torch.stack([iu, ju], 1), torch.stack([idn + 1, jdn], 1)])
    b = torch.cat([torch.stack([iu + 1, ju], 1), torch.stack([idn + 1, jdn + 1], 1)])
    c = torch.cat([torch.stack([iu, ju + 1], 1), torch.stack([idn, jdn + 1], 1)])
    w = torch.stack([a, b, c], 1).to(torch.float64) / freq          # (freq^2, 3, 2)
    A, B, C = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]                    # (20, 3)
    p = (A[:, None, None] + w[None, :, :, :1] * (B - A)[:, None, None] + w[None, :, :, 1:] * (C - A)[:, None, None])
    p = p.reshape(-1, 3, 3)
    return p / p.norm(dim=-1, keepdim=True)


def _displaced(freq, gen):
    """A displaced sphere of radius about 1: radius 1 + 0.1 x a sum of random sinusoids."""
    d = _geodesic(freq)
    k = torch.randn(8, 3, generator=gen, device="cuda", dtype=torch.float64)
    k = k / k.norm(dim=1, keepdim=True) * torch.tensor([3., 4., 6., 8., 11., 15., 20., 27.], device="cuda")[:, None]
    ph = torch.rand(8, generator=gen, device="cuda", dtype=torch.float64) * 2 * math.pi
    amp = torch.tensor([3., 2.5, 2., 1.5, 1.2, 1., .7, .5], device="cuda", dtype=torch.float64)
    r = torch.sin(d @ k.T.to(torch.float64) + ph) @ (amp / amp.sum())
    return d * (1.0 + 0.1 * r)[..., None]


def _mesh_scene(freq, seed):
    tri = _displaced(freq, _gen(seed)).reshape(-1, 9).to(torch.float32).cpu().numpy()
    d = abi.SceneDesc()
    d.add_material((0.7, 0.7, 0.7), 0.5, 0.5, abi.M_LAMBERTIAN)
    d.tri_vertices = tri
    d.tri_material = np.zeros(tri.shape[0], np.uint32)
    pts = tri.reshape(-1, 3).astype(np.float64)
    d.bounds_min, d.bounds_max = tuple(pts.min(0)), tuple(pts.max(0))
    d.camera = abi.Camera(512, 1.0, (0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 45.0, (0.5, 0.6, 0.8))
    return d


def _spheres_scene(width, seed):
    """The 1080p workload's scene for any seed: 200 displaced spheres of 20,480 triangles on the
    ground (Lambertian / GGX / glass), a volume box, two area lights."""
    gen, rng = _gen(seed), np.random.default_rng(seed)
    d = abi.SceneDesc()
    ground = d.add_material((0.6, 0.6, 0.6), 0.5, 0.5, abi.M_LAMBERTIAN)
    base = torch.tensor([[-30, 0, -30, -30, 0, 30, 30, 0, -30], [30, 0, -30, -30, 0, 30, 30, 0, 30]],
                        dtype=torch.float32, device="cuda")
    parts, mats = [base], [np.full(2, ground, np.uint32)]
    shapes = [_displaced(32, gen) for _ in range(8)]
    for k in range(200):
        x, z = rng.uniform(-10, 10, 2)
        r = rng.uniform(0.3, 1.0)
        rough, col = float(rng.uniform(0.05, 0.8)), tuple(rng.uniform(0.2, 0.9, 3))
        if k % 3 == 0:
            m = d.add_material(col, 0.5, 0.5, abi.M_LAMBERTIAN)
        elif k % 3 == 1:
            m = d.add_material(col, rough, rough, abi.M_OPAQUE)
        else:
            m = d.add_material((1.0, 1.0, 1.0), 0.5, 0.5, abi.M_SPECULAR_DIELECTRIC, eta=1.5)
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        t = shapes[k % 8] @ torch.tensor(q * r, device="cuda") + torch.tensor([x, r, z], device="cuda",
                                                                               dtype=torch.float64)
        parts.append(t.reshape(-1, 9).to(torch.float32))
        mats.append(np.full(t.shape[0], m, np.uint32))
    vol = d.add_material((1.0, 1.0, 1.0), 0.5, 0.5, abi.M_VOLUME, sigma_t=0.5, albedo=0.8)
    c = np.array([[sx, sy, sz] for sx in (-1.5, 1.5) for sy in (0.01, 3.01) for sz in (1.5, 4.5)])
    quads = [(1, 5, 3, 7), (0, 2, 4, 6), (0, 1, 2, 3), (4, 6, 5, 7), (2, 3, 6, 7), (0, 4, 1, 5)]
    box = [np.concatenate([c[i] for i in t]) for a, b, e, g in quads for t in ((a, b, e), (b, g, e))]
    parts.append(torch.tensor(np.array(box), dtype=torch.float32, device="cuda"))
    mats.append(np.full(len(box), vol, np.uint32))
    tri = torch.cat(parts)
    d.tri_vertices, d.tri_material = tri.cpu().numpy(), np.concatenate(mats)
    for q in ((-5.0, 12.0, 0.0), (5.0, 12.0, 5.0)):
        d.lights.append(dict(center=q, normal=(0.0, -1.0, 0.0), width=4.0, height=4.0, color=(12.0, 12.0, 12.0),
                             visible=1))
    pts = tri.reshape(-1, 3)
    d.bounds_min, d.bounds_max = tuple(pts.amin(0).tolist()), tuple(pts.amax(0).tolist())
    d.camera = abi.Camera(width, 16.0 / 9.0, (0.0, 7.0, 24.0), (0.0, 1.0, 0.0), 40.0, (0.05, 0.06, 0.08))
    return d


def _desc(scene, width, seed):
    if scene == "cornell":
        return P.cornell_box(width=width, seed=seed)
    if scene == "random":
        return P.random_scene(seed, width=width)
    return _spheres_scene(width, seed)


def _rays(n, seed):
    """Origins uniform in [-2, 2]^3, directions uniform on the sphere (n, 8): o, tmin, d, tmax."""
    g = _gen(seed)
    r = torch.empty(n, 8, device="cuda")
    r[:, :3] = torch.rand(n, 3, generator=g, device="cuda") * 4 - 2
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    r[:, 4:7] = (d / d.norm(dim=1, keepdim=True)).float()
    r[:, 3], r[:, 7] = 0.001, 999999.0
    return r


def _images(n, h, w, seed):
    """n rendered-looking frames: a noisy image, its G-buffer and the clean image.  Blocks of plain
    albedo, smooth normals, depths and light, a sky region without a hit, heavy-tailed noise."""
    g = _gen(seed)

    def field(c, cell, mode):
        x = torch.rand(n, c, max(2, h // cell), max(2, w // cell), generator=g, device="cuda")
        kw = {} if mode == "nearest" else dict(align_corners=False)
        return torch.nn.functional.interpolate(x, (h, w), mode=mode, **kw).permute(0, 2, 3, 1)
    albedo = 0.1 + 0.8 * field(3, 40, "nearest")
    nrm = field(3, 48, "bilinear") * 2 - 1
    nrm = nrm / nrm.norm(dim=-1, keepdim=True).clamp(min=1e-3)
    depth = 4 + 26 * field(1, 64, "bilinear")
    light = (3 * field(1, 80, "bilinear") ** 2 + 0.02)
    hit = (field(1, 96, "bilinear") < 0.62).float()
    clean = hit * albedo * light + (1 - hit) * torch.tensor([0.05, 0.06, 0.08], device="cuda")
    sd = 0.6 * hit
    noise = torch.exp(sd * torch.randn(n, h, w, 1, generator=g, device="cuda") - sd * sd / 2)
    fly = (torch.rand(n, h, w, 1, generator=g, device="cuda") < 0.002).float() * 12 * hit
    rgb = (clean * noise + fly * albedo).contiguous()
    gb = torch.zeros(n, h, w, 8, device="cuda")
    gb[..., 0:3] = nrm * hit
    gb[..., 3:4] = torch.where(hit > 0, depth, torch.full_like(depth, 999999.0))
    gb[..., 4:7] = albedo * hit
    gb[..., 7:8] = (0.3 * light * hit) ** 2
    return rgb, gb, clean.contiguous()


def _weights(seed):
    """A network at the start of its training: He-normal weights, zero biases, a small last layer."""
    g = np.random.default_rng(seed)
    parts = []
    for k, (ci, co, _) in enumerate(SPECS):
        std = math.sqrt(2 / (9 * ci)) * (0.1 if k == len(SPECS) - 1 else 1.0)
        parts += [g.normal(0, std, 9 * ci * co), np.zeros(co)]
    return np.concatenate(parts).astype(np.float32)


def _context(case):
    ctx = api.Context(0)
    width, compressed = LAYOUTS[case["layout"]]
    ctx.set_bvh_width(width)
    ctx.set_bvh_compression(compressed)
    if "slots" in case:
        ctx.set_wavefront(case["slots"])
    return ctx


def _camera(case, moved):
    w, h = case["width"], case["height"]
    return abi.Camera(w, w / (h + 0.5), (0.05 * moved, 2.0, 12.0), (0.0, 0.8, 0.0), 40.0)


def _triangles(case, seed):
    n = case["triangles"]
    t = _displaced(max(1, math.ceil(math.sqrt(n / 20))), _gen(seed)).reshape(-1, 9).to(torch.float32)
    return t[torch.randperm(t.shape[0], generator=_gen(seed + 1), device="cuda")[:n]].contiguous()


_EXTRA_C = [[-1.0, 3.0, 0.5], [1.5, 2.5, -0.5]]        # two lights
_EXTRA_B = [[-1.5, 2.999, 0.0, 0.0, -0.5, 3.001, 1.0, 0.0], [1.0, 2.499, -1.0, 0.0, 2.0, 2.501, 0.0, 0.0]]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind in ("probe", "trace"):
        s["scene"] = api.Scene(_context(case), _mesh_scene(case["freq"], seed)).init()
        rays = _rays(case["rays"], seed + 1)
        if kind == "probe":
            s["rays"] = rays.cpu().numpy().view(abi.RAY_DTYPE).reshape(-1)
        else:
            s["rays"], s["hits"] = rays, torch.zeros(case["rays"], 4, device="cuda")
    elif kind == "build":
        tri = _triangles(case, seed)
        n = case["triangles"] + 2
        pts = tri.reshape(-1, 3).double()
        i32 = dict(dtype=torch.int32, device="cuda")
        s.update(tri=tri, lo=pts.amin(0).tolist(), hi=pts.amax(0).tolist(),
                 centroids=torch.tensor(_EXTRA_C, dtype=torch.float64, device="cuda"),
                 boxes=torch.tensor(_EXTRA_B, dtype=torch.float32, device="cuda"),
                 out=dict(keys=torch.zeros(n, dtype=torch.int64, device="cuda"), order=torch.zeros(n, **i32),
                          children=torch.zeros(n - 1, 2, **i32), node_range=torch.zeros(n - 1, 2, **i32),
                          node_boxes=torch.zeros(n - 1, 8, device="cuda"),
                          leaf_boxes=torch.zeros(n, 8, device="cuda")),
                 scratch=torch.zeros(api.Device.scratch_bytes(n), dtype=torch.uint8, device="cuda"))
    elif kind == "render":
        sc = api.Scene(_context(case), _desc(case["scene"], case["width"], seed)).init()
        s.update(scene=sc, seed=int(seed), rgb=torch.zeros(sc.height, sc.width, 3, device="cuda"),
                 rgba8=torch.zeros(sc.height, sc.width, 4, dtype=torch.uint8, device="cuda"),
                 gbuffer=torch.zeros(sc.height, sc.width, 8, device="cuda") if case["gbuffer"] else None)
    elif kind == "batch":
        s["ctx"] = _context(case)
        s["jobs"] = []
        for k, job in enumerate(case["jobs"].split()):
            size, spp = (int(x) for x in job.split("x"))
            sc = api.Scene(s["ctx"], _desc("random", size, seed + k)).init()
            s["jobs"].append(dict(scene=sc, spp=spp, seed=int(seed) + k,
                                  rgb=torch.zeros(sc.height, sc.width, 3, device="cuda"),
                                  gbuffer=torch.zeros(sc.height, sc.width, 8, device="cuda"), **PATH))
    elif kind == "denoise":
        s["net"] = Denoiser(0)
        s["net"].load(training.DEFAULT_WEIGHTS)
        rgb, gb, _ = _images(1, case["height"], case["width"], seed)
        s.update(rgb=rgb[0], gbuffer=gb[0], out=torch.zeros_like(rgb[0]))
    elif kind == "train":
        s["net"] = Denoiser(0)
        s["net"].params = _weights(seed)
        s["rgb"], s["gbuffer"], s["target"] = _images(case["batch"], case["size"], case["size"], seed)
    else:
        rgb, gb, _ = _images(1, case["height"], case["width"], seed)
        prev, _, _ = _images(1, case["height"], case["width"], seed + 1)
        s.update(ctx=api.Context(0), rgb=rgb[0], gbuffer=gb[0], prev=prev[0], out=torch.zeros_like(rgb[0]),
                 camera=_camera(case, 1 if case["moving"] else 0), before=_camera(case, 0))
    return s


# ---------------------------------------------------------------- the passes
def run(s):
    kind = s["kind"]
    if kind == "probe":
        h = s["scene"].trace(s["rays"])
        return dict(t=h["t"], prim=h["prim"], u=h["u"], v=h["v"])
    if kind == "trace":
        if s["case"]["rebuild"]:
            s["scene"].buildBVH()
        h = s["scene"].trace(s["rays"], s["hits"])
        return dict(t=h[:, 0], prim=h[:, 1].view(torch.int32), u=h[:, 2], v=h[:, 3])
    if kind == "build":
        api.Device.buildBVH(s["centroids"], s["boxes"], s["tri"], s["lo"], s["hi"], s["out"], s["scratch"])
        return s["out"]
    if kind == "render":
        c = s["case"]
        depth = PATH if c["estimator"] == "config" else {}
        r = s["scene"].render(spp=c["spp"], integrator=INTEGRATORS[c["integrator"]], seed=s["seed"], rgb=s["rgb"],
                              rgba8=s["rgba8"], gbuffer=s["gbuffer"],
                              estimator=abi.ESTIMATOR_CONFIG if depth else abi.ESTIMATOR_REFERENCE, **depth)
        return dict(rgb=r["rgb"], rgba8=r["rgba8"], gbuffer=r["gbuffer"], rays=r["rays"])
    if kind == "batch":
        r = api.render_batch(s["ctx"], s["jobs"])
        return dict(rgb=[j["rgb"] for j in r["jobs"]], gbuffer=[j["gbuffer"] for j in r["jobs"]], rays=r["rays"])
    if kind == "denoise":
        return s["net"].denoise(s["rgb"], s["gbuffer"], s["out"])
    if kind == "train":
        loss = s["net"].train_step(s["rgb"], s["gbuffer"], s["target"], lr=1e-4)
        return dict(loss=loss, grads=s["net"].grads())
    out = api.filter_bilateral(s["ctx"], s["rgb"], s["gbuffer"], s["out"])
    return api.filter_temporal(s["ctx"], out, s["prev"], s["gbuffer"], s["camera"], s["before"])


# ---------------------------------------------------------------- work
_LEVEL = [0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 3, 3, 2, 2, 1, 1, 0, 0, 0]   # U-Net level of each convolution
# Queries per sample and operations per query (box and triangle tests of an ordered, pruned binary
# traversal: 36 per node visit, 40 per triangle) of the scenes, as counted on such scenes.
_PER_SAMPLE = {"cornell": 8.0, "random": 4.0, "spheres": 3.6}
_PER_QUERY = {"cornell": 36 * 17 + 40 * 3, "random": 36 * 30 + 40 * 2, "spheres": 36 * 69 + 40 * 3}


def _conv_flops(pixels):
    return 2 * 9 * pixels * sum(ci * co / 4 ** l for (ci, co, _), l in zip(SPECS, _LEVEL))


def work(case):
    kind = case["kind"]
    if kind in ("probe", "trace"):
        tri = 20 * case["freq"] ** 2
        return dict(bytes=48 * case["rays"] + 36 * tri * (2 if case.get("rebuild") else 1),
                    flops=(36 * 9 + 40) * case["rays"])
    if kind == "build":
        n = case["triangles"] + 2
        return dict(bytes=(36 + 8 + 4 + 8 + 8 + 32 + 32) * n, flops=0)
    if kind == "render":
        w = case["width"]
        px = w * (int(w / (16 / 9)) if case["scene"] == "spheres" else w)
        tri = {"cornell": 34, "random": 80000, "spheres": 4096014}[case["scene"]]
        q = px * case["spp"] * _PER_SAMPLE[case["scene"]]
        return dict(bytes=36 * tri + px * (12 + 4 + (32 if case["gbuffer"] else 0)),
                    flops=q * _PER_QUERY[case["scene"]])
    if kind == "batch":
        jobs = [tuple(int(x) for x in j.split("x")) for j in case["jobs"].split()]
        return dict(bytes=sum(36 * 80000 + 44 * a * a for a, _ in jobs),
                    flops=sum(a * a * spp for a, spp in jobs) * _PER_SAMPLE["random"] * _PER_QUERY["random"])
    params = 4 * sum(9 * ci * co + co for ci, co, _ in SPECS)
    if kind == "denoise":
        px = case["width"] * case["height"]
        return dict(bytes=px * (12 + 32 + 12) + params, flops=_conv_flops(px))
    if kind == "train":
        px = case["batch"] * case["size"] ** 2
        return dict(bytes=px * (12 + 32 + 12) + 7 * params, flops=3 * _conv_flops(px))
    px = case["width"] * case["height"]
    return dict(bytes=px * (12 + 32 + 12 + 12), flops=px * 66 * 30)


# ---------------------------------------------------------------- 64-bit results
def _exact_hits(tri, rays):
    tri, rays = tri.double().reshape(-1, 3, 3), rays.double()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    out = [torch.full((rays.shape[0],), v, dtype=torch.float64, device="cuda") for v in (-1.0, 0.0, 0.0)]
    prim = torch.full((rays.shape[0],), -1, dtype=torch.int32, device="cuda")
    step = max(1, 60_000_000 // tri.shape[0])
    for a in range(0, rays.shape[0], step):
        o, d = rays[a:a + step, None, :3], rays[a:a + step, None, 4:7]
        h = torch.linalg.cross(d, e2[None])
        det = (e1[None] * h).sum(-1)
        s = o - p0[None]
        u = (s * h).sum(-1) / det
        q = torch.linalg.cross(s, e1[None])
        v = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0.001) & (t <= 999999.0)
        t = torch.where(ok, t, torch.inf)
        best, k = t.min(1)
        hit = best < torch.inf
        rows = torch.arange(k.shape[0], device="cuda")[hit]
        out[0][a + rows], prim[a + rows] = best[hit], k[hit].int()
        out[1][a + rows], out[2][a + rows] = u[rows, k[hit]], v[rows, k[hit]]
    return dict(t=out[0], prim=prim, u=out[1], v=out[2])


def _exact_build(case, seed):
    s = prepare(case, seed)
    tri = s["tri"].double().reshape(-1, 3, 3)
    lo = torch.cat([s["boxes"][:, 0:3].double(), tri.amin(1) - 1e-4])
    hi = torch.cat([s["boxes"][:, 4:7].double(), tri.amax(1) + 1e-4])
    c = torch.cat([s["centroids"], (tri[:, 0] + tri[:, 1] + tri[:, 2]) / 3.0])
    mn = torch.tensor(s["lo"], dtype=torch.float64, device="cuda") - 1.0
    mx = torch.tensor(s["hi"], dtype=torch.float64, device="cuda") + 1.0
    cell = ((c - mn) / (mx - mn) * 1024.0).clamp(0.0, 1023.0).long()
    code = torch.zeros(c.shape[0], dtype=torch.int64, device="cuda")
    for b in range(10):
        for axis in range(3):
            code |= ((cell[:, axis] >> b) & 1) << (3 * b + 2 - axis)
    n = c.shape[0]
    key = (code << 32) | torch.arange(n, device="cuda")
    key, order = key.sort()
    box = torch.cat([lo, -hi], 1)[order]        # the union of boxes is a minimum of these six

    def delta(i, j):                            # common prefix of keys i and j (they all differ), -1 outside
        ok = (j >= 0) & (j < n)
        x = key[i] ^ key[j.clamp(0, n - 1)]
        hi_, lo_ = (x >> 32).double(), (x & 0xFFFFFFFF).double()
        p = torch.where(hi_ > 0, 32 - torch.frexp(hi_).exponent, 64 - torch.frexp(lo_).exponent)
        return torch.where(ok, p, torch.full_like(p, -1))
    i = torch.arange(n - 1, device="cuda")
    d = torch.where(delta(i, i + 1) > delta(i, i - 1), 1, -1)
    least = delta(i, i - d)
    length = torch.zeros_like(i)
    for b in reversed(range(max(1, n.bit_length()))):
        length = torch.where(delta(i, i + (length + (1 << b)) * d) > least, length + (1 << b), length)
    first, last = torch.minimum(i, i + length * d), torch.maximum(i, i + length * d)
    node = torch.zeros(n - 1, 6, dtype=torch.float64, device="cuda")
    table, span = box, 1                        # table[k]: the union of box k .. k + span - 1
    while span <= n:
        here = (last - first + 1 >= span) & (last - first + 1 < 2 * span)
        node[here] = torch.minimum(table[first[here]], table[last[here] - span + 1])
        if 2 * span > n:
            break
        table, span = torch.minimum(table[:n - 2 * span + 1], table[span:n - span + 1]), 2 * span

    def pair(b):
        out = torch.zeros(b.shape[0], 8, dtype=torch.float64, device="cuda")
        out[:, 0:3], out[:, 4:7] = b[:, :3], -b[:, 3:]
        return out
    return dict(keys=key, order=order.int(), children=None, node_range=torch.stack([first, last], 1).int(),
                node_boxes=pair(node), leaf_boxes=pair(box))


def _exact_net(params, rgb, gb):
    """The denoiser's forward pass in 64 bits: params is the flat parameter tensor (differentiable)."""
    F = torch.nn.functional
    n, h, w, _ = rgb.shape
    rgb, gb = rgb.double(), gb.double()
    r = rgb.clamp(min=0)
    nrm = gb[..., 0:3]
    l1 = nrm.abs().sum(-1, keepdim=True)
    q = torch.where(l1 > 0, nrm[..., :2] / l1.clamp(min=1e-300), nrm[..., :2])
    fold = (1 - q.abs().flip(-1)) * torch.where(q >= 0, 1.0, -1.0).double()
    octa = torch.where((nrm[..., 2:3] < 0) & (l1 > 0), fold, q)
    depth = gb[..., 3:4]
    dep = torch.where(depth >= 999999.0, torch.ones_like(depth), depth / (1 + depth))
    lum = torch.log1p((rgb @ torch.tensor([0.2126, 0.7152, 0.0722], device="cuda", dtype=torch.float64)).clamp(min=0))
    win = F.pad(lum[:, None], (1, 1, 1, 1), mode="replicate").unfold(2, 3, 1).unfold(3, 3, 1).reshape(n, h, w, 9)
    var = win.var(-1, unbiased=False, keepdim=True)
    feat = torch.cat([torch.log1p(r), gb[..., 4:7], octa, dep, var, torch.log1p(gb[..., 7:8].clamp(min=0).sqrt())], -1)
    feat = F.pad(feat, (0, 32 - feat.shape[-1])).permute(0, 3, 1, 2)
    feat = F.pad(feat, (0, -w % 16, 0, -h % 16))
    layers = layer_slices()

    def conv(k, x):
        _, ws, bs, shape = layers[k]
        wt = params[ws].reshape(3, 3, shape[1], shape[2]).permute(3, 2, 0, 1)
        y = F.conv2d(x, wt, params[bs], padding=1)
        return y.relu() if SPECS[k][2] else y
    skips, x = [], feat
    for level in range(5):
        x = conv(2 * level + 1, conv(2 * level, x))
        if level < 4:
            skips.append(x)
            x = F.avg_pool2d(x, 2)
    for level in range(4):
        x = torch.cat([F.interpolate(x, scale_factor=2, mode="nearest"), skips[3 - level]], 1)
        x = conv(11 + 2 * level, conv(10 + 2 * level, x))
    wts = conv(18, x)[:, :25, :h, :w].softmax(1)
    pad = F.pad(r.permute(0, 3, 1, 2), (2, 2, 2, 2), mode="replicate")
    out = 0
    for k in range(25):
        out = out + wts[:, k:k + 1] * pad[:, :, k // 5:k // 5 + h, k % 5:k % 5 + w]
    return out.permute(0, 2, 3, 1)


def _exact_filter(case, seed):
    s = prepare(case, seed)
    gb, h, w = s["gbuffer"].double(), case["height"], case["width"]
    img = s["rgb"].double()
    for axis in (1, 0):
        acc, total = torch.zeros_like(img), torch.zeros(h, w, 1, dtype=torch.float64, device="cuda")
        for i in range(-16, 17):
            at = (torch.arange(img.shape[axis], device="cuda") + i).clamp(0, img.shape[axis] - 1)
            p, g = img.index_select(axis, at), gb.index_select(axis, at)
            e = (i * i / (2 * 8.0 ** 2) + ((p - img) ** 2).sum(-1) / (2 * 5.0 ** 2)
                 + ((g - gb)[..., :3] ** 2).sum(-1) / (2 * 0.1 ** 2) + (g - gb)[..., 3] ** 2 / (2 * 0.2 ** 2))
            wt = torch.exp(-e)[..., None]
            acc, total = acc + wt * p, total + wt
        img = acc / total

    def frame(c):
        f, at = np.array(c.look_from), np.array(c.look_at)
        fwd = at - f
        focal = float(np.linalg.norm(fwd))
        fwd = fwd / focal
        right = np.cross(fwd, [0.0, 1.0, 0.0])
        right /= np.linalg.norm(right)
        vh = 2 * math.tan(math.radians(c.vfov_deg) / 2) * focal
        return f, right, np.cross(right, fwd), fwd, focal, vh * w / h, vh
    f, right, up, fwd, focal, vw, vh = frame(s["camera"])
    x = (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w - 0.5
    y = (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h - 0.5
    vec = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)  # noqa: E731
    d = vec(fwd) * focal + x[None, :, None] * vw * vec(right) + y[:, None, None] * vh * vec(up)
    pos = vec(f) + gb[..., 3:4] * d / d.norm(dim=-1, keepdim=True)
    f, right, up, fwd, focal, vw, vh = frame(s["before"])
    v = pos - vec(f)
    z = v @ vec(fwd)
    u, t = 0.5 + (v @ vec(right)) / z * focal / vw, 0.5 + (v @ vec(up)) / z * focal / vh
    inside = (gb[..., 3] < 999999.0) & (u >= 0) & (t >= 0) & (u <= 1) & (t <= 1)
    i = torch.where(inside, (u * w).clamp(0, w - 1), torch.arange(w, device="cuda")[None, :].double()).long()
    j = torch.where(inside, (t * h).clamp(0, h - 1), torch.arange(h, device="cuda")[:, None].double()).long()
    return 0.1 * img + 0.9 * s["prev"].double()[j, i]


def exact(case, seed):
    kind = case["kind"]
    if kind == "probe" and 20 * case["freq"] ** 2 * case["rays"] <= 1_000_000_000:
        tri = torch.from_numpy(_mesh_scene(case["freq"], seed).tri_vertices).cuda()
        return _exact_hits(tri, _rays(case["rays"], seed + 1))
    if kind == "build":
        return _exact_build(case, seed)
    if kind == "denoise":
        params = torch.from_numpy(np.load(training.DEFAULT_WEIGHTS)["params"]).cuda().double()
        rgb, gb, _ = _images(1, case["height"], case["width"], seed)
        with torch.no_grad():
            return _exact_net(params, rgb, gb)
    if kind == "train":
        params = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_()
        rgb, gb, target = _images(case["batch"], case["size"], case["size"], seed)
        px = rgb[..., 0].numel() * 3
        loss = 0.0
        for k in range(case["batch"]):
            out = _exact_net(params, rgb[k:k + 1], gb[k:k + 1])
            part = ((out.clamp(min=0) + 1e-3).sqrt() - (target[k:k + 1].double() + 1e-3).sqrt()).abs().sum() / px
            part.backward()
            loss += float(part.detach())
        return dict(loss=loss, grads=params.grad)
    if kind == "filter":
        return _exact_filter(case, seed)
    return None   # a path tracer's images and 10M-ray hit lists: minutes in 64 bits
