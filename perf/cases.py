"""The renders and queries whose speed matters: the work a program has this
library do, through its public entry points.

Each case is a dict of plain values; `kind` names the entry point, `scene` the
scene family (the workloads of rustracer_b200/configs.py, varied by the seed).

  frame     GpuScene.render_accumulate into CUDA tensors: a still, or one step of
            a progressive render.  `photons` > 0 rebuilds the caustic map first,
            as a program whose lights or gems move does every frame; `guide`
            bounces from a frozen learned proposal.
  preview   render_accumulate and develop: what an interactive viewer does per frame.
  pass      GpuScene.render_tiles: the reference's own signature, one sample
            pass into host memory with a mask of converged pixels.
  batch     GpuScene.render_batch: many small requests of one scene.
  rays      GpuScene.trace_closest on CUDA tensors: ray queries of a host program.
  load      GpuScene(builder): copying a mesh and building its hierarchy, then the
            first query on it.
  guide     GpuScene.guide_loss_grad: the training direction of the proposal.
"""
import functools
import math
import random

import numpy as np
import torch

from rustracer_b200 import configs, photons
from rustracer_b200.renderer import GpuScene, guide_params, pass_params
from rustracer_b200.scene import Material, SceneBuilder, make_camera

LEVELS, TABLE, NIN, NOUT, NOUTP = 16, 1 << 19, 64, 41, 48      # the proposal network's shape


# ── the cases ────────────────────────────────────────────────────────────────
def listed():
    return [
        # a viewer's frame while the camera moves: launches and latency are all of it
        dict(name="preview_box_160x120", kind="preview", scene="box", width=160, height=120, spp=1, depth=8, hero=1),
        # the small workload of the benchmark: one pool of paths, a handful of bounces
        dict(name="box_256x256_16spp", kind="frame", scene="box", width=256, height=256, spp=16, depth=8, hero=4),
        # the headline workload: 1.3M triangles of a rough conductor under a sky map
        dict(name="mesh8_1080p_64spp", kind="frame", scene="mesh", levels=8, width=1920, height=1080, spp=64,
             depth=12, hero=4),
        # one progressive sample pass of the reference's loop at an odd size, a third
        # of the pixels converged, single-wavelength paths, host memory
        dict(name="mesh7_pass_961x541", kind="pass", scene="mesh", levels=7, width=961, height=541, spp=1, depth=50,
             hero=1),
        # a gem on a plane: dispersion, long paths, the caustic map rebuilt every frame
        dict(name="gem_720p_16spp_2Mphotons", kind="frame", scene="gem", width=1280, height=720, spp=16, depth=32,
             hero=4, photons=2_000_000),
        # the reference's own benchmark room: analytic gems, PBR, a physical sky with
        # its sun, and a caustic map with a wide fixed-radius gather
        dict(name="room_1200x800_8spp", kind="frame", scene="room", width=1200, height=800, spp=8, depth=50, hero=1,
             photons=500_000),
        # participating media: procedural noise and a constant-density ball
        dict(name="media_640x360_16spp", kind="frame", scene="media", width=640, height=360, spp=16, depth=24, hero=4),
        # the frozen learned proposal in the slit-lit room with a voxel-grid medium
        dict(name="guided_1280x720_4spp", kind="frame", scene="guided", width=1280, height=720, spp=4, depth=24,
             hero=4, guide=True),
        # a server packing thumbnails of one scene
        dict(name="batch_24_thumbnails", kind="batch", scene="mesh", levels=6, jobs=24, width=320, spp=32, depth=12,
             hero=4),
        # ray queries from a host program: incoherent rays against a large mesh
        dict(name="rays_4M_mesh7", kind="rays", scene="mesh", levels=7, n=4_000_003),
        # opening a scene: 327,680 triangles
        dict(name="load_mesh7", kind="load", scene="mesh", levels=7, n=65_536),
        # the backward direction of the learned proposal on one minibatch
        dict(name="guide_grad_65536", kind="guide", scene="box", n=65_536),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# most path samples of a drawn frame, so that none costs more than the largest listed case
MOST_SAMPLES = dict(box=24_000_000, mesh=64_000_000, gem=12_000_000, room=6_000_000, media=6_000_000,
                    guided=3_000_000)


def draw(rng):
    kind = rng.choice(["preview", "frame", "frame", "frame", "frame", "pass", "batch", "rays", "load", "guide"])
    if kind == "rays":
        return dict(kind=kind, scene="mesh", levels=rng.randint(4, 8), n=_logint(rng, 16_000, 8_000_000))
    if kind == "load":
        return dict(kind=kind, scene="mesh", levels=rng.randint(4, 7), n=_logint(rng, 16_000, 200_000))
    if kind == "guide":
        return dict(kind=kind, scene="box", n=_logint(rng, 1_000, 200_000))
    if kind == "batch":
        c = dict(kind=kind, scene=rng.choice(["mesh", "box"]), jobs=rng.randint(2, 48), width=_logint(rng, 48, 480),
                 spp=_logint(rng, 1, 64), depth=rng.randint(4, 16), hero=rng.choice([1, 4]))
        if c["scene"] == "mesh":
            c["levels"] = rng.randint(4, 7)
        while c["jobs"] * c["width"] ** 2 * c["spp"] > 48_000_000:
            c["spp"] = max(1, c["spp"] // 2)
            c["jobs"] = max(2, c["jobs"] * 3 // 4)
        return c
    scene = {"preview": lambda: rng.choice(["box", "mesh"]), "pass": lambda: rng.choice(["box", "mesh"]),
             "frame": lambda: rng.choice(["box", "mesh", "mesh", "gem", "room", "media", "guided"])}[kind]()
    width = _logint(rng, 96, 1920)
    height = max(64, int(width * rng.choice([1.0, 0.75, 0.5625])) | rng.randint(0, 1))
    c = dict(kind=kind, scene=scene, width=width, height=height, spp=1, depth=_logint(rng, 4, 50),
             hero=1 if scene == "room" else rng.choice([1, 4]))
    if scene == "mesh":
        c["levels"] = rng.randint(4, 8)
    if kind == "frame":
        c["spp"] = max(1, min(_logint(rng, 1, 64), MOST_SAMPLES[scene] // (width * height)))
        if scene in ("gem", "room"):
            c["photons"] = _logint(rng, 50_000, 2_000_000)
        if scene == "guided":
            c["guide"] = True
    return c


# ── scenes ───────────────────────────────────────────────────────────────────
@functools.lru_cache(maxsize=None)
def _sphere(levels):
    return configs.icosphere(levels)


@functools.lru_cache(maxsize=None)
def _sky(width, height, variant):
    return configs.sky_env(width, height, seed=variant)


def _mesh_scene(levels, seed, aspect, env=(1024, 512)):
    """A bumpy ball (20·4^levels triangles) of a rough gold-like conductor on a
    diffuse floor under a sky map with a sun: the icosphere workload with its bumps
    drawn from the seed (random plane waves, amplitude falling with frequency)."""
    rng = np.random.default_rng(seed)
    V, F = _sphere(levels)
    bump = np.zeros(len(V), np.float32)
    Vf = V.astype(np.float32)
    for k in range(20):
        w = rng.normal(size=3)
        f = 2.0 * 2.0 ** (k / 5.0)
        w = (w / np.linalg.norm(w) * f).astype(np.float32)
        bump += np.cos(Vf @ w + np.float32(rng.uniform(0, 2 * math.pi))) * np.float32(0.08 / f)
    V = V * (1.0 + bump.astype(np.float64))[:, None]
    fn = np.cross(V[F[:, 1]] - V[F[:, 0]], V[F[:, 2]] - V[F[:, 0]])
    N = np.stack([sum(np.bincount(F[:, k], weights=fn[:, a], minlength=len(V)) for k in range(3))
                  for a in range(3)], 1)
    N /= np.linalg.norm(N, axis=1, keepdims=True)
    sb = SceneBuilder()
    sb.spectral_range = 1
    n, k = configs.gold_like_nk()
    sb.add_mesh(V, F, sb.add_material(Material.spectral_metal_nk(380.0, 50.0, n, k, roughness=0.2)), N)
    floor = sb.add_material(Material.lambertian((0.5, 0.5, 0.5)))
    sb.add_quad((-10.0, -1.1, -10.0), (0.0, 0.0, 20.0), (20.0, 0.0, 0.0), floor)
    sky, _ = _sky(env[0], env[1], 2 + seed % 3)
    sb.set_env(sky)
    a = rng.uniform(-0.5, 0.5)
    cam = make_camera((3.6 * math.sin(a), 0.45, 3.6 * math.cos(a)), (0.0, -0.15, 0.0), vfov=40.0, aspect=aspect)
    return sb, cam


def _builder(case, seed):
    """(SceneBuilder, camera, photon params or None) of a case and seed."""
    aspect = case.get("width", 1) / case.get("height", 1)
    scene = case["scene"]
    j = random.Random(seed)
    if scene == "mesh":
        env = (2048, 1024) if case["levels"] >= 8 else (1024, 512)
        return _mesh_scene(case["levels"], seed, aspect, env) + (None,)
    if scene == "box":
        sb, st = configs.box_scene(hero=case.get("hero", 1))
        sb.spheres.clear()
        sb.add_sphere((j.uniform(0.25, 0.35), 0.18, j.uniform(0.55, 0.65)), 0.18,
                      sb.add_material(Material.lambertian((0.73, 0.73, 0.73))))
        sb.add_sphere((j.uniform(0.65, 0.75), 0.18, j.uniform(0.3, 0.4)), 0.18,
                      sb.add_material(Material.spectral_dielectric_cauchy(1.5, 0.0042)))
    elif scene == "media":
        sb, st = configs.media_box_scene(hero=case["hero"], density=j.uniform(3.0, 5.0))
    elif scene == "guided":
        sb, st = configs.guided_box_scene(hero=case["hero"], density=j.uniform(3.0, 5.0), grid_res=64)
    elif scene == "gem":
        sb, st = configs.gem_scene(hero=case["hero"], photons=case["photons"])
        cam = make_camera((j.uniform(-0.4, 0.4), 1.55, 2.2), (0.0, 0.35, 0.0), vfov=32.0, aspect=aspect)
        return sb, cam, st["photon_params"](seed + 1)
    else:
        sb, st = configs.gem_room_scene()
        cam = make_camera((j.uniform(-0.3, 0.3), 3.4, -9.0), (0.0, 2.247, 1.1993), vfov=36.0, aspect=aspect)
        return sb, cam, photons.caustic_params(sb, case["photons"], st["radius"], seed=seed + 1)
    cam = make_camera((0.5 + j.uniform(-0.1, 0.1), 0.5, -1.4), (0.5, 0.5, 0.5), vfov=40.0, aspect=aspect)
    return sb, cam, None


def _outputs(pixels, flat=False):
    shape = (pixels[0] * pixels[1],) if flat else pixels
    rgb = (shape[0] * 3,) if flat else shape + (3,)
    return (torch.zeros(rgb, dtype=torch.float32, device="cuda"), torch.zeros(rgb, dtype=torch.float32, device="cuda"),
            torch.zeros(shape, dtype=torch.int32, device="cuda"))


def _rays(n, seed):
    """Incoherent rays: origins in a shell around the ball, aimed at points inside it."""
    g = torch.Generator().manual_seed(seed)
    o = torch.nn.functional.normalize(torch.randn(n, 3, generator=g), dim=1) * (1.2 + 2.0 * torch.rand(n, 1, generator=g))
    at = torch.nn.functional.normalize(torch.randn(n, 3, generator=g), dim=1) * (1.3 * torch.rand(n, 1, generator=g))
    r = torch.empty(n, 8)
    r[:, 0:3], r[:, 3:6], r[:, 6], r[:, 7] = o, torch.nn.functional.normalize(at - o, dim=1), 1e-3, math.inf
    return r.cuda()


def _guide_weights(seed):
    """Parameters as after some training: Glorot layers, a hash table whose entries
    spread over ±0.1, so that lobes follow position and direction."""
    rng = np.random.default_rng(seed)
    p = np.zeros(3 * 64 * 64 + NOUTP * 64 + LEVELS * TABLE * 2, np.float32)
    for l in range(4):
        rows = NOUTP if l == 3 else 64
        lim = math.sqrt(6.0 / (64 + (NOUT if l == 3 else 64)))
        W = rng.uniform(-lim, lim, (rows, 64)).astype(np.float32)
        W[NOUT if l == 3 else rows:] = 0.0
        p[l * 4096:l * 4096 + rows * 64] = W.reshape(-1)
    p[15360:] = rng.random(LEVELS * TABLE * 2, dtype=np.float32) * np.float32(0.2) - np.float32(0.1)
    return p


def _guide_samples(n, seed):
    """Training records of a room: positions, unit normals, outgoing and sampled
    directions, weights with the long tail that path radiance has."""
    rng = np.random.default_rng(seed + 17)
    unit = lambda: (lambda v: v / np.linalg.norm(v, axis=1, keepdims=True))(rng.normal(size=(n, 3)))
    N, D = unit(), unit()
    D = np.where((N * D).sum(1, keepdims=True) < 0, -D, D)
    return np.concatenate([rng.random((n, 3)), N, unit(), D, rng.lognormal(-1.0, 1.2, (n, 1))], 1).astype(np.float32)


# ── what a program holds before the call ─────────────────────────────────────
def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind)
    sb, cam, ph = _builder(case, seed)
    if kind == "load":
        st.update(builder=sb, rays=_rays(case["n"], seed))
        return st
    scene = GpuScene(sb)
    st.update(scene=scene, cam=cam, photons=ph)
    if kind == "rays":
        st.update(rays=_rays(case["n"], seed), hits=torch.zeros((case["n"], 4), dtype=torch.int32, device="cuda"))
        return st
    if kind == "guide":
        scene.guide_init(guide_params(record_capacity=1 << 16, domain=((0, 0, 0), (1, 1, 1))))
        scene.guide_set_params(_guide_weights(seed))
        st["samples"] = _guide_samples(case["n"], seed)
        return st
    if kind == "batch":
        sizes, j = random.Random(case["jobs"]), random.Random(seed)    # the seed moves the cameras, not the sizes
        jobs = []
        for k in range(case["jobs"]):
            w = max(16, int(case["width"] * sizes.uniform(0.6, 1.0)))
            h = max(16, int(w * sizes.choice([1.0, 0.75, 0.5625])))
            a = j.uniform(-0.4, 0.4)
            eye, at = ((3.6 * math.sin(a), 0.45, 3.6 * math.cos(a)), (0.0, -0.15, 0.0)) if case["scene"] == "mesh" \
                else ((0.5 + 0.2 * a, 0.5, -1.4), (0.5, 0.5, 0.5))
            jobs.append(dict(cam=make_camera(eye, at, vfov=40.0, aspect=w / h), width=w, height=h,
                             spp=max(1, int(case["spp"] * sizes.uniform(0.5, 1.0))), seed=seed * 1000 + k))
        tot = sum(q["width"] * q["height"] for q in jobs)
        st.update(jobs=jobs, shared=pass_params(16, 16, max_depth=case["depth"], hero=case["hero"]),
                  outputs=_outputs((1, tot), flat=True))
        return st
    W, H = case["width"], case["height"]
    if case.get("guide"):
        scene.guide_init(guide_params(record_capacity=1 << 16))
        scene.guide_set_params(_guide_weights(3))
        scene.guide_mode(1)
    st["params"] = pass_params(W, H, 0, case["spp"], max_depth=case["depth"], hero=case["hero"], seed=seed)
    if kind == "pass":
        st.update(scratch=np.zeros((H, W, 3), np.float32), depth=case["depth"], hero=case["hero"], seed=seed,
                  converged=(np.random.default_rng(seed).random((H, W)) < 0.33).astype(np.uint8))
    else:
        st["outputs"] = _outputs((H, W))
        if kind == "preview":
            st["rgb8"] = torch.zeros((H, W, 3), dtype=torch.uint8, device="cuda")
    return st


def run(st):
    kind = st["kind"]
    if kind == "load":
        scene = GpuScene(st["builder"])
        hits = scene.trace_closest(st["rays"], torch.empty((st["rays"].shape[0], 4), dtype=torch.int32, device="cuda"))
        scene.close()
        return hits
    scene = st["scene"]
    if kind == "rays":
        return scene.trace_closest(st["rays"], st["hits"])
    if kind == "guide":
        return scene.guide_loss_grad(st["samples"])
    if kind == "batch":
        s, m, c = st["outputs"]
        scene.render_batch(st["jobs"], st["shared"], outputs=(s, m, c))
        return s, m, c
    if kind == "pass":
        p = st["params"]
        return scene.render_tiles(st["scratch"], st["converged"], 0, 1, p.width, p.height, st["cam"],
                                  max_depth=st["depth"], hero=st["hero"], seed=st["seed"])
    if st["photons"] is not None:
        scene.photon_build(st["photons"])
    out = scene.render_accumulate(st["cam"], st["params"], outputs=st["outputs"])
    if kind == "preview":
        p = st["params"]
        return tuple(out) + (scene.develop(p.width, p.height, linear=out[0], out=st["rgb8"]),)
    return tuple(out)


# ── what a pass cannot do without ────────────────────────────────────────────
# mean ray segments (extension and shadow rays) of one path sample of each family
SEGMENTS = dict(box=9.0, mesh=3.0, gem=7.0, room=9.0, media=9.0, guided=6.0)
PRIMS = dict(box=8, gem=2290, room=1430, media=8, guided=2310)


def _prims(case):
    return 20 * 4 ** case["levels"] if case["scene"] == "mesh" else PRIMS[case["scene"]]


def _ray_flops(prims):
    # one 8-wide node (8 boxes × 18 operations) per level and two primitive tests of 50
    return (math.log(max(prims, 8), 8) + 1.0) * 144.0 + 100.0


def work(case):
    kind, prims = case["kind"], _prims(case)
    if kind == "guide":
        # the gradient leaves whole; three products per layer and row, forward and backward
        params = 15360 + LEVELS * TABLE * 2
        return dict(bytes=4.0 * params + 52.0 * case["n"] + 2.0 * params, flops=case["n"] * 6.0 * 15360)
    geometry = prims * 72.0                                     # corners and normals
    if kind == "rays":
        return dict(bytes=case["n"] * 48.0 + prims * 36.0, flops=case["n"] * _ray_flops(prims))
    if kind == "load":
        return dict(bytes=2.0 * geometry + case["n"] * 48.0,
                    flops=prims * math.log2(prims) * 20.0 + case["n"] * _ray_flops(prims))
    if kind == "batch":
        pixels = case["jobs"] * (0.8 * case["width"]) ** 2 * 0.77
        samples = pixels * case["spp"] * 0.75
    else:
        pixels = case["width"] * case["height"]
        samples = pixels * case["spp"] * (0.67 if kind == "pass" else 1.0)
    extra = case.get("photons", 0)
    flops = samples * SEGMENTS[case["scene"]] * (_ray_flops(prims) + 200.0) + extra * 3.0 * (_ray_flops(prims) + 100.0)
    if case.get("guide"):
        flops += samples * 2.0 * 2.0 * 15360
    return dict(bytes=geometry + pixels * (12.0 if kind == "pass" else 31.0 if kind == "preview" else 28.0)
                + extra * 0.12 * 48.0, flops=flops)


# ── the values in 64 bits ────────────────────────────────────────────────────
def exact(case, seed):
    """Images are defined by their paths' random streams and hits are whole numbers:
    neither has a value apart from the run.  The proposal's loss and gradient do."""
    if case["kind"] != "guide":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.from_numpy(_guide_weights(seed)).to(dev).double()
    s = torch.from_numpy(_guide_samples(case["n"], seed)).to(dev).double()
    pos, nrm, wo, d, w = s[:, 0:3], s[:, 3:6], s[:, 6:9], s[:, 9:12], s[:, 12]
    Ws = [p[l * 4096:l * 4096 + (NOUTP if l == 3 else 64) * 64].reshape(-1, 64).requires_grad_(True) for l in range(4)]
    table = p[15360:].reshape(LEVELS, TABLE, 2).requires_grad_(True)
    feats, res = [], 4.0
    for l in range(LEVELS):                                     # Müller et al. 2022: the multiresolution hash grid
        r = max(2, int(res))
        res *= 1.32
        x = pos * r
        c = x.floor().clamp(max=r - 1).long()
        f = x - c
        acc = 0.0
        for k in range(8):
            q = [c[:, a] + ((k >> a) & 1) for a in range(3)]
            if (r + 1) ** 3 <= TABLE:
                idx = q[0] + (r + 1) * (q[1] + (r + 1) * q[2])
            else:
                idx = (q[0] ^ (q[1] * 2654435761) ^ (q[2] * 805459861)) & (TABLE - 1)
            wk = 1.0
            for a in range(3):
                wk = wk * (f[:, a] if (k >> a) & 1 else 1.0 - f[:, a])
            acc = acc + wk[:, None] * table[l][idx]
        feats.append(acc)
    th = torch.acos(wo[:, 2].clamp(-1, 1)) / math.pi            # Müller et al. 2019: one-blob of the angles
    ph = (torch.atan2(wo[:, 1], wo[:, 0]) + math.pi) / (2.0 * math.pi)
    bins = torch.arange(16, device=dev, dtype=torch.float64) + 0.5
    h = torch.cat(feats + [torch.exp(-0.5 * (16.0 * t[:, None] - bins) ** 2) for t in (th, ph)], 1)
    for l in range(3):
        h = torch.relu(h @ Ws[l].T)
    o = (h @ Ws[3].T)[:, :NOUT]
    lob = o[:, :40].reshape(-1, 8, 5)
    mu = torch.nn.functional.normalize(lob[:, :, :3], dim=2)
    kap = torch.exp(lob[:, :, 3].clamp(-5.0, 5.0))
    cosd = (mu * d[:, None, :]).sum(2)
    dens = kap / (2 * math.pi * -torch.expm1(-2 * kap)) * torch.exp(kap * (cosd - 1))
    pg = (torch.softmax(lob[:, :, 4], 1) * dens).sum(1)
    pb = (nrm * d).sum(1).clamp(min=0) / math.pi
    alpha = 0.5 * torch.sigmoid(o[:, 40])
    mix = (alpha * pg.detach() + (1 - alpha) * pb).clamp(min=1e-8)
    n = float(case["n"])
    # the lobes descend −w·log p_vmf, the fraction −w·log p_mix with the lobes held fixed
    ((-w * torch.log(pg.clamp(min=1e-8))).sum() / n + (-w * torch.log(mix)).sum() / n).backward()
    grad = torch.cat([q.grad.reshape(-1) for q in Ws] + [table.grad.reshape(-1)])
    loss = (-w * torch.log((alpha * pg + (1 - alpha) * pb).clamp(min=1e-8))).sum()
    return float(loss), grad.detach().cpu().numpy()
