"""The work that a user of the renderer has it do, as cases that can be timed.

Every case goes through ``lsystemeditor_b200.pathtracer.PathTracer`` the way an
editor, a batch job or an optimisation loop calls it: scene, camera and
parameters are set in ``prepare``, ``run`` is one complete call sequence with
its result read back into pinned host memory.  Kinds:

  frame    reset, render to the sample budget or to convergence, read back
  waves    reset, then single waves with a read-back after each (the
           progressive display of an editor viewport)
  load     upload a host mesh (device BVH build), first wave, read back
  grow     loft a procedural tree on the device, build, preview passes, first
           wave, read back (the edit loop of a procedural scene)
  batch    several uneven trees in one render
  forest   one view of an instanced forest under sun and sky
  adjoint  one optimisation step: new materials, forward render with the
           per-sample record, read back, path-replay gradient
  rays     closest-hit queries from host arrays (surface picking, visibility)

The geometries are the benchmark grammars of ``lsystemeditor_b200.scene`` and
are kept once per process; the seed of ``prepare`` draws the materials, the
camera and, for rays and gradients, the query data.
"""
import functools
import math

import numpy as np
import torch

from lsystemeditor_b200 import scene as S
from lsystemeditor_b200.pathtracer import PathTracer
from lsystemeditor_b200.records import MATERIAL_DTYPE, TEXTURE_DTYPE, default_material, default_params, look_at_camera


# --- cases ------------------------------------------------------------------
def _frame(name, scene, width, height, min_spp, max_spp, wavelengths, depth, lens=False, sky=False, mis=False,
           rel=0.01):
    return dict(name=name, kind="frame", scene=scene, width=width, height=height, min_spp=min_spp, max_spp=max_spp,
                wavelengths=wavelengths, depth=depth, lens=lens, sky=sky, mis=mis, rel=rel)


def listed():
    return [
        # the smallest call: a thumbnail-sized viewport, one sample per pixel, thin lens, after a camera move
        _frame("thumbnail", "bracket", 96, 64, 1, 1, 0, 32, lens=True),
        # the repository's small workload as it stands: 256^2, 64 spp fixed, 4 hero wavelengths, depth 8
        _frame("small-frame", "bracket", 256, 256, 64, 64, 4, 8),
        # glass, metal, subsurface, textures under an environment map, ragged image size, the default depth
        _frame("materials-sky", "zoo", 641, 359, 16, 16, 0, 32, sky=True),
        # the repository's large workload (1M triangles, 1024^2, 8 wavelengths, depth 12, relative std-error
        # 0.01) with its adaptive budget cut at 256 of 1024 samples per pixel
        _frame("large-frame", "tree7", 1024, 1024, 16, 256, 8, 12),
        # small lights found by emitter MIS: real shadow rays through the canopy
        _frame("emitter-mis", "tree7", 513, 511, 32, 32, 0, 12, mis=True),
        # an editor's progressive display of the large scene: a wave, a read-back, a wave, ...
        dict(name="progressive", kind="waves", scene="tree7", width=1024, height=1024, waves=4, wavelengths=0, depth=12),
        # opening a scene: a 1M-triangle host mesh uploaded and built, first wave shown
        dict(name="open-mesh", kind="load", scene="tree7", width=640, height=360, waves=1, wavelengths=0, depth=12),
        # editing a procedural scene: device loft and build of 131k triangles, previews, first wave
        dict(name="regrow", kind="grow", iterations=6, width=800, height=450, levels=3, waves=1, depth=12),
        # uneven scenes in one render (relative std-error stop, black-pixel stop, emitter MIS)
        dict(name="batch", kind="batch", count=6, first=0, size=320, min_spp=16, max_spp=64, depth=12),
        # instanced forest: 200 instances of 3 trees, sun + sky, 8 wavelengths, depth 16
        dict(name="forest", kind="forest", width=960, height=540, spp=8, wavelengths=8, depth=16),
        # the repository's differentiation workload: 512^2, 64 spp forward + 64 spp adjoint, 10 materials
        dict(name="adjoint", kind="adjoint", width=512, height=512, spp=64, depth=8),
        # 200k closest-hit queries from host memory, results back in host memory
        dict(name="rays", kind="rays", scene="bracket", n=200_003),
    ]


def _odd(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "waves", "load", "grow", "batch", "forest", "adjoint", "rays"])
    wl = rng.choice([0, 4, 8])
    if kind == "rays":
        return dict(kind=kind, scene=rng.choice(["bracket", "tree7"]), n=_odd(rng, 1, 1_000_000))
    w, h = _odd(rng, 33, 1024), _odd(rng, 33, 1024)
    if kind == "waves":
        return dict(kind=kind, scene=rng.choice(["bracket", "tree7"]), width=w, height=h, waves=rng.randint(1, 8),
                    wavelengths=wl, depth=rng.choice([8, 12, 32]))
    if kind == "load":
        return dict(kind=kind, scene=rng.choice(["bracket", "tree7", "zoo"]), width=w, height=h, waves=rng.randint(1, 4),
                    wavelengths=wl, depth=rng.choice([8, 12]))
    if kind == "grow":
        return dict(kind=kind, iterations=rng.choice([4, 5, 6, 7]), width=w, height=h, levels=rng.randint(0, 4),
                    waves=rng.randint(1, 4), depth=rng.choice([8, 12]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 8), first=rng.randint(0, 3), size=_odd(rng, 64, 320),
                    min_spp=rng.choice([4, 16]), max_spp=rng.choice([16, 32, 64]), depth=12)
    if kind == "forest":
        return dict(kind=kind, width=w, height=h, spp=rng.randint(1, 8), wavelengths=wl, depth=rng.choice([8, 16]))
    if kind == "adjoint":
        return dict(kind=kind, width=_odd(rng, 64, 512), height=_odd(rng, 64, 512), spp=rng.choice([4, 16, 37, 64]),
                    depth=8)
    scene = rng.choice(["bracket", "zoo", "tree7"])
    spp = _odd(rng, 1, 64)
    return dict(kind="frame", scene=scene, width=w, height=h, min_spp=spp, max_spp=rng.choice([spp, 2 * spp]),
                wavelengths=wl, depth=rng.choice([8, 12, 32]), lens=rng.random() < 0.3, sky=rng.random() < 0.3,
                mis=scene != "zoo" and rng.random() < 0.3, rel=0.02)


# --- geometry (the seed does not enter: kept once per process) -----------------
@functools.lru_cache(maxsize=None)
def _geometry(name):
    """(mesh, centre, extent) of a named scene."""
    if name == "bracket":
        mesh = S.config0_scene().mesh
        body = mesh.positions[:20000].reshape(-1, 3)
    elif name == "zoo":
        mesh = _zoo()
        body = mesh.positions[:2400].reshape(-1, 3)
    else:
        tubes = _tubes(int(name[4:]), 7, 64)
        mesh = tubes.host_mesh()
        body = mesh.positions[: 2 * tubes.sides * len(tubes.radii) + 2 * len(tubes.leaves)].reshape(-1, 3)
    lo, hi = body.min(0), body.max(0)
    return mesh, (lo + hi) * 0.5, float((hi - lo).max())


@functools.lru_cache(maxsize=None)
def _tubes(iterations, seed, sides):
    return S.tree_tubes(iterations=iterations, seed=seed, sides=sides, rings=16)


@functools.lru_cache(maxsize=None)
def _batch(count, first):
    """Uneven trees of the batching grammar: iterations 4..7, L-system seeds 100, 101, ..."""
    return [_tubes(4 + (k * 3 + first) % 4, 100 + k, 48) for k in range(count)]


@functools.lru_cache(maxsize=None)
def _forest():
    return S.forest_scene(trees=3, instances=200, extent=120.0, iterations=(6, 7), views=1)


@functools.lru_cache(maxsize=None)
def _bands():
    return S.config3_scene().mesh


def _zoo():
    """Small triangles of eight materials (one per lobe combination of the BSDF), two textures, ground and light."""
    rng = np.random.default_rng(3)
    n = 2400
    c = rng.uniform(-2.5, 2.5, (n, 1, 3))
    pos = (c + rng.normal(scale=0.5, size=(n, 3, 3))).astype(np.float32)
    face = np.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0])
    face /= np.linalg.norm(face, axis=1, keepdims=True) + 1e-12
    nrm = (face[:, None, :] + rng.normal(scale=0.2, size=(n, 3, 3))).astype(np.float32)
    mats = [default_material(r=0.7, g=0.6, b=0.5, roughness=0.6, albedo_tex=1),
            default_material(r=0.9, g=0.8, b=0.3, roughness=0.25, metallic=1.0),
            default_material(r=0.95, g=0.95, b=0.95, roughness=0.02, transmission=1.0, ior=1.5),
            default_material(r=0.9, g=0.9, b=0.95, roughness=0.4, transmission=1.0, ior=1.33),
            default_material(r=0.6, g=0.9, b=0.6, roughness=0.5, transmission=0.3, thin=1.0),
            default_material(r=0.8, g=0.5, b=0.4, roughness=0.5, subsurface=1.0, scatter_radius_r=0.3,
                             scatter_radius_g=0.1, scatter_radius_b=0.05),
            default_material(r=0.5, g=0.5, b=0.5, roughness=0.9, diffuse_roughness=0.2, specular=0.3, roughness_tex=2),
            default_material(r=1.0, g=0.9, b=0.8, emission=4.0)]
    tex = np.zeros(3, TEXTURE_DTYPE)
    tex[1]["kind"], tex[1]["p0"], tex[1]["p1"], tex[1]["p2"] = 2, [8, 8, 0.1, 0], [0.1, 0.1, 0.1, 0], [0.9, 0.9, 0.9, 0]
    tex[2]["kind"], tex[2]["p0"] = 3, [6.0, 0.5, 0.9, 0.1]
    soup = S.HostMesh(pos, nrm, rng.uniform(0, 1, (n, 3, 2)).astype(np.float32), (np.arange(n) % 8).astype(np.uint32),
                      np.array(mats, MATERIAL_DTYPE), tex)
    ground = S.quad_mesh((0, -3.2, 0), (12, 0, 0), (0, 0, -12), default_material(r=0.5, g=0.5, b=0.5, roughness=1.0),
                         normal=(0, 1, 0))
    light = S.quad_mesh((0, 4.0, 0), (2, 0, 0), (0, 0, 2), default_material(r=1, g=1, b=1, emission=8.0),
                        normal=(0, -1, 0))
    return S.HostMesh.concat([soup, ground, light])


# --- what the seed draws -------------------------------------------------------
def _materials(mats, rng):
    """The bank with other colours and roughnesses (emitters keep theirs)."""
    out = mats.copy()
    for m in out:
        if m["emission"] == 0.0:
            for ch in "rgb":
                m[ch] = np.clip(m[ch] * rng.uniform(0.8, 1.2), 0.02, 0.98)
            m["roughness"] = np.clip(m["roughness"] * rng.uniform(0.8, 1.2), 0.02, 1.0)
    return out


def _with_materials(mesh, rng):
    return S.HostMesh(mesh.positions, mesh.normals, mesh.uvs, mesh.material_ids, _materials(mesh.materials, rng),
                      mesh.textures)


def _camera(rng, centre, extent, width, height, lens=False):
    dist = extent * 0.5 / math.tan(math.radians(20.0)) * 1.2
    az = rng.uniform(-0.3, 0.3)
    eye = (centre[0] + dist * math.sin(az), centre[1] + rng.uniform(0.0, 0.1) * dist, centre[2] + dist * math.cos(az))
    kw = dict(aperture_radius=0.02 * extent, focus_distance=dist) if lens else {}
    return look_at_camera(eye, centre, fov_y_deg=40.0, aspect=width / height, **kw)


def _sky(rng, width=64, height=32):
    v = (np.arange(height) + 0.5) / height
    img = np.stack([0.3 + 0.7 * (1 - v), 0.4 + 0.5 * (1 - v), 0.8 + 0.2 * (1 - v)], -1)[:, None, :].repeat(width, 1)
    img[height // 5, width // 3] = [40.0, 38.0, 30.0]
    return (img + rng.uniform(0, 0.05, img.shape)).astype(np.float32)


def _pinned(width, height):
    return (torch.empty((height, width, 4), dtype=torch.float32, pin_memory=True).numpy(),
            torch.empty((height, width), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32),
            torch.empty((height, width), dtype=torch.uint8, pin_memory=True).numpy())


def _black(**kw):
    return default_params(background_r=0.0, background_g=0.0, background_b=0.0, russian_roulette_min_depth=3, **kw)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = dict(case=case, pt=PathTracer(0))
    pt = st["pt"]
    if kind == "batch":
        tubes = _batch(case["count"], case["first"])
        sizes = [(case["size"] + 32 * (k % 3),) * 2 for k in range(len(tubes))]
        pt.batch_configure(sizes)
        for k, t in enumerate(tubes):
            pt.batch_set_tubes(k, t)
            pt.set_materials(_materials(t.extra.materials, rng), scene=k)
            lo, hi = t.bounds()
            w, h = sizes[k]
            pt.batch_set_camera(k, _camera(rng, (lo + hi) * 0.5, float((hi - lo).max()), w, h))
        pt.set_params(_black(max_path_depth=case["depth"], min_samples=case["min_spp"],
                             max_samples_per_pixel=case["max_spp"], relative_error_threshold=0.02, adaptive_criterion=2,
                             emitter_mis=1))
        return st
    if kind == "rays":
        mesh, _, _ = _geometry(case["scene"])
        pt.configure(16, 16, mesh)
        lo, hi = mesh.bounds()
        n = case["n"]
        st["origins"] = rng.uniform(lo - 1.0, hi + 1.0, (n, 3)).astype(np.float32)
        st["dirs"] = (rng.uniform(lo, hi, (n, 3)) - st["origins"]).astype(np.float32)
        return st
    w, h = case["width"], case["height"]
    st["out"] = _pinned(w, h)
    pt.configure(w, h)
    if kind == "forest":
        scene, cams, params, sun = _forest()
        objects = [scene.objects[0], *scene.objects[1:]]
        objects[0] = _with_materials(objects[0], rng)
        pt.set_instances(objects, scene.instances)
        pt.set_distant_light(**sun)
        az = rng.uniform(0.0, 2.0 * math.pi)
        pt.set_camera(look_at_camera((56.0 * math.sin(az), 6.0, 56.0 * math.cos(az)), (0.0, 4.0, 0.0), fov_y_deg=40.0,
                                     aspect=w / h))
        p = params.copy()
        p["max_path_depth"] = case["depth"]
        p["min_samples"] = p["max_samples_per_pixel"] = case["spp"]
        p["spectral_wavelengths"] = case["wavelengths"]
        pt.set_params(p)
        return st
    if kind == "grow":
        st["tubes"] = _tubes(case["iterations"], 7, 64)
        st["materials"] = _materials(st["tubes"].extra.materials, rng)
        lo, hi = st["tubes"].bounds()
        pt.set_camera(_camera(rng, (lo + hi) * 0.5, float((hi - lo).max()), w, h))
        pt.set_preview_steps_per_level(case["levels"])
        pt.set_params(_black(max_path_depth=case["depth"]))
        return st
    if kind == "adjoint":
        mesh = _bands()
        mats = mesh.materials.copy()
        mats[:8] = S.diff_materials(rng, 8)
        mats["emission"][9] = rng.uniform(5.0, 20.0)
        st["materials"] = mats
        pt.set_mesh(mesh)
        body = mesh.positions[:20000].reshape(-1, 3)
        lo, hi = body.min(0), body.max(0)
        pt.set_camera(_camera(rng, (lo + hi) * 0.5, float((hi - lo).max()), w, h))
        pt.set_params(_black(max_path_depth=case["depth"], min_samples=case["spp"], max_samples_per_pixel=case["spp"]))
        pt.record_samples(case["spp"])
        st["target"] = rng.uniform(0.0, 0.5, (h, w, 3)).astype(np.float32)
        return st
    mesh, centre, extent = _geometry(case["scene"])
    st["mesh"] = _with_materials(mesh, rng)
    if kind != "load":
        pt.set_mesh(st["mesh"])
    pt.set_camera(_camera(rng, centre, extent, w, h, case.get("lens", False)))
    if case.get("sky", False):
        pt.set_environment(_sky(rng))
    spp = dict(min_samples=case["min_spp"], max_samples_per_pixel=case["max_spp"], adaptive_criterion=1,
               relative_error_threshold=case["rel"], emitter_mis=int(case["mis"])) if kind == "frame" else {}
    pt.set_params(_black(max_path_depth=case["depth"], spectral_wavelengths=case["wavelengths"], **spp))
    return st


def _image(out):
    return {"rgba": out[0], "counts": out[1].view(np.int32), "converged": out[2]}


def run(st):
    case, pt = st["case"], st["pt"]
    kind = case["kind"]
    if kind == "rays":
        r = pt.trace_rays(st["origins"], st["dirs"])
        return {"t": r["t"], "normal": r["normal"], "uv": r["uv"], "hit": r["hit"].view(np.uint8),
                "tri": r["tri"].view(np.int32)}
    if kind == "batch":
        pt.reset_accumulation()
        pt.render(0)
        return [_image(pt.batch_readback(k)) for k in range(case["count"])]
    if kind == "load":
        pt.set_mesh(st["mesh"])
    elif kind == "grow":
        pt.batch_set_tubes(0, st["tubes"])
        pt.set_materials(st["materials"])
    elif kind == "adjoint":
        pt.set_materials(st["materials"])
    pt.reset_accumulation()
    if kind == "waves":
        for _ in range(case["waves"]):
            pt.render(1)
            pt.readback(st["out"])
        return _image(st["out"])
    pt.render(case.get("waves", 0))
    pt.readback(st["out"])
    res = _image(st["out"])
    if kind == "grow":
        res["previews"] = [pt.preview(k) for k in range(case["levels"])]
    elif kind == "adjoint":
        residual = st["out"][0][..., :3] - st["target"]
        grad, _ = pt.backward(2.0 * residual, case["spp"], materials=len(st["materials"]))
        res["grad"] = grad
    return res


# --- what a pass cannot do without ----------------------------------------------
# Arithmetic per ray and per shaded vertex: a ray of these scenes visits about 6
# eight-wide nodes (8 slab tests of 20 operations) and tests about 5 triangles
# (47 operations); a vertex takes about 400 operations.  Rays per sample: 1.5
# (counted on the large workload).
_RAY_FLOPS = 6 * 8 * 20 + 5 * 47
_VERTEX_FLOPS = 400


def work(case):
    kind = case["kind"]
    if kind == "rays":
        tris = 972_262 if case["scene"] == "tree7" else 20_004
        return {"bytes": case["n"] * (32 + 1 + 4 + 4 + 12 + 8) + 36 * tris, "flops": case["n"] * _RAY_FLOPS}
    if kind == "batch":
        tubes = _batch(case["count"], case["first"])
        tris = sum(t.triangle_count for t in tubes)
        pixels = sum((case["size"] + 32 * (k % 3)) ** 2 for k in range(len(tubes)))
        samples, rays = pixels * 0.5 * (case["min_spp"] + case["max_spp"]), 2.5
    else:
        pixels = case["width"] * case["height"]
        rays = 1.5
        if kind == "forest":
            tris, samples, rays = _forest()[0].unique_triangles, pixels * case["spp"], 3.0
        elif kind == "grow":
            tris, samples = _tubes(case["iterations"], 7, 64).triangle_count, pixels * (case["waves"] + 0.33)
        elif kind == "adjoint":
            tris, samples = 20_004, 2 * pixels * case["spp"]
        else:
            tris = {"bracket": 20_004, "zoo": 2_404, "tree7": 972_262}[case["scene"]]
            samples = pixels * (0.9 * case["max_spp"] if kind == "frame" else case["waves"])
            rays = 4.0 if case["scene"] == "zoo" else 1.5
    n = 36 * tris + 64 * tris + 21 * pixels * (case["waves"] if kind == "waves" else 1)
    return {"bytes": n, "flops": samples * rays * (_RAY_FLOPS + _VERTEX_FLOPS)}


# --- exact values ----------------------------------------------------------------
def exact(case, seed):
    """The hit parameter t of the ray queries by brute force over all triangles in 64 bits (0 where nothing is hit).

    A rendered image is an estimate from the renderer's own random numbers: there is no 64-bit value to hold it to
    without them.  The queries of the 972k-triangle scene would take too long.
    """
    if case["kind"] != "rays" or case["scene"] != "bracket":
        return None
    rng = np.random.default_rng(seed)
    mesh = _geometry(case["scene"])[0]
    lo, hi = mesh.bounds()
    n = case["n"]
    origins = rng.uniform(lo - 1.0, hi + 1.0, (n, 3)).astype(np.float32)
    dirs = (rng.uniform(lo, hi, (n, 3)) - origins).astype(np.float32)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.from_numpy(np.ascontiguousarray(mesh.positions)).to(dev, torch.float64).reshape(-1, 3, 3)
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    o = torch.from_numpy(origins).to(dev, torch.float64)
    d = torch.from_numpy(dirs).to(dev, torch.float64)
    d = d / d.norm(dim=1, keepdim=True)
    # the ray/triangle equations as matrix products over (rays, triangles), with the ray's moment m = o x d:
    # det = -d . (e1 x e2), t = (o - v0) . (e1 x e2) / det, u = (m . e2 - d . (e2 x v0)) / det, w likewise
    ng = torch.linalg.cross(e1, e2)
    best = torch.empty(n, dtype=torch.float64, device=dev)
    step = max(1, 60_000_000 // len(v0))
    for a in range(0, n, step):
        oc, dc = o[a:a + step], d[a:a + step]
        m = torch.linalg.cross(oc, dc)
        det = -(dc @ ng.T)
        t = (oc @ ng.T - (v0 * ng).sum(1)) / det
        u = ((m @ e2.T) - dc @ torch.linalg.cross(e2, v0).T) / det
        w = -((m @ e1.T) - dc @ torch.linalg.cross(e1, v0).T) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0) & (t < 1e6)
        tc = torch.where(ok, t, torch.full_like(t, math.inf)).amin(1)
        best[a:a + step] = torch.where(torch.isfinite(tc), tc, torch.zeros_like(tc))
    return {"t": best.cpu().numpy(), "normal": None, "uv": None, "hit": None, "tri": None}
