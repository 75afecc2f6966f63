"""Sizes where the bookkeeping of the list-building and cooperative kernels has
edges.

* Build: triangle counts around the widths of a compressed node, a leaf and a
  treelet; every ray's hit equals the oracle's brute force over all triangles.
* Adjoint: samples with a gradient are listed and replayed 32 at a time.  The
  gradient from the forward render's sample record equals the one that replays
  every path for its radiance, for fewer jobs than lanes, ragged images and
  sparse image gradients.  Both sum the same terms, of samples whose radiance
  differs by FP32 rounding, in another order: 1e-3 of the largest entry.
* Previews: several levels in one launch equal the levels of a renderer that
  has only the coarser ones.
* Next-bounce list and routing: more path slots than one step per warp covers.
"""
import numpy as np
import pytest

from lsystemeditor_b200.pathtracer import PathTracer
from lsystemeditor_b200.records import default_params
from tests.helpers import random_soup, rays_through_bounds, zoo_camera, zoo_scene
from tests.test_gpu_adjoint import _render, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 9, 15, 16, 17, 31, 33, 64, 129, 300])
def test_build_sizes_match_brute_force(tracer, oracle, n, passes):
    mesh = random_soup(n, seed=n, extent=1.0, size=0.6)
    o, d = rays_through_bounds(mesh, 2000, seed=n + 1)
    tracer.set_bvh_options(passes)
    tracer.configure(8, 8, mesh)
    tracer.set_bvh_options(1)
    g = tracer.trace_rays(o, d)
    r = oracle.scene(mesh).trace_bruteforce(o, d)
    assert g["hit"].any()
    assert np.array_equal(g["hit"], r["hit"])
    for k in ("t", "tri"):
        assert np.array_equal(g[k][g["hit"]], r[k][r["hit"]]), k


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("w, h, spp", [(1, 1, 1), (31, 1, 1), (33, 1, 2), (3, 43, 5), (61, 47, 3)])
def test_adjoint_lists_match_full_replay(tracer, w, h, spp, sparse):
    spec, _ = _setup(tracer, w, h, spp)
    rng = np.random.default_rng(w + h)
    d_image = rng.uniform(0.5, 1.5, (h, w, 3)).astype(np.float32)
    if sparse:
        d_image[rng.uniform(size=(h, w)) < 0.9] = 0.0
    tracer.record_samples(0)
    _render(tracer, spec.mesh.materials, spp)
    full, _ = tracer.backward(d_image, spp)
    tracer.record_samples(spp)
    _render(tracer, spec.mesh.materials, spp)
    listed, _ = tracer.backward(d_image, spp)
    tracer.record_samples(0)
    assert np.isfinite(full).all()
    assert np.abs(listed - full).max() <= 1e-3 * np.abs(full).max()


@pytest.mark.parametrize("w, h, levels", [(1, 1, 1), (7, 3, 3), (65, 33, 2), (40, 24, 18)])
def test_previews_in_one_launch(tracer, w, h, levels):
    mesh = zoo_scene(n_per_mat=40, seed=2)

    def previews(t, width, height, n):
        t.configure(width, height, mesh)
        t.set_camera(zoo_camera(w, h))
        t.set_params(default_params(background_r=0.2, background_g=0.3, background_b=0.4))
        t.set_preview_steps_per_level(n)
        t.render_previews()
        out = [t.preview(k) for k in range(n)]
        t.set_preview_steps_per_level(0)
        return out

    both = previews(tracer, w, h, levels)
    for k, img in enumerate(both):
        ds = 1 << (levels - k)
        assert img.shape[:2] == (max(h // ds, 1), max(w // ds, 1))
        assert np.isfinite(img).all() and (img[..., 3] == 1.0).all()
    # level 0 of a renderer with one level draws with the same seed (1) at half its size
    ph, pw = both[0].shape[:2]
    with PathTracer(0) as one:
        assert np.array_equal(previews(one, 2 * pw, 2 * ph, 1)[0], both[0])


def test_more_slots_than_one_step_per_warp(tracer):
    """2.6M path slots: every warp of the list pass takes several steps, the last one ragged."""
    w, h = 1601, 1599
    tracer.configure(w, h, zoo_scene(n_per_mat=20, seed=8))
    tracer.set_camera(zoo_camera(w, h))
    tracer.set_params(default_params(max_path_depth=4, min_samples=1, max_samples_per_pixel=1, background_r=0.4,
                                     background_g=0.5, background_b=0.6))
    out = []
    for mode in (1, 2):
        tracer.set_extend_mode(mode)
        tracer.reset_accumulation()
        tracer.render(0)
        out.append(tracer.readback())
    tracer.set_extend_mode(0)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 130_000, 131_073, 300_001])
def test_ray_queries_through_staged_copies(tracer, n):
    """Queries on both sides of the size from which host arrays are staged through pinned slices (4 MB in: 131072
    rays), with partial last slices, give what one query of the same rays in small parts gives."""
    mesh = zoo_scene(n_per_mat=30, seed=5)
    tracer.configure(8, 8, mesh)
    o, d = rays_through_bounds(mesh, n, seed=7)
    for _ in range(3):  # (transfers of this size are staged from the fifth on: two per query)
        whole = tracer.trace_rays(o, d)
    parts = [tracer.trace_rays(o[a:a + 60_000], d[a:a + 60_000]) for a in range(0, n, 60_000)]
    for k, v in whole.items():
        assert np.array_equal(v, np.concatenate([p[k] for p in parts])), k


@pytest.mark.parametrize("n", [40_000, 559_241, 900_001])
def test_staged_mesh_upload(tracer, n):
    """A mesh comes back bit for bit below and above the size (32 MB of normals and uvs) from which its arrays are
    staged through pinned slices at once."""
    mesh = random_soup(n, seed=2, extent=30.0, size=0.2, materials=3)
    tracer.configure(8, 8, mesh)
    back = tracer.export_mesh()
    for name in ("positions", "normals", "uvs", "material_ids"):
        assert np.array_equal(getattr(back, name), getattr(mesh, name)), name
