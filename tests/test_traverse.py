"""Whole-warp traversal (csrc/pt_traverse.cuh) and the plane decode of the
compressed nodes (csrc/pt_trace.cuh).

* CPU: the permute-and-subtract decode gives every plane byte exactly.
* GPU: the whole-warp kernels render what the one-ray-per-lane traversal
  renders, bit for bit, where their bookkeeping has edges: fewer rays than
  lanes, one more than a warp, a chunk or a block, single-triangle scenes, every
  hit an exact tie, rays with degenerate directions, one scene of a batch
  instanced and the others flat.
"""
import numpy as np
import pytest

from lsystemeditor_b200.records import default_params, look_at_camera
from lsystemeditor_b200.scene import HostMesh, placement
from tests.helpers import random_soup, zoo_camera, zoo_scene


def test_plane_decode_is_exact():
    """Byte j of a plane word placed under 0x4B0000.. (2^23) and 2^23 subtracted is float(byte): the plane
    parameters are then those of fmaf(float(q), a, b), whatever a and b."""
    f = np.float32
    words = (np.arange(256, dtype=np.uint64)[:, None] * np.array([1, 1 << 8, 1 << 16, 1 << 24], np.uint64)).astype(np.uint32)
    words = words | np.uint32(0x5A5A5A5A) & ~np.array([0xFF, 0xFF00, 0xFF0000, 0xFF000000], np.uint32)
    for j in range(4):
        sources = np.concatenate([words[:, j].copy().view(np.uint8).reshape(-1, 4),
                                  np.broadcast_to(np.array([0, 0, 0, 0x4B], np.uint8), (256, 4))], 1)
        for first in (0x7540, 0x7541):  # the two lanes of a pair; the kernel adds the pair's first byte
            if (first & 1) != (j & 1):
                continue
            selector = first + (j & 2)
            picked = sources[:, [(selector >> (4 * k)) & 7 for k in range(4)]]
            q = np.ascontiguousarray(picked).view(np.uint32).reshape(-1).view(f) - f(8388608.0)
            assert np.array_equal(q, np.arange(256, dtype=f))


def _images(t, mode):
    t.set_extend_mode(mode)
    t.reset_accumulation()
    t.render(0)
    out = [t.batch_readback(k) for k in range(len(t.batch_sizes))]
    assert t.stats()["stack_overflows"] == 0
    return [a for o in out for a in o]


def _same(t):
    warp, lane = _images(t, 1), _images(t, 2)
    for k, (a, b) in enumerate(zip(warp, lane)):
        assert np.array_equal(a, b), f"array {k} differs"
    if warp[0].size > 1000:  # (a pixel or a row alone may be black)
        assert warp[0][..., :3].max() > 0


def _tied(mesh, copies):
    """Every triangle `copies` times: each hit is an exact tie."""
    return HostMesh(np.repeat(mesh.positions, copies, 0), np.repeat(mesh.normals, copies, 0),
                    np.repeat(mesh.uvs, copies, 0), np.tile(np.arange(copies, dtype=np.uint32) % len(mesh.materials),
                                                            mesh.triangle_count), mesh.materials, mesh.textures)


SCENES = {
    "one triangle": lambda: random_soup(1, seed=1, extent=0.1, size=2.0),
    "soup": lambda: zoo_scene(n_per_mat=100, seed=4),
    "ties": lambda: _tied(random_soup(60, seed=2, size=1.0, materials=4), 7),
}


@pytest.mark.gpu
@pytest.mark.parametrize("scene", sorted(SCENES))
@pytest.mark.parametrize("width, height, spp", [(1, 1, 1), (33, 1, 1), (3, 43, 1), (37, 29, 5)])
def test_render_matches_single_lane_traversal(tracer, scene, width, height, spp):
    tracer.configure(width, height, SCENES[scene]())
    tracer.set_camera(zoo_camera(width, height))
    for mis in (0, 1):
        tracer.set_params(default_params(max_path_depth=8, min_samples=spp, max_samples_per_pixel=spp, emitter_mis=mis,
                                         background_r=0.4, background_g=0.5, background_b=0.6))
        _same(tracer)
    tracer.set_extend_mode(0)


@pytest.mark.gpu
def test_degenerate_directions(tracer):
    """A field of view so narrow that every camera ray is the axis itself (quirk Q1)."""
    tracer.configure(40, 31, zoo_scene(n_per_mat=100, seed=4))
    cam = look_at_camera((0.3, 0.1, 9.0), (0.3, 0.1, 0.0), fov_y_deg=1.0e-8, aspect=40 / 31)
    cam["orientation"] = (1.0, 0.0, 0.0, 0.0)
    tracer.set_camera(cam)
    tracer.set_params(default_params(max_path_depth=6, min_samples=3, max_samples_per_pixel=3, background_r=0.4,
                                     background_g=0.5, background_b=0.6))
    _same(tracer)
    tracer.set_extend_mode(0)


@pytest.mark.gpu
@pytest.mark.parametrize("instanced", [(0,), (1,), (0, 2)])
def test_batch_of_flat_and_instanced_scenes(tracer, instanced):
    sizes = [(31, 17), (16, 40), (45, 9)]
    mesh = zoo_scene(n_per_mat=60, seed=6)
    tracer.batch_configure(sizes)
    for k, (w, h) in enumerate(sizes):
        if k in instanced:
            place = [(placement(0.2 * j - 0.2, 0.1 * j, 0.7 * j, 0.6 + 0.2 * j), 0) for j in range(3)]
            tracer.set_instances([mesh], place + place[:1], scene=k)  # (the last instance ties with the first)
        else:
            tracer.batch_set_mesh(k, mesh)
        tracer.batch_set_camera(k, zoo_camera(w, h))
    tracer.set_params(default_params(max_path_depth=8, min_samples=4, max_samples_per_pixel=4, background_r=0.4,
                                     background_g=0.5, background_b=0.6))
    _same(tracer)
    tracer.set_extend_mode(0)
