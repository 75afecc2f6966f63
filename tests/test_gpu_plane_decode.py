"""The kernels' decode of the quantised child planes, through the hits.

Triangles in axis-aligned planes have boxes without thickness: a near plane decoded above, or a far plane below its
value puts the entry behind the exit and the triangle is never tested.  With whole coordinates a box's planes lie
exactly on the quantised ones, with no room to spare, and coordinates up to 255 in nodes of all sizes reach every value
of a plane byte.  Every hit must be the brute-force one.  (Triangles that overlap in one plane are not for this test:
of two hits closer together than the box test is exact a ray may return either.)
"""
import numpy as np
import pytest

from lsystemeditor_b200.pathtracer import PathTracer
from lsystemeditor_b200.records import MATERIAL_DTYPE, TEXTURE_DTYPE, default_material, default_params, look_at_camera
from lsystemeditor_b200.scene import HostMesh

pytestmark = pytest.mark.gpu


def _flat(n, rng, span, axis):
    """n triangles in planes perpendicular to the axis, every coordinate a whole number."""
    pos = rng.integers(0, span + 1, (n, 3, 3)).astype(np.float32)
    pos[:, :, axis] = rng.integers(0, span + 1, (n, 1))
    a, b = (axis + 1) % 3, (axis + 2) % 3
    pos[:, 1, a] = pos[:, 0, a] + rng.integers(1, 6, n)  # a right angle at the first corner: none is a line
    pos[:, 1, b] = pos[:, 0, b]
    pos[:, 2, b] = pos[:, 0, b] + rng.integers(1, 6, n)
    pos[:, 2, a] = pos[:, 0, a]
    nrm = np.zeros_like(pos)
    nrm[..., axis] = 1.0
    return HostMesh(pos, nrm, np.zeros((n, 3, 2), np.float32), np.zeros(n, np.uint32),
                    np.array([default_material()], MATERIAL_DTYPE), np.zeros(0, TEXTURE_DTYPE))


@pytest.mark.parametrize("n", [8, 300, 3000])
def test_flat_boxes_are_hit(tracer, oracle, n):
    span = 255
    rng = np.random.default_rng(span + n)
    mesh = HostMesh.concat([_flat(n, rng, span, axis) for axis in range(3)])
    tracer.configure(8, 8, mesh)
    pick = rng.integers(0, 3 * n, 20_000)
    weights = rng.uniform(0.1, 1.0, (20_000, 3))
    target = ((weights / weights.sum(1, keepdims=True))[..., None] * mesh.positions[pick]).sum(1)
    origins = rng.uniform(-0.5 * span, 1.5 * span, (20_000, 3)).astype(np.float32)
    dirs = (target - origins).astype(np.float32)
    g = tracer.trace_rays(origins, dirs)
    r = oracle.scene(mesh).trace_bruteforce(origins, dirs)
    assert r["hit"].mean() > 0.99
    for k in ("hit", "tri", "t"):
        assert np.array_equal(g[k], r[k]), k


def test_whole_warp_kernels_see_flat_boxes(tracer):
    """The same boxes in the render kernels: one white triangle wall of 256 x 1 strips in planes x = 0 .. 255, lit by
    nothing but a white background, shows no strip missing: a camera ray that meets a strip takes the strip's colour."""
    n = 256
    pos = np.zeros((2 * n, 3, 3), np.float32)
    for q in range(n):
        corners = np.array([[q, q, 0], [q, q + 1, 0], [q, q + 1, 16], [q, q, 16]], np.float32)
        pos[2 * q], pos[2 * q + 1] = corners[[0, 1, 2]], corners[[0, 2, 3]]
    nrm = np.zeros_like(pos)
    nrm[..., 0] = -1.0
    mesh = HostMesh(pos, nrm, np.zeros((2 * n, 3, 2), np.float32), np.zeros(2 * n, np.uint32),
                    np.array([default_material(r=0.0, g=0.0, b=0.0, specular=0.0, emission=0.0)], MATERIAL_DTYPE),
                    np.zeros(0, TEXTURE_DTYPE))
    w, h = 64, 512
    tracer.configure(w, h, mesh)
    tracer.set_camera(look_at_camera((-40.0, 128.0, 8.0), (0.0, 128.0, 8.0), fov_y_deg=30.0, aspect=w / h))
    tracer.set_params(default_params(max_path_depth=1, min_samples=4, max_samples_per_pixel=4, background_r=1.0,
                                     background_g=1.0, background_b=1.0))
    out = []
    for mode in (1, 2):
        tracer.set_extend_mode(mode)
        tracer.reset_accumulation()
        tracer.render(0)
        out.append(tracer.readback()[0].copy())
    tracer.set_extend_mode(0)
    assert np.array_equal(out[0], out[1])
    # the middle of the wall fills the middle rows: no ray gets through to the background's full white
    with PathTracer(0) as t:
        t.configure(8, 8, mesh)
        y = np.linspace(100.0, 156.0, 4001, dtype=np.float32)
        o = np.broadcast_to(np.array([-40.0, 0.0, 8.5], np.float32), (4001, 3)).copy()
        o[:, 1] = y
        d = np.broadcast_to(np.array([1.0, 1.0e-3, 1.0e-3], np.float32), (4001, 3)).copy()
        assert t.trace_rays(o, d)["hit"].all()
