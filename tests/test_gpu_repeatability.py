"""A render repeats bit for bit where hits lie closer together than the box test is exact.

Overlapping rectangles in one plane: every ray that meets them has several hits within a few ulps of each other, and
which of them a box culls depends on the order of its tests.  That order may not depend on which parts of a ray idle
lanes have taken over (csrc/pt_traverse.cuh), which differs from run to run; so images that repeat are the whole test,
without a tolerance.
"""
import numpy as np
import pytest

from lsystemeditor_b200.records import MATERIAL_DTYPE, TEXTURE_DTYPE, default_material, default_params, look_at_camera
from lsystemeditor_b200.scene import HostMesh
from tests.helpers import random_soup

pytestmark = pytest.mark.gpu


def _coplanar(n, rng, size, offset):
    """n axis-aligned rectangles in the planes at +-offset and +-2 offset of the three axes."""
    pos = np.zeros((2 * n, 3, 3), np.float32)
    nrm = np.zeros_like(pos)
    for i in range(n):
        axis = int(rng.integers(0, 3))
        others = [k for k in range(3) if k != axis]
        corner = np.zeros((4, 3))
        corner[:, axis] = offset * (1 + int(rng.integers(0, 2))) * (-1 if axis == 1 else 1)
        centre, half = rng.uniform(-size, size, 2), rng.uniform(0.02 * size, 0.5 * size, 2)
        for k, signs in enumerate(((-1, -1), (1, -1), (1, 1), (-1, 1))):
            corner[k, others] = centre + np.array(signs) * half
        pos[2 * i], pos[2 * i + 1] = corner[[0, 1, 2]], corner[[0, 2, 3]]
        nrm[2 * i:2 * i + 2, :, axis] = 1.0
    mats = np.array([default_material(r=rng.uniform(0.1, 0.9), g=rng.uniform(0.1, 0.9), b=rng.uniform(0.1, 0.9),
                                      roughness=rng.uniform(0.05, 1.0)) for _ in range(16)], MATERIAL_DTYPE)
    return HostMesh(pos, nrm, rng.uniform(0, 1, (2 * n, 3, 2)).astype(np.float32),
                    rng.integers(0, 16, 2 * n).astype(np.uint32), mats, np.zeros(0, TEXTURE_DTYPE))


@pytest.mark.parametrize("seed, n, size, offset, height, w, h", [
    (1, 2000, 100.0, 10.0, 0.01, 256, 160), (2, 300, 10.0, 1.0, 0.01, 256, 160), (3, 2000, 100.0, 10.0, 0.1, 64, 48),
    (4, 40, 1000.0, 100.0, 1.0, 64, 48), (5, 2000, 1000.0, 1.0, 0.001, 64, 48), (6, 2000, 10.0, 1.0, 0.5, 33, 1)])
def test_coplanar_rectangles_render_the_same_every_time(tracer, seed, n, size, offset, height, w, h):
    rng = np.random.default_rng(seed)
    soup = random_soup(3000, seed=seed, extent=2.0 * size, size=0.05 * size, materials=2)
    tracer.configure(w, h, HostMesh.concat([_coplanar(n, rng, size, offset), soup]))
    tracer.set_camera(look_at_camera((0.37 * offset, height - offset, 0.21 * offset),
                                     (0.3 * size, -offset - 0.2 * height, 0.4 * size), fov_y_deg=70.0, aspect=w / h))
    tracer.set_params(default_params(max_path_depth=8, min_samples=16, max_samples_per_pixel=16, background_r=0.4,
                                     background_g=0.5, background_b=0.6))
    first = None
    for _ in range(6):
        tracer.reset_accumulation()
        tracer.render(0)
        image = tracer.readback()[0].copy()
        if first is None:
            first = image
            assert image[..., :3].max() > 0
        assert np.array_equal(image, first)
