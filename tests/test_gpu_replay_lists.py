"""Previews of every level and gradients that are not zero, where their lists begin and end.

* Every level of previews rendered together equals the finest level of a renderer that has that level as its last (same
  seed, same size), bit for bit; the levels around the sixteenth, where a second launch takes over, also match the
  oracle's preview on the same random numbers (relative RMSE 1e-3, as for whole images).
* The gradient of sparse image gradients at pixels that see the scene, listed from the sample record, equals the replayed one:
  the same terms in another order, 1e-3 of the largest entry.
"""
import numpy as np
import pytest

from lsystemeditor_b200.pathtracer import PathTracer
from lsystemeditor_b200.records import default_params
from tests.helpers import rel_rmse, zoo_camera, zoo_scene
from tests.test_gpu_adjoint import _render, _setup

pytestmark = pytest.mark.gpu


def _previews(t, width, height, levels, mesh, camera):
    t.configure(width, height, mesh)
    t.set_camera(camera)
    t.set_params(default_params(background_r=0.2, background_g=0.3, background_b=0.4))
    t.set_preview_steps_per_level(levels)
    t.render_previews()
    out = [t.preview(k) for k in range(levels)]
    t.set_preview_steps_per_level(0)
    return out


@pytest.mark.parametrize("w, h, levels", [(65, 33, 4), (7, 3, 3), (128, 96, 5), (40, 24, 18)])
def test_every_level_equals_the_finest_of_its_own_renderer(tracer, w, h, levels):
    mesh, camera = zoo_scene(n_per_mat=40, seed=2), zoo_camera(w, h)
    together = _previews(tracer, w, h, levels, mesh, camera)
    with PathTracer(0) as alone:
        for k, img in enumerate(together):
            ph, pw = img.shape[:2]
            assert (img[..., 3] == 1.0).all()
            assert np.array_equal(_previews(alone, 2 * pw, 2 * ph, k + 1, mesh, camera)[k], img), k


def test_levels_of_the_second_launch_match_the_oracle(tracer, oracle):
    w, h, n, stride = 96, 80, 18, 80
    mesh, camera = zoo_scene(n_per_mat=120, seed=5), zoo_camera(w, h)
    images = _previews(tracer, w, h, n, mesh, camera)
    params = default_params(background_r=0.2, background_g=0.3, background_b=0.4, max_path_depth=4)
    scene = oracle.scene(mesh)
    for k in (15, 16, 17):
        ph, pw = images[k].shape[:2]
        assert (ph, pw) == (h >> (n - k), w >> (n - k))
        with PathTracer(0) as t:
            t.configure(pw, ph, mesh)
            t.set_preview_steps_per_level(k)
            tape = t.rng_tape(0, 1, stride)[0]
        ref, err = scene.render_preview(camera, params, pw, ph, tape, stride)
        assert err == 0
        e = rel_rmse(images[k][..., :3], ref[..., :3])
        assert np.all(e <= 1e-3), (k, e)


@pytest.mark.parametrize("keep", [1, 31, 33, 100])
@pytest.mark.parametrize("w, h, spp", [(31, 31, 3), (33, 29, 2), (61, 47, 3)])
def test_sparse_gradients_of_pixels_that_see_the_tree(tracer, w, h, spp, keep):
    spec, _ = _setup(tracer, w, h, spp)
    tracer.record_samples(0)
    image = _render(tracer, spec.mesh.materials, spp)
    rng = np.random.default_rng(w + h + keep)
    d_image = np.zeros((h, w, 3), np.float32)
    seen = np.argwhere((np.abs(image - 0.4) > 1e-3).any(-1))  # (the sky is a grey 0.4)
    assert len(seen) >= 20
    for y, x in seen[rng.permutation(len(seen))[:keep]]:
        d_image[y, x] = rng.uniform(0.5, 1.5, 3)
    full, _ = tracer.backward(d_image, spp)
    tracer.record_samples(spp)
    _render(tracer, spec.mesh.materials, spp)
    listed, _ = tracer.backward(d_image, spp)
    tracer.record_samples(0)
    assert np.isfinite(full).all() and np.abs(full).max() > 0
    assert np.abs(listed - full).max() <= 1e-3 * np.abs(full).max()
