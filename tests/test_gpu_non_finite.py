"""A mesh with infinite, NaN or very large coordinates is built, queried and rendered without an error, and leaves
nothing behind.

What such triangles return is not specified (Moller-Trumbore passes NaN through its comparisons, as the reference's
does); what they may not do is damage the tree: the boxes above them are infinite, and the exponent of an infinite box
must still fit the byte that a node has for it.
"""
import numpy as np
import pytest

from lsystemeditor_b200.records import default_params
from tests.helpers import random_soup, rays_through_bounds, zoo_camera

pytestmark = pytest.mark.gpu

BAD = {"inf": [np.inf], "-inf": [-np.inf], "both": [np.inf, -np.inf], "nan": [np.nan],
       "large": [3.0e38, -3.0e38], "mixed": [np.inf, -np.inf, np.nan, 3.0e38]}


@pytest.mark.parametrize("kind", sorted(BAD))
@pytest.mark.parametrize("n, bad", [(1, 1), (9, 1), (64, 5), (900, 40)])
def test_non_finite_triangles(tracer, oracle, kind, n, bad):
    good = random_soup(n, seed=n, extent=1.0, size=0.4)
    mesh = random_soup(n, seed=n, extent=1.0, size=0.4)
    rng = np.random.default_rng(n)
    for k, t in enumerate(rng.permutation(n)[:bad]):
        mesh.positions[t, rng.integers(0, 3), rng.integers(0, 3)] = BAD[kind][k % len(BAD[kind])]
    o, d = rays_through_bounds(good, 3000, seed=n + 1)
    tracer.configure(24, 16, mesh)
    assert tracer.trace_rays(o, d)["tri"].max() < n
    tracer.set_camera(zoo_camera(24, 16))
    tracer.set_params(default_params(max_path_depth=4, min_samples=2, max_samples_per_pixel=2, background_r=0.4,
                                     background_g=0.5, background_b=0.6))
    for mode in (1, 2):
        tracer.set_extend_mode(mode)
        tracer.reset_accumulation()
        tracer.render(0)
        assert np.isfinite(tracer.readback()[0]).all()
    tracer.set_extend_mode(0)
    tracer.set_mesh(good)
    g, r = tracer.trace_rays(o, d), oracle.scene(good).trace_bruteforce(o, d)
    assert np.array_equal(g["hit"], r["hit"]) and np.array_equal(g["tri"][g["hit"]], r["tri"][r["hit"]])
