"""A scene that does not fit is refused, and the next call on the same renderer is as if nothing had been."""
import numpy as np
import pytest

from lsystemeditor_b200.pathtracer import PathTracer, PathTracerError
from tests.helpers import random_soup, rays_through_bounds

pytestmark = pytest.mark.gpu

MB = 1 << 20


# room for the mesh's arrays (90 MB) but not its shading records; for those, but not the build's scratch memory
@pytest.mark.parametrize("room", [112, 230])
def test_mesh_that_does_not_fit(room):
    import torch
    mesh = random_soup(900_001, seed=4, extent=30.0, size=0.2, materials=3)
    o, d = rays_through_bounds(mesh, 2000, seed=3)
    with PathTracer(0) as t, PathTracer(0) as other:
        t.configure(8, 8)
        other.configure(8, 8, mesh)
        torch.cuda.synchronize()
        hold = []
        for step in (1 << 30, 64 * MB, 4 * MB):
            while torch.cuda.mem_get_info()[0] - step > room * MB:
                hold.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        with pytest.raises(PathTracerError, match="OUT_OF_MEMORY"):
            t.set_mesh(mesh)
        hold.clear()
        torch.cuda.empty_cache()
        t.set_mesh(mesh)
        a, b = t.trace_rays(o, d), other.trace_rays(o, d)
    assert a["hit"].any()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
