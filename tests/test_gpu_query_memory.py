"""What a ray query keeps of the device's memory."""
import pytest

from lsystemeditor_b200.pathtracer import PathTracer
from tests.helpers import random_soup, rays_through_bounds

pytestmark = pytest.mark.gpu

KEPT = 128 << 20   # a query's buffer, 76 bytes per ray, is kept up to this size
GRAIN = 4 << 20    # cudaMalloc's granularity


@pytest.mark.parametrize("n, kept", [(1000, True), (1_700_000, True), (1_800_000, False), (3_000_000, False)])
def test_memory_kept_by_a_query(n, kept):
    import torch
    mesh = random_soup(500, seed=1)
    with PathTracer(0) as t:
        t.configure(8, 8, mesh)
        o, d = rays_through_bounds(mesh, n, seed=2)
        t.trace_rays(o[:10], d[:10])
        before = torch.cuda.mem_get_info()[0]
        for _ in range(2):
            assert t.trace_rays(o, d)["hit"].any()
        held = before - torch.cuda.mem_get_info()[0]
    assert held <= (min(76 * n, KEPT) + GRAIN if kept else GRAIN)
