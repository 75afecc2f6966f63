"""What a ray query keeps of the device's memory, and the error of one that cannot have any."""
import multiprocessing
import threading
from concurrent.futures import ProcessPoolExecutor

import pytest

from lsystemeditor_b200.pathtracer import PathTracer, PathTracerError
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


def _query_while_another_thread_captures():
    import torch
    mesh = random_soup(500, seed=1)
    x = torch.zeros(16, device="cuda")
    t = PathTracer(0)
    t.configure(8, 8, mesh)
    o, d = rays_through_bounds(mesh, 1000, seed=2)
    t.trace_rays(o[:10], d[:10])
    said = []

    def query():
        try:
            t.trace_rays(o, d)
            said.append("traced")
        except PathTracerError as e:
            said.append(str(e))

    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode="global"):
            x + 1
            thread = threading.Thread(target=query)
            thread.start()
            thread.join()
    except Exception:
        pass  # (the refused call ends the capture)
    torch.cuda.synchronize()
    t.trace_rays(o, d)
    return said[0]


def test_refused_allocation_is_not_called_out_of_memory():
    """While another thread captures a graph in global mode no device memory can be had: a CUDA error, not a lack of
    memory, and the next query works."""
    with ProcessPoolExecutor(1, mp_context=multiprocessing.get_context("spawn")) as pool:
        said = pool.submit(_query_while_another_thread_captures).result(300)
    assert "PT_ERR_CUDA" in said and "captur" in said
