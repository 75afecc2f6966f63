"""Staged uploads and downloads (csrc/pt_hostcopy.cuh) at the sizes where they begin and end, on the GPU.

Everything runs in one process of its own, whose copier is made ready first: whether it is, its three threads show.
What comes back must be what went in, bit for bit; a query's answer must be that of the same rays in small parts.
"""
import multiprocessing
import os
import threading
import traceback
from concurrent.futures import ProcessPoolExecutor

import numpy as np
import pytest

from lsystemeditor_b200.pathtracer import PathTracer, PathTracerError
from lsystemeditor_b200.scene import HostMesh
from tests.helpers import random_soup, rays_through_bounds, zoo_scene

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _threads() -> int:
    return len(os.listdir("/proc/self/task"))


def _soup(n, seed):
    return random_soup(n, seed=seed, extent=30.0, size=0.2, materials=3)


def _same(mesh, back):
    for name in ("positions", "normals", "uvs", "material_ids"):
        assert np.array_equal(getattr(back, name), getattr(mesh, name)), name


_held = []  # the renderer that keeps the process's copier


def _make_ready() -> int:
    """Queries until 96 MB went plainly and one transfer was staged; the number of threads that appeared."""
    t = PathTracer(0)
    _held.append(t)
    mesh = zoo_scene(n_per_mat=30, seed=5)
    t.configure(8, 8, mesh)
    o, d = rays_through_bounds(mesh, 1_000_000, seed=1)
    t.trace_rays(o[:1000], d[:1000])
    before = _threads()
    for _ in range(3):  # (32 MB in, 29 MB out)
        t.trace_rays(o, d)
    return _threads() - before


def _queries(n):
    mesh = zoo_scene(n_per_mat=30, seed=5)
    o, d = rays_through_bounds(mesh, n, seed=7)
    with PathTracer(0) as t:
        t.configure(8, 8, mesh)
        whole = t.trace_rays(o, d)
        parts = [t.trace_rays(o[a:a + 60_000], d[a:a + 60_000]) for a in range(0, n, 60_000)]
    assert whole["hit"].any()
    for k, v in whole.items():
        assert np.array_equal(v, np.concatenate([p[k] for p in parts])), k


def _mesh(n, caller_stream, pinned):
    import torch
    mesh = _soup(n, seed=2)
    if pinned:
        arrays = [torch.from_numpy(a.view(np.int32)).pin_memory() for a in
                  (mesh.positions, mesh.normals, mesh.uvs, mesh.material_ids)]
        mesh = HostMesh(*[a.numpy().view(np.float32) for a in arrays[:3]], arrays[3].numpy().view(np.uint32),
                        mesh.materials, mesh.textures)
    with PathTracer(0) as t:
        t.configure(8, 8)
        stream = torch.cuda.Stream()
        if caller_stream:
            t.set_stream(stream.cuda_stream)
        for _ in range(2):
            t.set_mesh(mesh)
            _same(mesh, t.export_mesh())
        o, d = rays_through_bounds(mesh, 2000, seed=3)
        hits = t.trace_rays(o, d)
        t.set_stream(None)
    small = HostMesh(mesh.positions.copy(), mesh.normals.copy(), mesh.uvs.copy(), mesh.material_ids.copy(),
                     mesh.materials, mesh.textures)
    _held[0].set_mesh(small)
    again = _held[0].trace_rays(o, d)
    for k in hits:
        assert np.array_equal(hits[k], again[k]), k


def _two_at_once():
    meshes = [_soup(700_000 + 3 * k, seed=k) for k in range(3)]
    errors = []

    def work(mesh, k):
        try:
            with PathTracer(0) as t:
                t.configure(8, 8)
                o, d = rays_through_bounds(mesh, 450_000 + k, seed=k)
                first = None
                for _ in range(3):
                    t.set_mesh(mesh)
                    _same(mesh, t.export_mesh())
                    r = t.trace_rays(o, d)
                    first = first or r
                    for name in r:
                        assert np.array_equal(r[name], first[name]), name
        except BaseException as e:  # (a thread's own failure does not reach the test)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(m, k)) for k, m in enumerate(meshes)]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not errors, errors


def _failing_build():
    """The build runs out of device memory while the normals and uvs are on their way: the call ends with the error,
    and the next one is as if nothing had been."""
    import torch
    mesh = _soup(900_001, seed=4)
    with PathTracer(0) as t:
        t.configure(8, 8)
        torch.cuda.synchronize()
        hold = []
        for step in (1 << 30, 64 * MB, 4 * MB):  # leave room for the mesh's arrays (90 MB), not for its records
            while torch.cuda.mem_get_info()[0] - step > 112 * MB:
                hold.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        with pytest.raises(PathTracerError, match="OUT_OF_MEMORY"):
            t.set_mesh(mesh)
        hold.clear()
        torch.cuda.empty_cache()
        t.set_mesh(mesh)
        _same(mesh, t.export_mesh())


def _run(f, *a):
    """What went wrong in f(*a), as text."""
    try:
        f(*a)
    except Exception:
        return traceback.format_exc()
    return None


def _report(failure):
    assert failure is None, failure


@pytest.fixture(scope="module")
def staging():
    """A process whose copier stages."""
    if (os.cpu_count() or 1) <= 4:
        pytest.skip("staging needs more than four processors")
    with ProcessPoolExecutor(1, mp_context=multiprocessing.get_context("spawn")) as pool:
        assert pool.submit(_make_ready).result(300) == 3, "the copier's threads were not made"
        yield lambda f, *a: _report(pool.submit(_run, f, *a).result(300))


# 32 bytes in and 29 out per ray: 12 MB in, and 12 MB out, with a last slice of a few bytes
@pytest.mark.parametrize("n", [393_215, 393_216, 393_217, 433_895, 600_001])
def test_queries(staging, n):
    staging(_queries, n)


# 40 and 60 bytes per triangle: the second pair of arrays, then the first is staged, then the second goes beside the build
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("caller_stream", [False, True])
@pytest.mark.parametrize("n", [209_716, 314_573, 559_241, 900_001])
def test_mesh(staging, n, caller_stream, pinned):
    staging(_mesh, n, caller_stream, pinned)


def test_renderers_of_several_threads(staging):
    staging(_two_at_once)


def test_build_that_fails_during_the_upload(staging):
    staging(_failing_build)
