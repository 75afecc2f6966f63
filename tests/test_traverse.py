"""Plane decode of the compressed nodes (csrc/pt_trace.cuh), on the CPU: the decoded near / far plane
parameters bracket the exact ones for node scales, directions and origins over the ranges that a scene can have.
"""
import numpy as np


def test_plane_decode_is_conservative():
    rng = np.random.default_rng(7)
    n = 400_000
    f = np.float32
    scale = np.ldexp(f(1.0), rng.integers(-30, 8, n)).astype(f)
    idir = (np.exp(rng.normal(0.0, 4.0, n)) * rng.choice([-1.0, 1.0], n)).astype(f)
    q = rng.integers(0, 256, n)
    # origins from inside the node to 2^20 of its extents away
    p = rng.normal(0.0, 5.0, n).astype(f)
    o = (p + scale * 256.0 * rng.uniform(-1.0, 1.0, n) * np.exp2(rng.uniform(-4.0, 20.0, n))).astype(f)
    rel = (p - o).astype(f)
    exact = (q * scale.astype(np.float64) + rel) * idir          # the plane's parameter from the rounded p - o
    a = (scale * f(32768.0) * idir).astype(f)
    b = (rel.astype(np.float64) * idir - a).astype(f)            # fma: one rounding
    pad = np.abs(a).astype(np.float64) * 2.0 ** -22
    near, far = (b - pad).astype(f), (b + pad).astype(f)
    plane = (f(1.0) + q.astype(f) * f(2.0 ** -15)).astype(f)
    assert np.array_equal((plane.view(np.uint32) >> 8) & 0xFF, q), "the byte sits in bits 8..15"
    t0 = (plane.astype(np.float64) * a + near).astype(f)
    t1 = (plane.astype(np.float64) * a + far).astype(f)
    slack = np.abs(exact) * 2.0 ** -22                           # half of what the slab test's tExit is widened by
    assert np.all(t0 <= exact + slack) and np.all(t1 >= exact - slack)
    # and the boxes stay tight: within 1/64 of a quantum (plus rounding)
    quantum = np.abs(scale.astype(np.float64) * idir)
    assert np.all(t1.astype(np.float64) - t0 <= quantum / 32.0 + np.abs(exact) * 2.0 ** -21)
