"""Traversal of the rays the packed slab test does not cover and of batch
sizes around the warp: axis-parallel directions (an infinite inverse in one or
two components, also negative zeros), origins on slab planes (0 x inf), a
finite tmax, and 1 to 4,097 rays.  Hits, visibility and visit counts must be
the oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _rays(n, kind):
    rng = np.random.default_rng(n)
    r = np.zeros(n, abi.RAY)
    r["o"] = rng.uniform((-0.9, 0.1, -0.9), (0.9, 1.9, 3.0), (n, 3))
    d = rng.normal(size=(n, 3))
    if kind != "general":
        axis = rng.integers(0, 3, n)
        for k in range(3):
            zero = axis == k if kind == "two" else axis != k
            d[zero, k] = np.where(rng.random(zero.sum()) < 0.5, 0.0, -0.0)
    if kind == "planes":       # origins exactly on walls, box faces and tessellation lines
        r["o"] = np.round(r["o"] * 4.0) / 4.0
        r["o"][: n // 2, 1] = 0.0
    r["d"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["tmax"] = np.where(rng.random(n) < 0.5, np.finfo(np.float32).max, 1.5)
    return r


@pytest.mark.parametrize("kind", ["general", "one", "two", "planes"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 129, 4097])
def test_rays_match_oracle(ctx, oracle, n, kind):
    desc = scenes.cornell_box(seed=2, target_tris=3000)
    nodes, idx = oracle.bvh_build(desc.triangles)
    ctx.upload(desc)
    ctx.bvh_import(nodes, idx)
    rays = _rays(n, kind)
    hits, visits, tests = oracle.trace_closest(desc.triangles, nodes, idx, rays)
    assert ctx.trace_closest(rays).tobytes() == hits.tobytes()
    assert ctx.trace_counters() == (visits, tests)
    vis, visits, tests = oracle.trace_any(desc.triangles, nodes, idx, rays)
    assert np.array_equal(ctx.trace_any(rays), vis)
    assert ctx.trace_counters() == (visits, tests)
