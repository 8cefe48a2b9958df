"""QuadTrees at refinements that make levels wider than the build's block.

A level holds up to 1 / refine_fraction cells.  Regions of up to 2,048
records are built by 128 threads, so below 1 / 128 a level can hold more
cells than threads; up to the budget of 256 cells a level reaches 171.
Trees must equal the oracle's node for node (children identical, flux within
1e-5 relative: float32 weights summed with compensation against float64)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import guide_oracle as go
from pathguidingdissertation_gb300 import abi, scenes
from test_gpu_guide_oracle import _compare_trees

pytestmark = pytest.mark.gpu


def _even_records(n, seed):
    """n records in random places, directions uniform over the sphere (and so
    over the trees' (u, v) square), nearly equal Li."""
    rng = np.random.default_rng(seed)
    r = np.zeros(n, abi.PATH_VERTEX)
    r["position"] = rng.uniform(-2, 2, (n, 3))
    r["normal"] = (0, 0, 1)
    u = rng.random((n, 2))
    z = 2.0 * u[:, 0] - 1.0
    phi = 2.0 * np.pi * u[:, 1] - np.pi
    s = np.sqrt(np.maximum(0.0, 1.0 - z * z))
    r["wi"] = np.stack([s * np.cos(phi), s * np.sin(phi), z], 1)
    r["Li"] = rng.uniform(0.9, 1.1, (n, 3))
    return r


def _widest_level(tree):
    depth = [0] * len(tree)
    for i, (_, child) in enumerate(tree):
        for c in child:
            if c >= 0:
                depth[c] = depth[i] + 1
    return int(np.bincount(depth).max())


# (region_records, refinement share, records, threads of the build)
CASES = [(1024, 0.003, 8192, 128), (2048, 0.002, 8192, 128), (600, 0.001, 4800, 128), (1024, 1e-6, 8192, 128),
         (2048, 1.0, 8192, 128), (2049, 0.002, 8196, 512), (4096, 0.0005, 8192, 512)]


@pytest.mark.parametrize("compensate", [0.0, 0.5])
@pytest.mark.parametrize("region_records,refine,n,threads", CASES)
def test_fine_refinement_matches_oracle(ctx, region_records, refine, n, threads, compensate):
    ctx.upload(scenes.cornell_box(seed=1, width=8, height=8))
    ctx.guide_configure(region_records=region_records, refine_fraction=refine, compensate=compensate)
    ctx.cache_build(_even_records(n, 11))
    nodes, out = ctx.cache_export()
    regions, qnodes, _ = ctx.guide_export()
    g = go.Guide(nodes, out, region_max=region_records, rho=refine, compensate=compensate)
    assert len(g.regions) >= 2
    if refine < 1.0:
        assert max(_widest_level(t) for t in g.trees) > 128
    _compare_trees(regions, qnodes, g, atol_rel=1e-6 if compensate else 0.0)
