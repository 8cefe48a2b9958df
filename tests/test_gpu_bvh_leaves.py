"""Leaves that the level-by-level phase of the GPU BVH build leaves whole:
triangles no plane separates, in groups of up to many thousands, whose ids
are copied to the leaf order in pieces of 1,024.  The tree must be the
oracle's node for node and the order a permutation."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import scenes
from test_gpu_bvh_build import _canonical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [[129], [1023], [1024], [1025], [2048], [2049], [70001], [3000, 1, 1025, 40, 129, 2048],
                                    [1500] * 9])
def test_groups_of_coincident_triangles(ctx, oracle, groups):
    desc = scenes.triangle_soup(sum(groups), seed=7, extent=5.0, size=0.3)
    p = desc.triangles["v"]["p"]
    at = np.random.default_rng(3).permutation(len(p))  # the groups' members lie apart in the input
    first = 0
    for g in groups:
        p[at[first:first + g]] = p[at[first]]
        first += g
    ctx.upload(desc)
    ctx.bvh_build()
    nodes, idx = ctx.bvh_export()
    o_nodes, o_idx = oracle.bvh_build(desc.triangles)
    assert sorted(idx.tolist()) == list(range(len(p)))
    assert len(nodes) == len(o_nodes)
    assert _canonical(nodes, idx) == _canonical(o_nodes, o_idx)
