"""The GPU BVH build at the sizes where it changes hands: subtrees finished
by one warp (up to 128 triangles), one chunk and several chunks of the
level-by-level phase (2,048 triangles each), leaves of any size (coincident
centroids, which no plane splits) and uneven splits (triangle sizes over six
decades).  The tree must be the oracle's node for node."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import scenes

pytestmark = pytest.mark.gpu


def _canonical(nodes, idx):
    """Sorted (kind, first box bytes, triangle set) of every node."""
    out, stack = [], [(0, 0)]
    sets = {}
    while stack:
        i, done = stack.pop()
        n = nodes[i]
        if n["used"] > 0:
            sets[i] = tuple(sorted(idx[n["left_first"]:n["left_first"] + n["used"]].tolist()))
        elif not done:
            stack += [(i, 1), (int(n["left_first"]), 0), (int(n["left_first"]) + 1, 0)]
            continue
        else:
            sets[i] = tuple(sorted(sets[int(n["left_first"])] + sets[int(n["left_first"]) + 1]))
        out.append((bool(n["used"] > 0), (n["bmin"] + 0.0).tobytes() + (n["bmax"] + 0.0).tobytes(), sets[i]))
    return sorted(out)


def _soup(n, kind):
    desc = scenes.triangle_soup(n, seed=n, extent=5.0, size=0.3)
    rng = np.random.default_rng(n + 1)
    p = desc.triangles["v"]["p"]
    if kind == "coincident":      # half of the triangles are copies of one
        p[: n // 2] = p[0]
    elif kind == "scales":        # clusters inside clusters
        p *= (10.0 ** rng.uniform(-6, 0, n)).astype(np.float32)[:, None, None]
    elif kind == "flat":          # one axis has no extent
        p[..., 1] = 0.25
    return desc


@pytest.mark.parametrize("kind", ["soup", "coincident", "scales", "flat"])
@pytest.mark.parametrize("n", [1, 4, 5, 31, 33, 127, 128, 129, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 9001])
def test_build_matches_oracle_at_limits(ctx, oracle, n, kind):
    desc = _soup(n, kind)
    ctx.upload(desc)
    ctx.bvh_build()
    nodes, idx = ctx.bvh_export()
    o_nodes, o_idx = oracle.bvh_build(desc.triangles)
    assert sorted(idx.tolist()) == list(range(n))
    assert len(nodes) == len(o_nodes)
    assert _canonical(nodes, idx) == _canonical(o_nodes, o_idx)
