"""The radiance cache's tree at the sizes where its build changes hands:
one leaf, one shared-memory subtree (up to 2,048 records), the level-by-level
phase in front of it, and regions above and below the subtree size.  Checked
against the definition alone: every node's bounds are its records', a node
of more than 8 records splits on its longest axis with the used/2 smallest
coordinates on the left, and every record is in exactly one leaf."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi

pytestmark = pytest.mark.gpu


def _records(n, seed, ties):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, abi.PATH_VERTEX)
    r["position"] = rng.normal(size=(n, 3)) * (3.0, 1.0, 2.0)
    if ties:
        r["position"][: n // 2] = np.round(r["position"][: n // 2])
    r["normal"] = (0, 1, 0)
    d = rng.normal(size=(n, 3))
    r["wi"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["Li"] = rng.uniform(0.1, 1.0, (n, 3))
    r["Li"][:, 0] = np.arange(n)
    return r


@pytest.mark.parametrize("region", [256, 1024, 16384])
@pytest.mark.parametrize("n,ties", [(1, 0), (8, 0), (9, 0), (16, 0), (17, 1), (255, 0), (1025, 1), (2047, 0), (2048, 0),
                                    (2049, 0), (4096, 1), (4099, 0), (33333, 1)])
def test_tree_at_build_limits(ctx, n, ties, region):
    ctx.guide_configure(region_records=region)
    recs = _records(n, n, ties)
    ctx.cache_build(recs)
    nodes, out = ctx.cache_export()
    assert np.array_equal(np.sort(out["Li"][:, 0]), np.arange(n))
    assert np.array_equal(out["position"], recs["position"][out["Li"][:, 0].astype(np.int64)])
    regions, _, _ = ctx.guide_export()
    want_regions = []
    seen = 0
    stack = [(0, 0, n, True)]
    while stack:
        i, first, used, above = stack.pop()
        nd, p = nodes[i], out["position"][first:first + used]
        seen += 1
        np.testing.assert_array_equal(nd["bmin"], p.min(axis=0))
        np.testing.assert_array_equal(nd["bmax"], p.max(axis=0))
        if above and used <= region:
            want_regions.append((first, used, i))
            above = False
        if used <= 8:
            assert (nd["left"], nd["right"], nd["offset"], nd["used"]) == (-1, -1, first, used)
            continue
        assert nd["used"] == 0
        axis = int(np.argmax((nd["bmax"] - nd["bmin"]).astype(np.float32)))  # ties to the lower axis
        assert p[:used // 2, axis].max() <= p[used // 2:, axis].min()
        stack.append((int(nd["left"]), first, used // 2, above))
        stack.append((int(nd["right"]), first + used // 2, used - used // 2, above))
    assert seen == len(nodes)
    assert sorted((int(r["first"]), int(r["count"]), int(r["node"])) for r in regions) == sorted(want_regions)


@pytest.mark.parametrize("n,k", [(1, 1), (5, 8), (9, 31), (300, 32), (300, 33), (40, 64), (5000, 1), (5000, 64)])
def test_knn_at_list_ends(ctx, n, k):
    """Lists of one, a full warp, one more, and longer than the cache; equal
    distances (duplicated records) keep the lower index first.  The distance
    is the float32 expression of the brute force."""
    recs = _records(n, n + k, ties=True)
    recs["position"][n // 2:] = recs["position"][: n - n // 2]
    ctx.cache_build(recs)
    _, out = ctx.cache_export()
    rng = np.random.default_rng(k)
    q = np.concatenate([out["position"][rng.integers(0, n, 40)], rng.normal(size=(60, 3)) * 3]).astype(np.float32)
    idx, d2 = ctx.cache_knn(q, k)
    d = out["position"][None, :, :] - q[:, None, :]
    ref = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
    order = np.argsort(ref, axis=1, kind="stable")[:, :k]
    m = min(n, k)
    assert np.array_equal(idx[:, :m], order[:, :m])
    assert np.array_equal(d2[:, :m], np.take_along_axis(ref, order[:, :m], 1))
    assert np.all(idx[:, m:] == -1) and np.all(np.isinf(d2[:, m:]))
