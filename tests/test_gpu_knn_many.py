"""Nearest records of many queries at once (a thread per query) against the
same queries in small calls (a warp per query): the same tree walk and the
same comparisons, so the indexes and distances are equal bit for bit, ties
and lists that stay short included."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 40, 5000])
@pytest.mark.parametrize("k", [1, 7, 8, 16, 17])
def test_many_queries_equal_few(ctx, n, k):
    rng = np.random.default_rng(n + k)
    recs = np.zeros(n, abi.PATH_VERTEX)
    recs["position"] = rng.uniform(-2, 2, (n, 3)).round(1)  # coarse: many equal distances
    recs["normal"] = recs["wi"] = (0, 0, 1)
    recs["Li"] = 1.0
    ctx.upload(scenes.cornell_box(seed=1, width=8, height=8))
    ctx.cache_build(recs)
    limit = 16384 + 6144 * k
    q = rng.uniform(-2.5, 2.5, (limit + 1, 3)).astype(np.float32)
    q[::3] = q[::3].round(1)
    q[5] = 1e20  # squared distances overflow: nothing is found
    pieces = [ctx.cache_knn(q[i:i + 16000], k) for i in range(0, len(q), 16000)]
    want_i, want_d = (np.concatenate([p[j] for p in pieces]) for j in (0, 1))
    finite = np.arange(len(q)) != 5
    assert (want_i[finite, min(n, k) - 1] >= 0).all() and (want_i[:, n:] == -1).all() and (want_i[5] == -1).all()
    assert np.isinf(want_d[5]).all() and np.isinf(want_d[:, n:]).all()
    for m in (limit - 1, limit, limit + 1):
        idx, d2 = ctx.cache_knn(q[:m], k)
        np.testing.assert_array_equal(idx, want_i[:m])
        np.testing.assert_array_equal(d2, want_d[:m])
