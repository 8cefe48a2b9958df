"""Small waves run in one launch (a thread per path), larger ones and renders
with stage times on the wavefront kernels.  Both must trace the same paths:
equal ray counts, and films that differ only by the order of the float32
sums (at most 16 samples a pixel here: a relative bound of 16 roundings,
16 x 2^-24 < 1e-6 of the pixel's sum of magnitudes)."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [abi.MODE_PLAIN, abi.MODE_GUIDED_LI, abi.MODE_GUIDED_QUADTREE, abi.MODE_GUIDED_PSS])
@pytest.mark.parametrize("size,spp", [((1, 1), 3), ((7, 5), 1), ((64, 64), 16), ((255, 257), 1), ((256, 257), 1)])
def test_small_wave_matches_wavefront(ctx, mode, size, spp):
    desc = scenes.material_zoo(seed=3, width=size[0], height=size[1], env=True)
    ctx.upload(desc)
    ctx.bvh_build()
    if mode in (abi.MODE_GUIDED_QUADTREE, abi.MODE_GUIDED_PSS):
        train = abi.MODE_PLAIN if mode == abi.MODE_GUIDED_QUADTREE else mode
        ctx.clear()
        ctx.render(8, mode=train, seed=2, max_depth=6, record_paths=8)
    films, counts = [], []
    for timing in (False, True):
        ctx.clear()
        ctx.render(spp, mode=mode, seed=5, max_depth=6, timing=timing)
        films.append(ctx.film(squares=True)[:2])
        st = ctx.render_stats()
        counts.append((st.extension_rays, st.shadow_rays, st.paths))
    assert counts[0] == counts[1] and counts[0][0] >= spp * size[0] * size[1]
    for a, b in zip(*films):
        np.testing.assert_allclose(a, b, rtol=2e-6, atol=0)


def test_small_wave_records_the_same_vertices(ctx):
    """The records of a small training render are those of the wavefront (as
    sets: their order is the order of arrival)."""
    ctx.upload(scenes.cornell_box(seed=1, width=48, height=40))
    ctx.bvh_build()
    got = []
    for timing in (False, True):
        ctx.clear()
        ctx.render(4, mode=abi.MODE_PLAIN, seed=7, max_depth=6, record_paths=4, timing=timing)
        _, rec = ctx.cache_export()
        got.append(np.sort(rec.view(np.float32).reshape(-1, 12).copy().view("V48").ravel()))
    assert np.array_equal(got[0], got[1])
