"""Evaluation parameters belong to the scene they were set for."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import scenes
from pathguidingdissertation_gb300.api import Context

pytestmark = pytest.mark.gpu


def _scene(n_objects, env, width, height):
    return scenes.interior(seed=3, target_tris=4000, n_objects=n_objects, width=width, height=height, env_width=2 * env,
                           env_height=env)


def test_a_new_upload_starts_from_its_own_parameters(ctx):
    """13 materials and a 32x16 map with parameters set, then 43 materials and
    a 128x64 map: the second scene's image and gradients are those of a
    context that never saw the first (one wave, sums in a fixed order: equal
    bits for the image)."""
    first = _scene(10, 16, 32, 24)
    ctx.upload(first)
    ctx.bvh_build()
    n = len(first.materials)
    ctx.diff_set_params(env=0.5 * first.env, albedo_offset=np.full((n, 3), 0.05, np.float32),
                        roughness=np.full(n, 0.4, np.float32))
    ctx.diff_render(2, seed=4, max_depth=4)
    second = _scene(40, 64, 40, 30)
    assert len(second.materials) > n and second.env.size > first.env.size
    fresh = Context(0)
    dimg = np.random.default_rng(1).normal(size=(30, 40, 3)).astype(np.float32)
    out = []
    for c in (ctx, fresh):
        c.upload(second)
        c.bvh_build()
        out.append((c.diff_render(4, seed=6, max_depth=5), *c.diff_adjoint(dimg, 4, seed=6, max_depth=5)))
    fresh.close()
    assert out[1][0].any()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for got, want in zip(out[0][1:], out[1][1:]):
        np.testing.assert_allclose(got, want, rtol=1e-6, atol=1e-6 * np.abs(want).max())
