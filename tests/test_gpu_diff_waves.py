"""Differentiable renders at the sizes where their kernels change: one path,
partial warps and tiles, the largest call of one thread per path (65,536) and
the smallest wavefront, one and several waves (2^24 paths of the primal, 2^22
of the adjoint), every depth limit end.  On a scene lit by its environment
alone the image is linear in the texels, so for any adjoint image d:
<d, image> = <gradient, texels>.  Both sides sum the same float32 terms of one
sign-free random d: a bound of 1e-4 of the terms' magnitude covers float32
rounding of the terms (2^-24 each, errors of either sign) with the gradient's
rounding to float32."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,spp,depth", [((1, 1), 1, 3), ((7, 5), 3, 0), ((33, 31), 5, 16), ((64, 48), 16, 8),
                                            ((256, 256), 1, 6), ((257, 256), 1, 6),
                                            ((512, 512), 17, 4), ((512, 512), 65, 2)])
def test_adjoint_is_the_transpose_of_the_primal(ctx, size, spp, depth):
    desc = scenes.terrain(grid=64, seed=4, width=size[0], height=size[1], env_width=64, env_height=32, sun_peak=20.0)
    ctx.upload(desc)
    ctx.bvh_build()
    rng = np.random.default_rng(spp)
    d = rng.uniform(0.5, 1.5, (size[1], size[0], 3)).astype(np.float32)
    img = ctx.diff_render(spp, seed=9, max_depth=depth)
    g_env, _, _ = ctx.diff_adjoint(d, spp, seed=9, max_depth=depth)
    lhs = float(np.sum(d.astype(np.float64) * img))
    rhs = float(np.sum(g_env.astype(np.float64) * desc.env))
    assert abs(lhs - rhs) <= 1e-4 * abs(lhs), (lhs, rhs)
    # masked samples contribute nothing: the gradient is additive over pixels
    half = d.copy()
    half[: size[1] // 2] = 0.0
    a = ctx.diff_adjoint(half, spp, seed=9, max_depth=depth)
    b = ctx.diff_adjoint(d - half, spp, seed=9, max_depth=depth)
    np.testing.assert_allclose(a[0] + b[0], g_env, rtol=1e-4, atol=1e-6 * float(np.abs(g_env).max()))
