"""Calls that ask for more device memory than there is: they return an error,
and the context goes on working with what fits.

The shortage is made by holding the device's free memory, all but a stated
rest, in one allocation for the length of a test; nothing is launched that
lacks its buffers."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

GB = 1 << 30


@contextlib.contextmanager
def only_free(rest: int):
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    if free <= rest + GB:
        pytest.skip("the device has too little free memory for this test")
    held = torch.empty(free - rest, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _film(ctx):
    return ctx.film()[0].astype(np.float64)


def _assert_close(got, want):
    # same paths; only the order of the film's float additions differs
    assert want.any() and np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-3)) < 1e-4


def test_render_after_a_render_that_did_not_fit(ctx):
    """512x512 x 64 samples need 3.1 GB of path state in one wave, one sample 49 MB."""
    ctx.upload(scenes.cornell_box(seed=1, width=512, height=512))
    ctx.bvh_build()
    ctx.clear()
    ctx.render(1, mode=abi.MODE_PLAIN, seed=3, max_depth=6)
    want = _film(ctx)
    ctx.render(1, mode=abi.MODE_PLAIN, seed=4, max_depth=6, record_paths=1)
    recorded = ctx.cache_stats().records
    assert recorded > 0
    ctx.clear()
    with only_free(3 * GB // 2):
        with pytest.raises(abi.PgxError) as err:
            ctx.render(64, mode=abi.MODE_PLAIN, seed=3, max_depth=6)
        assert err.value.code == abi.PGX_ERR_CUDA and "memory" in str(err.value)
        assert ctx.film()[2] == 0 and not _film(ctx).any()
        ctx.render(1, mode=abi.MODE_PLAIN, seed=3, max_depth=6)
        _assert_close(_film(ctx), want)
        # recording needs more per path: 8 samples do not fit, one does
        with pytest.raises(abi.PgxError):
            ctx.render(8, mode=abi.MODE_PLAIN, seed=3, max_depth=16, record_paths=8)
        ctx.cache_build_from_render()  # the vertices of the last recording are still there
        assert ctx.cache_stats().records == recorded
        ctx.clear()
        ctx.render(1, mode=abi.MODE_PLAIN, seed=3, max_depth=6, record_paths=1)
        _assert_close(_film(ctx), want)
    ctx.clear()
    ctx.render(64, mode=abi.MODE_PLAIN, seed=3, max_depth=6)
    assert ctx.film()[2] == 64


def test_differentiable_calls_fit_their_waves_to_the_memory(ctx):
    """512x512 x 40 samples: full waves need 2.1 GB (primal) and, with 17
    depths of vertex records, 6.5 GB (adjoint); smaller ones give the same
    image bit for bit and the same gradient up to the order of its double
    sums."""
    ctx.upload(scenes.interior(seed=3, target_tris=3000, n_objects=10, width=512, height=512, env_width=64,
                               env_height=32))
    ctx.bvh_build()
    dimg = np.random.default_rng(2).normal(size=(512, 512, 3)).astype(np.float32)
    want = ctx.diff_render(40, seed=5, max_depth=16)
    want_grads = ctx.diff_adjoint(dimg, 40, seed=5, max_depth=16)
    ctx.close()
    fresh = type(ctx)(0)
    fresh.upload(scenes.interior(seed=3, target_tris=3000, n_objects=10, width=512, height=512, env_width=64,
                                 env_height=32))
    fresh.bvh_build()
    with only_free(3 * GB // 2):
        np.testing.assert_array_equal(fresh.diff_render(40, seed=5, max_depth=16), want)
        for got, ref in zip(fresh.diff_adjoint(dimg, 40, seed=5, max_depth=16), want_grads):
            # sums of up to 1.7e8 doubles of mixed signs in another order
            # (2^-53 x terms x mean magnitude), rounded to float at the end
            np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-6 * np.abs(ref).max())
    fresh.close()
