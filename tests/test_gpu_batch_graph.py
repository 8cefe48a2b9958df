"""A batch replays its captured graph only where it is the graph of the call:
every tuning field that shapes the launches is part of the decision, and so
are the path-state buffers whose addresses the graph holds."""
from __future__ import annotations

import numpy as np
import pytest

from pathguidingdissertation_gb300 import abi, scenes
from pathguidingdissertation_gb300.api import Batch, Context

pytestmark = pytest.mark.gpu


def _ctx(seed, width, height):
    c = Context(0)
    c.upload(scenes.cornell_box(seed=seed, width=width, height=height))
    c.bvh_build()
    c.clear()
    return c


def _films(ctxs):
    return [c.film()[0].astype(np.float64) for c in ctxs]


def _assert_close(got, want):
    # same paths; only the order of the film's float additions differs
    for a, r in zip(got, want):
        assert r.any() and np.max(np.abs(a - r) / np.maximum(np.abs(r), 1e-3)) < 1e-4


def test_stack_depth_is_part_of_the_graph(pgx_lib):
    sizes = [(1, 48, 48), (2, 64, 32)]
    ctxs, solo = [_ctx(*s) for s in sizes], [_ctx(*s) for s in sizes]
    for c in solo:
        c.render(2, mode=abi.MODE_PLAIN, seed=9, max_depth=8)
    want = _films(solo)
    b = Batch(ctxs)
    for sh in (4, 8, 16, 8):
        for again in (0, 1):
            for c in ctxs:
                c.clear()
            b.set_tuning(1 << 20, 8, 16, stack_shared=sh)
            b.render(2, seed=9, max_depth=8)
            assert b.stats().graph_replayed == again
            _assert_close(_films(ctxs), want)
    b.close()
    for c in ctxs + solo:
        c.close()


def test_reallocated_state_is_not_replayed(pgx_lib):
    """Autotuning tries waves up to twice the batch's paths; where that
    reallocates the path state, the graph captured before must not run."""
    sizes = [(1, 512, 512), (2, 512, 512), (3, 512, 640)]
    ctxs, solo = [_ctx(*s) for s in sizes], [_ctx(*s) for s in sizes]
    for c in solo:
        c.render(2, mode=abi.MODE_PLAIN, seed=9, max_depth=4)
    want = _films(solo)
    b = Batch(ctxs)
    b.set_tuning(1 << 20, 8, 16)  # 1.7 M paths: two waves
    b.render(2, seed=9, max_depth=4)
    _assert_close(_films(ctxs), want)
    b.autotune(spp=2, max_depth=4)  # tries waves of 2^21
    for again in (0, 1):
        for c in ctxs:
            c.clear()
        b.set_tuning(1 << 20, 8, 16)
        b.render(2, seed=9, max_depth=4)
        assert b.stats().graph_replayed == again
        _assert_close(_films(ctxs), want)
    b.close()
    for c in ctxs + solo:
        c.close()
