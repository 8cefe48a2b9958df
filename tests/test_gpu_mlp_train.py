"""The training kernel at the ends of its tiles (128 samples, one tile a block
at a time).  Samples of weight zero add exact zeros, so one weighted sample
anywhere among them has exactly the gradient it has alone; and a
permutation of the samples only changes the order of float32 sums: n terms of
either sign, 2 n 2^-24 of the sum of their magnitudes, itself about sqrt(n)
times the sum's norm."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo
from pathguidingdissertation_gb300 import abi

pytestmark = pytest.mark.gpu

LO, HI = np.array([-1.0, 0.0, -2.0], np.float32), np.array([3.0, 2.0, 1.0], np.float32)


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    unit = lambda: (lambda v: v / np.linalg.norm(v, axis=1, keepdims=True))(rng.normal(size=(n, 3)))  # noqa: E731
    s = np.zeros(n, abi.RADIANCE_SAMPLE)
    s["position"] = rng.uniform(LO - 0.1, HI + 0.1, (n, 3))
    s["normal"], s["wo"], s["wi"] = unit(), unit(), unit()
    s["weight"] = rng.uniform(0.1, 2.0, n)
    return s


@pytest.fixture()
def net(ctx):
    ctx.mlp_init(1, LO, HI)
    ctx.mlp_set_params(mo.init_params(3))
    return ctx


@pytest.mark.parametrize("n,at", [(2, 1), (128, 127), (129, 128), (300, 5), (152 * 128 + 1, 152 * 128), (40000, 39999)])
def test_one_weighted_sample_anywhere(net, n, at):
    s = _samples(n, n)
    s["weight"] = 0.0
    s["weight"][at] = 0.75
    grad, loss = net.mlp_gradient(s)
    alone, alone_loss = net.mlp_gradient(s[at:at + 1])
    assert np.array_equal(grad, alone) and loss == alone_loss
    assert np.any(grad != 0)


@pytest.mark.parametrize("n", [31, 127, 128, 129, 300])
def test_permutation_changes_only_sums(net, n):
    s = _samples(n, n)
    a, _ = net.mlp_gradient(s)
    b, _ = net.mlp_gradient(s[np.random.default_rng(1).permutation(n)])
    assert np.linalg.norm(a - b) <= 2.0 * n ** 1.5 * 2.0 ** -24 * np.linalg.norm(a)
