"""The weight gradient of the learned stage where its split over blocks
changes: fewer tiles than blocks, several tiles a block with and without a
remainder, and blocks' partials summed over a large batch.

A batch of B copies of one sample has the gradient of that sample: the mean
squared error divides by B, every tile's partial is the single sample's
divided by B, exactly so when B is a power of two, and B of each are summed.
The two gradients therefore differ by the FP32 rounding of the sums alone:
at most 100 additions in a row (tiles of a block, blocks of a warp, warps) of
2^-24 each, relative to the sum of the partials' sizes, which is below the
number of one sample's tiles (64 at most here) times the result's:
100 * 2^-24 * 64 = 4e-4 of each layer's norm.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import learned_oracle as lo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,batch", [(16, 64), (32, 64), (48, 32), (64, 16), (64, 64)])
def test_gradient_of_copies_is_the_samples_gradient(sg, nx, batch):
    st = sg.LearnedCorrection(nx)
    try:
        rng = np.random.default_rng(nx)
        w = np.zeros(lo.NUM_PARAMS, np.float32)
        w[: lo.NET_PARAMS] = rng.uniform(-0.1, 0.1, lo.NET_PARAMS) * lo.param_mask()
        w[lo.NET_PARAMS] = 1.0
        st.weights = w
        x = rng.standard_normal((1, st.nc, 2)).astype(np.float32)
        t = rng.standard_normal((1, st.nc)).astype(np.float32)
        _, one = st.gradient(x, t)
        _, many = st.gradient(np.repeat(x, batch, 0), np.repeat(t, batch, 0))
        _, again = st.gradient(np.repeat(x, batch, 0), np.repeat(t, batch, 0))
        assert np.array_equal(many, again)
        for l in range(lo.LAYERS):
            sl = slice(l * lo.LAYER_P, (l + 1) * lo.LAYER_P)
            d = np.linalg.norm(many[sl].astype(float) - one[sl])
            assert d <= 4e-4 * np.linalg.norm(one[sl].astype(float)), l
    finally:
        st.close()
