"""The sizer's forward and backward kernel around its tile of 64 samples and past one tile per
resident block, against the FP64 oracle (fp32 sums of up to n terms: the bounds test_gpu_sizer.py
derives for hundreds of samples hold for all of these, as a block sums a few hundred itself)."""
import numpy as np
import pytest

import mlp_oracle as M


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 1000, 30011])
def test_mlp_matches_fp64(renderer, n):
    renderer.sizer_init(seed=n)
    params = renderer.sizer_params().astype(np.float64)
    rng = np.random.default_rng(n)
    x = np.abs(rng.normal(2.0, 1.5, (n, M.N_IN))).astype(np.float32)
    t = rng.normal(3.0, 1.0, (n, M.N_OUT)).astype(np.float32)
    want = M.predict(params, x)
    assert np.abs(renderer.sizer_predict(x) - want).max() <= 1e-4 * np.abs(want).max() + 1e-5
    grad, loss = renderer.sizer_gradient(x, t)
    lo, go = M.loss_and_grad(params, x, t)
    assert abs(loss - lo) <= 1e-4 * abs(lo) + 1e-6
    assert np.abs(grad.astype(np.float64) - go).max() <= 2e-4 * np.abs(go).max() + 1e-7
