"""Loss and gradient at the edges of the gradient kernel's tiles (64 samples)
and of its grid (two blocks per SM), against the numpy oracle in 64 bits.
Tolerance: sums of n FP32 terms in runs of at most 64 x tiles per block and a
tree, weights exactly as the kernel holds them: a relative 2-norm error of
n-independent order 2^-24 x sqrt(64 + tiles) x a few terms per sum; 1e-5
leaves a factor of 20."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 148 * 2 * 64 - 1, 148 * 2 * 64 + 1, 50_000])
def test_gradient_at_tile_edges(gpu, n):
    rng = np.random.default_rng(n)
    params = MO.to_bf16((rng.standard_normal(MO.P) * 0.3).astype(np.float32))
    m = gpu.Model(0, params=params)
    x = rng.gamma(2.0, 2.0, (n, 16)).astype(np.float32)
    y = rng.standard_normal(n).astype(np.float32)
    for _ in range(2):  # the kept scratch of the first call serves the second
        loss, g = m.grad(x, y)
        ref_loss, ref_g = MO.loss_and_grad(params, x, y)
        assert abs(loss - ref_loss) <= 1e-5 * ref_loss
        assert np.linalg.norm(g - ref_g) <= 1e-5 * np.linalg.norm(ref_g)
