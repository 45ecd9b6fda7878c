"""The weight gradients of the tcgen05 path (W % 128 == 0) against the warp-level
MMA kernels', layer by layer, at fewer tiles than CTAs, at more with a remainder,
and at rows of one to three tiles.

Both paths sum the same bfloat16 products in FP32; they differ by activations and
gradients that round to the other bfloat16 neighbour (2^-8 of the value at most)
after another order of accumulation, once per layer: 6 layers forward and back, so
6 * 2^-8 of a gradient's norm.  A missing or misplaced halo row, column or chunk
changes it by a tenth or more at these heights."""
import numpy as np
import pytest

from test_gpu_cnn import _layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,B", [(8, 128, 1), (8, 384, 1), (40, 256, 8), (16, 256, 5)])
def test_weight_gradients_match_the_warp_mma_ones(gpu, monkeypatch, H, W, B):
    import torch
    from rot2d3c_gb300.closure import CNN
    rng = np.random.default_rng(H + W + B)
    x = torch.from_numpy(rng.standard_normal((B, H, W, 8)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal((B, H, W, 2)).astype(np.float32)).cuda()
    grads = []
    for mode in ("tcgen05", "mma"):
        monkeypatch.setenv("R2D3C_CNN_CONV", mode)
        net = CNN(H, W, B, seed=11)
        grads.append([net.gradients(x, t, B)[1] for _ in range(2)])
    (a, a2), (b, _) = grads
    assert np.array_equal(a, a2)  # a fixed order of summation
    for l, slices in enumerate(_layer_slices()):
        for sl in slices:
            assert np.linalg.norm(a[sl] - b[sl]) <= 6 / 256 * np.linalg.norm(b[sl]), (l, sl)
