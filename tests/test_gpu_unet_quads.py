"""The U-Net's convolutions that also make the 2 x 2 sums behind them and read a concatenation where
its parts are (csrc/unet.cu): every level's sums by the convolution or by a kernel of its own, at
images whose edges cut the 16 x 16 tiles.

The forward of a batch (sums made by the convolutions on all levels, or on some) equals that of its
images alone (fewer tiles: other levels' by a kernel of their own) bit for bit.  Gradients: the bounds
of tests/test_gpu_unet.py (6e-2 a layer, 3e-2 on average, relative L2) for the reason given there."""
import numpy as np
import pytest

import test_gpu_unet_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(9, 104, 136), (148, 16, 24), (2, 200, 184)])
def test_forward_with_sums_by_the_convolutions(B, H, W):
    tiles.test_batched_forward_equals_single_images(B, H, W)


@pytest.mark.parametrize("B,H,W", [(4, 104, 136), (1, 200, 184), (22, 40, 24)])
def test_gradients_with_sums_by_the_convolutions(B, H, W):
    tiles.test_gradients_match_the_oracle(B, H, W)
