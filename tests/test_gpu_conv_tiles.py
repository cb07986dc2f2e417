"""Edges of the convolution's tiles (conv_tc.cu): 126 output columns a tile, two or four rows where
the tiles fill the SMs and half of that where they do not, remainders of each; against the FP64
oracle with the tolerance of test_gpu_conv.py (FP32 accumulation, one rounding to bf16)."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from test_gpu_conv import close_bf16, inputs, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (5, 125), (3, 126), (7, 127), (2, 253), (301, 261)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 64), (64, 32)])
def test_conv_tile_edges(cin, cout, H, W):
    x, w, b = inputs(cin, cout, H, W, 100 * H + W)
    got, _ = run(cin, cout, H, W, x, w, b, relu=1)
    want = U.relu(U.conv3x3(x, w, b.astype(np.float32).astype(np.float64)))
    close_bf16(got, want, U.conv3x3(np.abs(x), np.abs(w)).max())
