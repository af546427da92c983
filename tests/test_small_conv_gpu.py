"""Convolutions of every size class under CCT_ALGO_AUTO: the fp32 kernels that small layers take, and the split reductions
and uneven channel tiles of the tensor-core kernels, against the CPU restatement.  Tolerance: the 1e-4 of tests/parity.py
(fp32 products summed over at most a few thousand terms stay two orders below it, the tensor-core path's split operands one)."""
import pytest

from tests.parity import assert_close, make_inputs

pytestmark = pytest.mark.gpu

AUTO, TENSOR = 0, 2

# B, D, n, o, k, s, p, g
SHAPES = [
    (1, 1, 5, 1, 1, 1, 0, 1),         # one channel, one filter, one column per lane
    (3, 3, 7, 5, 3, 1, 1, 1),         # three channels: no split of the input channels; five filters: a tile of four and one
    (3, 4, 7, 8, 3, 1, 1, 1),         # four channels: the warps share positions
    (2, 9, 6, 9, 3, 2, 1, 1),         # stride 2, channels that do not divide over the warps
    (2, 70, 9, 18, 3, 1, 1, 2),       # 35 channels per group over up to sixteen warps
    (5, 6, 13, 20, 5, 1, 0, 1), (2, 6, 14, 12, 5, 2, 2, 1), (2, 3, 30, 33, 7, 2, 3, 1), (2, 3, 17, 9, 7, 1, 3, 1),
    (1, 4, 47, 24, 11, 4, 0, 1), (1, 3, 46, 30, 11, 4, 5, 1),
    (40, 2, 19, 70, 3, 1, 0, 1),      # 11 560 pixels: several chunks per block of the weight gradient, three channel tiles
    (1, 128, 9, 200, 3, 1, 1, 1),     # 81 pixels: reduction split over CTAs, forward and data gradient
    (1, 36, 6, 293, 3, 1, 1, 1), (1, 293, 6, 24, 3, 1, 1, 1),  # prime channel counts: the last channel tile is shorter
    (2, 64, 13, 263, 3, 2, 1, 1), (7, 40, 15, 96, 3, 1, 1, 1),
]


@pytest.mark.parametrize("algo", [AUTO, TENSOR])
@pytest.mark.parametrize("shape", SHAPES)
def test_small_and_split_convolutions(ctx, port, shape, algo):
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    X, W, b, dY = make_inputs(17, B, D, n, o, k, s, p, g)
    Y, dX, dW, db, used = conv_layer(ctx, X, W, b, dY, k, s, p, g, algo=algo)
    assert used == TENSOR
    dXr, dWr, dbr = port.conv_backward(X, W, dY, k, s, p, g)
    for a, r, name in ((Y, port.conv_forward(X, W, b, k, s, p, g), "Y"), (dX, dXr, "dX"), (dW, dWr, "dW"), (db, dbr, "db")):
        assert_close(a, r.reshape(a.shape), name)
