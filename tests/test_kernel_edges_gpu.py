"""The branches that a layer's sizes choose between, each at the sizes where it can go wrong: edges of tiles, remainders, the
smallest and largest of its range."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest
import torch

from caffecontroll_b200 import FullyConnectedBridge, Layer, LogicalCube, capi
from oracle import pyoracle
from tests.parity import assert_close, make_inputs

pytestmark = pytest.mark.gpu

TENSOR = 2


def vp(p):
    return C.c_void_p(p)


# Window rows loaded in 16-byte blocks (stride a multiple of four, no padding), k-blocks that cross images, odd planes whose
# blocks are misaligned, the tensor's ends, groups; then narrow data gradients with padding and stride.  Tolerance:
# tests/parity.py (1e-4; the split operands stay below 2e-5).
@pytest.mark.parametrize("shape", [
    (1, 3, 11, 8, 11, 4, 0, 1), (3, 3, 47, 24, 11, 4, 0, 1), (5, 4, 23, 17, 8, 4, 0, 1), (2, 2, 61, 128, 13, 8, 0, 1),
    (2, 6, 39, 40, 11, 4, 0, 2), (2, 4, 30, 9, 9, 4, 0, 1), (2, 3, 40, 16, 11, 4, 5, 1),
    (6, 20, 28, 32, 5, 1, 2, 1), (9, 16, 33, 64, 3, 1, 1, 1), (4, 24, 29, 80, 5, 2, 2, 1), (3, 3, 57, 96, 11, 4, 0, 1),
])
def test_convolution_shapes(ctx, port, shape):
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    X, W, b, dY = make_inputs(29, B, D, n, o, k, s, p, g)
    Y, dX, dW, db, used = conv_layer(ctx, X, W, b, dY, k, s, p, g, algo=TENSOR)
    assert used == TENSOR
    dXr, dWr, dbr = port.conv_backward(X, W, dY, k, s, p, g)
    for a, r, name in ((Y, port.conv_forward(X, W, b, k, s, p, g), "Y"), (dX, dXr, "dX"), (dW, dWr, "dW"), (db, dbr, "db")):
        assert_close(a, r.reshape(a.shape), name)


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("shape", [
    (32, 30, 40, 134, 3, 1, 1, 1), (9, 16, 33, 64, 3, 1, 1, 1), (6, 20, 28, 32, 5, 1, 2, 1), (4, 8, 14, 24, 3, 1, 0, 1),
    (32, 96, 27, 256, 5, 1, 2, 2),
])
def test_a_gradient_that_is_not_finite_stays_in_its_window(ctx, shape, value):
    """dX outside the window of one element of dY does not depend on that element, whatever it is: bit for bit."""
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    X, W, b, dY = make_inputs(31, B, D, n, o, k, s, p, g)
    W = np.where(W == 0, np.float32(0.01), W)
    m = (n + 2 * p - k) // s + 1
    where = (B - 1, o // g - 1, m // 2, m // 2 + 1)
    dY[where] = 0
    _, clean, _, _, _ = conv_layer(ctx, X, W, b, dY, k, s, p, g, algo=TENSOR)
    dY[where] = value
    _, dX, _, _, used = conv_layer(ctx, X, W, b, dY, k, s, p, g, algo=TENSOR)
    assert used == TENSOR
    bad = ~np.isfinite(dX)
    window = np.zeros(dX.shape, bool)
    y, x = where[2] - p, where[3] - p
    window[B - 1, :D // g, max(y, 0):y + k, max(x, 0):x + k] = True
    assert np.array_equal(bad, window)
    assert np.array_equal(dX[~window], clean[~window])


# Forward passes without padding (no bounds test on the gathered operand), reductions that end inside a block of 32, fewer pixels
# than a tile, groups; and one with padding.
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("shape", [(1, 3, 11, 8, 11, 4, 0, 1), (3, 3, 47, 96, 11, 4, 0, 1), (2, 10, 15, 130, 3, 1, 0, 2), (5, 7, 12, 70, 2, 2, 0, 1),
                                   (9, 33, 9, 80, 1, 1, 0, 1), (2, 3, 20, 72, 7, 2, 3, 1)])
def test_an_input_that_is_not_finite_stays_in_its_windows(ctx, shape, value):
    """Y outside the windows that hold one element of X does not depend on that element: bit for bit."""
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    X, W, b, _ = make_inputs(41, B, D, n, o, k, s, p, g)
    W = np.where(W == 0, np.float32(0.01), W)
    m = (n + 2 * p - k) // s + 1
    where = (B - 1, 0, n // 2, n // 2)
    X[where] = 0
    clean = conv_layer(ctx, X, W, b, None, k, s, p, g, algo=TENSOR)[0]
    X[where] = value
    Y = conv_layer(ctx, X, W, b, None, k, s, p, g, algo=TENSOR)[0]
    inside = [r * s - p <= n // 2 < r * s - p + k for r in range(m)]
    window = np.zeros(Y.shape, bool)
    window[B - 1, :o // g] = np.outer(inside, inside)
    assert np.array_equal(~np.isfinite(Y), window)
    assert np.array_equal(Y[~window], clean[~window])


@pytest.mark.parametrize("algo", [capi.ALGO_AUTO, TENSOR])
def test_many_groups(ctx, port, algo):
    """4096 groups of one channel are 65 536 rows of a packed operand; 65 600 groups (forward only) are more channel tiles than a
    grid has in y."""
    from caffecontroll_b200 import conv_layer
    for B, g, n, backward in ((2, 4096, 5, True), (1, 65600, 3, False)):
        X, W, b, dY = make_inputs(37, B, g, n, g, 3, 1, 1, g, bias=backward)  # (65 600 biases do not fit in shared memory)
        Y, dX, dW, db, used = conv_layer(ctx, X, W, b, dY if backward else None, 3, 1, 1, g, algo=algo)
        assert used == TENSOR
        assert_close(Y, port.conv_forward(X, W, b if backward else np.zeros(g, np.float32), 3, 1, 1, g).reshape(Y.shape), "Y")
        if backward:
            for a, r, name in zip((dX, dW, db), port.conv_backward(X, W, dY, 3, 1, 1, g), ("dX", "dW", "db")):
                assert_close(a, r.reshape(a.shape), name)


# The tensor core truncates.  An instruction adds eight products to a sum: the sum loses half a place on average, each product,
# aligned to it and cut two bits below its last place, an eighth - 1.5 places in all.  A place is 2^-23 .. 2^-24 of the sum
# (0.72 * 2^-23 on average) and over positive data the sum grows steadily (half its final value on average), so N instructions
# at full magnitude lose N * 1.5 * 0.72 * 2^-24 = N * 2^-23.9; the operand split adds less than 2^-21.  `chain`: the pass's
# accumulation chain in blocks of 32 products, one such instruction per eight products.
@pytest.mark.parametrize("shape,which,chain", [
    ((48, 96, 24, 41, 5, 1, 2, 1), "Y", 75), ((64, 64, 20, 64, 3, 1, 1, 1), "dX", 18),
    ((48, 96, 24, 41, 5, 1, 2, 1), "dW", 58), ((64, 64, 20, 64, 3, 1, 1, 1), "dW", 28),
    # 38 blocks, 76 at the two additions per block that narrow tiles may take; units of the weight gradient's splits, three
    # additions per block on wide tiles; uneven channel tiles
    ((32, 30, 40, 134, 3, 1, 1, 1), "dX", 76), ((32, 48, 28, 134, 3, 1, 1, 1), "dX", 76),
    ((8, 158, 45, 136, 5, 1, 2, 1), "dW", 3 * 57), ((5, 272, 25, 208, 5, 1, 2, 2), "dW", 3 * 20), ((40, 64, 30, 337, 3, 1, 1, 1), "dW", 3 * 58),
])
def test_accumulation_error(ctx, shape, which, chain):
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    m = (n + 2 * p - k) // s + 1
    gen = torch.Generator().manual_seed(B + o)
    X, W, dY = (torch.rand(sh, generator=gen) for sh in ((B, D, n, n), (o, D // g, k, k), (B, o, m, m)))
    Y, dX, dW, db, used = conv_layer(ctx, X.numpy(), W.numpy(), np.zeros(o, np.float32), dY.numpy(), k, s, p, g, algo=TENSOR)
    assert used == TENSOR
    Xd, Wd, dYd = X.double().requires_grad_(), W.double().requires_grad_(), dY.double()
    Yr = torch.nn.functional.conv2d(Xd, Wd, None, s, p, 1, g)
    Yr.backward(dYd)
    got, ref = {"Y": (Y, Yr.detach()), "dX": (dX, Xd.grad), "dW": (dW, Wd.grad)}[which]
    err = float((torch.from_numpy(got).double() - ref).norm() / ref.norm())
    assert err <= 4 * chain * 2.0 ** -23.9 + 2.0 ** -21, "%s: relative error %.2e, chain of %d" % (which, err, chain)


# One product per sum, so that nothing averages out.  x = hi + lo, hi cut to tf32's 11 bits; lo has up to 13 bits, of which the tensor
# core reads 11 (2^-21 of x's power of two); lo * lo is left out (2^-20); two more additions cut the sum (2^-22): 2^-20 + 2 * 2^-21 +
# 2^-22 of the product for two operands split so.  (Cross terms of operands with eight bits: 2^-17.)  Sums without a product are 0.
ONE_PRODUCT = 2.25 * 2.0 ** -20


def assert_products(got, ref, name):
    off = np.abs(got.astype(np.float64) - ref)
    assert np.all(off <= ONE_PRODUCT * np.abs(ref)), "%s: %.2e of a product" % (name, (off / np.maximum(np.abs(ref), 1e-30)).max())


# Filters with a single weight, each of another channel: Y and dX are single products; one element of dY per channel and every input
# channel of its own tile: so is dW.  Tiles of 64 columns and of more, reductions of seven, eight and many blocks of 32, each of the
# kernels for the weight gradient: gather (at least 512 lowered rows), dY through tensor memory (257 - 384), shorter ones.
@pytest.mark.parametrize("shape", [
    (3, 224, 14, 80, 1, 1, 0, 1), (3, 256, 14, 200, 1, 1, 0, 1), (3, 264, 14, 64, 1, 1, 0, 1), (4, 300, 13, 136, 3, 1, 1, 1),
    (8, 512, 27, 272, 1, 1, 0, 2), (24, 28, 40, 100, 3, 1, 1, 1), (24, 12, 40, 28, 3, 1, 1, 1), (40, 3, 115, 96, 11, 4, 0, 1),
])
def test_single_products(ctx, shape):
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    m = (n + 2 * p - k) // s + 1
    rng = np.random.default_rng(D + o)
    X, dY = (rng.standard_normal(sh).astype(np.float32) for sh in ((B, D, n, n), (B, o, m, m)))
    W = np.zeros((o, D // g, k, k), np.float32)
    at = np.arange(o)
    W[at, at % (o // g) % (D // g), at % k, at // k % k] = rng.standard_normal(o)
    one = np.zeros_like(dY)
    one[at % B, at, at % m, at // m % m] = rng.standard_normal(o)
    conv = lambda x, w, dy: conv_layer(ctx, x, w, np.zeros(o, np.float32), dy, k, s, p, g, algo=TENSOR)  # noqa: E731
    Y, dX, _, _, used = conv(X, W, dY)
    dW = conv(X, W, one)[2]
    assert used == TENSOR

    def exact(dy):
        x, w = (torch.from_numpy(t).double().requires_grad_() for t in (X, W))
        y = torch.nn.functional.conv2d(x, w, None, s, p, 1, g)
        y.backward(torch.from_numpy(dy).double())
        return y.detach().numpy(), x.grad.numpy(), w.grad.numpy()

    y, dx, _ = exact(dY)
    assert_products(Y, y, "Y")
    if o <= D:  # (otherwise several filters share a channel)
        assert_products(dX, dx, "dX")
    assert_products(dW, exact(one)[2].reshape(dW.shape), "dW")


# One feature per image, one output per image: every sum of the three passes is a single product.
@pytest.mark.parametrize("B,K,o", [(130, 2052, 4224), (70, 2304, 5000), (17, 4164, 4100), (256, 4608, 4608)])
def test_single_products_of_inner_products(ctx, B, K, o):
    rng = np.random.default_rng(K)
    W, at = rng.standard_normal((o, K)).astype(np.float32), np.arange(B)
    X, dY, b = np.zeros((B, K), np.float32), np.zeros((B, o), np.float32), np.zeros(o, np.float32)
    X[at, rng.permutation(K)[:B]], dY[at, rng.permutation(o)[:B]] = rng.standard_normal((2, B))
    c = {name: LogicalCube.from_numpy(ctx, t.reshape(1, 1, *t.reshape(-1, t.shape[-1]).shape))
         for name, t in (("X", X), ("W", W), ("b", b), ("dY", dY), ("Y", 0 * dY), ("dX", 0 * X), ("dW", 0 * W), ("db", 0 * b))}
    plan, q = C.c_void_p(), {name: cube.ptr for name, cube in c.items()}
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, q["X"], q["W"], q["b"], q["Y"], 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, q["X"], q["W"], q["dY"], q["dX"], q["dW"], q["db"], 0, None, 1.0), "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    X, W, dY = (t.astype(np.float64) for t in (X, W, dY))
    for name, ref in (("Y", X @ W.T), ("dX", dY @ W), ("dW", dY.T @ X)):
        assert_products(c[name].download().reshape(ref.shape), ref, name)
    for cube in c.values():
        cube.free()


# Data of random sign: both sides of the line of 64 columns, reductions that are no multiple of 32 or of eight channels.  Relative
# 2-norms: the operand split below 2^-21, the truncating additions as above, three per eight products at the most.  Chains: the whole
# reduction, of the weight gradient at most 19 blocks of 32 pixels (1 200 and 1 250 blocks in splits of nine for the last two), which
# keeps the bound at 1.6e-5 where a missing cross term gives 4e-4.
@pytest.mark.parametrize("shape", [
    (3, 224, 14, 80, 1, 1, 0, 1), (3, 256, 14, 80, 1, 1, 0, 1), (3, 257, 14, 65, 1, 1, 0, 1), (3, 264, 14, 64, 1, 1, 0, 1),
    (5, 29, 15, 130, 3, 1, 1, 1), (2, 160, 17, 272, 3, 1, 1, 2), (4, 40, 19, 300, 5, 2, 2, 1),
    (24, 28, 40, 75, 3, 1, 1, 1), (25, 28, 40, 170, 3, 1, 1, 1),  # both operands of the weight gradient in shared memory
])
def test_sums_of_random_sign(ctx, shape):
    from caffecontroll_b200 import conv_layer
    B, D, n, o, k, s, p, g = shape
    m = (n + 2 * p - k) // s + 1
    gen = torch.Generator().manual_seed(D + o)
    X, W, dY = (torch.randn(sh, generator=gen) for sh in ((B, D, n, n), (o, D // g, k, k), (B, o, m, m)))
    Y, dX, dW, db, used = conv_layer(ctx, X.numpy(), W.numpy(), np.zeros(o, np.float32), dY.numpy(), k, s, p, g, algo=TENSOR)
    assert used == TENSOR
    Xd, Wd, dYd = X.double().requires_grad_(), W.double().requires_grad_(), dY.double()
    Yr = torch.nn.functional.conv2d(Xd, Wd, None, s, p, 1, g)
    Yr.backward(dYd)
    for got, ref, products in ((Y, Yr.detach(), D // g * k * k), (dX, Xd.grad, o // g * k * k), (dW, Wd.grad, min(B * m * m, 19 * 32))):
        err = float((torch.from_numpy(got).double() - ref).norm() / ref.norm())
        assert err <= 4 * 3 * (products // 32 + 1) * 2.0 ** -23.9 + 2.0 ** -21, "relative error %.2e" % err


def test_the_largest_values(ctx):
    """The largest fp32 numbers, which no rounding of an operand may turn into Inf, times small ones."""
    from caffecontroll_b200 import conv_layer
    B, D, n, o = 2, 320, 8, 96
    rng = np.random.default_rng(5)
    X = rng.choice(np.float32([3.4028234e38, -3.4e38, 1.0]), (B, D, n, n)).astype(np.float32)
    W = (1e-12 * rng.standard_normal((o, D, 1, 1))).astype(np.float32)
    Y = conv_layer(ctx, X, W, np.zeros(o, np.float32), None, 1, 1, 0, 1, algo=TENSOR)[0]
    ref = np.einsum("bdyx,od->boyx", X.astype(np.float64), W[:, :, 0, 0].astype(np.float64))
    assert np.isfinite(Y).all() and np.linalg.norm(Y / 1e26 - ref / 1e26) <= 1e-5 * np.linalg.norm(ref / 1e26)


# Inner products: one product, features that are no multiple of four (padded copies or the fp32 kernel), both sides of the
# line between the fp32 and the tensor-core kernel, batches at the accumulator widths of 64, 128 and 256 columns.
# Tolerance: products of unit values summed over K: split operands leave 2^-20 of the sum of magnitudes, far below 1e-4.
@pytest.mark.parametrize("B,K,o", [(1, 1, 1), (3, 5, 7), (50, 500, 10), (33, 1023, 129), (64, 515, 2050), (65, 2049, 513),
                                   (128, 1026, 514), (129, 770, 1027), (257, 301, 260)])
def test_inner_product_sizes(ctx, B, K, o):
    rng = np.random.default_rng(B + K + o)
    X, W, b, dY = (rng.standard_normal(s).astype(np.float32) for s in ((B, K, 1, 1), (o, K, 1, 1), (o,), (B, o, 1, 1)))
    xin = Layer(LogicalCube.from_numpy(ctx, X), LogicalCube(ctx, 1, 1, K, B))
    out = Layer(LogicalCube(ctx, 1, 1, o, B), LogicalCube.from_numpy(ctx, dY))
    fc = FullyConnectedBridge(xin, out, True)
    fc.p_model_cube.upload(W)
    fc.p_bias_cube.upload(b)
    fc.forward()
    fc.backward()
    ctx.sync()
    X2, W2, dY2 = X.reshape(B, K).astype(np.float64), W.reshape(o, K).astype(np.float64), dY.reshape(B, o).astype(np.float64)
    for cube, r, name in ((out.p_data_cube, X2 @ W2.T + b, "Y"), (xin.p_gradient_cube, dY2 @ W2, "dX"),
                          (fc.p_model_gradient_cube, dY2.T @ X2, "dW"), (fc.p_bias_gradient_cube, dY2.sum(0), "db")):
        got = cube.download()
        assert_close(got, r.astype(np.float32).reshape(got.shape), name)
    fc.close()


# Chains of many blocks of 32: padded and ragged features, batches at the edges of the accumulator widths.  Relative 2-norms: see
# test_sums_of_random_sign.
@pytest.mark.parametrize("B,K,o", [(130, 2050, 4224), (70, 2304, 5000), (17, 4164, 4100), (256, 4608, 4608)])
def test_inner_product_long_chains(ctx, B, K, o):
    gen = torch.Generator(device="cuda").manual_seed(K)
    make = lambda *sh: torch.randn(sh, generator=gen, device="cuda")  # noqa: E731
    X, W, b, dY = make(B, K), make(o, K), make(o), make(B, o)
    Y, dX, dW, db = torch.zeros_like(dY), torch.zeros_like(X), torch.zeros_like(W), torch.zeros_like(b)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    Xd, Wd, dYd = X.double(), W.double(), dY.double()
    for got, ref, products in ((Y, Xd @ Wd.T + b.double(), K), (dX, dYd @ Wd, o), (dW, dYd.T @ Xd, B)):
        err = float((got.double() - ref).norm() / ref.norm())
        assert err <= 4 * 3 * (min(products, 96 * 32) // 32 + 1) * 2.0 ** -23.9 + 2.0 ** -21, "relative error %.2e" % err


# dX written over dY, the whole of it or a part, where the bias gradient would ride with the launch that writes dX: bit for bit what
# separate buffers give, every time.
@pytest.mark.parametrize("B,K,shift", [(256, 1024, 0), (40, 2048, 0), (130, 1024, 64), (130, 1024, -64)])
def test_inner_product_gradient_in_place(ctx, B, K, shift):
    gen = torch.Generator(device="cuda").manual_seed(B)
    make = lambda *sh: torch.randn(sh, generator=gen, device="cuda")  # noqa: E731
    X, W, dY = make(B, K), make(K, K), make(B, K)
    apart, dWs, dbs = torch.zeros_like(X), [torch.zeros_like(W) for _ in range(2)], [torch.zeros(K, device="cuda") for _ in range(2)]
    both, plan, q = torch.zeros(B * K + 128, device="cuda"), C.c_void_p(), lambda t: t.data_ptr()
    over, inside = both[64:64 + B * K], both[64 + shift:64 + shift + B * K]  # dY, dX
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, K, 1, C.byref(plan)), "plan", ctx.h)
    run = lambda dy, dx, k: capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dy), q(dx), q(dWs[k]), q(dbs[k]), 0, None, 1.0),  # noqa: E731
                                       "backward", ctx.h)
    run(dY, apart, 0)
    for _ in range(5):
        over.copy_(dY.view(-1))
        torch.cuda.synchronize()
        run(over, inside, 1)
        ctx.sync()
        assert torch.equal(inside.view(B, K), apart) and torch.equal(dWs[0], dWs[1]) and torch.equal(dbs[0], dbs[1])
    ctx.lib.cct_fc_plan_destroy(plan)


# Outputs over operands in layers of the fp32 kernels, with and without splits of a reduction, where an operand off a 16-byte boundary brings a
# layer of the tensor cores there, and on the tensor cores (alone, both contractions together, rows in padded copies): Y over X, dX over dY, dX over the weights, bit for bit what separate buffers give, every time.
@pytest.mark.parametrize("B,K,off", [(64, 32, 0), (256, 200, 0), (450, 210, 0), (577, 256, 0), (640, 256, 0), (385, 200, 0), (40, 256, 0), (256, 640, 1),
                                     (256, 640, 0), (64, 800, 0), (130, 1026, 0)])
def test_inner_products_over_their_operands(ctx, B, K, off):
    gen = torch.Generator(device="cuda").manual_seed(B)
    make = lambda *sh: torch.randn(sh, generator=gen, device="cuda")  # noqa: E731
    X, W, dY, b = make(B, K), make(K, K), make(B, K), make(K)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, K, 1, C.byref(plan)), "plan", ctx.h)

    def run(over):
        words = off + (B + K) * K
        spare = lambda: torch.zeros(words, device="cuda")[off:]  # noqa: E731
        x, w, dy, y, dx, dw, db = (spare() for _ in range(7))
        for buffer, values in ((x, X), (w, W), (dy, dY)):
            buffer[:values.numel()].copy_(values.view(-1))
        if over == "Y over X":
            y = x
        elif over == "dX over dY":
            dx = dy
        elif over == "dX over W":
            dx = w
        torch.cuda.synchronize()
        if over in ("", "Y over X"):
            capi.check(ctx.lib.cct_fc_forward(plan, q(x), q(w), q(b), q(y), 1, None, 1.0), "forward", ctx.h)
        if over != "Y over X":
            capi.check(ctx.lib.cct_fc_backward(plan, q(x), q(w), q(dy), q(dx), q(dw), q(db), 0, None, 1.0), "backward", ctx.h)
        ctx.sync()
        return y[:B * K], dx[:B * K], dw[:K * K], db[:K]

    apart = run("")
    for _ in range(5):
        assert torch.equal(run("Y over X")[0], apart[0])
        for over in ("dX over dY", "dX over W"):
            for got, want, name in zip(run(over)[1:], apart[1:], ("dX", "dW", "db")):
                assert torch.equal(got, want), (over, name)
    ctx.lib.cct_fc_plan_destroy(plan)
    for got, ref, name in zip(apart, ((X.double() @ W.double().T + b.double()).clamp(min=0), dY.double() @ W.double(),
                                      dY.double().T @ X.double(), dY.double().sum(0)), ("Y", "dX", "dW", "db")):
        assert_close(got.cpu().numpy(), ref.float().view(-1).cpu().numpy(), name)


# Operands four bytes off a 16-byte boundary, which no tensor map describes: all of them, or one at a time, with feature counts
# that are and are not multiples of four, above the size of the fp32 kernel.  Tolerance as above.
@pytest.mark.parametrize("B,K,o", [(129, 772, 1027), (129, 770, 1028), (130, 1024, 512), (40, 2051, 1030)])
@pytest.mark.parametrize("shifted", ["X", "W", "dY", "X W dY dX dW Y"])
def test_inner_product_alignment(ctx, B, K, o, shifted):
    rng = np.random.default_rng(B + K + o)
    sizes = {"X": (B, K), "W": (o, K), "b": (1, o), "dY": (B, o), "Y": (B, o), "dX": (B, K), "dW": (o, K), "db": (1, o)}
    host, base, ptr = {}, {}, {}
    for name, sh in sizes.items():
        host[name] = rng.standard_normal(sh).astype(np.float32)
        shift = 1 if name in shifted.split() else 0
        base[name] = LogicalCube.from_numpy(ctx, np.concatenate([np.full(shift, 7, np.float32), host[name].ravel(), np.full(3, 7, np.float32)]))
        ptr[name] = base[name].ptr + 4 * shift
    plan = C.c_void_p()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, ptr["X"], ptr["W"], ptr["b"], ptr["Y"], 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, ptr["X"], ptr["W"], ptr["dY"], ptr["dX"], ptr["dW"], ptr["db"], 0, None, 1.0),
               "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    X, W, dY = (host[n].astype(np.float64) for n in ("X", "W", "dY"))
    for name, r in (("Y", X @ W.T + host["b"]), ("dX", dY @ W), ("dW", dY.T @ X), ("db", dY.sum(0)[None])):
        shift = 1 if name in shifted.split() else 0
        got = base[name].download().ravel()
        assert_close(got[shift:shift + r.size].reshape(r.shape), r.astype(np.float32), name)
        assert np.all(got[:shift] == 7) and np.all(got[shift + r.size:] == 7)  # nothing beside the output


def test_inner_product_of_many_rows_off_the_boundary(ctx):
    """More row tiles than a grid has in y, in the kernel that takes an X off a 16-byte boundary.  Tolerance: parity (dW adds
    2 097 169 / 8 rounded products per chain: 2^-25 sqrt(n / 2) of the sum, 1.1e-5)."""
    B, K, o = 65536 * 32 + 17, 8, 12
    gen = torch.Generator(device="cuda").manual_seed(3)
    make = lambda n: torch.empty(n, device="cuda").uniform_(-1, 1, generator=gen)  # noqa: E731
    X, W, b, dY = make(B * K + 1)[1:], make(o * K), make(o), make(B * o)
    Y, dX, dW, db = torch.zeros(B * o, device="cuda"), torch.zeros(B * K, device="cuda"), torch.zeros_like(W), torch.zeros_like(b)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    Xd, Wd, dYd = X.double().view(B, K), W.double().view(o, K), dY.double().view(B, o)
    for got, ref, name in ((Y, Xd @ Wd.T + b.double(), "Y"), (dX, dYd @ Wd, "dX"), (dW, dYd.T @ Xd, "dW"), (db, dYd.sum(0), "db")):
        assert_close(got.cpu().numpy(), ref.float().flatten().cpu().numpy(), name)


# More than 2^31 elements in X and dX, more than 2^32 in W and dW.  Tolerance: parity (dW for the second only: its reduction over
# the batch is one chain, whose truncation alone is 2e-3 after 270 000 images).
@pytest.mark.parametrize("B,K,o", [(270000, 8192, 16), (4, 65536, 66000)])
def test_inner_product_beyond_32_bits(ctx, B, K, o):
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB")
    gen = torch.Generator(device="cuda").manual_seed(K)
    make = lambda r, c: torch.empty(r * c, device="cuda").uniform_(-1, 1, generator=gen).view(r, c)  # noqa: E731
    X, W, dY, b = make(B, K), make(o, K), make(B, o), make(1, o)
    Y, dX, dW, db = torch.zeros_like(dY), torch.zeros_like(X), torch.zeros_like(W), torch.zeros_like(b)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    rows, outs = sorted({0, 1, B // 2, B - 1}), sorted({0, 1, o // 2, o - 1})  # 64-bit products of some rows, the last among them
    Xd, Wd, dYd = X[rows].double(), W[outs].double(), dY[rows].double()
    checks = [(Y[rows][:, outs], Xd @ Wd.T + b[0, outs].double(), "Y"),
              (dX[rows], sum(dYd[:, j:j + 4096] @ W[j:j + 4096].double() for j in range(0, o, 4096)), "dX")]
    if B < 1000:
        checks.append((dW[outs], dY[:, outs].double().T @ X.double(), "dW"))
    for got, ref, name in checks:
        assert_close(got.cpu().numpy(), ref.float().cpu().numpy(), name)


def test_sgd_in_one_launch_equals_one_launch_per_tensor(ctx):
    """Bit for bit, over tails, chunks of one tensor that end inside a vector, and buffers off a 16-byte boundary."""
    rng = np.random.default_rng(5)
    items, cubes = (capi.SgdItem * 6)(), []
    for i, (n, shift, lam) in enumerate([(1, 0, 0.0), (7, 1, 5e-4), (4096, 0, 5e-4), (4099, 0, 0.0), (100003, 0, 5e-4), (70001, 3, 5e-4)]):
        values = [rng.standard_normal(n + shift).astype(np.float32) for _ in range(3)]
        pair = [[LogicalCube.from_numpy(ctx, v.reshape(1, -1, 1, 1)) for v in values] for _ in range(2)]
        one, many = ([c.ptr + 4 * shift for c in cs] for cs in pair)
        capi.check(ctx.lib.cct_sgd_step(ctx.h, n, vp(one[0]), vp(one[1]), vp(one[2]), 0.01, 0.9, lam), "sgd", ctx.h)
        items[i] = capi.SgdItem(n, many[0], many[1], many[2], 0.01, 0.9, lam)
        cubes.append(pair)
    capi.check(ctx.lib.cct_sgd_step_multi(ctx.h, 6, items), "sgd multi", ctx.h)
    ctx.sync()
    for one, many in cubes:
        for a, b in zip(one, many):
            assert np.array_equal(a.download(), b.download())


# Strips of windows and of 2 x 2 blocks: planes smaller than a strip, strips that are cut off, odd and even planes.
@pytest.mark.parametrize("B,D,n,k,s", [(1, 1, 3, 3, 2), (2, 3, 4, 3, 2), (3, 5, 8, 3, 2), (1, 7, 23, 3, 2), (5, 17, 13, 3, 2),
                                       (1, 3, 2, 2, 2), (3, 5, 7, 2, 2), (2, 9, 24, 2, 2)])
def test_pooling_planes(ctx, port, B, D, n, k, s):
    m = (n - k) // s + 1
    rng = np.random.default_rng(n)
    A = rng.integers(-3, 4, (B, D, n, n)).astype(np.float32)  # many equal values: the first maximum has to win
    dP = rng.standard_normal((B, D, m, m)).astype(np.float32)
    Yr, idxr = port.maxpool_forward(A, k, s)
    cA, cdP = LogicalCube.from_numpy(ctx, A), LogicalCube.from_numpy(ctx, dP)
    cY, cI, cdA = LogicalCube(ctx, m, m, D, B), LogicalCube(ctx, m, m, D, B), LogicalCube(ctx, n, n, D, B)
    capi.check(ctx.lib.cct_maxpool_forward(ctx.h, vp(cA.ptr), vp(cY.ptr), vp(cI.ptr), B * D, n, k, s), "pool fwd", ctx.h)
    capi.check(ctx.lib.cct_maxpool_backward(ctx.h, vp(cdP.ptr), vp(cI.ptr), vp(cdA.ptr), B * D, n, k, s), "pool bwd", ctx.h)
    ctx.sync()
    assert np.array_equal(cY.download(), Yr) and np.array_equal(cI.download().view(np.int32), idxr.reshape(B, D, m, m))
    assert np.array_equal(cdA.download(), port.maxpool_backward(dP, idxr, n))


def test_normalisation_with_subnormal_powers(ctx):
    """scale^-beta below 2^-126 times a large x: the product is an ordinary number.  Tolerance: the exponent -beta log2(scale), up
    to 130 in fp32, is off by up to 130 * 2^-23 = 1.6e-5 (relative error ln 2 of that), a subnormal power keeps 18 bits or more:
    below 1e-4."""
    B, D, n, alpha, beta = 1, 24, 4, 1.0, 1.3
    X = np.zeros((B, D, n, n), np.float32)
    X[0, ::8] = np.float32(10.0) ** np.linspace(14.0, 15.6, n * n, dtype=np.float32).reshape(n, n)
    x = X.astype(np.float64)
    pad = np.pad(x * x, ((0, 0), (2, 2), (0, 0), (0, 0)))
    scale = 1 + alpha / 5 * sum(pad[:, j:j + D] for j in range(5))
    power = scale ** -beta
    assert (power < 2.0 ** -126).any() and (power > 2.0 ** -132).all()
    cX, cY = LogicalCube.from_numpy(ctx, X), LogicalCube(ctx, n, n, D, B)
    capi.check(ctx.lib.cct_lrn_forward(ctx.h, cX.ptr, cY.ptr, None, B, D, n * n, 5, alpha, beta), "lrn fwd", ctx.h)
    ctx.sync()
    got, want = cY.download()[0, ::8], (x * power)[0, ::8]
    assert np.max(np.abs(got - want) / want) < 1e-4


@pytest.mark.parametrize("B,classes", [(1, 1), (1, 2), (7, 1024), (5, 1025), (3, 4001), (63, 1000), (64, 40), (65, 40), (33, 1030), (1030, 1030)])
def test_softmax_class_counts(ctx, B, classes):
    """Tolerance: parity's 1e-4 against the fp32 sums' (classes + B) * 2^-24 < 3e-4 of terms that are positive, in practice 1e-6."""
    rng = np.random.default_rng(classes)
    X = (3 * rng.standard_normal((B, classes, 1, 1))).astype(np.float32)
    labels = rng.integers(0, classes, B).astype(np.float32)
    pr, lr, gr = pyoracle.np_softmax_loss(X, labels, scale=1.0 / B)
    cX, cL = LogicalCube.from_numpy(ctx, X), LogicalCube.from_numpy(ctx, labels.reshape(B, 1, 1, 1))
    cP, cG, cIL, cLoss = (LogicalCube(ctx, 1, 1, d, b) for d, b in ((classes, B), (classes, B), (1, B), (1, 1)))
    for _ in range(2):
        capi.check(ctx.lib.cct_softmax_loss_forward(ctx.h, vp(cX.ptr), vp(cL.ptr), vp(cP.ptr), vp(cIL.ptr), vp(cLoss.ptr), B,
                                                    classes), "softmax fwd", ctx.h)
        capi.check(ctx.lib.cct_softmax_loss_backward(ctx.h, vp(cP.ptr), vp(cL.ptr), vp(cG.ptr), B, classes, 1.0 / B),
                   "softmax bwd", ctx.h)
        ctx.sync()
        assert_close(cP.download(), pr, "probabilities")
        assert abs(float(cLoss.download().reshape(-1)[0]) - lr) <= 1e-4 * abs(lr) + 1e-6
        assert_close(cG.download(), gr, "gradient")


@pytest.mark.parametrize("B", [64, 3000])
def test_losses_beside_one_another(B):
    """Two calls of one context, captured into graphs and replayed on two streams at once: each gives its own sum."""
    from caffecontroll_b200 import Context
    C_, streams = 1000, [torch.cuda.Stream() for _ in range(2)]
    own = Context(0, stream=streams[0].cuda_stream)
    gen = torch.Generator(device="cuda").manual_seed(B)
    graphs, losses, want = [], [], []
    for i in range(2):
        X = 3 * torch.randn((B, C_), generator=gen, device="cuda")
        labels = torch.randint(0, C_, (B,), generator=gen, device="cuda").float()
        prob, image, loss = torch.zeros_like(X), torch.zeros(B, device="cuda"), torch.zeros(1, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            for _ in range(20):
                capi.check(own.lib.cct_softmax_loss_forward(own.h, X.data_ptr(), labels.data_ptr(), prob.data_ptr(), image.data_ptr(),
                                                            loss.data_ptr(), B, C_), "softmax", own.h)
        graphs.append((g, X, labels, prob, image))
        losses.append(loss)
        want.append(float(torch.nn.functional.cross_entropy(X.double(), labels.long(), reduction="sum")))
    for _ in range(20):
        for i in range(2):
            losses[i].fill_(-1)
        torch.cuda.synchronize()
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                graphs[i][0].replay()
        torch.cuda.synchronize()
        for i in range(2):
            assert abs(float(losses[i]) - want[i]) <= 1e-4 * want[i]
    own.close()


def small_network(ctx):
    from caffecontroll_b200.net import Net, parse_prototxt, solver_from_message
    from tests.test_net_gpu import B, NET, SOLVER
    net_param, solver = parse_prototxt(NET.replace("dropout_ratio: 0.5", "dropout_ratio: 0.4")), solver_from_message(parse_prototxt(SOLVER))
    rng = np.random.default_rng(3)
    net = Net(ctx, net_param, solver, B, fuse=True)
    data = [(rng.standard_normal((B, 3, 67, 67)).astype(np.float32), rng.integers(0, 12, B).astype(np.float32)) for _ in range(2)]
    net.set_input(*data[0])
    return net, data


def graph_launches(ctx, net):
    n = C.c_ulonglong()
    capi.check(ctx.lib.cct_program_graph_launches(net._program, C.byref(n)), "cct_program_graph_launches", ctx.h)
    return n.value


def parameters(net):
    net.ctx.sync()
    return [pb.get_model_cube().download() for _, pb in net.param_bridges()]


def test_recorded_step_equals_the_bridges_one_by_one(ctx):
    """Steps through the recorded program (the first walks, the second records its walk, the later ones are graph launches), a
    change of a bridge's switch that has to be noticed, a second recording: the same bits as a network whose bridges are walked
    through."""
    results = []
    for recorded in (True, False):
        net, _ = small_network(ctx)
        for i in range(9):
            if i == 5:
                net.bridges[net.names.index("fc7")].needs_to_calc_backward_grad = False
            if not recorded:
                net.forward()
                net.backward()
                continue
            net.step()
            other = LogicalCube(ctx, 1, 1, 1, 1)  # objects that are not the network's do not matter, nor does an equal value
            other.ptr, net.labels.ptr = other.ptr, net.labels.ptr + 0
            other.free()
            assert (net._program is None) == (i in (0, 5)), i
            if net._program is not None:
                assert graph_launches(ctx, net) == {1: 0, 2: 1, 3: 2, 4: 3, 6: 0, 7: 1, 8: 2}[i]
        results.append(parameters(net))
        net.close()
    for a, b in zip(*results):
        assert np.array_equal(a, b)


def test_steps_that_alternate_between_input_buffers(ctx):
    """A double-buffered loader: the same bits as copying each batch into one buffer, and next to no recordings."""
    results = []
    for alternate in (True, False):
        net, data = small_network(ctx)
        buffers = [tuple(LogicalCube.from_numpy(ctx, a if a.ndim == 4 else a.reshape(-1, 1, 1, 1)) for a in d) for d in data]
        own = net.input.p_data_cube.ptr, net.labels.ptr
        recordings, record = [], net._record
        net._record = lambda: recordings.append(1) or record()
        for i in range(40):
            if alternate:
                net.input.p_data_cube.ptr, net.labels.ptr = (c.ptr for c in buffers[i % 2])
                net.loss_bridge.p_data_labels = net.labels
            else:
                net.set_input(*data[i % 2])
            net.step()
        assert len(recordings) == (5 if alternate else 1)  # at steps 1, 4, 9, 18 and 35, each given up at the next
        results.append(parameters(net))
        net.input.p_data_cube.ptr, net.labels.ptr = own
        net.close()
        for pair in buffers:
            for c in pair:
                c.free()
    for a, b in zip(*results):
        assert np.array_equal(a, b)


def test_replaced_methods_end_a_recording(ctx):
    """What a program replaces on a network that has recorded its calls is called from the next step on."""
    net, _ = small_network(ctx)
    for _ in range(3):
        net.step()
    assert graph_launches(ctx, net) == 1
    calls = []
    name, pb = net.param_bridges()[0]
    backward = pb.backward
    pb.backward = lambda begin_allreduce=True: (calls.append(name), backward(begin_allreduce))
    net.step()
    assert calls == [name] and net._program is None
    del pb.backward
    while net._program is None:
        net.step()
    net.step()
    net.ops.allreduce_begin = lambda ptr, count: calls.append(count)
    net.step()
    assert len(calls) == 1 + len(net.pbridges)
    del net.ops.allreduce_begin
    while net._program is None:
        net.step()
    net.ops.world_size = lambda: 2  # a process group that was set up later
    net.ops.allreduce_begin = lambda ptr, count: calls.append(count)
    net.step()
    assert len(calls) == 1 + 2 * len(net.pbridges) and net._program is None
    net.close()


def test_recording_is_one_threads_own(ctx):
    """While a thread records, another thread's calls on the same context are carried out, and it may record itself."""
    import threading
    from caffecontroll_b200.layers import ReLUBridge
    x = np.linspace(-1, 1, 64, dtype=np.float32).reshape(2, 2, 4, 4)
    mk = lambda v: Layer(LogicalCube.from_numpy(ctx, v), LogicalCube.from_numpy(ctx, 0 * v))  # noqa: E731
    mine, theirs = [(mk(x), mk(7 + 0 * x)) for _ in range(2)]
    relu, other = ReLUBridge(*mine, ctx), ReLUBridge(*theirs, ctx)
    program, failures = C.c_void_p(), []

    def beside():
        try:
            own = C.c_void_p()
            other.forward()
            capi.check(ctx.lib.cct_program_begin(ctx.h, C.byref(own)), "begin", ctx.h)
            other.backward()
            capi.check(ctx.lib.cct_program_end(own), "end", ctx.h)
            ctx.lib.cct_program_destroy(own)
        except Exception as e:
            failures.append(e)

    capi.check(ctx.lib.cct_program_begin(ctx.h, C.byref(program)), "begin", ctx.h)
    relu.forward()
    t = threading.Thread(target=beside)
    t.start()
    t.join()
    capi.check(ctx.lib.cct_program_end(program), "end", ctx.h)
    ctx.sync()
    assert not failures
    assert np.array_equal(theirs[1].p_data_cube.download(), np.maximum(x, 0))
    assert np.all(mine[1].p_data_cube.download() == 7)  # recorded, not carried out
    launches = C.c_ulonglong()
    for run in range(3):
        theirs[1].p_data_cube.upload(7 + 0 * x)
        mine[1].p_data_cube.upload(7 + 0 * x)
        capi.check(ctx.lib.cct_program_run(program), "run", ctx.h)
        ctx.sync()
        assert np.array_equal(mine[1].p_data_cube.download(), np.maximum(x, 0))
        assert np.all(theirs[1].p_data_cube.download() == 7)  # the other thread's call is no part of it
        capi.check(ctx.lib.cct_program_graph_launches(program, C.byref(launches)), "graph launches", ctx.h)
        assert launches.value == run  # the first run call by call
    ctx.lib.cct_program_destroy(program)


# Host-buffer calls that move the batch in slices: a last slice of one image, the kernels that the weight gradient can be, and
# layers of few pixels and many filters, whose data gradient leaves split sums in the buffer that the weight gradient uses too.
@pytest.mark.parametrize("shape", [(17, 3, 47, 24, 11, 4, 0, 1), (33, 6, 31, 40, 5, 1, 2, 1), (16, 64, 9, 48, 3, 1, 1, 1),
                                   (16, 48, 14, 256, 3, 1, 1, 1), (32, 48, 14, 256, 3, 1, 1, 1), (16, 32, 13, 384, 3, 1, 1, 1),
                                   (16, 16, 28, 192, 5, 1, 2, 1), (16, 16, 7, 64, 3, 1, 1, 1), (33, 1, 65, 136, 11, 4, 5, 1),
                                   (19, 14, 16, 208, 5, 1, 0, 1)])
@pytest.mark.parametrize("with_dx", [True, False])
@pytest.mark.parametrize("algo", [capi.ALGO_AUTO, TENSOR])
def test_sliced_host_calls(ctx, port, shape, with_dx, algo):
    B, D, n, o, k, s, p, g = shape
    X, W, b, dY = make_inputs(31, B, D, n, o, k, s, p, g)
    plan = C.c_void_p()
    desc = capi.ConvDesc(B, D, n, o, k, s, p, g, 1, algo)
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "plan", ctx.h)
    Y, dX, dW, db = (np.full_like(a, np.nan) for a in (dY, X, W, b))
    host = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    capi.check(ctx.lib.cct_conv_forward_host(plan, host(X), host(W), host(b), host(Y), 0), "forward", ctx.h)
    dXr, dWr, dbr = port.conv_backward(X, W, dY, k, s, p, g)
    assert_close(Y, port.conv_forward(X, W, b, k, s, p, g).reshape(Y.shape), "Y")
    for _ in range(2):
        for a in (dX, dW, db):
            a.fill(np.nan)
        capi.check(ctx.lib.cct_conv_backward_host(plan, None, None, host(dY), host(dX) if with_dx else None, host(dW), host(db)),
                   "backward", ctx.h)
        for a, r, name in [(dW, dWr, "dW"), (db, dbr, "db")] + ([(dX, dXr, "dX")] if with_dx else []):
            assert_close(a, r.reshape(a.shape), name)
    ctx.lib.cct_conv_plan_destroy(plan)


# At most 32 classes: the largest batch of one block, one more, sums in several pieces; 33 classes: the largest batch of a cluster and one more.
@pytest.mark.parametrize("B,classes", [(1, 32), (31, 10), (128, 32), (129, 32), (2049, 3), (64, 33), (65, 33)])
def test_softmax_of_few_classes(ctx, B, classes):
    test_softmax_class_counts(ctx, B, classes)


# Inner products of the fp32 kernels: one feature, rows that are and are not multiples of four floats or on a 16-byte boundary, tiles of four
# images and outputs that are not full, fewer and more steps of the reduction than a block has warps, a data gradient with and without
# splits; the two gradients in one launch.  Tolerance: n products added in fp32 in any order, n * 2^-24 of the sum of their magnitudes,
# and a few roundings more.
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("B,K,o", [(1, 1, 1), (2, 68, 9), (3, 5, 7), (5, 36, 130), (50, 4096, 10), (64, 500, 10), (33, 127, 257), (4, 60, 1021), (9, 2052, 21),
                                   (13, 1028, 300), (100, 400, 300)])
def test_small_inner_products(ctx, B, K, o, shift):
    gen = torch.Generator(device="cuda").manual_seed(B + K + o)
    make = lambda r, c: torch.randn(r * c + shift, device="cuda", generator=gen)[shift:].view(r, c)  # noqa: E731
    X, W, b, dY = make(B, K), make(o, K), make(1, o), make(B, o)
    keep, keep_in = ((torch.rand(s, device="cuda", generator=gen) < 0.5).int() for s in ((B, o), (B, K)))
    Y, dX, dW, db = torch.zeros_like(dY), torch.zeros_like(X), torch.zeros_like(W), torch.zeros_like(b)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    before = capi.kernel_launches()
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 1, q(keep), 2.0), "forward", ctx.h)
    forward = capi.kernel_launches()
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 1, q(keep_in), 2.0), "backward", ctx.h)
    # (100 images off a 16-byte boundary: too many products for loads of one word, fp32 tiles in three splits)
    assert forward - before == (2 if (B, shift) == (100, 1) else 1) and capi.kernel_launches() - forward == (2 if o >= 256 else 1)
    ctx.sync()
    Xd, Wd, dYd = X.double(), W.double(), dY.double()
    back = keep_in * 2.0 * (X > 0)
    checks = [(Y, (Xd @ Wd.T + b.double()).clamp(min=0) * keep * 2, (Xd.abs() @ Wd.abs().T + b.double().abs()) * 2, K + 2, "Y"),
              (dX, dYd @ Wd * back, dYd.abs() @ Wd.abs() * 2, o + 2, "dX"), (dW, dYd.T @ Xd, dYd.abs().T @ Xd.abs(), B, "dW"),
              (db, dYd.sum(0)[None], dYd.abs().sum(0)[None], B, "db")]
    for got, ref, size, n, name in checks:
        assert torch.all((got.double() - ref).abs() <= (n + 4) * 2.0 ** -24 * size), name
    # an output over an operand: the same bits as apart
    for out, over, call in ((Y, X, lambda t: ctx.lib.cct_fc_forward(plan, q(t), q(W), q(b), q(t), 1, q(keep), 2.0)),
                            (dW, W, lambda t: ctx.lib.cct_fc_backward(plan, q(X), q(t), q(dY), None, q(t), q(db), 0, None, 1.0)),
                            (dX, X, lambda t: ctx.lib.cct_fc_backward(plan, q(t), q(W), q(dY), q(t), q(dW), q(db), 1, q(keep_in), 2.0))):
        if out.numel() <= over.numel():
            both = over.clone()
            torch.cuda.synchronize()
            capi.check(call(both), "over", ctx.h)
            ctx.sync()
            assert torch.equal(both.view(-1)[:out.numel()], out.view(-1))
    ctx.lib.cct_fc_plan_destroy(plan)


# Layers whose passes take different kernels: dot products forward, tensor cores backward (with padded rows too); tensor cores forward, fp32
# tiles backward; fp32 tiles with splits forward.  Rows on and off a 16-byte boundary.  Tolerance: parity.
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("B,K,o", [(1, 4096, 1000), (4, 4093, 1001), (256, 1000, 100), (128, 999, 333), (60, 333, 300)])
def test_inner_products_of_mixed_plans(ctx, B, K, o, shift):
    gen = torch.Generator(device="cuda").manual_seed(B + K + o)
    make = lambda r, c: torch.randn(r * c + shift, device="cuda", generator=gen)[shift:].view(r, c)  # noqa: E731
    X, W, b, dY = make(B, K), make(o, K), make(1, o), make(B, o)
    Y, dX, dW, db = torch.zeros_like(dY), torch.zeros_like(X), torch.zeros_like(W), torch.zeros_like(b)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 0, None, 1.0), "forward", ctx.h)
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    Xd, Wd, dYd = X.double(), W.double(), dY.double()
    for got, ref, name in ((Y, Xd @ Wd.T + b.double(), "Y"), (dX, dYd @ Wd, "dX"), (dW, dYd.T @ Xd, "dW"), (db, dYd.sum(0)[None], "db")):
        assert_close(got.cpu().numpy(), ref.float().cpu().numpy(), name)


# Both sides of the lines of the dot products against routes of two launches: reductions that fill a part of a warp's step, rows off a 16-byte
# boundary with few and with many images, short and long reductions.  Tolerance: parity.
@pytest.mark.parametrize("B,K,o,shift,launches", [(32, 16, 2048, 0, 1), (384, 16, 2048, 0, 2), (64, 512, 500, 0, 1), (64, 512, 500, 1, 2), (64, 512, 700, 1, 2),
                                                  (8, 1024, 1000, 1, 1), (20, 1024, 1000, 1, 2), (128, 1024, 128, 1, 2), (50, 4096, 10, 1, 1),
                                                  (32, 2100, 130, 1, 1), (4, 4096, 1000, 1, 1), (8, 2100, 1250, 0, 1), (8, 2101, 1250, 0, 1)])
def test_lines_of_the_dot_products(ctx, B, K, o, shift, launches):
    gen = torch.Generator(device="cuda").manual_seed(B + K + o)
    make = lambda r, c: torch.randn(r * c + shift, device="cuda", generator=gen)[shift:].view(r, c)  # noqa: E731
    X, W, b, Y = make(B, K), make(o, K), make(1, o), make(B, o)
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    before = capi.kernel_launches()
    capi.check(ctx.lib.cct_fc_forward(plan, q(X), q(W), q(b), q(Y), 0, None, 1.0), "forward", ctx.h)
    assert capi.kernel_launches() - before == launches
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    assert_close(Y.cpu().numpy(), (X.double() @ W.double().T + b.double()).float().cpu().numpy(), "Y")


# Both sides of the line between one launch and two for both contractions on the tensor cores, in one round of tiles and in more.  Tolerance: parity.
@pytest.mark.parametrize("B,K,o,launches", [(128, 4096, 256, 2), (128, 4096, 512, 3), (64, 4096, 512, 2), (64, 3136, 1000, 3), (128, 6272, 512, 2), (128, 5436, 400, 2),
                                            (128, 6272, 552, 3)])
def test_lines_of_the_merged_launch(ctx, B, K, o, launches):
    test_backward_passes_of_long_batches(ctx, B, K, o, launches)


# Both sides of the line between the fp32 tiles and the tensor cores in backward passes of layers that are not small: a batch that makes one
# block's chain long, blocks for every SM several times over.  Tolerance: parity.
@pytest.mark.parametrize("B,K,o,launches", [(256, 784, 128, 1), (640, 1000, 100, 3), (4096, 784, 128, 3), (8192, 64, 512, 1), (1024, 256, 256, 1)])
def test_backward_passes_of_long_batches(ctx, B, K, o, launches):
    gen = torch.Generator(device="cuda").manual_seed(B + K + o)
    make = lambda r, c: torch.randn(r, c, device="cuda", generator=gen)  # noqa: E731
    X, W, dY = make(B, K), make(o, K), make(B, o)
    dX, dW, db = torch.zeros_like(X), torch.zeros_like(W), torch.zeros(o, device="cuda")
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    before = capi.kernel_launches()
    capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
    assert capi.kernel_launches() - before == launches
    ctx.sync()
    ctx.lib.cct_fc_plan_destroy(plan)
    for got, ref, name in ((dX, dY.double() @ W.double(), "dX"), (dW, dY.double().T @ X.double(), "dW"), (db, dY.double().sum(0), "db")):
        assert_close(got.cpu().numpy(), ref.float().cpu().numpy(), name)


# Both gradients of a small layer with stride 1 in one launch and, where dX lies over X, one after the other.  Tolerance: parity (fp32
# products, sums of at most 24 x 25 and 36 864 of them).
@pytest.mark.parametrize("shape", [(5, 1, 9, 7, 5, 1, 0, 1), (6, 2, 11, 24, 3, 1, 1, 2), (3, 8, 10, 5, 1, 1, 0, 1), (2, 3, 13, 9, 7, 1, 3, 1),
                                   (64, 1, 28, 20, 5, 1, 0, 1), (4, 12, 8, 16, 3, 1, 1, 1)])
def test_small_gradients_in_one_launch(ctx, shape):
    B, D, n, o, k, s, p, g = shape
    m = (n + 2 * p - k) // s + 1
    gen = torch.Generator(device="cuda").manual_seed(o)
    X, W, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, D, n, n), (o, D // g, k, k), (B, o, m, m)))
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    desc = capi.ConvDesc(B, D, n, o, k, s, p, g, 1, capi.ALGO_AUTO)
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "plan", ctx.h)

    def run(x, w, dx, dw):
        db = torch.zeros(o, device="cuda")
        torch.cuda.synchronize()
        before = capi.kernel_launches()
        capi.check(ctx.lib.cct_conv_backward(plan, q(x), q(w), q(dY), q(dx), q(dw), q(db)), "backward", ctx.h)
        ctx.sync()
        return dx, dw, db, capi.kernel_launches() - before

    dX, dW, db, launches = run(X, W, torch.zeros_like(X), torch.zeros_like(W))
    assert launches == 2
    x = X.clone()
    over = run(x, W, x, torch.zeros_like(W))
    ctx.lib.cct_conv_plan_destroy(plan)
    assert over[3] == 3 and torch.equal(over[1], dW) and torch.equal(over[2], db)
    Xd, Wd = X.double().requires_grad_(), W.double().requires_grad_()
    torch.nn.functional.conv2d(Xd, Wd, None, s, p, 1, g).backward(dY.double())
    for got, ref, name in ((dX, Xd.grad, "dX"), (over[0], Xd.grad, "dX over X"), (dW, Wd.grad, "dW"), (db, dY.double().sum((0, 2, 3)), "db")):
        assert_close(got.cpu().numpy(), ref.float().cpu().numpy(), name)


# Both contractions of a backward pass in one launch of the tensor-core kernel: a slot for every tile and up to two tiles a slot, one output
# tile, outputs that no tensor map describes, and the sum of dY where there is a bias; dX over X: one launch more.  Tolerance: parity.
@pytest.mark.parametrize("B,K,o,bias", [(64, 800, 500, 1), (16, 2048, 1000, 0), (128, 516, 512, 1), (40, 2051, 1030, 1), (1, 1300, 1028, 0)])
def test_two_contractions_in_one_launch(ctx, B, K, o, bias):
    gen = torch.Generator(device="cuda").manual_seed(B + K + o)
    make = lambda r, c: torch.randn(r, c, device="cuda", generator=gen)  # noqa: E731
    X, W, dY, keep = make(B, K), make(o, K), make(B, o), (torch.rand(B, K, device="cuda", generator=gen) < 0.5).int()
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, bias, C.byref(plan)), "plan", ctx.h)

    def run(x, dx):
        dW, db = torch.zeros_like(W), torch.zeros(o, device="cuda")
        torch.cuda.synchronize()
        before = capi.kernel_launches()
        capi.check(ctx.lib.cct_fc_backward(plan, q(x), q(W), q(dY), q(dx), q(dW), q(db), 1, q(keep), 2.0), "backward", ctx.h)
        ctx.sync()
        return dx, dW, db, capi.kernel_launches() - before

    dX, dW, db, launches = run(X, torch.zeros_like(X))
    x = X.clone()
    over = run(x, x)
    ctx.lib.cct_fc_plan_destroy(plan)
    pads = 2 * (K % 4 != 0) + (o % 4 != 0)
    assert launches == 2 + pads and over[3] == 3 + pads
    Xd, Wd, dYd = X.double(), W.double(), dY.double()
    refs = [(dYd @ Wd) * keep * 2 * (X > 0), dYd.T @ Xd] + [dYd.sum(0)] * bias
    for got in ((dX, dW, db), over):
        for a, r, name in zip(got, refs, ("dX", "dW", "db")):
            assert_close(a.cpu().numpy(), r.float().cpu().numpy(), name)


@pytest.fixture(scope="session")
def keep_sms(ctx, tmp_path_factory):
    """keep_sms(n): launches leave n SMs free from now on, as while a gradient reduction is in flight."""
    at = tmp_path_factory.mktemp("keep")
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caffecontroll_b200", "csrc")
    (at / "keep.cu").write_text('#include "%s/cct_internal.h"\nextern "C" void keep(cct_ctx* ctx, int sms) { ctx->reserved_sms = sms; }\n' % csrc)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-o", str(at / "keep.so"), str(at / "keep.cu")], check=True)
    lib = C.CDLL(str(at / "keep.so"))
    lib.keep.argtypes = [C.c_void_p, C.c_int]
    return lambda n: lib.keep(ctx.h, n)


def kernels_of(ctx, call):
    """Names of the library's kernels that a call launches, template arguments included."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        ctx.sync()
    names = [re.match(r"(?:void )?(\w+(?:<[^(]*>)?)\(", e.name.replace("(anonymous namespace)::", "")) for e in prof.events()]
    return [n.group(1) for n in names if n]


# gather_conv_kernel<SETS, MODE, ONE> with a CTA per tile (ONE) by tap and by run of channels, two and four producer sets, with and without
# splits, strides and groups; the last slot and one tile past it; 32 k-blocks and 33; wgrad_kernel<M-tiles, ...> with one M-tile per CTA where more
# would fit, and with two.  Persistent (all SMs but one kept), the same bits; tolerance against float64: parity.
@pytest.mark.parametrize("shape,forward,weight,data", [
    ((37, 50, 21, 75, 3, 2, 1, 1), "<2, 0, true>", "<1, 5>", "<2, 0, true>"), ((1, 256, 13, 384, 3, 1, 1, 1), "<2, 1, true>", None, "<2, 1, true>"),
    ((1, 96, 27, 256, 5, 1, 2, 2), "<2, 1, true>", None, "<2, 1, true>"), ((9, 17, 33, 65, 3, 1, 1, 1), "<2, 0, true>", "<2, 5>", "<2, 0, true>"),
    ((74, 32, 16, 130, 3, 1, 1, 1), "<4, 1, true>", "<2, 9>", "<2, 0, false>"), ((75, 32, 16, 130, 3, 1, 1, 1), "<2, 1, false>", "<2, 9>", "<2, 0, false>"),
    ((74, 31, 16, 130, 3, 1, 1, 1), "<4, 0, true>", "<2, 9>", "<2, 0, false>"), ((4, 100, 29, 300, 5, 1, 1, 1), "<4, 0, true>", None, "<4, 0, false>"),
    ((38, 96, 10, 300, 5, 1, 1, 1), "<4, 1, true>", None, "<4, 0, false>"), ((52, 33, 31, 40, 3, 2, 1, 1), "<2, 0, true>", None, "<4, 1, true>"),
    ((58, 64, 7, 17, 1, 2, 0, 1), "<2, 1, true>", "<1, 2>", "<2, 0, true>"), ((2, 33, 17, 300, 3, 1, 1, 1), "<2, 0, true>", "<1, 10>", "<2, 0, true>"),
    ((78, 64, 21, 8, 3, 2, 1, 1), "<2, 1, true>", None, "<2, 1, true>"), ((148, 64, 21, 8, 3, 2, 1, 1), "<2, 1, true>", None, "<2, 1, false>"),
    ((48, 256, 13, 51, 3, 2, 1, 1), "<2, 1, true>", None, "<4, 0, false>"), ((32, 16, 31, 24, 11, 4, 2, 1), "<2, 1, true>", None, "<2, 1, true>"),
    ((64, 16, 31, 24, 11, 4, 2, 1), "<2, 1, true>", None, "<2, 1, false>"),
    ((37, 1024, 16, 130, 1, 1, 0, 1), "<2, 1, true>", None, "<2, 0, false>"), ((37, 1056, 16, 130, 1, 1, 0, 1), "<2, 1, false>", None, "<4, 0, false>"),
])
def test_a_cta_per_tile(ctx, keep_sms, shape, forward, weight, data):
    B, D, n, o, k, s, p, g = shape
    m = (n + 2 * p - k) // s + 1
    gen = torch.Generator(device="cuda").manual_seed(D)
    X, W, b, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, D, n, n), (o, D // g, k, k), (o,), (B, o, m, m)))
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    desc = capi.ConvDesc(B, D, n, o, k, s, p, g, 1, TENSOR)
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "plan", ctx.h)

    def run():
        Y, dX, dW, db = (torch.full_like(t, 7) for t in (dY, X, W, b))
        torch.cuda.synchronize()
        there = kernels_of(ctx, lambda: capi.check(ctx.lib.cct_conv_forward(plan, q(X), q(W), q(b), q(Y), 1), "forward", ctx.h))
        back = kernels_of(ctx, lambda: capi.check(ctx.lib.cct_conv_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db)), "backward", ctx.h))
        last = [name for name in back if name.startswith("gather_conv_kernel")][-1]
        return (Y, dX, dW, db), ["".join(x for x in there if x.startswith("gather_conv")), "".join(x for x in back if x.startswith("wgrad_kernel")), last]

    got, names = run()
    assert names[0] == "gather_conv_kernel" + forward and names[2] == "gather_conv_kernel" + data
    assert weight is None or names[1] == "wgrad_kernel" + weight
    keep_sms(torch.cuda.get_device_properties(0).multi_processor_count - 1)
    try:
        kept, kept_names = run()
    finally:
        keep_sms(0)
    ctx.lib.cct_conv_plan_destroy(plan)
    assert "true" not in kept_names[0] + kept_names[2]
    Xd, Wd, bd = (t.double().requires_grad_() for t in (X, W, b))
    out = torch.nn.functional.conv2d(Xd, Wd, bd, s, p, 1, g)
    out.backward(dY.double())
    for a, c, r, name in zip(got, kept, (out.detach().clamp(min=0), Xd.grad, Wd.grad, bd.grad), ("Y", "dX", "dW", "db")):
        assert torch.equal(a, c), name
        assert_close(a.cpu().numpy(), r.float().cpu().numpy(), name)


def test_two_contractions_beside_a_reduction(ctx, keep_sms):
    """Both contractions of an inner product's backward pass with fewer SMs: in one launch where there are at most two tiles a slot, else in two;
    the same bits."""
    B, K, o = 64, 800, 500
    gen = torch.Generator(device="cuda").manual_seed(9)
    X, W, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, K), (o, K), (B, o)))
    plan, q, results = C.c_void_p(), lambda t: t.data_ptr(), []
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_fc_plan_create(ctx.h, B, K, o, 1, C.byref(plan)), "plan", ctx.h)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for kept, launches in ((0, 2), (8, 2), (sms - 40, 2), (sms - 4, 3), (sms - 1, 3)):
        dX, dW, db = torch.zeros_like(X), torch.zeros_like(W), torch.zeros(o, device="cuda")
        torch.cuda.synchronize()
        before = capi.kernel_launches()
        keep_sms(kept)
        try:
            capi.check(ctx.lib.cct_fc_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db), 0, None, 1.0), "backward", ctx.h)
        finally:
            keep_sms(0)
        ctx.sync()
        assert capi.kernel_launches() - before == launches, kept
        results.append((dX, dW, db))
    ctx.lib.cct_fc_plan_destroy(plan)
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    for a, r, name in zip(results[0], (dY.double() @ W.double(), dY.double().T @ X.double(), dY.double().sum(0)), ("dX", "dW", "db")):
        assert_close(a.cpu().numpy(), r.float().cpu().numpy(), name)


# One-channel data gradients of 5 x 5 windows: four and eight rows per lane on both sides of one lot of four for every SM, planes that end inside
# a lane's rows, alone and beside the weight gradient.  Tolerance: parity.
@pytest.mark.parametrize("shape,rows,launches", [
    ((1, 1, 28, 20, 5, 1, 0, 1), 4, 2), ((64, 1, 28, 20, 5, 1, 0, 1), 8, 2), ((128, 1, 12, 32, 5, 1, 0, 1), 4, 3), ((16, 1, 40, 32, 5, 1, 0, 1), 8, 3),
    ((64, 1, 28, 32, 5, 1, 0, 1), 8, 2), ((128, 1, 28, 20, 5, 1, 2, 1), 4, 3), ((64, 1, 32, 32, 5, 1, 2, 1), 8, 3), ((118, 1, 6, 42, 5, 1, 2, 1), 4, 3), ((64, 1, 32, 8, 5, 1, 2, 1), 8, 3),
])
def test_rows_of_one_channel(ctx, shape, rows, launches):
    B, D, n, o, k, s, p, g = shape
    m = n + 2 * p - k + 1
    gen = torch.Generator(device="cuda").manual_seed(n + o)
    X, W, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, D, n, n), (o, D, k, k), (B, o, m, m)))
    dX, dW, db = torch.full_like(X, 7), torch.zeros_like(W), torch.zeros(o, device="cuda")
    plan, q = C.c_void_p(), lambda t: t.data_ptr()
    desc = capi.ConvDesc(B, D, n, o, k, s, p, g, 1, capi.ALGO_AUTO)
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "plan", ctx.h)
    names = kernels_of(ctx, lambda: capi.check(ctx.lib.cct_conv_backward(plan, q(X), q(W), q(dY), q(dX), q(dW), q(db)), "backward", ctx.h))
    ctx.lib.cct_conv_plan_destroy(plan)
    mine = [name for name in names if name.startswith("small_conv_kernel")]
    assert len(names) == launches and len(mine) == 1 and mine[0].endswith(", %d>" % rows), names
    Xd, Wd = X.double().requires_grad_(), W.double().requires_grad_()
    torch.nn.functional.conv2d(Xd, Wd, None, s, p).backward(dY.double())
    for got, ref, name in ((dX, Xd.grad, "dX"), (dW, Wd.grad, "dW"), (db, dY.double().sum((0, 2, 3)), "db")):
        assert_close(got.cpu().numpy(), ref.float().cpu().numpy(), name)


# The data gradient of a small layer beside its weight gradient, in a launch of its own with the timing switched on, and over X, from few channels for
# eight warps to more than two a warp: the same bits.
@pytest.mark.parametrize("shape", [(16, 6, 30, 12, 3, 1, 1, 1), (3, 8, 10, 5, 1, 1, 0, 1), (5, 1, 9, 7, 5, 1, 0, 1), (6, 2, 11, 24, 3, 1, 1, 2), (64, 1, 28, 20, 5, 1, 0, 1),
                                   (2, 3, 13, 9, 7, 1, 3, 1), (4, 12, 8, 4, 3, 1, 1, 1), (4, 12, 8, 3, 3, 1, 1, 1), (8, 7, 18, 23, 5, 1, 2, 1)])
def test_small_data_gradients_alone_and_in_company(ctx, shape):
    B, D, n, o, k, s, p, g = shape
    m = n + 2 * p - k + 1
    gen = torch.Generator(device="cuda").manual_seed(o)
    X, W, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, D, n, n), (o, D // g, k, k), (B, o, m, m)))
    plan, q, results = C.c_void_p(), lambda t: t.data_ptr(), []
    desc = capi.ConvDesc(B, D, n, o, k, s, p, g, 1, capi.ALGO_AUTO)
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "plan", ctx.h)
    for timed, over in ((0, False), (1, False), (0, True)):
        capi.check(ctx.lib.cct_conv_plan_enable_timing(plan, timed), "timing", ctx.h)
        x = X.clone()
        dX, dW, db = x if over else torch.zeros_like(X), torch.zeros_like(W), torch.zeros(o, device="cuda")
        torch.cuda.synchronize()
        before = capi.kernel_launches()
        capi.check(ctx.lib.cct_conv_backward(plan, q(x), q(W), q(dY), q(dX), q(dW), q(db)), "backward", ctx.h)
        ctx.sync()
        assert capi.kernel_launches() - before == (3 if timed or over else 2)
        results.append((dX, dW, db))
    ctx.lib.cct_conv_plan_destroy(plan)
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
