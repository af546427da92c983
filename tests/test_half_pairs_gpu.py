"""Contractions whose operands are split into pairs of fp16 (the larger ones): each form of the kernel against 64-bit sums, the scale at its limits,
operands that are not split so, values that are not finite, rows of gradients whose ends lie inside a word."""
import ctypes as C

import numpy as np
import pytest
import torch

from caffecontroll_b200 import capi

pytestmark = pytest.mark.gpu

TENSOR = 2


class Layer:
    """A convolution of the tensor cores on torch's memory; every call waits for the device."""

    def __init__(self, ctx, shape):
        self.ctx, self.shape = ctx, shape
        B, D, n, o, k, s, p, g = shape
        self.m = (n + 2 * p - k) // s + 1
        self.plan = C.c_void_p()
        capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(capi.ConvDesc(B, D, n, o, k, s, p, g, 1, TENSOR)), C.byref(self.plan)), "plan", ctx.h)

    def close(self):
        self.ctx.lib.cct_conv_plan_destroy(self.plan)

    def operands(self, seed, positive=False):
        B, D, n, o, k, s, p, g = self.shape
        gen = torch.Generator(device="cuda").manual_seed(seed)
        X, dY = (torch.randn(sh, device="cuda", generator=gen) for sh in ((B, D, n, n), (B, o, self.m, self.m)))
        W, b = 0.02 * torch.randn((o, D // g, k, k), device="cuda", generator=gen), torch.randn(o, device="cuda", generator=gen)
        return (X.abs(), W.abs(), b, dY.abs()) if positive else (X, W, b, dY)

    def forward(self, X, W, b):
        Y = torch.full((X.shape[0], W.shape[0], self.m, self.m), 7.0, device="cuda")
        torch.cuda.synchronize()
        capi.check(self.ctx.lib.cct_conv_forward(self.plan, X.data_ptr(), W.data_ptr(), b.data_ptr(), Y.data_ptr(), 0), "forward", self.ctx.h)
        self.ctx.sync()
        return Y

    def backward(self, X, W, dY):
        dX, dW, db = torch.full_like(X, 7), torch.full_like(W, 7), torch.full((W.shape[0],), 7.0, device="cuda")
        torch.cuda.synchronize()
        capi.check(self.ctx.lib.cct_conv_backward(self.plan, X.data_ptr(), W.data_ptr(), dY.data_ptr(), dX.data_ptr(), dW.data_ptr(), db.data_ptr()),
                   "backward", self.ctx.h)
        self.ctx.sync()
        return dX, dW, db

    def exact(self, X, W, b, dY):
        _, _, _, _, _, s, p, g = self.shape
        X, W, dY = X.double(), W.double(), dY.double()
        return (torch.nn.functional.conv2d(X, W, b.double(), s, p, 1, g), torch.nn.grad.conv2d_input(X.shape, W, dY, s, p, 1, g),
                torch.nn.grad.conv2d_weight(X, W.shape, dY, s, p, 1, g), dY.sum((0, 2, 3)))


@pytest.fixture
def layer(ctx):
    made = []

    def make(shape):
        made.append(Layer(ctx, shape))
        return made[-1]
    yield make
    for one in made:
        one.close()


def off(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


def bound(products):
    """Three instructions per 16 products, each of which cuts the sum by 1.5 places of 0.72 * 2^-24 on average (see test_accumulation_error; four times
    that), and the split: 2^-22 of a value cut, 2^-24 rounded, for two operands, and lo * lo left out (2^-20): below 2^-19."""
    return 4 * 6 * (products // 32 + 1) * 2.0 ** -23.9 / 2 + 2.0 ** -19


def launches(ctx, call):
    count = [C.c_ulonglong(), C.c_ulonglong()]
    ctx.lib.cct_kernel_launches(C.byref(count[0]))
    call()
    ctx.lib.cct_kernel_launches(C.byref(count[1]))
    return count[1].value - count[0].value


# Runs of eight channels and single ones; one and two CTAs per SM; groups; strides; odd images (rows of gradients that end inside a word and
# a block of 32); reductions that are no multiple of 32; split reductions.  Launches: the look at the operands, packing, contraction and the sum of
# its splits; the look, the split of dY, contraction, sums and packing, contraction and the sum of its splits.
@pytest.mark.parametrize("shape,forward,backward", [
    ((67, 256, 13, 384, 3, 1, 1, 1), (3, 4), (5, 6)), ((67, 250, 17, 300, 3, 1, 1, 1), (3, 4), (5, 6)), ((64, 96, 27, 256, 5, 1, 2, 2), (3,), (4, 5, 6, 7)),
    ((50, 192, 31, 320, 3, 2, 1, 1), (2, 3, 4), (5,)), ((64, 384, 13, 384, 3, 1, 1, 2), (3,), (5,)), ((25, 120, 41, 160, 5, 1, 2, 1), (3, 4), (5, 6)),
    ((64, 1024, 27, 600, 1, 1, 0, 1), (2, 3), (5,)),
    # data gradients by tall blocks of pixels, two launches: by eight and single channels, strides, groups, one and two CTAs per SM
    ((128, 96, 27, 256, 5, 1, 2, 2), (3,), (6, 7)), ((64, 24, 60, 256, 5, 2, 2, 1), (2, 3, 4), (6, 7)), ((256, 20, 24, 50, 5, 1, 0, 1), (2,), (5, 6)),
    ((50, 31, 43, 250, 5, 1, 2, 1), (3, 4), (6, 7)),
    # weight gradients of 320 - 511 lowered rows, by the gather kernel
    ((100, 16, 40, 128, 5, 1, 2, 1), (2, 3), (6, 7)), ((100, 45, 41, 333, 3, 1, 1, 1), (3, 4), (6, 7)),
    # weight gradients of 257 - 384 lowered rows with stride 4, two launches as well: odd and even rows of pixels, window rows at every place of their
    # 16-byte blocks, tiles of filters that end inside a quadrant, groups
    ((90, 2, 200, 128, 12, 4, 0, 1), (2,), (6, 7)), ((90, 3, 190, 128, 10, 4, 0, 1), (2,), (6, 7)), ((90, 2, 201, 128, 13, 4, 0, 1), (2,), (6, 7)),
    ((64, 4, 199, 256, 12, 4, 0, 2), (2, 3), (6, 7)), ((128, 3, 150, 120, 11, 4, 0, 1), (2,), (6, 7)),
])
def test_pairs_of_fp16(ctx, layer, shape, forward, backward):
    B, D, n, o, k, s, p, g = shape
    at = layer(shape)
    X, W, b, dY = at.operands(D)
    assert launches(ctx, lambda: at.forward(X, W, b)) in forward and launches(ctx, lambda: at.backward(X, W, dY)) in backward
    Y, (dX, dW, db) = at.forward(X, W, b), at.backward(X, W, dY)
    # with stride 4 db is a row of the weight gradient (the row of ones), a chain of up to 176 blocks as the others; otherwise fp32 sums
    chains = (D // g * k * k, o // g * k * k, 176 * 32, 176 * 32 if s == 4 else 1)
    for got, ref, products, name in zip((Y, dX, dW, db), at.exact(X, W, b, dY), chains, ("Y", "dX", "dW", "db")):
        assert off(got, ref) <= bound(products), name


SHAPE = (67, 256, 13, 384, 3, 1, 1, 1)


@pytest.mark.parametrize("up", [-40, -20, 20, 40])
def test_scaled_operands_give_the_same_bits(layer, up):
    """A power of two goes into the scale: the products' bits do not change as long as nothing leaves fp32's range."""
    at = layer(SHAPE)
    X, W, b, dY = at.operands(1)
    b.zero_()
    Y, (dX, dW, _) = at.forward(X, W, b), at.backward(X, W, dY)
    f = 2.0 ** up
    assert torch.equal(at.forward(X * f, W, b), Y * f)
    dX2, dW2, _ = at.backward(X, W, dY * f)
    assert torch.equal(dX2, dX * f) and torch.equal(dW2, dW * f)
    dX3, dW3, _ = at.backward(X * f, W, dY / f)
    assert torch.equal(dX3, dX / f) and torch.equal(dW3, dW)


# Operands that are not split into fp16: largest values beyond 2^46 and below 2^-45, images so far below the largest value that fp16 would lose them, one
# value far above all others; and all zeros, which are.  Every image is right by its own measure.
@pytest.mark.parametrize("what", ["large", "small", "one image", "one value", "weights", "zeros"])
def test_operands_far_apart(layer, what):
    at = layer(SHAPE)
    X, W, b, dY = at.operands(2)
    b.zero_()
    if what == "large":
        X, dY = X * 2.0 ** 60, dY * 2.0 ** 50
    elif what == "small":
        X, dY = X * 2.0 ** -60, dY * 2.0 ** -60
    elif what == "one image":
        X[3] *= 1e-9
        dY[5] *= 1e-9
    elif what == "one value":
        X[0, 0, 0, 0], dY[1, 1, 1, 1] = 1e9, 1e9
    elif what == "weights":
        W[:, 0] *= 1e9
    else:
        X.zero_()
        dY.zero_()
    Y, (dX, dW, db) = at.forward(X, W, b), at.backward(X, W, dY)
    Yr, dXr, dWr, _ = at.exact(X, W, b, dY)
    if what == "zeros":
        assert not Y.any() and not dX.any() and not dW.any() and not db.any()
        return
    for image in range(SHAPE[0]):
        assert off(Y[image], Yr[image]) <= 2 * bound(256 * 9), image
        assert off(dX[image], dXr[image]) <= 2 * bound(384 * 9), image
    assert off(dW, dWr) <= 2 * bound(176 * 32)


STRIDE_4 = [(90, 2, 201, 128, 13, 4, 0, 1), (128, 3, 150, 120, 11, 4, 0, 1)]
TALL = [(128, 96, 27, 256, 5, 1, 2, 2), (64, 24, 60, 256, 5, 2, 2, 1), (256, 20, 24, 50, 5, 1, 0, 1), (50, 31, 43, 250, 5, 1, 2, 1)]


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("shape", [SHAPE] + TALL + STRIDE_4)
def test_values_that_are_not_finite(layer, shape, value):
    """They reach their windows, and nothing else changes by a bit; the calls after them are what those before them were."""
    at = layer(shape)
    B, D, n, o, k, s, p, g = shape
    X, W, b, dY = at.operands(3)
    W = torch.where(W == 0, torch.full_like(W, 0.01), W)
    where = [(B - 1, 9, at.m - 1, at.m // 2), (0, o - 1, 0, 0), (B // 2, 3, at.m // 2, at.m // 2)]
    X[B - 1, D - 1, 6, 7] = 0
    for w in where:
        dY[w] = 0
    Y, (dX, dW, db) = at.forward(X, W, b), at.backward(X, W, dY)
    Xn, dYn = X.clone(), dY.clone()
    Xn[B - 1, D - 1, 6, 7] = value
    for w in where:
        dYn[w] = value
    ones = torch.ones_like(W)
    inside = torch.nn.functional.conv2d((Xn != X).float(), ones, None, s, p, 1, g) != 0
    Yn = at.forward(Xn, W, b)
    assert not torch.isfinite(Yn[inside]).any() and torch.equal(Yn[~inside], Y[~inside])
    inside = torch.nn.grad.conv2d_input(X.shape, ones, (dYn != dY).float(), s, p, 1, g) != 0
    dXn, dWn, dbn = at.backward(X, W, dYn)
    assert not torch.isfinite(dXn[inside]).any() and torch.equal(dXn[~inside], dX[~inside])
    others = torch.ones(o, dtype=torch.bool, device="cuda")
    others[[w[1] for w in where]] = False
    assert torch.equal(dWn[others], dW[others]) and not torch.isfinite(dbn[~others]).any() and torch.equal(dbn[others], db[others])
    taps = torch.nn.grad.conv2d_weight((Xn != X).float(), W.shape, torch.ones_like(dY), s, p, 1, g) != 0
    dWn = at.backward(Xn, W, dY)[1]
    assert not torch.isfinite(dWn[taps]).any() and torch.equal(dWn[~taps], dW[~taps])
    assert torch.equal(at.forward(X, W, b), Y) and all(torch.equal(u, v) for u, v in zip(at.backward(X, W, dY), (dX, dW, db)))


@pytest.mark.parametrize("shape", [t for t in TALL if t[5] == 1])  # (with a stride a block of one period has zero weights for some pixels as well)
def test_many_values_that_are_not_finite(layer, shape):
    """More than a data gradient by tall blocks keeps a list of: it takes the others, and back."""
    at = layer(shape)
    _, _, _, _, _, s, p, g = shape
    X, W, b, dY = at.operands(8)
    clean = at.backward(X, W, dY)[0]
    wild = dY.clone()
    wild[1, 2, :, 3] = float("nan")
    inside = torch.nn.grad.conv2d_input(X.shape, torch.ones_like(W), torch.isnan(wild).float(), s, p, 1, g) != 0
    dX = at.backward(X, W, wild)[0]
    assert torch.isnan(dX[inside]).all() and off(dX[~inside], clean[~inside].double()) <= 4 * bound(shape[3] // g * shape[4] ** 2)
    assert torch.equal(at.backward(X, W, dY)[0], clean)


def test_one_way_after_the_other(layer):
    """The rows of dY hold one form after the other: what an earlier call has left behind the last image does not show."""
    at = layer(SHAPE)
    X, W, b, dY = at.operands(4)
    first = at.backward(X, W, dY)
    far = dY.clone()
    far[0] *= 1e-12
    other = at.backward(X, W, far)
    wild = dY.clone()
    wild[-1, :, -1, -1] = float("nan")
    at.backward(X, W, wild)
    assert all(torch.equal(u, v) for u, v in zip(at.backward(X, W, far), other))
    assert all(torch.equal(u, v) for u, v in zip(at.backward(X, W, dY), first))


@pytest.mark.parametrize("shape", [(37, 384, 13, 256, 3, 1, 1, 1), (64, 384, 14, 512, 3, 1, 1, 2), (65, 256, 13, 384, 3, 1, 1, 1), TALL[0]])
def test_pooled_gradients_in_rows(ctx, layer, shape):
    """The pooling kernel writes the rows of dY itself: the gradients of the chain pool -> ReLU -> convolution against 64 bits, and twice the same."""
    B, D, n, o, k, s, p, g = shape
    at = layer(shape)
    X, W, b, _ = at.operands(5)
    m, q = at.m, (at.m - 3) // 2 + 1
    capi.check(ctx.lib.cct_conv_plan_reserve_fusion(at.plan), "reserve", ctx.h)
    Y = at.forward(X, W, b).clamp_(min=0)
    P, index = torch.nn.functional.max_pool2d(Y, 3, 2, return_indices=True)
    assert P.shape[-1] == q
    index, dP = index.int().contiguous(), torch.randn(P.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    runs = []
    for _ in range(2):
        dX, dW, db = torch.full_like(X, 7), torch.full_like(W, 7), torch.full((o,), 7.0, device="cuda")
        torch.cuda.synchronize()
        f = capi.BwdFusion(None, index.data_ptr(), dP.data_ptr(), 3, 2, 0, P.data_ptr())
        capi.check(ctx.lib.cct_conv_backward_fused(at.plan, X.data_ptr(), W.data_ptr(), None, C.byref(f), dX.data_ptr(), dW.data_ptr(), db.data_ptr()),
                   "backward", ctx.h)
        ctx.sync()
        runs.append((dX, dW, db))
    dY = torch.zeros(B, o, m * m, device="cuda", dtype=torch.double)
    dY.scatter_add_(2, index.long().view(B, o, -1), (dP * (P > 0)).double().view(B, o, -1))
    _, dXr, dWr, dbr = at.exact(X, W, b, dY.view(B, o, m, m))
    for got, ref, products, name in zip(runs[0], (dXr, dWr, dbr), (o // g * k * k, 176 * 32, 1), ("dX", "dW", "db")):
        assert off(got, ref) <= bound(products), name
    assert all(torch.equal(u, v) for u, v in zip(*runs))
    # one that is not finite: the pixels of the window of the element that it goes to
    at_most = (P[1, 2] > 0).nonzero()[0].tolist()
    dP[1, 2, at_most[0], at_most[1]] = float("nan")
    dX = torch.full_like(X, 7)
    torch.cuda.synchronize()
    capi.check(ctx.lib.cct_conv_backward_fused(at.plan, X.data_ptr(), W.data_ptr(), None, C.byref(f), dX.data_ptr(), dW.data_ptr(), db.data_ptr()),
               "backward", ctx.h)
    ctx.sync()
    hit = torch.zeros(B, o, m * m, device="cuda")
    hit[1, 2, index[1, 2, at_most[0], at_most[1]]] = 1
    inside = torch.nn.grad.conv2d_input(X.shape, torch.ones_like(W), hit.view(B, o, m, m), s, p, 1, g) != 0
    assert torch.isnan(dX[inside]).all() and torch.equal(dX[~inside], runs[0][0][~inside])
