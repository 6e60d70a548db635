"""Kernels for small problems against float64: convolutions below the tensor cores' size, the
squeeze-and-excite block, products of a few rows. All are fp32 dot products of K terms in another
order than the oracle's; each of the at most K + 8 roundings of a partial sum is off by at most
2^-24 of sum |a||b|, so (K + 8) * 2^-24 * sum |a||b| bounds the error whatever the order."""
import numpy as np
import pytest
import torch

from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _run(build, inputs, kinds=None):
    g = ir.Graph()
    vals = [g.add_input(f"in{i}", a.shape) for i, a in enumerate(inputs)]
    g.outputs.append(build(g, *vals))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        if kinds:
            assert [e["kind"] for e in sess.schedule()] == kinds
        return sess.run(list(inputs))[0]
    finally:
        sess.close()


def _conv(g, x, w, b, k=1, s=1, p=0):
    return g.op("Conv2d", x, g.new_init(w), g.new_init(b), kernel_shape=[k, k], strides=[s, s], padding=[p] * 4,
                dilations=[1, 1], group=1, auto_pad="")


# n, c, h, oc, kernel, stride, pad, gate: one K step and several (cluster split), channel counts off
# the tile, planes whose rows are not whole float4s, columns across images, more than 148 tiles
@pytest.mark.parametrize("n,c,h,oc,k,s,p,gate", [
    (1, 16, 8, 16, 1, 1, 0, False), (1, 240, 14, 80, 1, 1, 0, True), (3, 61, 7, 37, 1, 1, 0, True),
    (2, 960, 3, 5, 1, 1, 0, False), (1, 3, 33, 16, 3, 2, 1, False), (2, 7, 9, 12, 5, 1, 2, False),
    (1, 16, 112, 16, 1, 1, 0, False), (5, 9, 31, 33, 1, 1, 0, True), (1, 33, 17, 40, 1, 2, 0, False)])
def test_small_convolution(cuda_lib, n, c, h, oc, k, s, p, gate):
    rng = np.random.default_rng(c * h + oc)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32)
    w = rng.standard_normal((oc, c, k, k)).astype(np.float32)
    b = rng.standard_normal(oc).astype(np.float32)
    gt = rng.random((n, c, 1, 1)).astype(np.float32)
    oh = (h + 2 * p - k) // s + 1
    r = rng.standard_normal((n, oc, oh, oh)).astype(np.float32)

    def build(g, xi, ri, gi=None):
        y = _conv(g, g.op("Mul", xi, gi) if gate else xi, w, b, k, s, p)
        return g.op("Add", g.op("ReLU", y), ri)
    got = _run(build, [x, r] + ([gt] if gate else []), ["conv_fp32_simt"])
    xg = torch.from_numpy(x * gt if gate else x).double()
    conv = lambda a, f, bias: torch.nn.functional.conv2d(a, f, bias, stride=s, padding=p)
    want = torch.relu(conv(xg, torch.from_numpy(w).double(), torch.from_numpy(b).double())).numpy() + r
    mass = conv(xg.abs(), torch.from_numpy(w).double().abs(), torch.from_numpy(b).double().abs()).numpy() + np.abs(r)
    assert (np.abs(got - want) <= (c * k * k + 8) * EPS * mass).all()


# The same kernel behind another one, where it makes a pass over zeros ahead of its first: a block of the cluster
# without a K step, K steps beyond the ring, tiles over many images, a single K step, a window.
@pytest.mark.parametrize("n,c,h,oc,k,p,gate", [
    (1, 160, 7, 80, 1, 0, True), (1, 2048, 5, 20, 1, 0, True), (1, 1600, 4, 33, 1, 0, True), (40, 36, 2, 17, 1, 0, False),
    (33, 40, 3, 7, 1, 0, True), (1, 8, 14, 16, 5, 2, False), (3, 31, 6, 18, 3, 1, False)])
def test_small_convolution_behind_a_kernel(cuda_lib, n, c, h, oc, k, p, gate):
    rng = np.random.default_rng(c * h + oc)
    x, gt, r = (rng.standard_normal(d).astype(np.float32) for d in ((n, c, h, h), (n, c, 1, 1), (n, oc, h, h)))
    w, b = rng.standard_normal((oc, c, k, k)).astype(np.float32), rng.standard_normal(oc).astype(np.float32)

    def build(g, xi, ri, gi=None):
        xi = g.op("Sqrt", g.op("ReLU", xi))
        return g.op("Add", g.op("ReLU", _conv(g, g.op("Mul", xi, gi) if gate else xi, w, b, k, 1, p)), ri)
    got = _run(build, [x, r] + ([gt] if gate else []))
    xs = np.sqrt(np.maximum(x, 0))
    xg = torch.from_numpy(xs * gt if gate else xs).double()
    conv = lambda a, f, bias: torch.nn.functional.conv2d(a, f, bias, padding=p)
    want = torch.relu(conv(xg, torch.from_numpy(w).double(), torch.from_numpy(b).double())).numpy() + r
    mass = conv(xg.abs(), torch.from_numpy(w).double().abs(), torch.from_numpy(b).double().abs()).numpy() + np.abs(r)
    assert (np.abs(got - want) <= (c * k * k + 8) * EPS * mass).all()


# Pointwise on the tensor cores with K cut over a cluster of two, four or eight: channels of a block that are no multiple of sixteen
# or of the eight under way at once, a last tile with channels that do not exist, ragged pixels. Bound: that of the split products.
@pytest.mark.parametrize("n,c,h,oc", [(4, 672, 14, 112), (5, 512, 9, 130), (1, 2048, 7, 500), (8, 1024, 8, 47), (32, 240, 14, 80), (13, 960, 6, 161)])
@pytest.mark.parametrize("act,res,gate", [(None, False, False), ("ReLU", True, False), (None, True, True)])
def test_pointwise_convolution_cut_over_a_cluster(cuda_lib, n, c, h, oc, act, res, gate):
    rng = np.random.default_rng(c + oc)
    x, r = rng.standard_normal((n, c, h, h)).astype(np.float32), rng.standard_normal((n, oc, h, h)).astype(np.float32)
    w, b, gt = rng.standard_normal((oc, c, 1, 1)).astype(np.float32), rng.standard_normal(oc).astype(np.float32), rng.random((n, c, 1, 1)).astype(np.float32)

    def build(g, xi, *more):
        y = _conv(g, g.op("Mul", xi, more[-1]) if gate else xi, w, b)
        y = g.op(act, y) if act else y
        return g.op("Add", y, more[0]) if res else y
    got = _run(build, [x] + ([r] if res else []) + ([gt] if gate else []), ["gemm_tf32x3_tcgen05"])
    xg = (x * gt if gate else x).astype(np.float64).transpose(0, 2, 3, 1)
    back = lambda a: a.transpose(0, 3, 1, 2)
    want = back(xg @ w[:, :, 0, 0].T.astype(np.float64) + b)
    mass = back(np.abs(xg) @ np.abs(w[:, :, 0, 0].T).astype(np.float64) + np.abs(b))
    want = np.maximum(want, 0) if act else want
    want = want + r if res else want
    assert (np.abs(got - want) <= 1e-5 * np.abs(want) + 5e-6 * mass).all()


# one, two and three images per cluster, with a remainder; planes with and without whole float4s
@pytest.mark.parametrize("n,c,h,s", [(1, 72, 28, 24), (3, 960, 7, 240), (19, 120, 14, 32), (41, 36, 5, 4), (1, 8, 1, 8)])
def test_squeeze_excite_block(cuda_lib, n, c, h, s):
    rng = np.random.default_rng(c + h)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32) + 0.5
    w1, w2 = (rng.standard_normal(d).astype(np.float32) / 4 for d in ((s, c, 1, 1), (c, s, 1, 1)))
    b1, b2 = rng.standard_normal(s).astype(np.float32), rng.standard_normal(c).astype(np.float32)

    def build(g, xi):
        z = g.op("ReLU", _conv(g, g.op("GlobalAveragePool", xi), w1, b1))
        return g.op("HardSigmoid", _conv(g, z, w2, b2), alpha=0.2, beta=0.5)
    got = _run(build, [x], ["squeeze_excite"])[:, :, 0, 0]
    x64, a1, a2 = x.astype(np.float64), w1[:, :, 0, 0].astype(np.float64), w2[:, :, 0, 0].astype(np.float64)
    mean = x64.mean((2, 3))
    hid = np.maximum(mean @ a1.T + b1, 0)
    z = hid @ a2.T + b2
    # errors of the means and of the first product pass through |W| with slope at most one
    e_mean = (h * h + 8) * EPS * np.abs(x64).mean((2, 3))
    e_hid = e_mean @ np.abs(a1).T + (c + 8) * EPS * (np.abs(mean) @ np.abs(a1).T + np.abs(b1))
    e_z = e_hid @ np.abs(a2).T + (s + 8) * EPS * (hid @ np.abs(a2).T + np.abs(b2))
    assert (np.abs(got - np.clip(0.2 * z + 0.5, 0, 1)) <= 0.2 * e_z + 4 * EPS).all()


# Depthwise convolution, activation, squeeze-and-excite block: means from the convolution's kernel (rows of whole float4s
# and others, several planes a block with a remainder, stride two, one image and clusters of two) or, where its planes
# are too large for that, from the block itself. The convolution's own result is held to its taps' rounding.
@pytest.mark.parametrize("n,c,h,k,st,s,pooled", [
    (1, 72, 28, 5, 2, 24, True), (2, 120, 28, 5, 1, 32, True), (3, 36, 7, 5, 1, 12, True), (19, 40, 14, 3, 1, 8, True),
    (1, 44, 9, 3, 1, 4, True), (2, 24, 14, 5, 2, 8, True), (1, 8, 5, 5, 1, 8, True), (1, 16, 40, 3, 1, 8, False), (2, 12, 61, 3, 1, 4, False)])
@pytest.mark.parametrize("act", ["ReLU", "HardSwish"])
def test_depthwise_in_front_of_squeeze_excite(cuda_lib, n, c, h, k, st, s, pooled, act):
    rng = np.random.default_rng(c + h)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32)
    f, fb = rng.standard_normal((c, 1, k, k)).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    w1, w2 = (rng.standard_normal(d).astype(np.float32) / 4 for d in ((s, c, 1, 1), (c, s, 1, 1)))
    b1, b2 = rng.standard_normal(s).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    g = ir.Graph()
    y = g.op("Conv2d", g.add_input("x", x.shape), g.new_init(f), g.new_init(fb), kernel_shape=[k, k], strides=[st, st],
             padding=[k // 2] * 4, dilations=[1, 1], group=c, auto_pad="")
    y = g.op("Mul", y, g.op("HardSigmoid", y)) if act == "HardSwish" else g.op(act, y)
    z = g.op("ReLU", _conv(g, g.op("GlobalAveragePool", y), w1, b1))
    g.outputs += [y, g.op("HardSigmoid", _conv(g, z, w2, b2), alpha=0.2, beta=0.5)]
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        plan = sess.schedule()
        assert [e["kind"] for e in plan] == ["conv_depthwise", "squeeze_excite"]
        planes = 4.0 * n * c * ((h - 1) // st + 1) ** 2
        assert (plan[1]["bytes"] < planes + 4 * (2 * c * s)) == pooled
        got_y, got = sess.run([x])
    finally:
        sess.close()
    conv = lambda a, b: torch.nn.functional.conv2d(torch.from_numpy(a).double(), torch.from_numpy(b).double(), None, stride=st, padding=k // 2,
                                                   groups=c).numpy()
    y64 = conv(x, f) + fb[:, None, None]
    e_y = (k * k + 2) * EPS * (conv(np.abs(x), np.abs(f)) + np.abs(fb)[:, None, None])
    if act == "HardSwish":                             # slope at most 1.5, four roundings
        y64, e_y = y64 * np.clip(0.2 * y64 + 0.5, 0, 1), 1.5 * e_y + 4 * EPS * np.abs(y64)
    else:
        y64 = np.maximum(y64, 0)
    assert (np.abs(got_y - y64) <= e_y).all()
    hw, a1, a2 = y64.shape[2] * y64.shape[3], w1[:, :, 0, 0].astype(np.float64), w2[:, :, 0, 0].astype(np.float64)
    mean = y64.mean((2, 3))
    hid = np.maximum(mean @ a1.T + b1, 0)
    e_mean = (hw + 8) * EPS * np.abs(y64).mean((2, 3)) + e_y.mean((2, 3))
    e_hid = e_mean @ np.abs(a1).T + (c + 8) * EPS * (np.abs(mean) @ np.abs(a1).T + np.abs(b1))
    e_z = e_hid @ np.abs(a2).T + (s + 8) * EPS * (hid @ np.abs(a2).T + np.abs(b2))
    want = np.clip(0.2 * (hid @ a2.T + b2) + 0.5, 0, 1)
    assert (np.abs(got[:, :, 0, 0] - want) <= 0.2 * e_z + 4 * EPS).all()


@pytest.mark.parametrize("m,k,n", [(1, 4, 3), (1, 768, 1000), (2, 132, 17), (3, 256, 10), (4, 60, 33), (9, 1280, 65), (32, 960, 1280)])
def test_product_of_a_few_rows(cuda_lib, m, k, n):
    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = rng.standard_normal((n, k)).astype(np.float32)
    b = rng.standard_normal(n).astype(np.float32)
    got = _run(lambda g, x: g.op("ReLU", g.op("Gemm", x, g.new_init(w), g.new_init(b), alpha=0.5, beta=2.0, trans_a=False,
                                              trans_b=True)), [a], ["gemm_fp32_rows"])
    a64, w64 = a.astype(np.float64), w.astype(np.float64)
    want = np.maximum(0.5 * (a64 @ w64.T) + 2.0 * b, 0)
    assert (np.abs(got - want) <= (k + 8) * EPS * (0.5 * (np.abs(a64) @ np.abs(w64).T) + 2.0 * np.abs(b))).all()
    w2 = np.ascontiguousarray(w.T)     # stored [K, N]: transposed once at create
    got = _run(lambda g, x: g.op("MatMul", x, g.new_init(w2)), [a], ["gemm_fp32_rows"])
    assert (np.abs(got - a64 @ w64.T) <= (k + 8) * EPS * (np.abs(a64) @ np.abs(w64).T)).all()


# 3xTF32 with a tensor-memory accumulator that truncates after every MMA step of 8 products: two
# operands of 22 bits and K / 8 * 3 truncations of at most 2^-23 each of the partial sum, with
# the bound the other tensor-core tests use for the latter: 1e-5 |want| + 5e-6 sum |a||b|.
# Channel counts off the 16s, K off the 8s and 32s, planes of odd size, K cut over a cluster of
# eight, several channel tiles, windows, a gate; residual and bias always.
@pytest.mark.parametrize("n,c,h,oc,k,s,p,gate", [
    (10, 21, 57, 27, 1, 1, 0, True), (3, 960, 7, 160, 1, 1, 0, True), (2, 672, 14, 112, 1, 1, 0, False),
    (5, 40, 28, 241, 1, 1, 0, False), (8, 3, 97, 33, 3, 2, 1, False), (1, 72, 14, 80, 5, 1, 2, False),
    (5, 1, 512, 16, 1, 1, 0, True), (1, 4096, 5, 300, 1, 1, 0, False), (32, 16, 40, 64, 1, 1, 0, False),
    # wide channel tiles with a table and a cluster's exchange beside the ring
    (8, 256, 14, 256, 3, 1, 1, False), (1, 256, 28, 512, 3, 1, 1, False), (1, 256, 32, 480, 3, 1, 1, False),
    (16, 128, 14, 256, 3, 1, 1, False), (2, 448, 14, 250, 3, 1, 1, False),
    # walking blocks that have an SM to themselves
    (6, 117, 57, 216, 1, 1, 0, True), (6, 117, 57, 215, 1, 1, 0, False)])
def test_tensor_core_convolution(cuda_lib, n, c, h, oc, k, s, p, gate):
    rng = np.random.default_rng(c * h + oc)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32)
    w = rng.standard_normal((oc, c, k, k)).astype(np.float32)
    b = rng.standard_normal(oc).astype(np.float32)
    gt = rng.random((n, c, 1, 1)).astype(np.float32)
    oh = (h + 2 * p - k) // s + 1
    r = rng.standard_normal((n, oc, oh, oh)).astype(np.float32)

    def build(g, xi, ri, gi=None):
        y = _conv(g, g.op("Mul", xi, gi) if gate else xi, w, b, k, s, p)
        return g.op("Add", g.op("ReLU", y), ri)
    got = _run(build, [x, r] + ([gt] if gate else []), ["gemm_tf32x3_tcgen05"])
    xg = torch.from_numpy(x * gt if gate else x).double()
    conv = lambda a, f, bias: torch.nn.functional.conv2d(a, f, bias, stride=s, padding=p)
    want = torch.relu(conv(xg, torch.from_numpy(w).double(), torch.from_numpy(b).double())).numpy() + r
    mass = conv(xg.abs(), torch.from_numpy(w).double().abs(), torch.from_numpy(b).double().abs()).numpy() + np.abs(r)
    assert (np.abs(got - want) <= 1e-5 * np.abs(want) + 5e-6 * mass).all()


# Rows of whole float4s with the paddings of the vector form, other paddings and rows, results whose rows are not
# whole float4s, planes smaller than the filter. K * K + 2 roundings of terms bounded by the sum of magnitudes.
@pytest.mark.parametrize("n,c,h,w,k,s,p", [
    (2, 5, 28, 28, 3, 1, 1), (1, 7, 56, 112, 3, 2, 1), (2, 3, 16, 20, 5, 1, 2), (3, 4, 28, 28, 5, 2, 2), (1, 9, 12, 8, 3, 1, 0),
    (1, 3, 9, 4, 5, 2, 1), (2, 3, 14, 14, 3, 1, 1), (1, 2, 6, 12, 3, 2, 0), (1, 2, 8, 8, 3, 1, 2), (1, 3, 1, 4, 3, 1, 1)])
def test_depthwise_convolution(cuda_lib, n, c, h, w, k, s, p):
    rng = np.random.default_rng(h * w + k)
    x, f, b = (rng.standard_normal(d).astype(np.float32) for d in ((n, c, h, w), (c, 1, k, k), (c,)))
    got = _run(lambda g, xi: g.op("ReLU", g.op("Conv2d", xi, g.new_init(f), g.new_init(b), kernel_shape=[k, k], strides=[s, s],
                                               padding=[p] * 4, dilations=[1, 1], group=c, auto_pad="")), [x], ["conv_depthwise"])
    conv = lambda a, q, r: torch.nn.functional.conv2d(torch.from_numpy(a).double(), torch.from_numpy(q).double(),
                                                      torch.from_numpy(r).double(), stride=s, padding=p, groups=c).numpy()
    assert (np.abs(got - np.maximum(conv(x, f, b), 0)) <= (k * k + 2) * EPS * conv(np.abs(x), np.abs(f), np.abs(b))).all()


# Filter and bias computed by the steps in front: nothing of them may be read before these have finished.
@pytest.mark.parametrize("n,c,h,oc,kinds", [
    (1, 48, 12, 40, "conv_fp32_simt"), (2, 256, 28, 96, "gemm_tf32x3_tcgen05")])
def test_convolution_with_computed_filter(cuda_lib, n, c, h, oc, kinds):
    rng = np.random.default_rng(c)
    x, w, b = (rng.standard_normal(d).astype(np.float32) for d in ((n, c, h, h), (oc, c, 1, 1), (oc,)))
    w2, b2 = rng.standard_normal(w.shape).astype(np.float32), rng.standard_normal(b.shape).astype(np.float32)

    def build(g, xi, wi, bi):
        return g.op("Conv2d", xi, g.op("Mul", wi, g.new_init(w2)), g.op("Mul", bi, g.new_init(b2)), kernel_shape=[1, 1],
                    strides=[1, 1], padding=[0] * 4, dilations=[1, 1], group=1, auto_pad="")
    g = ir.Graph()
    vals = [g.add_input(f"in{i}", a.shape) for i, a in enumerate((x, w, b))]
    g.outputs.append(build(g, *vals))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    assert kinds in [e["kind"] for e in sess.schedule()]
    t = lambda a: torch.from_numpy(a).double()
    for i in range(3):       # other operands on each run
        xs = [np.roll(a, i, 0) * np.float32(1 + i) for a in (x, w, b)]
        got = sess.run(xs)[0]
        wd, bd = t(xs[1] * w2), t(xs[2] * b2)
        want = torch.nn.functional.conv2d(t(xs[0]), wd, bd).numpy()
        mass = torch.nn.functional.conv2d(t(xs[0]).abs(), wd.abs(), bd.abs()).numpy()
        assert (np.abs(got - want) <= 1e-5 * np.abs(want) + 5e-6 * mass).all()
    sess.close()


# An MLP behind a LayerNormalization: both products on clusters that share a tile along K, the first one
# writing the halves the second one takes. Rows off the tiles, K off the K-blocks, N off the tile widths.
# fp16-split products: 1e-5 |want| + 5e-6 sum |a||b| each (as in the other tests of the format); the first
# one's error reaches the second through |w2| (Gelu has slope at most 1.13).
@pytest.mark.parametrize("m,d,hidden", [(33, 192, 768), (197, 768, 3072), (129, 200, 328), (128, 1024, 64), (700, 384, 1536)])
def test_few_row_products_on_clusters(cuda_lib, m, d, hidden):
    rng = np.random.default_rng(m + d)
    x = rng.standard_normal((m, d)).astype(np.float32)
    gam, bet = (1 + 0.1 * rng.standard_normal(d)).astype(np.float32), (0.1 * rng.standard_normal(d)).astype(np.float32)
    w1 = (rng.standard_normal((d, hidden)) / np.sqrt(d)).astype(np.float32)
    w2 = (rng.standard_normal((hidden, d)) / np.sqrt(hidden)).astype(np.float32)
    b1, b2 = rng.standard_normal(hidden).astype(np.float32), rng.standard_normal(d).astype(np.float32)

    def build(g, xi):
        h = g.op("LayerNormalization", xi, g.new_init(gam), g.new_init(bet), axis=-1, epsilon=1e-6, stash_type=1)
        h = g.op("Gelu", g.op("Add", g.op("MatMul", h, g.new_init(w1)), g.new_init(b1)))
        return g.op("Add", xi, g.op("Add", g.op("MatMul", h, g.new_init(w2)), g.new_init(b2)))
    got = _run(build, [x], ["layer_norm", "gemm_f16x3_cluster_tcgen05", "gemm_f16x3_cluster_tcgen05"])
    t = lambda a: torch.from_numpy(a).double()
    h = torch.nn.functional.layer_norm(t(x), (d,), t(gam), t(bet), 1e-6)
    z = h @ t(w1) + t(b1)
    e1 = 1e-5 * z.abs() + 5e-6 * (h.abs() @ t(w1).abs()) + 1e-5 * (h.abs() @ t(w1).abs())   # LayerNorm itself: 1e-5
    a = torch.nn.functional.gelu(z, approximate="tanh")
    want = t(x) + a @ t(w2) + t(b2)
    bound = 1.13 * e1 @ t(w2).abs() + 1e-5 * want.abs() + 6e-6 * (a.abs() @ t(w2).abs())
    assert (np.abs(got - want.numpy()) <= bound.numpy()).all()


def test_few_row_products_beyond_the_fixed_scale(cuda_lib):
    """A hidden layer of magnitude 1000 leaves the fixed scale of the halves (255): the session goes on with the
    kernels that split their operand themselves (65504), and only beyond that with 3xTF32."""
    m, d, hidden = 197, 384, 1536
    rng = np.random.default_rng(3)
    x = rng.standard_normal((m, d)).astype(np.float32)
    w1 = (1000 * rng.standard_normal((d, hidden)) / np.sqrt(d)).astype(np.float32)
    w2 = (rng.standard_normal((hidden, d)) / np.sqrt(hidden)).astype(np.float32)
    w3 = (rng.standard_normal((d, d)) / np.sqrt(d)).astype(np.float32)
    g = ir.Graph()
    one, zero = g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32))
    xi, scale = g.add_input("x", x.shape), g.add_input("scale", (1,))
    h = g.op("LayerNormalization", xi, one, zero, axis=-1, epsilon=1e-6, stash_type=1)
    g.outputs.append(g.op("MatMul", g.op("Gelu", g.op("MatMul", h, g.new_init(w1))), g.new_init(w2)))
    g.outputs.append(g.op("MatMul", g.op("Mul", xi, scale), g.new_init(w3)))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    kinds = lambda: {e["kind"] for e in sess.schedule()}
    t = lambda a: torch.from_numpy(a).double()
    ln = lambda a: torch.nn.functional.layer_norm(a, (d,), None, None, 1e-6)
    want = [torch.nn.functional.gelu(ln(t(x)) @ t(w1), approximate="tanh") @ t(w2), t(x) @ t(w3)]
    try:
        assert "gemm_f16x3_cluster_tcgen05" in kinds()
        for factor, there in ((1.0, {"gemm_f16x3_tcgen05"}), (1.0, {"gemm_f16x3_tcgen05"}), (1e6, {"gemm_tf32x3_tcgen05"})):
            got = sess.run([x, np.array([factor], np.float32)])
            assert {k for k in kinds() if k.startswith("gemm")} == there, kinds()
            for a, b in zip(got, (want[0], factor * want[1])):
                assert np.linalg.norm(a - b.numpy()) <= 1e-5 * np.linalg.norm(b.numpy())
    finally:
        sess.close()


# eight rows a block, in parts of 1024 floats of K: one part, a whole and a ragged second one, fewer quads than lanes, rows and
# columns off the tile; a row of A without finite values stays in its row
# (up to 256 floats of K it is not staged)
@pytest.mark.parametrize("m,k,n", [(5, 1024, 33), (8, 1028, 16), (13, 2048, 17), (31, 2564, 40), (6, 20, 5), (7, 256, 19), (17, 260, 19)])
def test_product_of_eight_rows_in_parts_of_k(cuda_lib, m, k, n):
    rng = np.random.default_rng(m * k + n)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = rng.standard_normal((n, k)).astype(np.float32)
    a[1, k - 1] = np.inf
    got = _run(lambda g, x: g.op("Gemm", x, g.new_init(w), g.new_init(np.zeros(n, np.float32)), alpha=1.0, beta=1.0, trans_a=False,
                                 trans_b=True), [a], ["gemm_fp32_rows"])
    assert np.isinf(got[1]).all()
    rest = np.arange(m) != 1
    a64, w64 = a[rest].astype(np.float64), w.astype(np.float64)
    assert (np.abs(got[rest] - a64 @ w64.T) <= (k + 8) * EPS * (np.abs(a64) @ np.abs(w64).T)).all()


# 31 to 45 images are three a cluster; the widest vectors that the block takes, one image and four a cluster
@pytest.mark.parametrize("n,c,h,s", [(47, 36, 5, 4), (2, 2560, 2, 512), (61, 3056, 1, 16), (47, 2560, 2, 512)])
def test_squeeze_excite_block_with_four_images_a_cluster(cuda_lib, n, c, h, s):
    test_squeeze_excite_block(cuda_lib, n, c, h, s)


# ... and behind a depthwise convolution that leaves the means
def test_squeeze_excite_block_with_four_images_a_cluster_from_means(cuda_lib):
    test_depthwise_in_front_of_squeeze_excite(cuda_lib, 47, 2688, 2, 3, 1, 384, True, "ReLU")
