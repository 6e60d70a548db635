"""Error against float64 of the kernels that took products over from others, on inputs as they meet (normal
activations, weights of variance 1 / K): none is further off than the path it replaced. The bounds are what
that path measured on these very inputs (2-norm of the difference over 2-norm of the result); the tensor core
truncates its sum at every instruction, so a longer chain on one accumulator shows here at once."""
import numpy as np
import pytest
import torch

from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder

pytestmark = pytest.mark.gpu


def _rel(graph, x, want, kind):
    sess = CudaSessionBuilder(ir.Model(graph, 13)).build()
    try:
        kinds = [e["kind"] for e in sess.schedule()]
        assert kind in kinds, kinds
        got = torch.from_numpy(sess.run([x])[0]).double().cuda()
        assert [e["kind"] for e in sess.schedule()] == kinds
    finally:
        sess.close()
    return ((got - want).norm() / want.norm()).item()


def _t(a):
    return torch.from_numpy(a).double().cuda()


# GEMM over a column buffer, 3xTF32, K in up to 32 slices
@pytest.mark.parametrize("n,c,h,oc,k,pad,bound", [
    (1, 2048, 7, 512, 1, 0, 3.40e-7), (1, 480, 32, 480, 1, 0, 2.69e-7), (1, 64, 56, 64, 3, 1, 2.94e-7), (2, 448, 14, 64, 3, 1, 1.21e-6),
    (1, 64, 56, 256, 1, 0, 1.94e-7), (8, 64, 56, 256, 1, 0, 3.08e-7), (13, 112, 12, 672, 1, 0, 5.51e-7)])
def test_convolution(cuda_lib, n, c, h, oc, k, pad, bound):
    rng = np.random.default_rng(c * h + oc)
    x = np.abs(rng.standard_normal((n, c, h, h))).astype(np.float32)
    w = (rng.standard_normal((oc, c, k, k)) / np.sqrt(c * k * k)).astype(np.float32)
    b = rng.standard_normal(oc).astype(np.float32)
    g = ir.Graph()
    g.outputs.append(g.op("ReLU", g.op("Conv2d", g.add_input("x", x.shape), g.new_init(w), g.new_init(b), kernel_shape=[k, k],
                                       strides=[1, 1], padding=[pad] * 4, dilations=[1, 1], group=1, auto_pad="")))
    want = torch.relu(torch.nn.functional.conv2d(_t(x), _t(w), _t(b), padding=pad))
    assert _rel(g, x, want, "gemm_tf32x3_tcgen05") <= bound


# the one-CTA kernel with two accumulators (first three), the CTA-pair kernel
@pytest.mark.parametrize("m,d,n,bound", [(37, 768, 2304, 1.45e-7), (394, 384, 1152, 1.43e-7), (1386, 384, 384, 1.38e-7),
                                         (197, 768, 2304, 3.49e-7), (2885, 768, 768, 9.8e-7)])
def test_few_row_product(cuda_lib, m, d, n, bound):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, d)).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b = rng.standard_normal(n).astype(np.float32)
    g = ir.Graph()
    h = g.op("LayerNormalization", g.add_input("x", x.shape), g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32)),
             axis=-1, epsilon=1e-6, stash_type=1)
    g.outputs.append(g.op("Add", g.op("MatMul", h, g.new_init(w)), g.new_init(b)))
    want = torch.nn.functional.layer_norm(_t(x), (d,), None, None, 1e-6) @ _t(w) + _t(b)
    assert _rel(g, x, want, "gemm_f16x3_cluster_tcgen05") <= bound


# Full-range products (gemm_mode 3) of few rows: the one-CTA kernel's error on these inputs. Ragged rows, columns and K, K over a
# cluster of two to eight, a single K-block; with each epilogue. Scaled inputs, which the fp16 formats could not hold.
@pytest.mark.parametrize("m,d,n,bound", [(198, 768, 2304, 4.91e-7), (394, 384, 1152, 4.94e-7), (1386, 384, 384, 4.71e-7),
                                         (198, 1536, 384, 6.4e-7), (788, 192, 576, 2.54e-7), (333, 520, 332, 1.84e-7),
                                         (1001, 100, 516, 2.75e-7), (129, 36, 1028, 2.75e-7), (515, 32, 2052, 2.75e-7)])
@pytest.mark.parametrize("act,res,scale", [(None, False, 1.0), ("Gelu", False, 1.0), ("ReLU", True, 1e6)])
def test_full_range_product(cuda_lib, m, d, n, bound, act, res, scale):
    rng = np.random.default_rng(m + n)
    x = (scale * rng.standard_normal((m, d))).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b = (scale * rng.standard_normal(n)).astype(np.float32)
    r = (scale * rng.standard_normal((m, n))).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    y = g.op("Add", g.op("MatMul", xi, g.new_init(w)), g.new_init(b))
    y = g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    sess = CudaSessionBuilder(ir.Model(g, 13)).with_gemm_mode(3).build()
    try:
        assert [(e["kind"], e["launches"]) for e in sess.schedule()] == [("gemm_tf32x3_tcgen05", 1)]   # no second kernel for slices
        got = torch.from_numpy(sess.run([x] + ([r] if res else []))[0]).double().cuda()
    finally:
        sess.close()
    want = _t(x) @ _t(w) + _t(b)
    want = torch.relu(want) if act == "ReLU" else torch.nn.functional.gelu(want, approximate="tanh") if act else want
    want = want + _t(r) if res else want
    # Gelu's slope is at most 1.13, its rational tanh is off by 1e-7 of the result
    assert ((got - want).norm() / want.norm()).item() <= bound * (1.0 if not act else 2.0 if act == "Gelu" else 1.0)


# beyond 256 tokens separate 3xTF32 and fp32 products, up to 256 the kernel on operands from fp32; on a given
# projection (one of 577 tokens) and behind its GEMM
@pytest.mark.parametrize("B,T,H,projection,bound", [
    (2, 577, 12, False, 7.49e-7), (1, 577, 12, True, 1.04e-6), (2, 401, 6, True, 9.92e-7), (3, 145, 6, True, 9.41e-7),
    (1, 226, 12, True, 1.63e-6)])
def test_attention_in_blocks_of_keys(cuda_lib, B, T, H, projection, bound):
    rng = np.random.default_rng(T + H)
    D = 64 * H
    x = rng.standard_normal((B, T, D if projection else 3 * D)).astype(np.float32)
    w = (rng.standard_normal((D, 3 * D)) / np.sqrt(D)).astype(np.float32)
    b = (0.1 * rng.standard_normal(3 * D)).astype(np.float32)
    g = ir.Graph()
    i64 = lambda v: g.new_init(np.asarray(v, np.int64))
    qkv = g.add_input("x", x.shape)
    if projection:
        qkv = g.op("LayerNormalization", qkv, g.new_init(np.ones(D, np.float32)), g.new_init(np.zeros(D, np.float32)), axis=-1,
                   epsilon=1e-6, stash_type=1)
        qkv = g.op("Add", g.op("MatMul", qkv, g.new_init(w)), g.new_init(b))
    q, k, v = g.add_node("Split", [qkv, i64([D, D, D])], 3, axis=2)
    heads = lambda t: g.op("Reshape", g.op("Transpose", g.op("Reshape", t, i64([B, T, H, 64])), perm=[0, 2, 1, 3]), i64([B * H, T, 64]))
    q, k, v = heads(q), heads(k), heads(v)
    s = g.op("Mul", g.op("MatMul", q, g.op("Transpose", k, perm=[0, 2, 1])), g.new_init(np.array([0.125], np.float32)))
    o = g.op("Reshape", g.op("MatMul", g.op("Softmax", s, axis=-1), v), i64([B, H, T, 64]))
    g.outputs.append(g.op("Reshape", g.op("Transpose", o, perm=[0, 2, 1, 3]), i64([B, T, D])))
    tx = _t(x)
    if projection:
        tx = torch.nn.functional.layer_norm(tx, (D,), None, None, 1e-6) @ _t(w) + _t(b)
    tq, tk, tv = [u.reshape(B, T, H, 64).transpose(1, 2) for u in tx.split(D, dim=2)]
    want = (torch.softmax(0.125 * (tq @ tk.transpose(2, 3)), -1) @ tv).transpose(1, 2).reshape(B, T, D)
    assert _rel(g, x, want, "attention_flash_tcgen05") <= bound
