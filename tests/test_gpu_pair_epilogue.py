"""Epilogues of the CTA-pair GEMM against float64 at the edges of its tiles (256 x 256; blocks of 16 x 16 within): a
row or a few columns beyond whole tiles, columns that are whole float4s but not whole groups of eight, K-sliced
last tiles. The bound is the one of all fp16-split products: 1e-5 of the result and 5e-6 of sum |a||b|. Then its form with
short accumulators, and the range of the halves that both write for a next product."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(a).double().cuda()


def _run(graph, inputs, kinds):
    sess = CudaSessionBuilder(ir.Model(graph, 13)).build()
    try:
        assert [e["kind"] for e in sess.schedule()] == kinds
        return torch.from_numpy(sess.run(inputs)[0]).double().cuda()
    finally:
        sess.close()


@pytest.mark.parametrize("m,n,k", [(2817, 1544, 264), (6305, 772, 392), (2561, 2308, 384)])
@pytest.mark.parametrize("act", [None, "ReLU", "Gelu", "HardSwish"])
@pytest.mark.parametrize("bias,res", [(False, False), (True, False), (False, True), (True, True)])
def test_pair_epilogues(cuda_lib, m, n, k, act, bias, res):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32)
    b = rng.standard_normal(n).astype(np.float32)
    r = rng.standard_normal((m, n)).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    y = g.op("MatMul", xi, g.new_init(w))
    y = g.op("Add", y, g.new_init(b)) if bias else y
    y = g.op("Mul", y, g.op("HardSigmoid", y)) if act == "HardSwish" else g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    got = _run(g, [x] + ([r] if res else []), ["act_f16_split", "gemm_f16x3_pair_tcgen05"])
    want, mass, slack = _t(x) @ _t(w), _t(x).abs() @ _t(w).abs(), 0
    if bias:
        want, mass = want + _t(b), mass + _t(b).abs()
    if act == "HardSwish":
        want = want * (0.2 * want + 0.5).clamp(0, 1)
        mass = 2 * mass                             # its slope is at most 1.5
    elif act:
        slack = 1e-6 * want.abs() if act == "Gelu" else 0   # the rational tanh and its cancellation against 1
        want = torch.relu(want) if act == "ReLU" else torch.nn.functional.gelu(want, approximate="tanh")
    if res:
        want, mass = want + _t(r), mass + _t(r).abs()
    assert ((got - want).abs() <= 1e-5 * want.abs() + 5e-6 * mass + slack).all()


# alpha, beta and C beside the product: whole float4s and single elements, a tile cut along K (k 1544), too.
@pytest.mark.parametrize("m,n,k", [(2817, 1540, 264), (6305, 2306, 392), (2561, 1284, 1544)])
@pytest.mark.parametrize("alpha,beta,full", [(0.5, 1.0, False), (1.0, -2.0, False), (0.5, 2.0, True), (1.0, 1.0, True)])
def test_pair_epilogues_with_factors(cuda_lib, m, n, k, alpha, beta, full):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    c = rng.standard_normal((m, n) if full else n).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ci = g.add_input("c", c.shape) if full else g.new_init(c)
    g.outputs.append(g.op("Gemm", xi, g.new_init(w), ci, alpha=alpha, beta=beta, trans_a=False, trans_b=True))
    got = _run(g, [x] + ([c] if full else []), ["act_f16_split", "gemm_f16x3_pair_tcgen05"])
    want = alpha * (_t(x) @ _t(w).T) + beta * _t(c)
    mass = alpha * (_t(x).abs() @ _t(w).abs().T) + abs(beta) * _t(c).abs()
    assert ((got - want).abs() <= 1e-5 * want.abs() + 5e-6 * mass).all()


@pytest.mark.parametrize("m,h,n", [(2817, 1544, 512), (2561, 2312, 768)])
def test_pair_writes_split_results_with_ragged_columns(cuda_lib, m, h, n):
    """The first product's result exists only as fp16 halves (16 bytes of a row per lane); columns end inside a
    64-column group."""
    rng = np.random.default_rng(h)
    x = rng.standard_normal((m, 384)).astype(np.float32)
    w1 = (rng.standard_normal((384, h)) / np.sqrt(384)).astype(np.float32)
    b1 = rng.standard_normal(h).astype(np.float32)
    w2 = (rng.standard_normal((h, n)) / np.sqrt(h)).astype(np.float32)
    g = ir.Graph()
    y = g.op("ReLU", g.op("Add", g.op("MatMul", g.add_input("x", x.shape), g.new_init(w1)), g.new_init(b1)))
    g.outputs.append(g.op("MatMul", y, g.new_init(w2)))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        assert [e["kind"] for e in sess.schedule()][:2] == ["act_f16_split", "gemm_f16x3_pair_tcgen05"]
        got = torch.from_numpy(sess.run([x])[0]).double().cuda()
    finally:
        sess.close()
    h64 = torch.relu(_t(x) @ _t(w1) + _t(b1))
    h_err = 1e-5 * h64 + 5e-6 * (_t(x).abs() @ _t(w1).abs() + _t(b1).abs())
    want = h64 @ _t(w2)
    bound = 1e-5 * want.abs() + 5e-6 * (h64 @ _t(w2).abs()) + h_err @ _t(w2).abs()
    assert ((got - want).abs() <= bound).all()


# Products that the kernel for few rows would take more than a round for: CTA pairs on 256 x 192 tiles whose accumulators
# are given up every one or two K-blocks. Bound: what the few-row kernel measured on these inputs. The last two have ragged rows,
# columns and K.
@pytest.mark.parametrize("m,d,n,bound", [(3152, 768, 768, 2.09e-7), (12672, 384, 384, 1.51e-7), (788, 768, 3072, 2.11e-7),
                                         (6304, 384, 384, 1.53e-7), (3081, 840, 780, 2.35e-7), (8001, 520, 324, 1.62e-7)])
@pytest.mark.parametrize("act,res", [(None, False), ("ReLU", True)])
def test_pairs_with_short_accumulators(cuda_lib, m, d, n, bound, act, res):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, d)).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b = rng.standard_normal(n).astype(np.float32)
    r = rng.standard_normal((m, n)).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    h = g.op("LayerNormalization", xi, g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32)), axis=-1, epsilon=1e-6,
             stash_type=1)
    y = g.op("Add", g.op("MatMul", h, g.new_init(w)), g.new_init(b))
    y = g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    got = _run(g, [x] + ([r] if res else []), ["layer_norm", "gemm_f16x3_pair_sums_tcgen05"])
    y = torch.nn.functional.layer_norm(_t(x), (d,), None, None, 1e-6) @ _t(w) + _t(b)
    y = torch.relu(y) if act else y
    want = y + _t(r) if res else y
    assert ((got - want).norm() / want.norm()).item() <= bound
    assert ((got - want).abs() <= 1e-5 * want.abs() + 2e-5).all()


# The same with a long K, behind a product that leaves the halves: tiles of 128 columns, and (last) of 192. Bound: what the few-row
# kernel measured on these inputs (at K = 1096 and 1992 on the line between), the error of the operand, 1.5e-7, included.
@pytest.mark.parametrize("m,d,n,bound", [(1576, 3072, 768, 5.79e-7), (1182, 4096, 1024, 7.80e-7), (2177, 1096, 772, 2.6e-7),
                                         (2100, 1992, 900, 4.1e-7), (1970, 1280, 1280, 2.86e-7)])
@pytest.mark.parametrize("act,res", [(None, False), ("ReLU", True)])
def test_pairs_with_short_accumulators_and_long_k(cuda_lib, m, d, n, bound, act, res):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, 256)).astype(np.float32)
    w0 = (rng.standard_normal((256, d)) / 16).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b = rng.standard_normal(n).astype(np.float32)
    r = rng.standard_normal((m, n)).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    h = g.op("LayerNormalization", xi, g.new_init(np.ones(256, np.float32)), g.new_init(np.zeros(256, np.float32)), axis=-1,
             epsilon=1e-6, stash_type=1)
    y = g.op("Add", g.op("MatMul", g.op("ReLU", g.op("MatMul", h, g.new_init(w0))), g.new_init(w)), g.new_init(b))
    y = g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    got = _run(g, [x] + ([r] if res else []), ["layer_norm"] + 2 * ["gemm_f16x3_pair_sums_tcgen05"])
    y = torch.relu(torch.nn.functional.layer_norm(_t(x), (256,), None, None, 1e-6) @ _t(w0)) @ _t(w) + _t(b)
    y = torch.relu(y) if act else y
    want = y + _t(r) if res else y
    assert ((got - want).norm() / want.norm()).item() <= bound
    assert ((got - want).abs() <= 1e-5 * want.abs() + 2e-5).all()


# Where tiles of 128 or 192 columns are chosen over long accumulators with K-slices and over two rounds of the few-row kernel: one and
# two rounds, one and two K-blocks on an accumulator, ragged rows, columns and K. Bound: the few-row kernel's, 1.5e-7 at K = 384 and
# 2.1e-7 from 768 on.
@pytest.mark.parametrize("m,d,n", [(9838, 384, 384), (2148, 1024, 1024), (2885, 768, 2304), (10241, 392, 380), (1343, 264, 3004),
                                   (2049, 1000, 1028), (4223, 360, 1532)])
@pytest.mark.parametrize("act,res", [(None, False), ("ReLU", True), ("Gelu", False)])
def test_pairs_with_short_accumulators_beside_the_others(cuda_lib, m, d, n, act, res):
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, d)).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b, r = rng.standard_normal(n).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    h = g.op("LayerNormalization", xi, g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32)), axis=-1, epsilon=1e-6,
             stash_type=1)
    y = g.op("Add", g.op("MatMul", h, g.new_init(w)), g.new_init(b))
    y = g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    got = _run(g, [x] + ([r] if res else []), ["layer_norm", "gemm_f16x3_pair_sums_tcgen05"])
    y = torch.nn.functional.layer_norm(_t(x), (d,), None, None, 1e-6) @ _t(w) + _t(b)
    y = {None: lambda v: v, "ReLU": torch.relu, "Gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](y)
    want = y + _t(r) if res else y
    bound = (2.1e-7 if d > 576 else 1.5e-7) * (2 if act == "Gelu" else 1)    # of the product; Gelu's own 2e-7
    assert ((got - want).norm() / want.norm()).item() <= bound
    assert ((got - want).abs() <= 1e-5 * want.abs() + 2e-5).all()


@pytest.mark.parametrize("act", [None, "ReLU", "Gelu"])
@pytest.mark.parametrize("bias,res", [(False, False), (True, False), (False, True), (True, True)])
def test_every_epilogue_with_short_accumulators(cuda_lib, act, bias, res):
    rng = np.random.default_rng(5)
    m, d, n = 3081, 840, 780
    x = rng.standard_normal((m, d)).astype(np.float32)
    w = (rng.standard_normal((d, n)) / np.sqrt(d)).astype(np.float32)
    b, r = rng.standard_normal(n).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    g = ir.Graph()
    xi = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if res else None
    y = g.op("LayerNormalization", xi, g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32)), axis=-1, epsilon=1e-6,
             stash_type=1)
    y = g.op("MatMul", y, g.new_init(w))
    y = g.op("Add", y, g.new_init(b)) if bias else y
    y = g.op(act, y) if act else y
    g.outputs.append(g.op("Add", y, ri) if res else y)
    got = _run(g, [x] + ([r] if res else []), ["layer_norm", "gemm_f16x3_pair_sums_tcgen05"])
    y = torch.nn.functional.layer_norm(_t(x), (d,), None, None, 1e-6) @ _t(w)
    y = y + _t(b) if bias else y
    y = {None: lambda v: v, "ReLU": torch.relu, "Gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](y)
    want = y + _t(r) if res else y
    assert ((got - want).norm() / want.norm()).item() <= 2.35e-7 * (2 if act == "Gelu" else 1)   # of the product; Gelu's own 2e-7
    assert ((got - want).abs() <= 1e-5 * want.abs() + 2e-5).all()


_NO_PAIRS = """
import numpy as np
from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder
x = np.random.default_rng(0).standard_normal((3152, 768)).astype(np.float32)
g = ir.Graph()
h = g.op("LayerNormalization", g.add_input("x", x.shape), g.new_init(np.ones(768, np.float32)), g.new_init(np.zeros(768, np.float32)),
         axis=-1, epsilon=1e-6, stash_type=1)
g.outputs.append(g.op("MatMul", h, g.new_init(2 * np.eye(768, dtype=np.float32))))
sess = CudaSessionBuilder(ir.Model(g, 13)).build()
assert [e["kind"] for e in sess.schedule()] == ["layer_norm", "gemm_f16x3_cluster_tcgen05"]
y = sess.run([x])[0].astype(np.float64)
x = x.astype(np.float64)
want = 2 * (x - x.mean(1, keepdims=True)) / np.sqrt(x.var(1, keepdims=True) + 1e-6)
assert np.linalg.norm(y - want) <= 1e-6 * np.linalg.norm(want)
"""


def test_without_room_for_a_pair_the_few_row_kernel_stays(cuda_lib):
    """One SM for the persistent kernels: no CTA pair fits, and the product is not handed to them."""
    env = dict(os.environ, ALTIUS_CUDA_TC_SMS="1")
    r = subprocess.run([sys.executable, "-c", _NO_PAIRS], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# ---- range of the halves a product writes for the next one --------------------------------------
# Reported (and repeated on another plan): anything beyond 255, and a warp's part of a tile with nothing of 2^-11 or more.
def _mlp(x, w1, w2, b1=None, act=None, r=None, norm=True):
    g = ir.Graph()
    h = g.add_input("x", x.shape)
    ri = g.add_input("r", r.shape) if r is not None else None
    if norm:
        h = g.op("LayerNormalization", h, g.new_init(np.ones(x.shape[1], np.float32)), g.new_init(np.zeros(x.shape[1], np.float32)), axis=-1,
                 epsilon=1e-6, stash_type=1)
    h = g.op("MatMul", h, g.new_init(w1))
    h = g.op("Add", h, g.new_init(b1)) if b1 is not None else h
    h = g.op(act, h) if act else h
    h = g.op("Add", h, ri) if r is not None else h
    g.outputs.append(g.op("MatMul", h, g.new_init(w2)))
    sess = CudaSessionBuilder(ir.Model(g, 13)).build()
    try:
        before = [e["kind"] for e in sess.schedule()]
        got = torch.from_numpy(sess.run([x] + ([r] if r is not None else []))[0]).double().cuda()
        after = [e["kind"] for e in sess.schedule()]
    finally:
        sess.close()
    y = torch.nn.functional.layer_norm(_t(x), x.shape[1:], None, None, 1e-6) if norm else _t(x)
    y = y @ _t(w1)
    y = y + _t(b1) if b1 is not None else y
    y = {None: lambda v: v, "ReLU": torch.relu, "Gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](y)
    y = y + _t(r) if r is not None else y
    return got, y @ _t(w2), before, after


def _weights(rng, d, h, n):
    return ((rng.standard_normal((d, h)) / np.sqrt(d)).astype(np.float32), (rng.standard_normal((h, n)) / np.sqrt(h)).astype(np.float32))


def _rel(got, want):
    return ((got - want).norm() / want.norm()).item()


# Short accumulators behind a LayerNormalization, tiles of 256 x 256 without one; the epilogues that are compiled in and those that are not.
@pytest.mark.parametrize("m,d,h,n,norm", [(3152, 768, 768, 768, True), (1576, 384, 1536, 384, True), (6304, 384, 1536, 384, False)])
@pytest.mark.parametrize("act,bias,res", [(None, True, False), ("ReLU", True, False), ("ReLU", False, False), ("Gelu", False, False),
                                          ("ReLU", True, True), ("Gelu", True, True)])
def test_tiny_results_are_reported(cuda_lib, m, d, h, n, norm, act, bias, res):
    rng = np.random.default_rng(m + h)
    w1, w2 = _weights(rng, d, h, n)
    tiny = np.float32(1e-8)
    b1 = tiny * rng.standard_normal(h).astype(np.float32) if bias else None
    r = tiny * rng.standard_normal((m, h)).astype(np.float32) if res else None
    x = rng.standard_normal((m, d)).astype(np.float32)
    got, want, before, after = _mlp(x, tiny * w1, w2, b1, act, r, norm)
    assert before[1] == ("gemm_f16x3_pair_sums_tcgen05" if norm else "gemm_f16x3_pair_tcgen05") and before != after
    assert _rel(got, want) <= 3e-5                   # 3xTF32, of positive values: 1.3e-5; as halves 6e-3


# One tile of tiny rows, whose warps have a tile of normal ones, too: its rows live on K positions where the weights are small.
@pytest.mark.parametrize("m,d,h,n,norm", [(12672, 384, 384, 384, True), (12672, 384, 1536, 384, False)])
def test_a_tile_of_tiny_results_is_reported(cuda_lib, m, d, h, n, norm):
    rng = np.random.default_rng(m + h)
    w1, w2 = _weights(rng, d, h, n)
    w1[:d // 2] *= np.float32(1e-7)
    x = rng.standard_normal((m, d)).astype(np.float32)
    x[:256] = 0
    x[:256, :d // 2] = rng.permuted(np.tile(np.float32([1, -1]), (256, d // 4)), axis=1)     # a mean of zero, whatever the order
    got, want, before, after = _mlp(x, w1, w2, norm=norm)
    assert before != after
    assert _rel(got[:256], want[:256]) <= 3e-5       # as halves 7e-4


# In range the halves stay: M, N and K off the tiles, N a multiple of 8 but not of 16; one value beyond 255 goes to another plan.
@pytest.mark.parametrize("m,d,h,n,norm", [(1577, 392, 1544, 384, True), (3081, 776, 776, 520, True), (6305, 392, 1544, 384, False)])
@pytest.mark.parametrize("act,bias,res", [(None, False, False), ("Gelu", True, False), ("ReLU", False, False), ("Gelu", True, True)])
@pytest.mark.parametrize("beyond", [False, True])
def test_results_as_halves(cuda_lib, m, d, h, n, norm, act, bias, res, beyond):
    rng = np.random.default_rng(m + h)
    w1, w2 = _weights(rng, d, h, n)
    b1 = rng.standard_normal(h).astype(np.float32) if bias or beyond else None
    if beyond:
        b1[h - 1] = 300
    r = rng.standard_normal((m, h)).astype(np.float32) if res else None
    x = rng.standard_normal((m, d)).astype(np.float32)
    got, want, before, after = _mlp(x, w1, w2, b1, act, r, norm)
    assert before[1] == ("gemm_f16x3_pair_sums_tcgen05" if norm else "gemm_f16x3_pair_tcgen05")
    assert (before != after) == beyond
    assert _rel(got, want) <= 2e-6
