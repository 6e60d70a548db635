"""CPU-only tests of the session library's host side: the C ABI surface, shape
inference, lowering / fusion and the arena plan (sessions built with
`plan_only`, which creates nothing on a GPU), and error reporting at create time."""
import collections
import os
import re

import numpy as np
import pytest

from altius_b200 import configs, ir, session
from altius_b200.session import CudaSessionBuilder, SessionError
from helpers import run_oracle, single_op_model

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def plan(model, fuse=True):
    return CudaSessionBuilder(model).with_plan_only(True).with_fusion(fuse).build()


def test_library_exports_every_declared_symbol():
    header = open(os.path.join(ROOT, "include", "altius_session_cuda.h")).read()
    declared = set(re.findall(r"\b(altius_(?:cuda|model)_\w+)\s*\(", header))
    assert declared == set(session.ABI_SYMBOLS)
    lib = session.load_library()
    for name in declared:
        assert hasattr(lib, name), name


def test_plan_only_session_refuses_to_run():
    model, feeds = configs.mnist_cnn()
    s = plan(model)
    with pytest.raises(SessionError) as e:
        s.run(list(feeds.values()))
    assert e.value.status == 5


@pytest.mark.parametrize("fn,kw", [(configs.mnist_cnn, {}), (configs.micrograph, dict(batch=2)),
                                   (configs.vit_base_16, dict(batch=2, depth=1)),
                                   (configs.deit_small_distilled_16, dict(batch=2, depth=1)),
                                   (configs.mobilenet_v3_large, dict(batch=1))])
def test_inferred_output_shapes_match_the_oracle(fn, kw):
    model, feeds = fn(**kw)
    s = plan(model)
    want = run_oracle(model, feeds.values(), threads=8, sgemm="openblas")
    assert [tuple(shape) for shape, _ in s.output_info] == [w.shape for w in want]
    assert [np.dtype(dt) for _, dt in s.output_info] == [w.dtype for w in want]


def test_fusion_folds_the_expected_chains():
    model, _ = configs.micrograph(batch=2)
    kinds = collections.Counter(e["kind"] for e in plan(model).schedule())
    assert kinds == {"layer_norm_bias_gelu_residual": 1, "softmax_scaled": 1, "reduce_mean_max": 1}
    assert plan(model, fuse=False).launches_per_run == 8
    # algorithmic bytes of the fused kernels at the benchmark's size
    model, _ = configs.micrograph(batch=64)
    by_kind = {e["kind"]: e for e in plan(model).schedule()}
    x_bytes = 64 * 197 * 768 * 4
    assert abs(by_kind["layer_norm_bias_gelu_residual"]["bytes"] - 2 * x_bytes) < 1e5
    assert by_kind["softmax_scaled"]["bytes"] == 2 * 64 * 12 * 197 * 197 * 4
    assert by_kind["reduce_mean_max"]["bytes"] == x_bytes + 2 * 64 * 197 * 4   # one pass over X for both

    model, _ = configs.vit_base_16(batch=2, depth=2)
    kinds = collections.Counter(e["kind"] for e in plan(model).schedule())
    gemms = sum(v for k, v in kinds.items() if k.startswith("gemm"))
    assert gemms == 2 * 4 + 2          # per layer: qkv, proj, mlp1, mlp2; patch embed; head
    # Split/Reshape/Transpose/QK^T/scale/Softmax/PV/merge in one kernel: with few heads a block per tile of
    # 128 queries, else a block per head
    assert kinds["attention_flash_tcgen05"] == 2
    assert kinds["gemm_fp32_rows"] == 1           # the head: two rows
    big = collections.Counter(e["kind"] for e in plan(configs.vit_base_16(batch=32, depth=2)[0]).schedule())
    assert big["attention_tma_tcgen05"] == 2 and big["gemm_f16x3_pair_tcgen05"] == 2 * 4 + 1
    assert not any(k in kinds for k in ("split_copy", "transpose_copy", "softmax", "softmax_scaled"))
    unfused = collections.Counter(e["kind"] for e in plan(model, fuse=False).schedule())
    assert unfused["split_copy"] == 6 and unfused["softmax"] == 2
    assert kinds["layer_norm"] == 2 * 2 + 1
    assert kinds.get("binary_Add", 0) == 1        # only the position embedding stays a kernel
    assert "unary_gelu" not in kinds

    model, _ = configs.mobilenet_v3_large(batch=1)
    kinds = collections.Counter(e["kind"] for e in plan(model).schedule())
    assert "unary_hard_sigmoid" not in kinds and "unary_relu" not in kinds and "binary_Add" not in kinds
    # Squeeze-excite: pool and both products in one kernel, the gate in the operand loads of the
    # pointwise convolution behind it.
    assert kinds["binary_Mul"] == 0 and kinds["squeeze_excite"] == 8 and kinds["global_avg_pool"] == 1
    assert kinds["conv_depthwise"] == 15
    assert kinds["gemm_fp32_rows"] == 2                # the 1 x 1 head convolution and the classifier
    assert kinds["conv_fp32_simt"] + kinds["gemm_tf32x3_tcgen05"] == 31

    # At the benchmark's batch all convolutions run on the tensor cores with the planes read in place.
    model, _ = configs.mobilenet_v3_large(batch=32)
    steps = plan(model).schedule()
    kinds = collections.Counter(e["kind"] for e in steps)
    assert kinds["binary_Mul"] == 0 and kinds["im2col"] == 0 and kinds["transpose_copy"] == 0
    assert kinds["gemm_tf32x3_tcgen05"] == 31 and kinds["squeeze_excite"] == 8
    assert collections.Counter(e["kind"] for e in plan(model, fuse=False).schedule())["binary_Mul"] >= 8
    assert "filter_pack" not in kinds                  # prepared once at create, not per run
    cuda_cores = CudaSessionBuilder(model).with_plan_only(True).with_gemm_mode(1).build().schedule()
    assert sum(e["kind"] == "gemm_fp32_simt" for e in cuda_cores) == 49
    assert not any(e["kind"].endswith("tcgen05") for e in cuda_cores)


def test_the_schedule_names_the_kernel_of_a_product():
    """Behind a LayerNormalization: the few-row kernel, beyond a round of it CTA pairs with short accumulators, or long ones."""
    def kind(m, d, n):
        g = ir.Graph()
        one, zero = g.new_init(np.ones(d, np.float32)), g.new_init(np.zeros(d, np.float32))
        h = g.op("LayerNormalization", g.add_input("x", (m, d)), one, zero, axis=-1, epsilon=1e-6, stash_type=1)
        g.outputs.append(g.op("MatMul", h, g.new_init(np.zeros((d, n), np.float32))))
        return plan(ir.Model(g, 13)).schedule()[-1]["kind"]
    assert kind(197, 768, 2304) == kind(2885, 768, 768) == "gemm_f16x3_cluster_tcgen05"
    assert kind(3152, 768, 768) == kind(12672, 384, 384) == "gemm_f16x3_pair_sums_tcgen05"
    assert kind(6304, 768, 2304) == "gemm_f16x3_pair_tcgen05"


def test_flops_of_vit_match_the_published_count():
    model, _ = configs.vit_base_16(batch=1, depth=12)
    flops = sum(e["flops"] for e in plan(model).schedule())
    assert abs(flops / 1e9 - 35.13) < 0.05


def test_arena_reuses_memory():
    model, _ = configs.vit_base_16(batch=4, depth=12)
    # gemm_mode 1: no transposed / split weight copies live in the arena
    s = CudaSessionBuilder(model).with_plan_only(True).with_gemm_mode(1).build()
    total = 0
    for v in range(len(model.graph.values)):
        if v in model.graph.inits:
            continue
        shape, dt = s.value_info(v)
        total += int(np.prod(shape)) * np.dtype(dt).itemsize
    assert s.arena_bytes < total / 8


def test_constant_only_nodes_are_not_in_the_per_run_schedule():
    model, _ = configs.mnist_cnn()
    kinds = [e["kind"] for e in plan(model).schedule()]
    assert kinds == ["conv_fp32_simt", "max_pool"] * 2 + ["gemm_fp32_rows"]


def test_convolutions_beyond_the_direct_kernels_go_through_the_gemm():
    """More than 4096 products per result: a column buffer, or planes read as they are / transposed."""
    def conv(c, h, oc, k):
        x, w = np.zeros((4, c, h, h), np.float32), np.zeros((oc, c, k, k), np.float32)
        return [e["kind"] for e in plan(single_op_model("Conv2d", [x], [w, np.zeros(oc, np.float32)], kernel_shape=[k, k],
                                                        strides=[1, 1], padding=[k // 2] * 4, dilations=[1, 1], group=1,
                                                        auto_pad="")).schedule()]
    assert conv(512, 14, 64, 3) == ["im2col", "gemm_tf32x3_tcgen05"]
    assert conv(4100, 8, 64, 1) == ["gemm_tf32x3_tcgen05"]
    assert conv(4100, 7, 64, 1) == ["transpose_copy", "gemm_tf32x3_tcgen05"]


def _mlp_behind_layer_norm(m, d, n):
    g = ir.Graph()
    f = lambda *shape: g.new_init(np.zeros(shape, np.float32))
    h = g.op("LayerNormalization", g.add_input("x", (m, d)), f(d), f(d), axis=-1, epsilon=1e-6, stash_type=1)
    h = g.op("Gelu", g.op("Add", g.op("MatMul", h, f(d, n)), f(n)))
    g.outputs.append(g.op("Add", g.op("MatMul", h, f(n, d)), f(d)))
    return ir.Model(g, 13)


@pytest.mark.parametrize("m", [1, 32, 33, 65, 128, 129, 197, 577, 1386, 6304])
def test_products_of_any_size_lower(m):
    """Whoever writes an operand as halves and the product that takes it decide by one rule: around every
    limit of it (operations, rows, K and N off the multiples) the graph lowers, the operand's producer included."""
    for d in (64, 72, 100, 128, 200, 384, 1032):
        for n in (32, 64, 66, 128, 256, 1024):
            kinds = [e["kind"] for e in plan(_mlp_behind_layer_norm(m, d, n)).schedule()]
            assert sum(k.startswith("gemm") for k in kinds) == 2, (m, d, n, kinds)


@pytest.mark.parametrize("dim,heads", [(64, 1), (128, 2), (192, 3), (256, 4)])
def test_narrow_transformers_lower(dim, heads):
    for batch in (1, 2, 3, 4, 9):
        for px in (48, 96, 224):
            plan(configs.vision_transformer(batch, dim, 2, heads, 4 * dim, 1, img=px)[0])


@pytest.mark.parametrize("px,batch,kind", [(96, 1, "attention_fused"), (96, 32, "attention_fused"), (112, 8, "attention_fused"),
                                           (128, 32, "attention_tma_tcgen05"), (224, 32, "attention_tma_tcgen05"),
                                           (224, 1, "attention_flash_tcgen05"), (240, 1, "attention_flash_tcgen05"),
                                           (240, 32, "attention_flash_tcgen05"), (384, 2, "attention_flash_tcgen05")])
def test_attention_kernel_by_tokens_and_heads(px, batch, kind):
    """fp32 up to 64 tokens; halves of the projection by TMA, a block per head up to 208 and per tile of queries
    with few heads and beyond."""
    model, _ = configs.vision_transformer(batch, 384, 1, 6, 1536, 1, img=px)
    kinds = [e["kind"] for e in plan(model).schedule()]
    assert [k for k in kinds if k.startswith("attention")] == [kind]
    assert "softmax_scaled" not in kinds and "act_f16_split" not in kinds[kinds.index(kind):]


@pytest.mark.parametrize("toggle,batch", [("ALTIUS_CUDA_NO_FUSED_SPLIT", 2), ("ALTIUS_CUDA_NO_ATTENTION_TMA", 2), (None, 0)])
def test_long_attention_without_its_kernel_is_separate_operators(monkeypatch, toggle, batch):
    """Beyond 256 tokens only the kernel on halves of the projection takes the fused chain; where these are not
    planned, or there is nothing to compute, the operators stay."""
    if toggle:
        monkeypatch.setenv(toggle, "1")
    B, T, H = batch, 300, 2
    D = 64 * H
    g = ir.Graph()
    i64 = lambda v: g.new_init(np.asarray(v, np.int64))
    qkv = g.op("MatMul", g.add_input("x", (B, T, D)), g.new_init(np.zeros((D, 3 * D), np.float32)))
    q, k, v = g.add_node("Split", [qkv, i64([D, D, D])], 3, axis=2)
    heads = lambda t: g.op("Reshape", g.op("Transpose", g.op("Reshape", t, i64([B, T, H, 64])), perm=[0, 2, 1, 3]), i64([B * H, T, 64]))
    q, k, v = heads(q), heads(k), heads(v)
    s = g.op("Softmax", g.op("MatMul", q, g.op("Transpose", k, perm=[0, 2, 1])), axis=-1)
    o = g.op("Reshape", g.op("MatMul", s, v), i64([B, H, T, 64]))
    g.outputs.append(g.op("Reshape", g.op("Transpose", o, perm=[0, 2, 1, 3]), i64([B, T, D])))
    kinds = [e["kind"] for e in plan(ir.Model(g, 13)).schedule()]
    assert "softmax" in kinds and not any(k.startswith("attention") for k in kinds), kinds


@pytest.mark.parametrize("m,k,n,rows", [(1, 1024, 32000, True), (4, 4096, 4096, True), (32, 768, 1000, True), (24, 768, 3072, True),
                                         (32, 768, 3072, False), (9, 1024, 32000, False), (16, 4096, 4096, False), (33, 768, 1000, False)])
def test_few_rows_take_the_kernel_that_streams_the_weights_while_they_are_small(m, k, n, rows):
    x, w = np.zeros((m, k), np.float32), np.zeros((n, k), np.float32)
    kinds = [e["kind"] for e in plan(single_op_model("Gemm", [x], [w], alpha=1.0, beta=1.0, trans_a=False, trans_b=True)).schedule()]
    assert kinds == (["gemm_fp32_rows"] if rows else ["gemm_f16x3_tcgen05"])


def test_errors_are_reported_at_create():
    a = np.zeros((1, 3, 28, 28), np.float32)
    b = np.zeros((3, 1, 2), np.float32)
    with pytest.raises(SessionError) as e:
        plan(single_op_model("Add", [a, b]))
    assert e.value.status == 2 and "broadcast" in str(e.value)
    with pytest.raises(SessionError) as e:
        plan(single_op_model("Clip", [a]))
    assert e.value.status == 3 and "Kernel not implemented" in str(e.value)
    x = np.zeros((2, 3, 4), np.float32)
    with pytest.raises(SessionError) as e:
        plan(single_op_model("Softmax", [x], axis=1))
    assert e.value.status == 3
    with pytest.raises(SessionError) as e:                 # dangling value id
        g = ir.Graph()
        i = g.add_input("x", (2, 2))
        g.nodes.append(ir.Node("ReLU", [i], [99]))
        g.outputs.append(99)
        plan(ir.Model(g))
    assert e.value.status == 1
    with pytest.raises(RuntimeError):
        session.InferenceSession(configs.mnist_cnn()[0], backend="interpreter")


def test_resize_and_expand_shapes():
    """shape.rs:148-160 (Expand) and :209-254 (Resize: sizes, or floor(dims * scales) for the
    asymmetric / nearest / floor pattern only)."""
    x = np.zeros((2, 3, 10, 10), np.float32)
    none = np.zeros(0, np.float32)
    s = plan(single_op_model("Resize", [x], [none, none, np.array([2, 3, 25, 15], np.int64)], mode="linear"))
    assert s.output_info[0][0] == (2, 3, 25, 15)
    assert [e["kind"] for e in s.schedule()] == ["resize_bilinear"]
    s = plan(single_op_model("Resize", [x], [none, np.array([1, 1, 2.5, 2.5], np.float32)], mode="nearest",
                             coordinate_transformation_mode="asymmetric", nearest_mode="floor"))
    assert s.output_info[0][0] == (2, 3, 25, 25)
    with pytest.raises(SessionError) as e:               # 3-input form outside the one supported pattern
        plan(single_op_model("Resize", [x], [none, np.array([1, 1, 2, 2], np.float32)], mode="linear",
                             coordinate_transformation_mode="asymmetric", nearest_mode="floor"))
    assert e.value.status == 3 and "Unsupported pattern" in str(e.value)
    i = np.zeros((1, 1, 1, 7), np.int64)
    s = plan(single_op_model("Expand", [i], [np.array([1, 1, 4, 7], np.int64)]))
    assert s.output_info[0][0] == (1, 1, 4, 7) and [e["kind"] for e in s.schedule()] == ["expand_copy"]
    with pytest.raises(SessionError) as e:
        plan(single_op_model("Expand", [np.zeros((3,), np.float32)], [np.array([2, 4], np.int64)]))
    assert e.value.status == 2


def test_create_without_a_gpu_fails_loudly():
    lib = session.load_library()
    if lib.altius_cuda_device_count() > 0:
        pytest.skip("a GPU is visible")
    model, _ = configs.mnist_cnn()
    with pytest.raises(SessionError) as e:
        CudaSessionBuilder(model).build()
    assert e.value.status == 5 and "no CPU fallback" in str(e.value)
