"""The attention kernel that takes keys in blocks of 128, against float64.

Bound, per output row: the projection is off by e = 5e-6 sum|x||w| (the bound of every split GEMM
here), the scores by scale * (e_q |k| + |q| e_k + 5e-6 |q||k|); a score off by d moves a softmax weight by at
most a factor exp(2 d), and the second product adds 5e-6 sum p|v| and p e_v."""
import numpy as np
import pytest
import torch

from altius_b200 import ir
from altius_b200.session import CudaSessionBuilder

pytestmark = pytest.mark.gpu


def _model(B, T, H, w, b, scale_op, projection):
    D = 64 * H
    g = ir.Graph()
    i64 = lambda v: g.new_init(np.asarray(v, np.int64))
    x = g.add_input("x", (B, T, D if projection else 3 * D))
    qkv = g.op("Add", g.op("MatMul", x, g.new_init(w)), g.new_init(b)) if projection else x
    q, k, v = g.add_node("Split", [qkv, i64([D, D, D])], 3, axis=2)

    def heads(t):
        t = g.op("Transpose", g.op("Reshape", t, i64([B, T, H, 64])), perm=[0, 2, 1, 3])
        return g.op("Reshape", t, i64([B * H, T, 64]))
    q, k, v = heads(q), heads(k), heads(v)
    s = g.op("MatMul", q, g.op("Transpose", k, perm=[0, 2, 1]))
    if scale_op:
        s = g.op(scale_op, s, g.new_init(np.array([0.125 if scale_op == "Mul" else 8.0], np.float32)))
    o = g.op("Reshape", g.op("MatMul", g.op("Softmax", s, axis=-1), v), i64([B, H, T, 64]))
    g.outputs.append(g.op("Reshape", g.op("Transpose", o, perm=[0, 2, 1, 3]), i64([B, T, D])))
    return ir.Model(g, 13)


# Tokens: two blocks and their edges, several with a last one of 1, 65, 76 and 128 keys, tiles of one row, sums of
# one and more runs of two blocks, in the last one a run of one block;
# items: fewer than blocks, a second round for some groups; "peaks" makes the running maximum move by more
# than the lazy threshold in every block.
@pytest.mark.parametrize("B,T,H,scale_op,projection,peaks", [
    (3, 129, 12, "Mul", True, False), (6, 200, 12, "Div", True, False), (12, 209, 12, "Mul", True, False),
    (9, 256, 12, "Mul", True, True), (2, 257, 2, "Mul", False, False), (1, 577, 12, "Mul", False, True),
    (5, 577, 12, "Mul", True, False), (3, 321, 1, "Div", False, True), (1, 1024, 3, None, False, False),
    (2, 513, 3, "Mul", False, True), (3, 1100, 2, "Mul", False, True), (20, 300, 12, "Mul", True, True)])
def test_flash_attention(cuda_lib, B, T, H, scale_op, projection, peaks):
    rng = np.random.default_rng(T + H)
    D = 64 * H
    x = rng.standard_normal((B, T, D if projection else 3 * D)).astype(np.float32)
    w = (0.05 * rng.standard_normal((D, 3 * D))).astype(np.float32)
    b = (0.1 * rng.standard_normal(3 * D)).astype(np.float32)
    if scale_op is None:
        x *= 0.35
    if peaks:                                   # keys that grow with their position
        x = x * (1 + 2 * np.arange(T, dtype=np.float32) / T)[None, :, None]
    sess = CudaSessionBuilder(_model(B, T, H, w, b, scale_op, projection)).build()
    try:
        kinds = [e["kind"] for e in sess.schedule()]
        assert kinds[-1] == "attention_flash_tcgen05", kinds
        got = sess.run([x])[0]
        assert [e["kind"] for e in sess.schedule()] == kinds      # no range fallback
    finally:
        sess.close()
    tx, tw = torch.from_numpy(x).double().cuda(), torch.from_numpy(w).double().cuda()
    if projection:
        qkv = tx @ tw + torch.from_numpy(b).double().cuda()
        e = 5e-6 * (tx.abs() @ tw.abs()) + 1e-6 * qkv.abs()
    else:
        qkv, e = tx, 5e-7 * tx.abs()            # the halves keep 22 bits
    split = lambda t: [u.reshape(B, T, H, 64).transpose(1, 2) for u in t.split(D, dim=2)]
    (q, k, v), (eq, ek, ev) = split(qkv), split(e)
    scale = 1.0 if scale_op is None else 0.125
    p = torch.softmax(scale * (q @ k.transpose(2, 3)), dim=-1)
    es = scale * (eq @ k.abs().transpose(2, 3) + q.abs() @ ek.transpose(2, 3) + 5e-6 * (q.abs() @ k.abs().transpose(2, 3)))
    want = (p @ v).transpose(1, 2).reshape(B, T, D).cpu().numpy()
    grow = torch.expm1(2 * es.amax(-1, keepdim=True))
    bound = (grow * (p @ v.abs()) + p @ ev + 5e-6 * (p @ v.abs())).transpose(1, 2).reshape(B, T, D).cpu().numpy()
    assert np.isfinite(got).all()
    err = np.abs(got - want)
    print("largest share of the bound", (err / bound).max(), "rel", np.linalg.norm(got - want) / np.linalg.norm(want))
    assert (err <= bound).all()


def test_values_beyond_the_fixed_scale_take_the_plan_without_it(cuda_lib):
    """Values of up to 4000 leave the fixed scale (255): the session goes on with the operators one by one, in
    the same mode; the products of constant weights stay on fp16 halves, which hold 65504."""
    B, T, H = 2, 300, 2
    D = 64 * H
    rng = np.random.default_rng(1)
    x = rng.standard_normal((B, T, D)).astype(np.float32)
    w = (rng.standard_normal((D, 3 * D)) / np.sqrt(D)).astype(np.float32)
    w[:, 2 * D:] *= 1000
    b = np.zeros(3 * D, np.float32)
    sess = CudaSessionBuilder(_model(B, T, H, w, b, "Mul", True)).build()
    try:
        assert "attention_flash_tcgen05" in [e["kind"] for e in sess.schedule()]
        for _ in range(2):
            got = sess.run([x])[0]
        kinds = [e["kind"] for e in sess.schedule()]
        assert "attention_flash_tcgen05" not in kinds and "softmax_scaled" in kinds
        assert any(k.startswith("gemm_f16x3") for k in kinds), kinds
    finally:
        sess.close()
    q, k, v = [u.reshape(B, T, H, 64).transpose(1, 2) for u in (torch.from_numpy(x).double() @ torch.from_numpy(w).double()).split(D, dim=2)]
    want = (torch.softmax(0.125 * (q @ k.transpose(2, 3)), dim=-1) @ v).transpose(1, 2).reshape(B, T, D).numpy()
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
