"""tx_mha_forward_f32 -- the layer as one call, projections on fp16 pairs (csrc/gemm_x3.cuh) -- at the edges of its tiles:
partial k-stages, partial row and column tiles, rows longer than the split pass keeps in registers, more than one
accumulator chunk, separate and shared inputs."""
import numpy as np
import pytest

import oracle
import tensorax_b200 as ts
from conftest import assert_close_fp16, assert_close_fp32, seeded
from tensorax_b200 import _C
from tensorax_b200.nn.attention import MultiHeadAttention

pytestmark = pytest.mark.gpu

NAMES = ("q", "k", "v", "out")


def layer(E, H, bias, **kw):
    mha = MultiHeadAttention(E, H, bias=bias, **kw).cuda()
    for i, n in enumerate(NAMES):
        mha._parameters[n + "_weight"] = ts.Tensor(seeded(50 + i, E, E) / np.sqrt(E), device="cuda")
        if bias:
            mha._parameters[n + "_bias"] = ts.Tensor(0.1 * seeded(60 + i, E), device="cuda")
    return mha, {n: p.numpy() for n, p in mha._parameters.items() if p is not None}


@pytest.mark.parametrize("B,Sq,Sk,E,H,bias", [
    (1, 1, 1, 8, 1, True), (2, 5, 7, 40, 2, True), (1, 129, 129, 72, 3, False), (3, 43, 43, 200, 5, True),
    (2, 130, 65, 256, 4, True), (1, 260, 260, 320, 5, False), (1, 70, 70, 1088, 17, True), (2, 64, 300, 512, 8, True),
])
def test_layer_against_the_composition_of_cpu_ops(B, Sq, Sk, E, H, bias):
    mha, params = layer(E, H, bias)
    x, y = seeded(1, B, Sq, E), seeded(2, B, Sk, E)
    xt, yt = ts.Tensor(x, device="cuda"), ts.Tensor(y, device="cuda")
    names = [mha._parameters[n + "_weight"]._c_tensor for n in NAMES]
    biases = [mha._parameters[n + "_bias"]._c_tensor if bias else None for n in NAMES]
    assert _C.multi_head_attention(xt._c_tensor, yt._c_tensor, yt._c_tensor, names, biases, H) is not None
    got = mha(xt, yt, yt).numpy()
    assert_close_fp32(got, oracle.mha_forward_f32(x, y, y, params, H, None), atol=2e-5)   # four chained fp32 stages
    assert np.array_equal(got, mha(xt, yt, yt).numpy())
    if Sq == Sk:
        same = mha(xt, xt, xt, causal=True, kv_lens=[max(1, Sk - 3)] * B).numpy()
        i, j = np.arange(Sq)[:, None], np.arange(Sk)[None, :]
        m = np.where((j <= i) & (j < max(1, Sk - 3)), 0.0, -np.inf).astype(np.float32)
        m = np.ascontiguousarray(np.broadcast_to(m, (B, H, Sq, Sk)))
        ref = oracle.mha_forward_f32(x, x, x, params, H, m)
        assert_close_fp32(same, ref, atol=2e-5)
        assert_close_fp32(mha(xt, xt, xt, ts.Tensor(m, device="cuda")).numpy(), ref, atol=2e-5)


@pytest.mark.parametrize("E,H", [(128, 2), (256, 2)])
def test_fp16_attention_step(E, H):
    mha, params = layer(E, H, True, attention_dtype="float16")
    x = seeded(3, 2, 150, E)
    got = mha(ts.Tensor(x, device="cuda"), ts.Tensor(x, device="cuda"), ts.Tensor(x, device="cuda")).numpy()
    assert_close_fp16(got, oracle.mha_forward_f32(x, x, x, params, H, None))


def test_rows_of_any_magnitude_keep_their_relative_precision():
    """Row scaling by powers of two: rows of 1e-20, 1 and 1e20 side by side, each as exact as the others.  (Without biases and
    with one key, the layer is (x Wv^T) Wo^T; float64 reference; bound: 22-bit operands and fp32 sums over E = 256,
    twice: 2 * 256 * 2^-23 worst, 1e-6 in norm.)"""
    E, H = 256, 4
    mha, params = layer(E, H, False)
    x = seeded(4, 3, 1, E) * np.array([1e-20, 1.0, 1e20]).reshape(3, 1, 1)
    x = x.astype(np.float32)
    q = ts.Tensor(seeded(5, 3, 1, E), device="cuda")
    xt = ts.Tensor(x, device="cuda")
    got = mha(q, q, xt).numpy()
    ref = x.astype(np.float64) @ params["v_weight"].astype(np.float64).T @ params["out_weight"].astype(np.float64).T
    for b in range(3):
        assert np.linalg.norm(got[b] - ref[b]) <= 1e-6 * np.linalg.norm(ref[b])


@pytest.mark.parametrize("E,H", [(512, 8), (384, 3), (240, 5)])
@pytest.mark.parametrize("scale", [1.0, 1e-4, 1e6])
def test_halves_written_by_the_projections(E, H, scale):
    """From the projections into the attention step (head dims 64, 128, 48; partial row tiles), with values of any size.
    Bound: four chained fp32 stages, 2e-5 of the result."""
    mha, params = layer(E, H, False)
    x, y = seeded(6, 2, 301, E), (scale * seeded(7, 2, 333, E)).astype(np.float32)
    k = seeded(8, 2, 333, E)
    got = mha(*(ts.Tensor(t, device="cuda") for t in (x, k, y))).numpy()
    ref = oracle.mha_forward_f32(x, k, y, params, H, None)
    assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("a,b", [(36, -30), (-36, 30), (34, -8)])
def test_products_in_range_of_operands_near_its_ends(a, b):
    """Inputs of 1e36 and value weights of 1e-30, or the other way round: the projections' results are ordinary numbers."""
    E, H = 64, 2
    mha, params = layer(E, H, False)
    w = (params["v_weight"] * np.float32(10.0) ** b).astype(np.float32)
    mha._parameters["v_weight"] = ts.Tensor(w, device="cuda")
    q, x = seeded(12, 2, 5, E), (seeded(13, 2, 1, E) * 10.0 ** a / 8).astype(np.float32)
    got = mha(ts.Tensor(q, device="cuda"), ts.Tensor(q[:, :1].copy(), device="cuda"), ts.Tensor(x, device="cuda")).numpy()
    ref = x.astype(np.float64) @ w.astype(np.float64).T @ params["out_weight"].astype(np.float64).T
    assert np.linalg.norm(got - ref) <= 2e-6 * np.linalg.norm(np.broadcast_to(ref, got.shape))


@pytest.mark.parametrize("E,H,Sq,Sk", [(72, 3, 70, 70), (256, 4, 130, 65), (1088, 17, 33, 40)])
def test_outliers_inside_a_row(E, H, Sq, Sk):
    """Elements far below their row's largest, which the weights leave out: the projections see the small ones alone.  Float64
    reference of the layer with one key per query row's batch element left visible; bound: fp32 sums over E, twice."""
    mha, params = layer(E, H, True)
    w = params["v_weight"].copy()
    w[:, 0] = 0
    mha._parameters["v_weight"] = ts.Tensor(w, device="cuda")
    x, y, z = seeded(9, 2, Sq, E), seeded(10, 2, Sk, E), seeded(11, 2, Sk, E)
    z[..., 0] = 1e9
    got = mha(*(ts.Tensor(t, device="cuda") for t in (x, y, z)), kv_lens=[1, 1]).numpy()
    v0 = z[:, :1].astype(np.float64) @ w.astype(np.float64).T + params["v_bias"]
    ref = np.broadcast_to(v0 @ params["out_weight"].astype(np.float64).T + params["out_bias"], got.shape)
    assert np.linalg.norm(got - ref) <= 5e-6 * np.linalg.norm(ref)


def test_outliers_in_the_weights_and_in_the_attention_result():
    """Whole weight rows of small numbers beside one large one that the input leaves out, and a head of the attention result
    far above all others that the output weights leave out (fp32 and fp16 attention results of the layer alike)."""
    E, H, S = 128, 4, 60
    mha, params = layer(E, H, False)
    x = seeded(14, 2, S, E)
    x[..., 5] = 0
    w = params["v_weight"].copy()
    w[:, 5] = 1e9
    mha._parameters["v_weight"] = ts.Tensor(w, device="cuda")
    got = mha(*(ts.Tensor(x, device="cuda"),) * 3).numpy()
    ref = oracle.mha_forward_f32(x, x, x, dict(params, v_weight=w), H, None)
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    mha, params = layer(E, H, False)
    w, o = params["v_weight"].copy(), params["out_weight"].copy()
    w[:32] *= np.float32(1e9)
    o[:, :32] = 0
    mha._parameters["v_weight"], mha._parameters["out_weight"] = ts.Tensor(w, device="cuda"), ts.Tensor(o, device="cuda")
    got = mha(*(ts.Tensor(x, device="cuda"),) * 3).numpy()
    ref = oracle.mha_forward_f32(x, x, x, dict(params, v_weight=w, out_weight=o), H, None)
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
