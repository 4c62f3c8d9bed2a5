"""The fp32 tensor-core path on operands of unequal magnitude.  The fp16 pairs are scaled by powers of two per row of Q and per
64-key tile of K and V, so that (a) a power of two taken out of a tensor leaves every bit of the result alone, and (b) small
numbers beside large ones keep fp32-grade precision; what scaling cannot hold goes to the exact kernel.  Reference: float64."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close_fp32, seeded
from gpu_util import sdpa_device
from tensorax_b200 import _lib

pytestmark = pytest.mark.gpu

B, H, S = 2, 4, 333


def inputs(dk, dv, seed=0):
    return [seeded(70 + seed + i, B, H, S, d).copy() for i, d in enumerate((dk, dk, dv))]


def exact64(q, k, v, mask=None):
    q, k, v = (x.astype(np.float64) for x in (q, k, v))
    s = q @ k.transpose(0, 1, 3, 2) / np.sqrt(q.shape[3])
    if mask is not None:
        s = s + mask
    e = np.exp(s - s.max(-1, keepdims=True))
    return (e @ v) / e.sum(-1, keepdims=True)


@pytest.mark.parametrize("dk,dv", [(64, 64), (80, 80), (128, 128), (40, 100)])
@pytest.mark.parametrize("masked", [False, True])
def test_powers_of_two_leave_every_bit_alone(dk, dv, masked):
    q, k, v = inputs(dk, dv)
    m = seeded(75, B, H, S, S) if masked else None
    base, _ = sdpa_device(q, k, v, mask=m)
    assert_close_fp32(base, oracle.sdpa_f32(q, k, v, m))
    for a in (-30, -7, 5, 30):
        f = np.float32(2.0 ** a)
        assert np.array_equal(sdpa_device(q * f, k / f, v, mask=m)[0], base)
        assert np.array_equal(sdpa_device(q, k, v * f, mask=m)[0], base * f)
    for j in range(S):                                        # rows of Q, each with its own factor, against K's
        q[:, :, j] *= np.float32(2.0 ** (j % 5 - 2))
    assert_close_fp32(sdpa_device(q, k, v, mask=m)[0], oracle.sdpa_f32(q, k, v, m))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("d", [64, 80, 128])
@pytest.mark.parametrize("f", [1e3, 1e4, 1e6])
def test_small_queries_and_large_keys(d, f, masked):
    q, k, v = inputs(d, d, 10)
    q, k = (q / f).astype(np.float32), (k * f).astype(np.float32)
    m = seeded(76, B, H, S, S) if masked else None
    assert_close_fp32(sdpa_device(q, k, v, mask=m)[0].astype(np.float64), exact64(q, k, v, m), atol=2e-6)
    assert_close_fp32(sdpa_device(k, q, v, mask=m)[0].astype(np.float64), exact64(k, q, v, m), atol=2e-6)


@pytest.mark.parametrize("d", [64, 80])
def test_small_head_and_small_tiles_of_v_beside_large_ones(d):
    q, k, v = inputs(d, d, 20)
    v[:, 1] *= np.float32(1e-4)
    v[0, 2] *= np.float32(1e-30)
    v[1, 3, 64:128] *= np.float32(1e-9)                       # a whole tile of keys
    got, ref = sdpa_device(q, k, v)[0], exact64(q, k, v)
    for b in range(B):
        for h in range(H):
            assert np.linalg.norm(got[b, h] - ref[b, h]) <= 2e-6 * np.linalg.norm(ref[b, h])
    v[:, :, 5] *= np.float32(1e-6)                            # one key of a tile: its row alone, where only it is seen
    m = np.full((B, H, S, S), -np.inf, np.float32)
    m[..., 5] = 0
    got, ref = sdpa_device(q, k, v, mask=m)[0], v[:, :, 5:6].astype(np.float64)
    for b in range(B):
        for h in range(H):
            assert np.linalg.norm(got[b, h] - ref[b, h]) <= 2e-6 * np.sqrt(S) * np.linalg.norm(ref[b, h])


@pytest.mark.parametrize("d", [64, 80, 128])
@pytest.mark.parametrize("f", [30.0, 1500.0, 1e6, 1e15])
def test_keys_of_small_weight_and_large_values(d, f):
    """One key of weight 1 and a tile of others whose weights times values still count: 1e-8 * 1500 and the like."""
    q, k, v = inputs(d, d, 50)
    q *= np.float32(0.1)
    v[:, :, 64:128] = np.float32(f) * (2 + v[:, :, 64:128].clip(-1, 1))
    m = np.full((B, H, S, S), -np.inf, np.float32)
    m[..., 5] = 0
    m[..., 64:128] = np.float32(np.log(1e-5 / f))
    ref = exact64(q, k, v, m)
    for e in (1.0, 2.0 ** -20):
        got = sdpa_device(q, k, v * np.float32(e), mask=m)[0]
        if f < 1e4:
            assert np.abs(got - ref * e).max() <= 2e-6 * e
        else:                                                 # too far apart: the exact kernel, with its own bound
            exact, _ = sdpa_device(q, k, v * np.float32(e), mask=m, flags=_lib.TX_SDPA_FORCE_SIMT)
            assert np.array_equal(got, exact) and np.abs(got - ref * e).max() <= 1e-5 * e


def test_garbage_behind_a_mask_and_mismatched_outliers():
    q, k, v = inputs(80, 80, 30)
    m = np.zeros((B, H, S, S), np.float32)
    m[..., 100:110] = -np.inf
    ref = exact64(q, k, v, m)
    for big in (1e6, 1e30):
        kb, vb = k.copy(), v.copy()
        vb[:, :, 100:110] = big
        assert_close_fp32(sdpa_device(q, k, vb, mask=m)[0].astype(np.float64), ref, atol=2e-6)
        kb[:, :, 100:110] = big
        assert_close_fp32(sdpa_device(q, kb, v, mask=m)[0].astype(np.float64), ref, atol=2e-6)
    # large values that never meet: 1e5 * 0 and 0 * 1e5
    q[..., 0], k[..., 0], q[..., 1], k[..., 1] = 1e5, 0, 0, 1e5
    assert_close_fp32(sdpa_device(q, k, v)[0].astype(np.float64), exact64(q, k, v), atol=2e-6)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_values_that_are_not_finite(which, bad):
    t = inputs(80, 80, 40)
    t[which][1, 2, 70, 3] = bad
    exact, _ = sdpa_device(*t, flags=_lib.TX_SDPA_FORCE_SIMT)
    assert np.array_equal(sdpa_device(*t)[0], exact, equal_nan=True)


@pytest.mark.parametrize("Hq,Hkv,Sk", [(6, 2, 64), (4, 1, 65), (3, 3, 1025)])
def test_factors_follow_grouped_heads_lengths_and_partial_tiles(Hq, Hkv, Sk):
    q, k, v = seeded(80, 2, Hq, 300, 64), seeded(81, 2, Hkv, Sk, 64), seeded(82, 2, Hkv, Sk, 64)
    for j in range(0, Sk, 64):
        k[:, :, j:j + 64] *= np.float32(2.0 ** (j // 64 % 3 - 1))
        v[:, :, j:j + 64] *= np.float32(2.0 ** (j // 64 % 5 - 2))
    for h in range(Hkv):
        v[:, h] *= np.float32(10.0 ** h)
    lens = [Sk, max(1, Sk - 20)]
    got, _ = sdpa_device(q, k, v, causal=True, kv_lens=lens)
    ref = oracle.sdpa_structured(q, k, v, causal=True, kv_lens=lens)
    for h in range(Hq):
        assert np.abs(got[:, h] - ref[:, h]).max() <= 1e-5 * 10.0 ** (h // (Hq // Hkv)) * 4


@pytest.mark.parametrize("shape,causal", [((2, 16, 1600, 128), True), ((1, 3, 2400, 64), False)])
def test_a_declined_call_costs_what_the_exact_kernel_costs(shape, causal):
    """The stand-in behind the tensor-core kernel uses the whole chip when it has to work: at most half as much again as
    the exact kernel by itself, split pass included (best of five each; it was four times at the first shape)."""
    B, H, S, d = shape
    lib = _lib.load()
    q, k, v = (torch.randn(shape, device="cuda") for _ in range(3))
    v[0, 0, 0] *= 1e-6
    out = torch.zeros(shape, device="cuda")

    def best(flags):
        desc = _lib.SdpaDesc(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), mask=None, kv_lens=None, out=out.data_ptr(), batch=B,
                             q_heads=H, kv_heads=H, seq_q=S, seq_k=S, d_k=d, d_v=d, dtype=_lib.TX_DTYPE_F32, causal=int(causal),
                             flags=flags, stream=None, lse=None)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            _lib.check(lib.tx_sdpa_forward(ctypes.byref(desc)))
            b.record()
            _lib.check(lib.tx_sdpa_finish(None))
            times.append(a.elapsed_time(b))
        return min(times[1:]), out.clone()

    exact, ref = best(_lib.TX_SDPA_FORCE_SIMT)
    declined, got = best(0)
    assert torch.equal(got, ref)
    assert declined <= 1.5 * exact, (declined, exact)
