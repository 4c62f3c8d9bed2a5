"""Few query rows per K/V head (csrc/sdpa_decode.cuh) against the oracle at the sizes where the kernel's partitions end:
one key, less than a stage, shares that leave later CTAs of a cluster without keys, one row more than a row group."""
import numpy as np
import pytest

import oracle
from conftest import FP16_ATOL, assert_close_fp32, seeded
from gpu_util import sdpa_device
from tensorax_b200 import _lib

pytestmark = pytest.mark.gpu

CASES = [
    # B, Hq, Hkv, Sq, Sk, causal, kv_lens, mask
    (1, 1, 1, 1, 1, False, None, False),
    (2, 4, 1, 1, 129, False, [129, 1], False),
    (3, 8, 1, 1, 1000, False, [1000, 0, 31], False),      # batch 1 sees no key: NaN rows, as the reference
    (1, 9, 1, 1, 4097, False, None, False),               # one row more than a row group
    (2, 4, 4, 1, 300, False, None, True),                 # the reference's padding-mask form
    (1, 2, 1, 3, 200, True, None, False),                 # several rows per head, causal
    (40, 8, 4, 1, 333, False, "ramp", False),             # lengths on the device; from the host: test_kv_lens_host_gpu.py
]


@pytest.mark.parametrize("dtype", [np.float32, np.float16])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_decode_against_oracle(case, d, dtype):
    B, Hq, Hkv, Sq, Sk, causal, lens, masked = CASES[case]
    if lens == "ramp":
        lens = [1 + (7 * i) % Sk for i in range(B)]
    q = seeded(10 + case, B, Hq, Sq, d).astype(dtype)
    k, v = (seeded(20 + case + j, B, Hkv, Sk, d).astype(dtype) for j in range(2))
    wide = [x.astype(np.float32) for x in (q, k, v)]
    if masked:
        m = np.where(np.arange(Sk) < 150, 0.0, -np.inf).astype(np.float32)
        m = np.ascontiguousarray(np.broadcast_to(m, (B, Hq, Sq, Sk)))
        got, _ = sdpa_device(q, k, v, mask=m)
        ref = oracle.sdpa_f32(*wide, m)
    else:
        outs, _ = sdpa_device(q, k, v, causal=causal, kv_lens=lens, repeats=2)
        got = outs[0]
        assert np.array_equal(got.view(np.uint32), outs[1].view(np.uint32))
        ref = oracle.sdpa_structured(*wide, causal=causal, kv_lens=lens)
    # fp32 arithmetic on both input types; fp16 calls of less than 128 keys stay on the tensor cores
    assert_close_fp32(got, ref, **({"atol": FP16_ATOL} if dtype == np.float16 and Sk < 128 else {}))


def test_statistics_and_fp16_result():
    B, Hq, Hkv, Sk, d = 2, 8, 2, 700, 128
    q = seeded(1, B, Hq, 1, d).astype(np.float16)
    k, v = (seeded(2 + j, B, Hkv, Sk, d).astype(np.float16) for j in range(2))
    got, lse, _ = sdpa_device(q, k, v, flags=_lib.TX_SDPA_OUT_F16, want_lse=True)
    k32, q32 = np.repeat(k.astype(np.float64), Hq // Hkv, axis=1), q.astype(np.float64)
    s = (q32 @ k32.transpose(0, 1, 3, 2)) / np.sqrt(d)
    np.testing.assert_allclose(lse, np.log2(np.exp(s).sum(-1)), rtol=0, atol=1e-5)
    ref = oracle.sdpa_structured(*(x.astype(np.float32) for x in (q, k, v)))
    assert np.abs(got.astype(np.float32) - ref).max() <= FP16_ATOL


def test_dense_mask_of_lowest_floats_is_a_uniform_average():
    """The reference starts its running max at -FLT_MAX: a row masked with it everywhere averages V."""
    q, k, v = seeded(5, 1, 2, 1, 64), seeded(6, 1, 2, 40, 64), seeded(7, 1, 2, 40, 64)
    m = np.full((1, 2, 1, 40), np.finfo(np.float32).min, np.float32)
    got, _ = sdpa_device(q, k, v, mask=m)
    assert_close_fp32(got, oracle.sdpa_f32(q, k, v, m))
