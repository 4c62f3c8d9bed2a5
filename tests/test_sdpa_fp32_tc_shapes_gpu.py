"""The fp32 tensor-core kernel (csrc/sdpa_tc_x3.cuh) at head dims that fill its operand panels in part, at d_k != d_v, and
with the dense additive mask, against the oracle; bounds: 1e-5, the fp32 figure."""
import numpy as np
import pytest

import oracle
from conftest import assert_close_fp32, seeded
from gpu_util import sdpa_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv", [(4, 4), (12, 20), (32, 32), (40, 40), (68, 68), (80, 80), (96, 96), (124, 128), (128, 32), (16, 100)])
@pytest.mark.parametrize("Sq,Sk,causal", [(129, 193, False), (200, 200, True)])
def test_partly_filled_panels(dk, dv, Sq, Sk, causal):
    B, Hq, Hkv = 2, 4, 2
    q, k, v = seeded(1, B, Hq, Sq, dk), seeded(2, B, Hkv, Sk, dk), seeded(3, B, Hkv, Sk, dv)
    lens = [Sk, Sk - 70]
    outs, tc = sdpa_device(q, k, v, causal=causal, kv_lens=lens, repeats=2)
    assert tc
    assert np.array_equal(outs[0], outs[1])
    assert_close_fp32(outs[0], oracle.sdpa_structured(q, k, v, causal=causal, kv_lens=lens))


@pytest.mark.parametrize("d", [32, 64, 80, 128])
@pytest.mark.parametrize("Sq,Sk", [(128, 64), (130, 260), (257, 323), (64, 1001)])     # rows of the mask 16-byte aligned and not
@pytest.mark.parametrize("kind", ["causal", "random", "rows"])
def test_dense_masks(d, Sq, Sk, kind):
    B, H = 4, 6                                          # enough rows for none to go to the decoding kernel
    q, k, v = seeded(11, B, H, Sq, d), seeded(12, B, H, Sk, d), seeded(13, B, H, Sk, d)
    if kind == "causal":
        m = np.where(np.arange(Sk)[None, :] <= np.arange(Sq)[:, None], 0.0, -np.inf)
        m = np.broadcast_to(m, (B, H, Sq, Sk))
    else:
        m = 2.0 * seeded(14, B, H, Sq, Sk)
        if kind == "rows":
            m[:, :, 3] = -np.inf                         # 0/0 rows
            m[:, 1, Sq - 1] = np.finfo(np.float32).min   # uniform average
            m[0, 0, 5, : Sk // 2] = -1e9
    m = np.ascontiguousarray(m, dtype=np.float32)
    got, tc = sdpa_device(q, k, v, mask=m)
    assert tc
    with np.errstate(all="ignore"):
        ref = oracle.sdpa_f32(q, k, v, m)
    assert_close_fp32(got, ref)


def test_small_values_of_v_keep_their_relative_precision():
    """A hi / lo pair is exact to 2^-25 absolutely: a V of 1e-4 would lose four digits, so it goes to the exact kernel."""
    q, k, v = seeded(21, 1, 2, 200, 80), seeded(22, 1, 2, 200, 80), 1e-4 * seeded(23, 1, 2, 200, 80)
    got, _ = sdpa_device(q, k, v)
    ref = oracle.sdpa_f32(q, k, v.astype(np.float32))
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
