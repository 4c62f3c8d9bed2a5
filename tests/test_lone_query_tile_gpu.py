"""A call whose last pair of 128-row query tiles has only one live tile, with many key tiles and many CTAs: the first
QK^T of such a CTA can complete before its producer warp reaches its loop, which once made the producer wait for a
release that had already happened (and the call give up after two seconds)."""
import numpy as np
import pytest

import oracle
from conftest import assert_close_fp16, seeded
from gpu_util import sdpa_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Sq", [5, 70, 300])
def test_many_lone_tiles_with_long_key_sequences(d, Sq):
    B, Hq, Hkv, Sk = 8, 32, 8, 2100
    q = seeded(1, B, Hq, Sq, d).astype(np.float16)
    k, v = (seeded(2 + j, B, Hkv, Sk, d).astype(np.float16) for j in range(2))
    lens = [2100, 1100, 1500, 2000, 2047, 2048, 2049, 1]
    got, tc = sdpa_device(q, k, v, kv_lens=lens)
    assert tc
    for bh in (0, 77, 130, 255):
        b, h = divmod(bh, Hq)
        ref = oracle.sdpa_structured(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), kv_lens=lens, heads=[bh])
        assert_close_fp16(got[b, h], ref[b, h])
