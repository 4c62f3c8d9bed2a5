"""Backward items cut over a thread-block cluster: small launches, where a CTA of the cluster may have one tile, a few or
none, and the partial gradients are added through shared memory.  Oracle and bounds as in test_sdpa_backward_gpu.py."""
import numpy as np
import pytest

import oracle
from conftest import seeded
from test_sdpa_backward_gpu import assert_grad_close, backward_device, widen

pytestmark = pytest.mark.gpu

SHAPES = [
    # B, Hq, Hkv, Sq, Sk, d, causal, lens
    (1, 1, 1, 128, 128, 64, False, None),         # one query tile, two key tiles: hardly anything to cut
    (1, 1, 1, 1025, 1025, 64, True, None),        # a lone last row; late key tiles have fewer tiles than CTAs
    (2, 6, 2, 300, 700, 64, False, [700, 65]),    # grouped heads; keys behind the length: items without a tile
    (2, 3, 1, 333, 97, 128, True, [97, 0]),       # no valid key in one batch element: NaN in every gradient
    (1, 4, 4, 1024, 1024, 128, True, None),
    (1, 2, 1, 127, 513, 128, False, [129]),
    (1, 1, 1, 600, 600, 256, True, None),         # two CTAs a key tile, each cut again
    (1, 2, 2, 65, 1000, 256, False, [640]),
]


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,d,causal,lens", SHAPES)
def test_cut_items(B, Hq, Hkv, Sq, Sk, d, causal, lens):
    q = seeded(90, B, Hq, Sq, d).astype(np.float16)
    k, v = (seeded(s, B, Hkv, Sk, d).astype(np.float16) for s in (91, 92))
    g = seeded(93, B, Hq, Sq, d)
    _, _, runs = backward_device(q, k, v, g, causal=causal, kv_lens=lens, repeats=2)
    n = B if lens is None else sum(x > 0 for x in lens)                  # batch elements with a valid key come first
    refs = oracle.sdpa_backward(widen(q[:n]), widen(k[:n]), widen(v[:n]), g[:n], causal=causal, kv_lens=lens and lens[:n])
    for got, again, ref, name in zip(runs[0], runs[1], refs, ("dq", "dk", "dv")):
        assert np.array_equal(got, again, equal_nan=True)                # the order of the sums is fixed
        assert_grad_close(got[:n], ref, name)
        assert np.isnan(got[n:]).all()
