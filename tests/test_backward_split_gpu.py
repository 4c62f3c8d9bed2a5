"""Backward items cut over a thread-block cluster: small launches, where a CTA of the cluster may have one tile, a few or
none, and the partial gradients are added through shared memory.  Oracle and bounds as in test_sdpa_backward_gpu.py."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import seeded
from tensorax_b200 import _lib
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


@pytest.mark.parametrize("S,d", [(300, 64), (700, 128)])
def test_calls_back_to_back_read_their_own_preprocess(S, d):
    """Backward calls enqueued one behind the other without a wait, each with another upstream gradient and the same
    workspace from the pool: bit for bit what each gives alone."""
    lib, shape = _lib.load(), (2, 4, S, d)
    q, k, v = (torch.empty(shape, device="cuda", dtype=torch.float16).normal_() for _ in range(3))
    out, lse = torch.zeros(shape, device="cuda"), torch.zeros(shape[:3], device="cuda")
    fwd = _lib.SdpaDesc(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), mask=None, kv_lens=None, out=out.data_ptr(), batch=2,
                        q_heads=4, kv_heads=4, seq_q=S, seq_k=S, d_k=d, d_v=d, dtype=_lib.TX_DTYPE_F16, causal=1, flags=0,
                        stream=None, lse=lse.data_ptr())
    _lib.check(lib.tx_sdpa_forward(ctypes.byref(fwd)))
    gs = [torch.randn(shape, device="cuda") * 4.0 ** i for i in range(6)]

    def grads(wait):
        res = [[torch.zeros(shape, device="cuda") for _ in range(3)] for _ in gs]
        torch.cuda.synchronize()
        for g, r in zip(gs, res):
            _lib.check(lib.tx_sdpa_backward(ctypes.byref(_lib.SdpaBwdDesc(
                q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), dout=g.data_ptr(), lse=lse.data_ptr(),
                kv_lens=None, dq=r[0].data_ptr(), dk=r[1].data_ptr(), dv=r[2].data_ptr(), batch=2, q_heads=4, kv_heads=4,
                seq_q=S, seq_k=S, d=d, causal=1, flags=0, stream=None))))
            if wait:
                _lib.check(lib.tx_sdpa_finish(None))
        _lib.check(lib.tx_sdpa_finish(None))
        return res

    alone = grads(True)
    for _ in range(10):
        for a, b in zip(grads(False), alone):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
