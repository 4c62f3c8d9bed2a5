"""Key lengths given as a host array (TX_SDPA_KV_LENS_HOST) are read during the call, however many there are, from whatever
memory they are in, and also while the call is recorded in a CUDA graph."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
import tensorax_b200 as ts
import tensorax_b200.functional as F
from conftest import assert_close_fp32, seeded
from tensorax_b200 import _lib

pytestmark = pytest.mark.gpu


def descriptor(q, k, v, out, lens, stream=None):
    B, H, Sq, d = q.shape
    return _lib.SdpaDesc(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), mask=None, kv_lens=lens, out=out.data_ptr(), batch=B,
                         q_heads=H, kv_heads=H, seq_q=Sq, seq_k=k.shape[2], d_k=d, d_v=d, dtype=_lib.TX_DTYPE_F32, causal=0,
                         flags=_lib.TX_SDPA_KV_LENS_HOST, stream=stream, lse=None)


def tensors(B, Sq=40, Sk=70):
    g = torch.Generator(device="cuda").manual_seed(B)
    q, k, v = (torch.randn(B, 2, s, 64, device="cuda", generator=g) for s in (Sq, Sk, Sk))
    return q, k, v, torch.zeros_like(q)


def want(q, k, v, lens):
    return oracle.sdpa_structured(*(t.cpu().numpy() for t in (q, k, v)), kv_lens=list(lens))


@pytest.mark.parametrize("B", [32, 33, 40, 1000, 2049])
def test_pinned_array_overwritten_right_after_the_call(B):
    lib = _lib.load()
    q, k, v, out = tensors(B, 3, 70)
    lens = (np.arange(B) * 7 % 70 + 1).astype(np.int32)
    busy = torch.randn(8192, 8192, device="cuda")
    torch.cuda.synchronize()
    ptr = lib.tx_host_alloc_pinned(B * 4)
    try:
        host = (ctypes.c_int32 * B).from_address(ptr)
        host[:] = lens.tolist()
        for _ in range(3):                                    # some milliseconds in the (default) stream ahead of the call
            busy @ busy
        _lib.check(lib.tx_sdpa_forward(ctypes.byref(descriptor(q, k, v, out, ptr))))
        host[:] = [1] * B
        _lib.check(lib.tx_sdpa_finish(None))
    finally:
        _lib.check(lib.tx_host_free_pinned(ptr))
    rows = [0, 31, B // 2, B - 1]
    assert_close_fp32(out.cpu().numpy()[rows], want(q[rows], k[rows], v[rows], lens[rows]))


@pytest.mark.parametrize("B", [8, 40])
def test_captured_call_keeps_the_lengths_it_was_recorded_with(B):
    lib, stream = _lib.load(), torch.cuda.Stream()
    q, k, v, out = tensors(B)
    lens = (np.arange(B) * 5 % 70 + 1).astype(np.int32)
    host = (ctypes.c_int32 * B)(*lens.tolist())
    d = descriptor(q, k, v, out, ctypes.addressof(host), ctypes.c_void_p(stream.cuda_stream))
    torch.cuda.synchronize()
    _lib.check(lib.tx_sdpa_forward(ctypes.byref(d)))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        _lib.check(lib.tx_sdpa_forward(ctypes.byref(d)))
    host[:] = [1] * B
    out.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert_close_fp32(out.cpu().numpy(), want(q, k, v, lens))


@pytest.mark.parametrize("B", [32, 33, 70])
def test_python_layer_forward_and_backward(B):
    S, d = 150, 64
    lens = [1 + 11 * i % S for i in range(B)]
    q, k, v = (seeded(60 + i, B, 1, S, d).astype(np.float16) for i in range(3))
    g = seeded(63, B, 1, S, d)
    leaves = [ts.Tensor(x, dtype="float16", device="cuda", requires_grad=True) for x in (q, k, v)]
    out = F.scaled_dot_product_attention_ex(*leaves, kv_lens=lens)
    wide = [x.astype(np.float32) for x in (q, k, v)]
    assert np.abs(out.numpy() - oracle.sdpa_structured(*wide, kv_lens=lens)).max() <= 2e-3
    out.backward(ts.Tensor(g, device="cuda"))
    for leaf, ref in zip(leaves, oracle.sdpa_backward(*wide, g, kv_lens=lens)):
        assert np.linalg.norm(leaf.grad.numpy() - ref) <= 5e-3 * np.linalg.norm(ref)
