"""Calls of several launches, where a launch starts under its predecessor's end, recorded in a CUDA graph and replayed on
other inputs: bit for bit what the same calls give outside the graph."""
import ctypes

import pytest
import torch

from tensorax_b200 import _lib

pytestmark = pytest.mark.gpu


def p(t):
    return t.data_ptr()


@pytest.mark.parametrize("S", [512, 1000])
def test_fp32_forward_in_a_graph(S):
    lib, stream = _lib.load(), torch.cuda.Stream()
    q, k, v = (torch.empty(2, 8, S, 64, device="cuda").normal_() for _ in range(3))
    out = torch.zeros_like(q)
    d = _lib.SdpaDesc(q=p(q), k=p(k), v=p(v), mask=None, kv_lens=None, out=p(out), batch=2, q_heads=8, kv_heads=8, seq_q=S,
                      seq_k=S, d_k=64, d_v=64, dtype=_lib.TX_DTYPE_F32, causal=1, flags=0,
                      stream=ctypes.c_void_p(stream.cuda_stream), lse=None)
    check_replays(stream, lambda: _lib.check(lib.tx_sdpa_forward(ctypes.byref(d))), (q, k, v), (out,))


@pytest.mark.parametrize("S,dim", [(300, 64), (1025, 128)])
def test_backward_in_a_graph(S, dim):
    lib, stream = _lib.load(), torch.cuda.Stream()
    q, k, v = (torch.empty(2, 4, S, dim, device="cuda", dtype=torch.float16).normal_() for _ in range(3))
    g, out, lse = torch.randn(2, 4, S, dim, device="cuda"), torch.zeros(2, 4, S, dim, device="cuda"), torch.zeros(2, 4, S, device="cuda")
    grads = [torch.zeros(2, 4, S, dim, device="cuda") for _ in range(3)]
    st = ctypes.c_void_p(stream.cuda_stream)
    fwd = _lib.SdpaDesc(q=p(q), k=p(k), v=p(v), mask=None, kv_lens=None, out=p(out), batch=2, q_heads=4, kv_heads=4, seq_q=S,
                        seq_k=S, d_k=dim, d_v=dim, dtype=_lib.TX_DTYPE_F16, causal=1, flags=0, stream=st, lse=p(lse))
    bwd = _lib.SdpaBwdDesc(q=p(q), k=p(k), v=p(v), out=p(out), dout=p(g), lse=p(lse), kv_lens=None, dq=p(grads[0]),
                           dk=p(grads[1]), dv=p(grads[2]), batch=2, q_heads=4, kv_heads=4, seq_q=S, seq_k=S, d=dim, causal=1,
                           flags=0, stream=st)

    def step():
        _lib.check(lib.tx_sdpa_forward(ctypes.byref(fwd)))
        _lib.check(lib.tx_sdpa_backward(ctypes.byref(bwd)))

    check_replays(stream, step, (q, k, v, g), (out, *grads))


def check_replays(stream, call, inputs, outputs):
    torch.cuda.synchronize()
    call()                                                   # kernels loaded and attributes set outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        call()
    for _ in range(3):
        for t in inputs:
            t.normal_()
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        want = [t.clone() for t in outputs]
        for t in outputs:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outputs, want))
