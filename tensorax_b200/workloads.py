"""Run one named SDPA workload through the C ABI on synthetic device-resident data and print its time.

    python -m tensorax_b200.workloads fwd --batch 4 --heads 8 --seq 4096 --d 256
    python -m tensorax_b200.workloads bwd --batch 2 --heads 8 --seq 4096 --d 128 --iters 2 --warmup 2
    python -m tensorax_b200.workloads fwd --fp32 --batch 8 --heads 32 --kv-heads 8 --seq-q 1 --seq 4096   (a decoding step)
    python -m tensorax_b200.workloads mha --batch 4 --heads 16 --seq 1024 --d 64 --causal                  (the fp32 layer)

For shapes other than the benchmark's (bench.py measures BASELINE config 2 only) and for profiler
captures of one kernel: `--iters/--warmup` fix the number of launches, nothing else runs on the GPU.
Timing is host wall-clock around `iters` back-to-back launches and one `tx_sdpa_finish`.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import time

import numpy as np

from . import _lib


def _randn_f16(rng, n):
    return _lib.to_device(rng.standard_normal(n, dtype=np.float32).astype(np.float16))


def _layer(a, rng, lib):
    """MultiHeadAttention in float32, from its input to its output, through the package's own layer."""
    from .nn.attention import MultiHeadAttention
    from .tensor import Tensor
    E = a.heads * a.d
    layer = MultiHeadAttention(E, a.heads).cuda()
    x = Tensor(rng.standard_normal((a.batch, a.seq, E), dtype=np.float32), device="cuda")
    visible = 0.5 * a.seq * (a.seq + 1) if a.causal else float(a.seq) * a.seq
    flops = 8.0 * a.batch * a.seq * E * E + 4.0 * a.batch * E * visible
    return _time(a, lib, lambda: layer(x, x, x, causal=a.causal), flops,
                 f"mha fp32 B{a.batch} H{a.heads} S{a.seq} d{a.d}" + (" causal" if a.causal else ""))


def _time(a, lib, launch, flops, name) -> int:
    for _ in range(a.warmup):
        launch()
    _lib.check(lib.tx_sdpa_finish(None))
    t0 = time.perf_counter()
    for _ in range(a.iters):
        launch()
    _lib.check(lib.tx_sdpa_finish(None))
    ms = (time.perf_counter() - t0) / max(a.iters, 1) * 1e3
    print(json.dumps({"workload": name, "ms": ms, "tflops_algorithmic": flops / (ms * 1e-3) / 1e12, "iters": a.iters,
                      "kernels_launched": int(lib.tx_kernel_launch_count())}))
    return 0


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("what", choices=["fwd", "bwd", "mha"])
    ap.add_argument("--batch", type=int, default=4)
    ap.add_argument("--heads", type=int, default=8)
    ap.add_argument("--kv-heads", type=int, default=0, help="K/V heads (default: same as --heads)")
    ap.add_argument("--seq", type=int, default=4096)
    ap.add_argument("--seq-q", type=int, default=0, help="query rows (default: same as --seq; forward only)")
    ap.add_argument("--d", type=int, default=128)
    ap.add_argument("--causal", action="store_true")
    ap.add_argument("--out-f16", action="store_true", help="fp16 result (TX_SDPA_OUT_F16)")
    ap.add_argument("--fp32", action="store_true", help="float32 inputs (forward only)")
    ap.add_argument("--mask", action="store_true", help="dense additive mask, causal (float32 forward only)")
    ap.add_argument("--iters", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--seed", type=int, default=0)
    a = ap.parse_args(argv)
    B, H, S, D = a.batch, a.heads, a.seq, a.d
    Hkv, Sq = a.kv_heads or H, a.seq_q or a.seq
    lib = _lib.load()
    if not lib.tx_cuda_is_available():
        raise RuntimeError("no CUDA device: this package has no CPU compute path")
    rng = np.random.default_rng(a.seed)
    nq, nk = B * H * Sq * D, B * Hkv * S * D
    if (a.mask or Sq != S) and (a.what != "fwd" or a.causal or (a.mask and not a.fp32)):
        raise SystemExit("--mask and --seq-q are for forward passes without --causal, --mask for --fp32")
    if a.what == "mha":
        return _layer(a, rng, lib)
    if a.fp32:
        if a.what != "fwd":
            raise SystemExit("--fp32 is a forward workload")
        q, k, v = (_lib.to_device(rng.standard_normal(n, dtype=np.float32)) for n in (nq, nk, nk))
    else:
        q, k, v = _randn_f16(rng, nq), _randn_f16(rng, nk), _randn_f16(rng, nk)
    flags = _lib.TX_SDPA_OUT_F16 if a.out_f16 else 0
    out = _lib.DeviceBuffer(nq * (2 if a.out_f16 else 4))
    lse = _lib.DeviceBuffer(B * H * Sq * 4)
    mask = None
    if a.mask:
        m = np.where(np.arange(S)[None, :] <= np.arange(Sq)[:, None], 0.0, -np.inf).astype(np.float32)
        mask = _lib.to_device(np.ascontiguousarray(np.broadcast_to(m, (B, H, Sq, S))))
    fwd = _lib.SdpaDesc(q=q.ptr, k=k.ptr, v=v.ptr, mask=mask.ptr if mask else None, kv_lens=None, out=out.ptr, batch=B, q_heads=H,
                        kv_heads=Hkv, seq_q=Sq, seq_k=S, d_k=D, d_v=D,
                        dtype=_lib.TX_DTYPE_F32 if a.fp32 else _lib.TX_DTYPE_F16, causal=int(a.causal),
                        flags=flags, stream=None, lse=lse.ptr if a.what == "bwd" else None)
    visible = 0.5 * S * (S + 1) if a.causal else float(Sq) * S
    if a.what == "fwd":
        def launch():
            _lib.check(lib.tx_sdpa_forward(ctypes.byref(fwd)))
        flops = 4.0 * B * H * visible * D
    else:
        _lib.check(lib.tx_sdpa_forward(ctypes.byref(fwd)))
        _lib.check(lib.tx_sdpa_finish(None))
        g = _lib.to_device(rng.standard_normal(nq, dtype=np.float32))
        dq, dk, dv = _lib.DeviceBuffer(nq * 4), _lib.DeviceBuffer(nk * 4), _lib.DeviceBuffer(nk * 4)
        bwd = _lib.SdpaBwdDesc(q=q.ptr, k=k.ptr, v=v.ptr, out=out.ptr, dout=g.ptr, lse=lse.ptr, kv_lens=None,
                               dq=dq.ptr, dk=dk.ptr, dv=dv.ptr, batch=B, q_heads=H, kv_heads=Hkv, seq_q=S, seq_k=S,
                               d=D, causal=int(a.causal), flags=flags, stream=None)

        def launch():
            _lib.check(lib.tx_sdpa_backward(ctypes.byref(bwd)))
        flops = 10.0 * B * H * visible * D           # the rule's five GEMMs
    name = f"{a.what} {'fp32' if a.fp32 else 'fp16'} B{B} Hq{H} Hkv{Hkv} " + (f"Sq{Sq} " if Sq != S else "") + f"S{S} d{D}"
    return _time(a, lib, launch, flops, name + (" causal" if a.causal else "") + (" dense mask" if a.mask else ""))


if __name__ == "__main__":
    raise SystemExit(main())
