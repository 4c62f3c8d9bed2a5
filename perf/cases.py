"""The workloads this package's speed is measured on: what a program that uses it has it do.

Every case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` gives another case of the
same ranges, ``prepare(case, seed)`` makes what the program has in hand before the call, ``run(state)`` is one pass
through the public entry points, ``work(case)`` what a pass cannot do without, ``tolerance(case)`` how far two correct
implementations of the same precision may be apart.

Six kinds of work ("kind"):
  sdpa     ``functional.scaled_dot_product_attention`` (float32) and ``..._mma_fp16`` / ``..._ex`` (float16): prefill
           and cross attention, with or without a causal mask and per-batch key lengths
  masked   float32 attention with the reference's dense additive mask [B, H, Sq, Sk]
  gqa      ``nn.GroupedQueryAttention.forward_bhsd``: prefill with shared K/V heads
  decode   one query token per sequence against a K/V cache: ``tx_sdpa_forward`` on buffers the serving loop keeps,
           enqueued without waiting; the cache's valid part given as key lengths or as the reference's padding mask
           [B, H, 1, Sk], which it takes for a single query row only
  train    forward with saved statistics, then ``Tensor.backward``
  mha      ``nn.MultiHeadAttention``: projections, attention, output projection

Query lengths of the float16 prefill and training passes keep the last 256 rows more than half full.  With a lone last
128-row query tile the float16 kernel that this file was written beside could lose a wait, and a pass that gives up has
no time to compare with; single-row passes are in float32, or at head width 256, for the same reason.
"""
import ctypes
import math

import torch

import tensorax_b200.functional as F
from tensorax_b200 import _C, _lib
from tensorax_b200.nn.attention import GroupedQueryAttention, MultiHeadAttention, ScaledDotProductAttention
from tensorax_b200.tensor import Tensor

_DTYPES = {"float32": torch.float32, "float16": torch.float16}
_SIZES = {"float32": 4, "float16": 2}


def _case(kind, B, Hq, Hkv, Sq, Sk, d, dtype="float16", causal=False, lens="full", name=None, **more):
    c = {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hkv, "Sq": Sq, "Sk": Sk, "d": d, "dtype": dtype, "causal": causal,
         "lens": lens, **more}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # The smallest call: the parity configuration of the float32 path.  Launch and host time only.
        _case("sdpa", 1, 2, 2, 128, 128, 64, "float32", name="fp32_small"),
        # float32 attention at a head width and a length that are no tile multiples.
        _case("sdpa", 2, 8, 8, 1000, 1000, 80, "float32", name="fp32_ragged_d80"),
        # The reference's own mask form: a dense causal mask, as create_causal_mask builds it.
        _case("masked", 4, 8, 8, 512, 512, 64, "float32", name="fp32_dense_mask"),
        # The shortest row of the reference's sweep: many calls of this size make up a small model's step.
        _case("sdpa", 4, 8, 8, 256, 256, 64, name="fp16_short_d64"),
        # The benchmark configuration: long sequences, narrow heads.
        _case("sdpa", 4, 8, 8, 8192, 8192, 64, name="fp16_long_d64"),
        # Wide heads.
        _case("sdpa", 4, 8, 8, 4096, 4096, 256, name="fp16_wide_d256"),
        # A padded batch of prompts of different lengths, causal.
        _case("sdpa", 4, 16, 16, 4096, 4096, 128, causal=True, lens="half", name="fp16_causal_padded_d128"),
        # Prefill with four query heads per K/V head, long context: the largest call.
        _case("gqa", 8, 32, 8, 8192, 8192, 128, causal=True, name="gqa_prefill_d128"),
        # One decoding step of a batch of such sequences: the K/V cache is read once, nothing else is large.
        _case("decode", 8, 32, 8, 1, 4096, 128, "float32", lens="half", mask=False, name="gqa_decode_d128"),
        # A training step's attention: forward and the three gradients.
        _case("train", 4, 16, 16, 2048, 2048, 128, causal=True, name="train_causal_d128"),
        # The same at an odd length with padding, narrow heads and shared K/V heads.
        _case("train", 2, 12, 4, 921, 921, 64, causal=True, lens="half", name="train_ragged_d64"),
        # A float32 attention layer from its input to its output.
        _case("mha", 4, 16, 16, 1024, 1024, 64, "float32", causal=True, name="mha_fp32"),
    ]


# ------------------------------------------------------------------ more cases of the same ranges
def _log_int(rng, lo, hi):
    """Uniform in the logarithm; every value between the bounds, odd ones too."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _two_tiles(n):
    return n if (n - 1) % 256 >= 128 else n + 128


def _largest_flops():
    return max(work(c)["flops"] for c in listed())


def _draw_once(rng):
    kind = rng.choice(["sdpa", "sdpa16", "sdpa16", "masked", "gqa", "decode", "decode", "train", "train", "mha"])
    if kind == "sdpa":
        Sq = _log_int(rng, 16, 4096)
        return _case("sdpa", rng.randint(1, 4), rng.randint(1, 16), 0, Sq, rng.choice([Sq, _log_int(rng, 16, 4096)]),
                     rng.choice([32, 64, 80, 96, 128]), "float32", causal=rng.random() < 0.3)
    if kind == "sdpa16":
        Sq = _two_tiles(_log_int(rng, 128, 8064))
        return _case("sdpa", rng.randint(1, 8), rng.randint(1, 16), 0, Sq, rng.choice([Sq, Sq, _log_int(rng, 64, 8192)]),
                     rng.choice([64, 64, 128, 128, 256, 512]), causal=rng.random() < 0.5,
                     lens=rng.choice(["full", "half"]))
    if kind == "masked":
        Sq = _log_int(rng, 32, 1024)
        return _case("masked", rng.randint(1, 4), rng.randint(1, 16), 0, Sq, Sq, rng.choice([32, 64, 128]), "float32")
    if kind == "gqa":
        S, hkv = _two_tiles(_log_int(rng, 256, 8064)), rng.choice([1, 2, 4, 8])
        return _case("gqa", rng.randint(1, 8), hkv * rng.choice([2, 4, 8]), hkv, S, S, rng.choice([64, 128]), causal=True,
                     lens=rng.choice(["full", "half"]))
    if kind == "decode":
        hkv = rng.choice([1, 2, 4, 8])
        dtype, d = rng.choice([("float32", 64), ("float32", 128), ("float32", 128), ("float16", 256)])
        return _case("decode", _log_int(rng, 1, 32), hkv * rng.choice([1, 2, 4, 8]), hkv, 1, _log_int(rng, 128, 8192), d,
                     dtype, lens=rng.choice(["full", "half"]), mask=dtype == "float32" and rng.random() < 0.3)
    if kind == "train":
        S, hkv = _two_tiles(_log_int(rng, 128, 3968)), rng.choice([2, 4, 8])
        return _case("train", rng.randint(1, 4), hkv * rng.choice([1, 1, 4]), hkv, S, S, rng.choice([64, 128, 256]),
                     causal=rng.random() < 0.7, lens=rng.choice(["full", "half"]))
    dtype = rng.choice(["float32", "float16"])
    S = _log_int(rng, 32, 1920) if dtype == "float32" else _two_tiles(_log_int(rng, 128, 1920))
    return _case("mha", rng.randint(1, 4), rng.choice([4, 8, 16]), 0, S, S, rng.choice([64, 128]), dtype,
                 causal=rng.random() < 0.7)


def draw(rng):
    most = _largest_flops()
    while True:
        c = _draw_once(rng)
        c["Hkv"] = c["Hkv"] or c["Hq"]
        # float32 and dense-mask passes cost more per operation than the float16 ones the bound comes from
        if work(c)["flops"] * (64 if c["dtype"] == "float32" else 1) <= most:
            return c


# ------------------------------------------------------------------ what the program has in hand
def _lengths(case, seed):
    """Valid keys of each sequence: all of them, or uniform in [Sk/2, Sk] as a padded batch has them."""
    if case["lens"] == "full":
        return None
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    lo = max(case["Sk"] // 2, 1)
    return torch.randint(lo, case["Sk"] + 1, (case["B"],), generator=g).tolist()


def _put(t, requires_grad=False):
    """A torch CUDA tensor's values in a tensor of the package."""
    t = t.contiguous()
    dtype = "float16" if t.dtype == torch.float16 else "float32"
    impl = _C.TensorImpl(list(t.shape), dtype, "cuda")
    _lib.check(_lib.load().tx_cuda_memcpy_d2d(impl.data_ptr, t.data_ptr(), t.numel() * t.element_size()))
    return Tensor._wrap(impl, requires_grad)


class _Shared:
    """A tensor of the package as an object torch can look at without a copy; keeps the tensor alive."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.__cuda_array_interface__ = {"shape": tensor.shape, "typestr": "<f2" if tensor.dtype == "float16" else "<f4",
                                         "data": (tensor._c_tensor.data_ptr, False), "version": 2}


def _view(tensor):
    return torch.as_tensor(_Shared(tensor), device="cuda")


def _desc(case, q, k, v, out, mask, lens):
    f16 = case["dtype"] == "float16"
    return _lib.SdpaDesc(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), mask=mask.data_ptr() if mask is not None else None,
                         kv_lens=lens.data_ptr() if lens is not None else None, out=out.data_ptr(), batch=case["B"],
                         q_heads=case["Hq"], kv_heads=case["Hkv"], seq_q=case["Sq"], seq_k=case["Sk"], d_k=case["d"],
                         d_v=case["d"], dtype=_lib.TX_DTYPE_F16 if f16 else _lib.TX_DTYPE_F32, causal=0,
                         flags=_lib.TX_SDPA_OUT_F16 if f16 else 0,
                         stream=ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), lse=None)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, B, Hq, Hkv, Sq, Sk, d = (case[n] for n in ("kind", "B", "Hq", "Hkv", "Sq", "Sk", "d"))
    dtype = _DTYPES[case["dtype"]]

    def normal(*shape, scale=1.0, dtype=dtype):
        return (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * scale).to(dtype)

    s = {"case": case, "lens": _lengths(case, seed)}
    if kind == "mha":
        E = Hq * d
        layer = MultiHeadAttention(E, Hq, device="cuda", attention_dtype=case["dtype"])
        for n in ("q", "k", "v", "out"):
            layer._parameters[n + "_weight"] = _put(normal(E, E, scale=E ** -0.5, dtype=torch.float32))
            layer._parameters[n + "_bias"] = _put(normal(E, scale=0.1, dtype=torch.float32))
        s["layer"], s["x"] = layer, _put(normal(B, Sq, E, dtype=torch.float32))
        return s
    # queries and keys of unit variance; where K/V heads are shared they are scaled by a half
    kv_scale = 0.5 if kind in ("gqa", "decode") else 1.0
    q, k, v = normal(B, Hq, Sq, d), normal(B, Hkv, Sk, d, scale=kv_scale), normal(B, Hkv, Sk, d, scale=kv_scale)
    if kind == "decode":
        lens = None if s["lens"] is None else torch.tensor(s["lens"], dtype=torch.int32, device="cuda")
        mask = None
        if case["mask"]:
            valid = torch.full((B,), Sk, device="cuda") if lens is None else lens
            hidden = torch.arange(Sk, device="cuda") >= valid.view(B, 1, 1, 1)
            mask = torch.zeros(B, Hq, 1, Sk, device="cuda").masked_fill(hidden, -math.inf)
            lens = None
        out = torch.empty((B, Hq, Sq, d), dtype=dtype, device="cuda")
        s.update(q=q, k=k, v=v, mask=mask, lens=lens, out=out, lib=_lib.load(), desc=_desc(case, q, k, v, out, mask, lens))
        return s
    grad = kind == "train"
    s["q"], s["k"], s["v"] = _put(q, grad), _put(k, grad), _put(v, grad)
    if kind == "masked":
        hidden = torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1)
        mask = torch.zeros(Sq, Sk, device="cuda").masked_fill(hidden, -math.inf)
        s["mask"] = _put(mask.expand(B, Hq, Sq, Sk))
        s["layer"] = ScaledDotProductAttention()
    elif kind == "gqa":
        s["layer"] = GroupedQueryAttention(Hq, Hkv)
    elif kind == "train":
        s["grad"] = _put(normal(B, Hq, Sq, d, dtype=torch.float32))
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        _lib.check(s["lib"].tx_sdpa_forward(ctypes.byref(s["desc"])))
        return s["out"]
    if kind == "mha":
        x = s["x"]
        return _view(s["layer"](x, x, x, causal=case["causal"]))
    q, k, v = s["q"], s["k"], s["v"]
    if kind == "masked":
        return _view(s["layer"](q, k, v, s["mask"]))
    if kind == "gqa":
        return _view(s["layer"].forward_bhsd(q, k, v, causal=case["causal"], kv_lens=s["lens"]))
    if kind == "train":
        q.grad = k.grad = v.grad = None
        out = F.scaled_dot_product_attention_ex(q, k, v, causal=case["causal"], kv_lens=s["lens"])
        out.backward(s["grad"])
        return [_view(out), _view(q.grad), _view(k.grad), _view(v.grad)]
    if case["causal"] or s["lens"] is not None:
        return _view(F.scaled_dot_product_attention_ex(q, k, v, causal=case["causal"], kv_lens=s["lens"]))
    if case["dtype"] == "float16":
        return _view(F.scaled_dot_product_attention_mma_fp16(q, k, v))
    return _view(F.scaled_dot_product_attention(q, k, v))


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind, B, Hq, Hkv, Sq, Sk, d = (case[n] for n in ("kind", "B", "Hq", "Hkv", "Sq", "Sk", "d"))
    size = _SIZES[case["dtype"]]
    # lengths uniform in [Sk/2, Sk] average three quarters of the keys
    keys = Sk if case["lens"] == "full" else 0.75 * Sk
    if case["causal"]:
        # row i sees min(i + 1, keys) of them
        n = min(Sq, keys)
        scores = n * (n + 1) / 2 + max(Sq - keys, 0) * keys
    elif kind == "masked":
        scores = Sq * Sk                 # a dense mask says nothing beforehand
    else:
        scores = Sq * keys
    attention = 4.0 * B * Hq * scores * d
    rows_q, rows_k = B * Hq * Sq * d, B * Hkv * keys * d
    if kind == "mha":
        E = Hq * d
        return {"bytes": 4.0 * (2 * B * Sq * E + 4 * E * E + 4 * E), "flops": attention + 8.0 * B * Sq * E * E}
    if kind == "train":
        # out, dQ, dK, dV written and dO read in float32
        return {"bytes": size * (rows_q + 2 * rows_k) + 4.0 * (3 * rows_q + 2 * B * Hkv * Sk * d), "flops": 3.5 * attention}
    out = rows_q * (size if kind == "decode" else 4)
    mask = 4.0 * B * Hq * Sq * Sk if kind == "masked" or case.get("mask") else 0.0
    return {"bytes": size * (rows_q + 2 * rows_k) + out + mask, "flops": attention}


def tolerance(case):
    if case["dtype"] == "float32":
        # sums of 32-bit products; a layer chains four of them
        return {"rel": 2e-5 if case["kind"] == "mha" else 1e-5}
    # 11 significand bits in the operands: probabilities in the forward pass, their gradients too in the backward one
    return {"rel": 4e-3 if case["kind"] == "train" else 2e-3}
