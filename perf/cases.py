"""The attention calls that are timed: what a program that uses this package has it compute.

Listed are calls of ``sageattn`` and ``sageattn_quantized_kv`` over the range of the repository's
own benchmark shapes (``sageattention_rdna3_b200/benchmark_attn.py``: image-generation self- and
cross-attention, VAE attention, a ragged GQA transformer) and of ``bench.py``'s workloads (causal
with an offset in K, causal GQA with outliers, one long sequence): from one call of about ten
microseconds to one of ten milliseconds.  ``draw`` gives further cases of the same families.

Inputs are synthetic, N(0, 1) as in the benchmark, with two variations that occur in trained models:
``offset`` adds a per-channel constant from U(-4, 4) to K (what ``smooth_k`` is for), ``outliers``
scales 1 % of the entries of Q and K by 20.
"""
from __future__ import annotations

import math

import torch

from sageattention_rdna3_b200 import quantize_kv, sageattn, sageattn_quantized_kv

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _case(name, batch, heads, kv_heads, q_len, kv_len, head_dim, dtype, layout, causal=False, smooth_k=False, lse=False,
          values="normal", call="sageattn"):
    case = dict(call=call, batch=batch, heads=heads, kv_heads=kv_heads, q_len=q_len, kv_len=kv_len, head_dim=head_dim,
                dtype=dtype, layout=layout, causal=causal, smooth_k=smooth_k, lse=lse, values=values)
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # The prompt of a GQA text encoder: one short odd sequence, latency of the call itself.
        _case("gqa_117", 1, 48, 12, 117, 117, 128, "bf16", "NHD"),
        # An image attending to a text prompt of 77 tokens (an odd kv length, less than one tile).
        _case("cross_77", 1, 10, 10, 4096, 77, 64, "fp16", "NHD"),
        # The inner blocks of an image UNet: short self-attention, still the un-quantised kernel.
        _case("self_1024", 1, 20, 20, 1024, 1024, 64, "fp16", "NHD"),
        # A diffusion transformer attending to a 512-token prompt, bf16.
        _case("cross_512", 1, 16, 16, 4096, 512, 128, "bf16", "NHD"),
        # The outer blocks of an image UNet at 1024 x 1024 pixels (the reference's headline shape).
        _case("self_4096_d64", 1, 10, 10, 4096, 4096, 64, "fp16", "NHD"),
        # Self-attention of a diffusion transformer at the same resolution.
        _case("self_4096_d128", 1, 16, 16, 4096, 4096, 128, "bf16", "NHD"),
        # Image and text tokens in one sequence: GQA, a length that is no multiple of anything.
        _case("gqa_4213", 1, 48, 12, 4213, 4213, 128, "bf16", "NHD"),
        # The attention block of a VAE, which programs run in fp32: few heads, long sequence.
        _case("vae_16384_fp32", 1, 4, 4, 16384, 16384, 128, "fp32", "NHD"),
        # Prefill of a decoder with an offset in K, smoothed.
        _case("causal_8192", 2, 32, 32, 8192, 8192, 128, "bf16", "HND", causal=True, smooth_k=True, values="offset"),
        # Prefill of a GQA decoder whose Q and K have outliers.
        _case("causal_gqa_4096", 4, 32, 8, 4096, 4096, 128, "bf16", "HND", causal=True, values="outliers"),
        # Video-length self-attention of a diffusion transformer.
        _case("self_32768", 1, 24, 24, 32768, 32768, 128, "fp16", "NHD"),
        # A few new tokens of each of 4 sequences against a long prefix that was quantised once; the
        # log-sum-exp is there to combine the result with the attention among the new tokens.
        _case("cached_prefix_8192", 4, 32, 8, 64, 8192, 128, "bf16", "HND", smooth_k=True, lse=True, values="offset",
              call="sageattn_quantized_kv"),
    ]


# No drawn case does more arithmetic than the largest listed one.
_MOST_FLOPS = 4.0 * 24 * 32768.0 ** 2 * 128


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    while True:
        family = rng.choice(["image", "image", "text", "decoder", "decoder", "vae", "cached"])
        dtype = rng.choice(["fp16", "bf16"])
        layout = rng.choice(["NHD", "HND"])
        dim = rng.choice([64, 128])
        if family == "image":            # self-attention over an image or a video
            heads = rng.choice([8, 10, 16, 20, 24])
            n = _log_int(rng, 256, 32768)
            case = _case(None, rng.choice([1, 1, 2]), heads, heads, n, n, dim, dtype, layout,
                         values=rng.choice(["normal", "outliers"]))
        elif family == "text":           # an image attending to a prompt
            heads = rng.choice([8, 10, 16, 20, 24])
            case = _case(None, rng.choice([1, 1, 2]), heads, heads, _log_int(rng, 256, 16384), _log_int(rng, 16, 1024), dim,
                         dtype, layout)
        elif family == "decoder":        # prefill, with or without GQA
            kv_heads = rng.choice([4, 8, 16, 32])
            n = _log_int(rng, 64, 8192)
            smooth = rng.choice([True, False])
            case = _case(None, rng.choice([1, 2, 4]), kv_heads * rng.choice([1, 1, 4]), kv_heads, n, n, dim, dtype, layout,
                         causal=True, smooth_k=smooth, lse=rng.choice([False, False, True]),
                         values="offset" if smooth else rng.choice(["normal", "outliers"]))
        elif family == "vae":            # fp32 program, few heads
            heads = rng.choice([1, 3, 4])
            n = _log_int(rng, 1024, 24576)
            case = _case(None, 1, heads, heads, n, n, 128, "fp32", layout)
        else:                            # keys and values quantised once: a prompt, or a prefix
            kv_heads = rng.choice([4, 8, 16])
            smooth = rng.choice([True, False])
            case = _case(None, rng.choice([1, 2, 4]), kv_heads * rng.choice([1, 2, 4]), kv_heads, _log_int(rng, 16, 4096),
                         _log_int(rng, 256, 16384), dim, dtype, layout, smooth_k=smooth, lse=rng.choice([False, True]),
                         values="offset" if smooth else "normal", call="sageattn_quantized_kv")
        if work(case)["flops"] <= _MOST_FLOPS:
            return case


def _shape(case, heads, length):
    if case["layout"] == "HND":
        return (case["batch"], heads, length, case["head_dim"])
    return (case["batch"], length, heads, case["head_dim"])


def prepare(case, seed):
    dtype = _DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)

    q = normal(_shape(case, case["heads"], case["q_len"]))
    k = normal(_shape(case, case["kv_heads"], case["kv_len"]))
    v = normal(_shape(case, case["kv_heads"], case["kv_len"]))
    if case["values"] == "offset":
        k += torch.rand(_shape(dict(case, batch=1), case["kv_heads"], 1), generator=gen, device="cuda", dtype=dtype) * 8 - 4
    elif case["values"] == "outliers":
        for t in (q, k):
            t *= 1 + 19 * (torch.rand(t.shape, generator=gen, device="cuda") < 0.01).to(dtype)
    state = dict(case=case, q=q)
    if case["call"] == "sageattn_quantized_kv":
        state["kv"] = quantize_kv(k, v, tensor_layout=case["layout"], smooth_k=case["smooth_k"])
    else:
        state["k"], state["v"] = k, v
    return state


def run(state):
    case = state["case"]
    if case["call"] == "sageattn_quantized_kv":
        return sageattn_quantized_kv(state["q"], state["kv"], is_causal=case["causal"], return_lse=case["lse"])
    return sageattn(state["q"], state["k"], state["v"], tensor_layout=case["layout"], is_causal=case["causal"],
                    smooth_k=case["smooth_k"], return_lse=case["lse"])


def work(case):
    q_len, kv_len, dim = case["q_len"], case["kv_len"], case["head_dim"]
    pairs = float(q_len) * kv_len
    if case["causal"]:                   # row i sees keys 0 .. i
        m = min(q_len, kv_len)
        pairs = m * (m + 1) / 2.0 + (q_len - m) * kv_len
    q_elems = case["batch"] * case["heads"] * q_len * dim
    kv_elems = case["batch"] * case["kv_heads"] * kv_len * dim
    size = 4 if case["dtype"] == "fp32" else 2
    kv_bytes = kv_elems * (1 + 2) if case["call"] == "sageattn_quantized_kv" else 2 * kv_elems * size
    lse_bytes = q_elems // dim * 4 if case["lse"] else 0
    return {"bytes": 2 * q_elems * size + kv_bytes + lse_bytes, "flops": 4.0 * case["batch"] * case["heads"] * pairs * dim}


def tolerance(case):
    # Compared with the same computation on the same int8 values, scales and fp16 values in 64 bits,
    # rounded once to the output type, over the listed and 24 drawn cases: at most rel 9.6e-4 and max
    # 7.8e-3 (one unit in the last place) for bf16 outputs, 3.3e-4 and 1.7e-3 for fp16 (P is rounded to
    # fp16; fp32 calls compute in fp16), 3e-7 for the log-sum-exp.  Four times that.
    if case["dtype"] == "bf16":
        return {"rel": 3.8e-3, "max": 3.2e-2}
    return {"rel": 1.4e-3, "max": 7e-3}


def _quantised(x, group, factor):
    """int8 values (as float64) and one scale per `group` rows of x [..., rows, head_dim], which is first multiplied by `factor`."""
    rows = x.shape[-2]
    x = torch.nn.functional.pad(x.float(), (0, 0, 0, -rows % group)).unflatten(-2, (-1, group))
    largest = (x * factor).abs().amax((-1, -2), keepdim=True).clamp_min(1e-7)
    y = x * (127.0 / largest * factor)
    values = torch.trunc(y + torch.where(y < 0, -0.5, 0.5)).clamp(-128, 127)
    scale = (largest / 127.0).expand(*x.shape[:-1], 1)
    return values.double().flatten(-3, -2)[..., :rows, :], scale.double().flatten(-3, -2)[..., :rows, :]


def _un_quantised(case):
    """The documented choice between the un-quantised and the INT8 kernel, by the length of K."""
    if case["call"] == "sageattn_quantized_kv":
        return False
    q_len, kv_len = case["q_len"], case["kv_len"]
    if case["head_dim"] == 64:
        if case["causal"] or q_len < kv_len:
            return kv_len <= 6144
        return kv_len <= (2048 if case["layout"] == "HND" else 3072)
    return kv_len <= (4096 if q_len * 2 < kv_len else 2048)


def exact(case, seed):
    """The softmax and both products in 64 bits, on the values that the path is defined on: the int8 values and scales of
    Q and K (the inputs in 16 bits for the un-quantised kernel) and V in fp16."""
    made = dict(case, call="sageattn")
    state = prepare(made, seed)
    q, k, v = (state[n].half() if case["dtype"] == "fp32" else state[n] for n in "qkv")
    if case["layout"] == "NHD":
        q, k, v = (t.transpose(1, 2) for t in (q, k, v))
    dim, rep = case["head_dim"], case["heads"] // case["kv_heads"]
    sm_scale, log2e = dim ** -0.5, torch.tensor(math.log2(math.e), dtype=torch.float32)
    factor = (torch.tensor(sm_scale, dtype=torch.float32) * log2e).item()
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    lse = torch.empty(q.shape[:3], dtype=torch.float64, device=q.device)
    for b in range(case["batch"]):
        for h in range(case["heads"]):
            qh, kh, vh = q[b, h], k[b, h // rep], v[b, h // rep].half().double()
            shift = None
            if _un_quantised(case):
                qh, kh = qh.double() * factor, kh.double()
            else:
                if case["smooth_k"]:
                    mean = kh.float().mean(0).to(kh.dtype)
                    shift = qh.double() @ mean.double() * sm_scale
                    kh = kh.float() - mean.float()
                (qi, qs), (ki, ks) = _quantised(qh, 32, factor), _quantised(kh, 16, 1.0)
                qh, kh = qi * qs, ki * ks
            for r in range(0, case["q_len"], 4096):
                s = qh[r:r + 4096] @ kh.T
                if case["causal"]:
                    s.masked_fill_(torch.ones(s.shape, dtype=torch.bool, device=s.device).triu_(r + 1), -math.inf)
                top = s.amax(1, keepdim=True)
                s = s.sub_(top).mul_(math.log(2.0)).exp_()
                total = s.sum(1, keepdim=True)
                out[b, h, r:r + 4096] = s @ vh / total
                lse[b, h, r:r + 4096] = (top[:, 0] * math.log(2.0)) + total[:, 0].log()
            if shift is not None:
                lse[b, h] += shift
    if case["layout"] == "NHD":
        out = out.transpose(1, 2).contiguous()
    return (out, lse) if case["lse"] else out
