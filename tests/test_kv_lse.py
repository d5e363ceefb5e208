"""The log-sum-exp of a call against smoothed cached keys: q . mean comes with the preparation of Q and is added by
whatever launch writes the log-sum-exp."""
import pytest
import torch

import helpers as H


def _compare(B, Hkv, rep, Sq, Skv, D, dtype, layout, causal, schedule):
    """Bit for bit what the launch without a mean and sage_lse_add_q_mean behind it give."""
    from sageattention_rdna3_b200 import _native, quantize_kv, sageattn_quantized_kv
    ops = _native.load_ops()
    g = torch.Generator(device="cpu").manual_seed(Sq + D)
    q, k, v = (torch.randn(B, h, s, D, generator=g).to(dtype).cuda() for h, s in ((Hkv * rep, Sq), (Hkv, Skv), (Hkv, Skv)))
    k += 3.0
    if layout == "NHD":
        q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
    lay = 1 if layout == "HND" else 0
    kv = quantize_kv(k, v, layout, smooth_k=True)
    try:
        H.set_streamk(schedule)
        o, lse = sageattn_quantized_kv(q, kv, is_causal=causal, return_lse=True)
        from dataclasses import replace
        o2, lse2 = sageattn_quantized_kv(q, replace(kv, k_mean=None), is_causal=causal, return_lse=True)
    finally:
        H.set_streamk(-1)
    ops.lse_add_q_mean(lse2, q, kv.k_mean, lay, D ** -0.5)
    assert torch.equal(o, o2)
    assert torch.equal(lse, lse2)


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", [0, 1])
@pytest.mark.parametrize("layout,causal", [("HND", False), ("NHD", False), ("HND", True)])
@pytest.mark.parametrize("B,Hkv,rep,Sq,Skv,D,dtype", [
    (1, 1, 1, 1, 16, 64, torch.float16),          # one row
    (2, 2, 4, 31, 300, 128, torch.bfloat16),      # folded heads (HND), a group that is not full
    (1, 3, 2, 200, 1500, 64, torch.bfloat16),     # two query tiles, the second ragged
])
def test_equals_the_sum_of_two_launches(B, Hkv, rep, Sq, Skv, D, dtype, layout, causal, schedule):
    _compare(B, Hkv, rep, Sq, Skv, D, dtype, layout, causal, schedule)


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hkv,rep,Sq,Skv,D,dtype,layout", [
    (1, 149, 1, 1280, 129, 64, torch.bfloat16, "NHD"),     # whole items
    (10, 15, 8, 160, 200, 128, torch.bfloat16, "HND"),     # whole items of folded heads
    (1, 10, 1, 4096, 4000, 64, torch.float16, "HND"),      # cut and merged, the last KV tile ragged
    (1, 83, 2, 250, 3500, 128, torch.float16, "NHD"),      # the same, the second query tile ragged too
])
def test_pairs_of_query_tiles(tmp_path, B, Hkv, rep, Sq, Skv, D, dtype, layout):
    """... and where two query tiles share a CTA, which schedules 0 and 1 exclude."""
    from test_pairs import _assert_pairs
    _assert_pairs(tmp_path, B, Hkv * rep, Hkv, Sq, Skv, D, "int8", layout)
    _compare(B, Hkv, rep, Sq, Skv, D, dtype, layout, False, -1)
