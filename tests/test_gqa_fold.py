"""Folding of the query heads of a GQA group into one row axis (csrc/internal.h) and the log-sum-exp
correction for smooth_k (csrc/merge_kernels.cuh)."""
import ctypes
import subprocess

import pytest
import torch

import helpers as H


def _fold_rule(tmp_path):
    """sage_gqa_fold(Hq, Hkv, Sq, o_stride_h, o_stride_s, is_causal), compiled for the host."""
    from sageattention_rdna3_b200.build import CSRC
    src = tmp_path / "fold.cpp"
    src.write_text(f'#include "{CSRC}/internal.h"\n'
                   'extern "C" int fold(long hq, long hkv, long sq, long sh, long ss, int c) '
                   '{ return sage_gqa_fold(hq, hkv, sq, sh, ss, c); }\n')
    lib = tmp_path / "fold.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    fold = ctypes.CDLL(str(lib)).fold
    fold.argtypes = [ctypes.c_long] * 5 + [ctypes.c_int]
    return fold


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", [0, 1])
@pytest.mark.parametrize("B,Hkv,rep,Sq,Skv,D,dtype", [
    (2, 2, 4, 1, 300, 128, torch.bfloat16),       # 4 rows of four heads in one tile
    (1, 3, 2, 64, 1000, 64, torch.float16),       # two heads fill a tile exactly
    (1, 2, 4, 31, 257, 128, torch.float16),       # heads end inside a 32-row scale group
    (2, 1, 8, 33, 129, 64, torch.bfloat16),       # two scale groups per head, the second of one row
    (1, 2, 3, 85, 640, 128, torch.float16),       # the folded rows are one short of two tiles
    (1, 2, 2, 160, 513, 64, torch.float16),       # more than a tile per head: 3 instead of 4 tiles
])
def test_folded_heads_match_the_unfolded_launch(tmp_path, B, Hkv, rep, Sq, Skv, D, dtype, schedule):
    """HND outputs are folded, NHD outputs (rows of a head not adjacent to the next head's) are not.  The
    same int8 values and scales: what differs is the rounding of P (fp16) where a warp holds other
    rows, and the order of the merge; the outputs are rounded to 16 bits once more."""
    from sageattention_rdna3_b200 import quantize_kv, sageattn_quantized_kv
    g = torch.Generator(device="cpu").manual_seed(Sq * 7 + D)
    q = torch.randn(B, Hkv * rep, Sq, D, generator=g).to(dtype).cuda()
    k = (torch.randn(B, Hkv, Skv, D, generator=g) + 1.0).to(dtype).cuda()
    v = torch.randn(B, Hkv, Skv, D, generator=g).to(dtype).cuda()
    nhd = [t.transpose(1, 2).clone(memory_format=torch.contiguous_format) for t in (q, k, v)]
    fold = _fold_rule(tmp_path)                   # the two launches that are compared are not the same one
    assert fold(Hkv * rep, Hkv, Sq, q.stride(1), q.stride(2), 0) == rep
    assert fold(Hkv * rep, Hkv, Sq, nhd[0].stride(2), nhd[0].stride(1), 0) == 1
    try:
        H.set_streamk(schedule)
        o, lse = sageattn_quantized_kv(q, quantize_kv(k, v, "HND", smooth_k=True), return_lse=True)
        o2, lse2 = sageattn_quantized_kv(nhd[0], quantize_kv(nhd[1], nhd[2], "NHD", smooth_k=True), return_lse=True)
    finally:
        H.set_streamk(-1)
    o2 = o2.transpose(1, 2).float()
    ulp = 2.0 ** (-10 if dtype == torch.float16 else -7)
    assert (o.float() - o2).norm() <= ulp * o2.norm()
    assert (lse - lse2).abs().max() <= 1e-5 * lse2.abs().max()
    ref = torch.nn.functional.scaled_dot_product_attention(
        q.double(), k.double().repeat_interleave(rep, 1), v.double().repeat_interleave(rep, 1))
    assert (o.double() - ref).norm() <= 2e-2 * ref.norm()          # the int8 rounding of Q and K
    ref_lse = torch.logsumexp(q.double() @ k.double().repeat_interleave(rep, 1).transpose(2, 3) * D ** -0.5, -1)
    assert (lse - ref_lse).abs().max() <= 5e-2


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["HND", "NHD"])
@pytest.mark.parametrize("B,Hkv,rep,Sq,D,dtype", [(1, 1, 1, 1, 64, torch.float16), (2, 3, 4, 37, 128, torch.bfloat16),
                                                  (1, 5, 2, 513, 64, torch.bfloat16)])
def test_lse_correction_against_64_bits(B, Hkv, rep, Sq, D, dtype, layout):
    from sageattention_rdna3_b200 import _native
    ops = _native.load_ops()
    g = torch.Generator(device="cpu").manual_seed(D + Sq)
    q = torch.randn(B, Hkv * rep, Sq, D, generator=g).to(dtype).cuda()
    mean = (torch.randn(B, Hkv, D, generator=g) * 3).to(dtype).cuda()
    lse = torch.randn(B, Hkv * rep, Sq, generator=g).cuda()
    want = lse.double() + 0.25 * torch.einsum("bhsd,bhd->bhs", q.double(), mean.double().repeat_interleave(rep, 1))
    ops.lse_add_q_mean(lse, q if layout == "HND" else q.transpose(1, 2).contiguous(), mean, 1 if layout == "HND" else 0, 0.25)
    # D products of magnitude up to 4 * 9 in fp32
    assert (lse - want).abs().max() <= D * 36 * 2.0 ** -24


def test_fold_rule_on_the_host(tmp_path):
    """The rule itself, compiled for the host: folded only where tiles are saved and the output allows it."""
    fold = _fold_rule(tmp_path)
    for sq in list(range(1, 300)) + [4096, 5000]:
        for hkv, rep in ((1, 1), (2, 2), (8, 4), (3, 8)):
            hq = hkv * rep
            fewer = -(-rep * sq // 128) < rep * -(-sq // 128)
            assert fold(hq, hkv, sq, sq * 128, 128, 0) == (rep if fewer else 1)
            assert fold(hq, hkv, sq, sq * 128, 128, 1) == 1                      # causal: rows are positions
            assert fold(hq, hkv, sq, 128, hq * 128, 0) == (rep if fewer and sq * hq == 1 else 1)   # NHD
            assert fold(hq, hkv, sq, sq * 128 + 8, 128, 0) == 1                  # padded heads
    assert fold(4, 0, 8, 8, 1, 0) == 1 and fold(4, 2, 0, 0, 1, 0) == 1 and fold(5, 2, 8, 8, 1, 0) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hkv,rep,Sq,Skv,D,dtype", [
    (2, 2, 4, 1, 300, 128, torch.bfloat16),
    (1, 2, 4, 31, 257, 128, torch.float16),       # the rows of a warp belong to two heads
    (2, 1, 8, 33, 129, 64, torch.bfloat16),
    (1, 2, 2, 160, 513, 64, torch.float16),
])
def test_scattering_launch_folds_like_the_plain_one(B, Hkv, rep, Sq, Skv, D, dtype):
    """Every copy that a scattering launch writes equals the result of the plain launch bit for bit, also where
    that one folds the heads (which rows share a warp decides when a running maximum moves, and with it the
    rounding of P).  Keys that grow along the sequence make the maxima move."""
    from sageattention_rdna3_b200 import check_status, sageattn
    g = torch.Generator(device="cpu").manual_seed(Sq + D)
    q = (torch.randn(B, Hkv * rep, Sq, D, generator=g) * 4).to(dtype).cuda()
    k = (torch.randn(B, Hkv, Skv, D, generator=g) * torch.linspace(0.5, 4.0, Skv)[:, None]).to(dtype).cuda()
    v = torch.randn(B, Hkv, Skv, D, generator=g).to(dtype).cuda()
    try:
        H.set_streamk(0)
        want = sageattn(q, k, v, kernel="int8")
        out = torch.empty_like(q)
        copies = [torch.full_like(q, float("nan")) for _ in range(3)]
        got = sageattn(q, k, v, kernel="int8", out=out, scatter_to=[c.data_ptr() for c in copies])
    finally:
        H.set_streamk(-1)
    check_status()
    assert torch.equal(got, want)
    for c in copies:
        assert torch.equal(c, want)


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D", [
    (8, 32, 8, 64, 8192, 128),       # 256 tiles, which stay on the plain launch; folded 128, which do not
    (4, 32, 8, 64, 8192, 128),       # persistent either way
])
def test_workspace_that_the_query_asks_for_is_used(B, Hq, Hkv, Sq, Skv, D):
    """A caller of the C ABI that allocates what sage_attn_workspace_bytes says gets the launch that the operator
    takes: it writes partial results to the workspace, and the output is the same bit for bit."""
    from sageattention_rdna3_b200 import _native
    lib, ops = _native.load_abi(), _native.load_ops()
    H.set_streamk(-1)
    q, k = H.randn((B, Hq, Sq, D), 0, torch.float16).cuda(), H.randn((B, Hkv, Skv, D), 1, torch.float16).cuda()
    v = H.randn((B, Hkv, Skv, D), 2, torch.float16).cuda()
    q_i8, q_scale, k_i8, k_scale, _ = H.abi_quant(q, k, None, "HND", D ** -0.5)
    want = ops.qk_int8_sv_f16_attn(q_i8, k_i8, v, torch.empty_like(q), q_scale, k_scale, 1, 0, 1.0)
    n = lib.sage_attn_workspace_bytes(B, Hq, Sq, Skv, D, 0)
    assert n > 0
    ws = torch.full((n // 4,), float("nan"), device="cuda")
    o, vs = torch.empty_like(q), H.strided(v, "HND")
    H._check(lib.sage_qk_int8_sv_f16_attn_ws(q_i8.data_ptr(), k_i8.data_ptr(), ctypes.byref(vs), o.data_ptr(), Hq * Sq * D,
                                             Sq * D, D, q_scale.data_ptr(), k_scale.data_ptr(), 0, B, Hq, Hkv, Sq, Skv, D, 0,
                                             None, None, None, ws.data_ptr(), n, H._stream()), "sage_qk_int8_sv_f16_attn_ws")
    torch.cuda.synchronize()
    assert not torch.isnan(ws).all()
    assert torch.equal(o, want)
