"""The launch with two query tiles per CTA (csrc/pair_kernel.cuh) and the rule that chooses it (csrc/internal.h)."""
import ctypes
import subprocess

import pytest
import torch

import helpers as H


def _rule(tmp_path, name="sage_takes_pairs"):
    from sageattention_rdna3_b200.build import CSRC
    src = tmp_path / "rule.cpp"
    src.write_text(f'#include "{CSRC}/internal.h"\n'
                   f'extern "C" int rule(long i, long q, long k, int d, int f, int s) {{ return {name}(i, q, k, d, f, s); }}\n')
    lib = tmp_path / f"{name}.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    rule = ctypes.CDLL(str(lib)).rule
    rule.argtypes = [ctypes.c_long] * 3 + [ctypes.c_int] * 3
    return rule


@pytest.mark.parametrize("items,nq,nkv,D,qkf,taken", [
    (740, 10, 12, 128, 0, 1), (740, 10, 13, 128, 0, 0), (739, 10, 5, 128, 0, 0), (444, 10, 4, 128, 0, 1), (443, 10, 4, 128, 0, 0),
    (592, 10, 8, 64, 0, 1), (592, 10, 9, 64, 0, 0), (740, 7, 2, 64, 0, 0), (825, 9, 6, 64, 0, 1), (825, 9, 7, 64, 0, 0), (740, 9, 4, 64, 0, 1), (740, 9, 5, 64, 0, 0),
    (300, 29, 29, 64, 0, 0), (310, 31, 29, 64, 0, 0), (740, 1, 1, 64, 1, 0),
    (740, 10, 8, 64, 1, 1), (740, 10, 9, 64, 1, 0), (740, 10, 12, 128, 1, 1), (739, 10, 1, 128, 1, 0), (444, 10, 1, 64, 1, 1),
    (160, 32, 32, 64, 0, 1), (148, 32, 32, 64, 0, 0), (178, 32, 32, 64, 0, 0), (160, 32, 15, 64, 0, 0), (160, 32, 40, 128, 0, 1),
    (160, 32, 41, 128, 0, 0), (148, 32, 16, 128, 1, 1), (147, 32, 16, 128, 1, 0), (160, 32, 16, 64, 1, 0),
    # cut launches: half pairs, a round hardly begun, long items, spans that reach over the end of an item
    (320, 31, 29, 64, 0, 1), (320, 31, 32, 64, 0, 0), (180, 71, 71, 64, 0, 1), (180, 71, 72, 64, 0, 0), (170, 19, 19, 64, 0, 1), (170, 19, 20, 64, 0, 0), (152, 16, 21, 64, 0, 0),
    (157, 2, 21, 64, 0, 1), (160, 32, 96, 64, 0, 1), (160, 32, 97, 64, 0, 0), (165, 129, 96, 64, 0, 0), (320, 128, 128, 64, 0, 0),
    (160, 32, 36, 128, 0, 1), (160, 32, 37, 128, 0, 0), (167, 2, 28, 128, 0, 1), (167, 2, 32, 128, 0, 0), (168, 55, 20, 128, 0, 1),
    (170, 19, 40, 128, 0, 0), (162, 18, 20, 128, 1, 1), (365, 9, 60, 128, 1, 1),
])
def test_rule_on_the_host(tmp_path, items, nq, nkv, D, qkf, taken):
    assert _rule(tmp_path)(items, nq, nkv, D, qkf, 148) == taken


@pytest.mark.parametrize("items,nq,nkv,D,qkf,filled", [
    (444, 10, 4, 128, 0, 1), (455, 10, 4, 128, 0, 0), (534, 10, 4, 128, 0, 0), (535, 10, 4, 128, 0, 1), (455, 10, 1, 128, 0, 1),
    (600, 15, 2, 128, 0, 0), (508, 4, 4, 64, 0, 0), (552, 6, 4, 64, 0, 1), (740, 10, 12, 128, 0, 1), (600, 10, 3, 64, 1, 1),
    (160, 32, 32, 64, 0, 1), (620, 9, 1, 128, 0, 0), (738, 123, 1, 128, 0, 1),
])
def test_rounds_that_are_badly_filled(tmp_path, items, nq, nkv, D, qkf, filled):
    assert _rule(tmp_path, "sage_pairs_fill")(items, nq, nkv, D, qkf, 148) == filled


def _assert_pairs(tmp_path, B, Hq, Hkv, Sq, Skv, D, kernel, layout):
    """The call is one that the rule takes (int8: with the heads of a GQA group folded where that is done)."""
    sms, rep = torch.cuda.get_device_properties(0).multi_processor_count, Hq // Hkv
    if kernel == "int8" and layout == "HND" and -(-rep * Sq // 128) < rep * -(-Sq // 128):
        Hq, Sq = Hkv, rep * Sq
    nq, nkv = -(-Sq // 128), -(-Skv // 128)
    case = B * Hq * -(-nq // 2), nq, nkv, D, int(kernel == "direct"), sms
    assert sms != 148 or (_rule(tmp_path)(*case) and _rule(tmp_path, "sage_pairs_fill")(*case))


def _calls(q, k, v, layout, kernel):
    from sageattention_rdna3_b200 import sageattn
    try:
        H.set_streamk(-1)
        pairs = sageattn(q, k, v, tensor_layout=layout, return_lse=True, kernel=kernel)
        H.set_streamk(0)
        plain = sageattn(q, k, v, tensor_layout=layout, return_lse=True, kernel=kernel)
    finally:
        H.set_streamk(-1)
    return pairs, plain


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["int8", "direct"])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D,dtype,layout", [
    (2, 93, 31, 1024, 1, 64, torch.float16, "HND"),        # 744 items of one key
    (1, 149, 149, 1280, 129, 64, torch.bfloat16, "NHD"),   # 745 items, the second KV tile of one key
    (1, 165, 33, 1150, 200, 128, torch.bfloat16, "HND"),   # nine query tiles: half a pair empty, the last rows ragged
    (5, 30, 30, 1281, 256, 128, torch.float16, "NHD"),     # a last query tile of one row
    (10, 120, 15, 160, 200, 128, torch.bfloat16, "HND"),   # int8: GQA heads folded into ten tiles of 1280 rows
])
def test_whole_items_equal_the_plain_launch(tmp_path, B, Hq, Hkv, Sq, Skv, D, dtype, layout, kernel):
    """A row's softmax does not depend on what else its CTA works on: bit for bit the result of one tile per CTA."""
    _assert_pairs(tmp_path, B, Hq, Hkv, Sq, Skv, D, kernel, layout)
    q, k, v = (H.randn((B, h, s, D), i, dtype).cuda() for i, (h, s) in enumerate(((Hq, Sq), (Hkv, Skv), (Hkv, Skv))))
    q[:, :, 5] *= 30                                       # rows whose maximum moves
    if layout == "NHD":
        q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
    (o, lse), (o2, lse2) = _calls(q, k, v, layout, kernel)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D,dtype,kernel", [
    (1, 10, 10, 4096, 4096, 64, torch.float16, "int8"),    # 160 items of 32 tiles on 148 SMs
    (1, 51, 17, 1500, 2001, 64, torch.bfloat16, "int8"),   # two rounds and 10 over, ragged
    (3, 53, 53, 250, 2433, 128, torch.bfloat16, "int8"),   # one pair per head, a last KV tile of one key
    (1, 20, 20, 2048, 2048, 128, torch.float16, "direct"),
    (1, 73, 73, 1100, 2048, 128, torch.bfloat16, "direct"),    # half pairs, 69 items over: 32 rows per CTA of the merge
])
def test_cut_items_match_the_plain_launch(tmp_path, B, Hq, Hkv, Sq, Skv, D, dtype, kernel):
    """Parts of an item are merged in fp32.  What may differ from the plain launch, element by element: one rounding of
    the output in either, and P rounded to fp16 against another maximum in either (2^-11 of its value, or 2^-25 of
    its largest value for what is below fp16's normal numbers)."""
    from sageattention_rdna3_b200 import sageattn
    _assert_pairs(tmp_path, B, Hq, Hkv, Sq, Skv, D, kernel, "HND")
    q, k, v = (H.randn((B, h, s, D), i, dtype) for i, (h, s) in enumerate(((Hq, Sq), (Hkv, Skv), (Hkv, Skv))))
    q[:, :, 3::31] *= 12                                   # rows whose maximum moves
    k[:, :, Skv // 2 :: 97] *= 3                           # ... by more in the later parts
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    junk = torch.full((160 << 20,), float("nan"), device="cuda")     # what the allocator hands out as workspace
    del junk
    (o, lse), (o2, lse2) = _calls(q, k, v, "HND", kernel)
    assert not torch.equal(o, o2)                          # another launch
    weighted = _calls(q, k, v.abs(), "HND", kernel)[1][0].float()    # sum of p |v| / l
    ulp = 2.0 ** (-10 if dtype == torch.float16 else -7)
    bound = ulp * o2.float().abs() + 2.0 ** -10 * (1 + ulp) * weighted + 2.0 ** -24 * Skv * v.abs().max().float()
    worst = ((o.float() - o2.float()).abs() / bound).max()
    assert worst <= 1, worst
    assert ((lse - lse2).abs() <= 1e-5 * lse2.abs().clamp_min(1.0)).all()


@pytest.mark.gpu
def test_wait_that_cannot_complete_gives_a_status():
    from sageattention_rdna3_b200 import _native, check_status, sageattn
    lib = _native.load_abi()
    q, k, v = (H.randn((1, 149, s, 64), i, torch.float16).cuda() for i, s in enumerate((1280, 128, 128)))
    good = sageattn(q, k, v, kernel="int8")
    check_status()
    try:
        lib.sage_test_set_wait_limit_us(20000)
        lib.sage_test_drop_v_load(1)
        sageattn(q, k, v, kernel="int8")
        with pytest.raises(RuntimeError, match="device status"):
            check_status()
    finally:
        lib.sage_test_drop_v_load(0)
        lib.sage_test_set_wait_limit_us(0)
    assert torch.equal(sageattn(q, k, v, kernel="int8"), good)
    check_status()


@pytest.mark.gpu
def test_workspace_that_is_not_needed_may_be_anywhere():
    """Whole items use no workspace, and the plain launch that would take them otherwise does not look at it either."""
    from sageattention_rdna3_b200 import _native
    lib = _native.load_abi()
    n_heads, Sq, Skv, D = 259, 512, 256, 64
    q, k, v = (H.randn((1, n_heads, s, D), i, torch.float16).cuda() for i, s in enumerate((Sq, Skv, Skv)))
    q_i8, q_scale, k_i8, k_scale, _ = H.abi_quant(q, k, None, "HND", D ** -0.5)
    ws = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
    outs = []
    for schedule, offset in ((0, 0), (-1, 0), (-1, 4)):
        o, vs, status = torch.empty_like(q), H.strided(v, "HND"), torch.zeros(1, dtype=torch.int32, device="cuda")
        H.set_streamk(schedule)
        try:
            rc = lib.sage_qk_int8_sv_f16_attn_ws(q_i8.data_ptr(), k_i8.data_ptr(), ctypes.byref(vs), o.data_ptr(), n_heads * Sq * D,
                                                 Sq * D, D, q_scale.data_ptr(), k_scale.data_ptr(), 0, 1, n_heads, n_heads, Sq, Skv,
                                                 D, 0, None, None, status.data_ptr(), ws.data_ptr() + offset, ws.numel() - 16,
                                                 H._stream())
        finally:
            H.set_streamk(-1)
        assert rc == 0, lib.sage_last_error()
        assert int(status.item()) == 0
        outs.append(o)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert not ws.any()


CASES_IN_USE = [
    (149, 1280, 129, 64, torch.bfloat16, "int8"),          # whole items
    (10, 4096, 4096, 64, torch.float16, "int8"),           # cut
    (20, 2048, 2048, 128, torch.float16, "direct"),        # cut
]


@pytest.mark.gpu
@pytest.mark.parametrize("heads,Sq,Skv,D,dtype,kernel", CASES_IN_USE)
def test_slices_of_larger_tensors(tmp_path, heads, Sq, Skv, D, dtype, kernel):
    """Q, K, V and the output as slices: the same bits as for contiguous tensors, and nothing written beside the output."""
    from sageattention_rdna3_b200 import sageattn
    _assert_pairs(tmp_path, 1, heads, heads, Sq, Skv, D, kernel, "NHD")
    qs = H.randn((1, Sq, heads, 2 * D), 0, dtype).cuda()
    kvs = H.randn((1, Skv, 2, heads, D + 8), 1, dtype).cuda()
    q, k, v = qs[..., D:], kvs[:, :, 0, :, 8:], kvs[:, :, 1, :, :D]
    buf = torch.full((1, Sq + 3, heads, D + 16), 7.0, dtype=dtype, device="cuda")
    out = buf[:, 2:-1, :, 8:-8]
    sageattn(q, k, v, tensor_layout="NHD", kernel=kernel, out=out)
    want = sageattn(q.contiguous(), k.contiguous(), v.contiguous(), tensor_layout="NHD", kernel=kernel)
    assert torch.equal(out, want)
    out.fill_(7.0)
    assert (buf == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,Sq,Skv,D,dtype,kernel", CASES_IN_USE)
def test_captured_and_on_two_streams(tmp_path, heads, Sq, Skv, D, dtype, kernel):
    """A captured call replayed on new inputs, and calls in flight on two streams, each with its workspace."""
    from sageattention_rdna3_b200 import check_status, sageattn
    _assert_pairs(tmp_path, 1, heads, heads, Sq, Skv, D, kernel, "HND")
    sets = [[H.randn((1, heads, s, D), 3 * n + i, dtype).cuda() for i, s in enumerate((Sq, Skv, Skv))] for n in range(2)]
    want = [sageattn(*t, kernel=kernel) for t in sets]
    mine = [t.clone() for t in sets[0]]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        sageattn(*mine, kernel=kernel)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = sageattn(*mine, kernel=kernel)
    for n in (0, 1):
        for a, b in zip(mine, sets[n]):
            a.copy_(b)
        graph.replay()
        assert torch.equal(out, want[n])
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(4):
        for n, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[n].append(sageattn(*sets[n], kernel=kernel))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[n]) for n in (0, 1) for o in got[n])
    check_status()
