"""The un-quantised launch that takes V in bf16 and converts it in shared memory (csrc/attn_kernel.cuh, VBF)."""
import ctypes
import subprocess

import pytest
import torch

import helpers as H


@pytest.mark.parametrize("items,nq,nkv,causal,D,inside", [
    (48, 1, 1, 0, 128, 1), (100000, 64, 1, 0, 128, 0), (100000, 64, 1, 0, 64, 1), (592, 64, 1, 0, 128, 1), (593, 64, 1, 0, 128, 0),
    (1000, 3, 1, 0, 128, 1), (64, 4, 4, 0, 128, 1), (64, 4, 5, 0, 128, 0), (149, 1, 2, 0, 128, 0), (148, 2, 2, 0, 128, 1),
    (112, 7, 7, 1, 128, 1), (128, 8, 8, 1, 128, 0), (148, 8, 8, 0, 64, 1), (149, 8, 8, 0, 64, 0), (20, 3, 20, 1, 64, 1),
])
def test_rule_on_the_host(tmp_path, items, nq, nkv, causal, D, inside):
    from sageattention_rdna3_b200.build import CSRC
    src = tmp_path / "rule.cpp"
    src.write_text(f'#include "{CSRC}/internal.h"\n'
                   'extern "C" int rule(long i, long q, long k, int c, int d) { return sage_few_v_tiles(i, q, k, c, d, 148); }\n')
    lib = tmp_path / "rule.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    rule = ctypes.CDLL(str(lib)).rule
    rule.argtypes = [ctypes.c_long] * 3 + [ctypes.c_int] * 2
    assert rule(items, nq, nkv, causal, D) == inside


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["HND", "NHD"])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D,causal", [
    (1, 2, 1, 1, 1, 64, False),                   # one row, one key
    (2, 4, 2, 130, 127, 128, False),              # two query tiles, a key short of a tile
    (1, 8, 8, 300, 128, 64, False),               # exactly one tile
    (1, 4, 4, 257, 385, 128, False),              # four tiles, the last of one key: rings of two, refilled
    (1, 8, 2, 500, 500, 128, True),
    (1, 3, 3, 900, 1000, 64, False),              # eight tiles, rings of two
    (1, 160, 160, 128, 60, 128, False),           # more items than SMs: rings of one tile
    (1, 160, 160, 100, 100, 128, True),
    (1, 8, 8, 700, 700, 64, True),
    (1, 160, 32, 200, 300, 64, False),            # two items per SM
])
def test_same_bits_as_with_the_conversion_ahead(B, Hq, Hkv, Sq, Skv, D, causal, layout):
    """The conversion is the same rounding wherever it is done, infinities and what overflows fp16 included."""
    from sageattention_rdna3_b200 import _native, sageattn
    ops = _native.load_ops()
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or \
        _native.load_abi().sage_direct_takes_bf16_v(B, Hq, Sq, Skv, D, int(causal))
    q, k, v = (H.randn((B, h, s, D), i, torch.bfloat16).cuda() for i, (h, s) in enumerate(((Hq, Sq), (Hkv, Skv), (Hkv, Skv))))
    v[:, :, :, 5] *= 1e-7                          # fp16 subnormals
    v[0, 0, -1, 3] = 1e6                           # overflows to infinity
    if layout == "NHD":
        q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
    lay = 1 if layout == "HND" else 0
    o, lse = sageattn(q, k, v, tensor_layout=layout, is_causal=causal, return_lse=True)
    o2, lse2 = torch.empty_like(q), torch.empty_like(lse)
    try:
        H.set_streamk(0)                           # the launch ahead and the plain launch behind it
        ops.bf16_attn(q, k, ops.v_to_f16(v, lay), o2, lay, 1, int(causal), D ** -0.5, lse=lse2)
    finally:
        H.set_streamk(-1)
    assert torch.equal(o.nan_to_num(7.0), o2.nan_to_num(7.0))
    assert torch.equal(o.isnan(), o2.isnan())
    assert torch.equal(lse, lse2)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["HND", "NHD"])
@pytest.mark.parametrize("B,heads,S,D", [(1, 8, 128, 64), (2, 48, 117, 128), (1, 20, 512, 128), (1, 18, 1000, 64)])
def test_output_over_the_values(B, heads, S, D, layout):
    """`out` may be V, or lie in the same buffer: what a call with few tiles reads and what it writes are kept apart."""
    from sageattention_rdna3_b200 import sageattn
    shape = (B, heads, S, D) if layout == "HND" else (B, S, heads, D)
    q, k, v = (H.randn(shape, i, torch.bfloat16).cuda() for i in range(3))
    want = sageattn(q, k, v, tensor_layout=layout, kernel="direct")
    for _ in range(5):
        o = v.clone()
        assert torch.equal(sageattn(q, k, o, tensor_layout=layout, kernel="direct", out=o), want)
    flat = torch.empty(q.numel() + 8 * D, dtype=q.dtype, device="cuda")      # V starts 8 rows behind the output
    vs, o = flat[8 * D:].view(shape), flat[:q.numel()].view(shape)
    vs.copy_(v)
    assert torch.equal(sageattn(q, k, vs, tensor_layout=layout, kernel="direct", out=o), want)
