"""Schedule of causal launches (csrc/internal.h): the last group of heads of a plain launch has its own size, and which
launches are persistent."""
import ctypes
import subprocess

import pytest
import torch

import helpers as H


def _rules(tmp_path):
    from sageattention_rdna3_b200.build import CSRC
    src = tmp_path / "rules.cpp"
    src.write_text(f'#include "{CSRC}/internal.h"\n'
                   'extern "C" int tail(int n, int g, int nq, double b, int sms) { return sage_tail_group_first(n, g, nq, b, sms); }\n'
                   'extern "C" int streamk(long n, long t, double m, int d) { return sage_causal_streamk(n, t, m, d); }\n')
    lib = tmp_path / "rules.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    rules = ctypes.CDLL(str(lib))
    rules.tail.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double, ctypes.c_int]
    rules.streamk.argtypes = [ctypes.c_long, ctypes.c_long, ctypes.c_double, ctypes.c_int]
    return rules


def test_every_item_has_one_block(tmp_path):
    """The kernel's map from block to (head, query tile), for whole GQA groups, odd numbers of heads, one tile, and
    heads too large to share the L2."""
    tail = _rules(tmp_path).tail
    for n_heads in (1, 3, 7, 8, 9, 20, 24, 63, 128):
        for group in (8, 9, 12):
            for nq in (1, 2, 18, 64):
                for kv_bytes in (0.0, 1e5, 3e6, 5e7):
                    first = tail(n_heads, group, nq, kv_bytes, 148)
                    assert 0 <= first <= n_heads and first % group == 0
                    items = set()
                    for block in range(n_heads * nq):
                        if block < first * nq:
                            g_first = block // (nq * group) * group
                            size, within = group, block - g_first * nq
                        else:
                            g_first, size, within = first, n_heads - first, block - first * nq
                        items.add((g_first + within % size, nq - 1 - within // size))
                    assert items == {(h, t) for h in range(n_heads) for t in range(nq)}


@pytest.mark.parametrize("heads,tiles,D,persistent", [
    (1, 7, 64, 0), (1, 8, 64, 1), (4, 7, 64, 0), (4, 8, 64, 1), (5, 40, 64, 1), (5, 64, 64, 0), (4, 96, 64, 0), (6, 13, 64, 0),
    (6, 32, 64, 1), (6, 40, 64, 0), (8, 20, 64, 0),
    (1, 7, 128, 0), (1, 8, 128, 1), (2, 7, 128, 0), (2, 8, 128, 1), (3, 32, 128, 1), (4, 19, 128, 0), (4, 20, 128, 1), (4, 40, 128, 1),
    (5, 40, 128, 0),
    (10, 24, 128, 0), (64, 64, 128, 0),
])
def test_few_long_causal_heads_are_cut_into_spans(tmp_path, heads, tiles, D, persistent):
    steps = heads * tiles * (tiles + 1) // 2
    assert _rules(tmp_path).streamk(heads, tiles, steps / min(steps, 296), D) == persistent


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hq,Hkv,S,D,dtype", [
    (1, 9, 9, 257, 128, torch.bfloat16),         # one group and a left-over head in the last group
    (2, 12, 3, 300, 64, torch.float16),          # GQA groups of 4 in groups of 8, un-quantised kernel
    (1, 40, 40, 2176, 128, torch.float16),       # two groups before the last one
])
def test_many_heads_are_their_heads(B, Hq, Hkv, S, D, dtype):
    """A head's result does not depend on where its items stand: bit for bit that of a launch of the head alone."""
    from sageattention_rdna3_b200 import sageattn
    q, k, v = (H.randn((B, h, S, D), i, dtype).cuda() for i, h in enumerate((Hq, Hkv, Hkv)))
    try:
        H.set_streamk(0)
        o = sageattn(q, k, v, is_causal=True)
        for b in range(B):
            for h in range(0, Hq, 5):
                one = [t[b:b + 1, i:i + 1].contiguous() for t, i in ((q, h), (k, h * Hkv // Hq), (v, h * Hkv // Hq))]
                assert torch.equal(o[b:b + 1, h:h + 1], sageattn(*one, is_causal=True)), (b, h)
    finally:
        H.set_streamk(-1)
