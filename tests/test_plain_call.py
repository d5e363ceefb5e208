"""The short way of a plain ``sageattn`` call (``sageattn_plain`` in csrc/torch_ops.cpp) against the long
way through core.py: same choice of kernel, same results, and whatever is not plain falls through."""
import pytest
import torch

from sageattention_rdna3_b200 import _native


def test_what_is_not_plain_falls_through():
    plain = _native.load_module().sageattn_plain
    q = torch.randn(1, 2, 16, 64, dtype=torch.float16)
    assert plain(q, q, q, "HND", False, None, False) is None            # not CUDA tensors
    assert plain(q, q, None, "HND", False, None, False) is None
    assert plain(torch.nn.Parameter(q), q, q, "HND", False, None, False) is None
    assert plain(q, q, q, "HND", False, None) is None                   # another number of arguments
    assert plain(q, q, q, "XYZ", False, None, False) is None
    assert plain(q, q, q, 1, False, None, False) is None
    assert plain(q, q, q, "HND", 0, None, False) is None
    assert plain(q, q, q, "HND", False, 1, False) is None


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("layout", ["HND", "NHD"])
@pytest.mark.parametrize("causal", [False, True])
def test_same_route_and_result_as_the_long_way(D, layout, causal, monkeypatch):
    """Lengths on both sides of every threshold; an empty keyword dict takes the short way, ``kernel=``
    the long one."""
    from sageattention_rdna3_b200 import core, sageattn
    import sageattention_rdna3_b200._C as C
    tiny = torch.randn(1, 1, 8, 64, dtype=torch.float16, device="cuda")
    sageattn(tiny, tiny, tiny)                                           # the first call registers the device
    for q_len, kv_len in ((1, 1), (33, 77), (2048, 2048), (2049, 2049), (3072, 3072), (3073, 3073), (100, 4096), (100, 4097),
                          (2047, 4096), (2048, 4096), (6144, 6144), (100, 6145), (6145, 6145)):
        if causal and q_len != kv_len:
            continue
        shape = (lambda n: (1, 1, n, D)) if layout == "HND" else (lambda n: (1, n, 1, D))
        q, k, v = (torch.randn(shape(n), dtype=torch.float16, device="cuda") for n in (q_len, kv_len, kv_len))
        direct = core.use_direct_kernel(D, layout, causal, q_len, kv_len)
        short = C.sageattn_plain(q, k, v, layout, causal, None, False)
        assert short is not None
        long = sageattn(q, k, v, tensor_layout=layout, is_causal=causal, kernel="direct" if direct else "int8")
        assert torch.equal(short, long), (q_len, kv_len)


@pytest.mark.gpu
def test_refusals_and_switches_stay(monkeypatch):
    from sageattention_rdna3_b200 import sageattn
    import sageattention_rdna3_b200._C as C
    q = torch.randn(1, 4, 40, 64, dtype=torch.float16, device="cuda")
    o = sageattn(q, q, q)
    assert torch.equal(sageattn(q, q, q), o) and torch.equal(C.sageattn_plain(q, q, q, "HND", False, None, False), o)
    with pytest.raises(AssertionError, match="head_dim"):
        sageattn(q[..., :32], q[..., :32], q[..., :32])
    with pytest.raises(AssertionError, match="same dtype"):
        sageattn(q, q.bfloat16(), q)
    with pytest.raises(AssertionError, match="strides"):
        sageattn(torch.randn(1, 4, 40, 68, dtype=torch.float16, device="cuda")[..., :64], q, q)
    with pytest.raises(AssertionError, match="multiple of num_kv_heads"):
        sageattn(q, q[:, :3], q[:, :3])
    odd = torch.randn(1, 4, 40, 68, dtype=torch.float16, device="cuda")[..., :64]
    assert C.sageattn_plain(q, odd, odd, "HND", False, None, False) is None         # copied by the long way
    assert torch.equal(sageattn(q, odd, odd), sageattn(q, odd.contiguous(), odd.contiguous()))
    assert sageattn(q.float(), q.float(), q.float()).dtype == torch.float32
    assert sageattn(q[:, :, :0], q, q).shape == (1, 4, 0, 64)
    assert sageattn(q, q[:, :, :0], q[:, :, :0]).abs().sum() == 0
    for name, value in (("SAGEATTN_KERNEL", "int8"), ("SAGEATTN_B200_CHECK_STATUS", "1"), ("SAGEATTN_DIRECT_THRESHOLD_D64", "8")):
        with monkeypatch.context() as m:
            m.setenv(name, value)
            assert C.sageattn_plain(q, q, q, "HND", False, None, False) is None
            sageattn(q, q, q)
    with pytest.raises(RuntimeError):                                    # no batching rule, as before
        torch.func.vmap(lambda t: sageattn(t, t, t))(q[None].repeat(2, 1, 1, 1, 1))
