"""Kernels that start before the one ahead of them in the stream has ended: every read and write still comes
after it."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("D,S,smooth,dtype", [(64, 256, False, torch.float16), (128, 2300, True, torch.bfloat16),
                                              (64, 4096, False, torch.bfloat16)])
def test_back_to_back_calls_on_buffers_that_change(D, S, smooth, dtype):
    """One launch, several, and several with the persistent form: the inputs are overwritten between calls
    without a synchronisation, and the scratch of one call is the allocator's next answer to the other."""
    from sageattention_rdna3_b200 import sageattn
    torch.manual_seed(0)
    inputs = [[torch.randn(1, 3, S, D, device="cuda").to(dtype) for _ in range(3)] for _ in range(4)]
    want = []
    for q, k, v in inputs:
        want.append(sageattn(q, k, v, smooth_k=smooth))
        torch.cuda.synchronize()
    q, k, v = (torch.empty_like(t) for t in inputs[0])
    got = []
    for i in range(40):
        for dst, src in zip((q, k, v), inputs[i % 4]):
            dst.copy_(src)
        got.append(sageattn(q, k, v, smooth_k=smooth))
    torch.cuda.synchronize()
    inner = sageattn(q, k, v, smooth_k=smooth)
    torch.cuda.synchronize()                     # the value of the chain, with nothing overlapped
    chain = sageattn(inner, k, v, smooth_k=smooth)
    torch.cuda.synchronize()
    chained = [sageattn(sageattn(q, k, v, smooth_k=smooth), k, v, smooth_k=smooth) for _ in range(8)]
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 4]) for i, o in enumerate(got))
    assert all(torch.equal(o, chain) for o in chained)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["HND", "NHD"])
@pytest.mark.parametrize("schedule", [0, 1])
def test_cached_keys_back_to_back(layout, schedule):
    """Four dependent kernels per call (Q, attention, merge, log-sum-exp), folded (HND) and not; the queries are
    overwritten between calls, and the output of one call is the query of the next."""
    import helpers
    from sageattention_rdna3_b200 import quantize_kv, sageattn_quantized_kv
    torch.manual_seed(1)
    shape = lambda h, s: (2, h, s, 128) if layout == "HND" else (2, s, h, 128)
    queries = [torch.randn(shape(8, 48), device="cuda").bfloat16() for _ in range(4)]
    kv = quantize_kv(torch.randn(shape(2, 900), device="cuda").bfloat16() + 1, torch.randn(shape(2, 900), device="cuda").bfloat16(),
                     layout, smooth_k=True)
    try:
        helpers.set_streamk(schedule)
        want = []
        for x in queries + [None]:
            want.append(sageattn_quantized_kv(want[-1][0] if x is None else x, kv, return_lse=True))
            torch.cuda.synchronize()
        q, got = torch.empty_like(queries[0]), []
        for i in range(32):
            q.copy_(queries[i % 4])
            got.append(sageattn_quantized_kv(q, kv, return_lse=True))
            if i % 4 == 3:
                got.append(sageattn_quantized_kv(got[-1][0], kv, return_lse=True))
        torch.cuda.synchronize()
    finally:
        helpers.set_streamk(-1)
    for i, (o, lse) in enumerate(got):
        assert torch.equal(o, want[i % 5][0]) and torch.equal(lse, want[i % 5][1]), i


@pytest.mark.gpu
def test_two_streams_at_once():
    """Calls on two streams whose kernels run beside each other: each gets its own results."""
    from sageattention_rdna3_b200 import sageattn
    torch.manual_seed(2)
    work = [([torch.randn(1, 4, s, d, device="cuda").to(t) for _ in range(3)], kw, torch.cuda.Stream())
            for s, d, t, kw in ((2304, 128, torch.bfloat16, dict(smooth_k=True)),
                                (1500, 64, torch.float16, dict(is_causal=True, kernel="int8")))]
    want = [sageattn(*x, **kw) for x, kw, _ in work]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for i, (x, kw, stream) in enumerate(work):
            with torch.cuda.stream(stream):
                got[i].append(sageattn(*x, **kw))
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(o, want[i]) for o in got[i])


def test_nothing_shared_is_taken_before_the_kernel_ahead_has_ended():
    """Read from the source (a kernel that breaks this may wait for ever, so it is not run): in the attention
    kernel nothing before the first dependency wait of the normal path allocates TMEM, starts a copy or reads
    global memory through the parameters."""
    import re
    from sageattention_rdna3_b200.build import CSRC
    text = re.sub(r"//[^\n]*", "", (CSRC / "attn_kernel.cuh").read_text())
    body = text[text.index("\nsage_attn_kernel("):]
    setup = body.index("mbar_init(q_full")
    before = body[setup:body.index("grid_dependency_wait();", setup)]
    for word in ("tmem_alloc", "load_q(", "load_k(", "tma_load", "p.status", "p.q_scale", "__ldg", "atomic"):
        assert word not in before, word
    assert body.index("tmem_alloc(") > body.index("grid_dependency_wait();", setup)
    # and the successor is not let in before the block has its own TMEM (the barrier behind the allocation)
    alloc = body.index("tmem_alloc(")
    assert body.index("grid_launch_dependents();") > body.index("__syncthreads();", alloc)


@pytest.mark.gpu
@pytest.mark.parametrize("H,S,D,dtype,kernel,smooth", [
    (4, 4096, 128, torch.bfloat16, "int8", False), (8, 2304, 128, torch.bfloat16, "int8", True),
    (4, 4500, 64, torch.float16, "int8", False), (8, 2048, 64, torch.bfloat16, "direct", False),
    (6, 3072, 64, torch.bfloat16, "direct", False)])
def test_small_launches_get_an_sm_per_block(H, S, D, dtype, kernel, smooth):
    """128 to 144 plain attention blocks behind a preparation that lets them start early: no SM runs two of them
    while others run none (counted by the kernel itself)."""
    import ctypes
    import helpers
    from sageattention_rdna3_b200 import _native, sageattn
    lib = _native.load_abi()
    n_sms = torch.cuda.get_device_properties(0).multi_processor_count
    items = H * -(-S // 128)
    if items > n_sms:
        pytest.skip("needs an SM for every block")

    def counts():
        c = (ctypes.c_uint32 * 1024)()
        assert lib.sage_test_sm_arrivals(c, 1024) == 0
        return list(c)

    torch.manual_seed(0)
    q, k, v = (torch.randn(1, S, H, D, device="cuda").to(dtype) for _ in range(3))
    call = lambda: sageattn(q, k, v, tensor_layout="NHD", kernel=kernel, smooth_k=smooth)
    try:
        helpers.set_streamk(0)
        call()
        for _ in range(4):
            torch.cuda.synchronize()
            before = counts()
            torch.cuda._sleep(1_000_000)         # about half a millisecond: both launches are queued before either runs
            call()
            torch.cuda.synchronize()
            new = [b - a for a, b in zip(before, counts())]
            assert sum(new) == items and max(new) == 1
    finally:
        helpers.set_streamk(-1)
