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
    chained = [sageattn(sageattn(q, k, v, smooth_k=smooth), k, v, smooth_k=smooth) for _ in range(8)]
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 4]) for i, o in enumerate(got))
    assert all(torch.equal(o, chained[0]) for o in chained)
