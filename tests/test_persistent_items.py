"""Persistent launches against the plain one where only some items, or none, are cut: what is not a number, and items of
one tile."""
import pytest
import torch

import helpers as H


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", [-1, 1])
@pytest.mark.parametrize("B,Hq,Sq,Skv,D,kernel", [
    (1, 20, 2048, 2048, 128, "direct"),     # pairs of query tiles: whole and cut items in one launch
    (1, 10, 4096, 4096, 64, "int8"),        # the same, quantised
    (1, 3, 300, 1500, 64, "direct"),        # too few items for pairs
])
def test_not_a_number_is_where_it_is_in_one_piece(B, Hq, Sq, Skv, D, kernel, schedule):
    from sageattention_rdna3_b200 import sageattn
    q, k, v = (H.randn((B, Hq, s, D), i, torch.float16) for i, s in enumerate((Sq, Skv, Skv)))
    q[:, :, 7] *= 500                       # one key takes all the weight: that of other parts underflows
    v[:, 1::5, 3, 9] = float("nan")         # ... and 0 * NaN is NaN
    v[:, 2::5, -1, 11] = float("inf")
    if kernel == "direct":                  # (the quantisation makes numbers of these)
        q[:, :, 130] = float("nan")         # all scores of a row
        k[:, 0::4, Skv // 3, 2] = float("inf")   # one score of each row is infinite: NaN for a positive one
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    try:
        H.set_streamk(0)
        want, want_lse = sageattn(q, k, v, kernel=kernel, return_lse=True)
        H.set_streamk(schedule)
        got, got_lse = sageattn(q, k, v, kernel=kernel, return_lse=True)
    finally:
        H.set_streamk(-1)
    assert want.isnan().any() and not want.isnan().all()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got_lse.isnan(), want_lse.isnan()) and torch.equal(got_lse.isinf(), want_lse.isinf())
    # elsewhere: one rounding of the output, and that of P against other maxima (fp16)
    ok = want.isfinite() & got.isfinite()
    assert (got[ok].float() - want[ok].float()).norm() <= 2.0 ** -10 * want[ok].float().norm()


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["int8", "direct"])
@pytest.mark.parametrize("B,heads,Sq,Skv,D,causal", [(1, 1, 1, 1, 64, False), (2, 301, 300, 128, 128, False), (1, 300, 128, 77, 64, True)])
def test_items_of_one_tile(B, heads, Sq, Skv, D, causal, kernel):
    """One tile per item: nothing is cut, and every output is written without a merge."""
    from sageattention_rdna3_b200 import check_status, sageattn
    q, k, v = (H.randn((B, heads, s, D), i, torch.bfloat16).cuda() for i, s in enumerate((Sq, Skv, Skv)))
    outs = []
    for schedule in (0, 1):
        try:
            H.set_streamk(schedule)
            out = torch.full_like(q, float("nan"))
            outs.append(sageattn(q, k, v, is_causal=causal, kernel=kernel, return_lse=True, out=out))
        finally:
            H.set_streamk(-1)
    check_status()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
