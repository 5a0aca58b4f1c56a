"""Element-wise bids with the inclusive share step as one key-stationary sweep, against the column-sum and main passes it replaces in
training forwards (which the goldens and the oracle hold), on both block sizes and ragged lengths."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(pkg, q, k, v, bid, shift, eps, fused, share=1):
    lib, L = pkg._lib.load(), pkg._lib
    n, seq = q.shape[1], q.shape[2]
    out, ssum, total = (torch.empty(n, seq, *s, device=DEV) for s in ((64,), (), ()))
    carry = torch.zeros(n, (seq + 31) // 32, seq, device=DEV)
    args = (*(x.data_ptr() for x in (q, k, v)), L.BF16, L.PREC["bf16"], n, seq, 64, 0.125, eps, L.BID[bid])
    st = torch.cuda.current_stream().cuda_stream
    if fused:
        rc = lib.dilution_variant_forward_fused(*args, shift, carry.data_ptr(), total.data_ptr(), out.data_ptr(), ssum.data_ptr(), st)
    else:
        rc = lib.dilution_variant_forward(*args, share, shift, None, None, carry.data_ptr(), total.data_ptr(), out.data_ptr(),
                                          ssum.data_ptr(), None, st)
    L.check(rc, "variant forward")
    return out, ssum, total, carry


def _inputs(rows, seq, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(rows * seq)
    q, k, v = (torch.randn(1, rows, seq, 64, device=DEV, generator=g) for _ in range(3))
    return (q * std).bfloat16(), k.bfloat16(), v.bfloat16()


# 128 and 512 keys per block (200 blocks of 512), lengths around tiles, half tiles and checkpoints
@pytest.mark.parametrize("rows,seq", [(1, 1), (2, 31), (1, 65), (3, 127), (2, 513), (1, 1777), (200, 129), (67, 1100), (100, 1024)])
@pytest.mark.parametrize("bid,shift", [("sigmoid", 1.0), ("sigshift", 40.0), ("expshift", 1000.0)])
@pytest.mark.parametrize("eps,std", [(1e-9, 1.0), (1e-30, 8.0)])
def test_sweep_matches_the_two_passes(rows, seq, bid, shift, eps, std):
    pkg = load_package()
    x = _inputs(rows, seq, std)
    (out, ssum, total, carry), (ref, rsum, rtotal, rcarry) = (_run(pkg, *x, bid, shift, eps, fused) for fused in (True, False))
    # demands are fp32 sums of the same bids in another order; every fourth exponential is a polynomial (2e-7)
    assert ((total - rtotal).abs() <= 2e-5 * rtotal.abs() + 1e-30).all()
    block = torch.arange(carry.shape[1], device=DEV)[:, None] * 32
    seen = torch.arange(seq, device=DEV)[None] < block         # what a backward reads: keys in front of a block's first query
    assert ((carry - rcarry).abs() <= 2e-5 * rcarry.abs() + 1e-30)[:, seen].all()
    # both round shares to 8 bits, at different values where the demands' last bits differ: 2^-8 of a share each
    assert ((ssum - rsum).abs() <= 2.0 ** -7 * rsum.abs() + 1e-6).all()
    assert (out - ref).abs().max().item() <= 2.0 ** -6 * ref.abs().max().item()


def test_a_query_that_is_not_a_number_stays_in_its_rows_and_demands():
    pkg = load_package()
    q, k, v = _inputs(2, 700)
    q[0, 0, 300] = float("nan")
    out, _, total, _ = _run(pkg, q, k, v, "sigmoid", 1.0, 1e-9, True)
    assert out[0, 300].isnan().all() and out[0, :300].isfinite().all() and out[1].isfinite().all()
    assert total[0, :301].isnan().all() and total[0, 301:].isfinite().all()


def _one_large_score(rows, seq, row, key, score):
    """q, k, v with one score of that size, of query `row` and key `key` of the first row; no other score of that key is above 0."""
    q, k, v = _inputs(rows, seq, 0.5)
    q[0, 0, :, 0], q[0, 0, row], k[0, 0, key] = 0.0, 0.0, 0.0
    q[0, 0, row, 0], k[0, 0, key, 0] = score / 2, 16.0
    return q, k, v


# both block sizes; every position modulo four (one exponential in four is a polynomial), the first and the last of a chunk of 32
@pytest.mark.parametrize("rows,seq", [(2, 200), (200, 600)])
@pytest.mark.parametrize("row", [60, 61, 62, 63, 64, 67, 96])
@pytest.mark.parametrize("score", [88.5, 89.5, 98.5, 150.0, 400.0])
@pytest.mark.parametrize("fused", [True, False])
def test_an_expshift_bid_that_overflows_spoils_its_own_row(rows, seq, row, score, fused):
    """exp(88.5) is an fp32 number, exp(89.5) is not: its demand is infinite from there on and its own row is inf / inf, but later
    rows are finite: nobody gets a share of that key any more."""
    pkg = load_package()
    key = 40
    out, ssum, total, carry = _run(pkg, *_one_large_score(rows, seq, row, key, score), "expshift", 1.0, 1e-9, fused)
    over = score > 88.7
    nan_rows = out[0].isnan().any(-1).nonzero().flatten().tolist()
    assert nan_rows == ([row] if over else []), nan_rows
    assert out[1:].isfinite().all() and not total.isnan().any()
    if over:
        assert total[0, key] == float("inf") and out[0, row].isnan().all() and ssum[0, row].isnan()
        assert (carry[0, row // 32 + 1:, key] == float("inf")).all()
    else:
        assert abs(total[0, key].item() / 2.7230907e38 - 1) < 1e-4            # exp(88.5)
    keep = torch.ones(seq, dtype=torch.bool, device=DEV)
    keep[key] = False
    assert total[0, keep].isfinite().all() and carry[0, :, :key].isfinite().all()


@pytest.mark.parametrize("row", [60, 61, 62, 63, 67, 127])
@pytest.mark.parametrize("share", [0, 2])
@pytest.mark.parametrize("score", [88.5, 89.5, 150.0])
def test_an_expshift_bid_that_overflows_without_the_inclusive_step(row, share, score):
    """Its share, and the row's sum, are infinite; later shares of the key after the exclusive step are 0."""
    pkg = load_package()
    q, k, v = _one_large_score(2, 200, row, 40, score)
    v = (v.float() * 0.1).bfloat16()                         # (the bid times a value, in fp32, is to be finite)
    out, ssum, _, _ = _run(pkg, q, k, v, "expshift", 1.0, 1.0, False, share)
    over = score > 88.7
    assert out[0].isnan().any(-1).nonzero().flatten().tolist() == ([row] if over else [])
    assert out[1].isfinite().all() and ssum[0, row].isinf().item() is over
    if not over:                                             # all of the row's share
        assert (out[0, row] - v[0, 0, 40].float()).abs().max().item() < 2e-3


def test_training_calls_take_it():
    pkg = load_package()
    x, y = ([t.requires_grad_(True) for t in _inputs(rows, 2048)] for rows in (8, 7))
    for share, name, x in ((True, "tc_forward_fused", x), ("exclusive", "tc_forward_main", x), (True, "tc_forward_main", y)):
        pkg._lib.profile(True)
        pkg._lib.profile_collect()
        pkg.kernels_bid.dilution_attention(*x, dot_precision="bf16", bid="sigmoid", share_cumsum=share)
        names = set(pkg._lib.profile_collect())
        pkg._lib.profile(False)
        assert name in names, names


def test_deterministic_algorithms_keep_the_two_passes():
    pkg = load_package()
    x = [t.requires_grad_(True) for t in _inputs(8, 2048)]
    call = lambda: pkg.kernels_bid.dilution_attention(*x, dot_precision="bf16", bid="sigmoid", share_cumsum=True)      # noqa: E731
    sweep = call().detach()
    torch.use_deterministic_algorithms(True)
    try:
        pkg._lib.profile(True)
        pkg._lib.profile_collect()
        got = [call().detach() for _ in range(3)]
        names = set(pkg._lib.profile_collect())
        pkg._lib.profile(False)
    finally:
        torch.use_deterministic_algorithms(False)
    assert "tc_forward_main" in names and "tc_forward_fused" not in names, names
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert (sweep - got[0]).abs().max().item() < 1e-2                      # both round their shares to bf16


def test_other_calls_are_refused():
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    one = 256                                                 # never dereferenced
    for dtype, prec, d, bid in ((L.F32, L.PREC["tf32"], 64, "sigmoid"), (L.BF16, L.PREC["bf16"], 32, "sigmoid"),
                                (L.BF16, L.PREC["bf16"], 64, "softmax"), (L.BF16, L.PREC["bf16"], 64, "relu")):
        assert lib.dilution_variant_forward_fused(one, one, one, dtype, prec, 1, 8, d, 0.125, 1e-9, L.BID[bid], 1.0, one, one, one,
                                                  one, None) == 2
