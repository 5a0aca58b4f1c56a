"""Shares are taken two at a time from one reciprocal where every demand lies between 1e-18 and 1e18, one at a time
elsewhere: an expshift bid whose bids are far beyond that, and an eps far below it (a C ABI argument), against 64 bits.  Bounds
of the other bf16 tests."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _dense(q, k, v, bid, eps):
    a = (q.double() @ k.double().transpose(-1, -2)) * 0.125
    t = a.shape[-1]
    mask = torch.ones(t, t, device=a.device).triu(1).bool()
    p = bid(a.masked_fill(mask, float("-inf")))
    share = p / (p.cumsum(-2) + eps)
    return p, share @ v.double() / (share.sum(-1, keepdim=True) + 1e-9)


@pytest.mark.parametrize("shift", [1e-25, 1e-20, 64.0])
def test_expshift_bids_of_any_size(shift):
    pkg = load_package()
    q, k, v, _ = make_inputs(1, 2, 300, 64, 31)
    qb, kb, vb = (x.bfloat16().to(DEV) for x in (q, k, v))
    got = pkg.kernels_bid.dilution_attention_forward(qb, kb, vb, dot_precision="bf16", bid="expshift", share_cumsum=True,
                                                     shift=shift)
    _, ref = _dense(qb, kb, vb, lambda a: a.exp() / shift, 1e-9)
    assert (got.double() - ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("eps", [1e-9, 1e-30])
@pytest.mark.parametrize("fused", [False, True])
def test_eps_of_any_size(eps, fused):
    """Keys that grow along the sequence: a late key's first bids are far above, an early key's late ones far below."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    t, d = 200, 64
    q, k, v, _ = make_inputs(1, 1, t, d, 5, scales=(1.5, 1.5, 1.0, 1.0))
    qb, kb, vb = (x.bfloat16().to(DEV) for x in (q, k, v))
    f = lambda *s: torch.empty(*s, device=DEV)
    rmax, rden, total, ssum, out, carry = f(t), f(t), f(t), f(t), f(t, d), f((t + 31) // 32, t)
    st = torch.cuda.current_stream().cuda_stream
    p = [x.data_ptr() for x in (qb, kb, vb)]
    L.check(lib.dilution_rowstats(p[0], p[1], L.BF16, 2, 1, t, t, 0, d, 0.125, rmax.data_ptr(), rden.data_ptr(), st), "rowstats")
    if fused:
        L.check(lib.dilution_forward_fused(*p, L.BF16, 2, 1, t, d, 0.125, eps, rmax.data_ptr(), rden.data_ptr(), carry.data_ptr(),
                                           total.data_ptr(), out.data_ptr(), ssum.data_ptr(), st), "fused")
    else:
        L.check(lib.dilution_colsum_scan(p[0], p[1], L.BF16, 2, 1, t, t, 0, d, 0.125, rmax.data_ptr(), rden.data_ptr(), None, 32,
                                         carry.data_ptr(), total.data_ptr(), st), "colsum")
        L.check(lib.dilution_forward_main(*p, L.BF16, 2, 1, t, t, 0, d, 0.125, eps, rmax.data_ptr(), rden.data_ptr(),
                                          carry.data_ptr(), 32, None, out.data_ptr(), ssum.data_ptr(), None, st), "main")
    bid, ref = _dense(qb, kb, vb, lambda a: torch.softmax(a, -1), eps)
    assert bid[bid > 0].min().item() > 1e-12          # nothing near the 2^-125 at which every fourth exponential ends
    assert rel_err(out.double().cpu(), ref[0, 0].cpu()) < 2e-2


@pytest.mark.parametrize("rows,seq", [(1, 200), (52, 2049)])
@pytest.mark.parametrize("eps", [1e-30, 1e20])
@pytest.mark.parametrize("path", ["sweep32", "sweep64", "two passes"])
def test_row_sums_under_an_eps_outside_the_range_of_pairs(path, eps, rows, seq):
    """Every sweep (blocks of 128 and of 512 keys, checkpoints every 32 and 64 rows) and the main pass without pairs.  Shares of
    1e-20 are summed as bf16."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    q, k, v, _ = make_inputs(1, rows, seq, 64, 6, scales=(1.0, 1.0, 1.0, 1.0))
    qb, kb, vb = (x.bfloat16().to(DEV) for x in (q, k, v))
    step = 64 if path == "sweep64" else 32
    f = lambda *s: torch.empty(rows, *s, device=DEV)
    rmax, rden, total, ssum, out, carry = f(seq), f(seq), f(seq), f(seq), f(seq, 64), f((seq + step - 1) // step, seq)
    st = torch.cuda.current_stream().cuda_stream
    p = [x.data_ptr() for x in (qb, kb, vb)]
    stats = rmax.data_ptr(), rden.data_ptr()
    L.check(lib.dilution_rowstats(p[0], p[1], L.BF16, 2, rows, seq, seq, 0, 64, 0.125, *stats, st), "rowstats")
    if path == "two passes":
        L.check(lib.dilution_colsum_scan(p[0], p[1], L.BF16, 2, rows, seq, seq, 0, 64, 0.125, *stats, None, step,
                                         carry.data_ptr(), total.data_ptr(), st), "colsum")
        L.check(lib.dilution_forward_main(*p, L.BF16, 2, rows, seq, seq, 0, 64, 0.125, eps, *stats, carry.data_ptr(), step, None,
                                          out.data_ptr(), ssum.data_ptr(), None, st), "main")
    else:
        L.check(lib.dilution_forward_fused_rows(*p, L.BF16, 2, rows, seq, 64, 0.125, eps, *stats, step, carry.data_ptr(),
                                                total.data_ptr(), out.data_ptr(), ssum.data_ptr(), st), "fused")
    for r in (0, rows - 1):
        bid, ref = _dense(qb[0, r], kb[0, r], vb[0, r], lambda a: torch.softmax(a, -1), eps)
        share = bid / (bid.cumsum(-2) + eps)
        assert (ssum[r].double() / share.sum(-1) - 1).abs().max().item() < 2.0 ** -8          # bf16 shares, half an ulp
        if eps < 1:
            assert rel_err(out[r].double().cpu(), ref.cpu()) < 2e-2
            assert rel_err(total[r].double().cpu(), bid.sum(-2).cpu()) < 1e-4


@pytest.mark.parametrize("base", [float("inf"), 1e30])
def test_a_key_that_is_all_demanded_already(base):
    """A starting demand that is infinite (or far above the range of pairs) takes the key out of every row."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    t = 200
    q, k, v, _ = make_inputs(1, 1, t, 64, 7, scales=(1.0, 1.0, 1.0, 1.0))
    qb, kb, vb = (x.bfloat16().to(DEV) for x in (q, k, v))
    f = lambda *s: torch.empty(*s, device=DEV)
    rmax, rden, total, ssum, out, carry = f(t), f(t), f(t), f(t), f(t, 64), f((t + 31) // 32, t)
    demand = torch.zeros(t, device=DEV)
    demand[5] = base
    st = torch.cuda.current_stream().cuda_stream
    p, stats = [x.data_ptr() for x in (qb, kb, vb)], (rmax.data_ptr(), rden.data_ptr())
    L.check(lib.dilution_rowstats(p[0], p[1], L.BF16, 2, 1, t, t, 0, 64, 0.125, *stats, st), "rowstats")
    L.check(lib.dilution_colsum_scan(p[0], p[1], L.BF16, 2, 1, t, t, 0, 64, 0.125, *stats, None, 32, carry.data_ptr(),
                                     total.data_ptr(), st), "colsum")
    L.check(lib.dilution_forward_main(*p, L.BF16, 2, 1, t, t, 0, 64, 0.125, 1e-9, *stats, carry.data_ptr(), 32,
                                      demand.data_ptr(), out.data_ptr(), ssum.data_ptr(), None, st), "main")
    bid, _ = _dense(qb, kb, vb, lambda a: torch.softmax(a, -1), 1e-9)
    share = (bid / (bid.cumsum(-2) + 1e-9))[0, 0]
    share[:, 5] = 0.0
    ref = share @ vb[0, 0].double() / (share.sum(-1, keepdim=True) + 1e-9)
    assert rel_err(out.double().cpu(), ref.cpu()) < 2e-2
