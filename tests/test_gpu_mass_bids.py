"""relu, relu2 and softplus bids of bf16 heads of 64 on the tcgen05 kernels (from 641 tokens on): forward and
backward against the oracle and against the tile kernels ("tf32" on the same tensors), at edges of the 128-row tiles and
64-query half-steps.

Bounds: those of the other bf16 bids.  bf16 shares and Jacobian terms carry 2^-9 each; a row's gradient is a sum
of them, a single value is off by a few times that against the largest."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O
from test_gpu_variants import check_grads

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _grads(KB, x, dout, prec, bid, share):
    leaves = [t.to(DEV).requires_grad_(True) for t in x]
    out = KB.dilution_attention(*leaves, dot_precision=prec, bid=bid, share_cumsum=share)
    return (out.detach(), *torch.autograd.grad(out, leaves, dout.to(DEV)))


def _check_out(out, ref, share):
    """Exclusive share step, p / (c + eps): where a key's whole demand is one barely positive bid, an fp32 score's
    rounding (2^-21 of its terms) over that score, twice that for relu2, is the relative error of c, without a bound for
    a single row.  Such rows are few: 2-norm there, every value elsewhere."""
    if share == "exclusive":
        assert ((out - ref).norm() / ref.norm()).item() < 2e-2
    else:
        assert (out - ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("seq", [641, 703, 768, 1025, 1087, 1300])
@pytest.mark.parametrize("share", [True, "exclusive", False])
@pytest.mark.parametrize("bid", ["relu", "relu2", "softplus"])
def test_mass_bids_on_the_tensor_cores(bid, share, seq):
    pkg = load_package()
    KB = pkg.kernels_bid
    q, k, v, dout = make_inputs(1, 3, seq, 64, 900 + seq, scales=(0.7, 0.7, 1.0, 1.0))
    x = [t.bfloat16() for t in (q, k, v)]
    ref, *rgrads = O.variant_backward(*(t.float() for t in x), dout, bid, share, 1.0)
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out, *grads = _grads(KB, x, dout, "bf16", bid, share)
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert {"tc_rowstats", "tc_forward_main", "tc_backward_ghat", "tc_backward_main"} <= names, names
    assert not any(n.startswith("simt_") for n in names), names
    _check_out(out.cpu(), ref, share)
    check_grads(share, grads, rgrads, 2e-2)
    tile_out, *tile_grads = _grads(KB, x, dout, "tf32", bid, share)
    _check_out(out, tile_out, share)
    check_grads(share, grads, [t.float().cpu() for t in tile_grads], 2e-2)
    # forward only, with the row mass and the demand totals
    _, aux = KB.dilution_attention_forward(*(t.to(DEV) for t in x), dot_precision="bf16", return_aux=True, bid=bid,
                                           share_cumsum=share)
    _, tile = KB.dilution_attention_forward(*(t.to(DEV) for t in x), dot_precision="tf32", return_aux=True, bid=bid,
                                            share_cumsum=share)
    assert torch.equal(aux["rmax"], tile["rmax"]) and rel_err(aux["rden"].cpu(), tile["rden"].cpu()) < 1e-4
    assert rel_err(aux["committed_total"].cpu(), O.variant_bids(x[0].float(), x[1].float(), bid, 1.0).sum(-2)) < 1e-3


@pytest.mark.parametrize("bid", ["relu", "relu2", "softplus"])
def test_rows_without_mass_bid_uniformly(bid):
    """Queries against the keys: no score of the first 40 rows is positive.  relu and relu2 rows have no
    mass there and bid uniformly with a zero Jacobian; softplus rows keep theirs."""
    pkg = load_package()
    q, k, v, dout = make_inputs(1, 2, 1100, 64, 5, scales=(0.7, 0.7, 1.0, 1.0))
    q[:, :, :40] = -3.0 * k[:, :, :40].mean(dim=(0, 1, 2))
    k[:, :, :40] = k[:, :, :40].mean(dim=(0, 1, 2)) * torch.linspace(0.5, 1.5, 40)[:, None]
    x = [t.bfloat16() for t in (q, k, v)]
    ref, *rgrads = O.variant_backward(*(t.float() for t in x), dout, bid, True, 1.0)
    out, *grads = _grads(pkg.kernels_bid, x, dout, "bf16", bid, True)
    assert (out.cpu() - ref).abs().max().item() < 2e-2
    check_grads(True, grads, rgrads, 2e-2)
    if bid != "softplus":
        assert not grads[0][:, :, :40].any()


@pytest.mark.parametrize("bid", ["relu", "softplus"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_that_are_not_finite_reach_the_same_outputs(bid, value):
    """One key and, in another row, one query that are not finite: the outputs that are not finite are the tile kernels'."""
    pkg = load_package()
    q, k, v, _ = make_inputs(1, 2, 800, 64, 6, scales=(0.7, 0.7, 1.0, 1.0))
    k[0, 0, 302, 3] = value
    q[0, 1, 403, 5] = value
    x = [t.bfloat16().to(DEV) for t in (q, k, v)]
    out, tile = (pkg.kernels_bid.dilution_attention_forward(*x, dot_precision=p, bid=bid) for p in ("bf16", "tf32"))
    assert torch.equal(torch.isfinite(out).all(-1), torch.isfinite(tile).all(-1))
