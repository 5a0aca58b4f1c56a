"""The exact fp32 passes of few blocks, shared by clusters of 2, 4 and 8 CTAs: every split and the unsplit form, ragged last
tiles and ranks without a tile, against the oracle (1e-4, as the other "ieee" tests) for the operator, and for a bid whose
reverse pass runs twice."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O
from test_gpu_variants import check_grads

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,seq,d", [(1, 65, 64), (2, 129, 32), (3, 300, 128), (4, 512, 64), (4, 577, 16), (19, 513, 64),
                                        (37, 200, 64), (2, 1500, 64), (100, 130, 64)])
def test_exact_operator(dtype, rows, seq, d):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, rows, seq, d, 40 + seq)
    q, k, v = (t.to(dtype).float() for t in (q, k, v))
    ref, *grads = O.dilution_backward(q, k, v, dout)
    leaves = [t.to(DEV, dtype).requires_grad_(True) for t in (q, k, v)]
    out = pkg.dilution_attention(*leaves, dot_precision="ieee")
    out.backward(dout.to(DEV))
    assert rel_err(out.detach().cpu(), ref) < 1e-4
    for name, t, g in zip(("dq", "dk", "dv"), leaves, grads):
        # a bf16 gradient is rounded once
        assert rel_err(t.grad.float().cpu(), g) < (1e-4 if dtype == torch.float32 else 2.0 ** -8), name


@pytest.mark.parametrize("bid,share", [("softplus", True), ("minshift", "exclusive"), ("sigmoid", False)])
def test_bids(bid, share):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, 2, 400, 64, 9)
    ref, *grads = O.variant_backward(q, k, v, dout, bid, share, 1.0)
    leaves = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    out = pkg.kernels_bid.dilution_attention(*leaves, dot_precision="ieee", bid=bid, share_cumsum=share)
    out.backward(dout.to(DEV))
    assert rel_err(out.detach().cpu(), ref) < 1e-4
    check_grads(share, [t.grad for t in leaves], grads, 2e-3)
