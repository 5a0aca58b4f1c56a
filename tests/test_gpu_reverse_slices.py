"""The reverse pass of the sigmoid's bid in slices of 32 queries: the route at its edge, lengths around slices, half tiles and blocks,
flat and peaked bids, against the oracle."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("seq", [1535, 1536, 1537, 1567, 1569, 1601, 1664, 1665, 2049])
@pytest.mark.parametrize("bid,shift,share,std", [("sigmoid", 1.0, True, 0.5), ("sigmoid", 1.0, True, 4.0), ("sigshift", 30.0, True, 0.5),
                                                 ("sigmoid", 1.0, "exclusive", 0.5)])
def test_gradients(seq, bid, shift, share, std):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, 3, seq, 64, 7 + seq, scales=(std, 0.5, 1.0, 1.0))
    qb, kb, vb = (t.bfloat16() for t in (q, k, v))
    _, *grads = O.variant_backward(qb.float(), kb.float(), vb.float(), dout, bid, share, shift)
    leaves = [t.to(DEV).requires_grad_(True) for t in (qb, kb, vb)]
    out = pkg.kernels_bid.dilution_attention(*leaves, dot_precision="bf16", bid=bid, share_cumsum=share, shift=shift)
    out.backward(dout.to(DEV))
    # shares, pdp and do' have 8 bits, a gradient is a sum of many of either sign: 2e-2 of its largest value, as for the other
    # kernels of bf16 tensors.  The exclusive step's dq and dk are differences of 1e9-fold terms, so only dv has a value
    for t, grad, exact in zip(leaves, grads, (share is True, share is True, True)):
        assert t.grad.isfinite().all()
        if exact:
            assert rel_err(t.grad.float().cpu(), grad) < 2e-2


def test_it_is_as_exact_as_the_pass_of_shorter_rows():
    """The 2-norm error against the fp32 path's gradients, on both sides of the line."""
    pkg = load_package()
    errors = {}
    for seq in (1535, 1536):
        x = make_inputs(1, 4, seq, 64, 3, scales=(0.5, 0.5, 1.0, 1e-2))
        got = []
        for precision in ("bf16", "ieee"):
            leaves = [t.bfloat16().to(DEV).requires_grad_(True) for t in x[:3]]
            ops = leaves if precision == "bf16" else [t.detach().float().requires_grad_(True) for t in leaves]
            out = pkg.kernels_bid.dilution_attention(*ops, dot_precision=precision, bid="sigmoid", share_cumsum=True)
            got.append([g.float() for g in torch.autograd.grad(out, ops, x[3].to(DEV))])
        errors[seq] = [((a - b).norm() / b.norm()).item() for a, b in zip(*got)]
    for long, short in zip(errors[1536], errors[1535]):
        assert long < 1.1 * short, errors                     # the same operands and roundings
