"""The reverse pass of the sigmoid's bid in slices of 32 queries: the route at its edge, lengths around slices, half tiles and blocks,
flat and peaked bids, against the oracle; both share steps with an eps of 1 against 64 bits; values that are not finite."""

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


@pytest.mark.parametrize("seq", [1535, 1536, 1567, 1665])
@pytest.mark.parametrize("share", [1, 2])
def test_gradients_with_a_large_eps_against_64_bits(seq, share):
    """With eps = 1 no demand is small, and the exclusive step's dq and dk have values to compare: 1e9-fold terms that cancel
    otherwise.  Shares, pdp, do' and the gradients have 8 bits: 2-norm errors of 2.9e-3, largest 5e-3 of the largest value."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    n, eps = 3, 1.0
    g = torch.Generator(device=DEV).manual_seed(seq)
    q, k, v = (torch.randn(n, seq, 64, device=DEV, generator=g).bfloat16() for _ in range(3))
    dout = torch.randn(n, seq, 64, device=DEV, generator=g) * 1e-2
    out, ssum, total = (torch.empty(n, seq, *s, device=DEV) for s in ((64,), (), ()))
    carry = torch.zeros(n, (seq + 31) // 32, seq, device=DEV)
    st = torch.cuda.current_stream().cuda_stream
    args = (*(x.data_ptr() for x in (q, k, v)), L.BF16, L.PREC["bf16"], n, seq, 64, 0.125, eps, L.BID["sigmoid"], share, 1.0)
    parts = [x.data_ptr() for x in (carry, total)]
    L.check(lib.dilution_variant_forward(*args, None, None, *parts, out.data_ptr(), ssum.data_ptr(), None, st), "forward")
    scratch = torch.empty(lib.dilution_backward_scratch_bytes(n, seq, 64), device=DEV, dtype=torch.uint8)
    grads = [torch.empty_like(q) for _ in range(3)]
    L.check(lib.dilution_variant_backward(*args, dout.data_ptr(), out.data_ptr(), None, None, *parts, ssum.data_ptr(), None,
                                          scratch.data_ptr(), *(x.data_ptr() for x in grads), st), "backward")
    leaves = [x.double().requires_grad_(True) for x in (q, k, v)]
    p = torch.sigmoid(leaves[0] @ leaves[1].mT / 8)
    p = p.masked_fill(torch.ones(seq, seq, device=DEV, dtype=torch.bool).triu(1), 0.0)
    demand = p.cumsum(1) if share == 1 else p.cumsum(1) - p
    shares = p / (demand + eps)
    ref = shares / (shares.sum(-1, keepdim=True) + eps) @ leaves[2]
    assert ((out - ref).norm() / ref.norm()).item() < 4e-3
    for got, want in zip(grads, torch.autograd.grad(ref, leaves, dout.double())):
        assert ((got - want).norm() / want.norm()).item() < 6e-3
        assert (got - want).abs().max().item() < 1.5e-2 * want.abs().max().item()


@pytest.mark.parametrize("what,value", [("q", "nan"), ("k", "nan"), ("v", "nan"), ("v", "inf")])
@pytest.mark.parametrize("pos", [3, 700, 1589])
@pytest.mark.parametrize("share", [True, "exclusive"])
def test_values_that_are_not_finite(what, value, pos, share):
    """Outputs and gradients are finite where the exact path's are, and the other row's stay what they are."""
    pkg = load_package()
    x = list(make_inputs(1, 2, 1590, 64, 4, scales=(1.0, 1.0, 1.0, 1e-2)))
    x[:3] = [t.bfloat16() for t in x[:3]]

    def run(precision):
        leaves = [(t if precision == "bf16" else t.float()).to(DEV).requires_grad_(True) for t in x[:3]]
        out = pkg.kernels_bid.dilution_attention(*leaves, dot_precision=precision, bid="sigmoid", share_cumsum=share)
        return [t.float() for t in (out.detach(), *torch.autograd.grad(out, leaves, x[3].to(DEV)))]

    clean = run("bf16")
    x["qkv".index(what)][0, 0, pos, 5] = float(value)
    for got, exact, before in zip(run("bf16"), run("ieee"), clean):
        assert torch.equal(got.isfinite(), exact.isfinite())
        assert got[0, 1].isfinite().all()
        if share is True:       # a sum of dq or of the output in another order may round to the next bf16
            assert rel_err(got[0, 1].cpu(), before[0, 1].cpu()) < 2.0 ** -8
