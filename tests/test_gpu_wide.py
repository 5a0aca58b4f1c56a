"""Rows of 256 bytes on the tcgen05 kernels: bf16 heads of 128 under "bf16" and fp32 heads of 16, 32 and 64
under "tf32" (values as bf16 pairs hi + lo), forward and backward against the oracle at the edges of the 128-row tiles
and 64-query half-steps.

Bounds.  bf16: those of the other bf16 tests.  fp32: a product of two hi + lo operands drops lo * lo and the bits
below lo, 2^-16 of each term; scores of standard deviation 1 reach 6, so p and the shares are off by
at most 6 * 2^-16 = 1e-4 relative and a gradient, which multiplies two of them, by a few times that."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("seq", [1, 63, 64, 65, 128, 129, 257, 700, 1100])
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 128), (torch.float32, 64), (torch.float32, 32), (torch.float32, 16)])
def test_wide_rows_match_the_oracle(kernels, dtype, d, seq):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, 3, seq, d, 300 + seq, scales=(1.0, 1.0, 1.0, 1e-1))
    q, k, v = (x.to(dtype) for x in (q, k, v))
    ref = O.dilution_backward(q.float(), k.float(), v.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    prec = "bf16" if dtype == torch.bfloat16 else "tf32"
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out = kernels.dilution_attention(qs, ks, vs, dot_precision=prec)
    out.backward(dout.to(DEV))
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert {"tc_wide_forward_main", "tc_wide_backward_main"} <= names and not any(n.startswith("simt_") for n in names), names
    tol, gtol = (2e-2, 3e-2) if dtype == torch.bfloat16 else (2e-4, 5e-4)
    assert (out.detach().cpu() - ref[0]).abs().max().item() < tol
    for name, r, x in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert x.grad.dtype == dtype and torch.isfinite(x.grad).all(), name
        # a single row's gradients are rounding noise on an identically zero dq and dk
        if seq > 1 or name == "dv":
            assert rel_err(x.grad.float().cpu(), r) < gtol, name
    # forward only: the row pass without its product, demand totals and every checkpoint's last row
    got, aux = kernels.dilution_attention_forward(qs.detach(), ks.detach(), vs.detach(), dot_precision=prec, return_aux=True)
    assert (got.cpu() - ref[0]).abs().max().item() < tol and aux["bwd_block_m"] == 32 and aux["pk"] is None
    demand = O.demand_totals(q.float(), k.float())
    assert rel_err(aux["committed_total"].cpu(), demand) < tol


@pytest.mark.parametrize("dtype,d,tol", [(torch.bfloat16, 128, 3e-2), (torch.float32, 64, 5e-4)])
def test_wide_rows_with_peaked_scores_and_saved_pk(kernels, dtype, d, tol):
    """Scores of standard deviation 8: the row pass moves its reference and rescales both halves of its accumulators.
    p carries the score's error times its magnitude, 50 * 2^-16."""
    q, k, v, dout = make_inputs(1, 2, 900, d, 71, scales=(2.83, 2.83, 1.0, 1e-1))
    q, k, v = (x.to(dtype) for x in (q, k, v))
    prec = "bf16" if dtype == torch.bfloat16 else "tf32"
    _, aux = kernels.dilution_attention_forward(q.to(DEV), k.to(DEV), v.to(DEV), dot_precision=prec, return_aux=True,
                                                _save_pk=True)
    assert rel_err(aux["pk"].reshape(1, 2, 900, d).cpu(), O.query_correction(q.float(), k.float())) < max(tol / 3, 1e-3)
    rmax, rden = O.row_stats(q.float(), k.float())
    lse = (aux["rmax"] + torch.log2(aux["rden"])).reshape(1, 2, 900).cpu()
    assert (lse - (rmax + torch.log2(rden))).abs().max().item() < 2e-3
    ref = O.dilution_backward(q.float(), k.float(), v.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    kernels.dilution_attention(qs, ks, vs, dot_precision=prec).backward(dout.to(DEV))
    for name, r, x in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert rel_err(x.grad.float().cpu(), r) < max(tol, 2e-3), name


def test_wide_entry_points_refuse_other_cases():
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    one = 256      # never dereferenced
    rc = lib.dilution_wide_forward(one, one, one, L.BF16, 1, 64, 64, 0.125, 1e-9, one, one, one, one, one, one, None, None)
    assert rc == 2 and b"heads of 128" in lib.dilution_last_error()
    rc = lib.dilution_split_operands(one, one, one, 64, 128, one, one, one, None)
    assert rc == 1 and b"16, 32, 64" in lib.dilution_last_error()
