"""Which calls take the fused sweep, at the edges of the rule, and both sides of it against the oracle."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 74 blocks of 256 keys at 1536 tokens, 101 of them, 256 blocks of 512 from 1024 tokens on, and (40 x 2560) the CTAs of 512 keys
@pytest.mark.parametrize("rows,seq,sweep", [(12, 1536, True), (13, 1536, False), (17, 1536, True), (17, 1535, False), (127, 1024, False),
                                            (128, 1024, True), (128, 1023, False), (12, 2304, True), (39, 2559, True), (40, 2560, True)])
def test_training_calls(rows, seq, sweep):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, rows, seq, 64, 3 + seq, scales=(0.5, 0.5, 1.0, 1e-2))
    leaves = [t.bfloat16().to(DEV).requires_grad_(True) for t in (q, k, v)]
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out = pkg.kernels.dilution_attention(*leaves, dot_precision="bf16")
    out.backward(dout.to(DEV))
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert ("tc_forward_fused" in names, "tc_forward_main" in names) == (sweep, not sweep), names
    r = rows - 1                                      # the rows are independent
    ref, *grads = O.dilution_backward(*(t[:, r:].bfloat16().float() for t in (q, k, v)), dout[:, r:])
    # operands are exact, shares and pdp have 8 bits: 2^-8 of an output, a few of a gradient's largest value
    assert (out[:, r:].detach().cpu() - ref).abs().max().item() < 2e-2
    for t, grad in zip(leaves, grads):
        assert rel_err(t.grad[:, r:].float().cpu(), grad) < 3e-2


@pytest.mark.parametrize("seq,sweep", [(2048, False), (2049, True)])
def test_calls_that_no_backward_follows(seq, sweep):
    pkg = load_package()
    x = [t.bfloat16().to(DEV) for t in make_inputs(1, 2, seq, 64, 5, scales=(1.0, 1.0, 1.0, 1.0))[:3]]
    assert pkg.kernels._takes_sweep(pkg._lib.BF16, pkg._lib.PREC["bf16"], 2, seq, seq, 64, 64) is sweep
    out, aux = pkg.kernels.dilution_attention_forward(*x, dot_precision="bf16", return_aux=True)
    ref, demand = O.dilution_chunked(*(t.float().cpu() for t in x), return_demand=True)
    assert (out.cpu() - ref).abs().max().item() < 2e-2
    assert rel_err(aux["committed_total"].cpu().reshape(demand.shape), demand) < 1e-4
