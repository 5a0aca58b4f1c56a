"""Training forwards of many short rows take the column-sum and main passes, others the fused sweep: the choice at its
edges, and both sides of it against the oracle."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,seq,short", [(74, 100, True), (73, 256, False), (37, 257, True), (10, 2048, True),
                                            (9, 2048, False), (10, 2049, False)])
def test_route_and_gradients(rows, seq, short):
    pkg = load_package()
    q, k, v, dout = make_inputs(1, rows, seq, 64, 17 + seq, scales=(0.5, 0.5, 1.0, 1e-2))
    leaves = [t.bfloat16().to(DEV).requires_grad_(True) for t in (q, k, v)]
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out = pkg.kernels.dilution_attention(*leaves, dot_precision="bf16")
    out.backward(dout.to(DEV))
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert ("tc_forward_main" in names, "tc_forward_fused" in names) == (short, not short), names
    # the rows are independent: the first and the last one
    for r in (0, rows - 1):
        ref, *grads = O.dilution_backward(*(t[:, r:r + 1].bfloat16().float() for t in (q, k, v)), dout[:, r:r + 1])
        assert (out[:, r:r + 1].detach().cpu() - ref).abs().max().item() < 2e-2
        for t, g in zip(leaves, grads):
            assert rel_err(t.grad[:, r:r + 1].float().cpu(), g) < 3e-2
