"""The demand that a long prompt leaves, key by key against 64 bits: keys whose bids are large early and small later, keys that get
the same bid from every query, and ordinary ones.

Bound: a bid is 2^(s - l) with s and l below 32 in size, each rounded once (2^-20 of a log2, 6.6e-7 of a bid), an exponential of
2.4e-7 and a log-sum-exp out of polynomials of 2.7e-6; the sum itself, of thousands of bids, may add nothing to that."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
DEV = "cuda"
BOUND = 2 * 6.6e-7 + 2.4e-7 + 2.7e-6


def _total(q, k):
    """Column sums of the causal softmax of one (seq, 64) row in 64 bits."""
    t = q.shape[0]
    kd, total = k.double(), torch.zeros(t, device=DEV, dtype=torch.float64)
    for a in range(0, t, 1024):
        b = min(t, a + 1024)
        s = q[a:b].double() @ kd[:b].T / 8.0
        s.masked_fill_(torch.arange(b, device=DEV)[None, :] > torch.arange(a, b, device=DEV)[:, None], -math.inf)
        total[:b] += torch.softmax(s, -1).sum(0)
    return total


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("kind", ["ordinary", "peaked", "sink", "constant"])
@pytest.mark.parametrize("rows,seq", [(2, 65536), (52, 2111)])
def test_demand_of_a_sweep(rows, seq, kind, training):
    if training and seq > 4096:
        rows, seq = 8, 16384                 # (checkpoints every 32 rows: 9 GB at 65536)
    g = torch.Generator(device=DEV).manual_seed(41)
    q, k, v = (torch.randn(1, rows, seq, 64, device=DEV, generator=g) for _ in range(3))
    if kind == "peaked":
        q *= 2.0
    elif kind in ("sink", "constant"):       # feature 0 is key 0's alone
        q *= 0.3
        k[..., 0] = 0.0
        k[:, :, 0] = 0.0
        k[:, :, 0, 0] = 8.0
        if kind == "sink":                   # a bid of about 0.9 from the first half, of about 1e-3 from the second
            q[..., 0] = 13.0
            q[:, :, seq // 2:, 0] = 4.0
        else:                                # about 0.3 from everybody
            q[..., 0] = (0.43 * torch.arange(1, seq + 1, device=DEV)).log()
    q, k, v = (x.bfloat16() for x in (q, k, v))
    pkg = load_package()
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    _, aux = pkg.kernels.dilution_attention_forward(q, k, v, dot_precision="bf16", return_aux=True, _training=training)
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert "tc_forward_fused" in names
    for r in (0, rows - 1):
        ref = _total(q[0, r], k[0, r])
        err = ((aux["committed_total"][0, r].double() - ref) / ref).abs()
        assert err.max().item() < BOUND, (kind, err.argmax().item(), err.max().item())
