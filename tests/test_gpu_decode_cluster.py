"""A cached step of few keys in all runs as one launch of clusters: lengths at the edges of its warps, chunks and limits,
for both attentions, against 64-bit arithmetic on the same tensors and against the three-launch step.

Bounds: fp32 sums of a few thousand terms, 1e-5 of the largest value; a bf16 output row is rounded once, 2^-8."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dilution", [True, False])
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 64), (torch.bfloat16, 128), (torch.float32, 16), (torch.float32, 64)])
@pytest.mark.parametrize("rows,length", [(3, 1), (3, 31), (3, 256), (3, 257), (2, 513), (37, 2048), (2, 2049), (38, 1792),
                                         (1, 4095), (5, 8192), (1, 8193)])
def test_step(dilution, dtype, d, rows, length):
    pkg = load_package()
    g = torch.Generator(device=DEV).manual_seed(length + d)
    cap = length + 3
    k, v = (torch.randn(1, rows, cap, d, device=DEV, generator=g).to(dtype) for _ in range(2))
    q1, k1, v1 = (torch.randn(1, rows, 1, d, device=DEV, generator=g).to(dtype) for _ in range(3))
    committed = torch.rand(1, rows, cap, device=DEV, generator=g)
    cache = dict(k=k.clone(), v=v.clone(), len=length - 1)
    if dilution:
        cache["committed"] = committed.clone()
    step = pkg.dilution_decode_append_step if dilution else pkg.softmax_decode_append_step
    y = step(q1, k1, v1, cache)
    kk = torch.cat([k[:, :, :length - 1], k1], 2).double()
    vv = torch.cat([v[:, :, :length - 1], v1], 2).double()
    p = torch.softmax((q1.double() @ kk.transpose(-1, -2)) / math.sqrt(d), -1)[:, :, 0]
    share = p
    if dilution:
        c = committed[:, :, :length].double()
        c[:, :, -1] = 0.0
        share = p / (c + p + 1e-9)
        assert (cache["committed"][:, :, :length].double() - (c + p)).abs().max().item() < 1e-5
        assert torch.equal(cache["committed"][:, :, length:], committed[:, :, length:])
    ref = torch.einsum("bhj,bhjd->bhd", share, vv) / (share.sum(-1, keepdim=True) + (1e-9 if dilution else 0.0))
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5) * ref.abs().max().item()
    assert cache["len"] == length and (y[:, :, 0].double() - ref).abs().max().item() < tol
    for new, old, row in ((cache["k"], k, k1), (cache["v"], v, v1)):
        assert torch.equal(new[:, :, length - 1:length], row)
        assert torch.equal(new[:, :, :length - 1], old[:, :, :length - 1]) and torch.equal(new[:, :, length:], old[:, :, length:])
