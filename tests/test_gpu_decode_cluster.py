"""A cached step of few keys in all runs as one launch of clusters: lengths at the edges of its warps, chunks and limits,
for both attentions, against 64-bit arithmetic on the same tensors; which form runs on either side of the limit; and
the two forms against each other on the same row.

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


def _step(pkg, q1, k1, v1, k, v, committed, length, pos_dev=False):
    """(out, demand, names of the kernels) of one step on copies of the cache."""
    cache = dict(k=k.clone(), v=v.clone(), committed=committed.clone(), len=length - 1)
    if pos_dev:
        cache["pos_dev"] = torch.tensor([length - 1], device=DEV, dtype=torch.int32)
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    y = pkg.dilution_decode_append_step(q1, k1, v1, cache)
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    return y, cache["committed"], names


def _cache(rows, cap, d, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    k, v = (torch.randn(1, rows, cap, d, device=DEV, generator=g).to(dtype) for _ in range(2))
    new = tuple(torch.randn(1, rows, 1, d, device=DEV, generator=g).to(dtype) for _ in range(3))
    return new, k, v, torch.rand(1, rows, cap, device=DEV, generator=g)


ONE, THREE = {"decode_step"}, {"decode_scores", "decode_sweep", "decode_finalize"}


# two CTAs per SM at one per 256 keys (at most eight), 1024 keys and 128 KB of either cache per CTA
@pytest.mark.parametrize("dtype,d,rows,length,want", [
    (torch.bfloat16, 64, 296, 256, ONE), (torch.bfloat16, 64, 297, 256, THREE), (torch.bfloat16, 64, 148, 512, ONE),
    (torch.bfloat16, 64, 149, 512, THREE), (torch.bfloat16, 64, 37, 8192, ONE), (torch.bfloat16, 64, 1, 8193, THREE),
    (torch.bfloat16, 128, 1, 4096, ONE), (torch.bfloat16, 128, 1, 4097, THREE), (torch.float32, 64, 1, 4097, THREE)])
def test_which_form_runs(dtype, d, rows, length, want):
    pkg = load_package()
    new, k, v, committed = _cache(rows, length + 2, d, dtype, 3)
    assert _step(pkg, *new, k, v, committed, length)[2] == want


@pytest.mark.parametrize("dtype,d", [(torch.float32, 64), (torch.bfloat16, 64), (torch.bfloat16, 128)])
@pytest.mark.parametrize("length", [1, 255, 513, 1500])
def test_both_forms_of_a_step_agree(dtype, d, length):
    """A row on its own and the same row among 300: one launch and three.  Partial sums over other chunks, 1e-5; a bf16 output
    is rounded once."""
    pkg = load_package()
    new, k, v, committed = _cache(1, length + 2, d, dtype, length)
    y1, c1, names1 = _step(pkg, *new, k, v, committed, length)
    many = [t.expand(1, 300, *t.shape[2:]).contiguous() for t in (*new, k, v, committed)]
    y3, c3, names3 = _step(pkg, *many, length)
    assert names1 == ONE and names3 == THREE
    scale = y1.float().abs().max().item()
    assert (y3[:, 299:].float() - y1.float()).abs().max().item() < (2.0 ** -7 if dtype == torch.bfloat16 else 1e-5) * scale
    assert (c3[:, 299:] - c1).abs().max().item() < 1e-5


@pytest.mark.parametrize("length", [1, 33, 700, 2999])
def test_length_on_the_device_below_capacity(length):
    """pos_dev: chunks follow the capacity, so most ranks of the cluster may be left without a key."""
    pkg = load_package()
    new, k, v, committed = _cache(3, 3000, 64, torch.bfloat16, length)
    y, c, names = _step(pkg, *new, k, v, committed, length, pos_dev=True)
    ref, rc, _ = _step(pkg, *new, k, v, committed, length)
    assert names == ONE
    assert (y.float() - ref.float()).abs().max().item() < 2.0 ** -7 * ref.float().abs().max().item()
    assert (c - rc).abs().max().item() < 1e-5
