"""Row passes of many blocks: ragged lengths around the tiles, and a reference exponent that has to move, against 64 bits."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _exact(q, k, v, row):
    z = (q[0, row].double() @ k[0, row].double().T) / math.sqrt(64)
    z = z.masked_fill(torch.ones_like(z, dtype=torch.bool).triu(1), float("-inf"))
    return torch.softmax(z, -1), torch.logsumexp(z, -1)


# 1024 blocks of 256 queries and more in rows of 2048 tokens and more, one row less, and one token
@pytest.mark.parametrize("rows,seq", [(128, 2048), (127, 2048), (128, 2047), (114, 2049), (114, 2111), (114, 2177), (103, 2433)])
@pytest.mark.parametrize("std", [1.0, 24.0])
def test_row_pass_against_64_bits(rows, seq, std):
    pkg = load_package()
    g = torch.Generator(device=DEV).manual_seed(rows + seq)
    q, k, v = (torch.randn(1, rows, seq, 64, device=DEV, generator=g).bfloat16() for _ in range(3))
    q = (q.float() * std).bfloat16()                      # scores of deviation std: later tiles outgrow the first one's reference
    out = pkg.softmax_attention_forward(q, k, v)
    lib = pkg._lib.load()
    stats = torch.empty(2, rows, seq, device=DEV)
    pk = torch.empty(rows, seq, 64, device=DEV)
    stream = torch.cuda.current_stream().cuda_stream
    pkg._lib.check(lib.dilution_rowstats_pk(q.data_ptr(), k.data_ptr(), pkg._lib.BF16, pkg._lib.PREC["bf16"], rows, seq, 64, 0.125,
                                            stats[0].data_ptr(), stats[1].data_ptr(), pk.data_ptr(), stream), "rowstats_pk")
    for row in (0, rows // 2, rows - 1):
        p, lse = _exact(q, k, v, row)
        # P~ has 8 bits: a product's error is at most 2^-8 of sum p |b|, its fp32 sums' and the special-function unit's 1e-5 of it
        bound = 2.0 ** -8 * 1.01
        ref = p @ v[0, row].double()
        size = p @ v[0, row].double().abs()
        assert ((out[0, row].double() - ref).abs() <= bound * size + 2.0 ** -8 * ref.abs() + 1e-6).all()     # (and out is bf16)
        ref, size = 0.125 * (p @ k[0, row].double()), 0.125 * (p @ k[0, row].double().abs())
        assert ((pk[row].double() - ref).abs() <= bound * size + 1e-6).all()
        got = (stats[0, row].double() + torch.log2(stats[1, row].double())) * math.log(2)
        assert ((got - lse).abs() <= 2e-6 * lse.abs().clamp(min=1.0) + 2e-6).all()


# rows of 256 bytes: bf16 heads of 128, fp32 heads as hi + lo planes; 148 blocks of 256 queries and one less
@pytest.mark.parametrize("rows,seq", [(148, 100), (74, 257), (148, 129), (50, 700), (147, 100)])
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 128), (torch.float32, 64), (torch.float32, 32)])
@pytest.mark.parametrize("std", [1.0, 24.0])
def test_wide_row_pass_against_64_bits(rows, seq, dtype, d, std):
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    g = torch.Generator(device=DEV).manual_seed(rows + seq + d)
    q, k, v = (torch.randn(rows, seq, d, device=DEV, generator=g) for _ in range(3))
    q, k, v = (q * std).to(dtype), k.to(dtype), v.to(dtype)
    st = torch.cuda.current_stream().cuda_stream
    code, ops = L.BF16, (q, k, v)
    if dtype == torch.float32:
        code, ops = L.F32, tuple(torch.empty(rows, seq, 128, device=DEV, dtype=torch.bfloat16) for _ in range(3))
        L.check(lib.dilution_split_operands(*(x.data_ptr() for x in (q, k, v)), rows * seq, d, *(x.data_ptr() for x in ops), st), "split")
    f32 = dict(device=DEV, dtype=torch.float32)
    rmax, rden, total, ssum = (torch.empty(rows, seq, **f32) for _ in range(4))
    carry, out, pk = torch.empty(rows, (seq + 31) // 32, seq, **f32), torch.empty(rows, seq, d, **f32), torch.empty(rows, seq, d, **f32)
    scale = d ** -0.5
    L.check(lib.dilution_wide_forward(*(x.data_ptr() for x in ops), code, rows, seq, d, scale, 1e-9,
                                      *(x.data_ptr() for x in (rmax, rden, carry, total, out, ssum, pk)), st), "wide forward")
    for row in (0, rows - 1):
        z = (q[row].double() @ k[row].double().T) * scale
        size = (q[row].double().abs() @ k[row].double().abs().T) * scale
        z = z.masked_fill(torch.ones_like(z, dtype=torch.bool).triu(1), float("-inf"))
        p, lse = torch.softmax(z, -1), torch.logsumexp(z, -1)
        # operands keep 16 bits as pairs (exact in bf16), so a score is off by 2^-16 of the sum of its terms' sizes, and P~ by that and 2^-16
        off = (2.0 ** -16 * size).amax(-1) if dtype == torch.float32 else torch.zeros_like(lse)
        got = (rmax[row].double() + torch.log2(rden[row].double())) * math.log(2)
        assert ((got - lse).abs() <= off + 2e-6 * lse.abs().clamp(min=1.0) + 2e-6).all()
        ref, width = scale * (p @ k[row].double()), scale * (p @ k[row].double().abs())
        assert ((pk[row].double() - ref).abs() <= (2 * off[:, None] + 2.0 ** -14) * width + 1e-6).all()
