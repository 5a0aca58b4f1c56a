"""Row passes of many blocks: pairs of query tiles with an issuing warp.  The route at its edge, ragged lengths around the tiles, and a
reference exponent that has to move, against 64 bits."""

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


# rows x pairs of tiles: 512 of them and more; one less takes the kernel of single tiles
@pytest.mark.parametrize("rows,seq", [(512, 1), (512, 64), (512, 127), (512, 129), (256, 257), (171, 513), (128, 1000), (511, 200)])
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
