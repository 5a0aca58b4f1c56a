"""Row passes with an issuing warp (wide rows; narrow ones of 6144 tokens in 256 blocks of 256 queries): a row's results are the same
bits whatever the number of rows in the call and on both sides of the line between the kernels, and hold against 64 bits."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(rows, seq, d, std, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(rows + seq)
    q, k, v = (torch.randn(rows, seq, d, device=DEV, generator=g) for _ in range(3))
    return (q * std).to(dtype), k.to(dtype), v.to(dtype)


def _narrow(q, k, v):
    """Softmax attention, and row statistics with pk."""
    pkg = load_package()
    rows, seq = q.shape[:2]
    lib, L = pkg._lib.load(), pkg._lib
    rmax, rden, pk = (torch.empty(rows, seq, *s, device=DEV) for s in ((), (), (64,)))
    L.check(lib.dilution_rowstats_pk(q.data_ptr(), k.data_ptr(), L.BF16, L.PREC["bf16"], rows, seq, 64, 0.125, rmax.data_ptr(),
                                     rden.data_ptr(), pk.data_ptr(), torch.cuda.current_stream().cuda_stream), "rowstats_pk")
    return [pkg.softmax_attention_forward(q[None], k[None], v[None])[0], rmax, rden, pk]


def _wide(q, k, v):
    """Row statistics and pk of dilution_wide_forward."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    rows, seq, d = q.shape
    st = torch.cuda.current_stream().cuda_stream
    code, ops = L.BF16, (q, k, v)
    if q.dtype == torch.float32:
        code, ops = L.F32, tuple(torch.empty(rows, seq, 128, device=DEV, dtype=torch.bfloat16) for _ in range(3))
        L.check(lib.dilution_split_operands(*(x.data_ptr() for x in (q, k, v)), rows * seq, d, *(x.data_ptr() for x in ops), st), "split")
    rmax, rden, total, ssum, out, pk = (torch.empty(rows, seq, *s, device=DEV) for s in ((), (), (), (), (d,), (d,)))
    carry = torch.empty(rows, (seq + 31) // 32, seq, device=DEV)
    L.check(lib.dilution_wide_forward(*(x.data_ptr() for x in ops), code, rows, seq, d, d ** -0.5, 1e-9,
                                      *(x.data_ptr() for x in (rmax, rden, carry, total, out, ssum, pk)), st), "wide forward")
    return [rmax, rden, pk]


@pytest.mark.parametrize("std", [1.0, 24.0])
@pytest.mark.parametrize("rows,seq,few,d,dtype", [
    (128, 2048, 64, 64, torch.bfloat16), (100, 3001, 9, 64, torch.bfloat16), (11, 6200, 10, 64, torch.bfloat16), (37, 1000, 36, 128, torch.bfloat16),
    (148, 100, 5, 128, torch.bfloat16), (74, 300, 2, 64, torch.float32), (148, 65, 147, 32, torch.float32)])
def test_a_row_does_not_depend_on_how_many_there_are(rows, seq, few, d, dtype, std):
    x = _inputs(rows, seq, d, std, dtype)
    call = _narrow if (d, dtype) == (64, torch.bfloat16) else _wide
    for many, one in zip(call(*x), call(*(t[:few].contiguous() for t in x))):
        assert torch.equal(many[:few], one)


@pytest.mark.parametrize("what", [0, 1, 2])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("pos", [3, 70, 6143, 6199])
def test_values_that_are_not_finite(what, value, pos):
    """What such a value does is the same in a call of 264 blocks of 256 queries and in one of 240, bit for bit."""
    x = _inputs(11, 6200, 64, 1.0)
    x[what][1, pos, 5] = value
    for many, one in zip(_narrow(*x), _narrow(*(t[:10].contiguous() for t in x))):
        assert torch.equal(many[:10].isnan(), one.isnan()) and torch.equal(many[:10].nan_to_num(7.0), one.nan_to_num(7.0))
        assert many[0].isfinite().all() and many[2:].isfinite().all()


@pytest.mark.parametrize("std", [1.0, 24.0])
def test_both_sides_of_the_line(std):
    x = _inputs(11, 6144, 64, std)
    # (the reference exponents of a warp's 32 queries move together: the last warp has a row less)
    for at, under in zip(_narrow(*x), _narrow(*(t[:, :6143].contiguous() for t in x))):
        assert torch.equal(at[:, :6112], under[:, :6112])


@pytest.mark.parametrize("rows,q_off,tq", [(11, 0, 6145), (256, 6016, 128), (256, 6144, 13), (128, 6016, 257), (86, 5760, 513), (11, 128, 6050)])
@pytest.mark.parametrize("std", [1.0, 24.0])
def test_slices_of_queries_against_64_bits(rows, q_off, tq, std):
    """Queries [q_off, q_off + tq) of rows of 6300 keys."""
    pkg = load_package()
    lib, L = pkg._lib.load(), pkg._lib
    q, k, v = _inputs(rows, 6300, 64, std)
    q = q[:, q_off:q_off + tq].contiguous()
    out, (rmax, rden) = torch.empty_like(q), (torch.empty(rows, tq, device=DEV) for _ in range(2))
    L.check(lib.dilution_softmax_forward(*(x.data_ptr() for x in (q, k, v)), L.BF16, L.PREC["bf16"], rows, tq, 6300, q_off, 64, 0.125,
                                         rmax.data_ptr(), rden.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream),
            "softmax_forward")
    for row in (0, rows - 1):
        z = (q[row].double() @ k[row].double().T) / 8
        z = z.masked_fill(torch.ones_like(z, dtype=torch.bool).triu(1 + q_off), float("-inf"))
        p, lse = torch.softmax(z, -1), torch.logsumexp(z, -1)
        ref, size = p @ v[row].double(), p @ v[row].double().abs()
        # P~ and out have 8 bits, the sums are fp32
        assert ((out[row].double() - ref).abs() <= 2.0 ** -8 * 1.01 * size + 2.0 ** -8 * ref.abs() + 1e-6).all()
        got = (rmax[row].double() + torch.log2(rden[row].double())) * math.log(2)
        assert ((got - lse).abs() <= 2e-6 * lse.abs().clamp(min=1.0) + 2e-6).all()
