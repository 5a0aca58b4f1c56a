"""Tensors with NaN and infinities on the tcgen05 kernels: the same outputs are NaN and infinite as on the exact fp32 path,
every other output keeps its value, and nothing that a value is may steer a warp: its lanes meet in warp-wide TMEM loads and in the release of
TMEM."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"
SEQ = 300
PATHS = [(torch.bfloat16, 64, "bf16"), (torch.bfloat16, 128, "bf16"), (torch.float32, 64, "tf32"), (torch.float32, 32, "tf32")]


def run(x, dtype, prec, training):
    """(out, gradients) of one call; no gradients from a forward-only one."""
    pkg = load_package()
    leaves = [t.to(DEV, dtype) for t in x]
    if not training:
        return pkg.dilution_attention_forward(*leaves, dot_precision=prec), ()
    leaves = [t.requires_grad_(True) for t in leaves]
    out = pkg.dilution_attention(*leaves, dot_precision=prec)
    return out.detach(), torch.autograd.grad(out, leaves, torch.full_like(out, 1e-2))


def same_as_exact(x, dtype, prec, training):
    """Outputs are NaN, infinite and finite where the exact path's are (same operands, fp32 products)."""
    out, grads = run(x, dtype, prec, training)
    ref, _ = run([t.to(dtype).float() for t in x], torch.float32, "ieee", False)
    assert torch.equal(out.isnan(), ref.isnan())
    assert torch.equal(out.isinf(), ref.isinf()) and torch.equal(out[out.isinf()], ref[ref.isinf()])
    ok = ref.isfinite()
    assert (out[ok] - ref[ok]).abs().max().item() < 2e-2
    return out, ref, grads


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("what", ["q", "k"])
@pytest.mark.parametrize("pos", [0, 34, 130, 258, SEQ - 2])
@pytest.mark.parametrize("dtype,d,prec", PATHS)
def test_a_nan_row_leaves_its_warp_whole(dtype, d, prec, pos, what, training):
    """A NaN query has no score to take a maximum of, at lanes of several warps and in the last, ragged tile."""
    x = list(make_inputs(1, 2, SEQ, d, 11))[:3]
    x["qk".index(what)][0, 1, pos, 3] = float("nan")
    out, _, grads = same_as_exact(x, dtype, prec, training)
    assert out[0, 1, pos].isnan().all() and out[0, 0].isfinite().all()
    for g in grads:
        assert g[0, 0].isfinite().all()
    # the next call on the same device
    run([t[:, :1] for t in x], dtype, prec, training)[0].isfinite().all().item()


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("what", ["q", "k", "v"])
@pytest.mark.parametrize("pos", [3, 128, 129, 130, 131, 259, SEQ - 1])
@pytest.mark.parametrize("dtype,d,prec", PATHS[1:])
def test_a_nan_comes_through_every_exponential(dtype, d, prec, pos, what, training):
    """Every fourth exponential of a row is a polynomial, at each position modulo four and in the last row.  (A masked
    share of 0 makes NaN of a NaN value: the rows in front of it in its tile, 64 rows of the exact path and 128 here, are
    left out.)"""
    x = list(make_inputs(1, 2, SEQ, d, 12))[:3]
    x["qkv".index(what)][0, 0, pos, 5] = float("nan")
    if what != "v":
        same_as_exact(x, dtype, prec, training)
        return
    out, _ = run(x, dtype, prec, training)
    x[2][0, 0, pos, 5] = 0.0
    clean, _ = run(x, dtype, prec, training)
    assert out[0, 0, pos:, 5].isnan().all()
    keep = torch.ones_like(out, dtype=torch.bool)
    keep[0, 0, pos // 128 * 128:, 5] = False
    assert torch.equal(out[keep], clean[keep])


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), 3.4e38, -3.4e38])
@pytest.mark.parametrize("pos", [4, 129, 130, 131, SEQ - 1])
@pytest.mark.parametrize("dtype,d,prec", PATHS[1:])
def test_a_score_of_minus_infinity_is_a_bid_of_zero(dtype, d, prec, pos, value):
    """A key's infinite feature against queries of the other sign: its scores are -inf, nobody bids for it and every output
    is finite.  3.4e38 is past the largest bf16 and rounds to an infinity there."""
    q, k, v, _ = make_inputs(1, 2, SEQ, d, 13)
    q[0, 0, :, 5] = -torch.copysign(q[0, 0, :, 5].abs() + 0.1, torch.tensor(value))
    k[0, 0, pos, 5] = value
    x = [q, k, v]
    for training in (False, True):
        out, ref, grads = same_as_exact(x, dtype, prec, training)
        assert ref.isfinite().all()
    _, exact = run([t.to(dtype).float() for t in x], torch.float32, "ieee", True)
    for name, g, r in zip(("dq", "dk", "dv"), grads, exact):
        ok = r.isfinite()
        if name == "dq":             # 0 * inf in the key's feature, for the rows of its 128-row tile too
            ok[0, 0, pos // 128 * 128:, 5] = False
        assert ((g.float() - r)[ok].norm() / r[ok].norm()).item() < 1e-2, name
    _, aux = load_package().dilution_attention_forward(*(t.to(DEV, dtype) for t in x), dot_precision=prec, return_aux=True)
    assert aux["committed_total"].isfinite().all()


@pytest.mark.parametrize("seq", [700, 768])
def test_a_key_that_nobody_bids_for_under_the_softplus_bid(seq):
    q, k, v, dout = make_inputs(1, 2, seq, 64, 15)
    q[0, 0, :, 5] = -(q[0, 0, :, 5].abs() + 0.1)
    k[0, 0, 131, 5] = float("inf")
    kb = load_package().kernels_bid
    got = []
    for prec in ("bf16", "tf32"):      # tf32 on the same tensors: the tile kernels
        leaves = [t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v)]
        out = kb.dilution_attention(*leaves, dot_precision=prec, bid="softplus")
        got.append((out.detach(), *(g.float() for g in torch.autograd.grad(out, leaves, dout.to(DEV)))))
    for name, a, b in zip(("out", "dq", "dk", "dv"), *got):
        ok = b.isfinite()
        if name == "dq":
            ok[0, 0, 128:, 5] = False
        assert ok.float().mean().item() > 0.98, name
        assert ((a - b)[ok].norm() / b[ok].norm()).item() < 1e-2, name


@pytest.mark.parametrize("what", ["q", "k"])
@pytest.mark.parametrize("dtype,d,prec", PATHS[1:])
def test_an_infinite_score_makes_its_rows_nan(dtype, d, prec, what):
    x = list(make_inputs(1, 2, SEQ, d, 14))[:3]
    x["qk".index(what)][0, 0, 131, 5] = float("inf")
    same_as_exact(x, dtype, prec, True)


def test_hi_and_lo_planes_of_values_that_are_not_finite():
    """hi + lo of every kind of value, and of its neighbours as if it were not there."""
    lib = load_package()._lib.load()
    clean = make_inputs(1, 1, 8, 32, 17)[0][0, 0]
    x = clean.clone()
    odd = [float("inf"), float("-inf"), float("nan"), 3.4e38, -3.4e38]
    for n, value in enumerate(odd):
        x[n, 6 + n] = value
    got = []
    for t in (x.to(DEV), clean.to(DEV)):
        planes = [torch.empty(8, 128, device=DEV, dtype=torch.bfloat16) for _ in range(3)]
        assert lib.dilution_split_operands(t.data_ptr(), t.data_ptr(), t.data_ptr(), 8, 32, *(p.data_ptr() for p in planes),
                                           torch.cuda.current_stream().cuda_stream) == 0
        got.append(planes[0].float().cpu())
    hi, lo = got[0][:, :64], got[0][:, 64:]
    assert (hi[0, 6], lo[0, 6]) == (1.0, float("inf")) and (hi[1, 7], lo[1, 7]) == (-1.0, float("-inf"))
    assert hi[2, 8].isnan() and lo[2, 8].isnan()
    for n, sign in ((3, 1), (4, -1)):
        assert hi[n, 6 + n] == sign * torch.finfo(torch.bfloat16).max
        assert abs((hi[n, 6 + n].double() + lo[n, 6 + n].double()).item() / x[n, 6 + n].item() - 1) < 2.0 ** -15
    for n in range(5):
        for p in got:
            p[n, [6 + n, 70 + n]] = 0.0
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("signs", [(1.0,), (-1.0,), (1.0, 1.0), (1.0, -1.0)])
@pytest.mark.parametrize("pos", [0, 63, 129, 131, SEQ - 1])
@pytest.mark.parametrize("path", PATHS[1:] + ["softplus"])
def test_infinite_values_make_infinite_outputs(path, pos, signs):
    """The rows that see an infinite value are infinite in its column, and NaN where they see both signs; shares multiplied as
    hi + lo would make NaN of all of them.  (Rows in front of it in its 128-row tile: 0 * inf, as above.)"""
    pkg = load_package()
    dtype, d, prec = (torch.bfloat16, 64, None) if path == "softplus" else path
    seq = 700 if path == "softplus" else SEQ

    def call(x, exact):
        if path == "softplus":       # tf32 on the same tensors: the tile kernels
            return pkg.kernels_bid.dilution_attention_forward(*(t.to(DEV, dtype) for t in x), bid="softplus",
                                                              dot_precision="tf32" if exact else "bf16")
        return run([t.to(dtype).float() for t in x], torch.float32, "ieee", False)[0] if exact else run(x, dtype, prec, True)[0]

    x = list(make_inputs(1, 2, seq, d, 16))[:3]
    clean = call(x, False)
    at = [pos, pos + 70][:len(signs)] if pos + 70 < seq else [pos - 70 * n for n in range(len(signs))][::-1]
    pos = at[0]
    for p, s in zip(at, signs):
        x[2][0, 1, p, 7] = s * float("inf")
    out, ref = call(x, False)[0, 1, :, 7].cpu(), call(x, True)[0, 1, :, 7].cpu()
    want = torch.zeros(seq)
    for p, s in zip(at, signs):
        want[p:] += s * float("inf")
    sees = [i for i in range(pos, seq) if all(i >= p or i < p // 128 * 128 for p in at)]      # no masked infinity in the tile
    for got in (out, ref):
        assert torch.equal(got[sees].nan_to_num(5.0, 1.0, -1.0), want[sees].nan_to_num(5.0, 1.0, -1.0))
    full = call(x, False)
    keep = torch.ones_like(full, dtype=torch.bool)
    keep[0, 1, pos // 128 * 128:, 7] = False
    assert torch.equal(full[keep], clean[keep])


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("what", ["q", "k"])
@pytest.mark.parametrize("pos", [3, 128, 129, 130, 131, 259, SEQ - 1])
def test_a_nan_comes_through_every_exponential_of_bf16_heads_of_64(pos, what, training):
    x = list(make_inputs(1, 2, SEQ, 64, 12))[:3]
    x["qk".index(what)][0, 0, pos, 5] = float("nan")
    same_as_exact(x, torch.bfloat16, "bf16", training)


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("what", ["q", "k"])
@pytest.mark.parametrize("pos", [1000, 1001, 1002, 1003])
def test_a_nan_in_a_sweep_of_512_keys(pos, what, training):
    """A NaN query makes every demand NaN that it bids for, a NaN key its own, and both every output from there on, in a call
    of 256 blocks of 512 keys or more."""
    rows, seq = 52, 2049
    x = [t.bfloat16().to(DEV) for t in make_inputs(1, rows, seq, 64, 18)[:3]]
    x["qk".index(what)][0, 1, pos, 5] = float("nan")
    pkg = load_package()
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out, aux = pkg.kernels.dilution_attention_forward(*x, dot_precision="bf16", return_aux=True, _training=training)
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert "tc_forward_fused" in names
    total = aux["committed_total"]
    assert out[0, 1, pos:].isnan().all() and out[0, 1, :pos].isfinite().all()
    assert total[0, 1, pos].isnan() and (what == "k" or total[0, 1, :pos].isnan().all())
    for other in (0, 2, rows - 1):
        assert out[0, other].isfinite().all() and total[0, other].isfinite().all()
