"""Gradient parity of the autograd op against autograd through the reference
(stored goldens) and the CPU oracle.  Mirrors tests/test_kernels.py:109-202."""

from __future__ import annotations

import pytest
import torch

from conftest import golden, load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("seq", [8, 64, 257, 1024, 2049])
def test_backward_matches_oracle_autograd_fp32(kernels, seq):
    q, k, v, dout = make_inputs(2, 4, seq, 64, seq)
    _, rdq, rdk, rdv = O.dilution_backward(q, k, v, dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    kernels.dilution_attention(qs, ks, vs, dot_precision="ieee").backward(dout.to(DEV))
    for name, ref, got in (("dq", rdq, qs.grad), ("dk", rdk, ks.grad), ("dv", rdv, vs.grad)):
        err = rel_err(got.cpu(), ref)
        assert err < 2e-3, f"{name} {err}"            # the reference's bound
        assert err < 1e-4, f"{name} {err}"            # fp32 kernels: 1e-4 relative


@pytest.mark.parametrize("t", [1, 8, 65, 257])
def test_backward_small_goldens(kernels, t):
    g = golden("small_cases.npz")
    c = {k[len(f"t{t}_"):]: torch.from_numpy(g[k]) for k in g.files if k.startswith(f"t{t}_")}
    qs, ks, vs = (c[n].to(DEV).requires_grad_(True) for n in "qkv")
    kernels.dilution_attention(qs, ks, vs, dot_precision="ieee").backward(c["dout"].to(DEV))
    for name, got in (("dq", qs.grad), ("dk", ks.grad), ("dv", vs.grad)):
        assert rel_err(got.cpu(), c[name]) < 1e-4, name


# "ieee": fp32 FMAs, 1e-4 of the oracle.  "tf32": tensor-core products on operands rounded to
# 10 mantissa bits with fp32 accumulation (the reference's own meaning of the mode,
# kernels.py:318-325), within 5e-3 of the fp32 oracle.
@pytest.mark.parametrize("prec,tol", [("ieee", 1e-4), ("tf32", 5e-3)])
@pytest.mark.parametrize("head_dim", [16, 32, 128])
def test_backward_other_head_dims(kernels, head_dim, prec, tol):
    q, k, v, dout = make_inputs(1, 2, 130, head_dim, 500 + head_dim)
    ref, rdq, rdk, rdv = O.dilution_backward(q, k, v, dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision=prec)
    out.backward(dout.to(DEV))
    assert rel_err(out.detach().cpu(), ref) < tol
    for name, ref, got in (("dq", rdq, qs.grad), ("dk", rdk, ks.grad), ("dv", rdv, vs.grad)):
        assert rel_err(got.cpu(), ref) < tol, name


@pytest.mark.parametrize("seq", [64, 257, 1100])
def test_tf32_products_head_dim_64(kernels, seq):
    q, k, v, dout = make_inputs(2, 3, seq, 64, 900 + seq)
    ref, rdq, rdk, rdv = O.dilution_backward(q, k, v, dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision="tf32")
    out.backward(dout.to(DEV))
    assert rel_err(out.detach().cpu(), ref) < 5e-3
    for name, ref, got in (("dq", rdq, qs.grad), ("dk", rdk, ks.grad), ("dv", rdv, vs.grad)):
        assert rel_err(got.cpu(), ref) < 5e-3, name


@pytest.mark.parametrize("head_dim", [32, 128])
def test_bf16_tensors_other_head_dims(kernels, head_dim):
    """bf16 tensors whose head size the tcgen05 kernels do not take: tile kernels with
    tensor-core products, against the oracle on the same bf16-rounded inputs."""
    q, k, v, dout = make_inputs(1, 3, 300, head_dim, 70 + head_dim, scales=(0.5, 0.5, 1.0, 1.0))
    qb, kb, vb = (x.bfloat16() for x in (q, k, v))
    ref, rdq, rdk, rdv = O.dilution_backward(qb.float(), kb.float(), vb.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (qb, kb, vb))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
    out.backward(dout.to(DEV).bfloat16())
    assert (out.detach().float().cpu() - ref).abs().max().item() < 2e-2
    for name, ref, got in (("dq", rdq, qs.grad), ("dk", rdk, ks.grad), ("dv", rdv, vs.grad)):
        assert rel_err(got.float().cpu(), ref) < 2e-2, name


def test_backward_finite_grads(kernels):
    q, k, v, _ = make_inputs(1, 2, 96, 64, 1)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    kernels.dilution_attention(qs, ks, vs, dot_precision="ieee").sum().backward()
    for t in (qs, ks, vs):
        assert t.grad is not None and torch.isfinite(t.grad).all()


@pytest.mark.parametrize("seq", [257, 1100])
def test_bf16_mode_forward_and_backward(kernels, seq):
    """dot_precision="bf16": bf16 tensor-core operands, fp32 cumsum/share maths."""
    q, k, v, dout = make_inputs(2, 4, seq, 64, 5)
    ref, rdq, rdk, rdv = O.dilution_backward(q, k, v, dout)
    qb, kb, vb = (x.to(DEV).bfloat16().requires_grad_(True) for x in (q, k, v))
    out = kernels.dilution_attention(qb, kb, vb, dot_precision="bf16")
    out.backward(dout.to(DEV).bfloat16())
    assert torch.isfinite(out).all() and out.dtype == torch.float32
    assert (out.detach().cpu() - ref).abs().max().item() < 5e-2
    for name, gr, t in (("dq", rdq, qb), ("dk", rdk, kb), ("dv", rdv, vb)):
        assert t.grad.dtype == torch.bfloat16
        err = rel_err(t.grad.float().cpu(), gr)
        assert torch.isfinite(t.grad).all() and err < 1e-1, f"{name} {err}"   # reference bound
    # same bf16-rounded inputs: 2e-2 max-abs on outputs and gradients
    r2 = O.dilution_backward(qb.detach().float().cpu(), kb.detach().float().cpu(), vb.detach().float().cpu(),
                             dout.bfloat16().float())
    assert (out.detach().cpu() - r2[0]).abs().max().item() < 2e-2
    for name, gr, t in (("dq", r2[1], qb), ("dk", r2[2], kb), ("dv", r2[3], vb)):
        assert (t.grad.float().cpu() - gr).abs().max().item() < 2e-2, name
        assert rel_err(t.grad.float().cpu(), gr) < 3e-2, name


def test_training_shape_inputs_bf16_small_t(kernels):
    """The benchmark's value distribution (q,k ~ 0.5 N, dout ~ 1e-2 N) at T=2048."""
    q, k, v, dout = make_inputs(1, 2, 2048, 64, 1339, scales=(0.5, 0.5, 1.0, 1e-2))
    qb, kb, vb = (x.bfloat16() for x in (q, k, v))
    ref = O.dilution_backward(qb.float(), kb.float(), vb.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (qb, kb, vb))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
    out.backward(dout.to(DEV))
    assert (out.detach().cpu() - ref[0]).abs().max().item() < 2e-2
    for name, gr, t in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert (t.grad.float().cpu() - gr).abs().max().item() < 2e-2, name
        assert rel_err(t.grad.float().cpu(), gr) < 5e-2, name


def test_bf16_training_step_runs_on_the_tensor_core_kernels(pkg, kernels):
    """Forward and backward of the bf16 op launch tcgen05 kernels only (plus the
    small elementwise pre/post kernels): no fp32-FMA kernel on the training path."""
    q, k, v, dout = make_inputs(1, 2, 900, 64, 77, scales=(0.5, 0.5, 1.0, 1e-2))
    qs, ks, vs = (x.bfloat16().to(DEV).requires_grad_(True) for x in (q, k, v))
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    kernels.dilution_attention(qs, ks, vs, dot_precision="bf16").backward(dout.to(DEV))
    torch.cuda.synchronize()
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    # passes 2 and 3: one key-stationary sweep, or the column-sum pass plus the main pass
    fwd = {"tc_forward_fused", "tc_normalize_out"} if kernels.TC_FUSED_FORWARD else {"tc_colsum_scan", "tc_forward_main"}
    if kernels.TC_SAVE_PK:      # pass 1 saves pk; the correction pass has only its key half left
        want = {"tc_rowstats_pk", "tc_backward_prep", "tc_backward_main", "tc_backward_key_correction",
                "tc_dq_from_pk"} | fwd
    else:
        want = {"tc_rowstats", "tc_backward_prep", "tc_backward_main", "tc_backward_correction", "tc_cast_dq"} | fwd
    assert names == want, names
    ref = O.dilution_backward(qs.detach().float().cpu(), ks.detach().float().cpu(), vs.detach().float().cpu(), dout)
    for name, gr, t in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert rel_err(t.grad.float().cpu(), gr) < 3e-2, name


def test_host_buffer_entry_point_matches_device_op(kernels):
    """dilution_attention_host (pinned host tensors in and out, slabs pipelined over
    streams) returns what the device op returns."""
    q, k, v, dout = make_inputs(2, 3, 300, 64, 901, scales=(0.5, 0.5, 1.0, 1e-2))
    qb, kb, vb = (x.bfloat16().pin_memory() for x in (q, k, v))
    dout = dout.pin_memory()
    out, dq, dk, dv = kernels.dilution_attention_host(qb, kb, vb, dout, dot_precision="bf16", slabs=4)
    torch.cuda.synchronize()
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (qb, kb, vb))
    ref = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
    ref.backward(dout.to(DEV))
    assert torch.equal(out, ref.detach().cpu())
    assert torch.equal(dv, vs.grad.cpu())
    # dq and ghat (hence dk) are accumulated across key blocks with floating-point reductions
    # whose order varies between runs
    assert rel_err(dq.float(), qs.grad.float().cpu()) < 2e-2
    assert rel_err(dk.float(), ks.grad.float().cpu()) < 2e-3
    fwd_only = kernels.dilution_attention_host(qb, kb, vb, dot_precision="bf16", slabs=3)
    torch.cuda.synchronize()
    # the forward-only call takes its row statistics from the plain row pass, the training call
    # from the row pass that also saves pk: same values up to the last bits
    assert (fwd_only - out).abs().max().item() < 1e-3


def test_backward_size_independent_properties_at_16k(kernels):
    """T=16384, one (b,h) row, bf16, tensor-core kernels: identities of the true gradient that
    need no T^2 oracle.
    (a) the scores depend on q and k only through q.k, so <q, dq> == <k, dk>;
    (b) out is linear in v (out = A v, dv = A^T dout), so <v, dv> == <out, dout>;
    (c) the gradients are linear in dout."""
    t, d = 16384, 64
    q, k, v, dout = make_inputs(1, 1, t, d, 21, scales=(0.5, 0.5, 1.0, 1e-2))
    _, _, _, dout2 = make_inputs(1, 1, t, d, 22, scales=(0.5, 0.5, 1.0, 1e-2))

    def run(g):
        qs, ks, vs = (x.bfloat16().to(DEV).requires_grad_(True) for x in (q, k, v))
        out = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
        out.backward(g.to(DEV))
        return out.detach(), qs, ks, vs

    out, qs, ks, vs = run(dout)
    dq, dk, dv = (x.grad.double() for x in (qs, ks, vs))
    assert all(torch.isfinite(x).all() for x in (dq, dk, dv))
    qdq = (qs.detach().double() * dq).sum().item()
    kdk = (ks.detach().double() * dk).sum().item()
    scale_qk = (qs.detach().double() * dq).abs().sum().item()
    assert abs(qdq - kdk) < 2e-3 * scale_qk, (qdq, kdk, scale_qk)
    vdv = (vs.detach().double() * dv).sum().item()
    odo = (out.double() * dout.to(DEV).double()).sum().item()
    scale_v = (out.double() * dout.to(DEV).double()).abs().sum().item()
    assert abs(vdv - odo) < 2e-3 * scale_v, (vdv, odo, scale_v)
    _, q2, k2, v2 = run(dout2)
    _, q3, k3, v3 = run(dout + dout2)
    for name, a, b, c in (("dq", qs, q2, q3), ("dk", ks, k2, k3), ("dv", vs, v2, v3)):
        s = a.grad.float() + b.grad.float()
        assert rel_err(c.grad.float().cpu(), s.cpu()) < 2e-2, name


@pytest.mark.parametrize("seq", [1, 2, 63, 64, 65, 127, 128, 129, 192, 193, 320])
def test_bf16_tensor_path_backward_ragged_lengths(kernels, seq):
    """Lengths around the 64-row checkpoint and 128-row tile boundaries (half-steps that are
    partly or wholly past the end, a single tile, one row) on the tensor-core kernels."""
    q, k, v, dout = make_inputs(1, 3, seq, 64, 300 + seq, scales=(0.5, 0.5, 1.0, 1e-1))
    qb, kb, vb = (x.bfloat16() for x in (q, k, v))
    ref = O.dilution_backward(qb.float(), kb.float(), vb.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (qb, kb, vb))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
    out.backward(dout.to(DEV))
    assert (out.detach().cpu() - ref[0]).abs().max().item() < 2e-2
    for name, gr, t in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert torch.isfinite(t.grad).all(), name
        assert (t.grad.float().cpu() - gr).abs().max().item() < 2e-2, name


@pytest.mark.parametrize("scale", [2.0, 4.0, 8.0])
def test_bf16_backward_peaked_attention(kernels, scale):
    """Scores with a standard deviation of 4, 16 and 64: softmax rows close to one-hot, keys whose
    first bids are tiny.  The demand must be accumulated forwards from its checkpoints and the
    suffix of dk_share backwards; either sum taken in the other direction loses these cases."""
    q, k, v, dout = make_inputs(1, 2, 1024, 64, 5, scales=(scale, scale, 1.0, 1e-1))
    qb, kb, vb = (x.bfloat16() for x in (q, k, v))
    ref = O.dilution_backward(qb.float(), kb.float(), vb.float(), dout)
    qs, ks, vs = (x.to(DEV).requires_grad_(True) for x in (qb, kb, vb))
    out = kernels.dilution_attention(qs, ks, vs, dot_precision="bf16")
    out.backward(dout.to(DEV))
    assert rel_err(out.detach().cpu(), ref[0]) < 1e-2
    for name, gr, t in (("dq", ref[1], qs), ("dk", ref[2], ks), ("dv", ref[3], vs)):
        assert torch.isfinite(t.grad).all(), name
        assert rel_err(t.grad.float().cpu(), gr) < 3e-2, name


@pytest.mark.parametrize("dtype,d,prec", [(torch.bfloat16, 64, "bf16"), (torch.bfloat16, 128, "bf16"),
                                          (torch.float32, 64, "tf32"), (torch.float32, 32, "tf32"),
                                          (torch.float32, 64, "ieee")])
@pytest.mark.parametrize("bid", ["softmax", "sigmoid", "softplus"])
def test_saved_tensor_hooks_that_round(kernels, bid, dtype, d, prec):
    """A hook that keeps 12 bits of the mantissa of what is saved as fp32 costs about that much in the gradients: nothing but
    fp32 values may be saved as fp32.  Bound: 2^-12 on the demands, 1/(row sums), log-sum-exps of up to 16 (2^-8 of a bid) and pk
    of sums that cancel to a tenth."""
    def rounding(x):
        return (x.view(torch.int32) & ~0x7FF).view(torch.float32) if x.dtype == torch.float32 else x

    pkg = load_package()
    q, k, v, dout = (x.to(DEV) for x in make_inputs(1, 2, 200, d, 77))
    leaves = [x.to(dtype).requires_grad_(True) for x in (q, k, v)]

    def grads():
        if bid == "softmax":
            out = kernels.dilution_attention(*leaves, dot_precision=prec)
        else:
            out = pkg.kernels_bid.dilution_attention(*leaves, dot_precision=prec, bid=bid)
        return torch.autograd.grad(out, leaves, dout)

    plain = grads()
    with torch.autograd.graph.saved_tensors_hooks(rounding, lambda x: x):
        rounded = grads()
    for name, a, b in zip(("dq", "dk", "dv"), rounded, plain):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 4e-2, name
