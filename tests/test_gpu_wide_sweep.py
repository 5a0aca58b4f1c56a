"""The key-stationary sweep in blocks of 512 keys (256 of them or more) at the edges of its blocks, warpgroups and half tiles,
with checkpoints every 32 rows (a training forward) and every 64 (a prompt), against the two passes and, in the first and last
row, the oracle; and the choice between the two at its edges."""

from __future__ import annotations

import pytest
import torch

from conftest import load_package, make_inputs, rel_err
from oracle import dilution_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _forward(K, x, training, fused):
    saved, K.TC_FUSED_FORWARD = K.TC_FUSED_FORWARD, fused
    try:
        out, aux = K.dilution_attention_forward(*x, dot_precision="bf16", return_aux=True, _training=training)
    finally:
        K.TC_FUSED_FORWARD = saved
    return out, aux


@pytest.mark.parametrize("training", [True, False])
@pytest.mark.parametrize("rows,seq", [(52, 2049), (52, 2111), (52, 2175), (52, 2176), (52, 2177), (52, 2305), (43, 2561),
                                      (43, 3072), (37, 3137)])
def test_sweep_of_512_keys(rows, seq, training):
    pkg = load_package()
    K = pkg.kernels
    x = [t.bfloat16().to(DEV) for t in make_inputs(1, rows, seq, 64, 60 + seq, scales=(1.0, 1.0, 1.0, 1.0))[:3]]
    pkg._lib.profile(True)
    pkg._lib.profile_collect()
    out, aux = _forward(K, x, training, True)
    names = set(pkg._lib.profile_collect())
    pkg._lib.profile(False)
    assert "tc_forward_fused" in names and "tc_forward_main" not in names, names
    ref_out, ref = _forward(K, x, training, False)
    assert aux["bwd_block_m"] == ref["bwd_block_m"] == (32 if training else 64)
    assert (out - ref_out).abs().max().item() < 1e-2                     # both round their shares to bf16
    assert rel_err(aux["committed_total"], ref["committed_total"]) < 1e-4
    assert rel_err(aux["ssum"], ref["ssum"]) < 1e-2
    step = aux["bwd_block_m"]
    scale = max(1.0, ref["carry"][:, -1].abs().max().item())
    for rb in range(aux["carry"].shape[1]):
        end = min((rb + 1) * step, seq)
        assert (aux["carry"][:, rb, :end] - ref["carry"][:, rb, :end]).abs().max().item() < 1e-4 * scale, rb
    for r in (0, rows - 1):
        want = O.dilution_chunked(*(t[:, r:r + 1].float().cpu() for t in x), chunk=512)
        assert (out[:, r:r + 1].cpu() - want).abs().max().item() < 2e-2


def _route(rows, seq, training):
    pkg = load_package()
    return pkg.kernels._takes_sweep(pkg._lib.BF16, pkg._lib.PREC["bf16"], rows, seq, seq, 64, 32 if training else 64)


@pytest.mark.parametrize("rows,seq,training,sweep", [(52, 2048, False, False), (52, 2049, False, True), (51, 2049, False, True),
                                                     (1, 2049, False, True), (10, 2559, True, True), (10, 2560, True, True),
                                                     (12, 2304, True, True), (32, 4096, True, True), (31, 4096, True, True),
                                                     (12, 1536, True, True), (13, 1536, True, False), (16, 1600, True, True)])
def test_route(rows, seq, training, sweep):
    assert _route(rows, seq, training) is sweep


def test_deterministic_algorithms_keep_the_two_passes():
    pkg = load_package()
    x = [t.bfloat16().to(DEV) for t in make_inputs(1, 52, 2111, 64, 71, scales=(1.0, 1.0, 1.0, 1.0))[:3]]
    sweep = pkg.kernels.dilution_attention_forward(*x, dot_precision="bf16")
    torch.use_deterministic_algorithms(True)
    try:
        pkg._lib.profile(True)
        pkg._lib.profile_collect()
        got = [pkg.kernels.dilution_attention_forward(*x, dot_precision="bf16", return_aux=True) for _ in range(3)]
        names = set(pkg._lib.profile_collect())
        pkg._lib.profile(False)
        assert pkg.kernels._takes_sweep(pkg._lib.BF16, pkg._lib.PREC["bf16"], 52, 2111, 2111, 64, 32)      # a training forward
    finally:
        torch.use_deterministic_algorithms(False)
    assert "tc_forward_main" in names and "tc_forward_fused" not in names, names
    for out, aux in got[1:]:
        assert torch.equal(out, got[0][0]) and torch.equal(aux["committed_total"], got[0][1]["committed_total"])
    assert (sweep - got[0][0]).abs().max().item() < 1e-2                  # both round their shares to bf16


@pytest.mark.parametrize("rows,seq,sweep", [(11, 2304, True), (12, 2304, False), (10, 2559, True), (10, 2560, False), (11, 2559, False),
                                            (51, 2559, False), (52, 2559, True), (32, 4096, True), (31, 4096, False)])
def test_route_under_deterministic_algorithms(rows, seq, sweep):
    """Training calls keep the two passes, whose outputs repeat, beyond 100 blocks of 256 keys or 2559 tokens and up to 256 blocks of 512;
    calls that no backward follows always do."""
    torch.use_deterministic_algorithms(True)
    try:
        assert _route(rows, seq, True) is sweep and _route(rows, seq, False) is False
    finally:
        torch.use_deterministic_algorithms(False)
