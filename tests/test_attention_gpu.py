# SPDX-License-Identifier: Apache-2.0
"""tcgen05 causal attention forward kernel against fp32 masked-softmax attention."""
import math

import pytest
import torch

import core_scheduler_b200 as cs
from core_scheduler_b200 import ops
from helpers import attention_reference

C = cs._C
pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 3), (2, 1024, 4), (1, 384, 2)])
def test_forward_matches_reference(B, T, H):
    D = 64
    torch.manual_seed(B * 1000 + T + H)
    qkv = torch.randn(B, T, 3 * H * D, device="cuda").to(BF)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, 1.0 / math.sqrt(D))
    torch.cuda.synchronize()
    assert rc == 0
    assert C.attention_status()[0] == 0
    q, k, v = qkv.float().view(B, T, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v).reshape(B, T, H * D)
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)
    s = torch.einsum("bthd,bshd->bhts", q, k) / math.sqrt(D)
    mask = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
    ref_lse = torch.logsumexp(s.masked_fill(~mask, float("-inf")), dim=-1)
    assert torch.allclose(lse, ref_lse, atol=2e-2, rtol=1e-3)


def test_unsupported_shapes_are_declined():
    qkv = torch.randn(1, 100, 3 * 2 * 64, device="cuda").to(BF)  # T not a multiple of 128
    rc, _, _ = C.attention_forward_tcgen05(qkv, 2, 0.125)
    assert rc == -1
    qkv = torch.randn(1, 128, 3 * 2 * 32, device="cuda").to(BF)  # head dimension 32
    rc, _, _ = C.attention_forward_tcgen05(qkv, 2, 0.125)
    assert rc == -1


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 3), (1, 1024, 2), (1, 384, 2)])
def test_backward_matches_reference(B, T, H):
    """dQ, dK, dV written into the packed layout equal autograd through fp32 masked-softmax attention."""
    D = 64
    torch.manual_seed(7 * B + T + H)
    qkv = torch.randn(B, T, 3 * H * D, device="cuda").to(BF)
    dout = torch.randn(B, T, H * D, device="cuda").to(BF)
    scale = 1.0 / math.sqrt(D)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, scale)
    assert rc == 0
    dqkv, delta = C.attention_backward_tcgen05(qkv, out, dout, lse, H, scale)
    torch.cuda.synchronize()
    assert C.attention_status()[0] == 0
    qr = qkv.float().requires_grad_(True)
    q, k, v = qr.view(B, T, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v).reshape(B, T, H * D)
    ref.backward(dout.float())
    ref_delta = (ref.detach() * dout.float()).view(B, T, H, D).sum(-1).permute(0, 2, 1)
    assert torch.allclose(delta, ref_delta, atol=5e-2, rtol=2e-2)
    got, want = dqkv.float().view(B, T, 3, H, D), qr.grad.view(B, T, 3, H, D)
    for i, name in enumerate(("dq", "dk", "dv")):
        err = (got[:, :, i] - want[:, :, i]).abs().max().item()
        ref_mag = want[:, :, i].abs().max().item()
        assert err <= 3e-2 * max(1.0, ref_mag), (name, err, ref_mag)


def test_backward_through_the_op_uses_own_kernels(gpu_scheduler, monkeypatch):
    """With the tcgen05 engine selected, forward_packed/backward_packed run this library's kernels end to end."""
    monkeypatch.setenv("CS_ATTENTION_ENGINE", "tcgen05")
    s = gpu_scheduler
    B, T, H, D = 2, 256, 4, 64
    qkv = torch.randn(B, T, 3 * H * D, device="cuda").to(BF)
    do = torch.randn(B, T, H * D, device="cuda").to(BF)
    st = C.attention_init(s, is_causal=True)
    before = C.kernel_launch_count()
    out = C.attention_forward_packed(s, st, cs.from_torch(qkv), H)
    dqkv = C.attention_backward_packed(s, st, cs.from_torch(do))
    s.synchronize()
    assert C.kernel_launch_count() - before == 4  # 1 forward + 3 backward launches, no library kernel
    qr = qkv.float().requires_grad_(True)
    q, k, v = qr.view(B, T, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v).reshape(B, T, H * D)
    ref.backward(do.float())
    assert torch.allclose(out.raw().float(), ref, atol=2e-2, rtol=2e-2)
    assert (dqkv.raw().float() - qr.grad).abs().max().item() < 5e-2


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 3), (1, 512, 2)])
def test_non_causal_forward_and_backward_match_reference(B, T, H):
    """The same kernels without the mask: every query attends to every key."""
    D = 64
    torch.manual_seed(11 * B + T + H)
    qkv = torch.randn(B, T, 3 * H * D, device="cuda").to(BF)
    dout = torch.randn(B, T, H * D, device="cuda").to(BF)
    scale = 1.0 / math.sqrt(D)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, scale, causal=False)
    assert rc == 0
    dqkv, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, scale, causal=False)
    torch.cuda.synchronize()
    assert C.attention_status()[0] == 0
    qr = qkv.float().requires_grad_(True)
    q, k, v = qr.view(B, T, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v, causal=False).reshape(B, T, H * D)
    ref.backward(dout.float())
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)
    s = torch.einsum("bthd,bshd->bhts", q, k) * scale
    assert torch.allclose(lse, torch.logsumexp(s, dim=-1), atol=2e-2, rtol=1e-3)
    got, want = dqkv.float().view(B, T, 3, H, D), qr.grad.view(B, T, 3, H, D)
    for i, name in enumerate(("dq", "dk", "dv")):
        err = (got[:, :, i] - want[:, :, i]).abs().max().item()
        assert err <= 3e-2 * max(1.0, want[:, :, i].abs().max().item()), (name, err)


def test_non_causal_attention_through_the_op_stays_on_own_kernels(gpu_scheduler):
    s = gpu_scheduler
    B, T, H, D = 2, 256, 2, 64
    qkv = torch.randn(B, T, 3 * H * D, device="cuda").to(BF)
    st = C.attention_init(s, is_causal=False)
    fallbacks = C.library_fallbacks()
    before = C.kernel_launch_count()
    out = C.attention_forward_packed(s, st, cs.from_torch(qkv), H)
    s.synchronize()
    assert C.kernel_launch_count() - before == 1 and C.library_fallbacks() == fallbacks
    q, k, v = qkv.float().view(B, T, 3, H, D).unbind(2)
    assert torch.allclose(out.raw().float(), attention_reference(q, k, v, causal=False).reshape(B, T, H * D), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,T,H", [(5, 384, 13), (2, 1024, 12), (1, 2176, 9), (149, 128, 1)])
def test_blocks_dealt_to_persistent_ctas(B, T, H, causal):
    """More 128-row blocks than SMs, an odd number of them and of tiles in each: the backward pipeline runs across block
    boundaries. Keys grow along the sequence, so that the forward pass has to move its reference maximum more than once.
    P, dS and the results are rounded to bf16 (2^-9 each); in the 2-norm of a gradient that stays below 1e-2."""
    D = 64
    torch.manual_seed(B + T + H)
    qkv = torch.randn(B, T, 3, H, D, device="cuda")
    qkv[:, :, 1] *= torch.linspace(0.3, 4.0, T, device="cuda")[None, :, None, None]
    qkv = qkv.view(B, T, 3 * H * D).to(BF)
    dout = torch.randn(B, T, H * D, device="cuda").to(BF)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, 0.125, causal=causal)
    assert rc == 0
    dqkv, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, 0.125, causal=causal)
    again, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, 0.125, causal=causal)
    torch.cuda.synchronize()
    assert C.attention_status()[0] == 0
    assert torch.equal(dqkv, again)  # no atomics: the same bits every time
    qr = qkv.double().requires_grad_(True)
    q, k, v = qr.view(B, T, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v, causal=causal).reshape(B, T, H * D)
    ref.backward(dout.double())
    assert ((out.double() - ref).norm() / ref.norm()).item() < 6e-3
    got, want = dqkv.double().view(B, T, 3, H, D), qr.grad.view(B, T, 3, H, D)
    for i in range(3):
        assert ((got[:, :, i] - want[:, :, i]).norm() / want[:, :, i].norm()).item() < 1e-2


@pytest.mark.parametrize("row", [0, 37, 63, 64, 127, 190])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_a_query_that_is_not_finite_stays_with_the_keys_it_sees(row, value):
    """Causal backward with one query row whose log-sum-exp is NaN or infinite: the keys after it get the same bits as without
    it, in dV and in dK, and no other query's dQ changes."""
    B, T, H, D = 1, 256, 2, 64
    torch.manual_seed(row)
    qkv, dout = torch.randn(B, T, 3 * H * D, device="cuda").to(BF), torch.randn(B, T, H * D, device="cuda").to(BF)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, 0.125, causal=True)
    assert rc == 0
    clean, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, 0.125, causal=True)
    bad_lse = lse.clone()
    bad_lse[0, 1, row] = value
    got, _ = C.attention_backward_tcgen05(qkv, out, dout, bad_lse, H, 0.125, causal=True)
    clean, got = clean.view(T, 3, H, D), got.view(T, 3, H, D)
    assert torch.equal(got[:, :, 0], clean[:, :, 0])  # the other head
    assert torch.equal(got[row + 1:, 1:, 1], clean[row + 1:, 1:, 1])
    others = torch.arange(T, device="cuda") != row
    assert torch.equal(got[others, 0, 1], clean[others, 0, 1])


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("scale", [0.125, 0.0, -0.125])
def test_backward_of_a_given_forward_takes_any_scale(scale, causal):
    """dqkv from an output and a log-sum-exp computed elsewhere. bf16 P, dS and results: below 1e-2 in the 2-norm."""
    B, T, H, D = 2, 256, 3, 64
    torch.manual_seed(5)
    qkv, dout = torch.randn(B, T, 3 * H * D, device="cuda").to(BF), torch.randn(B, T, H * D, device="cuda").to(BF)
    qr = qkv.double().requires_grad_(True)
    q, k, v = (x.transpose(1, 2) for x in qr.view(B, T, 3, H, D).unbind(2))
    s = q @ k.transpose(2, 3) * scale
    if causal:
        s = s.masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ref = (s.softmax(-1) @ v).transpose(1, 2).reshape(B, T, H * D)
    ref.backward(dout.double())
    lse = s.detach().logsumexp(-1).float().contiguous()
    got, _ = C.attention_backward_tcgen05(qkv, ref.detach().to(BF), dout, lse, H, scale, causal=causal)
    assert ((got.double() - qr.grad).norm() / qr.grad.norm()).item() < 1e-2


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("scale", [0.0, -0.125, -1.0, 1e-30])
def test_forward_and_backward_at_any_scale(gpu_scheduler, scale, causal):
    """Several key blocks through the op, at scales of zero and below. bf16 P and results: 6e-3 in the 2-norm forward, 1e-2 backward."""
    s = gpu_scheduler
    B, T, H, D = 1, 384, 2, 64
    torch.manual_seed(9)
    qkv, dout = torch.randn(B, T, 3 * H * D, device="cuda").to(BF), torch.randn(B, T, H * D, device="cuda").to(BF)
    op = ops.Attention(s, is_causal=causal, scale=scale)
    fallbacks = C.library_fallbacks()
    out = op.forward_packed(cs.from_torch(qkv), H)
    dqkv = op.backward_packed(cs.from_torch(dout))
    s.synchronize()
    assert C.library_fallbacks() == fallbacks
    qr = qkv.double().requires_grad_(True)
    q, k, v = (x.transpose(1, 2) for x in qr.view(B, T, 3, H, D).unbind(2))
    scores = q @ k.transpose(2, 3) * scale
    if causal:
        scores = scores.masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ref = (scores.softmax(-1) @ v).transpose(1, 2).reshape(B, T, H * D)
    ref.backward(dout.double())
    assert ((out.raw().double() - ref).norm() / ref.norm()).item() < 6e-3
    assert ((dqkv.raw().double() - qr.grad).norm() / qr.grad.norm()).item() < 1e-2


@pytest.mark.parametrize("B,T,H", [(3, 2048, 13), (149, 128, 1)])
def test_a_query_that_is_not_finite_among_many_blocks(B, T, H):
    """Several 128-row blocks a CTA, one of them with a NaN log-sum-exp: the CTAs concerned take another loop than the rest. Keys the
    query cannot see, other heads and sequences keep their values; those blocks round P' and dS' alike, so only the order of
    fp32 operations inside an element differs: 2^-7 of the largest gradient."""
    D, b, h, row = 64, B // 2, H // 2, T - 100
    torch.manual_seed(T)
    qkv, dout = torch.randn(B, T, 3 * H * D, device="cuda").to(BF), torch.randn(B, T, H * D, device="cuda").to(BF)
    rc, out, lse = C.attention_forward_tcgen05(qkv, H, 0.125, causal=True)
    assert rc == 0
    clean, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, 0.125, causal=True)
    lse[b, h, row] = float("nan")
    got, _ = C.attention_backward_tcgen05(qkv, out, dout, lse, H, 0.125, causal=True)
    torch.cuda.synchronize()
    assert C.attention_status()[0] == 0
    clean, got = clean.view(B, T, 3, H, D).float(), got.view(B, T, 3, H, D).float()
    bad = got.isnan().any(-1)  # [B, T, 3, H]
    want = torch.zeros_like(bad)
    want[b, row, 0, h] = True          # dQ of the query itself
    want[b, :row + 1, 1:, h] = True    # dK and dV of the keys it sees
    assert torch.equal(bad, want)
    assert ((got - clean)[~bad].abs().max() / clean.abs().max()).item() < 2 ** -7
