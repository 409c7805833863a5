# SPDX-License-Identifier: Apache-2.0
"""sm_100a kernels against plain PyTorch fp32 references of the same op (GPU only)."""
import math

import pytest
import torch
import torch.nn.functional as F

import core_scheduler_b200 as cs
from helpers import T, TorchGPT2, attention_reference

C = cs._C
pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def bf16_close(a, b, atol=2e-2, rtol=2e-2):
    return torch.allclose(a.float(), b.float(), atol=atol, rtol=rtol)


def test_native_kernels_are_the_path_that_runs(gpu_scheduler):
    s = gpu_scheduler
    before = C.kernel_launch_count()
    st = C.gelu_init(s)
    C.gelu_forward(s, st, T(torch.randn(1024, device="cuda", dtype=BF)))
    s.synchronize()
    assert C.get_backend() == "fused"
    assert C.kernel_launch_count() > before


@pytest.mark.parametrize("rows,d", [(64, 768), (1000, 1024), (37, 1280), (8, 256), (5, 2048), (3, 4096)])
def test_layernorm_forward_backward(gpu_scheduler, rows, d):
    s = gpu_scheduler
    torch.manual_seed(0)
    st = C.layer_norm_init(s, [d])  # fp32 parameters
    st.weight.raw().uniform_(0.5, 1.5)
    st.bias.raw().uniform_(-0.5, 0.5)
    x = torch.randn(rows, d, device="cuda").mul_(2).add_(0.5).to(BF)
    dy = torch.randn(rows, d, device="cuda").to(BF)
    res = torch.randn(rows, d, device="cuda").to(BF)
    xr = x.float().requires_grad_(True)
    w = st.weight.raw().clone().requires_grad_(True)
    b = st.bias.raw().clone().requires_grad_(True)
    yr = F.layer_norm(xr, (d,), w, b)
    yr.backward(dy.float())
    with cs.autocast(s, BF):
        y = C.layer_norm_forward(s, st, T(x))
    dx = C.layer_norm_backward(s, st, T(dy), T(res))
    s.synchronize()
    assert y.raw().dtype == BF
    assert bf16_close(y.raw(), yr)
    assert bf16_close(dx.raw(), xr.grad + res.float(), atol=4e-2)
    assert torch.allclose(st.grad_weight.raw(), w.grad, atol=2e-2 * math.sqrt(rows), rtol=2e-2)
    assert torch.allclose(st.grad_bias.raw(), b.grad, atol=2e-2 * math.sqrt(rows), rtol=2e-2)
    # second micro-step accumulates
    with cs.autocast(s, BF):
        C.layer_norm_forward(s, st, T(x))
    C.layer_norm_backward(s, st, T(dy))
    s.synchronize()
    assert torch.allclose(st.grad_bias.raw(), 2 * b.grad, atol=4e-2 * math.sqrt(rows), rtol=2e-2)


@pytest.mark.parametrize("n", [8, 1000, 1 << 20, (1 << 20) + 3])
def test_gelu_and_add(gpu_scheduler, n):
    s = gpu_scheduler
    x = torch.randn(n, device="cuda").mul_(3).to(BF)
    dy = torch.randn(n, device="cuda").to(BF)
    st = C.gelu_init(s)
    y = C.gelu_forward(s, st, T(x))
    dx = C.gelu_backward(s, st, T(dy))
    xr = x.float().requires_grad_(True)
    yr = F.gelu(xr)
    yr.backward(dy.float())
    s.synchronize()
    assert bf16_close(y.raw(), yr)
    assert bf16_close(dx.raw(), xr.grad)
    if n % 8 == 0:
        z = C.utils_add(s, T(x), T(dy))
        s.synchronize()
        assert bf16_close(z.raw(), x.float() + dy.float())


def test_embedding_token_position(gpu_scheduler):
    s = gpu_scheduler
    V, P, d, B, Tn = 1000, 64, 256, 4, 48
    te, pe = C.embedding_init(s, V, d), C.embedding_init(s, P, d)
    idx = torch.randint(0, V, (B, Tn), device="cuda")
    idx[0, :8] = 7  # duplicates exercise the atomics
    with cs.autocast(s, BF):
        y = C.embedding_forward_token_position(s, te, pe, T(idx))
    ref = te.weight.raw()[idx] + pe.weight.raw()[:Tn][None]
    dy = torch.randn(B, Tn, d, device="cuda").to(BF)
    C.embedding_backward_token_position(s, te, pe, T(dy))
    s.synchronize()
    assert bf16_close(y.raw(), ref)
    gte = torch.zeros(V, d, device="cuda").index_add_(0, idx.reshape(-1), dy.float().reshape(-1, d))
    gpe = torch.zeros(P, d, device="cuda")
    gpe[:Tn] = dy.float().sum(0)
    assert torch.allclose(te.grad_weight.raw(), gte, atol=1e-3)
    assert torch.allclose(pe.grad_weight.raw(), gpe, atol=1e-3)


@pytest.mark.parametrize("n", [1000, 1 << 20])
@pytest.mark.parametrize("amsgrad", [False, True])
def test_adamw_kernel_fp32_master_with_bf16_copy(gpu_scheduler, n, amsgrad):
    from test_optimizer_module import adamw_reference

    s = gpu_scheduler
    w0 = torch.randn(n, device="cuda")
    w = T(w0.clone())
    C.working_copy(s, w, BF)  # creates the bf16 working copy the kernel refreshes
    st = C.adamw_init(s, w, lr=1e-2, beta1=0.9, beta2=0.95, weight_decay=0.1, amsgrad=amsgrad)
    wr, m, v = w0.clone(), torch.zeros_like(w0), torch.zeros_like(w0)
    vmax = torch.zeros_like(w0) if amsgrad else None
    for t in range(1, 4):
        g = torch.randn(n, device="cuda")
        C.adamw_step(s, st, w, T(g))
        wr, m, v, vmax = adamw_reference(wr, g, m, v, t, 1e-2, 0.9, 0.95, 1e-8, 0.1, vmax)
    s.synchronize()
    assert torch.allclose(w.raw(), wr, rtol=1e-4, atol=1e-5)
    assert torch.allclose(st.m.raw(), m, rtol=1e-4, atol=1e-6)
    assert torch.equal(w.lp(), w.raw().to(BF))


def test_adamw_kernel_bf16_gradients(gpu_scheduler):
    s = gpu_scheduler
    w = T(torch.randn(4096, device="cuda"))
    ref = w.raw().clone()
    st = C.adamw_init(s, w, lr=1e-2, weight_decay=0.0)
    g = torch.randn(4096, device="cuda").to(BF)
    C.adamw_step(s, st, w, T(g))
    s.synchronize()
    # first step of Adam moves every weight by ~lr * sign(g)
    assert torch.allclose(w.raw(), ref - 1e-2 * torch.sign(g.float()), atol=1e-4)


def test_clip_grad_norm_kernels(gpu_scheduler):
    s = gpu_scheduler
    g1 = torch.randn(100000, device="cuda") * 3
    g2 = (torch.randn(5000, device="cuda") * 3).to(BF)
    ref = torch.cat([g1, g2.float()]).norm()
    norm = C.utils_clip_grad_norm_(s, [T(g1), T(g2)], 1.0)
    s.synchronize()
    assert torch.allclose(norm.raw(), ref, rtol=1e-3)
    assert abs(torch.cat([g1, g2.float()]).norm().item() - 1.0) < 2e-2


def test_transposed_working_copy(gpu_scheduler):
    s = gpu_scheduler
    w = T(torch.randn(300, 200, device="cuda"))
    wt = C.working_copy_transposed(s, w, BF)
    s.synchronize()
    assert torch.equal(wt.raw(), w.raw().t().to(BF))


@pytest.mark.parametrize("M,K,N", [(256, 128, 256), (300, 768, 2304), (1024, 3072, 768), (128, 64, 100)])
def test_linear_paths_bf16(gpu_scheduler, M, K, N):
    """Forward (+residual, +GELU companion), dgrad and fp32-accumulated wgrad against fp32 math."""
    s = gpu_scheduler
    torch.manual_seed(1)
    st = C.linear_init(s, K, N, bias=False, gelu_epilogue=True)
    st.weight.raw().normal_(0, 0.05)
    x = torch.randn(M, K, device="cuda").to(BF)
    res = torch.randn(M, N, device="cuda").to(BF)
    dy = torch.randn(M, N, device="cuda").mul_(0.1).to(BF)
    w = st.weight.raw().to(BF).float()
    with cs.autocast(s, BF):
        y = C.linear_forward(s, st, T(x))
    dx = C.linear_backward_input(s, st, T(dy))
    C.linear_backward_parameter(s, st, T(dy))
    with cs.autocast(s, BF):
        C.linear_forward(s, st, T(x))
    C.linear_backward_parameter(s, st, T(dy))  # accumulates
    s.synchronize()
    ref = x.float() @ w.t()
    assert bf16_close(y.raw(), ref, atol=3e-2)
    assert bf16_close(y.companion(), F.gelu(ref), atol=3e-2)
    assert bf16_close(dx.raw(), dy.float() @ w, atol=3e-2)
    gw = dy.float().t() @ x.float()
    assert st.grad_weight.raw().dtype == torch.float32
    assert torch.allclose(st.grad_weight.raw(), 2 * gw, atol=5e-2, rtol=2e-2)
    st2 = C.linear_init(s, K, N, bias=False)
    st2.weight.raw().copy_(st.weight.raw())
    with cs.autocast(s, BF):
        y2 = C.linear_forward(s, st2, T(x), T(res))
    s.synchronize()
    assert bf16_close(y2.raw(), ref + res.float(), atol=4e-2)


def test_gelu_linear_bf16(gpu_scheduler):
    s = gpu_scheduler
    M, K, N = 512, 1024, 256
    st = C.gelu_linear_init(s, K, N, bias=False)
    st.weight.raw().normal_(0, 0.05)
    x = torch.randn(M, K, device="cuda").to(BF)
    dy = torch.randn(M, N, device="cuda").mul_(0.1).to(BF)
    with cs.autocast(s, BF):
        y = C.gelu_linear_forward(s, st, T(x))
    dx = C.gelu_linear_backward_input(s, st, T(dy))
    C.gelu_linear_backward_parameter(s, st, T(dy))
    s.synchronize()
    xr = x.float().requires_grad_(True)
    w = st.weight.raw().to(BF).float().requires_grad_(True)
    yr = F.gelu(xr) @ w.t()
    yr.backward(dy.float())
    assert bf16_close(y.raw(), yr, atol=3e-2)
    assert bf16_close(dx.raw(), xr.grad, atol=3e-2)
    assert torch.allclose(st.grad_weight.raw(), w.grad, atol=5e-2, rtol=2e-2)


@pytest.mark.parametrize("rows,d,V,valid", [(256, 128, 512, 500), (1000, 768, 2048, 2048), (130, 256, 1280, 1279)])
def test_fused_classifier_cross_entropy(gpu_scheduler, rows, d, V, valid):
    s = gpu_scheduler
    torch.manual_seed(2)
    lin = C.linear_init(s, d, V, bias=False)
    lin.weight.raw().normal_(0, 0.05)
    st = C.linear_cross_entropy_init(s, lin, valid_classes=valid)
    x = torch.randn(rows, d, device="cuda").to(BF)
    t = torch.randint(0, valid, (rows,), device="cuda")
    t[3] = -100
    with cs.autocast(s, BF):
        loss = C.linear_cross_entropy_forward(s, st, T(x), T(t))
    dx = C.linear_cross_entropy_backward(s, st)
    s.synchronize()
    xr = x.float().requires_grad_(True)
    w = lin.weight.raw().to(BF).float().requires_grad_(True)
    lr = F.cross_entropy((xr @ w.t())[:, :valid], t)
    lr.backward()
    assert abs(loss.raw().item() - lr.item()) < 2e-2
    assert bf16_close(dx.raw(), xr.grad, atol=2e-3, rtol=5e-2)
    assert torch.allclose(lin.grad_weight.raw(), w.grad, atol=2e-3, rtol=5e-2)


def test_attention_bf16_packed(gpu_scheduler):
    s = gpu_scheduler
    B, Tn, H, D = 2, 256, 4, 64
    qkv = torch.randn(B, Tn, 3 * H * D, device="cuda").to(BF)
    st = C.attention_init(s, is_causal=True)
    out = C.attention_forward_packed(s, st, T(qkv), H)
    do = torch.randn(B, Tn, H * D, device="cuda").to(BF)
    dqkv = C.attention_backward_packed(s, st, T(do))
    s.synchronize()
    qr = qkv.float().requires_grad_(True)
    q, k, v = qr.view(B, Tn, 3, H, D).unbind(2)
    ref = attention_reference(q, k, v).reshape(B, Tn, H * D)
    ref.backward(do.float())
    assert bf16_close(out.raw(), ref, atol=3e-2)
    assert bf16_close(dqkv.raw(), qr.grad, atol=5e-2, rtol=5e-2)


def _train_losses(s, backend, steps=4):
    C.set_backend(backend)
    try:
        cs.manual_seed(0)
        cfg = cs.GPT2Config(n_layer=2, n_head=4, n_embd=256, block_size=128, vocab_size=1000, padded_vocab_size=1024)
        m = cs.GPT2(s, cfg)
        flat = C.flatten_parameters(s, m, lp_dtype=BF)
        opt = cs.AdamW(s, m, lr=1e-3, beta1=0.9, beta2=0.95, weight_decay=0.1, flat=flat)
        g = torch.Generator(device="cuda").manual_seed(3)
        ids = torch.randint(0, 1000, (4, 129), device="cuda", generator=g)
        x, y = T(ids[:, :-1].contiguous()), T(ids[:, 1:].contiguous())
        first = {k: v.raw().clone() for k, v in m.named_parameters().items()}
        losses = []
        for _ in range(steps):
            with cs.autocast(s, BF):
                loss = m.forward_loss(s, x, y)
            m.backward_loss(s)
            if not losses:
                s.synchronize()
                grads = {k: v.raw().clone() for k, v in m.named_gradients().items()}
            opt.step(s)
            opt.zero_grad(s)
            losses.append(cs.to_torch(s, loss).item())
        return losses, first, grads, (ids[:, :-1], ids[:, 1:])
    finally:
        C.set_backend("fused")


def test_gpt2_bf16_training_matches_fp32_autograd_and_library_backend(gpu_scheduler):
    s = gpu_scheduler
    fused, params, grads, (ids, lab) = _train_losses(s, "fused")
    lib, _, _, _ = _train_losses(s, "library")
    ref = TorchGPT2(2, 4, 256, 128, 1024, 1000).cuda()
    ref.load_from(params)
    lr = ref(ids, lab)
    lr.backward()
    assert abs(fused[0] - lr.item()) < 3e-2
    assert abs(lib[0] - lr.item()) < 3e-2
    assert fused[-1] < fused[0]
    for a, b in zip(fused, lib):
        assert abs(a - b) < 5e-2
    for k in ("lm_head.weight", "1.mlp.fc2.weight", "0.attn.c_attn.weight", "0.ln1.weight", "wpe.weight"):
        g, r = grads[k].float(), ref.p(k).grad
        err = (g - r).norm() / (r.norm() + 1e-12)
        assert err < 5e-2, (k, err.item())


@pytest.mark.parametrize("rows,d,offset", [(1, 8, 0), (50, 768, 0), (333, 1000, 0), (64, 264, 1)])
def test_embedding_backward_hot_ids_and_unaligned_table(gpu_scheduler, rows, d, offset):
    """Most rows add into one id; the gradient table starts at any fp32 element (vector or scalar reductions). Up to `rows` fp32
    additions in any order: an error of rows * 2^-24 of the largest partial sum."""
    s = gpu_scheduler
    torch.manual_seed(rows + d)
    V = 40
    te = C.embedding_init(s, V, d)
    idx = torch.randint(0, V, (rows,), device="cuda")
    idx[: rows // 2 + 1] = 7
    dy = torch.randn(rows, d, device="cuda").to(BF)
    store = torch.zeros(V * d + offset, device="cuda")
    te.grad_weight.set_raw(store[offset:].view(V, d))
    with cs.autocast(s, BF):
        y = C.embedding_forward(s, te, T(idx))
    C.embedding_backward(s, te, T(dy))
    s.synchronize()
    assert torch.equal(y.raw(), te.weight.raw()[idx].to(BF))
    want = torch.zeros(V, d, device="cuda", dtype=torch.float64).index_add_(0, idx, dy.double())
    bound = rows * 2.0 ** -24 * torch.zeros(V, d, device="cuda", dtype=torch.float64).index_add_(0, idx, dy.double().abs()).max()
    assert (te.grad_weight.raw().double() - want).abs().max() <= bound


@pytest.mark.parametrize("rows,d", [(1, 8), (3, 256), (5, 264), (4099, 760), (2500, 1600), (1030, 2048), (2, 2056)])
def test_layernorm_column_kernels(gpu_scheduler, rows, d):
    """Widths around a warp's 256 columns and the 2048 limit, row counts around the group of four, more rows than one wave of
    CTAs, and the accumulation into existing gradients. bf16 outputs: half an ulp, 2^-9; fp32 sums over the rows: 1e-5."""
    s = gpu_scheduler
    torch.manual_seed(rows + d)
    st = C.layer_norm_init(s, [d])
    st.weight.raw().uniform_(0.5, 1.5)
    st.bias.raw().uniform_(-0.5, 0.5)
    x, dy, res = (torch.randn(rows, d, device="cuda").mul_(2).add_(0.5).to(BF) for _ in range(3))
    xr = x.double().requires_grad_(True)
    w, b = (t.raw().double().requires_grad_(True) for t in (st.weight, st.bias))
    yr = F.layer_norm(xr, (d,), w, b)
    yr.backward(dy.double())

    def rel(a, want):
        return ((a.double() - want).norm() / want.norm()).item()

    for step in (1, 2):
        with cs.autocast(s, BF):
            y = C.layer_norm_forward(s, st, T(x))
        dx = C.layer_norm_backward(s, st, T(dy), T(res))
        s.synchronize()
        assert rel(y.raw(), yr.detach()) < 2e-3 and rel(dx.raw(), xr.grad + res.double()) < 3e-3
        assert rel(st.grad_weight.raw(), step * w.grad) < 1e-5 and rel(st.grad_bias.raw(), step * b.grad) < 1e-5


@pytest.mark.parametrize("rows,n", [(1, 8), (31, 72), (64, 3072), (65, 64), (3000, 5120), (70001, 136)])
def test_bias_gradient_column_sums(gpu_scheduler, rows, n):
    """One block per column group and several, remainders of both; stored, then accumulated. A term goes through one addition per
    64 rows of its block, 8 more on the way to the block's sum, one per 8 blocks and 4 more among the blocks: that many times 2^-24
    of the sum of magnitudes. Whole numbers add up exactly."""
    s = gpu_scheduler
    torch.manual_seed(rows + n)
    st = C.linear_init(s, 8, n, bias=True)
    x, dy = torch.zeros(rows, 8, device="cuda", dtype=BF), torch.randn(rows, n, device="cuda").to(BF)
    parts = max(1, min(-(-592 // -(-n // 64)), -(-rows // 64), 64))
    depth = -(-rows // (64 * parts)) + 8 + -(-parts // 8) + 4
    for whole in (False, True):
        if whole:
            dy = torch.randint(-9, 10, (rows, n), device="cuda").to(BF)
        st.zero_grad()
        want, bound = dy.double().sum(0), depth * 2.0 ** -24 * dy.double().abs().sum(0) + 1e-30
        for step in (1, 2):
            with cs.autocast(s, BF):
                C.linear_forward(s, st, T(x))
            C.linear_backward_parameter(s, st, T(dy))
            s.synchronize()
            assert ((st.grad_bias.raw().double() - step * want).abs() <= (0 if whole else step * bound)).all()
    assert st.grad_bias.raw().shape == (n,) and st.grad_bias.raw().dtype == torch.float32


def test_bias_gradient_is_as_close_as_pairwise_sums(gpu_scheduler):
    """20000 rows: the half dozen additions that are made near the magnitude of the result leave about sqrt(6) * 2^-24 / sqrt(3) in
    the 2-norm (a chain of all partial rows left 1.0e-7, the library's reduction 7e-8)."""
    s = gpu_scheduler
    torch.manual_seed(3)
    st = C.linear_init(s, 8, 1024, bias=True)
    x, dy = torch.zeros(20000, 8, device="cuda", dtype=BF), torch.randn(20000, 1024, device="cuda").to(BF)
    with cs.autocast(s, BF):
        C.linear_forward(s, st, T(x))
    C.linear_backward_parameter(s, st, T(dy))
    s.synchronize()
    want = dy.double().sum(0)
    assert ((st.grad_bias.raw().double() - want).norm() / want.norm()).item() < (6 / 3) ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("d", [8, 56, 88, 768, 896, 1000, 1792, 2048, 2304])
def test_layernorm_of_constant_rows_is_the_bias(gpu_scheduler, d):
    """Rows of one value: their sum is exact in fp32 (8 + 12 bits), so the mean is the value, the deviation zero, and the result
    the bias to the last bit, however far rstd magnifies."""
    s = gpu_scheduler
    st = C.layer_norm_init(s, [d])
    st.weight.raw().uniform_(0.5, 1.5)
    st.bias.raw().uniform_(-0.5, 0.5)
    x = torch.tensor([100.5, -0.0302734375, 3.015625, 1e4, -7.0], device="cuda").to(BF)[:, None].expand(5, d).contiguous()
    with cs.autocast(s, BF):
        y = C.layer_norm_forward(s, st, T(x))
    s.synchronize()
    assert torch.equal(y.raw(), st.bias.raw().to(BF).expand(5, d))


@pytest.mark.parametrize("rows,d", [(1, 768), (3, 776), (2, 512), (5, 584), (7, 592), (4737, 256), (9999, 768), (2961, 776), (1300, 520)])
def test_layernorm_where_its_dispatch_changes(gpu_scheduler, rows, d):
    """Around 768 columns (a warp or a CTA per row forward), 592 (columns per block of the gradient sum) and a multiple of 256,
    with odd row counts below and above one wave of CTAs: the bounds of the test above."""
    test_layernorm_column_kernels(gpu_scheduler, rows, d)


@pytest.mark.parametrize("first,last", [(0, 32), (0, 128), (64, 96), (0, 512), (480, 500)])
def test_nan_logits_of_whole_chunks_reach_the_loss(gpu_scheduler, first, last):
    """NaN in all logits of one 32-column chunk, of a half tile, of every column, or of the last columns before the end of the
    vocabulary (the epilogue looks at 32 columns at a time): the row's loss is NaN, as log_softmax has it."""
    s = gpu_scheduler
    torch.manual_seed(0)
    lin = C.linear_init(s, 64, 512, bias=False)
    s.synchronize()
    lin.weight.raw()[first:last] = float("nan")
    ce = C.linear_cross_entropy_init(s, lin, valid_classes=500)
    x = torch.randn(40, 64, device="cuda").to(BF)
    target = torch.full((40,), 300, device="cuda")
    with cs.autocast(s, BF):
        loss = C.linear_cross_entropy_forward(s, ce, T(x), T(target))
    s.synchronize()
    assert torch.isnan(loss.raw()).all()


def test_classifier_gradient_keeps_subnormal_probabilities(gpu_scheduler):
    """One row with logits 0 .. -100: probabilities down to 2^-133, bf16's smallest number, come back as gradients. bf16 keeps
    fewer bits there: half of 2^-133 beside 2^-8 of the value."""
    s = gpu_scheduler
    lin = C.linear_init(s, 64, 64, bias=False)
    s.synchronize()
    w = lin.weight.raw()
    w.zero_()
    w[:, 0] = torch.linspace(0, -100, 64, device="cuda")
    ce = C.linear_cross_entropy_init(s, lin)
    x = torch.zeros(1, 64, device="cuda", dtype=BF)
    x[0, 0] = 1
    with cs.autocast(s, BF):
        C.linear_cross_entropy_forward(s, ce, T(x), T(torch.zeros(1, dtype=torch.int64, device="cuda")))
    C.linear_cross_entropy_backward(s, ce)
    s.synchronize()
    p = torch.softmax(w[:, 0].to(BF).double(), 0)[1:]
    got = lin.grad_weight.raw()[1:, 0].double()
    assert ((got - p).abs() <= 2.0 ** -8 * p + 2.0 ** -133 * 0.51).all()
    assert (got[p > 2.0 ** -132] > 0).all()


@pytest.mark.parametrize("rows,vocab,padded", [(3, 7, 8), (70, 300, 304), (2500, 512, 512), (33, 1000, 1000), (9, 7160, 7160), (9, 8190, 8192), (9, 8200, 8200)])
def test_classifier_loss_over_vocabulary_sizes(gpu_scheduler, rows, vocab, padded):
    """Rows of less than one chunk a thread, the last width with fewer than 256 threads, 64 and 66 softmax partials a row, more rows
    than CTAs. The reference starts from the bf16 logits, so that the loss is left with fp32 sums (and logits that round the
    other way: 2^-9 of one in a few); gradients are bf16, 5e-3 in the norm."""
    s = gpu_scheduler
    torch.manual_seed(rows + vocab)
    lin = C.linear_init(s, 64, padded, bias=False)
    ce = C.linear_cross_entropy_init(s, lin, valid_classes=vocab)
    x, target = torch.randn(rows, 64, device="cuda").to(BF), torch.randint(0, vocab, (rows,), device="cuda")
    target[0] = vocab - 1
    s.synchronize()
    with cs.autocast(s, BF):
        loss = C.linear_cross_entropy_forward(s, ce, T(x), T(target))
    dx = C.linear_cross_entropy_backward(s, ce)
    s.synchronize()
    w = lin.weight.raw().to(BF).double()
    logits = (x.double() @ w[:vocab].t()).to(BF).double().requires_grad_(True)
    ref = F.cross_entropy(logits, target)
    ref.backward()
    assert abs(loss.raw().double().item() - ref.item()) < 1e-4 * max(1.0, ref.item())
    dw = torch.zeros_like(w)
    dw[:vocab] = logits.grad.t() @ x.double()
    assert ((dx.raw().double() - logits.grad @ w[:vocab]).norm() / (logits.grad @ w[:vocab]).norm()).item() < 5e-3
    assert ((lin.grad_weight.raw().double() - dw).norm() / dw.norm()).item() < 5e-3


@pytest.mark.parametrize("batch,seq,d", [(1, 1, 8), (2, 57, 1280), (3, 5, 264), (1, 37, 1288), (4, 592, 264), (3, 790, 264), (5, 1000, 768)])
def test_token_and_position_embedding_pieces(gpu_scheduler, batch, seq, d):
    """Rows of one piece and several, whole and not, on both sides of the row count from which backward gives a row one warp. The
    forward sum is one fp32 addition, rounded once; gradients are fp32 sums of at most batch * seq terms."""
    s = gpu_scheduler
    torch.manual_seed(batch * seq + d)
    V = 30
    te, pe = C.embedding_init(s, V, d), C.embedding_init(s, 1024, d)
    idx = torch.randint(0, V, (batch, seq), device="cuda")
    dy = torch.randn(batch, seq, d, device="cuda").to(BF)
    with cs.autocast(s, BF):
        y = C.embedding_forward_token_position(s, te, pe, T(idx))
    C.embedding_backward_token_position(s, te, pe, T(dy))
    s.synchronize()
    assert torch.equal(y.raw(), (te.weight.raw()[idx] + pe.weight.raw()[:seq]).to(BF))
    want = torch.zeros(V, d, device="cuda", dtype=torch.float64).index_add_(0, idx.view(-1), dy.double().view(-1, d))
    size = torch.zeros(V, d, device="cuda", dtype=torch.float64).index_add_(0, idx.view(-1), dy.double().abs().view(-1, d))
    count = torch.bincount(idx.view(-1), minlength=V)[:, None]
    assert ((te.grad_weight.raw().double() - want).abs() <= count * 2.0 ** -24 * size).all()
    assert ((pe.grad_weight.raw()[:seq].double() - dy.double().sum(0)).abs() <= batch * 2.0 ** -24 * dy.double().abs().sum(0)).all()
