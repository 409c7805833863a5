# SPDX-License-Identifier: Apache-2.0
"""tcgen05 GEMM kernel: every layout/epilogue against fp32 PyTorch math, including ragged tiles."""
import pytest
import torch
import torch.nn.functional as F

import core_scheduler_b200 as cs

C = cs._C
pytestmark = pytest.mark.gpu
BF = torch.bfloat16
TN, NT = 0, 1
STORE, RESIDUAL, GELU_DUAL, DGELU, STORE_F32, ACCUM_F32, CE = range(7)


def rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


def operands(M, N, K):
    torch.manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, device="cuda").to(BF)
    b = torch.randn(N, K, device="cuda").mul_(0.1).to(BF)
    return a, b


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 768), (300, 2304, 768), (1000, 776, 200), (77, 8, 72),
                                   (4096, 768, 3072), (129, 264, 1032)])
def test_tn_store_and_bias(M, N, K):
    a, b = operands(M, N, K)
    ref = a.float() @ b.float().t()
    d = torch.full((M, N), float("nan"), device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, TN, STORE) == 0
    assert rel(d, ref) < 4e-3
    bias = torch.randn(N, device="cuda").to(BF)
    assert C.gemm_bf16(a, b, d, TN, STORE, bias=bias) == 0
    assert rel(d, ref + bias.float()) < 4e-3
    assert C.gemm_status()[0] == 0


def test_output_padding_is_untouched():
    """Rows/columns outside [M, N] of a strided output must never be written."""
    M, N, K = 200, 520, 128
    a, b = operands(M, N, K)
    big = torch.full((M + 8, N + 16), 7.0, device="cuda", dtype=BF)
    d = big[:M, :N]
    assert C.gemm_bf16(a, b, d, TN, STORE) == 0
    torch.cuda.synchronize()
    assert rel(d, a.float() @ b.float().t()) < 4e-3
    assert (big[M:] == 7).all() and (big[:, N:] == 7).all()


@pytest.mark.parametrize("M,N,K", [(256, 768, 768), (1000, 776, 264)])
def test_tn_residual_gelu_dual_dgelu(M, N, K):
    a, b = operands(M, N, K)
    ref = a.float() @ b.float().t()
    aux = torch.randn(M, N, device="cuda").to(BF)
    d = torch.empty(M, N, device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, TN, RESIDUAL, aux=aux) == 0
    assert rel(d, ref + aux.float()) < 4e-3
    d2 = torch.empty_like(d)
    assert C.gemm_bf16(a, b, d, TN, GELU_DUAL, d2=d2) == 0
    assert rel(d, ref) < 4e-3
    assert rel(d2, F.gelu(d.float())) < 4e-3  # GELU of the stored (rounded) pre-activation
    assert C.gemm_bf16(a, b, d, TN, DGELU, aux=aux) == 0
    x = aux.float().requires_grad_(True)
    F.gelu(x).backward(torch.ones_like(x))
    assert rel(d, ref * x.grad) < 5e-3


@pytest.mark.parametrize("Kr,M,N", [(64, 128, 256), (4096, 768, 2304), (1000, 200, 776), (16384, 768, 768), (520, 1032, 264)])
def test_nt_weight_gradient_store_and_accumulate(Kr, M, N):
    torch.manual_seed(Kr + M + N)
    a = torch.randn(Kr, M, device="cuda").to(BF)
    b = torch.randn(Kr, N, device="cuda").mul_(0.1).to(BF)
    ref = a.float().t() @ b.float()
    d = torch.full((M, N), float("nan"), device="cuda")
    assert C.gemm_bf16(a, b, d, NT, STORE_F32) == 0
    assert rel(d, ref) < 1e-4
    assert C.gemm_bf16(a, b, d, NT, ACCUM_F32) == 0
    assert rel(d, 2 * ref) < 1e-4
    assert C.gemm_status()[0] == 0


def test_tn_fp32_output():
    a, b = operands(256, 512, 4096)
    d = torch.zeros(256, 512, device="cuda")
    assert C.gemm_bf16(a, b, d, TN, STORE_F32) == 0
    assert rel(d, a.float() @ b.float().t()) < 1e-4


@pytest.mark.parametrize("M,V,K,valid", [(256, 1024, 128, 1000), (300, 1288, 256, 1288), (128, 50304, 64, 50257)])
def test_cross_entropy_epilogue_partials(M, V, K, valid):
    a, b = operands(M, V, K)
    tiles = C.gemm_ce_stat_tiles(V)
    stats = torch.full((M, tiles, 2), float("nan"), device="cuda")
    d = torch.empty(M, V, device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, TN, CE, stats=stats, n_valid=valid) == 0
    torch.cuda.synchronize()
    logits = d.float()[:, :valid]
    m = stats[..., 0].max(dim=1).values
    lse = m + torch.log((stats[..., 1] * torch.exp(stats[..., 0] - m[:, None]).nan_to_num(0.0)).sum(1))
    assert torch.allclose(lse, torch.logsumexp(logits, dim=1), atol=2e-3)
    assert rel(d, a.float() @ b.float().t()) < 4e-3


def test_unsupported_shapes_are_declined():
    a = torch.randn(64, 60, device="cuda").to(BF)  # K not a multiple of 8
    b = torch.randn(64, 60, device="cuda").to(BF)
    d = torch.empty(64, 64, device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, TN, STORE) == -1


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (4096, 768, 2304), (1000, 776, 264), (16384, 3072, 768), (100, 264, 136)])
def test_tm_input_gradient_layout(M, N, K):
    """A [M,K] row-major times B [K,N] row-major (the weight as stored): dX = dY * W."""
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(BF)
    b = torch.randn(K, N, device="cuda").mul_(0.1).to(BF)
    d = torch.full((M, N), float("nan"), device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, 2, STORE) == 0
    ref = a.float() @ b.float()
    assert rel(d, ref) < 4e-3
    aux = torch.randn(M, N, device="cuda").to(BF)
    assert C.gemm_bf16(a, b, d, 2, DGELU, aux=aux) == 0
    x = aux.float().requires_grad_(True)
    F.gelu(x).backward(torch.ones_like(x))
    assert rel(d, ref * x.grad) < 5e-3
    assert C.gemm_status()[0] == 0


@pytest.mark.parametrize("layout", [TN, 2])
@pytest.mark.parametrize("M,N,K", [(129, 8, 72), (384, 72, 200), (1536, 768, 768), (1000, 136, 64), (6000, 1288, 72), (2048, 2304, 328)])
def test_narrow_tiles_with_every_epilogue(M, N, K, layout):
    """Shapes whose output has too few 256-column tiles for the chip take 128- or 64-column ones: remainders in rows, columns
    and K, one column tile and many, with each bf16 epilogue. bf16 results: half an ulp, 2^-9 of the value, in the norm."""
    a, b = operands(M, N, K)
    bb = b if layout == TN else b.t().contiguous()
    ref = a.float() @ b.float().t()
    aux, bias = torch.randn(M, N, device="cuda").to(BF), torch.randn(N, device="cuda").to(BF)
    guard = torch.full((M + 3, N + 8), 7.0, device="cuda", dtype=BF)
    d, d2 = guard[:M, :N], torch.empty(M, N + 8, device="cuda", dtype=BF)[:, :N]
    assert C.gemm_bf16(a, bb, d, layout, STORE, bias=bias) == 0
    assert rel(d, ref + bias.float()) < 4e-3
    wide_aux = torch.empty(M, N + 8, device="cuda", dtype=BF)[:, :N].copy_(aux)  # the auxiliary operand has the output's row stride
    assert C.gemm_bf16(a, bb, d, layout, RESIDUAL, aux=wide_aux, bias=bias) == 0
    assert rel(d, ref + bias.float() + aux.float()) < 4e-3
    assert C.gemm_bf16(a, bb, d, layout, DGELU, aux=wide_aux) == 0
    x = aux.float().requires_grad_(True)
    F.gelu(x).backward(torch.ones_like(x))
    assert rel(d, ref * x.grad) < 5e-3
    assert C.gemm_bf16(a, bb, d, layout, GELU_DUAL, d2=d2, bias=bias) == 0
    assert rel(d, ref + bias.float()) < 4e-3 and rel(d2, F.gelu(ref + bias.float())) < 4e-3
    assert (guard[M:] == 7).all() and (guard[:, N:] == 7).all()
    assert C.gemm_status()[0] == 0


def test_gelu_epilogue_limits():
    """Infinite and very large pre-activations of either sign: GELU is x on the right and zero on the left, never NaN."""
    a = torch.zeros(256, 64, device="cuda", dtype=BF)
    a[:, 0] = 1
    b = torch.zeros(256, 64, device="cuda", dtype=BF)
    b[:6, 0] = torch.tensor([float("inf"), 3e38, -3e38, -20.0, 20.0, float("-inf")])
    d, d2 = torch.empty(256, 256, device="cuda", dtype=BF), torch.empty(256, 256, device="cuda", dtype=BF)
    assert C.gemm_bf16(a, b, d, TN, GELU_DUAL, d2=d2, bias=None) == 0
    big = b[1, 0].item()
    assert torch.equal(d[7, :6], b[:6, 0]) and not d2.isnan().any()
    assert d2[7, 0].item() == float("inf") and d2[7, 5].item() == 0
    assert d2[7, 1].item() == big and d2[7, 2].item() == 0 and d2[7, 3].item() == 0 and d2[7, 4].item() == 20


@pytest.mark.parametrize("spread", [1.0, 100.0, 3e37])
@pytest.mark.parametrize("M,N,n_valid", [(130, 512, 512), (64, 640, 600), (256, 136, 130)])
def test_softmax_partials_hold_the_exact_maximum(M, N, n_valid, spread):
    """(max, sum-exp) of every 128-column half tile: the maximum is the stored logit itself, the sum that of exp(x - max), at
    magnitudes up to where a product with log2(e) overflows. ex2.approx is within 2 ulp, 2^-22; at most 128 fp32 additions."""
    torch.manual_seed(M + N)
    a, b = torch.zeros(M, 64, device="cuda", dtype=BF), (torch.randn(N, 64, device="cuda") * spread).to(BF)
    a[torch.arange(M), torch.arange(M) % 64] = 1  # each row of logits is a column of b
    d = torch.empty(M, N, device="cuda", dtype=BF)
    tiles = 2 * ((N + 255) // 256)
    stats = torch.full((M, tiles, 2), 7.0, device="cuda")
    assert C.gemm_bf16(a, b, d, TN, 6, stats=stats, n_valid=n_valid) == 0
    x = d.double()
    x[:, n_valid:] = float("-inf")
    x = torch.nn.functional.pad(x, (0, tiles * 128 - N), value=float("-inf")).view(M, tiles, 128)
    mx = x.amax(-1)
    assert torch.equal(stats[..., 0].double(), mx)
    want = torch.where(mx > float("-inf"), (x - mx[..., None]).exp().sum(-1), torch.zeros_like(mx))
    assert ((stats[..., 1].double() - want).abs() <= (128 * 2.0 ** -24 + 2.0 ** -20) * want).all()


@pytest.mark.parametrize("M,N,K", [(844, 1024, 3072), (1200, 1024, 3072), (1500, 1024, 3072), (1500, 768, 2304), (2000, 768, 2304), (5, 1024, 3072)])
def test_input_gradient_widths_beside_a_weight_gradient(M, N, K):
    """Input gradients whose tile width depends on what their layer's weight gradient leaves free, on both sides of the line, and
    that weight gradient. bf16 results: half an ulp, 2^-9 of the value, in the norm; fp32 ones: sums of M terms."""
    torch.manual_seed(M + N)
    dy, w, x = (torch.randn(*shape, device="cuda").to(BF) for shape in ((M, K), (K, N), (M, N)))
    dx = torch.empty(M, N, device="cuda", dtype=BF)
    assert C.gemm_bf16(dy, w, dx, 2, STORE) == 0
    assert rel(dx, dy.float() @ w.float()) < 4e-3
    dw = torch.empty(K, N, device="cuda")
    assert C.gemm_bf16(dy, x, dw, 1, 4) == 0
    assert rel(dw, dy.float().t() @ x.float()) < 1e-4
    assert C.gemm_status()[0] == 0
