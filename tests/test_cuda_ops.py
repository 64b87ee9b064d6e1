"""Every sm_100a kernel against the plain-PyTorch fp32 statement of the same op (ops/ref.py)."""

import math

import pytest
import torch

from tinyllmforge_b200.ops import ref
from tinyllmforge_b200.ops.cuda import decode_chunking

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    from tinyllmforge_b200.ops.cuda import CudaOps
    o = CudaOps()
    yield o
    o.check_status()


def _rand(*shape, scale=1.0, dtype=BF):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _close(a, b, atol, rtol):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    bad = (err > tol).sum().item()
    assert bad == 0, f"{bad}/{a.numel()} elements off; max err {err.max().item():.4g} (max ref {b.abs().max().item():.4g})"


# ----------------------------------------------------------------------------- GEMM (tcgen05)
@pytest.mark.parametrize("M,N,K,mode", [
    (1, 128, 64, 0), (16, 256, 128, 0), (7, 1024, 1024, 0), (64, 4096, 1024, 0), (200, 1024, 2048, 0),
    (256, 6144, 1024, 0), (128, 128, 64, 1), (300, 384, 256, 1), (1000, 1024, 1024, 0), (4096, 4096, 1024, 0),
    (130, 200, 72, 1), (33, 136, 200, 2), (256, 1024, 3072, 2),
    # one rank's shapes of the 32B architecture split 8 ways: qkv, o_proj, down_proj at decode and prefill sizes
    (64, 1280, 5120, 0), (64, 5120, 1024, 0), (64, 5120, 3200, 0), (2048, 1280, 5120, 0), (2048, 5120, 3200, 0),
])
def test_gemm_matches_fp32(ops, M, N, K, mode):
    torch.manual_seed(M * 7 + N)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    out = ops.linear(x, w, force_mode=mode)
    want = x.float() @ w.float().t()
    _close(out, want, atol=2e-2, rtol=2e-2)
    ops.check_status()


@pytest.mark.parametrize("M,I,K,mode", [(8, 256, 128, 0), (100, 3072, 1024, 0), (256, 1536, 1024, 2), (700, 3072, 1024, 0), (384, 512, 256, 1),
                                        (64, 3200, 5120, 0), (2048, 3200, 5120, 0)])
def test_gemm_silu_mul_epilogue(ops, M, I, K, mode):
    torch.manual_seed(M + I)
    x, w = _rand(M, K), _rand(2 * I, K, scale=0.05)
    out = ops.linear_silu_mul(x, w, force_mode=mode)
    gu = x.float() @ w.float().t()
    want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    _close(out, want, atol=2e-2, rtol=2e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,splits", [
    (256, 1024, 2048, 8), (256, 1024, 3072, 8), (200, 4096, 1024, 4), (16, 1024, 2048, 4), (1, 1024, 1024, 2),
    (64, 1024, 2048, 8), (128, 512, 1024, 1), (40, 384, 448, 4), (256, 151936 // 8, 1024, 1),
])
def test_gemm_decode_kernel_split_k(ops, M, N, K, splits):
    """Weight-tile kernel with K split over a thread-block cluster and the DSMEM reduction."""
    torch.manual_seed(M + N + splits)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    out = ops.linear(x, w, force_mode=2, force_splits=splits)
    _close(out, x.float() @ w.float().t(), atol=2e-2, rtol=2e-2)
    again = ops.linear(x, w, force_mode=2, force_splits=splits)
    assert torch.equal(out, again)                       # fixed reduction order: bit-reproducible
    ops.check_status()


@pytest.mark.parametrize("M,I,K,splits", [(256, 3072, 1024, 4), (256, 3072, 1024, 1), (24, 1536, 1024, 2), (100, 512, 2048, 8), (8, 256, 256, 2)])
def test_gemm_decode_kernel_silu_split_k(ops, M, I, K, splits):
    torch.manual_seed(M + I + splits)
    x, w = _rand(M, K), _rand(2 * I, K, scale=0.05)
    out = ops.linear_silu_mul(x, w, force_mode=2, force_splits=splits)
    gu = x.float() @ w.float().t()
    _close(out, torch.nn.functional.silu(gu[:, :I]) * gu[:, I:], atol=2e-2, rtol=2e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,bc,silu", [
    (256, 4096, 1024, 64, False), (200, 1024, 2048, 16, False), (130, 1000, 512, 32, False), (96, 3072, 1024, 32, True),
    (256, 3072, 1024, 64, True), (140, 1536, 256, 16, True), (700, 2048, 1024, 32, False),
])
def test_gemm_token_kernel_narrow_feature_tiles(ops, M, N, K, bc, silu):
    """Token-tile kernel with 16/32/64-feature tiles (large decode batches: direct epilogue, no K split)."""
    torch.manual_seed(M + N + bc)
    x, w = _rand(M, K), _rand((2 if silu else 1) * N, K, scale=0.05)
    f = ops.linear_silu_mul if silu else ops.linear
    out = f(x, w, force_mode=1, force_block_c=bc)
    ref = x.float() @ w.float().t()
    if silu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    _close(out, ref, atol=2e-2, rtol=2e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,bc,splits,silu", [
    (256, 4096, 1024, 64, 1, False), (256, 1024, 2048, 64, 4, False), (200, 1024, 3072, 32, 2, False), (130, 2048, 4096, 128, 1, False),
    (256, 3072, 1024, 64, 1, True), (96, 1536, 2048, 32, 2, True), (256, 512, 1024, 128, 1, True), (8, 256, 128, 16, 1, False),
])
def test_gemm_decode_kernel_deep_ring(ops, M, N, K, bc, splits, silu):
    """The one-CTA-per-SM variant of the weight-tile kernel (ring of ~200 KB) gives the same bits as the two-per-SM one."""
    torch.manual_seed(M + N + bc)
    x, w = _rand(M, K), _rand((2 if silu else 1) * N, K, scale=0.05)
    f = ops.linear_silu_mul if silu else ops.linear
    deep = f(x, w, force_mode=2, force_splits=splits, force_block_c=bc, force_deep=2)
    shallow = f(x, w, force_mode=2, force_splits=splits, force_block_c=bc, force_deep=1)
    ref = x.float() @ w.float().t()
    if silu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    _close(deep, ref, atol=2e-2, rtol=2e-2)
    assert torch.equal(deep, shallow)
    ops.check_status()


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (16, 1280, 1024), (50, 1024, 3200 - 3200 % 128), (64, 6400, 5120), (200, 1024, 2048), (600, 384, 256)])
def test_gemm_fp8_block_scaled(ops, M, N, K):
    """e4m3 weights with 128 x 128 block scales, activations quantised per token and 128 features."""
    from tinyllmforge_b200.ops.quant import Fp8BlockWeight, linear_fp8_ref, quantize_activations_ref
    torch.manual_seed(M + N)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    wq = Fp8BlockWeight.quantize(w)
    # the CUDA quantiser agrees with the PyTorch statement
    xq = torch.empty(M, K, dtype=torch.uint8, device="cuda")
    xs = torch.empty(K // 128, (M + 3) // 4 * 4, dtype=torch.float32, device="cuda")
    ops.C.quant_fp8(x, xq, xs)
    q_ref, s_ref = quantize_activations_ref(x)
    assert torch.allclose(xs[:, :M], s_ref, rtol=1e-6)
    assert (xq.view(torch.float8_e4m3fn).float() - q_ref.float()).abs().max() <= 32          # at most one e4m3 step at the top of the range
    out = ops.linear_fp8(x, wq)            # the e4m3 kernel itself (ops.linear expands the weight to bf16 for many tokens)
    # the GEMM itself, checked on exactly the operands it saw: the CUDA-quantised activations, dequantised in fp32
    xd = xq.view(torch.float8_e4m3fn).float().view(M, K // 128, 128) * xs[:, :M].t()[..., None]
    _close(out, xd.view(M, K) @ wq.dequantize().t(), atol=2e-2, rtol=2e-2)
    _close(out, linear_fp8_ref(x, wq), atol=0.15, rtol=5e-2)          # PyTorch quantiser may round ties differently
    exact = x.float() @ w.float().t()
    rel = (out.float() - exact).norm() / exact.norm()
    assert rel < 0.06, rel                                              # quantisation error itself stays small
    ops.check_status()


# ----------------------------------------------------------------------------- GEMMs with norm / residual fused in
@pytest.mark.parametrize("M,N,K,mode,silu", [
    (1, 4096, 1024, 0, False), (8, 4096, 1024, 2, False), (64, 4096, 1024, 0, False), (200, 4096, 1024, 0, False), (256, 6144, 4096, 0, False),
    (700, 4096, 1024, 0, False), (4096, 2048, 1024, 0, False), (5, 3072, 1024, 0, True), (16, 3072, 1024, 2, True), (100, 3072, 1024, 0, True),
    (256, 1536, 1024, 2, True), (700, 3072, 1024, 0, True), (130, 12288, 4096, 0, True), (33, 1024, 2048, 2, False),
])
def test_gemm_with_folded_input_norm(ops, M, N, K, mode, silu):
    """(x @ W'.T) * rsqrt(mean(x^2) + eps) per row, W' = W * gamma, against rms_norm(x) * gamma @ W.T in fp32; x is a residual
    stream with rows of very different magnitudes."""
    torch.manual_seed(M + N + K)
    x = (_rand(M, K).float() * torch.logspace(-1, 1.5, M, device="cuda")[:, None]).to(BF)
    gamma = (1 + 0.2 * torch.randn(K, device="cuda")).to(BF)
    w = _rand(2 * N if silu else N, K, scale=0.05)
    w_folded = (w.float() * gamma.float()[None, :]).to(BF)
    parts = (K + 127) // 128          # the sums of squares arrive in pieces of 128 features, as the producing GEMM writes them
    ssq = (x.float() ** 2).view(M, parts, -1).sum(-1).contiguous()
    got = ops.linear_scaled(x, w_folded, ssq, 1e-6, silu_mul=silu, force_mode=mode)
    xn = x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)
    want = xn @ w_folded.float().t()
    if silu:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    _close(got, want, atol=3e-2, rtol=3e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,mode,tune", [
    (1, 1024, 2048, 0, 0), (7, 1024, 3072, 0, 0), (64, 1024, 2048, 0, 0), (200, 1024, 3072, 0, 0), (256, 1024, 2048, 2, 8), (256, 4096, 12288, 0, 0),
    (33, 1024, 1024, 2, 1), (300, 1024, 2048, 0, 0), (4096, 1024, 3072, 0, 0), (1000, 4096, 4096, 0, 0), (130, 200, 72, 1, 0), (19, 136, 200, 2, 0),
    (700, 1100, 256, 1, 0), (40, 5120, 3200, 0, 0),
])
def test_gemm_with_residual_add_and_sum_of_squares(ops, M, N, K, mode, tune):
    """residual += x @ W.T in the epilogue (rounded like a bf16 GEMM followed by a bf16 add) plus the per-row sums of squares."""
    torch.manual_seed(M * 3 + N + K)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    residual = _rand(M, N, scale=2.0)
    want = ((x.float() @ w.float().t()).to(BF).float() + residual.float()).to(BF)
    parts = (N + 127) // 128
    ssq = torch.full((M, parts), float("nan"), dtype=torch.float32, device="cuda")     # every entry must be written
    res = residual.clone()
    ops.linear_residual(x, w, res, ssq, force_mode=mode, tune=tune)
    _close(res, want, atol=6e-2, rtol=2e-2)
    sq = torch.nn.functional.pad(res.float() ** 2, (0, parts * 128 - N)).view(M, parts, 128).sum(-1)
    assert torch.allclose(ssq, sq, rtol=1e-3, atol=1e-3)                               # of the values actually stored
    ssq2 = torch.empty_like(ssq)
    res2 = residual.clone()
    ops.linear_residual(x, w, res2, ssq2, force_mode=mode, tune=tune)
    assert torch.equal(res2, res) and torch.equal(ssq2, ssq)                           # no dependence on scheduling
    ops.check_status()


@pytest.mark.parametrize("M,N,K,bc,kg,silu", [
    (256, 6144, 4096, 0, 4, False), (64, 4096, 4096, 0, 4, False), (200, 4096, 12288, 0, 4, False), (16, 1280, 5120, 128, 2, False),
    (100, 5120, 3200, 0, 3, False), (256, 12288, 4096, 0, 4, True), (50, 3200, 5120, 0, 8, True), (130, 1000, 520, 64, 1, False),
    (300, 1536, 1024, 64, 2, True), (1, 256, 64, 0, 1, False), (7, 136, 4104, 128, 5, False),
])
def test_gemm_stream_k_matches_fp32(ops, M, N, K, bc, kg, silu):
    """Token-tile kernel with the (tile, K group) units dealt out evenly over the CTAs: partial tiles go through the
    scratch buffer and are summed by the CTA that arrives last."""
    torch.manual_seed(M + N + K)
    x, w = _rand(M, K), _rand(2 * N if silu else N, K, scale=0.05)
    fn = ops.linear_silu_mul if silu else ops.linear
    out = fn(x, w, force_mode=3, force_splits=kg, force_block_c=bc)
    ref_ = x.float() @ w.float().t()
    want = torch.nn.functional.silu(ref_[:, :N]) * ref_[:, N:] if silu else ref_
    _close(out, want, atol=2e-2, rtol=2e-2)
    out2 = fn(x, w, force_mode=3, force_splits=kg, force_block_c=bc)
    assert torch.equal(out, out2)                      # partial sums are added in the order of their K ranges
    ops.check_status()


@pytest.mark.parametrize("M,N,K,kg", [(256, 4096, 4096, 4), (64, 4096, 12288, 4), (130, 1024, 3072, 2), (40, 5120, 3200, 4)])
def test_gemm_stream_k_with_the_fused_epilogues(ops, M, N, K, kg):
    torch.manual_seed(M + K)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    residual = _rand(M, N, scale=2.0)
    want = ((x.float() @ w.float().t()).to(BF).float() + residual.float()).to(BF)
    parts = (N + 127) // 128
    ssq = torch.full((M, parts), float("nan"), dtype=torch.float32, device="cuda")
    res = residual.clone()
    ops.linear_residual(x, w, res, ssq, force_mode=3, tune=kg)
    _close(res, want, atol=6e-2, rtol=2e-2)
    sq = torch.nn.functional.pad(res.float() ** 2, (0, parts * 128 - N)).view(M, parts, 128).sum(-1)
    assert torch.allclose(ssq, sq, rtol=1e-3, atol=1e-3)
    res2, ssq2 = residual.clone(), torch.empty_like(ssq)
    ops.linear_residual(x, w, res2, ssq2, force_mode=3, tune=kg)
    assert torch.equal(res2, res) and torch.equal(ssq2, ssq)
    # folded input norm as a row scale
    pk = (K + 127) // 128
    ssq_in = (x.float() ** 2).view(M, pk, -1).sum(-1).contiguous()
    got = ops.linear_scaled(x, w, ssq_in, 1e-6, force_mode=3, tune=kg)
    xn = x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)
    _close(got, xn @ w.float().t(), atol=3e-2, rtol=3e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,kg,silu", [
    (256, 256, 64, 0, False), (512, 512, 256, 0, False), (256, 6144, 4096, 0, False), (256, 6144, 4096, 4, False), (8192, 4096, 1024, 0, False),
    (200, 4096, 4096, 4, False), (100, 1280, 5120, 2, False), (1000, 1100, 520, 0, False), (700, 1100, 520, 3, False), (4096, 3072, 1024, 0, True),
    (256, 12288, 4096, 4, True), (130, 1536, 1024, 2, True), (300, 200, 72, 0, True), (1, 128, 64, 0, False),
])
def test_gemm_cta_pair_kernel_matches_fp32(ops, M, N, K, kg, silu):
    """One 256 x 256 UMMA per pair of SMs (cta_group::2): each CTA loads its 128 tokens and half of the weight rows."""
    torch.manual_seed(M + N + K)
    x, w = _rand(M, K), _rand(2 * N if silu else N, K, scale=0.05)
    fn = ops.linear_silu_mul if silu else ops.linear
    out = fn(x, w, force_mode=4, force_splits=kg)
    ref_ = x.float() @ w.float().t()
    want = torch.nn.functional.silu(ref_[:, :N]) * ref_[:, N:] if silu else ref_
    _close(out, want, atol=2e-2, rtol=2e-2)
    assert torch.equal(out, fn(x, w, force_mode=4, force_splits=kg))
    ops.check_status()


@pytest.mark.parametrize("M,N,K,kg", [(256, 4096, 4096, 4), (2048, 1024, 3072, 0), (130, 1024, 3072, 2)])
def test_gemm_cta_pair_kernel_with_the_fused_epilogues(ops, M, N, K, kg):
    torch.manual_seed(M + K)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    residual = _rand(M, N, scale=2.0)
    want = ((x.float() @ w.float().t()).to(BF).float() + residual.float()).to(BF)
    parts = (N + 127) // 128
    ssq = torch.full((M, parts), float("nan"), dtype=torch.float32, device="cuda")
    res = residual.clone()
    ops.linear_residual(x, w, res, ssq, force_mode=4, tune=kg)
    _close(res, want, atol=6e-2, rtol=2e-2)
    sq = torch.nn.functional.pad(res.float() ** 2, (0, parts * 128 - N)).view(M, parts, 128).sum(-1)
    assert torch.allclose(ssq, sq, rtol=1e-3, atol=1e-3)
    pk = (K + 127) // 128
    ssq_in = (x.float() ** 2).view(M, pk, -1).sum(-1).contiguous()
    got = ops.linear_scaled(x, w, ssq_in, 1e-6, force_mode=4, tune=kg)
    xn = x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)
    _close(got, xn @ w.float().t(), atol=3e-2, rtol=3e-2)
    ops.check_status()


@pytest.mark.parametrize("M,N,K,silu", [(600, 1280, 1024, False), (2048, 3200, 5120, True), (1000, 5120, 3200, False)])
def test_fp8_weights_with_many_tokens_are_expanded_and_multiplied_in_bf16(ops, M, N, K, silu):
    """Prefill-sized GEMM on a block-scaled e4m3 weight: the weight is expanded to bf16 (exactly: e4m3 x scale rounded to
    bf16) right before the bf16 GEMM, which must not read it early; activations are not quantised."""
    from tinyllmforge_b200.ops.quant import Fp8BlockWeight
    torch.manual_seed(N + K)
    w = _rand(2 * N if silu else N, K, scale=0.05)
    wq = Fp8BlockWeight.quantize(w)
    wd = wq.dequantize()
    assert torch.equal(ops._expand_fp8(wq), wd.to(BF))
    for seed in range(3):                              # the scratch buffer is overwritten between calls
        x = _rand(M, K)
        got = (ops.linear_silu_mul if silu else ops.linear)(x, wq)
        ref_ = x.float() @ wd.to(BF).float().t()
        want = torch.nn.functional.silu(ref_[:, :N]) * ref_[:, N:] if silu else ref_
        _close(got, want, atol=2e-2, rtol=2e-2)
        other = Fp8BlockWeight.quantize(_rand(2 * N if silu else N, K, scale=0.05))
        ops._expand_fp8(other)
    ops.check_status()


@pytest.mark.parametrize("mode", [5, 6])
@pytest.mark.parametrize("M,N,K,S,silu", [
    (256, 4096, 4096, 4, False), (64, 6144, 4096, 6, False), (200, 4096, 12288, 4, False), (16, 1280, 5120, 8, False),
    (100, 5120, 3200, 3, False), (130, 1536, 4096, 4, True), (50, 3200, 5120, 2, True), (7, 136, 4104, 5, False), (300, 1000, 2048, 2, False),
])
def test_gemm_split_k_with_reduce_kernel(ops, M, N, K, S, silu, mode):
    """K split S ways, one (tile, K range) per CTA or CTA pair; a second kernel adds the partial tiles and runs the epilogue."""
    torch.manual_seed(M + N + K)
    x, w = _rand(M, K), _rand(2 * N if silu else N, K, scale=0.05)
    fn = ops.linear_silu_mul if silu else ops.linear
    out = fn(x, w, force_mode=mode, force_splits=S)
    ref_ = x.float() @ w.float().t()
    want = torch.nn.functional.silu(ref_[:, :N]) * ref_[:, N:] if silu else ref_
    _close(out, want, atol=2e-2, rtol=2e-2)
    assert torch.equal(out, fn(x, w, force_mode=mode, force_splits=S))
    ops.check_status()


@pytest.mark.parametrize("mode", [5, 6])
@pytest.mark.parametrize("M,N,K,S", [(256, 4096, 4096, 4), (64, 4096, 12288, 8), (130, 1024, 3072, 2), (40, 5120, 3200, 4)])
def test_gemm_split_k_with_reduce_kernel_and_fused_epilogues(ops, M, N, K, S, mode):
    torch.manual_seed(M + K)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    residual = _rand(M, N, scale=2.0)
    want = ((x.float() @ w.float().t()).to(BF).float() + residual.float()).to(BF)
    parts = (N + 127) // 128
    ssq = torch.full((M, parts), float("nan"), dtype=torch.float32, device="cuda")
    res = residual.clone()
    ops.linear_residual(x, w, res, ssq, force_mode=mode, tune=S)
    _close(res, want, atol=6e-2, rtol=2e-2)
    sq = torch.nn.functional.pad(res.float() ** 2, (0, parts * 128 - N)).view(M, parts, 128).sum(-1)
    assert torch.allclose(ssq, sq, rtol=1e-3, atol=1e-3)
    res2, ssq2 = residual.clone(), torch.empty_like(ssq)
    ops.linear_residual(x, w, res2, ssq2, force_mode=mode, tune=S)
    assert torch.equal(res2, res) and torch.equal(ssq2, ssq)
    pk = (K + 127) // 128
    ssq_in = (x.float() ** 2).view(M, pk, -1).sum(-1).contiguous()
    got = ops.linear_scaled(x, w, ssq_in, 1e-6, force_mode=mode, tune=S)
    xn = x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)
    _close(got, xn @ w.float().t(), atol=3e-2, rtol=3e-2)
    ops.check_status()


@pytest.mark.parametrize("T,K,nq,nkv,bs,folded", [(64, 1024, 16, 8, 256, True), (256, 1024, 16, 8, 256, False), (33, 4096, 32, 8, 16, True),
                                                 (200, 512, 8, 1, 64, False), (1, 256, 4, 2, 256, True)])
def test_qkv_gemm_with_norm_rope_and_cache_store_in_its_epilogue(ops, T, K, nq, nkv, bs, folded):
    """The qkv projection whose epilogue normalises q and k per head, rotates them and writes k / v into the paged cache,
    against the fp32 statement of the same chain (projection rounded to bf16, then q/k-norm + RoPE + store)."""
    torch.manual_seed(T + K)
    D, nblk = 128, 8 + T // bs
    x = _rand(T, K)
    w = _rand((nq + 2 * nkv) * D, K, scale=0.05)
    qw, kw = _rand(D, scale=0.2) + 1, _rand(D, scale=0.2) + 1
    table = ref.rope_table(4096, D, 1e6, "cuda")
    pos = torch.randint(0, 4096, (T,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(nblk * bs, device="cuda")[:T].to(torch.int32)
    if T > 2:
        slots[1] = -1
    kc, vc = torch.zeros(nblk, nkv, bs, D, dtype=BF, device="cuda"), torch.zeros(nblk, nkv, bs, D, dtype=BF, device="cuda")
    kc2, vc2 = kc.clone(), vc.clone()
    ssq = None
    proj = x.float() @ w.float().t()
    if folded:
        parts = (K + 127) // 128
        ssq = (x.float() ** 2).view(T, parts, -1).sum(-1).contiguous()
        proj = proj * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6)
    q = ops.linear_qkv_rope_store(x, w, ssq, 1e-6, qw, kw, 1e-6, table, pos, slots, kc, vc, nq, nkv)
    q_want = ref.qk_norm_rope_store(proj.to(BF), qw, kw, 1e-6, table, pos, slots, kc2, vc2, nq, nkv, D)
    _close(q, q_want, 3e-2, 3e-2)
    _close(kc, kc2, 3e-2, 3e-2)
    _close(vc, vc2, 2e-2, 2e-2)
    if T > 2:
        assert torch.count_nonzero(kc) == torch.count_nonzero(kc2)          # the row with slot -1 was not stored
    ops.check_status()


@pytest.mark.parametrize("T,K,nq,nkv,bs,folded", [(257, 1024, 16, 8, 256, True), (511, 512, 5, 1, 64, False), (1025, 4096, 32, 8, 256, True),
                                                 (3000, 256, 3, 3, 16, True), (700, 1024, 2, 1, 128, False)])
def test_qkv_gemm_of_prompts_with_norm_rope_and_cache_store_in_its_epilogue(ops, T, K, nq, nkv, bs, folded):
    """More than 256 rows: CTA pairs, two heads per tile (q and k, k and v in one tile; an odd number of heads; ragged last rows)."""
    test_qkv_gemm_with_norm_rope_and_cache_store_in_its_epilogue(ops, T, K, nq, nkv, bs, folded)


@pytest.mark.parametrize("folded", [True, False])
@pytest.mark.parametrize("T,K,nq,nkv", [(300, 2048, 16, 8), (1500, 4096, 5, 1), (2000, 4096, 16, 4), (700, 2560, 8, 2)])
def test_qkv_gemm_of_prompts_gives_the_bits_of_the_two_kernels(ops, T, K, nq, nkv, folded):
    """With the input norm folded in (one GPU) and without it (ranks of several, which hold a part of the heads)."""
    torch.manual_seed(T)
    x, w = _rand(T, K), _rand((nq + 2 * nkv) * 128, K, scale=0.05)
    qw, kw = _rand(128, scale=0.2) + 1, _rand(128, scale=0.2) + 1
    ssq = (x.float() ** 2).view(T, K // 128, -1).sum(-1).contiguous() if folded else None
    table = ref.rope_table(4096, 128, 1e6, "cuda")
    pos = torch.randint(0, 4096, (T,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(2048, device="cuda")[:T].to(torch.int32)
    caches = [torch.zeros(8, nkv, 256, 128, dtype=BF, device="cuda") for _ in range(4)]
    got = ops.linear_qkv_rope_store(x, w, ssq, 1e-6, qw, kw, 1e-6, table, pos, slots, caches[0], caches[1], nq, nkv)
    proj = ops.linear_scaled(x, w, ssq, 1e-6) if folded else ops.linear(x, w)
    want = ops.qk_norm_rope_store(proj, qw, kw, 1e-6, table, pos, slots, caches[2], caches[3], nq, nkv, 128)
    assert torch.equal(got.view(-1), want.view(-1)) and torch.equal(caches[0], caches[2]) and torch.equal(caches[1], caches[3])
    ops.check_status()


def test_qkv_gemm_route_of_prompts(ops):
    """One kernel where pairs have several tiles each (74 pairs; hidden sizes from 4096) or many (2560); two kernels else, as for fp8 weights."""
    weight = lambda heads, hidden: torch.empty(heads * 128, hidden, dtype=BF, device="meta")
    route = lambda rows, heads, hidden: ops.qkv_rope_store_in_gemm(rows, 128, weight(heads, hidden), True)
    assert route(3777, 48, 4096) and route(1024, 48, 4096) and route(2048, 24, 4096) and route(3777, 48, 2560) and route(8192, 6, 4096)
    assert not (route(300, 48, 4096) or route(768, 48, 4096) or route(1024, 24, 4096) or route(3777, 6, 4096) or route(1500, 48, 2560))
    assert not (route(200, 48, 4096) or route(16000, 32, 2048) or route(16000, 32, 1024) or ops.qkv_rope_store_in_gemm(3777, 64, weight(48, 4096), True))


def test_embedding_sum_of_squares(ops):
    V, H, T = 512, 1024, 37
    table = _rand(V, H)
    ids = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    out, ssq, scratch = ops.embedding_ssq(ids, table, 0)
    assert torch.equal(out, table[ids.long()])
    assert ssq.shape == (T, H // 128) == scratch.shape
    assert torch.allclose(ssq.sum(-1), (out.float() ** 2).sum(-1), rtol=1e-4)
    assert torch.count_nonzero(ssq[:, 1:]) == 0


def test_gemm_strided_input(ops):
    big = _rand(64, 3 * 256)
    x = big[:, 256:512]          # row stride 768, 16-byte aligned start
    w = _rand(128, 256, scale=0.05)
    _close(ops.linear(x, w), x.float() @ w.float().t(), 2e-2, 2e-2)


# ----------------------------------------------------------------------------- norms / activation / gathers
@pytest.mark.parametrize("rows,H", [(1, 1024), (37, 1024), (5, 4096), (3, 5120), (2, 256), (4, 8192)])
def test_rms_norm(ops, rows, H):
    x, w = _rand(rows, H), _rand(H, scale=0.3) + 1
    _close(ops.rms_norm(x, w, 1e-6), ref.rms_norm(x, w, 1e-6), 1e-2, 1e-2)


@pytest.mark.parametrize("rows,H", [(1, 1024), (33, 1024), (6, 4096), (3, 5120)])
def test_add_rms_norm(ops, rows, H):
    x, r, w = _rand(rows, H), _rand(rows, H), _rand(H, scale=0.3) + 1
    want_y, want_r = ref.add_rms_norm(x, r, w, 1e-6)
    r2 = r.clone()
    y, r_out = ops.add_rms_norm(x, r2, w, 1e-6)
    assert r_out.data_ptr() == r2.data_ptr()
    assert torch.equal(r_out, want_r)
    _close(y, want_y, 1e-2, 1e-2)


def test_silu_mul(ops):
    x = _rand(77, 2 * 3072, scale=2.0)
    _close(ops.silu_mul(x), ref.silu_mul(x), 1e-2, 1e-2)


def test_embedding_shard_and_gather(ops):
    w = _rand(1000, 1024)
    ids = torch.tensor([0, 999, 1000, 1500, 2000, 1234], dtype=torch.int32, device="cuda")
    got = ops.embedding(ids, w, 1000)
    assert torch.equal(got, ref.embedding(ids, w, 1000))
    idx = torch.tensor([5, 0, 3], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.select_rows(got, idx), got[idx.long()])


# ----------------------------------------------------------------------------- q/k norm + rope + KV store
@pytest.mark.parametrize("T,nq,nkv,bs", [(1, 16, 8, 256), (50, 16, 8, 16), (9, 4, 1, 64)])
def test_qk_norm_rope_store(ops, T, nq, nkv, bs):
    D, nblk = 128, 8
    qkv = _rand(T, (nq + 2 * nkv) * D)
    qw, kw = _rand(D, scale=0.2) + 1, _rand(D, scale=0.2) + 1
    table = ref.rope_table(4096, D, 1e6, "cuda")
    pos = torch.randint(0, 4096, (T,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(nblk * bs, device="cuda")[:T].to(torch.int32)
    if T > 2:
        slots[1] = -1
    kc, vc = torch.zeros(nblk, nkv, bs, D, dtype=BF, device="cuda"), torch.zeros(nblk, nkv, bs, D, dtype=BF, device="cuda")
    kc2, vc2 = kc.clone(), vc.clone()
    q = ops.qk_norm_rope_store(qkv, qw, kw, 1e-6, table, pos, slots, kc, vc, nq, nkv, D)
    q_want = ref.qk_norm_rope_store(qkv, qw, kw, 1e-6, table, pos, slots, kc2, vc2, nq, nkv, D)
    _close(q, q_want, 2e-2, 2e-2)
    _close(kc, kc2, 2e-2, 2e-2)
    assert torch.equal(vc, vc2)
    ops.check_status()


def test_qk_norm_rope_store_rounds_in_a_fixed_order(ops):
    """A head's bits: sums of squares as sum + (a^2 + b^2), an eight-element run per lane, then a tree over eight lanes; rotation as
    x1 c - round(x2 s) and x1 s + round(x2 c).  Products of bf16 numbers are exact in fp32 and those with a table entry in 64 bits, so both
    can be stated exactly; another order differs in a few of the 16 million elements (3 to 6 for the sums, over 120 for the rotation)."""
    T, nq, nkv = 8192, 16, 8
    torch.manual_seed(0)
    qkv = _rand(T, (nq + 2 * nkv) * 128)
    w = _rand(128, scale=0.2) + 1
    table = ref.rope_table(4096, 128, 1e6, "cuda")
    pos = torch.randint(0, 4096, (T,), dtype=torch.int32, device="cuda")
    slots = torch.arange(T, dtype=torch.int32, device="cuda")
    kc, vc = torch.zeros(32, nkv, 256, 128, dtype=BF, device="cuda"), torch.zeros(32, nkv, 256, 128, dtype=BF, device="cuda")
    x = qkv.view(T, -1, 128)[:, :nq].float()
    squares = (x * x).view(T, nq, 2, 8, 8)
    sums = torch.zeros(T, nq, 8, device="cuda")
    for e in range(8):
        sums = sums + (squares[:, :, 0, :, e] + squares[:, :, 1, :, e])
    for step in (1, 2, 4):
        sums = sums + sums[..., [i ^ step for i in range(8)]]
    normed = (x * torch.rsqrt(sums[..., :1] / 128 + 1e-6)).to(BF).float() * w.float()
    got = ops.qk_norm_rope_store(qkv, w, w, 1e-6, table, pos, slots, kc, vc, nq, nkv, 128, do_rope=False)
    assert torch.equal(got, normed.to(BF))
    x1, x2 = x[..., :64].double(), x[..., 64:].double()
    c, s = table[pos.long()][:, None].double().split(64, -1)
    want = torch.cat([x1 * c - (x2 * s).float().double(), x1 * s + (x2 * c).float().double()], -1).float().to(BF)
    got = ops.qk_norm_rope_store(qkv, None, None, 1e-6, table, pos, slots, kc, vc, nq, nkv, 128)
    assert torch.equal(got, want)
    ops.check_status()


# ----------------------------------------------------------------------------- attention
class _Batch:
    pass


def _paged_case(q_lens, k_lens, nq, nkv, bs, seed=0):
    torch.manual_seed(seed)
    D = 128
    S = len(q_lens)
    nblk_per = [-(-k // bs) for k in k_lens]
    total = sum(nblk_per) + 3
    perm = torch.randperm(total).tolist()
    width = max(nblk_per) + 1
    bt = torch.full((S, width), -1, dtype=torch.int32)
    p = 0
    for s, n in enumerate(nblk_per):
        bt[s, :n] = torch.tensor(perm[p:p + n], dtype=torch.int32)
        p += n
    kc, vc = _rand(total, nkv, bs, D), _rand(total, nkv, bs, D)
    T = sum(q_lens)
    q = _rand(T, nq, D)
    b = _Batch()
    b.cu_seqlens_q = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device="cuda")
    b.context_lens = torch.tensor(k_lens, dtype=torch.int32, device="cuda")
    b.block_tables = bt.cuda()
    b.num_seqs = b.padded_seqs = S
    b.max_seqlen_q, b.max_seqlen_k = max(q_lens), max(k_lens)
    b.table_width = width
    return q, kc, vc, b


@pytest.mark.parametrize("mode", ["flat", "chunked"])
@pytest.mark.parametrize("k_lens,nq,nkv,bs", [
    ([1], 16, 8, 256), ([5, 300, 64, 1000], 16, 8, 256), ([17, 33, 250], 8, 2, 16), ([700, 2011, 129], 32, 8, 256),
    ([40, 90], 8, 8, 32), ([513, 77], 8, 1, 64), ([300, 1000, 70, 2], 40, 8, 256), ([129, 640, 33], 64, 8, 256), ([50, 400], 6, 2, 64), ([700, 2011, 129], 8, 1, 256),
    ([300, 65, 2], 10, 1, 64), ([700, 129], 24, 2, 256), ([500, 1], 15, 1, 128), ([64, 513], 32, 2, 256),          # groups over 8: slices of 5 and 4 heads
])
def test_decode_attention(ops, k_lens, nq, nkv, bs, mode, monkeypatch):
    monkeypatch.setattr(ops, "decode_attention_mode", mode)
    q, kc, vc, b = _paged_case([1] * len(k_lens), k_lens, nq, nkv, bs)
    b.is_prefill = False
    got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("mode", ["flat", "chunked"])
def test_decode_attention_reports_a_length_the_block_table_cannot_describe(ops, mode, monkeypatch):
    """A context length written too large on the host (one block more than the table has) is clamped on the device: the
    status word gets the bad-index bit, every access stays inside the table and the scratch, the other rows are right."""
    monkeypatch.setattr(ops, "decode_attention_mode", mode)
    k_lens = [300, 100, 520]
    q, kc, vc, b = _paged_case([1] * 3, k_lens, 16, 8, 256)
    b.is_prefill = False
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, 3)
    b.context_lens = b.context_lens.clone()
    b.context_lens[1] = (b.table_width + 1) * 256
    b.block_tables = b.block_tables.clone()
    b.block_tables[1, 1:] = b.block_tables[1, 0]        # the clamped row reads valid blocks; its result is not checked
    ops.check_status()
    got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    torch.cuda.synchronize()
    word = int(ops.status[0].item())
    assert word & 4, word
    ops.status.zero_()
    _close(got[[0, 2]], want[[0, 2]], 2e-2, 2e-2)


@pytest.mark.parametrize("mode", ["flat", "chunked"])
def test_decode_attention_padding_rows(ops, mode, monkeypatch):
    monkeypatch.setattr(ops, "decode_attention_mode", mode)
    q, kc, vc, b = _paged_case([1, 1, 1], [100, 0, 7], 16, 8, 256)
    b.is_prefill = False
    got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    assert torch.count_nonzero(got[1]) == 0
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, 3)
    _close(got[[0, 2]], want[[0, 2]], 2e-2, 2e-2)


@pytest.mark.parametrize("mode", ["flat", "chunked"])
@pytest.mark.parametrize("k_lens,nq,nkv,bs", [
    ([1, 2, 64, 65, 300, 1000, 0, 256, 257, 512], 16, 8, 256), ([17, 33, 250, 16, 1], 8, 2, 16), ([700, 2011, 129, 128], 32, 8, 256),
    ([40, 90, 64], 8, 8, 32), ([513, 77], 8, 1, 64), (list(range(1, 140, 3)), 16, 8, 128), ([300, 1000, 70, 2], 40, 8, 256),
    ([129, 640, 33], 64, 8, 256), ([300, 0, 64], 10, 1, 64), ([129, 500], 32, 2, 256),
])
def test_decode_attention_from_raw_qkv(ops, k_lens, nq, nkv, bs, mode, monkeypatch):
    """q/k-norm + rotation + KV store inside the attention kernel == qk_norm_rope_store followed by attention:
    same output, same cache contents (the step's token of every sequence sits at position len - 1)."""
    monkeypatch.setattr(ops, "decode_attention_mode", mode)
    S, D = len(k_lens), 128
    _, kc, vc, b = _paged_case([1] * S, [max(k, 1) for k in k_lens], nq, nkv, bs, seed=7)
    b.context_lens = torch.tensor(k_lens, dtype=torch.int32, device="cuda")
    b.is_prefill = False
    torch.manual_seed(11)
    qkv = _rand(S, (nq + 2 * nkv) * D)
    qw, kw = _rand(D, scale=0.2) + 1, _rand(D, scale=0.2) + 1
    table = ref.rope_table(4096, D, 1e6, "cuda")
    lens = b.context_lens.long()
    pos = (lens - 1).clamp(min=0).to(torch.int32)
    blk = b.block_tables.long()[torch.arange(S), ((lens - 1).clamp(min=0) // bs).cpu()]
    slots = torch.where(lens > 0, blk.cuda() * bs + (lens - 1) % bs, torch.full_like(lens, -1)).to(torch.int32)
    kc1, vc1, kc2, vc2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    q = ops.qk_norm_rope_store(qkv, qw, kw, 1e-6, table, pos, slots, kc1, vc1, nq, nkv, D)
    want = ops.attention(q, kc1, vc1, b, D ** -0.5)
    got = ops.decode_attention_qkv(qkv, qw, kw, 1e-6, table, kc2, vc2, b, nq, D ** -0.5)
    live = [i for i, n in enumerate(k_lens) if n > 0]
    _close(got[live], want[live], 2e-2, 2e-2)
    _close(kc2, kc1, 1e-2, 1e-2)
    assert torch.equal(vc2, vc1)
    for i, n in enumerate(k_lens):
        if n == 0:
            assert torch.count_nonzero(got[i]) == 0
    ops.check_status()


@pytest.mark.parametrize("nq,nkv", [(8, 8), (16, 8), (24, 8), (32, 8), (40, 8), (64, 8), (2, 1), (5, 1)])
def test_decode_attention_with_chunks_longer_than_asked_for(ops, nq, nkv, monkeypatch):
    """One sequence of 2000 tokens under a table for more, from ready queries and from the raw projection."""
    test_decode_attention_from_raw_qkv(ops, [2000], nq, nkv, 256, "chunked", monkeypatch)
    test_decode_attention(ops, [2000], nq, nkv, 256, "chunked", monkeypatch)


@pytest.mark.parametrize("nq", [32, 64])
def test_decode_attention_from_raw_qkv_over_a_list_of_chunks(ops, nq, monkeypatch):
    """More possible chunks than two waves of CTAs: each walks the list of live ones, several in a row, through one ring."""
    k_lens = [(1 + 977 * i) % 4000 for i in range(32)]
    k_lens[5] = k_lens[31] = 0
    test_decode_attention_from_raw_qkv(ops, k_lens, nq, 8, 256, "chunked", monkeypatch)


@pytest.mark.parametrize("k_lens,nq,nkv", [([300, 1000, 70, 2], 32, 8), ([129, 640, 33, 2011], 40, 8), ([50, 400, 900], 8, 2)])
def test_decode_attention_cuda_core_variant_for_groups_of_4_and_5(ops, k_lens, nq, nkv, monkeypatch):
    """The flat kernel runs groups of 4..8 q heads per KV head on the tensor cores by default (covered by the tests above); the
    CUDA-core kernel stays selectable for them and must agree too."""
    monkeypatch.setattr(ops, "decode_attention_mode", "flat")
    q, kc, vc, b = _paged_case([1] * len(k_lens), k_lens, nq, nkv, 256)
    b.is_prefill = False
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    ops.C.decode_attention_set_tc_min_group(9)
    try:
        got = ops.attention(q, kc, vc, b, 128 ** -0.5)
        torch.cuda.synchronize()
    finally:
        ops.C.decode_attention_set_tc_min_group(4)
    _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("k_lens,nq,nkv,bs,chunk,max_chunks", [
    ([1, 63, 64, 65, 0, 128, 129, 700], 32, 8, 256, 64, 16),           # edges of tiles and chunks, a padding row, every sequence cut
    ([2000, 5], 8, 2, 64, 64, 32),                                     # few sequences: fewer and longer chunks than asked for
    ([9000], 4, 1, 256, 64, 141), ([9000], 2, 1, 256, 64, 141), ([20000, 3000], 5, 1, 512, 64, 313),      # more than 24 of them
    ([9000, 1, 700, 3000], 32, 8, 256, 64, 141), ([9000, 1, 700, 3000], 16, 8, 256, 64, 141),             # more than 128 to merge
    ([0, 640, 641, 1], 10, 2, 128, 128, 6), ([300, 511], 12, 2, 256, 64, 8), ([300, 511], 7, 1, 256, 256, 2), ([900] * 3, 16, 2, 512, 1024, 1),
    ([17 * i % 900 for i in range(70)], 32, 8, 256, 64, 15),           # more items than two waves: walked as a list, three ballots of sequences
])
def test_decode_attention_chunks_on_tensor_cores(ops, k_lens, nq, nkv, bs, chunk, max_chunks):
    """Groups of 4 to 8 heads (and one of 2); weights and sums are fp32, so what is left is the rounding of the bf16 result (2^-9 of values of unit size)."""
    q, kc, vc, b = _paged_case([1] * len(k_lens), k_lens, nq, nkv, bs, seed=4)
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    B = len(k_lens)
    part_o = torch.full((B * nq * max_chunks * 128,), float("nan"), device="cuda")
    part_ml = torch.full((B * nq * max_chunks * 2,), float("nan"), device="cuda")
    got = torch.full((B, nq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.C.decode_attention(q, kc, vc, b.block_tables, b.context_lens, got, part_o, part_ml, chunk, max_chunks, 128 ** -0.5, ops.status)
    for i, n in enumerate(k_lens):
        if n == 0:
            assert torch.count_nonzero(got[i]) == 0
        else:
            _close(got[i], want.view(B, -1)[i], 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("k_lens,nq,nkv", [([700, 5, 300], 16, 8), ([700, 5, 300], 32, 8), ([1500], 8, 8)])
def test_decode_attention_with_a_scratch_that_begins_anywhere(ops, k_lens, nq, nkv):
    """Views at an odd number of floats from an aligned address, few and more than eight chunks to merge."""
    q, kc, vc, b = _paged_case([1] * len(k_lens), k_lens, nq, nkv, 256, seed=8)
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    for chunk in (64, 256):
        max_chunks = -(-max(k_lens) // chunk)
        need = len(k_lens) * nq * max_chunks
        part_o, part_ml = torch.empty(need * 128 + 1, device="cuda")[1:], torch.empty(need * 2 + 1, device="cuda")[1:]
        got = torch.empty(len(k_lens), nq * 128, dtype=BF, device="cuda")
        ops.C.decode_attention(q, kc, vc, b.block_tables, b.context_lens, got, part_o, part_ml, chunk, max_chunks, 128 ** -0.5, ops.status)
        _close(got, want.view_as(got), 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("nq,nkv", [(16, 8), (32, 8), (40, 8), (64, 8)])
@pytest.mark.parametrize("n,chunk", [(4500, 256), (30000, 1536)])
def test_decode_attention_keeps_weights_and_sums_in_fp32(ops, nq, nkv, n, chunk):
    """The partial results of chunks, which are fp32, against 64 bits: values without a common direction, so that sums of some hundred weights of
    like size nearly cancel and an error of 2^-24 in each shows.  Multiply-adds of fp32 numbers give 2.1e-7 for 256 tokens, 3.9e-7 for 1536
    (and 1.5e-7, 2.3e-7 in the logarithm of the sums); weights of 16 bits would give 1.7e-6."""
    q, kc, vc, b = _paged_case([1, 1], [n, n], nq, nkv, 256, seed=10)
    parts = -(-n // chunk)
    part_o, part_ml = torch.empty(2 * nq * parts * 128, device="cuda"), torch.empty(2 * nq * parts * 2, device="cuda")
    out = torch.empty(2, nq * 128, dtype=BF, device="cuda")
    ops.C.decode_attention(q, kc, vc, b.block_tables, b.context_lens, out, part_o, part_ml, chunk, parts, 128 ** -0.5, ops.status)
    error = size = 0.0
    for s in range(2):
        at = b.block_tables[s, :-(-n // 256)].long()
        k, v = (c[at].transpose(0, 1).reshape(nkv, -1, 128)[:, :n].double() for c in (kc, vc))
        scores = q[s].double().view(nkv, -1, 128) @ k.transpose(1, 2) * (128 ** -0.5 * math.log2(math.e))
        for c in range(parts):
            here = scores[..., c * chunk:(c + 1) * chunk]
            want = torch.softmax(here * math.log(2), -1) @ v[:, c * chunk:(c + 1) * chunk]
            got = part_o.view(2, nkv, -1, parts, 128)[s, :, :, c].double()
            error, size = error + (got - want).square().sum(), size + want.square().sum()
            ml = part_ml.view(2, nkv, -1, parts, 2)[s, :, :, c].double()
            assert (torch.log2(ml[..., 1]) + ml[..., 0] - torch.logsumexp(here * math.log(2), -1) / math.log(2)).square().mean().sqrt() < 3e-7
    assert (error / size).sqrt() < 5e-7
    ops.check_status()


@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("k_lens,nq,nkv", [([300, 64, 1000, 1], 16, 8), ([300, 64, 1000, 1], 32, 8), ([700, 129], 10, 2), ([500, 90], 8, 1)])
def test_decode_attention_with_infinite_values(ops, k_lens, nq, nkv, raw):
    """An infinite value under a positive weight makes an infinite sum, two of opposite signs, or a NaN, make a NaN; all other elements are what
    they are without.  Among the values of cached tokens and of the newest one."""
    S = len(k_lens)
    q, kc, vc, b = _paged_case([1] * S, k_lens, nq, nkv, 256, seed=9)
    b.is_prefill = False
    qkv = _rand(S, (nq + 2 * nkv) * 128)
    put = lambda s, tok, d, value: vc[int(b.block_tables[s, tok // 256]), :, tok % 256, d].fill_(value)
    put(0, 5, 7, math.inf), put(0, 200, 8, -math.inf), put(0, 70, 100, math.inf), put(0, 130, 100, -math.inf), put(0, 131, 99, math.nan)
    for s, n in enumerate(k_lens):
        put(s, n // 2, 20, math.inf)
        qkv[s, (nq + nkv) * 128 + 21] = math.inf                     # the newest token's, first KV head
    if raw:
        slots = torch.stack([b.block_tables[s, (n - 1) // 256] * 256 + (n - 1) % 256 for s, n in enumerate(k_lens)]).to(torch.int32)
        table = ref.rope_table(4096, 128, 1e6, "cuda")
        pos = b.context_lens - 1
        kc1, vc1 = kc.clone(), vc.clone()
        q1 = ops.qk_norm_rope_store(qkv, None, None, 1e-6, table, pos, slots, kc1, vc1, nq, nkv, 128)
        want = ref.attention(q1, kc1, vc1, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, S)
        got = ops.decode_attention_qkv(qkv, None, None, 1e-6, table, kc, vc, b, nq, 128 ** -0.5)
    else:
        want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, S)
        got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    got, want = got.view_as(want).float(), want.float()
    finite = torch.isfinite(want)
    assert (~finite).sum() > 2 * nq and torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[got.isinf()], want[want.isinf()]) and torch.equal(got.isinf(), want.isinf())
    _close(got[finite], want[finite], 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("k_lens,nkv", [([2000], 8), ([200 + 131 * i for i in range(13)], 8), ([3000, 70], 1)])
def test_decode_attention_that_keeps_its_order(ops, k_lens, nkv, raw, monkeypatch):
    """Models with fp8 weights: four heads per KV head bit for bit as two pairs of them, which always run on the CUDA cores, and in chunks of
    exactly the size that batch and KV heads ask for, whatever the group."""
    B = len(k_lens)
    q, kc, vc, b = _paged_case([1] * B, k_lens, 4 * nkv, nkv, 256, seed=12)
    b.is_prefill = False
    qkv = _rand(B, 6 * nkv * 128)
    monkeypatch.setattr(ops, "decode_attention_mode", "chunked")
    monkeypatch.setattr(ops, "decode_keep_order", True)
    def run(heads):
        if not raw:
            return ops.attention(q.view(B, nkv, 4, 128)[:, :, heads].reshape(B, -1, 128).contiguous(), kc, vc, b, 128 ** -0.5)
        part = qkv.view(B, 6 * nkv, 128)
        part = torch.cat([part[:, :4 * nkv].view(B, nkv, 4, 128)[:, :, heads].reshape(B, -1, 128), part[:, 4 * nkv:]], 1).reshape(B, -1).contiguous()
        return ops.decode_attention_qkv(part, None, None, 1e-6, None, kc, vc, b, len(heads) * nkv, 128 ** -0.5, do_rope=False)
    whole = run([0, 1, 2, 3]).view(B, nkv, 4, 128)
    for pair in ([0, 1], [2, 3]):
        assert torch.equal(run(pair).view(B, nkv, 2, 128), whole[:, :, pair])
    chunk = decode_chunking(B, nkv, 256, b.table_width * 256)[0]
    assert chunk == (64 if B * nkv < 16 else 256)
    chunks = -(-max(k_lens) // chunk)
    part_o, part_ml = torch.empty(B * 4 * nkv * chunks * 128, device="cuda"), torch.full((B * 4 * nkv * chunks * 2,), float("nan"), device="cuda")
    out = torch.empty(B, 4 * nkv * 128, dtype=BF, device="cuda")
    ops.C.decode_attention(q, kc, vc, b.block_tables, b.context_lens, out, part_o, part_ml, chunk, chunks, 128 ** -0.5, ops.status, True)
    for s, n in enumerate(k_lens):
        live = -(-n // chunk)
        if live > 1:
            assert not torch.isnan(part_ml.view(B, 4 * nkv, chunks, 2)[s, :, :live]).any() and torch.isnan(part_ml.view(B, 4 * nkv, chunks, 2)[s, :, live:]).all()
    if not raw:
        assert torch.equal(out, whole.reshape(B, -1))
    ops.check_status()


@pytest.mark.parametrize("nq,nkv", [(16, 8), (32, 8)])
def test_decode_attention_refuses_a_cache_that_is_not_aligned(ops, nq, nkv):
    """Every kernel copies cache rows 16 bytes at a time; a cache that begins elsewhere is an error on the host."""
    q, kc, vc, b = _paged_case([1], [50], nq, nkv, 64)
    odd = torch.zeros(vc.numel() + 4, dtype=BF, device="cuda")[4:].view(vc.shape)
    got = torch.empty(1, nq * 128, dtype=BF, device="cuda")
    for k, v in ((kc, odd), (odd, vc)):
        with pytest.raises(RuntimeError):
            ops.C.decode_attention(q, k, v, b.block_tables, b.context_lens, got, None, None, 128, 1, 128 ** -0.5, ops.status)
    ops.check_status()


@pytest.mark.parametrize("batch,lo,hi,nq,nkv", [(64, 100, 1500, 16, 8), (200, 1, 700, 16, 8), (300, 3000, 3100, 8, 2), (7, 1, 4000, 32, 8),
                                                (70, 100, 2500, 64, 8)])
def test_decode_attention_flat_partition_many_sequences(ops, batch, lo, hi, nq, nkv, monkeypatch):
    """Enough tiles that every CTA's range spans several (sequence, head) items and most items are cut at most once;
    lengths from 1 token to several thousand, zero-length rows in between; both kernels against the fp32 statement,
    twice in a row (the scratch keeps stale partials from the first call)."""
    g = torch.Generator().manual_seed(batch)
    k_lens = torch.randint(lo, hi + 1, (batch,), generator=g).tolist()
    for i in range(3, batch, 17):
        k_lens[i] = 0
    q, kc, vc, b = _paged_case([1] * batch, k_lens, nq, nkv, 256, seed=batch)
    b.is_prefill = False
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    live = [i for i, n in enumerate(k_lens) if n > 0]
    for mode in ("flat", "flat", "chunked"):
        monkeypatch.setattr(ops, "decode_attention_mode", mode)
        got = ops.attention(q, kc, vc, b, 128 ** -0.5)
        _close(got[live], want[live], 2e-2, 2e-2)
        assert torch.count_nonzero(got[3]) == 0
    ops.check_status()


@pytest.mark.parametrize("q_lens,k_lens,nq,nkv,bs", [
    ([64], [64], 16, 8, 256), ([1, 100, 257], [1, 100, 257], 16, 8, 256), ([30, 70], [286, 70], 8, 2, 256),
    ([50, 200], [50, 200], 4, 4, 16), ([10], [522], 8, 1, 32), ([1000], [1000], 2, 1, 256),
    ([300, 129, 128, 1], [812, 129, 640, 1], 8, 2, 128), ([513, 40], [513, 1064], 4, 1, 256), ([128, 256], [128, 256], 16, 8, 512),
])
def test_prefill_attention(ops, q_lens, k_lens, nq, nkv, bs):
    q, kc, vc, b = _paged_case(q_lens, k_lens, nq, nkv, bs, seed=1)
    b.is_prefill = True
    got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("q_lens,k_lens,nq,nkv,bs", [
    ([130] * 9 + [1, 127, 128, 129, 256, 257], [130] * 9 + [1, 127, 128, 129, 256, 257], 16, 8, 256),
    ([1000, 3, 700], [1000, 3, 700], 32, 8, 256),                                # few sequences, several rounds of items per CTA
    ([5 + 3 * i for i in range(70)], [5 + 3 * i + 128 * (i % 3) for i in range(70)], 4, 2, 128),      # three ballots of sequences, prefixes
    ([300, 0, 129, 640, 0, 1, 511], [300, 0, 1153, 700, 256, 2, 511], 12, 4, 256),          # odd group: row pairs, with and without a second tile; empty ones
    ([257] * 20, [257] * 20, 5, 5, 512),
    ([256] * 3 + [64] * 9, [2304] * 3 + [2112] * 9, 32, 8, 256),                 # a prefix shared in length
])
def test_prefill_attention_two_tiles_per_cta(ops, q_lens, k_lens, nq, nkv, bs):
    """More tiles than SMs: items of two heads or two row tiles, dealt out over persistent CTAs (tolerance of the test above: bf16 operands and weights)."""
    assert sum(-(-n // 128) for n in q_lens) * nq > torch.cuda.get_device_properties(0).multi_processor_count
    q, kc, vc, b = _paged_case(q_lens, k_lens, nq, nkv, bs, seed=2)
    b.is_prefill = True
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    for _ in range(2):
        got = ops.attention(q, kc, vc, b, 128 ** -0.5)
        _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("seqs,nq,nkv", [(1, 1, 1), (40, 4, 2), (40, 5, 5)])
def test_prefill_attention_adds_row_sums_in_pairs(ops, seqs, nq, nkv):
    """One query tile per CTA, and two (heads of a group, or rows).  The scores are whole numbers, so the weights are powers of two: 1 + 2^-9,
    then 2^-18, then twice 2^-24 (the rest vanishes), and only the first value is 1.  Added pair by pair, the last two survive: the sum is
    1 + 2^-9 + 2^-18 + 2^-23 and the result 2^-8 below 1.  One by one they are lost and the result, a tie in bf16, is 1."""
    n = 128
    q, kc, vc, b = _paged_case([n] * seqs, [n] * seqs, nq, nkv, 256)
    b.is_prefill = True
    exponents = torch.full((n,), -200.0)
    for key, e in ((0, 0), (1, -9), (8, -18), (16, -24), (17, -24)):
        exponents[key] = e
    q.zero_(), kc.zero_(), vc.zero_()
    q[:, :, 0] = 1
    kc[:, :, :n, 0] = exponents.cuda().to(BF)
    vc[:, :, 0] = 1
    got = ops.attention(q, kc, vc, b, math.log(2)).view(seqs, n, nq * 128)          # times log2(e): a factor of exactly one
    assert torch.all(got[:, 18:].float() == 1 - 2.0 ** -8)
    ops.check_status()


@pytest.mark.parametrize("scale", [0.0, -0.05])
@pytest.mark.parametrize("q_lens,k_lens", [([300], [300]), ([300] * 12, [300] * 6 + [684] * 6)])
def test_prefill_attention_with_a_scale_that_is_not_positive(ops, q_lens, k_lens, scale):
    """Zero (every visible key counts the same) and less, with few query tiles and with many (each row sees a key of each of its tiles)."""
    q, kc, vc, b = _paged_case(q_lens, k_lens, 8, 4, 256, seed=6)
    b.is_prefill = True
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, scale, b.num_seqs)
    _close(ops.attention(q, kc, vc, b, scale), want, 2e-2, 2e-2)
    ops.check_status()


def _growing_keys(q, kc, b, nq, nkv, bs):
    """Adds a direction to q and k along which the keys grow from one 128-key tile to the next: the maxima of a part of the rows (a third of
    them, of different heads) jump by 10 to 40 in the exponent of 2 again and again, others by less than the 8 from which O is rescaled, a third not."""
    u = torch.nn.functional.normalize(torch.randn(128, device="cuda"), dim=0)
    strength = torch.tensor([0.0, 1.0, 6.0], device="cuda")[torch.randint(0, 3, q.shape[:2], device="cuda")] * (1 + torch.rand(q.shape[:2], device="cuda"))
    q += (strength[..., None] * u * 128 ** 0.5).to(BF)
    for s in range(b.num_seqs):
        for i in range(-(-int(b.context_lens[s]) // bs)):
            tile = (i * bs + torch.arange(bs, device="cuda")) // 128
            kc[b.block_tables[s, i]] += (1.5 * tile[:, None] * u).to(BF)


@pytest.mark.parametrize("q_lens,k_lens,nq,nkv,bs", [
    ([900], [900], 4, 2, 256), ([100, 300], [1400, 800], 3, 1, 128),                                     # one query tile per CTA
    ([1000, 300, 77], [1000, 300, 77], 32, 8, 256), ([200] * 6, [1224] * 6, 16, 8, 256),                 # two: heads of a group
    ([700, 129, 300], [700, 1153, 300], 27, 9, 256), ([400] * 5, [900] * 5, 10, 10, 512),                # two: rows of a head
])
def test_prefill_attention_with_growing_maxima(ops, q_lens, k_lens, nq, nkv, bs):
    """O is read back, scaled and stored between two products with V (tolerance of the tests above: bf16 operands and weights)."""
    q, kc, vc, b = _paged_case(q_lens, k_lens, nq, nkv, bs, seed=3)
    b.is_prefill = True
    _growing_keys(q, kc, b, nq, nkv, bs)
    want = ref.attention(q, kc, vc, b.cu_seqlens_q, b.context_lens, b.block_tables, 128 ** -0.5, b.num_seqs)
    got = ops.attention(q, kc, vc, b, 128 ** -0.5)
    _close(got, want, 2e-2, 2e-2)
    ops.check_status()


@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("nq,nkv", [(16, 8), (24, 8)])
def test_prefill_attention_does_not_depend_on_the_batch(ops, nq, nkv, grow):
    """A sequence alone (one query tile per CTA), the same one among others (two), and computed in portions that are no multiples of a tile:
    the same bits, so a prompt computed in portions or beside others gives the tokens it gives by itself.  Also where maxima grow, and with
    another sequence's queries behind the last rows of a tile."""
    lens = [1000, 333, 129, 64] + [300] * 8
    q, kc, vc, b = _paged_case(lens, lens, nq, nkv, 256, seed=5)
    b.is_prefill = True
    if grow:
        _growing_keys(q, kc, b, nq, nkv, 256)
    whole = ops.attention(q, kc, vc, b, 128 ** -0.5)
    at = 0
    for i, n in enumerate(lens[:4]):
        for first, last in [(0, n), (0, n // 3), (n // 3, n - n // 4), (n - n // 4, n)]:
            one = _Batch()
            one.is_prefill, one.num_seqs, one.padded_seqs, one.table_width = True, 1, 1, b.table_width
            one.cu_seqlens_q = torch.tensor([0, last - first], dtype=torch.int32, device="cuda")
            one.context_lens = torch.tensor([last], dtype=torch.int32, device="cuda")
            one.block_tables = b.block_tables[i:i + 1].contiguous()
            one.max_seqlen_q, one.max_seqlen_k = last - first, last
            rows = slice(at + first, at + last)
            assert torch.equal(ops.attention(q[rows].contiguous(), kc, vc, one, 128 ** -0.5), whole[rows]), (i, first, last)
        at += n
    ops.check_status()


# ----------------------------------------------------------------------------- sampler
def _header(step, seed):
    h = torch.zeros(16, dtype=torch.int32)
    h[9], h[10], h[11] = step, seed & 0x7FFFFFFF, 0
    return h.cuda()


def test_sampler_greedy_and_gumbel_match_reference(ops):
    torch.manual_seed(3)
    rows, vocab = 6, 151936
    logits = _rand(rows, vocab, scale=3.0)
    temps = torch.tensor([0.0, 0.6, 1.0, 0.0, 2.0, 0.3], device="cuda")
    ids, best = ops.sample_shard(logits, temps, _header(11, 1234), 0)
    want_ids, want_best = ref.sample(logits.cpu(), temps.cpu(), 1234, 11, 0)
    _close(best.cpu(), want_best, 1e-3, 1e-4)
    assert torch.equal(ids.cpu().long()[[0, 3]], logits.float().argmax(-1).cpu()[[0, 3]])
    # sampled rows: the chosen id must be (near-)optimal under the reference's perturbed scores
    assert (ids.cpu().long() == want_ids).float().mean() >= 0.8


def test_sampler_is_invariant_to_vocab_sharding(ops):
    torch.manual_seed(4)
    rows, vocab, tp = 5, 4096 * 4, 4
    logits = _rand(rows, vocab, scale=2.0)
    temps = torch.full((rows,), 0.8, device="cuda")
    hdr = _header(5, 99)
    full_ids, _ = ops.sample_shard(logits, temps, hdr, 0)
    shard = vocab // tp
    vals, ids = [], []
    for r in range(tp):
        i, v = ops.sample_shard(logits[:, r * shard:(r + 1) * shard], temps, hdr, r * shard)
        ids.append(i)
        vals.append(v)
    out = torch.empty(rows, dtype=torch.int32, device="cuda")
    ops.C.sample_merge_ranks(torch.stack(vals), torch.stack(ids), out)
    assert torch.equal(out, full_ids)


@pytest.mark.parametrize("vocab,start", [(16, 0), (80, 0), (72, 16)])
def test_sampler_distribution(ops, vocab, start):
    """Empirical frequencies over many rows follow softmax(logits / T): one group (level 2 alone), several groups (level 1
    picks the group, level 2 the token), and a shard whose last group is partial."""
    T, n = 0.7, 6000
    base = torch.linspace(-2, 2, vocab, device="cuda")[torch.randperm(vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(vocab))]
    logits = base.to(BF)[None].repeat(n, 1).contiguous()
    temps = torch.full((n,), T, device="cuda")
    ids, _ = ops.sample_shard(logits, temps, _header(1, 7), start)
    freq = torch.bincount(ids.long().cpu() - start, minlength=vocab).float() / n
    want = torch.softmax(logits[0].float().cpu() / T, -1)
    assert (freq - want).abs().max() < 0.025


@pytest.mark.parametrize("rows,vocab,start", [(8, 151936, 0), (64, 75968, 75968), (200, 40000, 40000), (256, 151936, 0)])
def test_lm_head_gemm_samples_in_its_epilogue_like_the_two_kernel_path(ops, rows, vocab, start):
    """LM head + sampling in one kernel (logits never written) picks exactly the tokens of GEMM -> logits -> sampler:
    the same bf16-rounded logits, the same noise per (row, global token id); greedy rows (T = 0) are the arg-max."""
    torch.manual_seed(rows + vocab)
    K = 1024
    hidden, w = _rand(rows, K), _rand(vocab, K, scale=0.05)
    temps = torch.full((rows,), 0.6, device="cuda")
    temps[::3] = 0.0
    temps[1::5] = 1.3
    hdr = _header(step=11, seed=5)
    assert ops.can_sample_in_lm_head(rows, w)
    ids, best = ops.lm_head_sample_shard(hidden, w, temps, hdr, start)
    logits = ops.linear(hidden, w)
    want_ids, want_best = ops.sample_shard(logits, temps, hdr, start)
    assert torch.equal(ids, want_ids)
    assert torch.equal(best, want_best)
    greedy = (temps == 0).nonzero().flatten()
    assert torch.equal(ids[greedy].long() - start, logits[greedy].float().argmax(-1))
    ops.check_status()


# ----------------------------------------------------------------------------- bounded waits
def test_peer_flag_wait_runs_out_and_reports_status(ops):
    """Failure detection on the device: a consumer waits for a peer that never signals (the flag word is simply
    never written), gives up after its time limit, sets the status bit, and the context stays usable."""
    import time
    H, rows = 1024, 4
    parts = torch.zeros(2, rows, H, dtype=BF, device="cuda")             # both "ranks'" partial buffers live on this GPU
    signal = torch.zeros(8, dtype=torch.int32, device="cuda")
    epoch = torch.ones(1, dtype=torch.int32, device="cuda")            # this rank claims one completed production ...
    signal[0] = 1                                                       # ... rank 0's flag is there, rank 1's never arrives
    normal_mode = torch.zeros(1, dtype=torch.int32, device="cuda")      # the measurement-mode switch stays off
    out = torch.empty(rows, H, dtype=BF, device="cuda")
    torch.cuda.synchronize()
    t0 = time.monotonic()
    ops.C.tp_reduce_rms_norm(2, 0, [parts[0].data_ptr(), parts[1].data_ptr()], 0, 0, signal.data_ptr(), epoch.data_ptr(), int(0.2e9),
                             normal_mode.data_ptr(), None, out, None, None, 1e-6, ops.status)
    torch.cuda.synchronize()
    assert 0.15 < time.monotonic() - t0 < 5.0
    with pytest.raises(RuntimeError, match="peer flag wait ran out"):
        ops.check_status()
    ops.check_status()                                                  # the word was cleared; nothing else is wrong
    x = _rand(8, 1024)
    assert torch.isfinite(ops.rms_norm(x, torch.ones(1024, dtype=BF, device="cuda"), 1e-6).float()).all()
