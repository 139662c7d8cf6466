"""GEMM paths chosen by shape: K split over the pairs of a cluster, odd row blocks on CTA pairs, and the block-scaled GEMM
whose SwiGLU result leaves quantised."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(m, n, k, seed=0):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    a = torch.randn(m, k, device='cuda', generator=gen).bfloat16()
    b = (torch.randn(n, k, device='cuda', generator=gen) * 0.05).bfloat16()
    return a, b


def _close(d, want):
    # one rounding to bf16 (2^-9 of the value) on top of fp32 sums (a few 1e-6 of the largest); twice that
    assert torch.all((d.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max())


def _swiglu(full):
    t = full.view(full.shape[0], -1, 2, 128)
    return (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(full.shape[0], -1)


@pytest.mark.parametrize('m,n,k', [(1, 256, 1024), (128, 256, 512), (129, 512, 576), (256, 3584, 4096), (256, 4096, 1792), (300, 1024, 1088),
                                   (257, 4096, 8192), (512, 4352, 1024), (16, 256, 64)])
def test_split_k_matches_the_unsplit_product(m, n, k):
    from msccl.ops import check_gemm_errors, gemm_bf16
    a, b = _operands(m, n, k)
    full = a.double() @ b.double().t()
    _close(gemm_bf16(a, b), full)
    _close(gemm_bf16(a, b, epilogue='swiglu'), _swiglu(full))
    check_gemm_errors()
    # rows beyond M and columns beyond the result are left alone
    holder = torch.full((m + 2, n + 64), 7.0, device='cuda', dtype=torch.bfloat16)
    gemm_bf16(a, b, out=holder[1:m + 1, :n])
    assert torch.all(holder[0] == 7) and torch.all(holder[m + 1] == 7) and torch.all(holder[1:, n:] == 7)
    _close(holder[1:m + 1, :n], full)


@pytest.mark.parametrize('m,n,k', [(16, 3584, 4096), (128, 256, 1024), (256, 3584, 4096), (256, 4096, 1792), (300, 7168, 7168)])
@pytest.mark.parametrize('epilogue', ['none', 'swiglu'])
def test_split_k_is_as_exact_as_the_unsplit_sum(m, n, k, epilogue):
    """Both kinds of sum are fp32; what is left of either error is the rounding of the result, 1.66e-3 of its norm.  The two may
    round a few values (below 1 %) to different sides; measured, the split sum was never further from 64 bits."""
    from msccl.ops import check_gemm_errors, gemm_bf16
    a, b = _operands(m, n, k, 3)
    want = a.double() @ b.double().t()
    if epilogue == 'swiglu':
        want = _swiglu(want)
    split, whole = gemm_bf16(a, b, epilogue=epilogue), gemm_bf16(a, b, epilogue=epilogue, pair=True)
    assert torch.equal(split, gemm_bf16(a, b, epilogue=epilogue))          # the order of the parts is fixed
    check_gemm_errors()
    assert float((split != whole).float().mean()) < 0.01
    assert float((split.double() - want).norm()) <= 1.001 * float((whole.double() - want).norm())


@pytest.mark.parametrize('m,n,k', [(1, 256, 128), (128, 512, 256), (130, 256, 1024), (384, 768, 1792), (640, 256, 128)])
def test_block_scaled_gemm_on_pairs_behind_an_odd_row_block(m, n, k):
    from msccl.ops import check_gemm_errors
    from msccl.ops.gemm import gemm_mxfp8, quantize_mxfp8_packed
    a, b = _operands(m, n, k, 1)
    (aq, sa), (bq, sb) = quantize_mxfp8_packed(a), quantize_mxfp8_packed(b)
    assert torch.equal(gemm_mxfp8(aq, sa, bq, sb), gemm_mxfp8(aq, sa, bq, sb, pair=False))
    check_gemm_errors()


@pytest.mark.parametrize('m,n,k', [(128, 256, 128), (256, 512, 512), (384, 1024, 256), (1024, 7168, 1024)])
def test_quantised_swiglu_epilogue(m, n, k):
    from msccl.ops import check_gemm_errors
    from msccl.ops.gemm import dequantize_mxfp8, gemm_mxfp8_swiglu, quantize_mxfp8, quantize_mxfp8_packed
    a, b = _operands(m, n, k, 2)
    (aq, sa), (bq, sb) = quantize_mxfp8_packed(a), quantize_mxfp8_packed(b)
    q = torch.empty(m, n // 2, dtype=torch.float8_e4m3fn, device='cuda')
    sf = torch.full((m // 128 * (n // 256) * 512,), 255, dtype=torch.uint8, device='cuda')
    gemm_mxfp8_swiglu(aq, sa, bq, sb, q, sf)
    check_gemm_errors()
    h = _swiglu((dequantize_mxfp8(*quantize_mxfp8(a.float())).double() @ dequantize_mxfp8(*quantize_mxfp8(b.float())).double().t()))
    want_q, want_sf = quantize_mxfp8_packed(h.to(torch.bfloat16))
    # a bf16 value on the other side of a rounding or e4m3 boundary may differ; nearly all bytes are the same
    assert (q.view(torch.uint8) != want_q.view(torch.uint8)).float().mean() < 0.02
    assert (sf != want_sf).float().mean() < 0.002
