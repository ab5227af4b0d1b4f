"""MXFP8 GEMM on SM pairs (more than one wave of one-CTA tiles): both tile widths, with row and column tails."""
import pytest
import torch

from archscale_b200.ops import backend, mxfp8

pytestmark = pytest.mark.gpu


# (2048, 2112): 128-wide tiles (both widths need two waves of pairs), half a tile of columns at the end; the others 192-wide
@pytest.mark.parametrize("M,N,K", [(2048, 2112, 256), (3000, 1928, 384), (2304, 1728, 128)])
def test_pair_gemm_matches_dequantised_fp32(M, N, K):
    torch.manual_seed(2)
    a = (torch.randn(M, K, device="cuda") * torch.logspace(-1, 1, K, device="cuda")).bfloat16()
    b = (torch.randn(N, K, device="cuda") * (1 + torch.arange(N, device="cuda").view(-1, 1) % 7)).bfloat16()
    aq, asf = mxfp8.quantize(a)
    bq, bsf = mxfp8.quantize(b)
    ar = mxfp8.dequantize_ref(aq.view(torch.float8_e4m3fn), mxfp8.unchunk_scales_ref(asf, M, K))
    br = mxfp8.dequantize_ref(bq.view(torch.float8_e4m3fn), mxfp8.unchunk_scales_ref(bsf, N, K))
    ref = ar.double() @ br.double().t()
    big = ref.abs().max().item()
    out = mxfp8.gemm(aq, asf, bq, bsf, out_f32=True)
    assert (out.double() - ref).abs().max().item() <= 1e-4 * big          # K ≤ 384 products summed in fp32
    assert torch.equal(out, mxfp8.gemm(aq, asf, bq, bsf, out_f32=True))
    assert torch.equal(mxfp8.gemm(aq, asf, bq, bsf), out.bfloat16())      # the other output type: the same sums, rounded
    acc = torch.ones(M, N, device="cuda")
    mxfp8.gemm(aq, asf, bq, bsf, acc=acc, alpha=0.5)
    assert (acc.double() - (1 + 0.5 * ref)).abs().max().item() <= 1e-4 * big
    assert backend.require_extension().device_status() == 0
