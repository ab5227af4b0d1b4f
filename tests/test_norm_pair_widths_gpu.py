"""RMSNorm backward with a row split over two warps: widths that fill neither the last chunk nor the second warp's share."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stream", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 1032), (5, 1280), (333, 1536), (70, 1544), (2500, 1984), (9, 2040), (64, 2048)])
def test_add_rms_norm_backward_widths(rows, cols, stream):
    from archscale_b200 import ops
    torch.manual_seed(7)
    dev = "cuda"
    res = torch.randn(rows, cols, device=dev).to(stream).requires_grad_(True)
    h = torch.randn(rows, cols, device=dev).bfloat16().requires_grad_(True)
    w = (1 + 0.1 * torch.randn(cols, device=dev)).requires_grad_(True)
    x, n = ops.add_rms_norm(res, h, w, 1e-5, 0.25, torch.bfloat16, stream)
    gx, gn = torch.randn_like(x), torch.randn_like(n)
    got = torch.autograd.grad((x, n), (res, h, w), (gx, gn))
    rd, hd, wd = (t.detach().double().requires_grad_(True) for t in (res, h, w))
    xd = rd + 0.25 * hd
    xs = xd + (x.detach().double() - xd.detach())               # the stream is rounded before it is normalised
    nd = xs * torch.rsqrt(xs.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    ref = torch.autograd.grad((xs, nd), (rd, hd, wd), (gx.double(), gn.double()))
    assert float((n.double() - nd).abs().max()) <= 2 ** -8 * float(nd.abs().max())
    # results in bf16 carry 2^-9 relative each, those in fp32 the rounding of sums over `cols` or `rows` terms
    for a, r in zip(got, ref):
        tol = 4e-3 if a.dtype == torch.bfloat16 else 1e-5
        assert float((a.double() - r).norm()) <= tol * float(r.norm())
