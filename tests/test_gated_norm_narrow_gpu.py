"""Backward of the gated RMSNorm in groups of at most 256 columns (half the registers, more CTAs) against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,groups,g", [(1, 3, 8), (23, 64, 8), (25, 16, 64), (1000, 16, 64), (7111, 1, 128), (49, 1, 256), (1000, 2, 256),
                                           (1000, 2, 264)])
def test_narrow_groups(rows, groups, g, dtype):
    from archscale_b200.ops.norm import gated_rms_norm
    torch.manual_seed(8)
    n = groups * g
    mk = lambda: torch.randn(rows, n, device="cuda").to(dtype).requires_grad_(True)
    x, z, gy = mk(), mk(), mk().detach()
    w = (1 + 0.2 * torch.randn(n, device="cuda")).requires_grad_(True)
    for nbg in (True, False):
        got = torch.autograd.grad(gated_rms_norm(x, w, z, 1e-5, g, nbg), (x, w, z), gy)
        xd, wd, zd = refs = [t.detach().double().requires_grad_(True) for t in (x, w, z)]
        s = torch.nn.functional.silu(zd)
        xin = (xd if nbg else xd * s).view(rows, groups, g)
        nrm = (xin * torch.rsqrt(xin.pow(2).mean(-1, keepdim=True) + 1e-5)).view(rows, n) * wd
        ref = torch.autograd.grad(nrm * s if nbg else nrm, refs, gy.double())
        # bf16 results are rounded once (2^-9); fp32: sums over up to 264 columns or 7111 rows and the fast exponential
        for a, r in zip(got, ref):
            assert float((a.double() - r).norm()) <= (4e-3 if a.dtype == torch.bfloat16 else 2e-6) * float(r.norm())
