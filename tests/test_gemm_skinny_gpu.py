"""Products of a few dozen rows without gradients (csrc/gemm_skinny.cu): against fp64, and the route against the general one."""
import pytest
import torch
import torch.nn.functional as F

from archscale_b200.models.layers import Linear
from archscale_b200.ops import backend, gemm

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def _w(n, k, pad=0):
    """(n, k) weight rows with `pad` more elements between them."""
    return (torch.randn(n, k + pad, device="cuda") / k ** 0.5).bfloat16()[:, :k]


# K tails (no multiple of 64), one K block (no split), row tails, row strides, one token, a full block of tokens
@pytest.mark.parametrize("M,N,K,pad", [(1, 8, 64, 0), (41, 1024, 1024, 0), (64, 136, 72, 8), (63, 5632, 1000, 0), (17, 264, 2816, 24),
                                       (64, 32000, 128, 0)])
def test_skinny_linear_matches_fp64(M, N, K, pad):
    torch.manual_seed(0)
    x, w = torch.randn(1, M, K, device="cuda").bfloat16(), _w(N, K, pad)
    with torch.no_grad():
        n0 = backend.launches()
        y = gemm.linear(x, w)
        assert backend.launches() == n0 + 1 and y.shape == (1, M, N)
        again = gemm.linear(x, w)
    ref = x.double() @ w.double().t()
    # one rounding to bf16 of an fp32 sum: relative 2^-9 at most, as the library's result
    assert _rel(y, ref) < 2.0 ** -8 and _rel(y, ref) < 1.05 * _rel(F.linear(x, w), ref) + 1e-6
    assert torch.equal(y, again)
    assert backend.require_extension().device_status() == 0


@pytest.mark.parametrize("M,I,K", [(1, 8, 64), (41, 2816, 1024), (64, 72, 200)])
def test_skinny_swiglu_matches_the_unfused_pair(M, I, K):
    torch.manual_seed(1)
    x, w = torch.randn(M, K, device="cuda").bfloat16(), _w(2 * I, K)
    with torch.no_grad():
        y = gemm.linear_swiglu(x, w)
    g, u = (x.double() @ w.double().t()).bfloat16().double().chunk(2, -1)
    assert _rel(y, F.silu(g) * u) < 2.0 ** -7       # two roundings to bf16 before the product, one after it


def test_skinny_multi_takes_weights_that_are_not_neighbours():
    torch.manual_seed(2)
    x = torch.randn(2, 21, 256, device="cuda").bfloat16()
    layers = [Linear(256, n, bias=False, device="cuda", dtype=torch.bfloat16) for n in (512, 128, 136)]
    with torch.no_grad():
        fused = gemm.linear_multi(x, layers, keep_fused=True)
        parts = gemm.linear_multi(x, layers)
    assert fused.shape == (2, 21, 776)
    for p, f, l in zip(parts, fused.split([512, 128, 136], -1), layers):
        assert torch.equal(p, f)
        assert _rel(p, x.double() @ l.weight.double().t()) < 2.0 ** -8


def test_route_needs_no_gradients_and_few_rows():
    x, w = torch.randn(41, 64, device="cuda").bfloat16(), _w(64, 64)
    wide = torch.randn(41, 128, device="cuda").bfloat16()[:, 64:]
    assert not gemm._skinny_ok(x, (w,))                                       # gradients on
    with torch.no_grad():
        assert gemm._skinny_ok(x, (w,))
        assert not gemm._skinny_ok(torch.randn(65, 64, device="cuda").bfloat16(), (w,))
        assert not gemm._skinny_ok(wide, (w,)) and not gemm._skinny_ok(x.float(), (w,)) and not gemm._skinny_ok(x[:0], (w,))
        assert _rel(gemm.linear(wide, w), wide.double() @ w.double().t()) < 2.0 ** -8
        with torch.autograd.forward_ad.dual_level():
            assert not gemm._skinny_ok(x, (w,))
        with pytest.raises(RuntimeError):
            gemm.linear(x, _w(64, 72))
