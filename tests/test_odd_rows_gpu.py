"""Token counts that are no multiple of 8 on the tcgen05 GEMM: the three layouts, the fp32 accumulation and the layers."""
import pytest
import torch
import torch.nn.functional as F

from archscale_b200.ops import backend, gemm

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def _mk(*s, pad=0):
    return (torch.randn(*s[:-1], s[-1] + pad, device="cuda") * 0.5).bfloat16()[..., :s[-1]]


# below, at and past a tile of 256 rows and a K block of 64; one row; row strides
@pytest.mark.parametrize("T", [1, 65, 129, 255, 257, 1001, 4099])
@pytest.mark.parametrize("I,O,pad", [(64, 8, 0), (136, 264, 8)])
def test_products_with_any_number_of_rows(T, I, O, pad):
    torch.manual_seed(0)
    x, w, dy = _mk(T, I, pad=pad), _mk(O, I, pad=pad), _mk(T, O, pad=pad)
    n0 = backend.launches()
    y = gemm.matmul_nt(x, w)
    dx = gemm.matmul_nn(dy, _mk(O, I)) if O >= 64 else None
    assert backend.launches() > n0
    # one rounding to bf16 of an fp32 sum
    assert _rel(y, x.double() @ w.double().t()) < 2.0 ** -8
    if dx is not None:
        w2 = _mk(O, I, pad=pad)
        assert _rel(gemm.matmul_nn(dy, w2), dy.double() @ w2.double()) < 2.0 ** -8
    ref = dy.double().t() @ x.double()
    assert _rel(gemm.matmul_tn(dy, x), ref) < 2.0 ** -8
    acc = torch.full((O, I), 0.25, device="cuda")
    gemm.matmul_tn_acc_(acc, dy, x)
    if T >= 64:
        assert _rel(acc, ref + 0.25) < 1e-5                     # fp32 sums of bf16 products, added in fp32
    assert backend.require_extension().device_status() == 0


@pytest.mark.parametrize("T", [67, 513, 2731])
def test_layers_agree_with_the_library_route(T):
    torch.manual_seed(1)
    x = _mk(1, T, 256).requires_grad_()
    w, w2 = (_mk(n, 256).requires_grad_() for n in (512, 144))
    for fn, ref in ((lambda: gemm.linear(x, w), lambda: F.linear(x.float(), w.float())),
                    (lambda: gemm.linear_swiglu(x, w), lambda: F.silu(F.linear(x.float(), w.float())[..., :256]) *
                     F.linear(x.float(), w.float())[..., 256:]),
                    (lambda: gemm.linear(x, w2), lambda: F.linear(x.float(), w2.float()))):
        y, r = fn(), ref()
        g = torch.randn_like(y)
        leaves = [x, w2 if y.shape[-1] == 144 else w]
        got, want = torch.autograd.grad(y, leaves, g), torch.autograd.grad(r, leaves, g.float())
        assert _rel(y, r) < 2.0 ** -7
        for a, b in zip(got, want):
            assert _rel(a, b) < 2.0 ** -7                       # gradients pass one more bf16 tensor each


@pytest.mark.parametrize("T", [1, 67, 1001])
def test_a_small_bias_is_added_before_the_rounding(T):
    torch.manual_seed(2)
    x, w = _mk(T, 256), _mk(512, 256)
    b = torch.full((512,), 2.0 ** -9, device="cuda", dtype=torch.bfloat16)      # far below an ulp of most of the products (up to 2^-4)
    y, ref = gemm.linear(x, w, b), x.double() @ w.double().t() + b.double()
    # half an ulp (at most 2^-8 of the value), and fp32 sums of 256 products of magnitude below 8
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 256 * 8 * 2.0 ** -24).all())
    # the bias survives on average; a second rounding drops it where an ulp exceeds 2^-8: the mean of n rounding errors, each
    # within ulp / 2 <= 2^-8 |ref|, stays within 6 of its standard deviations
    err = (y.double() - ref)
    if T > 1:
        assert abs(float(err.mean())) < 6 * 2.0 ** -8 * float(ref.norm()) / ref.numel()
