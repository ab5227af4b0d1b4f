"""Selective scan with the time axis in parts: the state handed from part to part, against the recurrence in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, L, Di, a_scale, dtype=torch.float32):
    torch.manual_seed(9)
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)
    A = -(0.5 + torch.rand(Di, 16, device="cuda")) * a_scale
    bias = torch.full((Di,), -4.0, device="cuda")                     # dt about 0.02: a state lives for many hundred steps
    return dict(u=mk(B, L, Di), delta=(0.3 * torch.randn(B, L, Di, device="cuda")).to(dtype), A=A, B=mk(B, L, 16), C=mk(B, L, 16),
                D=torch.randn(Di, device="cuda"), z=mk(B, L, Di), delta_bias=bias)


def _run(x, cu=None, softplus=True):
    from archscale_b200.ops.selective_scan import selective_scan
    return selective_scan(x["u"], x["delta"], x["A"], x["B"], x["C"], x["D"], z=x["z"], delta_bias=x["delta_bias"], delta_softplus=softplus,
                          cu_seqlens=cu, channel_last=True)


def _oracle(x, cuts=(), softplus=True):
    v = {k: t.double() for k, t in x.items()}
    dt = v["delta"] + v["delta_bias"]
    dt = torch.nn.functional.softplus(dt) if softplus else dt
    B, L, Di = v["u"].shape
    h, ys = v["u"].new_zeros(B, Di, 16), []
    for t in range(L):
        if t in cuts:
            h = torch.zeros_like(h)
        h = torch.exp(dt[:, t, :, None] * v["A"]) * h + (dt[:, t] * v["u"][:, t])[..., None] * v["B"][:, t, None]
        ys.append((h * v["C"][:, t, None]).sum(-1))
    y = torch.stack(ys, 1) + v["D"] * v["u"]
    return y * torch.nn.functional.silu(v["z"])


def _parts(B, L, Di):
    """Length of a part by the rule of the launch (a multiple of 64)."""
    n = min(-(-49152 // (B * Di)), L // 512)
    assert B * Di < 8192 and n >= 3
    return -(-(-(-L // n)) // 64) * 64


# L 2304 = four parts of 576 (a state keeps e^-0.06 .. e^-17 of itself over one), 2500 = four of 640 with a short last one
@pytest.mark.parametrize("a_scale", [0.005, 0.05, 1.0])
@pytest.mark.parametrize("B,L,cuts", [
    (1, 2304, None), (2, 2304, None), (1, 2500, None),
    (1, 2304, ()),                                                    # one document
    (1, 2304, (700,)),                                                # inside the second part: the first and the last two hold none
    (1, 2304, (1152,)),                                               # on the edge between the second and the third part
    (1, 2304, (1151, 1153)), (1, 2304, (600, 1800, 2303)), (1, 2500, (10, 2400)),
])
def test_state_crosses_parts(B, L, cuts, a_scale):
    x = _inputs(B, L, 48, a_scale)
    assert _parts(B, L, 48) == (576 if L == 2304 else 640)
    cu = None if cuts is None else torch.tensor([0, *cuts, L], dtype=torch.int32, device="cuda")
    y, yr = _run(x, cu), _oracle(x, cuts or ())
    # the recurrence rounds at every step (2^-24 of the state); a state of thousands of steps' memory collects sqrt(L) of them
    assert float((y.double() - yr).norm()) <= 1e-5 * float(yr.norm())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("cut", [700, 1152, 1500])
def test_documents_stay_separate(bad, cut):
    """A state that is not finite ends with its document, whether or not the next one starts in another part."""
    L = 2304
    x = _inputs(1, L, 48, 0.05)
    cu = torch.tensor([0, cut, L], dtype=torch.int32, device="cuda")
    clean = _run(x, cu)
    x["u"][0, 5, 3] = bad
    y = _run(x, cu)
    assert torch.equal(y[:, cut:], clean[:, cut:])
    assert not bool(torch.isfinite(y[0, 5:cut, 3]).all())


def test_growing_states():
    """exp(A·Σdt) of a part beyond the largest float meets a state that is zero or small: the product is what the steps give."""
    L, Di = 2304, 48
    x = _inputs(1, L, Di, 1.0)
    x["A"], x["delta_bias"] = torch.ones(Di, 16, device="cuda"), torch.zeros(Di, device="cuda")
    x["delta"] = torch.full((1, L, Di), 0.2, device="cuda")           # e^115 per part of 576 steps
    x["u"][:, :2100] = 0.0                                            # the state leaves zero in the last part
    x["u"][:, 2104:] = 0.0
    y, yr = _run(x, softplus=False), _oracle(x, softplus=False)
    assert float((y.double() - yr).norm()) <= 1e-4 * float(yr.norm())  # 200 steps, each with the rounded exponential (2^-22)
    x["delta"][:, :1152] = 0.0                                        # the state 1e-30 in front of the third part grows e^115-fold
    x["u"].zero_()
    x["u"][:, 1151] = 1e-30
    x["delta"][:, 1151] = 1.0
    x["delta"][:, 1728:] = 0.0
    y, yr = _run(x, softplus=False), _oracle(x, softplus=False)
    assert bool(torch.isfinite(yr.float()).all())
    assert float((y.double() - yr).norm()) <= 1e-4 * float(yr.norm())
