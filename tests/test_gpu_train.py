"""The one-node training path (mta_train_fwd / mta_train_bwd) against autograd through a plain PyTorch evaluation in float64,
at lengths around the tile edges, and the float32 score-plane products behind it."""
import types

import pytest
import torch
import torch.nn.functional as F

from multitokenatention_triton_b200 import MTAAttentionTriton, _lib, ops
from multitokenatention_triton_b200.autograd_ops import MTAFunction

pytestmark = pytest.mark.gpu
DEV = "cuda"


def torch_mta(q, k, v, w1, W1, w2, W2):
    S = q.size(-2)
    dead = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)

    def conv(x, w):
        p = (w.size(-1) - 1) // 2
        return F.conv2d(F.pad(x.masked_fill(dead, 0.0), (p, p, w.size(-2) - 1, 0)), w.unsqueeze(1), groups=x.size(1))

    s = conv(q @ k.transpose(2, 3) * q.size(-1) ** -0.5, w1)
    s = torch.einsum("oh,bhqk->boqk", W1, s).masked_fill(dead, float("-inf")).softmax(-1)
    s = torch.einsum("oh,bhqk->boqk", W2, conv(s, w2).masked_fill(dead, 0.0))
    return (s @ v).transpose(1, 2)


@pytest.mark.parametrize("S,H,D,ker,ker2,dtype", [
    (1, 8, 64, (3, 5), (3, 3), torch.bfloat16), (127, 16, 128, (6, 11), (3, 3), torch.bfloat16),
    (129, 8, 64, (2, 3), (6, 11), torch.float16), (200, 12, 64, (11, 15), (7, 9), torch.bfloat16),
    (321, 16, 128, (6, 11), (6, 11), torch.float16), (67, 8, 32, (3, 5), (3, 3), torch.float32),
    (130, 16, 64, (11, 15), (11, 15), torch.float32), (96, 64, 128, (5, 5), (3, 3), torch.bfloat16)])
def test_training_step(S, H, D, ker, ker2, dtype):
    cfg = types.SimpleNamespace(use_mta=True, query_kernel_size=ker[0], key_kernel_size=ker[1], after_sm_query_kernel_size=ker2[0],
                                after_sm_key_kernel_size=ker2[1], pre_sm_linear_head=True, post_sm_linear_head=True, pad_key="both",
                                init_method="identity", dim=H * D)
    g = torch.Generator(device=DEV).manual_seed(S)
    m = MTAAttentionTriton(H, cfg, dropout=0.0, causal=True).to(DEV, dtype)
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 2:
                p.copy_(torch.eye(H, device=DEV) + 0.1 * torch.randn(H, H, device=DEV, generator=g))
            else:
                p.copy_(torch.randn(p.shape, device=DEV, generator=g) * (p[0].numel()) ** -0.5)
                p[:, -1, p.shape[2] // 2] += 1.0
    x = [torch.randn(2, H, S, D, device=DEV, generator=g).to(dtype).requires_grad_() for _ in range(3)]
    up = torch.randn(2, S, H, D, device=DEV, generator=g).to(dtype)
    out = m(*x, None, None)
    out.backward(up)
    _lib.device_status()
    w = [m.mta_conv_triton.weight, m.wpsm_triton.weight, m.mta_conv_after_sm_triton.weight, m.wposm_triton.weight]
    ref_in = [t.detach().double().requires_grad_() for t in x + w]
    ref = torch_mta(*ref_in)
    ref.backward(up.double())
    tol = {torch.float32: 2e-5, torch.float16: 6e-3, torch.bfloat16: 4e-2}[dtype]
    for name, got, want in zip(("out", "dq", "dk", "dv", "dw1", "dW1", "dw2", "dW2"), [out] + [t.grad for t in x + w],
                               [ref] + [t.grad for t in ref_in]):
        err = float((got.detach().double() - want.detach()).norm() / want.detach().norm().clamp_min(1e-30))
        if S == 1 and name in ("dq", "dk", "dw1", "dW1"):       # a softmax over one key has no gradient
            assert float(want.abs().max()) < 1e-12 and float(got.abs().max()) < 1e-2, name
            continue
        assert err <= tol, f"{name}: relative error {err:.3e}"


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S,D", [(4, 8), (60, 100), (64, 64), (68, 128), (132, 36), (260, 128)])
def test_float32_products(S, D, causal):
    g = torch.Generator(device=DEV).manual_seed(S + D)
    q, k, v = (torch.randn(2, 3, S, D, device=DEV, generator=g) for _ in range(3))
    p = torch.rand(2, 3, S, S, device=DEV, generator=g)
    mask = (lambda t: t.tril()) if causal else (lambda t: t)
    s = ops.qk_scores_fwd(q, k, 0.25, causal)
    assert torch.allclose(s.double(), mask(q.double() @ k.double().transpose(2, 3) * 0.25), atol=2e-5, rtol=1e-5)
    pn = p.clone()
    if causal:
        pn.masked_fill_(torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1), float("nan"))
    o = ops.pv_fwd(pn, v, causal)
    assert torch.allclose(o.double(), mask(p.double()) @ v.double(), atol=5e-5, rtol=1e-5)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("H,W,R,S,dtype", [(8, 8, 1, 1, torch.bfloat16), (127, 120, 6, 11, torch.float16), (128, 96, 2, 16, torch.bfloat16),
                                           (129, 136, 7, 17, torch.bfloat16), (260, 48, 16, 15, torch.float16), (64, 328, 20, 3, torch.bfloat16),
                                           (640, 640, 11, 15, torch.bfloat16)])
def test_conv_weight_gradient_tensor_cores(H, W, R, S, dtype, causal):
    """Planes around the 128-row, 48-key step, odd and even tap counts, several flushes; NaN above the diagonal."""
    g = torch.Generator(device=DEV).manual_seed(H + W)
    x, dy = (torch.randn(2, 3, H, W, device=DEV, generator=g).to(dtype) for _ in range(2))
    dead = torch.arange(W, device=DEV)[None, :] > torch.arange(H, device=DEV)[:, None]
    xr, dr = x.double(), dy.double()
    if causal:
        xr, dr = xr.masked_fill(dead, 0.0), dr.masked_fill(dead, 0.0)
        x, dy = x.masked_fill(dead, float("nan")), dy.masked_fill(dead, float("nan"))
    got = ops.conv2d_bwd_weight(x, dy, (R, S), causal)
    _lib.device_status()
    pad = (S - 1) // 2
    xp = F.pad(xr, (pad, S - 1 - pad, R - 1, 0))
    want = torch.stack([torch.stack([(xp[:, :, i:i + H, j:j + W] * dr).sum((0, 2, 3)) for j in range(S)], -1) for i in range(R)], -2)
    bound = (xr.abs().sum((0, 2, 3)).max() * 3).item()
    assert float((got.double() - want).abs().max()) <= 2e-6 * bound + 1e-5


def setup_step(B, S, H, D, ker, ker2, dtype, w_dtype, seed):
    """q, k, v, the four weights and an upstream gradient in the layout of the module's output."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = [torch.randn(B, H, S, D, device=DEV, generator=g).to(dtype) for _ in range(3)]
    conv = [torch.randn(H, *k, device=DEV, generator=g) * (k[0] * k[1]) ** -0.5 for k in (ker, ker2)]
    for w in conv:
        w[:, -1, w.shape[2] // 2] += 1.0
    mix = [torch.eye(H, device=DEV) + 0.1 * torch.randn(H, H, device=DEV, generator=g) for _ in range(2)]
    up = torch.randn(B, S, H, D, device=DEV, generator=g).to(dtype)
    return x, [t.to(w_dtype) for t in (conv[0], mix[0], conv[1], mix[1])], up


# Long enough for the head mixes on tcgen05 (16 heads from a padded row of 1024 on, 8 heads from 1536), and float32 weights with 16-bit
# activations, whose convs and head mixes run on other kernels.  Tolerances as above: the same stages round.
@pytest.mark.parametrize("S,H,D,ker,ker2,dtype,w_dtype", [
    (1030, 16, 64, (6, 11), (3, 3), torch.bfloat16, torch.bfloat16), (1024, 16, 128, (7, 7), (7, 7), torch.float16, torch.float16),
    (1543, 8, 64, (3, 5), (3, 3), torch.bfloat16, torch.bfloat16), (1021, 16, 64, (6, 11), (3, 3), torch.bfloat16, torch.float32),
    (200, 12, 128, (11, 15), (3, 3), torch.float16, torch.float32), (130, 64, 64, (5, 5), (3, 3), torch.bfloat16, torch.float32)])
def test_long_and_mixed_precision_steps(S, H, D, ker, ker2, dtype, w_dtype):
    x, w, up = setup_step(1, S, H, D, ker, ker2, dtype, w_dtype, S)
    leaves = [t.requires_grad_() for t in x + w]
    out = MTAFunction.apply(*leaves).transpose(1, 2)
    out.backward(up)
    _lib.device_status()
    ref_in = [t.detach().double().requires_grad_() for t in leaves]
    ref = torch_mta(*ref_in)
    ref.backward(up.double())
    tol = {torch.float16: 6e-3, torch.bfloat16: 4e-2}[dtype]
    for name, got, want in zip(("out", "dq", "dk", "dv", "dw1", "dW1", "dw2", "dW2"), [out] + [t.grad for t in leaves],
                               [ref] + [t.grad for t in ref_in]):
        err = float((got.detach().double() - want.detach()).norm() / want.detach().norm())
        assert err <= tol, f"{name}: relative error {err:.3e}"
    assert all(t.grad.dtype == t.dtype for t in leaves)


NEEDS = [tuple(i == j for j in range(7)) for i in range(7)] + [
    (True, False, False, False, False, False, False), (True, True, True, False, False, False, False),
    (False, False, False, True, True, True, True), (False, False, True, False, False, False, True), (False, True, False, False, True, False, False)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradients_that_are_not_asked_for(dtype):
    """Every gradient alone and some together: bit for bit those of the whole step, and nothing where none is wanted."""
    x, w, up = setup_step(2, 130, 16, 64, (6, 11), (3, 3), dtype, dtype, 7)
    out, saved = ops.mta_train_fwd(*x, *w)
    g = up.transpose(1, 2)
    whole = ops.mta_train_bwd(g, saved, *x, *w, (True,) * 7)
    for needs in NEEDS:
        part = ops.mta_train_bwd(g, saved, *x, *w, needs)
        for i, (a, b) in enumerate(zip(part, whole)):
            assert (a is None) == (not needs[i])
            assert a is None or torch.equal(a, b), f"{needs}: gradient {i}"
    # frozen weights through autograd
    xs = [t.clone().requires_grad_(i != 1) for i, t in enumerate(x)]
    MTAFunction.apply(*xs, *w).backward(g)
    _lib.device_status()
    assert torch.equal(xs[0].grad, whole[0]) and xs[1].grad is None and torch.equal(xs[2].grad, whole[2])


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float16, 20), (torch.float32, 64), (torch.float32, 33)])
def test_layouts_of_the_upstream_gradient(dtype, D):
    """(B,S,H,D) and (B,H,S,D) contiguous, neither, off a 16-byte boundary, and the expanded one of a sum."""
    B, S, H = 2, 67, 8
    x, w, up = setup_step(B, S, H, D, (3, 5), (3, 3), dtype, dtype, D)
    out, saved = ops.mta_train_fwd(*x, *w)
    whole = ops.mta_train_bwd(up.transpose(1, 2), saved, *x, *w, (True,) * 7)
    odd = torch.empty(up.numel() + 1, device=DEV, dtype=dtype)
    odd[1:].copy_(up.flatten())
    wide = torch.zeros(B, S, H, D + 3, device=DEV, dtype=dtype)
    wide[..., :D].copy_(up)
    for g in (up.transpose(1, 2).contiguous(), odd[1:].view(B, S, H, D).transpose(1, 2), wide[..., :D].transpose(1, 2)):
        for a, b in zip(ops.mta_train_bwd(g, saved, *x, *w, (True,) * 7), whole):
            # an unaligned gradient takes other product kernels: the same sums in another order
            err = float((a.double() - b.double()).norm() / b.double().norm())
            assert err <= {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1e-2}[dtype]
    ones = ops.mta_train_bwd(torch.ones(B, H, S, D, device=DEV, dtype=dtype), saved, *x, *w, (True,) * 7)
    leaves = [t.clone().requires_grad_() for t in x + w]
    MTAFunction.apply(*leaves).sum().backward()
    _lib.device_status()
    for a, b in zip(leaves, ones):
        assert torch.equal(a.grad, b)
