"""Up to 16 row taps on the tensor-core convs (one output staging tile, two staged score tiles): each against the CUDA-core path."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, conv64, conv64_bwd_input, npf, rel_fro, rel_max

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("S,R,Sk,causal,dtype", [(264, 9, 9, True, torch.bfloat16), (520, 11, 15, True, torch.float16), (136, 16, 17, True, torch.bfloat16),
                                                 (384, 13, 3, False, torch.float16)])
def test_conv2d(S, R, Sk, causal, dtype):
    g = torch.Generator(device=DEV).manual_seed(S)
    x, gr = (torch.randn(3, 5, S, S, device=DEV, generator=g).to(dtype) for _ in range(2))
    w = (torch.randn(5, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(dtype)
    if causal:
        x, gr = (t.masked_fill(torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1), float("nan")) for t in (x, gr))
    got = {}
    for variant in (0, 1):
        _lib.set_variant("conv2d", variant)
        try:
            got[variant] = ops.conv2d_fwd(x, w, causal), ops.conv2d_bwd_input(gr, w, causal)
        finally:
            _lib.set_variant("conv2d", 0)
    _lib.device_status()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got[0], got[1]):
        assert float((a.float() - b.float()).abs().max()) <= 2 * ulp * float(b.float().abs().max())


@pytest.mark.parametrize("S,D,R,Sk", [(257, 128, 7, 9), (130, 128, 11, 15), (400, 128, 16, 17), (200, 64, 14, 11)])
def test_conv_attention_and_scores_in_the_conv(S, D, R, Sk):
    g = torch.Generator(device=DEV).manual_seed(S + R)
    q, k, v = (torch.randn(2, 8, S, D, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w = (torch.randn(8, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(torch.bfloat16)
    mix = [(torch.eye(8, device=DEV) + 0.1 * torch.randn(8, 8, device=DEV, generator=g)).to(torch.bfloat16) for _ in range(2)]
    one = ops.conv_attn_fwd(q, k, v, w, True, D ** -0.5), ops.mta_fused_fwd(q, k, v, w, mix[0], w, mix[1])
    _lib.set_variant("gemm", 1)
    _lib.set_variant("conv2d", 1)
    try:
        ref = ops.conv_attn_fwd(q, k, v, w, True, D ** -0.5), ops.mta_fused_fwd(q, k, v, w, mix[0], w, mix[1])
    finally:
        _lib.set_variant("gemm", 0)
        _lib.set_variant("conv2d", 0)
    _lib.device_status()
    for a, b in zip(one, ref):
        assert rel_fro(npf(a), npf(b)) <= 1e-2 and rel_max(npf(a), npf(b)) <= 3e-2


# A long launch of the score + conv kernel works through its planes in groups: bit-identical to launches of one group.
@pytest.mark.parametrize("R,Sk", [(6, 11), (11, 15)])
def test_long_launches_equal_short_ones(R, Sk):
    g = torch.Generator(device=DEV).manual_seed(R)
    q, k, v = (torch.randn(16, 16, 1030, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w = (torch.randn(16, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(torch.bfloat16)
    mix = [(torch.eye(16, device=DEV) + 0.1 * torch.randn(16, 16, device=DEV, generator=g)).to(torch.bfloat16) for _ in range(2)]
    whole = ops.mta_fused_fwd(q, k, v, w, mix[0], w, mix[1])
    for b in (0, 7, 15):
        assert torch.equal(whole[b:b + 1], ops.mta_fused_fwd(q[b:b + 1], k[b:b + 1], v[b:b + 1], w, mix[0], w, mix[1]))
    _lib.device_status()


# The same kernels against references that share nothing with them: the conv and its input gradient in float64 (a result may be off by its own
# rounding - half a unit in the last of 8 or 11 significant bits, so 2^-8 or 2^-11 of it - and by the float32 sum of up to 272 products:
# 272 * 2^-24 of the sum of their magnitudes, which is about 11),
# the attention forwards against the oracle.
@pytest.mark.parametrize("S,R,Sk,causal,dtype", [(264, 9, 9, True, torch.bfloat16), (520, 11, 15, True, torch.float16), (136, 16, 17, True, torch.bfloat16),
                                                 (384, 13, 3, False, torch.float16), (200, 7, 7, True, torch.float16)])
def test_conv2d_against_float64(S, R, Sk, causal, dtype):
    g = torch.Generator(device=DEV).manual_seed(S)
    x, gr = (torch.randn(3, 5, S, S, device=DEV, generator=g).to(dtype) for _ in range(2))
    w = (torch.randn(5, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(dtype)
    got = ops.conv2d_fwd(x, w, causal), ops.conv2d_bwd_input(gr, w, causal)
    _lib.device_status()
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got, (conv64(x, w, causal), conv64_bwd_input(gr, w, causal))):
        assert bool(((a.double() - b).abs() <= u * b.abs() + 2e-4).all())


@pytest.mark.parametrize("S,D,R,Sk", [(257, 128, 7, 9), (130, 128, 11, 15), (400, 128, 16, 17), (200, 64, 14, 11)])
def test_attention_against_the_oracle(S, D, R, Sk):
    g = torch.Generator(device=DEV).manual_seed(S + R)
    q, k, v = (torch.randn(1, 8, S, D, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w = (torch.randn(8, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(torch.bfloat16)
    mix = [(torch.eye(8, device=DEV) + 0.1 * torch.randn(8, 8, device=DEV, generator=g)).to(torch.bfloat16) for _ in range(2)]
    attn, mta = ops.conv_attn_fwd(q, k, v, w, True, D ** -0.5), ops.mta_fused_fwd(q, k, v, w, mix[0], w, mix[1])
    _lib.device_status()
    n = [npf(t) for t in (q, k, v, w, mix[0], mix[1])]
    assert_parity(npf(attn), orc.conv_attn_fwd(*n[:4], True, D ** -0.5, orc.ROUND_NONE), torch.bfloat16, "conv attention")
    assert_parity(npf(mta), orc.mta_fwd(*n[:5], n[3], n[5], True, ROUND[torch.bfloat16]), torch.bfloat16, "forward")
