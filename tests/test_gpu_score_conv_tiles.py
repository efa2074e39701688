"""The convs with their input in tensor memory at the edges of their tiles: 4 (33 - R) query rows in four groups of 33 - R, 112 keys."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, conv64, conv64_bwd_input, npf

pytestmark = pytest.mark.gpu
DEV = "cuda"


# lengths around one group, one tile of rows, one tile of keys and two of them; the fewest and the most row taps; float32 weights
@pytest.mark.parametrize("S,R,Sk,D,dtype,w32", [
    (26, 6, 11, 128, torch.bfloat16, False), (28, 6, 11, 128, torch.bfloat16, False), (107, 6, 11, 128, torch.bfloat16, False),
    (109, 6, 11, 64, torch.float16, False), (111, 6, 11, 128, torch.bfloat16, False), (112, 6, 11, 64, torch.bfloat16, False),
    (113, 6, 11, 128, torch.float16, False), (217, 6, 11, 128, torch.bfloat16, True), (225, 6, 17, 64, torch.bfloat16, False),
    (129, 1, 1, 64, torch.bfloat16, False), (113, 1, 3, 128, torch.float16, True), (125, 2, 3, 128, torch.bfloat16, False),
    (69, 16, 17, 128, torch.bfloat16, True), (137, 16, 17, 64, torch.float16, False), (233, 11, 15, 128, torch.bfloat16, False)])
def test_tile_edges(S, R, Sk, D, dtype, w32):
    g = torch.Generator().manual_seed(S * 100 + R)
    q, k, v = (torch.randn(1, 8, S, D, generator=g).to(dtype) for _ in range(3))
    wd = torch.float32 if w32 else dtype
    w = (torch.randn(8, R, Sk, generator=g) * (R * Sk) ** -0.5).to(wd)
    w2 = (torch.randn(8, 3, 3, generator=g) / 3).to(wd)
    mix = [(torch.eye(8) + 0.1 * torch.randn(8, 8, generator=g)).to(wd) for _ in range(2)]
    args = (q, k, v, w, mix[0], w2, mix[1])
    got = npf(ops.mta_fused_fwd(*[t.to(DEV) for t in args]))
    _lib.device_status()
    assert_parity(got, orc.mta_fwd(*[npf(t) for t in args], True, ROUND[dtype]), dtype, f"S={S} {R}x{Sk}")


# the conv alone and its input gradient: a result may be off by half a unit in its last place (2^-8 or 2^-11 of it) and by the float32 sum of
# up to 272 products, 272 * 2^-24 of their magnitudes, which add up to about 11
@pytest.mark.parametrize("S,R,Sk,causal,dtype,w32", [(107, 6, 11, True, torch.bfloat16, False), (108, 6, 11, False, torch.float16, False),
                                                     (113, 6, 11, True, torch.float16, True), (225, 6, 11, False, torch.bfloat16, False),
                                                     (129, 1, 1, True, torch.bfloat16, False), (112, 2, 4, True, torch.bfloat16, False),
                                                     (69, 16, 17, True, torch.bfloat16, True), (137, 16, 17, False, torch.float16, True),
                                                     (233, 11, 15, True, torch.bfloat16, False)])
def test_conv2d_tile_edges(S, R, Sk, causal, dtype, w32):
    g = torch.Generator(device=DEV).manual_seed(S * 100 + R)
    x = torch.randn(2, 3, S, S, device=DEV, generator=g).to(dtype)
    w = (torch.randn(3, R, Sk, device=DEV, generator=g) * (R * Sk) ** -0.5).to(torch.float32 if w32 else dtype)
    nan = x.masked_fill(torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1), float("nan")) if causal else x
    pairs = [(ops.conv2d_fwd(nan, w, causal), conv64(x, w, causal))]
    if Sk % 2 == 1:
        pairs.append((ops.conv2d_bwd_input(nan, w, causal), conv64_bwd_input(x, w, causal)))
    _lib.device_status()
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in pairs:
        assert bool(((a.double() - b).abs() <= u * b.abs() + 2e-4).all())


# the conv attention: tiles of 80 keys, units of 4 (33 - R) rows
@pytest.mark.parametrize("S,R,Sk,D,dtype,w32", [(1, 6, 11, 64, torch.bfloat16, False), (27, 6, 11, 128, torch.float16, False), (79, 6, 11, 128, torch.bfloat16, False),
                                                (81, 6, 11, 64, torch.bfloat16, True), (109, 6, 11, 128, torch.bfloat16, False), (161, 1, 1, 128, torch.float16, False),
                                                (129, 2, 3, 64, torch.bfloat16, False), (137, 16, 17, 128, torch.bfloat16, True), (241, 16, 17, 64, torch.float16, False),
                                                (321, 11, 15, 128, torch.bfloat16, False)])
def test_conv_attention_tile_edges(S, R, Sk, D, dtype, w32):
    g = torch.Generator().manual_seed(S * 100 + R)
    q, k, v = (torch.randn(2, 4, S, D, generator=g).to(dtype) for _ in range(3))
    w = (torch.randn(4, R, Sk, generator=g) * (R * Sk) ** -0.5).to(torch.float32 if w32 else dtype)
    _lib.reset_launch_count()
    got = npf(ops.conv_attn_fwd(*[t.to(DEV) for t in (q, k, v, w)], True, D ** -0.5))
    assert _lib.launch_count() == 1
    _lib.device_status()
    assert_parity(got, orc.conv_attn_fwd(*[npf(t) for t in (q, k, v, w)], True, None, orc.ROUND_NONE), dtype, f"S={S} {R}x{Sk}")
