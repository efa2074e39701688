"""The second conv and the second head mix as one kernel (small convs)."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, npf, rel_fro

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(B, H, S, D, cq2, ck2, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, H, S, D, generator=g).to(dtype) for _ in range(3))
    w1 = (torch.randn(H, 3, 5, generator=g) * 15 ** -0.5).to(dtype)
    w2 = (torch.randn(H, cq2, ck2, generator=g) * (cq2 * ck2) ** -0.5).to(dtype)
    mix = [(torch.eye(H) + 0.02 ** 0.5 * torch.randn(H, H, generator=g)).to(dtype) for _ in range(2)]
    return q, k, v, w1, mix[0], w2, mix[1]


# one tile of 128 keys and two, the first key of a tile, rows that are no multiple of a group; every number of heads and conv it takes
@pytest.mark.parametrize("H,S,cq2,ck2,dtype", [(16, 1, 3, 3, torch.bfloat16), (16, 9, 3, 3, torch.float16), (32, 127, 2, 3, torch.bfloat16), (64, 65, 3, 3, torch.float16),
                                               (8, 256, 3, 3, torch.bfloat16), (8, 273, 2, 3, torch.float16), (16, 257, 3, 3, torch.bfloat16),
                                               (16, 385, 3, 3, torch.float16), (16, 300, 2, 3, torch.bfloat16), (32, 258, 3, 3, torch.float16),
                                               (32, 391, 2, 3, torch.bfloat16), (64, 259, 3, 3, torch.bfloat16), (64, 263, 2, 3, torch.float16)])
def test_against_the_oracle(H, S, cq2, ck2, dtype):
    args = _inputs(1, H, S, 128, cq2, ck2, dtype, S + H)
    dev = [t.to(DEV) for t in args]
    _lib.set_stage_trace(True)
    try:
        got = ops.mta_fused_fwd(*dev)
        assert [n for n, _ in _lib.stage_times_ms()][-2:] == ["conv2+head_mix2", "pv"]
    finally:
        _lib.set_stage_trace(False)
    part, lo, hi = torch.zeros_like(got), S // 7, max(S - 3, S // 7 + 1)
    ops.mta_fused_fwd(*dev, True, rows=(lo, hi), out=part)
    _lib.device_status()
    assert_parity(npf(got), orc.mta_fwd(*[npf(t) for t in args], True, ROUND[dtype]), dtype, f"H={H} S={S} {cq2}x{ck2}")
    assert torch.equal(part[:, :, lo:hi], got[:, :, lo:hi]), "a row range gives the same bits"


# both round the conv's output and the mix's to 16 bits and sum in float32, in another order: some results round the other way
@pytest.mark.parametrize("B,H,S,dtype", [(3, 16, 640, torch.bfloat16), (1, 16, 1300, torch.float16), (2, 32, 511, torch.bfloat16), (1, 64, 700, torch.float16)])
def test_against_the_two_kernels(B, H, S, dtype):
    args = [t.to(DEV) for t in _inputs(B, H, S, 128, 3, 3, dtype, S)]
    one = ops.mta_fused_fwd(*args)
    try:
        _lib.set_variant("conv2d", 3)
        _lib.set_variant("fused", 3)
        two = ops.mta_fused_fwd(*args)
    finally:
        _lib.set_variant("conv2d", 0)
        _lib.set_variant("fused", 0)
    _lib.device_status()
    assert rel_fro(npf(one), npf(two)) <= (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)


@pytest.mark.parametrize("H,S,D", [(8, 64, 64), (8, 128, 128), (16, 128, 64), (16, 1024, 64), (16, 128, 128)])
def test_the_choice_does_not_depend_on_the_head_dimension(H, S, D):
    args = [t.to(DEV) for t in _inputs(1, H, S, D, 3, 3, torch.bfloat16, S + D)]
    _lib.set_stage_trace(True)
    try:
        ops.mta_fused_fwd(*args)
        assert [n for n, _ in _lib.stage_times_ms()][-2:] == ["conv2+head_mix2", "pv"]
    finally:
        _lib.set_stage_trace(False)
