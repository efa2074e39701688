"""The score + conv kernel at the edges of its tiles: 4 (33 - R) query rows in four groups of 33 - R, 112 keys."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, npf

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
