"""The float32 products in their forms for few and for many tiles: a sum does not depend on the form, so the bits are the same."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from util import max_abs, npf

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("S,D", [(4, 64), (64, 32), (68, 64), (132, 128), (260, 64), (320, 36)])
def test_few_tiles_equal_many(S, D):
    g = torch.Generator(device=DEV).manual_seed(S + D)
    q, k, v = (torch.randn(4, 60, S, D, device=DEV, generator=g) for _ in range(3))       # 240 planes: many tiles
    s, p = ops.qk_scores_fwd(q, k, D ** -0.5, causal=True), torch.randn(4, 60, S, S, device=DEV, generator=g)
    o = ops.pv_fwd(p, v, causal=True)
    for b, h in ((0, 0), (3, 57)):
        few = slice(b, b + 1), slice(h, h + 2)
        assert torch.equal(ops.qk_scores_fwd(q[few].contiguous(), k[few].contiguous(), D ** -0.5, causal=True).tril(), s[few].tril())
        assert torch.equal(ops.pv_fwd(p[few].contiguous(), v[few].contiguous(), causal=True), o[few])
    _lib.device_status()
    dead = torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1)
    ref = torch.matmul(q.double(), k.double().transpose(2, 3)) * D ** -0.5
    assert max_abs(npf(s.tril()), npf(ref.masked_fill(dead, 0.0))) <= 1e-4 and max_abs(npf(o), npf(torch.matmul(p.double().masked_fill(dead, 0.0), v.double()))) <= 1e-3
