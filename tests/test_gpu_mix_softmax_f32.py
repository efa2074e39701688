"""Head mix + softmax in float32 as one kernel: the edges of its rows and groups of threads, against float64."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one thread's keys and one more, one pass of a CTA's threads and one more, the longest rows that fit; head counts around the paddings
@pytest.mark.parametrize("N,C,S,scale", [(2, 1, 4, 1.0), (1, 8, 5, 1.0), (1, 3, 127, 1.0), (2, 8, 516, 1.0), (1, 16, 1028, 3.0), (1, 12, 260, 1.0), (1, 16, 2052, 1.0),
                                         (1, 17, 132, 1.0), (1, 32, 516, 1.0), (1, 33, 260, 1.0), (1, 64, 256, 2.0), (1, 64, 860, 1.0), (1, 64, 864, 1.0)])
def test_against_float64(N, C, S, scale):
    g = torch.Generator(device=DEV).manual_seed(S * 100 + C)
    x = torch.randn(N, C, S, S, device=DEV, generator=g) * scale
    W = torch.eye(C, device=DEV) + 0.1 * torch.randn(C, C, device=DEV, generator=g)
    dead = torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1)
    got = ops.head_linear_softmax_fwd(x.masked_fill(dead, float("nan")), W)
    _lib.device_status()
    logits = torch.einsum("oh,nhpk->nopk", W.double(), x.double())
    want = torch.softmax(logits.masked_fill(dead, float("-inf")), dim=-1)
    # a logit is off by up to C + 1 roundings of the sum of its terms' magnitudes, at most 2^-24 each; a probability by twice that (its own and
    # the row's largest), the exponential's 2^-21 of |logit - largest| <= 2^-17 and a few roundings
    bound = 2 * (C + 1) * 2.0 ** -24 * torch.einsum("oh,nhpk->nopk", W.abs().double(), x.abs().double()).amax(-1, keepdim=True) + 2.0 ** -17
    assert bool(((got.double() - want).abs() <= bound * want + 1e-30).all())
    assert bool((got.masked_select(dead) == 0).all())
