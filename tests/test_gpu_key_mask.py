"""A boolean (batch, keys) mask on the fused causal forward (mta_masked_fwd) against the masked oracle: padding on either side,
holes, sequences with no key at all for their first queries, lengths around the 32-key words and the 128-key tiles, head counts
and dtypes on and off the tensor-core head mix."""
import numpy as np
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from multitokenatention_triton_b200.synthetic import MTAWorkload, make_mta_inputs
from oracle import mta_oracle as orc
from util import assert_parity, npf

pytestmark = pytest.mark.gpu
DEV = "cuda"


def key_mask(S, seed):
    """Right padding, left padding, holes, everything kept."""
    g = torch.Generator().manual_seed(seed)
    keep = torch.ones(4, S, dtype=torch.bool)
    keep[0, max(1, S * 2 // 3):] = False
    keep[1, :S // 3] = False
    keep[2] = torch.rand(S, generator=g) < 0.6
    return keep


@pytest.mark.parametrize("S,H,D,cq,ck,dtype", [
    (1, 8, 64, 3, 5, torch.bfloat16), (31, 16, 64, 3, 3, torch.float16), (33, 12, 64, 6, 11, torch.bfloat16), (96, 64, 64, 2, 3, torch.bfloat16),
    (129, 16, 128, 6, 11, torch.bfloat16), (300, 8, 64, 7, 9, torch.float16), (65, 16, 32, 3, 5, torch.float32), (130, 12, 36, 6, 11, torch.float32),
    (72, 7, 33, 3, 3, torch.float32)])
def test_key_mask(S, H, D, cq, ck, dtype):
    wl = MTAWorkload("keymask", 4, H, S, D, cq, ck, 3, 3, dtype, seed=700 + S, random_post_conv=True)
    inp = make_mta_inputs(wl)
    keep = key_mask(S, S)
    names = ("w1", "W1", "w2", "W2")
    out = ops.mta_masked_fwd(*(inp[x].to(DEV) for x in ("q", "k", "v")), keep.to(DEV), *(inp[x].to(DEV) for x in names))
    _lib.device_status()
    dead = ~keep[:, None, None, :] | torch.ones(S, S, dtype=torch.bool).triu(1)
    full = torch.zeros(4, H, S, S).masked_fill_(dead.expand(4, H, S, S), float("-inf"))
    with np.errstate(all="ignore"):
        ref = orc.mta_fwd_masked(*(npf(inp[x]) for x in ("q", "k", "v", *names)), npf(full), True)
    assert np.isfinite(npf(out)).all()
    assert_parity(npf(out), ref, dtype, f"S{S} H{H}")


def test_float32_weights_with_16_bit_activations():
    wl = MTAWorkload("keymask", 4, 16, 136, 64, 3, 5, 3, 3, torch.bfloat16, seed=5, random_post_conv=True)
    inp = make_mta_inputs(wl)
    keep = key_mask(136, 9).to(DEV)
    args = [inp[x].to(DEV) for x in ("q", "k", "v")]
    w = [inp[x].to(DEV) for x in ("w1", "W1", "w2", "W2")]
    a = ops.mta_masked_fwd(*args, keep, *w)
    b = ops.mta_masked_fwd(*args, keep, *(t.float() for t in w))
    _lib.device_status()
    assert_parity(npf(b), npf(a), torch.bfloat16, "float32 weights")
