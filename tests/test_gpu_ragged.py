"""Sequence lengths that are no multiple of anything: the 16-bit forward keeps its score planes with padded rows, so the
tensor-core kernels take them too.  The workspace is filled with NaN bit patterns first: nothing in the padding, above the
diagonal or left over from another call may reach the result."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from multitokenatention_triton_b200.synthetic import MTAWorkload, make_mta_inputs
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, npf

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("S,H,D,cq,ck,dtype", [
    (1, 8, 64, 3, 5, torch.bfloat16), (65, 16, 128, 6, 11, torch.bfloat16), (127, 12, 64, 6, 11, torch.float16),
    (129, 64, 64, 2, 3, torch.bfloat16), (201, 16, 128, 11, 15, torch.bfloat16), (259, 32, 64, 7, 9, torch.float16)])
def test_forward_ragged(S, H, D, cq, ck, dtype):
    wl = MTAWorkload("ragged", 2, H, S, D, cq, ck, 3, 3, dtype, seed=900 + S, random_post_conv=True)
    inp = make_mta_inputs(wl)
    args = [inp[k].to(DEV) for k in ("q", "k", "v", "w1", "W1", "w2", "W2")]
    nbytes = _lib.lib().mta_workspace_bytes(2, H, S, D, cq, ck, 3, 3, 0, S, _lib.dtype_code(args[0]))
    ws = torch.full((nbytes,), 255, dtype=torch.uint8, device=DEV)
    out = ops.mta_fused_fwd(*args, True, workspace=ws)
    _lib.device_status()
    a = [npf(inp[k]) for k in ("q", "k", "v", "w1", "W1", "w2", "W2")]
    assert_parity(npf(out), orc.mta_fwd(*a, True, ROUND[dtype]), dtype, f"S{S} H{H} D{D} {cq}x{ck}")
