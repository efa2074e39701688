"""Sequence lengths that are no multiple of anything: the 16-bit forward keeps its score planes with padded rows, so the
tensor-core kernels take them too.  The workspace is filled with NaN bit patterns first: nothing in the padding, above the
diagonal or left over from another call may reach the result."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib, ops
from multitokenatention_triton_b200.synthetic import MTAWorkload, make_mta_inputs
from oracle import mta_oracle as orc
from util import ROUND, assert_parity, conv64, conv64_bwd_input, npf, rel_fro

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


# The stand-alone ops on rows that are not 16-byte aligned, from the size on at which they work on copies with padded rows (1M to 8M scores),
# against the CUDA-core kernels; the first and last elements of the tensors lie inside a 16-byte piece.
@pytest.mark.parametrize("S,H,causal,dtype,offset", [
    (1025, 4, True, torch.bfloat16, 0), (839, 6, False, torch.float16, 3), (1502, 2, True, torch.float16, 0), (1023, 16, True, torch.bfloat16, 1),
    (515, 64, True, torch.bfloat16, 0), (390, 14, False, torch.bfloat16, 5)])
def test_stand_alone_ops_on_unaligned_rows(S, H, causal, dtype, offset):
    g = torch.Generator(device=DEV).manual_seed(S)
    x, gr = (torch.randn(H * S * S + offset, device=DEV, generator=g).to(dtype)[offset:].view(1, H, S, S) for _ in range(2))
    upper = torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1)
    if causal:
        for t in (x, gr):
            t.masked_fill_(upper, float("nan"))
    w = (torch.randn(H, 6, 11, device=DEV, generator=g) / 8).to(dtype)
    mix = torch.randn(H, H, device=DEV, generator=g).to(dtype)
    got = {}
    for variant in (0, 1):
        _lib.set_variant("conv2d", variant)
        _lib.set_variant("head_linear", variant)
        try:
            got[variant] = (ops.conv2d_fwd(x, w, causal), ops.conv2d_bwd_input(gr, w, causal), ops.head_linear_fwd(x, mix, causal, -3.3),
                            ops.head_linear_bwd_input(gr, mix, causal), ops.conv2d_bwd_weight(x, gr, (6, 11), causal),
                            ops.head_linear_bwd_weight(x, gr, causal))
        finally:
            _lib.set_variant("conv2d", 0)
            _lib.set_variant("head_linear", 0)
    _lib.device_status()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got[0][:4], got[1][:4]):
        assert float((a.float() - b.float()).abs().max()) <= 2 * ulp * float(b.float().abs().max())
        if causal:
            assert torch.equal(a.masked_select(upper), b.masked_select(upper))
    for a, b in zip(got[0][4:], got[1][4:]):
        assert rel_fro(npf(a), npf(b)) <= 1e-4


@pytest.mark.parametrize("S,H,causal,dtype,offset", [
    (1025, 4, True, torch.bfloat16, 0), (839, 6, False, torch.float16, 3), (1502, 2, True, torch.float16, 0), (1023, 16, True, torch.bfloat16, 1),
    (515, 64, True, torch.bfloat16, 0), (390, 14, False, torch.bfloat16, 5)])
def test_stand_alone_ops_on_unaligned_rows_against_float64(S, H, causal, dtype, offset):
    """A result plane may be off by its own rounding (half a unit in the last of 8 or 11 significant bits, so 2^-8 or 2^-11 of it)
    and by a float32 sum of up to 66 products; a weight gradient by float32 sums of a block, whose errors do not add up over the
    blocks."""
    g = torch.Generator(device=DEV).manual_seed(S)
    x, gr = (torch.randn(H * S * S + offset, device=DEV, generator=g).to(dtype)[offset:].view(1, H, S, S) for _ in range(2))
    w = (torch.randn(H, 6, 11, device=DEV, generator=g) / 8).to(dtype)
    mix = (torch.randn(H, H, device=DEV, generator=g) * H ** -0.5).to(dtype)
    got = (ops.conv2d_fwd(x, w, causal), ops.conv2d_bwd_input(gr, w, causal), ops.head_linear_fwd(x, mix, causal, -3.5),
           ops.head_linear_bwd_input(gr, mix, causal))
    dw, dmix = ops.conv2d_bwd_weight(x, gr, (6, 11), causal), ops.head_linear_bwd_weight(x, gr, causal)
    _lib.device_status()
    dead = torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1)
    xd, gd = x.double(), gr.double()
    if causal:
        xd, gd = xd.masked_fill(dead, 0.0), gd.masked_fill(dead, 0.0)
    mixed = torch.einsum("oh,bhpq->bopq", mix.double(), xd), torch.einsum("oh,bopq->bhpq", mix.double(), gd)
    if causal:
        mixed[0].masked_fill_(dead, -3.5)
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got, (conv64(xd, w, causal), conv64_bwd_input(gd, w, causal), *mixed)):
        assert bool(((a.double() - b).abs() <= u * b.abs() + 1e-4).all())
    xp = torch.nn.functional.pad(xd, (5, 5, 5, 0))
    want = torch.stack([torch.stack([(xp[:, :, i:i + S, j:j + S] * gd).sum((0, 2, 3)) for j in range(11)], -1) for i in range(6)], -2)
    assert float((dw.double() - want).norm() / want.norm()) <= 1e-5
    want = torch.einsum("bopq,bhpq->oh", gd, xd)
    assert float((dmix.double() - want).norm() / want.norm()) <= 1e-5


def test_stand_alone_ops_without_room_for_copies(monkeypatch):
    """Two more planes than the result needs are not to be had: the ops run as they do without copies."""
    S, H = 1025, 16
    x, g = (torch.randn(1, H, S, S, device=DEV).to(torch.bfloat16) for _ in range(2))
    w, mix = torch.randn(H, 6, 11, device=DEV).to(torch.bfloat16), torch.randn(H, H, device=DEV).to(torch.bfloat16)
    L, st, shape, bf16 = _lib.lib(), torch.cuda.current_stream().cuda_stream, (1, H, S, S), _lib.MTA_BF16
    want = [torch.empty_like(x) for _ in range(4)] + [torch.empty(H, 6, 11, device=DEV), torch.empty(H, H, device=DEV)]
    conv_ws, mix_ws = L.mta_conv2d_bwd_weight_workspace_bytes(*shape, 6, 11), L.mta_head_linear_bwd_weight_workspace_bytes(H)
    ws = torch.empty(max(conv_ws, mix_ws), dtype=torch.uint8, device=DEV)
    y = [t.data_ptr() for t in want]
    for rc in (L.mta_conv2d_fwd(x.data_ptr(), w.data_ptr(), y[0], *shape, 6, 11, 1, bf16, bf16, st),
               L.mta_conv2d_bwd_input(x.data_ptr(), w.data_ptr(), y[1], *shape, 6, 11, 1, bf16, bf16, st),
               L.mta_head_linear_fwd(x.data_ptr(), mix.data_ptr(), y[2], *shape, 1, -3.5, bf16, bf16, st),
               L.mta_head_linear_bwd_input(x.data_ptr(), mix.data_ptr(), y[3], *shape, 1, bf16, bf16, st),
               L.mta_conv2d_bwd_weight(x.data_ptr(), g.data_ptr(), y[4], ws.data_ptr(), conv_ws, *shape, 6, 11, 1, bf16, st),
               L.mta_head_linear_bwd_weight(x.data_ptr(), g.data_ptr(), y[5], ws.data_ptr(), mix_ws, *shape, 1, bf16, st)):
        _lib.check(rc, "without a workspace")
    real = torch.empty

    def empty(*a, **k):
        if k.get("dtype") == torch.uint8 and a[0] >= 2 * x.numel() * 2:
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*a, **k)

    monkeypatch.setattr(torch, "empty", empty)
    got = [ops.conv2d_fwd(x, w, True), ops.conv2d_bwd_input(x, w, True), ops.head_linear_fwd(x, mix, True, -3.5),
           ops.head_linear_bwd_input(x, mix, True), ops.conv2d_bwd_weight(x, g, (6, 11), True), ops.head_linear_bwd_weight(x, g, True)]
    monkeypatch.undo()
    _lib.device_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("S,variant", [(960, 2), (961, 3), (1021, 3), (1024, 3), (2048, 3), (2049, 2)])
def test_lengths_of_one_padded_row_take_one_head_mix(S, variant):
    """The second head mix of 16 heads, where it is a kernel of its own (the second conv is not small), is chosen by the padded row: bit for bit
    what the kernel of that row gives, not the other's."""
    g = torch.Generator(device=DEV).manual_seed(S)
    q, k, v = (torch.randn(1, 16, S, 64, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w = torch.randn(16, 3, 5, device=DEV, generator=g).to(torch.bfloat16)
    mix = torch.randn(16, 16, device=DEV, generator=g).to(torch.bfloat16)
    out = {}
    for n in (0, 2, 3):
        _lib.set_variant("head_linear", n)
        try:
            out[n] = ops.mta_fused_fwd(q, k, v, w, mix, w, mix)
        finally:
            _lib.set_variant("head_linear", 0)
    _lib.device_status()
    assert torch.equal(out[0], out[variant]) and not torch.equal(out[2], out[3])
