"""A kernel that starts while its predecessor still runs must not work on what a predecessor that gave up has left.

The predecessor is a kernel whose bounded wait, limited to a few milliseconds, runs out: the call behind it passes the host's
check, its first kernel starts early, and the flag goes up only then.  Nothing may be written and the next call is refused."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
N, H, S, D, R, K = 1, 16, 256, 128, 6, 11
BF16 = _lib.MTA_BF16


def _rand(*shape):
    return torch.randn(*shape, device=DEV).to(torch.bfloat16)


def _calls():
    """name -> (call(out pointer, stream), bytes of the buffer its tcgen05 kernel writes first)"""
    L = _lib.lib()
    p = {"x": _rand(N, H, S, S), "g": _rand(N, H, S, S), "q": _rand(N, H, S, D), "k": _rand(N, H, S, D), "v": _rand(N, H, S, D),
         "w": _rand(H, R, K), "W": _rand(H, H), "o": _rand(N, H, S, D), "dw": torch.zeros(H * max(R * K, H), device=DEV)}
    a = {n: t.data_ptr() for n, t in p.items()}
    plane, heads = N * H * S * S * 2, N * H * S * D * 2
    conv_ws = L.mta_conv2d_bwd_weight_workspace_for(N, H, S, S, R, K, BF16)
    mix_ws = L.mta_head_linear_bwd_weight_workspace_for(N, H, S, S, BF16)
    fused_ws = L.mta_workspace_bytes(N, H, S, D, R, K, R, K, 0, S, BF16)
    calls = {
        "conv2d": (lambda y, st: L.mta_conv2d_fwd(a["x"], a["w"], y, N, H, S, S, R, K, 1, BF16, BF16, st), plane),
        "conv2d_mma": (lambda y, st: L.mta_conv2d_fwd(a["x"], a["w"], y, N, H, S, S, R, K, 1, BF16, BF16, st), plane),
        "conv2d_bwd_input": (lambda y, st: L.mta_conv2d_bwd_input(a["x"], a["w"], y, N, H, S, S, R, K, 1, BF16, BF16, st), plane),
        "head_linear": (lambda y, st: L.mta_head_linear_fwd(a["x"], a["W"], y, N, H, S, S, 1, 0.0, BF16, BF16, st), plane),
        "head_linear_softmax": (lambda y, st: L.mta_head_linear_softmax_fwd(a["x"], a["W"], y, N, H, S, S, BF16, BF16, st), plane),
        "qk_scores": (lambda y, st: L.mta_qk_scores_fwd(a["q"], a["k"], y, N, H, S, D, 1.0, 1, 1, BF16, st), plane),
        "pv": (lambda y, st: L.mta_pv_fwd(a["x"], a["v"], y, N, H, S, D, 1, BF16, st), heads),
        "conv_attn": (lambda y, st: L.mta_conv_attn_fwd(a["q"], a["k"], a["v"], a["w"], y, 0, 0, N, H, S, D, R, K, 1, 1.0, BF16, BF16, st),
                      heads),
        # the kernels below write slots or planes of the workspace, which later kernels of the call read
        "conv2d_bwd_weight": (lambda y, st: L.mta_conv2d_bwd_weight_as(a["x"], a["g"], a["dw"], _lib.MTA_F32, y, conv_ws, N, H, S, S, R,
                                                                       K, 1, BF16, st), conv_ws),
        "head_linear_bwd_weight": (lambda y, st: L.mta_head_linear_bwd_weight_as(a["x"], a["g"], a["dw"], _lib.MTA_F32, y, mix_ws, N, H,
                                                                                 S, S, 1, BF16, st), mix_ws),
        "fused": (lambda y, st: L.mta_fused_fwd(a["q"], a["k"], a["v"], a["w"], a["W"], a["w"], a["W"], a["o"], y, fused_ws, N, H, S, D,
                                                R, K, R, K, 0, S, 1, BF16, BF16, st), plane),
    }
    return p, calls


@pytest.mark.parametrize("name", ["conv2d", "conv2d_mma", "conv2d_bwd_input", "head_linear", "head_linear_softmax", "qk_scores", "pv", "conv_attn",
                                  "conv2d_bwd_weight", "head_linear_bwd_weight", "fused"])
def test_the_successor_of_a_kernel_that_gave_up_writes_nothing(name):
    keep, calls = _calls()
    call, nbytes = calls[name]
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    room = max(nbytes, L.mta_workspace_bytes(N, H, S, D, R, K, R, K, 0, S, BF16))
    good = torch.zeros(room, dtype=torch.uint8, device=DEV)
    buf = torch.full((room,), 0x5A, dtype=torch.uint8, device=DEV)
    # the kernels without bounded waits, such as the mma.sync head mix, carry on
    _lib.set_variant("head_linear", 3 if name in ("head_linear", "fused") else 0)
    _lib.set_variant("conv2d", 2 if name == "conv2d_mma" else 0)
    try:
        _lib.check(call(good.data_ptr(), st), name)          # a first call also does what only a first call does
        _lib.device_status()
        for _ in range(5):                                   # a host that pauses longer than the wait has its call refused
            _lib.check(L.mta_inject_late_wait_timeout(st), "inject")
            rc = call(buf.data_ptr(), st)
            assert L.mta_device_status(st) == 4
            if rc != 4:
                break
        _lib.check(rc, name)
    finally:
        _lib.set_variant("head_linear", 0)
        _lib.set_variant("conv2d", 0)
        L.mta_device_status(st)
    assert bool((buf[:nbytes] == 0x5A).all()), "written after the predecessor gave up"
    _lib.check(call(buf.data_ptr(), st), name)               # and afterwards the call works again
    _lib.device_status()
    assert bool((buf[:nbytes] != 0x5A).any())
    del keep
