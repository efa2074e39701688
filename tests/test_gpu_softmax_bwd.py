"""The softmax gradient's rows in registers: 1, 2, 4 or 8 chunks a lane by the row length, and longer rows walked twice.  The gradients
of q and k (whole, and of the last, longest rows) against autograd in float64 at lengths just up to and past each step."""
import pytest
import torch

from multitokenatention_triton_b200 import _lib
from multitokenatention_triton_b200.autograd_ops import MTAFunction
from test_gpu_train import torch_mta

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("S,dtype", [(256, torch.bfloat16), (264, torch.float16), (519, torch.bfloat16), (1024, torch.float16),
                                     (1025, torch.bfloat16), (2048, torch.bfloat16), (2056, torch.float16), (128, torch.float32),
                                     (132, torch.float32), (260, torch.float32), (513, torch.float32), (1024, torch.float32),
                                     (1028, torch.float32)])
def test_rows(S, dtype):
    H, D = 8, 32
    g = torch.Generator(device=DEV).manual_seed(S)
    x = [torch.randn(1, H, S, D, device=DEV, generator=g).to(dtype) for _ in range(3)]
    ws = []
    for shape in ((H, 2, 3), (H, H), (H, 2, 3), (H, H)):
        w = torch.randn(shape, device=DEV, generator=g) * 0.1
        if len(shape) == 2:
            w += torch.eye(H, device=DEV)
        else:
            w[:, -1, 1] += 1.0
        ws.append(w.to(dtype))
    up = torch.randn(1, S, H, D, device=DEV, generator=g).to(dtype)
    ins = [t.detach().requires_grad_() for t in (x[0], x[1], x[2], *ws)]
    out = MTAFunction.apply(*ins).transpose(1, 2)
    out.backward(up)
    _lib.device_status()
    ref_in = [t.detach().double().requires_grad_() for t in ins]
    torch_mta(*ref_in).backward(up.double())
    tol = {torch.float32: 2e-5, torch.float16: 6e-3, torch.bfloat16: 4e-2}[dtype]      # the bounds of the whole training step
    for i in (0, 1):
        got, want = ins[i].grad.double(), ref_in[i].grad
        assert float((got - want).norm() / want.norm()) <= tol
    got, want = ins[0].grad[:, :, -8:].double(), ref_in[0].grad[:, :, -8:]
    assert float((got - want).norm() / want.norm()) <= 2 * tol


@pytest.mark.parametrize("S,dtype", [(31, torch.bfloat16), (256, torch.bfloat16), (257, torch.float16), (519, torch.bfloat16), (1024, torch.bfloat16),
                                     (1033, torch.float16), (2056, torch.bfloat16), (128, torch.float32), (135, torch.float32),
                                     (513, torch.float32), (1024, torch.float32), (1029, torch.float32)])
def test_every_chunk_counts_once(S, dtype):
    """Entry by entry.  Queries of 0 make a row's probabilities 1 / n; the convs and mixes are identities; the values of a head are 0 but for eight
    neighbouring keys, which alone make up the row's dot product; keys with a single 1 hand the gradient of 64 scores to one entry of dq each."""
    H, D, G = 8, 64, 1024.0
    g = torch.Generator(device=DEV).manual_seed(S)
    first = [min(max(k, 0), S - 8) for k in (0, 124, 248, 256, S // 2 // 8 * 8, (S - 1) // 8 * 8, S - 16, S - 8)]
    q, k, v = (torch.zeros(1, H, S, D, device=DEV, dtype=dtype) for _ in range(3))
    seen = torch.zeros(H, D, dtype=torch.long, device=DEV)
    for h, f in enumerate(first):
        v[0, h, f:f + 8, 0] = (1 + torch.rand(8, device=DEV, generator=g)).to(dtype)
        at = torch.cat([torch.arange(f, f + 8, device=DEV), torch.randperm(S, device=DEV, generator=g)[:D - 8]])
        seen[h, :len(at)] = at
        for j, key in enumerate(at.tolist()):
            k[0, h, key, j] = 1.0
    up = torch.zeros(1, S, H, D, device=DEV, dtype=dtype)
    up[..., 0] = G
    ins = [t.requires_grad_() for t in (q, k, v)]
    w, mix = torch.ones(H, 1, 1, device=DEV, dtype=dtype), torch.eye(H, device=DEV, dtype=dtype)
    MTAFunction.apply(*ins, w, mix, w, mix).transpose(1, 2).backward(up)
    _lib.device_status()
    n = torch.arange(1, S + 1, device=DEV, dtype=torch.float64)[None, :, None]
    below = torch.ones(S, S, dtype=torch.bool, device=DEV).tril()
    dp = (G * v[0, :, :, 0].detach().double())[:, None, :] * below                      # [head, query, key]
    dot = dp.sum(-1, keepdim=True) / n
    pick = seen[:, None, :].expand(H, S, D)
    live = below.expand(H, S, S).gather(2, pick)
    filled = torch.arange(D, device=DEV) < min(D, 8 + S)
    want = ((dp.gather(2, pick) - dot) / n * live * filled) * D ** -0.5
    # p (twice: in the dot and in front), the result and dq are rounded once each; the exponential, its sum and the dot in float32
    u = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    bound = (5 * u + 2.0 ** -18) * (dp.gather(2, pick) + dot) / n * D ** -0.5
    assert bool(((ins[0].grad[0].double() - want).abs() <= bound + 1e-30).all())
