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
