"""The work that users of this package have it do, as cases that can be timed one by one.

Every case is one call (or one forward + backward) of a public module, with the inputs resident on the GPU:

  forward    MTAAttentionTriton under no_grad: prefill and evaluation
  train      MTAAttentionTriton, output and the gradients of q, k, v and all four weights: a training step's share
  masked     MTAAttentionTriton(use_mask=True) under no_grad with a (batch, keys) padding mask: a batch of sequences of
             different lengths
  conv       Conv2dTriton alone on a score plane; with `grad`, forward and both gradients
  head_mix   TritonLinearHead alone on probabilities; with `grad`, forward and both gradients
  conv_attn  TritonConvAttention: softmax(scale * conv(Q K^T)) V

All are causal, as in the reference's benchmarks.  Sizes are those of the package's five workloads, of the sweep in
benchmark_seq_len.py and of the reference's published sweeps; `draw` spreads over the same ranges, lengths that are no
multiple of anything among them.
"""
import types

import torch

from multitokenatention_triton_b200 import Conv2dTriton, MTAAttentionTriton, TritonConvAttention, TritonLinearHead

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}


def _case(name, op, dtype, batch, heads, seq, dim=128, kernel=(6, 11), kernel2=(3, 3), grad=False):
    c = {"op": op, "dtype": dtype, "batch": batch, "heads": heads, "seq": seq, "dim": dim, "cq": kernel[0], "ck": kernel[1],
         "cq2": kernel2[0], "ck2": kernel2[1], "grad": grad}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short prompt: launches and host time count
        _case("forward_s128_bf16", "forward", "bf16", 1, 16, 128, kernel2=(6, 11)),
        # the small float32 configuration the parity suite starts from
        _case("forward_s256_fp32", "forward", "fp32", 2, 8, 256, dim=64, kernel=(3, 5)),
        # a prompt length as it comes: odd, no multiple of a tile
        _case("forward_s1021_bf16", "forward", "bf16", 2, 16, 1021),
        # the half-precision point of the reference's published sweep
        _case("forward_s2048_fp16", "forward", "fp16", 1, 16, 2048, kernel=(7, 7), kernel2=(7, 7)),
        # the float32 point of the published sweep
        _case("forward_s2048_fp32", "forward", "fp32", 1, 16, 2048, dim=64, kernel=(11, 15), kernel2=(11, 15)),
        # the headline configuration: long prompts, eight at a time
        _case("forward_s4096_bf16", "forward", "bf16", 8, 16, 4096),
        # a training step at the end of the sequence-length sweep
        _case("train_s1024_bf16", "train", "bf16", 4, 16, 1024, kernel2=(6, 11), grad=True),
        # a float32 training step of the published sweep
        _case("train_s1024_fp32", "train", "fp32", 1, 16, 1024, dim=64, kernel=(11, 15), kernel2=(11, 15), grad=True),
        # four prompts of different lengths, padded on the right
        _case("masked_s1024_bf16", "masked", "bf16", 4, 16, 1024),
        # the conv on its own, as a layer of a model that is trained
        _case("conv_s2048_bf16", "conv", "bf16", 4, 16, 2048, grad=True),
        # the head mix on its own, likewise
        _case("head_mix_s2048_bf16", "head_mix", "bf16", 4, 16, 2048, grad=True),
        # the conv attention at the headline shape
        _case("conv_attn_s4096_bf16", "conv_attn", "bf16", 8, 16, 4096),
    ]


# The most entries of all score planes together (batch * heads * seq^2) of a drawn case.
LIMIT = {"forward": 1 << 30, "conv_attn": 1 << 30, "train": 1 << 26, "masked": 1 << 26, "conv": 1 << 28, "head_mix": 1 << 28}


def draw(rng):
    op = rng.choice(["forward", "forward", "forward", "train", "train", "masked", "conv", "head_mix", "conv_attn"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    heads = rng.choice([8, 12, 16, 16, 32, 64])
    kernel = rng.choice([(2, 3), (3, 5), (3, 9), (4, 7), (5, 5), (6, 11), (6, 11), (7, 7), (7, 9), (11, 15)])
    grad = op == "train" or (op in ("conv", "head_mix") and rng.random() < 0.5)
    limit = LIMIT[op] >> (3 if dtype == "fp32" and op in ("forward", "conv_attn") else 0)
    longest = min(4096, int((limit / heads) ** 0.5))
    seq = round(64 * (longest / 64) ** rng.random())
    if rng.random() < 0.5:
        seq = max(64, seq // 64 * 64)
    fits = max(1, min(8, limit // (heads * seq * seq)))
    batch = rng.randint(1, fits)
    return _case(None, op, dtype, batch, heads, seq, dim=rng.choice([64, 128]), kernel=kernel,
                 kernel2=kernel if rng.random() < 0.5 else (3, 3), grad=grad)


def _conv_kernel(g, heads, rows, cols):
    """Random taps plus one on the current query and key."""
    w = torch.randn(heads, rows, cols, device="cuda", generator=g) * (rows * cols) ** -0.5
    w[:, rows - 1, cols // 2] += 1.0
    return w


def _mix(g, heads):
    return torch.eye(heads, device="cuda") + 0.02 ** 0.5 * torch.randn(heads, heads, device="cuda", generator=g)


def _module(case):
    h = case["heads"]
    if case["op"] == "conv":
        return Conv2dTriton(h, (case["cq"], case["ck"]), causal=True)
    if case["op"] == "head_mix":
        return TritonLinearHead(h, causal=True)
    if case["op"] == "conv_attn":
        return TritonConvAttention(h, (case["cq"], case["ck"]), causal=True)
    mta = types.SimpleNamespace(use_mta=True, query_kernel_size=case["cq"], key_kernel_size=case["ck"],
                                after_sm_query_kernel_size=case["cq2"], after_sm_key_kernel_size=case["ck2"],
                                pre_sm_linear_head=True, post_sm_linear_head=True, pad_key="both", init_method="identity",
                                dim=h * case["dim"])
    return MTAAttentionTriton(h, mta, dropout=0.0, causal=True, use_mask=case["op"] == "masked")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    b, h, s, d = case["batch"], case["heads"], case["seq"], case["dim"]
    m = _module(case).to("cuda", dtype)
    m.train(case["grad"])
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 2:
                p.copy_(_mix(g, h))
            else:
                p.copy_(_conv_kernel(g, h, p.shape[1], p.shape[2]))
    q, k, v = (torch.randn(b, h, s, d, device="cuda", generator=g).to(dtype) for _ in range(3))
    mask = upstream = None
    if case["op"] == "conv":
        inputs = [torch.matmul(q, k.transpose(2, 3)) * d ** -0.5]
    elif case["op"] == "head_mix":
        # causal rows that sum to one, zero above the diagonal; plane by plane, for the float32 temporaries' sake
        dead = torch.ones(s, s, device="cuda", dtype=torch.bool).triu(1)
        probs = torch.empty(b, h, s, s, device="cuda", dtype=dtype)
        for n in range(b):
            logits = torch.randn(h, s, s, device="cuda", generator=g).masked_fill_(dead, float("-inf"))
            probs[n] = torch.softmax(logits, dim=-1)
        inputs = [probs]
    else:
        inputs = [q, k, v]
    if case["op"] == "masked":
        lengths = torch.randint(s // 2, s + 1, (b, 1), device="cuda", generator=g)
        mask = torch.arange(s, device="cuda")[None, :] < lengths
    if case["grad"]:
        inputs = [t.requires_grad_() for t in inputs]
        shape = (b, s, h, d) if case["op"] == "train" else (b, h, s, s)
        upstream = torch.randn(shape, device="cuda", generator=g).to(dtype)
    return {"op": case["op"], "module": m, "inputs": inputs, "mask": mask, "upstream": upstream, "scale": d ** -0.5}


def _call(state):
    m, inputs = state["module"], state["inputs"]
    if state["op"] in ("forward", "train", "masked"):
        return m(*inputs, state["mask"], None)
    if state["op"] == "conv_attn":
        return m(*inputs, True, state["scale"])[0]
    return m(*inputs)


def run(state):
    if state["upstream"] is None:
        with torch.no_grad():
            return _call(state)
    leaves = state["inputs"] + list(state["module"].parameters())
    for t in leaves:
        t.grad = None
    out = _call(state)
    out.backward(state["upstream"])
    return [out.detach()] + [t.grad for t in leaves]


def work(case):
    b, h, s, d, e = case["batch"], case["heads"], case["seq"], case["dim"], SIZE[case["dtype"]]
    lower, full = b * h * s * (s + 1) // 2, b * h * s * s
    conv1, conv2, mix = 2 * case["cq"] * case["ck"], 2 * case["cq2"] * case["ck2"], 2 * h
    if case["op"] == "conv":
        per, weights, bytes_ = conv1, h * case["cq"] * case["ck"], e * (lower + full)
    elif case["op"] == "head_mix":
        per, weights, bytes_ = mix, h * h, e * (lower + full)
    elif case["op"] == "conv_attn":
        per, weights, bytes_ = 4 * d + conv1, h * case["cq"] * case["ck"], e * 4 * b * h * s * d
    else:
        per, weights = 4 * d + conv1 + conv2 + 2 * mix, h * (case["cq"] * case["ck"] + case["cq2"] * case["ck2"] + 2 * h)
        bytes_ = e * 4 * b * h * s * d
        if case["op"] == "masked":
            bytes_ += b * s
    bytes_ += e * weights
    flops = per * lower
    if case["grad"]:
        # the upstream gradient in, a gradient of every input and weight out; every product has two gradients
        bytes_ = 2 * bytes_
        flops = 3 * flops
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # 16-bit paths round at every stage; float32 is sums of up to a few thousand terms and one exponential
    rel = {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]
    return {"rel": 2 * rel if case["op"] == "train" else rel}
