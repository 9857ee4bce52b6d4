"""The work a user of this framework has it do, as cases that can be timed and compared.

Seven kinds of call, each through the public interface (`turbogpt_b200.bridge`, or the C ABI where the
caller keeps device pointers or pinned buffers):

  reference   training the reference architecture (width 16, arg-max attention, SwiGLU, Muon) the way its
              host program does: a chunk of steps under OneCycle, the chunk's losses, the weights
  train       training a GPT: a chunk of steps, its losses, and a snapshot of the weights in pinned memory
  host        training a GPT on batches the caller streams from pinned host memory, losses after every step
  batch       one evaluation with logits, losses and all gradients on the host, BF16 or FP32
  predict     the next-byte logits of one context, host call to host logits (the sampling loop's call)
  projection  one linear layer's three products on device tensors: y, dx and dw
  attention   causal attention forward and backward on device tensors

`listed()` names the sizes of the repository's own configurations and tests; `draw()` takes sizes from the
whole range those stand for.
"""
import ctypes
import math

import numpy as np
import torch

from turbogpt_b200 import bridge
from turbogpt_b200.bridge import Config, ConfigEx, Native

CORPUS = 1 << 20  # bytes of the training corpus
MOST_FLOPS = 1.5e14  # of a drawn training pass; the long-context case below is the largest at 1.8e14


def listed():
    return [
        # The smallest training call: the reference architecture at its own test's size (64 tokens a step),
        # where a step is launches and latency.
        dict(name="reference-tiny", kind="reference", depth=4, context=4, batch=16, steps=32),
        # The reference host's shipped experiment: batch 2880, context 4.
        dict(name="reference-experiment", kind="reference", depth=4, context=4, batch=2880, steps=32),
        # The 4-layer, 256-wide model that step-by-step comparisons are made on, as a BF16 and as an FP32
        # (check mode) evaluation that brings logits and every gradient back.
        dict(name="gradients-bf16", kind="batch", depth=4, width=256, hidden=1024, context=256, batch=8, fp32=False),
        dict(name="gradients-fp32", kind="batch", depth=4, width=256, hidden=1024, context=256, batch=8, fp32=True),
        # Training that same small model: 2048 tokens a step, an ordinary experiment on one GPU.
        dict(name="train-small", kind="train", depth=4, width=256, hidden=1024, context=256, batch=8, muon=False, steps=16),
        # Sizes off every tile: an odd batch, a context that is no multiple of 64, a width that is no multiple
        # of 256, a last partial tile of tokens; Muon on the hidden matrices.
        dict(name="train-ragged", kind="train", depth=6, width=384, hidden=1536, context=333, batch=7, muon=True, steps=4),
        # The main workload: 12 layers, d 768, context 1024, micro-batch 32, AdamW.
        dict(name="train-gpt", kind="train", depth=12, width=768, hidden=3072, context=1024, batch=32, muon=False, steps=8),
        # The larger, longer-context model with Muon.
        dict(name="train-long", kind="train", depth=16, width=1024, hidden=4096, context=4096, batch=8, muon=True, steps=3),
        # A caller that feeds its own bytes and reads the losses after every step, at a small micro-batch.
        dict(name="train-host-bytes", kind="host", depth=12, width=768, hidden=3072, context=1024, batch=4, muon=False, steps=4),
        # Sampling from the main model: one context in, 256 logits out; latency.
        dict(name="predict", kind="predict", depth=12, width=768, hidden=3072, context=1024),
        # The kernel calls at the main workload's sizes: the MLP's up projection and its two gradients,
        # attention forward and backward.
        dict(name="projection", kind="projection", tokens=32768, out=3072, width=768),
        dict(name="attention", kind="attention", batch=32, heads=12, context=1024),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["reference", "train", "train", "host", "batch", "predict", "projection", "attention"])
    if kind == "reference":
        context = rng.randint(2, 16)
        unit = 16 // math.gcd(16, context)  # the engine takes whole 16-token groups
        batch = max(1, _log_int(rng, 16, 4096) // unit) * unit
        return dict(kind=kind, depth=rng.randint(2, 8), context=context, batch=max(batch, 4), steps=rng.choice([8, 16, 32]))
    if kind == "projection":
        return dict(kind=kind, tokens=_log_int(rng, 256, 65536), out=8 * _log_int(rng, 16, 512), width=8 * _log_int(rng, 16, 512))
    if kind == "attention":
        context = _log_int(rng, 64, 4096)
        heads = rng.randint(2, 16)
        return dict(kind=kind, batch=max(1, min(64, int(_log_int(rng, 1024, 65536) / context))), heads=heads, context=context)
    width = 64 * rng.randint(2, 16)
    depth = rng.randint(2, 16)
    hidden = width * 4 if rng.random() < 0.7 else 64 * rng.randint(width // 64, width // 16)
    if kind == "predict":
        return dict(kind=kind, depth=depth, width=width, hidden=hidden, context=_log_int(rng, 64, 2048))
    if kind == "batch":
        width = 64 * rng.randint(2, 8)
        context = _log_int(rng, 32, 512)
        return dict(kind=kind, depth=rng.randint(2, 6), width=width, hidden=4 * width, context=context,
                    batch=max(1, _log_int(rng, 256, 4096) // context), fp32=rng.random() < 0.4)
    context = _log_int(rng, 64, 4096)
    steps = rng.choice([2, 3, 4])
    batch = max(1, _log_int(rng, 1024, 32768) // context)
    case = dict(kind=kind, depth=depth, width=width, hidden=hidden, context=context, batch=batch, muon=rng.random() < 0.4, steps=steps)
    while work(case)["flops"] > MOST_FLOPS:
        if case["batch"] > 1:
            case["batch"] //= 2
        else:
            case["depth"] //= 2
    return case


# ---------------------------------------------------------------------------------- inputs ---

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed & 0x7fffffff)


def _corpus(seed, size=CORPUS):
    """Order-2 Markov bytes with Dirichlet(0.1) transition rows; 4096 chains advance together."""
    g = _generator(seed)
    table = torch._standard_gamma(torch.full((65536, 256), 0.1, device="cuda"), generator=g) + 1e-30
    cdf = (table / table.sum(1, keepdim=True)).cumsum(1)
    chains = 4096
    a = torch.randint(0, 256, (chains,), generator=g, device="cuda")
    b = torch.randint(0, 256, (chains,), generator=g, device="cuda")
    out = torch.empty(size // chains, chains, dtype=torch.uint8, device="cuda")
    for t in range(size // chains):
        u = torch.rand(chains, 1, generator=g, device="cuda")
        c = (cdf[a * 256 + b] < u).sum(1).clamp_(max=255)
        out[t] = c
        a, b = b, c
    return out.t().contiguous().view(-1).cpu().numpy()


def _windows(data, seed, count, context):
    """`count` windows of the corpus and their successors, in pinned memory, as a data loader keeps them."""
    ends = np.random.default_rng(seed).integers(context, len(data) - 1, count)
    index = ends[:, None] - context + np.arange(context)[None]
    return torch.from_numpy(data[index]).pin_memory(), torch.from_numpy(data[index + 1]).pin_memory()


def _configuration(case, seed, batch):
    base = Config(depth=case["depth"], context=case["context"], batch=batch, learning_rate=3e-4, beta1=.9, beta2=.95,
                  weight_decay=.1, clip=1.0, seed=1 + seed % 100003, ns_steps=5)
    ex = ConfigEx.gpt(base, case["width"], case["width"] // 64, case["hidden"])
    ex.hidden_optimizer = bridge.HIDDEN_MUON if case.get("muon") else bridge.HIDDEN_ADAMW
    ex.precision = bridge.PRECISION_FP32 if case.get("fp32") else bridge.PRECISION_BF16
    return ex


def _weights(ex, seed):
    """N(0, 0.02) matrices, residual projections scaled by 1/sqrt(2 depth), unit norm scales, zero biases."""
    layout = bridge.parameter_layout(ex)
    w = torch.randn(bridge.load_library().tg_ex_parameter_count(ctypes.byref(ex)), generator=_generator(seed + 1), device="cuda") * .02
    vectors = 0
    for offset, rows, cols in layout[1:]:  # after the embedding
        if cols == 0:
            w[offset:offset + rows] = 1.0 - vectors % 2  # a norm's scale, then its bias
            vectors += 1
        elif rows == ex.width:
            w[offset:offset + rows * cols] *= (2 * ex.base.depth) ** -.5
    pinned = torch.empty(w.numel(), pin_memory=True)
    pinned.copy_(w)
    return pinned


class _Engine:
    """An engine and what its caller keeps beside it; the engine's memory goes back with the last reference."""

    def __init__(self, case, ex, weights):
        self.case = case
        self.native = Native(ex)
        self.weights = weights  # pinned: loaded from here, snapshots are written here
        self.native.check(self.native.lib.tg_set_weights(self.native.handle, weights.data_ptr()))

    def snapshot(self):
        self.native.check(self.native.lib.tg_get_weights(self.native.handle, self.weights.data_ptr()))
        return self.weights

    def __del__(self):
        if hasattr(self, "native"):
            self.native.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "projection":
        return _prepare_projection(case, seed)
    if kind == "attention":
        return _prepare_attention(case, seed)
    if kind == "reference":
        base = Config(depth=case["depth"], context=case["context"], batch=case["batch"], seed=1 + seed % 100003)
        ex = ConfigEx.reference(base)
        weights = torch.from_numpy(bridge.initialize_weights(ex)).pin_memory()
        state = _Engine(case, ex, weights)
        state.native.set_onecycle(1 << 19)
        state.native.set_data(_corpus(seed))
        return state
    ex = _configuration(case, seed, case.get("batch", 1))
    state = _Engine(case, ex, _weights(ex, seed))
    data = _corpus(seed)
    if kind == "train":
        state.native.set_data(data)
    elif kind == "host":
        x, y = _windows(data, seed, case["steps"] * case["batch"], case["context"])
        shape = (case["steps"], case["batch"], case["context"])
        state.x, state.y = x.numpy().reshape(shape), y.numpy().reshape(shape)
        state.keep = x, y
    else:
        x, y = _windows(data, seed, case.get("batch", 1), case["context"])
        state.x, state.y, state.keep = x.numpy(), y.numpy(), (x, y)
    return state


class _Tensors:
    pass


def _prepare_projection(case, seed):
    m, n, k = case["tokens"], case["out"], case["width"]
    g = _generator(seed)
    s = _Tensors()
    s.case = case
    s.x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    s.w = (torch.randn(n, k, generator=g, device="cuda") * k ** -.5).bfloat16()
    s.dy = torch.randn(m, n, generator=g, device="cuda").bfloat16()
    s.y = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    s.dx = torch.empty(m, k, device="cuda", dtype=torch.bfloat16)
    s.dw = torch.empty(n, k, device="cuda")
    return s


def _prepare_attention(case, seed):
    tokens, width = case["batch"] * case["context"], case["heads"] * 64
    g = _generator(seed)
    s = _Tensors()
    s.case = case
    s.qkv = torch.randn(tokens, 3 * width, generator=g, device="cuda").bfloat16()
    s.dout = torch.randn(tokens, width, generator=g, device="cuda").bfloat16()
    s.out = torch.empty(tokens, width, device="cuda", dtype=torch.bfloat16)
    s.lse = torch.empty(case["batch"], case["heads"], case["context"], device="cuda")
    s.dqkv = torch.empty_like(s.qkv)
    return s


# ------------------------------------------------------------------------------------ calls ---

def _check(status):
    if status < 0:
        raise RuntimeError(bridge.load_library().tg_error().decode())


def run(state):
    case = state.case
    kind = case["kind"]
    if kind in ("reference", "train"):
        state.native.train(case["steps"])
        return {"losses": state.native.training_losses(case["steps"]), "weights": state.snapshot()}
    if kind == "host":
        losses = [state.native.train_batch(x, y) for x, y in zip(state.x, state.y)]
        return {"losses": losses, "weights": state.snapshot()}
    if kind == "batch":
        logits, gradients, losses = state.native.batch(state.x, state.y)
        return {"logits": logits, "gradients": gradients, "losses": losses}
    if kind == "predict":
        return state.native.predict(state.x)
    lib, stream = bridge.load_library(), torch.cuda.current_stream().cuda_stream
    if kind == "projection":
        m, n, k = case["tokens"], case["out"], case["width"]
        _check(lib.tg_ex_gemm(state.x.data_ptr(), k, 1, state.w.data_ptr(), k, 1, state.y.data_ptr(), n, m, n, k, 0, 1, stream))
        _check(lib.tg_ex_gemm(state.dy.data_ptr(), n, 1, state.w.data_ptr(), 1, k, state.dx.data_ptr(), k, m, k, n, 0, 1, stream))
        _check(lib.tg_ex_gemm(state.dy.data_ptr(), 1, n, state.x.data_ptr(), 1, k, state.dw.data_ptr(), k, n, k, m, 1, 1, stream))
        return state.y, state.dx, state.dw
    sizes = case["batch"], case["context"], case["heads"], 64
    _check(lib.tg_ex_attention_forward(state.qkv.data_ptr(), state.out.data_ptr(), state.lse.data_ptr(), *sizes, 1, stream))
    _check(lib.tg_ex_attention_backward(state.qkv.data_ptr(), state.out.data_ptr(), state.dout.data_ptr(), state.lse.data_ptr(),
                                        state.dqkv.data_ptr(), *sizes, 1, stream))
    return state.out, state.lse, state.dqkv


# ------------------------------------------------------------------------------------- work ---

def _newton_schulz(rows, cols, steps=5):
    r, n = min(rows, cols), max(rows, cols)
    return steps * (4.0 * r * r * n + 2.0 * r ** 3)


def work(case):
    kind = case["kind"]
    if kind == "projection":
        m, n, k = case["tokens"], case["out"], case["width"]
        return {"bytes": 2.0 * (2 * m * k + 2 * m * n + n * k) + 4.0 * n * k, "flops": 6.0 * m * n * k}
    if kind == "attention":
        tokens, width, t = case["batch"] * case["context"], case["heads"] * 64, case["context"]
        return {"bytes": 2.0 * tokens * width * 8 + 4.0 * tokens * case["heads"],
                "flops": 7.0 * tokens * (t + 1) * width}  # 2 + 5 products over the causal half
    if kind == "reference":
        w, hd, depth, t = 16, 48, case["depth"], case["context"]
        matrices = depth * (4 * w * w + 3 * hd * w) + 256 * w
        tokens = case["batch"] * t
        parameters = depth * (4 * w * w + 3 * hd * w + 2 * w) + 2 * 256 * w + w
        step = tokens * (6.0 * matrices + 6.0 * (t + 1) / 2 * w * depth)
        step += depth * (_newton_schulz(3 * w, w) + _newton_schulz(w, w) + 3 * _newton_schulz(hd, w))
        return {"bytes": case["steps"] * (24.0 * parameters + 2.0 * tokens + 4.0 * t) + 4.0 * parameters,
                "flops": case["steps"] * step}
    w, hd, depth, t = case["width"], case["hidden"], case["depth"], case["context"]
    hidden_matrices = depth * (4 * w * w + 2 * hd * w)
    matrices = hidden_matrices + 256 * w
    parameters = matrices + (2 * depth + 1) * 2 * w
    tokens = case.get("batch", 1) * t
    forward = tokens * (2.0 * matrices + 2.0 * (t + 1) * w * depth)
    if kind == "predict":  # the head is needed at the last position only
        return {"bytes": 2.0 * parameters + t + 1024.0, "flops": forward - 2.0 * (tokens - 1) * 256 * w}
    backward = tokens * (4.0 * matrices + 5.0 * (t + 1) * w * depth)
    if kind == "batch":
        element = 4.0 if case["fp32"] else 2.0
        return {"bytes": element * parameters + 4.0 * parameters + tokens * (2.0 + 1024.0), "flops": forward + backward}
    step = forward + backward
    if case.get("muon"):
        step += depth * (_newton_schulz(3 * w, w) + _newton_schulz(w, w) + 2 * _newton_schulz(hd, w))
    return {"bytes": case["steps"] * (24.0 * parameters + 2.0 * tokens + 4.0 * t) + 4.0 * parameters,
            "flops": case["steps"] * step}


def tolerance(case):
    # FP32 check mode: FP32 products and sums throughout.  Everything else computes in BF16 (8 significant bits)
    # with FP32 sums, and returns BF16 tensors or FP32 values computed from BF16 activations.  Muon's Newton-Schulz
    # steps raise the small singular directions of a gradient to the size of the large ones, its rounding error with
    # them: starting weights that differ by 1e-6 end a chunk of 4 to 32 steps up to 0.7e-2 apart.
    if case.get("fp32"):
        return {"rel": 1e-5}
    return {"rel": 2e-2 if case["kind"] == "reference" or case.get("muon") else 1e-2}
