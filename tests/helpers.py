"""Shared by the parity tests: error measures of the reference's tests/verify.py:10-11."""
import math

import numpy as np
import torch
from torch.nn import functional as F

from oracle.model import specification


def relative(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12))


def max_relative(a, b):
    """Largest elementwise error relative to the largest reference magnitude."""
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-30))


def evaluation_in_64_bits(arch, flat, x, y):
    """Logits and the flat gradient of the mean loss of a GPT (`Arch.gpt`) in 64 bits, on the GPU."""
    flat, device = torch.as_tensor(flat).cuda().double(), "cuda"
    x, y = (torch.as_tensor(v.astype(np.int64)).to(device) for v in (x, y))
    offset, p = 0, {}
    for name, shape in specification(arch):
        n = math.prod(shape)
        p[name], offset = flat[offset:offset + n].reshape(shape).clone().requires_grad_(), offset + n
    (B, T), W, D = x.shape, arch.width, arch.width // arch.heads
    mask = torch.ones(T, T, dtype=torch.bool, device=device).tril()
    norm = lambda h, name: F.layer_norm(h, (W,), p[name + "w"], p[name + "b"], 1e-5)
    h = F.embedding(x, p["embedding"])
    for l in range(arch.depth):
        q, k, v = [t.reshape(B, T, arch.heads, D).transpose(1, 2) for t in F.linear(norm(h, f"{l}.ln1"), p[f"{l}.qkv"]).split(W, -1)]
        scores = (q @ k.transpose(-1, -2) / math.sqrt(D)).masked_fill(~mask, -math.inf)
        h = h + F.linear((torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(B, T, W), p[f"{l}.attention"])
        h = h + F.linear(F.gelu(F.linear(norm(h, f"{l}.ln2"), p[f"{l}.gate"])), p[f"{l}.projection"])
    logits = F.linear(norm(h, "final"), p["embedding"])
    F.cross_entropy(logits.flatten(0, 1), y.flatten()).backward()
    return logits.detach().cpu().numpy(), torch.cat([p[name].grad.flatten() for name, _ in specification(arch)]).cpu().numpy()
