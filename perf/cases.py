"""Timing cases of the library: what a Clef-Omni engine has it do, through `OmniBackend`.

Three kinds of pass:
  block   one MoE block, `begin` + `encode_moe`, on activations that are in device memory.  Short
          batches are decode steps and server micro-batches, long ones packed prefill.
  layers  a decoder pass over a packed batch of records: the residual stream is filled with the
          embeddings, then `encode_layer` (attention half, norm, MoE block) runs for each layer.
          Two layers stand for the model's 48, as all of them cost the same.
  host    one MoE block on activations in page-locked host memory, `forward_host`: uploads, block
          and download, synchronous.

Geometry everywhere: hidden 2048, 128 experts, top-8, intermediate 768, 32 query and 4 key/value
heads of 128; BF16 weights N(0, 0.02), BF16 activations N(0, 1), FP32 residual stream.  A caller
waits (`complete`) once per model pass, so the passes here end without it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cleffa_b200 import OmniBackend, workloads

H, F, E, TOP = workloads.H, workloads.F, workloads.E, workloads.TOP
QKV, ATTN = 5120, 4096          # columns of the q|k|v projection and of the attention output
HEADS, HEAD_DIM = 32, 128
MAX_TOKENS = 16384              # the most tokens of one attention pass, and of one arena pass of the block
LAYERS = 2


def listed():
    return [
        # one decode step of one user: eight experts' weights, launches and latency
        dict(name="block, 1 token", kind="block", tokens=1, records=1, skew=False),
        # a small server micro-batch: about half of the experts are touched
        dict(name="block, 9 tokens", kind="block", tokens=9, records=1, skew=False),
        # a full micro-batch: every expert's weights are streamed for a few rows each
        dict(name="block, 128 tokens", kind="block", tokens=128, records=1, skew=False),
        # one short prompt, an odd number of tokens
        dict(name="block, 511 tokens", kind="block", tokens=511, records=1, skew=False),
        # packed prefill of eight prompts, the benchmark's own workload
        dict(name="block, 4096 tokens", kind="block", tokens=4096, records=8, skew=False),
        # routing as skewed as it gets: Zipf(1.2) popularity, the hottest expert at ten times the mean
        dict(name="block, 8192 tokens, skewed", kind="block", tokens=8192, records=1, skew=True),
        # one long prompt, the largest arena pass
        dict(name="block, 16384 tokens", kind="block", tokens=MAX_TOKENS, records=1, skew=False),
        # a short utterance through whole layers
        dict(name="layers, 37 tokens", kind="layers", tokens=37, records=1, skew=False),
        # a few short prompts of ragged lengths
        dict(name="layers, 1030 tokens, 6 records", kind="layers", tokens=1030, records=6, skew=False),
        # packed prefill of eight prompts through whole layers
        dict(name="layers, 4096 tokens, 8 records", kind="layers", tokens=4096, records=8, skew=False),
        # one long document: causal attention over 16384 keys
        dict(name="layers, 16384 tokens", kind="layers", tokens=MAX_TOKENS, records=1, skew=False),
        # an engine whose activations live in host memory
        dict(name="host, 4096 tokens", kind="host", tokens=4096, records=8, skew=False),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    case = _draw(rng)
    while any(all(known[k] == v for k, v in case.items()) for known in listed()):
        case = _draw(rng)
    return case


def _draw(rng):
    kind = rng.choices(("block", "layers", "host"), weights=(5, 4, 1))[0]
    tokens = _log_int(rng, *((64, 8192) if kind == "host" else (1, MAX_TOKENS)))
    records = rng.randint(1, max(1, min(16, tokens // 16)))
    return dict(kind=kind, tokens=tokens, records=records, skew=kind == "block" and tokens >= 1024 and rng.random() < 0.3)


class State:
    """A program's context, its bound weights and one batch."""

    def __init__(self, backend):
        self.backend = backend

    def __del__(self):
        self.backend.close()


_stream = None


def _use_stream():
    """The stream that the program's own work and the library's kernels share."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    torch.cuda.set_stream(_stream)
    return _stream.cuda_stream


def _bounds(case, seed):
    return workloads.varlen_bounds(seed, case["tokens"], case["records"])


def prepare(case, seed):
    T, n_layer = case["tokens"], LAYERS if case["kind"] == "layers" else 1
    state = State(OmniBackend(0, stream=_use_stream()))
    b = state.backend
    b.reserve(T, n_layer=n_layer)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, mean=0.0, std=0.02, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device="cuda").normal_(mean, std, generator=g)

    bias = torch.from_numpy(workloads.zipf_bias(seed)).cuda() if case["skew"] else None
    for layer in range(n_layer):
        b.bind_layer(layer, normal(E, H), normal(E, 2 * F, H), normal(E, H, F), bias=bias)
    state.bounds = _bounds(case, seed)
    if case["kind"] == "layers":
        ones = dict(mean=1.0, std=0.1, dtype=torch.float32)
        for layer in range(n_layer):
            b.bind_attention(layer, normal(H, **ones), normal(QKV, H), normal(H, ATTN), normal(HEAD_DIM, **ones), normal(HEAD_DIM, **ones))
            b.bind_norm(layer, normal(H, **ones))
        state.pos = torch.from_numpy(np.ascontiguousarray(workloads.make_positions(seed, state.bounds).T)).cuda()
        state.embeddings = normal(T, H, std=1.0, dtype=torch.float32)
        state.x = torch.empty_like(state.embeddings)
    else:
        state.xn = normal(T, H, std=1.0)
        state.x = torch.zeros(T, H, dtype=torch.float32, device="cuda")
        if case["kind"] == "host":
            state.xn, state.x = state.xn.cpu().pin_memory(), state.x.cpu().pin_memory()
    state.run = {"block": _run_block, "layers": _run_layers, "host": _run_host}[case["kind"]]
    return state


def _run_block(s):
    s.backend.begin()
    s.backend.encode_moe(0, s.xn, s.x, s.bounds)


def _run_layers(s):
    s.backend.begin()
    s.x.copy_(s.embeddings)
    for layer in range(LAYERS):
        s.backend.encode_layer(layer, s.x, s.pos, s.bounds)


def _run_host(s):
    s.backend.forward_host(0, s.xn, s.x, s.bounds)


def run(state):
    """One pass; the block adds into the residual `x`, which is its output."""
    state.run(state)
    return state.x


def _experts_touched(tokens, skew):
    """Expected number of experts that at least one of the tokens is routed to."""
    if not skew:
        return E * (1.0 - (1.0 - TOP / E) ** tokens)
    # router logits are N(0, 0.02 * sqrt(2048)) plus the bias; its permutation does not matter
    logits = np.random.default_rng(0).normal(0.0, 0.02 * math.sqrt(H), (512, E)) + workloads.zipf_bias(0)
    chosen = np.argsort(-logits, axis=1)[:, :TOP]
    share = np.bincount(chosen.ravel(), minlength=E) / len(logits)
    return float((1.0 - (1.0 - np.clip(share, 0.5 / len(logits), 1.0)) ** tokens).sum())


def work(case):
    T, layers = case["tokens"], LAYERS if case["kind"] == "layers" else 1
    weights = 2 * E * H + _experts_touched(T, case["skew"]) * 2 * 3 * F * H
    flops = T * (2 * E * H + TOP * 2 * 3 * F * H)
    tokens = 4 * H + 4 * H                               # the residual in and out
    if case["kind"] == "layers":
        weights += 2 * (QKV * H + H * ATTN)
        lengths = np.diff(_bounds(case, 0)).astype(np.float64)
        flops += T * 2 * (QKV * H + H * ATTN) + 4 * HEAD_DIM * HEADS * float((lengths * (lengths + 1) / 2).sum())
    else:
        tokens += 2 * H                                  # the normed activations
    return dict(bytes=layers * weights + T * tokens, flops=layers * flops)


def tolerance(case):
    # BF16 operands and BF16 intermediates (h and the experts' outputs; q, k, v and the attention
    # output): 2.4e-3 to 4e-3 against FP64.  Single elements: a few times the rounding step of the
    # largest values; in a second layer also a token whose eighth expert changes at a near tie (its
    # weight of about 0.08 times an expert output of up to 5 standard deviations of 0.3, twice).
    return dict(rel=5e-3, max=0.25 if case["kind"] == "layers" else 0.1)
