"""The work a user of this library has it do, as cases that can be timed and compared.

A case is one pass of the mixture-of-experts feed-forward layer (or of a short stack of
them, or of the dense block of the same architecture) through the public entry points of
``biv_b200.moe``, on weights in the GGUF block formats and rows as a model's norm leaves
them.  The listed cases span what an inference engine asks for: one token of one
conversation, a batch of decode steps, the verification of drafted tokens through several
layers, prompts from a few hundred to many thousand rows, rows that live in host memory, the
dense block.  ``draw`` gives more of the same ranges.

  call    "moe"     rows on the device, a new output, the caller's current stream
          "moe_"    rows and output kept by the caller, on the engine's one stream (the layers
                    of a model run one after another there)
          "host"    page-locked host rows in, host rows out, finished on return
          "stack"   layers one after another on the residual, norm included, on that stream
          "dense"   the dense feed-forward block
"""
import math

import numpy as np
import torch

from biv_b200 import workloads as W
from biv_b200.moe import Moe, MoeStack

# the weight types of the benchmark's configurations: (gate and up, down)
TYPES = {"q4_k": (W.Q4_K, W.Q4_K), "q4_k/q6_k": (W.Q4_K, W.Q6_K), "q5_k/q6_k": (W.Q5_K, W.Q6_K),
         "q8_0": (W.Q8_0, W.Q8_0), "bf16": (W.BF16, W.BF16)}
# how unequal the experts' popularity is: all alike; a N(0, 1) bias of the router's logits;
# the benchmark's Zipf(1.1) bias
SKEWS = ("balanced", "normal", "zipf")
EPS = 1e-6
_DEV = "cuda:0"


def _moe(name, call, types, tokens, skew="balanced", layers=1, n_embd=2048, n_expert=256, k=8, ff=512):
    c = dict(call=call, types=types, tokens=tokens, skew=skew, layers=layers, n_embd=n_embd,
             n_expert=n_expert, k=k, ff=ff)
    return dict(c, name=name) if name else c


def _dense(name, types, tokens, n_embd, ff):
    return _moe(name, "dense", types, tokens, n_embd=n_embd, n_expert=1, k=1, ff=ff)


def listed():
    return [
        # one conversation, one token: latency, launches, the weights of eight experts
        _moe("decode_1_q4_k", "moe_", "q4_k", 1),
        # a server's decode step: 64 sequences, a token each, some experts much in demand
        _moe("decode_64_q4_k", "moe_", "q4_k", 64, "normal"),
        # 32 sequences x 5 drafted tokens verified through four layers of the model
        _moe("verify_160_q5_k_x4", "stack", "q5_k/q6_k", 160, layers=4),
        # a small batch of an engine that keeps its activations on the host
        _moe("host_16_q8_0", "host", "q8_0", 16),
        # unquantised experts, a batch too small for one row per expert
        _moe("decode_33_bf16", "moe_", "bf16", 33),
        # a prompt of ordinary, ragged length on the commonest mix of 4-bit files
        _moe("prompt_509_q4_k_q6_k", "moe", "q4_k/q6_k", 509),
        # a long prompt, Zipf-skewed experts
        _moe("prompt_4096_q8_0", "moe", "q8_0", 4096, "zipf"),
        # the largest pass: unquantised experts, many prompts at once
        _moe("prompt_16384_bf16", "moe", "bf16", 16384),
        # the same kind of pass for rows that come from and go back to host memory
        _moe("host_8192_bf16", "host", "bf16", 8192),
        # the dense block: one token, and a ragged prompt
        _dense("dense_1_q4_k", "q4_k", 1, 4096, 12288),
        _dense("dense_300_q8_0", "q8_0", 300, 4096, 12288),
    ]


def _log_uniform(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    types = rng.choice(sorted(TYPES))
    call = rng.choice(["moe", "moe", "moe_", "moe_", "host", "stack", "dense"])
    # quantised layers up to a long prompt, unquantised ones up to the largest pass
    most = 16384 if types == "bf16" else 4096
    if call == "dense":
        return _dense(None, types, _log_uniform(rng, 1, 512), rng.choice([1024, 2048, 4096]),
                      rng.choice([3072, 6144, 8192, 12288]))
    skew = rng.choice(SKEWS)
    n_expert, k = rng.choice([(64, 6), (128, 8), (256, 8)])
    n_embd, ff = rng.choice([(1024, 512), (2048, 512), (2048, 768)])
    if call == "stack":
        layers = rng.randint(2, 4)
        return _moe(None, call, types, _log_uniform(rng, 1, 512), skew, layers, min(n_embd, 2048),
                    min(n_expert, 128) if types == "bf16" else n_expert, k, 512)
    if call == "host":
        most //= 2
    return _moe(None, call, types, _log_uniform(rng, 1, most), skew, 1, n_embd, n_expert, k, ff)


# --------------------------------------------------------------------------
# inputs

def _host(t):
    """Device bytes as a numpy array: what a mapped model file is to the library."""
    buf = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    buf.copy_(t)
    return buf.numpy().reshape(-1)


def _uniform_f16(g, n, lo, hi):
    return torch.empty(n, device=_DEV).uniform_(lo, hi, generator=g).half()


def _weights(g, ty, n, rows, cols):
    """``n`` matrices of weights with a standard deviation of about 0.02, a model's."""
    if ty in (W.Q4_K, W.Q5_K, W.Q6_K):
        bb = W.row_size(ty, 256)
        nblk = n * rows * cols // 256
        raw = torch.randint(-2**31, 2**31 - 1, ((nblk * bb + 3) // 4,), dtype=torch.int32, device=_DEV,
                            generator=g).view(torch.uint8)[:nblk * bb].view(nblk, bb)
        # uniform quants and sub-block scales (6 bits; 8 signed bits for Q6_K): the block
        # scale puts the values where a model's are, the minimum's scale centres them
        if ty == W.Q6_K:
            raw[:, 208:210] = _uniform_f16(g, nblk, 1.0e-5, 2.0e-5).view(nblk, 1).view(torch.uint8)
        else:
            half = 7.5 if ty == W.Q4_K else 15.5
            d = _uniform_f16(g, nblk, 0.45e-3 / half, 0.75e-3 / half)
            raw[:, 0:2] = d.view(nblk, 1).view(torch.uint8)
            raw[:, 2:4] = (d.float() * half).half().view(nblk, 1).view(torch.uint8)
        return W.ExpertStack(ty, cols, rows, n, _host(raw))
    if ty == W.BF16:
        w = torch.empty(n * rows * cols, dtype=torch.bfloat16, device=_DEV).normal_(0, 0.02, generator=g)
        return W.ExpertStack(ty, cols, rows, n, _host(w.view(torch.uint8)))
    assert ty == W.Q8_0
    w = torch.empty(n * rows * cols // 32, 32, device=_DEV).normal_(0, 0.02, generator=g)
    d = w.abs().amax(dim=1, keepdim=True) / 127
    raw = torch.empty(w.shape[0], 34, dtype=torch.uint8, device=_DEV)
    raw[:, 0:2] = d.half().view(torch.uint8)
    raw[:, 2:] = (w / d).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    return W.ExpertStack(ty, cols, rows, n, _host(raw))


def _bias(rng, skew, n_expert):
    if skew == "normal":
        return rng.standard_normal(n_expert)
    if skew == "zipf":
        return -1.1 * W.ZIPF_ALPHA * np.log(rng.permutation(n_expert) + 1.0)
    return np.zeros(n_expert)


def _layer(g, c, seed):
    rng = np.random.default_rng(seed)
    gate_ty, down_ty = TYPES[c["types"]]
    e, ne, ff = c["n_embd"], c["n_expert"], c["ff"]
    router = rng.standard_normal((ne, e), dtype=np.float32) * np.float32(0.02)
    router[:, 0] = _bias(rng, c["skew"], ne)     # column 0 of the rows is the constant 1
    layer = W.MoeLayer(e, ne, c["k"], ff, ff, router, gate=_weights(g, gate_ty, ne, ff, e),
                       up=_weights(g, gate_ty, ne, ff, e), down=_weights(g, down_ty, ne, e, ff))
    layer.sh_gate, layer.sh_up = _weights(g, gate_ty, 1, ff, e), _weights(g, gate_ty, 1, ff, e)
    layer.sh_down = _weights(g, down_ty, 1, e, ff)
    layer.sh_gate_inp = rng.standard_normal(e, dtype=np.float32) * np.float32(0.02)
    return layer


class _State:
    pass


_engine_streams = []


def _engine_stream():
    if not _engine_streams:
        _engine_streams.append(torch.cuda.Stream(_DEV))
    return _engine_streams[0]


def prepare(case, seed):
    c, n, e = case, case["tokens"], case["n_embd"]
    g = torch.Generator(device=_DEV).manual_seed(seed)
    s = _State()
    s.call = c["call"]
    s.stream = _engine_stream() if s.call in ("moe_", "stack") else None
    x = torch.empty(n, e, device=_DEV).normal_(generator=g)
    h = x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + EPS)      # as the norm leaves the rows
    h[:, 0] = 1.0
    if s.call == "dense":
        gate_ty, down_ty = TYPES[c["types"]]
        s.layers = [Moe.dense(_weights(g, gate_ty, 1, c["ff"], e), _weights(g, gate_ty, 1, c["ff"], e),
                              _weights(g, down_ty, 1, e, c["ff"]), n)]
    else:
        s.layers = [Moe(_layer(g, c, seed * 64 + l), n) for l in range(c["layers"])]
    s.h = h
    if s.call == "moe_":
        s.out = torch.empty_like(h)
    elif s.call == "host":
        s.h = torch.empty(n, e, pin_memory=True)
        s.h.copy_(h)
        s.out = torch.empty(n, e, pin_memory=True)
    elif s.call == "stack":
        w = 1.0 + 0.1 * np.random.default_rng(seed).standard_normal((c["layers"], e))
        w[:, 0] = 1.0
        for m, row in zip(s.layers, w):
            m.set_post_norm(row, EPS)
        s.h = x
        s.h[:, 0] = 1.0
        s.out = torch.empty_like(x)
        s.stack = MoeStack(s.layers)
    torch.cuda.synchronize()
    return s


def run(s):
    m = s.layers[0]
    if s.call in ("moe", "dense"):
        return m.moe(s.h)
    if s.call == "host":
        return m.moe_host(s.h, s.out)
    with torch.cuda.stream(s.stream):
        if s.call == "moe_":
            return m.moe_(s.h, s.out, accumulate=False)
        s.out.copy_(s.h)          # the residual as the layers before left it
        return s.stack.forward_(s.out)


# --------------------------------------------------------------------------
# what a pass cannot do without

def _experts_hit(c):
    """Distinct experts a batch selects, from the distribution of the router's logits."""
    if c["call"] == "dense":
        return 1
    rng = np.random.default_rng(0)
    n = min(c["tokens"], 2048)
    sigma = 0.02 * math.sqrt(c["n_embd"])
    logits = _bias(rng, c["skew"], c["n_expert"]) + sigma * rng.standard_normal((n, c["n_expert"]))
    return len(np.unique(np.argpartition(-logits, c["k"] - 1, axis=1)[:, :c["k"]]))


def work(case):
    c = case
    n, e, ff, ne = c["tokens"], c["n_embd"], c["ff"], c["n_expert"]
    gate_ty, down_ty = TYPES[c["types"]]
    expert = 2 * ff * W.row_size(gate_ty, e) + e * W.row_size(down_ty, ff)
    shared, routed = (0, 1) if c["call"] == "dense" else (1, c["k"])
    weights = (_experts_hit(c) + shared) * expert + (ne + 1) * e * 4 * shared
    flops = 2.0 * n * (routed + shared) * 3 * e * ff + 2.0 * n * (ne + 1) * e * shared
    # the rows come in once and go out once, however many layers they pass
    return {"bytes": c["layers"] * weights + 2 * n * e * 4, "flops": c["layers"] * flops}


def tolerance(case):
    if case["call"] == "stack":
        # a rounding difference in one layer can move a top-k choice of the next
        return {"rel": 3e-3, "max": 2e-1}
    if case["types"] == "bf16":
        # bf16 weights on f32 rows, which the path keeps to about 2^-17
        return {"rel": 1e-4, "max": 1e-3}
    # the SwiGLU rows are quantised to int8: a rounding difference in the products before moves
    # a value by one step now and then, and with it that expert's output for the token
    return {"rel": 1e-3, "max": 1e-2}
