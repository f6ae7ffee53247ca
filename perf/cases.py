"""What is timed of this framework: the passes a program built on it makes, through its public entry points.

``listed()`` names twelve of them, ``draw(rng)`` gives one more of the same ranges.  Each case is a dict of plain values
with a ``kind``:

  causal         ``RFA.apply`` on given features, forward and backward (the boundary the headline number is quoted at)
  layer_train    one training step of a ``CausalAttention`` layer in fp16 with padded sequences: every gradient
  layer_prefill  the same layer without gradients (evaluation, scoring, the prompt of a generation)
  layer_decode   one token through the layer with its running state (``saved_state``)
  decode         one token for a large batch through ``ops.decode_step_fused`` (the serving loop's inner call)
  cross          encoder keys -> state -> decoder queries, from the per-head vectors, forward and backward, padded keys
  features       ``random_project`` alone, forward and backward

Inputs are N(0, 1) vectors, normalised by the feature map as the path itself does, and orthogonal random matrices from
``construct_random_matrices.orf``, one per head; padded sequences have lengths uniform in [T/2, T].
"""
import math

import numpy as np
import torch

from rfa_b200 import CausalAttention, ops
from rfa_b200.construct_random_matrices import orf
from rfa_b200.cross_attention import cross_rfa_query, cross_rfa_state
from rfa_b200.rfa import RFA
from rfa_b200.utils import SCALE, random_project

DEV = "cuda"


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # upstream's checking size and a debugging user's: a few heads, half a thousand tokens; launches and latency
        _causal("causal_small", 2, 4, 512),
        # machine translation, what upstream's package was written for: a batch of many short sentences
        _causal("causal_sentences", 96, 16, 45),
        # a language model's evaluation batch: few sequences, a length that is a multiple of nothing
        _causal("causal_ragged", 3, 12, 1531),
        # the headline workload
        _causal("causal_headline", 8, 16, 2048),
        # one long document, the longest the repository's benchmark runs
        _causal("causal_long", 1, 32, 131072),
        # a small model: 8 heads of 32, 32 random features pairs per head
        _causal("causal_d32", 8, 8, 1024, head_dim=32, proj_dim=32),
        # training step of a layer of a base-size decoder on a padded batch of sentences
        dict(name="layer_train", kind="layer_train", batch=24, heads=8, tokens=150, padded=True),
        # prompt pass of a large layer at the headline batch, padded
        dict(name="layer_prefill", kind="layer_prefill", batch=8, heads=16, tokens=2048, padded=True),
        # interactive generation: the smallest call a served model makes per layer and token
        dict(name="layer_decode", kind="layer_decode", batch=8, heads=16),
        # batch generation: the state of 4096 heads streams from memory for every token
        dict(name="decode_batch", kind="decode", batch=256, heads=16),
        # encoder-decoder training at the cross-attention workload of the benchmark
        dict(name="cross_train", kind="cross", batch=16, heads=16, queries=1024, keys=1024),
        # a single-precision program (a module used without .half(), a gradient check): the feature map in fp32
        dict(name="features_fp32", kind="features", batch=4, heads=16, tokens=1024, head_dim=64, proj_dim=64, dtype="float32"),
    ]


def _causal(name, batch, heads, tokens, head_dim=64, proj_dim=64):
    return dict(name=name, kind="causal", batch=batch, heads=heads, tokens=tokens, head_dim=head_dim, proj_dim=proj_dim)


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["causal"] * 5 + ["layer_train", "layer_prefill", "layer_decode", "decode", "cross", "cross", "features"])
    if kind == "causal":
        if rng.random() < 0.7:                       # the sizes the models use: 64 features pairs, heads of 64
            heads = rng.choice([4, 8, 12, 16, 32])
            tokens = _log(rng, 16, 131072)
            batch = _log(rng, 1, max(1, min(128, 4194304 // (heads * tokens))))
            head_dim, proj_dim = 64, 64
        else:                                        # other widths upstream's kernels take
            head_dim, proj_dim = rng.choice([(32, 32), (40, 48), (128, 64), (128, 128)])
            heads, tokens, batch = rng.choice([4, 8]), _log(rng, 16, 512), _log(rng, 1, 16)
        case = _causal("", batch, heads, tokens, head_dim, proj_dim)
        del case["name"]
        return case
    if kind in ("layer_train", "layer_prefill"):
        heads, tokens = rng.choice([8, 16]), _log(rng, 16, 2048)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(64, 16384 // tokens))), heads=heads, tokens=tokens, padded=rng.random() < 0.7)
    if kind == "layer_decode":
        return dict(kind=kind, batch=_log(rng, 1, 128), heads=rng.choice([8, 16]))
    if kind == "decode":
        return dict(kind=kind, batch=_log(rng, 1, 512), heads=rng.choice([8, 12, 16]))
    if kind == "cross":
        queries, keys = _log(rng, 16, 2048), _log(rng, 16, 2048)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(96, 16384 // max(queries, keys)))), heads=rng.choice([8, 16]), queries=queries, keys=keys)
    head_dim, proj_dim = rng.choice([(64, 64), (64, 64), (32, 32), (128, 128)])
    tokens = _log(rng, 16, 2048)
    return dict(kind=kind, batch=_log(rng, 1, max(1, min(64, 4096 // tokens))), heads=rng.choice([8, 16]), tokens=tokens, head_dim=head_dim,
                proj_dim=proj_dim, dtype=rng.choice(["float32", "float32", "float16"]))


# ------------------------------------------------------------------------------------------------ inputs
def _matrices(heads, head_dim, proj_dim, seed):
    np.random.seed(seed % (1 << 32))
    return torch.tensor(np.stack([orf(head_dim=head_dim, proj_dim=max(proj_dim, head_dim))[:proj_dim] for _ in range(heads)]),
                        dtype=torch.float32, device=DEV)


def _randn(gen, *shape, dtype=torch.float16):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=dtype)


def _features(x, w):
    """The feature map in plain tensor operations: inputs do not depend on the code that is timed."""
    x = x.float()
    u = torch.einsum("tbhd,hkd->tbhk", x / (torch.linalg.vector_norm(x, dim=-1, keepdim=True) + 1e-3), w)
    return (torch.cat([u.sin(), u.cos()], dim=-1) * SCALE).half()


def _padding(gen, batch, tokens):
    """[batch, tokens] with True at the padded positions, lengths uniform in [tokens / 2, tokens]."""
    lengths = torch.randint((tokens + 1) // 2, tokens + 1, (batch, 1), generator=gen, device=DEV)
    return torch.arange(tokens, device=DEV)[None, :] >= lengths


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind, B, H = case["kind"], case["batch"], case["heads"]
    if kind == "causal":
        T, d, D = case["tokens"], case["head_dim"], case["proj_dim"]
        w = _matrices(H, d, D, seed)
        q, k = (_features(_randn(gen, T, B, H, d), w).view(T, B * H, 2 * D).requires_grad_() for _ in range(2))
        v = _randn(gen, T, B * H, d).requires_grad_()
        return dict(kind=kind, leaves=[q, k, v], g=_randn(gen, T, B * H, d))
    if kind in ("layer_train", "layer_prefill", "layer_decode"):
        T, d = case.get("tokens", 1), 64
        torch.manual_seed(seed)
        layer = CausalAttention(embed_dim=H * d, num_heads=H, head_dim=d, proj_dim=64).to(DEV).half()
        state = dict(kind=kind, layer=layer, x=_randn(gen, T, B, H * d), w=_matrices(H, d, 64, seed).half())
        if kind == "layer_decode":
            k = _features(_randn(gen, 64, B, H, d), state["w"].float()).float()       # the state a prompt leaves
            v = _randn(gen, 64, B, H, d).float()
            state["saved"] = dict(prev_s=torch.einsum("tbhk,tbhd->bhkd", k, v).contiguous(), prev_z=k.sum(dim=0))
        else:
            state["pad"] = _padding(gen, B, T) if case["padded"] else None
        if kind == "layer_train":
            state["x"].requires_grad_()
            state["g"] = _randn(gen, T, B, H * d)
        return state
    if kind == "decode":
        d, D = 64, 64
        w = _matrices(H, d, D, seed)
        k = _features(_randn(gen, 16, B, H, d), w).float()
        v = _randn(gen, 16, B, H, d).float()
        return dict(kind=kind, q=_randn(gen, B, H, d), k=_randn(gen, B, H, d), v=_randn(gen, B, H, d), w=w,
                    s=torch.einsum("tbhk,tbhd->bhkd", k, v).contiguous(), z=k.sum(dim=0))
    if kind == "cross":
        Tq, Tk, d = case["queries"], case["keys"], 64
        leaves = [_randn(gen, Tq, B, H, d), _randn(gen, Tk, B, H, d), _randn(gen, Tk, B, H, d), _matrices(H, d, 64, seed)]
        return dict(kind=kind, leaves=[t.requires_grad_() for t in leaves], pad=_padding(gen, B, Tk), g=_randn(gen, Tq, B, H, d))
    T, d, D, dtype = case["tokens"], case["head_dim"], case["proj_dim"], getattr(torch, case["dtype"])
    leaves = [_randn(gen, T, B, H, d, dtype=dtype).requires_grad_(), _matrices(H, d, D, seed).requires_grad_()]
    return dict(kind=kind, leaves=leaves, g=_randn(gen, T, B, H, 2 * D, dtype=dtype))


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "layer_train":
        layer, x = state["layer"], state["x"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        y = layer(x, state["w"], key_padding_mask=state["pad"])
        y.backward(state["g"])
        return [y, x.grad] + [p.grad for p in layer.parameters()]
    if kind == "layer_prefill":
        with torch.no_grad():
            return state["layer"](state["x"], state["w"], key_padding_mask=state["pad"])
    if kind == "layer_decode":
        with torch.no_grad():
            y = state["layer"](state["x"], state["w"], saved_state=state["saved"])
        return [y, state["saved"]["prev_s"], state["saved"]["prev_z"]]
    if kind == "decode":
        y = ops.decode_step_fused(state["q"], state["k"], state["v"], state["w"], SCALE, state["s"], state["z"])
        return [y, state["s"], state["z"]]
    leaves = state["leaves"]
    for t in leaves:
        t.grad = None
    if kind == "causal":
        y = RFA.apply(*leaves)
    elif kind == "cross":
        q, k, v, w = leaves
        s, z = cross_rfa_state(random_project(x=k, random_matrices=w), v, state["pad"])
        y = cross_rfa_query(random_project(x=q, random_matrices=w), s, z)
    else:
        y = random_project(x=leaves[0], random_matrices=leaves[1])
    y.backward(state["g"])
    return [y] + [t.grad for t in leaves]


# ------------------------------------------------------------------------------------------------ the least it takes
def work(case):
    """Bytes: each array of a forward and of a backward read or written once by each (a backward starts when the forward
    has returned and its inputs have left the chip).  Flops: the products of the recurrent form, which grow with T only."""
    kind, B, H = case["kind"], case["batch"], case["heads"]
    if kind == "causal":
        n, d, K = B * H * case["tokens"], case["head_dim"], 2 * case["proj_dim"]
        return dict(bytes=n * 2 * ((2 * K + 2 * d) + (4 * K + 3 * d)), flops=n * 14 * K * d)
    if kind == "features":
        n, d, D = B * H * case["tokens"], case["head_dim"], case["proj_dim"]
        return dict(bytes=n * (3 * d + 4 * D) * (4 if case["dtype"] == "float32" else 2), flops=n * 8 * d * D)
    d, K = 64, 128
    if kind == "decode":
        return dict(bytes=B * H * (2 * 4 * (K * d + K) + 4 * 2 * d) + H * 4 * d * d, flops=B * H * (4 * K * d + 4 * d * d))
    if kind == "cross":
        nq, nk = B * H * case["queries"], B * H * case["keys"]
        return dict(bytes=2 * d * (nq * 5 + nk * 6) + H * 12 * d * d, flops=(nq * 6 + nk * 6) * K * d + (nq + nk) * 8 * d * d)
    E, n = H * d, B * case.get("tokens", 1)
    weights = 4 * E * (E + 1)
    if kind == "layer_decode":
        return dict(bytes=2 * weights + B * H * 2 * 4 * (K * d + K) + 4 * n * E, flops=n * (8 * E * E + H * (4 * K * d + 4 * d * d)))
    if kind == "layer_prefill":
        return dict(bytes=2 * weights + 4 * n * E, flops=n * (8 * E * E + H * (4 * K * d + 4 * d * d)))
    return dict(bytes=2 * 3 * weights + 2 * 5 * n * E, flops=n * (24 * E * E + H * (14 * K * d + 16 * d * d)))


def tolerance(case):
    """About four times what the path differs from itself computed in fp64 from the same inputs (largest over its outputs;
    "max" grows with the length of a sequence, and is what the longest ones show)."""
    kind, built = case["kind"], (case.get("head_dim", 64), case.get("proj_dim", 64)) == (64, 64)
    if kind == "features" and case["dtype"] == "float32":
        return dict(rel=1.2e-6, max=1.4e-5)                # fp32 throughout: 3.0e-7, 3.3e-6
    if kind == "features":
        return dict(rel=1.7e-3, max=1e-2) if built else dict(rel=9e-4, max=2e-3)      # 4.1e-4, 2.3e-3; 2.1e-4, 4.9e-4
    if kind == "causal":
        return dict(rel=1.9e-3, max=0.1) if built else dict(rel=9e-4, max=2e-3)       # 4.7e-4, 2.4e-2; 2.1e-4, 4.9e-4
    if kind in ("decode", "layer_decode"):
        return dict(rel=1.2e-3, max=4e-3)                  # 3.0e-4, 9.3e-4
    return dict(rel=3.4e-3, max=0.03)                      # layers and cross attention: 8.5e-4, 7.7e-3
