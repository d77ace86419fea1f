"""The calls that a structure-prediction program makes to this framework, at the sizes it makes them, for timing.

A prediction runs, in order: the trunk (pair blocks on the N x N pair tensor, 48 of them per recycling), the sampler (one
network evaluation per diffusion step, 100 to 200 steps, one to five samples) and the confidence head (once per sample).
Complexes have from a few dozen tokens (a peptide, a single domain) to about two thousand; token counts are whatever the
sequence gives, so most are odd.  Everything is inference; the trunk and the confidence head run in bfloat16, the network of
the sampler in bfloat16 under autocast or, as the models were trained, in float32.

Inputs and weights are drawn on the GPU from the seed: activations ~ N(0, 1), matrices ~ N(0, 1 / fan_in), LayerNorm scales
around one, and a tail of padding tokens and atoms as batching leaves it.
"""
from __future__ import annotations

import math
import types

import torch

from kfold_b200 import confidence, modules, sampler

DEVICE = "cuda"
C_S = 384           # single / conditioning channels
C_ATOM, C_ATOMPAIR = 128, 16
SINGLE_HEADS, TRI_HEADS = 16, 4
CONF_BLOCKS = 4
# token transformer of the diffusion network: width -> blocks (16 heads each; head dim 48 and 64)
TOKEN_BLOCKS = {768: 24, 1024: 16}


def listed():
    return [
        # One Pairformer block (c_z = 128, c_s = 384), the unit of the trunk; a peptide: the call is all latency and launches.
        {"name": "block-64", "kind": "block", "tokens": 64, "pad": 0.0, "dtype": "bf16"},
        # A small protein: an odd token count, as nearly every sequence has.
        {"name": "block-251", "kind": "block", "tokens": 251, "pad": 0.05, "dtype": "bf16"},
        # The common complex, and the size that the benchmark reports.
        {"name": "block-768", "kind": "block", "tokens": 768, "pad": 0.1, "dtype": "bf16"},
        # The largest complexes: N^3 work and gigabyte-sized pair tensors.
        {"name": "block-2048", "kind": "block", "tokens": 2048, "pad": 0.05, "dtype": "bf16"},
        # The same block in float32: users who check or fine-compare structures run without autocast.
        {"name": "block-160-f32", "kind": "block", "tokens": 160, "pad": 0.0, "dtype": "f32"},
        # K-Fold's own trunk block (c_z = 256: two triangle multiplications and a transition), odd and common sizes.
        {"name": "tri-333", "kind": "tri", "tokens": 333, "pad": 0.0, "dtype": "bf16"},
        {"name": "tri-768", "kind": "tri", "tokens": 768, "pad": 0.1, "dtype": "bf16"},
        # One evaluation of the diffusion network, called eagerly: a single small structure (latency, about 240 launches) ...
        {"name": "step-96x1", "kind": "step", "tokens": 96, "atoms": 736, "samples": 1, "width": 768, "pad": 0.0, "dtype": "bf16"},
        # ... the common complex with five samples ...
        {"name": "step-768x5", "kind": "step", "tokens": 768, "atoms": 6016, "samples": 5, "width": 768, "pad": 0.1, "dtype": "bf16"},
        # ... and float32 at the production width, the precision in which the reference samples.
        {"name": "step-301x1-f32", "kind": "step", "tokens": 301, "atoms": 2400, "samples": 1, "width": 1024, "pad": 0.02, "dtype": "f32"},
        # A whole sampler run with the default number of steps, the network replayed as a CUDA graph.
        {"name": "sample-384x5", "kind": "sample", "tokens": 384, "atoms": 3008, "samples": 5, "width": 768, "steps": 100, "pad": 0.05,
         "dtype": "bf16"},
        # The confidence head on one sample: four blocks at c_z = 256 and the float32 output heads over all pairs.
        {"name": "confidence-400", "kind": "confidence", "tokens": 400, "pad": 0.05, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "tri", "step", "step", "step", "sample", "confidence"])
    pad = round(rng.choice([0.0, rng.uniform(0.0, 0.15)]), 3)
    if kind == "block":
        f32 = rng.random() < 0.2
        return {"kind": kind, "tokens": _log_int(rng, 40, 256 if f32 else 1600), "pad": pad, "dtype": "f32" if f32 else "bf16"}
    if kind == "tri":
        return {"kind": kind, "tokens": _log_int(rng, 64, 1024), "pad": pad, "dtype": "bf16"}
    if kind == "confidence":
        return {"kind": kind, "tokens": _log_int(rng, 64, 500), "pad": pad, "dtype": "bf16"}
    f32 = kind == "step" and rng.random() < 0.3
    tokens = _log_int(rng, 48, 384 if f32 or kind == "sample" else 800)
    case = {"kind": kind, "tokens": tokens, "atoms": 32 * max(2, int(tokens * rng.uniform(6.0, 9.0)) // 32),
            "samples": rng.randint(1, 5), "width": rng.choice(sorted(TOKEN_BLOCKS)), "pad": pad, "dtype": "f32" if f32 else "bf16"}
    if kind == "sample":
        case["steps"] = rng.randint(20, 80)
    return case


# ------------------------------------------------------------------------------------------------ inputs and weights
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _normal(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype)


def _weights(module, gen):
    """Random weights of the architecture: matrices N(0, 1 / fan_in), LayerNorm scales and offsets spread around 1 and 0, the
    gates of the conditioned layers starting nearly closed, as they are trained."""
    module = module.to(DEVICE)
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() == 2:
                p.normal_(0.0, p.shape[1] ** -0.5, generator=gen)
            else:
                p.normal_(0.0, 0.1, generator=gen)
                if name.endswith("weight"):
                    p.add_(1.0)
                elif name.endswith("linear_ada_out.bias") or name.endswith("transition.linear_g.bias"):
                    p.sub_(2.0)
    return module


def _mask(n, pad):
    m = torch.ones(n, dtype=torch.bool, device=DEVICE)
    if int(pad * n):
        m[n - int(pad * n):] = False
    return m


def _pair_mask(m):
    return (m[:, None] & m[None, :]).unsqueeze(0).contiguous()


class _Normals:
    """The sampler's source of normals: a generator of its own, so that a seed gives one structure."""

    def __init__(self, seed):
        self.seed, self.gen = seed, torch.Generator(device=DEVICE)

    def restart(self):
        self.gen.manual_seed(self.seed)
        return self

    def randn(self, shape):
        return torch.randn(tuple(shape), generator=self.gen, device=DEVICE, dtype=torch.float32)


def _autocast(case):
    return torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["dtype"] == "bf16")


def _network(case, gen, coords):
    """The diffusion network with its weights, and what the program has computed once for the complex: atom features, window
    pair features, the token pair bias of all blocks, index and masks."""
    nt, na, width = case["tokens"], case["atoms"], case["width"]
    with torch.device(DEVICE):
        net = modules.DiffusionStack(channel_a=width, channel_s=C_S, channel_z=128, channel_atom=C_ATOM, channel_atompair=C_ATOMPAIR,
                                     channel_coords=coords, token_transformer_blocks=TOKEN_BLOCKS[width])
    net = _weights(net, gen)
    state = {"net": net, "q": _normal(gen, 1, na, C_ATOM), "c": _normal(gen, 1, na, C_ATOM),
             "p": _normal(gen, 1, na // 32, 32, 128, C_ATOMPAIR),
             "token_index": torch.randint(0, nt, (1, na), generator=gen, device=DEVICE).sort(-1).values,
             "atom_mask": _mask(na, case["pad"] / 4).unsqueeze(0), "token_mask": _mask(nt, case["pad"]).unsqueeze(0)}
    with torch.no_grad(), _autocast(case):
        state["pair_bias"] = net.get_pair_bias(_normal(gen, 1, nt, nt, 128, dtype=_dtype(case)))
    return state


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def prepare(case, seed):
    gen = _generator(seed)
    kind, n = case["kind"], case["tokens"]
    state = {"case": case}
    if kind in ("block", "tri"):
        with torch.device(DEVICE):
            mod = modules.PairformerBlock(128, C_S, TRI_HEADS, SINGLE_HEADS) if kind == "block" else modules.TriangularBlock(256)
        state["net"] = _weights(mod, gen)
        state["z"] = _normal(gen, 1, n, n, 128 if kind == "block" else 256, dtype=_dtype(case))
        m = _mask(n, case["pad"])
        state["pair_mask"] = _pair_mask(m)
        if kind == "block":
            state["s"], state["mask"] = _normal(gen, 1, n, C_S, dtype=_dtype(case)), m.unsqueeze(0)
    elif kind == "confidence":
        with torch.device(DEVICE):
            mod = confidence.ConfidenceHead(channel_s=C_S, channel_z=256, num_heads_attn=SINGLE_HEADS, num_blocks=CONF_BLOCKS)
        state["net"] = _weights(mod, gen)
        state["z"], state["s"] = _normal(gen, 1, n, n, 256, dtype=torch.bfloat16), _normal(gen, 1, n, C_S, dtype=torch.bfloat16)
        state["x"] = _normal(gen, 1, n, 3) * 15.0
        state["mask"] = _mask(n, case["pad"]).unsqueeze(0)
    elif kind == "step":
        state.update(_network(case, gen, 3))
        state["r"] = _normal(gen, 1, case["samples"], case["atoms"], 3) * 4.0
        state["s"] = _normal(gen, 1, case["samples"], n, C_S)
    else:
        pre = _network(case, gen, 6)
        state["sampler"] = sampler.KFoldECSI(sampler.KFoldECSI.Config(), pre["net"])
        state["precomputed"] = {k: pre[k] for k in ("q", "c", "p", "pair_bias")}
        atom = types.SimpleNamespace(pad_mask=pre["atom_mask"], token_index=pre["token_index"],
                                     prior_coords=_normal(gen, 1, case["atoms"], 1, 3) * 10.0)
        state["f_input"] = types.SimpleNamespace(atom=atom, token=types.SimpleNamespace(pad_mask=pre["token_mask"]))
        state["s_inputs"] = _normal(gen, 1, n, C_S)
        state["normals"] = _Normals(int(seed))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    with torch.no_grad():
        if kind == "block":
            return state["net"](state["z"], state["s"], state["pair_mask"], state["mask"])
        if kind == "tri":
            return state["net"](state["z"], state["pair_mask"])
        with _autocast(case):
            if kind == "confidence":
                return state["net"].forward_single(state["z"], state["s"], state["x"], state["mask"])
            if kind == "step":
                return state["net"].step(state["r"], state["q"], state["c"], state["p"], state["token_index"], state["atom_mask"],
                                         state["s"], state["pair_bias"], state["token_mask"])
            return state["sampler"].sample_structure(state["f_input"], state["s_inputs"], None, num_steps=case["steps"],
                                                     num_samples=case["samples"], precomputed=state["precomputed"],
                                                     rng=state["normals"].restart(), cuda_graph=True)["coordinates"]


# ------------------------------------------------------------------------------------------------ algorithmic work
def _tri_mul(n, c):      # flops, weights
    return 2.0 * n ** 3 * c + 2.0 * n * n * c * 6 * c, 6 * c * c


def _transition(rows, c, factor):
    return 2.0 * rows * c * 3 * factor * c, 3 * factor * c * c


def _single_attention(n, c):
    return 2.0 * n * c * 5 * c + 4.0 * n * n * c, 5 * c * c


def _pair_single(n, c_z, tri_att):
    """One block: (flops, weight elements) of the pair track and the single track."""
    parts = [_tri_mul(n, c_z), _tri_mul(n, c_z), _transition(n * n, c_z, 4), _single_attention(n, C_S), _transition(n, C_S, 4),
             (2.0 * n * n * c_z * SINGLE_HEADS, c_z * SINGLE_HEADS)]
    if tri_att:
        one = (2.0 * n * n * c_z * (5 * c_z + TRI_HEADS) + 4.0 * n ** 3 * c_z, 5 * c_z * c_z + TRI_HEADS * c_z)
        parts += [one, one]
    return sum(f for f, _ in parts), sum(w for _, w in parts)


def _step_work(case):
    """One evaluation of the diffusion network: (flops, weight elements, bytes of activations in and out, bytes of the pair
    bias and the window pair features, which every evaluation reads)."""
    nt, na, ns, c = case["tokens"], case["atoms"], case["samples"], case["width"]
    blocks, e = TOKEN_BLOCKS[c], 4 if case["dtype"] == "f32" else 2
    rows_t, rows_a, ca, windows = ns * nt, ns * na, C_ATOM, na // 32
    token = 2.0 * rows_t * (c * 5 * c + c * 6 * c) + 4.0 * ns * nt * nt * c + 2.0 * rows_t * C_S * 6 * c
    atom = 2.0 * rows_a * (ca * 5 * ca + ca * 6 * ca) + 4.0 * rows_a * 128 * ca + 2.0 * na * ca * 8 * ca + 2.0 * windows * 4096 * C_ATOMPAIR * 4
    flops = blocks * token + 6 * atom + 2.0 * 2 * rows_a * ca * c + 2.0 * rows_t * C_S * c
    weights = blocks * (11 * c * c + 6 * C_S * c) + 6 * (11 + 8) * ca * ca + 2 * ca * c + C_S * c
    bias = float(blocks) * 16 * nt * nt * e + 4.0 * windows * 4096 * C_ATOMPAIR
    acts = 4.0 * (rows_a * 6 + rows_t * C_S + 2 * na * ca)
    return flops, weights, acts, bias


def work(case):
    kind, n = case["kind"], case["tokens"]
    e = 4 if case["dtype"] == "f32" else 2
    if kind in ("block", "tri"):
        if kind == "block":
            flops, weights = _pair_single(n, 128, True)
            return {"bytes": 2.0 * e * (n * n * 128 + n * C_S) + n * n + e * weights, "flops": flops}
        parts = [_tri_mul(n, 256), _tri_mul(n, 256), _transition(n * n, 256, 4)]
        return {"bytes": 2.0 * e * n * n * 256 + n * n + e * sum(w for _, w in parts), "flops": sum(f for f, _ in parts)}
    if kind == "confidence":
        flops, weights = _pair_single(n, 256, False)
        flops = CONF_BLOCKS * flops + 2.0 * n * n * 256 * 128 + 2.0 * n * C_S * 1248
        return {"bytes": 2.0 * n * n * 256 + 4.0 * n * n * 128 + 2.0 * n * C_S + 4.0 * n * 1248 + 2.0 * CONF_BLOCKS * weights, "flops": flops}
    flops, weights, acts, bias = _step_work(case)
    if kind == "step":
        return {"bytes": acts + bias + e * weights, "flops": flops}
    # every step of the sampler also conditions the single representation on the noise level (two transitions)
    flops += 2.0 * n * C_S * C_S * 12
    return {"bytes": case["steps"] * (4.0 * 9 * case["samples"] * case["atoms"] + bias + e * weights), "flops": case["steps"] * flops}


def tolerance(case):
    # float32 computes with 24-bit operands and float32 sums through a few dozen layers; bfloat16 rounds every operand to 8 bits
    return {"rel": 2e-5} if case["dtype"] == "f32" else {"rel": 1e-2}
