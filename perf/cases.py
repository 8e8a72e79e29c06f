"""Performance cases of the framework: the work its users have it do, through the public modules.

A case is one call of a module (or of a short stack of modules, as a model holds them) on tensors that are on the GPU.
The kinds and what they stand for:

- ``trunk``        the Pairformer trunk, eager: one prediction per length, so shapes change from call to call
- ``graphed``      the same trunk behind ``trunk.graphed``: a server that sees one shape again and again
- ``triangle``     the four triangle operations on their own, as a model with its own block structure calls them
- ``pairmixer``    the PairMixer trunk (triangle multiplications and transition)
- ``opm``          the outer product mean of an alignment
- ``embedder``     the whole sequence embedder: pair initialisation, one recycle, an MSA block, PairMixer blocks
- ``diffusion``    token blocks of one denoising step: several samples share one static pair tensor
- ``atoms``        atom-window blocks of one denoising step
- ``conditioning`` the pairwise conditioning of the diffusion module, once per system
- ``accurate``     a PairMixer block in the fp32-accurate mode

Trunks have 4 blocks where a model has 48: the blocks are alike, so the time of a pass is proportional to their number.
Weights are random with the scale of the modules' own initialisation, and LayerNorm and bias vectors are moved off
their initial constants as training moves them.  Inputs are N(0, 1) except masks (the last 7 % of the tokens padded),
one-hot MSA rows and their flags.
"""
from __future__ import annotations

import math

import torch

import bioemu2_b200 as b

DEV = "cuda"
C_S, C_Z, C_MSA = 384, 128, 64          # single, pair and MSA widths of the trunk
C_TOK, C_ATOM, C_ATOM_PAIR = 768, 128, 16  # token and atom widths of the diffusion module
S_INPUT = 456                            # input embedding of the sequence embedder
W_Q, W_K = 32, 128                       # atom attention window: queries, keys


def listed():
    return [
        # a short peptide: every kernel is tiny, launches and host work are what the call costs
        {"name": "trunk_n64", "kind": "trunk", "n": 64, "blocks": 4, "dtype": "float32"},
        # an ordinary protein whose length is a multiple of nothing
        {"name": "trunk_n203", "kind": "trunk", "n": 203, "blocks": 4, "dtype": "float32"},
        # the benchmark's trunk size
        {"name": "trunk_n512", "kind": "trunk", "n": 512, "blocks": 4, "dtype": "float32"},
        # a service with one padded length, captured once
        {"name": "graphed_n128", "kind": "graphed", "n": 128, "blocks": 4, "dtype": "float32"},
        # the large-system pair operations, on a bf16 pair tensor
        {"name": "triangle_n1536_bf16", "kind": "triangle", "n": 1536, "dtype": "bfloat16"},
        {"name": "pairmixer_n384", "kind": "pairmixer", "n": 384, "batch": 1, "blocks": 4, "dtype": "float32"},
        # the deep alignment of the benchmark
        {"name": "opm_s1024_n384_bf16", "kind": "opm", "n": 384, "s": 1024, "dtype": "bfloat16"},
        {"name": "embedder_n256_s128", "kind": "embedder", "n": 256, "s": 128},
        {"name": "diffusion_n256_m8", "kind": "diffusion", "n": 256, "m": 8},
        {"name": "atoms_4096_m8", "kind": "atoms", "n": 4096, "m": 8},
        {"name": "conditioning_n384", "kind": "conditioning", "n": 384},
        {"name": "accurate_n200", "kind": "accurate", "n": 200},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["trunk", "trunk", "graphed", "triangle", "pairmixer", "opm", "embedder", "diffusion", "atoms",
                       "conditioning", "accurate"])
    if kind in ("trunk", "graphed"):
        # bf16 pair and single tensors are what a caller that keeps its activations in bf16 passes
        return {"kind": kind, "n": _log_int(rng, 24, 512 if kind == "trunk" else 320), "blocks": 4,
                "dtype": rng.choice(["float32", "float32", "bfloat16"])}
    if kind == "triangle":
        return {"kind": kind, "n": _log_int(rng, 64, 1536), "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "pairmixer":
        batch = rng.choice([1, 1, 2])
        return {"kind": kind, "n": _log_int(rng, 48, 720 // batch), "batch": batch, "blocks": 4,
                "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "opm":
        return {"kind": kind, "n": _log_int(rng, 40, 400), "s": _log_int(rng, 16, 1024),
                "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "embedder":
        return {"kind": kind, "n": _log_int(rng, 48, 320), "s": _log_int(rng, 8, 256)}
    if kind == "diffusion":
        return {"kind": kind, "n": _log_int(rng, 32, 448), "m": rng.randint(1, 8)}
    if kind == "atoms":
        return {"kind": kind, "n": W_Q * _log_int(rng, 8, 192), "m": rng.randint(1, 8)}
    if kind == "conditioning":
        return {"kind": kind, "n": _log_int(rng, 48, 512)}
    return {"kind": kind, "n": _log_int(rng, 32, 256)}


# ------------------------------------------------------------------------------------------------ inputs and modules
def _weights(module, gen):
    """Seeded weights for a module built on the GPU: matrices as ``nn.Linear`` initialises them, vectors a little off
    the constants they start from (LayerNorm weights and the gate bias of triangle attention 1, other biases 0)."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.ndim >= 2:
                bound = 1.0 / math.sqrt(p.shape[1])
                p.uniform_(-bound, bound, generator=gen)
            else:
                start = 1.0 if name.endswith(("weight", "linear_g.bias")) else 0.0
                p.copy_(start + 0.05 * torch.randn(p.shape, device=p.device, generator=gen))
    return module.eval()


def _build(gen, make):
    with torch.device(DEV):
        module = make()
    return _weights(module, gen)


def _token_mask(batch, n):
    mask = torch.ones(batch, n, dtype=torch.bool, device=DEV)
    mask[:, n - max(1, round(n * 37 / 512)):] = False
    return mask


def _msa_features(gen, s, n):
    tok = _token_mask(1, n)
    rows = torch.randint(0, 33, (1, s, n), device=DEV, generator=gen)

    def u():
        return torch.rand(1, s, n, device=DEV, generator=gen)

    return {
        "msa": torch.nn.functional.one_hot(rows, 33).float(),
        "msa_mask": tok[:, None, :] & (u() > 0.1),
        "has_deletion": (u() < 0.2).float(),
        "deletion_value": u(),
        "msa_paired": (u() < 0.5).float(),
        "token_pad_mask": tok,
    }


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind, n = case["kind"], case["n"]
    dtype = getattr(torch, case.get("dtype", "float32"))

    def randn(*shape, dt=dtype):
        return torch.randn(*shape, device=DEV, generator=gen).to(dt)

    st = {"kind": kind}
    if kind in ("trunk", "graphed"):
        trunk = _build(gen, lambda: b.PairformerModule(C_S, C_Z, case["blocks"]))
        st.update(s=randn(1, n, C_S), z=randn(1, n, n, C_Z), mask=_token_mask(1, n))
        st["call"] = trunk if kind == "trunk" else trunk.graphed(st["s"], st["z"], st["mask"])
    elif kind == "triangle":
        st["ops"] = [_build(gen, make) for make in (b.TriangleMultiplicationOutgoing, b.TriangleMultiplicationIncoming,
                                                    b.TriangleAttentionStartingNode, b.TriangleAttentionEndingNode)]
        tok = _token_mask(1, n)
        st.update(z=randn(1, n, n, C_Z), mask=tok[:, :, None] & tok[:, None, :])
    elif kind == "pairmixer":
        st["call"] = _build(gen, lambda: b.PairMixerModule(C_S, C_Z, case["blocks"]))
        tok = _token_mask(case["batch"], n)
        st.update(s=randn(case["batch"], n, C_S), z=randn(case["batch"], n, n, C_Z), mask=tok[:, :, None] & tok[:, None, :])
    elif kind == "opm":
        st["call"] = _build(gen, lambda: b.OuterProductMean(C_MSA, 32, C_Z))
        rows = torch.rand(1, case["s"], 1, device=DEV, generator=gen) > 0.1
        st.update(m=randn(1, case["s"], n, C_MSA), mask=rows.expand(1, case["s"], n).contiguous())
    elif kind == "embedder":
        st["call"] = _build(gen, lambda: b.PairMixerSequenceEmbedder(C_S, C_Z, S_INPUT, msa_s=C_MSA, msa_blocks=1, num_blocks=2))
        st.update(s=randn(1, n, S_INPUT), feats=dict(_msa_features(gen, case["s"], n), pair_init_terms=randn(1, n, n, C_Z)))
    elif kind == "diffusion":
        st["layers"] = [_build(gen, lambda: b.ConditionedTransformerLayer(
            dim=C_TOK, dim_pairwise=C_Z, dim_cond=C_TOK, heads=16, transition_hidden=4 * C_TOK,
            lns_scale=1.0 / math.sqrt(i + 1))) for i in range(4)]
        st.update(x=randn(case["m"], n, C_TOK), c=randn(case["m"], n, C_TOK), z=randn(1, n, n, C_Z), mask=_token_mask(1, n),
                  m=case["m"])
        # the pair tensor is the same in every denoising step: its biases are projected once
        st["cache"] = b.PairBiasCache([layer.attention.pair_bias_attn for layer in st["layers"]])
        st["cache"].prepare(st["z"])
    elif kind == "atoms":
        st["layers"] = [_build(gen, lambda: b.ConditionedTransformerLayer(
            dim=C_ATOM, dim_pairwise=C_ATOM_PAIR, dim_cond=C_ATOM, heads=4, transition_hidden=2 * C_ATOM,
            is_sliding_window=True, window_queries=W_Q, window_keys=W_K)) for _ in range(3)]
        st.update(x=randn(case["m"], n, C_ATOM), c=randn(case["m"], n, C_ATOM), z=randn(1, n // W_Q, W_Q, W_K, C_ATOM_PAIR),
                  mask=_token_mask(1, n), m=case["m"])
    elif kind == "conditioning":
        st["call"] = _build(gen, lambda: b.PairwiseConditioning(C_Z, C_Z))
        st.update(z=randn(1, n, n, C_Z), rel=randn(1, n, n, C_Z))
    else:
        st["call"] = _build(gen, lambda: b.PairMixerLayer(C_S, C_Z))
        tok = _token_mask(1, n)
        st.update(s=randn(1, n, C_S), z=randn(1, n, n, C_Z), mask=tok[:, :, None] & tok[:, None, :])
    return st


@torch.no_grad()
def run(st):
    kind = st["kind"]
    if kind in ("trunk", "pairmixer"):
        return st["call"](st["s"], st["z"], st["mask"])
    if kind == "graphed":
        return st["call"](st["s"], st["z"], st["mask"])
    if kind == "triangle":
        return [op(st["z"], st["mask"]) for op in st["ops"]]
    if kind == "opm":
        return st["call"](st["m"], st["mask"])
    if kind == "embedder":
        return st["call"](st["s"], st["feats"], num_steps_recycle=1)
    if kind in ("diffusion", "atoms"):
        x = st["x"]
        for layer in st["layers"]:
            x = layer(x, st["z"], st["c"], st["mask"], st["m"])
        return x
    if kind == "conditioning":
        return st["call"](st["z"], st["rel"])
    with b.precision.matmul_precision("ieee"):
        return st["call"](st["s"], st["z"], st["mask"])


# ------------------------------------------------------------------------------------------------ what a pass costs
def _trimul(n):  # projections 128 -> 512, contraction, projections 2 x (128 -> 128)
    return 256 * n ** 3 + 196608 * n * n


def _triatt(n):  # q | k | v | g, 4-head bias, scores and weighted sum, output projection
    return 512 * n ** 3 + 164864 * n * n


def _linear(rows, *widths):
    return sum(2 * rows * i * o for i, o in widths)


def _opm(s, n):
    return 2 * s * n * n * 1024 + _linear(n * n, (1024, 128)) + _linear(s * n, (64, 64))


def work(case):
    """Each input and weight (as bf16) read once, each output written once; multiply and add count as two."""
    kind, n = case["kind"], case["n"]
    e = 2 if case.get("dtype") == "bfloat16" else 4
    pair, p = n * n * C_Z, n * n
    transition = _linear(p, (128, 512), (128, 512), (512, 128))
    if kind in ("trunk", "graphed"):
        block = 2 * _trimul(n) + 2 * _triatt(n) + transition + _linear(p, (128, 16)) + 4 * p * C_S
        block += _linear(n, *[(C_S, C_S)] * 5, *[(C_S, 4 * C_S)] * 3)
        return {"bytes": 2 * e * (pair + n * C_S) + n + 2 * case["blocks"] * 3.1e6, "flops": case["blocks"] * block}
    if kind == "triangle":
        return {"bytes": 5 * e * pair + p, "flops": 2 * _trimul(n) + 2 * _triatt(n)}
    if kind == "pairmixer":
        return {"bytes": case["batch"] * (2 * e * pair + p) + 2 * case["blocks"] * 3.9e5,
                "flops": case["batch"] * case["blocks"] * (2 * _trimul(n) + transition)}
    if kind == "opm":
        return {"bytes": e * (case["s"] * n * C_MSA + pair) + case["s"] * n, "flops": _opm(case["s"], n)}
    if kind == "embedder":
        s = case["s"]
        mixer = 2 * _trimul(n) + transition
        msa = _linear(s * n, (64, 256), (64, 256), (64, 256), (256, 64), (256, 64), (256, 64), (40, 64), (64, 256))
        msa += 2 * s * p * 256 + _linear(p, (128, 8)) + _opm(s, n) + mixer
        recycle = _linear(p, (128, 128)) + _linear(n, (C_S, C_S))
        return {"bytes": 2 * 4 * pair + 4 * s * n * (33 + 3) + s * n + 4 * n * (S_INPUT + C_S),
                "flops": 2 * (recycle + msa + 2 * mixer)}
    if kind == "diffusion":
        rows, d = case["m"] * n, C_TOK
        layer = _linear(rows, (d, 6 * d), *[(d, d)] * 5, *[(d, 4 * d)] * 3) + 4 * case["m"] * p * d
        return {"bytes": 3 * 4 * rows * d + 4 * (2 * p * 16 + 2 * 23 * d * d), "flops": 4 * layer}
    if kind == "atoms":
        rows, d = case["m"] * n, C_ATOM
        layer = _linear(rows, (d, 6 * d), *[(d, d)] * 5, *[(d, 2 * d)] * 3) + 4 * rows * W_K * d
        layer += _linear(n * W_K, (C_ATOM_PAIR, 4))
        return {"bytes": 3 * 4 * rows * d + 4 * n * W_K * C_ATOM_PAIR, "flops": 3 * layer}
    if kind == "conditioning":
        return {"bytes": 3 * 4 * pair, "flops": _linear(p, (256, 128), *[(128, 256)] * 6)}
    return {"bytes": 2 * 4 * pair + p, "flops": 2 * _trimul(n) + transition}


def tolerance(case):
    if case["kind"] == "accurate":
        return {"rel": 5e-5}  # products of split fp32 operands, about 2^-16 each
    return {"rel": 1e-2}      # bf16 operands, fp32 accumulation
