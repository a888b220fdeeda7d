"""Work that a user of this framework has it do, as cases that can be timed and compared.

Six paths, each through the public entry point that an inference program calls:

  trunk        ``ops.pairformer_stack_``: Pairformer blocks over a pair and a single representation (one recycle runs 48 of
               them, the confidence head 4; the time is linear in the blocks, so a case runs a few)
  trimul       ``ops.triangle_multiplication_``: outgoing, then incoming edges (the stand-alone operator)
  diffusion    ``PackedDiffusionTransformer.forward``: the 24-block transformer of one denoising step (200 per sample)
  pair_logits  ``PackedDiffusionTransformer.pair_logits``: once per inference, before the denoising steps
  atoms        ``ops.cross_attention``: the core of the atom cross attention, windows of 32 queries x 128 keys
  grid_op      ``torch.ops._alpha_attention.grid_self_attn_forward``: the registered operator, argument by argument as the
               reference's wrapper passes it

Sizes and widths are those of the model this repository implements (pair 128, single 384, token 768, 16 heads).  The model
(weights) is made once per process, as a program loads its checkpoint once; inputs come from the seed.
"""
from __future__ import annotations

import functools
import math

import torch

import __graft_entry__ as _entry

_entry.load_package()
from distributed_xfold_b200 import diffusion, op_library, ops  # noqa: E402

DEV = "cuda"
BF16 = torch.bfloat16
C_PAIR, C_SINGLE, C_TOKEN, HEADS, DIFF_BLOCKS = 128, 384, 768, 16, 24
WINDOW_Q, WINDOW_K, ATOM_C, ATOM_HEADS, ATOM_D = 32, 128, 128, 4, 32


def listed():
    return [
        # a short peptide: nothing but launches and latency
        {"name": "trunk 37 x4", "path": "trunk", "tokens": 37, "blocks": 4, "mask": "none"},
        # a small protein, a token count that is a multiple of nothing, padded at its end
        {"name": "trunk 255 x4", "path": "trunk", "tokens": 255, "blocks": 4, "mask": "tail"},
        # an ordinary protein
        {"name": "trunk 600 x2", "path": "trunk", "tokens": 600, "blocks": 2, "mask": "tail"},
        # the benchmark's size and masks (10 % of the tokens padded at random)
        {"name": "trunk 1024 x2", "path": "trunk", "tokens": 1024, "blocks": 2, "mask": "random"},
        # a large complex, the token count of the end-to-end configuration
        {"name": "trunk 1536 x1", "path": "trunk", "tokens": 1536, "blocks": 1, "mask": "none"},
        # the operator on its own, at its own configuration
        {"name": "trimul 768", "path": "trimul", "tokens": 768, "mask": "none"},
        # a denoising step: a short peptide, five samples of an ordinary protein in one batch, the largest configuration
        {"name": "diffusion 77 x1", "path": "diffusion", "tokens": 77, "samples": 1, "mask": "none"},
        {"name": "diffusion 384 x5", "path": "diffusion", "tokens": 384, "samples": 5, "mask": "tail"},
        {"name": "diffusion 2048 x1", "path": "diffusion", "tokens": 2048, "samples": 1, "mask": "none"},
        # the step-invariant part of the diffusion transformer
        {"name": "pair_logits 1000", "path": "pair_logits", "tokens": 1000},
        # about eight atoms per token of a 1024-token complex
        {"name": "atoms 8200", "path": "atoms", "atoms": 8200},
        # the operator interface at an ordinary, ragged size
        {"name": "grid_op 300", "path": "grid_op", "tokens": 300, "mask": "tail"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # the trunk and the denoising steps are where an inference spends its time
    path = rng.choice(["trunk"] * 5 + ["diffusion"] * 3 + ["trimul", "pair_logits", "atoms", "grid_op"])
    mask = rng.choice(["none", "tail", "random"])
    if path == "trunk":
        n = _log(rng, 32, 1536)
        return {"path": path, "tokens": n, "blocks": 4 if n <= 300 else 2 if n <= 1024 else 1, "mask": mask}
    if path == "diffusion":
        n = _log(rng, 40, 2048)
        return {"path": path, "tokens": n, "samples": rng.choice([1, 5]) if n <= 400 else 1, "mask": mask}
    if path == "trimul":
        return {"path": path, "tokens": _log(rng, 48, 1280), "mask": mask}
    if path == "pair_logits":
        return {"path": path, "tokens": _log(rng, 40, 1536)}
    if path == "atoms":
        return {"path": path, "atoms": _log(rng, 200, 16384)}
    return {"path": path, "tokens": _log(rng, 40, 640), "mask": mask}


# ---------------------------------------------------------------------------------------------------------------
# the model: Linear weights ~ N(0, 1 / fan_in), LayerNorm scales about 1 and offsets about 0, as in a trained network
# ---------------------------------------------------------------------------------------------------------------
class _Maker:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device=DEV)

    def lin(self, state, name, n_out, n_in, bias=False):
        state[name + ".weight"] = self.randn(n_out, n_in) * n_in ** -0.5
        if bias:
            state[name + ".bias"] = self.randn(n_out) * 0.1

    def norm(self, state, name, c, bias=True):
        state[name + ".weight"] = 1.0 + 0.1 * self.randn(c)
        if bias:
            state[name + ".bias"] = 0.1 * self.randn(c)

    def trimul(self, state, p):
        c = C_PAIR
        self.norm(state, p + "left_norm_input", c)
        self.lin(state, p + "projection", 2 * c, c)
        self.lin(state, p + "gate", 2 * c, c)
        self.norm(state, p + "center_norm", c)
        self.lin(state, p + "output_projection", c, c)
        self.lin(state, p + "gating_linear", c, c)

    def grid(self, state, p):
        c = C_PAIR
        self.norm(state, p + "act_norm", c)
        self.lin(state, p + "pair_bias_projection", 4, c)
        for n in ("q_projection", "k_projection", "v_projection", "gating_query", "output_projection"):
            self.lin(state, p + n, c, c)

    def transition(self, state, p, c, factor=4):
        self.norm(state, p + "input_layer_norm", c)
        self.lin(state, p + "transition1", 2 * factor * c, c)
        self.lin(state, p + "transition2", c, factor * c)

    def adaln(self, state, p, c, c_cond):
        self.norm(state, p + "single_cond_layer_norm", c_cond, bias=False)
        self.lin(state, p + "single_cond_scale", c, c_cond, bias=True)
        self.lin(state, p + "single_cond_bias", c, c_cond)

    def adaln_zero(self, state, p, c_in, c, c_cond):
        self.lin(state, p + "transition2", c, c_in)
        if c_cond:
            self.lin(state, p + "adaptive_zero_cond", c, c_cond, bias=True)

    def attention(self, state, p, c, c_cond):
        if c_cond:
            self.adaln(state, p + "adaptive_layernorm.", c, c_cond)
        else:
            self.norm(state, p + "adaptive_layernorm.layer_norm", c)
        self.lin(state, p + "q_projection", c, c, bias=True)
        for n in ("k_projection", "v_projection", "gating_query"):
            self.lin(state, p + n, c, c)
        self.adaln_zero(state, p + "adaptive_zero_init.", c, c, c_cond)

    def block(self, p):
        s = {}
        self.trimul(s, p + "triangle_multiplication_outgoing.")
        self.trimul(s, p + "triangle_multiplication_incoming.")
        self.grid(s, p + "pair_attention1.")
        self.grid(s, p + "pair_attention2.")
        self.transition(s, p + "pair_transition.", C_PAIR)
        self.norm(s, p + "single_pair_logits_norm", C_PAIR)
        self.lin(s, p + "single_pair_logits_projection", HEADS, C_PAIR)
        self.attention(s, p + "single_attention_.", C_SINGLE, 0)
        self.transition(s, p + "single_transition.", C_SINGLE)
        return s


@functools.lru_cache(maxsize=None)
def _trunk(blocks):
    m = _Maker(2)
    return ops.PackedPairformerStack(ops.PackedPairformerBlock(m.block(""), "", DEV) for _ in range(blocks))


@functools.lru_cache(maxsize=None)
def _trimul():
    m, s = _Maker(1), {}
    m.trimul(s, "out.")
    m.trimul(s, "in.")
    return ops.PackedTriMul(s, "out.", DEV), ops.PackedTriMul(s, "in.", DEV)


@functools.lru_cache(maxsize=None)
def _diffusion():
    m, s = _Maker(7), {}
    m.norm(s, "pair_input_layer_norm", C_PAIR)
    for i in range(DIFF_BLOCKS // 4):
        m.lin(s, f"pair_logits_projection.{i}", 4 * HEADS, C_PAIR)
    for i in range(DIFF_BLOCKS):
        m.attention(s, f"self_attention.{i}.", C_TOKEN, C_SINGLE)
        p = f"transition_block.{i}."
        m.adaln(s, p + "adaptive_layernorm.", C_TOKEN, C_SINGLE)
        m.lin(s, p + "transition1", 4 * C_TOKEN, C_TOKEN)
        m.adaln_zero(s, p + "adaptive_zero_init.", 2 * C_TOKEN, C_TOKEN, C_SINGLE)
    return diffusion.PackedDiffusionTransformer(s, "", DEV, HEADS, DIFF_BLOCKS, 4)


def _heads(m, c_in, heads, d):
    return (m.randn(c_in, heads, d) * c_in ** -0.5).to(BF16)


@functools.lru_cache(maxsize=None)
def _atoms():
    m = _Maker(9)
    qw, kw, vw, gw = (_heads(m, ATOM_C, ATOM_HEADS, ATOM_D) for _ in range(4))
    return ops.PackedCrossAttention(qw, 0.1 * m.randn(1, ATOM_HEADS, ATOM_D), kw, vw, gw, DEV)


@functools.lru_cache(maxsize=None)
def _grid():
    op_library.register()
    m = _Maker(11)
    w = {n: _heads(m, C_PAIR, 4, 32) for n in ("query_w", "key_w", "value_w", "gating_w")}
    w["output_w"] = (m.randn(4, 32, C_PAIR) * C_PAIR ** -0.5).to(BF16)
    return w


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _token_mask(case, n, g):
    m = torch.ones(n, device=DEV)
    if case["mask"] == "tail":      # tokens up to a bucket's size
        m[n - max(1, n // 12):] = 0
    elif case["mask"] == "random":
        m = (torch.rand(n, generator=g, device=DEV) >= 0.1).float()
        m[0] = 1
    return m


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)

    def randn(*shape, dtype=BF16):
        return torch.randn(*shape, generator=g, device=DEV, dtype=dtype)

    path = case["path"]
    st = {"path": path}
    if path in ("trunk", "trimul"):
        n = case["tokens"]
        st["z0"] = randn(n, n, C_PAIR)
        st["z"] = torch.empty_like(st["z0"])
        st["seq_mask"] = _token_mask(case, n, g)
        st["pair_mask"] = st["seq_mask"][:, None] * st["seq_mask"][None, :]
        if path == "trimul":
            st["w"] = _trimul()
        else:
            st["w"] = _trunk(case["blocks"])
            st["s0"] = randn(n, C_SINGLE)
            st["s"] = torch.empty_like(st["s0"])
    elif path in ("diffusion", "pair_logits"):
        n = case["tokens"]
        st["w"] = _diffusion()
        pair = randn(n, n, C_PAIR)
        if path == "pair_logits":
            st["pair"] = pair
        else:
            st["logits"] = st["w"].pair_logits(pair)
            st["mask"] = _token_mask(case, n, g)
            st["cond"] = randn(n, C_SINGLE)
            shape = (n, C_TOKEN) if case["samples"] == 1 else (case["samples"], n, C_TOKEN)
            st["act0"] = randn(*shape)
            st["act"] = torch.empty_like(st["act0"])
    elif path == "atoms":
        b = (case["atoms"] + WINDOW_Q - 1) // WINDOW_Q
        st["w"] = _atoms()
        st["q"] = randn(b, WINDOW_Q, ATOM_C)
        st["m"] = randn(b, WINDOW_K, ATOM_C)
        # pair term plus the key mask of each window (atoms beyond the chain's ends)
        keep = torch.rand(b, 1, 1, WINDOW_K, generator=g, device=DEV) >= 0.1
        st["bias"] = randn(b, ATOM_HEADS, WINDOW_Q, WINDOW_K, dtype=torch.float32) + 1e9 * (keep.float() - 1.0)
    else:
        n = case["tokens"]
        st["w"] = _grid()
        st["x"] = randn(n, n, C_PAIR)
        m = _token_mask(case, n, g)
        st["bias"] = (1e9 * (m[:, None] * m[None, :] - 1.0))[:, None, None, :].contiguous()
        st["nb"] = randn(4, n, n, dtype=torch.float32)
    return st


def run(st):
    path = st["path"]
    if path == "trunk":     # a recycle starts from new embeddings, in the buffers that the program keeps
        st["z"].copy_(st["z0"])
        st["s"].copy_(st["s0"])
        return ops.pairformer_stack_(st["z"], st["s"], st["pair_mask"], st["seq_mask"], st["w"])
    if path == "trimul":
        st["z"].copy_(st["z0"])
        ops.triangle_multiplication_(st["z"], st["pair_mask"], st["w"][0], True)
        return ops.triangle_multiplication_(st["z"], st["pair_mask"], st["w"][1], False)
    if path == "diffusion":  # a denoising step starts from the noisy positions' new token activations
        st["act"].copy_(st["act0"])
        return st["w"].forward(st["act"], st["mask"], st["cond"], st["logits"])
    if path == "pair_logits":
        return st["w"].pair_logits(st["pair"])
    if path == "atoms":
        return ops.cross_attention(st["q"], st["m"], st["bias"], st["w"])
    w = st["w"]
    return torch.ops._alpha_attention.grid_self_attn_forward(st["x"], st["bias"], st["nb"], w["query_w"], w["key_w"],
                                                             w["value_w"], w["gating_w"], w["output_w"], 32, 32)


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two right answers may be apart
# ---------------------------------------------------------------------------------------------------------------
def _trimul_flops(n):
    return 2.0 * n ** 3 * C_PAIR + 12.0 * n * n * C_PAIR * C_PAIR


def work(case):
    path, c = case["path"], C_PAIR
    if path in ("trunk", "trimul"):
        n = case["tokens"]
        io = 2.0 * n * n * c * 2 + n * n * 4
        if path == "trimul":
            return {"bytes": io + 2 * 6 * c * c * 2, "flops": 2 * _trimul_flops(n)}
        cs = C_SINGLE
        att = 10.0 * n * n * c * c + 4.0 * n ** 3 * c + 2.0 * n * n * c * 4
        single = 10.0 * n * cs * cs + 4.0 * n * n * cs + 24.0 * n * cs * cs + 2.0 * n * n * c * HEADS
        per_block = 2 * _trimul_flops(n) + 2 * att + 24.0 * n * n * c * c + single
        weights = (2 * 6 + 2 * 5 + 12) * c * c * 2 + 17 * cs * cs * 2
        return {"bytes": io + 4.0 * n * cs + case["blocks"] * weights, "flops": case["blocks"] * per_block}
    if path == "diffusion":
        n, s, ct, cc = case["tokens"], case["samples"], C_TOKEN, C_SINGLE
        per_block = s * (10.0 * n * ct * ct + 4.0 * n * n * ct + 12.0 * n * ct * ct) + 12.0 * n * cc * ct
        weights = (5 + 6) * ct * ct * 2 + 6 * cc * ct * 2
        logits = HEADS * n * n * 2
        return {"bytes": DIFF_BLOCKS * (weights + logits) + 2.0 * s * n * ct * 2 + n * cc * 2, "flops": DIFF_BLOCKS * per_block}
    if path == "pair_logits":
        n, h = case["tokens"], DIFF_BLOCKS * HEADS
        return {"bytes": n * n * c * 2.0 + h * n * ((n + 7) // 8 * 8) * 2.0 + h * c * 4, "flops": 2.0 * n * n * c * h}
    if path == "atoms":
        b, hd = (case["atoms"] + WINDOW_Q - 1) // WINDOW_Q, ATOM_HEADS * ATOM_D
        proj = 2.0 * b * (WINDOW_Q + WINDOW_K) * ATOM_C * 2 * hd
        io = b * ((WINDOW_Q + WINDOW_K) * ATOM_C * 2.0 + ATOM_HEADS * WINDOW_Q * WINDOW_K * 4.0 + WINDOW_Q * hd * 2.0)
        return {"bytes": io + 4 * ATOM_C * hd * 2, "flops": proj + 4.0 * b * WINDOW_Q * WINDOW_K * hd}
    n = case["tokens"]
    return {"bytes": 2.0 * n * n * c * 2 + 4.0 * n * n * 4 + n * n * 4 + 5 * c * c * 2, "flops": 10.0 * n * n * c * c + 4.0 * n ** 3 * c}


def tolerance(case):
    # bf16 storage between the operators: about 4e-3 per block on the updated representation; the pair logits are a
    # float32 product rounded to float16
    if case["path"] == "pair_logits":
        return {"rel": 1e-3, "max": 5e-3}
    if case["path"] == "diffusion" or case.get("blocks", 1) > 2:
        return {"rel": 2e-2}
    return {"rel": 1e-2}
