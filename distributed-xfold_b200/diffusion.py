"""DiffusionTransformer on the sm_100a kernels (reference: nn/d_diffusion_transformer.py:37-310).

24 blocks in 6 super-blocks; per block  act += AttentionPairBias(act, mask, pair_logits, single_cond)
and  act += DiffusionTransition(act, single_cond).  A step is one C-ABI call (``xfold_diffusion_transformer_fwd``):

    conditioning             -> the LayerNorms of single_cond and two GEMMs for the modulations and gates of many blocks
    AdaptiveLayerNorm        -> LayerNorm with fused modulation
    q/k/v/gate projections   -> one GEMM with query bias and D^-0.5 folded into the epilogue
    attention (16 x 48 -> 64)-> flash kernel with the prepared pair logits
    AdaLNZero                -> output GEMM whose epilogue multiplies by sigmoid(cond) per token row and adds the residual
    DiffusionTransition      -> GEMM with SwiGLU epilogue, then the AdaLNZero GEMM

The pair logits depend only on the step-invariant ``pair_cond``; ``pair_logits()`` computes them once
per inference (the reference recomputes them every denoising step, nn/d_diffusion_transformer.py:299-305;
results are identical).  Samples are independent: ``shard_samples`` gives each rank its share by the
reference's ShardInfo rule (d_alphafold3.py:381-385); no collective is needed inside the transformer.
"""
from __future__ import annotations

import ctypes as C
from typing import Dict, List, Optional

import torch

from . import _cabi, ops
from .distribute_utils import ShardInfo

State = Dict[str, torch.Tensor]
BF16 = torch.bfloat16


class _PackedAdaLN:
    """AdaptiveLayerNorm with conditioning: scale and shift projections stacked into one [2c, c_cond] GEMM."""

    def __init__(self, state: State, prefix: str, device):
        self.cond_ln_g = ops._f32(state[prefix + "single_cond_layer_norm.weight"], device)
        w = torch.cat([state[prefix + "single_cond_scale.weight"], state[prefix + "single_cond_bias.weight"]], 0)
        self.w = ops._b16(w, device)
        c = state[prefix + "single_cond_scale.weight"].shape[0]
        b = torch.zeros(2 * c)
        b[:c] = state[prefix + "single_cond_scale.bias"].detach().float().cpu()
        self.b = ops._f32(b, device)
        self.c = c

    def __call__(self, x: torch.Tensor, cond: torch.Tensor) -> torch.Tensor:
        cn = ops.layernorm(cond, self.cond_ln_g, None)
        mod = ops.linear(cn, self.w, self.b)                      # [N, 2c]: scale | shift
        sc, sh = mod[:, : self.c].contiguous(), mod[:, self.c:].contiguous()
        return ops.layernorm(x, mod_scale=sc, mod_shift=sh)       # sigmoid(scale) * LN(x) + shift


def _conditioning(state: State, p_att: str, p_tr: str):
    """The conditioning projections of one block: (modulations [4c, c_cond], their bias [4c], gates [2c, c_cond], their
    bias [2c], scales of the two LayerNorms of the conditioning [2, c_cond])."""
    mod, mod_b, gate, gate_b, ln_g = [], [], [], [], []
    for p in (p_att, p_tr):
        ln = p + "adaptive_layernorm."
        ln_g.append(state[ln + "single_cond_layer_norm.weight"].detach().float()[None])
        scale_b = state[ln + "single_cond_scale.bias"].detach().float()
        mod += [state[ln + n + ".weight"].detach().float() for n in ("single_cond_scale", "single_cond_bias")]
        mod_b += [scale_b, torch.zeros_like(scale_b)]
        w = state[p + "adaptive_zero_init.adaptive_zero_cond.weight"].detach().float()
        b = state.get(p + "adaptive_zero_init.adaptive_zero_cond.bias")
        gate.append(w)
        gate_b.append(w.new_zeros(w.shape[0]) if b is None else b.detach().float())
    return mod, mod_b, gate, gate_b, ln_g


class PackedDiffusionBlock:
    def __init__(self, state: State, p_att: str, p_tr: str, device, num_head: int = 16):
        self.att = ops.PackedSelfAttention(state, p_att, device, num_head)
        self.tr_w1 = ops._b16(ops.pack_swiglu_weight(state[p_tr + "transition1.weight"]), device)
        self.tr_w2 = ops._b16(state[p_tr + "adaptive_zero_init.transition2.weight"], device)
        self.c = _cabi.DiffusionBlockWeights(ops._ptr(self.att.w_qkvg), ops._ptr(self.att.bias), ops._ptr(self.att.scale),
                                             ops._ptr(self.att.w_out), ops._ptr(self.tr_w1), ops._ptr(self.tr_w2))


class PackedDiffusionTransformer:
    def __init__(self, state: State, prefix: str, device, num_head: int = 16, num_blocks: int = 24,
                 super_block_size: int = 4):
        self.num_head, self.num_blocks, self.sb = num_head, num_blocks, super_block_size
        self.pair_ln_g = ops._f32(state.get(prefix + "pair_input_layer_norm.weight"), device)
        self.pair_ln_b = ops._f32(state.get(prefix + "pair_input_layer_norm.bias"), device)
        self.pl_w = ops._f32(torch.cat([state[prefix + f"pair_logits_projection.{i}.weight"]
                                        for i in range(num_blocks // super_block_size)], 0), device)
        names = [(prefix + f"self_attention.{i}.", prefix + f"transition_block.{i}.") for i in range(num_blocks)]
        self.blocks = [PackedDiffusionBlock(state, p_att, p_tr, device, num_head) for p_att, p_tr in names]
        parts = [_conditioning(state, p_att, p_tr) for p_att, p_tr in names]
        stack = [torch.cat([t for p in parts for t in p[k]], 0) for k in range(5)]
        self.w_mod, self.w_gate = ops._b16(stack[0], device), ops._b16(stack[2], device)
        self.b_mod, self.b_gate, self.ln_cond = (ops._f32(stack[k], device) for k in (1, 3, 4))
        a = self.blocks[0].att
        self._arr = (_cabi.DiffusionBlockWeights * num_blocks)(*[b.c for b in self.blocks])
        self.c = _cabi.DiffusionWeights(a.C, self.w_mod.shape[1], a.H, a.Dp, self.blocks[0].tr_w2.shape[1], num_blocks,
                                        ops._ptr(self.w_mod), ops._ptr(self.b_mod), ops._ptr(self.w_gate),
                                        ops._ptr(self.b_gate), self._arr, ops._ptr(self.ln_cond))

    def pair_logits(self, pair_cond: torch.Tensor) -> List[torch.Tensor]:
        """[N, N, 128] bf16 -> per super-block float16 [super_block_size, heads, N, pad8(N)], the prepared operand of the
        attention kernel (values times log2(e)): half the resident bytes of the float32 logits, and no conversion inside
        the 200 denoising steps.  ('n s (b h) -> b h n s', nn/d_diffusion_transformer.py:301-305.)"""
        prepared = ops.pair_logits_prepared(pair_cond, self.pair_ln_g, self.pair_ln_b, self.pl_w)
        return list(prepared.reshape(-1, self.sb, self.num_head, *prepared.shape[1:]).unbind(0))

    def forward(self, act: torch.Tensor, mask: Optional[torch.Tensor], single_cond: torch.Tensor,
                pair_logits: List[torch.Tensor]) -> torch.Tensor:
        """act bf16 [S, N, 768] or [N, 768] (updated in place and returned); single_cond bf16 [N, 384]."""
        ops._need_cuda(act, mask, single_cond)
        assert act.dtype == BF16 and act.is_contiguous() and act.shape[-1] == self.c.C
        assert single_cond.dtype == BF16 and single_cond.is_contiguous()
        s = 1 if act.dim() == 2 else act.shape[0]
        n = act.shape[-2]
        assert tuple(single_cond.shape) == (n, self.c.C_cond)
        shape = (self.num_head, n, (n + 7) // 8 * 8)
        ptrs, held = (C.c_void_p * self.num_blocks)(), []
        for i in range(0, self.num_blocks, self.sb):
            t, blocks = pair_logits[i // self.sb], min(self.sb, self.num_blocks - i)
            if not isinstance(t, torch.Tensor):
                t = torch.stack(list(t))
            ops._need_cuda(t)
            if t.dtype == torch.float32:   # plain logits [super_block_size, heads, N, N]
                t = ops.prepare_pair_bias(t.reshape(-1, n, n).contiguous()).reshape(-1, *shape)
            assert t.dtype == torch.float16 and t.shape[0] >= blocks and tuple(t.shape[1:]) == shape
            assert t.is_contiguous() or t[0].is_contiguous()
            base, step = t.data_ptr(), t.stride(0) * 2
            for j in range(blocks):
                ptrs[i + j] = base + j * step
            held.append(t)
        if mask is not None:
            mask = mask.to(torch.float32).contiguous()
        dev = ops._dev(act)
        lib = _cabi.load()
        ws = ops._Workspace.get(dev, lib.xfold_diffusion_workspace_bytes(s, n, C.byref(self.c)))
        rc = lib.xfold_diffusion_transformer_fwd(_cabi.ctx(dev), ops._ptr(act), s, n, ops._ptr(mask), ops._ptr(single_cond),
                                                 C.byref(self.c), ptrs, ops._ptr(ws), ws.numel(), ops._stream(dev))
        _cabi.check(rc, dev, "xfold_diffusion_transformer_fwd")
        return act


def shard_samples(num_samples: int, world: int, rank: int) -> slice:
    """Samples owned by ``rank`` (ShardInfo rule, d_alphafold3.py:381-385)."""
    return ShardInfo(num_samples, world).get_shard_slice_list()[rank]
