"""`transformers` attention-backend callable built on `intra_llm_attn`.

The reference ships a PyTorch restatement of the kernel's language-model patterns as an
ALL_ATTENTION_FUNCTIONS-style callable (experiments/llm/intra_token_attn.py:112-134): two Scatter
layers, then two 64-aligned-window layers, repeating, with dense attention for single-token decode
steps because the patterns are prefill-only. This module offers the same callable with the prefill
running on the B200 kernels: query/key/value arrive as (B, H, S, D) and are handed to the kernel as
(B, S, H, D) views without copies. The decode step is dense over the cache, as in the reference: on the
library's decode kernel for bf16 caches with or without a padding mask, else, and for multi-head caches that
SDPA is quicker on, one SDPA call.

    from transformers import AttentionInterface
    AttentionInterface.register("intra_b200", make_intra_attention())
    model = AutoModelForCausalLM.from_pretrained(..., attn_implementation="intra_b200")
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .interface import _llm, decode_attn

NUM_GROUPS = 8          # intra_token_attn.py:22-24
WINDOW_BACK = 512
WINDOW_CHUNK = 64


def layer_masktype(layer_idx: int) -> int:
    """Kernel mask id of a layer: 0 (Scatter) for layer_idx % 4 in {0, 1}, 4 (window) otherwise
    (intra_token_attn.py:112-114)."""
    return 0 if layer_idx % 4 in (0, 1) else 4


def _kernel_is_quicker(units, S, masked):
    """Is the decode kernel quicker than SDPA on caches of S keys with as many KV heads as query heads, `units` of them in
    the batch? With one query row per KV head it has nothing to reuse. Measured on one B200, us:
    * without a mask its GPU time is 0.9-1.7 times SDPA's over 8-8192 units of 17-24000 keys, except where its 8 CTAs per
      unit fill the chip (32 units, K and V of 28 / 64 / 100 MB: 8.1 / 14.1 / 18.7 against 8.4 / 15.3 / 19.9). But its way
      to the launch is shorter, which decides calls of up to 44 MB: 13-14.4 a call against 15.4-19.3 (replayed from a CUDA
      graph, where that does not count, such calls take 4-14 against 3-12). Below 24 units the kernel takes a second launch
      from 28 MB on (20.7 a call against 19.3), and beyond 256 units its GPU time shows (512 units, 44 MB: 17.5 against
      15.7; 1024: 16.8-18.6 against 15.8-17.0 from the shortest caches on);
    * with a mask it is quicker, but for the shortest caches of many units: up to 32 keys of 4096 units a call takes 64
      against 59 (2048 units: 33 against 39).
    The choice goes by sizes alone: a call that is captured runs what its warm-up ran."""
    if masked:
        return S > 32 or units < 4096
    nbytes = units * S * 512                         # K and V
    if 28 <= units <= 37:
        return nbytes <= 100e6
    return units <= 512 and nbytes <= (44e6 if 24 <= units <= 256 else 28e6)


def make_intra_attention(num_groups: int = NUM_GROUPS, back: int = WINDOW_BACK, chunk: int = WINDOW_CHUNK,
                         force_masktype=None):
    """Returns `fn(module, query, key, value, attention_mask=None, scaling=None, dropout=0.0, **kw)`
    -> (output (B, S, H, D), None), the signature transformers expects of an attention backend."""
    if chunk != 64:
        raise ValueError("the window kernel aligns its lookback to 64-query blocks")
    window = back + chunk      # a 64-query block sees itself plus `back` earlier tokens

    def intra_attention_forward(module, query, key, value, attention_mask=None, scaling=None, dropout=0.0,
                                **kwargs):
        if query.shape[2] == 1:          # decode step: dense over the cache, as the reference does
            rep = query.shape[1] // key.shape[1]
            if rep != 1 or _kernel_is_quicker(query.shape[0] * query.shape[1], key.shape[2], attention_mask is not None):
                out = decode_attn(query, key, value, attention_mask, scaling)
                if out is not None:
                    return out, None
            k2 = key.repeat_interleave(rep, dim=1) if rep > 1 else key
            v2 = value.repeat_interleave(rep, dim=1) if rep > 1 else value
            am = attention_mask[:, :, :, : k2.shape[-2]] if attention_mask is not None else None
            o = F.scaled_dot_product_attention(query, k2, v2, attn_mask=am, scale=scaling, is_causal=False)
            return o.transpose(1, 2).contiguous(), None
        mt = force_masktype if force_masktype is not None else layer_masktype(getattr(module, "layer_idx", 0))
        if torch.is_grad_enabled():          # the kernels are forward-only; this callable is, too
            query, key, value = query.detach(), key.detach(), value.detach()
        out = _llm(query, key, value, 2, 1, "scatter" if mt == 0 else "window", num_groups, window, scaling, True, False, None)
        return out, None

    return intra_attention_forward
