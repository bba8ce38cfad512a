"""KV-cached incremental decode for the Qwen3 stack (prompt expansion / "magic prompt").

``prefill`` runs the prompt once and fills a per-layer cache with the normalised, rotated keys and the values;
``decode_step`` then processes ONE token: one-row q / k / v projections, append k and v at the current position, and a
single-query grouped-query attention over the cache (each query head reads the cache of its key/value group, no
``repeat`` of the cache), followed by the MLP; ``logits`` applies the final norm and the (tied or separate) output
head to the last position. ``generate`` loops decode + host sampling until EOS or ``max_new_tokens``
(serenitymojo/llm/decoder.mojo:1-150, serenitymojo/llm/sqa.mojo:1-116)."""
from __future__ import annotations

from typing import List, Optional, Sequence

import torch

from .. import ops
from ..models.layers import globally_hooked, own_parameters
from ..models.text.qwen3 import _MLP, _Norm, _W, Qwen3Config, Qwen3Encoder, _rope
from ..ops import native
from .sampler import Rng, SamplerConfig, sample


def single_query_attention(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, length: int,
                           scale: Optional[float] = None) -> torch.Tensor:
    """q [B, H, Dh] (one position), caches [B, Hkv, T, Dh] valid up to ``length`` -> [B, H, Dh]. Query head h reads
    key/value head h // (H / Hkv); scores and the weighted sum are accumulated in fp32."""
    B, H, Dh = q.shape
    Hkv = k_cache.shape[1]
    rep = H // Hkv
    scale = scale if scale is not None else Dh ** -0.5
    qg = q.view(B, Hkv, rep, Dh).float()
    k = k_cache[:, :, :length].float()
    v = v_cache[:, :, :length].float()
    s = torch.einsum("bgrd,bgtd->bgrt", qg, k) * scale
    p = torch.softmax(s, dim=-1)
    return torch.einsum("bgrt,bgtd->bgrd", p, v).reshape(B, H, Dh).to(q.dtype)


class KVCache:
    def __init__(self, cfg: Qwen3Config, batch: int, max_len: int, dtype, device):
        shape = (cfg.num_hidden_layers, batch, cfg.num_key_value_heads, max_len, cfg.head_dim)
        self.k = torch.zeros(shape, dtype=dtype, device=device)
        self.v = torch.zeros(shape, dtype=dtype, device=device)
        self.length = 0
        self.max_len = max_len
        self.rope = None                # (cos, sin) [positions, head_dim] for the fused decode step, filled by the prefill on the GPU


class Qwen3Decoder:
    """Wraps a :class:`Qwen3Encoder` (same weights, same parameter names) with an output head for generation."""

    def __init__(self, encoder: Qwen3Encoder, lm_head: Optional[torch.Tensor] = None):
        self.enc = encoder
        self.cfg = encoder.cfg
        self.lm_head = lm_head          # [vocab, hidden]; None: tied to the embedding table

    def _angles(self, pos: torch.Tensor, dtype):
        c = self.cfg
        inv = 1.0 / (c.rope_theta ** (torch.arange(0, c.head_dim, 2, device=pos.device).float() / c.head_dim))
        ang = pos.float()[:, None] * inv[None]
        emb = torch.cat((ang, ang), dim=-1)
        return emb.cos().to(dtype), emb.sin().to(dtype)

    def _native(self, x: torch.Tensor) -> bool:
        """Whether the fused decode-step kernels cover this configuration: bf16 on the GPU, 16-byte rows, heads of up to 256. They
        round to bf16 where the separate operations do."""
        c = self.cfg
        return (native.use_native(x) and x.dtype == torch.bfloat16 and c.qk_norm and c.hidden_size % 8 == 0 and c.hidden_size <= 16384
                and c.intermediate_size % 8 == 0 and c.head_dim % 8 == 0 and c.head_dim <= 256 and x.numel() > 0
                and c.num_attention_heads % c.num_key_value_heads == 0)

    def _fused_layers(self, x: torch.Tensor, cache: KVCache, pos: int, batch: Optional[int] = None):
        """Per layer ((norm, q, k, v, biases, q norm, k norm), (o, norm, gate, up, down)) for the fused kernels, or None when the
        separate operations have to run: a module that a program hooked, replaced or gave another epsilon or bias, weights or
        caches of another type, shape or layout. Looked at anew on every step. x [rows, hidden]: one row per sequence at ``pos``, or
        (``batch`` given) the rows of a prompt that ends there."""
        c, rope = self.cfg, getattr(cache, "rope", None)
        if rope is None or not self._native(x) or pos >= native.ops().llm_decode_attention_max() or x.dim() != 2 or globally_hooked():
            return None
        D, Dh, F, eps = c.hidden_size, c.head_dim, c.intermediate_size, c.rms_norm_eps
        Q, KV = c.num_attention_heads * Dh, c.num_key_value_heads * Dh
        layers, flat, has = [], [], None
        for l in self.enc.model.layers:
            l = l._modules
            a, mlp, norm = l["self_attn"]._modules, l["mlp"], own_parameters(l["input_layernorm"], _Norm)
            post, q_norm, k_norm = own_parameters(l["post_attention_layernorm"], _Norm), own_parameters(a["q_norm"], _Norm), own_parameters(a["k_norm"], _Norm)
            if own_parameters(mlp, _MLP) is None or norm is None or post is None or q_norm is None or k_norm is None:
                return None
            if not l["input_layernorm"].eps == l["post_attention_layernorm"].eps == a["q_norm"].eps == a["k_norm"].eps == eps:
                return None
            m, ps = mlp._modules, []
            for mod in (a["q_proj"], a["k_proj"], a["v_proj"], a["o_proj"], m["gate_proj"], m["up_proj"], m["down_proj"]):
                p = own_parameters(mod, _W)
                if p is None or mod.__dict__.get("bias") is not None:      # a plain tensor in the place of the parameter
                    return None
                ps.append(p)
            q, k, v, o, gate, up, down = ps
            if "bias" in o or "bias" in gate or "bias" in up or "bias" in down:
                return None
            bias = [p.get("bias") for p in (q, k, v)]
            some = [t for t in bias if t is not None]
            if has is None:
                has = len(some)
            try:
                qkv = (norm["weight"], q["weight"], k["weight"], v["weight"], *bias, q_norm["weight"], k_norm["weight"])
                rest = (o["weight"], post["weight"], gate["weight"], up["weight"], down["weight"])
            except KeyError:                                               # a weight that is no parameter any more
                return None
            if len(some) != has or has not in (0, 3):
                return None
            layers.append((qkv, rest))
            flat += [t for t in qkv if t is not None] if has == 0 else qkv
            flat += rest
        # one call looks at type, device, layout, alignment and shape of all weights: the launches refuse what the separate
        # operations broadcast or copy
        shapes = [D, 0, Q, D, KV, D, KV, D, *([Q, 0, KV, 0, KV, 0] if has else []), Dh, 0, Dh, 0, D, Q, D, 0, F, D, F, D, D, F]
        kv = (len(layers), x.shape[0] if batch is None else batch, c.num_key_value_heads, cache.k.shape[3] if cache.k.dim() == 5 else 0, Dh)
        if kv[3] <= pos or cache.k.shape != kv or cache.v.shape != kv or any(t.dim() != 2 or t.shape[0] <= pos or t.shape[1] != Dh for t in rope):
            return None
        ok = native.ops().bf16_operands_ok
        return layers if ok([x, cache.k, cache.v, *rope], [-1, 0]) and (not layers or flat[0].device == x.device and ok(flat, shapes)) else None

    @torch.no_grad()
    def prefill(self, ids: torch.Tensor, max_len: int) -> "tuple[torch.Tensor, KVCache]":
        """ids [B, S] -> (hidden of the last position [B, hidden], cache holding positions 0..S-1)."""
        c, m = self.cfg, self.enc.model
        B, S = ids.shape
        x = m.embed_tokens(ids)
        cache = KVCache(c, B, max_len, x.dtype, ids.device)
        cos, sin = self._angles(torch.arange(S, device=ids.device), x.dtype)
        cos, sin = cos[None, None], sin[None, None]
        mask = torch.full((S, S), float("-inf"), device=ids.device, dtype=x.dtype).triu(1)[None, None]
        rep = c.num_attention_heads // c.num_key_value_heads
        if self._native(x):
            reach = min(max_len, native.ops().llm_decode_attention_max())
            cache.rope = self._angles(torch.arange(reach, device=ids.device), x.dtype)        # for the decode steps
        # an embedding that a program hooked or replaced may return anything the modules take: rows in another order stay with them
        plain = cache.rope is not None and S > 0 and x.shape == (B, S, c.hidden_size) and x.is_contiguous() and native.direct(x)
        layers = self._fused_layers(x.view(B * S, -1), cache, S - 1, B) if plain else None
        if layers is not None:
            # updated in place: the embedding's output stays as it is
            o, x2, y = native.ops(), x.view(B * S, -1).clone(), None
            for li, (qkv, out_mlp) in enumerate(layers):
                q, k, v = o.llm_prompt_qkv(x2, y, *qkv, *cache.rope, cache.k[li], cache.v[li], c.rms_norm_eps)
                attn = torch.nn.functional.scaled_dot_product_attention(q, k, v, attn_mask=mask).transpose(1, 2).reshape(B, S, -1)
                y = o.llm_prompt_mlp(x2, attn, *out_mlp, c.rms_norm_eps)
            cache.length = S
            return (x2 + y if y is not None else x2).view(B, S, -1)[:, -1], cache
        for li, l in enumerate(m.layers):
            a = l.self_attn
            h = l.input_layernorm(x)
            q = a.q_norm(a.q_proj(h).view(B, S, c.num_attention_heads, c.head_dim)).transpose(1, 2)
            k = a.k_norm(a.k_proj(h).view(B, S, c.num_key_value_heads, c.head_dim)).transpose(1, 2)
            v = a.v_proj(h).view(B, S, c.num_key_value_heads, c.head_dim).transpose(1, 2)
            q, k = _rope(q, cos, sin), _rope(k, cos, sin)
            cache.k[li, :, :, :S] = k
            cache.v[li, :, :, :S] = v
            o = torch.nn.functional.scaled_dot_product_attention(q, k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1),
                                                                 attn_mask=mask)
            x = x + a.o_proj(o.transpose(1, 2).reshape(B, S, -1))
            x = x + l.mlp(l.post_attention_layernorm(x))
        cache.length = S
        return x[:, -1], cache

    @torch.no_grad()
    def decode_step(self, token: torch.Tensor, cache: KVCache) -> torch.Tensor:
        """token [B] at position ``cache.length`` -> hidden [B, hidden]; the cache grows by one."""
        c, m = self.cfg, self.enc.model
        B = token.shape[0]
        pos = cache.length
        if pos >= cache.max_len:
            raise RuntimeError("KV cache is full")
        x = m.embed_tokens(token)                                         # [B, hidden]
        layers = self._fused_layers(x, cache, pos)
        if layers is not None:
            o, H, eps, scale, y = native.ops(), c.num_attention_heads, c.rms_norm_eps, c.head_dim ** -0.5, None
            for li, (qkv, out_mlp) in enumerate(layers):
                q = o.llm_qkv(x, y, *qkv, *cache.rope, cache.k[li], cache.v[li], pos, eps)
                y = o.llm_out_mlp(x, o.llm_decode_attention(q, cache.k[li], cache.v[li], H, pos + 1, scale), *out_mlp, eps)
            cache.length = pos + 1
            return x + y if y is not None else x
        cos, sin = self._angles(torch.tensor([pos], device=token.device), x.dtype)
        for li, l in enumerate(m.layers):
            a = l.self_attn
            h = l.input_layernorm(x)
            q = _rope(a.q_norm(a.q_proj(h).view(B, c.num_attention_heads, c.head_dim)), cos, sin)
            k = _rope(a.k_norm(a.k_proj(h).view(B, c.num_key_value_heads, c.head_dim)), cos, sin)
            cache.k[li, :, :, pos] = k
            cache.v[li, :, :, pos] = a.v_proj(h).view(B, c.num_key_value_heads, c.head_dim)
            o = single_query_attention(q, cache.k[li], cache.v[li], pos + 1)
            x = x + a.o_proj(o.reshape(B, -1))
            x = x + l.mlp(l.post_attention_layernorm(x))
        cache.length = pos + 1
        return x

    @torch.no_grad()
    def logits(self, hidden: torch.Tensor) -> torch.Tensor:
        h = self.enc.model.norm(hidden)
        w = self.lm_head if self.lm_head is not None else self.enc.model.embed_tokens.weight
        if (native.use_native(h) and native.direct(h, w) and h.dtype == w.dtype == torch.bfloat16 and h.dim() == w.dim() == 2 and 0 < h.shape[0] <= 8
                and h.shape[1] == w.shape[1] and h.shape[1] % 8 == 0 and native.ops().bf16_operands_ok([h, w], [-1, 0])):
            # products of bf16 values are exact in fp32 and the few-row kernel sums in fp32: the table needs no fp32 copy
            return ops.functional._gemm([h], [w], out_fp32=True)
        return h.float() @ w.float().t()

    @torch.no_grad()
    def generate(self, prompt_ids: Sequence[int], max_new_tokens: int, cfg: SamplerConfig = SamplerConfig(),
                 eos_ids: Sequence[int] = (), device=None) -> List[int]:
        dev = device or next(self.enc.parameters()).device
        ids = torch.tensor([list(prompt_ids)], dtype=torch.long, device=dev)
        hidden, cache = self.prefill(ids, ids.shape[1] + max_new_tokens)
        rng = Rng(cfg.seed)
        out: List[int] = []
        for _ in range(max_new_tokens):
            tok = sample(self.logits(hidden)[0].tolist(), cfg, rng)
            out.append(tok)
            if tok in eos_ids or cache.length >= cache.max_len:
                break
            hidden = self.decode_step(torch.tensor([tok], dtype=torch.long, device=dev), cache)
        return out
