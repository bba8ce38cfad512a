"""The workloads whose speed is tracked: one pass each through the public entry points of the package.

Six kinds of work cover what a user has the framework do:

* ``flux``       text-to-image denoising with the FLUX.1-shaped 12 B MMDiT through ``FluxPipeline.denoise``
* ``flux_lora``  one LoRA rank-16 training step of the same model through ``FlowMatchTrainer.step``
* ``sdxl``       one guided denoise step of the SDXL UNet (conditional and unconditional sample in one batch)
* ``sdxl_lora``  one LoRA rank-16 training step of that UNet (forward and backward of convolutions, norms, attention)
* ``vae``        the FLUX image autoencoder, encode or decode
* ``video``      one denoise step of the LTX-2-shaped 13 B video DiT, bf16 or with fp8-resident block weights
* ``llm``        prompt expansion with the Qwen3-4B-shaped decoder: prefill, then one token at a time

Weights are random with the variance a trained network of that width has (1 / fan-in), inputs are unit normal like
latents and text features. All of it is drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import torch

from mojodiffusion_b200 import ops
from mojodiffusion_b200.llm.decoder import Qwen3Decoder
from mojodiffusion_b200.models.mmdit import MMDiT, flux1_dev_config
from mojodiffusion_b200.models.text.qwen3 import Qwen3Config, Qwen3Encoder
from mojodiffusion_b200.models.unet import UNet, sdxl_config
from mojodiffusion_b200.models.vae import AutoencoderKL, flux_vae_config
from mojodiffusion_b200.models.video_dit import VideoDiT, ltx2_config
from mojodiffusion_b200.pipeline.flux import FluxPipeline
from mojodiffusion_b200.training import lora as L
from mojodiffusion_b200.training.optim import FusedAdamW
from mojodiffusion_b200.training.trainer import FlowMatchTrainer

DEV = "cuda"
BF16 = torch.bfloat16


# ---- the cases -------------------------------------------------------------------------------------------------
def listed():
    return [
        # the headline of the benchmark: one step of a 1024 x 1024 image (64 x 64 packed latent tokens, 512 text tokens)
        dict(name="flux_1024", kind="flux", batch=1, h=64, w=64, text=512, steps=1),
        # two images of an odd aspect ratio in one batch, a text length that fills no tile
        dict(name="flux_ragged_batch2", kind="flux", batch=2, h=47, w=35, text=333, steps=1),
        # a whole four-step 256 x 256 preview: streaming the weights and launching bound it, not arithmetic
        dict(name="flux_256_preview", kind="flux", batch=1, h=16, w=16, text=256, steps=4),
        # LoRA training at 1024 x 1024 with per-block recompute, the default of the training benchmark
        dict(name="flux_lora_1024", kind="flux_lora", batch=1, h=64, w=64, text=512, recompute=True),
        # LoRA training at about 512 x 512 in an aspect-ratio bucket, activations kept
        dict(name="flux_lora_bucket", kind="flux_lora", batch=1, h=27, w=37, text=512, recompute=False),
        # one guided SDXL step at 1024 x 1024
        dict(name="sdxl_1024", kind="sdxl", images=1, h=128, w=128),
        # SDXL LoRA training in an aspect-ratio bucket (832 x 1216)
        dict(name="sdxl_lora_bucket", kind="sdxl_lora", images=1, h=104, w=152),
        # the last stage of every image: latent to 1024 x 1024 pixels
        dict(name="vae_decode_1024", kind="vae", way="decode", images=1, h=128, w=128),
        # caching latents of a dataset: three images of an odd size (latent 61 x 89)
        dict(name="vae_encode_ragged", kind="vae", way="encode", images=3, h=61, w=89),
        # a clip of 6144 latent tokens, bf16 weights
        dict(name="video_bf16", kind="video", batch=1, frames=8, h=24, w=32, text=256, fp8=False),
        # a shorter clip of an odd size with the fp8-resident serving weights
        dict(name="video_fp8_ragged", kind="video", batch=1, frames=7, h=17, w=23, text=201, fp8=True),
        # a 45-token prompt and eight generated tokens: latency of the smallest calls
        dict(name="llm_expand", kind="llm", prompt=45, new=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo_area, hi_area, step=1):
    """(h, w) of a log-uniform area and an aspect ratio from 1:2 to 2:1, both multiples of ``step``."""
    area = math.exp(rng.uniform(math.log(lo_area), math.log(hi_area)))
    ratio = math.exp(rng.uniform(-math.log(2.0), math.log(2.0)))
    h = max(1, int(math.sqrt(area * ratio) / step)) * step
    return h, max(1, int(area / h / step)) * step


def draw(rng):
    kind = rng.choice(["flux", "flux", "flux_lora", "flux_lora", "sdxl", "sdxl_lora", "vae", "vae", "video", "video", "llm"])
    if kind == "flux":
        batch = rng.choice([1, 1, 2])
        h, w = _sides(rng, 256, 4096 // batch)
        return dict(kind=kind, batch=batch, h=h, w=w, text=rng.randint(64, 512), steps=rng.randint(2, 4) if h * w * batch < 1024 else 1)
    if kind == "flux_lora":
        recompute = rng.random() < 0.5
        h, w = _sides(rng, 256, 3600 if recompute else 2304)
        return dict(kind=kind, batch=1, h=h, w=w, text=rng.choice([rng.randint(64, 512), 512]), recompute=recompute)
    if kind == "sdxl":
        h, w = _sides(rng, 64 * 64, 128 * 128, 4)
        return dict(kind=kind, images=1 if h * w > 8192 else rng.choice([1, 2]), h=h, w=w)
    if kind == "sdxl_lora":
        h, w = _sides(rng, 64 * 64, 104 * 152, 4)
        return dict(kind=kind, images=1, h=h, w=w)
    if kind == "vae":
        h, w = _sides(rng, 32 * 32, 128 * 128)
        return dict(kind=kind, way=rng.choice(["decode", "encode"]), images=1 if h * w > 6000 else rng.randint(1, 3), h=h, w=w)
    if kind == "video":
        frames = rng.randint(1, 9)
        h, w = _sides(rng, 128, max(129, 6144 // frames if frames > 2 else 2048))
        return dict(kind=kind, batch=1, frames=frames, h=h, w=w, text=rng.randint(64, 256), fp8=rng.random() < 0.5)
    return dict(kind="llm", prompt=_log_int(rng, 9, 512), new=rng.randint(4, 12))


# ---- what a program holds before the call --------------------------------------------------------------------------
#: projections that write back into a transformer's residual stream
BACK = ("attn.proj.weight", "mlp.2.weight", "linear2.weight", "to_out.0.weight", "ff.net.2.weight", "o_proj.weight", "down_proj.weight")


@torch.no_grad()
def _fill(model, gen, depth=1):
    """Matrices and convolutions normal with variance 1 / fan-in, divided by 2 x depth where a branch joins the residual
    stream (what keeps a stack of 50 blocks as well conditioned as a trained one), biases small, norm weights around one."""
    for name, p in model.named_parameters():
        if p.dim() >= 2:
            fan_in = p.shape[-1] if p.dim() == 2 else p[0].numel()
            std = 0.02 if "table" in name or "embed_tokens" in name else fan_in ** -0.5
            p.normal_(0.0, std * (2 * depth) ** -0.5 if name.endswith(BACK) else std, generator=gen)
        else:
            norm = name.endswith("scale") or name.endswith("weight")
            p.normal_(1.0 if norm else 0.0, 0.05, generator=gen)
    return model


def _lora(model, inject, gen):
    """Rank-16 adapters in mid-training: both factors non-zero."""
    slots = inject(model, rank=16, alpha=16.0)
    params = L.lora_parameters(slots)
    with torch.no_grad():
        for s in slots:
            s.down.normal_(0.0, s.down.shape[1] ** -0.5, generator=gen)
            s.up.normal_(0.0, 0.01, generator=gen)
    return params, FusedAdamW(params, lr=1e-4, max_grad_norm=1.0)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)

    def rn(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device=DEV, dtype=dtype)

    kind = case["kind"]
    s = dict(case=case)
    if kind in ("flux", "flux_lora"):
        cfg = flux1_dev_config()
        model = _fill(MMDiT(cfg, BF16, DEV), gen, cfg.depth_double + cfg.depth_single)
        B, S = case["batch"], case["h"] * case["w"]
        s.update(x=rn(B, S, cfg.in_channels), txt=rn(B, case["text"], cfg.context_dim, dtype=BF16), y=rn(B, cfg.vec_dim, dtype=BF16))
        if kind == "flux":
            s["pipe"] = FluxPipeline(model.eval(), DEV)
        else:
            params, opt = _lora(model, L.inject_flux_lora, gen)
            model.gradient_checkpointing = case["recompute"]
            model.train()
            s.update(params=params, trainer=FlowMatchTrainer(model, params, opt), noise=rn(B, S, cfg.in_channels),
                     sigma=torch.rand(B, generator=gen, device=DEV) * 0.8 + 0.1)
    elif kind in ("sdxl", "sdxl_lora"):
        cfg = sdxl_config()
        model = _fill(UNet(cfg, BF16, DEV), gen)
        n = case["images"] * (2 if kind == "sdxl" else 1)
        s.update(model=model, x=rn(case["images"], cfg.in_channels, case["h"], case["w"]), ctx=rn(n, 77, cfg.context_dim, dtype=BF16),
                 y=rn(n, cfg.adm_in_channels, dtype=BF16), t=torch.randint(50, 950, (1,), generator=gen, device=DEV).float().expand(n).contiguous())
        if kind == "sdxl":
            model.eval()
        else:
            s["params"], s["opt"] = _lora(model, L.inject_sdxl_lora, gen)
            s["noise"] = rn(*s["x"].shape)
            model.train()
    elif kind == "vae":
        cfg = flux_vae_config()
        s["model"] = _fill(AutoencoderKL(cfg, BF16, DEV), gen).eval()
        n, h, w = case["images"], case["h"], case["w"]
        s["x"] = rn(n, cfg.z_channels, h, w) if case["way"] == "decode" else rn(n, 3, 8 * h, 8 * w).clamp_(-1, 1)
    elif kind == "video":
        cfg = ltx2_config()
        model = _fill(VideoDiT(cfg, BF16, DEV), gen, cfg.depth).eval()
        if case["fp8"]:
            model.to_fp8(4, 46)
        S = case["frames"] * case["h"] * case["w"]
        s.update(model=model, x=rn(case["batch"], S, cfg.in_channels), ctx=rn(case["batch"], case["text"], cfg.context_dim, dtype=BF16),
                 t=torch.rand(case["batch"], generator=gen, device=DEV))
    else:
        cfg = Qwen3Config()
        s["dec"] = Qwen3Decoder(_fill(Qwen3Encoder(cfg, BF16, DEV), gen, cfg.num_hidden_layers).eval())
        s["ids"] = torch.randint(0, cfg.vocab_size, (1, case["prompt"]), generator=gen, device=DEV)
        # the continuation is given: a sampled one would hang on the last bit of nearly equal logits
        s["next"] = torch.randint(0, cfg.vocab_size, (case["new"], 1), generator=gen, device=DEV)
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "flux":
        return s["pipe"].denoise(s["x"], s["txt"], s["y"], steps=case["steps"], guidance=3.5, hw=(case["h"], case["w"]))
    if kind == "flux_lora":
        loss = s["trainer"].step(s["x"], s["txt"], s["y"], sigma=s["sigma"], noise=s["noise"], hw=(case["h"], case["w"]))
        return {"loss": loss, "grads": torch.cat([p.grad.reshape(-1) for p in s["params"]])}
    if kind == "sdxl":
        with torch.no_grad():
            n = case["images"]
            eps = s["model"](torch.cat((s["x"], s["x"])).to(BF16), s["t"], s["ctx"], s["y"]).float()
            return s["x"] - 0.05 * (eps[n:] + 7.0 * (eps[:n] - eps[n:]))
    if kind == "sdxl_lora":
        s["opt"].zero_grad(set_to_none=True)
        xt = (0.7 * s["x"] + 0.714 * s["noise"]).to(BF16)
        loss = (s["model"](xt, s["t"], s["ctx"], s["y"]).float() - s["noise"]).square().mean()
        loss.backward()
        s["opt"].step()
        return {"loss": loss.detach(), "grads": torch.cat([p.grad.reshape(-1) for p in s["params"]])}
    if kind == "vae":
        with torch.no_grad():
            return s["model"].decode(s["x"]) if case["way"] == "decode" else s["model"].encode(s["x"], sample=False)
    if kind == "video":
        with torch.no_grad():
            return s["model"](s["x"].to(BF16), s["ctx"], s["t"], (case["frames"], case["h"], case["w"]))
    hidden, cache = s["dec"].prefill(s["ids"], case["prompt"] + case["new"])
    out = [s["dec"].logits(hidden)]
    for token in s["next"]:
        out.append(s["dec"].logits(s["dec"].decode_step(token, cache)))
    return torch.cat(out)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def _attn(batch, q, k, width):
    return 4.0 * batch * q * k * width


def _unet_work(images, h, w, ctx_len=77):
    """Multiply-adds x 2 and weight bytes of one SDXL UNet forward over ``images`` samples."""
    c = sdxl_config()
    flops = weights = 0.0
    px = h * w

    def conv(cin, cout, k, pix):
        nonlocal flops, weights
        flops += 2.0 * images * pix * cin * cout * k * k
        weights += cin * cout * k * k

    def lin(cin, cout, rows):
        nonlocal flops, weights
        flops += 2.0 * images * rows * cin * cout
        weights += cin * cout

    def res(cin, cout, pix):
        conv(cin, cout, 3, pix)
        conv(cout, cout, 3, pix)
        lin(4 * c.model_channels, cout, 1)
        if cin != cout:
            conv(cin, cout, 1, pix)

    def spatial(ch, depth, pix):
        nonlocal flops
        lin(ch, ch, pix)
        lin(ch, ch, pix)
        for _ in range(depth):
            lin(ch, 4 * ch, pix)                                       # self-attention q, k, v, out
            lin(ch, 2 * ch, pix)                                       # cross-attention q, out
            lin(c.context_dim, 2 * ch, ctx_len)
            lin(ch, 8 * ch, pix)
            lin(4 * ch, ch, pix)
            flops += _attn(images, pix, pix, ch) + _attn(images, pix, ctx_len, ch)

    mc, ch = c.model_channels, c.model_channels
    conv(c.in_channels, mc, 3, px)
    chans = [ch]
    levels = len(c.channel_mult)
    for i, m in enumerate(c.channel_mult):
        pix = px // 4 ** i
        for _ in range(c.num_res_blocks):
            res(ch, m * mc, pix)
            ch = m * mc
            spatial(ch, c.transformer_depth[i], pix) if c.transformer_depth[i] else None
            chans.append(ch)
        if i != levels - 1:
            conv(ch, ch, 3, pix // 4)
            chans.append(ch)
    pix = px // 4 ** (levels - 1)
    res(ch, ch, pix)
    spatial(ch, c.transformer_depth[-1], pix)
    res(ch, ch, pix)
    for i in reversed(range(levels)):
        pix = px // 4 ** i
        for j in range(c.num_res_blocks + 1):
            res(ch + chans.pop(), c.channel_mult[i] * mc, pix)
            ch = c.channel_mult[i] * mc
            spatial(ch, c.transformer_depth[i], pix) if c.transformer_depth[i] else None
            if i and j == c.num_res_blocks:
                conv(ch, ch, 3, pix * 4)
    conv(ch, c.out_channels, 3, px)
    return flops, weights


def _vae_work(way, images, h, w):
    c = flux_vae_config()
    flops = weights = 0.0

    def conv(cin, cout, k, pix):
        nonlocal flops, weights
        flops += 2.0 * images * pix * cin * cout * k * k
        weights += cin * cout * k * k

    def res(cin, cout, pix):
        conv(cin, cout, 3, pix)
        conv(cout, cout, 3, pix)
        if cin != cout:
            conv(cin, cout, 1, pix)

    top, levels, small = c.ch * c.ch_mult[-1], len(c.ch_mult), h * w
    res(top, top, small)
    res(top, top, small)
    conv(top, 4 * top, 1, small)
    flops += _attn(images, small, small, top)
    if way == "decode":
        conv(c.z_channels, top, 3, small)
        ch = top
        for i in reversed(range(levels)):
            pix = small * 4 ** (levels - 1 - i)
            for _ in range(c.num_res_blocks + 1):
                res(ch, c.ch * c.ch_mult[i], pix)
                ch = c.ch * c.ch_mult[i]
            if i:
                conv(ch, ch, 3, 4 * pix)
        conv(ch, 3, 3, small * 64)
        return flops, weights, images * small * (4 * c.z_channels + 64 * 3 * 2)
    conv(3, c.ch, 3, small * 64)
    ch = c.ch
    for i in range(levels):
        pix = small * 4 ** (levels - 1 - i)
        for _ in range(c.num_res_blocks):
            res(ch, c.ch * c.ch_mult[i], pix)
            ch = c.ch * c.ch_mult[i]
        if i != levels - 1:
            conv(ch, ch, 3, pix // 4)
    conv(top, 2 * c.z_channels, 3, small)
    return flops, weights, images * small * (64 * 3 * 4 + 4 * c.z_channels)


def work(case):
    kind = case["kind"]
    if kind in ("flux", "flux_lora"):
        c = flux1_dev_config()
        D, B = c.hidden, case["batch"]
        si, st = case["h"] * case["w"], case["text"]
        S, blocks = si + st, c.depth_double + c.depth_single
        linear = 2.0 * B * (S * blocks * 12 * D * D + (2 * si * c.in_channels + st * c.context_dim) * D)
        attn = blocks * _attn(B, S, S, D)
        weights = D * D * (c.depth_double * 36 + c.depth_single * 15 + 8.0) + D * (c.context_dim + c.vec_dim)
        io = B * (8.0 * si * c.in_channels + 2 * st * c.context_dim)
        if kind == "flux":
            return {"bytes": case["steps"] * (2 * weights + io), "flops": case["steps"] * (linear + attn)}
        adapters = 16 * D * (c.depth_double * 2 * (3 * 2 + 2 + 5 + 5) + c.depth_single * (3 * 2 + 5 + 6.0))
        # forward, input gradients (frozen weights have none of their own), the five products of the attention backward;
        # the weights are read by both directions, an adapter entry moves weight, gradient and two fp32 moments
        return {"bytes": 4 * weights + 2 * io + adapters * 24, "flops": 2 * linear + 3.5 * attn + 6.0 * B * S * adapters}
    if kind == "sdxl":
        flops, weights = _unet_work(2 * case["images"], case["h"], case["w"])
        return {"bytes": 2 * weights + case["images"] * case["h"] * case["w"] * 32.0, "flops": flops}
    if kind == "sdxl_lora":
        flops, weights = _unet_work(case["images"], case["h"], case["w"])
        return {"bytes": 4 * weights, "flops": 2.2 * flops}
    if kind == "vae":
        flops, weights, io = _vae_work(case["way"], case["images"], case["h"], case["w"])
        return {"bytes": 2 * weights + io, "flops": flops}
    if kind == "video":
        c = ltx2_config()
        D, B, S, T = c.hidden, case["batch"], case["frames"] * case["h"] * case["w"], case["text"]
        block = 6.0 * D * D + 2 * D * c.ffn_hidden                     # per latent token: q, k, v, out, cross q, out, feed-forward
        cross = 2.0 * D * c.context_dim                               # per text token: cross k, v
        flops = c.depth * (2.0 * B * (S * block + T * cross) + _attn(B, S, S, D) + _attn(B, S, T, D))
        weights = c.depth * (block + cross)
        per = 2.0 if not case["fp8"] else (2.0 * (c.depth - 42) + 42) / c.depth
        return {"bytes": weights * per + B * (S * c.in_channels * 6.0 + T * c.context_dim * 2), "flops": flops}
    c = Qwen3Config()
    n, layers = case["new"], c.num_hidden_layers
    kv = c.num_key_value_heads * c.head_dim
    layer = c.hidden_size * (2 * c.num_attention_heads * c.head_dim + 2 * kv + 3.0 * c.intermediate_size)
    head = float(c.hidden_size * c.vocab_size)
    tokens = case["prompt"] + n
    cache = sum(case["prompt"] + i for i in range(n + 1)) * 4.0 * kv * layers
    return {"bytes": (n + 1) * 2 * (layers * layer + head) + cache + (n + 1) * 4.0 * c.vocab_size,
            "flops": 2 * tokens * layers * layer + 2 * (n + 1) * head + 4.0 * layers * c.num_attention_heads * c.head_dim * (case["prompt"] ** 2 / 2 + n * tokens)}


# ---- how far another correct implementation may be off -------------------------------------------------------------------
#: Largest relative errors, about four times what was measured on the listed cases between this package's kernels and the
#: same models on PyTorch's library kernels in bf16 (flux 0.008, video 0.009, sdxl 0.005, vae 0.012) or, for the training
#: steps and the fp8 weights, between two tilings of the GEMM and two forms of the exponential (flux_lora 0.0026, sdxl_lora
#: 0.005, which is also what two runs of its split sums differ by, fp8 0.0125: one bf16 rounding can move an activation by a
#: whole fp8 step). Single gradient entries are off by more than that share of their root mean square (up to 0.4 measured).
#: The decoder's own bf16 roundings of scores and probabilities decide for ``llm``.
REL = {"flux": 0.03, "flux_lora": 0.015, "sdxl": 0.02, "sdxl_lora": 0.025, "vae": 0.03, "video": 0.03, "llm": 0.02}


def tolerance(case):
    return {"rel": REL[case["kind"]], "max": 0.99} if case["kind"].endswith("lora") else {"rel": REL[case["kind"]]}
