"""Kernel variants chosen by size: each against the plain fp32 statement of the op at the sizes where it can go wrong."""
import math

import pytest
import torch

import mojodiffusion_b200.ops as O
from mojodiffusion_b200.ops import native, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"
if torch.cuda.is_available():
    native.load(True)


def _rand(*shape, scale=1.0, seed=0, dtype=torch.bfloat16):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def _close(out, want, name, rel=0.0):
    """bf16 outputs of fp32 sums: the rounding of the value (2^-9, doubled because two sums may round to neighbours), plus ``rel``
    of the largest value for what the inputs of that rounding may differ by."""
    native.check_status(out)
    assert out.shape == want.shape and torch.isfinite(out.float()).all(), name
    w = want.float()
    err = (out.float() - w).abs()
    bound = w.abs() * 2.0 ** -8 + (rel + 1e-5) * float(w.abs().max())
    assert bool((err <= bound).all()), f"{name}: {float((err - bound).max())} over the bound, largest {float(w.abs().max())}"


# rows 1 / 2 / 4 / 8 are the kernel's own sizes, 3 / 5 / 7 repeat a row, 9 is the first on the tiled kernel; K = 8 leaves 31 lanes
# idle, 264 / 520 end in a partial step; N = 1000 ends inside a block, 9480 takes four columns per warp on 148 SMs
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 7, 8, 9])
@pytest.mark.parametrize("N,K", [(56, 8), (1000, 264), (5000, 520), (9480, 3072)])
def test_few_row_gemm(M, N, K):
    x, w = _rand(M, K, seed=M), _rand(N, K, scale=1 / math.sqrt(K), seed=2)
    bias, gate, res = _rand(N, seed=7), _rand(M, N, seed=8), _rand(M, N, seed=9)
    _close(O.linear(x, w), x.float() @ w.float().t(), f"plain {M}x{N}x{K}")
    for act in ("gelu_tanh", "silu", "gelu"):
        out = O.linear(x, w, bias, act=act, residual=res, gate=gate, rows_per_group=1)
        _close(out, ref.linear(x, w, bias, act, res, gate, 1, out_dtype=torch.float32), f"{act} {M}x{N}x{K}", rel=1e-4)
    x2, w2 = _rand(M, 24, seed=3), _rand(N, 24, scale=0.1, seed=4)
    _close(O.linear(x, w, extra=[(x2, w2)]), x.float() @ w.float().t() + x2.float() @ w2.float().t(), f"two segments {M}x{N}x{K}")
    if N % 16 == 0:
        _close(O.linear_glu(x, w, bias, "silu"), ref.linear_glu(x.float(), w.float(), bias.float(), "silu"), f"paired {M}x{N}x{K}", rel=1e-4)


# fp8 on the CTA-pair kernel (M > 128 rows and enough tiles), with both scales in its epilogue; ragged in M, N and K
@pytest.mark.parametrize("M,N,K", [(129, 256, 128), (300, 4096, 400), (2737, 1032, 4096)])
def test_fp8_pair_gemm(M, N, K):
    x, w = _rand(M, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2)
    wq, ws = O.fp8_quant_rows(w)
    xq, xs = O.fp8_quant_rows(x)
    bias, res = _rand(N, seed=7), _rand(M, N, seed=9)
    want = (xq.float() @ wq.float().t()) * xs[:, None] * ws[None] + bias.float()
    _close(O.fp8_linear(x, wq, ws, bias), want, f"fp8 {M}x{N}x{K}", rel=1e-4)
    _close(O.fp8_linear(x, wq, ws, bias, residual=res), want + res.float(), f"fp8 residual {M}x{N}x{K}", rel=1e-4)


def _conv_ref(x, w, bias, stride=1, offset=0):
    y = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).float(), w.permute(0, 3, 1, 2).float(), bias.float(), padding=1).permute(0, 2, 3, 1)
    return y[:, offset::stride, offset::stride]


def test_conv3x3_many_tiles_per_cluster():
    from mojodiffusion_b200.ops import conv as C
    for Cin, Cout in ((64, 128), (128, 128), (192, 96), (128, 256)):   # several tiles per persistent cluster: every ring wraps
        x, w = _rand(1, 200, 333, Cin, seed=1), _rand(Cout, 3, 3, Cin, scale=1 / math.sqrt(9 * Cin), seed=2)
        with torch.no_grad():
            _close(C.conv2d_nhwc(x, w, _rand(Cout, seed=3)), _conv_ref(x, w, _rand(Cout, seed=3)), f"{Cin} -> {Cout}")


# one patch (its partner of the pair lies past the batch), images smaller than a patch, ragged edges both ways, an odd number of
# patches; output channels below, at and beyond one 256-wide tile
@pytest.mark.parametrize("N,H,W", [(1, 8, 16), (1, 5, 3), (2, 17, 33), (1, 9, 47), (3, 31, 50)])
@pytest.mark.parametrize("Cin,Cout", [(64, 8), (128, 64), (64, 128), (192, 320), (128, 512), (64, 648)])
def test_conv3x3_pair_tiles(N, H, W, Cin, Cout):
    from mojodiffusion_b200.ops import conv as C
    x, w = _rand(N, H, W, Cin, seed=1), _rand(Cout, 3, 3, Cin, scale=1 / math.sqrt(9 * Cin), seed=2)
    bias, res = _rand(Cout, seed=3), _rand(N, H, W, Cout, seed=4)
    with torch.no_grad():
        _close(C.conv2d_nhwc(x, w, bias), _conv_ref(x, w, bias), "plain")
        _close(C.conv2d_nhwc(x, w, bias, act="silu", residual=res), torch.nn.functional.silu(_conv_ref(x, w, bias)) + res.float(), "act + residual", rel=1e-4)
        for off in (0, 1):
            _close(C.conv2d_nhwc(x, w, bias, stride=2, offset=off), _conv_ref(x, w, bias, 2, off), f"stride 2 from {off}")
        w1 = _rand(Cout, 1, 1, Cin, scale=1 / math.sqrt(Cin), seed=5)
        _close(C.conv2d_nhwc(x, w1, bias, padding=0), x.float() @ w1[:, 0, 0].float().t() + bias.float(), "1 x 1")


# decoder layer kernels against the same stack in fp32 on the CPU: rows of one, eight and nine sequences (few-row / tiled
# projections), head widths with one and with several rotary pairs per lane, with and without biases
@pytest.mark.parametrize("B,S,H,Hkv,Dh,bias", [(1, 1, 4, 2, 64, False), (2, 11, 4, 1, 128, False), (8, 3, 6, 6, 40, True), (9, 65, 2, 2, 256, False)])
def test_decoder_layers(B, S, H, Hkv, Dh, bias):
    from mojodiffusion_b200.llm.decoder import Qwen3Decoder
    from mojodiffusion_b200.models.text.qwen3 import Qwen3Config, Qwen3Encoder
    cfg = Qwen3Config(vocab_size=200, hidden_size=264, intermediate_size=520, num_hidden_layers=3, num_attention_heads=H, num_key_value_heads=Hkv,
                      head_dim=Dh, qkv_bias=bias)
    enc = Qwen3Encoder(cfg, torch.bfloat16, DEV).eval()
    g = torch.Generator(device=DEV).manual_seed(0)
    with torch.no_grad():
        for n, p in enc.named_parameters():
            p.normal_(0.0, p.shape[-1] ** -0.5, generator=g) if p.dim() == 2 else p.normal_(0.0 if n.endswith("bias") else 1.0, 0.1, generator=g)
    cpu = Qwen3Encoder(cfg, torch.float32).eval()
    cpu.load_state_dict({k: v.float().cpu() for k, v in enc.state_dict().items()})
    ids = torch.randint(0, 200, (B, S), generator=torch.Generator().manual_seed(1))
    nxt = torch.randint(0, 200, (4, B), generator=torch.Generator().manual_seed(2))
    outs = []
    for dec, dev in ((Qwen3Decoder(enc), DEV), (Qwen3Decoder(cpu), "cpu")):
        h, cache = dec.prefill(ids.to(dev), S + 4)
        out = [dec.logits(h)]
        for t in nxt:
            out.append(dec.logits(dec.decode_step(t.to(dev), cache)))
        outs.append(torch.stack(out).float().cpu())
    native.check_status(torch.empty(0, device=DEV))
    # about twenty bf16 roundings of 2^-9 / sqrt(3) each per layer, added in quadrature over three layers and the head, doubled
    err = float((outs[0] - outs[1]).norm() / outs[1].norm())
    assert err < 2 * 2.0 ** -9 / 3 ** 0.5 * 64 ** 0.5, err


def test_few_row_gemm_accumulates_fp32():
    from mojodiffusion_b200.ops.functional import _gemm
    for M in (1, 3, 8, 40):
        x, w, out = _rand(M, 264, seed=1), _rand(120, 264, seed=2, scale=0.1), _rand(M, 120, seed=3, dtype=torch.float32)
        want = out + x.float() @ w.float().t()
        _gemm([x], [w], out=out, out_fp32=True, accumulate=True)
        native.check_status(out)
        assert float((out - want).abs().max()) < 2e-5 * float(want.abs().max()), M


# groups of 3 / 4 / 10 / 80 channels, slabs of whole groups beyond 2048 channels, one pixel, images that end inside a chunk
@pytest.mark.parametrize("N,HW,C,G", [(1, 1, 64, 2), (2, 1000, 24, 8), (3, 4097, 128, 32), (2, 777, 320, 32), (2, 300, 2560, 32), (1, 50, 4096, 32),
                                      (1, 300000, 8, 2)])
def test_group_norm_forward_and_backward(N, HW, C, G):
    from mojodiffusion_b200.ops import conv as K
    x = _rand(N, 1, HW, C, seed=1) * 2 + 3                      # a mean of several standard deviations
    w, b, dy = _rand(C, seed=2), _rand(C, seed=3), _rand(N, 1, HW, C, seed=4)
    for act in (None, "silu"):
        with torch.no_grad():
            y = K.group_norm_nhwc(x, w, b, G, 1e-6, act)
        leaf = [t.float().requires_grad_() for t in (x, w, b)]
        want = torch.nn.functional.group_norm(leaf[0].permute(0, 3, 1, 2).double(), G, leaf[1].double(), leaf[2].double(), 1e-6).permute(0, 2, 3, 1)
        want = torch.nn.functional.silu(want) if act else want
        _close(y, want, f"forward {act}", rel=1e-5)
        want.backward(dy.double())
        p = [t.clone().requires_grad_() for t in (x, w, b)]
        K.group_norm_nhwc(*p, G, 1e-6, act).backward(dy)
        _close(p[0].grad, leaf[0].grad, f"dx {act}", rel=1e-4)
        for i in (1, 2):                                        # fp32 sums over the pixels, then bf16: 2^-9 and the sum's own 1e-4
            err = float((p[i].grad.float() - leaf[i].grad).norm() / leaf[i].grad.norm())
            assert err < 2.0 ** -8 + 1e-3, (act, i, err)


# one wide head: odd key counts (padded score rows), fewer rows than a tile, several chunks of rows when the scores pass the
# bound, a width that is no multiple of 16
@pytest.mark.parametrize("B,Sq,Skv,Dh", [(1, 5, 3, 512), (3, 333, 333, 512), (2, 300, 1001, 136), (1, 9000, 17001, 256)])
def test_wide_single_head_attention(B, Sq, Skv, Dh):
    q, k, v = (_rand(B, s, 1, Dh, seed=i) for i, s in ((1, Sq), (2, Skv), (3, Skv)))
    with torch.no_grad():
        out = O.attention(q, k, v)
        pad = torch.empty(B, Sq, 2 * Dh, dtype=torch.bfloat16, device=DEV)
        pad[..., :Dh] = q[:, :, 0]
        strided = O.attention(pad[..., :Dh].unflatten(-1, (1, Dh)), k, v)
    native.check_status(out)
    want = torch.cat([torch.softmax(q[b, :, 0].float() @ k[b, :, 0].float().t() / math.sqrt(Dh), -1) @ v[b, :, 0].float() for b in range(B)]).view(B, Sq, 1, Dh)
    # probabilities and the result are rounded to bf16 once each: 2^-9 / sqrt(3) of their size, in quadrature, doubled
    assert float((out.float() - want).norm() / want.norm()) < 2 * 2.0 ** -9 * (2 / 3) ** 0.5
    assert torch.equal(out, strided)


@pytest.mark.parametrize("cols", [1, 3, 4, 1000, 16384, 16385, 40001])
def test_softmax_rows(cols):
    ld = (cols + 7) // 8 * 8
    s = torch.full((7, ld), float("nan"), device=DEV)            # what the padding holds does not matter
    s[:, :cols] = _rand(7, cols, scale=4, dtype=torch.float32)
    s[1, :cols // 2] = float("-inf")
    s[2, :cols] = 1e30
    s[3, cols - 1] = float("nan")
    p = torch.empty(7, ld, dtype=torch.bfloat16, device=DEV)
    torch.ops.mdb200.softmax_rows(s[:, :cols], p[:, :cols], 0.7)
    want = torch.softmax(s[:, :cols].double() * 0.7, -1)
    assert torch.isnan(p[3, :cols]).all()
    keep = [0, 1, 2, 4, 5, 6]
    # bf16 rounding (2^-9) and the exponential's and sum's 1e-5, doubled
    assert bool(((p[keep][:, :cols].double() - want[keep]).abs() <= want[keep] * 2 * (2.0 ** -9 + 1e-5) + 1e-38).all())


# one-pass q / k norm + rotation and the head gates against the fp32 module on the CPU: one and several heads per thread block
# step, two samples (rotary rows repeat), a token count off every tile
@pytest.mark.parametrize("hidden,heads,head_dim", [(256, 4, 64), (384, 3, 128), (4352, 34, 128)])
def test_video_attention_rows(hidden, heads, head_dim):
    from mojodiffusion_b200.models.video_dit import VideoAttention, VideoDiTConfig
    axes = (head_dim // 2, head_dim // 4, head_dim // 4)
    cfg = VideoDiTConfig(hidden=hidden, heads=heads, head_dim=head_dim, axes_dim=axes)
    att = VideoAttention(cfg, False, torch.bfloat16, DEV)
    with torch.no_grad():
        for i, (n, p) in enumerate(att.named_parameters()):
            p.copy_(_rand(*p.shape, seed=i, scale=p.shape[-1] ** -0.5) if p.dim() == 2 else _rand(*p.shape, seed=i, scale=0.1) + (1.0 if "norm" in n else 0.0))
        ids = torch.stack(torch.meshgrid(torch.arange(3.), torch.arange(5.), torch.arange(7.), indexing="ij"), -1).reshape(-1, 3)
        cos, sin = O.rope_table(ids.to(DEV), axes, 10000.0)
        x = _rand(2, 105, hidden, seed=50)
        out = att(x, None, cos, sin)
        native.check_status(out)
        cpu = VideoAttention(cfg, False, torch.float32, None)
        cpu.load_state_dict({k: v.float().cpu() for k, v in att.state_dict().items()})
        want = cpu(x.float().cpu(), None, cos.cpu(), sin.cpu())
    # projections, q / k, probabilities, attention and gated output are rounded to bf16 once each: five in quadrature, doubled
    assert float((out.float().cpu() - want).norm() / want.norm()) < 2 * 2.0 ** -9 * (5 / 3) ** 0.5


def test_fp8_projections_share_quantised_rows():
    from mojodiffusion_b200.models.layers import Linear, packed_projection
    from mojodiffusion_b200.models.video_dit import FP8Linear
    lins = [FP8Linear(Linear(384, n, True, torch.bfloat16, DEV)) for n in (256, 64, 128)]
    for shape in ((2, 150, 384), (5, 384)):
        x = _rand(*shape, seed=1)
        with torch.no_grad():
            got = packed_projection(x, lins)
            want = torch.cat([l(x) for l in lins], -1)
        native.check_status(got)
        assert torch.equal(got, want)


# few tiles against a long reduction: the launch shares each tile's K range over a cluster. Rows and columns off the tile, K off
# the 64-wide step, a second segment that starts inside a share, N below one 8-column group of the finish
@pytest.mark.parametrize("M,N,K", [(9, 64, 4096), (45, 2560, 9728), (256, 3072, 12288), (200, 40, 3080), (512, 1000, 2056), (130, 20, 8200), (512, 3072, 15360),
                                   (300, 3000, 6200)])
def test_cluster_split_k(M, N, K):
    from mojodiffusion_b200.ops.functional import _gemm
    N8 = (N + 7) // 8 * 8
    x, w = _rand(M, K, seed=1), _rand(N8, K, scale=1 / math.sqrt(K), seed=2)
    bias, gate, res = _rand(N, seed=7), _rand(2, N8, seed=8)[:, :N], _rand(M, N8, seed=9)[:, :N]
    want = x.float() @ w[:N].float().t()
    _close(_gemm([x], [w[:N]]), want, "plain")
    _close(_gemm([x], [w[:N]], out_fp32=True), want, "fp32 out")
    x2, w2 = _rand(M, 16, seed=3), _rand(N, 16, scale=0.1, seed=4)
    full = ref.linear(x, w[:N], bias, "gelu_tanh", res, gate, (M + 1) // 2, [(x2, w2)], out_dtype=torch.float32)
    _close(_gemm([x, x2], [w[:N], w2], bias=bias, residual=res, gate=gate, rows_per_group=(M + 1) // 2, act=1), full, "epilogue", rel=1e-4)
    _close(_gemm([x], [w.t().contiguous()], b_mn=True), x.float() @ w.float().t(), "B read transposed")
    M8 = (M + 7) // 8 * 8
    xt = _rand(K, M8, seed=5)
    _close(_gemm([xt], [w.t().contiguous()], a_mn=True, b_mn=True, alpha=0.5), 0.5 * xt.float().t() @ w.float().t(), "both read transposed", rel=1e-4)


# every combination of epilogue terms on whole and ragged tiles of the lone and the pair kernel (N = 1160 leaves 8 columns of a
# 128-wide group, M = 300 rows beyond a tile; bn 512 is the pair kernel)
@pytest.mark.parametrize("bn", [128, 256, 512])
@pytest.mark.parametrize("N", [1152, 1160])
def test_epilogue_terms(bn, N):
    from mojodiffusion_b200.ops.functional import _gemm
    from mojodiffusion_b200.ops.reference import act_code
    M, K = 300, 200
    x, w = _rand(M, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2)
    bias, gate, res = _rand(N, seed=7), _rand(2, N, seed=8), _rand(M, N, seed=9)
    for act in (None, "silu", "gelu_tanh", "gelu"):
        for b in (None, bias):
            for g, r in ((None, None), (None, res), (gate, res), (gate, None)):
                out = _gemm([x], [w], bias=b, residual=r, gate=g, rows_per_group=150, act=act_code(act), bn=bn)
                want = ref.linear(x, w, b, act, r, g, 150, out_dtype=torch.float32) if g is None or r is not None else \
                    ref.linear(x, w, b, act, out_dtype=torch.float32) * gate.float().repeat_interleave(150, 0)
                _close(out, want, f"{bn} {N} {act} bias {b is not None} gate {g is not None} residual {r is not None}", rel=1e-4)
    for act in ("silu", "gelu_tanh", "gelu"):
        for second in (0, 1):
            out = _gemm([x], [w], bias=bias, act=act_code(act), pair_offset=N // 2, act_on_second=second, bn=bn)
            _close(out, ref.linear_glu(x.float(), w.float(), bias.float(), act, bool(second)), f"paired {bn} {N} {act} {second}", rel=1e-4)


# rows on the block kernel (2048 .. 16384) give the bytes and scales of the one-warp kernel, which takes the same rows padded with
# zeros beyond 16384; a zero row, a row with an infinity, strided rows
@pytest.mark.parametrize("D", [2048, 2056, 4096, 5000, 16384])
def test_fp8_quant_rows_block(D):
    x = _rand(37, D, seed=1)
    x[3] = 0
    x[4, D - 1] = float("inf")
    x[5] *= 1e-30
    pad = torch.zeros(37, 16392, dtype=torch.bfloat16, device=DEV)
    pad[:, :D] = x
    wq, ws = torch.ops.mdb200.fp8_quant_rows(pad)
    for src in (x, pad[:, :D]):
        q, s = torch.ops.mdb200.fp8_quant_rows(src)
        assert torch.equal(s, ws) and torch.equal(q.view(torch.uint8), wq[:, :D].contiguous().view(torch.uint8))


# a row of linear(whole_k=True) has the same bits whatever rows come with it: few rows, rows that the launch would share over a
# cluster, and whole tiles; a K and an N that are padded to the 16-byte rule; the autograd route and its input gradient
@pytest.mark.parametrize("N,K", [(2560, 9728), (512, 8192), (64, 4096), (60, 4100)])
def test_whole_k_rows_do_not_depend_on_their_number(N, K):
    x, w, bias, dy = _rand(300, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2), _rand(N, seed=3), _rand(300, N, seed=4)
    full, full_dx = O.linear(x, w, bias, whole_k=True), None
    _close(full, x.float() @ w.float().t() + bias.float(), f"{N}x{K}", rel=1e-4)
    for m in (300, 1, 7, 8, 9, 45, 129, 256):
        assert torch.equal(O.linear(x[:m], w, bias, whole_k=True), full[:m]), m
        leaf = x[:m].clone().requires_grad_()
        y = O.linear(leaf, w, bias, whole_k=True)
        assert torch.equal(y, full[:m]), m
        y.backward(dy[:m])
        full_dx = leaf.grad if full_dx is None else full_dx
        assert torch.equal(leaf.grad, full_dx[:m]), m
    native.check_status(full)


# projections of the text encoders at long reductions: a token's row does not depend on the length of the prompt
def test_text_encoder_projections_do_not_depend_on_prompt_length():
    from mojodiffusion_b200.models.text import clip, gpt_oss, qwen3, t5
    for lin in (clip._Lin(5120, 1280, torch.bfloat16, DEV), t5._W(10240, 4096, torch.bfloat16, DEV), gpt_oss._Lin(4096, 2880, torch.bfloat16, DEV),
                qwen3._W(9728, 2560, torch.bfloat16, DEV, True)):
        x = _rand(1, 300, lin.weight.shape[1], seed=1)
        with torch.no_grad():
            full = lin(x)
            for n in (1, 8, 9, 45, 129):
                assert torch.equal(lin(x[:, :n]), full[:, :n]), (type(lin).__module__, n)


# what a program does to the q / k norms of a video attention takes effect: a hook on either side, an epsilon of one of them, another
# module in its place (its hook-free twin on the fp32 CPU path is the oracle)
@pytest.mark.parametrize("change", ["pre-hook", "hook", "global hook", "eps", "module", "forward"])
def test_video_attention_keeps_to_its_norm_modules(change):
    from mojodiffusion_b200.models.video_dit import VideoAttention, VideoDiTConfig
    cfg = VideoDiTConfig(hidden=256, heads=4, head_dim=64, axes_dim=(32, 16, 16))
    ids = torch.stack(torch.meshgrid(torch.arange(3.), torch.arange(5.), torch.arange(7.), indexing="ij"), -1).reshape(-1, 3)
    cos, sin = O.rope_table(ids.to(DEV), cfg.axes_dim, 10000.0)
    x, handles = _rand(2, 105, 256, seed=50), []
    att = VideoAttention(cfg, False, torch.bfloat16, DEV)
    cpu = VideoAttention(cfg, False, torch.float32, None)
    with torch.no_grad():
        for i, (n, p) in enumerate(att.named_parameters()):
            p.copy_(_rand(*p.shape, seed=i, scale=p.shape[-1] ** -0.5) if p.dim() == 2 else _rand(*p.shape, seed=i, scale=0.1) + (1.0 if "norm" in n else 0.0))
        cpu.load_state_dict({k: v.float().cpu() for k, v in att.state_dict().items()})
        plain = att(x, None, cos, sin)
        for m in (att, cpu):
            if change == "pre-hook":
                m.q_norm.register_forward_pre_hook(lambda mod, args: (args[0].roll(1, -1),))
            elif change == "hook":
                m.k_norm.register_forward_hook(lambda mod, args, out: out.roll(1, -1))
            elif change == "global hook":
                norms = (m.q_norm, m.k_norm)
                handles.append(torch.nn.modules.module.register_module_forward_hook(lambda mod, args, out, norms=norms: out.roll(1, -1) if mod is norms[1] else None))
            elif change == "eps":
                m.k_norm.eps = 1.0
            elif change == "module":
                m.k_norm = torch.nn.Identity()
            else:
                m.q_norm.forward = lambda t: t * 0.5
        try:
            with torch.no_grad():
                out, want = att(x, None, cos, sin), cpu(x.float().cpu(), None, cos.cpu(), sin.cpu())
        finally:
            for h in handles:
                h.remove()
    native.check_status(out)
    # as above, and one rounding more where the norm stands apart from the rotation
    bound = 2 * 2.0 ** -9 * (6 / 3) ** 0.5
    assert float((out.float().cpu() - want).norm() / want.norm()) < bound
    assert float((plain.float().cpu() - want).norm() / want.norm()) > 4 * bound         # the change does show


# fp8 projections that a program has changed get their own input, not the shared quantised rows
@pytest.mark.parametrize("change", ["pre-hook", "subclass", "forward"])
def test_changed_fp8_projections_quantise_their_own_rows(change):
    from mojodiffusion_b200.models.layers import Linear, packed_projection
    from mojodiffusion_b200.models.video_dit import FP8Linear

    class Halved(FP8Linear):
        def forward(self, x, act=None, residual=None, gate=None, rows_per_group=1, out=None):
            return super().forward(x * 0.5, act, residual, gate, rows_per_group, out)

    lins = [(Halved if change == "subclass" and i == 1 else FP8Linear)(Linear(384, n, True, torch.bfloat16, DEV)) for i, n in enumerate((256, 64, 128))]
    if change == "pre-hook":
        lins[1].register_forward_pre_hook(lambda mod, args: (args[0] * 0.5,))
    elif change == "forward":
        plain = lins[1].forward
        lins[1].forward = lambda x, out=None: plain(x * 0.5, out=out)
    x = _rand(2, 150, 384, seed=1)
    with torch.no_grad():
        got = packed_projection(x, lins)
        want = torch.cat([O.fp8_linear(x * 0.5 if i == 1 else x, l.weight, l.weight_scale, l.bias) for i, l in enumerate(lins)], -1)
    native.check_status(got)
    assert torch.equal(got, want)


# a block of columns inside a wider buffer: the columns beside it keep what they held
@pytest.mark.parametrize("cols", [1, 2, 3, 5, 1001, 16385, 16391])
def test_softmax_rows_writes_its_columns_only(cols):
    ld = (cols + 7) // 8 * 8 + 8
    s, p = _rand(5, ld, seed=1, dtype=torch.float32), _rand(5, ld, seed=2)
    beside = p[:, cols:].clone()
    torch.ops.mdb200.softmax_rows(s[:, :cols], p[:, :cols], 1.0)
    assert torch.equal(p[:, cols:], beside)
    want = torch.softmax(s[:, :cols].double(), -1)
    assert bool(((p[:, :cols].double() - want).abs() <= want * 2 * (2.0 ** -9 + 1e-5)).all())


# a constant group is normalised to zero, so only the bias is left whatever the weight; 1 / sqrt(eps) times the weight overflows
def test_group_norm_large_weight_on_a_constant_group():
    from mojodiffusion_b200.ops import conv as K
    x, w, b = torch.full((1, 4, 4, 64), 3.0, dtype=torch.bfloat16, device=DEV), torch.full((64,), 3e38, dtype=torch.bfloat16, device=DEV), _rand(64, seed=1)
    with torch.no_grad():
        assert torch.equal(K.group_norm_nhwc(x, w, b, 8, 1e-6), b.expand(1, 4, 4, 64))


def test_head_gate_rounds_as_the_torch_statement():
    o, logit = _rand(2000, 32, 128, seed=1), _rand(2000, 32, seed=2, scale=20.0)
    want = (o.float() * (2.0 * torch.sigmoid(logit.float()))[..., None]).to(torch.bfloat16)
    torch.ops.mdb200.head_gate(o, logit)
    assert torch.equal(o, want)


# identity weights make the gated MLP of a decoder step silu(h) * h of its normalised input, and rows of +-1 normalise to +-1 exactly:
# the result is known to the bit, here for every bf16 value from 2^-7 to 87
def test_decoder_mlp_rounds_a_precise_silu():
    bits = torch.arange(0x3c00, 0x42b0, dtype=torch.int32).to(torch.int16)
    ln = bits.view(torch.bfloat16).to(DEV)
    D = ln.numel()
    eye = torch.eye(D, dtype=torch.bfloat16, device=DEV)
    x = torch.ones(2, D, dtype=torch.bfloat16, device=DEV)
    x[1] = -1
    h = x * ln
    out = torch.ops.mdb200.llm_out_mlp(x, torch.zeros(2, D, dtype=torch.bfloat16, device=DEV), eye, ln, eye, eye, eye, 1e-6)
    native.check_status(out)
    assert torch.equal(out, torch.nn.functional.silu(h.double()).float().to(torch.bfloat16) * h)


# one-hot keys and values: the outputs are the probabilities. Errors beyond the bf16 rounding (2^-8) are those of the fp32
# exponential, sum and quotient, a few 2^-24
def test_decode_attention_probabilities():
    B, H, Dh, T = 8, 32, 128, 128
    q = torch.zeros(B, H * Dh, dtype=torch.bfloat16, device=DEV)
    q.copy_(-torch.rand(B, H * Dh, generator=torch.Generator().manual_seed(1)) * 60)
    eye = torch.eye(T, Dh, dtype=torch.bfloat16, device=DEV).expand(B, H, T, Dh).contiguous()
    out = torch.ops.mdb200.llm_decode_attention(q, eye, eye, H, T, 1.0).view(B, H, T).double()
    want = torch.softmax(q.view(B, H, Dh).double(), -1)
    worst = float(((out - want).abs() / want - 2.0 ** -8).max())
    assert worst < 16 * 2.0 ** -24, worst


# one wide head in the forms that only the torch operations have: batch or value width that differ, vmap, forward-mode AD, a
# dispatch mode; the plain call is the oracle of each
@pytest.mark.parametrize("form", ["one key batch", "value width", "many key heads", "vmap", "forward AD", "dispatch mode"])
def test_wide_single_head_attention_other_forms(form):
    from torch.autograd import forward_ad
    from torch.utils._python_dispatch import TorchDispatchMode
    B, Sq, Skv, Dh = 3, 33, 2000, 512
    q, k, v = (_rand(B, s, 1, Dh, seed=i) for i, s in ((1, Sq), (2, Skv), (3, Skv)))
    assert O.functional._wide_ok(q, k, v)                       # the plain call is on the GEMMs
    with torch.no_grad():
        plain = O.attention(q, k, v)
        if form == "one key batch":
            got, want = O.attention(q, k[:1], v[:1]), O.attention(q, k[:1].repeat(B, 1, 1, 1), v[:1].repeat(B, 1, 1, 1))
        elif form == "value width":
            got, want = O.attention(q, k, v[..., :256]), plain[..., :256]
        elif form == "many key heads":
            got = O.attention(q, torch.cat((k, k), 2), torch.cat((v, v), 2))
            want = torch.cat((plain, plain), 2)
        elif form == "vmap":
            got, want = torch.func.vmap(O.attention)(q[:, None], k[:, None], v[:, None])[:, 0], plain
        elif form == "forward AD":
            # the library kernel has none: it says so and does not drop the tangent
            with forward_ad.dual_level(), pytest.raises(NotImplementedError):
                O.attention(q, k, forward_ad.make_dual(v, _rand(B, Skv, 1, Dh, seed=9)))
            got = want = plain
        else:
            seen = []

            class Log(TorchDispatchMode):
                def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                    seen.append(str(func))
                    return func(*args, **(kwargs or {}))
            with Log():
                got = O.attention(q, k, v)
            want = plain
            assert any("attention" in s or "softmax" in s for s in seen), seen
    assert got.shape == want.shape and float((got.float() - want.float()).norm() / want.float().norm()) < 2.0 ** -7


# what a program does to the modules, weights or cache of a decoder takes effect in the decode step and nothing that the separate
# operations take is refused: the same change on the fp32 CPU stack is the oracle
@pytest.mark.parametrize("change", ["none", "norm hook", "projection hook", "global pre-hook", "epsilon", "bias", "plain bias", "module", "forward", "weight offset",
                                    "beams", "strided cache", "no tables", "token column", "table offset", "vmap logits"])
def test_decode_step_keeps_to_its_modules(change):
    from mojodiffusion_b200.llm.decoder import Qwen3Decoder
    from mojodiffusion_b200.models.text.qwen3 import Qwen3Config, Qwen3Encoder
    cfg = Qwen3Config(vocab_size=200, hidden_size=264, intermediate_size=520, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64)
    enc, cpu = Qwen3Encoder(cfg, torch.bfloat16, DEV).eval(), Qwen3Encoder(cfg, torch.float32).eval()
    g = torch.Generator(device=DEV).manual_seed(0)
    with torch.no_grad():
        for n, p in enc.named_parameters():
            p.normal_(0.0, p.shape[-1] ** -0.5, generator=g) if p.dim() == 2 else p.normal_(1.0, 0.1, generator=g)
    cpu.load_state_dict({k: v.float().cpu() for k, v in enc.state_dict().items()})
    B = 1 if change == "token column" else 3
    ids, tok = torch.randint(0, 200, (B, 7), generator=torch.Generator().manual_seed(1)), torch.randint(0, 200, (B,), generator=torch.Generator().manual_seed(2))
    handles, outs = [], []
    for e, dev in ((enc, DEV), (cpu, "cpu")):
        dec, l = Qwen3Decoder(e), e.model.layers[1]
        hidden, cache = dec.prefill(ids.to(dev), 12)
        t = tok.to(dev)
        if change == "norm hook":
            l.input_layernorm.register_forward_hook(lambda mod, args, out: out * 2)
        elif change == "projection hook":
            l.mlp.down_proj.register_forward_pre_hook(lambda mod, args: (args[0] * 2,))
        elif change == "global pre-hook":
            k_norm = l.self_attn.k_norm
            handles.append(torch.nn.modules.module.register_module_forward_pre_hook(lambda mod, args, k_norm=k_norm: (args[0].roll(1, -1),) if mod is k_norm else None))
        elif change == "epsilon":
            l.self_attn.q_norm.eps = 4.0
        elif change == "bias":
            l.self_attn.o_proj.bias = torch.nn.Parameter(_rand(264, seed=5).to(dev, l.self_attn.o_proj.weight.dtype))
        elif change == "plain bias":
            l.mlp.up_proj.bias = _rand(520, seed=5).to(dev, l.mlp.up_proj.weight.dtype)
        elif change == "module":
            l.mlp = torch.nn.Identity()
        elif change == "forward":
            l.mlp.forward = lambda h: h * 0.5
        elif change == "weight offset":
            w = e.model.norm.weight.data
            for n in (l.self_attn.k_norm, l.input_layernorm):
                buf = torch.empty(n.weight.numel() + 1, dtype=w.dtype, device=dev)
                buf[1:] = n.weight.data * 2
                n.weight.data = buf[1:]
        elif change == "beams":
            cache.k, cache.v = cache.k[:, :1].expand(-1, B, -1, -1, -1).clone(), cache.v[:, :1].expand(-1, B, -1, -1, -1).clone()
        elif change == "strided cache":
            cache.k, cache.v = (c.transpose(2, 3).contiguous().transpose(2, 3) for c in (cache.k, cache.v))
        elif change == "no tables":
            del cache.rope
        elif change == "token column":
            t = t[:, None]
        elif change == "table offset":
            table = torch.empty(200 * 264 + 4, dtype=e.model.embed_tokens.weight.dtype, device=dev)
            table[4:] = e.model.embed_tokens.weight.data.flatten()
            dec.lm_head = table[4:].view(200, 264)
        try:
            h = dec.decode_step(t, cache)
            h = dec.decode_step(t, cache) if change != "token column" else h[:, 0]
            if change == "vmap logits":
                outs.append(torch.func.vmap(lambda r: dec.logits(r[None])[0])(h).float().cpu())
            else:
                outs.append(dec.logits(h).float().cpu())
        finally:
            while handles:
                handles.pop().remove()
    native.check_status(torch.empty(0, device=DEV))
    # as for the layers above, with two layers
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 2 * 2.0 ** -9 / 3 ** 0.5 * 44 ** 0.5


# the GEMM form of one wide head rounds its result only: 2^-9 / sqrt(3) of its size, doubled for the spread of that estimate (one bf16 term per
# probability adds as much again). Odd key counts, one key, several chunks of rows, a width off 16
@pytest.mark.parametrize("B,Sq,Skv,Dh", [(1, 5, 3, 512), (2, 7, 1, 512), (3, 333, 333, 512), (2, 300, 1001, 136), (1, 5000, 17001, 256)])
def test_wide_attention_on_gemms_rounds_once(B, Sq, Skv, Dh):
    q, k, v = (_rand(B, s, 1, Dh, seed=i) for i, s in ((1, Sq), (2, Skv), (3, Skv)))
    out = O.functional._wide_attention(q, k, v, 1 / math.sqrt(Dh))
    native.check_status(out)
    want = torch.cat([torch.softmax(q[b, :, 0].double() @ k[b, :, 0].double().t() / math.sqrt(Dh), -1) @ v[b, :, 0].double() for b in range(B)]).view(B, Sq, 1, Dh)
    assert float((out.double() - want).norm() / want.norm()) < 2 * 2.0 ** -9 / 3 ** 0.5


def test_epilogue_terms_of_narrow_tiles():
    for N in (640, 1160):
        test_epilogue_terms(64, N)


# rows of 64, 128 and 256 items: the widths at which the one-pass q / k kernel changes its block
@pytest.mark.parametrize("hidden,heads,head_dim", [(512, 8, 64), (528, 33, 16), (1024, 16, 64), (2048, 16, 128), (4096, 32, 128)])
def test_video_attention_row_blocks(hidden, heads, head_dim):
    test_video_attention_rows(hidden, heads, head_dim)


# sizes drawn over the range that the launch chooses its form for, in the three operand layouts, against the fp32 product
@pytest.mark.parametrize("seed", range(8))
def test_gemm_forms_left_to_the_launch(seed):
    import random
    from mojodiffusion_b200.ops.functional import _gemm
    r = random.Random(seed)
    for _ in range(12):
        M, N, K = (int(round(math.exp(r.uniform(math.log(lo), math.log(hi))))) for lo, hi in ((1, 5000), (8, 6000), (8, 6000)))
        N8, K8, M8 = ((t + 7) // 8 * 8 for t in (N, K, M))
        x, w, bias, res = _rand(M, K8, seed=1)[:, :K], _rand(N, K8, scale=1 / math.sqrt(K), seed=2)[:, :K], _rand(N, seed=3), _rand(M, N, seed=4)
        want = x.float() @ w.float().t()
        _close(_gemm([x], [w]), want, f"NT {M}x{N}x{K}")
        _close(_gemm([x], [w], bias=bias, residual=res, act=2), ref.linear(x, w, bias, "silu", res, None, 1, out_dtype=torch.float32), f"terms {M}x{N}x{K}", rel=1e-4)
        wt, xt = torch.zeros(K, N8, dtype=torch.bfloat16, device=DEV), torch.zeros(K, M8, dtype=torch.bfloat16, device=DEV)
        wt[:, :N], xt[:, :M] = w.t(), x.t()
        _close(_gemm([x], [wt[:, :N]], b_mn=True), want, f"NN {M}x{N}x{K}")
        _close(_gemm([xt[:, :M]], [wt[:, :N]], a_mn=True, b_mn=True), want, f"TN {M}x{N}x{K}")


# beyond 2048 channels: pixels on either side of the lines between one block per group and chunks of pixels (forward 512, backward 160)
@pytest.mark.parametrize("N,HW", [(1, 8), (2, 159), (1, 160), (1, 511), (2, 512)])
def test_group_norm_wide_tensors_of_few_pixels(N, HW):
    test_group_norm_forward_and_backward(N, HW, 2560, 32)


# rows that leave through a tensor map: many short tiles per CTA (the staging buffers take turns), rows and columns that end inside a
# store's 32 x 64 box, two gates in one warp's rows, an output between other columns and one in the place of the residual
# (the two shapes without a width are left to the launch, which takes clusters for them: their rows leave the other way)
@pytest.mark.parametrize("M,N,K,bn", [(30000, 64, 64, 64), (30000, 192, 64, 256), (20000, 320, 64, 512), (20000, 72, 128, 128), (300, 200, 320, 128), (129, 24, 72, 64), (300, 200, 320, 0), (129, 24, 72, 0)])
@pytest.mark.parametrize("terms", ["bias", "gelu", "gate", "slice"])
def test_bulk_epilogue(M, N, K, bn, terms):
    from mojodiffusion_b200.ops.functional import _gemm
    x, w, b = _rand(M, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2), _rand(N, seed=3)
    want = x.float() @ w.float().t() + b.float()
    if terms == "bias":
        got = _gemm([x], [w], bias=b, bn=bn)
    elif terms == "gelu":
        want, got = torch.nn.functional.gelu(want, approximate="tanh"), _gemm([x], [w], bias=b, act=1, bn=bn)
    elif terms == "gate":
        gate, out, rows = _rand(3, N, seed=4), _rand(M, N, seed=5), (M + 2) // 3
        want = out.float() + want * gate.float().repeat_interleave(rows, 0)[:M]
        got = _gemm([x], [w], bias=b, residual=out, gate=gate, rows_per_group=rows, out=out, bn=bn)
    else:
        wide = torch.zeros(M, 3 * N, device=DEV, dtype=torch.bfloat16)
        got = _gemm([x], [w], bias=b, out=wide[:, N:2 * N], bn=bn)
        assert not wide[:, :N].any() and not wide[:, 2 * N:].any()
    _close(got, want, f"{terms} {M}x{N}x{K}", rel=1e-4)


# one and two tiles of each stream, last tiles of one row or key, one warpgroup without a tile
@pytest.mark.parametrize("Sq,Skv", [(1, 1), (65, 64), (128, 65), (257, 129), (64, 300), (300, 193)])
@pytest.mark.parametrize("Dh", [64, 128])
def test_attention_few_tiles(Sq, Skv, Dh):
    q, k, v = (_rand(2, s, 3, Dh, seed=i).requires_grad_(True) for i, s in enumerate((Sq, Skv, Skv)))
    do = _rand(2, Sq, 3, Dh, seed=5)
    o = O.attention(q, k, v)
    got = torch.autograd.grad(o, (q, k, v), do)
    q2, k2, v2 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    want = torch.nn.functional.scaled_dot_product_attention(*(t.transpose(1, 2) for t in (q2, k2, v2))).transpose(1, 2)
    wants = torch.autograd.grad(want, (q2, k2, v2), do.double())
    native.check_status(o)
    # P, dS and the result are rounded to bf16 once each (2^-9 relative), o once more on its way into delta
    for a, b, n in zip((o, *got), (want, *wants), ("o", "dq", "dk", "dv")):
        err = float((a.double() - b).norm() / b.norm().clamp_min(1e-9)) if b.norm() > 1e-6 else float(a.double().norm())
        assert err < 4 * 2.0 ** -9, (n, err)


@pytest.mark.parametrize("B,S,bias", [(1, 1, False), (1, 45, False), (2, 9, True), (3, 130, False)])
def test_prompt_layers_keep_every_bit(B, S, bias):
    """The fused prompt and the modules (one of them hooked, which the fused path leaves to itself) give the same bits."""
    from mojodiffusion_b200.llm.decoder import Qwen3Decoder
    from mojodiffusion_b200.models.text.qwen3 import Qwen3Config, Qwen3Encoder
    cfg = Qwen3Config(vocab_size=512, hidden_size=384, intermediate_size=776, num_hidden_layers=3, num_attention_heads=6, num_key_value_heads=2,
                      head_dim=128, qkv_bias=bias)
    torch.manual_seed(0)
    enc = Qwen3Encoder(cfg, torch.bfloat16, DEV).eval()
    for n, p in enc.named_parameters():
        p.data.normal_(1.0 if n.endswith("norm.weight") or "layernorm" in n else 0.0, 0.05)
    dec, ids = Qwen3Decoder(enc), torch.randint(0, 512, (B, S), device=DEV)
    fused, routes = dec._fused_layers, []
    dec._fused_layers = lambda *a: routes.append(fused(*a)) or routes[-1]
    h, cache = dec.prefill(ids, S + 3)
    handle = enc.model.layers[1].input_layernorm.register_forward_hook(lambda *a: None)
    h2, cache2 = dec.prefill(ids, S + 3)
    handle.remove()
    native.check_status(h)
    assert len(routes) == 2 and len(routes[0]) == 3 and routes[1] is None
    assert torch.equal(h, h2) and torch.equal(cache.k, cache2.k) and torch.equal(cache.v, cache2.v)
    # an embedding whose output is laid out in another order goes to the modules, as every tensor they take
    handle = enc.model.embed_tokens.register_forward_hook(lambda m, a, y: y.transpose(1, 2).contiguous().transpose(1, 2))
    h3, cache3 = dec.prefill(ids, S + 3)
    handle.remove()
    assert len(routes) == 2 + (S == 1) and h3.shape == h.shape and torch.isfinite(h3.float()).all()
    # its norms add the squares of a row in another order: a few bf16 roundings on the way
    assert float((h3.float() - h.float()).norm() / h.float().norm()) < 2.0 ** -6


@pytest.mark.parametrize("H,Dh", [(1, 64), (2, 64), (3, 128), (6, 128), (8, 128), (1, 256), (2, 256)])
@pytest.mark.parametrize("interleaved", [True, False])
def test_qk_norm_rope_backward_heads_per_warp(H, Dh, interleaved):
    S, D = 37, H * Dh
    buf, d = _rand(2, S, 3 * D, seed=1), _rand(2, S, 3 * D, seed=2)
    wq, wk = _rand(Dh, seed=3), _rand(Dh, seed=4)
    ang = torch.rand(S, Dh // 2, generator=torch.Generator().manual_seed(5)).to(DEV) * 6
    cos, sin = ang.cos(), ang.sin()
    out = d.clone()
    native.ops().qk_norm_rope_bwd(out, buf, wq, wk, cos, sin, H, Dh, 0, D, 1e-6, interleaved, True, 0, 0)
    x = buf.double().requires_grad_(True)
    y = []
    for part, w in ((0, wq), (1, wk)):
        t = x[..., part * D:(part + 1) * D].unflatten(-1, (H, Dh))
        t = t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        c, s = cos.double()[:, None], sin.double()[:, None]
        if interleaved:
            a, b = t[..., 0::2], t[..., 1::2]
            t = torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)
        else:
            a, b = t[..., :Dh // 2], t[..., Dh // 2:]
            t = torch.cat((a * c - b * s, b * c + a * s), -1)
        y.append(t.flatten(-2))
    (torch.cat(y, -1) * d[..., :2 * D].double()).sum().backward()
    _close(out[..., :2 * D], x.grad[..., :2 * D], f"{H} {Dh}", rel=1e-5)
    assert torch.equal(out[..., 2 * D:], d[..., 2 * D:])


@pytest.mark.parametrize("bias,train_w,scale", [(True, False, 1.0), (False, False, 0.5), (True, True, 1.0)])
def test_adapted_layer_nodes_agree(bias, train_w, scale):
    """The native autograd node of an adapted layer against the one in Python: outputs and gradients, also through saved-tensor hooks."""
    from mojodiffusion_b200.ops.functional import _LoraLinearFn
    x, w, A, B = _rand(77, 64, seed=1), _rand(96, 64, scale=0.1, seed=2), _rand(16, 64, scale=0.1, seed=3), _rand(96, 16, scale=0.1, seed=4)
    b = _rand(96, seed=5) if bias else None
    leaves = [t.requires_grad_(True) for t in (x, A, B)] + ([t.requires_grad_(True) for t in (w, b)] if train_w else [])
    want = _LoraLinearFn.apply(x, w, b, A, B, scale)
    dy = _rand(77, 96, seed=6)
    gw = torch.autograd.grad(want, leaves, dy)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t), t)[1], lambda t: t):
        got = O.lora_linear(x, w, b, A, B, scale)
    gg = torch.autograd.grad(got, leaves, dy)
    assert len(seen) == 6 and torch.equal(got, want) and all(torch.equal(a, c) for a, c in zip(gg, gw))


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 5, 7, 3), (3, 9, 4, 70), (1, 33, 17, 8)])
@pytest.mark.parametrize("layout", ["rows", "planar", "slice"])
def test_pad_channels(shape, layout):
    N, H, W, C = shape
    x = _rand(N, H, W, C)
    if layout == "planar":
        x = _rand(N, C, H, W).permute(0, 2, 3, 1)
    elif layout == "slice":
        x = _rand(N, H + 2, W + 1, C + 3)[:, 1:-1, 1:, 2:C + 2]
    for cp in ((C + 7) // 8 * 8, (C + 63) // 64 * 64):
        got = native.ops().pad_channels(x, cp)
        assert got.is_contiguous() and torch.equal(got, torch.nn.functional.pad(x, (0, cp - C)))


# the pointwise kernel, the few-row kernel, a lone tile of each width and the pair
@pytest.mark.parametrize("route", ["pointwise", "rows", 64, 128, 256, 512])
def test_gelu_is_the_single_precision_tanh_form(route):
    """0.5 x (1 + tanh(u)) with the tanh rounded to single precision, as torch evaluates it: it is -1, and the result zero, from -6 down.
    A form without that cancellation is as good, but gives other bits to a model that was run with this one."""
    from mojodiffusion_b200.ops.functional import _gemm
    rows = 4 if route == "rows" else 300
    x = torch.linspace(-12, 6, 64).repeat(rows, 1).bfloat16().to(DEV) + _rand(rows, 64, scale=0.05)
    eye = torch.eye(64, device=DEV, dtype=torch.bfloat16)
    got = O.activation(x, "gelu_tanh") if route == "pointwise" else _gemm([x], [eye], act=1, bn=0 if route == "rows" else route)
    native.check_status(got)
    want = torch.nn.functional.gelu(x.float(), approximate="tanh")
    # tanh in [-1, -0.5] is a multiple of 2^-24; the approximate exponential and division may take its neighbours
    assert bool(((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + x.float().abs() * 2.0 ** -23).all())
    assert bool((x <= -6).any()) and not got[x <= -6].any()


# one row, a warp without a row, tiles of one row, K off 64, rows and columns that end inside a store's box, several gates in a warp's rows
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (31, 24, 72), (33, 200, 320), (129, 136, 64), (257, 328, 200)])
@pytest.mark.parametrize("bn", [64, 128, 256, 512])
def test_epilogue_rounds_each_product(M, N, K, bn):
    """Scales, bias, gate and residual as separate fp32 operations on the same accumulator give the same bits: no product is contracted
    with the sum that follows it."""
    from mojodiffusion_b200.ops.functional import _gemm
    x, w, b, res = _rand(M, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2), _rand(N, seed=3), _rand(M, N, seed=5)
    rows = (M + 4) // 5
    gate = _rand(5, N, seed=4)
    each = gate.float().repeat_interleave(rows, 0)[:M]
    acc = _gemm([x], [w], out_fp32=True, bn=bn)
    got = _gemm([x], [w], bias=b, residual=res, gate=gate, rows_per_group=rows, bn=bn)
    assert torch.equal(got, ((acc + b.float()) * each + res.float()).bfloat16())
    assert torch.equal(_gemm([x], [w], gate=gate, rows_per_group=rows, bn=bn), (acc * each).bfloat16())
    assert torch.equal(_gemm([x], [w], bias=b, alpha=0.3, bn=bn), (acc * torch.tensor(0.3, device=DEV) + b.float()).bfloat16())
    if K % 16 == 0:
        (xq, xs), (wq, ws) = O.fp8_quant_rows(x), O.fp8_quant_rows(w)
        acc = _gemm([xq], [wq], out_fp32=True, bn=bn)
        got = _gemm([xq], [wq], bias=b, residual=res, row_scale=xs, col_scale=ws, bn=bn)
        assert torch.equal(got, (acc * xs[:, None] * ws + b.float() + res.float()).bfloat16())
    native.check_status(got)


@pytest.mark.parametrize("scale", [1.0, 0.5])
@pytest.mark.parametrize("where", ["nowhere", "forward", "backward"])
def test_adapted_layer_recomputed_across_a_mode(where, scale):
    """A dispatch mode around one direction only makes the layer run the Python node there and the native one in the other."""
    import contextlib
    from torch.utils._python_dispatch import TorchDispatchMode
    from torch.utils.checkpoint import checkpoint

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    x, w, b = _rand(77, 64, seed=1).requires_grad_(True), _rand(96, 64, scale=0.1, seed=2), _rand(96, seed=5)
    A, B = _rand(16, 64, scale=0.1, seed=3).requires_grad_(True), _rand(96, 16, scale=0.1, seed=4).requires_grad_(True)
    dy = _rand(77, 96, seed=6)
    want = torch.autograd.grad(O.lora_linear(x, w, b, A, B, scale), (x, A, B), dy)
    with Watch() if where == "forward" else contextlib.nullcontext():
        y = checkpoint(lambda t: O.lora_linear(t, w, b, A, B, scale), x, use_reentrant=False)
    with Watch() if where == "backward" else contextlib.nullcontext():
        got = torch.autograd.grad(y, (x, A, B), dy)
    assert all(torch.equal(a, c) for a, c in zip(got, want))


@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_adapted_layer_notices_a_changed_factor(scale):
    x, w = _rand(77, 64, seed=1).requires_grad_(True), _rand(96, 64, scale=0.1, seed=2)
    A, B = _rand(16, 64, scale=0.1, seed=3).requires_grad_(True), _rand(96, 16, scale=0.1, seed=4).requires_grad_(True)
    y = O.lora_linear(x, w, None, A, B, scale)
    with torch.no_grad():
        B.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(_rand(77, 96, seed=6))


@pytest.mark.parametrize("H,Dh", [(24, 128), (10, 64), (3, 128), (2, 256)])
@pytest.mark.parametrize("interleaved", [True, False])
def test_qk_norm_rope_backward_rounds_one_product(H, Dh, interleaved):
    """The rotation alone, bit by bit: one product of each pair is rounded to fp32, the other one joins it in a fused multiply-add."""
    S, D = 1536, H * Dh
    d = _rand(1, S, 2 * D, seed=2)
    ang = (torch.rand(S, Dh // 2, generator=torch.Generator().manual_seed(5)) * 6).to(DEV)
    cos, sin = ang.cos(), ang.sin()
    out = d.clone()
    native.ops().qk_norm_rope_bwd(out, d, None, None, cos, sin, H, Dh, 0, D, 1e-6, interleaved, False, 0, 0)
    g, c, s = d.unflatten(-1, (2 * H, Dh)).float(), cos[:, None], sin[:, None]

    def fma(p, q, r):                                  # products of 8 and 24 bits are exact in fp64
        return (p.double() * q.double() + r.double()).float()
    if interleaved:
        a, b = g[..., 0::2], g[..., 1::2]
        want = torch.stack((fma(a, c, b * s), fma(b, c, -(a * s))), -1).flatten(-2)
    else:
        a, b = g[..., :Dh // 2], g[..., Dh // 2:]
        want = torch.cat((fma(b, s, a * c), fma(b, c, -(a * s))), -1)
    native.check_status(out)
    assert torch.equal(out, want.flatten(-2).bfloat16())


@pytest.mark.parametrize("form", ["plain", "extra", "adapted"])
def test_linear_writes_a_range_of_tokens(form):
    """An output whose leading dimensions have no common stride cannot be flattened without a copy; one that can is written in place."""
    x, w, A, B = _rand(2, 3, 64, seed=1), _rand(72, 64, scale=0.1, seed=2), _rand(8, 64, scale=0.1, seed=3), _rand(72, 8, scale=0.1, seed=4)
    buf = torch.zeros(2, 5, 72, device=DEV, dtype=torch.bfloat16)

    def run(out):
        if form == "adapted":
            return O.lora_linear(x, w, None, A, B, 1.0, out=out)
        return O.linear(x, w, out=out, extra=[(x, w)] if form == "extra" else ())
    want = run(None)
    assert want.shape == (2, 3, 72) and want.any()
    got = run(buf[:, 1:4])
    native.check_status(got)
    assert torch.equal(buf[:, 1:4], want) and not buf[:, ::4].any()
    wide = torch.zeros(2, 3, 3 * 72, device=DEV, dtype=torch.bfloat16)
    run(wide[..., 72:144])
    assert torch.equal(wide[..., 72:144], want) and not wide[..., :72].any() and not wide[..., 144:].any()


# a bias, residual, gate or output off 16 bytes leaves the bulk stores: the kernels whose lanes store their own rows
@pytest.mark.parametrize("M,N,K", [(33, 200, 320), (257, 328, 200)])
@pytest.mark.parametrize("bn", [64, 128, 256, 512])
@pytest.mark.parametrize("off", ["bias", "residual", "gate", "out"])
def test_gemm_terms_off_sixteen_bytes(M, N, K, bn, off):
    from mojodiffusion_b200.ops.functional import _gemm

    def place(t, name):
        if off != name:
            return t
        wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 3, device=DEV, dtype=t.dtype) if t.dim() > 1 else torch.zeros(t.numel() + 1, device=DEV, dtype=t.dtype)
        part = wide[..., 1:1 + t.shape[-1]]
        part.copy_(t)
        return part
    x, w = _rand(M, K, seed=1), _rand(N, K, scale=1 / math.sqrt(K), seed=2)
    b, res, gate, out = (place(_rand(*s, seed=i), n) for i, (s, n) in enumerate((((N,), "bias"), ((M, N), "residual"), ((3, N), "gate"), ((M, N), "out"))))
    rows = (M + 2) // 3
    want = ((x.float() @ w.float().t() + b.float()) * gate.float().repeat_interleave(rows, 0)[:M] + res.float())
    got = _gemm([x], [w], bias=b, residual=res, gate=gate, rows_per_group=rows, out=out, bn=bn)
    assert got.data_ptr() == out.data_ptr()
    _close(got, want, f"{off} {M}x{N}x{K} bn {bn}", rel=1e-4)


# a lone CTA's tile, pairs of 256 and 128 channels, the resident filter, stride 2; images whose edges cut the patches
@pytest.mark.parametrize("n,h,w,cin,cout,size,stride", [(1, 9, 17, 64, 64, 5, 1), (2, 70, 150, 128, 256, 3, 1), (2, 150, 150, 192, 128, 3, 1),
                                                        (1, 270, 150, 64, 128, 3, 1), (1, 34, 50, 64, 128, 3, 2)])
@pytest.mark.parametrize("off", ["bias", "residual"])
def test_conv_terms_off_sixteen_bytes(n, h, w, cin, cout, size, stride, off):
    from mojodiffusion_b200.ops import conv as C
    x, f = _rand(n, h, w, cin, seed=1), _rand(cout, size, size, cin, scale=1 / math.sqrt(size * size * cin), seed=2)
    b = _rand(cout + 1, seed=3)[1 if off == "bias" else 0:][:cout]
    want = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), f.double().permute(0, 3, 1, 2), b.double(), stride, size // 2).permute(0, 2, 3, 1)
    res = None
    if off == "residual" and stride == 1:
        res = _rand(n * h * w * cout + 1, seed=4)[1:].view(n, h, w, cout)
        want = want + res.double()
    _close(C.conv2d_nhwc(x, f, b, stride, size // 2, residual=res), want, f"{off} {n}x{h}x{w} {cin}->{cout}", rel=1e-4)
