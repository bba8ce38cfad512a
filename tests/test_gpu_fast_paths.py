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
    for Cin, Cout in ((64, 128), (128, 256)):                  # several tiles per persistent cluster: every ring wraps
        x, w = _rand(1, 200, 333, Cin, seed=1), _rand(Cout, 3, 3, Cin, scale=1 / math.sqrt(9 * Cin), seed=2)
        with torch.no_grad():
            _close(C.conv2d_nhwc(x, w, _rand(Cout, seed=3)), _conv_ref(x, w, _rand(Cout, seed=3)), f"{Cin} -> {Cout}")


# one patch (its partner of the pair lies past the batch), images smaller than a patch, ragged edges both ways, an odd number of
# patches; 8 / 64, 128 / 320 and 512 / 648 output channels take the 64-, 128- and 256-wide tiles on some of the sizes
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
