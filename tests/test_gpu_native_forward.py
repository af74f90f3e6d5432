"""What only the native host path uses, against the separate operators and the Python code it stands for: same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _codebook(gen, bits, dev):
    cb = torch.sort(torch.randn(2 ** bits, generator=gen) * 1.2)[0].to(dev)
    return cb, (cb[:-1] + cb[1:]) / 2


# rows around the 32-row blocks, 128-row CTAs and 256-row pair tiles; slabs of 64, 128 and 192 columns; one and several tiles per
# pair; streamed and stationary weight
@pytest.mark.parametrize("M,N,K,bits", [(1, 64, 64, 4), (31, 320, 128, 2), (197, 768, 192, 3), (255, 1536, 384, 4), (257, 256, 1536, 4),
                                        (1576, 3072, 768, 3), (7289, 768, 192, 2), (12608, 1536, 384, 4)])
@pytest.mark.parametrize("bias", [True, False])
def test_gemm_with_gelu_and_quantizer_equals_the_two_operators(pkg, cuda_device, M, N, K, bits, bias):
    gen = torch.Generator().manual_seed(M + N + K)
    cb, th = _codebook(gen, bits, cuda_device)
    x = torch.randn(M, K, generator=gen)
    x[:: 7] *= 40.0                                       # GELU arguments beyond the polynomial's range, both signs
    w = torch.randn(N, K, generator=gen) * K ** -0.5
    if M > 100:
        x[13] = 6.0e4                                     # overflows fp16: a row of infinities and NaN
        w[:, 0] = w[:, 0].abs() + 1.0
    x, w = x.half().to(cuda_device), w.half().to(cuda_device)
    b = torch.randn(N, generator=gen).to(cuda_device) if bias else None
    h = pkg.ops.dense_weight_gemm(x, w, b)
    want = pkg.ops.quantize_activation_dequant(h, th, cb, bits, 64, torch.float16, True)
    with pkg._cabi.option("ARCQ_GELU_GEMM", 1):           # at every size, not only where the dispatch takes it
        got = pkg.ops.dense_weight_gemm_gelu_quant(x, w, b, th, cb, bits, 64)
    assert pkg.ops.device_status() == 0
    nan = want.isnan()
    assert torch.equal(got.isnan(), nan)
    assert torch.equal(got.masked_fill(nan, 0), want.masked_fill(nan, 0))
    assert pkg._cabi.last_gemm_kernel() == pkg._cabi.GEMM_PAIR_DENSE_GELU_QUANT


@pytest.mark.parametrize("name,bits", [("deit_tiny", 3), ("deit_small", 4), ("deit_base", 2)])
def test_native_forward_equals_the_python_forward(pkg, cuda_device, name, bits, monkeypatch):
    """Batch sizes on both sides of every size rule; the weights go through two scratch matrices in turn."""
    model = pkg.create_vit(name, seed=1)
    model.blocks = torch.nn.ModuleList(list(model.blocks)[:3])
    model = model.half().to(cuda_device)
    gen = torch.Generator().manual_seed(5)
    images = torch.randn(40, 3, 224, 224, generator=gen).half().to(cuda_device)
    with torch.no_grad():
        model = pkg.quantise_model(model, images[:4], bits)
        got = {b: model(images[:b]) for b in (1, 2, 3, 8, 17, 40)}
        monkeypatch.setattr(pkg.vit.VisionTransformer, "_forward_native", lambda self, x: None)
        for b, y in got.items():
            assert torch.equal(y, model(images[:b])), f"batch {b}"
    assert pkg.ops.device_status() == 0


def _packed_layer(pkg, bits, K, N, dev, on_the_fly, bias=True):
    gen = torch.Generator().manual_seed(K + N + bits)
    linear = torch.nn.Linear(K, N, bias=bias)
    with torch.no_grad():
        linear.weight.copy_(torch.randn(N, K, generator=gen) * 0.03)
        if bias:
            linear.bias.copy_(torch.randn(N, generator=gen) * 0.1)
    cb, th = _codebook(gen, bits, dev)
    return pkg.pack_linear(linear.to(dev), bits, cb, th, group_size=64, on_the_fly=on_the_fly), gen


# packed rows of 24, 72, 120 and 192 bytes (the last a multiple of 16); rows of x on both sides of the quantizers' size rule
@pytest.mark.parametrize("K,N", [(64, 64), (192, 576), (320, 48), (512, 192)])
@pytest.mark.parametrize("M", [1, 197, 12700])
def test_three_bit_rows_of_any_length_equal_the_packed_operators(pkg, cuda_device, K, N, M):
    """The packed linears against quantize_activation + arcq_linear_forward on their buffers, which rebuilds rows that are no
    multiple of 16 bytes in fp32 with one rounding: same bits."""
    for on_the_fly, dtype in ((True, torch.float16), (False, torch.float32), (False, torch.bfloat16)):
        layer, gen = _packed_layer(pkg, 3, K, N, cuda_device, on_the_fly)
        x = torch.randn(M, K, generator=gen).to(dtype).to(cuda_device)
        b = layer._buffers
        codes = pkg.ops.quantize_activation(x, layer.activation_thresholds, layer.activation_codebook, 3, 64)
        want = pkg.ops.arcq_linear_forward(*codes, b["packed_weight_codes"], b["weight_center"], b["weight_scale"], b["weight_code_sum"],
                                           b["activation_codebook"], b["weight_codebook"], b.get("bias", b.get("bias_tensor")), 3, 64, K, N,
                                           torch.float16 if on_the_fly else torch.float32)
        assert torch.equal(layer(x), want)
        wide = torch.empty(M, K + 8, dtype=dtype, device=cuda_device)[:, :K].copy_(x)      # not contiguous: the Python route
        assert torch.equal(layer(wide), want)
    assert pkg.ops.device_status() == 0
