"""The pair GEMM's tiles: pairs that change slabs from tile to tile, and the bias that goes with them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# K = 768 streams both operands: fewer tiles than pairs, one more than a round, several rounds; slabs of every width, ragged rows,
# widths that leave a slab to one half of the epilogue warps (32, 96, 160); from K = 1024 on the last round in halves: one tile of it,
# several, half a round
@pytest.mark.parametrize("M,N,K", [(1, 32, 768), (300, 96, 768), (300, 160, 768), (1000, 2304, 768), (6305, 768, 768), (6305, 3072, 768),
                                   (19001, 768, 768), (700, 384, 1536),
                                   (12608, 384, 1536), (6305, 768, 1024), (19001, 768, 1024), (9473, 512, 1088)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("bias", ["none", "aligned", "offset"])
def test_every_tile_gets_its_columns_and_its_bias(pkg, cuda_device, M, N, K, dtype, bias):
    gen = torch.Generator(device=cuda_device).manual_seed(M + N)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    w = (torch.randn(N, K, generator=gen, device=cuda_device) * K ** -0.5).half()
    store = torch.randn(N + 1, generator=gen, device=cuda_device) * 4
    b = None if bias == "none" else store[:N] if bias == "aligned" else store[1:]      # the last one not 16-byte aligned
    y = pkg.ops.dense_weight_gemm(x, w, b, dtype)
    want = x.double() @ w.double().t() + (0 if b is None else b.double())
    # fp32 sums of K products of unit variance, then one rounding to the output type
    tol = 2.0 ** -24 * K + want.abs() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -23)
    assert bool(((y.double() - want).abs() <= tol + 2.0 ** -25).all())
    # a row does not depend on the tile it falls in, a whole one or a half
    with pkg._cabi.option("ARCQ_PAIR_SPLIT", 0):
        assert torch.equal(pkg.ops.dense_weight_gemm(x, w, b, dtype), y)
        with pkg._cabi.option("ARCQ_PAIR_STAGGER", 1):          # pairs that keep their slabs
            assert torch.equal(pkg.ops.dense_weight_gemm(x, w, b, dtype), y)
    with pkg._cabi.option("ARCQ_PAIR_STAGGER", 0):
        assert torch.equal(pkg.ops.dense_weight_gemm(x, w, b, dtype), y)
    part = pkg.ops.dense_weight_gemm(x[M // 2:].contiguous(), w, b, dtype)
    assert torch.equal(part, y[M // 2:])
    assert pkg.ops.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(6305, 3072, 768), (19001, 3072, 768), (300, 768, 768), (5000, 1536, 384)])
@pytest.mark.parametrize("offset", [0, 1])
def test_the_quantising_epilogue_gets_its_bias(pkg, cuda_device, M, N, K, offset):
    gen = torch.Generator(device=cuda_device).manual_seed(M + N)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    w = (torch.randn(N, K, generator=gen, device=cuda_device) * 0.4 * K ** -0.5).half()
    b = (torch.randn(N + 1, generator=gen, device=cuda_device))[offset:N + offset]
    cb = torch.linspace(-2.2, 2.2, 16, device=cuda_device)
    th = (cb[:-1] + cb[1:]) / 2
    with pkg._cabi.option("ARCQ_GELU_GEMM", 1):
        got = pkg.ops.dense_weight_gemm_gelu_quant(x, w, b, th, cb, 4, 64)
    h = pkg.ops.dense_weight_gemm(x, w, b, torch.float16)
    want = pkg.ops.quantize_activation_dequant(h, th, cb, 4, 64, torch.float16, pre_gelu=True)
    assert torch.equal(got, want)
    assert pkg.ops.device_status() == 0
