"""Residual add + LayerNorm (+ quantizer): blocks that take several tiles, ragged ends, and the sum of two fp16 values."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one tile of 128 groups, one row more or less, and more tiles than blocks (592 on 148 SMs) with a ragged last one
@pytest.mark.parametrize("K,M", [(192, 42), (192, 43), (192, 25301), (384, 21), (384, 22), (384, 12651), (768, 10), (768, 11), (768, 6333),
                                 (768, 13001)])
@pytest.mark.parametrize("with_y", [True, False])
def test_tiles_of_a_block(pkg, cuda_device, K, M, with_y):
    gen = torch.Generator(device=cuda_device).manual_seed(K + M)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    y = (torch.randn(M, K, generator=gen, device=cuda_device) * 0.5).half() if with_y else None
    norm = torch.nn.LayerNorm(K, eps=1e-6).to(cuda_device)
    with torch.no_grad():
        norm.weight.normal_(1, 0.1, generator=gen)
        norm.bias.normal_(0, 0.1, generator=gen)
    cb = torch.linspace(-2.2, 2.2, 16, device=cuda_device)
    th = (cb[:-1] + cb[1:]) / 2
    s0, h0 = pkg.ops.add_layernorm(x, y, norm)
    want = pkg.ops.quantize_activation_dequant(h0, th, cb, 4, 64, torch.float16)
    with pkg._cabi.option("ARCQ_LNQ_SMALL", 0):
        s1, xhat, h1 = pkg.ops.add_layernorm_quant(x, y, norm, th, cb, 4, 64, want_h=True)
    assert torch.equal(s0, s1) and torch.equal(h0, h1) and torch.equal(xhat, want)
    ref = torch.nn.functional.layer_norm(s0.double(), (K,), norm.weight.double(), norm.bias.double(), 1e-6)
    # fp16 rounds by 2^-11 of the value (2^-25 where it is subnormal); the fp32 steps before it (statistics, product, sum) lose at most
    # 2^-21 of |normalised value * gamma| + |beta| + 1, whatever is left of them after a cancellation: below 8 for these inputs
    assert bool(((h0.double() - ref).abs() <= ref.abs() * 2.0 ** -11 + 2.0 ** -25 + 8 * 2.0 ** -21).all())
    assert pkg.ops.device_status() == 0


def test_residual_sum_is_rounded_once(pkg, cuda_device):
    """Every pair of exponents, with values that make ties: what the fp32 sum rounds to."""
    exps = torch.arange(-24, 16, device=cuda_device)
    mant = torch.tensor([1.0, 1 + 2.0 ** -10, 1.5, 2 - 2.0 ** -10, 1 + 2.0 ** -1 + 2.0 ** -10], device=cuda_device)
    v = (mant[None] * 2.0 ** exps[:, None].float()).half().flatten()
    v = torch.cat([v, -v, torch.zeros(1, device=cuda_device).half(), torch.tensor([float("inf")], device=cuda_device).half()])
    a, b = torch.meshgrid(v, v, indexing="ij")
    n = a.numel() // 384 * 384
    x, y = a.flatten()[:n].view(-1, 384).contiguous(), b.flatten()[:n].view(-1, 384).contiguous()
    norm = torch.nn.LayerNorm(384, eps=1e-6).to(cuda_device)
    s, _ = pkg.ops.add_layernorm(x, y, norm)
    want = (x.float() + y.float()).half()
    assert torch.equal(torch.nan_to_num(s.float(), nan=1e9), torch.nan_to_num(want.float(), nan=1e9))


@pytest.mark.parametrize("K,M", [(192, 43), (384, 12651), (768, 13001)])      # one tile, and several tiles a block
@pytest.mark.parametrize("with_y", [True, False])
def test_a_wait_for_the_rows_that_runs_out(pkg, cuda_device, K, M, with_y):
    """No poll: the kernel ends, says so in the status word and has stored nothing, and the next launch is none the worse."""
    gen = torch.Generator(device=cuda_device).manual_seed(K + M)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    y = torch.randn(M, K, generator=gen, device=cuda_device).half()
    gamma, beta = torch.ones(K, device=cuda_device).half(), torch.zeros(K, device=cuda_device).half()
    cb = torch.linspace(-2.2, 2.2, 16, device=cuda_device)
    th = (cb[:-1] + cb[1:]) / 2
    lib = pkg._cabi.load()

    def run():
        outs = [torch.full((M, K), 77.0, device=cuda_device).half() for _ in range(3)]
        torch.cuda.synchronize()
        rc = lib.arcq_add_layernorm_act_quant_unpack(
            x.data_ptr(), y.data_ptr() if with_y else None, gamma.data_ptr(), beta.data_ptr(), pkg._cabi.DT_F16, 1e-6, M, K, th.data_ptr(),
            cb.data_ptr(), 4, 64, outs[0].data_ptr() if with_y else None, outs[1].data_ptr(), outs[2].data_ptr(), 0, None, 0, None)
        assert rc == 0
        return outs
    with pkg._cabi.option("ARCQ_LNQ_SMALL", 0):
        want = run()
        with pkg._cabi.option("ARCQ_POLL_LIMIT", 0):
            got = run()
        assert pkg.ops.device_status() == 0x411
        assert pkg.ops.device_status() == 0
        assert all(bool((o == 77.0).all()) for o in got)
        assert all(torch.equal(a, b) for a, b in zip(run(), want))
    assert pkg.ops.device_status() == 0
