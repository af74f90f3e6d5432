"""Layer constants that an operator has to copy for its call: the kernels read them early, so the copy has to be written before they start."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _every_other(t):
    """The same values in memory that is not contiguous."""
    wide = torch.zeros(t.numel(), 2, device=t.device, dtype=t.dtype)
    wide[:, 0] = t
    return wide[:, 0]


@pytest.mark.parametrize("M,K", [(5, 192), (3001, 384)])
def test_a_copy_made_for_the_call_is_what_the_kernel_reads(pkg, cuda_device, M, K):
    gen = torch.Generator(device=cuda_device).manual_seed(M)
    ops = pkg.ops
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    w = (torch.randn(K, K, generator=gen, device=cuda_device) * K ** -0.5).half()
    books = torch.sort(torch.randn(20, 16, generator=gen, device=cuda_device))[0]
    biases = torch.randn(20, K, generator=gen, device=cuda_device)
    norms = [torch.nn.LayerNorm(K).to(cuda_device).double() for _ in books]
    singles = [torch.nn.LayerNorm(K).to(cuda_device) for _ in books]
    with torch.no_grad():
        for a, b, bias in zip(norms, singles, biases):
            b.weight.copy_(1 + bias / 8)
            a.weight.copy_(b.weight)
    ths = (books[:, :-1] + books[:, 1:]) / 2
    torch.cuda.synchronize()

    def run(change, norm):
        out = []
        for cb, th, bias, n in zip(books, ths, biases, norm):
            out.append(ops.quantize_activation_dequant(x, change(th), change(cb), 4, 64, torch.float16))
            out.append(ops.dense_weight_gemm(x, w, change(bias)))
            out.extend(ops.add_layernorm(x, None, n))
            out.extend(ops.add_layernorm_quant(x, x, n, change(th), change(cb), 4))
        return out
    assert all(torch.equal(a, b) for a, b in zip(run(_every_other, norms), run(lambda t: t, singles)))
    assert ops.device_status() == 0
