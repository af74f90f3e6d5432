"""Reconstruction from packed codes: the kernel with wide stores against the one that takes any alignment, and both against torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# less than a block, two chunks of which the second is missing, whole rounds and more
@pytest.mark.parametrize("R,K", [(1, 64), (3, 192), (37, 704), (1000, 384), (9473, 3072)])
@pytest.mark.parametrize("bits", [4, 3, 2])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_wide_stores_give_the_same_values(pkg, cuda_device, R, K, bits, dtype):
    gen = torch.Generator(device=cuda_device).manual_seed(R + K + bits)
    x = torch.randn(R, K, generator=gen, device=cuda_device) * 3 + 1
    cb = torch.sort(torch.randn(2 ** bits, generator=gen, device=cuda_device))[0]
    th = (cb[:-1] + cb[1:]) / 2
    packed, mu, sg, cs = pkg.ops.quantize_activation(x, th, cb, bits, 64)
    got = pkg.ops.dequant(packed, mu, sg, cs, cb, bits, 64, dtype)                       # right behind the kernel that wrote the codes
    buf = torch.zeros(R * K + 9, dtype=dtype, device=cuda_device)
    off = pkg.ops.dequant(packed, mu, sg, cs, cb, bits, 64, dtype, out=buf[1:])         # not 16-byte aligned
    assert torch.equal(got, off) and float(buf[0]) == 0 and bool((buf[1 + R * K:] == 0).all())
    codes = pkg.packing.unpack_codes(packed.cpu(), bits, K).to(cuda_device)
    want = mu.repeat_interleave(64, 1) + sg.repeat_interleave(64, 1) * (cb[codes] - (cs / 64).repeat_interleave(64, 1))
    assert torch.equal(got, want.to(dtype))


# the kernel starts while the one before it in the stream may still run: a codebook that is that one's output, written in place, and a
# strided one, which the operator copies right before its launch
@pytest.mark.parametrize("R,K", [(1, 64), (300, 384)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("strided", [False, True])
def test_levels_written_right_before_the_call(pkg, cuda_device, R, K, dtype, strided):
    gen = torch.Generator(device=cuda_device).manual_seed(R + K)
    x = torch.randn(R, K, generator=gen, device=cuda_device)
    books = torch.sort(torch.randn(64, 16, generator=gen, device=cuda_device))[0]
    packed, mu, sg, cs = pkg.ops.quantize_activation(x, (books[0, :-1] + books[0, 1:]) / 2, books[0].contiguous(), 4, 64)
    idx = pkg.packing.unpack_codes(packed.cpu(), 4, K).to(cuda_device)
    wide = torch.zeros(16, 2, device=cuda_device)
    outs = [torch.empty(R, K, dtype=dtype, device=cuda_device) for _ in books]
    torch.cuda.synchronize()
    for cb, out in zip(books, outs):
        wide[:, 0].copy_(cb)
        levels = wide[:, 0] if strided else wide.view(-1)[:16].copy_(cb)
        pkg.ops.dequant(packed, mu, sg, cs, levels, 4, 64, dtype, out=out)
    for cb, out in zip(books, outs):
        want = mu.repeat_interleave(64, 1) + sg.repeat_interleave(64, 1) * (cb[idx] - (cs / 64).repeat_interleave(64, 1))
        assert torch.equal(out, want.to(dtype))
