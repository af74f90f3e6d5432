"""The packed linear in one launch against the two launches it stands for: the same bits, whatever rows and columns a block takes."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(pkg, dev, K, N, bits, on_the_fly, bias=True, pre_gelu=False, seed=0):
    gen = torch.Generator(device=dev).manual_seed(K + N + bits + seed)
    linear = torch.nn.Linear(K, N, bias=bias, device=dev)
    with torch.no_grad():
        linear.weight.normal_(0, 0.02, generator=gen)
        if bias:
            linear.bias.normal_(0, 1, generator=gen)
    cb = torch.linspace(-2.3, 2.4, 2 ** bits, device=dev)
    th = (cb[:-1] + cb[1:]) / 2
    layer = pkg.pack_linear(linear, bits, cb, th, group_size=64, on_the_fly=on_the_fly)
    if pre_gelu:
        layer.pre_gelu = True
    return layer, gen


class _Job(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("packed", "mu", "sigma", "codesum", "codebook", "out")] + [
        ("rows", ctypes.c_int64), ("K", ctypes.c_int64), ("bits", ctypes.c_int)]


def _call(pkg, layer, x, y):
    """The C entry point, into an output of the caller's."""
    ptr = lambda t: t.data_ptr()
    job = _Job(ptr(layer.packed_weight_codes), ptr(layer.weight_center), ptr(layer.weight_scale), ptr(layer.weight_code_sum),
               ptr(layer.weight_codebook), None, y.shape[1], x.shape[1], 4)
    rc = pkg._cabi.load().arcq_packed_linear_small(0, ptr(x), pkg._cabi.DT_F16, x.shape[0], ptr(layer.activation_thresholds),
                                                   ptr(layer.activation_codebook), 0, ctypes.byref(job), ptr(layer.bias_tensor), ptr(y),
                                                   pkg._cabi.DT_F16, None)
    assert rc == 0, pkg._cabi.last_error()


def _both(pkg, layer, x):
    """Outputs of the one launch (forced) and of the two."""
    with pkg._cabi.option("ARCQ_SMALL_LINEAR", 1):
        one = layer(x)
        assert pkg._cabi.last_gemm_kernel() == pkg._cabi.GEMM_SMALL_LINEAR
    with pkg._cabi.option("ARCQ_SMALL_LINEAR", 0):
        two = layer(x)
        assert pkg._cabi.last_gemm_kernel() != pkg._cabi.GEMM_SMALL_LINEAR
    assert pkg.ops.device_status() == 0
    return one, two


# rows around the blocks of 8 to 128, one group and many, one slab and many, 3-bit rows of an odd number of groups (other operands)
@pytest.mark.parametrize("M,K,N", [(1, 64, 16), (1, 3072, 768), (7, 192, 192), (8, 384, 1536), (9, 768, 48), (33, 192, 576), (64, 1536, 384),
                                   (65, 384, 384), (129, 192, 192), (197, 192, 768), (560, 192, 192)])
@pytest.mark.parametrize("bits", [4, 3, 2])
@pytest.mark.parametrize("form", ["half", "half gelu", "half no bias", "float", "float from f16", "float from bf16"])
def test_one_launch_equals_two(pkg, cuda_device, M, K, N, bits, form):
    layer, gen = _layer(pkg, cuda_device, K, N, bits, form.startswith("half"), bias="no bias" not in form, pre_gelu="gelu" in form)
    dtype = {"half": torch.float16, "float": torch.float32}.get(form, torch.bfloat16 if "bf16" in form else torch.float16)
    x = torch.randn(M, K, generator=gen, device=cuda_device)
    x[:, :3] *= 20.0
    one, two = _both(pkg, layer, x.to(dtype))
    assert one.dtype == two.dtype and torch.equal(one, two)


@pytest.mark.parametrize("R", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("bn", [16, 32, 48, 64, 96, 128, 192])
def test_rows_and_columns_of_a_block(pkg, cuda_device, R, bn):
    M, K, N = 133, 192, 576
    layer, gen = _layer(pkg, cuda_device, K, N, 4, True)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    with pkg._cabi.option("ARCQ_SMALL_R", R), pkg._cabi.option("ARCQ_SMALL_BN", bn), pkg._cabi.option("ARCQ_SMALL_LINEAR", 1):
        fits = bool(pkg._cabi.load().arcq_packed_linear_small_applies(M, N, K))
        assert fits == (N % bn == 0 and -(-M // R) * (N // bn) <= torch.cuda.get_device_properties(cuda_device).multi_processor_count)
        if fits:
            assert torch.equal(*_both(pkg, layer, x))


def test_infinities_and_nan_stay_in_their_rows(pkg, cuda_device):
    layer, gen = _layer(pkg, cuda_device, 384, 384, 4, True)
    x = torch.randn(40, 384, generator=gen, device=cuda_device).half()
    x[3, 5], x[11, 200], x[39, 383] = float("inf"), float("nan"), 6.0e4
    one, two = _both(pkg, layer, x)
    assert torch.equal(one.isnan(), two.isnan()) and torch.equal(one.nan_to_num(0), two.nan_to_num(0))
    assert not bool(one[[0, 1, 2, 4, 10, 12, 38]].isnan().any())


def test_a_wait_that_runs_out(pkg, cuda_device):
    """No poll for the products: the status word says so, and the next call is right."""
    layer, gen = _layer(pkg, cuda_device, 192, 192, 4, True)
    x = torch.randn(20, 192, generator=gen, device=cuda_device).half()
    with pkg._cabi.option("ARCQ_SMALL_LINEAR", 1), pkg._cabi.option("ARCQ_POLL_LIMIT", 0):
        layer(x)
        torch.cuda.synchronize()
        assert pkg.ops.device_status() == 0x601
    assert torch.equal(*_both(pkg, layer, x))


@pytest.mark.parametrize("polls", [0, 1, 2, 3, 5, 8])
@pytest.mark.parametrize("M,K,N", [(20, 192, 192), (33, 768, 768), (128, 192, 768)])
def test_no_row_is_missing_without_a_word(pkg, cuda_device, polls, M, K, N):
    """Waits that may run out in some warps of a block and not in others: what is not in the output is in the status word."""
    layer, gen = _layer(pkg, cuda_device, K, N, 4, True)
    x = torch.randn(M, K, generator=gen, device=cuda_device).half()
    want, _ = _both(pkg, layer, x)
    y = torch.empty(M, N, device=cuda_device).half()
    for _ in range(20):
        y.fill_(777.0)
        torch.cuda.synchronize()
        with pkg._cabi.option("ARCQ_SMALL_LINEAR", 1), pkg._cabi.option("ARCQ_POLL_LIMIT", polls):
            _call(pkg, layer, x, y)
        status = pkg.ops.device_status()
        assert status in (0, 0x601)
        assert bool(((y == want) | (y == 777.0)).all()) and (status != 0 or torch.equal(y, want))
    assert torch.equal(layer(x), want) and pkg.ops.device_status() == 0


def test_new_inputs_streams_and_capture(pkg, cuda_device):
    layer, gen = _layer(pkg, cuda_device, 192, 192, 4, True)
    xs = [torch.randn(m, 192, generator=gen, device=cuda_device).half() for m in (5, 50, 197)]
    want = [_both(pkg, layer, x)[1] for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    got = []
    for _ in range(20):
        for s, x in zip(streams, xs):
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(layer(x))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i % 3]) for i, y in enumerate(got))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = layer(xs[2])
        z = layer(y)                       # the one launch behind itself
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want[2]) and torch.equal(z, layer(want[2]))


def test_a_captured_call_takes_what_the_gpu_does_faster(pkg, cuda_device):
    """192 x 192: eight rows in one launch either way, 197 only where the host's time counts; the same bits."""
    layer, gen = _layer(pkg, cuda_device, 192, 192, 4, True)
    for M, captured in ((8, True), (197, False)):
        x = torch.randn(M, 192, generator=gen, device=cuda_device).half()
        want = layer(x)
        assert pkg._cabi.last_gemm_kernel() == pkg._cabi.GEMM_SMALL_LINEAR
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = layer(x)
            assert (pkg._cabi.last_gemm_kernel() == pkg._cabi.GEMM_SMALL_LINEAR) == captured
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
