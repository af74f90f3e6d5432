"""What only the native host path uses, against the separate operators and the Python code it stands for: same bits."""
import ctypes
import subprocess
import sys

import pytest
import torch

from conftest import ROOT

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
        got = {b: model._forward_native(images[:b]) for b in (1, 2, 3, 8, 17, 40)}
        assert all(y is not None for y in got.values())      # the native forward took them all
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


def _small_model(pkg, name, bits, dev, blocks=2):
    model = pkg.create_vit(name, seed=1)
    model.blocks = torch.nn.ModuleList(list(model.blocks)[:blocks])
    model = model.half().to(dev)
    images = torch.randn(8, 3, 224, 224, generator=torch.Generator().manual_seed(5)).half().to(dev)
    with torch.no_grad():
        for n, p in model.named_parameters():                  # LayerNorms that do something
            if "norm" in n:
                p.add_(torch.randn(p.shape, generator=torch.Generator().manual_seed(len(n))).to(p) * 0.2)
        return pkg.quantise_model(model, images[:4], bits), images


@torch.no_grad()
def test_a_captured_forward_outlives_what_later_calls_do(pkg, cuda_device):
    """A graph of the native forward, then calls that the native forward does not take, allocations and changed parameters of
    another model: the replay still gives the bits of the capture."""
    model, images = _small_model(pkg, "deit_small", 4, cuda_device)
    want = model(images).clone()
    runner = pkg.GraphedModel(model, images)
    model(images.contiguous(memory_format=torch.channels_last))
    model(images[::2])
    model(images.float()[:, :, ::1].half())
    filler = [torch.full((n,), float("nan"), device=cuda_device) for n in (96, 192, 384, 768) for _ in range(64)]
    assert torch.equal(runner(images), want)
    del filler


@torch.no_grad()
def test_layernorm_parameters_are_read_on_every_call(pkg, cuda_device):
    """Written through .data (no version count), replaced, or in another type: the next forward sees them, on the native and on the
    Python route."""
    model, images = _small_model(pkg, "deit_small", 4, cuda_device)
    strided = images[::2].contiguous(memory_format=torch.channels_last)
    seen = []
    for change in (lambda n: None, lambda n: n.weight.data.mul_(1.5), lambda n: n.bias.data.add_(0.25),
                   lambda n: setattr(n, "weight", torch.nn.Parameter(n.weight * 0.5))):
        for norm in (model.blocks[1].norm1, model.norm):
            change(norm)
        seen.append(model(images[::2].contiguous()))
        assert torch.equal(seen[-1], model(strided))
    for i in range(1, len(seen)):
        assert not torch.equal(seen[i], seen[i - 1])
    for norm in (model.blocks[1].norm1, model.norm):
        norm.float()                                           # the same values
    assert torch.equal(model(images[::2].contiguous()), seen[-1])
    assert pkg.ops.device_status() == 0


# rows of the lane-layout kernels and of the general one; one row, a ragged tile and many tiles
@pytest.mark.parametrize("K", [192, 384, 768, 1000])
@pytest.mark.parametrize("M", [1, 2500])
@torch.no_grad()
def test_layernorm_kernels_read_parameters_of_any_type(pkg, cuda_device, K, M):
    gen = torch.Generator().manual_seed(K + M)
    x, y = (torch.randn(M, K, generator=gen).half().to(cuda_device) for _ in range(2))
    cb, th = _codebook(gen, 4, cuda_device)
    for dtype in (torch.float16, torch.bfloat16):
        norm = torch.nn.LayerNorm(K, eps=1e-6)
        norm.weight.copy_(torch.randn(K, generator=gen)), norm.bias.copy_(torch.randn(K, generator=gen))
        norm = norm.to(dtype).to(cuda_device)
        wide = torch.nn.LayerNorm(K, eps=1e-6).to(cuda_device)
        wide.weight.copy_(norm.weight), wide.bias.copy_(norm.bias)
        for a, b in zip(pkg.ops.add_layernorm(x, y, norm), pkg.ops.add_layernorm(x, y, wide)):
            assert torch.equal(a, b)
        if K != 1000:
            for a, b in zip(pkg.ops.add_layernorm_quant(x, y, norm, th, cb, 4), pkg.ops.add_layernorm_quant(x, y, wide, th, cb, 4)):
                assert torch.equal(a, b)
    assert pkg.ops.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@torch.no_grad()
def test_autocast_gives_what_the_python_forward_gives(pkg, cuda_device, dtype, monkeypatch):
    model, images = _small_model(pkg, "deit_small", 4, cuda_device)
    plain = model(images)
    with torch.autocast("cuda", dtype):
        got = model(images)
        monkeypatch.setattr(pkg.vit.VisionTransformer, "_forward_native", lambda self, x: None)
        want = model(images)
    assert got.dtype == want.dtype and torch.equal(got, want)
    assert dtype != torch.float16 or torch.equal(got, plain)
    assert pkg.ops.device_status() == 0


def _counting(calls):
    def forward(self, x, **kw):
        calls.append(type(self).__name__)
        return type(self).forward(self, x, **kw)
    return forward


@torch.no_grad()
def test_changes_after_the_first_forward_are_seen(pkg, cuda_device, monkeypatch):
    """eps, and a forward set on an instance or on a class, against the Python forward; inputs that are not taken keep the plan."""
    model, images = _small_model(pkg, "deit_small", 4, cuda_device)
    before = model(images)
    model.blocks[0].norm1.eps, model.norm.eps = 0.5, 0.25
    got = model(images)
    assert not torch.equal(got, before)
    plan = pkg.vit._PLANS[model]
    assert torch.equal(model(images.contiguous(memory_format=torch.channels_last)), got)        # the Python forward
    handle = model.blocks[0].mlp.register_forward_hook(lambda *a: None)
    assert torch.equal(model(images), got)
    handle.remove()
    assert pkg.vit._PLANS[model] is plan
    calls = []
    for module in (model.patch_embed, model.blocks[1].attn, model.blocks[0].mlp, model.blocks[1].mlp.fc2, model.head):
        module.forward = _counting(calls).__get__(module)
        assert torch.equal(model(images), got) and calls.pop() == type(module).__name__ and not calls
        del module.forward
        assert torch.equal(model(images), got) and not calls
    attention = pkg.vit.Attention.forward
    monkeypatch.setattr(pkg.vit.Attention, "forward", lambda self, x, **kw: calls.append(1) or attention(self, x, **kw))
    assert torch.equal(model(images), got) and len(calls) == 2
    assert pkg.ops.device_status() == 0


@torch.no_grad()
def test_a_bias_that_is_a_parameter(pkg, cuda_device):
    """An assigned Parameter is not among the module's buffers, where the native call looks."""
    for on_the_fly, name in ((True, "bias_tensor"), (False, "bias")):
        layer, gen = _packed_layer(pkg, 4, 192, 64, cuda_device, on_the_fly)
        x = torch.randn(50, 192, generator=gen).to(torch.float16 if on_the_fly else torch.float32).to(cuda_device)
        bias = getattr(layer, name)
        want = layer(x)
        delattr(layer, name)
        setattr(layer, name, torch.nn.Parameter(bias.clone()))
        assert name not in layer._buffers and torch.equal(layer(x), want)
    model, images = _small_model(pkg, "deit_tiny", 4, cuda_device)
    want = model(images)
    fc1 = model.blocks[0].mlp.fc1
    bias = fc1.bias_tensor
    del fc1.bias_tensor
    fc1.bias_tensor = torch.nn.Parameter(bias.clone())
    assert torch.equal(model(images), want)
    assert pkg.ops.device_status() == 0


def test_arguments_of_other_types_are_the_python_codes(pkg, cuda_device):
    cb, th = _codebook(torch.Generator().manual_seed(1), 4, cuda_device)
    x = torch.randn(8, 128, device=cuda_device)
    want = pkg.ops.quantize_activation(x, th, cb, 4, 64)
    for bits in (4.0, "4"):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            pkg.ops.quantize_activation(x, th, cb, bits, 64)
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            pkg.ops.dequant(*want, cb, bits, 64)
    for a, b in zip(pkg.ops.quantize_activation(x, th, cb, 4, 64, 1, 0), want):
        assert torch.equal(a, b)
    assert pkg.ops.quantize_activation(x, th, cb, 4, 64, False)[3] is None


@torch.no_grad()
def test_modes_and_subclasses_see_what_the_python_forward_shows_them(pkg, cuda_device):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            names.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))

    class Dispatched(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            names.append(str(func))
            return func(*args, **(kwargs or {}))

    class Image(torch.Tensor):
        pass

    model, images = _small_model(pkg, "deit_small", 4, cuda_device)
    want = model(images)
    names = []
    with Seen():
        assert torch.equal(model(images), want)
    assert names.count("scaled_dot_product_attention") == 2 and names.count("linear") == 2
    names = []
    with Dispatched():
        assert torch.equal(model(images), want)
    assert any("attention" in n for n in names)
    assert model._forward_native(images.as_subclass(Image)) is None
    assert torch.equal(model(images.as_subclass(Image)).as_subclass(torch.Tensor), want)
    with torch.device(cuda_device):                            # a default device is no reason to leave the native forward
        assert torch.equal(model._forward_native(images), want)


@torch.no_grad()
def test_other_threads_run_while_a_native_call_waits_for_the_gpu(pkg, cuda_device):
    """Calls pile up behind a busy GPU until the launch queue is full and the last one has to wait; another Python thread goes on
    meanwhile."""
    import threading
    import time
    model, images = _small_model(pkg, "deit_tiny", 4, cuda_device)
    layer = model.blocks[0].mlp.fc1
    rows = torch.randn(8, 192, device=cuda_device).half()
    for call in (lambda: model(images), lambda: layer(rows)):
        for _ in range(3):
            call()
        torch.cuda.synchronize()
        gaps, stop = [], threading.Event()

        def tick():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(0.001)
                now = time.perf_counter()
                gaps.append(now - last)
                last = now

        thread = threading.Thread(target=tick)
        thread.start()
        torch.cuda._sleep(1_500_000_000)                     # cycles: 0.8 s
        start = time.perf_counter()
        for _ in range(1500):
            call()
            if time.perf_counter() - start > 0.5:
                break
        waited = time.perf_counter() - start
        stop.set()
        thread.join()
        torch.cuda.synchronize()
        assert waited > 0.5 and max(gaps) < 0.25, (waited, max(gaps))
    assert pkg.ops.device_status() == 0


class _UnpackJob(ctypes.Structure):
    _fields_ = ([(n, ctypes.c_void_p) for n in ("packed", "mu", "sigma", "codesum", "codebook", "out")]
                + [("rows", ctypes.c_int64), ("K", ctypes.c_int64), ("bits", ctypes.c_int)])


@pytest.mark.parametrize("bits", [4, 3, 2])
@pytest.mark.parametrize("M", [0, 5])
def test_unpack_jobs_of_every_entry_point_run_whatever_the_rows(pkg, cuda_device, bits, M):
    lib, gen = pkg._cabi.load(), torch.Generator().manual_seed(bits)
    K, N, st = 384, 64, torch.cuda.current_stream().cuda_stream
    cb, th = _codebook(gen, bits, cuda_device)
    packed, mu, sg, cs = pkg.ops.quantize_activation(torch.randn(N, K, generator=gen).to(cuda_device), th, cb, bits, 64)
    want = pkg.ops.unpack_weight_f16(packed, mu, sg, cs, cb, bits, 64)
    x, h = torch.randn(M + 1, K, generator=gen).half().to(cuda_device), torch.empty(M + 1, K, dtype=torch.float16, device=cuda_device)
    one = torch.ones(K, device=cuda_device)

    def run(call):
        out = torch.zeros(N, K, dtype=torch.float16, device=cuda_device)
        job = _UnpackJob(*(t.data_ptr() for t in (packed, mu, sg, cs, cb, out)), N, K, bits)
        assert call(ctypes.addressof(job)) == 0
        assert torch.equal(out, want)

    p = [ctypes.c_void_p(t.data_ptr()) for t in (x, h, th, cb, one)]
    i64, vp = ctypes.c_int64, ctypes.c_void_p
    run(lambda j: lib.arcq_act_quant_unpack(0, p[0], 1, i64(M), i64(K), p[2], p[3], bits, 64, p[1], 1, 0, vp(j), 1, vp(st)))
    run(lambda j: lib.arcq_add_layernorm_act_quant_unpack(x.data_ptr(), None, one.data_ptr(), one.data_ptr(), 0, 1e-6, M, K, th.data_ptr(),
                                                          cb.data_ptr(), bits, 64, None, None, h.data_ptr(), 0, j, 1, st))
    run(lambda j: lib.arcq_dense_weight_gemm_unpack(p[0], vp(want.data_ptr()), None, i64(M), i64(N), i64(K), p[1], 1, vp(j), 1, vp(st)))
    assert pkg.ops.device_status() == 0


def test_gemm_layout_does_not_depend_on_the_first_question(pkg, cuda_device):
    """In a fresh process, whichever of the two forms of the pair GEMM is asked about first: the same room beside both."""
    code = ("import sys, ctypes; sys.path.insert(0, '.'); import __graft_entry__ as e, torch; torch.zeros(1, device='cuda')\n"
            "l = e.import_package()._cabi.load(); f = l.arcq_dense_weight_gemm_unpack_room; f.restype = ctypes.c_int64\n"
            "i = ctypes.c_int64\n"
            "print([f(i(m), i(n), i(k), q) for q in (%s) for m, n, k in ((12608, 1152, 384), (3000, 768, 3072), (12608, 3072, 768))])")
    rooms = [eval(subprocess.run([sys.executable, "-c", code % order], cwd=ROOT, capture_output=True, text=True, check=True).stdout)
             for order in ("0, 1", "1, 0")]
    assert rooms[0] == rooms[1][3:] + rooms[1][:3]
