"""The attention kernel between the qkv and proj linears and its form that also runs proj's activation quantizer: against an fp64
evaluation and the library kernel, and -- for the quantizer form -- bit for bit against the quantizer kernel applied to the plain
form's output.  Then where the modules take it, what they show of it, and where they take the library's attention."""
import subprocess
import sys

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from conftest import ROOT

pytestmark = pytest.mark.gpu


def _fp64(qkv, B, T, H):
    q = qkv.double().reshape(B, T, 3, H, 64).permute(2, 0, 3, 1, 4)
    s = (q[0] @ q[1].transpose(-1, -2)) / 8.0
    return (torch.softmax(s, -1) @ q[2]).transpose(1, 2).reshape(B * T, H * 64)


def _library(qkv, B, T, H):
    q = qkv.reshape(B, T, 3, H, 64).permute(2, 0, 3, 1, 4)
    return F.scaled_dot_product_attention(q[0], q[1], q[2]).transpose(1, 2).reshape(B * T, H * 64)


@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (1, 16, 1), (2, 197, 3), (3, 64, 2), (2, 200, 6), (1, 256, 2), (4, 5, 12),
                                   (16, 197, 6)])
def test_attention_kernel(pkg, oracle, cuda_device, B, T, H):
    gen = torch.Generator().manual_seed(B * 1000 + T + H)
    qkv = (torch.randn(B * T, 3 * H * 64, generator=gen) * 1.5).half().to(cuda_device)
    out = pkg.ops.attention(qkv, B, T, H)
    assert out.dtype == torch.float16 and tuple(out.shape) == (B * T, H * 64)
    ref = _fp64(qkv, B, T, H)
    err = float((out.double() - ref).abs().max())
    err_lib = float((_library(qkv, B, T, H).double() - ref).abs().max())
    assert err <= max(2.5e-3, 1.5 * err_lib), (err, err_lib)          # fp16 outputs of magnitude ~1-4
    # images do not see each other: the first image alone gives the same rows
    alone = pkg.ops.attention(qkv[:T].contiguous(), 1, T, H)
    assert torch.equal(alone, out[:T])
    for bits in (4, 3, 2):
        cb = torch.sort(torch.randn(2 ** bits, generator=gen) * 1.1)[0].to(cuda_device)
        th = (cb[:-1] + cb[1:]) / 2
        xq = pkg.ops.attention(qkv, B, T, H, th, cb, bits)
        want = pkg.ops.quantize_activation_dequant(out, th, cb, bits, 64, torch.float16)
        assert torch.equal(xq, want), bits
    # the quantizer form against the CPU oracle on the plain form's output (first rows)
    rows = slice(0, min(B * T, 24))
    cb = np.sort(np.random.default_rng(T).normal(size=16).astype(np.float32) * 1.1)
    th = ((cb[:-1] + cb[1:]) / np.float32(2)).astype(np.float32)
    xq = pkg.ops.attention(qkv, B, T, H, torch.from_numpy(th).to(cuda_device), torch.from_numpy(cb).to(cuda_device), 4)
    codes, mu, sg, cs = oracle.quantize(out[rows].float().cpu().numpy(), th, cb, 64)
    want = oracle.dequant(codes, mu, sg, cb, 64).astype(np.float16)
    assert np.array_equal(xq[rows].cpu().numpy(), want)
    assert pkg.ops.device_status() == 0


def test_attention_kernel_rejects_what_it_does_not_take(pkg, cuda_device):
    qkv = torch.zeros(300 * 2, 3 * 64, dtype=torch.float16, device=cuda_device)
    with pytest.raises(RuntimeError):
        pkg.ops.attention(qkv, 2, 300, 1)                 # more than 256 tokens
    with pytest.raises(RuntimeError):
        pkg.ops.attention(qkv, 3, 197, 1)                 # row count does not match


def test_model_with_the_attention_kernel(pkg, cuda_device):
    """The ViT skeleton with ``Attention.implementation = "kernel"``: attention and proj's quantizer in one launch.
    The first block's attention output equals the library's to fp16 rounding; whole-model logits stay finite and
    close (they differ like any two fp16 attention implementations do, amplified by the quantizers downstream)."""
    dev = cuda_device
    gen = torch.Generator().manual_seed(13)
    model = pkg.create_vit("deit_tiny", seed=3).half().to(dev)
    x = torch.randn(4, 3, 224, 224, generator=gen).half().to(dev)
    from importlib import import_module
    attn_cls = type(model.blocks[0].attn)
    saved = attn_cls.implementation
    try:
        with torch.no_grad():
            model = pkg.quantise_model(model, x, 4)
            attn_cls.implementation = "sdpa"
            y0 = model(x).clone()
            attn_cls.implementation = "kernel"
            y1 = model(x).clone()
            g1 = pkg.GraphedModel(model, x)(x).clone()
        assert torch.equal(y1, g1)
        assert bool(torch.isfinite(y1).all()) and pkg.ops.device_status() == 0
        rms = float(y0.float().pow(2).mean().sqrt())
        assert float((y1.float() - y0.float()).pow(2).mean().sqrt()) < 0.5 * rms
    finally:
        attn_cls.implementation = saved


@pytest.mark.parametrize("B,T,H", [(3, 17, 2), (2, 33, 1), (2, 128, 3), (2, 129, 3), (1, 144, 2), (1, 224, 1), (1, 225, 1), (2, 240, 2),
                                   (3, 255, 1), (130, 100, 3), (70, 197, 6)])
def test_attention_kernel_tile_edges(pkg, cuda_device, B, T, H):
    """Token counts around the edges of the products (multiples of 16), of the score pieces (32), of the query tiles (128) and of
    the tensor-memory layout, and more heads than blocks.  An output is a convex combination of fp16 values up to 8: rounding P and
    the output to fp16 gives at most 2^-11 of the largest value each, 2^-10 * 8 in all."""
    gen = torch.Generator().manual_seed(T)
    qkv = (torch.randn(B * T, 3 * H * 64, generator=gen) * 1.5).clamp(-8, 8).half().to(cuda_device)
    out = pkg.ops.attention(qkv, B, T, H)
    ref = _fp64(qkv, B, T, H)
    assert float((out.double() - ref).abs().max()) <= 8 * 2.0 ** -10
    # no further from 64 bits than the library's kernel, over the whole matrix
    err = [float((y.double() - ref).norm() / ref.norm()) for y in (out, _library(qkv, B, T, H))]
    assert err[0] <= 1.05 * err[1], err
    cb = torch.linspace(-2.5, 2.5, 8, device=cuda_device)
    th = (cb[:-1] + cb[1:]) / 2
    assert torch.equal(pkg.ops.attention(qkv, B, T, H, th, cb, 3), pkg.ops.quantize_activation_dequant(out, th, cb, 3, 64, torch.float16))
    assert pkg.ops.device_status() == 0


def test_attention_kernel_extreme_scores(pkg, cuda_device):
    """Large scores of one sign (nothing but the maximum may decide which exponentials survive), equal scores, and values that are
    not finite: like softmax in the library."""
    B, T, H = 2, 197, 1
    gen = torch.Generator().manual_seed(5)
    qkv = torch.randn(B * T, 192, generator=gen)
    qkv[:T, :64], qkv[:T, 64:128] = 30.0, -30.0 - torch.rand(T, 1, generator=gen)      # scores around -7200
    qkv[T:, :64] = 0.0                                                                # equal scores
    x = qkv.half().to(cuda_device)
    out, ref = pkg.ops.attention(x, B, T, H), _fp64(x, B, T, H)
    assert float((out.double() - ref).abs().max()) <= 8 * 2.0 ** -10
    x[3, 0] = float("nan")                                                            # one query: its row only
    x[T + 5, 70] = float("inf")                                                       # one key of the second image
    got, want = pkg.ops.attention(x, B, T, H), _library(x, B, T, H)
    assert torch.equal(got.isnan().any(1), want.isnan().any(1))
    assert torch.equal(got[4:T], out[4:T])
    assert pkg.ops.device_status() == 0


def test_chosen_back_ends_are_kept(pkg, cuda_device, monkeypatch):
    """A program that chooses among the library's attention back ends gets the one it chose: in the model's one call, in the Python
    forward and from the attention module alone."""
    gen = torch.Generator().manual_seed(14)
    model = pkg.create_vit("deit_tiny", seed=3).half().to(cuda_device)
    x = torch.randn(2, 3, 224, 224, generator=gen).half().to(cuda_device)
    tokens = torch.randn(2, 197, 192, generator=gen).half().to(cuda_device)
    attn = model.blocks[0].attn
    forward_native = pkg.vit.VisionTransformer._forward_native
    calls = (lambda: model(x), lambda: model(x), lambda: attn(tokens))
    with torch.no_grad():
        model = pkg.quantise_model(model, x, 4)
        for call, native in zip(calls, (True, False, False)):
            monkeypatch.setattr(pkg.vit.VisionTransformer, "_forward_native", forward_native if native else lambda self, x: None)
            own = call().clone()
            with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):
                chosen = call().clone()
                monkeypatch.setattr(type(attn), "implementation", "sdpa")
                want = call().clone()
                monkeypatch.setattr(type(attn), "implementation", "auto")
            assert torch.equal(chosen, want) and not torch.equal(chosen, own)


def _block(pkg, dev, name="deit_tiny", bits=4):
    """A packed block in a model of one, and input of its attention."""
    model = pkg.create_vit(name, seed=3)
    model.blocks = torch.nn.ModuleList(list(model.blocks)[:1])
    model = model.half().to(dev)
    gen = torch.Generator().manual_seed(14)
    images = torch.randn(2, 3, 224, 224, generator=gen).half().to(dev)
    with torch.no_grad():
        model = pkg.quantise_model(model, images, bits)
    return model, images, torch.randn(2, 197, model.embed_dim, generator=gen).half().to(dev)


@pytest.mark.parametrize("name,bits", [("deit_small", 4), ("deit_tiny", 3)])      # proj takes a reconstruction, and does not
@torch.no_grad()
def test_attention_of_nothing(pkg, cuda_device, name, bits):
    """No images, and no tokens."""
    model, _, x = _block(pkg, cuda_device, name, bits)
    attn = model.blocks[0].attn
    for empty in (x[:0], x[:, :0]):
        assert attn(empty).shape == empty.shape
    C = 64 * model.num_heads
    for quantizer in ((), (attn.proj.activation_thresholds, attn.proj.activation_codebook, bits)):
        assert pkg.ops.attention(x.new_empty(0, 3 * C), 0, 197, model.num_heads, *quantizer).shape == (0, C)
    assert pkg.ops.device_status() == 0


def _pre_hook(proj, seen, monkeypatch):
    proj.register_forward_pre_hook(lambda m, args, kwargs: seen.append((args, kwargs)), with_kwargs=True)


def _hook(proj, seen, monkeypatch):
    proj.register_forward_hook(lambda m, args, kwargs, y: seen.append((args, kwargs)), with_kwargs=True)


def _global_pre_hook(proj, seen, monkeypatch):
    module = torch.nn.modules.module
    monkeypatch.setattr(module, "_global_forward_pre_hooks", {0: lambda m, args: seen.append((args, {})) if m is proj else None})


def _own_forward(proj, seen, monkeypatch):
    proj.forward = lambda x: seen.append(((x,), {})) or type(proj).forward(proj, x)


def _class_forward(proj, seen, monkeypatch):
    forward = type(proj).forward
    monkeypatch.setattr(type(proj), "forward", lambda self, x: (seen.append(((x,), {})) if self is proj else None) or forward(self, x))


@pytest.mark.parametrize("watch", [_pre_hook, _hook, _global_pre_hook, _own_forward, _class_forward])
@torch.no_grad()
def test_what_watches_proj_sees_the_attention_output(pkg, cuda_device, watch, monkeypatch):
    """Hooks on proj, and a forward of its own that takes x only, get what the attention gives and nothing else; same bits."""
    model, images, x = _block(pkg, cuda_device)
    attn = model.blocks[0].attn
    want, seen = attn(x), []
    qkv = attn.qkv(x)
    watch(attn.proj, seen, monkeypatch)
    assert torch.equal(attn(x), want)
    (given,), kwargs = seen.pop()
    assert not kwargs and not seen
    C = 64 * model.num_heads
    assert torch.equal(given.reshape(-1, C), pkg.ops.attention(qkv.reshape(-1, 3 * C), 2, 197, model.num_heads))
    error = (given.reshape(-1, C).double() - _fp64(qkv.reshape(-1, 3 * C), 2, 197, model.num_heads)).abs().max()
    assert float(error) <= 2.0 ** -10 * float(qkv.abs().max())         # P and the output rounded to fp16


class _OnAttention(torch.overrides.TorchFunctionMode):
    """A function mode that knows the library's attention by identity and puts something in its place."""

    def __init__(self, instead):
        super().__init__()
        self.calls, self.instead = 0, instead

    def __torch_function__(self, func, types, args=(), kwargs=None):
        if func is F.scaled_dot_product_attention:
            self.calls += 1
            return self.instead(*args, **(kwargs or {}))
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("whole", [False, True])                   # the attention module, the model
@torch.no_grad()
def test_a_function_mode_sees_and_replaces_the_attention(pkg, cuda_device, whole, monkeypatch):
    model, images, x = _block(pkg, cuda_device)
    call = (lambda: model(images)) if whole else (lambda: model.blocks[0].attn(x))
    want = call()
    sdpa = F.scaled_dot_product_attention
    with _OnAttention(sdpa) as seen:
        assert torch.equal(call(), want) and seen.calls == 1
    cls = type(model.blocks[0].attn)
    for instead in (lambda q, k, v: torch.zeros_like(q), lambda q, k, v: sdpa(q, k, v, is_causal=True), lambda q, k, v: sdpa(q, k, q),
                    lambda q, k, v: sdpa(q, k, v, scale=0.5), lambda q, k, v: torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v):
        results = []
        for implementation in ("auto", "sdpa"):
            monkeypatch.setattr(cls, "implementation", implementation)
            with _OnAttention(instead) as seen:
                results.append(call())
            assert seen.calls == 1
        assert torch.equal(*results) and not torch.equal(results[0], want)
    assert pkg.ops.device_status() == 0


@torch.no_grad()
def test_a_dispatch_mode_sees_the_attention_operator(pkg, cuda_device):
    """By the framework's own name: its counter of operations knows it.  Same bits, also in inference mode."""
    from torch.utils.flop_counter import FlopCounterMode
    model, _, x = _block(pkg, cuda_device)
    attn = model.blocks[0].attn
    want = attn(x)
    with FlopCounterMode(display=False) as counter:
        assert torch.equal(attn(x), want)
    assert counter.get_total_flops() == 4 * 2 * model.num_heads * 197 * 197 * 64
    with torch.inference_mode(), FlopCounterMode(display=False):
        assert torch.equal(attn(x), want)
    with torch.autocast("cuda", torch.float16), FlopCounterMode(display=False):
        assert torch.equal(attn(x), want)
    assert pkg.ops.device_status() == 0


_BACK_ENDS = ("MATH", "EFFICIENT_ATTENTION", "FLASH_ATTENTION", "CUDNN_ATTENTION")


# the slowest first; the order that the framework starts with and leaves when it is first asked for a back end
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (2, 1, 0, 3)])
@pytest.mark.parametrize("native", [True, False])
@torch.no_grad()
def test_a_set_order_of_the_back_ends_is_kept(pkg, cuda_device, native, order, monkeypatch):
    """All four back ends in an order of the program's: the library's attention runs, in the model's one call and in the attention
    module."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    model, images, _ = _block(pkg, cuda_device)
    if not native:
        monkeypatch.setattr(pkg.vit.VisionTransformer, "_forward_native", lambda self, x: None)
    own = model(images)
    monkeypatch.setattr(type(model.blocks[0].attn), "implementation", "kernel")
    assert torch.equal(model(images), own)                      # the library has run by now, in the calibration
    monkeypatch.setattr(type(model.blocks[0].attn), "implementation", "auto")
    with sdpa_kernel([getattr(SDPBackend, _BACK_ENDS[i]) for i in order], set_priority=True):
        chosen = model(images)
        monkeypatch.setattr(type(model.blocks[0].attn), "implementation", "sdpa")
        assert torch.equal(chosen, model(images)) and not torch.equal(chosen, own)
    assert pkg.ops.device_status() == 0


def test_the_order_of_a_fresh_process_is_no_choice(cuda_device):
    """Before the library's attention has run, and after."""
    code = """
import sys; sys.path.insert(0, '.')
import torch, __graft_entry__ as entry
from torch.nn.attention import SDPBackend as B, sdpa_kernel
untouched = entry.import_package()._cabi.host().attention_back_ends_as_they_come
assert untouched()
with sdpa_kernel([B.FLASH_ATTENTION, B.EFFICIENT_ATTENTION, B.MATH, B.CUDNN_ATTENTION], set_priority=True):
    assert not untouched()
q = torch.randn(1, 1, 8, 64, device='cuda').half()
torch.nn.functional.scaled_dot_product_attention(q, q, q)
assert untouched()
"""
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)


@torch.no_grad()
def test_qkv_that_the_kernel_cannot_read_in_place(pkg, cuda_device):
    """A hook that gives back qkv two bytes off, and one with a gap between its rows: read from a copy, same bits."""
    model, _, x = _block(pkg, cuda_device)
    attn = model.blocks[0].attn
    want = attn(x)

    def off(m, args, y):
        return torch.empty(y.numel() + 1, dtype=y.dtype, device=y.device)[1:].reshape(y.shape).copy_(y)

    def gap(m, args, y):
        return torch.empty(*y.shape[:-1], y.shape[-1] + 3, dtype=y.dtype, device=y.device)[..., :-3].copy_(y)

    for hook in (off, gap):
        handle = attn.qkv.register_forward_hook(hook)
        assert torch.equal(attn(x), want)
        handle.remove()
    assert pkg.ops.device_status() == 0


@torch.no_grad()
def test_a_graph_of_operators_has_the_librarys_attention(pkg, cuda_device, monkeypatch):
    model, _, x = _block(pkg, cuda_device)
    attn = model.blocks[0].attn
    got = torch.compile(attn, backend="eager")(x)
    monkeypatch.setattr(type(attn), "implementation", "sdpa")
    assert torch.equal(got, attn(x))
    assert pkg.ops.device_status() == 0


def test_probabilities_are_divided_by_a_correctly_rounded_sum(pkg, cuda_device):
    """Equal scores: every probability before the division is one and the sum is T.  The values are halfway between two fp16 numbers
    times T, in two summands that fp16 holds, so which way an output is rounded depends on the last bit of 1 / T in fp32."""
    gen = torch.Generator().manual_seed(3)
    for T in range(2, 257):
        half = (2048 + 2 * torch.randint(0, 1024, (64,), generator=gen) + 1).float() / 2048       # twelve bits, in [1, 2)
        qkv = torch.zeros(T, 192)
        qkv[0, 128:] = (half * T).half().float()
        qkv[1, 128:] = half * T - qkv[0, 128:]
        assert torch.equal(qkv.half().float(), qkv)
        want = ((half * T) * torch.tensor(T, dtype=torch.float32).reciprocal()).half()
        got = pkg.ops.attention(qkv.half().to(cuda_device), 1, T, 1).cpu()
        assert torch.equal(got, want.expand(T, 64)), T
    assert pkg.ops.device_status() == 0


@pytest.mark.parametrize("B,T", [(1, 17), (1, 197), (200, 197)])       # one item, two of a head, several blocks an SM and heads a block
def test_waits_of_the_attention_kernel_that_run_out(pkg, cuda_device, B, T):
    """With no polls every warp gives up at its first wait: the kernel ends and leaves its code in the status word, and the next launch
    is none the worse."""
    H = 3
    qkv = torch.randn(B * T, 3 * H * 64, generator=torch.Generator().manual_seed(T)).half().to(cuda_device)
    want = pkg.ops.attention(qkv, B, T, H)
    cb = torch.linspace(-2.5, 2.5, 16, device=cuda_device)
    for quantizer in ((), ((cb[:-1] + cb[1:]) / 2, cb, 4)):
        with pkg._cabi.option("ARCQ_POLL_LIMIT", 0):
            pkg.ops.attention(qkv, B, T, H, *quantizer)
        assert pkg.ops.device_status() == 0x501
        assert pkg.ops.device_status() == 0
    assert torch.equal(pkg.ops.attention(qkv, B, T, H), want)
    assert pkg.ops.device_status() == 0


@pytest.mark.parametrize("polls", [1, 2, 4, 8])
@pytest.mark.parametrize("B,T", [(1, 17), (1, 197), (200, 197)])
def test_waits_of_some_warps_that_run_out(pkg, cuda_device, polls, B, T):
    """A few polls: some warps' waits run out and others' do not.  The kernel ends, a result that is not the whole one has left its code,
    and the next launch is none the worse."""
    H = 3
    qkv = torch.randn(B * T, 3 * H * 64, generator=torch.Generator().manual_seed(T)).half().to(cuda_device)
    cb = torch.linspace(-2.5, 2.5, 16, device=cuda_device)
    for quantizer in ((), ((cb[:-1] + cb[1:]) / 2, cb, 4)):
        want = pkg.ops.attention(qkv, B, T, H, *quantizer)
        for _ in range(5):
            with pkg._cabi.option("ARCQ_POLL_LIMIT", polls):
                got = pkg.ops.attention(qkv, B, T, H, *quantizer)
            status = pkg.ops.device_status()
            assert status in (0, 0x501) and (status != 0 or torch.equal(got, want))
        assert torch.equal(pkg.ops.attention(qkv, B, T, H, *quantizer), want)
    assert pkg.ops.device_status() == 0


@torch.no_grad()
def test_auto_is_the_kernel_between_packed_linears(pkg, cuda_device, monkeypatch):
    model, images, x = _block(pkg, cuda_device, "deit_small")
    attn = model.blocks[0].attn
    got = [attn(x), model(images), model._forward_native(images)]
    monkeypatch.setattr(type(attn), "implementation", "kernel")
    assert model._forward_native(images) is None
    for y, want in zip(got, (attn(x), model(images), model(images))):
        assert torch.equal(y, want)
    monkeypatch.setattr(type(attn), "implementation", "sdpa")
    assert not torch.equal(got[0], attn(x))


def _replaced(attn, monkeypatch):
    library = F.scaled_dot_product_attention
    monkeypatch.setattr(F, "scaled_dot_product_attention", lambda *a, **k: library(*a, **k))


def _asks_for_gradients(attn, monkeypatch):
    attn.qkv = torch.nn.Linear(192, 576).half().to(attn.qkv.packed_weight_codes.device)


def _autocast(attn, monkeypatch):
    """Entered around the call."""


@pytest.mark.parametrize("why", [_replaced, _asks_for_gradients, _autocast])
def test_where_the_library_attention_stays(pkg, cuda_device, why, monkeypatch):
    """A function in its place, a qkv that wants a gradient, autocast to another type: bit for bit the library's route."""
    model, _, x = _block(pkg, cuda_device)
    attn = model.blocks[0].attn
    why(attn, monkeypatch)
    results = []
    for implementation in ("auto", "sdpa"):
        monkeypatch.setattr(type(attn), "implementation", implementation)
        with torch.autocast("cuda", torch.bfloat16, enabled=why is _autocast), torch.set_grad_enabled(why is _asks_for_gradients):
            results.append(attn(x).detach())
    assert torch.equal(*results)
    monkeypatch.undo()
    with torch.no_grad():
        assert not torch.equal(attn(x), results[0])              # without the reason: the kernel
    assert pkg.ops.device_status() == 0


# one to six items a block (both halves of tensor memory in turn), heads of one and of two query tiles, splits of the keys for the two
# threads of a row: all of them lower, uneven, even, the longest
@pytest.mark.parametrize("B,T,H", [(1, 5, 1), (150, 17, 1), (40, 33, 5), (75, 64, 6), (30, 100, 12), (150, 129, 1), (40, 197, 12), (60, 240, 6), (37, 256, 12)])
def test_items_of_a_block_one_after_the_other(pkg, cuda_device, B, T, H):
    gen = torch.Generator(device=cuda_device).manual_seed(B + T + H)
    qkv = torch.randn(B * T, 3 * H * 64, generator=gen, device=cuda_device).half()
    out = pkg.ops.attention(qkv, B, T, H)
    q, k, v = qkv.double().view(B, T, 3, H, 64).permute(2, 0, 3, 1, 4)
    want = (torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v).transpose(1, 2).reshape(B * T, H * 64)
    # probabilities rounded to fp16 (2^-11 of each, times |v| < 6), the output's own rounding, fp32 sums of T terms
    assert float((out.double() - want).abs().max()) <= 6 * 2.0 ** -11 + 2.0 ** -11 * float(want.abs().max()) + T * 6 * 2.0 ** -22
    part = pkg.ops.attention(qkv[-T:].contiguous(), 1, T, H)              # the last image on its own: other blocks, other halves
    assert torch.equal(part, out[-T:])
    assert pkg.ops.device_status() == 0
