"""What surrounds the attention kernel on the host, with a stand-in for the library: no GPU."""
import contextlib
import subprocess
import sys
import types

import pytest
import torch
from torch.nn.attention import SDPBackend, sdpa_kernel

from conftest import ROOT


@pytest.mark.parametrize("quantise", [False, True])
def test_attention_launches_on_the_device_of_its_tensors(pkg, monkeypatch, quantise):
    """The stand-in records the device that is current when the kernel is launched and the one whose stream it is given."""
    current, launches = ["the current device"], []

    @contextlib.contextmanager
    def device(d):
        current.append(d)
        yield
        current.pop()

    def launch(*args):
        launches.append((current[-1], args[-1]))
        return 0

    ops = pkg.ops
    monkeypatch.setattr(ops, "_dev", lambda t, *_: t.contiguous())
    monkeypatch.setattr(ops, "_stream", lambda: ("stream of", current[-1]))
    monkeypatch.setattr(ops._cabi, "load", lambda: types.SimpleNamespace(arcq_attention=launch, arcq_attention_act_quant=launch))
    monkeypatch.setattr(torch.cuda, "device", device)
    qkv = torch.zeros(2 * 5, 3 * 64, dtype=torch.float16)
    out = ops.attention(qkv, 2, 5, 1, *((torch.zeros(15), torch.zeros(16)) if quantise else ()))
    assert launches == [(qkv.device, ("stream of", qkv.device))] and current == ["the current device"]
    assert out.shape == (10, 64)


def test_an_empty_batch_is_nothing_to_do(pkg):
    """Tensors of an empty batch have null pointers; null pointers of any other batch, and bad shapes of an empty one, are refused."""
    lib, some = pkg._cabi.load(), 16
    assert lib.arcq_attention(None, 0, 197, 3, 64, None, None) == 0
    assert lib.arcq_attention_act_quant(None, 0, 197, 3, 64, some, some, 4, 64, None, None) == 0
    for args in ((None, 1, 197, 3, 64, None, None), (some, 1, 197, 3, 64, None, None), (None, 0, 0, 3, 64, None, None),
                 (None, 0, 257, 3, 64, None, None), (None, 0, 197, 3, 32, None, None)):
        assert lib.arcq_attention(*args) < 0
    assert lib.arcq_attention_act_quant(None, 0, 197, 3, 64, None, some, 4, 64, None, None) < 0


def test_a_choice_among_the_librarys_back_ends_is_noticed(pkg):
    """A back end left out, or all of them in an order of the program's own."""
    untouched = pkg._cabi.host().attention_back_ends_as_they_come
    every = [SDPBackend.FLASH_ATTENTION, SDPBackend.EFFICIENT_ATTENTION, SDPBackend.MATH, SDPBackend.CUDNN_ATTENTION]
    assert untouched()
    for i in range(4):
        with sdpa_kernel(every[:i] + every[i + 1:]):
            assert not untouched()
    with sdpa_kernel(every[::-1], set_priority=True):
        assert not untouched()
    with sdpa_kernel(every):
        assert untouched()
    with sdpa_kernel(every[3:] + every[:3], set_priority=True):     # what the framework settles on
        assert untouched()
    assert untouched()


def test_an_attention_put_in_the_librarys_place_before_the_import_is_noticed():
    """By the attention module and by the native forward, whose reasons not to run are looked at in this order."""
    code = """
import sys; sys.path.insert(0, '.')
import torch, torch.nn.functional as F
library = F.scaled_dot_product_attention
F.scaled_dot_product_attention = lambda *a, **k: library(*a, **k)
import __graft_entry__ as entry
vit = entry.import_package().vit
def differs(): return [n for c, n, f in vit._STANDS_FOR if getattr(c, n) is not f], F.scaled_dot_product_attention is vit._LIBRARY_ATTENTION
assert differs() == (['scaled_dot_product_attention'], False), differs()
F.scaled_dot_product_attention = library
assert differs() == ([], True), differs()
"""
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)


def test_a_block_can_be_traced_symbolically(pkg):
    """A tracer's proxies are asked nothing that has no answer yet."""
    block = pkg.vit.Block(128, 2)
    x = torch.randn(2, 5, 128, generator=torch.Generator().manual_seed(1))
    graph = torch.fx.symbolic_trace(block)
    assert any(n.target is torch.nn.functional.scaled_dot_product_attention for n in graph.graph.nodes)
    assert torch.equal(graph(x), block(x))
