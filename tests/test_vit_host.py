"""ViT skeleton and the CPU whole-model oracle (no GPU)."""
import pytest
import torch

from oracle.fakequant_vit import OracleViT


def test_skeleton_names_and_sizes(pkg):
    m = pkg.create_vit("deit_small", seed=0)
    names = pkg.quantised_linear_names(m)
    assert len(names) == 48 and names[:4] == ["blocks.0.attn.qkv", "blocks.0.attn.proj", "blocks.0.mlp.fc1",
                                             "blocks.0.mlp.fc2"]
    sd = m.state_dict()
    assert tuple(sd["blocks.3.attn.qkv.weight"].shape) == (1152, 384)
    assert tuple(sd["blocks.3.mlp.fc1.weight"].shape) == (1536, 384)
    assert tuple(sd["pos_embed"].shape) == (1, 197, 384) and tuple(sd["head.weight"].shape) == (1000, 384)
    n_q = sum(sd[n + ".weight"].numel() for n in names)
    assert n_q == 21_233_664                      # quantised weights of DeiT-S
    same = pkg.create_vit("deit_small", seed=0).state_dict()
    assert all(torch.equal(sd[k], same[k]) for k in sd)


def test_oracle_vit_is_deterministic_and_batch_invariant(pkg):
    m = pkg.create_vit("deit_tiny", seed=1)
    dim, heads, depth = pkg.DEIT_CONFIGS["deit_tiny"]
    o = OracleViT(m.state_dict(), dim, heads, 2, bits=4)     # two blocks keep the CPU suite short
    x = torch.randn(4, 3, 224, 224, generator=torch.Generator().manual_seed(2))
    o(x)                                                      # calibrates
    cap = {}
    y = o(x, cap)
    assert torch.equal(y, o(x))
    halves = torch.cat([o(x[:2]), o(x[2:])])
    assert torch.allclose(y, halves, atol=1e-5)
    assert set(cap) == set(o.layer_names()) and cap["blocks.1.mlp.fc2"]["x"].shape == (4 * 197, 768)
    cb = o.codebooks["blocks.0.attn.qkv"]["act_cb"]
    assert cb.shape == (16,) and (cb == 0).sum() == 1


def _packed_on_cpu(pkg, blocks=2):
    m = pkg.create_vit("deit_tiny", seed=1)
    m.blocks = torch.nn.ModuleList(list(m.blocks)[:blocks])
    cb = torch.linspace(-2.6, 2.6, 16)
    th = (cb[:-1] + cb[1:]) / 2
    return pkg.pack_model_with_codebooks(m, {n: dict(act_cb=cb, act_th=th, w_cb=cb, w_th=th) for n in pkg.quantised_linear_names(m)}, 4)


def _own(self, x, **kw):
    return type(self).forward(self, x, **kw)


CHANGES = {
    "eps of a block's norm": lambda m: setattr(m.blocks[1].norm2, "eps", 1e-3),
    "eps of the last norm": lambda m: setattr(m.norm, "eps", 1e-3),
    "attention's forward": lambda m: setattr(m.blocks[0].attn, "forward", _own.__get__(m.blocks[0].attn)),
    "mlp's forward": lambda m: setattr(m.blocks[1].mlp, "forward", _own.__get__(m.blocks[1].mlp)),
    "a linear's forward": lambda m: setattr(m.blocks[1].mlp.fc1, "forward", _own.__get__(m.blocks[1].mlp.fc1)),
    "patch embedding's forward": lambda m: setattr(m.patch_embed, "forward", _own.__get__(m.patch_embed)),
    "head's forward": lambda m: setattr(m.head, "forward", _own.__get__(m.head)),
    "weight form": lambda m: setattr(m.blocks[0].attn.proj, "weight_form", "packed"),
    "attention form": lambda m: setattr(m.blocks[0].attn, "implementation", "kernel"),
    "heads": lambda m: setattr(m.blocks[0].attn, "num_heads", 4),
    "a block less": lambda m: m.blocks.__delitem__(1),
    "a block more": lambda m: m.blocks.append(m.blocks[0]),
    "another module": lambda m: setattr(m, "head", torch.nn.Linear(192, 1000)),
}
STILL_NATIVE = ("eps", "a block", "another module")


@pytest.mark.parametrize("what", CHANGES)
def test_plan_of_the_native_forward_is_void_once_the_model_changes(pkg, what):
    """The check comes before everything that needs a GPU: False for a void plan, None for an input that is not taken."""
    m, x = _packed_on_cpu(pkg), torch.zeros(1, 3, 224, 224)
    host = pkg._cabi.host()
    plan = pkg.vit._make_plan(m)
    assert not callable(plan) and host.vit_forward(plan, x) is None
    CHANGES[what](m)
    assert host.vit_forward(plan, x) is False
    plan = pkg.vit._make_plan(m)
    if what.startswith(STILL_NATIVE):
        assert not callable(plan) and host.vit_forward(plan, x) is None
    else:
        assert callable(plan) and plan()                      # refused, for a reason that holds


def test_a_model_that_was_refused_is_looked_at_again(pkg):
    m, x = _packed_on_cpu(pkg), torch.zeros(1, 3, 224, 224)
    CHANGES["mlp's forward"](m)
    why = pkg.vit._make_plan(m)
    assert callable(why) and why()
    del m.blocks[1].mlp.forward
    assert not why() and not callable(pkg.vit._make_plan(m))
    handle = m.blocks[0].attn.register_forward_hook(lambda *a: None)
    plan = pkg.vit._make_plan(m)                              # hooks decline a call, they do not void the plan
    assert pkg._cabi.host().vit_forward(plan, x) is None
    handle.remove()
    assert pkg._cabi.host().vit_forward(plan, x) is None
