"""The work a user of this package has it do, as cases that can be timed and compared.

A case is a dict of plain values.  Its ``kind`` says which public entry point it goes through:

* ``graph``   a packed DeiT behind ``GraphedModel`` (serving loop with a fixed batch shape, inputs in device memory)
* ``eager``   the same model called as a module (a host program that swapped the packed linears in and kept its own loop)
* ``host``    the same model behind ``HostPipeline``: pinned host batches in, logits in host memory out
* ``linear``  one packed linear called as a module: ``chain`` "half" is ``ARCQPackedLinearOnTheFly`` (fp16 in and out),
              "float" is ``ARCQPackedLinear`` (fp32 out, packed activation codes in between)
* ``codec``   the activation codec alone: ``quantize_activation`` (packed codes and statistics) and ``dequant`` back

Models, widths, code widths and batch sizes are those of this repository's benchmark and tests: DeiT-Tiny / Small / Base at
224 x 224 (197 tokens), 4- and 3-bit codes (2-bit in the operators too), group size 64, random-init weights.  Images have
the make-up of normalised photographs (a colour cast, soft structure, some noise); a layer's inputs are normal with a few
channels 20 times as large as the rest.
"""
from __future__ import annotations

import math

import torch

import __graft_entry__ as entry

TOKENS, PATCH_COLS, CLASSES, GROUP = 197, 3 * 16 * 16, 1000, 64
WIDTH = {"deit_tiny": 192, "deit_small": 384, "deit_base": 768}
DEPTH = 12
HOST_BATCHES = 4
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
# (K, N) of qkv, proj, fc1 and fc2 for a model width
LAYERS = [lambda d: (d, 3 * d), lambda d: (d, d), lambda d: (d, 4 * d), lambda d: (4 * d, d)]


def listed():
    return [
        # one image at a time: an interactive request, all launches and latency
        dict(name="small w4 graph b1", kind="graph", model="deit_small", bits=4, batch=1),
        # the benchmark's batch
        dict(name="small w4 graph b64", kind="graph", model="deit_small", bits=4, batch=64),
        # 3-bit codes (rows that do not end on a byte boundary of a code)
        dict(name="small w3 graph b64", kind="graph", model="deit_small", bits=3, batch=64),
        # the narrow model, 3-bit packed rows of 72 bytes, and a last batch of a data set that is not full
        dict(name="tiny w3 graph b37", kind="graph", model="deit_tiny", bits=3, batch=37),
        # the wide model with the whole global batch of the benchmark on one GPU: the largest call
        dict(name="base w4 graph b1024", kind="graph", model="deit_base", bits=4, batch=1024),
        # modules called from a Python loop without a graph: host work and launches count
        dict(name="small w4 eager b8", kind="eager", model="deit_small", bits=4, batch=8),
        # images and logits in host memory, four batches through the double-buffered runner
        dict(name="small w4 host b64", kind="host", model="deit_small", bits=4, batch=64),
        # a single layer, the smallest call: one image through proj of the narrow model
        dict(name="linear half w4 197x192x192", kind="linear", chain="half", bits=4, M=197, K=192, N=192),
        # a single layer with a long reduction (fc2 of the wide model), a ragged number of rows
        dict(name="linear half w4 3001x3072x768", kind="linear", chain="half", bits=4, M=3001, K=3072, N=768),
        # the fp32 layer of the reference's extension path at the size of its unit workload (8 images, fc1)
        dict(name="linear float w4 1576x384x1536", kind="linear", chain="float", bits=4, M=1576, K=384, N=1536),
        # the fp32 layer with 3-bit rows of 72 bytes, a full batch
        dict(name="linear float w3 12608x192x576", kind="linear", chain="float", bits=3, M=12608, K=192, N=576),
        # encode and decode of an activation matrix that is kept packed in between
        dict(name="codec w4 f32 12608x384", kind="codec", bits=4, M=12608, K=384, dtype="f32"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choices(["graph", "eager", "host", "linear", "codec"], [0.4, 0.12, 0.08, 0.3, 0.1])[0]
    if kind in ("graph", "eager", "host"):
        model = rng.choices(["deit_tiny", "deit_small", "deit_base"], [0.25, 0.45, 0.3])[0]
        hi = {"graph": 256, "eager": 64, "host": 128}[kind]
        return dict(kind=kind, model=model, bits=rng.choice([4, 4, 3]), batch=_log_int(rng, 1, hi))
    if kind == "linear":
        K, N = rng.choice(LAYERS)(rng.choice([192, 384, 768]))
        return dict(kind=kind, chain=rng.choice(["half", "half", "float"]), bits=rng.choice([4, 4, 3, 2]),
                    M=_log_int(rng, 1, 128 * TOKENS), K=K, N=N)
    return dict(kind=kind, bits=rng.choice([4, 4, 3, 2]), M=_log_int(rng, 1, 128 * TOKENS),
                K=64 * rng.choice([1, 3, 6, 12, 24, 48, rng.randint(1, 48)]), dtype=rng.choice(["f32", "f16", "bf16"]))


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(gen, M, K, dtype):
    x = torch.randn(M, K, generator=gen, device="cuda")
    x[:, torch.randperm(K, generator=gen, device="cuda")[:4]] *= 20.0
    return x.to(dtype)


def _images(gen, batch):
    x = torch.randn(batch, 3, 224, 224, generator=gen, device="cuda") * 0.2
    x += torch.randn(batch, 3, 1, 1, generator=gen, device="cuda")
    soft = torch.randn(batch, 3, 7, 7, generator=gen, device="cuda") * 0.7
    return (x + torch.nn.functional.interpolate(soft, size=(224, 224), mode="bilinear")).half()


def _model(pkg, case, seed, gen):
    """Random-init DeiT, packed, its codebooks fitted on a few images and frozen: what a serving program loads once.
    The class token and the positions get the size they have in trained models, large against what one block adds:
    with both at 0.02 the logits are all branch noise, and one rounding difference moves them by a quarter of their size
    through the codes that flip behind it (with 3 bits by half)."""
    model = pkg.create_vit(case["model"], seed=seed).half().cuda()
    size = WIDTH[case["model"]] / 80 * (1.5 if case["bits"] == 3 else 1)
    with torch.no_grad():
        model.cls_token.normal_(0.0, size, generator=gen)
        model.pos_embed.normal_(0.0, size / 4, generator=gen)
        return pkg.quantise_model(model, _images(gen, min(case["batch"], 8)), case["bits"])


def prepare(case, seed):
    pkg = entry.import_package()
    gen = _generator(seed)
    kind = case["kind"]
    if kind in ("graph", "eager", "host"):
        model = _model(pkg, case, seed, gen)
        if kind == "eager":
            return dict(kind=kind, model=model, x=_images(gen, case["batch"]))
        x = _images(gen, case["batch"])
        runner = pkg.GraphedModel(model, x)
        if kind == "graph":
            return dict(kind=kind, model=model, runner=runner, x=x)
        host = [_images(gen, case["batch"]).cpu().pin_memory() for _ in range(HOST_BATCHES)]
        return dict(kind=kind, model=model, pipe=pkg.HostPipeline(runner, host[0], (case["batch"], CLASSES)), host=host)
    if kind == "linear":
        M, K, N = case["M"], case["K"], case["N"]
        x = _activations(gen, M, K, torch.float16 if case["chain"] == "half" else torch.float32)
        linear = torch.nn.Linear(K, N, device="cuda")
        with torch.no_grad():
            linear.weight.normal_(0.0, 0.02, generator=gen)
            linear.bias.normal_(0.0, 0.01, generator=gen)
        cb, th = pkg.codebook.calibrate_codebook(_activations(gen, 256, K, torch.float32), case["bits"], GROUP)
        layer = pkg.pack_linear(linear, case["bits"], cb, th, group_size=GROUP, on_the_fly=case["chain"] == "half")
        return dict(kind=kind, layer=layer, x=x)
    x = _activations(gen, case["M"], case["K"], DTYPES[case["dtype"]])
    cb, th = pkg.codebook.calibrate_codebook(_activations(gen, 256, case["K"], torch.float32), case["bits"], GROUP)
    return dict(kind=kind, ops=pkg.ops, x=x, cb=cb, th=th, bits=case["bits"])


# ------------------------------------------------------------------------------------------------ one pass
@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "graph":
        return state["runner"](state["x"])
    if kind == "eager":
        return state["model"](state["x"])
    if kind == "host":
        logits = []
        state["pipe"].run(state["host"], on_result=lambda t: logits.append(t.clone()))
        return logits
    if kind == "linear":
        return state["layer"](state["x"])
    ops, bits = state["ops"], state["bits"]
    packed, center, scale, code_sum = ops.quantize_activation(state["x"], state["th"], state["cb"], bits, GROUP)
    return packed, center, scale, code_sum, ops.dequant(packed, center, scale, code_sum, state["cb"], bits, GROUP)


# ------------------------------------------------------------------------------------------------ what it cannot do without
def _linear_work(M, K, N, bits, x_bytes, y_bytes):
    weight = N * K * bits / 8 + 12 * N * K / GROUP + 4 * N
    return M * K * x_bytes + weight + M * N * y_bytes, 2.0 * M * N * K


def work(case):
    kind, bits = case["kind"], case["bits"]
    if kind in ("graph", "eager", "host"):
        d, batches = WIDTH[case["model"]], HOST_BATCHES if kind == "host" else 1
        images = case["batch"] * batches
        weights = sum(_linear_work(0, *layer(d), bits, 2, 2)[0] for layer in LAYERS) * DEPTH
        weights += 2 * (PATCH_COLS * d + d * CLASSES + (TOKENS + 2) * d + 4 * DEPTH * d)
        flops = sum(_linear_work(TOKENS, *layer(d), bits, 2, 2)[1] for layer in LAYERS) * DEPTH
        flops += DEPTH * 4.0 * TOKENS * TOKENS * d                     # q k^T and p v over all heads
        flops += 2.0 * (TOKENS - 1) * PATCH_COLS * d + 2.0 * d * CLASSES
        return {"bytes": weights * batches + images * (3 * 224 * 224 * 2 + CLASSES * 2), "flops": images * flops}
    M, K = case["M"], case["K"]
    if kind == "linear":
        half = case["chain"] == "half"
        b, f = _linear_work(M, K, case["N"], bits, 2 if half else 4, 2 if half else 4)
        return {"bytes": b, "flops": f}
    packed = M * K * bits / 8 + 12 * M * K / GROUP
    return {"bytes": M * K * DTYPES[case["dtype"]].itemsize + packed + 2 * M * K, "flops": 12.0 * M * K}


def tolerance(case):
    if case["kind"] in ("graph", "eager", "host"):
        # 48 layers re-quantise to 3 or 4 bits: where an fp16 rounding differs, codes flip, and the logits of two correct
        # implementations (library and own attention, say) lie 0.5 to 1.5 % apart; those of two images 3 to 15 %
        return {"rel": 2.5e-2, "max": 0.25}
    return {"rel": 1e-3 if case["kind"] == "codec" else 2e-3}
