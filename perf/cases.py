"""The work that users of this package have it do, as cases that can be timed and compared.

A case goes through the public entry points only: `tx.step` of the optimizers (eager with and without donated
buffers, behind global-norm clipping, and captured in a CUDA graph), `reconstruct_weights` / `set_fp32_params`
(checkpoint export and import) and the moment codecs.  Shapes are those of the configurations the package is
benchmarked and tested on (square matrices with their bias, the ResNet-50, GPT-2-small and Llama-3-8B pytrees)
and scaled relatives of them.
"""

from __future__ import annotations

import math

import torch

import flashoptim_jax_b200 as fo
from flashoptim_jax_b200 import clipping, schedules
from flashoptim_jax_b200 import tree as pytree

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
FACTORY = {"adam": fo.flash_adam, "adamw": fo.flash_adamw, "lion": fo.flash_lion, "sgd": fo.flash_sgd, "sgdw": fo.flash_sgdw}
# learning rate and weight decay of the benchmark's configurations
HPARAMS = {"adam": dict(learning_rate=1e-3, weight_decay=0.0), "adamw": dict(learning_rate=1e-3, weight_decay=1e-2),
           "lion": dict(learning_rate=1e-4, weight_decay=1e-2), "sgd": dict(learning_rate=1e-2, momentum=0.9, nesterov=True),
           "sgdw": dict(learning_rate=1e-2, momentum=0.9, weight_decay=1e-2)}
MAX_PARAMS = 1_500_000_000  # of a drawn case; below the largest listed one


def _step(tree, opt, **more):
    case = {"what": "step", "tree": tree, "opt": opt, "dtype": "bf16", "grads": "bf16", "bits": 24, "quantize": True, "group": 32,
            "fused": True, "donate": True, "graph": False, "clip": False}
    case.update(more)
    return case


def listed():
    return [
        # one layer's matrix and bias at the smallest size of the reference's step benchmark: latency of a call
        dict(_step("square", "adamw", rows=256, cols=256, grads="f32"), name="adamw_256"),
        # an odd-shaped fp16 matrix under Lion (fp16 mixed precision): ragged ends, rows that are no multiple of a group
        dict(_step("square", "lion", rows=2999, cols=1777, dtype="f16", grads="f16"), name="lion_f16_2999x1777"),
        # coarser quantization groups (fewer scales to keep), fp32 gradients as an accumulation buffer leaves them
        dict(_step("square", "adamw", rows=4096, cols=4096, bits=32, group=128, grads="f32"), name="adamw_group128_4096"),
        # the reference's unfused text on its single-matrix configuration
        dict(_step("square", "adamw", rows=2048, cols=2048, fused=False), name="adamw_unfused_2048"),
        # image classification: 161 leaves, most of them tiny fp32 vectors; the recipe's no-decay group
        dict(_step("resnet", "sgdw", width=64, layers=50), name="resnet50_sgdw"),
        # the GPT-2 pretraining recipe: global-norm clipping in front of AdamW, warm-up + cosine schedule
        dict(_step("gpt2", "adamw", width=768, layers=12, vocab=50257, clip=True), name="gpt2_small_adamw_clip"),
        # the same pytree under Lion with the step captured in a CUDA graph
        dict(_step("gpt2", "lion", width=768, layers=12, vocab=50257, graph=True), name="gpt2_small_lion_graph"),
        # without donation (the default): the caller keeps the old parameters and state
        dict(_step("llama", "adamw", width=1024, layers=1, vocab=0, donate=False), name="layer_adamw_copied"),
        # one GPU's part of a large language model, 32-bit master weights: embeddings, four layers, head (the largest)
        dict(_step("llama", "adamw", width=4096, layers=4, vocab=128256, bits=32), name="llama_4_layers_adamw32"),
        # fp32 weights of a model for evaluation or export, and back into parameters and error-correction codes
        {"what": "export", "dtype": "bf16", "bits": 24, "width": 1024, "layers": 4, "vocab": 8192, "name": "export_fp32"},
        {"what": "import", "dtype": "bf16", "bits": 32, "width": 2048, "layers": 2, "vocab": 32000, "name": "import_fp32"},
        # both moments of a leaf quantized (state converted from another optimizer) and read back
        {"what": "codec", "rows": 4096, "cols": 4096, "group": 32, "name": "codec_4096"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _options(rng, case):
    """Options as they are met: mostly the defaults."""
    case["dtype"] = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
    case["grads"] = rng.choice([case["dtype"], "f32"])
    case["bits"] = rng.choice([24, 32]) if case["dtype"] != "f32" else None
    if case["dtype"] != "f32" and rng.random() < 0.1:
        case["bits"] = None
    case["quantize"] = rng.random() < 0.85
    case["group"] = rng.choice([32, 32, 32, 64, 128, 256, 16])
    case["fused"] = rng.random() < 0.8
    return case


def draw(rng):
    while True:
        kind = rng.choice(["square", "square", "square", "resnet", "gpt2", "gpt2", "llama", "copied", "export", "import", "codec"])
        if kind == "square":
            rows = _log(rng, 64, 16384)
            cols = rows if rng.random() < 0.4 else max(1, min(16384, int(rows * math.exp(rng.uniform(-1.4, 1.4)))))
            case = _options(rng, _step("square", rng.choice(["adamw", "adamw", "adam", "lion", "sgd", "sgdw"]), rows=rows, cols=cols))
        elif kind == "resnet":
            case = _step("resnet", rng.choice(["sgdw", "sgdw", "adamw"]), width=_log(rng, 16, 96), layers=rng.choice([26, 50, 101]),
                         graph=rng.random() < 0.3)
        elif kind == "gpt2":
            case = _step("gpt2", rng.choice(["adamw", "lion"]), width=16 * _log(rng, 8, 100), layers=rng.randint(2, 24),
                         vocab=_log(rng, 257, 50257), bits=rng.choice([24, 32]))
            case["graph"] = rng.random() < 0.4
            case["clip"] = not case["graph"] and rng.random() < 0.6
        elif kind == "llama":
            case = _step("llama", rng.choice(["adamw", "adamw", "lion"]), width=128 * _log(rng, 4, 32), layers=rng.randint(1, 6),
                         vocab=_log(rng, 8192, 128256), bits=rng.choice([24, 32]))
        elif kind == "copied":
            case = _step("llama", rng.choice(["adamw", "lion", "sgdw"]), width=32 * _log(rng, 4, 128), layers=1, vocab=0,
                         bits=rng.choice([24, 32]), donate=False)
        elif kind in ("export", "import"):
            case = {"what": kind, "dtype": rng.choice(["bf16", "bf16", "f16"]), "bits": rng.choice([24, 32]), "width": 32 * _log(rng, 4, 96),
                    "layers": rng.randint(1, 3), "vocab": _log(rng, 257, 64000)}
        else:
            case = {"what": "codec", "rows": _log(rng, 64, 16384), "cols": _log(rng, 64, 16384), "group": rng.choice([32, 32, 64, 128, 16])}
        if sum(math.prod(shape) for shape, _ in _shapes(case).values()) <= MAX_PARAMS:
            return case


# ---- shapes: {leaf name: (shape, kind)}; "w" weights in the case's dtype, "zero" biases in it, "f32" fp32 vectors ----


def _shapes(case):
    if case["what"] == "codec" or case.get("tree") == "square":
        return {"w": ((case["rows"], case["cols"]), "w"), "b": ((case["cols"],), "zero")}
    if case["what"] != "step":
        return _llama(case)
    return {"resnet": _resnet, "gpt2": _gpt2, "llama": _llama}[case["tree"]](case)


def _resnet(case):
    """Bottleneck ResNet: HWIO convolution kernels, BatchNorm scale / bias pairs, classifier (161 leaves for 50 layers)."""
    w = case["width"]
    shapes = {"stem_conv/kernel": ((7, 7, 3, w), "w"), "stem_bn/scale": ((w,), "f32"), "stem_bn/bias": ((w,), "f32")}
    cin = w
    for stage, blocks in enumerate({26: (2, 2, 2, 2), 50: (3, 4, 6, 3), 101: (3, 4, 23, 3)}[case["layers"]]):
        f = w << stage
        for block in range(blocks):
            p = f"layer{stage}_block{block}/"
            convs = [("conv1", "bn1", (1, 1, cin, f)), ("conv2", "bn2", (3, 3, f, f)), ("conv3", "bn3", (1, 1, f, 4 * f))]
            if block == 0:
                convs.append(("proj_conv", "proj_bn", (1, 1, cin, 4 * f)))
            for conv, bn, shape in convs:
                shapes[p + conv + "/kernel"] = (shape, "w")
                shapes[p + bn + "/scale"] = ((shape[-1],), "f32")
                shapes[p + bn + "/bias"] = ((shape[-1],), "f32")
            cin = 4 * f
    shapes["fc/kernel"] = ((cin, 1000), "w")
    shapes["fc/bias"] = ((1000,), "f32")
    return shapes


def _gpt2(case):
    d = case["width"]
    shapes = {"wte": ((case["vocab"], d), "w"), "wpe": ((1024, d), "w"), "ln_f.scale": ((d,), "f32"), "ln_f.bias": ((d,), "f32")}
    for i in range(case["layers"]):
        p = f"h.{i:02d}."
        for ln in ("ln_1", "ln_2"):
            shapes[p + ln + ".scale"] = ((d,), "f32")
            shapes[p + ln + ".bias"] = ((d,), "f32")
        for name, rows, cols in (("c_attn", d, 3 * d), ("attn_proj", d, d), ("c_fc", d, 4 * d), ("mlp_proj", 4 * d, d)):
            shapes[p + name + ".w"] = ((rows, cols), "w")
            shapes[p + name + ".b"] = ((cols,), "zero")
    return shapes


def _llama(case):
    """Embeddings and head (none for vocab 0), layers with grouped-query attention and a gated MLP, RMSNorm weights."""
    d = case["width"]
    kv, ff = max(32, d // 4), d * 7 // 2
    shapes = {"norm": ((d,), "f32")}
    if case["vocab"]:
        shapes["tok_embeddings"] = ((case["vocab"], d), "w")
        shapes["lm_head"] = ((case["vocab"], d), "w")
    for i in range(case["layers"]):
        p = f"layers.{i:02d}."
        for name, shape in (("wq", (d, d)), ("wk", (d, kv)), ("wv", (d, kv)), ("wo", (d, d)), ("w1", (d, ff)), ("w3", (d, ff)), ("w2", (ff, d))):
            shapes[p + name] = (shape, "w")
        shapes[p + "attention_norm"] = ((d,), "f32")
        shapes[p + "ffn_norm"] = ((d,), "f32")
    return shapes


# ---- inputs ---------------------------------------------------------------------------------------------------


def _randn(shape, gen):
    return torch.randn(shape, device="cuda", generator=gen)


def _params(case, gen):
    dt = DTYPES[case["dtype"]]
    out = {}
    for name, (shape, kind) in _shapes(case).items():
        if kind == "f32":
            out[name] = torch.ones(shape, device="cuda") + 0.01 * _randn(shape, gen)
        elif kind == "zero":
            out[name] = torch.zeros(shape, device="cuda", dtype=dt)
        else:
            out[name] = (_randn(shape, gen) * 0.02).to(dt)
    return out


def _grads(case, params, gen, resting):
    """Normal draws, 0.01 % of the entries a hundred times as large; the embedding rows in `resting` (tokens that never
    occur) have none."""
    out = {}
    for name, p in params.items():
        g = _randn(p.shape, gen).mul_(1e-3)
        flat = g.view(-1)
        at = torch.randint(flat.numel(), (flat.numel() // 10000 + 1,), device="cuda", generator=gen)
        flat[at] = flat[at] * 100.0
        if name in resting:
            g[resting[name]] = 0.0
        out[name] = g.to(torch.float32 if p.dtype == torch.float32 else DTYPES[case["grads"]])
    return out


def _arena(tree):
    """The tree with its tensors laid out one after another (512-byte starts, as an allocator gives them) in one buffer
    per dtype, and those buffers: the outputs of a step that updates a model's tensors in place."""
    leaves, treedef = pytree.tree_flatten(tree)
    real = [i for i, x in enumerate(leaves) if x.dim() > 0]  # the step count and the 0-d markers of absent buffers stay as they are
    used, place = {}, {}
    for i in real:
        dt, step = leaves[i].dtype, 512 // leaves[i].element_size()
        place[i] = used.get(dt, 0)
        used[dt] = place[i] + -(-leaves[i].numel() // step) * step
    buffers = {dt: torch.zeros(n, dtype=dt, device="cuda") for dt, n in used.items()}
    for i in real:
        view = buffers[leaves[i].dtype][place[i]:place[i] + leaves[i].numel()].view(leaves[i].shape)
        leaves[i] = view.copy_(leaves[i])
    return treedef.unflatten(leaves), {str(dt): b for dt, b in buffers.items()}


def _no_decay(path, _leaf):
    last = str(path[-1])
    return last.endswith("bias") or "bn" in last


def _optimizer(case):
    kw = dict(HPARAMS[case["opt"]], master_weight_bits=case["bits"], quantize=case["quantize"], group_size=case["group"],
              fused=case["fused"], donate=case["donate"], capturable=case["graph"])
    if case["tree"] == "resnet":
        kw["param_groups"] = [{"params": _no_decay, "weight_decay": 0.0}]
    if case["tree"] == "llama":
        kw["param_groups"] = [{"params": lambda path, _leaf: "norm" in str(path[-1]), "weight_decay": 0.0}]
    if case["clip"]:
        kw["learning_rate"] = schedules.warmup_cosine(20000, 100, kw["learning_rate"])
    tx = FACTORY[case["opt"]](**kw)
    return clipping.clip_by_global_norm(tx, 1.0) if case["clip"] else tx


class _Training:
    """What a training program holds: the optimizer, parameters, state, and gradients that arrive in two buffers by turns."""


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["what"] == "codec":
        shape = (case["rows"], case["cols"])
        m = _randn(shape, gen) * 1e-3
        return {"what": "codec", "group": case["group"], "m": m, "v": (_randn(shape, gen) * 1e-3).square_()}
    if case["what"] == "import":
        template = {k: torch.empty_like(v) for k, v in _params(case, gen).items()}
        weights = {k: 0.02 * _randn(v.shape, gen) for k, v in template.items()}
        return {"what": "import", "weights": weights, "template": template, "bits": case["bits"]}
    if case["what"] == "export":
        weights = {k: 0.02 * _randn(v.shape, gen) for k, v in _params(case, gen).items()}
        template = {k: torch.empty(s, device="cuda", dtype=torch.float32 if kind == "f32" else DTYPES[case["dtype"]])
                    for k, (s, kind) in _shapes(case).items()}
        params, ecc = fo.set_fp32_params(weights, template, master_weight_bits=case["bits"])
        return {"what": "export", "params": params, "ecc": ecc}
    t = _Training()
    t.tx = _optimizer(case)
    params = _params(case, gen)
    resting = {}
    if "tok_embeddings" in params:  # a tenth of the vocabulary does not occur in the data
        rows = params["tok_embeddings"].shape[0]
        resting["tok_embeddings"] = torch.randperm(rows, device="cuda", generator=gen)[:rows // 10]
    t.grads = [_grads(case, params, gen, resting) for _ in range(2)]
    t.turn = 0
    opt = t.tx.init(params)
    if case["donate"]:
        (t.params, t.opt), t.buffers = _arena((params, opt))
    else:
        t.params, t.opt, t.buffers = params, opt, None
    del params, opt
    t.graph = None
    side = torch.cuda.Stream() if case["graph"] else torch.cuda.current_stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for g in t.grads:  # training has begun: moments and error-correction codes are not zero
            t.params, t.opt = t.tx.step(t.params, t.opt, g)
    torch.cuda.current_stream().wait_stream(side)
    if case["graph"]:
        torch.cuda.synchronize()
        t.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(t.graph):
            t.params, t.opt = t.tx.step(t.params, t.opt, t.grads[0])
    return t


def run(state):
    if isinstance(state, _Training):
        if state.graph is not None:
            state.graph.replay()
        else:
            state.turn ^= 1
            state.params, state.opt = state.tx.step(state.params, state.opt, state.grads[state.turn])
        opt = state.opt["opt"] if isinstance(state.opt, dict) else state.opt
        if state.buffers is not None:
            return {"count": opt.count, **state.buffers}
        return {"params": state.params, "opt": tuple(opt)}
    if state["what"] == "export":
        return fo.reconstruct_weights(state["params"], state["ecc"])
    if state["what"] == "import":
        return fo.set_fp32_params(state["weights"], state["template"], master_weight_bits=state["bits"])
    group = state["group"]
    m, v = fo.quantize_momentum(state["m"], group), fo.quantize_variance(state["v"], group)
    return (*m, *v, fo.dequantize_momentum(m, group), fo.dequantize_variance(v, group))


# ---- what a pass cannot do without -----------------------------------------------------------------------------


def work(case):
    nbytes = flops = 0.0
    for shape, kind in _shapes(case).values():
        n = math.prod(shape)
        if case["what"] == "codec":
            if kind == "w":  # values in, codes and scales out, and the way back, for two moments
                nbytes += 2 * 2 * n * (4 + 1 + 2 / case["group"])
                flops += 2 * 15 * n
            continue
        f32 = kind == "f32" or case["dtype"] == "f32"
        ecc = 0 if f32 or case["bits"] is None else (case["bits"] - 16) // 8
        if case["what"] != "step":  # fp32 weights on one side, parameter and code on the other; fp32 leaves are passed on
            if not f32:
                nbytes += n * (4 + 2 + ecc)
                flops += 5 * n
            continue
        adam = case["opt"] in ("adam", "adamw")
        moments = (2 if adam else 1) * ((1 + 2 / case["group"]) if case["quantize"] else 4)
        grad = 4 if f32 or case["grads"] == "f32" else 2
        nbytes += n * (grad + 2 * ((4 if f32 else 2) + ecc + moments))
        flops += n * (57 if adam else 25)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Every stored bit is defined by the arithmetic (one IEEE rounding per written operation), so a step's outputs are
    exact.  The one exception is the order in which clipping adds up the squares of the gradients: the last place of
    the fp32 norm may differ, hence that of the fp32 leaves' rescaled gradients, and a code that sits on a tie."""
    if case.get("clip"):
        return {"rel": 1e-5, "max": 1e-2, "differ": 1e-4}
    return "exact"
