"""Workloads by which the speed of this framework is judged, and plain 64-bit restatements of them.

Two kinds of work, each through the entry points that a user's program calls:

* ``train``: one optimizer step of a model - forward, backward, update - on inputs that are on the GPU.  GPT through
  ``parallel.FSDP`` (one rank), ResNet-50 through ``parallel.dp.DataParallel`` with fp16 and a loss scale on the device.
* ``serve``: one step of the continuous-batching engine through ``Engine.feed``: the next token of ``rows`` running sequences
  (decode), whole prompts of new ones, or both in one batch.  Running sequences grow by a token a pass, as they do in earnest
  (an answer has some hundred tokens); prompts are released when they are done, so their places come free for the next.

Model sizes are those of the benchmarks under ``bench/``.  Weights are drawn at random; tokens are uniform.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch
import torch.nn.functional as TF
from torch.utils.checkpoint import checkpoint

GROW = 2048             # tokens by which a running sequence may grow before it starts over
SCORED = 16             # last places of a prompt whose logits are asked for
VOCAB = 32000
SIZES = {  # width, heads, kv_heads, dense ff, experts, top, expert ff, shared ff
    "2b": (2048, 16, 4, 5632, 32, 4, 1024, 1536),
    "7b": (4096, 32, 8, 11008, 32, 4, 2048, 2816),
}
FAMILIES = ("llama", "zidalix", "nufupel", "potodra", "lerosun")


# ---------------------------------------------------------------- the cases
def listed():
    def serve(name, model, size, rows=0, ctx=0, prompts=0, prompt=0, layers=8):
        return {"name": name, "kind": "serve", "model": model, "size": size, "layers": layers, "rows": rows, "ctx": ctx,
                "prompts": prompts, "prompt": prompt}

    return [
        # the two-layer float32 decoder that a first training script runs: nothing but launches and latency
        {"name": "train tiny decoder f32", "kind": "gpt", "dtype": "float32", "width": 128, "heads": 4, "layers": 2, "ff": 512, "act": "relu",
         "vocab": 1024, "batch": 8, "seq": 64},
        # a small GPT with ragged sizes: a batch of three, a sequence that is no multiple of a tile
        {"name": "train small GPT ragged", "kind": "gpt", "dtype": "bfloat16", "width": 1024, "heads": 8, "layers": 4, "ff": 4096,
         "act": "gelu", "vocab": 16000, "batch": 3, "seq": 1000},
        # the GPT-1.3B training step
        {"name": "train GPT 1.3B", "kind": "gpt", "dtype": "bfloat16", "width": 2048, "heads": 16, "layers": 24, "ff": 8192, "act": "gelu",
         "vocab": 50304, "batch": 8, "seq": 2048},
        # a middle-sized GPT on short sequences
        {"name": "train GPT 350M", "kind": "gpt", "dtype": "bfloat16", "width": 1024, "heads": 8, "layers": 24, "ff": 4096, "act": "gelu",
         "vocab": 50304, "batch": 4, "seq": 1024},
        # the ResNet-50 training step in fp16
        {"name": "train ResNet-50", "kind": "resnet", "images": 256, "side": 224},
        # a lone user of the INT4 server: latency of a token
        serve("llama int4 decode 1", "llama", "7b", rows=1, ctx=1100),
        # a busy INT4 server between arrivals
        serve("llama int4 decode 48", "llama", "7b", rows=48, ctx=1250),
        # a busy INT4 server as a request arrives: a prompt beside the running sequences
        serve("llama int4 arrival", "llama", "7b", rows=24, ctx=900, prompts=1, prompt=1531),
        # decoding over latents with a long context
        serve("zidalix decode 16", "zidalix", "7b", rows=16, ctx=2200),
        # prompts of several lengths through windows and mixtures of experts
        serve("nufupel prompts", "nufupel", "2b", prompts=3, prompt=1900),
        # many running sequences with matrix memories, windows and four residual streams
        serve("potodra decode 64", "potodra", "2b", rows=64, ctx=600),
        # prompts through talking heads and the delta rule
        serve("lerosun prompts", "lerosun", "2b", prompts=2, prompt=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gpt"] * 3 + ["resnet"] + ["serve"] * 8)
    if kind == "gpt" and rng.random() < 0.3:
        heads = rng.choice([2, 4, 8])
        return {"kind": "gpt", "dtype": "float32", "width": 32 * heads, "heads": heads, "layers": rng.randint(1, 4), "ff": 128 * heads,
                "act": rng.choice(["relu", "gelu"]), "vocab": 8 * _log(rng, 32, 500), "batch": rng.randint(1, 16), "seq": 8 * rng.randint(2, 16)}
    if kind == "gpt":
        heads = rng.randint(4, 16)
        return {"kind": "gpt", "dtype": "bfloat16", "width": 128 * heads, "heads": heads, "layers": rng.randint(1, 12), "ff": 512 * heads,
                "act": rng.choice(["relu", "gelu"]), "vocab": 64 * _log(rng, 64, 786), "batch": rng.randint(1, 8), "seq": _log(rng, 64, 2048)}
    if kind == "resnet":
        return {"kind": "resnet", "images": _log(rng, 8, 256), "side": 32 * rng.randint(4, 7)}
    model, phase = rng.choice(FAMILIES), rng.choice(["decode", "decode", "prompt", "both"])
    rows = 0 if phase == "prompt" else _log(rng, 1, 64)
    prompts = 0 if phase == "decode" else rng.randint(1, 3)
    # prompts of a few tokens up to a whole step's budget; the running sequences' contexts fit the pool three times over
    return {"kind": "serve", "model": model, "size": rng.choice(["2b", "2b", "7b"]), "layers": 8, "rows": rows,
            "ctx": _log(rng, 64, 2048 if rows <= 32 else 1024) if rows else 0, "prompts": prompts,
            "prompt": _log(rng, 24, 4096 // max(prompts, 1)) if prompts else 0}


def _lengths(case):
    """(context of every running sequence, length of every prompt): they differ, as those of real users do."""
    ctx = [case["ctx"] - (i * 37) % max(1, case["ctx"] // 4) for i in range(case["rows"])]
    prompt = [case["prompt"] - i * (case["prompt"] // 5) for i in range(case["prompts"])]
    return ctx, prompt


# ---------------------------------------------------------------- weights of the training models
def _gpt_units(case):
    """(unit, [(parameter, shape)]): how a user finds the gradients in the engine's flat buffers."""
    d, ff, v = case["width"], case["ff"], case["vocab"]

    def block(i):
        p = f"blocks.{i}."
        return [(p + "ln1.weight", (d,)), (p + "ln1.bias", (d,)), (p + "attn.qkv_weight", (d, 3 * d)), (p + "attn.qkv_bias", (3 * d,)),
                (p + "attn.out_proj.weight", (d, d)), (p + "attn.out_proj.bias", (d,)), (p + "ln2.weight", (d,)), (p + "ln2.bias", (d,)),
                (p + "mlp_fc1.weight", (d, ff)), (p + "mlp_fc1.bias", (ff,)), (p + "mlp_fc2.weight", (ff, d)), (p + "mlp_fc2.bias", (d,))]
    first = [("token_emb.weight", (v, d)), ("pos_emb.weight", (case["seq"], d))]
    last = [("ln_final.weight", (d,)), ("ln_final.bias", (d,)), ("head.weight", (d, v))]
    return [("embeddings", first)] + [(f"blocks.{i}", block(i)) for i in range(case["layers"])] + [("tail", last)]


def _train_weights(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
    out = {}
    for _, params in _gpt_units(case):
        for name, shape in params:
            r = torch.randn(shape, generator=g, device="cuda")
            norm = ".ln" in name or name.startswith("ln_final")
            w = 0.02 * r if len(shape) > 1 else 1 + 0.1 * r if norm and name.endswith("weight") else 0.02 * r
            out[name] = w.to(getattr(torch, case["dtype"]))
    return out


def _tokens(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 2)
    t = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=g, device="cuda")
    return t[:, :-1], t[:, 1:]


def _conv_shapes():
    """ResNet-50's parameters in the order of the model."""
    def bn(p, c):
        return [(p + "weight", (c,)), (p + "bias", (c,))]

    out = [("conv1.weight", (64, 147))] + bn("bn1.", 64)
    cin, n = 64, 0
    for i, count in enumerate((3, 4, 6, 3)):
        w = 64 * 2 ** i
        for j in range(count):
            p = f"blocks.{n}."
            out += [(p + "conv1.weight", (w, cin))] + bn(p + "bn1.", w) + [(p + "conv2.weight", (w, 9 * w))] + bn(p + "bn2.", w)
            out += [(p + "conv3.weight", (4 * w, w))] + bn(p + "bn3.", 4 * w)
            if j == 0:
                out += [(p + "downsample.conv.weight", (4 * w, cin))] + bn(p + "downsample.bn.", 4 * w)
            cin, n = 4 * w, n + 1
    return out + [("fc.weight", (2048, 1000)), ("fc.bias", (1000,))]


def _conv_weights(seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
    out = {}
    for name, shape in _conv_shapes():
        r = torch.randn(shape, generator=g, device="cuda")
        if len(shape) == 2:
            w = r * (0.02 if name == "fc.weight" else math.sqrt(2.0 / shape[1]))
        else:
            # the last norm of a block starts small, so that blocks begin near the identity
            w = (0.2 if ".bn3." in name else 1.0) * (1 + 0.1 * r) if name.endswith("weight") else 0.02 * r
        out[name] = w.half()
    return out


def _images(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 2)
    x = torch.randn(case["images"], 3, case["side"], case["side"], generator=g, device="cuda").half().contiguous(memory_format=torch.channels_last)
    return x, torch.randint(0, 1000, (case["images"],), generator=g, device="cuda")


# ---------------------------------------------------------------- configurations of the served models
def _config(case):
    width, H, G, ff, E, top, eff, sff = SIZES[case["size"]]
    L, model = case["layers"], case["model"]
    head = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    rot = {"base": 1e6, "dims": 128}
    base = {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}}
    dense = {"kind": "dense", "ff": ff}
    if model == "llama":
        return {"vocab_size": VOCAB, "seq_len": 8192, "d_model": width, "num_heads": H, "num_kv_heads": H, "num_layers": L, "ffn_dim": ff}
    if model == "zidalix":
        m = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
             "rot": {"base": 1e6, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        return {**base, "logit_scale": 1.0, "layers": [
            {"type": "latent_attention", "mixer": dict(m, kv_from=i - 1) if i % 4 == 3 else m, "mlp": {**dense, "limit": 7.0}} for i in range(L)]}
    if model == "nufupel":
        band = {"base": 1e6, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
        moe = {"kind": "moe", "router": {"experts": E, "top": top}, "expert": {"ff": eff}, "shared": {"ff": sff}}
        return {**base, "logit_softcap": 30.0, "layers": [
            {"type": "attention_2" if i % 2 else "attention", "mixer": {**head, "mask": {"size": (1024, 2048)[i % 2]}, **({"rot": band} if i % 2 else {})},
             "mlp": moe if i else dense} for i in range(L)]}
    if model == "potodra":
        att, mem = {**head, "rot": rot}, {"heads": H, "dim": 128, "vdim": 128}
        mixers = [("attention", {**att, "mask": {"size": 1024, "keep_first": 16}, "softcap": 30.0})] + [("mlstm", {**mem, "gate_cap": 15.0})] * 2 + \
            [("parallel", {"left": att, "right": {**mem, "kv_heads": H, "conv": 4}, "left_scale": 0.5, "right_scale": 0.5})]
        # dense feed-forwards of as many weights as the other models': which experts its groups open turns on less than 16 bits hold
        wide = {"kind": "dense", "ff": ff * 3 // 2}
        return {**base, "streams": 4, "layers": [{"type": mixers[i % 4][0], "mixer": mixers[i % 4][1], "mlp": wide} for i in range(L)]}
    att, mem = {**head, "rot": rot, "mask": {"size": 1024}}, {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4}
    return {**base, "loop": None, "layers": [{"type": "attention" if i % 4 == 3 else "delta", "mixer": att if i % 4 == 3 else mem, "mlp": dense}
                                             for i in range(L)]}


def _model_config(case):
    from rumus_b200.models.lerosun import LerosunConfig
    from rumus_b200.models.llama import LlamaConfig
    from rumus_b200.models.nufupel import NufupelConfig
    from rumus_b200.models.potodra import PotodraConfig
    from rumus_b200.models.zidalix import ZidalixConfig
    classes = {"llama": LlamaConfig, "zidalix": ZidalixConfig, "nufupel": NufupelConfig, "potodra": PotodraConfig, "lerosun": LerosunConfig}
    return classes[case["model"]].from_dict(_config(case))


def _serving_weights(config, seed):
    """Random weights; routers are as peaked as trained ones, so that the last expert of a choice has little weight."""
    return {k: t * 4 if k.endswith("mlp.router") else t for k, t in config.random_weights(seed, device="cuda").items()}


def _sequences(case, seed):
    """Token ids: running sequences with the tokens they will go on with, prompts."""
    g = torch.Generator().manual_seed(seed * 7 + 3)
    ctx, prompt = _lengths(case)

    def ids(n):
        return torch.randint(0, VOCAB, (n,), generator=g).tolist()

    return [ids(n + GROW) for n in ctx], [ids(n) for n in prompt]


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "gpt":
        from rumus_b200.models import GPT, GPTConfig
        from rumus_b200.parallel import FSDP
        dt = getattr(torch, case["dtype"])
        model = GPT(GPTConfig(case["vocab"], case["seq"], case["width"], case["heads"], case["layers"], case["ff"], case["act"]), dev, dt)
        weights = _train_weights(case, seed)
        with torch.no_grad():
            for name, p in model.named_parameters():
                p.copy_(weights[name])
        engine = FSDP(model, lr=1e-4)
        x, y = _tokens(case, seed)
        return SimpleNamespace(case=case, model=model, engine=engine, x=x, y=y)
    if case["kind"] == "resnet":
        from rumus_b200.models import ResNet50
        from rumus_b200.optim import SGD, GradScaler
        from rumus_b200.parallel.dp import DataParallel
        model = ResNet50(device=dev, dtype=torch.float16)
        weights = _conv_weights(seed)
        with torch.no_grad():
            for name, p in model.named_parameters():
                p.copy_(weights[name])
        dp = DataParallel(model)
        scaler = GradScaler(init_scale=32768.0, device_side=True)
        scaler._ensure(dev)
        x, y = _images(case, seed)
        return SimpleNamespace(case=case, model=model, dp=dp, opt=SGD(model.parameters(), lr=0.01, momentum=0.9), scaler=scaler, x=x, y=y)
    from rumus_b200.serve import Engine, ServeConfig
    config = _model_config(case)
    running, prompts = _sequences(case, seed)
    blocks = sum(-(-len(s) // 64) + 1 for s in running + prompts) + 8
    longest = max(len(s) for s in running + prompts)
    cfg = ServeConfig(model=config, num_blocks=blocks, max_batch=len(running) + len(prompts), max_seq_len=longest)
    weights = None if case["model"] == "llama" else _serving_weights(config, seed)
    s = SimpleNamespace(case=case, engine=Engine(cfg, dev, seed=seed, weights=weights), running=running, prompts=prompts, ctx=_lengths(case)[0], pos=None)
    _start(s)
    if running:
        run(s)          # a server's first token is behind it
    return s


def _start(s):
    """The running sequences' contexts into the cache, a few at a time."""
    if s.pos is not None:
        for i in range(len(s.running)):
            s.engine.release(i)
    for i in range(0, len(s.running), 4):
        s.engine.feed([(j, s.running[j][:s.ctx[j]], []) for j in range(i, min(i + 4, len(s.running)))])
    s.pos = list(s.ctx)


def run(state):
    s, kind = state, state.case["kind"]
    if kind == "gpt":
        s.engine.zero_grad()
        loss = s.model(s.x, s.y)
        loss.backward()
        s.engine.step()
        return {"loss": loss.detach(), "grads": [u.flat_grad for u in s.engine.units], "weights": [u.master for u in s.engine.units]}
    if kind == "resnet":
        from rumus_b200.ops import functional as F
        s.dp.zero_grad()
        loss = F.cross_entropy_loss(s.model(s.x), s.y)
        s.dp.begin_backward(s.scaler.inv_scale)
        s.scaler.scale(loss).backward()
        found = s.dp.all_reduce_grads()
        s.opt.grad_scale, s.opt.skip_flag = None, found
        s.scaler.found_inf = found
        s.opt.step()
        s.scaler.update()
        return {"loss": loss.detach(), "grads": [b.flat for b in s.dp.buckets]}
    n = len(s.running)
    if n and s.pos[0] + 1 >= s.ctx[0] + GROW:
        _start(s)
    portions = [(i, [s.running[i][s.pos[i]]], [0]) for i in range(n)]
    portions += [(n + j, t, list(range(max(0, len(t) - SCORED), len(t)))) for j, t in enumerate(s.prompts)]
    logits = s.engine.feed(portions)
    for i in range(n):
        s.pos[i] += 1
    for j in range(len(s.prompts)):
        s.engine.release(n + j)
    return logits


# ---------------------------------------------------------------- what a pass cannot do without
def _attention_work(lengths, heads, width, window=None):
    """Operations of causal attention over whole prompts; ``width``: multiply-adds of a query and a key together."""
    pairs = sum(min(i + 1, window or i + 1) for n in lengths for i in range(n))
    return 2.0 * heads * width * pairs


def work(case):
    if case["kind"] == "gpt":
        d, ff, L, T = case["width"], case["ff"], case["layers"], case["batch"] * case["seq"]
        params = sum(math.prod(s) for _, ps in _gpt_units(case) for _, s in ps)
        mats = L * (4 * d * d + 2 * d * ff) + d * case["vocab"]
        flops = 6.0 * T * mats + 3 * _attention_work([case["seq"]], case["heads"], 2 * d // case["heads"]) * case["batch"]
        e = 4 if case["dtype"] == "float32" else 2
        # weights in, gradients out, fp32 master and two moments in and out, weights out
        return {"bytes": params * (3 * e + 24.0) + 16.0 * T, "flops": flops}
    if case["kind"] == "resnet":
        side, macs, out = case["side"], 0, (case["side"] + 1) // 2
        macs += out * out * 64 * 147
        out = (out + 1) // 2
        cin = 64
        for i, count in enumerate((3, 4, 6, 3)):
            w = 64 * 2 ** i
            for j in range(count):
                first = j == 0
                macs += out * out * cin * w
                out = (out + 1) // 2 if first and i else out
                macs += out * out * (9 * w * w + 4 * w * w + (4 * w * cin if first else 0))
                cin = 4 * w
        params = sum(math.prod(s) for _, s in _conv_shapes())
        return {"bytes": params * 2.0 * 6 + case["images"] * 3.0 * side * side * 2, "flops": 6.0 * case["images"] * macs}
    width, H, G, ff, E, top, eff, sff = SIZES[case["size"]]
    ctx, prompt = _lengths(case)
    rows, T = len(ctx), len(ctx) + sum(prompt)
    scored = rows + sum(min(SCORED, n) for n in prompt)
    hd, by, fl = H * 128, 0.0, 0.0

    def product(n, e=2.0, tokens=T):
        nonlocal by, fl
        by += n * e
        fl += 2.0 * n * tokens

    def cache(token, window=None):       # bytes a token keeps
        nonlocal by
        by += token * (sum(min(c, window or c) for c in ctx) + sum(prompt))

    def memory(heads):                   # a matrix state per sequence in and out, fp32; a few operations per element and token
        nonlocal by, fl
        by += (2 * rows + len(prompt)) * heads * 128 * 128 * 4.0
        fl += T * heads * 128 * 128 * 6.0

    for layer in range(case["layers"]) if case["model"] == "llama" else _config(case)["layers"]:
        if case["model"] == "llama":
            product(width * 3 * hd + hd * width + 3 * width * ff, 0.5 + 4 / 128)
            cache(4.0 * hd)
            fl += _attention_work(prompt, H, 256) + 4.0 * 128 * H * sum(ctx)
            continue
        kind, m, mlp = layer["type"], layer["mixer"], layer["mlp"]
        window = m.get("mask", {}).get("size")
        if kind == "latent_attention":
            product(width * (H * 192 + hd) + hd * width + 512 * 2 * hd + (0 if m.get("kv_from") is not None else 576 * width))
            cache(576 * 2.0)
            fl += _attention_work(prompt, H, 320) + 2.0 * H * (576 + 512) * sum(ctx)
        elif kind in ("attention", "attention_2"):
            gate = {"potodra": 0, "lerosun": H}.get(case["model"], H if kind == "attention_2" else hd)
            values = 0 if case["model"] == "lerosun" else G * 128
            product(width * (hd + G * 128 + values + gate) + hd * width)
            cache((G * 128 + values) * 2.0, window)
            mixed = H if case["model"] == "lerosun" else 0
            fl += _attention_work(prompt, H, 256 + mixed, window) + 2.0 * (256 + mixed) * H * sum(min(c, window) for c in ctx)
        elif kind == "mlstm":
            product(width * 4 * hd + hd * width)
            memory(H)
        elif kind == "delta":
            product(width * 4 * hd + hd * width)
            memory(H)
        else:
            product(width * (hd + 2 * G * 128) + hd * width + width * 3 * hd + hd * width + 2 * 128 * (width + hd))
            cache(G * 512.0)
            memory(H)
            fl += _attention_work(prompt, H, 256) + 4.0 * 128 * H * sum(ctx)
        if mlp["kind"] == "dense":
            product((2 if case["model"] == "potodra" else 3) * width * mlp["ff"])
        else:
            product(3 * width * sff + width * E)
            met = E * (1 - (1 - top / E) ** T)
            by += met * 3 * width * eff * 2
            fl += 2.0 * T * top * 3 * width * eff
    product(width * VOCAB, tokens=scored)
    return {"bytes": by + 4.0 * scored * VOCAB, "flops": fl}


def tolerance(case):
    """Four times what the path shows against 64 bits, or against itself in another order of sums."""
    if case["kind"] == "gpt":
        # gradients of bf16 or TF32 products through all layers; ``max``: single elements are sums of thousands of rounded terms
        return {"rel": 0.02, "max": 0.9}
    if case["kind"] == "resnet":
        return {"rel": 0.03, "max": 0.95}
    # bf16 activations through eight layers; a mixture may choose another expert where two are as good
    return {"rel": 0.03, "max": 0.9}


# ---------------------------------------------------------------- 64 bits: training
def exact(case, seed):
    w = work(case)
    if case["kind"] == "gpt":
        return _exact_train(case, seed) if w["flops"] < 250e12 else None
    if case["kind"] == "resnet":
        return _exact_resnet(case, seed)
    ctx, prompt = _lengths(case)
    # contexts are computed as well: two operations per weight and token
    per_token = (w["flops"] / (len(ctx) + sum(prompt)))
    return _exact_serve(case, seed) if per_token * (sum(ctx) + sum(prompt)) < 300e12 else None


def _flat(parts, align, multiple):
    out = []
    for t in parts:
        out += [t.reshape(-1), t.new_zeros(-t.numel() % align)]
    flat = torch.cat(out)
    return torch.cat([flat, flat.new_zeros(-flat.numel() % multiple)])


def _rope_halves(x, base, dims, neighbours=False, freq=None, factor=1.0):
    """x [..., T, heads, d]: pair i is (i, i + dims / 2), or (2 i, 2 i + 1) with ``neighbours``."""
    half = dims // 2
    if freq is None:
        freq = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    ang = torch.arange(x.shape[-3], dtype=torch.float64, device=x.device)[:, None] * freq
    c, s = (ang.cos() * factor)[:, None], (ang.sin() * factor)[:, None]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :half], x[..., half:dims])
    a, b = u * c - v * s, v * c + u * s
    turned = torch.stack([a, b], -1).flatten(-2) if neighbours else torch.cat([a, b], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _train_attention(qkv, H, hd):
    B, S, _ = qkv.shape
    q, k, v = (t.view(B, S, H, hd) for t in qkv.split(H * hd, -1))
    see = torch.ones(S, S, dtype=torch.bool, device=qkv.device).tril()
    out = []
    for b in range(B):
        s = torch.einsum("ihd,jhd->hij", q[b], k[b]) * hd ** -0.5
        out.append(torch.einsum("hij,jhd->ihd", s.masked_fill(~see, -math.inf).softmax(-1), v[b]))
    return torch.stack(out).reshape(B, S, H * hd)


def _exact_train(case, seed):
    units = _gpt_units(case)
    w = {k: t.double().requires_grad_() for k, t in _train_weights(case, seed).items()}
    x, y = _tokens(case, seed)
    d, H = case["width"], case["heads"]

    def block(h, i):
        p = {k[len(f"blocks.{i}."):]: t for k, t in w.items() if k.startswith(f"blocks.{i}.")}
        a = TF.layer_norm(h, (d,), p["ln1.weight"], p["ln1.bias"], 1e-5) @ p["attn.qkv_weight"] + p["attn.qkv_bias"]
        h = h + _train_attention(a, H, d // H) @ p["attn.out_proj.weight"] + p["attn.out_proj.bias"]
        m = TF.layer_norm(h, (d,), p["ln2.weight"], p["ln2.bias"], 1e-5) @ p["mlp_fc1.weight"] + p["mlp_fc1.bias"]
        m = torch.relu(m) if case["act"] == "relu" else TF.gelu(m, approximate="tanh")
        return h + m @ p["mlp_fc2.weight"] + p["mlp_fc2.bias"]

    def tail(h, y):
        h = TF.layer_norm(h, (d,), w["ln_final.weight"], w["ln_final.bias"], 1e-5)
        return TF.cross_entropy(h @ w["head.weight"], y, reduction="sum")

    h = w["token_emb.weight"][x] + w["pos_emb.weight"][:x.shape[1]]
    for i in range(case["layers"]):
        h = checkpoint(block, h, i, use_reentrant=False)
    loss = sum(checkpoint(tail, h[b], y[b], use_reentrant=False) for b in range(x.shape[0])) / y.numel()
    loss.backward()
    grads, weights = [], []
    for _, ps in units:
        grads.append(_flat([w[n].grad for n, _ in ps], 128, 512))
        # the first step of Adam: both moments are the gradient's own
        weights.append(_flat([(w[n] - 1e-4 * w[n].grad / (w[n].grad.abs() + 1e-8)).detach() for n, _ in ps], 128, 512))
        for n, _ in ps:
            w[n].grad = None
    return {"loss": loss.detach(), "grads": grads, "weights": weights}


def _exact_resnet(case, seed):
    w = {k: t.double().requires_grad_() for k, t in _conv_weights(seed).items()}
    x, y = _images(case, seed)

    def conv(h, name, k, stride):
        t = w[name + ".weight"]
        return TF.conv2d(h, t.view(t.shape[0], -1, k, k), stride=stride, padding=k // 2)

    def norm(h, name):
        return TF.batch_norm(h, None, None, w[name + ".weight"], w[name + ".bias"], True, 0.1, 1e-5)

    def block(h, p, stride, down):
        skip = norm(conv(h, p + "downsample.conv", 1, stride), p + "downsample.bn") if down else h
        h = torch.relu(norm(conv(h, p + "conv1", 1, 1), p + "bn1"))
        h = torch.relu(norm(conv(h, p + "conv2", 3, stride), p + "bn2"))
        return torch.relu(norm(conv(h, p + "conv3", 1, 1), p + "bn3") + skip)

    h = TF.max_pool2d(torch.relu(norm(conv(x.double(), "conv1", 7, 2), "bn1")), 3, 2, 1)
    n = 0
    for i, count in enumerate((3, 4, 6, 3)):
        for j in range(count):
            h = checkpoint(block, h, f"blocks.{n}.", 2 if j == 0 and i else 1, j == 0, use_reentrant=False)
            n += 1
    loss = TF.cross_entropy(h.mean((2, 3)) @ w["fc.weight"] + w["fc.bias"], y)
    loss.backward()
    buckets, cur, size = [], [], 0
    for name, _ in reversed(_conv_shapes()):        # buckets of 25 MB in the order of backward
        cur.append(w[name].grad)
        size += cur[-1].numel() * 2
        if size >= 25 << 20:
            buckets.append(_flat(cur, 64, 16))
            cur, size = [], 0
    # the first layers' gradients have no such value: fp16 activations that round to the other side of a ReLU or to another maximum,
    # block after block, move them by a tenth of their norm
    return {"loss": loss.detach(), "grads": [buckets[0]] + [None] * (len(buckets) - 1 + bool(cur))}


# ---------------------------------------------------------------- 64 bits: serving
def _attend(q, k, v, scale, window=None, keep=0, cap=None, sink=None, mix=None):
    """q [T, H, d], k [T, G, d], v [T, G, e] of one sequence."""
    T, H, per = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    i = torch.arange(T, device=q.device)
    gap = i[:, None] - i[None]
    see = gap >= 0
    if window:
        see &= (gap < window) | (i[None] < keep)

    def rows(heads):
        s = torch.einsum("ihd,jhd->hij", q[:, heads], k[:, [h // per for h in heads]]) * scale
        return cap * torch.tanh(s / cap) if cap else s

    out = torch.empty(T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    every = torch.einsum("gh,hij->gij", mix, rows(list(range(H)))) if mix is not None else None
    for h in range(H):
        s = (every[h] if every is not None else rows([h])[0]).masked_fill(~see, -math.inf)
        top = s.max(-1, keepdim=True).values
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0)
        out[:, h] = (e / den) @ v[:, h // per]
    return out


def _each(f, *xs):
    """f over the sequences of a batch."""
    return torch.stack([f(*ts) for ts in zip(*xs)])


def _short_conv(x, taps):
    n = taps.shape[1]
    wide = torch.cat([x.new_zeros(x.shape[0], n - 1, x.shape[2]), x], 1)
    return TF.silu(sum(wide[:, j:j + x.shape[1]] * taps[:, j] for j in range(n)))


def _delta_memory(q, k, v, g, beta):
    """q, k [B, T, H, d], v [B, T, H, e], g [B, T, H, d or 1], beta [B, T, H] -> [B, T, H, e]."""
    S = q.new_zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3])
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        S *= g[:, t, :, :, None]
        new = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhd,bhde->bhe", k[:, t], S))
        S += k[:, t, :, :, None] * new[:, :, None]
        out[:, t] = torch.einsum("bhd,bhde->bhe", q[:, t], S)
    return out


def _delta(h, w, p, m, eps, decays, gate):
    B, T = h.shape[:2]
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]

    def unit(x):
        return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)

    def part(name, n, size):
        return _short_conv(h @ w[p + name].T, w[p + name + ".conv"]).view(B, T, n, size)

    per = H // G
    q, k = unit(part("q", G, d)).repeat_interleave(per, 2) * d ** -0.5, unit(part("k", G, d)).repeat_interleave(per, 2)
    o = _delta_memory(q, k, part("v", H, e), decays, torch.sigmoid(h @ w[p + "b"].T))
    return (_rms(o, eps) * w[p + "norm"] * gate.view(B, T, H, e)).flatten(2) @ w[p + "o"].T


def _mlstm(h, w, p, m, eps):
    B, T = h.shape[:2]
    H, d, e, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k = (h @ w[p + "q"].T).view(B, T, H, d) * d ** -0.5, (h @ w[p + "k"].T).view(B, T, H, d)
    v = (h @ w[p + "v"].T).view(B, T, H, e)
    i = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    f = TF.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    S, n, top = q.new_zeros(B, H, d, e), q.new_zeros(B, H, d), q.new_zeros(B, H)
    out = torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(f[:, t] + top, i[:, t])
        keep, put = torch.exp(f[:, t] + top - new)[..., None], torch.exp(i[:, t] - new)[..., None]
        S = S.mul_(keep[..., None]).add_((put * k[:, t])[..., None] * v[:, t, :, None])
        n, top = keep * n + put * k[:, t], new
        den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[:, t] = torch.einsum("bhd,bhde->bhe", q[:, t], S) / den[..., None]
    return (_rms(out, eps).flatten(2) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def _unit(h, w, p, act):
    return (act(h @ w[p + "gate"].T.double()) * (h @ w[p + "up"].T.double())) @ w[p + "down"].T.double()


def _clamped(h, w, p, limit):
    g, u = (h @ w[p + "gate"].T.double()).clamp(max=limit), (h @ w[p + "up"].T.double()).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].T.double()


def _experts(h, chosen, weight, f):
    """h [N, d]; expert ``chosen`` [N, top] with ``weight``; f(x, expert)."""
    y = torch.zeros_like(h)
    for e in chosen.unique().tolist():
        row, place = (chosen == e).nonzero(as_tuple=True)
        y.index_add_(0, row, weight[row, place, None] * f(h[row], e))
    return y


def _mix_nufupel(h, w, p, m):
    x = h.flatten(0, 1)
    top = (x @ w[p + "router"].T + w[p + "router.b"]).topk(m["router"]["top"], -1)
    y = _unit(x, w, p + "shared.", TF.silu) + _experts(x, top.indices, top.values.softmax(-1), lambda t, e: _unit(t, w, f"{p}e{e}.", TF.silu))
    return y.view_as(h)


def _int4(w):
    """A weight [in, out] as the server keeps it: groups of 128 inputs, 16 steps between the least and the largest, fp16 scale and zero."""
    K, N = w.shape
    g = TF.pad(w, (0, 0, 0, -K % 128)).view(-1, 128, N)
    lo, hi = g.min(1).values, g.max(1).values
    scale = (hi - lo) / 15.0
    zero = (-lo / scale).half().float()
    scale = scale.half().float()
    q = torch.clamp(torch.round(g / scale[:, None] + zero[:, None]), 0, 15)
    return ((q.double() - zero.double()[:, None]) * scale.double()[:, None]).view(-1, N)[:K]


def _llama_hidden(c, seed, tokens):
    g = torch.Generator(device="cuda").manual_seed(seed)
    d, ff, H = c["d_model"], c["ffn_dim"], c["num_heads"]

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda") * 0.02

    x = rnd(VOCAB, d).bfloat16().double()[tokens]
    for _ in range(c["num_layers"]):
        qkv, o = _int4(torch.cat([rnd(d, d), rnd(d, d), rnd(d, d)], 1)), _int4(rnd(d, d))
        gate_up, down = _int4(torch.cat([rnd(d, ff), rnd(d, ff)], 1)), _int4(rnd(ff, d))
        q, k, v = ((t.view(*t.shape[:2], H, -1)) for t in (_rms(x, 1e-5) @ qkv).split(d, -1))
        q, k = _rope_halves(q, 10000.0, d // H), _rope_halves(k, 10000.0, d // H)
        a = _each(lambda q, k, v: _attend(q, k, v, (d // H) ** -0.5), q, k, v)
        x = x + a.flatten(2) @ o
        g1, u = (_rms(x, 1e-5) @ gate_up).chunk(2, -1)
        x = x + (TF.silu(g1) * u) @ down
    return _rms(x, 1e-5), rnd(d, VOCAB).bfloat16().double()


def _zidalix_hidden(c, w, tokens):
    x, store, eps = w["embed"][tokens], {}, c["norm"]["eps"]
    B, T = tokens.shape
    y = c["layers"][0]["mixer"]["rot"]
    sc, dims = y["scaling"], y["dims"]

    def turns(t):
        return dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(y["base"]))

    lo, hi = max(math.floor(turns(sc["fast"])), 0), min(math.ceil(turns(sc["slow"])), dims - 1)
    n = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f, ramp = y["base"] ** (-2.0 * n / dims), ((n - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f, factor = f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0

    def turn(t):
        return _rope_halves(t, y["base"], dims, True, f, factor)

    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, D, V, R = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
        h = _rms(x, eps) * w[f"l{i}.norm1"]
        q = (h @ w[p + "q"].T).view(B, T, H, -1)
        q = torch.cat([q[..., :D], turn(q[..., D:])], -1)
        if m.get("kv_from") is None:
            z = h @ w[p + "dkv"].T
            store[i] = _rms(z[..., :R], eps) * w[p + "dkv.norm"], turn(z[..., None, R:])
        lat, kr = store[i if m.get("kv_from") is None else m["kv_from"]]
        k = torch.cat([(lat @ w[p + "uk"].T).view(B, T, H, D), kr.expand(B, T, H, -1)], -1)
        v = (lat @ w[p + "uv"].T).view(B, T, H, V)
        o = _each(lambda q, k, v: _attend(q, k, v, m["scale"], sink=w[p + "sink"]), q, k, v).flatten(2)
        out = (o * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
        x = x + out + _clamped(_rms(x, eps) * w[f"l{i}.norm2"], w, f"l{i}.mlp.", layer["mlp"]["limit"])
    return _rms(x, eps) * w["final.norm"], w["head"].T


def _nufupel_hidden(c, w, tokens):
    x, eps = w["embed"][tokens], c["norm"]["eps"]
    B, T = tokens.shape
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, G = m["heads"], m["kv_heads"]
        h = _rms(x, eps) * (1 + w[f"l{i}.norm1"])
        q, k, v = ((h @ w[p + n].T).view(B, T, s, 128) for n, s in (("q", H), ("k", G), ("v", G)))
        gate = torch.sigmoid(h @ w[p + "g"].T)
        if layer["type"] == "attention_2":
            r, s = m["rot"], m["rot"]["scaling"]
            f = r["base"] ** (-2.0 * torch.arange(r["dims"] // 2, dtype=torch.float64, device=x.device) / r["dims"])
            wave = 2 * math.pi / f
            blend = (s["original"] / wave - s["low"]) / (s["high"] - s["low"])
            mid = (1 - blend) * f / s["factor"] + blend * f
            f = torch.where(wave > s["original"] / s["low"], f / s["factor"], torch.where(wave < s["original"] / s["high"], f, mid))
            q = _rope_halves(_rms(q, eps) * w[p + "q.norm"], 0, r["dims"], freq=f)
            k = _rope_halves(_rms(k, eps) * w[p + "k.norm"], 0, r["dims"], freq=f)
        o = _each(lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], sink=w[p + "sink"]), q, k, v)
        o = o * (gate[..., None] if layer["type"] == "attention_2" else gate.view_as(o))
        n = f"l{i}.mlp."
        y = _unit(h, w, n, lambda t: TF.gelu(t, approximate="tanh")) if layer["mlp"]["kind"] == "dense" else _mix_nufupel(h, w, n, layer["mlp"])
        x = x + o.flatten(2) @ w[p + "o"].T + y
    return _rms(x, eps) * (1 + w["final.norm"]), w["head"].T


def _potodra_hidden(c, w, tokens):
    eps = c["norm"]["eps"]
    B, T = tokens.shape
    xs = w["embed"][tokens].unsqueeze(2).repeat(1, 1, c["streams"], 1)

    def attention(h, p, m, neighbours, sink):
        H, G = m["heads"], m["kv_heads"]
        q, k, v = ((h @ w[p + n].T + w[p + n + ".b"]).view(B, T, s, 128) for n, s in (("q", H), ("k", G), ("v", G)))
        q, k = (_rope_halves(t, m["rot"]["base"], m["rot"]["dims"], neighbours) for t in (q, k))
        mask = m.get("mask") or {}
        o = _each(lambda q, k, v: _attend(q, k, v, m["scale"], mask.get("size"), mask.get("keep_first", 0), m.get("softcap"), sink), q, k, v)
        return o.flatten(2) @ w[p + "o"].T

    def mixer(h, p, layer):
        m = layer["mixer"]
        if layer["type"] == "attention":
            return attention(h, p, m, False, w[p + "sink"])
        if layer["type"] == "mlstm":
            return _mlstm(h, w, p, m, eps)
        r, o = m["right"], p + "right."
        step = TF.softplus(h @ w[o + "a1"].T @ w[o + "a2"].T + w[o + "dt_bias"]).view(B, T, r["heads"], r["dim"])
        gate = torch.sigmoid(h @ w[o + "g1"].T @ w[o + "g2"].T)
        right = _delta(h, w, o, r, eps, torch.exp(-torch.exp(w[o + "A_log"])[:, None] * step), gate)
        return m["left_scale"] * attention(h, p + "left.", m["left"], True, None) + m["right_scale"] * right

    for i, layer in enumerate(c["layers"]):
        def sublayer(xs, n, f):
            hc = f"l{i}.hc{n}."
            y = f(_rms(torch.einsum("s,btsd->btd", w[hc + "in"], xs), eps) * w[f"l{i}.norm{n}"])
            return torch.einsum("su,btsd->btud", w[hc + "mix"], xs) + w[hc + "out"][:, None] * y[:, :, None]

        def feed_forward(h, p=f"l{i}.mlp."):
            return torch.relu(h @ w[p + "up"].T.double()) ** 2 @ w[p + "down"].T.double()

        xs = sublayer(xs, 1, lambda h: mixer(h, f"l{i}.mix.", layer))
        xs = sublayer(xs, 2, feed_forward)
    return _rms(xs.sum(2), eps) * w["final.norm"], w["embed"].T


def _lerosun_hidden(c, w, tokens):
    eps = c["norm"]["eps"]
    B, T = tokens.shape
    x = _rms(w["embed"][tokens], eps) * w["embed.norm"]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, G = m["heads"], m["kv_heads"]
        h = _rms(x, eps) * w[f"l{i}.norm1"]
        if layer["type"] == "attention":
            q, k = ((h @ w[p + n].T + w[p + n + ".b"]).view(B, T, s, 128) for n, s in (("q", H), ("k", G)))
            qr, kr = (_rope_halves(t, m["rot"]["base"], m["rot"]["dims"]) for t in (q, k))
            qr = qr * w[p + "temp"][:, None]
            o = _each(lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], sink=w[p + "sink"], mix=w[p + "talk"]), qr, kr, k)
            y = (o * torch.sigmoid(h @ w[p + "g"].T)[..., None]).flatten(2) @ w[p + "o"].T
        else:
            g = torch.exp(-torch.exp(w[p + "A_log"]) * TF.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
            y = _delta(h, w, p, m, eps, g[..., None], TF.silu(h @ w[p + "g"].T))
        x = x + w[f"l{i}.ls1"] * y
        x = x + w[f"l{i}.ls2"] * _unit(_rms(x, eps) * w[f"l{i}.norm2"], w, f"l{i}.mlp.", torch.relu)
    return _rms(x, eps) * w["final.norm"], w["head"].T


class _Doubles(dict):
    """Weights in 64 bits as they are asked for; those of feed-forward layers stay as they are until they are used."""

    def __getitem__(self, k):
        t = super().__getitem__(k)
        return t if ".mlp." in k and k.rsplit(".", 1)[-1] in ("gate", "up", "down") else t.double()


def _exact_serve(case, seed):
    running, prompts = _sequences(case, seed)
    ctx = _lengths(case)[0]
    # prepare has fed the context and one token, the pass feeds the next
    seqs = [s[:n + 2] for s, n in zip(running, ctx)] + prompts
    wanted = [1] * len(running) + [min(SCORED, len(p)) for p in prompts]
    c = _config(case)
    w = None if case["model"] == "llama" else _Doubles(_serving_weights(_model_config(case), seed))
    out, group = [None] * len(seqs), 16
    with torch.no_grad():
        for first in range(0, len(seqs), group):
            part = seqs[first:first + group]
            # causal: what follows a sequence's end changes nothing before it
            tokens = torch.zeros(len(part), max(map(len, part)), dtype=torch.int64)
            for i, s in enumerate(part):
                tokens[i, :len(s)] = torch.tensor(s)
            tokens = tokens.cuda()
            hidden = {"zidalix": _zidalix_hidden, "nufupel": _nufupel_hidden, "potodra": _potodra_hidden, "lerosun": _lerosun_hidden}
            x, head = _llama_hidden(c, seed, tokens) if w is None else hidden[case["model"]](c, w, tokens)
            for i, s in enumerate(part):
                y = x[i, len(s) - wanted[first + i]:len(s)] @ head
                cap = c.get("logit_softcap")
                out[first + i] = cap * torch.tanh(y / cap) if cap else y * c.get("logit_scale", 1.0)
    return torch.cat(out)
