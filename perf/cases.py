"""What this framework is used for, as a list of timed cases: single quantized Linears, the training-side pair of a LoRA layer,
quantized Llama and GPT-2 models that read prompts and decode, and the two decoders built from a list of layers.

Every case goes through `ruai_b200.nn`.  Weights are the library's seeded synthetic ones (normal, 0.02), quantized on the
device when a state is prepared; token ids are uniform; activations of single Linears are normal with a few large channels.
`exact` restates every path in float64 torch, on the GPU, from the definition of the synthetic weights.
"""
import math

import numpy as np
import torch

from ruai_b200 import nn

GROUP = 32  # rows of an int4 scale group

LLAMAS = {  # vocabulary, width, feed-forward, heads, key heads, head width, rotation base, tied head, layers of the real model
    "8b": dict(V=128256, d=4096, ff=14336, H=32, KV=8, hd=128, theta=500000.0, tied=0, L=32),
    "1.1b": dict(V=32000, d=2048, ff=5632, H=32, KV=4, hd=64, theta=10000.0, tied=0, L=22),
    "135m": dict(V=49152, d=576, ff=1536, H=9, KV=3, hd=64, theta=10000.0, tied=1, L=30),
}
GPT2 = dict(V=50257, n_pos=1024, d=768, L=12, H=12)
ZAZASUN = {  # layers by the kind of their token mixer, width, and the mixers' sizes
    "1b": dict(V=32000, d=2048, ff=5632, attention=dict(heads=16, kv_heads=4, dim=64, vdim=128), wkv=dict(heads=32, dim=64), hgrn2=dict(heads=16, dim=128, vdim=128)),
    "8b": dict(V=128256, d=4096, ff=14336, attention=dict(heads=16, kv_heads=4, dim=128, vdim=256), wkv=dict(heads=64, dim=64), hgrn2=dict(heads=32, dim=128, vdim=128)),
}
LOTORAX = {
    "1b": dict(V=32000, d=2048, ff=5632, eff=1408, latent=dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512), delta=dict(heads=16, kv_heads=8, dim=128, vdim=128, conv=4)),
    "8b": dict(V=128256, d=4096, ff=14336, eff=2048, latent=dict(heads=32, dim=128, rot_dim=64, vdim=128, kv_rank=512), delta=dict(heads=32, kv_heads=16, dim=128, vdim=128, conv=4)),
}
EXPERTS, TOP, RANK, WINDOW, KEEP, POSITIONS = 32, 4, 64, 1024, 4, 4096


def listed():
    return [
        # the smallest call: one token through one square Linear, the micro benchmark of quantized matvecs
        dict(name="linear-int8-1row", kind="linear", bits=8, m=1, k=2048, n=2048, dtype="f32", bias=False),
        # a few dozen rows of half-precision activations, nothing a multiple of a tile
        dict(name="linear-int4-ragged", kind="linear", bits=4, m=37, k=1504, n=1500, dtype="f16", bias=True),
        # the largest Linear: the gate of an 8B-shaped layer over four thousand tokens
        dict(name="linear-int4-4096rows", kind="linear", bits=4, m=4096, k=4096, n=14336, dtype="f32", bias=False),
        # fine-tuning on a frozen quantized base: forward with the adapter, gradient of the activations
        dict(name="lora-int4-256rows", kind="lora", bits=4, m=256, k=2048, n=2048, rank=16),
        # a short prompt continued greedily by GPT-2 small, and the prompt's own logits
        dict(name="gpt2-int8-generate", kind="generate", model="gpt2", bits=8, prompt=16, new=32, temperature=0.0, top_k=0, top_p=1.0),
        # sixteen users of the smallest Llama, a few steps each with the ids on the device
        dict(name="135m-int4-b16-steps", kind="steps", model="135m", layers=30, bits=4, B=16, ctx=256, new=8),
        # one user of the 8B shape deep in a conversation (an eighth of the layers)
        dict(name="8b-int4-b1-steps", kind="steps", model="8b", layers=4, bits=4, B=1, ctx=1024, new=8),
        # a serving batch
        dict(name="1.1b-int8-b64-steps", kind="steps", model="1.1b", layers=22, bits=8, B=64, ctx=256, new=4),
        # a chat turn: prompt of 512 tokens, then a few tokens whose logits the host reads
        dict(name="1.1b-int4-serve", kind="serve", model="1.1b", layers=22, bits=4, B=1, prompt=512, new=16),
        # a long prompt on the 8B shape: time to the first token
        dict(name="8b-int8-prompt", kind="serve", model="8b", layers=4, bits=8, B=1, prompt=2000, new=0),
        # the layer-list decoders in bf16: a long prompt, then a few tokens
        dict(name="zazasun-8b-serve", kind="zazasun", shape="8b", stack="attention,wkv,hgrn2", dtype="bfloat16", prompt=2048, new=4),
        dict(name="lotorax-1b-serve", kind="lotorax", shape="1b", stack="delta-dense,latent-moe,latent-dense,delta-moe", loop=True, dtype="bfloat16", prompt=1024, new=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "lora", "generate", "steps", "steps", "serve", "serve", "zazasun", "lotorax"])
    bits = rng.choice([8, 4])
    if kind == "linear":
        k = _log(rng, 16, 448) * 32 if bits == 4 else _log(rng, 512, 14336)
        n = _log(rng, 512, 14336)
        return dict(kind=kind, bits=bits, m=min(_log(rng, 1, 4096), 4096 * 4096 * 14336 // (k * n)), k=k, n=n, dtype=rng.choice(["f32", "f32", "f16", "bf16"]), bias=rng.random() < 0.5)
    if kind == "lora":
        return dict(kind=kind, bits=bits, m=_log(rng, 1, 512), k=_log(rng, 16, 128) * 32, n=_log(rng, 512, 4096), rank=rng.choice([4, 8, 16, 64]))
    if kind == "generate":
        sampled = rng.random() < 0.5
        return dict(kind=kind, model=rng.choice(["gpt2", "135m"]), bits=bits, prompt=_log(rng, 4, 256), new=_log(rng, 8, 48), temperature=0.8 if sampled else 0.0,
                    top_k=rng.choice([0, 40]) if sampled else 0, top_p=rng.choice([1.0, 0.9]) if sampled else 1.0)
    if kind in ("steps", "serve"):
        model = rng.choice(list(LLAMAS))
        layers = {"8b": rng.randint(1, 4), "1.1b": rng.randint(4, 22), "135m": rng.randint(10, 30)}[model]
        if kind == "steps":
            return dict(kind=kind, model=model, layers=layers, bits=bits, B=_log(rng, 1, 64), ctx=_log(rng, 32, 400), new=rng.randint(2, 8))
        B = rng.choice([1, 1, 1, 2, 5])
        return dict(kind=kind, model=model, layers=layers, bits=bits, B=B, prompt=_log(rng, 8, 2000 // B), new=rng.randint(0, 8))
    shape, stacks = rng.choice(["1b", "8b"]), ["attention", "wkv", "hgrn2"] if kind == "zazasun" else ["delta-dense", "latent-dense", "latent-moe", "delta-moe"]
    case = dict(kind=kind, shape=shape, stack=",".join(rng.choice(stacks) for _ in range(rng.randint(1, 3))), dtype="float32" if shape == "1b" and rng.random() < 0.3 else "bfloat16",
                prompt=_log(rng, 8, 2048), new=rng.randint(0, 6))
    return dict(case, loop=False) if kind == "lotorax" else case


# ---- states and passes ----------------------------------------------------------------------------------------------

_NP = {"f32": np.float32, "f16": np.float16, "bf16": np.uint16}
_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_DTYPE = {"f32": nn.F32, "f16": nn.F16, "bf16": nn.BF16}


class _Memory:
    """A device tensor of the library as torch sees it, without a copy."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": t.np_dtype.str, "data": (t.ptr.value, False), "version": 2}


def _view(t):
    v = torch.as_tensor(_Memory(t), device="cuda")
    return v.view(torch.bfloat16) if t.rdtype == nn.BF16 else v


def _normal(seed, salt, shape, std=1.0):
    g = torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return torch.randn(shape, generator=g, device="cuda") * std


def _activations(seed, salt, m, k):
    """Normal, with one channel in a hundred ten times as large."""
    x = _normal(seed, salt, (m, k))
    big = torch.from_numpy(np.random.RandomState((int(seed) + salt) % (1 << 31)).rand(k) < 0.01).to(x.device)
    return torch.where(big, x * 10.0, x)


def _put(dev, x, dtype="f32"):
    x = x.to(_TORCH[dtype])
    a = (x.view(torch.int16) if dtype == "bf16" else x).cpu().numpy()
    return nn.Tensor.from_numpy(dev, a.view(_NP[dtype]), _DTYPE[dtype])


def _ids(seed, salt, shape, vocab):
    return np.random.RandomState((int(seed) * 7919 + salt) % (1 << 31)).randint(0, vocab, shape).astype(np.int32)


def _vocab(case):
    return GPT2["V"] if case.get("model") == "gpt2" else (LLAMAS[case["model"]] if "model" in case else (ZAZASUN if case["kind"] == "zazasun" else LOTORAX)[case["shape"]])["V"]


def _model(dev, case, seed):
    if case["model"] == "gpt2":
        m = nn.GPT2(dev, nn.GPT2Config(GPT2["V"], GPT2["n_pos"], GPT2["d"], GPT2["L"], GPT2["H"]))
    else:
        c = LLAMAS[case["model"]]
        m = nn.Llama(dev, nn.LlamaConfig(c["V"], c["d"], c["ff"], case.get("layers", c["L"]), c["H"], c["KV"], c["hd"], 2048, 1e-5, c["theta"], c["tied"]))
    m.load_synthetic(_seed(seed), case["bits"], GROUP)
    return m


def _seed(seed):
    return int(seed) % (1 << 31)


def prepare(case, seed):
    dev, kind = nn.Device.cuda(0), case["kind"]
    if kind in ("linear", "lora"):
        k, n = case["k"], case["n"]
        w = _normal(seed, 1, (k, n), 0.02).cpu().numpy()
        bias = _normal(seed, 2, (n,)).cpu().numpy() if case.get("bias") else None
        x = _put(dev, _activations(seed, 3, case["m"], k), case.get("dtype", "f32"))
        if kind == "linear":
            lin = nn.Linear(dev, w, bias)
            lin.quantize_int8() if case["bits"] == 8 else lin.quantize_int4(GROUP)
            return dict(kind=kind, lin=lin, x=x)
        base = nn.QWeight.int8(dev, *nn.quantize_int8_device(dev, w)) if case["bits"] == 8 else nn.QWeight.int4(dev, *nn.quantize_int4_device(dev, w, GROUP), GROUP)
        return dict(kind=kind, base=base, x=x, a=_put(dev, _normal(seed, 4, (k, case["rank"]), k ** -0.5)), b=_put(dev, _normal(seed, 5, (case["rank"], n), 0.02)),
                    g=_put(dev, _normal(seed, 6, (case["m"], n))), scale=16.0 / case["rank"])
    V = _vocab(case)
    if kind == "generate":
        return dict(kind=kind, model=_model(dev, case, seed), prompt=_ids(seed, 1, (case["prompt"],), V), new=case["new"], temperature=case["temperature"], top_k=case["top_k"],
                    top_p=case["top_p"], seed=_seed(seed))
    if kind == "steps":  # the conversation so far is in the cache; every pass continues it from the same place
        m, B, ctx = _model(dev, case, seed), case["B"], case["ctx"]
        m.cache_reserve(B, ctx + case["new"] + 1)
        m.forward_cached(_ids(seed, 1, (B, ctx), V), want_logits=False)
        ids = _ids(seed, 2, (case["new"] + 1, B), V)
        return dict(kind=kind, model=m, B=B, ctx=ctx, ids=[nn.Tensor.from_numpy(dev, i) for i in ids[:-1]], last=ids[-1][:, None])
    if kind == "serve":
        m, B = _model(dev, case, seed), case["B"]
    else:
        m, B = _layer_list(dev, case, seed), 1
    m.cache_reserve(B, case["prompt"] + case["new"])
    return dict(kind="serve", model=m, prompt=_ids(seed, 1, (B, case["prompt"]), V), ids=_ids(seed, 2, (case["new"], B, 1), V))


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return _view(state["lin"].forward(state["x"]))
    if kind == "lora":
        y = nn.linear_lora_forward(state["x"], state["base"], state["a"], state["b"], state["scale"])
        return _view(y), _view(nn.matmul_q_grad_input(state["g"], state["base"]))
    m = state["model"]
    if kind == "generate":
        m.cache_clear()
        logits = m.forward_cached(state["prompt"][None, :])
        if state["temperature"] > 0:
            return logits, m.generate_sampled(state["prompt"], state["new"], state["temperature"], state["top_k"], state["top_p"], state["seed"])
        return logits, m.generate(state["prompt"], state["new"])
    if kind == "steps":
        m.cache_assume(state["B"], state["ctx"])
        picked = [m.decode_step(state["B"], i.ptr) for i in state["ids"]]
        return np.stack(picked), m.forward_cached(state["last"])
    m.cache_clear()
    return [m.forward_cached(state["prompt"])] + [m.forward_cached(i) for i in state["ids"]]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def _weight_bytes(k, n, bits):
    return k * n * bits / 8 + (4 * n if bits == 8 else 4 * n * (k // GROUP))


def work(case):
    kind = case["kind"]
    if kind in ("linear", "lora"):
        m, k, n, e = case["m"], case["k"], case["n"], {"f32": 4}.get(case.get("dtype", "f32"), 2)
        w, io = _weight_bytes(k, n, case["bits"]), m * (k + n) * e
        if kind == "linear":
            return {"bytes": w + io + (4 * n if case["bias"] else 0), "flops": 2.0 * m * k * n}
        return {"bytes": w + 2 * io + 4 * case["rank"] * (k + n), "flops": 4.0 * m * k * n + 2.0 * m * case["rank"] * (k + n)}
    passes = {"generate": [(1, 0, case.get("prompt"))] * 2 + [(1, case.get("prompt", 0) + i, 1) for i in range(case["new"] - 1)],
              "steps": [(case.get("B"), case.get("ctx", 0) + i, 1) for i in range(case["new"] + 1)]}.get(
        kind, [(case.get("B", 1), 0, case.get("prompt"))] + [(case.get("B", 1), case.get("prompt", 0) + i, 1) for i in range(case["new"])])
    total = {"bytes": 0.0, "flops": 0.0}
    for B, past, T in passes:
        if "model" in case:
            w, f, kv, at, V, d = _quantized_work(case)
        else:
            w, f, kv, at, V, d = _layer_list_work(case, B * T)
        keys = T * past + T * (T + 1) / 2  # pairs of a query and a key it sees
        total["bytes"] += w + B * ((past + 2 * T) * kv + 4 * T * d + 4 * V)
        total["flops"] += B * (T * f + at * keys + 2.0 * d * V)
    return total


def _quantized_work(case):
    """Weight bytes of a step, flops per token, cache bytes per position, attention flops per query and key, vocabulary, width."""
    if case["model"] == "gpt2":
        d, L, V, H, hd, kv = GPT2["d"], GPT2["L"], GPT2["V"], GPT2["H"], GPT2["d"] // GPT2["H"], GPT2["H"]
        shapes = [(d, 3 * d), (d, d), (d, 4 * d), (4 * d, d)]
    else:
        c = LLAMAS[case["model"]]
        d, L, V, H, hd, kv = c["d"], case.get("layers", c["L"]), c["V"], c["H"], c["hd"], c["KV"]
        shapes = [(d, (H + 2 * kv) * hd), (H * hd, d), (d, 2 * c["ff"]), (c["ff"], d)]
    return (L * sum(_weight_bytes(k, n, case["bits"]) for k, n in shapes) + _weight_bytes(d, V, 8), 2.0 * L * sum(k * n for k, n in shapes), 8.0 * L * kv * hd, 4.0 * L * H * hd, V, d)


def _layer_list_work(case, tokens):
    e = 2 if case["dtype"] == "bfloat16" else 4
    cfg = _layer_list_cfg(case)
    params = active = kv = at = 0.0
    for i in _schedule(cfg):
        layer, d = cfg["layers"][i], cfg["width"]
        m = layer["mixer"]
        hk, hv = m["heads"] * m["dim"], m["heads"] * m.get("vdim", m["dim"])
        if layer["type"] == "attention":
            p = d * (2 * hk + m["kv_heads"] * (2 * m["dim"] + m["vdim"]) + hv)
            kv += 4 * m["kv_heads"] * (2 * m["dim"] + m["vdim"])
            at += m["heads"] * (4 * m["dim"] + 4 * m["vdim"])
        elif layer["type"] == "wkv":
            p = d * 5 * hk + RANK * (d + hk)
        elif layer["type"] == "hgrn2":
            p = d * (2 * hk + 2 * hv)
        elif layer["type"] == "delta":
            p = d * (2 * m["kv_heads"] * m["dim"] + 3 * hv + 2 * m["heads"])
        else:
            p = d * (m["heads"] * (m["dim"] + m["rot_dim"] + 1) + m["kv_rank"] + m["rot_dim"] + hv) + m["kv_rank"] * (hk + hv)
            kv += 4 * (m["kv_rank"] + m["rot_dim"])
            at += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        mlp = layer["mlp"]
        one = 3 * d * mlp["ff"] if mlp["kind"] == "dense" else 3 * d * mlp["expert"]["ff"]
        used, stored = (1, 1) if mlp["kind"] == "dense" else (TOP, min(EXPERTS, TOP * tokens))
        params += p + one * stored
        active += p + one * used
    if cfg.get("loop"):
        params, active = params + 2 * cfg["loop"]["times"] * cfg["width"] ** 2, active + 2 * cfg["loop"]["times"] * cfg["width"] ** 2
    return e * (params + cfg["vocab"] * cfg["width"]), 2.0 * active, kv, at, cfg["vocab"], cfg["width"]


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 8e-3}[case["dtype"]]}
    if kind == "lora":
        return {"rel": 1e-5}
    if kind in ("generate", "steps"):  # a pick between two logits that agree to five digits may go either way
        return {"rel": 1e-4, "differ": 0.25 if kind == "generate" else 0.05}
    if kind == "serve":
        return {"rel": 1e-4}
    if case["dtype"] == "float32":
        return {"rel": 1e-4}
    if "moe" in case["stack"]:  # an expert more or less where two scores are nearly equal
        return {"rel": 3e-1}
    return {"rel": 4e-2 if kind == "zazasun" else 1e-1}


# ---- the layer-list decoders ----------------------------------------------------------------------------------------

def _layer_list_cfg(case):
    if case["kind"] == "zazasun":
        c = ZAZASUN[case["shape"]]
        at = c["attention"]
        mixers = {"attention": dict(at, mask=dict(size=WINDOW, keep_first=KEEP), scale=at["dim"] ** -0.5, diff=0.5), "wkv": c["wkv"], "hgrn2": c["hgrn2"]}
        layers = [{"type": k, "mixer": mixers[k], "mlp": {"ff": c["ff"], "kind": "dense"}} for k in case["stack"].split(",")]
        return {"architecture": "Zazasun", "layers": layers, "max_positions": POSITIONS, "norm": {"eps": 1e-5}, "vocab": c["V"], "width": c["d"]}
    c = LOTORAX[case["shape"]]
    lat = c["latent"]
    rot = dict(base=10000.0, dims=lat["rot_dim"], scaling=dict(factor=8.0, original=2048, fast=16.0, slow=1.0))
    mixers = {"latent": ("latent_attention", dict(lat, scale=(lat["dim"] + lat["rot_dim"]) ** -0.5, rot=rot)), "delta": ("delta", c["delta"])}
    mlps = {"dense": {"kind": "dense", "ff": c["ff"]}, "moe": {"kind": "moe", "expert": {"ff": c["eff"]}, "router": {"experts": EXPERTS, "top": TOP}}}
    layers = []
    for part in case["stack"].split(","):
        mix, mlp = part.split("-")
        layers.append({"type": mixers[mix][0], "mixer": mixers[mix][1], "mlp": mlps[mlp]})
    cfg = {"architecture": "Lotorax", "embedding": {"scale": c["d"] ** 0.5}, "layers": layers, "norm": {"eps": 1e-5}, "vocab": c["V"], "width": c["d"]}
    if case["loop"]:
        cfg["loop"] = {"start": 1, "stop": 3, "times": 2}
    return cfg


def _layer_list(dev, case, seed):
    cfg = _layer_list_cfg(case)
    m = nn.Zazasun(dev, nn.ZazasunConfig(cfg, RANK)) if case["kind"] == "zazasun" else nn.Lotorax(dev, nn.LotoraxConfig(cfg))
    m.load_synthetic(_seed(seed), case["dtype"])
    return m


def _schedule(cfg):
    n, loop = len(cfg["layers"]), cfg.get("loop")
    return list(range(n)) if not loop else list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def _named_tensors(case):
    """(name, rows, columns, standard deviation, constant) in the order that numbers them."""
    cfg, out = _layer_list_cfg(case), []
    d, zaza = cfg["width"], case["kind"] == "zazasun"

    def add(name, rows, cols, std=0.02, fill=0.0):
        out.append((name, rows, cols, std, fill))

    def norm(name):
        add(name, 1, d, 0.0, 1.0)
        add(name + ".b", 1, d, 0.0, 0.0)

    add("embed", cfg["vocab"], d)
    if zaza:
        add("pos", cfg["max_positions"], d)
    elif cfg.get("loop"):
        add("loop.in", d, 2 * d)
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        x, H, dim, vdim = p + "mix.", m["heads"], m["dim"], m.get("vdim", m["dim"])
        if zaza:
            add(p + "norm1", 1, 1, 0.0, 1.0)
            add(p + "shift", 1, d, 0.0, 0.5)
        else:
            norm(p + "norm1")
            norm(p + "norm1b")
        if layer["type"] == "attention":
            for n, rows in (("q", 2 * H * dim), ("k", 2 * m["kv_heads"] * dim), ("v", m["kv_heads"] * vdim)):
                add(x + n, rows, d)
            for n in ("q.norm", "k.norm"):
                add(x + n, 1, dim, 0.0, 1.0)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                add(x + n, 1, dim, 0.1)
        elif layer["type"] == "wkv":
            for n in "rkvgw":
                add(x + "mu." + n, 1, d, 0.0, 0.5)
            for n in "rkvg":
                add(x + n, H * dim, d)
            add(x + "w1", RANK, d)
            add(x + "w2", H * dim, RANK)
            add(x + "w0", 1, H * dim, 0.0, -2.0)
            add(x + "u", H, dim, 0.3)
            add(x + "norm", 1, H * dim, 0.0, 1.0)
        elif layer["type"] == "hgrn2":
            add(x + "q", H * dim, d)
            add(x + "f", H * dim, d)
            add(x + "f.b", 1, H * dim, 0.0, 1.0)
            add(x + "lower", 1, H * dim, 0.0, 0.5)
            add(x + "v", H * vdim, d)
            add(x + "norm", 1, vdim, 0.0, 1.0)
        elif layer["type"] == "latent_attention":
            add(x + "q", H * (dim + m["rot_dim"]), d)
            add(x + "dkv", m["kv_rank"] + m["rot_dim"], d)
            add(x + "dkv.norm", 1, m["kv_rank"], 0.0, 1.0)
            add(x + "uk", H * dim, m["kv_rank"])
            add(x + "uv", H * vdim, m["kv_rank"])
            add(x + "sink", 1, H, 0.5)
            add(x + "g", H, d)
        else:
            for n, rows in (("q", m["kv_heads"] * dim), ("k", m["kv_heads"] * dim), ("v", H * vdim)):
                add(x + n, rows, d)
                add(x + n + ".conv", rows, m["conv"], 0.5)
            add(x + "b", H, d)
            add(x + "a", H, d)
            add(x + "A_log", 1, H, 0.5)
            add(x + "dt_bias", 1, H, 0.0, -3.0)
            add(x + "norm", 1, vdim, 0.0, 1.0)
            add(x + "g", H * vdim, d)
        add(x + "o", d, H * vdim)
        if not zaza:
            norm(p + "norm2")
            norm(p + "norm2b")
        moe = mlp["kind"] == "moe"
        for e in range(EXPERTS if moe else 1):
            s, ff = p + "mlp." + (f"e{e}." if moe else ""), mlp["expert"]["ff"] if moe else mlp["ff"]
            add(s + "gate", ff, d)
            add(s + "up", ff, d)
            add(s + "down", d, ff)
        if moe:
            add(p + "mlp.router", EXPERTS, d)
            add(p + "mlp.correction", 1, EXPERTS, 0.0, 0.0)
    if zaza:
        add("final.norm", 1, 1, 0.0, 1.0)
    else:
        norm("final.norm")
    add("head", cfg["vocab"], d)
    return out


# ---- the same in float64 --------------------------------------------------------------------------------------------

_MASK = (1 << 64) - 1


def _i64(v):
    v &= _MASK
    return v - (1 << 64) if v >> 63 else v


def _mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & _MASK
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _MASK
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _MASK
    return z ^ (z >> 31)


def _synthetic(seed, tensor, rows, cols, std):
    """The library's synthetic normal tensor in float32: twelve 16-bit uniforms out of three hashes per element."""
    key, count = _mix64((_seed(seed) * 0xD6E8FEB86659FD93 + tensor) & _MASK), rows * cols
    mult = np.float32(std / 65535.99999237060546875)
    out = torch.empty(count, device="cuda")
    for at in range(0, count, 1 << 26):
        n = min(1 << 26, count - at)
        base = torch.arange(at, at + n, device="cuda", dtype=torch.int64).mul_(3).add_(_i64(key + 0x9E3779B97F4A7C15))
        s = torch.full((n,), -393210, device="cuda", dtype=torch.int64)
        for r in range(3):
            z = base + r
            z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * _i64(0xBF58476D1CE4E5B9)
            z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * _i64(0x94D049BB133111EB)
            z ^= (z >> 31) & ((1 << 33) - 1)
            for shift in (0, 16, 32, 48):
                s += (z >> shift) & 0xFFFF
        out[at : at + n] = s.to(torch.float32) * float(mult)
    return out.view(rows, cols)


def _dequantized(w, bits):
    """w [k, n] f32 through the int8 (column) or int4 (group of rows and column) quantizer and back, in float64."""
    k, n = w.shape
    g = w.view(1, k, n) if bits == 8 else w.view(k // GROUP, GROUP, n)
    top = 127.0 if bits == 8 else 7.0
    mx = g.abs().amax(1, keepdim=True)
    scale = torch.where(mx > 0, mx / torch.full_like(mx, top), torch.ones_like(mx))  # by a tensor: a scalar divisor may become a product with its inverse
    q = g / scale
    q = torch.sign(q) * torch.floor(q.abs().double() + 0.5)
    return (q.clamp(-127.0 if bits == 8 else -8.0, top) * scale.double()).view(k, n)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, eps):
    return (x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, keepdim=True, unbiased=False) + eps)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _softmax_values(q, k, v, scale, window=None, keep=0, sink=None):
    """q [H, T, e], k [G, T, e], v [G, T, f], heads in groups: causal, the last `window` positions and the first `keep`."""
    H, T, out = q.shape[0], q.shape[1], []
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    hidden = (j > i) | ((i - j >= window) & (j >= keep)) if window else j > i
    for h in range(H):
        g = h // (H // k.shape[0])
        s = (q[h] @ k[g].T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[g])
    return torch.stack(out)


def _exact_quantized(case, seed, ids, rows):
    """Logits [B, rows, V] of the token matrix ids [B, T] at some of its positions."""
    bits, gpt = case["bits"], case["model"] == "gpt2"
    c = dict(GPT2, KV=GPT2["H"], hd=64) if gpt else LLAMAS[case["model"]]
    d, L, V, H, KV, hd = c["d"], case.get("layers", c["L"]), c["V"], c["H"], c["KV"], c["hd"]
    B, T = ids.shape
    tok = torch.from_numpy(ids.astype(np.int64)).cuda()
    embed = _synthetic(seed, 0x10000000, V, d, 0.02)
    x = embed[tok].double()
    if gpt:
        x = x + _synthetic(seed, 0x10000002, c["n_pos"], d, 0.02)[:T].double()
    else:
        inv = (torch.tensor(c["theta"], dtype=torch.float32) ** (-torch.arange(0, hd, 2, dtype=torch.float32) / hd)).double().cuda()
        angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * inv
        cos, sin = torch.cat([angle.cos()] * 2, 1), torch.cat([angle.sin()] * 2, 1)

        def turn(t):
            return t * cos + torch.cat([-t[..., hd // 2 :], t[..., : hd // 2]], -1) * sin

    for l in range(L):
        def w(kind, k, n):
            return _dequantized(_synthetic(seed, 16 * l + kind, k, n, 0.02), bits)

        def b(kind, n):
            return _synthetic(seed, 16 * l + kind, 1, n, 0.02).double()

        h = _layer_norm(x, 1e-5) if gpt else _rms(x, 1e-5)
        if gpt:
            q, k, v = (h @ w(7, d, 3 * d) + b(11, 3 * d)).split(d, -1)
        else:
            q, k, v = h @ w(0, d, H * hd), h @ w(1, d, KV * hd), h @ w(2, d, KV * hd)
        q, k, v = (t.view(B, T, -1, hd).transpose(1, 2) for t in (q, k, v))
        if not gpt:
            q, k = turn(q), turn(k)
        a = torch.stack([_softmax_values(q[s], k[s], v[s], hd ** -0.5) for s in range(B)]).transpose(1, 2).reshape(B, T, H * hd)
        if gpt:
            x = x + a @ w(8, d, d) + b(12, d)
            x = x + _gelu(_layer_norm(x, 1e-5) @ w(9, d, 4 * d) + b(13, 4 * d)) @ w(10, 4 * d, d) + b(14, d)
        else:
            x = x + a @ w(3, H * hd, d)
            h = _rms(x, 1e-5)
            x = x + (_silu(h @ w(4, d, c["ff"])) * (h @ w(5, d, c["ff"]))) @ w(6, c["ff"], d)
    x = (_layer_norm if gpt else _rms)(x[:, rows], 1e-5)
    return x @ _dequantized(embed.T.contiguous() if gpt or c["tied"] else _synthetic(seed, 0x10000001, d, V, 0.02), 8)


def _exact_layer_list(case, seed, ids, rows):
    cfg, numbered = _layer_list_cfg(case), {t[0]: (i, t) for i, t in enumerate(_named_tensors(case))}
    eps, T, zaza = cfg["norm"]["eps"], len(ids), case["kind"] == "zazasun"

    def w(name, f32=False):
        i, (_, r, c, std, fill) = numbered[name]
        t = _synthetic(seed, 0x60000000 + i, r, c, float(np.float32(std))) if std else torch.full((r, c), fill, device="cuda")
        return t if f32 else t.double()

    def shifted(h, mu):
        return h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * mu

    def heads(t, n):
        return t.view(T, n, -1).transpose(0, 1)

    def mixer(h, layer, p):
        m = layer["mixer"]
        H, dim, vdim = m["heads"], m["dim"], m.get("vdim", m["dim"])
        if layer["type"] == "attention":
            G = m["kv_heads"]
            q = _rms((h @ w(p + "q").T).view(T, H, 2, dim), eps) * w(p + "q.norm")
            k = _rms((h @ w(p + "k").T).view(T, G, 2, dim), eps) * w(p + "k.norm")
            v = heads(h @ w(p + "v").T, G)
            lam = torch.exp((w(p + "lq1") * w(p + "lk1")).sum()) - torch.exp((w(p + "lq2") * w(p + "lk2")).sum()) + m["diff"]
            a = [_softmax_values(q[:, :, c].transpose(0, 1), k[:, :, c].transpose(0, 1), v, m["scale"], WINDOW, KEEP) for c in (0, 1)]
            o = _rms(a[0] - lam * a[1], eps) * (1.0 - m["diff"])
            return o.transpose(0, 1).reshape(T, H * vdim) @ w(p + "o").T
        if layer["type"] == "latent_attention":
            R = m["rot_dim"]
            q, dkv = heads(h @ w(p + "q").T, H), h @ w(p + "dkv").T
            c = _rms(dkv[:, : m["kv_rank"]], eps) * w(p + "dkv.norm")
            s = m["rot"]["scaling"]
            f = m["rot"]["base"] ** (-torch.arange(0, R, 2, device="cuda", dtype=torch.float64) / R)
            lo, hi = (R * math.log(s["original"] / (2 * math.pi * s[t])) / (2 * math.log(m["rot"]["base"])) for t in ("fast", "slow"))
            lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), R - 1)
            ramp = ((torch.arange(R // 2, device="cuda", dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
            angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * (f / s["factor"] * ramp + f * (1.0 - ramp))
            cos, sin = (0.1 * math.log(s["factor"]) + 1.0) * angle.cos(), (0.1 * math.log(s["factor"]) + 1.0) * angle.sin()

            def turn(t):
                u, v = t[..., 0::2], t[..., 1::2]
                return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)

            k = torch.cat([heads(c @ w(p + "uk").T, H), turn(dkv[:, m["kv_rank"] :]).expand(H, T, R)], -1)
            o = _softmax_values(torch.cat([q[..., :dim], turn(q[..., dim:])], -1), k, heads(c @ w(p + "uv").T, H), m["scale"], sink=w(p + "sink")[0])
            o = o * torch.sigmoid(h @ w(p + "g").T).T[:, :, None]
            return o.transpose(0, 1).reshape(T, H * vdim) @ w(p + "o").T
        o = torch.empty((T, H, vdim), device="cuda", dtype=torch.float64)
        S = torch.zeros((H, dim, vdim), device="cuda", dtype=torch.float64)
        if layer["type"] == "wkv":
            mix = {n: shifted(h, w(p + "mu." + n)) for n in "rkvgw"}
            r, k, v = ((mix[n] @ w(p + n).T).view(T, H, dim) for n in "rkv")
            decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).view(T, H, dim)
            u = w(p + "u")
            for t in range(T):
                kv = k[t, :, :, None] * v[t, :, None, :]
                o[t] = (r[t, :, :, None] * (S + u[:, :, None] * kv)).sum(1)
                S = decay[t, :, :, None] * S + kv
            return (_rms(o, eps).view(T, H * dim) * w(p + "norm") * _silu(mix["g"] @ w(p + "g").T)) @ w(p + "o").T
        if layer["type"] == "hgrn2":
            q, v, low = _silu(h @ w(p + "q").T).view(T, H, dim), (h @ w(p + "v").T).view(T, H, vdim), w(p + "lower")
            f = (low + (1.0 - low) * torch.sigmoid(h @ w(p + "f").T + w(p + "f.b"))).view(T, H, dim)
            for t in range(T):
                S = f[t, :, :, None] * S + (1.0 - f[t])[:, :, None] * v[t, :, None, :]
                o[t] = (q[t, :, :, None] * S).sum(1)
            return (_rms(o, eps) * w(p + "norm")).view(T, H * vdim) @ w(p + "o").T
        G, n = m["kv_heads"], m["conv"]

        def conv(name):
            x, taps = h @ w(p + name).T, w(p + name + ".conv")
            x = torch.cat([torch.zeros((n - 1, x.shape[1]), device="cuda", dtype=torch.float64), x])
            return _silu(sum(x[i : i + T] * taps[:, i] for i in range(n)))

        q, k = (conv(s).view(T, G, dim) for s in "qk")
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q * dim ** -0.5, k))
        v, beta = conv("v").view(T, H, vdim), torch.sigmoid(h @ w(p + "b").T)
        decay = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(h @ w(p + "a").T + w(p + "dt_bias")))
        for t in range(T):
            S = S * decay[t, :, None, None]
            S = S + k[t, :, :, None] * (beta[t, :, None] * (v[t] - (k[t, :, :, None] * S).sum(1)))[:, None, :]
            o[t] = (q[t, :, :, None] * S).sum(1)
        o = _rms(o, eps) * w(p + "norm") * _silu(h @ w(p + "g").T).view(T, H, vdim)
        return o.view(T, H * vdim) @ w(p + "o").T

    def gated(h, p, act):
        return (act(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T

    def feed_forward(h, layer, p):
        if layer["mlp"]["kind"] == "dense":
            return gated(h, p, _gelu if zaza else torch.relu)
        s = torch.sigmoid(h @ w(p + "router").T)
        chosen = torch.topk(s, TOP, -1).indices
        out = torch.zeros_like(h)
        for e in range(EXPERTS):
            t = (chosen == e).any(-1).nonzero()[:, 0]
            if len(t):
                out[t] += s[t, e, None] * gated(h[t], f"{p}e{e}.", _silu)
        return out

    x = w("embed", True)[torch.from_numpy(ids.astype(np.int64)).cuda()].double()
    if zaza:
        x = x + w("pos")[:T]
        for i in _schedule(cfg):
            p = f"l{i}."
            h = _rms(x, eps) * w(p + "norm1")
            x = x + mixer(shifted(h, w(p + "shift")), cfg["layers"][i], p + "mix.") + feed_forward(h, cfg["layers"][i], p + "mlp.")
        return _rms(x[rows], eps) @ w("head").T
    x = x0 = x * cfg["embedding"]["scale"]
    for i in _schedule(cfg):
        p = f"l{i}."
        if cfg.get("loop") and i == cfg["loop"]["start"]:
            x = torch.cat([x, x0], 1) @ w("loop.in").T
        x = x + _layer_norm(mixer(_layer_norm(x, eps), cfg["layers"][i], p + "mix."), eps)
        x = x + _layer_norm(feed_forward(_layer_norm(x, eps), cfg["layers"][i], p + "mlp."), eps)
    return _layer_norm(x[rows], eps) @ w("head").T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linear", "lora"):
        w = _dequantized(_normal(seed, 1, (case["k"], case["n"]), 0.02), case["bits"])
        x = _activations(seed, 3, case["m"], case["k"]).to(_TORCH[case.get("dtype", "f32")]).double()
        y = x @ w
        if kind == "linear":
            return y + _normal(seed, 2, (case["n"],)).double() if case["bias"] else y
        a, b = _normal(seed, 4, (case["k"], case["rank"]), case["k"] ** -0.5).double(), _normal(seed, 5, (case["rank"], case["n"]), 0.02).double()
        return y + (x @ a @ b) * (16.0 / case["rank"]), _normal(seed, 6, (case["m"], case["n"])).double() @ w.T
    V = _vocab(case)
    if kind == "generate":  # the picks have no 64-bit value
        return _exact_quantized(case, seed, _ids(seed, 1, (1, case["prompt"]), V), [-1])[:, 0], None
    if kind == "steps":
        ids = np.concatenate([_ids(seed, 1, (case["B"], case["ctx"]), V), _ids(seed, 2, (case["new"] + 1, case["B"]), V).T], 1)
        return None, _exact_quantized(case, seed, ids, [-1])[:, 0]
    B, T = case.get("B", 1), case["prompt"] + case["new"]
    ids, rows = np.concatenate([_ids(seed, 1, (B, case["prompt"]), V), _ids(seed, 2, (case["new"], B, 1), V)[:, :, 0].T], 1), list(range(case["prompt"] - 1, T))
    if kind == "serve":
        y = _exact_quantized(case, seed, ids, rows)
    elif case["dtype"] == "bfloat16" and "moe" in case["stack"]:
        return None  # which experts a token goes to is a choice that bf16 makes otherwise for one token in ten
    else:
        y = _exact_layer_list(case, seed, ids[0], rows)[None]
    return [y[:, i] for i in range(len(rows))]
