"""What a user of this library has it do, as cases that a timer can run: listed ones and drawn ones of the same ranges.

Six kinds of work, each through the public entry points of tl_b200:

  linear    quantized linear layers on their own (QTensor, Tensor.matmul_quantized), one to several hundred activation rows
  generate  one sequence decoded greedily in a session with a cached context (Decoder.generate)
  batch     several sequences decoded together, the caller choosing the tokens (Decoder.step_batch)
  prompt    a prompt run at once, the logits of a few of its tokens read (Decoder.prefill_logits)
  ops       the chatbot program's decode steps, one library call per op (chatbot.PerOpLlama)
  layered   a bf16 model described by a config.json: a prompt, then decode steps (Decoder on a TensorMap with a config)

Sizes are those of the repository's benchmark (TinyLlama-, Llama-3-8B- and 70B-shaped models, Mukutar and Rukedra at width 2048), with fewer
layers where whole models would take long to make.  Weights are random in genuine GGUF blocks, scaled as a trained model's: a
weight matrix keeps the size of what it multiplies, so attention spreads over its context and logits stay moderate.
"""
import json
import math
import random

import numpy as np
import torch

import tl_b200 as tl
from tl_b200 import synth
from tl_b200.chatbot import PerOpLlama

SHAPES = {"tiny": synth.TINYLLAMA, "8b": synth.LLAMA3_8B, "70b": synth.LLAMA3_70B}
TYPES = {"q4_0": synth.Q4_0, "q8_0": synth.Q8_0, "q4_k": synth.Q4_K, "q6_k": synth.Q6_K}
VOCABS = {"tiny": 32000, "8b": 32000, "70b": 16000}      # with few layers a whole head would outweigh them


def listed():
    return [
        # one token through a short stack of small layers, call by call: latency and launches are the time
        dict(name="linear-1row-2048", kind="linear", type="q4_k", rows=1, k=2048, n=2048, depth=4),
        # four tokens (a small batch, or a draft to check) through a wide layer: the streaming matvec at its widest
        dict(name="linear-4rows-q8", kind="linear", type="q8_0", rows=4, k=4096, n=14336, depth=1),
        # sixteen rows through the largest matrix there is, an output head
        dict(name="linear-16rows-head", kind="linear", type="q4_k", rows=16, k=4096, n=128256, depth=1),
        # a prompt's rows through a feed-forward projection: the tensor-core product
        dict(name="linear-512rows", kind="linear", type="q4_k", rows=512, k=4096, n=14336, depth=1),
        # a chat with the small model: short context, f32 cache, the whole depth
        dict(name="generate-tiny", kind="generate", shape="tiny", layers=22, vocab=32000, type="q4_0", head="q4_0", kv_f16=False, context=128, steps=32),
        # a chat with the 8B model: 2048 cached tokens, f16 cache, its whole vocabulary
        dict(name="generate-8b", kind="generate", shape="8b", layers=8, vocab=128256, type="q4_k", head="q6_k", kv_f16=True, context=2048, steps=16),
        # a server's step over sixteen sequences
        dict(name="batch-16-8b", kind="batch", shape="8b", layers=4, vocab=32000, type="q4_k", head="q6_k", kv_f16=True, context=1024, steps=8, batch=16),
        # a long prompt of the 8B model
        dict(name="prompt-2048-8b", kind="prompt", shape="8b", layers=4, vocab=32000, type="q4_k", head="q6_k", kv_f16=True, tokens=2048, rows=4),
        # a question of a few hundred tokens to the small model: a ragged length, heads of 64, f32 cache
        dict(name="prompt-333-tiny", kind="prompt", shape="tiny", layers=8, vocab=32000, type="q8_0", head="q8_0", kv_f16=False, tokens=333, rows=4),
        # the program as its compiler emits it, one call per op, a cache that grows by concatenation
        dict(name="ops-tiny", kind="ops", shape="tiny", layers=4, vocab=32000, type="q4_0", head="q4_0", context=512, steps=4),
        # a question and the beginning of its answer, two layers of each Mukutar mixer
        dict(name="mukutar-answer", kind="layered", model="mukutar", width=2048, heads=16, ff=5632, layers=6, vocab=32768, window=4096, prompt=512, steps=16),
        # the same with one layer of each Rukedra mixer, dense and expert feed-forwards; a ragged prompt
        dict(name="rukedra-answer", kind="layered", model="rukedra", width=2048, heads=16, ff=5632, layers=3, vocab=32768, window=4096, prompt=509, steps=16),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over their logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "generate", "batch", "prompt", "ops", "layered"])
    if kind == "linear":
        k = 256 * _log(rng, 4, 56)
        c = dict(kind=kind, type=rng.choice(sorted(TYPES)), rows=_log(rng, 1, 512), k=k, n=k, depth=1)
        if rng.random() < 0.25:
            c["depth"] = rng.randint(2, 4)
        else:
            c["n"] = _log(rng, 1000, 32000)
        return c
    if kind == "layered":
        return dict(kind=kind, model=rng.choice(["mukutar", "rukedra"]), width=rng.choice([1024, 1536, 2048]), heads=rng.choice([8, 12, 16]), ff=256 * rng.randint(8, 22),
                    layers=3, vocab=32768, window=rng.choice([256, 4096]), prompt=_log(rng, 24, 800), steps=rng.randint(2, 16))
    shape = rng.choice(["tiny", "tiny", "8b"] if kind == "ops" else ["tiny", "8b", "70b"])
    c = dict(kind=kind, shape=shape, layers=1 if shape == "70b" else rng.randint(2, 4), vocab=VOCABS[shape], type=rng.choice(["q4_0", "q8_0", "q4_k", "q6_k"]))
    c["head"] = "q6_k" if c["type"] == "q4_k" else c["type"]
    if kind == "ops":
        return dict(c, context=_log(rng, 16, 1500), steps=rng.randint(1, 4))
    c["kv_f16"] = rng.random() < 0.67
    if kind == "prompt":
        return dict(c, tokens=_log(rng, 17, 1024 if shape == "70b" else 2048), rows=rng.randint(1, 4))
    if kind == "batch":
        return dict(c, context=_log(rng, 16, 1500), steps=rng.randint(2, 8), batch=rng.randint(2, 16))
    return dict(c, context=_log(rng, 16, 4000), steps=rng.randint(4, 24))


# ---- inputs -------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _blocks(gen, t, n, k, std):
    """Random GGUF blocks of an [n, k] matrix whose values have about this standard deviation, as bytes on the GPU."""
    per, nb = synth.BLOCK[t]
    count = n * k // per
    out = torch.randint(0, 256, (count, nb), dtype=torch.uint8, device="cuda", generator=gen)

    def scale(by, at):
        d = (by * (0.5 + torch.rand(count, 1, device="cuda", generator=gen))).half()
        out[:, at:at + 2] = d.view(torch.uint8)
        return d

    if t == synth.Q4_0:
        scale(std / 4.6, 0)
    elif t == synth.Q8_0:
        scale(std / 74, 0)
    elif t == synth.Q4_K:                      # minima of 7.5 steps, so that the values lie around zero
        out[:, 2:4] = (scale(std / 167, 0).float() * 7.5).half().view(torch.uint8)
        out[:, 8:12] = out[:, 4:8]
        out[:, 12:16] = (out[:, 12:16] & 15) * 17
    else:
        scale(std / 1350, 208)
    return out


def _host(t):
    return t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy()


def _tokens(seed, count, vocab):
    rng = random.Random(seed * 7919 + count)
    return [rng.randrange(vocab) for _ in range(count)]


def _llama_cfg(case):
    return dict(SHAPES[case["shape"]], n_layers=case["layers"], vocab=case["vocab"])


def _llama_parts(case, gen):
    """(name, type, shape, bytes on the GPU) of every tensor, in the order they are drawn."""
    cfg = _llama_cfg(case)
    for name, t, shape in synth.llama_tensor_specs(cfg, TYPES[case["type"]], TYPES[case["head"]], synth.Q8_0):
        if len(shape) == 1:
            yield name, t, shape, 1.0 + 0.1 * torch.randn(shape[0], device="cuda", generator=gen)
        else:
            yield name, t, shape, _blocks(gen, t, shape[0], shape[1], 1.0 if name.startswith("token_embd") else shape[1] ** -0.5)


def _context(case, gen, cfg):
    """Cached keys and values [tokens, KV heads * head size] of one sequence and layer, values that f16 holds."""
    shape = (2, case["context"], cfg["n_kv_heads"] * cfg["head_dim"])
    return torch.randn(shape, device="cuda", generator=gen).half().float()


def _layered_cfg(case):
    W, heads, window = case["width"], case["heads"], case["window"]
    if case["model"] == "mukutar":
        mix = [("retention", dict(heads=heads, dim=128, vdim=128, rot=dict(base=10000.0, dims=128), decay=[1.0 - 2.0 ** (-5 - 6 * i / heads) for i in range(heads)])),
               ("general_delta", dict(heads=heads, dim=128)),
               ("attention", dict(heads=heads, kv_heads=heads // 4, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=window)))]
        ffn = [dict(kind="dense", ff=case["ff"])]
        extra = dict(architecture="Mukutar", norm=dict(eps=1e-5))
    else:
        lat = dict(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5,
                   rot=dict(base=10000.0, dims=64, scaling=dict(factor=8.0, original=4096, fast=32.0, slow=1.0)))
        mix = [("latent_attention_2", lat), ("latent_attention", dict(lat, q_rank=768, mask=dict(size=window))), ("mingru", dict(width=W))]
        e = case["ff"] // 4
        ffn = [dict(kind="dense", ff=case["ff"]),
               dict(kind="moe", expert=dict(ff=e), shared=dict(ff=2 * e), router=dict(experts=64, top=6, scale=2.5, groups=dict(count=8, keep=3)))]
        extra = dict(architecture="Rukedra", norm=dict(eps=1e-6, groups=2), logit_softcap=30.0)
    return dict(extra, vocab=case["vocab"], width=W,
                layers=[dict(type=mix[i % 3][0], mixer=mix[i % 3][1], mlp=ffn[i % len(ffn)]) for i in range(case["layers"])])


def _layered_parts(case, gen):
    """(name, bf16 values on the GPU) of every tensor; spreads as synth.mukutar_tensor and synth.rukedra_tensor give them."""
    cfg, muk = _layered_cfg(case), case["model"] == "mukutar"
    for name, shape in (synth.mukutar_specs(cfg, rank=128) if muk else synth.rukedra_specs(cfg)).items():
        x = torch.randn(shape, device="cuda", generator=gen)
        leaf = name.split(".", 1)[-1]
        if len(shape) == 2:
            x = x if name == "embed" else x * ((3.0 if name.endswith("router") else 1.0) * shape[1] ** -0.5)
        elif not muk:
            x = 0.5 * x if name.endswith(".b") else 1.0 + 0.2 * x
        elif leaf.startswith("ls"):
            x = 0.5 + 0.1 * x
        elif leaf in ("mix.r1", "mix.r2"):
            x = 0.2 + 0.3 * x.abs()
        elif leaf == "mix.norm":
            x = 1.0 + 0.1 * x
        elif leaf == "mlp.act":
            x = 0.5 + 0.3 * x
        elif leaf not in ("mix.sink", "mix.w0", "mix.a.b"):
            x = 0.1 * x
        yield name, x.bfloat16()


def prepare(case, seed):
    tl.init(0)
    gen, kind = _gen(seed), case["kind"]
    if kind == "linear":
        t = TYPES[case["type"]]
        ws = [tl.QTensor.from_gguf_bytes(t, case["n"], case["k"], _host(_blocks(gen, t, case["n"], case["k"], case["k"] ** -0.5))) for _ in range(case["depth"])]
        x = tl.Tensor.from_numpy(torch.randn(case["rows"], case["k"], device="cuda", generator=gen).cpu().numpy())
        return dict(case=case, x=x, weights=ws)
    wmap = tl.TensorMap.new()
    if kind == "layered":
        cfg = _layered_cfg(case)
        for name, x in _layered_parts(case, gen):
            wmap.add(name, synth.BF16, tuple(x.shape), _host(x))
        wmap.set_config(json.dumps(cfg))
        dec = tl.Decoder(None, wmap, max_seq=case["prompt"] + case["steps"])
        return dict(case=case, map=wmap, dec=dec, tokens=_tokens(seed, case["prompt"] + case["steps"], case["vocab"]))
    cfg = _llama_cfg(case)
    for name, t, shape, data in _llama_parts(case, gen):
        wmap.add(name, t, shape, _host(data))
    s = dict(case=case, map=wmap)
    if kind == "prompt":
        s["tokens"] = _tokens(seed, case["tokens"], case["vocab"])
        s["want"] = _want(case)
        s["dec"] = tl.Decoder(cfg, wmap, kv_f16=case["kv_f16"], max_seq=case["tokens"])
    elif kind == "ops":
        s["tokens"] = _tokens(seed, case["steps"], case["vocab"])
        s["dec"] = PerOpLlama(cfg, wmap, max_seq=case["context"] + case["steps"])
        s["past"] = []
        for layer in range(case["layers"]):
            k, v = _context(case, gen, cfg).cpu().numpy()
            s["dec"].seed_cache(layer, k, v)
            s["past"].append((s["dec"].cache.get_k(layer), s["dec"].cache.get_v(layer)))
    else:
        B = case.get("batch", 1)
        s["tokens"] = _tokens(seed, B * case["steps"] if kind == "batch" else 1, case["vocab"])
        s["dec"] = tl.Decoder(cfg, wmap, kv_f16=case["kv_f16"], max_seq=case["context"] + case["steps"], batch=B)
        for b in range(B):
            for layer in range(case["layers"]):
                k, v = _context(case, gen, cfg).cpu().numpy()
                if kind == "batch":
                    s["dec"].kv_write_seq(b, layer, 0, k, v)
                else:
                    s["dec"].kv_write(layer, 0, k, v)
    return s


def _want(case):
    """The places whose logits are read: the last token, and others evenly before it."""
    n, r = case["tokens"], case["rows"]
    return [n * (i + 1) // r - 1 for i in range(r)]


class _Device:
    """A library tensor as what torch takes without a copy."""

    def __init__(self, t, shape):
        self.t = t
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(tl.lib().tlb_tensor_data(t.h), False), version=3)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "linear":
        y = s["x"].matmul_quantized(s["weights"][0])
        for w in s["weights"][1:]:
            y = y.rms_norm(None, 1e-5).matmul_quantized(w)
        return torch.as_tensor(_Device(y, (c["rows"], c["n"])), device="cuda")
    d, toks = s["dec"], s["tokens"]
    if kind == "generate":
        out = d.generate(toks[0], c["context"], c["steps"])
        return dict(tokens=np.array(out, dtype=np.int64), logits=d.logits())
    if kind == "batch":
        B = c["batch"]
        for i in range(c["steps"]):
            d.step_batch(toks[i * B:(i + 1) * B], [c["context"] + i] * B)
        return dict(logits=d.logits_batch())
    if kind == "prompt":
        return dict(logits=d.prefill_logits(toks, 0, want=s["want"]))
    if kind == "ops":
        for layer, (k, v) in enumerate(s["past"]):
            d.cache.update(layer, k, v)
        for i, t in enumerate(toks):
            d.step_native([t], c["context"] + i)
        return dict(logits=torch.as_tensor(_Device(d.last_logits, (1, c["vocab"])), device="cuda"))
    n = c["prompt"]
    first = d.prefill_logits(toks[:n], 0, want=[n - 1])
    for i in range(n, n + c["steps"]):
        d.step(toks[i], i)
    return dict(first=first, last=d.logits())


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _llama_linear(cfg):
    """Weights of one layer's matrices."""
    d, qd, kvd = cfg["d_model"], cfg["n_heads"] * cfg["head_dim"], cfg["n_kv_heads"] * cfg["head_dim"]
    return d * (qd + 2 * kvd) + qd * d + 3 * d * cfg["ffn"]


def work(case):
    kind = case["kind"]
    if kind == "linear":
        per, r = synth.bytes_per_weight(TYPES[case["type"]]), case["rows"]
        return dict(bytes=case["depth"] * case["n"] * case["k"] * per + 4 * r * (case["k"] + case["n"]), flops=2.0 * case["depth"] * r * case["n"] * case["k"])
    if kind == "layered":
        cfg = _layered_cfg(case)
        specs = synth.mukutar_specs(cfg, rank=128) if case["model"] == "mukutar" else synth.rukedra_specs(cfg)
        size = {n: int(np.prod(s)) for n, s in specs.items() if n != "embed"}
        all_w = float(sum(size.values()))
        used, head = all_w, float(size["head"])
        for lay in cfg["layers"]:
            if lay["mlp"]["kind"] == "moe":                     # a token's own experts among the stored ones
                r = lay["mlp"]["router"]
                used -= 3.0 * case["width"] * lay["mlp"]["expert"]["ff"] * (r["experts"] - r["top"])
        n, steps = case["prompt"], case["steps"]
        return dict(bytes=2 * (all_w + used * steps), flops=2.0 * ((used - head) * (n + steps) + head * (1 + steps)))
    cfg = _llama_cfg(case)
    per, lin, head = synth.bytes_per_weight(TYPES[case["type"]]), case["layers"] * _llama_linear(cfg), case["vocab"] * cfg["d_model"]
    head_b, kvd = head * synth.bytes_per_weight(TYPES[case["head"]]), cfg["n_kv_heads"] * cfg["head_dim"]
    elem = 2 if case.get("kv_f16") else 4
    if kind == "prompt":
        n = case["tokens"]
        att = 4.0 * case["layers"] * cfg["n_heads"] * cfg["head_dim"] * n * (n + 1) / 2
        return dict(bytes=lin * per + head_b + 2 * case["layers"] * n * kvd * elem + 4 * n * cfg["d_model"] + 4 * case["rows"] * case["vocab"],
                    flops=2.0 * n * lin + att + 2.0 * case["rows"] * head)
    B, steps, mid = case.get("batch", 1), case["steps"], case["context"] + case["steps"] / 2
    kv = 2.0 * case["layers"] * kvd * elem * mid * B
    return dict(bytes=steps * (lin * per + head_b + kv + 4 * B * case["vocab"]),
                flops=steps * B * (2.0 * (lin + head) + 4.0 * case["layers"] * cfg["n_heads"] * cfg["head_dim"] * mid))


def tolerance(case):
    """About four times the error against 64 bits that each precision shows."""
    kind = case["kind"]
    if kind == "linear":                       # one row: 23-bit activations; two to four: 16 bits; above: f16
        return {"rel": 1e-5 if case["rows"] == 1 else 1.6e-4 if case["rows"] <= 4 else 2e-3}
    if kind in ("generate", "ops"):            # f32 throughout, or f16 cache rows
        return {"rel": 1e-3 if case.get("kv_f16") else 1e-5}
    return {"rel": 2e-2 if kind == "layered" else 4e-3}      # bf16 operands; f16 operands


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _values(raw, t):
    """GGUF blocks (bytes on the GPU) -> float64 values, one block per row."""
    f16 = lambda at: raw[:, at:at + 2].contiguous().view(torch.float16).double()
    if t == synth.Q4_0:
        q = raw[:, 2:]
        return f16(0) * (torch.cat([q & 15, q >> 4], 1).double() - 8)
    if t == synth.Q8_0:
        return f16(0) * raw[:, 2:].contiguous().view(torch.int8).double()
    if t == synth.Q4_K:
        s = raw[:, 4:16].int()
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], 1).double()
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)], 1).double()
        q = raw[:, 16:].reshape(-1, 4, 32)
        q = torch.stack([q & 15, q >> 4], 2).reshape(-1, 8, 32).double()
        return ((f16(0) * sc)[:, :, None] * q - (f16(2) * mn)[:, :, None]).reshape(-1, 256)
    lo, hi, sc = raw[:, :128].reshape(-1, 2, 2, 32), raw[:, 128:192].reshape(-1, 2, 1, 32), raw[:, 192:208].contiguous().view(torch.int8)
    q = torch.cat([lo & 15, lo >> 4], 2).int()                            # [block, half, quarter, 32]
    q = q | torch.cat([(hi >> s) & 3 for s in (0, 2, 4, 6)], 2).int() << 4
    return ((f16(208) * sc.double())[:, :, None] * (q.reshape(-1, 16, 16) - 32).double()).reshape(-1, 256)


def _rms(x, eps):
    return x / torch.sqrt(torch.mean(x * x, -1, keepdim=True) + eps)


def _turn_pairs(x, pos, speeds, gain=1.0):
    """x [tokens, heads, dim]: neighbours as complex numbers, turned by position * speed."""
    a = pos.double()[:, None, None] * speeds
    u, v, c, s = x[..., 0::2], x[..., 1::2], gain * torch.cos(a), gain * torch.sin(a)
    return torch.stack([u * c - v * s, u * s + v * c], -1).flatten(-2)


def _attend(q, k, v, scale, window=None, bias=None, sink=None):
    """q [n, H, d] are the last n of the tokens of k [T, H, d], v [T, H, dv]."""
    n, T = q.shape[0], k.shape[0]
    dist = torch.arange(T - n, T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    out = dist < 0
    if window is not None:
        out = out | (dist >= window)
    o = torch.empty(n, q.shape[1], v.shape[2], dtype=torch.float64, device="cuda")
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h].T * scale
        if bias is not None:
            s = s - bias[0][h] * torch.log1p(bias[1][h] * dist.clamp(min=0))
        s = s.masked_fill(out, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        o[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, h]
    return o


class _Llama:
    def __init__(self, case, gen):
        self.cfg = _llama_cfg(case)
        self.w = {n: (x.double() if len(shape) == 1 else _values(x, t).reshape(shape)) for n, t, shape, x in _llama_parts(case, gen)}

    def forward(self, tokens, pos0, past):
        """past: a list of [2, tokens, KV heads, head size] per layer, extended in place; logits of every new token."""
        c, w = self.cfg, self.w
        H, G, D, n = c["n_heads"], c["n_kv_heads"], c["head_dim"], len(tokens)
        pos = torch.arange(pos0, pos0 + n, device="cuda")
        speeds = float(c["rope_base"]) ** (-2.0 * torch.arange(D // 2, device="cuda", dtype=torch.float64) / D)
        x = w["token_embd.weight"][torch.tensor(tokens, device="cuda")]
        for i in range(c["n_layers"]):
            p = "blk.%d." % i
            h = _rms(x, c["eps"]) * w[p + "attn_norm.weight"]
            q, k, v = ((h @ w[p + "attn_%s.weight" % a].T).reshape(n, -1, D) for a in "qkv")
            new = torch.stack([_turn_pairs(k, pos, speeds), v])
            past[i] = new if past[i] is None else torch.cat([past[i], new], 1)
            kv = past[i].repeat_interleave(H // G, 2)
            x = x + _attend(_turn_pairs(q, pos, speeds), kv[0], kv[1], c["attn_scale"]).reshape(n, -1) @ w[p + "attn_output.weight"].T
            h = _rms(x, c["eps"]) * w[p + "ffn_norm.weight"]
            g = h @ w[p + "ffn_gate.weight"].T
            x = x + (g * torch.sigmoid(g) * (h @ w[p + "ffn_up.weight"].T)) @ w[p + "ffn_down.weight"].T
        return (_rms(x, c["eps"]) * w["output_norm.weight"]) @ w["output.weight"].T


def _mukutar(cfg, w, tokens):
    n, eps = len(tokens), cfg["norm"]["eps"]
    pos = torch.arange(n, device="cuda")
    norm = lambda x, name: _rms(x, eps) * (1.0 + w[name])
    x = w["embed"][torch.tensor(tokens, device="cuda")]
    for i, lay in enumerate(cfg["layers"]):
        p, m = "l%d." % i, lay["mixer"]
        q_, H, D = p + "mix.", m["heads"], m["dim"]
        h = norm(x, p + "norm1")
        lin = lambda name: h @ w[q_ + name].T
        if lay["type"] == "attention":
            q, k, v = ((lin(a) + w[q_ + a + ".b"]).reshape(n, -1, D) for a in "qkv")
            k, v = (t.repeat_interleave(H // m["kv_heads"], 1) for t in (k, v))
            o = _attend(q, k, v, m["scale"], m["mask"]["size"], (w[q_ + "r1"], w[q_ + "r2"]), w[q_ + "sink"]).reshape(n, -1)
        elif lay["type"] == "retention":
            half, rot = m["rot"]["dims"] // 2, m["rot"]
            a = pos.double()[:, None, None] * float(rot["base"]) ** (-2.0 * torch.arange(half, device="cuda", dtype=torch.float64) / rot["dims"])
            turn = lambda t: torch.cat([t[..., :half] * torch.cos(a) - t[..., half:2 * half] * torch.sin(a),
                                        t[..., half:2 * half] * torch.cos(a) + t[..., :half] * torch.sin(a), t[..., 2 * half:]], -1)
            q, k, v = turn(lin("q").reshape(n, H, D)), turn(lin("k").reshape(n, H, D)) * D ** -0.5, lin("v").reshape(n, H, -1)
            decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")
            dist = (pos[:, None] - pos[None]).double()
            o = torch.stack([torch.where(dist >= 0, decay[e] ** dist.clamp(min=0), 0.0) * (q[:, e] @ k[:, e].T) @ v[:, e] for e in range(H)], 1)
            g = lin("g")
            o = _rms(o, eps).reshape(n, -1) * g * torch.sigmoid(g)
        else:
            r, k, v = (lin(a).reshape(n, H, D) for a in "rkv")
            f = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(lin("w1")) @ w[q_ + "w2"].T + w[q_ + "w0"])).reshape(n, H, D, 1)
            a = torch.sigmoid(lin("a") + w[q_ + "a.b"]).reshape(n, H, D)
            u = k / torch.sqrt(torch.sum(k * k, -1, keepdim=True) + 1e-6)
            au = (a * u)[..., None]
            S, o = torch.zeros(H, D, D, dtype=torch.float64, device="cuda"), torch.empty_like(r)
            for t in range(n):
                seen = u[t][:, None, :] @ S
                S = f[t] * S - au[t] * seen + k[t][:, :, None] * v[t][:, None, :]
                o[t] = (r[t][:, None, :] @ S)[:, 0]
            o = _rms(o, eps).reshape(n, -1) * w[q_ + "norm"] * torch.sigmoid(lin("g"))
        x = x + w[p + "ls1"] * (o @ w[q_ + "o"].T)
        z = norm(x, p + "norm2") @ w[p + "mlp.up"].T
        a, b, c, e = w[p + "mlp.act"]
        x = x + w[p + "ls2"] * ((a * _rms(z, eps) + b * _rms(z * z, eps) + c * _rms(z ** 3, eps) + e) @ w[p + "mlp.down"].T)
    return norm(x, "final.norm") @ w["head"].T


def _turn_speeds(dims, base, s):
    i = torch.arange(dims // 2, device="cuda", dtype=torch.float64)
    f = float(base) ** (-2.0 * i / dims)
    where = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
    slow = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return slow * f / s["factor"] + (1.0 - slow) * f, 0.1 * math.log(s["factor"]) + 1.0


def _rukedra(cfg, w, tokens):
    n, eps, groups = len(tokens), cfg["norm"]["eps"], cfg["norm"]["groups"]
    pos = torch.arange(n, device="cuda")
    norm = lambda x, name: _rms(x.reshape(n, groups, -1), eps).reshape(n, -1) * w[name]
    silu = lambda z: z * torch.sigmoid(z)
    gelu = lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
    gated = lambda p, h, act: (act(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T
    x = w["embed"][torch.tensor(tokens, device="cuda")]
    for i, lay in enumerate(cfg["layers"]):
        p, m, f = "l%d." % i, lay["mixer"], lay["mlp"]
        q_ = p + "mix."
        h = norm(x, p + "norm1")
        if lay["type"] == "mingru":
            g, v = torch.sigmoid(h @ w[q_ + "z"].T + w[q_ + "z.b"]), h @ w[q_ + "x"].T + w[q_ + "x.b"]
            v = g * torch.where(v >= 0, v + 0.5, torch.sigmoid(v))
            S, o = torch.zeros_like(v[0]), torch.empty_like(v)
            for t in range(n):
                S = o[t] = (1.0 - g[t]) * S + v[t]
            y = o * silu(h @ w[q_ + "g"].T)
        else:
            H, d, R = m["heads"], m["dim"], m["kv_rank"]
            latent = lay["type"] == "latent_attention"
            q = (_rms(h @ w[q_ + "dq"].T, eps) * w[q_ + "dq.norm"]) @ w[q_ + "uq"].T if latent else h @ w[q_ + "q"].T
            q = q.reshape(n, H, -1)
            speeds, gain = _turn_speeds(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
            kv = h @ w[q_ + "dkv"].T
            c = _rms(kv[:, :R], eps) * w[q_ + "dkv.norm"]
            kr = _turn_pairs(kv[:, None, R:], pos, speeds, gain).expand(n, H, -1)
            k = torch.cat([(c @ w[q_ + "uk"].T).reshape(n, H, d), kr], 2)
            q = torch.cat([q[..., :d], _turn_pairs(q[..., d:], pos, speeds, gain)], 2)
            y = _attend(q, k, (c @ w[q_ + "uv"].T).reshape(n, H, -1), m["scale"], m["mask"]["size"] if latent else None).reshape(n, -1)
            if latent:
                y = y * torch.sigmoid(h @ w[q_ + "g"].T)
        y = y @ w[q_ + "o"].T
        x = x + norm(y * torch.sigmoid(h @ w[p + "rg1"].T + w[p + "rg1.b"]), p + "norm1b")
        h, p2 = norm(x, p + "norm2"), p + "mlp."
        if f["kind"] == "dense":
            y = gated(p2, h, gelu)
        else:
            r = f["router"]
            s = torch.sigmoid(h @ w[p2 + "router"].T)
            parts = s.reshape(n, r["groups"]["count"], -1)
            kept = torch.topk(torch.topk(parts, 2, -1).values.sum(-1), r["groups"]["keep"], -1).indices
            open_ = torch.zeros(parts.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, kept, True)
            top = torch.topk(s.masked_fill(~open_[..., None].expand_as(parts).reshape(n, -1), -1.0), r["top"], -1)
            weight = top.values / top.values.sum(-1, keepdim=True) * r["scale"]
            y = torch.sigmoid(h @ w[p2 + "shared.sg"].T) * gated(p2 + "shared.", h, silu)
            for e in range(r["experts"]):
                row, col = torch.nonzero(top.indices == e, as_tuple=True)
                if len(row):
                    y[row] += weight[row, col][:, None] * gated("%se%d." % (p2, e), h[row], silu)
        x = x + norm(y * torch.sigmoid(h @ w[p + "rg2"].T + w[p + "rg2.b"]), p + "norm2b")
    cap = cfg["logit_softcap"]
    return cap * torch.tanh(norm(x, "final.norm") @ w["head"].T / cap)


def exact(case, seed):
    gen, kind = _gen(seed), case["kind"]
    if kind == "linear":
        t = TYPES[case["type"]]
        ws = [_values(_blocks(gen, t, case["n"], case["k"], case["k"] ** -0.5), t).reshape(case["n"], case["k"]) for _ in range(case["depth"])]
        y = torch.randn(case["rows"], case["k"], device="cuda", generator=gen).double() @ ws[0].T
        for w in ws[1:]:
            y = _rms(y, 1e-5) @ w.T
        return y
    if kind == "layered":
        toks = _tokens(seed, case["prompt"] + case["steps"], case["vocab"])
        w = {name: x.double() for name, x in _layered_parts(case, gen)}
        y = (_mukutar if case["model"] == "mukutar" else _rukedra)(_layered_cfg(case), w, toks)
        return dict(first=y[case["prompt"] - 1:case["prompt"]].cpu().numpy(), last=y[-1].cpu().numpy())
    cfg, m = _llama_cfg(case), _Llama(case, gen)
    L, G, D = case["layers"], cfg["n_kv_heads"], cfg["head_dim"]
    if kind == "prompt":
        y = m.forward(_tokens(seed, case["tokens"], case["vocab"]), 0, [None] * L)
        return dict(logits=y[_want(case)].cpu().numpy())
    past = lambda: [_context(case, gen, cfg).double().reshape(2, -1, G, D) for _ in range(L)]
    if kind == "ops":
        return dict(logits=m.forward(_tokens(seed, case["steps"], case["vocab"]), case["context"], past())[-1:])
    if kind == "batch":
        B = case["batch"]
        toks = _tokens(seed, B * case["steps"], case["vocab"])
        return dict(logits=np.stack([m.forward(toks[b::B], case["context"], past())[-1].cpu().numpy() for b in range(B)]))
    kv, tok, gap = past(), _tokens(seed, 1, case["vocab"])[0], math.inf
    for i in range(case["steps"]):
        y = m.forward([tok], case["context"] + i, kv)[0]
        top = torch.topk(y, 2)
        tok = int(top.indices[0])
        gap = min(gap, float(top.values[0] - top.values[1])) if i + 1 < case["steps"] else gap
    # two tokens nearly equal: another correct run may go on with the other one
    near = gap < 5e-4 * float(torch.sqrt(torch.mean(y * y)))
    return dict(tokens=None, logits=None if near else y.cpu().numpy())
