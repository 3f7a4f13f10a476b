"""The work that users of this framework have it do, as cases that can be timed and compared.

Kinds of case, all through the public entry points:

* ``product``: quantized products over device tensors, as an embedder with its own runtime calls them (`swlm_op_qgemm_dev`); a pass
  multiplies by several weight matrices one after the other, as the layers of a model do, so that weights come from memory.
* ``attention``: flash-decode over a caller's cache (`swlm_op_flash_decode_dev`).
* ``decode``: a model's decode loop with the tokens chosen by the host (`InferenceModel.decode`), then its logits.
* ``prompt``: one prompt into an empty sequence (`InferenceModel.prefill`), then its logits.
* ``batch``: one step of continuous batching over an fp32-stream model (`InferenceModel.run_batch`): decoding sequences beside a
  portion of a prompt, logits for a sampler.

Model widths are those of the framework's own configurations; the Llama shape has fewer layers here (they are alike) so that inputs
can be made anew often. Weights are drawn around zero with about unit gain, keys sharp enough that attention is not a plain mean.
"""
import math
import zlib

import numpy as np
import torch

import __graft_entry__

GROUP = 64
KV_Q8_GROUP32 = 0x10


def listed():
    return [
        # one token through projections the size of a 7B model's: the smallest call, one launch each
        {"name": "product_1x4096x4096", "kind": "product", "rows": 1, "k": 4096, "n": 4096, "weights": 32},
        # a decode batch through the widest projection of the 8B shape
        {"name": "product_16x4096x14336", "kind": "product", "rows": 16, "k": 4096, "n": 14336, "weights": 8},
        # a prompt's products
        {"name": "product_512x4096x14336", "kind": "product", "rows": 512, "k": 4096, "n": 14336, "weights": 4},
        # a serving batch with long contexts
        {"name": "attention_8x8192", "kind": "attention", "batch": 8, "context": 8192, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # one user, the 8B shape: the headline loop
        {"name": "llama_decode_1", "kind": "decode", "model": "llama", "layers": 8, "batch": 1, "context": 4096, "ragged": False, "kv": 0, "steps": 16},
        # sequences sharing one pass over the weights
        {"name": "llama_decode_16", "kind": "decode", "model": "llama", "layers": 4, "batch": 16, "context": 4096, "ragged": False, "kv": 0, "steps": 8},
        # a larger batch, no power of two, every sequence at its own place
        {"name": "llama_decode_41", "kind": "decode", "model": "llama", "layers": 4, "batch": 41, "context": 4091, "ragged": True, "kv": 0, "steps": 4},
        # the memory-saving cache: 8-bit groups of 32
        {"name": "llama_decode_1_q8", "kind": "decode", "model": "llama", "layers": 4, "batch": 1, "context": 8192, "ragged": False, "kv": KV_Q8_GROUP32, "steps": 16},
        # time to the first token
        {"name": "llama_prompt_4096", "kind": "prompt", "model": "llama", "layers": 4, "tokens": 4096},
        # a small hybrid model, where launches and latency are most of a step
        {"name": "lfm2_decode_1", "kind": "decode", "model": "lfm2", "layers": 16, "batch": 1, "context": 2048, "ragged": False, "kv": 0, "steps": 16},
        # and its prompt, an odd length
        {"name": "lfm2_prompt_2011", "kind": "prompt", "model": "lfm2", "layers": 16, "tokens": 2011},
        # a step of the batch scheduler over the latent-attention design: fifteen users decode while a prompt comes in
        {"name": "vuzunex_batch_15+497", "kind": "batch", "layers": 4, "decoding": 15, "context": 4096, "portion": 497},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["product", "product", "attention", "decode", "decode", "decode", "prompt", "batch"])
    if kind == "product":
        k, n = rng.choice([(4096, 4096), (4096, 6144), (4096, 14336), (14336, 4096), (2048, 2048), (2048, 8192), (8192, 2048), (2048, 3072)])
        rows = _log(rng, 1, 1024)
        return {"kind": kind, "rows": rows, "k": k, "n": n, "weights": max(2, min(32, 300_000_000 // (k * n) + 1))}
    if kind == "attention":
        batch = _log(rng, 1, 64)
        return {"kind": kind, "batch": batch, "context": min(32768, max(64, _log(rng, 256, 131072) // batch + rng.randrange(64))), "heads": 32,
                "kv_heads": 8, "head_dim": rng.choice([64, 128])}
    if kind == "decode":
        model = rng.choice(["llama", "llama", "lfm2"])
        batch = rng.choice([1, 1, _log(rng, 2, 16), rng.randint(17, 48)])
        kv = KV_Q8_GROUP32 if model == "llama" and batch <= 4 and rng.random() < 0.3 else 0
        return {"kind": kind, "model": model, "layers": 4 if model == "llama" else 16, "batch": batch, "context": _log(rng, 64, 8192 if batch == 1 else 4096),
                "ragged": batch > 1 and rng.random() < 0.7, "kv": kv, "steps": 16 if batch == 1 else 8 if batch <= 16 else 4}
    if kind == "prompt":
        model = rng.choice(["llama", "lfm2"])
        return {"kind": kind, "model": model, "layers": 4 if model == "llama" else 16, "tokens": _log(rng, 40, 4096)}
    decoding, portion = rng.choice([(_log(rng, 1, 16), 0), (0, _log(rng, 16, 1024)), (_log(rng, 1, 16), _log(rng, 16, 1024))])
    return {"kind": kind, "layers": 4, "decoding": decoding, "context": _log(rng, 64, 4096), "portion": portion}


# ---- what the values are ---------------------------------------------------------------------------------------------

def _generator(seed, name):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)


def _q4(seed, name, n, k, gain=1.0):
    """(words int32 [n, k/8], scales, biases bf16 [n, k/64]): uniform nibbles, weights around zero, outputs of about `gain`."""
    g = _generator(seed, name)
    words = torch.randint(-2 ** 31, 2 ** 31, (n, k // 8), generator=g, device="cuda", dtype=torch.int32)
    unit = gain / (4.61 * math.sqrt(k))
    scales = (unit * (0.7 + 0.6 * torch.rand((n, k // GROUP), generator=g, device="cuda"))).bfloat16()
    biases = (-7.5 * scales.float() + 0.1 * unit * torch.randn((n, k // GROUP), generator=g, device="cuda")).bfloat16()
    return words, scales, biases


def _normal(seed, name, shape, std=1.0, mean=0.0):
    return (mean + std * torch.randn(shape, generator=_generator(seed, name), device="cuda")).bfloat16()


def _tensor(seed, name, kind, shape):
    """One tensor of a model's inventory. Results that join the residual stream are a fraction of it, as in a trained model."""
    if kind == "q4":
        joins = name.endswith(("o_proj", "out_proj", "down_proj", "feed_forward.w2"))
        return _q4(seed, name, shape[0], shape[1], 0.25 * math.sqrt(shape[1]) if "embed" in name else 0.12 if joins else 1.0)
    if kind == "norm":
        return _normal(seed, name, shape, 0.05, 1.0)
    if kind == "norm0":
        return _normal(seed, name, shape, 0.05)
    if kind == "matrix":
        return _normal(seed, name, shape, 1.0 / math.sqrt(shape[1]))
    return _normal(seed, name, shape, 0.3 if kind == "conv" else 1.0)


def _host(t):
    t = t.cpu()
    return t.view(torch.int16).numpy().view(np.uint16) if t.dtype == torch.bfloat16 else t.numpy()


def _tokens(seed, name, shape, vocab):
    return torch.randint(0, vocab, shape, generator=_generator(seed, name), device="cuda").cpu().numpy().astype(np.int32)


def _contexts(case):
    """Rows in the cache of each sequence: all alike, or from the whole context down to a quarter of it."""
    batch, context = case.get("batch", case.get("decoding")), case["context"]
    if not case.get("ragged", True) or batch == 1:
        return [context] * batch
    return [max(1, round(context * (1.0 - 0.75 * b / (batch - 1)))) for b in range(batch)]


def _cached(seed, which, layer, b, shape):
    """Rows of one sequence [kv heads, rows, head_dim]; keys (0) are drawn wider than values (1)."""
    return _normal(seed, f"cache{which}.{layer}.{b}", shape, 2.0 if which == 0 else 1.0)


# ---- the models ------------------------------------------------------------------------------------------------------

def _builder(pkg, case):
    max_seq = (case["context"] + case["steps"] if case["kind"] == "decode" else case.get("tokens", 0)) + 8
    batch = case.get("batch", 1)
    if case["kind"] == "batch":
        P = pkg.vuzunex
        mixer = P.LatentAttention(16, 128, 64, 128, 512, 192 ** -0.5, 10000.0, 64, P.RotaryScaling(40.0, 4096.0, 32.0, 1.0))
        layers = [P.Layer(mixer, 8192, i) for i in range(case["layers"])]
        return pkg.VuzunexPlanBuilder(pkg.VuzunexConfig(vocab=32768, width=2048, layers=layers, max_seq=max(case["context"], case["portion"]) + 64,
                                                        max_batch=case["decoding"] + (case["portion"] > 0)))
    if case["model"] == "lfm2":
        config = pkg.lfm2_like_config(max_seq=max_seq, max_batch=batch)
    else:
        config = pkg.llama3_8b_config(max_seq=max_seq, max_batch=batch)
        config.layers, config.quantized_embedding, config.kv_scheme = case["layers"], True, case.get("kv", 0)
    return pkg.DispatchPlanBuilder(config)


class _Weights:
    """name -> the host arrays that the loader takes, one tensor at a time."""

    def __init__(self, builder, seed):
        self.seed, self.inventory = seed, {name: (kind, shape) for name, kind, shape, _ in builder.tensors()}

    def __getitem__(self, name):
        kind, shape = self.inventory[name]
        t = _tensor(self.seed, name, kind, shape)
        return tuple(_host(p).view(np.uint32) if p.dtype == torch.int32 else _host(p) for p in t) if kind == "q4" else _host(t)


class _Exact:
    """The same tensors in 64 bits."""

    def __init__(self, builder, seed):
        self.seed, self.inventory = seed, {name: (kind, shape) for name, kind, shape, _ in builder.tensors()}

    def rows(self, name, at=None):
        kind, shape = self.inventory[name]
        t = _tensor(self.seed, name, kind, shape)
        if kind != "q4":
            return (t if at is None else t[at]).double()
        return _dequantized(*(p if at is None else p[at] for p in t))

    def times(self, x, name):
        kind, shape = self.inventory[name]
        t = _tensor(self.seed, name, kind, shape)
        return _product(x, *t) if kind == "q4" else x @ t.double().T


def _dequantized(words, scales, biases):
    q = (words.unsqueeze(-1) >> torch.arange(0, 32, 4, device=words.device, dtype=torch.int32)) & 15
    q = q.reshape(words.shape[0], -1, GROUP).double()
    return (q * scales.double().unsqueeze(-1) + biases.double().unsqueeze(-1)).reshape(words.shape[0], -1)


def _product(x, words, scales, biases):
    return torch.cat([x @ _dequantized(words[a:a + 8192], scales[a:a + 8192], biases[a:a + 8192]).T for a in range(0, words.shape[0], 8192)], dim=1)


# ---- preparing -------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    pkg = __graft_entry__.load_package()
    store = pkg.WeightStore(0)
    state = {"case": case, "store": store, "lib": store.lib}
    if case["kind"] == "product":
        state["names"] = [f"w{i}" for i in range(case["weights"])]
        for name in state["names"]:
            words, scales, biases = _q4(seed, name, case["n"], case["k"])
            store.add_q4_mlx(name, _host(words).view(np.uint32), _host(scales), _host(biases))
        state["x"] = _normal(seed, "x", (case["weights"], case["rows"], case["k"]))
        state["y"] = torch.empty((case["weights"], case["rows"], case["n"]), dtype=torch.bfloat16, device="cuda")
        state["stream"] = torch.cuda.Stream()
    elif case["kind"] == "attention":
        b, ctx, h, kvh, d = (case[f] for f in ("batch", "context", "heads", "kv_heads", "head_dim"))
        state["q"], state["k"], state["v"] = _attention_inputs(case, seed)
        state["out"] = torch.empty((b, h, d), dtype=torch.bfloat16, device="cuda")
        state["scratch"] = torch.empty(store.lib.swlm_op_flash_decode_scratch_bytes(b, h, kvh, d, ctx), dtype=torch.uint8, device="cuda")
        state["stream"] = torch.cuda.Stream()
    else:
        builder = _builder(pkg, case)
        model = state["model"] = pkg.load_model(store, builder, _Weights(builder, seed))
        vocab = builder.config.vocab
        if case["kind"] == "decode":
            c = builder.config
            state["positions"] = _contexts(case)
            for layer in range(c.kv_layer_count):
                for b, rows in enumerate(state["positions"]):
                    for which in (0, 1):
                        cached = _host(_cached(seed, which, layer, b, (c.kv_heads, rows, c.head_dim)))
                        for head in range(c.kv_heads):
                            model.write_kv(which, layer, b, head, cached[head])
            state["tokens"] = _tokens(seed, "tokens", (case["steps"], case["batch"]), vocab)
        elif case["kind"] == "prompt":
            state["tokens"] = _tokens(seed, "tokens", (1, case["tokens"]), vocab)
        else:
            contexts, tokens, portion = _batch_tokens(case, seed, vocab)
            state["positions"] = contexts + ([0] if case["portion"] else [])
            for b, t in enumerate(tokens):
                model.run_batch([(b, t[:-1].tolist(), [])], logits=False)
            state["entries"] = [(b, t[-1:].tolist(), [0]) for b, t in enumerate(tokens)]
            if case["portion"]:
                state["entries"].append((len(tokens), portion.tolist(), [case["portion"] - 1]))
    torch.cuda.synchronize()
    return state


def _attention_inputs(case, seed):
    b, ctx, h, kvh, d = (case[f] for f in ("batch", "context", "heads", "kv_heads", "head_dim"))
    return _normal(seed, "q", (b, h, d)), _normal(seed, "k", (b, kvh, ctx, d), 2.0), _normal(seed, "v", (b, kvh, ctx, d))


def _batch_tokens(case, seed, vocab):
    """Rows in the cache of the decoding sequences, their tokens (the last one is to be decoded), the portion's tokens."""
    contexts = _contexts(case) if case["decoding"] else []
    return contexts, [_tokens(seed, f"sequence{b}", (c + 1,), vocab) for b, c in enumerate(contexts)], _tokens(seed, "portion", (case["portion"],), vocab)


# ---- one pass --------------------------------------------------------------------------------------------------------

def run(state):
    case, lib = state["case"], state["lib"]
    if case["kind"] == "product":
        x, y, stream = state["x"], state["y"], state["stream"].cuda_stream
        for i, name in enumerate(state["names"]):
            lib.check(lib.swlm_op_qgemm_dev(state["store"].handle, name.encode(), case["rows"], x[i].data_ptr(), y[i].data_ptr(), stream))
        return y
    if case["kind"] == "attention":
        b, ctx, h, kvh, d = (case[f] for f in ("batch", "context", "heads", "kv_heads", "head_dim"))
        lib.check(lib.swlm_op_flash_decode_dev(state["store"].handle, b, h, kvh, d, ctx, ctx, 1.0 / math.sqrt(d), state["q"].data_ptr(),
                                               state["k"].data_ptr(), state["v"].data_ptr(), state["out"].data_ptr(),
                                               state["scratch"].data_ptr(), state["stream"].cuda_stream))
        return state["out"]
    model = state["model"]
    if case["kind"] == "batch":
        model.set_positions(state["positions"])
        return model.run_batch(state["entries"])[0]
    if case["kind"] == "decode":
        model.set_positions(state["positions"])
        for t in state["tokens"]:
            model.decode(t)
    else:
        model.reset_sequence(0)
        model.prefill(state["tokens"])
    return torch.from_numpy(model.logits().view(np.int16)).view(torch.bfloat16)


# ---- what it takes, and how exact it is --------------------------------------------------------------------------------

def work(case):
    if case["kind"] == "product":
        k, n, m, w = case["k"], case["n"], case["rows"], case["weights"]
        return {"bytes": w * (0.5625 * k * n + 2 * m * (k + n)), "flops": 2.0 * w * m * k * n}
    if case["kind"] == "attention":
        b, ctx, h, kvh, d = (case[f] for f in ("batch", "context", "heads", "kv_heads", "head_dim"))
        return {"bytes": 4.0 * b * ctx * kvh * d + 4 * b * h * d, "flops": 4.0 * b * ctx * h * d}
    builder = _builder(__graft_entry__.load_package(), case)
    c = builder.config
    if case["kind"] == "batch":
        m, rows, matrices = c.layers[0].mixer, case["decoding"] + case["portion"], c.weight_elems()
        wanted = case["decoding"] + (case["portion"] > 0)
        context = sum(_contexts(case)) if case["decoding"] else 0
        attended = context + case["portion"] * (case["portion"] + 1) / 2
        return {"bytes": 2.0 * matrices + 2.0 * case["layers"] * (m.kv_rank + m.rot_dim) * (context + case["portion"]) + 4 * wanted * c.vocab,
                "flops": 2.0 * rows * (matrices - c.vocab * c.width) + 2.0 * wanted * c.vocab * c.width
                + 2.0 * case["layers"] * m.heads * attended * (m.dim + m.rot_dim + m.vdim)}
    head = c.hidden * c.vocab
    weights, row = c.q4_weight_elems() - head, 4.0 * c.kv_heads * c.head_dim
    if case["kind"] == "prompt":
        n = case["tokens"]
        return {"bytes": 0.5625 * (weights + head) + row * c.kv_layer_count * n + 2 * c.vocab,
                "flops": 2.0 * n * weights + 2.0 * head + 4.0 * c.kv_layer_count * c.heads * c.head_dim * n * (n + 1) / 2}
    cached, b, t = sum(_contexts(case)), case["batch"], case["steps"]
    if case["kv"]:
        row = row / 2 * 36 / 32
    return {"bytes": t * (0.5625 * (weights + head) + row * c.kv_layer_count * cached + 2 * b * c.vocab),
            "flops": t * (2.0 * b * (weights + head) + 4.0 * c.kv_layer_count * c.heads * c.head_dim * cached)}


def tolerance(case):
    if case["kind"] in ("product", "attention"):
        return {"rel": 8e-3, "max": 3e-2}     # results are rounded to bf16, sums are 32 bits wide
    return {"rel": 3e-2, "max": 0.3}          # activations between the layers are bf16


def exact(case, seed):
    if case["kind"] == "product":
        x = _normal(seed, "x", (case["weights"], case["rows"], case["k"])).double()
        return torch.stack([_product(x[i], *_q4(seed, f"w{i}", case["n"], case["k"])) for i in range(case["weights"])])
    if case["kind"] == "attention":
        q, k, v = _attention_inputs(case, seed)
        return torch.stack([_attend(q[b].double(), k[b].double(), v[b].double()) for b in range(case["batch"])])
    builder = _builder(__graft_entry__.load_package(), case)
    if case["kind"] == "batch":
        _, tokens, portion = _batch_tokens(case, seed, builder.config.vocab)
        sequences = tokens + ([portion] if case["portion"] else [])
        return torch.cat([_vuzunex_logits(builder, seed, t) for t in sequences])
    return _llama_logits(builder, case, seed)


def _attend(q, k, v):
    """q [heads, d] over k, v [kv heads, rows, d]."""
    qg = q.reshape(k.shape[0], -1, q.shape[-1])
    return (torch.softmax(qg @ k.transpose(1, 2) / math.sqrt(q.shape[-1]), dim=-1) @ v).reshape(q.shape)


def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps) * weight


def _rotate(x, positions, base):
    """Rotate-half over the last axis of x [tokens, heads, d]."""
    half = x.shape[-1] // 2
    angle = positions.double()[:, None, None] * base ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = angle.cos(), angle.sin()
    return torch.cat([x[..., :half] * c - x[..., half:] * s, x[..., half:] * c + x[..., :half] * s], dim=-1)


def _causal(q, k, v, scale):
    """q [tokens, heads, d] over k, v [tokens, kv heads, ...] of the same sequence."""
    n, group, out = q.shape[0], q.shape[1] // k.shape[1], []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T) * scale
        s.masked_fill_(torch.ones((n, n), dtype=torch.bool, device=q.device).triu(1), -math.inf)
        out.append(torch.softmax(s, dim=-1) @ v[:, h // group])
    return torch.stack(out, dim=1)


def _llama_logits(builder, case, seed):
    """Logits behind the last token of a prompt, or of decode steps over the prepared cache; Llama and LFM2 layers."""
    c, w = builder.config, _Exact(builder, seed)
    h, kvh, d, lfm2 = c.heads, c.kv_heads, c.head_dim, c.family == "lfm2"
    if case["kind"] == "prompt":
        tokens, batch, steps, contexts = _tokens(seed, "tokens", (1, case["tokens"]), c.vocab).T, 1, case["tokens"], [0]
    else:
        tokens, batch, steps, contexts = _tokens(seed, "tokens", (case["steps"], case["batch"]), c.vocab), case["batch"], case["steps"], _contexts(case)
    x = w.rows("model.embed_tokens.weight", torch.from_numpy(tokens.astype(np.int64)).cuda().reshape(-1)).reshape(steps, batch, -1)
    position = torch.arange(steps, device="cuda")
    kv = 0
    for i in range(c.layers):
        p = f"model.layers.{i}."
        n = _rms(x, w.rows(p + ("operator_norm.weight" if lfm2 else "input_layernorm.weight")), c.norm_eps).reshape(steps * batch, -1)
        if c.is_attention_layer(i):
            q, k, v = (w.times(n, p + f"self_attn.{s}_proj").reshape(steps, batch, -1, d) for s in "qkv")
            if lfm2:
                q, k = _rms(q, w.rows(p + "self_attn.q_layernorm.weight"), c.norm_eps), _rms(k, w.rows(p + "self_attn.k_layernorm.weight"), c.norm_eps)
            out = []
            for b in range(batch):
                at = position + contexts[b]
                qb, kb = _rotate(q[:, b], at, c.rope_theta), _rotate(k[:, b], at, c.rope_theta)
                if case["kind"] == "prompt":
                    out.append(_causal(qb, kb, v[:, b], d ** -0.5))
                    continue
                keys, values = (torch.cat([_cached(seed, s, kv, b, (kvh, contexts[b], d)).double(), new.transpose(0, 1)], dim=1)
                                for s, new in ((0, kb), (1, v[:, b])))
                out.append(torch.stack([_attend(qb[t], keys[:, :contexts[b] + t + 1], values[:, :contexts[b] + t + 1]) for t in range(steps)]))
            x = x + w.times(torch.stack(out, dim=1).reshape(steps * batch, h * d), p + ("self_attn.out_proj" if lfm2 else "self_attn.o_proj")).reshape(x.shape)
            kv += 1
        else:
            gate_in, gate_out, u = w.times(n, p + "conv.in_proj").reshape(steps, batch, -1).chunk(3, dim=-1)
            taps = w.rows(p + "conv.conv.weight")
            u = torch.cat([torch.zeros((c.conv_kernel - 1, *u.shape[1:]), dtype=u.dtype, device="cuda"), gate_in * u])
            y = gate_out * sum(u[j:j + steps] * taps[:, j] for j in range(c.conv_kernel))
            x = x + w.times(y.reshape(steps * batch, -1), p + "conv.out_proj").reshape(x.shape)
        n = _rms(x, w.rows(p + ("ffn_norm.weight" if lfm2 else "post_attention_layernorm.weight")), c.norm_eps).reshape(steps * batch, -1)
        gate, up, down = (p + s for s in (("feed_forward.w1", "feed_forward.w3", "feed_forward.w2") if lfm2 else ("mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")))
        x = x + w.times(torch.nn.functional.silu(w.times(n, gate)) * w.times(n, up), down).reshape(x.shape)
    n = _rms(x[-1], w.rows("model.embedding_norm.weight" if lfm2 else "model.norm.weight"), c.norm_eps)
    return w.times(n, "model.embed_tokens.weight" if c.tie_embeddings else "lm_head")


def _vuzunex_logits(builder, seed, tokens):
    """Logits [1, vocab] behind the last token of one sequence."""
    c, w = builder.config, _Exact(builder, seed)
    x = w.rows("embed", torch.from_numpy(tokens.astype(np.int64)).cuda()) * c.embedding_scale
    n, at = x.shape[0], torch.arange(x.shape[0], device="cuda").double()
    for i, layer in enumerate(c.layers):
        p, m, eps = f"l{i}.", layer.mixer, c.norm_eps
        s, pair = m.rot_scaling, torch.arange(m.rot_dims // 2, device="cuda", dtype=torch.float64)
        f = m.rot_base ** (-2.0 * pair / m.rot_dims)
        low, high = (m.rot_dims * math.log(s.original / (2 * math.pi * turns)) / (2 * math.log(m.rot_base)) for turns in (s.fast, s.slow))
        low, high = max(math.floor(low), 0), min(math.ceil(high), m.rot_dims - 1)
        ramp = ((pair - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        angle = at[:, None, None] * (f / s.factor * ramp + f * (1.0 - ramp))
        cos, sin = (t * (0.1 * math.log(s.factor) + 1.0) for t in (angle.cos(), angle.sin()))

        def turn(z):
            u, v = z[..., :m.rot_dims // 2], z[..., m.rot_dims // 2:m.rot_dims]
            return torch.cat([u * cos - v * sin, v * cos + u * sin, z[..., m.rot_dims:]], dim=-1)

        a = _rms(x, 1.0 + w.rows(p + "norm1"), eps)
        q = w.times(a, p + "mix.q").reshape(n, m.heads, m.dim + m.rot_dim)
        down = w.times(a, p + "mix.dkv")
        latent, shared = _rms(down[:, :m.kv_rank], w.rows(p + "mix.dkv.norm"), eps), turn(down[:, None, m.kv_rank:])
        q = torch.cat([q[..., :m.dim], turn(q[..., m.dim:])], dim=-1)
        k = torch.cat([w.times(latent, p + "mix.uk").reshape(n, m.heads, m.dim), shared.expand(n, m.heads, m.rot_dim)], dim=-1)
        o = _causal(q, k, w.times(latent, p + "mix.uv").reshape(n, m.heads, m.vdim), m.scale) * torch.sigmoid(w.times(a, p + "mix.g"))[:, :, None]
        x = x + _rms(w.times(o.reshape(n, -1), p + "mix.o"), 1.0 + w.rows(p + "norm1b"), eps)
        a = _rms(x, 1.0 + w.rows(p + "norm2"), eps)
        a = torch.nn.functional.gelu(w.times(a, p + "mlp.gate"), approximate="tanh") * w.times(a, p + "mlp.up")
        x = x + _rms(w.times(a, p + "mlp.down"), 1.0 + w.rows(p + "norm2b"), eps)
    return w.times(_rms(x[-1:], 1.0 + w.rows("final.norm"), c.norm_eps), "head")
