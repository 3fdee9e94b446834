"""The workloads this framework is timed on: what its users run, through the public entry points, over the sizes they run it at.

Five kinds of case, named by ``kind``:

* ``decode``: one request on a quantised GGUF model (Q4_K with Q6_K for the output head, ``attn_v`` and ``ffn_down``) through ``GGUFModel``, its
  prompt in the cache; a pass takes ``steps`` tokens, each handed over by the caller (``stream``: a server that streams) or all in one scripted run;
* ``prompt``: the prompt pass of such a model up to the first token's logits, or (``score``) the logits of every position;
* ``serve``: requests of different lengths in the batching engine over its paged cache, from their prompts through ``steps`` tokens each;
* ``train``: one training step (forward, backward, AdamW on fp32 masters that also writes the bf16 weights) of the Llama-style or the character model;
* ``attention``: ``flash_attention`` forward and backward on its own, as a module of a user's own model calls it.

The model shapes are those of the benchmarks (``bench.py``, ``benchmarks/``) with fewer layers, since a layer costs the same at every depth.
Weights and inputs are random (projections into the residual stream scaled down by the number of layers, as is usual at initialisation); ids that a sampler would have chosen are given, so that a pass is the same every time."""
import math
import os
import tempfile

import torch
import torch.nn.functional as F

Q4_K, Q6_K, F32 = 12, 14, 0                     # type numbers of the GGUF format
ROPE_GGUF, ROPE_LLAMA = 1e6, 1e4
EPS_GGUF, EPS_LLAMA = 1e-6, 1e-5
LR, BETAS, DECAY = 3e-4, (0.9, 0.95), 0.1       # AdamW of the training benchmarks


def _decode(name, layers, hidden, heads, kv_heads, ffn, vocab, prompt, steps, stream):
    return dict(name=name, kind="decode", layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, head_dim=128, ffn=ffn, vocab=vocab,
                prompt=prompt, steps=steps, stream=stream)


def _prompt(name, layers, hidden, heads, kv_heads, ffn, vocab, prompt, score):
    return dict(name=name, kind="prompt", layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, head_dim=128, ffn=ffn, vocab=vocab,
                prompt=prompt, score=score)


def _serve(name, layers, hidden, heads, kv_heads, ffn, vocab, requests, shortest, longest, steps):
    return dict(name=name, kind="serve", layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, ffn=ffn, vocab=vocab, requests=requests,
                shortest=shortest, longest=longest, steps=steps)


def _train(name, model, layers, hidden, heads, kv_heads, ffn, vocab, batch, seq):
    return dict(name=name, kind="train", model=model, layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, ffn=ffn, vocab=vocab, batch=batch, seq=seq)


def _attention(name, batch, queries, keys, heads, kv_heads, head_dim, causal):
    return dict(name=name, kind="attention", batch=batch, queries=queries, keys=keys, heads=heads, kv_heads=kv_heads, head_dim=head_dim, causal=causal)


def listed():
    return [
        # a small chat model answering one user, token by token: launches and hand-overs count, not bytes
        _decode("decode-small", 4, 1024, 16, 8, 2048, 4096, 16, 16, True),
        # the headline: a 4B-class model at batch 1 (its width and vocabulary, a third of its layers), generation without a caller in between
        _decode("decode-4b", 12, 2560, 32, 8, 9728, 151936, 128, 32, False),
        # a short question to the same model: time to the first token
        _prompt("prompt-128", 12, 2560, 32, 8, 9728, 151936, 128, False),
        # a long context (a document, a conversation) to the same model, of no round length
        _prompt("prompt-1999", 12, 2560, 32, 8, 9728, 151936, 1999, False),
        # ranking or verifying a short text: the logits of every position
        _prompt("score-57", 12, 2560, 32, 8, 9728, 151936, 57, True),
        # the engine with one request
        _serve("serve-1", 16, 2048, 16, 4, 5632, 32000, 1, 512, 512, 32),
        # the engine with a full batch of requests of different lengths
        _serve("serve-32", 16, 2048, 16, 4, 5632, 32000, 32, 61, 509, 32),
        # a 7B-class model (a quarter of its layers) with long prompts, one key head per query head
        _serve("serve-7b", 8, 4096, 32, 32, 11008, 32000, 8, 1500, 2048, 16),
        # a training step of the 1.1B model (4 of its 22 layers), half the benchmark's sequences per GPU
        _train("train-1b", "llama", 4, 2048, 32, 4, 5632, 32000, 4, 2048),
        # a training step of the 7B model (2 of its 32 layers), one sequence of 4096
        _train("train-7b", "llama", 2, 4096, 32, 32, 11008, 32000, 1, 4096),
        # the character model: a small network, many launches
        _train("train-char", "chargpt", 4, 384, 6, 6, 1536, 65, 64, 256),
        # attention by itself, an odd length, grouped heads
        _attention("attention-odd", 2, 4001, 4001, 32, 8, 128, True),
    ]


def draw(rng):
    def log(lo, hi, step=1):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))

    kind = rng.choice(["decode", "prompt", "prompt", "serve", "serve", "train", "train", "attention"])
    if kind in ("decode", "prompt"):
        hidden = log(512, 2560, 256)
        heads, kv_heads = rng.choice([(8, 2), (16, 8), (20, 5), (32, 8), (24, 24)])
        shape = (rng.randint(1, 8), hidden, heads, kv_heads, log(1024, 9728, 256), log(999, 100000))
        if kind == "decode":
            return {k: v for k, v in _decode("", *shape, log(9, 1500), rng.randint(1, 32), rng.random() < 0.5).items() if k != "name"}
        score = rng.random() < 0.3
        return {k: v for k, v in _prompt("", *shape, log(9, 200 if score else 1999), score).items() if k != "name"}
    if kind == "serve":
        heads, kv_heads, head_dim = rng.choice([(8, 1, 64), (16, 4, 64), (32, 4, 64), (16, 16, 64), (8, 4, 128), (16, 4, 128), (16, 16, 128), (24, 3, 128)])
        longest = log(16, 2000)
        requests = log(1, max(1, min(48, 14000 // longest)))
        return {k: v for k, v in _serve("", rng.randint(1, 8), heads * head_dim, heads, kv_heads, log(512, 8192, 8), log(1000, 50000, 8), requests,
                                        max(2, int(longest * rng.uniform(0.1, 1.0))), longest, rng.randint(1, 24)).items() if k != "name"}
    if kind == "train":
        if rng.random() < 0.3:
            heads = rng.randint(2, 8)
            return {k: v for k, v in _train("", "chargpt", rng.randint(1, 4), heads * 64, heads, heads, heads * 256, rng.randint(30, 200), log(2, 64), log(31, 256)).items()
                    if k != "name"}
        heads, kv_heads, head_dim = rng.choice([(4, 1, 64), (8, 2, 64), (16, 4, 64), (32, 4, 64), (8, 8, 128), (12, 4, 128), (16, 8, 128), (24, 24, 128)])
        seq = log(33, 4096)
        return {k: v for k, v in _train("", "llama", rng.randint(1, 4), heads * head_dim, heads, kv_heads, log(256, 8192, 8), log(500, 32000, 8),
                                        log(1, max(1, min(16, 6000 // seq))), seq).items() if k != "name"}
    heads, kv_heads = rng.choice([(2, 2), (8, 2), (12, 4), (16, 16), (32, 4), (32, 8)])
    queries = log(17, 4001)
    causal = rng.random() < 0.6
    keys = queries if causal else log(17, 4001)
    return {k: v for k, v in _attention("", log(1, max(1, min(32, 8000 // max(queries, keys)))), queries, keys, heads, kv_heads, rng.choice([64, 128]), causal).items()
            if k != "name"}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))


def _normal(g, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * std + mean).to(dtype)


def _into(case, cols):
    """Standard deviation of a projection into the residual stream."""
    return (cols * 2 * case["layers"]) ** -0.5


def _ids(g, n, vocab):
    return torch.randint(0, vocab, (n,), generator=g, device="cuda").tolist()


def _half_bytes(x):
    return x.to(torch.float16).view(torch.uint8).reshape(*x.shape, 2)


def _q4k(g, rows, cols, std):
    """Q4_K blocks: sub-block s of a block holds d * sc[s] * q - dmin * m[s]; here m = sc and dmin = 7.5 d, so values spread around zero."""
    n = rows * cols // 256
    q = (torch.randn(n, 8, 32, generator=g, device="cuda") * 3.2 + 7.5).round().clamp(0, 15).to(torch.uint8)
    sc = torch.randint(24, 64, (n, 8), generator=g, device="cuda", dtype=torch.uint8)
    d = (torch.rand(n, 1, generator=g, device="cuda") * 0.4 + 0.8) * (std / (3.2 * 44.0))
    packed = torch.cat([sc[:, :4] & 63 | (sc[:, 4:] >> 4) << 6] * 2 + [sc[:, 4:] & 15 | (sc[:, 4:] & 15) << 4], 1)
    quants = q[:, 0::2] | q[:, 1::2] << 4
    return torch.cat([_half_bytes(d).reshape(n, 2), _half_bytes(d * 7.5).reshape(n, 2), packed, quants.reshape(n, 128)], 1).reshape(rows, -1)


def _q6k(g, rows, cols, std):
    """Q6_K blocks: group j of 16 values holds d * sc[j] * (q - 32)."""
    n = rows * cols // 256
    q = (torch.randn(n, 2, 4, 32, generator=g, device="cuda") * 10 + 32).round().clamp(0, 63).to(torch.uint8)      # [half][quarter][value]
    low = torch.cat([q[:, :, 0] & 15 | (q[:, :, 2] & 15) << 4, q[:, :, 1] & 15 | (q[:, :, 3] & 15) << 4], 2)
    high = q[:, :, 0] >> 4 | q[:, :, 1] >> 4 << 2 | q[:, :, 2] >> 4 << 4 | q[:, :, 3] >> 4 << 6
    sc = torch.randint(60, 120, (n, 16), generator=g, device="cuda", dtype=torch.uint8)
    d = (torch.rand(n, 1, generator=g, device="cuda") * 0.4 + 0.8) * (std / (10 * 90.0))
    return torch.cat([low.reshape(n, 128), high.reshape(n, 64), sc, _half_bytes(d).reshape(n, 2)], 1).reshape(rows, -1)


def _half_of(b):
    return b.contiguous().view(torch.float16).double()


def _wide_q4k(raw, rows, cols):
    b = raw.reshape(-1, 144)
    s = b[:, 4:16].to(torch.int32)
    sc = torch.cat([s[:, :4] & 63, s[:, 8:] & 15 | s[:, :4] >> 6 << 4], 1).double()
    mn = torch.cat([s[:, 4:8] & 63, s[:, 8:] >> 4 | s[:, 4:8] >> 6 << 4], 1).double()
    q = b[:, 16:].reshape(-1, 4, 32)
    q = torch.stack([q & 15, q >> 4], 2).reshape(-1, 8, 32).double()
    w = (_half_of(b[:, 0:2]) * sc)[:, :, None] * q - (_half_of(b[:, 2:4]) * mn)[:, :, None]
    return w.reshape(rows, cols)


def _wide_q6k(raw, rows, cols):
    b = raw.reshape(-1, 210)
    low, high = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 32)
    q = torch.stack([low[:, :, 0] & 15 | (high & 3) << 4, low[:, :, 1] & 15 | (high >> 2 & 3) << 4,
                     low[:, :, 0] >> 4 | (high >> 4 & 3) << 4, low[:, :, 1] >> 4 | (high >> 6 & 3) << 4], 2)
    sc = b[:, 192:208].contiguous().view(torch.int8).double() * _half_of(b[:, 208:210])
    return ((q.reshape(-1, 16, 16).double() - 32) * sc[:, :, None]).reshape(rows, cols)


def _gguf_tensors(case, seed):
    """(name, shape, type, data) of a model's tensors in file order; the ids come from the same generator afterwards."""
    g = _gen(seed)
    H, Q, K, I, V = case["hidden"], case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"], case["ffn"], case["vocab"]
    out = []

    def mat(name, rows, cols, kind, std=None):
        std = cols ** -0.5 if std is None else std
        out.append((name, (rows, cols), kind, (_q4k if kind == Q4_K else _q6k)(g, rows, cols, std)))

    def vec(name, n):
        out.append((name, (n,), F32, _normal(g, n, std=0.05, mean=1.0, dtype=torch.float32)))

    mat("token_embd.weight", V, H, Q4_K, 1.0)
    for i in range(case["layers"]):
        p = "blk.%d." % i
        vec(p + "attn_norm.weight", H)
        mat(p + "attn_q.weight", Q, H, Q4_K)
        mat(p + "attn_k.weight", K, H, Q4_K)
        mat(p + "attn_v.weight", K, H, Q6_K)
        vec(p + "attn_q_norm.weight", case["head_dim"])
        vec(p + "attn_k_norm.weight", case["head_dim"])
        mat(p + "attn_output.weight", H, Q, Q4_K, _into(case, Q))
        vec(p + "ffn_norm.weight", H)
        mat(p + "ffn_gate.weight", I, H, Q4_K)
        mat(p + "ffn_up.weight", I, H, Q4_K)
        mat(p + "ffn_down.weight", H, I, Q6_K, _into(case, I))
    vec("output_norm.weight", H)
    mat("output.weight", V, H, Q6_K)
    return out, _ids(g, case["prompt"] + case.get("steps", 0), V)


def _gguf_model(case, seed):
    from prometorch_b200.io.gguf import GGUFWriter
    from prometorch_b200.io.gguf_model import GGUFModel
    tensors, ids = _gguf_tensors(case, seed)
    most = case["prompt"] + case.get("steps", 0) + 1
    with tempfile.TemporaryDirectory(prefix="gguf_") as folder:
        w = GGUFWriter(os.path.join(folder, "model.gguf"))
        for key, value in (("general.architecture", "qwen3"), ("general.name", "random"), ("general.alignment", 32), ("qwen3.embedding_length", case["hidden"]),
                           ("qwen3.block_count", case["layers"]), ("qwen3.attention.head_count", case["heads"]),
                           ("qwen3.attention.head_count_kv", case["kv_heads"]), ("qwen3.feed_forward_length", case["ffn"]), ("qwen3.context_length", 4096),
                           ("qwen3.rope.freq_base", ROPE_GGUF), ("qwen3.attention.layer_norm_rms_epsilon", EPS_GGUF),
                           ("qwen3.attention.key_length", case["head_dim"]), ("qwen3.attention.value_length", case["head_dim"])):
            w.add(key, value)
        for name, shape, kind, data in tensors:
            w.add_tensor(name, shape, kind, data)
        w.write()
        del tensors
        model = GGUFModel(w.path, device="cuda", max_seq=max(64, most), want_logits=True)
    return model, ids


def _lens(case):
    """Lengths of the prompts: spread evenly from the shortest to the longest, in mixed order."""
    n = case["requests"]
    return [case["longest"] - (i * 5 % n) * (case["longest"] - case["shortest"]) // max(1, n - 1) for i in range(n)]


def _serve_weights(case, seed):
    """A checkpoint's tensors under their Hugging Face names."""
    g = _gen(seed)
    D, I, V = case["hidden"], case["ffn"], case["vocab"]
    kv = D // case["heads"] * case["kv_heads"]
    sd = {"model.embed_tokens.weight": _normal(g, V, D)}
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        for name, rows, cols in (("self_attn.q_proj", D, D), ("self_attn.k_proj", kv, D), ("self_attn.v_proj", kv, D), ("self_attn.o_proj", D, D),
                                 ("mlp.gate_proj", I, D), ("mlp.up_proj", I, D), ("mlp.down_proj", D, I)):
            sd[p + name + ".weight"] = _normal(g, rows, cols, std=_into(case, cols) if name in ("self_attn.o_proj", "mlp.down_proj") else cols ** -0.5)
        sd[p + "input_layernorm.weight"] = _normal(g, D, std=0.1, mean=1.0)
        sd[p + "post_attention_layernorm.weight"] = _normal(g, D, std=0.1, mean=1.0)
    sd["model.norm.weight"] = _normal(g, D, std=0.1, mean=1.0)
    sd["lm_head.weight"] = _normal(g, V, D, std=D ** -0.5)
    lens = _lens(case)
    return sd, [_ids(g, n + case["steps"], V) for n in lens], lens


def _train_weights(case, seed):
    """Parameters by name, as a run some way into training would have them, and the tokens [batch, seq + 1]."""
    g = _gen(seed)
    D, I, V = case["hidden"], case["ffn"], case["vocab"]
    kv = D // case["heads"] * case["kv_heads"]
    w = {}

    def norm(name, bias=False):
        w[name + ".weight"] = _normal(g, D, std=0.1, mean=1.0)
        if bias:
            w[name + ".bias"] = _normal(g, D, std=0.1)

    def mat(name, rows, cols, bias=False, std=None):
        w[name + ".weight"] = _normal(g, rows, cols, std=cols ** -0.5 if std is None else std)
        if bias:
            w[name + ".bias"] = _normal(g, rows, std=0.02)

    if case["model"] == "llama":
        mat("embed", V, D, std=1.0)
        for i in range(case["layers"]):
            p = "blocks.%d." % i
            norm(p + "attn_norm")
            mat(p + "attn.qkv", D + 2 * kv, D)
            mat(p + "attn.out", D, D, std=_into(case, D))
            norm(p + "mlp_norm")
            mat(p + "mlp.gate_up", 2 * I, D)
            mat(p + "mlp.down", D, I, std=_into(case, I))
        norm("norm")
        mat("lm_head", V, D)
    else:
        mat("wte", V, D, std=0.1)
        mat("wpe", case["seq"], D, std=0.1)
        for i in range(case["layers"]):
            p = "blocks.%d." % i
            norm(p + "ln1", True)
            norm(p + "ln2", True)
            mat(p + "qkv", 3 * D, D, True)
            mat(p + "proj", D, D, True, _into(case, D))
            mat(p + "fc", I, D, True)
            mat(p + "fc2", D, I, True, _into(case, I))
        norm("ln_f", True)
    tokens = torch.randint(0, V, (case["batch"], case["seq"] + 1), generator=g, device="cuda")
    return w, tokens


def _attention_inputs(case, seed):
    g = _gen(seed)
    B, H, Hk, D = case["batch"], case["heads"], case["kv_heads"], case["head_dim"]
    return (_normal(g, B, case["queries"], H, D), _normal(g, B, case["keys"], Hk, D), _normal(g, B, case["keys"], Hk, D), _normal(g, B, case["queries"], H, D))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        model, ids = _gguf_model(case, seed)
        if kind == "decode":
            model.prefill(ids[:case["prompt"]])
        return dict(case=case, model=model, ids=ids)
    if kind == "serve":
        from prometorch_b200.serve.llm import PAGE, LLMEngine, LlamaConfig, LlamaWeights
        sd, ids, lens = _serve_weights(case, seed)
        most = max(lens) + case["steps"]
        cfg = LlamaConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["ffn"], num_hidden_layers=case["layers"],
                          num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], max_position_embeddings=most + 1,
                          rms_norm_eps=EPS_LLAMA, rope_theta=ROPE_LLAMA, eos_token_id=-1)
        engine = LLMEngine(device="cuda", max_pages=sum(-(-len(t) // PAGE) for t in ids), max_active=case["requests"])
        engine.set_weights(LlamaWeights.from_state_dict(cfg, sd))
        return dict(case=case, engine=engine, ids=ids, lens=lens)
    if kind == "train":
        from prometorch_b200.optim import AdamW
        w, tokens = _train_weights(case, seed)
        with torch.device("cuda"):
            if case["model"] == "llama":
                from prometorch_b200.models.llama import Llama, LlamaConfig
                model = Llama(LlamaConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], num_layers=case["layers"], num_heads=case["heads"],
                                          num_kv_heads=case["kv_heads"], intermediate_size=case["ffn"], max_seq=case["seq"], rope_theta=ROPE_LLAMA,
                                          rms_eps=EPS_LLAMA))
            else:
                from prometorch_b200.models.gpt import CharGPT, GPTConfig
                model = CharGPT(GPTConfig(vocab_size=case["vocab"], block_size=case["seq"], n_layer=case["layers"], n_head=case["heads"],
                                          n_embd=case["hidden"]))
        model = model.to(torch.bfloat16)
        model.load_state_dict(w, strict=False)
        params = [p for _, p in sorted(model.named_parameters())]
        masters = [torch.nn.Parameter(p.detach().float().clone(), requires_grad=False) for p in params]
        opt = AdamW(masters, lr=LR, betas=BETAS, weight_decay=DECAY, fused=True)
        for mp, p in zip(masters, params):
            p.grad = torch.zeros_like(p)
            opt.set_grad_source(mp, p.grad)
            opt.attach_lowp(mp, p.data)
        return dict(case=case, model=model, opt=opt, params=params, masters=masters, tokens=tokens)
    q, k, v, do = _attention_inputs(case, seed)
    return dict(case=case, q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), do=do)


# ------------------------------------------------------------------------------------------------ one pass
def _kept(model):
    """The step's logits in a tensor of their own: the engine's buffer is overwritten by the next step and goes with the model."""
    with torch.cuda.stream(model.stream):
        return model.logits_view().clone()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "decode":
        model, ids, n = state["model"], state["ids"], case["prompt"]
        if not case["stream"]:
            model.run_script(ids[n:], 1, pos0=n)
            return {"logits": _kept(model)}
        out = []
        for i, t in enumerate(ids[n:]):
            model.forward_decode(t, n + i)
            out.append(_kept(model))
        return out
    if kind == "prompt":
        model, ids = state["model"], state["ids"]
        if case["score"]:
            return {"logits": model.prefill(ids, return_logits=True)}
        model.prefill(ids[:-1])
        model.forward_decode(ids[-1], len(ids) - 1)
        return {"logits": _kept(model)}
    if kind == "serve":
        engine, ids, lens = state["engine"], state["ids"], state["lens"]
        seqs = [engine.open_sequence() for _ in lens]
        out = [engine.feed([(s, t[:n], [n - 1]) for s, t, n in zip(seqs, ids, lens)])]
        for i in range(case["steps"]):
            out.append(engine.feed([(s, [t[n + i]], [0]) for s, t, n in zip(seqs, ids, lens)]))
        for s in seqs:
            engine.close_sequence(s)
        return out
    if kind == "train":
        model, opt, tokens = state["model"], state["opt"], state["tokens"]
        model.zero_grad(set_to_none=False)
        loss = model(tokens[:, :-1], tokens[:, 1:])
        loss.backward()
        opt.step()
        out = {"loss": loss.detach(), "grads": [p.grad for p in state["params"]]}
        if case["model"] == "llama":
            out["weights"] = [p.detach() for p in state["masters"]]
        return out
    from prometorch_b200.ops.attention import flash_attention
    q, k, v = state["q"], state["k"], state["v"]
    o = flash_attention(q, k, v, causal=case["causal"])
    return [o.detach(), *torch.autograd.grad(o, (q, k, v), state["do"])]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_params(case):
    head_dim = case.get("head_dim") or case["hidden"] // case["heads"]
    Q, K = case["heads"] * head_dim, case["kv_heads"] * head_dim
    return case["hidden"] * (2 * Q + 2 * K), case["hidden"] * case["ffn"], Q, K


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, Tq, Tk, H, Hk, D = (case[k] for k in ("batch", "queries", "keys", "heads", "kv_heads", "head_dim"))
        pairs = Tq * (Tq + 1) / 2 if case["causal"] else Tq * Tk
        return {"bytes": 2.0 * B * D * (4 * Tq * H + 4 * Tk * Hk), "flops": 14.0 * B * H * D * pairs}
    attn, ffn, Q, K = _layer_params(case)
    L, V, D = case["layers"], case["vocab"], case["hidden"]
    if kind in ("decode", "prompt"):
        v, o = D * K, D * Q
        weights = L * ((attn - v + 2 * ffn) * 144 / 256 + (v + ffn) * 210 / 256)
        head = V * D * 210 / 256
        n = case["prompt"]
        if kind == "decode":
            S = case["steps"]
            context = S * n + S * (S + 1) / 2
            return {"bytes": S * (weights + head + 4.0 * V) + 4.0 * L * K * context, "flops": 2.0 * S * (L * (attn + 3 * ffn) + V * D) + 4.0 * L * Q * context}
        rows = n if case["score"] else 1
        return {"bytes": weights + head + n * D * 144 / 256 + 4.0 * L * K * n + 4.0 * V * rows,
                "flops": 2.0 * n * L * (attn + 3 * ffn) + 2.0 * rows * V * D + 4.0 * L * Q * n * (n + 1) / 2}
    params = L * (attn + 3 * ffn) + V * D
    if kind == "serve":
        lens, S = _lens(case), case["steps"]
        context = sum(S * n + S * (S + 1) / 2 for n in lens)
        tokens = sum(lens) + S * len(lens)
        logits = (1 + S) * len(lens)
        return {"bytes": 2.0 * params * (1 + S) + 4.0 * L * K * (context + sum(lens)) + 4.0 * V * logits + 2.0 * D * tokens,
                "flops": 2.0 * tokens * (params - V * D) + 2.0 * logits * V * D + 4.0 * L * Q * (context + sum(n * (n + 1) / 2 for n in lens))}
    n, T = case["batch"] * case["seq"], case["seq"]
    gates = 3 if case["model"] == "llama" else 2
    params = L * (attn + gates * ffn) + V * D
    held = params + (V * D if case["model"] == "llama" else 0)
    # bf16 weights read twice and written, gradients written and read, masters and both moments read and written
    return {"bytes": held * (3 * 2.0 + 2 * 2.0 + 6 * 4.0), "flops": 6.0 * n * params + 14.0 * L * Q * case["batch"] * T * (T + 1) / 2}


def tolerance(case):
    # bf16 throughout (decode: 8-bit activations).  Attention alone is 0.0025 from 64 bits; through the layers of a model outputs and
    # gradients are up to 0.011 from it, and what the order of fp32 sums decides, repeated by the roundings after it, up to 0.005.
    return {"rel": 0.01, "max": 0.2} if case["kind"] == "attention" else {"rel": 0.025, "max": 0.6}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rotate(x, theta):
    """x [T, heads, D], pairs (j, j + D/2)."""
    T, _, D = x.shape
    inv = theta ** (-torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    a = torch.arange(T, dtype=torch.float64, device=x.device)[:, None] * inv
    c, s = a.cos()[:, None], a.sin()[:, None]
    x, y = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([x * c - y * s, y * c + x * s], -1)


def _attend(q, k, v, causal):
    """q [Tq, H, D], k and v [Tk, Hk, D]."""
    H, Hk, D = q.shape[1], k.shape[1], q.shape[2]
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // Hk)].T * D ** -0.5
        if causal:
            s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h // (H // Hk)])
    return torch.stack(out, 1)


def _exact_gguf(case, seed):
    tensors, ids = _gguf_tensors(case, seed)
    raw = {name: (kind, shape, data) for name, shape, kind, data in tensors}

    def w(name):
        kind, shape, data = raw[name]
        return data.double() if kind == F32 else (_wide_q4k if kind == Q4_K else _wide_q6k)(data, *shape)

    d = case["head_dim"]
    kind, shape, data = raw["token_embd.weight"]
    x = _wide_q4k(data[torch.tensor(ids, device="cuda")], len(ids), shape[1])
    T = len(ids)
    for i in range(case["layers"]):
        p = "blk.%d." % i
        h = _rms(x, w(p + "attn_norm.weight"), EPS_GGUF)
        q, k, v = ((h @ w(p + "attn_%s.weight" % n).T).reshape(T, -1, d) for n in "qkv")
        q = _rotate(_rms(q, w(p + "attn_q_norm.weight"), EPS_GGUF), ROPE_GGUF)
        k = _rotate(_rms(k, w(p + "attn_k_norm.weight"), EPS_GGUF), ROPE_GGUF)
        x = x + _attend(q, k, v, True).reshape(T, -1) @ w(p + "attn_output.weight").T
        h = _rms(x, w(p + "ffn_norm.weight"), EPS_GGUF)
        x = x + (F.silu(h @ w(p + "ffn_gate.weight").T) * (h @ w(p + "ffn_up.weight").T)) @ w(p + "ffn_down.weight").T
    rows = T if case.get("score") else case["steps"] if case.get("stream") else 1
    logits = _rms(x[-rows:], w("output_norm.weight"), EPS_GGUF) @ w("output.weight").T
    if case["kind"] == "decode" and case["stream"]:
        return list(logits)
    return {"logits": logits if case.get("score") else logits[0]}


def _exact_serve(case, seed):
    sd, ids, lens = _serve_weights(case, seed)
    d = case["hidden"] // case["heads"]
    cuts = [len(t) for t in ids]
    x = sd["model.embed_tokens.weight"][torch.tensor([t for s in ids for t in s], device="cuda")].double()
    for i in range(case["layers"]):
        w = lambda n: sd["model.layers.%d.%s.weight" % (i, n)].double()
        h = _rms(x, w("input_layernorm"), EPS_LLAMA)
        q, k, v = ((h @ w("self_attn.%s_proj" % n).T).reshape(x.shape[0], -1, d).split(cuts) for n in "qkv")
        a = torch.cat([_attend(_rotate(qs, ROPE_LLAMA), _rotate(ks, ROPE_LLAMA), vs, True).reshape(len(qs), -1) for qs, ks, vs in zip(q, k, v)])
        x = x + a @ w("self_attn.o_proj").T
        h = _rms(x, w("post_attention_layernorm"), EPS_LLAMA)
        x = x + (F.silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    head = sd["lm_head.weight"].double()
    x = _rms(x, sd["model.norm.weight"], EPS_LLAMA).split(cuts)
    return [torch.stack([s[n - 1 + i] for s, n in zip(x, lens)]) @ head.T for i in range(case["steps"] + 1)]


def _exact_train(case, seed):
    w, tokens = _train_weights(case, seed)
    w = {k: t.double().requires_grad_() for k, t in w.items()}
    H, d, T = case["heads"], case["hidden"] // case["heads"], case["seq"]
    Q, K = H * d, case["kv_heads"] * d
    total = tokens[:, 1:].numel()
    loss = 0.0
    for row in tokens:                                    # one sequence's graph at a time
        if case["model"] == "llama":
            x = w["embed.weight"][row[:-1]]
            for i in range(case["layers"]):
                p = "blocks.%d." % i
                q, k, v = (_rms(x, w[p + "attn_norm.weight"], EPS_LLAMA) @ w[p + "attn.qkv.weight"].T).split([Q, K, K], -1)
                a = _attend(_rotate(q.reshape(T, -1, d), ROPE_LLAMA), _rotate(k.reshape(T, -1, d), ROPE_LLAMA), v.reshape(T, -1, d), True)
                x = x + a.reshape(T, -1) @ w[p + "attn.out.weight"].T
                g, u = (_rms(x, w[p + "mlp_norm.weight"], EPS_LLAMA) @ w[p + "mlp.gate_up.weight"].T).chunk(2, -1)
                x = x + (F.silu(g) * u) @ w[p + "mlp.down.weight"].T
            logits = _rms(x, w["norm.weight"], EPS_LLAMA) @ w["lm_head.weight"].T
        else:
            def layer_norm(x, n):
                return F.layer_norm(x, x.shape[-1:], w[n + ".weight"], w[n + ".bias"])

            def linear(x, n):
                return x @ w[n + ".weight"].T + w[n + ".bias"]
            x = w["wte.weight"][row[:-1]] + w["wpe.weight"][:T]
            for i in range(case["layers"]):
                p = "blocks.%d." % i
                q, k, v = linear(layer_norm(x, p + "ln1"), p + "qkv").reshape(T, 3, H, d).unbind(1)
                x = x + linear(_attend(q, k, v, True).reshape(T, -1), p + "proj")
                x = x + linear(F.gelu(linear(layer_norm(x, p + "ln2"), p + "fc"), approximate="tanh"), p + "fc2")
            logits = layer_norm(x, "ln_f") @ w["wte.weight"].T
        part = F.cross_entropy(logits, row[1:], reduction="sum") / total
        part.backward()
        loss += part.detach()
    names = sorted(w)
    out = {"loss": loss, "grads": [w[n].grad for n in names]}
    if case["model"] == "llama":                          # the first AdamW step: both moments, corrected, are the gradient's own
        out["weights"] = [w[n].detach() * (1 - LR * DECAY) - LR * w[n].grad / (w[n].grad.abs() + 1e-8) for n in names]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "attention":
        q, k, v, do = (t.double() for t in _attention_inputs(case, seed))
        out = [[], [], [], []]
        for b in range(case["batch"]):
            x = [t[b].requires_grad_() for t in (q, k, v)]
            grads = [torch.zeros_like(t) for t in x]
            group = case["heads"] // case["kv_heads"]
            o = []
            for h in range(case["heads"]):                # one head's graph at a time
                j = h // group
                oh = _attend(x[0][:, h:h + 1], x[1][:, j:j + 1], x[2][:, j:j + 1], case["causal"])
                for acc, gr in zip(grads, torch.autograd.grad(oh, x, do[b][:, h:h + 1])):
                    acc += gr
                o.append(oh.detach())
            for place, t in zip(out, [torch.cat(o, 1), *grads]):
                place.append(t)
        return [torch.stack(t) for t in out]
    if kind == "train":
        return _exact_train(case, seed)
    with torch.no_grad():
        return _exact_serve(case, seed) if kind == "serve" else _exact_gguf(case, seed)
