"""Performance cases of the framework: what its users run, through the entry points they call.

Five kinds of work:

* `step`    one decode step of one sparse-attention layer (`SocketAttention.sparse_decode`): the new token's
            key and value go into the cache, the query is hashed, every cached key scored, a list selected and
            attended to.  Sizes of the benchmark's configurations and of their shards over several GPUs.
* `lists`   the same span for callers that keep the original operators and their layouts
            (`build_sparse_list_decode`, `sparse_attention_fwd`).
* `append`  a prompt's keys and values go into the cache with their bucket codes and norms (`KVCache.append`).
* `prompt`  a portion of a prompt through a whole decoder (`Decoder.forward_portion`), fresh or behind an
            earlier portion: last logits, caches and recurrent states.
* `token`   one decoded token through a whole decoder (`Decoder.decode_given_token`), its CUDA graph replayed.

The decoders have the benchmark's shapes with random weights; the Transformer has the layers of the 8B shape,
four of them.  Weights are drawn here and loaded as a checkpoint is, so that `exact` can restate the
arithmetic in float64 without the framework's code.
"""
from __future__ import annotations

import math

import torch

# what the trace runner and the benchmark set: sums of split matrix products stay in fp32, fp32 products stay fp32
torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
torch.backends.cuda.matmul.allow_tf32 = False

DEV = "cuda:0"
TABLES, PLANES, HEAD = 32, 8, 128
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
BYTES = {"bf16": 2, "f16": 2, "f32": 4}


# ------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: the CPU-sized fp32 configuration, where launches and latency are everything
        dict(name="step 4k f32", kind="step", B=1, H=32, G=8, T=4096, topk=256, sink=16, window=64, dtype="f32"),
        # one user with a 32K context: the second benchmark configuration
        dict(name="step 32k", kind="step", B=1, H=32, G=8, T=32768, topk=1024, sink=64, window=128, dtype="bf16"),
        # four long contexts: the headline configuration
        dict(name="step 128k x4", kind="step", B=4, H=32, G=8, T=131072, topk=2048, sink=64, window=256, dtype="bf16"),
        # one GPU's share of a 70B-shape layer (one KV head, 8 query heads), batch 8, ragged length, fp16 cache
        dict(name="step 64k shard f16", kind="step", B=8, H=8, G=1, T=65003, topk=2048, sink=64, window=256, dtype="f16"),
        # a caller that swapped only the two operators, ragged length
        dict(name="lists 12k", kind="lists", B=1, H=32, G=8, T=12345, topk=1024, sink=64, window=128, dtype="bf16"),
        # writing a prompt of 8192 tokens into one layer's cache
        dict(name="append 8k", kind="append", B=1, G=8, start=0, S=8192, dtype="bf16"),
        # a chat turn: 1501 more tokens behind 2500 cached ones
        dict(name="radapel 2k turn", kind="prompt", model="radapel", size="2k", B=1, start=2500, S=1501),
        # a whole document at the larger size
        dict(name="radapel 4k prompt", kind="prompt", model="radapel", size="4k", B=1, start=0, S=8000),
        # a long document at the smaller size, many windows long
        dict(name="timalorn 2k long", kind="prompt", model="timalorn", size="2k", B=1, start=0, S=32000),
        # a single user's next token
        dict(name="radapel 4k token", kind="token", model="radapel", size="4k", B=1, T=7777),
        # a batch of users' next tokens
        dict(name="timalorn 2k token x8", kind="token", model="timalorn", size="2k", B=8, T=5001),
        # sparse decode inside the Llama-shaped decoder
        dict(name="transformer token", kind="token", model="transformer", size="8b", B=1, T=32768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "lists", "append", "prompt", "prompt", "token"])
    if kind == "step":
        H, G = rng.choice([(32, 8), (32, 8), (16, 4), (8, 2), (4, 1), (8, 1), (64, 8)])
        B = rng.choice([1, 1, 2, 3, 4, 8])
        T = _log(rng, 1000, min(131072, 4 * 8 * 131072 // (B * G)))
        sink, window = rng.choice([(64, 128), (64, 256), (16, 64), (4, 1), (0, 100)])
        return dict(kind=kind, B=B, H=H, G=G, T=T, topk=rng.choice([64, 256, 1024, 2048, T // 32 + 1]), sink=sink, window=window,
                    dtype=rng.choice(["bf16", "bf16", "bf16", "f16", "f32"]))
    if kind == "lists":
        H, G = rng.choice([(32, 8), (16, 4), (8, 1), (8, 8)])
        return dict(kind=kind, B=rng.choice([1, 1, 2]), H=H, G=G, T=_log(rng, 700, 32768), topk=rng.choice([64, 256, 1000, 2048]),
                    sink=rng.choice([0, 16, 64]), window=rng.choice([1, 64, 128]), dtype=rng.choice(["bf16", "bf16", "f16", "f32"]))
    if kind == "append":
        return dict(kind=kind, B=rng.choice([1, 1, 2, 4]), G=rng.choice([1, 2, 4, 8]), start=rng.choice([0, 0, 1000, 7777]),
                    S=_log(rng, 16, 12000), dtype=rng.choice(["bf16", "bf16", "f16", "f32"]))
    size = rng.choice(["2k", "2k", "4k"])
    if kind == "prompt":
        B = rng.choice([1, 1, 1, 2, 4, 8])
        S = _log(rng, 2, (24000 if size == "2k" else 6000) // B)
        start = rng.choice([0, 0, rng.randrange(1, 6000)])
        return dict(kind=kind, model=rng.choice(["radapel", "timalorn"]), size=size, B=B, start=start, S=max(S, 4 - start, 2))
    model = rng.choice(["radapel", "timalorn", "transformer"])
    if model == "transformer":
        return dict(kind=kind, model=model, size="8b", B=rng.choice([1, 2, 4]), T=_log(rng, 1500, 60000))
    B = rng.choice([1, 1, 2, 3, 4, 8])
    return dict(kind=kind, model=model, size=size, B=B, T=_log(rng, 50, (24000 if size == "2k" else 8000) // B))


def _random(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return g, lambda *s: torch.randn(*s, generator=g, device=DEV)


def _prototypes():
    r = torch.arange(1 << PLANES, device=DEV)
    return torch.stack([((r >> (PLANES - 1 - p)) & 1) * 2.0 - 1.0 for p in range(PLANES)])


# ------------------------------------------------------------------------------------------- decoders
SHAPES = {"2k": dict(width=2048, heads=16, kv=4, ff=5632, rank=512, ssm=64, memory=(8, 128, 256)),
          "4k": dict(width=4096, heads=32, kv=8, ff=14336, rank=512, ssm=128, memory=(8, 256, 512))}
VOCAB, CHUNK, WINDOW, TURNED = 32768, 8192, 4096, 64
TRANSFORMER = dict(block_size=131072, vocab_size=32768, n_layer=4, n_head=32, n_local_heads=8, dim=4096,
                   intermediate_size=14336, rope_base=500000, heavy_const=1024, sink_size=64, window_size=128)


def _config(case):
    if case["model"] == "transformer":
        return {"architecture": "Transformer", **TRANSFORMER}
    z = SHAPES[case["size"]]
    H, G, F = z["heads"], z["kv"], z["ff"]
    if case["model"] == "radapel":
        mlp = {"kind": "dense", "ff": F, "limit": 7.0}
        att = {"type": "attention", "mlp": mlp, "mixer": {"heads": H, "kv_heads": G, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5,
                                                          "bias_max": 1024, "mask": {"size": CHUNK}}}
        lat = {"type": "latent_attention", "mlp": mlp,
               "mixer": {"heads": H, "dim": HEAD, "rot_dim": TURNED, "vdim": HEAD, "kv_rank": z["rank"],
                         "scale": (HEAD + TURNED) ** -0.5, "rot": {"base": 500000.0, "dims": TURNED}}}
        ssm = {"type": "mamba2", "mlp": None,
               "mixer": {"heads": z["ssm"], "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
        return {"architecture": "Radapel", "vocab": VOCAB, "width": z["width"], "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                "layers": [att, att, lat, ssm], "loop": {"start": 1, "stop": 4, "times": 2}}
    mlp = {"kind": "dense", "ff": F}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": H, "kv_heads": G, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "softcap": 50.0,
                     "mask": {"size": WINDOW},
                     "rot": {"base": 500000.0, "dims": TURNED,
                             "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}}
    MH, N, P = z["memory"]
    mem = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": MH, "dim": N, "vdim": P, "gate_cap": 15.0}}
    return {"architecture": "Timalorn", "vocab": VOCAB, "width": z["width"], "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "layers": [att, mem, att, mem, dict(att, weights_of=0), dict(mem, weights_of=1), att]}


def _owner(cfg, i):
    while cfg["layers"][i].get("weights_of") is not None:
        i = cfg["layers"][i]["weights_of"]
    return i


def _runs(cfg):
    """(layer whose tensors are used, pass of the loop that begins here or None) in running order."""
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if loop is None:
        return [(_owner(cfg, i), None) for i in range(n)]
    a, b = loop["start"], loop["stop"]
    return ([(i, None) for i in range(a)] + [(i, t if i == a else None) for t in range(loop["times"]) for i in range(a, b)] +
            [(i, None) for i in range(b, n)])


def _tensor_shapes(cfg):
    if cfg["architecture"] == "Transformer":
        W, F, qkv = cfg["dim"], cfg["intermediate_size"], cfg["dim"] + 2 * cfg["n_local_heads"] * HEAD
        out = {"tok_embeddings.weight": (cfg["vocab_size"], W), "norm.weight": (W,), "output.weight": (cfg["vocab_size"], W)}
        for i in range(cfg["n_layer"]):
            p = f"layers.{i}."
            out.update({p + "attention.wqkv.weight": (qkv, W), p + "attention.wo.weight": (W, W),
                        p + "attention.planes": (TABLES, PLANES, HEAD), p + "attention.protos_T": (PLANES, 1 << PLANES),
                        p + "feed_forward.w13.weight": (2 * F, W), p + "feed_forward.w2.weight": (W, F),
                        p + "ffn_norm.weight": (W,), p + "attention_norm.weight": (W,)})
        return out
    V, W = cfg["vocab"], cfg["width"]
    out = {"embed": (V, W), "final.norm": (W,), "head": (V, W)}
    if cfg.get("loop"):
        out["loop.in"], out["loop.step"] = (W, 2 * W), (cfg["loop"]["times"], W)
    for i, e in enumerate(cfg["layers"]):
        if e.get("weights_of") is not None:
            continue
        m, p = e["mixer"], f"l{i}."
        H = m["heads"]
        norms = ["norm1"]
        if e["type"] == "attention":
            D, G = m["dim"], m["kv_heads"]
            mix = {"q": (H * D, W), "k": (G * D, W), "o": (W, H * D)}
            mix.update({"v": (G * D, W), "rel": (32, H)} if "bias_max" in m else {"sink": (H,)})
        elif e["type"] == "latent_attention":
            K, R, D = m["kv_rank"], m["rot_dim"], m["dim"]
            mix = {"q": (H * (D + R), W), "dkv": (K + R, W), "dkv.norm": (K,), "uk": (H * D, K), "uv": (H * D, K), "sink": (H,),
                   "o": (W, H * D)}
        elif e["type"] == "mamba2":
            inner, ch = H * m["vdim"], H * m["vdim"] + 2 * m["groups"] * m["state"]
            mix = {"in": (inner + ch + H, W), "conv": (ch, m["conv"]), "conv.b": (ch,), "dt_bias": (H,), "A_log": (H,), "D": (H,),
                   "norm": (inner,), "o": (W, inner)}
        else:
            N, P = m["dim"], m["vdim"]
            mix = {"q": (H * N, W), "k": (H * N, W), "v": (H * P, W), "g": (H * P, W), "o": (W, H * P), "norm": (H * P,),
                   "i": (H, W), "i.b": (H,), "f": (H, W), "f.b": (H,)}
        out.update({p + "mix." + k: v for k, v in mix.items()})
        if cfg["architecture"] == "Radapel":
            norms += ["norm1b"] + (["norm2", "norm2b"] if e["mlp"] is not None else [])
        out.update({p + k: (W,) for k in norms})
        if e["mlp"] is not None:
            F = e["mlp"]["ff"]
            out.update({p + "mlp.gate": (F, W), p + "mlp.up": (F, W), p + "mlp.down": (W, F)})
    return out


def _weights(cfg, seed):
    """A checkpoint: matrices of variance 1 / inputs, norms near one, recurrence constants in their usual ranges."""
    g, randn = _random(seed)
    out = {}
    for name, shape in _tensor_shapes(cfg).items():
        leaf = name.split("mix.")[-1] if "mix." in name else name.split(".")[-1]
        x = randn(*shape)
        if "norm" in name.split("mix.")[-1]:
            x = 1.0 + 0.1 * x
        elif leaf == "planes":
            pass
        elif leaf == "protos_T":
            x = _prototypes()
        elif leaf == "A_log":
            x = torch.log(1.0 + 15.0 * torch.rand(shape, generator=g, device=DEV))
        elif leaf == "dt_bias":
            x = torch.log(torch.expm1(torch.exp(-6.9 + 4.6 * torch.rand(shape, generator=g, device=DEV))))
        elif leaf == "D":
            x = torch.ones_like(x)
        elif leaf == "f.b":
            x = 3.0 + x
        elif leaf in ("embed", "step", "i.b", "conv.b", "rel"):
            x = 0.5 * x
        elif leaf != "sink" and name != "tok_embeddings.weight":
            x = x * shape[-1] ** -0.5
        out[name] = x.to(torch.bfloat16)
    for i, e in enumerate(cfg.get("layers", [])):       # keys that lean towards their queries, as a trained memory's do
        if e["type"] == "mlstm" and e.get("weights_of") is None:
            k = out[f"l{i}.mix.k"].float() + out[f"l{i}.mix.q"].float()
            out[f"l{i}.mix.k"] = (k * 0.5 ** 0.5).to(torch.bfloat16)
    return out


def _tokens(case, seed):
    n = case["start"] + case["S"] if case["kind"] == "prompt" else case["T"] + 1
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return torch.randint(0, VOCAB, (case["B"], n), generator=g, device=DEV)


def _live(caches, total):
    """Caches and states that the next token reads, rows beyond the live length left out."""
    out = []
    for c in caches:
        if hasattr(c, "conv"):                          # state space
            out += [c.state, c.conv]
        elif hasattr(c, "S"):                           # matrix memory
            out += [c.S, c.n, c.m]
        elif hasattr(c, "k"):                           # the current chunk
            n = (total - 1) % c.k.shape[1] + 1
            out += [c.k[:, :n], c.v[:, :n]]
        else:                                           # rows of the window, or of the whole sequence
            out.append(c.rows[:, :min(total, c.rows.shape[1])])
    return out


# ------------------------------------------------------------------------------------------- prepare and run
def _layer_inputs(case, seed):
    """One layer's queries, keys and values: keys with uneven channels, one in a hundred near a query's direction."""
    B, H, G, T = case["B"], case["H"], case["G"], case["T"]
    dt = DTYPES[case["dtype"]]
    g, randn = _random(seed)
    planes = randn(TABLES, PLANES, HEAD).to(dt)
    q = randn(B, H, HEAD).to(dt)
    channel = torch.exp(randn(HEAD))
    k = torch.empty(B, T + 1, G, HEAD, dtype=dt, device=DEV)
    v = torch.empty(B, T + 1, G, HEAD, dtype=dt, device=DEV)
    for b in range(B):
        kb = randn(T + 1, G, HEAD) * channel
        direction = q[b, ::H // G].float()
        near = 0.8 * direction / direction.norm(dim=-1, keepdim=True) + 0.2 * randn(T + 1, G, HEAD)
        planted = torch.rand(T + 1, G, 1, generator=g, device=DEV) < 0.01
        k[b] = torch.where(planted, near, kb).to(dt)
        v[b] = randn(T + 1, G, HEAD).to(dt)
    return planes, q, k, v


def _append_inputs(case, seed):
    B, S, G, dt = case["B"], case["S"], case["G"], DTYPES[case["dtype"]]
    _, randn = _random(seed)
    planes = randn(TABLES, PLANES, HEAD).to(dt)
    channel = torch.exp(randn(HEAD))
    return planes, (randn(B, S, G, HEAD) * channel).to(dt), randn(B, S, G, HEAD).to(dt)


def _list_inputs(case, seed):
    """What the original decode branch hands to its two operators: bucket probabilities, codes and norms expanded to
    the query heads, the live keys and values."""
    planes, q, k, v = _layer_inputs(dict(case, T=case["T"] - 1), seed)
    rep = case["H"] // case["G"]
    k, v = k.transpose(1, 2).contiguous(), v.transpose(1, 2).contiguous()
    probs = _probabilities(q.double(), planes.double()).float()
    codes = _codes(k, planes).to(torch.int16).repeat_interleave(rep, 1).transpose(2, 3).contiguous()
    norms = torch.linalg.vector_norm(v.float(), dim=-1).half().repeat_interleave(rep, 1)
    return q, k, v, probs, codes, norms, torch.ones(norms.shape, dtype=torch.bool, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        from socket_b200.attention import SocketAttention
        planes, q, k, v = _layer_inputs(case, seed)
        B, T, dt = case["B"], case["T"], DTYPES[case["dtype"]]
        attn = SocketAttention(case["H"], case["G"], HEAD, L=TABLES, P=PLANES, heavy_const=case["topk"], sink_size=case["sink"],
                               window_size=case["window"], planes=planes, protos_T=_prototypes(), dtype=dt, device=DEV)
        cache = attn.setup_cache(B, T + 64, dtype=dt)
        for s in range(0, T, 16384):
            e = min(T, s + 16384)
            cache.append(torch.arange(s, e, device=DEV), k[:, s:e], v[:, s:e], attn.planes)
        return dict(kind=kind, attn=attn, q=q, k=k[:, T:].contiguous(), v=v[:, T:].contiguous(), pos=torch.tensor([T], device=DEV),
                    state=[cache.k_cache, cache.v_cache, cache.k_hard, cache.v_norm, cache.prefill_len])
    if kind == "lists":
        q, k, v, probs, codes, norms, allowed = _list_inputs(case, seed)
        return dict(kind=kind, lists=(probs, codes, norms, allowed, case["sink"], case["window"], case["topk"]), q=q, k=k, v=v)
    if kind == "append":
        from socket_b200.attention import KVCache
        planes, k, v = _append_inputs(case, seed)
        start, S = case["start"], case["S"]
        cache = KVCache(case["B"], start + S + 8, case["G"], HEAD, L=TABLES, R=1 << PLANES, dtype=k.dtype, device=DEV)
        return dict(kind=kind, cache=cache, pos=torch.arange(start, start + S, device=DEV), k=k, v=v, planes=planes)
    from socket_b200.registry import build_model
    cfg = _config(case)
    tensors = _weights(cfg, seed)
    model = build_model(cfg, {n: tuple(t.shape) for n, t in tensors.items()}, dtype=torch.bfloat16, device=DEV)
    model.load_tensors(tensors)
    del tensors
    tokens = _tokens(case, seed)
    B, total = tokens.shape
    model.setup_caches(B, total + 8)
    if case["model"] == "transformer":                  # a context that another worker computed
        model.setup_decode(B, "sparse")
        keys = _context(case, seed)
        for layer in model.layers:
            k, v = next(keys)
            layer.attention.kv_cache.append(torch.arange(total - 1, device=DEV), k, v, layer.attention.planes)
        state = [t for y in model.layers for t in (y.attention.kv_cache.k_cache, y.attention.kv_cache.v_cache,
                                                   y.attention.kv_cache.k_hard, y.attention.kv_cache.v_norm)]
        return dict(kind=kind, model=model, token=tokens[:, -1:].contiguous(), at=total - 1, state=state)
    if kind == "token":
        model.setup_decode(B)
        model.prefill(tokens[:, :-1])
        return dict(kind=kind, model=model, token=tokens[:, -1:].contiguous(), at=total - 1, state=_live(model.caches, total))
    if case["start"]:
        model.prefill(tokens[:, :case["start"]])
    return dict(kind=kind, model=model, tokens=tokens[:, case["start"]:].contiguous(), at=case["start"],
                state=_live(model.caches, total))


def run(state):
    kind = state["kind"]
    if kind == "step":
        return [state["attn"].sparse_decode(state["q"], state["k"], state["v"], state["pos"])] + state["state"]
    if kind == "lists":
        from socket_b200.kernels.sparse import build_sparse_list_decode, sparse_attention_fwd
        lst, length = build_sparse_list_decode(*state["lists"])
        return [sparse_attention_fwd(state["q"], state["k"], state["v"], lst, length), lst, length]
    if kind == "append":
        cache = state["cache"]
        cache.append(state["pos"], state["k"], state["v"], state["planes"])
        return [cache.k_cache, cache.v_cache, cache.k_hard, cache.v_norm, cache.prefill_len]
    if kind == "token":
        return [state["model"].decode_given_token(state["token"], state["at"])] + state["state"]
    return [state["model"].forward_portion(state["tokens"], state["at"])] + state["state"]


# ------------------------------------------------------------------------------------------- work and tolerance
def _selected(case):
    T = case["T"] + (case["kind"] != "lists")
    sink, window = min(case["sink"], T), min(case["window"], T)
    return max(1, sink + min(window, T - sink)) + min(case["topk"], T)


def _model_work(cfg, B, start, S):
    """Bytes and operations of S tokens of B sequences behind `start` cached ones."""
    rows, total = B * S, start + S
    shapes = _tensor_shapes(cfg)
    size = lambda p: sum(math.prod(s) for n, s in shapes.items() if n.startswith(p) and len(s) == 2)  # noqa: E731
    read = sum(math.prod(s) for n, s in shapes.items() if n != "embed") * 2 + rows * cfg["width"] * 2
    flops, moved = 2.0 * B * VOCAB * cfg["width"], 4.0 * B * VOCAB
    for i, first in _runs(cfg):
        e = cfg["layers"][i]
        m = e["mixer"]
        flops += 2.0 * rows * (size(f"l{i}.") + (size("loop.in") if first is not None else 0))
        if e["type"] == "mamba2":
            state = m["heads"] * m["state"] * m["vdim"]
            flops += 6.0 * rows * state
            moved += 4.0 * B * state * (2 if start else 1)
        elif e["type"] == "mlstm":
            state = m["heads"] * m["dim"] * m["vdim"]
            flops += 6.0 * rows * state
            moved += 4.0 * B * state * (2 if start else 1)
        else:
            span = m["mask"]["size"] if "mask" in m else total
            if "bias_max" in m:                         # chunks: positions seen, summed over the portion's tokens
                seen = sum(p % span + 1 for p in range(start, total))
                old = start % span
            else:
                seen = sum(min(p + 1, span) for p in range(start, total))
                old = min(start, span)
            kv = 2 * m["dim"] if "kv_rank" not in m else 2 * m["dim"] + m["rot_dim"]
            flops += 2.0 * B * m["heads"] * seen * kv
            row = (m["kv_rank"] + m["rot_dim"]) if "kv_rank" in m else m["kv_heads"] * (2 * m["dim"] if "bias_max" in m
                                                                                       else m["dim"] + TURNED)
            moved += 2.0 * B * row * (old + min(S, span))
    return {"bytes": read + moved, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "append":
        n, es = case["B"] * case["S"] * case["G"], BYTES[case["dtype"]]
        return {"bytes": n * (4 * HEAD * es + TABLES + 2), "flops": 2.0 * n * TABLES * PLANES * HEAD}
    if kind in ("step", "lists"):
        B, H, G, T, es = case["B"], case["H"], case["G"], case["T"], BYTES[case["dtype"]]
        rows = min(B * H * _selected(case), B * G * T)
        scan = B * G * T * (TABLES + 2) if kind == "step" else B * H * T * (2 * TABLES + 3)
        return {"bytes": scan + rows * 2 * HEAD * es + 2 * B * H * HEAD * es,
                "flops": 1.0 * B * H * T * TABLES + 4.0 * B * H * _selected(case) * HEAD}
    cfg = _config(case)
    if case["model"] != "transformer":
        return _model_work(cfg, case["B"], *((case["start"], case["S"]) if kind == "prompt" else (case["T"], 1)))
    params = sum(math.prod(s) for n, s in _tensor_shapes(cfg).items() if n != "tok_embeddings.weight")
    layer = work(dict(kind="step", B=case["B"], H=cfg["n_head"], G=cfg["n_local_heads"], T=case["T"], topk=cfg["heavy_const"],
                      sink=cfg["sink_size"], window=cfg["window_size"], dtype="bf16"))
    return {"bytes": 2 * params + cfg["n_layer"] * layer["bytes"], "flops": 2.0 * case["B"] * params + cfg["n_layer"] * layer["flops"]}


def tolerance(case):
    if case["kind"] == "append":                        # copies and codes are exact, a norm may round to its neighbour in fp16
        return {"rel": 5e-4, "max": 2e-3}
    if case["kind"] in ("step", "lists"):
        # another order of the fp32 sums lets near-ties of scores change places, and with them a key of the list
        rel = {"bf16": 1e-2, "f16": 4e-3, "f32": 1e-3}[case["dtype"]]
        return {"rel": rel, "max": 0.1, "differ": 1e-3}
    return {"rel": 0.03, "max": 0.5, "differ": 1e-5}    # bf16 activations through seven layers


# ------------------------------------------------------------------------------------------- the same in 64 bits
def _codes(keys, planes):
    """Bucket of every key [B,G,T,D] in every table: the signs of its products with the table's planes, first plane
    most significant."""
    flat = planes.double().reshape(TABLES * PLANES, -1).t()
    bits = 2 ** torch.arange(PLANES - 1, -1, -1, device=keys.device)
    out = torch.empty(*keys.shape[:3], TABLES, dtype=torch.uint8, device=keys.device)
    for b in range(keys.shape[0]):
        for g in range(keys.shape[1]):
            sign = keys[b, g].double() @ flat >= 0
            out[b, g] = (sign.view(-1, TABLES, PLANES) * bits).sum(-1).to(torch.uint8)
    return out


def _probabilities(q, planes):
    t = torch.tanh(torch.einsum("bhd,lpd->bhlp", q, planes)) / math.sqrt(q.shape[-1])
    return torch.softmax(torch.einsum("bhlp,pr->bhlr", t, _prototypes().double()), -1)


def _sparse_attention(q, k, v, codes, norms, probs, topk, sink, window):
    """q [B,H,D]; k, v [B,G,T,D]; codes [B,G,T,L]; norms [B,G,T] -> [B,H,D]: softmax over first, last and top-scored keys,
    each counted as often as it is listed."""
    B, H, D = q.shape
    G, T = k.shape[1:3]
    sink, window = min(sink, T), min(window, T)
    base = torch.cat([torch.arange(sink, device=DEV), torch.arange(max(T - window, sink), T, device=DEV)])
    if base.numel() == 0:
        base = torch.tensor([T - 1], device=DEV)
    out = torch.empty(B, H, D, dtype=torch.float64, device=DEV)
    for b in range(B):
        for h in range(H):
            g = h // (H // G)
            score = torch.zeros(T, dtype=torch.float64, device=DEV)
            for table in range(TABLES):
                score += probs[b, h, table].double()[codes[b, g, :, table].long()]
            rows = torch.cat([base, torch.topk(score * norms[b, g].double(), min(topk, T)).indices])
            p = torch.softmax(k[b, g, rows].double() @ q[b, h].double() / math.sqrt(D), 0)
            out[b, h] = p @ v[b, g, rows].double()
    return out


def _norms(v):
    return torch.linalg.vector_norm(v.float(), dim=-1).half()


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, eps):
    return _rms(x - x.mean(-1, keepdim=True), w, eps)


def _frequencies(rot):
    """Angle per position of each pair; with scaling, slow pairs turn slower, pairs between are blended."""
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, device=DEV, dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    if s is None:
        return f, 1.0
    pair = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _turn(x, rot, halves):
    """Rotate the last axis of x [B,S,...,dims] by each position's angles: interleaved pairs, or element i with i + dims / 2."""
    f, gain = _frequencies(rot)
    a = torch.arange(x.shape[1], device=DEV, dtype=torch.float64)[:, None] * f
    for _ in range(x.dim() - 3):
        a = a.unsqueeze(1)
    c, s = torch.cos(a) * gain, torch.sin(a) * gain
    u, v = x.chunk(2, -1) if halves else (x[..., 0::2], x[..., 1::2])
    y = (u * c - v * s, v * c + u * s)
    return torch.cat(y, -1) if halves else torch.stack(y, -1).flatten(-2)


def _attend(q, k, v, scale, span, chunks, bias=None, cap=0.0, sink=None):
    """Causal attention q [B,S,H,D], k, v [B,S,G,D]: inside chunks of `span` positions, or over the last `span` ones."""
    B, S, H, _ = q.shape
    rep, out = H // k.shape[2], torch.empty(*q.shape[:3], v.shape[3], dtype=q.dtype, device=DEV)
    step = 256
    for i0 in range(0, S, step):
        i1 = min(S, i0 + step)
        lo = i0 // span * span if chunks else max(0, i0 - span + 1)
        i, j = torch.arange(i0, i1, device=DEV)[:, None], torch.arange(lo, i1, device=DEV)[None]
        seen = (j <= i) & ((i // span == j // span) if chunks else (i - j < span))
        for b in range(B):
            for h in range(H):
                s = q[b, i0:i1, h] @ k[b, lo:i1, h // rep].t() * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                if bias is not None:
                    s = s + bias[h][(i - j).clamp(0, bias.shape[1] - 1)]
                s = s.masked_fill(~seen, -math.inf)
                top = s.amax(-1, keepdim=True)
                if sink is not None:
                    top = torch.maximum(top, sink[h])
                e = torch.exp(s - top)
                den = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0)
                out[b, i0:i1, h] = e / den @ v[b, lo:i1, h // rep]
    return out


def _bias_per_distance(rel, far):
    """[H, far + 1] from rows per bucket: half of them one distance each, the others growing logarithmically to `far`."""
    rows = rel.shape[0]
    half = rows // 2
    n = torch.arange(far + 1, dtype=torch.float64)
    grown = half + torch.floor(torch.log(n.clamp(min=1) / half) / math.log(far / half) * (rows - half) + 1e-9)
    at = torch.where(n < half, n, grown).clamp(max=rows - 1).long()
    return rel[at.to(DEV)].t()


def _chunk_attention(h, w, m):
    B, S, _ = h.shape
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (h @ w["q"].t()).view(B, S, H, D), (h @ w["k"].t()).view(B, S, G, D), (h @ w["v"].t()).view(B, S, G, D)
    C = m["mask"]["size"]
    y = _attend(q, k, v, m["scale"], C, True, bias=_bias_per_distance(w["rel"], m["bias_max"]))
    lo = (S - 1) // C * C
    return y.flatten(2) @ w["o"].t(), [k[:, lo:], v[:, lo:]]


def _latent_attention(h, w, m, eps):
    B, S, _ = h.shape
    H, D, R, K = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    q, dkv = (h @ w["q"].t()).view(B, S, H, D + R), h @ w["dkv"].t()
    c, turned = _rms(dkv[..., :K], w["dkv.norm"], eps), _turn(dkv[..., K:], m["rot"], False)
    q = torch.cat([q[..., :D], _turn(q[..., D:], m["rot"], False)], -1)
    k = torch.cat([(c @ w["uk"].t()).view(B, S, H, D), turned[:, :, None].expand(B, S, H, R)], -1)
    y = _attend(q, k, (c @ w["uv"].t()).view(B, S, H, D), m["scale"], S, False, sink=w["sink"])
    return y.flatten(2) @ w["o"].t(), [torch.cat([c, turned], -1)]


def _window_attention(h, w, m):
    B, S, _ = h.shape
    H, G, D, R, W = m["heads"], m["kv_heads"], m["dim"], m["rot"]["dims"], m["mask"]["size"]
    q, k = (h @ w["q"].t()).view(B, S, H, D), (h @ w["k"].t()).view(B, S, G, D)
    turn = lambda x: torch.cat([x[..., R:], _turn(x[..., :R], m["rot"], True)], -1)  # noqa: E731
    kr = turn(k)
    y = _attend(turn(q), kr, k, m["scale"], W, False, cap=m["softcap"], sink=w["sink"])
    rows = torch.cat([k, kr[..., D - R:]], -1)          # a position p lives in row p % W
    ring = torch.empty(B, min(S, W), G, D + R, dtype=h.dtype, device=DEV)
    last = torch.arange(max(0, S - W), S, device=DEV)
    ring[:, last % W] = rows[:, last]
    return y.flatten(2), [ring]


def _state_space(h, w, m, eps):
    B, S, _ = h.shape
    H, P, N, G, taps = m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
    inner, parts = H * P, m["norm_groups"]
    z, xbc, dt = (h @ w["in"].t()).split([inner, inner + 2 * G * N, H], -1)
    padded = torch.cat([xbc.new_zeros(B, taps - 1, xbc.shape[2]), xbc], 1)
    conv = sum(padded[:, j:j + S] * w["conv"][:, j] for j in range(taps)) + w["conv.b"]
    x, Bm, C = (conv / (1 + torch.exp(-conv))).split([inner, G * N, G * N], -1)
    x, Bm, C = x.reshape(B, S, H, P), Bm.reshape(B, S, G, N).repeat_interleave(H // G, 2), C.reshape(B, S, G, N).repeat_interleave(H // G, 2)
    dt = torch.logaddexp(dt + w["dt_bias"], dt.new_zeros(()))
    rate = -torch.exp(w["A_log"])
    st, y = x.new_zeros(B, H, N, P), torch.empty_like(x)
    for s in range(0, S, 64):                           # blocks: tokens of a block see its state and one another
        e = min(S, s + 64)
        cum = torch.cumsum(dt[:, s:e] * rate, 1).transpose(1, 2)                       # [B,H,t]
        keep = torch.tril(torch.ones(e - s, e - s, dtype=torch.bool, device=DEV))
        pair = torch.einsum("bthn,bshn->bhts", C[:, s:e], Bm[:, s:e])
        pair = pair * torch.exp((cum[..., :, None] - cum[..., None, :]).masked_fill(~keep, -math.inf)) * dt[:, s:e].transpose(1, 2)[:, :, None]
        y[:, s:e] = (torch.einsum("bhts,bshp->bthp", pair, x[:, s:e]) +
                     torch.einsum("bthn,bhnp->bthp", C[:, s:e], st) * torch.exp(cum).transpose(1, 2)[..., None])
        left = torch.exp(cum[..., -1:] - cum).transpose(1, 2) * dt[:, s:e]
        st = st * torch.exp(cum[..., -1])[..., None, None] + torch.einsum("bshn,bshp->bhnp", Bm[:, s:e] * left[..., None], x[:, s:e])
    y = (y + w["D"][:, None] * x).reshape(B, S, inner) * (z / (1 + torch.exp(-z)))
    y = _rms(y.view(B, S, parts, -1), 1.0, eps).reshape(B, S, inner) * w["norm"]
    return y @ w["o"].t(), [st, padded[:, S:]]


def _memory(h, w, m, eps):
    B, S, _ = h.shape
    H, N, P, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k = (h @ w["q"].t()).view(B, S, H, N) * N ** -0.5, (h @ w["k"].t()).view(B, S, H, N)
    v = (h @ w["v"].t()).view(B, S, H, P)
    gate = lambda n: cap * torch.tanh((h @ w[n].t() + w[n + ".b"]) / cap)  # noqa: E731
    b = torch.cumsum(torch.nn.functional.logsigmoid(gate("f")), 1).transpose(1, 2)     # [B,H,S]
    a = gate("i").transpose(1, 2) - b
    M = torch.cummax(a, -1).values.clamp(min=0)         # the running maximum m_t is b_t + M_t, from 0
    st, n, at = h.new_zeros(B, H, N, P), h.new_zeros(B, H, N), h.new_zeros(B, H)
    o = torch.empty_like(v)
    for s in range(0, S, 64):
        e = min(S, s + 64)
        keep = torch.tril(torch.ones(e - s, e - s, dtype=torch.bool, device=DEV))
        pair = torch.einsum("bthn,bshn->bhts", q[:, s:e], k[:, s:e])
        pair = pair * torch.exp((a[..., None, s:e] - M[..., s:e, None]).masked_fill(~keep, -math.inf))
        old = torch.exp(at[..., None] - M[..., s:e])
        num = torch.einsum("bhts,bshp->bthp", pair, v[:, s:e]) + torch.einsum("bthn,bhnp,bht->bthp", q[:, s:e], st, old)
        den = pair.sum(-1) + torch.einsum("bthn,bhn,bht->bht", q[:, s:e], n, old)
        den = torch.maximum(den.abs(), torch.exp(-(b + M)[..., s:e])) + 1e-6
        o[:, s:e] = num / den.transpose(1, 2)[..., None]
        end = M[..., e - 1]
        kw = k[:, s:e] * torch.exp(a[..., s:e] - end[..., None]).transpose(1, 2)[..., None]
        st = st * torch.exp(at - end)[..., None, None] + torch.einsum("bshn,bshp->bhnp", kw, v[:, s:e])
        n = n * torch.exp(at - end)[..., None] + kw.sum(1)
        at = end
    o = _rms(o, 1.0, eps).reshape(B, S, H * P) * w["norm"]
    return o / (1 + torch.exp(-(h @ w["g"].t()))), [st, n, (b + M)[..., -1]]


def _exact_decoder(cfg, tokens, weights):
    w = {n: t.double() for n, t in weights.items()}
    eps = cfg["norm"]["eps"]
    x0 = x = w["embed"][tokens] * cfg["embedding"]["scale"]
    radapel, state = cfg["architecture"] == "Radapel", []
    for i, first in _runs(cfg):
        e, p = cfg["layers"][i], f"l{i}."
        m, mix = e["mixer"], {n[len(p) + 4:]: t for n, t in w.items() if n.startswith(p + "mix.")}
        mlp = {n[len(p) + 4:]: t for n, t in w.items() if n.startswith(p + "mlp.")}
        if radapel:
            if first is not None:
                x = torch.cat([x, x0], -1) @ w["loop.in"].t() + w["loop.step"][first]
            h = _rms(x, w[p + "norm1"], eps)
            if e["type"] == "attention":
                y, s = _chunk_attention(h, mix, m)
            else:
                y, s = (_latent_attention if e["type"] == "latent_attention" else _state_space)(h, mix, m, eps)
            x = x + _rms(y, w[p + "norm1b"], eps)
            if mlp:
                h, limit = _rms(x, w[p + "norm2"], eps), e["mlp"]["limit"]
                gate, up = (h @ mlp["gate"].t()).clamp(max=limit), (h @ mlp["up"].t()).clamp(-limit, limit)
                x = x + _rms((gate / (1 + torch.exp(-1.702 * gate)) * (up + 1)) @ mlp["down"].t(), w[p + "norm2b"], eps)
        else:
            h = _layer_norm(x, w[p + "norm1"], eps)
            y, s = _window_attention(h, mix, m) if e["type"] == "attention" else _memory(h, mix, m, eps)
            gate = h @ mlp["gate"].t()
            x = x + y @ mix["o"].t() + (gate / (1 + torch.exp(-gate)) * (h @ mlp["up"].t())) @ mlp["down"].t()
        state += s
    last = (_rms if radapel else _layer_norm)(x[:, -1:], w["final.norm"], eps) @ w["head"].t()
    return last, state


def _context(case, seed):
    """Keys and values [B,T,G,D] of the cached context, layer by layer."""
    _, randn = _random(seed + 2)
    shape = (case["B"], case["T"], TRANSFORMER["n_local_heads"], HEAD)
    for _ in range(TRANSFORMER["n_layer"]):
        yield (randn(*shape) * torch.exp(0.5 * randn(HEAD))).to(torch.bfloat16), randn(*shape).to(torch.bfloat16)


def _exact_transformer(case, seed):
    cfg = _config(case)
    w = _weights(cfg, seed)
    token, B, T, G = _tokens(case, seed)[:, -1], case["B"], case["T"], cfg["n_local_heads"]
    H, cap = cfg["n_head"], (case["T"] + 9 + 7) // 8 * 8
    i = torch.arange(0, HEAD, 2, device=DEV).float()
    angle = torch.arange(cap, device=DEV).float()[:, None] * (1.0 / (cfg["rope_base"] ** (i / HEAD)))
    c, s = (t[T].to(torch.bfloat16).double() for t in (torch.cos(angle), torch.sin(angle)))   # the table is bf16 by design

    def turn(x):
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    x = w["tok_embeddings.weight"][token].double()
    state = []
    for n, (k, v) in enumerate(_context(case, seed)):
        m = {a[len(f"layers.{n}."):]: t.double() for a, t in w.items() if a.startswith(f"layers.{n}.")}
        h = _rms(x, m["attention_norm.weight"], 1e-5)
        q, k1, v1 = (h @ m["attention.wqkv.weight"].t()).split([H * HEAD, G * HEAD, G * HEAD], -1)
        q, k1, v1 = turn(q.view(B, H, HEAD)), turn(k1.view(B, G, HEAD)), v1.view(B, G, HEAD)
        k = torch.cat([k.transpose(1, 2).double(), k1[:, :, None]], 2)
        v = torch.cat([v.transpose(1, 2).double(), v1[:, :, None]], 2)
        planes, norms = m["attention.planes"], torch.linalg.vector_norm(v, dim=-1)
        y = _sparse_attention(q, k, v, _codes(k, planes), norms.half(), _probabilities(q, planes), cfg["heavy_const"],
                              cfg["sink_size"], cfg["window_size"])
        x = x + y.reshape(B, -1) @ m["attention.wo.weight"].t()
        h = _rms(x, m["ffn_norm.weight"], 1e-5)
        a, b = (h @ m["feed_forward.w13.weight"].t()).chunk(2, -1)
        x = x + (a / (1 + torch.exp(-a)) * b) @ m["feed_forward.w2.weight"].t()
        pad = lambda t: torch.nn.functional.pad(t, (0, 0, 0, cap - T - 1))  # noqa: E731
        state += [pad(k), pad(v), None, pad(norms[..., None])[..., 0]]
    return [_rms(x, w["norm.weight"].double(), 1e-5) @ w["output.weight"].double().t()] + state


def exact(case, seed):
    kind = case["kind"]
    if kind == "append":
        planes, k, v = _append_inputs(case, seed)
        start = case["start"]
        pad = lambda t: torch.nn.functional.pad(t.transpose(1, 2), (0, 0, start, 8))  # noqa: E731
        norms = torch.linalg.vector_norm(v.double(), dim=-1)[..., None]
        return [pad(k), pad(v), None, pad(norms)[..., 0], None]
    if kind == "step":
        planes, q, k, v = _layer_inputs(case, seed)
        k, v = (torch.nn.functional.pad(t.transpose(1, 2), (0, 0, 0, 63)) for t in (k, v))
        kl, vl = k[:, :, :case["T"] + 1], v[:, :, :case["T"] + 1]
        out = _sparse_attention(q, kl, vl, _codes(kl, planes), _norms(vl), _probabilities(q.double(), planes.double()),
                                case["topk"], case["sink"], case["window"])
        return [out, k, v, None, torch.linalg.vector_norm(v.float(), dim=-1), None]
    if kind == "lists":
        q, k, v, probs, _, norms, _ = _list_inputs(case, seed)
        planes = _layer_inputs(dict(case, T=case["T"] - 1), seed)[0]
        out = _sparse_attention(q, k, v, _codes(k, planes), norms[:, ::case["H"] // case["G"]], probs, case["topk"], case["sink"],
                                case["window"])
        return [out, None, None]
    if case["model"] == "transformer":
        return _exact_transformer(case, seed)
    cfg = _config(case)
    logits, state = _exact_decoder(cfg, _tokens(case, seed), _weights(cfg, seed))
    return [logits if kind == "prompt" else logits[:, 0]] + state
