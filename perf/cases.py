"""What is measured: training steps and serving steps of language models through the framework's model interface.

* ``train``: ``compute_next_token_loss`` of a model on an ``LmExample`` and its backward pass, as a training step on one GPU does
  it; the loss and every parameter's gradient come back.
* ``prefill``: ``model.decode`` over packed prompts that all start here, as the serving engine runs them: keys and values enter the
  page caches, the last token of every prompt is scored.
* ``decode``: one serving round, ``model.decode`` of one new token per sequence over the page caches and the sampler on its logits,
  captured once in a CUDA graph and replayed, as the serving engine does with ``use_cuda_graph``.

Widths, heads and vocabularies are those of this repository's configs (``config/*.yaml``) and serving benchmark; the models have a
few of their layers, so that a pass is a few milliseconds and not the same layer over and over.  Weights are drawn like an
initialised model's, tokens uniformly, prompt and context lengths ragged."""
import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

PAGE = 16

MODELS = {
    # config/gpt2_small_b200.yaml with its tokenizer's vocabulary: head size 64, learned positions, biases, a tied head
    "gpt2_small": dict(family="gpt2", hidden=768, heads=12, vocab=50257, positions=1024),
    # config/llama2_7b_b200.yaml: the training benchmark's model
    "llama2_7b": dict(family="llama", hidden=4096, ff=11008, heads=32, kv=32, size=128, vocab=32000),
    # config/qwen3_1_7b.yaml: grouped queries, norms of the heads
    "qwen3_1_7b": dict(family="qwen3", hidden=2048, ff=6144, heads=16, kv=8, size=128, vocab=32000),
    # config/gated_deltanet_400m.yaml: linear attention with a matrix state
    "gated_deltanet": dict(family="gdn", hidden=1024, ff=2816, heads=8, size=128, vocab=50257),
    # the serving benchmark's models (levanter_b200/inference/bench_decode.py)
    "llama3_8b": dict(family="llama", hidden=4096, ff=14336, heads=32, kv=8, size=128, vocab=128256),
    "llama_1b": dict(family="llama", hidden=2048, ff=8192, heads=32, kv=8, size=64, vocab=128256),
}
THETA = 500000.0


def listed():
    return [
        # a training step on documents packed to the context of GPT-2 small, the size that is trained on one GPU
        dict(name="train_gpt2_small", kind="train", model="gpt2_small", layers=4, batch=8, length=1024, documents=1, recompute=False),
        # a small ragged batch: fine-tuning, tests, evaluation while training; latency and launches count
        dict(name="train_gpt2_short", kind="train", model="gpt2_small", layers=2, batch=3, length=333, documents=1, recompute=False),
        # the training benchmark's micro-batch
        dict(name="train_llama2_7b", kind="train", model="llama2_7b", layers=2, batch=2, length=4096, documents=1, recompute=False),
        # documents packed into one sequence (segment ids), grouped queries, a length that is no multiple of a tile
        dict(name="train_qwen3_packed", kind="train", model="qwen3_1_7b", layers=4, batch=2, length=3000, documents=5, recompute=False),
        # linear attention at its config's length, layers recomputed in the backward pass as its config asks
        dict(name="train_gdn", kind="train", model="gated_deltanet", layers=2, batch=4, length=4096, documents=1, recompute=True),
        # one ragged sequence: fine-tuning on long documents
        dict(name="train_gdn_short", kind="train", model="gated_deltanet", layers=2, batch=1, length=1500, documents=1, recompute=False),
        # one short prompt arrives: the time to the first token
        dict(name="prefill_1", kind="prefill", model="llama_1b", layers=4, batch=1, length=200, ragged=False),
        # a full prefill step of the engine
        dict(name="prefill_16", kind="prefill", model="llama3_8b", layers=4, batch=16, length=1024, ragged=True),
        # one user, a small model: the latency of a round
        dict(name="decode_1", kind="decode", model="llama_1b", layers=2, batch=1, length=300, ragged=False),
        # a few users
        dict(name="decode_8", kind="decode", model="llama3_8b", layers=4, batch=8, length=1500, ragged=True),
        # the serving benchmark's batch over long contexts
        dict(name="decode_64", kind="decode", model="llama3_8b", layers=4, batch=64, length=4096, ragged=True),
        # 256 concurrent requests with prompts of up to 2048 and 256 new tokens
        dict(name="decode_256", kind="decode", model="llama3_8b", layers=4, batch=256, length=2304, ragged=True),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train", "train", "prefill", "decode", "decode"])
    if kind == "train":
        model, layers, most, longest = rng.choice([("gpt2_small", 4, 8192, 1024), ("llama2_7b", 2, 8192, 4096), ("qwen3_1_7b", 4, 8192, 4096),
                                                   ("gated_deltanet", 2, 16384, 4096)])
        length = _log_uniform(rng, 192, longest)
        if rng.random() < 0.4:
            length = length // 64 * 64
        return dict(kind=kind, model=model, layers=rng.randint(1, layers), batch=_log_uniform(rng, 1, max(1, min(16, most // length))), length=length,
                    documents=rng.randint(2, 8) if model in ("llama2_7b", "qwen3_1_7b") and rng.random() < 0.4 else 1, recompute=rng.random() < 0.3)
    model = rng.choice(["llama3_8b", "llama_1b"])
    if kind == "prefill":
        batch = _log_uniform(rng, 1, 16)
        length = _log_uniform(rng, 16, 16384 // batch if batch > 4 else 4096)
    else:
        batch, length = _log_uniform(rng, 1, 256), 0
        length = _log_uniform(rng, 32, 2304 if batch > 64 else 4096)
    return dict(kind=kind, model=model, layers=rng.randint(2, 4), batch=batch, length=length, ragged=rng.random() < 0.7)


# ---------------------------------------------------------------------------------------------------------------- inputs from a seed
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt) % (1 << 62))


def _shapes(case):
    """Name -> (shape, kind) of the model's parameters; kind: w (a matrix), n (a norm's weight), b (a bias), a, d (decays)."""
    m, out = MODELS[case["model"]], {}
    E, V = m["hidden"], m["vocab"]
    if m["family"] == "gpt2":
        for i in range(case["layers"]):
            p = f"transformer.blocks.{i}."
            out.update({p + "ln_1.weight": ((E,), "n"), p + "ln_1.bias": ((E,), "b"), p + "attn.c_attn.weight": ((3 * E, E), "w"),
                        p + "attn.c_attn.bias": ((3 * E,), "b"), p + "attn.c_proj.weight": ((E, E), "w"), p + "attn.c_proj.bias": ((E,), "b"),
                        p + "ln_2.weight": ((E,), "n"), p + "ln_2.bias": ((E,), "b"), p + "mlp.c_fc.weight": ((4 * E, E), "w"),
                        p + "mlp.c_fc.bias": ((4 * E,), "b"), p + "mlp.c_proj.weight": ((E, 4 * E), "w"), p + "mlp.c_proj.bias": ((E,), "b")})
        out.update({"transformer.ln_f.weight": ((E,), "n"), "transformer.ln_f.bias": ((E,), "b"),
                    "embeddings.token_embeddings.weight": ((V, E), "w"), "embeddings.position_embeddings.weight": ((m["positions"], E), "w")})
        return out
    ff, H, D = m["ff"], m["heads"], m["size"]
    for i in range(case["layers"]):
        if m["family"] == "gdn":
            p = f"layers.{i}."
            out.update({p + "attn_norm.weight": ((E,), "n"), p + "mlp_norm.weight": ((E,), "n")})
            out.update({p + f"attn.{x}_proj.weight": ((H * D, E), "w") for x in "qkvg"})
            out.update({p + f"attn.{x}_proj.weight": ((H, E), "w") for x in "ab"})
            out.update({p + f"attn.{x}_conv1d.weight": ((H * D, 1, 4), "c") for x in "qkv"})
            out.update({p + "attn.o_proj.weight": ((E, H * D), "w"), p + "attn.A_log": ((H,), "a"), p + "attn.dt_bias": ((H,), "d"),
                        p + "attn.o_norm_weight": ((D,), "n")})
        else:
            p = f"transformer.layers.{i}."
            out.update({p + "input_layernorm.weight": ((E,), "n"), p + "post_attention_layernorm.weight": ((E,), "n"),
                        p + "self_attn.q_proj.weight": ((H * D, E), "w"), p + "self_attn.k_proj.weight": ((m["kv"] * D, E), "w"),
                        p + "self_attn.v_proj.weight": ((m["kv"] * D, E), "w"), p + "self_attn.o_proj.weight": ((E, H * D), "w")})
            if m["family"] == "qwen3":
                out.update({p + "self_attn.q_norm.weight": ((D,), "n"), p + "self_attn.k_norm.weight": ((D,), "n")})
        out.update({p + "mlp.gate_proj.weight": ((ff, E), "w"), p + "mlp.up_proj.weight": ((ff, E), "w"), p + "mlp.down_proj.weight": ((E, ff), "w")})
    out["norm.weight" if m["family"] == "gdn" else "transformer.norm.weight"] = ((E,), "n")
    out["embeddings.weight" if m["family"] == "gdn" else "embeddings.token_embeddings.weight"] = ((V, E), "w")
    out["lm_head.weight"] = ((V, E), "w")
    return out


def _weights(case, seed):
    """The parameters' values in bf16, made from the seed alone."""
    g, out = _generator(seed, 1), {}
    for name, (shape, kind) in _shapes(case).items():
        x = torch.empty(shape, dtype=torch.bfloat16 if kind == "w" else torch.float32, device="cuda")
        if kind == "a":  # decay rates of 1 to 16
            x.uniform_(1.0, 16.0, generator=g).log_()
        elif kind == "d":  # time steps of 0.001 to 0.1, through the inverse of softplus
            x.uniform_(math.log(0.001), math.log(0.1), generator=g).exp_()
            x = x + torch.log(-torch.expm1(-x))
        else:
            x.normal_(0.0, 0.3 if kind == "c" else 0.02, generator=g)
            if kind == "n":
                x += 1.0
        out[name] = x.bfloat16()
    return out


def _tokens(case, seed, count):
    return torch.randint(0, MODELS[case["model"]]["vocab"], (count,), generator=_generator(seed, 2), device="cuda", dtype=torch.int32)


def _segments(case, seed):
    """Document numbers ``[batch, length]`` of packed sequences, or None."""
    if case["documents"] == 1:
        return None
    r = np.random.RandomState(seed % (1 << 31))
    cuts = np.stack([np.isin(np.arange(case["length"]), r.choice(np.arange(1, case["length"]), case["documents"] - 1, replace=False))
                     for _ in range(case["batch"])])
    return torch.from_numpy(np.cumsum(cuts, axis=1).astype(np.int32)).cuda()


def _lengths(case, seed):
    """Tokens of each sequence: the prompts, or the contexts that a decode round reads (its new token included)."""
    if not case["ragged"]:
        return [case["length"]] * case["batch"]
    r = np.random.RandomState(seed % (1 << 31))
    return [int(x) for x in r.randint(max(2, case["length"] // 16), case["length"] + 1, case["batch"])]


def _config(case):
    m = MODELS[case["model"]]
    kw = dict(hidden_dim=m["hidden"], num_layers=case["layers"], num_heads=m["heads"], gradient_checkpointing=bool(case.get("recompute")))
    if m["family"] == "gpt2":
        from levanter_b200.models.gpt2 import Gpt2Config

        return Gpt2Config(seq_len=m["positions"], scale_attn_by_inverse_layer_idx=True, **kw)
    kw.update(seq_len=max(case["length"], 128), intermediate_dim=m["ff"])
    if m["family"] == "gdn":
        from levanter_b200.models.gated_deltanet import GatedDeltaNetConfig

        return GatedDeltaNetConfig(head_k_dim=m["size"], head_v_dim=m["size"], **kw)
    from levanter_b200.layers.rotary import DefaultRotaryEmbeddingsConfig
    from levanter_b200.models.llama import LlamaConfig
    from levanter_b200.models.qwen import Qwen3Config

    kw.update(num_kv_heads=m["kv"], rope=DefaultRotaryEmbeddingsConfig(theta=THETA))
    return Qwen3Config(head_dim=m["size"], **kw) if m["family"] == "qwen3" else LlamaConfig(**kw)


def _model(case, seed):
    w = _weights(case, seed)
    model = _config(case).build(MODELS[case["model"]]["vocab"], device="cuda", dtype=torch.bfloat16)
    params = dict(model.named_parameters())
    assert set(params) == set(w), set(params) ^ set(w)
    for name, p in params.items():
        assert p.shape == w[name].shape, name
        p.data = w[name]
    return model


def _table(case, lengths):
    """A page table that holds ``lengths`` tokens of every sequence; the pages of the sequences lie among one another, as they do after
    some rounds of decoding."""
    from levanter_b200.inference.page_table import PageTable

    per_seq = -(-(case["length"] + 1) // PAGE)
    t = PageTable.init(len(lengths) * per_seq, len(lengths), PAGE, per_seq)
    for s in range(len(lengths)):
        t, _ = t.assign_seq_id_to_seq(s)
    done = [0] * len(lengths)
    for part in (0.5, 0.75, 1.0):
        for s, n in enumerate(lengths):
            upto = int(n * part) if part < 1 else n
            if upto > done[s]:
                t, _ = t.allocate_for_seq(np.full(upto - done[s], s, np.int32), np.arange(done[s], upto, dtype=np.int32))
                done[s] = upto
    return t


def _cache_values(case, seed, index, like):
    """What the tokens before this round left in the cache of layer ``index``: keys and values of about the size that the layers make."""
    return like.normal_(0.0, 0.9, generator=_generator(seed, 100 + index))


def _decode_batch(case, seed):
    lengths = _lengths(case, seed)
    t = _table(case, [n - 1 for n in lengths])
    slots, pos = np.arange(len(lengths), dtype=np.int32), np.array([n - 1 for n in lengths], dtype=np.int32)
    t, info = t.allocate_for_seq(slots, pos)
    return t, info, pos


def _prefill_batch(case, seed):
    from levanter_b200.inference.page_table import INVALID, PageTable

    lengths = _lengths(case, seed)
    per_seq = -(-(case["length"] + 1) // PAGE)
    t = PageTable.init(len(lengths) * per_seq, len(lengths), PAGE, per_seq)
    for s in range(len(lengths)):
        t, _ = t.assign_seq_id_to_seq(s)
    pad = -sum(lengths) % 256  # the engine's padding of packed prompts
    slots = np.concatenate([np.full(n, s, np.int32) for s, n in enumerate(lengths)] + [np.full(pad, INVALID, np.int32)])
    pos = np.concatenate([np.arange(n, dtype=np.int32) for n in lengths] + [np.full(pad, INVALID, np.int32)])
    t, info = t.allocate_for_seq(slots, pos)
    info.prefill_segment_ids = torch.from_numpy(np.where(slots == INVALID, -1, slots).astype(np.int32))
    rows = np.cumsum(lengths) - 1
    return t, info, np.where(pos == INVALID, 0, pos).astype(np.int32), rows.astype(np.int64), lengths


# ---------------------------------------------------------------------------------------------------------------- the framework's passes
def prepare(case, seed):
    model = _model(case, seed)
    if case["kind"] == "train":
        from levanter_b200.models.lm_model import LmExample

        tokens = _tokens(case, seed, case["batch"] * case["length"]).view(case["batch"], case["length"])
        return dict(kind="train", model=model.train(), example=LmExample.causal(tokens, segment_ids=_segments(case, seed)))
    model.eval()
    if case["kind"] == "prefill":
        table, info, pos, rows, _ = _prefill_batch(case, seed)
        cache = model.initial_cache(table, dtype=torch.bfloat16)
        return dict(kind="prefill", model=model, cache=cache, info=info.to("cuda"), pos=torch.from_numpy(pos).cuda(),
                    rows=torch.from_numpy(rows).cuda(), tokens=_tokens(case, seed, len(pos)))
    from levanter_b200.layers.sampler import Sampler

    table, info, pos = _decode_batch(case, seed)
    cache = model.initial_cache(table, dtype=torch.bfloat16)
    for i, c in enumerate(cache):
        _cache_values(case, seed, i, c.kv_pages)
    state = dict(kind="decode", model=model, cache=cache, info=info.to("cuda"), pos=torch.from_numpy(pos).cuda(), tokens=_tokens(case, seed, len(pos)),
                 temperatures=torch.zeros(len(pos), dtype=torch.float32, device="cuda"),
                 keys=torch.arange(len(pos), dtype=torch.int64, device="cuda") + seed, sampler=Sampler())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            _round(state)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        state["outputs"] = _round(state)
    state["graph"] = graph
    return state


def _round(s):
    with torch.no_grad():
        logits, cache = s["model"].decode(s["tokens"], s["cache"], s["info"], s["pos"])
        _, logprobs = s["sampler"](logits, s["temperatures"], key=s["keys"])
    return dict(logits=logits, logprobs=logprobs, pages=[c.kv_pages for c in cache])


def run(state):
    if state["kind"] == "decode":
        state["graph"].replay()
        return state["outputs"]
    model = state["model"]
    if state["kind"] == "prefill":
        with torch.no_grad():
            logits, cache = model.decode(state["tokens"], state["cache"], state["info"], state["pos"], logit_rows=state["rows"])
        return dict(logits=logits, pages=[c.kv_pages for c in cache])
    from levanter_b200.models.lm_model import compute_next_token_loss

    model.zero_grad(set_to_none=True)
    loss = compute_next_token_loss(model, state["example"])
    loss.backward()
    return dict(loss=loss.detach(), grads={n: p.grad for n, p in model.named_parameters()})


# ---------------------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    m, L, B, S = MODELS[case["model"]], case["layers"], case["batch"], case["length"]
    E, V = m["hidden"], m["vocab"]
    weights = sum(math.prod(shape) for shape, _ in _shapes(case).values())
    tables = V * E + (m["positions"] * E if m["family"] == "gpt2" else 0)  # rows of embeddings are looked up, not multiplied
    body = weights - tables - (0 if m["family"] == "gpt2" else V * E)
    size = m.get("size", 64)
    width = m["heads"] * size
    if case["kind"] == "train":
        seen = S / case["documents"]  # documents of this many tokens on average
        per_pair = 0 if m["family"] == "gdn" else 2 * 2 * width * seen / 2
        per_state = 3 * 2 * size * size * m["heads"] if m["family"] == "gdn" else 0  # predict, write, read of a state
        flops = 3 * B * S * (2 * body + 2 * V * E + L * (per_pair + per_state))
        return dict(bytes=2 * 2 * weights, flops=flops)
    mean = S if not case["ragged"] else (S + max(2, S // 16)) / 2
    kv = 2 * m["kv"] * size
    if case["kind"] == "prefill":
        rows = B * mean
        return dict(bytes=2 * (body + V * E + rows * (E + L * kv) + B * V), flops=rows * (2 * body + L * 2 * 2 * width * mean / 2) + B * 2 * V * E)
    return dict(bytes=2 * (body + V * E + B * (E + L * kv * mean + V)), flops=B * (2 * body + 2 * V * E + L * 2 * 2 * width * mean))


def tolerance(case):
    # bf16 weights, activations and products over a few layers.  Four times the distance to 64 bits that was measured: 0.026 for the
    # gradients of the smallest parameters (0.02 for matrices), 0.017 for what serving returns
    return dict(rel=0.1 if case["kind"] == "train" else 0.06)


# ---------------------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope(x, pos):
    """``x [..., tokens, heads, size]`` turned by its positions, dimension ``i`` with ``i + size / 2``."""
    half = x.shape[-1] // 2
    inv = 1.0 / THETA ** (torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = (pos.double()[..., None] * inv)[..., None, :]
    u, v = x[..., :half], x[..., half:]
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), dim=-1)


def _attend(q, k, v, mask):
    """``q [S, H, D]``, ``k, v [K, KV, D]``, ``mask [S, K]``, a few heads at a time."""
    group, out = q.shape[1] // k.shape[1], []
    for h in range(k.shape[1]):
        s = torch.einsum("shd,kd->hsk", q[:, h * group:(h + 1) * group], k[:, h]) * q.shape[-1] ** -0.5
        p = torch.softmax(s.masked_fill(~mask, -math.inf), dim=-1)
        out.append(torch.einsum("hsk,kd->shd", p, v[:, h]))
    return torch.cat(out, dim=1)


def _causal(S, segments=None):
    i = torch.arange(S, device="cuda")
    m = i[:, None] >= i[None, :]
    return m if segments is None else m & (segments[:, None] == segments[None, :])


def _mlp(x, w, p):
    return (F.silu(x @ w[p + "gate_proj.weight"].t()) * (x @ w[p + "up_proj.weight"].t())) @ w[p + "down_proj.weight"].t()


def _qkv(m, h, w, p, pos):
    D, lead = m["size"], h.shape[:-1]
    q, k, v = ((h @ w[p + f"{x}_proj.weight"].t()).view(*lead, -1, D) for x in "qkv")
    if m["family"] == "qwen3":
        q, k = _rms(q, w[p + "q_norm.weight"], 1e-5), _rms(k, w[p + "k_norm.weight"], 1e-5)
    return _rope(q, pos), _rope(k, pos), v


def _llama_layer(m, x, w, p, segments):
    B, S, _ = x.shape
    h = _rms(x, w[p + "input_layernorm.weight"], 1e-5)
    q, k, v = _qkv(m, h, w, p + "self_attn.", torch.arange(S, device=x.device))
    o = torch.stack([_attend(q[b], k[b], v[b], _causal(S, None if segments is None else segments[b])) for b in range(B)])
    x = x + o.reshape(B, S, -1) @ w[p + "self_attn.o_proj.weight"].t()
    return x + _mlp(_rms(x, w[p + "post_attention_layernorm.weight"], 1e-5), w, p + "mlp.")


def _gpt2_layer(m, x, w, p, index):
    B, S, E = x.shape
    lin = lambda t, n: t @ w[p + n + ".weight"].t() + w[p + n + ".bias"]  # noqa: E731
    h = F.layer_norm(x, (E,), w[p + "ln_1.weight"], w[p + "ln_1.bias"], 1e-5)
    q, k, v = lin(h, "attn.c_attn").view(B, S, 3, m["heads"], -1).unbind(2)
    o = torch.stack([_attend(q[b] / (index + 1.0), k[b], v[b], _causal(S)) for b in range(B)])
    x = x + lin(o.reshape(B, S, E), "attn.c_proj")
    h = F.layer_norm(x, (E,), w[p + "ln_2.weight"], w[p + "ln_2.bias"], 1e-5)
    return x + lin(F.gelu(lin(h, "mlp.c_fc"), approximate="tanh"), "mlp.c_proj")


def _delta_rule(q, k, v, g, beta):
    """The gated delta rule over ``[B, H, L, D]`` in blocks of 32 positions: the writes of a block solve a triangular system."""
    B, H, L, D = q.shape
    C = 32
    pad = -L % C
    if pad:
        q, k, v = (F.pad(t, (0, 0, 0, pad)) for t in (q, k, v))
        g, beta = F.pad(g, (0, pad)), F.pad(beta, (0, pad))
    S, out = q.new_zeros(B, H, D, D), []
    low = torch.tril(torch.ones(C, C, dtype=torch.bool, device=q.device))
    eye = torch.eye(C, dtype=q.dtype, device=q.device)
    for n in range(0, L + pad, C):
        qn, kn, vn, bn = (t[:, :, n:n + C] for t in (q, k, v, beta))
        c = g[:, :, n:n + C].cumsum(-1)
        decay = (c[..., :, None] - c[..., None, :]).masked_fill(~low, -math.inf).exp()
        system = eye + torch.tril((kn @ kn.transpose(-1, -2)) * decay, -1) * bn[..., None]
        writes = torch.linalg.solve_triangular(system, bn[..., None] * (vn - c.exp()[..., None] * (kn @ S)), upper=False, unitriangular=True)
        out.append(c.exp()[..., None] * (qn @ S) + ((qn @ kn.transpose(-1, -2)) * decay) @ writes)
        S = S * c[..., -1, None, None].exp() + (kn * (c[..., -1:] - c).exp()[..., None]).transpose(-1, -2) @ writes
    return torch.cat(out, dim=2)[:, :, :L]


def _gdn_layer(m, x, w, p):
    B, S, E = x.shape
    H, D = m["heads"], m["size"]
    a = p + "attn."
    h = _rms(x, w[p + "attn_norm.weight"], 1e-6)

    def short(name):
        y = (h @ w[a + f"{name}_proj.weight"].t()).transpose(1, 2)
        y = F.conv1d(F.pad(y, (3, 0)), w[a + f"{name}_conv1d.weight"], groups=H * D)
        return F.silu(y.transpose(1, 2)).view(B, S, H, D)

    q, k, v = short("q"), short("k"), short("v")
    beta = torch.sigmoid(h @ w[a + "b_proj.weight"].t())
    g = -w[a + "A_log"].exp() * F.softplus(h @ w[a + "a_proj.weight"].t() + w[a + "dt_bias"])
    q, k, v = (t.transpose(1, 2) for t in (F.normalize(q, dim=-1) * D ** -0.5, F.normalize(k, dim=-1), v))
    o = _delta_rule(q, k, v, g.transpose(1, 2), beta.transpose(1, 2)).transpose(1, 2)
    o = _rms(o, w[a + "o_norm_weight"], 1e-6) * F.silu((h @ w[a + "g_proj.weight"].t()).view(B, S, H, D))
    x = x + o.reshape(B, S, H * D) @ w[a + "o_proj.weight"].t()
    return x + _mlp(_rms(x, w[p + "mlp_norm.weight"], 1e-6), w, p + "mlp.")


def _exact_train(case, seed):
    m, L = MODELS[case["model"]], case["layers"]
    w = {n: t.double().requires_grad_() for n, t in _weights(case, seed).items()}
    tokens = _tokens(case, seed, case["batch"] * case["length"]).view(case["batch"], -1).long()
    segments = _segments(case, seed)
    if m["family"] == "gpt2":
        x = w["embeddings.token_embeddings.weight"][tokens] + w["embeddings.position_embeddings.weight"][:case["length"]]
        for i in range(L):
            x = checkpoint(_gpt2_layer, m, x, w, f"transformer.blocks.{i}.", i, use_reentrant=False)
        x = F.layer_norm(x, (m["hidden"],), w["transformer.ln_f.weight"], w["transformer.ln_f.bias"], 1e-5)
        head = w["embeddings.token_embeddings.weight"]
    elif m["family"] == "gdn":
        x = w["embeddings.weight"][tokens]
        for i in range(L):
            x = checkpoint(_gdn_layer, m, x, w, f"layers.{i}.", use_reentrant=False)
        x, head = _rms(x, w["norm.weight"], 1e-6), w["lm_head.weight"]
    else:
        x = w["embeddings.token_embeddings.weight"][tokens]
        for i in range(L):
            x = checkpoint(_llama_layer, m, x, w, f"transformer.layers.{i}.", segments, use_reentrant=False)
        x, head = _rms(x, w["transformer.norm.weight"], 1e-5), w["lm_head.weight"]

    def summed(xs, ts):
        return F.cross_entropy(xs @ head.t(), ts, reduction="sum")

    # every token but a sequence's last one has a target, the first of the next document too
    keep = torch.ones(tokens.shape, dtype=torch.bool, device="cuda")
    keep[:, -1] = False
    rows, target = x[keep], tokens.roll(-1, dims=1)[keep]
    loss = sum(checkpoint(summed, rows[i:i + 2048], target[i:i + 2048], use_reentrant=False) for i in range(0, len(rows), 2048)) / len(rows)
    loss.backward()
    return dict(loss=loss.detach(), grads={n: t.grad for n, t in w.items()})


def _exact_serve(case, seed):
    """Prefill and decode: the sequences' tokens, their positions, and for decode the keys and values already in the pages."""
    m, L = MODELS[case["model"]], case["layers"]
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    if case["kind"] == "prefill":
        table, info, pos, rows, lengths = _prefill_batch(case, seed)
        spans = [(e - n, e) for n, e in zip(lengths, np.cumsum(lengths))]
    else:
        table, info, pos = _decode_batch(case, seed)
        spans = [(s, s + 1) for s in range(len(pos))]
    tokens, dests = _tokens(case, seed, len(pos)).long(), info.new_token_dests.cuda().long()
    pos = torch.from_numpy(pos).cuda().long()
    used = spans[-1][1]
    x, pages = w["embeddings.token_embeddings.weight"][tokens[:used]], []
    for i in range(L):
        p = f"transformer.layers.{i}."
        cache = torch.zeros(table.num_pages, PAGE, 2 * m["kv"], m["size"], dtype=torch.bfloat16, device="cuda")
        if case["kind"] == "decode":
            _cache_values(case, seed, i, cache)
        cache = cache.double()
        q, k, v = _qkv(m, _rms(x, w[p + "input_layernorm.weight"], 1e-5), w, p + "self_attn.", pos[:used])
        flat = cache.view(-1, m["kv"], 2, m["size"])
        flat[dests[:used]] = torch.stack((k, v), dim=2)
        if case["kind"] == "prefill":
            o = [_attend(q[a:b], k[a:b], v[a:b], _causal(b - a)) for a, b in spans]
        else:
            o = []
            for s in range(used):
                n = int(pos[s]) + 1
                kv = cache[info.page_indices[s, :-(-n // PAGE)].cuda().long()].view(-1, m["kv"], 2, m["size"])[:n]
                o.append(_attend(q[s:s + 1], kv[:, :, 0], kv[:, :, 1], torch.ones(1, n, dtype=torch.bool, device="cuda")))
        x = x + torch.cat(o).reshape(used, -1) @ w[p + "self_attn.o_proj.weight"].t()
        x = x + _mlp(_rms(x, w[p + "post_attention_layernorm.weight"], 1e-5), w, p + "mlp.")
        pages.append(cache)
    x = _rms(x, w["transformer.norm.weight"], 1e-5)
    if case["kind"] == "prefill":
        return dict(logits=x[torch.from_numpy(rows).cuda()] @ w["lm_head.weight"].t(), pages=pages)
    logits = x @ w["lm_head.weight"].t()
    return dict(logits=logits, logprobs=torch.log_softmax(logits, dim=-1).amax(-1), pages=pages)


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    with torch.no_grad():
        return _exact_serve(case, seed)
