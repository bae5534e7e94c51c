"""The work that programs have this framework do, at sizes from the smallest call to the largest: requests served by the three kinds
of decoder (GPT-2 in f32, the Ministral shape with 4- and 8-bit weights, a layered hybrid of attention, delta rule and experts in bf16),
a decoder driven one program call per token, and the paged attention that a host engine calls by itself.

A case is a dict of plain values. `prepare` loads the model and makes the prompts, `run` serves them once through the public entry
points, `exact` computes the same outputs in 64 bits with torch alone. A model's weights depend on its configuration only, as a
checkpoint's would; prompts, the ids that a step is given and caches come from the seed."""
from __future__ import annotations

import math
import zlib
from types import SimpleNamespace

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from gptrs_b200 import backend, model as gm, ops, ptir  # noqa: E402

D = torch.float64
# width -> query heads, kv heads, feed-forward size (Ministral shape); heads are 128 wide
MINISTRAL = {1024: (8, 2, 3072), 2048: (16, 4, 6144), 3072: (32, 8, 9216)}
# width -> attention (heads, kv heads, chunk), delta rule (heads, rank), experts (number, top, groups, kept groups, size); heads are 128 wide
HYBRID = {1024: ((8, 2, 1024), (8, 64), (16, 4, 4, 2, 768)), 2048: ((16, 4, 2048), (16, 128), (32, 6, 4, 2, 1024))}
GPT = dict(layers=12, width=768, heads=12, ff=3072, vocab=50257, context=1024)


def listed():
    return [
        # One user of the f32 model: a prompt of 32 ids, 64 tokens one by one (host ids in, sampled ids out, every step).
        dict(name="gpt2-chat", kind="gpt", batch=1, prompt=32, new=64),
        # The same model scoring a long prompt: nearly the whole context at once.
        dict(name="gpt2-prompt", kind="gpt", batch=1, prompt=937, new=0),
        # A handful of sequences of unequal lengths side by side.
        dict(name="gpt2-batch", kind="gpt", batch=6, prompt=60, new=24),
        # The f32 model driven from outside, every token one call of a prepared program, K/V handles in and out.
        dict(name="gpt2-program", kind="program", capacity=128, start=40, new=16),
        # One user of the 26-layer model with 4-bit weights: a question of a few hundred ids and the start of the answer.
        dict(name="w4-chat", kind="ministral", bits=4, width=3072, layers=26, vocab=131072, batch=1, prompt=200, new=32),
        # A server's full batch on the same model: 64 ragged prompts, then every sequence advances together.
        dict(name="w4-serve", kind="ministral", bits=4, width=3072, layers=26, vocab=131072, batch=64, prompt=128, new=32),
        # Long prompts on a few layers of it: reading documents.
        dict(name="w4-prompts", kind="ministral", bits=4, width=3072, layers=4, vocab=32768, batch=4, prompt=2048, new=0),
        # 8-bit weights, a small batch of a smaller model.
        dict(name="w8-batch", kind="ministral", bits=8, width=2048, layers=4, vocab=32768, batch=7, prompt=150, new=32),
        # The hybrid reading prompts.
        dict(name="hybrid-prompts", kind="hybrid", width=2048, layers=4, vocab=32768, batch=4, prompt=2000, new=0),
        # The hybrid generating for a batch.
        dict(name="hybrid-serve", kind="hybrid", width=2048, layers=4, vocab=32768, batch=48, prompt=40, new=32),
        # Decode attention over a paged cache, called by a host engine: 64 sequences with 512 to 8192 cached tokens.
        dict(name="attention-ragged", kind="attention", batch=64, low=512, high=8192),
        # The same for one sequence in the middle of a chat.
        dict(name="attention-one", kind="attention", batch=1, low=1500, high=1500),
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["gpt", "program", "ministral", "ministral", "hybrid", "attention"])
    if kind == "attention":
        low, high = sorted((_log_uniform(rng, 100, 8192), _log_uniform(rng, 100, 8192)))
        return dict(kind=kind, batch=_log_uniform(rng, 1, 64), low=low, high=high)
    if kind == "program":
        capacity = rng.choice([64, 128, 256])
        new = rng.randint(4, 24)
        return dict(kind=kind, capacity=capacity, start=rng.randint(1, capacity - new), new=new)
    if kind == "gpt":
        batch = _log_uniform(rng, 1, 8)
        if rng.random() < 0.4:
            return dict(kind=kind, batch=batch, prompt=_log_uniform(rng, 32, 937 // batch), new=0)
        return dict(kind=kind, batch=batch, prompt=_log_uniform(rng, 2, 900 // batch), new=rng.randint(4, 48))
    width = rng.choice(list(MINISTRAL if kind == "ministral" else HYBRID))
    sizes = dict(kind=kind, width=width, layers=4 if kind == "hybrid" else rng.choice([2, 4, 6]), vocab=32768)
    if kind == "ministral":
        sizes["bits"] = rng.choice([4, 4, 8])
    if rng.random() < 0.5:   # prompts
        batch = _log_uniform(rng, 1, 8)
        return dict(sizes, batch=batch, prompt=_log_uniform(rng, 100, 8192 // batch if batch > 1 else 4000), new=0)
    batch = _log_uniform(rng, 1, 64)
    return dict(sizes, batch=batch, prompt=_log_uniform(rng, 8, 8192 // max(batch, 16)), new=rng.randint(8, 32))


# ---- inputs ------------------------------------------------------------------------------------------------------------------
def _generator(*key):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(repr(key).encode()))


def _lengths(case, seed):
    """Prompt lengths of a batch: the first has `prompt` ids, the others 40 to 100 % of that."""
    rng = np.random.default_rng([seed, 1])
    n = case["prompt"]
    return [n] + [int(v) for v in rng.integers(max(1, n * 2 // 5), n + 1, case["batch"] - 1)]


def _tokens(case, seed):
    """Per sequence its prompt, and the ids that the steps behind it are given: [batch][new + 1]."""
    rng = np.random.default_rng([seed, 2])
    vocab = case.get("vocab", GPT["vocab"])
    prompts = [rng.integers(0, vocab, n).astype(np.int32) for n in _lengths(case, seed)]
    return prompts, rng.integers(0, vocab, (case["batch"], case["new"] + 1)).astype(np.int32)


def _rows(case):
    """Most rows of a forward pass: as many as the prompts have, up to 8192."""
    return max(64, min(8192, case["batch"] * case["prompt"]))


def _config(case):
    context = (case["prompt"] + case["new"] + 16 + 15) // 16 * 16
    if case["kind"] == "gpt":
        return gm.ModelConfig(gm.KIND_GPT, GPT["layers"], GPT["width"], GPT["heads"], GPT["heads"], 64, GPT["ff"], GPT["vocab"], GPT["context"], 1e-5,
                              max_seqs=case["batch"], max_tokens=min(_rows(case), GPT["context"]), max_logit_rows=case["batch"], use_pdl=1)
    pages = dict(max_seqs=case["batch"], max_tokens=_rows(case), max_logit_rows=case["batch"], kv_pages=case["batch"] * (context // 16) + 8,
                 max_pages_per_seq=context // 16, use_pdl=1)
    if case["kind"] == "ministral":
        heads, kv, ff = MINISTRAL[case["width"]]
        return gm.ModelConfig(gm.KIND_MINISTRAL, case["layers"], case["width"], heads, kv, 128, ff, case["vocab"], context, 1e-5, 1e6, 128,
                              weight_mode=gm.MODE_W4A16 if case["bits"] == 4 else gm.MODE_W8A16, **pages)
    (h, g, chunk), (dh, rank), (experts, top, groups, keep, ff) = HYBRID[case["width"]]
    moe = dict(mlp=gm.MLP_EXPERTS, d_ff=ff, experts=experts, top=top, groups=groups, keep=keep)
    att = gm.LayerConfig(heads=h, kv_heads=g, dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0, mask=gm.MASK_CHUNK, mask_size=chunk,
                         distance_bias=gm.DISTANCE_LOG, proj_bias=1, mixer=gm.MIXER_GROUPED_ATTENTION, **moe)
    delta = gm.LayerConfig(heads=dh, kv_heads=dh, dim=128, vdim=128, taps=4, decay_rank=rank, gate_rank=rank, mixer=gm.MIXER_CHANNEL_DELTA, **moe)
    return gm.ModelConfig.layered([att, delta] * (case["layers"] // 2), case["width"], case["vocab"], context, 1e-6, block=gm.BLOCK_SANDWICH,
                                  learned_positions=context, weight_mode=gm.MODE_BF16, **pages)


def _model_key(case):
    return tuple((k, case[k]) for k in ("kind", "bits", "width", "layers", "vocab") if k in case)


def _normal(shape, std, key, mean=0.0):
    return torch.empty(shape, device="cuda").normal_(mean, std, generator=_generator(*key))


def _weights(key, shapes):
    """(name, f32 tensor) one after another: what a checkpoint of this model holds. The ids that follow each other are likely ones, as in
    a trained model: the head's row t + 1 points along the embedding of t."""
    kind = dict(key)["kind"]
    for name, shape in shapes.items():
        last, k = name.rsplit(".", 1)[-1], (key, name)
        if kind in ("gpt", "program"):
            t = torch.ones(shape, device="cuda") if last == "gamma" else _normal(shape, 0.02, k)
        elif kind == "ministral":
            if last == "gamma":
                t = 1 + _normal(shape, 0.1, k)
            elif name == "tok_embeddings.weight":
                t = _normal(shape, 2.0, k)
            elif name == "lm_head":
                t = (_normal(shape[::-1], 2.0, (key, "tok_embeddings.weight")).roll(1, 0).t() * 0.01).contiguous()
            else:
                t = _normal(shape, 0.02, k)
        else:
            t = _hybrid_weight(key, name, last, shape).bfloat16().float()
        yield name, t


def _hybrid_weight(key, name, last, shape):
    """Norm gains around 1, projections of unit output scale, decays spread between quick and slow. A token keeps a code in the last
    channels (one per expert) that no layer adds to and that the routers read: as in a trained model, few choices of experts are close."""
    experts = HYBRID[dict(key)["width"]][2][0]
    g = _generator(key, name)
    normal = torch.empty(shape, device="cuda").normal_(generator=g)
    uniform = torch.empty(shape, device="cuda").uniform_(generator=g)
    if "norm" in last:
        t = 1 + 0.2 * normal
        if last in ("norm1b", "norm2b"):
            t[-experts:] = 0
        elif last == "norm2":
            t[-experts:] = 1
        return t
    if last == "router":
        t = torch.zeros(shape, device="cuda")
        t[:, -experts:] = 6 * torch.eye(experts, device="cuda")
        return t
    if name == "embed":
        order = torch.rand((shape[0], experts), device="cuda", generator=g).argsort(1)
        normal[:, -experts:] = 2.0 * (order - (experts - 1) / 2) / experts
        return normal
    if name == "pos":
        normal[:, -experts:] = 0
        return 0.5 * normal
    if name == "head":
        return _hybrid_weight(key, "embed", "embed", shape).roll(1, 0) * shape[-1] ** -0.5
    if last == "conv":
        t = 0.5 * normal
        t[:, -1] += 0.7
        return t
    if last == "r1":
        return 0.2 + 0.8 * uniform
    if last == "r2":
        return 0.05 + 1.45 * uniform
    if last == "A_log":
        return torch.log(0.3 + 2.7 * uniform)
    if last == "dt_bias":
        return -6.0 * uniform
    if last == "b" and len(shape) == 1:
        return 0.3 * normal
    return normal * shape[-1] ** -0.5


def prepare(case, seed):
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    if case["kind"] == "program":
        return _prepare_program(case, seed)
    cfg = _config(case)
    m = gm.LoadedModel(cfg, namespace=zlib.crc32(repr(_model_key(case)).encode()))
    for name, w in _weights(_model_key(case), cfg.param_shapes()):
        m.load_param(name, w)
    m.finalize()
    prompts, given = _tokens(case, seed)
    return SimpleNamespace(kind=case["kind"], model=m, prompts=prompts, given=given, new=case["new"], slots=list(range(case["batch"])))


# ---- one pass -----------------------------------------------------------------------------------------------------------------
def run(s):
    if s.kind == "attention":
        out, _ = ops.paged_attention_decode(s.q, s.pool, s.table, s.slot, s.lengths, 32, 8, s.longest)
        return out
    if s.kind == "program":
        return _run_program(s)
    m = s.model
    for slot in s.slots:
        m.reset_sequence(slot)
    ids = []
    if len(s.slots) == 1:
        _, first = m.prefill(0, s.prompts[0])
        ids.append([first])
    else:
        ids.append(m.prefill_many(s.slots, s.prompts))
    if s.new:
        steps = gm.Generator(m, s.given[:, 0])
        for j in range(s.new):
            ids.append(steps.step(s.given[:, j]))
    # the last step is sampled by the program itself, from the logits
    at = [m.sequence_length(slot) for slot in s.slots]
    logits, _ = m.forward_with_decode_cache(s.given[:, s.new], s.slots, at, s.slots)
    return {"ids": np.array(ids, dtype=np.int32), "logits": logits}


# ---- the model driven through programs ------------------------------------------------------------------------------------------
def _gpt_shape():
    return SimpleNamespace(kind="gpt", n_layers=GPT["layers"], d_model=GPT["width"], n_q=GPT["heads"], n_kv=GPT["heads"], hd=64, d_mlp=GPT["ff"],
                           vocab=GPT["vocab"], ctx=GPT["context"], eps=1e-5, rot=0)


def _program_caches(case, seed):
    """Keys and values of the tokens before `start`, [layer][2][heads][capacity][64]."""
    c = _normal((GPT["layers"], 2, GPT["heads"], case["capacity"], 64), 0.5, (seed, "caches"))
    c[:, :, :, case["start"]:] = 0
    return c


def _prepare_program(case, seed):
    be = backend.CudaBackend()
    builder, names = ptir.decode_step_program(_gpt_shape(), case["capacity"])
    shapes = {n: tuple(p.dims) for n, p in zip(names, builder.params) if not n.startswith("@")}
    weights = {n: be.materialize(w.cpu().numpy()) for n, w in _weights((("kind", "program"),), shapes)}
    caches = [[be.materialize(t) for t in layer] for layer in _program_caches(case, seed).cpu().numpy()]
    given = np.random.default_rng([seed, 3]).integers(0, GPT["vocab"], case["new"]).astype(np.int32)
    return SimpleNamespace(kind="program", backend=be, program=be.prepare(builder.to_json()), names=names, weights=weights, caches=caches, given=given,
                           start=case["start"])


def _run_program(s):
    be, caches, ids = s.backend, s.caches, []
    for j, token in enumerate(s.given):
        pos = s.start + j
        small = {"@tokens": np.array([token], np.int32), "@positions": np.array([pos], np.int32),
                 "@update_starts": np.array([0, pos, 0], np.int32), "@query_start": np.array([pos], np.int32)}
        inputs = []
        for n in s.names:
            if n in small:
                inputs.append(be.materialize(small[n]))
            elif n.startswith("@"):
                inputs.append(caches[int(n[2:])][n[1] == "v"])
            else:
                inputs.append(s.weights[n])
        out = s.program.run(inputs)
        caches = [(out[1 + 2 * l], out[2 + 2 * l]) for l in range(GPT["layers"])]
        ids.append(be.sample_decode_token(out[0], 0.0))
    return {"ids": np.array(ids, dtype=np.int32), "logits": be.to_literal(out[0])}


# ---- paged attention by itself -----------------------------------------------------------------------------------------------
def _attention_inputs(case, seed):
    """Lengths, queries [batch][32][128], and a function that gives the keys and values [length][2][8][128] of a sequence."""
    rng = np.random.default_rng([seed, 4])
    lengths = [int(v) for v in rng.integers(case["low"], case["high"] + 1, case["batch"])]
    q = _normal((case["batch"], 32, 128), 1.0, (seed, "q")).bfloat16()
    return lengths, q, lambda b: _normal((lengths[b], 2, 8, 128), 1.0, (seed, "kv", b)).bfloat16()


def _prepare_attention(case, seed):
    lengths, q, kv = _attention_inputs(case, seed)
    per = (max(lengths) + 15) // 16
    pool = ops.new_kv_pool(case["batch"] * per, 8, q.device)
    table = torch.randperm(case["batch"] * per, device="cuda", generator=_generator(seed, "pages")).int().view(case["batch"], per)
    cos, sin = torch.ones((per * 16, 64), device="cuda"), torch.zeros((per * 16, 64), device="cuda")
    for b, n in enumerate(lengths):   # fills the cache as an engine would (keys that are rotated already)
        rows = torch.cat([torch.zeros((n, 32 * 128), dtype=torch.bfloat16, device="cuda"), kv(b).view(n, -1)], 1).contiguous()
        ops.rope_kv_append(rows, torch.arange(n, dtype=torch.int32, device="cuda"), torch.full((n,), b, dtype=torch.int32, device="cuda"), table, cos, sin, 128,
                           pool, 32, 8)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    return SimpleNamespace(kind="attention", q=q, pool=pool, table=table, slot=torch.arange(case["batch"], dtype=torch.int32, device="cuda"), lengths=i32(lengths),
                           longest=max(lengths))


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------
def _quantised(w, bits):
    """f32 [in][out] -> the values that symmetric weights of 4 bits (scales in f16 per 128 inputs) or 8 bits (per output) stand for."""
    n_in, n_out = w.shape
    g = w.view(n_in // 128, 128, n_out) if bits == 4 else w.view(1, n_in, n_out)
    scale = (g.abs().amax(1, keepdim=True) / (7.0 if bits == 4 else 127.0)).half().float()
    low = -8 if bits == 4 else -127
    q = torch.where(scale > 0, (g / scale).round(), 0.0).clamp(low, 7 if bits == 4 else 127)
    return (q * scale).view(n_in, n_out)


def _layer_norm(x, g, b):
    return (x - x.mean(-1, keepdim=True)) / (x.var(-1, unbiased=False, keepdim=True) + 1e-5).sqrt() * g + b


def _rms(x, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def _attend(q, k, v, scale, mask, bend=None):
    """q [T][H][d], k and v [S][G][d], mask [T][S] -> [T][H][d], a kv head at a time; `bend` changes the scores of a range of heads."""
    group, out = q.shape[1] // k.shape[1], torch.empty_like(q)
    for h in range(k.shape[1]):
        own = slice(h * group, (h + 1) * group)
        s = torch.einsum("tgd,sd->gts", q[:, own], k[:, h]) * scale
        if bend is not None:
            s = bend(s, own)
        out[:, own] = torch.einsum("gts,sd->tgd", s.masked_fill(~mask, -math.inf).softmax(-1), v[:, h])
    return out


def _causal(n):
    return torch.ones((n, n), dtype=torch.bool, device="cuda").tril()


def _exact_plain(case, spans, tokens, positions, want, caches=None, kind=None):
    """Logits [len(want)][vocab] of the GPT and Ministral shapes for packed sequences (`spans` of rows); `caches`: keys and values of one
    sequence's earlier tokens."""
    kind = kind or case["kind"]
    gpt = kind != "ministral"
    cfg = _config(dict(case, kind="gpt" if gpt else kind, batch=1, prompt=case.get("prompt", 1)))
    key = (("kind", "program"),) if kind == "program" else _model_key(case)
    shapes = cfg.param_shapes()

    def w(name):
        _, t = next(iter(_weights(key, {name: shapes[name]})))
        if not gpt and t.dim() == 2 and name != "tok_embeddings.weight":
            t = _quantised(t, case["bits"])
        return t.to(D)

    x = w("tok_embeddings.weight")[tokens]
    heads, kv, hd = cfg.n_q_heads, cfg.n_kv_heads, cfg.head_dim
    if gpt:
        x = x + w("pos_embeddings")[positions]
    else:
        angle = positions[:, None].to(D) * (1e6 ** (-torch.arange(0, hd, 2, device="cuda", dtype=D) / hd))
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    for l in range(cfg.n_layers):
        p = f"blocks.{l}."
        h = _layer_norm(x, w(p + "ln_1.gamma"), w(p + "ln_1.beta")) if gpt else _rms(x, 1e-5) * w(p + "norm_1.gamma")
        qkv = h @ w(p + "attention.w_qkv") + (w(p + "attention.b_qkv") if gpt else 0)
        q, k, v = (t.reshape(len(x), -1, hd) for t in qkv.split([heads * hd, kv * hd, kv * hd], 1))
        if not gpt:
            q, k = (torch.cat([t[..., :hd // 2] * cos - t[..., hd // 2:] * sin, t[..., hd // 2:] * cos + t[..., :hd // 2] * sin], -1) for t in (q, k))
        o = torch.empty_like(q)
        for a, b in spans:
            mask = _causal(b - a)
            ks, vs = k[a:b], v[a:b]
            if caches is not None:
                ks, vs = (torch.cat([c.transpose(0, 1), t]) for c, t in zip(caches[l], (ks, vs)))
                mask = torch.cat([mask.new_ones((b - a, len(ks) - (b - a))), mask], 1)
            o[a:b] = _attend(q[a:b], ks, vs, hd ** -0.5, mask)
        x = x + o.flatten(1) @ w(p + "attention.w_out") + (w(p + "attention.b_out") if gpt else 0)
        if gpt:
            h = _layer_norm(x, w(p + "ln_2.gamma"), w(p + "ln_2.beta")) @ w(p + "feed_forward.w_in") + w(p + "feed_forward.b_in")
            x = x + torch.nn.functional.gelu(h) @ w(p + "feed_forward.w_out") + w(p + "feed_forward.b_out")
        else:
            h = _rms(x, 1e-5) * w(p + "norm_2.gamma")
            x = x + (torch.nn.functional.silu(h @ w(p + "feed_forward.w_gate")) * (h @ w(p + "feed_forward.w_up"))) @ w(p + "feed_forward.w_down")
    x = x[want]
    x = _layer_norm(x, w("final_ln.gamma"), w("final_ln.beta")) if gpt else _rms(x, 1e-5) * w("final_norm.gamma")
    return x @ w("lm_head")


def _delta(h, w, heads, spans):
    """The gated delta rule with a decay per key channel over packed sequences: one step of the recurrence at a time, all sequences together."""
    def conv(x, taps):
        out = torch.zeros_like(x)
        for a, b in spans:
            for j in range(taps.shape[1]):
                back = taps.shape[1] - 1 - j
                out[a + back:b] += taps[:, j] * x[a:b - back] if b - a > back else 0
        return torch.nn.functional.silu(out)

    def unit(x):
        return x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()

    q, k, v = (conv(h @ w[n].T, w[n + ".conv"]).view(len(h), heads, 128) for n in "qkv")
    q, k, beta = unit(q) * 128 ** -0.5, unit(k), torch.sigmoid(h @ w["b"].T)
    a = (h @ w["a1"].T @ w["a2"].T).view(len(h), heads, 128)
    decay = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a + w["dt_bias"].view(heads, 128)))
    longest = max(b - a for a, b in spans)
    state, o = torch.zeros((len(spans), heads, 128, 128), dtype=D, device="cuda"), torch.empty_like(v)
    first = torch.tensor([a for a, _ in spans], device="cuda")
    length = torch.tensor([b - a for a, b in spans], device="cuda")
    order = length.argsort(descending=True)
    first, length = first[order], length[order].tolist()
    for t in range(longest):
        n = sum(1 for m in length if m > t)
        at = first[:n] + t
        s = state[:n]
        s *= decay[at][..., None]
        u = beta[at][..., None] * (v[at] - torch.einsum("nhdv,nhd->nhv", s, k[at]))
        s += k[at][..., None] * u[..., None, :]
        o[at] = torch.einsum("nhdv,nhd->nhv", s, q[at])
    gate = torch.sigmoid(h @ w["g1"].T @ w["g2"].T).view(len(h), heads, 128)
    return (_rms(o, 1e-6) * w["norm"] * gate).flatten(1) @ w["o"].T


def _mixture(h, w, experts, top, groups, keep):
    s = (h @ w["router"].T).softmax(-1)
    best = s.view(len(h), groups, -1).amax(-1).topk(keep, -1).indices
    allowed = torch.zeros((len(h), groups), dtype=torch.bool, device="cuda").scatter_(1, best, True).repeat_interleave(experts // groups, 1)
    chosen = s.masked_fill(~allowed, -1).topk(top, -1).indices
    out = torch.zeros_like(h)
    for e in range(experts):
        rows = (chosen == e).any(1).nonzero()[:, 0]
        if len(rows):
            x = h[rows]
            y = (torch.nn.functional.silu(x @ w[f"e{e}.gate"].T) * (x @ w[f"e{e}.up"].T)) @ w[f"e{e}.down"].T
            out[rows] += s[rows, e, None] * y
    return out


def _exact_hybrid(case, spans, tokens, positions, want):
    cfg, key = _config(case), _model_key(case)
    w = {n: t.to(D) for n, t in _weights(key, cfg.param_shapes())}
    (heads, kv, chunk), (delta_heads, _), (experts, top, groups, keep, _) = HYBRID[case["width"]]
    x = w["embed"][tokens] + w["pos"][positions]
    for l in range(case["layers"]):
        part = lambda s: {n[len(f"l{l}.{s}."):]: t for n, t in w.items() if n.startswith(f"l{l}.{s}.")}  # noqa: E731
        h, mix = _rms(x, 1e-6) * w[f"l{l}.norm1"], part("mix")
        if l % 2:
            y = _delta(h, mix, delta_heads, spans)
        else:
            q, k, v = ((h @ mix[n].T + mix[n + ".b"]).view(len(h), -1, 128) for n in "qkv")
            o = torch.empty_like(q)
            for a, b in spans:
                at = torch.arange(b - a, device="cuda")
                far = (at[:, None] - at).clamp(min=0).to(D)

                def bend(s, own):
                    return 30.0 * torch.tanh(s / 30.0) - mix["r1"][own, None, None] * torch.log1p(mix["r2"][own, None, None] * far)

                o[a:b] = _attend(q[a:b], k[a:b], v[a:b], 128 ** -0.5, _causal(b - a) & (at[:, None] // chunk == at // chunk), bend)
            y = o.flatten(1) @ mix["o"].T + mix["o.b"]
        x = x + _rms(y, 1e-6) * w[f"l{l}.norm1b"]
        x = x + _rms(_mixture(_rms(x, 1e-6) * w[f"l{l}.norm2"], part("mlp"), experts, top, groups, keep), 1e-6) * w[f"l{l}.norm2b"]
    return (_rms(x[want], 1e-6) * w["final.norm"]) @ w["head"].T


def exact(case, seed):
    if case["kind"] == "attention":
        lengths, q, kv = _attention_inputs(case, seed)
        out = []
        for b, n in enumerate(lengths):
            k, v = kv(b).to(D).unbind(1)
            out.append(_attend(q[b:b + 1].to(D), k, v, 128 ** -0.5, torch.ones((1, n), dtype=torch.bool, device="cuda"))[0].flatten())
        return torch.stack(out)
    if case["kind"] == "program":
        given = torch.from_numpy(np.random.default_rng([seed, 3]).integers(0, GPT["vocab"], case["new"])).cuda()
        caches = _program_caches(case, seed)[:, :, :, :case["start"]].to(D)
        at = case["start"] + torch.arange(case["new"], device="cuda")
        return {"ids": None, "logits": _exact_plain(case, [(0, case["new"])], given, at, [case["new"] - 1], caches)}
    prompts, given = _tokens(case, seed)
    rows = [np.concatenate([p, g]) for p, g in zip(prompts, given)]
    ends = np.cumsum([len(r) for r in rows])
    spans = [(int(e) - len(r), int(e)) for e, r in zip(ends, rows)]
    tokens = torch.from_numpy(np.concatenate(rows)).long().cuda()
    positions = torch.cat([torch.arange(b - a, device="cuda") for a, b in spans])
    want = torch.tensor([b - 1 for _, b in spans], device="cuda")
    return {"ids": None, "logits": (_exact_hybrid if case["kind"] == "hybrid" else _exact_plain)(case, spans, tokens, positions, want)}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def work(case):
    """Every step reads its weights and its cache once; multiplications with weights and in attention count."""
    kind = case["kind"]
    if kind == "attention":
        n = case["batch"] * (case["low"] + case["high"]) / 2
        return {"bytes": n * 4096 + case["batch"] * 2 * 32 * 128 * 2, "flops": n * 4 * 32 * 128}
    b, new = case.get("batch", 1), case["new"]
    mean = case["start"] if kind == "program" else case["prompt"] * (1 + 0.7 * (b - 1)) / b   # cached tokens of a sequence when the steps begin
    steps = new + (kind != "program")
    passes = 0 if kind == "program" else math.ceil(b * mean / _rows(case))
    rows = b * (steps + (mean if passes else 0))
    seen = b * steps * (mean + steps / 2)                       # cached tokens that the decode steps read
    pairs = seen + (b * mean * mean / 2 if passes else 0)       # scores per head
    active = None
    if kind in ("gpt", "program"):
        layers, d, size = GPT["layers"], GPT["width"], 4.0
        per_layer, head, token = 4 * d * d + 2 * d * GPT["ff"], d * GPT["vocab"], 2 * d * 4
        width = d
    elif kind == "ministral":
        heads, kv, ff = MINISTRAL[case["width"]]
        layers, d, size = case["layers"], case["width"], 0.5 + 2 / 128 if case["bits"] == 4 else 1.0
        per_layer, head, token = d * 128 * (2 * heads + 2 * kv) + 3 * d * ff, d * case["vocab"], kv * 2 * 128 * 2
        width = heads * 128
    else:
        (heads, kv, _), (dh, rank), (experts, top, _, _, ff) = HYBRID[case["width"]]
        layers, d, size = case["layers"], case["width"], 2.0
        mixers = (d * 128 * (2 * heads + 2 * kv) + d * 128 * 4 * dh + 2 * rank * (d + 128 * dh)) / 2
        per_layer, head, token = mixers + experts * 3 * d * ff, d * case["vocab"], kv * 2 * 128 * 2 / 2
        active = mixers + top * 3 * d * ff
        width = heads * 128 / 2
    weights = layers * per_layer
    state = 2 * b * (steps + passes) * (layers / 2) * HYBRID[case["width"]][1][0] * 128 * 128 * 4 if kind == "hybrid" else 0
    nbytes = (steps + passes) * (weights + head) * size + layers * token * (seen + rows) + state + b * case.get("vocab", GPT["vocab"]) * 4
    flops = 2 * rows * layers * (active or per_layer) + 2 * b * (steps + (1 if passes else 0)) * head + 4 * pairs * layers * width
    if kind == "hybrid":
        flops += rows * (layers / 2) * HYBRID[case["width"]][1][0] * 8 * 128 * 128
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Against 64 bits the logits are off by 4e-7 in f32, by 4e-3 to 1.5e-2 in bf16 (more with more layers); another order of the sums, or
    another place of a rounding to bf16, moves them by as much."""
    if case["kind"] in ("gpt", "program"):
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    if case["kind"] == "attention":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 0.03, "max": 0.3, "differ": 0.005}
