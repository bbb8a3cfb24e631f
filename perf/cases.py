"""The work this framework is measured on: forward passes of its models as a serving program runs them, and paged decode attention by itself.

A case is one call pattern of one model:

  decode    every sequence feeds one token, its context is in the paged cache (``CudaModel.forward``)
  prompts   whole prompts, all of them in one forward
  mixed     one step of continuous batching: decoding sequences and portions of prompts whose beginning is in the cache
  generate  short prompts and then token after token; the way models with state slots decode, since a state cannot be fed the same token twice
  attention paged decode attention through the C ABI, on buffers that the caller owns (``orion_cuda_paged_decode_attention_noalloc``)

Lengths are spread evenly between ``shortest`` and ``longest``. The models are the shapes of ``bench.py`` with their first ``layers`` layers and
a vocabulary of 32768, all weights random from the seed.
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch
import torch.nn.functional as F

orion = importlib.import_module("orionserve-rs_b200")

BLOCK, VOCAB = 16, 32768
PATTERNS = 64  # kinds of tokens that the routers of the mixtures tell apart
MOST_EXACT_FLOPS = 3.5e14  # about 15 s in 64 bits

# The Llama and Qwen2 layouts: configuration 1 of the benchmark (f32), the Llama-3-8B shape, the Qwen2-7B shape.
DENSE = {
    "tiny": dict(hidden_size=256, num_attention_heads=4, num_kv_heads=2, head_dim=64, ffn_dim=688, rope_theta=10000.0, rms_norm_eps=1e-5),
    "llama": dict(hidden_size=4096, num_attention_heads=32, num_kv_heads=8, head_dim=128, ffn_dim=14336, rope_theta=500000.0, rms_norm_eps=1e-5),
    "qwen2": dict(hidden_size=3584, num_attention_heads=28, num_kv_heads=4, head_dim=128, ffn_dim=18944, rope_theta=1000000.0, rms_norm_eps=1e-6,
                  has_qkv_bias=True),
}
# The layer-list designs, at the two sizes that the benchmark runs them at.
LAYERED = {
    "metapel": {2048: dict(ffn=8192, heads=16, rank=512, window=1024), 4096: dict(ffn=16384, heads=32, rank=512, window=1024)},
    "zulozen": {2048: dict(ffn=8192, heads=16, expert=1408, shared=2816), 4096: dict(ffn=16384, heads=32, expert=2816, shared=5632)},
    "belizen": {2048: dict(ffn=5504, heads=16, expert=1408, shared=2816), 4096: dict(ffn=11008, heads=32, expert=2816, shared=5632)},
    "vusenex": {2048: dict(heads=16, rank=512, expert=2112, shared=4224), 4096: dict(heads=32, rank=512, expert=4224, shared=8448)},
}
EXPERTS, TOP, IDENTITY, GROUPS, KEEP = 16, 2, 2, 4, 2
STATEFUL = ("metapel", "belizen")


def listed():
    return [
        # configuration 1 in the f32 build: eight short chats, one token each; the smallest step there is
        dict(name="tiny f32 decode 8", design="tiny", width=256, layers=2, kind="decode", sequences=8, shortest=32, longest=160),
        # one user in a chat
        dict(name="llama decode 1", design="llama", width=4096, layers=8, kind="decode", sequences=1, shortest=1024, longest=1024),
        # the headline batch
        dict(name="llama decode 64", design="llama", width=4096, layers=8, kind="decode", sequences=64, shortest=1024, longest=1024),
        # a full server: many requests behind one system prompt, of unequal length by now
        dict(name="qwen2 decode 128", design="qwen2", width=3584, layers=8, kind="decode", sequences=128, shortest=1089, longest=1407),
        # a step of continuous batching with a budget of 512 tokens
        dict(name="llama mixed 512", design="llama", width=4096, layers=8, kind="mixed", sequences=96, shortest=131, longest=2047, portions=1, rows=416,
             start=512),
        # prompts without a cache, the largest batch
        dict(name="llama prompts 4x2048", design="llama", width=4096, layers=8, kind="prompts", sequences=4, shortest=2048, longest=2048),
        # decode attention by itself, ragged contexts
        dict(name="attention 64", design="attention", kind="attention", sequences=64, shortest=512, longest=8192),
        # the same for one user: launch and latency
        dict(name="attention 1", design="attention", kind="attention", sequences=1, shortest=2371, longest=2371),
        # recurrence and latent attention: a short prompt and an answer, 16 users
        dict(name="metapel generate 16", design="metapel", width=2048, layers=8, kind="generate", sequences=16, shortest=97, longest=131, steps=40),
        # mixtures of experts, 16 users
        dict(name="zulozen decode 16", design="zulozen", width=2048, layers=8, kind="decode", sequences=16, shortest=1024, longest=1024),
        # linear attention and windows, prompts of odd lengths
        dict(name="belizen prompts 4", design="belizen", width=2048, layers=8, kind="prompts", sequences=4, shortest=1531, longest=2047),
        # latent attention and keys that are values, one prompt
        dict(name="vusenex prompt 2048", design="vusenex", width=2048, layers=8, kind="prompts", sequences=1, shortest=2048, longest=2048),
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    design = rng.choice(["tiny", "llama", "llama", "llama", "qwen2", "qwen2", "attention", "metapel", "zulozen", "belizen", "vusenex"])
    if design == "attention":
        n, longest = _log(rng, 1, 256), _log(rng, 512, 8192)
        return dict(design=design, kind="attention", sequences=n, shortest=rng.randint(min(512, longest), longest), longest=longest)
    layers = 8
    if design in LAYERED:
        width = rng.choice([2048, 2048, 4096])
        layers = 8 if width == 2048 else 4
    else:
        width = DENSE[design]["hidden_size"]
        layers = 2 if design == "tiny" else 8
    case = dict(design=design, width=width, layers=layers, kind=rng.choice(["decode", "decode", "prompts", "mixed"]))
    if design in STATEFUL:
        case["kind"] = rng.choice(["generate", "prompts"])
    if design == "tiny":
        case.update(kind="decode", sequences=_log(rng, 1, 16), longest=rng.randint(64, 192))
        case["shortest"] = rng.randint(32, case["longest"])
    elif case["kind"] == "decode":
        case["sequences"] = _log(rng, 1, 192)
        case["longest"] = _log(rng, 64, min(4096, 131072 // case["sequences"]))
        case["shortest"] = rng.randint(max(1, case["longest"] // 2), case["longest"])
    elif case["kind"] == "prompts":
        case["longest"] = _log(rng, 64, 2048)
        case["sequences"] = _log(rng, 1, 8192 // case["longest"])
        case["shortest"] = rng.randint(max(1, case["longest"] // 2), case["longest"])
    elif case["kind"] == "mixed":
        case.update(sequences=_log(rng, 1, 128), longest=rng.randint(256, 2048), shortest=rng.randint(32, 255), portions=rng.randint(1, 3),
                    start=16 * rng.randint(0, 64))
        case["rows"] = max(16, (512 - case["sequences"]) // case["portions"] - rng.randint(0, 20))
    else:
        case.update(sequences=_log(rng, 1, 64), longest=_log(rng, 32, 128), steps=rng.randint(8, 48))
        case["shortest"] = rng.randint(max(1, case["longest"] // 2), case["longest"])
    return case


# ---- sizes -------------------------------------------------------------------------------------------------------------------------------

def _spread(low, high, n):
    """n lengths over low .. high, in an order that is neither sorted nor random."""
    return [low + int(round((high - low) * ((i * 0.6180339887498949 + 0.5) % 1.0))) for i in range(n)] if n > 1 else [high]


def _lengths(case):
    """(context, rows fed) of every sequence of the measured forward, in the order of the batch."""
    contexts = _spread(case["shortest"], case["longest"], case["sequences"])
    if case["kind"] in ("prompts", "generate"):
        return [(c, c) for c in contexts]
    out = [(c, 1) for c in contexts]
    if case["kind"] == "mixed":
        out += [(case["start"] + case["rows"], case["rows"])] * case["portions"]
    return out


def _specs(design, width, layers):
    """The layers of a layer-list design as ``bench.py`` sets them up."""
    z = LAYERED[design][width]
    att = dict(heads=z["heads"], dim=128, value_dim=128)
    if design == "metapel":
        gru = orion.LayerSpec("mingru", z["ffn"], width=width)
        lat = orion.LayerSpec("latent_attention", z["ffn"], rot_dim=64, kv_rank=z["rank"], window=z["window"], rope_dims=64, rope_base=10000.0,
                              scale=192 ** -0.5, **att)
        return [lat if i % 2 else gru for i in range(layers)]
    if design == "zulozen":
        att.update(kv_heads=z["heads"] // 4, chunk=2048, rope_dims=64, rope_base=10000.0, scale=128 ** -0.5, qk_norm=True, sinks=True, head_gate=True)
        dense = orion.LayerSpec("attention", z["ffn"], activation="relu2", ffn_bias=True, **att)
        mix = orion.LayerSpec("attention", z["expert"], experts=EXPERTS, experts_per_token=TOP, shared_dim=z["shared"], **att)
        return [mix if i % 2 else dense for i in range(layers)]
    if design == "belizen":
        gla = dict(heads=z["heads"], dim=64, value_dim=128, decay_tau=8.0, decay_rank=16)
        att.update(kv_heads=z["heads"] // 4, window=1024, keep_first=8, rope_dims=64, rope_base=10000.0, yarn=orion.Yarn(2.0, 4096.0, 32.0, 1.0),
                   rope_halves=True, scale=128 ** -0.5, softcap=20.0, qk_norm="per_head", qkv_bias=True, value_gate=True)
        dense = dict(ffn_dim=z["ffn"], activation="geglu_tanh")
        mix = dict(ffn_dim=z["expert"], experts=EXPERTS, experts_per_token=TOP, router="softmax", router_identity=IDENTITY, expert_form="clamped",
                   expert_limit=7.0, shared_dim=z["shared"], shared_limit=7.0)
        return [orion.LayerSpec("attention" if i % 2 else "gla", **(att if i % 2 else gla), **(mix if i % 4 in (1, 2) else dense)) for i in range(layers)]
    att.update(ffn_dim=z["expert"], scale=128 ** -0.5, experts=EXPERTS, experts_per_token=TOP, router="softmax_renorm", router_groups=GROUPS,
               router_keep=KEEP, expert_form="gelu", shared_dim=z["shared"])
    lat = orion.LayerSpec("latent_attention", kv_rank=z["rank"], ungated=True, **att)
    joint = orion.LayerSpec("attention", kv_heads=z["heads"] // 4, qk_norm=True, qkv_bias=True, sinks="zero", keys_as_values=True, distance_bias=True,
                            q_temp=orion.QueryTemperature(0.1, 512.0), **att)
    return [joint if i % 2 else lat for i in range(layers)]


def _metadata(case):
    design, width, layers = case["design"], case["width"], case["layers"]
    if design in DENSE:
        return orion.ModelMetadata(architecture="qwen2" if design == "qwen2" else "llama", name=design, num_layers=layers,
                                   vocab_size=1024 if design == "tiny" else VOCAB, max_position_embeddings=8192, **DENSE[design])
    common = dict(architecture=design.capitalize(), name=design, hidden_size=width, vocab_size=VOCAB, layers=_specs(design, width, layers), norm_eps=1e-6)
    more = {"metapel": dict(conv_taps=4), "zulozen": dict(block="sandwich", untied_lm_head=True, residual_mult=0.5),
            "belizen": dict(block="prenorm", residual_mult=0.5, embed_scale=8.0, logit_softcap=25.0),
            "vusenex": dict(block="gated_postnorm", untied_lm_head=True, scalar_norms=True, max_positions=8192, bigram=orion.Bigram(32749, 37, 101))}
    return orion.LayeredMetadata(**common, **more[design])


def _shapes(case, meta):
    """Names and shapes of the model's tensors, in a fixed order."""
    t = {}
    if case["design"] in DENSE:
        H, D, ff = meta.hidden_size, meta.head_dim, meta.ffn_dim
        q, k = meta.num_attention_heads * D, meta.num_kv_heads * D
        t["model.embed_tokens.weight"], t["model.norm.weight"], t["lm_head.weight"] = (meta.vocab_size, H), (H,), (meta.vocab_size, H)
        for i in range(meta.num_layers):
            p = f"model.layers.{i}."
            t[p + "input_layernorm.weight"] = t[p + "post_attention_layernorm.weight"] = (H,)
            for n, rows in (("q", q), ("k", k), ("v", k)):
                t[f"{p}self_attn.{n}_proj.weight"] = (rows, H)
                if meta.has_qkv_bias:
                    t[f"{p}self_attn.{n}_proj.bias"] = (rows,)
            t[p + "self_attn.o_proj.weight"], t[p + "mlp.gate_proj.weight"], t[p + "mlp.up_proj.weight"] = (H, q), (ff, H), (ff, H)
            t[p + "mlp.down_proj.weight"] = (H, ff)
        return t
    H, design = meta.hidden_size, case["design"]
    gain = () if meta.scalar_norms else (H,)
    t["embed"], t["final.norm"] = (VOCAB, H), gain
    if meta.untied_lm_head:
        t["head"] = (VOCAB, H)
    if design == "vusenex":
        t["bigram"], t["pos"] = (meta.bigram.buckets + 1, H), (meta.max_positions, H)
    for i, s in enumerate(meta.layers):
        p = f"l{i}."
        q, k, v = s.heads * s.dim, s.kv_heads * s.dim, s.kv_heads * s.value_dim
        t[p + "norm1"] = gain
        if design == "metapel":
            t[p + "canon1"] = t[p + "canon2"] = (H, meta.conv_taps)
            t[p + "mlp.up"], t[p + "mlp.down"] = (s.ffn_dim, H), (H, s.ffn_dim)
        if design == "zulozen":
            t[p + "norm1b"] = t[p + "norm2"] = t[p + "norm2b"] = (H,)
        if design == "belizen":
            t[p + "norm2"] = (H,)
        if design == "vusenex":
            t[p + "rg1"], t[p + "rg1.b"], t[p + "norm2"], t[p + "rg2"], t[p + "rg2.b"] = (H, H), (H,), (), (H, H), (H,)
        if s.mixer == "mingru":
            for n in "zxg":
                t[f"{p}mix.{n}"] = (s.width, H)
            t[p + "mix.z.b"], t[p + "mix.x.b"], t[p + "mix.o"] = (s.width,), (s.width,), (H, s.width)
        elif s.mixer == "latent_attention":
            t[p + "mix.q"] = (s.heads * (s.dim + s.rot_dim), H)
            t[p + "mix.dkv"], t[p + "mix.dkv.norm"] = (s.kv_rank + s.rot_dim, H), (s.kv_rank,)
            t[p + "mix.uk"], t[p + "mix.uv"], t[p + "mix.o"] = (q, s.kv_rank), (s.heads * s.value_dim, s.kv_rank), (H, s.heads * s.value_dim)
            if not s.ungated:
                t[p + "mix.g"] = (s.heads * s.value_dim, H)
        elif s.mixer == "gla":
            kk, vv = s.heads * s.dim, s.heads * s.value_dim
            t[p + "mix.q"], t[p + "mix.k"], t[p + "mix.v"], t[p + "mix.g"] = (kk, H), (kk, H), (vv, H), (vv, H)
            t[p + "mix.a1"], t[p + "mix.a2"], t[p + "mix.a2.b"] = (s.decay_rank, H), (kk, s.decay_rank), (kk,)
            t[p + "mix.norm"], t[p + "mix.o"] = (s.value_dim,), (H, vv)
        else:
            t[p + "mix.q"], t[p + "mix.k"], t[p + "mix.o"] = (q, H), (k, H), (H, s.heads * s.value_dim)
            if not s.keys_as_values:
                t[p + "mix.v"] = (v, H)
            if design == "zulozen":
                t[p + "mix.q.norm"], t[p + "mix.k.norm"], t[p + "mix.sink"], t[p + "mix.g"] = (q,), (k,), (s.heads,), (s.heads, H)
            elif design == "belizen":
                t[p + "mix.q.b"], t[p + "mix.k.b"], t[p + "mix.v.b"] = (q,), (k,), (v,)
                t[p + "mix.q.norm"] = t[p + "mix.k.norm"] = (s.dim,)
                t[p + "mix.g"] = (s.heads * s.value_dim, H)
            else:
                t[p + "mix.q.b"], t[p + "mix.k.b"], t[p + "mix.q.norm"], t[p + "mix.k.norm"] = (q,), (k,), (q,), (k,)
                t[p + "mix.r1"] = t[p + "mix.r2"] = (s.heads,)
        if s.experts:
            outputs = s.experts + s.router_identity
            t[p + "mlp.router"] = (outputs, H)
            if design == "belizen":
                t[p + "mlp.correction"] = (outputs,)
            for name, ff in [(f"e{j}", s.ffn_dim) for j in range(s.experts)] + [("shared", s.shared_dim)]:
                if s.expert_form != "gelu":
                    t[f"{p}mlp.{name}.gate"] = (ff, H)
                t[f"{p}mlp.{name}.up"], t[f"{p}mlp.{name}.down"] = (ff, H), (H, ff)
        elif design == "zulozen":
            t[p + "mlp.up"], t[p + "mlp.up.b"], t[p + "mlp.down"], t[p + "mlp.down.b"] = (s.ffn_dim, H), (s.ffn_dim,), (H, s.ffn_dim), (H,)
        elif design == "belizen":
            t[p + "mlp.gate"], t[p + "mlp.up"], t[p + "mlp.down"] = (s.ffn_dim, H), (s.ffn_dim, H), (H, s.ffn_dim)
    return t


# ---- weights and inputs ------------------------------------------------------------------------------------------------------------------

class _Weights:
    """Random bf16 tensors on the GPU, each made from (seed, its place in the list) alone, when it is asked for.

    Matrices have 1 / sqrt(inputs), gains stand around one, biases are of visible size. The routers of the mixtures read a few dimensions of the
    stream into which only the embedding writes: trained routers are as decided, and rounding then does not move a token to another expert."""

    def __init__(self, case, meta, seed):
        self.design, self.shapes, self.seed = case["design"], _shapes(case, meta), seed
        self.order = {n: i for i, n in enumerate(self.shapes)}
        self.mixtures = any("router" in n for n in self.shapes)
        rng = np.random.default_rng([seed, 1])
        self.kind = torch.from_numpy(rng.permutation(VOCAB) % PATTERNS).cuda()

    def __getitem__(self, name):
        shape = self.shapes[name]
        g = torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + self.order[name]) % (1 << 62))
        x = torch.empty(shape, device="cuda").normal_(generator=g)
        leaf = name.rsplit(".", 1)[-1]
        if leaf == "b" or leaf == "bias":
            x = (1.0 if name.endswith("a2.b") else 0.0) + (1.5 if name.endswith("a2.b") else 0.5) * x
        elif "norm" in name:
            x = 1.0 + 0.1 * x
        elif leaf == "sink":
            x = 1.0 + x
        elif leaf == "r1":
            x = 0.2 + x.abs()
        elif leaf == "r2":
            x = 0.05 + 0.3 * x.abs()
        elif leaf == "correction":
            x = 0.02 * x
        elif leaf.startswith("canon"):
            x = 0.4 * x
        elif name == "pos":
            x = 0.3 * x
        elif name not in ("embed", "bigram", "model.embed_tokens.weight"):
            x = x / math.sqrt(shape[-1])
        if self.mixtures:
            self._decide(name, leaf, x)
        return x.bfloat16()

    def _decide(self, name, leaf, x):
        P = PATTERNS
        if name == "embed":
            x[:, :P] = 3.0 * torch.eye(P, device="cuda")[self.kind]
        elif name in ("bigram", "pos"):
            x[:, :P] = 0.0
        elif leaf in ("o", "down") and x.dim() == 2:
            x[:P] = 0.0
        elif leaf in ("norm1b", "norm2b") and x.dim() == 1 or name.endswith("down.b"):
            x[:P] = 0.0
        elif leaf == "norm2" and x.dim() == 1:
            x[:P] = 1.0
        elif leaf == "router":
            rng = np.random.default_rng([self.seed, 2, self.order[name]])
            n, z = x.shape[0], np.empty((x.shape[0], P), np.float32)
            for p in range(P):
                z[:, p] = rng.uniform(-1.6, -1.2, n)
                if self.design == "vusenex":  # the best of two groups
                    best = [g * (n // GROUPS) + rng.integers(n // GROUPS) for g in rng.permutation(GROUPS)[:TOP]]
                else:
                    best = rng.permutation(n)[:TOP]
                z[best, p] = rng.permutation([0.6, 1.2])
            x.zero_()
            x[:, :P] = torch.from_numpy(z).cuda()


_staging = []


def _pinned(n):
    if not _staging or _staging[0].numel() < n:
        _staging[:] = [torch.empty(n, dtype=torch.bfloat16, pin_memory=True)]
    return _staging[0][:n]


def _model(case, seed, blocks, rows, sequences):
    """A model with its weights, loaded tensor by tensor as from a checkpoint."""
    meta, backend = _metadata(case), orion.CudaBackend(0)
    dtype = orion.DType.F32 if case["design"] == "tiny" else orion.DType.BF16
    cls = orion.CudaTransformerModel if case["design"] in DENSE else orion.CudaLayeredModel
    model = cls(meta, blocks, BLOCK, backend, compute_dtype=dtype, max_batch_tokens=rows, max_batch_sequences=sequences)
    weights = _Weights(case, meta, seed)
    for name, shape in weights.shapes.items():
        x = weights[name].reshape(-1)
        host = _pinned(max(x.numel(), 1 << 24))[:x.numel()]
        host.copy_(x)
        model.load_tensor(name, host.view(torch.int16).numpy(), shape, orion.DType.BF16)
    model.finalize()
    return model


def _texts(case, seed):
    """The tokens of every sequence, with those of the steps of a generation."""
    rng = np.random.default_rng([seed, 3])
    vocab = 1024 if case["design"] == "tiny" else VOCAB
    return [rng.integers(0, vocab, c + case.get("steps", 0)).astype(np.uint32) for c, _ in _lengths(case)]


def prepare(case, seed):
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    lengths, texts = _lengths(case), _texts(case, seed)
    n = len(lengths)
    blocks = [(len(t) + BLOCK - 1) // BLOCK for t in texts]
    pool = sum(blocks) + 16
    most = 8192  # rows of a forward
    model = _model(case, seed, pool, most, max(n, 64))
    order = np.random.default_rng([seed, 4]).permutation(pool).astype(np.uint32)
    ends = np.cumsum(blocks)
    tables = [np.ascontiguousarray(order[e - b:e]) for e, b in zip(ends, blocks)]
    slots = np.arange(n, dtype=np.uint32) if model.num_state_slots() else None

    def batch(parts, prefill):
        """parts: (sequence, first position, positions after it)"""
        tabs = [tables[s] for s, _, _ in parts]
        if len({len(t) for t in tabs}) == 1:
            tabs = np.stack(tabs)
        return orion.ForwardBatch(np.concatenate([texts[s][a:b] for s, a, b in parts]), np.concatenate([np.arange(a, b, dtype=np.uint32) for _, a, b in parts]),
                                  np.array([s + 1 for s, _, _ in parts], np.uint64), np.array([b - a for _, a, b in parts], np.uint64),
                                  np.array([b for _, _, b in parts], np.uint64), tabs, has_prefill=prefill,
                                  state_slots=None if slots is None else slots[[s for s, _, _ in parts]])

    # what earlier steps left in the cache
    portion, room = [], most
    for s, (context, rows) in enumerate(lengths):
        at = 0
        while at < context - rows:
            take = min(room, context - rows - at)
            portion.append((s, at, at + take))
            at, room = at + take, room - take
            if room == 0:
                model.forward(batch(portion, True))
                portion, room = [], most
    if portion:
        model.forward(batch(portion, True))
    batches = [batch([(s, c - r, c) for s, (c, r) in enumerate(lengths)], case["kind"] != "decode")]
    if case["kind"] == "generate":
        batches += [batch([(s, c + k, c + k + 1) for s, (c, _) in enumerate(lengths)], False) for k in range(case["steps"])]
    size = n * model.metadata().vocab_size
    # page-locked buffers that the logits of a forward come back in
    return {"model": model, "batches": batches, "outs": [torch.empty(size, pin_memory=True).numpy() for _ in batches]}


def run(state):
    if "call" in state:
        return state["call"]()
    return [state["model"].forward(b, out=o).logits for b, o in zip(state["batches"], state["outs"])]


# ---- attention by itself -----------------------------------------------------------------------------------------------------------------

HEADS, KV_HEADS, DIM = 32, 8, 128


def _attention_inputs(case, seed):
    contexts = _spread(case["shortest"], case["longest"], case["sequences"])
    blocks = [(c + BLOCK - 1) // BLOCK for c in contexts]
    pool = sum(blocks) + 64
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.empty(len(contexts), HEADS, DIM, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    arena = torch.empty(pool, KV_HEADS, 2, BLOCK, DIM, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    table = torch.randperm(pool, generator=g, device="cuda")[:sum(blocks)]
    return contexts, blocks, q, arena, table


def _prepare_attention(case, seed):
    contexts, blocks, q, arena, table = _attention_inputs(case, seed)
    n = len(contexts)
    positions = torch.tensor([c - 1 for c in contexts], dtype=torch.int32, device="cuda")
    sequences = torch.arange(n, dtype=torch.int32, device="cuda")
    offsets = torch.tensor(np.concatenate([[0], np.cumsum(blocks)]), dtype=torch.int32, device="cuda")
    flat, out = table.int(), torch.empty_like(q)
    lib, ptr = orion._ffi.lib(), [t.data_ptr() for t in (q, arena, positions, sequences, flat, offsets, out)]
    keep = (q, arena, positions, sequences, flat, offsets)

    def call():
        orion.errors.check(lib.orion_cuda_paged_decode_attention_noalloc(
            0, ptr[0], ptr[1], arena.shape[0], KV_HEADS, HEADS, ptr[2], ptr[3], ptr[4], ptr[5], n, max(contexts) - 1, 0, ptr[6],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return out

    return {"call": call, "keep": keep}


def _exact_attention(case, seed):
    contexts, blocks, q, arena, table = _attention_inputs(case, seed)
    # the arena keeps the 16-byte groups of a row permuted by slot & 7
    place = (torch.arange(DIM // 8, device="cuda")[None] ^ (torch.arange(BLOCK, device="cuda") & 7)[:, None])
    out, at = torch.empty(q.shape, dtype=torch.float64, device="cuda"), 0
    for i, (c, b) in enumerate(zip(contexts, blocks)):
        x = arena[table[at:at + b]].reshape(b, KV_HEADS, 2, BLOCK, DIM // 8, 8)
        x = torch.gather(x, 4, place[None, None, None, :, :, None].expand(x.shape)).double()
        k, v = (x[:, :, j].reshape(b, KV_HEADS, BLOCK, DIM).transpose(0, 1).reshape(KV_HEADS, b * BLOCK, DIM)[:, :c] for j in (0, 1))
        p = torch.softmax(q[i].double().view(KV_HEADS, HEADS // KV_HEADS, DIM) @ k.transpose(1, 2) * DIM ** -0.5, -1)
        out[i] = (p @ v).reshape(HEADS, DIM)
        at += b
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------------

def _reached(rows):
    """Experts that the tokens of `rows` rows reach on average."""
    return EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** rows)


def _forward_work(case, meta, parts):
    """(bytes, flops) of one forward. parts: (context, rows) of every sequence."""
    rows, outs, V = sum(r for _, r in parts), len(parts), meta.vocab_size
    H, es = meta.hidden_size, 4 if case["design"] == "tiny" else 2

    def keys(most):  # (query, key) pairs, keys read from the cache
        return (sum(sum(min(i, most) for i in range(c - r + 1, c + 1)) for c, r in parts),
                sum(min(c - r, most + r) for c, r in parts))

    table = es * H * min(rows, V) + es * H * V + 4 * V * outs  # embedding rows, head, logits
    if case["design"] in DENSE:
        q, k = meta.num_attention_heads * meta.head_dim, meta.num_kv_heads * meta.head_dim
        n = H * (q + 2 * k) + q * H + 3 * H * meta.ffn_dim
        pairs, cached = keys(1 << 30)
        per_layer = (es * n + es * 2 * k * (cached + rows), 2 * n * rows + 4 * pairs * q)
        return table + meta.num_layers * per_layer[0], 2 * outs * V * H + meta.num_layers * per_layer[1]
    bytes_, flops = table, 2 * outs * V * H
    for s in meta.layers:
        cache = 0
        pairs, cached = keys(s.window + s.keep_first if s.window else s.chunk or 1 << 30)
        if s.mixer == "mingru":
            n = 4 * H * s.width
            cache, flops = 8 * s.width * outs, flops + 6 * rows * s.width
        elif s.mixer == "latent_attention":
            q, v = s.heads * s.dim, s.heads * s.value_dim
            n = H * (q + s.heads * s.rot_dim + s.kv_rank + s.rot_dim + (0 if s.ungated else v)) + v * H + (q + v) * s.kv_rank
            cache = es * (s.kv_rank + s.rot_dim) * (cached + rows)
            flops += 2 * pairs * s.heads * (s.dim + s.rot_dim + s.value_dim)
        elif s.mixer == "gla":
            k, v = s.heads * s.dim, s.heads * s.value_dim
            n = H * (2 * k + 2 * v + s.decay_rank) + k * s.decay_rank + v * H
            cache, flops = 8 * k * s.value_dim * outs, flops + 4 * rows * k * s.value_dim
        else:
            per_token = s.kv_heads * (s.dim if s.keys_as_values else s.dim + s.value_dim)
            n = H * (s.heads * s.dim + per_token) + s.heads * s.value_dim * H
            n += H * s.heads * s.value_dim if s.value_gate else H * s.heads if s.head_gate else 0
            cache = es * per_token * (cached + rows)
            flops += 2 * pairs * s.heads * (s.dim + s.value_dim)
        if case["design"] == "vusenex":
            n += 2 * H * H
        if s.experts:
            one, outputs = (2 if s.expert_form == "gelu" else 3) * H * s.ffn_dim, s.experts + s.router_identity
            n += H * outputs + one // s.ffn_dim * s.shared_dim
            bytes_ += int(es * _reached(rows) * one)
            flops += int(2 * TOP * s.experts / outputs * one * rows)
        else:
            n += (3 if s.activation == "geglu_tanh" else 2) * H * s.ffn_dim
        bytes_, flops = bytes_ + es * n + cache, flops + 2 * n * rows
    return bytes_, flops


def work(case):
    if case["kind"] == "attention":
        contexts = _spread(case["shortest"], case["longest"], case["sequences"])
        return {"bytes": sum(c * KV_HEADS * DIM * 4 + HEADS * DIM * 4 for c in contexts), "flops": sum(4 * c * HEADS * DIM for c in contexts)}
    meta, lengths = _metadata(case), _lengths(case)
    steps = [lengths] + [[(c + k + 1, 1) for c, _ in lengths] for k in range(case.get("steps", 0))]
    got = [_forward_work(case, meta, p) for p in steps]
    return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}


def tolerance(case):
    """About four times the distance from ``exact``, measured: 6e-7 in the f32 build (whose sums another order would move further), 2.2e-3
    of one attention in bf16, 2.2e-3 to 4.8e-3 of whole models in bf16, 8.5e-3 where nothing normalises what a sublayer reads."""
    if case["design"] == "tiny":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "attention":
        return {"rel": 8e-3, "max": 5e-2}
    return {"rel": 3e-2, "max": 0.25} if case["design"] == "vusenex" else {"rel": 2e-2, "max": 0.15}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------------------

def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _heads(x, n):
    return x.view(x.shape[0], n, -1)


def _turn(x, pos, freq, mult, halves):
    """Rotates the first 2 len(freq) entries of every head; pairs are half of them apart or neighbours."""
    n = freq.numel()
    ang = pos.double()[:, None, None] * freq
    c, s = ang.cos() * mult, ang.sin() * mult
    u, v = (x[..., :n], x[..., n:2 * n]) if halves else (x[..., 0:2 * n:2], x[..., 1:2 * n:2])
    a, b = u * c - v * s, v * c + u * s
    y = torch.cat([a, b], -1) if halves else torch.stack([a, b], -1).flatten(-2)
    return torch.cat([y, x[..., 2 * n:]], -1)


def _frequencies(dims, base, yarn=None):
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = base ** (-2.0 * i / dims)
    if yarn is None:
        return f, 1.0

    def dim_of(turns):
        return dims * math.log(yarn.original / (2 * math.pi * turns)) / (2 * math.log(base))

    low, high = max(math.floor(dim_of(yarn.fast)), 0), min(math.ceil(dim_of(yarn.slow)), dims - 1)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
    return f / yarn.factor * ramp + f * (1 - ramp), 0.1 * math.log(yarn.factor) + 1.0


def _attend(q, k, v, scale, seen=None, sink=None, cap=0.0, bias=None):
    """q [T, heads, D], k and v [T, kv heads, D] of one sequence from its first position. seen(i, j): whether i sees j <= i; sink: further logits
    in the denominators, one per head; bias(i - j): [heads, ..] taken off the scores."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device="cuda")
    j = torch.arange(T, device="cuda")
    step = max(16, min(T, (1 << 28) // (H * T)))
    for a in range(0, T, step):
        i = j[a:a + step, None]
        n = i.shape[0]
        s = torch.einsum("tgmd,jgd->gmtj", q[a:a + n].view(n, G, H // G, -1), k).reshape(H, n, T) * scale
        if bias is not None:
            s = s - bias((i - j).clamp(min=0))
        if cap:
            s = cap * torch.tanh(s / cap)
        mask = j <= i
        s.masked_fill_(~(mask if seen is None else mask & seen(i, j)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.view(H, 1, 1).expand(H, n, 1)], -1)
        p = torch.softmax(s, -1)[..., :T]
        out[a:a + n] = torch.einsum("gmtj,jgd->tgmd", p.reshape(G, H // G, n, T), v).reshape(n, H, -1)
    return out


class _Exact:
    def __init__(self, case, seed):
        self.case, self.meta = case, _metadata(case)
        self.w = _Weights(case, self.meta, seed)
        self.texts = [torch.from_numpy(t.astype(np.int64)).cuda() for t in _texts(case, seed)]
        self.tokens = torch.cat(self.texts)
        self.ends = np.cumsum([len(t) for t in self.texts])
        self.pos = torch.cat([torch.arange(len(t), device="cuda") for t in self.texts])

    def weight(self, name):
        return self.w[name].double()

    def linear(self, x, name):
        return x @ self.weight(name).T

    def each(self, f, *xs):
        """f of every sequence's rows, put together again."""
        return torch.cat([f(*(x[e - len(t):e] for x in xs)) for e, t in zip(self.ends, self.texts)])

    def by_rows(self, f, x):
        return torch.cat([f(c) for c in x.split(32768)])

    def logits(self):
        """Of the rows that the measured forwards return, forward by forward."""
        x, head = (self.dense if self.case["design"] in DENSE else self.layered)()
        lengths = _lengths(self.case)
        first = [e - len(t) + c - 1 for e, t, (c, _) in zip(self.ends, self.texts, lengths)]
        out = []
        for k in range(1 + self.case.get("steps", 0)):
            y = x([r + k for r in first]) @ head.T
            cap = getattr(self.meta, "logit_softcap", 0.0)
            out.append(cap * torch.tanh(y / cap) if cap else y)
        return out

    def dense(self):
        m = self.meta
        x = self.weight("model.embed_tokens.weight")[self.tokens]
        freq, _ = _frequencies(m.head_dim, m.rope_theta)
        for i in range(m.num_layers):
            p = f"model.layers.{i}."
            h = _rms(x, self.weight(p + "input_layernorm.weight"), m.rms_norm_eps)
            q, k, v = (self.linear(h, f"{p}self_attn.{n}_proj.weight") + (self.weight(f"{p}self_attn.{n}_proj.bias") if m.has_qkv_bias else 0.0) for n in "qkv")
            q, k = (_turn(_heads(y, n), self.pos, freq, 1.0, True) for y, n in ((q, m.num_attention_heads), (k, m.num_kv_heads)))
            y = self.each(lambda *a: _attend(*a, m.head_dim ** -0.5), q, k, _heads(v, m.num_kv_heads))
            x = x + self.linear(y.flatten(1), p + "self_attn.o_proj.weight")
            wg, wu, wd = (self.weight(f"{p}mlp.{n}_proj.weight") for n in ("gate", "up", "down"))
            norm = self.weight(p + "post_attention_layernorm.weight")

            def ffn(c):
                h = _rms(c, norm, m.rms_norm_eps)
                return c + (F.silu(h @ wg.T) * (h @ wu.T)) @ wd.T

            x = self.by_rows(ffn, x)
        norm = self.weight("model.norm.weight")
        return lambda rows: _rms(x[rows], norm, m.rms_norm_eps), self.weight("lm_head.weight")

    def layered(self):
        m, eps, w = self.meta, self.meta.norm_eps, self.weight
        mult = m.residual_mult
        x = w("embed")[self.tokens] * m.embed_scale
        if m.bigram is not None:
            before = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), self.tokens[:-1]])
            row = (before * m.bigram.mul_prev + self.tokens * m.bigram.mul_cur) % m.bigram.buckets
            x = x + w("bigram")[torch.where(self.pos == 0, m.bigram.buckets, row)] + w("pos")[self.pos]
        for i, s in enumerate(m.layers):
            p = f"l{i}."
            mixer = getattr(self, s.mixer)
            if m.block == "parallel":
                h = _rms(x, w(p + "norm1"), eps)
                y = mixer(h + self.conv(h, p + "canon1"), s, p + "mix.")
                u = h + self.conv(h, p + "canon2")
                x = x + y + self.linear(F.gelu(self.linear(u, p + "mlp.up"), approximate="tanh"), p + "mlp.down")
            elif m.block == "sandwich":
                x = x + mult * _rms(mixer(_rms(x, w(p + "norm1"), eps), s, p + "mix."), w(p + "norm1b"), eps)
                x = x + mult * _rms(self.feed(_rms(x, w(p + "norm2"), eps), s, p + "mlp."), w(p + "norm2b"), eps)
            elif m.block == "prenorm":
                x = x + mult * mixer(_rms(x, w(p + "norm1"), eps), s, p + "mix.")
                x = x + mult * self.feed(_rms(x, w(p + "norm2"), eps), s, p + "mlp.")
            else:
                x = x + _rms(torch.sigmoid(self.linear(x, p + "rg1") + w(p + "rg1.b")) * mixer(x, s, p + "mix."), w(p + "norm1"), eps)
                x = x + _rms(torch.sigmoid(self.linear(x, p + "rg2") + w(p + "rg2.b")) * self.feed(x, s, p + "mlp."), w(p + "norm2"), eps)
        return lambda rows: _rms(x[rows], w("final.norm"), eps), w("head" if m.untied_lm_head else "embed")

    def conv(self, h, name):
        taps = self.weight(name)
        n = taps.shape[1]
        return self.each(lambda c: sum(F.pad(c, (0, 0, n - 1 - j, 0))[:len(c)] * taps[:, j] for j in range(n)), h)

    def mingru(self, h, s, p):
        z = torch.sigmoid(self.linear(h, p + "z") + self.weight(p + "z.b"))
        u = self.linear(h, p + "x") + self.weight(p + "x.b")
        c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))

        def scan(z, c):
            state, out = torch.zeros_like(c[0]), torch.empty_like(c)
            for t in range(len(z)):
                state = torch.lerp(state, c[t], z[t])
                out[t] = state
            return out

        return self.linear(self.each(scan, z, c) * F.silu(self.linear(h, p + "g")), p + "o")

    def latent_attention(self, h, s, p):
        q, dkv = _heads(self.linear(h, p + "q"), s.heads), self.linear(h, p + "dkv")
        c = _rms(dkv[:, :s.kv_rank], self.weight(p + "dkv.norm"), self.meta.norm_eps)
        k, v = _heads(self.linear(c, p + "uk"), s.heads), _heads(self.linear(c, p + "uv"), s.heads)
        if s.rot_dim:
            freq, _ = _frequencies(s.rope_dims, s.rope_base)
            q = torch.cat([q[..., :s.dim], _turn(q[..., s.dim:], self.pos, freq, 1.0, False)], -1)
            turned = _turn(dkv[:, None, s.kv_rank:], self.pos, freq, 1.0, False)
            k = torch.cat([k, turned.expand(-1, s.heads, -1)], -1)
        seen = (lambda i, j: i - j < s.window) if s.window else None
        y = self.each(lambda *a: _attend(*a, s.scale, seen), q, k, v).flatten(1)
        return self.linear(y if s.ungated else y * torch.sigmoid(self.linear(h, p + "g")), p + "o")

    def gla(self, h, s, p):
        q, k, v = (_heads(self.linear(h, p + n), s.heads) for n in "qkv")
        decay = torch.sigmoid(self.linear(self.linear(h, p + "a1"), p + "a2") + self.weight(p + "a2.b")) ** (1.0 / s.decay_tau)

        def scan(q, k, v, a):
            state, out = torch.zeros(s.heads, s.dim, s.value_dim, dtype=torch.float64, device="cuda"), torch.empty_like(v)
            for t in range(len(q)):
                state = torch.baddbmm(state * a[t, :, :, None], k[t, :, :, None], v[t, :, None])
                out[t] = torch.bmm(q[t, :, None], state)[:, 0]
            return out

        y = self.each(scan, q * s.dim ** -0.5, k, v, _heads(decay, s.heads))
        y = _rms(y, self.weight(p + "norm"), self.meta.norm_eps).flatten(1)
        return self.linear(y * F.silu(self.linear(h, p + "g")), p + "o")

    def attention(self, h, s, p):
        w, eps = self.weight, self.meta.norm_eps
        q, k = self.linear(h, p + "q"), self.linear(h, p + "k")
        v = None if s.keys_as_values else self.linear(h, p + "v")
        if s.qkv_bias:
            q, k = q + w(p + "q.b"), k + w(p + "k.b")
            v = v if v is None else v + w(p + "v.b")
        v = k if s.keys_as_values else v
        if s.qk_norm is True:
            q, k = (_heads(_rms(x, w(f"{p}{n}.norm"), eps), c) for x, n, c in ((q, "q", s.heads), (k, "k", s.kv_heads)))
        else:
            q, k = (_rms(_heads(x, c), w(f"{p}{n}.norm"), eps) for x, n, c in ((q, "q", s.heads), (k, "k", s.kv_heads)))
        if s.rope_dims:
            freq, turn = _frequencies(s.rope_dims, s.rope_base, s.yarn)
            q, k = (_turn(x, self.pos, freq, turn, s.rope_halves) for x in (q, k))
        if s.q_temp:
            grown = torch.log(torch.floor((self.pos.double() + 1) / s.q_temp.every) + 1.0)
            q = q * (1.0 + s.q_temp.coef * grown)[:, None, None]
        seen = bias = sink = None
        if s.chunk:
            seen = lambda i, j: i // s.chunk == j // s.chunk  # noqa: E731
        if s.window:
            seen = lambda i, j: (i - j < s.window) | (j < s.keep_first)  # noqa: E731
        if s.distance_bias:
            r1, r2 = w(p + "r1")[:, None, None], w(p + "r2")[:, None, None]
            bias = lambda d: r1 * torch.log1p(r2 * d)  # noqa: E731
        if s.sinks:
            sink = w(p + "sink") if s.sinks is True else torch.zeros(s.heads, dtype=torch.float64, device="cuda")
        y = self.each(lambda *a: _attend(*a, s.scale, seen, sink, s.softcap, bias), q, k, _heads(v, s.kv_heads))
        if s.head_gate:
            y = y * torch.sigmoid(self.linear(h, p + "g"))[..., None]
        y = y.flatten(1)
        return self.linear(y * torch.sigmoid(self.linear(h, p + "g")) if s.value_gate else y, p + "o")

    def expert(self, h, s, name, limit):
        up = self.linear(h, name + ".up")
        if s.expert_form == "gelu":
            return self.linear(F.gelu(up), name + ".down")
        gate = self.linear(h, name + ".gate")
        if s.expert_form == "clamped":
            gate = gate.clamp(max=limit)
            return self.linear(gate * torch.sigmoid(1.702 * gate) * (up.clamp(-limit, limit) + 1.0), name + ".down")
        return self.linear(F.silu(gate) * up, name + ".down")

    def feed(self, h, s, p):
        w = self.weight
        if not s.experts:
            if s.activation == "relu2":
                return self.linear(F.relu(self.linear(h, p + "up") + w(p + "up.b")).square(), p + "down") + w(p + "down.b")
            return self.linear(F.gelu(self.linear(h, p + "gate"), approximate="tanh") * self.linear(h, p + "up"), p + "down")
        z = self.linear(h, p + "router")
        score = torch.sigmoid(z) if s.router == "sigmoid_input" else torch.softmax(z, -1)
        order = score + w(p + "correction") if s.router == "softmax" else score
        if s.router_groups:
            best = score.view(len(h), s.router_groups, -1).amax(-1)
            kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(s.router_keep, -1).indices, True)
            order = order.masked_fill(~kept.repeat_interleave(s.experts // s.router_groups, 1), -math.inf)
        chosen = order.topk(s.experts_per_token, -1).indices
        weight = score.gather(1, chosen)
        if s.router == "softmax_renorm":
            weight = weight / weight.sum(-1, keepdim=True)
        y = self.expert(h, s, p + "shared", s.shared_limit)
        for e in range(s.experts + s.router_identity):
            rows, place = torch.nonzero(chosen == e, as_tuple=True)
            if len(rows):
                x, by = h[rows], weight[rows, place][:, None]
                if s.router == "sigmoid_input":
                    y[rows] += self.expert(by * x, s, f"{p}e{e}", 0.0)
                else:
                    y[rows] += by * (self.expert(x, s, f"{p}e{e}", s.expert_limit) if e < s.experts else x)
        return y


def exact(case, seed):
    if case["kind"] == "attention":
        return _exact_attention(case, seed)
    meta, lengths = _metadata(case), _lengths(case)
    whole = [(c + case.get("steps", 0),) * 2 for c, _ in lengths]
    if _forward_work(case, meta, whole)[1] > MOST_EXACT_FLOPS:
        return None
    with torch.no_grad():
        return _Exact(case, seed).logits()
