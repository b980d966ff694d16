"""What the engine is timed on: the layers a model is made of, each through the part's own `forward` on a step of real
rows against a paged cache, and the whole engine fed token by token as a replay does it.

A case says which part (`kind`), of which size, in which number type, and what the step brings: `requests` entries of
`tokens` new tokens each, behind `context` tokens that every request already holds.  One token a request is decoding (the
part is then replayed from a CUDA graph, as the engine replays such steps); more is a portion of a prompt, run eagerly.
The sizes are those of the shapes and designs this repository measures (flambeau_b200/measure): widths 2,048, 4,096 and
5,120, heads of 128.  Inputs are rows as a norm leaves them (unit variance, in the engine's type), weights N(0, 0.02), keys
and values of unit variance.

kinds   gqa            grouped-query attention: product, rotation and cache write, attention under a window, output product
        latent         attention over cached latents with a sink per head (32-bit softmax weights)
        diff           differential attention within chunks, with a norm and a rotation on both maps
        delta          gated delta rule, a decay per head          channel_delta   a decay per head and key channel
        linear         gated linear attention (a decay per channel)
        mlp            SiLU-gated feed-forward                     experts         routed experts with a shared expert
        replay         the whole engine: prompts in, given token ids step by step, logits out
"""
from __future__ import annotations

import hashlib
import math

import torch

PAGE = 16
VOCAB = 32000                 # of the whole models; single parts need no vocabulary
EPS = 1e-6

# the sizes of the designs: w(idth), heads H on G key/value heads, window (chunk of `diff`), gated feed-forward,
# experts (how many, how many a token takes, inner size, shared expert's inner size)
SIZES = {
    "1b": dict(w=2048, H=16, G=4, window=1024, ff=8192, E=32, K=4, eff=1024, sff=4096),
    "7b": dict(w=4096, H=32, G=8, window=4096, ff=14336, E=64, K=6, eff=1792, sff=3584),
    "12b": dict(w=5120, H=32, G=8, window=0, ff=14336, E=0, K=0, eff=0, sff=0),
}
HD = 128                      # head size of every design (64 for each of the two maps of `diff`)
LATENT = 256                  # a cached latent row
TAPS, RANK, TAU, DIFF = 4, 128, 16.0, 0.5
REPLAY_LAYERS = 4
STATEFUL = ("delta", "channel_delta", "linear")
CACHED = ("gqa", "latent", "diff")


def _case(kind, size, requests, tokens, context=0, dtype="bfloat16", **more):
    return dict(kind=kind, size=size, requests=requests, tokens=tokens, context=context, dtype=dtype, **more)


def listed():
    return [
        # one user alone: a single row through the feed-forward, which is reading its weights once (the smallest call)
        dict(_case("mlp", "1b", 1, 1), name="mlp_decode_1"),
        # serving eight users at a long context: the benchmark's decode step, one layer's attention
        dict(_case("gqa", "7b", 8, 1, 8191), name="gqa_decode_8"),
        # the prompt of the benchmark, one layer's attention
        dict(_case("gqa", "7b", 1, 2048), name="gqa_prompt_2048"),
        # a prompt's chunk of 512 beside 25 decoded rows, as the scheduler mixes them: the feed-forward sees 537 rows
        dict(_case("mlp", "12b", 1, 537), name="mlp_mixed_537"),
        # the true 32-bit path that logits are checked on: a portion behind a cached prefix, odd sizes
        dict(_case("gqa", "7b", 1, 301, 500, dtype="float32"), name="gqa_float32_301"),
        # eight users decoding against cached latents
        dict(_case("latent", "7b", 8, 1, 8171), name="latent_decode_8"),
        # a whole prompt over latents
        dict(_case("latent", "7b", 1, 2048), name="latent_prompt_2048"),
        # a whole prompt of differential attention (one chunk)
        dict(_case("diff", "7b", 1, 2048), name="diff_prompt_2048"),
        # a whole prompt through the recurrence with a decay per channel
        dict(_case("channel_delta", "7b", 1, 2048), name="channel_delta_prompt_2048"),
        # three users' portions of odd length in one step through the recurrence with a decay per head
        dict(_case("delta", "1b", 3, 343), name="delta_portions_3x343"),
        # a whole prompt through routed experts (the largest call)
        dict(_case("experts", "7b", 1, 2048), name="experts_prompt_2048"),
        # the whole engine: three prompts of odd lengths, then given tokens step by step, logits of every step
        dict(_case("replay", "7b", 3, 173, steps=24), name="replay_3x173"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gqa", "gqa", "mlp", "mlp", "latent", "diff", "delta", "channel_delta", "linear", "experts", "replay"])
    size = rng.choice(["1b", "7b", "12b"] if kind in ("gqa", "mlp", "latent", "diff") else ["1b", "7b"])
    dtype = "float32" if kind not in ("experts", "replay") and rng.random() < 0.12 else "bfloat16"
    if kind == "replay":
        return _case(kind, size, rng.randint(1, 4), _log(rng, 9, 180), steps=rng.randint(4, 24))
    if rng.random() < 0.4:                                    # decoding
        requests = _log(rng, 1, 64 if dtype == "bfloat16" else 8)
        context = _log(rng, 40, 8191 if requests <= 16 else 3000) if kind in CACHED else 0
        return _case(kind, size, requests, 1, context, dtype=dtype)
    requests = rng.choice([1, 1, 1, 2, 3, 4])
    most = (2048 if dtype == "bfloat16" else 320) // requests
    context = rng.choice([0, _log(rng, 10, 2000)]) if kind in CACHED else 0
    if dtype == "float32":
        context = min(context, 500)
    return _case(kind, size, requests, _log(rng, 17, most), context, dtype=dtype)


# ---- what a user's program has in hand ---------------------------------------------------------------------------
def _random(seed, name, shape, std=1.0, mean=0.0):
    """float32 on the GPU, from the seed and the name alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    t = torch.randn(shape, generator=g, dtype=torch.float32, device="cuda")
    return t.mul_(std).add_(mean)


def _weight(seed, name, shape, dtype):
    """A tensor of a model file as the engine holds it."""
    leaf = name.split(".")[-1]
    if leaf == "norm" or name.endswith(("norm.weight", "layernorm.weight")):
        std, mean = 0.1, 1.0
    elif leaf in ("lq1", "lk1", "lq2", "lk2"):
        std, mean = 0.1, 0.0
    elif leaf == "conv":
        std, mean = 0.25, 0.0
    elif leaf in ("A_log", "dt_bias", "a2", "g2"):
        std, mean = (0.1 if leaf in ("a2", "g2") else 0.5), 0.0
    elif leaf == "sink" or name.endswith("a2.b"):
        std, mean = 1.0, 0.0
    else:
        std, mean = 0.02, 0.0
    return _random(seed, name, shape, std, mean).to(dtype)


def _part(case):
    """(mixer, feed-forward) of the case as data; the part that is timed and the least that a layer needs beside it."""
    from flambeau_b200.parts.spec import PartSpec
    s, kind = SIZES[case["size"]], case["kind"]
    w, H, G = s["w"], s["H"], s["G"]
    rotary = PartSpec("position", "rotary_half", dict(head_dim=HD, theta=10000.0))
    if kind == "gqa":
        return PartSpec("mixer", "attention", dict(width=w, num_heads=H, num_kv_heads=G, head_dim=HD, window=s["window"],
                                                   position=rotary), "mix."), None
    if kind == "latent":
        return PartSpec("mixer", "latent_attention", dict(
            width=w, num_heads=H, head_dim=HD, rot_dim=0, value_dim=HD, kv_rank=LATENT, q_rank=None, window=0,
            scale=HD ** -0.5, eps=EPS, gate=False, sink=True), "mix."), None
    if kind == "diff":
        half = PartSpec("position", "rotary_half", dict(head_dim=HD // 2, theta=1e6))
        return PartSpec("mixer", "diff_attention", dict(
            width=w, num_heads=H, num_kv_heads=G, key_dim=HD // 2, value_dim=HD, chunk=s["window"] or 8192,
            scale=(HD // 2) ** -0.5, diff=DIFF, eps=EPS, bias=True, out_bias=False, head_gate=False, qk_norm=True,
            position=half), "mix."), None
    if kind in ("delta", "channel_delta"):
        more = dict(decay="channel", gate="sigmoid", low_rank_gate=True, rank=RANK) if kind == "channel_delta" else {}
        return PartSpec("mixer", "gated_delta", dict(
            width=w, num_heads=H, num_qk_heads=H if kind == "channel_delta" else G, key_dim=HD, value_dim=HD, conv=TAPS,
            eps=EPS, unit_eps=EPS, **more), "mix."), None
    if kind == "linear":
        return PartSpec("mixer", "gated_linear_attention", dict(
            width=w, num_heads=H, key_dim=HD, value_dim=HD, tau=TAU, eps=EPS, decay_rank=16), "mix."), None
    small = PartSpec("mixer", "attention", dict(width=w, num_heads=1, num_kv_heads=1, head_dim=16), "mix.")
    if kind == "mlp":
        return small, PartSpec("feed_forward", "gated_mlp", dict(width=w, inner=s["ff"], activation="silu"), "mlp.")
    return small, PartSpec("feed_forward", "routed_experts", dict(
        width=w, inner=s["eff"], experts=s["E"], top=s["K"], activation="relu_squared", shared_inner=s["sff"],
        router_bias=False), "mlp.")


def _bind(model, seed, dtype):
    for part in model.parts():
        part.bind({name: _weight(seed, name, spec.shape, dtype) for name, spec in part.tensor_specs().items()})


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _live(case):
    """The first position of the context that the step's first token still sees."""
    s, context = SIZES[case["size"]], case["context"]
    if case["kind"] == "gqa" and s["window"]:
        return max(0, context - s["window"] + 1)
    if case["kind"] == "diff":
        chunk = s["window"] or 8192
        return context // chunk * chunk
    return 0


def _context(case, seed):
    """Keys and values of every request's live context, logically ordered: [requests, live, key/value heads, size]."""
    s, dt = SIZES[case["size"]], _dtype(case)
    live, heads = case["context"] - _live(case), 1 if case["kind"] == "latent" else s["G"]
    size = LATENT if case["kind"] == "latent" else HD
    k = _random(seed, "context k", (case["requests"], live, heads, size)).to(dt)
    v = k if case["kind"] == "latent" else _random(seed, "context v", (case["requests"], live, heads, size)).to(dt)
    return k, v


def _rows(case, seed):
    n = case["requests"] * case["tokens"]
    return _random(seed, "rows", (n, SIZES[case["size"]]["w"])).to(_dtype(case))


class _PartState:
    """One part in an engine whose requests hold `context` tokens, and a step of `tokens` more for each."""

    def __init__(self, case, seed):
        import flambeau_b200.models  # noqa: F401  (registers the parts)
        from flambeau_b200.engine.batch import Entry
        from flambeau_b200.engine.runtime import Runtime
        from flambeau_b200.engine.step import Engine, EngineOptions
        from flambeau_b200.models.decoder import DecoderModel
        from flambeau_b200.parts.spec import LayerCall, ModelSpec, PartSpec
        w, n_req, n_tok, context = SIZES[case["size"]]["w"], case["requests"], case["tokens"], case["context"]
        mixer, ffn = _part(case)
        norm = lambda p: PartSpec("norm", "rmsnorm", dict(width=w, eps=EPS), p)  # noqa: E731
        block = dict(mixer=mixer, mixer_norm=norm("norm1."))
        if ffn is not None:
            block.update(feed_forward=ffn, feed_forward_norm=norm("norm2."))
        spec = ModelSpec(hidden_size=w, vocab_size=16,
                         embedding=PartSpec("embedding", "token_embedding", dict(vocab=16, width=w), "embed."),
                         layers=[PartSpec("block", "pre_norm", block, "")], order=[LayerCall(0)], final_norm=norm("final."),
                         head=PartSpec("head", "lm_head", dict(vocab=16, width=w), "head."))
        rt = Runtime("cuda:0", case["dtype"], PAGE)
        model = DecoderModel(spec, rt)
        _bind(model, seed, rt.dtype)
        total = context + n_tok + 2 * PAGE
        engine = Engine(model, EngineOptions(dtype=case["dtype"], page_size=PAGE, cache_tokens=n_req * total + 512,
                                             max_requests=n_req, max_step_tokens=n_req * n_tok, max_seq_len=total))
        self.engine, cache = engine, engine.cache
        layer = model.layers[0]
        self.part, self.is_mixer = (layer.mixer, True) if ffn is None else (layer.feed_forward, False)
        entries = [Entry(f"request {i}", [1] * n_tok, []) for i in range(n_req)]
        for e in entries:
            engine.admit(e.request_id)
            left = context
            while left > 0:
                k = min(left, 256)
                cache.reserve(e.request_id, k)
                cache.commit(e.request_id, k)
                left -= k
            cache.reserve(e.request_id, n_tok)
        self.batch = engine.buffers.build(entries, cache, 16)
        if self.batch.seq_slot != list(range(n_req)):
            raise RuntimeError("requests do not sit in the slots in their order")
        for g in cache.groups:
            for c in g.owners:
                g.k[c].zero_()
                g.v[c].zero_()
        if case["kind"] in CACHED and context > 0:
            self._fill(case, seed)
        self.h = _rows(case, seed)
        self.pools, self.recurrent = (), None
        view = cache.view(0, self.batch.tables, self.batch.table_bases)
        if case["kind"] in CACHED:
            self.pools = (view.k_pool,) if case["kind"] == "latent" else (view.k_pool, view.v_pool)
        if case["kind"] in STATEFUL:
            state = view.state.view(n_req, -1)
            s = SIZES[case["size"]]["H"] * HD * HD
            self.state, self.recurrent = state, (state[:, :s], state[:, s:])
        self.fresh = n_tok > 1               # a prompt's first portion starts on a zeroed state; decoding carries it on
        self.graph = None
        if n_tok == 1:
            self._capture()

    def _fill(self, case, seed):
        """The context's keys and values into the pages that the step's block tables name."""
        g = self.engine.cache.groups[0]
        owner, first, last = g.owners[0], _live(case), case["context"]
        k, v = _context(case, seed)
        pos = torch.arange(first, last, device="cuda")
        for i in range(case["requests"]):
            page = self.batch.tables[0][i].long()[pos // PAGE - int(self.batch.table_bases[0][i])]
            g.k[owner][page, :, pos % PAGE] = k[i]
            if case["kind"] != "latent":
                g.v[owner][page, :, pos % PAGE] = v[i]

    def _capture(self):
        """As the engine does it for steps of decoded tokens: once eagerly, then captured."""
        self.step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        ws, step_ws = self.engine.runtime.ws, self.engine.step_ws
        ws.frozen = step_ws.frozen = True
        kv, self.batch.max_kv_len = self.batch.max_kv_len, self.engine.max_seq_len
        try:
            with torch.cuda.graph(graph):
                self.out = self.step()
        finally:
            ws.frozen = step_ws.frozen = False
            self.batch.max_kv_len = kv
        self.graph = graph
        if self.recurrent is not None:
            self.state.zero_()

    def step(self):
        from flambeau_b200.engine.step import StepContext
        from flambeau_b200.parts.block import ResidualStream
        e = self.engine
        e.runtime.ws.reset()
        e.step_ws.reset()
        ctx = StepContext(e, self.batch)
        x = ctx.open_stream(self.h.shape[1])
        x.zero_()
        if self.fresh and self.recurrent is not None:
            self.state.zero_()
        ctx.stream_x, ctx.pending_slabs = x, 1
        if self.is_mixer:
            self.part.forward(ctx, self.h, ctx.delta, 0)
        else:
            self.part.forward(ctx, self.h, ctx.delta)
        ResidualStream(x, ctx.delta, ctx.pending_slabs).settle(ctx)
        return x

    def run(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            self.out = self.step()
        return dict(out=self.out, pools=list(self.pools), state=list(self.recurrent or ()))


def _replay_config(case):
    s = SIZES[case["size"]]
    return dict(architectures=["MistralForCausalLM"], rms_norm_eps=1e-5, tie_word_embeddings=False, hidden_act="silu",
                hidden_size=s["w"], num_hidden_layers=REPLAY_LAYERS, num_attention_heads=s["H"], num_key_value_heads=s["G"],
                head_dim=HD, intermediate_size=s["ff"], vocab_size=VOCAB, rope_theta=10000.0, sliding_window=s["window"],
                max_position_embeddings=32768)


def _replay_tokens(case, seed):
    """[requests, prompt + steps] token ids; the prompts' lengths differ by a few."""
    n = case["tokens"] + 2 * case["requests"] + case["steps"]
    ids = _random(seed, "tokens", (case["requests"], n)).mul_(1e4).long().remainder_(VOCAB)
    lengths = [case["tokens"] + 2 * i for i in range(case["requests"])]
    return [ids[i, :lengths[i] + case["steps"]].tolist() for i in range(case["requests"])], lengths


class _ReplayState:
    """A small model in an engine, and the token ids that it is fed."""

    def __init__(self, case, seed):
        import flambeau_b200.models  # noqa: F401
        from flambeau_b200.config.registry import resolve
        from flambeau_b200.engine.runtime import Runtime
        from flambeau_b200.engine.step import Engine, EngineOptions
        from flambeau_b200.models.decoder import DecoderModel
        arch = resolve("MistralForCausalLM")
        config = arch.config_class.from_dict(_replay_config(case))
        rt = Runtime("cuda:0", case["dtype"], PAGE)
        model = DecoderModel(arch.build_spec(config), rt)
        _bind(model, seed, rt.dtype)
        self.ids, self.lengths = _replay_tokens(case, seed)
        self.steps = case["steps"]
        most = max(len(i) for i in self.ids) + PAGE
        self.engine = Engine(model, EngineOptions(
            dtype=case["dtype"], page_size=PAGE, cache_tokens=case["requests"] * (most + PAGE) + 256,
            max_requests=case["requests"], max_step_tokens=sum(self.lengths), max_seq_len=most))

    def run(self):
        """All prompts in one step, then one token a request and step; the logits of every step."""
        names = list(range(len(self.ids)))
        step = self.engine.step
        kept = [step([(i, self.ids[i][:n], [n - 1]) for i, n in zip(names, self.lengths)]).clone()]
        for t in range(self.steps):
            entries = [(i, [self.ids[i][n + t]], [0]) for i, n in zip(names, self.lengths)]
            kept.append(step(entries, end=names if t == self.steps - 1 else ()).clone())
        return kept


def prepare(case, seed):
    return _ReplayState(case, seed) if case["kind"] == "replay" else _PartState(case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _seen(case):
    """(query, key) pairs of one head, and keys that are read, over all requests."""
    s, c, t = SIZES[case["size"]], case["context"], case["tokens"]
    pairs = 0
    for p in range(c, c + t):
        if case["kind"] == "gqa" and s["window"]:
            pairs += min(p + 1, s["window"])
        elif case["kind"] == "diff":
            pairs += p % (s["window"] or 8192) + 1
        else:
            pairs += p + 1
    return case["requests"] * pairs, case["requests"] * (c - _live(case) + t)


def work(case):
    s, kind, b = SIZES[case["size"]], case["kind"], 4 if case["dtype"] == "float32" else 2
    w, H, G, n = s["w"], s["H"], s["G"], case["requests"] * case["tokens"]
    rows = n * w * (b + 4)                                              # normalised rows in, the float32 delta out
    if kind == "replay":
        layer = w * HD * (2 * H + 2 * G) + 3 * w * s["ff"]
        steps, n = 1 + case["steps"], n + case["requests"] * case["steps"]
        return dict(bytes=steps * (REPLAY_LAYERS * layer + w * VOCAB) * b,
                    flops=2.0 * n * REPLAY_LAYERS * layer + 2.0 * steps * case["requests"] * w * VOCAB)
    if kind == "mlp":
        return dict(bytes=3 * w * s["ff"] * b + rows, flops=6.0 * n * w * s["ff"])
    if kind == "experts":
        distinct = s["E"] * (1.0 - (1.0 - s["K"] / s["E"]) ** n)
        return dict(bytes=(2 * distinct * w * s["eff"] + 2 * w * s["sff"] + w * s["E"]) * b + rows,
                    flops=4.0 * n * w * (s["K"] * s["eff"] + s["sff"]) + 2.0 * n * w * s["E"])
    if kind in STATEFUL:
        Gq = G if kind == "delta" else H
        maps = w * HD * (2 * Gq + 2 * H + (H if kind != "channel_delta" else 0)) + w * 2 * H
        if kind == "channel_delta":
            maps += 2 * w * RANK + 2 * H * HD * RANK
        return dict(bytes=maps * b + rows + 2 * case["requests"] * H * HD * HD * 4, flops=2.0 * n * maps + 7.0 * n * H * HD * HD)
    pairs, keys = _seen(case)
    if kind == "latent":
        maps = w * (2 * H * HD + LATENT) + 2 * H * HD * LATENT
        return dict(bytes=maps * b + rows + (keys + n) * LATENT * b, flops=2.0 * n * maps + 4.0 * pairs * H * LATENT)
    maps = w * HD * (2 * H + 2 * G)
    # (differential attention has two score maps of half the size, and both weigh the values)
    per_pair = 4.0 * HD if kind == "gqa" else 2.0 * HD + 4.0 * HD
    return dict(bytes=maps * b + rows + (keys + n) * 2 * G * HD * b, flops=2.0 * n * maps + per_pair * pairs * H)


def tolerance(case):
    # Measured against the 64-bit results: 2.9e-6 in 32 bits; 0.0017 to 0.0043 for one part in 16 bits and 0.016 for the
    # logits of a whole model, whose roundings travel through all layers.  Stated: about four times that (the whole model:
    # what two such results lie apart).
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5, "max": 1e-3}
    if case["kind"] == "replay":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 1.5e-2, "max": 0.15}


# ---- the same in 64 bits, from the formulas -------------------------------------------------------------------------
F64 = torch.float64


def _over_rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turn(x, first, theta):
    """x [n, heads, d] at positions first, first + 1, ...: dimension i is turned together with i + d / 2."""
    n, d = x.shape[0], x.shape[-1]
    f = torch.tensor([theta ** (-2.0 * i / d) for i in range(d // 2)], dtype=F64, device=x.device)
    a = (torch.arange(first, first + n, dtype=F64, device=x.device)[:, None] * f)[:, None]
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _weights_of(q, k, first_q, first_k, scale, window=0, sink=None):
    """Softmax weights [n, keys] of one head."""
    i = torch.arange(first_q, first_q + q.shape[0], device=q.device)[:, None]
    j = torch.arange(first_k, first_k + k.shape[0], device=q.device)[None]
    seen = (j <= i) & ((i - j < window) if window else (j >= 0))
    z = ((q @ k.T) * scale).masked_fill(~seen, -math.inf)
    top = z.max(-1, keepdim=True).values
    if sink is not None:
        top = torch.maximum(top, sink)
    z = torch.exp(z - top)
    return z / (z.sum(-1, keepdim=True) + (torch.exp(sink - top) if sink is not None else 0.0))


def _exact_attention(case, seed, W, h, i):
    """The mixer's output for request i's rows h."""
    s, kind, context = SIZES[case["size"]], case["kind"], case["context"]
    H, G, n, first = s["H"], s["G"], h.shape[0], _live(case)
    kc, vc = (t[i].to(F64) for t in _context(case, seed))
    heads = []
    if kind == "gqa":
        q = _turn((h @ W("mix.q_proj.weight", (H * HD, s["w"])).T).view(n, H, HD), context, 10000.0)
        k = _turn((h @ W("mix.k_proj.weight", (G * HD, s["w"])).T).view(n, G, HD), context, 10000.0)
        k, v = torch.cat([kc, k]), torch.cat([vc, (h @ W("mix.v_proj.weight", (G * HD, s["w"])).T).view(n, G, HD)])
        for x in range(H):
            g = x // (H // G)
            heads.append(_weights_of(q[:, x], k[:, g], context, first, HD ** -0.5, s["window"]) @ v[:, g])
        return torch.cat(heads, -1) @ W("mix.o_proj.weight", (s["w"], H * HD)).T
    if kind == "latent":
        c = _over_rms(h @ W("mix.dkv", (LATENT, s["w"])).T) * W("mix.dkv.norm", (LATENT,))
        c = torch.cat([kc[:, 0], c])
        q = (h @ W("mix.q", (H * HD, s["w"])).T).view(n, H, HD)
        uk, uv = (W("mix." + t, (H * HD, LATENT)).view(H, HD, LATENT) for t in ("uk", "uv"))
        sink = W("mix.sink", (H,))
        for x in range(H):
            p = _weights_of(q[:, x] @ uk[x], c, context, first, HD ** -0.5, sink=sink[x])
            heads.append((p @ c) @ uv[x].T)
        return torch.cat(heads, -1) @ W("mix.o", (s["w"], H * HD)).T
    d, chunk = HD // 2, s["window"] or 8192
    q = (h @ W("mix.q", (H * HD, s["w"])).T + W("mix.q.b", (H * HD,))).view(n, 2 * H, d)
    k = (h @ W("mix.k", (G * HD, s["w"])).T + W("mix.k.b", (G * HD,))).view(n, 2 * G, d)
    v = (h @ W("mix.v", (G * HD, s["w"])).T + W("mix.v.b", (G * HD,))).view(n, G, HD)
    q = _turn(_over_rms(q) * W("mix.q.norm", (d,)), context, 1e6)
    k = _turn(_over_rms(k) * W("mix.k.norm", (d,)), context, 1e6)
    k, v = torch.cat([kc.reshape(-1, 2 * G, d), k]), torch.cat([vc, v])
    lam = float(torch.exp((W("mix.lq1", (d,)) * W("mix.lk1", (d,))).sum())
                - torch.exp((W("mix.lq2", (d,)) * W("mix.lk2", (d,))).sum())) + DIFF
    out = []
    starts = sorted({context} | {p for p in range(context, context + n) if p % chunk == 0})
    for x in range(H):
        g, rows = x // (H // G), []
        for a, b in zip(starts, starts[1:] + [context + n]):          # the rows of one chunk see that chunk's keys
            f = max(first, a // chunk * chunk)
            m = [_weights_of(q[a - context:b - context, 2 * x + j], k[f - first:b - first, 2 * g + j], a, f, d ** -0.5)
                 @ v[f - first:b - first, g] for j in (0, 1)]
            rows.append(_over_rms(m[0] - lam * m[1]) * (1.0 - DIFF))
        out.append(torch.cat(rows))
    return torch.cat(out, -1) @ W("mix.o", (s["w"], H * HD)).T


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_recurrence(case, W, h):
    """The mixer's output for one request's rows from a zero state, and the state [H, dk, dv] behind them."""
    s, kind = SIZES[case["size"]], case["kind"]
    H, n, w = s["H"], h.shape[0], s["w"]
    Gq = s["G"] if kind == "delta" else H
    beta = None
    if kind == "linear":
        q, k, v = ((h @ W("mix." + t, (H * HD, w)).T).view(n, H, HD) for t in "qkv")
        q = q * HD ** -0.5
        z = (h @ W("mix.a1", (16, w)).T) @ W("mix.a2", (H * HD, 16)).T + W("mix.a2.b", (H * HD,))
        decay = torch.sigmoid(z).pow(1.0 / TAU).view(n, H, HD)
        gate = _silu(h @ W("mix.g", (H * HD, w)).T).view(n, H, HD)
    else:
        def conv(name, heads):
            x, taps = h @ W(f"mix.{name}", (heads * HD, w)).T, W(f"mix.{name}.conv", (heads * HD, TAPS))
            x = torch.cat([x.new_zeros(TAPS - 1, x.shape[1]), x])
            return _silu(sum(x[j:j + n] * taps[:, j] for j in range(TAPS))).view(n, heads, HD)

        def unit(x):
            return x / torch.sqrt((x * x).sum(-1, keepdim=True) + EPS)
        q, k = unit(conv("q", Gq)) * HD ** -0.5, unit(conv("k", Gq))
        q, k = (t.repeat_interleave(H // Gq, 1) for t in (q, k))
        v = conv("v", H)
        beta = torch.sigmoid(h @ W("mix.b", (H, w)).T)
        rate = torch.exp(W("mix.A_log", (H,)))
        if kind == "delta":
            z = (h @ W("mix.a", (H, w)).T + W("mix.dt_bias", (H,)))[..., None]
            gate = _silu(h @ W("mix.g", (H * HD, w)).T).view(n, H, HD)
        else:
            z = ((h @ W("mix.a1", (RANK, w)).T) @ W("mix.a2", (H * HD, RANK)).T + W("mix.dt_bias", (H * HD,))).view(n, H, HD)
            gate = torch.sigmoid((h @ W("mix.g1", (RANK, w)).T) @ W("mix.g2", (H * HD, RANK)).T).view(n, H, HD)
        decay = torch.exp(-rate[:, None] * torch.nn.functional.softplus(z, threshold=40.0))
    S, out = h.new_zeros(H, HD, HD), []
    for t in range(n):
        S = S * decay[t][..., None]
        u = v[t]
        if beta is not None:
            u = beta[t][:, None] * (u - (k[t][:, None] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][..., None], u[:, None])
        out.append((q[t][:, None] @ S)[:, 0])
    o = _over_rms(torch.stack(out)) * W("mix.norm", (HD,)) * gate
    return o.reshape(n, H * HD) @ W("mix.o", (w, H * HD)).T, S


def _exact_experts(s, W, h):
    z = h @ W("mlp.router", (s["E"], s["w"])).T
    best = z.topk(s["K"], -1)
    share = torch.softmax(best.values, -1)
    act = lambda x: torch.relu(x).square()  # noqa: E731
    out = act(h @ W("mlp.shared.up", (s["sff"], s["w"])).T) @ W("mlp.shared.down", (s["w"], s["sff"])).T
    out = out * torch.sigmoid(h @ W("mlp.shared.sg", (1, s["w"])).T)
    for e in range(s["E"]):
        rows, place = (best.indices == e).nonzero(as_tuple=True)
        if rows.numel():
            y = act(h[rows] @ W(f"mlp.e{e}.up", (s["eff"], s["w"])).T) @ W(f"mlp.e{e}.down", (s["w"], s["eff"])).T
            out.index_add_(0, rows, y * share[rows, place][:, None])
    return out


def _exact_mlp(W, h, p, w, ff):
    a = _silu(h @ W(p + "gate_proj.weight", (ff, w)).T) * (h @ W(p + "up_proj.weight", (ff, w)).T)
    return a @ W(p + "down_proj.weight", (w, ff)).T


def _exact_replay(case, seed, W):
    s = SIZES[case["size"]]
    w, H, G = s["w"], s["H"], s["G"]
    ids, lengths = _replay_tokens(case, seed)
    table = W("model.embed_tokens.weight", (VOCAB, w))
    xs = [table[torch.tensor(i[:-1] + i[-1:], device="cuda")] for i in ids]

    def norm(x, name):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * W(name, (w,))
    for layer in range(REPLAY_LAYERS):
        p = f"model.layers.{layer}."
        for r, x in enumerate(xs):
            n, h = x.shape[0], norm(x, p + "input_layernorm.weight")
            q = _turn((h @ W(p + "self_attn.q_proj.weight", (H * HD, w)).T).view(n, H, HD), 0, 10000.0)
            k = _turn((h @ W(p + "self_attn.k_proj.weight", (G * HD, w)).T).view(n, G, HD), 0, 10000.0)
            v = (h @ W(p + "self_attn.v_proj.weight", (G * HD, w)).T).view(n, G, HD)
            a = [_weights_of(q[:, i], k[:, i // (H // G)], 0, 0, HD ** -0.5, s["window"]) @ v[:, i // (H // G)] for i in range(H)]
            x = x + torch.cat(a, -1) @ W(p + "self_attn.o_proj.weight", (w, H * HD)).T
            xs[r] = x + _exact_mlp(W, norm(x, p + "post_attention_layernorm.weight"), p + "mlp.", w, s["ff"])
    head = W("lm_head.weight", (VOCAB, w))
    logits = [norm(x[n - 1:], "model.norm.weight") @ head.T for x, n in zip(xs, lengths)]
    return [torch.stack([l[t] for l in logits]) for t in range(case["steps"] + 1)]


def exact(case, seed):
    s, dt, kept = SIZES[case["size"]], _dtype(case), {}

    def W(name, shape):
        if name not in kept:
            if len(kept) > 12:                     # (float64 weights of a whole model need not all be held at once)
                kept.clear()
            kept[name] = _weight(seed, name, shape, dt).to(F64)
        return kept[name]
    if case["kind"] == "replay":
        return _exact_replay(case, seed, W)
    h, n = _rows(case, seed).to(F64), case["tokens"]
    pools, state = [], []
    if case["kind"] == "mlp":
        out = _exact_mlp(W, h, "mlp.", s["w"], s["ff"])
    elif case["kind"] == "experts":
        out = _exact_experts(s, W, h)
    else:
        outs, states = [], []
        for i in range(case["requests"]):
            rows = h[i * n:(i + 1) * n]
            if case["kind"] in CACHED:
                outs.append(_exact_attention(case, seed, W, rows, i))
            else:
                o, S = _exact_recurrence(case, W, rows)
                outs.append(o)
                states.append(S.transpose(1, 2).reshape(-1))        # (a slot keeps a value dimension's keys side by side)
        out = torch.cat(outs)
        if states:
            state = [torch.stack(states), None]
        else:
            pools = [None] * (1 if case["kind"] == "latent" else 2)
    return dict(out=out, pools=pools, state=state)
