"""The work that is measured: what programs over this framework have it do.

Whole steps of a Llama decoder through ``StepRunner`` (a prompt, a decode step replayed from its CUDA
graph, a prompt in 32-bit), and single mixers and feed-forwards through ``Part.forward``, as a model's
blocks call them. Sizes are those of ``bench.py`` (the TinyLlama-1.1B, Llama-2-7B and Llama-3-8B shapes
and the "2k" and "4k" sizes of the other designs). Steps in which every request brings one token are
replayed from a CUDA graph, as the engine does.

``exact`` computes each case in 64 bits with plain torch, from the same (bfloat16 or 32-bit) weights
and inputs and without rounding in between.
"""
import functools
import math

import torch

DEVICE = "cuda:0"
PAGE = 32

SHAPES = {
    "tinyllama": dict(layers=22, width=2048, heads=32, kv_heads=4, dim=64, ff=5632, vocab=32000, theta=10000.0),
    "llama2-7b": dict(layers=32, width=4096, heads=32, kv_heads=32, dim=128, ff=11008, vocab=32000, theta=10000.0),
    "llama3-8b": dict(layers=32, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=128256, theta=500000.0),
}
# per size: latent attention; capped attention (a_); the delta rules (d_, g_); the state space (s_); experts
SIZES = {
    "2k": dict(width=2048, heads=32, dim=32, rot_dim=32, vdim=64, kv_rank=256, scale=0.125, a_heads=32, a_kv=4, a_dim=64,
               d_heads=16, d_kv=16, rank=64, g_heads=32, g_dim=64, s_heads=64, s_groups=8, experts=16, top=4, expert_ff=1408),
    "4k": dict(width=4096, heads=32, dim=64, rot_dim=64, vdim=128, kv_rank=512, scale=0.088, a_heads=32, a_kv=8, a_dim=128,
               d_heads=32, d_kv=16, rank=128, g_heads=32, g_dim=128, s_heads=128, s_groups=8, experts=16, top=4, expert_ff=2752),
}
D_DIM, TAPS, WINDOW, KEEP, CAP = 128, 4, 1024, 4, 30.0
S_VDIM, S_STATE = 64, 128
DECAY_SCALE = math.exp(-0.5)
EPS = 1e-5


def listed():
    return [
        # the engine's headline: eight conversations at 2,048 positions, one token each
        dict(name="llama decode 8 at 2048", kind="decode", shape="tinyllama", requests=8, context=2048),
        # a prompt as long as the model's context, in one step
        dict(name="llama prompt 2048", kind="prompt", shape="tinyllama", layers=22, tokens=2048, requests=1, dtype="bfloat16"),
        # the 32-bit mode (checks of a checkpoint, trace replays): two prompts in one step
        dict(name="llama prompt 500, 32-bit", kind="prompt", shape="tinyllama", layers=2, tokens=500, requests=2, dtype="float32"),
        # continuous batching in a wide model: prompt portions of several requests behind what is cached already
        dict(name="attention, three portions", kind="attention", shape="llama3-8b", tokens=1221, requests=3, past=3001),
        # a feed-forward of a step that carries a few hundred tokens
        dict(name="feed-forward 333", kind="feed_forward", shape="llama3-8b", tokens=333),
        # the smallest step of a model with experts: eight decoded tokens, replayed
        dict(name="experts 8", kind="experts", size="2k", tokens=8, requests=8),
        # prompts through the mixers of the other designs
        dict(name="latent attention 2048", kind="latent", size="2k", tokens=2048, requests=1, past=0),
        dict(name="capped attention 2048", kind="capped", size="2k", tokens=2048, requests=1, past=0),
        dict(name="channel delta rule 2048", kind="channel_delta", size="2k", tokens=2048, requests=1),
        # ragged: four requests, among them the end of one that is a few dozen tokens
        dict(name="head delta rule, four prompts", kind="head_delta", size="4k", tokens=1511, requests=4),
        dict(name="general delta rule 2048", kind="general_delta", size="2k", tokens=2048, requests=1),
        dict(name="state space 2048", kind="state_space", size="2k", tokens=2048, requests=1),
    ]


def draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["decode", "prompt", "prompt32", "attention", "feed_forward", "experts", "latent", "capped",
                       "channel_delta", "head_delta", "general_delta", "state_space"])
    if kind == "decode":
        return dict(kind=kind, shape="tinyllama", requests=spread(1, 16), context=spread(32, 2048))
    if kind == "prompt":
        tokens = spread(2, 2048)
        return dict(kind=kind, shape="tinyllama", layers=22, tokens=tokens, requests=min(rng.randint(1, 4), tokens), dtype="bfloat16")
    if kind == "prompt32":
        tokens = spread(2, 480)
        return dict(kind="prompt", shape="tinyllama", layers=2, tokens=tokens, requests=min(rng.randint(1, 4), tokens), dtype="float32")
    tokens = spread(2, 2048)
    requests = min(rng.randint(1, 4), tokens)
    if kind == "attention":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), tokens=tokens, requests=requests, past=rng.choice([0, spread(1, 4096)]))
    if kind == "feed_forward":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), tokens=tokens)
    if kind in ("latent", "capped"):
        return dict(kind=kind, size=rng.choice(sorted(SIZES)), tokens=tokens, requests=requests, past=rng.choice([0, spread(1, 2048)]))
    return dict(kind=kind, size=rng.choice(sorted(SIZES)), tokens=tokens, requests=requests)


def prepare(case, seed):
    return _KINDS[case["kind"]](case, seed).ready()


def run(state):
    return state.run()


def exact(case, seed):
    with torch.no_grad():
        return _KINDS[case["kind"]](case, seed).exact()


def work(case):
    return _KINDS[case["kind"]](case, 0).work()


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 2e-5, "max": 8e-4}           # 4e-6 off ``exact``
    # bfloat16 operands: 2e-3 to 4e-3 off ``exact`` for a layer, 2e-2 behind 22 layers
    return {"rel": 0.03, "max": 0.6} if case["kind"] in ("decode", "prompt") else {"rel": 0.015, "max": 0.4}


# ------------------------------------------------------------------------------------------- common ground
class _Draws:
    """Values on the device from a seed, each call's own."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(*shape, generator=self.g, device=DEVICE) * std + mean).to(dtype)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(*shape, generator=self.g, device=DEVICE) * (high - low) + low

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.g, device=DEVICE).tolist()


@functools.lru_cache(maxsize=None)
def _kernels(dtype):
    """The kernel set that a program keeps: one per compute dtype."""
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps(DEVICE, tensor_cores=dtype == torch.bfloat16)


def _lengths(tokens, requests):
    """The step's tokens split unevenly: 1 : 3 : 5 : ... , at least one each."""
    out = [max(1, tokens * (2 * i + 1) // (requests * requests)) for i in range(requests - 1)]
    return out + [tokens - sum(out)]


def _f64(t):
    return t.double()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _step_times(lengths, fn):
    """Walks several requests' tokens side by side: ``fn(rows, members)`` for the k-th token of every request that has one."""
    first = [sum(lengths[:i]) for i in range(len(lengths))]
    for k in range(max(lengths)):
        members = [r for r, n in enumerate(lengths) if k < n]
        fn(torch.tensor([first[r] + k for r in members], device=DEVICE), torch.tensor(members, device=DEVICE))


class _Part:
    """One part, called as a model's block calls it: ``forward`` on the step's normed input, its output in 32-bit. ``past``: what
    its cache holds of every request before the step (a recurrent part starts every pass from the state a new request
    has, unless the step decodes: then the state goes on from pass to pass)."""
    registry, name = "mixer", ""

    def __init__(self, case, seed):
        self.case = case
        self.z = dict(SHAPES[case["shape"]]) if "shape" in case else dict(SIZES[case["size"]])
        self.tokens, self.requests, self.past = case["tokens"], case.get("requests", 1), case.get("past", 0)
        self.lengths = _lengths(self.tokens, self.requests)
        self.decodes = self.tokens == self.requests and "requests" in case
        self.dtype = torch.bfloat16
        self.seed = seed

    def draw_all(self):
        d = _Draws(self.seed)
        self.h = d.normal(self.tokens, self.z["width"], dtype=self.dtype)
        self.weights = self.draw_weights(d)
        # pages in an order of their own
        self.pages_each = [(self.past + n + PAGE - 1) // PAGE for n in self.lengths]
        total = sum(self.pages_each)
        order = torch.randperm(total, generator=d.g, device=DEVICE).to(torch.int32)
        self.table = torch.full((self.requests, max(self.pages_each)), -1, dtype=torch.int32, device=DEVICE)
        at = 0
        for r, n in enumerate(self.pages_each):
            self.table[r, :n] = order[at:at + n]
            at += n
        self.pools = self.draw_pools(d, total)

    def draw_pools(self, d, pages):
        return None

    def matrix(self, d, *shape, std=0.02):
        return d.normal(*shape, std=std, dtype=self.dtype)

    def ready(self):
        from garuda_b200.engine.batch import StepBatch, StepContext, Workspace
        from garuda_b200.parts import LayerCache, PartSpec, build_part
        self.draw_all()
        ops = _kernels(self.dtype)
        self.part = build_part(self.registry, PartSpec(self.name, self.params()))
        self.part.load(self.weights, ops, self.dtype)
        self.weights = None
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEVICE)
        cu = [sum(self.lengths[:i]) for i in range(self.requests + 1)]
        batch = StepBatch(
            num_tokens=self.tokens, num_requests=self.requests, token_ids=i32([0] * self.tokens),
            positions=i32([self.past + k for n in self.lengths for k in range(n)]),
            token_req=i32([r for r, n in enumerate(self.lengths) for _ in range(n)]), cu_q=i32(cu),
            kv_lens=i32([self.past + n for n in self.lengths]), slots=i32(list(range(self.requests))), block_tables=[self.table],
            logit_rows=i32([]), num_logit_rows=0, max_q_len=max(self.lengths), max_kv_len=self.past + max(self.lengths),
            min_q_len=min(self.lengths))
        self.ctx = StepContext(batch=batch, ws=Workspace(torch.device(DEVICE)), ops=ops, dtype=self.dtype)
        self.cache = None
        if self.registry == "mixer":
            need = self.part.cache_need()
            if self.pools is not None:
                self.cache = LayerCache(need=need, k=self.pools[0], v=self.pools[1] if len(self.pools) > 1 else None,
                                        block_table=self.table, page_size=PAGE)
            else:
                self.state = torch.zeros(self.requests, *need.shape, dtype=need.dtype, device=DEVICE)
                self.cache = LayerCache(need=need, state=self.state)
        self.graph = None
        if self.decodes:
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                self.call()                      # tables and scratch that are made on first use
            torch.cuda.current_stream().wait_stream(stream)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                self.out = self.call()
            self.graph = graph
            if self.pools is None and self.cache is not None:
                self.state.zero_()
        return self

    def call(self):
        args = (self.ctx, self.h) + ((self.cache,) if self.registry == "mixer" else ())
        self.ctx.step_cache.clear()
        return self.part.forward(*args)

    def run(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            if self.cache is not None and self.pools is None:
                self.state.zero_()               # every request starts: its state is that of no tokens
            self.out = self.call()
        if self.cache is None:
            return self.out
        if self.pools is None:
            return {"y": self.out, "state": self.state}
        return {"y": self.out, "cache": list(self.pools)}

    # pages in 64 bits: rows of a request's positions, and back
    def gather(self, pool, r):
        pages = self.table[r, :self.pages_each[r]].long()
        rows = pool[pages].transpose(1, 2).reshape(len(pages) * PAGE, pool.shape[1], pool.shape[3])
        return rows[:self.past + self.lengths[r]]

    def scatter(self, pool, r, rows):
        positions = torch.arange(self.past, self.past + self.lengths[r], device=DEVICE)
        pool[self.table[r].long()[positions // PAGE], :, positions % PAGE] = rows

    def rows_of(self, r):
        first = sum(self.lengths[:r])
        return slice(first, first + self.lengths[r])


def _attend(q, k, v, scale, first, window=0, keep=0, cap=0.0):
    """q [n, H, d] at positions first .., k and v [m, G, .] from position 0, in 64 bits: [n, H, vdim]."""
    n, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=torch.float64, device=q.device)
    j = torch.arange(k.shape[0], device=q.device)
    for lo in range(0, n, 512):
        i = first + torch.arange(lo, min(lo + 512, n), device=q.device)
        seen = j[None, :] <= i[:, None]
        if window:
            seen &= (i[:, None] - j[None, :] < window) | (j[None, :] < keep)
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("nhd,md->hnm", q[lo:lo + 512, heads], k[:, g]) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~seen, -math.inf).softmax(-1)
            out[lo:lo + 512, heads] = torch.einsum("hnm,md->nhd", s, v[:, g])
    return out


def _turn(x, positions, freqs, neighbours):
    """Rotates [n, heads, 2 * len(freqs)]: pairs (2i, 2i + 1), or (i, i + half)."""
    angle = positions.double()[:, None, None] * freqs
    c, s = angle.cos(), angle.sin()
    if neighbours:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    half = len(freqs)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _seen_keys(lengths, past, window=0, keep=0):
    total = 0
    for n in lengths:
        for i in range(past, past + n):
            total += i + 1 if not window or i + 1 <= window else window + min(keep, i + 1 - window)
    return total


# ------------------------------------------------------------------------------------------- Llama, whole
class _Llama:
    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.z = dict(SHAPES[case["shape"]])
        self.z["layers"] = case.get("layers", self.z["layers"])
        self.dtype = getattr(torch, case.get("dtype", "bfloat16"))

    def names(self):
        z = self.z
        w, q, kv = z["width"], z["heads"] * z["dim"], z["kv_heads"] * z["dim"]
        out = {"model.embed_tokens.weight": (z["vocab"], w), "lm_head.weight": (z["vocab"], w), "model.norm.weight": (w,)}
        for l in range(z["layers"]):
            p = f"model.layers.{l}."
            out.update({p + "self_attn.q_proj.weight": (q, w), p + "self_attn.k_proj.weight": (kv, w),
                        p + "self_attn.v_proj.weight": (kv, w), p + "self_attn.o_proj.weight": (w, q),
                        p + "mlp.gate_proj.weight": (z["ff"], w), p + "mlp.up_proj.weight": (z["ff"], w),
                        p + "mlp.down_proj.weight": (w, z["ff"]), p + "input_layernorm.weight": (w,),
                        p + "post_attention_layernorm.weight": (w,)})
        return out

    def draw_weights(self):
        d = _Draws(self.seed)
        out = {n: d.normal(*s, std=0.02, dtype=self.dtype) if len(s) == 2 else d.normal(*s, std=0.1, mean=1.0)
               for n, s in self.names().items()}
        return d, out

    def build(self, max_requests, max_positions, kv_tokens):
        """The runner that ``Engine`` makes, over weights that are on the device already."""
        from garuda_b200 import StepRunner
        from garuda_b200.cache.manager import CacheConfig, PagedCache
        from garuda_b200.config.registry import build_model
        z = self.z
        _, model = build_model(dict(
            architectures=["LlamaForCausalLM"], model_type="llama", rms_norm_eps=EPS, tie_word_embeddings=False,
            hidden_size=z["width"], num_hidden_layers=z["layers"], num_attention_heads=z["heads"],
            num_key_value_heads=z["kv_heads"], head_dim=z["dim"], intermediate_size=z["ff"], vocab_size=z["vocab"],
            rope_theta=z["theta"], max_position_embeddings=max_positions))
        d, weights = self.draw_weights()
        ops = _kernels(self.dtype)
        model.load(weights, ops, self.dtype)
        cache = PagedCache(model, CacheConfig(page_size=PAGE, max_tokens=kv_tokens, max_requests=max_requests,
                                              max_positions=max_positions), self.dtype, DEVICE)
        return d, StepRunner(model, cache, ops, self.dtype, DEVICE)

    def exact_logits(self, weights, sequences):
        """Logits at each sequence's last position; one list of token ids per request."""
        z, w = self.z, weights
        freqs = torch.tensor([z["theta"] ** (-2.0 * i / z["dim"]) for i in range(z["dim"] // 2)], dtype=torch.float64, device=DEVICE)
        lengths = [len(s) for s in sequences]
        ids = torch.tensor([t for s in sequences for t in s], device=DEVICE)
        x = _f64(w["model.embed_tokens.weight"])[ids]
        where = torch.cat([torch.arange(n, device=DEVICE) for n in lengths])
        for l in range(z["layers"]):
            p = f"model.layers.{l}."
            m = lambda name: _f64(w[p + name])
            h = _rms(x, EPS) * m("input_layernorm.weight")
            q = _turn((h @ m("self_attn.q_proj.weight").T).unflatten(1, (z["heads"], z["dim"])), where, freqs, False)
            k = _turn((h @ m("self_attn.k_proj.weight").T).unflatten(1, (z["kv_heads"], z["dim"])), where, freqs, False)
            v = (h @ m("self_attn.v_proj.weight").T).unflatten(1, (z["kv_heads"], z["dim"]))
            at, mixed = 0, []
            for n in lengths:
                mixed.append(_attend(q[at:at + n], k[at:at + n], v[at:at + n], z["dim"] ** -0.5, 0))
                at += n
            x = x + torch.cat(mixed).flatten(1) @ m("self_attn.o_proj.weight").T
            h = _rms(x, EPS) * m("post_attention_layernorm.weight")
            act = torch.nn.functional.silu(h @ m("mlp.gate_proj.weight").T) * (h @ m("mlp.up_proj.weight").T)
            x = x + act @ m("mlp.down_proj.weight").T
        ends = torch.tensor(lengths, device=DEVICE).cumsum(0) - 1
        return (_rms(x[ends], EPS) * _f64(w["model.norm.weight"])) @ _f64(w["lm_head.weight"]).T

    def layer_weights(self):
        z = self.z
        return z["width"] * z["dim"] * (2 * z["heads"] + 2 * z["kv_heads"]) + 3 * z["width"] * z["ff"]

    def work_of(self, tokens, rows, cached, scores):
        """``tokens`` run, ``rows`` of logits, ``cached`` positions read from the cache, ``scores`` query-key pairs per head."""
        z, item = self.z, self.dtype.itemsize
        weights = z["layers"] * self.layer_weights() + z["vocab"] * z["width"] + tokens * z["width"]
        kv = z["layers"] * 2 * z["kv_heads"] * z["dim"]
        flops = 2 * tokens * z["layers"] * self.layer_weights() + 2 * rows * z["vocab"] * z["width"] \
            + 4 * z["layers"] * z["heads"] * z["dim"] * scores
        return {"bytes": item * (weights + kv * (cached + tokens)) + 4 * rows * z["vocab"], "flops": flops}


class _Prompt(_Llama):
    """Prompts from their first token, in one step; logits at each one's last place."""

    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.lengths = _lengths(case["tokens"], case["requests"])

    def sequences(self, d):
        return [d.ids(n, self.z["vocab"]) for n in self.lengths]

    def ready(self):
        from garuda_b200 import StepEntry
        d, self.runner = self.build(len(self.lengths), 2048, sum(self.lengths) + PAGE * len(self.lengths))
        self.entries = [StepEntry(r, s, [len(s) - 1]) for r, s in enumerate(self.sequences(d))]
        return self

    def run(self):
        logits = self.runner.run(self.entries)
        for e in self.entries:
            self.runner.end(e.request)
        return logits

    def exact(self):
        d, w = self.draw_weights()
        return self.exact_logits(w, self.sequences(d))

    def work(self):
        return self.work_of(sum(self.lengths), len(self.lengths), 0, _seen_keys(self.lengths, 0))


class _Decode(_Llama):
    """One token for each of several requests; every pass is the next position."""
    AHEAD = 2048

    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.requests, self.context = case["requests"], case["context"]

    def tokens(self, d):
        return [d.ids(self.context + self.AHEAD, self.z["vocab"]) for _ in range(self.requests)]

    def fill(self):
        from garuda_b200 import StepEntry
        for r in range(self.requests):
            if self.at:
                self.runner.end(r)
            for lo in range(0, self.context - 1, 2048):
                self.runner.run([StepEntry(r, self.ids[r][lo:min(lo + 2048, self.context - 1)], [])])
        self.at = self.context - 1

    def ready(self):
        from garuda_b200.engine.graph import DecodeGraphs
        most = self.context + self.AHEAD
        d, self.runner = self.build(self.requests, most, self.requests * (most + PAGE))
        self.runner.graphs = DecodeGraphs(self.runner, self.requests)
        self.runner.graphs.warm()
        self.ids, self.at = self.tokens(d), 0
        self.fill()
        return self

    def run(self):
        from garuda_b200 import StepEntry
        if self.at == self.context + self.AHEAD:
            self.fill()
        logits = self.runner.run([StepEntry(r, [self.ids[r][self.at]], [0]) for r in range(self.requests)])
        self.at += 1
        return logits

    def exact(self):
        if self.requests * self.context > 20000:
            return None
        d, w = self.draw_weights()
        return self.exact_logits(w, [s[:self.context] for s in self.tokens(d)])

    def work(self):
        return self.work_of(self.requests, self.requests, self.requests * (self.context - 1), self.requests * self.context)


# ------------------------------------------------------------------------------------------- Llama, its parts
class _Attention(_Part):
    name = "paged_attention"

    def params(self):
        z = self.z
        return dict(width=z["width"], heads=z["heads"], kv_heads=z["kv_heads"], head_dim=z["dim"],
                    position={"name": "rotary", "params": {"theta": z["theta"], "head_dim": z["dim"]}})

    def draw_weights(self, d):
        z = self.z
        q, kv = z["heads"] * z["dim"], z["kv_heads"] * z["dim"]
        return {"q_proj.weight": self.matrix(d, q, z["width"]), "k_proj.weight": self.matrix(d, kv, z["width"]),
                "v_proj.weight": self.matrix(d, kv, z["width"]), "o_proj.weight": self.matrix(d, z["width"], q)}

    def draw_pools(self, d, pages):
        return [d.normal(pages, self.z["kv_heads"], PAGE, self.z["dim"], dtype=self.dtype) for _ in range(2)]

    def exact(self):
        self.draw_all()
        z, w, h = self.z, self.weights, _f64(self.h)
        freqs = torch.tensor([z["theta"] ** (-2.0 * i / z["dim"]) for i in range(z["dim"] // 2)], dtype=torch.float64, device=DEVICE)
        pools, mixed = [_f64(p) for p in self.pools], []
        for r, n in enumerate(self.lengths):
            hr, where = h[self.rows_of(r)], torch.arange(self.past, self.past + n, device=DEVICE)
            q = _turn((hr @ _f64(w["q_proj.weight"]).T).unflatten(1, (z["heads"], z["dim"])), where, freqs, False)
            k = _turn((hr @ _f64(w["k_proj.weight"]).T).unflatten(1, (z["kv_heads"], z["dim"])), where, freqs, False)
            self.scatter(pools[0], r, k)
            self.scatter(pools[1], r, (hr @ _f64(w["v_proj.weight"]).T).unflatten(1, (z["kv_heads"], z["dim"])))
            mixed.append(_attend(q, self.gather(pools[0], r), self.gather(pools[1], r), z["dim"] ** -0.5, self.past))
        return {"y": torch.cat(mixed).flatten(1) @ _f64(w["o_proj.weight"]).T, "cache": pools}

    def work(self):
        z = self.z
        weights = z["width"] * z["dim"] * (2 * z["heads"] + 2 * z["kv_heads"])
        row = 2 * z["kv_heads"] * z["dim"]
        return {"bytes": 2 * (weights + self.tokens * z["width"] + row * (self.requests * self.past + self.tokens)) + 4 * self.tokens * z["width"],
                "flops": 2 * self.tokens * weights + 4 * z["heads"] * z["dim"] * _seen_keys(self.lengths, self.past)}


class _FeedForward(_Part):
    registry, name = "feed_forward", "swiglu"

    def params(self):
        return dict(width=self.z["width"], inner=self.z["ff"])

    def draw_weights(self, d):
        z = self.z
        return {"gate_proj.weight": self.matrix(d, z["ff"], z["width"]), "up_proj.weight": self.matrix(d, z["ff"], z["width"]),
                "down_proj.weight": self.matrix(d, z["width"], z["ff"])}

    def exact(self):
        self.draw_all()
        w, h = self.weights, _f64(self.h)
        act = torch.nn.functional.silu(h @ _f64(w["gate_proj.weight"]).T) * (h @ _f64(w["up_proj.weight"]).T)
        return act @ _f64(w["down_proj.weight"]).T

    def work(self):
        z = self.z
        weights = 3 * z["width"] * z["ff"]
        return {"bytes": 2 * (weights + self.tokens * z["width"]) + 4 * self.tokens * z["width"], "flops": 2 * self.tokens * weights}


# ------------------------------------------------------------------------------------------- the other designs' parts
class _Experts(_Part):
    """Sixteen gated experts of which a token uses four, a softmax over the chosen ones."""
    registry, name = "feed_forward", "routed_experts"

    def params(self):
        z = self.z
        return dict(width=z["width"], experts=z["experts"], top=z["top"], inner=z["expert_ff"], limit=7.0)

    def draw_weights(self, d):
        z = self.z
        out = {"router": self.matrix(d, z["experts"], z["width"]), "router.b": d.normal(z["experts"], std=0.02)}
        for e in range(z["experts"]):
            out[f"e{e}.gate"], out[f"e{e}.up"] = (self.matrix(d, z["expert_ff"], z["width"]) for _ in range(2))
            out[f"e{e}.down"] = self.matrix(d, z["width"], z["expert_ff"])
        return out

    def exact(self):
        self.draw_all()
        z, w, h = self.z, self.weights, _f64(self.h)
        best, chosen = (h @ _f64(w["router"]).T + _f64(w["router.b"])).topk(z["top"], -1)
        share = best.softmax(-1)
        y = torch.zeros(self.tokens, z["width"], dtype=torch.float64, device=DEVICE)
        for e in range(z["experts"]):
            token, place = (chosen == e).nonzero(as_tuple=True)
            he = h[token]
            g, u = (he @ _f64(w[f"e{e}.gate"]).T).clamp(max=7.0), (he @ _f64(w[f"e{e}.up"]).T).clamp(-7.0, 7.0)
            out = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ _f64(w[f"e{e}.down"]).T
            y.index_add_(0, token, out * share[token, place][:, None])
        return y

    def work(self):
        z = self.z
        one = 3 * z["width"] * z["expert_ff"]
        used = z["experts"] * (1.0 - (1.0 - z["top"] / z["experts"]) ** self.tokens)     # experts that some token chose, on average
        return {"bytes": 2 * (used * one + z["experts"] * z["width"] + self.tokens * z["width"]) + 4 * self.tokens * z["width"],
                "flops": 2 * self.tokens * (z["top"] * one + z["experts"] * z["width"])}


class _Latent(_Part):
    """Attention over a cached latent that all heads share."""
    name = "latent_attention"

    def params(self):
        z = self.z
        return dict(width=z["width"], heads=z["heads"], dim=z["dim"], rot_dim=z["rot_dim"], vdim=z["vdim"], kv_rank=z["kv_rank"],
                    scale=z["scale"], eps=EPS)

    def draw_weights(self, d):
        z = self.z
        return {"q": self.matrix(d, z["heads"] * (z["dim"] + z["rot_dim"]), z["width"]),
                "dkv": self.matrix(d, z["kv_rank"] + z["rot_dim"], z["width"]), "dkv.norm": d.normal(z["kv_rank"], std=0.1, mean=1.0),
                "uk": self.matrix(d, z["heads"] * z["dim"], z["kv_rank"], std=0.06),
                "uv": self.matrix(d, z["heads"] * z["vdim"], z["kv_rank"], std=0.06),
                "o": self.matrix(d, z["width"], z["heads"] * z["vdim"])}

    def draw_pools(self, d, pages):
        return [d.normal(pages, 1, PAGE, self.z["kv_rank"] + self.z["rot_dim"], dtype=self.dtype)]

    def exact(self):
        self.draw_all()
        z, w, h = self.z, {n: _f64(t) for n, t in self.weights.items()}, _f64(self.h)
        dim, rot, rank, H = z["dim"], z["rot_dim"], z["kv_rank"], z["heads"]
        freqs = torch.tensor([10000.0 ** (-2.0 * i / rot) for i in range(rot // 2)], dtype=torch.float64, device=DEVICE)
        uk, uv = w["uk"].view(H, dim, rank), w["uv"].view(H, z["vdim"], rank)
        pool, mixed = _f64(self.pools[0]), []
        for r, n in enumerate(self.lengths):
            hr, where = h[self.rows_of(r)], torch.arange(self.past, self.past + n, device=DEVICE)
            q = (hr @ w["q"].T).unflatten(1, (H, dim + rot))
            c = hr @ w["dkv"].T
            row = torch.cat([_rms(c[:, :rank], EPS) * w["dkv.norm"], _turn(c[:, None, rank:], where, freqs, True)[:, 0]], -1)
            self.scatter(pool, r, row[:, None])
            kept = self.gather(pool, r)
            ql = torch.cat([torch.einsum("nhd,hdc->nhc", q[..., :dim], uk), _turn(q[..., dim:], where, freqs, True)], -1)
            lat = _attend(ql, kept, kept[..., :rank], z["scale"], self.past)
            mixed.append(torch.einsum("nhc,hvc->nhv", lat, uv).flatten(1))
        return {"y": torch.cat(mixed) @ w["o"].T, "cache": [pool]}

    def work(self):
        z = self.z
        H, rank, row = z["heads"], z["kv_rank"], z["kv_rank"] + z["rot_dim"]
        weights = z["width"] * (H * (z["dim"] + z["rot_dim"]) + row + H * z["vdim"]) + H * rank * (z["dim"] + z["vdim"])
        return {"bytes": 2 * (weights + self.tokens * z["width"] + row * (self.requests * self.past + self.tokens)) + 4 * self.tokens * z["width"],
                "flops": 2 * self.tokens * weights + 2 * H * (row + rank) * _seen_keys(self.lengths, self.past)}


class _Capped(_Part):
    """Attention without positions: capped scores, a window that keeps the first positions, a sink, biases."""
    name = "capped_sink_attention"

    def params(self):
        z = self.z
        return dict(width=z["width"], heads=z["a_heads"], kv_heads=z["a_kv"], dim=z["a_dim"], softcap=CAP, window=WINDOW,
                    keep_first=KEEP, sink=True, bias=True)

    def draw_weights(self, d):
        z = self.z
        q, kv = z["a_heads"] * z["a_dim"], z["a_kv"] * z["a_dim"]
        return {"q": self.matrix(d, q, z["width"]), "k": self.matrix(d, kv, z["width"]), "v": self.matrix(d, kv, z["width"]),
                "o": self.matrix(d, z["width"], q), "q.b": d.normal(q, std=0.02), "k.b": d.normal(kv, std=0.02), "v.b": d.normal(kv, std=0.02)}

    def draw_pools(self, d, pages):
        return [d.normal(pages, self.z["a_kv"], PAGE, self.z["a_dim"], dtype=self.dtype) for _ in range(2)]

    def exact(self):
        self.draw_all()
        z, w, h = self.z, {n: _f64(t) for n, t in self.weights.items()}, _f64(self.h)
        H, G, dim = z["a_heads"], z["a_kv"], z["a_dim"]
        pools, mixed = [_f64(p) for p in self.pools], []
        for r, n in enumerate(self.lengths):
            hr = h[self.rows_of(r)]
            q = (hr @ w["q"].T + w["q.b"]).unflatten(1, (H, dim))
            self.scatter(pools[0], r, (hr @ w["k"].T + w["k.b"]).unflatten(1, (G, dim)))
            self.scatter(pools[1], r, (hr @ w["v"].T + w["v.b"]).unflatten(1, (G, dim)))
            k, v = (self.gather(p, r) for p in pools)
            # the sink: a key whose score is zero and whose value is nothing
            i = torch.arange(self.past, self.past + n, device=DEVICE)[:, None]
            j = torch.arange(self.past + n, device=DEVICE)[None, :]
            seen = (j <= i) & ((i - j < WINDOW) | (j < KEEP))
            out = torch.empty(n, H, dim, dtype=torch.float64, device=DEVICE)
            for g in range(G):
                heads = slice(g * (H // G), (g + 1) * (H // G))
                s = CAP * torch.tanh(torch.einsum("nhd,md->hnm", q[:, heads], k[:, g]) * dim ** -0.5 / CAP)
                e = torch.exp(s - CAP).masked_fill(~seen, 0.0)
                p = e / (e.sum(-1, keepdim=True) + math.exp(-CAP))
                out[:, heads] = torch.einsum("hnm,md->nhd", p, v[:, g])
            mixed.append(out.flatten(1))
        return {"y": torch.cat(mixed) @ w["o"].T, "cache": pools}

    def work(self):
        z = self.z
        weights = z["width"] * z["a_dim"] * 2 * (z["a_heads"] + z["a_kv"])
        cached = self.requests * min(self.past, WINDOW + KEEP)
        return {"bytes": 2 * (weights + self.tokens * z["width"] + 2 * z["a_kv"] * z["a_dim"] * (cached + self.tokens)) + 4 * self.tokens * z["width"],
                "flops": 2 * self.tokens * weights + 4 * z["a_heads"] * z["a_dim"] * _seen_keys(self.lengths, self.past, WINDOW, KEEP)}


def _inverse_softplus(y):
    return y + torch.log(-torch.expm1(-y))


class _Recurrent(_Part):
    def conv(self, x, kernel, bias=None):
        """Causal convolution over time per channel of every request's rows, then SiLU, and the kept last inputs."""
        taps, out, kept = kernel.shape[1], [], []
        for r in range(self.requests):
            rows = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=x.dtype, device=x.device), x[self.rows_of(r)]])
            y = sum(rows[i:i + self.lengths[r]] * kernel[:, i] for i in range(taps))
            out.append(torch.nn.functional.silu(y if bias is None else y + bias))
            kept.append(rows[self.lengths[r]:].flatten())
        return torch.cat(out), torch.stack(kept)

    def step_sizes(self, d, *shape):
        """Biases whose softplus lies between 0.001 and 0.1, evenly over the logarithm, as such layers are initialized."""
        return _inverse_softplus(torch.exp(d.uniform(*shape, low=math.log(1e-3), high=math.log(0.1))))


class _Delta(_Recurrent):
    """The gated delta rule, with a decay per key channel or per head."""
    per_head = False
    name = "channel_delta_rule"

    def params(self):
        z = self.z
        more = {} if self.per_head else dict(decay_rank=z["rank"], gate_rank=z["rank"])
        return dict(width=z["width"], heads=z["d_heads"], kv_heads=z["d_kv"], dim=D_DIM, vdim=D_DIM, taps=TAPS, eps=EPS, **more)

    def draw_weights(self, d):
        z = self.z
        H, qk, v, m = z["d_heads"], z["d_kv"] * D_DIM, z["d_heads"] * D_DIM, self.matrix
        out = {"q": m(d, qk, z["width"]), "k": m(d, qk, z["width"]), "v": m(d, v, z["width"]), "b": m(d, H, z["width"]),
               "o": m(d, z["width"], v), "q.conv": d.normal(qk, TAPS, std=0.4), "k.conv": d.normal(qk, TAPS, std=0.4),
               "v.conv": d.normal(v, TAPS, std=0.4), "A_log": torch.log(d.uniform(H, low=1.0, high=16.0)),
               "norm": d.normal(D_DIM, std=0.1, mean=1.0), "dt_bias": self.step_sizes(d, H if self.per_head else v)}
        if self.per_head:
            out.update(a=m(d, H, z["width"]), g=m(d, v, z["width"]))
        else:
            out.update(a1=m(d, z["rank"], z["width"]), a2=m(d, H * D_DIM, z["rank"]), g1=m(d, z["rank"], z["width"]), g2=m(d, v, z["rank"]))
        return out

    def exact(self):
        self.draw_all()
        z, w, h = self.z, {n: _f64(t) for n, t in self.weights.items()}, _f64(self.h)
        H, G, T, F = z["d_heads"], z["d_kv"], self.tokens, torch.nn.functional
        act, kept = self.conv(torch.cat([h @ w[n].T for n in "qkv"], -1), torch.cat([w[n + ".conv"] for n in "qkv"]))
        q, k, v = act.split([G * D_DIM, G * D_DIM, H * D_DIM], -1)
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        q = (unit(q.view(T, G, D_DIM)) * D_DIM ** -0.5).repeat_interleave(H // G, 1)
        k = unit(k.view(T, G, D_DIM)).repeat_interleave(H // G, 1)
        v, beta = v.view(T, H, D_DIM), torch.sigmoid(h @ w["b"].T)
        pre = h @ w["a"].T if self.per_head else h @ w["a1"].T @ w["a2"].T
        rate = torch.exp(w["A_log"]) if self.per_head else torch.exp(w["A_log"]).repeat_interleave(D_DIM)
        decay = torch.exp(-rate * F.softplus(pre + w["dt_bias"])).view(T, H, -1)
        S, o = torch.zeros(self.requests, H, D_DIM, D_DIM, dtype=torch.float64, device=DEVICE), torch.empty_like(v)

        def token(rows, members):
            s = S[members] * decay[rows][..., None]
            u = beta[rows][..., None] * (v[rows] - torch.einsum("rhkv,rhk->rhv", s, k[rows]))
            s = s + k[rows][..., None] * u[..., None, :]
            S[members] = s
            o[rows] = torch.einsum("rhkv,rhk->rhv", s, q[rows])

        _step_times(self.lengths, token)
        if self.per_head:
            gate = F.silu(h @ w["g"].T)
        else:
            gate = torch.sigmoid(h @ w["g1"].T @ w["g2"].T)
        y = ((_rms(o, EPS) * w["norm"]).flatten(1) * gate) @ w["o"].T
        return {"y": y, "state": torch.cat([S.flatten(1), kept], -1)}

    def work(self):
        z = self.z
        H, qk, v = z["d_heads"], z["d_kv"] * D_DIM, z["d_heads"] * D_DIM
        weights = z["width"] * (2 * qk + 2 * v + H) + (z["width"] * (H + v) if self.per_head else z["rank"] * (2 * z["width"] + 2 * v))
        return {"bytes": 2 * (weights + self.tokens * z["width"]) + 4 * self.tokens * z["width"] + 8 * self.requests * H * D_DIM * D_DIM,
                "flops": self.tokens * (2 * weights + 7 * H * D_DIM * D_DIM)}


class _HeadDelta(_Delta):
    per_head = True
    name = "head_delta_rule"


class _GeneralDelta(_Recurrent):
    """The generalized delta rule: a decay and a removal rate per key channel."""
    name = "general_delta_rule"

    def params(self):
        z = self.z
        return dict(width=z["width"], heads=z["g_heads"], dim=z["g_dim"], eps=EPS, decay_scale=DECAY_SCALE, decay_rank=z["rank"])

    def draw_weights(self, d):
        z = self.z
        n, m = z["g_heads"] * z["g_dim"], self.matrix
        out = {name: m(d, n, z["width"]) for name in ("r", "k", "v", "a", "g")}
        # decays from a few tokens to a few hundred
        out.update({"a.b": d.normal(n, std=0.5), "w1": m(d, z["rank"], z["width"]), "w2": m(d, n, z["rank"], std=0.1),
                    "w0": d.uniform(n, low=-5.0, high=1.0), "norm": d.normal(n, std=0.1, mean=1.0), "o": m(d, z["width"], n)})
        return out

    def exact(self):
        self.draw_all()
        z, w, h = self.z, {n: _f64(t) for n, t in self.weights.items()}, _f64(self.h)
        H, D, T = z["g_heads"], z["g_dim"], self.tokens
        r, k, v = ((h @ w[n].T).view(T, H, D) for n in "rkv")
        decay = torch.exp(-DECAY_SCALE * torch.sigmoid(torch.tanh(h @ w["w1"].T) @ w["w2"].T + w["w0"])).view(T, H, D)
        a = torch.sigmoid(h @ w["a"].T + w["a.b"]).view(T, H, D)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, o = torch.zeros(self.requests, H, D, D, dtype=torch.float64, device=DEVICE), torch.empty_like(v)

        def token(rows, members):
            old = S[members]
            seen = torch.einsum("rhkv,rhk->rhv", old, u[rows])
            s = old * decay[rows][..., None] - (a[rows] * u[rows])[..., None] * seen[..., None, :] + k[rows][..., None] * v[rows][..., None, :]
            S[members] = s
            o[rows] = torch.einsum("rhkv,rhk->rhv", s, r[rows])

        _step_times(self.lengths, token)
        y = (_rms(o, EPS).flatten(1) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T
        return {"y": y, "state": S.flatten(1)}

    def work(self):
        z = self.z
        H, D = z["g_heads"], z["g_dim"]
        weights = 6 * z["width"] * H * D + z["rank"] * (z["width"] + H * D)
        return {"bytes": 2 * (weights + self.tokens * z["width"]) + 4 * self.tokens * z["width"] + 8 * self.requests * H * D * D,
                "flops": self.tokens * (2 * weights + 9 * H * D * D)}


class _StateSpace(_Recurrent):
    """The selective state space with one decay per head and token."""
    name = "state_space_duality"

    def params(self):
        z = self.z
        return dict(width=z["width"], heads=z["s_heads"], groups=z["s_groups"], state=S_STATE, vdim=S_VDIM, taps=TAPS, eps=EPS)

    def draw_weights(self, d):
        z = self.z
        H, inner = z["s_heads"], z["s_heads"] * S_VDIM
        channels = inner + 2 * z["s_groups"] * S_STATE
        return {"in": self.matrix(d, inner + channels + H, z["width"]), "conv": d.normal(channels, TAPS, std=0.4),
                "conv.b": d.normal(channels, std=0.1), "dt_bias": self.step_sizes(d, H), "A_log": torch.log(d.uniform(H, low=1.0, high=16.0)),
                "D": d.normal(H, std=0.3, mean=1.0), "norm": d.normal(inner, std=0.1, mean=1.0), "o": self.matrix(d, z["width"], inner)}

    def exact(self):
        self.draw_all()
        zz, w, h = self.z, {n: _f64(t) for n, t in self.weights.items()}, _f64(self.h)
        H, G, T, F = zz["s_heads"], zz["s_groups"], self.tokens, torch.nn.functional
        inner, gs = H * S_VDIM, G * S_STATE
        z, xbc, d = (h @ w["in"].T).split([inner, inner + 2 * gs, H], -1)
        act, kept = self.conv(xbc, w["conv"], w["conv.b"])
        x = act[:, :inner].view(T, H, S_VDIM)
        B, C = (act[:, inner + i * gs:inner + (i + 1) * gs].view(T, G, S_STATE).repeat_interleave(H // G, 1) for i in range(2))
        dt = F.softplus(d + w["dt_bias"])
        decay = torch.exp(-torch.exp(w["A_log"]) * dt)
        S, y = torch.zeros(self.requests, H, S_VDIM, S_STATE, dtype=torch.float64, device=DEVICE), torch.empty_like(x)

        def token(rows, members):
            s = S[members] * decay[rows][..., None, None] + (dt[rows][..., None] * x[rows])[..., None] * B[rows][..., None, :]
            S[members] = s
            y[rows] = torch.einsum("rhvs,rhs->rhv", s, C[rows]) + w["D"][:, None] * x[rows]

        _step_times(self.lengths, token)
        out = (_rms(y.flatten(1) * F.silu(z), EPS) * w["norm"]) @ w["o"].T
        return {"y": out, "state": torch.cat([S.flatten(1), kept], -1)}

    def work(self):
        z = self.z
        inner = z["s_heads"] * S_VDIM
        weights = z["width"] * (3 * inner + 2 * z["s_groups"] * S_STATE + z["s_heads"])
        return {"bytes": 2 * (weights + self.tokens * z["width"]) + 4 * self.tokens * z["width"] + 8 * self.requests * inner * S_STATE,
                "flops": self.tokens * (2 * weights + 5 * inner * S_STATE)}


_KINDS = {"decode": _Decode, "prompt": _Prompt, "attention": _Attention, "feed_forward": _FeedForward, "experts": _Experts,
          "latent": _Latent, "capped": _Capped, "channel_delta": _Delta, "head_delta": _HeadDelta, "general_delta": _GeneralDelta,
          "state_space": _StateSpace}
