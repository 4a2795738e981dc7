"""What the library's users have it do, as cases that can be timed and compared.

Whole steps of the Qwen3 model through ``Engine.step`` (prompts and single tokens, bfloat16 and true 32-bit), and the layers
that the other architectures are made of, each alone through the registered part's ``forward``: routed experts, the gated
delta rule, attention beside a state-space mixer, retention and differential attention.  Sizes are the presets'; weights and
inputs are drawn here from the case's seed.

A case is ``{"call", "sizes", "dtype", "step", "batch", "tokens"}``: ``step`` is ``"prompt"`` (``batch`` new sequences of up to
``tokens`` tokens, the first of exactly that many and the others shorter by turns) or ``"token"`` (one more token for each of
``batch`` sequences that hold about ``tokens`` already).  A layer's single-token step runs as a captured CUDA graph, which is
how the engine runs the whole model's.
"""

import math
import zlib

import torch

from idempotent_llm_b200.api import LM, build_model
from idempotent_llm_b200.cache import SequenceCache
from idempotent_llm_b200.config.presets import preset
from idempotent_llm_b200.engine import declare_weights
from idempotent_llm_b200.engine.batch import context_from_packed, pack_step_host
from idempotent_llm_b200.kernels import Kernels
from idempotent_llm_b200.parts import FEED_FORWARDS, MIXERS, Runtime

DEVICE = "cuda:0"
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
F64 = torch.float64


# ------------------------------------------------------------------------------------------------------- the cases
def _case(name, call, sizes, dtype, step, batch, tokens):
    return {"name": name, "call": call, "sizes": sizes, "dtype": dtype, "step": step, "batch": batch, "tokens": tokens}


def listed():
    return [
        # one user waiting for the next token: the smallest whole call, launches and latencies
        _case("model-token-1", "model", "qwen3-0.6b", "bfloat16", "token", 1, 1500),
        # the first answer to a long prompt
        _case("model-prompt-2048", "model", "qwen3-0.6b", "bfloat16", "prompt", 1, 2048),
        # the 32-bit path that other runs are checked against: a small batch decoding ...
        _case("model32-token-8", "model", "qwen3-0.6b", "float32", "token", 8, 400),
        # ... and its prompts, of unequal lengths
        _case("model32-prompt-2x350", "model", "qwen3-0.6b", "float32", "prompt", 2, 350),
        # experts chosen by a router: a long prompt, a full decoding batch, prompts at the large sizes
        _case("experts-prompt-2048", "experts", "zazulix-0.6b", "bfloat16", "prompt", 1, 2048),
        _case("experts-token-64", "experts", "tosodra-0.6b", "bfloat16", "token", 64, 0),
        _case("experts-prompt-4x1000-large", "experts", "pununex-8b", "bfloat16", "prompt", 4, 1000),
        # the recurrence with the longest serial chain: a long prompt, a full decoding batch
        _case("delta-prompt-2048", "gated_delta", "pununex-0.6b", "bfloat16", "prompt", 1, 2048),
        _case("delta-token-64", "gated_delta", "pununex-0.6b", "bfloat16", "token", 64, 300),
        # attention and a state-space mixer side by side, several prompts of unequal lengths at once
        _case("parallel-prompt-4x1500", "parallel", "lunulix-0.6b", "bfloat16", "prompt", 4, 1500),
        # a retention layer, an odd prompt
        _case("retention-prompt-1777", "retention", "zazulix-0.6b", "bfloat16", "prompt", 1, 1777),
        # two softmax maps per head behind short filters, a few ordinary prompts
        _case("differential-prompt-3x1000", "differential_attention", "zazulix-0.6b", "bfloat16", "prompt", 3, 1000),
    ]


# call -> (presets, most sequences of a prompt step, longest prompt, most sequences of a single-token step, longest context)
_RANGES = {
    "model": (("qwen3-0.6b",), 4, 2048, 64, 1500),
    "experts": (("zazulix-0.6b", "tosodra-0.6b", "pununex-0.6b", "pununex-8b"), 8, 2048, 64, 0),
    "gated_delta": (("pununex-0.6b", "pununex-8b"), 8, 2048, 64, 500),
    "parallel": (("lunulix-0.6b",), 8, 2048, 64, 500),
    "retention": (("zazulix-0.6b", "zazulix-8b"), 8, 2048, 64, 500),
    "differential_attention": (("zazulix-0.6b", "zazulix-8b"), 8, 2048, 64, 500),
}


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    call = rng.choice(sorted(_RANGES))
    presets, seqs, longest, batch, context = _RANGES[call]
    sizes = rng.choice(presets)
    dtype = rng.choice(("bfloat16", "float32")) if call == "model" else "bfloat16"
    step = rng.choice(("prompt", "token"))
    if dtype == "float32":
        seqs, longest, batch, context = 2, 350, 16, 400
    if step == "prompt":
        most = 2100 if call == "model" else 6000            # tokens of a step in all
        tokens = _log_uniform(rng, 12, longest)
        n = max(1, min(_log_uniform(rng, 1, seqs), most // tokens))
        return {"call": call, "sizes": sizes, "dtype": dtype, "step": step, "batch": n, "tokens": tokens}
    return {"call": call, "sizes": sizes, "dtype": dtype, "step": step, "batch": _log_uniform(rng, 1, batch),
            "tokens": rng.randint(min(8, context), context)}


def _lengths(case):
    """Tokens of each sequence: the first has ``tokens``, the others down to half of it."""
    n, t = case["batch"], case["tokens"]
    return [t - (i * t) // (2 * n) for i in range(n)]


# ------------------------------------------------------------------------------------------------------- inputs
def _rng(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((zlib.crc32(name.encode()) << 20) + seed)


def _value(decl, seed):
    """A tensor of a checkpoint: matrices as the presets draw them, decays and step sizes as trained models have them (rates
    from 1 to 16, steps from 0.001 to 0.1)."""
    g = _rng(seed, decl.name)
    if decl.name.endswith("A_log"):
        return torch.log(1.0 + 15.0 * torch.rand(decl.shape, generator=g, device=DEVICE))
    if decl.name.endswith("dt_bias"):
        step = torch.exp(math.log(1e-3) + math.log(100.0) * torch.rand(decl.shape, generator=g, device=DEVICE))
        return step + torch.log(-torch.expm1(-step))         # softplus of it is the step
    t = torch.randn(tuple(decl.free if n == -1 else n for n in decl.shape), generator=g, device=DEVICE)
    if decl.init in ("filter", "unit_normal"):
        return 0.5 * t
    return 1.0 + 0.1 * t if decl.init == "one_plus_normal" else 0.02 * t


def _weights(decls, seed, dtype):
    return {d.name: _value(d, seed).to(dtype) for d in decls if not d.optional}


def _tokens(case, seed, vocab, lengths):
    g = _rng(seed, "tokens")
    return [torch.randint(0, vocab, (n,), generator=g, device=DEVICE).tolist() for n in lengths]


def _rows(seed, name, n, width, dtype):
    """A layer's input: rows as a norm leaves them."""
    return torch.randn((n, width), generator=_rng(seed, name), device=DEVICE).to(dtype)


def _part_spec(case):
    """(registry, spec, name prefix) of the case's layer: the first of its kind in the preset."""
    for layer in preset(case["sizes"]).to_model_spec().layers:
        if case["call"] == "experts":
            if layer.feed_forward is not None and layer.feed_forward.kind == "routed_experts":
                return FEED_FORWARDS, layer.feed_forward, layer.prefix
        elif layer.mixer.kind == case["call"]:
            return MIXERS, layer.mixer, layer.prefix
    raise ValueError(f"{case['sizes']} has no {case['call']}")


# ------------------------------------------------------------------------------------------------------- whole steps
class _Model:
    """A loaded model and a step's tokens.  A single-token step goes back to the same place before each pass."""

    def __init__(self, case, seed):
        config = preset(case["sizes"])
        dtype = DTYPES[case["dtype"]]
        weights = _weights(declare_weights(config.to_model_spec()), seed, dtype)
        lengths = _lengths(case)
        room = sum(n + 65 for n in lengths) + 64
        model = build_model(config, weights, dtype, DEVICE)
        self.lm = LM(model, config, max_tokens=room, max_seqs=len(lengths), max_seq_len=max(lengths) + 64)
        engine = self.lm.engine
        prompts = _tokens(case, seed, config.vocab_size, lengths)
        self.prompts = self.slots = None
        if case["step"] == "prompt":
            self.prompts = prompts
        else:
            self.lengths = lengths
            self.slots = [engine.open() for _ in prompts]
            engine.step(list(zip(self.slots, prompts)))
            self.next = _tokens(case, seed + 1, config.vocab_size, [1] * len(prompts))

    def run(self):
        engine = self.lm.engine
        if self.prompts is not None:
            slots = [engine.open() for _ in self.prompts]
            logits = engine.step(list(zip(slots, self.prompts)))
            for s in slots:
                engine.close(s)
            return logits
        for s, n in zip(self.slots, self.lengths):
            engine.cache.set_length(s, n)
        return engine.step(list(zip(self.slots, self.next)))


# ------------------------------------------------------------------------------------------------------- one layer
class _Layer:
    """A part with its weights and cache, and a step's rows.  A prompt's pass starts from the zero state of new sequences; a
    single-token pass is one token further each time (its keys and values at the same place)."""

    def __init__(self, case, seed):
        registry, spec, prefix = _part_spec(case)
        dtype = DTYPES[case["dtype"]]
        cls = registry.get(spec.kind)
        rt = Runtime(device=torch.device(DEVICE), dtype=dtype, kernels=Kernels(dtype, DEVICE))
        self.part = cls(spec, _weights(cls.declare(spec, prefix), seed, dtype), prefix, rt)
        self.mixes = registry is MIXERS
        lengths = _lengths(case)
        prompt = case["step"] == "prompt"
        self.kv = self.state = self.graph = None
        slots = list(range(len(lengths)))
        if self.mixes:
            self.cache = SequenceCache({0: cls.cache_need(spec)}, sum(n + 65 for n in lengths), dtype, DEVICE,
                                       max_seqs=len(lengths), max_seq_len=max(lengths) + 64)
            slots = [self.cache.alloc_slot() for _ in lengths]
            self.cache.reserve([(s, n + 1) for s, n in zip(slots, lengths)])
            self.cache.flush()
            self.kv, self.state = self.cache.view(0), self.cache.state_of(0)
        if prompt or self.mixes:
            self._step(slots, [0] * len(slots), lengths, _rows(seed, "x", sum(lengths), spec.hidden, dtype), True)
        if not prompt:
            if self.mixes:
                self._pass()                             # the sequences' earlier tokens
            self._step(slots, lengths, [1] * len(slots), _rows(seed, "next", len(slots), spec.hidden, dtype), False)
            self._capture()
        self.zero = prompt and self.state is not None

    def _step(self, slots, starts, lengths, x, eager):
        tokens = [[0] * n for n in lengths]
        packed, n, q_lens = pack_step_host(slots, starts, tokens)
        self.ctx = context_from_packed(packed.to(DEVICE), n, slots, q_lens, starts, host_tokens=tokens if eager else None)
        self.x = x

    def _pass(self):
        self.ctx.memo.clear()                            # a step makes its own position tables
        if self.mixes:
            return self.part.forward(self.x, self.ctx, self.kv, self.state, True)
        return self.part.forward(self.x, self.ctx)

    def _capture(self):
        keep = None if self.state is None else self.state.clone()
        for _ in range(2):
            self._pass()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = self._pass()
        if keep is not None:
            self.state.copy_(keep)

    def run(self):
        if self.graph is not None:
            self.graph.replay()
        else:
            if self.zero:
                self.state.zero_()
            self.out = self._pass()
        return (self.out, self.state) if self.state is not None else self.out


def prepare(case, seed):
    with torch.no_grad():
        return _Model(case, seed) if case["call"] == "model" else _Layer(case, seed)


def run(state):
    with torch.no_grad():
        return state.run()


# ------------------------------------------------------------------------------------------------------- work
def _size(dtype):
    return 2 if dtype == "bfloat16" else 4


def _pairs(case):
    """(query, key) pairs that causal attention scores."""
    total = 0
    for n in _lengths(case):
        total += n * (n + 1) // 2 if case["step"] == "prompt" else n + 1
    return total


def work(case):
    """Weights and cached rows read once, inputs and outputs once; a multiply and an add for every number of a product."""
    lengths = _lengths(case)
    e = _size(case["dtype"])
    n = sum(lengths) if case["step"] == "prompt" else len(lengths)
    rows = sum(lengths) if case["step"] == "prompt" else sum(lengths) + len(lengths)      # cached rows written or read
    if case["call"] == "model":
        c = preset(case["sizes"])
        wide = c.num_attention_heads * c.head_dim
        kv = c.num_key_value_heads * c.head_dim
        layer = c.hidden_size * (2 * wide + 2 * kv + 3 * c.intermediate_size)
        head = c.vocab_size * c.hidden_size
        flops = c.num_hidden_layers * (2 * n * layer + 4 * _pairs(case) * wide) + 2 * len(lengths) * head
        bytes_ = e * (c.num_hidden_layers * (layer + 2 * rows * kv) + head) + 4 * len(lengths) * c.vocab_size
        return {"bytes": bytes_, "flops": flops}
    _, s, _ = _part_spec(case)
    stream = n * s.hidden * (e + 4)                                              # the rows in, the 32-bit sum out
    if case["call"] == "experts":
        used = min(s.n_experts, n * s.top)
        shared = 3 * s.hidden * s.shared.intermediate if s.shared is not None else 0
        one = 3 * s.hidden * s.intermediate
        real = s.top * s.n_experts / (s.n_experts + s.n_identity)
        router = (s.n_experts + s.n_identity) * s.hidden
        return {"bytes": stream + e * (used * one + shared + router), "flops": 2 * n * (real * one + shared + router)}
    weights, flops, state, cached = _mixer_work(case, s, n, _pairs(case))
    return {"bytes": stream + e * weights + 4 * state * len(lengths) + e * cached * rows, "flops": 2 * n * weights + flops}


def _mixer_work(case, s, n, pairs):
    """(weights, operations beside the products, 32-bit state floats moved per sequence, cached numbers per row)."""
    moved = 1 if case["step"] == "prompt" else 2                                 # written, or read and written
    if s.kind == "gated_delta":
        q, v = s.kv_heads * s.key_dim, s.heads * s.value_dim
        gate = s.hidden * v if s.gate == "silu" else 0
        weights = s.hidden * (2 * q + 2 * v + 2 * s.heads) + gate
        return weights, 8 * n * v * s.key_dim, moved * (v * s.key_dim + (s.conv_taps - 1) * (2 * q + v)), 0
    if s.kind == "retention":
        q, v = s.heads * s.key_dim, s.heads * s.value_dim
        return s.hidden * (2 * q + 3 * v), 5 * n * v * s.key_dim, moved * v * s.key_dim, 0
    if s.kind == "differential_attention":
        q, k, v = 2 * s.n_heads * s.key_dim, 2 * s.n_kv_heads * s.key_dim, s.n_kv_heads * s.value_dim
        out = s.n_heads * s.value_dim
        weights = s.hidden * (q + k + v + s.n_heads + out)
        return weights, pairs * (2 * q + 4 * out), moved * (s.conv_taps - 1) * (q + k + v), k + v
    a, b = (branch.mixer for branch in s.branches)                               # attention beside the state-space mixer
    q, k, v = a.n_heads * a.key_dim, a.n_kv_heads * a.key_dim, a.n_kv_heads * a.value_dim
    out, inner, gn = a.n_heads * a.value_dim, b.heads * b.head_dim, b.groups * b.state
    weights = s.hidden * (q + k + v + 2 * out + 3 * inner + 2 * gn + b.heads)
    state = (a.conv_taps - 1) * (q + k + v) + (b.conv_taps - 1) * (inner + 2 * gn) + inner * b.state
    return weights, pairs * (2 * q + 2 * out) + 5 * n * inner * b.state, moved * state, k + v


# ------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times what the library differs by from the same sums in 64 bits: 2.3e-6 in the 32-bit model, 6.2e-3 in the
    bfloat16 one, 5.5e-3 where one softmax map is taken off another, 1.7e-3 in the other layers."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["call"] in ("model", "differential_attention"):
        return {"rel": 2.5e-2}
    return {"rel": 7e-3}


# ------------------------------------------------------------------------------------------------------- in 64 bits
def _norm(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(rot):
    i = torch.arange(rot.dim // 2, dtype=F64, device=DEVICE)
    f = float(rot.theta) ** (-2.0 * i / rot.dim)
    sc = getattr(rot, "scaling", None)
    if sc is not None:                               # by wavelength: short waves kept, long ones slowed, a blend between
        wave = 2.0 * math.pi / f
        blend = (sc.original / wave - sc.low) / (sc.high - sc.low)
        f = torch.where(wave < sc.original / sc.high, f,
                        torch.where(wave > sc.original / sc.low, f / sc.factor, (1.0 - blend) * f / sc.factor + blend * f))
    return f


def _turn(x, rot):
    """x [T, heads, d]: dim i turned with dim i + dims / 2 over the first dims."""
    half = rot.dim // 2
    a = torch.arange(x.shape[0], dtype=F64, device=DEVICE)[:, None] * _frequencies(rot)[None, :]
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], dim=-1)


def _filter(u, w, bias=None):
    """u [T, C], w [C, taps]: the last tap meets the token itself, zeros before the start."""
    T, taps = u.shape[0], w.shape[1]
    y = torch.zeros_like(u)
    for j in range(taps):
        back = taps - 1 - j
        if back < T:
            y[back:] += w[:, j] * u[:T - back]
    return y if bias is None else y + bias


def _attend(q, k, v, scale, sink=None):
    """Causal softmax attention; q-head h reads kv-head h // (H / G); ``sink`` [H]: one more term of the denominator."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    out = torch.zeros(T, H, v.shape[-1], dtype=F64, device=DEVICE)
    hidden = torch.ones(T, T, dtype=torch.bool, device=DEVICE).triu(1)
    for h in range(H):
        s = ((q[:, h] @ k[:, h // per].T) * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :T] @ v[:, h // per]
    return out


def _recur(q, k, v, decay, beta=None):
    """S <- decay S (rows by key dim); u = v, or beta (v - S^T k); S <- S + k u^T; o = S^T q.  q, k [T, H, d], v [T, H, dv],
    decay broadcast to [T, H, d], beta [T, H]."""
    T, H, d = k.shape
    S = torch.zeros(H, d, v.shape[-1], dtype=F64, device=DEVICE)
    out = torch.empty_like(v)
    for t in range(T):
        S = S * decay[t][:, :, None]
        u = v[t]
        if beta is not None:
            u = beta[t][:, None] * (u - (k[t][:, None, :] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None, :])
        out[t] = (q[t][:, None, :] @ S)[:, 0]
    return out


def _gated(x, w, p, names):
    return (_silu(x @ w[p + names.gate].T) * (x @ w[p + names.up].T)) @ w[p + names.down].T


def _exact_delta(x, w, p, s):
    T, nm = x.shape[0], s.names
    q, k, v = (_silu(_filter(x @ w[p + n].T, w[p + n + nm.conv])) for n in (nm.q, nm.k, nm.v))
    unit = lambda z: z / torch.sqrt((z * z).sum(dim=-1, keepdim=True) + 1e-6)    # noqa: E731
    per = s.heads // s.kv_heads
    q, k = (unit(z.view(T, s.kv_heads, s.key_dim)).repeat_interleave(per, dim=1) for z in (q, k))
    beta = torch.sigmoid(x @ w[p + nm.beta].T)
    step = torch.nn.functional.softplus(x @ w[p + nm.decay].T + w[p + nm.dt_bias])
    decay = torch.exp(-torch.exp(w[p + nm.a_log]) * step)[:, :, None].expand(T, s.heads, s.key_dim)
    o = _recur(q * s.key_dim ** -0.5, k, v.view(T, s.heads, s.value_dim), decay, beta)
    o = _norm(o, s.norm_eps, w[p + nm.norm]).reshape(T, -1) * _silu(x @ w[p + nm.gate].T)
    return o @ w[p + nm.o].T


def _exact_retention(x, w, p, s):
    T, nm = x.shape[0], s.names
    q, k = (_turn((x @ w[p + n].T).view(T, s.heads, s.key_dim), s.position) for n in (nm.q, nm.k))
    v = (x @ w[p + nm.v].T).view(T, s.heads, s.value_dim)
    decay = torch.tensor(s.decay, dtype=F64, device=DEVICE)[None, :, None].expand(T, s.heads, s.key_dim)
    o = _norm(_recur(q, k * s.key_dim ** -0.5, v, decay), s.eps).reshape(T, -1)
    return (o * _silu(x @ w[p + nm.gate].T)) @ w[p + nm.o].T


def _exact_differential(x, w, p, s):
    T, nm = x.shape[0], s.names
    q, k, v = (_filter(x @ w[p + n].T, w[p + n + nm.conv]) for n in (nm.q, nm.k, nm.v))
    q, k = (_turn(z.reshape(T, -1, s.key_dim), s.position) for z in (q, k))
    q, k = q.view(T, s.n_heads, 2, s.key_dim), k.view(T, s.n_kv_heads, 2, s.key_dim)
    v = v.view(T, s.n_kv_heads, s.value_dim)
    a, b = (_attend(q[:, :, m], k[:, :, m], v, s.softmax_scale) for m in (0, 1))
    one, two = (torch.exp((w[p + i] * w[p + j]).sum()) for i, j in ((nm.lambda_q1, nm.lambda_k1), (nm.lambda_q2, nm.lambda_k2)))
    o = _norm(a - (one - two + s.diff) * b, s.eps) * (1.0 - s.diff) * torch.sigmoid(x @ w[p + nm.gate].T)[:, :, None]
    return o.reshape(T, -1) @ w[p + nm.o].T


def _exact_parallel(x, w, p, s):
    T = x.shape[0]
    left, right = s.branches
    a, q = left.mixer, p + s.prefix + left.prefix
    nm = a.names
    u = [_filter(x @ w[q + n].T, w[q + n + nm.conv]) for n in (nm.q, nm.k, nm.v)]
    u = [z.view(T, h, -1) for z, h in zip(u, (a.n_heads, a.n_kv_heads, a.n_kv_heads))]
    o = _attend(_turn(u[0], a.position), _turn(u[1], a.position), u[2], a.softmax_scale, w[q + nm.sink])
    first = (o.reshape(T, -1) * torch.sigmoid(x @ w[q + nm.gate].T)) @ w[q + nm.o].T
    b, q = right.mixer, p + s.prefix + right.prefix
    nm = b.names
    inner, gn = b.heads * b.head_dim, b.groups * b.state
    z, xbc, dt = (x @ w[q + nm.w_in].T).split([inner, inner + 2 * gn, b.heads], dim=1)
    xbc = _silu(_filter(xbc, w[q + nm.conv], w[q + nm.conv_bias]))
    v, B, C = xbc.split([inner, gn, gn], dim=1)
    v = v.reshape(T, b.heads, b.head_dim)
    B, C = (m.reshape(T, b.groups, b.state).repeat_interleave(b.heads // b.groups, dim=1) for m in (B, C))
    dt = torch.nn.functional.softplus(dt + w[q + nm.dt_bias])
    decay = torch.exp(-torch.exp(w[q + nm.a_log]) * dt)[:, :, None].expand(T, b.heads, b.state)
    y = _recur(C, B * dt[:, :, None], v, decay) + w[q + nm.d][None, :, None] * v
    y = y.reshape(T, inner) * _silu(z)
    y = _norm(y.view(T, b.norm_groups, -1), b.norm_eps).reshape(T, inner) * w[q + nm.norm]
    return left.scale * first + right.scale * (y @ w[q + nm.o].T)


def _exact_experts(x, w, p, s):
    z = x @ w[p + s.router].T
    scores = torch.softmax(z, dim=-1) if s.scores == "softmax" else torch.sigmoid(z)
    choice = scores + w[p + s.correction] if s.correction is not None else scores
    groups = choice.view(x.shape[0], s.groups, -1)
    best = groups.topk(min(s.group_top, groups.shape[-1]), dim=-1).values.sum(dim=-1)
    kept = torch.zeros_like(best).scatter(1, best.topk(s.groups_keep, dim=-1).indices, 1.0).bool()
    chosen = groups.masked_fill(~kept[:, :, None], -math.inf).flatten(1).topk(s.top, dim=-1).indices
    weight = scores.gather(1, chosen)
    if s.renormalize:
        weight = weight / (weight.sum(dim=-1, keepdim=True) + 1e-20)
    weight = weight * s.scale
    out = torch.zeros_like(x)
    if s.shared is not None:
        out = _gated(x, w, p, s.shared.names)
        if s.shared_gate is not None:
            out = out * torch.sigmoid(x @ w[p + s.shared_gate].T)
    for e in range(s.n_experts + s.n_identity):
        row, k = (chosen == e).nonzero(as_tuple=True)
        mine = weight[row, k][:, None]
        if e >= s.n_experts:
            out[row] += mine * x[row]
        elif s.weight_on == "input":
            out[row] += _gated(mine * x[row], w, p + s.expert.format(e), s.names)
        else:
            out[row] += mine * _gated(x[row], w, p + s.expert.format(e), s.names)
    return out


def _exact_model(config, w, tokens):
    """Logits of a sequence's last token."""
    c = config
    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEVICE)].to(F64)
    rot = config.to_model_spec().layers[0].mixer.position
    T = x.shape[0]
    for i in range(c.num_hidden_layers):
        m = {n: w[f"model.layers.{i}.{n}.weight"].to(F64) for n in (
            "input_layernorm", "self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "self_attn.q_norm",
            "self_attn.k_norm", "post_attention_layernorm", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        h = _norm(x, c.rms_norm_eps, m["input_layernorm"])
        q, k, v = ((h @ m[f"self_attn.{n}_proj"].T).view(T, -1, c.head_dim) for n in "qkv")
        q = _turn(_norm(q, c.rms_norm_eps, m["self_attn.q_norm"]), rot)
        k = _turn(_norm(k, c.rms_norm_eps, m["self_attn.k_norm"]), rot)
        x = x + _attend(q, k, v, c.head_dim ** -0.5).reshape(T, -1) @ m["self_attn.o_proj"].T
        h = _norm(x, c.rms_norm_eps, m["post_attention_layernorm"])
        x = x + (_silu(h @ m["mlp.gate_proj"].T) * (h @ m["mlp.up_proj"].T)) @ m["mlp.down_proj"].T
    return _norm(x[-1], c.rms_norm_eps, w["model.norm.weight"].to(F64)) @ w["model.embed_tokens.weight"].to(F64).T


_EXACT = {"gated_delta": _exact_delta, "retention": _exact_retention, "differential_attention": _exact_differential,
          "parallel": _exact_parallel, "experts": _exact_experts}


def exact(case, seed):
    """The same sums in 64 bits; the moved state of a layer has no value here."""
    with torch.no_grad():
        lengths, dtype = _lengths(case), DTYPES[case["dtype"]]
        token = case["step"] == "token"
        if sum(lengths) > 16000:
            return None
        if case["call"] == "model":
            config = preset(case["sizes"])
            w = _weights(declare_weights(config.to_model_spec()), seed, dtype)
            tokens = _tokens(case, seed, config.vocab_size, lengths)
            if token:
                tokens = [a + b for a, b in zip(tokens, _tokens(case, seed + 1, config.vocab_size, [1] * len(lengths)))]
            return torch.stack([_exact_model(config, w, t) for t in tokens])
        registry, s, p = _part_spec(case)
        w = {k: v.to(F64) for k, v in _weights(registry.get(s.kind).declare(s, p), seed, dtype).items()}
        layer = _EXACT[case["call"]]
        new = _rows(seed, "next", len(lengths), s.hidden, dtype).to(F64) if token else None
        if registry is FEED_FORWARDS:
            return layer(new if token else _rows(seed, "x", sum(lengths), s.hidden, dtype).to(F64), w, p, s)[None]
        rows, at = [], 0
        x = _rows(seed, "x", sum(lengths), s.hidden, dtype).to(F64)
        for i, n in enumerate(lengths):
            mine = x[at:at + n]
            at += n
            rows.append(layer(torch.cat([mine, new[i:i + 1]]), w, p, s)[-1:] if token else layer(mine, w, p, s))
        out = torch.cat(rows)[None]
        keeps = registry.get(s.kind).cache_need(s).state_shape is not None
        return (out, None) if keeps else out
