"""What this framework's speed is measured on: its layers, each called through its part, and one whole model.

A case is one part of a decoder layer (`part`), in the layer sizes of one of `SIZES`, over the packed rows of one step:
`batch` sequences that bring up to `tokens` tokens each on top of up to `past` earlier ones (`ragged`: sequence b of B brings
(b + 1) / B of them, else all the same).  tokens == 1 is a decode step.  A pass is the part's forward over those rows, as a
model's step calls it: normed rows in, the layer's branch out, keys and values or the recurrent state written to the cache.
"generate" is a whole Llama engine: prompts, then single tokens, logits of every step.
"""
import math

import torch

from longbow_quarrel_b200 import architectures  # noqa: F401  (registers parts and architectures)
from longbow_quarrel_b200.cache import Cache
from longbow_quarrel_b200.engine import Engine
from longbow_quarrel_b200.engine.step import make_context, pack_step
from longbow_quarrel_b200.kernels import ops
from longbow_quarrel_b200.parts.base import Runtime
from longbow_quarrel_b200.parts.registry import make_part
from longbow_quarrel_b200.parts.spec import PartSpec
from longbow_quarrel_b200.weights import random_weights

EPS = 1e-5
DEVICE = "cuda:0"
VOCAB = 32000

# Layer sizes: the Llama 3 shapes of 1B and 8B that the benchmark uses for every design, and a small one.
SIZES = {
    "small": dict(width=512, heads=8, kv=2, dim=64, ff=1536, latent_heads=4, q_rank=192, kv_rank=128, experts=16, top=4, expert_ff=256, shared_ff=512),
    "1b": dict(width=2048, heads=32, kv=8, dim=64, ff=8192, latent_heads=16, q_rank=768, kv_rank=512, experts=64, top=6, expert_ff=1408, shared_ff=2816),
    "8b": dict(width=4096, heads=32, kv=8, dim=128, ff=14336, latent_heads=32, q_rank=1536, kv_rank=512, experts=64, top=6, expert_ff=2048, shared_ff=4096),
}
NOPE, ROT, VALUE = 128, 64, 128         # a latent head's unrotated, rotated and value sizes
GROUPS, KEEP, ROUTE_SCALE = 8, 3, 2.5   # the router's groups of experts
CAP, TAU, RANK, TAPS = 15.0, 16.0, 64, 4


def _case(name, part, size, dtype="bfloat16", batch=1, tokens=1, past=0, ragged=False):
    return {"name": name, "part": part, "size": size, "dtype": dtype, "batch": batch, "tokens": tokens, "past": past, "ragged": ragged}


def listed():
    return [
        # one user's decode step through an attention layer: launches and latency
        _case("attention_decode_b1", "attention", "1b", past=130),
        # the true 32-bit path, in which a model is checked, over a few short prompts
        _case("attention_prompt_f32", "attention", "small", "float32", 3, 300, ragged=True),
        # several users' prompts of unequal lengths in one step
        _case("attention_prompt_8b", "attention", "8b", batch=4, tokens=2048, ragged=True),
        # a prompt through a layer with a fixed decay per head
        _case("retention_prompt_1b", "retention", "1b", tokens=2048),
        # portions of long prompts, going on from a state, through a layer with exponential gates
        _case("mlstm_portion_8b", "mlstm", "8b", batch=3, tokens=1025, past=500, ragged=True),
        # a prompt through a layer whose key channels decay each at its own rate
        _case("channel_decay_prompt_8b", "channel_decay", "8b", tokens=2048),
        # a prompt, and a batch's single tokens, through attention over latent rows
        _case("latent_prompt_1b", "latent", "1b", tokens=2048),
        _case("latent_decode_b8", "latent", "1b", batch=8, past=2048),
        # a prompt, and a batch's single tokens, through routed experts
        _case("experts_prompt_1b", "experts", "1b", tokens=2048),
        _case("experts_decode_b8", "experts", "1b", batch=8, past=100),
        # prompts through the gated delta rule
        _case("delta_prompt_1b", "delta", "1b", batch=2, tokens=1500, ragged=True),
        # a batch answered by a whole model: prompts, then tokens one by one
        _case("generate_8b", "generate", "8b", batch=8, tokens=512, past=32, ragged=True),
    ]


def draw(rng):
    """Any part, in any of its sizes: prompts and portions of 2 to 2,500 rows in all, decode batches of 1 to 32."""
    part = rng.choice(["attention", "retention", "mlstm", "channel_decay", "latent", "experts", "delta", "attention", "latent", "experts", "generate"])
    size = rng.choice(["small", "1b", "8b"])
    ragged = rng.random() < 0.6
    dtype = "float32" if size == "small" and rng.random() < 0.3 else "bfloat16"
    past = 0 if part in ("delta", "experts") or rng.random() < 0.5 else _log(rng, 1, 3000)
    if part == "generate":
        return _drawn(part, "8b" if size == "8b" else "1b", "bfloat16", rng.randint(1, 8), _log(rng, 3, 500), rng.randint(2, 32), ragged)
    if rng.random() < 0.3 and part in ("attention", "latent", "experts"):
        return _drawn(part, size, dtype, _log(rng, 1, 32), 1, past, ragged)
    batch = rng.choice([1, 1, 2, 3, 5, 8])
    most = (600 if dtype == "float32" else 2500) // batch
    return _drawn(part, size, dtype, batch, _log(rng, 2, most), past, ragged)


def _drawn(part, size, dtype, batch, tokens, past, ragged):
    case = _case("", part, size, dtype, batch, tokens, past, ragged)
    del case["name"]
    return case


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------------------- what a case is made of

def _lengths(case):
    """(new tokens, earlier tokens) of every sequence."""
    B = case["batch"]
    share = lambda n, b: -(-n * (b + 1) // B) if case["ragged"] else n
    new = [max(1, share(case["tokens"], b)) for b in range(B)]
    return new, [share(case["past"], B - 1 - b) for b in range(B)]


def _decays(heads):
    return tuple(1.0 - 2.0 ** (-5 - 3 * h / heads) for h in range(heads))


def _rope(dims, base):
    return PartSpec("rope", {"head_dim": dims, "theta": base})


def _part(case, runtime):
    z = SIZES[case["size"]]
    D, H, dim = z["width"], z["heads"], z["dim"]
    matrix = dict(hidden_size=D, n_heads=H, key_dim=dim, value_dim=dim, eps=EPS)
    kind = case["part"]
    if kind == "attention":
        spec = PartSpec("attention", dict(hidden_size=D, n_heads=H, n_kv_heads=z["kv"], head_dim=dim, scale=dim ** -0.5, position=_rope(dim, 500000.0)))
    elif kind == "retention":
        spec = PartSpec("retention", dict(matrix, decay=_decays(H), position=_rope(dim, 10000.0)))
    elif kind == "mlstm":
        spec = PartSpec("mlstm", dict(matrix, gate_cap=CAP))
    elif kind == "channel_decay":
        spec = PartSpec("channel_decay", dict(matrix, tau=TAU, rank=RANK))
    elif kind == "latent":
        spec = PartSpec("latent_attention", dict(hidden_size=D, n_heads=z["latent_heads"], head_dim=NOPE, rot_dim=ROT, value_dim=VALUE, q_rank=z["q_rank"],
                                                 kv_rank=z["kv_rank"], scale=(NOPE + ROT) ** -0.5, eps=EPS, position=_rope(ROT, 10000.0), gate="sigmoid"))
    elif kind == "experts":
        return make_part("ffn", PartSpec("routed_experts", dict(
            hidden_size=D, n_experts=z["experts"], top=z["top"], expert_size=z["expert_ff"], activation="gelu", groups=GROUPS, keep_groups=KEEP,
            route_scale=ROUTE_SCALE, shared_size=z["shared_ff"])), runtime)
    else:
        spec = PartSpec("channel_delta", dict(matrix, taps=TAPS, rank=RANK, gate_rank=RANK))
    return make_part("mixer", spec, runtime)


def _generator(seed, salt):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 1000 + salt)


def _rows(case, seed, n, width):
    """Normed rows as a layer's first norm hands them on."""
    x = torch.randn((n, width), generator=_generator(seed, 1), device=DEVICE)
    return (x / x.square().mean(dim=1, keepdim=True).add(EPS).sqrt()).to(_dtype(case))


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _earlier(case, seed, b, past):
    """What the cache holds of sequence b: keys (and values) of its earlier tokens, or its state."""
    z, g = SIZES[case["size"]], _generator(seed, 100 + b)
    H, dim, kind = z["heads"], z["dim"], case["part"]
    normal = lambda *shape: torch.randn(shape, generator=g, device=DEVICE)
    if kind == "attention":
        return normal(z["kv"], past, dim).to(_dtype(case)), normal(z["kv"], past, dim).to(_dtype(case))
    if kind == "latent":
        return (normal(1, past, z["kv_rank"] + ROT).to(_dtype(case)),)
    if kind == "mlstm":     # one more row for the running maximum, one more column for the normaliser
        state = normal(H, dim + 1, dim + 1)
        state[:, dim] = normal(H, 1).abs()
        return state if past else torch.zeros_like(state)
    state = normal(H, dim, dim)
    return state if past else torch.zeros_like(state)


def prepare(case, seed):
    if case["part"] == "generate":
        return _prepare_engine(case, seed)
    new, past = _lengths(case)
    device = torch.device(DEVICE)
    context = -(-max(n + p for n, p in zip(new, past)) // 64) * 64
    runtime = Runtime(device=device, dtype=_dtype(case), max_context=context)
    part = _part(case, runtime)
    ops.prepare(runtime.dtype, verbose=False, extra=tuple(getattr(part, "kernel_libraries", ())))
    part.load(random_weights(part.weights(), seed, _dtype(case), device))
    state = {"case": case, "part": part, "h": _rows(case, seed, sum(new), SIZES[case["size"]]["width"]), "view": None, "start": [], "kept": []}
    slots = list(range(len(new)))
    needs = part.step_needs()
    if case["part"] != "experts":
        cache = Cache({0: part.cache_need()}, sum(-(-(n + p) // 64) * 64 for n, p in zip(new, past)), context, runtime.dtype, device, max_slots=len(new))
        slots = [cache.alloc_slot() for _ in new]
        for slot, n, p in zip(slots, new, past):
            cache.reserve(slot, n + p)
        cache.upload()
        view = state["view"] = cache.view(0)
        state["cache"] = cache
        if case["part"] in ("attention", "latent"):
            for b, (slot, p) in enumerate(zip(slots, past)):
                at = torch.arange(p, device=device)
                page, place = view.page_table[slot].long()[at // 64], at % 64
                for pool, rows in zip((view.k_pages, view.v_pages), _earlier(case, seed, b, p)):
                    pool[page, :, place] = rows.transpose(0, 1)
            state["kept"] = [t for t in (view.k_pages, view.v_pages) if t is not None]
        else:
            state["kept"] = list(view) if isinstance(view, (tuple, list)) else [view]
            if case["part"] != "delta":
                for b, (slot, p) in enumerate(zip(slots, past)):
                    view[slot] = _earlier(case, seed, b, p)
            state["start"] = [t.clone() for t in state["kept"]]
    flat, info = pack_step([(s, [0] * n) for s, n in zip(slots, new)], None, past, needs)
    state["ctx"] = make_context(torch.from_numpy(flat).to(device), info, slots)
    return state


def _llama(case):
    z = SIZES[case["size"]]
    return dict(architectures=["LlamaForCausalLM"], hidden_size=z["width"], num_hidden_layers=2, num_attention_heads=z["heads"], num_key_value_heads=z["kv"],
                head_dim=z["dim"], intermediate_size=z["ff"], vocab_size=VOCAB, rope_theta=500000.0, rms_norm_eps=EPS, tie_word_embeddings=False,
                max_position_embeddings=8192)


def _tokens(case, seed):
    """Prompts, and the tokens that follow them one by one (a case's `past` says how many steps)."""
    new, _ = _lengths(case)
    g = torch.Generator().manual_seed(int(seed))
    draw_ = lambda n: torch.randint(0, VOCAB, (n,), generator=g).tolist()
    return [draw_(n) for n in new], [draw_(len(new)) for _ in range(case["past"])]


def _prepare_engine(case, seed):
    prompts, steps = _tokens(case, seed)
    context = max(map(len, prompts)) + len(steps)
    engine = Engine.from_config(_llama(case), seed=int(seed), max_batch=len(prompts), max_context=context,
                                max_tokens=sum(-(-(len(p) + len(steps)) // 64) * 64 for p in prompts), device=DEVICE)
    state = {"case": case, "engine": engine, "prompts": prompts, "steps": steps}
    run(state)          # an engine that has served before: its steps are captured
    return state


def run(state):
    case = state["case"]
    if case["part"] == "generate":
        engine = state["engine"]
        slots = [engine.new_sequence() for _ in state["prompts"]]
        logits = [engine.step(list(zip(slots, state["prompts"]))).clone()]
        for tokens in state["steps"]:
            logits.append(engine.step([(s, [t]) for s, t in zip(slots, tokens)]).clone())
        for slot in slots:
            engine.end_sequence(slot)
        return logits
    part = state["part"]
    if case["part"] == "experts":
        return part.forward(state["h"], state["ctx"], None)
    for kept, start in zip(state["kept"], state["start"]):
        kept.copy_(start)                       # every pass goes on from the same state
    out = part.forward(state["h"], state["ctx"], state["view"], None)
    return [out, *state["kept"]]


# ---------------------------------------------------------------------------- what a pass cannot do without

def _numel(case):
    """The part's weights, and those that a row passes through."""
    z = SIZES[case["size"]]
    D, H, dim, kv = z["width"], z["heads"], z["dim"], z["kv"]
    kind = case["part"]
    if kind == "attention":
        n = D * (H + 2 * kv) * dim + D * H * dim
    elif kind == "latent":
        Hl = z["latent_heads"]
        n = D * (z["q_rank"] + z["kv_rank"] + ROT + Hl * VALUE) + z["q_rank"] * Hl * (NOPE + ROT) + z["kv_rank"] * Hl * (NOPE + VALUE) + D * Hl * VALUE
    elif kind == "mlstm":
        n = 5 * D * H * dim + 2 * H * D
    elif kind == "channel_decay":
        n = 5 * D * H * dim + RANK * (D + H * dim)
    elif kind == "delta":
        n = 4 * D * H * dim + 2 * RANK * (D + H * dim) + H * D
    else:
        n = 5 * D * H * dim
    return n


def work(case):
    z = SIZES[case["size"]]
    D, H, dim = z["width"], z["heads"], z["dim"]
    new, past = _lengths(case)
    T, wide = sum(new), 4 if case["dtype"] == "float32" else 2
    if case["part"] == "generate":
        layer = D * (H + 2 * z["kv"]) * dim + D * H * dim + 3 * D * z["ff"]
        passes, B = case["past"] + 1, len(new)
        pairs = sum(sum(range(1, n + case["past"] + 1)) for n in new)
        kv_read = sum((n + i) * 2 * z["kv"] * dim for n in new for i in range(case["past"]))
        return {"bytes": passes * (2 * layer + VOCAB * D) * wide + 2 * kv_read * wide + passes * B * VOCAB * 4,
                "flops": 2.0 * (T + B * case["past"]) * 2 * layer + 2.0 * passes * B * VOCAB * D + 2 * 4.0 * H * dim * pairs}
    rows = T * D * (wide + 4)
    if case["part"] == "experts":
        E, top = z["experts"], z["top"]
        hit = E * (1.0 - (1.0 - top / E) ** T)          # experts that some row chooses, on average
        each, rest = 2 * D * z["expert_ff"], 2 * D * z["shared_ff"] + (E + 1) * D
        return {"bytes": rows + (hit * each + rest) * wide, "flops": 2.0 * T * (top * each + rest)}
    n = _numel(case)
    pairs = sum(p * m + m * (m + 1) / 2 for m, p in zip(new, past))
    if case["part"] == "attention":
        return {"bytes": rows + n * wide + (sum(past) + T) * 2 * z["kv"] * dim * wide, "flops": 2.0 * T * n + 4.0 * H * dim * pairs}
    if case["part"] == "latent":
        Hl = z["latent_heads"]
        # Keys and values are expanded per token for a prompt; single tokens read the latent rows as they are.
        per_pair = 2.0 * Hl * ((NOPE + ROT + VALUE) if case["tokens"] > 1 else (2 * z["kv_rank"] + ROT))
        return {"bytes": rows + n * wide + (sum(past) + T) * (z["kv_rank"] + ROT) * wide, "flops": 2.0 * T * n + per_pair * pairs}
    states = 2 * 4 * len(new) * H * dim * dim
    return {"bytes": rows + n * wide + states, "flops": 2.0 * T * n + 4.0 * T * H * dim * dim}


# About four times what is seen between the path and `exact`: 0.0025 to 0.0047 for a layer in bfloat16 (rows, weights and
# probabilities of eight bits; the delta rule's inputs stay 32-bit sums: 0.0017), 0.012 for two layers and the head, 8e-7 in 32-bit.
TOLERANCE = {"attention": 0.016, "retention": 0.016, "mlstm": 0.018, "channel_decay": 0.016, "latent": 0.016, "experts": 0.012, "delta": 0.008, "generate": 0.05}


def tolerance(case):
    return {"rel": 5e-6 if case["dtype"] == "float32" else TOLERANCE[case["part"]]}


# ---------------------------------------------------------------------------- the same in 64 bits

def _rotate(x, pos, base):
    """x [T, heads, d]: pairs (i, i + d / 2) turn by pos * base^(-2i / d)."""
    half = x.shape[-1] // 2
    a = pos[:, None, None].double() * torch.tensor(float(base), dtype=torch.float64, device=x.device) ** (-torch.arange(half, device=x.device).double() / half)
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _norm(x, gain=None):
    y = x / (x.square().mean(-1, keepdim=True) + EPS).sqrt()
    return y if gain is None else y * gain


def _attend(q, k, v, past, scale):
    """q [T, H, d] at positions past.., k [L, G, d], v [L, G, dv] -> [T, H, dv]."""
    T, H = q.shape[:2]
    G, out = k.shape[1], []
    hidden = torch.arange(k.shape[0], device=q.device)[None] > torch.arange(past, past + T, device=q.device)[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), dim=1) @ v[:, h * G // H])
    return torch.stack(out, dim=1)


def _exact_attention(case, w, h, past, earlier):
    z = SIZES[case["size"]]
    H, G, d = z["heads"], z["kv"], z["dim"]
    T = h.shape[0]
    pos = torch.arange(past, past + T, device=h.device)
    q, k, v = ((h @ w[f"{n}_proj.weight"].T).view(T, -1, d) for n in "qkv")
    k, v = torch.cat([earlier[0].transpose(0, 1), _rotate(k, pos, 500000.0)]), torch.cat([earlier[1].transpose(0, 1), v])
    return _attend(_rotate(q, pos, 500000.0), k, v, past, d ** -0.5).reshape(T, H * d) @ w["o_proj.weight"].T, (k, v)


def _exact_latent(case, w, h, past, earlier):
    z = SIZES[case["size"]]
    H, R, T = z["latent_heads"], z["kv_rank"], h.shape[0]
    pos = torch.arange(past, past + T, device=h.device)
    q = (_norm(h @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(T, H, NOPE + ROT)
    down = h @ w["dkv"].T
    row = torch.cat([_norm(down[:, :R], w["dkv.norm"]), _rotate(down[:, None, R:], pos, 10000.0)[:, 0]], dim=1)
    row = torch.cat([earlier[0][0], row])
    c, shared = row[:, :R], row[:, None, R:].expand(-1, H, -1)
    k = torch.cat([(c @ w["uk"].T).view(-1, H, NOPE), shared], dim=2)
    q = torch.cat([q[..., :NOPE], _rotate(q[..., NOPE:], pos, 10000.0)], dim=2)
    out = _attend(q, k, (c @ w["uv"].T).view(-1, H, VALUE), past, (NOPE + ROT) ** -0.5).reshape(T, H * VALUE)
    return (out * torch.sigmoid(h @ w["g"].T)) @ w["o"].T, (row[:, None],)


def _exact_matrix(case, w, h, past, state):
    """The mixers with a matrix state, token by token; returns the branch and the state's record."""
    z, kind = SIZES[case["size"]], case["part"]
    H, d, T = z["heads"], z["dim"], h.shape[0]
    q, k, v = ((h @ w[n].T).view(T, H, d) for n in "qkv")
    keep, put = None, torch.ones(T, H, 1, dtype=h.dtype, device=h.device)
    if kind == "retention":
        pos = torch.arange(past, past + T, device=h.device)
        q, k = _rotate(q, pos, 10000.0), _rotate(k, pos, 10000.0) * d ** -0.5
        keep = torch.tensor(_decays(H), dtype=torch.float64, device=h.device)[None, :, None].expand(T, H, 1)
    elif kind == "channel_decay":
        q = q * d ** -0.5
        keep = torch.exp(torch.nn.functional.logsigmoid((h @ w["a1"].T) @ w["a2"].T + w["a2.b"]) / TAU).view(T, H, d)
    S = state
    if kind == "mlstm":
        q = q * d ** -0.5
        m = state[:, d, 0]
        S = state[:, :d]
        log_i = CAP * torch.tanh((h @ w["i"].T + w["i.b"]) / CAP)
        log_f = torch.nn.functional.logsigmoid(CAP * torch.tanh((h @ w["f"].T + w["f.b"]) / CAP))
        v = torch.cat([v, torch.ones_like(v[..., :1])], dim=2)
        keep, put, top = [], [], []
        for t in range(T):
            last, m = m, torch.maximum(log_f[t] + m, log_i[t])
            keep.append(torch.exp(log_f[t] + last - m))
            put.append(torch.exp(log_i[t] - m))
            top.append(m)
        keep, put, top = (torch.stack(x)[..., None] for x in (keep, put, top))
    out = []
    for t in range(T):
        S = keep[t][..., None] * S + (put[t] * k[t])[..., None] * v[t][:, None]
        out.append((S * q[t][..., None]).sum(1))
    o = torch.stack(out)
    if kind == "mlstm":
        o = o[..., :d] / (torch.maximum(o[..., d:].abs(), torch.exp(-top)) + 1e-6)
        S = torch.cat([S, m[:, None, None].expand(-1, 1, d + 1)], dim=1)
    o = _norm(o).reshape(T, H * d)
    if kind != "retention":
        o = o * (w["norm"] if kind == "mlstm" else w["norm"].repeat(H))
    g = h @ w["g"].T
    return (o * (torch.sigmoid(g) if kind == "mlstm" else torch.nn.functional.silu(g))) @ w["o"].T, S


def _exact_delta(case, w, h):
    """The gated delta rule with a decay per key channel, from an empty state; the convolution's last inputs have no value here."""
    z = SIZES[case["size"]]
    H, d, T = z["heads"], z["dim"], h.shape[0]

    def conv(n):
        x = torch.nn.functional.pad(h @ w[n].T, (0, 0, TAPS - 1, 0))
        return torch.nn.functional.silu(sum(w[n + ".conv"][:, j] * x[j:j + T] for j in range(TAPS))).view(T, H, d)
    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k, v = unit(conv("q")) * d ** -0.5, unit(conv("k")), conv("v")
    b = torch.sigmoid(h @ w["b"].T)[..., None]
    a = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus((h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(T, H, d))
    S, out = torch.zeros(H, d, d, dtype=h.dtype, device=h.device), []
    for t in range(T):
        S = a[t][..., None] * S
        u = b[t] * (v[t] - (S * k[t][..., None]).sum(1))
        S = S + k[t][..., None] * u[:, None]
        out.append((S * q[t][..., None]).sum(1))
    o = (_norm(torch.stack(out)) * w["norm"]).reshape(T, H * d)
    return (o * torch.sigmoid((h @ w["g1"].T) @ w["g2"].T)) @ w["o"].T, S


def _exact_experts(case, w, h):
    z = SIZES[case["size"]]
    E, top, T = z["experts"], z["top"], h.shape[0]
    act = torch.nn.functional.gelu
    s = torch.sigmoid(h @ w["router"].T)
    groups = s.view(T, GROUPS, E // GROUPS).topk(2, dim=2).values.sum(2).topk(KEEP, dim=1).indices
    open_ = torch.zeros(T, GROUPS, dtype=torch.bool, device=h.device).scatter_(1, groups, True).repeat_interleave(E // GROUPS, dim=1)
    chosen, ids = s.masked_fill(~open_, -1.0).topk(top, dim=1)
    weights = chosen / (chosen.sum(1, keepdim=True) + 1e-20) * ROUTE_SCALE
    out = torch.sigmoid(h @ w["shared.sg"].T) * (act(h @ w["shared.up"].T) @ w["shared.down"].T)
    for e in range(E):
        row, place = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, row, weights[row, place, None] * (act(h[row] @ w[f"e{e}.up"].T) @ w[f"e{e}.down"].T))
    return out


def _exact_engine(case, seed):
    z = SIZES[case["size"]]
    H, G, d = z["heads"], z["kv"], z["dim"]
    engine = Engine.from_config(_llama(case), seed=int(seed), max_tokens=64, max_batch=1, device=DEVICE)      # its table of weights' names and shapes
    table = engine.model.weight_table()
    engine.close()
    w = {n: t.double() for n, t in random_weights(table, int(seed), torch.bfloat16, DEVICE, 0.02, 0.0).items()}
    prompts, steps = _tokens(case, seed)
    logits = []
    for b, prompt in enumerate(prompts):
        x = w["model.embed_tokens.weight"][torch.tensor(prompt + [s[b] for s in steps], device=DEVICE)]
        T = x.shape[0]
        pos = torch.arange(T, device=DEVICE)
        for i in range(2):
            p = f"model.layers.{i}."
            h = _norm(x, w[p + "input_layernorm.weight"])
            q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].T).view(T, -1, d) for n in "qkv")
            a = _attend(_rotate(q, pos, 500000.0), _rotate(k, pos, 500000.0), v, 0, d ** -0.5).reshape(T, H * d)
            x = x + a @ w[p + "self_attn.o_proj.weight"].T
            h = _norm(x, w[p + "post_attention_layernorm.weight"])
            x = x + (torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        logits.append(_norm(x[len(prompt) - 1:], w["model.norm.weight"]) @ w["lm_head.weight"].T)
    return [torch.stack([sequence[i] for sequence in logits]) for i in range(len(steps) + 1)]


def exact(case, seed):
    if case["part"] == "generate":
        return _exact_engine(case, seed)
    new, past = _lengths(case)
    state = prepare(case, seed)          # the weights' names, and where the cache's pages lie
    w = {n: t.double() for n, t in random_weights(state["part"].weights(), seed, _dtype(case), DEVICE).items()}
    h, out, row = state["h"].double(), [], 0
    kept = [t.double() for t in state["kept"]]
    for b, (n, p) in enumerate(zip(new, past)):
        mine = h[row:row + n]
        row += n
        if case["part"] == "experts":
            out.append(_exact_experts(case, w, mine))
        elif case["part"] == "delta":
            o, kept[0][b] = _exact_delta(case, w, mine)
            out.append(o)
        elif case["part"] in ("attention", "latent"):
            earlier = [t.double() for t in _earlier(case, seed, b, p)]
            o, rows = (_exact_attention if case["part"] == "attention" else _exact_latent)(case, w, mine, p, earlier)
            out.append(o)
            at = torch.arange(n + p, device=h.device)
            page = state["view"].page_table[state["ctx"].h_slots[b]].long()[at // 64]
            for pool, r in zip(kept, rows):
                pool[page, :, at % 64] = r
        else:
            o, kept[0][b] = _exact_matrix(case, w, mine, p, _earlier(case, seed, b, p).double())
            out.append(o)
    out = torch.cat(out)
    if case["part"] == "experts":
        return out
    return [out, kept[0], None] if case["part"] == "delta" else [out, *kept]
