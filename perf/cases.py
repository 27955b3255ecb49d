"""What this library is measured on: requests that a program brings to it, from their token ids to their logits.

A case is one serving of a batch of requests by Falcon-H1 (the layer sizes of bench.py: 1.5B, 3B and 7B, random weights):
the prompts go through LLM.step together, then perhaps a further turn of every conversation, then `new` one-token steps
through the engine's decode step, with the token ids given (as in the replay of a trace or the scoring of a text, so that
one token on the edge between two does not change all that follow it).  A pass acquires its slots and gives them back.

Outputs are the logits of every prompt's last token, those of every turn's last token, the tokens that the decode steps
picked and the logits of the last of them.
"""
import math
import random

import torch

import tinyllama_c_b200 as tlc
from tinyllama_c_b200.config import config_from_dict
from tinyllama_c_b200.engine import EngineBackend
from tinyllama_c_b200.weights import build_model

_COMMON = dict(
    architectures=["FalconH1ForCausalLM"], model_type="falcon_h1", head_dim=128, num_key_value_heads=2, rope_theta=1e11,
    rms_norm_eps=1e-5, mamba_n_groups=1, mamba_d_state=256, mamba_d_conv=4, mamba_chunk_size=128, mamba_conv_bias=True,
    mamba_proj_bias=False, mamba_rms_norm=True, mamba_norm_before_gate=False, embedding_multiplier=5.66,
    lm_head_multiplier=0.039, key_multiplier=0.39, attention_in_multiplier=1.0, attention_out_multiplier=0.94,
    ssm_in_multiplier=1.25, ssm_out_multiplier=0.24, mlp_multipliers=[0.88, 0.3], ssm_multipliers=[0.35, 0.25, 0.7, 0.5, 0.35])
CONFIGS = {
    "1.5B": dict(_COMMON, vocab_size=65536, hidden_size=2048, num_hidden_layers=24, num_attention_heads=8,
                 intermediate_size=4096, max_position_embeddings=4096, tie_word_embeddings=True, mamba_d_ssm=3072,
                 mamba_n_heads=48, mamba_d_head=64),
    "3B": dict(_COMMON, vocab_size=65536, hidden_size=2560, num_hidden_layers=32, num_attention_heads=10,
               intermediate_size=8192, max_position_embeddings=4096, tie_word_embeddings=True, mamba_d_ssm=4096,
               mamba_n_heads=32, mamba_d_head=128),
    "7B": dict(_COMMON, vocab_size=130048, hidden_size=3072, num_hidden_layers=44, num_attention_heads=12,
               intermediate_size=12288, max_position_embeddings=8320, tie_word_embeddings=False, mamba_d_ssm=3072,
               mamba_n_heads=24, mamba_d_head=128),
}
STEP_TOKENS = 8192            # prompts share a step up to this many tokens, as in LLM.generate


def _case(name, size, batch, lo, hi, new, turn=0, sampled=False, dtype="bfloat16"):
    """Prompts of lo..hi tokens; `turn`: up to this many tokens a further turn brings; `sampled`: temperature, top-k, top-p,
    min-p and repeat penalty (the command line's defaults) in place of the largest logit."""
    case = dict(size=size, batch=batch, lo=lo, hi=hi, turn=turn, new=new, sampled=sampled, dtype=dtype)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user's chat: a short prompt, an answer token by token
        _case("chat-1", "1.5B", 1, 96, 96, 32),
        # the benchmark's serving point: eight requests of 512 tokens
        _case("chat-8", "1.5B", 8, 512, 512, 32),
        # a full server: 64 short unequal requests, sampled as the command line does by default
        _case("serve-64-sampled", "1.5B", 64, 16, 128, 12, sampled=True),
        # two long documents, a short answer to each: decoding far from the start of the context
        _case("documents-2", "1.5B", 2, 3300, 3800, 32),
        # conversations that go on: prompts, then a turn of a few dozen tokens each, then the answer
        _case("turns-6", "1.5B", 6, 200, 700, 16, turn=90),
        # the smallest call: the first token after a handful of tokens
        _case("prompt-23", "1.5B", 1, 23, 23, 0),
        # an ordinary question, of a size that fills no tile
        _case("prompt-333", "1.5B", 1, 333, 333, 0),
        # the benchmark's prompt
        _case("prompt-2048", "1.5B", 1, 2048, 2048, 0),
        # the middle model's workload: 16 unequal prompts, sampled answers
        _case("ragged-16-3b", "3B", 16, 64, 1100, 20, sampled=True),
        # the largest model serving a batch
        _case("serve-32-7b", "7B", 32, 24, 100, 10),
        # the largest model reading a long text
        _case("prompt-8192-7b", "7B", 1, 8192, 8192, 0),
        # true 32-bit arithmetic, for checks of a model against other implementations
        _case("float32-2", "1.5B", 2, 60, 250, 10, dtype="float32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chat", "serve", "document", "turns", "prompt", "ragged", "float32"])
    size = rng.choice(["1.5B", "1.5B", "1.5B", "3B", "7B"])
    new = rng.randint(6, 32) if size == "1.5B" else rng.randint(4, 12)
    sampled = rng.random() < 0.4
    if kind == "chat":
        batch, n = _log_int(rng, 1, 16), _log_int(rng, 16, 512)
        return _case(None, size, batch, max(1, n // 2), n, new, sampled=sampled)
    if kind == "serve":
        batch = rng.randint(17, 64)
        lo = _log_int(rng, 4, 40)
        return _case(None, size, batch, lo, lo + rng.randint(1, 80), min(new, 12), sampled=sampled)
    if kind == "document":
        n = _log_int(rng, 1500, 3900)
        return _case(None, size, rng.randint(1, 2), n - 100, n, min(new, 16), sampled=sampled)
    if kind == "turns":
        n = _log_int(rng, 32, 900)
        return _case(None, size, rng.randint(1, 8), max(1, n // 3), n, min(new, 16), turn=_log_int(rng, 1, 300))
    if kind == "prompt":
        n = _log_int(rng, 5, 4000 if size != "7B" else 8100)
        return _case(None, size, 1, n, n, 0)
    if kind == "ragged":
        hi = _log_int(rng, 100, 1800)
        return _case(None, size, rng.randint(3, 6 if hi > 700 else 14), max(1, hi // 20), hi, min(new, 12), sampled=sampled)
    return _case(None, "1.5B", rng.randint(1, 4), 5, _log_int(rng, 12, 300), rng.randint(2, 10), dtype="float32")


def _lengths(case):
    """The prompts' and the turns' lengths: a property of the case, not of the seed."""
    r = random.Random("%s %s %s" % (case["batch"], case["lo"], case["hi"]))
    prompts = [r.randint(case["lo"], case["hi"]) for _ in range(case["batch"])]
    return prompts, [r.randint(1, case["turn"]) for _ in prompts] if case["turn"] else []


def _sizes(c):
    D, H, KV, hd = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    Di, Hs, G, N = c["mamba_d_ssm"], c["mamba_n_heads"], c["mamba_n_groups"], c["mamba_d_state"]
    return D, H, KV, hd, Di, Hs, c["mamba_d_head"], G, N, Di + 2 * G * N, c["intermediate_size"], c["vocab_size"], c["num_hidden_layers"]


def _weights(case, seed):
    """Random weights by tensor name: matrices N(0, 0.02) in bfloat16, norms around 1, the state-space constants over the
    ranges that trained models have (A in 1..16, time steps in 1e-3..0.1)."""
    c = CONFIGS[case["size"]]
    D, H, KV, hd, Di, Hs, P, G, N, Cd, F, V, L = _sizes(c)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev, W = dict(device="cuda"), {}

    def normal(name, *shape, mean=0.0, std=0.02, dtype=torch.bfloat16):
        W[name] = torch.empty(shape, dtype=dtype, **dev).normal_(mean, std, generator=g)

    def uniform(*shape):
        return torch.rand(shape, generator=g, **dev)

    normal("model.embed_tokens.weight", V, D)
    if not c["tie_word_embeddings"]:
        normal("lm_head.weight", V, D)
    normal("model.final_layernorm.weight", D, mean=60.0, std=6.0)     # logits that spread over a few units, as trained ones do
    for l in range(L):
        p = "model.layers.%d." % l
        for n in ("input_layernorm", "pre_ff_layernorm"):
            normal(p + n + ".weight", D, mean=1.0, std=0.1)
        for n, rows, cols in (("q", H * hd, D), ("k", KV * hd, D), ("v", KV * hd, D), ("o", D, H * hd)):
            normal(p + "self_attn.%s_proj.weight" % n, rows, cols)
        for n, rows, cols in (("gate", F, D), ("up", F, D), ("down", D, F)):
            normal(p + "feed_forward.%s_proj.weight" % n, rows, cols)
        normal(p + "mamba.in_proj.weight", Di + Cd + Hs, D)
        normal(p + "mamba.out_proj.weight", D, Di)
        normal(p + "mamba.conv1d.weight", Cd, 1, c["mamba_d_conv"], std=0.3)
        normal(p + "mamba.conv1d.bias", Cd)
        normal(p + "mamba.norm.weight", Di, mean=1.0, std=0.1)
        W[p + "mamba.A_log"] = torch.log(1.0 + 15.0 * uniform(Hs))
        dt = torch.exp(uniform(Hs) * (math.log(0.1) - math.log(1e-3)) + math.log(1e-3))
        W[p + "mamba.dt_bias"] = dt + torch.log(-torch.expm1(-dt))
        normal(p + "mamba.D", Hs, mean=1.0, std=0.1, dtype=torch.float32)
    return W


def _tokens(case, seed):
    """Every sequence's token ids: its prompt, its turn and the ids that its decode steps bring."""
    prompts, turns = _lengths(case)
    r = random.Random("tokens %d" % seed)
    V = CONFIGS[case["size"]]["vocab_size"]
    ids = lambda n: [r.randrange(V) for _ in range(n)]  # noqa: E731
    return [ids(n) for n in prompts], [ids(n) for n in turns], [ids(case["new"]) for _ in prompts]


def _params(case, seed):
    return tlc.SamplingParams(seed=seed) if case["sampled"] else tlc.GREEDY


def prepare(case, seed):
    """A program's model with its cache, its requests, and the decode step captured for this batch (as a server has it
    after its first request)."""
    config = config_from_dict(dict(CONFIGS[case["size"]]))
    model = build_model(config)
    model.bind(_weights(case, seed), getattr(torch, case["dtype"]), torch.device("cuda:0"))
    prompts, turns, forced = _tokens(case, seed)
    total = [len(p) + (len(turns[i]) if turns else 0) + case["new"] for i, p in enumerate(prompts)]
    llm = tlc.LLM(model, dtype=case["dtype"], max_tokens=sum(-(-n // 64) * 64 for n in total) + 64, max_seqs=case["batch"] + 1)
    graphs = {}
    state = dict(llm=llm, graphs=graphs, backend=EngineBackend(llm.model, llm.cache, _params(case, seed), graphs, True),
                 prompts=prompts, turns=turns, forced=forced)
    if case["new"]:
        run(state)
    return state


def _step_all(llm, slots, tokens):
    """Unequal rows of tokens in steps of at most STEP_TOKENS (a single sequence may be longer); the last tokens' logits."""
    out, i = [], 0
    while i < len(slots):
        j, n = i + 1, len(tokens[i])
        while j < len(slots) and n + len(tokens[j]) <= STEP_TOKENS:
            n += len(tokens[j])
            j += 1
        out.append(llm.step([tlc.StepEntry(s, t, (len(t) - 1,)) for s, t in zip(slots[i:j], tokens[i:j])]))
        i = j
    return out[0] if len(out) == 1 else torch.cat(out)


def run(state):
    llm, backend = state["llm"], state["backend"]
    prompts, turns, forced = state["prompts"], state["turns"], state["forced"]
    B = len(prompts)
    slots = [llm.cache.acquire() for _ in range(B)]
    out = {"prompt": _step_all(llm, slots, prompts)}
    seen = [list(p) for p in prompts]
    if turns:
        out["turn"] = _step_all(llm, slots, turns)
        for s, t in zip(seen, turns):
            s.extend(t)
    picked = []
    for k in range(len(forced[0])):
        entries = [(slot, [f[k]]) for slot, f in zip(slots, forced)]
        for s, f in zip(seen, forced):
            s.append(f[k])
        picked.append(backend.decode_step(entries, seen, range(B), [k] * B))
    if picked:
        out["picked"] = torch.tensor(picked, dtype=torch.int32)
        # (the graph of the last step: the one for the longest context that was captured)
        graph = max(state["graphs"].values(), key=lambda g: g.max_context)
        out["last"] = graph.logits[:B].clone()
    for s in slots:
        llm.cache.release(s)
    return out


def _layer_weights(c):
    D, H, KV, hd, Di, Hs, P, G, N, Cd, F, V, L = _sizes(c)
    return D * (H + 2 * KV) * hd + H * hd * D + D * (Di + Cd + Hs) + Di * D + 3 * D * F


def work(case):
    """Every step reads the weights once, the live keys and values (in their stored type) and the sequences' states, and
    writes the new ones and the logits that are asked for."""
    c = CONFIGS[case["size"]]
    D, H, KV, hd, Di, Hs, P, G, N, Cd, F, V, L = _sizes(c)
    size = 4 if case["dtype"] == "float32" else 2
    prompts, turns = _lengths(case)
    matrices = L * _layer_weights(c)
    state = L * (Hs * P * N + (c["mamba_d_conv"] - 1) * Cd) * 4
    kv = L * 2 * KV * hd * size
    nbytes = flops = 0

    def step(starts, lens):
        nonlocal nbytes, flops
        T, B = sum(lens), len(lens)
        nbytes += (matrices + V * D) * size + kv * (sum(starts) + T) + state * (B + sum(s > 0 for s in starts)) + B * V * 4
        flops += 2 * T * matrices + 2 * B * V * D + L * T * Hs * P * N * 6
        flops += L * 4 * H * hd * sum(n * s + n * (n + 1) // 2 for s, n in zip(starts, lens))

    i = 0
    while i < len(prompts):
        j, n = i + 1, prompts[i]
        while j < len(prompts) and n + prompts[j] <= STEP_TOKENS:
            n += prompts[j]
            j += 1
        step([0] * (j - i), prompts[i:j])
        i = j
    at = list(prompts)
    if turns:
        step(at, turns)
        at = [a + t for a, t in zip(at, turns)]
    for _ in range(case["new"]):
        step(at, [1] * len(at))
        at = [a + 1 for a in at]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the path was measured to be off 64-bit arithmetic (bfloat16: 0.007 to 0.015, largest value 0.07; 32
    bits: 4e-6, largest value 1.7e-5), and what other kernels of the same precision change among the picked tokens: with
    two logits as near to each other as that another one is picked, 1 to 4 in 100 greedy and up to 10 in 100 sampled ones."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 8e-5, "differ": 0.05}
    return {"rel": 5e-2, "max": 0.25, "differ": 0.4}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _attention64(c, q, k, v):
    """Causal attention of [B, T, heads, hd]; the rotation's angle is a 32-bit product of position and frequency, as every
    32-bit engine has it."""
    B, T, H, hd = q.shape
    KV = k.shape[2]
    inv = (1.0 / torch.pow(torch.tensor(float(c["rope_theta"]), dtype=torch.float64),
                           torch.arange(hd // 2, dtype=torch.float64) * 2 / hd)).float().to(q.device)
    ang = (torch.arange(T, device=q.device, dtype=torch.float32)[:, None] * inv).double()
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def turn(x):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    q, k = turn(q), turn(k)
    out = torch.empty_like(q)
    rows = max(1, min(T, (1 << 27) // max(1, T * B * (H // KV))))
    for g in range(KV):
        heads = slice(g * H // KV, (g + 1) * H // KV)
        kg, vg = k[:, :, g], v[:, :, g]
        for t in range(0, T, rows):
            e = min(T, t + rows)
            s = torch.einsum("bthd,bsd->bhts", q[:, t:e, heads], kg[:, :e]) / math.sqrt(hd)
            hidden = torch.arange(e, device=q.device)[None, :] > torch.arange(t, e, device=q.device)[:, None]
            out[:, t:e, heads] = torch.einsum("bhts,bsd->bthd", s.masked_fill_(hidden, -math.inf).softmax(-1), vg[:, :e])
    return out.reshape(B, T, H * hd)


def _scan64(x, Bm, Cm, dt, A, Dskip, chunk=64):
    """y of S <- S exp(dt A) + (dt x) B, y = S C + D x, a chunk of rows at a time; x [B, T, heads, P], B and C [B, T, N]."""
    B, T, Hs, P = x.shape
    S = x.new_zeros(B, Hs, P, Bm.shape[-1])
    y = torch.empty_like(x)
    for t in range(0, T, chunk):
        e = min(T, t + chunk)
        xc, bc, cc, dc = x[:, t:e], Bm[:, t:e], Cm[:, t:e], dt[:, t:e]
        cum = torch.cumsum(dc * A, 1)                                                 # [B, q, heads]
        gap = (cum[:, :, None] - cum[:, None]).permute(0, 3, 1, 2)                    # [B, heads, q, q]
        M = torch.exp(torch.where(torch.ones_like(gap, dtype=torch.bool).tril(), gap, -math.inf)) * (cc @ bc.transpose(1, 2))[:, None]
        xd = xc * dc[..., None]
        y[:, t:e] = torch.einsum("bhqs,bshp->bqhp", M, xd) + torch.einsum("bqn,bhpn->bqhp", cc, S) * cum.exp()[..., None]
        left = torch.exp(cum[:, -1:] - cum)                                           # from each row to the chunk's end
        S = S * cum[:, -1].exp()[:, :, None, None] + torch.einsum("bqhp,bqn->bhpn", xd * left[..., None], bc)
    return y + x * Dskip[:, None]


def _logits64(case, W, rows, wanted):
    """Logits of the wanted positions of every row of token ids, whole sequences at a time; rows padded at their ends."""
    c = CONFIGS[case["size"]]
    D, H, KV, hd, Di, Hs, P, G, N, Cd, F, V, L = _sizes(c)
    eps, d = c["rms_norm_eps"], torch.float64
    w = lambda name: W[name].to(d)  # noqa: E731
    silu = torch.nn.functional.silu
    T = max(len(r) for r in rows)
    ids = torch.tensor([r + [0] * (T - len(r)) for r in rows], device="cuda")
    x = W["model.embed_tokens.weight"][ids].to(d) * c["embedding_multiplier"]
    B = len(rows)
    m = c["ssm_multipliers"]
    for l in range(L):
        p = "model.layers.%d." % l
        n = _rms(x, w(p + "input_layernorm.weight"), eps)
        na = n * c["attention_in_multiplier"]
        q, k, v = ((na @ w(p + "self_attn.%s_proj.weight" % s).T).view(B, T, -1, hd) for s in "qkv")
        x = x + _attention64(c, q, k * c["key_multiplier"], v) @ w(p + "self_attn.o_proj.weight").T * c["attention_out_multiplier"]
        del q, k, v
        z, xs, bs, cs, dt = (n * c["ssm_in_multiplier"] @ w(p + "mamba.in_proj.weight").T).split([Di, Di, N, N, Hs], -1)
        u = torch.cat([xs * m[1], bs * m[2], cs * m[3]], -1).transpose(1, 2)
        u = torch.nn.functional.conv1d(torch.nn.functional.pad(u, (c["mamba_d_conv"] - 1, 0)), w(p + "mamba.conv1d.weight"),
                                       w(p + "mamba.conv1d.bias"), groups=Cd)
        xs, bs, cs = silu(u).transpose(1, 2).split([Di, N, N], -1)
        y = _scan64(xs.reshape(B, T, Hs, P), bs, cs, torch.nn.functional.softplus(dt * m[4] + w(p + "mamba.dt_bias")),
                    -torch.exp(w(p + "mamba.A_log")), w(p + "mamba.D")).reshape(B, T, Di)
        y = _rms(y * silu(z * m[0]), w(p + "mamba.norm.weight"), eps)
        x = x + y @ w(p + "mamba.out_proj.weight").T * c["ssm_out_multiplier"]
        del z, xs, bs, cs, u, y, n, na
        n = _rms(x, w(p + "pre_ff_layernorm.weight"), eps)
        a = silu(n @ w(p + "feed_forward.gate_proj.weight").T * c["mlp_multipliers"][0]) * (n @ w(p + "feed_forward.up_proj.weight").T)
        x = x + a @ w(p + "feed_forward.down_proj.weight").T * c["mlp_multipliers"][1]
        del n, a
    at = [(b, t) for b, ts in enumerate(wanted) for t in ts]
    f = _rms(x[[b for b, _ in at], [t for _, t in at]], w("model.final_layernorm.weight"), eps)
    return f @ w("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight").T * c["lm_head_multiplier"]


def exact(case, seed):
    W = _weights(case, seed)
    prompts, turns, forced = _tokens(case, seed)
    keys = ["prompt"] + ["turn"] * bool(turns) + ["last"] * bool(case["new"])
    rows, wanted = [], []
    for i, p in enumerate(prompts):
        t = turns[i] if turns else []
        rows.append(p + t + forced[i])
        ends = {"prompt": len(p), "turn": len(p) + len(t), "last": len(rows[-1])}
        wanted.append([ends[k] - 1 for k in keys])
    got, at = [None] * len(rows), 0
    order = sorted(range(len(rows)), key=lambda i: len(rows[i]))
    while at < len(order):                          # rows of like lengths together, as many as memory allows
        n = 1
        while at + n < len(order) and (n + 1) * len(rows[order[at + n]]) <= 8192:
            n += 1
        some = order[at:at + n]
        y = _logits64(case, W, [rows[i] for i in some], [wanted[i] for i in some]).view(n, len(keys), -1)
        for k, i in enumerate(some):
            got[i] = y[k]
        at += n
    y = torch.stack(got)
    out = {key: y[:, k] for k, key in enumerate(keys)}
    if case["new"]:
        out["picked"] = None
    return out
