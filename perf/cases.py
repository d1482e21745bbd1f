"""What is timed: steps of the models that this package runs, through ``load_model``, ``CacheManager`` and ``ModelRunner``.

Kinds of a case (``"kind"``):

  prompt   requests are opened, ONE step takes all their prompts (ragged lengths) and returns every prompt's last logits, and they
           are closed: the time to the first token.
  decode   requests whose contexts are cached take one token each in one step: what a generating server does most of the time.
           After the step every request is set back to its context, as a program that tries several continuations does.
  mixed    one request's next prompt portion beside one token of every other request, in one step: chunked prefill under load.
  turn     a short conversation turn: open, one step with all prompts, ``steps`` decode steps of given tokens, close.  For models
           that hold recurrent states, where a step cannot be taken back, this is also how decoding is timed.

Weights are the package's seeded random ones (``load_model(config, random_seed=...)``), token ids uniform-random, as in the
package's own benchmark.  ``exact`` draws the same weights and computes the logits of whole sequences in 64 bits with plain torch.

Models with routed experts are not among the cases: a near tie in a router sends a token to another expert when a sum is rounded
differently, and the logits of two correct implementations are then not comparable.
"""
import hashlib
import math

import torch

from mini_hisparse_b200 import CacheConfig, CacheManager, load_model
from mini_hisparse_b200.engine import ModelRunner, StepEntry

DEVICE = "cuda:0"

# width, heads, kv heads, head size, feed-forward width, vocabulary
SHAPES = {
    "tiny-a": (64, 4, 2, 16, 176, 512),            # the package's smallest test configuration
    "tiny-b": (96, 3, 1, 32, 256, 1000),           # the second one
    "1k": (1024, 16, 4, 64, 4096, 32000),          # a generic small model with heads of 64
    "2k": (2048, 16, 4, 128, 8192, 32000),         # the two sizes at which the package compares its designs
    "4k": (4096, 32, 8, 128, 14336, 32000),
    "7b": (3584, 28, 4, 128, 18944, 152064),       # the shape of the package's headline benchmark
    "14b": (5120, 40, 8, 128, 13824, 152064),      # the shapes of its two serving workloads
    "32b": (5120, 40, 8, 128, 27648, 152064),
}


def listed():
    return [
        # the smallest calls: a tiny float32 model answers four prompts of very different lengths; launches and host work count
        case("tiny chat float32", "qwen2", "tiny-b", 3, "float32", "turn", batch=4, context=257, spread=1.0, steps=24, page=32),
        # one user, long context: every weight is read for one token
        case("decode 1 x 4096", "qwen2", "7b", 8, "bfloat16", "decode", batch=1, context=4096),
        # the headline: eight users with about 4,096 tokens each
        case("decode 8 x 4096", "qwen2", "7b", 8, "bfloat16", "decode", batch=8, context=4096, spread=0.1),
        # a busy server: 64 users, contexts from a few hundred to 2,400 tokens
        case("decode 64 x 2400", "qwen2", "7b", 8, "bfloat16", "decode", batch=64, context=2400, spread=0.8),
        # the time to the first token of a 2,048-token prompt
        case("prompt 2048", "qwen2", "7b", 8, "bfloat16", "prompt", batch=1, context=2048),
        # the 14B serving mix: a portion of 512 tokens beside 31 users who are generating
        case("portion 512 beside 31", "qwen2", "14b", 4, "bfloat16", "mixed", batch=32, context=2800, spread=0.9, tokens=512),
        # the 32B long-prompt workload: the last portion of an 8,192-token prompt
        case("portion 2048 at 6144", "qwen2", "32b", 2, "bfloat16", "mixed", batch=1, context=6144, tokens=2048),
        # the 32-bit path at full width: three ragged prompts
        case("prompts 3 x 250 float32", "qwen2", "7b", 2, "float32", "prompt", batch=3, context=250, spread=0.5),
        # the other designs at the sizes of their comparison: first tokens, and turns in which decoding has the larger part
        case("koronex prompt 2048", "koronex", "4k", 8, "bfloat16", "prompt", batch=1, context=2048),
        case("koronex turn 8 x 300", "koronex", "2k", 8, "bfloat16", "turn", batch=8, context=300, spread=0.6, steps=24),
        case("dotivik turn 4 x 700", "dotivik", "2k", 8, "bfloat16", "turn", batch=4, context=700, spread=0.5, steps=16),
        case("zetenex prompts 3 x 1000", "zetenex", "2k", 8, "bfloat16", "prompt", batch=3, context=1000, spread=0.7),
    ]


def case(name, model, shape, layers, dtype, kind, batch, context, spread=0.0, tokens=0, steps=0, page=16):
    """``context``: the longest prompt or cached context; request i of ``batch`` has it less its share of ``spread`` of it."""
    c = dict(model=model, shape=shape, layers=layers, dtype=dtype, kind=kind, batch=batch, context=context, spread=spread,
             tokens=tokens, steps=steps, page=page)
    return dict(name=name, **c) if name else c


def draw(rng):
    """Another case of the same ranges: batches of 1 to 64, contexts of tens to thousands, odd lengths, every kind and model."""
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    page = rng.choice((16, 16, 16, 32, 64))
    spread = round(rng.uniform(0.0, 0.9), 2)
    what = rng.choice(("tiny", "decode", "decode", "prompt", "mixed", "float32", "design", "design"))
    if what == "tiny":
        return case("", "qwen2", rng.choice(("tiny-a", "tiny-b")), rng.randint(2, 4), rng.choice(("float32", "float32", "bfloat16")), "turn",
                    batch=rng.randint(1, 6), context=log(5, 250), spread=spread, steps=rng.randint(4, 24), page=page)
    if what == "decode":
        shape, batch = rng.choice(("7b", "7b", "1k", "4k")), log(1, 64)
        return case("", "qwen2", shape, rng.randint(2, 8), "bfloat16", "decode", batch=batch,
                    context=log(64, min(8000, 100000 // batch)), spread=spread, page=page)
    if what == "prompt":
        batch = rng.randint(1, 4)
        return case("", "qwen2", rng.choice(("7b", "1k", "4k")), rng.randint(2, 6), "bfloat16", "prompt", batch=batch,
                    context=log(40, 2048 // batch), spread=spread, page=page)
    if what == "mixed":
        shape, tokens, batch = rng.choice(("14b", "32b", "4k", "1k")), log(64, 2000), log(1, 32)
        return case("", "qwen2", shape, 2, "bfloat16", "mixed", batch=batch, context=log(300, min(6000, 60000 // batch)),
                    spread=spread, tokens=tokens, page=page)
    if what == "float32":
        return case("", "qwen2", rng.choice(("1k", "2k", "7b")), 2, "float32", rng.choice(("prompt", "turn")), batch=rng.randint(1, 4),
                    context=log(30, 250), spread=spread, steps=8, page=page)
    batch, kind = rng.randint(1, 8), rng.choice(("prompt", "turn"))
    return case("", rng.choice(("koronex", "dotivik", "zetenex")), rng.choice(("2k", "2k", "4k")), 8, "bfloat16", kind, batch=batch,
                context=log(40, (2048 if kind == "prompt" else 1600) // batch), spread=spread,
                steps=rng.randint(8, 24) if kind == "turn" else 0, page=page)


# ---- the calls -------------------------------------------------------------------------------------------------------------------
def lengths(c):
    """Prompt or context lengths of a case's requests, longest first, with odd ones among them."""
    n = c["batch"]
    return [max(1, int(c["context"] * (1.0 - c["spread"] * i / max(1, n - 1)))) for i in range(n)]


def new_tokens(c):
    """Tokens of every request in the timed steps behind its context."""
    if c["kind"] == "prompt":
        return [0] * c["batch"]
    if c["kind"] == "turn":
        return [c["steps"]] * c["batch"]
    return [c["tokens"] if c["kind"] == "mixed" and i == 0 else 1 for i in range(c["batch"])]


def token_ids(c, seed):
    """Per request: the ids of its prompt or context, and those that follow."""
    g = torch.Generator().manual_seed(seed)
    vocab = SHAPES[c["shape"]][5]
    both = [(n, m) for n, m in zip(lengths(c), new_tokens(c))]
    return [(torch.randint(0, vocab, (n,), generator=g).tolist(), torch.randint(0, vocab, (m,), generator=g).tolist()) for n, m in both]


def prepare(c, seed):
    model = load_model(config_of(c), device=DEVICE, dtype=c["dtype"], random_seed=seed)
    ids = token_ids(c, seed)
    pages = sum(-(-(len(a) + len(b)) // c["page"]) + 1 for a, b in ids)
    cache = CacheManager(model.cache_needs, CacheConfig(num_pages=pages, page_size=c["page"], max_requests=c["batch"],
                                                        dtype=model.rt.dtype, device=DEVICE))
    runner = ModelRunner(model, cache)
    if c["kind"] in ("decode", "mixed"):
        for i, (context, _) in enumerate(ids):
            cache.open(i)
            for at in range(0, len(context), 2048):
                runner.step([StepEntry(i, context[at:at + 2048], [])])
    return dict(case=c, runner=runner, cache=cache, ids=ids)


def run(state):
    c, runner, cache, ids = state["case"], state["runner"], state["cache"], state["ids"]
    if c["kind"] in ("decode", "mixed"):
        logits = runner.step([StepEntry(i, new, [len(new) - 1]) for i, (_, new) in enumerate(ids)])
        for i, (context, _) in enumerate(ids):
            cache.requests[i].length = len(context)
        return logits
    for i in range(len(ids)):
        cache.open(i)
    logits = runner.step([StepEntry(i, prompt, [len(prompt) - 1]) for i, (prompt, _) in enumerate(ids)])
    if c["kind"] == "turn":
        rows = [logits.clone()]          # a step's logits are overwritten by the next one
        for s in range(c["steps"]):
            rows.append(runner.step([StepEntry(i, [new[s]], [0]) for i, (_, new) in enumerate(ids)]).clone())
        logits = torch.stack(rows)
    for i in range(len(ids)):
        cache.close(i)
    return logits


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def work(c):
    cfg, size = config_of(c), 2 if c["dtype"] == "bfloat16" else 4
    steps = 1 + (c["steps"] if c["kind"] == "turn" else 0)
    vocab = SHAPES[c["shape"]][5]
    table = {name: math.prod(t[0]) for name, t in tensors(c["model"], cfg).items()}
    head = table.pop("lm_head.weight" if c["model"] == "qwen2" else "head", None)
    gathered = [table.pop(n) for n in ("model.embed_tokens.weight", "embed", "side.embed") if n in table]
    head = head or gathered[0]                                  # a tied head is read whole
    runs = [sum(n for name, n in table.items() if name.startswith(prefix_of(c["model"], i))) for i in layer_runs(cfg)]
    rest = sum(n for name, n in table.items() if not any(name.startswith(prefix_of(c["model"], i)) for i in set(layer_runs(cfg))))
    weights = sum(runs) + rest
    ids = list(zip(lengths(c), new_tokens(c)))
    if c["kind"] in ("prompt", "turn"):
        segments = [[(0, n) for n, _ in ids]] + [[(n + s, 1) for n, _ in ids] for s in range(steps - 1)]
    else:
        segments = [ids]
    bytes_, flops = 0.0, 0.0
    for seg in segments:
        n = sum(m for _, m in seg)
        bytes_ += size * (weights + head) + 4 * len(seg) * vocab
        flops += 2.0 * weights * n + 2.0 * head * len(seg)
        for heads, key, value, row, window in attentions(c["model"], cfg):
            for start, m in seg:
                seen = min(start + m, window + m)
                bytes_ += size * row * (seen + (m if start else 0))
                pairs = m * start + m * (m + 1) / 2 if start + m <= window else m * min(window, start + m / 2)
                flops += 2.0 * heads * (key + value) * pairs
        state = recurrent_state(c["model"], cfg)
        bytes_ += 2 * 4 * state * len(seg)
        flops += 5.0 * state * n
    return dict(bytes=bytes_, flops=flops)


def attentions(model, cfg):
    """(heads, key width, value width, numbers cached per position, window) of every attention layer run."""
    out, far = [], 1 << 30
    if model == "qwen2":
        d = cfg["head_dim"]
        return [(cfg["num_attention_heads"], d, d, 2 * cfg["num_key_value_heads"] * d, far)] * cfg["num_hidden_layers"]
    for i in layer_runs(cfg):
        kind, m = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"]
        m = m["left"] if kind == "parallel" else m
        if kind in ("lightning", "mingru"):
            continue
        window = (m.get("mask") or {}).get("size", far)
        if kind == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            out.append((m["heads"], row, m["kv_rank"], row, window))
        else:
            maps = 2 if model == "dotivik" else 1
            out.append((m["heads"] * maps, m["dim"], m["vdim"], m["kv_heads"] * (maps * m["dim"] + m["vdim"]), window))
    return out


def recurrent_state(model, cfg):
    """Numbers of recurrent state of one request over all layer runs."""
    n = 0
    for i in layer_runs(cfg) if model != "qwen2" else ():
        kind, m = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"]
        n += {"lightning": lambda: m["heads"] * m["dim"] * m["vdim"], "mingru": lambda: m["width"],
              "parallel": lambda: m["right"]["inner"] * m["right"]["state"]}.get(kind, lambda: 0)()
    return n


def tolerance(c):
    """bfloat16: the package's logits lie 0.004 to 0.019 from exact()'s (every product's operands are rounded to 8 bits, layer by
    layer), so two correct implementations differ by up to 0.027.  float32: 3e-7 to 7e-6 from it, by the length of the sums."""
    return {"rel": 3e-5, "max": 1e-3} if c["dtype"] == "float32" else {"rel": 0.03, "max": 0.5}


# ---- configurations --------------------------------------------------------------------------------------------------------------
def config_of(c):
    width, heads, kv_heads, dim, ff, vocab = SHAPES[c["shape"]]
    layers, scale = c["layers"], dim ** -0.5
    dense = dict(kind="dense", ff=ff)
    if c["model"] == "qwen2":
        return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", vocab_size=vocab, hidden_size=width, intermediate_size=ff,
                    num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim, rms_norm_eps=1e-6,
                    rope_theta=1e6, tie_word_embeddings=c["shape"] == "tiny-a", max_position_embeddings=32768)
    if c["model"] == "koronex":       # one lightning layer, two windowed attention layers and one that reads the second's keys
        att = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, mask=dict(size=1024), rot=dict(dims=dim // 2, base=10000.0), scale=scale)
        decay = [1.0 - 2.0 ** (-(3 + 5 * h / (heads - 1))) for h in range(heads)]
        light = dict(type="lightning", mixer=dict(heads=heads, dim=dim, vdim=dim, decay=decay), mlp=dense)
        out = [light if i % 4 == 0 else dict(type="attention", mixer=dict(att, kv_from=i - 1) if i % 4 == 3 else att, mlp=dense)
               for i in range(layers)]
        return dict(architecture="Koronex", vocab=vocab, width=width, embedding=dict(scale=1.0), norm=dict(eps=1e-5), postln_alpha=1.0,
                    token_side=dict(dim=64), layers=out)
    repeat = 2                        # layers in the middle that run twice
    stored = layers - repeat
    loop = dict(start=(stored - repeat) // 2, stop=(stored - repeat) // 2 + repeat, times=2)
    if c["model"] == "dotivik":       # latent attention and attention with two score maps
        lat = dict(heads=heads, dim=dim, rot_dim=32, vdim=dim, kv_rank=96, scale=(dim + 32) ** -0.5, mask=dict(size=1024),
                   rot=dict(dims=32, base=10000.0))
        att = dict(heads=heads // 2, kv_heads=kv_heads // 2, dim=dim // 2, vdim=dim, scale=(dim // 2) ** -0.5, softcap=50.0, diff=0.5,
                   rot=dict(dims=dim // 2, base=10000.0))
        out = [dict(type="attention" if i % 3 == 1 else "latent_attention", mixer=att if i % 3 == 1 else lat, mlp=dense) for i in range(stored)]
        return dict(architecture="Dotivik", vocab=vocab, width=width, norm=dict(eps=1e-5), layers=out, loop=loop)
    par = dict(left=dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, scale=scale, q_temp=dict(coef=0.1, every=1024)), left_scale=0.7,
               right=dict(inner=width, state=16, dt_rank=width // 16, conv=4), right_scale=0.7)
    out = [dict(type="mingru" if i % 3 else "parallel", mixer=dict(width=width) if i % 3 else par, mlp=dense) for i in range(stored)]
    return dict(architecture="Zetenex", vocab=vocab, width=width, norm=dict(eps=1e-5), canon=dict(taps=4),
                embedding=dict(scale=float(width) ** 0.5), layers=out, loop=loop)


def layer_runs(cfg):
    """The layers in the order in which they run."""
    n, loop = cfg.get("num_hidden_layers") or len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return list(range(n))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def prefix_of(model, i):
    return f"model.layers.{i}." if model == "qwen2" else f"l{i}."


def tensors(model, cfg):
    """{checkpoint name: (shape, mean, standard deviation, whether it is a matrix in the compute dtype)}."""
    def matrix(*shape, std=0.02):
        return (shape, 0.0, std, True)

    def vector(*shape, mean=0.0, std=0.02):
        return (shape, mean, std, False)

    def weight(n):
        return vector(n, mean=1.0, std=0.1)

    t = {}
    if model == "qwen2":
        H, I, V, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
        q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
        t["model.embed_tokens.weight"] = matrix(V, H)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            t[p + "input_layernorm.weight"] = t[p + "post_attention_layernorm.weight"] = weight(H)
            for n, rows in (("q", q), ("k", kv), ("v", kv)):
                t[p + f"self_attn.{n}_proj.weight"], t[p + f"self_attn.{n}_proj.bias"] = matrix(rows, H), vector(rows)
            t[p + "self_attn.o_proj.weight"] = matrix(H, q)
            t[p + "mlp.gate_proj.weight"] = t[p + "mlp.up_proj.weight"] = matrix(I, H)
            t[p + "mlp.down_proj.weight"] = matrix(H, I)
        t["model.norm.weight"] = weight(H)
        if not cfg["tie_word_embeddings"]:
            t["lm_head.weight"] = matrix(V, H)
        return t
    W, V = cfg["width"], cfg["vocab"]
    t["embed"] = matrix(V, W)
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        x = p + "mix."
        if layer["type"] == "lightning":
            n = m["heads"] * m["dim"]
            t.update({x + k: matrix(n, W) for k in "qkvg"})
            t.update({x + "o": matrix(W, n), x + "norm": weight(n)})
        elif layer["type"] == "mingru":
            t.update({x + k: matrix(W, W) for k in "zxgo"})
            t.update({x + "z.b": vector(W, std=0.5), x + "x.b": vector(W, std=0.5)})
        elif layer["type"] == "latent_attention":
            h, row = m["heads"], m["kv_rank"] + m["rot_dim"]
            t.update({x + "q": matrix(h * (m["dim"] + m["rot_dim"]), W), x + "uk": matrix(h * m["dim"], m["kv_rank"]),
                      x + "uv": matrix(h * m["vdim"], m["kv_rank"]), x + "o": matrix(W, h * m["vdim"]), x + "dkv": matrix(row, W),
                      x + "dkv.norm": weight(m["kv_rank"]), x + "g": matrix(h, W)})
        elif model == "koronex":
            q, kv = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
            t.update({x + "q": matrix(q, W), x + "g": matrix(q, W), x + "o": matrix(W, q), x + "q.norm": weight(q),
                      x + "sink": vector(m["heads"], std=1.0)})
            if "kv_from" not in m:
                t.update({x + "k": matrix(kv, W), x + "v": matrix(kv, W), x + "k.norm": weight(kv)})
        else:
            a, maps = (m["left"], 1) if model == "zetenex" else (m, 2)
            y = x + ("left." if model == "zetenex" else "")
            t.update({y + "q": matrix(a["heads"] * maps * a["dim"], W), y + "k": matrix(a["kv_heads"] * maps * a["dim"], W),
                      y + "v": matrix(a["kv_heads"] * a["vdim"], W), y + "g": matrix(a["heads"], W), y + "o": matrix(W, a["heads"] * a["vdim"])})
            if model == "dotivik":
                t.update({x + n: vector(a["dim"], std=0.1) for n in ("lq1", "lk1", "lq2", "lk2")})
            else:
                b, y = m["right"], x + "right."
                n, N, R = b["inner"], b["state"], b["dt_rank"]
                t.update({y + "in": matrix(2 * n, W), y + "conv": vector(n, b["conv"], std=0.5), y + "conv.b": vector(n, std=0.1),
                          y + "x": matrix(R + 2 * N, n), y + "dt": matrix(n, R), y + "dt.b": vector(n, mean=-2.0, std=1.0),
                          y + "A_log": vector(n, N, std=1.0), y + "D": vector(n, mean=1.0, std=0.1), y + "o": matrix(W, n)})
        norms = ("norm1",) if model == "dotivik" else ("norm1", "norm2")
        t.update({p + n: weight(W) for n in norms})
        t.update({p + "mlp.up": matrix(ff, W), p + "mlp.down": matrix(W, ff)})
        if model == "dotivik":
            t[p + "mlp.gate"] = matrix(ff, W)
        if model == "koronex":
            d = cfg["token_side"]["dim"]
            t.update({p + "side.gate": matrix(d, W), p + "side.proj": matrix(W, d), p + "side.norm": weight(W)})
        if model == "zetenex":
            t.update(dyt(p + "norm1", W) | dyt(p + "norm2", W))
            t.update({p + "canon1": vector(W, 4, std=0.3), p + "canon2": vector(W, 4, std=0.3)})
    t["final.norm"] = weight(W)
    if model == "koronex":
        t.update({"head": matrix(V, W), "side.embed": matrix(V, len(cfg["layers"]) * cfg["token_side"]["dim"])})
    if model == "dotivik":
        t["loop.in"] = matrix(W, 2 * W)
    if model == "zetenex":
        t["loop.step"] = vector(cfg["loop"]["times"], W, std=0.1)
        t.update(dyt("final.norm", W))
    return t


def dyt(name, W):
    return {name: ((W,), 1.0, 0.1, False), name + ".b": ((W,), 0.0, 0.1, False), name + ".alpha": ((), 0.6, 0.1, False)}


# ---- the same logits in 64 bits, whole sequences at once -------------------------------------------------------------------------
class Weights:
    """The seeded random weights by name, each drawn when it is asked for."""

    def __init__(self, c, cfg, seed):
        self.table, self.seed, self.matrix = tensors(c["model"], cfg), seed, getattr(torch, c["dtype"])

    def __getitem__(self, name):
        shape, mean, std, matrix = self.table[name]
        number = int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:8], "little") & ((1 << 63) - 1)
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(number)
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE)
        t.normal_(mean, std, generator=gen)
        return (t.to(self.matrix) if matrix else t).double()


def exact(c, seed):
    """Logits as run() returns them."""
    cfg = config_of(c)
    w = Weights(c, cfg, seed)
    ids = token_ids(c, seed)
    seqs = [a + b for a, b in ids]
    cuts = [0]
    for s in seqs:
        cuts.append(cuts[-1] + len(s))
    tokens = torch.tensor(sum(seqs, []), device=DEVICE)
    spans = [slice(a, b) for a, b in zip(cuts, cuts[1:])]
    x = {"qwen2": qwen2, "koronex": koronex, "dotivik": dotivik, "zetenex": zetenex}[c["model"]](cfg, w, tokens, spans)
    if c["kind"] == "turn":
        rows = [[s.start + len(a) - 1 + k for s, (a, _) in zip(spans, ids)] for k in range(c["steps"] + 1)]
    else:
        rows = [s.stop - 1 for s in spans]
    x = x[torch.tensor(rows, device=DEVICE)]
    head = "lm_head.weight" if "lm_head.weight" in w.table else "head" if "head" in w.table else \
        "embed" if "embed" in w.table else "model.embed_tokens.weight"
    return x @ w[head].T


def mean_square(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def silu(z):
    return z * torch.sigmoid(z)


def in_parts(f, x, rows=16384):
    return torch.cat([f(x[a:a + rows]) for a in range(0, x.shape[0], rows)])


def turned(t, dims, base, interleaved=False):
    """t [T, n, d] of positions 0 .. T-1: pairs of the first ``dims`` elements turn by position * base^(-2i / dims)."""
    i = torch.arange(dims // 2, dtype=t.dtype, device=t.device)
    a = torch.arange(t.shape[0], dtype=t.dtype, device=t.device)[:, None] * base ** (-2.0 * i / dims)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    first = slice(0, dims, 2) if interleaved else slice(0, dims // 2)
    second = slice(1, dims, 2) if interleaved else slice(dims // 2, dims)
    u, v, out = t[..., first], t[..., second], t.clone()
    out[..., first], out[..., second] = u * cos - v * sin, v * cos + u * sin
    return out


def attend(q, k, v, scale, window=None, sink=None, cap=None):
    """q [T, H, d] over k [T, G, d], v [T, G, dv]: causal softmax attention of one sequence, [T, H, dv]."""
    T, H, _ = q.shape
    G = k.shape[1]
    k, v = k.transpose(0, 1)[:, None], v.transpose(0, 1)[:, None]                       # [G, 1, T, .]
    out = []
    part = max(1, (1 << 28) // (H * T))
    for a in range(0, T, part):
        rows = torch.arange(a, min(T, a + part), device=q.device)
        s = q[a:a + part].transpose(0, 1).reshape(G, H // G, len(rows), -1) @ k.transpose(-1, -2) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        back = rows[:, None] - torch.arange(T, device=q.device)
        s.masked_fill_((back < 0) | (back >= (window or T)), -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.view(G, H // G, 1, 1).expand(-1, -1, len(rows), 1)), -1)
        s = torch.softmax(s, -1)[..., :T]
        out.append((s @ v).reshape(H, len(rows), -1).transpose(0, 1))
    return torch.cat(out)


def qwen2(cfg, w, tokens, spans):
    eps, d, x = cfg["rms_norm_eps"], cfg["head_dim"], w["model.embed_tokens.weight"][tokens]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = mean_square(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].T + w[p + f"self_attn.{n}_proj.bias"]).view(len(h), -1, d) for n in "qkv")
        theta = cfg["rope_theta"]
        o = torch.cat([attend(turned(q[s], d, theta), turned(k[s], d, theta), v[s], d ** -0.5) for s in spans])
        x = x + o.flatten(1) @ w[p + "self_attn.o_proj.weight"].T
        gate, up, down = (w[p + f"mlp.{n}_proj.weight"].T for n in ("gate", "up", "down"))
        norm = w[p + "post_attention_layernorm.weight"]
        x = in_parts(lambda y: y + (silu(mean_square(y, eps) * norm @ gate) * (mean_square(y, eps) * norm @ up)) @ down, x)
    return mean_square(x, eps) * w["model.norm.weight"]


def koronex(cfg, w, tokens, spans):
    eps, alpha, x, kept = cfg["norm"]["eps"], cfg["postln_alpha"], w["embed"][tokens] * cfg["embedding"]["scale"], {}
    side, table = cfg["token_side"]["dim"], w["side.embed"][tokens]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        gate = torch.sigmoid(x @ w[p + "mix.g"].T)
        if layer["type"] == "lightning":
            q, k, v = (silu(x @ w[p + "mix." + n].T).view(len(x), m["heads"], -1) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float32, device=DEVICE).double().log()[:, None, None]
            o = torch.cat([lightning(q[s], k[s], v[s], decay) for s in spans]).flatten(1)
            y = mean_square(o, eps) * w[p + "mix.norm"] * gate
        else:
            def heads(name, n):
                return (mean_square(x @ w[p + f"mix.{name}"].T, eps) * w[p + f"mix.{name}.norm"]).view(len(x), n, -1)

            r, base = m["rot"]["dims"], m["rot"]["base"]
            if "kv_from" not in m:
                kept[i] = heads("k", m["kv_heads"]), (x @ w[p + "mix.v"].T).view(len(x), m["kv_heads"], -1)
            k, v = kept[m.get("kv_from", i)]
            q, sink = heads("q", m["heads"]), w[p + "mix.sink"]
            y = torch.cat([attend(turned(q[s], r, base), turned(k[s], r, base), v[s], m["scale"], m["mask"]["size"], sink)
                           for s in spans]).flatten(1) * gate
        x = mean_square(alpha * x + y @ w[p + "mix.o"].T, eps) * w[p + "norm1"]
        x = mean_square(alpha * x + torch.relu(x @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T, eps) * w[p + "norm2"]
        y = (gelu(x @ w[p + "side.gate"].T) * table[:, i * side:(i + 1) * side]) @ w[p + "side.proj"].T
        x = x + mean_square(y, eps) * w[p + "side.norm"]
    return mean_square(x, eps) * w["final.norm"]


def lightning(q, k, v, log_decay):
    """q, k, v [T, H, d]: o_t = sum over j <= t of decay^(t - j) (q_t . k_j) v_j."""
    t = torch.arange(q.shape[0], device=q.device, dtype=q.dtype)
    back = t[:, None] - t
    fade = torch.where(back >= 0, torch.exp(log_decay * back.clamp(min=0)), torch.zeros((), dtype=q.dtype, device=q.device))
    return ((q.transpose(0, 1) @ k.permute(1, 2, 0) * fade) @ v.transpose(0, 1)).transpose(0, 1)


def dotivik(cfg, w, tokens, spans):
    eps, x, start = cfg["norm"]["eps"], w["embed"][tokens], cfg["loop"]["start"]
    x0 = x

    def norm(y, name):
        y = y - y.mean(-1, keepdim=True)
        return mean_square(y, eps) * w[name]

    for i in layer_runs(cfg):
        if i == start:
            x = torch.cat((x, x0), -1) @ w["loop.in"].T
        p, layer = f"l{i}.", cfg["layers"][i]
        m, h = layer["mixer"], norm(x, f"l{i}.norm1")
        T, H, d, r, base = len(h), m["heads"], m["dim"], m["rot"]["dims"], m["rot"]["base"]
        window, cap = (m.get("mask") or {}).get("size"), m.get("softcap")
        q = h @ w[p + "mix.q"].T
        if layer["type"] == "attention":
            q, k = (y.view(T, -1, 2, d) for y in (q, h @ w[p + "mix.k"].T))
            v = (h @ w[p + "mix.v"].T).view(T, m["kv_heads"], -1)
            lam = torch.exp((w[p + "mix.lq1"] * w[p + "mix.lk1"]).sum()) - torch.exp((w[p + "mix.lq2"] * w[p + "mix.lk2"]).sum()) + m["diff"]
            one, two = (torch.cat([attend(turned(q[s, :, n], r, base, True), turned(k[s, :, n], r, base, True), v[s], m["scale"], window, cap=cap)
                                   for s in spans]) for n in (0, 1))
            o = mean_square(one - lam * two, eps) * (1.0 - m["diff"])
        else:
            q, down, rank = q.view(T, H, -1), h @ w[p + "mix.dkv"].T, m["kv_rank"]
            low = mean_square(down[:, :rank], eps) * w[p + "mix.dkv.norm"]
            k, v = ((low @ w[p + "mix." + n].T).view(T, H, -1) for n in ("uk", "uv"))
            o = []
            for s in spans:
                qr, kr = turned(q[s, :, d:], r, base), turned(down[s, None, rank:], r, base).expand(-1, H, -1)
                o.append(attend(torch.cat((q[s, :, :d], qr), -1), torch.cat((k[s], kr), -1), v[s], m["scale"], window))
            o = torch.cat(o)
        o = (o * torch.sigmoid(h @ w[p + "mix.g"].T)[:, :, None]).flatten(1)
        x = x + o @ w[p + "mix.o"].T + (gelu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return norm(x, "final.norm")


def zetenex(cfg, w, tokens, spans):
    eps, x, opened, start = cfg["norm"]["eps"], w["embed"][tokens] * cfg["embedding"]["scale"], 0, cfg["loop"]["start"]
    x0 = x

    def norm(y, name):
        return torch.tanh(w[name + ".alpha"] * y) * w[name] + w[name + ".b"]

    def convolved(h, filters):
        out = []
        for s in spans:
            padded = torch.cat((h.new_zeros(filters.shape[1] - 1, h.shape[1]), h[s]))
            out.append(sum(padded[j:j + s.stop - s.start] * filters[:, j] for j in range(filters.shape[1])))
        return torch.cat(out)

    for i in layer_runs(cfg):
        if i == start:
            x, opened = (x + x0 if opened else x) + w["loop.step"][opened], opened + 1
        p, layer = f"l{i}.", cfg["layers"][i]
        m, h = layer["mixer"], norm(x, f"l{i}.norm1")
        h = h + convolved(h, w[p + "canon1"])
        if layer["type"] == "mingru":
            z = torch.sigmoid(h @ w[p + "mix.z"].T + w[p + "mix.z.b"])
            u = h @ w[p + "mix.x"].T + w[p + "mix.x.b"]
            u = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            y = torch.zeros_like(u)
            for s in spans:
                S = torch.zeros_like(u[0])
                for t in range(s.start, s.stop):
                    y[t] = S = torch.addcmul(u[t], 1 - z[t], S)
            y = (y * silu(h @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
        else:
            y = m["left_scale"] * unit_attention(h, w, p + "mix.left.", m["left"], eps, spans) \
                + m["right_scale"] * selective_scan(h, w, p + "mix.right.", m["right"], spans, convolved)
        x = x + y
        h = norm(x, p + "norm2")
        h = h + convolved(h, w[p + "canon2"])
        x = x + gelu(h @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T
    return norm(x, "final.norm")


def unit_attention(h, w, p, m, eps, spans):
    q, k = (mean_square((h @ w[p + n].T).view(len(h), -1, m["dim"]), eps) for n in "qk")
    v = (h @ w[p + "v"].T).view(len(h), m["kv_heads"], -1)
    out = []
    for s in spans:
        at = torch.arange(s.stop - s.start, device=h.device, dtype=h.dtype)
        warm = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1)
        out.append(attend(q[s] * warm[:, None, None], k[s], v[s], m["scale"]))
    return (torch.cat(out) * torch.sigmoid(h @ w[p + "g"].T)[:, :, None]).flatten(1) @ w[p + "o"].T


def selective_scan(h, w, p, m, spans, convolved):
    n, N, R = m["inner"], m["state"], m["dt_rank"]
    xz = h @ w[p + "in"].T
    x = silu(convolved(xz[:, :n], w[p + "conv"]) + w[p + "conv.b"])
    low = x @ w[p + "x"].T
    dt = torch.nn.functional.softplus(low[:, :R] @ w[p + "dt"].T + w[p + "dt.b"], threshold=1e9)
    A, y = -torch.exp(w[p + "A_log"]), torch.zeros_like(x)
    for s in spans:
        S = torch.zeros_like(A)
        for t in range(s.start, s.stop):
            S = torch.addcmul((dt[t] * x[t])[:, None] * low[t, R:R + N], torch.exp(dt[t][:, None] * A), S)
            y[t] = S @ low[t, R + N:]
    return ((y + w[p + "D"] * x) * silu(xz[:, n:])) @ w[p + "o"].T
