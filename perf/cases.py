"""The work that users of wick_b200 have it do, as cases that can be timed and compared.

A case is one pass through the public entry points: a prompt step, a few decode steps of a batch that is under way, a later
portion of a prompt whose beginning is cached, a whole ``generate``.  Three of the served designs stand for all: Qwen3 (the
dense decoder; layer sizes of the 8B, 14B and 32B models and of a small one), Nibotar (attention over blocks of positions,
experts chosen by a table) and Kikopel (attention through a cached latent, a recurrence, PolyNorm feed-forwards).  Designs
whose experts are chosen by scores are left out: there two correct implementations send single tokens to different experts,
so that their outputs cannot be held against each other.

Weights are seeded random numbers in the layer sizes of those models; where a model has more layers than a case names,
the case runs the first ones (every layer of a model does the same work; the roundings of 36 layers to bfloat16 add up to
3 % of the logits, too much to hold two implementations against each other).  Decode steps are fed given tokens, as
``bin/trace_run`` does, so that their logits can be compared; afterwards the sequences are taken back to where they were.
"""
import hashlib
import math
import random

import torch

import wick_b200 as wick

# Layer sizes: Qwen3 as bench.py names them, "2k" and "4k" as in the comparisons of designs there.
QWEN3 = {"2k": dict(width=2048, heads=16, kv=4, dim=128, ff=5120, layers=8, vocab=32768),
         "8b": dict(width=4096, heads=32, kv=8, dim=128, ff=12288, layers=36, vocab=151936),
         "14b": dict(width=5120, heads=40, kv=8, dim=128, ff=17408, layers=40, vocab=151936),
         "32b": dict(width=5120, heads=64, kv=8, dim=128, ff=25600, layers=64, vocab=151936)}
NIBOTAR = {"2k": dict(width=2048, heads=16, kv=4, dim=128, layers=8, vocab=32768, mask=1024, dense_ff=8192, experts=8, top=2,
                      expert_ff=1536, shared_ff=2048),
           "4k": dict(width=4096, heads=32, kv=8, dim=128, layers=4, vocab=32768, mask=2048, dense_ff=16384, experts=16, top=2,
                      expert_ff=2048, shared_ff=4096)}
KIKOPEL = {"2k": dict(width=2048, heads=16, dim=128, layers=8, vocab=32768, window=1024, ff=7680, q_rank=768, kv_rank=512,
                      rot_dim=64),
           "4k": dict(width=4096, heads=32, dim=128, layers=4, vocab=32768, window=2048, ff=15360, q_rank=1536, kv_rank=512,
                      rot_dim=64)}
SIZES = {"qwen3": QWEN3, "nibotar": NIBOTAR, "kikopel": KIKOPEL}
PAIRS = {"buckets": 65521, "mul_prev": 36313, "mul_cur": 27191}
DEVICE = "cuda:0"


def _case(design, size, layers, dtype, job, batch, low, high, cached, steps, name=None, sampling="greedy"):
    """low, high: the prompts' lengths lie between them; cached: tokens of each sequence that were run before; steps: decode
    steps of one pass (for "generate": tokens of each sequence)."""
    c = dict(design=design, size=size, layers=layers, dtype=dtype, job=job, batch=batch, low=low, high=high, cached=cached,
             steps=steps, sampling=sampling)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One token of one conversation on a small model: the smallest call, all latency.
        _case("qwen3", "2k", 8, "bfloat16", "decode", 1, 300, 300, 0, 1, "decode_2k_b1"),
        # The headline: 8 sequences of 512-token prompts on the 8B model, mid-generation.
        _case("qwen3", "8b", 20, "bfloat16", "decode", 8, 512, 512, 0, 4, "decode_8b_b8"),
        # A full batch of unequal conversations.
        _case("qwen3", "8b", 12, "bfloat16", "decode", 64, 64, 1536, 0, 4, "decode_8b_b64"),
        # Few long conversations, eight query heads to a key head, an odd batch.
        _case("qwen3", "32b", 6, "bfloat16", "decode", 5, 2900, 3950, 0, 4, "decode_32b_long"),
        # A short question: time to the first token.
        _case("qwen3", "8b", 12, "bfloat16", "prompt", 1, 100, 100, 0, 0, "prompt_8b_100"),
        # A document: one 2,048-token prompt on the 8B model.
        _case("qwen3", "8b", 20, "bfloat16", "prompt", 1, 2048, 2048, 0, 0, "prompt_8b_2048"),
        # Sixteen unequal prompts that start together.
        _case("qwen3", "14b", 8, "bfloat16", "prompt", 16, 64, 2048, 0, 0, "prompt_14b_ragged"),
        # The next turn of long conversations: new tokens behind what the cache holds.
        _case("qwen3", "8b", 12, "bfloat16", "portion", 2, 333, 777, 3100, 0, "portion_8b"),
        # The 32-bit path from prompt to tokens through generate().
        _case("qwen3", "2k", 8, "float32", "generate", 4, 17, 130, 0, 12, "generate_2k_f32"),
        # Nibotar: prompts, and a batch mid-generation.
        _case("nibotar", "4k", 4, "bfloat16", "prompt", 3, 500, 1700, 0, 0, "nibotar_prompt"),
        _case("nibotar", "2k", 8, "bfloat16", "decode", 8, 1400, 1600, 0, 4, "nibotar_decode"),
        # Kikopel: four requests from their prompts to their answers (its recurrence cannot be taken back, so both in one).
        _case("kikopel", "4k", 4, "bfloat16", "turn", 4, 500, 1500, 0, 12, "kikopel_turn"),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "portion", "generate", "nibotar", "nibotar", "kikopel"])
    if kind == "decode":
        size = rng.choice(["2k", "8b", "14b", "32b"])
        batch = _spread(rng, 1, 64)
        low = _spread(rng, 16, 3900 if batch <= 12 else 1500)
        high = min(max(low, _spread(rng, 64, 3900)), max(low, 40000 // batch))
        return _case("qwen3", size, rng.randint(4, 10), "bfloat16", "decode", batch, low, high, 0, rng.randint(1, 4))
    if kind == "prompt":
        size = rng.choice(["2k", "8b", "14b", "32b"])
        batch = _spread(rng, 1, 16)
        high = _spread(rng, 8, 12000 // batch if batch > 3 else 4000)
        return _case("qwen3", size, rng.randint(3, 6), "bfloat16", "prompt", batch, _spread(rng, max(1, high // 8), high), high, 0, 0)
    if kind == "portion":
        batch = _spread(rng, 1, 4)
        high = _spread(rng, 16, 1000)
        return _case("qwen3", rng.choice(["2k", "8b", "14b"]), rng.randint(3, 8), "bfloat16", "portion", batch,
                     max(2, high // 2), high, _spread(rng, 100, 3000), 0)
    if kind == "generate":
        return _case("qwen3", "2k", rng.randint(2, 8), "float32", "generate", rng.randint(1, 9), 5, _spread(rng, 8, 200), 0,
                     rng.randint(2, 12), sampling=rng.choice(["greedy", "default"]))
    if kind == "nibotar":
        size = rng.choice(["2k", "4k"])
        layers = rng.randint(2, NIBOTAR[size]["layers"])
        if rng.random() < 0.5:
            batch = _spread(rng, 1, 6)
            high = _spread(rng, 30, 6000 // batch if batch > 1 else 4000)
            return _case("nibotar", size, layers, "bfloat16", "prompt", batch, max(1, high // 3), high, 0, 0)
        high = _spread(rng, 60, 2500)
        return _case("nibotar", size, layers, "bfloat16", "decode", _spread(rng, 1, 24), high // 2, high, 0, rng.randint(1, 4))
    size = rng.choice(["2k", "4k"])
    batch = _spread(rng, 1, 8)
    high = _spread(rng, 20, 4000 // batch)
    return _case("kikopel", size, rng.randint(3, KIKOPEL[size]["layers"]), "bfloat16", "turn", batch, max(1, high // 3), high, 0,
                 rng.randint(1, 12))


# ---- configurations and their tensors --------------------------------------------------------------------------------
def _config(case):
    z, n = SIZES[case["design"]][case["size"]], case["layers"]
    d = z["dim"]
    if case["design"] == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], hidden_size=z["width"], num_attention_heads=z["heads"],
                    num_key_value_heads=z["kv"], head_dim=d, intermediate_size=z["ff"], num_hidden_layers=n,
                    vocab_size=z["vocab"], max_position_embeddings=40960, rope_theta=1000000.0, rms_norm_eps=1e-6,
                    tie_word_embeddings=False)
    if case["design"] == "nibotar":
        mixer = dict(heads=z["heads"], kv_heads=z["kv"], dim=d, vdim=d, scale=d ** -0.5, v_mix=True, mask={"size": z["mask"]},
                     rot={"dims": d, "base": 1000000.0})
        moe = {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "router": {"experts": z["experts"], "top": z["top"]},
               "shared": {"ff": z["shared_ff"]}}
        return dict(architecture="Nibotar", vocab=z["vocab"], width=z["width"], norm={"eps": 1e-5}, postln_alpha=2.0,
                    logit_softcap=30.0, layers=[dict(type="attention", mixer=mixer, mlp={"kind": "dense", "ff": z["dense_ff"]}
                                                     if i == 0 else moe) for i in range(n)])
    latent = dict(heads=z["heads"], dim=d, rot_dim=z["rot_dim"], vdim=d, q_rank=z["q_rank"], kv_rank=z["kv_rank"],
                  scale=(d + z["rot_dim"]) ** -0.5, mask={"size": z["window"]}, rot={"dims": z["rot_dim"], "base": 10000.0})
    hgrn2 = dict(heads=z["width"] // 128, dim=128, vdim=128)
    layers = [dict(type="hgrn2" if i % 4 == 2 else "latent_attention", mixer=hgrn2 if i % 4 == 2 else latent,
                   mlp={"kind": "dense", "ff": z["ff"]}) for i in range(n)]
    return dict(architecture="Kikopel", vocab=z["vocab"], width=z["width"], norm={"eps": 1e-5}, residual_mult=0.5,
                embedding={"scale": 1.0, "bigram": PAIRS}, layers=layers)


def _tensors(case):
    """name -> (shape, kind) of every tensor of the case's model, layer by layer.  Kinds: "matrix" N(0, 0.02) in the compute
    dtype; vectors in 32 bits: "one" 1 + N(0, 0.1), "zero" N(0, 0.1), "unit" U(0.2, 0.8), "bias" 1 + N(0, 1); "table"."""
    z, n = SIZES[case["design"]][case["size"]], case["layers"]
    w, d, v, t = z["width"], z["dim"], z["vocab"], {}

    def matrix(name, rows, cols):
        t[name] = ((rows, cols), "matrix")

    if case["design"] == "qwen3":
        q, kv = z["heads"] * d, z["kv"] * d
        matrix("model.embed_tokens.weight", v, w)
        for i in range(n):
            p = f"model.layers.{i}."
            for name, rows, cols in (("self_attn.q_proj", q, w), ("self_attn.k_proj", kv, w), ("self_attn.v_proj", kv, w),
                                     ("self_attn.o_proj", w, q), ("mlp.gate_proj", z["ff"], w), ("mlp.up_proj", z["ff"], w),
                                     ("mlp.down_proj", w, z["ff"])):
                matrix(p + name + ".weight", rows, cols)
            for name, size in (("input_layernorm", w), ("post_attention_layernorm", w), ("self_attn.q_norm", d), ("self_attn.k_norm", d)):
                t[p + name + ".weight"] = ((size,), "one")
        t["model.norm.weight"] = ((w,), "one")
        matrix("lm_head.weight", v, w)
        return t
    matrix("embed", v, w)
    if case["design"] == "nibotar":
        q, kv = z["heads"] * d, z["kv"] * d
        for i in range(n):
            m, f = f"l{i}.mix.", f"l{i}.mlp."
            for name, rows in (("q", q), ("k", kv), ("v", kv)):
                matrix(m + name, rows, w)
                t[m + name + ".b"] = ((rows,), "zero")
            matrix(m + "o", w, q)
            t[m + "q.norm"], t[m + "k.norm"] = ((q,), "one"), ((kv,), "one")
            t[m + "sink"], t[m + "vmix"] = ((z["heads"],), "zero"), ((), "unit")
            t[f"l{i}.norm1"] = t[f"l{i}.norm2"] = ((w,), "zero")
            if i == 0:
                matrix(f + "up", z["dense_ff"], w)
                matrix(f + "down", w, z["dense_ff"])
                continue
            for e, ff in [(f"e{k}.", z["expert_ff"]) for k in range(z["experts"])] + [("shared.", z["shared_ff"])]:
                matrix(f + e + "gate", ff, w)
                matrix(f + e + "up", ff, w)
                matrix(f + e + "down", w, ff)
            t[f + "table"] = ((v, z["top"], z["experts"]), "table")
        t["final.norm"] = ((w,), "zero")
    else:
        matrix("bigram", PAIRS["buckets"] + 1, w)
        h, dr, qr, kr = z["heads"], z["rot_dim"], z["q_rank"], z["kv_rank"]
        for i in range(n):
            m = f"l{i}.mix."
            if i % 4 == 2:
                for name in ("q", "f", "v", "o"):
                    matrix(m + name, w, w)
                t[m + "f.b"], t[m + "lower"], t[m + "norm"] = ((w,), "bias"), ((w,), "unit"), ((128,), "one")
            else:
                for name, rows, cols in (("dq", qr, w), ("uq", h * (d + dr), qr), ("dkv", kr + dr, w), ("uk", h * d, kr),
                                         ("uv", h * d, kr), ("g", h * d, w), ("o", w, h * d)):
                    matrix(m + name, rows, cols)
                t[m + "dq.norm"], t[m + "dkv.norm"] = ((qr,), "one"), ((kr,), "one")
            t[f"l{i}.norm1"] = t[f"l{i}.norm2"] = ((), "one")
            matrix(f"l{i}.mlp.up", z["ff"], w)
            matrix(f"l{i}.mlp.down", w, z["ff"])
            t[f"l{i}.mlp.act"] = ((4,), "one")
        t["final.norm"] = ((), "one")
    matrix("head", v, w)
    return t


def _weights(case, seed):
    """A function from a tensor's name to its values, from the seed and the name alone."""
    table = _tensors(case)
    dtype = getattr(torch, case["dtype"])

    def get(name):
        if name not in table:
            return None
        shape, kind = table[name]
        g = torch.Generator(device=DEVICE)
        g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
        if kind == "matrix":
            return torch.empty(shape, dtype=dtype, device=DEVICE).normal_(0.0, 0.02, generator=g)
        if kind == "table":                            # every id's experts: the first of a random order of all
            return torch.rand((shape[0], shape[2]), generator=g, device=DEVICE).argsort(1)[:, :shape[1]].to(torch.int32).contiguous()
        if kind == "unit":
            return 0.2 + 0.6 * torch.rand(shape, generator=g, device=DEVICE)
        x = torch.randn(shape, generator=g, device=DEVICE)
        return {"one": 1.0 + 0.1 * x, "zero": 0.1 * x, "bias": 1.0 + x}[kind]

    return get


def _lens(case):
    rng = random.Random(f"{case['batch']}:{case['low']}:{case['high']}")
    return [rng.randint(case["low"], case["high"]) for _ in range(case["batch"])]


def _tokens(case, seed):
    """(what is cached before, the prompts, the tokens that the decode steps are fed) of every sequence, as lists."""
    vocab = SIZES[case["design"]][case["size"]]["vocab"]
    g = torch.Generator()
    g.manual_seed(7 * seed + 1)
    ids = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()  # noqa: E731
    lens = _lens(case)
    return [ids(case["cached"]) for _ in lens], [ids(n) for n in lens], [ids(case["steps"]) for _ in lens]


# ---- what a user's program has, and a pass ---------------------------------------------------------------------------
def prepare(case, seed):
    cached, prompts, feed = _tokens(case, seed)
    cfg = wick.config_from_json(_config(case))
    model = wick.Model(wick.get_architecture(cfg.architecture).build_spec(cfg), getattr(torch, case["dtype"]), DEVICE)
    model.load(_weights(case, seed))
    longest = [len(c) + len(p) + case["steps"] for c, p in zip(cached, prompts)]
    eng = wick.Engine(model, max_tokens=sum((n + 63) // 64 * 64 for n in longest) + 64)
    state = dict(case=case, eng=eng, prompts=prompts, feed=[[[f[k]] for f in feed] for k in range(case["steps"])])
    if case["job"] in ("decode", "portion"):           # sequences under way: the prompts (or their first portions) are in the cache
        state["slots"] = [eng.open_seq() for _ in prompts]
        eng.step(state["slots"], prompts if case["job"] == "decode" else cached)
        state["held"] = [eng.seq_len(s) for s in state["slots"]]
    if case["job"] != "generate":                      # a program that has served before: the steps it captures are captured
        run(state)
    return state


def run(state):
    return {"decode": _run_decode, "portion": _run_portion, "prompt": _run_turn, "turn": _run_turn,
            "generate": _run_generate}[state["case"]["job"]](state)


def _run_decode(state):
    eng, slots = state["eng"], state["slots"]
    out = [eng.step(slots, tokens).clone() for tokens in state["feed"]]
    for s, n in zip(slots, state["held"]):
        eng.truncate_seq(s, n)
    return out


def _run_portion(state):
    eng, slots = state["eng"], state["slots"]
    out = eng.step(slots, state["prompts"])
    for s, n in zip(slots, state["held"]):
        eng.truncate_seq(s, n)
    return out


def _run_turn(state):
    eng = state["eng"]
    slots = [eng.open_seq() for _ in state["prompts"]]
    out = [eng.step(slots, state["prompts"])]
    out += [eng.step(slots, tokens).clone() for tokens in state["feed"]]
    for s in slots:
        eng.close_seq(s)
    return out


class _KeepingLogits:
    """A batch under way whose every step's logits are kept."""

    def __init__(self, run, logits):
        self.run, self.logits, self.depth = run, logits, run.depth

    def start(self, slots, prompts, limits):
        self.run.start(slots, prompts, limits)
        self.logits.append(self.run.last_logits.clone())

    def launch(self, slots):
        self.run.launch(slots)
        self.logits.append(self.run.last_logits.clone())

    def collect(self):
        return self.run.collect()


def _run_generate(state):
    case, eng, logits = state["case"], state["eng"], []
    sampler = wick.SamplerConfig.greedy() if case["sampling"] == "greedy" else wick.SamplerConfig()
    got = wick.generate(eng, state["prompts"], wick.GenOptions(max_tokens=case["steps"], sampler=sampler, max_batch=case["batch"]),
                        run_factory=lambda engine, opts, stops, n: _KeepingLogits(engine.begin_run(opts.sampler, stops), logits))
    return {"tokens": [torch.tensor(r.tokens) for r in got], "logits": logits}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _steps_of(case):
    """The steps of a pass, each as a list of (tokens held before, new tokens) of every sequence."""
    lens = _lens(case)
    if case["job"] == "decode":
        return [[(n + k, 1) for n in lens] for k in range(case["steps"])]
    first = [[(case["cached"], n) for n in lens]]
    more = case["steps"] - 1 if case["job"] == "generate" else case["steps"]
    return first + [[(n + k, 1) for n in lens] for k in range(more)]


def work(case):
    z, n_layers = SIZES[case["design"]][case["size"]], case["layers"]
    size = 4 if case["dtype"] == "float32" else 2
    table = _tensors(case)
    numbers = lambda keep: sum(math.prod(s) for k, (s, kind) in table.items() if kind == "matrix" and keep(k))  # noqa: E731
    expert = lambda k: ".mlp.e" in k  # noqa: E731
    head = z["vocab"] * z["width"]
    dense = numbers(lambda k: not expert(k) and k not in ("embed", "bigram", "head", "model.embed_tokens.weight", "lm_head.weight"))
    experts = numbers(expert)
    share = z["top"] / z["experts"] if "experts" in z else 0.0
    window = z.get("window")
    flops = nbytes = 0.0
    for step in _steps_of(case):
        new, rows = sum(q for _, q in step), len(step)
        flops += 2.0 * new * (dense + experts * share) + 2.0 * rows * head
        touched = 1.0 - (1.0 - share) ** new if experts else 0.0
        nbytes += size * (dense + experts * touched + head + new * z["width"]) + 4.0 * rows * z["vocab"]
        for i in range(n_layers):
            for start, q in step:
                if case["design"] == "kikopel" and i % 4 == 2:   # a record of 128 x 128 numbers a head, read and written
                    nbytes += 2 * 4.0 * z["width"] * 128
                    flops += 4.0 * q * z["width"] * 128
                    continue
                lo, kept = 0, start
                pairs = q * start + q * (q + 1) / 2
                if case["design"] == "nibotar":                  # keys of the query's own block of positions
                    size_b = z["mask"]
                    lo = start // size_b * size_b
                    pairs = sum(p % size_b + 1 for p in range(start, start + q))
                    kept = start - lo
                elif window is not None and start + q > window:
                    pairs = sum(min(p + 1, window) for p in range(start, start + q))
                    kept = min(start, window)
                row = z["kv_rank"] + z["rot_dim"] if case["design"] == "kikopel" else 2 * z["kv"] * z["dim"]
                per_pair = 2 * z["dim"] + (z["rot_dim"] if case["design"] == "kikopel" else 0)
                nbytes += size * row * (kept + q)
                flops += 2.0 * pairs * z["heads"] * per_pair
    return {"bytes": nbytes, "flops": flops}


# ---- tolerances and the same results in 64 bits ----------------------------------------------------------------------
def tolerance(case):
    """Measured between decode steps and prompt steps of the same tokens, whose sums run in other orders: bfloat16 Qwen3 of 12 / 24
    layers 0.018 / 0.025 of the norm and at most 0.10 / 0.16 of the root mean square, Nibotar and Kikopel 0.005 and 0.025; against
    64 bits, the 32-bit path 5e-6 of the norm."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.0}
    return {"rel": 0.03, "max": 0.4} if case["design"] == "qwen3" else {"rel": 0.02, "max": 0.1}


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(positions, dims, base):
    """The designs' angles are 32-bit products of a position and an inverse frequency."""
    inv = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=DEVICE).float()
    a = (positions.float()[:, None] * inv[None, :]).double()[:, None, :]
    return torch.cos(a), torch.sin(a)


def _turn(x, positions, base, neighbours=False):
    """x [n, heads, d]: pairs (i, i + d / 2), or neighbours (2 i, 2 i + 1), turned by the position's angles."""
    d = x.shape[-1]
    c, s = _angles(positions, d, base)
    a, b = (x[..., 0::2], x[..., 1::2]) if neighbours else (x[..., :d // 2], x[..., d // 2:])
    a, b = a * c - b * s, b * c + a * s
    return torch.stack([a, b], -1).flatten(-2) if neighbours else torch.cat([a, b], -1)


def _attend(q, k, v, scale, see, sink=None):
    """q [n, H, d], k [n, G, d], v [n, G, e]; see(i, j): whether query i sees key j.  [n, H, e], a key head at a time."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(n, device=DEVICE)
    hidden = ~see(i[:, None], i[None, :])
    out = torch.empty((n, H, v.shape[2]), dtype=q.dtype, device=DEVICE)
    for h in range(H):
        g = h * G // H
        s = (q[:, h] @ k[:, g].T) * scale
        s.masked_fill_(hidden, -math.inf)
        m = s.max(-1, keepdim=True).values
        if sink is not None:
            m = torch.maximum(m, sink[h])
        e = torch.exp(s - m)
        den = e.sum(-1, keepdim=True)
        if sink is not None:
            den = den + torch.exp(sink[h] - m)
        out[:, h] = (e @ v[:, g]) / den
    return out


def _exact_rows(case, get, tokens, rows):
    """Logits in 64 bits of whole sequences at the given places of each; [sum of places, vocab], sequence by sequence."""
    z, cfg = SIZES[case["design"]][case["size"]], _config(case)
    W = lambda name: get(name).double()  # noqa: E731
    ids = [torch.tensor(t, device=DEVICE) for t in tokens]
    pos = [torch.arange(len(t), device=DEVICE) for t in tokens]
    cuts = [len(t) for t in tokens]
    flat = torch.cat(ids)
    H, d, each = z["heads"], z["dim"], lambda x: x.split(cuts)
    silu = lambda x: x * torch.sigmoid(x)  # noqa: E731
    if case["design"] == "qwen3":
        eps, base, scale = cfg["rms_norm_eps"], cfg["rope_theta"], d ** -0.5
        x = get("model.embed_tokens.weight")[flat].double()
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, eps) * W(p + "input_layernorm.weight")
            q = _rms((h @ W(p + "self_attn.q_proj.weight").T).view(-1, H, d), eps) * W(p + "self_attn.q_norm.weight")
            k = _rms((h @ W(p + "self_attn.k_proj.weight").T).view(-1, z["kv"], d), eps) * W(p + "self_attn.k_norm.weight")
            v = (h @ W(p + "self_attn.v_proj.weight").T).view(-1, z["kv"], d)
            a = torch.cat([_attend(_turn(qs, ps, base), _turn(ks, ps, base), vs, scale, lambda i, j: j <= i)
                           for qs, ks, vs, ps in zip(each(q), each(k), each(v), pos)])
            x = x + a.flatten(1) @ W(p + "self_attn.o_proj.weight").T
            h = _rms(x, eps) * W(p + "post_attention_layernorm.weight")
            x = x + (silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
        at = torch.cat([xs[r] for xs, r in zip(each(x), rows)])
        return (_rms(at, eps) * W("model.norm.weight")) @ W("lm_head.weight").T
    eps = cfg["norm"]["eps"]
    x = get("embed")[flat].double()
    if case["design"] == "nibotar":
        alpha, cap, first = cfg["postln_alpha"], cfg["logit_softcap"], None
        gated = lambda h, p: (silu(h @ W(p + "gate").T) * (h @ W(p + "up").T)) @ W(p + "down").T  # noqa: E731
        for i, L in enumerate(cfg["layers"]):
            m, p = L["mixer"], f"l{i}.mix."
            q, k, v = (x @ W(p + n).T + W(p + n + ".b") for n in ("q", "k", "v"))
            q, k = (_rms(q, eps) * W(p + "q.norm")).view(-1, H, d), (_rms(k, eps) * W(p + "k.norm")).view(-1, z["kv"], d)
            first, v = (v, v) if first is None else (first, (1 - W(p + "vmix")) * v + W(p + "vmix") * first)
            base, block, sink = m["rot"]["base"], m["mask"]["size"], W(p + "sink")
            a = torch.cat([_attend(_turn(qs, ps, base, True), _turn(ks, ps, base, True), vs, m["scale"],
                                   lambda i, j: (j <= i) & (j // block == i // block), sink)
                           for qs, ks, vs, ps in zip(each(q), each(k), each(v.view(-1, z["kv"], d)), pos)])
            x = _rms(alpha * x + a.flatten(1) @ W(p + "o").T, eps) * (1 + W(f"l{i}.norm1"))
            p = f"l{i}.mlp."
            if L["mlp"]["kind"] == "dense":
                f = torch.relu(x @ W(p + "up").T).square() @ W(p + "down").T
            else:
                f, chosen = gated(x, p + "shared."), get(p + "table")[flat]
                for e in range(z["experts"]):
                    mine = (chosen == e).any(1).nonzero()[:, 0]
                    f[mine] += gated(x[mine], f"{p}e{e}.") / z["top"]
            x = _rms(alpha * x + f, eps) * (1 + W(f"l{i}.norm2"))
        at = torch.cat([xs[r] for xs, r in zip(each(x), rows)])
        return cap * torch.tanh((_rms(at, eps) * (1 + W("final.norm"))) @ W("head").T / cap)
    mult, dr, pairs = cfg["residual_mult"], z["rot_dim"], get("bigram")
    at_row = [torch.cat([t.new_full((1,), PAIRS["buckets"]), (t[:-1] * PAIRS["mul_prev"] + t[1:] * PAIRS["mul_cur"]) % PAIRS["buckets"]])
              for t in ids]
    x = x + pairs[torch.cat(at_row)].double()
    for i, L in enumerate(cfg["layers"]):
        m, p = L["mixer"], f"l{i}.mix."
        if L["type"] == "hgrn2":
            low = W(p + "lower")
            f = (low + (1 - low) * torch.sigmoid(x @ W(p + "f").T + W(p + "f.b"))).view(-1, m["heads"], 128)
            q, v = silu(x @ W(p + "q").T).view(-1, m["heads"], 128), (x @ W(p + "v").T).view(-1, m["heads"], 128)
            o = []
            for qs, fs, vs in zip(each(q), each(f), each(v)):
                S = torch.zeros((m["heads"], 128, 128), dtype=x.dtype, device=DEVICE)
                for t in range(qs.shape[0]):
                    S = torch.lerp(vs[t][:, None, :].expand_as(S), S, fs[t][:, :, None].expand_as(S))
                    o.append((qs[t][:, None, :] @ S)[:, 0])
            a = (_rms(torch.stack(o), eps) * W(p + "norm")).flatten(1)
        else:
            q = ((_rms(x @ W(p + "dq").T, eps) * W(p + "dq.norm")) @ W(p + "uq").T).view(-1, H, d + dr)
            down = x @ W(p + "dkv").T
            c = _rms(down[:, :z["kv_rank"]], eps) * W(p + "dkv.norm")
            k, v = (c @ W(p + "uk").T).view(-1, H, d), (c @ W(p + "uv").T).view(-1, H, d)
            base, window, out = m["rot"]["base"], m["mask"]["size"], []
            for qs, ks, vs, rs, ps in zip(each(q), each(k), each(v), each(down[:, None, z["kv_rank"]:]), pos):
                qs = torch.cat([qs[..., :d], _turn(qs[..., d:], ps, base)], -1)
                ks = torch.cat([ks, _turn(rs, ps, base).expand(-1, H, -1)], -1)
                out.append(_attend(qs, ks, vs, m["scale"], lambda i, j: (j <= i) & (i - j < window)))
            a = torch.cat(out).flatten(1) * torch.sigmoid(x @ W(p + "g").T)
        x = x + mult * W(f"l{i}.norm1") * _rms(a @ W(p + "o").T, eps)
        y, c = x @ W(f"l{i}.mlp.up").T, W(f"l{i}.mlp.act")
        y = c[0] * _rms(y, eps) + c[1] * _rms(y * y, eps) + c[2] * _rms(y * y * y, eps) + c[3]
        x = x + mult * W(f"l{i}.norm2") * _rms(y @ W(f"l{i}.mlp.down").T, eps)
    at = torch.cat([xs[r] for xs, r in zip(each(x), rows)])
    return (_rms(at, eps) * W("final.norm")) @ W("head").T


def exact(case, seed):
    get = _weights(case, seed)
    cached, prompts, feed = _tokens(case, seed)
    if case["job"] == "generate":
        if case["sampling"] != "greedy":               # (what is drawn decides what follows)
            return None
        seqs, logits = [list(p) for p in prompts], []
        for _ in range(case["steps"]):
            z = _exact_rows(case, get, seqs, [[len(s) - 1] for s in seqs])
            logits.append(z)
            for s, t in zip(seqs, z.argmax(1).tolist()):
                s.append(t)
        return {"tokens": [torch.tensor(s[len(p):]) for s, p in zip(seqs, prompts)], "logits": logits}
    if sum(len(c) + len(p) for c, p in zip(cached, prompts)) * work_of_a_token(case) > 4e14:
        return None                                    # (over about 20 seconds)
    seqs = [c + p + f for c, p, f in zip(cached, prompts, feed)]
    first = 0 if case["job"] == "decode" else -1       # the first wanted row: of the first token fed, or of the prompt's last
    rows = [list(range(len(c) + len(p) + first, len(s))) for c, p, s in zip(cached, prompts, seqs)]
    z = _exact_rows(case, get, seqs, rows)
    z = z.view(len(seqs), len(rows[0]), -1)
    out = [z[:, k].contiguous() for k in range(z.shape[1])]
    return out[0] if case["job"] == "portion" else out


def work_of_a_token(case):
    """Operations of one token in the matrix products."""
    return 2.0 * sum(math.prod(s) for s, kind in _tensors(case).values() if kind == "matrix" and len(s) == 2)
