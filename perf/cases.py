"""Workloads of the library: layers and whole steps as a program runs them, at the sizes of the named configurations.

A case names a `part` and a `phase`:

    block     one pre-norm layer of the Llama decoder on the 32-bit stream
    delta     the gated delta rule mixer          (Gikepel sizes)
    ssm       the selective state-space mixer     (Gikepel sizes)
    latent    the latent attention mixer          (Gikepel sizes; with window, sinks and head gates the Dufizen sizes)
    gla       the gated linear attention mixer    (Dufizen sizes)
    experts   a mixture of experts                (Pikalix sizes; `relu2`: Dufizen sizes)
    model     a whole Llama model through `Stepper`

    prefill   new prompts, launched as the step function launches them
    decode    one token for each sequence, captured in a CUDA graph as the library captures its decode steps

Layers get their inputs, weights, cached keys and values and carried states from a seed; `exact` states each of them in
64-bit torch over the same numbers.  A mixer's pass goes on from the state it finds, like the next portion of a long prompt.
"""
import math

import torch

from gpt_fast_b200 import Stepper, Transformer, ops
from gpt_fast_b200.cache import EntryView
from gpt_fast_b200.config.registry import architecture_for, config_from_name
from gpt_fast_b200.config.spec import PartSpec
from gpt_fast_b200.ops.types import BatchMeta, PagedKV
from gpt_fast_b200.parts import FEED_FORWARDS, MIXERS, POSITIONS, build_block, build_part
from gpt_fast_b200.parts.residual import Branch, Residual

F64 = torch.float64
PAGE = 64
TAPS = 4
YARN = dict(type="yarn", factor=8.0, original=4096, fast=32.0, slow=1.0)


def listed():
    return [
        # one token of one chat on the flagship size: the smallest call of a served model, bound by the layer's weights and its launches
        dict(name="llama8b-layer-decode-1", part="block", phase="decode", model="llama-3.1-8b", dtype="bfloat16", seqs=1, lo=911, hi=911),
        # a long prompt on the flagship size: the products on the tensor cores and causal attention
        dict(name="llama8b-layer-prefill-2048", part="block", phase="prefill", model="llama-3.1-8b", dtype="bfloat16", seqs=1, lo=2048, hi=2048),
        # sixteen prompts of unequal length packed into one step, as a server admits them
        dict(name="llama3b-layer-packed-16", part="block", phase="prefill", model="llama-3.2-3b", dtype="bfloat16", seqs=16, lo=64, hi=1024),
        # the true 32-bit path, by which results are checked: two short prompts
        dict(name="llama3b-layer-float32", part="block", phase="prefill", model="llama-3.2-3b", dtype="float32", seqs=2, lo=61, hi=137),
        # a whole decode step of a served batch: embedding to logits through the step function
        dict(name="llama3b-model-decode-16", part="model", phase="decode", model="llama-3.2-3b", dtype="bfloat16", seqs=16, lo=64, hi=512),
        # the recurrent mixers over a prompt
        dict(name="delta-prefill-2048", part="delta", phase="prefill", dtype="bfloat16", seqs=1, lo=2048, hi=2048, heads=16, dim=128, width=2048),
        dict(name="ssm-prefill-ragged", part="ssm", phase="prefill", dtype="bfloat16", seqs=3, lo=77, hi=1500, heads=64, dim=64, width=2048),
        dict(name="gla-prefill-2048", part="gla", phase="prefill", dtype="bfloat16", seqs=1, lo=2048, hi=2048, heads=16, dim=128, width=2048),
        # a recurrent mixer in a decode step of a small batch: launches, and the states read and written once
        dict(name="delta-decode-8", part="delta", phase="decode", dtype="bfloat16", seqs=8, lo=512, hi=512, heads=16, dim=128, width=2048),
        # latent attention over a long prompt: every head against one cached row per token
        dict(name="latent-prefill-4096", part="latent", phase="prefill", dtype="bfloat16", seqs=1, lo=4096, hi=4096, heads=16, dim=128, width=2048, window=0),
        # experts of a prompt, and of a decode step, where every chosen expert's weights stream through once
        dict(name="experts-prefill-2048", part="experts", phase="prefill", dtype="bfloat16", seqs=1, lo=2048, hi=2048, experts=16, top=3, hidden=1792, width=2048, relu2=False),
        dict(name="experts-decode-8", part="experts", phase="decode", dtype="bfloat16", seqs=8, lo=1, hi=1, experts=16, top=3, hidden=1792, width=2048, relu2=False),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    part = rng.choice(["block", "block", "block", "model", "delta", "ssm", "gla", "latent", "latent", "experts"])
    phase = rng.choice(["prefill", "prefill", "decode"])
    c = dict(part=part, phase=phase, dtype="bfloat16")
    if phase == "decode":
        c.update(seqs=between(1, 64), lo=between(16, 512))
        c["hi"] = between(c["lo"], 2048)
    else:
        c["seqs"] = between(1, 16)
        c["hi"] = between(1, 4096 // c["seqs"])
        c["lo"] = between(1, c["hi"])
    if part == "block":
        c["model"] = rng.choice(["llama-3.1-8b", "llama-3.2-3b"])
        if phase == "prefill" and rng.random() < 0.25:
            c.update(dtype="float32", seqs=rng.randint(1, 3), hi=between(8, 80))
            c["lo"] = between(2, c["hi"])
    elif part == "model":
        c.update(model="llama-3.2-3b", seqs=min(c["seqs"], 24), hi=between(16, 384))
        if phase == "prefill":
            c["seqs"] = min(c["seqs"], 4)
        c["lo"] = between(8, c["hi"])
    elif part == "experts":
        c.update(experts=rng.choice([8, 16, 32]), top=rng.choice([2, 3, 4]), hidden=rng.choice([768, 1792]), width=rng.choice([1024, 2048]),
                 relu2=rng.random() < 0.5)
    elif part == "ssm":
        c.update(heads=rng.choice([16, 32, 64]), dim=64, width=rng.choice([1024, 2048]))
    else:
        c.update(heads=rng.choice([4, 8, 16]), dim=rng.choice([64, 128]), width=rng.choice([1024, 2048]))
        if part == "latent":
            c.update(dim=128, window=rng.choice([0, 0, 256, 1024]))
    return c


# ---- the numbers of a case -------------------------------------------------------------------------------

def lengths(case):
    """Per sequence, new tokens of a prompt (prefill) or cached tokens (decode): spread evenly from lo to hi, unsorted."""
    n, lo, hi = case["seqs"], case["lo"], case["hi"]
    v = [hi if n == 1 else lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return v[1::2] + v[0::2]


def counts(case):
    """(cached tokens, new tokens) per sequence."""
    v = lengths(case)
    return (v, [1] * len(v)) if case["phase"] == "decode" else ([0] * len(v), v)


class Numbers:
    """Tensors from a seed, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) + 1)

    def normal(self, shape, std=1.0, dtype=torch.float32, mean=0.0):
        t = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=self.g)
        if std != 1.0:
            t *= std
        return t + mean if mean else t

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, device="cuda", generator=self.g) * (hi - lo) + lo

    def matrix(self, *shape, dtype):
        return self.normal(shape, shape[-1] ** -0.5, dtype)


def dtype_of(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def spec_of(case):
    cfg = config_from_name(case["model"])
    arch = architecture_for(cfg)
    return arch.build_spec(arch.parse(cfg)), cfg


def llama_sizes(cfg):
    H = cfg["num_attention_heads"]
    return dict(D=cfg["hidden_size"], H=H, G=cfg["num_key_value_heads"], d=cfg["hidden_size"] // H, F=cfg["intermediate_size"],
                V=cfg["vocab_size"], layers=cfg["num_hidden_layers"], eps=cfg["rms_norm_eps"])


def llama_layer(r, s, dt):
    D, H, G, d, F = s["D"], s["H"], s["G"], s["d"], s["F"]
    return {"mixer.wq": r.matrix(H * d, D, dtype=dt), "mixer.wk": r.matrix(G * d, D, dtype=dt), "mixer.wv": r.matrix(G * d, D, dtype=dt),
            "mixer.wo": r.matrix(D, H * d, dtype=dt), "feed_forward.w1": r.matrix(F, D, dtype=dt), "feed_forward.w3": r.matrix(F, D, dtype=dt),
            "feed_forward.w2": r.matrix(D, F, dtype=dt), "mixer_norm.weight": r.normal((D,), 0.1, dt, 1.0),
            "ffn_norm.weight": r.normal((D,), 0.1, dt, 1.0)}


def step_sizes(r, n):
    """Biases whose softplus spreads over 0.001 to 0.1, as recurrent models start from."""
    dt = torch.exp(r.uniform((n,), math.log(1e-3), math.log(0.1)))
    return dt + torch.log(-torch.expm1(-dt))


def mixer_numbers(case, r):
    """(constructor arguments, weights) of a mixer or of the experts."""
    dt, D = dtype_of(case), case["width"]
    vec = lambda n: r.normal((n,), 0.1, torch.float32, 1.0)  # noqa: E731
    if case["part"] == "experts":
        E, F = case["experts"], case["hidden"]
        w = {"router": r.matrix(E, D, dtype=dt), "up": r.matrix(E, F, D, dtype=dt), "down": r.matrix(E, D, F, dtype=dt),
             "correction": r.normal((E,), 0.01), "shared_up": r.matrix(F, D, dtype=dt), "shared_down": r.matrix(D, F, dtype=dt)}
        if not case["relu2"]:
            w.update(gate=r.matrix(E, F, D, dtype=dt), shared_gate=r.matrix(F, D, dtype=dt))
        args = dict(dim=D, hidden=F, n_experts=E, top=case["top"], score="softmax" if case["relu2"] else "sigmoid_plain", shared_hidden=F,
                    activation="relu2" if case["relu2"] else "glu", groups=(4, 2, 1 if case["relu2"] else 2))
        return args, w
    H, d = case["heads"], case["dim"]
    if case["part"] == "ssm":
        N, inner = 128, H * d
        w = {"w_in": r.matrix(2 * inner + 2 * N + H, D, dtype=dt), "conv": r.normal((inner + 2 * N, TAPS), 0.5), "conv_bias": r.normal((inner + 2 * N,), 0.1),
             "dt_bias": step_sizes(r, H), "a_log": torch.log(r.uniform((H,), 1.0, 16.0)), "skip": vec(H), "norm": vec(inner),
             "wo": r.matrix(D, inner, dtype=dt)}
        return dict(dim=D, n_head=H, head_dim=d, n_state=N, n_groups=1, norm_groups=1, taps=TAPS, eps=1e-5), w
    if case["part"] == "delta":
        w = {k: r.matrix(H * d, D, dtype=dt) for k in ("wq", "wk", "wv")}
        w.update(wb=r.matrix(H, D, dtype=dt), wa1=r.matrix(128, D, dtype=dt), wa2=r.matrix(H * d, 128, dtype=dt), wg1=r.matrix(128, D, dtype=dt),
                 wg2=r.matrix(H * d, 128, dtype=dt), dt_bias=step_sizes(r, H * d), a_log=torch.log(r.uniform((H,), 1.0, 16.0)), norm=vec(d),
                 wo=r.matrix(D, H * d, dtype=dt), **{k: r.normal((H * d, TAPS), 0.5) for k in ("q_conv", "k_conv", "v_conv")})
        return dict(dim=D, n_head=H, n_qk=H, head_dim=d, v_head_dim=d, taps=TAPS, decay_rank=128, gate_rank=128, eps=1e-5), w
    if case["part"] == "gla":
        w = {k: r.matrix(H * d, D, dtype=dt) for k in ("wq", "wk", "wv", "wg")}
        w.update(wa1=r.matrix(16, D, dtype=dt), wa2=r.matrix(H * d, 16, dtype=dt), a2_bias=r.normal((H * d,), 0.5), norm=vec(d), wo=r.matrix(D, H * d, dtype=dt))
        return dict(dim=D, n_head=H, head_dim=d, v_head_dim=d, decay_rank=16, tau=16.0, eps=1e-5), w
    R, rot, windowed = 512, 64, bool(case["window"])
    w = {"wq": r.matrix(H * (d + rot), D, dtype=dt), "wdkv": r.matrix(R + rot, D, dtype=dt), "wg": r.matrix(H if windowed else H * d, D, dtype=dt),
         "wuk": r.matrix(H * d, R, dtype=dt), "wuv": r.matrix(H * d, R, dtype=dt), "wo": r.matrix(D, H * d, dtype=dt), "latent_norm": vec(R)}
    args = dict(dim=D, n_head=H, head_dim=d, rot_dim=rot, v_head_dim=d, rank=R, scale=0.0722, eps=1e-5)
    if windowed:
        w["sink"] = r.normal((H,))
        args.update(window=case["window"], sink=True, head_gate=True)
    return args, w


def carried(case, r):
    """What the sequences bring along: [seqs, floats] of state (zeros ahead of a prompt's first token)."""
    n, d = case["seqs"], case["dim"]
    inner = case["heads"] * d
    body = inner * (128 if case["part"] == "ssm" else d)
    conv = {"ssm": inner + 256, "delta": 3 * inner, "gla": 0}[case["part"]] * (TAPS - 1)
    if case["phase"] == "decode":
        return torch.cat([r.normal((n, body), 0.05), r.normal((n, conv))], 1)
    return torch.zeros(n, body + conv, device="cuda")


def pages(case, seed):
    """Page table [seqs, pages] (the pool's pages in shuffled order) and the number of pages."""
    ctx, new = counts(case)
    need = [-(-(a + b) // PAGE) for a, b in zip(ctx, new)]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(int(seed))).to(torch.int32)
    table, o = torch.full((len(need), max(need)), -1, dtype=torch.int32), 0
    for i, k in enumerate(need):
        table[i, :k] = order[o:o + k]
        o += k
    return table.cuda(), sum(need)


def pools(case, r, n_pages, heads, dim, v_dim):
    def make(width):
        if case["phase"] == "decode":
            return r.normal((n_pages, heads, PAGE, width), 1.0, dtype_of(case))
        return torch.zeros(n_pages, heads, PAGE, width, dtype=dtype_of(case), device="cuda")
    return make(dim), make(v_dim)


def cached(pool, table, seq, n):
    """The first n rows of a sequence out of the pool: [n, heads, dim]."""
    p = pool[table[seq, :-(-n // PAGE)].long()]
    return p.transpose(1, 2).reshape(-1, pool.shape[1], pool.shape[3])[:n].to(F64)


def batch_of(case):
    ctx, new = counts(case)
    cu = [0]
    for q in new:
        cu.append(cu[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    return BatchMeta(i32(cu), i32([i for i, q in enumerate(new) for _ in range(q)]), i32(list(range(len(new)))), i32(ctx), len(new), cu[-1],
                     max(new), max(a + b for a, b in zip(ctx, new)), ops.new_status("cuda"))


def prompts(case, seed, vocab):
    g = torch.Generator().manual_seed(int(seed) + 5)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lengths(case)]


def model_weights(r, s):
    dt = torch.bfloat16
    w = {"embed.weight": r.normal((s["V"], s["D"]), 0.02, dt), "final_norm.weight": r.normal((s["D"],), 0.1, dt, 1.0)}
    for i in range(s["layers"]):
        w.update({f"layers.{i}.{k}": v for k, v in llama_layer(r, s, dt).items()})
    w["head.weight"] = w["embed.weight"]
    return w


# ---- what a program has in hand, and one pass --------------------------------------------------------------

def prepare(case, seed):
    r = Numbers(seed)
    if case["part"] == "model":
        return prepare_model(case, seed, r)
    batch = batch_of(case)
    state = {"batch": batch, "overlap": case["part"] not in ("gla", "experts")}
    if case["part"] == "block":
        spec, cfg = spec_of(case)
        s = llama_sizes(cfg)
        position = build_part(POSITIONS, spec.layers[0].position)
        block = build_block(spec.layers[0], s["D"], dtype_of(case), position)
        w = llama_layer(r, s, dtype_of(case))
        for name, part in block.parts().items():
            part.load({k[len(name) + 1:]: v for k, v in w.items() if k.startswith(name + ".")})
        table, n_pages = pages(case, seed)
        position.prepare(table.shape[1] * PAGE, "cuda")
        k, v = pools(case, r, n_pages, s["G"], s["d"], s["d"])
        x = r.normal((batch.n_tokens, s["D"]))
        view = EntryView(kv=PagedKV(k, v, table, PAGE))

        def call():
            stream = Residual(x.clone())
            block.forward(stream, batch, view, append=True)
            return {"x": stream.tensor(), "k": k, "v": v}
    else:
        dt, T, D = dtype_of(case), batch.n_tokens, case["width"]
        args, w = mixer_numbers(case, r)
        h = r.normal((T, D), 1.0, dt)
        out = {}
        if case["part"] == "experts":
            part = build_part(FEED_FORWARDS, PartSpec("moe", args), dtype=dt)
            forward = lambda y: part.forward(h, y)  # noqa: E731
        else:
            position, kind = None, {"ssm": "state_space", "delta": "delta_rule", "gla": "gla", "latent": "latent_attention"}[case["part"]]
            if case["part"] == "latent":
                position = build_part(POSITIONS, PartSpec("rope", dict(head_dim=64, base=10000.0, scaling=YARN, pairing="interleaved", freq_dtype="float64")))
                table, n_pages = pages(case, seed)
                position.prepare(table.shape[1] * PAGE, "cuda")
                k, v = pools(case, r, n_pages, 1, 576, 0)
                view, out = EntryView(kv=PagedKV(k, v, table, PAGE)), {"latents": k}
            else:
                view = EntryView(state=carried(case, r))
                out = {"state": view.state}
                state["before"] = view.state.clone()
            part = build_part(MIXERS, PartSpec(kind, args), dtype=dt, position=position)
            forward = lambda y: part.forward(h, batch, view, y)  # noqa: E731
        part.load(w)

        def call():
            y = Branch(T, D, h.device)
            forward(y)
            return dict(out, y=y.tensor())
    state["call"] = call                            # (also what keeps a graph's weights and inputs alive)
    if case["phase"] == "decode":
        ops.set_launch_overlap(state["overlap"])
        call()                                      # loads the kernels
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            result = call()
        if "before" in state:
            result["state"].copy_(state.pop("before"))
        state.update(graph=graph, result=result)
    return state


def prepare_model(case, seed, r):
    spec, cfg = spec_of(case)
    s = llama_sizes(cfg)
    model = Transformer(spec, torch.bfloat16, "cuda")
    model.load_params(model_weights(r, s))
    toks = prompts(case, seed, s["V"])
    # pages for the steps to come: a served sequence goes on for thousands of tokens
    cache = model.new_cache(max_tokens=case["seqs"] * 4096, max_seqs=case["seqs"], max_seq_len=4096)
    stepper = Stepper.of(model, cache)
    if case["phase"] == "prefill":
        return {"stepper": stepper, "prompts": toks}
    slots = cache.begin(len(toks))
    stepper.step(slots, toks, "none")
    for i in slots:
        cache.reserve(i, 4096)
    step = stepper.decode_batch(slots)
    step.tokens.copy_(torch.tensor([(7 * t[-1] + 1) % s["V"] for t in toks], dtype=torch.int32))
    before = cache.lengths.clone()
    for _ in range(2):                              # an eager step, then the captured one
        step.run()
        cache.lengths.copy_(before)
        cache.note_advance(slots, [-1] * len(slots))
    return {"step": step}


def run(state):
    if "step" in state:
        return state["step"].run()
    if "stepper" in state:
        cache = state["stepper"].cache
        slots = cache.begin(len(state["prompts"]))
        logits = state["stepper"].step(slots, state["prompts"], "last")
        cache.end(slots)
        return logits
    ops.set_launch_overlap(state["overlap"])
    if "graph" in state:
        state["graph"].replay()
        return state["result"]
    return state["call"]()


# ---- what a pass cannot do without -------------------------------------------------------------------------

def work(case):
    ctx, new = counts(case)
    T, b = sum(new), 4 if case["dtype"] == "float32" else 2
    seen = sum(sum(min(c + i + 1, case.get("window") or c + i + 1) for i in range(q)) for c, q in zip(ctx, new))
    rows = sum(min(c, case.get("window") or c) + q for c, q in zip(ctx, new))
    if case["part"] in ("block", "model"):
        s = llama_sizes(config_from_name(case["model"]))
        weights = s["D"] * s["d"] * (2 * s["H"] + 2 * s["G"]) + 3 * s["D"] * s["F"]
        flops = 2.0 * T * weights + 4.0 * seen * s["H"] * s["d"]
        moved = b * (weights + 2 * rows * s["G"] * s["d"]) + 8.0 * T * s["D"]
        if case["part"] == "model":
            n = case["seqs"]
            moved = s["layers"] * (moved - 8.0 * T * s["D"]) + 2.0 * s["V"] * s["D"] + 4.0 * n * s["V"]
            flops = s["layers"] * flops + 2.0 * n * s["V"] * s["D"]
        return {"bytes": moved, "flops": flops}
    D = case["width"]
    if case["part"] == "experts":
        E, F, mats = case["experts"], case["hidden"], 2 if case["relu2"] else 3
        busy = E * (1 - (1 - case["top"] / E) ** T) + 1                    # experts that some token chooses, and the shared one
        return {"bytes": 2.0 * busy * mats * F * D + 6.0 * T * D, "flops": 2.0 * T * ((case["top"] + 1) * mats * F * D + E * D)}
    H, d = case["heads"], case["dim"]
    if case["part"] == "latent":
        gates = H if case["window"] else H * d
        weights = D * (H * (d + 64) + 576 + gates) + 2 * H * d * 512 + D * H * d
        return {"bytes": 2.0 * weights + 6.0 * T * D + 2.0 * 576 * rows, "flops": 2.0 * T * weights + 2.0 * seen * H * (576 + 512)}
    inner = H * d
    weights = {"ssm": D * (3 * inner + 256 + H), "delta": D * (4 * inner + H + 256) + 256 * inner, "gla": D * (5 * inner + 16) + 16 * inner}[case["part"]]
    per_state = 128 if case["part"] == "ssm" else d
    steps = 2.0 * T * inner * per_state * (3 if case["part"] == "delta" else 2)
    return {"bytes": 2.0 * weights + 6.0 * T * D + 8.0 * case["seqs"] * inner * per_state, "flops": 2.0 * T * weights + steps}


def tolerance(case):
    # Against 64-bit sums over the same inputs a 32-bit layer is 1e-6 off, a bfloat16 layer 0.3 to 0.7 % (every projection is rounded
    # once or twice), the whole 28-layer model 1 to 2 %.  Single numbers stand further out than the norm does.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03 if case["part"] == "model" else 0.02, "max": 0.9}


# ---- the same in 64-bit ------------------------------------------------------------------------------------

def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def turn(x, pos, freqs, amplitude=1.0):
    """Neighbouring pairs of x [T, heads, dims] turned by pos * freqs."""
    ang = pos.to(F64)[:, None, None] * freqs
    c, s = torch.cos(ang) * amplitude, torch.sin(ang) * amplitude
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def llama_frequencies(cfg, d):
    f = float(cfg["rope_theta"]) ** (-2.0 * torch.arange(d // 2, dtype=F64, device="cuda") / d)
    sc = cfg.get("rope_scaling")
    if not sc:
        return f
    turns = sc["original_max_position_embeddings"] * f / (2 * math.pi)
    blend = ((turns - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])).clamp(0, 1)
    return f * (blend + (1 - blend) / sc["factor"])


def yarn(dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)
    at = lambda turns: dims * math.log(YARN["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(YARN["fast"])), 0), min(math.ceil(at(YARN["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / YARN["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(YARN["factor"]) + 1.0


def attend(q, k, v, scale, first, window=0, sink=None):
    """q [T, H, d] at positions first.., k [S, G, d], v [S, G, dv]."""
    T, H, S, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        n = torch.arange(first, first + T, device="cuda")[:, None] - torch.arange(S, device="cuda")[None]
        s = s.masked_fill((n < 0) | (n >= window if window else n < 0), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :S] @ v[:, h * G // H])
    return torch.stack(out, 1)


def exact_llama(x, w, s, freqs, past):
    """One layer on x [T, D]; past = (keys, values) of the sequence's cached tokens, [n, G, d] each."""
    w = {k: v.to(F64) for k, v in w.items()}
    T, first = x.shape[0], past[0].shape[0]
    pos = torch.arange(first, first + T, device="cuda")
    h = rms(x, s["eps"]) * w["mixer_norm.weight"]
    q = turn((h @ w["mixer.wq"].T).view(T, s["H"], s["d"]), pos, freqs)
    k = torch.cat([past[0], turn((h @ w["mixer.wk"].T).view(T, s["G"], s["d"]), pos, freqs)])
    v = torch.cat([past[1], (h @ w["mixer.wv"].T).view(T, s["G"], s["d"])])
    x = x + attend(q, k, v, s["d"] ** -0.5, first).reshape(T, -1) @ w["mixer.wo"].T
    h = rms(x, s["eps"]) * w["ffn_norm.weight"]
    x = x + (silu(h @ w["feed_forward.w1"].T) * (h @ w["feed_forward.w3"].T)) @ w["feed_forward.w2"].T
    return x, k[first:], v[first:]


def put(pool, table, seq, first, rows):
    """rows [n, heads, dim] into a sequence's places from position `first` on."""
    p = torch.arange(first, first + rows.shape[0], device="cuda")
    pool[table[seq, p // PAGE].long(), :, p % PAGE] = rows


def convolved(u, w, bias, before):
    """Causal convolution and SiLU of u [T, C] behind the inputs `before` [taps - 1, C]; also the last taps - 1 inputs."""
    full = torch.cat([before, u])
    y = sum(full[j:j + u.shape[0]] * w[:, j] for j in range(TAPS))
    return silu(y if bias is None else y + bias), full[-(TAPS - 1):]


def exact_ssm(h, w, case, carry):
    H, P, N, T = case["heads"], case["dim"], 128, h.shape[0]
    inner = H * P
    proj = h @ w["w_in"].T
    S = carry[:inner * N].view(H, N, P).clone()
    xbc, last = convolved(proj[:, inner:2 * inner + 2 * N], w["conv"], w["conv_bias"], carry[inner * N:].view(TAPS - 1, -1))
    x, B, C = xbc[:, :inner].view(T, H, P), xbc[:, inner:inner + N], xbc[:, inner + N:]
    dt = torch.nn.functional.softplus(proj[:, 2 * inner + 2 * N:] + w["dt_bias"])
    decay, y = torch.exp(-torch.exp(w["a_log"]) * dt), []
    for t in range(T):
        S = decay[t][:, None, None] * S + B[t][None, :, None] * (dt[t][:, None] * x[t])[:, None, :]
        y.append(torch.einsum("hnp,n->hp", S, C[t]) + w["skip"][:, None] * x[t])
    y = rms(torch.stack(y).view(T, inner) * silu(proj[:, :inner]), 1e-5) * w["norm"]
    return y @ w["wo"].T, torch.cat([S.flatten(), last.flatten()])


def exact_delta(h, w, case, carry):
    H, d, T = case["heads"], case["dim"], h.shape[0]
    S = carry[:H * d * d].view(H, d, d).clone()
    u = torch.cat([h @ w[k].T for k in ("wq", "wk", "wv")], 1)
    u, last = convolved(u, torch.cat([w["q_conv"], w["k_conv"], w["v_conv"]]), None, carry[H * d * d:].view(TAPS - 1, -1))
    q, k, v = (t.reshape(T, H, d) for t in u.split(H * d, 1))
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    beta = torch.sigmoid(h @ w["wb"].T)
    z = torch.nn.functional.softplus(h @ w["wa1"].T @ w["wa2"].T + w["dt_bias"]).view(T, H, d)
    g, o = torch.exp(-torch.exp(w["a_log"])[:, None] * z), []
    for t in range(T):
        S = g[t][:, :, None] * S
        e = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * e[:, None, :]
        o.append(torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5)
    gate = torch.sigmoid(h @ w["wg1"].T @ w["wg2"].T).view(T, H, d)
    return (rms(torch.stack(o), 1e-5) * w["norm"] * gate).view(T, H * d) @ w["wo"].T, torch.cat([S.flatten(), last.flatten()])


def exact_gla(h, w, case, carry):
    H, d, T = case["heads"], case["dim"], h.shape[0]
    S = carry.view(H, d, d).clone()
    q, k, v = ((h @ w[n].T).view(T, H, d) for n in ("wq", "wk", "wv"))
    a, o = (torch.sigmoid(h @ w["wa1"].T @ w["wa2"].T + w["a2_bias"]) ** (1.0 / 16.0)).view(T, H, d), []
    for t in range(T):
        S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        o.append(torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5)
    o = (rms(torch.stack(o), 1e-5) * w["norm"]).view(T, H * d)
    return (o * silu(h @ w["wg"].T)) @ w["wo"].T, S.flatten()


def exact_latent(h, w, case, past):
    H, d, T, first = case["heads"], case["dim"], h.shape[0], past.shape[0]
    pos, (freqs, amp) = torch.arange(first, first + T, device="cuda"), yarn(64, 10000.0)
    q = (h @ w["wq"].T).view(T, H, d + 64)
    down = h @ w["wdkv"].T
    rows = torch.cat([rms(down[:, :512], 1e-5) * w["latent_norm"], turn(down[:, None, 512:], pos, freqs, amp)[:, 0]], 1)
    seen = torch.cat([past, rows])
    k = torch.cat([(seen[:, :512] @ w["wuk"].T).view(-1, H, d), seen[:, None, 512:].expand(-1, H, 64)], 2)
    v = (seen[:, :512] @ w["wuv"].T).view(-1, H, d)
    o = attend(torch.cat([q[..., :d], turn(q[..., d:], pos, freqs, amp)], 2), k, v, 0.0722, first, case["window"], w.get("sink"))
    gate = torch.sigmoid(h @ w["wg"].T).view(T, H, -1)
    return (o * gate).reshape(T, H * d) @ w["wo"].T, rows


def exact_experts(h, w, case):
    T, E, top = h.shape[0], case["experts"], case["top"]
    z = h @ w["router"].T
    s = torch.softmax(z, -1) if case["relu2"] else torch.sigmoid(z)
    c = s + w["correction"]
    best = c.view(T, 4, E // 4).topk(1 if case["relu2"] else 2, -1).values.sum(-1)
    kept = torch.zeros_like(best).scatter_(1, best.topk(2, -1).indices, 1.0).repeat_interleave(E // 4, 1)
    chosen = c.masked_fill(kept == 0, -math.inf).topk(top, -1).indices

    def expert(x, up, down, gate):
        a = torch.relu(x @ up.to(F64).T) ** 2 if gate is None else silu(x @ gate.to(F64).T) * (x @ up.to(F64).T)
        return a @ down.to(F64).T
    y = expert(h, w["shared_up"], w["shared_down"], w.get("shared_gate"))
    for e in range(E):
        t, j = (chosen == e).nonzero(as_tuple=True)
        if t.numel():
            y.index_add_(0, t, s[t, e][:, None] * expert(h[t], w["up"][e], w["down"][e], None if case["relu2"] else w["gate"][e]))
    return y


def exact(case, seed):
    r = Numbers(seed)
    ctx, new = counts(case)
    cuts = [0]
    for q in new:
        cuts.append(cuts[-1] + q)
    if case["part"] == "model":
        s = llama_sizes(config_from_name(case["model"]))
        w, freqs = model_weights(r, s), llama_frequencies(config_from_name(case["model"]), s["d"])
        toks = prompts(case, seed, s["V"])
        if case["phase"] == "decode":
            toks = [t + [(7 * t[-1] + 1) % s["V"]] for t in toks]
        xs = [w["embed.weight"][torch.tensor(t, device="cuda")].to(F64) for t in toks]
        none = torch.zeros(0, s["G"], s["d"], dtype=F64, device="cuda")
        for i in range(s["layers"]):
            layer = {k[len(f"layers.{i}."):]: v.to(F64) for k, v in w.items() if k.startswith(f"layers.{i}.")}
            xs = [exact_llama(x, layer, s, freqs, (none, none))[0] for x in xs]
        last = torch.stack([x[-1] for x in xs])
        h = rms(last, s["eps"]) * w["final_norm.weight"].to(F64)
        return torch.cat([h @ part.to(F64).T for part in w["head.weight"].split(16384)], 1)
    if case["part"] == "block":
        cfg = config_from_name(case["model"])
        s = llama_sizes(cfg)
        w, freqs = llama_layer(r, s, dtype_of(case)), llama_frequencies(cfg, s["d"])
        table, n_pages = pages(case, seed)
        k, v = pools(case, r, n_pages, s["G"], s["d"], s["d"])
        x, k64, v64, out = r.normal((cuts[-1], s["D"])).to(F64), k.to(F64), v.to(F64), []
        for i, n in enumerate(ctx):
            y, kn, vn = exact_llama(x[cuts[i]:cuts[i + 1]], w, s, freqs, (cached(k, table, i, n), cached(v, table, i, n)))
            put(k64, table, i, n, kn)
            put(v64, table, i, n, vn)
            out.append(y)
        return {"x": torch.cat(out), "k": k64, "v": v64}
    args, w = mixer_numbers(case, r)
    h = r.normal((cuts[-1], case["width"]), 1.0, dtype_of(case)).to(F64)
    if case["part"] == "experts":
        return {"y": exact_experts(h, {k: v if v.dim() > 2 else v.to(F64) for k, v in w.items()}, case)}
    w = {k: v.to(F64) for k, v in w.items()}
    parts = [h[a:b] for a, b in zip(cuts, cuts[1:])]
    if case["part"] == "latent":
        table, n_pages = pages(case, seed)
        k, _ = pools(case, r, n_pages, 1, 576, 0)
        k64, out = k.to(F64), []
        for i, n in enumerate(ctx):
            y, rows = exact_latent(parts[i], w, case, cached(k, table, i, n)[:, 0])
            put(k64, table, i, n, rows[:, None])
            out.append(y)
        return {"latents": k64, "y": torch.cat(out)}
    before = carried(case, r).to(F64)
    fn = {"ssm": exact_ssm, "delta": exact_delta, "gla": exact_gla}[case["part"]]
    got = [fn(p, w, case, before[i]) for i, p in enumerate(parts)]
    return {"state": torch.stack([g[1] for g in got]), "y": torch.cat([g[0] for g in got])}
