"""What a user of the library has it do, as cases that can be timed: inputs, one pass, its work, its exact result.

The cases are single layers (a feed-forward, attention, the head, routed experts, mixers with a state) built from the part
registries as a model builds them, and three whole models through the step function and the replayed decode step.  Widths
are those of the configurations this repository benchmarks (Llama-3.1-8B, Llama-3.2-1B and Llama-2-13B shapes, and the
2048- and 4096-wide sizes of its other architectures); weights and inputs are random with the scales such models have.

Every case's ``kind`` names the path; ``draw`` gives more cases of the same ranges."""
import math
import random

import torch

from ithaca_b200.cache.cache import SequenceCache
from ithaca_b200.config import config_from_dict
from ithaca_b200.config.spec import PartSpec
from ithaca_b200.engine.context import ContextBuilder
from ithaca_b200.engine.graph import GraphDecoder
from ithaca_b200.engine.model import build_model, weight_manifest
from ithaca_b200.engine.step import Stepper
from ithaca_b200.parts import FEED_FORWARDS, HEADS, MIXERS, NORMS, POSITIONS, Runtime

DEVICE = "cuda:0"
EPS = 1e-5
ROPE = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
        "original_max_position_embeddings": 8192}
THETA = 500000.0

# width, heads, kv heads, head size, feed-forward, vocabulary
SHAPES = {"8b": (4096, 32, 8, 128, 14336, 128256), "1b": (2048, 32, 8, 64, 8192, 128256), "13b": (5120, 40, 40, 128, 13824, 32000)}


def listed():
    return [
        # a step of a decoding batch at the benchmark's context: what serving does most of the time
        {"name": "decode step 8b x8", "kind": "decode", "shape": "8b", "layers": 4, "batch": 8, "held": 4095},
        # a batch of unequal prompts entering together (the 1B configuration's workload)
        {"name": "prompt step 1b", "kind": "prompts", "shape": "1b", "layers": 4, "dtype": "bfloat16", "sequences": 12, "new_from": 16, "new_to": 2048},
        # the 32-bit path: a small batch of prompts in true 32-bit arithmetic
        {"name": "prompt step 1b float32", "kind": "prompts", "shape": "1b", "layers": 2, "dtype": "float32", "sequences": 3, "new_from": 30, "new_to": 300},
        # the feed-forward of a long prompt
        {"name": "feed-forward 8b prompt", "kind": "mlp", "shape": "8b", "tokens": 2048},
        # the feed-forward of a large decoding batch
        {"name": "feed-forward 8b x64", "kind": "mlp", "shape": "8b", "tokens": 64},
        # attention of prompts and of a later piece of a prompt, unequal lengths
        {"name": "attention 8b prompts", "kind": "attention", "shape": "8b", "sequences": 3, "new_from": 400, "new_to": 2048, "held": 1000},
        # attention of a decoding batch over a full cache
        {"name": "attention 8b x48", "kind": "attention", "shape": "8b", "sequences": 48, "new_from": 1, "new_to": 1, "held": 3500},
        # the last norm and the head for one sequence: the smallest call
        {"name": "head 1b x1", "kind": "head", "shape": "1b", "rows": 1},
        # routed experts over a prompt
        {"name": "experts prompt", "kind": "moe", "hidden": 2048, "inner": 1024, "experts": 32, "top": 4, "tokens": 4096},
        # a matrix state corrected token by token, two prompts
        {"name": "delta rule prompts", "kind": "delta", "hidden": 2048, "heads": 16, "groups": 4, "head": 128, "sequences": 2, "new_from": 1000, "new_to": 3000, "held": 0},
        # attention over one low-rank row per token, a prompt
        {"name": "latent attention prompt", "kind": "latent", "hidden": 2048, "heads": 16, "head": 128, "rope": 64, "rank": 512, "sequences": 1, "new_from": 4096, "new_to": 4096, "held": 0},
        # a diagonal state per channel, two prompts
        {"name": "selective scan prompts", "kind": "scan", "hidden": 2048, "inner": 4096, "state": 16, "rank": 128, "sequences": 2, "new_from": 1000, "new_to": 3000, "held": 0},
    ]


def spread(rng, lo, hi):
    """A whole number of [lo, hi], even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["decode", "prompts", "prompts32", "mlp", "mlp", "attention", "attention", "head", "moe", "delta", "latent", "scan"])
    shape = rng.choice(["8b", "1b", "13b"])
    if kind == "decode":
        batch = spread(rng, 1, 64)
        return {"kind": kind, "shape": rng.choice(["8b", "1b"]), "layers": rng.randint(1, 4), "batch": batch, "held": spread(rng, 30, min(8000, 32768 // batch))}
    if kind == "prompts":
        n = spread(rng, 1, 12)
        to = spread(rng, 100, 2048)
        return {"kind": kind, "shape": rng.choice(["8b", "1b"]), "layers": rng.randint(1, 2), "dtype": "bfloat16", "sequences": n, "new_from": spread(rng, 16, to), "new_to": to}
    if kind == "prompts32":
        to = spread(rng, 20, 300)
        return {"kind": "prompts", "shape": "1b", "layers": rng.randint(1, 2), "dtype": "float32", "sequences": rng.randint(1, 3), "new_from": spread(rng, 1, to), "new_to": to}
    if kind == "mlp":
        return {"kind": kind, "shape": shape, "tokens": spread(rng, 1, 2048)}
    if kind == "attention":
        if rng.random() < 0.5:
            n = spread(rng, 1, 64)
            return {"kind": kind, "shape": shape, "sequences": n, "new_from": 1, "new_to": 1, "held": spread(rng, 40, min(8000, 60000 // n))}
        n, to = rng.randint(1, 4), spread(rng, 20, 2048)
        return {"kind": kind, "shape": shape, "sequences": n, "new_from": spread(rng, 2, to), "new_to": to, "held": rng.choice([0, spread(rng, 20, 4000)])}
    if kind == "head":
        return {"kind": kind, "shape": shape, "rows": spread(rng, 1, 64)}
    if kind == "moe":
        e = rng.choice([(2048, 1024, 32, 4), (4096, 3584, 16, 2), (2048, 1024, 16, 4)])
        return {"kind": kind, "hidden": e[0], "inner": e[1], "experts": e[2], "top": e[3], "tokens": spread(rng, 1, 4096)}
    wide = rng.random() < 0.4
    many = {"sequences": spread(rng, 1, 64), "new_from": 1, "new_to": 1, "held": rng.randint(40, 300)} if rng.random() < 0.3 else None
    if many is None:
        to = spread(rng, 60, 3000)
        many = {"sequences": rng.randint(1, 3), "new_from": spread(rng, 10, to), "new_to": to, "held": 0}
    hidden = 4096 if wide else 2048
    if kind == "delta":
        return dict({"kind": kind, "hidden": hidden, "heads": hidden // 128, "groups": hidden // 512, "head": 128}, **many)
    if kind == "latent":
        return dict({"kind": kind, "hidden": hidden, "heads": hidden // 128, "head": 128, "rope": 64, "rank": 512}, **many)
    return dict({"kind": kind, "hidden": hidden, "inner": 2 * hidden, "state": 16, "rank": hidden // 16}, **many)


# -- sizes ---------------------------------------------------------------------------------------------------------------
def lengths(case):
    """How many tokens every sequence brings: spread over the case's range, the same for every seed."""
    lo, hi, n = case["new_from"], case["new_to"], case["sequences"]
    r = random.Random(f"{lo} {hi} {n}")
    return [hi] + [r.randint(lo, hi) for _ in range(n - 1)]


def held(case):
    """How many positions every sequence holds before the pass: the last of them all of ``held``, the others less."""
    n, h = case["sequences"], case["held"]
    if h == 0:
        return [0] * n
    r = random.Random(f"{h} {n}")
    return [r.randint(max(1, h // 4), h) for _ in range(n - 1)] + [h]


def llama_config(case):
    d, nh, nkv, hd, ff, vocab = SHAPES[case["shape"]]
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": d, "num_hidden_layers": case["layers"], "num_attention_heads": nh,
            "num_key_value_heads": nkv, "head_dim": hd, "intermediate_size": ff, "vocab_size": vocab, "rope_theta": THETA,
            "rope_scaling": dict(ROPE), "rms_norm_eps": EPS, "max_position_embeddings": 16384,
            "tie_word_embeddings": case["shape"] == "1b", "torch_dtype": "bfloat16"}


# -- random tensors, the same for prepare() and exact() ---------------------------------------------------------------------
class Source:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(generator=self.g)
        return t.mul_(std).add_(mean).to(dtype)

    def weight(self, rows, cols):
        """A projection's matrix: its results have the scale of its inputs."""
        return self.normal(rows, cols, std=cols ** -0.5)

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.g, device=DEVICE).tolist()


def part_tensors(case, src):
    """The tensors of a layer's part by name, and the part's specification."""
    k = case["kind"]
    if k == "mlp":
        d, _, _, _, ff, _ = SHAPES[case["shape"]]
        return {"gate": src.weight(ff, d), "up": src.weight(ff, d), "down": src.weight(d, ff)}, PartSpec(
            "gated_mlp", {"hidden_size": d, "intermediate_size": ff, "activation": "silu"}, {r: r for r in ("gate", "up", "down")})
    if k == "attention":
        d, nh, nkv, hd, _, _ = SHAPES[case["shape"]]
        return {"q": src.weight(nh * hd, d), "k": src.weight(nkv * hd, d), "v": src.weight(nkv * hd, d), "o": src.weight(d, nh * hd)}, PartSpec(
            "attention", {"hidden_size": d, "n_heads": nh, "n_kv_heads": nkv, "head_dim": hd, "window": None, "scale": None}, {r: r for r in "qkvo"})
    if k == "moe":
        d, ff, E = case["hidden"], case["inner"], case["experts"]
        t = {"router": src.normal(E, d, std=2 * d ** -0.5)}
        for e in range(E):
            t[f"g{e}"], t[f"u{e}"], t[f"d{e}"] = src.weight(ff, d), src.weight(ff, d), src.weight(d, ff)
        return t, PartSpec("moe", {"hidden_size": d, "intermediate_size": ff, "n_experts": E, "top": case["top"], "n_groups": 4, "group_keep": 2},
                           {"router": "router", "gate": "g{e}", "up": "u{e}", "down": "d{e}"})
    if k == "delta":
        d, H, G, hd = case["hidden"], case["heads"], case["groups"], case["head"]
        t = {"q": src.weight(G * hd, d), "k": src.weight(G * hd, d), "v": src.weight(H * hd, d), "g": src.weight(H * hd, d), "b": src.weight(H, d),
             "a": src.weight(H, d), "A_log": src.normal(H, std=0.5, mean=-2.0, dtype=torch.float32), "dt_bias": src.normal(H, std=0.5, dtype=torch.float32),
             "norm": src.normal(hd, std=0.1, mean=1.0, dtype=torch.float32), "o": src.weight(d, H * hd)}
        for r, rows in (("q_conv", G * hd), ("k_conv", G * hd), ("v_conv", H * hd)):
            t[r] = src.normal(rows, 4, std=0.5, dtype=torch.float32)
        return t, PartSpec("gated_delta", {"hidden_size": d, "n_heads": H, "n_qk_heads": G, "head_dim": hd, "v_head_dim": hd, "conv_taps": 4,
                                           "norm_eps": 1e-6}, {r: r for r in t})
    if k == "latent":
        d, H, hd, rd, rank = case["hidden"], case["heads"], case["head"], case["rope"], case["rank"]
        t = {"q": src.weight(H * (hd + rd), d), "dkv": src.weight(rank + rd, d), "dkv_norm": src.normal(rank, std=0.1, mean=1.0, dtype=torch.float32),
             "uk": src.weight(H * hd, rank), "uv": src.weight(H * hd, rank), "g": src.weight(H * hd, d), "o": src.weight(d, H * hd)}
        return t, PartSpec("latent_attention", {"hidden_size": d, "n_heads": H, "head_dim": hd, "rope_dim": rd, "v_head_dim": hd, "kv_rank": rank,
                                                "scale": (hd + rd) ** -0.5, "norm_eps": 1e-6, "window": None, "head_gate": "wide"}, {r: r for r in t})
    if k == "scan":
        d, inner, N, R = case["hidden"], case["inner"], case["state"], case["rank"]
        t = {"in": src.weight(2 * inner, d), "conv": src.normal(inner, 4, std=0.5, dtype=torch.float32), "conv_bias": src.normal(inner, std=0.1, dtype=torch.float32),
             "x": src.weight(R + 2 * N, inner), "dt": src.weight(inner, R), "dt_bias": src.normal(inner, std=0.5, mean=-3.0, dtype=torch.float32),
             "A_log": torch.log(torch.arange(1, N + 1, dtype=torch.float32, device=DEVICE)).expand(inner, N).contiguous(),
             "D": src.normal(inner, std=0.1, mean=1.0, dtype=torch.float32), "o": src.weight(d, inner)}
        return t, PartSpec("mamba1", {"hidden_size": d, "inner": inner, "state": N, "dt_rank": R, "conv_taps": 4}, {r: r for r in t})
    raise ValueError(k)


def model_tensors(case, src):
    _, cfg = config_from_dict(llama_config(case))
    out = {}
    for name, req in weight_manifest(cfg.model_spec()).items():
        shape = tuple(req.shape)
        if len(shape) == 1:
            out[name] = src.normal(*shape, std=0.05, mean=1.0)
        elif "embed_tokens" in name:
            out[name] = src.normal(*shape, std=0.02)
        else:
            out[name] = src.weight(*shape)
    return out


STATES = {"delta": "delta_state", "scan": "scan_state"}


# -- the calls ----------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    src, k = Source(seed), case["kind"]
    rt = Runtime(case.get("dtype", "bfloat16"), DEVICE)
    if k in ("decode", "prompts"):
        arch, cfg = config_from_dict(llama_config(case))
        model = build_model(arch, cfg, model_tensors(case, src), rt)
        if k == "prompts":
            new, old = lengths(case), [0] * case["sequences"]
        else:
            new, old = [1] * case["batch"], [case["held"]] * case["batch"]
        pages = sum(-(-(a + b) // 64) for a, b in zip(new, old))
        cache = SequenceCache(model.cache_requests(), max_tokens=64 * pages, kv_dtype=rt.kv_dtype, device=DEVICE)
        step = Stepper(model, cache, max_step_tokens=16384)
        slots = [cache.alloc_slot() for _ in new]
        history = [src.ids(n, cfg.vocab_size) for n in old]
        tokens = [src.ids(n, cfg.vocab_size) for n in new]
        state = {"kind": k, "cache": cache, "step": step, "slots": slots, "tokens": tokens, "old": old}
        if k == "decode":
            for s, h in zip(slots, history):
                step.step([s], [h], None)
            state["decoder"] = GraphDecoder(step)
            run(state)                      # the step of this shape is captured once, as a decoding program does
        return state
    if k == "mlp":
        t, spec = part_tensors(case, src)
        part = FEED_FORWARDS.get(spec.kind)(spec, t, rt)
        x = src.normal(case["tokens"], spec["hidden_size"])
        return {"kind": k, "part": part, "x": x, "y": torch.empty(x.shape, dtype=torch.float32, device=DEVICE)}
    if k == "moe":
        t, spec = part_tensors(case, src)
        part = FEED_FORWARDS.get(spec.kind)(spec, t, rt)
        x = src.normal(case["tokens"], spec["hidden_size"])
        return {"kind": k, "part": part, "x": x, "y": torch.empty(x.shape, dtype=torch.float32, device=DEVICE)}
    if k == "head":
        d, _, _, _, _, vocab = SHAPES[case["shape"]]
        t = {"norm": src.normal(d, std=0.05, mean=1.0), "head": src.weight(vocab, d)}
        norm = NORMS.get("rmsnorm")(PartSpec("rmsnorm", {"size": d, "eps": EPS}, {"weight": "norm"}), t, rt)
        head = HEADS.get("lm_head")(PartSpec("lm_head", {"vocab_size": vocab, "hidden_size": d}, {"weight": "head"}), t, rt)
        return {"kind": k, "norm": norm, "head": head, "x": src.normal(case["rows"], d, std=3.0, dtype=torch.float32)}
    t, spec = part_tensors(case, src)
    if k == "attention":
        pos = PartSpec("rotary", {"rotary_dim": spec["head_dim"], "theta": THETA, "pairing": "half", "scaling": dict(ROPE)})
    elif k == "latent":
        pos = PartSpec("rotary", {"rotary_dim": spec["rope_dim"], "theta": THETA, "pairing": "interleaved", "scaling": None})
    else:
        pos = None
    more = {"position": POSITIONS.get("rotary")(pos, {}, rt)} if pos is not None else {}
    part = MIXERS.get(spec.kind)(spec, t, rt, **more)
    new, old = lengths(case), held(case)
    cache = SequenceCache({0: part.cache_requests()}, max_tokens=64 * sum(-(-(a + b) // 64) for a, b in zip(new, old)),
                          max_slots=case["sequences"], device=DEVICE)
    slots = [cache.alloc_slot() for _ in new]
    assert slots == list(range(len(slots)))
    build = ContextBuilder(DEVICE)

    def context(counts, start, which):
        cache.reserve(which, counts)
        cols = max(-(-(a + b) // 64) for a, b in zip(counts, start))
        tables = [cache.table.table_rows(g, which, cols) for g in range(len(cache.kv_groups))]
        return build.build(which, [[0] * n for n in counts], start, [[] for _ in counts], tables)

    past = [src.normal(n, spec["hidden_size"]) if n else None for n in old]
    for s, n in zip(slots, old):
        if n:
            y = torch.empty((n, spec["hidden_size"]), dtype=torch.float32, device=DEVICE)
            part.forward(past[s], context([n], [0], [s]), cache.layer(0), y, True, accumulate=False)
            cache.commit([s], [n])
    x = src.normal(sum(new), spec["hidden_size"])
    return {"kind": k, "part": part, "layer": cache.layer(0), "cache": cache, "ctx": context(new, old, slots), "x": x,
            "y": torch.empty(x.shape, dtype=torch.float32, device=DEVICE)}


def run(state):
    """A layer's result (float32, as it would join the residual stream) and, of a mixer with a state of fixed size, that
    state; a model's logits."""
    k = state["kind"]
    if k in ("mlp", "moe"):
        state["part"].forward(state["x"], None, state["y"], accumulate=False)
        return state["y"]
    if k == "head":
        return state["head"].forward(state["norm"].forward(state["x"]))
    if k in ("decode", "prompts"):
        for s, n in zip(state["slots"], state["old"]):
            state["cache"].truncate(s, n)
        if k == "decode":
            return state["decoder"].step(state["slots"], state["tokens"])[0]
        return state["step"].step(state["slots"], state["tokens"], "last")
    state["part"].forward(state["x"], state["ctx"], state["layer"], state["y"], True, accumulate=False)
    if k in STATES:
        return state["y"], state["layer"].state(STATES[k])
    return state["y"]


# -- what a pass cannot do without -----------------------------------------------------------------------------------------
def pairs(new, old):
    """(query, key) pairs under the causal mask."""
    return sum(n * o + n * (n + 1) // 2 for n, o in zip(new, old))


def work(case):
    k = case["kind"]
    if k in ("mlp", "head", "moe"):
        if k == "moe":
            d, ff, T = case["hidden"], case["inner"], case["tokens"]
            met = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** T)         # experts that some token meets
            return {"bytes": met * 3 * d * ff * 2 + T * d * 6, "flops": 2 * T * (3 * d * ff * case["top"] + d * case["experts"])}
        d, _, _, _, ff, vocab = SHAPES[case["shape"]]
        T, n = (case["tokens"], 3 * ff) if k == "mlp" else (case["rows"], vocab)
        return {"bytes": n * d * 2 + T * d * 6 if k == "mlp" else n * d * 2 + T * (d + n) * 4, "flops": 2 * T * n * d}
    if k in ("decode", "prompts"):
        d, nh, nkv, hd, ff, vocab = SHAPES[case["shape"]]
        new = [1] * case["batch"] if k == "decode" else lengths(case)
        old = [case["held"]] * case["batch"] if k == "decode" else [0] * len(new)
        size = 4 if case.get("dtype") == "float32" else 2
        T, per = sum(new), d * (2 * nh + 2 * nkv) * hd + 3 * d * ff
        cache = sum(new) + sum(old)
        return {"bytes": case["layers"] * (per * 2 + cache * 2 * nkv * hd * size) + vocab * d * 2 + len(new) * vocab * 4,
                "flops": case["layers"] * (2 * T * per + 4 * nh * hd * pairs(new, old)) + 2 * len(new) * vocab * d}
    new, old = lengths(case), held(case)
    T = sum(new)
    if k == "attention":
        d, nh, nkv, hd, _, _ = SHAPES[case["shape"]]
        per = d * (2 * nh + 2 * nkv) * hd
        return {"bytes": per * 2 + (T + sum(old)) * 2 * nkv * hd * 2 + T * d * 6, "flops": 2 * T * per + 4 * nh * hd * pairs(new, old)}
    d = case["hidden"]
    if k == "latent":
        H, hd, rd, rank = case["heads"], case["head"], case["rope"], case["rank"]
        per = d * (H * (hd + rd) + rank + rd + 2 * H * hd)
        # a score is head + rope products and a value head more, once keys and values are formed from the rows (or, for few
        # queries, the same carried into the rows' space)
        each = 2 * H * hd * rank
        return {"bytes": (per + each) * 2 + (T + sum(old)) * (rank + rd) * 2 + T * d * 6,
                "flops": 2 * T * (per + each) + 2 * H * (2 * hd + rd) * pairs(new, old)}
    if k == "delta":
        H, G, hd = case["heads"], case["groups"], case["head"]
        per = d * (2 * G * hd + 3 * H * hd + 2 * H)
        return {"bytes": per * 2 + len(new) * H * hd * hd * 4 * (2 if case["held"] else 1) + T * d * 6, "flops": 2 * T * per + 6 * T * H * hd * hd}
    inner, N, R = case["inner"], case["state"], case["rank"]
    per = d * 3 * inner + (2 * R + 2 * N) * inner
    return {"bytes": per * 2 + len(new) * inner * N * 4 * (2 if case["held"] else 1) + T * d * 6, "flops": 2 * T * per + 6 * T * inner * N}


def tolerance(case):
    """About four times the distance measured from the results in 64 bits.  32-bit: sums of some thousand float products in
    another order (4e-6).  16-bit: a layer rounds its operands and one or two intermediate results to 8 bits of mantissa (2 to
    4e-3); in a whole model such a change travels on through the layers behind it (9e-3)."""
    if case.get("dtype") == "float32":
        return {"rel": 1.5e-5, "max": 2e-4}
    if case["kind"] in ("decode", "prompts"):
        return {"rel": 3e-2, "max": 0.3}
    if case["kind"] == "moe":
        return {"rel": 1.5e-2, "max": 0.9}          # two experts' scores may be as good as equal: such a token differs whole
    return {"rel": 1.5e-2, "max": 0.2}


# -- the results in 64 bits ------------------------------------------------------------------------------------------------
def f64(t):
    return t.to(torch.float64)


def frequencies(dim, scaled):
    f = [THETA ** (-2.0 * i / dim) for i in range(dim // 2)]
    if scaled:
        low, high, factor = ROPE["low_freq_factor"], ROPE["high_freq_factor"], ROPE["factor"]
        for i, v in enumerate(f):
            turns = ROPE["original_max_position_embeddings"] * v / (2 * math.pi)
            mix = min(1.0, max(0.0, (turns - low) / (high - low)))
            f[i] = (1 - mix) * v / factor + mix * v
    return torch.tensor(f, dtype=torch.float64, device=DEVICE).to(torch.float32)       # the table is float32 by definition


def rotate(x, positions, freq, neighbours=False):
    """x [T, heads, size] turned by position; pairs are (i, i + half) or neighbours.  The angle is a float32 product by definition."""
    a = f64(positions.to(torch.float32)[:, None] * freq[None])[:, None, :]
    c, s = torch.cos(a), torch.sin(a)
    if neighbours:
        x0, x1 = x[..., 0::2], x[..., 1::2]
        return torch.stack((x0 * c - x1 * s, x0 * s + x1 * c), dim=-1).flatten(-2)
    x0, x1 = x.chunk(2, dim=-1)
    return torch.cat((x0 * c - x1 * s, x0 * s + x1 * c), dim=-1)


def attend64(q, k, v, scale):
    """q [n, H, a] behind k [m, G, a], v [m, G, c]: causal, the last query sees every key."""
    n, H, _ = q.shape
    m, G, _ = k.shape
    out = torch.empty((n, H, v.shape[2]), dtype=torch.float64, device=DEVICE)
    for lo in range(0, n, 2048):
        hi = min(n, lo + 2048)
        seen = torch.arange(m, device=DEVICE)[None] <= (torch.arange(lo, hi, device=DEVICE) + m - n)[:, None]
        for g in range(G):
            hs = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("nha,ma->hnm", q[lo:hi, hs], k[:, g]) * scale
            s = s.masked_fill(~seen, -math.inf).softmax(-1)
            out[lo:hi, hs] = torch.einsum("hnm,mc->nhc", s, v[:, g])
    return out


def rms64(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * f64(w)


def mlp64(x, gate, up, down):
    return (torch.nn.functional.silu(x @ f64(gate).T) * (x @ f64(up).T)) @ f64(down).T


def llama64(case, src):
    d, nh, nkv, hd, _, vocab = SHAPES[case["shape"]]
    w = model_tensors(case, src)
    new = [1] * case["batch"] if case["kind"] == "decode" else lengths(case)
    old = [case["held"]] * case["batch"] if case["kind"] == "decode" else [0] * len(new)
    history = [src.ids(n, vocab) for n in old]
    tokens = [src.ids(n, vocab) for n in new]
    freq, out = frequencies(hd, True), []
    head = f64(w["lm_head.weight"] if "lm_head.weight" in w else w["model.embed_tokens.weight"])
    for a, b in zip(history, tokens):
        ids = torch.tensor(a + b, device=DEVICE)
        at = torch.arange(len(ids), device=DEVICE)
        h = f64(w["model.embed_tokens.weight"][ids])
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            x = rms64(h, w[p + "input_layernorm.weight"], EPS)
            q, k, v = (x @ f64(w[f"{p}self_attn.{r}_proj.weight"]).T for r in "qkv")
            q, k = rotate(q.view(-1, nh, hd), at, freq), rotate(k.view(-1, nkv, hd), at, freq)
            o = attend64(q, k, v.view(-1, nkv, hd), hd ** -0.5).flatten(1)
            h = h + o @ f64(w[p + "self_attn.o_proj.weight"]).T
            x = rms64(h, w[p + "post_attention_layernorm.weight"], EPS)
            h = h + mlp64(x, w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"], w[p + "mlp.down_proj.weight"])
        out.append(rms64(h[-1:], w["model.norm.weight"], EPS) @ head.T)
    return torch.cat(out)


def conv64(x, w):
    """The causal convolution over time of one sequence's channels: x [T, c], w [c, taps], the last tap meets the current token."""
    taps = w.shape[1]
    z = torch.cat((torch.zeros((taps - 1, x.shape[1]), dtype=torch.float64, device=DEVICE), x))
    return sum(z[i:i + len(x)] * f64(w[:, i]) for i in range(taps))


def delta64(case, t, x, states, slot, before):
    """One sequence; ``before``: positions it held (their state is kept beside the new one)."""
    H, G, hd = case["heads"], case["groups"], case["head"]
    q, k, v = (torch.nn.functional.silu(conv64(x @ f64(t[r]).T, t[r + "_conv"])) for r in "qkv")
    q, k = (z.view(-1, G, hd).repeat_interleave(H // G, 1) for z in (q, k))
    q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
    q, v = q * hd ** -0.5, v.view(-1, H, hd)
    b = torch.sigmoid(x @ f64(t["b"]).T)
    g = torch.exp(-torch.exp(f64(t["A_log"])) * torch.nn.functional.softplus(x @ f64(t["a"]).T + f64(t["dt_bias"])))
    S, o = torch.zeros((H, hd, hd), dtype=torch.float64, device=DEVICE), []            # [head, value, key]
    for n in range(len(x)):
        S = S * g[n][:, None, None]
        u = b[n][:, None] * (v[n] - torch.einsum("hvk,hk->hv", S, k[n]))
        S = S + u[:, :, None] * k[n][:, None, :]
        o.append(torch.einsum("hvk,hk->hv", S, q[n]))
        if n + 1 == before or n + 1 == len(x):
            states[slot, n & 1] = S
    o = rms64(torch.stack(o), t["norm"], 1e-6).flatten(1) * torch.nn.functional.silu(x @ f64(t["g"]).T)
    return o @ f64(t["o"]).T


def scan64(case, t, x, states, slot, before):
    inner, N, R = case["inner"], case["state"], case["rank"]
    u, z = (x @ f64(t["in"]).T).chunk(2, dim=1)
    u = torch.nn.functional.silu(conv64(u, t["conv"]) + f64(t["conv_bias"]))
    r, B, C = (u @ f64(t["x"]).T).split((R, N, N), dim=1)
    dt = torch.nn.functional.softplus(r @ f64(t["dt"]).T + f64(t["dt_bias"]))
    A = -torch.exp(f64(t["A_log"]))
    S, y = torch.zeros((inner, N), dtype=torch.float64, device=DEVICE), []
    for n in range(len(x)):
        S = torch.exp(dt[n][:, None] * A) * S + (dt[n] * u[n])[:, None] * B[n]
        y.append(S @ C[n])
        if n + 1 == before or n + 1 == len(x):
            states[slot, n & 1] = S
    y = (torch.stack(y) + f64(t["D"]) * u) * torch.nn.functional.silu(z)
    return y @ f64(t["o"]).T


def latent64(case, t, x, before):
    H, hd, rd, rank = case["heads"], case["head"], case["rope"], case["rank"]
    at, freq = torch.arange(len(x), device=DEVICE), frequencies(rd, False)
    q, ck = (x[before:] @ f64(t["q"]).T).view(-1, H, hd + rd), x @ f64(t["dkv"]).T
    q = torch.cat((q[..., :hd], rotate(q[..., hd:], at[before:], freq, True)), -1)
    c = rms64(ck[:, :rank], t["dkv_norm"], 1e-6)
    turned = rotate(ck[:, None, rank:], at, freq, True).expand(-1, H, -1)
    k = torch.cat(((c @ f64(t["uk"]).T).view(-1, H, hd), turned), -1)
    o = attend64(q, k, (c @ f64(t["uv"]).T).view(-1, H, hd), (hd + rd) ** -0.5).flatten(1)
    return (o * torch.sigmoid(x[before:] @ f64(t["g"]).T)) @ f64(t["o"]).T


def attention64(case, t, x, before):
    d, nh, nkv, hd, _, _ = SHAPES[case["shape"]]
    at, freq = torch.arange(len(x), device=DEVICE), frequencies(hd, True)
    q = rotate((x[before:] @ f64(t["q"]).T).view(-1, nh, hd), at[before:], freq)
    k = rotate((x @ f64(t["k"]).T).view(-1, nkv, hd), at, freq)
    return attend64(q, k, (x @ f64(t["v"]).T).view(-1, nkv, hd), hd ** -0.5).flatten(1) @ f64(t["o"]).T


def moe64(case, t, x):
    E, top = case["experts"], case["top"]
    scores = (x @ f64(t["router"]).T).softmax(-1)
    best = scores.view(len(x), 4, -1).amax(-1)
    kept = torch.zeros_like(best).scatter_(1, best.topk(2, dim=1).indices, 1.0).repeat_interleave(E // 4, 1)
    chosen = (scores * kept).topk(top, dim=1).indices
    y = torch.zeros_like(x)
    for e in range(E):
        rows = (chosen == e).any(1).nonzero()[:, 0]
        if len(rows):
            y[rows] += scores[rows, e, None] * mlp64(x[rows], t[f"g{e}"], t[f"u{e}"], t[f"d{e}"])
    return y


def exact(case, seed):
    src, k = Source(seed), case["kind"]
    if k in ("decode", "prompts"):
        return llama64(case, src)
    if k == "head":
        d, _, _, _, _, vocab = SHAPES[case["shape"]]
        norm, head = src.normal(d, std=0.05, mean=1.0), src.weight(vocab, d)
        return rms64(f64(src.normal(case["rows"], d, std=3.0, dtype=torch.float32)), norm, EPS) @ f64(head).T
    t, spec = part_tensors(case, src)
    if k in ("mlp", "moe"):
        x = f64(src.normal(case["tokens"], spec["hidden_size"]))
        return mlp64(x, t["gate"], t["up"], t["down"]) if k == "mlp" else moe64(case, t, x)
    new, old = lengths(case), held(case)
    past = [f64(src.normal(n, spec["hidden_size"])) if n else None for n in old]
    xs = f64(src.normal(sum(new), spec["hidden_size"])).split(new)
    xs = [x if p is None else torch.cat((p, x)) for p, x in zip(past, xs)]
    if k in ("attention", "latent"):
        one = attention64 if k == "attention" else latent64
        return torch.cat([one(case, t, x, n) for x, n in zip(xs, old)])
    if k == "delta":
        states = torch.zeros((len(new), 2, case["heads"], case["head"], case["head"]), dtype=torch.float64, device=DEVICE)
    else:
        states = torch.zeros((len(new), 2, case["inner"], case["state"]), dtype=torch.float64, device=DEVICE)
    one = delta64 if k == "delta" else scan64
    y = torch.cat([one(case, t, x, states, i, n)[n:] for i, (x, n) in enumerate(zip(xs, old))])
    return y, states
