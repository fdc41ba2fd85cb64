"""What the engine's speed is measured on: the work a program has it do, case by case.

Every layer kind of the Qwen3 dense engine and, of each further design, the mixer or feed-forward that sets it apart, each
called as the model calls it (a part built through the registry, a step's arrays built by the step builder, pages and
states in the cache's storage); and whole calls through ``ModelRunner.step`` that return logits.  A case's portions
(new tokens and tokens already cached of every request) follow from its numbers alone.

Sizes: Qwen3-8B and -4B layers (atom_b200/benchmarks/sizes.py) and the designs at width 2048 with 16 heads and width
1024 with 8 (atom_b200/benchmarks/designs.py).
"""
import math
import random
import zlib

import numpy as np
import torch

from atom_b200.benchmarks.designs import simivik_config
from atom_b200.cache import CacheManager
from atom_b200.cache.storage import CacheStorage
from atom_b200.config import EngineConfig, config_from_dict
from atom_b200.engine.batch import StepBuilder, StepEntry
from atom_b200.engine.runner import ModelRunner
from atom_b200.parts import registry
from atom_b200.parts.base import Runtime, Workspace
from atom_b200.parts.spec import PartSpec

DEV = "cuda:0"
PAGE = 16
EPS = 1e-5
QWEN_EPS = 1e-6
THETA = 1000000.0
VOCAB, LAYERS = 32000, 2            # of the whole model
HIDDEN, HEADS, KV, HEAD, FF = 4096, 32, 8, 128, 12288


# ------------------------------------------------------------------------------------------------------------ the cases


def listed():
    return [
        # a short conversation with 13 users: their prompts in one step, then tokens one by one (whole model, logits)
        {"name": "serve", "kind": "serve", "requests": 13, "tokens": 1501, "past": 0, "steps": 12},
        # the feed-forward of one decoded token of a small model: the smallest call, a read of its weights
        {"name": "mlp_one_row", "kind": "mlp", "hidden": 2560, "ff": 9728, "requests": 1, "tokens": 1, "past": 0},
        # ... and of a prompt's portion of a large one
        {"name": "mlp_portion", "kind": "mlp", "hidden": 4096, "ff": 12288, "requests": 3, "tokens": 1901, "past": 0},
        # attention of prompts in one step, some of them continuing
        {"name": "attention_prompts", "kind": "attention", "dtype": "bfloat16", "requests": 3, "tokens": 6007, "past": 3000},
        # attention of a full decode batch over long contexts
        {"name": "attention_decode", "kind": "attention", "dtype": "bfloat16", "requests": 64, "tokens": 64, "past": 4100},
        # attention of prompts where a program asked for true 32-bit
        {"name": "attention_float32", "kind": "attention", "dtype": "float32", "requests": 2, "tokens": 1030, "past": 400},
        # Nurinex: attention with mixed heads beside a recurrence with a decay per channel
        {"name": "nurinex_mixer", "kind": "nurinex", "width": 2048, "requests": 2, "tokens": 2048, "past": 0},
        # Mugulorn: attention through a latent, a window of 1024
        {"name": "mugulorn_latent", "kind": "mugulorn", "width": 2048, "requests": 2, "tokens": 2048, "past": 700},
        # Simivik: lightning attention (a state per head, one decay per head)
        {"name": "simivik_lightning", "kind": "simivik", "width": 2048, "requests": 3, "tokens": 2048, "past": 900},
        # Kibotar: gated linear attention (a state per head, a decay per channel and token)
        {"name": "kibotar_gla", "kind": "kibotar", "width": 2048, "requests": 2, "tokens": 2048, "past": 900},
        # Vudezen: 16 routed and 4 identity experts in groups beside a shared one
        {"name": "vudezen_experts", "kind": "vudezen", "width": 2048, "requests": 4, "tokens": 1000, "past": 0},
        # Vunepel: differential attention within chunks of 1024
        {"name": "vunepel_attention", "kind": "vunepel", "width": 2048, "requests": 2, "tokens": 2048, "past": 700},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["serve", "mlp", "attention", "attention", "nurinex", "mugulorn", "simivik", "kibotar", "vudezen",
                       "vunepel"])
    if kind == "serve":
        n = rng.randint(1, 13)
        return {"kind": kind, "requests": n, "tokens": max(n, log(13, 1501)), "past": 0, "steps": rng.randint(2, 12)}
    if kind == "mlp":
        hidden, ff = rng.choice([(2560, 9728), (4096, 12288)])
        return {"kind": kind, "hidden": hidden, "ff": ff, "requests": 1, "tokens": log(1, 1901), "past": 0}
    if kind == "attention":
        if rng.random() < 0.4:
            n = log(1, 64)
            return {"kind": kind, "dtype": "bfloat16", "requests": n, "tokens": n, "past": log(17, 4100)}
        if rng.random() < 0.5:
            return {"kind": kind, "dtype": "float32", "requests": rng.randint(1, 4), "tokens": log(4, 1030), "past": rng.randint(0, 400)}
        return {"kind": kind, "dtype": "bfloat16", "requests": rng.randint(1, 8), "tokens": log(8, 6007), "past": rng.randint(0, 3000)}
    width = 2048 if kind == "nurinex" else rng.choice([1024, 2048, 2048])
    if kind != "nurinex" and rng.random() < 0.25:          # a step of single tokens
        n = rng.randint(1, 32)
        return {"kind": kind, "width": width, "requests": n, "tokens": n, "past": log(17, 900)}
    n = rng.randint(1, 6)
    return {"kind": kind, "width": width, "requests": n, "tokens": max(n, log(40, 2048)), "past": rng.choice([0, 0, log(17, 900)])}


def _portions(case):
    """[(tokens cached before, new tokens)] of the case's requests, from its numbers alone."""
    n, total, past = case["requests"], case["tokens"], case["past"]
    rng = random.Random("%d %d %d" % (n, total, past))
    cut = [rng.uniform(0.3, 1.7) for _ in range(n)]
    new = [1 + int((total - n) * c / sum(cut)) for c in cut]
    new[0] += total - sum(new)
    old = [rng.randint(past // 2, past) for _ in range(n)]
    if total > n > 1:
        old[0] = 0                       # one prompt of a step begins
    return list(zip(old, new))


# -------------------------------------------------------------------------------------------------------------- values


def _rand(seed, name, shape, scale=1.0, dtype=torch.bfloat16, uniform=None):
    gen = torch.Generator(device=DEV)
    gen.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
    if uniform is not None:
        t = torch.rand(shape, generator=gen, device=DEV) * (uniform[1] - uniform[0]) + uniform[0]
    else:
        t = torch.randn(shape, generator=gen, device=DEV) * scale
    return t.to(dtype)


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _weights(case, seed):
    """Parameter name -> tensor of the case's part: matrices keep the variance of what they multiply, norm weights lie
    around one, decays reach from nearly nothing forgotten to most of it."""
    dt, k = _dtype(case), case["kind"]
    w = {}

    def mat(name, rows, cols):
        w[name] = _rand(seed, name, (rows, cols), cols ** -0.5, dt)

    def norm(name, n):
        w[name] = _rand(seed, name, (n,), dtype=dt, uniform=(0.8, 1.2))

    if k == "mlp":
        mat("gate_up.weight", 2 * case["ff"], case["hidden"])
        mat("down.weight", case["hidden"], case["ff"])
        return w
    if k == "attention":
        mat("qkv.weight", (HEADS + 2 * KV) * HEAD, HIDDEN)
        mat("o.weight", HIDDEN, HEADS * HEAD)
        norm("q_norm.weight", HEAD)
        norm("k_norm.weight", HEAD)
        return w
    W = case["width"]
    H = W // 128
    G = H // 4
    if k == "nurinex":
        mat("left.qkv.weight", (H + 2 * G) * 128, W)
        mat("left.o.weight", W, H * 128)
        w["left.rel"] = _rand(seed, "rel", (32, H), 0.5, dt)
        w["left.talk"] = (torch.eye(H, device=DEV) + _rand(seed, "talk", (H, H), 0.1, torch.float32)).to(dt)
        w["left.sink"] = _rand(seed, "sink", (H,), 1.0, dt)
        w["right.mu"] = _rand(seed, "mu", (5, W), dtype=dt, uniform=(0.25, 0.75))
        for n in "rkvg":
            mat("right.%s.weight" % n, W, W)
        mat("right.w1.weight", 64, W)
        mat("right.w2.weight", W, 64)
        w["right.w0"] = _rand(seed, "w0", (W,), dtype=dt, uniform=(-6.0, 0.5))
        w["right.u"] = _rand(seed, "u", (W // 64, 64), 0.5, dt)
        norm("right.norm", W)
        mat("right.o.weight", W, W)
        norm("left.out", W)
        norm("right.out", W)
    elif k == "mugulorn":
        mat("in.weight", W // 2 + W // 4 + 64 + H * 128, W)
        norm("dq.norm", W // 2)
        norm("dkv.norm", W // 4)
        mat("uq.weight", H * 192, W // 2)
        mat("uk.weight", H * 128, W // 4)
        mat("uv.weight", H * 128, W // 4)
        w["sink"] = _rand(seed, "sink", (H,), 1.0, dt)
        mat("o.weight", W, H * 128)
    elif k == "simivik":
        mat("qkvg.weight", 4 * H * 128, W)
        norm("norm", H * 128)
        mat("o.weight", W, H * 128)
    elif k == "kibotar":
        mat("in.weight", 4 * H * 128 + 64, W)
        mat("a2.weight", H * 128, 64)
        w["a2.bias"] = _rand(seed, "a2.bias", (H * 128,), dtype=dt, uniform=(-2.0, 6.0))
        norm("norm", 128)
        mat("o.weight", W, H * 128)
    elif k == "vudezen":
        w["router.weight"] = torch.cat([_rand(seed, "router", (20, W), W ** -0.5, dt), torch.zeros((4, W), dtype=dt, device=DEV)])
        w["correction"] = _rand(seed, "correction", (20,), 0.02, dt)
        mat("gate_up.weight", 16 * 2 * W, W)
        mat("down.weight", 16 * W, W)
        mat("shared.gate_up.weight", 2 * W, W)
        mat("shared.down.weight", W, W)
    elif k == "vunepel":
        mat("in.weight", 2 * H * 64 + 2 * G * 64 + G * 128, W)
        mat("o.weight", W, H * 128)
        w["lambdas"] = _rand(seed, "lambdas", (4, 64), 0.1, dt)
        norm("q_norm", 64)
        norm("k_norm", 64)
    return w


def _serve_weights(seed):
    w = {"embedding.weight": _rand(seed, "embedding", (VOCAB, HIDDEN))}
    for i in range(LAYERS):
        p = "layers.%d." % i
        w[p + "mixer_norm.weight"] = _rand(seed, p + "n1", (HIDDEN,), uniform=(0.8, 1.2))
        for n, t in _weights({"kind": "attention"}, seed + 101 * i).items():
            w[p + "mixer." + n] = t
        w[p + "ffn_norm.weight"] = _rand(seed, p + "n2", (HIDDEN,), uniform=(0.8, 1.2))
        for n, t in _weights({"kind": "mlp", "hidden": HIDDEN, "ff": FF}, seed + 101 * i).items():
            w[p + "ffn." + n] = t
    w["final_norm.weight"] = _rand(seed, "norm", (HIDDEN,), uniform=(0.8, 1.2))
    w["lm_head.weight"] = _rand(seed, "head", (VOCAB, HIDDEN), HIDDEN ** -0.5)
    return w


def _decays(H):
    return simivik_config(H * 128, H, 2)["layers"][1]["mixer"]["decay"]


def _spec(case):
    """(registry category, PartSpec) of the case's part."""
    k = case["kind"]
    if k == "mlp":
        return "ffn", PartSpec("gated_silu", {"hidden_size": case["hidden"], "intermediate_size": case["ff"]})
    if k == "attention":
        return "mixer", PartSpec("paged_attention", {
            "hidden_size": HIDDEN, "num_heads": HEADS, "num_kv_heads": KV, "head_dim": HEAD, "qk_norm": True, "norm_eps": QWEN_EPS,
            "position": PartSpec("rope_neox", {"rotary_dim": HEAD, "theta": THETA, "max_position": 40960})})
    W = case["width"]
    H = W // 128
    G = H // 4
    if k == "nurinex":
        left = PartSpec("mixed_head_attention", {
            "hidden_size": W, "num_heads": H, "num_kv_heads": G, "key_dim": 128, "value_dim": 128, "scale": 128 ** -0.5,
            "norm_eps": EPS, "value_norm": True, "head_mixing": True, "sink": True, "bias_rows": 32, "bias_max_distance": 4096,
            "temp_coef": 0.5, "temp_every": 64})
        right = PartSpec("decayed_state_mixing", {"hidden_size": W, "num_heads": W // 64, "head_dim": 64, "decay_rank": 64, "norm_eps": EPS})
        return "mixer", PartSpec("side_by_side", {"hidden_size": W, "norm_eps": EPS, "members": {"left": left, "right": right}})
    if k == "mugulorn":
        return "mixer", PartSpec("latent_attention", {
            "hidden_size": W, "num_heads": H, "head_dim": 128, "rot_dim": 64, "value_dim": 128, "q_rank": W // 2, "kv_rank": W // 4,
            "scale": 192 ** -0.5, "norm_eps": EPS, "position": PartSpec("rope_yarn", {"rotary_dim": 64, "theta": THETA}),
            "window": 1024, "cache_window": 1024, "sink": True, "gate": True})
    if k == "simivik":
        return "mixer", PartSpec("lightning_attention", {"hidden_size": W, "num_heads": H, "key_dim": 128, "value_dim": 128,
                                                         "decay": _decays(H), "norm_eps": EPS})
    if k == "kibotar":
        return "mixer", PartSpec("gated_linear_attention", {"hidden_size": W, "num_heads": H, "key_dim": 128, "value_dim": 128,
                                                            "decay_rank": 64, "tau": 8.0, "norm_eps": EPS})
    if k == "vudezen":
        return "ffn", PartSpec("routed_experts", {
            "hidden_size": W, "num_experts": 16, "top": 2, "intermediate_size": W, "shared_size": W, "score": "softmax",
            "renormalize": True, "weight_on": "output", "correction": True, "groups": (4, 2), "identity": 4, "factor": 1.5,
            "sum_eps": 1e-20, "limit": 7.0, "shared_limit": 7.0})
    return "mixer", PartSpec("differential_attention", {
        "hidden_size": W, "num_heads": H, "num_kv_heads": G, "key_dim": 64, "value_dim": 128, "scale": 64 ** -0.5, "diff": 0.4,
        "norm_eps": EPS, "position": PartSpec("rope_yarn", {"rotary_dim": 64, "theta": THETA}), "chunk": 1024})


def _width(case):
    return case.get("width") or case.get("hidden") or HIDDEN


def _cached(case, seed, i, old):
    """What request i has in the cache: entry -> [vectors, old, size] for pages, state -> array."""
    k, dt = case["kind"], _dtype(case)

    def r(name, shape, scale=1.0, dtype=dt):
        return _rand(seed, "past %s %d" % (name, i), shape, scale if old else 0.0, dtype)

    if k == "attention":
        return {"k": r("k", (KV, old, HEAD)), "v": r("v", (KV, old, HEAD))}, {}
    W = _width(case)
    H = W // 128
    G = H // 4
    if k == "nurinex":
        return ({"k": r("k", (G, old, 128)), "v": r("v", (G, old, 128))},
                {"right.wkv": r("wkv", (W // 64, 64, 64), 1.0, torch.float32), "right.shift": r("shift", (W,))})
    if k == "mugulorn":
        return {"latent": r("latent", (1, old, W // 4 + 64))}, {}
    if k in ("simivik", "kibotar"):
        return {}, {"S": r("S", (H, 128, 128), 1.0, torch.float32)}
    if k == "vunepel":
        return {"k": r("k", (2 * G, old, 64)), "v": r("v", (G, old, 128))}, {}
    return {}, {}


def _prompts(case, seed):
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 5])
    return [rng.integers(0, VOCAB, new + case["steps"]).tolist() for _, new in _portions(case)]


# ---------------------------------------------------------------------------------------------------------- prepare, run


def prepare(case, seed):
    if case["kind"] == "serve":
        return _prepare_serve(case, seed)
    dt = _dtype(case)
    rt = Runtime(dt, torch.device(DEV), Workspace(torch.device(DEV)))
    category, spec = _spec(case)
    part = registry.build(category, spec)
    part.bind(_weights(case, seed), rt)
    part.after_load()
    ports = _portions(case)
    need = part.cache_need() if category == "mixer" else None
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    pages = sum(-(-(o + n) // PAGE) for o, n in ports) + 1
    manager = CacheManager({0: need} if need is not None else {}, PAGE, pages, len(ports))
    storage = CacheStorage(manager, dt, torch.device(DEV))
    builder = StepBuilder(manager, DEV, 1 << 30, status)
    view = storage.view(0) if need is not None else None
    entries, targets = [], []
    for i, (old, new) in enumerate(ports):
        manager.admit(i)
        page_rows, states = _cached(case, seed, i, old)
        if old:
            manager.extend(i, old)
            manager.commit(i, old)
        manager.extend(i, old + new)
        if old and page_rows:
            table = torch.tensor(manager.table(i, view.group)[: -(-old // PAGE)], device=DEV)
            for name, rows in page_rows.items():
                for p in range(table.numel()):
                    if int(table[p]) < 0:
                        continue
                    part_rows = rows[:, p * PAGE:min(old, (p + 1) * PAGE)]
                    dst = view.pages[name][int(table[p])]
                    dst.view(-1, PAGE, dst.shape[-1])[:, : part_rows.shape[1]].copy_(part_rows)
        if old:
            for name, value in states.items():
                view.states[name][manager.requests[i].state_slot].copy_(value)
        entries.append(StepEntry(i, [0] * new, ()))
        targets.append(old + new)
    step = builder.build(entries, targets)
    x = _rand(seed, "x", (case["tokens"], _width(case)), dtype=dt)
    return {"part": part, "x": x, "step": step, "view": view, "mixer": category == "mixer", "keep": (manager, storage, builder)}


def _prepare_serve(case, seed):
    cfg = {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": LAYERS, "hidden_size": HIDDEN, "num_attention_heads": HEADS,
           "num_key_value_heads": KV, "head_dim": HEAD, "intermediate_size": FF, "vocab_size": VOCAB, "rope_theta": THETA,
           "rms_norm_eps": QWEN_EPS, "tie_word_embeddings": False, "max_position_embeddings": 4096, "hidden_act": "silu",
           "attention_bias": False}
    prompts = _prompts(case, seed)
    pages = sum(-(-len(p) // PAGE) for p in prompts) + 8
    runner = ModelRunner(EngineConfig(model="", dtype="bfloat16", load_dummy="random", seed=1, kv_cache_block_size=PAGE,
                                      num_kvcache_blocks=pages, max_num_seqs=16, max_num_batched_tokens=2048),
                         config_from_dict(cfg))
    mine = _serve_weights(seed)
    for path, part, _ in runner.model.named_parts():
        for name in part.params():
            getattr(part, "w_" + name.replace(".", "_")).copy_(mine[path + "." + name])
        part.after_load()
    state = {"runner": runner, "prompts": prompts, "steps": case["steps"]}
    run(state)                        # an engine in service has its buffers and its graphs
    return state


def run(state):
    if "runner" in state:
        runner, prompts, steps = state["runner"], state["prompts"], state["steps"]
        n = [len(p) - steps for p in prompts]
        out = [runner.step([StepEntry(i, p[: n[i]], (n[i] - 1,)) for i, p in enumerate(prompts)]).clone()]
        for k in range(steps):
            out.append(runner.step([StepEntry(i, [p[n[i] + k]], (0,)) for i, p in enumerate(prompts)]).clone())
        for i in range(len(prompts)):
            runner.finish(i)
        return out
    part, view = state["part"], state["view"]
    if not state["mixer"]:
        return {"out": part.forward(state["x"], state["step"])}
    got = {"out": part.forward(state["x"], state["step"], view, True)}
    for name, t in view.pages.items():
        got["pages " + name] = t
    for name, t in view.states.items():
        got["state " + name] = t
    return got


# ------------------------------------------------------------------------------------------- the same in 64 bits, by itself


def _rms(x, eps, w=None):
    y = x / (x.square().mean(-1, keepdim=True) + eps).sqrt()
    return y if w is None else y * w


def _rotate(x, pos, dims):
    """x [T, heads, size]: pairs (i, i + dims / 2) of the first ``dims`` numbers turned by pos * THETA^(-2i / dims)."""
    f = THETA ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEV) / dims)
    a = (pos.double()[:, None] * f)[:, None]
    x1, x2, rest = x[..., : dims // 2], x[..., dims // 2:dims], x[..., dims:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin(), rest], -1)


def _attend(q, k, v, scale, seen, sink=None, lam=None):
    """q [n, heads, dk], k [m, kv, dk], v [m, kv, dv], seen [n, m] -> [n, heads, dv]; query h reads head h // (heads / kv)."""
    n, heads, _ = q.shape
    group, out = heads // k.shape[1], torch.empty((n, heads, v.shape[2]), dtype=torch.float64, device=DEV)
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T * scale).masked_fill_(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        p = s.softmax(1)
        out[:, h] = (p[:, :-1] if sink is not None else p) @ v[:, h // group]
    return out


def _requests(case, seed):
    """(request, its tokens cached before, slice of its new rows, positions of these, what is cached)."""
    at = 0
    for i, (old, new) in enumerate(_portions(case)):
        pages, states = _cached(case, seed, i, old)
        yield (i, old, slice(at, at + new), torch.arange(old, old + new, device=DEV),
               {n: t.double().transpose(0, 1) for n, t in pages.items()}, {n: t.double() for n, t in states.items()})
        at += new


def _causal(old, pos):
    return torch.arange(old + len(pos), device=DEV)[None] <= pos[:, None]


def _attention64(w, x, old, pos, kc, vc):
    qkv = x @ w["qkv.weight"].T
    q, k, v = qkv.split([HEADS * HEAD, KV * HEAD, KV * HEAD], 1)
    q = _rotate(_rms(q.unflatten(1, (HEADS, HEAD)), QWEN_EPS, w["q_norm.weight"]), pos, HEAD)
    k = _rotate(_rms(k.unflatten(1, (KV, HEAD)), QWEN_EPS, w["k_norm.weight"]), pos, HEAD)
    k, v = torch.cat([kc, k]), torch.cat([vc, v.unflatten(1, (KV, HEAD))])
    return _attend(q, k, v, HEAD ** -0.5, _causal(old, pos)).flatten(1) @ w["o.weight"].T


def _mlp64(w, x):
    gate, up = (x @ w["gate_up.weight"].T).chunk(2, 1)
    return (torch.nn.functional.silu(gate) * up) @ w["down.weight"].T


def _states(S, q, k, v, decay, before=False, bonus=None):
    """The recurrence S <- diag(decay) S + k v^T token by token; o = S^T q after the token's own term, or with ``before``
    of the state in front of it plus the bonus' share of the token."""
    o = torch.empty_like(v)
    for t in range(len(q)):
        kv = k[t][:, :, None] * v[t][:, None, :]
        if before:
            o[t] = torch.einsum("hk,hkv->hv", q[t], S + bonus[:, :, None] * kv)
            S = decay[t][:, :, None] * S + kv
        else:
            S = decay[t][:, :, None] * S + kv
            o[t] = torch.einsum("hk,hkv->hv", q[t], S)
    return o, S


def _nurinex64(case, seed, w, x):
    W = case["width"]
    H = W // 128
    G, H2 = H // 4, W // 64
    silu = torch.nn.functional.silu
    out, wkvs, shifts = torch.empty_like(x), [], []
    half, rows = 16, 32

    def bucket(n):
        return n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(4096 / half) * (rows - half))))

    for i, old, s, pos, pages, states in _requests(case, seed):
        h = x[s]
        q, k, v = (h @ w["left.qkv.weight"].T).split([H * 128, G * 128, G * 128], 1)
        k = torch.cat([pages["k"], k.unflatten(1, (G, 128))])
        v = torch.cat([pages["v"], _rms(v.unflatten(1, (G, 128)), EPS)])
        q = q.unflatten(1, (H, 128))
        temp = 1 + 0.5 * torch.log(torch.floor((pos.double() + 1) / 64) + 1)
        dist = (pos[:, None] - torch.arange(old + len(pos), device=DEV)[None])
        table = torch.tensor([bucket(d) for d in range(old + len(pos))], device=DEV)
        seen = dist >= 0
        b = table[dist.clamp(min=0)]
        scores = torch.stack([q[:, g] @ k[:, g // 4].T * (128 ** -0.5 * temp)[:, None] + w["left.rel"][:, g][b] for g in range(H)])
        o = torch.empty((len(pos), H, 128), dtype=torch.float64, device=DEV)
        for g in range(H):
            m = torch.einsum("g,gij->ij", w["left.talk"][g], scores).masked_fill_(~seen, -math.inf)
            o[:, g] = torch.cat([m, w["left.sink"][g].expand(len(pos), 1)], 1).softmax(1)[:, :-1] @ v[:, g // 4]
        left = o.flatten(1) @ w["left.o.weight"].T
        before = torch.cat([states["right.shift"][None], h[:-1]])
        mix = [h + (before - h) * w["right.mu"][j] for j in range(5)]
        r, k, v, g = (mix[j] @ w["right.%s.weight" % n].T for j, n in enumerate("rkvg"))
        d = torch.tanh(mix[4] @ w["right.w1.weight"].T) @ w["right.w2.weight"].T + w["right.w0"]
        heads = lambda t: t.unflatten(1, (H2, 64))  # noqa: E731
        y, S = _states(states["right.wkv"], heads(r), heads(k), heads(v), torch.exp(-torch.exp(heads(d))), True, w["right.u"])
        right = (_rms(y, EPS).flatten(1) * w["right.norm"] * silu(g)) @ w["right.o.weight"].T
        out[s] = (_rms(left, EPS, w["left.out"]) + _rms(right, EPS, w["right.out"])) / 2
        wkvs.append(S)
        shifts.append(h[-1])
    return {"out": out, "pages k": None, "pages v": None, "state right.wkv": torch.stack(wkvs), "state right.shift": torch.stack(shifts)}


def _mugulorn64(case, seed, w, x):
    W = case["width"]
    H, R = W // 128, W // 4
    out = torch.empty_like(x)
    for i, old, s, pos, pages, _ in _requests(case, seed):
        dq, c, kr, g = (x[s] @ w["in.weight"].T).split([W // 2, R, 64, H * 128], 1)
        q = (_rms(dq, EPS, w["dq.norm"]) @ w["uq.weight"].T).unflatten(1, (H, 192))
        past = pages["latent"][:, 0]
        c = torch.cat([past[:, :R], _rms(c, EPS, w["dkv.norm"])])
        kr = torch.cat([past[:, R:], _rotate(kr[:, None], pos, 64)[:, 0]])
        k = torch.cat([(c @ w["uk.weight"].T).unflatten(1, (H, 128)), kr[:, None].expand(-1, H, -1)], 2)
        v = (c @ w["uv.weight"].T).unflatten(1, (H, 128))
        q = torch.cat([q[..., :128], _rotate(q[..., 128:], pos, 64)], 2)
        dist = pos[:, None] - torch.arange(old + len(pos), device=DEV)[None]
        o = _attend(q, k, v, 192 ** -0.5, (dist >= 0) & (dist < 1024), w["sink"])
        out[s] = (o.flatten(1) * torch.sigmoid(g)) @ w["o.weight"].T
    return {"out": out, "pages latent": None}


def _simivik64(case, seed, w, x):
    H, silu, S_out, out = case["width"] // 128, torch.nn.functional.silu, [], torch.empty_like(x)
    lam = torch.tensor(_decays(H), dtype=torch.float64, device=DEV)[:, None].expand(H, 128)
    for i, old, s, pos, _, states in _requests(case, seed):
        q, k, v, g = (x[s] @ w["qkvg.weight"].T).chunk(4, 1)
        heads = lambda t: silu(t).unflatten(1, (H, 128))  # noqa: E731
        o, S = _states(states["S"], heads(q), heads(k), heads(v), [lam] * len(pos))
        out[s] = (_rms(o.flatten(1), EPS, w["norm"]) * torch.sigmoid(g)) @ w["o.weight"].T
        S_out.append(S)
    return {"out": out, "state S": torch.stack(S_out)}


def _kibotar64(case, seed, w, x):
    H, S_out, out = case["width"] // 128, [], torch.empty_like(x)
    for i, old, s, pos, _, states in _requests(case, seed):
        n = H * 128
        q, k, v, g, a = (x[s] @ w["in.weight"].T).split([n, n, n, n, 64], 1)
        alpha = torch.sigmoid(a @ w["a2.weight"].T + w["a2.bias"]) ** 0.125
        heads = lambda t: t.unflatten(1, (H, 128))  # noqa: E731
        o, S = _states(states["S"], heads(q) * 128 ** -0.5, heads(k), heads(v), heads(alpha))
        out[s] = (_rms(o, EPS, w["norm"]).flatten(1) * torch.nn.functional.silu(g)) @ w["o.weight"].T
        S_out.append(S)
    return {"out": out, "state S": torch.stack(S_out)}


def _vudezen64(w, x):
    W = x.shape[1]

    def ffn(h, gate_up, down):
        g, u = (h @ gate_up.T).chunk(2, 1)
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ down.T

    score = (x @ w["router.weight"][:20].T).softmax(1)
    choice = score + w["correction"]
    best = choice.unflatten(1, (4, 5)).amax(2)
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(2, 1).indices, True).repeat_interleave(5, 1)
    ids = choice.masked_fill(~kept, -math.inf).topk(2, 1).indices
    wts = score.gather(1, ids)
    wts = wts / (wts.sum(1, keepdim=True) + 1e-20) * 1.5
    out = ffn(x, w["shared.gate_up.weight"], w["shared.down.weight"])
    gate_up, down = w["gate_up.weight"].view(16, 2 * W, W), w["down.weight"].view(16, W, W)
    for e in range(20):
        rows, j = (ids == e).nonzero(as_tuple=True)
        if len(rows):
            f = ffn(x[rows], gate_up[e], down[e]) if e < 16 else x[rows]
            out.index_add_(0, rows, f * wts[rows, j][:, None])
    return {"out": out}


def _vunepel64(case, seed, w, x):
    H, out = case["width"] // 128, torch.empty_like(x)
    G = H // 4
    l1, k1, l2, k2 = w["lambdas"]
    lam = torch.exp(l1 @ k1) - torch.exp(l2 @ k2) + 0.4
    for i, old, s, pos, pages, _ in _requests(case, seed):
        q, k, v = (x[s] @ w["in.weight"].T).split([2 * H * 64, 2 * G * 64, G * 128], 1)
        q = _rotate(_rms(q.unflatten(1, (2 * H, 64)), EPS, w["q_norm"]), pos, 64)
        k = _rotate(_rms(k.unflatten(1, (2 * G, 64)), EPS, w["k_norm"]), pos, 64)
        k, v = torch.cat([pages["k"], k]), torch.cat([pages["v"], v.unflatten(1, (G, 128))])
        key = torch.arange(old + len(pos), device=DEV)[None]
        seen = (key <= pos[:, None]) & (key // 1024 == pos[:, None] // 1024)
        one, two = (_attend(q[:, m::2], k[:, m::2], v, 64 ** -0.5, seen) for m in (0, 1))
        out[s] = (_rms(one - lam * two, EPS) * 0.6).flatten(1) @ w["o.weight"].T
    return {"out": out, "pages k": None, "pages v": None}


def _serve64(case, seed):
    w = _serve_weights(seed)
    by_step = [[] for _ in range(case["steps"] + 1)]
    empty = torch.zeros((0, KV, HEAD), dtype=torch.float64, device=DEV)
    rows = []
    for p in _prompts(case, seed):
        rows.append(w["embedding.weight"][torch.tensor(p, device=DEV)].double())
    for i in range(LAYERS):
        lw = {n[len("layers.%d." % i):]: t.double() for n, t in w.items() if n.startswith("layers.%d." % i)}
        att = {n[6:]: t for n, t in lw.items() if n.startswith("mixer.")}
        ffn = {n[4:]: t for n, t in lw.items() if n.startswith("ffn.")}
        for j, r in enumerate(rows):
            pos = torch.arange(len(r), device=DEV)
            r = r + _attention64(att, _rms(r, QWEN_EPS, lw["mixer_norm.weight"]), 0, pos, empty, empty)
            rows[j] = r + _mlp64(ffn, _rms(r, QWEN_EPS, lw["ffn_norm.weight"]))
    head, norm = w["lm_head.weight"].double(), w["final_norm.weight"].double()
    for r in rows:
        logits = _rms(r[-case["steps"] - 1:], QWEN_EPS, norm) @ head.T
        for k in range(case["steps"] + 1):
            by_step[k].append(logits[k])
    return [torch.stack(x) for x in by_step]


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return _serve64(case, seed)
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    x = _rand(seed, "x", (case["tokens"], _width(case)), dtype=_dtype(case)).double()
    if kind == "mlp":
        return {"out": _mlp64(w, x)}
    if kind == "attention":
        out = [_attention64(w, x[s], old, pos, pages["k"], pages["v"]) for _, old, s, pos, pages, _ in _requests(case, seed)]
        return {"out": torch.cat(out), "pages k": None, "pages v": None}
    if kind == "vudezen":
        return _vudezen64(w, x)
    return {"nurinex": _nurinex64, "mugulorn": _mugulorn64, "simivik": _simivik64, "kibotar": _kibotar64,
            "vunepel": _vunepel64}[kind](case, seed, w, x)


# ------------------------------------------------------------------------------------------------------ work, tolerances


def work(case):
    """One read of the weights and of the rows and cached keys that are looked at, one write of the results; the products'
    operations and the attention's over the pairs that are seen (the recurrences': two per state element and row)."""
    kind, T, ports = case["kind"], case["tokens"], _portions(case)
    size = 4 if case.get("dtype") == "float32" else 2

    def pairs(window=1 << 30):
        return sum(sum(min(p + 1, window) for p in range(o, o + n)) for o, n in ports)

    keys = sum(o + n for o, n in ports)
    if kind == "mlp":
        h, f = case["hidden"], case["ff"]
        return {"bytes": 2 * (3 * h * f + 2 * T * h), "flops": 6 * T * h * f}
    att = HIDDEN * HEAD * (2 * HEADS + 2 * KV)
    if kind == "attention":
        return {"bytes": size * (att + 2 * T * HIDDEN + 2 * (keys + T) * KV * HEAD), "flops": 2 * T * att + 4 * HEADS * HEAD * pairs()}
    if kind == "serve":
        layer, steps = att + 3 * HIDDEN * FF, case["steps"]
        rows = T + case["requests"] * steps
        n = sum((a + steps) * (a + steps + 1) // 2 for _, a in ports)
        cached = sum(a * (steps + 1) + steps * (steps + 1) // 2 for _, a in ports)
        return {"bytes": 2 * (steps + 1) * (LAYERS * layer + VOCAB * HIDDEN) + 4 * KV * HEAD * LAYERS * cached + 4 * VOCAB * case["requests"] * (steps + 1),
                "flops": LAYERS * (2 * rows * layer + 4 * HEADS * HEAD * n) + 2 * VOCAB * HIDDEN * case["requests"] * (steps + 1)}
    W = case["width"]
    H = W // 128
    G = H // 4
    io = 4 * T * W
    n_req = len(ports)
    if kind == "nurinex":
        mats = W * 128 * (2 * H + 2 * G) + 5 * W * W + 128 * W
        return {"bytes": 2 * mats + io + 4 * keys * G * 128 + 8 * n_req * W * 64,
                "flops": 2 * T * mats + 4 * H * 128 * pairs() + 2 * H * H * pairs() + 4 * T * W * 64}
    if kind == "mugulorn":
        mats = W * (W // 2 + W // 4 + 64 + 2 * H * 128) + H * 192 * (W // 2) + 2 * H * 128 * (W // 4)
        seen = sum(min(o, 1023) + n for o, n in ports)
        return {"bytes": 2 * mats + io + 2 * seen * (W // 4 + 64), "flops": 2 * T * mats + 2 * H * 320 * pairs(1024)}
    if kind in ("simivik", "kibotar"):
        mats = 5 * W * W + (128 * W if kind == "kibotar" else 0)
        return {"bytes": 2 * mats + io + 8 * n_req * W * 128, "flops": 2 * T * mats + 4 * T * W * 128}
    if kind == "vudezen":
        hit = 16 * (1 - (1 - 1 / 16) ** (1.6 * T))             # experts that are chosen by some row, as expected
        return {"bytes": int(2 * 3 * W * W * (hit + 1) + io), "flops": int(2 * T * 3 * W * W * 2.6)}
    mats = W * (2 * H * 64 + 2 * G * 64 + G * 128 + H * 128)
    n = sum(sum(p % 1024 + 1 for p in range(o, o + a)) for o, a in ports)
    return {"bytes": 2 * mats + io + 2 * keys * G * 256, "flops": 2 * T * mats + 2 * H * (128 + 256) * n}


def tolerance(case):
    """About four times the distance from the same in 64 bits: what bfloat16 rows between a layer's kernels (and, in the
    whole model, between its layers) give, or the order of sums over 4096 numbers in 32 bits."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    return {"rel": {"mlp": 1e-2, "simivik": 1e-2, "serve": 1.25e-2, "vudezen": 1.25e-2, "attention": 1.6e-2}.get(case["kind"], 2e-2)}
