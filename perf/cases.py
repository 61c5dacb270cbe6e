"""The work whose speed this repository is measured by: whole steps of the engine at the headline layer sizes, and
single layers (a decoder block, recurrent mixers, differential attention, routed experts), each through the entry point
that a program built on the package calls.

Sizes are those of ``bench.py`` (Qwen2.5-1.5B and 7B layer sizes; the layer sizes it gives the other designs).  Weights
are random with the scale of trained ones, contexts are random rows in the cache; the gates of the recurrent mixers
have the ranges that their designs start training from (decays from a few tokens to thousands).
"""
import math
import random
import zlib

import torch

from coheryn_ai_studio_b200.cache import CacheManager
from coheryn_ai_studio_b200.config import Qwen2Config
from coheryn_ai_studio_b200.config.qwen2 import qwen2_model_spec
from coheryn_ai_studio_b200.config.spec import PartSpec
from coheryn_ai_studio_b200.engine import StepEntry, StepRunner
from coheryn_ai_studio_b200.parts.base import FEED_FORWARDS, MIXERS, POSITIONS, LayerCache, Runtime, StepContext, build_part
from coheryn_ai_studio_b200.parts.model import DecoderModel

PAGE = 16
DEVICE = "cuda:0"
QWEN = {  # layer sizes of bench.py's headline and of its serving workload
    "1.5b": dict(width=1536, ff=8960, heads=12, kv_heads=2, head_dim=128, vocab=151936, layers=28, eps=1e-6, theta=1e6),
    "7b": dict(width=3584, ff=18944, heads=28, kv_heads=4, head_dim=128, vocab=152064, layers=28, eps=1e-6, theta=1e6),
}


def listed():
    return [
        # One user, a short conversation: a decode step of the whole model for one request (latency).
        dict(name="decode_1", kind="decode", model="1.5b", layers=28, batch=1, context=700),
        # The headline of bench.py: a decode step of the whole model for eight requests at context 4,096.
        dict(name="decode_8", kind="decode", model="1.5b", layers=28, batch=8, context=4096),
        # The other headline: a prompt of 2,048 tokens through the whole model to the logits of its last token.
        dict(name="prompt_2048", kind="prompt", model="1.5b", layers=28, tokens=2048),
        # A serving batch decoding: one block for 64 requests with contexts of every length up to 4,096.
        dict(name="block_decode_64", kind="block", model="1.5b", dtype="bf16", prompts="", decodes=64, context=4096),
        # A step of continuous batching at the 7B layer sizes: portions of prompts (one of them continued) beside decoding
        # requests; odd lengths, as users bring them.
        dict(name="block_mixed_7b", kind="block", model="7b", dtype="bf16", prompts="1337+0 403+1024 96+0", decodes=37, context=2048),
        # The 32-bit path, which the reference's own numerics are compared in: two short prompts.
        dict(name="block_float32", kind="block", model="1.5b", dtype="f32", prompts="217+0 96+31", decodes=0, context=0),
        # Kapudra's gated delta rule (a decay per head and key channel), a long prompt.
        dict(name="delta_2048", kind="delta", width=1536, heads=12, kv_heads=12, dim=128, vdim=128, per="channel", lengths="2048"),
        # Tutunex's (a decay per head): prompts of several users in one step, of odd lengths.
        dict(name="delta_ragged", kind="delta", width=1536, heads=12, kv_heads=12, dim=128, vdim=128, per="head", lengths="1021 407 130 2"),
        # Its decoding: a token for each of 32 requests, bound by the state that it reads and writes.
        dict(name="delta_decode_32", kind="delta", width=1536, heads=12, kv_heads=12, dim=128, vdim=128, per="channel",
             lengths=" ".join(["1"] * 32)),
        # Kapudra's matrix memory, a long prompt.
        dict(name="memory_2048", kind="memory", width=1536, heads=8, dim=128, vdim=256, lengths="2048"),
        # Tutunex's differential attention over chunks, a long prompt.
        dict(name="maps_2048", kind="maps", width=1536, heads=12, kv_heads=2, dim=64, vdim=128, chunk=1024, lengths="2048"),
        # Guvusun's routed experts, a long prompt.
        dict(name="experts_2048", kind="experts", width=2048, ff=1024, experts=30, identity=2, top=4, groups=4, keep=2, tokens=2048),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "block", "block", "block", "delta", "delta", "delta", "memory", "memory", "maps", "maps", "experts"])
    if kind == "decode":
        batch = _log_int(rng, 1, 48)
        return dict(kind=kind, model="1.5b", layers=rng.choice([4, 12, 28]), batch=batch, context=_log_int(rng, 64, min(4096, 32768 // batch)))
    if kind == "prompt":
        return dict(kind=kind, model="1.5b", layers=rng.choice([4, 12, 28]), tokens=_log_int(rng, 17, 2048))
    if kind == "block":
        dtype = rng.choice(["bf16", "bf16", "bf16", "f32"])
        model = rng.choice(["1.5b", "7b"]) if dtype == "bf16" else "1.5b"
        most = 1800 if dtype == "bf16" else 320
        prompts = []
        for _ in range(rng.randrange(0, 4)):
            prompts.append("%d+%d" % (_log_int(rng, 2, most // 3), rng.choice([0, 0, rng.randrange(1, 1500)])))
        decodes = _log_int(rng, 1, 64) if dtype == "bf16" and (not prompts or rng.random() < 0.6) else 0
        if not prompts and not decodes:
            prompts = ["%d+0" % _log_int(rng, 2, most)]
        return dict(kind=kind, model=model, dtype=dtype, prompts=" ".join(prompts), decodes=decodes, context=_log_int(rng, 64, 4096) if decodes else 0)
    if kind in ("delta", "memory", "maps"):
        if kind != "maps" and rng.random() < 0.25:
            lengths = [1] * _log_int(rng, 1, 32)
        else:
            lengths = [_log_int(rng, 2, 2048 // n) for n in [rng.randrange(1, 6)] for _ in range(n)]
        lengths = " ".join(map(str, lengths))
        if kind == "memory":
            return dict(kind=kind, width=rng.choice([1536, 2560]), heads=8, dim=rng.choice([64, 128]), vdim=rng.choice([128, 256]), lengths=lengths)
        if kind == "maps":
            heads, kv = rng.choice([(12, 2), (20, 4)])
            return dict(kind=kind, width=128 * heads, heads=heads, kv_heads=kv, dim=64, vdim=128, chunk=rng.choice([0, 512, 1024]), lengths=lengths)
        heads, kv = rng.choice([(12, 12), (16, 16), (12, 4)])
        return dict(kind=kind, width=128 * heads, heads=heads, kv_heads=kv, dim=rng.choice([64, 128]), vdim=rng.choice([64, 128]),
                    per=rng.choice(["channel", "head"]), lengths=lengths)
    return dict(kind=kind, width=2048, ff=1024, experts=30, identity=2, top=4, groups=4, keep=2, tokens=_log_int(rng, 1, 2048))


# ------------------------------------------------------------------------------------------------ inputs from the seed
def _rand(seed, tag, shape, scale=1.0, mean=0.0, dtype=torch.bfloat16):
    """Normal values of one tensor: the same for the same seed and tag."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed((int(seed) << 32) ^ zlib.crc32(tag.encode()))
    x = torch.empty(tuple(shape), dtype=torch.float32 if math.prod(shape) < (1 << 22) else dtype, device=DEVICE)
    return x.normal_(mean, scale, generator=g).to(dtype)


def _uniform(seed, tag, shape, lo, hi):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((int(seed) << 32) ^ zlib.crc32(tag.encode()))
    return torch.empty(tuple(shape), device=DEVICE).uniform_(lo, hi, generator=g)


def _ids(seed, tag, n, vocab):
    r = random.Random("%d %s" % (seed, tag))
    return [r.randrange(vocab) for _ in range(n)]


def _i32(values):
    return torch.tensor(values, dtype=torch.int32).to(DEVICE)


def _qwen_weight(seed, name, shape, layers, dtype=torch.bfloat16):
    """Matrices scaled by their inputs, those that add to the stream also by the depth; norms about one, biases small."""
    if name.endswith("norm.weight"):
        return _rand(seed, name, shape, 0.1, 1.0, dtype)
    if name.endswith("bias"):
        return _rand(seed, name, shape, 0.1, 0.0, dtype)
    if "embed_tokens" in name:
        return _rand(seed, name, shape, 0.05, 0.0, dtype)
    depth = 1.0 / math.sqrt(2 * layers) if "o_proj" in name or "down_proj" in name else 1.0
    return _rand(seed, name, shape, depth * shape[1] ** -0.5, 0.0, dtype)


def _qwen_config(z, layers, vocab):
    return Qwen2Config(vocab_size=vocab, hidden_size=z["width"], intermediate_size=z["ff"], num_hidden_layers=layers,
                       num_attention_heads=z["heads"], num_key_value_heads=z["kv_heads"], head_dim=z["head_dim"],
                       max_position_embeddings=32768, rms_norm_eps=z["eps"], rope_theta=z["theta"], tie_word_embeddings=True)


def _qwen_model(case, seed, layers, vocab, dtype=torch.bfloat16):
    z = QWEN[case["model"]]
    model = DecoderModel(qwen2_model_spec(_qwen_config(z, layers, vocab)), Runtime(dtype, torch.device(DEVICE)))
    model.bind({n: _qwen_weight(seed, n, s.shape, layers, dtype) for n, s in model.tensor_specs().items()})
    return model


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


# ------------------------------------------------------------------------------------------------ whole steps
GROWTH = 512      # a decoding request starts again from its first length after so many tokens


def _decode_lengths(case):
    r = random.Random("lengths %d %d" % (case["batch"], case["context"]))
    return [case["context"] - r.randrange(0, max(1, case["context"] // 4)) for _ in range(case["batch"])]


def _context_rows(case, seed, layer, request, n):
    z = QWEN[case["model"]]
    return _rand(seed, "context %d %d" % (layer, request), (2, n, z["kv_heads"], z["head_dim"]))


def _admit(s):
    for rid, n in zip(s["ids"], s["lengths"]):
        s["cache"].admit(rid)
        s["cache"].reserve(rid, [0] * n)
        s["cache"].commit(rid)
    s["grown"] = 0


def _prepare_decode(case, seed):
    z = QWEN[case["model"]]
    model = _qwen_model(case, seed, case["layers"], z["vocab"])
    lengths, batch = _decode_lengths(case), case["batch"]
    most = case["context"] + GROWTH + PAGE
    cache = CacheManager(model.cache_requirements(), [e.cache_from for e in model.spec.schedule], torch.bfloat16, torch.device(DEVICE),
                         page_size=PAGE, num_pages=batch * -(-most // PAGE), max_requests=batch, prefix_reuse=False)
    s = dict(cache=cache, runner=StepRunner(model, cache, use_graphs=True, graph_max_kv_len=most), lengths=lengths,
             ids=["r%d" % b for b in range(batch)])
    _admit(s)
    for layer, c in enumerate(cache.layer_caches()):
        for b, n in enumerate(lengths):
            rows = _context_rows(case, seed, layer, b, n)
            at = torch.arange(n, device=DEVICE)
            page = _i32(cache.block_table(s["ids"][b], c.group)).long()[at // PAGE]
            c.k[page, :, at % PAGE] = rows[0]
            c.v[page, :, at % PAGE] = rows[1]
    s["entries"] = [StepEntry(rid, [t], [0]) for rid, t in zip(s["ids"], _ids(seed, "tokens", batch, z["vocab"]))]
    return s


def _prepare_prompt(case, seed):
    z = QWEN[case["model"]]
    model = _qwen_model(case, seed, case["layers"], z["vocab"])
    cache = CacheManager(model.cache_requirements(), [e.cache_from for e in model.spec.schedule], torch.bfloat16, torch.device(DEVICE),
                         page_size=PAGE, num_pages=-(-case["tokens"] // PAGE) + 1, max_requests=1, prefix_reuse=False)
    return dict(cache=cache, runner=StepRunner(model, cache, use_graphs=True),
                entry=StepEntry("p", _ids(seed, "tokens", case["tokens"], z["vocab"]), [case["tokens"] - 1]))


# ------------------------------------------------------------------------------------------------ one step for single layers
def _requests(case):
    """(new tokens, tokens before them) of every request of the step."""
    if "lengths" in case:
        return [(int(n), 0) for n in case["lengths"].split()]
    got = [tuple(int(v) for v in p.split("+")) for p in case["prompts"].split()]
    r = random.Random("requests %d %d" % (case["decodes"], case["context"]))
    return got + [(1, r.randrange(case["context"] // 4, case["context"])) for _ in range(case["decodes"])]


def _pages(case):
    """Pages of every request, in an order as a pool in use hands them out."""
    need = [-(-(n + before) // PAGE) for n, before in _requests(case)]
    order = list(range(sum(need)))
    random.Random("pages %d" % sum(need)).shuffle(order)
    cut = [sum(need[:i]) for i in range(len(need) + 1)]
    return [order[a:b] for a, b in zip(cut, cut[1:])]


def _step(case, token_ids=None):
    req, pages = _requests(case), _pages(case)
    new, total = [n for n, _ in req], [n + b for n, b in req]
    T = sum(new)
    positions = [p for n, b in req for p in range(b, b + n)]
    owner = [i for i, n in enumerate(new) for _ in range(n)]
    cu = [sum(new[:i]) for i in range(len(new) + 1)]
    width = max(len(p) for p in pages)
    tables = _i32([p + [-1] * (width - len(p)) for p in pages])
    slots = _i32([pages[o][p // PAGE] * PAGE + p % PAGE for o, p in zip(owner, positions)])
    return StepContext(num_tokens=T, num_requests=len(req), token_ids=_i32(token_ids or [0] * T), positions=_i32(positions),
                       token_req=_i32(owner), cu_q=_i32(cu), kv_lens=_i32(total), block_tables=[tables], slots=[slots],
                       state_slots=_i32(list(range(len(req)))), q_lens=new, kv_lens_host=total, max_q_len=max(new), max_kv_len=max(total))


def _pool(case, seed, which, kv_heads, dim, dtype):
    pages = sum(len(p) for p in _pages(case))
    return _rand(seed, which + " pool", (pages + 1, kv_heads, PAGE, dim), dtype=dtype)


def _prepare_block(case, seed):
    z, dtype = QWEN[case["model"]], _dtype(case)
    model = _qwen_model(case, seed, 1, 64, dtype)
    step = _step(case)
    return dict(model=model, step=step, x=_rand(seed, "stream", (step.num_tokens, z["width"]), dtype=torch.float32),
                cache=LayerCache("paged", 0, PAGE, _pool(case, seed, "k", z["kv_heads"], z["head_dim"], dtype),
                                 _pool(case, seed, "v", z["kv_heads"], z["head_dim"], dtype)))


def _mixer_params(case):
    if case["kind"] == "delta":
        p = dict(hidden_size=case["width"], num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=case["dim"],
                 v_head_dim=case["vdim"], conv_taps=4, eps=1e-6)
        if case["per"] == "head":
            return "gated_delta_rule", dict(p, decay="head", low_rank=False, gate_activation="silu")
        return "gated_delta_rule", dict(p, decay_rank=64, gate_rank=64)
    if case["kind"] == "memory":
        return "matrix_memory", dict(hidden_size=case["width"], num_heads=case["heads"], head_dim=case["dim"], v_head_dim=case["vdim"],
                                     gate_cap=15.0, eps=1e-6)
    return "attention_maps", dict(hidden_size=case["width"], num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=case["dim"],
                                  v_head_dim=case["vdim"], scale=case["dim"] ** -0.5, maps=2, lambda_init=0.5,
                                  chunk=case["chunk"] or None, eps=1e-6, float32_output=True)


def _part_weight(seed, name, shape):
    if name in ("lq1", "lk1", "lq2", "lk2"):
        return _rand(seed, name, shape, 0.1)
    if name.endswith("norm"):
        return _rand(seed, name, shape, 0.1, 1.0)
    if name.endswith("conv"):
        return _rand(seed, name, shape, shape[1] ** -0.5)
    if name == "A_log":      # rates from 1 to 16
        return _uniform(seed, name, shape, 0.0, math.log(16.0)).to(torch.bfloat16)
    if name == "dt_bias":    # step sizes from a thousandth to a tenth
        dt = torch.exp(_uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)))
        return torch.log(torch.expm1(dt)).to(torch.bfloat16)
    if name == "f.b":        # forget gates from 0.95 to 0.998
        return _uniform(seed, name, shape, 3.0, 6.0).to(torch.bfloat16)
    if name == "i.b":
        return _rand(seed, name, shape, 1.0, -2.0)
    if name == "correction":
        return _rand(seed, name, shape, 0.01)
    scale = shape[-1] ** -0.5
    return _rand(seed, name, shape, 0.3 * scale if name in ("a", "a2") else scale)


def _mixer(case, seed):
    kind, params = _mixer_params(case)
    runtime = Runtime(torch.bfloat16, torch.device(DEVICE))
    extra = {}
    if case["kind"] == "maps":
        rot = PartSpec("rope_computed", dict(rotary_dim=case["dim"], theta=500000.0,
                                             scaling=dict(factor=8.0, original=8192, fast=32.0, slow=1.0)))
        extra["position"] = build_part(POSITIONS, "position", rot, runtime)
    part = build_part(MIXERS, "mixer", PartSpec(kind, params), runtime, **extra)
    w = {n: _part_weight(seed, n, s.shape) for n, s in part.tensor_specs().items()}
    part.bind(w)
    return part, w


def _prepare_mixer(case, seed):
    part, w = _mixer(case, seed)
    step = _step(case)
    s = dict(part=part, step=step, x=_rand(seed, "input", (step.num_tokens, case["width"])))
    if case["kind"] == "maps":
        s["cache"] = LayerCache("paged", 0, PAGE, _pool(case, seed, "k", case["kv_heads"], 2 * case["dim"], torch.bfloat16),
                                _pool(case, seed, "v", case["kv_heads"], case["vdim"], torch.bfloat16))
    else:
        need = part.cache_requirement()
        s["cache"] = LayerCache("state", state=torch.zeros((step.num_requests,) + tuple(need.shape), dtype=need.dtype, device=DEVICE))
        if step.max_q_len == 1:
            s["cache"].state.copy_(_start_state(case, seed, s["cache"].state.shape))
    return s


def _start_state(case, seed, shape):
    """The state of decoding requests: as a prompt leaves it, small numbers (and a normaliser and maximum of a memory)."""
    st = _rand(seed, "state", shape, 0.1, dtype=torch.float32)
    if case["kind"] == "memory":
        H, dk, dv = case["heads"], case["dim"], case["vdim"]
        st[:, H * dk * dv + H * dk:] = 0.0
    return st


def _prepare_experts(case, seed):
    part = build_part(FEED_FORWARDS, "feed_forward", PartSpec("routed_experts", dict(
        hidden_size=case["width"], expert_size=case["ff"], experts=case["experts"], top=case["top"], identity=case["identity"],
        groups=case["groups"], keep=case["keep"], scale=2.5, correction=True, activation="silu")), Runtime(torch.bfloat16, torch.device(DEVICE)))
    part.bind({n: _part_weight(seed, n, s.shape) for n, s in part.tensor_specs().items()})
    return dict(part=part, step=_step(dict(lengths=str(case["tokens"]))), x=_rand(seed, "input", (case["tokens"], case["width"])))


def prepare(case, seed):
    s = {"decode": _prepare_decode, "prompt": _prepare_prompt, "block": _prepare_block, "delta": _prepare_mixer,
         "memory": _prepare_mixer, "maps": _prepare_mixer, "experts": _prepare_experts}[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(s):
    kind = s["kind"]
    if kind == "decode":
        if s["grown"] == GROWTH:
            for rid in s["ids"]:
                s["cache"].free(rid)
            _admit(s)
        s["grown"] += 1
        return {"logits": s["runner"].step(s["entries"])}
    if kind == "prompt":
        s["cache"].admit("p")
        logits = s["runner"].step([s["entry"]])
        s["cache"].free("p")
        return {"logits": logits}
    step = s["step"]
    step.native, step.shared = None, {}
    if kind == "block":
        stream = s["x"].clone()          # the embedding's output, which a block adds to in place
        stream, delta = s["model"].layers[0].forward(stream, None, step, s["cache"])
        normed = s["model"].final_norm.forward(stream, delta)
        return {"stream": stream, "normed": normed, "k": s["cache"].k, "v": s["cache"].v}
    if kind == "experts":
        return {"y": s["part"].forward(s["x"], step)}
    if kind == "maps":
        return {"y": s["part"].forward(s["x"], step, s["cache"]), "k": s["cache"].k, "v": s["cache"].v}
    if step.max_q_len > 1:               # a prompt starts from a zeroed state, as a request that has just been admitted
        s["cache"].state.zero_()
    y = s["part"].forward(s["x"], step, s["cache"])
    return {"y": y, "state": s["cache"].state}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_params(z):
    qkv = (z["heads"] + 2 * z["kv_heads"]) * z["head_dim"]
    return z["width"] * qkv + z["heads"] * z["head_dim"] * z["width"] + 3 * z["width"] * z["ff"]


def _attended(requests):
    """Keys that the new tokens see, added up, and cached rows that have to be read."""
    return sum(n * b + n * (n + 1) // 2 for n, b in requests), sum(n + b for n, b in requests)


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt", "block"):
        z = QWEN[case["model"]]
        if kind == "decode":
            req, layers = [(1, n) for n in _decode_lengths(case)], case["layers"]
        elif kind == "prompt":
            req, layers = [(case["tokens"], 0)], case["layers"]
        else:
            req, layers = _requests(case), 1
        T, item = sum(n for n, _ in req), 4 if case.get("dtype") == "f32" else 2
        seen, held = _attended(req)
        flops = layers * (2.0 * T * _layer_params(z) + 4.0 * z["heads"] * z["head_dim"] * seen)
        size = layers * (_layer_params(z) * item + 2.0 * z["kv_heads"] * z["head_dim"] * item * held)
        if kind == "block":
            return {"bytes": size + T * z["width"] * (8 + item), "flops": flops}
        rows = len(req)
        return {"bytes": size + 2.0 * z["vocab"] * z["width"] + 4.0 * rows * z["vocab"] + 2.0 * T * z["width"],
                "flops": flops + 2.0 * rows * z["vocab"] * z["width"]}
    W = case["width"]
    if kind == "experts":
        T = case["tokens"]
        pairs = T * case["top"] * case["experts"] / (case["experts"] + case["identity"])
        used = case["experts"] * (1.0 - (1.0 - case["top"] / (case["experts"] + case["identity"])) ** T)
        return {"bytes": 2.0 * 3 * W * case["ff"] * used + T * W * 6.0, "flops": 6.0 * pairs * W * case["ff"] + 2.0 * T * W * 32}
    T, B = sum(n for n, _ in _requests(case)), len(_requests(case))
    H, dk, dv = case["heads"], case["dim"], case["vdim"]
    if kind == "maps":
        G, chunk = case["kv_heads"], case["chunk"] or 1 << 30
        seen = sum(p % chunk + 1 for n, _ in _requests(case) for p in range(n))
        params = W * (2 * H * dk + 2 * G * dk + G * dv) + H * dv * W
        return {"bytes": 2.0 * params + T * W * 6.0 + 2.0 * T * G * (2 * dk + dv), "flops": 2.0 * T * params + 2.0 * H * seen * (2 * dk + 2 * dv)}
    if kind == "memory":
        params = W * (2 * H * dk + 3 * H * dv + 2 * H)
        return {"bytes": 2.0 * params + T * W * 6.0 + 8.0 * B * H * (dk * dv + dk + 1), "flops": 2.0 * T * params + 6.0 * T * H * dk * dv}
    G = case["kv_heads"]
    params = W * (2 * G * dk + 2 * H * dv + H)
    params += 64 * (2 * W + H * dk + H * dv) if case["per"] == "channel" else W * (H + H * dv)
    return {"bytes": 2.0 * params + T * W * 6.0 + 8.0 * B * (H * dk * dv + 3 * (2 * G * dk + H * dv)), "flops": 2.0 * T * params + 8.0 * T * H * dk * dv}


def tolerance(case):
    """bfloat16 activations between the kernels give each layer a few thousandths; a whole model adds up its layers."""
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        return {"rel": 0.03, "max": 0.3}
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.01, "max": 0.2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, angle, amp=1.0):
    """x [T, heads, d]: channel i turns with channel i + d/2 by angle [T, d/2]."""
    h = angle.shape[1]
    a, b, c, s = x[..., :h], x[..., h:2 * h], (angle.cos() * amp)[:, None], (angle.sin() * amp)[:, None]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, seen, scale):
    """q [T, H, d], k [S, G, d], v [S, G, dv], seen [T, S]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    s = torch.einsum("tghd,sgd->ghts", q.view(T, G, H // G, -1), k) * scale
    p = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
    return torch.einsum("ghts,sgd->tghd", p, v).reshape(T, H, -1)


def _qwen_layer(z, w, x, positions, spans, context, dtype):
    """One block on x [T, width]; spans: (first row, rows) of every request; context(r): its earlier k and v or None."""
    T, hd, H, G = x.shape[0], z["head_dim"], z["heads"], z["kv_heads"]
    f = z["theta"] ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=x.device) / hd)
    angle = positions.double()[:, None] * f[None]
    h = _rms(x, z["eps"]) * w("input_layernorm.weight")
    q, k, v = (h @ w("self_attn.%s_proj.weight" % n).T + w("self_attn.%s_proj.bias" % n) for n in "qkv")
    q, k, v = _turn(q.view(T, H, hd), angle), _turn(k.view(T, G, hd), angle), v.view(T, G, hd)
    out = torch.empty((T, H, hd), dtype=torch.float64, device=x.device)
    for r, (at, n) in enumerate(spans):
        kk, vv, old = k[at:at + n], v[at:at + n], context(r)
        if old is not None:
            kk, vv = torch.cat([old[0].double(), kk]), torch.cat([old[1].double(), vv])
        S = kk.shape[0]
        seen = torch.arange(S, device=x.device)[None] <= torch.arange(S - n, S, device=x.device)[:, None]
        out[at:at + n] = _attend(q[at:at + n], kk, vv, seen, hd ** -0.5)
    x = x + out.view(T, -1) @ w("self_attn.o_proj.weight").T
    h = _rms(x, z["eps"]) * w("post_attention_layernorm.weight")
    g = h @ w("mlp.gate_proj.weight").T
    return x, (g * torch.sigmoid(g) * (h @ w("mlp.up_proj.weight").T)) @ w("mlp.down_proj.weight").T


def _qwen_shapes(z):
    W, F, qd, kd = z["width"], z["ff"], z["heads"] * z["head_dim"], z["kv_heads"] * z["head_dim"]
    return {"input_layernorm.weight": (W,), "post_attention_layernorm.weight": (W,), "self_attn.q_proj.weight": (qd, W),
            "self_attn.q_proj.bias": (qd,), "self_attn.k_proj.weight": (kd, W), "self_attn.k_proj.bias": (kd,),
            "self_attn.v_proj.weight": (kd, W), "self_attn.v_proj.bias": (kd,), "self_attn.o_proj.weight": (W, qd),
            "mlp.gate_proj.weight": (F, W), "mlp.up_proj.weight": (F, W), "mlp.down_proj.weight": (W, F)}


def _exact_model(case, seed):
    z, layers = QWEN[case["model"]], case["layers"]
    shapes = _qwen_shapes(z)
    table = _qwen_weight(seed, "model.embed_tokens.weight", (z["vocab"], z["width"]), layers)
    if case["kind"] == "decode":
        lengths = _decode_lengths(case)
        ids, spans = _ids(seed, "tokens", case["batch"], z["vocab"]), [(b, 1) for b in range(case["batch"])]
        positions = torch.tensor(lengths, device=DEVICE)
    else:
        ids, spans = _ids(seed, "tokens", case["tokens"], z["vocab"]), [(0, case["tokens"])]
        positions = torch.arange(case["tokens"], device=DEVICE)
    x = table[torch.tensor(ids, device=DEVICE)].double()
    for i in range(layers):
        def w(n):
            return _qwen_weight(seed, "model.layers.%d.%s" % (i, n), shapes[n], layers).double()

        def context(r):
            return _context_rows(case, seed, i, r, lengths[r]) if case["kind"] == "decode" else None
        x, d = _qwen_layer(z, w, x, positions, spans, context, torch.float64)
        x = x + d
    x = x[-1:] if case["kind"] == "prompt" else x
    h = _rms(x, z["eps"]) * _qwen_weight(seed, "model.norm.weight", (z["width"],), layers).double()
    return {"logits": torch.cat([h @ t.double().T for t in table.split(16384)], 1)}


def _exact_block(case, seed):
    z, dtype, req, pages = QWEN[case["model"]], _dtype(case), _requests(case), _pages(case)
    shapes = _qwen_shapes(z)
    kp, vp = (_pool(case, seed, n, z["kv_heads"], z["head_dim"], dtype) for n in "kv")

    def context(r):
        n = req[r][1]
        if not n:
            return None
        at = torch.arange(n, device=DEVICE)
        page = torch.tensor(pages[r], device=DEVICE)[at // PAGE]
        return kp[page, :, at % PAGE], vp[page, :, at % PAGE]
    spans, at = [], 0
    for n, _ in req:
        spans.append((at, n))
        at += n
    positions = torch.tensor([p for n, b in req for p in range(b, b + n)], device=DEVICE)
    x = _rand(seed, "stream", (at, z["width"]), dtype=torch.float32).double()
    x, d = _qwen_layer(z, lambda n: _qwen_weight(seed, "model.layers.0." + n, shapes[n], 1, dtype).double(), x, positions, spans, context, torch.float64)
    x = x + d
    h = _rms(x, z["eps"]) * _qwen_weight(seed, "model.norm.weight", (z["width"],), 1, dtype).double()
    return {"stream": x, "normed": h, "k": None, "v": None}


def _exact_maps(case, seed):
    H, G, d, dv, W = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["width"]
    w = {n: _part_weight(seed, n, s).double() for n, s in (
        ("q", (2 * H * d, W)), ("k", (2 * G * d, W)), ("v", (G * dv, W)), ("o", (W, H * dv)),
        ("lq1", (d,)), ("lk1", (d,)), ("lq2", (d,)), ("lk2", (d,)))}
    x = _rand(seed, "input", (sum(n for n, _ in _requests(case)), W)).double()
    i = torch.arange(d // 2, dtype=torch.float64, device=DEVICE)
    f = 500000.0 ** (-2.0 * i / d)       # interpolated by parts (YaRN): factor 8, 8,192 positions, 32 and 1 turns
    where = [d * math.log(8192 / (2.0 * math.pi * t)) / (2.0 * math.log(500000.0)) for t in (32.0, 1.0)]
    lo, hi = max(math.floor(where[0]), 0), min(math.ceil(where[1]), d - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f, amp = f / 8.0 * ramp + f * (1.0 - ramp), 0.1 * math.log(8.0) + 1.0
    lam = math.exp(float(w["lq1"] @ w["lk1"])) - math.exp(float(w["lq2"] @ w["lk2"])) + 0.5
    out, at = [], 0
    for n, _ in _requests(case):
        h, pos = x[at:at + n], torch.arange(n, device=DEVICE)
        at += n
        angle = pos.double()[:, None] * f[None]
        q, k = _turn((h @ w["q"].T).view(n, 2 * H, d), angle, amp), _turn((h @ w["k"].T).view(n, 2 * G, d), angle, amp)
        v = (h @ w["v"].T).view(n, G, dv)
        chunk = case["chunk"] or 1 << 30
        seen = (pos[None] <= pos[:, None]) & (pos[None] // chunk == pos[:, None] // chunk)
        a = [_attend(q[:, m::2].contiguous(), k[:, m::2].contiguous(), v, seen, d ** -0.5) for m in (0, 1)]
        out.append((_rms(a[0] - lam * a[1], 1e-6) * 0.5).view(n, -1) @ w["o"].T)
    return {"y": torch.cat(out), "k": None, "v": None}


def _exact_recurrent(case, seed):
    H, dk, dv, W, req = case["heads"], case["dim"], case["vdim"], case["width"], _requests(case)
    x = _rand(seed, "input", (sum(n for n, _ in req), W)).double()
    started = max(n for n, _ in req) == 1
    delta = case["kind"] == "delta"
    G = case.get("kv_heads", H)
    C = 2 * G * dk + H * dv
    size = H * dk * dv + (3 * C if delta else H * dk + H)
    state = _start_state(case, seed, (len(req), size)).double() if started else torch.zeros((len(req), size), dtype=torch.float64, device=DEVICE)

    def w(n, *shape):
        return _part_weight(seed, n, shape).double()

    def silu(z):
        return z * torch.sigmoid(z)
    v = x @ w("v", H * dv, W).T
    if delta:
        raw = torch.cat([x @ w("q", G * dk, W).T, x @ w("k", G * dk, W).T, v], 1)
        taps = torch.cat([w("q.conv", G * dk, 4), w("k.conv", G * dk, 4), w("v.conv", H * dv, 4)])
        beta = torch.sigmoid(x @ w("b", H, W).T)
        if case["per"] == "channel":
            pre = x @ w("a1", 64, W).T @ w("a2", H * dk, 64).T + w("dt_bias", H * dk)
            gate = torch.sigmoid(x @ w("g1", 64, W).T @ w("g2", H * dv, 64).T)
        else:
            pre = x @ w("a", H, W).T + w("dt_bias", H)
            gate = silu(x @ w("g", H * dv, W).T)
        pre = pre.view(len(x), H, -1)
        decay = torch.exp(-torch.exp(w("A_log", H))[:, None] * torch.nn.functional.softplus(pre, threshold=60.0))
        norm = w("norm", dv)
    else:
        q, k = (x @ w("q", H * dk, W).T).view(-1, H, dk) * dk ** -0.5, (x @ w("k", H * dk, W).T).view(-1, H, dk)
        v = v.view(-1, H, dv)
        li = 15.0 * torch.tanh((x @ w("i", H, W).T + w("i.b", H)) / 15.0)
        lf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w("f", H, W).T + w("f.b", H)) / 15.0))
        gate, norm = torch.sigmoid(x @ w("g", H * dv, W).T), w("norm", H * dv).view(H, dv)
    out, at = torch.empty((len(x), H, dv), dtype=torch.float64, device=DEVICE), 0
    for r, (n, _) in enumerate(req):
        S = state[r, :H * dk * dv].view(H, dk, dv).clone()
        if delta:
            rows = torch.cat([state[r, H * dk * dv:].view(3, C), raw[at:at + n]])
            y = silu(sum(rows[j:j + n] * taps[:, j] for j in range(4)))
            qq, kk = (t.reshape(n, G, dk) for t in (y[:, :G * dk], y[:, G * dk:2 * G * dk]))
            qq, kk = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (qq, kk))
            qq, kk = (t.repeat_interleave(H // G, 1) for t in (qq * dk ** -0.5, kk))
            vv = y[:, 2 * G * dk:].reshape(n, H, dv)
            for t in range(n):
                S = decay[at + t][..., None] * S
                u = beta[at + t][:, None] * (vv[t] - torch.einsum("hkv,hk->hv", S, kk[t]))
                S = S + kk[t][..., None] * u[:, None]
                out[at + t] = torch.einsum("hkv,hk->hv", S, qq[t])
            state[r, H * dk * dv:] = rows[-3:].reshape(-1)
        else:
            nn, m = state[r, H * dk * dv:H * dk * (dv + 1)].view(H, dk).clone(), state[r, H * dk * (dv + 1):].clone()
            for t in range(n):
                mx = torch.maximum(lf[at + t] + m, li[at + t])
                a, b = torch.exp(lf[at + t] + m - mx), torch.exp(li[at + t] - mx)
                S = a[:, None, None] * S + b[:, None, None] * k[at + t][..., None] * v[at + t][:, None]
                nn, m = a[:, None] * nn + b[:, None] * k[at + t], mx
                den = torch.maximum((nn * q[at + t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                out[at + t] = torch.einsum("hkv,hk->hv", S, q[at + t]) / den[:, None]
            state[r, H * dk * dv:H * dk * (dv + 1)], state[r, H * dk * (dv + 1):] = nn.reshape(-1), m
        state[r, :H * dk * dv] = S.reshape(-1)
        at += n
    o = (_rms(out, 1e-6) * norm).view(len(x), -1) * gate
    return {"y": o @ w("o", W, H * dv).T, "state": state}


def _exact_experts(case, seed):
    W, F, E, out_n, top = case["width"], case["ff"], case["experts"], case["experts"] + case["identity"], case["top"]
    x = _rand(seed, "input", (case["tokens"], W)).double()
    s = torch.softmax(x @ _part_weight(seed, "router", (out_n, W)).double().T, -1)
    choice = s + _part_weight(seed, "correction", (out_n,)).double()
    best = choice.view(len(x), case["groups"], -1).amax(-1)
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(case["keep"], -1).indices, True)
    ids = choice.masked_fill(~kept.repeat_interleave(out_n // case["groups"], 1), -math.inf).topk(top, -1).indices
    weights = s.gather(1, ids)
    weights = weights / (weights.sum(-1, keepdim=True) + 1e-20) * 2.5
    share = torch.zeros_like(s).scatter_(1, ids, weights)
    y = x * share[:, E:].sum(-1, keepdim=True)
    for e in range(E):
        rows = share[:, e].nonzero()[:, 0]
        g, u, d = (_part_weight(seed, "e%d.%s" % (e, n), (F, W) if n != "down" else (W, F)).double() for n in ("gate", "up", "down"))
        h = x[rows]
        a = h @ g.T
        y[rows] += share[rows, e, None] * ((a * torch.sigmoid(a) * (h @ u.T)) @ d.T)
    return {"y": y}


def exact(case, seed):
    with torch.no_grad():
        return {"decode": _exact_model, "prompt": _exact_model, "block": _exact_block, "delta": _exact_recurrent,
                "memory": _exact_recurrent, "maps": _exact_maps, "experts": _exact_experts}[case["kind"]](case, seed)
