"""What the engine is timed on: prompts in, tokens and logits out, through its public entry points.

Every case is one batch of requests and one of three ways to have it done:

* ``serve``: the step function as a serving loop drives it.  Requests are admitted with their sampling parameters,
  prompts go through in steps of at most 2,048 tokens, then every request decodes with steps launched one ahead of
  the tokens' way back; the distribution of the token after the last comes back as logits.
* ``score``: prompts in, logits of the last places out (one ``step.run`` per 2,048 tokens), as a trace replay or an
  evaluation of completions does it.
* ``generate``: ``LLM.generate`` over more requests than run at a time, prompts of many lengths and limits of their
  own, so that steps mix prompt portions with single tokens; the completions are then scored.

The models are the Qwen3 sizes of the bench and three of the other designs at the bench's width of 2,048 (the
mechanisms of the rest are theirs in other arrangements).  Weights are seeded and random, shaped like trained ones in
the two ways that matter for comparing results: the token after a token, and the experts a token goes to, are decided
by a clear margin instead of by the last bit.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from tokamak_b200 import LLM, SamplingParams
from tokamak_b200.config import architecture_of
from tokamak_b200.engine.core import EngineCore
from tokamak_b200.engine.step import SamplingRow, StepEntry
from tokamak_b200.models.decoder import DecoderModel
from tokamak_b200.weights.random_init import random_tensors

BUDGET = 2048           # most prompt tokens of a step
PAGE = 16
STD = 0.02


# ------------------------------------------------------------------------------------------------ models

def qwen3(layers, hidden, heads, ff, tied):
    return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": ff,
            "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": tied,
            "max_position_embeddings": 40960}


def ketalix():
    """Windowed attention (caps, sinks, blended values) and gated linear attention in turn."""
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5 * 2.0, "softcap": 30.0,
           "mask": {"size": 1024}, "rot": {"base": 1e6, "dims": 128}, "v_mix": True}
    gla = {"heads": 8, "dim": 128, "vdim": 256, "tau": 16.0, "rank": 16}
    layers = [{"type": "attention" if i % 2 == 0 else "gla", "mixer": att if i % 2 == 0 else gla,
               "mlp": {"kind": "dense", "ff": 8192}} for i in range(8)]
    return {"architecture": "Ketalix", "vocab": 65536, "width": 2048, "norm": {"eps": 1e-6},
            "embedding": {"scale": 1.0}, "layers": layers}


def logivik():
    """Latent attention (windowed; rotated with sinks and a gate) and the gated delta rule in turn."""
    win = {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": 1536, "scale": 128 ** -0.5,
           "mask": {"size": 1024}}
    rot = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
           "rot": {"base": 1e6, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    delta = {"heads": 8, "kv_heads": 4, "dim": 128, "vdim": 256, "conv": 4}
    order = [("latent_attention_2", win), ("delta", delta), ("latent_attention", rot), ("delta", delta)]
    layers = [{"type": order[i % 4][0], "mixer": order[i % 4][1], "mlp": {"kind": "dense", "ff": 8192}} for i in range(8)]
    return {"architecture": "Logivik", "vocab": 65536, "width": 2048, "norm": {"eps": 1e-6},
            "embedding": {"scale": 1.0}, "layers": layers}


def tarivik():
    """Chunked attention beside a state-space half, HGRN2, mLSTM; a mixture of 8 experts, 2 used, in every layer."""
    par = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}},
           "right": {"heads": 32, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 4},
           "left_scale": 0.7, "right_scale": 0.6}
    rec = {"heads": 8, "dim": 128, "vdim": 256}
    mlp = {"kind": "moe", "expert": {"ff": 4096}, "router": {"experts": 8, "top": 2, "groups": {"count": 4, "keep": 2}}}
    order = [("parallel", par), ("hgrn2", rec), ("parallel", par), ("mlstm", dict(rec, gate_cap=15.0))]
    layers = [{"type": order[i % 4][0], "mixer": order[i % 4][1], "mlp": mlp} for i in range(8)]
    return {"architecture": "Tarivik", "vocab": 65536, "width": 2048, "max_positions": 32768,
            "norm": {"eps": 1e-5, "groups": 8}, "canon": {"taps": 4}, "layers": layers}


MODELS = {
    "qwen3-0.6b": lambda: qwen3(28, 1024, 16, 3072, True),
    "qwen3-8b": lambda: qwen3(36, 4096, 32, 12288, False),
    "ketalix": ketalix, "logivik": logivik, "tarivik": tarivik,
}


def sizes_of(raw) -> tuple[int, int]:
    return (raw["vocab_size"], raw["hidden_size"]) if "vocab_size" in raw else (raw["vocab"], raw["width"])


def expected_of(raw):
    arch = architecture_of(raw)
    return DecoderModel.expected_tensors(arch.build_spec(arch.parse(raw)))


def make_weights(case, seed):
    """``(tensors by name, the token that follows each token)``, made on the device from the seed.

    Random weights as the engine's own seeded folders have them, except: products that add to the residual stream
    shrink with the depth or by their layer scale, and so do queries that read the stream as it is, whose scores would
    be all or nothing;
    embedded rows have elements of size one and an untied head holds them permuted, so that the next token is decided
    clearly, sampled or not; routers and embedded rows share directions, so that a token's experts are."""
    raw = MODELS[case["model"]]()
    vocab, width = sizes_of(raw)
    dtype = getattr(torch, case["dtype"])
    expected = expected_of(raw)
    w = random_tensors(expected, seed, STD, 0.1, dtype, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    layers = raw.get("num_hidden_layers") or len(raw["layers"])
    embed = w["model.embed_tokens.weight" if "model.embed_tokens.weight" in w else "embed"]
    embed.mul_(1.0 / STD)
    for name, t in w.items():
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            t.mul_((2 * layers) ** -0.5)
        elif name.endswith((".canon1", ".canon2")):
            t.mul_(0.4)
        elif name.endswith((".ls1", ".ls2")):
            t.mul_(0.3)
        elif raw.get("architecture") == "Logivik" and name.endswith(("mix.q", "mix.uq")):
            t.mul_(0.3)
    if raw.get("architecture") == "Tarivik":
        router = raw["layers"][0]["mlp"]["router"]
        dirs = F.normalize(torch.randn(1 + router["experts"], width, generator=gen, device="cuda"), dim=-1)
        picks = torch.rand(vocab, router["experts"], generator=gen, device="cuda").topk(router["top"], dim=-1).indices
        embed.copy_((embed.float() + 24.0 * (dirs[0] + dirs[1:][picks].sum(1))).to(dtype))
        for name, t in w.items():
            if name.endswith("mlp.router"):
                order = torch.randperm(router["experts"], generator=gen, device="cuda")
                t.copy_(((2.0 * dirs[1:][order] - dirs[0]) / 6.0).to(dtype).to(t.dtype))
            elif name.endswith("mlp.correction"):
                t.mul_(0.1)
    follows = torch.arange(vocab, device="cuda")
    if not raw.get("tie_word_embeddings"):
        follows = torch.randperm(vocab, generator=gen, device="cuda")
        w["lm_head.weight" if "lm_head.weight" in w else "head"][follows] = (3.0 * F.normalize(embed.float(), dim=-1)).to(dtype)
    for name, req in expected.items():
        if name in w and req.role in ("vector", "bias", "fraction", "matrix_f32"):
            w[name] = w[name].float()
    return w, follows


# ------------------------------------------------------------------------------------------------ cases

def case_of(name, how, model, requests, prompt, new=0, *, want=1, ragged=0.5, dtype="bfloat16", slots=0,
            temperature=0.0, top_k=0, top_p=1.0):
    c = dict(how=how, model=model, requests=requests, prompt=prompt, new=new, want=want, ragged=ragged, dtype=dtype,
             slots=slots or requests, temperature=temperature, top_k=top_k, top_p=top_p)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a short question to the smallest model, a few tokens back; all latency and launches
        case_of("0.6b short answer", "serve", "qwen3-0.6b", 1, 25, 12),
        # one user's chat turn at 8B, sampled as most programs sample
        case_of("8b one chat turn", "serve", "qwen3-8b", 1, 500, 32, temperature=0.8, top_p=0.95),
        # a handful of users at once, the bench's batch
        case_of("8b batch of 8", "serve", "qwen3-8b", 8, 1000, 48),
        # a loaded server: many requests, short prompts of all lengths, top-k sampling
        case_of("8b batch of 64", "serve", "qwen3-8b", 64, 150, 24, temperature=0.7, top_k=50, ragged=0.8),
        # the bench's prompt: one full step of prompt tokens
        case_of("8b prompt of 2048", "score", "qwen3-8b", 1, 2048),
        # short prompts of odd lengths in one step, as between two full ones
        case_of("8b three short prompts", "score", "qwen3-8b", 3, 131),
        # the offline batch: 32 requests of which 16 run at a time, mixed steps throughout
        case_of("0.6b offline batch", "generate", "qwen3-0.6b", 32, 300, 64, slots=16, ragged=0.9),
        # the 32-bit path, which checks of a model run in: logits of every place of a completion
        case_of("0.6b scored in float32", "score", "qwen3-0.6b", 2, 150, want=32, dtype="float32"),
        # recurrent and latent designs: prompts and decoding
        case_of("ketalix batch of 8", "serve", "ketalix", 8, 400, 40),
        case_of("logivik batch of 8", "serve", "logivik", 8, 400, 40),
        case_of("logivik prompt of 2000", "score", "logivik", 1, 2000, want=4),
        # recurrences and mixtures of experts
        case_of("tarivik batch of 8", "serve", "tarivik", 8, 400, 40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another batch: any model, one to sixty-four requests, prompts of 16 to 4,000 tokens, at most 6,000 in all."""
    how = rng.choice(["serve", "serve", "serve", "score", "score", "generate"])
    model = rng.choice(["qwen3-0.6b", "qwen3-8b", "qwen3-8b", "ketalix", "logivik", "tarivik"])
    ragged = round(rng.uniform(0.0, 0.9), 2)
    if how == "generate":
        requests = _log(rng, 4, 32)
        return case_of(None, how, model, requests, _log(rng, 16, 4000 // requests), _log(rng, 8, 24), ragged=ragged,
                       slots=max(2, requests // rng.choice([1, 2, 3])))
    if how == "score":
        if model == "qwen3-0.6b" and rng.random() < 0.5:
            return case_of(None, how, model, _log(rng, 1, 4), _log(rng, 16, 200), want=_log(rng, 1, 16), ragged=ragged,
                           dtype="float32")
        requests = _log(rng, 1, 16)
        return case_of(None, how, model, requests, _log(rng, 16, min(4000, 6000 // requests)), want=_log(rng, 1, 16), ragged=ragged)
    requests = _log(rng, 1, 64)
    sampling = rng.choice([{}, {}, dict(temperature=0.8, top_p=0.95), dict(temperature=0.7, top_k=50), dict(temperature=1.0)])
    return case_of(None, how, model, requests, _log(rng, 16, min(4000, 6000 // requests)), _log(rng, 6, 40 if requests <= 8 else 20), ragged=ragged, **sampling)


def lengths(case):
    """Prompt length of every request: the longest is ``prompt``, the others shorter by up to the share ``ragged``."""
    return [max(1, round(case["prompt"] * (1.0 - case["ragged"] * (0.618034 * i % 1.0)))) for i in range(case["requests"])]


def limits(case):
    """Tokens each request may generate: all the same, but for ``generate``, where they differ."""
    if case["how"] != "generate":
        return [case["new"]] * case["requests"]
    return [max(2, round(case["new"] * (1.0 - 0.8 * (0.414214 * i % 1.0)))) for i in range(case["requests"])]


def make_prompts(case, seed):
    vocab = sizes_of(MODELS[case["model"]]())[0]
    gen = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n,), generator=gen).tolist() for n in lengths(case)]


def prepare(case, seed):
    weights, _ = make_weights(case, seed)
    longest = max(lengths(case)) + case["new"] + 1
    need = sum(-(-(n + m + 1) // PAGE) * PAGE for n, m in zip(lengths(case), limits(case)))
    core = EngineCore("<random>", dtype=case["dtype"], tensors=weights, raw_config=MODELS[case["model"]](), max_seq_len=longest,
                      page_size=PAGE, pool_tokens=max(need, longest), max_slots=case["requests"], max_step_tokens=BUDGET)
    state = {"case": case, "core": core, "prompts": make_prompts(case, seed)}
    rows = dict(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"])
    if case["how"] == "generate":
        state["llm"] = LLM("<random>", _core=core, max_batch_size=case["slots"], max_num_batched_tokens=BUDGET, block_size=PAGE)
        state["sampling"] = [SamplingParams(max_new_tokens=m, ignore_eos=True, seed=i, **rows)
                             for i, m in enumerate(limits(case))]
    else:
        state["sampling"] = [SamplingRow(seed=i, **rows) for i in range(case["requests"])]
    return state


# ------------------------------------------------------------------------------------------------ one pass

def steps_of(prompts, want):
    """The prompts as steps of at most ``BUDGET`` tokens, in order; the last ``want`` places of each are wanted."""
    entries, room = [], BUDGET
    for i, tokens in enumerate(prompts):
        at = 0
        while at < len(tokens):
            n = min(room, len(tokens) - at)
            wanted = range(max(at, len(tokens) - want), at + n)
            entries.append(StepEntry(i, tokens[at:at + n], [p - at for p in wanted]))
            at, room = at + n, room - n
            if room == 0:
                yield entries
                entries, room = [], BUDGET
    if entries:
        yield entries


def score(core, prompts, want):
    logits = [core.step.run(entries) for entries in steps_of(prompts, want)]
    for i in range(len(prompts)):
        core.step.free(i)
    return logits[0] if len(logits) == 1 else torch.cat(logits)


def serve(core, prompts, sampling, new):
    step, tokens = core.step, [[] for _ in prompts]
    for i, row in enumerate(sampling):
        step.admit(i, row)
    for entries in steps_of(prompts, 1):
        got = step.run_and_sample(entries)
        for e, token in zip((e for e in entries if e.want), got):
            tokens[e.req_id].append(token)
    entries = [StepEntry(i, None, [0]) for i in range(len(prompts))]
    flight = step.launch_and_sample(entries)
    for left in range(new - 2, -1, -1):
        ahead = step.launch_and_sample(entries) if left else None
        for mine, token in zip(tokens, step.collect(flight)):
            mine.append(token)
        flight = ahead
    logits = step.run([StepEntry(i, mine[-1:], [0]) for i, mine in enumerate(tokens)])
    for i in range(len(prompts)):
        step.free(i)
    return tokens, logits


def run(state):
    case, core, prompts = state["case"], state["core"], state["prompts"]
    if case["how"] == "score":
        return {"logits": score(core, prompts, case["want"])}
    if case["how"] == "serve":
        tokens, logits = serve(core, prompts, state["sampling"], case["new"])
        return {"tokens": torch.tensor(tokens), "logits": logits}
    outs = state["llm"].generate(prompt_token_ids=prompts, sampling_params=state["sampling"])
    full = [p + o.output_token_ids for p, o in zip(prompts, outs)]
    return {"tokens": torch.tensor([t for o in outs for t in o.output_token_ids]), "logits": score(core, full, 1)}


# ------------------------------------------------------------------------------------------------ what a pass needs

def work(case):
    """Weights once per step that must come after another one, cached keys and values once per token that reads them,
    logits once; two operations per weight and token, and the attention's."""
    raw = MODELS[case["model"]]()
    vocab, width = sizes_of(raw)
    size = 2 if case["dtype"] == "bfloat16" else 4
    dense = experts = 0
    for name, req in expected_of(raw).items():
        n = math.prod(req.shape)
        if ".mlp.e" in name:
            experts += n
        elif len(req.shape) == 2 and not name.startswith(("embed", "pos", "model.embed", "lm_head", "head")):
            dense += n
    head = vocab * width
    router = raw["layers"][0]["mlp"].get("router") if "layers" in raw else None
    share = router["top"] / router["experts"] if router else 0.0
    if "layers" in raw:
        attn = []           # (bytes cached per token, operations per key, window)
        for lay in raw["layers"]:
            m = lay["mixer"].get("left", lay["mixer"])
            if "kv_heads" in m and "mask" in m:
                attn.append((2 * m["kv_heads"] * m["dim"] * size, 4 * m["heads"] * m["dim"], m["mask"]["size"]))
            elif "kv_rank" in m:
                row = m["kv_rank"] + m.get("rot_dim", 0)
                attn.append((row * size, 4 * m["heads"] * m["dim"], m.get("mask", {}).get("size", 1 << 30)))
    else:
        kv, d = raw["num_key_value_heads"], raw["head_dim"]
        attn = [(2 * kv * d * size, 4 * raw["num_attention_heads"] * d, 1 << 30)] * raw["num_hidden_layers"]

    def prompts(sizes):
        steps, tokens = -(-sum(sizes) // BUDGET), sum(sizes)
        keys = lambda n, w: sum(min(i + 1, w) for i in range(n))
        flops = 2.0 * tokens * (dense + share * experts) + sum(f * keys(n, w) for _, f, w in attn for n in sizes)
        touched = experts * (1.0 - (1.0 - share) ** (tokens / steps))
        return steps * size * (dense + touched) + tokens * sum(b for b, _, _ in attn), flops

    def decode(contexts):
        n = len(contexts)
        touched = experts * (1.0 - (1.0 - share) ** n)
        read = size * (dense + touched + head) + sum(b * min(c, w) for b, _, w in attn for c in contexts) + 4 * n * vocab
        return read, 2.0 * n * (dense + share * experts + head) + sum(f * min(c, w) for _, f, w in attn for c in contexts)

    lens, caps = lengths(case), limits(case)
    total, flops = prompts(lens)
    rows = sum(min(case["want"], n) for n in lens)
    if case["how"] == "score":
        return {"bytes": total + size * head + 4 * rows * vocab, "flops": flops + 2.0 * rows * head}
    if case["how"] == "serve":
        for s in range(case["new"]):
            b, f = decode([n + s + 1 for n in lens])
            total, flops = total + b, flops + f
        return {"bytes": total, "flops": flops}
    # all output tokens in steps of as many requests as run at a time; then the completions once more
    slots, out = min(case["slots"], case["requests"]), sum(caps)
    b, f = decode([n + m // 2 for n, m in zip(lens, caps)][:slots])
    b2, f2 = prompts([n + m for n, m in zip(lens, caps)])
    return {"bytes": total + b * out / slots + b2 + size * head + 4 * len(lens) * vocab,
            "flops": flops + f * out / slots + f2 + 2.0 * len(lens) * head}


def tolerance(case):
    """Logits of 16-bit activations are 0.2e-2 to 1.3e-2 (2-norm) off those in 64 bits, and two such results as much off
    each other; true 32-bit ones are 0.7e-6 off.  Tokens follow by clear margins."""
    if case["dtype"] == "float32":
        return {"rel": 4e-6, "max": 1e-3, "differ": 0.0}
    return {"rel": 0.03, "max": 0.9, "differ": 0.005}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

F64 = torch.float64


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def group_rms(x, w, groups, eps):
    return rms(x.view(*x.shape[:-1], groups, -1), eps).reshape(x.shape) * w


def attend(q, k, v, scale, *, window=None, chunk=None, softcap=None, sinks=None, slopes=None):
    """Causal attention of one request: ``q`` [T, H, d], ``k`` and ``v`` [T, G, .], a head at a time."""
    T, H, _ = q.shape
    at = torch.arange(T, device=q.device)
    far = at[:, None] - at[None, :]
    seen = far >= 0
    if window:
        seen &= far < window
    if chunk:
        seen &= at[:, None] // chunk == at[None, :] // chunk
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    for h in range(H):
        g = h // (H // k.shape[1])
        s = (q[:, h] @ k[:, g].T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if slopes is not None:
            s = s - slopes[h] * far
        s = s.masked_fill(~seen, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sinks is not None:
            top = torch.maximum(top, sinks[h])
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True)
        if sinks is not None:
            den = den + torch.exp(sinks[h] - top)
        out[:, h] = (e @ v[:, g]) / den
    return out


def turn_halves(x, theta):
    T, _, d = x.shape
    inv = 1.0 / (theta ** (torch.arange(0, d, 2, dtype=torch.float32, device=x.device) / d))
    a = (torch.arange(T, dtype=torch.float32, device=x.device)[:, None] * inv).to(F64)[:, None, :]
    u, v = x.chunk(2, dim=-1)
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), dim=-1)


def turn_pairs(x, freqs, mag=1.0):
    """Neighbouring pairs of the last axis turn by position times frequency; ``x`` [T, heads, d]."""
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None, None] * freqs
    c, s = a.cos() * mag, a.sin() * mag
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack((u * c - v * s, v * c + u * s), dim=-1).reshape(x.shape)


def pair_freqs(dims, base, scaling=None):
    i = torch.arange(dims // 2, dtype=F64, device="cuda")
    f = base ** (-2.0 * i / dims)
    if not scaling:
        return f, 1.0
    edge = lambda t: dims * math.log(scaling["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(edge(scaling["fast"])), 0), min(math.ceil(edge(scaling["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / scaling["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def causal_conv(x, taps):
    T, K = x.shape[0], taps.shape[1]
    padded = F.pad(x, (0, 0, K - 1, 0))
    return sum(taps[:, j] * padded[j:j + T] for j in range(K))


def scan(q, k, v, decay):
    """``S = decay S + k v^T``, ``o = S^T q``, all heads: ``q, k, decay`` [T, H, dk], ``v`` [T, H, dv]."""
    S = torch.zeros(*k.shape[1:], v.shape[-1], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = decay[t][..., None] * S + k[t][..., None] * v[t][:, None, :]
        out[t] = (S * q[t][..., None]).sum(1)
    return out


def mlstm_scan(q, k, v, gi, gf):
    S = torch.zeros(*k.shape[1:], v.shape[-1], dtype=F64, device=q.device)
    n, m = torch.zeros_like(k[0]), torch.zeros_like(gi[0])
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        m_new = torch.maximum(gf[t] + m, gi[t])
        a, b = torch.exp(gf[t] + m - m_new)[:, None], torch.exp(gi[t] - m_new)[:, None]
        m = m_new
        S = a[..., None] * S + (b * k[t])[..., None] * v[t][:, None, :]
        n = a * n + b * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[t] = (S * q[t][..., None]).sum(1) / den[:, None]
    return out


def delta_scan(q, k, v, beta, g):
    S = torch.zeros(*k.shape[1:], v.shape[-1], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = g[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - (S * k[t][..., None]).sum(1))
        S = S + k[t][..., None] * u[:, None, :]
        out[t] = (S * q[t][..., None]).sum(1)
    return out


class Sequences:
    """Rows of several requests, one after another; ``each`` applies a function request by request."""

    def __init__(self, sizes):
        self.sizes = sizes

    def each(self, f, *xs):
        return torch.cat([f(*part) for part in zip(*(x.split(self.sizes) for x in xs))])


def sub(w, prefix):
    """The tensors below a name, in 64 bits when asked for."""
    return lambda name: w[prefix + name].to(F64)


def qwen3_hidden(raw, w, x, seqs):
    heads, kv, d, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    for i in range(raw["num_hidden_layers"]):
        t = sub(w, f"model.layers.{i}.")
        h = rms(x, eps) * t("input_layernorm.weight")
        q = rms((h @ t("self_attn.q_proj.weight").T).view(-1, heads, d), eps) * t("self_attn.q_norm.weight")
        k = rms((h @ t("self_attn.k_proj.weight").T).view(-1, kv, d), eps) * t("self_attn.k_norm.weight")
        v = (h @ t("self_attn.v_proj.weight").T).view(-1, kv, d)
        o = seqs.each(lambda q, k, v: attend(turn_halves(q, raw["rope_theta"]), turn_halves(k, raw["rope_theta"]), v,
                                             d ** -0.5), q, k, v)
        x = x + o.flatten(1) @ t("self_attn.o_proj.weight").T
        h = rms(x, eps) * t("post_attention_layernorm.weight")
        x = x + (F.silu(h @ t("mlp.gate_proj.weight").T) * (h @ t("mlp.up_proj.weight").T)) @ t("mlp.down_proj.weight").T
    return rms(x, eps) * w["model.norm.weight"].to(F64)


def ketalix_hidden(raw, w, x, seqs):
    eps, first = raw["norm"]["eps"], None
    for i, lay in enumerate(raw["layers"]):
        t, m = sub(w, f"l{i}."), lay["mixer"]
        h, H, d, dv = rms(x, eps) * t("norm1"), m["heads"], m["dim"], m["vdim"]
        if lay["type"] == "attention":
            q, k = (h @ t("mix.q").T).view(-1, H, d), (h @ t("mix.k").T).view(-1, m["kv_heads"], d)
            v = (h @ t("mix.v").T).view(-1, m["kv_heads"], dv)
            first = v if first is None else first
            v = v + t("mix.vmix") * (first - v)
            freqs, _ = pair_freqs(m["rot"]["dims"], m["rot"]["base"])
            o = seqs.each(lambda q, k, v: attend(rms(turn_pairs(q, freqs), eps), rms(turn_pairs(k, freqs), eps), v, m["scale"],
                                                 window=m["mask"]["size"], softcap=m["softcap"], sinks=t("mix.sink")), q, k, v)
            y = o.flatten(1) @ t("mix.o").T
        else:
            alpha = torch.sigmoid((h @ t("mix.a1").T) @ t("mix.a2").T + t("mix.a2.b")).pow(1.0 / m["tau"]).view(-1, H, d)
            o = seqs.each(scan, (h @ t("mix.q").T).view(-1, H, d) * d ** -0.5, (h @ t("mix.k").T).view(-1, H, d),
                          (h @ t("mix.v").T).view(-1, H, dv), alpha)
            y = ((rms(o, eps) * t("mix.norm")).flatten(1) * F.silu(h @ t("mix.g").T)) @ t("mix.o").T
        x = x + rms(y, eps) * t("norm1b") * t("ls1")
        h = rms(x, eps) * t("norm2")
        y = (F.gelu(h @ t("mlp.gate").T, approximate="tanh") * (h @ t("mlp.up").T)) @ t("mlp.down").T
        x = x + rms(y, eps) * t("norm2b") * t("ls2")
    return rms(x, eps) * w["final.norm"].to(F64)


def logivik_hidden(raw, w, x, seqs):
    eps = raw["norm"]["eps"]
    for i, lay in enumerate(raw["layers"]):
        t, m = sub(w, f"l{i}."), lay["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if lay["type"] == "delta":
            conv = lambda n, heads: F.silu(seqs.each(lambda z: causal_conv(z, t(f"mix.{n}.conv")),
                                                     x @ t(f"mix.{n}").T)).view(x.shape[0], heads, -1)
            unit = lambda z: z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)
            rep = H // m["kv_heads"]
            q = (unit(conv("q", m["kv_heads"])) * d ** -0.5).repeat_interleave(rep, 1)
            k = unit(conv("k", m["kv_heads"])).repeat_interleave(rep, 1)
            g = torch.exp(-torch.exp(t("mix.A_log")) * F.softplus(x @ t("mix.a").T + t("mix.dt_bias")))
            o = seqs.each(delta_scan, q, k, conv("v", H), torch.sigmoid(x @ t("mix.b").T), g)
            y = ((rms(o, eps) * t("mix.norm")).flatten(1) * F.silu(x @ t("mix.g").T)) @ t("mix.o").T
        else:
            rank, dr = m["kv_rank"], m.get("rot_dim", 0)
            low = x @ t("mix.dkv").T
            c = rms(low[:, :rank], eps) * t("mix.dkv.norm")
            k, v = (c @ t("mix.uk").T).view(-1, H, d), (c @ t("mix.uv").T).view(-1, H, dv)
            if dr:
                q = (x @ t("mix.q").T).view(-1, H, d + dr)
                freqs, mag = pair_freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
                q_rot = seqs.each(lambda z: turn_pairs(z, freqs, mag), q[..., d:])
                k_rot = seqs.each(lambda z: turn_pairs(z, freqs, mag), low[:, None, rank:])
                q, k = torch.cat((q[..., :d], q_rot), -1), torch.cat((k, k_rot.expand(-1, H, -1)), -1)
                o = seqs.each(lambda q, k, v: attend(q, k, v, m["scale"], sinks=t("mix.sink")), q, k, v).flatten(1)
                o = o * torch.sigmoid(x @ t("mix.g").T)
            else:
                q = ((rms(x @ t("mix.dq").T, eps) * t("mix.dq.norm")) @ t("mix.uq").T).view(-1, H, d)
                o = seqs.each(lambda q, k, v: attend(q, k, v, m["scale"], window=m["mask"]["size"]), q, k, v).flatten(1)
            y = o @ t("mix.o").T
        x = x + rms(y, eps) * (1.0 + t("norm1"))
        y = (F.silu(x @ t("mlp.gate").T) * (x @ t("mlp.up").T)) @ t("mlp.down").T
        x = x + rms(y, eps) * (1.0 + t("norm2"))
    return rms(x, eps) * (1.0 + w["final.norm"].to(F64))


def tarivik_mixer(t, kind, m, h, eps, seqs):
    if kind == "parallel":
        left, right = (lambda n: t("mix.left." + n)), (lambda n: t("mix.right." + n))
        a = m["left"]
        H, G, d = a["heads"], a["kv_heads"], a["dim"]
        q = (rms(h @ left("q").T + left("q.b"), eps) * left("q.norm")).view(-1, H, d)
        k = (rms(h @ left("k").T + left("k.b"), eps) * left("k.norm")).view(-1, G, d)
        v = (h @ left("v").T + left("v.b")).view(-1, G, a["vdim"])
        slopes = [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)]
        o = seqs.each(lambda q, k, v: attend(q, k, v, a["scale"], chunk=a["mask"]["size"], sinks=left("sink"), slopes=slopes), q, k, v)
        y = (o.flatten(1) * torch.sigmoid(h @ left("g").T)) @ left("o").T
        b = m["right"]
        H, dv, N, G = b["heads"], b["vdim"], b["state"], b["groups"]
        z, xbc, dt = (h @ right("in").T).split([H * dv, H * dv + 2 * G * N, H], dim=-1)
        xbc = F.silu(seqs.each(lambda s: causal_conv(s, right("conv")), xbc) + right("conv.b"))
        s, B, C = xbc.split([H * dv, G * N, G * N], dim=-1)
        s, B, C = s.view(-1, H, dv), (B.view(-1, G, N).repeat_interleave(H // G, 1)), (C.view(-1, G, N).repeat_interleave(H // G, 1))
        dt = F.softplus(dt + right("dt_bias"))
        decay = torch.exp(-torch.exp(right("A_log")) * dt)[..., None].expand(-1, H, N)
        o = seqs.each(scan, C, B, dt[..., None] * s, decay) + right("D")[:, None] * s
        o = group_rms(o.flatten(1) * F.silu(z), right("norm"), b["norm_groups"], eps)
        return m["left_scale"] * y + m["right_scale"] * (o @ right("o").T)
    H, d, dv = m["heads"], m["dim"], m["vdim"]
    lin = lambda n: h @ t("mix." + n).T
    if kind == "hgrn2":
        f = (t("mix.lower") + (1.0 - t("mix.lower")) * torch.sigmoid(lin("f") + t("mix.f.b"))).view(-1, H, d)
        o = seqs.each(scan, F.silu(lin("q")).view(-1, H, d), 1.0 - f, lin("v").view(-1, H, dv), f)
        return (rms(o, eps) * t("mix.norm")).flatten(1) @ t("mix.o").T
    cap = m["gate_cap"]
    gi = cap * torch.tanh((lin("i") + t("mix.i.b")) / cap)
    gf = F.logsigmoid(cap * torch.tanh((lin("f") + t("mix.f.b")) / cap))
    o = seqs.each(mlstm_scan, lin("q").view(-1, H, d) * d ** -0.5, lin("k").view(-1, H, d), lin("v").view(-1, H, dv), gi, gf)
    return (rms(o, eps).flatten(1) * t("mix.norm") * torch.sigmoid(lin("g"))) @ t("mix.o").T


def tarivik_moe(t, r, h):
    n, keep = r["groups"]["count"], r["groups"]["keep"]
    s = torch.sigmoid(h @ t("mlp.router").T)
    choice = s + t("mlp.correction")
    groups = choice.view(-1, n, r["experts"] // n)
    kept = groups.topk(min(2, groups.shape[-1]), -1).values.sum(-1).topk(keep, -1).indices
    allowed = torch.zeros(len(h), n, dtype=torch.bool, device=h.device).scatter_(1, kept, True)
    chosen = groups.masked_fill(~allowed[..., None], -math.inf).flatten(1).topk(r["top"], -1).indices
    out = torch.zeros_like(h)
    for e in range(r["experts"]):
        rows, _ = torch.nonzero(chosen == e, as_tuple=True)
        y = (F.silu(h[rows] @ t(f"mlp.e{e}.gate").T) * (h[rows] @ t(f"mlp.e{e}.up").T)) @ t(f"mlp.e{e}.down").T
        out[rows] += s[rows, e, None] * y
    return out


def tarivik_hidden(raw, w, x, seqs):
    eps, groups = raw["norm"]["eps"], raw["norm"]["groups"]
    x = seqs.each(lambda z: z + w["pos"][:len(z)].to(F64), x)
    for i, lay in enumerate(raw["layers"]):
        t = sub(w, f"l{i}.")
        h = x + seqs.each(lambda z: causal_conv(z, t("canon1")), x)
        x = x + group_rms(tarivik_mixer(t, lay["type"], lay["mixer"], h, eps, seqs), t("norm1"), groups, eps)
        h = x + seqs.each(lambda z: causal_conv(z, t("canon2")), x)
        x = x + group_rms(tarivik_moe(t, lay["mlp"]["router"], h), t("norm2"), groups, eps)
    return group_rms(x, w["final.norm"].to(F64), groups, eps)


HIDDEN = {"qwen3-0.6b": qwen3_hidden, "qwen3-8b": qwen3_hidden, "ketalix": ketalix_hidden, "logivik": logivik_hidden,
          "tarivik": tarivik_hidden}


@torch.no_grad()
def exact(case, seed):
    """The logits in 64 bits over the whole sequences; the tokens are whole values and follow from the weights."""
    if work(case)["flops"] > 2.5e14:
        return None                     # minutes in 64 bits
    raw = MODELS[case["model"]]()
    w, follows = make_weights(case, seed)
    seqs = [torch.tensor(p, device="cuda") for p in make_prompts(case, seed)]
    rows = []
    for i, new in enumerate(limits(case)):
        made = []
        for _ in range(new if case["how"] != "score" else 0):
            made.append(follows[(made or [seqs[i][-1]])[-1]])
        seqs[i] = torch.cat([seqs[i], torch.stack(made)]) if made else seqs[i]
        rows.append(min(case["want"], len(seqs[i])))
    sizes = [len(s) for s in seqs]
    embed = w["model.embed_tokens.weight" if "model.embed_tokens.weight" in w else "embed"]
    x = HIDDEN[case["model"]](raw, w, embed[torch.cat(seqs)].to(F64), Sequences(sizes))
    last = torch.cat([part[-n:] for part, n in zip(x.split(sizes), rows)])
    head = w["lm_head.weight" if "lm_head.weight" in w else "head"] if not raw.get("tie_word_embeddings") else embed
    logits = last @ head.to(F64).T
    return {"logits": logits} if case["how"] == "score" else {"tokens": None, "logits": logits}
