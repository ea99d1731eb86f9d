"""The framework's work as a set of cases for timing: prompt steps, decode steps and token picks of random-weight
models, through the public entry points (`Stratum.step`, `launch_decode`/`collect`, `decode_step`, `Sampler.pick`).

A case is a dict of plain values:

  task      "prompt"  one pass takes the sequences' whole prompts in one step and gives the logits behind each
            "decode"  one pass takes `steps` given tokens for every sequence of a running batch: the steps are launched
                      one ahead of the host's reading, as generation launches them, the last one is read with its logits
            "pick"    one pass draws a token for every row of logits
  model     whose shape (MODELS): the three Llama shapes at full depth, the other decoders with four layers
  dtype     "bfloat16" (the serving kernels) or "float32" (the true 32-bit path)
  batch, longest, shortest   how many sequences, and between which lengths theirs lie (the first is the longest)

A decode pass leaves its sequences longer, as it does in use; the batch begins anew when their room is used up.  Token
ids are no outputs of the prompt and decode cases: with random weights one row in twenty has a runner-up nearer than
bfloat16's rounding, so two correct implementations pick different ids; the logits and every step's largest one say all.
The decoders with routed experts run with dense feed-forwards for the same reason: a token whose last chosen expert is
nearly tied changes its logits by far more than rounding does.

`exact` restates the models in float64 with torch alone.
"""
import hashlib
import math
import random

import numpy as np
import torch

from stratum_b200 import SamplingParams, StepEntry, Stratum
from stratum_b200.config import GetizenConfig, LlamaConfig, NibelornConfig, VitinexConfig
from stratum_b200.engine import expected_tensors, model_from_tensors
from stratum_b200.sampling import Pcg32, Sampler

DEVICE = "cuda"
ROOM = 1024                 # tokens a decode batch's sequences may grow by before it begins anew
FILL_TOKENS = 16384         # tokens of one step while a decode batch's prompts are run

# ---------------------------------------------------------------------------------------------- the models
LLAMA_8B = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": 32, "hidden_size": 4096,
    "intermediate_size": 14336, "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128,
    "vocab_size": 128256, "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "max_position_embeddings": 131072,
    "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                     "original_max_position_embeddings": 8192},
    "tie_word_embeddings": False, "hidden_act": "silu", "torch_dtype": "bfloat16"}
LLAMA_7B = dict(LLAMA_8B, num_key_value_heads=32, intermediate_size=11008, vocab_size=32000, rope_theta=10000.0,
                rope_scaling=None, max_position_embeddings=4096)
LLAMA_1B = dict(LLAMA_8B, num_hidden_layers=16, hidden_size=2048, intermediate_size=8192, head_dim=64,
                tie_word_embeddings=True, rope_scaling=dict(LLAMA_8B["rope_scaling"], factor=32.0))

# widths of a 1B and an 8B model for the other decoders: (width, heads, kv heads, dense gated size, dense plain size)
SIZES = {"1b": (2048, 16, 4, 5504, 8192), "8b": (4096, 32, 8, 10880, 16384)}


def vitinex(size):
    """Three state-space layers to one of latent attention, one pass of the loop."""
    width, heads, _, gated, _ = SIZES[size]
    dim, rank, q_rank = (64, 256, 768) if size == "1b" else (128, 512, 1536)
    latent = {"heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": rank, "q_rank": q_rank,
              "scale": (dim + dim // 2) ** -0.5, "rot": {"base": 10000.0, "dims": dim // 2}}
    ssm = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    mlp = {"kind": "dense", "ff": gated}
    layers = [{"type": "latent_attention", "mixer": latent, "mlp": mlp} if i == 3 else
              {"type": "mamba2", "mixer": ssm, "mlp": mlp} for i in range(4)]
    return {"architecture": "Vitinex", "vocab": 32768, "width": width, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
            "layers": layers, "loop": {"start": 0, "stop": 4, "times": 1}}


def nibelorn(size):
    """Three latent-attention layers to one of differential attention."""
    width, heads, kv, _, ff = SIZES[size]
    dim, rank = (64, 256) if size == "1b" else (128, 512)
    latent = {"heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": rank,
              "scale": (dim + dim // 2) ** -0.5, "rot": {"base": 10000.0, "dims": dim // 2}}
    diff = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "softcap": 30.0, "diff": 0.2,
            "q_temp": {"coef": 0.1, "every": 1024}}
    mlp = {"kind": "dense", "ff": ff}
    layers = [{"type": "attention", "mixer": diff, "mlp": mlp} if i == 2 else
              {"type": "latent_attention", "mixer": latent, "mlp": mlp} for i in range(4)]
    return {"architecture": "Nibelorn", "vocab": 32768, "width": width, "norm": {"eps": 1e-6}, "layers": layers}


def getizen(size):
    """Three layers of chunked attention beside a linear recurrence to one of retention."""
    width, heads, kv, gated, _ = SIZES[size]
    left = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
            "rot": {"base": 10000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    right = {"width": width, "blocks": width // 256, "conv": 4}
    ret = {"heads": heads, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 5 * h / heads) for h in range(heads)],
           "rot": {"base": 10000.0, "dims": 128}}
    mlp = {"kind": "dense", "ff": gated, "limit": 7.0}
    layers = [{"type": "retention", "mixer": ret, "mlp": mlp} if i == 3 else
              {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp} for i in range(4)]
    return {"architecture": "Getizen", "vocab": 32768, "width": width, "norm": {"eps": 1e-5, "groups": 2},
            "postln_alpha": 1.5, "layers": layers}


MODELS = {"llama-1b": (LlamaConfig, LLAMA_1B), "llama-7b": (LlamaConfig, LLAMA_7B), "llama-8b": (LlamaConfig, LLAMA_8B),
          **{f"{name}-{size}": (cls, make(size)) for size in SIZES
             for name, cls, make in (("vitinex", VitinexConfig, vitinex), ("nibelorn", NibelornConfig, nibelorn),
                                     ("getizen", GetizenConfig, getizen))}}
VOCAB = {m: raw.get("vocab_size") or raw["vocab"] for m, (_, raw) in MODELS.items()}


# ---------------------------------------------------------------------------------------------- the cases
def _prompt(model, batch, longest, shortest, dtype="bfloat16", name=None):
    return {"name": name, "task": "prompt", "model": model, "dtype": dtype, "batch": batch, "longest": longest,
            "shortest": shortest}


def _decode(model, batch, longest, shortest, steps, dtype="bfloat16", name=None):
    return {"name": name, "task": "decode", "model": model, "dtype": dtype, "batch": batch, "longest": longest,
            "shortest": shortest, "steps": steps}


def listed():
    return [
        # one person chatting with a small model: a token at a time, nothing to hide the launches behind
        _decode("llama-1b", 1, 201, 201, 1, name="llama1b decode 1"),
        # a small model serving many people, replies of about a thousand tokens so far
        _decode("llama-1b", 64, 1023, 300, 8, name="llama1b decode 64"),
        # the headline: eight conversations near four thousand tokens on the 8B shape
        _decode("llama-8b", 8, 3700, 3700, 8, name="llama8b decode 8"),
        # the other headline: one document read before an answer
        _prompt("llama-8b", 1, 2048, 2048, name="llama8b prompt 2048"),
        # chat turns that arrive together: short, of unequal lengths
        _prompt("llama-1b", 5, 187, 9, name="llama1b short prompts"),
        # eight unequal documents in one step, every head with keys of its own: the largest step
        _prompt("llama-7b", 8, 2048, 64, name="llama7b 8 prompts"),
        # the 32-bit path that results are checked against: a whole text, and tokens one by one
        _prompt("llama-1b", 1, 611, 611, dtype="float32", name="llama1b fp32 prompt"),
        _decode("llama-1b", 3, 450, 120, 2, dtype="float32", name="llama1b fp32 decode"),
        # picking a batch's next tokens with the usual filters
        {"name": "pick 24 rows", "task": "pick", "rows": 24, "vocab": 128256, "temperature": 0.8, "top_k": 50,
         "top_p": 0.95},
        # the other decoders: recurrences and latent attention over a text, latent and differential attention over
        # running conversations, chunked attention beside a recurrence over a batch of texts
        _prompt("vitinex-8b", 1, 2000, 2000, name="vitinex8b prompt"),
        _decode("nibelorn-8b", 6, 3000, 900, 8, name="nibelorn8b decode 6"),
        _prompt("getizen-8b", 3, 1500, 333, name="getizen8b 3 prompts"),
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("prompt", "prompt", "decode", "decode", "other prompt", "other decode", "fp32 prompt",
                       "fp32 decode", "pick"))
    if kind == "pick":
        top_k = rng.choice((0, _between(rng, 5, 300)))
        return {"task": "pick", "rows": _between(rng, 1, 64), "vocab": rng.choice((32000, 32768, 128256)),
                "temperature": round(rng.uniform(0.5, 1.2), 2), "top_k": top_k,
                "top_p": round(rng.uniform(0.7, 0.98), 2) if top_k == 0 or rng.random() < 0.5 else 1.0}
    if kind.startswith("other"):
        model = rng.choice(("vitinex-1b", "vitinex-8b", "nibelorn-1b", "nibelorn-8b", "getizen-1b", "getizen-8b"))
    else:
        model = "llama-1b" if kind.startswith("fp32") else rng.choice(("llama-1b", "llama-7b", "llama-8b"))
    if kind == "fp32 prompt":
        batch = rng.randint(1, 4)
        longest = _between(rng, 5, 1000 // batch)
    elif kind == "fp32 decode":
        batch = _between(rng, 1, 8)
        longest = _between(rng, 16, 1200 // batch)
    elif kind.endswith("prompt"):
        batch = _between(rng, 1, 8)
        longest = _between(rng, 5, min(4096, 6000 // batch))
    else:
        batch = _between(rng, 1, 64 if model == "llama-1b" else 16)
        longest = _between(rng, 30, min(4000, (40000 if model == "llama-1b" else 24000) // batch))
    shortest = rng.randint(max(4, longest // 8), longest)
    dtype = "float32" if kind.startswith("fp32") else "bfloat16"
    if kind.endswith("prompt"):
        case = _prompt(model, batch, longest, min(longest, shortest), dtype)
    else:
        case = _decode(model, batch, longest, shortest, rng.choice((1, 2, 8)), dtype)
    del case["name"]
    return case


def lengths(case):
    """Every sequence's tokens: the first is the longest, the others lie anywhere down to the shortest."""
    r = random.Random("%(batch)s %(longest)s %(shortest)s" % case)
    return [case["longest"]] + [r.randint(case["shortest"], case["longest"]) for _ in range(case["batch"] - 1)]


def _generator(seed, what):
    key = int.from_bytes(hashlib.sha256(f"{seed}:{what}".encode()).digest()[:7], "little")
    return torch.Generator(device=DEVICE).manual_seed(key)


def token_ids(case, seed):
    """One row of token ids per sequence, as long as its tokens and what it decodes from them."""
    more = ROOM if case["task"] == "decode" else 0
    ids = torch.randint(0, VOCAB[case["model"]], (case["batch"], case["longest"] + more), device=DEVICE,
                        generator=_generator(seed, "ids"))
    return ids.cpu().numpy()


def config_of(case):
    cls, raw = MODELS[case["model"]]
    return cls.from_dict(raw)


def make_weights(case, seed):
    """Matrices N(0, 0.02) as in bench.py; gains near one, small biases, and for the recurrences' constants the ranges
    that trained models start from.  A Llama's residual stream is a trained model's: the matrices that add to it are
    scaled by 1 / sqrt(2 layers) and the embeddings large enough to stay present through the depth (with plain N(0, 0.02)
    the rounding of bfloat16 alone moves the 8B shape's logits by 5 %)."""
    dtype = getattr(torch, case["dtype"])
    raw = MODELS[case["model"]][1]
    scales = {}
    if case["model"].startswith("llama"):
        into = (2 * raw["num_hidden_layers"]) ** -0.5
        scales = {"o_proj.weight": 0.02 * into, "down_proj.weight": 0.02 * into,
                  "embed_tokens.weight": 0.1 if raw["tie_word_embeddings"] else 0.6}
    out = {}
    for name, spec in expected_tensors(config_of(case)).items():
        if spec.optional:
            continue
        gen = _generator(seed, name)
        dt = dtype if spec.role == "matrix" else torch.float32
        if name.endswith((".A_log", ".dt_bias", ".lam")):
            u = torch.rand(spec.shape, device=DEVICE, generator=gen)
            if name.endswith(".A_log"):                       # decay rates of 1 to 16
                w = torch.log(1.0 + 15.0 * u)
            elif name.endswith(".dt_bias"):                   # steps of 0.001 to 0.1 before the input's share
                w = torch.log(torch.expm1(torch.exp(math.log(1e-3) + math.log(100.0) * u)))
            else:                                             # half-open gates decay by 0.9 to 0.999 a token
                w = torch.log(torch.expm1(-torch.log(0.9 + 0.099 * u) / 4.0))
        else:
            w = torch.randn(spec.shape, device=DEVICE, dtype=dt, generator=gen)
            if name.endswith(".conv"):
                w *= 0.3
            elif name.endswith((".lq1", ".lk1", ".lq2", ".lk2")):
                w *= 0.1
            elif name.endswith(".alpha"):
                w = 0.7 + 0.05 * w
            elif spec.init == "ones":
                w = 1.0 + 0.1 * w
            else:
                w *= next((v for end, v in scales.items() if name.endswith(end)), 0.02)
        out[name] = w.to(dt)
    return out


# ---------------------------------------------------------------------------------------------- one pass
class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["task"] == "pick":
        # a peaked head and a long tail, as a model's logits have
        z = torch.randn((case["rows"], case["vocab"]), device=DEVICE, generator=_generator(seed, "logits"))
        s.logits = z * 1.5 + 0.35 * torch.relu(z) ** 2
        s.sampler = Sampler(DEVICE)
        s.params = SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed)
        s.streams = [Pcg32(seed, i) for i in range(case["rows"])]
        return s
    lens = lengths(case)
    config = config_of(case)
    decode = case["task"] == "decode"
    pages = sum(-(-(n + (ROOM if decode else 0)) // 64) for n in lens)
    model = model_from_tensors(config, make_weights(case, seed), getattr(torch, case["dtype"]), DEVICE)
    s.llm = Stratum(dtype=case["dtype"], max_tokens=64 * pages, max_seqs=case["batch"], _model=model, _config=config)
    ids = token_ids(case, seed)
    if decode:
        s.prompts = [row[:n - case["steps"]].tolist() for row, n in zip(ids, lens)]
        s.follow = [[int(row[n - case["steps"] + k]) for row, n in zip(ids, lens)] for k in range(ROOM)]
        s.slots = []
        _begin(s)
        run(s)                                       # (the first pass captures the step's graph: a server's warm-up)
    else:
        s.prompts = [row[:n].tolist() for row, n in zip(ids, lens)]
        run(s)
        run(s)                                       # (a shape is captured when it is met for the second time)
    return s


def _begin(s):
    """The decode batch's sequences, up to the first token that a pass gives them."""
    for slot in s.slots:
        s.llm.release(slot)
    s.slots = [s.llm.acquire() for _ in s.prompts]
    chunk = min(2048, max(64, FILL_TOKENS // len(s.prompts)))
    for at in range(0, max(len(p) for p in s.prompts), chunk):
        s.llm.step([StepEntry(slot, p[at:at + chunk], []) for slot, p in zip(s.slots, s.prompts) if len(p) > at])
    s.done = 0


def run(s):
    case, task = s.case, s.case["task"]
    if task == "pick":
        ids, values = s.sampler.pick(s.logits, s.params, s.streams, want_values=True)
        return {"ids": ids, "values": values}
    llm = s.llm
    if task == "prompt":
        slots = [llm.acquire() for _ in s.prompts]
        logits = llm.step([StepEntry(slot, p, [len(p) - 1]) for slot, p in zip(slots, s.prompts)])
        for slot in slots:
            llm.release(slot)
        return logits
    if s.done + case["steps"] > ROOM:
        _begin(s)
    tokens = s.follow[s.done:s.done + case["steps"]]
    s.done += case["steps"]
    largest, flight = [], None
    for row in tokens[:-1]:                          # the next step is launched before this one's result is read
        ahead = llm.launch_decode(s.slots, row)
        if flight is not None:
            largest.append(llm.collect(flight)[1])
        flight = ahead
    if flight is not None:
        largest.append(llm.collect(flight)[1])
    _, values, logits = llm.decode_step(s.slots, tokens[-1], with_logits=True)
    largest.append(values)
    return {"largest": np.asarray(largest, dtype=np.float32), "logits": logits}


# ---------------------------------------------------------------------------------------------- what a pass needs
def _attention(model):
    """Per layer with attention: (heads, key size, value size, bytes of cache per token per element, window)."""
    raw = MODELS[model][1]
    if model.startswith("llama"):
        d = raw["head_dim"]
        one = (raw["num_attention_heads"], d, d, 2 * raw["num_key_value_heads"] * d, 0)
        return [one] * raw["num_hidden_layers"]
    out = []
    for layer in raw["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            # the heads' own keys and values for a text; a token's cache is the latent and the rotated part
            out.append((m["heads"], m["dim"] + m["rot_dim"], m["vdim"], m["kv_rank"] + m["rot_dim"], 0))
        elif layer["type"] == "attention":           # two maps over the same values
            out.append((2 * m["heads"], m["dim"], m["vdim"], m["kv_heads"] * (2 * m["dim"] + m["vdim"]), 0))
        elif layer["type"] == "parallel":
            a = m["left"]
            out.append((a["heads"], a["dim"], a["vdim"], a["kv_heads"] * (a["dim"] + a["vdim"]), a["mask"]["size"]))
    return out


def _matrices(model):
    """Weights that every token passes, and the head's."""
    head = body = 0
    tied = True
    for name, spec in expected_tensors(config_of({"model": model})).items():
        n = math.prod(spec.shape)
        if spec.optional or spec.role != "matrix":
            continue
        if name in ("model.embed_tokens.weight", "embed"):
            head = n
        elif name in ("lm_head.weight", "head"):
            tied = False
        else:
            body += n
    return body, head, tied


def _recurrences(model):
    """(multiply-adds per token, float32 numbers of state per sequence) of the recurrent mixers."""
    macs = state = 0
    for layer in MODELS[model][1].get("layers", ()):
        m = layer["mixer"]
        if layer["type"] == "mamba2":
            n = m["heads"] * m["vdim"] * m["state"]
        elif layer["type"] == "retention":
            n = m["heads"] * m["dim"] * m["vdim"]
        elif layer["type"] == "parallel":
            n = m["right"]["width"]
        else:
            continue
        macs, state = macs + 2 * n, state + n
    return macs, state


def work(case):
    if case["task"] == "pick":
        return {"bytes": case["rows"] * case["vocab"] * 4 + case["rows"] * 8, "flops": 2 * case["rows"] * case["vocab"]}
    size = 4 if case["dtype"] == "float32" else 2
    body, head, _ = _matrices(case["model"])
    macs, state = _recurrences(case["model"])
    att, lens, B, vocab = _attention(case["model"]), lengths(case), case["batch"], VOCAB[case["model"]]
    if case["task"] == "prompt":
        T = sum(lens)
        scores = sum(h * (dk + dv) * sum(min(p + 1, w or p + 1) for n in set(lens) for p in range(n)
                                         for _ in range(lens.count(n)))
                     for h, dk, dv, _, w in set(att) for _ in range(att.count((h, dk, dv, _, w))))
        flops = 2 * (body + macs) * T + 2 * head * B + 2 * scores
        moved = (body + head) * size + T * sum(c for *_, c, _ in att) * size + 8 * B * state + 4 * B * vocab
    else:
        k = case["steps"]
        flops = moved = 0
        for h, dk, dv, c, w in att:
            seen = sum(min(n + 1, w or n + 1) for n in lens)
            flops += 2 * k * h * (dk + dv) * seen
            moved += k * c * size * seen
        flops += 2 * k * B * (body + head + macs)
        moved += k * ((body + head) * size + 8 * B * state) + 4 * B * vocab
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["task"] == "pick":
        return "exact"
    # (measured against `exact`: 7e-6 in 32 bits, up to 1.5e-2 in bfloat16, where two orders of addition differ by as much)
    return {"rel": 3e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
F64 = torch.float64
MOST_EXACT_FLOPS = 4.5e14


def _lin(x, w, b=None):
    y = x @ w.to(F64).T
    return y if b is None else y + b.to(F64)


def _rms(x, eps, gain=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if gain is None else y * gain.to(F64)


def _frequencies(dims, base, scaling):
    """The rotation's frequencies; a Llama model's table is kept in 32 bits by definition, the others' likewise."""
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64)
    if scaling:
        wave, orig = 2 * math.pi / f, scaling["original"]
        s = (orig / wave - scaling["low"]) / (scaling["high"] - scaling["low"])
        mixed = (1 - s) * f / scaling["factor"] + s * f
        f = torch.where(wave < orig / scaling["high"], f, torch.where(wave > orig / scaling["low"], f / scaling["factor"], mixed))
    return f.to(torch.float32).to(DEVICE)


def _turn(x, freq, neighbours=False):
    """x [T, heads, m]: its first 2 len(freq) dimensions turned by position times frequency (a 32-bit product), in pairs
    (i, i + half) or (2i, 2i + 1)."""
    n = freq.numel()
    a = (torch.arange(x.shape[0], device=x.device, dtype=torch.float32)[:, None] * freq).to(F64)
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    y = x.clone()
    i, j = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if neighbours else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., i], x[..., j]
    y[..., i], y[..., j] = u * c - v * s, v * c + u * s
    return y


def _attend(q, k, v, scale, chunk=0, cap=0.0, block=512):
    """Causal attention of one sequence: q [T, H, d], k [T, G, d], v [T, G, e] -> [T, H, e]."""
    T, H, d = q.shape
    G, e = k.shape[1], v.shape[2]
    out = torch.empty((T, H, e), dtype=F64, device=q.device)
    kt, vt = k.permute(1, 2, 0), v.permute(1, 0, 2)                       # [G, d, T], [G, T, e]
    at = torch.arange(T, device=q.device)
    for b in range(0, T, block):
        n = min(block, T - b)
        lo = b // chunk * chunk if chunk else 0
        qb = q[b:b + n].view(n, G, H // G, d).permute(1, 2, 0, 3).reshape(G, -1, d)
        s = (qb @ kt[:, :, lo:b + n]).view(G, H // G, n, b + n - lo) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        i, j = at[b:b + n, None], at[None, lo:b + n]
        hidden = j > i
        if chunk:
            hidden = hidden | (i // chunk != j // chunk)
        p = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1)
        o = p.view(G, -1, b + n - lo) @ vt[:, lo:b + n]
        out[b:b + n] = o.view(G, H // G, n, e).permute(2, 0, 1, 3).reshape(n, H, e)
    return out


def _conv(x, taps, bias):
    """Causal convolution per channel; the last tap is the current token's."""
    n = taps.shape[1]
    y = bias.to(F64).expand_as(x).clone()
    for i in range(n):
        y[i:] += x[:x.shape[0] - i] * taps[:, n - 1 - i].to(F64)
    return y


def _each(lens, f, *rows):
    """f on every sequence's rows by themselves, put together again."""
    return torch.cat([f(*parts) for parts in zip(*(r.split(lens) for r in rows))])


class _Named:
    """A layer's weights by the ends of their names."""

    def __init__(self, weights, prefix):
        self.weights, self.prefix = weights, prefix

    def __getitem__(self, name):
        return self.weights[self.prefix + name]


def _exact_llama(raw, W, ids, lens):
    H, G, d, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    sc = raw["rope_scaling"]
    sc = sc and {"factor": sc["factor"], "low": sc["low_freq_factor"], "high": sc["high_freq_factor"],
                 "original": sc["original_max_position_embeddings"]}
    freq = _frequencies(d, raw["rope_theta"], sc)
    x = W["model.embed_tokens.weight"][ids].to(F64)
    for i in range(raw["num_hidden_layers"]):
        w = _Named(W, f"model.layers.{i}.")
        h = _rms(x, eps, w["input_layernorm.weight"])
        q, k, v = (_lin(h, w[f"self_attn.{n}_proj.weight"]) for n in "qkv")

        def attend(q, k, v):
            n = q.shape[0]
            o = _attend(_turn(q.view(n, H, d), freq), _turn(k.view(n, G, d), freq), v.view(n, G, d), d ** -0.5)
            return o.reshape(n, H * d)

        x = x + _lin(_each(lens, attend, q, k, v), w["self_attn.o_proj.weight"])
        h = _rms(x, eps, w["post_attention_layernorm.weight"])
        g = torch.nn.functional.silu(_lin(h, w["mlp.gate_proj.weight"])) * _lin(h, w["mlp.up_proj.weight"])
        x = x + _lin(g, w["mlp.down_proj.weight"])
    return _rms(x, eps, W["model.norm.weight"]), W["model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight"]


def _latent(m, w, h, lens, eps, neighbours):
    H, d, e, rank = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
    freq = _frequencies(m["rot"]["dims"], m["rot"]["base"], None)
    q = _lin(_rms(_lin(h, w["dq"]), eps, w["dq.norm"]), w["uq"]) if "q_rank" in m else _lin(h, w["q"])
    low = _lin(h, w["dkv"])
    c = _rms(low[:, :rank], eps, w["dkv.norm"])
    k, v = _lin(c, w["uk"]), _lin(c, w["uv"])

    def attend(q, k, kr, v):
        n = q.shape[0]
        q, kr = q.view(n, H, -1), _turn(kr.reshape(n, 1, -1), freq, neighbours)
        q = torch.cat([q[..., :d], _turn(q[..., d:], freq, neighbours)], -1)
        k = torch.cat([k.view(n, H, d), kr.expand(n, H, kr.shape[-1])], -1)
        return _attend(q, k, v.view(n, H, e), m["scale"])

    o = _each(lens, attend, q, k, low[:, rank:], v)
    if "q_rank" in m:
        o = o * torch.sigmoid(_lin(h, w["g"]))[..., None]
    return _lin(o.reshape(o.shape[0], H * e), w["o"])


def _state_space(m, w, h, lens, eps):
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    row = _lin(h, w["in"])
    z, dt = row[:, :inner], torch.nn.functional.softplus(row[:, 2 * inner + 2 * G * N:] + w["dt_bias"].to(F64), threshold=50)
    xbc = _each(lens, lambda r: _conv(r, w["conv"], w["conv.b"]), row[:, inner:2 * inner + 2 * G * N])
    xbc = torch.nn.functional.silu(xbc)
    decay = torch.exp(-torch.exp(w["A_log"].to(F64)) * dt)

    def scan(xbc, dt, decay):
        T = xbc.shape[0]
        x = xbc[:, :inner].view(T, H, P)
        b = (xbc[:, inner:inner + G * N].view(T, G, N)).repeat_interleave(H // G, 1)
        c = (xbc[:, inner + G * N:].view(T, G, N)).repeat_interleave(H // G, 1)
        dx = dt[..., None] * x
        S = torch.zeros((H, P, N), dtype=F64, device=h.device)
        y = torch.empty((T, H, P, 1), dtype=F64, device=h.device)
        for t in range(T):
            S.mul_(decay[t, :, None, None]).addcmul_(dx[t, :, :, None], b[t, :, None, :])
            torch.bmm(S, c[t, :, :, None], out=y[t])
        return (y[..., 0] + w["D"].to(F64)[:, None] * x).reshape(T, inner)

    y = _each(lens, scan, xbc, dt, decay) * torch.nn.functional.silu(z)
    y = _rms(y.view(y.shape[0], m["norm_groups"], -1), eps).reshape(y.shape) * w["norm"].to(F64)
    return _lin(y, w["o"])


def _exact_vitinex(raw, W, ids, lens):
    eps, mult = raw["norm"]["eps"], raw["residual_mult"]

    def ln(x, w):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w.to(F64), None, eps)

    x0 = W["embed"][ids].to(F64)
    x = _lin(torch.cat([x0, x0], -1), W["loop.in"]) + W["loop.step"][0].to(F64)
    for i, layer in enumerate(raw["layers"]):
        w, h = _Named(W, f"l{i}.mix."), ln(x, W[f"l{i}.norm1"])
        if layer["type"] == "mamba2":
            y = _state_space(layer["mixer"], w, h, lens, eps)
        else:
            y = _latent(layer["mixer"], w, h, lens, eps, True)
        x = x + mult * ln(y, W[f"l{i}.norm1b"])
        w, h = _Named(W, f"l{i}.mlp."), ln(x, W[f"l{i}.norm2"])
        g = torch.nn.functional.gelu(_lin(h, w["gate"], w["gate.b"]), approximate="tanh") * _lin(h, w["up"], w["up.b"])
        x = x + mult * ln(_lin(g, w["down"], w["down.b"]), W[f"l{i}.norm2b"])
    return ln(x, W["final.norm"]), W["embed"]


def _differential(m, w, h, lens, eps):
    H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_lin(h, w[n]) for n in "qkv")
    lam = math.exp(float((w["lq1"].to(F64) * w["lk1"].to(F64)).sum())) \
        - math.exp(float((w["lq2"].to(F64) * w["lk2"].to(F64)).sum())) + m["diff"]

    def attend(q, k, v):
        n = q.shape[0]
        p = torch.arange(n, device=q.device, dtype=F64)
        warm = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((p + 1) / m["q_temp"]["every"]) + 1.0)
        q, k = (q * warm[:, None]).view(n, H, 2, d), k.view(n, G, 2, d)
        a, b = (_attend(q[:, :, i], k[:, :, i], v.view(n, G, e), m["scale"], cap=m["softcap"]) for i in (0, 1))
        return _rms(a - lam * b, eps) * (1.0 - m["diff"])

    o = _each(lens, attend, q, k, v) * torch.sigmoid(_lin(h, w["g"]))[..., None]
    return _lin(o.reshape(o.shape[0], H * e), w["o"])


def _exact_nibelorn(raw, W, ids, lens):
    eps = raw["norm"]["eps"]

    def norm(x, name):
        return torch.tanh(W[name + ".alpha"].to(F64) * x) * W[name].to(F64) + W[name + ".b"].to(F64)

    x = W["embed"][ids].to(F64)
    for i, layer in enumerate(raw["layers"]):
        w, h = _Named(W, f"l{i}.mix."), norm(x, f"l{i}.norm1")
        if layer["type"] == "latent_attention":
            x = x + _latent(layer["mixer"], w, h, lens, eps, False)
        else:
            x = x + _differential(layer["mixer"], w, h, lens, eps)
        h = norm(x, f"l{i}.norm2")
        x = x + _lin(torch.nn.functional.gelu(_lin(h, W[f"l{i}.mlp.up"])), W[f"l{i}.mlp.down"])
    return norm(x, "final.norm"), W["head"]


def _chunked_and_recurrent(m, w, h, lens, eps):
    a, r = m["left"], m["right"]
    H, G, d, e, size = a["heads"], a["kv_heads"], a["dim"], a["vdim"], a["mask"]["size"]
    freq = _frequencies(a["rot"]["dims"], a["rot"]["base"], a["rot"]["scaling"])
    q = _rms(_lin(h, w["left.q"]), eps, w["left.q.norm"])
    k = _rms(_lin(h, w["left.k"]), eps, w["left.k.norm"])

    def attend(q, k, v):
        n = q.shape[0]
        q = _turn(q.view(n, H, d), freq) * w["left.temp"].to(F64)[:, None]
        o = _attend(q, _turn(k.view(n, G, d), freq), v.view(n, G, e), a["scale"], chunk=size)
        return o.reshape(n, H * e)

    o = _each(lens, attend, q, k, _lin(h, w["left.v"])) * torch.sigmoid(_lin(h, w["left.g"]))
    left = _rms(_lin(o, w["left.o"]), eps, w["left.out"])

    y = torch.nn.functional.gelu(_lin(h, w["right.y"], w["right.y.b"]), approximate="tanh")
    u = _each(lens, lambda x: _conv(x, w["right.conv"], w["right.conv.b"]), _lin(h, w["right.x"], w["right.x.b"]))
    ub = u.view(u.shape[0], r["blocks"], -1)
    gate, inp = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, w[f"right.{n}"].to(F64)) + w[f"right.{n}.b"].to(F64)).reshape(u.shape)
                 for n in ("ra", "ri"))
    log_a = -8.0 * gate * torch.nn.functional.softplus(w["right.lam"].to(F64), threshold=50)
    decay, push = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * inp * u

    def scan(decay, push):
        S, out = torch.zeros_like(push[0]), torch.empty_like(push)
        for t in range(push.shape[0]):
            torch.addcmul(push[t], decay[t], S, out=out[t])
            S = out[t]
        return out

    right = _rms(_lin(_each(lens, scan, decay, push) * y, w["right.o"]), eps, w["right.out"])
    return 0.5 * (left + right)


def _retention(m, w, h, lens, eps):
    H, d, e = m["heads"], m["dim"], m["vdim"]
    freq = _frequencies(m["rot"]["dims"], m["rot"]["base"], None)
    decay = torch.tensor(m["decay"], dtype=F64, device=h.device)[:, None, None]

    def scan(q, k, v):
        n = q.shape[0]
        q, k, v = _turn(q.view(n, H, d), freq), _turn(k.view(n, H, d), freq) / math.sqrt(d), v.view(n, H, e)
        S, o = torch.zeros((H, e, d), dtype=F64, device=h.device), torch.empty((n, H, e, 1), dtype=F64, device=h.device)
        for t in range(n):
            S.mul_(decay).addcmul_(v[t, :, :, None], k[t, :, None, :])
            torch.bmm(S, q[t, :, :, None], out=o[t])
        return _rms(o[..., 0], eps).reshape(n, H * e)

    o = _each(lens, scan, *(_lin(h, w[n]) for n in "qkv"))
    return _lin(o * torch.nn.functional.silu(_lin(h, w["g"])), w["o"])


def _exact_getizen(raw, W, ids, lens):
    eps, groups, alpha = raw["norm"]["eps"], raw["norm"]["groups"], raw["postln_alpha"]

    def norm(x, gain):
        return _rms(x.view(x.shape[0], groups, -1), eps).reshape(x.shape) * gain.to(F64)

    x = norm(W["embed"][ids].to(F64), W["embed.norm"])
    for i, layer in enumerate(raw["layers"]):
        mix = _chunked_and_recurrent if layer["type"] == "parallel" else _retention
        x = norm(alpha * x + mix(layer["mixer"], _Named(W, f"l{i}.mix."), x, lens, eps), W[f"l{i}.norm1"])
        w, lim = _Named(W, f"l{i}.mlp."), layer["mlp"]["limit"]
        g, u = torch.clamp(_lin(x, w["gate"]), max=lim), torch.clamp(_lin(x, w["up"]), -lim, lim)
        x = norm(alpha * x + _lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), w["down"]), W[f"l{i}.norm2"])
    return norm(x, W["final.norm"]), W["embed"]


def _exact_pick(case, seed):
    s = prepare(case, seed)
    ids, values = [], []
    for row, stream in zip(s.logits, s.streams):
        k = min(512, case["top_k"] or 512)
        best, at = torch.sort(row, descending=True, stable=True)          # the lower id first among equals
        p = torch.softmax((best[:k].to(F64) - best[0]) / np.float32(case["temperature"]), 0)
        keep = k if case["top_p"] >= 1 else min(k, int((torch.cumsum(p, 0) < float(np.float32(case["top_p"]))).sum()) + 1)
        cum = torch.cumsum(p[:keep], 0)
        i = min(keep - 1, int((cum <= stream.uniform() * cum[-1]).sum()))
        ids.append(int(at[i]))
        values.append(float(best[i]))
    return {"ids": np.asarray(ids), "values": np.asarray(values)}


@torch.no_grad()
def exact(case, seed):
    if case["task"] == "pick":
        return _exact_pick(case, seed)
    steps = case.get("steps", 0)
    lens = [n + (steps if case["task"] == "decode" else 0) for n in lengths(case)]
    body, head, _ = _matrices(case["model"])
    if 2.0 * body * sum(lens) > MOST_EXACT_FLOPS:
        return None
    W = make_weights(case, seed)
    ids = torch.from_numpy(np.concatenate([row[:n] for row, n in zip(token_ids(case, seed), lens)])).to(DEVICE)
    raw = MODELS[case["model"]][1]
    form = {"llama": _exact_llama, "vitinex": _exact_vitinex, "nibelorn": _exact_nibelorn, "getizen": _exact_getizen}
    h, table = form[case["model"].split("-")[0]](raw, W, ids, lens)
    ends = torch.tensor(lens, device=DEVICE).cumsum(0)
    if case["task"] == "prompt":
        return _lin(h[ends - 1], table)
    # the first of the passes that `run` makes stands behind the one that `prepare` made
    largest = [_lin(h[ends - steps + k], table) for k in range(steps)]
    return {"largest": torch.stack([z.max(-1).values for z in largest]), "logits": largest[-1]}
