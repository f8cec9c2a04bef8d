"""Performance cases: what users of this framework have it do, through its public entry points.

Three ways of using it are timed, each as one whole pass with its results on the host:

  loop    one request of the generation loop over an int4 decoder (`NativeLlmSession`): prompt, then token by token, the logits
          of every step taken (the caller samples)
  session a decode loop over a batch with key / value tensors as inputs and outputs (`CudaSession.run`), from a cached prefix on
  engine  batch steps over a ragged-batch module (`Engine.forward`), as a serving host or a replayed trace feeds them: prompts in
          portions, then one token per sequence and step, then the sequences are released

A case names a design and one of the three sizes whose hidden size, heads and feed-forward the benchmark uses (1b, 4b, 27b), a number
of layers, and the lengths of its sequences. Weights are random, on the grid of the stored type. Which experts a token takes does
not hang on rounding: some dimensions of the residual stream carry well separated levels of the token's own, no layer writes to
them, and the routers read nothing else.

`exact` computes the same logits with plain torch in 64 bits. It shares no code with the package but the seeded int4 weights.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from onyxia_b200 import ir, kipizen, lovuzen, models, mufevik, zusitar
from onyxia_b200.backend import CudaBackend
from onyxia_b200.checkpoint import Weights
from onyxia_b200.engine import Engine
from onyxia_b200.ir import HostTensor
from onyxia_b200.llm import NativeLlmSession

# hidden, heads, kv_heads, head_dim, ffn, recurrence blocks
SIZES = {"1b": (1152, 4, 1, 256, 6912, 9), "4b": (2560, 16, 4, 128, 10240, 10), "27b": (5376, 32, 16, 128, 21504, 21)}
VOCAB = 32768
EXPERTS, TOP, GROUPS, KEEP = 16, 4, 4, 2
EPS = 1e-6
RANK = 16            # of the map to the decays of gated linear attention
BIAS_ROWS = 32       # of a table of distance biases
STEP_TOKENS = 2048   # of prompts in one step, the scheduler's default
SCORED = 8           # last places of a prompt whose logits are wanted when nothing is generated
ENGINE_DESIGNS = ("lovuzen", "kipizen", "zusitar", "mufevik")


# ── the cases ──
def _engine_case(design, size, layers, batch, prompt, new, dtype="bf16", ragged=False):
    return {"way": "engine", "design": design, "size": size, "layers": layers, "dtype": dtype, "batch": batch, "prompt": prompt, "new": new, "ragged": ragged}


def _loop_case(model, layers, vocab, prompt, new):
    return {"way": "loop", "model": model, "layers": layers, "vocab": vocab, "prompt": prompt, "new": new}


def _session_case(layers, batch, context, new):
    return {"way": "session", "layers": layers, "batch": batch, "context": context, "new": new}


def listed():
    cases = {
        # the smallest: a short answer of the two-layer f32 decoder with explicit zero points; launches and host work count
        "c1_f32_answer": _loop_case("c1", 2, 32000, 16, 16),
        # the benchmark's request: the 26-layer decoder after a prompt of 512 tokens, its full vocabulary
        "int4_1b_request": _loop_case("1b", 26, 262144, 512, 32),
        # a long odd prompt of the int4 decoder whose answer is one token (classification)
        "int4_1b_prompt_2047": _loop_case("1b", 6, VOCAB, 2047, 0),
        # batched decode over a cached prefix at the width of the 27B architecture
        "int4_27b_batch64": _session_case(1, 64, 2048, 8),
        # one user with a long document: decode is bound by weights and a long context
        "lovuzen_27b_document": _engine_case("lovuzen", "27b", 1, 1, 8192, 32),
        # 32-bit arithmetic (--dtype float32), a few short ragged requests
        "lovuzen_1b_f32": _engine_case("lovuzen", "1b", 2, 3, 101, 16, dtype="f32", ragged=True),
        # a small serving batch whose users' prompts differ in length; the host samples, so every step's logits are taken
        "kipizen_1b_batch8": _engine_case("kipizen", "1b", 2, 8, 256, 32, ragged=True),
        # a prompt of 4096 tokens in one go through experts and windows
        "kipizen_1b_prompt_4096": _engine_case("kipizen", "1b", 2, 1, 4096, 0),
        # an ordinary prompt that fills no tile
        "zusitar_1b_prompt_1999": _engine_case("zusitar", "1b", 3, 1, 1999, 0),
        # a full serving batch: short questions, answers of 32 tokens
        "zusitar_4b_batch64": _engine_case("zusitar", "4b", 3, 64, 128, 32, ragged=True),
        # an ordinary prompt through mixed heads, gated linear attention and the delta rule
        "mufevik_4b_prompt_2048": _engine_case("mufevik", "4b", 2, 1, 2048, 0),
        # a single user who waits for every token
        "mufevik_1b_single": _engine_case("mufevik", "1b", 2, 1, 512, 48),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _spread(rng, low, high):
    """A whole number from low to high, its logarithm spread evenly."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def draw(rng):
    way = rng.choice(("loop", "session") + ("engine",) * 6)
    if way == "loop":
        if rng.random() < 0.3:
            return _loop_case("c1", 2, 32000, _spread(rng, 1, 128), _spread(rng, 4, 32))
        prompt = _spread(rng, 1, 2000)
        return _loop_case("1b", rng.randint(2, 8), VOCAB, prompt, rng.choice((0, _spread(rng, 4, 40))) if prompt > 8 else _spread(rng, 8, 40))
    if way == "session":
        batch = _spread(rng, 2, 64)
        return _session_case(rng.randint(1, 2), batch, _spread(rng, 130, 2048), rng.randint(4, 8))
    design = rng.choice(ENGINE_DESIGNS)
    size = rng.choice(("1b", "1b", "4b", "27b" if design == "lovuzen" else "1b"))
    f32 = size == "1b" and rng.random() < 0.12
    layers = 3 if design == "zusitar" else 1 if size == "27b" else 2
    if f32:
        return _engine_case(design, size, layers, _spread(rng, 1, 4), _spread(rng, 8, 128), _spread(rng, 4, 16), "f32", rng.random() < 0.5)
    batch = _spread(rng, 1, 64)
    prompt = _spread(rng, 16, min(4096, 8192 // batch))
    new = _spread(rng, 8, 40) if batch > 1 or rng.random() < 0.5 else 0
    return _engine_case(design, size, layers, batch, prompt, new, "bf16", rng.random() < 0.7)


# ── the sequences of a case ──
def _lengths(case):
    n, batch = case["prompt"], case["batch"]
    return [n - (i * 37) % (n // 4 + 1) if case["ragged"] else n for i in range(batch)]


def _steps(case):
    """Batch steps: (entries, whether their logits are taken); an entry is (sequence, first token, tokens, wanted places).
    Up to eight sequences the logits of every step come back, above that those of the last step."""
    lengths, new, batch = _lengths(case), case["new"], case["batch"]
    steps, entries, room = [], [], max(STEP_TOKENS, max(lengths) if new == 0 else 0)
    left = room
    for i, n in enumerate(lengths):
        at = 0
        while at < n:
            take = min(n - at, left)
            entries.append((i, at, take, list(range(max(0, take - SCORED), take)) if new == 0 and at + take == n else []))
            at, left = at + take, left - take
            if left == 0:
                steps.append((entries, new == 0))
                entries, left = [], room
    if entries:
        steps.append((entries, new == 0))
    for j in range(new):
        last = j == new - 1
        taken = batch <= 8 or last
        steps.append(([(i, n + j, 1, [0] if taken else []) for i, n in enumerate(lengths)], taken))
    return steps


def _tokens(rng, vocab, n):
    return rng.integers(0, vocab, n).tolist()


# ── designs of the engine: config.json's dictionary, weights ──
def _config(case):
    H, heads, kv, dim, ffn, blocks = SIZES[case["size"]]
    n = H // 128
    base = {"vocab": VOCAB, "width": H, "norm": {"eps": EPS}}
    rot = {"base": 10000.0, "dims": dim // 2}
    layers = []
    for i in range(case["layers"]):
        if case["design"] == "lovuzen":
            layers.append({"type": "parallel", "mlp": {"kind": "dense", "ff": ffn, "limit": 7.0}, "mixer": {
                "left": {"heads": heads, "kv_heads": kv, "dim": dim, "scale": dim ** -0.5, "bias_max": 128, "q_temp": {"coef": 0.1, "every": 1024}},
                "right": {"width": H, "blocks": blocks, "conv": 4}, "left_scale": 0.7, "right_scale": 0.7}})
        elif case["design"] == "kipizen":
            mlp = {"kind": "moe", "expert": {"ff": ffn // TOP}, "router": {"experts": EXPERTS, "top": TOP}}
            mixer = {"heads": n, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(1.0 + 7.0 * h / n) for h in range(n)]}
            if i % 2:
                mixer = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0, "mask": {"size": 4096},
                         "rot": dict(rot, scaling={"factor": 4.0})}
            layers.append({"type": "attention" if i % 2 else "lightning", "mixer": mixer, "mlp": mlp})
        elif case["design"] == "zusitar":
            ff = ffn // (TOP + 1) // 64 * 64
            mlp = {"kind": "moe", "expert": {"ff": ff, "limit": 7.0}, "shared": {"ff": ff, "limit": 7.0},
                   "router": {"experts": EXPERTS, "top": TOP, "scale": 2.5, "groups": {"count": GROUPS, "keep": KEEP}}}
            mixer = ({"heads": max(heads, 8), "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 1536 if H > 2000 else 768, "kv_rank": 512, "scale": 192 ** -0.5,
                      "rot": {"base": 10000.0, "dims": 64}},
                     {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0, "rot": rot},
                     {"inner": 2 * H, "state": 16, "dt_rank": -(-H // 128) * 8, "conv": 4})[i % 3]
            layers.append({"type": ("latent_attention", "attention", "mamba1")[i % 3], "mixer": mixer, "mlp": mlp if i else {"kind": "dense", "ff": ffn}})
        else:
            ff = ffn // (TOP + 1) // 64 * 64
            mlp = {"kind": "moe", "expert": {"ff": ff}, "shared": {"ff": ff}, "router": {"experts": EXPERTS, "top": TOP, "groups": {"count": GROUPS, "keep": KEEP}}}
            mixer = {"heads": n, "kv_heads": n, "dim": 128, "vdim": 128, "conv": 4}
            if i % 2 == 0:
                mixer = {"left": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "rot": rot},
                         "right": {"heads": n, "dim": 128, "vdim": 128, "tau": 16.0}}
            layers.append({"type": "delta" if i % 2 else "parallel", "mixer": mixer, "mlp": mlp})
    return dict(base, layers=layers, embedding={"scale": H ** 0.5}, streams=4, logit_scale=1.0)


def _package_config(case):
    """The package's form of the configuration, the module it belongs to and the shapes of its tensors."""
    kind, module = {"lovuzen": (lovuzen.LovuzenConfig, lovuzen), "kipizen": (kipizen.KipizenConfig, kipizen), "zusitar": (zusitar.ZusitarConfig, zusitar),
                    "mufevik": (mufevik.MufevikConfig, mufevik)}[case["design"]]
    cfg = kind.from_dict(_config(case))
    more = {"lovuzen": (BIAS_ROWS,), "mufevik": (RANK,)}.get(case["design"], ())
    return cfg, module, module.tensor_shapes(cfg, *more)


def _levels(gen, rows, grouped):
    """[rows, EXPERTS] evenly spaced levels, in an order of each row's own. Grouped: the two largest of a group are both above the two
    largest of the next one, in an order of the groups of the row's own."""
    down = torch.linspace(3.0, 3.0 / EXPERTS, EXPERTS, device="cuda")
    rand = lambda *s: torch.rand(s, generator=gen, device="cuda")  # noqa: E731
    if not grouped:
        return down[rand(rows, EXPERTS).argsort(1)]
    size = EXPERTS // GROUPS
    lead = down[:2 * GROUPS].reshape(GROUPS, 2)[rand(rows, GROUPS).argsort(1)]
    rest = down[2 * GROUPS:][rand(rows, EXPERTS - 2 * GROUPS).argsort(1)].reshape(rows, GROUPS, size - 2)
    both = torch.cat([lead, rest], 2)
    return both.gather(2, rand(rows, GROUPS, size).argsort(2)).reshape(rows, EXPERTS)


def _weights(case, seed):
    """Every tensor of the checkpoint as bf16 on the GPU."""
    design = case["design"]
    gen = torch.Generator("cuda").manual_seed(seed * 2 + 1)
    coded = 0 if design == "lovuzen" else EXPERTS   # leading dimensions of the stream that carry the levels
    rand = lambda s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    uniform = lambda s, lo, hi: lo + (hi - lo) * torch.rand(s, generator=gen, device="cuda")  # noqa: E731
    H, scale = SIZES[case["size"]][0], SIZES[case["size"]][0] ** 0.5 if design in ("kipizen", "zusitar") else 1.0
    out = {}
    for name, s in _package_config(case)[2].items():
        last = name.rsplit(".", 1)[-1]
        if name == "embed":
            a = rand(s) * (2.0 if coded else 1.0)
            if coded:
                a[:, :coded] = _levels(gen, s[0], design == "zusitar")
            a = a / scale
        elif last == "router":
            a = torch.zeros(s, device="cuda")
            order = torch.randperm(EXPERTS, generator=gen, device="cuda")
            if design == "zusitar":
                members = order.reshape(GROUPS, -1) % (EXPERTS // GROUPS)
                members = members.argsort(dim=1, stable=True)
                order = (torch.randperm(GROUPS, generator=gen, device="cuda")[:, None] * (EXPERTS // GROUPS) + members).reshape(-1)
            a[torch.arange(EXPERTS, device="cuda"), order] = {"kipizen": 2.0, "zusitar": 1.5, "mufevik": 3.0}[design]
        elif last == "correction":
            a = -0.5 - (torch.rand(s, generator=gen, device="cuda") < 0.5).float()
        elif name.endswith("router.b"):
            a = torch.zeros(s, device="cuda")
        elif last in ("norm1b", "norm2b"):
            a = 0.5 + 0.05 * rand(s)
            a[:coded] = 0.0
        elif name.endswith((".left.out", ".right.out")):
            a = 0.7 + 0.05 * rand(s)
            a[:coded] = 0.0
        elif last in ("norm", "norm1", "norm2", "D", "temp"):
            a = 1.0 + 0.1 * rand(s)
            if last == "norm2" and len(s) and design != "lovuzen":
                a[:coded] = 1.0
        elif last in ("ls1", "ls2"):
            a = 0.5 + 0.05 * rand(s)
        elif last == "in":
            a = rand(s) / math.sqrt(s[-1]) if design == "zusitar" else (1.0 + 0.1 * rand(s)) / s[0]
        elif last == "out":
            a = 1.0 + 0.1 * rand(s)
        elif last == "mix":
            a = 0.6 * torch.eye(s[0], device="cuda") + (0.4 + 0.05 * rand(s)) / s[0]
        elif last == "talk":
            a = 0.6 * torch.eye(s[0], device="cuda") + 0.5 * rand(s) / math.sqrt(s[0])
        elif last == "lam":
            a = uniform(s, -6.0, -1.0)
        elif name.endswith("a2.b"):
            a = uniform(s, -1.0, 5.0)
        elif name.endswith("dt.b"):
            a = uniform(s, -6.0, -2.0)
        elif last == "A_log" and len(s) == 2:
            a = torch.arange(1, s[1] + 1, device="cuda").float().log().expand(s)
        elif last in ("A_log", "dt_bias"):
            a = uniform(s, -4.0, -1.0)
        elif last in ("rel", "sink") or (last == "b" and s != (s[0], H)):
            a = 0.1 * rand(s)
        else:
            a = rand(s) / math.sqrt(s[-1])
            if coded and design != "zusitar" and (last == "down" or (last == "o" and ".left." not in name and ".right." not in name)):
                a[:coded] = 0.0
        out[name] = a.to(torch.bfloat16)
    return out


# ── int4 decoders ──
def _decoder(case):
    """The configuration; scales are small enough that the squares of random layers' results stay far from the end of f16."""
    if case["way"] == "session":
        cfg = models.config_gemma3_27b()
        cfg.vocab = VOCAB // 4
        cfg.scale_range = (0.0005, 0.002)
    else:
        cfg = models.config_c1() if case["model"] == "c1" else models.config_gemma3_1b()
        cfg.vocab = case["vocab"]
        if case["model"] == "1b":
            cfg.scale_range = (0.001, 0.004)
        cfg.max_positions = max(cfg.max_positions, case["prompt"] + case["new"])
    cfg.layers = case["layers"]
    return cfg


def _past(case, seed):
    """Keys and values of the cached prefix, [layers][2] of f16 [batch, kv_heads, context, dim]."""
    cfg = _decoder(case)
    gen = torch.Generator("cuda").manual_seed(seed)
    shape = (case["batch"], cfg.kv_heads, case["context"], cfg.head_dim)
    return [[torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16) for _ in range(2)] for _ in range(cfg.layers)]


# ── prepare and run ──
def prepare(case, seed):
    rng = np.random.default_rng([seed, 1])
    backend = CudaBackend((0,))
    if case["way"] == "loop":
        cfg = _decoder(case)
        llm = NativeLlmSession(backend, models.build_decoder(cfg, seed), case["prompt"] + case["new"] + 1)
        ids = _tokens(rng, cfg.vocab, case["prompt"] + case["new"])
        return {"way": "loop", "backend": backend, "llm": llm, "prompt": ids[:case["prompt"]], "next": ids[case["prompt"]:]}
    if case["way"] == "session":
        cfg = _decoder(case)
        session = backend.prepare(models.build_decoder(cfg, seed))
        ids = rng.integers(0, cfg.vocab, (case["new"], case["batch"], 1)).astype(np.int64)
        masks = [np.ones((case["batch"], case["context"] + j + 1), np.int64) for j in range(case["new"])]
        past = {}
        for l, pair in enumerate(_past(case, seed)):
            for part, t in zip(("key", "value"), pair):
                past[f"past_key_values.{l}.{part}"] = session.upload(HostTensor.from_numpy(t.cpu().numpy()))
        session.wait_idle()
        return {"way": "session", "backend": backend, "session": session, "ids": ids, "masks": masks, "past": past}
    cfg, module, _ = _package_config(case)
    weights = {k: v.view(torch.int16).cpu().numpy().view(np.uint16) for k, v in _weights(case, seed).items()}
    session = backend.prepare(module.build(cfg, Weights.from_bf16(weights), ir.F32 if case["dtype"] == "f32" else ir.BF16))
    lengths = _lengths(case)
    engine = Engine(session, sum(-(-(n + case["new"]) // 64) * 64 for n in lengths), case["batch"])
    tokens = [_tokens(rng, VOCAB, n + case["new"]) for n in lengths]
    steps = [([(i, tokens[i][at:at + n], want) for i, at, n, want in entries], taken) for entries, taken in _steps(case)]
    return {"way": "engine", "backend": backend, "engine": engine, "steps": steps, "batch": case["batch"]}


def run(state):
    out = []
    if state["way"] == "loop":
        llm = state["llm"]
        llm.reset()
        out.append(llm.step_logits(state["prompt"]))
        for token in state["next"]:
            out.append(llm.step_logits([token]))
        return out
    if state["way"] == "session":
        session, kv = state["session"], state["past"]
        for ids, mask in zip(state["ids"], state["masks"]):
            feed = {"input_ids": session.upload(HostTensor.from_numpy(ids)), "attention_mask": session.upload(HostTensor.from_numpy(mask))}
            results = dict(session.run({**feed, **kv}))
            kv = {"past_key_values." + k[len("present."):]: t for k, t in results.items() if k.startswith("present.")}
        return session.download(results["logits"]).numpy()
    engine = state["engine"]
    for entries, taken in state["steps"]:
        logits = engine.forward(entries, logits=taken)
        if taken:
            out.append(logits)
    for i in range(state["batch"]):
        engine.release(i)
    return out


# ── the work that a pass cannot do without ──
def _parts(case):
    """Of a design: elements of the dense tensors, per layer (experts, top, elements of one), per attention layer (cached bytes per token,
    FLOPs per query and key, window), and per sequence bytes of state."""
    cfg, shapes, size = _config(case), _package_config(case)[2], 4 if case["dtype"] == "f32" else 2
    count = lambda s: int(np.prod(s, dtype=np.int64))  # noqa: E731
    dense = sum(count(s) for k, s in shapes.items() if k not in ("embed", "head") and ".mlp.e" not in k)
    experts, attention, state = [], [], 0
    for l in cfg["layers"]:
        m, mlp = l["mixer"], l["mlp"]
        if mlp["kind"] == "moe":
            experts.append((EXPERTS, TOP, 3 * cfg["width"] * mlp["expert"]["ff"]))
        a = m.get("left", m) if l["type"] in ("parallel", "attention") else None
        if case["design"] == "lovuzen":
            attention.append((a["kv_heads"] * a["dim"] * size + 4, 4 * a["heads"] * a["dim"], 0))
            state += 4 * m["right"]["width"] * (1 + m["right"]["conv"])
        elif a:
            attention.append((a["kv_heads"] * (a["dim"] + a["vdim"]) * size, 2 * a["heads"] * (a["dim"] + a["vdim"]), (a.get("mask") or {}).get("size", 0)))
        if l["type"] == "latent_attention":
            attention.append(((m["kv_rank"] + m["rot_dim"]) * size, 2 * m["heads"] * (2 * m["kv_rank"] + m["rot_dim"]), 0))
        elif l["type"] == "mamba1":
            state += m["inner"] * (4 * m["state"] + size * m["conv"])
        elif l["type"] in ("lightning", "delta"):
            state += 4 * m["heads"] * m["dim"] * m["vdim"] + (size * m["conv"] * m["heads"] * 3 * m["dim"] if l["type"] == "delta" else 0)
        elif case["design"] == "mufevik":
            state += 4 * m["right"]["heads"] * m["right"]["dim"] * m["right"]["vdim"]
    return dense, experts, attention, state, size


def _decoder_work(cfg, sequences, taken):
    """Of one step of an int4 decoder: `sequences` (past, new) and rows whose logits are formed."""
    rows, esz = sum(n for _, n in sequences), 2 if cfg.act_dtype == ir.F16 else 4
    kv, q = cfg.kv_heads * cfg.head_dim, cfg.heads * cfg.head_dim
    layer = cfg.hidden * (2 * q + 2 * kv + 3 * cfg.ffn)
    head = cfg.hidden * cfg.vocab
    by = cfg.weight_bytes_per_token() + rows * cfg.hidden * esz + taken * cfg.vocab * esz
    fl = 2.0 * rows * cfg.layers * layer + 2.0 * taken * head
    for l in range(cfg.layers):
        w = cfg.layer_window(l)
        for past, new in sequences:
            seen = past + new if w < 0 else min(past + new, w + new)
            by += 2 * kv * esz * (seen + new)
            keys = sum(past + i + 1 if w < 0 else min(past + i + 1, w + 1) for i in range(new))
            fl += 4.0 * q * keys
    return by, fl


def work(case):
    by = fl = 0.0
    if case["way"] == "loop":
        cfg, n = _decoder(case), case["prompt"]
        # the f32 decoder forms the logits of all places of a prompt; one row is what its caller takes
        for past, new in [(0, n)] + [(n + j, 1) for j in range(case["new"])]:
            b, f = _decoder_work(cfg, [(past, new)], 1)
            by, fl = by + b, fl + f
        return {"bytes": by, "flops": fl}
    if case["way"] == "session":
        cfg = _decoder(case)
        for j in range(case["new"]):
            b, f = _decoder_work(cfg, [(case["context"] + j, 1)] * case["batch"], case["batch"])
            by, fl = by + b, fl + f
        return {"bytes": by, "flops": fl}
    dense, experts, attention, state, size = _parts(case)
    H = SIZES[case["size"]][0]
    for entries, _ in _steps(case):
        rows, wanted = sum(e[2] for e in entries), sum(len(e[3]) for e in entries)
        by += dense * size + rows * H * size + (wanted > 0) * H * VOCAB * size + wanted * VOCAB * 4 + 2 * state * len(entries)
        fl += 2.0 * rows * dense + 2.0 * wanted * H * VOCAB
        for many, top, each in experts:
            by += many * (1 - (1 - top / many) ** rows) * each * size
            fl += 2.0 * rows * top * each
        for per_token, per_pair, window in attention:
            for _, past, new, _ in entries:
                by += per_token * (min(past + new, window + new) if window else past + new) + per_token * new
                fl += per_pair * float(sum(min(past + i + 1, window) if window else past + i + 1 for i in range(new)))
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """Measured against `exact`: f32 up to 1.4e-6, bf16 up to 3.7e-3. The f16 decoders are off by 2e-4 to 2e-3, single tokens by 3e-2 (every
    operation rounds to f16, and a score or an overflowing square at an edge moves a whole row)."""
    if case["way"] == "engine":
        return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 0.015, "max": 0.15}
    return {"rel": 1e-5} if case["way"] == "loop" and case["model"] == "c1" else {"rel": 0.03, "max": 0.3}


# ── the same results in 64 bits ──
def _d(t):
    return t.double()


def _norm(x, w=None, eps=EPS):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * _d(w)


def _lin(x, w, b=None):
    y = x @ _d(w).T
    return y if b is None else y + _d(b)


def _sub(w, prefix):
    return {k[len(prefix):]: v for k, v in w.items() if k.startswith(prefix)}


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, base, dims, factor=1.0, neighbours=False):
    """x [B, T, heads, d]: rotation of the leading `dims` dimensions by position, in two halves or in neighbouring pairs."""
    half = dims // 2
    angle = (torch.arange(x.shape[1], device="cuda").double() / factor)[:, None] * base ** (-2.0 * torch.arange(half, device="cuda").double() / dims)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, half), slice(half, dims))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _weigh(s, first, window, sink=None):
    """Softmax weights of scores [B, n, T] of the queries at places `first` and on."""
    i = first + torch.arange(s.shape[1], device="cuda")[:, None]
    j = torch.arange(s.shape[2], device="cuda")[None]
    seen = (j <= i) & (j > i - window) if window else j <= i
    s = s.masked_fill(~seen, -math.inf)
    if sink is None:
        return torch.softmax(s, -1)
    return torch.softmax(torch.cat([s, sink.expand(s.shape[0], s.shape[1], 1)], -1), -1)[..., :-1]


def _attend(q, k, v, scale, softcap=0.0, window=0, sink=None, bias=None, talk=None):
    """Causal attention: q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv]; sink [H], bias [H, T] by distance, talk [H, H] mixes the heads' weights."""
    B, T, H, _ = q.shape
    share = H // k.shape[2]
    out = q.new_zeros(B, T, H, v.shape[-1])
    block = T if talk is None else 256
    for first in range(0, T, block):
        rows = slice(first, min(first + block, T))
        weights = []
        for h in range(H):
            s = q[:, rows, h] @ k[:, :, h // share].transpose(1, 2) * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if bias is not None:
                far = (torch.arange(T, device="cuda")[rows, None] - torch.arange(T, device="cuda")[None]).clamp(min=0)
                s = s + bias[h][far]
            w = _weigh(s, first, window, None if sink is None else sink[h])
            if talk is None:
                out[:, rows, h] = w @ v[:, :, h // share]
            else:
                weights.append(w)
        if talk is not None:
            mixed = torch.einsum("hg,gbij->hbij", talk, torch.stack(weights))
            for h in range(H):
                out[:, rows, h] = mixed[h] @ v[:, :, h // share]
    return out


def _conv(x, w, b=None):
    """Causal convolution per channel: x [B, T, C], w [C, taps], the last tap on the token itself."""
    taps = w.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    y = sum(padded[:, t:t + x.shape[1]] * _d(w)[:, t] for t in range(taps))
    return y if b is None else y + _d(b)


def _experts(h, w, chosen, weight, unit):
    flat, out = h.reshape(-1, h.shape[-1]), torch.zeros_like(h).reshape(-1, h.shape[-1])
    for e in range(EXPERTS):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        if len(rows):
            out[rows] += weight[rows, place][:, None] * unit(flat[rows], _sub(w, f"e{e}."))
    return out.reshape(h.shape)


def _open_groups(score, judged):
    """-inf where a score's group is not among the best ones."""
    shut = judged.argsort(1, descending=True)[:, KEEP:]
    closed = torch.zeros_like(judged).scatter(1, shut, 1.0).bool()
    return score.masked_fill(closed.repeat_interleave(EXPERTS // GROUPS, 1), -math.inf)


def _lovuzen_bias(rel):
    far, half = 128, BIAS_ROWS // 2
    row = []
    for n in range(far + 1):
        step = n
        if n >= half:
            step = math.log(n / half) / math.log(far / half) * (BIAS_ROWS - half)
            step = min(BIAS_ROWS - 1, half + math.floor(round(step) if abs(step - round(step)) < 1e-9 else step))
        row.append(step)
    return _d(rel)[row].T


def _lovuzen_layer(x, w, c):
    B, T, H = x.shape
    a, r = c["mixer"]["left"], c["mixer"]["right"]
    l, m = _sub(w, "mix.left."), _sub(w, "mix.right.")
    kp = _lin(x, l["k"])
    q = _norm(_lin(x, l["q"]), l["q.norm"]).reshape(B, T, a["heads"], a["dim"])
    k = _norm(kp, l["k.norm"]).reshape(B, T, a["kv_heads"], a["dim"])
    place = torch.arange(T, device="cuda").double()
    q = q * (1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((place + 1) / a["q_temp"]["every"]) + 1))[:, None, None]
    bias = _lovuzen_bias(l["rel"])
    bias = torch.cat([bias, bias[:, -1:].expand(-1, max(0, T - bias.shape[1]))], 1)
    left = _lin(_attend(q, k, kp.reshape(k.shape), a["scale"], bias=bias).reshape(B, T, -1), l["o"])
    y = torch.nn.functional.gelu(_lin(x, m["y"], m["y.b"]), approximate="tanh")
    u = _conv(_lin(x, m["x"], m["x.b"]), m["conv"], m["conv.b"])
    gate = lambda n: torch.sigmoid(torch.einsum("btki,koi->btko", u.reshape(B, T, r["blocks"], -1), _d(m[n])) + _d(m[n + ".b"])).reshape(u.shape)  # noqa: E731
    log_a = -8.0 * gate("ra") * torch.nn.functional.softplus(_d(m["lam"]))
    decay, entering = log_a.exp(), torch.sqrt(-torch.expm1(2.0 * log_a)) * gate("ri") * u
    S, states = torch.zeros_like(u[:, 0]), torch.empty_like(u)
    for t in range(T):
        S = decay[:, t] * S + entering[:, t]
        states[:, t] = S
    x = x + _d(w["ls1"]) * _norm(c["mixer"]["left_scale"] * left + c["mixer"]["right_scale"] * _lin(states * y, m["o"]), w["norm1"])
    limit, f = c["mlp"]["limit"], _sub(w, "mlp.")
    g, up = _lin(x, f["gate"]).clamp(max=limit), _lin(x, f["up"]).clamp(-limit, limit)
    return x + _d(w["ls2"]) * _norm(_lin(g * torch.sigmoid(1.702 * g) * (up + 1.0), f["down"]), w["norm2"])


def _kipizen_layer(x, w, c):
    B, T, H = x.shape
    h, m, a = _norm(x, w["norm1"]), _sub(w, "mix."), c["mixer"]
    if c["type"] == "attention":
        q, k, v = (_lin(h, m[n], m[n + ".b"]).reshape(B, T, heads, -1) for n, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
        q, k = (_norm(_turn(t, a["rot"]["base"], a["rot"]["dims"], a["rot"]["scaling"]["factor"])) for t in (q, k))
        y = _attend(q, k, v, a["scale"], a["softcap"], a["mask"]["size"], torch.zeros(a["heads"], device="cuda").double()).reshape(B, T, -1)
    else:
        q, k, v = (_silu(_lin(h, m[n])).reshape(B, T, a["heads"], -1) for n in "qkv")
        decay = torch.tensor(a["decay"], device="cuda", dtype=torch.float64)[:, None, None]
        S, o = q.new_zeros(B, a["heads"], a["dim"], a["vdim"]), torch.empty_like(v)
        for t in range(T):
            S = decay * S + k[:, t, :, :, None] * v[:, t, :, None]
            o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
        y = _norm(o.reshape(B, T, -1), m["norm"]) * torch.sigmoid(_lin(h, m["g"]))
    x = x + _lin(y, m["o"])
    h, f = _norm(x, w["norm2"]), _sub(w, "mlp.")
    z, chosen = _lin(h, f["router"], f["router.b"]).reshape(-1, EXPERTS).topk(TOP, 1)
    return x + _experts(h, f, chosen, torch.softmax(z, 1), lambda r, e: _lin(_silu(_lin(r, e["gate"])) * _lin(r, e["up"]), e["down"]))


def _zusitar_layer(x, w, c):
    B, T, H = x.shape
    h, m, a = _norm(x, w["norm1"]), _sub(w, "mix."), c["mixer"]
    if c["type"] == "attention":
        q, k, v = (_lin(h, m[n], m[n + ".b"]).reshape(B, T, heads, -1) for n, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
        q, k = (_turn(t, a["rot"]["base"], a["rot"]["dims"], neighbours=True) for t in (q, k))
        o = _attend(q, k, v, a["scale"], a["softcap"], 0, _d(m["sink"])) * torch.sigmoid(_lin(h, m["g"]))[..., None]
        y = _lin(o.reshape(B, T, -1), m["o"], m["o.b"])
    elif c["type"] == "latent_attention":
        n, rank = a["heads"], a["kv_rank"]
        q = _lin(_norm(_lin(h, m["dq"]), m["dq.norm"]), m["uq"]).reshape(B, T, n, -1)
        kv = _lin(h, m["dkv"])
        latent = _norm(kv[..., :rank], m["dkv.norm"])
        turn = lambda t: _turn(t, a["rot"]["base"], a["rot"]["dims"])  # noqa: E731
        q = torch.cat([q[..., :a["dim"]], turn(q[..., a["dim"]:])], -1)
        k = torch.cat([_lin(latent, m["uk"]).reshape(B, T, n, -1), turn(kv[..., None, rank:]).expand(-1, -1, n, -1)], -1)
        o = _attend(q, k, _lin(latent, m["uv"]).reshape(B, T, n, -1), a["scale"]).reshape(B, T, -1)
        y = _lin(o * torch.sigmoid(_lin(h, m["g"])), m["o"])
    else:
        inner, rank, n = a["inner"], a["dt_rank"], a["state"]
        u, z = _lin(h, m["in"]).split(inner, -1)
        u = _silu(_conv(u, m["conv"], m["conv.b"]))
        p = _lin(u, m["x"])
        dt = torch.nn.functional.softplus(_lin(p[..., :rank], m["dt"], m["dt.b"]))
        A, Bt, Ct = -torch.exp(_d(m["A_log"])), p[..., rank:rank + n], p[..., rank + n:]
        S, o = u.new_zeros(B, inner, n), torch.empty_like(u)
        for t in range(T):
            S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * u[:, t])[..., None] * Bt[:, t, None]
            o[:, t] = (S * Ct[:, t, None]).sum(-1)
        y = _lin((o + _d(m["D"]) * u) * _silu(z), m["o"])
    x = x + _norm(y, w["norm1b"])
    h, f = _norm(x, w["norm2"]), _sub(w, "mlp.")
    if c["mlp"]["kind"] == "dense":
        y = _lin(_silu(_lin(h, f["gate"])) * _lin(h, f["up"]), f["down"])
    else:
        limit = c["mlp"]["expert"]["limit"]

        def unit(r, e):
            g = _lin(r, e["gate"]).clamp(max=limit)
            return _lin(g * torch.sigmoid(1.702 * g) * (_lin(r, e["up"]).clamp(-limit, limit) + 1.0), e["down"])

        s = torch.sigmoid(_lin(h, f["router"])).reshape(-1, EXPERTS)
        judged = s.reshape(-1, GROUPS, EXPERTS // GROUPS).topk(2, 2)[0].sum(2)
        chosen = _open_groups(s, judged).topk(TOP, 1)[1]
        weight = s.gather(1, chosen)
        weight = weight / (weight.sum(1, keepdim=True) + 1e-20) * c["mlp"]["router"]["scale"]
        y = _experts(h, f, chosen, weight, unit) + unit(h, _sub(f, "shared."))
    return x + _norm(y, w["norm2b"])


def _mufevik_mixer(h, m, c):
    B, T, H = h.shape
    if c["type"] == "parallel":
        a, r, l, g = c["mixer"]["left"], c["mixer"]["right"], _sub(m, "left."), _sub(m, "right.")
        q, k, v = (_lin(h, l[n]).reshape(B, T, heads, -1) for n, heads in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])))
        q, k = (_turn(t, a["rot"]["base"], a["rot"]["dims"]) for t in (q, k))
        left = _lin(_attend(q * _d(l["temp"])[:, None], k, v, a["scale"], talk=_d(l["talk"])).reshape(B, T, -1), l["o"])
        q, k, v = (_lin(h, g[n]).reshape(B, T, r["heads"], -1) for n in "qkv")
        q = q * r["dim"] ** -0.5
        alpha = torch.sigmoid(_lin(_lin(h, g["a1"]), g["a2"], g["a2.b"])).pow(1.0 / r["tau"]).reshape(q.shape)
        S, o = q.new_zeros(B, r["heads"], r["dim"], r["vdim"]), torch.empty_like(v)
        for t in range(T):
            S = alpha[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None]
            o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
        right = _lin(_norm(o, g["norm"]).reshape(B, T, -1) * _silu(_lin(h, g["g"])), g["o"])
        return 0.5 * (_norm(left, l["out"]) + _norm(right, g["out"]))
    a = c["mixer"]
    q, k, v = (_silu(_conv(_lin(h, m[n]), m[n + ".conv"])).reshape(B, T, a["heads"], -1) for n in "qkv")
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k = unit(q) * a["dim"] ** -0.5, unit(k)
    decay = torch.exp(-torch.exp(_d(m["A_log"])) * torch.nn.functional.softplus(_lin(h, m["a"], m["dt_bias"])))
    beta = torch.sigmoid(_lin(h, m["b"]))
    S, o = q.new_zeros(B, a["heads"], a["dim"], a["vdim"]), torch.empty_like(v)
    for t in range(T):
        S = decay[:, t, :, None, None] * S
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None]
        o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
    return _lin(_norm(o, m["norm"]).reshape(B, T, -1) * _silu(_lin(h, m["g"])), m["o"])


def _mufevik_layer(x, w, c):
    """x [streams, B, T, width]."""

    def through(x, n, sublayer):
        p = _sub(w, f"hc{n}.")
        y = sublayer(_norm(torch.einsum("s,s...->...", _d(p["in"]), x)) * _d(w[f"norm{n}"]))
        return torch.einsum("st,s...->t...", _d(p["mix"]), x) + _d(p["out"]).reshape(-1, 1, 1, 1) * y

    def mixture(h):
        f = _sub(w, "mlp.")
        s = torch.softmax(_lin(h, f["router"]).reshape(-1, EXPERTS), 1)
        score = s + _d(f["correction"])
        chosen = _open_groups(score, score.reshape(-1, GROUPS, EXPERTS // GROUPS).amax(2)).topk(TOP, 1)[1]
        unit = lambda r, e: _lin(_silu(_lin(r, e["gate"])) * _lin(r, e["up"]), e["down"])  # noqa: E731
        return _experts(h, f, chosen, s.gather(1, chosen), unit) + torch.sigmoid(_lin(h, f["shared.sg"])) * unit(h, _sub(f, "shared."))

    x = through(x, 1, lambda h: _mufevik_mixer(h, _sub(w, "mix."), c))
    return through(x, 2, mixture)


def _exact_engine(case, seed):
    rng = np.random.default_rng([seed, 1])
    lengths, c, w = _lengths(case), _config(case), _weights(case, seed)
    tokens = [_tokens(rng, VOCAB, n + case["new"]) for n in lengths]
    ids = torch.zeros(len(tokens), max(map(len, tokens)), dtype=torch.int64)   # what follows a shorter sequence changes nothing in it
    for i, t in enumerate(tokens):
        ids[i, :len(t)] = torch.tensor(t)
    x = _d(w["embed"][ids.cuda()])
    if case["design"] == "lovuzen":
        x = _norm(x, w["embed.norm"])
    elif case["design"] in ("kipizen", "zusitar"):
        x = x * c["embedding"]["scale"]
    else:
        x = x.expand(c["streams"], -1, -1, -1)
    layer = {"lovuzen": _lovuzen_layer, "kipizen": _kipizen_layer, "zusitar": _zusitar_layer, "mufevik": _mufevik_layer}[case["design"]]
    for i, l in enumerate(c["layers"]):
        x = layer(x, _sub(w, f"l{i}."), l)
    if case["design"] == "mufevik":
        x = x.sum(0)
    x, head, out = _norm(x, w["final.norm"]), _d(w["embed" if case["design"] == "zusitar" else "head"]), []
    for entries, taken in _steps(case):
        if taken:
            out.append(torch.stack([x[i, at + p] for i, at, _, want in entries for p in want]) @ head.T)
    return out


def _exact_decoder(case, seed):
    cfg = _decoder(case)
    rng = np.random.default_rng([seed, 1])
    batch, context = case.get("batch", 1), case.get("context", 0)
    n = case["new"] + case.get("prompt", 0)
    if case["way"] == "session":
        ids, past = rng.integers(0, cfg.vocab, (n, batch, 1))[:, :, 0].T, _past(case, seed)
    else:
        ids, past = np.array([_tokens(rng, cfg.vocab, n)]), [[None, None]] * cfg.layers
    place = torch.arange(context, context + n, device="cuda")

    def lin(x, name, k, m):
        packed, scales, _ = models.nbits_arrays(cfg, seed, name, k, m)
        bits = torch.from_numpy(packed).cuda().reshape(m, -1)
        q = torch.stack([bits & 15, bits >> 4], 2).reshape(m, -1, 32).double() - 8.0
        return x @ (q * torch.from_numpy(scales).cuda().double().reshape(m, -1, 1)).reshape(m, -1)[:, :k].T

    def norm(x, name):
        return _norm(x, torch.from_numpy(models.norm_array(cfg, seed, name, cfg.hidden)).cuda(), cfg.eps)

    cos, sin = (torch.from_numpy(t).cuda().double()[place][:, None] for t in models.rope_caches(cfg))
    half, D, heads = cfg.head_dim // 2, cfg.head_dim, cfg.heads
    embed = torch.from_numpy(models.embed_array(cfg, seed)[np.unique(ids)]).cuda().double()
    x = embed[torch.from_numpy(np.searchsorted(np.unique(ids), ids)).cuda()]
    for l in range(cfg.layers):
        pre = f"/model/layers.{l}"
        h = norm(x, f"{pre}/input_layernorm")
        q, k, v = (lin(h, f"{pre}/attn/{t}_proj", cfg.hidden, m * D).reshape(batch, n, m, D) for t, m in (("q", heads), ("k", cfg.kv_heads), ("v", cfg.kv_heads)))
        q, k = (torch.cat([t[..., :half] * cos - t[..., half:] * sin, t[..., half:] * cos + t[..., :half] * sin], -1) for t in (q, k))
        k, v = (t if p is None else torch.cat([_d(p).transpose(1, 2), t], 1) for p, t in zip(past[l], (k, v)))
        o, w = torch.empty_like(q), cfg.layer_window(l)
        for hd in range(heads):
            g = hd // (heads // cfg.kv_heads)
            o[:, :, hd] = _weigh(q[:, :, hd] @ k[:, :, g].transpose(1, 2) * D ** -0.5, context, w + 1 if w >= 0 else 0) @ v[:, :, g]
        y = lin(o.reshape(batch, n, -1), f"{pre}/attn/o_proj", heads * D, cfg.hidden)
        x = x + (norm(y, f"{pre}/post_attention_layernorm") if cfg.sandwich_norms else y)
        h = norm(x, f"{pre}/pre_feedforward_layernorm")
        y = torch.nn.functional.gelu(lin(h, f"{pre}/mlp/gate_proj", cfg.hidden, cfg.ffn), approximate="tanh") * lin(h, f"{pre}/mlp/up_proj", cfg.hidden, cfg.ffn)
        y = lin(y, f"{pre}/mlp/down_proj", cfg.ffn, cfg.hidden)
        x = x + (norm(y, f"{pre}/post_feedforward_layernorm") if cfg.sandwich_norms else y)
    first = max(case.get("prompt", n) - 1, 0) if case["way"] == "loop" else n - 1
    logits = lin(norm(x, "/model/norm")[:, first:], "/lm_head", cfg.hidden, cfg.vocab)
    return logits if case["way"] == "session" else list(logits[0])


def exact(case, seed):
    with torch.no_grad():
        return _exact_engine(case, seed) if case["way"] == "engine" else _exact_decoder(case, seed)
