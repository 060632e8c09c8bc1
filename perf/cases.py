"""The work that users of this engine have it do, as cases that can be timed and checked.

A case is a batch of requests taken from their prompts to their last token through the step function
(``ModelRunner.step``), which generation, serving and trace replay all go through: prompts run in portions, then (or
beside other prompts' portions) one given token per request and step, and the logits of every wanted place come back.
Token ids are given rather than sampled, so that a rounding in one step does not change the inputs of the next.

Sizes are those of ``akas_b200/bench.py`` (the LFM2 layer sizes 350m, 700m and 1.2b, and Gigusun and Girelix at the same
widths). Weights are random; the parameters whose values decide what a mixer does (forget gates, step sizes, decays) are
spread over the range that such layers are initialised with, so that short and long memories both occur.

``exact`` restates the three designs in float64 with torch alone: whole sequences, no cache, token by token where a
recurrence is involved.
"""

from __future__ import annotations

import gc
import json
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

VOCAB = 65536
EPS = 1e-5
LAYERS = 16
# width, query heads, feed-forward width; 8 key/value heads of size 64 everywhere
SHAPES = {"350m": (1024, 16, 4608), "700m": (1536, 24, 6912), "1.2b": (2048, 32, 8192)}
KV_HEADS, HEAD = 8, 64
LFM2_ATTENTION = (2, 5, 8, 10, 12, 14)  # the other layers are short convolutions
GIGUSUN_KINDS = ("gla", "delta", "attention") * 5 + ("gla",)
THETA = 1000000.0
WINDOW, KEPT, SOFTCAP, TAU, RANK = 1024, 4, 30.0, 16.0, 64  # Gigusun's attention mask and cap, and its gates
EXPERTS, IDENTITY, TOP, GROUPS, KEEP = 14, 2, 4, 4, 2  # Girelix's router


# ------------------------------------------------------------------------------------------------ the cases


def _case(name, design, shape, requests, shortest, longest, portion, budget, steps, dtype="bfloat16", serving=False, score=False):
    """``requests`` prompts of ``shortest`` to ``longest`` tokens run in portions of at most ``portion`` tokens, at most
    ``budget`` in a step; then each request takes ``steps`` more tokens one by one, once all prompts are in, or, when
    ``serving``, as soon as its own prompt is in. ``score``: the logits of every prompt token are wanted."""
    return dict(name=name, design=design, shape=shape, dtype=dtype, requests=requests, shortest=shortest, longest=longest,
                portion=portion, budget=budget, steps=steps, serving=serving, score=score)


def listed():
    return [
        # one short question, a short answer: launches and latency are all there is
        _case("chat_350m_b1", "lfm2", "350m", 1, 23, 23, 2048, 8192, 16),
        # many users at once: portions of new prompts share every step with the requests that decode
        _case("serving_350m_b64", "lfm2", "350m", 64, 128, 1000, 512, 512, 24, serving=True),
        # trace replay in float32, the arithmetic that bfloat16 is checked against: every token's logits
        _case("score_350m_float32", "lfm2", "350m", 4, 60, 301, 2048, 8192, 8, dtype="float32", score=True),
        # one long document, then a short answer
        _case("long_700m_b1", "lfm2", "700m", 1, 30000, 30000, 2048, 8192, 8),
        # one user, a longer answer
        _case("decode_1.2b_b1", "lfm2", "1.2b", 1, 512, 512, 2048, 8192, 64),
        # the benchmark's batch: 8 requests whose 2,048-token prompts are cached, decoding
        _case("decode_1.2b_b8", "lfm2", "1.2b", 8, 2048, 2048, 2048, 8192, 128),
        # a full batch of requests of all lengths
        _case("decode_1.2b_b64", "lfm2", "1.2b", 64, 64, 1000, 2048, 8192, 64),
        # one prompt, its first token
        _case("prefill_1.2b_2048", "lfm2", "1.2b", 1, 2048, 2048, 2048, 8192, 0),
        # two prompts of odd lengths through windowed attention and matrix-state mixers
        _case("gigusun_prefill_1.2b", "gigusun", "1.2b", 2, 1337, 2048, 2048, 8192, 0),
        _case("gigusun_decode_1.2b_b8", "gigusun", "1.2b", 8, 200, 500, 2048, 8192, 64),
        # a prompt, and a small batch decoding, through two mixers side by side and a mixture of experts
        _case("girelix_prefill_700m", "girelix", "700m", 1, 2048, 2048, 2048, 8192, 0),
        _case("girelix_decode_700m_b8", "girelix", "700m", 8, 200, 500, 2048, 8192, 64),
    ]


def draw(rng):
    """Another batch of requests, of the kinds and ranges above, that costs no more than the largest of them."""
    def spread(low, high):  # whole numbers, evenly over their logarithm
        return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))

    most = max(_cost(c) for c in listed())
    while True:
        design = rng.choice(("lfm2", "lfm2", "lfm2", "gigusun", "girelix"))
        shape = rng.choice(("350m", "700m") if design == "girelix" else ("350m", "700m", "1.2b"))
        kind = rng.choice(("prefill", "decode", "decode", "serving", "score") if design == "lfm2" else ("prefill", "decode", "serving"))
        requests = spread(1, 64) if kind != "prefill" else spread(1, 8)
        longest = spread(16, 30000 if design == "lfm2" and requests == 1 else 4096)
        longest = min(longest, 1000) if kind in ("serving", "score") else longest
        shortest = longest if requests == 1 else rng.randint(max(1, longest // 8), longest)
        steps = 0 if kind == "prefill" else spread(4, 128)
        portion = rng.choice((512, 1024, 2048))
        case = _case("", design, shape, requests, shortest, longest, portion, portion if kind == "serving" else 8192, steps,
                     dtype="float32" if kind == "score" else "bfloat16", serving=kind == "serving", score=kind == "score")
        if kind == "score" and requests * longest > 2500:
            continue  # float32 is for checking: a few short texts
        if _rows(case) > 4200 or _cost(case) > most:
            continue
        case.pop("name")
        return case


def _lengths(case):
    """Prompt length of every request: evenly from the shortest to the longest, in a shuffled order."""
    n, low, high = case["requests"], case["shortest"], case["longest"]
    lengths = [high - (high - low) * i // max(1, n - 1) for i in range(n)]
    return [lengths[i * 37 % n] for i in range(n)] if n % 37 else lengths


def _plan(case):
    """The steps: lists of (request, first token, tokens, wanted places among them)."""
    lengths, total = _lengths(case), [n + case["steps"] for n in _lengths(case)]
    at = [0] * len(lengths)
    steps = []
    while any(a < t for a, t in zip(at, total)):
        step, room = [], case["budget"]
        prompts_in = all(a >= n for a, n in zip(at, lengths))
        for r, n in enumerate(lengths):
            if at[r] < n:
                k = min(case["portion"], n - at[r], room)
                if k:
                    step.append((r, at[r], k, tuple(range(k)) if case["score"] else (k - 1,) if at[r] + k == n else ()))
                    room -= k
            elif at[r] < total[r] and (prompts_in or case["serving"]):
                step.append((r, at[r], 1, (0,)))
        for r, _, k, _ in step:
            at[r] += k
        steps.append(step)
    return steps


def _rows(case):
    return sum(len(want) for step in _plan(case) for _, _, _, want in step)


# ------------------------------------------------------------------------------------------------ models


def _config(design, shape):
    """config.json of the design at a shape."""
    c, heads, ff = SHAPES[shape]
    if design == "lfm2":
        return dict(architectures=["Lfm2ForCausalLM"], model_type="lfm2", hidden_size=c, num_attention_heads=heads,
                    num_key_value_heads=KV_HEADS, intermediate_size=ff, block_auto_adjust_ff_dim=False, vocab_size=VOCAB,
                    num_hidden_layers=LAYERS, full_attn_idxs=list(LFM2_ATTENTION), rope_theta=THETA, norm_eps=EPS,
                    conv_L_cache=3, conv_bias=False, tie_embedding=True, max_position_embeddings=128000)
    if design == "gigusun":
        h = c // 128
        mixers = dict(
            attention=dict(heads=heads, kv_heads=KV_HEADS, dim=HEAD, vdim=HEAD, scale=HEAD ** -0.5, softcap=SOFTCAP,
                           mask=dict(size=WINDOW, keep_first=KEPT)),
            gla=dict(heads=h, dim=64, vdim=128, tau=TAU, rank=RANK),
            delta=dict(heads=h, kv_heads=h // 2, dim=128, vdim=128, conv=4))
        return dict(architecture="Gigusun", width=c, vocab=VOCAB, max_positions=8192, norm=dict(eps=EPS),
                    layers=[dict(type=k, mixer=mixers[k], mlp=dict(ff=_gigusun_ff(shape), kind="dense")) for k in GIGUSUN_KINDS])
    left = dict(heads=c // 128, kv_heads=2, dim=HEAD, vdim=HEAD, scale=HEAD ** -0.5, rot=dict(base=THETA, dims=HEAD))
    right = dict(heads=c // 256, dim=64, vdim=128, decay=_decays(c // 256))
    mlp = dict(kind="moe", expert=dict(ff=ff // 4), router=dict(experts=EXPERTS, identity=IDENTITY, top=TOP, groups=dict(count=GROUPS, keep=KEEP)))
    layer = dict(type="parallel", mixer=dict(left=left, right=right, left_scale=1.0, right_scale=1.0), mlp=mlp)
    return dict(architecture="Girelix", width=c, vocab=VOCAB, norm=dict(eps=EPS), residual_mult=0.5, layers=[layer] * LAYERS)


def _gigusun_ff(shape):
    return -(-(3 * SHAPES[shape][2] // 2) // 256) * 256  # two matrices with the parameters of SwiGLU's three


def _decays(heads):
    return [1.0 - 2.0 ** -(3 + 5 * i / max(1, heads - 1)) for i in range(heads)]


def _inventory(design, shape):
    """name -> (shape, rule) of every tensor of the checkpoint; rule "m" is a matrix, "o" a matrix that writes into the
    residual stream (initialised smaller the deeper the model), "t" a tied embedding (its logits spread over a few units, as
    a trained model's do), "e" an embedding by itself, a number the mean of a vector, a pair the range that a parameter is
    spread over."""
    c, heads, ff = SHAPES[shape]
    q, kv, t = heads * HEAD, KV_HEADS * HEAD, {}
    if design == "lfm2":
        t["model.embed_tokens.weight"] = ((VOCAB, c), "t")
        for i in range(LAYERS):
            p = f"model.layers.{i}."
            t[p + "operator_norm.weight"] = t[p + "ffn_norm.weight"] = ((c,), 1.0)
            if i in LFM2_ATTENTION:
                a = p + "self_attn."
                t.update({a + "q_proj.weight": ((q, c), "m"), a + "k_proj.weight": ((kv, c), "m"), a + "v_proj.weight": ((kv, c), "m"),
                          a + "out_proj.weight": ((c, q), "o"), a + "q_layernorm.weight": ((HEAD,), 1.0), a + "k_layernorm.weight": ((HEAD,), 1.0)})
            else:
                t.update({p + "conv.in_proj.weight": ((3 * c, c), "m"), p + "conv.conv.weight": ((c, 1, 3), (-0.5, 0.5)), p + "conv.out_proj.weight": ((c, c), "o")})
            f = p + "feed_forward."
            t.update({f + "w1.weight": ((ff, c), "m"), f + "w3.weight": ((ff, c), "m"), f + "w2.weight": ((c, ff), "o")})
        t["model.embedding_norm.weight"] = ((c,), 1.0)
        return t
    t.update({"embed": ((VOCAB, c), "e"), "head": ((VOCAB, c), "m")})
    if design == "gigusun":
        h, ff = c // 128, _gigusun_ff(shape)
        t.update({"pos": ((8192, c), "m"), "embed.norm": ((c,), 0.0), "final.norm": ((c,), 0.0)})
        for i, kind in enumerate(GIGUSUN_KINDS):
            p, m = f"l{i}.", f"l{i}.mix."
            t.update({p + "norm1": ((c,), 0.0), p + "norm2": ((c,), 0.0), p + "mlp.up": ((ff, c), "m"), p + "mlp.down": ((c, ff), "o"), p + "mlp.act": ((4,), 0.5)})
            if kind == "attention":
                t.update({m + "q": ((q, c), "m"), m + "k": ((kv, c), "m"), m + "v": ((kv, c), "m"), m + "o": ((c, q), "o"), m + "g": ((heads, c), "m"),
                          m + "r1": ((heads,), (0.0, 1.0)), m + "r2": ((heads,), (0.1, 1.0)), m + "q.norm": ((HEAD,), 1.0), m + "k.norm": ((HEAD,), 1.0)})
            elif kind == "gla":  # gates from 0.92 (a memory of a dozen tokens) to 0.9998
                t.update({m + "q": ((h * 64, c), "m"), m + "k": ((h * 64, c), "m"), m + "v": ((h * 128, c), "m"), m + "g": ((h * 128, c), "m"), m + "o": ((c, h * 128), "o"),
                          m + "norm": ((128,), 1.0), m + "a1": ((RANK, c), "m"), m + "a2": ((h * 64, RANK), "m"), m + "a2.b": ((h * 64,), (-1.0, 6.0))})
            else:
                t.update({m + "q": ((h * 64, c), "m"), m + "k": ((h * 64, c), "m"), m + "v": ((h * 128, c), "m"), m + "g": ((h * 128, c), "m"), m + "o": ((c, h * 128), "o"),
                          m + "q.conv": ((h * 64, 4), (-0.5, 0.5)), m + "k.conv": ((h * 64, 4), (-0.5, 0.5)), m + "v.conv": ((h * 128, 4), (-0.5, 0.5)),
                          m + "b": ((h, c), "m"), m + "a": ((h, c), "m"), m + "A_log": ((h,), (0.0, 2.7)), m + "dt_bias": ((h,), (-6.0, -2.0)), m + "norm": ((128,), 1.0)})
        return t
    e, l, r = ff // 4, c // 128, c // 256
    t["final.norm"] = ((c,), 1.0)
    for i in range(LAYERS):
        p = f"l{i}."
        t.update({p + "norm1": ((c,), 1.0), p + "ls1": ((c,), 1.0), p + "ls2": ((c,), 1.0)})
        m = p + "mix.left."
        t.update({m + "q": ((l * 64, c), "m"), m + "k": ((128, c), "m"), m + "o": ((c, l * 64), "o"), m + "sink": ((l,), 0.0)})
        m = p + "mix.right."
        t.update({m + "q": ((r * 64, c), "m"), m + "k": ((r * 64, c), "m"), m + "v": ((r * 128, c), "m"), m + "g": ((r * 128, c), "m"), m + "o": ((c, r * 128), "o"), m + "norm": ((r * 128,), 1.0)})
        t.update({p + "mlp.router": ((EXPERTS + IDENTITY, c), "m"), p + "mlp.correction": ((EXPERTS + IDENTITY,), 0.0)})
        for j in range(EXPERTS):
            x = p + f"mlp.e{j}."
            t.update({x + "gate": ((e, c), "m"), x + "up": ((e, c), "m"), x + "down": ((c, e), "o")})
    return t


def _tensors(design, shape, dtype):
    """(name, tensor) of the checkpoint, on the GPU: the same for every call with the same arguments."""
    g = torch.Generator(device="cuda").manual_seed(20240607)
    std = {"m": 0.02, "o": 0.02 / math.sqrt(2 * LAYERS), "t": 0.1, "e": 1.0}
    for name, (size, rule) in _inventory(design, shape).items():
        if isinstance(rule, tuple):
            x = torch.rand(size, device="cuda", generator=g) * (rule[1] - rule[0]) + rule[0]
        else:
            x = torch.randn(size, device="cuda", generator=g) * std.get(rule, 0.02)
            x += 0.0 if rule in std else rule
        yield name, x.to(torch.float32 if dtype == "float32" else torch.bfloat16)


_folder = {}  # the checkpoint written last: (design, shape, dtype) -> its folder
_runner = {}  # the engine built last: what the case needs of it -> the engine


def _engine(case):
    """The engine that a user's program keeps for such requests, with pages for all of them."""
    from safetensors.torch import save_file

    from akas_b200 import EngineConfig
    from akas_b200.engine.runner import ModelRunner

    context = -(-(case["longest"] + case["steps"] + 1) // 64) * 64
    model = (case["design"], case["shape"], case["dtype"])
    key = model + (case["requests"], context, case["portion"], case["budget"], tuple(_lengths(case)), case["steps"])
    if key not in _runner:
        _runner.clear()
        gc.collect()
        torch.cuda.empty_cache()
        if model not in _folder:
            _folder.clear()
            folder = tempfile.TemporaryDirectory(prefix="akas-perf-")
            (Path(folder.name) / "config.json").write_text(json.dumps(_config(*model[:2])))
            save_file({n: x.cpu() for n, x in _tensors(*model)}, str(Path(folder.name) / "model.safetensors"))
            _folder[model] = folder
        options = EngineConfig(dtype=case["dtype"], max_requests=case["requests"], context=context, page_size=64,
                               prefill_chunk=case["portion"], prefill_token_budget=case["budget"])
        _runner[key] = ModelRunner(_folder[model].name, options)
    return _runner[key]


# ------------------------------------------------------------------------------------------------ one pass


def _texts(case, seed):
    rng = np.random.default_rng([seed, 7])
    return [rng.integers(0, VOCAB, n + case["steps"]).tolist() for n in _lengths(case)]


def prepare(case, seed):
    from akas_b200 import StepEntry

    texts = _texts(case, seed)
    steps = [[StepEntry(f"r{r}", texts[r][first : first + k], want) for r, first, k, want in step] for step in _plan(case)]
    return dict(runner=_engine(case), steps=steps, requests=[f"r{r}" for r in range(len(texts))],
                logits=torch.empty((_rows(case), VOCAB), dtype=torch.float32, device="cuda"))


def run(state):
    runner, logits, row = state["runner"], state["logits"], 0
    for entries in state["steps"]:
        got = runner.step(entries)
        if got.shape[0]:  # a step's logits are valid until the next step
            logits[row : row + got.shape[0]].copy_(got)
            row += got.shape[0]
    for request in state["requests"]:
        runner.release(request)
    return logits


# ------------------------------------------------------------------------------------------------ what it costs


def work(case):
    """Every step reads the weights that its tokens need once, and each request's keys and values (or state) once;
    logits are written once. Operations: the products, and attention over the visible keys."""
    size = 4 if case["dtype"] == "float32" else 2
    design, shape = case["design"], case["shape"]
    c, heads, _ = SHAPES[shape]
    dense = expert = 0
    for name, (dims, _) in _inventory(design, shape).items():
        if len(dims) == 2 and name not in ("model.embed_tokens.weight", "embed", "pos", "head"):
            if ".mlp.e" in name:
                expert += dims[0] * dims[1]
            else:
                dense += dims[0] * dims[1]
    routed = TOP * EXPERTS / (EXPERTS + IDENTITY)  # real experts of a token
    if design == "lfm2":
        attention, row, rest, heads_here = len(LFM2_ATTENTION), 2 * KV_HEADS * HEAD, 2 * c * 4 * (LAYERS - len(LFM2_ATTENTION)), heads
    elif design == "gigusun":
        h = c // 128
        attention, row, heads_here = GIGUSUN_KINDS.count("attention"), 2 * KV_HEADS * HEAD, heads
        rest = 4 * h * 128 * (64 * GIGUSUN_KINDS.count("gla") + 128 * GIGUSUN_KINDS.count("delta"))
    else:
        attention, row, rest, heads_here = LAYERS, 2 * HEAD, 4 * c // 256 * 64 * 128 * LAYERS, c // 128
    moved = flops = 0.0
    for step in _plan(case):
        tokens, wanted = sum(k for _, _, k, _ in step), sum(len(w) for _, _, _, w in step)
        moved += size * (dense + expert * min(1.0, tokens * routed / EXPERTS)) + (size * VOCAB * c if wanted else 0) + 4.0 * wanted * VOCAB
        moved += size * tokens * c
        flops += 2.0 * tokens * (dense + expert * routed / EXPERTS) + 2.0 * wanted * VOCAB * c
        for _, first, k, _ in step:
            if design == "gigusun":
                seen = sum(min(first + i + 1, WINDOW + KEPT) for i in range(k))
                held = min(first + k, WINDOW + KEPT + k)
            else:
                seen, held = k * first + k * (k + 1) / 2, first + k
            moved += size * attention * row * (held + k) + 2 * rest
            flops += 4.0 * attention * heads_here * HEAD * seen + (rest * k if design != "lfm2" else 0)
    return dict(bytes=moved, flops=flops)


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case):
    """About four times the error of the present kernels against 64 bits (3e-6 in float32, 3e-3 for the matrix-state designs
    in bfloat16), and less than twice what two ways of computing LFM2 in bfloat16 differ by (up to 1.9e-2: gates multiply
    gates in its layers). A token whose router is near a tie may take another expert and be off in every logit."""
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5}
    return {"rel": 0.03, "max": 0.4} if case["design"] == "lfm2" else {"rel": 0.015, "max": 0.5}


# ------------------------------------------------------------------------------------------------ in 64 bits

F = torch.float64


def exact(case, seed):
    texts, lengths = _texts(case, seed), _lengths(case)
    places = [[] for _ in texts]  # per request the positions whose logits are wanted, with their rows
    row = 0
    for step in _plan(case):
        for r, first, _, want in step:
            for w in want:
                places[r].append((first + w, row))
                row += 1
    store = {n: x for n, x in _tensors(case["design"], case["shape"], case["dtype"])}
    w = lambda name: store[name].to(F)  # noqa: E731
    out = torch.empty((row, VOCAB), dtype=F, device="cuda")
    order = sorted(range(len(texts)), key=lambda r: lengths[r])
    with torch.no_grad():
        while order:  # requests of like lengths together, shorter ones padded at their end (every mixer is causal)
            batch = [order.pop()]
            widest = len(texts[batch[0]])
            while order and (len(batch) + 1) * widest <= 20000:
                batch.append(order.pop())
            ids = torch.zeros((len(batch), widest), dtype=torch.long, device="cuda")
            for b, r in enumerate(batch):
                ids[b, : len(texts[r])] = torch.tensor(texts[r], device="cuda")
            hidden = {"lfm2": _lfm2, "gigusun": _gigusun, "girelix": _girelix}[case["design"]](w, ids)
            head = w("model.embed_tokens.weight" if case["design"] == "lfm2" else "head")
            for b, r in enumerate(batch):
                at, rows = (torch.tensor(x, device="cuda") for x in zip(*places[r]))
                out[rows] = hidden[b, at] @ head.T
            del hidden, head
    return out


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x):
    return x * torch.sigmoid(x)


def _causal_taps(x, taps):
    """x [B, T, C], taps [C, L] whose last column weighs the current token."""
    n = taps.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return sum(padded[:, j : j + x.shape[1]] * taps[:, j] for j in range(n))


def _attend(q, k, v, weigh):
    """q [B, T, H, D] over k, v [B, T, G, .]: ``weigh(scores [H, queries, keys], query positions, key positions)`` gives
    the weights. Query by query block, since all scores at once may not fit."""
    B, T, H, _ = q.shape
    out = torch.empty((B, T, H, v.shape[-1]), dtype=F, device=q.device)
    rep = H // k.shape[2]
    step = max(1, min(T, int(3e8 / (H * T))))
    for b in range(B):
        kb, vb = (x[b].transpose(0, 1).repeat_interleave(rep, 0) for x in (k, v))
        for i in range(0, T, step):
            e = min(T, i + step)
            at, keys = torch.arange(i, e, device=q.device)[:, None], torch.arange(e, device=q.device)[None]
            scores = q[b, i:e].transpose(0, 1) @ kb[:, :e].transpose(1, 2)
            out[b, i:e] = (weigh(scores, at, keys) @ vb[:, :e]).transpose(0, 1)
    return out.flatten(2)


def _angles(T, dims, device):
    freq = THETA ** (-2.0 * torch.arange(dims // 2, dtype=F, device=device) / dims)
    a = torch.arange(T, dtype=F, device=device)[:, None] * freq
    return torch.cos(a)[:, None], torch.sin(a)[:, None]  # [T, 1, dims / 2]


def _lfm2(w, ids):
    B, T = ids.shape
    x = w("model.embed_tokens.weight")[ids]
    cos, sin = _angles(T, HEAD, ids.device)

    def rotate(y):  # channel i turns with channel i + D / 2
        a, b = y.chunk(2, -1)
        return torch.cat((a * cos - b * sin, a * sin + b * cos), -1)

    def weigh(scores, at, keys):
        return torch.softmax((scores * HEAD ** -0.5).masked_fill(keys > at, float("-inf")), -1)

    for i in range(LAYERS):
        p = f"model.layers.{i}."
        h = _rms(x) * w(p + "operator_norm.weight")
        if i in LFM2_ATTENTION:
            a = p + "self_attn."
            q, k, v = ((h @ w(a + n + "_proj.weight").T).unflatten(-1, (-1, HEAD)) for n in "qkv")
            q, k = rotate(_rms(q) * w(a + "q_layernorm.weight")), rotate(_rms(k) * w(a + "k_layernorm.weight"))
            x = x + _attend(q, k, v, weigh) @ w(a + "out_proj.weight").T
        else:
            gate, out, value = (h @ w(p + "conv.in_proj.weight").T).chunk(3, -1)
            x = x + (out * _causal_taps(gate * value, w(p + "conv.conv.weight")[:, 0])) @ w(p + "conv.out_proj.weight").T
        h, f = _rms(x) * w(p + "ffn_norm.weight"), p + "feed_forward."
        x = x + (_silu(h @ w(f + "w1.weight").T) * (h @ w(f + "w3.weight").T)) @ w(f + "w2.weight").T
    return _rms(x) * w("model.embedding_norm.weight")


def _gigusun(w, ids):
    x = _rms(w("embed")[ids] + w("pos")[: ids.shape[1]]) * (1 + w("embed.norm"))
    mixers = {"attention": _windowed, "gla": _gla, "delta": _delta}
    for i, kind in enumerate(GIGUSUN_KINDS):
        p = f"l{i}."
        x = x + mixers[kind](lambda n: w(p + "mix." + n), _rms(x) * (1 + w(p + "norm1")))
        z = (_rms(x) * (1 + w(p + "norm2"))) @ w(p + "mlp.up").T
        a, b, c, e = w(p + "mlp.act")
        x = x + (a * _rms(z) + b * _rms(z * z) + c * _rms(z ** 3) + e) @ w(p + "mlp.down").T
    return _rms(x) * (1 + w("final.norm"))


def _windowed(w, h):
    """Attention inside a window and to the first tokens, with a capped score, a penalty that grows with the logarithm of the
    distance, one more term exp(0) in the denominator and a gate per head."""
    q, k, v = ((h @ w(n).T).unflatten(-1, (-1, HEAD)) for n in "qkv")
    q, k = _rms(q) * w("q.norm"), _rms(k) * w("k.norm")
    r1, r2 = w("r1")[:, None, None], w("r2")[:, None, None]

    def weigh(scores, at, keys):
        s = SOFTCAP * torch.tanh(scores * HEAD ** -0.5 / SOFTCAP) - r1 * torch.log1p(r2 * (at - keys).clamp(min=0))
        e = torch.exp(s.masked_fill((keys > at) | ((at - keys >= WINDOW) & (keys >= KEPT)), float("-inf")))
        return e / (1 + e.sum(-1, keepdim=True))

    o = _attend(q, k, v, weigh).unflatten(-1, (-1, HEAD)) * torch.sigmoid(h @ w("g").T)[..., None]
    return o.flatten(2) @ w("o").T


def _gla(w, h):
    """S <- diag(alpha) S + k v^T, o = S^T q."""
    q, k = ((h @ w(n).T).unflatten(-1, (-1, 64)) for n in "qk")
    v = (h @ w("v").T).unflatten(-1, (-1, 128))
    alpha = (torch.sigmoid((h @ w("a1").T) @ w("a2").T + w("a2.b")) ** (1 / TAU)).unflatten(-1, (-1, 64))
    o, S = torch.empty_like(v), torch.zeros((*v[:, 0].shape[:2], 64, 128), dtype=F, device=h.device)
    for t in range(h.shape[1]):
        S = alpha[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    o = (_rms(o * 64 ** -0.5) * w("norm")).flatten(2)
    return (o * _silu(h @ w("g").T)) @ w("o").T


def _delta(w, h):
    """S <- g S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q."""
    q, k, v = (_silu(_causal_taps(h @ w(n).T, w(n + ".conv"))).unflatten(-1, (-1, 128)) for n in "qkv")
    q, k = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
    rep = v.shape[2] // q.shape[2]
    q, k = (y.repeat_interleave(rep, 2) for y in (q * 128 ** -0.5, k))
    beta = torch.sigmoid(h @ w("b").T)[..., None]
    decay = torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(h @ w("a").T + w("dt_bias")))[..., None, None]
    o, S = torch.empty_like(v), torch.zeros((*v[:, 0].shape[:2], 128, 128), dtype=F, device=h.device)
    for t in range(h.shape[1]):
        S = decay[:, t] * S
        u = beta[:, t] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * u[:, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    return ((_rms(o) * w("norm")).flatten(2) * _silu(h @ w("g").T)) @ w("o").T


def _girelix(w, ids):
    x = w("embed")[ids]
    cos, sin = _angles(ids.shape[1], HEAD, ids.device)

    def rotate(y):  # channel 2i turns with channel 2i + 1
        a, b = y[..., 0::2], y[..., 1::2]
        return torch.stack((a * cos - b * sin, b * cos + a * sin), -1).flatten(-2)

    for i in range(LAYERS):
        p = f"l{i}."
        h = _rms(x) * w(p + "norm1")
        m = p + "mix.left."
        q, k = ((h @ w(m + n).T).unflatten(-1, (-1, HEAD)) for n in "qk")
        sink = w(m + "sink")[:, None, None]

        def weigh(scores, at, keys):
            e = torch.exp((scores * HEAD ** -0.5).masked_fill(keys > at, float("-inf")))
            return e / (e.sum(-1, keepdim=True) + torch.exp(sink))

        total = _attend(rotate(q), rotate(k), k, weigh) @ w(m + "o").T
        total = total + _decayed(lambda n: w(p + "mix.right." + n), h)
        total = w(p + "ls1") * total + w(p + "ls2") * _experts(lambda n: w(p + "mlp." + n), h.flatten(0, 1)).view_as(h)
        x = x + 0.5 * total
    return _rms(x) * w("final.norm")


def _decayed(w, h):
    """S <- decay S + k v^T, o = S^T q, one decay per head."""
    q, k = (_silu(h @ w(n).T).unflatten(-1, (-1, 64)) for n in "qk")
    v = _silu(h @ w("v").T).unflatten(-1, (-1, 128))
    decay = torch.tensor(_decays(v.shape[2]), dtype=F, device=h.device)[:, None, None]
    o, S = torch.empty_like(v), torch.zeros((*v[:, 0].shape[:2], 64, 128), dtype=F, device=h.device)
    for t in range(h.shape[1]):
        S = decay * S + k[:, t, :, :, None] * v[:, t, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    return (_rms(o.flatten(2)) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _experts(w, h):
    """The weighted sum of the chosen experts' results; a router output past the real experts returns its input. The choice
    is by score plus correction among the outputs of the best groups, the weights are the plain scores, normalised."""
    n = EXPERTS + IDENTITY
    s = torch.softmax(h @ w("router").T, -1)
    choice = (s + w("correction")).unflatten(-1, (GROUPS, -1))
    best = torch.zeros(choice.shape[:2], dtype=torch.bool, device=h.device).scatter_(1, choice.amax(-1).topk(KEEP, -1).indices, True)
    chosen = choice.masked_fill(~best[..., None], float("-inf")).flatten(1).topk(TOP, -1).indices
    weight = torch.zeros_like(s).scatter_(1, chosen, s.gather(1, chosen))
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = weight[:, EXPERTS:].sum(-1, keepdim=True) * h
    for j in range(EXPERTS):
        at = weight[:, j].nonzero()[:, 0]
        y = h[at]
        out[at] += weight[at, j, None] * ((_silu(y @ w(f"e{j}.gate").T) * (y @ w(f"e{j}.up").T)) @ w(f"e{j}.down").T)
    return out
