"""Work that programs have this framework do, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs, weights, caches,
work lists) from a seed, ``run`` is one pass through the framework's entry points, ``exact`` the same numbers in 64 bits
by plain torch.  Kinds:

  serve, prefill   whole model steps at the Qwen2.5-0.5B layer sizes: a batch of requests answered from their
                   prompts, and one long prompt; they return logits
  wkv, hgrn2       the gated linear recurrences of Zazasun's mixers
  ssm              the state-space recurrence of Ratilorn's parallel layers
  delta            Vetevik's gated delta rule
  memory           Zugarax's matrix memory with its gates and norms
  diff             Zazasun's differential attention over the paged cache
  latent           Rozesun's and Zugarax's attention over latents
  sigmoid          Ratilorn's attention with sigmoid weights mixed across heads
  experts          the routed feed-forward of Bopilorn, Ratilorn and Vetevik
  mlp32            a dense gated feed-forward of the 32-bit path (``--dtype float32``)

``size`` picks the layer sizes "896" or "2048" of the benchmarks of the architectures.  ``rows`` lists the rows each
request of the step brings (a prompt portion, or 1 for a decoded token), ``before`` how many tokens each has cached.
"""

from __future__ import annotations

import math
import types

import numpy as np
import torch

from mini_llm_runtime_b200 import ops
from mini_llm_runtime_b200.cache import CacheManager
from mini_llm_runtime_b200.config import Qwen2Config
from mini_llm_runtime_b200.engine import ModelRunner, StepEntry
from mini_llm_runtime_b200.models import build_model
from mini_llm_runtime_b200.ops import AttentionBatch

PAGE = 16
QWEN = dict(vocab_size=151936, hidden_size=896, intermediate_size=4864, num_hidden_layers=24, num_attention_heads=14,
            num_key_value_heads=2, max_position_embeddings=32768, rms_norm_eps=1e-6, rope_theta=1000000.0,
            hidden_act="silu", tie_word_embeddings=True)
SIZES = {
    "wkv": {"896": dict(heads=14, dim=64, vdim=64), "2048": dict(heads=32, dim=64, vdim=64)},
    "hgrn2": {"896": dict(heads=7, dim=128, vdim=128), "2048": dict(heads=16, dim=128, vdim=128)},
    "ssm": {"896": dict(heads=14, vdim=64, n=64), "2048": dict(heads=32, vdim=64, n=128)},
    "delta": {"896": dict(heads=14, kv_heads=7, dim=64, vdim=64), "2048": dict(heads=32, kv_heads=16, dim=128, vdim=64)},
    "memory": {"896": dict(heads=7, dim=128, vdim=128), "2048": dict(heads=16, dim=128, vdim=128)},
    "diff": {"896": dict(heads=7, kv_heads=1, dim=64, vdim=128), "2048": dict(heads=16, kv_heads=4, dim=64, vdim=128)},
    "latent": {"896": dict(heads=14, rank=256, rot=32), "2048": dict(heads=16, rank=512, rot=64)},
    "sigmoid": {"896": dict(heads=14, kv_heads=2, dim=64), "2048": dict(heads=16, kv_heads=4, dim=128)},
    "experts": {"896": dict(width=896, inner=2432, experts=16, top=2), "2048": dict(width=2048, inner=1408, experts=64, top=6)},
    "mlp32": {"896": dict(width=896, ff=4864), "2048": dict(width=2048, ff=8192)},
}
RECURRENT = ("wkv", "hgrn2", "ssm", "delta", "memory")
ATTENTION = ("diff", "latent", "sigmoid")
WINDOW, KEEP_FIRST = 1024, 4
EPS = 1e-6
CAP = 15.0                # of the matrix memory's gates
LAMBDA, DIFF = 0.4, 0.5


# ---------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # eight chats answered together: prompts of mixed lengths in one step, then a dozen decoded tokens each
        dict(name="serve-8", kind="serve", rows="37,512,1,204,96,333,64,150", tokens=12),
        # a long document's prompt in one step, the time to the first token
        dict(name="prefill-2048", kind="prefill", rows="2048"),
        # one prompt portion of the scheduler's budget through a recurrent layer, a new request
        dict(name="wkv-prompt", kind="wkv", size="896", rows="2048", before="0"),
        # several prompts' portions of odd lengths in one step, some of them further portions, beside a decoded row
        dict(name="ssm-ragged", kind="ssm", size="2048", rows="1531,77,1,439", before="0,512,900,0"),
        # one prompt portion through a delta-rule layer
        dict(name="delta-prompt", kind="delta", size="2048", rows="2048", before="0"),
        # two prompts through a matrix-memory layer
        dict(name="memory-prompts", kind="memory", size="896", rows="1300,748", before="0,0"),
        # one prompt portion through windowed differential attention
        dict(name="diff-prompt", kind="diff", size="896", rows="2048", before="0", window=WINDOW),
        # the second portion of a prompt, attending to the first one's latents as well
        dict(name="latent-prompt", kind="latent", size="2048", rows="1024", before="1024", window=0),
        # a decode step of eight requests, windowed layer with sinks
        dict(name="latent-decode", kind="latent", size="2048", rows="1,1,1,1,1,1,1,1",
             before="2047,1990,310,2047,1500,77,1024,2040", window=WINDOW),
        # prompts of mixed lengths through sigmoid attention
        dict(name="sigmoid-prompts", kind="sigmoid", size="2048", rows="1450,401,197", before="0,0,0"),
        # the feed-forward of a full prompt portion
        dict(name="experts-2048", kind="experts", size="2048", rows="2048"),
        # the feed-forward of a step of the 32-bit path
        dict(name="mlp32-600", kind="mlp32", size="896", rows="600"),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _cut(rng, total, most):
    """``total`` rows as the portions of up to ``most`` requests."""
    count = rng.randint(1, max(1, min(most, total)))
    at = sorted(rng.sample(range(1, total), count - 1)) if count > 1 else []
    return [b - a for a, b in zip([0] + at, at + [total])]


def draw(rng):
    kind = rng.choice(("serve", "prefill", "wkv", "hgrn2", "ssm", "delta", "memory", "diff", "latent", "sigmoid",
                       "experts", "mlp32"))
    if kind == "serve":
        count = rng.randint(1, 8)
        return dict(kind=kind, rows=",".join(str(_log_uniform(rng, 1, 300)) for _ in range(count)), tokens=rng.randint(2, 10))
    if kind == "prefill":
        return dict(kind=kind, rows=str(_log_uniform(rng, 64, 3000)))
    size = rng.choice(("896", "2048"))
    if kind == "experts":
        return dict(kind=kind, size=size, rows=str(_log_uniform(rng, 1, 2500)))
    if kind == "mlp32":
        return dict(kind=kind, size=size, rows=str(_log_uniform(rng, 1, 1500)))
    if rng.random() < 0.25:
        rows = [1] * _log_uniform(rng, 1, 32)           # a decode step
        before = [_log_uniform(rng, 1, 3000) for _ in rows]
    else:
        rows = _cut(rng, _log_uniform(rng, 2, 4000), 6)
        before = [rng.choice((0, 0, _log_uniform(rng, 1, 2000))) for _ in rows]
    case = dict(kind=kind, size=size, rows=",".join(map(str, rows)), before=",".join(map(str, before)))
    if kind == "diff":
        case["window"] = WINDOW
    if kind == "latent":
        case["window"] = rng.choice((0, WINDOW))
    return case


def _numbers(case, key):
    return [int(v) for v in str(case[key]).split(",")]


# ---------------------------------------------------------------------------------------------------- inputs
class _Draw:
    """Random tensors on the GPU from a seed."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda")
        self.generator.manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        values = torch.randn(shape, generator=self.generator, device="cuda")
        return values.mul_(std).add_(mean).to(dtype)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(shape, generator=self.generator, device="cuda") * (high - low) + low

    def order(self, count):
        return torch.randperm(count, generator=self.generator, device="cuda")


def _segments(case):
    lengths, before = np.array(_numbers(case, "rows"), np.int32), np.array(_numbers(case, "before"), np.int32)
    starts = np.zeros_like(lengths)
    np.cumsum(lengths[:-1], out=starts[1:])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()      # noqa: E731
    return types.SimpleNamespace(
        seg_q_start=dev(starts), seg_q_len=dev(lengths), seg_pos0=dev(before), seg_slot=dev(np.arange(len(lengths))),
        num_segments=len(lengths), max_q_len=int(lengths.max()), lengths=lengths, positions=before, total=int(lengths.sum()),
        max_kv_len=int((lengths + before).max()))


def _spans(case):
    """(first row, rows, tokens before) of each request."""
    at = 0
    for count, before in zip(_numbers(case, "rows"), _numbers(case, "before")):
        yield at, count, before
        at += count


def _carried(d, ctx, *shape, std):
    """States of the requests: zeros where a request begins, else what earlier tokens left."""
    state = d.normal(ctx.num_segments, *shape, std=std)
    for index, before in enumerate(ctx.positions):
        if before == 0:
            state[index].zero_()
    return state


def _paged(d, ctx, *shapes, dtype=torch.bfloat16):
    """Page pools of the given (heads, entries, std) holding every position, in pages of mixed order, and their table."""
    need = [-(-int(n) // PAGE) for n in ctx.lengths + ctx.positions]
    pages = sum(need)
    order = d.order(pages).to(torch.int32)
    table = torch.full((ctx.num_segments, max(need)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for index, count in enumerate(need):
        table[index, :count] = order[at:at + count]
        at += count
    pools = [d.normal(pages, heads, PAGE, entries, std=std, dtype=dtype) for heads, entries, std in shapes]
    arrays, counts = ops.current().plan_attention(ctx.lengths, ctx.positions)
    arrays = {name: torch.from_numpy(np.ascontiguousarray(value)).cuda() for name, value in arrays.items()}
    batch = AttentionBatch(ctx.seg_q_start, ctx.seg_q_len, ctx.seg_pos0, ctx.seg_slot, table, ctx.num_segments, ctx.max_q_len,
                           ctx.max_kv_len, arrays, counts)
    return pools, batch


def _unit_heads(x, dim):
    """Rows whose heads have a root mean square of one, as normalised queries and keys have."""
    f = x.float()
    f = f.view(*f.shape[:-1], -1, dim)
    return (f / f.square().mean(-1, keepdim=True).sqrt()).reshape(x.shape).to(x.dtype)


def _wkv(case, d):
    s, ctx = SIZES["wkv"][case["size"]], _segments(case)
    inner = s["heads"] * s["dim"]
    r, k, v, gate = (d.normal(ctx.total, inner, std=0.6) for _ in range(4))
    return dict(s, ctx=ctx, r=r, k=k, v=v, gate=gate, raw=d.normal(ctx.total, inner, std=0.3),
                bias=d.uniform(inner, low=-5.0, high=0.5), bonus=d.normal(inner, std=0.3),
                weight=d.normal(inner, std=0.1, mean=1.0), state=_carried(d, ctx, s["heads"], s["dim"], s["vdim"], std=0.7))


def _hgrn2(case, d):
    s, ctx = SIZES["hgrn2"][case["size"]], _segments(case)
    n, values = s["heads"] * s["dim"], s["heads"] * s["vdim"]
    qfv = d.normal(ctx.total, 2 * n + values, std=0.8)        # one product yields all three
    return dict(s, ctx=ctx, q=qfv[:, :n], f=qfv[:, n:2 * n], v=qfv[:, 2 * n:], bias=d.normal(n, std=0.5, mean=1.0),
                lower=d.uniform(n), weight=d.normal(s["vdim"], std=0.1, mean=1.0),
                state=_carried(d, ctx, s["heads"], s["dim"], s["vdim"], std=0.5))


def _ssm(case, d):
    s, ctx = SIZES["ssm"][case["size"]], _segments(case)
    inner, n = s["heads"] * s["vdim"], s["n"]
    mixed = torch.nn.functional.silu(d.normal(ctx.total, inner + 2 * n))          # what the convolution leaves: [x | B | C]
    projected = d.normal(ctx.total, 2 * inner + 2 * n + s["heads"], std=0.5)
    return dict(s, ctx=ctx, x=mixed[:, :inner], B=mixed[:, inner:inner + n], C=mixed[:, inner + n:],
                dt=projected[:, 2 * inner + 2 * n:], dt_bias=d.uniform(s["heads"], low=-4.0, high=0.0),
                A_log=d.uniform(s["heads"], high=2.5), D=d.normal(s["heads"], std=0.1, mean=1.0),
                state=_carried(d, ctx, s["heads"], s["vdim"], n, std=0.5))


def _delta(case, d):
    s, ctx = SIZES["delta"][case["size"]], _segments(case)
    qk, inner, heads = s["kv_heads"] * s["dim"], s["heads"] * s["vdim"], s["heads"]
    mixed = torch.nn.functional.silu(d.normal(ctx.total, 2 * qk + inner))          # [q | k | v] behind their convolutions
    wide = 2 * qk + 2 * inner + 2 * heads
    rows = d.normal(ctx.total, wide + -wide % 8)
    at = 2 * qk + 2 * inner
    return dict(s, ctx=ctx, q=mixed[:, :qk], k=mixed[:, qk:2 * qk], v=mixed[:, 2 * qk:], a=rows[:, at:at + heads],
                b=rows[:, at + heads:at + 2 * heads], dt_bias=d.uniform(heads, low=-4.0, high=0.0),
                A_log=d.uniform(heads, high=2.5), state=_carried(d, ctx, heads, s["vdim"], s["dim"], std=0.3))


def _memory(case, d):
    s, ctx = SIZES["memory"][case["size"]], _segments(case)
    qk, inner, heads = s["heads"] * s["dim"], s["heads"] * s["vdim"], s["heads"]
    wide = 2 * qk + 2 * inner + 2 * heads
    rows = d.normal(ctx.total, wide + -wide % 8, std=0.8)          # one product yields [q | k | v | gate | i | f]
    at = 2 * qk + 2 * inner
    return dict(s, ctx=ctx, q=rows[:, :qk], k=rows[:, qk:2 * qk], v=rows[:, 2 * qk:2 * qk + inner],
                gate=rows[:, 2 * qk + inner:at], i=rows[:, at:at + heads], f=rows[:, at + heads:at + 2 * heads],
                i_bias=d.normal(heads, std=0.5, mean=-1.0), f_bias=d.uniform(heads, low=2.0, high=6.0),
                weight=d.normal(inner, std=0.1, mean=1.0), state=_carried(d, ctx, heads, s["vdim"] + 1, s["dim"], std=0.5),
                maximum=_carried(d, ctx, heads, std=0.5))


def _diff(case, d):
    s, ctx = SIZES["diff"][case["size"]], _segments(case)
    (k_pool, v_pool), batch = _paged(d, ctx, (s["kv_heads"], 2 * s["dim"], 1.0), (s["kv_heads"], s["vdim"], 0.6))
    q = _unit_heads(d.normal(ctx.total, 2 * s["heads"] * s["dim"], dtype=torch.bfloat16), s["dim"])
    return dict(s, batch=batch, q=q, k_pool=_unit_heads(k_pool, s["dim"]), v_pool=v_pool, window=case["window"])


def _latent(case, d):
    s, ctx = SIZES["latent"][case["size"]], _segments(case)
    width = s["rank"] + s["rot"]
    (pool,), batch = _paged(d, ctx, (1, width, 1.0))
    q = d.normal(ctx.total, s["heads"] * width, std=0.5, dtype=torch.bfloat16)
    return dict(s, batch=batch, q=q, pool=pool, window=case["window"], scale=0.08,
                sink=d.normal(s["heads"], std=0.5) if case["window"] else None)


def _sigmoid(case, d):
    s, ctx = SIZES["sigmoid"][case["size"]], _segments(case)
    heads, dim = s["heads"], s["dim"]
    (k_pool, v_pool), batch = _paged(d, ctx, (s["kv_heads"], dim, 1.0), (s["kv_heads"], dim, 0.6))
    q = _unit_heads(d.normal(ctx.total, heads * dim, dtype=torch.bfloat16), dim)
    talk = torch.eye(heads, device="cuda") + d.normal(heads, heads, std=0.1)
    return dict(s, batch=batch, q=q, k_pool=_unit_heads(k_pool, dim), v_pool=v_pool, r1=d.uniform(heads), r2=d.uniform(heads),
                bias=d.normal(heads, std=0.3), talk=talk)


def _experts(case, d):
    s, rows = SIZES["experts"][case["size"]], int(case["rows"])
    scores = torch.softmax(d.normal(rows, s["experts"]), dim=1)
    weights, chosen = torch.topk(scores, s["top"], dim=1)
    gate_up = d.normal(s["experts"], 2 * s["inner"], s["width"], std=0.03, dtype=torch.bfloat16)
    down = d.normal(s["experts"], s["width"], s["inner"], std=0.03, dtype=torch.bfloat16)
    return dict(s, x=d.normal(rows, s["width"], dtype=torch.bfloat16), chosen=chosen.int().contiguous(),
                weights=weights.contiguous(), gate_up=gate_up, down=down, block=64)


def _mlp32(case, d):
    s, rows = SIZES["mlp32"][case["size"]], int(case["rows"])
    return dict(s, x=d.normal(rows, s["width"]), gate_up=d.normal(2 * s["ff"], s["width"], std=0.03),
                down=d.normal(s["width"], s["ff"], std=0.03), block=64)


def _qwen_tensors(d):
    h, i, v = QWEN["hidden_size"], QWEN["intermediate_size"], QWEN["vocab_size"]
    kv = QWEN["num_key_value_heads"] * (h // QWEN["num_attention_heads"])
    matrix = lambda *shape: d.normal(*shape, std=0.02, dtype=torch.bfloat16)      # noqa: E731
    out = {"model.embed_tokens.weight": matrix(v, h), "model.norm.weight": d.normal(h, std=0.02, mean=1.0, dtype=torch.bfloat16)}
    for layer in range(QWEN["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        for name, rows in (("q", h), ("k", kv), ("v", kv)):
            out[p + f"self_attn.{name}_proj.weight"] = matrix(rows, h)
            out[p + f"self_attn.{name}_proj.bias"] = matrix(rows)
        out[p + "self_attn.o_proj.weight"] = matrix(h, h)
        out[p + "mlp.gate_proj.weight"], out[p + "mlp.up_proj.weight"] = matrix(i, h), matrix(i, h)
        out[p + "mlp.down_proj.weight"] = matrix(h, i)
        for name in ("input_layernorm", "post_attention_layernorm"):
            out[p + name + ".weight"] = d.normal(h, std=0.02, mean=1.0, dtype=torch.bfloat16)
    return out


def _token_lists(case, d):
    """Each request's prompt and the tokens that follow it."""
    extra = int(case.get("tokens", 0))
    return [torch.randint(0, QWEN["vocab_size"], (count + extra,), generator=d.generator, device="cuda").tolist()
            for count in _numbers(case, "rows")]


def _model(case, d):
    model = build_model(Qwen2Config(**QWEN), torch.bfloat16).load(_qwen_tensors(d), "cuda:0")
    tokens = _token_lists(case, d)
    longest = max(len(t) for t in tokens)
    cache = CacheManager(model.cache_needs(), page_size=PAGE, num_pages=sum(-(-len(t) // PAGE) for t in tokens),
                         max_requests=len(tokens), max_tokens_per_request=longest, dtype=torch.bfloat16, device="cuda:0",
                         max_step_tokens=max(4096, longest))
    prompts = [np.asarray(t[:n], dtype=np.int32) for t, n in zip(tokens, _numbers(case, "rows"))]
    follow = [t[n:] for t, n in zip(tokens, _numbers(case, "rows"))]
    return dict(runner=ModelRunner(model, cache), prompts=prompts, follow=follow)


_PREPARE = dict(serve=_model, prefill=_model, wkv=_wkv, hgrn2=_hgrn2, ssm=_ssm, delta=_delta, memory=_memory, diff=_diff,
                latent=_latent, sigmoid=_sigmoid, experts=_experts, mlp32=_mlp32)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, _Draw(seed)), kind=case["kind"])


# ---------------------------------------------------------------------------------------------------- one pass
def _answer(s):
    """Requests from their prompts to the last decoded token; the logits of every step."""
    runner, ids = s["runner"], [f"r{i}" for i in range(len(s["prompts"]))]
    for rid in ids:
        runner.cache.create_request(rid)
    logits = [runner.step([StepEntry(rid, prompt, [len(prompt) - 1]) for rid, prompt in zip(ids, s["prompts"])])]
    for step in range(len(s["follow"][0])):
        logits.append(runner.step([StepEntry(rid, [more[step]], [0]) for rid, more in zip(ids, s["follow"])]))
    for rid in ids:
        runner.cache.release(rid)
    return logits


def run(s):
    k, kind, bf16 = ops.current(), s["kind"], torch.bfloat16
    if kind in ("serve", "prefill"):
        return _answer(s)
    if kind == "wkv":
        out = k.bonus_recurrence(s["r"], s["k"], s["v"], s["raw"], s["gate"], s["bias"], s["bonus"], s["weight"], EPS,
                                 s["state"], s["ctx"], s["heads"], s["dim"], bf16)
        return [out, s["state"]]
    if kind == "hgrn2":
        out = k.forget_gate_recurrence(s["q"], s["f"], s["v"], s["bias"], s["lower"], s["weight"], EPS, s["state"], s["ctx"],
                                       s["heads"], s["dim"], s["vdim"], bf16)
        return [out, s["state"]]
    if kind == "ssm":
        out = k.state_space_scan(s["x"], s["B"], s["C"], s["dt"], s["dt_bias"], s["A_log"], s["D"], s["state"], s["ctx"],
                                 s["heads"], s["vdim"], s["n"], 1)
        return [out, s["state"]]
    if kind == "delta":
        out = k.delta_rule_scan(s["q"], s["k"], s["v"], s["a"], s["b"], s["dt_bias"], s["A_log"], s["state"], s["ctx"],
                                s["heads"], s["kv_heads"], s["dim"], s["vdim"], EPS)
        return [out, s["state"]]
    if kind == "memory":
        out = k.matrix_memory(s["q"], s["k"], s["v"], s["i"], s["f"], s["i_bias"], s["f_bias"], CAP, EPS, s["gate"], s["weight"],
                              EPS, s["state"], s["maximum"], s["ctx"], s["heads"], s["dim"], s["vdim"], bf16)
        return [out, s["state"], s["maximum"]]
    if kind == "diff":
        return k.differential_attention(s["q"], s["k_pool"], s["v_pool"], s["batch"], s["heads"], s["kv_heads"], s["dim"],
                                        s["vdim"], s["dim"] ** -0.5, s["window"], KEEP_FIRST, LAMBDA, EPS, 1.0 - DIFF)
    if kind == "latent":
        return k.latent_attention(s["q"], s["pool"], s["batch"], s["heads"], s["rank"], s["rot"], s["scale"], s["window"],
                                  s["sink"])
    if kind == "sigmoid":
        return k.sigmoid_attention(s["q"], s["k_pool"], s["v_pool"], s["batch"], s["heads"], s["kv_heads"], s["dim"], s["dim"],
                                   s["dim"] ** -0.5, distance=(s["r1"], s["r2"]), score_bias=s["bias"], head_mix=s["talk"])
    if kind == "experts":
        return k.routed_experts(s["x"], s["chosen"], s["weights"], s["gate_up"], s["down"], s["block"])
    hidden = k.linear_swiglu(s["x"], s["gate_up"], s["block"])
    return k.linear(hidden, s["down"])


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _pairs(case, window, keep):
    """(query, key) pairs that see each other, and the keys that some query of its request sees."""
    pairs = keys = 0
    for _, count, before in _spans(case):
        if window:
            pairs += sum(min(p + 1, window + min(keep, max(0, p + 1 - window))) for p in range(before, before + count))
            keys += min(before + count, window + count + keep)
        else:
            pairs += count * before + count * (count + 1) // 2
            keys += before + count
    return pairs, keys


def work(case):
    kind, rows = case["kind"], _numbers(case, "rows")
    total = sum(rows)
    if kind in ("serve", "prefill"):
        h, i, v, layers = QWEN["hidden_size"], QWEN["intermediate_size"], QWEN["vocab_size"], QWEN["num_hidden_layers"]
        kv = 2 * QWEN["num_key_value_heads"] * (h // QWEN["num_attention_heads"])
        per_layer = h * (h + kv) + h * h + 3 * h * i
        extra = int(case.get("tokens", 0))
        tokens, steps = total + extra * len(rows), 1 + extra
        pairs = sum((n + extra) * (n + extra + 1) // 2 for n in rows)
        read = sum(n * extra + extra * (extra + 1) // 2 for n in rows)
        return {"bytes": steps * 2 * (layers * per_layer + v * h) + (tokens + read) * layers * kv * 2 + steps * len(rows) * v * 4,
                "flops": 2 * tokens * layers * per_layer + 2 * steps * len(rows) * v * h + 4 * pairs * layers * h}
    s = SIZES[kind][case["size"]]
    if kind == "experts":
        used = min(s["experts"], round(s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** total)))
        matrices = 3 * s["inner"] * s["width"]
        return {"bytes": 2 * used * matrices + total * (s["width"] * 6 + s["top"] * 8), "flops": 2 * total * s["top"] * matrices}
    if kind == "mlp32":
        matrices = 3 * s["ff"] * s["width"]
        return {"bytes": 4 * matrices + 8 * total * s["width"], "flops": 2 * total * matrices}
    heads, requests = s["heads"], len(rows)
    if kind in ("wkv", "hgrn2"):
        cells, inputs = heads * s["dim"] * s["vdim"], heads * (5 * s["dim"] if kind == "wkv" else 2 * s["dim"] + s["vdim"])
        return {"bytes": total * (4 * inputs + 2 * heads * s["vdim"]) + 8 * requests * cells, "flops": 5 * total * cells}
    if kind == "ssm":
        cells = heads * s["vdim"] * s["n"]
        return {"bytes": 4 * total * (2 * heads * s["vdim"] + 2 * s["n"] + heads) + 8 * requests * cells, "flops": 5 * total * cells}
    if kind == "delta":
        cells = heads * s["vdim"] * s["dim"]
        return {"bytes": 4 * total * (2 * s["kv_heads"] * s["dim"] + 2 * heads * s["vdim"] + 2 * heads) + 8 * requests * cells,
                "flops": 7 * total * cells}
    if kind == "memory":
        cells = heads * (s["vdim"] + 1) * s["dim"]
        return {"bytes": total * (8 * heads * s["dim"] + 10 * heads * s["vdim"] + 8 * heads) + 8 * requests * cells,
                "flops": 5 * total * cells}
    pairs, keys = _pairs(case, case.get("window", 0), KEEP_FIRST if kind == "diff" else 0)
    if kind == "diff":
        return {"bytes": 2 * keys * s["kv_heads"] * (2 * s["dim"] + s["vdim"]) + 2 * total * heads * (2 * s["dim"] + s["vdim"]),
                "flops": 4 * pairs * heads * (s["dim"] + s["vdim"])}
    if kind == "latent":
        width = s["rank"] + s["rot"]
        return {"bytes": 2 * keys * width + total * heads * (2 * width + 4 * s["rank"]),
                "flops": 2 * pairs * heads * (width + s["rank"])}
    return {"bytes": 4 * keys * s["kv_heads"] * s["dim"] + 4 * total * heads * s["dim"],
            "flops": pairs * heads * (4 * s["dim"] + 2 * heads)}


# ---------------------------------------------------------------------------------------------------- 64-bit answers
def _d(x):
    return x.double()


def _rms(x):
    return (x.square().mean(-1, keepdim=True) + EPS).sqrt()


def _walk(case, state, token):
    """Advance every request's state token by token; ``token(index, row, S)`` returns (the new S, the row's result)."""
    rows, states = [], []
    for index, (first, count, _) in enumerate(_spans(case)):
        S = _d(state[index])
        for row in range(first, first + count):
            S, out = token(index, row, S)
            rows.append(out)
        states.append(S)
    return torch.stack(rows), torch.stack(states)


def _exact_gated(case, s):
    heads, dim, vdim = s["heads"], s["dim"], s["vdim"]
    per_head = lambda x, n: _d(x).reshape(-1, heads, n)      # noqa: E731
    v = per_head(s["v"], vdim)
    if case["kind"] == "wkv":
        r, b = per_head(s["r"], dim), per_head(s["k"], dim)
        a = per_head(torch.exp(-torch.exp(_d(s["raw"]) + _d(s["bias"]))), dim)
        bonus = _d(s["bonus"]).view(heads, dim)
        weight, gate = _d(s["weight"]).view(heads, vdim), per_head(torch.nn.functional.silu(_d(s["gate"])), vdim)
    else:
        lower = _d(s["lower"])
        a = per_head(lower + (1 - lower) * torch.sigmoid(_d(s["f"]) + _d(s["bias"])), dim)
        r, b = per_head(torch.nn.functional.silu(_d(s["q"])), dim), 1 - a
        weight, gate = _d(s["weight"]), 1.0

    def token(_, row, S):
        written = b[row][:, :, None] * v[row][:, None, :]
        if case["kind"] == "wkv":
            out = torch.einsum("hi,hij->hj", r[row], S + bonus[:, :, None] * written)
            return a[row][:, :, None] * S + written, out
        S = a[row][:, :, None] * S + written
        return S, torch.einsum("hi,hij->hj", r[row], S)

    o, state = _walk(case, s["state"], token)
    return [(o / _rms(o) * weight * gate).flatten(1), state]


def _exact_ssm(case, s):
    heads, vdim, n = s["heads"], s["vdim"], s["n"]
    dt = torch.nn.functional.softplus(_d(s["dt"]) + _d(s["dt_bias"]))
    decay = torch.exp(-torch.exp(_d(s["A_log"])) * dt)
    x, B, C, D = _d(s["x"]).reshape(-1, heads, vdim), _d(s["B"]), _d(s["C"]), _d(s["D"])

    def token(_, row, S):
        S = decay[row][:, None, None] * S + (dt[row][:, None] * x[row])[:, :, None] * B[row]
        return S, S @ C[row] + D[:, None] * x[row]

    y, state = _walk(case, s["state"], token)
    return [y.flatten(1), state]


def _exact_delta(case, s):
    heads, kv, dim, vdim = s["heads"], s["kv_heads"], s["dim"], s["vdim"]
    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + EPS).sqrt()      # noqa: E731
    spread = lambda x: unit(_d(x).reshape(-1, kv, dim)).repeat_interleave(heads // kv, dim=1)      # noqa: E731
    q, k, v = spread(s["q"]) * dim ** -0.5, spread(s["k"]), _d(s["v"]).reshape(-1, heads, vdim)
    g = torch.exp(-torch.exp(_d(s["A_log"])) * torch.nn.functional.softplus(_d(s["a"]) + _d(s["dt_bias"])))
    beta = torch.sigmoid(_d(s["b"]))

    def token(_, row, S):
        S = g[row][:, None, None] * S
        u = beta[row][:, None] * (v[row] - torch.einsum("hji,hi->hj", S, k[row]))
        S = S + u[:, :, None] * k[row][:, None, :]
        return S, torch.einsum("hji,hi->hj", S, q[row])

    y, state = _walk(case, s["state"], token)
    return [y.flatten(1), state]


def _exact_memory(case, s):
    heads, dim, vdim = s["heads"], s["dim"], s["vdim"]
    capped = lambda raw, bias: CAP * torch.tanh((_d(raw) + _d(bias)) / CAP)      # noqa: E731
    i, f = capped(s["i"], s["i_bias"]), torch.nn.functional.logsigmoid(capped(s["f"], s["f_bias"]))
    q, k = _d(s["q"]).reshape(-1, heads, dim) * dim ** -0.5, _d(s["k"]).reshape(-1, heads, dim)
    v = torch.cat([_d(s["v"]).reshape(-1, heads, vdim), torch.ones(q.shape[0], heads, 1, dtype=torch.float64, device="cuda")], 2)
    m = [_d(row) for row in s["maximum"]]

    def token(index, row, S):
        new = torch.maximum(f[row] + m[index], i[row])
        keep, write = torch.exp(f[row] + m[index] - new), torch.exp(i[row] - new)
        m[index] = new
        S = keep[:, None, None] * S + (write[:, None] * v[row])[:, :, None] * k[row][:, None, :]
        read = torch.einsum("hji,hi->hj", S, q[row])
        return S, read[:, :vdim] / (torch.maximum(read[:, vdim:].abs(), torch.exp(-new)[:, None]) + EPS)

    o, state = _walk(case, s["state"], token)
    gate = torch.sigmoid(_d(s["gate"]).reshape(-1, heads, vdim))
    return [(o / _rms(o) * _d(s["weight"]).view(heads, vdim) * gate).flatten(1), state, torch.stack(m)]


def _cached(pool, batch, index, count):
    """[heads, positions, entries] of one request's cached rows."""
    pages = pool[batch.block_table[index, :-(-count // PAGE)].long()]
    return _d(pages.permute(1, 0, 2, 3).reshape(pool.shape[1], -1, pool.shape[3])[:, :count])


def _visible(count, before, window, keep):
    i = torch.arange(before, before + count, device="cuda")[:, None]
    j = torch.arange(before + count, device="cuda")[None, :]
    seen = j <= i
    return seen & ((i - j < window) | (j < keep)) if window else seen


def _exact_diff(case, s):
    heads, dim, vdim, out = s["heads"], s["dim"], s["vdim"], []
    for index, (first, count, before) in enumerate(_spans(case)):
        keys, values = _cached(s["k_pool"], s["batch"], index, before + count), _cached(s["v_pool"], s["batch"], index, before + count)
        hidden = ~_visible(count, before, s["window"], KEEP_FIRST)
        q = _d(s["q"][first:first + count]).view(count, heads, 2, dim)
        rows = []
        for head in range(heads):
            kv = head // (heads // s["kv_heads"])
            maps = []
            for part in range(2):
                score = q[:, head, part] @ keys[kv][:, part * dim:(part + 1) * dim].T * dim ** -0.5
                maps.append(torch.softmax(score.masked_fill(hidden, -math.inf), 1) @ values[kv])
            o = maps[0] - LAMBDA * maps[1]
            rows.append(o / _rms(o) * (1.0 - DIFF))
        out.append(torch.cat(rows, 1))
    return torch.cat(out)


def _exact_latent(case, s):
    heads, rank, width, out = s["heads"], s["rank"], s["rank"] + s["rot"], []
    for index, (first, count, before) in enumerate(_spans(case)):
        keys = _cached(s["pool"], s["batch"], index, before + count)[0]
        hidden = ~_visible(count, before, s["window"], 0)
        q = _d(s["q"][first:first + count]).view(count, heads, width)
        rows = []
        for head in range(heads):
            score = (q[:, head] @ keys.T * s["scale"]).masked_fill(hidden, -math.inf)
            total = torch.logsumexp(score, 1, keepdim=True)
            if s["sink"] is not None:
                total = torch.logaddexp(total, _d(s["sink"][head]))
            rows.append(torch.exp(score - total) @ keys[:, :rank])
        out.append(torch.cat(rows, 1))
    return torch.cat(out)


def _exact_sigmoid(case, s):
    heads, dim, out = s["heads"], s["dim"], []
    group = heads // s["kv_heads"]
    for index, (first, count, before) in enumerate(_spans(case)):
        keys, values = _cached(s["k_pool"], s["batch"], index, before + count), _cached(s["v_pool"], s["batch"], index, before + count)
        for at in range(0, count, 256):
            part = min(256, count - at)
            q = _d(s["q"][first + at:first + at + part]).view(part, heads, dim)
            far = (torch.arange(before + at, before + at + part, device="cuda")[:, None]
                   - torch.arange(before + count, device="cuda")[None, :])
            seen = far >= 0
            distance = torch.log1p(_d(s["r2"])[:, None, None] * far.clamp_min(0))
            score = torch.einsum("rhd,hkd->hrk", q, keys.repeat_interleave(group, 0)) * dim ** -0.5
            w = torch.sigmoid(score - _d(s["r1"])[:, None, None] * distance + _d(s["bias"])[:, None, None]) * seen
            mixed = torch.einsum("hg,grk->hrk", _d(s["talk"]), w)
            out.append(torch.einsum("hrk,hkd->rhd", mixed, values.repeat_interleave(group, 0)).flatten(1))
    return torch.cat(out)


def _gate_up(both, block):
    both = both.view(both.shape[0], -1, 2, block)
    return (torch.nn.functional.silu(both[:, :, 0]) * both[:, :, 1]).flatten(1)


def _exact_experts(case, s):
    out = torch.zeros(s["x"].shape[0], s["width"], dtype=torch.float64, device="cuda")
    for expert in range(s["experts"]):
        row, place = torch.nonzero(s["chosen"] == expert, as_tuple=True)
        if row.numel():
            hidden = _gate_up(_d(s["x"][row]) @ _d(s["gate_up"][expert]).T, s["block"])
            out.index_add_(0, row, hidden @ _d(s["down"][expert]).T * _d(s["weights"][row, place])[:, None])
    return out


def _exact_mlp32(case, s):
    return _gate_up(_d(s["x"]) @ _d(s["gate_up"]).T, s["block"]) @ _d(s["down"]).T


def _exact_model(case, seed):
    d = _Draw(seed)
    w = _qwen_tensors(d)
    tokens = _token_lists(case, d)
    h, heads, kv_heads = QWEN["hidden_size"], QWEN["num_attention_heads"], QWEN["num_key_value_heads"]
    dim, eps = h // heads, QWEN["rms_norm_eps"]
    norm = lambda x, name: x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * _d(w[name])      # noqa: E731
    lengths = _numbers(case, "rows")
    flat = torch.tensor([t for some in tokens for t in some], device="cuda")
    x = _d(w["model.embed_tokens.weight"][flat])
    freq = QWEN["rope_theta"] ** (-torch.arange(0, dim, 2, dtype=torch.float64, device="cuda") / dim)
    positions = torch.cat([torch.arange(len(t), device="cuda") for t in tokens]).double()
    cos, sin = torch.cos(positions[:, None] * freq)[:, None], torch.sin(positions[:, None] * freq)[:, None]

    def turn(y):
        a, b = y[..., :dim // 2], y[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for layer in range(QWEN["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        y = norm(x, p + "input_layernorm.weight")
        q, k, v = ((y @ _d(w[p + f"self_attn.{n}_proj.weight"]).T + _d(w[p + f"self_attn.{n}_proj.bias"])).view(len(y), -1, dim)
                   for n in "qkv")
        q, k = turn(q), turn(k)
        mixed, at = [], 0
        for t in tokens:
            rows = slice(at, at + len(t))
            at += len(t)
            K, V = (z[rows].repeat_interleave(heads // kv_heads, 1).transpose(0, 1) for z in (k, v))
            score = q[rows].transpose(0, 1) @ K.transpose(1, 2) * dim ** -0.5
            hidden = torch.ones(len(t), len(t), dtype=torch.bool, device="cuda").triu(1)
            mixed.append((torch.softmax(score.masked_fill(hidden, -math.inf), -1) @ V).transpose(0, 1).flatten(1))
        x = x + torch.cat(mixed) @ _d(w[p + "self_attn.o_proj.weight"]).T
        y = norm(x, p + "post_attention_layernorm.weight")
        y = torch.nn.functional.silu(y @ _d(w[p + "mlp.gate_proj.weight"]).T) * (y @ _d(w[p + "mlp.up_proj.weight"]).T)
        x = x + y @ _d(w[p + "mlp.down_proj.weight"]).T
    x = norm(x, "model.norm.weight")
    starts = np.cumsum([0] + [len(t) for t in tokens])[:-1]
    head = _d(w["model.embed_tokens.weight"])
    return [x[torch.tensor([int(a) + n - 1 + step for a, n in zip(starts, lengths)], device="cuda")] @ head.T
            for step in range(1 + int(case.get("tokens", 0)))]


_EXACT = dict(wkv=_exact_gated, hgrn2=_exact_gated, ssm=_exact_ssm, delta=_exact_delta, memory=_exact_memory, diff=_exact_diff,
              latent=_exact_latent, sigmoid=_exact_sigmoid, experts=_exact_experts, mlp32=_exact_mlp32)


def exact(case, seed):
    if case["kind"] in ("serve", "prefill"):
        return _exact_model(case, seed)
    return _EXACT[case["kind"]](case, prepare(case, seed))


# About four times what the results of the listed and of some thirty drawn cases differ from the 64-bit answers by.  Results
# in bfloat16 set the figures of most kinds; serve and prefill go through 24 layers of them.
_TOLERANCE = {
    "serve": {"rel": 8e-2, "max": 0.4}, "prefill": {"rel": 8e-2, "max": 0.4},
    "wkv": {"rel": 7e-3, "max": 1.6e-2}, "hgrn2": {"rel": 7e-3, "max": 1.6e-2},
    "ssm": {"rel": 1e-6, "max": 1e-5}, "delta": {"rel": 1e-6, "max": 1e-5},
    "memory": {"rel": 1.4e-2, "max": 0.28},
    "diff": {"rel": 1e-2, "max": 5e-2}, "latent": {"rel": 5e-3, "max": 8e-2}, "sigmoid": {"rel": 1e-2, "max": 7e-2},
    "experts": {"rel": 7e-3, "max": 6e-2}, "mlp32": {"rel": 6e-6, "max": 4e-5},
}


def tolerance(case):
    return dict(_TOLERANCE[case["kind"]])
