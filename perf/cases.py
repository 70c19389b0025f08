"""Performance cases: engine steps (decode, prefill) of the served model families on one GPU.

Every case is a step of the engine over the first eighth of a preset's blocks at their full width, with an eighth of
its vocabulary, so that trunk and output head keep the full model's proportions: `ModelRunner.decode` replaying the
captured decode graph (with its upload and read-back), or `Executor.generate_batch` running prompts up to their first
token (admission, chunked prefill, head, release). The models are the framework's own `DenseModel` / `HybridModel`.

Sublayer inputs are forced. Chained NVFP4 layers turn a rounding difference in one sum into different 4-bit codes a few
kernels later, after which the outputs of two correct implementations are no longer comparable. So every projection
back into the hidden size (a dense layer's o_proj and down, a hybrid sublayer's output) is computed, kept as an output
of the case, and replaced in the residual stream by given rows of the same distribution. The kernels, their order and
their traffic are those of the plain model.

Returned: the logits and tokens, the outputs of every sublayer, the KV pool and the recurrent states.
"""
from __future__ import annotations

import math

import torch

from hibana_b200.engine.executor import Executor
from hibana_b200.engine.request import SamplingParams
from hibana_b200.models.dense import DenseModel
from hibana_b200.models.hybrid import HybridModel
from hibana_b200.target import ATTN, GATED_ATTN, GDN, LATENT_MOE, MAMBA2, MLP, get_target, scaled

DEVICE = "cuda"
PART = 8                      # an eighth of the depth and of the vocabulary
PREFILL_BUDGET = 4096         # tokens of one prefill forward (the engine's default budget)
MAX_TOKENS = 4096             # prompt tokens of a drawn prefill case
KV_TOKENS = 64 * 2048         # cached tokens of a drawn decode case
INPUT_AMAX = 48.0             # normed rows reach about 6, products of gate and up (or squares) about 40
KV_DTYPES = {"bf16": torch.bfloat16, "fp8": torch.float8_e4m3fn}


def listed() -> list:
    return [
        # one chat user on an idle engine: latency per token, bound by launches and the weight stream
        decode("dense-decode-1", "dense-27b", 1, 500),
        # a few users at different points of their conversations, sampling with temperature and nucleus cut
        decode("dense-decode-11-sampled", "dense-27b", 11, 3001, ragged=True, sampled=True),
        # the throughput point of the headline benchmark: 64 sequences past 2048-token prompts
        decode("dense-decode-64", "dense-27b", 64, 2048),
        # long documents with an fp8 cache
        decode("dense-decode-long-fp8", "dense-27b", 2, 30011, kv="fp8"),
        # time to first token of a short chat message: latency and launches
        prefill("dense-prefill-29", "dense-27b", "29"),
        # time to first token of the headline benchmark's prompt
        prefill("dense-prefill-2048", "dense-27b", "2048"),
        # a full prefill budget of mixed prompts, as a busy server packs them
        prefill("dense-prefill-mixed-4096", "dense-27b", "1801,37,640,1,1617"),
        # the hybrid 27B (gated delta rule + gated attention of head dim 256, fp8 cache by default), a few users
        decode("qwen38-decode-4", "qwen38", 4, 5003, kv="fp8", ragged=True),
        prefill("qwen38-prefill-1500", "qwen38", "1237,263", kv="fp8"),
        # the Mamba-2 mixture of experts (fp8 cache by default): one user, and the batch its benchmark runs
        decode("nemotron-decode-1", "nemotron", 1, 900, kv="fp8"),
        decode("nemotron-decode-16", "nemotron", 16, 8192, kv="fp8"),
        # a prompt longer than the prefill chunk: a full chunk and a ragged rest that continues its state
        prefill("nemotron-prefill-5000", "nemotron", "5000", kv="fp8"),
    ]


def decode(name, model, batch, context, kv="bf16", ragged=False, sampled=False) -> dict:
    return {"name": name, "step": "decode", "model": model, "batch": batch, "context": context, "kv": kv,
            "ragged": ragged, "sampled": sampled}


def prefill(name, model, prompts, kv="bf16") -> dict:
    return {"name": name, "step": "prefill", "model": model, "prompts": prompts, "kv": kv}


def _log_uniform(rng, lo, hi) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    """A decode step of 1 to 64 sequences with up to 32k cached tokens each, or a prefill of 8 to 4096 tokens in one
    to six prompts, of any of the three models and both cache formats."""
    model = rng.choice(("dense-27b", "dense-27b", "qwen38", "nemotron"))
    kv = rng.choice(("bf16", "fp8") if model == "dense-27b" else ("fp8", "fp8", "bf16"))
    if rng.random() < 0.55:
        batch = _log_uniform(rng, 1, 64)
        context = _log_uniform(rng, 32, min(32768, KV_TOKENS // batch))
        case = decode("", model, batch, context, kv, rng.random() < 0.5, rng.random() < 0.3)
    else:
        total = _log_uniform(rng, 8, MAX_TOKENS)
        parts = min(rng.choice((1, 1, 2, 3, 4, 6)), total)
        cuts = sorted(rng.sample(range(1, total), parts - 1)) if parts > 1 else []
        lens = [b - a for a, b in zip([0] + cuts, cuts + [total])]
        case = prefill("", model, ",".join(map(str, lens)), kv)
    del case["name"]
    return case


def _target(case):
    t = get_target(case["model"])
    return scaled(t, layers=len(t.layers) // PART, vocab=t.vocab // PART, mtp_layers=0, mtp_depth=0)


def _contexts(case) -> list:
    """Cached tokens per sequence, the new one included."""
    b, c = case["batch"], case["context"]
    return [max(2, int(c * (0.25 + 0.75 * (i + 1) / b))) for i in range(b)] if case["ragged"] else [max(2, c)] * b


def _prompts(case) -> list:
    return [int(n) for n in case["prompts"].split(",")]


class ForcedLinear:
    """A projection back into the hidden size whose result is kept while given rows take its place."""

    def __init__(self, lin, given):
        self._lin, self._given, self.results = lin, given, []

    def __getattr__(self, name):
        return getattr(self._lin, name)

    def __call__(self, x, *args, **kw):
        y = self._lin(x, *args, **kw)
        self.results.append(y)
        return self._given[:y.shape[0]]


class ForcedLayer:
    """The same for a whole sublayer of a hybrid model."""

    def __init__(self, sub, given):
        self._sub, self._given, self.results = sub, given, []

    def __getattr__(self, name):
        return getattr(self._sub, name)

    def forward(self, *args, **kw):
        y = self._sub.forward(*args, **kw)
        self.results.append(y)
        return self._given[:y.shape[0]]


def _force(model, rows, gen) -> list:
    """Puts the wrappers in; returns them."""
    # hidden rows of different tokens point partly the same way, as they do in trained models (less of it where a
    # router has to spread the tokens over its experts)
    common = 0.5 if model.target.experts else 1.0
    model.embed += (0.02 * common * torch.randn(model.target.hidden, generator=gen, device=DEVICE)).to(torch.bfloat16)

    def given():
        x = torch.randn(rows + 1, model.target.hidden, generator=gen, device=DEVICE)
        return (x[1:] + common * x[:1]).to(torch.bfloat16)

    forced = []
    if isinstance(model, DenseModel):
        for layer in model.layers:
            layer.o, layer.down = ForcedLinear(layer.o, given()), ForcedLinear(layer.down, given())
            forced += [layer.o, layer.down]
    else:
        for blk in model.blocks:
            for name in ("mixer", "ffn"):
                if getattr(blk, name) is not None:
                    setattr(blk, name, ForcedLayer(getattr(blk, name), given()))
                    forced.append(getattr(blk, name))
    return forced


class Logits:
    """Keeps what the model's output head returns."""

    def __init__(self, model):
        self._fn, self.results = model.logits, []
        model.logits = self

    def __call__(self, *args, **kw):
        y = self._fn(*args, **kw)
        self.results.append(y)
        return y


def _build(case, seed, max_batch, max_ctx, slots, rows):
    t = _target(case)
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    model = (DenseModel if t.family == "dense" else HybridModel)(t, DEVICE, seed=seed)
    ex = Executor(model, max_batch=max_batch, max_ctx=max(max_ctx, 256), kv_slots=max(slots, 256),
                  radix_cache=False, kv_dtype=KV_DTYPES[case["kv"]])
    for lin in model.linears():        # static activation scales, as a checkpoint brings them: the widest input's range
        if lin.fmt == "nvfp4":
            lin.set_input_amax(INPUT_AMAX)
    return t, gen, model, ex, _force(model, rows, gen), Logits(model)


def prepare(case, seed):
    return _prepare_decode(case, seed) if case["step"] == "decode" else _prepare_prefill(case, seed)


def _prepare_decode(case, seed):
    batch, lens = case["batch"], _contexts(case)
    max_batch = 1 << (batch - 1).bit_length()          # the engine's graph buckets are powers of two
    t, gen, model, ex, forced, logits = _build(case, seed, max_batch, max(lens), sum(lens) + 64, max(max_batch, 16 * batch))
    runner = ex.runner
    rows = [runner.alloc_row() for _ in lens]
    slots = [ex.kv.alloc(n) for n in lens]
    ids = torch.randint(0, t.vocab, (batch, 17), generator=gen, device=DEVICE).tolist()
    states = [ex.state_pool.alloc() for _ in lens] if ex.state_pool is not None else None
    for row, s in zip(rows, slots):
        runner.set_table(row, 0, s)
    # recurrent states of a running sequence: a few tokens through the model from an empty state
    if states is not None:
        for s in states:
            ex.state_pool.zero_slot(s)
        n = [min(16, len(s)) for s in slots]
        runner.forward_rows(rows, [i[:m] for i, m in zip(ids, n)], [0] * batch, [s[:m] for s, m in zip(slots, n)],
                            state_slots=states)
    # cached keys and values with the spread that random-init projections of normed rows give them, half of it an
    # offset per channel
    std = 0.02 * math.sqrt(t.hidden / 2)
    for layer in ex.kv.storage:
        for side in layer:
            for head in side:
                x = torch.randn(head.shape, generator=gen, device=DEVICE)
                head.copy_((x + torch.randn(head.shape[1], generator=gen, device=DEVICE)) * std)
    for f in forced + [logits]:
        f.results.clear()
    sampling = None
    if case["sampled"]:
        sampling = {"temp": [0.8] * batch, "top_k": [0] * batch, "top_p": [0.95] * batch,
                    "seed": [seed + i for i in range(batch)], "offs": [7] * batch}
    runner.capture([max_batch])
    step = (rows, [i[16] for i in ids], [n - 1 for n in lens], [s[-1] for s in slots], sampling, states)
    outputs = [f.results[-1] for f in forced] + [logits.results[-1]]
    return {"step": "decode", "runner": runner, "args": step, "outputs": outputs, "ex": ex, "batch": batch}


def _prepare_prefill(case, seed):
    lens = _prompts(case)
    t, gen, model, ex, forced, logits = _build(case, seed, len(lens), max(lens) + 8, sum(lens) + 64, PREFILL_BUDGET)
    prompts = [torch.randint(0, t.vocab, (n,), generator=gen, device=DEVICE).tolist() for n in lens]
    for f in forced + [logits]:
        f.results.clear()
    return {"step": "prefill", "prompts": prompts, "params": SamplingParams(max_tokens=1, ignore_eos=True), "ex": ex,
            "forced": forced, "logits": logits}


def run(state):
    ex = state["ex"]
    if state["step"] == "decode":
        # the same position on every pass: the step's work stays the same
        tokens = state["runner"].decode(*state["args"])
        rows = state["batch"]
        out = {"tokens": torch.tensor(tokens), "outputs": [o[:rows] for o in state["outputs"]]}
    else:
        for f in state["forced"]:
            f.results.clear()
        state["logits"].results.clear()
        reqs = ex.generate_batch(state["prompts"], state["params"], PREFILL_BUDGET)
        out = {"tokens": torch.tensor([r.output_ids for r in reqs]), "logits": list(state["logits"].results),
               "outputs": [list(f.results) for f in state["forced"]]}
    out["kv"] = ex.kv.storage[:, :, :, 1:]                  # slot 0 is the dummy that padded rows share
    if ex.state_pool is not None:
        out["conv"], out["ssm"] = ex.state_pool.conv[:, 1:], ex.state_pool.ssm[:, 1:]
    return out


def _weights(t, tokens: int) -> tuple:
    """(bytes of the weights that `tokens` tokens read, multiply-adds per token) of the trunk."""
    h, fp4 = t.hidden, 0.5625
    total, macs = 0.0, 0.0
    for mixer, ffn in t.layers:
        n4, n16 = 0, 0
        if mixer in (ATTN, GATED_ATTN):
            q = t.q_heads * t.head_dim
            n4 += h * (q * (2 if mixer == GATED_ATTN else 1) + 2 * t.kv_heads * t.head_dim) + q * h
        elif mixer == MAMBA2:
            n4 += h * (2 * t.mamba_inner + 2 * t.mamba_groups * t.mamba_state + t.mamba_heads) + t.mamba_inner * h
        elif mixer == GDN:
            n4 += h * (t.gdn_conv_dim + t.gdn_v_heads * t.gdn_head_dim) + t.gdn_v_heads * t.gdn_head_dim * h
            n16 += h * 2 * t.gdn_v_heads
        if ffn == MLP:
            n4 += 3 * h * t.ffn
        elif ffn == LATENT_MOE:
            expert = 2 * t.latent * t.expert_ffn
            distinct = t.experts * (1.0 - (1.0 - t.top_k / t.experts) ** tokens)
            n4 += 2 * h * t.shared_ffn
            n16 += h * t.experts + 2 * h * t.latent
            total += distinct * expert * fp4
            macs += t.top_k * expert
        total += n4 * fp4 + n16 * 2
        macs += n4 + n16
    return total, macs


def work(case) -> dict:
    """Weights once, the cached keys and values and the recurrent states read once, everything new written once."""
    t = _target(case)
    kv_tok = t.attn_layers * 2 * t.kv_heads * t.head_dim * (2 if case["kv"] == "bf16" else 1)
    qd = t.attn_layers * t.q_heads * t.head_dim
    if case["step"] == "decode":
        lens = _contexts(case)
        tokens = sampled = len(lens)
        pairs, read = sum(lens), sum(n - 1 for n in lens)
        states = 2 * t.state_bytes_per_slot * len(lens)
    else:
        lens = _prompts(case)
        tokens, sampled = sum(lens), len(lens)
        pairs, read = sum(n * (n + 1) // 2 for n in lens), 0
        states = t.state_bytes_per_slot * len(lens)
    weights, macs = _weights(t, tokens)
    outs = sum((m != "none") + (f != "none") for m, f in t.layers) * tokens * t.hidden * 2
    nbytes = (weights + t.vocab * t.hidden * 2 + read * kv_tok + tokens * kv_tok + states + outs
              + sampled * t.vocab * 4)
    return {"bytes": nbytes, "flops": 2 * macs * tokens + 2 * sampled * t.vocab * t.hidden + 4 * pairs * qd}


def tolerance(case) -> dict:
    """A sublayer quantises to 4 bits behind its attention or its recurrence: where two implementations' bf16 values
    differ in the last bit, some of the codes and block scales differ too. Measured between this repository's attention
    kernels (softmax weights in bf16 or fp32, other tiles and splits): 0.006 to 0.021 of a projection's result, and
    0.024 between the two forms of the delta rule's chunk phase."""
    return {"rel": 0.03, "max": 0.5, "differ": 0.01}
