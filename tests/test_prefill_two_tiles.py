"""Prefill attention with two Q tiles per CTA (csrc/attn_prefill.cu, attn_prefill_q2_kernel) and the rule that chooses it."""
import math

import pytest
import torch

from hibana_b200 import config as cfgmod
from hibana_b200.ops import attention


def test_two_q_tiles_rule_cpu():
    assert attention.two_q_tiles(1, 40, 8, 2048) and attention.two_q_tiles(16, 40, 8, 60)
    assert attention.two_q_tiles(1, 40, 8, 29) and attention.two_q_tiles(1, 40, 8, 225)
    assert not attention.two_q_tiles(1, 40, 8, 250) and not attention.two_q_tiles(1, 40, 8, 450)
    assert attention.two_q_tiles(1, 40, 8, 451) and attention.two_q_tiles(1, 128, 1, 2)
    with cfgmod.using(stable_numerics=True):
        assert not attention.two_q_tiles(1, 40, 8, 2048)


def test_two_q_tiles_rule_looks_at_the_context_cpu():
    """Within half a wave: 192 keys per row on average, whatever the prefix is; beyond one wave any context."""
    assert attention.two_q_tiles(1, 40, 8, 225, 225) and attention.two_q_tiles(1, 40, 8, 150, 256)
    assert not attention.two_q_tiles(1, 40, 8, 100, 256) and not attention.two_q_tiles(4, 40, 8, 50, 1024)
    assert not attention.two_q_tiles(1, 40, 8, 250, 250) and attention.two_q_tiles(1, 40, 8, 451, 16000)


def test_context_bound_reaches_the_rule_cpu(monkeypatch):
    """`max_ctx` of the call, or the width of the block table where the caller gives none."""
    from hibana_b200 import _native as nv
    seen = []

    class Lib:
        def hb_attn_prefill(self, *args):
            seen.append(args[13])
            return 0

    monkeypatch.setattr(nv, "use_native", lambda *t: True)
    monkeypatch.setattr(nv, "lib", Lib)
    monkeypatch.setattr(nv, "stream", lambda: 0)
    monkeypatch.setattr(nv, "device_state", lambda dev: type("S", (), {"status": torch.zeros(1)}))
    monkeypatch.setattr(attention, "_prefill_tensor_cores", lambda *a: True)
    pool = torch.empty(1100, 8, 128, dtype=torch.bfloat16)
    ip = torch.tensor([0, 100], dtype=torch.int32)
    call = lambda width, **kw: attention.paged_attention(  # noqa: E731
        torch.empty(100, 40, 128, dtype=torch.bfloat16), pool, pool, torch.zeros(1, width, dtype=torch.int32),
        torch.tensor([100], dtype=torch.int32), q_indptr=ip, max_rows=100, **kw)
    call(1000), call(200), call(1000, max_ctx=100), call(1000, max_ctx=1000)
    assert seen == [0, 1, 1, 0]


# rows and contexts: one tile, a second tile of one row, both tiles full, a tile more for the second one, prefixes that end on and
# off a tile, sequences with one tile or none of the block's rows
CASES = [([26], [26]), ([50], [50]), ([51], [64]), ([51], [65]), ([100, 1, 27], [128, 1, 192]), ([30, 129, 3], [300, 129, 3]),
         ([77], [1000])]


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,d", [(40, 8, 128), (8, 8, 64), (32, 2, 128), (7, 1, 64), (128, 1, 128)])
@pytest.mark.parametrize("scattered", [False, True])
@pytest.mark.parametrize("causal", [True, False])
def test_two_q_tiles_match_reference(hq, hkv, d, scattered, causal):
    """bf16 weights and a bf16 result: half an ulp each (2^-8) of the largest value that a row averages is an upper bound."""
    from hibana_b200 import _native as nv
    g = hq // hkv
    gen = torch.Generator(device="cuda").manual_seed(hq * d)
    for rows, ctxs in CASES:
        rows = [max(1, r * 5 // g) for r in rows]                   # the same tiles at every group size
        ctxs = [max(r, c) for r, c in zip(rows, ctxs)]
        slots = sum(ctxs) + 65
        st = torch.randn(2, hkv, slots, d, generator=gen, device="cuda").bfloat16()
        k, v = st[0].transpose(0, 1), st[1].transpose(0, 1)
        perm = torch.randperm(slots - 1, generator=gen, device="cuda") if scattered else torch.arange(slots - 1, device="cuda")
        idx = torch.zeros(len(ctxs), max(ctxs), dtype=torch.int32, device="cuda")
        o = 0
        for i, c in enumerate(ctxs):
            idx[i, :c] = perm[o:o + c].int() + 1
            o += c
        indptr = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        q = torch.randn(sum(rows), hq, d, generator=gen, device="cuda").bfloat16() * 2
        ctx = torch.tensor(ctxs, dtype=torch.int32, device="cuda")
        kw = dict(q_indptr=indptr, max_rows=max(rows), scale=1 / math.sqrt(d), causal=causal)
        saved = attention.two_q_tiles
        try:
            attention.two_q_tiles = lambda *a: True
            got = attention.paged_attention(q, k, v, idx, ctx, **kw)
        finally:
            attention.two_q_tiles = saved
        ref = attention.paged_attention_ref(q, k, v, idx, ctx, indptr, 1 / math.sqrt(d), causal=causal).float()
        vmax = v.float().abs().max().item()
        assert (got.float() - ref).abs().max().item() <= 2 * 2.0 ** -8 * vmax, (rows, ctxs)
        assert ((got.float() - ref).norm() / ref.norm()).item() <= 4e-3
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,d", [(40, 8, 128), (8, 8, 64)])
@pytest.mark.parametrize("spread", [1.0, 1.5, 3.0])
def test_two_q_tiles_are_as_close_as_one(hq, hkv, d, spread):
    """2-norm of the error against fp64 of the forms with two and with one Q tile, over 130 thousand outputs and more: rounding alone
    tells two forms apart by some 1e-3 of it."""
    gen = torch.Generator(device="cuda").manual_seed(d)
    rows, g = 600, hq // hkv
    st = torch.randn(2, hkv, rows + 65, d, generator=gen, device="cuda").bfloat16()
    k, v = st[0].transpose(0, 1), st[1].transpose(0, 1)
    q = (torch.randn(rows, hq, d, generator=gen, device="cuda") * spread).bfloat16()
    idx = torch.arange(rows, dtype=torch.int32, device="cuda")[None]
    ctx, indptr = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([rows], [0, rows]))
    hidden = torch.ones(rows, rows, dtype=torch.bool, device="cuda").triu(1)
    ref = torch.empty(rows, hq, d, dtype=torch.float64, device="cuda")
    for h in range(hq):
        s = q[:, h].double() @ k[:rows, h // g].double().t() / math.sqrt(d)
        ref[:, h] = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[:rows, h // g].double()
    err, saved = [], attention.two_q_tiles
    try:
        for two in (False, True):
            attention.two_q_tiles = lambda *a, two=two: two
            y = attention.paged_attention(q, k, v, idx, ctx, q_indptr=indptr, max_rows=rows)
            err.append((y.double() - ref).norm().item())
    finally:
        attention.two_q_tiles = saved
    assert err[1] <= 1.005 * err[0], err
