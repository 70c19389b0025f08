"""MoE routing and grouped expert GEMMs against plain-PyTorch references; EP ranges sum to the whole."""
import pytest
import torch

from hibana_b200.ops import moe


def test_route_ref_properties_cpu():
    lg = torch.randn(7, 16)
    ids, w = moe.route(lg, 4)
    assert ids.shape == (7, 4) and torch.allclose(w.sum(-1), torch.ones(7), atol=1e-5)
    top = torch.topk(torch.softmax(lg, -1), 4).indices
    assert torch.equal(ids.long().sort(-1).values, top.sort(-1).values)
    ids2, w2 = moe.route(lg, 3, sigmoid=True, sel_bias=torch.zeros(16), scale=2.5)
    assert torch.allclose(w2.sum(-1), torch.full((7,), 2.5), atol=1e-4)


def _weights(e, h, inter, act, fmt, dev, seed=0):
    g = torch.Generator().manual_seed(seed)
    n1 = 2 * inter if act == "swiglu" else inter
    fc1 = torch.randn(e, n1, h, generator=g) * 0.05
    fc2 = torch.randn(e, h, inter, generator=g) * 0.05
    return moe.ExpertWeights.create(fc1.to(dev), fc2.to(dev), act, fmt, in_amax=5.0, mid_amax=2.0)


def test_experts_ref_ep_halves_sum_cpu():
    ew = _weights(8, 64, 128, "swiglu", "bf16", "cpu")
    x = torch.randn(5, 64).bfloat16()
    ids, w = moe.route(torch.randn(5, 8), 2)
    whole = moe.experts_forward(x, ids, w, ew).float()
    parts = sum(moe.experts_forward(x, ids, w, ew, e_lo=lo, e_n=4).float() for lo in (0, 4))
    assert (whole - parts).abs().max() < 2e-2 * whole.abs().max() + 1e-3
    # a rank that keeps only experts 4..7 (global ids, local weights) computes the same partial sum
    kept = moe.experts_forward(x, ids, w, ew.slice(4, 4), id_base=4).float()
    assert torch.equal(kept, moe.experts_forward(x, ids, w, ew, e_lo=4, e_n=4).float())


@pytest.mark.gpu
@pytest.mark.parametrize("e,k,sig", [(8, 2, False), (512, 10, False), (512, 22, True), (60, 6, True)])
def test_route_gpu(e, k, sig):
    lg = torch.randn(33, e)
    bias = torch.randn(e) * 0.1 if sig else None
    ids, w = moe.route(lg, k, sigmoid=sig, sel_bias=bias, scale=1.7)
    ids_g, w_g = moe.route(lg.cuda(), k, sigmoid=sig, sel_bias=None if bias is None else bias.cuda(), scale=1.7)
    assert torch.equal(ids_g.cpu(), ids)
    assert torch.allclose(w_g.cpu(), w, atol=1e-5, rtol=1e-4)
    if sig:
        # many exactly equal scores around the k-th place: equal scores go to the lower expert index, in both the
        # one-CTA-per-token form (few tokens) and the one-warp-per-token form (many)
        for tokens in (7, 300):
            coarse = (torch.randn(tokens, e) * 2).round() / 2
            ids, w = moe.route(coarse, k, sigmoid=True, scale=1.0)
            ids_g, w_g = moe.route(coarse.cuda(), k, sigmoid=True, scale=1.0)
            assert torch.equal(ids_g.cpu(), ids)
            assert torch.allclose(w_g.cpu(), w, atol=1e-5, rtol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4", "w3"])
@pytest.mark.parametrize("t,e,k,h,inter,act", [(4, 8, 2, 256, 512, "swiglu"), (37, 16, 4, 256, 128, "relu2"),
                                               (300, 8, 2, 128, 256, "swiglu")])
def test_experts_forward_gpu(fmt, t, e, k, h, inter, act):
    ew = _weights(e, h, inter, act, fmt, "cpu", seed=1)
    g = torch.Generator().manual_seed(2)
    x = torch.randn(t, h, generator=g).bfloat16()
    ids, w = moe.route(torch.randn(t, e, generator=g), k)
    shared = torch.randn(t, h, generator=g).bfloat16()
    ref = moe.experts_forward(x, ids, w, ew, shared=shared).float()
    ewg = ew.to("cuda")
    got = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg, shared=shared.cuda()).float().cpu()
    tol = 3e-2 if fmt == "bf16" else 6e-2
    assert (got - ref).abs().max() <= tol * ref.abs().max() + 2e-3, (got - ref).abs().max()
    # expert-parallel ranges produce partial sums that add up to the whole
    lo = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg, e_lo=0, e_n=e // 2).float()
    hi = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg, e_lo=e // 2, e_n=e // 2).float()
    whole = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg).float()
    assert (lo + hi - whole).abs().max() <= 2e-2 * whole.abs().max() + 2e-3
    if fmt != "w3":    # a rank holding only the upper half of the experts: same partial sum from global ids
        kept = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg.slice(e // 2, e // 2), id_base=e // 2).float()
        assert torch.equal(kept, hi)
    # deterministic
    again = moe.experts_forward(x.cuda(), ids.cuda(), w.cuda(), ewg).float()
    assert torch.equal(again, whole)
    from hibana_b200 import _native as nv
    assert nv.read_status() == 0


def _share_case(seed=0, rows=12, e=64, k=6):
    g = torch.Generator().manual_seed(seed)
    ids, w = moe.route(torch.randn(rows, e, generator=g) * 2, k, sigmoid=True, scale=2.5)
    return ids, w


def test_expert_sharing_keeps_the_budget_and_the_guaranteed_choices_cpu():
    ids, w = _share_case()
    e, k, keep, budget = 64, 6, 2, 30
    assert len(set(ids.flatten().tolist())) > budget
    ids2, w2 = moe.share_experts(ids, w, e, keep, budget, scale=2.5)
    used = {int(ids2[r, j]) for r in range(ids.shape[0]) for j in range(k) if float(w2[r, j]) > 0}
    core = {int(x) for x in ids[:, :keep].flatten()}
    assert core <= used and len(used) <= max(budget, len(core))
    for r in range(ids.shape[0]):
        assert ids2[r, :keep].tolist() == ids[r, :keep].tolist()            # every row keeps its best choices
        live = w2[r] > 0
        assert abs(float(w2[r][live].sum()) - 2.5) < 1e-5                    # renormalised, router scale kept
        kept = [int(x) for x in ids2[r][live]]
        assert kept == [int(x) for x in ids[r] if int(x) in kept]            # rank order preserved
        assert all(int(x) == int(ids[r, 0]) for x in ids2[r][~live])         # lost slots: best expert, weight 0
    # a budget that covers everything changes nothing but the renormalisation
    ids3, w3 = moe.share_experts(ids, w, e, keep, 64, scale=2.5)
    assert torch.equal(ids3, ids) and torch.allclose(w3, w, atol=1e-6)


@pytest.mark.gpu
def test_expert_sharing_kernel_matches_reference():
    for seed, rows, e, k, keep, budget in ((0, 12, 64, 6, 2, 20), (1, 16, 512, 22, 4, 128), (2, 3, 512, 10, 1, 8)):
        ids, w = _share_case(seed, rows, e, k)
        want_i, want_w = moe.share_experts(ids, w, e, keep, budget, scale=1.7)
        got_i, got_w = moe.share_experts(ids.cuda(), w.cuda(), e, keep, budget, scale=1.7)
        assert torch.equal(got_i.cpu(), want_i)
        assert torch.allclose(got_w.cpu(), want_w, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("t,e,k,h,inter,act", [(129, 5, 2, 256, 384, "relu2"), (300, 40, 6, 512, 640, "relu2"),
                                               (700, 3, 2, 256, 2688, "relu2"), (300, 16, 4, 128, 192, "swiglu"),
                                               (1500, 64, 8, 1024, 704, "swiglu")])
def test_experts_forward_on_sm_pairs(t, e, k, h, inter, act, monkeypatch):
    """Chunks of 256 rows on SM pairs with the activation requantised in fc1's epilogue give the bytes of the one-CTA tiles
    followed by the quantiser: the same sums in the same order (empty, partial and several chunks per expert, a last
    weight tile of 128 rows, plans by one CTA and by a cluster)."""
    from hibana_b200 import _native as nv
    ew = _weights(e, h, inter, act, "nvfp4", "cpu", seed=3).to("cuda")
    g = torch.Generator().manual_seed(t)
    x = torch.randn(t, h, generator=g).bfloat16().cuda()
    logits = torch.randn(t, e, generator=g)
    logits[:, 0] += 3.0                       # a crowded expert
    logits[:, 1] -= 30.0                      # and an empty one
    ids, w = moe.route(logits, k)
    ids, w = ids.cuda(), w.cuda()
    assert moe.pair_rows(ew, t)
    got = moe.experts_forward(x, ids, w, ew)
    half = moe.experts_forward(x, ids, w, ew, e_lo=1, e_n=e - 2)
    monkeypatch.setattr(moe, "pair_rows", lambda *a: False)
    assert torch.equal(got, moe.experts_forward(x, ids, w, ew))
    assert torch.equal(half, moe.experts_forward(x, ids, w, ew, e_lo=1, e_n=e - 2))
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,topk,e,lo,n", [(1, 1, 8, 0, 8), (372, 22, 512, 0, 512), (373, 22, 512, 0, 512),
                                                (4096, 22, 512, 100, 300), (1025, 8, 60, 0, 60)])
def test_plan_places_pairs_in_order(tokens, topk, e, lo, n):
    """Segments, positions and work list of the routing plan (one CTA below 8192 pairs, a cluster of eight from there on)
    against a plain count: whole numbers, all equal."""
    from hibana_b200 import _native as nv
    g = torch.Generator().manual_seed(tokens)
    ids = torch.rand(tokens, e, generator=g).topk(topk, dim=1).indices.int()
    rows_cap = ((tokens * topk + 127) // 128) * 128 + min(n, tokens * topk) * 128
    bn, cap = 256, tokens * topk // 256 + 1 + e
    out = [torch.empty(m, dtype=torch.int32, device="cuda") for m in (e, e, tokens * topk, rows_cap, 1, cap, 1)]
    cnt, start, pos, src, total, tiles, n_tiles = out
    idc = ids.cuda()
    nv.check(nv.lib().hb_moe_plan(idc.data_ptr(), tokens, topk, e, lo, n, 0, cnt.data_ptr(), start.data_ptr(), pos.data_ptr(),
                                  src.data_ptr(), rows_cap, total.data_ptr(), bn, tiles.data_ptr(), n_tiles.data_ptr(), cap,
                                  nv.stream()), "hb_moe_plan")
    flat = ids.view(-1)
    held = (flat >= lo) & (flat < lo + n)
    want_cnt = torch.bincount(flat[held].long(), minlength=e)
    seg = (want_cnt + 127) // 128 * 128
    want_start = seg.cumsum(0) - seg
    assert cnt.cpu().tolist() == want_cnt.tolist() and int(total) == int(seg.sum())
    assert start.cpu().tolist() == want_start.tolist()
    want_pos = torch.full_like(flat, -1)
    want_src = torch.full((rows_cap,), -1, dtype=torch.int32)
    for x in range(lo, lo + n):
        at = (flat == x).nonzero()[:, 0]
        want_pos[at] = (want_start[x] + torch.arange(len(at))).int()
        want_src[int(want_start[x]):int(want_start[x]) + len(at)] = (at // topk).int()
    assert torch.equal(pos.cpu(), want_pos) and torch.equal(src.cpu(), want_src)
    want_tiles = [x * 4096 + c for x in range(e) for c in range(-(-int(want_cnt[x]) // bn))]
    assert int(n_tiles) == len(want_tiles) and tiles[:len(want_tiles)].cpu().tolist() == want_tiles
