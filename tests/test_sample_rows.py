"""Full-vocabulary and listed-candidate sampling at the edges of the row kernel: one warp of tokens, the longest row staged in
shared memory and the first that is not, more equal tokens than the ranking list holds, candidate counts around the listed form."""
import pytest
import torch

from hibana_b200.engine.rejection import distribution
from hibana_b200.ops import sampling

ROWS = 12


def _rows(kind: str, vocab: int) -> torch.Tensor:
    g = torch.Generator().manual_seed(vocab)
    x = torch.randn(ROWS, vocab, generator=g)
    if kind == "plain":
        return x * 2
    if kind == "ties":                     # a few distinct values, zeros of both signs: thousands of equal tokens at every cut
        return (x * 2).round() / 2
    x = x * 3
    x[:, ::3] = float("-inf")
    x[:, 1::7] = float("nan")
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [33, 4096, 52224, 52225])
@pytest.mark.parametrize("kind", ["plain", "ties", "holes"])
@pytest.mark.parametrize("top_k,top_p", [(0, 0.95), (0, 0.3), (65, 0.9), (3, 1.0), (4, 0.9), (64, 0.95)])
def test_row_kernel_draws_from_the_law(vocab, kind, top_k, top_p):
    x = _rows(kind, vocab)
    masked = kind == "holes"
    mask = None
    if masked:
        g = torch.Generator().manual_seed(1)
        mask = torch.randint(-2 ** 31, 2 ** 31 - 1, (ROWS, (vocab + 31) // 32), generator=g).to(torch.int32)
    temp = torch.tensor([0.8, 1.0, 0.3, 2.0] * 3)
    full = lambda v, dt: torch.full((ROWS,), v, dtype=dt)
    seeds, offs = torch.arange(ROWS) * 7919 + 5, torch.arange(ROWS) + 3
    dev = [t.cuda() for t in (x, temp, full(top_k, torch.int32), full(top_p, torch.float32), seeds, offs)]
    got = sampling.sample(*dev, mask.cuda() if masked else None).cpu()
    for r in range(ROWS):
        lg = x[r].double()
        allowed = ~lg.isnan()
        if masked:
            allowed &= ((mask[r][torch.arange(vocab) // 32] >> (torch.arange(vocab) % 32)) & 1).bool()
        lg[~allowed] = float("-inf")
        if 1 <= top_k <= 64:               # candidates in (value desc, index asc) order
            order = torch.sort(lg, descending=True, stable=True).indices[:top_k]
            w = torch.exp((lg[order] - lg[order[0]]) / float(temp[r]))
        else:
            order = torch.arange(vocab)
            w = distribution(lg[None].float(), float(temp[r]), top_k, 1.0)[0].double()
        w = w / w.sum()
        if top_p < 1:                      # smallest prefix in value order that reaches top_p
            by = torch.sort(lg[order], descending=True, stable=True).indices
            cum = torch.cumsum(w[by], 0)
            cut = int((cum >= top_p).nonzero()[0]) + 1
            drop = by[cut:]
            edge = float(w[by[cut - 1]])
            w[drop] = 0
        else:
            edge = 0.0
        kept = float(w.sum())
        u = sampling.uniform01(int(seeds[r]), int(offs[r])) * kept
        at = int((order == got[r]).nonzero()[0])
        after = float(w[:at + 1].sum())
        before = after - float(w[at])
        # fp32 sums of at most ceil(52225 / 256) + 256 + 13 terms, one after the other: 473 * 2^-24 < 3e-5 of the mass, and as much
        # again for the cut; a cut moved by that rounding moves the mass by the token at the edge where sums tie
        tol = 6e-5 + (edge if edge < 6e-5 else 0.0)
        assert before - tol <= u <= after + tol, (r, u, before, after)


@pytest.mark.gpu
def test_speculative_targets_on_staged_and_long_rows_agree():
    """The same law over a staged row and over one padded with forbidden tokens past the staging limit."""
    vocab, longer, b, k = 5000, 52300, 4, 2
    g = torch.Generator().manual_seed(2)
    x = torch.randn(b * (k + 1), vocab, generator=g).cuda() * 2
    pad = torch.full((b * (k + 1), longer), float("-inf"), device="cuda")
    pad[:, :vocab] = x
    drafts = x.argmax(1).view(b, k + 1)[:, :k].contiguous()
    drafts[0] = 17
    t = lambda v, dt: torch.full((b,), v, dtype=dt, device="cuda")
    args = (t(0.8, torch.float32), t(0, torch.int32), t(0.9, torch.float32), torch.arange(b, device="cuda") + 9,
            torch.arange(b, device="cuda"))
    a, pa = sampling.spec_targets(x, drafts, *args)
    c, pc = sampling.spec_targets(pad, drafts, *args)
    # other strides of the sums (the draw's chunks are 1/256 of the row): 473 * 2^-24 of the mass
    assert torch.allclose(pa, pc, atol=6e-5, rtol=0)
    assert (a == c).float().mean() > 0.8 and bool((a < vocab).all() and (c < vocab).all())


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [18992, 52300])
@pytest.mark.parametrize("top_k", [0, 3000])
def test_nucleus_that_ends_with_a_bucket(vocab, top_k):
    """top-p at the mass where a bucket of the nucleus search ends, give or take some floats, and just below 1: always a finite
    probability and a token of the nucleus (a search whose two tests disagree by a rounding finds no key there)."""
    temp, ulps = 0.8, 8
    x = torch.randn(vocab, generator=torch.Generator().manual_seed(1)) * 2
    order = torch.sort(x, descending=True, stable=True).indices[:top_k or vocab]
    v = x[order]
    w = torch.exp((v.double() - float(v[0])) / temp)
    cum = torch.cumsum(w, 0) / w.sum()
    bucket = ((v[0] - v) * (16 / temp)).floor()
    ends = (bucket[1:] != bucket[:-1]).nonzero().flatten()
    at = cum[ends][(cum[ends] > 0.05) & (cum[ends] < 0.9995)].float()
    ps = torch.cat([(at.view(torch.int32)[:, None] + torch.arange(-ulps, ulps + 1)).flatten().int().view(torch.float32),
                    torch.tensor([1 - 2.0 ** -24, 1 - 2.0 ** -23, 0.999999])])
    b = len(ps)
    full = lambda val, dt: torch.full((b,), val, dtype=dt, device="cuda")
    args = (full(temp, torch.float32), full(top_k, torch.int32), ps.cuda(), torch.arange(b, device="cuda") + 3,
            torch.arange(b, device="cuda"))
    rank = torch.full((vocab,), vocab, dtype=torch.long)
    rank[order] = torch.arange(len(order))
    before = torch.cat([cum - w / w.sum(), torch.tensor([2.0])])      # mass in front of a token; past the top-k cut: none of the law
    tol = 6e-5      # as above: fp32 sums
    tok = sampling.sample(x.cuda().expand(b, vocab), *args).cpu()
    assert (before[rank[tok].clamp_max(len(order))] <= ps.double() + tol).all()
    drafts = full(int(order[0]), torch.int64)[:, None]
    target, p_draft = (t.cpu() for t in sampling.spec_targets(x.cuda().expand(2 * b, vocab), drafts, *args))
    assert (before[rank[target[:, 1]].clamp_max(len(order))] <= ps.double() + tol).all()
    # the first token's share of the nucleus, whose mass is at least p and less than p and one more token
    kept = 1 / (w.sum() * p_draft[:, 0].double())
    edge = (w / w.sum())[torch.searchsorted(cum, ps.double()).clamp_max(len(order) - 1)]
    assert (kept >= ps.double() - tol).all() and (kept <= ps.double() + edge + tol).all()


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [4096, 52225])
@pytest.mark.parametrize("top_p", [1.0, 0.8])
def test_fewer_live_tokens_than_top_k(vocab, top_p):
    """A grammar that leaves 10 tokens and a top-k of 100: the law of those 10."""
    b = 32
    g = torch.Generator().manual_seed(4)
    x = torch.randn(2 * b, vocab, generator=g)
    live = torch.randperm(vocab, generator=g)[:10]
    words = torch.zeros((vocab + 31) // 32, dtype=torch.int64)
    for t in live.tolist():
        words[t // 32] |= 1 << (t % 32)
    mask = ((words + 2 ** 31) % 2 ** 32 - 2 ** 31).to(torch.int32).expand(2 * b, -1).contiguous()
    full = lambda val, dt: torch.full((2 * b,), val, dtype=dt)
    args = (full(0.8, torch.float32), full(100, torch.int32), full(top_p, torch.float32), torch.arange(2 * b) * 31 + 7,
            torch.arange(2 * b))
    got = sampling.sample(x.cuda(), *[a.cuda() for a in args], mask.cuda()).cpu()
    assert torch.equal(got, sampling.sample_ref(x, *args, mask))
    drafts = live[torch.arange(b) % 10][:, None]
    half = [a[:b] for a in args]
    got, p = sampling.spec_targets(x.cuda(), drafts.cuda(), *[a.cuda() for a in half], None, mask.cuda())
    want, pw = sampling.spec_targets_ref(x, drafts, *half, None, mask)
    assert torch.equal(got.cpu(), want) and torch.allclose(p.cpu(), pw, atol=1e-5, rtol=1e-5)


# more tokens than are listed within one bucket: rows whose logits lie close together, the last bucket, rows in several slabs of 2^18
@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [4097, 52224, 262145, 300000])
@pytest.mark.parametrize("spread", [0.001, 0.05, 40.0])
@pytest.mark.parametrize("top_k", [0, 2000])
def test_searches_that_have_to_be_narrowed(vocab, spread, top_k):
    """The nucleus' mass and its tokens, as at the bucket ends; with a top-k the candidates' search is narrowed first."""
    temp, tol = 0.8, 6e-5
    x = torch.randn(vocab, generator=torch.Generator().manual_seed(vocab)) * spread
    order = torch.sort(x, descending=True, stable=True).indices[:top_k or vocab]
    w = torch.exp((x[order].double() - float(x[order[0]])) / temp)
    cum = torch.cumsum(w, 0) / w.sum()
    ps = torch.tensor([0.01, 0.3, 0.77, 0.999, 1.0])
    b = len(ps)
    full = lambda val, dt: torch.full((b,), val, dtype=dt, device="cuda")
    args = (full(temp, torch.float32), full(top_k, torch.int32), ps.cuda(), torch.arange(b, device="cuda") + 3,
            torch.arange(b, device="cuda"))
    rank = torch.full((vocab,), vocab, dtype=torch.long)
    rank[order] = torch.arange(len(order))
    before = torch.cat([cum - w / w.sum(), torch.tensor([2.0])])
    tok = sampling.sample(x.cuda().expand(b, vocab), *args).cpu()
    assert (before[rank[tok].clamp_max(len(order))] <= ps.double() + tol).all()
    target, p_draft = (t.cpu() for t in sampling.spec_targets(x.cuda().expand(2 * b, vocab), full(int(order[0]), torch.int64)[:, None], *args))
    assert (before[rank[target[:, 1]].clamp_max(len(order))] <= ps.double() + tol).all()
    kept = 1 / (w.sum() * p_draft[:, 0].double())
    edge = (w / w.sum())[torch.searchsorted(cum, ps.double()).clamp_max(len(order) - 1)]
    # (sums of ceil(300000 / 256) terms one after the other and a tree: 1185 * 2^-24 of the mass)
    tol = max(tol, 1200 * 2.0 ** -24)
    assert (kept >= ps.double() - tol).all() and (kept <= ps.double() + edge + tol).all()
