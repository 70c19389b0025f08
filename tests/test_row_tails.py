"""Row kernels at the edges of their forms: expert combine, gated norm, tiled convolution."""
import pytest
import torch

from hibana_b200 import _native as nv
from hibana_b200.ops import basic, moe  # noqa: F401  (registers the kernels)


def _close(got, want, terms):
    """fp32 sums of `terms` values (2^-24 each, of the sum of their magnitudes, here below 64), then bf16 (half an ulp: 2^-8)."""
    assert ((got.double() - want).abs() <= terms * 2.0 ** -24 * 64 + 2.0 ** -8 * want.abs()).all()


# 16-byte rows (h, pitches), pairs, a last block that is partly empty, one expert to the limit of 32
@pytest.mark.gpu
@pytest.mark.parametrize("h,pitch", [(2048, 2048), (1032, 1040), (1024 + 8, 1032), (66, 66), (1030, 1032), (2, 2)])
@pytest.mark.parametrize("topk", [1, 8, 9, 32])
@pytest.mark.parametrize("with_shared", [False, True])
def test_combine(h, pitch, topk, with_shared):
    t, rows = 5, 70
    g = torch.Generator().manual_seed(h + topk)
    y = torch.randn(rows, pitch, generator=g).bfloat16().cuda()[:, :h]
    pos = torch.randint(0, rows, (t, topk), generator=g).int()
    pos[1] = -1
    pos[2, 0] = -1
    w = torch.rand(t, topk, generator=g)
    shared = torch.randn(t, pitch, generator=g).bfloat16().cuda()[:, :h] if with_shared else None
    out = torch.full((t + 1, pitch), 7.0, dtype=torch.bfloat16, device="cuda")
    posd, wd = pos.cuda(), w.cuda()
    nv.check(nv.lib().hb_moe_combine(y.data_ptr(), y.stride(0), posd.data_ptr(), wd.data_ptr(), nv.ptr(shared), pitch if with_shared else 0,
                                     out.data_ptr(), pitch, t, topk, h, nv.stream()), "hb_moe_combine")
    want = torch.where((pos >= 0)[..., None], y.cpu().double()[pos.clamp(min=0).long()], torch.zeros((), dtype=torch.float64))
    want = (want * w.double()[..., None]).sum(1) + (shared.cpu().double() if with_shared else 0)
    _close(out[:t, :h].cpu(), want, topk + 1)
    assert (out[:t, h:] == 7).all() and (out[t] == 7).all()


# two to four warps to a group; groups that leave lanes idle, one CTA and hundreds
@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 74, 99])
@pytest.mark.parametrize("gs", [264, 512, 640, 1000, 1024])
@pytest.mark.parametrize("norm_first", [False, True])
def test_gated_norm_of_wide_groups(rows, gs, norm_first):
    groups = 4 if rows != 99 else 3
    g = torch.Generator().manual_seed(gs + rows)
    x, z = (torch.randn(rows, groups * gs, generator=g).bfloat16() for _ in range(2))
    w = torch.randn(groups * gs, generator=g).bfloat16()
    got = basic.gated_rmsnorm(x.cuda(), z.cuda(), w.cuda(), 1e-5, gs, norm_first=norm_first).cpu()
    xd, zd = x.double(), z.double()
    gate = zd * torch.sigmoid(zd)
    v = (xd if norm_first else xd * gate).view(rows, groups, gs)
    n = (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5)).view(rows, -1) * w.double() * (gate if norm_first else 1.0)
    # the fast exponential is good to some 2^-21 for arguments of a few units
    assert ((got.double() - n).abs() <= (2.0 ** -8 + 2.0 ** -18) * n.abs() + 1e-6).all()


# one and two channels a thread (odd counts and pitches take one), tiles of 32 rows in batches of 8, sequences with and without a state
@pytest.mark.gpu
@pytest.mark.parametrize("channels,pitch", [(6, 6), (258, 320), (131, 131), (64, 67)])
@pytest.mark.parametrize("rows", [(33, 1, 40), (64, 65, 7), (3, 96, 2)])
def test_tiled_convolution(channels, pitch, rows):
    from hibana_b200.ops import recurrent
    g = torch.Generator().manual_seed(channels)
    x = torch.randn(sum(rows), pitch, generator=g).bfloat16()
    w, bias = torch.randn(channels, 4, generator=g).bfloat16(), torch.randn(channels, generator=g).bfloat16()
    state = torch.randn(5, channels, 3, generator=g).bfloat16()
    ip = torch.tensor([0, rows[0], rows[0] + rows[1], sum(rows)], dtype=torch.int32)
    slots, init = torch.tensor([3, 1, 4], dtype=torch.int32), torch.tensor([1, 0, 1], dtype=torch.int32)
    kw = dict(silu=True, max_rows=max(rows))
    want_state, got_state = state.clone(), state.cuda()
    want = recurrent.conv1d(x[:, :channels], w, bias, want_state, slots, slots, q_indptr=ip, has_init=init, **kw)
    got = recurrent.conv1d(x.cuda()[:, :channels], w.cuda(), bias.cuda(), got_state, slots.cuda(), slots.cuda(), q_indptr=ip.cuda(),
                           has_init=init.cuda(), **kw)
    # five fp32 terms of at most 16 and the fast exponential, then bf16
    assert ((got.cpu().double() - want.double()).abs() <= 2.0 ** -7 * want.double().abs() + 5 * 16 * 2.0 ** -23).all()
    assert torch.equal(got_state.cpu(), want_state)
