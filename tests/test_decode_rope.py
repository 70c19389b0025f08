"""RoPE and KV write inside the decode attention kernel, and its reads ahead of the wait (csrc/attn_decode.cu)."""
import math

import pytest
import torch

from hibana_b200.ops import attention, basic


def test_rope_in_kernel_needs_the_native_path_cpu():
    pool = torch.empty(8, 2, 128, dtype=torch.bfloat16)
    assert not attention.rope_in_kernel(torch.empty(1, 7 * 128, dtype=torch.bfloat16), pool, pool, 4, 2, 128, 128)


def test_rope_that_would_not_reach_its_kernel_is_refused_cpu(monkeypatch):
    """Calls whose dispatch leads elsewhere would attend with unrotated queries and write no K and V (or leave the kernel's rope armed
    for the next call): a ValueError, before anything is armed or launched."""
    from hibana_b200 import _native as nv
    from hibana_b200 import config as cfgmod
    called = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: called.append(name) or 0

    def call(dtype=torch.bfloat16, d=128, q_indptr=None, ready=True):
        pool = torch.zeros(40, 2, d, dtype=dtype)
        qkv = torch.zeros(1, 8 * d, dtype=torch.bfloat16)
        one = torch.ones(1, dtype=torch.int32)
        return attention.paged_attention(qkv[:, :4 * d].unflatten(1, (4, d)), pool, pool, torch.ones(1, 32, dtype=torch.int32), one,
                                         q_indptr=q_indptr, tables_ready=ready, rope=(qkv, one, one, torch.ones(d // 2)))

    with pytest.raises(ValueError, match="rope"):
        call()                                      # the CPU path
    monkeypatch.setattr(nv, "use_native", lambda *t: True)
    monkeypatch.setattr(nv, "lib", Lib)
    monkeypatch.setattr(nv, "stream", lambda: 0)
    monkeypatch.setattr(nv, "device_state", lambda dev: type("S", (), {"status": torch.zeros(1)}))
    for kw in (dict(d=96), dict(dtype=torch.float8_e4m3fn, d=64), dict(q_indptr=torch.tensor([0, 1], dtype=torch.int32)), dict(ready=False)):
        with pytest.raises(ValueError, match="rope"):
            call(**kw)
    with cfgmod.using(decode_attn="tc"), pytest.raises(ValueError, match="rope"):
        call()
    with cfgmod.using(stable_numerics=True), pytest.raises(ValueError, match="rope"):
        call(dtype=torch.float8_e4m3fn)
    assert called == []
    call()
    assert called[-3:] == ["hb_attn_decode_early", "hb_attn_decode_rope", "hb_attn_decode"]


# contexts that end in the first and the last row of a key tile, in the tile after, in one key, and across splits
CTX = [1, 2, 16, 17, 31, 32, 33, 64, 65, 500, 513, 1300]


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,d", [(40, 8, 128), (32, 2, 128), (8, 8, 64), (24, 4, 256)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("scattered", [False, True])
def test_fused_rope_equals_separate_kernels(hq, hkv, d, fp8, splits, scattered):
    """Outputs and both pools bit for bit: the same arithmetic on the same operands in the same order."""
    from hibana_b200 import _native as nv
    if fp8 and d == 64:
        pytest.skip("head dim 64: no tensor-core kernel for e4m3 pools")
    gen = torch.Generator(device="cuda").manual_seed(3)
    b, slots = len(CTX), sum(CTX) + 65
    store = torch.randn(2, hkv, slots, d, generator=gen, device="cuda") * 0.7
    kv_scale = 0.37 if fp8 else 1.0
    store = (store / kv_scale).to(torch.float8_e4m3fn) if fp8 else store.bfloat16()
    pools = [store.clone(), store.clone()]
    perm = torch.randperm(slots - 1, generator=gen, device="cuda") if scattered else torch.arange(slots - 1, device="cuda")
    idx = torch.zeros(b, max(CTX), dtype=torch.int32, device="cuda")
    o = 0
    for i, c in enumerate(CTX):
        idx[i, :c] = perm[o:o + c].int() + 1
        o += c
    ctx = torch.tensor(CTX, dtype=torch.int32, device="cuda")
    pos = ctx - 1
    new = idx.gather(1, pos.long()[:, None]).squeeze(1).contiguous()
    qkv = torch.randn(b, (hq + 2 * hkv) * d, generator=gen, device="cuda").bfloat16()
    inv = basic.rope_inv_freq(d, 1e6, device="cuda")
    ws = attention.AttnWorkspace(b, hq, d, splits, torch.device("cuda")) if splits > 1 else None
    kw = dict(scale=1 / math.sqrt(d), kv_scale=kv_scale, splits=splits, workspace=ws)
    k, v = pools[0][0].transpose(0, 1), pools[0][1].transpose(0, 1)
    q = basic.rope_kv_write(qkv, pos, new, inv, k, v, hq, hkv, d, kv_scale=kv_scale)
    want = attention.paged_attention(q, k, v, idx, ctx, **kw)
    k, v = pools[1][0].transpose(0, 1), pools[1][1].transpose(0, 1)
    assert attention.rope_in_kernel(qkv, k, v, hq, hkv, d, d)
    torch.cuda.synchronize()      # what `tables_ready` promises
    got = attention.paged_attention(qkv[:, :hq * d].unflatten(1, (hq, d)), k, v, idx, ctx, tables_ready=True,
                                    rope=(qkv, pos, new, inv), **kw)
    assert torch.equal(got, want)
    assert torch.equal(pools[0].view(torch.uint8), pools[1].view(torch.uint8))
    # tables read ahead of the wait, keys written by the separate kernel
    again = attention.paged_attention(q, k, v, idx, ctx, tables_ready=True, **kw)
    assert torch.equal(again, want)
    assert nv.read_status() == 0
