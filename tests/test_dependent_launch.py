"""Programmatic dependent launch changes when kernels start, never what they compute."""
import pytest
import torch

from hibana_b200.engine.executor import Executor
from hibana_b200.engine.request import SamplingParams
from hibana_b200.models.dense import DenseModel
from hibana_b200.models.hybrid import HybridModel
from hibana_b200.target import dense_tiny, get_target, scaled, tiny_hybrid_moe


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["dense", "hybrid"])
@pytest.mark.parametrize("graphs", [False, True])
def test_launch_levels_give_the_same_bits(family, graphs):
    """Prefill and decode of short and long prompts: tokens, KV pool and recurrent states of level 2 (every kernel of a step is
    launched as a dependent and may trigger its successor early) equal those of plain launches, run after run."""
    from hibana_b200 import _native as nv
    from hibana_b200.ops import gemm
    t = dense_tiny() if family == "dense" else tiny_hybrid_moe()
    model = (DenseModel if family == "dense" else HybridModel)(t, "cuda", seed=0)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, t.vocab, (n,), generator=g).tolist() for n in (1, 17, 65, 300)]

    def run(level):
        gemm.set_pdl(level)
        ex = Executor(model, max_batch=4, max_ctx=384, kv_slots=1024, radix_cache=False, use_graphs=graphs)
        if graphs:
            ex.capture_graphs()
        out = [r.output_ids for r in ex.generate_batch(prompts, SamplingParams(max_tokens=12, ignore_eos=True))]
        torch.cuda.synchronize()
        pools = [ex.kv.storage[:, :, :, 1:].clone()]
        if ex.state_pool is not None:
            pools += [ex.state_pool.conv[:, 1:].clone(), ex.state_pool.ssm[:, 1:].clone()]
        return out, pools

    try:
        want, pools = run(0)
        for _ in range(3):
            got, again = run(2)
            assert got == want
            assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(pools, again))
    finally:
        from hibana_b200 import config
        gemm.set_pdl(config.current().pdl)
    assert nv.read_status() == 0


# RoPE and KV write inside the attention of an e4m3 pool; the delta rule with its gates in clusters on a side stream and the scan that reads
# its states early; latent experts beside a shared one
SERVED = {
    "dense": lambda: dense_tiny(),
    "delta": lambda: scaled(get_target("qwen38"), layers=4, hidden=2048, ffn=1024, vocab=2048, mtp_layers=0, mtp_depth=0),
    "latent": lambda: scaled(get_target("nemotron"), layers=9, hidden=1024, vocab=2048, experts=32, top_k=4, expert_ffn=256,
                             shared_ffn=512, latent=256, mtp_layers=0, mtp_depth=0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("family", sorted(SERVED))
@pytest.mark.parametrize("sampled", [False, True])
def test_launch_levels_with_fp8_caches_and_sampled_rows(family, sampled):
    """As above: captured decode steps after prompts of odd lengths, fp8 caches, greedy and sampled with a nucleus cut."""
    from hibana_b200 import _native as nv
    from hibana_b200 import config
    from hibana_b200.ops import gemm
    t = SERVED[family]()
    model = (DenseModel if t.family == "dense" else HybridModel)(t, "cuda", seed=0)
    g = torch.Generator().manual_seed(6)
    prompts = [torch.randint(0, t.vocab, (n,), generator=g).tolist() for n in (1, 17, 130)]
    params = SamplingParams(max_tokens=16, ignore_eos=True, **(dict(temperature=0.8, top_p=0.9, seed=11) if sampled else {}))

    def run(level):
        gemm.set_pdl(level)
        ex = Executor(model, max_batch=4, max_ctx=256, kv_slots=1024, radix_cache=False, kv_dtype=torch.float8_e4m3fn)
        ex.capture_graphs()
        out = [r.output_ids for r in ex.generate_batch(prompts, params)]
        torch.cuda.synchronize()
        pools = [ex.kv.storage[:, :, :, 1:].clone()]
        if ex.state_pool is not None:
            pools += [ex.state_pool.conv[:, 1:].clone(), ex.state_pool.ssm[:, 1:].clone()]
        return out, pools

    try:
        want, pools = run(0)
        for _ in range(3):
            got, again = run(2)
            assert got == want
            assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(pools, again))
    finally:
        gemm.set_pdl(config.current().pdl)
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4", "w3"])
@pytest.mark.parametrize("t", [3, 100])
def test_expert_range_without_rows(fmt, t):
    """An expert range that no token is routed to, in a chain of dependents: its grouped GEMMs have nothing to do, but end behind
    what runs in front of them. Bits of the chain equal those of plain launches."""
    from hibana_b200 import _native as nv
    from hibana_b200 import config
    from hibana_b200.ops import gemm, moe
    g = torch.Generator().manual_seed(t)
    e, h, inter = 8, 512, 256
    ew = moe.ExpertWeights.create((torch.randn(e, 2 * inter, h, generator=g) * 0.05).cuda(),
                                  (torch.randn(e, h, inter, generator=g) * 0.05).cuda(), "swiglu", fmt, in_amax=5.0, mid_amax=2.0)
    x = torch.randn(t, 8192, generator=g).bfloat16().cuda()
    wide, back = ((torch.randn(n, k, generator=g) * 0.02).bfloat16().cuda() for n, k in ((h, 8192), (8192, h)))
    ids = torch.randint(0, 4, (t, 2), generator=g).int().cuda()
    w = torch.rand(t, 2, generator=g).cuda()

    def chain():
        y = x
        for _ in range(4):
            shared = gemm.linear_bf16(y, wide)
            y = gemm.linear_bf16(moe.experts_forward(shared, ids, w, ew, shared=shared, e_lo=4, e_n=4), back)
        return y, shared

    try:
        gemm.set_pdl(0)
        want, shared = chain()
        assert torch.equal(moe.experts_forward(shared, ids, w, ew, shared=shared, e_lo=4, e_n=4), shared)
        gemm.set_pdl(2)
        for _ in range(5):
            assert torch.equal(chain()[0], want)
    finally:
        gemm.set_pdl(config.current().pdl)
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4"])
@pytest.mark.parametrize("m", [4, 64, 300])
def test_weights_written_by_the_kernel_in_front(fmt, m):
    """A projection whose weights this library's kernels have just been launched to write (gathered, projected or quantised) waits for
    them, also where a norm that releases its successor at once runs in between."""
    from hibana_b200 import _native as nv
    from hibana_b200.ops import basic, gemm, nvfp4
    g = torch.Generator(device="cuda").manual_seed(m)
    n, k = 8192, 2048
    table = torch.randn(2 * n, k, generator=g, device="cuda").bfloat16() * 0.05
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    probe = torch.randn(32, n, generator=g, device="cuda").bfloat16()
    nw, gs = torch.ones(k, device="cuda").bfloat16(), torch.tensor(0.01, device="cuda")
    alpha = (gs * gs).reshape(1)
    step = torch.cuda.synchronize

    def run(between):
        out = []
        for i in range(4):
            ids = torch.randperm(2 * n, generator=torch.Generator().manual_seed(i))[:n].cuda()
            step()
            w = basic.embedding(ids, table)
            if fmt == "bf16":
                between()
                a = basic.rmsnorm(x, nw, 1e-6)
                between()
                y = gemm.linear_bf16(a, w)
                between()
                out += [y, gemm.linear_bf16(probe, y)]
            else:
                wq = nvfp4.quantize(w, gs)
                between()
                xq, _ = nvfp4.rmsnorm_quantize(x, nw, 1e-6, gs)
                between()
                out.append(gemm.linear_nvfp4(xq, wq, alpha))
                between()
                out.append(gemm.linear_nvfp4_silu_quant(xq, nvfp4.quantize(w, gs), alpha, gs).q.clone())
            step()
        return out

    got, want = run(lambda: None), run(step)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert nv.read_status() == 0


def test_only_promised_weights_are_fetched_early_cpu(monkeypatch):
    from hibana_b200 import _native as nv
    from hibana_b200.models.linear import Linear
    from hibana_b200.ops import gemm
    called = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: called.append(name) or 0

    lin = Linear(torch.randn(128, 64), "bf16")
    for name, fake in (("use_native", lambda *t: True), ("lib", Lib), ("stream", lambda: 0),
                       ("device_state", lambda dev: type("S", (), {"status": torch.zeros(1)}))):
        monkeypatch.setattr(nv, name, fake)
    monkeypatch.setattr(gemm, "_PDL_INIT", True)
    for rows, kernel in ((4, "hb_few_rows_bf16"), (40, "hb_gemm")):
        x = torch.randn(rows, 64).bfloat16()
        called.clear()
        lin(x)
        assert called == [kernel]
        gemm.linear_bf16(x, lin.weight)
        assert called == [kernel, "hb_gemm_plain", kernel]
