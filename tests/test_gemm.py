"""tcgen05 GEMM and NVFP4 quantiser against plain PyTorch fp32 references."""
import pytest
import torch

from hibana_b200 import _native as nv
from hibana_b200.ops import gemm, nvfp4


def test_e2m1_round_trip_cpu():
    codes = torch.arange(16, dtype=torch.int32)
    vals = nvfp4.e2m1_values(codes)
    assert torch.equal(nvfp4.e2m1_codes(vals) & 7, codes & 7)
    # ties go to the even mantissa
    x = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])
    assert nvfp4.e2m1_values(nvfp4.e2m1_codes(x)).tolist() == [0.0, 1.0, 1.0, 2.0, 2.0, 4.0, 4.0]


def test_swizzle_round_trip_cpu():
    sf = torch.randint(0, 255, (200, 20), dtype=torch.uint8)
    blocks = nvfp4.swizzle_sf(sf)
    assert blocks.shape == (2, 8, 512)
    assert torch.equal(nvfp4.unswizzle_sf(blocks, 200, 20), sf)
    r, g = 133, 7
    assert blocks[r // 128, g // 4, (r % 32) * 16 + ((r % 128) // 32) * 4 + g % 4] == sf[r, g]


def test_quant_dequant_error_cpu():
    x = torch.randn(64, 256)
    gs = float(x.abs().max()) / (6 * 448)
    q, sfb = nvfp4.quantize_ref(x, gs)
    y = nvfp4.dequantize_ref(q, sfb, gs)
    rel = (x - y).norm() / x.norm()
    assert rel < 0.12


def test_linear_nvfp4_cpu_reference():
    w = torch.randn(96, 128) * 0.02
    x = torch.randn(5, 128)
    wq = nvfp4.quantize_weight(w)
    gs = torch.tensor(float(x.abs().max()) / (6 * 448))
    xq = nvfp4.quantize(x.bfloat16(), gs)
    y = gemm.linear_nvfp4(xq, wq, gs * wq.gscale)
    ref = x @ w.t()
    assert (y.float() - ref).norm() / ref.norm() < 0.2


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (8, 5120, 5120), (64, 1024, 17408), (200, 384, 704),
                                   (300, 512, 1024), (1024, 2048, 4096)])
@pytest.mark.parametrize("epi", [gemm.EPI_STORE, gemm.EPI_RESIDUAL, gemm.EPI_SILU_MUL, gemm.EPI_STORE_F32])
def test_gemm_bf16(m, n, k, epi):
    dev = torch.device("cuda")
    x = (torch.randn(m, k, device=dev) * 0.5).bfloat16()
    w = (torch.randn(n, k, device=dev) * 0.05).bfloat16()
    res = torch.randn(m, n, device=dev).bfloat16() if epi == gemm.EPI_RESIDUAL else None
    y = gemm.linear_bf16(x, w, epilogue=epi, residual=res)
    ref = gemm._ref_epilogue(x.float() @ w.float().t(), epi, res)
    torch.cuda.synchronize()
    assert nv.read_status() == 0
    err = (y.float() - ref.float()).abs().max().item()
    scale = ref.float().abs().max().item()
    assert err <= 2e-2 * scale + 1e-3, (err, scale)


@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(1, 256), (7, 5120), (130, 704), (512, 17408)])
@pytest.mark.parametrize("mode", [nvfp4.MODE_PLAIN, nvfp4.MODE_SILU_SPLIT, nvfp4.MODE_SILU_PAIRS])
def test_quant_nvfp4_matches_reference(m, k, mode):
    dev = torch.device("cuda")
    cols = k if mode == nvfp4.MODE_PLAIN else 2 * k
    x = torch.randn(m, cols, device=dev).bfloat16()
    gs = torch.tensor(4.0 / (6 * 448), device=dev)
    got = nvfp4.quantize(x, gs, mode)
    y = x if mode == nvfp4.MODE_PLAIN else nvfp4._silu_mul(x, mode)
    packed, sfb = nvfp4.quantize_ref(y, gs)
    sf_got = nvfp4.unswizzle_sf(got.sf, m, k // 16)
    # silu uses __expf on the device: allow a handful of one-step differences in the fused modes
    mism_sf = (sf_got != sfb).float().mean().item()
    mism_q = (got.q != packed).float().mean().item()
    if mode == nvfp4.MODE_PLAIN:
        assert mism_sf == 0 and mism_q == 0
    else:
        assert mism_sf < 1e-3 and mism_q < 1e-2
    # padding scales are zero
    blocks = got.sf
    full = nvfp4.unswizzle_sf(blocks, blocks.shape[0] * 128, blocks.shape[1] * 4)
    assert full[m:].sum() == 0 and full[:, k // 16:].sum() == 0


@pytest.mark.gpu
def test_norm_quant_matches_reference():
    dev = torch.device("cuda")
    m, k = 37, 5120
    x = torch.randn(m, k, device=dev).bfloat16()
    res = torch.randn(m, k, device=dev).bfloat16()
    w = (torch.randn(k, device=dev) * 0.1 + 1).bfloat16()
    gs = torch.tensor(8.0 / (6 * 448), device=dev)
    res_ref = res.clone()
    ref_q, ref_y = nvfp4.rmsnorm_quantize(x.cpu(), w.cpu(), 1e-6, gs.cpu(), residual=(res_cpu := res_ref.cpu()),
                                          want_normed=True)
    got_q, got_y = nvfp4.rmsnorm_quantize(x, w, 1e-6, gs, residual=res, want_normed=True)
    assert torch.equal(res.cpu(), res_cpu)
    assert (got_y.cpu().float() - ref_y.float()).abs().max() < 0.05
    a, b = got_q.dequantize().cpu(), ref_q.dequantize()
    assert (a - b).norm() / b.norm() < 0.02


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 256, 256), (4, 5120, 5120), (16, 1024, 17408), (64, 34816, 5120),
                                   (200, 384, 768), (300, 512, 1024), (1024, 5120, 2560), (2048, 768, 640)])
def test_gemm_nvfp4(m, n, k):
    dev = torch.device("cuda")
    x = torch.randn(m, k, device=dev).bfloat16()
    w = torch.randn(n, k, device=dev) * 0.02
    wq = nvfp4.quantize_weight(w)
    gs = torch.tensor(float(x.float().abs().max()) / (6 * 448), device=dev)
    xq = nvfp4.quantize(x, gs)
    alpha = (gs * wq.gscale).reshape(1)
    y = gemm.linear_nvfp4(xq, wq, alpha)
    torch.cuda.synchronize()
    assert nv.read_status() == 0
    ref = xq.dequantize() @ wq.dequantize().t()
    err = (y.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1.5e-2 * scale + 1e-4, (err, scale)


@pytest.mark.gpu
def test_gemm_nvfp4_epilogues_and_splitk_deterministic():
    dev = torch.device("cuda")
    m, n, k = 8, 1024, 8192
    x = torch.randn(m, k, device=dev).bfloat16()
    wq = nvfp4.quantize_weight(torch.randn(n, k, device=dev) * 0.02)
    gs = torch.tensor(float(x.float().abs().max()) / (6 * 448), device=dev)
    xq = nvfp4.quantize(x, gs)
    alpha = (gs * wq.gscale).reshape(1)
    acc = xq.dequantize() @ wq.dequantize().t()
    res = torch.randn(m, n, device=dev).bfloat16()
    for epi in (gemm.EPI_RESIDUAL, gemm.EPI_SILU_MUL):
        y1 = gemm.linear_nvfp4(xq, wq, alpha, epilogue=epi, residual=res, splits=4)
        y2 = gemm.linear_nvfp4(xq, wq, alpha, epilogue=epi, residual=res, splits=4)
        y3 = gemm.linear_nvfp4(xq, wq, alpha, epilogue=epi, residual=res, splits=1)
        ref = gemm._ref_epilogue(acc, epi, res)
        assert torch.equal(y1, y2)
        for y in (y1, y3):
            assert (y.float() - ref.float()).abs().max() <= 2e-2 * ref.float().abs().max() + 1e-3
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 512, 1024), (4, 1280, 2560), (64, 768, 1152), (300, 640, 512), (2048, 1024, 2048)])
@pytest.mark.parametrize("dynamic", [False, True])
def test_fp8_gemm_matches_reference(m, n, k, dynamic):
    """e4m3 x e4m3 on tcgen05 (kind::f8f6f4) vs the fp32 product of the dequantised operands."""
    from hibana_b200.ops import fp8
    g = torch.Generator().manual_seed(m + n)
    x = (torch.randn(m, k, generator=g) * 1.5).bfloat16()
    w = fp8.Fp8Weight.quantize(torch.randn(n, k, generator=g) * 0.05)
    wc = fp8.Fp8Weight(w.q.cuda(), w.scale.cuda())
    if dynamic:
        q_ref, s_ref = fp8.quantize_rows(x)
        q, s = fp8.quantize_rows(x.cuda())
        assert torch.allclose(s.cpu(), s_ref, rtol=1e-3)
        ref = fp8.linear_fp8(q.cpu(), w, row_scales=s.cpu())
        got = fp8.linear_fp8(q, wc, row_scales=s)
    else:
        scale = torch.tensor([float(x.float().abs().max()) / 448.0])
        q = fp8.quantize_static(x.cuda(), scale.cuda())
        assert torch.equal(q.cpu().float(), fp8.quantize_static(x, scale).float())
        ref = fp8.linear_fp8(q.cpu(), w, x_scale=scale)
        got = fp8.linear_fp8(q, wc, x_scale=scale.cuda())
    err = (got.float().cpu() - ref.float()).abs().max() / ref.float().abs().max()
    assert float(err) < 1e-2, float(err)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 512, 1024), (8, 1280, 2560), (64, 640, 4352), (130, 300, 512), (256, 1024, 1024)])
def test_w3_dequant_fused_gemm(m, n, k):
    """3-bit codes expanded in shared memory and multiplied on tcgen05 vs fp32 over the dequantised matrix."""
    from hibana_b200.ops.w3gemm import W3Linear
    g = torch.Generator().manual_seed(k + m)
    w = torch.randn(n, k, generator=g) * 0.05
    x = torch.randn(m, k, generator=g).bfloat16()
    lin = W3Linear.from_weight(w, "cuda")
    ref = x.float() @ lin.w3.dequantize().t()
    got = lin(x.cuda()).float().cpu()
    err = (got - ref).abs().max() / ref.abs().max()
    assert float(err) < 1e-2, float(err)
    res = torch.randn(m, n, generator=g).bfloat16()
    got = lin(x.cuda(), epilogue=1, residual=res.cuda()).float().cpu()
    assert float((got - (ref + res.float())).abs().max() / ref.abs().max()) < 2e-2
    from hibana_b200 import _native as nv
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (7, 1024, 5120), (64, 4352, 5120), (64, 34816, 1024), (100, 512, 768),
                                   (300, 192, 512), (300, 96, 512), (384, 4352, 1024), (1000, 2176, 768), (2048, 1024, 512)])
def test_silu_mul_requant_epilogue_matches_two_kernels(m, n, k):
    """gate/up GEMM with the SiLU-mul + NVFP4 requant epilogue == the SiLU-mul GEMM followed by the quantiser,
    byte for byte (packed values and every scale byte of real rows), for unsplit and cluster split-K launches and
    for prefill-sized calls (more than 256 rows: tokens on the 128-row side of the MMA); and the dequantised result is close to the fp32 reference of the same op."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(m * 7 + n)
    w = torch.randn(n, k, device=dev, generator=g) * 0.05
    x = torch.randn(m, k, device=dev, generator=g).bfloat16()
    wq = nvfp4.quantize_weight(w)
    gs = torch.tensor(6.0 / (6 * 448), device=dev)
    xq = nvfp4.quantize(x, gs)
    alpha = (gs * wq.gscale).reshape(1)
    acc = xq.dequantize() @ wq.dequantize().t()
    ref = torch.nn.functional.silu(acc[:, 0::2]) * acc[:, 1::2]
    out_scale = (ref.abs().max() / (6 * 448)).reshape(()).float()      # no clipping: the error is rounding only
    two = nvfp4.quantize(gemm.linear_nvfp4(xq, wq, alpha, epilogue=gemm.EPI_SILU_MUL), out_scale)
    one = gemm.linear_nvfp4_silu_quant(xq, wq, alpha, out_scale)
    torch.cuda.synchronize()
    assert nv.read_status() == 0
    assert torch.equal(one.q, two.q)
    groups = n // 2 // 16
    assert torch.equal(nvfp4.unswizzle_sf(one.sf, m, groups), nvfp4.unswizzle_sf(two.sf, m, groups))
    err = (one.dequantize() - ref).norm() / ref.norm().clamp_min(1e-6)
    assert err < 0.15, err
    # a second call reuses the persistent buffers and must give the same bytes (captured graphs replay it)
    again = gemm.linear_nvfp4_silu_quant(xq, wq, alpha, out_scale)
    assert torch.equal(again.q, two.q)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(257, 256, 288), (300, 5120, 512), (511, 264, 256), (513, 336, 1312), (700, 18560, 256),
                                   (1025, 4096, 1088), (2048, 5120, 704), (4100, 2048, 320)])
@pytest.mark.parametrize("epi", [gemm.EPI_STORE, gemm.EPI_RESIDUAL, gemm.EPI_SILU_MUL])
def test_gemm_nvfp4_sm_pairs(m, n, k, epi):
    """Prefill-sized calls on SM pairs: ragged rows, columns and K tiles, last waves of every unit width. Bound per element:
    one bf16 rounding of the result (two with a residual) plus an fp32 accumulation of K / 64 block products."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(m + n + k)
    x = torch.randn(m, k, device=dev, generator=g).bfloat16()
    wq = nvfp4.quantize_weight(torch.randn(n, k, device=dev, generator=g) * 0.05)
    gs = torch.tensor(6.0 / (6 * 448), device=dev)
    xq = nvfp4.quantize(x, gs)
    alpha = (gs * wq.gscale).reshape(1)
    res = torch.randn(m, n, device=dev, generator=g).bfloat16() if epi == gemm.EPI_RESIDUAL else None
    y = gemm.linear_nvfp4(xq, wq, alpha, epilogue=epi, residual=res)
    torch.cuda.synchronize()
    assert nv.read_status() == 0
    a, b = xq.dequantize().double(), wq.dequantize().double()
    acc = a @ b.t()
    err = (k // 64 + 1) * 2.0 ** -22 * (a.abs() @ b.abs().t())
    if epi == gemm.EPI_SILU_MUL:
        gate, up = acc[:, 0::2], acc[:, 1::2]
        ref = torch.nn.functional.silu(gate) * up
        # |silu'| <= 1.1; the exponential and the division of the epilogue are good to 2^-20
        bound = 2.0 ** -8 * ref.abs() + 1.1 * err[:, 0::2] * up.abs() + err[:, 1::2] * gate.abs() + 2.0 ** -20 * ref.abs()
    else:
        ref = acc if res is None else acc + res.double()
        bound = 2.0 ** -8 * (ref.abs() + (acc.abs() if res is not None else 0)) + err
    assert bool(((y.double() - ref).abs() <= bound + 1e-30).all())


@pytest.mark.parametrize("n,k_tiles", [(5120, 80), (256, 20), (34816, 20)])
def test_stable_plan_does_not_depend_on_rows_cpu(n, k_tiles):
    from hibana_b200 import config as cfgmod
    with cfgmod.using(stable_numerics=True):
        plans = {gemm._plan(m, n, k_tiles, 0)[2] for m in (1, 16, 64, 65, 128, 129, 256)}
    assert len(plans) == 1
    s = plans.pop()
    assert s == 1 or s < -1       # negative: the launch lowers the number alike at every tile width


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(5120, 5120), (1024, 17408), (7168, 5120)])
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4", "fp8"])
def test_stable_numerics_rows_keep_their_bits_at_any_batch(n, k, fmt):
    """Under `stable_numerics` a row of a projection has the same bits however many rows share the call, on either side of
    the 64-token tile (two CTAs per SM) and of the 128-token one."""
    from hibana_b200 import config as cfgmod
    from hibana_b200.ops import fp8
    torch.manual_seed(4)
    x = torch.randn(256, k, device="cuda").bfloat16()
    w = torch.randn(n, k, device="cuda") * 0.02
    if fmt == "bf16":
        wb = w.bfloat16()
        run = lambda rows: gemm.linear_bf16(rows, wb, epilogue=gemm.EPI_STORE_F32)
    elif fmt == "nvfp4":
        wq, gs = nvfp4.quantize_weight(w), torch.tensor(6.0 / (6 * 448), device="cuda")
        alpha = (gs * wq.gscale).reshape(1)
        run = lambda rows: gemm.linear_nvfp4(nvfp4.quantize(rows, gs), wq, alpha, epilogue=gemm.EPI_STORE_F32)
    else:
        w8, scale = fp8.Fp8Weight.quantize(w), torch.tensor([6.0 / 448], device="cuda")
        run = lambda rows: fp8.linear_fp8(fp8.quantize_static(rows, scale), w8, x_scale=scale, epilogue=gemm.EPI_STORE_F32)
    with cfgmod.using(stable_numerics=True):
        want = run(x[:1]).clone()
        for m in (2, 16, 64, 65, 80, 128, 130, 256):
            assert torch.equal(run(x[:m])[:1], want), m
            assert m < 80 or torch.equal(run(x[:m])[:64], run(x[:64])), m
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("k,few", [(2688, 448), (2064, 448), (8192, 256), (6160, 256), (5120, 448), (1024, 448)])
def test_norm_quant_rows_do_not_depend_on_how_many_there_are(k, few):
    """Few rows hold the norm weights from the start, many read them late (2 and 4 chunks per thread): the same bytes."""
    torch.manual_seed(6)
    x, res = (torch.randn(few + 1, k, device="cuda").bfloat16() for _ in range(2))
    w, gs = torch.randn(k, device="cuda").bfloat16(), torch.tensor(0.01, device="cuda")
    out = []
    for m in (few, few + 1):
        r = res[:m].clone()
        q, y = nvfp4.rmsnorm_quantize(x[:m], w, 1e-6, gs, residual=r, want_normed=True)
        out.append((q.q[:few], nvfp4.unswizzle_sf(q.sf, m, k // 16)[:few], y[:few], r[:few]))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    ref = (x.float() + res.float()).bfloat16().float()[:few]
    ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + 1e-6) * w.float()
    assert bool(((out[0][2].float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(257, 64, 256), (257, 320, 288), (513, 320, 512), (513, 2112, 256), (300, 2112, 1024),
                                   (600, 10304, 256), (2048, 5120, 256)])
def test_requant_epilogue_on_sm_pairs_ragged(m, n, k):
    """SiLU-mul + requantisation with ragged rows, odd multiples of 32 features and a last wave of narrow units: every packed
    byte and every scale byte of the rows, padding groups included, as SiLU-mul followed by the quantiser leaves them."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    wq = nvfp4.quantize_weight(torch.randn(n, k, device="cuda", generator=g) * 0.05)
    gs, out_scale = torch.tensor(6.0 / (6 * 448), device="cuda"), torch.tensor(0.002, device="cuda")
    xq = nvfp4.quantize(torch.randn(m, k, device="cuda", generator=g).bfloat16(), gs)
    alpha = (gs * wq.gscale).reshape(1)
    two = nvfp4.quantize(gemm.linear_nvfp4(xq, wq, alpha, epilogue=gemm.EPI_SILU_MUL), out_scale)
    one = gemm.linear_nvfp4_silu_quant(xq, wq, alpha, out_scale)
    assert torch.equal(one.q, two.q) and one.sf.shape == two.sf.shape
    groups = 4 * one.sf.shape[1]
    assert torch.equal(nvfp4.unswizzle_sf(one.sf, m, groups), nvfp4.unswizzle_sf(two.sf, m, groups))
    assert nv.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m", [300, 257, 400])
def test_split_k_with_the_tokens_on_the_128_row_side(m):
    """A cluster per tile, the last of which has warps without rows: they read the peers' partials too and must not outlive them."""
    from hibana_b200 import _native as nv
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, 2048, generator=g, device="cuda").bfloat16()
    w = torch.randn(320, 2048, generator=g, device="cuda").bfloat16()
    want = x.double() @ w.double().t()
    for _ in range(20):
        y = gemm.linear_bf16(x, w, epilogue=gemm.EPI_STORE_F32, splits=4)
        # fp32 sums of k exact products: k * 2^-24 of the sum of their magnitudes
        assert ((y.double() - want).abs() <= 2048 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())).all()
    assert nv.read_status() == 0
