"""bf16 projections of up to 16 rows (csrc/few_rows.cu) against fp64."""
import pytest
import torch

from hibana_b200 import config as cfgmod
from hibana_b200.ops import gemm


def test_few_rows_rule_cpu():
    def ok(m, n, k, epi=gemm.EPI_STORE, res=None, **kw):
        return gemm.few_rows_ok(torch.empty(m, k, dtype=torch.bfloat16), torch.empty(n, k, dtype=torch.bfloat16), epi, res)
    assert ok(1, 512, 4096) and ok(16, 1024, 4096) and ok(8, 4096, 4096) and ok(4, 96, 5120, gemm.EPI_STORE_F32)
    assert not ok(17, 512, 4096) and not ok(16, 4096, 4096) and not ok(1, 8192, 5120) and not ok(1, 64, 60)
    assert not ok(1, 512, 4096, gemm.EPI_SILU_MUL) and not ok(1, 512, 4096, gemm.EPI_RESIDUAL, torch.empty(1, 512))
    x = torch.empty(4, 136, dtype=torch.bfloat16)
    w = torch.empty(64, 128, dtype=torch.bfloat16)
    assert gemm.few_rows_ok(x[:, :128], w, gemm.EPI_STORE, None) and not gemm.few_rows_ok(x[:, 4:132], w, gemm.EPI_STORE, None)
    with cfgmod.using(stable_numerics=True):
        assert not ok(1, 512, 4096)


# n and k around the tiles (16 features, 32-element steps, turns of 4, 8 and 16 warps, clusters of 8) and each of the kernel's forms
@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(1, 8), (17, 72), (16, 2048), (31, 2056), (96, 5120), (50, 1000), (512, 4096), (520, 2056), (4096, 1024), (4100, 264),
                                 (2368, 1032), (2384, 3304)])
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("f32", [True, False])
def test_few_rows_match_fp64(n, k, m, f32):
    """fp32 sums of k exact products in any order are off by at most k * 2^-24 of the sum of their magnitudes; rounding to bf16 (8
    significant bits: half an ulp is at most 2^-8 of the value) adds that."""
    from hibana_b200 import _native as nv
    g = torch.Generator(device="cuda").manual_seed(n * 31 + k + m)
    xs = torch.randn(m, k + 8, generator=g, device="cuda").bfloat16()
    x = xs[:, 8:]                                    # a column slice: rows with a pitch of their own
    w = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    epi = gemm.EPI_STORE_F32 if f32 else gemm.EPI_STORE
    assert gemm.few_rows_ok(x, w, epi, None)
    guard = torch.full((m + 2, n + 3), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    out = guard[1:m + 1, :n]
    gemm.linear_bf16(x, w, epilogue=epi, out=out)
    want = x.double() @ w.double().t()
    bound = k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + (0 if f32 else 2.0 ** -8) * want.abs()
    assert ((out.double() - want).abs() <= bound).all()
    assert (guard[0] == 7).all() and (guard[-1] == 7).all() and (guard[:, n:] == 7).all()
    assert nv.read_status() == 0


# the tcgen05 form cuts K into 8 pieces here, so that its chains of additions are short
@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(256, 1000), (300, 1536), (512, 4096), (4096, 1024)])
@pytest.mark.parametrize("m", [1, 8, 16])
def test_few_rows_are_as_close_as_the_tiles(n, k, m):
    """2-norm of the error against fp64 over N = n * m sums. A norm of N independent errors varies by 1 / sqrt(2 N) of itself, the
    quotient of two by 1 / sqrt(N): four times that is allowed, 25 % at N = 256 (chains twice as long are off by 75 % there)."""
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    want = x.double() @ w.double().t()
    splits = gemm._plan(m, n, (k + 63) // 64, 0)[2]
    few, tiles = ((gemm.linear_bf16(x, w, epilogue=gemm.EPI_STORE_F32, splits=s).double() - want).norm().item() for s in (None, splits))
    assert few <= (1 + 4 / (n * m) ** 0.5) * tiles, (few, tiles)
