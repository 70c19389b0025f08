"""Paged GQA attention over the token-granular KV pool (decode, speculative verify, chunked prefill).

`paged_attention` is the single entry: query rows of a ragged batch attend to their sequence's context through
the block table. Kernels: csrc/attn_prefill.cu (tcgen05 prefill, two Q tiles per CTA where `two_q_tiles` says so),
csrc/attn_decode.cu (tensor-core flash-decoding, up to 16 query rows per kv head, RoPE and KV write of a decode step inside),
csrc/attn.cu (general split-KV + LSE merge: NVFP4 KV, and fp8 KV under `stable_numerics`, with head dim 64 or off 16-byte
boundaries). The plain-PyTorch reference below is the CPU path
and the GPU tests' oracle. Reference counterparts: hibana/kernels/ops.py:131-161 (ragged prefill),
hibana/model/attention.py:69-126, hibana/kernels/csrc/verify_attn.cu.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from .. import _native as nv
from .. import config as cfgmod
from . import nvfp4

P, I, L, Fl = nv.P, nv.I, nv.L, nv.F
nv.register("hb_attn_paged", [P, P, P, L, L, P, L, P, P, P, P, P, P, I, I, I, I, I, I, I, Fl, I, Fl, I, P])

nv.register("hb_attn_merge", [P, P, P, L, I, I, P])
nv.register("hb_attn_fp4_scales", [P, P, L, L], void=True)
nv.register("hb_attn_merge_quant", [P, P, L, I, I, I, P, P, P, I, P])
nv.register("hb_attn_decode", [P, P, P, L, L, P, L, P, P, P, P, P, P, I, I, I, I, I, I, Fl, I, Fl, I, L, P, P])

nv.register("hb_attn_decode_fuse", [P, P, P, P, I], void=True)
nv.register("hb_attn_decode_early", [], void=True)
nv.register("hb_attn_decode_rope", [P, L, P, P, P, Fl], void=True)
nv.register("hb_attn_decode_tc", [P, P, P, L, L, P, L, P, P, P, P, P, P, I, I, I, I, I, I, Fl, I, L, P, P])
nv.register("hb_attn_decode_tc_profile", [P], void=True)
nv.register("hb_attn_prefill_profile", [P], void=True)
nv.register("hb_attn_decode_profile", [P], void=True)
nv.register("hb_attn_prefill", [P, P, P, L, L, P, L, P, P, P, P, P, P, I, I, I, I, I, I, Fl, I, Fl, I, L, P, P])

from ..hardware.b200 import NUM_SMS  # noqa: E402


# One pass of a bf16 decode CTA (two warps, a 32-key tile each). A pass is a chain of latencies, about 1.6 us: one sequence of
# 500 keys on 8 kv heads takes 15.1 us as one split and 11.3 us, merge included, in seven.
MIN_SPLIT_KEYS = 64
# The merge is a launch of about 4 us: as much as this many keys of a CTA. One sequence on 8 kv heads, whole / in ranges of 64:
# 128 keys 8.4 / 10.2 us, 256 keys 10.4 / 10.2, 320 keys 11.2 / 10.2; 8 sequences, whole / in two: 256 keys 10.4 / 11.4,
# 448 keys 13.3 / 13.4, 512 keys 14.2 / 13.3.
MIN_KEYS_SAVED = 224
DECODE_CTAS_PER_SM = 2      # csrc/attn_decode.cu: 64-thread CTAs with ~100 KB of rings, two share an SM


def choose_splits(batch: int, hkv: int, max_ctx: int, row_chunks: int = 1, slots: int = 0) -> int:
    """KV splits that fill whole waves of the resident CTA slots (the decode kernel streams from every resident
    CTA at once, so a last wave that is a third full costs a whole wave). Within the first wave a split may be as short as
    MIN_SPLIT_KEYS keys, where that takes MIN_KEYS_SAVED keys off every CTA: idle SMs take it. Beyond it one has at least
    256 keys, because shorter ones only leave more to merge (4 sequences of 5000 keys on 4 heads: 9 splits take 19.8 us and
    5.2 us of merge, 37 take 26.4 and 8.4). `max_ctx` is the limit that a captured launch is planned for, which the
    sequences may stay far below: an engine with a limit of 32k runs one of 500 keys in 37 splits, 16 of them with keys."""
    if cfgmod.current().stable_numerics:
        # row-count invariant: one pass over the keys in fixed tiles from position 0, so a token's attention sums
        # in the same order whether it is the only new row of its sequence or one of several verified rows
        return 1
    slots = slots or NUM_SMS * max(1, cfgmod.current().attn_ctas_per_sm)
    ctas = max(1, batch * hkv * row_chunks)
    cap = int(max(1, min(max_ctx // MIN_SPLIT_KEYS, 64)))
    best, best_eff = 1, 0.0
    for s in range(1, cap + 1):
        n = ctas * s
        if n > slots and s > max_ctx // 256:
            break
        eff = n / (-(-n // slots) * slots)
        if eff > best_eff + 0.02:     # prefer fewer splits unless the wave efficiency clearly improves
            best, best_eff = s, eff
    return best if max_ctx - -(-max_ctx // best) >= MIN_KEYS_SAVED else 1


# A split prefill writes fp32 partial rows and runs a merge: worth it when every CTA gets rid of this many of its key tiles
# (32 CTAs of 8 tiles: 22.3 us whole, 22.4 in four ranges; of 16 tiles 34.2 and 24.7; 40 / 8 heads of 128).
MIN_TILES_SAVED = 6


def prefill_splits(batch: int, hq: int, hkv: int, d: int, max_rows: int, max_ctx: int) -> int:
    """Context ranges of a tensor-core prefill (csrc/attn_prefill.cu): whole key tiles, two at least, and no more CTAs than
    one wave, of which an SM holds one. A second wave of ranges only adds partial rows to write and merge: 100 rows over
    30000 keys, 40 / 8 heads, 32 CTAs of whole contexts take 353 us, in 4 ranges 112, in 37 ranges 192; 100 rows over 500
    keys 16 us whole, 35 in 7 ranges."""
    if cfgmod.current().stable_numerics:
        return 1
    tiles = -(-max_ctx // (128 if d <= 128 else 64))
    blocks = batch * hkv * -(-max_rows // max(1, 128 // (hq // hkv)))
    room = min(NUM_SMS // max(1, blocks), 64)
    if room < 2:
        return 1
    per = max(2, -(-tiles // room))
    return -(-tiles // per) if tiles - per >= MIN_TILES_SAVED else 1


# Keys that a row sees on average up to which two Q tiles per CTA pay within half a wave of CTAs (`two_q_tiles`).
TWO_TILES_KEYS = 192


def two_q_tiles(batch: int, hq: int, hkv: int, max_rows: int, max_ctx: int = 0) -> bool:
    """Whether an unsplit bf16 prefill (head dims up to 128) over contexts of up to `max_ctx` keys runs two 128-row Q tiles per CTA
    (csrc/attn_prefill.cu, attn_prefill_q2_kernel). Against one tile per CTA, 40 / 8 heads of 128: more tiles than one wave of CTAs 1.4
    to 1.9 times as fast (460 tokens 24.9 -> 17.5 us, over 16000 keys 382 -> 253, 2048 tokens 111 -> 62). Within one wave a CTA has twice the
    rows to do while SMs stay idle, which every key tile pays for: prompts of 29 / 128 / 225 tokens 13.1 / 13.1 / 14.0 -> 8.8 / 11.1 /
    12.3, but four times 50 rows over 256 / 512 / 1024 keys 13.2 / 15.9 / 22.0 -> 13.9 / 17.9 / 26.0 (longer contexts are split,
    `prefill_splits`). So up to half a wave a row may see 192 keys on average: 150 rows over 256 keys gain 5 %, 100 lose 3 %.
    One form for all row counts under `stable_numerics`."""
    if cfgmod.current().stable_numerics:
        return False
    ctas = batch * hkv * -(-max_rows // max(1, 128 // (hq // hkv)))
    return ctas > NUM_SMS or 2 * ctas <= NUM_SMS and max_ctx - max_rows // 2 <= TWO_TILES_KEYS


def forward_splits(k_pool: torch.Tensor, v_pool: torch.Tensor, batch: int, hq: int, hkv: int, d: int, max_rows: int,
                   max_ctx: int) -> int:
    """KV splits of a ragged forward with up to `max_rows` new rows per sequence, for the kernel that will run it."""
    g = max(1, hq // max(hkv, 1))
    cfg = cfgmod.current()
    if max_rows * g > 16 and _prefill_tensor_cores(k_pool, v_pool, d, cfg):
        return prefill_splits(batch, hq, hkv, d, max_rows, max_ctx)
    ctas = batch * hkv * max(1, max_rows // max(1, 32 // g))       # the general kernel takes up to 32 query rows per CTA
    if ctas >= NUM_SMS:
        return 1
    splits = choose_splits(batch, hkv, max_ctx)
    if max_rows * g > 16:
        # Ranges of less than 256 keys only while about four CTAs per SM run. NVFP4 pools, 40 / 8 and 24 / 4 heads of 128 and
        # 256: 100 rows over 2000 keys, 7 ranges 363 and 466 us, 18 and 31 ranges 413 and 582; 29 rows over 500 keys, one
        # range 178 and 251 us, 7 ranges 71 and 87.
        splits = min(splits, max(max_ctx // 256, 4 * NUM_SMS // ctas, 1))
    return splits


class AttnWorkspace:
    """Split-KV partial buffers, allocated once (stable addresses for CUDA graphs)."""

    def __init__(self, rows: int, hq: int, d: int, splits: int, device: torch.device):
        self.rows, self.splits = rows, splits
        self.part_o = torch.empty(rows, hq, splits, d, dtype=torch.float32, device=device)
        self.part_lse = torch.empty(rows, hq, splits, dtype=torch.float32, device=device)
        # arrivals per (sequence, kv head) of the fused split merge: zero between launches (the kernel re-arms it)
        self.counter = torch.zeros(rows * hq, dtype=torch.int32, device=device)


def paged_attention_ref(q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, kv_indices: torch.Tensor,
                        ctx_len: torch.Tensor, q_indptr: Optional[torch.Tensor], scale: float, kv_scale: float = 1.0,
                        causal: bool = True) -> torch.Tensor:
    t, hq, d = q.shape
    hkv = k_pool.shape[1]
    g = hq // hkv
    out = torch.zeros(t, hq, d, dtype=torch.float32, device=q.device)
    b = ctx_len.shape[0]
    for i in range(b):
        r0 = int(q_indptr[i]) if q_indptr is not None else i
        r1 = int(q_indptr[i + 1]) if q_indptr is not None else i + 1
        rows = r1 - r0
        ctx = int(ctx_len[i])
        if rows == 0 or ctx == 0:
            continue
        idx = kv_indices[i, :ctx].long()
        if getattr(k_pool, "sf", None) is not None:     # NVFP4 pool: packed values + block scales
            from ..cache.kv_pool import dequant_rows
            k = dequant_rows(k_pool[idx], k_pool.sf[idx], kv_scale)
            v = dequant_rows(v_pool[idx], v_pool.sf[idx], kv_scale)
        else:
            k = k_pool[idx].float() * kv_scale     # [ctx, hkv, d]
            v = v_pool[idx].float() * kv_scale
        qq = q[r0:r1].float().view(rows, hkv, g, d)
        s = torch.einsum("rhgd,chd->rhgc", qq, k) * scale
        if causal:
            pos = torch.arange(ctx, device=q.device)[None, :]
            lim = (ctx - rows + torch.arange(rows, device=q.device))[:, None]
            s = s.masked_fill((pos > lim)[:, None, None, :], float("-inf"))
        p = torch.softmax(s, dim=-1)
        out[r0:r1] = torch.einsum("rhgc,chd->rhgd", p, v).reshape(rows, hq, d)
    return out.to(q.dtype)


def paged_attention(q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, kv_indices: torch.Tensor,
                    ctx_len: torch.Tensor, *, q_indptr: Optional[torch.Tensor] = None, max_rows: int = 1,
                    seq_rows: Optional[torch.Tensor] = None,
                    scale: Optional[float] = None, kv_scale: float = 1.0, causal: bool = True, splits: int = 1,
                    workspace: Optional[AttnWorkspace] = None, out: Optional[torch.Tensor] = None,
                    quant_scale: Optional[torch.Tensor] = None, tables_ready: bool = False, rope: Optional[tuple] = None,
                    max_ctx: int = 0):
    """q [T, Hq, D] bf16; pools [slots, Hkv, D]; kv_indices [B, max_ctx] int32; ctx_len [B] int32.

    Row r of sequence b (rows q_indptr[b]..q_indptr[b+1], or exactly one row when q_indptr is None) sees keys
    [0, ctx_len[b] - rows_b + r + 1) when causal. `max_rows` bounds rows per sequence (host value).
    `seq_rows` int32 [B] selects each sequence's row of kv_indices (identity when None).
    `quant_scale` (fp32 scalar tensor): return the rows [T, Hq * D] as an Nvfp4Tensor quantised with that static
    scale (the activation operand of the output projection); on the decode kernel this and the split merge happen
    inside the attention kernel, elsewhere a quantisation pass follows.
    `tables_ready`: the tables and all keys and values but those of the call's own rows were complete before the forward began
    with its embedding gather (a decode step): the decode kernel then fetches them while its predecessors still run.
    `rope` = (qkv, positions, slots, inv_freq), where `rope_in_kernel` allows it: q is a view of the projection's rows, and
    rotation and KV write happen inside the kernel instead of in `basic.rope_kv_write`.
    `max_ctx` (host value) bounds the context lengths; 0: the width of kv_indices does.
    """
    t, hq, d = q.shape
    hkv = k_pool.shape[1]
    scale = 1.0 / math.sqrt(d) if scale is None else scale
    if not nv.use_native(q, k_pool):
        if rope is not None:
            raise ValueError("rope in the attention kernel: no such kernel on the CPU (see rope_in_kernel)")
        idx = kv_indices if seq_rows is None else kv_indices[seq_rows.long()]
        res = paged_attention_ref(q, k_pool, v_pool, idx, ctx_len, q_indptr, scale, kv_scale, causal)
        if out is not None:
            out.copy_(res)
            res = out
        return res if quant_scale is None else nvfp4.quantize(res.reshape(t, hq * d), quant_scale)
    b = ctx_len.shape[0]
    if splits > 1 and (workspace is None or workspace.rows < t or workspace.part_o.shape[1:] != (hq, splits, d)):
        workspace = AttnWorkspace(t, hq, d, splits, q.device)
    fp8 = k_pool.dtype != torch.bfloat16
    cfg = cfgmod.current()
    kernel = _decode_kernel(k_pool, v_pool, d, max_rows * (hq // hkv), cfg, q, out)
    if rope is not None and not (kernel == "mma" and tables_ready and q_indptr is None):
        raise ValueError("rope in the attention kernel: a decode step that rope_in_kernel() allows, with tables_ready")
    if kernel is not None:
        st = nv.device_state(q.device)
        f8, tc = fp8, kernel == "tc"
        fuse = cfg.fuse_epilogues and not tc and (cfg.fuse_attn_tail or splits == 1)
        xq = None
        if fuse:
            qb = sfb = None
            if quant_scale is not None:
                qb, sfb = _quant_bufs(t, hq * d, q.device)
                xq = nvfp4.Nvfp4Tensor(qb, sfb, quant_scale, t, hq * d)
            nv.lib().hb_attn_decode_fuse(workspace.counter.data_ptr() if splits > 1 else None, nv.ptr(qb), nv.ptr(sfb),
                                         nv.ptr(quant_scale), sfb.shape[1] if sfb is not None else 0)
        if xq is None:
            out = torch.empty(t, hq, d, dtype=q.dtype, device=q.device) if out is None else out
        # decode_attn = "tc" selects the persistent tcgen05 kernel (head dim 128; csrc/attn_decode_tc.cu). It
        # matches the mma.sync kernel in isolation (123 vs 122 us at 64 x 2304 keys) but not yet inside the 27B
        # decode step (18.8 vs 15.8 ms per step), so the mma.sync kernel stays the default.
        args = (q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), k_pool.stride(0), k_pool.stride(1),
                kv_indices.data_ptr(), kv_indices.stride(0), nv.ptr(seq_rows), ctx_len.data_ptr(), nv.ptr(q_indptr),
                nv.ptr(out), workspace.part_o.data_ptr() if splits > 1 else None,
                workspace.part_lse.data_ptr() if splits > 1 else None, b, max_rows, hq, hkv, d, splits, scale)
        tail = (int(causal), k_pool.shape[0], st.status.data_ptr(), nv.stream())
        if tables_ready and not tc:
            nv.lib().hb_attn_decode_early()
        if rope is not None:
            qkv, positions, slots, inv_freq = rope
            nv.lib().hb_attn_decode_rope(qkv.data_ptr(), qkv.stride(0), positions.data_ptr(), slots.data_ptr(),
                                         inv_freq.data_ptr(), 1.0 / kv_scale)
        code = (nv.lib().hb_attn_decode_tc(*args, *tail) if tc
                else nv.lib().hb_attn_decode(*args, int(f8), kv_scale, *tail))
        nv.check(code, "hb_attn_decode")
        if xq is not None:
            return xq
        if splits > 1 and not fuse:
            if quant_scale is not None and cfg.fuse_epilogues:
                # the merge kernel writes the NVFP4 rows itself: no separate quantisation pass
                qb, sfb = _quant_bufs(t, hq * d, q.device)
                nv.check(nv.lib().hb_attn_merge_quant(workspace.part_o.data_ptr(), workspace.part_lse.data_ptr(), t,
                                                      hq, splits, d, qb.data_ptr(), sfb.data_ptr(),
                                                      quant_scale.data_ptr(), sfb.shape[1], nv.stream()),
                         "hb_attn_merge_quant")
                return nvfp4.Nvfp4Tensor(qb, sfb, quant_scale, t, hq * d)
            nv.check(nv.lib().hb_attn_merge(workspace.part_o.data_ptr(), workspace.part_lse.data_ptr(),
                                            out.data_ptr(), t * hq, splits, d, nv.stream()), "hb_attn_merge")
        return out if quant_scale is None else nvfp4.quantize(out.view(t, hq * d), quant_scale)
    out = torch.empty_like(q) if out is None else out
    res = _paged_general(q, k_pool, v_pool, kv_indices, ctx_len, q_indptr, max_rows, seq_rows, scale, kv_scale, causal,
                         splits, workspace, out, cfg, fp8, b, t, hq, hkv, d, max_ctx or kv_indices.shape[1])
    return res if quant_scale is None else nvfp4.quantize(res.view(t, hq * d), quant_scale)


def rope_in_kernel(qkv: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, hq: int, hkv: int, d: int, rot: int) -> bool:
    """Whether a decode step (one row per sequence) may hand its projection's rows to `paged_attention(rope=...)`: the
    tensor-core decode kernel on a bf16 or e4m3 pool, all of the head rotated, no q / k norm or gate in the rows, 16-byte
    aligned rows everywhere."""
    cfg = cfgmod.current()
    if not nv.use_native(qkv, k_pool) or cfg.decode_attn == "tc" or _decode_kernel(k_pool, v_pool, d, hq // hkv, cfg, qkv) != "mma":
        return False
    return (rot == d and qkv.stride(0) % 8 == 0 and qkv.stride(1) == 1 and qkv.data_ptr() % 16 == 0
            and k_pool.stride() == v_pool.stride() and k_pool.stride(2) == 1 and k_pool.stride(0) % 8 == 0
            and k_pool.stride(1) % 8 == 0 and k_pool.data_ptr() % 16 == 0 and v_pool.data_ptr() % 16 == 0)


def _decode_kernel(k_pool: torch.Tensor, v_pool: torch.Tensor, d: int, rows: int, cfg, q: Optional[torch.Tensor] = None,
                   out: Optional[torch.Tensor] = None) -> Optional[str]:
    """Kernel for `rows` query rows per kv head: "mma" (csrc/attn_decode.cu), "tc" (csrc/attn_decode_tc.cu, `decode_attn` setting) or
    None, the prefill and general kernels."""
    if rows > 16 or getattr(k_pool, "sf", None) is not None:
        return None
    if k_pool.dtype != torch.bfloat16:
        return "mma" if _fp8_tensor_cores(k_pool, v_pool, d, cfg, q, out) else None
    return None if d not in (64, 128, 256) else "tc" if d == 128 and cfg.decode_attn == "tc" else "mma"


def _fp8_tensor_cores(k_pool: torch.Tensor, v_pool: torch.Tensor, d: int, cfg, q: Optional[torch.Tensor] = None,
                      out: Optional[torch.Tensor] = None) -> bool:
    """Whether an e4m3 pool takes the tensor-core kernels: whole 128-byte column blocks per row and rows on 16-byte
    boundaries (bulk copies), query and output rows on 16-byte boundaries (16-byte accesses; the general kernel reads and
    writes them element by element). Under `stable_numerics` the general kernel stays: it sums a row's keys in the same order
    however many rows share the call, the tensor-core kernels have one form for up to 8 and one for up to 16 rows."""
    return (k_pool.dtype == torch.float8_e4m3fn and d in (128, 256) and not cfg.stable_numerics
            and k_pool.stride(0) % 16 == 0 and k_pool.stride(1) % 16 == 0 and k_pool.stride(2) == 1
            and v_pool.stride() == k_pool.stride()
            and k_pool.data_ptr() % 16 == 0 and v_pool.data_ptr() % 16 == 0
            and all(x is None or x.data_ptr() % 16 == 0 for x in (q, out)))


def _prefill_tensor_cores(k_pool: torch.Tensor, v_pool: torch.Tensor, d: int, cfg, q: Optional[torch.Tensor] = None,
                          out: Optional[torch.Tensor] = None) -> bool:
    """Whether more than 16 query rows per kv head run in csrc/attn_prefill.cu."""
    if getattr(k_pool, "sf", None) is not None or cfg.prefill_attn != "tc":
        return False
    return d in (64, 128, 256) if k_pool.dtype == torch.bfloat16 else _fp8_tensor_cores(k_pool, v_pool, d, cfg, q, out)


_QUANT_BUFS: dict = {}


def _quant_bufs(rows: int, k: int, device):
    """Persistent NVFP4 output buffers per shape (stable addresses for captured graphs); padding scales zeroed once."""
    key = (device, rows, k)
    bufs = _QUANT_BUFS.get(key)
    if bufs is None:
        qb, sfb = nvfp4._alloc(rows, k, device)
        sfb.zero_()
        bufs = _QUANT_BUFS[key] = (qb, sfb)
    return bufs


def _paged_general(q, k_pool, v_pool, kv_indices, ctx_len, q_indptr, max_rows, seq_rows, scale, kv_scale, causal,
                   splits, workspace, out, cfg, fp8, b, t, hq, hkv, d, max_ctx):
    if getattr(k_pool, "sf", None) is not None:
        fp8 = 2       # NVFP4 pool: the split-KV kernel dequantises rows as it loads them
        nv.lib().hb_attn_fp4_scales(k_pool.sf.data_ptr(), v_pool.sf.data_ptr(), k_pool.sf.stride(0), k_pool.sf.stride(1))
    if q_indptr is not None and _prefill_tensor_cores(k_pool, v_pool, d, cfg, q, out):
        st = nv.device_state(q.device)
        parts = (workspace.part_o.data_ptr(), workspace.part_lse.data_ptr()) if splits > 1 else (None, None)
        if splits <= 1:      # 1: two Q tiles per CTA, 0: one
            splits = int(two_q_tiles(b, hq, hkv, max_rows, max_ctx))
        nv.check(nv.lib().hb_attn_prefill(
            q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), k_pool.stride(0), k_pool.stride(1), kv_indices.data_ptr(),
            kv_indices.stride(0), nv.ptr(seq_rows), ctx_len.data_ptr(), q_indptr.data_ptr(), out.data_ptr(), *parts, splits,
            b, max_rows, hq, hkv, d, scale, int(fp8), kv_scale, int(causal), k_pool.shape[0], st.status.data_ptr(),
            nv.stream()), "hb_attn_prefill")
        if splits > 1:
            nv.check(nv.lib().hb_attn_merge(*parts, out.data_ptr(), t * hq, splits, d, nv.stream()), "hb_attn_merge")
        return out
    nv.check(nv.lib().hb_attn_paged(
        q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), k_pool.stride(0), k_pool.stride(1), kv_indices.data_ptr(),
        kv_indices.stride(0), nv.ptr(seq_rows), ctx_len.data_ptr(), nv.ptr(q_indptr), out.data_ptr(),
        workspace.part_o.data_ptr() if splits > 1 else None, workspace.part_lse.data_ptr() if splits > 1 else None,
        b, t, max_rows, hq, hkv, d, splits, scale, int(fp8), kv_scale, int(causal), nv.stream()), "hb_attn_paged",
             launches=2 if splits > 1 else 1)
    return out


TC_PROFILE_FIELDS = ("producer_wait", "tiles_tma", "tiles_gather", "issuer_wait_full", "issuer_wait_p",
                     "softmax_wait_s", "softmax_wait_pv", "epilogue", "softmax_total", "raises", "tiles", "ctas")


class DecodeTcProfile:
    """Role counters of the tcgen05 decode kernel (csrc/attn_decode_tc.cu), accumulated while the object lives."""

    def __init__(self, device):
        self.buf = torch.zeros(len(TC_PROFILE_FIELDS), dtype=torch.int64, device=device)
        nv.lib().hb_attn_decode_tc_profile(self.buf.data_ptr())

    def read(self) -> dict:
        torch.cuda.synchronize(self.buf.device)
        c = dict(zip(TC_PROFILE_FIELDS, self.buf.tolist()))
        tiles, ctas = max(c["tiles"], 1), max(c["ctas"], 1)
        out = {k: round(c[k] / tiles) for k in ("producer_wait", "issuer_wait_full", "issuer_wait_p",
                                                "softmax_wait_s", "softmax_wait_pv")}
        out.update(epilogue_per_cta=round(c["epilogue"] / ctas), total_per_cta=round(c["softmax_total"] / ctas),
                   tiles_per_cta=round(tiles / ctas, 1), raises_per_tile=round(c["raises"] / tiles, 3),
                   gather_share=round(c["tiles_gather"] / max(c["tiles_gather"] + c["tiles_tma"], 1), 3))
        return out

    def close(self) -> None:
        nv.lib().hb_attn_decode_tc_profile(None)
