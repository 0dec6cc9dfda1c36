"""Grouped bf16 GEMMs of the expert MLP on the tcgen05 kernel (forward, dgrad, wgrad).

Rows of all groups live in one matrix; ``group_off`` (int32[G+1], device) gives each group's row
range and every offset is a multiple of 128, so tiles never straddle two groups and the rows
between a group's real end and its padded end are zero.
"""
from __future__ import annotations

from typing import Optional

import torch

from .. import runtime
from ..utils.config import CONFIG

FORWARD, DGRAD, WGRAD = 0, 1, 2
STORE, SWIGLU, SWIGLU_BWD = 0, 1, 2
_BM, _BN, _BK = 128, 256, 64
# CTA-pair kernel (256 x 256 tiles, cta_group::2); set False to fall back to the one-CTA kernel.
USE_PAIR = CONFIG.gemm != "one"
# Rows of a raster band (see csrc/kernels/gemm_common.cuh); 0 = kernel default.
BAND_ROWS = CONFIG.band_rows
# CTA-pair weight gradients: True = epilogue threads write global memory row by row; False = staged tiles + TMA stores.
DIRECT_EPILOGUE = False


def row_align() -> int:
    """Rows every group must be padded to for the kernel in use."""
    return 256 if USE_PAIR else 128


_status = None
_maps: dict = {}


def _st():
    global _status
    if _status is None:
        _status = runtime.ext().StatusBlock()
    return _status


def check() -> None:
    """Raise if a GEMM launched through this module gave up on an mbarrier wait."""
    code, site, detail, seen, want = _st().read()
    if code:
        raise runtime.CollectiveTimeout(code, site, detail, seen, want)


def _tmap(t: torch.Tensor, box_rows: int):
    assert t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1
    key = (t.data_ptr(), t.shape[0], t.shape[1], t.stride(0), box_rows)
    m = _maps.get(key)
    if m is None:
        if len(_maps) > 4096:
            _maps.clear()
        m = runtime.ext().TensorMap2D(t.data_ptr(), t.shape[0], t.shape[1], t.stride(0), 64, box_rows)
        _maps[key] = m
    return m


def _out_maps(c: torch.Tensor, c2: Optional[torch.Tensor]):
    """Tensor maps of the outputs for the CTA-pair kernel's TMA stores (boxes of 64 columns x 128 rows)."""
    if not USE_PAIR:
        return None, None
    return _tmap(c, _BM), (_tmap(c2, _BM) if c2 is not None else None)


def _ctas() -> int:
    return torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count


def pad_group_offsets(counts: torch.Tensor) -> torch.Tensor:
    """int32[G+1] offsets with every group rounded up to row_align() rows (host/torch helper for tests)."""
    ra = row_align()
    padded = (counts.to(torch.int64) + ra - 1) // ra * ra
    off = torch.zeros(counts.numel() + 1, dtype=torch.int64, device=counts.device)
    off[1:] = torch.cumsum(padded, 0)
    return off.to(torch.int32)


def _tmap_bytes(t: torch.Tensor, box_rows: int):
    assert t.dtype == torch.uint8 and t.dim() == 2 and t.stride(1) == 1
    key = (t.data_ptr(), t.shape[0], t.shape[1], t.stride(0), box_rows, "u8")
    m = _maps.get(key)
    if m is None:
        m = runtime.ext().TensorMap2D.bytes(t.data_ptr(), t.shape[0], t.shape[1], t.stride(0), box_rows)
        _maps[key] = m
    return m


class TokScratch:
    """Arrival counters of the token-major kernel's partial tiles, kept by a caller that launches it again and again on one
    stream (an engine): one half serves a launch, which clears the other half for the next. Without it a launch clears its own."""

    def __init__(self, device):
        self.ctas = torch.cuda.get_device_properties(device).multi_processor_count
        self.counters = torch.zeros(2, self.ctas * runtime.ext().TOK_COUNTERS_PER_CTA, dtype=torch.int32, device=device)
        self.parity = 0
        # True while weights and group tables are older than the kernel that a launch follows in the stream (an engine whose routing
        # lies behind its dispatch): the launch may then start on them before that kernel has ended.
        self.early = False
        self.plans: dict = {}   # (mode, epilogue) -> the plan of the last launch; asked whether it fits before every other


_plans: dict = {}


def wide_tiles(epi: int, reduction: int, mean_rows: int, waves: float) -> bool:
    """Whether tiles of 512 tokens are taken instead of 256 for groups of about ``mean_rows`` rows (grouped_gemm_tokens.cu says what they
    save); ``waves`` is how many rounds of the GPU they make. What they save is power, so they are ahead in a stream of GEMMs and behind, or even,
    in a launch that follows other work; the lines lie where the first is several per cent and the second about nothing. us, 256 -> 512 tokens.

    SwiGLU forward: where a group fits one wide tile but not one of 256, and tiles are many. In a stream / after other work, 264, 320, 400, 440 rows:
    32 experts of 7168 x 2048 505 -> 477, 568 -> 534, 635 -> 603, 689 -> 663 / 497 -> 491, 562 -> 552, 640 -> 662, 695 -> 734; 10 of 4096 x 5632 (6
    waves) 265 -> 250, 290 -> 271, 327 -> 315 / 251 -> 251, 279 -> 271, 292 -> 302. Few tiles: 2 experts of 4096 x 2048 24 -> 48, 16 of them (3.5 waves)
    173 -> 183, 2 of 4096 x 14336 (3 waves) 157 -> 158 / 164 -> 166.
    Others: where tiles are long (the reduction) and many (the rows). 8 experts, reduction of 28672 with 440, 560, 750, 832, 2048 rows 682 -> 874, 870 -> 840,
    1182 -> 1060, 1246 -> 1145, 2966 -> 2778 / 560 rows 867 -> 926, 750 and 832 1151 -> 1139, 1285 -> 1215; of 14336 with 640, 1024, 1536, 4096 rows
    470 -> 450, 718 -> 718, 1111 -> 1053, 2796 -> 2460 / 454 -> 476, 741 -> 773, 1128 -> 1154; of 4096 with the SwiGLU backward and 4096, 8192 rows 2973 ->
    2794, 5912 -> 5426 / 3130 -> 3134, 6623 -> 6656. Below three waves (2 experts, 14336, 1536 and 3000 rows) 263 -> 279, 501 -> 494 / 310 -> 370,
    494 -> 554. Whole training steps of 1800 tokens (450 rows) with the data gradient of W13 wide 9920 -> 10190, of 12000, 16384, 32768 tokens
    against no wide tiles at all 26740 -> 25920, 34750 -> 33330, 66200 -> 61230. Shorter reductions lose at any size (plain, 3584 with 4096 rows 178 -> 189; a whole SwiGLU layer, 1024 with 444 rows 115 -> 122)."""
    if reduction < 4096:
        return False
    if epi == SWIGLU:
        return 272 <= mean_rows <= 368 and waves >= 5.5
    return mean_rows * reduction >= 16 << 20 and waves >= (3 if reduction >= 8192 else 6)


def _plan_key(mode: int, epi: int, granule: int, w: torch.Tensor, x: torch.Tensor, out: torch.Tensor, gu: Optional[torch.Tensor]) -> tuple:
    """Everything that a ``TokGemmPlan`` is made from or refuses by: another view, shape, type or device at the same address is
    another plan (or none)."""
    return (mode, epi, granule, BAND_ROWS, w.data_ptr(), w.dtype, w.shape, w.stride(), w.get_device(), x.data_ptr(), x.dtype, x.shape, x.stride(), x.get_device(),
            out.data_ptr(), out.dtype, out.shape, out.stride(), out.get_device(),
            None if gu is None else (gu.data_ptr(), gu.dtype, gu.shape, gu.stride(), gu.get_device()))


def wide_columns(row_tiles: int, columns: int, pairs: int, mean_rows: int) -> bool:
    """Whether weight gradients take tiles of 512 columns instead of 256 (grouped_gemm_pair.cu). Few rows: the tile's way out is the time, and half
    as many pass through; but tiles twice as large can leave more of the last wave idle, or of the only one. Many: the power cap is, and operand
    traffic saved is clock won. Between them neither, and two tiles of 256 in turn keep the tensor cores busier. us after other work, 256 -> 512 columns,
    16, 256, 500, 600, 660, 1600 rows: 8 experts of 4096 x 14336 277 -> 201, 368 -> 263, 460 -> 416, 508 -> 495, 532 -> 529, 1058 -> 1123; 32 of 1024 x 2048 (14 waves
    to 7) 54 -> 42, 61 -> 49, 76 -> 66, 78 -> 76, 80 -> 80, 177 -> 185; 8 of 2048 x 2048 (7 to 4) 28.7 -> 24.6, 32.8 -> 30.8, 41 -> 41, 43 -> 45, 45 -> 49, 74 -> 84; 4 of
    them (4 to 2) 20.5 -> 18.5, 22.6 -> 20.5, 26.6 -> 26.6, 28.7 -> 28.7, 28.7 -> 30.7, 47 -> 49; 8 of 1024 x 1024 (2 to 1) 14.3 -> 14.3, 16.4 -> 16.4, 18.4 -> 20.5;
    2 of them (1 to 1) 12.3 -> 14.3, 12.3 -> 16.3, 14.3 -> 18.4. In a stream, W13 of 8 of 4096 x 14336 with 1536, 2048, 4096, 8192 rows 1920 -> 1892, 2486 -> 2447,
    4897 -> 4850, 12177 -> 11402; whole training steps of 8192 tokens (2048 rows) 20050 -> 20065."""
    if columns % 512:
        return False
    narrow, wide = (-(-row_tiles * (columns // n) // pairs) for n in (256, 512))
    if mean_rows < 512:
        return narrow >= 4 and 14 * wide <= 8 * narrow
    return (narrow >= 14 if mean_rows <= 640 else mean_rows >= 1536) and 50 * wide <= 26 * narrow


def token_tile(epi: int, reduction: int, most_rows: int, mean_rows: int, groups: int, features: int, pairs: int) -> int:
    """Most tokens of a tile. Where no group can have more than a narrow tile holds, narrow tiles leave shared memory to the weights in flight."""
    if 0 < most_rows <= 128:
        return 64 if most_rows <= 64 else 128
    waves = groups * -(-mean_rows // 512) * (features / 256) / pairs
    return 512 if wide_tiles(epi, reduction, mean_rows, waves) else 256


def group_rows_hint(mean_rows: int, rows: int, groups: int, live_rows) -> int:
    """About how many rows a group has: the caller's ``mean_rows``, else those that the matrix holds, unless ``live_rows`` says that these
    are a capacity: then 0, unknown, and tiles are those that suit any number."""
    return mean_rows or (rows // groups if live_rows is None else 0)


def _tok_run(mode: int, epi: int, w: torch.Tensor, x: torch.Tensor, out: torch.Tensor, gu: Optional[torch.Tensor], group_off: torch.Tensor, live_rows,
             granule: int, timeout_s: float, ctas: Optional[int], gate, gate_tile_rows: int, scratch: Optional[TokScratch], most_rows: int = 0,
             mean_rows: int = 0) -> None:
    plan = scratch.plans.get((mode, epi)) if scratch is not None else None
    if plan is None or not plan.matches(w, x, out, gu, granule, BAND_ROWS):
        key = _plan_key(mode, epi, granule, w, x, out, gu)
        plan = _plans.get(key)
        if plan is None:
            if len(_plans) > 1024:
                _plans.clear()
            plan = _plans[key] = runtime.ext().TokGemmPlan(mode, epi, w, x, out, gu, granule, BAND_ROWS)
        if scratch is not None:
            scratch.plans[mode, epi] = plan
    n = scratch.ctas if scratch is not None else _ctas()
    counter_ptr, target = gate or (0, None)
    counters, parity, early = None, 0, False
    if scratch is not None:
        scratch.parity ^= 1
        counters, parity, early = scratch.counters, scratch.parity, scratch.early
    tile_n = token_tile(epi, x.shape[1], most_rows, group_rows_hint(mean_rows, x.shape[0], w.shape[0], live_rows), w.shape[0], w.shape[1 + mode], n // 2)
    plan.run(group_off, live_rows, _st().ptr(), int(timeout_s * 1e9), min(ctas or n, n), counter_ptr, target, gate_tile_rows, counters, parity, tile_n, early)


def grouped_gemm_fwd(a: torch.Tensor, w: torch.Tensor, group_off: torch.Tensor, out: torch.Tensor, swiglu: bool = False,
                     gate_up_out: Optional[torch.Tensor] = None, timeout_s: float = 5.0, gate=None, a_scales: Optional[torch.Tensor] = None,
                     group_rows: Optional[torch.Tensor] = None, gate_tile_rows: int = 0, ctas: Optional[int] = None,
                     live_rows: Optional[torch.Tensor] = None, granule: int = 32, scratch: Optional[TokScratch] = None, most_rows: int = 0,
                     mean_rows: int = 0) -> torch.Tensor:
    """out[rows of g] = a[rows of g] @ w[g].T  (a [R, K], w [G, N, K], out [R, N]).

    With ``swiglu`` the N columns of every 256-wide tile are [128 gate | 128 up] of the same 128
    features and ``out`` is [R, N/2] = silu(gate) * up; ``gate_up_out`` ([R, N]) optionally keeps
    the raw tile for the backward pass. ``gate=(counter_ptr, target)`` makes the TMA producer
    wait, group by group, until ``counter[g] >= target[g]`` (rows pushed by peers have landed);
    with ``gate_tile_rows`` > 0 the counters are per tile of that many rows of ``a`` instead of per
    group, so a tile is loaded as soon as its own rows are in.

    ``a`` may be uint8 e4m3 rows with ``a_scales`` (float [R, K/128], one scale per 128 elements):
    the CTA-pair kernel then converts them to bf16 tiles in shared memory on the way to the tensor
    core (no dequantised copy of ``a`` exists in global memory). ``group_rows`` (int32[G], real rows
    per group) makes that path treat the rows between a group's real and padded end as zeros.

    ``live_rows`` (int32[G], real rows per group; CTA-pair kernels, bf16 ``a``): only these rows, up to a multiple of
    ``granule`` (32 or 64), are computed and written. ``scratch``: see ``TokScratch``. ``most_rows`` > 0: no group has more real
    rows than this; ``mean_rows`` > 0: about how many they have (hints that size the tiles; the result does not depend on them but for
    the rounding of sums that are cut into parts).
    """
    G, N, K = w.shape
    assert a.shape[1] == K and K % _BK == 0 and N % _BN == 0 and a.shape[0] % _BM == 0
    assert out.shape[0] == a.shape[0] and out.shape[1] == (N // 2 if swiglu else N)
    if USE_PAIR and a.dtype == torch.bfloat16:
        assert a_scales is None
        _tok_run(FORWARD, SWIGLU if swiglu else STORE, w, a, out, gate_up_out, group_off, live_rows, granule, timeout_s, ctas, gate, gate_tile_rows, scratch, most_rows, mean_rows)
        return out
    C = runtime.ext()
    map_b = _tmap(w.view(G * N, K), 128 if USE_PAIR else _BN)
    if a.dtype == torch.uint8:
        assert USE_PAIR and a_scales is not None and K % 128 == 0 and a.is_contiguous(), "e4m3 operand: CTA-pair kernel, scales given, K a multiple of 128"
        map_a = _tmap_bytes(a, _BM)
    else:
        assert a_scales is None
        map_a = _tmap(a, _BM)
    C.grouped_gemm(FORWARD, SWIGLU if swiglu else STORE, map_a, map_b, group_off, N // _BN, 0, K, N,
                   0, out, gate_up_out, _st().ptr(), int(timeout_s * 1e9), min(ctas or _ctas(), _ctas()), *(gate or (0, None)), USE_PAIR, BAND_ROWS,
                   *_out_maps(out, gate_up_out), DIRECT_EPILOGUE and a_scales is None, a_scales, group_rows, gate_tile_rows)
    return out


def grouped_gemm_dgrad(dy: torch.Tensor, w: torch.Tensor, group_off: torch.Tensor, out: torch.Tensor, timeout_s: float = 5.0, gate=None,
                       swiglu_bwd_of: Optional[torch.Tensor] = None, live_rows: Optional[torch.Tensor] = None, granule: int = 64,
                       scratch: Optional[TokScratch] = None, most_rows: int = 0, mean_rows: int = 0) -> torch.Tensor:
    """out[rows of g] = dy[rows of g] @ w[g]  (dy [R, N], w [G, N, K], out [R, K]).

    With ``swiglu_bwd_of`` (the saved gate|up tiles [R, 2K]) the product is taken as d(act) and the
    epilogue writes d(gate|up) [R, 2K] into ``out`` instead (CTA-pair kernel only): the SwiGLU
    backward costs no extra pass over memory. ``live_rows``, ``granule``, ``scratch``, ``most_rows``, ``mean_rows``: as in ``grouped_gemm_fwd``.
    """
    G, N, K = w.shape
    assert dy.shape[1] == N and N % _BK == 0 and K % _BN == 0 and dy.shape[0] % _BM == 0
    if swiglu_bwd_of is not None:
        assert USE_PAIR and out.shape[1] == 2 * K and swiglu_bwd_of.shape == out.shape
    if USE_PAIR:
        _tok_run(DGRAD, SWIGLU_BWD if swiglu_bwd_of is not None else STORE, w, dy, out, swiglu_bwd_of, group_off, live_rows, granule, timeout_s, None, gate, 0, scratch, most_rows, mean_rows)
        return out
    C = runtime.ext()
    C.grouped_gemm(DGRAD, STORE, _tmap(dy, _BM), _tmap(w.view(G * N, K), _BK), group_off, K // _BN, 0, N, N, 0, out, None, _st().ptr(),
                   int(timeout_s * 1e9), _ctas(), *(gate or (0, None)), USE_PAIR, BAND_ROWS, *_out_maps(out, None), DIRECT_EPILOGUE)
    return out


def grouped_gemm_wgrad(dy: torch.Tensor, x: torch.Tensor, group_off: torch.Tensor, out: torch.Tensor, timeout_s: float = 5.0,
                       live_rows: Optional[torch.Tensor] = None, mean_rows: int = 0) -> torch.Tensor:
    """out[g] = dy[rows of g].T @ x[rows of g]  (dy [R, N], x [R, K], out [G, N, K]). ``mean_rows`` as in ``grouped_gemm_fwd``. Rows between a
    group's real end and its padded end must be zero in at least one operand and finite in both; with ``live_rows``
    (int32[G], real rows per group) that holds for the rows up to the next multiple of 64, the others are not read."""
    G, N, K = out.shape
    bm = 256 if USE_PAIR else _BM
    assert dy.shape[1] == N and x.shape[1] == K and N % bm == 0 and K % _BN == 0
    C = runtime.ext()
    mean = group_rows_hint(mean_rows, x.shape[0], G, live_rows)
    wide = USE_PAIR and not DIRECT_EPILOGUE and (mean > 0 or live_rows is None) and wide_columns(G * (N // bm), K, _ctas() // 2, mean)
    C.grouped_gemm(WGRAD, STORE, _tmap(dy, _BK), _tmap(x, _BK), group_off, K // (512 if wide else _BN), N // bm, 0, 0, N, out.view(G * N, K), None, _st().ptr(),
                   int(timeout_s * 1e9), _ctas(), 0, None, USE_PAIR, BAND_ROWS, *((_tmap(out.view(G * N, K), 32), None) if wide else _out_maps(out.view(G * N, K), None)), DIRECT_EPILOGUE, None, live_rows, 0, wide)
    return out
