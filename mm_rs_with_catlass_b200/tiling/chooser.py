"""Runtime tiling chooser: (op, M, N, K, world, dtype) -> :class:`TilingConfig`.

Order of precedence: an exact hit in the measured table, the nearest measured shape of the
same op / world / dtype in log-space (within a factor of two per dimension), then a heuristic
from a measured cost model: waves of tiles x the time of one wave, where a narrow tile costs far
more than its share of the output (it re-reads A once per column tile), so the widest tile wins
unless it leaves most SMs idle.

The reference only has the offline half of this (a sweep whose best rows are picked by hand,
examples/dynamic_tiling/utils/get_best_res.py:43-83; the default it falls back to is a
constant, examples/dynamic_tiling/dynamic_tiling.cpp:219-227).
"""
from __future__ import annotations

import functools
import math
import os
from typing import Optional

import torch

from .config import TilingConfig
from . import table as _table

_NUM_SMS = 148


# Measured on B200 (bf16, CUDA-graph replay): time of one wave of tiles relative to the 128 x 256
# single-CTA tile, per unit of output. Narrow tiles re-read A from L2 once per column tile and are
# bound by the fill rate of shared memory, so halving the width costs far more than half.
_TILE_EFF = {256: 1.0, 192: 0.85, 128: 0.56, 64: 0.43}
_PAIR_GAIN = {256: 1.18, 192: 1.18, 128: 1.35}     # 2-CTA tiles: each CTA fills half of B (192: pairs only)
# int8: a pair of 256 columns in a single wave loses to 128-column tiles (256 x 8192 x 1024: 16.4 against 12.8 us, 205 x 8192 x
# 3584: 21.8 against 19.9), and over several waves the choice is the same with either figure
_PAIR_GAIN_INT8 = {256: 1.10, 128: 1.35}
_PAIR_GAIN_FUSED = {256: 1.10, 128: 1.35}          # ... of a launch that also communicates (measured on 2 to 8 GPUs)


# Cost model of split_k, in SM cycles, fitted to 84 shapes (bf16 and int8; 4 to 1024 rows, N of 992 to 28672, K of 3584 to
# 28672): its choices lose 2 % on average against the best of all cuts that were measured, the direct kernel alone 28 %.
_TAIL_INT8 = 12000.0              # int8 products gain that much less from a cut tail than the model says (fitted)
_TAIL_INTAKE = 52.0               # the same for a pair tile of a product that fills the GPU
_INTAKE = {1: 46.0, 2: 42.0}      # bytes per cycle that one CTA takes in while most of the others do the same (pair: per CTA)
_HBM = 3600.0                     # bytes per cycle from HBM, all SMs
_PLANES = 3500.0                  # bytes per cycle of the planes, written and read through L2
_DOUBLE_EPILOGUE = 2500.0         # what a double tile's epilogue leaves uncovered
_LAUNCH = 10000.0                 # start, fill and drain of a kernel
_FOLD = 8000.0                    # the second kernel and the gap before it
_INT8_EPILOGUE = 10000.0          # the dequantising epilogue of the direct kernel, which the second kernel spreads over all SMs


def tile_cost(seg_rows: int, nseg: int, n: int, bn: int, pair: int, seg_cols: bool = False,
              gain: Optional[dict] = None) -> float:
    """Relative time of a GEMM whose rows come in ``nseg`` segments of ``seg_rows`` rows (tiles never
    straddle segments): waves of tiles x time of one wave. With ``seg_cols`` the output is cut into
    ``nseg`` column segments instead and ``seg_rows`` is the full row count."""
    bm = 128 * pair
    if seg_cols:
        tiles = math.ceil(seg_rows / bm) * nseg * math.ceil(math.ceil(n / nseg) / bn)
    else:
        tiles = nseg * math.ceil(seg_rows / bm) * math.ceil(n / bn)
    units = _NUM_SMS // pair
    waves = math.ceil(tiles / units)
    eff = _TILE_EFF[bn] * ((gain or _PAIR_GAIN)[bn] if pair == 2 else 1.0)
    return waves * bn / eff


@functools.lru_cache(maxsize=4096)
def tail_cut(m: int, n: int, k: int, elt: int, bn: int):
    """A local product on pair tiles (256 x bn): ``(waves, cut)`` with ``cut = (first, slices, k_slice)``
    when the tiles from ``first`` on, its last and nearly empty wave, are worth cutting along K so that
    they spread over all SMs, else None; ``waves`` is what the product then costs, in waves of tiles.

    The cut pays for its planes (written and read through L2) and for a second kernel, so it needs a long
    K. bf16 1024 x 5120 x 6144 (80 tiles on 74 pairs): 81 -> 64 us; 600 x 8192 x 14336: 149 -> 134 us; int8
    600 x 8192 x 14336: 101 -> 91 us; over 28 shapes the choice is within 5 % of the better form."""
    units = _NUM_SMS // 2
    tiles = -(-m // 256) * -(-n // bn)
    first, rest = tiles // units * units, tiles % units
    waves, kb = -(-tiles // units), -(-k * elt // 128)
    wave_time = kb * max(2.0 * bn, (128 + bn // 2) * 128 / _TAIL_INTAKE)
    best, best_time = None, 0.96 * (waves * wave_time + _LAUNCH)
    for s in range(2, 25) if rest else ():
        kbs = -(-(-(-kb // s)) // 2) * 2                      # K blocks per slice: whole pair stages
        if kbs < 8 or -(-kb // kbs) != s:
            continue
        t = first // units * wave_time + -(-rest * s // units) * kbs * wave_time / kb
        t += rest * s * 256.0 * bn * 8 / _PLANES + _LAUNCH + _FOLD + (_TAIL_INT8 if elt == 1 else 0.0)
        if t < best_time:
            best, best_time = (first, s, kbs * 128 // elt), t
    return (waves, None) if best is None else ((best_time - _LAUNCH) / wave_time, best)


@functools.lru_cache(maxsize=16384)
def double_plan(rows: int, cols: int, k: int, elt: int, bn: int, rows_k_major: bool = True):
    """A local product on double tiles, 256 ``rows`` x 2 bn ``cols``: ``(cycles, cut)`` with ``cut = (slices, k_slice)`` when the
    units of 256 x bn past the last full wave are worth cutting along K, else None.

    A K block of a double tile takes 122 + 3.8 bn cycles (bn 256: 1096, 192: 865; its MMAs: 4 bn), never less than the 610 of
    its issue. One of a unit by itself takes what its loads' latency leaves: 780 above 160 columns, else 560, or 660 where the
    operand under the rows is not K-contiguous (operands of zeros, K of 4096 to 8192)."""
    workers = _NUM_SMS // 2
    rt, ct, kb = -(-rows // 256), -(-cols // bn), -(-k * elt // 128)
    total = rt * ct
    twice, once = max(610.0, 122 + 3.8 * bn), 780.0 if bn > 160 else 560.0 if rows_k_major else 660.0

    def whole(units):          # the busiest pair, as the units are dealt out (double_item in csrc/include/catcoc/sched.h)
        waves = -(-units // workers)
        doubles = min(rt * (ct // 2), waves // 2 * workers, units // 2)
        singles, per, r = units - 2 * doubles, doubles // workers, doubles % workers
        level = min(singles, 2 * (workers - r)) if r else 0
        light = per * twice + -(-level // (workers - r)) * once
        heavy = (per + (r > 0)) * twice
        return kb * (max(heavy, light) + -(-(singles - level) // workers) * once) + (per + (r > 0)) * _DOUBLE_EPILOGUE

    hbm = (rows + cols) * k * elt / _HBM
    best, best_time = None, max(hbm, whole(total)) + _LAUNCH
    rest = total % workers
    full = whole(total - rest)
    for s in range(2, 33) if rest else ():
        kbs = -(-kb // s)
        if kbs < 8 or -(-kb // kbs) != s:
            continue
        t = max(hbm, full + -(-rest * s // workers) * kbs * once) + rest * s * 256.0 * bn * 8 / _PLANES + _LAUNCH + 2 * _FOLD
        if t < 0.94 * best_time:
            best, best_time = (s, kbs * 128 // elt), t
    return best_time, best


def double(m: int, n: int, k: int, elt: int, b_k_major: bool, swap: bool, limit: float) -> Optional[TilingConfig]:
    """The best tiling on double tiles whose predicted cycles are below ``limit``, else None. With B stored [K, N] the halves must
    be whole 128-byte blocks of columns for every CTA (192 columns: 3890 us where 256 take 3250, bf16 8192 x 28672 x 8192); with
    ``swap`` the output's rows may run along the tiles' columns, whose width then fits them: int8 614 x 8192 x 7168: 48 -> 32 us,
    bf16 302 x 14336 x 8192: 116 -> 74 us, 106 x 14336 x 8192 with B [N, K]: 58 -> 49 us.

    Over 120 shapes that this rule sends here (129 to 16384 rows, bf16 and int8, both storages of B) the product is 12 % faster
    on average than on the other tiles, in a loop; the worst lost 3 %."""
    best = None
    for turned in (False, True):
        if (turned and not swap) or (m <= 128 and not (turned and b_k_major)):
            continue           # few rows on the tiles' rows are mostly padding, and a [K, N] weight under them is slower to load
        rows, cols = (n, m) if turned else (m, n)
        for bn in ((256, 224, 192, 160, 128, 96, 64) if b_k_major or turned else (256,)):
            if bn > 64 and bn >= cols + 32:
                continue
            t, cut = double_plan(rows, cols, k, elt, bn, b_k_major if turned else True)
            # the cluster's start, an epilogue that nothing covers; turning the tile
            t += (5500.0 if turned else 4500.0) + (_INT8_EPILOGUE if elt == 1 else 0.0)
            if t < limit:
                limit, best = t, (bn, turned, cut)
    if best is None:
        return None
    bn, turned, cut = best
    return TilingConfig(bn=bn, swizzle=4, cta_pair=2, twice=True, swap=turned, cut_slices=cut[0] if cut else 0,
                        cut_k=cut[1] if cut else 0)


def heuristic(op: str, m: int, n: int, k: int, world: int, dtype: torch.dtype, b_k_major: bool = False,
              tails: bool = False) -> TilingConfig:
    """``tails``: the caller cuts the last wave along K where that pays (:func:`tail_cut`).
    ``b_k_major``: the caller can launch 192-column pair tiles, i.e. a local product with a B stored
    [N, K]. They fill waves that 256 columns leave nearly empty (8144 x 1696 x 5120: 124 -> 115 us;
    1024 x 5120 x 6152: 93 -> 85 us); single 192-column tiles were never the best of 20 shapes."""
    rows = m
    fused = world > 1 and op in ("matmul_reduce_scatter", "quant_matmul_reduce_scatter", "matmul_allreduce",
                                 "allgather_matmul")
    nseg = world if fused else 1
    seg_rows = max(1, rows // nseg)
    allreduce = op == "matmul_allreduce" and world > 1
    ar_cols = allreduce and n % (world * 8) == 0     # the all-reduce then splits ownership by columns
    if ar_cols:
        seg_rows = rows
    forced = os.environ.get("CATCOC_CTA_PAIR")
    best = None
    gain = _PAIR_GAIN_FUSED if fused else _PAIR_GAIN_INT8 if dtype == torch.int8 else _PAIR_GAIN
    for pair in (2, 1):
        if forced in ("1", "2") and pair != int(forced):
            continue
        if pair == 2 and ((seg_rows < 256 or seg_rows % 256 != 0) if fused else seg_rows <= 128):
            # ragged 256-row tiles of a segment are mostly padding; a local product has one ragged row of them
            # (8144 x 1696 x 5120: 146 us on single tiles, 124 on pairs)
            continue
        for bn in (256, 192, 128, 64):
            if pair == 2 and bn < 128:
                continue
            if bn == 192 and (pair == 1 or not b_k_major or fused or n <= 192 or dtype == torch.int8):
                continue
            if dtype == torch.int8 and (bn < 128 or (pair == 2 and bn < 256)):
                continue   # 8-bit [K, N] operands need a full 128-byte run of N per TMA box and CTA
            cost = tile_cost(seg_rows, nseg, n, bn, pair, seg_cols=ar_cols, gain=gain)
            if tails and pair == 2:
                cost = tail_cut(rows, n, k, dtype.itemsize, bn)[0] * bn / (_TILE_EFF[bn] * gain[bn])
            if best is None or cost < best[0] - 1e-9:
                best = (cost, bn, pair)
    if best is None:
        best = (0.0, 256, 1)
    _, bn, pair = best
    tiles_m = max(1, math.ceil(rows / 128))
    # column-group width: keep the concurrently running tiles roughly square in (rows, cols)
    # (measured on 8192 x 28672 x 8192 and 8192 x 8192 x 28672: groups of 3-4 column tiles run 3-5 % faster
    # than groups of 8 or 16)
    swizzle = 4 if tiles_m >= 8 else max(1, min(16, _NUM_SMS // max(1, tiles_m)))
    # measured at W = 8: the int32 partials of the quantised op are link bound, lagged owner
    # rounds overlap its owner-side reduce; the all-reduce gains from the NVLS broadcast (the op
    # layer drops the flag when the heap has no multicast alias) and from column ownership
    rounds = 4 if (op == "quant_matmul_reduce_scatter" and world > 1 and rows >= 2048) else 0
    if allreduce:
        return TilingConfig(bn=bn, swizzle=swizzle, cta_pair=pair, use_multicast=True, seg_dim=1 if ar_cols else -1)
    # the all-gather broadcasts its shard by multicast stores when the heap has the alias (measured at
    # M = 8192: 6 % faster than peer-by-peer stores on 4 GPUs, 7 % slower on 2, where one store per
    # 16 bytes reaches one peer either way)
    return TilingConfig(bn=bn, swizzle=swizzle, cta_pair=pair, rounds=rounds,
                        use_multicast=(op == "allgather_matmul" and world >= 4))


def split_k(m: int, n: int, k: int, elt: int, direct: TilingConfig):
    """``(slices, k_slice, bn)`` when a local product is faster with its K range cut into slices whose
    planes a second kernel sums, else None.

    With few output tiles the direct kernel runs a fraction of the SMs, or a last wave that is nearly
    empty, and one CTA's intake bounds it: a 128-byte K block of a tile costs its MMAs (2 cycles per
    column) or its bytes (all 128 rows of A are filled, whatever M is). Wide tiles cut into slices take
    in fewer bytes per column; the price is the planes and a second kernel. bf16, M = 128, 8192 x 28672:
    134 -> 94 us; M = 100, 3584 x 8192: 44 -> 29 us; int8, M = 128, 8192 x 28672: 106 -> 63 us."""
    return _split_k(m, n, k, elt, direct)[0]


@functools.lru_cache(maxsize=4096)
def _split_k(m: int, n: int, k: int, elt: int, direct: TilingConfig):
    """``split_k``'s answer and the cycles that the product then takes."""
    kb = -(-k * elt // 128)

    def unit(bn, pair):
        return max(2.0 * bn, (128 + bn // pair) * 128 / _INTAKE[pair])

    hbm = (n * k + m * k) * elt / _HBM
    pair, bn0 = (2 if direct.cta_pair == 2 else 1), direct.effective_bn
    waves = -(-(-(-m // (128 * pair)) * -(-n // bn0)) // (_NUM_SMS // pair))
    if pair == 2 and bn0 >= 128:
        waves = tail_cut(m, n, k, elt, bn0)[0]
    # (for 8-bit operands the model puts a cut rather high: 256 x 8192 x 7168 30.5 us direct, 25.7 cut)
    whole = max(hbm, waves * kb * unit(bn0, pair)) + _LAUNCH + (_INT8_EPILOGUE if elt == 1 else 0.0)
    best, best_time = None, (0.97 if elt == 1 else 0.95) * whole
    for bn in (256, 128):
        if n < bn and bn > 128:
            continue
        tiles = -(-m // 128) * -(-n // bn)
        for s in range(2, 33):
            kbs = -(-(-(-kb // s)) // 2) * 2                  # K blocks per slice: whole 256-byte stages
            if kbs < 8 or -(-kb // kbs) != s:
                continue
            t = max(hbm, -(-tiles * s // _NUM_SMS) * kbs * unit(bn, 1)) + s * m * n * 8 / _PLANES + _LAUNCH + _FOLD
            if t < best_time:
                best, best_time = (s, kbs * 128 // elt, bn), t
    return best, whole if best is None else best_time


def slice_k_groups(groups: int, m: int, n: int, k_total: int, dtype: torch.dtype) -> TilingConfig:
    """Tiling of the products of ``groups`` K ranges, [m, n] each, in one launch (16-bit).

    A double tile takes 1.77 times as long as a pair tile: 32 ranges of 440 rows, 2048 x 4096: 294 -> 260 us, 32 of 234, 2048 x
    2048: 111 -> 88 us."""
    return _slice_k_groups(groups, m, n, k_total, dtype, os.environ.get("CATCOC_CTA_PAIR"))


@functools.lru_cache(maxsize=4096)
def _slice_k_groups(groups: int, m: int, n: int, k_total: int, dtype: torch.dtype, forced: Optional[str]) -> TilingConfig:
    # (`forced` is read by the heuristic: a choice made under it is not one without it)
    t = heuristic("matmul", groups * m, n, k_total, 1, dtype)
    if t.cta_pair == 2 and math.ceil(m / 256) * 256 > 1.18 * math.ceil(m / 128) * 128:
        t = t.with_(cta_pair=1)
    if t.cta_pair == 2 and t.effective_bn == 256:
        tiles, workers = groups * math.ceil(m / 256), _NUM_SMS // 2
        if 1.77 * math.ceil(tiles * math.ceil(n / 512) / workers) < math.ceil(tiles * math.ceil(n / 256) / workers):
            t = t.with_(bn=256, twice=True)
    return t


def grouped(rows_total: int, rows_per_group: float, n: int, dtype: torch.dtype) -> TilingConfig:
    """Tiling of a launch over groups of rows: waves of the groups' own tiles x time of a wave. The rows per
    group are exact (an int) or a mean, which then leaves half a tile of padding in each group.

    A 256-row tile is 1.18 times as fast per row in a call by itself; back to back its padding costs power as
    well (32 ragged groups of 440 rows on average: 230 -> 210 us from a cold start, 273 -> 282 us in a loop;
    937 rows: 429 -> 388 us), so ragged groups count 1.10. Few rows per group: 16 groups of 9 rows, 4096 x 2048:
    59 -> 50 us on wide tiles (the tiles used to be chosen for the rows of all groups as one product)"""
    return _grouped(rows_total, rows_per_group, n, dtype, os.environ.get("CATCOC_CTA_PAIR"))


@functools.lru_cache(maxsize=4096, typed=True)      # an exact row count and an equal mean are different questions
def _grouped(rows_total: int, rows_per_group: float, n: int, dtype: torch.dtype, forced: Optional[str]) -> TilingConfig:
    exact = isinstance(rows_per_group, int)
    groups = rows_total / max(rows_per_group, 1e-9)
    best = (0.0, 256, 1)
    for pair in (2, 1):
        bm = 128 * pair
        if (forced in ("1", "2") and pair != int(forced)) or (pair == 2 and rows_per_group <= 64):
            continue
        row_tiles = groups * (math.ceil(rows_per_group / bm) if exact else max(1.0, rows_per_group / bm + 0.5))
        row_tiles = max(1, math.ceil(min(row_tiles, rows_total)))
        for bn in (256, 128, 64):
            if (pair == 2 and bn < 128) or (dtype == torch.int8 and (bn < 128 or (pair == 2 and bn < 256))):
                continue
            gain = 1.0 if pair == 1 else _PAIR_GAIN[bn] if exact else _PAIR_GAIN[bn] * 1.10 / 1.18
            cost = math.ceil(row_tiles * math.ceil(n / bn) / (_NUM_SMS // pair)) * bn / (_TILE_EFF[bn] * gain)
            if best[0] == 0.0 or cost < best[0] - 1e-9:
                best = (cost, bn, pair)
    return TilingConfig(bn=best[1], swizzle=4, cta_pair=best[2])


def token_groups(rows_total: int, groups: int, n: int, k: int, dtype: torch.dtype) -> TilingConfig:
    """Tiling of a product over ragged groups of rows of an A stored [M, K] (their extents are on the device): :func:`grouped`'s,
    or double tiles with swapped roles, whose columns fit each group's rows to 32 where the other tiles pad them to 128 or 256.

    Groups of 110 to 770 rows, 32 of them, 4096 x 2048: 256 -> 227 us; 16 of 539 on average, 4096 x 4096: 321 -> 278; int8, 8 of
    451, 4096 x 2048: 55 -> 49. Few rows per group are bound by the weights' bytes, and the narrow pairs stream them more slowly
    (64 groups of 18, 1408 x 2048: 74 against 88 us), as does a short K, whose epilogues nothing covers."""
    return _token_groups(rows_total, groups, n, k, dtype, os.environ.get("CATCOC_CTA_PAIR"))


@functools.lru_cache(maxsize=4096)
def _token_groups(rows_total: int, groups: int, n: int, k: int, dtype: torch.dtype, forced: Optional[str]) -> TilingConfig:
    rows = rows_total / max(1, groups)
    old = _grouped(rows_total, rows, n, dtype, forced)
    if forced == "1" or rows < 128 or groups > 128 or rows_total >= 1 << 24 or dtype not in (torch.float16, torch.bfloat16, torch.int8):
        return old
    if dtype == torch.int8 and old.cta_pair == 2:      # 32 groups of 837, 4096 x 4096: 445 us, 499 with swapped roles
        return old
    kb, fb, hbm = -(-k * dtype.itemsize // 128), -(-n // 256), groups * n * k * dtype.itemsize / _HBM
    total = count = 0.0
    for f in (0.375, 0.625, 0.875, 1.125, 1.375, 1.625):       # a spread of sizes around the mean
        t = math.ceil(rows * f / 512)
        w = min(512, math.ceil(rows * f / t / 32) * 32)
        total += t * (kb * (560 if w <= 128 else max(610.0, 122 + 1.9 * w)) + 6000) / 6
        count += t / 6
    waves = count * groups * fb / (_NUM_SMS // 2)
    uneven = min(math.ceil(waves) - waves, 0.5 if waves > 1 else 1.0) if waves < 4 else 0.35
    new = max(total * groups * fb / (_NUM_SMS // 2) + total / count * uneven, hbm)
    bm = 128 * old.cta_pair
    unit = {(256, 1): 900, (128, 1): 620, (64, 1): 500, (256, 2): 640, (128, 2): 430}[(old.effective_bn, old.cta_pair)]
    tiles = groups * max(1.0, rows / bm + 0.5) * -(-n // old.effective_bn)
    cycles = max(math.ceil(tiles / (_NUM_SMS // old.cta_pair)) * kb * unit, hbm)
    if new + _LAUNCH < (cycles + _LAUNCH) / (0.985 if dtype != torch.int8 else 1.02):
        return TilingConfig(bn=256, swizzle=4, cta_pair=2, twice=True, swap=True)
    return old


def choose(op: str, m: int, n: int, k: int, world: int, dtype: torch.dtype,
           table: Optional["_table.TilingTable"] = None, b_k_major: bool = False, tails: bool = False,
           doubles: bool = False, swap: bool = False) -> TilingConfig:
    """``doubles``: the caller can launch double tiles (local products), ``swap``: with swapped roles too."""
    tbl = table if table is not None else _table.default_table()
    hit = tbl.lookup(op, m, n, k, world, dtype)
    if hit is not None:
        return hit
    forced = os.environ.get("CATCOC_CTA_PAIR")
    if doubles and forced != "1":
        return _with_doubles(op, m, n, k, world, dtype, b_k_major, tails, swap, forced)
    return heuristic(op, m, n, k, world, dtype, b_k_major, tails)


@functools.lru_cache(maxsize=4096)
def _with_doubles(op: str, m: int, n: int, k: int, world: int, dtype: torch.dtype, b_k_major: bool, tails: bool, swap: bool,
                  forced: Optional[str]) -> TilingConfig:
    # (kept by the sizes: a call without a plan, such as one whose weight needs a padded copy, comes here each time)
    t, elt = heuristic(op, m, n, k, world, dtype, b_k_major, tails), dtype.itemsize
    cut, cycles = _split_k(m, n, k, elt, t)
    if cut is None and t.cta_pair == 2:
        bn = t.effective_bn
        cycles = tail_cut(m, n, k, elt, bn)[0] * -(-k * elt // 128) * max(2.0 * bn, (128 + bn // 2) * 128 / _TAIL_INTAKE) + _LAUNCH + (
            _INT8_EPILOGUE if elt == 1 else 0.0)
    return double(m, n, k, elt, b_k_major, swap, 0.99 * cycles) or t
