"""Column-major (transposed) index of a fixed minibatch, and the gradient that uses it.

When a shard's minibatches are fixed row slices (the cyclic cursor of the reference,
ml/data/DataSet.scala:15-21, with a shard size that is a multiple of the batch size), the set of
columns a batch touches never changes. Its transposed index is built once; a step then computes
the per-row coefficients and gathers them per column, which replaces the scatter into the
dim-sized accumulator, the touched bitmap and the compaction (see csrc/cuda/glm_kernels.cu).
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import List, Optional

import torch

from . import lib as L
from .glm import DeviceCSR

SHORT_MAX, MEDIUM_MAX, LONG_SEGMENT = 4, 512, 4096
TILE_ROWS_MAX = 49152   # coefficients of one row tile in shared memory: 192 KB
PAIR_SEGMENT = 256      # longest entry list behind one partial sum
HOT_SEGMENT = 64        # entries of a tile's list of a frequent column
HOT_MIN_ENTRIES = 8_000_000   # entries of the frequent columns from which on their lists pay (see `_hot_columns`)
SEG_SLOTS = 256         # >= TILE_ROWS_MAX / PAIR_SEGMENT segments per (tile, column) pair


@dataclass
class TiledPart:
    """Row-tiled form of the index: entries in (tile, column, row) order with 16-bit tile-local rows, one
    partial sum per (tile, column) pair, the pairs of a column consecutive in (column, tile) order."""
    tile_rows: int
    n_tiles: int
    n_pairs: int
    tile_pair_ptr: torch.Tensor   # int32 [n_tiles + 1]
    pair_ptr: torch.Tensor        # int32 [n_pairs + 1]
    lrow: torch.Tensor            # int16 bit patterns of the unsigned tile-local rows [nnz]
    pair_dst: torch.Tensor        # int32 [n_pairs]
    col_pair_ptr: torch.Tensor    # int32 [n_cols + 1]
    partial: Optional[torch.Tensor] = None   # float32 scratch [>= n_pairs]; may be shared between indices


@dataclass
class HotColumns:
    """Frequent columns of a batch as lists per (row tile, item), with tile-local rows (csrc/cuda/tiled_kernels.cu)."""
    args: L.HotColumnsArgs
    tensors: List[torch.Tensor]    # what `args` points into
    partial_floats: int            # scratch it needs

    def nbytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self.tensors)

    def bind(self, partial: torch.Tensor) -> None:
        """Scratch of the engine's step; batches that run one after another share it."""
        self.partial = partial
        self.args.partial = partial.data_ptr()


@dataclass
class BatchIndex:
    lo: int
    rows: int
    n_cols: int
    colptr: torch.Tensor      # int32 [n_cols + 1]
    rowidx: torch.Tensor      # int32 [nnz], batch-local rows, column-major
    svals: Optional[torch.Tensor]
    ucols: torch.Tensor       # int32 [n_cols] ascending distinct columns = gradient keys
    bins: torch.Tensor        # int32: positions of short columns, then of medium columns
    long_col: torch.Tensor
    long_e0: torch.Tensor
    long_e1: torch.Tensor
    n_short: int
    n_medium: int
    n_long: int
    meta: torch.Tensor        # int64 [4] = {n_cols, 1, 0, 0}
    tiled: Optional[TiledPart] = None   # when set, the per-column arrays above are empty
    hot: Optional[HotColumns] = None    # when set, `bins` holds the other columns only, and no column is long

    def nbytes(self) -> int:
        ts = [self.colptr, self.rowidx, self.ucols, self.bins, self.long_col, self.long_e0, self.long_e1]
        if self.tiled is not None:
            ts += [self.tiled.tile_pair_ptr, self.tiled.pair_ptr, self.tiled.lrow, self.tiled.pair_dst, self.tiled.col_pair_ptr]
        return sum(t.numel() * t.element_size() for t in ts) + (self.svals.numel() * 4 if self.svals is not None else 0) + (
            self.hot.nbytes() if self.hot is not None else 0)


def _build_tiled(csr: DeviceCSR, lo: int, hi: int, e0: int, e1: int, rows: torch.Tensor) -> BatchIndex:
    dev = csr.cols.device
    nrows = hi - lo
    n_tiles = max(1, -(-nrows // TILE_ROWS_MAX))
    tile_rows = ((-(-nrows // n_tiles)) + 3) // 4 * 4
    cols = csr.cols[e0:e1].long()
    tile = (rows // tile_rows).long()
    skey, order = torch.sort((tile << 32) | cols, stable=True)   # (tile, column); rows stay ascending inside a pair
    local = (rows.long() - tile * tile_rows)[order]
    lrow = torch.where(local >= 32768, local - 65536, local).to(torch.int16).contiguous()   # unsigned 16-bit patterns
    svals = None if csr.values is None else csr.values[e0:e1][order].contiguous()
    # pairs of the frequent columns are cut into segments of PAIR_SEGMENT entries (each with its own partial sum),
    # so that no warp is left with one very long list
    pk0, pc0 = torch.unique_consecutive(skey, return_counts=True)
    start0 = torch.cumsum(pc0, 0) - pc0
    rank = torch.arange(e1 - e0, device=dev) - torch.repeat_interleave(start0, pc0, output_size=e1 - e0)
    seg = rank // PAIR_SEGMENT
    skey_seg = skey * SEG_SLOTS + seg            # still ascending: seg grows inside a pair
    pkey_seg, pcnt = torch.unique_consecutive(skey_seg, return_counts=True)
    pkey, pseg = pkey_seg // SEG_SLOTS, pkey_seg % SEG_SLOTS
    n_pairs = int(pkey.numel())
    pair_ptr = torch.zeros(n_pairs + 1, dtype=torch.int32, device=dev)
    pair_ptr[1:] = torch.cumsum(pcnt, 0).to(torch.int32)
    ptile, pcol = pkey >> 32, pkey & 0xFFFFFFFF
    tile_pair_ptr = torch.searchsorted(ptile, torch.arange(n_tiles + 1, device=dev)).to(torch.int32)
    skey2, perm = torch.sort(((pcol << 20) | ptile) * SEG_SLOTS + pseg)   # (column, tile, segment)
    skey2 = skey2 // SEG_SLOTS
    pair_dst = torch.empty(n_pairs, dtype=torch.int32, device=dev)
    pair_dst[perm] = torch.arange(n_pairs, dtype=torch.int32, device=dev)
    ucols, ccnt = torch.unique_consecutive(skey2 >> 20, return_counts=True)
    n = int(ucols.numel())
    col_pair_ptr = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    col_pair_ptr[1:] = torch.cumsum(ccnt, 0).to(torch.int32)
    empty = torch.zeros(0, dtype=torch.int32, device=dev)
    part = TiledPart(tile_rows, n_tiles, n_pairs, tile_pair_ptr.contiguous(), pair_ptr, lrow, pair_dst, col_pair_ptr)
    return BatchIndex(lo, nrows, n, empty, empty, svals, ucols.to(torch.int32).contiguous(), empty, empty, empty, empty, 0, 0, 0,
                      torch.tensor([n, 1 if n else 0, 0, 0], dtype=torch.int64, device=dev), part)


def _hot_columns(ucols: torch.Tensor, colptr: torch.Tensor, rowidx: torch.Tensor, svals: Optional[torch.Tensor], cnt: torch.Tensor, rows: int,
                 budget: Optional[int] = None):
    """The columns with at least two entries per row tile on average (and more than the short ones'), and which they are;
    (None, None) where they hold too few entries to pay for tiles, partial sums and one more launch. Steps without and with
    lists, us: 3.4M entries of frequent columns 165 / 165, 5.6M 220 / 212, 7.9M 265 / 250, 11.3M 322 / 299; with values 3.9M
    142 / 145, 6.4M 179 / 179, 9.0M 221 / 217, 12.8M 270 / 261. Building them takes 0.2 ms more a batch of 15M entries (0.4 of
    30M with values), which 10 to 15 visits of the batch pay for.
    None too where building the lists, or the lists and their scratch afterwards, would take more than ``budget`` bytes."""
    if rowidx.numel() < HOT_MIN_ENTRIES:
        return None, None
    dev, lib = rowidx.device, L.lib()
    a = L.HotColumnsArgs()
    a.rows = rows
    a.row_tiles, a.tile_rows = _tiles(rows, TILE_ROWS_MAX)
    is_hot = cnt >= max(SHORT_MAX + 1, 2 * a.row_tiles)
    pos = torch.nonzero(is_hot).flatten().to(torch.int32)
    a.columns = pos.numel()
    if int(cnt[pos.long()].sum()) < HOT_MIN_ENTRIES:
        return None, None
    room = a.columns * (8 * a.row_tiles + 100)   # bounds and counts per tile; positions, items and places of the columns
    if budget is not None and room > budget:
        return None, None
    a.items = a.columns
    a.pos = L.ptr(pos)
    bound = torch.empty((a.row_tiles + 1, a.columns), dtype=torch.int32, device=dev)
    L.check(lib.skml_hot_bounds(C.byref(a), L.ptr(colptr), L.ptr(rowidx), L.ptr(bound), L.stream()), "skml_hot_bounds")
    per = bound[1:] - bound[:-1]
    k = (per.amax(0) + HOT_SEGMENT - 1) // HOT_SEGMENT
    item0 = torch.zeros(a.columns + 1, dtype=torch.int32, device=dev)
    torch.cumsum(k, 0, dtype=torch.int32, out=item0[1:])
    a.items = int(item0[-1])
    if a.row_tiles * a.items + rowidx.numel() // 4 >= L.DT_LISTS_MAX:
        return None, None
    room += 12 * a.row_tiles * a.items + 32 * a.items   # the lists' lengths, bounds and partial sums; the items' columns
    if budget is not None and room > budget:
        return None, None
    info = torch.stack([pos, item0[:-1], k, ucols[pos.long()].to(torch.int32)], 1).contiguous()
    wide = info[k > 1].contiguous()
    a.wide = wide.shape[0]
    column = torch.repeat_interleave(torch.arange(a.columns, device=dev, dtype=torch.int32), k, output_size=a.items)
    segment = torch.arange(a.items, device=dev, dtype=torch.int32) - item0[column]
    quads = per[:, column]
    quads.sub_(segment.mul_(HOT_SEGMENT)).clamp_(0, HOT_SEGMENT).add_(3).bitwise_right_shift_(2)
    ptr = torch.zeros(a.row_tiles * a.items + 1, dtype=torch.int32, device=dev)
    torch.cumsum(quads.flatten(), 0, dtype=torch.int32, out=ptr[1:])
    n = 4 * int(ptr[-1])
    if budget is not None and room + n * (2 if svals is None else 6) > budget:
        return None, None
    loc = torch.full((n,), a.tile_rows if a.tile_rows < 32768 else a.tile_rows - 65536, dtype=torch.int16, device=dev)   # unsigned 16-bit patterns
    val = None if svals is None else torch.zeros(n, dtype=torch.float32, device=dev)
    a.item0, a.info, a.wide_info, a.ptr, a.loc, a.val = L.ptr(item0), L.ptr(info), L.ptr(wide), L.ptr(ptr), L.ptr(loc), L.ptr(val)
    L.check(lib.skml_hot_fill(C.byref(a), L.ptr(bound), L.ptr(column), L.ptr(rowidx), L.ptr(svals), L.stream()), "skml_hot_fill")
    return HotColumns(a, [pos, item0, info, wide, ptr, loc] + ([val] if val is not None else []), int(a.row_tiles * a.items)), is_hot


def build_batch_index(csr: DeviceCSR, lo: int, hi: int, tiled: bool = False, hot: bool = False, hot_budget: Optional[int] = None) -> BatchIndex:
    """``tiled``: the row-tiled form (coefficients of a row tile in shared memory, no atomics); needs fewer than
    2^20 tiles, i.e. any batch that fits a GPU. ``hot``: the frequent columns of the per-column form as lists per row
    tile, where that pays and takes no more than ``hot_budget`` bytes (see `_hot_columns`)."""
    dev = csr.cols.device
    e0, e1 = int(csr.rowptr[lo]), int(csr.rowptr[hi])
    cols = csr.cols[e0:e1]
    counts = (csr.rowptr[lo + 1:hi + 1] - csr.rowptr[lo:hi])
    rows = torch.repeat_interleave(torch.arange(hi - lo, device=dev, dtype=torch.int32), counts, output_size=e1 - e0)
    if tiled and e1 > e0:
        return _build_tiled(csr, lo, hi, e0, e1, rows)
    scol, order = torch.sort(cols, stable=True)
    rowidx = rows[order].contiguous()
    svals = None if csr.values is None else csr.values[e0:e1][order].contiguous()
    ucols, cnt = torch.unique_consecutive(scol, return_counts=True)
    n = int(ucols.numel())
    colptr = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    colptr[1:] = torch.cumsum(cnt, 0).to(torch.int32)
    pos = torch.arange(n, device=dev, dtype=torch.int32)
    frequent, is_hot = _hot_columns(ucols, colptr, rowidx, svals, cnt, hi - lo, hot_budget) if hot and n else (None, None)
    if frequent is not None:
        none = torch.zeros(0, dtype=torch.int32, device=dev)
        short, medium = pos[cnt <= SHORT_MAX], pos[(cnt > SHORT_MAX) & ~is_hot]
        return BatchIndex(lo, hi - lo, n, colptr, rowidx, svals, ucols.to(torch.int32).contiguous(), torch.cat([short, medium]).contiguous(),
                          none, none, none, int(short.numel()), int(medium.numel()), 0, torch.tensor([n, 1, 0, 0], dtype=torch.int64, device=dev), hot=frequent)
    short = pos[cnt <= SHORT_MAX]
    medium = pos[(cnt > SHORT_MAX) & (cnt <= MEDIUM_MAX)]
    longs = pos[cnt > MEDIUM_MAX]
    nseg = (cnt[longs.long()] + LONG_SEGMENT - 1) // LONG_SEGMENT
    long_col = torch.repeat_interleave(longs, nseg)
    first = torch.cumsum(nseg, 0) - nseg
    seg = torch.arange(int(long_col.numel()), device=dev) - torch.repeat_interleave(first, nseg)
    le0 = colptr[long_col.long()].long() + seg * LONG_SEGMENT
    le1 = torch.minimum(le0 + LONG_SEGMENT, colptr[long_col.long() + 1].long())
    return BatchIndex(lo, hi - lo, n, colptr, rowidx, svals, ucols.to(torch.int32).contiguous(),
                      torch.cat([short, medium]).contiguous(), long_col.to(torch.int32).contiguous(),
                      le0.to(torch.int32).contiguous(), le1.to(torch.int32).contiguous(), int(short.numel()),
                      int(medium.numel()), int(long_col.numel()),
                      torch.tensor([n, 1 if n else 0, 0, 0], dtype=torch.int64, device=dev))


@dataclass
class DenseIndex:
    """Tiled copies of the entries of a batch that touches most coordinates (csrc/cuda/tiled_kernels.cu)."""
    lo: int
    rows: int
    args: L.DenseIndexArgs
    tensors: List[torch.Tensor]    # what `args` points into
    partial_floats: int            # scratch it needs

    def nbytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self.tensors)

    def bind(self, partial: torch.Tensor, coef: torch.Tensor) -> None:
        """Scratch of a step; batches that run one after another share it."""
        self.args.partial, self.args.coef = partial.data_ptr(), coef.data_ptr()


def _tiles(n: int, tile_max: int):
    tiles = max(1, -(-n // tile_max))
    return tiles, ((-(-n // tiles)) + 7) // 8 * 8


def build_dense_index(csr: DeviceCSR, lo: int, hi: int, budget: Optional[int] = None) -> Optional[DenseIndex]:
    """None where the batch touches no more than two thirds of the columns, or where the lists would be too short to be
    worth it (fewer than one entry per row tile and column): partial sums and list bounds then cost more than the
    scatter's atomics. The margins take the tiled form from six entries per
    row and column tile on; below, the padding and the partial sums cost more than gathers of w.
    None too where building it, or the index and its scratch afterwards, would take more than ``budget`` bytes."""
    dev, lib, rows, dim = csr.cols.device, L.lib(), hi - lo, csr.dim
    e0, e1 = int(csr.rowptr[lo]), int(csr.rowptr[hi])
    nnz = e1 - e0
    a = L.DenseIndexArgs()
    a.rows, a.dim = rows, dim
    a.row_tiles, a.tile_rows = _tiles(rows, TILE_ROWS_MAX)
    a.col_tiles, a.tile_cols = _tiles(dim, TILE_ROWS_MAX)
    if nnz < a.row_tiles * dim or 3 * nnz <= 2 * dim:
        return None
    if max(a.row_tiles * dim, a.col_tiles * rows) + nnz // 4 >= L.DT_LISTS_MAX:
        return None   # (lists and their quads, at most one more than a quarter of the entries each, are numbered in 32 bits)
    margins = nnz >= 6 * rows * a.col_tiles and a.col_tiles <= 256
    # counts and bounds of all lists, the sums in between, the partial sums of a step (the entries are added below)
    n_lists = (a.row_tiles * dim, a.col_tiles * rows if margins else 0)
    room = 8 * sum(n_lists) + 12 * max(n_lists) + 8 * dim
    if budget is not None and room > budget:
        return None
    cnt_c = torch.zeros(a.row_tiles * dim, dtype=torch.int32, device=dev)
    cnt_r = torch.empty(a.col_tiles * rows, dtype=torch.int32, device=dev) if margins else None
    L.check(lib.skml_dt_count(C.byref(a), L.ptr(csr.rowptr), L.ptr(csr.cols), lo, L.ptr(cnt_c), L.ptr(cnt_r), L.stream()), "skml_dt_count")

    any_c = cnt_c.view(a.row_tiles, dim).amax(0) if a.row_tiles > 1 else cnt_c
    if int(torch.count_nonzero(any_c)) <= dim * 2 // 3:
        return None

    def bounds(cnt):
        ptr = torch.zeros(cnt.numel() + 1, dtype=torch.int32, device=dev)
        torch.cumsum((cnt + 3) >> 2, 0, dtype=torch.int32, out=ptr[1:])
        return ptr, -(-4 * int(ptr[-1]) // 2 ** 20) * 2 ** 20   # whole megabytes: batches of one data set get buffers of one size

    def entries(n, pad):
        loc = torch.full((n,), pad if pad < 32768 else pad - 65536, dtype=torch.int16, device=dev)   # unsigned 16-bit patterns
        return loc, None if csr.values is None else torch.zeros(n, dtype=torch.float32, device=dev)

    c_ptr, n_c = bounds(cnt_c)
    r_ptr, n_r = bounds(cnt_r) if margins else (None, 0)
    if budget is not None and room + (n_c + n_r) * (2 if csr.values is None else 6) > budget:
        return None

    c_loc, c_val = entries(n_c, int(a.tile_rows))
    tensors = [c_ptr, c_loc] + ([c_val] if c_val is not None else [])
    a.c_ptr, a.c_loc, a.c_val = L.ptr(c_ptr), L.ptr(c_loc), L.ptr(c_val)
    if margins:
        r_loc, r_val = entries(n_r, int(a.tile_cols))
        tensors += [r_ptr, r_loc] + ([r_val] if r_val is not None else [])
        a.r_ptr, a.r_loc, a.r_val = L.ptr(r_ptr), L.ptr(r_loc), L.ptr(r_val)
    cursor = cnt_c.zero_()
    L.check(lib.skml_dt_fill(C.byref(a), L.ptr(csr.rowptr), L.ptr(csr.cols), L.ptr(csr.values), lo, nnz, L.ptr(cursor), L.stream()),
            "skml_dt_fill")
    return DenseIndex(lo, rows, a, tensors, int(max(n_lists)))


def glm_grad_dense(csr: DeviceCSR, di: DenseIndex, w: torch.Tensor, g: torch.Tensor, bitmap: torch.Tensor, partials: torch.Tensor,
                   status: torch.Tensor, loss_id: int, budget_s: float = 1.0) -> None:
    """The batch gradient (mean over the batch) in the zero accumulator ``g`` and its touched bitmap, for
    `compact_gradient`; the objective loss sum is added into partials[1]."""
    L.check(L.lib().skml_dt_gradient(C.byref(di.args), L.ptr(csr.rowptr), L.ptr(csr.cols), L.ptr(csr.values), L.ptr(csr.labels), di.lo,
                                     csr.nnz_padded, float(csr.avg_nnz), L.ptr(w), loss_id, 1.0 / max(1, di.rows),
                                     partials.data_ptr() + 8, L.ptr(g), L.ptr(bitmap), L.ptr(status), L.budget_cycles(budget_s),
                                     L.stream()), "skml_dt_gradient")
    L.count_launches(4 if di.args.r_ptr else 3)


def glm_grad_transposed(csr: DeviceCSR, bi: BatchIndex, w: torch.Tensor, coef: torch.Tensor, out_vals: torch.Tensor,
                        partials: torch.Tensor, status: torch.Tensor, loss_id: int, lam: float,
                        budget_s: float = 1.0) -> None:
    """out_vals[:bi.n_cols] = gradient values (mean over the batch + lam * w) for keys bi.ucols;
    the objective loss sum is added into partials[1]."""
    lib = L.lib()
    L.check(lib.skml_glm_coef(L.ptr(csr.rowptr), L.ptr(csr.cols), L.ptr(csr.values), L.ptr(csr.labels), bi.lo, bi.rows,
                              csr.nnz_padded, float(csr.avg_nnz), L.ptr(w), w.numel(), loss_id, 1.0 / max(1, bi.rows),
                              partials.data_ptr() + 8, L.ptr(coef), L.ptr(status), L.budget_cycles(budget_s), L.stream()),
            "skml_glm_coef")
    if bi.tiled is not None:
        tp = bi.tiled
        if tp.partial is None or tp.partial.numel() < tp.n_pairs:
            tp.partial = torch.zeros(max(tp.n_pairs, 1), dtype=torch.float32, device=coef.device)
        L.check(lib.skml_colsum_tiled(L.ptr(tp.tile_pair_ptr), L.ptr(tp.pair_ptr), L.ptr(tp.lrow), L.ptr(bi.svals),
                                      L.ptr(tp.pair_dst), L.ptr(tp.col_pair_ptr), L.ptr(bi.ucols), bi.rows, tp.tile_rows,
                                      tp.n_tiles, bi.n_cols, L.ptr(coef), L.ptr(w), float(lam), L.ptr(tp.partial),
                                      L.ptr(out_vals), L.stream()), "skml_colsum_tiled")
        L.count_launches(3)
        return
    if bi.hot is not None:
        # scratch of this call's own: the same index may be used on another stream or thread at the same time
        partial = torch.empty(bi.hot.partial_floats, dtype=torch.float32, device=coef.device)
        args = L.HotColumnsArgs.from_buffer_copy(bi.hot.args)
        args.partial = partial.data_ptr()
        L.check(lib.skml_hot_colsum(C.byref(args), L.ptr(bi.bins), bi.n_short, bi.n_medium, L.ptr(bi.colptr), L.ptr(bi.rowidx),
                                    L.ptr(bi.svals), L.ptr(bi.ucols), L.ptr(coef), L.ptr(w), float(lam), L.ptr(out_vals), None, None,
                                    L.stream()), "skml_hot_colsum")
        L.count_launches(3)
        return
    L.check(lib.skml_colsum(L.ptr(bi.colptr), L.ptr(bi.rowidx), L.ptr(bi.svals), L.ptr(bi.ucols), L.ptr(bi.bins),
                            L.ptr(bi.long_col), L.ptr(bi.long_e0), L.ptr(bi.long_e1), bi.n_short, bi.n_medium, bi.n_long,
                            bi.n_cols, L.ptr(coef), L.ptr(w), float(lam), L.ptr(out_vals), L.stream()), "skml_colsum")
    L.count_launches(2)
