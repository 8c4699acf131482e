// Gradient of a batch that touches most coordinates (the dense kind), over two tiled copies of its entries.
//
// A near-dense batch has many entries per column and per row, so both halves of the gradient are products of
// a sparse matrix with a vector that does not fit L1: margins gather w, column sums gather the coefficients,
// and every gather is a random 32-byte sector of L2 (155 G/s). The scatter form adds one float atomic per
// entry on top. Here the vector is cut into tiles that fit shared memory, and the batch's entries are laid
// out once, when the index is built, by (vector tile, row) for the margins and by (vector tile, column) for
// the column sums, with 16-bit tile-local positions. A block keeps one tile and sums its share of the (tile,
// item) lists, one lane per list; the partial sums, tile-major, are added up by a second kernel with
// consecutive reads. Lists are padded to four entries so that a lane reads them 8 and 16 bytes at a time; the
// padding points at a slot that holds zero.
// 500,000 rows x 200 values over 1M columns (100M entries, 1.3 GB of tiled copies read): see the measured
// figures at dt_partial_kernel.
//
// Reference behaviour restated (ml module): objective/GradientDescent.scala:23-51 (margins, coefficients,
// scatter-add); the kind is still decided by the compaction, as in gradient/DenseDoubleGradient.scala:64-94.
#include "glm_loss.cuh"
#include "skml_api.h"
#include "skml_device.cuh"

namespace {

constexpr int DT_THREADS = 1024;
constexpr int DT_LONG = 16;          // lists of more quads are summed by the whole warp
constexpr int DT_BATCH = 4;          // quads of a lane in flight
constexpr int DT_ROW_WARPS = 8;
constexpr int DT_MAX_COL_TILES = 256;
constexpr int DT_ROW_STAGE = 256;    // entries of a row that the fill puts in order in shared memory

// Entries per (row tile, column) and per (column tile, row); one warp per row.
__global__ void __launch_bounds__(DT_ROW_WARPS * 32)
dt_count_kernel(const long long* __restrict__ rowptr, const int* __restrict__ cols, long long row_lo, int rows, int tile_rows,
                int tile_cols, int col_tiles, int dim, int* __restrict__ cnt_cols, int* __restrict__ cnt_rows) {
    __shared__ int s_cnt[DT_ROW_WARPS][DT_MAX_COL_TILES];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = blockIdx.x * DT_ROW_WARPS + warp; r < rows; r += gridDim.x * DT_ROW_WARPS) {
        if (cnt_rows)
            for (int t = lane; t < col_tiles; t += 32) s_cnt[warp][t] = 0;
        __syncwarp();
        const long long e0 = rowptr[row_lo + r], e1 = rowptr[row_lo + r + 1];
        int* const cc = cnt_cols + (long long)(r / tile_rows) * dim;
        for (long long e = e0 + lane; e < e1; e += 32) {
            const int c = cols[e];
            atomicAdd(cc + c, 1);
            if (cnt_rows) atomicAdd(&s_cnt[warp][c / tile_cols], 1);
        }
        __syncwarp();
        if (cnt_rows)
            for (int t = lane; t < col_tiles; t += 32) cnt_rows[(long long)t * rows + r] = s_cnt[warp][t];
        __syncwarp();
    }
}

// The entries to their lists. The column lists fill up entry by entry at random places, so they have to stay in L2
// until they are full: the rows of a tile are walked `parts` times, each time for one range of columns whose lists
// take some 16 MB, and the walks are dealt to the warps in order. (One walk over 70 MB of lists ran at the rate of
// random DRAM sectors: 10 ms for 100M entries.) Everything else is read and written as a stream: a warp puts a row's
// entries in the order of its row lists in shared memory first (rows of up to DT_ROW_STAGE entries).
__global__ void __launch_bounds__(DT_ROW_WARPS * 32)
dt_fill_kernel(const long long* __restrict__ rowptr, const int* __restrict__ cols, const float* __restrict__ vals, long long row_lo,
               int rows, int tile_rows, int row_tiles, int tile_cols, int col_tiles, int dim, int parts, const int* __restrict__ c_ptr, int* __restrict__ cursor,
               unsigned short* __restrict__ c_loc, float* __restrict__ c_val, const int* __restrict__ r_ptr,
               unsigned short* __restrict__ r_loc, float* __restrict__ r_val) {
    __shared__ int s_at[DT_ROW_WARPS][DT_MAX_COL_TILES];
    __shared__ int s_dst[DT_ROW_WARPS][DT_MAX_COL_TILES];   // position of a tile's first staged entry
    __shared__ unsigned short s_loc[DT_ROW_WARPS][DT_ROW_STAGE];
    __shared__ unsigned char s_tile[DT_ROW_WARPS][DT_ROW_STAGE];
    __shared__ float s_val[DT_ROW_WARPS][DT_ROW_STAGE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int width = (dim + parts - 1) / parts;   // columns of a walk
    const long long walks = (long long)row_tiles * parts * tile_rows;
    for (long long q = (long long)blockIdx.x * DT_ROW_WARPS + warp; q < walks; q += (long long)gridDim.x * DT_ROW_WARPS) {
        const long long walk = q / tile_rows;
        const int rt = (int)(walk / parts), part = (int)(walk % parts), r = rt * tile_rows + (int)(q % tile_rows);
        if (r >= rows) continue;
        const int c_lo = part * width, c_hi = dim - c_lo < width ? dim : c_lo + width;
        const long long e0 = rowptr[row_lo + r], e1 = rowptr[row_lo + r + 1];
        const long long cbase = (long long)rt * dim;
        const unsigned short lr = (unsigned short)(r - rt * tile_rows);
        const bool by_row = r_ptr && part == 0, stage = by_row && e1 - e0 <= DT_ROW_STAGE;
        if (by_row) {
            for (int t = lane; t < col_tiles; t += 32) s_at[warp][t] = 0;
            __syncwarp();
        }
        if (stage) {   // entries per tile, then their first positions
            for (long long e = e0 + lane; e < e1; e += 32) atomicAdd(&s_at[warp][cols[e] / tile_cols], 1);
            __syncwarp();
            int before = 0;
            for (int t0 = 0; t0 < col_tiles; t0 += 32) {
                const int n = t0 + lane < col_tiles ? s_at[warp][t0 + lane] : 0;
                int inc = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                    if (lane >= o) inc += x;
                }
                if (t0 + lane < col_tiles) {
                    s_dst[warp][t0 + lane] = before + inc - n;
                    s_at[warp][t0 + lane] = before + inc - n;
                }
                before += __shfl_sync(0xFFFFFFFFu, inc, 31);
            }
            __syncwarp();
        }
        for (long long e = e0 + lane; e < e1; e += 32) {
            const int c = __ldcs(cols + e);
            const bool here = c >= c_lo && c < c_hi;
            const float v = vals && (here || by_row) ? __ldcs(vals + e) : 1.f;
            if (here) {
                const long long at = 4ll * c_ptr[cbase + c] + atomicAdd(cursor + cbase + c, 1);
                c_loc[at] = lr;
                if (vals) c_val[at] = v;
            }
            if (by_row) {
                const int ct = c / tile_cols;
                const int k = atomicAdd(&s_at[warp][ct], 1);
                if (stage) {
                    s_loc[warp][k] = (unsigned short)(c - ct * tile_cols);
                    s_tile[warp][k] = (unsigned char)ct;
                    if (vals) s_val[warp][k] = v;
                } else {
                    const long long ar = 4ll * r_ptr[(long long)ct * rows + r] + k;
                    r_loc[ar] = (unsigned short)(c - ct * tile_cols);
                    if (vals) r_val[ar] = v;
                }
            }
        }
        __syncwarp();
        if (stage) {
            for (int k = lane; k < (int)(e1 - e0); k += 32) {
                const int ct = s_tile[warp][k];
                const long long ar = 4ll * r_ptr[(long long)ct * rows + r] + (k - s_dst[warp][ct]);
                __stcs(r_loc + ar, s_loc[warp][k]);
                if (vals) __stcs(r_val + ar, s_val[warp][k]);
            }
            __syncwarp();
        }
    }
}

// Puts the quads of every 32 neighbouring lists of a tile in the order dt_partial_kernel reads them: the first quads of
// all lists, then the second quads of those that have one, and so on, so that a warp's loads are consecutive. The 32
// lists keep their place in memory. Groups with a list of more than DT_LONG quads stay list by list. One warp a group.
constexpr int DT_TURN_WARPS = 4;
template <bool HAS_VALS>
__global__ void __launch_bounds__(DT_TURN_WARPS * 32)
dt_interleave_kernel(const int* __restrict__ ptr, int tiles, int items, ushort4* __restrict__ loc, float4* __restrict__ val) {
    __shared__ float4 s_val[HAS_VALS ? DT_TURN_WARPS : 1][HAS_VALS ? 32 * DT_LONG : 1];
    __shared__ ushort4 s_loc[DT_TURN_WARPS][32 * DT_LONG];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int below = (1u << lane) - 1u;
    const int per_tile = (items + 31) / 32;
    const long long groups = (long long)tiles * per_tile;
    for (long long g = (long long)blockIdx.x * DT_TURN_WARPS + warp; g < groups; g += (long long)gridDim.x * DT_TURN_WARPS) {
        const int tile = (int)(g / per_tile), i = (int)(g % per_tile) * 32 + lane;
        const long long p = (long long)tile * items + i;
        const int q0 = i < items ? ptr[p] : 0, len = i < items ? ptr[p + 1] - q0 : 0;
        const int most = __reduce_max_sync(0xFFFFFFFFu, len);
        if (most > DT_LONG || most < 2) continue;
        const int first = __shfl_sync(0xFFFFFFFFu, q0, 0), total = __reduce_add_sync(0xFFFFFFFFu, len);
        for (int k = lane; k < total; k += 32) {
            s_loc[warp][k] = loc[first + k];
            if (HAS_VALS) s_val[warp][k] = val[first + k];
        }
        __syncwarp();
        int at = first;
        for (int j = 0; j < most; ++j) {
            const unsigned int have = __ballot_sync(0xFFFFFFFFu, len > j);
            if (len > j) {
                const int dst = at + __popc(have & below);
                loc[dst] = s_loc[warp][q0 - first + j];
                if (HAS_VALS) val[dst] = s_val[warp][q0 - first + j];
            }
            at += __popc(have);
        }
        __syncwarp();
    }
}

// First list p in [lo, hi) whose quads and lists before it reach `target`; a whole warp, 32 probes a round.
__device__ __forceinline__ int weighted_bound(const int* __restrict__ ptr, int lo, int hi, long long base, long long target) {
    const int lane = threadIdx.x & 31, first = lo;
    while (hi > lo) {
        const int step = (hi - lo + 32) / 33;   // probes lo + step - 1, lo + 2 step - 1, ... below hi
        const long long at = (long long)lo + (long long)(lane + 1) * step - 1;
        const bool less = at < hi && (long long)ptr[at] + (at - first) - base < target;
        const int n = __popc(__ballot_sync(0xFFFFFFFFu, less));   // probes that lie before the answer: the first n
        const long long nlo = (long long)lo + (long long)n * step, nhi = n == 32 ? (long long)hi : nlo + step - 1;
        lo = nlo < hi ? (int)nlo : hi;
        hi = nhi < hi ? (int)nhi : hi;
    }
    return lo;
}

// Shares of a tile's lists [p0, p1) of block `sub` of `blocks`, one per warp, by quads + lists, cut at whole groups of 32:
// warp w sums lists s_cut[w] to s_cut[w + 1].
__device__ __forceinline__ void dt_cuts(const int* __restrict__ ptr, int p0, int p1, int sub, int blocks, int* s_cut) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = DT_THREADS / 32;
    const long long base = ptr[p0], all = (long long)ptr[p1] - base + (p1 - p0);
    const long long share = (long long)sub * warps + warp, shares = (long long)blocks * warps;
    auto group_start = [&](int p) { return p0 + ((p - p0) & ~31); };
    const int cut = group_start(weighted_bound(ptr, p0, p1, base, all * share / shares));
    if (lane == 0) s_cut[warp] = cut;
    if (warp == warps - 1) {
        const int end = sub + 1 == blocks ? p1 : group_start(weighted_bound(ptr, p0, p1, base, all * (share + 1) / shares));
        if (lane == 0) s_cut[warps] = end;
    }
}

// One warp's lists [w0, w1): partial[p] = sum over list p of s_x[loc] * val.
template <bool HAS_VALS>
__device__ __forceinline__ void dt_lists(const float* s_x, int T, int w0, int w1, const int* __restrict__ ptr, const ushort4* __restrict__ loc,
                                         const float4* __restrict__ val, float* __restrict__ partial) {
    const int lane = threadIdx.x & 31;
    auto quad = [&](const ushort4 l, const float4 v) {
        return HAS_VALS ? fmaf(s_x[l.x], v.x, fmaf(s_x[l.y], v.y, fmaf(s_x[l.z], v.z, s_x[l.w] * v.w)))
                        : (s_x[l.x] + s_x[l.y]) + (s_x[l.z] + s_x[l.w]);
    };
    const ushort4 none = make_ushort4(T, T, T, T);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    // list bounds two rounds ahead, entries one round ahead as far as L2
    int nq0 = 0, nq1 = 0, mq0 = 0, mq1 = 0;
    auto bounds = [&](int p, int& a, int& e) {
        a = e = 0;
        if (p < w1) {
            a = ptr[p];
            e = ptr[p + 1];
        }
    };
    bounds(w0 + lane, nq0, nq1);
    bounds(w0 + 32 + lane, mq0, mq1);
    for (int b = w0; b < w1; b += 32) {
        const int p = b + lane;
        const int q0 = nq0, q1 = nq1;
        nq0 = mq0;
        nq1 = mq1;
        bounds(p + 64, mq0, mq1);
        {   // the next round's lists are neighbours: a line of 128 bytes a lane
            const int f = __shfl_sync(0xFFFFFFFFu, nq0, 0), l = __reduce_max_sync(0xFFFFFFFFu, nq1);
            if (HAS_VALS && f + 8 * lane < l) asm volatile("prefetch.global.L2 [%0];" ::"l"(val + f + 8 * lane));
            if (f + 16 * lane < l) asm volatile("prefetch.global.L2 [%0];" ::"l"(loc + f + 16 * lane));
        }
        float acc = 0.f;
        const int len = q1 - q0, most = __reduce_max_sync(0xFFFFFFFFu, len);
        if (most <= DT_LONG) {   // interleaved
            int at = __shfl_sync(0xFFFFFFFFu, q0, 0);
            for (int k = 0; k < most; k += DT_BATCH) {
                ushort4 l[DT_BATCH];
                float4 v[DT_BATCH];
#pragma unroll
                for (int u = 0; u < DT_BATCH; ++u) {
                    const unsigned int have = __ballot_sync(0xFFFFFFFFu, len > k + u);
                    const int q = at + __popc(have & ((1u << lane) - 1u));
                    at += __popc(have);
                    l[u] = len > k + u ? __ldg(loc + q) : none;
                    v[u] = HAS_VALS && len > k + u ? __ldg(val + q) : zero;
                }
#pragma unroll
                for (int u = 0; u < DT_BATCH; ++u)
                    if (len > k + u) acc += quad(l[u], v[u]);
            }
            if (p < w1) partial[p] = acc;
            continue;
        }
        if (len <= DT_LONG)
            for (int q = q0; q < q1; ++q) acc += quad(__ldg(loc + q), HAS_VALS ? __ldg(val + q) : zero);
        unsigned int longs = __ballot_sync(0xFFFFFFFFu, len > DT_LONG);
        while (longs) {   // frequent items: the warp sums one list at a time
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const int s0 = __shfl_sync(0xFFFFFFFFu, q0, src), s1 = __shfl_sync(0xFFFFFFFFu, q1, src);
            float part = 0.f;
            for (int q = s0 + lane; q < s1; q += 32 * DT_BATCH) {
                ushort4 l[DT_BATCH];
                float4 v[DT_BATCH];
#pragma unroll
                for (int u = 0; u < DT_BATCH; ++u) {
                    l[u] = q + 32 * u < s1 ? __ldg(loc + q + 32 * u) : none;
                    v[u] = HAS_VALS && q + 32 * u < s1 ? __ldg(val + q + 32 * u) : zero;
                }
#pragma unroll
                for (int u = 0; u < DT_BATCH; ++u) part += quad(l[u], v[u]);
            }
            part = warp_sum(part);
            if (lane == src) acc = part;
        }
        if (p < w1) partial[p] = acc;
    }
}

// partial[tile * items + item] = sum over the list of x[tile * T + loc] * val.
// Blocks of a tile, and the warps of a block, share its lists by quads + lists, cut at whole groups of 32.
// What bounds it: reading the lists (7 bytes an entry with padding). List by list a lane's loads were 20 and 40 bytes
// from its neighbour's, and the passes they took through L1 were the limit: 160 us for 100M entries, 149 with the next
// round's lists on their way into L2, 144 us (4.9 TB/s) with the lists interleaved (dt_interleave_kernel).
template <bool HAS_VALS>
__global__ void __launch_bounds__(DT_THREADS, 1)
dt_partial_kernel(const float* __restrict__ x, long long n, int T, int items, int blocks_per_tile, const int* __restrict__ ptr,
                  const ushort4* __restrict__ loc, const float4* __restrict__ val, float* __restrict__ partial) {
    skml_after_previous();
    extern __shared__ __align__(16) float s_x[];
    __shared__ int s_cut[DT_THREADS / 32 + 1];
    const int tile = blockIdx.x / blocks_per_tile, warp = threadIdx.x >> 5;
    const long long x0 = (long long)tile * T;
    const int nx = n - x0 < T ? (int)(n - x0) : T;
    for (int i = threadIdx.x; i < nx; i += DT_THREADS) s_x[i] = __ldg(x + x0 + i);
    if (threadIdx.x == 0) s_x[T] = 0.f;   // the padding's slot
    dt_cuts(ptr, tile * items, (tile + 1) * items, blockIdx.x % blocks_per_tile, blocks_per_tile, s_cut);
    __syncthreads();
    dt_lists<HAS_VALS>(s_x, T, s_cut[warp], s_cut[warp + 1], ptr, loc, val, partial);
}

// ---------------------------------------------------------------------------
// Column sums of a sparse batch with a transposed index (glm_kernels.cu): the frequent columns, which hold most entries,
// from lists per (row tile, column) with the tile's coefficients in shared memory, all others one lane each with gathers
// of the coefficients from L2. A list of the frequent columns holds at most HOT_SEGMENT entries, so that every group of
// 32 lists is interleaved and no warp has much more than another: a column takes as many items as its fullest tile needs.
// ---------------------------------------------------------------------------
constexpr int HOT_SEGMENT = 4 * DT_LONG;

__device__ __forceinline__ int rows_below(const int* __restrict__ rowidx, int e0, int e1, int row) {   // first entry of a row >= row
    while (e0 < e1) {
        const int mid = e0 + ((e1 - e0) >> 1);
        if (rowidx[mid] < row) e0 = mid + 1;
        else e1 = mid;
    }
    return e0;
}

// Where the entries of a frequent column begin in each row tile, and end: bound[tile][column], one row more than tiles.
__global__ void __launch_bounds__(256)
hot_bounds_kernel(const int* __restrict__ colptr, const int* __restrict__ rowidx, const int* __restrict__ pos, int columns, int T, int tiles,
                  int* __restrict__ bound) {
    const long long all = (long long)(tiles + 1) * columns;
    for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < all; p += (long long)gridDim.x * 256) {
        const int tile = (int)(p / columns), i = pos[p - (long long)tile * columns];
        const int e0 = colptr[i], e1 = colptr[i + 1];
        bound[p] = tile == 0 ? e0 : (tile == tiles ? e1 : rows_below(rowidx, e0, e1, tile * T));
    }
}

// The entries to their lists, a warp per list: the rows of a column ascend, so an item holds the next HOT_SEGMENT entries of
// its tile. 15M entries in 0.51M lists: 77 us; as a warp per (row tile, column), one of a column that is in every row walked
// 45,000 entries while the others had ended (0.70 ms).
__global__ void __launch_bounds__(256)
hot_fill_kernel(const int* __restrict__ bound, const int* __restrict__ rowidx, const float* __restrict__ svals, const int* __restrict__ item0,
                const int* __restrict__ item_column, int columns, int items, int T, int tiles, const int* __restrict__ ptr,
                unsigned short* __restrict__ loc, float* __restrict__ val) {
    const int lane = threadIdx.x & 31;
    const long long all = (long long)tiles * items;
    for (long long p = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); p < all; p += (long long)gridDim.x * 8) {
        const int tile = (int)(p / items), item = (int)(p - (long long)tile * items), h = item_column[item];
        const int* const from = bound + (long long)tile * columns + h;
        const int lo = from[0] + HOT_SEGMENT * (item - item0[h]), n = min(from[columns] - lo, HOT_SEGMENT);
        const long long at = 4ll * ptr[p];
        for (int k = lane; k < n; k += 32) {
            loc[at + k] = (unsigned short)(rowidx[lo + k] - tile * T);
            if (svals) val[at + k] = svals[lo + k];
        }
    }
}

struct ColdColumns {   // columns bins[0 .. n) of the index: the first n_short (at most four entries) one lane each, the others eight
    const int* bins;
    int n_short, n;
    const int* colptr;
    const int* rowidx;
    const float* svals;
    const int* ucols;
};

// The other columns. Positions two turns ahead, bounds one, up to four gathers of a lane in flight. Eight lanes read the
// rows (and values) of a longer column together: one lane each, as for the short ones, took 143 instead of 97 us for the
// launch at 1M rows of 30 values.
template <bool HAS_VALS, int LANES>
__device__ __forceinline__ void cold_columns(const ColdColumns& c, int first, int last, const float* __restrict__ coef, const float* __restrict__ w,
                                             float lambda, float* __restrict__ out) {
    const int sub = threadIdx.x & (LANES - 1), turn = (int)gridDim.x * (DT_THREADS / LANES), start = ((int)blockIdx.x * DT_THREADS + (int)threadIdx.x) / LANES;
    int t = first + start;
    auto position = [&](int k) { return k < last ? c.bins[k] : -1; };
    int ni = position(t), mi = position(t + turn), n0 = 0, n1 = 0, nu = 0;
    auto bounds = [&]() {
        if (ni < 0) return;
        n0 = c.colptr[ni];
        n1 = c.colptr[ni + 1];
        nu = c.ucols[ni];
    };
    bounds();
    for (; t - (int)(threadIdx.x & 31) / LANES < last; t += turn) {   // (the whole warp)
        const int i = ni, e0 = n0, e1 = i < 0 ? n0 : n1;
        const float wv = i < 0 || sub ? 0.f : __ldg(w + nu);   // a random sector of the model: issued first
        ni = mi;
        mi = position(t + 2 * turn);
        bounds();
        float acc = 0.f;
        const unsigned int end = (unsigned int)e1;   // (steps past the end do not wrap)
        for (unsigned int e = (unsigned int)(e0 + sub); e < end; e += 4 * LANES) {
            int r[4];
            float x[4], v[4];
#pragma unroll
            for (unsigned int u = 0; u < 4; ++u) {
                r[u] = e + u * LANES < end ? c.rowidx[e + u * LANES] : -1;
                x[u] = HAS_VALS && e + u * LANES < end ? c.svals[e + u * LANES] : 1.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = r[u] >= 0 ? __ldg(coef + r[u]) : 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) acc = fmaf(v[u], x[u], acc);
        }
        if (LANES > 1) {
            __syncwarp();
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        }
        if (i >= 0 && sub == 0) out[i] = acc + lambda * wv;
    }
}

// Both kinds in one launch: the lists are bound by shared memory, the other columns by random sectors (one of the model
// per column, most of them from DRAM), so half of the warps begin with either. 500,000 rows of 30: 22 us the lists, 54 the
// others, 57 together; colsum_kernel, whose gathers of coefficients are random sectors for all columns, took 95. With
// real values, 1M rows of 30: 97 against 141 (and 8 and 13 us for the sums of the partial sums).
template <bool HAS_VALS>
__global__ void __launch_bounds__(DT_THREADS, 1)
hot_colsum_kernel(const float* __restrict__ coef, int rows, int T, int items, int blocks_per_tile, int listed, const int* __restrict__ ptr,
                  const ushort4* __restrict__ loc, const float4* __restrict__ val, float* __restrict__ partial, ColdColumns cold,
                  const float* __restrict__ w, float lambda, float* __restrict__ out) {
    skml_after_previous();
    extern __shared__ __align__(16) float s_x[];
    __shared__ int s_cut[DT_THREADS / 32 + 1];
    const int tile = blockIdx.x / blocks_per_tile, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x < listed) {   // (blocks beyond the tiles' shares have cold columns only)
        const int x0 = tile * T, nx = rows - x0 < T ? rows - x0 : T;
        for (int i = threadIdx.x; i < nx; i += DT_THREADS) s_x[i] = __ldg(coef + x0 + i);
        if (threadIdx.x == 0) s_x[T] = 0.f;   // the padding's slot
        dt_cuts(ptr, tile * items, (tile + 1) * items, blockIdx.x % blocks_per_tile, blocks_per_tile, s_cut);
        __syncthreads();
    }
#pragma unroll 1
    for (int phase = 0; phase < 2; ++phase) {
        if (phase == (warp & 1)) {
            if ((int)blockIdx.x < listed) dt_lists<HAS_VALS>(s_x, T, s_cut[warp], s_cut[warp + 1], ptr, loc, val, partial);
        } else {
            cold_columns<HAS_VALS, 8>(cold, cold.n_short, cold.n, coef, w, lambda, out);
            cold_columns<HAS_VALS, 1>(cold, 0, cold.n_short, coef, w, lambda, out);
        }
    }
}

// Frequent columns from their partial sums, info[h] = {place in out, first item, items, column}: a lane per column of one
// item, a block per column of several (`wide`).
__global__ void __launch_bounds__(256)
hot_combine_kernel(const float* __restrict__ partial, int columns, int items, int tiles, const int4* __restrict__ info, const int4* __restrict__ wide,
                   int lane_blocks, const float* __restrict__ w, float lambda, float* __restrict__ out, StepLoss loss) {
    skml_after_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) loss.settle();
    if ((int)blockIdx.x < lane_blocks) {
        const int h = blockIdx.x * 256 + threadIdx.x;
        if (h >= columns) return;
        const int4 q = info[h];
        if (q.z > 1) return;
        const float wv = __ldg(w + q.w);
        float v = 0.f;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t) v += partial[(long long)t * items + q.y];
        out[q.x] = v + lambda * wv;
        return;
    }
    __shared__ float s_part[8];
    const int4 q = wide[blockIdx.x - lane_blocks];
    const float wv = threadIdx.x == 0 ? __ldg(w + q.w) : 0.f;
    float v = 0.f;
    const int all = tiles * q.z;
#pragma unroll 4
    for (int k = threadIdx.x; k < all; k += 256) {
        const int t = k / q.z;
        v += partial[(long long)t * items + q.y + (k - t * q.z)];
    }
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.f;
        for (int k = 0; k < 8; ++k) sum += s_part[k];
        out[q.x] = sum + lambda * wv;
    }
}

// Margins of the rows from their partial sums, loss and coefficient.
__global__ void __launch_bounds__(256)
dt_coef_kernel(const float* __restrict__ partial, int rows, int tiles, const float* __restrict__ labels, int loss_id, float inv_batch,
               double* __restrict__ acc, float* __restrict__ coef) {
    skml_after_previous();
    double loss = 0.0;
    for (int r = blockIdx.x * 256 + threadIdx.x; r < rows; r += gridDim.x * 256) {
        float pre = 0.f;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t) pre += partial[(long long)t * rows + r];
        const float y = labels[r];
        loss += (double)glm_loss(loss_id, pre, y);
        coef[r] = -glm_grad(loss_id, pre, y) * inv_batch;
    }
    const double total = block_sum_double(loss);
    if (threadIdx.x == 0 && total != 0.0) atomicAdd(acc, total);
}

// Whether this lane's list of a group of 32 holds an x that is not zero (asked by lanes with `mine`; the whole warp).
__device__ __noinline__ bool holds_nonzero(const float* __restrict__ x, int T, const ushort4* __restrict__ loc, int q0, int len, bool mine) {
    const int lane = threadIdx.x & 31, most = __reduce_max_sync(0xFFFFFFFFu, len);
    auto nonzero = [&](int q) {
        const ushort4 l = __ldg(loc + q);
        return (l.x != T && x[l.x] != 0.f) || (l.y != T && x[l.y] != 0.f) || (l.z != T && x[l.z] != 0.f) || (l.w != T && x[l.w] != 0.f);
    };
    bool some = false;
    if (most <= DT_LONG) {   // interleaved
        int at = __shfl_sync(0xFFFFFFFFu, q0, 0);
        for (int k = 0; k < most; ++k) {
            const unsigned int have = __ballot_sync(0xFFFFFFFFu, len > k);
            if (mine && len > k && !some) some = nonzero(at + __popc(have & ((1u << lane) - 1u)));
            at += __popc(have);
        }
    } else {
        for (unsigned int left = __ballot_sync(0xFFFFFFFFu, mine); left; left &= left - 1) {   // one list after another
            const int src = __ffs(left) - 1;
            const int s0 = __shfl_sync(0xFFFFFFFFu, q0, src), n = __shfl_sync(0xFFFFFFFFu, len, src);
            bool any = false;
            for (int k = lane; k - lane < n && !any; k += 32) any = __any_sync(0xFFFFFFFFu, k < n && nonzero(s0 + k));
            if (lane == src) some = any;
        }
    }
    return some;
}

// Column sums from their partial sums into the (cleared) accumulator, and the columns that the batch touches: those with
// an entry in a row whose coefficient is not zero, as in the scatter (rows outside the hinge have none, and a logistic
// slope may underflow). A partial sum other than zero says so; where all are zero the column's lists are looked through.
__global__ void __launch_bounds__(256)
dt_sum_kernel(const float* __restrict__ partial, int dim, int tiles, int T, const int* __restrict__ ptr, const ushort4* __restrict__ loc,
              const float* __restrict__ coef, float* __restrict__ g, unsigned int* __restrict__ bitmap) {
    skml_after_previous();
    const int lane = threadIdx.x & 31;
    for (int c = blockIdx.x * 256 + threadIdx.x; c - lane < dim; c += gridDim.x * 256) {   // a warp a word of 32 columns
        const bool in = c < dim;
        const float* const src = partial + (in ? c : dim - 1);
        float v = 0.f;
        unsigned int bits = 0;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t) {
            const float x = src[(long long)t * dim];
            bits |= __float_as_uint(x);
            v += x;
        }
        if (in) g[c] = v;
        bool touched = in && (bits << 1) != 0u;
        for (int t = 0; t < tiles && !__all_sync(0xFFFFFFFFu, touched || !in); ++t) {
            const long long p = (long long)t * dim + c;
            const int q0 = in ? ptr[p] : 0, len = in ? ptr[p + 1] - q0 : 0;
            const bool mine = !touched && len > 0;
            if (__any_sync(0xFFFFFFFFu, mine)) touched |= holds_nonzero(coef + (long long)t * T, T, loc, q0, len, mine);
        }
        const unsigned int m = __ballot_sync(0xFFFFFFFFu, touched);
        if (lane == 0) bitmap[c >> 5] = m;
    }
}

int dt_sms() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    }
    return n;
}

unsigned blocks_for(long long n, int per, int most_per_sm) {
    const long long b = (n + per - 1) / per, most = (long long)dt_sms() * most_per_sm;
    return (unsigned)(b < 1 ? 1 : b > most ? most : b);
}

int dt_partial(const float* x, long long n, int T, int tiles, int items, const int* ptr, const unsigned short* loc, const float* val,
               float* partial, cudaStream_t stream) {
    static bool ready = false;
    if (!ready) {
        cudaError_t e = cudaFuncSetAttribute(dt_partial_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * (SKML_DT_TILE_MAX + 4));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(dt_partial_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * (SKML_DT_TILE_MAX + 4));
        if (e != cudaSuccess) return (int)e;
        ready = true;
    }
    int bpt = dt_sms() / tiles;
    if (bpt < 1) bpt = 1;
    const size_t smem = 4 * ((size_t)T + 4);
    const ushort4* l = reinterpret_cast<const ushort4*>(loc);
    const float4* v = reinterpret_cast<const float4*>(val);
    if (val) skml_launch(dt_partial_kernel<true>, tiles * bpt, DT_THREADS, smem, stream, x, n, T, items, bpt, ptr, l, v, partial);
    else skml_launch(dt_partial_kernel<false>, tiles * bpt, DT_THREADS, smem, stream, x, n, T, items, bpt, ptr, l, v, partial);
    return (int)cudaGetLastError();
}

void dt_interleave(const int* ptr, long long tiles, long long items, unsigned short* loc, float* val, cudaStream_t stream) {
    const unsigned blocks = blocks_for(tiles * ((items + 31) / 32), DT_TURN_WARPS, 16);
    ushort4* const l = reinterpret_cast<ushort4*>(loc);
    float4* const v = reinterpret_cast<float4*>(val);
    if (val) dt_interleave_kernel<true><<<blocks, DT_TURN_WARPS * 32, 0, stream>>>(ptr, (int)tiles, (int)items, l, v);
    else dt_interleave_kernel<false><<<blocks, DT_TURN_WARPS * 32, 0, stream>>>(ptr, (int)tiles, (int)items, l, v);
}

bool hot_valid(const SkmlHotColumns* h) {
    return h && h->rows > 0 && h->rows < (1ll << 31) && h->columns > 0 && h->items >= h->columns && h->tile_rows > 0 && h->tile_rows <= SKML_DT_TILE_MAX &&
           h->row_tiles * h->tile_rows >= h->rows && h->row_tiles * h->items < SKML_DT_LISTS_MAX && h->wide >= 0;
}

bool dt_valid(const SkmlDenseIndex* d) {
    return d && d->rows > 0 && d->dim > 0 && d->rows < (1ll << 31) && d->dim < (1ll << 31) && d->tile_rows > 0 && d->tile_cols > 0 &&
           d->tile_rows <= SKML_DT_TILE_MAX && d->tile_cols <= SKML_DT_TILE_MAX && d->row_tiles * d->tile_rows >= d->rows &&
           d->col_tiles * d->tile_cols >= d->dim && d->row_tiles * d->dim < SKML_DT_LISTS_MAX && d->col_tiles * d->rows < SKML_DT_LISTS_MAX;
}

}  // namespace

extern "C" int skml_dt_count(const SkmlDenseIndex* d, const long long* rowptr, const int* cols, long long row_lo, int* cnt_cols,
                             int* cnt_rows, void* stream) {
    if (!dt_valid(d) || !cnt_cols || (cnt_rows && d->col_tiles > DT_MAX_COL_TILES)) return (int)cudaErrorInvalidValue;
    dt_count_kernel<<<blocks_for(d->rows, DT_ROW_WARPS, 8), DT_ROW_WARPS * 32, 0, (cudaStream_t)stream>>>(
        rowptr, cols, row_lo, (int)d->rows, (int)d->tile_rows, (int)d->tile_cols, (int)d->col_tiles, (int)d->dim, cnt_cols, cnt_rows);
    return (int)cudaGetLastError();
}

extern "C" int skml_dt_fill(const SkmlDenseIndex* d, const long long* rowptr, const int* cols, const float* vals, long long row_lo,
                            long long entries, int* cursor, void* stream) {
    if (!dt_valid(d) || !d->c_ptr || !d->c_loc || !cursor || (d->r_ptr && d->col_tiles > DT_MAX_COL_TILES)) return (int)cudaErrorInvalidValue;
    long long parts = entries / d->row_tiles * (vals ? 7 : 2) / (16 << 20) + 1;
    if (parts > d->dim) parts = d->dim;
    dt_fill_kernel<<<blocks_for(d->rows, DT_ROW_WARPS, 8), DT_ROW_WARPS * 32, 0, (cudaStream_t)stream>>>(
        rowptr, cols, vals, row_lo, (int)d->rows, (int)d->tile_rows, (int)d->row_tiles, (int)d->tile_cols, (int)d->col_tiles, (int)d->dim,
        (int)parts, d->c_ptr, cursor,
        d->c_loc, d->c_val, d->r_ptr, d->r_loc, d->r_val);
    dt_interleave(d->c_ptr, d->row_tiles, d->dim, d->c_loc, d->c_val, (cudaStream_t)stream);
    if (d->r_ptr) dt_interleave(d->r_ptr, d->col_tiles, d->rows, d->r_loc, d->r_val, (cudaStream_t)stream);
    return (int)cudaGetLastError();
}

extern "C" int skml_dt_gradient(const SkmlDenseIndex* d, const long long* rowptr, const int* cols, const float* vals, const float* labels,
                                long long row_lo, long long nnz_padded, double avg_nnz, const float* w, int loss_id, float inv_batch,
                                double* loss_acc, float* g, unsigned int* bitmap, unsigned int* status, long long budget, void* stream_) {
    if (!dt_valid(d) || !d->c_ptr || !d->partial || !d->coef) return (int)cudaErrorInvalidValue;
    cudaStream_t stream = (cudaStream_t)stream_;
    int rc;
    if (d->r_ptr) {
        rc = dt_partial(w, d->dim, (int)d->tile_cols, (int)d->col_tiles, (int)d->rows, d->r_ptr, d->r_loc, d->r_val, d->partial, stream);
        if (rc) return rc;
        skml_launch(dt_coef_kernel, blocks_for(d->rows, 256, 8), 256, 0, stream, d->partial, (int)d->rows, (int)d->col_tiles, labels + row_lo, loss_id,
                    inv_batch, loss_acc, d->coef);
        rc = (int)cudaGetLastError();
    } else {
        rc = skml_glm_coef(rowptr, cols, vals, labels, row_lo, d->rows, nnz_padded, avg_nnz, w, d->dim, loss_id, inv_batch, loss_acc, d->coef,
                           status, budget, stream_);
    }
    if (rc) return rc;
    rc = dt_partial(d->coef, d->rows, (int)d->tile_rows, (int)d->row_tiles, (int)d->dim, d->c_ptr, d->c_loc, d->c_val, d->partial, stream);
    if (rc) return rc;
    skml_launch(dt_sum_kernel, blocks_for(d->dim, 256, 8), 256, 0, stream, d->partial, (int)d->dim, (int)d->row_tiles, (int)d->tile_rows, d->c_ptr,
                reinterpret_cast<const ushort4*>(d->c_loc), d->coef, g, bitmap);
    return (int)cudaGetLastError();
}

extern "C" int skml_hot_bounds(const SkmlHotColumns* h, const int* colptr, const int* rowidx, int* bound, void* stream) {
    if (!hot_valid(h) || !h->pos || !bound) return (int)cudaErrorInvalidValue;
    hot_bounds_kernel<<<blocks_for((h->row_tiles + 1) * h->columns, 256, 8), 256, 0, (cudaStream_t)stream>>>(
        colptr, rowidx, h->pos, (int)h->columns, (int)h->tile_rows, (int)h->row_tiles, bound);
    return (int)cudaGetLastError();
}

extern "C" int skml_hot_fill(const SkmlHotColumns* h, const int* bound, const int* item_column, const int* rowidx, const float* svals, void* stream) {
    if (!hot_valid(h) || !bound || !item_column || !h->item0 || !h->ptr || !h->loc || (svals != nullptr) != (h->val != nullptr)) return (int)cudaErrorInvalidValue;
    hot_fill_kernel<<<blocks_for(h->row_tiles * h->items, 8, 8), 256, 0, (cudaStream_t)stream>>>(
        bound, rowidx, svals, h->item0, item_column, (int)h->columns, (int)h->items, (int)h->tile_rows, (int)h->row_tiles, h->ptr, h->loc, h->val);
    dt_interleave(h->ptr, h->row_tiles, h->items, h->loc, h->val, (cudaStream_t)stream);
    return (int)cudaGetLastError();
}

extern "C" int skml_hot_colsum(const SkmlHotColumns* h, const int* bins, int n_short, int n_medium, const int* colptr, const int* rowidx, const float* svals,
                               const int* ucols, const float* coef, const float* w, float lambda, float* out, double* partials, double* tmpl,
                               void* stream_) {
    if (!hot_valid(h) || !h->ptr || !h->loc || !h->partial || !h->info || n_short < 0 || n_medium < 0 || (svals != nullptr) != (h->val != nullptr)) return (int)cudaErrorInvalidValue;
    cudaStream_t stream = (cudaStream_t)stream_;
    static bool ready = false;
    if (!ready) {
        cudaError_t e = cudaFuncSetAttribute(hot_colsum_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * (SKML_DT_TILE_MAX + 4));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(hot_colsum_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * (SKML_DT_TILE_MAX + 4));
        if (e != cudaSuccess) return (int)e;
        ready = true;
    }
    int bpt = dt_sms() / (int)h->row_tiles;
    if (bpt < 1) bpt = 1;
    const int listed = (int)h->row_tiles * bpt, grid = listed > dt_sms() ? listed : dt_sms();
    const size_t smem = 4 * ((size_t)h->tile_rows + 4);
    const ushort4* l = reinterpret_cast<const ushort4*>(h->loc);
    const float4* v = reinterpret_cast<const float4*>(h->val);
    const ColdColumns cold{bins, n_short, n_short + n_medium, colptr, rowidx, svals, ucols};
    if (svals)
        skml_launch(hot_colsum_kernel<true>, grid, DT_THREADS, smem, stream, coef, (int)h->rows, (int)h->tile_rows, (int)h->items, bpt, listed, h->ptr, l, v,
                    h->partial, cold, w, lambda, out);
    else
        skml_launch(hot_colsum_kernel<false>, grid, DT_THREADS, smem, stream, coef, (int)h->rows, (int)h->tile_rows, (int)h->items, bpt, listed, h->ptr, l, v,
                    h->partial, cold, w, lambda, out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    const int lane_blocks = (int)((h->columns + 255) / 256);
    skml_launch(hot_combine_kernel, (unsigned)(lane_blocks + h->wide), 256, 0, stream, h->partial, (int)h->columns, (int)h->items, (int)h->row_tiles,
                reinterpret_cast<const int4*>(h->info), reinterpret_cast<const int4*>(h->wide_info),
                lane_blocks, w, lambda, out, StepLoss{partials, tmpl});
    return (int)cudaGetLastError();
}
