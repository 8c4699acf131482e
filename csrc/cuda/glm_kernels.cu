// Sparse generalized-linear-model numerics for sm_100a:
//   * skml_glm_grad      : per-row margin, loss and coefficient, fused with the scatter of
//                          coefficient * feature into the dense gradient accumulator
//                          (a few lanes per row, shuffle reductions, hot columns summed
//                          in shared memory, touched-coordinate bitmap)
//   * skml_compact_*     : touched bitmap -> sorted (key, value) list with L2 term and
//                          the |v| > 1e-8 filter; decides sparse vs dense kind
//   * skml_glm_validate  : margin, loss and confusion counts over a validation shard
//   * skml_update_*      : SGD / lazy-Adam updates used by the uncompressed baselines
//
// Reference behaviour restated (paths inside the reference project, module `ml`):
//   objective/GradientDescent.scala:23-51,70-87 (minibatch gradient, 1/batch, L2 on the
//   gradient's own coordinates), objective/Loss.scala:82-137 (log / hinge / square loss and
//   their negative derivatives, +-18 cut-offs), gradient/DenseDoubleGradient.scala:51-95
//   (scatter-add, countNNZ with |v| > 1e-8, toSparse, dense iff nnz > 2/3 dim),
//   util/ValidationUtil.scala:12-41, objective/Adam.scala:27-77,
//   objective/GradientDescent.scala:89-132.
#include <math.h>

#include "glm_loss.cuh"
#include "skml_api.h"
#include "skml_device.cuh"

#define GRAD_THREADS 1024
#define SKML_EPS 1e-8f
#define GRAD_RPI 4         // rows a warp scatters at a time
#define GRAD_PRIV 256      // hottest columns kept once per warp

__device__ __forceinline__ void red_add_f32(float* p, float v) {
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

__device__ __forceinline__ void red_add_v4(float* p, float4 v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

__device__ __forceinline__ void red_or_u32(unsigned int* p, unsigned int v) {
    asm volatile("red.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Training with a scatter: margin, loss, coefficient, coefficient * feature into the accumulator. Margins are taken as
// in glm_margin_kernel below (a warp's turn is up to 32 consecutive rows, 1 << GL lanes a row); the scatter then walks
// the same rows one warp per row, GRAD_RPI rows in flight, so that the columns a warp handles at a time are distinct
// inside each row and the hottest `priv` of them can live in a private copy per warp, without atomics. Columns up to
// `hot` meet in one copy per block, the rest go to L2.
// What bounds it is same-sector traffic in L2, some 4 ns each: with a tenth of the hot columns the adds took 217 us,
// and reading the touched bitmap (256 columns a sector) before every OR took 40. So a column is marked by the add that
// finds it zero, one of many (whoever comes first does; a sum that passes through zero again only repeats the OR), and
// there is one block per SM: every block flushes its hot columns to the same sectors.
// 100,000 rows of 30: 85 -> 43 us; 50,000: 48 -> 22 us; 7,500 rows of 20: 14.4 -> 9.2 us (before: tiles staged by bulk
// copies with two block barriers each, two blocks an SM).
// The shared columns are the frequent ones where indices are assigned by frequency. Where they are not, the frequent
// columns' adds meet in L2: 100,000 rows of 30 over 10M columns, columns permuted at random, take 293 us (before: 313).
template <int GL, bool HAS_VALS>
__global__ void __launch_bounds__(GRAD_THREADS, 1)
glm_scatter_kernel(const long long* __restrict__ rowptr, const int* __restrict__ cols, const float* __restrict__ vals,
                   const float* __restrict__ labels, long long row_lo, long long row_cnt, int iters, const float* __restrict__ w,
                   float* __restrict__ g, unsigned int* __restrict__ bitmap, int loss_id, float inv_batch, int hot, int priv,
                   double* __restrict__ acc) {
    skml_after_previous();
    extern __shared__ __align__(16) float s_hot[];   // [hot], then [warps][priv]
    constexpr int LANES = 1 << GL, ROWS = 32 >> GL, PER = 4;
    const int lane = threadIdx.x & 31, sub = lane & (LANES - 1), grp = lane >> GL, nwarps = blockDim.x / 32;
    float* const s_priv = s_hot + hot + (threadIdx.x >> 5) * priv;
    for (int i = threadIdx.x; i < hot + nwarps * priv; i += blockDim.x) s_hot[i] = 0.f;
    __syncthreads();
    const int bundle = ROWS * iters;
    const long long bundles = (row_cnt + bundle - 1) / bundle, stride = (long long)gridDim.x * nwarps;
    double loss_sum = 0.0;
    for (long long b = (long long)blockIdx.x * nwarps + (threadIdx.x >> 5); b < bundles; b += stride) {
        const long long r0 = b * bundle;   // within the batch
        const int nrows = row_cnt - r0 < bundle ? (int)(row_cnt - r0) : bundle;
        const long long e_mine = rowptr[row_lo + r0 + (lane < nrows ? lane : nrows)];
        const long long e_end = rowptr[row_lo + r0 + nrows];
        const int my_row = sub * ROWS + grp;   // the row this lane evaluates
        const float y = my_row < nrows ? labels[row_lo + r0 + my_row] : 0.f;
        const long long base = __shfl_sync(0xFFFFFFFFu, e_mine, 0);
        auto turn = [&](auto off_of) {   // offsets inside the bundle in 32 bits where they fit
            using T = decltype(off_of(0ll));
            const T mine = off_of(e_mine - base), last = off_of(e_end - base);
            const int* __restrict__ cp = cols + base;
            const float* __restrict__ vp = HAS_VALS ? vals + base : nullptr;
            auto start = [&](int row) { return __shfl_sync(0xFFFFFFFFu, mine, row & 31); };
            float pre = 0.f;
#pragma unroll 2
            for (int i = 0; i < iters; ++i) {
                const int row = i * ROWS + grp;
                const T lo = start(row), nx = start(row + 1), hi = row + 1 < 32 ? nx : last;
                float sum = 0.f;
                for (T k = lo + sub; k < hi; k += PER * LANES) {
                    int c[PER];
                    float x[PER], wv[PER];
#pragma unroll
                    for (int u = 0; u < PER; ++u) {
                        const bool ok = k + u * LANES < hi;
                        c[u] = ok ? __ldg(cp + k + u * LANES) : -1;
                        x[u] = HAS_VALS ? (ok ? __ldg(vp + k + u * LANES) : 0.f) : 1.f;
                    }
#pragma unroll
                    for (int u = 0; u < PER; ++u) wv[u] = c[u] >= 0 ? __ldg(w + c[u]) : 0.f;
#pragma unroll
                    for (int u = 0; u < PER; ++u) sum = fmaf(wv[u], x[u], sum);
                }
                __syncwarp();
#pragma unroll
                for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                if (sub == i) pre = sum;
            }
            float mine_coef = 0.f;
            if (my_row < nrows) {
                loss_sum += (double)glm_loss(loss_id, pre, y);
                mine_coef = -glm_grad(loss_id, pre, y) * inv_batch;
            }
            for (int r = 0; r < nrows; r += GRAD_RPI) {
                T lo[GRAD_RPI], hi[GRAD_RPI], longest = 0;
                float coef[GRAD_RPI];
#pragma unroll
                for (int u = 0; u < GRAD_RPI; ++u) {   // rows from nrows on are empty
                    const int row = r + u;
                    lo[u] = start(row);
                    const T nx = start(row + 1);
                    hi[u] = row + 1 < 32 ? nx : last;
                    coef[u] = __shfl_sync(0xFFFFFFFFu, mine_coef, (((row & (ROWS - 1)) << GL) | (row / ROWS)) & 31);
                    if (row >= 32 || coef[u] == 0.f) hi[u] = lo[u];
                    longest = max(longest, hi[u] - lo[u]);
                }
                for (T off = lane; off - lane < longest; off += 32) {
                    int c[GRAD_RPI];
                    float add[GRAD_RPI];
                    float old[GRAD_RPI];
#pragma unroll
                    for (int u = 0; u < GRAD_RPI; ++u) {
                        const bool ok = lo[u] + off < hi[u];
                        c[u] = ok ? __ldg(cp + lo[u] + off) : -1;
                        add[u] = HAS_VALS ? (ok ? coef[u] * __ldg(vp + lo[u] + off) : 0.f) : coef[u];
                    }
#pragma unroll
                    for (int u = 0; u < GRAD_RPI; ++u) {   // the adds first: their old values come back side by side
                        old[u] = 1.f;
                        if (c[u] < hot || c[u] < 0) continue;
                        if (bitmap) old[u] = atomicAdd(g + c[u], add[u]);
                        else red_add_f32(g + c[u], add[u]);
                    }
#pragma unroll
                    for (int u = 0; u < GRAD_RPI; ++u) {
                        if (c[u] >= hot && c[u] >= 0) {
                            if (old[u] == 0.f) red_or_u32(bitmap + (c[u] >> 5), 1u << (c[u] & 31));
                        } else if (c[u] >= priv) {
                            atomicAdd(&s_hot[c[u]], add[u]);
                        }
                        // one row's columns are distinct and a warp's accesses to shared memory are ordered: a plain
                        // read-modify-write is exact
                        if (c[u] >= 0 && c[u] < priv) s_priv[c[u]] += add[u];
                        __syncwarp();
                    }
                }
            }
        };
        if (e_end - base < (1ll << 30)) turn([](long long v) { return (int)v; });
        else turn([](long long v) { return v; });
    }
    __syncthreads();
    for (int i = threadIdx.x; i < priv; i += blockDim.x) {
        float t = s_hot[i];
        for (int k = 0; k < nwarps; ++k) t += s_hot[hot + k * priv + i];
        s_hot[i] = t;
    }
    __syncthreads();
    // flush the hot columns: an add per four columns with a non-zero sum (g is 16-byte aligned, or hot is 0), an OR per
    // 32 columns where a bit is missing
    constexpr int FLUSH = 2;
    for (int i0 = 4 * (threadIdx.x - lane); i0 < hot; i0 += 4 * FLUSH * blockDim.x) {
        unsigned int mark[FLUSH], word[FLUSH];
#pragma unroll
        for (int u = 0; u < FLUSH; ++u) {
            const int i = i0 + u * 4 * (int)blockDim.x + 4 * lane;
            mark[u] = 0u;
            word[u] = ~0u;
            if (i < hot) {
                if (bitmap) word[u] = __ldcg(bitmap + (i >> 5));
                const float4 v = *reinterpret_cast<const float4*>(s_hot + i);
                mark[u] = (v.x != 0.f ? 1u : 0u) | (v.y != 0.f ? 2u : 0u) | (v.z != 0.f ? 4u : 0u) | (v.w != 0.f ? 8u : 0u);
                if (mark[u]) red_add_v4(g + i, v);
            }
            mark[u] <<= 4 * (lane & 7);
        }
#pragma unroll
        for (int u = 0; u < FLUSH; ++u) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) mark[u] |= __shfl_xor_sync(0xFFFFFFFFu, mark[u], o);
            if ((lane & 7) == 0 && (mark[u] & ~word[u])) red_or_u32(bitmap + ((i0 + u * 4 * (int)blockDim.x + 4 * lane) >> 5), mark[u]);
        }
    }
    const double tot = block_sum_double(loss_sum);
    if (threadIdx.x == 0 && tot != 0.0) atomicAdd(&acc[0], tot);
}

// Margins without a scatter. MODE 1: validation (loss + confusion counts), MODE 2: per-row coefficients (the
// gradient is summed per column by the transposed-index kernels).
// A warp takes up to 32 consecutive rows, 32 >> GL of them at a time (`iters` times) with 1 << GL lanes each; every
// row's sum ends up in the lane that owns the row, so loss and coefficient are evaluated for all of them at once.
// What bounds it is the number of gathers of w: a fully divergent load takes a cycle of the L1 per lane even when
// it hits and an L1 line while it misses, so the weights of the first `hot` columns (the frequent ones where
// indices are assigned by frequency) are kept in shared memory, which serves some ten lanes a cycle, and nothing
// is staged that would take L1 away. 500,000 rows of 30: 80 -> 61 us; 1M rows of 30 with values: 208 -> 102 us
// (before: a warp per row, tiles staged by bulk copies, 103 warp instructions per 32 entries). Four blocks an SM instead of
// three (PER_SM), at 32 registers with a few spills: 58 and 99 us, 62,500 rows 15 -> 13; one block of 1024 threads with six
// times the hot columns took 80 and 129: what counts is the gathers in flight. That holds where they go to DRAM; see
// margin_launch_gl for where three blocks are the better choice.
#define MARGIN_THREADS 512
struct ClearSlots {   // out[slot[0 .. n)] = 0
    float* out;
    const int* slot;
    int n;
};
template <int MODE, int GL, bool HAS_VALS, int PER_SM>
__global__ void __launch_bounds__(MARGIN_THREADS, PER_SM)
glm_margin_kernel(const long long* __restrict__ rowptr, const int* __restrict__ cols, const float* __restrict__ vals,
                  const float* __restrict__ labels, long long row_lo, long long row_cnt, int iters, const float* __restrict__ w,
                  int hot, int loss_id, float inv_batch, double* __restrict__ acc, float* __restrict__ out, ClearSlots clear) {
    skml_after_previous();
    extern __shared__ __align__(16) float s_w[];
    if (MODE == 2)   // what the column sums behind this launch add to
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < clear.n; i += gridDim.x * blockDim.x) clear.out[clear.slot[i]] = 0.f;
    constexpr int LANES = 1 << GL, ROWS = 32 >> GL, PER = 4;   // rows of an iteration, entries of a lane in flight
    const int lane = threadIdx.x & 31, sub = lane & (LANES - 1), grp = lane >> GL;
    for (int i = threadIdx.x; i < hot / 4; i += blockDim.x) reinterpret_cast<float4*>(s_w)[i] = __ldg(reinterpret_cast<const float4*>(w) + i);
    __syncthreads();
    const int bundle = ROWS * iters;   // rows of a warp's turn
    const long long bundles = (row_cnt + bundle - 1) / bundle, stride = (long long)gridDim.x * (blockDim.x / 32);
    double loss_sum = 0.0;
    unsigned int tp = 0, tn = 0, fp = 0, fn = 0;
    for (long long b = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); b < bundles; b += stride) {
        const long long r0 = b * bundle;   // within the batch
        const int nrows = row_cnt - r0 < bundle ? (int)(row_cnt - r0) : bundle;
        const long long e_mine = rowptr[row_lo + r0 + (lane < nrows ? lane : nrows)];
        const long long e_end = rowptr[row_lo + r0 + nrows];
        const int my_row = sub * ROWS + grp;   // the row this lane evaluates
        const float y = my_row < nrows ? labels[row_lo + r0 + my_row] : 0.f;
        const long long base = __shfl_sync(0xFFFFFFFFu, e_mine, 0);
        const long long span = e_end - base;
        float pre = 0.f;
        auto row_sums = [&](auto off_of) {   // offsets inside the bundle in 32 bits where they fit
            using T = decltype(off_of(0ll));
            const T mine = off_of(e_mine - base), last = off_of(span);
            const int* __restrict__ cp = cols + base;
            const float* __restrict__ vp = HAS_VALS ? vals + base : nullptr;
#pragma unroll 2
            for (int i = 0; i < iters; ++i) {
                const int row = i * ROWS + grp;
                const T lo = __shfl_sync(0xFFFFFFFFu, mine, row), nx = __shfl_sync(0xFFFFFFFFu, mine, (row + 1) & 31);
                const T hi = row + 1 < 32 ? nx : last;   // rows from nrows on are empty: every later offset is the end
                float sum = 0.f;
                for (T k = lo + sub; k < hi; k += PER * LANES) {
                    int c[PER];
                    float x[PER], wv[PER];
#pragma unroll
                    for (int u = 0; u < PER; ++u) {
                        const bool ok = k + u * LANES < hi;
                        c[u] = ok ? __ldcs(cp + k + u * LANES) : -1;
                        x[u] = HAS_VALS ? (ok ? __ldcs(vp + k + u * LANES) : 0.f) : 1.f;
                    }
#pragma unroll
                    for (int u = 0; u < PER; ++u) {
                        wv[u] = 0.f;
                        if (c[u] >= hot) wv[u] = __ldg(w + c[u]);
                        else if (c[u] >= 0) wv[u] = s_w[c[u]];
                    }
#pragma unroll
                    for (int u = 0; u < PER; ++u) sum = fmaf(wv[u], x[u], sum);
                }
                __syncwarp();
#pragma unroll
                for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                if (sub == i) pre = sum;
            }
        };
        if (span < (1ll << 30)) row_sums([](long long v) { return (int)v; });
        else row_sums([](long long v) { return v; });
        if (my_row < nrows) {
            loss_sum += (double)glm_loss(loss_id, pre, y);
            if (MODE == 2) {
                out[r0 + my_row] = -glm_grad(loss_id, pre, y) * inv_batch;
            } else {
                const float z = pre * y;
                if (z > 0.f) {
                    if (pre > 0.f) ++tp; else ++tn;
                } else if (z < 0.f) {
                    if (pre > 0.f) ++fp; else ++fn;
                }
                if (out) out[r0 + my_row] = pre;
            }
        }
    }
    double tot = block_sum_double(loss_sum);
    if (threadIdx.x == 0 && tot != 0.0) atomicAdd(&acc[0], tot);
    if (MODE == 1) {
        double c0 = block_sum_double((double)tp), c1 = block_sum_double((double)tn);
        double c2 = block_sum_double((double)fp), c3 = block_sum_double((double)fn);
        if (threadIdx.x == 0) {
            if (c0 != 0.0) atomicAdd(&acc[1], c0);
            if (c1 != 0.0) atomicAdd(&acc[2], c1);
            if (c2 != 0.0) atomicAdd(&acc[3], c2);
            if (c3 != 0.0) atomicAdd(&acc[4], c3);
        }
    }
}

static int g_sm_count = 0;
static int sm_count() {
    if (g_sm_count == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (g_sm_count <= 0) g_sm_count = 148;
    }
    return g_sm_count;
}

// Columns [0, margin_hot) of w in shared memory: at most 8192 (32 KB, four blocks an SM keep 92 KB of L1), no more
// than a block has entries to look up (reading them in is then an eighth of the sectors of the gathers at most),
// whole 16-byte units. Below 1024 the copy is not worth its barrier.
static int margin_hot(long long entries, long long blocks, long long dim, const float* w) {
    long long hot = entries / (blocks > 0 ? blocks : 1);
    if (hot > 8192) hot = 8192;
    if (hot > dim) hot = dim;
    hot &= ~255ll;
    return hot < 1024 || ((uintptr_t)w & 15) ? 0 : (int)hot;
}

// Rows of a warp's turn (iterations of 32 >> gl rows, 1 << gl at most), warps per block and blocks, for blocks of at
// most `max_warps` warps, `per_sm` of them on an SM. Few rows: one turn for every warp slot of the chip, down to one
// iteration, in blocks of as many warps as spread the turns over all SMs. Many: of the turn lengths from half the
// maximum on, the one whose last round of turns is fullest (500,000 rows in turns of 32 are 2.2 rounds, of 24 are 2.93).
struct TurnShape {
    int iters, warps, grid;
};
static TurnShape turn_shape(long long row_cnt, int gl, int max_warps, int per_sm) {
    const long long blocks = (long long)per_sm * sm_count(), slots = blocks * max_warps, rows = 32 >> gl;
    const int most = 1 << gl;
    auto turns = [&](long long iters) { return (row_cnt + rows * iters - 1) / (rows * iters); };
    TurnShape t;
    const long long even = (row_cnt + rows * slots - 1) / (rows * slots);   // iterations in a single round
    t.iters = even < 1 ? 1 : (int)(even < most ? even : most);
    if (even > most) {
        double best = 0.0;
        for (int it = most; it >= (most + 1) / 2; --it) {
            const long long n = turns(it);
            const double fill = (double)n / (double)((n + slots - 1) / slots * slots);
            if (fill > best + 0.02) {
                best = fill;
                t.iters = it;
            }
        }
    }
    const long long n = turns(t.iters);
    long long warps = (n + blocks - 1) / blocks;
    if (warps > max_warps) warps = max_warps;
    t.warps = (int)warps;
    const long long grid = (n + warps - 1) / warps;
    t.grid = (int)(grid < blocks ? grid : blocks);
    return t;
}

template <int MODE, int GL>
static int margin_launch_gl(const long long* rowptr, const int* cols, const float* vals, const float* labels, long long row_lo,
                            long long row_cnt, double avg_nnz, const float* w, long long dim, int loss_id, float inv_batch, double* acc,
                            float* out, const ClearSlots& clear, cudaStream_t stream) {
    // Spills cost the validation's counters and the values more than a fourth block brings, unless the gathers miss L2.
    // Three / four blocks, us: dim 10M, 1M rows of 8 values 35 / 40 (validated 40 / 47, binary and validated 38 / 42), dim 1M,
    // 100,000 rows of 250 values 51 / 58 (56 / 65); dim 50M, 200,000 rows of 30 values 21.0 / 20.5, dim 100M, 1M rows 93 / 89.
    const bool four = (MODE == 2 && !vals) || dim > (16ll << 20);
    const TurnShape t = turn_shape(row_cnt, GL, MARGIN_THREADS / 32, four ? 4 : 3);
    const int iters = t.iters, warps = t.warps, grid = t.grid;
    const int hot = margin_hot((long long)(row_cnt * avg_nnz), grid, dim, w);
    auto launch = [&](auto kernel) {
        skml_launch(kernel, (unsigned)grid, (unsigned)(32 * warps), hot * sizeof(float), stream,
                    rowptr, cols, vals, labels, row_lo, row_cnt, iters, w, hot, loss_id, inv_batch, acc, out, clear);
    };
    if (vals) {
        if (four) launch(glm_margin_kernel<MODE, GL, true, 4>);
        else launch(glm_margin_kernel<MODE, GL, true, 3>);
    } else if (four || MODE == 2) {
        launch(glm_margin_kernel<MODE, GL, false, 4>);
    } else {
        launch(glm_margin_kernel<MODE, GL, false, 3>);
    }
    return (int)cudaGetLastError();
}

// Lanes per row: four entries of a lane are in flight at a time, so a row of the average length takes one trip.
template <int MODE>
static int margin_launch(const long long* rowptr, const int* cols, const float* vals, const float* labels, long long row_lo,
                         long long row_cnt, double avg_nnz, const float* w, long long dim, int loss_id, float inv_batch, double* acc,
                         float* out, cudaStream_t stream, const ClearSlots& clear = {nullptr, nullptr, 0}) {
    if (row_cnt <= 0) return 0;
    auto go = avg_nnz <= 16.0 ? margin_launch_gl<MODE, 2> : avg_nnz <= 40.0 ? margin_launch_gl<MODE, 3>
            : avg_nnz <= 96.0 ? margin_launch_gl<MODE, 4> : margin_launch_gl<MODE, 5>;
    return go(rowptr, cols, vals, labels, row_lo, row_cnt, avg_nnz, w, dim, loss_id, inv_batch, acc, out, clear, stream);
}

// Columns summed per block: no more than the caller allows, and only those whose adds would queue up in L2: with
// frequencies falling like 1 / rank, rank r of E entries gets about E / (9 r), so a sector of eight columns is busy
// for half a microsecond and more (4 to 10 ns an add) down to rank E / 110. The others would only lengthen the flush
// (7,500 rows of 20: 15 us with 8192 columns). Hot columns leave in 16-byte units.
static int grad_hot(long long entries, int limit, const float* g) {
    long long hot = entries / 128;
    if (hot < GRAD_PRIV) hot = GRAD_PRIV;
    if (hot > 16384) hot = 16384;
    if (hot > limit) hot = limit;
    return hot < 0 || ((uintptr_t)g & 15) ? 0 : (int)(hot & ~31ll);
}

template <int GL>
static int grad_launch_gl(const long long* rowptr, const int* cols, const float* vals, const float* labels, long long row_lo,
                          long long row_cnt, double avg_nnz, const float* w, float* g, unsigned int* bitmap, int loss_id,
                          float inv_batch, int hot_limit, double* acc, cudaStream_t stream) {
    const TurnShape t = turn_shape(row_cnt, GL, GRAD_THREADS / 32, 1);
    const int hot = grad_hot((long long)(row_cnt * avg_nnz), hot_limit, g), priv = hot < GRAD_PRIV ? hot : GRAD_PRIV;
    const size_t smem = ((size_t)hot + (size_t)priv * t.warps) * sizeof(float);
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(glm_scatter_kernel<GL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        cudaFuncSetAttribute(glm_scatter_kernel<GL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        attr_set = true;
    }
    if (vals)
        skml_launch(glm_scatter_kernel<GL, true>, t.grid, 32 * t.warps, smem, stream, rowptr, cols, vals, labels, row_lo, row_cnt, t.iters, w, g,
                    bitmap, loss_id, inv_batch, hot, priv, acc);
    else
        skml_launch(glm_scatter_kernel<GL, false>, t.grid, 32 * t.warps, smem, stream, rowptr, cols, vals, labels, row_lo, row_cnt, t.iters, w, g,
                    bitmap, loss_id, inv_batch, hot, priv, acc);
    return (int)cudaGetLastError();
}

extern "C" int skml_glm_grad(const long long* rowptr, const int* cols, const float* vals, const float* labels,
                             long long row_lo, long long row_cnt, long long nnz_padded, double avg_nnz,
                             const float* w, float* g, unsigned int* bitmap, int loss_id, float inv_batch, int hot,
                             double* loss_acc, unsigned int* status, long long budget, void* stream) {
    (void)nnz_padded;
    (void)status;
    (void)budget;   // nothing in it waits
    if (row_cnt <= 0) return 0;
    auto go = avg_nnz <= 16.0 ? grad_launch_gl<2> : avg_nnz <= 40.0 ? grad_launch_gl<3> : avg_nnz <= 96.0 ? grad_launch_gl<4> : grad_launch_gl<5>;
    return go(rowptr, cols, vals, labels, row_lo, row_cnt, avg_nnz, w, g, bitmap, loss_id, inv_batch, hot, loss_acc, (cudaStream_t)stream);
}

extern "C" int skml_glm_validate(const long long* rowptr, const int* cols, const float* vals, const float* labels,
                                 long long row_lo, long long row_cnt, long long nnz_padded, double avg_nnz,
                                 const float* w, long long dim, int loss_id, double* acc5, float* margins, unsigned int* status,
                                 long long budget, void* stream) {
    (void)nnz_padded;
    (void)status;
    (void)budget;   // nothing in it waits
    return margin_launch<1>(rowptr, cols, vals, labels, row_lo, row_cnt, avg_nnz, w, dim, loss_id, 1.f, acc5, margins, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Compaction of the touched bitmap into a sorted sparse gradient. A warp owns `wpw` consecutive bitmap
// words, walked 32 at a time; the count pass leaves one count per warp and one per block, and every block of
// the write pass adds up the blocks before its own, so there is no scan launch in between.
// What bounds it is the chain bitmap word -> g and w -> stores of each group of 32 words, so the split is
// by latency: as few words per warp as the count array allows (wpw = 8 up to 4M coordinates, one group of 32 up
// to 16M), which spreads 100k coordinates over 49 blocks. (One 1024-thread block per 131,072 coordinates put
// them on one SM: 39 + 2 + 30 us; 1M coordinates on eight: 55 + 2 + 31 us. Four groups a warp at 10M: 29 + 23 us.)
// meta[0] = nnz, meta[1] = kind (1 sparse, 2 dense, 0 empty)
// ---------------------------------------------------------------------------
#define COMPACT_THREADS 256
#define COMPACT_WARPS (COMPACT_THREADS / 32)
#define COMPACT_MIN_WPW 8
#define COMPACT_MAX_BLOCKS 2048  // every block of the write pass reads the totals of all (8 KB)
#define COMPACT_SPARSE_BITS 4    // words with at most this many bits are walked by one lane
#define COMPACT_DENSE_BATCH 8    // dense words whose loads are in flight together

struct CompactShape {
    int wpw;      // bitmap words per warp: the smallest power of two from COMPACT_MIN_WPW that needs no more than
                  // COMPACT_MAX_BLOCKS blocks
    int nwarps, nblocks;
};

static CompactShape compact_shape(long long dim) {
    const long long nwords = (dim + 31) / 32;
    CompactShape c;
    c.wpw = COMPACT_MIN_WPW;
    while (nwords > (long long)c.wpw * COMPACT_WARPS * COMPACT_MAX_BLOCKS) c.wpw *= 2;
    c.nwarps = (int)((nwords + c.wpw - 1) / c.wpw);
    c.nblocks = (c.nwarps + COMPACT_WARPS - 1) / COMPACT_WARPS;
    return c;
}

__global__ void __launch_bounds__(COMPACT_THREADS)
compact_count_kernel(float* __restrict__ g, const float* __restrict__ w, unsigned int* __restrict__ bitmap,
                     long long nwords, int dim, float lambda, int wpw, int nwarps, unsigned int* __restrict__ warp_counts) {
    skml_after_previous();
    // Words with few bits are walked by their own lane; words with many bits are walked by the whole
    // warp, one bit per lane, so that the g / w accesses of dense regions are coalesced. Loads are issued
    // in batches before any of them is consumed (several memory round trips in flight per warp).
    // The filtered value g + lambda * w is stored back into g so that the write pass reads one
    // array only.
    const int lane = threadIdx.x & 31;
    __shared__ unsigned int s_cnt[COMPACT_WARPS];
    const int gw = blockIdx.x * COMPACT_WARPS + (threadIdx.x >> 5);
    const long long wbase = (long long)gw * wpw;
    const long long wend = gw >= nwarps ? wbase : (wbase + wpw < nwords ? wbase + wpw : nwords);
    unsigned int cnt = 0;
    unsigned int next = wbase + lane < wend ? bitmap[wbase + lane] : 0u;
    for (long long gbase = wbase; gbase < wend; gbase += 32) {
        const long long wi = gbase + lane;
        const unsigned int bits = next;
        next = wi + 32 < wend ? bitmap[wi + 32] : 0u;   // one group ahead
        unsigned int keep = bits;
        const int pc = __popc(bits);
        if (pc > 0 && pc <= COMPACT_SPARSE_BITS) {
            int tpos[COMPACT_SPARSE_BITS];
            bool inb[COMPACT_SPARSE_BITS];
            float gv[COMPACT_SPARSE_BITS], wv[COMPACT_SPARSE_BITS];
            unsigned int b = bits;
#pragma unroll
            for (int j = 0; j < COMPACT_SPARSE_BITS; ++j) {
                tpos[j] = b ? __ffs(b) - 1 : -1;
                b &= b - 1;
                const long long k = wi * 32 + (tpos[j] < 0 ? 0 : tpos[j]);
                inb[j] = tpos[j] >= 0 && k < dim;
                gv[j] = inb[j] ? g[k] : 0.f;
                wv[j] = inb[j] ? w[k] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < COMPACT_SPARSE_BITS; ++j) {
                if (tpos[j] < 0) continue;
                if (!inb[j]) {  // a bit beyond dim (never set by the gradient kernel): drop it
                    keep &= ~(1u << tpos[j]);
                    continue;
                }
                const long long k = wi * 32 + tpos[j];
                const float v = gv[j] + lambda * wv[j];
                if (fabsf(v) > SKML_EPS) {
                    g[k] = v;
                } else {
                    keep &= ~(1u << tpos[j]);
                    g[k] = 0.f;
                }
            }
        }
        unsigned int dense = __ballot_sync(0xFFFFFFFFu, pc > COMPACT_SPARSE_BITS);
        while (dense) {
            int jj[COMPACT_DENSE_BATCH];
            unsigned int wb[COMPACT_DENSE_BATCH];
            float gv[COMPACT_DENSE_BATCH], wv[COMPACT_DENSE_BATCH];
#pragma unroll
            for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                jj[u] = dense ? __ffs(dense) - 1 : -1;
                dense &= dense - 1;
                wb[u] = __shfl_sync(0xFFFFFFFFu, bits, jj[u] < 0 ? 0 : jj[u]);
                const long long k = (gbase + (jj[u] < 0 ? 0 : jj[u])) * 32 + lane;
                const bool active = jj[u] >= 0 && ((wb[u] >> lane) & 1u) && k < dim;
                gv[u] = active ? g[k] : 0.f;
                wv[u] = active ? w[k] : 0.f;
                if (!active) wb[u] &= ~(1u << lane);
            }
#pragma unroll
            for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                if (jj[u] < 0) continue;  // uniform over the warp
                const bool active = (wb[u] >> lane) & 1u;
                bool ok = false;
                if (active) {
                    const long long k = (gbase + jj[u]) * 32 + lane;
                    const float v = gv[u] + lambda * wv[u];
                    ok = fabsf(v) > SKML_EPS;
                    g[k] = ok ? v : 0.f;
                }
                const unsigned int kb = __ballot_sync(0xFFFFFFFFu, ok);
                if (lane == jj[u]) keep = kb;
            }
        }
        if (keep != bits) bitmap[wi] = keep;
        cnt += __popc(keep);
    }
    cnt = warp_sum(cnt);
    if (lane == 0) {
        s_cnt[threadIdx.x >> 5] = cnt;
        if (gw < nwarps) warp_counts[gw] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = 0;
#pragma unroll
        for (int i = 0; i < COMPACT_WARPS; ++i) t += s_cnt[i];
        warp_counts[nwarps + blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(COMPACT_THREADS)
compact_write_kernel(float* __restrict__ g, const float* __restrict__ w, unsigned int* __restrict__ bitmap,
                     long long nwords, int dim, float lambda, int wpw, int nwarps,
                     const unsigned int* __restrict__ warp_counts, long long* __restrict__ meta, int* __restrict__ keys,
                     float* __restrict__ vals, float* __restrict__ dense_vals, long long capacity, unsigned int* status, StepLoss loss) {
    skml_after_previous();
    __shared__ unsigned int s_before[COMPACT_WARPS], s_total[COMPACT_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gw0 = blockIdx.x * COMPACT_WARPS, gw = gw0 + warp;
    const long long wbase = (long long)gw * wpw;
    const long long wend = gw >= nwarps ? wbase : (wbase + wpw < nwords ? wbase + wpw : nwords);
    unsigned int next = wbase + lane < wend ? bitmap[wbase + lane] : 0u;   // in flight while the counts are added up
    unsigned int before = 0, total = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += COMPACT_THREADS) {
        const unsigned int c = warp_counts[nwarps + i];
        total += c;
        if (i < (int)blockIdx.x) before += c;
    }
    before = warp_sum(before);
    total = warp_sum(total);
    if (lane == 0) {
        s_before[warp] = before;
        s_total[warp] = total;
    }
    __syncthreads();
    before = total = 0;
#pragma unroll
    for (int i = 0; i < COMPACT_WARPS; ++i) {
        before += s_before[i];
        total += s_total[i];
    }
    const int kind = total == 0 ? 0 : ((dense_vals != nullptr && (long long)total > (long long)dim * 2 / 3) ? 2 : 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        meta[0] = total;
        meta[1] = kind;
        loss.settle();
    }
    if (gw >= nwarps) return;
    if (kind == 2) {
        // dense kind: every coordinate is shipped. Kept coordinates already hold g + lambda*w
        // (count pass); all others contribute lambda * w alone.
        for (long long gbase = wbase; gbase < wend; gbase += 32) {
            const long long wi = gbase + lane;
            const unsigned int bits = next;
            next = wi + 32 < wend ? bitmap[wi + 32] : 0u;
            if (wi < wend) bitmap[wi] = 0;
            const int words = wend - gbase < 32 ? (int)(wend - gbase) : 32;
            for (int j0 = 0; j0 < words; j0 += COMPACT_DENSE_BATCH) {
                float v[COMPACT_DENSE_BATCH];
#pragma unroll
                for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                    const unsigned int wb = __shfl_sync(0xFFFFFFFFu, bits, (j0 + u) & 31);
                    const long long k = (gbase + j0 + u) * 32 + lane;
                    v[u] = 0.f;
                    if (j0 + u < words && k < dim) v[u] = ((wb >> lane) & 1u) ? g[k] : lambda * w[k];
                }
#pragma unroll
                for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                    const long long k = (gbase + j0 + u) * 32 + lane;
                    if (j0 + u < words && k < dim) {
                        dense_vals[k] = v[u];
                        g[k] = 0.f;
                    }
                }
            }
        }
        return;
    }
    long long out = before;   // keys in front of this warp's words
    for (int i = 0; i < warp; ++i) out += warp_counts[gw0 + i];
    bool overflow = false;
    for (long long gbase = wbase; gbase < wend; gbase += 32) {
        const long long wi = gbase + lane;
        const unsigned int bits = next;
        next = wi + 32 < wend ? bitmap[wi + 32] : 0u;
        const int pc = __popc(bits);
        unsigned int inc = (unsigned int)pc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += t;
        }
        const unsigned int ex = inc - (unsigned int)pc;
        const unsigned int grp_total = __shfl_sync(0xFFFFFFFFu, inc, 31);
        if (pc > 0 && pc <= COMPACT_SPARSE_BITS) {
            int tpos[COMPACT_SPARSE_BITS];
            float gv[COMPACT_SPARSE_BITS];
            unsigned int b = bits;
#pragma unroll
            for (int j = 0; j < COMPACT_SPARSE_BITS; ++j) {
                tpos[j] = b ? __ffs(b) - 1 : -1;
                b &= b - 1;
                gv[j] = tpos[j] >= 0 ? g[wi * 32 + tpos[j]] : 0.f;
            }
            long long pos = out + ex;
#pragma unroll
            for (int j = 0; j < COMPACT_SPARSE_BITS; ++j) {
                if (tpos[j] < 0) continue;
                const long long k = wi * 32 + tpos[j];
                if (pos < capacity) {
                    keys[pos] = (int)k;
                    vals[pos] = gv[j];
                } else {
                    overflow = true;
                }
                g[k] = 0.f;
                ++pos;
            }
        }
        unsigned int dense = __ballot_sync(0xFFFFFFFFu, pc > COMPACT_SPARSE_BITS);
        while (dense) {
            int jj[COMPACT_DENSE_BATCH];
            unsigned int wb[COMPACT_DENSE_BATCH], exj[COMPACT_DENSE_BATCH];
            float gv[COMPACT_DENSE_BATCH];
#pragma unroll
            for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                jj[u] = dense ? __ffs(dense) - 1 : -1;
                dense &= dense - 1;
                const int src = jj[u] < 0 ? 0 : jj[u];
                wb[u] = __shfl_sync(0xFFFFFFFFu, bits, src);
                exj[u] = __shfl_sync(0xFFFFFFFFu, ex, src);
                if (jj[u] < 0) wb[u] = 0u;
                gv[u] = ((wb[u] >> lane) & 1u) ? g[(gbase + src) * 32 + lane] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < COMPACT_DENSE_BATCH; ++u) {
                if (!((wb[u] >> lane) & 1u)) continue;
                const long long k = (gbase + jj[u]) * 32 + lane;
                const long long pos = out + exj[u] + __popc(wb[u] & ((1u << lane) - 1u));
                if (pos < capacity) {
                    keys[pos] = (int)k;
                    vals[pos] = gv[u];
                } else {
                    overflow = true;
                }
                g[k] = 0.f;
            }
        }
        if (bits) bitmap[wi] = 0;
        out += grp_total;
    }
    if (overflow) skml_set_status(status, SKML_CAPACITY, 0x20u);
}

static int compact_launch(float* g, const float* w, unsigned int* bitmap, int dim, float lambda, unsigned int* warp_counts,
                          long long* meta, int* keys, float* vals, float* dense_vals, long long capacity, unsigned int* status,
                          cudaStream_t stream, const StepLoss& loss = {nullptr, nullptr}) {
    const long long nwords = ((long long)dim + 31) / 32;
    const CompactShape c = compact_shape(dim);
    skml_launch(compact_count_kernel, c.nblocks, COMPACT_THREADS, 0, stream, g, w, bitmap, nwords, dim, lambda, c.wpw, c.nwarps, warp_counts);
    skml_launch(compact_write_kernel, c.nblocks, COMPACT_THREADS, 0, stream, g, w, bitmap, nwords, dim, lambda, c.wpw, c.nwarps, warp_counts,
                meta, keys, vals, dense_vals, capacity, status, loss);
    return (int)cudaGetLastError();
}

// skml_compact that also settles the step's loss partials.
extern "C" int skml_compact_settle(float* g, const float* w, unsigned int* bitmap, int dim, float lambda, unsigned int* block_counts, long long* meta,
                   int* keys, float* vals, float* dense_vals, long long capacity, unsigned int* status, double* partials, double* tmpl,
                   void* stream) {
    return compact_launch(g, w, bitmap, dim, lambda, block_counts, meta, keys, vals, dense_vals, capacity, status, (cudaStream_t)stream,
                          StepLoss{partials, tmpl});
}

extern "C" int skml_compact(float* g, const float* w, unsigned int* bitmap, int dim, float lambda,
                            unsigned int* block_counts, long long* meta, int* keys, float* vals, float* dense_vals,
                            long long capacity, unsigned int* status, void* stream_) {
    return compact_launch(g, w, bitmap, dim, lambda, block_counts, meta, keys, vals, dense_vals, capacity, status,
                          (cudaStream_t)stream_);
}

// Entries of the caller's count array.
extern "C" long long skml_compact_blocks(int dim) {
    const CompactShape c = compact_shape(dim);
    return c.nwarps + c.nblocks;
}

// ---------------------------------------------------------------------------
// Updates for the uncompressed baselines (the compressed path updates inside the
// fused decode kernel).
// opt[0] = lr, opt[1] = sqrt(1 - beta2^t) / (1 - beta1^t) for Adam.
// ---------------------------------------------------------------------------
// ms: elements between the moments of neighbouring coordinates (1: plain arrays; 4: m and v point into
// one array of per-coordinate quads, so both moments of a coordinate come with one memory sector).
__device__ __forceinline__ void apply_update(float* w, float* m, float* v, long long k, float gval, int adam,
                                             float lr, float adam_scale, long long ms) {
    if (!adam) {
        w[k] -= lr * gval;
    } else {
        const long long q = k * ms;
        float mt = 0.9f * m[q] + 0.1f * gval;
        float vt = 0.999f * v[q] + 0.001f * gval * gval;
        w[k] -= lr * adam_scale * mt / (sqrtf(vt) + 1e-8f);
        m[q] = mt;
        v[q] = vt;
    }
}

__global__ void update_dense_kernel(float* w, float* m, float* v, const float* g, long long dim, float scale,
                                    int adam, float lr, float adam_scale, int sparse_only, long long ms) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (long long)gridDim.x * blockDim.x) {
        float gv = g[i] * scale;
        if (sparse_only && gv == 0.f) continue;
        apply_update(w, m, v, i, gv, adam, lr, adam_scale, ms);
    }
}

__global__ void update_sparse_kernel(float* w, float* m, float* v, const int* keys, const float* vals,
                                     const long long* n_ptr, long long n_max, float scale, int adam, float lr,
                                     float adam_scale, long long ms, const unsigned int* status) {
    skml_after_previous();
    long long n = n_ptr ? *n_ptr : n_max;
    if (n > n_max) n = n_max;
    if (skml_failed(status)) n = 0;   // (read beside the count)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        apply_update(w, m, v, keys[i], vals[i] * scale, adam, lr, adam_scale, ms);
}

extern "C" int skml_update_dense(float* w, float* m, float* v, const float* g, long long dim, float scale, int adam,
                                 float lr, float adam_scale, int sparse_only, int adam_stride, void* stream) {
    int grid = sm_count() * 8;
    update_dense_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(w, m, v, g, dim, scale, adam, lr, adam_scale,
                                                                sparse_only, adam_stride > 1 ? adam_stride : 1);
    return (int)cudaGetLastError();
}

extern "C" int skml_update_sparse(float* w, float* m, float* v, const int* keys, const float* vals,
                                  const long long* n_ptr, long long n_max, float scale, int adam, float lr,
                                  float adam_scale, int adam_stride, const unsigned int* status, void* stream) {
    int grid = sm_count() * 8;
    skml_launch(update_sparse_kernel, grid, 256, 0, (cudaStream_t)stream, w, m, v, keys, vals, n_ptr, n_max, scale, adam, lr,
                adam_scale, adam_stride > 1 ? adam_stride : 1, status);
    return (int)cudaGetLastError();
}

// Sum of squares of the model in one launch: a contiguous slice per block, the partial sums added in
// block order by the last block to finish (so the result does not depend on the schedule).
constexpr int NORM_BLOCKS = 592;

__global__ void __launch_bounds__(256) weight_norm_kernel(const float* __restrict__ w, long long dim, double lambda,
                                                          double* __restrict__ sumsq_out, double* __restrict__ reg_out,
                                                          double* __restrict__ partials, unsigned int* __restrict__ counter) {
    skml_after_previous();
    const long long per = ((dim + gridDim.x - 1) / gridDim.x + 3) & ~3ll;
    const long long lo = per * blockIdx.x, hi = lo + per < dim ? lo + per : dim;
    double acc = 0.0;
    for (long long i = lo + 4ll * threadIdx.x; i < hi; i += 4ll * blockDim.x) {
        if (i + 4 <= hi) {
            const float4 v = *reinterpret_cast<const float4*>(w + i);  // lo is a multiple of 4: 16-byte aligned
            acc += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
        } else {
            for (long long j = i; j < hi; ++j) acc += (double)w[j] * w[j];
        }
    }
    __shared__ double sh[256];
    __shared__ bool last;
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = sh[0];
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) t += __ldcg(partials + b);
    sh[threadIdx.x] = t;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *counter = 0;
        if (sumsq_out) sumsq_out[0] = sh[0];
        if (reg_out) reg_out[0] = lambda * sqrt(sh[0]);
    }
}

extern "C" long long skml_weight_norm_scratch_bytes() { return (NORM_BLOCKS + 2) * 8; }

extern "C" int skml_weight_norm(const float* w, long long dim, double lambda, double* sumsq_out, double* reg_out,
                                void* scratch, void* stream) {
    if (!w || !scratch || dim < 0) return (int)cudaErrorInvalidValue;
    double* partials = reinterpret_cast<double*>(scratch);
    unsigned int* counter = reinterpret_cast<unsigned int*>(partials + NORM_BLOCKS);
    skml_launch(weight_norm_kernel, NORM_BLOCKS, 256, 0, (cudaStream_t)stream, w, dim, lambda, sumsq_out, reg_out, partials, counter);
    return (int)cudaGetLastError();
}

// Update from a dense accumulator on exactly the coordinates of the gathered key lists, clearing the
// accumulator on the way: the work is proportional to the number of gathered keys, not to the model
// dimension. One launch per list (keys are distinct inside a list, so a launch touches every word at
// most once); a coordinate shared by several lists is updated by the first one and found cleared
// (exactly zero, skipped) by the later ones. A sum that is exactly zero is a no-op, as in the
// `sparse_only` dense update.
__global__ void update_gathered_kernel(float* w, float* m, float* v, float* acc, const int* keys, const long long* count,
                                       long long stride, float scale, int adam, float lr, float adam_scale, long long ms,
                                       const unsigned int* status) {
    long long n = *count;
    if (n > stride) n = stride;
    if (skml_failed(status)) n = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int k = keys[i];
        const float g = acc[k];
        if (g == 0.f) continue;
        acc[k] = 0.f;
        apply_update(w, m, v, k, g * scale, adam, lr, adam_scale, ms);
    }
}

extern "C" int skml_update_gathered(float* w, float* m, float* v, float* acc, const int* keys, const long long* counts,
                                    long long stride, int lists, float scale, int adam, float lr, float adam_scale,
                                    int adam_stride, const unsigned int* status, void* stream) {
    for (int l = 0; l < lists; ++l) {
        update_gathered_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(w, m, v, acc, keys + (long long)l * stride,
                                                                                 counts + l, stride, scale, adam, lr, adam_scale,
                                                                                 adam_stride > 1 ? adam_stride : 1, status);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

// Scatter-add of (key, value) lists into a dense accumulator (raw key/value all-gather
// baseline: local sum of the gathered lists).
__global__ void scatter_kv_kernel(float* acc, const int* keys, const float* vals, const long long* counts,
                                  long long stride, int lists) {
    for (int l = 0; l < lists; ++l) {
        long long n = counts[l];
        if (n > stride) n = stride;
        const int* k = keys + (long long)l * stride;
        const float* v = vals + (long long)l * stride;
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
             i += (long long)gridDim.x * blockDim.x)
            atomicAdd(acc + k[i], v[i]);
    }
}

// One launch per list: inside a list every key occurs once, so its adds touch distinct words, and
// stream order fixes the order in which the lists reach a word. Every rank therefore computes the
// same floating-point sums (a single launch over all lists would let blocks run ahead into later
// lists, and three or more addends in varying order round differently).
extern "C" int skml_scatter_kv(float* acc, const int* keys, const float* vals, const long long* counts,
                               long long stride, int lists, void* stream) {
    for (int l = 0; l < lists; ++l) {
        scatter_kv_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(acc, keys + (long long)l * stride,
                                                                            vals + (long long)l * stride, counts + l, stride, 1);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Synthetic data generation on the device.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double u01(uint64_t h) { return (double)(h >> 11) * (1.0 / 9007199254740992.0); }

__device__ __forceinline__ float normal_from(uint64_t h1, uint64_t h2) {
    double a = u01(h1), b = u01(h2);
    if (a < 1e-300) a = 1e-300;
    return (float)(sqrt(-2.0 * log(a)) * cospi(2.0 * b));
}

__global__ void gen_wstar_kernel(float* w, long long dim, double density, uint64_t seed) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (long long)gridDim.x * blockDim.x) {
        bool on = density >= 1.0 || u01(skml_rand(seed, 0xA1u, (uint64_t)i, 0)) < density;
        w[i] = on ? normal_from(skml_rand(seed, 0xA2u, (uint64_t)i, 0), skml_rand(seed, 0xA3u, (uint64_t)i, 0)) : 0.f;
    }
}

extern "C" int skml_gen_wstar(float* w, long long dim, double density, unsigned long long seed, void* stream) {
    gen_wstar_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(w, dim, density, seed);
    return (int)cudaGetLastError();
}

// 0-based Zipf(s) rank from a uniform draw: the density x^-s on [1, dim+1) inverted in
// closed form (s == 0: uniform).
__device__ __forceinline__ int zipf_rank(double u, int dim, double s, double top_pow, double inv_a, double log_top) {
    double x;
    if (s == 0.0) x = 1.0 + u * dim;
    else if (inv_a == 0.0) x = exp(u * log_top);
    else x = pow(1.0 + u * (top_pow - 1.0), inv_a);
    long long r = (long long)x - 1;
    if (r < 0) r = 0;
    if (r >= dim) r = dim - 1;
    return (int)r;
}

#define GEN_WARPS 8
#define GEN_MAX_K 256
// One warp per row. Candidates are drawn in rounds of 32; a candidate is kept if it is
// new to the row (compared with the kept list and with lower lanes of the round).
__global__ void __launch_bounds__(GEN_WARPS * 32)
gen_rows_kernel(int* __restrict__ cols, float* __restrict__ vals, float* __restrict__ labels, long long row_offset,
                long long rows, int dim, int k, double s, int value_kind, int task, float noise,
                const float* __restrict__ wstar, uint64_t seed) {
    __shared__ int s_cols[GEN_WARPS][GEN_MAX_K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double a = 1.0 - s;
    const bool is_one = fabs(a) < 1e-9;
    const double inv_a = is_one ? 0.0 : 1.0 / a;
    const double top_pow = is_one ? 0.0 : pow((double)dim + 1.0, a);
    const double log_top = log((double)dim + 1.0);
    for (long long r = (long long)blockIdx.x * GEN_WARPS + warp; r < rows; r += (long long)gridDim.x * GEN_WARPS) {
        const uint64_t gid = (uint64_t)(row_offset + r);
        int have = 0;
        unsigned int round = 0;
        while (have < k && round < 4096) {
            uint64_t h = skml_rand(seed, gid, (uint64_t)round * 32 + lane, 0xC0u);
            int c = zipf_rank(u01(h), dim, s, top_pow, inv_a, log_top);
            bool fresh = true;
            for (int j = 0; j < have; ++j)
                if (s_cols[warp][j] == c) fresh = false;
            unsigned int same = __match_any_sync(0xFFFFFFFFu, c);
            if ((same & ((1u << lane) - 1u)) != 0) fresh = false;  // a lower lane drew the same column
            unsigned int m = __ballot_sync(0xFFFFFFFFu, fresh);
            int pos = have + __popc(m & ((1u << lane) - 1u));
            if (fresh && pos < k) s_cols[warp][pos] = c;
            have += __popc(m);
            if (have > k) have = k;
            ++round;
            __syncwarp();
        }
        // values, margin, label
        float sq = 0.f;
        for (int j = lane; j < k; j += 32) {
            float v = 1.f;
            if (value_kind == 1) v = (float)u01(skml_rand(seed, gid, j, 0xC1u)) + 1e-12f;
            else if (value_kind == 2) v = normal_from(skml_rand(seed, gid, j, 0xC2u), skml_rand(seed, gid, j, 0xC3u));
            sq += v * v;
        }
        sq = warp_sum(sq);
        float scale = value_kind == 1 ? rsqrtf(sq) : 1.f;
        float margin = 0.f;
        for (int j = lane; j < k; j += 32) {
            float v = 1.f;
            if (value_kind == 1) v = ((float)u01(skml_rand(seed, gid, j, 0xC1u)) + 1e-12f) * scale;
            else if (value_kind == 2) v = normal_from(skml_rand(seed, gid, j, 0xC2u), skml_rand(seed, gid, j, 0xC3u));
            int c = j < have ? s_cols[warp][j] : 0;
            cols[r * k + j] = c;
            if (vals) vals[r * k + j] = v;
            margin += wstar[c] * v;
        }
        margin = warp_sum(margin);
        if (lane == 0) {
            float y;
            float nz = noise != 0.f ? noise * normal_from(skml_rand(seed, gid, 1, 0xC4u), skml_rand(seed, gid, 2, 0xC4u)) : 0.f;
            if (task == 0) {
                float p = 1.f / (1.f + __expf(-margin));
                y = u01(skml_rand(seed, gid, 0, 0xC5u)) < (double)p ? 1.f : -1.f;
            } else if (task == 1) {
                y = margin + nz >= 0.f ? 1.f : -1.f;
            } else {
                y = margin + nz;
            }
            labels[r] = y;
        }
        __syncwarp();
    }
}

extern "C" int skml_gen_rows(int* cols, float* vals, float* labels, long long row_offset, long long rows, int dim,
                             int k, double s, int value_kind, int task, float noise, const float* wstar,
                             unsigned long long seed, void* stream) {
    if (k > GEN_MAX_K || k > dim || k < 1) return -1;
    long long blocks = (rows + GEN_WARPS - 1) / GEN_WARPS;
    long long cap = (long long)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    gen_rows_kernel<<<(unsigned)blocks, GEN_WARPS * 32, 0, (cudaStream_t)stream>>>(
        cols, vals, labels, row_offset, rows, dim, k, s, value_kind, task, noise, wstar, seed);
    return (int)cudaGetLastError();
}

extern "C" int skml_sm_count() { return sm_count(); }

// ---------------------------------------------------------------------------
// Transposed-index gradient. For a shard whose minibatches are fixed row slices, the batch's
// column-major index (distinct columns, their row lists) is built once. A step then needs the
// per-row coefficients (glm_margin_kernel<2>) and, per distinct column c of the batch,
//     value[c] = sum over the batch rows r that contain c of coef[r] * x[r][c]  +  lambda * w[c],
// which is a gather of coefficients (an L2-resident array of batch-size floats) instead of a
// scatter into the dim-sized accumulator: no atomics, no touched bitmap, no compaction, and the
// keys come out sorted because the column list is. Columns are binned by their number of
// entries when the index is built: one thread, one warp or one block per column.
// (Equivalent of ml/gradient/DenseDoubleGradient.scala:51-57 + toSparse for a known sparsity
// pattern.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float colsum_range(const int* __restrict__ rowidx, const float* __restrict__ svals,
                                              const float* __restrict__ coef, int e0, int e1, int start, int stride) {
    // four entries in flight: one after the other, each is two trips to L2 (1.9M entries 18.3 -> 15.7 us, 7.5M 51 -> 48,
    // 0.15M 5.7 -> 4.4)
    float acc = 0.f;
    const unsigned int end = (unsigned int)e1;   // (steps past the end do not wrap)
    for (unsigned int e = (unsigned int)(e0 + start); e < end; e += 4u * stride) {
        int r[4];
        float x[4], c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned int at = e + (unsigned int)(u * stride);
            r[u] = at < end ? rowidx[at] : -1;
            x[u] = svals && at < end ? svals[at] : 1.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = r[u] >= 0 ? __ldg(coef + r[u]) : 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (r[u] >= 0) acc = fmaf(c[u], x[u], acc);
    }
    return acc;
}

// bins[0..n_short) thread per column, bins[n_short..n_short+n_medium) warp per column (bins hold
// positions into ucols / colptr). Long columns are cut into segments of a few thousand entries at
// build time: item j = (long_col[j], [long_e0[j], long_e1[j])), one block each, partial sums added
// atomically into `out` (which the caller zeroes for that reason).
__global__ void __launch_bounds__(256)
colsum_kernel(const int* __restrict__ colptr, const int* __restrict__ rowidx, const float* __restrict__ svals,
              const int* __restrict__ ucols, const int* __restrict__ bins, const int* __restrict__ long_col,
              const int* __restrict__ long_e0, const int* __restrict__ long_e1, int n_short, int n_medium, int n_long,
              int short_blocks, int medium_blocks, const float* __restrict__ coef, const float* __restrict__ w,
              float lambda, float* __restrict__ out, StepLoss loss) {
    skml_after_previous();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int b = blockIdx.x;
    if (b == 0 && threadIdx.x == 0) loss.settle();
    if (b < short_blocks) {
        const int t = b * 256 + threadIdx.x;
        if (t < n_short) {
            const int i = bins[t];
            const float wv = __ldg(w + ucols[i]);   // issued first: this DRAM gather overlaps the coefficient chain
            out[i] = colsum_range(rowidx, svals, coef, colptr[i], colptr[i + 1], 0, 1) + lambda * wv;
        }
        return;
    }
    b -= short_blocks;
    if (b < medium_blocks) {
        const int t = b * 8 + warp;
        if (t < n_medium) {
            const int i = bins[n_short + t];
            const float wv = lane == 0 ? __ldg(w + ucols[i]) : 0.f;
            float v = colsum_range(rowidx, svals, coef, colptr[i], colptr[i + 1], lane, 32);
            v = warp_sum(v);
            if (lane == 0) out[i] = v + lambda * wv;
        }
        return;
    }
    b -= medium_blocks;
    if (b < n_long) {
        __shared__ float s_part[8];
        const int i = long_col[b];
        const int e0 = long_e0[b];
        float v = colsum_range(rowidx, svals, coef, e0, long_e1[b], threadIdx.x, 256);
        v = warp_sum(v);
        if (lane == 0) s_part[warp] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.f;
            for (int k = 0; k < 8; ++k) t += s_part[k];
            if (e0 == colptr[i]) t += lambda * w[ucols[i]];  // the column's first segment carries the L2 term
            atomicAdd(out + i, t);
        }
    }
}

// skml_glm_coef that also zeroes out[slot[0 .. n_slots)], for the column sums that add to them.
extern "C" int skml_glm_coef_clear(const long long* rowptr, const int* cols, const float* vals, const float* labels, long long row_lo, long long row_cnt,
                   double avg_nnz, const float* w, long long dim, int loss_id, float inv_batch, double* loss_acc, float* coef_out,
                   float* out, const int* slot, int n_slots, void* stream) {
    return margin_launch<2>(rowptr, cols, vals, labels, row_lo, row_cnt, avg_nnz, w, dim, loss_id, inv_batch, loss_acc, coef_out,
                            (cudaStream_t)stream, ClearSlots{out, slot, n_slots});
}

extern "C" int skml_glm_coef(const long long* rowptr, const int* cols, const float* vals, const float* labels,
                             long long row_lo, long long row_cnt, long long nnz_padded, double avg_nnz,
                             const float* w, long long dim, int loss_id, float inv_batch, double* loss_acc, float* coef_out,
                             unsigned int* status, long long budget, void* stream) {
    (void)nnz_padded;
    (void)status;
    (void)budget;   // nothing in it waits
    return margin_launch<2>(rowptr, cols, vals, labels, row_lo, row_cnt, avg_nnz, w, dim, loss_id, inv_batch, loss_acc, coef_out,
                            (cudaStream_t)stream);
}

// Local-id batches (streamed minibatches whose column indices were replaced on the host by their
// position in the batch's sorted list of distinct columns): the weights of those columns are
// gathered once into a compact array, the gradient is scattered into a compact accumulator, and
// the sparse gradient's values are read off it in key order. The accumulators and the touched-bit
// words of the range are cleared for the next step.
__global__ void gather_compact_kernel(const float* __restrict__ w, const int* __restrict__ ucols, int n,
                                      float* __restrict__ wc) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) wc[i] = w[ucols[i]];
}

__global__ void finalize_compact_kernel(float* __restrict__ gc, const float* __restrict__ wc, float lambda, int n,
                                        float* __restrict__ vals, unsigned int* __restrict__ bitmap) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        vals[i] = gc[i] + lambda * wc[i];
        gc[i] = 0.f;
        if (bitmap && i < (n + 31) / 32) bitmap[i] = 0u;
    }
}

extern "C" int skml_gather_compact(const float* w, const int* ucols, int n, float* wc, void* stream) {
    if (n <= 0) return 0;
    gather_compact_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(w, ucols, n, wc);
    return (int)cudaGetLastError();
}

extern "C" int skml_finalize_compact(float* gc, const float* wc, float lambda, int n, float* vals, unsigned int* bitmap,
                                     void* stream) {
    if (n <= 0) return 0;
    finalize_compact_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(gc, wc, lambda, n, vals, bitmap);
    return (int)cudaGetLastError();
}

static int colsum_launch(const int* colptr, const int* rowidx, const float* svals, const int* ucols, const int* bins, const int* long_col,
                         const int* long_e0, const int* long_e1, int n_short, int n_medium, int n_long, const float* coef, const float* w,
                         float lambda, float* out, const StepLoss& loss, cudaStream_t stream) {
    const int short_blocks = (n_short + 255) / 256, medium_blocks = (n_medium + 7) / 8;
    const long long blocks = (long long)short_blocks + medium_blocks + n_long;
    if (blocks <= 0 && !loss.partials) return 0;
    skml_launch(colsum_kernel, (unsigned)(blocks > 0 ? blocks : 1), 256, 0, stream, colptr, rowidx, svals, ucols, bins, long_col, long_e0, long_e1,
                n_short, n_medium, n_long, short_blocks, medium_blocks, coef, w,
                lambda, out, loss);
    return (int)cudaGetLastError();
}

// The long columns' slots are zero already (skml_glm_coef_clear); also settles the step's loss partials.
extern "C" int skml_colsum_settle(const int* colptr, const int* rowidx, const float* svals, const int* ucols, const int* bins, const int* long_col,
                  const int* long_e0, const int* long_e1, int n_short, int n_medium, int n_long, const float* coef, const float* w,
                  float lambda, float* out, double* partials, double* tmpl, void* stream) {
    return colsum_launch(colptr, rowidx, svals, ucols, bins, long_col, long_e0, long_e1, n_short, n_medium, n_long, coef, w, lambda, out,
                         StepLoss{partials, tmpl}, (cudaStream_t)stream);
}

extern "C" int skml_colsum(const int* colptr, const int* rowidx, const float* svals, const int* ucols, const int* bins,
                           const int* long_col, const int* long_e0, const int* long_e1, int n_short, int n_medium,
                           int n_long, int n_cols, const float* coef, const float* w, float lambda, float* out,
                           void* stream) {
    const cudaError_t e = cudaMemsetAsync(out, 0, (size_t)n_cols * sizeof(float), (cudaStream_t)stream);
    if (e != cudaSuccess) return (int)e;
    return colsum_launch(colptr, rowidx, svals, ucols, bins, long_col, long_e0, long_e1, n_short, n_medium, n_long, coef, w, lambda, out,
                         StepLoss{nullptr, nullptr}, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Row-tiled form of the transposed index. The per-column gather of `coef[row]` above costs one random
// 32-byte L2 sector per batch entry. Here the batch rows are cut into tiles of `tile_rows` rows whose
// coefficients fit in shared memory (196 KB for 49,152 rows), the index is ordered by (tile, column,
// row) with 16-bit tile-local rows, and a block that owns (a share of) a tile gathers from shared
// memory. One partial sum per (tile, column) pair goes to `partial[pair_dst[p]]`, a position in
// (column, tile) order, so the second kernel adds a column's partial sums from consecutive words, in
// tile order: no atomics anywhere, the result is bit-reproducible.
// ---------------------------------------------------------------------------
constexpr int CT_SHORT = 8;   // pairs of up to this many entries are summed by one lane

template <bool HAS_VALS>
__global__ void __launch_bounds__(1024, 1)
coltile_partial_kernel(const float* __restrict__ coef, int rows, int tile_rows, const int* __restrict__ tile_pair_ptr,
                       int blocks_per_tile, const int* __restrict__ pair_ptr, const unsigned short* __restrict__ lrow,
                       const float* __restrict__ svals, const int* __restrict__ pair_dst, float* __restrict__ partial) {
    extern __shared__ __align__(16) float s_coef[];
    const int tile = blockIdx.x / blocks_per_tile, sub = blockIdx.x % blocks_per_tile;
    const int r0 = tile * tile_rows, nr = min(tile_rows, rows - r0);
    {   // the tile's coefficients (r0 is a multiple of 4 floats: 16-byte aligned rows)
        const float4* src = reinterpret_cast<const float4*>(coef + r0);
        float4* dst = reinterpret_cast<float4*>(s_coef);
        const int nv = nr / 4;
        for (int i = threadIdx.x; i < nv; i += blockDim.x) dst[i] = __ldg(src + i);
        for (int i = 4 * nv + threadIdx.x; i < nr; i += blockDim.x) s_coef[i] = __ldg(coef + r0 + i);
    }
    __syncthreads();
    // this block's share of the tile's pairs: cut by entries (pairs are not split), found by binary search
    const int p0 = tile_pair_ptr[tile], p1 = tile_pair_ptr[tile + 1];
    __shared__ int s_my[2];
    if (threadIdx.x < 2) {
        const long long e0 = pair_ptr[p0], e1 = pair_ptr[p1];
        const int which = sub + threadIdx.x;
        int pos;
        if (which == 0) pos = p0;
        else if (which >= blocks_per_tile) pos = p1;
        else {
            const long long target = e0 + (e1 - e0) * which / blocks_per_tile;
            int lo = p0, hi = p1;
            while (lo < hi) {   // first pair that starts at or after the target entry
                const int mid = (lo + hi) >> 1;
                if ((long long)pair_ptr[mid] < target) lo = mid + 1;
                else hi = mid;
            }
            pos = lo;
        }
        s_my[threadIdx.x] = pos;
    }
    __syncthreads();
    const int my0 = s_my[0], my1 = s_my[1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // the warps share the block's pairs by entries too (a warp that drew the frequent columns' pairs would
    // otherwise have many times the work of the others)
    int w0 = my0, w1 = my1;
    if (lane < 2 && my1 > my0) {
        const long long e0 = pair_ptr[my0], e1 = pair_ptr[my1];
        const int which = warp + lane;
        int pos;
        if (which == 0) pos = my0;
        else if (which >= nwarps) pos = my1;
        else {
            const long long target = e0 + (e1 - e0) * which / nwarps;
            int lo = my0, hi = my1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if ((long long)pair_ptr[mid] < target) lo = mid + 1;
                else hi = mid;
            }
            pos = lo;
        }
        if (lane == 0) w0 = pos;
        else w1 = pos;
    }
    w0 = __shfl_sync(0xFFFFFFFFu, w0, 0);
    w1 = __shfl_sync(0xFFFFFFFFu, w1, 1);
    for (int base = w0; base < w1; base += 32) {
        const int p = base + lane;
        const bool valid = p < w1;
        const int e0 = valid ? __ldg(pair_ptr + p) : 0, e1 = valid ? __ldg(pair_ptr + p + 1) : 0;
        const int len = e1 - e0;
        float acc = 0.f;
        if (valid && len <= CT_SHORT) {
            for (int e = e0; e < e1; ++e) acc = fmaf(s_coef[lrow[e]], HAS_VALS ? svals[e] : 1.f, acc);
        }
        unsigned int longs = __ballot_sync(0xFFFFFFFFu, valid && len > CT_SHORT);
        while (longs) {   // the warp sums one long pair at a time (fixed order: lane stride, shuffle tree)
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const int se0 = __shfl_sync(0xFFFFFFFFu, e0, src), se1 = __shfl_sync(0xFFFFFFFFu, e1, src);
            float part = 0.f, part2 = 0.f;   // two independent chains: the loads of a round overlap
            int e = se0 + lane;
            for (; e + 32 < se1; e += 64) {
                const unsigned short r0 = lrow[e], r1 = lrow[e + 32];
                part = fmaf(s_coef[r0], HAS_VALS ? svals[e] : 1.f, part);
                part2 = fmaf(s_coef[r1], HAS_VALS ? svals[e + 32] : 1.f, part2);
            }
            if (e < se1) part = fmaf(s_coef[lrow[e]], HAS_VALS ? svals[e] : 1.f, part);
            part = warp_sum(part + part2);
            if (lane == src) acc = part;
        }
        if (valid) partial[__ldg(pair_dst + p)] = acc;
    }
}

__global__ void __launch_bounds__(256)
colsum_combine_kernel(const int* __restrict__ col_pair_ptr, const float* __restrict__ partial, const int* __restrict__ ucols,
                      const float* __restrict__ w, float lambda, int n_cols, float* __restrict__ out) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_cols; c += gridDim.x * blockDim.x) {
        const int q0 = col_pair_ptr[c], q1 = col_pair_ptr[c + 1];
        float v = 0.f;
        for (int q = q0; q < q1; ++q) v += partial[q];   // tile order
        out[c] = v + lambda * __ldg(w + ucols[c]);
    }
}

extern "C" int skml_colsum_tiled(const int* tile_pair_ptr, const int* pair_ptr, const unsigned short* lrow, const float* svals,
                                 const int* pair_dst, const int* col_pair_ptr, const int* ucols, int rows, int tile_rows,
                                 int n_tiles, int n_cols, const float* coef, const float* w, float lambda, float* partial,
                                 float* out, void* stream_) {
    if (n_cols <= 0 || n_tiles <= 0) return 0;
    if (tile_rows <= 0 || tile_rows > 65536 || (tile_rows & 3) || (long long)n_tiles * tile_rows < rows) return (int)cudaErrorInvalidValue;
    cudaStream_t stream = (cudaStream_t)stream_;
    static bool ready = false;
    if (!ready) {
        cudaError_t e = cudaFuncSetAttribute(coltile_partial_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 * 4 - 40 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(coltile_partial_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536 * 4 - 40 * 1024);
        if (e != cudaSuccess) return (int)e;
        ready = true;
    }
    const int tr = tile_rows < rows ? tile_rows : ((rows + 3) & ~3);
    const size_t smem = (size_t)tr * sizeof(float);
    if (smem > 65536 * 4 - 40 * 1024) return (int)cudaErrorInvalidValue;
    int bpt = sm_count() / n_tiles;
    if (bpt < 1) bpt = 1;
    const unsigned grid = (unsigned)(n_tiles * bpt);
    if (svals)
        coltile_partial_kernel<true><<<grid, 1024, smem, stream>>>(coef, rows, tile_rows, tile_pair_ptr, bpt, pair_ptr, lrow, svals,
                                                                  pair_dst, partial);
    else
        coltile_partial_kernel<false><<<grid, 1024, smem, stream>>>(coef, rows, tile_rows, tile_pair_ptr, bpt, pair_ptr, lrow, svals,
                                                                   pair_dst, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    colsum_combine_kernel<<<sm_count() * 8, 256, 0, stream>>>(col_pair_ptr, partial, ucols, w, lambda, n_cols, out);
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// skml_compact_noalloc: the compaction above for callers that must not allocate.
// (Declared and documented in skml_noalloc.h; it has no counterpart in the reference.)
//
// The only scratch memory of the compaction is the array of counts. Here
// it lives in a file-scope device array instead of a caller-supplied buffer, so the call
// needs no cudaMalloc, no cudaFree and no allocating library routine.
// ---------------------------------------------------------------------------
#include <stdio.h>

#include <mutex>

#include "skml_noalloc.h"

// one count per warp and one per block of the largest shape
static __device__ __align__(256) unsigned int g_noalloc_block_counts[(COMPACT_WARPS + 1) * COMPACT_MAX_BLOCKS];

#define NOALLOC_MAX_DEVICES 64
static unsigned int* g_noalloc_scratch_ptr[NOALLOC_MAX_DEVICES];  // device address of the array, per device
static std::mutex g_noalloc_mutex;

// In host code the array's name is only a handle of the symbol, not a device address:
// the address is asked for once per device, with that device current.
static int noalloc_scratch(unsigned int** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return (int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_scratch_ptr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_block_counts);
        if (e != cudaSuccess) return (int)e;
        g_noalloc_scratch_ptr[dev] = static_cast<unsigned int*>(p);
    }
    *out = g_noalloc_scratch_ptr[dev];
    return 0;
}

extern "C" int skml_compact_noalloc(float* g, const float* w, unsigned int* bitmap, int dim, float lambda,
                                    long long* meta, int* keys, float* vals, long long capacity,
                                    unsigned int* status, void* stream_) {
    if (dim <= 0 || !g || !w || !bitmap || !meta || !keys || !vals || !status) {
        fprintf(stderr, "skml_compact_noalloc: null pointer or non-positive dim\n");
        return SKML_NOALLOC_BAD_ARGUMENT;
    }
    if ((long long)dim > SKML_NOALLOC_MAX_DIM) {
        fprintf(stderr, "skml_compact_noalloc: dim %d exceeds the built-in scratch (at most %lld coordinates); "
                        "use skml_compact with a caller-owned block_counts buffer\n", dim, (long long)SKML_NOALLOC_MAX_DIM);
        return SKML_NOALLOC_TOO_LARGE;
    }
    unsigned int* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    // every entry of the scratch that is read (one per warp and block) is rewritten by the count kernel of this
    // call, so nothing of an earlier call has to be cleared
    return compact_launch(g, w, bitmap, dim, lambda, scratch, meta, keys, vals, nullptr, capacity, status, (cudaStream_t)stream_);
}
