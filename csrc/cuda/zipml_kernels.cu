// Baseline compressor "Zip" on the device: the ZipML quantizer (split points by repeated halving of
// the candidate set, keeping split the pairs whose merge would cost the largest squared error), the
// bucket codes that travel between ranks, and the inverse (code -> bucket midpoint, scatter-add of
// several ranks' lists). Nothing here reads a value back to the host: the number of non-zeros, the
// number of halving rounds and the number of buckets all stay on the device.
//
// Behaviour follows ml/gradient/ZipGradient.scala:70-129 of the reference with the one repair the CPU
// oracle shares (the unpaired last candidate of an odd round is kept; the reference bumps the wrong
// counter and loses it): sort, prefix sums of v and v^2 in double, per round the error
//   l2 + mean^2 * m - 2 * mean * l1
// of every adjacent candidate pair, the thr-th largest error as threshold, pairs at or above it
// (the first thr of them in index order) stay split. Decode value of a bucket = midpoint of its edges.
//
// The split search is one cooperative launch. A round is a map over the candidate pairs, a selection and
// an ordered compaction, and the candidate set halves from round to round, so the search reads about two
// entries per value; what bounds it is the chain of some twenty rounds. While a round has more than
// Z_ALONE pairs they are cut into one slice per block: every block selects the keys of its slice that can
// be among the round's largest, publishes them, and after a grid barrier selects among all blocks' lists,
// which also tells it how many pairs the blocks before it keep split. The rest is block 0's alone, about
// 2 us a round. (One block for all rounds took 822 us for 330,000 values.)
// A barrier that gives up reports to the caller's status word; the tables are then those of an earlier call, so the
// kernels behind the search, and the update behind them, do nothing once the word is set.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include <cub/device/device_radix_sort.cuh>

#include "skml_api.h"
#include "skml_device.cuh"

namespace {

constexpr int ZT = 1024;           // threads of the split search
constexpr int Z_MAX_BUCKETS = 8192;     // the split and midpoint tables are staged in shared memory
constexpr int Z_KPT = 8;                // values a thread handles per tile of the prefix sums
constexpr int Z_ALONE = ZT * Z_KPT;     // pairs one block handles in shared memory: below, a barrier costs more than it saves
constexpr int Z_MAX_BLOCKS = 148;
// Candidates block 0 keeps in shared memory for the last rounds, a pair a thread: where the blocks' lists were, so that the
// block stays below the 164 KB that leave 92 KB of L1 (2048 of them in memory of their own: the search of 233,000 values 154 us
// instead of 139). With two pairs' loads in flight in the rounds before: 233,000 values 145 -> 139 us, 48,000 99 -> 92, 16,000 97 -> 90.
constexpr int Z_TAIL = 1536;

constexpr int Z_FLIGHT = 2;             // pairs of a thread whose loads are in flight together
constexpr int Z_SORT_KEYS = 8;          // values a thread of the sort keeps in registers
constexpr int Z_SORT_ALONE = 6144;      // values that one block sorts (44 KB of shared memory)

// What the blocks of the sort and of the split search share; the barrier words are cleared before the sort.
struct ZShared {
    unsigned int bar, sort_bar, pad[14];
    unsigned int digits[Z_MAX_BLOCKS][256];               // sort: values per digit in every block's slice
    double sum_v[Z_MAX_BLOCKS], sum_v2[Z_MAX_BLOCKS];     // sums over the blocks' slices of values
    unsigned long long cand[Z_ALONE];                     // blocks x kept pairs of a round at most
};

struct ZScratch {
    float* sorted_in;        // values padded with +inf, or the sort's second buffer
    float* sorted;           // ascending
    double2* rt;             // prefix sums of v and of v^2
    int* idx_a;              // candidate split positions (double buffered)
    int* idx_b;
    unsigned long long* err; // order-preserving keys of the pair errors
    ZShared* shared;
    void* cub_temp;
    size_t cub_bytes;
};

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

size_t cub_temp_bytes(long long n_max) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, bytes, (const float*)nullptr, (float*)nullptr, (int)n_max);
    return bytes;
}

size_t carve(unsigned char* base, long long n_max, ZScratch* z) {
    size_t o = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base ? base + o : nullptr;
        o += al256(bytes);
        return p;
    };
    const size_t n = (size_t)n_max;
    float* a = reinterpret_cast<float*>(take(4 * n));
    float* b = reinterpret_cast<float*>(take(4 * n));
    double2* rt = reinterpret_cast<double2*>(take(16 * n));
    int* ia = reinterpret_cast<int*>(take(4 * n));
    int* ib = reinterpret_cast<int*>(take(4 * n));
    unsigned long long* e = reinterpret_cast<unsigned long long*>(take(8 * (n / 2 + 1)));
    ZShared* sh = reinterpret_cast<ZShared*>(take(sizeof(ZShared)));
    const size_t cb = cub_temp_bytes(n_max);
    void* ct = take(cb);
    if (z) *z = ZScratch{a, b, rt, ia, ib, e, sh, ct, cb};
    return o;
}

__global__ void zip_pad_kernel(const float* __restrict__ vals, const long long* __restrict__ n_ptr, long long n_max,
                               float* __restrict__ out) {
    long long n = *n_ptr;
    if (n > n_max) n = n_max;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_max; i += (long long)gridDim.x * blockDim.x)
        out[i] = i < n ? vals[i] : __int_as_float(0x7F800000);
}

// Ascending order of the values: least significant digit first, eight bits a pass, all four passes in one cooperative
// launch. A warp owns consecutive values and ranks 32 of them at a time among those of their digit; a block publishes its
// slice's digit counts, and behind a grid barrier every block adds up those it needs. Bound by the seven barriers and the
// trips to L2 between them. 330,000 values: 43 us; cub's sort, six kernels and six fills with the gaps between them, took 88.
// ALONE: one block, whose values stay in shared memory between the passes: a pack of 3,000 values 66 us instead of 72, of 4,097
// (two blocks otherwise) 72 instead of 85; with cub's sort 64 and 68, of 6,000 87 instead of 97 and 118.
template <bool ALONE>
__global__ void __launch_bounds__(ZT, 1)
zip_sort_kernel(const float* __restrict__ vals, const long long* __restrict__ n_ptr, long long n_max, unsigned int* buf_a, unsigned int* buf_b,
                ZShared* __restrict__ shared, unsigned int* status) {
    skml_after_previous();
    using Count = typename std::conditional<ALONE, unsigned short, unsigned int>::type;
    __shared__ Count s_cnt[ZT / 32][256];
    __shared__ unsigned int s_tot[ALONE ? 1 : 4][256], s_bef[ALONE ? 1 : 4][256], s_base[256], s_warp[8], s_buf[ALONE ? Z_SORT_ALONE : 1];
    const unsigned int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x, b = blockIdx.x;
    long long n64 = *n_ptr;
    if (n64 > n_max) n64 = n_max;
    const unsigned int n = (unsigned int)n64;
    const unsigned int per = ((n + nb - 1) / nb + ZT - 1) / ZT * ZT, wper = per / 32;   // at most Z_SORT_KEYS values a thread
    const unsigned int lo = min(n, b * per + warp * wper), hi = min(n, lo + wper);
    unsigned int passed = 0;
    for (int pass = 0; pass < 4; ++pass) {
        const unsigned int* const src = pass == 2 ? buf_b : buf_a;
        unsigned int* const dst = pass == 0 || pass == 2 ? buf_a : buf_b;
        const int shift = 8 * pass;
        unsigned int x[Z_SORT_KEYS], same[Z_SORT_KEYS];
#pragma unroll
        for (int e = 0; e < Z_SORT_KEYS; ++e) {
            const unsigned int i = lo + 32 * e + lane;
            x[e] = 0;
            if (i < hi) x[e] = pass ? (ALONE ? s_buf[i] : __ldcg(src + i)) : f2ord(vals[i]);
        }
        for (unsigned int d = lane; d < 256; d += 32) s_cnt[warp][d] = 0;
        __syncwarp();
#pragma unroll
        for (int e = 0; e < Z_SORT_KEYS; ++e) {
            if (lo + 32 * e >= hi) break;   // (the whole warp)
            const bool in = lo + 32 * e + lane < hi;
            const unsigned int d = (x[e] >> shift) & 255u;
            same[e] = __ballot_sync(0xFFFFFFFFu, in);   // lanes with this lane's digit (a ballot per bit: faster than a match of the warp)
#pragma unroll
            for (int k = 0; k < 8; ++k) same[e] &= __ballot_sync(0xFFFFFFFFu, (d >> k) & 1u) ^ ((d >> k & 1u) - 1u);
            if (in && (int)lane == __ffs(same[e]) - 1) s_cnt[warp][d] += (Count)__popc(same[e]);
            __syncwarp();
        }
        __syncthreads();
        unsigned int run = 0;
        if (tid < 256) {   // what the warps before it hold, and the slice's counts
#pragma unroll 8
            for (int w = 0; w < ZT / 32; ++w) {
                const unsigned int c = s_cnt[w][tid];
                s_cnt[w][tid] = (Count)run;
                run += c;
            }
            if (!ALONE) shared->digits[b][tid] = run;
        }
        if (!ALONE) {
            if (!skml_grid_barrier(&shared->sort_bar, nb, status, 2000000000ll, 0x64u, passed)) return;
            const unsigned int d = tid & 255, part = tid >> 8;
            unsigned int tot = 0, bef = 0;
#pragma unroll 8
            for (unsigned int q = part; q < nb; q += 4) {
                const unsigned int c = __ldcg(&shared->digits[q][d]);
                tot += c;
                if (q < b) bef += c;
            }
            s_tot[part][d] = tot;
            s_bef[part][d] = bef;
            __syncthreads();
        }
        unsigned int tot = 0, inc = 0;
        if (tid < 256) {
            tot = ALONE ? run : s_tot[0][tid] + s_tot[ALONE ? 0 : 1][tid] + s_tot[ALONE ? 0 : 2][tid] + s_tot[ALONE ? 0 : 3][tid];
            inc = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if ((int)lane >= o) inc += v;
            }
            if (lane == 31) s_warp[warp] = inc;
        }
        __syncthreads();
        if (tid < 256) {
            unsigned int before = inc - tot;
            if (!ALONE)
                for (int part = 0; part < 4; ++part) before += s_bef[ALONE ? 0 : part][tid];
            for (unsigned int w = 0; w < warp; ++w) before += s_warp[w];
            s_base[tid] = before;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < Z_SORT_KEYS; ++e) {
            if (lo + 32 * e >= hi) break;
            const bool in = lo + 32 * e + lane < hi;
            const unsigned int d = (x[e] >> shift) & 255u;
            if (in) {
                const unsigned int at = s_base[d] + s_cnt[warp][d] + (unsigned int)__popc(same[e] & ((1u << lane) - 1u));
                if (ALONE && pass < 3) s_buf[at] = x[e];   // (everyone has read its values of this pass)
                else dst[at] = pass < 3 ? x[e] : __float_as_uint(ord2f(x[e]));
            }
            __syncwarp();
            if (in && (int)lane == __ffs(same[e]) - 1) s_cnt[warp][d] += (Count)__popc(same[e]);
            __syncwarp();
        }
        if (pass == 3) return;
        if (ALONE) __syncthreads();
        else if (!skml_grid_barrier(&shared->sort_bar, nb, status, 2000000000ll, 0x65u, passed)) return;
    }
}

// order-preserving map of a double onto an unsigned 64-bit key
__device__ __forceinline__ unsigned long long zkey(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// block-wide exclusive scan of one unsigned value per thread; returns the exclusive prefix, `total` to all
__device__ __forceinline__ unsigned int zscan(unsigned int v, unsigned int* sh_warp, unsigned int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    __syncthreads();  // the previous call's readers are done
    if (lane == 31) sh_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned int w = sh_warp[lane], winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int x = __shfl_up_sync(0xFFFFFFFFu, winc, o);
            if (lane >= o) winc += x;
        }
        sh_warp[lane] = winc - w;
        if (lane == 31) sh_warp[32] = winc;
    }
    __syncthreads();
    total = sh_warp[32];
    return sh_warp[warp] + inc - v;
}

// block-wide exclusive scans of two doubles per thread (pairwise adds in a fixed order)
__device__ __forceinline__ void zscan_double2(double& va, double& vb, double2* sh_warp, double& total_a, double& total_b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double a = va, b = vb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xFFFFFFFFu, a, o), y = __shfl_up_sync(0xFFFFFFFFu, b, o);
        if (lane >= o) {
            a = __dadd_rn(x, a);
            b = __dadd_rn(y, b);
        }
    }
    __syncthreads();  // the previous call's readers are done
    if (lane == 31) sh_warp[warp] = make_double2(a, b);
    __syncthreads();
    if (warp == 0) {
        double wa = sh_warp[lane].x, wb = sh_warp[lane].y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double x = __shfl_up_sync(0xFFFFFFFFu, wa, o), y = __shfl_up_sync(0xFFFFFFFFu, wb, o);
            if (lane >= o) {
                wa = __dadd_rn(x, wa);
                wb = __dadd_rn(y, wb);
            }
        }
        sh_warp[lane] = make_double2(wa, wb);
    }
    __syncthreads();
    total_a = sh_warp[31].x;
    total_b = sh_warp[31].y;
    double ea = __shfl_up_sync(0xFFFFFFFFu, a, 1), eb = __shfl_up_sync(0xFFFFFFFFu, b, 1);
    if (lane == 0) ea = eb = 0.0;
    if (warp) {
        ea = __dadd_rn(sh_warp[warp - 1].x, ea);
        eb = __dadd_rn(sh_warp[warp - 1].y, eb);
    }
    va = ea;
    vb = eb;
}

// Squared error of merging the values between two prefix sums apart, as a sortable key.
__device__ __forceinline__ unsigned long long merge_error(double l1, double l2, double cnt) {
    const double mean = __ddiv_rn(l1, cnt);
    return zkey(__dadd_rn(__dadd_rn(l2, __dmul_rn(__dmul_rn(mean, mean), cnt)), -__dmul_rn(__dmul_rn(2.0, mean), l1)));
}

// Squared errors of merging the candidate pairs p0 .. p0 + count (pair i: the values from its first candidate up to the
// next pair's), by the whole block. A pair ends where the next one begins, so a lane fetches the sums in front of its own
// pair, one random sector, and takes those behind it from the lane above. (Four sectors a pair: 158 instead of 146 us for
// the search at 330,000 values.)
__device__ __forceinline__ void pair_errors(const ZScratch& z, const int* idx, unsigned int p0, unsigned int count, unsigned int split_num,
                                            unsigned int n, unsigned long long* key) {
    const unsigned int lane = threadIdx.x & 31;
    struct Front {
        int at;
        double2 sum;
    };
    auto place = [&](unsigned int pair) { return 2 * pair >= split_num ? (int)n : __ldcg(idx + 2 * pair); };   // where a pair begins
    auto sum_to = [&](int at) { return at ? z.rt[at - 1] : make_double2(0.0, 0.0); };                          // the sums up to there
    // Z_FLIGHT pairs of a thread at a time: a pair is two trips to L2, one behind the other (one block alone, 7,400 pairs: 10 us
    // with one in flight)
    for (unsigned int i0 = 0; i0 < count; i0 += Z_FLIGHT * ZT) {
        Front lo[Z_FLIGHT], hi[Z_FLIGHT];
#pragma unroll
        for (int u = 0; u < Z_FLIGHT; ++u) {
            const unsigned int i = i0 + u * ZT + threadIdx.x;
            lo[u].at = i < count ? place(p0 + i) : 0;
            hi[u].at = i < count && (lane == 31 || i + 1 >= count) ? place(p0 + i + 1) : 0;
        }
#pragma unroll
        for (int u = 0; u < Z_FLIGHT; ++u) {
            lo[u].sum = sum_to(lo[u].at);
            hi[u].sum = sum_to(hi[u].at);
        }
#pragma unroll
        for (int u = 0; u < Z_FLIGHT; ++u) {
            const unsigned int i = i0 + u * ZT + threadIdx.x;
            const bool last = lane == 31 || i + 1 >= count;
            Front up;
            up.at = __shfl_down_sync(0xFFFFFFFFu, lo[u].at, 1);
            up.sum.x = __shfl_down_sync(0xFFFFFFFFu, lo[u].sum.x, 1);
            up.sum.y = __shfl_down_sync(0xFFFFFFFFu, lo[u].sum.y, 1);
            if (last) up = hi[u];
            if (i < count) {
                const double l1 = __dadd_rn(up.sum.x, lo[u].at ? -lo[u].sum.x : 0.0), l2 = __dadd_rn(up.sum.y, lo[u].at ? -lo[u].sum.y : 0.0);
                key[i] = merge_error(l1, l2, (double)(up.at - lo[u].at));
            }
        }
    }
}

struct ZSmem {
    unsigned long long key[Z_ALONE];   // errors of the block's slice of a round, where they fit
    unsigned int hist[ZT];             // select_largest
    unsigned int warp[33];
    double2 dwarp[32];
    unsigned int digit, above, ncand, fill;
    // the last rounds (at most Z_TAIL candidates, of one block): their positions and the prefix sums in front of them
    struct Tail {
        int pos[Z_TAIL];
        double sum_v[Z_TAIL], sum_v2[Z_TAIL];
    };
    union {
        unsigned long long all[Z_ALONE];   // the lists of all blocks
        Tail tail[2];                      // a round reads one and writes the other
    };
};
static_assert(Z_TAIL <= 2 * ZT && sizeof(ZSmem) <= 162 * 1024, "a pair a thread; the 164 KB carve-out");

// Threshold for the k largest of keys[0, count), in shared memory or global (0 = no key, k keys at least): the k-th
// largest, or a value that exactly k keys reach (`exact`). Radix select, ten bits a pass from the top: a
// shared-memory count per digit, one digit per thread. Two or three passes settle real errors, because it
// stops as soon as the keys down to a digit's are k. A function of its own: the kernel runs its stages a few
// times per round, and with everything inlined it spent more time fetching instructions than executing.
// (Counting against several thresholds per step without a histogram cost 5,000 to 15,000 cycles a selection.)
__device__ __noinline__ unsigned long long select_largest(ZSmem& sm, const unsigned long long* keys, unsigned int count, unsigned int k,
                                                          bool& exact) {
    const unsigned int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long prefix = 0;   // the digits settled so far
    exact = false;
    for (int shift = 54;; shift = max(0, shift - 10)) {
        const int bits = shift == 54 ? 10 : min(10, 54 - shift - ((54 - shift - 1) / 10) * 10);
        const int top = shift + bits;   // bits from here up are the prefix's
        sm.hist[tid] = 0;
        __syncthreads();
        for (unsigned int i = tid; i < count; i += ZT) {
            const unsigned long long key = keys[i];
            if (key && (top == 64 || (key >> top) == (prefix >> top))) atomicAdd(&sm.hist[(unsigned int)(key >> shift) & ((1u << bits) - 1u)], 1u);
        }
        __syncthreads();
        // thread t looks at digit 1023 - t: keys in the digits above it
        const unsigned int mine = sm.hist[ZT - 1 - tid];
        unsigned int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if ((int)lane >= o) inc += x;
        }
        if (lane == 31) sm.warp[warp] = inc;
        __syncthreads();
        const unsigned int w = sm.warp[lane];
        const unsigned int above = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u) + inc - mine;
        if (above < k && k <= above + mine) {   // one thread: the k-th largest has this digit
            sm.digit = ZT - 1 - tid;
            sm.above = above;
            sm.ncand = mine;
        }
        __syncthreads();
        prefix |= (unsigned long long)sm.digit << shift;
        k -= sm.above;
        exact = sm.ncand == k;
        if (exact || shift == 0) return prefix;
    }
}

// The last rounds: at most Z_TAIL candidates in shared memory, a pair per thread; the
// selection is the block's. Every thread keeps count of the set.
__device__ void tail_rounds(ZSmem& sm, int bin_num, double end_v, double end_v2, int n, unsigned int& split_num, unsigned int& rounds,
                            unsigned int& which) {
    const unsigned int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    while (split_num > (unsigned int)bin_num) {
        const ZSmem::Tail& in = sm.tail[which];
        ZSmem::Tail& out = sm.tail[which ^ 1];
        const unsigned int pairs = split_num / 2, odd = split_num & 1u;
        int want = bin_num / 2 - (int)odd;
        if (want < 1) want = 1;
        const unsigned int thr_num = min((unsigned int)want, pairs);
        unsigned long long key = 0;
        if (i < pairs) {
            const bool last = 2 * i + 2 >= split_num;
            const double hv = last ? end_v : in.sum_v[2 * i + 2], hv2 = last ? end_v2 : in.sum_v2[2 * i + 2];
            const int hp = last ? n : in.pos[2 * i + 2];
            key = merge_error(__dadd_rn(hv, -in.sum_v[2 * i]), __dadd_rn(hv2, -in.sum_v2[2 * i]), (double)(hp - in.pos[2 * i]));
            sm.key[i] = key;
        }
        __syncthreads();
        bool exact;
        const unsigned long long thr = thr_num < pairs ? select_largest(sm, sm.key, pairs, thr_num, exact) : 1ull;
        const unsigned int flags = __ballot_sync(0xFFFFFFFFu, key >= thr);
        if (lane == 0) sm.warp[warp] = (unsigned int)__popc(flags);
        __syncthreads();
        const unsigned int c = sm.warp[lane];
        const unsigned int all = __reduce_add_sync(0xFFFFFFFFu, c);
        const unsigned int at = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? c : 0u) + (unsigned int)__popc(flags & ((1u << lane) - 1u));
        const unsigned int m = pairs + min(all, thr_num) + odd;
        if (m >= split_num) break;   // no progress: stop with the current set
        // candidate slots of the next set, thread by thread: first candidates, second ones that stay, an odd last one
        const unsigned int to = i < pairs ? i + min(at, thr_num) : m - 1;
        const int copies = i < pairs ? (key >= thr && at < thr_num ? 2 : 1) : (odd && i == pairs ? 1 : 0);
        for (int q = 0; q < copies; ++q) {
            out.pos[to + q] = in.pos[2 * i + q];
            out.sum_v[to + q] = in.sum_v[2 * i + q];
            out.sum_v2[to + q] = in.sum_v2[2 * i + q];
        }
        __syncthreads();
        split_num = m;
        which ^= 1;
        ++rounds;
    }
}

// meta_out: [0] buckets, [1] zero bucket, [2] halving rounds run; range_out: min, max of the values.
__global__ void __launch_bounds__(ZT, 1)
zip_splits_kernel(ZScratch z, const long long* __restrict__ n_ptr, long long n_max, int bin_num,
                  float* __restrict__ splits_out, float* __restrict__ mids_out, int* __restrict__ meta_out,
                  float* __restrict__ range_out, unsigned int* status) {
    skml_after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ZSmem& sm = *reinterpret_cast<ZSmem*>(smem_raw);
    unsigned int* const sh_warp = sm.warp;
    ZShared& g = *z.shared;
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned int nb = gridDim.x, b = blockIdx.x;
    unsigned int passed = 0;
    auto barrier = [&](unsigned int stage) { return skml_grid_barrier(&g.bar, nb, status, 2000000000ll, stage, passed); };
    long long n64 = *n_ptr;
    if (n64 > n_max) n64 = n_max;
    const unsigned int n = (unsigned int)n64;
    if (n == 0) {
        if (tid == 0 && b == 0) {
            meta_out[0] = 0;
            meta_out[1] = 0;
            meta_out[2] = 0;
        }
        return;
    }
    const float* s = z.sorted;
    // prefix sums of v and v^2: a slice of the values per block, tiles of Z_KPT values per thread carried from
    // tile to tile; every addition in a fixed order. A slice of one tile stays in registers while the blocks
    // exchange their sums, a longer one is added up first.
    {
        const unsigned int per = (n + nb - 1) / nb, lo = min(n, per * b), hi = min(n, lo + per);
        const bool one_tile = per <= (unsigned int)Z_ALONE;
        double carry_a = 0.0, carry_b = 0.0, ta = 0.0, tb = 0.0;
        if (nb > 1 && !one_tile) {
            double a = 0.0, q = 0.0;
            for (unsigned int i = lo + tid; i < hi; i += ZT) {
                const double v = (double)s[i];
                a = __dadd_rn(a, v);
                q = __dadd_rn(q, __dmul_rn(v, v));
            }
            zscan_double2(a, q, sm.dwarp, ta, tb);
        }
        for (unsigned int base = lo; base < hi || base == lo; base += Z_ALONE) {
            const unsigned int i0 = base + Z_KPT * tid;
            float v[Z_KPT];
            double a = 0.0, q = 0.0;
#pragma unroll
            for (int j = 0; j < Z_KPT; ++j) {
                v[j] = i0 + j < hi ? s[i0 + j] : 0.f;
                a = __dadd_rn(a, (double)v[j]);
                q = __dadd_rn(q, __dmul_rn((double)v[j], (double)v[j]));
            }
            double tile_a, tile_b;
            zscan_double2(a, q, sm.dwarp, tile_a, tile_b);
            if (base == lo && nb > 1) {
                if (tid == 0) {
                    g.sum_v[b] = one_tile ? tile_a : ta;
                    g.sum_v2[b] = one_tile ? tile_b : tb;
                }
                if (!barrier(0x60u)) return;
                for (unsigned int k = lane; k < b; k += 32) {
                    carry_a = __dadd_rn(carry_a, __ldcg(&g.sum_v[k]));
                    carry_b = __dadd_rn(carry_b, __ldcg(&g.sum_v2[k]));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    carry_a = __dadd_rn(carry_a, __shfl_xor_sync(0xFFFFFFFFu, carry_a, o));
                    carry_b = __dadd_rn(carry_b, __shfl_xor_sync(0xFFFFFFFFu, carry_b, o));
                }
            }
            a = __dadd_rn(carry_a, a);
            q = __dadd_rn(carry_b, q);
#pragma unroll
            for (int j = 0; j < Z_KPT; ++j) {
                a = __dadd_rn(a, (double)v[j]);
                q = __dadd_rn(q, __dmul_rn((double)v[j], (double)v[j]));
                if (i0 + j < hi) {
                    z.rt[i0 + j] = make_double2(a, q);
                    z.idx_a[i0 + j] = (int)(i0 + j);
                }
            }
            carry_a = __dadd_rn(carry_a, tile_a);
            carry_b = __dadd_rn(carry_b, tile_b);
        }
        if (nb > 1 && !barrier(0x61u)) return;
    }
    __syncthreads();
    int* idx = z.idx_a;
    int* nxt = z.idx_b;
    unsigned int split_num = n, rounds = 0;
    while (split_num > (unsigned int)bin_num) {
        const unsigned int pairs = split_num / 2, odd = split_num & 1u;
        const bool alone = nb == 1 || pairs <= Z_ALONE;
        if (alone && b != 0) return;   // block 0 goes on by itself
        if (split_num <= (unsigned int)Z_TAIL) break;   // and its first warp finishes
        int want = bin_num / 2 - (int)odd;
        if (want < 1) want = 1;
        const unsigned int thr_num = min((unsigned int)want, pairs);
        // this block's pairs; their errors stay in shared memory where they fit
        const unsigned int per = alone ? pairs : (pairs + nb - 1) / nb;
        const unsigned int p0 = alone ? 0u : min(pairs, per * b), p1 = alone ? pairs : min(pairs, p0 + per), mine = p1 - p0;
        unsigned long long* const key = per <= (unsigned int)Z_ALONE ? sm.key : z.err + p0;
        pair_errors(z, idx, p0, mine, split_num, n, key);
        __syncthreads();
        // keys of the slice at or above `thr` stay split (the first thr_num of the round's, in index order)
        unsigned long long thr = 1;
        bool exact = thr_num >= mine;   // no more than thr_num keys of the slice reach thr
        if (!exact) thr = select_largest(sm, key, mine, thr_num, exact);
        unsigned int before = 0;   // pairs at or above the round's threshold in the blocks before this one
        if (!alone) {
            // publish the slice's largest keys (at most thr_num: with more equal ones than that it does not
            // matter which), then select among everybody's
            if (tid == 0) sm.fill = 0;
            __syncthreads();
            for (int pass = exact ? 1 : 0; pass < 2; ++pass) {   // first those above thr, then those equal to it
                const unsigned long long lo = pass ? thr : thr + 1, hi = pass && !exact ? thr : ~0ull;
                for (unsigned int i = tid; i < mine; i += ZT) {
                    const unsigned long long k = key[i];
                    if (k >= lo && k <= hi) {
                        const unsigned int at = atomicAdd(&sm.fill, 1u);
                        if (at < thr_num) g.cand[b * thr_num + at] = k;
                    }
                }
                __syncthreads();
            }
            // slots without a key hold none (a block with fewer pairs than thr_num)
            for (unsigned int at = min(sm.fill, thr_num) + tid; at < thr_num; at += ZT) g.cand[b * thr_num + at] = 0ull;
            if (!barrier(0x62u)) return;
            for (unsigned int q = tid; q < nb * thr_num; q += ZT) sm.all[q] = __ldcg(&g.cand[q]);   // blocks x thr_num <= Z_ALONE
            __syncthreads();
            thr = select_largest(sm, sm.all, nb * thr_num, thr_num, exact);
            unsigned int cnt = 0;
            for (unsigned int q = tid; q < b * thr_num; q += ZT) cnt += sm.all[q] >= thr ? 1u : 0u;
            zscan(cnt, sh_warp, before);
        }
        // ordered compaction, a tile of ZT pairs at a time: the first thr_num pairs at or above the threshold keep
        // their second candidate
        unsigned int flagged = before;
        for (unsigned int base = 0; base < mine; base += ZT) {
            const unsigned int i = p0 + base + tid;
            const bool in = base + tid < mine;
            const int first = in ? __ldcg(idx + 2 * i) : 0, second = in ? __ldcg(idx + 2 * i + 1) : 0;   // on their way during the scan
            const bool f = in && key[base + tid] >= thr;
            unsigned int tile_total;
            const unsigned int at = flagged + zscan(f ? 1u : 0u, sh_warp, tile_total);
            if (in) {
                const unsigned int pos = i + min(at, thr_num);
                nxt[pos] = first;
                if (f && at < thr_num) nxt[pos + 1] = second;
            }
            flagged += tile_total;
        }
        // all blocks together keep thr_num second candidates: at least that many keys reach the threshold
        const unsigned int kept_total = alone ? min(flagged, thr_num) : thr_num;
        const unsigned int m = pairs + kept_total + odd;
        if (m >= split_num) break;  // no progress: stop with the current set (uniform for the block; never while several work)
        if (odd && tid == 0 && b == 0) nxt[pairs + kept_total] = __ldcg(idx + split_num - 1);
        if (alone) __syncthreads();
        else if (!barrier(0x63u)) return;
        int* sw = idx;
        idx = nxt;
        nxt = sw;
        split_num = m;
        ++rounds;
    }
    if (b != 0) return;
    if (split_num > (unsigned int)bin_num && split_num <= (unsigned int)Z_TAIL) {
        for (unsigned int i = tid; i < split_num; i += ZT) {
            const int at = __ldcg(idx + i);
            sm.tail[0].pos[i] = at;
            const double2 sum = at ? z.rt[at - 1] : make_double2(0.0, 0.0);
            sm.tail[0].sum_v[i] = sum.x;
            sm.tail[0].sum_v2[i] = sum.y;
        }
        __syncthreads();
        unsigned int which = 0;
        tail_rounds(sm, bin_num, z.rt[n - 1].x, z.rt[n - 1].y, (int)n, split_num, rounds, which);
        for (unsigned int i = tid; i < split_num; i += ZT) idx[i] = sm.tail[which].pos[i];
    }
    __syncthreads();
    // split values (duplicates dropped), bucket midpoints, zero bucket
    const float vmin = s[0], vmax = s[n - 1];
    const unsigned int raw = split_num > 1 ? split_num - 1 : 1u;
    // a round that cannot shrink the set any further stops the search one or two candidates early
    // (only with very few buckets): the tables hold bin_num + 2 entries for that case
    const unsigned int cap = min(raw, (unsigned int)bin_num + 1u);
    unsigned int total_distinct = 0;
    for (unsigned int base = 0; base < cap; base += ZT) {
        const unsigned int i = base + tid;
        float v = 0.f;
        bool fresh = false;
        if (i < cap) {
            v = split_num > 1 ? s[idx[i + 1]] : s[0];
            fresh = i == 0 || v != s[idx[i]];
        }
        unsigned int tile_total;
        const unsigned int pos = total_distinct + zscan(fresh ? 1u : 0u, sh_warp, tile_total);
        if (fresh) splits_out[pos] = v;
        total_distinct += tile_total;
    }
    __syncthreads();
    const unsigned int buckets = total_distinct + 1u;
    for (unsigned int i = tid; i < buckets; i += ZT) {
        const double left = i == 0 ? (double)vmin : (double)splits_out[i - 1];
        const double right = i + 1 == buckets ? (double)vmax : (double)splits_out[i];
        mids_out[i] = (float)(0.5 * (left + right));
    }
    int negs = 0;   // the splits ascend: the zero bucket is the number of negative ones
    for (unsigned int base = 0; base + 1 < buckets; base += ZT) {
        const unsigned int i = base + tid;
        negs += __syncthreads_count(i + 1 < buckets && splits_out[i] < 0.f);
    }
    if (tid == 0) {
        meta_out[0] = (int)buckets;
        meta_out[1] = vmin > 0.f ? 0 : (vmax < 0.f ? (int)buckets - 1 : negs);
        meta_out[2] = (int)rounds;
        range_out[0] = vmin;
        range_out[1] = vmax;
    }
}

// bucket of every value = number of splits <= value; one or two bytes per code
__global__ void __launch_bounds__(256)
zip_code_kernel(const float* __restrict__ vals, const long long* __restrict__ n_ptr, long long n_max,
                const float* __restrict__ splits, const int* __restrict__ meta, int code_bytes,
                unsigned char* __restrict__ codes, const unsigned int* __restrict__ status) {
    skml_after_previous();
    extern __shared__ float sh_splits[];
    long long n = *n_ptr;
    if (n > n_max) n = n_max;
    if (skml_failed(status)) n = 0;   // (read beside the counts)
    const int nb = meta[0], ns = nb > 0 ? nb - 1 : 0;
    for (int i = threadIdx.x; i < ns; i += blockDim.x) sh_splits[i] = splits[i];
    __syncthreads();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = vals[i];
        int lo = 0, hi = ns;  // first split > v
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sh_splits[mid] <= v) lo = mid + 1;
            else hi = mid;
        }
        if (code_bytes == 1) codes[i] = (unsigned char)lo;
        else reinterpret_cast<unsigned short*>(codes)[i] = (unsigned short)lo;
    }
}

__global__ void __launch_bounds__(256)
zip_unpack_scatter_kernel(float* __restrict__ acc, const int* __restrict__ keys, const unsigned char* __restrict__ codes,
                          const float* __restrict__ mids, const long long* __restrict__ count, long long key_stride,
                          int code_bytes, int table_len, float* __restrict__ vals_out, const unsigned int* __restrict__ status) {
    skml_after_previous();
    extern __shared__ float sh_mids[];
    long long n = *count;
    if (n > key_stride) n = key_stride;
    if (skml_failed(status)) n = 0;
    for (int i = threadIdx.x; i < table_len; i += blockDim.x) sh_mids[i] = mids[i];
    __syncthreads();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        unsigned int c = code_bytes == 1 ? codes[i] : reinterpret_cast<const unsigned short*>(codes)[i];
        if (c >= (unsigned int)table_len) c = table_len - 1;
        const float f = sh_mids[c];
        if (vals_out) vals_out[i] = f;
        if (acc) atomicAdd(acc + keys[i], f);
    }
}

int zip_sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    }
    return n;
}

}  // namespace

extern "C" long long skml_zipml_scratch_bytes(long long n_max) {
    if (n_max < 1 || n_max > 0x7FFFFFFFll) return -1;
    return (long long)carve(nullptr, n_max, nullptr);
}

extern "C" int skml_zipml_code_bytes(int bin_num) { return bin_num + 2 <= 256 ? 1 : 2; }

// entries of the split / midpoint tables of one list
extern "C" int skml_zipml_table_len(int bin_num) { return bin_num + 2; }

// vals[0..*n_ptr) -> codes (one per value), mids[bin_num + 2] (decode value of every bucket),
// meta[3] (buckets, zero bucket, rounds), range[2]. splits: bin_num + 2 floats for the split points.
extern "C" int skml_zipml_pack(const float* vals, const long long* n_ptr, long long n_max, int bin_num, void* scratch,
                               long long scratch_bytes, float* splits, float* mids, int* meta, float* range,
                               unsigned char* codes, unsigned int* status, void* stream) {
    if (!status || bin_num < 2 || bin_num + 2 > Z_MAX_BUCKETS || n_max < 1 || n_max > 0x7FFFFFFFll) return (int)cudaErrorInvalidValue;
    ZScratch z;
    if ((long long)carve(reinterpret_cast<unsigned char*>(scratch), n_max, &z) > scratch_bytes) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(z.shared, 0, offsetof(ZShared, digits), s);   // the barriers' words
    if (e != cudaSuccess) return (int)e;
    long long sorters = n_max <= Z_SORT_ALONE ? 1 : (n_max + 4095) / 4096;
    if (sorters > Z_MAX_BLOCKS) sorters = Z_MAX_BLOCKS;
    if (sorters > zip_sm_count()) sorters = zip_sm_count();
    if (n_max <= sorters * ZT * Z_SORT_KEYS) {   // (beyond, passes over memory are what a sort costs)
        unsigned int* a = reinterpret_cast<unsigned int*>(z.sorted_in);
        unsigned int* b = reinterpret_cast<unsigned int*>(z.sorted);
        if (sorters == 1) e = skml_launch(zip_sort_kernel<true>, 1, ZT, 0, s, vals, n_ptr, n_max, a, b, z.shared, status);
        else e = skml_launch_as(true, zip_sort_kernel<false>, (unsigned)sorters, ZT, 0, s, vals, n_ptr, n_max, a, b, z.shared, status);
    } else {
        zip_pad_kernel<<<zip_sm_count() * 4, 256, 0, s>>>(vals, n_ptr, n_max, z.sorted_in);
        e = cub::DeviceRadixSort::SortKeys(z.cub_temp, z.cub_bytes, z.sorted_in, z.sorted, (int)n_max, 0, 32, s);
    }
    if (e != cudaSuccess) return (int)e;
    // a block per slice of about 2048 values, as many as their lists of kept pairs have room for
    long long blocks = (n_max + 2047) / 2048;
    const int keep = bin_num / 2 > 1 ? bin_num / 2 : 1;
    if (blocks > Z_ALONE / keep) blocks = Z_ALONE / keep;
    if (blocks > Z_MAX_BLOCKS) blocks = Z_MAX_BLOCKS;
    if (blocks > zip_sm_count()) blocks = zip_sm_count();
    if (blocks < 1 || n_max <= 2 * Z_ALONE) blocks = 1;
    static bool ready = false;
    if (!ready) {
        e = cudaFuncSetAttribute(zip_splits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ZSmem));
        if (e != cudaSuccess) return (int)e;
        ready = true;
    }
    e = skml_launch_as(true, zip_splits_kernel, (unsigned)blocks, ZT, sizeof(ZSmem), s, z, n_ptr, n_max, bin_num, splits, mids, meta, range, status);
    if (e != cudaSuccess) return (int)e;
    const int cb = skml_zipml_code_bytes(bin_num);
    skml_launch(zip_code_kernel, zip_sm_count() * 4, 256, sizeof(float) * (size_t)(bin_num + 2), s, vals, n_ptr, n_max, splits, meta, cb, codes, status);
    return (int)cudaGetLastError();
}

// One launch per list, in list order (every rank adds the lists to a coordinate in the same order).
// mids: `lists` tables of bin_num + 2 floats; codes: `lists` arrays code_stride bytes apart.
extern "C" int skml_zipml_unpack_scatter(float* acc, const int* keys, const unsigned char* codes, const float* mids,
                                         const long long* counts, long long key_stride, long long code_stride,
                                         int lists, int bin_num, float* vals_out, const unsigned int* status, void* stream) {
    if (bin_num < 2 || bin_num + 2 > Z_MAX_BUCKETS) return (int)cudaErrorInvalidValue;
    const int cb = skml_zipml_code_bytes(bin_num);
    for (int l = 0; l < lists; ++l) {
        const int tl = bin_num + 2;
        skml_launch(zip_unpack_scatter_kernel, zip_sm_count() * 4, 256, sizeof(float) * (size_t)tl, (cudaStream_t)stream,
                    acc, keys ? keys + (long long)l * key_stride : nullptr, codes + (long long)l * code_stride,
                    mids + (long long)l * tl, counts + l, key_stride, cb, tl, vals_out ? vals_out + (long long)l * key_stride : nullptr, status);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}
