// DeltaAdaptive key codec as a stand-alone call (the fused exchange codes keys inside its own kernels). Behaviour
// follows the reference's live key encoder, binary/DeltaAdaptiveEncoder.java:23-146:
//   bitsNeeded_i = floor(log2(delta_i)) + 1 (1 for a first key of 0), histogram over 1..31;
//   interval count m in {2, 4, 8, 16} (fallback 1) and fixed vs unary flags chosen by the estimated
//   bits per key; flag = need - 1 in log2(m) bits (fixed) or `need` ones and a zero (unary) with
//   need = ceil(bitsNeeded / (32 / m)); delta in (32 / m) * need bits; both most significant bit
//   first in two separate streams in java.util.BitSet order (stream bit p = bit (p & 31) of 32-bit
//   word p >> 5).
//
// Every kernel cuts the keys into contiguous runs of whole tiles, one run per block, so the prefix sums over runs are short
// enough for every block to add up on its own. Encoding is one cooperative launch (two where its output would be large, see
// skml_da_encode), and so is decoding of fixed-width flags where a tile a block is enough (1.2M keys; otherwise three launches,
// and two more where flags are unary). What bounds both at ordinary sizes is the chain of trips to L2, two or three from block to block among them, and the
// host's calls around the one wait. 1M keys there and back: 64 us, 80 as seven launches (plan, pack, widths, keys, offsets
// and fills; 43 us of kernels against 27 here), 300 with library scans.
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "skml_api.h"
#include "skml_device.cuh"

namespace {

constexpr int KT = 1024;
constexpr int KPT = 8;              // adjacent keys of a thread
constexpr int KEY_TILE = KT * KPT;
constexpr int KEY_BLOCKS = 192;     // at most one block per SM: a grid barrier of 592 small blocks took twice as long
constexpr int STAGE_F = KEY_TILE * 17 / 32 + 2;   // words of one tile's flag bits (at most 17 a key, plus a word of misalignment)
constexpr int STAGE_D = KEY_TILE + 2;             // the same for its delta bits (at most 32 a key)
constexpr int LT = 256, LPT = 4, L_TILE = LT * LPT, L_BLOCKS = 592;   // unary flags, long lists: four small blocks per SM
constexpr long long KEY_BUDGET = 2000000000ll;    // cycles a grid barrier waits at most

// What a block tells the others it tells in words that say themselves that they are there, and who needs them polls the
// words: a grid barrier (fence, count, poll, fence) and the loads behind it are four trips to L2, this is two. 1M keys encoded
// 18.7 -> 17.3 us, decoded 15.9 -> 9.6; 10,000 keys 16.9 -> 15.4 and 9.8 -> 7.1; 1.2M 18.9 -> 18.4 and 18.1 -> 8.6.
constexpr unsigned int ROW_HERE = 1u << 31, ROW_BAD = 1u << 30;         // beside a run's count of a width (runs are below 2^30 keys)
constexpr unsigned long long SUM_HERE = 1ull << 63, SUM_GONE = 1ull << 50;   // beside a tile's sum (192 of them are below 2^40)

struct KeyWork {
    unsigned long long told_a[KEY_BLOCKS], told_b[KEY_BLOCKS];   // decode: sums over the tiles; cleared by the host
    unsigned int ticket, status;        // encode: cleared by the host; status: SkmlStatus (SKML_BAD_INPUT: keys not strictly increasing, or negative)
    unsigned int pad[30];
    unsigned int hist[KEY_BLOCKS][32];  // encode: delta widths of the runs; cleared by the host
    unsigned long long run_a[L_BLOCKS], run_b[L_BLOCKS];       // decode of long lists: sums over the runs
    unsigned long long zeros[L_BLOCKS];
};

struct Runs {
    long long per_run;
    int runs;
};

Runs runs_for(long long n, long long tile, int blocks) {
    const long long tiles = (n + tile - 1) / tile;
    long long per = (tiles + blocks - 1) / blocks;
    if (per < 1) per = 1;
    Runs r;
    r.per_run = per * tile;
    r.runs = (int)((tiles + per - 1) / per);
    if (r.runs < 1) r.runs = 1;
    return r;
}

__device__ __forceinline__ int bits_needed(int d) { return d <= 0 ? 1 : 32 - __clz((unsigned int)d); }

// Exclusive sum over the block's threads; `total` = the block's sum. Two barriers.
template <int THREADS, class T>
__device__ __forceinline__ T block_scan(T v, T* part, T& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    __syncthreads();   // the previous call's readers are done
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    const T x = lane < THREADS / 32 ? part[lane] : T(0);
    total = warp_sum(x);
    return warp_sum(lane < warp ? x : T(0)) + inc - v;
}

// Polls a block's word, `v` on, until `here` is set in it; false where that takes more than `budget` cycles. (With sleeps of 10
// to 200 ns between the polls, 1M keys were decoded in 10.8 us instead of 9.6.)
template <class T, class Load>
__device__ __forceinline__ bool await_word(T& v, T here, long long budget, Load load) {
    const long long t0 = clock64();
    while (!(v & here)) {
        if (clock64() - t0 > budget) return false;
        v = load();
    }
    return true;
}

// Sum of what the first `count` blocks tell, a thread per block; SUM_GONE or more where one of them has not told it in time.
// `part`: KEY_BLOCKS / 32 words that nobody else writes. (Not inlined: with the
// loop twice in the kernel, decoding 1M keys took 16.7 us instead of 10.8.)
__device__ __noinline__ unsigned long long told_before(const unsigned long long* told, int count, long long budget, unsigned long long* part) {
    const int warp = threadIdx.x >> 5;
    if (warp < KEY_BLOCKS / 32) {
        unsigned long long v = 0;
        if ((int)threadIdx.x < count) {
            const unsigned long long* const word = told + threadIdx.x;
            v = ld_relaxed_gpu64(word);
            v = await_word(v, SUM_HERE, budget, [=] { return ld_relaxed_gpu64(word); }) ? v & ~SUM_HERE : SUM_GONE;
        }
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) part[warp] = v;
    }
    __syncthreads();
    unsigned long long sum = 0;
#pragma unroll
    for (int w = 0; w < KEY_BLOCKS / 32; ++w) sum += part[w];
    return sum;
}

// Sum of sums[0, count) of a launch before, by the whole block.
template <int THREADS>
__device__ __forceinline__ unsigned long long block_sum_before(const unsigned long long* sums, int count, unsigned long long* part) {
    unsigned long long v = 0, total;
    for (int i = threadIdx.x; i < count; i += THREADS) v += __ldcg(sums + i);
    block_scan<THREADS>(v, part, total);
    return total;
}

// Interval counts, widths and flag of a delta under m intervals of b = 1 << lb bits.
struct Code {
    unsigned int fv, fw, dw;   // flag value, flag width, delta width
};
__device__ __forceinline__ Code code_of(unsigned int delta, unsigned int lb, unsigned int fb, unsigned int kind) {
    const unsigned int iv = ((unsigned int)bits_needed((int)delta) + (1u << lb) - 1u) >> lb;
    Code c;
    c.fw = kind ? iv + 1 : fb;
    c.fv = kind ? (1u << (iv + 1)) - 2u : iv - 1;
    c.dw = iv << lb;
    return c;
}

// Deltas of a thread's keys i0 .. i0 + KPT (0 beyond hi). `bad`: keys that are negative or do not ascend.
__device__ __forceinline__ void load_deltas(const int* __restrict__ keys, long long i0, long long hi, unsigned int (&d)[KPT], bool& bad) {
    const int lane = threadIdx.x & 31;
    int k[KPT];
    if (i0 + KPT <= hi && (reinterpret_cast<uintptr_t>(keys) & 15) == 0) {   // (i0 is a multiple of KPT)
#pragma unroll
        for (int q = 0; q < KPT / 4; ++q) {
            const int4 v = *reinterpret_cast<const int4*>(keys + i0 + 4 * q);
            k[4 * q] = v.x; k[4 * q + 1] = v.y; k[4 * q + 2] = v.z; k[4 * q + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int u = 0; u < KPT; ++u) k[u] = i0 + u < hi ? keys[i0 + u] : 0;
    }
    int prev = __shfl_up_sync(0xFFFFFFFFu, k[KPT - 1], 1);
    if (lane == 0) prev = i0 > 0 && i0 <= hi ? keys[i0 - 1] : 0;
#pragma unroll
    for (int u = 0; u < KPT; ++u) {
        const bool in = i0 + u < hi;
        if (in && (k[u] < prev || (k[u] == prev && i0 + u > 0) || k[u] < 0)) bad = true;
        d[u] = in ? (unsigned int)k[u] - (unsigned int)prev : 0u;
        prev = k[u];
    }
}

// A thread's bits on their way to a zeroed shared-memory word array, most significant bit of every value first (stream
// bit p = bit (p & 31) of word p >> 5): words between its first and its last are its own, those two it may share.
struct BitWriter {
    unsigned int* word;
    unsigned long long acc;
    unsigned int have;
    bool shared;
    __device__ __forceinline__ BitWriter(unsigned int* words, unsigned int off) : word(words + (off >> 5)), acc(0), have(off & 31u), shared((off & 31u) != 0) {}
    __device__ __forceinline__ void put(unsigned int value, unsigned int nb) {   // nb <= 32
        if (nb == 0) return;
        acc |= (unsigned long long)(__brev(value) >> (32u - nb)) << have;
        have += nb;
        if (have >= 32u) {
            if (shared) atomicOr(word, (unsigned int)acc);
            else *word = (unsigned int)acc;
            shared = false;
            ++word;
            acc >>= 32;
            have -= 32u;
        }
    }
    __device__ __forceinline__ void close() {
        if (have && (unsigned int)acc) atomicOr(word, (unsigned int)acc);
    }
};

// Interval count and flag kind of the DeltaAdaptive key code (reference: binary/DeltaAdaptiveEncoder.java:23-112), by one
// warp: prob[w] (shared memory) = share of the deltas of width w. The reference's estimates in the same double arithmetic,
// operation by operation (explicit round-to-nearest intrinsics keep the compiler from fusing multiply-adds), but a lane per
// interval of every interval count: as one lane per count they were a chain of a hundred additions.
__device__ __forceinline__ void da_mode(const double* prob, unsigned int& num, unsigned int& kind) {
    const int lane = threadIdx.x & 31, q = lane < 2 ? 0 : (lane < 6 ? 1 : (lane < 14 ? 2 : 3)), i = lane - ((2 << q) - 2);
    double ip = 0.0;
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < (16 >> q) && lane < 30) ip = __dadd_rn(ip, prob[i * (16 >> q) + j]);
    const double term = __dmul_rn((double)(i + 1), ip);
    const int m = 2 << (lane & 3), b = 16 >> (lane & 3);   // lanes 0 to 3: the estimates of 2, 4, 8 and 16 intervals
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const double t = __shfl_sync(0xFFFFFFFFu, term, (m - 2 + k) & 31);
        if (k < m) sum = __dadd_rn(sum, t);
    }
    const double t1 = __dadd_rn(__dmul_rn(sum, (double)b), (double)((lane & 3) + 1)), t2 = __dadd_rn(__dmul_rn(sum, (double)(b + 1)), 1.0);
    double best = 32.0;
    num = 1;
    kind = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double fixed = __shfl_sync(0xFFFFFFFFu, t1, k), unary = __shfl_sync(0xFFFFFFFFu, t2, k);
        if (fixed < best) {
            best = fixed;
            num = 2u << k;
            kind = 0;
        }
        if (unary < best) {
            best = unary;
            num = 2u << k;
            kind = 1;
        }
    }
}

// One stream on its way through shared memory. A tile's whole words are stored; the word it ends in goes on to the
// next tile, the word a run starts in belongs to the run before, and the run's last word is completed with the first
// bits of the run behind it (write_tails), so that nobody shares a word and nothing has to be cleared first.
struct Out {
    unsigned int* words;
    unsigned long long at;   // stream bit of the next key
    unsigned int carry;      // bits of the word `at` lies in
    bool mine;               // whether that word is this run's
};

__device__ __forceinline__ void open_tile(unsigned int* stage, unsigned int nbits, const Out& o) {
    const unsigned int words = ((unsigned int)(o.at & 31ull) + nbits) / 32u + 1u;
    for (unsigned int i = threadIdx.x; i < words; i += KT) stage[i] = i ? 0u : o.carry;
}

__device__ __forceinline__ void flush_tile(const unsigned int* stage, Out& o, unsigned int nbits) {
    const unsigned int end = (unsigned int)(o.at & 31ull) + nbits, full = end >> 5;
    unsigned int* dst = o.words + (o.at >> 5);
    for (unsigned int w = threadIdx.x; w < full; w += KT)
        if (w || o.mine) dst[w] = stage[w];
    o.carry = end & 31u ? stage[full] : 0u;
    o.mine = o.mine || full;
    o.at += nbits;
}

// The words the run ends in, by one warp: up to 32 keys behind the run have bits there.
__device__ __forceinline__ void write_tails(const int* __restrict__ keys, long long hi, long long n, unsigned int lb, unsigned int fb,
                                            unsigned int kind, const Out& f, const Out& d) {
    const unsigned int lane = threadIdx.x & 31;
    const long long i = hi + lane;
    Code c{0, 0, 0};
    unsigned int delta = 0;
    if (i < n) {
        delta = (unsigned int)keys[i] - (unsigned int)keys[i - 1];
        c = code_of(delta, lb, fb, kind);
    }
    unsigned int inc = c.fw + (c.dw << 16);   // at most 17 * 32 and 32 * 32
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= (unsigned int)o) inc += t;
    }
    const unsigned int fo = (unsigned int)(f.at & 31ull) + (inc & 0xFFFFu) - c.fw, dof = (unsigned int)(d.at & 31ull) + (inc >> 16) - c.dw;
    const unsigned int fbits = __reduce_or_sync(0xFFFFFFFFu, c.fw && fo < 32u ? (__brev(c.fv) >> (32u - c.fw)) << fo : 0u);
    const unsigned int dbits = __reduce_or_sync(0xFFFFFFFFu, c.dw && dof < 32u ? (__brev(delta) >> (32u - c.dw)) << dof : 0u);
    if (lane == 0) {
        if (f.mine && (f.at & 31ull)) f.words[f.at >> 5] = f.carry | fbits;
        if (d.mine && (d.at & 31ull)) d.words[d.at >> 5] = d.carry | dbits;
        if (hi == n) {   // the streams are counted in 64-bit words
            const unsigned long long fw = (f.at + 31ull) >> 5, dw = (d.at + 31ull) >> 5;
            if (fw & 1ull) f.words[fw] = 0u;
            if (dw & 1ull) d.words[dw] = 0u;
        }
    }
}

// Encoding in one cooperative launch: every run's histogram of delta widths, told to all blocks, the mode and the run's
// first bits from the histograms (every block adds up all, and those of the runs before its own), then the streams.
// Runs of one tile keep their deltas in registers meanwhile. 17.3 us at 1M keys, 15.4 at 10,000: latency.
// Mode and lengths are reported once every block has all histograms, where nothing can fail any more: what the host does
// with them, it does beside the streams.
// `words`: where the streams go, the flags and, from the next whole 64-bit word on, the deltas; `room` 64-bit words of it.
// Null: mode and lengths only. `planned`: a launch of that kind has left the histograms of these keys in the workspace.
__global__ void __launch_bounds__(KT, 1)
da_encode_kernel(const int* __restrict__ keys, long long n, long long per_run, KeyWork* __restrict__ wk, unsigned int* words,
                 unsigned long long room, bool planned, unsigned long long* done, unsigned long long seq) {
    extern __shared__ __align__(16) unsigned int s_stage[];
    unsigned int* const s_f = s_stage;
    unsigned int* const s_d = s_stage + STAGE_F;
    __shared__ unsigned int s_h[KT / 32][32], s_all[KT / 32][32], s_before[KT / 32][32];
    __shared__ unsigned long long s_part[KT / 32], s_at[4];
    __shared__ double s_prob[32];
    __shared__ unsigned int s_mode[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    bool bad = false;
    unsigned int x[KPT];
    if (!planned) {
        unsigned int count = 0;   // lane w counts width w
        for (long long t0 = lo; t0 < hi; t0 += KEY_TILE) {
            const long long i0 = t0 + (long long)KPT * threadIdx.x;
            load_deltas(keys, i0, hi, x, bad);
#pragma unroll
            for (int u = 0; u < KPT; ++u) {   // a ballot per bit of the width: all lanes would meet in a few counters
                const int width = bits_needed((int)x[u]) & 31;
                unsigned int of_lane = __ballot_sync(0xFFFFFFFFu, i0 + u < hi);
#pragma unroll
                for (int k = 0; k < 5; ++k) of_lane &= __ballot_sync(0xFFFFFFFFu, (width >> k) & 1) ^ (((unsigned int)lane >> k & 1u) - 1u);
                count += (unsigned int)__popc(of_lane);
            }
        }
        s_h[warp][lane] = count;
        if (bad) skml_set_status(&wk->status, SKML_BAD_INPUT, 0x70u);
        const unsigned int any = __syncthreads_or(bad) ? ROW_BAD : 0u;
        if (warp == 0) {
            unsigned int t = 0;
            for (int w = 0; w < KT / 32; ++w) t += s_h[w][lane];
            st_relaxed_gpu(&wk->hist[blockIdx.x][lane], ROW_HERE | any | t);
        }
    }
    {   // all runs' histograms, a width per lane, a warp's rows in flight together
        constexpr int ROWS = KEY_BLOCKS / (KT / 32);
        unsigned int row[ROWS], all = 0, before = 0;
        bool stop = false;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int r = warp + j * (KT / 32);
            row[j] = r < (int)gridDim.x ? ld_relaxed_gpu(&wk->hist[r][lane]) : ROW_HERE;
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int r = warp + j * (KT / 32);
            if (!await_word(row[j], ROW_HERE, KEY_BUDGET, [=] { return ld_relaxed_gpu(&wk->hist[r][lane]); })) {
                skml_set_status(&wk->status, SKML_TIMEOUT_BARRIER, 0x71u);
                stop = true;
                break;
            }
            stop = stop || (row[j] & ROW_BAD);
            const unsigned int t = row[j] & (ROW_BAD - 1u);
            all += t;
            if (r < (int)blockIdx.x) before += t;
        }
        s_all[warp][lane] = all;
        s_before[warp][lane] = before;
        if (__syncthreads_or(stop)) return;   // (the same in every block, but for waits that run out: the status says so)
    }
    unsigned int total = 0;
    if (warp == 0) {
        for (int w = 0; w < KT / 32; ++w) total += s_all[w][lane];
        s_prob[lane] = __ddiv_rn((double)total, (double)(n > 0 ? n : 1));
        __syncwarp();
        unsigned int num, mode;
        da_mode(s_prob, num, mode);
        if (lane == 0) {
            s_mode[0] = num;
            s_mode[1] = mode;
        }
    } else if (warp == 1) {
        unsigned int t = 0;
        for (int w = 0; w < KT / 32; ++w) t += s_before[w][lane];
        s_before[0][lane] = t;
    }
    __syncthreads();
    const unsigned int m = s_mode[0], kind = s_mode[1], lb = (unsigned int)__clz(m) - 26u, fb = 5u - lb;   // 32 / m bits an interval
    if (warp == 0) {
        const unsigned int before = s_before[0][lane];
        const unsigned int iv = ((lane ? (unsigned int)lane : 32u) + (1u << lb) - 1u) >> lb, fw = kind ? iv + 1 : fb, dw = iv << lb;
        const unsigned long long f0 = warp_sum((unsigned long long)before * fw), d0 = warp_sum((unsigned long long)before * dw);
        const unsigned long long fa = warp_sum((unsigned long long)total * fw), da = warp_sum((unsigned long long)total * dw);
        if (lane == 0) {
            s_at[0] = f0;
            s_at[1] = d0;
            s_at[2] = fa;
            s_at[3] = da;
        }
    }
    __syncthreads();
    const unsigned long long fwords = (s_at[2] + 63ull) >> 6, dwords = (s_at[3] + 63ull) >> 6;
    if (!planned && threadIdx.x == 0 && atomicAdd(&wk->ticket, 1u) == gridDim.x - 1) {
        done[1] = (unsigned long long)m | ((unsigned long long)kind << 32);
        done[2] = s_at[2];
        done[3] = s_at[3];
        __threadfence_system();
        skml_store_done(done, seq, &wk->status);
    }
    if (!words || fwords + dwords > room) return;   // (the same in every block; the host compares the lengths too)
    Out f{words, s_at[0], 0u, (s_at[0] & 31ull) == 0}, d{words + 2 * fwords, s_at[1], 0u, (s_at[1] & 31ull) == 0};
    for (long long t0 = lo; t0 < hi; t0 += KEY_TILE) {
        const long long i0 = t0 + (long long)KPT * threadIdx.x;
        if (planned || per_run > KEY_TILE) load_deltas(keys, i0, hi, x, bad);
        unsigned int fsum = 0, dsum = 0;   // at most 17 and 32 bits a key
#pragma unroll
        for (int u = 0; u < KPT; ++u)
            if (i0 + u < hi) {
                const Code c = code_of(x[u], lb, fb, kind);
                fsum += c.fw;
                dsum += c.dw;
            }
        unsigned long long bits;
        const unsigned long long ex = block_scan<KT>(((unsigned long long)dsum << 32) | fsum, s_part, bits);
        open_tile(s_f, (unsigned int)bits, f);
        open_tile(s_d, (unsigned int)(bits >> 32), d);
        __syncthreads();
        BitWriter wf(s_f, (unsigned int)(f.at & 31ull) + (unsigned int)ex), wd(s_d, (unsigned int)(d.at & 31ull) + (unsigned int)(ex >> 32));
#pragma unroll
        for (int u = 0; u < KPT; ++u)
            if (i0 + u < hi) {
                const Code c = code_of(x[u], lb, fb, kind);
                wf.put(c.fv, c.fw);
                wd.put(x[u], c.dw);
            }
        wf.close();
        wd.close();
        __syncthreads();
        flush_tile(s_f, f, (unsigned int)bits);
        flush_tile(s_d, d, (unsigned int)(bits >> 32));
        // (the next tile's words are cleared behind the barriers of its scan)
    }
    if (warp == 0) write_tails(keys, hi, n, lb, fb, kind, f, d);
}

struct Streams {
    const unsigned int* flag_words;
    const unsigned int* delta_words;
    long long flag_lim, delta_lim;    // 32-bit words
    const long long* zero_pos;        // unary flags: where every key's flag ends
    unsigned int m;
    int unary;
};

// Interval counts of a thread's N keys (at most eight), from i0 on (0 beyond `hi`).
template <int N>
__device__ __forceinline__ void intervals(const Streams& s, long long i0, long long hi, unsigned int (&iv)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u) iv[u] = 0;
    if (i0 >= hi) return;
    if (s.unary) {
        long long before = i0 ? s.zero_pos[i0 - 1] : -1;
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (i0 + u < hi) {
                const long long z = s.zero_pos[i0 + u];
                iv[u] = (unsigned int)(z - before - 1);
                before = z;
            }
        return;
    }
    const unsigned int fb = 31u - (unsigned int)__clz(s.m);   // at most 4
    unsigned long long win = 0;
    if (fb) {
        const unsigned long long off = (unsigned long long)i0 * fb;
        const long long w = (long long)(off >> 5);
        const unsigned int lo = w < s.flag_lim ? s.flag_words[w] : 0u, hw = w + 1 < s.flag_lim ? s.flag_words[w + 1] : 0u;
        win = ((unsigned long long)lo | ((unsigned long long)hw << 32)) >> (off & 31ull);
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
        if (i0 + u < hi) {
            const unsigned int bits = fb ? (unsigned int)(win >> (fb * u)) & ((1u << fb) - 1u) : 0u;
            iv[u] = (fb ? __brev(bits) >> (32u - fb) : 0u) + 1u;
        }
}

// Unary flags: zero bits of every run of flag words (a key's flag ends at its zero bit).
__global__ void __launch_bounds__(LT) da_zero_count_kernel(const unsigned int* __restrict__ flag_words, long long flag_bits, long long per_run,
                                                           KeyWork* __restrict__ wk) {
    __shared__ unsigned long long s_part[LT / 32];
    const long long nw = (flag_bits + 31) >> 5, lo = per_run * blockIdx.x, hi = lo + per_run < nw ? lo + per_run : nw;
    unsigned long long v = 0, total;
    for (long long w = lo + threadIdx.x; w < hi; w += LT) {
        const long long rest = flag_bits - (w << 5);
        v += __popc(~flag_words[w] & (rest >= 32 ? 0xFFFFFFFFu : ((1u << rest) - 1u)));
    }
    block_scan<LT>(v, s_part, total);
    if (threadIdx.x == 0) wk->zeros[blockIdx.x] = total;
}

// Stream position of the i-th zero bit.
__global__ void __launch_bounds__(LT) da_zero_pos_kernel(const unsigned int* __restrict__ flag_words, long long flag_bits, long long per_run,
                                                         const KeyWork* __restrict__ wk, long long n, long long* __restrict__ pos) {
    __shared__ unsigned long long s_part[LT / 32];
    const long long nw = (flag_bits + 31) >> 5, lo = per_run * blockIdx.x, hi = lo + per_run < nw ? lo + per_run : nw;
    unsigned long long base = block_sum_before<LT>(wk->zeros, blockIdx.x, s_part);
    for (long long w0 = lo; w0 < hi; w0 += LT) {
        const long long w = w0 + threadIdx.x;
        unsigned int z = 0;
        if (w < hi) {
            const long long rest = flag_bits - (w << 5);
            z = ~flag_words[w] & (rest >= 32 ? 0xFFFFFFFFu : ((1u << rest) - 1u));
        }
        unsigned long long total;
        unsigned long long idx = base + block_scan<LT>((unsigned long long)__popc(z), s_part, total);
        while (z) {
            const int bit = __ffs(z) - 1;
            z &= z - 1;
            if (idx < (unsigned long long)n) pos[idx] = (w << 5) + bit;
            ++idx;
        }
        base += total;
    }
}

// Bits of the deltas of a thread's keys.
template <int N>
__device__ __forceinline__ unsigned int delta_bits(const Streams& s, const unsigned int (&iv)[N]) {
    unsigned int t = 0;
#pragma unroll
    for (int u = 0; u < N; ++u) t += iv[u];
    return t * (32u / s.m);
}

// Keys of a tile, each counted from its thread's first one: k[u] = sum of the deltas up to the thread's u-th. `bit`: the
// tile's first delta bit, then the next tile's. Returns the thread's sum.
template <int THREADS, int N>
__device__ __forceinline__ unsigned int tile_keys(const Streams& s, const unsigned int (&iv)[N], unsigned long long& bit, unsigned int* part32,
                                                  unsigned int (&k)[N]) {
    const unsigned int b = 32u / s.m;
    unsigned int total;
    unsigned long long off = bit + block_scan<THREADS>(delta_bits(s, iv), part32, total);
    bit += total;
    unsigned int dsum = 0;
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const unsigned int dw = b * iv[u];
        unsigned int d = 0;
        if (dw && dw <= 32u) {
            const long long w = (long long)(off >> 5);
            const unsigned int x0 = w < s.delta_lim ? s.delta_words[w] : 0u, x1 = w + 1 < s.delta_lim ? s.delta_words[w + 1] : 0u;
            d = __brev(__funnelshift_r(x0, x1, (unsigned int)(off & 31ull)) << (32u - dw));
        }
        off += dw;
        dsum += d;
        k[u] = dsum;
    }
    return dsum;
}

// What the blocks before this one would have told it, found by itself: delta bits and sum of the keys [0, lo).
__device__ __noinline__ void before_run(Streams s, long long lo, unsigned int* part32, unsigned long long& bit, unsigned int& sum) {
    bit = 0;
    sum = 0;
    for (long long t0 = 0; t0 < lo; t0 += KEY_TILE) {
        unsigned int iv[KPT], k[KPT], tile_sum;
        intervals(s, t0 + (long long)KPT * threadIdx.x, lo, iv);
        block_scan<KT>(tile_keys<KT>(s, iv, bit, part32, k), part32, tile_sum);
        sum += tile_sum;
    }
}

// Decoding in one cooperative launch, where a block has one tile: its delta bits, told to the blocks behind it, its keys
// counted from the key before them, their sum told, too, and the sum of the tiles before it added; flags and keys stay in registers.
// The caller is not told how the launch went, so it cannot fail: where a wait runs out, the block works out for itself
// what it waited for, and tells the others what they wait for all the same.
__global__ void __launch_bounds__(KT, 1)
da_decode_kernel(Streams s, long long n, KeyWork* __restrict__ wk, int* __restrict__ keys, long long budget) {
    __shared__ unsigned long long s_part[KT / 32], s_told[2][KEY_BLOCKS / 32];
    __shared__ unsigned int s_part32[KT / 32];
    const long long lo = (long long)KEY_TILE * blockIdx.x, i0 = lo + (long long)KPT * threadIdx.x;
    unsigned int iv[KPT], k[KPT], sum, add = 0;
    bool together = gridDim.x > 1;   // (one block has nothing to wait for)
    unsigned long long bit = 0;
    intervals(s, i0, n, iv);
    if (together) {
        unsigned long long total;
        block_scan<KT>((unsigned long long)delta_bits(s, iv), s_part, total);
        if (threadIdx.x == 0) st_relaxed_gpu64(&wk->told_a[blockIdx.x], SUM_HERE | total);
        bit = told_before(wk->told_a, blockIdx.x, budget, s_told[0]);
        together = bit < SUM_GONE;
        if (!together) before_run(s, lo, s_part32, bit, add);
    }
    const unsigned int before = block_scan<KT>(tile_keys<KT>(s, iv, bit, s_part32, k), s_part32, sum);   // keys are below 2^31: 32-bit sums are exact
    if (gridDim.x > 1 && threadIdx.x == 0) st_relaxed_gpu64(&wk->told_b[blockIdx.x], SUM_HERE | sum);
    if (together) {
        const unsigned long long keys_before = told_before(wk->told_b, blockIdx.x, budget, s_told[1]);
        if (keys_before < SUM_GONE) add = (unsigned int)keys_before;
        else before_run(s, lo, s_part32, bit, add);
    }
    add += before;
    if (i0 + KPT <= n && (reinterpret_cast<uintptr_t>(keys) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < KPT / 4; ++q)
            *reinterpret_cast<uint4*>(keys + i0 + 4 * q) = make_uint4(k[4 * q] + add, k[4 * q + 1] + add, k[4 * q + 2] + add, k[4 * q + 3] + add);
    } else {
#pragma unroll
        for (int u = 0; u < KPT; ++u)
            if (i0 + u < n) keys[i0 + u] = (int)(k[u] + add);
    }
}

// Longer lists, and unary flags, where two launches have come before and the stream is never idle for the host: three
// launches, a run of tiles per block and four small blocks per SM, which hide one another's trips to memory. With the runs of
// tiles in one block of 1024 per SM and grid barriers, 2M keys took 38 us instead of 28, 20M 206 instead of 143 and 100M 1870
// instead of 1430; 100,000 keys with unary flags 35 instead of 32. (Fixed-width flags, one launch instead of three: 100,000
// keys 11.7 instead of 17.3, 1M 13.1 instead of 19.3, fill and gaps with them.)
// Delta bits of every run.
__global__ void __launch_bounds__(LT) da_width_kernel(Streams s, long long n, long long per_run, KeyWork* __restrict__ wk) {
    __shared__ unsigned long long s_part[LT / 32];
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    unsigned long long v = 0, total;
    for (long long t0 = lo; t0 < hi; t0 += L_TILE) {
        unsigned int iv[LPT];
        intervals(s, t0 + LPT * (long long)threadIdx.x, hi, iv);
        v += delta_bits(s, iv);
    }
    block_scan<LT>(v, s_part, total);
    if (threadIdx.x == 0) wk->run_a[blockIdx.x] = total;
}

// Keys of every run counted from the key before it, and the runs' sums.
__global__ void __launch_bounds__(LT) da_extract_kernel(Streams s, long long n, long long per_run, KeyWork* __restrict__ wk, int* __restrict__ keys) {
    __shared__ unsigned long long s_part[LT / 32];
    __shared__ unsigned int s_part32[LT / 32];
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    unsigned long long bit = block_sum_before<LT>(wk->run_a, blockIdx.x, s_part);
    unsigned int sum = 0;
    for (long long t0 = lo; t0 < hi; t0 += L_TILE) {
        const long long i0 = t0 + LPT * (long long)threadIdx.x;
        unsigned int iv[LPT], k[LPT], tile_sum;
        intervals(s, i0, hi, iv);
        const unsigned int before = sum + block_scan<LT>(tile_keys<LT>(s, iv, bit, s_part32, k), s_part32, tile_sum);
#pragma unroll
        for (int u = 0; u < LPT; ++u)
            if (i0 + u < hi) keys[i0 + u] = (int)(k[u] + before);
        sum += tile_sum;
    }
    if (threadIdx.x == 0) wk->run_b[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(LT) da_offset_kernel(long long n, long long per_run, const KeyWork* __restrict__ wk, int* __restrict__ keys) {
    __shared__ unsigned long long s_part[LT / 32];
    if (blockIdx.x == 0) return;
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    const int add = (int)block_sum_before<LT>(wk->run_b, blockIdx.x, s_part);
    for (long long i = lo + threadIdx.x; i < hi; i += LT) keys[i] += add;
}

constexpr size_t ENCODE_SMEM = 4 * (size_t)(STAGE_F + STAGE_D);

// Blocks of a cooperative launch of a kernel on the current device (0: an error, asked for again by the next call). Asked
// for once per device: a kernel's limit of dynamic shared memory is set for one device only.
constexpr int KEY_DEVICES = 64;
template <class K>
int resident_blocks(K kernel, size_t smem, std::atomic<int> (&known)[KEY_DEVICES]) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const bool keep = dev >= 0 && dev < KEY_DEVICES;
    if (keep) {
        const int have = known[dev].load(std::memory_order_acquire);
        if (have) return have;
    }
    if (smem && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, KT, smem) != cudaSuccess || per_sm < 1)
        return 0;
    const int blocks = sms < KEY_BLOCKS ? sms : KEY_BLOCKS;
    if (keep) known[dev].store(blocks, std::memory_order_release);
    return blocks;
}

}  // namespace

extern "C" long long skml_da_workspace_bytes() { return (long long)sizeof(KeyWork); }

// The mode's estimate counts floor(w / b) + 1 intervals of b bits for a delta of w bits, at least as many as it takes, so the
// streams are no longer than the least estimate: 32 bits a key (the fallback's), and no more than that of 16 intervals with
// fixed flags, w + 2 + 4 bits. The deltas add up to the last key, below 2^31: their w, at most log2(delta) + 1, are
// log2(2^31 / n) + 1 on average at most. (And each stream's last word.)
extern "C" long long skml_da_words(long long n) {
    int log2n = 0;
    while ((n >> log2n) > 1) ++log2n;
    const long long bits = 38 - log2n < 32 ? 38 - log2n : 32;
    return n > 0 ? (bits * n + 63) / 64 + 4 : 0;
}

extern "C" int skml_da_encode(const int* keys, long long n, void* workspace, unsigned long long* words, long long n_words, int planned,
                              unsigned long long* done, unsigned int* status_out, void* stream) {
    if (n < 0 || n_words < 0 || !workspace || !done || !status_out || (n && !keys) || (planned && !words)) return (int)cudaErrorInvalidValue;
    static std::atomic<int> known[KEY_DEVICES];
    const int blocks = resident_blocks(da_encode_kernel, ENCODE_SMEM, known);
    if (blocks < 1) return (int)cudaErrorLaunchOutOfResources;
    cudaStream_t s = (cudaStream_t)stream;
    KeyWork* wk = reinterpret_cast<KeyWork*>(workspace);
    cudaError_t e = cudaSuccess;
    const Runs r = runs_for(n, KEY_TILE, blocks);
    if (!planned) e = cudaMemsetAsync(&wk->ticket, 0, offsetof(KeyWork, hist) - offsetof(KeyWork, ticket) + r.runs * sizeof(wk->hist[0]), s);
    if (e != cudaSuccess) return (int)e;
    unsigned long long seq = ((*done >> 32) + 1) & 0xFFFFFFFFull;
    long long per_run = r.per_run;
    unsigned int* out = reinterpret_cast<unsigned int*>(words);
    unsigned long long room = (unsigned long long)n_words;
    bool have_plan = planned != 0;
    void* args[] = {&keys, &n, &per_run, &wk, &out, &room, &have_plan, &done, &seq};
    e = cudaLaunchCooperativeKernel((const void*)da_encode_kernel, dim3((unsigned)r.runs), dim3(KT), args, ENCODE_SMEM, s);
    if (e != cudaSuccess) return (int)e;
    *status_out = 0;
    if (!planned) {
        const int rc = skml_wait_done(done, seq, &wk->status, status_out, s);
        if (rc || *status_out) return rc;
    }
    if (words && ((done[2] + 63ull) >> 6) + ((done[3] + 63ull) >> 6) > room) *status_out = SKML_CAPACITY;
    return 0;
}

extern "C" int skml_da_decode(const unsigned long long* flag_words, long long n_flag_words, const unsigned long long* delta_words,
                              long long n_delta_words, long long n, int num_intervals, int unary, long long flag_bits, void* workspace,
                              long long* zero_pos, int* keys, long long budget_cycles, void* stream) {
    if (num_intervals < 1 || num_intervals > 16 || (num_intervals & (num_intervals - 1)) || !workspace || (unary && !zero_pos))
        return (int)cudaErrorInvalidValue;
    if (n <= 0) return 0;
    static std::atomic<int> known[KEY_DEVICES];
    const int blocks = resident_blocks(da_decode_kernel, 0, known);
    if (blocks < 1) return (int)cudaErrorLaunchOutOfResources;
    cudaStream_t s = (cudaStream_t)stream;
    KeyWork* wk = reinterpret_cast<KeyWork*>(workspace);
    Streams st;
    st.flag_words = reinterpret_cast<const unsigned int*>(flag_words);
    st.delta_words = reinterpret_cast<const unsigned int*>(delta_words);
    st.flag_lim = 2 * n_flag_words;
    st.delta_lim = 2 * n_delta_words;
    st.zero_pos = zero_pos;
    st.m = (unsigned int)num_intervals;
    st.unary = unary != 0;
    if (unary) {
        const long long nw = (flag_bits + 31) >> 5;
        if (nw > st.flag_lim) return (int)cudaErrorInvalidValue;
        const Runs f = runs_for(nw, L_TILE, L_BLOCKS);
        da_zero_count_kernel<<<f.runs, LT, 0, s>>>(st.flag_words, flag_bits, f.per_run, wk);
        da_zero_pos_kernel<<<f.runs, LT, 0, s>>>(st.flag_words, flag_bits, f.per_run, wk, n, zero_pos);
    }
    const Runs r = runs_for(n, KEY_TILE, blocks);
    if (r.per_run > KEY_TILE || (unary && r.runs > 1)) {
        const Runs l = runs_for(n, L_TILE, L_BLOCKS);
        da_width_kernel<<<l.runs, LT, 0, s>>>(st, n, l.per_run, wk);
        da_extract_kernel<<<l.runs, LT, 0, s>>>(st, n, l.per_run, wk, keys);
        da_offset_kernel<<<l.runs, LT, 0, s>>>(n, l.per_run, wk, keys);
        return (int)cudaGetLastError();
    }
    if (r.runs > 1) {
        const cudaError_t e = cudaMemsetAsync(wk, 0, offsetof(KeyWork, ticket), s);
        if (e != cudaSuccess) return (int)e;
    }
    long long budget = budget_cycles > 0 ? budget_cycles : KEY_BUDGET;
    void* args[] = {&st, &n, &wk, &keys, &budget};
    return (int)cudaLaunchCooperativeKernel((const void*)da_decode_kernel, dim3((unsigned)r.runs), dim3(KT), args, 0, s);
}
