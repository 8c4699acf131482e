// DeltaAdaptive key codec as a stand-alone call (the fused exchange codes keys inside its own kernels). Behaviour
// follows the reference's live key encoder, binary/DeltaAdaptiveEncoder.java:23-146:
//   bitsNeeded_i = floor(log2(delta_i)) + 1 (1 for a first key of 0), histogram over 1..31;
//   interval count m in {2, 4, 8, 16} (fallback 1) and fixed vs unary flags chosen by the estimated
//   bits per key; flag = need - 1 in log2(m) bits (fixed) or `need` ones and a zero (unary) with
//   need = ceil(bitsNeeded / (32 / m)); delta in (32 / m) * need bits; both most significant bit
//   first in two separate streams in java.util.BitSet order (stream bit p = bit (p & 31) of 32-bit
//   word p >> 5).
//
// Every kernel cuts the keys into at most KEY_BLOCKS contiguous runs of whole 1024-key tiles, one run per
// block, so the prefix sums over runs are short enough for every block to add up on its own: encoding is two
// launches (a run's histogram of delta widths gives its stream lengths for every mode, so one pass decides
// the mode and every offset), decoding three (five with unary flags). What bounds both at ordinary sizes is
// launches and the one wait for the stream lengths that the caller allocates by: 1M keys there and back took
// 35 launches and 300 us as maps over keys with library scans between them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "skml_api.h"
#include "skml_device.cuh"

namespace {

constexpr int KT = 256;
constexpr int KEY_TILE = 1024;      // four adjacent keys a thread
constexpr int KEY_BLOCKS = 592;     // four blocks per SM
constexpr int STAGE_F = 548;        // words of one tile's flag bits (at most 17 a key, plus a word of misalignment)
constexpr int STAGE_D = 1028;       // the same for its delta bits (at most 32 a key)

struct KeyWork {
    unsigned int ticket, status;    // status bit 0: keys not strictly increasing (or negative)
    unsigned int m, kind;
    unsigned int pad[12];
    unsigned int total[32];         // encode: delta widths of all keys
    unsigned long long flag_off[KEY_BLOCKS], delta_off[KEY_BLOCKS];   // encode: first bits of the runs
    alignas(16) unsigned int hist[KEY_BLOCKS][32];                                // encode: delta widths of the runs
    unsigned long long run_a[KEY_BLOCKS], run_b[KEY_BLOCKS];          // decode: sums over the runs
};

struct Runs {
    long long tiles_per_run;
    int runs;
};

Runs runs_for(long long n) {
    const long long tiles = (n + KEY_TILE - 1) / KEY_TILE;
    Runs r;
    r.tiles_per_run = (tiles + KEY_BLOCKS - 1) / KEY_BLOCKS;
    if (r.tiles_per_run < 1) r.tiles_per_run = 1;
    r.runs = (int)((tiles + r.tiles_per_run - 1) / r.tiles_per_run);
    if (r.runs < 1) r.runs = 1;
    return r;
}

__device__ __forceinline__ int bits_needed(int d) { return d <= 0 ? 1 : 32 - __clz((unsigned int)d); }

// Exclusive sum over the 256 threads of the block; `total` = the block's sum. Two barriers.
template <class T>
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
    T base = 0, all = 0;
#pragma unroll
    for (int w = 0; w < KT / 32; ++w) {
        const T x = part[w];
        if (w < warp) base += x;
        all += x;
    }
    total = all;
    return base + inc - v;
}

// Sum of sums[0, count) by the whole block.
__device__ __forceinline__ unsigned long long sum_before(const unsigned long long* sums, int count, unsigned long long* part) {
    unsigned long long v = 0, total;
    for (int i = threadIdx.x; i < count; i += KT) v += __ldcg(sums + i);
    block_scan(v, part, total);
    return total;
}

// Pass 1: histogram of the delta widths of every run. The last block adds them up, chooses the mode and turns
// the runs' histograms into stream offsets.
__global__ void __launch_bounds__(KT) da_plan_kernel(const int* __restrict__ keys, long long n, long long per_run, KeyWork* __restrict__ wk,
                                                     unsigned long long* done, unsigned long long seq) {
    __shared__ unsigned int s_h[KT / 32][32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s_h[warp][lane] = 0;
    __syncwarp();
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    bool bad = false;
    for (long long i0 = lo; i0 < hi; i0 += 4 * KT) {
        int k[4], p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * KT + threadIdx.x;
            k[u] = i < hi ? keys[i] : 0;
            p[u] = i < hi && i ? keys[i - 1] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + u * KT + threadIdx.x;
            if (i >= hi) continue;
            if (k[u] < p[u] || (k[u] == p[u] && i > 0) || k[u] < 0) bad = true;
            atomicAdd(&s_h[warp][bits_needed((int)((unsigned int)k[u] - (unsigned int)p[u])) & 31], 1u);
        }
    }
    if (bad) atomicOr(&wk->status, 1u);
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned int t = 0;
        for (int w = 0; w < KT / 32; ++w) t += s_h[w][lane];
        wk->hist[blockIdx.x][lane] = t;
        if (t) red_add_gpu(&wk->total[lane], t);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&wk->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int runs = (int)gridDim.x;
    __shared__ double s_prob[32], s_t[2][4];
    __shared__ unsigned int s_mode[2];
    if (warp == 0) {
        s_prob[lane] = __ddiv_rn((double)__ldcg(&wk->total[lane]), (double)(n > 0 ? n : 1));
        __syncwarp();
        // the reference's estimates in the same double arithmetic, operation by operation (explicit
        // round-to-nearest intrinsics keep the compiler from fusing multiply-adds), one lane per interval count
        if (lane < 4) {
            const int m = 2 << lane, b = 32 / m;
            double sum = 0.0;
            for (int i = 0; i < m; ++i) {
                double ip = 0.0;
                for (int j = 0; j < b; ++j) ip = __dadd_rn(ip, s_prob[i * b + j]);
                sum = __dadd_rn(sum, __dmul_rn((double)(i + 1), ip));
            }
            s_t[0][lane] = __dadd_rn(__dmul_rn(sum, (double)b), (double)(lane + 1));
            s_t[1][lane] = __dadd_rn(__dmul_rn(sum, (double)(b + 1)), 1.0);
        }
        __syncwarp();
        if (lane == 0) {
            double best = 32.0;
            unsigned int num = 1, kind = 0;
            for (int q = 0; q < 4; ++q)
                for (unsigned int k = 0; k < 2; ++k)
                    if (s_t[k][q] < best) {
                        best = s_t[k][q];
                        num = 2u << q;
                        kind = k;
                    }
            s_mode[0] = wk->m = num;
            s_mode[1] = wk->kind = kind;
        }
    }
    __syncthreads();
    const unsigned int m = s_mode[0], kind = s_mode[1], b = 32u / m, lb = 31u - (unsigned int)__clz(b), fb = 5u - lb;   // powers of two
    // bits of the streams up to every run
    __shared__ unsigned long long s_part[KT / 32];
    unsigned long long base_f = 0, base_d = 0;
    for (int r0 = 0; r0 < runs; r0 += KT) {
        const int r = r0 + (int)threadIdx.x;
        unsigned long long f = 0, d = 0;
        if (r < runs) {
            uint4 h[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) h[q] = ld_cg_v4(reinterpret_cast<const uint4*>(wk->hist[r]) + q);
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const unsigned int k = 4u * q + c, cnt = c == 0 ? h[q].x : (c == 1 ? h[q].y : (c == 2 ? h[q].z : h[q].w));
                    const unsigned int iv = ((k ? k : 32u) + b - 1) >> lb;
                    f += (unsigned long long)cnt * (kind ? iv + 1 : fb);
                    d += (unsigned long long)cnt * (b * iv);
                }
        }
        unsigned long long tf, td;
        const unsigned long long ef = block_scan(f, s_part, tf), ed = block_scan(d, s_part, td);
        if (r < runs) {
            wk->flag_off[r] = base_f + ef;
            wk->delta_off[r] = base_d + ed;
        }
        base_f += tf;
        base_d += td;
    }
    if (threadIdx.x == 0) {
        done[1] = (unsigned long long)m | ((unsigned long long)kind << 32);
        done[2] = base_f;
        done[3] = base_d;
        __threadfence_system();
        skml_store_done(done, seq, &wk->status);
    }
}

// Writes `nb` (<= 32) bits of `value`, most significant first, at bit `off` of a zeroed shared-memory word array.
__device__ __forceinline__ void put_bits(unsigned int* words, unsigned int off, unsigned int value, unsigned int nb) {
    if (nb == 0) return;
    const unsigned int rv = __brev(value) >> (32u - nb);  // stream order: bit j of rv is stream bit off + j
    const unsigned int sh = off & 31u, w = off >> 5;
    atomicOr(&words[w], rv << sh);
    if (sh + nb > 32u) atomicOr(&words[w + 1], rv >> (32u - sh));
}

// One tile's bits from shared memory to the stream: whole words are stored, the first and last may be shared
// with the neighbouring tiles and are completed with atomic ORs (the streams start from zero).
__device__ __forceinline__ void flush_bits(unsigned int* words, const unsigned int* stage, unsigned long long start, unsigned int nbits) {
    if (nbits == 0) return;
    const unsigned int sh = (unsigned int)(start & 31ull), nw = (sh + nbits + 31u) >> 5;
    unsigned int* dst = words + (start >> 5);
    for (unsigned int w = threadIdx.x; w < nw; w += KT) {
        const unsigned int v = stage[w];
        if ((w == 0 && sh != 0) || (w == nw - 1 && ((sh + nbits) & 31u) != 0)) {
            if (v) atomicOr(dst + w, v);
        } else {
            dst[w] = v;
        }
    }
}

// Pass 2: the two streams.
__global__ void __launch_bounds__(KT) da_pack_kernel(const int* __restrict__ keys, long long n, long long per_run, const KeyWork* __restrict__ wk,
                                                     unsigned int* flag_words, unsigned int* delta_words) {
    __shared__ unsigned int s_f[STAGE_F], s_d[STAGE_D], s_part[KT / 32];
    const unsigned int m = wk->m, kind = wk->kind, b = 32u / m, fb = 31u - (unsigned int)__clz(m);
    unsigned long long fs = wk->flag_off[blockIdx.x], ds = wk->delta_off[blockIdx.x];
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    for (long long t0 = lo; t0 < hi; t0 += KEY_TILE) {
        const long long i0 = t0 + 4 * threadIdx.x;
        int prev = i0 > 0 && i0 < hi ? keys[i0 - 1] : 0;
        unsigned int d[4], fv[4], fw[4], dw[4], packed = 0;   // flag bits (<= 17408 a tile) low, delta bits (<= 32768) high
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            d[u] = fv[u] = fw[u] = dw[u] = 0;
            if (i0 + u < hi) {
                const int k = keys[i0 + u];
                d[u] = (unsigned int)k - (unsigned int)prev;
                prev = k;
                const unsigned int iv = ((unsigned int)bits_needed((int)d[u]) + b - 1) / b;
                fw[u] = kind ? iv + 1 : fb;
                fv[u] = kind ? (1u << (iv + 1)) - 2u : iv - 1;
                dw[u] = b * iv;
                packed += fw[u] + (dw[u] << 16);
            }
        }
        for (int i = threadIdx.x; i < STAGE_F; i += KT) s_f[i] = 0;
        for (int i = threadIdx.x; i < STAGE_D; i += KT) s_d[i] = 0;
        unsigned int total;
        const unsigned int ex = block_scan(packed, s_part, total);   // its barriers also publish the cleared words
        unsigned int fo = (unsigned int)(fs & 31ull) + (ex & 0xFFFFu), dof = (unsigned int)(ds & 31ull) + (ex >> 16);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            put_bits(s_f, fo, fv[u], fw[u]);
            put_bits(s_d, dof, d[u], dw[u]);
            fo += fw[u];
            dof += dw[u];
        }
        __syncthreads();
        flush_bits(flag_words, s_f, fs, total & 0xFFFFu);
        flush_bits(delta_words, s_d, ds, total >> 16);
        fs += total & 0xFFFFu;
        ds += total >> 16;
        __syncthreads();   // the staging words are cleared again by the next tile
    }
}

struct Streams {
    const unsigned int* flag_words;
    const unsigned int* delta_words;
    long long flag_lim, delta_lim;    // 32-bit words
    const long long* zero_pos;        // unary flags: where every key's flag ends
    unsigned int m;
    int unary;
};

// Interval counts of keys i0..i0+3 (0 beyond `hi`).
__device__ __forceinline__ void intervals(const Streams& s, long long i0, long long hi, unsigned int (&iv)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) iv[u] = 0;
    if (i0 >= hi) return;
    if (s.unary) {
        long long before = i0 ? s.zero_pos[i0 - 1] : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u < hi) {
                const long long z = s.zero_pos[i0 + u];
                iv[u] = (unsigned int)(z - before - 1);
                before = z;
            }
        return;
    }
    const unsigned int fb = 31u - (unsigned int)__clz(s.m);
    unsigned long long win = 0;
    if (fb) {
        const unsigned long long off = (unsigned long long)i0 * fb;
        const long long w = (long long)(off >> 5);
        const unsigned int lo = w < s.flag_lim ? s.flag_words[w] : 0u, hw = w + 1 < s.flag_lim ? s.flag_words[w + 1] : 0u;
        win = ((unsigned long long)lo | ((unsigned long long)hw << 32)) >> (off & 31ull);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (i0 + u < hi) {
            const unsigned int bits = fb ? (unsigned int)(win >> (fb * u)) & ((1u << fb) - 1u) : 0u;
            iv[u] = (fb ? __brev(bits) >> (32u - fb) : 0u) + 1u;
        }
}

// Unary flags: zero bits of every run of flag words (a key's flag ends at its zero bit).
__global__ void __launch_bounds__(KT) da_zero_count_kernel(const unsigned int* __restrict__ flag_words, long long flag_bits, long long per_run,
                                                           KeyWork* __restrict__ wk) {
    __shared__ unsigned long long s_part[KT / 32];
    const long long nw = (flag_bits + 31) >> 5, lo = per_run * blockIdx.x, hi = lo + per_run < nw ? lo + per_run : nw;
    unsigned long long v = 0, total;
    for (long long w = lo + threadIdx.x; w < hi; w += KT) {
        const long long rest = flag_bits - (w << 5);
        v += __popc(~flag_words[w] & (rest >= 32 ? 0xFFFFFFFFu : ((1u << rest) - 1u)));
    }
    block_scan(v, s_part, total);
    if (threadIdx.x == 0) wk->run_a[blockIdx.x] = total;
}

// Stream position of the i-th zero bit.
__global__ void __launch_bounds__(KT) da_zero_pos_kernel(const unsigned int* __restrict__ flag_words, long long flag_bits, long long per_run,
                                                         const KeyWork* __restrict__ wk, long long n, long long* __restrict__ pos) {
    __shared__ unsigned long long s_part[KT / 32];
    const long long nw = (flag_bits + 31) >> 5, lo = per_run * blockIdx.x, hi = lo + per_run < nw ? lo + per_run : nw;
    unsigned long long base = sum_before(wk->run_a, blockIdx.x, s_part);
    for (long long w0 = lo; w0 < hi; w0 += KT) {
        const long long w = w0 + threadIdx.x;
        unsigned int z = 0;
        if (w < hi) {
            const long long rest = flag_bits - (w << 5);
            z = ~flag_words[w] & (rest >= 32 ? 0xFFFFFFFFu : ((1u << rest) - 1u));
        }
        unsigned long long total;
        unsigned long long idx = base + block_scan((unsigned long long)__popc(z), s_part, total);
        while (z) {
            const int bit = __ffs(z) - 1;
            z &= z - 1;
            if (idx < (unsigned long long)n) pos[idx] = (w << 5) + bit;
            ++idx;
        }
        base += total;
    }
}

// Delta bits of every run.
__global__ void __launch_bounds__(KT) da_width_kernel(Streams s, long long n, long long per_run, KeyWork* __restrict__ wk) {
    __shared__ unsigned long long s_part[KT / 32];
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    unsigned long long v = 0, total;
    for (long long t0 = lo; t0 < hi; t0 += KEY_TILE) {
        unsigned int iv[4];
        intervals(s, t0 + 4 * threadIdx.x, hi, iv);
        v += (iv[0] + iv[1] + iv[2] + iv[3]) * (32u / s.m);
    }
    block_scan(v, s_part, total);
    if (threadIdx.x == 0) wk->run_a[blockIdx.x] = total;
}

// Keys of every run counted from the key before it, and the runs' sums.
__global__ void __launch_bounds__(KT) da_extract_kernel(Streams s, long long n, long long per_run, KeyWork* __restrict__ wk, int* __restrict__ keys) {
    __shared__ unsigned long long s_part[KT / 32];
    __shared__ unsigned int s_part32[KT / 32];
    const unsigned int b = 32u / s.m;
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    unsigned long long bit = sum_before(wk->run_a, blockIdx.x, s_part), sum = 0;
    for (long long t0 = lo; t0 < hi; t0 += KEY_TILE) {
        const long long i0 = t0 + 4 * threadIdx.x;
        unsigned int iv[4];
        intervals(s, i0, hi, iv);
        unsigned int total;
        unsigned long long off = bit + block_scan((iv[0] + iv[1] + iv[2] + iv[3]) * b, s_part32, total);
        bit += total;
        unsigned int d[4], dsum = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned int dw = b * iv[u];
            d[u] = 0;
            if (dw && dw <= 32u) {
                const long long w = (long long)(off >> 5);
                const unsigned int x0 = w < s.delta_lim ? s.delta_words[w] : 0u, x1 = w + 1 < s.delta_lim ? s.delta_words[w + 1] : 0u;
                d[u] = __brev(__funnelshift_r(x0, x1, (unsigned int)(off & 31ull)) << (32u - dw));
            }
            off += dw;
            dsum += d[u];
        }
        unsigned int tile_sum;
        unsigned int key = (unsigned int)sum + block_scan(dsum, s_part32, tile_sum);   // keys are below 2^31: 32-bit sums are exact
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            key += d[u];
            if (i0 + u < hi) keys[i0 + u] = (int)key;
        }
        sum += tile_sum;
    }
    if (threadIdx.x == 0) wk->run_b[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(KT) da_offset_kernel(long long n, long long per_run, const KeyWork* __restrict__ wk, int* __restrict__ keys) {
    __shared__ unsigned long long s_part[KT / 32];
    if (blockIdx.x == 0) return;
    const long long lo = per_run * blockIdx.x, hi = lo + per_run < n ? lo + per_run : n;
    const int add = (int)sum_before(wk->run_b, blockIdx.x, s_part);
    for (long long i = lo + threadIdx.x; i < hi; i += KT) keys[i] += add;
}

}  // namespace

extern "C" long long skml_da_workspace_bytes() { return (long long)sizeof(KeyWork); }

extern "C" int skml_da_plan(const int* keys, long long n, void* workspace, unsigned long long* done, unsigned int* status_out, void* stream) {
    if (n < 0 || !workspace || !done || !status_out) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    KeyWork* wk = reinterpret_cast<KeyWork*>(workspace);
    cudaError_t e = cudaMemsetAsync(wk, 0, offsetof(KeyWork, flag_off), s);
    if (e != cudaSuccess) return (int)e;
    const Runs r = runs_for(n);
    const unsigned long long seq = ((*done >> 32) + 1) & 0xFFFFFFFFull;
    da_plan_kernel<<<r.runs, KT, 0, s>>>(keys, n, r.tiles_per_run * KEY_TILE, wk, done, seq);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    return skml_wait_done(done, seq, &wk->status, status_out, s);
}

extern "C" int skml_da_pack(const int* keys, long long n, const void* workspace, unsigned long long* flag_words, long long n_flag_words,
                            unsigned long long* delta_words, long long n_delta_words, void* stream) {
    if (n <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
    if (delta_words == flag_words + n_flag_words) {   // one allocation: one fill
        e = cudaMemsetAsync(flag_words, 0, 8 * (size_t)(n_flag_words + n_delta_words), s);
    } else {
        if (n_flag_words) e = cudaMemsetAsync(flag_words, 0, 8 * (size_t)n_flag_words, s);
        if (e == cudaSuccess && n_delta_words) e = cudaMemsetAsync(delta_words, 0, 8 * (size_t)n_delta_words, s);
    }
    if (e != cudaSuccess) return (int)e;
    const Runs r = runs_for(n);
    da_pack_kernel<<<r.runs, KT, 0, s>>>(keys, n, r.tiles_per_run * KEY_TILE, reinterpret_cast<const KeyWork*>(workspace),
                                         reinterpret_cast<unsigned int*>(flag_words), reinterpret_cast<unsigned int*>(delta_words));
    return (int)cudaGetLastError();
}

extern "C" int skml_da_decode(const unsigned long long* flag_words, long long n_flag_words, const unsigned long long* delta_words,
                              long long n_delta_words, long long n, int num_intervals, int unary, long long flag_bits, void* workspace,
                              long long* zero_pos, int* keys, void* stream) {
    if (num_intervals < 1 || num_intervals > 16 || (num_intervals & (num_intervals - 1)) || !workspace || (unary && !zero_pos))
        return (int)cudaErrorInvalidValue;
    if (n <= 0) return 0;
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
        const Runs f = runs_for(nw);
        da_zero_count_kernel<<<f.runs, KT, 0, s>>>(st.flag_words, flag_bits, f.tiles_per_run * KEY_TILE, wk);
        da_zero_pos_kernel<<<f.runs, KT, 0, s>>>(st.flag_words, flag_bits, f.tiles_per_run * KEY_TILE, wk, n, zero_pos);
    }
    const Runs r = runs_for(n);
    const long long per = r.tiles_per_run * KEY_TILE;
    da_width_kernel<<<r.runs, KT, 0, s>>>(st, n, per, wk);
    da_extract_kernel<<<r.runs, KT, 0, s>>>(st, n, per, wk, keys);
    if (r.runs > 1) da_offset_kernel<<<r.runs, KT, 0, s>>>(n, per, wk, keys);
    return (int)cudaGetLastError();
}
