// Device-side building blocks shared by all sm_100a kernels of this library:
// status words, bounded waits (grid barrier, flag wait), order-preserving float keys,
// sorts and searches in shared memory, the end of a checked call, and system-scope
// loads/stores used on peer-mapped memory.
//
// Every wait in this file has a clock64() budget. When it runs out the kernel
// records a status word and returns normally, so the CUDA context stays usable.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "skml_common.h"

#define SKML_BLOCK 1024
#define SKML_WARPS (SKML_BLOCK / 32)

// The kernels of a step follow one another on one stream. Launched by skml_launch (programmatic stream serialization) a
// kernel is set up while the one before it ends, and waits here, before it touches memory, until that one has completed
// and its stores are visible: 2 us between kernels became about 1 (an epoch of ten small steps 1058 -> 993 us). Every kernel
// launched that way calls this first. No kernel lets the next one start early: what a block would do before it waits is
// nothing, and the blocks would take the place of others.
__device__ __forceinline__ void skml_after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
static inline cudaError_t skml_launch_as(bool cooperative, void (*kernel)(P...), unsigned int grid, unsigned int block, size_t smem,
                                         cudaStream_t stream, A... args) {
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeCooperative;
    attrs[1].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attrs;
    cfg.numAttrs = cooperative ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
static inline cudaError_t skml_launch(void (*kernel)(P...), unsigned int grid, unsigned int block, size_t smem, cudaStream_t stream, A... args) {
    return skml_launch_as(false, kernel, grid, block, smem, stream, args...);
}

enum SkmlStatus {
    SKML_OK = 0,
    SKML_TIMEOUT_BARRIER = 1,
    SKML_TIMEOUT_PEER = 2,
    SKML_BAD_HEADER = 3,
    SKML_CAPACITY = 4,
    SKML_BAD_INPUT = 5,
};

// status word: low 8 bits = code, bits 8..31 = detail (stage, peer, ...). First error wins.
__device__ __forceinline__ void skml_set_status(unsigned int* status, unsigned int code, unsigned int detail) {
    atomicCAS(status, 0u, code | (detail << 8));
}

// Whether an earlier launch has reported an error (null: nobody asks).
__device__ __forceinline__ bool skml_failed(const unsigned int* status) { return status && (*status & 0xFFu) != SKML_OK; }

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_sys(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_sys(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint4 ld_cg_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_v4(uint4* p, uint4 v) {
    asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ---------------------------------------------------------------------------
// Table positions of one key for sketches whose rows all use the three integer mixers (BJ, Mix64,
// TW: what skml_pick_hashes draws for up to three rows). Equal to skml_hash(ids[r], key, size) for
// every row and every key, with about a third of the instructions of the general routine: the three
// mixers are computed once and handed to the rows, and `x % size` is a 32-bit reciprocal
// multiplication with one correction step (q = mulhi(x, floor(2^32 / size)) is the quotient or one
// less). Java semantics: the remainder keeps the sign of the dividend and is then moved up by size.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned int skml_recip32(unsigned int size) {
    if (size <= 1u) return 0xFFFFFFFFu;
    const unsigned int q = 0xFFFFFFFFu / size;   // floor(2^32 / size) is one more where size divides 2^32
    return q + (0xFFFFFFFFu - q * size == size - 1u ? 1u : 0u);
}
__device__ __forceinline__ int skml_java_mod(unsigned int code, unsigned int size, unsigned int recip) {
    const bool neg = (int)code < 0;
    const unsigned int a = neg ? 0u - code : code;
    unsigned int r = a - __umulhi(a, recip) * size;
    if (r >= size) r -= size;
    return (int)(neg ? (r ? size - r : 0u) : r);
}
template <int MAXR>
__device__ __forceinline__ void skml_hash_rows_mixers(const unsigned char* ids, int rows, int key, unsigned int size,
                                                      unsigned int recip, int* out) {
    const unsigned int h0 = skml_mix_bj((unsigned int)key), h1 = skml_mix_64((unsigned int)key), h2 = skml_mix_tw((unsigned int)key);
#pragma unroll
    for (int r = 0; r < MAXR; ++r) {
        if (r >= rows) continue;
        const int id = ids[r];
        out[r] = skml_java_mod(id == 0 ? h0 : (id == 1 ? h1 : h2), size, recip);
    }
}

// ---------------------------------------------------------------------------
// Grid barrier for cooperative launches. *bar counts arrivals: zero when the kernel starts, nblocks more
// per barrier, and put back to zero by the kernel's last block. `passed` is the caller's count of arrivals
// of the barriers before this one. A block adds itself and polls until everyone has: one trip to L2 and
// one poll, no second word for the last block to release. The status word is polled beside the count, in
// the same flight: a block that reported an error may have left the kernel and will never arrive, and
// nobody goes on after an error.
// Returns false (on every thread of the block) when the wait budget ran out or an error was reported; the
// host then clears the workspace.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned int ld_relaxed_gpu(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu(unsigned int* p, unsigned int v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_gpu64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void red_add_gpu(unsigned int* p, unsigned int v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

static __device__ __noinline__ bool skml_grid_barrier_at(unsigned int* bar, unsigned int nblocks, unsigned int* status,
                                                         long long budget, unsigned int stage, unsigned int target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned int st;
        if (nblocks > 1) {
            __threadfence();
            red_add_gpu(bar, 1u);
            const long long t0 = clock64();
            unsigned int ns = 0;
            while (true) {
                const unsigned int now = ld_relaxed_gpu(bar);
                st = ld_relaxed_gpu(status);
                if (now >= target || (st & 0xFFu) != SKML_OK) break;
                if (clock64() - t0 > budget) {
                    skml_set_status(status, SKML_TIMEOUT_BARRIER, stage);
                    ok = 0;
                    break;
                }
                if (ns) __nanosleep(ns);
                if (ns < 200) ns += 10;
            }
            __threadfence();
        } else {
            st = ld_relaxed_gpu(status);
        }
        s_ok = ok && (st & 0xFFu) == SKML_OK;
    }
    __syncthreads();
    return s_ok != 0;
}
__device__ __forceinline__ bool skml_grid_barrier(unsigned int* bar, unsigned int nblocks, unsigned int* status,
                                                  long long budget, unsigned int stage, unsigned int& passed) {
    passed += nblocks;
    return skml_grid_barrier_at(bar, nblocks, status, budget, stage, passed);
}

// Waits until *flag == want (system scope). Thread 0 of the block polls.
__device__ __forceinline__ bool skml_wait_flag(const unsigned long long* flag, unsigned long long want,
                                               unsigned int* status, long long budget, unsigned int detail) {
    long long t0 = clock64();
    unsigned int ns = 32;
    while (ld_acquire_sys(flag) != want) {
        if (clock64() - t0 > budget) {
            skml_set_status(status, SKML_TIMEOUT_PEER, detail);
            return false;
        }
        __nanosleep(ns);
        if (ns < 1000) ns *= 2;
    }
    return true;
}

// ---------------------------------------------------------------------------
// Order-preserving map float -> uint32 (ascending floats give ascending keys).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned int f2ord(float f) {
    unsigned int b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned int k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Block sum of doubles; the result is valid on thread 0.
__device__ __forceinline__ double block_sum_double(double v) {
    __shared__ double s_part[SKML_WARPS];
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0;
    if (threadIdx.x < 32) {
        r = threadIdx.x < (blockDim.x >> 5) ? s_part[threadIdx.x] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

// ---------------------------------------------------------------------------
// One merge round of sorted runs of LEN keys: an element's place in the merged pair of runs is its place in
// its own run plus the number of the other run's keys before it (a binary search; the left run wins ties).
// A warp's 64 elements belong to one run, so its 32 searches run side by side on neighbouring keys.
// `remote`: where another block of the cluster takes a copy (shared::cluster address; 0: none).
template <int LEN>
__device__ __forceinline__ void merge_round(const unsigned int* __restrict__ src, unsigned int* __restrict__ dst, unsigned int remote = 0) {
    const int lane = threadIdx.x & 31, i0 = (threadIdx.x >> 5) * 64 + lane;
    const int run = i0 / LEN;
    const unsigned int* other = src + (run ^ 1) * LEN;
    const unsigned int x0 = src[i0], x1 = src[i0 + 32];
    int p0 = 0, p1 = 0;
    if (run & 1) {   // uniform over the warp
#pragma unroll
        for (int step = LEN / 2; step > 0; step >>= 1) {
            if (other[p0 + step - 1] <= x0) p0 += step;
            if (other[p1 + step - 1] <= x1) p1 += step;
        }
        p0 += other[p0] <= x0;
        p1 += other[p1] <= x1;
    } else {
#pragma unroll
        for (int step = LEN / 2; step > 0; step >>= 1) {
            if (other[p0 + step - 1] < x0) p0 += step;
            if (other[p1 + step - 1] < x1) p1 += step;
        }
        p0 += other[p0] < x0;
        p1 += other[p1] < x1;
    }
    const int base = (run & ~1) * LEN + (i0 & (LEN - 1));
    dst[base + p0] = x0;
    dst[base + 32 + p1] = x1;
    if (remote) {
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote + 4u * (unsigned int)(base + p0)), "r"(x0) : "memory");
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote + 4u * (unsigned int)(base + 32 + p1)), "r"(x1) : "memory");
    }
    __syncthreads();
}

// Ascending order of 256 keys by one warp, eight adjacent ones a lane: a bitonic network whose steps of distance 8 and more
// are shuffles. Keys of descending stretches are inverted, so that every comparison is a minimum and a maximum.
__device__ __forceinline__ void warp_sort_256(unsigned int (&a)[8]) {
    const unsigned int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 256; k <<= 1) {
        if (k >= 8) {   // stretches of k keys: whole lanes from here on
            const unsigned int now = k < 256 && (lane & (k / 8)) ? 0xFFFFFFFFu : 0u, before = k > 8 && (lane & (k / 16)) ? 0xFFFFFFFFu : 0u;
#pragma unroll
            for (int e = 0; e < 8; ++e) a[e] ^= now ^ before;
        }
#pragma unroll
        for (int j = k / 2; j >= 8; j >>= 1) {
            const bool upper = (lane & (j / 8)) != 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned int o = __shfl_xor_sync(0xFFFFFFFFu, a[e], j / 8);
                a[e] = upper ? max(a[e], o) : min(a[e], o);
            }
        }
#pragma unroll
        for (int j = k / 2 < 4 ? k / 2 : 4; j > 0; j >>= 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (e & j) continue;
                const bool down = k < 8 && (e & k);   // (inside a lane)
                const unsigned int x = a[e], y = a[e + j];
                a[e] = down ? max(x, y) : min(x, y);
                a[e + j] = down ? min(x, y) : max(x, y);
            }
        }
    }
}

// Ascending sort of 2048 unsigned keys in shared memory (16-byte aligned) by a block of 1024 threads, `tmp` a second array of
// that size. Eight warps sort 256 keys each in registers, three merge rounds by binary search follow with one block barrier each.
// What bounds it is the chain of dependent steps, and shared memory's passes in the merge rounds. In every block of a compress
// launch, with its result sent to the other block instead of fetched: 10,000 keys 35.0 -> 33.8 us, 170,000 with coded tables
// 67.5 -> 65.7, against 32 warps of 64 keys and five merge rounds.
// `remote`: a copy of the result in another block of the cluster (see merge_round), complete behind a cluster barrier.
__device__ __forceinline__ void block_sort_2048(unsigned int* s, unsigned int* tmp, unsigned int remote = 0) {
    if (threadIdx.x < 256) {
        uint4* const at = reinterpret_cast<uint4*>(s) + 2 * threadIdx.x;
        const uint4 x = at[0], y = at[1];
        unsigned int a[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        warp_sort_256(a);
        uint4* const to = reinterpret_cast<uint4*>(tmp) + 2 * threadIdx.x;
        to[0] = make_uint4(a[0], a[1], a[2], a[3]);
        to[1] = make_uint4(a[4], a[5], a[6], a[7]);
    }
    __syncthreads();
    merge_round<256>(tmp, s);
    merge_round<512>(s, tmp);
    merge_round<1024>(tmp, s, remote);
}

// Upper bounds of K values side by side in an ascending array of n floats: element i lies at a[i + i / 32], and
// NaNs (below nothing) fill up to 2 top - 1 elements, top = search_top(n). The elements a halving step may read
// are powers of two apart, in two or four banks of a plain array (37 passes of shared memory per warp at 255
// elements, half of what bounded S3); with the gaps they lie in different banks.
__device__ __forceinline__ int search_top(int n) { return n > 255 ? 1 << (31 - __clz(n)) : 128; }
__device__ __forceinline__ int search_slot(int i) { return i + (i >> 5); }
template <int K>
__device__ __forceinline__ void upper_bounds_f(const float* a, int top, const float (&x)[K], int (&pos)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) pos[k] = 0;   // search_slot of the position so far
    for (int step = top; step > 128; step >>= 1) {
        const int inc = search_slot(step);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (a[pos[k] + inc - 2] <= x[k]) pos[k] += inc;
    }
#pragma unroll
    for (int step = 128; step > 0; step >>= 1) {
        const int inc = search_slot(step), at = step >= 32 ? inc - 2 : inc - 1;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (a[pos[k] + at] <= x[k]) pos[k] += inc;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) pos[k] -= pos[k] / 33;
}

// Number of elements of the ascending array a[0..n) that are <= x (upper bound).
__device__ __forceinline__ int upper_bound_u(const unsigned int* a, int n, unsigned int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ int lower_bound_u(const unsigned int* a, int n, unsigned int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// Checked calls: the kernel's last block stores (sequence number, status word) into a pinned host word and
// the caller polls that word, instead of a device-to-host copy and a stream synchronisation (15 us and more
// on top of a 35 us kernel). A kernel that reported an error may end without the store: the stream is
// queried now and then, and once it has drained the status word is read the plain way.
// The caller goes on while the kernel's blocks are still leaving, so every block fences after its last store and
// before it counts itself, and the last one fences after it has counted and before it reads the status here: whoever
// has seen the word sees every block's outputs, on any stream.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void skml_store_done(unsigned long long* word, unsigned long long seq, const unsigned int* status) {
    if (word) st_release_sys(word, (seq << 32) | ld_relaxed_gpu(status));
}

static inline int skml_wait_done(volatile unsigned long long* word, unsigned long long seq, const unsigned int* status,
                                 unsigned int* status_out, cudaStream_t stream) {
    for (unsigned long long spins = 1;; ++spins) {
        const unsigned long long v = *word;
        if ((v >> 32) == (seq & 0xFFFFFFFFull)) {
            __atomic_thread_fence(__ATOMIC_ACQUIRE);   // what the kernel left beside the word is read after it
            *status_out = (unsigned int)v;
            return 0;
        }
        if ((spins & 0x3FFF) == 0) {
            const cudaError_t q = cudaStreamQuery(stream);
            if (q == cudaErrorNotReady) continue;
            if (q != cudaSuccess) return (int)q;
            if ((*word >> 32) == (seq & 0xFFFFFFFFull)) continue;
            cudaError_t e = cudaMemcpyAsync(status_out, status, sizeof(unsigned int), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            return (int)e;
        }
    }
}
