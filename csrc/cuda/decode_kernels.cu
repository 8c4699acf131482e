// Fused decode + aggregate + update for sm_100a: the receiving side of the gradient
// exchange in one persistent cooperative kernel.
//   D0  bounded wait for the arrival flags of all ranks' payloads (written by the peers'
//       compress kernels straight into this GPU's memory), header validation, work table
//   D1  per 1024-key chunk (restart points make chunks independent): flag bits -> delta
//       widths -> scan -> gather -> prefix sum = keys; grouped MinMaxSketch query
//       (furthest-from-zero over the rows); dequantize
//   Replicas must end bit-identical, so the order of the float adds per coordinate is fixed:
//   * one payload: keys are unique inside it, every value is applied by the thread that
//     decoded it (SGD step, lazy Adam step, or plain sum);
//   * several short payloads: D1 stashes (key, value) pairs; after one grid barrier every
//     block owns a key range (quantiles of the longest key list), finds its slice of every
//     (rank, group) list by binary search and applies the slices rank by rank with block
//     barriers only. Lazy Adam first sums the ranks' values per coordinate (plain floats in
//     the zeroed accumulator array), then the first rank holding the coordinate applies the
//     moment update and clears the sum;
//   * several long payloads (SGD): one decode-and-apply pass per rank, grid barrier in between;
//   * a dense-kind payload among them: per-rank passes for SGD; for Adam 64-bit fixed-point
//     accumulators (integer adds commute) and a claim pass (atomic exchange with zero).
//
// Reference behaviour restated (paths inside the reference project):
//   sketch/.../binary/DeltaBinaryEncoder.java:42-53 (key decode),
//   sketch/.../sketch/frequency/MinMaxSketch.java:64-73, GroupedMinMaxSketch.java:123-146,
//   ml/.../gradient/SketchGradient.scala:57-68, Gradient.scala:44-49 (sum over workers),
//   ml/.../algorithm/GeneralizedLinearModel.scala:150 (1/workerNum),
//   ml/.../objective/GradientDescent.scala:89-117, Adam.scala:27-77 (updates).
#include "decode_common.cuh"

// The header fields that are needed after the work table is built.
struct HdrLite {
    unsigned int kind, cell_bits, bin_num, zero_idx;
    unsigned long long off_dense_codes, off_bucket_values;
    double loss_partials[4];
};

struct DecSmem {
    HdrLite hdr[SKML_MAX_PEERS];
    int nitems;
    unsigned long long total_chunks, total_keys;
    int any_dense;
    unsigned long long rank_key_begin[SKML_MAX_PEERS + 1];
    int rank_item_begin[SKML_MAX_PEERS + 1];
    int ref_item;    // the (rank, group) list with the most keys: its quantiles are the blocks' key-range bounds
    int small_passes;   // a pass per payload would leave most blocks with one chunk or none
    int shift;       // fixed-point: accumulator = value * 2^shift
    double inv_world;
    int ok;
    int max_items;
    int nhuf;        // items whose table arrives Huffman-coded
    DecItem items[1];  // max_items entries (dynamic shared memory)
};

// How the payloads are applied.
struct DecForm {
    bool direct;       // linear update (SGD / plain sum): payloads applied in rank order, no accumulators
    bool adam_plain;   // Adam without fixed-point accumulators (no dense payload, and one payload or a value scratch)
    bool two_phase;    // several payloads: decode everything first, then ordered apply
};
// Several payloads are decoded into the scratch first and applied by key range when a per-rank
// pass would leave most blocks with one chunk or none (the pass latency then dominates). Long
// payloads keep the blocks busy in per-rank passes and skip the scratch round trip; Adam has no
// per-rank mode, so it always takes the scratch.
__device__ __forceinline__ DecForm decode_form(const DP& p, const DecSmem& s) {
    DecForm f;
    f.direct = p.adam_v == nullptr;
    f.adam_plain = !f.direct && !s.any_dense && (p.world == 1 || p.val_scratch != nullptr);
    f.two_phase = (f.direct || f.adam_plain) && p.world > 1 && p.val_scratch != nullptr && (s.small_passes || f.adam_plain);
    return f;
}

// D0: wait, validate, build the work table (identically in every block).
__device__ bool decode_prepare(const DP& p, DecSmem& s) {
    // the full headers sit in the (still idle) table staging area while the work table is built
    SkmlHeader* full = reinterpret_cast<SkmlHeader*>(reinterpret_cast<unsigned char*>(&s) + p.tab_off);
    if (threadIdx.x == 0) s.ok = 1;
    __syncthreads();
    // one thread per rank polls that rank's arrival flag (bounded), so the waits overlap
    if (threadIdx.x < p.world && p.flag[threadIdx.x] &&
        !skml_wait_flag(p.flag[threadIdx.x], p.step + 1, p.status, p.budget, (unsigned int)threadIdx.x))
        s.ok = 0;
    __syncthreads();
    if (!s.ok) return false;
    // headers -> shared memory (L2 loads: the bytes were written by other GPUs)
    for (int t = threadIdx.x; t < p.world * (SKML_HEADER_BYTES / 16); t += blockDim.x) {
        int r = t / (SKML_HEADER_BYTES / 16), i = t % (SKML_HEADER_BYTES / 16);
        reinterpret_cast<uint4*>(&full[r])[i] = ld_cg_v4(reinterpret_cast<const uint4*>(p.payload[r]) + i);
    }
    __syncthreads();
    bool bad = false;
    if (threadIdx.x < p.world) {
        const SkmlHeader& h = full[threadIdx.x];
        bool good = h.magic == SKML_MAGIC && h.version == SKML_VERSION && h.header_checksum == skml_header_checksum(&h) &&
                    h.step == p.step && h.rank == (unsigned int)threadIdx.x && h.dim == (unsigned long long)p.dim &&
                    h.total_bytes <= (unsigned long long)p.slot_capacity && h.dtype == SKML_F32 &&
                    h.group_num <= SKML_MAX_GROUPS && h.row_num <= SKML_MAX_ROWS && h.kind <= SKML_KIND_DENSE &&
                    (h.kind != SKML_KIND_SPARSE || ((h.off_group_table & 15ull) == 0 &&
                                                    h.off_group_table + sizeof(SkmlGroupEntry) * h.group_num <= h.total_bytes)) &&
                    (h.kind == SKML_KIND_EMPTY || (h.bin_num >= 1 && h.bin_num <= SKML_GPU_MAX_BINS && h.zero_idx < h.bin_num)) &&
                    (h.kind != SKML_KIND_SPARSE || ((h.key_encoder == SKML_KEYS_DELTA_BINARY || h.key_encoder == SKML_KEYS_DELTA_ADAPTIVE) &&
                                                    h.restart_interval == SKML_RESTART_INTERVAL &&
                                                    (h.cell_bits == 8 || h.cell_bits == 16 || (h.cell_bits == 0 && p.tab_scratch))));
        if (!good) {
            skml_set_status(p.status, SKML_BAD_HEADER, (unsigned int)threadIdx.x);
            bad = true;
        }
        HdrLite& l = s.hdr[threadIdx.x];
        l.kind = h.kind;
        l.cell_bits = h.cell_bits;
        l.bin_num = h.bin_num;
        l.zero_idx = h.zero_idx;
        l.off_dense_codes = h.off_dense_codes;
        l.off_bucket_values = h.off_bucket_values;
        for (int i = 0; i < 4; ++i) l.loss_partials[i] = h.loss_partials[i];
    }
    // group entries: one thread per (rank, group) fetches its 64-byte entry (independent loads), while the first warp is
    // still checking the headers: only the offsets the fetch itself needs are looked at first
    const int gcap = p.max_items / p.world;
    for (int t = (threadIdx.x + DEC_THREADS - 32) % DEC_THREADS; t < p.world * gcap; t += DEC_THREADS) {
        const int r = t / gcap, g = t % gcap;
        const SkmlHeader& h = full[r];
        DecItem& it = s.items[t];
        it.e.n = 0;
        if (h.kind == SKML_KIND_SPARSE && g < (int)h.group_num && h.group_num <= SKML_MAX_GROUPS && (h.off_group_table & 15ull) == 0 &&
            h.off_group_table <= (unsigned long long)p.slot_capacity && h.row_num <= SKML_MAX_ROWS &&
            h.off_group_table + sizeof(SkmlGroupEntry) * h.group_num <= (unsigned long long)p.slot_capacity) {
            const uint4* src = reinterpret_cast<const uint4*>(p.payload[r] + h.off_group_table + g * sizeof(SkmlGroupEntry));
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(&it.e);  // 8-byte aligned in DecItem
#pragma unroll
            for (int q = 0; q < (int)(sizeof(SkmlGroupEntry) / 16); ++q) {
                const uint4 v = ld_cg_v4(src + q);
                dst[2 * q] = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
                dst[2 * q + 1] = (unsigned long long)v.z | ((unsigned long long)v.w << 32);
            }
            if (it.e.n) {
                const unsigned long long lim = h.total_bytes;
                const bool good = it.e.col_num > 0 && (unsigned long long)h.row_num * it.e.col_num < (1ull << 31) &&
                                  it.e.table_off + (h.cell_bits ? (unsigned long long)h.row_num * it.e.col_num * (h.cell_bits / 8) : 16ull) <= lim &&
                                  (it.e.flag_off & 7ull) == 0 && (it.e.restart_off & 15ull) == 0 && it.e.flag_off + 8ull * it.e.n_flag_words <= lim && it.e.delta_off + 8ull * it.e.n_delta_words <= lim &&
                                  it.e.restart_off + 16ull * ((it.e.n + SKML_RESTART_INTERVAL - 1) / SKML_RESTART_INTERVAL) <= lim &&
                                  (h.key_encoder == SKML_KEYS_DELTA_BINARY
                                       ? 2ull * it.e.n <= 64ull * it.e.n_flag_words
                                       : (it.e.flag_kind <= 1u && it.e.num_intervals >= 1u && it.e.num_intervals <= 16u &&
                                          (it.e.num_intervals & (it.e.num_intervals - 1u)) == 0u &&
                                          (it.e.num_intervals > 1u || it.e.flag_kind == 0u)));
                it.enc = h.key_encoder;
                it.base = p.payload[r];
                it.tab = it.base + it.e.table_off;
                it.huffman = h.cell_bits == 0 ? 1u : 0u;
                it.cell_bits = it.huffman ? (h.bin_num <= 256 ? 8u : 16u) : h.cell_bits;  // Huffman: width of the expanded table
                it.zero = h.zero_idx;
                it.rows = h.row_num;
                it.off_bv = h.off_bucket_values;
                it.recip = skml_recip32(it.e.col_num);
                it.mixers = 0;
                if (h.row_num <= 3) {
                    unsigned int seen = 0;
                    it.row_of[0] = it.row_of[1] = it.row_of[2] = 3;
                    for (unsigned int q = 0; q < h.row_num; ++q)
                        if (it.e.hash_ids[q] < 3) {
                            it.row_of[it.e.hash_ids[q]] = (unsigned char)q;
                            seen |= 1u << it.e.hash_ids[q];
                        }
                    it.mixers = __popc(seen) == (int)h.row_num ? 1 : 0;
                }
                it.col_magic = good && !it.mixers ? skml_fastmod_magic(it.e.col_num) : 0ull;   // (a 64-bit division)
                it.chunk_prefix = good ? 0ull : 1ull;  // scratch use until the compaction below: 1 = failed validation
            }
        }
    }
    if (__syncthreads_or(bad)) return false;
    if (threadIdx.x == 32) {   // the per-rank header facts
        int dense = 0, e = 0;
        double mx = 0.0;
        for (int r = 0; r < p.world; ++r) {
            const SkmlHeader& h = full[r];
            if (h.kind == SKML_KIND_EMPTY) continue;
            mx = fmax(mx, fmax(fabs(h.min_value), fabs(h.max_value)));
            if (h.kind == SKML_KIND_DENSE) dense = 1;
            else if ((int)h.group_num > gcap) {
                skml_set_status(p.status, SKML_BAD_HEADER, 0x300u | (unsigned int)r);
                s.ok = 0;
            }
        }
        if (mx > 0.0 && isfinite(mx)) frexp(mx, &e);
        s.shift = 60 - e;
        s.any_dense = dense;
        s.inv_world = 1.0 / (double)p.world;
    }
    // The work table: the non-empty (rank, group) lists moved to the front in (rank, group) order, each
    // with the number of chunks and keys in front of it. Warp 0 does it 32 slots at a time (ballot for the
    // positions, shuffle scans for the prefixes).
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int ni = 0, nhuf = 0;
        unsigned long long chunks = 0, keys = 0, tab_used = 0;
        int ref = 0;
        unsigned int ref_n = 0, key_pad = 0;
        const int nslots = p.world * gcap;
        for (int base = 0; base < nslots; base += 32) {
            const int t = base + lane;
            const bool in = t < nslots;
            const int r = in ? t / gcap : 0, g = in ? t % gcap : 0;
            const bool v = in && s.items[t].e.n != 0;
            const unsigned int n = v ? s.items[t].e.n : 0u;
            const bool failed = v && s.items[t].chunk_prefix != 0ull;
            const bool huf = v && s.items[t].huffman != 0u;
            unsigned long long c_inc = (n + SKML_RESTART_INTERVAL - 1) / SKML_RESTART_INTERVAL, k_inc = (n + 3ull) & ~3ull;   // (stashed four at a time)
            unsigned long long b_inc = huf ? skml_align16((unsigned long long)s.items[t].rows * s.items[t].e.col_num * (s.items[t].cell_bits / 8)) : 0ull;
            const unsigned long long c_own = c_inc, k_own = k_inc, b_own = b_inc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long c2 = __shfl_up_sync(0xFFFFFFFFu, c_inc, o), k2 = __shfl_up_sync(0xFFFFFFFFu, k_inc, o),
                                         b2 = __shfl_up_sync(0xFFFFFFFFu, b_inc, o);
                if (lane >= o) {
                    c_inc += c2;
                    k_inc += k2;
                    b_inc += b2;
                }
            }
            const unsigned int vm = __ballot_sync(0xFFFFFFFFu, v);
            const int pos = ni + __popc(vm & ((1u << lane) - 1u));
            if (in && g == 0) {   // what lies in front of rank r's first slot
                s.rank_key_begin[r] = keys + k_inc - k_own;
                s.rank_item_begin[r] = pos;
            }
            if (__any_sync(0xFFFFFFFFu, v && pos != t)) {   // some slot before is empty: entries move forward
                DecItem it;
                if (v) it = s.items[t];
                __syncwarp();   // every lane holds its entry in registers
                if (v) s.items[pos] = it;
            }
            if (v) {
                DecItem& it = s.items[pos];
                it.chunk_prefix = chunks + c_inc - c_own;
                it.key_prefix = keys + k_inc - k_own;
                if (huf) it.tab = p.tab_scratch + tab_used + b_inc - b_own;
            }
            const unsigned int fm = __ballot_sync(0xFFFFFFFFu, failed);
            if (fm) {
                const int r_bad = __shfl_sync(0xFFFFFFFFu, r, __ffs(fm) - 1);
                if (lane == 0) {
                    skml_set_status(p.status, SKML_BAD_HEADER, 0x100u | (unsigned int)r_bad);
                    s.ok = 0;
                }
            }
            // the longest list (the first of equals) gives the apply its range bounds
            unsigned int best_n = n;
            int best_pos = v ? pos : 0x7FFFFFFF;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned int on = __shfl_xor_sync(0xFFFFFFFFu, best_n, o);
                const int op = __shfl_xor_sync(0xFFFFFFFFu, best_pos, o);
                if (on > best_n || (on == best_n && op < best_pos)) {
                    best_n = on;
                    best_pos = op;
                }
            }
            if (best_n > ref_n) {
                ref_n = best_n;
                ref = best_pos;
            }
            chunks += __shfl_sync(0xFFFFFFFFu, c_inc, 31);
            keys += __shfl_sync(0xFFFFFFFFu, k_inc, 31);
            key_pad += __reduce_add_sync(0xFFFFFFFFu, (unsigned int)(k_own - n));
            tab_used += __shfl_sync(0xFFFFFFFFu, b_inc, 31);
            ni += __popc(vm);
            nhuf += __popc(__ballot_sync(0xFFFFFFFFu, huf));
            __syncwarp();
        }
      if (lane == 0) {
        if (tab_used > (unsigned long long)p.tab_capacity) {
            skml_set_status(p.status, SKML_CAPACITY, 0x41u);
            s.ok = 0;
        }
        if (keys - key_pad > (unsigned long long)p.key_capacity) {
            skml_set_status(p.status, SKML_CAPACITY, 0x40u);
            s.ok = 0;
        }
        for (int r = p.world; r <= SKML_MAX_PEERS; ++r) {
            s.rank_key_begin[r] = keys;
            s.rank_item_begin[r] = ni;
        }
        s.ref_item = ref;
        s.nitems = ni;
        s.nhuf = nhuf;
        s.total_chunks = chunks;
        s.total_keys = keys;
        s.small_passes = chunks < 4ull * gridDim.x * (unsigned long long)p.world ? 1 : 0;
      }
    }
    __syncthreads();
    return s.ok != 0;
}

// Huffman-coded sketch tables -> 8/16-bit bucket codes in the scratch, before any key is decoded
// (binary/HuffmanEncoder.java:126-166 decodes by walking a tree; here the code words, left-aligned and
// sorted, are searched with the next 32 stream bits: in a prefix code the word that matches is the
// largest one not above them). A block works on one item at a time; its threads each decode a stretch
// of cells from a restart offset (every `head[3]` cells; a table without restart offsets is decoded by
// one thread). Never-written cells (Integer.MAX_VALUE) become the zero bucket, as in the narrow form.
// What bounds it is the chain of a stretch's 128 cells, some 60 cycles each: the next stream bits wait in a 64-bit
// window, words of up to DEC_HUF_LUT bits are looked up in a table of all prefixes, and a warp takes as few
// stretches (16 at most) as keep all warps busy, with their part of the stream staged in shared memory first:
// the lanes refill their windows at different cells, so every load from L2 would hold up all of them.
// (Two L2 loads and a search per cell took 80 us for 200,000 keys' tables.)
__device__ __noinline__ void expand_tables(const DP& p, DecSmem& s) {
    if (s.nhuf == 0) return;
    unsigned char* area = reinterpret_cast<unsigned char*>(&s) + p.tab_off;
    unsigned int* la = reinterpret_cast<unsigned int*>(area);                       // left-aligned code words, ascending
    unsigned short* sym = reinterpret_cast<unsigned short*>(la + DEC_HUF_MAX_ITEMS);  // their symbols (0xFFFF = never written)
    unsigned char* len = reinterpret_cast<unsigned char*>(sym + DEC_HUF_MAX_ITEMS);
    // [prefix of DEC_HUF_LUT bits]: symbol | code length << 16, 0 = longer code; the records as they arrived
    unsigned int* lut = reinterpret_cast<unsigned int*>(area + 7 * DEC_HUF_MAX_ITEMS + 1);   // 7 x 513 + 1 is a multiple of 8
    int* recs = reinterpret_cast<int*>(lut + (1 << DEC_HUF_LUT));
    static_assert((7 * DEC_HUF_MAX_ITEMS + 1) % 4 == 0 && 7 * DEC_HUF_MAX_ITEMS + 1 + (4 << DEC_HUF_LUT) + 12 * DEC_HUF_MAX_ITEMS <= DEC_TAB_SMEM &&
                  7 * DEC_HUF_MAX_ITEMS + 1 + (4 << DEC_HUF_LUT) + DEC_THREADS / 8 * DEC_HUF_STAGE <= DEC_TAB_SMEM,
                  "the expander's tables fit the staged-table area");
    __shared__ unsigned int s_head[4];
    __shared__ int s_bad;
    // blocks are dealt to the Huffman items round-robin; the blocks of one item share its stretches
    const int H = s.nhuf, B = (int)gridDim.x;
    int seen = 0;
    for (int i = 0; i < s.nitems; ++i) {
        const DecItem& it = s.items[i];
        if (!it.huffman) continue;
        const int mine = seen++;
        int helper = 0, nhelp = 1;
        if (H <= B) {
            if ((int)blockIdx.x % H != mine) continue;
            helper = (int)blockIdx.x / H;
            nhelp = (B - mine + H - 1) / H;
        } else if (mine % B != (int)blockIdx.x) {
            continue;
        }
        const unsigned char* sec = it.base + it.e.table_off;
        __syncthreads();
        if (threadIdx.x < 4) s_head[threadIdx.x] = __ldcg(reinterpret_cast<const unsigned int*>(sec) + threadIdx.x);
        if (threadIdx.x == 0) s_bad = 0;
        __syncthreads();
        const unsigned int nitems = s_head[0], nwords = s_head[1], cells = s_head[2], interval = s_head[3];
        const unsigned long long lim = reinterpret_cast<const SkmlHeader*>(it.base)->total_bytes;
        const unsigned int want = it.rows * it.e.col_num;
        const unsigned long long stream_off = it.e.table_off + 16ull + 12ull * nitems;
        const unsigned long long restart_off = skml_align16(stream_off + 8ull * nwords);
        const unsigned int nseg = interval ? (cells + interval - 1) / interval : 1u;
        if (nitems == 0 || nitems > DEC_HUF_MAX_ITEMS || cells != want || stream_off + 8ull * nwords > lim ||
            (interval && restart_off + 4ull * nseg > lim)) {
            if (threadIdx.x == 0) skml_set_status(p.status, SKML_BAD_HEADER, 0x600u | (unsigned int)(i & 0xFF));
            continue;
        }
        // code words: rank sort by the left-aligned word
        for (unsigned int a = threadIdx.x; a < 3 * nitems; a += blockDim.x) recs[a] = __ldcg(reinterpret_cast<const int*>(sec + 16) + a);
        __syncthreads();
        for (unsigned int a = threadIdx.x; a < nitems; a += blockDim.x) {
            const int value = recs[3 * a], bits = recs[3 * a + 1], nb = recs[3 * a + 2];
            if (nb < 1 || nb > 32) {
                s_bad = 1;
                continue;
            }
            const unsigned int mine_la = (unsigned int)bits << (32 - nb);
            unsigned int r = 0;
            for (unsigned int b = 0; b < nitems; ++b) {
                const int nbb = recs[3 * b + 2];
                const unsigned int other = (nbb >= 1 && nbb <= 32) ? (unsigned int)recs[3 * b + 1] << (32 - nbb) : 0u;
                if (other < mine_la || (other == mine_la && b < a)) ++r;
            }
            la[r] = mine_la;
            len[r] = (unsigned char)nb;
            sym[r] = value == 0x7FFFFFFF ? (unsigned short)it.zero : (unsigned short)value;
        }
        __syncthreads();
        if (s_bad) {
            if (threadIdx.x == 0) skml_set_status(p.status, SKML_BAD_HEADER, 0x700u | (unsigned int)(i & 0xFF));
            continue;
        }
        auto search = [&](unsigned int x) {   // largest word <= x
            unsigned int a = 0, b = nitems;
            while (b - a > 1) {
                const unsigned int mid = (a + b) >> 1;
                if (la[mid] <= x) a = mid;
                else b = mid;
            }
            return a;
        };
        for (unsigned int e = threadIdx.x; e < (1u << DEC_HUF_LUT); e += blockDim.x) {
            const unsigned int a = search(e << (32 - DEC_HUF_LUT));
            lut[e] = len[a] <= DEC_HUF_LUT ? (unsigned int)sym[a] | ((unsigned int)len[a] << 16) : 0u;
        }
        __syncthreads();
        const unsigned int* words = reinterpret_cast<const unsigned int*>(it.base + stream_off);
        const unsigned int wlim = 2u * nwords;
        const unsigned int* restart = reinterpret_cast<const unsigned int*>(it.base + restart_off);
        unsigned char* out = const_cast<unsigned char*>(it.tab);
        // one stretch by one thread; word(w): stream word w with its most significant bit first
        auto stretch = [&](unsigned int pos, unsigned int c0, unsigned int c1, auto word) {
            unsigned int w = pos >> 5;
            unsigned long long win = (((unsigned long long)word(w) << 32) | word(w + 1)) << (pos & 31u);   // next bit on top
            int have = 64 - (int)(pos & 31u);
            w += 2;
            auto next = [&]() {
                const unsigned int x = (unsigned int)(win >> 32);
                unsigned int v = lut[x >> (32 - DEC_HUF_LUT)], n = v >> 16;
                if (n == 0) {
                    const unsigned int a = search(x);
                    v = sym[a];
                    n = len[a];
                }
                win <<= n;
                have -= (int)n;
                if (have <= 32) {
                    win |= (unsigned long long)word(w++) << (32 - have);
                    have += 32;
                }
                return v & 0xFFFFu;
            };
            unsigned int c = c0;
            if (it.cell_bits == 8) {
                for (; c + 4 <= c1 && (c & 3u) == 0; c += 4) {   // whole words
                    unsigned int v = next();
                    v |= next() << 8;
                    v |= next() << 16;
                    v |= next() << 24;
                    *reinterpret_cast<unsigned int*>(out + c) = v;
                }
                for (; c < c1; ++c) out[c] = (unsigned char)next();
            } else {
                for (; c < c1; ++c) reinterpret_cast<unsigned short*>(out)[c] = (unsigned short)next();
            }
        };
        auto from_payload = [&](unsigned int w) { return w < wlim ? __brev(__ldcg(words + w)) : 0u; };
        if (!interval) {
            if (helper == 0 && threadIdx.x == 0) stretch(0u, 0u, cells, from_payload);
            continue;
        }
        const unsigned int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (unsigned int)nhelp * (DEC_THREADS / 32);
        const unsigned int per = min(16u, (nseg + warps - 1) / warps);
        unsigned int* const stage = reinterpret_cast<unsigned int*>(recs) + warp * DEC_HUF_STAGE;   // (the records are sorted by now)
        for (unsigned int s0 = ((unsigned int)helper * (DEC_THREADS / 32) + warp) * per; s0 < nseg; s0 += warps * per) {
            const unsigned int sg = s0 + lane;
            const bool mine = lane < per && sg < nseg;
            const unsigned int pos = sg < nseg ? __ldcg(restart + sg) : 32u * wlim;   // lane `per`: where the turn's stretches end
            const unsigned int first = __shfl_sync(0xFFFFFFFFu, pos, 0) >> 5, last = __shfl_sync(0xFFFFFFFFu, pos, (int)per) >> 5;
            const unsigned int nw = last - first + 1;
            __syncwarp();
            const bool staged = last >= first && nw <= DEC_HUF_STAGE;
            if (staged)
                for (unsigned int w = lane; w < nw; w += 32) stage[w] = from_payload(first + w);
            __syncwarp();
            if (mine) {
                const unsigned int c0 = sg * interval, c1 = min(cells, c0 + interval);
                if (staged) stretch(pos, c0, c1, [&](unsigned int w) { return w - first < nw ? stage[w - first] : 0u; });
                else stretch(pos, c0, c1, from_payload);
            }
            __syncwarp();
        }
    }
    __syncthreads();
}

// D1 for sparse payloads: one 1024-key chunk per block iteration, DEC_KPT adjacent keys per
// thread (256 threads), so that every thread has several independent load chains in flight and
// several blocks share an SM.
__device__ void decode_accumulate(const DP& p, DecSmem& s, int i_begin, int i_end, float& dsq) {
    __shared__ unsigned int s_part[6][DEC_THREADS / 32];  // [3 scans x chunk parity]
    __shared__ unsigned short s_pos[SKML_RESTART_INTERVAL];  // delta_adaptive with unary flags: where every key's flag ends
    int par = 0;
    // Every block takes a contiguous run of chunks, so that consecutive chunks belong to the same
    // (rank, group) list and its sketch table, when it fits, is staged in shared memory once and
    // then queried there: three random L2 sectors per key become one coalesced read of the table.
    // Runs differ by one chunk at most: with equal runs (6 where 5.06 is the mean) a sixth of the blocks had none.
    // (One range of the model per block, a share of every list, was tried for single payloads: an update alone is
    // faster in key order, 59 against 81 us for 2.2M keys of 50M, but the shares come out uneven, 0 to 2 chunks where
    // one is the mean, and the launch took 89 instead of 81 us, 41 instead of 25 at 0.4M keys.)
    const unsigned long long run0 = i_begin < i_end ? s.items[i_begin].chunk_prefix : 0ull;
    const unsigned long long run_n = (i_end < s.nitems ? s.items[i_end].chunk_prefix : s.total_chunks) - run0;
    const unsigned int run_end = (unsigned int)(run0 + run_n * (blockIdx.x + 1) / gridDim.x);
    unsigned int ch = (unsigned int)(run0 + run_n * blockIdx.x / gridDim.x);
    int item = i_begin;
    unsigned char* tab_area = p.tab_off ? reinterpret_cast<unsigned char*>(&s) + p.tab_off : nullptr;
    int staged = -1;
    const unsigned char* stab = nullptr;
    const DecForm form = decode_form(p, s);
    const bool sums = p.out_sum != nullptr, two_phase = form.two_phase, direct = form.direct, adam = form.adam_plain;
    const float iw = (float)s.inv_world;
    float* const dst = sums ? p.out_sum : p.w;
    ChunkHead head;
    auto fetch = [&]() {   // the head of chunk `ch`
        while (item + 1 < i_end && ch >= s.items[item + 1].chunk_prefix) ++item;
        head = fetch_head(s.items[item], ch - (unsigned int)s.items[item].chunk_prefix);
    };
    if (ch < run_end) fetch();
    while (ch < run_end) {
        const DecItem& it = s.items[item];
        const unsigned int j = ch - (unsigned int)it.chunk_prefix;
        if (item != staged) {
            staged = item;
            stab = stage_table(it, tab_area);
        }
        const ChunkHead now = head;
        if (++ch < run_end) fetch();
        ChunkKeys c;
        decode_keys(p, it, j, now, s_part[par], s_part[2 + par], s_part[4 + par], s_pos, c);
        if (c.i0 < c.cnt) {
            // What the update reads does not depend on the sketch: its loads (random sectors of the model) start before
            // the queries, for all keys of the thread at once. Keys are unique inside a payload, so no store below
            // touches what another key of the thread loads.
            float old[DEC_KPT], mom[DEC_KPT], vel[DEC_KPT];
#pragma unroll
            for (int u = 0; u < DEC_KPT; ++u) {
                old[u] = mom[u] = vel[u] = 0.f;
                if (c.keys[u] == 0xFFFFFFFFu) continue;
                if (two_phase) continue;
                if (direct) {
                    old[u] = dst[c.keys[u]];
                } else if (adam && !sums) {
                    old[u] = p.w[c.keys[u]];
                    mom[u] = p.adam_m[c.keys[u] * p.adam_stride];
                    vel[u] = p.adam_v[c.keys[u] * p.adam_stride];
                }
            }
            float bv[DEC_KPT];
            query_keys(it, stab, c.keys, bv);
            const unsigned long long at = it.key_prefix + c.first + c.i0;   // a multiple of four, as every list's start
            if (two_phase) {
                // stash (key, value): the ordered apply passes read them back coalesced
                *reinterpret_cast<int4*>(p.key_scratch + at) = make_int4((int)c.keys[0], (int)c.keys[1], (int)c.keys[2], (int)c.keys[3]);
                *reinterpret_cast<float4*>(p.val_scratch + at) = make_float4(bv[0] * iw, bv[1] * iw, bv[2] * iw, bv[3] * iw);
            } else if (direct) {  // single payload: keys are unique inside it, plain read-modify-write
#pragma unroll
                for (int u = 0; u < DEC_KPT; ++u) {
                    if (c.keys[u] == 0xFFFFFFFFu) continue;
                    const float g = bv[u] * iw, nw = sums ? old[u] + g : old[u] - p.lr * g;
                    dst[c.keys[u]] = nw;
                    if (!sums) dsq += (nw - old[u]) * (nw + old[u]);
                }
            } else if (adam) {  // single payload: the decoded value is the whole gradient of its key
#pragma unroll
                for (int u = 0; u < DEC_KPT; ++u)
                    if (c.keys[u] != 0xFFFFFFFFu && bv[u] != 0.f) dsq += apply_loaded(p, c.keys[u], bv[u] * iw, old[u], mom[u], vel[u]);
            } else {
                *reinterpret_cast<int4*>(p.key_scratch + at) = make_int4((int)c.keys[0], (int)c.keys[1], (int)c.keys[2], (int)c.keys[3]);
#pragma unroll
                for (int u = 0; u < DEC_KPT; ++u) {
                    const long long fx = c.keys[u] != 0xFFFFFFFFu ? to_fixed((double)bv[u] * s.inv_world, s.shift) : 0ll;
                    if (fx) atomicAdd(reinterpret_cast<unsigned long long*>(p.acc + c.keys[u]), (unsigned long long)fx);
                }
            }
        }
        par ^= 1;   // no barrier here: the next chunk's scans use the other parity of s_part
    }
    __syncthreads();
}

// Ordered apply of one rank's stashed (key, value) pairs: keys are unique inside a payload, so the
// plain read-modify-write needs no atomics; four independent pairs per thread and iteration.
__device__ __noinline__ void apply_stashed(const DP& p, unsigned long long begin, unsigned long long end, float& dsq) {
    const unsigned long long gsz = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long t = begin + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < end; t += 4 * gsz) {
        unsigned int k[4];
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned long long tt = t + u * gsz;
            k[u] = tt < end ? (unsigned int)__ldcg(p.key_scratch + tt) : 0xFFFFFFFFu;
            v[u] = tt < end ? __ldcg(p.val_scratch + tt) : 0.f;
        }
        float old[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float* dst = p.out_sum ? p.out_sum : p.w;
            old[u] = k[u] < (unsigned long long)p.dim ? dst[k[u]] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k[u] < (unsigned long long)p.dim) {
                if (p.out_sum) p.out_sum[k[u]] = old[u] + v[u];
                else {
                    const float nw = old[u] - p.lr * v[u];
                    p.w[k[u]] = nw;
                    dsq += (nw - old[u]) * (nw + old[u]);
                }
            }
    }
}

// One rank's slice of the block's key range. The groups of one rank hold disjoint keys, so their slices are walked as one
// concatenated list: `ends` are the slices' ends in it, `shift` what an entry's place in it lacks to its place in the
// scratch. A thread takes four independent entries per iteration.
struct OwnedEntries {
    unsigned int k[4];   // 0xFFFFFFFF: none
    float v[4];
};
template <bool VALUES>
__device__ __forceinline__ void owned_fetch(const DP& p, const DecSmem& s, const unsigned long long* shift, const unsigned long long* ends, int r,
                                            unsigned int q, OwnedEntries& e) {
    int i = s.rank_item_begin[r];
    const int i1 = s.rank_item_begin[r + 1];
    const unsigned int total = i < i1 ? (unsigned int)ends[i1 - 1] : 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const unsigned int qq = q + u * DEC_THREADS;
        e.k[u] = 0xFFFFFFFFu;
        e.v[u] = 0.f;
        if (qq < total) {
            while (qq >= (unsigned int)ends[i]) ++i;
            const unsigned long long pos = shift[i] + qq;
            e.k[u] = (unsigned int)__ldcg(p.key_scratch + pos);
            if (VALUES) e.v[u] = __ldcg(p.val_scratch + pos);
        }
    }
}

// OP 0: SGD step / plain sum; OP 1: add into the float accumulators; OP 2: Adam update of every coordinate whose
// accumulated sum is non-zero, then clear it. `e`: the thread's first entries, loaded by the caller; those of rank `next`
// (negative: none) are there when the pass ends. A block barrier ends it.
// Entries are loaded while the weights before them arrive where a pass is an iteration or little more and waits for one trip
// after the other; longer passes, whose sectors come from DRAM, load them behind the stores: eight payloads of 60,000 keys
// 42 us (44 with the loads behind the barrier), of 62,500 rows (430,000 keys) 122 (131), of 1M keys of 50M 431 (458 with the
// loads ahead), two of 4M with Adam 1155 (1229). Adam's sweeps find the sums of shorter slices in L2 already: eight of 600,000
// keys, slices of 675, 702 (715).
template <int OP>
__device__ __forceinline__ void owned_pass(const DP& p, DecSmem& s, const unsigned long long* shift, const unsigned long long* ends, int r, int next,
                                           OwnedEntries& e, float& dsq) {
    const int i1 = s.rank_item_begin[r + 1];
    const unsigned int total = s.rank_item_begin[r] < i1 ? (unsigned int)ends[i1 - 1] : 0u;
    float* dst = OP == 0 ? (p.out_sum ? p.out_sum : p.w) : p.fsum;
    const long long ds = OP == 0 ? 1ll : p.fsum_stride;
    const bool many = total > (OP == 0 ? 5 : 2) * DEC_THREADS;
    OwnedEntries ahead;
    for (unsigned int q = threadIdx.x;; q += 4 * DEC_THREADS) {
        float old[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) old[u] = e.k[u] < (unsigned long long)p.dim ? dst[e.k[u] * ds] : 0.f;
        const bool more = q + 4 * DEC_THREADS < total;
        if (!many) {
            if (more) owned_fetch<OP != 2>(p, s, shift, ends, r, q + 4 * DEC_THREADS, ahead);
            else if (next >= 0) owned_fetch<OP != 2>(p, s, shift, ends, next, threadIdx.x, ahead);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (e.k[u] >= (unsigned long long)p.dim) continue;
            if (OP == 0) {
                const float nw = p.out_sum ? old[u] + e.v[u] : old[u] - p.lr * e.v[u];
                dst[e.k[u] * ds] = nw;
                if (!p.out_sum) dsq += (nw - old[u]) * (nw + old[u]);
            } else if (OP == 1) dst[e.k[u] * ds] = old[u] + e.v[u];
            else if (old[u] != 0.f) {
                dst[e.k[u] * ds] = 0.f;
                dsq += apply_one(p, e.k[u], old[u]);
            }
        }
        if (many) {
            if (more) owned_fetch<OP != 2>(p, s, shift, ends, r, q + 4 * DEC_THREADS, ahead);
            else if (next >= 0) owned_fetch<OP != 2>(p, s, shift, ends, next, threadIdx.x, ahead);
        }
        e = ahead;
        if (!more) break;
    }
    __syncthreads();
}
template <int OP>
__device__ __forceinline__ void owned_passes(const DP& p, DecSmem& s, const unsigned long long* shift, const unsigned long long* ends, float& dsq) {
    OwnedEntries e;
    owned_fetch<OP != 2>(p, s, shift, ends, 0, threadIdx.x, e);
    for (int r = 0; r < p.world; ++r) owned_pass<OP>(p, s, shift, ends, r, r + 1 < p.world ? r + 1 : -1, e, dsq);
}

// Barrier-free ordered apply. The key space is cut into DEC_OWN_RANGES x blocks ranges at the quantiles
// of the longest key list; a block owns one range per round, dealt in snake order (round 0: range b,
// round 1: range 2B - 1 - b, ...). Low keys are the frequent ones and sit in L2 while the high ones
// miss to DRAM, so a block's ranges cost about the same in sum although single ranges differ several
// times. For each of its ranges the block finds its slice of every (rank, group) list by binary search
// in the stashed keys and applies the slices rank by rank with only a block barrier in between: all
// updates of one coordinate happen in one block, in rank order, so replicas stay bit-identical.
__device__ void apply_owned(const DP& p, DecSmem& s, float& dsq) {
    if (s.nitems == 0) return;
    unsigned long long* seg = reinterpret_cast<unsigned long long*>(&s.items[p.max_items]);  // [2 * DEC_OWN_RANGES][max_items]
    __shared__ unsigned long long s_bound[2 * DEC_OWN_RANGES];
    // SGD: one range per block (more ranges even out the blocks but do not shorten the launch: the random
    // DRAM sectors bound it in total). Lazy Adam sweeps a range 2 x ranks times, and smaller ranges keep its
    // sectors in L2 between the sweeps; where a block has fewer than 2048 keys, the sweeps' latency is what counts.
    const int rounds = p.adam_v && s.total_keys >= 2048ull * gridDim.x ? DEC_OWN_RANGES : 1;
    if (threadIdx.x < 2 * rounds) {
        const DecItem& ref = s.items[s.ref_item];
        const unsigned long long B = gridDim.x, total = (unsigned long long)rounds * B;
        const unsigned long long round = threadIdx.x >> 1;
        const unsigned long long range = (round & 1ull) ? (round + 1ull) * B - 1ull - blockIdx.x : round * B + blockIdx.x;
        const unsigned long long j = range + (threadIdx.x & 1);   // lower / upper bound of the range
        unsigned long long v;
        if (j == 0) v = 0ull;
        else if (j >= total) v = 1ull << 32;
        else v = (unsigned long long)(unsigned int)__ldcg(p.key_scratch + ref.key_prefix + j * (unsigned long long)ref.e.n / total);
        s_bound[threadIdx.x] = v;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * rounds * s.nitems; t += blockDim.x) {
        const int item = t / (2 * rounds), which = t % (2 * rounds);
        const DecItem& it = s.items[item];
        const unsigned long long bound = s_bound[which];
        const int* list = p.key_scratch + it.key_prefix;
        unsigned int lo = 0, hi = it.e.n;
        while (lo < hi) {  // first position whose key is >= bound: three probes a step, half as many trips to L2 as with one
            const unsigned int len = hi - lo, m1 = lo + len / 4, m2 = lo + len / 2, m3 = m2 + (hi - m2) / 2;
            const unsigned int k1 = (unsigned int)__ldcg(list + m1), k2 = (unsigned int)__ldcg(list + m2), k3 = (unsigned int)__ldcg(list + m3);
            if ((unsigned long long)k2 < bound) {
                if ((unsigned long long)k3 < bound) lo = m3 + 1;
                else {
                    lo = m2 + 1;
                    hi = m3;
                }
            } else if ((unsigned long long)k1 < bound) {
                lo = m1 + 1;
                hi = m2;
            } else {
                hi = m1;
            }
        }
        seg[(size_t)which * p.max_items + item] = it.key_prefix + lo;
    }
    __syncthreads();
    // begin and end of every slice -> end in the rank's concatenated slices, and shift (a warp's lane per rank and range)
    for (int t = threadIdx.x; t < rounds * p.world; t += blockDim.x) {
        const int r = t % p.world;
        unsigned long long* const b = seg + (size_t)(2 * (t / p.world)) * p.max_items;
        unsigned long long* const e = b + p.max_items;
        unsigned long long end = 0;
        for (int i = s.rank_item_begin[r]; i < s.rank_item_begin[r + 1]; ++i) {
            const unsigned long long before = end;
            end += e[i] - b[i];
            b[i] -= before;
            e[i] = end;
        }
    }
    __syncthreads();
    for (int round = 0; round < rounds; ++round) {
        const unsigned long long* shift = seg + (size_t)(2 * round) * p.max_items;
        const unsigned long long* ends = shift + p.max_items;
        if (p.adam_v) {
            // Adam: sum the ranks' values per coordinate in rank order (plain floats in the zeroed
            // sums), then let the first rank that holds a coordinate apply the update and clear the sum.
            owned_passes<1>(p, s, shift, ends, dsq);
            owned_passes<2>(p, s, shift, ends, dsq);
        } else {
            owned_passes<0>(p, s, shift, ends, dsq);
        }
    }
}

// D1 for dense payloads: every coordinate carries a bucket code. Four adjacent coordinates per thread, so that codes
// and weights move in vectors, and the bucket values wait in shared memory. (One coordinate at a time, with the bucket
// value from L2, took 43 us for 1M coordinates.)
__device__ void decode_accumulate_dense(const DP& p, DecSmem& s, int r_begin, int r_end, float& dsq) {
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float* const bv = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(&s) + p.tab_off);
    static_assert(4 * SKML_GPU_MAX_BINS <= DEC_TAB_SMEM, "the bucket values fit the staged-table area");
    float* const dst = p.out_sum ? p.out_sum : p.w;
    const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    for (int r = r_begin; r < r_end; ++r) {
        const HdrLite& h = s.hdr[r];
        if (h.kind != SKML_KIND_DENSE) continue;
        const unsigned char* codes = p.payload[r] + h.off_dense_codes;
        __syncthreads();   // nobody reads the area any more
        for (unsigned int b = threadIdx.x; b < h.bin_num; b += blockDim.x)
            bv[b] = __ldcg(reinterpret_cast<const float*>(p.payload[r] + h.off_bucket_values) + b);
        __syncthreads();
        const unsigned int bin_num = h.bin_num, zero = h.zero_idx;
        const bool narrow = h.cell_bits == 8;
        for (long long q = gid; q < (p.dim + 3) / 4; q += gsz) {   // (a code section is padded to 16 bytes)
            const long long i0 = 4 * q;
            unsigned int c[4];
            if (narrow) {
                const unsigned int x = __ldcg(reinterpret_cast<const unsigned int*>(codes) + q);
#pragma unroll
                for (int u = 0; u < 4; ++u) c[u] = (x >> (8 * u)) & 0xFFu;
            } else {
                const uint2 x = __ldcg(reinterpret_cast<const uint2*>(codes) + q);
                c[0] = x.x & 0xFFFFu; c[1] = x.x >> 16; c[2] = x.y & 0xFFFFu; c[3] = x.y >> 16;
            }
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = bv[c[u] < bin_num ? c[u] : zero];
            if (p.adam_v) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (i0 + u >= p.dim) continue;
                    const long long fx = to_fixed((double)v[u] * s.inv_world, s.shift);
                    if (fx) atomicAdd(reinterpret_cast<unsigned long long*>(p.acc + i0 + u), (unsigned long long)fx);
                }
            } else if (vec && i0 + 4 <= p.dim) {
                float4 old = *reinterpret_cast<float4*>(dst + i0), nw;
                const float iw = (float)s.inv_world;
                if (p.out_sum) {
                    nw = make_float4(old.x + v[0] * iw, old.y + v[1] * iw, old.z + v[2] * iw, old.w + v[3] * iw);
                } else {
                    nw = make_float4(old.x - p.lr * (v[0] * iw), old.y - p.lr * (v[1] * iw), old.z - p.lr * (v[2] * iw),
                                     old.w - p.lr * (v[3] * iw));
                    dsq += (nw.x - old.x) * (nw.x + old.x);
                    dsq += (nw.y - old.y) * (nw.y + old.y);
                    dsq += (nw.z - old.z) * (nw.z + old.z);
                    dsq += (nw.w - old.w) * (nw.w + old.w);
                }
                *reinterpret_cast<float4*>(dst + i0) = nw;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i0 + u < p.dim) dsq += apply_direct(p, i0 + u, v[u] * (float)s.inv_world);
            }
        }
    }
}

// D2: claim and update.
__device__ __noinline__ void decode_update(const DP& p, DecSmem& s, float& dsq) {
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s.any_dense) {
        for (long long i = gid; i < p.dim; i += gsz) {
            long long a = p.acc[i];
            if (a) {
                p.acc[i] = 0;
                dsq += apply_one(p, i, (float)from_fixed(a, s.shift));
            }
        }
    } else {
        // four independent claims per thread and iteration: their round trips overlap
        for (long long t = gid; t < (long long)s.total_keys; t += 4 * gsz) {
            long long k[4], a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const long long tt = t + u * gsz;
                k[u] = tt < (long long)s.total_keys ? (long long)(unsigned int)p.key_scratch[tt] : p.dim;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                a[u] = k[u] < p.dim ? (long long)atomicExch(reinterpret_cast<unsigned long long*>(p.acc + k[u]), 0ull) : 0ll;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (a[u]) dsq += apply_one(p, k[u], (float)from_fixed(a[u], s.shift));
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.loss_out) {
        double l[4] = {0, 0, 0, 0};
        for (int r = 0; r < p.world; ++r)
            for (int i = 0; i < 4; ++i) l[i] += s.hdr[r].loss_partials[i];
        for (int i = 0; i < 4; ++i) p.loss_out[i] = l[i];
    }
}

// The launch's end. Adds its change of the squared weight norm to the running sum; the last block to arrive
// turns the sum into the regularisation loss of the next batch (lambda * ||w||_2, un-squared as in
// ml/objective/Loss.scala:48-53) so that no step passes over the whole model for it, and puts the control words back.
// One count for both: a second one behind the first was another trip to L2 for every block. With that, the work table where it
// is and a block per SM for few keys: 10,000 keys 16.5 -> 15.0 us, 26,000 with Adam 18.9 -> 17.2, 430,000 20.7 -> 19.5.
template <bool FUSED>
__device__ void finish_launch(const DP& p, float dsq) {
    if (!FUSED && !p.wsq) return;
    __shared__ double s_red[DEC_THREADS / 32];
    if (p.wsq) {
        const double d = warp_sum((double)dsq);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (p.wsq) {
            double t = 0.0;
            for (int w = 0; w < DEC_THREADS / 32; ++w) t += s_red[w];
            if (t != 0.0) atomicAdd(p.wsq, t);
        }
        if (p.wsq || p.done_word) __threadfence();   // (a checked call returns before the kernel ends, see skml_store_done)
        const unsigned int prev = atomicAdd(&p.ctrl[2], 1u);
        if (prev == gridDim.x - 1) {
            p.ctrl[2] = 0;
            p.ctrl[0] = 0;   // nobody is in a grid barrier any more
            unsigned long long now;   // the kernel's true end (block 0's stamp is its own)
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (FUSED) reinterpret_cast<unsigned long long*>(p.ctrl)[16 + (int)(p.step & 1)] = now;
            if (p.wsq || p.done_word) __threadfence();
            if (p.wsq && p.reg_out) {
                const double w2 = *reinterpret_cast<volatile double*>(p.wsq);
                p.reg_out[0] = p.reg_lambda * sqrt(w2 > 0.0 ? w2 : 0.0);
            }
            skml_store_done(p.done_word, p.done_seq, p.status);
        }
    }
}

// The forms that few launches take (coded tables, stashed passes, claims) are functions of their own, out of the way of the
// code that every launch fetches: 26,000 keys with Adam 17.0 -> 16.6 us. (The apply by key ranges out of line: eight payloads of
// 430,000 keys 120 -> 129; the query of other than integer mixers: 26,000 keys 16.3, but 430,000 18.9 -> 19.6.)
template <bool FUSED>
__global__ void __launch_bounds__(DEC_THREADS, DEC_BLOCKS_PER_SM) decode_update_kernel(const __grid_constant__ DP p, int stage) {
    skml_after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DecSmem& s = *reinterpret_cast<DecSmem*>(smem_raw);
    float dsq = 0.f;  // this thread's share of the change of ||w||^2
    unsigned int passed = 0;   // arrivals of the grid barriers so far
    if (FUSED && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        reinterpret_cast<unsigned long long*>(p.ctrl)[8 + 4 * (int)(p.step & 1)] = t;
    }
    if (!decode_prepare(p, s)) return;
    if (s.nhuf) {  // tables that arrived Huffman-coded become plain bucket codes first
        if (FUSED || stage == 0) expand_tables(p, s);
        if (FUSED) {
            if (!skml_grid_barrier(p.ctrl, gridDim.x, p.status, p.budget, 0x2Eu, passed)) return;
        }
    }
    if (!FUSED && stage == 0) return;
    if (FUSED && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        reinterpret_cast<unsigned long long*>(p.ctrl)[9 + 4 * (int)(p.step & 1)] = t;
    }
    // Payloads applied one after the other take a pass per rank (un-fused: pass `stage - 1`), the rest one over all
    // lists. One call for every form: the passes are most of the kernel's code.
    const DecForm form = decode_form(p, s);
    const bool ordered = form.direct || form.adam_plain, per_rank = ordered && !form.two_phase;
    for (int r = 0; r < (per_rank ? p.world : 1); ++r) {
        if (FUSED || stage == r + 1) {
            decode_accumulate(p, s, per_rank ? s.rank_item_begin[r] : 0, per_rank ? s.rank_item_begin[r + 1] : s.nitems, dsq);
            if (s.any_dense && !form.two_phase) decode_accumulate_dense(p, s, per_rank ? r : 0, per_rank ? r + 1 : p.world, dsq);
        }
        if (FUSED && per_rank && r + 1 < p.world) {
            if (!skml_grid_barrier(p.ctrl, gridDim.x, p.status, p.budget, 0x30u + r, passed)) return;
        }
    }
    if (ordered) {
        if (form.two_phase) {
            if (FUSED) {
                if (!skml_grid_barrier(p.ctrl, gridDim.x, p.status, p.budget, 0x2Fu, passed)) return;
                if (blockIdx.x == 0 && threadIdx.x == 0) {
                    unsigned long long t;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                    reinterpret_cast<unsigned long long*>(p.ctrl)[10 + 4 * (int)(p.step & 1)] = t;
                }
            }
            // Phase 2 without dense payloads (un-fused: stage 2): key-range-owned apply, no grid barrier.
            if (!s.any_dense) {
                if (FUSED || stage == 2) apply_owned(p, s, dsq);
            } else
            // Phase 2 with dense payloads (un-fused: stage r + 2): one apply pass per rank, in rank order.
            for (int r = 0; r < p.world; ++r) {
                if (FUSED || stage == r + 2) {
                    apply_stashed(p, s.rank_key_begin[r], s.rank_key_begin[r + 1], dsq);
                    if (s.any_dense) decode_accumulate_dense(p, s, r, r + 1, dsq);
                }
                if (FUSED && r + 1 < p.world) {
                    if (!skml_grid_barrier(p.ctrl, gridDim.x, p.status, p.budget, 0x30u + r, passed)) return;
                }
            }
        }
        if ((FUSED || stage == 1) && blockIdx.x == 0 && threadIdx.x == 0 && p.loss_out) {
            double l[4] = {0, 0, 0, 0};
            for (int r = 0; r < p.world; ++r)
                for (int i = 0; i < 4; ++i) l[i] += s.hdr[r].loss_partials[i];
            for (int i = 0; i < 4; ++i) p.loss_out[i] = l[i];
        }
        if (FUSED && blockIdx.x == 0 && threadIdx.x == 0) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (!form.two_phase) reinterpret_cast<unsigned long long*>(p.ctrl)[10 + 4 * (int)(p.step & 1)] = t;
            reinterpret_cast<unsigned long long*>(p.ctrl)[11 + 4 * (int)(p.step & 1)] = t;
        }
        finish_launch<FUSED>(p, dsq);
        return;
    }
    if (FUSED) {
        if (!skml_grid_barrier(p.ctrl, gridDim.x, p.status, p.budget, 0x21u, passed)) return;
    }
    if (FUSED && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        reinterpret_cast<unsigned long long*>(p.ctrl)[10 + 4 * (int)(p.step & 1)] = t;
    }
    if (FUSED || stage == 2) decode_update(p, s, dsq);
    if (FUSED && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        reinterpret_cast<unsigned long long*>(p.ctrl)[11 + 4 * (int)(p.step & 1)] = t;
    }
    finish_launch<FUSED>(p, dsq);
}

extern "C" long long skml_decode_workspace_bytes(long long world, long long group_num) {
    (void)world;
    (void)group_num;
    return 256;
}

extern "C" int skml_decode_update(const SkmlDecodeArgs* a, void* stream_) {
    if (!a || !a->acc || !a->key_scratch || !a->workspace || !a->status) return (int)cudaErrorInvalidValue;
    if (a->world < 1 || a->world > SKML_MAX_PEERS) return (int)cudaErrorInvalidValue;
    if (!a->out_sum && !a->w) return (int)cudaErrorInvalidValue;
    cudaStream_t stream = (cudaStream_t)stream_;
    DP p;
    for (int i = 0; i < SKML_MAX_PEERS; ++i) {
        p.payload[i] = a->payload[i];
        p.flag[i] = a->flag[i];
    }
    p.world = (int)a->world;
    p.slot_capacity = a->slot_capacity;
    p.step = a->step;
    p.dim = a->dim;
    p.w = a->w;
    p.adam_m = a->adam_m;
    p.adam_v = a->adam_v;
    p.adam_stride = a->adam_stride > 1 ? a->adam_stride : 1;
    if (p.adam_stride == 4 && a->adam_m) {
        p.fsum = a->adam_m + 2;   // packed quads {m, v, sum, -}: the three words of a coordinate share a sector
        p.fsum_stride = 4;
    } else {
        p.fsum = reinterpret_cast<float*>(a->acc);
        p.fsum_stride = 1;
    }
    p.lr = (float)a->lr;
    p.adam_scale = (float)a->adam_scale;
    p.acc = a->acc;
    p.key_scratch = a->key_scratch;
    p.val_scratch = a->val_scratch;
    p.tab_scratch = a->table_scratch;
    p.tab_capacity = a->table_capacity;
    p.wsq = a->out_sum ? nullptr : a->weight_sumsq;
    p.reg_out = a->reg_out;
    p.reg_lambda = a->reg_lambda;
    p.done_word = a->done_word;
    p.done_seq = a->done_seq;
    p.key_capacity = a->key_capacity;
    p.loss_out = a->loss_out;
    p.out_sum = a->out_sum;
    p.ctrl = reinterpret_cast<unsigned int*>(a->workspace);
    p.status = a->status;
    p.budget = a->budget_cycles > 0 ? a->budget_cycles : 2000000000ll;
    // the (rank, group) table lives in dynamic shared memory: world x groups entries
    long long groups = a->max_groups > 0 ? a->max_groups : SKML_MAX_GROUPS;
    if (groups > SKML_MAX_GROUPS) groups = SKML_MAX_GROUPS;
    p.max_items = (int)(a->world * groups);
    // dynamic shared memory: work table, two slice bounds per entry, then the staged-table area
    const size_t smem_items = (sizeof(DecSmem) + (size_t)p.max_items * (sizeof(DecItem) + 16 * DEC_OWN_RANGES) + 15) & ~(size_t)15;
    p.tab_off = (int)smem_items;
    const size_t smem = smem_items + DEC_TAB_SMEM;
    static int sms = 0;
    static size_t cached_smem = 0;
    static int max_grid = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
        const int cap = (int)(sizeof(DecSmem) + (size_t)DEC_MAX_ITEMS * (sizeof(DecItem) + 16 * DEC_OWN_RANGES) + 16 + DEC_TAB_SMEM);
        cudaError_t e0 = cudaFuncSetAttribute(decode_update_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
        if (e0 == cudaSuccess)
            e0 = cudaFuncSetAttribute(decode_update_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
        if (e0 != cudaSuccess) {
            sms = 0;
            return (int)e0;
        }
    }
    if (cached_smem != smem) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_update_kernel<true>, DEC_THREADS, smem);
        max_grid = per_sm * sms;
        cached_smem = smem;
    }
    // Few keys: a block per SM, where each has a chunk at most (as many as a list's end takes more per group; a dense payload
    // has a code per coordinate). The other blocks would only stand in line at the launch's end (see finish_launch
    // for what this and a single count gave).
    int grid = a->grid > 0 ? (int)a->grid : DEC_BLOCKS_PER_SM * sms;
    const long long few = (long long)sms * SKML_RESTART_INTERVAL;
    if (a->grid <= 0 && a->world == 1 && a->key_capacity + groups * SKML_RESTART_INTERVAL <= few && (a->slot_capacity < a->dim || a->dim <= few)) grid = sms;
    cudaError_t e;
    if (a->fused) {
        if (max_grid < 1) return (int)cudaErrorLaunchOutOfResources;
        if (grid > max_grid) grid = max_grid;
        return (int)skml_launch_as(true, decode_update_kernel<true>, (unsigned)grid, DEC_THREADS, smem, stream, p, -1);
    }
    // stages: Adam = accumulate + claims; SGD over several payloads with a value scratch = decode +
    // one apply pass per rank; otherwise one pass per rank
    const int nst = a->adam_v ? 2 : ((a->world > 1 && a->val_scratch) ? (int)a->world + 1 : (int)a->world);
    for (int st = a->table_scratch ? 0 : 1; st <= nst; ++st) {
        decode_update_kernel<false><<<grid, DEC_THREADS, smem, stream>>>(p, st);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

extern "C" int skml_decode_sum_checked(SkmlDecodeArgs* a, unsigned int* status_out, void* stream) {
    if (!a || !a->done_word || !a->fused || !a->out_sum || !status_out) return (int)cudaErrorInvalidValue;
    const cudaError_t e = cudaMemsetAsync(a->out_sum, 0, (size_t)a->dim * sizeof(float), (cudaStream_t)stream);
    if (e != cudaSuccess) return (int)e;
    a->done_seq = ((*a->done_word >> 32) + 1) & 0xFFFFFFFFull;
    const int rc = skml_decode_update(a, stream);
    if (rc) return rc;
    return skml_wait_done(a->done_word, a->done_seq, a->status, status_out, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Peer memory helpers (one process per GPU, same node).
// ---------------------------------------------------------------------------
extern "C" int skml_ipc_get_handle(void* dev_ptr, unsigned char* handle64) {
    cudaIpcMemHandle_t h;
    cudaError_t e = cudaIpcGetMemHandle(&h, dev_ptr);
    if (e != cudaSuccess) return (int)e;
    memcpy(handle64, &h, sizeof(h));
    return 0;
}

extern "C" int skml_ipc_open_handle(const unsigned char* handle64, void** dev_ptr) {
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, sizeof(h));
    return (int)cudaIpcOpenMemHandle(dev_ptr, h, cudaIpcMemLazyEnablePeerAccess);
}

extern "C" int skml_ipc_close(void* dev_ptr) { return (int)cudaIpcCloseMemHandle(dev_ptr); }

// A zeroed device allocation of its own (cudaMalloc): the IPC handle of a receive region then names
// exactly that region, whatever a caching allocator does with the rest of the memory.
extern "C" int skml_region_alloc(long long bytes, void** dev_ptr) {
    if (bytes <= 0 || !dev_ptr) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaMalloc(dev_ptr, (size_t)bytes);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaMemset(*dev_ptr, 0, (size_t)bytes);
}

extern "C" int skml_region_free(void* dev_ptr) { return (int)cudaFree(dev_ptr); }

extern "C" int skml_enable_peer_access(int peer_device) {
    cudaError_t e = cudaDeviceEnablePeerAccess(peer_device, 0);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
        cudaGetLastError();
        return 0;
    }
    return (int)e;
}
