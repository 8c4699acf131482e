// Fused SketchML compress + publish for sm_100a.
//
// One persistent cooperative kernel (one block per SM, 1024 threads) runs the whole
// sender side of the gradient exchange:
//   S1  mergeable quantile summary of the values (sorted shared-memory tiles, k = 128
//       samples per run, pairwise merge + keep-every-second carry chain), min / max
//   S2  weighted-rank query of the merged summaries -> q-1 raw split points
//   S3  dedupe splits, zero bucket, bucket midpoints, group edges; bucketize every value and
//       count the keys of every bucket group per warp slice
//   S4  group sizes -> payload layout; every key goes to its group's contiguous (still key-sorted)
//       staging list; grouped MinMaxSketch insert (atomicMin on packed cells; for large gradients, as a stage of its
//       own, into tables in shared memory whose copies are merged in S6)
//   S5  the groups' key lists are coded in 1024-key chunks like a plain array: delta widths, byte
//       offsets, flag bytes, delta bytes staged per warp, one restart point per chunk. A block owns a
//       contiguous run of chunks and learns its byte offset from the blocks before it (their
//       published byte counts), so no grid barrier sits inside this stage
//   S6  header and group table; sketch tables narrowed to 8/16-bit bucket codes; the finished
//       payload is stored into every peer's receive slot with 16-byte peer stores, then the
//       arrival flags are released (system scope). There is no separate all-gather.
// Grid-wide dependencies are bounded software barriers, or, where a block needs only counts of the
// others, words that carry the launch's number beside the count and are polled with the same bound
// (a cooperative launch guarantees co-residency). With `fused = 0` the same stage functions run as
// separate launches.
//
// Reference behaviour restated (paths inside the reference project, module `sketch`):
//   quantization/QuantileQuantizer.java:27-50, sketch/quantile/HeapQuantileSketch.java:73-143,
//   293-323, sketch/quantile/QSketchUtils.java:45-82, base/Quantizer.java:39-92,
//   sketch/frequency/FSketchUtils.java:9-47, MinMaxSketch.java:27-55,
//   GroupedMinMaxSketch.java:103-121, binary/DeltaBinaryEncoder.java:26-39, and
//   ml/gradient/SketchGradient.scala:24-48.
#include <cooperative_groups.h>
#include <stdio.h>

#include "skml_api.h"
#include "skml_device.cuh"

#define MAX_GRID 192
#define SK_K 128            // samples per run
#define TILE 2048           // values sorted at once
#define TILE_W 16           // TILE / SK_K: weight of a sample taken from a full tile
#define MAX_LEVELS 24
#define FP_SHIFT 20         // fixed-point fraction bits of sample weights
#define MAX_SAMPLE 16        // largest sampling factor of the bottom-level sampler
#define HUF_MAX_SYMS 512     // symbols per bucket group the device Huffman coder accepts
#define HUF_RESTART 128      // cells between two restart offsets of a Huffman-coded table
#define AP_STAGE_F 548       // staging words of one chunk's flag bits (<= 17 bits per key, plus a word of misalignment)
#define AP_STAGE_D 1028      // the same for its delta bits (<= 32 bits per key)

struct CP {
    const int* keys;
    const float* vals;
    const long long* meta;
    long long n_max, dim;
    int q, G, rows;
    double col_ratio;
    unsigned long long seed, step;
    unsigned int rank, world;
    const double* loss_partials;
    unsigned char* payload;
    long long slot_capacity;
    unsigned char* peer_payload[SKML_MAX_PEERS];
    unsigned long long* peer_flag[SKML_MAX_PEERS];
    unsigned int* ctrl;
    unsigned int* run_vals;
    unsigned int* run_cnt;
    unsigned long long* run_w;
    unsigned int* splits_raw;
    unsigned int* warp_cnt;          // [grid * 32 warps][SKML_MAX_GROUPS]: keys of every group in every warp slice
    unsigned long long* blk_cnt;     // [SKML_MAX_GROUPS + 2][MAX_GRID]: the same per block, and its least and largest value (tagged)
    unsigned long long* blk_bytes;   // [SKML_MAX_GROUPS][MAX_GRID]: delta bytes of the chunks every block owns, per group (tagged)
    unsigned int* blk_flag;          // [grid]: epoch in which the block has published all of its counts
    unsigned short* chunk_part;      // [8 * chunks]: delta bytes of a chunk's eighths (128 keys)
    unsigned int* chunk_off;         // [2 * chunks]: delta-byte offset of a chunk inside its owner's part of the group
                                     // (delta_adaptive: flag-bit and delta-bit offsets)
    unsigned long long* blk_bits;    // delta_adaptive: [2 * SKML_MAX_GROUPS][2][MAX_GRID] flag bits / delta bits per block and group (tagged halves)
    unsigned int* blk_done;          // bit streams on several ranks: [grid] epoch in which the block finished writing its chunks
    unsigned int* key_hist;          // delta_adaptive: [SKML_MAX_GROUPS][32] keys per delta width, zeroed in S1
    int key_encoder;
    int huffman;                     // sketch tables travel Huffman-coded (cell_bits = 0)
    int sample_splits;               // split points from a sample every cluster draws alike (no S2, two grid barriers fewer)
    unsigned int* cell_hist;         // Huffman: [bin_num + groups] cells per symbol, zeroed in S1
    unsigned long long* blk_tbits;   // Huffman: [SKML_MAX_GROUPS][2][MAX_GRID] code bits per block (in the tables' turn) and group (tagged halves)
    unsigned int* tchunk_off;        // Huffman: [table chunks] bit offset of a chunk inside its owner's part of the stream
    unsigned short* bins;
    int* gkeys;                      // keys, grouped: group g's list starts at Layout::goff[g]
    unsigned int* tables;
    long long tables_cap;
    unsigned char* gcodes;           // insert in shared memory: rank codes of the keys, in the order of gkeys
    long long copies_cap;            // insert in shared memory: bytes of the tables' copies (they lie where `tables` does)
    int priv;                        // insert in shared memory: the launch's parameters allow it (see priv_layout)
    float priv_least[4], priv_parts; // and where it pays (priv_pays, priv_passes)
    unsigned int* status;
    long long budget;
    const float* given_splits;
    int n_given;
    float given_min, given_max;
    const float* dense_vals;                             // values of the dense kind (null: not this launch's business)
    long long n_value;                                   // count and kind when meta is null
    int kind_value;
    int zero_slot;                                       // clear the local slot first
    int decode_follows;                                  // whoever waits for the arrival flag is behind this launch on its stream
    unsigned long long* done_word;                       // pinned host word for the status (checked calls)
    unsigned long long done_seq;
    unsigned long long sample_rand;                      // draw behind the sample's offset (host: seed, step, rank)
    int mixers;                                          // every row of every group uses an integer mixer (<= 3 rows)
    unsigned char hash_ids[SKML_MAX_GROUPS][SKML_MAX_ROWS];  // hash rows of every group (host: seed, step, rank, group)
};

struct QInfo {
    int nsplits, bin_num, zero_idx, cell_bits;
    float minv, maxv;
    int edges[SKML_MAX_GROUPS];
};

struct Layout {
    unsigned int n_g[SKML_MAX_GROUPS];
    unsigned int col[SKML_MAX_GROUPS];
    unsigned int goff[SKML_MAX_GROUPS];            // start of the group's staging list (a multiple of 4 entries)
    unsigned int chunk_prefix[SKML_MAX_GROUPS + 1]; // chunks of the groups before, group-major chunk numbering
    unsigned int base_rank[SKML_MAX_GROUPS];       // keys of the group in the blocks before this one
    unsigned long long bytes_g[SKML_MAX_GROUPS];   // delta bytes of the group (block 0, for the header)
    unsigned long long flag_bits[SKML_MAX_GROUPS], delta_bits[SKML_MAX_GROUPS];  // delta_adaptive: stream lengths
    unsigned int num_iv[SKML_MAX_GROUPS], flag_kind[SKML_MAX_GROUPS];            // delta_adaptive: the groups' modes
    unsigned long long off_keys;                   // delta_adaptive: start of the per-group [flags | deltas] sections
    // Huffman-coded tables: symbol range, cells, present symbols, code bits, chunk numbering, stream / restart starts
    unsigned int sym_lo[SKML_MAX_GROUPS], nsym[SKML_MAX_GROUPS], cells[SKML_MAX_GROUPS], items[SKML_MAX_GROUPS];
    unsigned int tchunk_prefix[SKML_MAX_GROUPS + 1];
    unsigned long long tbits[SKML_MAX_GROUPS], tstream_off[SKML_MAX_GROUPS], trestart_off[SKML_MAX_GROUPS];
    unsigned long long table_off[SKML_MAX_GROUPS], flag_off[SKML_MAX_GROUPS], delta_off[SKML_MAX_GROUPS],
        restart_off[SKML_MAX_GROUPS], tab32_off[SKML_MAX_GROUPS];
    unsigned long long col_magic[SKML_MAX_GROUPS];  // ceil(2^64 / col) for the division-free modulo (other hash rows only)
    unsigned int recip[SKML_MAX_GROUPS];            // floor(2^32 / col) for the mixer-only hash path
    unsigned char hash_ids[SKML_MAX_GROUPS][SKML_MAX_ROWS];  // CP's, where the lanes of a warp may differ in the group
    unsigned long long unit_prefix[SKML_MAX_GROUPS + 1];  // 16-byte units of the narrow tables of the groups before
    // insert in shared memory (priv_layout): parts a row's cells are cut into, cells of a part, parts of the groups
    // before, the groups' first unit of work (four keys against one part), units per block, bytes of a copy
    unsigned int parts[SKML_MAX_GROUPS], part_len[SKML_MAX_GROUPS], part_prefix[SKML_MAX_GROUPS + 1];
    unsigned long long work_prefix[SKML_MAX_GROUPS + 1], work_per;
    unsigned int copy_stride;
    int priv;
    unsigned long long off_bv, off_gt, off_flags, off_restart, off_tables, off_deltas, total_bytes;
    int overflow;
};

struct WsLayout {
    long long ctrl, run_vals, run_cnt, run_w, splits_raw, warp_cnt, blk_cnt, blk_bytes, blk_flag, chunk_off, chunk_part, blk_bits, blk_done, key_hist, cell_hist, blk_tbits, tchunk_off, bins, gkeys, gcodes, tables,
        total;
    long long tables_cap, copies_cap;
};

static inline long long al256(long long x) { return (x + 255) & ~255ll; }

#define PRIV_MIN_KEYS 1250000    // least number of keys of an insert in shared memory (see priv_thresholds)
#define PRIV_MIN_ROOM 4000000    // insert in shared memory where only room for so many keys is known, not how many there are (see fill_params)
#define PRIV_UNITS 2             // units of four keys a thread inserts per round
#define PRIV_MAX_PARTS 2048      // parts of all groups' rows (their blocks are listed in shared memory)
#define PRIV_BYTES (136 * 1024)  // cells that fit a block's shared memory

// Keys from which on the insert in shared memory pays (priv_layout): it hashes a key once per row and part of the row
// (`passes`: parts a row on average), where an atomic per row and key has to be saved by it, and puts the keys and their codes
// into lists first, a fixed price and one per key. Whole calls, atomics / shared memory in us, eight groups of 250 buckets:
//   three rows: 1M keys 79 / 79, 1.5M 91 / 86, 2M 105 / 95, 4M 187 / 144; in two parts 2.5M 122 / 126, 3M 156 / 139, 10M 371 / 323;
//               in three 2.5M 130 / 151, 4M 205 / 193, 6M 268 / 255, 10M 383 / 384; in four 4M 215 / 224, 6M 277 / 293; tables of
//               10 MB, three parts 3M 131 / 153, 4M 160 / 187
//   two rows:   1M 68 / 73, 2M 91 / 93, 2.5M 103 / 101, 4M 139 / 134; in two parts 4M 136 / 146, 6M 192 / 183, 10M 292 / 274;
//               in three 10M 296 / 314
//   one row:    2M 76 / 86, 4M 108 / 122, 6M 151 / 144; in two parts 10M 215 / 227
// More than eight groups (the lists are made by ballots then): three rows, 1.5M 98 / 100, 2M 112 / 113, 3M 145 / 135; in two
// parts 4M 201 / 204, 10M 426 / 415. Tables of 32-bit cells that leave L2 make atomics dear: 72 MB 541 / 466, 120 MB 862 / 569.
// least[k]: keys from which on k + 1 passes pay.
static void priv_thresholds(long long rows, long long G, double col_ratio, float least[4]) {
    const double scale = G > 8 ? 1.6 : 1.0, bytes = 4.0 * (double)rows * (col_ratio > 1e-9 ? col_ratio : 1e-9);   // of 32-bit cells, a key
    const double one = rows >= 3 ? PRIV_MIN_KEYS : (rows == 2 ? 2.5e6 : 6e6), two = rows >= 3 ? 3e6 : 6e6, three = 24e6 / bytes > 4e6 ? 24e6 / bytes : 4e6;
    const double out = 64e6 / bytes > one * scale ? 64e6 / bytes : one * scale;
    least[0] = (float)(one * scale);
    least[1] = (float)(rows >= 2 && two * scale < out ? two * scale : out);
    least[2] = (float)(rows >= 3 && three * scale < out ? three * scale : out);
    least[3] = (float)out;
}
// `hashed` / `rows`: passes, a little above a whole number counting as that. A launch's start takes the groups to be alike
// (`slack` 1); once they are known the insert is given up only where it clearly does not pay, since the tables have to be
// cleared then.
static __host__ __device__ inline bool priv_pays(const float (&least)[4], float keys, float hashed, float rows, float slack) {
    const float parts = hashed - 0.25f * slack * rows;
    if (parts > 4.f * rows) return false;
    return keys * slack >= (parts <= rows ? least[0] : (parts <= 2.f * rows ? least[1] : (parts <= 3.f * rows ? least[2] : least[3])));
}
// Parts of a row if the groups are alike; `parts`: parts of a group that holds one key.
static __host__ __device__ inline float priv_passes(float keys, float parts) { return fmaxf(ceilf(keys * parts), 1.f); }

// Whether launches of these sizes may insert in shared memory: enough keys, rows of integer mixers only, codes of a byte.
static inline bool priv_sizes(long long n_max, long long q, long long rows, long long G, double col_ratio) {
    if (n_max < PRIV_MIN_KEYS || rows > 3 || q > 256) return false;
    float least[4];
    priv_thresholds(rows, G, col_ratio, least);
    return (float)n_max >= least[0];
}

// Bytes of the copies that blocks make of the parts they have worked on: at most one copy per block and part border.
static inline long long copies_bytes(long long n_max, long long G, long long rows, double col_ratio, long long grid) {
    const long long cells = (long long)(col_ratio * (double)n_max) + 2;
    const long long len = cells < PRIV_BYTES ? cells : PRIV_BYTES;
    return (grid + rows * (2 * cells / PRIV_BYTES + G)) * (len + 32);
}

// `priv`: with what the insert in shared memory takes, a byte a key and the copies. (It lies behind everything else but the
// tables.)
static WsLayout ws_layout(long long n_max, long long q, long long G, long long rows, double col_ratio, long long grid, bool priv) {
    WsLayout L;
    long long o = 0;
    L.ctrl = o; o += 256;
    L.run_vals = o; o += al256(grid * SK_K * 4);
    L.run_cnt = o; o += al256(grid * 4);
    L.run_w = o; o += al256(grid * 8);
    L.splits_raw = o; o += al256(q * 4);
    L.warp_cnt = o; o += al256(grid * SKML_WARPS * SKML_MAX_GROUPS * 4);
    L.blk_cnt = o; o += al256(MAX_GRID * (SKML_MAX_GROUPS + 2) * 8);
    L.blk_bytes = o; o += al256(MAX_GRID * SKML_MAX_GROUPS * 8);
    L.blk_flag = o; o += al256(grid * 4);
    L.chunk_off = o; o += al256((n_max / SKML_RESTART_INTERVAL + SKML_MAX_GROUPS + 8) * 8);
    L.chunk_part = o; o += al256((n_max / SKML_RESTART_INTERVAL + SKML_MAX_GROUPS + 8) * 16);
    L.blk_bits = o; o += al256(2 * SKML_MAX_GROUPS * 2 * MAX_GRID * 8);
    L.blk_done = o; o += al256(grid * 4);
    L.key_hist = o; o += al256(SKML_MAX_GROUPS * 32 * 4);
    L.cell_hist = o; o += al256((SKML_GPU_MAX_BINS + SKML_MAX_GROUPS) * 4);
    L.blk_tbits = o; o += al256(SKML_MAX_GROUPS * 2 * MAX_GRID * 8);
    L.tchunk_off = o; o += al256(((rows * ((long long)(col_ratio * (double)n_max) + 2 + G) + 64) / 1024 + SKML_MAX_GROUPS + 8) * 4);
    L.bins = o; o += al256(n_max * 2);
    L.gkeys = o; o += al256((n_max + 4 * SKML_MAX_GROUPS + 8) * 4);
    L.tables_cap = rows * ((long long)(col_ratio * (double)n_max) + 2 + G) + 64 + 4 * G;  // groups' tables start at multiples of 4 cells
    L.gcodes = o; o += priv ? al256(n_max + 4 * SKML_MAX_GROUPS + 8) : 0;
    L.copies_cap = priv ? copies_bytes(n_max, G, rows, col_ratio, grid) : 0;
    if (L.copies_cap < L.tables_cap * 4) L.copies_cap = L.tables_cap * 4;
    L.tables = o; o += al256(L.copies_cap);
    L.total = o;
    return L;
}

extern "C" long long skml_compress_workspace_bytes(long long n_max, long long bin_num, long long group_num,
                                                   long long row_num, double col_ratio, long long grid) {
    if (grid <= 0 || grid > MAX_GRID) grid = MAX_GRID;
    return ws_layout(n_max, bin_num, group_num, row_num, col_ratio, grid, priv_sizes(n_max, bin_num, row_num, group_num, col_ratio)).total;
}

extern "C" long long skml_compress_workspace_least(long long n_max, long long bin_num, long long group_num,
                                                   long long row_num, double col_ratio, long long grid) {
    if (grid <= 0 || grid > MAX_GRID) grid = MAX_GRID;
    return ws_layout(n_max, bin_num, group_num, row_num, col_ratio, grid, false).total;
}

// Upper bound of the payload size for n_max non-zeros (sparse kind) or dim codes (dense kind).
static __host__ __device__ inline long long payload_bound(long long n_max, long long dim, long long bin_num, long long group_num,
                                                          long long row_num, double col_ratio) {
    long long G = group_num, R = SKML_RESTART_INTERVAL;
    long long head = SKML_HEADER_BYTES + (long long)skml_align16(4 * bin_num) + SKML_GROUP_ENTRY_BYTES * G;
    long long flags = 17 * n_max / 8 + 24 * G + 16;   // delta_adaptive with unary flags: up to 17 flag bits per key
    long long restart = 16 * (n_max / R + G) + 16 * G;
    long long cells = row_num * ((long long)(col_ratio * (double)n_max) + 2 * G);
    // two bytes per cell cover 8/16-bit codes and any Huffman stream (at most 10 bits per cell); the
    // Huffman sections add their code books (12 bytes per symbol) and one restart offset per 128 cells
    long long tables = 2 * cells + 32 * G + 12 * (bin_num + G) + cells / 32 + 96 * G;
    long long deltas = 4 * n_max + 24 * G;
    long long sparse = head + flags + restart + tables + deltas + 64;
    long long dense = head + 2 * dim + 64;
    long long cap = sparse > dense ? sparse : dense;
    return (cap + 255) & ~255ll;
}

extern "C" long long skml_payload_capacity(long long n_max, long long dim, long long bin_num, long long group_num,
                                           long long row_num, double col_ratio) {
    return payload_bound(n_max, dim, bin_num, group_num, row_num, col_ratio);
}

// ---------------------------------------------------------------------------
// shared memory carve-up (dynamic, one block per SM)
// ---------------------------------------------------------------------------
// Per-warp scratch of the Huffman code construction.
struct HufScratch {
    unsigned int cnt[HUF_MAX_SYMS];       // cells per symbol
    unsigned int w[HUF_MAX_SYMS + 2];     // leaf weights, ascending; two more that are never the smaller ones
    unsigned int iw[HUF_MAX_SYMS + 2];    // weights of the internal nodes, in creation order (ascending), likewise
    unsigned short ord[HUF_MAX_SYMS];     // symbol of the i-th lightest leaf
    unsigned short pl[HUF_MAX_SYMS];      // parent (internal node) of every leaf
    unsigned short pi[HUF_MAX_SYMS];      // parent of every internal node
    unsigned int next[34];                // symbols per code length, then the next code word of every length
};

// The quantile stages (S1, S2) and the coding stage (S5) never hold data at the same time, so their
// arrays share one region: the smaller the block's shared memory, the more of the SM's 256 KB is left
// as L1 for the scatter and coding passes, which keep many loads in flight.
struct SmemQuantile {
    alignas(16) unsigned int tile[TILE];
    unsigned int levels[MAX_LEVELS][SK_K];
    unsigned int run[SK_K];
    unsigned int merge[2 * SK_K];
    unsigned int tail[SK_K];
    unsigned long long e_acc[SK_K];
    alignas(16) unsigned int runs_all[MAX_GRID * SK_K];   // S2: all blocks' runs; S1: scratch of the sort
    unsigned int runs_cnt[MAX_GRID];
    unsigned long long runs_w[MAX_GRID];
};
struct SmemCoding {
    unsigned int stage_f[4][AP_STAGE_F];            // delta_adaptive: one chunk's flag / delta bits per sub-block
    unsigned int stage_d[4][AP_STAGE_D];            // (also the staging of the Huffman table streams)
    unsigned char huf_len[SKML_GPU_MAX_BINS + SKML_MAX_GROUPS];   // Huffman: code length / code word per symbol slot
    unsigned int huf_code[SKML_GPU_MAX_BINS + SKML_MAX_GROUPS];
    HufScratch huf_scratch[8];
};

// S3's copy of the split points, laid out for upper_bounds_f (the quantile stages are over, coding has not begun).
struct SmemSearch {
    float a[SKML_GPU_MAX_BINS + SKML_GPU_MAX_BINS / 32];
};

// S5, plain key code: byte counts of a run of chunks (measuring), then every warp's delta bytes on their way out.
#define MEASURE_CHUNKS 2048  // chunks whose byte counts are kept in shared memory at a time
struct SmemPack {
    union {
        uint4 stage[SKML_WARPS][34];   // 128 keys of at most 4 bytes, at any offset in the first unit
        unsigned int tot[MEASURE_CHUNKS];
    };
};
static_assert(sizeof(SmemPack) <= offsetof(SmemCoding, huf_len), "the Huffman code tables outlive the key code's staging");

// S4, insert in shared memory: a warp's turn of 128 elements, put in the groups' order (rank code | group << 8).
struct SmemPart {
    unsigned int key[SKML_WARPS][128];
    unsigned short tag[SKML_WARPS][128];
};

struct Smem {
    float splits[SKML_GPU_MAX_BINS];               // stages S3..S6
    union {
        SmemQuantile qs;
        SmemCoding cs;
        SmemSearch ss;
        SmemPack ps;
        uint2 priv_blocks[PRIV_MAX_PARTS];         // merge of the copies: a part's first block and its number of blocks
        SmemPart part;
    };
    // stages S3..S6
    unsigned char grp_lut[SKML_GPU_MAX_BINS];      // bucket -> group
    unsigned char rank_lut[256], code_bin[256];    // insert in shared memory: bucket -> rank code, edge + rank code -> bucket
    QInfo qi;
    Layout lay;
    unsigned int wcnt[SKML_WARPS][SKML_MAX_GROUPS];
    unsigned int wbase[SKML_WARPS][SKML_MAX_GROUPS];
    unsigned long long my_bytes[SKML_MAX_GROUPS];   // delta bytes of the chunks this block owns, per group
    unsigned long long pre_bytes[SKML_MAX_GROUPS];  // the same, summed over the blocks before this one
    unsigned long long my_bits[2 * SKML_MAX_GROUPS], pre_bits[2 * SKML_MAX_GROUPS];  // delta_adaptive: flag / delta bits
    unsigned long long my_tbits[SKML_MAX_GROUPS], pre_tbits[SKML_MAX_GROUPS];
    unsigned int sub_part[4][8];                    // scan scratch of the four 256-thread sub-blocks
    unsigned int sub_total[4], sub_off[4];
    unsigned long long sums[5];                      // layout_from_counts: totals of its five prefix sums
    unsigned int scan[2][SKML_WARPS];                // block_rank scratch, alternating
    unsigned int row[SKML_MAX_GROUPS + 2];           // S3: the block's counts, least and largest value
    alignas(16) SkmlHeader hdr;                      // copied out in 16-byte units
    int flag;
};


// 164 KB is a shared-memory carve-out step of the SM: staying under it (with the block's static shared
// memory and the 1 KB the system reserves) leaves 92 KB of L1; measured, the scatter + insert stage of
// 2.3M keys takes 69 us with that L1 and 120 us with the 28 KB that the next step (228 KB) leaves.
static_assert(2 * TILE + SKML_GPU_MAX_BINS <= MAX_GRID * SK_K, "S1: the sort's scratch, the split points, the other half");
static_assert(offsetof(Smem, hdr) % 16 == 0, "the header is read in 16-byte units");
static_assert(sizeof(Smem) <= 162 * 1024, "the compress kernels' shared memory must stay below the 164 KB carve-out");

// Insert in shared memory: the cells lie behind the first 256 split points (all there are with codes of a byte) and in
// the stages' shared region.
#define PRIV_SPLITS 256
static_assert(offsetof(Smem, qs) == SKML_GPU_MAX_BINS * 4, "the cells need one piece of shared memory");
static_assert(offsetof(Smem, grp_lut) - PRIV_SPLITS * 4 >= PRIV_BYTES && PRIV_BYTES % 16 == 0, "room for the cells");

__device__ __forceinline__ unsigned int lanemask_lt() {
    unsigned int m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Control words (u32): [1] launches so far; [2] blocks that are done (finish_publish); from ctrl_set on, four words of one
// launch: arrivals of its grid barriers, and the minimum (inverted) and maximum of its values. Launches take one of two
// sets in turn, and a launch clears the set of the next one, so none has to wait at its end until everyone is done with its own.
__device__ __forceinline__ unsigned int* ctrl_set(unsigned int* ctrl, unsigned int epoch) { return ctrl + 4 + 4 * (epoch & 1u); }
enum { CTRL_BAR = 0, CTRL_MIN = 1, CTRL_MAX = 2 };

// A launch's first words: `epoch` names it. The set behind it is nobody's now (its last user has ended).
template <bool FUSED>
__device__ __forceinline__ unsigned int ctrl_open(unsigned int* ctrl) {
    const unsigned int epoch = ld_relaxed_gpu(&ctrl[1]) + 1u;
    if (FUSED && blockIdx.x == 0 && threadIdx.x < 4) ctrl_set(ctrl, epoch + 1u)[threadIdx.x] = 0u;
    return epoch;
}
// Behind a grid barrier: every block has read the number.
__device__ __forceinline__ void ctrl_advance(unsigned int* ctrl, unsigned int epoch) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st_relaxed_gpu(&ctrl[1], epoch);
}

// Block 0 leaves a nanosecond time stamp per stage in the control words (u64 at ctrl[16 + 2 i]);
// skml tools read them to show where a fused launch spends its time.
__device__ __forceinline__ void stage_stamp(unsigned int* ctrl, int i) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        reinterpret_cast<unsigned long long*>(ctrl)[8 + i] = t;
    }
}

// Clears the local slot from byte `from` (a multiple of 16) on, in 16-byte units; a capacity that is no multiple of 16
// keeps its last bytes to the tail. Nothing orders the callers' stores against those of other blocks: bytes that
// another block writes in the same launch need a grid barrier in between.
__device__ __noinline__ void clear_slot(const CP& p, long long from, long long gid, long long gsz) {
    uint4* z4 = reinterpret_cast<uint4*>(p.payload);
    for (long long i = from / 16 + gid; i < p.slot_capacity / 16; i += gsz) __stcs(z4 + i, make_uint4(0, 0, 0, 0));
    if (gid < (p.slot_capacity & 15)) p.payload[(p.slot_capacity & ~15ll) + gid] = 0;
}

// ---------------------------------------------------------------------------
// S1: quantile summary
// ---------------------------------------------------------------------------
// Merge the sorted runs a[128] and b[128] into s.qs.merge (ascending) with a bitonic merge.
__device__ __forceinline__ void merge_runs(Smem& s, const unsigned int* a, const unsigned int* b) {
    for (int t = threadIdx.x; t < SK_K; t += blockDim.x) {
        s.qs.merge[t] = a[t];
        s.qs.merge[2 * SK_K - 1 - t] = b[t];
    }
    __syncthreads();
    for (int j = SK_K; j > 0; j >>= 1) {
        for (int t = threadIdx.x; t < SK_K; t += blockDim.x) {
            int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
            unsigned int x = s.qs.merge[i], y = s.qs.merge[i | j];
            if (x > y) {
                s.qs.merge[i] = y;
                s.qs.merge[i | j] = x;
            }
        }
        __syncthreads();
    }
}

// Carry s.qs.run (weight TILE_W << level0) up the level chain.
__device__ __forceinline__ void carry_run(Smem& s, unsigned int& occupied, int level, const CP& p, unsigned long long salt) {
    while (true) {
        if (!(occupied & (1u << level))) {
            for (int t = threadIdx.x; t < SK_K; t += blockDim.x) s.qs.levels[level][t] = s.qs.run[t];
            occupied |= 1u << level;
            __syncthreads();
            return;
        }
        merge_runs(s, s.qs.levels[level], s.qs.run);
        unsigned int off = (unsigned int)(skml_rand(p.seed, p.step, ((unsigned long long)p.rank << 32) | blockIdx.x,
                                                    salt * 64 + level) & 1u);
        for (int t = threadIdx.x; t < SK_K; t += blockDim.x) s.qs.run[t] = s.qs.merge[2 * t + off];
        occupied &= ~(1u << level);
        __syncthreads();
        ++level;
        if (level >= MAX_LEVELS) return;  // unreachable for n < 2^31
    }
}

// The block's share of the values -> one run of at most SK_K samples in s.qs.tile[0, cnt) with weight w.
__device__ void summarize_slice(const CP& p, Smem& s, unsigned int* set, const float* __restrict__ vals, long long n, unsigned int& run_cnt,
                                unsigned long long& run_w) {
    run_cnt = 0;
    run_w = 0;
    // Bottom-level sampler (as in KLL sketches): of every f consecutive values one is kept at random
    // with weight f, so one 2048-sort covers f * 2048 values and enters the level chain as one run
    // of weight 16 f. f is the smallest power of two (<= MAX_SAMPLE) for which every block has one
    // sort to do; min and max still see every value.
    const long long ntiles = (n + TILE - 1) / TILE;
    int f = 1, lf = 0;
    while (f < MAX_SAMPLE && ntiles > (long long)f * gridDim.x) {
        f <<= 1;
        ++lf;
    }
    const long long ST = (long long)f * TILE;
    const long long nst = (n + ST - 1) / ST;
    const long long t0 = blockIdx.x;  // super tiles are dealt round-robin: t0, t0 + grid, ...
    if (t0 >= nst || n <= 0) return;
    unsigned int occupied = 0;
    int tail_cnt = 0;
    unsigned long long tail_w = 0;
    unsigned int kmin = 0xFFFFFFFFu, kmax = 0u;
    const unsigned long long salt0 = p.seed ^ (p.step * 0x9E3779B97F4A7C15ull) ^ ((unsigned long long)p.rank << 40);
    for (long long st = t0; st < nst; st += gridDim.x) {
        const long long base = st * ST;
        const long long m = (n - base) < ST ? (n - base) : ST;  // values of this super tile
        if (m == ST) {
            for (int t = threadIdx.x; t < TILE; t += blockDim.x) {
                const float* src = vals + base + (long long)t * f;
                const unsigned int pick = (unsigned int)(skml_splitmix64(salt0 ^ (unsigned long long)(base + t)) >> 40) & (unsigned int)(f - 1);
                unsigned int chosen = 0;
                if (f == 1) {
                    chosen = f2ord(src[0]);
                    kmin = min(kmin, chosen);
                    kmax = max(kmax, chosen);
                } else if (f == 2) {
                    const float2 q = *reinterpret_cast<const float2*>(src);
                    const unsigned int k0 = f2ord(q.x), k1 = f2ord(q.y);
                    kmin = min(kmin, min(k0, k1));
                    kmax = max(kmax, max(k0, k1));
                    chosen = pick ? k1 : k0;
                } else {
                    for (int j = 0; j < f / 4; ++j) {
                        const float4 q = reinterpret_cast<const float4*>(src)[j];
                        const unsigned int k0 = f2ord(q.x), k1 = f2ord(q.y), k2 = f2ord(q.z), k3 = f2ord(q.w);
                        kmin = min(min(kmin, k0), min(min(k1, k2), k3));
                        kmax = max(max(kmax, k0), max(max(k1, k2), k3));
                        if ((int)(pick >> 2) == j) {
                            const unsigned int r = pick & 3u;
                            chosen = r == 0 ? k0 : (r == 1 ? k1 : (r == 2 ? k2 : k3));
                        }
                    }
                }
                s.qs.tile[t] = chosen;
            }
            __syncthreads();
            if (st == t0) stage_stamp(p.ctrl, 10);
            block_sort_2048(s.qs.tile, s.qs.runs_all);
            if (st == t0) stage_stamp(p.ctrl, 11);
            const unsigned int off = (unsigned int)(skml_rand(p.seed, p.step, ((unsigned long long)p.rank << 32) | blockIdx.x,
                                                              0x7200u + (unsigned long long)((st - t0) / gridDim.x)) & (TILE_W - 1));
            for (int t = threadIdx.x; t < SK_K; t += blockDim.x) s.qs.run[t] = s.qs.tile[t * TILE_W + off];
            __syncthreads();
            carry_run(s, occupied, lf, p, (unsigned long long)((st - t0) / gridDim.x) + 1);
            continue;
        }
        // the last, partial super tile of the whole input: slot t samples the valid part of its f values
        const int ms = (int)((m + f - 1) / f);  // slots that hold a value
        for (int t = threadIdx.x; t < TILE; t += blockDim.x) {
            unsigned int chosen = 0xFFFFFFFFu;
            const long long g0 = base + (long long)t * f;
            if (g0 < n) {
                const int valid = (int)((n - g0) < f ? (n - g0) : f);
                const unsigned int pick = (unsigned int)((skml_splitmix64(salt0 ^ (unsigned long long)(base + t)) >> 40) % (unsigned int)valid);
                for (int j = 0; j < valid; ++j) {
                    const unsigned int k = f2ord(vals[g0 + j]);
                    kmin = min(kmin, k);
                    kmax = max(kmax, k);
                    if ((unsigned int)j == pick) chosen = k;
                }
            }
            s.qs.tile[t] = chosen;
        }
        __syncthreads();
        block_sort_2048(s.qs.tile, s.qs.runs_all);
        int stride = 1;
        while ((ms + stride - 1) / stride > SK_K) stride <<= 1;
        tail_cnt = (ms + stride - 1) / stride;
        const unsigned int off = stride > 1 ? (unsigned int)(skml_rand(p.seed, p.step, p.rank, 0x7100u) % stride) : 0u;
        for (int t = threadIdx.x; t < tail_cnt; t += blockDim.x) {
            int idx = t * stride + (int)off;
            if (idx > ms - 1) idx = ms - 1;
            s.qs.tail[t] = s.qs.tile[idx];
        }
        tail_w = (((unsigned long long)m) << FP_SHIFT) / (unsigned long long)tail_cnt;
        __syncthreads();
    }
    stage_stamp(p.ctrl, 12);
    // block min / max -> global (stored so that an all-zero word means "nothing yet")
    {
        unsigned int a = kmin, b = kmax;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = min(a, __shfl_xor_sync(0xFFFFFFFFu, a, o));
            b = max(b, __shfl_xor_sync(0xFFFFFFFFu, b, o));
        }
        // one pair of atomics per block: thousands of same-address atomics would serialise in L2
        __shared__ unsigned int s_mn[SKML_WARPS], s_mx[SKML_WARPS];
        if ((threadIdx.x & 31) == 0) {
            s_mn[threadIdx.x >> 5] = a;
            s_mx[threadIdx.x >> 5] = b;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            a = s_mn[threadIdx.x];
            b = s_mx[threadIdx.x];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                a = min(a, __shfl_xor_sync(0xFFFFFFFFu, a, o));
                b = max(b, __shfl_xor_sync(0xFFFFFFFFu, b, o));
            }
            if (threadIdx.x == 0) {
                atomicMax(&set[CTRL_MIN], ~a);
                atomicMax(&set[CTRL_MAX], b);
            }
        }
    }
    stage_stamp(p.ctrl, 13);
    // collapse the levels (+ tail) into one run (the sort buffer is free now)
    int nruns = __popc(occupied) + (tail_cnt > 0 ? 1 : 0);
    unsigned int* out = s.qs.tile;
    if (nruns == 1) {
        const unsigned int* src;
        int cnt;
        unsigned long long w;
        if (tail_cnt > 0) {
            src = s.qs.tail; cnt = tail_cnt; w = tail_w;
        } else {
            int lv = __ffs(occupied) - 1;
            src = s.qs.levels[lv]; cnt = SK_K; w = ((unsigned long long)TILE_W << lv) << FP_SHIFT;
        }
        for (int t = threadIdx.x; t < cnt; t += blockDim.x) out[t] = src[t];
        run_cnt = (unsigned int)cnt;
        run_w = w;
        return;
    }
    // several runs: exclusive cumulative weight of every sample, then 128 mid-rank samples
    unsigned long long Wc = 0;
    for (int lv = 0; lv < MAX_LEVELS; ++lv)
        if (occupied & (1u << lv)) Wc += (unsigned long long)SK_K * (((unsigned long long)TILE_W << lv) << FP_SHIFT);
    Wc += (unsigned long long)tail_cnt * tail_w;
    const int total_samples = __popc(occupied) * SK_K + tail_cnt;
    for (int sidx = threadIdx.x; sidx < total_samples; sidx += blockDim.x) {
        // locate (run a, index i): occupied levels in ascending order, then the tail
        int a = -1, i = sidx, seen = 0;
        for (int lv = 0; lv < MAX_LEVELS; ++lv) {
            if (!(occupied & (1u << lv))) continue;
            if (i < SK_K) { a = lv; break; }
            i -= SK_K;
            ++seen;
        }
        const unsigned int value = a >= 0 ? s.qs.levels[a][i] : s.qs.tail[i];
        const unsigned long long wa = a >= 0 ? (((unsigned long long)TILE_W << a) << FP_SHIFT) : tail_w;
        unsigned long long e = (unsigned long long)i * wa;
        for (int lv = 0; lv < MAX_LEVELS; ++lv) {
            if (!(occupied & (1u << lv)) || lv == a) continue;
            unsigned long long wl = ((unsigned long long)TILE_W << lv) << FP_SHIFT;
            bool before = a < 0 || lv < a;  // runs earlier in the order win ties
            int c = before ? upper_bound_u(s.qs.levels[lv], SK_K, value) : lower_bound_u(s.qs.levels[lv], SK_K, value);
            e += (unsigned long long)c * wl;
        }
        if (tail_cnt > 0 && a >= 0) e += (unsigned long long)lower_bound_u(s.qs.tail, tail_cnt, value) * tail_w;
        // targets t_j = (2j+1) * Wc / 256, j = 0..127, covered iff e <= t_j < e + wa
        long long j = (long long)((e << 7) / Wc) - 1;
        if (j < 0) j = 0;
        for (; j < SK_K; ++j) {
            unsigned long long tj = ((unsigned long long)(2 * j + 1) * (Wc >> 8));
            if (tj < e) continue;
            if (tj >= e + wa) break;
            out[j] = value;
        }
        (void)seen;
    }
    run_cnt = SK_K;
    run_w = Wc / SK_K;
}

// --- thread-block cluster primitives (distributed shared memory) ---
__device__ __forceinline__ unsigned int cluster_ctarank() {
    unsigned int r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned int cluster_nctarank() {
    unsigned int r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// hardware barrier of the cluster's blocks (blocks that have exited count as arrived)
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared-memory address of `ptr` (a location in this block's shared memory) in block `rank` of the cluster
__device__ __forceinline__ unsigned int dsmem_addr(const void* ptr, unsigned int rank) {
    const unsigned int a = (unsigned int)__cvta_generic_to_shared(ptr);
    unsigned int r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ unsigned int ld_dsmem_u32(unsigned int addr) {
    unsigned int v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_dsmem_u64(unsigned int addr) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}

// Two weighted runs a (s.qs.tile[0, ca), weight wa) and b (s.qs.tile[SK_K, SK_K + cb), weight wb) -> SK_K samples
// at the mid ranks (2j + 1) / (2 SK_K) of their union, left in s.qs.tile[0, SK_K); returns the new weight.
__device__ unsigned long long merge_two_runs(Smem& s, unsigned int ca, unsigned long long wa, unsigned int cb,
                                             unsigned long long wb) {
    const unsigned int* a = s.qs.tile;
    const unsigned int* b = s.qs.tile + SK_K;
    const unsigned long long Wc = (unsigned long long)ca * wa + (unsigned long long)cb * wb;
    for (unsigned int sidx = threadIdx.x; sidx < ca + cb; sidx += blockDim.x) {
        const bool from_a = sidx < ca;
        const unsigned int i = from_a ? sidx : sidx - ca;
        const unsigned int value = from_a ? a[i] : b[i];
        const unsigned long long w = from_a ? wa : wb;
        // weight in front of the sample; run a wins ties
        const unsigned long long e = (unsigned long long)i * w +
            (from_a ? (unsigned long long)lower_bound_u(b, (int)cb, value) * wb : (unsigned long long)upper_bound_u(a, (int)ca, value) * wa);
        long long j = (long long)((e << 7) / Wc) - 1;
        if (j < 0) j = 0;
        for (; j < SK_K; ++j) {
            const unsigned long long tj = (unsigned long long)(2 * j + 1) * (Wc >> 8);
            if (tj < e) continue;
            if (tj >= e + w) break;
            s.qs.merge[j] = value;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < SK_K; t += blockDim.x) s.qs.tile[t] = s.qs.merge[t];
    __syncthreads();
    return Wc / SK_K;
}

// S1: every block summarises its share of the values; the blocks of a thread-block cluster then merge
// their runs in shared memory (the cluster's first block reads the others' runs through distributed
// shared memory) and only the merged run goes to global memory, so S2 has 1 / cluster-size as many runs
// to load and to rank against. Launched without clusters the cluster is the block itself.
__device__ __noinline__ void stage_summary(const CP& p, Smem& s, unsigned int* set, const float* __restrict__ vals, long long n) {
    __shared__ unsigned int s_pub_cnt;
    __shared__ unsigned long long s_pub_w;
    unsigned int cnt;
    unsigned long long w;
    summarize_slice(p, s, set, vals, n, cnt, w);
    const unsigned int cs = cluster_nctarank(), cr = cluster_ctarank();
    if (threadIdx.x == 0) {
        s_pub_cnt = cnt;
        s_pub_w = w;
    }
    __syncthreads();
    if (cs > 1) {
        cluster_sync_all();   // every block's run, count and weight are in its shared memory
        if (cr == 0) {
            for (unsigned int r = 1; r < cs; ++r) {
                const unsigned int cb = ld_dsmem_u32(dsmem_addr(&s_pub_cnt, r));
                const unsigned long long wb = ld_dsmem_u64(dsmem_addr(&s_pub_w, r));
                if (cb == 0 || cb > SK_K) continue;   // uniform over the block
                const unsigned int src = dsmem_addr(s.qs.tile, r);
                unsigned int* dst = cnt ? s.qs.tile + SK_K : s.qs.tile;
                for (unsigned int t = threadIdx.x; t < cb; t += blockDim.x) dst[t] = ld_dsmem_u32(src + 4u * t);
                __syncthreads();
                if (cnt == 0) {
                    cnt = cb;
                    w = wb;
                } else {
                    w = merge_two_runs(s, cnt, w, cb, wb);
                    cnt = SK_K;
                }
            }
        } else {
            cnt = 0;   // this block's samples travel in the first block's run
            w = 0;
        }
        cluster_sync_all();   // nobody reads the others' shared memory any more
    }
    unsigned int* out = p.run_vals + (long long)blockIdx.x * SK_K;
    for (unsigned int t = threadIdx.x; t < cnt; t += blockDim.x) out[t] = s.qs.tile[t];
    if (threadIdx.x == 0) {
        p.run_cnt[blockIdx.x] = cnt;
        p.run_w[blockIdx.x] = w;
    }
}

// Warp-wide exclusive prefix sum; `total` = the warp's sum.
__device__ __forceinline__ unsigned long long warp_prefix(unsigned long long v, unsigned long long& total) {
    const int lane = threadIdx.x & 31;
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    return inc - v;
}

// S1, sample form. Every thread-block cluster draws the SAME stratified sample of the values (one value
// per stride of n / m positions, the offset a function of (seed, step, rank)), so every block ends up with
// the same split points without a grid barrier and without S2. The two blocks of a cluster sort one half
// of a 4096-value sample each and leave it in the other's shared memory, too: split t is the
// value of rank floor(m (t + 1) / q) in the union of the two sorted halves, found by a merge-path search
// over both. Without clusters a block sorts 2048 values alone.
// The rank error of a split is that of an m-value sample (standard deviation at most 0.8 % of n at
// m = 4096), the same order as the k = 128 summary's; inputs of up to m values are summarised exactly.
// Minimum and maximum of ALL values are taken by the count stage, which reads every value anyway.
// The splits stay in the block's shared memory (raw_splits); block 0 also leaves them in the workspace.
__device__ __forceinline__ unsigned int* raw_splits(Smem& s) { return s.qs.runs_all + TILE; }

// x mod n, n < 2^31: the upper half reduced first, then a quotient in double, one off at most.
__device__ __forceinline__ unsigned int mod_u64(unsigned long long x, unsigned int n) {
    const unsigned long long y = ((unsigned long long)((unsigned int)(x >> 32) % n) << 32) | (unsigned int)x;   // below n 2^32
    const unsigned long long q = (unsigned long long)((double)y * __drcp_rn((double)n));
    long long r = (long long)(y - q * n);
    if (r < 0) r += n;
    if (r >= (long long)n) r -= n;
    return (unsigned int)r;
}

// Where sample t of this block's half lies (below n), and how large sample and half are.
struct SamplePlace {
    int lh, half, m;            // log2 of the halves, which one, sample size
    unsigned long long off;
    __device__ __forceinline__ long long at(int t, long long n) const {   // -1: none
        const long long j = ((long long)t << lh) + half;
        if (j >= m) return -1;
        // m is a power of two (TILE * halves) whenever it is not n itself
        return n > m ? (long long)(((unsigned long long)j * (unsigned long long)n + off) >> (11 + lh)) : j;
    }
};
__device__ __forceinline__ SamplePlace sample_place(const CP& p, long long n) {
    SamplePlace f;
    f.lh = cluster_nctarank() >= 2 ? 1 : 0;
    f.half = (int)cluster_ctarank() & ((1 << f.lh) - 1);
    const int M = TILE << f.lh;
    f.m = n < M ? (int)n : M;
    f.off = n > f.m ? mod_u64(p.sample_rand, (unsigned int)n) : 0u;
    return f;
}

__device__ void stage_sample_splits(const CP& p, Smem& s, const float* __restrict__ vals, long long n) {
    const SamplePlace f = sample_place(p, n);
    const int m = f.m, mine = (m - f.half + (1 << f.lh) - 1) >> f.lh, theirs = m - mine;   // samples in this block's half, and the other
    if (f.lh) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this block runs: its shared memory may be written
#pragma unroll
    for (int t = threadIdx.x; t < TILE; t += SKML_BLOCK) {
        const long long pos = f.at(t, n);
        s.qs.tile[t] = pos >= 0 ? f2ord(__ldg(vals + pos)) : 0xFFFFFFFFu;
    }
    __syncthreads();
    // the other block's sorted half arrives behind the split points, which nothing else uses
    unsigned int* const their = raw_splits(s) + SKML_GPU_MAX_BINS;
    unsigned int remote = 0;
    if (f.lh) {
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        remote = dsmem_addr(their, (unsigned int)f.half ^ 1u);
    }
    block_sort_2048(s.qs.tile, s.qs.runs_all, remote);
    if (f.lh) cluster_sync_all();   // both halves are in both blocks
    const double inv_q = 1.0 / (double)p.q;
    for (int t = threadIdx.x; t < p.q - 1; t += blockDim.x) {
        int k = (int)((double)m * ((double)(t + 1) * inv_q));   // target rank in the sample (m <= 4096)
        if (k > m - 1) k = m - 1;
        // i = how many of the k values before the answer come from this block's half (ties: this half first)
        int lo = k - theirs > 0 ? k - theirs : 0, hi = k < mine ? k : mine;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const int j = k - mid;
            const bool ok = j >= theirs || s.qs.tile[mid - 1] <= their[j];
            if (ok) lo = mid;
            else hi = mid - 1;
        }
        const int j = k - lo;
        const unsigned int a = lo < mine ? s.qs.tile[lo] : 0xFFFFFFFFu;
        const unsigned int b = j < theirs ? their[j] : 0xFFFFFFFFu;
        const unsigned int key = a < b ? a : b;
        raw_splits(s)[t] = key;
        if (blockIdx.x == 0) p.splits_raw[t] = key;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// S2: weighted-rank query over all published runs -> splits_raw[q-1] (ordered keys)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long rank_target(long long n, int t, double inv_q) {
    unsigned long long r = (unsigned long long)((double)n * ((double)(t + 1) * inv_q));
    if (r > (unsigned long long)(n - 1)) r = (unsigned long long)(n - 1);
    return r << FP_SHIFT;
}

__device__ __noinline__ void stage_query(const CP& p, Smem& s, long long n) {
    if (n <= 0) return;
    const int nb = gridDim.x;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        s.qs.runs_cnt[t] = p.run_cnt[t];
        s.qs.runs_w[t] = p.run_w[t];
    }
    __syncthreads();
    {
        // all published runs -> shared memory, 16 bytes per load and several loads in flight per thread
        const uint4* src = reinterpret_cast<const uint4*>(p.run_vals);
        const int nv = nb * (SK_K / 4);
        for (int t0 = threadIdx.x; t0 < nv; t0 += 4 * blockDim.x) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int t = t0 + u * blockDim.x;
                // runs that a cluster merged away are empty: nothing to fetch
                v[u] = (t < nv && (4 * t) % SK_K < (int)s.qs.runs_cnt[(4 * t) / SK_K]) ? ld_cg_v4(src + t) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int t = t0 + u * blockDim.x;
                if (t >= nv) continue;
                const int c = (4 * t) / SK_K, i = (4 * t) % SK_K, cnt = (int)s.qs.runs_cnt[c];
                s.qs.runs_all[4 * t] = i < cnt ? v[u].x : 0xFFFFFFFFu;
                s.qs.runs_all[4 * t + 1] = i + 1 < cnt ? v[u].y : 0xFFFFFFFFu;
                s.qs.runs_all[4 * t + 2] = i + 2 < cnt ? v[u].z : 0xFFFFFFFFu;
                s.qs.runs_all[4 * t + 3] = i + 3 < cnt ? v[u].w : 0xFFFFFFFFu;
            }
        }
    }
    __syncthreads();
    // total weight: every warp sums a strided share, lanes combine by shuffle (all threads need it)
    unsigned long long Wtot = 0;
    for (int c = threadIdx.x & 31; c < nb; c += 32) Wtot += (unsigned long long)s.qs.runs_cnt[c] * s.qs.runs_w[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) Wtot += __shfl_xor_sync(0xFFFFFFFFu, Wtot, o);
    const double inv_q = 1.0 / (double)p.q;
    const int i = threadIdx.x & (SK_K - 1), part = threadIdx.x / SK_K, parts = blockDim.x / SK_K;
    for (int c = blockIdx.x; c < nb; c += gridDim.x) {
        const int cnt = (int)s.qs.runs_cnt[c];
        if (cnt == 0) continue;  // uniform over the block
        if (threadIdx.x < SK_K) s.qs.e_acc[threadIdx.x] = 0ull;
        __syncthreads();
        if (i < cnt) {
            const unsigned int value = s.qs.runs_all[c * SK_K + i];
            unsigned long long e = 0;
            for (int c2 = part; c2 < nb; c2 += parts) {
                int cnt2 = (int)s.qs.runs_cnt[c2];
                if (cnt2 == 0) continue;
                int k;
                if (c2 == c) k = i;
                else if (c2 < c) k = upper_bound_u(s.qs.runs_all + c2 * SK_K, cnt2, value);
                else k = lower_bound_u(s.qs.runs_all + c2 * SK_K, cnt2, value);
                e += (unsigned long long)k * s.qs.runs_w[c2];
            }
            atomicAdd(&s.qs.e_acc[i], e);
        }
        __syncthreads();
        if (threadIdx.x < cnt) {
            const unsigned int value = s.qs.runs_all[c * SK_K + threadIdx.x];
            const unsigned long long e = s.qs.e_acc[threadIdx.x], w = s.qs.runs_w[c];
            const bool last = e + w >= Wtot;
            // smallest t with target >= e
            int lo = 0, hi = p.q - 1;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (rank_target(n, mid, inv_q) >= e) hi = mid;
                else lo = mid + 1;
            }
            for (int t = lo; t < p.q - 1; ++t) {
                unsigned long long r = rank_target(n, t, inv_q);
                if (!last && r >= e + w) break;
                p.splits_raw[t] = value;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// S3 prelude: unique splits, zero bucket, group edges (every block, in shared memory)
// ---------------------------------------------------------------------------
// Positions of the kept items of one round of blockDim items (thread order), and how many of them are
// negative: one block barrier. `par` alternates between calls.
__device__ __forceinline__ unsigned int block_rank(Smem& s, int par, bool keep, bool neg, unsigned int& total, unsigned int& total_neg) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int km = __ballot_sync(0xFFFFFFFFu, keep), nm = __ballot_sync(0xFFFFFFFFu, keep && neg);
    if (lane == 0) s.scan[par][warp] = (unsigned int)__popc(km) | ((unsigned int)__popc(nm) << 16);
    __syncthreads();
    const unsigned int c = s.scan[par][lane];
    const unsigned int all = __reduce_add_sync(0xFFFFFFFFu, c), before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? c & 0xFFFFu : 0u);
    total = all & 0xFFFFu;
    total_neg = all >> 16;
    return before + (unsigned int)__popc(km & lanemask_lt());
}

// Distinct splits, zero bucket and group edges, in the shared memory of every block.
// in_smem: the raw split points are in raw_splits(s) (sample form, same launch), otherwise in the workspace.
// minmax_ready = false: the minimum and maximum of the values are not known yet (sample form before the
// count stage has run); the zero bucket does not need them (see below), set_minmax follows later.
__device__ void load_quantizer(const CP& p, Smem& s, const unsigned int* set, bool in_smem = false, bool minmax_ready = true) {
    const bool given = p.given_splits != nullptr;
    const int nraw = given ? p.n_given : p.q - 1;
    auto raw = [&](int i) { return given ? p.given_splits[i] : ord2f(in_smem ? raw_splits(s)[i] : __ldcg(p.splits_raw + i)); };
    unsigned int base = 0, negs = 0;
    int par = 0;
    for (int b = 0; b < nraw; b += blockDim.x, par ^= 1) {
        const int i = b + threadIdx.x;
        float v = 0.f;
        bool keep = false;
        if (i < nraw) {
            v = raw(i);
            keep = i == 0 || v != raw(i - 1);
        }
        unsigned int total, total_neg;
        const unsigned int pos = block_rank(s, par, keep, v < 0.f, total, total_neg);
        if (keep) s.splits[base + pos] = v;
        base += total;
        negs += total_neg;
    }
    if (threadIdx.x < 32) {
        QInfo& q = s.qi;
        const int lane = threadIdx.x, bin_num = (int)base + 1, G = p.G;
        float minv = 0.f, maxv = 0.f;
        if (given) {
            minv = p.given_min;
            maxv = p.given_max;
        } else if (minmax_ready) {
            minv = ord2f(~__ldcg(set + CTRL_MIN));
            maxv = ord2f(__ldcg(set + CTRL_MAX));
        }
        // The splits ascend, so the zero bucket (the first whose upper split is not negative) is their number of
        // negative ones. With splits taken from the data, min > 0 means every split is positive and max < 0 that
        // every split is negative, so that count gives the first two cases' answers too; they stay for given splits.
        int z = (int)negs;
        if ((given || minmax_ready) && minv > 0.f) z = 0;
        else if ((given || minmax_ready) && maxv < 0.f) z = bin_num - 1;
        // group edges as skml_group_edges, one lane per group: from the third group on an edge is the one before it
        // plus a constant, cut at bin_num
        int edge = bin_num;
        if (G == 2 && lane == 0) edge = z;
        if (G > 2 && lane < G - 1) {
            int bpg = bin_num / G;
            if (bpg < 1) bpg = 1;
            const int rem = z % bpg;
            const int e0 = z < bpg ? z : (rem < bpg / 2 ? bpg + rem : rem);
            edge = lane == 0 ? e0 : min(e0 + lane * bpg, bin_num);
        }
        if (lane < G) q.edges[lane] = edge;
        if (lane == 0) {
            q.nsplits = (int)base;
            q.bin_num = bin_num;
            q.cell_bits = bin_num <= 256 ? 8 : 16;
            q.minv = minv;
            q.maxv = maxv;
            q.zero_idx = z;
            // NaN or infinite gradient values cannot be bucketized (the reference's sketch throws on NaN)
            if (!isfinite(minv) || !isfinite(maxv)) skml_set_status(p.status, SKML_BAD_INPUT, 0x35u);
        }
    }
    __syncthreads();
}

// Sample form, once the values have all been looked at: their minimum or maximum, as order-preserving keys (one thread;
// the caller has a block barrier after it).
__device__ __forceinline__ void set_extreme(const CP& p, Smem& s, bool least, unsigned int key) {
    const float v = ord2f(key);
    if (least) s.qi.minv = v;
    else s.qi.maxv = v;
    if (!isfinite(v)) skml_set_status(p.status, SKML_BAD_INPUT, 0x35u);
}

// What a block tells the others of its counts: word i of all blocks lies in words[i * MAX_GRID ...], the count below the
// number of the launch (none in staged launches, where a launch's end is the barrier), so that whoever reads the number has
// the count with it. By one warp, behind a block barrier; the block's earlier stores come before it.
template <bool FUSED>
__device__ __forceinline__ void publish_row(unsigned long long* words, const unsigned int* row, int count, unsigned int epoch) {
    if (FUSED) __threadfence();
    for (int i = threadIdx.x & 31; i < count; i += 32) st_relaxed_gpu64(words + i * MAX_GRID + blockIdx.x, ((unsigned long long)(FUSED ? epoch : 0u) << 32) | row[i]);
}

// One word of the blocks [0, count), lane l those of blocks l, l + 32, ...: c[k] (undefined beyond). Waits for them where `wait`;
// false where the budget ran out (reported) or, `stop`, where an error has been reported: that block may never come.
template <bool WAIT>
__device__ __forceinline__ bool read_row(const CP& p, const unsigned long long* words, unsigned int count, unsigned int epoch, unsigned int where,
                                         bool stop, unsigned int (&c)[MAX_GRID / 32]) {
    const unsigned int lane = threadIdx.x & 31;
    const long long t0 = WAIT ? clock64() : 0;
    for (unsigned int ns = 0;; ns = min(ns + 20u, 200u)) {
        if (ns) __nanosleep(ns);
        unsigned long long v[MAX_GRID / 32];
#pragma unroll
        for (int k = 0; k < MAX_GRID / 32; ++k) v[k] = lane + 32 * k < count ? ld_relaxed_gpu64(words + lane + 32 * k) : (unsigned long long)epoch << 32;
        const unsigned int st = WAIT && stop ? ld_relaxed_gpu(p.status) : 0u;   // (in the same flight)
        bool here = true;
#pragma unroll
        for (int k = 0; k < MAX_GRID / 32; ++k) {
            here = here && (unsigned int)(v[k] >> 32) == epoch;
            c[k] = (unsigned int)v[k];
        }
        if (!WAIT) return true;
        if (__any_sync(0xFFFFFFFFu, (st & 0xFFu) != SKML_OK)) return false;
        if (__all_sync(0xFFFFFFFFu, here)) return true;
        if (__any_sync(0xFFFFFFFFu, clock64() - t0 > p.budget)) {
            if (lane == 0) skml_set_status(p.status, SKML_TIMEOUT_BARRIER, where);
            return false;
        }
    }
}

__device__ __forceinline__ float bucket_value(const Smem& s, int b) {
    const QInfo& q = s.qi;
    if (q.bin_num == 1) return 0.5f * (q.minv + q.maxv);
    if (b == 0) return 0.5f * (q.minv + s.splits[0]);
    if (b == q.bin_num - 1) return 0.5f * (s.splits[q.nsplits - 1] + q.maxv);
    return 0.5f * (s.splits[b - 1] + s.splits[b]);
}

// ---------------------------------------------------------------------------
// Element stages. The unit of work of S3 and S4 is a warp: warp w of block b owns one contiguous
// slice of the (key-sorted) input. S5 works on the groups' contiguous lists in 1024-key chunks.
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long vslice_size(long long n) {
    const long long nv = (long long)gridDim.x * SKML_WARPS;
    long long c = (n + nv - 1) / nv;
    return (c + 31) / 32 * 32;
}

template <bool PRIV>
__device__ __forceinline__ void build_group_lut(const CP& p, Smem& s) {
    for (int b = threadIdx.x; b < s.qi.bin_num; b += blockDim.x) {
        int g = 0;   // the edges ascend: the group is the number of edges at or below the bucket
        for (int e = 0; e < p.G - 1; ++e) g += s.qi.edges[e] <= b ? 1 : 0;
        s.grp_lut[b] = (unsigned char)g;
        if (PRIV) {
            // rank of the bucket's cell among those of its group: by distance from the zero bucket, the lower bucket first
            const int lo = g ? s.qi.edges[g - 1] : 0, hi = s.qi.edges[g], z = s.qi.zero_idx;
            const int below = z - lo, above = hi - 1 - z, d = b < z ? z - b : b - z;
            int rank = d;
            if (below <= 0) rank = b - lo;
            else if (above <= 0) rank = hi - 1 - b;
            else if (d) rank = 1 + min(d - 1, below) + min(d - 1, above) + (b > z && d <= below ? 1 : 0);
            s.rank_lut[b] = (unsigned char)rank;
            s.code_bin[lo + rank] = (unsigned char)b;
        }
    }
    __syncthreads();
}

// The split points into s.ss; the caller's barrier follows. Returns the search's first step.
__device__ __forceinline__ int build_search(Smem& s) {
    const int n = s.qi.nsplits, top = search_top(n);
    for (int i = threadIdx.x; i < 2 * top - 1; i += blockDim.x) s.ss.a[search_slot(i)] = i < n ? s.splits[i] : __int_as_float(0x7FC00000);
    return top;
}

// Group lists keep the keys' order, so a warp ranks its elements by group: one ballot per bit of the group number
// gives every lane the mask of its own group, and lane g that of group g. (__match_any_sync and counters in shared
// memory took twice the instructions.)
template <int BITS>
__device__ __forceinline__ void group_masks(bool valid, int g, unsigned int& own, unsigned int& of_lane) {
    const int lane = threadIdx.x & 31;
    own = of_lane = __ballot_sync(0xFFFFFFFFu, valid);
#pragma unroll
    for (int k = 0; k < BITS; ++k) {
        const unsigned int b = __ballot_sync(0xFFFFFFFFu, (g >> k) & 1);
        own &= b ^ (((unsigned int)g >> k & 1u) - 1u);
        of_lane &= b ^ (((unsigned int)lane >> k & 1u) - 1u);
    }
}

// U searches side by side, the next turn's values on their way.
template <int U>
__device__ __forceinline__ void count_turns(Smem& s, int top, int rem, const float* __restrict__ vals, unsigned short* __restrict__ bins,
                                            const float (&first_val)[2], int (&first_bin)[2], unsigned int& kmin, unsigned int& kmax) {
    const int warp = threadIdx.x >> 5;
    float nval[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nval[u] = u < 2 ? first_val[u] : (32 * u < rem ? vals[32 * u] : 0.f);
    for (int i0 = 0; i0 < rem; i0 += 32 * U) {
        float val[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            val[u] = nval[u];
            if (i0 + 32 * (U + u) < rem) nval[u] = vals[i0 + 32 * (U + u)];
        }
        int bin[U];
        upper_bounds_f(s.ss.a, top, val, bin);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + 32 * u >= rem) break;
            bins[i0 + 32 * u] = (unsigned short)bin[u];
            if (u < 2 && i0 == 0) first_bin[u] = bin[u];
            atomicAdd(&s.wcnt[warp][s.grp_lut[bin[u]]], 1u);
            const unsigned int k = f2ord(val[u]);
            kmin = min(kmin, k);
            kmax = max(kmax, k);
        }
    }
}

// S3: bucket of every value; keys of every group in every warp slice.
// Bound by instruction issue: a conflict-free search unrolled for up to 255 splits, 32-bit positions inside the slice
// and shared-memory counts instead of a match of the warp took it from 58 to 31 us at 10M values.
// `first_val`: the values of this lane's first two elements where the caller has them in flight already; their
// buckets are left in `first_bin`.
template <bool FUSED, bool PRIV>
__device__ void stage_count(const CP& p, Smem& s, unsigned int* set, unsigned int epoch, long long n, bool track_minmax, const float (&first_val)[2],
                            int (&first_bin)[2]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int kmin = 0xFFFFFFFFu, kmax = 0u;
    const int top = build_search(s);
    build_group_lut<PRIV>(p, s);
    const long long sub = vslice_size(n);
    const long long vb = (long long)blockIdx.x * SKML_WARPS + warp;
    long long lo = vb * sub, hi = lo + sub;
    if (lo > n) lo = n;
    if (hi > n) hi = n;
    s.wcnt[warp][lane] = 0;
    __syncwarp();
    const int rem = (int)(hi - lo) - lane;   // this lane's elements: 0, 32, ... below it
    const float* const vals = p.vals + lo + lane;
    unsigned short* const bins = p.bins + lo + lane;
    // 32 U values a turn: short slices are not worth a second pair of searches, long ones want the loads in flight (2.3M
    // values: 11.3 -> 10.1 us, 10M: 32 -> 27.6)
    if (!PRIV || sub <= 64) count_turns<2>(s, top, rem, vals, bins, first_val, first_bin, kmin, kmax);
    else count_turns<4>(s, top, rem, vals, bins, first_val, first_bin, kmin, kmax);
    kmin = __reduce_min_sync(0xFFFFFFFFu, kmin);
    kmax = __reduce_max_sync(0xFFFFFFFFu, kmax);
    if (lane == 0) {
        s.scan[0][warp] = kmin;
        s.scan[1][warp] = kmax;
    }
    // (one launch for all stages: the slices' counts stay in shared memory)
    if (!FUSED && lane < p.G) p.warp_cnt[vb * SKML_MAX_GROUPS + lane] = s.wcnt[warp][lane];
    __syncthreads();
    for (int i = warp; i < p.G + 2; i += SKML_WARPS) {   // the block's totals, a warp each
        const unsigned int v = i < p.G ? __reduce_add_sync(0xFFFFFFFFu, s.wcnt[lane][i])
                                       : (i == p.G ? __reduce_min_sync(0xFFFFFFFFu, s.scan[0][lane]) : __reduce_max_sync(0xFFFFFFFFu, s.scan[1][lane]));
        if (lane == 0) s.row[i] = v;
    }
    __syncthreads();
    if (warp == 0) publish_row<FUSED>(p.blk_cnt, s.row, p.G + 2, epoch);
    if (!FUSED && track_minmax && threadIdx.x == 0 && s.row[p.G] <= s.row[p.G + 1]) {   // staged launches: for the next ones
        atomicMax(&set[CTRL_MIN], ~s.row[p.G]);
        atomicMax(&set[CTRL_MAX], s.row[p.G + 1]);
    }
}

// S4 prelude: group sizes, table sizes, hash rows and every section offset that does not depend on
// the key code (every block computes the same layout); this block's and its warps' starting ranks.
// One launch for all stages: waits for every block's row of counts. Whoever has seen them all is behind a grid barrier: a
// row is stored behind a fence, and nothing is counted in one place first. (An arrival, a poll for the last one and only then
// the loads of the counts took 4.3 us of every launch. This, the counts of S5 sent likewise, the narrow tables by other blocks
// than the keys' and the flag without a count, together: 26,000 keys 37.5 -> 29.5 us, 430,000 57.5 -> 48.5, 2.27M 105.5 -> 100.7.)
// False on every thread where the wait ran out, or on an error.
template <bool FUSED>
__device__ bool layout_from_counts(const CP& p, Smem& s, unsigned int epoch, bool want_minmax) {
    const int G = p.G, nb = gridDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Layout& L = s.lay;
    bool ok = true;
    for (int i = warp; i < (want_minmax ? G + 2 : G); i += SKML_WARPS) {
        // the blocks' totals (before this block / all blocks), lanes striding over the blocks; this
        // block's own 32 slices are scanned over the lanes for the warps' starting ranks
        unsigned int c[MAX_GRID / 32];
        ok = read_row<FUSED>(p, p.blk_cnt + i * MAX_GRID, nb, epoch, 3u, true, c) && ok;
        if (i >= G) {   // least and largest value
            unsigned int v = i == G ? 0xFFFFFFFFu : 0u;
#pragma unroll
            for (int k = 0; k < MAX_GRID / 32; ++k)
                if (lane + 32 * k < nb) v = i == G ? min(v, c[k]) : max(v, c[k]);
            v = i == G ? __reduce_min_sync(0xFFFFFFFFu, v) : __reduce_max_sync(0xFFFFFFFFu, v);
            if (lane == 0) set_extreme(p, s, i == G, v);
            continue;
        }
        const int g = i;
        unsigned int before = 0, total = 0;
#pragma unroll
        for (int k = 0; k < MAX_GRID / 32; ++k) {
            if (lane + 32 * k < nb) total += c[k];
            if (lane + 32 * k < (int)blockIdx.x) before += c[k];
        }
        const unsigned int own = FUSED ? s.wcnt[lane][g] : __ldcg(&p.warp_cnt[((long long)blockIdx.x * SKML_WARPS + lane) * SKML_MAX_GROUPS + g]);
        total = __reduce_add_sync(0xFFFFFFFFu, total);
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        unsigned int inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += t;
        }
        s.wbase[lane][g] = inc - own;
        if (lane == 0) {
            L.n_g[g] = total;
            L.base_rank[g] = before;
        }
        if (lane < SKML_MAX_ROWS) L.hash_ids[g][lane] = p.hash_ids[g][lane];
    }
    if (FUSED && warp == 0) __threadfence();   // the others' stores before their rows, too
    if (!__syncthreads_and(ok)) return false;
    // One lane per group, one warp per quantity: sizes, then prefix sums over the lanes. (One thread that walked the
    // groups took 3 us of a 62 us launch at 10,000 keys.)
    const bool adaptive = p.key_encoder == SKML_KEYS_DELTA_ADAPTIVE;
    if (warp < 5) {
        const unsigned int n = lane < G ? L.n_g[lane] : 0u;
        unsigned long long v = 0;
        unsigned int col = 0;
        if (warp == 2 || warp == 3) {
            if (n) {
                col = (unsigned int)ceil((double)n * p.col_ratio);
                if (col < 1) col = 1;
            }
            const unsigned long long cells = (unsigned long long)p.rows * col;
            v = warp == 2 ? skml_align16(cells * (s.qi.cell_bits / 8)) : (cells + 3ull) & ~3ull;
        } else if (warp == 0) {
            v = n && !adaptive ? skml_align16(8ull * ((2ull * n + 63) / 64)) : 0ull;   // flag bytes
        } else if (warp == 1) {
            v = ((unsigned long long)((n + SKML_RESTART_INTERVAL - 1) / SKML_RESTART_INTERVAL) << 32) | ((n + 3u) & ~3u);  // chunks | staging entries
        } else if (lane < G) {
            // the key code adds at most four bytes per key (delta_adaptive: 49 bits): refuse now what cannot
            // fit in the worst case
            v = skml_align16(4ull * n + 8) + (adaptive ? skml_align16(17ull * n / 8 + 8) : 0ull);
        }
        unsigned long long total;
        const unsigned long long o = warp_prefix(v, total);
        if (lane < G) {
            if (warp == 0) L.flag_off[lane] = o;
            else if (warp == 1) {
                L.goff[lane] = (unsigned int)o;
                L.chunk_prefix[lane] = (unsigned int)(o >> 32);
            } else if (warp == 2) {
                L.table_off[lane] = o;
                L.unit_prefix[lane] = o / 16;
                L.col[lane] = col;
                L.recip[lane] = skml_recip32(col);
            } else if (warp == 3) {
                L.tab32_off[lane] = o;
                if (!p.mixers) L.col_magic[lane] = col ? skml_fastmod_magic(col) : 0ull;
            }
        }
        if (lane == 0) s.sums[warp] = total;
    }
    __syncthreads();
    if (warp == 0) {   // the sections' starts
        const unsigned long long off_gt = SKML_HEADER_BYTES + skml_align16(4ull * p.q);
        const unsigned long long off_flags = off_gt + (unsigned long long)SKML_GROUP_ENTRY_BYTES * G;
        const unsigned int chunks = (unsigned int)(s.sums[1] >> 32);
        const unsigned long long off_restart = off_flags + s.sums[0], off_tables = off_restart + 16ull * chunks;
        const unsigned long long off_deltas = off_tables + s.sums[2];
        if (lane < G) {
            L.flag_off[lane] += off_flags;
            L.restart_off[lane] = off_restart + 16ull * L.chunk_prefix[lane];
            L.table_off[lane] += off_tables;
        }
        if (lane == 0) {
            L.off_bv = SKML_HEADER_BYTES;
            L.off_gt = off_gt;
            L.off_flags = off_flags;
            L.off_restart = off_restart;
            L.off_tables = off_tables;
            L.off_deltas = off_deltas;
            L.off_keys = off_deltas;  // delta_adaptive: both key sections of every group follow the tables
            L.chunk_prefix[G] = chunks;
            L.unit_prefix[G] = s.sums[2] / 16;
            L.overflow = (off_deltas + s.sums[4] > (unsigned long long)p.slot_capacity) || (s.sums[3] + 4 > (unsigned long long)p.tables_cap);
            if (L.overflow) skml_set_status(p.status, SKML_CAPACITY, 0x30u);
        }
    }
    __syncthreads();
    return true;
}

// Insert in shared memory (large gradients, plain tables). A cell of the sketch is decided by the rank of its bucket among
// the buckets of its group, a byte where a group has at most 255 of them, so a row of a group's table is small enough for
// a block's shared memory, or a few parts of it are. Work is (part of a row, four keys of the group's list); the units of
// all parts, one part behind the other, are dealt to the blocks in equal runs. A block hashes its keys for one row, keeps
// the least codes in shared memory and leaves a copy of the part; the copies of a part are merged when the tables are
// written to the payload. Bound by the hashes' instructions and the latency of the rounds; atomics in L2, three a key, by
// L2's rate (121 G/s). Insert and all, S4 and S5 of such launches (three rows of 0.2 cells a key; atomics / shared memory, us):
// 2.27M keys 76 / 59, 10M 302 / 247.
// Sets L.priv where it pays (priv_pays): the keys of large groups are hashed once per part, so a group of many parts (few
// distinct values: one group holds nearly every key) is left to the atomics.
__device__ void priv_layout(const CP& p, Smem& s) {
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31, G = p.G;
    if (threadIdx.x < 32) {
        unsigned int parts = 0, len = 0;
        unsigned long long work = 0;
        if (lane < G && L.n_g[lane]) {
            const unsigned int room = PRIV_BYTES - 16u;   // (a part starts at its place in a 16-byte unit)
            parts = (L.col[lane] + room - 1u) / room;
            len = (L.col[lane] + parts - 1u) / parts;
            work = (unsigned long long)p.rows * parts * ((L.n_g[lane] + 3u) / 4u);
        }
        unsigned long long nparts, units;
        const unsigned long long part0 = warp_prefix((unsigned long long)p.rows * parts, nparts), work0 = warp_prefix(work, units);
        const unsigned int longest = __reduce_max_sync(0xFFFFFFFFu, len);
        unsigned long long keys;
        warp_prefix(lane < G ? (unsigned long long)L.n_g[lane] : 0ull, keys);
        if (lane < G) {
            L.parts[lane] = parts;
            L.part_len[lane] = len;
            L.part_prefix[lane] = (unsigned int)part0;
            L.work_prefix[lane] = work0;
        }
        if (lane == 0) {
            L.part_prefix[G] = (unsigned int)nparts;
            L.work_prefix[G] = units;
            L.work_per = (units + gridDim.x - 1) / gridDim.x;
            L.copy_stride = (longest + 15u + 15u) & ~15u;
            L.priv = nparts <= PRIV_MAX_PARTS && priv_pays(p.priv_least, (float)keys, 4.f * (float)units, (float)p.rows * (float)keys, 1.3f) &&
                     (nparts + gridDim.x) * L.copy_stride <= (unsigned long long)p.copies_cap;
        }
    }
    __syncthreads();
}

// Units [u0, u1) of one group's keys against one part of one row: cells lo .. lo + len of the row at cells[at ..].
// Two block barriers per round instead of an atomic per key: codes smaller than the cell's are stored plainly, so where
// several threads meet in a cell any of them may win; behind the barrier every thread that has stored looks again, and
// those that find a larger code (few) repeat it with compare-and-swap, while nobody stores plainly.
template <int MIXER>
__device__ __forceinline__ void priv_insert(const CP& p, const Layout& L, int g, unsigned int u0, unsigned int u1, unsigned int lo,
                                            unsigned int len, unsigned int at, unsigned char* cells) {
    const unsigned int n = L.n_g[g], col = L.col[g], recip = L.recip[g];
    const int4* const keys = reinterpret_cast<const int4*>(p.gkeys + L.goff[g]);                       // (lists start at multiples of four)
    const unsigned int* const codes = reinterpret_cast<const unsigned int*>(p.gcodes + L.goff[g]);
    int4 nk[PRIV_UNITS];
    unsigned int nc[PRIV_UNITS];
    auto fetch = [&](unsigned int u) {
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q) {
            nk[q] = make_int4(0, 0, 0, 0);
            nc[q] = 0;
            if (u + q * SKML_BLOCK < u1) {
                nk[q] = __ldcg(keys + u + q * SKML_BLOCK);
                nc[q] = __ldcg(codes + u + q * SKML_BLOCK);
            }
        }
    };
    fetch(u0 + threadIdx.x);
    for (unsigned int base = u0; base < u1; base += PRIV_UNITS * SKML_BLOCK) {
        const unsigned int u = base + threadIdx.x;
        unsigned int c[PRIV_UNITS], pos[PRIV_UNITS][4];
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q) {
            const int k[4] = {nk[q].x, nk[q].y, nk[q].z, nk[q].w};
            const unsigned int uq = u + q * SKML_BLOCK;
            c[q] = nc[q];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned int h = MIXER == 0 ? skml_mix_bj((unsigned int)k[i]) : (MIXER == 1 ? skml_mix_64((unsigned int)k[i]) : skml_mix_tw((unsigned int)k[i]));
                const unsigned int x = (unsigned int)skml_java_mod(h, col, recip) - lo;
                pos[q][i] = x < len && uq < u1 && 4u * uq + i < n ? x + at : ~0u;
            }
        }
        fetch(u + PRIV_UNITS * SKML_BLOCK);
        unsigned char old[PRIV_UNITS][4];
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) old[q][i] = pos[q][i] != ~0u ? *(volatile unsigned char*)(cells + pos[q][i]) : 0;
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned int code = (c[q] >> (8 * i)) & 0xFFu;
                if (code < old[q][i]) *(volatile unsigned char*)(cells + pos[q][i]) = (unsigned char)code;
                else pos[q][i] = ~0u;
            }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) old[q][i] = pos[q][i] != ~0u ? *(volatile unsigned char*)(cells + pos[q][i]) : 0;
#pragma unroll
        for (int q = 0; q < PRIV_UNITS; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned int code = (c[q] >> (8 * i)) & 0xFFu;
                if (code < old[q][i]) {
                    unsigned int* const word = reinterpret_cast<unsigned int*>(cells) + (pos[q][i] >> 2);
                    const unsigned int shift = 8u * (pos[q][i] & 3u);
                    unsigned int seen = *(volatile unsigned int*)word;
                    while (((seen >> shift) & 0xFFu) > code) {
                        const unsigned int was = atomicCAS(word, seen, (seen & ~(0xFFu << shift)) | (code << shift));
                        if (was == seen) break;
                        seen = was;
                    }
                }
            }
        __syncthreads();
    }
}

__device__ void stage_insert(const CP& p, Smem& s) {
    const Layout& L = s.lay;
    if (L.overflow) return;
    unsigned char* const cells = reinterpret_cast<unsigned char*>(s.splits + PRIV_SPLITS);
    unsigned long long w = L.work_per * blockIdx.x;
    unsigned long long w1 = w + L.work_per;
    if (w1 > L.work_prefix[p.G]) w1 = L.work_prefix[p.G];
    int g = 0;
    while (w < w1) {   // one part of a row after the other
        while (g + 1 < p.G && w >= L.work_prefix[g + 1]) ++g;
        const unsigned int per_part = (L.n_g[g] + 3u) / 4u;
        const unsigned int t = (unsigned int)((w - L.work_prefix[g]) / per_part);
        const unsigned long long part_w = L.work_prefix[g] + (unsigned long long)t * per_part;
        const unsigned int u0 = (unsigned int)(w - part_w), u1 = (unsigned int)min((unsigned long long)per_part, w1 - part_w);
        const unsigned int row = t / L.parts[g], lo = (t - row * L.parts[g]) * L.part_len[g];
        const unsigned int len = min(L.part_len[g], L.col[g] - lo);
        const unsigned int at = (unsigned int)(((unsigned long long)row * L.col[g] + lo) & 15ull), units = (at + len + 15u) / 16u;
        uint4* const cells4 = reinterpret_cast<uint4*>(cells);
        for (unsigned int i = threadIdx.x; i < units; i += SKML_BLOCK) cells4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncthreads();
        const int id = L.hash_ids[g][row];
        if (id == 0) priv_insert<0>(p, L, g, u0, u1, lo, len, at, cells);
        else if (id == 1) priv_insert<1>(p, L, g, u0, u1, lo, len, at, cells);
        else priv_insert<2>(p, L, g, u0, u1, lo, len, at, cells);
        __syncthreads();
        // the blocks and the parts of a run of work ascend together: block + part names a copy
        uint4* const out = reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(p.tables) +
                                                    (unsigned long long)(blockIdx.x + L.part_prefix[g] + t) * L.copy_stride);
        for (unsigned int i = threadIdx.x; i < units; i += SKML_BLOCK) __stcg(out + i, cells4[i]);
        __syncthreads();
        w = part_w + u1;
    }
}

// S4: every key goes to its group's staging list (stable, so the lists stay sorted);
// grouped MinMaxSketch insert with atomics in L2.
// `nkey`, `nbin`: keys and buckets of this lane's first two elements (one launch for all stages). What bounds it is
// the rate of atomics in L2: three a key, 121 G/s at 10M keys; a plain count of 100M random keys reaches 156 G/s.
template <bool FUSED>
__device__ void stage_scatter(const CP& p, Smem& s, long long n, int (&nkey)[2], int (&nbin)[2]) {
    const int G = p.G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Layout& L = s.lay;
    if (L.overflow) return;
    if (!FUSED) build_group_lut<false>(p, s);   // (otherwise the group table is the count stage's)
    const long long sub = vslice_size(n);
    const long long vb = (long long)blockIdx.x * SKML_WARPS + warp;
    long long lo = vb * sub, hi = lo + sub;
    if (lo > n) lo = n;
    if (hi > n) hi = n;
    const int zero = s.qi.zero_idx;
    unsigned int run = 0;   // lane g: staging position of the next key of group g in this slice
    if (lane < G) run = L.goff[lane] + L.base_rank[lane] + s.wbase[warp][lane];
    const int len = (int)(hi - lo), rem = len - lane;   // this lane's elements: 0, 32, ... below rem
    const int* const keys = p.keys + lo + lane;
    const unsigned short* const bins = p.bins + lo + lane;
    if (!FUSED) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (32 * u < rem) {
                nkey[u] = keys[32 * u];
                nbin[u] = bins[32 * u];
            }
    }
    for (int i0 = 0; i0 < len; i0 += 64) {
        const int key[2] = {nkey[0], nkey[1]}, bin[2] = {nbin[0], nbin[1]};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + 64 + 32 * u;
            if (i < rem) {
                nkey[u] = keys[i];
                nbin[u] = bins[i];
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool valid = i0 + 32 * u < rem;
            const int g = valid ? (int)s.grp_lut[bin[u]] : 0;
            unsigned int own, of_lane;
            if (G <= 8) group_masks<3>(valid, g, own, of_lane);
            else group_masks<5>(valid, g, own, of_lane);
            const unsigned int base = __shfl_sync(0xFFFFFFFFu, run, g);
            run += (unsigned int)__popc(of_lane);   // (of lanes beyond the last group nobody asks)
            if (!valid) continue;
            p.gkeys[base + (unsigned int)__popc(own & lanemask_lt())] = key[u];
            const unsigned int cell = skml_pack_cell(bin[u], zero);
            const int col = (int)L.col[g];
            unsigned int* tab = p.tables + L.tab32_off[g];
            int pos[SKML_MAX_ROWS];
            if (p.mixers) {
                skml_hash_rows_mixers<3>(L.hash_ids[g], p.rows, key[u], (unsigned int)col, L.recip[g], pos);
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    if (r < p.rows) atomicMin(tab + (long long)r * col + pos[r], cell);
            } else if (p.rows <= 4) {
                skml_hash_rows<4>(L.hash_ids[g], p.rows, key[u], col, L.col_magic[g], pos);
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < p.rows) atomicMin(tab + (long long)r * col + pos[r], cell);
            } else {
                skml_hash_rows<SKML_MAX_ROWS>(L.hash_ids[g], p.rows, key[u], col, L.col_magic[g], pos);
#pragma unroll
                for (int r = 0; r < SKML_MAX_ROWS; ++r)
                    if (r < p.rows) atomicMin(tab + (long long)r * col + pos[r], cell);
            }
        }
        __syncwarp();
    }
}

// S4 where the insert follows in shared memory: the lists get the keys and their rank codes.
// Up to eight groups: 128 elements a turn, four adjacent ones a lane. A lane's counts of all groups are the bytes of one
// word, so that one scan of the warp ranks the turn's elements; they are put in group order in shared memory and leave it
// in runs. (A ballot per bit of the group number for every 32 elements took four times the instructions: 66 us of 10M keys.)
__device__ __forceinline__ void partition_turns(const CP& p, Smem& s, int len, unsigned int run, const int* __restrict__ keys,
                                                const unsigned short* __restrict__ bins) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int* const s_key = s.part.key[warp];
    unsigned short* const s_tag = s.part.tag[warp];
    const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;   // (slices start at multiples of 32 elements)
    int nkey[4], nbin[4];
    auto fetch = [&](int i0) {
        const int i = i0 + 4 * lane;
        if (vec && i + 4 <= len) {
            const int4 k = __ldg(reinterpret_cast<const int4*>(keys + i));
            const uint2 b = *reinterpret_cast<const uint2*>(bins + i);
            nkey[0] = k.x; nkey[1] = k.y; nkey[2] = k.z; nkey[3] = k.w;
            nbin[0] = (int)(b.x & 0xFFFFu); nbin[1] = (int)(b.x >> 16); nbin[2] = (int)(b.y & 0xFFFFu); nbin[3] = (int)(b.y >> 16);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                nkey[u] = i + u < len ? keys[i + u] : 0;
                nbin[u] = i + u < len ? (int)bins[i + u] : 0;
            }
        }
    };
    fetch(0);
    for (int i0 = 0; i0 < len; i0 += 128) {
        int key[4], bin[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            key[u] = nkey[u];
            bin[u] = nbin[u];
        }
        fetch(i0 + 128);
        const int have = len - i0 - 4 * lane;   // this lane's elements
        unsigned int g[4];
        unsigned long long own = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            g[u] = u < have ? s.grp_lut[bin[u]] : 0u;
            if (u < have) own += 1ull << (8 * g[u]);
        }
        unsigned long long inc = own;   // (128 elements at most: no byte overflows)
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += t;
        }
        const unsigned long long all = __shfl_sync(0xFFFFFFFFu, inc, 31);
        // bytes of `start`: elements of the groups before (the sum over the lower bytes, below 256 each)
        const unsigned long long start = (all << 8) * 0x0101010101010101ull;
        unsigned long long at = start + inc - own;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u < have) {
                const unsigned int r = (unsigned int)(at >> (8 * g[u])) & 0xFFu;
                s_key[r] = (unsigned int)key[u];
                s_tag[r] = (unsigned short)(s.rank_lut[bin[u]] | (g[u] << 8));
                at += 1ull << (8 * g[u]);
            }
        }
        __syncwarp();
        // lane g: where group g's first element of this turn goes, less its place in the turn
        const unsigned int base = lane < 8 ? run - ((unsigned int)(start >> (8 * lane)) & 0xFFu) : 0u;
        if (lane < 8) run += (unsigned int)(all >> (8 * lane)) & 0xFFu;
        const int turn = min(128, len - i0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = 32 * u + lane;
            const unsigned int tag = q < turn ? s_tag[q] : 0u;
            const unsigned int to = __shfl_sync(0xFFFFFFFFu, base, (int)(tag >> 8)) + (unsigned int)q;
            if (q < turn) {
                p.gkeys[to] = (int)s_key[q];
                p.gcodes[to] = (unsigned char)tag;
            }
        }
        __syncwarp();
    }
}

// More groups: a ballot per bit of the group number.
__device__ void stage_partition(const CP& p, Smem& s, long long n) {
    constexpr int U = 4;
    const int G = p.G, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Layout& L = s.lay;
    if (L.overflow) return;
    const long long sub = vslice_size(n);
    const long long vb = (long long)blockIdx.x * SKML_WARPS + warp;
    long long lo = vb * sub, hi = lo + sub;
    if (lo > n) lo = n;
    if (hi > n) hi = n;
    unsigned int run = 0;   // lane g: staging position of the next key of group g in this slice
    if (lane < G) run = L.goff[lane] + L.base_rank[lane] + s.wbase[warp][lane];
    const int len = (int)(hi - lo), rem = len - lane;   // this lane's elements: 0, 32, ... below rem
    if (G <= 8) {
        partition_turns(p, s, len, run, p.keys + lo, p.bins + lo);
        return;
    }
    const int* const keys = p.keys + lo + lane;
    const unsigned short* const bins = p.bins + lo + lane;
    int nkey[U], nbin[U];
    auto fetch = [&](int i0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            nkey[u] = nbin[u] = 0;
            if (i0 + 32 * u < rem) {
                nkey[u] = keys[i0 + 32 * u];
                nbin[u] = bins[i0 + 32 * u];
            }
        }
    };
    fetch(0);
    for (int i0 = 0; i0 < len; i0 += 32 * U) {
        int key[U], bin[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            key[u] = nkey[u];
            bin[u] = nbin[u];
        }
        fetch(i0 + 32 * U);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool valid = i0 + 32 * u < rem;
            const int g = valid ? (int)s.grp_lut[bin[u]] : 0;
            unsigned int own, of_lane;
            group_masks<5>(valid, g, own, of_lane);
            const unsigned int to = __shfl_sync(0xFFFFFFFFu, run, g) + (unsigned int)__popc(own & lanemask_lt());
            run += (unsigned int)__popc(of_lane);   // (of lanes beyond the last group nobody asks)
            if (valid) {
                p.gkeys[to] = key[u];
                p.gcodes[to] = s.rank_lut[bin[u]];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// S5: delta-binary key code of the groups' lists. Chunks of 1024 keys are numbered group-major; a
// block owns a contiguous run of them and works on four at a time (one per 256-thread sub-block,
// four adjacent keys per thread).
// ---------------------------------------------------------------------------
struct ChunkWork {
    int g;                  // group, -1 = no chunk for this sub-block
    unsigned int j;         // chunk index inside the group
    unsigned int cnt;       // keys in the chunk
    int k[4];               // this thread's keys
    unsigned int w[4];      // their delta widths in bytes (0 = no key)
    unsigned int d[4];      // their deltas
    unsigned int wsum;
    int prev0;              // key before the chunk's first key (0 at the start of a group)
};

// A chunk's keys on their way from memory.
struct ChunkFetch {
    int g;
    unsigned int j, cnt;
    int4 k;
    int before;   // a warp's first lane: the key before its first one
};

// `g`: a group at or before the chunk's.
__device__ __forceinline__ ChunkFetch fetch_chunk(const CP& p, const Layout& L, unsigned int ch, unsigned int ch_end, int G, int g) {
    const unsigned int i0 = 4u * (threadIdx.x & 255);
    ChunkFetch f;
    f.g = -1;
    f.j = f.cnt = 0;
    f.k = make_int4(0, 0, 0, 0);
    f.before = 0;
    if (ch >= ch_end) return f;
    while (g + 1 < G && ch >= L.chunk_prefix[g + 1]) ++g;
    f.g = g;
    f.j = ch - L.chunk_prefix[g];
    const unsigned int first = f.j * SKML_RESTART_INTERVAL;
    f.cnt = min((unsigned int)SKML_RESTART_INTERVAL, L.n_g[g] - first);
    const int* list = p.gkeys + L.goff[g] + first;
    if (i0 < f.cnt) {
        f.k = *reinterpret_cast<const int4*>(list + i0);  // goff and first are multiples of 4
        if ((threadIdx.x & 31) == 0 && first + i0 > 0) f.before = list[(int)i0 - 1];
    }
    return f;
}

__device__ __forceinline__ void expand_chunk(const ChunkFetch& f, ChunkWork& c) {
    const unsigned int i0 = 4u * (threadIdx.x & 255);
    c.g = f.g;
    c.j = f.j;
    c.cnt = f.cnt;
    c.wsum = 0;
    c.k[0] = f.k.x; c.k[1] = f.k.y; c.k[2] = f.k.z; c.k[3] = f.k.w;
    // the key before this thread's first key: the lane below holds it, except at a warp's start
    int prev = __shfl_up_sync(0xFFFFFFFFu, c.k[3], 1);
    if ((threadIdx.x & 31) == 0) prev = f.before;
    c.prev0 = f.before;   // (meant for the sub-block's first thread)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        c.w[u] = c.d[u] = 0;
        if (i0 + u < f.cnt) {
            c.d[u] = (unsigned int)(c.k[u] - prev);
            c.w[u] = (unsigned int)skml_delta_bytes(c.d[u]);
            c.wsum += c.w[u];
            prev = c.k[u];
        }
    }
}

__device__ __forceinline__ void load_chunk(const CP& p, const Layout& L, unsigned int ch, unsigned int ch_end, int G, ChunkWork& c) {
    expand_chunk(fetch_chunk(p, L, ch, ch_end, G, 0), c);
}

// Exclusive scan of `v` over the 256 threads of this thread's sub-block; `total` = the sub-block's sum.
// One block barrier inside; `par` alternates between calls.
__device__ __forceinline__ unsigned int sub_scan(Smem& s, unsigned int v, unsigned int& total) {
    const int lane = threadIdx.x & 31, sw = (threadIdx.x >> 5) & 7, sb = threadIdx.x >> 8;
    unsigned int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    __syncthreads();  // the previous call's readers are done
    if (lane == 31) s.sub_part[sb][sw] = inc;
    __syncthreads();
    unsigned int base = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const unsigned int x = s.sub_part[sb][w];
        if (w < sw) base += x;
        tot += x;
    }
    total = tot;
    return base + inc - v;
}

// Group of a group-major chunk (or table chunk) number.
__device__ __forceinline__ int group_of_chunk(const unsigned int* prefix, int G, unsigned int ch) {
    int g = 0;
    while (g + 1 < G && ch >= prefix[g + 1]) ++g;
    return g;
}

// Pass A: byte counts of this block's chunks -> chunk offsets inside the block's part of each group,
// the block's byte totals per group (published for the blocks after it). A block with one round of chunks keeps
// them (`c`, `boff`, `total`; offsets in s.sub_off) and does not read its keys again. Longer runs need the totals
// only: every warp adds up eighths of chunks on its own, the next one's keys on their way, without a barrier
// per chunk (a scan and three barriers per round took 31 us at 66 chunks a block).
template <bool FUSED>
__device__ void pack_measure(const CP& p, Smem& s, unsigned int epoch, unsigned int my_begin, unsigned int my_end, ChunkWork& c, unsigned int& boff,
                             unsigned int& total) {
    const Layout& L = s.lay;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < SKML_MAX_GROUPS) s.my_bytes[threadIdx.x] = 0;
    if (my_end - my_begin <= 4) {
        load_chunk(p, L, my_begin + (threadIdx.x >> 8), my_end, p.G, c);
        boff = sub_scan(s, c.wsum, total);
        if ((threadIdx.x & 255) == 0) s.sub_total[threadIdx.x >> 8] = total;
        __syncthreads();
        const unsigned int q = threadIdx.x;
        if (q < 4 && my_begin + q < my_end) {
            const int g = group_of_chunk(L.chunk_prefix, p.G, my_begin + q);
            unsigned int off = 0;
            for (unsigned int k = 0; k < q; ++k)
                if (my_begin + k >= L.chunk_prefix[g]) off += s.sub_total[k];
            s.sub_off[q] = off;
            atomicAdd(&s.my_bytes[g], (unsigned long long)s.sub_total[q]);
        }
    } else {
        unsigned int* const tot = s.ps.tot;
        for (unsigned int b0 = my_begin; b0 < my_end; b0 += MEASURE_CHUNKS) {
            const unsigned int nb = min((unsigned int)MEASURE_CHUNKS, my_end - b0);
            for (unsigned int i = threadIdx.x; i < nb; i += blockDim.x) tot[i] = 0;
            __syncthreads();
            // warp w: eighth w % 8 of the chunks w / 8, w / 8 + 4, ... (the lanes of a fetch take their keys by thread number)
            ChunkFetch f = fetch_chunk(p, L, b0 + (warp >> 3), b0 + nb, p.G, 0);
            for (unsigned int ch = warp >> 3; ch < nb; ch += 4) {
                const ChunkFetch nf = fetch_chunk(p, L, b0 + ch + 4, b0 + nb, p.G, f.g < 0 ? 0 : f.g);
                ChunkWork x;
                expand_chunk(f, x);
                const unsigned int bytes = __reduce_add_sync(0xFFFFFFFFu, x.wsum);
                if (lane == 0) {
                    p.chunk_part[8ull * (b0 + ch) + (warp & 7)] = (unsigned short)bytes;
                    if (bytes) atomicAdd(&tot[ch], bytes);
                }
                f = nf;
            }
            __syncthreads();
            if (warp == 0) {   // running offsets per group, 32 chunks a turn
                for (unsigned int i0 = 0; i0 < nb; i0 += 32) {
                    const unsigned int i = i0 + lane;
                    const unsigned int t = i < nb ? tot[i] : 0u;
                    const int g = i < nb ? group_of_chunk(L.chunk_prefix, p.G, b0 + i) : -1;
                    unsigned int inc = t;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                        if (lane >= o) inc += x;
                    }
                    // the chunks of a group are neighbours: subtract what lies before the group's first lane
                    const unsigned int same = __match_any_sync(0xFFFFFFFFu, g);
                    const int head = __ffs(same) - 1, tail = 31 - __clz(same);
                    const unsigned int before = __shfl_sync(0xFFFFFFFFu, inc - t, head), upto = __shfl_sync(0xFFFFFFFFu, inc, tail);
                    if (i < nb) p.chunk_off[b0 + i] = (unsigned int)s.my_bytes[g] + inc - t - before;
                    __syncwarp();
                    if (g >= 0 && lane == head) s.my_bytes[g] += upto - before;
                    __syncwarp();
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    // (32 bits: a delta of more than a byte is 256 at least, and those of a group's keys add up to less than 2^31)
    if ((int)threadIdx.x < p.G)
        st_relaxed_gpu64(p.blk_bytes + threadIdx.x * MAX_GRID + blockIdx.x, ((unsigned long long)(FUSED ? epoch : 0u) << 32) | (unsigned int)s.my_bytes[threadIdx.x]);
}

// Bounded wait for the publications (epoch words) of blocks [0, count); false on every thread when one is missing.
__device__ bool wait_published(const CP& p, const unsigned int* flags, unsigned int count, unsigned int epoch, unsigned int where) {
    bool ok = true;
    if (threadIdx.x < count) {
        const long long t0 = clock64();
        unsigned int ns = 0;
        while (ld_acquire_gpu(&flags[threadIdx.x]) != epoch) {
            if (clock64() - t0 > p.budget) {
                skml_set_status(p.status, SKML_TIMEOUT_BARRIER, where);
                ok = false;
                break;
            }
            if (ns) __nanosleep(ns);
            if (ns < 200) ns += 20;
        }
    }
    return __syncthreads_and(ok) != 0;
}

// Sum of one word of the blocks [0, count) (see read_row), by a warp.
template <bool WAIT>
__device__ __forceinline__ bool sum_row(const CP& p, const unsigned long long* words, unsigned int count, unsigned int epoch, unsigned int where,
                                        unsigned long long& sum) {
    unsigned int c[MAX_GRID / 32];
    const bool ok = read_row<WAIT>(p, words, count, epoch, where, false, c);
    sum = 0;
#pragma unroll
    for (int k = 0; k < MAX_GRID / 32; ++k) sum += (threadIdx.x & 31) + 32 * k < count ? c[k] : 0u;
    sum = warp_sum(sum);
    return ok;
}

// The same for numbers of 64 bits, whose halves are words of their own: halves 2 i and 2 i + 1 of the i-th number of block `at`.
template <bool FUSED>
__device__ __forceinline__ void put_halves(unsigned long long* words, unsigned int i, unsigned int at, unsigned int epoch, unsigned long long v) {
    const unsigned long long tag = (unsigned long long)(FUSED ? epoch : 0u) << 32;
    st_relaxed_gpu64(words + (2 * i) * MAX_GRID + at, tag | (v & 0xFFFFFFFFull));
    st_relaxed_gpu64(words + (2 * i + 1) * MAX_GRID + at, tag | (v >> 32));
}
__device__ __forceinline__ unsigned long long get_halves(const unsigned long long* words, unsigned int i, unsigned int at) {
    return (__ldcg(words + (2 * i) * MAX_GRID + at) & 0xFFFFFFFFull) | (__ldcg(words + (2 * i + 1) * MAX_GRID + at) << 32);
}
template <bool WAIT>
__device__ __forceinline__ bool sum_halves(const CP& p, const unsigned long long* words, unsigned int i, unsigned int count, unsigned int epoch,
                                           unsigned int where, unsigned long long& sum) {
    unsigned long long lo, hi;
    const bool a = sum_row<WAIT>(p, words + (2 * i) * MAX_GRID, count, epoch, where, lo), b = sum_row<WAIT>(p, words + (2 * i + 1) * MAX_GRID, count, epoch, where, hi);
    sum = lo + (hi << 32);
    return a && b;
}

// Byte totals of the blocks before this one (they own the chunks before this block's run, so the
// sums give this block's starting offsets and the sizes of all earlier groups); a warp per group.
template <bool WAIT>
__device__ void pack_prefix(const CP& p, Smem& s, unsigned int epoch) {
    bool ok = true;
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < p.G) {
        unsigned long long v;
        ok = sum_row<WAIT>(p, p.blk_bytes + warp * MAX_GRID, blockIdx.x, epoch, 0x50u, v);
        if (lane == 0) s.pre_bytes[warp] = v;
    }
    ok = __syncthreads_and(ok) != 0;
    if (warp == 0) {
        // section starts of the groups this block can reach: all earlier groups are complete in pre_bytes
        // (plus this block's own part of the group its run starts in)
        unsigned long long size = 0, all;
        if (lane < p.G && L.n_g[lane]) size = skml_align16(8ull * ((s.pre_bytes[lane] + s.my_bytes[lane] + 7) / 8));
        const unsigned long long o = warp_prefix(size, all);
        if (lane < p.G) L.delta_off[lane] = L.off_deltas + o;
        if (lane == 0 && !ok) L.overflow = 1;
    }
    __syncthreads();
}

// Flag bytes, delta bytes and restart point of one eighth of a chunk (a warp, four adjacent keys a lane). `at`: byte
// offset of the chunk in its group's deltas; `before`: the chunk's bytes before this warp's; `lane_off`: this warp's
// bytes before this lane's; `bytes`: this warp's. The delta bytes are put together in shared memory at the alignment
// they have in the payload and leave in 16-byte units (bytes at the two ends, which neighbours share); byte stores
// from every lane, and scans and barriers of 256 threads per chunk, took 48 us of 10M keys.
__device__ __forceinline__ void pack_emit(const CP& p, Smem& s, const ChunkWork& c, unsigned long long at, unsigned int before,
                                          unsigned int lane_off, unsigned int bytes) {
    const Layout& L = s.lay;
    const int t = threadIdx.x & 255, lane = threadIdx.x & 31, g = c.g;
    const unsigned int first = c.j * SKML_RESTART_INTERVAL, i0 = 4u * t;
    // flags: (w - 1) most significant bit first at stream bits 2i, 2i+1 -> one byte per four keys
    // (a group's last chunk also writes the zero padding up to the section's 16-byte end: there the
    // threads beyond the last key hold widths of zero)
    const unsigned int flag_bytes = (L.n_g[g] + 63u) / 64u * 16u;
    const unsigned int fbyte = first / 4 + t;
    if (fbyte < flag_bytes) {
        unsigned int fb = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned int fv = c.w[u] ? c.w[u] - 1u : 0u;
            fb |= (((fv >> 1) & 1u) | ((fv & 1u) << 1)) << (2 * u);
        }
        p.payload[L.flag_off[g] + fbyte] = (unsigned char)fb;
    }
    const unsigned long long to = L.delta_off[g] + at + before;
    const unsigned int sh = (unsigned int)(to & 15ull), end = sh + bytes;
    uint4* const units = s.ps.stage[threadIdx.x >> 5];
    unsigned char* const stage = reinterpret_cast<unsigned char*>(units);
    __syncwarp();   // the previous bytes have left
    if (i0 < c.cnt) {
        unsigned char* dst = stage + sh + lane_off;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // the delta's bytes, most significant first and each bit-reversed: the reversed word's bytes in memory order
            const unsigned int x = c.w[u] ? __brev(c.d[u]) >> (32u - 8u * c.w[u]) : 0u;
            if (c.w[u] > 0) dst[0] = (unsigned char)x;
            if (c.w[u] > 1) dst[1] = (unsigned char)(x >> 8);
            if (c.w[u] > 2) {
                dst[2] = (unsigned char)(x >> 16);
                dst[3] = (unsigned char)(x >> 24);
            }
            dst += c.w[u];
        }
    }
    __syncwarp();
    unsigned char* const out = p.payload + (to - sh);
    const unsigned int u0 = (sh + 15u) / 16u, u1 = end / 16u;   // whole units
    for (unsigned int u = u0 + lane; u < u1; u += 32) st_v4(reinterpret_cast<uint4*>(out) + u, units[u]);
    // lanes 0 - 15: the unit the bytes start in, where they do not fill it from its start; lanes 16 - 31: the one they end in
    const unsigned int b = (lane & 16 ? 16u * u1 : 0u) + (lane & 15);
    if ((lane & 16 ? u1 >= u0 : sh != 0u) && b >= sh && b < end) out[b] = stage[b];
    if (t == 224 && c.j + 1 == (L.n_g[g] + SKML_RESTART_INTERVAL - 1) / SKML_RESTART_INTERVAL) {
        // the group's last chunk: clear the padding between the last delta byte and the section's end
        const unsigned long long endb = at + before + bytes;
        for (unsigned long long a = endb; a < skml_align16(8ull * ((endb + 7) / 8)); ++a) p.payload[L.delta_off[g] + a] = 0;
    }
    if (t == 0) {
        SkmlRestart r;
        r.prev_key = (unsigned int)c.prev0;
        r.flag_bit_off = 2u * first;
        r.delta_bit_off = 8ull * at;
        *reinterpret_cast<SkmlRestart*>(p.payload + L.restart_off[g] + (unsigned long long)c.j * sizeof(SkmlRestart)) = r;
    }
}

// Pass B: the key code of this block's chunks. `c`, `boff`, `total`: pass A's only round, where it had one (`kept`).
// Of longer runs every warp takes its eighths on its own, the next one's keys on their way.
__device__ void pack_write(const CP& p, Smem& s, unsigned int my_begin, unsigned int my_end, bool kept, ChunkWork& c, unsigned int boff,
                           unsigned int total) {
    if (s.lay.overflow) return;
    const unsigned int sb = threadIdx.x >> 8, lane = threadIdx.x & 31, eighth = (threadIdx.x >> 5) & 7;
    if (my_end - my_begin <= 4) {
        unsigned int off = s.sub_off[sb];
        if (!kept) {   // staged launches: pass A's counts were in another launch's registers and shared memory
            load_chunk(p, s.lay, my_begin + sb, my_end, p.G, c);
            boff = sub_scan(s, c.wsum, total);
            if ((threadIdx.x & 255) == 0) s.sub_total[sb] = total;
            __syncthreads();
            off = 0;
            for (unsigned int k = 0; k < sb && c.g >= 0; ++k)
                if (my_begin + k >= s.lay.chunk_prefix[c.g]) off += s.sub_total[k];
        }
        const unsigned int before = __shfl_sync(0xFFFFFFFFu, boff, 0);
        const unsigned int bytes = __shfl_sync(0xFFFFFFFFu, boff + c.wsum, 31) - before;
        if (c.g >= 0) pack_emit(p, s, c, s.pre_bytes[c.g] + off, before, boff - before, bytes);
    } else {
        const unsigned int ch0 = my_begin + sb;
        ChunkFetch f = fetch_chunk(p, s.lay, ch0, my_end, p.G, 0);
        // lane k < 8: bytes of the chunk's eighth k; all lanes: the chunk's offset
        auto part_of = [&](unsigned int ch) { return ch < my_end && lane < eighth ? (unsigned int)__ldcg(&p.chunk_part[8ull * ch + lane]) : 0u; };
        unsigned int part = part_of(ch0), off = ch0 < my_end ? __ldcg(&p.chunk_off[ch0]) : 0u;
        for (unsigned int ch = ch0; ch < my_end; ch += 4) {
            const ChunkFetch nf = fetch_chunk(p, s.lay, ch + 4, my_end, p.G, f.g);
            const unsigned int npart = part_of(ch + 4), noff = ch + 4 < my_end ? __ldcg(&p.chunk_off[ch + 4]) : 0u;
            ChunkWork x;
            expand_chunk(f, x);
            unsigned int inc = x.wsum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= (unsigned int)o) inc += t;
            }
            pack_emit(p, s, x, s.pre_bytes[x.g] + off, __reduce_add_sync(0xFFFFFFFFu, part), inc - x.wsum,
                      __shfl_sync(0xFFFFFFFFu, inc, 31));
            f = nf;
            part = npart;
            off = noff;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// S5, DeltaAdaptive key code (the reference's live encoder, binary/DeltaAdaptiveEncoder.java:23-112).
// Flags and deltas are bit streams: per group, every delta takes b * iv bits (b = 32 / m bits per
// interval, iv = intervals needed) and a flag of log2(m) bits holding iv - 1, or iv one-bits and a
// zero-bit ("unary" flags); m and the flag kind minimise the estimated bits per key over the group's
// histogram of delta widths. Chunk starts are therefore bit positions, adjacent chunks share stream
// words, and the sections' sizes depend on the data: the two sections of a group follow each other
// at the end of the payload, and the (pre-zeroed) shared words are completed with atomic ORs.
// ---------------------------------------------------------------------------
__device__ __noinline__ void push_bytes(const CP& p, unsigned long long lo, unsigned long long hi);

__device__ __forceinline__ int da_bits_needed(unsigned int d) { return d == 0u ? 1 : 32 - __clz(d); }

// Pass 0: histogram of the delta widths of this block's chunks, per group, added to the global one.
__device__ void apack_histogram(const CP& p, Smem& s, unsigned int my_begin, unsigned int my_end) {
    const Layout& L = s.lay;
    unsigned int* hist = s.cs.stage_d[0];  // [G][32], the staging area is idle in this pass
    for (int t = threadIdx.x; t < SKML_MAX_GROUPS * 32; t += blockDim.x) hist[t] = 0;
    __syncthreads();
    for (unsigned int c0 = my_begin; c0 < my_end; c0 += 4) {
        ChunkWork c;
        load_chunk(p, L, c0 + (threadIdx.x >> 8), my_end, p.G, c);
        if (c.g >= 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c.w[u]) atomicAdd(&hist[c.g * 32 + (da_bits_needed(c.d[u]) & 31)], 1u);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < p.G * 32; t += blockDim.x)
        if (hist[t]) atomicAdd(&p.key_hist[t], hist[t]);
}

__device__ __forceinline__ unsigned long long stream_bytes(unsigned long long bits) { return skml_align16(8ull * ((bits + 63) / 64)); }

// Pass 1 prelude (every block): interval count and flag kind of every group from the complete
// histogram. The histogram also gives the exact lengths of the two bit streams of every group, so the
// whole layout of the key sections is known here, before a single key is coded.
__device__ __forceinline__ void apack_modes(const CP& p, Smem& s, int first, int step) {   // a warp per group, lane = delta width
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31;
    for (int g = first; g < p.G; g += step) {
        double* prob = reinterpret_cast<double*>(s.cs.stage_d) + 32 * g;   // (the staging area is idle until pass 2)
        const unsigned int h = __ldcg(&p.key_hist[g * 32 + lane]), n = L.n_g[g];
        prob[lane] = __ddiv_rn((double)h, (double)(n > 0 ? n : 1));
        __syncwarp();
        // the reference's estimates in the same double arithmetic, operation by operation (explicit round-to-nearest
        // intrinsics keep the compiler from fusing multiply-adds), one lane per interval count m
        double t1 = 0.0, t2 = 0.0;
        if (lane < 4) {
            const int m = 2 << lane, b = 32 / m;
            double sum = 0.0;
            for (int i = 0; i < m; ++i) {
                double ip = 0.0;
                for (int j = 0; j < b; ++j) ip = __dadd_rn(ip, prob[i * b + j]);
                sum = __dadd_rn(sum, __dmul_rn((double)(i + 1), ip));
            }
            t1 = __dadd_rn(__dmul_rn(sum, (double)b), (double)(lane + 1));
            t2 = __dadd_rn(__dmul_rn(sum, (double)(b + 1)), 1.0);
        }
        double best = 32.0;
        unsigned int num = 1, kind = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double a = __shfl_sync(0xFFFFFFFFu, t1, q), c = __shfl_sync(0xFFFFFFFFu, t2, q);
            if (a < best) {
                best = a;
                num = 2u << q;
                kind = 0;
            }
            if (c < best) {
                best = c;
                num = 2u << q;
                kind = 1;
            }
        }
        const unsigned int b = 32u / num, fb = 31u - (unsigned int)__clz(num);
        const unsigned int need = lane ? (unsigned int)lane : 32u;   // bin 0 holds the 32-bit deltas (need & 31)
        const unsigned long long iv = (need + b - 1) / b;
        const unsigned long long fbits = warp_sum((unsigned long long)h * (kind ? iv + 1 : fb));
        const unsigned long long dbits = warp_sum((unsigned long long)h * b * iv);
        if (lane == 0) {
            L.num_iv[g] = num;
            L.flag_kind[g] = kind;
            L.flag_bits[g] = fbits;
            L.delta_bits[g] = dbits;
        }
    }
}

// And the key sections' places behind what lies before them (one warp).
__device__ __forceinline__ void apack_places(const CP& p, Smem& s) {
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31;
    {
        const bool any = lane < p.G && L.n_g[lane];
        const unsigned long long f = any ? stream_bytes(L.flag_bits[lane]) : 0ull, d = any ? stream_bytes(L.delta_bits[lane]) : 0ull;
        unsigned long long all;
        const unsigned long long o = L.off_keys + warp_prefix(f + d, all);
        if (lane < p.G) {
            L.flag_off[lane] = o;
            L.delta_off[lane] = o + f;
        }
        if (lane == 0) {
            L.total_bytes = L.off_keys + all;
            if (L.total_bytes > (unsigned long long)p.slot_capacity) {
                L.overflow = 1;
                skml_set_status(p.status, SKML_CAPACITY, 0x37u);
            }
        }
    }
}

__device__ void apack_choose(const CP& p, Smem& s) {
    apack_modes(p, s, threadIdx.x >> 5, SKML_WARPS);
    __syncthreads();
    if (threadIdx.x < 32) apack_places(p, s);
    __syncthreads();
}


struct KeyCode {
    unsigned int fv, fw, dw;  // flag value / width, delta width (the delta value is the delta itself)
};
__device__ __forceinline__ KeyCode da_code(unsigned int d, unsigned int m, unsigned int kind) {
    const int b = 32 / (int)m, fb = 31 - __clz(m);
    const int iv = (da_bits_needed(d) + b - 1) / b;
    KeyCode k;
    k.fw = kind ? (unsigned int)(iv + 1) : (unsigned int)fb;
    k.fv = kind ? ((1u << (iv + 1)) - 2u) : (unsigned int)(iv - 1);
    k.dw = (unsigned int)(b * iv);
    return k;
}

// Writes `nb` (<= 32) bits of `value`, most significant first, at bit offset `off` of a zeroed
// shared-memory word array (stream bit p = bit (p & 31) of word p >> 5, as in java.util.BitSet).
__device__ __forceinline__ void put_bits_shared(unsigned int* words, unsigned int off, unsigned int value, unsigned int nb) {
    if (nb == 0) return;
    const unsigned int rv = __brev(value) >> (32u - nb);
    const unsigned int sh = off & 31u, w = off >> 5;
    atomicOr(&words[w], rv << sh);
    if (sh + nb > 32u) atomicOr(&words[w + 1], rv >> (32u - sh));
}

// Pass 1: flag and delta bits of this block's chunks -> chunk bit offsets inside the block's part of
// each group, the block's bit totals per group (published for the blocks after it).
template <bool FUSED>
__device__ void apack_measure(const CP& p, Smem& s, unsigned int epoch, unsigned int my_begin, unsigned int my_end) {
    const Layout& L = s.lay;
    if (threadIdx.x < 2 * SKML_MAX_GROUPS) s.my_bits[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned int c0 = my_begin; c0 < my_end; c0 += 4) {
        ChunkWork c;
        load_chunk(p, L, c0 + (threadIdx.x >> 8), my_end, p.G, c);
        unsigned int packed = 0;  // flag bits (<= 17408 per chunk) in the low half, delta bits (<= 32768) above
        if (c.g >= 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c.w[u]) {
                    const KeyCode k = da_code(c.d[u], L.num_iv[c.g], L.flag_kind[c.g]);
                    packed += k.fw + (k.dw << 16);
                }
        }
        unsigned int total;
        sub_scan(s, packed, total);
        if ((threadIdx.x & 255) == 0) s.sub_total[threadIdx.x >> 8] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int q = 0; q < 4 && c0 + q < my_end; ++q) {
                int g = 0;
                while (g + 1 < p.G && c0 + q >= L.chunk_prefix[g + 1]) ++g;
                p.chunk_off[2 * (c0 + q)] = (unsigned int)s.my_bits[2 * g];
                p.chunk_off[2 * (c0 + q) + 1] = (unsigned int)s.my_bits[2 * g + 1];
                s.my_bits[2 * g] += s.sub_total[q] & 0xFFFFu;
                s.my_bits[2 * g + 1] += s.sub_total[q] >> 16;
            }
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < 2 * p.G) put_halves<FUSED>(p.blk_bits, threadIdx.x, blockIdx.x, epoch, s.my_bits[threadIdx.x]);
}

// Bit totals of the blocks before this one -> this block's starting bit offsets inside the streams.
template <bool WAIT>
__device__ void apack_prefix(const CP& p, Smem& s, unsigned int epoch) {
    bool ok = true;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int g = warp; g < 2 * p.G; g += SKML_WARPS) {
        unsigned long long v;
        ok = sum_halves<WAIT>(p, p.blk_bits, g, blockIdx.x, epoch, 0x52u, v) && ok;
        if (lane == 0) s.pre_bits[g] = v;
    }
    if (!__syncthreads_and(ok) && threadIdx.x == 0) s.lay.overflow = 1;
    __syncthreads();
}

// One stream segment staged in shared memory -> the payload: whole words are stored, the first and
// the last word may be shared with the neighbouring chunks and are completed with atomic ORs.
__device__ __forceinline__ void flush_stream(unsigned int* dst_words, const unsigned int* stage, unsigned long long start_bit,
                                             unsigned int nbits) {
    if (nbits == 0) return;
    const unsigned int sh = (unsigned int)(start_bit & 31ull);
    const unsigned int nw = (sh + nbits + 31u) >> 5;
    unsigned int* dst = dst_words + (start_bit >> 5);
    for (unsigned int w = threadIdx.x & 255; w < nw; w += 256) {
        const unsigned int v = stage[w];
        const bool shared_word = (w == 0 && sh != 0) || (w == nw - 1 && ((sh + nbits) & 31u) != 0);
        if (shared_word) {
            if (v) atomicOr(dst + w, v);
        } else {
            dst[w] = v;
        }
    }
}

// Pass 2: the bit streams and restart points of this block's chunks.
__device__ void apack_write(const CP& p, Smem& s, unsigned int my_begin, unsigned int my_end) {
    const Layout& L = s.lay;
    if (L.overflow) return;
    const int t = threadIdx.x & 255, sb = threadIdx.x >> 8;
    for (unsigned int c0 = my_begin; c0 < my_end; c0 += 4) {
        ChunkWork c;
        const unsigned int ch = c0 + sb;
        load_chunk(p, L, ch, my_end, p.G, c);
        KeyCode kc[4];
        unsigned int packed = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            kc[u].fv = kc[u].fw = kc[u].dw = 0;
            if (c.g >= 0 && c.w[u]) {
                kc[u] = da_code(c.d[u], L.num_iv[c.g], L.flag_kind[c.g]);
                packed += kc[u].fw + (kc[u].dw << 16);
            }
        }
        for (int i = t; i < AP_STAGE_F; i += 256) s.cs.stage_f[sb][i] = 0;
        for (int i = t; i < AP_STAGE_D; i += 256) s.cs.stage_d[sb][i] = 0;
        unsigned int total;
        const unsigned int ex = sub_scan(s, packed, total);  // (its barriers also publish the cleared staging words)
        unsigned long long fs = 0, ds = 0;
        if (c.g >= 0) {
            fs = s.pre_bits[2 * c.g] + __ldcg(&p.chunk_off[2 * ch]);
            ds = s.pre_bits[2 * c.g + 1] + __ldcg(&p.chunk_off[2 * ch + 1]);
            unsigned int fo = (unsigned int)(fs & 31ull) + (ex & 0xFFFFu), dof = (unsigned int)(ds & 31ull) + (ex >> 16);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                put_bits_shared(s.cs.stage_f[sb], fo, kc[u].fv, kc[u].fw);
                put_bits_shared(s.cs.stage_d[sb], dof, c.d[u], kc[u].dw);
                fo += kc[u].fw;
                dof += kc[u].dw;
            }
        }
        __syncthreads();
        if (c.g >= 0) {
            flush_stream(reinterpret_cast<unsigned int*>(p.payload + L.flag_off[c.g]), s.cs.stage_f[sb], fs, total & 0xFFFFu);
            flush_stream(reinterpret_cast<unsigned int*>(p.payload + L.delta_off[c.g]), s.cs.stage_d[sb], ds, total >> 16);
            if (t == 0) {
                SkmlRestart r;
                r.prev_key = (unsigned int)c.prev0;
                r.flag_bit_off = (unsigned int)fs;
                r.delta_bit_off = ds;
                *reinterpret_cast<SkmlRestart*>(p.payload + L.restart_off[c.g] + (unsigned long long)c.j * sizeof(SkmlRestart)) = r;
            }
        }
        __syncthreads();  // the staging words are cleared again by the next round
    }
}

// The restart points and the 16-byte units of the two bit streams that hold bits of this block only
// -> the peers' slots. Units that hold a block border are sent by the last block once every block is done.
__device__ __noinline__ void apush_own_chunks(const CP& p, Smem& s, unsigned int my_begin, unsigned int my_end) {
    const Layout& L = s.lay;
    if (p.world <= 1 || L.overflow || my_begin >= my_end) return;
    __syncthreads();
    for (int g = 0; g < p.G; ++g) {
        const unsigned int c0 = max(my_begin, L.chunk_prefix[g]), c1 = min(my_end, L.chunk_prefix[g + 1]);
        if (c0 >= c1) continue;
        const bool last = c1 == L.chunk_prefix[g + 1];
        push_bytes(p, L.restart_off[g] + 16ull * (c0 - L.chunk_prefix[g]), L.restart_off[g] + 16ull * (c1 - L.chunk_prefix[g]));
        for (int k = 0; k < 2; ++k) {
            const unsigned long long a = s.pre_bits[2 * g + k], b = a + s.my_bits[2 * g + k];
            const unsigned long long lo = 16ull * ((a + 127) / 128), hi = last ? stream_bytes(k ? L.delta_bits[g] : L.flag_bits[g]) : 16ull * (b / 128);
            const unsigned long long base = k ? L.delta_off[g] : L.flag_off[g];
            if (hi > lo) push_bytes(p, base + lo, base + hi);
        }
    }
}

// The last block, after every block has written its chunks: the stream units that hold a block border.
__device__ __noinline__ void apush_borders(const CP& p, Smem& s) {
    const Layout& L = s.lay;
    if (p.world <= 1 || L.overflow) return;
    const unsigned int total = L.chunk_prefix[p.G];
    unsigned int per = (total + gridDim.x - 1) / gridDim.x;
    per = (per + 3u) & ~3u;
    const unsigned int b = threadIdx.x;
    if (b >= 1 && b < gridDim.x && (unsigned long long)per * b < total) {
        const unsigned int cs = per * b;
        int g = 0;
        while (g + 1 < p.G && cs >= L.chunk_prefix[g + 1]) ++g;
        if (cs != L.chunk_prefix[g]) {  // the run of block b starts inside group g
            unsigned long long a[2] = {0, 0};
            for (unsigned int q = 0; q < b; ++q) {
                a[0] += get_halves(p.blk_bits, 2 * g, q);
                a[1] += get_halves(p.blk_bits, 2 * g + 1, q);
            }
            for (int k = 0; k < 2; ++k) {
                if ((a[k] & 127ull) == 0) continue;
                const unsigned long long off = (k ? L.delta_off[g] : L.flag_off[g]) + 16ull * (a[k] / 128);
                const uint4 v = ld_cg_v4(reinterpret_cast<const uint4*>(p.payload + off));
                for (unsigned int r = 0; r < p.world; ++r)
                    if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + off), v);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// S5, Huffman-coded sketch tables (cell_bits = 0; the reference codes every table this way when it
// serialises a sketch: sketch/frequency/MinMaxSketch.java:88-97, binary/HuffmanEncoder.java:88-124).
// Section of one group: u32 {items, 64-bit words, cells, restart interval}; items x {i32 value,
// i32 code, i32 code length}, ascending by value; the code stream (most significant bit first in
// java.util.BitSet order); then, 16-byte aligned, one u32 stream offset per 128 cells (not in the
// reference: it lets a decoder start anywhere). The symbols of a group are the buckets of its range
// plus the "never written" cell (Integer.MAX_VALUE), at most HUF_MAX_SYMS of them. Any prefix code is
// valid on the wire (the items carry the codes); the coder builds an optimal one from the cell
// histogram and assigns canonical code words.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned int huf_slot(const Layout& L, int g, unsigned int cell) {
    const unsigned int sidx = cell == SKML_EMPTY_CELL ? L.nsym[g] - 1u : (cell & 0xFFFFu) - L.sym_lo[g];
    return L.sym_lo[g] + (unsigned int)g + (sidx < L.nsym[g] ? sidx : L.nsym[g] - 1u);
}

// Table chunks (1024 cells of one group's table, group-major) of the block whose turn it is: a contiguous run.
__device__ __forceinline__ void tchunk_run(const Layout& L, int G, unsigned int turn, unsigned int& t_begin, unsigned int& t_end) {
    const unsigned int total = L.tchunk_prefix[G];
    unsigned int per = (total + gridDim.x - 1) / gridDim.x;
    per = (per + 3u) & ~3u;
    t_begin = min(total, per * turn);
    t_end = min(total, t_begin + per);
}

struct CellWork {
    int g;
    unsigned int j, cnt;      // chunk index inside the group's table, cells in the chunk
    unsigned int cell[4];     // this thread's cells (32-bit working form)
};

__device__ __forceinline__ void load_cells(const CP& p, const Layout& L, unsigned int ch, unsigned int ch_end, int G, CellWork& c) {
    const unsigned int t = threadIdx.x & 255;
    c.g = -1;
    c.cnt = 0;
    c.j = 0;
    if (ch >= ch_end) return;
    int g = 0;
    while (g + 1 < G && ch >= L.tchunk_prefix[g + 1]) ++g;
    c.g = g;
    c.j = ch - L.tchunk_prefix[g];
    const unsigned int first = c.j * 1024u;
    c.cnt = min(1024u, L.cells[g] - first);
    const unsigned int* tab = p.tables + L.tab32_off[g] + first;
#pragma unroll
    for (int u = 0; u < 4; ++u) c.cell[u] = 4u * t + u < c.cnt ? __ldcg(tab + 4u * t + u) : SKML_EMPTY_CELL;
}

// Symbol ranges, cell counts and table chunks of the groups (every block, thread 0).
__device__ void huf_ranges(const CP& p, Smem& s) {
    Layout& L = s.lay;
    if (threadIdx.x == 0) {
        unsigned int ch = 0;
        for (int g = 0; g < p.G; ++g) {
            const int lo = g ? s.qi.edges[g - 1] : 0, hi = s.qi.edges[g];
            L.sym_lo[g] = (unsigned int)lo;
            L.nsym[g] = (unsigned int)(hi > lo ? hi - lo : 0) + 1u;
            L.cells[g] = (unsigned int)p.rows * L.col[g];
            L.tchunk_prefix[g] = ch;
            ch += (L.cells[g] + 1023u) / 1024u;
            if (L.n_g[g] && L.nsym[g] > HUF_MAX_SYMS) {
                L.overflow = 1;
                skml_set_status(p.status, SKML_BAD_INPUT, 0x38u);
            }
        }
        L.tchunk_prefix[p.G] = ch;
    }
    __syncthreads();
}

// Pass 0: histogram of the cell symbols of this block's table chunks, added to the global one.
__device__ void huf_histogram(const CP& p, Smem& s, unsigned int t_begin, unsigned int t_end) {
    const Layout& L = s.lay;
    unsigned int* hist = s.cs.huf_code;  // idle until the codes are built
    for (int t = threadIdx.x; t < SKML_GPU_MAX_BINS + SKML_MAX_GROUPS; t += blockDim.x) hist[t] = 0;
    __syncthreads();
    for (unsigned int c0 = t_begin; c0 < t_end; c0 += 4) {
        CellWork c;
        load_cells(p, L, c0 + (threadIdx.x >> 8), t_end, p.G, c);
        if (c.g >= 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (4u * (threadIdx.x & 255) + u < c.cnt) atomicAdd(&hist[huf_slot(L, c.g, c.cell[u])], 1u);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < s.qi.bin_num + p.G; t += blockDim.x)
        if (hist[t]) atomicAdd(&p.cell_hist[t], hist[t]);
    __syncthreads();
}

// Optimal prefix code of every group from the complete histogram (every block; one warp per group,
// eight groups at a time), canonical code words, section sizes and the layout that follows the tables.
// Only the merges are a chain (one lane, the two candidates of either queue read side by side); sorting,
// code lengths (a walk to the root per leaf) and code words are the whole warp's. (One lane for all of it,
// reading the histogram from L2, was some 35 us of a launch.)
// ADAPTIVE: the other warps choose the key code's modes meanwhile, and its places follow (170,000 keys: with the counts sent by themselves and the
// tables coded by other blocks than the keys, the launch 66 -> 54 us; 560,000 keys 96 -> 84).
template <bool ADAPTIVE>
__device__ void huf_build(const CP& p, Smem& s) {
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    HufScratch* scratch = s.cs.huf_scratch;
    for (int t = threadIdx.x; t < SKML_GPU_MAX_BINS + SKML_MAX_GROUPS; t += blockDim.x) {
        s.cs.huf_len[t] = 0;
        s.cs.huf_code[t] = 0;
    }
    __syncthreads();
    if (warp < 8 && !L.overflow) {
        HufScratch& h = scratch[warp];
        for (int g = warp; g < p.G; g += 8) {
            const unsigned int n = L.nsym[g], base = L.sym_lo[g] + (unsigned int)g;
            if (L.n_g[g] == 0) {
                if (lane == 0) {
                    L.items[g] = 0;
                    L.tbits[g] = 0;
                }
                continue;
            }
            unsigned int m = 0;   // symbols that occur
            for (unsigned int a = lane; a < n; a += 32) {
                const unsigned int c = __ldcg(&p.cell_hist[base + a]);
                h.cnt[a] = c;
                m += c ? 1u : 0u;
            }
            m = __reduce_add_sync(0xFFFFFFFFu, m);
            h.next[lane] = 0;
            if (lane < 2) h.next[32 + lane] = 0;
            __syncwarp();
            // rank sort of the present symbols by (count, symbol): every lane ranks its symbols
            for (unsigned int a = lane; a < n; a += 32) {
                const unsigned int ca = h.cnt[a];
                if (!ca) continue;
                unsigned int r = 0;
                for (unsigned int b = 0; b < n; ++b) {
                    const unsigned int cb = h.cnt[b];
                    if (cb && (cb < ca || (cb == ca && b < a))) ++r;
                }
                h.ord[r] = (unsigned short)a;
                h.w[r] = ca;
            }
            if (lane < 2) h.w[m + lane] = 0xFFFFFFFFu;
            __syncwarp();
            if (lane == 0 && m > 1) {
                // two-queue construction: leaves and internal nodes are both consumed in ascending weight, leaves first
                unsigned int li = 0, ii = 0;
                h.iw[0] = h.iw[1] = 0xFFFFFFFFu;
                for (unsigned int ni = 0; ni + 1 < m; ++ni) {
                    const unsigned int l0 = h.w[li], l1 = h.w[li + 1], i0 = h.iw[ii], i1 = h.iw[ii + 1];
                    const bool leaf_a = l0 <= i0;
                    const bool leaf_b = (leaf_a ? l1 : l0) <= (leaf_a ? i0 : i1);
                    h.iw[ni] = (leaf_a ? l0 : i0) + (leaf_b ? (leaf_a ? l1 : l0) : (leaf_a ? i0 : i1));
                    h.iw[ni + 1] = h.iw[ni + 2] = 0xFFFFFFFFu;
                    if (leaf_a) h.pl[li++] = (unsigned short)ni;
                    else h.pi[ii++] = (unsigned short)ni;
                    if (leaf_b) h.pl[li++] = (unsigned short)ni;
                    else h.pi[ii++] = (unsigned short)ni;
                }
            }
            __syncwarp();
            unsigned long long bits = 0;
            unsigned int longest = 0;
            for (unsigned int i = lane; i < m; i += 32) {
                unsigned int len = 1;   // (a single symbol gets the one-bit code 0)
                if (m > 1)
                    for (unsigned int j = h.pl[i]; j != m - 2; j = h.pi[j]) ++len;   // node m - 2 is the root
                s.cs.huf_len[base + h.ord[i]] = (unsigned char)(len < 32 ? len : 32);
                if (len < 32) atomicAdd(&h.next[len], 1u);
                longest = max(longest, len);
                bits += (unsigned long long)h.w[i] * len;
            }
            bits = warp_sum(bits);
            longest = __reduce_max_sync(0xFFFFFFFFu, longest);
            __syncwarp();
            // canonical code words: lengths ascending, symbols ascending inside a length
            unsigned int first = 0;
            for (int k = 1; k < lane; ++k) first = (first + h.next[k]) << 1;
            __syncwarp();
            h.next[lane] = first;
            __syncwarp();
            for (unsigned int a0 = 0; a0 < n; a0 += 32) {
                const unsigned int a = a0 + lane, len = a < n ? s.cs.huf_len[base + a] : 0u;
                const unsigned int same = __match_any_sync(0xFFFFFFFFu, len);
                if (len && len < 32) s.cs.huf_code[base + a] = h.next[len] + (unsigned int)__popc(same & lanemask_lt());
                __syncwarp();
                if (len && len < 32 && (same & lanemask_lt()) == 0) h.next[len] += (unsigned int)__popc(same);
                __syncwarp();
            }
            if (lane == 0) {
                if (longest > 31) {
                    L.overflow = 1;
                    skml_set_status(p.status, SKML_BAD_INPUT, 0x39u);
                }
                L.items[g] = m;
                L.tbits[g] = bits;
            }
            __syncwarp();
        }
    } else if (ADAPTIVE && warp >= 8) {
        apack_modes(p, s, warp - 8, SKML_WARPS - 8);
    }
    __syncthreads();
    if (warp == 0) {   // sections start at multiples of 16, so their sizes do not depend on where
        const unsigned int n = lane < p.G ? L.n_g[lane] : 0u;
        unsigned long long stream = 0, restart = 0, size = 0, all, worst;
        if (n) {
            stream = 16ull + 12ull * L.items[lane];
            restart = skml_align16(stream + 8ull * ((L.tbits[lane] + 63) / 64));
            size = skml_align16(restart + 4ull * ((L.cells[lane] + HUF_RESTART - 1) / HUF_RESTART));
        }
        const unsigned long long o = L.off_tables + warp_prefix(size, all);
        const bool adaptive = p.key_encoder == SKML_KEYS_DELTA_ADAPTIVE;
        warp_prefix(lane < p.G ? skml_align16(4ull * n + 8) + (adaptive ? skml_align16(17ull * n / 8 + 8) : 0ull) : 0ull, worst);
        if (lane < p.G) {
            L.table_off[lane] = o;
            if (n) {
                L.tstream_off[lane] = o + stream;
                L.trestart_off[lane] = o + restart;
            }
        }
        if (lane == 0) {
            L.off_deltas = L.off_keys = L.off_tables + all;
            if (L.off_deltas + worst > (unsigned long long)p.slot_capacity && !L.overflow) {
                L.overflow = 1;
                skml_set_status(p.status, SKML_CAPACITY, 0x3Au);
            }
        }
        __syncwarp();
        if (ADAPTIVE) apack_places(p, s);
    }
    __syncthreads();
}

// Pass 1: code bits of this block's table chunks -> chunk offsets inside the block's part of each
// group's stream, the block's bit totals per group (published with the key counts).
template <bool FUSED>
__device__ void huf_measure(const CP& p, Smem& s, unsigned int epoch, unsigned int turn, unsigned int t_begin, unsigned int t_end) {
    const Layout& L = s.lay;
    if (threadIdx.x < SKML_MAX_GROUPS) s.my_tbits[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned int c0 = t_begin; c0 < t_end; c0 += 4) {
        CellWork c;
        load_cells(p, L, c0 + (threadIdx.x >> 8), t_end, p.G, c);
        unsigned int bits = 0;
        if (c.g >= 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (4u * (threadIdx.x & 255) + u < c.cnt) bits += s.cs.huf_len[huf_slot(L, c.g, c.cell[u])];
        }
        unsigned int total;
        sub_scan(s, bits, total);
        if ((threadIdx.x & 255) == 0) s.sub_total[threadIdx.x >> 8] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int q = 0; q < 4 && c0 + q < t_end; ++q) {
                int g = 0;
                while (g + 1 < p.G && c0 + q >= L.tchunk_prefix[g + 1]) ++g;
                p.tchunk_off[c0 + q] = (unsigned int)s.my_tbits[g];
                s.my_tbits[g] += s.sub_total[q];
            }
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < p.G) put_halves<FUSED>(p.blk_tbits, threadIdx.x, turn, epoch, s.my_tbits[threadIdx.x]);
}

// Table bits of the blocks whose turn is before this one's.
template <bool WAIT>
__device__ void huf_prefix(const CP& p, Smem& s, unsigned int epoch, unsigned int turn) {
    bool ok = true;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < p.G) {
        unsigned long long v;
        ok = sum_halves<WAIT>(p, p.blk_tbits, warp, turn, epoch, 0x53u, v);
        if (lane == 0) s.pre_tbits[warp] = v;
    }
    if (!__syncthreads_and(ok) && threadIdx.x == 0) s.lay.overflow = 1;
    __syncthreads();
}

// Pass 2: code streams and restart offsets of this block's table chunks; section head and items by
// the block that owns a group's first chunk.
__device__ void huf_write(const CP& p, Smem& s, unsigned int t_begin, unsigned int t_end) {
    const Layout& L = s.lay;
    if (L.overflow) return;
    const int t = threadIdx.x & 255, sb = threadIdx.x >> 8;
    for (unsigned int c0 = t_begin; c0 < t_end; c0 += 4) {
        CellWork c;
        const unsigned int ch = c0 + sb;
        load_cells(p, L, ch, t_end, p.G, c);
        unsigned int len[4], code[4], bits = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            len[u] = code[u] = 0;
            if (c.g >= 0 && 4u * t + u < c.cnt) {
                const unsigned int slot = huf_slot(L, c.g, c.cell[u]);
                len[u] = s.cs.huf_len[slot];
                code[u] = s.cs.huf_code[slot];
                bits += len[u];
            }
        }
        for (int i = t; i < AP_STAGE_D; i += 256) s.cs.stage_d[sb][i] = 0;
        unsigned int total;
        const unsigned int ex = sub_scan(s, bits, total);
        unsigned long long start = 0;
        if (c.g >= 0) {
            start = s.pre_tbits[c.g] + __ldcg(&p.tchunk_off[ch]);
            unsigned int off = (unsigned int)(start & 31ull) + ex;
            if (4u * t < c.cnt && ((c.j * 1024u + 4u * t) % HUF_RESTART) == 0)
                reinterpret_cast<unsigned int*>(p.payload + L.trestart_off[c.g])[(c.j * 1024u + 4u * t) / HUF_RESTART] =
                    (unsigned int)(start + ex);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                put_bits_shared(s.cs.stage_d[sb], off, code[u], len[u]);
                off += len[u];
            }
        }
        __syncthreads();
        if (c.g >= 0) {
            flush_stream(reinterpret_cast<unsigned int*>(p.payload + L.tstream_off[c.g]), s.cs.stage_d[sb], start, total);
            if (c.j == 0) {
                // this sub-block owns the group's first chunk: section head and items (ascending by value)
                const int g = c.g;
                unsigned int* head = reinterpret_cast<unsigned int*>(p.payload + L.table_off[g]);
                if (t == 0) {
                    head[0] = L.items[g];
                    head[1] = (unsigned int)((L.tbits[g] + 63) / 64);
                    head[2] = L.cells[g];
                    head[3] = HUF_RESTART;
                }
                if (t < 32) {
                    const unsigned int base = L.sym_lo[g] + (unsigned int)g, n = L.nsym[g];
                    unsigned int seen = 0;
                    for (unsigned int a0 = 0; a0 < n; a0 += 32) {
                        const unsigned int a = a0 + t;
                        const unsigned int ln = a < n ? s.cs.huf_len[base + a] : 0u;
                        const unsigned int present = __ballot_sync(0xFFFFFFFFu, ln != 0);
                        if (ln) {
                            int* rec = reinterpret_cast<int*>(head + 4) + 3 * (seen + __popc(present & ((1u << t) - 1u)));
                            rec[0] = a + 1 == n ? 0x7FFFFFFF : (int)(L.sym_lo[g] + a);
                            rec[1] = (int)s.cs.huf_code[base + a];
                            rec[2] = (int)ln;
                        }
                        seen += __popc(present);
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Absolute byte range of the 16-byte units that hold only bits [a, b) of a stream starting at byte
// `base` (4-byte aligned): from the first unit boundary at or after bit a to the last one at or before b.
__device__ __forceinline__ void own_units(unsigned long long base, unsigned long long a, unsigned long long b,
                                          unsigned long long& lo, unsigned long long& hi) {
    lo = 16ull * ((8ull * base + a + 127ull) / 128ull);
    hi = 16ull * ((8ull * base + b) / 128ull);
}

// The parts of the coded tables this block wrote -> the peers' slots (units that hold a block border
// are sent by block 0 once every block is done).
__device__ __noinline__ void huf_push_own(const CP& p, Smem& s, unsigned int t_begin, unsigned int t_end) {
    const Layout& L = s.lay;
    if (p.world <= 1 || L.overflow || t_begin >= t_end) return;
    __syncthreads();
    for (int g = 0; g < p.G; ++g) {
        const unsigned int c0 = max(t_begin, L.tchunk_prefix[g]), c1 = min(t_end, L.tchunk_prefix[g + 1]);
        if (c0 >= c1) continue;
        const bool first = c0 == L.tchunk_prefix[g], last = c1 == L.tchunk_prefix[g + 1];
        const unsigned long long a = s.pre_tbits[g], b = a + s.my_tbits[g];
        unsigned long long lo, hi;
        own_units(L.tstream_off[g], a, b, lo, hi);
        if (first) lo = L.table_off[g];          // head, items and the stream's first bits
        if (last) hi = L.trestart_off[g];        // the stream's padding up to the restart offsets
        if (hi > lo) push_bytes(p, lo, hi);
        // restart offsets of the block's chunks (1024 / HUF_RESTART per chunk)
        const unsigned int e0 = (c0 - L.tchunk_prefix[g]) * (1024u / HUF_RESTART);
        unsigned int e1 = (c1 - L.tchunk_prefix[g]) * (1024u / HUF_RESTART);
        const unsigned int ne = (L.cells[g] + HUF_RESTART - 1) / HUF_RESTART;
        unsigned long long r1 = L.trestart_off[g] + 4ull * min(e1, ne);
        if (last) r1 = skml_align16(r1);
        push_bytes(p, L.trestart_off[g] + 4ull * e0, r1);
        (void)e1;
    }
}

// Block 0, after every block has written: the units of the table streams that hold a block border.
__device__ __noinline__ void huf_push_borders(const CP& p, Smem& s) {
    const Layout& L = s.lay;
    if (p.world <= 1 || L.overflow) return;
    const unsigned int total = L.tchunk_prefix[p.G];
    unsigned int per = (total + gridDim.x - 1) / gridDim.x;
    per = (per + 3u) & ~3u;
    const unsigned int b = threadIdx.x;
    if (b >= 1 && b < gridDim.x && (unsigned long long)per * b < total) {
        const unsigned int cs = per * b;
        int g = 0;
        while (g + 1 < p.G && cs >= L.tchunk_prefix[g + 1]) ++g;
        if (cs != L.tchunk_prefix[g]) {
            unsigned long long a = 0;
            for (unsigned int q = 0; q < b; ++q) a += get_halves(p.blk_tbits, g, q);
            const unsigned long long bit = 8ull * L.tstream_off[g] + a;
            if (bit & 127ull) {
                const unsigned long long off = 16ull * (bit / 128ull);
                const uint4 v = ld_cg_v4(reinterpret_cast<const uint4*>(p.payload + off));
                for (unsigned int r = 0; r < p.world; ++r)
                    if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + off), v);
            }
        }
    }
}

// Contiguous run of chunks of this block, a multiple of four (the chunks of one round) per block, and how
// many blocks have one.
__device__ __forceinline__ unsigned int chunk_run(const Layout& L, int G, unsigned int& my_begin, unsigned int& my_end) {
    const unsigned int total = L.chunk_prefix[G];
    unsigned int per = (total + gridDim.x - 1) / gridDim.x;
    per = (per + 3u) & ~3u;
    my_begin = min(total, per * blockIdx.x);
    my_end = min(total, my_begin + per);
    return per ? (total + per - 1) / per : 0u;
}

// S6 prelude: every group's delta bytes from all blocks' counts -> delta section offsets, total size.
template <bool WAIT>
__device__ bool layout_finish(const CP& p, Smem& s, unsigned int epoch, unsigned int nactive) {
    Layout& L = s.lay;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool ok = true;
    if (warp < p.G) {
        unsigned long long v;
        ok = sum_row<WAIT>(p, p.blk_bytes + warp * MAX_GRID, nactive, epoch, 0x51u, v);
        if (lane == 0) L.bytes_g[warp] = v;
    }
    if (!__syncthreads_and(ok)) return false;
    if (warp == 0) {
        unsigned long long size = 0, all;
        if (lane < p.G && L.n_g[lane]) size = skml_align16(8ull * ((L.bytes_g[lane] + 7) / 8));
        const unsigned long long o = warp_prefix(size, all);
        if (lane < p.G) L.delta_off[lane] = L.off_deltas + o;
        if (lane == 0) {
            L.total_bytes = L.off_deltas + all;
            if (L.total_bytes > (unsigned long long)p.slot_capacity) {
                L.overflow = 1;
                skml_set_status(p.status, SKML_CAPACITY, 0x36u);
            }
        }
    }
    __syncthreads();
    return true;
}

// Fill helpers run inside S1 (they do not depend on the summary). priv: the sketch is not expected to be inserted in
// p.tables; where it is after all, a second call fills the tables only.
__device__ void stage_prepare(const CP& p, long long n, bool priv, bool tables_only = false) {
    // working sketch cells start "empty"
    long long cells = (long long)p.rows * ((long long)(p.col_ratio * (double)n) + 2 + p.G) + 4 * p.G;
    if (cells > p.tables_cap - 4) cells = p.tables_cap - 4;
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    uint4* t4 = reinterpret_cast<uint4*>(p.tables);
    if (!priv)
        for (long long i = gid; i < (cells + 3) / 4; i += gsz) t4[i] = ones;
    if (tables_only) return;
    if (p.zero_slot) clear_slot(p, 0, gid, gsz);   // (two grid barriers lie before the first byte of the payload)
    if (p.key_encoder == SKML_KEYS_DELTA_ADAPTIVE || p.huffman) {
        // the bit streams are completed with atomic ORs where chunks meet: they start from zero
        long long bound = payload_bound(n, 0, p.q, p.G, p.rows, p.col_ratio);
        if (bound > p.slot_capacity) bound = p.slot_capacity;
        uint4 z = make_uint4(0, 0, 0, 0);
        uint4* z4 = reinterpret_cast<uint4*>(p.payload);
        if (!p.zero_slot)
            for (long long i = gid + SKML_HEADER_BYTES / 16; i < bound / 16; i += gsz) z4[i] = z;
        for (long long i = gid; i < SKML_MAX_GROUPS * 32; i += gsz) p.key_hist[i] = 0;
        for (long long i = gid; i < SKML_GPU_MAX_BINS + SKML_MAX_GROUPS; i += gsz) p.cell_hist[i] = 0;
    }
}

// Header, bucket values and group table, stored locally and into every peer's slot, by the block that calls it.
__device__ void write_header(const CP& p, Smem& s, long long n, int kind) {
    const Layout& L = s.lay;
    const QInfo& q = s.qi;
    const bool sparse = kind == SKML_KIND_SPARSE && !L.overflow;
    if (kind != SKML_KIND_EMPTY && (kind == SKML_KIND_DENSE || sparse)) {
        float* bv = reinterpret_cast<float*>(p.payload + SKML_HEADER_BYTES);
        const int padded = (int)(skml_align16(4ull * p.q) / 4);
        for (int b = threadIdx.x; b < padded; b += blockDim.x) bv[b] = b < q.bin_num ? bucket_value(s, b) : 0.f;
    }
    if (sparse && threadIdx.x >= 32 && threadIdx.x < 32 + p.G) {
        const int g = threadIdx.x - 32;
        const bool any = L.n_g[g] != 0;
        SkmlGroupEntry e;
        e.n = L.n_g[g];
        e.col_num = L.col[g];
        for (int i = 0; i < 8; ++i) e.hash_ids[i] = any ? p.hash_ids[g][i] : 0;
        e.table_off = any ? L.table_off[g] : 0;
        e.flag_off = any ? L.flag_off[g] : 0;
        e.n_flag_words = (unsigned int)((2ull * L.n_g[g] + 63) / 64);
        e.num_intervals = 4;
        e.delta_off = any ? L.delta_off[g] : 0;
        e.n_delta_words = (unsigned int)((L.bytes_g[g] + 7) / 8);
        e.flag_kind = 0;
        if (p.key_encoder == SKML_KEYS_DELTA_ADAPTIVE) {
            e.n_flag_words = (unsigned int)((L.flag_bits[g] + 63) / 64);
            e.n_delta_words = (unsigned int)((L.delta_bits[g] + 63) / 64);
            e.num_intervals = any ? L.num_iv[g] : 0;
            e.flag_kind = any ? L.flag_kind[g] : 0;
        }
        e.restart_off = any ? L.restart_off[g] : 0;
        *reinterpret_cast<SkmlGroupEntry*>(p.payload + L.off_gt + (unsigned long long)g * sizeof(SkmlGroupEntry)) = e;
    }
    if (threadIdx.x < 32) {   // the header is put together in shared memory by one warp
        const int lane = threadIdx.x;
        SkmlHeader& h = s.hdr;
        for (int i = lane; i < SKML_HEADER_BYTES / 4; i += 32) reinterpret_cast<unsigned int*>(&h)[i] = 0u;
        __syncwarp();
        if (lane < 4 && p.loss_partials) h.loss_partials[lane] = p.loss_partials[lane];
        if (lane == 0) {
            h.magic = SKML_MAGIC;
            h.version = SKML_VERSION;
            const unsigned int hk = (kind == SKML_KIND_SPARSE && L.overflow) ? (unsigned int)SKML_KIND_EMPTY : (unsigned int)kind;
            h.kind = hk;
            h.dtype = SKML_F32;
            h.step = p.step;
            h.rank = p.rank;
            h.world = p.world;
            h.dim = (unsigned long long)p.dim;
            h.seed = p.seed;
            h.total_bytes = SKML_HEADER_BYTES;
            if (hk != SKML_KIND_EMPTY) {
                h.nnz = (unsigned long long)n;
                h.bin_num = (unsigned int)q.bin_num;
                h.zero_idx = (unsigned int)q.zero_idx;
                h.cell_bits = (kind == SKML_KIND_SPARSE && p.huffman) ? 0u : (unsigned int)q.cell_bits;
                h.min_value = (double)q.minv;
                h.max_value = (double)q.maxv;
                h.off_bucket_values = SKML_HEADER_BYTES;
            }
            if (hk == SKML_KIND_SPARSE) {
                h.group_num = (unsigned int)p.G;
                h.row_num = (unsigned int)p.rows;
                h.col_ratio = p.col_ratio;
                h.key_encoder = (unsigned int)p.key_encoder;
                h.restart_interval = SKML_RESTART_INTERVAL;
                h.off_group_table = L.off_gt;
                h.off_key_flags = L.off_flags;
                h.off_restart = L.off_restart;
                h.off_tables = L.off_tables;
                h.off_key_deltas = L.off_deltas;
                h.total_bytes = L.total_bytes;
            } else if (hk == SKML_KIND_DENSE) {
                h.off_dense_codes = SKML_HEADER_BYTES + skml_align16(4ull * p.q);
                h.total_bytes = skml_align16(h.off_dense_codes + (unsigned long long)p.dim * (q.cell_bits / 8));
            }
        }
        __syncwarp();
        if (lane == 0) h.header_checksum = skml_header_checksum(&h);
        __syncwarp();
        if (lane < SKML_HEADER_BYTES / 16) reinterpret_cast<uint4*>(p.payload)[lane] = reinterpret_cast<const uint4*>(&h)[lane];
    }
    // this block wrote the head of the payload (header, bucket values, group table): it also stores it
    // into the peers' slots, so that no other block has to wait for it
    __syncthreads();
    if (p.world > 1) {
        unsigned long long head = SKML_HEADER_BYTES;
        if (sparse) head = L.off_flags;
        else if (kind == SKML_KIND_DENSE) head = SKML_HEADER_BYTES + skml_align16(4ull * p.q);
        const uint4* src = reinterpret_cast<const uint4*>(p.payload);
        for (unsigned long long i = threadIdx.x; i < head / 16; i += blockDim.x) {
            const uint4 v = ld_cg_v4(src + i);
            for (unsigned int r = 0; r < p.world; ++r)
                if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r]) + i, v);
        }
    }
}

// ---------------------------------------------------------------------------
// S6: narrow tables, store everything into the peers' slots, release the flags
// ---------------------------------------------------------------------------
__device__ void copy_range_to_peers(const CP& p, unsigned long long lo, unsigned long long hi) {
    if (p.world <= 1 || hi <= lo) return;
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long units = (long long)((hi - lo) / 16);
    const uint4* src = reinterpret_cast<const uint4*>(p.payload + lo);
    for (long long i = gid; i < units; i += gsz) {
        uint4 v = ld_cg_v4(src + i);
        for (unsigned int r = 0; r < p.world; ++r)
            if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + lo) + i, v);
    }
}

// The block barrier orders every thread's stores before thread 0's fence, and the fence before the count, so one
// thread fences for the block (1024 threads fencing at system scope took 7 us); peers' memory needs system scope.
// A checked call returns on the last block's word, before the kernel has ended: that word must carry the other blocks'
// stores (and statuses) too. Only a launch alone, without flag and word, leaves its readers to the end of the kernel; so does
// one whose only reader is behind it on its stream, and the block that writes the header sets the flag then (`header`): fence,
// count and flag took 3.7 us at the end of every step.
template <bool FUSED>
__device__ void finish_publish(const CP& p, unsigned int* set, bool header) {
    if (FUSED && p.world == 1 && !p.done_word && (p.decode_follows || !p.peer_flag[0])) {
        if (header && threadIdx.x == 0 && p.peer_flag[0]) *(volatile unsigned long long*)p.peer_flag[0] = p.step + 1;
        return;
    }
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (p.world > 1) __threadfence_system();
        else if (p.peer_flag[0] || p.done_word) __threadfence();
        unsigned int prev = atomicAdd(&p.ctrl[2], 1u);
        s_last = prev == gridDim.x - 1;
        if (s_last) {
            p.ctrl[2] = 0;
            if (!FUSED) set[CTRL_MIN] = set[CTRL_MAX] = 0;   // (a staged launch opens no set of its own)
            __threadfence();
            skml_store_done(p.done_word, p.done_seq, p.status);
        }
    }
    __syncthreads();
    // the last block to arrive raises the arrival flags, one thread per rank so that the releases (each
    // orders this GPU's earlier peer stores before its flag) run side by side instead of one after another
    if (s_last && threadIdx.x < p.world && p.peer_flag[threadIdx.x]) {
        __threadfence_system();
        st_release_sys(p.peer_flag[threadIdx.x], p.step + 1);
    }
}

// Sketch tables: 32-bit working cells -> 8/16-bit bucket codes, stored locally and into the peers' slots.
// `first`: the block that begins, the first one without keys to code where there is one (10,000 keys: 2.2 us less).
__device__ void narrow_tables(const CP& p, Smem& s, unsigned int first) {
    const Layout& L = s.lay;
    if (L.overflow) return;
    const int G = p.G, cb = s.qi.cell_bits, per = 16 / (cb / 8);  // cells per 16-byte unit
    const unsigned int turn = blockIdx.x >= first ? blockIdx.x - first : blockIdx.x + gridDim.x - first;
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)turn * blockDim.x + threadIdx.x;
    const long long units = (long long)L.unit_prefix[G];
    const unsigned int zero = (unsigned int)s.qi.zero_idx;
    auto code_of = [&](unsigned int cell) { return cell == SKML_EMPTY_CELL ? zero : cell; };
    for (long long u = gid; u < units; u += gsz) {
        int g = 0;
        while (g + 1 < G && (unsigned long long)u >= L.unit_prefix[g + 1]) ++g;
        const long long j = u - (long long)L.unit_prefix[g];
        const long long left = (long long)p.rows * L.col[g] - j * per;   // cells from this unit on
        // a group's working table starts at a multiple of four cells, so the unit is `per / 4` 16-byte loads
        const uint4* src = reinterpret_cast<const uint4*>(p.tables + L.tab32_off[g]) + j * (per / 4);
        unsigned int words[4] = {0, 0, 0, 0};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            if (4 * t >= per) break;
            uint4 c = make_uint4(0, 0, 0, 0);
            if (4 * t < left) c = ld_cg_v4(src + t);
            const unsigned int x0 = 4 * t < left ? code_of(c.x) & 0xFFFFu : 0u, x1 = 4 * t + 1 < left ? code_of(c.y) & 0xFFFFu : 0u;
            const unsigned int x2 = 4 * t + 2 < left ? code_of(c.z) & 0xFFFFu : 0u, x3 = 4 * t + 3 < left ? code_of(c.w) & 0xFFFFu : 0u;
            if (cb == 8) words[t] = (x0 & 0xFFu) | ((x1 & 0xFFu) << 8) | ((x2 & 0xFFu) << 16) | (x3 << 24);
            else if (t < 2) {
                words[2 * t] = x0 | (x1 << 16);
                words[2 * t + 1] = x2 | (x3 << 16);
            }
        }
        uint4 v = make_uint4(words[0], words[1], words[2], words[3]);
        const unsigned long long off = L.table_off[g] + 16ull * j;
        st_v4(reinterpret_cast<uint4*>(p.payload + off), v);
        for (unsigned int r = 0; r < p.world; ++r)
            if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + off), v);
    }
}

// The copies of the sketch's parts (stage_insert) -> bucket codes, stored locally and into the peers' slots.
__device__ void merge_copies(const CP& p, Smem& s) {
    const Layout& L = s.lay;
    if (L.overflow) return;
    const int G = p.G;
    for (unsigned int t = threadIdx.x; t < L.part_prefix[G]; t += SKML_BLOCK) {
        int g = 0;
        while (g + 1 < G && t >= L.part_prefix[g + 1]) ++g;
        const unsigned int per_part = (L.n_g[g] + 3u) / 4u;
        const unsigned long long w0 = L.work_prefix[g] + (unsigned long long)(t - L.part_prefix[g]) * per_part;
        const unsigned int b0 = (unsigned int)(w0 / L.work_per), b1 = (unsigned int)((w0 + per_part - 1) / L.work_per);
        s.priv_blocks[t] = make_uint2(b0, b1 - b0 + 1u);
    }
    __syncthreads();
    const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long units = (long long)L.unit_prefix[G];
    const unsigned int zero = (unsigned int)s.qi.zero_idx;
    for (long long u = gid; u < units; u += gsz) {
        int g = 0;
        while (g + 1 < G && (unsigned long long)u >= L.unit_prefix[g + 1]) ++g;
        const unsigned long long j = (unsigned long long)u - L.unit_prefix[g];
        const unsigned int col = L.col[g], parts = L.parts[g], plen = L.part_len[g];
        const unsigned long long c0 = 16ull * j, c1 = min(c0 + 16ull, (unsigned long long)p.rows * col);   // cells of this unit
        uint4 m = make_uint4(~0u, ~0u, ~0u, ~0u);
        for (unsigned long long c = c0; c < c1;) {   // the parts that have cells in it: one, two at a border
            const unsigned int row = (unsigned int)(c / col), in_row = (unsigned int)(c - (unsigned long long)row * col), part = in_row / plen;
            const unsigned int t = L.part_prefix[g] + row * parts + part;
            const unsigned long long first = (unsigned long long)row * col + (unsigned long long)part * plen;
            const uint2 blocks = s.priv_blocks[t];
            const unsigned char* src = reinterpret_cast<const unsigned char*>(p.tables) + (unsigned long long)(blocks.x + t) * L.copy_stride +
                                       16ull * (j - first / 16ull);
#pragma unroll 4
            for (unsigned int b = 0; b < blocks.y; ++b) {
                const uint4 v = ld_cg_v4(reinterpret_cast<const uint4*>(src + (unsigned long long)b * L.copy_stride));
                m.x = __vminu4(m.x, v.x);
                m.y = __vminu4(m.y, v.y);
                m.z = __vminu4(m.z, v.z);
                m.w = __vminu4(m.w, v.w);
            }
            c = min(first + plen, (unsigned long long)(row + 1) * col);
        }
        const unsigned int lo = g ? (unsigned int)s.qi.edges[g - 1] : 0u, left = (unsigned int)(c1 - c0);
        auto bucket = [&](unsigned int code, unsigned int i) {
            return i >= left ? 0u : (code == 0xFFu ? zero : (unsigned int)s.code_bin[lo + code]);
        };
        auto word = [&](unsigned int x, unsigned int i) {
            return bucket(x & 0xFFu, i) | (bucket((x >> 8) & 0xFFu, i + 1) << 8) | (bucket((x >> 16) & 0xFFu, i + 2) << 16) |
                   (bucket(x >> 24, i + 3) << 24);
        };
        const uint4 v = make_uint4(word(m.x, 0), word(m.y, 4), word(m.z, 8), word(m.w, 12));
        const unsigned long long off = L.table_off[g] + 16ull * j;
        st_v4(reinterpret_cast<uint4*>(p.payload + off), v);
        for (unsigned int r = 0; r < p.world; ++r)
            if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + off), v);
    }
    __syncthreads();
}

// Bytes [lo, hi) of the local payload -> the same bytes of every peer's slot, by this block alone:
// 16-byte stores for the aligned interior, byte stores for a ragged head or tail (two blocks that
// share a 16-byte unit each store only their own bytes of it).
__device__ __noinline__ void push_bytes(const CP& p, unsigned long long lo, unsigned long long hi) {
    if (p.world <= 1 || hi <= lo) return;
    const unsigned long long a0 = (lo + 15ull) & ~15ull, a1 = hi & ~15ull;
    if (a0 < a1) {
        const uint4* src = reinterpret_cast<const uint4*>(p.payload + a0);
        for (unsigned long long i = threadIdx.x; i < (a1 - a0) / 16; i += blockDim.x) {
            const uint4 v = ld_cg_v4(src + i);
            for (unsigned int r = 0; r < p.world; ++r)
                if (r != p.rank && p.peer_payload[r]) st_v4(reinterpret_cast<uint4*>(p.peer_payload[r] + a0) + i, v);
        }
    }
    const unsigned long long head_end = a0 < hi ? a0 : hi, tail_begin = a1 > head_end ? a1 : head_end;
    const unsigned long long ragged = (head_end - lo) + (hi - tail_begin);
    for (unsigned long long i = threadIdx.x; i < ragged; i += blockDim.x) {
        const unsigned long long a = i < head_end - lo ? lo + i : tail_begin + (i - (head_end - lo));
        const unsigned char v = __ldcg(p.payload + a);
        for (unsigned int r = 0; r < p.world; ++r)
            if (r != p.rank && p.peer_payload[r]) p.peer_payload[r][a] = v;
    }
}

// The flag bytes, restart points and delta bytes this block wrote for its chunks -> the peers' slots.
__device__ __noinline__ void push_own_chunks(const CP& p, Smem& s, unsigned int my_begin, unsigned int my_end) {
    const Layout& L = s.lay;
    if (p.world <= 1 || L.overflow || my_begin >= my_end) return;
    __syncthreads();  // this block's own stores are visible to all its threads
    for (int g = 0; g < p.G; ++g) {
        const unsigned int c0 = max(my_begin, L.chunk_prefix[g]), c1 = min(my_end, L.chunk_prefix[g + 1]);
        if (c0 >= c1) continue;
        const unsigned int ja = c0 - L.chunk_prefix[g], jb = c1 - L.chunk_prefix[g];
        const bool last = c1 == L.chunk_prefix[g + 1];
        const unsigned long long flag_bytes = skml_align16(8ull * ((2ull * L.n_g[g] + 63) / 64));
        const unsigned long long f1 = min(flag_bytes, 256ull * jb);
        push_bytes(p, L.flag_off[g] + 256ull * ja, L.flag_off[g] + (last ? flag_bytes : f1));
        push_bytes(p, L.restart_off[g] + 16ull * ja, L.restart_off[g] + 16ull * jb);
        unsigned long long d0 = s.pre_bytes[g], d1 = s.pre_bytes[g] + s.my_bytes[g];
        if (last) d1 = skml_align16(8ull * ((d1 + 7) / 8));  // the zero padding written with the last chunk
        push_bytes(p, L.delta_off[g] + d0, L.delta_off[g] + d1);
    }
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
#define STAGE_BARRIER(stage_id)                                                           \
    if (FUSED) {                                                                          \
        if (!skml_grid_barrier(set + CTRL_BAR, gridDim.x, p.status, p.budget, stage_id, passed)) return; \
        stage_stamp(p.ctrl, stage_id);                                                    \
    }

// Dense kind: one narrow bucket code per coordinate, written straight into the local
// payload and every peer's slot.
template <bool FUSED>
__device__ void dense_stages(const CP& p, Smem& s, unsigned int* set, unsigned int epoch, const float* __restrict__ vals, int stage) {
    unsigned int passed = 0;   // arrivals of the grid barriers so far
    const long long n = p.dim;
    const bool given = p.given_splits != nullptr;
    // sample form: the splits are in every block after S1; the extremes of the values (needed for the bucket
    // values in the header only) are collected by the code pass, and the header is written after it
    const bool sample = p.sample_splits != 0 && !given;
    if (FUSED || stage == 1) {
        if (sample) stage_sample_splits(p, s, vals, n);
        else if (!given) stage_summary(p, s, set, vals, n);
    }
    if (!sample) {
        STAGE_BARRIER(1)
        if ((FUSED || stage == 2) && !given) stage_query(p, s, n);
        STAGE_BARRIER(2)
    }
    if (FUSED || stage == 3) {
        load_quantizer(p, s, set, FUSED && sample, !sample);
        if (s.qi.bin_num > SKML_GPU_MAX_BINS) {
            if (threadIdx.x == 0) skml_set_status(p.status, SKML_BAD_INPUT, 0x33u);
            return;
        }
        if (threadIdx.x == 0) s.lay.overflow = 0;
        __syncthreads();
        const int cb = s.qi.cell_bits;
        const unsigned long long off_codes = SKML_HEADER_BYTES + skml_align16(4ull * p.q);
        const unsigned long long total = skml_align16(off_codes + (unsigned long long)n * (cb / 8));
        if (total > (unsigned long long)p.slot_capacity) {
            if (threadIdx.x == 0) skml_set_status(p.status, SKML_CAPACITY, 0x34u);
            return;
        }
        if (!sample && blockIdx.x == 0) write_header(p, s, n, SKML_KIND_DENSE);
        const long long gsz = (long long)gridDim.x * blockDim.x, gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        // What lies before the end of the codes is written whole (header and bucket values by block 0, the code section
        // with its padding below) and not cleared: with sampled splits no grid barrier lies in between, so a late block
        // would clear codes that another one has written.
        if (p.zero_slot) clear_slot(p, (long long)total, gid, gsz);
        unsigned int kmin = 0xFFFFFFFFu, kmax = 0u;
        // Four adjacent values per thread: one vector load, four searches side by side, one store. (Sixteen values a
        // thread, searched one after another, left two thirds of the threads idle at 1M coordinates: 25 us.)
        const long long units = (long long)((total - off_codes) / (cb / 2));   // with the section's zero padding
        const int top = build_search(s);
        __syncthreads();
        const bool vec = (reinterpret_cast<uintptr_t>(vals) & 15) == 0;
        for (long long u = gid; u < units; u += gsz) {
            const long long i0 = 4 * u;
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (vec && i0 + 4 <= n) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(vals) + u);
                x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
            } else {
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (i0 + t < n) x[t] = vals[i0 + t];
            }
            int code[4];
            upper_bounds_f(s.ss.a, top, x, code);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (i0 + t < n) {
                    const unsigned int k = f2ord(x[t]);
                    kmin = min(kmin, k);
                    kmax = max(kmax, k);
                } else {
                    code[t] = 0;
                }
            }
            auto put = [&](unsigned char* at) {
                if (cb == 8)
                    reinterpret_cast<unsigned int*>(at)[u] =
                        (unsigned int)code[0] | ((unsigned int)code[1] << 8) | ((unsigned int)code[2] << 16) | ((unsigned int)code[3] << 24);
                else
                    reinterpret_cast<uint2*>(at)[u] =
                        make_uint2((unsigned int)code[0] | ((unsigned int)code[1] << 16), (unsigned int)code[2] | ((unsigned int)code[3] << 16));
            };
            put(p.payload + off_codes);
            for (unsigned int r = 0; r < p.world; ++r)
                if (r != p.rank && p.peer_payload[r]) put(p.peer_payload[r] + off_codes);
        }
        if (sample) {   // one pair of atomics per warp
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                kmin = min(kmin, __shfl_xor_sync(0xFFFFFFFFu, kmin, o));
                kmax = max(kmax, __shfl_xor_sync(0xFFFFFFFFu, kmax, o));
            }
            if ((threadIdx.x & 31) == 0 && kmin <= kmax) {
                atomicMax(&set[CTRL_MIN], ~kmin);
                atomicMax(&set[CTRL_MAX], kmax);
            }
        }
    }
    STAGE_BARRIER(3)
    if (FUSED) ctrl_advance(p.ctrl, epoch);
    if (FUSED || stage == 4) {
        if (sample) {
            if (!FUSED) load_quantizer(p, s, set);   // staged launches: the extremes are complete now
            else if (threadIdx.x < 2) set_extreme(p, s, threadIdx.x == 0, threadIdx.x == 0 ? ~__ldcg(set + CTRL_MIN) : __ldcg(set + CTRL_MAX));
            __syncthreads();
            if (!FUSED) {
                if (threadIdx.x == 0) s.lay.overflow = 0;
                __syncthreads();
            }
            if (blockIdx.x == 0) write_header(p, s, n, SKML_KIND_DENSE);
        }
        finish_publish<FUSED>(p, set, blockIdx.x == 0);
    }
}

// As a function of its own, for the launches that rarely need it.
__device__ __noinline__ void dense_stages_apart(const CP& p, Smem& s, unsigned int* set, unsigned int epoch, const float* __restrict__ vals) {
    dense_stages<true>(p, s, set, epoch, vals, -1);
}

// STAGE < 0: all stages in one cooperative launch; otherwise only that stage.
// ADAPTIVE / HUFFMAN: the key encoder and the table coder are compile-time choices, so that the default
// path (delta_binary keys, plain tables) carries none of the other coders' registers. PRIV: launches that may have enough
// keys for the insert in shared memory (its code costs the others 2 us). DENSE: launches that may be of the dense kind.
// A launch runs most of its code once, so what it does not need should not lie between what it does: fetching instructions
// is a good part of a short stage, and most of it where the step's other kernels have put them out of L2. Without the dense
// kind's stages, and with the sketch form of S1 and S2 and the stores to peers out of line: 430,000 keys in a step 49.3 -> 43.2 us,
// 2.27M 100.3 -> 93.3, 26,000 29.1 -> 28.5; a dense launch of 1M coordinates 27.9 -> 22.8. (The stages of the insert in shared
// memory, the sample, the quantizer or the layout out of line too: 2.27M keys 100 to 102, 10M 323 -> 343 to 346. The dense
// stages as a function of their own: 27.9 -> 34, but the insert in shared memory compiles the better for it, 2.27M keys 93.3 -> 92.1
// and 10M 323 -> 313, so launches of PRIV have them so.)
template <bool FUSED, bool ADAPTIVE, bool HUFFMAN, bool PRIV, bool DENSE>
__global__ void __launch_bounds__(SKML_BLOCK, 1) compress_sparse_kernel(const __grid_constant__ CP p, int stage) {
    skml_after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    unsigned int passed = 0;   // arrivals of the grid barriers so far
    long long n = p.n_value, kind = p.kind_value;
    if (p.meta) {
        n = p.meta[0];
        kind = p.meta[1];
    }
    const unsigned int epoch = ctrl_open<FUSED>(p.ctrl);   // names this launch's publications
    unsigned int* const set = ctrl_set(p.ctrl, epoch);
    if (kind == SKML_KIND_DENSE) {  // un-fused launches leave it to the dense kernel's stages
        if (FUSED && p.dense_vals) {
            if (PRIV) dense_stages_apart(p, s, set, epoch, p.dense_vals);
            else if (DENSE) dense_stages<FUSED>(p, s, set, epoch, p.dense_vals, stage);
        }
        return;
    }
    if (n > p.n_max) {
        if (threadIdx.x == 0) skml_set_status(p.status, SKML_CAPACITY, 0x31u);
        n = 0;
    }
    if (n <= 0) {  // empty gradient: header-only payload
        if (FUSED || stage == 8) {
            if (threadIdx.x == 0) {
                s.lay.overflow = 0;
                s.qi.bin_num = 0;
            }
            __syncthreads();
            if (blockIdx.x == 0) {
                if (p.zero_slot) {   // by this block alone, before its own header
                    clear_slot(p, 0, threadIdx.x, blockDim.x);
                    __syncthreads();
                }
                write_header(p, s, 0, SKML_KIND_EMPTY);   // locally and into the peers' slots
            }
            finish_publish<FUSED>(p, set, blockIdx.x == 0);
        }
        return;
    }
    const bool given = p.given_splits != nullptr;
    if (FUSED) stage_stamp(p.ctrl, 0);
    // sample form of the split search: S1 ends with the splits in every block, S2 and two grid barriers drop out
    const bool sample = p.sample_splits != 0 && !given;
    // this lane's first two elements: their values are wanted after S1, their keys after S3, the loads start here
    float first_val[2] = {0.f, 0.f};
    int first_key[2] = {0, 0}, first_bin[2] = {0, 0};
    if (FUSED || stage == 3) {
        const long long sub = vslice_size(n), lo = sub * ((long long)blockIdx.x * SKML_WARPS + (threadIdx.x >> 5));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long long k = 32 * u + (threadIdx.x & 31);
            if (k < sub && lo + k < n) {
                first_val[u] = p.vals[lo + k];
                if (FUSED) first_key[u] = p.keys[lo + k];
            }
        }
    }
    bool priv = PRIV && priv_pays(p.priv_least, (float)n, priv_passes((float)n, p.priv_parts), 1.f, 1.f);   // insert in shared memory
    if (FUSED || stage == 1) {
        stage_prepare(p, n, priv);
        stage_stamp(p.ctrl, 8);
        if (sample) stage_sample_splits(p, s, p.vals, n);
        else if (!given) stage_summary(p, s, set, p.vals, n);
        stage_stamp(p.ctrl, 9);
    }
    if (sample) {
        if (FUSED) {
            stage_stamp(p.ctrl, 1);
            stage_stamp(p.ctrl, 2);
        }
    } else {
        STAGE_BARRIER(1)
        if ((FUSED || stage == 2) && !given) stage_query(p, s, n);
        STAGE_BARRIER(2)
    }
    if (FUSED || stage == 3) {
        load_quantizer(p, s, set, FUSED && sample, !sample);
        if (s.qi.bin_num > SKML_GPU_MAX_BINS) {
            if (threadIdx.x == 0) skml_set_status(p.status, SKML_BAD_INPUT, 0x32u);
            return;
        }
        stage_count<FUSED, PRIV>(p, s, set, epoch, n, sample, first_val, first_bin);
    }
    if (FUSED || stage == 4) {
        if (!FUSED) load_quantizer(p, s, set);
        if (!layout_from_counts<FUSED>(p, s, epoch, FUSED && sample)) return;
        if (FUSED) {
            ctrl_advance(p.ctrl, epoch);
            stage_stamp(p.ctrl, 3);
        }
        if (priv) {
            priv_layout(p, s);
            priv = s.lay.priv != 0;
            if (!priv) {   // the same in every block
                stage_prepare(p, n, false, true);
                if (!skml_grid_barrier(set + CTRL_BAR, gridDim.x, p.status, p.budget, 0x14u, passed)) return;
            }
        }
        if (priv) stage_partition(p, s, n);
        else stage_scatter<FUSED>(p, s, n, first_key, first_bin);
    }
    STAGE_BARRIER(4)
    if (priv) {
        stage_insert(p, s);
        stage_stamp(p.ctrl, 7);
    }
    // S5: key code and publication. In one cooperative launch a block waits only for the counts of the
    // blocks before it (they are resident, and never wait for a later block), and the last block for all of
    // them before it writes the header (it has the fewest chunks, none where there are fewer than blocks); after an
    // insert in shared memory every block waits for all of them, behind its own keys, before it merges the copies;
    // staged launches split the stage at those points. The delta_adaptive
    // code needs the groups' complete histograms of delta widths first: one more grid barrier.
    unsigned int my_begin = 0, my_end = 0, t_begin = 0, t_end = 0, nactive = 0, turn = 0;
    constexpr bool adaptive = ADAPTIVE, huffman = HUFFMAN;
    if (FUSED || stage >= 5) {
        if (!FUSED) {
            load_quantizer(p, s, set);
            layout_from_counts<FUSED>(p, s, epoch, false);
        }
        nactive = chunk_run(s.lay, p.G, my_begin, my_end);
        if (huffman) {
            huf_ranges(p, s);
            // the tables' chunks begin behind the blocks that have keys to code
            turn = blockIdx.x >= nactive ? blockIdx.x - nactive : blockIdx.x + gridDim.x - nactive;
            tchunk_run(s.lay, p.G, turn, t_begin, t_end);
        }
    }
    if (FUSED || stage == 5) {
        if (huffman) {
            if (!s.lay.overflow) huf_histogram(p, s, t_begin, t_end);
        } else if (adaptive && !priv) {
            narrow_tables(p, s, nactive);   // the tables are complete since S4
        }
        if (adaptive && !s.lay.overflow) apack_histogram(p, s, my_begin, my_end);
    }
    if (FUSED && (adaptive || huffman)) {
        if (!skml_grid_barrier(set + CTRL_BAR, gridDim.x, p.status, p.budget, 0x15u, passed)) return;
    }
    if (FUSED || stage >= 6) {
        // code tables and the layout behind the tables (every block; staged launches repeat it per stage)
        if (huffman) huf_build<ADAPTIVE>(p, s);
        else if (adaptive) apack_choose(p, s);
    }
    ChunkWork cw;
    unsigned int boff = 0, btotal = 0;
    if (FUSED || stage == 6) {
        if (adaptive) apack_measure<FUSED>(p, s, epoch, my_begin, my_end);
        else if (my_begin < my_end) pack_measure<FUSED>(p, s, epoch, my_begin, my_end, cw, boff, btotal);
        if (huffman) huf_measure<FUSED>(p, s, epoch, turn, t_begin, t_end);
    }
    if (FUSED && priv) {   // (counts carry the number themselves, the copies of an insert in shared memory do not)
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            st_relaxed_gpu(&p.blk_flag[blockIdx.x], epoch);
        }
    }
    if (!huffman && !adaptive && !priv && (FUSED || stage == 6)) narrow_tables(p, s, nactive);   // while the publications travel
    const bool borders = (adaptive || huffman) && p.world > 1;  // stream words shared by two blocks are sent by the last block at the end
    if (FUSED || stage == 7) {
        if (!FUSED) {  // the block's own counts again (shared memory does not survive a launch)
            if (threadIdx.x < SKML_MAX_GROUPS) {
                s.my_bytes[threadIdx.x] = (unsigned int)p.blk_bytes[threadIdx.x * MAX_GRID + blockIdx.x];
                s.my_tbits[threadIdx.x] = get_halves(p.blk_tbits, threadIdx.x, turn);
            }
            if (threadIdx.x < 2 * SKML_MAX_GROUPS) s.my_bits[threadIdx.x] = get_halves(p.blk_bits, threadIdx.x, blockIdx.x);
            __syncthreads();
        }
        if (adaptive) {
            apack_prefix<FUSED>(p, s, epoch);
            apack_write(p, s, my_begin, my_end);
            if (p.world > 1) apush_own_chunks(p, s, my_begin, my_end);
        } else if (my_begin < my_end) {
            pack_prefix<FUSED>(p, s, epoch);
            pack_write(p, s, my_begin, my_end, FUSED && my_end - my_begin <= 4, cw, boff, btotal);
            if (p.world > 1) push_own_chunks(p, s, my_begin, my_end);
        }
        if (huffman) {
            huf_prefix<FUSED>(p, s, epoch, turn);
            huf_write(p, s, t_begin, t_end);
            if (p.world > 1) huf_push_own(p, s, t_begin, t_end);
        }
        if (priv) {   // every block has made its copies before it published its counts
            if (!wait_published(p, p.blk_flag, gridDim.x, epoch, 0x54u)) return;
            merge_copies(p, s);
        }
        if (FUSED && borders) {
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                st_relaxed_gpu(&p.blk_done[blockIdx.x], epoch);
            }
        }
        if (FUSED) stage_stamp(p.ctrl, 5);
    }
    if (FUSED || stage == 8) {
        if (blockIdx.x == gridDim.x - 1) {
            if (FUSED && borders && !wait_published(p, p.blk_done, gridDim.x, epoch, 0x51u)) return;
            if (adaptive && borders) apush_borders(p, s);
            if (!adaptive && !layout_finish<FUSED>(p, s, epoch, nactive)) return;
            if (huffman && borders) huf_push_borders(p, s);
            write_header(p, s, n, SKML_KIND_SPARSE);
        }
        finish_publish<FUSED>(p, set, blockIdx.x == gridDim.x - 1);
        if (FUSED) stage_stamp(p.ctrl, 6);
    }
}

template <bool FUSED>
__global__ void __launch_bounds__(SKML_BLOCK, 1) compress_dense_kernel(const __grid_constant__ CP p, int stage) {
    skml_after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if ((p.meta ? p.meta[1] : p.kind_value) != SKML_KIND_DENSE) return;
    const unsigned int epoch = ctrl_open<FUSED>(p.ctrl);
    dense_stages<FUSED>(p, *reinterpret_cast<Smem*>(smem_raw), ctrl_set(p.ctrl, epoch), epoch, p.vals, stage);
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static int device_sms() {
    static int cached = 0;
    if (cached == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cached = sms > 0 ? sms : 148;
    }
    return cached;
}

static int fill_params(const SkmlCompressArgs* a, CP& p, int& grid) {
    if (!a || (!a->meta && (a->kind_value < 0 || a->kind_value > 2 || a->n_value < 0)) || !a->payload || !a->workspace || !a->status) return (int)cudaErrorInvalidValue;
    if (a->bin_num < 2 || a->bin_num > SKML_GPU_MAX_BINS) return (int)cudaErrorInvalidValue;
    if (a->group_num < 1 || a->group_num > SKML_MAX_GROUPS) return (int)cudaErrorInvalidValue;
    if (a->row_num < 1 || a->row_num > SKML_MAX_ROWS) return (int)cudaErrorInvalidValue;
    if (a->world < 1 || a->world > SKML_MAX_PEERS || a->rank < 0 || a->rank >= a->world) return (int)cudaErrorInvalidValue;
    if (a->n_max >= (1ll << 31) || a->dim >= (1ll << 31)) return (int)cudaErrorInvalidValue;
    if (a->key_encoder != SKML_KEYS_DELTA_BINARY && a->key_encoder != SKML_KEYS_DELTA_ADAPTIVE) return (int)cudaErrorInvalidValue;
    grid = a->grid > 0 ? (int)a->grid : device_sms();
    if (grid > MAX_GRID) grid = MAX_GRID;
    bool priv_room = priv_sizes(a->n_max, a->bin_num, a->row_num, a->group_num, a->col_ratio);
    WsLayout L = ws_layout(a->n_max, a->bin_num, a->group_num, a->row_num, a->col_ratio, grid, priv_room);
    if (L.total > a->workspace_bytes && priv_room) {   // (a workspace of the least size)
        priv_room = false;
        L = ws_layout(a->n_max, a->bin_num, a->group_num, a->row_num, a->col_ratio, grid, false);
    }
    if (L.total > a->workspace_bytes) return (int)cudaErrorInvalidValue;
    p.keys = a->keys;
    p.vals = a->vals;
    p.meta = a->meta;
    p.n_max = a->n_max;
    p.dim = a->dim;
    p.q = (int)a->bin_num;
    p.G = (int)a->group_num;
    p.rows = (int)a->row_num;
    p.col_ratio = a->col_ratio;
    p.seed = a->seed;
    p.step = a->step;
    p.rank = (unsigned int)a->rank;
    p.world = (unsigned int)a->world;
    p.loss_partials = a->loss_partials;
    p.payload = a->payload;
    p.slot_capacity = a->slot_capacity;
    for (int i = 0; i < SKML_MAX_PEERS; ++i) {
        p.peer_payload[i] = a->peer_payload[i];
        p.peer_flag[i] = a->peer_flag[i];
    }
    unsigned char* ws = a->workspace;
    p.ctrl = reinterpret_cast<unsigned int*>(ws + L.ctrl);
    p.run_vals = reinterpret_cast<unsigned int*>(ws + L.run_vals);
    p.run_cnt = reinterpret_cast<unsigned int*>(ws + L.run_cnt);
    p.run_w = reinterpret_cast<unsigned long long*>(ws + L.run_w);
    p.splits_raw = reinterpret_cast<unsigned int*>(ws + L.splits_raw);
    p.warp_cnt = reinterpret_cast<unsigned int*>(ws + L.warp_cnt);
    p.blk_cnt = reinterpret_cast<unsigned long long*>(ws + L.blk_cnt);
    p.blk_bytes = reinterpret_cast<unsigned long long*>(ws + L.blk_bytes);
    p.blk_flag = reinterpret_cast<unsigned int*>(ws + L.blk_flag);
    p.chunk_part = reinterpret_cast<unsigned short*>(ws + L.chunk_part);
    p.chunk_off = reinterpret_cast<unsigned int*>(ws + L.chunk_off);
    p.blk_bits = reinterpret_cast<unsigned long long*>(ws + L.blk_bits);
    p.blk_done = reinterpret_cast<unsigned int*>(ws + L.blk_done);
    p.key_hist = reinterpret_cast<unsigned int*>(ws + L.key_hist);
    p.key_encoder = (int)a->key_encoder;
    p.huffman = a->cell_bits == 0 ? 1 : 0;
    p.sample_splits = a->quantile_summary == 1 ? 0 : 1;
    p.cell_hist = reinterpret_cast<unsigned int*>(ws + L.cell_hist);
    p.blk_tbits = reinterpret_cast<unsigned long long*>(ws + L.blk_tbits);
    p.tchunk_off = reinterpret_cast<unsigned int*>(ws + L.tchunk_off);
    p.gkeys = reinterpret_cast<int*>(ws + L.gkeys);
    p.bins = reinterpret_cast<unsigned short*>(ws + L.bins);
    p.tables = reinterpret_cast<unsigned int*>(ws + L.tables);
    p.tables_cap = L.tables_cap;
    p.gcodes = ws + L.gcodes;
    p.copies_cap = L.copies_cap;
    p.status = a->status;
    p.budget = a->budget_cycles > 0 ? a->budget_cycles : 2000000000ll;
    p.given_splits = a->given_splits;
    p.n_given = (int)a->n_given;
    p.given_min = (float)a->given_min;
    p.given_max = (float)a->given_max;
    p.dense_vals = a->dense_vals;
    p.n_value = a->n_value;
    p.kind_value = (int)a->kind_value;
    p.zero_slot = a->zero_slot != 0;
    p.decode_follows = a->decode_follows != 0;
    p.done_word = a->done_word;
    p.done_seq = a->done_seq;
    // draws that depend on the launch's parameters only are made here, once, instead of by every block
    p.sample_rand = skml_rand(p.seed, p.step, p.rank, 0x7300u);
    p.mixers = p.rows <= 3;
    for (int g = 0; g < p.G; ++g) {
        skml_pick_hashes(p.seed, p.step, p.rank, (unsigned int)g, p.rows, p.hash_ids[g]);
        for (int r = 0; r < p.rows && p.mixers; ++r) p.mixers = p.hash_ids[g][r] < 3;
    }
    // codes of a byte, 255 meaning "no key": at most 255 buckets in a group (of 256 buckets, from three groups on a group has
    // at most 171)
    const int bins = a->given_splits ? (int)a->n_given + 1 : p.q;
    // A launch that could insert in shared memory but has too few keys for it is 3 to 4.6 us slower than one of the plain
    // kernel (247,000 keys 45.1 -> 48.3, 426,000 54.7 -> 59.3, 722,000 68.8 -> 72.2). Where the number is on the device only
    // (gradients that were scattered and compacted: one key to three to nine entries where columns are frequent and rare, up
    // to one each where they are alike), n_max says little: 4M keys of 6M alike 149 -> 139, but 247,000 to 722,000 of 1.1M to
    // 4.5M keys the above.
    const long long enough = a->meta && a->n_bound <= 0 ? PRIV_MIN_ROOM : 0;
    const long long n_known = !a->meta ? a->n_value : (a->n_bound > 0 && a->n_bound < a->n_max ? a->n_bound : a->n_max);
    p.priv = priv_room && p.mixers && !p.huffman && n_known >= enough && n_known >= PRIV_MIN_KEYS && (bins <= 255 || (bins == 256 && p.G >= 3));
    if (p.priv) {
        priv_thresholds(p.rows, p.G, p.col_ratio, p.priv_least);
        p.priv_parts = (float)(p.col_ratio / p.G / (PRIV_BYTES - 16));
        p.priv = priv_pays(p.priv_least, (float)n_known, priv_passes((float)n_known, p.priv_parts), 1.f, 1.f);
    }
    return 0;
}

// Byte offset, inside the workspace, of the q - 1 split points the last launch queried from its
// summary (order-preserving 32-bit images of the floats, before duplicates are dropped). Debug
// tooling reads them to recompute a payload on the CPU from the same splits.
extern "C" long long skml_compress_splits_offset(long long n_max, long long bin_num, long long group_num,
                                                 long long row_num, double col_ratio, long long grid) {
    long long g = grid > 0 ? grid : device_sms();
    if (g > MAX_GRID) g = MAX_GRID;
    return ws_layout(n_max, bin_num, group_num, row_num, col_ratio, g, false).splits_raw;   // (in front of all that differs)
}

// Function attributes and the co-residency limit are looked up once per kernel (one process
// drives one GPU), so a steady-state launch makes a single runtime call.
static int g_last_cluster = 0;   // blocks per cluster of the most recent compress launch (0: none yet)

struct LaunchCache {
    bool ready = false;
    int max_grid = 0;
    int cluster = 1;   // blocks per thread-block cluster (2 where that many clusters fit the device at once)
};

// One launch through the extensible API: cooperative when `coop`, in clusters of `cluster` blocks.
template <class K>
static cudaError_t launch_ex(K kernel, int grid, int cluster, bool coop, const CP& p, int stage, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(SKML_BLOCK);
    cfg.dynamicSmemBytes = sizeof(Smem);
    cfg.stream = stream;
    cudaLaunchAttribute attrs[3];
    unsigned int na = 0;
    if (coop) {
        attrs[na].id = cudaLaunchAttributeCooperative;
        attrs[na].val.cooperative = 1;
        ++na;
    }
    if (cluster > 1) {
        attrs[na].id = cudaLaunchAttributeClusterDimension;
        attrs[na].val.clusterDim.x = (unsigned int)cluster;
        attrs[na].val.clusterDim.y = 1;
        attrs[na].val.clusterDim.z = 1;
        ++na;
    }
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
    cfg.attrs = attrs;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kernel, p, stage);
}

template <class K>
static int launch_stages(K fused_kernel, K staged_kernel, LaunchCache& cache, CP& p, int grid, bool fused, int nstages,
                         cudaStream_t stream) {
    cudaError_t e;
    if (!cache.ready) {
        e = cudaFuncSetAttribute(fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
        if (e != cudaSuccess) return (int)e;
        e = cudaFuncSetAttribute(staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
        if (e != cudaSuccess) return (int)e;
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_kernel, SKML_BLOCK, sizeof(Smem));
        if (per_sm < 1) return (int)cudaErrorLaunchOutOfResources;
        cache.max_grid = per_sm * device_sms();
        // pairs of blocks as clusters when the whole grid still fits the device at once that way
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cache.max_grid & ~1);
        cfg.blockDim = dim3(SKML_BLOCK);
        cfg.dynamicSmemBytes = sizeof(Smem);
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        const char* knob = getenv("SKML_COMPRESS_CLUSTER");   // "1": plain blocks, no clusters
        if (knob && knob[0] == '1' && knob[1] == 0) {
            cache.cluster = 1;
        } else if (cudaOccupancyMaxActiveClusters(&nclusters, fused_kernel, &cfg) == cudaSuccess && 2 * nclusters >= (cache.max_grid & ~1) &&
            cache.max_grid >= 2)
            cache.cluster = 2;
        else
            cudaGetLastError();  // a refused query is not an error of the caller
        cache.ready = true;
    }
    if (grid > cache.max_grid) grid = cache.max_grid;
    int cluster = cache.cluster;
    if (grid < 2 * cluster) cluster = 1;   // tiny grids (tests) keep plain blocks
    if (cluster > 1) grid -= grid % cluster;
    if (fused) {
        e = launch_ex(fused_kernel, grid, cluster, true, p, -1, stream);
        if (e != cudaSuccess && cluster > 1) {
            // the device refuses cooperative clusters of this shape: plain blocks from now on
            cudaGetLastError();
            cache.cluster = cluster = 1;
            e = launch_ex(fused_kernel, grid, 1, true, p, -1, stream);
        }
        g_last_cluster = cluster;
        return (int)e;
    }
    g_last_cluster = cluster;
    for (int st = 1; st <= nstages; ++st) {
        e = launch_ex(staged_kernel, grid, st == 1 ? cluster : 1, false, p, st, stream);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

// Blocks per thread-block cluster of the most recent compress launch of this process (2 where the device
// takes the whole grid as cooperative clusters of two, 1 for plain blocks, 0 before the first launch).
extern "C" int skml_compress_cluster_size() { return g_last_cluster; }

extern "C" int skml_compress_sparse(const SkmlCompressArgs* a, void* stream) {
    CP p;
    int grid = 0;
    int rc = fill_params(a, p, grid);
    if (rc) return rc;
    static LaunchCache cache[7];
    const bool adaptive = p.key_encoder == SKML_KEYS_DELTA_ADAPTIVE, huffman = p.huffman != 0;
    const bool fused = a->fused != 0, priv = fused && !huffman && p.priv, dense = p.dense_vals != nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    auto go = [&](auto kernel, auto staged, int which) { return launch_stages(kernel, staged, cache[which], p, grid, fused, 8, st); };
    if (adaptive && huffman) return go(compress_sparse_kernel<true, true, true, false, true>, compress_sparse_kernel<false, true, true, false, false>, 0);
    if (huffman) return go(compress_sparse_kernel<true, false, true, false, true>, compress_sparse_kernel<false, false, true, false, false>, 1);
    if (adaptive && priv) return go(compress_sparse_kernel<true, true, false, true, false>, compress_sparse_kernel<false, true, false, false, false>, 2);
    if (adaptive) return go(compress_sparse_kernel<true, true, false, false, true>, compress_sparse_kernel<false, true, false, false, false>, 3);
    const auto plain = compress_sparse_kernel<false, false, false, false, false>;
    if (priv) return go(compress_sparse_kernel<true, false, false, true, false>, plain, 4);
    return dense ? go(compress_sparse_kernel<true, false, false, false, true>, plain, 5) : go(compress_sparse_kernel<true, false, false, false, false>, plain, 6);
}

extern "C" int skml_compress_dense(const SkmlCompressArgs* a, void* stream) {
    CP p;
    int grid = 0;
    int rc = fill_params(a, p, grid);
    if (rc) return rc;
    static LaunchCache cache;
    return launch_stages(compress_dense_kernel<true>, compress_dense_kernel<false>, cache, p, grid, a->fused != 0, 4,
                         (cudaStream_t)stream);
}

extern "C" int skml_compress_checked(SkmlCompressArgs* a, unsigned int* status_out, void* stream) {
    if (!a || !a->done_word || !a->fused || !status_out) return (int)cudaErrorInvalidValue;
    a->done_seq = ((*a->done_word >> 32) + 1) & 0xFFFFFFFFull;
    const int rc = skml_compress_sparse(a, stream);
    if (rc) return rc;
    return skml_wait_done(a->done_word, a->done_seq, a->status, status_out, (cudaStream_t)stream);
}
