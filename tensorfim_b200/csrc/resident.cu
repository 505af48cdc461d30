// RESIDENT engine: the batched search with its state on the device.
//
// Same search and pruning as mine_batched (mine.cu) -- families of children counted as
// masked Gram blocks, candidate restriction, equal-support pruning, head-union-tail
// lookahead with the tail-pair filter or the learned proposal, dynamic tail order, root
// filter -- but the family records, the DFS stack, the lookahead queue, the mask-slot
// free list and the MFI output live in device memory, and two kernels drive it:
//   k_res_pack    (one block) pops families from the top of the device stack into a wave:
//                 count-job descriptors, counted rows, tiles and output offsets;
//   k_res_expand  (one warp per counted row) turns a counted row into the child's MFI
//                 test, equal-support pruning, tail (sorted by support in the warp),
//                 child mask, lookahead decision (tail-pair filter, or the proposal MLP
//                 evaluated in the warp) and pushes the child onto the stack.
// Between them the counting kernels of count_lop3.cu / count_b1.cu run on the wave.  The
// host reads one small status record per wave (to size the launches and grow pools) and
// copies the MFIs back once at the end.
#include <cub/cub.cuh>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <numeric>

#include "search_error.h"
#include "tfim_internal.h"

namespace tfim {
namespace {

struct alignas(16) DFam {
    int32_t slot, item;        // base mask = masks[slot] & B[item] (either optional)
    int32_t head_off, head_len;
    int32_t F_off, nF, nT;     // F list in the item pool, tail = its first nT entries
    int32_t sup;
    int32_t next_row;          // rows handed to waves
    int32_t rows_done;         // rows expanded
    int32_t state;             // 0 ready, 1 waiting on its lookahead, 2 finished
    int32_t top;               // 1: the family of the empty prefix
    int32_t W, n;              // its transactions: words per bitmap row, and their number
    int32_t pad[2];
};

struct DLook {
    int32_t fam, slot, log, pad;
};

// A prefix mask to build after an expand: masks[dst] = (slot >= 0 ? masks[slot] : ~0) &
// (item >= 0 ? B[item] : ~0) & (t >= 0 ? B[t] : ~0) & AND of B[items[off + q]], q < n, over W words.
struct MaskJob {
    int32_t dst, slot, item, t, off, n, W, pad;
};

// A family to project (see "projection" below): its F list's rows compressed to the
// transactions of its prefix, `sup` of them, become the rows row0 .. row0 + nF of the row table,
// each of Wp words, from word `woff` of the pool on.
struct PJob {
    int32_t fam, item, F_off, nF, Wp, row0, sup, pad;
    int64_t woff;
};

enum { kJobFam = 0, kJobLook = 1 };
struct DJob {
    int32_t fam, kind, r0, nr, slot, log;
    int32_t cls, sl3;          // tile group (kGrp*, or kGrps: the projected counter's); word slices
    // exclusive prefixes of the tile groups over the wave's jobs.  CUDA-core tiles: dense
    // families' first (the register-blocked launch), then heavy jobs', then the light ones'
    int32_t pre[6];
    int32_t sup, pad;          // its family's support
};

// Tile groups of a wave: the order of DJob::pre.
enum { kGrpDense = 0, kGrpHeavy, kGrpLight, kGrpB1, kGrpTc, kGrpGram, kGrps };

// Phases of a wave (device-time stamps) and counter classes of a count job.
enum { kPhPack = 0, kPhZero, kPhLop3, kPhB1, kPhTc, kPhProj, kPhGram, kPhExpand, kPhMasks, kPhases };
enum { kClsLop3 = 0, kClsB1 = 1, kClsProj = 2, kClsTc = 3, kClsGram = 4, kClasses = 5 };

struct ResStatus {
    int32_t stack_n, look_n, fam_n, item_n, head_n, mfi_n, mfi_item_n, slot_n, free_n, free_taken, defer_n, log_n;
    int32_t jobs, rows, tiles_l3, tiles_b1, n_proj, n_mjobs;   // n_mjobs: masks the last expand asked for
    int32_t pj_n, pj_rows;                   // families to project, their rows in all,
    int64_t pj_words;                        // and the words these take
    int64_t pj_groups;                       // at most so many groups of 32 items hold their columns
    int64_t out_total;
    int32_t max_cols, max_head, starved, error;
    // grow: the wave the pack built does not fit the pools; nothing was consumed and the
    // g_* fields hold its size, for the host to grow the pools and pack again
    int32_t grow, g_rows, g_jobs, g_max_head, g_max_cols, waves;
    int64_t g_out, g_tiles;
    int32_t launch_id, next3, next1;         // next3 / next1: tile counters of the persistent counters
    int32_t tiles_l3d;                       // the first tiles_l3d CUDA-core tiles are dense families'
    int32_t tiles_tc, small;                  // packed tcgen05 family counter: tiles; the wave is the device loop's
    int32_t tiles_gr, next_gr;               // CUDA-core Gram counter: tiles, tile counter
    unsigned long long launch_t0;
    unsigned long long supports, nodes, lookaheads, hits, skipped, pep;
    // superset check: MFIs [0, sup_done) are in the item -> MFI index the expand reads
    int32_t sup_done, loop_go;               // loop_go: 1 run the packed wave, 0 leave, 2 leave (time limit)
    unsigned long long sup_pruned;
    // phase stamps of the current wave (first block start, last block end; %globaltimer ns)
    // and their durations summed over the search; the pack folds and resets them
    unsigned long long ph_s[kPhases], ph_e[kPhases], ph_ns[kPhases];
    // committed count jobs per counter class: algorithmic bytes (every operand row read once,
    // every count written once), bit-ops (supports x transactions), supports, jobs
    unsigned long long cls_bytes[kClasses], cls_bitops[kClasses], cls_sup[kClasses], cls_jobs[kClasses];
};

// Pool capacities, in entries.  A wave is packed only when the worst case of its expand fits.
struct Caps {
    int64_t fam, item, head, mfi, mfi_items, looks, slots, log, rows;
};
__host__ __device__ __forceinline__ bool wave_fits(const Caps& c, const ResStatus& st, int64_t rows, int64_t jobs,
                                                   int64_t out_total, int64_t max_head, int64_t max_cols, bool log_on) {
    const int64_t list = max_head + 2 + max_cols;
    return st.fam_n + rows + 1 <= c.fam && st.item_n + 2 * out_total + rows + 1 <= c.item &&
           st.head_n + rows * list + 1 <= c.head && st.mfi_n + rows + jobs + 1 <= c.mfi &&
           st.mfi_item_n + (rows + jobs) * list + 1 <= c.mfi_items && rows + 1 <= c.looks &&
           st.slot_n + 2 * rows + 2 <= c.slots && (!log_on || st.log_n + rows + 1 <= c.log) && rows <= c.rows;
}

struct ResPtrs {
    // pools
    DFam* fams;
    int32_t* items;
    int32_t* heads;
    int32_t* stack;
    DLook* looks;
    int32_t* free_slots;
    int32_t* defer;
    int32_t* mfi_off;
    int32_t* mfi_len;
    int32_t* mfi_sup;
    int32_t* mfi_items;
    float* log_feat;
    float* log_label;
    // wave
    DJob* djobs;
    MaskJob* mjobs;
    JobDesc* jobs;
    RowDesc* rows;
    int32_t* row_job;
    int32_t* row_local;
    TileDesc* tiles_l3;
    TileDesc* tiles_b1;
    TileDesc* tiles_tc;
    TileDesc* tiles_gr;
    int32_t* pk_list;             // jobs of each packed tile (kPkJobs entries)
    int32_t* counts;
    // constants
    const uint32_t* bitmap;
    uint32_t* masks;
    const int32_t* dense_freq;
    const uint8_t* is_root;
    const __nv_bfloat16* mlp_w;   // BF16 weights of the proposal (nullptr: none)
    const float* mlp_p;           // FP32 parameters (biases read from here)
    ResStatus* st;
    int64_t W, n_bits;
    int32_t min_count;
    int32_t wave_rows;            // cap on rows per wave
    int64_t cap_out, cap_tiles;
    int32_t counter;              // TFIM_COUNTER_*
    int32_t la_mode;              // 0 off, 1 filtered, 2 learned, 3 every node
    int32_t log_on;
    float proposal_threshold;
    int64_t kslice_min;           // b1 word slice when tiles are few (multiple of 64)
    int32_t sm_count;
    int32_t* proj_list;           // family jobs counted by the projected counter
    float avg_len;                // mean reduced transaction length
    int32_t csr_ok;               // the reduced transaction list repeats no id within a row
    int32_t proj_auto;            // let the automatic counter choice pick the projected counter
    int32_t b1_min_rows, b1_min_cols;   // automatic choice: tensor path from this job shape
    float l3_slices_per_sm, b1_tiles_per_sm;   // work split targets per wave
    float l3_dense_slices_per_sm;               // ... of dense families' CUDA-core tiles
    int32_t tc_min_work;                       // automatic choice of the tcgen05 family counter
    float tc_min_density, tc_tiles_per_sm;
    int32_t gram_min_rows;                     // ... and of the CUDA-core Gram counter
    Caps caps;
    int64_t row_bytes;            // bytes of one bitmap row (algorithmic traffic accounting)
    const struct RowSum* row_sum; // first pass of the expand precomputed per wave row (or nullptr)
    // graph-driven wave loop: stop after wave_limit waves or max_launch_ns of device time
    int32_t wave_limit, launch_id;
    unsigned long long max_launch_ns;
    // superset check (nullptr: off): bit k of word sup_index[x * sup_words + k / 32] is set
    // when MFI k holds item x, for items x < sup_items and MFIs k < sup_words * 32
    uint32_t* sup_index;
    int32_t sup_words, sup_items;
    // projected rows: an id >= n_base of an F list is row id - n_base of this table, a copy of
    // item vitem[id - n_base]'s row over the transactions of its family's universe
    int32_t n_base;
    const uint32_t** vrows;
    int32_t* vitem;
    PJob* pjobs;
    int32_t* pj_off;              // per family to project: bits before each tile, tiles + 1 entries
    uint32_t* pj_pool;
    // transactions as rows, for the projection: pj_chunks x N32 transactions x pj_gc words of 32 items
    // (positions in the top family's order), and per family its column at each position (or -1) and
    // the groups of each chunk with columns; null when the rows are compressed word by word
    uint32_t* pj_tm;
    int16_t* pj_inv;
    uint32_t* pj_gbits;
    int32_t* pj_pos;
    int32_t pj_chunks, pj_gc;
    ResStatus* h_st;              // pinned copy of the status record, written by the host-driven packs
};
// The dense item id of an F list entry.
__device__ __forceinline__ int32_t item_of(const ResPtrs& p, int32_t id) { return id < p.n_base ? id : p.vitem[id - p.n_base]; }
__device__ __forceinline__ const uint32_t* row_of(const ResPtrs& p, int32_t id) {
    return id < p.n_base ? p.bitmap + (int64_t)id * p.W : p.vrows[id - p.n_base];
}

// The first pass of the expand over one counted row: extensions (count >= min_count, own
// column excluded), equal-support extensions, tail extensions, whether an equal-support
// extension lies outside the tail (the subtree is pruned), and the column blocks of
// `column_block(nF)` columns that hold an extension.
struct RowSum {
    int32_t n_ext, n_eq, n_tail, prune;
    unsigned long long blocks;
    int64_t pad;
};
__host__ __device__ __forceinline__ int column_block(int nF) { return max(128, (((nF + 63) >> 6) + 31) & ~31); }

// Arguments of the graph-driven wave loop, kept in device memory so that growing a pool
// only rewrites this record (the captured launches stay valid).
struct ResArgs {
    ResPtrs p;
    CountArgs a3, a1, ap, atc, agr;   // CUDA-core, b1, projected, tcgen05 family and Gram counters
};

__device__ __forceinline__ unsigned long long globaltimer() { return dev_globaltimer(); }

// Projected counting pays when the prefix holds few transactions: it walks the base's set
// bits (W words) and looks up about 6 entries per item of each of its sup transactions,
// against the bitmap counters' (rows + columns + 1) x W words.
__device__ __forceinline__ bool use_proj(const ResPtrs& p, const JobDesc& jd, int32_t sup) {
    if (!p.csr_ok || jd.n_cols > kProjMaxCols || (jd.base_slot >= 0 && jd.base_item >= 0)) return false;
    if (jd.base_slot < 0 && jd.base_item < 0) return false;
    if (p.counter == TFIM_COUNTER_PROJ) return true;
    if (p.counter != TFIM_COUNTER_AUTO || !p.proj_auto) return false;
    const double proj = (double)p.W + (double)sup * 6.0 * (double)p.avg_len;
    const double bitmap = (double)(jd.n_rows + jd.n_cols + 1) * (double)p.W;
    return proj < bitmap;
}

__host__ __device__ __forceinline__ int64_t lmin(int64_t a, int64_t b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ int64_t lmax(int64_t a, int64_t b) { return a > b ? a : b; }

// Packed tcgen05 counter, automatic choice: a 128-column tile costs about 128 cycles per 64
// transactions whatever its jobs' tail rows, a register-blocked CUDA-core tile about 0.17 per
// row and column; on the 6.3M-row dense database the counting of the later waves took 20.1 / 18.1
// ms from 4 / 8 tail rows on.  Short rows stay with the CUDA cores, whose launch is the
// shorter one (10,000 rows, W = 320: 0.71 against 0.66 ms a mine).
constexpr int kPkMinRows = 8, kPkMinWords = 1024;
// and, over the wave, rows x columns x words, below which the second launch and its packing cost more
// than they save (a 1M-row sparse mine 1.69 / 1.72 ms with its one packed wave on the CUDA cores /
// packed; a 49,000-row dense one 2.62 / 2.56 ms with its waves below 2e8 / 5e7 on the CUDA cores).
constexpr float kPkMinWork = 1e8f;
// Narrow dense families of short rows stay with the Gram counter.  It neither gains nor costs much: 49,000 /
// 98,000 / 196,000 rows of the dense database mine in 2.28 / 2.93 / 2.89 ms with it and in 2.26 / 2.90 / 2.87 ms
// with their jobs in packed tiles or CUDA-core tiles.
constexpr int kGramMaxWords = 4096;

constexpr int kPackThreads = 1024;
constexpr int kPackItems = 4;
// A wave of at most this many rows x columns x words is counted inside the device loop (mines at
// 3e7 / 1e8 / 2e8 / 6e8: 2M dense rows 0.395 / 0.314 / 0.314 / 0.313 ms, 196,000 rows of the dense
// replicated database at 10% 1.03 / 0.91 / 0.90 / 1.02 ms).
constexpr float kLoopMaxWork = 2e8f;
// The empty prefix's family up to this many items^2 x words is counted there too (10,000-row dense
// database 0.394 -> 0.368 ms a mine, 70,000 rows at 90% 0.109 -> 0.088; beyond, the tensor tiles win).
constexpr double kLoopTopWork = 1e7;
constexpr int kPackCand = kPackThreads * kPackItems;

// The packed tcgen05 counter takes a family job (its rows are a run of its columns) of at most
// kPkMaxCols columns: always when that counter is asked for, and in the automatic choice from
// kPkMinRows tail rows on when its prefix is dense enough that skipping zero words (which the
// CUDA-core tiles do and the tensor tiles do not) saves little.
__device__ __forceinline__ bool use_tc(const ResPtrs& p, const JobDesc& jd, int32_t sup, int32_t n) {
    if (jd.n_cols < 1 || jd.n_cols > kPkMaxCols || jd.n_rows < 1) return false;
    if (p.counter == TFIM_COUNTER_I8) return true;
    if (p.counter != TFIM_COUNTER_AUTO) return false;
    if (jd.n_rows < kPkMinRows || jd.words < kPkMinWords || (int64_t)jd.n_rows * jd.n_cols < p.tc_min_work) return false;
    const float d = n > 0 ? fminf(1.f, 128.f * (float)sup / (float)n) : 1.f;
    return d >= p.tc_min_density;
}
// Jobs per packed tile by columns: 8, 16, 24, 32, 40, 64 or 128 rows of the tile each.
constexpr int kPkClasses = 7;
__device__ __forceinline__ int pk_class(int cols) {
    return cols <= 40 ? max(0, (cols - 1) >> 3) : cols <= 64 ? 5 : 6;
}
__device__ __forceinline__ int pk_per(int cls) { return cls <= 3 ? 16 / (cls + 1) : cls == 4 ? 3 : cls == 5 ? 2 : 1; }

// The CUDA-core Gram counter takes a dense family job of at most kGramMaxCols columns (and at
// most 128 blocks of 4 x 4 pairs) over rows of fewer than kGramMaxWords words: a dense prefix has no
// zero word for the general tiles to skip, and the columns are read once per job instead of once per
// eight rows.
__device__ __forceinline__ bool use_gram(const ResPtrs& p, const JobDesc& jd, int32_t sup, int32_t n) {
    // tails of 1 or 2 rows are memory-bound in any kernel (8 bit-ops per byte and row); the
    // general tiles handle them as well, and measured faster on the dense benchmark
    if (jd.n_cols < 1 || jd.n_cols > kGramMaxCols || jd.n_rows < p.gram_min_rows) return false;
    if (((jd.n_rows + 3) / 4) * ((jd.n_cols + 3) / 4) > 128 || jd.words >= kGramMaxWords) return false;
    if (p.counter != TFIM_COUNTER_AUTO) return false;
    const float d = n > 0 ? fminf(1.f, 128.f * (float)sup / (float)n) : 1.f;
    return d >= p.tc_min_density;
}

__device__ __forceinline__ bool use_b1_shape(const ResPtrs& p, int nr, int nc) {
    if (p.counter == TFIM_COUNTER_LOP3) return false;
    if (p.counter == TFIM_COUNTER_TENSOR) return true;
    return nr >= p.b1_min_rows && nc >= p.b1_min_cols;
}
__device__ __forceinline__ int64_t l3_tiles(int nr, int nc) { return (int64_t)((nr + kLop3Rows - 1) / kLop3Rows) * ((nc + 63) / 64); }
__device__ __forceinline__ int64_t b1_tiles(int nr, int nc) { return (int64_t)((nr + kB1Rows - 1) / kB1Rows) * ((nc + kB1Cols - 1) / kB1Cols); }

// ---------------------------------------------------------------------------------- pack
// One block.  Phases: (0) recycle the mask slots released by the last expand; (1) one job
// per queued lookahead; (2) families from the top of the stack, 4096 candidates per pass,
// with block scans deciding how many fit the wave's row and output budgets; (3) the counted
// rows and row->job maps; (4) tiles.  Every phase is block-parallel; jobs are ordered by their
// row offsets, which the row writer binary-searches, as the tile writers do the prefixes of
// their group.
//
// The kernel is a chain of latencies on one SM while the other 147 wait, so each phase scans
// all its quantities in one pass of warp shuffles (two barriers) and the binary searches run
// on prefixes held in shared memory.  Measured per launch: 10,000-row dense database 39 -> 18
// us, 1M-row sparse one 60 -> 38 us, 6.3M-row dense one 147 -> 100 us.
constexpr int kPackSearch = 5120;   // jobs whose prefixes fit the shared search arrays

// Exclusive prefixes of N values per thread over the block, and their totals.  `sm` holds
// N * 33 values; `any` = false: this warp's values are all zero.
template <int N, typename T>
__device__ __forceinline__ void block_scan(T (&v)[N], T (&ex)[N], T (&tot)[N], T* sm, bool any) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5;
    T inc[N];
#pragma unroll
    for (int k = 0; k < N; k++) inc[k] = v[k];
    if (any) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; k++) {
                const T x = __shfl_up_sync(0xffffffffu, inc[k], o);
                if (lane >= o) inc[k] += x;
            }
    }
    if (lane == 31)
#pragma unroll
        for (int k = 0; k < N; k++) sm[k * 33 + warp] = inc[k];
    __syncthreads();
    if (warp < N) {   // warp k scans value k's warp totals
        const T own = lane < warps ? sm[warp * 33 + lane] : T(0);
        T x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < warps) sm[warp * 33 + lane] = x - own;
        if (lane == 31) sm[warp * 33 + 32] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) {
        ex[k] = sm[k * 33 + warp] + inc[k] - v[k];
        tot[k] = sm[k * 33 + 32];
    }
    __syncthreads();   // sm is reused
}

// The last entry of the ascending a[0 .. n) that is <= t (a[0] <= t).
template <typename A>
__device__ __forceinline__ int last_le(const A& at, int n, int32_t t) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (at(mid) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Word slices of `n` tiles of `words` words each when a wave's tiles hold `total` words in all
// and should make about `want` slices: the slice length in words, a multiple of 64.
__device__ __forceinline__ int64_t slice_words(int64_t total, int64_t want) {
    return lmax(1, (total / lmax(want, 1) + 63) / 64) * 64;
}

// NT: threads of the block.  LOOP: the wave loop on the device (k_res_loop), which counts waves of
// at most kLoopMaxWork itself; these get no tiles.
template <int NT, bool LOOP>
__device__ __forceinline__ void res_pack(const ResPtrs& p) {
    constexpr int kPackThreads = NT, kPackCand = NT * kPackItems;
    __shared__ int64_t sm64[2 * 33];
    __shared__ int32_t sm32[kPkClasses * 33];
    __shared__ int32_t s_pre[kPackSearch];
    __shared__ int32_t s_src[kPackSearch];
    __shared__ int32_t s_n_jobs, s_rows_total, s_done, s_max_cols, s_max_head, s_stack_after, s_kstop, s_fit;
    __shared__ int64_t s_out_total;
    __shared__ float s_cost, s_pk_work, s_pk_cost, s_work;
    __shared__ unsigned long long s_words[3];   // words of the wave's b1 / tcgen05 / Gram tiles
    ResStatus* st = p.st;
    const int tid = threadIdx.x, lane = tid & 31;
    // (0) recycle
    const int32_t taken = min(st->free_taken, st->free_n);
    const int32_t fn = st->free_n - taken, dn = st->defer_n;
    const int32_t n_look = st->look_n;
    for (int k = tid; k < dn; k += kPackThreads) p.free_slots[fn + k] = p.defer[k];
    if (tid < kPhases) {
        // the last wave's phases: add their durations, clear the stamps, stamp this pack
        const unsigned long long s0 = st->ph_s[tid], e0 = st->ph_e[tid];
        if (s0 != ~0ull && e0 > s0) st->ph_ns[tid] += e0 - s0;
        st->ph_s[tid] = tid == kPhPack ? globaltimer() : ~0ull;
        st->ph_e[tid] = 0;
    }
    if (tid == 32) {
        s_n_jobs = n_look; s_rows_total = n_look; s_out_total = 0; s_max_cols = 0; s_max_head = 0; s_done = 0;
        s_stack_after = st->stack_n;
        s_cost = s_pk_work = s_pk_cost = s_work = 0.f;
        s_words[0] = s_words[1] = s_words[2] = 0;
        st->n_proj = 0;
        st->n_mjobs = 0;
        st->grow = 0;
        st->starved = 0;
        // MFIs of the finished waves are indexed (k_index_mfis ran after the last expand)
        if (p.sup_index) st->sup_done = min(st->mfi_n, p.sup_words * 32);
        if (st->launch_id != p.launch_id) {
            st->launch_id = p.launch_id;
            st->launch_t0 = globaltimer();
        }
    }
    __syncthreads();
    if (tid == 0) {
        st->free_n = fn + dn;
        st->free_taken = 0;
        st->defer_n = 0;
    }
    // (1) lookahead jobs
    for (int base = 0; base < n_look; base += kPackThreads) {
        const int k = base + tid;
        int64_t v[1] = {0}, ex[1], tot[1];
        DLook L{};
        DFam f{};
        if (k < n_look) {
            L = p.looks[k];
            f = p.fams[L.fam];
            v[0] = f.nF - f.nT + 1;
            atomicMax(&s_max_cols, (int32_t)v[0]);
        }
        block_scan<1>(v, ex, tot, sm64, base + (tid & ~31) < n_look);
        if (k < n_look) {
            DJob dj{};
            dj.fam = L.fam; dj.kind = kJobLook; dj.nr = 1; dj.slot = L.slot; dj.log = L.log; dj.sl3 = 1; dj.sup = f.sup;
            p.djobs[k] = dj;
            JobDesc jd;
            jd.base_slot = -1; jd.base_item = -1; jd.n_rows = 1; jd.n_cols = (int32_t)v[0];
            jd.row_off = k; jd.col_off = f.F_off + f.nT; jd.out_off = s_out_total + ex[0]; jd.self_col = f.nF - f.nT;
            jd.words = f.W;
            p.jobs[k] = jd;
            if (k < kPackSearch) {
                s_pre[k] = k;
                s_src[k] = -1 - L.slot;
            }
        }
        __syncthreads();
        if (tid == 0) s_out_total += tot[0];
        __syncthreads();
    }
    // (2) families from the top of the stack
    while (!s_done) {
        const int32_t avail = s_stack_after;
        const int32_t n_c = min(avail, kPackCand);
        if (n_c == 0) break;
        const int64_t rows_left = (int64_t)p.wave_rows - s_rows_total;
        const int64_t out_left = p.cap_out - s_out_total;
        const int64_t out_base = s_out_total;
        const int32_t rows_base = s_rows_total, jobs_base = s_n_jobs;
        const bool any = (tid & ~31) * kPackItems < n_c;
        int32_t fid[kPackItems];
        int64_t rv[kPackItems], ov[kPackItems];
        int32_t nf[kPackItems], hl[kPackItems];
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            const int k = tid * kPackItems + q;
            fid[q] = k < n_c ? p.stack[avail - 1 - k] : -1;
        }
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            rv[q] = ov[q] = 0;
            nf[q] = hl[q] = 0;
            if (fid[q] >= 0) {
                const DFam f = p.fams[fid[q]];
                const int32_t rem = f.state == 0 ? f.nT - f.next_row : 0;
                rv[q] = rem;
                ov[q] = (int64_t)rem * f.nF;
                nf[q] = f.nF;
                hl[q] = f.head_len;
            }
        }
        if (tid == 0) s_kstop = n_c;
        int64_t tr[2] = {0, 0}, ex[2], tot[2];
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            tr[0] += rv[q];
            tr[1] += ov[q];
        }
        block_scan<2>(tr, ex, tot, sm64, any);
        // take per candidate and the first stop point
        int32_t take[kPackItems];
        int64_t o_at[kPackItems];
        int kstop = n_c;
        int64_t rb = ex[0], ob = ex[1];
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            const int k = tid * kPackItems + q;
            take[q] = -1;
            o_at[q] = ob;
            if (k < n_c) {
                const int64_t r1 = rb + rv[q], o1 = ob + ov[q];
                if (r1 <= rows_left && o1 <= out_left) {
                    take[q] = (int32_t)rv[q];
                } else if (rb < rows_left && ob < out_left) {
                    take[q] = (int32_t)lmin(lmin(rows_left - rb, (out_left - ob) / max(1, nf[q])), rv[q]);
                    if (take[q] == 0 && rb == 0 && ob == 0 && jobs_base == 0) atomicExch(&st->starved, 1);
                }
                if (take[q] < 0 || (rv[q] > 0 && take[q] < rv[q])) kstop = min(kstop, k);
                rb = r1;
                ob = o1;
            }
        }
        if (kstop < n_c) atomicMin(&s_kstop, kstop);
        __syncthreads();
        const int32_t ks = s_kstop;
        // jobs: candidates before the stop point with rows left, and the stop point if it takes rows
        bool hj[kPackItems];
        int32_t jv[2] = {0, 0}, jx[2], jt[2];
        int32_t mcol = 0, mhead = 0;
        int64_t contrib = 0;
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            const int k = tid * kPackItems + q;
            hj[q] = k < n_c && ((k < ks && rv[q] > 0) || (k == ks && take[q] > 0));
            if (hj[q]) {
                jv[0] += 1;
                jv[1] += take[q];
                mcol = max(mcol, nf[q]);
                mhead = max(mhead, hl[q]);
                contrib += (int64_t)take[q] * nf[q];
            }
        }
        block_scan<2>(jv, jx, jt, sm32, any);
        if (any) {
            mcol = __reduce_max_sync(0xffffffffu, mcol);
            mhead = __reduce_max_sync(0xffffffffu, mhead);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, o);
            if (lane == 0) {
                atomicMax(&s_max_cols, mcol);
                atomicMax(&s_max_head, mhead);
                if (contrib) atomicAdd((unsigned long long*)&s_out_total, (unsigned long long)contrib);
            }
        }
        int32_t jid = jobs_base + jx[0], row = rows_base + jx[1];
#pragma unroll
        for (int q = 0; q < kPackItems; q++) {
            if (!hj[q]) continue;
            const DFam f = p.fams[fid[q]];
            DJob dj{};
            dj.fam = fid[q]; dj.kind = kJobFam; dj.r0 = f.next_row; dj.nr = take[q]; dj.slot = -1; dj.log = -1; dj.sl3 = 1;
            dj.sup = f.sup;
            p.djobs[jid] = dj;   // next_row advances when the wave is committed
            JobDesc jd;
            jd.base_slot = f.slot; jd.base_item = f.item; jd.n_rows = take[q]; jd.n_cols = f.nF;
            jd.row_off = row;
            jd.col_off = f.F_off;
            // outputs: every candidate before this one contributed rv * nF, this one take * nF
            jd.out_off = out_base + o_at[q];
            jd.self_col = -1; jd.words = f.W; jd.r0 = f.next_row;
            p.jobs[jid] = jd;
            if (jid < kPackSearch) {
                s_pre[jid] = row;
                s_src[jid] = f.F_off + f.next_row;
            }
            jid++;
            row += take[q];
        }
        __syncthreads();
        if (tid == 0) {
            s_n_jobs = jobs_base + jt[0];
            s_rows_total = rows_base + jt[1];
            s_stack_after = avail - ks;   // candidates before the stop point are consumed
            if (ks < n_c || s_rows_total >= p.wave_rows || n_c < kPackCand || s_stack_after == 0) s_done = 1;
        }
        __syncthreads();
    }
    const int32_t nj = s_n_jobs, rows_total = s_rows_total;
    const bool in_sm = nj <= kPackSearch;
    // (3) rows
    for (int32_t g = tid; g < rows_total; g += kPackThreads) {
        int j, r;
        int32_t src;
        if (in_sm) {
            j = last_le([&](int k) { return s_pre[k]; }, nj, g);
            r = g - s_pre[j];
            src = s_src[j];
        } else {
            j = last_le([&](int k) { return p.jobs[k].row_off; }, nj, g);
            r = g - p.jobs[j].row_off;
            const DJob dj = p.djobs[j];
            src = dj.kind == kJobFam ? p.jobs[j].col_off + dj.r0 : -1 - dj.slot;
        }
        p.rows[g] = src >= 0 ? RowDesc{-1, p.items[src + r]} : RowDesc{-1 - src, -1};
        p.row_job[g] = j;
        p.row_local[g] = r;
    }
    // (4) tiles.  Pass 1 picks each job's counter and sums the estimated cost of its CUDA-core
    // tiles and the words of the others; pass 2 gives every job its own number of word slices (a
    // heavy job -- dense prefix, many rows and columns, long rows -- is split so that no tile
    // runs far longer than the wave's average) and forms the prefix sums the tile writers search.
    auto l3_cost = [&](const JobDesc& jd, const DJob& dj, int32_t n) -> float {
        float d = 1.f;   // fraction of 128-bit base positions that are nonzero
        if (dj.kind == kJobFam && (jd.base_slot >= 0 || jd.base_item >= 0) && n > 0)
            d = fminf(1.f, 128.f * (float)dj.sup / (float)n);
        const float nr = (float)min(jd.n_rows, kLop3Rows), nc = (float)min(jd.n_cols, 64);
        return (float)(jd.words >> 2) * (1.f + d * (2.f + nr + nr * nc / 32.f));
    };
    if (LOOP) {   // rows x columns x words of the wave
        float work = 0.f;
        for (int j = tid; j < nj; j += kPackThreads) {
            const JobDesc jd = p.jobs[j];
            work += (float)jd.n_rows * (float)jd.n_cols * (float)jd.words;
        }
        if ((tid & ~31) < nj) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) work += __shfl_xor_sync(0xffffffffu, work, o);
            if (lane == 0) atomicAdd(&s_work, work);
        }
        __syncthreads();
    }
    const bool small = LOOP && s_work <= kLoopMaxWork;
    if (small)
        for (int j = tid; j < nj; j += kPackThreads) {
            p.djobs[j].cls = kGrpLight;
            p.djobs[j].pad = p.fams[p.djobs[j].fam].n;
        }
    if (!small) {
        float cost = 0.f, pk_work = 0.f, pk_cost = 0.f;   // of the packed jobs: pairs x words; as CUDA-core tiles
        unsigned long long w1 = 0, wt = 0, wg = 0;
        for (int j = tid; j < nj; j += kPackThreads) {
            const JobDesc jd = p.jobs[j];
            const DJob dj = p.djobs[j];
            const bool fam = dj.kind == kJobFam;
            const int32_t n = p.fams[dj.fam].n;
            int cls;
            if (fam && use_proj(p, jd, dj.sup)) {
                cls = kGrps;
                p.proj_list[atomicAdd(&st->n_proj, 1)] = j;
            } else if (fam && use_gram(p, jd, dj.sup, n)) {
                cls = kGrpGram;
                wg += (unsigned long long)jd.words;
            } else if (fam && use_tc(p, jd, dj.sup, n)) {
                cls = kGrpTc;
                wt += (unsigned long long)(jd.words / pk_per(pk_class(jd.n_cols)) + 1);
                pk_work += (float)jd.n_rows * (float)jd.n_cols * (float)jd.words;
                pk_cost += (float)l3_tiles(jd.n_rows, jd.n_cols) * l3_cost(jd, dj, n);
            } else if (fam && use_b1_shape(p, jd.n_rows, jd.n_cols)) {
                cls = kGrpB1;
                w1 += (unsigned long long)(b1_tiles(jd.n_rows, jd.n_cols) * jd.words);
            } else {
                // Tiles of dense families and of their lookaheads (the family's prefix holds at
                // least 1/16 of its transactions, so no 128-bit position is zero to skip) come
                // first, for the register-blocked dense launch
                cls = 16 * (int64_t)dj.sup >= n ? kGrpDense : kGrpLight;
                cost += (float)l3_tiles(jd.n_rows, jd.n_cols) * l3_cost(jd, dj, n);
            }
            p.djobs[j].cls = cls;
            p.djobs[j].pad = n;
        }
        if ((tid & ~31) < nj) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                cost += __shfl_xor_sync(0xffffffffu, cost, o);
                pk_work += __shfl_xor_sync(0xffffffffu, pk_work, o);
                pk_cost += __shfl_xor_sync(0xffffffffu, pk_cost, o);
                w1 += __shfl_xor_sync(0xffffffffu, w1, o);
                wt += __shfl_xor_sync(0xffffffffu, wt, o);
                wg += __shfl_xor_sync(0xffffffffu, wg, o);
            }
            if (lane == 0) {
                atomicAdd(&s_cost, cost);
                if (w1) atomicAdd(&s_words[0], w1);
                if (wt) {
                    atomicAdd(&s_words[1], wt);
                    atomicAdd(&s_pk_work, pk_work);
                    atomicAdd(&s_pk_cost, pk_cost);
                }
                if (wg) atomicAdd(&s_words[2], wg);
            }
        }
        __syncthreads();
    }
    // a wave whose packed jobs are little work in all counts them on the CUDA cores instead.  The
    // shared sums are only read from here on: what the decision changes stays in registers
    const bool few_pk = p.counter == TFIM_COUNTER_AUTO && s_words[1] > 0 && s_pk_work < kPkMinWork;
    const int64_t pk_words = few_pk ? 0 : (int64_t)s_words[1];
    const float l3_total = s_cost + (few_pk ? s_pk_cost : 0.f);
    // the wave's estimated CUDA-core cost over (slices per SM x SMs): the cost of one tile
    // slice; dense families are split more finely (their own target), which shortens the
    // launch's tail on large dense databases
    const float target = fmaxf(l3_total / (p.l3_slices_per_sm * (float)p.sm_count), 1.f);
    const float target_d = fmaxf(l3_total / (p.l3_dense_slices_per_sm * (float)p.sm_count), 1.f);
    const int64_t sw_b1 = slice_words((int64_t)s_words[0], (int64_t)(p.b1_tiles_per_sm * (float)p.sm_count));
    const int64_t sw_tc = slice_words(pk_words, (int64_t)(p.tc_tiles_per_sm * (float)p.sm_count));
    const int64_t sw_gr = slice_words((int64_t)s_words[2], (int64_t)(p.l3_slices_per_sm * (float)p.sm_count));
    int32_t tot[kGrps] = {0, 0, 0, 0, 0, 0};
    for (int base = 0; base < (small ? 0 : nj); base += kPackThreads) {
        const int j = base + tid;
        int32_t v[kGrps] = {0, 0, 0, 0, 0, 0}, ex[kGrps], t[kGrps];
        if (j < nj) {
            const JobDesc jd = p.jobs[j];
            DJob* djp = p.djobs + j;
            const DJob dj = *djp;
            const int64_t W = jd.words;
            int64_t sl = 1, per = 1;   // word slices, tiles per slice
            int cls = dj.cls;
            if (few_pk && cls == kGrpTc) cls = 16 * (int64_t)dj.sup >= dj.pad ? kGrpDense : kGrpLight;
            if (cls <= kGrpLight) {
                const float cost = l3_cost(jd, dj, dj.pad);
                sl = lmin(lmax(1, W / 256), lmax(1, (int64_t)ceilf(cost / (cls == kGrpDense ? target_d : target))));
                // heavy jobs (cost at least half the slice target) before the light ones, so that the
                // longest tiles are dispatched first and the light ones fill in behind them
                if (cls == kGrpLight && cost >= 0.5f * target) cls = kGrpHeavy;
                per = l3_tiles(jd.n_rows, jd.n_cols);
            } else if (cls < kGrps) {
                const int64_t sw = cls == kGrpB1 ? sw_b1 : sw_gr;
                sl = (W + sw - 1) / sw;
                if (cls == kGrpB1) per = b1_tiles(jd.n_rows, jd.n_cols);
            }
            if (cls < kGrps && cls != kGrpTc) {
                const int64_t wsl = ((W / 64 + sl - 1) / sl) * 64;
                sl = wsl > 0 ? (W + wsl - 1) / wsl : 1;
                djp->sl3 = (int32_t)sl;
                djp->cls = cls;
#pragma unroll
                for (int k = 0; k < kGrps; k++) v[k] = k == cls ? (int32_t)lmin(per * sl, 1 << 30) : 0;
            }
        }
        block_scan<kGrps>(v, ex, t, sm32, base + (tid & ~31) < nj);
        if (j < nj)
#pragma unroll
            for (int k = 0; k < kGrps; k++) p.djobs[j].pre[k] = tot[k] + ex[k];
#pragma unroll
        for (int k = 0; k < kGrps; k++) tot[k] += t[k];
    }
    // packed tiles: the jobs of a class fill them in order; the tiles of class k follow those of
    // class k - 1
    int32_t n_pk = 0;          // packed tiles before slicing
    int32_t TT = 0;            // and in word slices
    int32_t pk_first[kPkClasses] = {0, 0, 0, 0, 0, 0, 0}, pk_jobs[kPkClasses] = {0, 0, 0, 0, 0, 0, 0};
    // counts the word slices of the packed tiles and, with `write`, writes them; a slice holds at
    // most 2^18 words, so that FP32 sums stay exact
    auto pk_tiles = [&](bool write) -> int32_t {
        int32_t run = 0;
        for (int base = 0; base < n_pk; base += kPackThreads) {
            const int b = base + tid;
            int32_t n = 0, per = 1, v[1] = {0}, ex[1], t[1];
            int64_t W = 0, wsl = 64;
            if (b < n_pk) {
#pragma unroll
                for (int k = 0; k < kPkClasses; k++)
                    if (pk_jobs[k] > 0 && b >= pk_first[k]) {   // the last such class holds tile b
                        per = pk_per(k);
                        n = min(per, pk_jobs[k] - (b - pk_first[k]) * per);
                    }
                for (int i = 0; i < n; i++) W = lmax(W, (int64_t)p.jobs[p.pk_list[b * kPkJobs + i]].words);
                const int64_t sw = lmin(sw_tc, 1 << 18), sl = lmax(1, (W + sw - 1) / sw);
                wsl = lmax(1, (W / 64 + sl - 1) / sl) * 64;
                v[0] = (int32_t)((W + wsl - 1) / wsl);
            }
            block_scan<1>(v, ex, t, sm32, base + (tid & ~31) < n_pk);
            if (write)
                for (int32_t q = 0; q < v[0]; q++)
                    p.tiles_tc[run + ex[0] + q] = TileDesc{b * kPkJobs, 0, n, per, 0, (int32_t)(q * wsl),
                                                           (int32_t)lmin(W, (q + 1) * wsl), 0};
            run += t[0];
        }
        return run;
    };
    if (!small && pk_words > 0) {
        for (int base = 0; base < nj; base += kPackThreads) {
            const int j = base + tid;
            int32_t v[kPkClasses] = {0, 0, 0, 0, 0, 0, 0}, ex[kPkClasses], t[kPkClasses];
            const bool in = j < nj && p.djobs[j].cls == kGrpTc;
            const int pc = in ? pk_class(p.jobs[j].n_cols) : 0;
            if (in)
#pragma unroll
                for (int k = 0; k < kPkClasses; k++) v[k] = k == pc;
            block_scan<kPkClasses>(v, ex, t, sm32, base + (tid & ~31) < nj);
#pragma unroll
            for (int k = 0; k < kPkClasses; k++) {
                if (in && k == pc) p.djobs[j].pre[kGrpTc] = pk_jobs[k] + ex[k];
                pk_jobs[k] += t[k];
            }
        }
#pragma unroll
        for (int k = 0; k < kPkClasses; k++) {
            pk_first[k] = n_pk;
            n_pk += (pk_jobs[k] + pk_per(k) - 1) / pk_per(k);
        }
        for (int j = tid; j < nj; j += kPackThreads) {
            const DJob dj = p.djobs[j];
            if (dj.cls != kGrpTc) continue;
            const int pc = pk_class(p.jobs[j].n_cols), per = pk_per(pc);
            int32_t first = 0;
#pragma unroll
            for (int k = 0; k < kPkClasses; k++)
                if (k == pc) first = pk_first[k];
            p.pk_list[(first + dj.pre[kGrpTc] / per) * kPkJobs + dj.pre[kGrpTc] % per] = j;
        }
        __syncthreads();   // the lists are read below
        TT = pk_tiles(false);
    }
    const int64_t T3 = (int64_t)tot[kGrpDense] + tot[kGrpHeavy] + tot[kGrpLight], T1 = tot[kGrpB1], TG = tot[kGrpGram];
    // the wave is committed only when the worst case of its expand fits the pools
    if (tid == 0) {
        const bool fit = s_out_total <= p.cap_out && T1 <= p.cap_tiles && T3 <= p.cap_tiles && TT <= p.cap_tiles &&
                         TG <= p.cap_tiles &&
                         wave_fits(p.caps, *st, rows_total, nj, s_out_total, s_max_head, s_max_cols, p.log_on != 0);
        s_fit = fit;
        if (!fit) {
            st->grow = 1;
            st->g_rows = rows_total;
            st->g_jobs = nj;
            st->g_out = s_out_total;
            st->g_max_head = s_max_head;
            st->g_max_cols = s_max_cols;
            st->g_tiles = lmax(lmax(lmax(T1, T3), TT), TG);
            st->jobs = 0; st->rows = 0; st->tiles_l3 = 0; st->tiles_l3d = 0; st->tiles_b1 = 0; st->tiles_tc = 0;
            st->tiles_gr = 0; st->n_proj = 0;
            st->out_total = 0;
            st->ph_e[kPhPack] = globaltimer();
        }
    }
    __syncthreads();   // s_fit; s_pre is free
    if (!s_fit) return;
    // commit: the families hand out their rows; the wave's work per counter class (warp sums, one
    // atomic per warp and class)
    {
        unsigned long long cb[kClasses], cbo[kClasses], cs[kClasses], cj[kClasses];
#pragma unroll
        for (int k = 0; k < kClasses; k++) cb[k] = cbo[k] = cs[k] = cj[k] = 0;
        for (int j = tid; j < nj; j += kPackThreads) {
            const JobDesc jd = p.jobs[j];
            const DJob dj = p.djobs[j];
            if (dj.kind == kJobFam) p.fams[dj.fam].next_row = dj.r0 + dj.nr;
            const int cls = dj.cls <= kGrpLight ? kClsLop3
                            : dj.cls == kGrpB1  ? kClsB1
                            : dj.cls == kGrpTc  ? kClsTc
                            : dj.cls == kGrpGram ? kClsGram
                                                 : kClsProj;
            const unsigned long long nbase = (jd.base_slot >= 0) + (jd.base_item >= 0);
            const unsigned long long sup = (unsigned long long)jd.n_rows * (unsigned long long)jd.n_cols;
            const unsigned long long by = (unsigned long long)((dj.pad + 7) / 8) *
                                              ((unsigned long long)jd.n_rows + jd.n_cols + nbase) + 4ull * sup;
#pragma unroll
            for (int k = 0; k < kClasses; k++)
                if (cls == k) {
                    cb[k] += by;
                    cbo[k] += sup * (unsigned long long)dj.pad;
                    cs[k] += sup;
                    cj[k] += 1;
                }
        }
        if ((tid & ~31) < nj) {
#pragma unroll
            for (int k = 0; k < kClasses; k++) {
                if (!__any_sync(0xffffffffu, cj[k] != 0)) continue;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    cb[k] += __shfl_xor_sync(0xffffffffu, cb[k], o);
                    cbo[k] += __shfl_xor_sync(0xffffffffu, cbo[k], o);
                    cs[k] += __shfl_xor_sync(0xffffffffu, cs[k], o);
                    cj[k] += __shfl_xor_sync(0xffffffffu, cj[k], o);
                }
                if (lane == 0) {
                    atomicAdd(&st->cls_bytes[k], cb[k]);
                    atomicAdd(&st->cls_bitops[k], cbo[k]);
                    atomicAdd(&st->cls_sup[k], cs[k]);
                    atomicAdd(&st->cls_jobs[k], cj[k]);
                }
            }
        }
    }
    // the tiles of one group: `base` = the group's first entry of its tile list
    auto emit = [&](int grp, TileDesc* out, int64_t first) {
        const int32_t n = tot[grp];
        if (n == 0) return;
        if (in_sm) {
            for (int j = tid; j < nj; j += kPackThreads) s_pre[j] = p.djobs[j].pre[grp];
            __syncthreads();
        }
        for (int32_t t = tid; t < n; t += kPackThreads) {
            // the job owning tile t: jobs of other groups share the prefix of the next one of this group
            const int j = in_sm ? last_le([&](int k) { return s_pre[k]; }, nj, t)
                                : last_le([&](int k) { return p.djobs[k].pre[grp]; }, nj, t);
            const JobDesc jd = p.jobs[j];
            const DJob dj = p.djobs[j];
            const int32_t local = t - dj.pre[grp];
            const int64_t W = jd.words, wsl = ((W / 64 + dj.sl3 - 1) / dj.sl3) * 64;
            if (grp == kGrpGram) {
                // rows 0 .. n_rows of the job are its columns dj.r0 .. dj.r0 + n_rows
                const int64_t w0 = local * wsl;
                out[first + t] = TileDesc{j, 0, jd.n_rows, 0, jd.n_cols, (int32_t)w0, (int32_t)lmin(W, w0 + wsl), dj.r0};
            } else {
                const int tr = grp == kGrpB1 ? kB1Rows : kLop3Rows, tc = grp == kGrpB1 ? kB1Cols : 64;
                const int cg = (jd.n_cols + tc - 1) / tc;
                const int bt = cg * ((jd.n_rows + tr - 1) / tr);
                const int slice = local / bt, within = local - slice * bt;
                const int rg = within / cg, cc = within - rg * cg;
                const int64_t w0 = slice * wsl;
                out[first + t] = TileDesc{j, rg * tr, min(tr, jd.n_rows - rg * tr), cc * tc, min(jd.n_cols, cc * tc + tc),
                                          (int32_t)w0, (int32_t)lmin(W, w0 + wsl), grp == kGrpDense ? 1 : 0};
            }
        }
        __syncthreads();   // s_pre is reused
    };
    emit(kGrpDense, p.tiles_l3, 0);
    emit(kGrpHeavy, p.tiles_l3, tot[kGrpDense]);
    emit(kGrpLight, p.tiles_l3, (int64_t)tot[kGrpDense] + tot[kGrpHeavy]);
    emit(kGrpB1, p.tiles_b1, 0);
    if (TT > 0) pk_tiles(true);
    emit(kGrpGram, p.tiles_gr, 0);
    if (tid == 0) {
        st->small = small ? 1 : 0;
        st->jobs = nj;
        st->rows = rows_total;
        st->tiles_l3 = (int32_t)T3;
        st->tiles_l3d = tot[kGrpDense];
        st->tiles_b1 = (int32_t)T1;
        st->tiles_tc = TT;
        st->tiles_gr = (int32_t)TG;
        st->out_total = s_out_total;
        st->max_cols = s_max_cols;
        st->max_head = s_max_head;
        st->stack_n = s_stack_after;
        st->look_n = 0;
        st->nodes += rows_total;
        st->supports += s_out_total;
        st->ph_e[kPhPack] = globaltimer();
    }
}

// The status record into pinned host memory (one block).
__device__ __forceinline__ void publish_status(const ResPtrs& p) {
    __syncthreads();
    static_assert(sizeof(ResStatus) % 8 == 0, "the record is copied in 8-byte words");
    const volatile unsigned long long* from = reinterpret_cast<const volatile unsigned long long*>(p.st);
    unsigned long long* to = reinterpret_cast<unsigned long long*>(p.h_st);
    for (int i = threadIdx.x; i < (int)(sizeof(ResStatus) / 8); i += blockDim.x) to[i] = from[i];
}

__global__ void __launch_bounds__(kPackThreads) k_res_pack(ResPtrs p) {
    res_pack<kPackThreads, false>(p);
    publish_status(p);
}
__global__ void __launch_bounds__(kPackThreads) k_res_pack_g(const ResArgs* __restrict__ args) {
    const ResPtrs p = args->p;
    res_pack<kPackThreads, false>(p);
}

// ---------------------------------------------------------------------------------- expand helpers
__device__ __forceinline__ int32_t pop_slot(const ResPtrs& p) {
    const int32_t k = atomicAdd(&p.st->free_taken, 1);
    const int32_t fn = p.st->free_n;
    if (k < fn) return p.free_slots[fn - 1 - k];
    return atomicAdd(&p.st->slot_n, 1);
}
__device__ __forceinline__ void release_slot(const ResPtrs& p, int32_t s) {
    if (s < 0) return;
    const int32_t k = atomicAdd(&p.st->defer_n, 1);
    p.defer[k] = s;
}

// Record a mask for k_build_masks (lane 0 of the calling warp).
__device__ __forceinline__ void emit_mask(const ResPtrs& p, int32_t dst, int32_t slot, int32_t item, int32_t t, int32_t off,
                                          int32_t n, int32_t W, int lane) {
    if (lane == 0) {
        const int32_t k = atomicAdd(&p.st->n_mjobs, 1);
        p.mjobs[k] = MaskJob{dst, slot, item, t, off, n, W, 0};
    }
}

// Sort an emitted MFI's item list (distinct dense ids) in descending order in place: a rank
// sort with two items per lane when it holds at most 64 items (longer lists are sorted by the
// host, which checks every list).
__device__ void warp_sort_desc(int32_t* a, int n, int lane) {
    if (n > 64 || n < 2) return;
    __syncwarp();
    const int32_t v0 = lane < n ? a[lane] : INT_MIN, v1 = lane + 32 < n ? a[lane + 32] : INT_MIN;
    int r0 = 0, r1 = 0;
    for (int j = 0; j < n; j++) {
        const int32_t x = __shfl_sync(0xffffffffu, j < 32 ? v0 : v1, j & 31);
        r0 += x > v0;
        r1 += x > v1;
    }
    __syncwarp();
    if (lane < n) a[r0] = v0;
    if (lane + 32 < n) a[r1] = v1;
    __syncwarp();
}

__device__ void warp_emit_mfi(const ResPtrs& p, const int32_t* head, int head_len, int32_t t, const int32_t* extra_cols,
                              int n_extra, const int32_t* F, int32_t sup, int lane) {
    // max dense id decides the root rule
    int32_t mx = t;
    for (int q = lane; q < head_len; q += 32) mx = max(mx, head[q]);
    for (int q = lane; q < n_extra; q += 32) mx = max(mx, item_of(p, F[extra_cols[q]]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (!p.is_root[mx]) return;
    const int len = head_len + 1 + n_extra;
    int32_t k = 0, off = 0;
    if (lane == 0) {
        k = atomicAdd(&p.st->mfi_n, 1);
        off = atomicAdd(&p.st->mfi_item_n, len);
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    off = __shfl_sync(0xffffffffu, off, 0);
    for (int q = lane; q < head_len; q += 32) p.mfi_items[off + q] = head[q];
    if (lane == 0) p.mfi_items[off + head_len] = t;
    for (int q = lane; q < n_extra; q += 32) p.mfi_items[off + head_len + 1 + q] = item_of(p, F[extra_cols[q]]);
    warp_sort_desc(p.mfi_items + off, len, lane);
    if (lane == 0) {
        p.mfi_off[k] = off;
        p.mfi_len[k] = len;
        p.mfi_sup[k] = len == 1 ? p.dense_freq[t] : sup;   // a root's own frequency is its F1 count
    }
}

// Whether some indexed MFI (ids below `done`) holds every item of head[0, nh) and tail[0, nt):
// one index word per lane, ANDed over the items until every lane's word is zero.  Items
// beyond the index hold no indexed MFI.
__device__ bool warp_covered(const ResPtrs& p, int32_t done, const int32_t* head, int nh, const int32_t* tail, int nt,
                             int lane) {
    const int nw = (done + 31) >> 5;
    const int n = nh + nt;
    for (int w0 = 0; w0 < nw; w0 += 32) {
        const int w = w0 + lane;
        uint32_t acc = w < nw ? ~0u : 0u;
        if (w == nw - 1 && (done & 31)) acc = (1u << (done & 31)) - 1u;
        for (int q = 0; q < n; q++) {
            if (!__any_sync(0xffffffffu, acc != 0u)) break;
            const int32_t x = q < nh ? head[q] : item_of(p, tail[q - nh]);
            if (x < 0 || x >= p.sup_items) acc = 0u;
            else if (acc) acc &= p.sup_index[(int64_t)x * p.sup_words + w];
        }
        if (__any_sync(0xffffffffu, acc != 0u)) return true;
    }
    return false;
}

__device__ void finish_row(const ResPtrs& p, DFam* f, int lane) {
    if (lane == 0) {
        const int32_t done = atomicAdd(&f->rows_done, 1) + 1;
        if (done == f->nT) {
            release_slot(p, f->slot);
            f->state = 2;
        }
    }
}

// The proposal network on one warp: lane i holds feature i.
__device__ float warp_mlp(const ResPtrs& p, float x, int lane) {
    const __nv_bfloat16* w = p.mlp_w;
    const float* P = p.mlp_p;
    constexpr int kIn = 32, kH = 64;
    constexpr int oW1 = 0, oB1 = kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH, oB3 = oW3 + kH;
    float h1a = P[oB1 + lane], h1b = P[oB1 + lane + 32];
    for (int i = 0; i < kIn; i++) {
        const float xi = __shfl_sync(0xffffffffu, x, i);
        h1a = fmaf(__bfloat162float(w[oW1 + lane * kIn + i]), xi, h1a);
        h1b = fmaf(__bfloat162float(w[oW1 + (lane + 32) * kIn + i]), xi, h1b);
    }
    h1a = fmaxf(h1a, 0.f);
    h1b = fmaxf(h1b, 0.f);
    float h2a = P[oB2 + lane], h2b = P[oB2 + lane + 32];
    for (int j = 0; j < kH; j++) {
        const float hj = __shfl_sync(0xffffffffu, j < 32 ? h1a : h1b, j & 31);
        h2a = fmaf(__bfloat162float(w[oW2 + lane * kH + j]), hj, h2a);
        h2b = fmaf(__bfloat162float(w[oW2 + (lane + 32) * kH + j]), hj, h2b);
    }
    float z = __bfloat162float(w[oW3 + lane]) * fmaxf(h2a, 0.f) + __bfloat162float(w[oW3 + lane + 32]) * fmaxf(h2b, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    z += P[oB3];
    return 1.f / (1.f + expf(-z));
}

// ---------------------------------------------------------------------------------- expand
// One warp per counted row of the wave.
__device__ void expand_row(const ResPtrs& p, int64_t g, int lane) {
    ResStatus* st = p.st;
    const int32_t jid = p.row_job[g];
    const int32_t r = p.row_local[g];
    const DJob dj = p.djobs[jid];
    const JobDesc jd = p.jobs[jid];
    const int32_t* crow = p.counts + jd.out_off + (int64_t)r * jd.n_cols;
    const int32_t minc = p.min_count;
    DFam* fp = p.fams + dj.fam;
    const DFam f = *fp;
    const int32_t* F = p.items + f.F_off;

    if (dj.kind == kJobLook) {
        const int32_t self = crow[jd.n_cols - 1];
        bool ext = false;
        for (int c = lane; c < jd.n_cols - 1; c += 32) ext |= crow[c] >= minc;
        ext = __any_sync(0xffffffffu, ext);
        if (lane == 0) {
            release_slot(p, dj.slot);
            if (dj.log >= 0) p.log_label[dj.log] = self >= minc ? 1.f : 0.f;
        }
        if (self >= minc) {
            if (lane == 0) atomicAdd(&st->hits, 1ull);
            if (!ext) {
                // head + whole tail: the tail is F[0..nT)
                const int32_t* head = p.heads + f.head_off;
                // emit head + F[0] ... F[nT-1]: treat F[0] as "t" and the rest as extra columns
                int32_t mx = -1;
                for (int q = lane; q < f.head_len; q += 32) mx = max(mx, head[q]);
                for (int q = lane; q < f.nT; q += 32) mx = max(mx, item_of(p, F[q]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                if (mx >= 0 && p.is_root[mx]) {
                    const int len = f.head_len + f.nT;
                    int32_t k = 0, off = 0;
                    if (lane == 0) {
                        k = atomicAdd(&st->mfi_n, 1);
                        off = atomicAdd(&st->mfi_item_n, len);
                    }
                    k = __shfl_sync(0xffffffffu, k, 0);
                    off = __shfl_sync(0xffffffffu, off, 0);
                    for (int q = lane; q < f.head_len; q += 32) p.mfi_items[off + q] = head[q];
                    for (int q = lane; q < f.nT; q += 32) p.mfi_items[off + f.head_len + q] = item_of(p, F[q]);
                    warp_sort_desc(p.mfi_items + off, len, lane);
                    if (lane == 0) {
                        p.mfi_off[k] = off;
                        p.mfi_len[k] = len;
                        p.mfi_sup[k] = len == 1 ? p.dense_freq[item_of(p, F[0])] : self;
                    }
                }
            }
            if (lane == 0) {
                release_slot(p, f.slot);
                fp->state = 2;
            }
        } else if (lane == 0) {
            fp->state = 0;
            const int32_t k = atomicAdd(&st->stack_n, 1);
            p.stack[k] = dj.fam;
        }
        return;
    }

    // a family row: the child X = head(P) + t
    const int32_t i = dj.r0 + r;
    const int32_t nT = f.nT, nF = f.nF;
    const int32_t t = F[i];
    const int32_t supc = crow[i];
    if (supc < minc) {   // cannot happen: t is in F(P)
        if (lane == 0) atomicExch(&st->error, kErrRow);
        finish_row(p, fp, lane);
        return;
    }
    // scan the row: extensions, equal-support items, tail.  Four loads in flight per lane;
    // `blocks` marks the column blocks of `bs` columns that hold an extension, so that the
    // later passes read only those.
    bool prune = false;
    int n_ext = 0, n_eq = 0, n_tail = 0;
    const int bs = column_block(nF);   // nF / bs <= 64, a multiple of 32
    unsigned long long blocks = 0;
    if (p.row_sum) {
        const RowSum rs = p.row_sum[g];
        n_ext = rs.n_ext; n_eq = rs.n_eq; n_tail = rs.n_tail; prune = rs.prune != 0; blocks = rs.blocks;
    }
    for (int c0 = 0; c0 < (p.row_sum ? 0 : nF); c0 += 128) {
        int32_t v4[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int c = c0 + 32 * u + lane;
            v4[u] = c < nF && c != i ? crow[c] : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int c = c0 + 32 * u + lane;
            const int32_t v = v4[u];
            const bool e = v >= minc;
            const bool in_tail = c > i && c < nT;
            const bool eq = e && v == supc;
            prune |= eq && !in_tail;
            if (e) blocks |= 1ull << (c / bs);
            n_ext += __popc(__ballot_sync(0xffffffffu, e));
            n_eq += __popc(__ballot_sync(0xffffffffu, eq));
            n_tail += __popc(__ballot_sync(0xffffffffu, e && !eq && in_tail));
        }
    }
    prune = __any_sync(0xffffffffu, prune);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) blocks |= __shfl_xor_sync(0xffffffffu, blocks, o);
    if (prune) {
        if (lane == 0) atomicAdd(&st->pep, 1ull);
        finish_row(p, fp, lane);
        return;
    }
    const int32_t* head = p.heads + f.head_off;
    const int n_rest = n_ext - n_eq;
    if (n_rest == 0 || n_tail == 0) {
        if (n_rest == 0) {
            // MFI: head + t + the equal-support items.  Gather their columns into the item
            // pool's scratch (the emit reads F[col]).
            int32_t eoff = 0;
            if (lane == 0 && n_eq) eoff = atomicAdd(&st->item_n, n_eq);
            eoff = __shfl_sync(0xffffffffu, eoff, 0);
            int32_t* ecols = p.items + eoff;
            int pos = 0;
            for (unsigned long long bm = n_eq ? blocks : 0ull; bm; bm &= bm - 1) {
                const int b0 = (__ffsll((long long)bm) - 1) * bs;
                for (int c0 = b0; c0 < min(nF, b0 + bs); c0 += 32) {
                    const int c = c0 + lane;
                    const int32_t v = c < nF && c != i ? crow[c] : -1;
                    const bool eq = v >= minc && v == supc;
                    const unsigned bal = __ballot_sync(0xffffffffu, eq);
                    if (eq) ecols[pos + __popc(bal & ((1u << lane) - 1u))] = c;
                    pos += __popc(bal);
                }
            }
            __syncwarp();
            warp_emit_mfi(p, head, f.head_len, item_of(p, t), ecols, n_eq, F, supc, lane);
        }
        finish_row(p, fp, lane);
        return;
    }
    // the child family: head' = head + t + eq; F' = sorted tail, then the other extensions
    const int head_len = f.head_len + 1 + n_eq;
    int32_t fid = 0, foff = 0, hoff = 0;
    if (lane == 0) {
        fid = atomicAdd(&st->fam_n, 1);
        foff = atomicAdd(&st->item_n, n_rest + n_tail);   // + staging for the unsorted tail
        hoff = atomicAdd(&st->head_n, head_len);
    }
    fid = __shfl_sync(0xffffffffu, fid, 0);
    foff = __shfl_sync(0xffffffffu, foff, 0);
    hoff = __shfl_sync(0xffffffffu, hoff, 0);
    int32_t* Fc = p.items + foff;              // n_rest entries
    int32_t* stage = p.items + foff + n_rest;  // n_tail tail columns in column order
    int32_t* hc = p.heads + hoff;
    for (int q = lane; q < f.head_len; q += 32) hc[q] = head[q];
    if (lane == 0) hc[f.head_len] = item_of(p, t);
    int pos_eq = 0, pos_tail = 0, pos_rest = 0;
    for (unsigned long long bm = blocks; bm; bm &= bm - 1) {
        const int b0 = (__ffsll((long long)bm) - 1) * bs;
        for (int c0 = b0; c0 < min(nF, b0 + bs); c0 += 32) {
            const int c = c0 + lane;
            const int32_t v = c < nF && c != i ? crow[c] : -1;
            const bool e = v >= minc;
            const bool eq = e && v == supc;
            const bool tl = e && !eq && c > i && c < nT;
            const bool rs = e && !eq && !tl;
            const unsigned lt = (1u << lane) - 1u;
            const unsigned bq = __ballot_sync(0xffffffffu, eq), bt = __ballot_sync(0xffffffffu, tl),
                           br = __ballot_sync(0xffffffffu, rs);
            if (eq) hc[f.head_len + 1 + pos_eq + __popc(bq & lt)] = item_of(p, F[c]);
            if (tl) stage[pos_tail + __popc(bt & lt)] = c;
            if (rs) Fc[n_tail + pos_rest + __popc(br & lt)] = F[c];
            pos_eq += __popc(bq);
            pos_tail += __popc(bt);
            pos_rest += __popc(br);
        }
    }
    __syncwarp();
    // tail sorted by (support, column), written as items to Fc[0 .. n_tail)
    if (n_tail <= 32) {
        unsigned long long key = ~0ull;
        if (lane < n_tail) {
            const int32_t c = stage[lane];
            key = ((unsigned long long)(uint32_t)crow[c] << 32) | (uint32_t)c;
        }
        // bitonic sort across the warp, ascending
        for (int k = 2; k <= 32; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
                const bool up = (lane & k) == 0;
                const bool lower = (lane & j) == 0;
                const bool take_min = (lower == up);
                key = take_min ? min(key, other) : max(key, other);
            }
        if (lane < n_tail) Fc[lane] = F[(int32_t)(key & 0xffffffffu)];
    } else if (n_tail <= 4096) {
        for (int a = lane; a < n_tail; a += 32) {
            const int32_t ca = stage[a];
            const unsigned long long ka = ((unsigned long long)(uint32_t)crow[ca] << 32) | (uint32_t)ca;
            int rank = 0;
            for (int b = 0; b < n_tail; b++) {
                const int32_t cb = stage[b];
                const unsigned long long kb = ((unsigned long long)(uint32_t)crow[cb] << 32) | (uint32_t)cb;
                rank += kb < ka;
            }
            Fc[rank] = F[ca];
        }
    } else {
        for (int a = lane; a < n_tail; a += 32) Fc[a] = F[stage[a]];
    }
    __syncwarp();
    // superset check: every itemset of the child's subtree lies inside head' + tail; when an
    // MFI of an earlier wave holds them all, none of those itemsets is a new maximal set
    if (p.sup_index && warp_covered(p, p.st->sup_done, hc, head_len, Fc, n_tail, lane)) {
        if (lane == 0) atomicAdd(&st->sup_pruned, 1ull);
        finish_row(p, fp, lane);
        return;
    }
    // base mask of the child
    int32_t cslot = -1, citem = -1;
    if (f.slot < 0 && f.item < 0) {
        citem = t;
    } else {
        if (lane == 0) cslot = pop_slot(p);
        cslot = __shfl_sync(0xffffffffu, cslot, 0);
        emit_mask(p, cslot, f.slot, f.item, t, 0, 0, f.W, lane);
    }
    // lookahead decision
    bool issue = false;
    float feat = 0.f;
    int log_idx = -1;
    const int list_len = n_tail + 1 + (f.item >= 0 ? 1 : 0);
    if (p.la_mode != 0 && n_tail >= 2 && list_len <= kMaxListLen) {
        // tail-pair filter: rows of tail items that are in this job's row range
        int pairs = 0, pairs_ok = 0;
        for (int a = 0; a < n_tail; a++) {
            const int32_t ra = stage[a];
            if (ra < dj.r0 || ra >= dj.r0 + dj.nr) continue;
            const int32_t* rowa = p.counts + jd.out_off + (int64_t)(ra - dj.r0) * jd.n_cols;
            for (int b = a + 1 + lane; b < n_tail; b += 32) {
                pairs++;
                pairs_ok += rowa[stage[b]] >= minc;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
            pairs_ok += __shfl_xor_sync(0xffffffffu, pairs_ok, o);
        }
        const bool filtered = pairs_ok < pairs;
        if (filtered && p.la_mode != 3) {
            if (lane == 0) atomicAdd(&st->skipped, 1ull);
        } else {
            issue = true;
            if (p.la_mode == 2 || p.log_on) {
                // features (same definitions as the host engine's)
                double mn = 1e30, mn2 = 1e30, mx = 0, sum = 0, sum2 = 0, logprod = 0;
                int gt90 = 0, gt99 = 0;
                for (int a = 0; a < n_tail; a++) {
                    const double rr = (double)crow[stage[a]] / (double)supc;
                    if (rr < mn) { mn2 = mn; mn = rr; } else if (rr < mn2) mn2 = rr;
                    mx = fmax(mx, rr);
                    sum += rr;
                    sum2 += rr * rr;
                    logprod += log(fmax(rr, 1e-12));
                    gt90 += rr > 0.9;
                    gt99 += rr > 0.99;
                }
                const int k = n_tail;
                const double mean = sum / k, var = fmax(0.0, sum2 / k - mean * mean);
                const double minc_d = max(1, minc);
                const bool top_child = f.top != 0;
                const double pf = pairs ? (double)pairs_ok / (double)pairs : 1.0;
                double v = 0.0;
                switch (lane) {
                    case 0: v = head_len / 16.0; break;
                    case 1: v = k / 32.0; break;
                    case 2: v = n_rest / 64.0; break;
                    case 3: v = (double)supc / (double)lmax(1, p.n_bits); break;
                    case 4: v = log2(1.0 + supc) / 24.0; break;
                    case 5: v = mn; break;
                    case 6: v = mean; break;
                    case 7: v = mx; break;
                    case 8: v = fmin(mn * supc / minc_d, 8.0) / 8.0; break;
                    case 9: v = exp(logprod); break;
                    case 10: v = fmax(-8.0, fmin(8.0, logprod + log(supc / minc_d))) / 8.0; break;
                    case 11: v = pf; break;
                    case 12: v = (n_rest - k) / 64.0; break;
                    case 13: v = minc_d / (double)lmax(1, p.n_bits); break;
                    case 14: v = fmin(supc / minc_d, 64.0) / 64.0; break;
                    case 15: v = sqrt(var); break;
                    case 16: v = k > 1 ? mn2 : mn; break;
                    case 17: v = (double)gt90 / k; break;
                    case 18: v = (double)gt99 / k; break;
                    case 19: v = log2(1.0 + k) / 6.0; break;
                    case 20: v = n_eq / 8.0; break;
                    case 21: v = nT / 64.0; break;
                    case 22: v = (double)i / (double)max(1, nT); break;
                    case 23: v = top_child ? 1.0 : 0.0; break;
                    default: v = 0.0;
                }
                feat = (float)v;
                if (p.la_mode == 2 && p.mlp_w) {
                    const float prob = warp_mlp(p, feat, lane);
                    if (prob < p.proposal_threshold) {
                        issue = false;
                        if (lane == 0) atomicAdd(&st->skipped, 1ull);
                    }
                }
            }
        }
    }
    if (issue && p.log_on) {
        if (lane == 0) log_idx = atomicAdd(&st->log_n, 1);
        log_idx = __shfl_sync(0xffffffffu, log_idx, 0);
        p.log_feat[(int64_t)log_idx * 32 + lane] = feat;
        if (lane == 0) p.log_label[log_idx] = 0.f;
    }
    // the child record
    if (lane == 0) {
        DFam ch;
        ch.slot = cslot; ch.item = citem; ch.head_off = hoff; ch.head_len = head_len;
        ch.F_off = foff; ch.nF = n_rest; ch.nT = n_tail; ch.sup = supc;
        ch.next_row = 0; ch.rows_done = 0; ch.state = issue ? 1 : 0; ch.top = 0;
        ch.W = f.W; ch.n = f.n;
        p.fams[fid] = ch;
    }
    if (issue) {
        int32_t ls = 0;
        if (lane == 0) ls = pop_slot(p);
        ls = __shfl_sync(0xffffffffu, ls, 0);
        // mask of head + tail: the child's base (the parent's sources and t) & the tail rows
        emit_mask(p, ls, f.slot, f.item, t, foff, n_tail, f.W, lane);
        if (lane == 0) {
            const int32_t q = atomicAdd(&st->look_n, 1);
            p.looks[q] = DLook{fid, ls, log_idx, 0};
            atomicAdd(&st->lookaheads, 1ull);
        }
    } else if (lane == 0) {
        const int32_t k = atomicAdd(&st->stack_n, 1);
        p.stack[k] = fid;
    }
    __syncwarp();
    finish_row(p, fp, lane);
}

__global__ void __launch_bounds__(256) k_res_expand(ResPtrs p) {
    phase_begin(&p.st->ph_s[kPhExpand]);
    const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (g < p.st->rows) expand_row(p, g, threadIdx.x & 31);
    phase_end(&p.st->ph_e[kPhExpand]);
}

// The masks the expand asked for, with the whole grid: every mask is cut into the same number
// of parts, at least two per block in all (one warp building a 1,000,000-bit mask alone would
// take a chain of ~250 dependent load rounds), strided over the blocks.
__device__ __forceinline__ void build_masks(const ResPtrs& p) {
    const int32_t n = p.st->n_mjobs;
    if (n <= 0) return;
    // a part holds at least a block's width (rows of a bitmap are below 2^31 transactions)
    const int32_t most = (int32_t)((p.W / 4 + 255) / 256);
    const int32_t parts = max(1, min(most, (int32_t)((2 * gridDim.x + n - 1) / n)));
    const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    const int64_t units = (int64_t)n * parts;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        const int32_t job = parts == 1 ? (int32_t)u : (int32_t)(u / parts), part = (int32_t)(u - (int64_t)job * parts);
        const MaskJob mj = p.mjobs[job];
        const int32_t W4 = mj.W >> 2, per = (W4 + parts - 1) / parts;
        const int32_t c0 = part * per, c1 = min(W4, c0 + per);
        uint4* d = reinterpret_cast<uint4*>(p.masks + (int64_t)mj.dst * p.W);
        const uint4* sm = mj.slot >= 0 ? reinterpret_cast<const uint4*>(p.masks + (int64_t)mj.slot * p.W) : nullptr;
        const uint4* si = mj.item >= 0 ? reinterpret_cast<const uint4*>(row_of(p, mj.item)) : nullptr;
        const uint4* st = mj.t >= 0 ? reinterpret_cast<const uint4*>(row_of(p, mj.t)) : nullptr;
        for (int32_t w = c0 + (int32_t)threadIdx.x; w < c1; w += blockDim.x) {
            uint4 v = ones;
            auto andv = [&](uint4 x) { v.x &= x.x; v.y &= x.y; v.z &= x.z; v.w &= x.w; };
            if (sm) andv(sm[w]);
            if (si) andv(__ldg(si + w));
            if (st) andv(__ldg(st + w));
            for (int q = 0; q < mj.n; q++) andv(__ldg(reinterpret_cast<const uint4*>(row_of(p, p.items[mj.off + q])) + w));
            d[w] = v;
        }
    }
}
__global__ void __launch_bounds__(256) k_build_masks(ResPtrs p) {
    phase_begin(&p.st->ph_s[kPhMasks]);
    build_masks(p);
    phase_end(&p.st->ph_e[kPhMasks]);
}

// Add the MFIs emitted since the last pack to the superset index: one warp per MFI, one
// atomicOr per item.  An MFI holding an item beyond the index is left out (it then prunes
// nothing); so are MFIs beyond the index's capacity.
__device__ void index_mfis(const ResPtrs& p) {
    if (!p.sup_index) return;
    const int32_t lo = p.st->sup_done;
    const int32_t hi = min(p.st->mfi_n, p.sup_words * 32);
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t k = lo + (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; k < hi; k += warps) {
        const int32_t off = p.mfi_off[k], len = p.mfi_len[k];
        bool ok = true;
        for (int q = lane; q < len; q += 32) {
            const int32_t x = p.mfi_items[off + q];
            ok &= x >= 0 && x < p.sup_items;
        }
        if (!__all_sync(0xffffffffu, ok)) continue;
        const uint32_t bit = 1u << (k & 31);
        for (int q = lane; q < len; q += 32)
            atomicOr(&p.sup_index[(int64_t)p.mfi_items[off + q] * p.sup_words + (k >> 5)], bit);
    }
}
__global__ void __launch_bounds__(256) k_index_mfis(ResPtrs p) {
    phase_begin(&p.st->ph_s[kPhMasks]);
    index_mfis(p);
    phase_end(&p.st->ph_e[kPhMasks]);
}

// Families waiting on the stack that an MFI found since their creation covers: a fresh
// family (no row handed out, not waiting on a lookahead) whose head and whole tail lie inside
// an indexed MFI is marked finished and its mask slot released; the pack then pops it without
// a job.  One warp per stack entry, from the top, over the entries the next waves take first.
__device__ void prune_stack(const ResPtrs& p) {
    if (!p.sup_index) return;
    ResStatus* st = p.st;
    const int32_t done = min(st->mfi_n, p.sup_words * 32);   // k_index_mfis has indexed these
    const int32_t n = st->stack_n;
    const int32_t depth = min(n, 4 * p.wave_rows);
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; k < depth; k += warps) {
        const int32_t fid = p.stack[n - 1 - k];
        DFam* fp = p.fams + fid;
        const DFam f = *fp;
        if (f.state != 0 || f.next_row != 0 || f.rows_done != 0 || f.top) continue;
        if (warp_covered(p, done, p.heads + f.head_off, f.head_len, p.items + f.F_off, f.nT, lane) && lane == 0) {
            fp->state = 2;
            release_slot(p, f.slot);
            atomicAdd(&st->sup_pruned, 1ull);
        }
    }
}
__global__ void __launch_bounds__(256) k_prune_stack(ResPtrs p) {
    phase_begin(&p.st->ph_s[kPhMasks]);
    prune_stack(p);
    phase_end(&p.st->ph_e[kPhMasks]);
}

// The family of the empty prefix (an n x n count block whose rows are its tail, nT = nF = n) is
// counted in its upper triangle.  This pass reads that once, 32 x 32 entries per block: it
// forms the expand's first pass over every row (`out`, cleared before) and writes the lower triangle
// where it matters, the entries of at least minc, and the diagonal.  6,156 items: 104 us as a
// mirror of the whole triangle and a pass over the rows, 51 us so.
__global__ void __launch_bounds__(256) k_top_finish(int32_t* __restrict__ M, int32_t n, const int32_t* __restrict__ diag,
                                                    int32_t minc, RowSum* __restrict__ out) {
    __shared__ int32_t tile[32][33];
    const int32_t bi = blockIdx.x, bj = blockIdx.y;   // rows bj, columns bi of the upper triangle
    if (bj > bi) return;
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int bs = column_block(n);   // a multiple of 32: a tile's columns lie in one block
    int any = 0;
    for (int k = ty; k < 32; k += 8) {
        const int32_t r = bj * 32 + k, c = bi * 32 + lane;
        const int32_t v = r < n && c < n && r < c ? M[(int64_t)r * n + c] : -1;
        tile[k][lane] = v;
        const bool e = v >= minc, eq = e && v == diag[r];
        const unsigned be = __ballot_sync(0xffffffffu, e), bq = __ballot_sync(0xffffffffu, eq);
        any |= be != 0;
        if (lane == 0 && be) {   // extensions of row r in its tail
            atomicAdd(&out[r].n_ext, __popc(be));
            if (bq) atomicAdd(&out[r].n_eq, __popc(bq));
            if (be & ~bq) atomicAdd(&out[r].n_tail, __popc(be & ~bq));
            atomicOr(&out[r].blocks, 1ull << (bi * 32 / bs));
        }
    }
    if (bi == bj && threadIdx.x < 32 && bi * 32 + lane < n) {
        const int32_t r = bi * 32 + lane;
        M[(int64_t)r * n + r] = diag[r];
    }
    if (!__syncthreads_or(any)) return;
    for (int k = ty; k < 32; k += 8) {
        const int32_t c = bi * 32 + k, r = bj * 32 + lane;   // row c of the lower triangle, column r
        const int32_t v = tile[lane][k];
        const bool e = v >= minc, eq = e && v == diag[c];
        const unsigned be = __ballot_sync(0xffffffffu, e), bq = __ballot_sync(0xffffffffu, eq);
        if (e) M[(int64_t)c * n + r] = v;
        if (lane == 0 && be) {   // extensions of row c outside its tail
            atomicAdd(&out[c].n_ext, __popc(be));
            if (bq) {
                atomicAdd(&out[c].n_eq, __popc(bq));
                atomicOr(&out[c].prune, 1);
            }
            atomicOr(&out[c].blocks, 1ull << (bj * 32 / bs));
        }
    }
}

// ---------------------------------------------------------------------------------- projection
// The subtree under a child {t} of the empty prefix counts only transactions that hold t.  When
// these are at most half of the database, the family is moved to a universe of its own: the
// rows of its F list are compressed to the set bits of t's row (bit k of a compressed row = the
// k-th transaction of t), and the family and all its descendants count there with an all-ones
// base, over sup(t) instead of N transactions.  Supports do not change.  It pays from a few tail
// rows on: a family reads its rows again for every one of them.
// Measured on the 6.3M-row dense database (267 items, minsup 6%): counting of the later waves
// 62 -> 25 ms and masks 1.8 -> 0.6 ms, for 2.2 ms of compression.  Lines at
// 3/4 and 19/20 of N instead of 1/2 moved the mine by less than its noise, as did 2 tail rows.
// The plan is made once, after the first wave, and leaves out the families that wait on a lookahead then
// (state 1): these and their subtrees count over all transactions.  With the learned proposal they are
// few (72 lookaheads in all at 12.5M rows, 42 ms a mine), with the tail-pair filter alone
// many (3,321, 100 ms).
constexpr int kProjMinTail = 4;        // tail rows from which a family is projected
constexpr int kProjTile = 64;          // words of a row per tile; rows are padded to this
constexpr int kProjGroups = 13;        // most groups of 32 items in a transposed chunk (odd)
constexpr int kProjWarps = 20;
constexpr int kProjWords = 1024;       // word by word: words of a row per block,
constexpr int kProjWordTiles = kProjWords / kProjTile;
constexpr int kProjThreads = kProjWords / 8;
constexpr int kProjCols = 4;           // and rows compressed between two barriers
// Columns per group of 32 items from which rows are compressed by transposing.  Its cost is per
// group with columns, the word-by-word way's per column: 2.2 and 5.6 ms at 21 columns a group (the
// 6.3M-row dense database), so they meet near 8.  The number of groups is only bounded here,
// by all groups or one per column (7 columns a group by that bound there), hence the lower line.
constexpr int kProjMinCols = 6;

// One block: the children of the empty prefix worth projecting, their places in the row table
// and the pool.
__global__ void __launch_bounds__(kPackThreads) k_proj_plan(ResPtrs p) {
    __shared__ int64_t sm64[4 * 33];
    const int tid = threadIdx.x;
    const int32_t n_fam = p.st->fam_n;
    int64_t cnt = 0, rows = 0, words = 0, groups = 0;
    const int32_t n_groups = (p.fams[0].nF + 31) / 32;
    for (int32_t base = 1; base < n_fam; base += kPackThreads) {
        const int32_t fid = base + tid;
        DFam f{};
        bool on = false;
        if (fid < n_fam) {
            f = p.fams[fid];
            on = f.state == 0 && f.slot < 0 && f.item >= 0 && f.nT >= kProjMinTail && 2 * (int64_t)f.sup <= f.n &&
                 64 * (int64_t)f.sup >= f.n;
        }
        const int64_t Wp = ((int64_t)f.sup + 2047) / 2048 * 64;
        int64_t v[4] = {on ? 1 : 0, on ? f.nF : 0, on ? f.nF * Wp : 0, on ? min(f.nF, n_groups) : 0}, ex[4], tot[4];
        block_scan<4>(v, ex, tot, sm64, true);
        if (on)
            p.pjobs[cnt + ex[0]] =
                PJob{fid, f.item, f.F_off, f.nF, (int32_t)Wp, (int32_t)(rows + ex[1]), f.sup, 0, words + ex[2]};
        cnt += tot[0];
        rows += tot[1];
        words += tot[2];
        groups += tot[3];
    }
    if (tid == 0) {
        p.st->pj_groups = groups;
        p.st->pj_n = (int32_t)cnt;
        p.st->pj_rows = (int32_t)rows;
        p.st->pj_words = words;
    }
}

// Set bits of every tile of every base row: half a warp per (family, tile).  Also the positions
// of the top family's items.
__global__ void __launch_bounds__(256) k_proj_count(ResPtrs p, int32_t n_pj) {
    const int64_t nt = p.W / kProjTile;
    const int lane = threadIdx.x & 31;
    if (p.pj_pos)
        for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < p.fams[0].nF; i += gridDim.x * blockDim.x)
            p.pj_pos[p.items[p.fams[0].F_off + i]] = i;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), half = (nt + 1) / 2;
    for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < n_pj * half; u += warps) {
        const int64_t k = u / half, tile = 2 * (u % half) + (lane >> 4);
        const uint4* row = reinterpret_cast<const uint4*>(row_of(p, p.pjobs[k].item));
        int32_t n = 0;
        if (tile < nt) {
            const uint4 x = __ldg(row + tile * (kProjTile / 4) + (lane & 15));
            n = __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
        }
#pragma unroll
        for (int o = 8; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
        if ((lane & 15) == 0 && tile < nt) p.pj_off[k * (nt + 1) + tile + 1] = n;
    }
}

// Bits before each tile: one warp per family.
__global__ void __launch_bounds__(256) k_proj_scan(ResPtrs p, int32_t n_pj) {
    const int64_t nt = p.W / kProjTile;
    const int lane = threadIdx.x & 31;
    const int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (k >= n_pj) return;
    int32_t* off = p.pj_off + k * (nt + 1);
    int32_t sum = 0;
    if (lane == 0) off[0] = 0;
    for (int64_t t0 = 1; t0 <= nt; t0 += 32) {
        const int64_t t = t0 + lane;
        int32_t x = t <= nt ? off[t] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (t <= nt) off[t] = sum + x;
        sum += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0 && sum != p.pjobs[k].sup) atomicExch(&p.st->error, kErrProjected);
}

// The row table's entries, zeros in the padding, and what the chosen way of compressing needs: the
// family's columns by position, or zeros in the words that two tiles share.  One block per family.
__global__ void __launch_bounds__(256) k_proj_init(ResPtrs p) {
    const PJob q = p.pjobs[blockIdx.x];
    const int64_t nt = p.W / kProjTile;
    const int32_t* off = p.pj_off + (int64_t)blockIdx.x * (nt + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = warp; c < q.nF; c += blockDim.x >> 5) {
        uint32_t* dst = p.pj_pool + q.woff + (int64_t)c * q.Wp;
        if (lane == 0) {
            p.vrows[q.row0 + c] = dst;
            p.vitem[q.row0 + c] = p.items[q.F_off + c];
        }
        if (!p.pj_tm)
            for (int64_t t = lane; t * kProjWordTiles < nt; t += 32) {
                const int32_t w = off[t * kProjWordTiles] >> 5;
                if (w < q.Wp) dst[w] = 0;
            }
        for (int32_t w = (q.sup >> 5) + lane; w < q.Wp; w += 32) dst[w] = 0;
    }
    if (!p.pj_tm) return;
    const int32_t n_g = p.pj_chunks * p.pj_gc;
    int16_t* inv = p.pj_inv + (int64_t)blockIdx.x * n_g * 32;
    for (int32_t i = threadIdx.x; i < n_g * 32; i += blockDim.x) inv[i] = -1;
    __syncthreads();
    for (int32_t c = threadIdx.x; c < q.nF; c += blockDim.x) inv[p.pj_pos[p.items[q.F_off + c]]] = (int16_t)c;
    __syncthreads();
    for (int32_t h = warp; h < p.pj_chunks; h += blockDim.x >> 5) {
        uint32_t m = 0;
        for (int32_t g = 0; g < p.pj_gc; g++) m |= (uint32_t)__any_sync(0xffffffffu, inv[(h * p.pj_gc + g) * 32 + lane] >= 0) << g;
        if (lane == 0) p.pj_gbits[(int64_t)blockIdx.x * p.pj_chunks + h] = m;
    }
}

// Transposes a 32 x 32 bit matrix in registers: bit i of v[j] becomes bit j of v[i].
__device__ __forceinline__ void transpose32(uint32_t (&v)[32]) {
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const uint32_t x = v[k], y = v[k + 16];
        v[k] = __byte_perm(x, y, 0x5410);
        v[k + 16] = __byte_perm(x, y, 0x7632);
    }
#pragma unroll
    for (int k = 0; k < 32; k++)
        if (!(k & 8)) {
            const uint32_t x = v[k], y = v[k + 8];
            v[k] = __byte_perm(x, y, 0x6240);
            v[k + 8] = __byte_perm(x, y, 0x7351);
        }
#pragma unroll
    for (int e = 2; e >= 0; e--) {
        const int sh = 1 << e;
        const uint32_t m = sh == 4 ? 0x0f0f0f0fu : sh == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int k = 0; k < 32; k++)
            if (!(k & sh)) {
                const uint32_t x = v[k], y = v[k + sh];
                v[k] = (x & m) | ((y << sh) & ~m);
                v[k + sh] = ((x >> sh) & m) | (y & ~m);
            }
    }
}

// The database with its transactions as rows: one block per 1,024 transactions and chunk of item
// groups, a warp per group.
__global__ void __launch_bounds__(32 * kProjGroups) k_proj_tm(ResPtrs p) {
    extern __shared__ uint32_t tm_out[];   // [1024][gc], one word of padding per 32 transactions
    const int gc = p.pj_gc, h = blockIdx.y, lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int64_t w0 = (int64_t)blockIdx.x * 32;
    const int32_t n0 = p.fams[0].nF, at = (h * gc + g) * 32;
    const int32_t* F = p.items + p.fams[0].F_off;
    uint32_t v[32];
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = at + j < n0 ? __ldg(row_of(p, F[at + j]) + w0 + lane) : 0;
    transpose32(v);
#pragma unroll
    for (int j = 0; j < 32; j++) tm_out[(32 * lane + j) * gc + g + lane] = v[j];
    __syncthreads();
    uint32_t* dst = p.pj_tm + ((int64_t)h * p.W + w0) * 32 * gc;
    for (int i = threadIdx.x; i < 1024 * gc; i += blockDim.x) dst[i] = tm_out[i + i / (32 * gc)];
}

// Compresses families' rows a tile of 2,048 transactions at a time.  The tile's transactions lie in
// shared memory as rows of item bits; a warp lists a family's transactions of the tile, and a
// thread picks the 32 of one compressed word, transposes their 32 x 32 bits in registers and stores
// the words of the group's columns.  Work is per word written, not per word read: about 500
// instructions for 32 words of up to 32 columns.  A tile writes the words whose first bit is its own; the
// up to 31 transactions that the last one lacks are fetched from the tiles behind.  Odd row lengths
// spread the gathered words over the banks.  Bound by the load/store pipe (list, gathers and scattered
// stores): 24 warps instead of 20, and the next family's words loaded ahead, changed nothing.
// Measured on the 6.3M-row dense database (267 items, minsup 6%): 2.1 ms and 0.14 ms for the
// transposed copy, against 5.6 ms word by word (k_proj_words).
__global__ void __launch_bounds__(32 * kProjWarps, 1) k_proj_rows(ResPtrs p, int32_t n_pj, int32_t parts) {
    extern __shared__ __align__(16) uint32_t pr_smem[];
    const int gc = p.pj_gc, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nt = p.W / kProjTile;
    constexpr int T = kProjTile * 32, kZero = T + 32 * kProjWarps;   // staged rows: the tile, each warp's 32, a zero row
    uint32_t* rows = pr_smem;
    uint16_t* list = reinterpret_cast<uint16_t*>(pr_smem + (((kZero + 1) * gc + 3) & ~3)) + warp * (T + 32);
    for (int i = threadIdx.x; i < gc; i += blockDim.x) rows[kZero * gc + i] = 0;
    for (int64_t u = blockIdx.x; u < nt * p.pj_chunks * parts; u += gridDim.x) {
        const int part = (int)(u % parts), h = (int)(u / parts % p.pj_chunks);
        const int64_t tile = u / parts / p.pj_chunks;
        const uint32_t* tm = p.pj_tm + (int64_t)h * p.W * 32 * gc;
        __syncthreads();
        {
            const uint4* src = reinterpret_cast<const uint4*>(tm + tile * T * gc);
            for (int i = threadIdx.x; i < T / 4 * gc; i += blockDim.x) reinterpret_cast<uint4*>(rows)[i] = __ldg(src + i);
        }
        __syncthreads();
        for (int32_t k = part + parts * warp; k < n_pj; k += parts * kProjWarps) {
            const uint32_t gbits = p.pj_gbits[(int64_t)k * p.pj_chunks + h];
            if (!gbits) continue;
            const PJob q = p.pjobs[k];
            const int32_t off0 = p.pj_off[(int64_t)k * (nt + 1) + tile], off1 = p.pj_off[(int64_t)k * (nt + 1) + tile + 1];
            const int32_t wa = (off0 + 31) >> 5, n_w = min((off1 + 31) >> 5, q.Wp) - wa;
            if (n_w <= 0) continue;
            const uint32_t* base = row_of(p, q.item);
            // the family's transactions, as offsets into `rows`, from list[off0 % 32] on
            const int32_t lead = off0 & 31;
            const uint2 m2 = __ldg(reinterpret_cast<const uint2*>(base + tile * kProjTile) + lane);
            int32_t n = __popc(m2.x) + __popc(m2.y), pre = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o) pre += y;
            }
            pre += lead - n;
            for (uint32_t m = m2.x; m; m &= m - 1) list[pre++] = (uint16_t)((64 * lane + __ffs(m) - 1) * gc);
            for (uint32_t m = m2.y; m; m &= m - 1) list[pre++] = (uint16_t)((64 * lane + 31 + __ffs(m)) * gc);
            const int32_t end = lead + off1 - off0;                       // list entries used
            const int32_t need = min(32 * (wa + n_w), q.sup) - off1;      // transactions to fetch from behind
            for (int32_t i = lane; end + i < 32 * ((end + 31) >> 5); i += 32)
                list[end + i] = (uint16_t)((i < need ? T + 32 * warp + i : kZero) * gc);
            uint32_t* far = rows + (T + 32 * warp) * gc;   // the fetched transactions' rows
            int32_t got = 0;
            for (int64_t w = (tile + 1) * kProjTile; got < need && w < p.W; w += 32) {   // W is a multiple of 64
                uint32_t m = __ldg(base + w + lane);
                const int32_t c = __popc(m);
                int32_t at = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t y = __shfl_up_sync(0xffffffffu, at, o);
                    if (lane >= o) at += y;
                }
                const int32_t all = __shfl_sync(0xffffffffu, at, 31);
                at += got - c;
                for (; m && at < need; m &= m - 1, at++) far[at] = (uint32_t)(32 * (w + lane) + __ffs(m) - 1);
                got += all;
            }
            if (need > 0) {
                __syncwarp();
                const uint32_t t = lane < min(need, got) ? far[lane] : 0;
                __syncwarp();
#pragma unroll 4
                for (int i = 0; i < need * gc; i += 32) {
                    const int e = min((i + lane) / gc, 31);
                    const int64_t te = __shfl_sync(0xffffffffu, t, e);
                    if (i + lane < need * gc) far[i + lane] = __ldg(tm + te * gc + (i + lane - e * gc));
                }
            }
            __syncwarp();
            const int32_t total = __popc(gbits) * n_w;
            const int32_t first = 32 * (wa - (off0 >> 5));                // list entry of word wa's first bit
            for (int32_t e = lane; e < total; e += 32) {
                const int32_t gi = e / n_w, w = e - gi * n_w;
                uint32_t gm = gbits;
                for (int i = 0; i < gi; i++) gm &= gm - 1;
                const int g = __ffs(gm) - 1;
                const uint4* idx = reinterpret_cast<const uint4*>(list + first + 32 * w);
                const uint32_t* src = rows + g;
                uint32_t v[32];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint4 x = idx[t];
                    v[8 * t] = src[x.x & 0xffffu];
                    v[8 * t + 1] = src[x.x >> 16];
                    v[8 * t + 2] = src[x.y & 0xffffu];
                    v[8 * t + 3] = src[x.y >> 16];
                    v[8 * t + 4] = src[x.z & 0xffffu];
                    v[8 * t + 5] = src[x.z >> 16];
                    v[8 * t + 6] = src[x.w & 0xffffu];
                    v[8 * t + 7] = src[x.w >> 16];
                }
                transpose32(v);
                const uint4* cols = reinterpret_cast<const uint4*>(p.pj_inv + ((int64_t)k * p.pj_chunks * gc + h * gc + g) * 32);
                uint32_t* dst = p.pj_pool + q.woff + wa + w;
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint4 x = __ldg(cols + t);
                    const uint32_t c4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int32_t c = (int16_t)(c4[i >> 1] >> (16 * (i & 1)));
                        if (c >= 0) dst[(int64_t)c * q.Wp] = v[8 * t + i];
                    }
                }
            }
            __syncwarp();
        }
    }
}

// The same word by word, for families whose few columns are spread over many items: the rows of
// one (family, kProjWords words) per block.  A thread owns 8 words of the tile and
// keeps their five move masks (the parallel-suffix compress of H. S. Warren, Hacker's Delight,
// 7-4) in registers for all rows; per row it loads its 32 bytes, compresses each word and
// appends it to a bit run that it flushes word by word into the row's shared output, which
// then goes out whole.  Tiles of all families at one place run together, so that the database's
// rows are read from L2.
__global__ void __launch_bounds__(kProjThreads, 4) k_proj_words(ResPtrs p, int32_t n_pj) {
    __shared__ uint32_t out[kProjCols][kProjWords + 2];
    __shared__ int32_t s_warp[kProjThreads / 32];
    const int64_t nt = p.W / kProjTile, nw = (nt + kProjWordTiles - 1) / kProjWordTiles;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kProjCols * (kProjWords + 2); i += kProjThreads) (&out[0][0])[i] = 0;
    for (int64_t u = blockIdx.x; u < n_pj * nw; u += gridDim.x) {
        const int64_t tile = u / n_pj, k = u % n_pj;
        const PJob q = p.pjobs[k];
        const int32_t* off = p.pj_off + k * (nt + 1);
        const int32_t t0 = off[tile * kProjWordTiles], bits = off[min((tile + 1) * kProjWordTiles, nt)] - t0;
        if (bits == 0) continue;
        const int64_t w4 = tile * (kProjWords / 4) + tid * 2;   // this thread's words, 16 bytes each
        const bool in = w4 * 4 < p.W;                          // W is a multiple of 64 words
        uint32_t m[8], mv[8][5];
        int32_t n_of[8], n_all = 0;
        {
            const uint4* row = reinterpret_cast<const uint4*>(row_of(p, q.item));
            const uint4 a = in ? __ldg(row + w4) : make_uint4(0, 0, 0, 0), b = in ? __ldg(row + w4 + 1) : make_uint4(0, 0, 0, 0);
            m[0] = a.x; m[1] = a.y; m[2] = a.z; m[3] = a.w; m[4] = b.x; m[5] = b.y; m[6] = b.z; m[7] = b.w;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint32_t x = m[i], mk = ~x << 1;
            n_of[i] = __popc(x);
            n_all += n_of[i];
#pragma unroll
            for (int s = 0; s < 5; s++) {
                uint32_t mp = mk ^ (mk << 1);
                mp ^= mp << 2;
                mp ^= mp << 4;
                mp ^= mp << 8;
                mp ^= mp << 16;
                mv[i][s] = mp & x;
                x = (x ^ mv[i][s]) | (mv[i][s] >> (1 << s));
                mk &= ~mp;
            }
        }
        int32_t pre = n_all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += y;
        }
        if (lane == 31) s_warp[warp] = pre;
        __syncthreads();
        pre -= n_all;
        for (int w = 0; w < warp; w++) pre += s_warp[w];
        const int32_t start = (t0 & 31) + pre;          // this thread's first bit in the tile's output
        const int32_t n_words = ((t0 & 31) + bits + 31) >> 5;
        for (int c0 = 0; c0 < q.nF; c0 += kProjCols) {
            const int nc = min(kProjCols, q.nF - c0);
            for (int c = 0; c < nc; c++) {
                const uint4* row = reinterpret_cast<const uint4*>(row_of(p, p.items[q.F_off + c0 + c]));
                uint32_t x[8];
                const uint4 a = in ? __ldg(row + w4) : make_uint4(0, 0, 0, 0), b = in ? __ldg(row + w4 + 1) : make_uint4(0, 0, 0, 0);
                x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
                uint32_t lo = 0;
                int32_t n = start & 31, at = start >> 5;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    uint32_t y = x[i] & m[i];
#pragma unroll
                    for (int s = 0; s < 5; s++) {
                        const uint32_t t = y & mv[i][s];
                        y = (y ^ t) | (t >> (1 << s));
                    }
                    lo |= y << n;
                    const uint32_t hi = __funnelshift_l(y, 0u, n);
                    n += n_of[i];
                    if (n >= 32) {
                        if (lo) atomicOr(&out[c][at], lo);
                        lo = hi;
                        n -= 32;
                        at++;
                    }
                }
                if (lo) atomicOr(&out[c][at], lo);
            }
            __syncthreads();
            for (int i = tid; i < nc * n_words; i += kProjThreads) {
                const int c = i / n_words, w = i - c * n_words;
                const uint32_t v = out[c][w];
                out[c][w] = 0;
                uint32_t* dst = p.pj_pool + q.woff + (int64_t)(c0 + c) * q.Wp + (t0 >> 5) + w;
                // a word that a neighbouring tile writes too was zeroed before
                if ((w == 0 && (t0 & 31)) || (w == n_words - 1 && ((t0 + bits) & 31))) {
                    if (v) atomicOr(dst, v);
                } else {
                    *dst = v;
                }
            }
            __syncthreads();
        }
    }
}

// Dynamic shared memory of k_proj_tm and k_proj_rows at `gc` groups per chunk.
constexpr int proj_tm_smem(int gc) { return (1024 * gc + 32) * 4; }
constexpr int proj_rows_smem(int gc) {
    return ((((kProjTile * 32 + 32 * kProjWarps + 1) * gc + 3) & ~3) * 4) + kProjWarps * (kProjTile * 32 + 32) * 2;
}

// The families move to their universes: one block per family.
__global__ void __launch_bounds__(128) k_proj_commit(ResPtrs p) {
    const PJob q = p.pjobs[blockIdx.x];
    for (int c = threadIdx.x; c < q.nF; c += blockDim.x) p.items[q.F_off + c] = p.n_base + q.row0 + c;
    if (threadIdx.x == 0) {
        DFam* f = p.fams + q.fam;
        f->slot = -1;
        f->item = -1;
        f->W = q.Wp;
        f->n = q.sup;
    }
}

// The search's initial state, one launch: parts of pinned host memory to their places on the device
// (in place of a copy each).  Sizes are rounded up to 16 bytes on both sides.
struct SetupPart {
    const uint4* src;
    uint4* dst;
    int64_t n16;
};
struct SetupParts {
    SetupPart part[16];
    int32_t n;
};
__global__ void __launch_bounds__(256) k_res_setup(SetupParts s) {   // blockIdx.y: the part
    const SetupPart q = s.part[blockIdx.y];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < q.n16; i += (int64_t)gridDim.x * blockDim.x)
        q.dst[i] = q.src[i];
}

// ---------------------------------------------------------------------------------- device loop
// Searches over short rows are chains of small waves: a 10,000-row dense database takes eight
// waves of about 10 us of counting, and each cost a launch of every phase, a clear, a status copy
// and a host wait, 85 us.  This kernel runs such waves back to back with its whole grid resident
// (cooperative launch): block 0 packs, then all blocks count, expand and build masks, with a grid
// barrier after each.  A wave of more than kLoopMaxWork, and one that needs larger pools, is left
// to the host.  Measured, a call: 10,000-row dense mine 0.70 -> 0.48 ms (31 us a wave), 2M-row one 0.45 ->
// 0.35 ms.
constexpr int kLoopThreads = 512;
constexpr int kLoopMaxWords = 4096;     // rows of the databases that take it;
constexpr int kLoopDenseWords = 1 << 16; // of dense ones (minimum support at least 1/64 of the transactions)
constexpr int kLoopCols = 8;            // columns a warp counts at once
constexpr uint32_t kLoopSpin = 1u << 22;

// All blocks of the grid (`target` arrivals); false when the wait expired.  The fences order the
// phases' plain loads and stores, as those of a grid-wide sync do.
__device__ __forceinline__ bool grid_barrier(uint32_t* bar, uint32_t target) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        uint32_t k = 0;
        while (*(volatile uint32_t*)bar < target && ++k < kLoopSpin) __nanosleep(20);
        s_ok = k < kLoopSpin;
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
}

// Word slices of a wave's rows: enough for two tasks per warp, of at least 256 words.
__device__ __forceinline__ int32_t loop_slices(const ResPtrs& p) {
    const int64_t tasks = (int64_t)max(p.st->rows, 1) * max((p.st->max_cols + kLoopCols - 1) / kLoopCols, 1);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    return (int32_t)lmax(1, lmin((2 * warps + tasks - 1) / tasks, p.W / 256));
}

// Counts of the wave's rows: one warp per row, kLoopCols columns and word slice (several slices add
// into cleared counts).  Masks, lists and counts are written during this kernel, so only bitmap
// rows are read through the read-only path.
__device__ __forceinline__ void loop_count(const ResPtrs& p, int32_t slices) {
    const int32_t rows = p.st->rows, chunks = (p.st->max_cols + kLoopCols - 1) / kLoopCols;
    const int lane = threadIdx.x & 31;
    const int32_t warps = gridDim.x * (blockDim.x >> 5);
    const int64_t tasks = (int64_t)rows * chunks;
    for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < tasks * slices; u += warps) {
        const int32_t slice = (int32_t)(u / tasks);
        const int64_t t = u - slice * tasks;
        const int32_t g = (int32_t)(t / chunks), c0 = (int32_t)(t % chunks) * kLoopCols;
        const JobDesc jd = p.jobs[p.row_job[g]];
        if (c0 >= jd.n_cols) continue;
        const RowDesc rd = p.rows[g];
        const uint4* bm = jd.base_slot >= 0 ? reinterpret_cast<const uint4*>(p.masks + (int64_t)jd.base_slot * p.W) : nullptr;
        const uint4* bi = jd.base_item >= 0 ? reinterpret_cast<const uint4*>(row_of(p, jd.base_item)) : nullptr;
        const uint4* rm = rd.slot >= 0 ? reinterpret_cast<const uint4*>(p.masks + (int64_t)rd.slot * p.W) : nullptr;
        const uint4* ri = rd.item >= 0 ? reinterpret_cast<const uint4*>(row_of(p, rd.item)) : nullptr;
        const uint4* col[kLoopCols];   // null: all ones
        int32_t acc[kLoopCols];
#pragma unroll
        for (int k = 0; k < kLoopCols; k++) {
            const int32_t c = min(c0 + k, jd.n_cols - 1);
            const int32_t id = c == jd.self_col ? -1 : p.items[jd.col_off + c];
            col[k] = id >= 0 ? reinterpret_cast<const uint4*>(row_of(p, id)) : nullptr;
            acc[k] = 0;
        }
        const int32_t W4 = jd.words >> 2, per = (W4 + slices - 1) / slices;
        for (int32_t w = slice * per + lane; w < min(W4, (slice + 1) * per); w += 32) {
            uint4 v = make_uint4(~0u, ~0u, ~0u, ~0u);
            auto andv = [&](uint4 x) { v.x &= x.x; v.y &= x.y; v.z &= x.z; v.w &= x.w; };
            if (bm) andv(bm[w]);
            if (bi) andv(__ldg(bi + w));
            if (rm) andv(rm[w]);
            if (ri) andv(__ldg(ri + w));
#pragma unroll
            for (int k = 0; k < kLoopCols; k++) {
                const uint4 x = col[k] ? __ldg(col[k] + w) : make_uint4(~0u, ~0u, ~0u, ~0u);
                acc[k] += __popc(v.x & x.x) + __popc(v.y & x.y) + __popc(v.z & x.z) + __popc(v.w & x.w);
            }
        }
        int32_t mine = 0;
#pragma unroll
        for (int k = 0; k < kLoopCols; k++) {
            const int32_t n = __reduce_add_sync(0xffffffffu, acc[k]);
            if (lane == k) mine = n;
        }
        if (lane < kLoopCols && c0 + lane < jd.n_cols) {
            int32_t* out = p.counts + jd.out_off + (int64_t)p.row_local[g] * jd.n_cols + c0 + lane;
            if (slices == 1) *out = mine;
            else if (mine) atomicAdd(out, mine);
        }
    }
}

__global__ void __launch_bounds__(kLoopThreads, 1) k_res_loop(ResPtrs p, uint32_t* bar) {
    ResStatus* st = p.st;
    uint32_t arrived = 0;
    bool first = true;
    while (true) {
        if (blockIdx.x == 0) {
            // a launch gives the device back after max_launch_ns; the next one continues
            const bool late = !first && globaltimer() - st->launch_t0 > p.max_launch_ns;
            if (__syncthreads_or(late)) {
                if (threadIdx.x == 0) st->loop_go = 2;
            } else {
                res_pack<kLoopThreads, true>(p);
                __syncthreads();
                if (threadIdx.x == 0) st->loop_go = st->jobs > 0 && st->small && !st->error ? 1 : 0;
            }
        }
        first = false;
        bool ok = grid_barrier(bar, arrived += gridDim.x);
        if (!ok || st->loop_go != 1) {
            if (!ok && threadIdx.x == 0) atomicExch(&st->error, kErrWait);
            if (blockIdx.x == 0) publish_status(p);
            return;
        }
        phase_begin(&st->ph_s[kPhLop3]);
        const int32_t slices = loop_slices(p);
        if (slices > 1) {
            const int64_t n = st->out_total;
            for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
                p.counts[i] = 0;
            if (!grid_barrier(bar, arrived += gridDim.x)) {
                if (threadIdx.x == 0) atomicExch(&st->error, kErrWait);
                if (blockIdx.x == 0) publish_status(p);
                return;
            }
        }
        loop_count(p, slices);
        phase_end(&st->ph_e[kPhLop3]);
        ok = grid_barrier(bar, arrived += gridDim.x);
        if (ok) {
            phase_begin(&st->ph_s[kPhExpand]);
            const int32_t rows = st->rows;
            const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
            for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < rows; g += warps)
                expand_row(p, g, threadIdx.x & 31);
            phase_end(&st->ph_e[kPhExpand]);
            ok = grid_barrier(bar, arrived += gridDim.x);
        }
        if (ok) {
            phase_begin(&st->ph_s[kPhMasks]);
            build_masks(p);
            phase_end(&st->ph_e[kPhMasks]);
            if (blockIdx.x == 0 && threadIdx.x == 0) st->waves += 1;
            ok = grid_barrier(bar, arrived += gridDim.x);
        }
        if (!ok) {
            if (threadIdx.x == 0) atomicExch(&st->error, kErrWait);
            if (blockIdx.x == 0) publish_status(p);
            return;
        }
    }
}

// ---------------------------------------------------------------------------------- graph loop
// The wave loop as a graph: a conditional WHILE node whose body is
//   pack -> zero the count block -> persistent counters -> persistent expand -> control.
// Every kernel reads its arguments from the ResArgs record and its sizes from the status
// record, so the launch shapes are fixed.  The control kernel ends the loop when the search
// is done, when the pack asks for larger pools or reports an error, or after the slice's
// wave / time limit; the host then reads the status once.

// Zero the wave's count block and the persistent counters' tile counters.
__global__ void __launch_bounds__(256) k_res_zero(const ResArgs* __restrict__ args) {
    ResStatus* st = args->p.st;
    int32_t* counts = args->p.counts;
    phase_begin(&st->ph_s[kPhZero]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->next3 = 0;
        st->next1 = 0;
        st->next_gr = 0;
    }
    const int64_t n = st->out_total;
    const int64_t n4 = n >> 2;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int4* c4 = reinterpret_cast<int4*>(counts);
    for (int64_t i = i0; i < n4; i += stride) c4[i] = make_int4(0, 0, 0, 0);
    for (int64_t i = (n4 << 2) + i0; i < n; i += stride) counts[i] = 0;
    phase_end(&st->ph_e[kPhZero]);
}

__global__ void __launch_bounds__(256) k_res_expand_g(const ResArgs* __restrict__ args) {
    const ResPtrs p = args->p;
    const int lane = threadIdx.x & 31;
    phase_begin(&p.st->ph_s[kPhExpand]);
    const int32_t rows = p.st->rows;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < rows; g += warps) expand_row(p, g, lane);
    phase_end(&p.st->ph_e[kPhExpand]);
}

__global__ void __launch_bounds__(256) k_build_masks_g(const ResArgs* __restrict__ args) {
    const ResPtrs p = args->p;
    phase_begin(&p.st->ph_s[kPhMasks]);
    build_masks(p);
    phase_end(&p.st->ph_e[kPhMasks]);
}

__global__ void __launch_bounds__(256) k_index_mfis_g(const ResArgs* __restrict__ args) {
    phase_begin(&args->p.st->ph_s[kPhMasks]);
    index_mfis(args->p);
    phase_end(&args->p.st->ph_e[kPhMasks]);
}
__global__ void __launch_bounds__(256) k_prune_stack_g(const ResArgs* __restrict__ args) {
    phase_begin(&args->p.st->ph_s[kPhMasks]);
    prune_stack(args->p);
    phase_end(&args->p.st->ph_e[kPhMasks]);
}

__global__ void k_res_control(const ResArgs* __restrict__ args, cudaGraphConditionalHandle h) {
    if (threadIdx.x != 0) return;
    ResStatus* st = args->p.st;
    const bool progressed = st->jobs > 0;
    if (progressed) st->waves += 1;
    const bool go = progressed && !st->error && !st->grow && !st->starved && st->waves < args->p.wave_limit &&
                    globaltimer() - st->launch_t0 < args->p.max_launch_ns;
    cudaGraphSetConditional(h, go ? 1u : 0u);
}

// ------------------------------------------------------------------------ output order
// The MFIs leave the device in their output order: descending support, then item lists
// (each in descending order) compared lexicographically, larger first.  The sort key packs
// the support and the two largest items in as few bits as the database needs, complemented so
// that an ascending radix sort gives that order; where 64 bits do not hold them (i_bits = 0), 32
// bits of support and the largest item.  Lists whose keys are equal are finished on the host.
struct MfiKey {
    int32_t s_bits, i_bits;
    __host__ __device__ int bits() const { return i_bits ? s_bits + 2 * i_bits : 64; }
};
__device__ __forceinline__ uint64_t mfi_key(MfiKey f, const int32_t* items, int32_t l, uint32_t sup) {
    int32_t a = -1, b = -1;   // the two largest items
    for (int32_t q = 0; q < l; q++) {
        const int32_t x = items[q];
        if (x > a) {
            b = a;
            a = x;
        } else if (x > b) {
            b = x;
        }
    }
    if (!f.i_bits) return ((uint64_t)(0xFFFFFFFFu - sup) << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)(a + 1));
    const uint64_t im = (1ull << f.i_bits) - 1, smax = (1ull << f.s_bits) - 1;
    return ((smax - sup) << (2 * f.i_bits)) | ((im - (uint64_t)(a + 1)) << f.i_bits) | (im - (uint64_t)(b + 1));
}

__global__ void __launch_bounds__(256) k_mfi_keys(const int32_t* __restrict__ off, const int32_t* __restrict__ len,
                                                  const int32_t* __restrict__ sup, const int32_t* __restrict__ items,
                                                  int32_t n, MfiKey f, uint64_t* __restrict__ keys,
                                                  int32_t* __restrict__ idx) {
    for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        keys[k] = mfi_key(f, items + off[k], len[k], (uint32_t)sup[k]);
        idx[k] = k;
    }
}

// Few MFIs (at most kFinishMax): one block forms the keys, sorts, places lengths, supports and items
// in output order and hands them to pinned host memory, in place of six launches and three
// copies (1,612 MFIs: 57 us of read-back in all against 75).
// Up to 1,024 MFIs are sorted one to a thread (129 MFIs: 31 us with four, 17 with one).
constexpr int kFinishThreads = 1024, kFinishMax = kFinishThreads * 4;
constexpr int64_t kFinishMaxItems = 1 << 16;
template <int kFinishItems>
__global__ void __launch_bounds__(kFinishThreads) k_mfi_finish(const int32_t* off, const int32_t* len, const int32_t* sup,
                                                               const int32_t* items, int32_t n, int64_t ni, MfiKey f,
                                                               uint4* dev, uint4* host) {
    typedef cub::BlockRadixSort<uint64_t, kFinishThreads, kFinishItems, int32_t> Sort;
    constexpr int kMax = kFinishThreads * kFinishItems;
    __shared__ union {
        typename Sort::TempStorage sort;
        int32_t scan[33];
        struct { int32_t from[kMax], to[kMax]; } g;   // each MFI's place before and after
    } sm;
    // keys, lengths, supports, items: one after the other, as the host reads them
    uint64_t* d_key = reinterpret_cast<uint64_t*>(dev);
    int32_t* d_len = reinterpret_cast<int32_t*>(d_key + n);
    int32_t* d_sup = d_len + n;
    int32_t* d_items = d_sup + n;
    const int tid = threadIdx.x;
    uint64_t key[kFinishItems];
    int32_t idx[kFinishItems];
#pragma unroll
    for (int q = 0; q < kFinishItems; q++) {
        const int32_t k = tid * kFinishItems + q;
        idx[q] = k;
        key[q] = k < n ? mfi_key(f, items + off[k], len[k], (uint32_t)sup[k]) : ~0ull;
    }
    Sort(sm.sort).Sort(key, idx, 0, f.bits());   // stable: the padding (all ones) stays last
    __syncthreads();
    int32_t l[kFinishItems], v[1] = {0}, ex[1], tot[1];
#pragma unroll
    for (int q = 0; q < kFinishItems; q++) {
        l[q] = tid * kFinishItems + q < n ? len[idx[q]] : 0;
        v[0] += l[q];
    }
    block_scan<1>(v, ex, tot, sm.scan, true);
    int32_t o = ex[0];
#pragma unroll
    for (int q = 0; q < kFinishItems; q++) {
        const int32_t k = tid * kFinishItems + q;
        if (k < n) {
            d_key[k] = key[q];
            d_len[k] = l[q];
            d_sup[k] = sup[idx[q]];
            sm.g.from[k] = idx[q];
            sm.g.to[k] = o;
            o += l[q];
        }
    }
    __syncthreads();
    // items: eight lanes per MFI
    for (int32_t k = tid >> 3; k < n; k += kFinishThreads >> 3) {
        const int32_t m = sm.g.from[k], src = off[m], ll = len[m], dst = sm.g.to[k];
        for (int32_t x = tid & 7; x < ll; x += 8) d_items[dst + x] = items[src + x];
    }
    __syncthreads();
    const int64_t n16 = ((int64_t)n * 16 + ni * 4 + 15) >> 4;
    for (int64_t i = tid; i < n16; i += kFinishThreads) host[i] = dev[i];
}

// Lengths and supports in sorted order.
__global__ void __launch_bounds__(256) k_mfi_permute(const int32_t* __restrict__ idx, const int32_t* __restrict__ len,
                                                     const int32_t* __restrict__ sup, int32_t n,
                                                     int32_t* __restrict__ len_o, int32_t* __restrict__ sup_o) {
    for (int32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int32_t k = idx[q];
        len_o[q] = len[k];
        sup_o[q] = sup[k];
    }
}

// Item lists in sorted order: one warp per MFI.
__global__ void __launch_bounds__(256) k_mfi_gather(const int32_t* __restrict__ idx, const int32_t* __restrict__ off,
                                                    const int32_t* __restrict__ items, const int32_t* __restrict__ off_o,
                                                    const int32_t* __restrict__ len_o, int32_t n,
                                                    int32_t* __restrict__ items_o) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < n; q += warps) {
        const int32_t* src = items + off[idx[q]];
        int32_t* dst = items_o + off_o[q];
        for (int32_t x = lane; x < len_o[q]; x += 32) dst[x] = src[x];
    }
}

// ---------------------------------------------------------------------------------- host
struct Pool {
    void* p = nullptr;
    size_t bytes = 0;
};

int grow(Pool& b, size_t need, cudaStream_t s, size_t min_bytes = 1 << 16) {
    if (need <= b.bytes && b.p) return TFIM_OK;
    size_t cap = std::max<size_t>(need + need / 2, min_bytes);
    void* np = nullptr;
    TFIM_TRY(dev_alloc(&np, cap, s));
    if (b.p && b.bytes) TFIM_CUDA(cudaMemcpyAsync(np, b.p, b.bytes, cudaMemcpyDeviceToDevice, s));
    dev_free(b.p, s);
    b.p = np;
    b.bytes = cap;
    return TFIM_OK;
}

// The captured wave loop.  Its launches read ResArgs at `args` and sizes from the status
// record at `status`; it is rebuilt when either moves or the set of counters changes.
struct WaveGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const void* args = nullptr;
    const void* status = nullptr;
    int with_proj = -1;
    void release() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        args = status = nullptr;
        with_proj = -1;
    }
};

int build_wave_graph(WaveGraph& G, const ResArgs* d_args, ResStatus* d_status, bool with_proj, const int64_t* red_off,
                     const int32_t* red_items, cudaStream_t s) {
    G.release();
    int sm = 148, dev = 0, occ3 = 1, occ1 = 1, occp = 1, occe = 1, occg = 1;
    TFIM_CUDA(cudaGetDevice(&dev));
    TFIM_CUDA(cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev));
    TFIM_TRY(persistent_occupancy(&occ3, &occ1, &occp));
    TFIM_TRY(configure_pk_kernel());
    TFIM_TRY(occupancy_gram(&occg));
    TFIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occe, k_res_expand_g, 256, 0));
    TFIM_CUDA(cudaGraphCreate(&G.graph, 0));
    cudaGraphConditionalHandle h;
    TFIM_CUDA(cudaGraphConditionalHandleCreate(&h, G.graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    TFIM_CUDA(cudaGraphAddNode(&node, G.graph, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    TFIM_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    int rc = TFIM_OK;
    do {
        k_res_pack_g<<<1, kPackThreads, 0, s>>>(d_args);
        k_res_zero<<<sm * 4, 256, 0, s>>>(d_args);
        if ((rc = launch_count_lop3_persistent(&d_args->a3, &d_status->tiles_l3, &d_status->next3, sm * std::max(1, occ3), s)))
            break;
        if ((rc = launch_count_b1_persistent(&d_args->a1, &d_status->tiles_b1, &d_status->next1, sm * std::max(1, occ1), s)))
            break;
        if (with_proj &&
            (rc = launch_count_proj_persistent(&d_args->ap, &d_status->n_proj, sm * std::max(1, occp), red_off, red_items, s)))
            break;
        if ((rc = launch_count_pk_persistent(&d_args->atc, &d_status->tiles_tc, sm, s))) break;
        if ((rc = launch_count_gram_persistent(&d_args->agr, &d_status->tiles_gr, &d_status->next_gr, sm * std::max(1, occg),
                                               s)))
            break;
        k_res_expand_g<<<sm * std::max(1, occe), 256, 0, s>>>(d_args);
        k_build_masks_g<<<sm * 8, 256, 0, s>>>(d_args);
        k_index_mfis_g<<<sm, 256, 0, s>>>(d_args);
        k_prune_stack_g<<<sm, 256, 0, s>>>(d_args);
        k_res_control<<<1, 32, 0, s>>>(d_args, h);
    } while (0);
    cudaGraph_t captured = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(s, &captured);
    if (rc != TFIM_OK) return rc;
    TFIM_CUDA(ec);
    TFIM_CUDA(cudaGetLastError());
    TFIM_CUDA(cudaGraphInstantiate(&G.exec, G.graph, 0));
    G.args = d_args;
    G.status = d_status;
    G.with_proj = with_proj ? 1 : 0;
    return TFIM_OK;
}

}  // namespace

struct ResidentState {
    Pool fams, items, heads, stack, looks, free_slots, defer, mfi_off, mfi_len, mfi_sup, mfi_items, log_feat, log_label;
    Pool djobs, jobs, rows, row_job, row_local, tiles_l3, tiles_b1, tiles_tc, tiles_gr, counts, status, is_root, dense_freq, top_pos,
        top_diag, proj_list, args, top_sum, mjobs, sup_index;
    Pool pk_list, loop_bar;
    Pool pjobs, pj_off, pj_pool, vrows, vitem;              // projected families
    Pool ord_keys, ord_idx, ord_meta, ord_items, ord_tmp;   // output order of the MFIs
    size_t mem_total = 0;                                   // the device's memory (0: not asked for yet)
    HostBuf h_status, h_args, h_res, h_setup, h_first, h_tiles;
    // the database's part of the search's initial state (root flags, the top family in
    // increasing support order), computed at a context's first resident mine and its pinned
    // staging reused by later mines; setup_uid names the context it belongs to
    uint64_t setup_uid = 0;
    std::vector<char> is_root_h;
    std::vector<int32_t> F0;
    size_t setup_total = 0;
    WaveGraph graph;
    int32_t launch_id = 0;
    void release(cudaStream_t s) {
        graph.release();
        for (Pool* b : {&fams, &items, &heads, &stack, &looks, &free_slots, &defer, &mfi_off, &mfi_len, &mfi_sup, &mfi_items,
                        &log_feat, &log_label, &djobs, &jobs, &rows, &row_job, &row_local, &tiles_l3, &tiles_b1, &tiles_tc, &tiles_gr, &counts,
                        &status, &is_root, &dense_freq, &top_pos, &top_diag, &proj_list, &args, &top_sum, &mjobs,
                        &sup_index, &pk_list, &loop_bar, &pjobs, &pj_off, &pj_pool, &vrows, &vitem, &ord_keys, &ord_idx, &ord_meta, &ord_items, &ord_tmp}) {
            dev_free(b->p, s);
            b->p = nullptr;
            b->bytes = 0;
        }
        h_status.release();
        h_args.release();
        h_res.release();
        h_setup.release();
        h_first.release();
        h_tiles.release();
    }
};

void free_resident(ResidentState* r, cudaStream_t s) {
    if (!r) return;
    r->release(s);
    delete r;
}

// Resident-engine pools and mask pools of closed contexts, one of each per device.  A
// context that closes after its work has finished hands them over (its stream is idle); the
// next context's first resident mine on that device adopts them, so a database opened again
// starts from pools already grown to the last search's size instead of growing (and copying)
// them from their minimum.  tfim_release_cached frees them.
namespace {
std::mutex g_cache_mu;
ResidentState* g_cached_res[64] = {};
DevBuf g_cached_masks[64];
}  // namespace

void stash_resident(tfim_ctx* c) {
    const int dev = c->device;
    if (dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> lk(g_cache_mu);
    if (c->resident) {
        c->resident->graph.release();   // its launches hold this context's transaction list
        // the projected rows, which may be many GB, go back to the device's pool: their size is this
        // database's own
        dev_free(c->resident->pj_pool.p, c->stream);
        c->resident->pj_pool = Pool{};
        if (g_cached_res[dev]) free_resident(g_cached_res[dev], c->stream);
        g_cached_res[dev] = c->resident;
        c->resident = nullptr;
    }
    if (c->d_masks.p && c->d_masks.bytes > g_cached_masks[dev].bytes) {
        g_cached_masks[dev].release();
        g_cached_masks[dev] = c->d_masks;
        // the closing context's stream is idle and about to be destroyed: a cached buffer
        // holds no stream (freed on the default stream, adopted onto the adopter's)
        g_cached_masks[dev].stream = nullptr;
        c->d_masks.p = nullptr;
        c->d_masks.bytes = 0;
    }
}

void adopt_resident(tfim_ctx* c) {
    const int dev = c->device;
    if (dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> lk(g_cache_mu);
    if (!c->resident && g_cached_res[dev]) {
        c->resident = g_cached_res[dev];
        g_cached_res[dev] = nullptr;
    }
    if (g_cached_masks[dev].p && g_cached_masks[dev].bytes > c->d_masks.bytes) {
        c->d_masks.release();
        c->d_masks = g_cached_masks[dev];
        c->d_masks.stream = c->stream;
        g_cached_masks[dev].p = nullptr;
        g_cached_masks[dev].bytes = 0;
    }
}

int release_cached(int dev) {
    std::lock_guard<std::mutex> lk(g_cache_mu);
    for (int d = 0; d < 64; d++) {
        if (dev >= 0 && d != dev) continue;
        stream_release(d);
        if (!g_cached_res[d] && !g_cached_masks[d].p) continue;
        TFIM_CUDA(cudaSetDevice(d));
        if (g_cached_res[d]) free_resident(g_cached_res[d], nullptr);
        g_cached_res[d] = nullptr;
        g_cached_masks[d].stream = nullptr;
        g_cached_masks[d].release();
        TFIM_CUDA(cudaDeviceSynchronize());
    }
    return TFIM_OK;
}

namespace {
// Sorts the n MFIs of the pool (ni items) into output order on the device and queues the
// copies of their sort keys (hkey[n]), lengths then supports (hmeta[2n]) and items
// (hitems[ni]) into pinned host memory; they are valid once the stream has finished.
int order_mfis(ResidentState& R, const tfim_ctx* c, const ResPtrs& P, int32_t n, int64_t ni, int sm_count,
               cudaStream_t s, uint64_t* hkey, int32_t* hmeta, int32_t* hitems) {
    int32_t max_sup = 0;
    for (int32_t f : c->dense_freq) max_sup = std::max(max_sup, f);
    auto width = [](uint32_t x) { int b = 1; while (b < 32 && (x >> b)) b++; return b; };
    MfiKey f{width((uint32_t)std::max<int64_t>(max_sup, c->n_bits)), width((uint32_t)c->info.n_dense)};
    if (f.s_bits + 2 * f.i_bits > 64) f.i_bits = 0;
    if (n <= kFinishMax && ni <= kFinishMaxItems) {
        TFIM_TRY(grow(R.ord_items, (size_t)n * 16 + (size_t)ni * 4 + 16, s));
        auto finish = n <= kFinishThreads ? k_mfi_finish<1> : k_mfi_finish<4>;
        finish<<<1, kFinishThreads, 0, s>>>(P.mfi_off, P.mfi_len, P.mfi_sup, P.mfi_items, n, ni, f, (uint4*)R.ord_items.p,
                                            (uint4*)hkey);
        TFIM_CUDA(cudaGetLastError());
        return TFIM_OK;
    }
    size_t t_sort = 0, t_scan = 0;
    TFIM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t_sort, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                              (const int32_t*)nullptr, (int32_t*)nullptr, n, 0, f.bits(), s));
    TFIM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t_scan, (const int32_t*)nullptr, (int32_t*)nullptr, n, s));
    TFIM_TRY(grow(R.ord_keys, (size_t)n * 16, s));
    TFIM_TRY(grow(R.ord_idx, (size_t)n * 8, s));
    TFIM_TRY(grow(R.ord_meta, ((size_t)n * 3 + 1) * 4, s));
    TFIM_TRY(grow(R.ord_items, (size_t)std::max<int64_t>(ni, 1) * 4, s));
    TFIM_TRY(grow(R.ord_tmp, std::max<size_t>(std::max(t_sort, t_scan), 16), s));
    uint64_t* k_in = (uint64_t*)R.ord_keys.p;
    uint64_t* k_out = k_in + n;
    int32_t* i_in = (int32_t*)R.ord_idx.p;
    int32_t* i_out = i_in + n;
    int32_t* len_o = (int32_t*)R.ord_meta.p;
    int32_t* sup_o = len_o + n;
    int32_t* off_o = sup_o + n;
    int32_t* items_o = (int32_t*)R.ord_items.p;
    const unsigned grid = (unsigned)std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)sm_count * 8);
    k_mfi_keys<<<grid, 256, 0, s>>>(P.mfi_off, P.mfi_len, P.mfi_sup, P.mfi_items, n, f, k_in, i_in);
    TFIM_CUDA(cudaGetLastError());
    size_t t = R.ord_tmp.bytes;
    TFIM_CUDA(cub::DeviceRadixSort::SortPairs(R.ord_tmp.p, t, k_in, k_out, i_in, i_out, n, 0, f.bits(), s));
    k_mfi_permute<<<grid, 256, 0, s>>>(i_out, P.mfi_len, P.mfi_sup, n, len_o, sup_o);
    TFIM_CUDA(cudaGetLastError());
    t = R.ord_tmp.bytes;
    TFIM_CUDA(cub::DeviceScan::ExclusiveSum(R.ord_tmp.p, t, len_o, off_o, n, s));
    const unsigned ggrid = (unsigned)std::min<int64_t>(((int64_t)n + 7) / 8, (int64_t)sm_count * 8);
    k_mfi_gather<<<ggrid, 256, 0, s>>>(i_out, P.mfi_off, P.mfi_items, off_o, len_o, n, items_o);
    TFIM_CUDA(cudaGetLastError());
    TFIM_CUDA(cudaMemcpyAsync(hkey, k_out, (size_t)n * 8, cudaMemcpyDeviceToHost, s));
    TFIM_CUDA(cudaMemcpyAsync(hmeta, len_o, (size_t)n * 8, cudaMemcpyDeviceToHost, s));   // len_o, sup_o
    if (ni) TFIM_CUDA(cudaMemcpyAsync(hitems, items_o, (size_t)ni * 4, cudaMemcpyDeviceToHost, s));
    return TFIM_OK;
}

// Finishes the output order on the host: item lists longer than 64 (the device sorts
// shorter ones as it emits them) are sorted, then each run of equal sort keys is ordered by
// the full comparison of item lists.
void finish_mfi_order(MfiSet& M, const uint64_t* key) {
    const size_t n = M.size();
    for (size_t k = 0; k < n; k++)
        if (M.off[k + 1] - M.off[k] > 64)
            std::sort(M.items.begin() + M.off[k], M.items.begin() + M.off[k + 1], std::greater<int32_t>());
    std::vector<int32_t> idx, items;
    for (size_t a = 0; a < n;) {
        size_t b = a + 1;
        while (b < n && key[b] == key[a]) b++;
        if (b - a > 1) {
            idx.resize(b - a);
            for (size_t q = a; q < b; q++) idx[q - a] = (int32_t)q;
            std::sort(idx.begin(), idx.end(), [&](int32_t x, int32_t y) {
                return std::lexicographical_compare(M.items.begin() + M.off[y], M.items.begin() + M.off[y + 1],
                                                    M.items.begin() + M.off[x], M.items.begin() + M.off[x + 1]);
            });
            items.assign(M.items.begin() + M.off[a], M.items.begin() + M.off[b]);
            const int64_t base = M.off[a];
            int64_t o = base;
            for (int32_t q : idx) {
                const int64_t l = M.off[q + 1] - M.off[q];
                std::copy(items.begin() + (M.off[q] - base), items.begin() + (M.off[q] - base) + l, M.items.begin() + o);
                o += l;
            }
            // supports are equal within the run; the offsets follow the new lengths
            std::vector<int64_t> lens(b - a);
            for (size_t q = 0; q < idx.size(); q++) lens[q] = M.off[idx[q] + 1] - M.off[idx[q]];
            for (size_t q = 0; q < idx.size(); q++) M.off[a + q + 1] = M.off[a + q] + lens[q];
        }
        a = b;
    }
}
}  // namespace

namespace {
// A search that a tensor-core counter left with incomplete counts reports that counter's wait.
int check_search(tfim_ctx* c, int32_t error) {
    if (error == 0) return TFIM_OK;
    int32_t status = 0;
    TFIM_CUDA(cudaMemcpyAsync(&status, c->d_status.p, 4, cudaMemcpyDeviceToHost, c->stream));
    TFIM_CUDA(cudaStreamSynchronize(c->stream));
    TFIM_TRY(tensor_status_check(status));
    TFIM_CHECK(error != kErrWait, search_error_status(error), "resident search: a wait of the device loop's grid barrier expired");
    set_error("resident search invariant failed (code %d)", error);
    return search_error_status(error);
}

int search_resident(tfim_ctx* c, const tfim_mine_opts* o, tfim_mine_stats* stt, bool may_project, bool* projected) {
    const auto t_entry = std::chrono::steady_clock::now();
    cudaStream_t s = c->stream;
    const int32_t d = c->n_counted;
    const int32_t minc = c->info.min_count;
    const int64_t W = c->W;
    const int32_t la_mode = o->lookahead;
    TFIM_CHECK(la_mode != 2 || c->proposal, TFIM_E_STATE, "lookahead mode 2 needs a proposal network (tfim_set_proposal)");
    if (!c->resident) adopt_resident(c);
    if (!c->resident) c->resident = new ResidentState();
    ResidentState& R = *c->resident;
    c->la_feats.clear();
    c->la_labels.clear();

    const bool fresh_setup = R.setup_uid != c->uid;
    if (fresh_setup) {
        R.is_root_h.assign((size_t)c->info.n_dense + 1, 0);
        for (int32_t r : c->roots) R.is_root_h[r] = 1;
        // top family: the counted items frequent by bitmap support, increasing support
        R.F0.clear();
        const bool ordered = (int32_t)c->support_order.size() == d;
        for (int32_t k = 0; k < d; k++) {
            const int32_t e = ordered ? c->support_order[k] : k;
            if (c->bit_support[e] >= minc) R.F0.push_back(e);
        }
        if (!ordered)
            std::stable_sort(R.F0.begin(), R.F0.end(),
                             [&](int32_t a, int32_t b) { return c->bit_support[a] < c->bit_support[b]; });
    }
    const std::vector<char>& is_root = R.is_root_h;
    const std::vector<int32_t>& F0 = R.F0;
    // the parked id 0 used as a root: the reference's search for that root (host driver)
    if (c->info.n_dense > d && is_root[d]) TFIM_TRY(mine_plain_roots(c, {d}, stt));
    const int32_t n0 = (int32_t)F0.size();
    if (n0 == 0) return TFIM_OK;

    int sm_count = 148;
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
    }
    const tfim_tuning tn = tuning();
    const int32_t wave_rows = o->wave_cap > 0 ? o->wave_cap : tn.wave_rows;
    const int64_t top_out = (int64_t)n0 * n0;
    const bool small = o->small_pools != 0;
    const size_t gmin = small ? 64 : (1 << 16);
    auto grow = [&](Pool& b, size_t need, cudaStream_t st) { return tfim::grow(b, need, st, gmin); };
    int64_t cap_out = small ? top_out : std::max<int64_t>(top_out, 64LL << 20);
    int64_t cap_tiles = small ? 64 : 1LL << 21;
    int64_t cap_rows = std::max<int64_t>(wave_rows, n0) + 64;

    // initial capacities (the first wave's ensure grows them to what its expand needs)
    int64_t cap_fam = small ? 1 : std::max<int64_t>(4 * n0, 1 << 16);
    int64_t cap_item = small ? n0 : std::max<int64_t>(4 * top_out + 2 * n0, 1 << 20);   // holds the top family's list
    int64_t cap_head = 1 << 20, cap_mfi = 1 << 16, cap_mfi_items = 1 << 20, cap_slots = 1 << 12, cap_log = 1 << 16;
    if (small) cap_head = cap_mfi = cap_mfi_items = cap_slots = cap_log = 1;
    TFIM_TRY(grow(R.status, sizeof(ResStatus) + 16, s));
    TFIM_TRY(grow(R.fams, cap_fam * sizeof(DFam), s));
    TFIM_TRY(grow(R.items, cap_item * 4, s));
    TFIM_TRY(grow(R.heads, cap_head * 4, s));
    TFIM_TRY(grow(R.stack, cap_fam * 4, s));
    TFIM_TRY(grow(R.looks, cap_rows * sizeof(DLook), s));
    TFIM_TRY(grow(R.free_slots, cap_slots * 4, s));
    TFIM_TRY(grow(R.defer, cap_slots * 4, s));
    TFIM_TRY(grow(R.mfi_off, cap_mfi * 4, s));
    TFIM_TRY(grow(R.mfi_len, cap_mfi * 4, s));
    TFIM_TRY(grow(R.mfi_sup, cap_mfi * 4, s));
    TFIM_TRY(grow(R.mfi_items, cap_mfi_items * 4, s));
    if (o->log_lookahead) {
        TFIM_TRY(grow(R.log_feat, cap_log * 32 * 4, s));
        TFIM_TRY(grow(R.log_label, cap_log * 4, s));
    }
    TFIM_TRY(grow(R.djobs, cap_rows * sizeof(DJob), s));
    TFIM_TRY(grow(R.jobs, cap_rows * sizeof(JobDesc), s));
    TFIM_TRY(grow(R.rows, cap_rows * sizeof(RowDesc), s));
    TFIM_TRY(grow(R.row_job, cap_rows * 4, s));
    TFIM_TRY(grow(R.row_local, cap_rows * 4, s));
    TFIM_TRY(grow(R.proj_list, cap_rows * 4, s));
    TFIM_TRY(grow(R.pk_list, cap_rows * kPkJobs * 4, s));   // at most one tile per job
    TFIM_TRY(grow(R.mjobs, (2 * cap_rows + 2) * sizeof(MaskJob), s));   // at most two masks per expanded row
    TFIM_TRY(grow(R.tiles_l3, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.tiles_b1, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.tiles_tc, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.tiles_gr, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.counts, cap_out * 4, s));
    TFIM_TRY(grow(R.is_root, is_root.size(), s));
    TFIM_TRY(grow(R.dense_freq, (size_t)std::max<int32_t>(c->info.n_dense, 1) * 4, s));
    TFIM_TRY(grow(R.top_pos, (size_t)std::max<int32_t>(c->info.n_dense, 1) * 4, s));
    TFIM_TRY(grow(R.top_diag, (size_t)n0 * 4, s));
    // superset index (opts.superset): d items x sup_words words (about 32 MiB; MFIs past its
    // capacity are not indexed and prune nothing), cleared for every mine
    const bool sup_on = o->superset != 0;
    const int32_t sup_words = (int32_t)std::min<int64_t>(65536, std::max<int64_t>(32, (8LL << 20) / std::max(d, 1)));
    if (sup_on) {
        const size_t sup_bytes = (size_t)d * (size_t)sup_words * 4;
        TFIM_TRY(grow(R.sup_index, sup_bytes, s));
        TFIM_CUDA(cudaMemsetAsync(R.sup_index.p, 0, sup_bytes, s));
    }
    // mask slots (grown on demand)
    int64_t slot_cap = c->d_masks.bytes / ((size_t)W * 4);

    // top family counting: pair co-occurrence or the symmetric bitmap Gram (cost model)
    int top_mode;
    {
        const double nF = n0;
        const bool b1 = o->counter != TFIM_COUNTER_LOP3 &&
                        (o->counter == TFIM_COUNTER_TENSOR || (nF >= tn.b1_min_rows && nF >= tn.b1_min_cols));
        const bool i8 = o->counter != TFIM_COUNTER_LOP3 && o->counter != TFIM_COUNTER_TENSOR && nF >= tn.i8_min_rows &&
                        nF >= tn.i8_min_cols;
        const double rate = i8 ? tn.rate_i8_bitops : b1 ? tn.rate_b1_bitops : tn.rate_lop3_bitops;
        const double bitmap_s = nF * nF * (double)c->n_bits / 2.0 / rate;
        const double pairs_s = c->red_pair_work / 2.0 / tn.rate_pair_incr + nF * nF * 4.0 / kTuneHbmBytes;
        if (o->top_counter == 1) top_mode = 1;
        else if (o->top_counter == 2) top_mode = c->csr_exact ? 2 : 1;
        else top_mode = (c->csr_exact && pairs_s < bitmap_s) ? 2 : 1;
    }
    const bool top_b1 = o->counter == TFIM_COUNTER_TENSOR ||
                        (o->counter != TFIM_COUNTER_LOP3 && n0 >= tn.b1_min_rows && n0 >= tn.b1_min_cols);
    // the tcgen05 wave counter (38 items x 2M transactions: 17 us against 143 on the CUDA-core tiles)
    const bool top_i8 = o->counter != TFIM_COUNTER_LOP3 && o->counter != TFIM_COUNTER_TENSOR && n0 >= tn.i8_min_rows &&
                        n0 >= tn.i8_min_cols;

    // the projected counter, which reads the transaction list, may be picked
    const bool may_list = c->csr_exact && (o->counter == TFIM_COUNTER_PROJ ||
                                           (o->counter == TFIM_COUNTER_AUTO && (o->proj_auto >= 0 ? o->proj_auto : tn.proj_auto)));
    const bool use_graph = o->use_graphs != 0;
    // small waves run in the device loop; a small enough family of the empty prefix is its first wave
    const bool loop = !use_graph && W <= (64 * (int64_t)minc >= c->n_bits ? kLoopDenseWords : kLoopMaxWords) && !sup_on && !may_list &&
                      (o->counter == TFIM_COUNTER_AUTO || o->counter == TFIM_COUNTER_LOP3);
    // Children of the empty prefix move to universes of their own when the database is long enough
    // for a wave's counting to outweigh the extra status read (small_pools: any length, so that
    // short ones exercise it), some frequent item lies in at most half of it, and no counter that
    // reads the transaction list may be picked.
    const bool project = may_project && (W >= (1 << 12) || small) && 2 * (int64_t)c->bit_support[F0.front()] <= c->n_bits &&
                         64 * (int64_t)minc >= c->n_bits && !may_list;
    const bool top_loop = loop && !project && o->top_counter == 0 && top_mode == 1 && n0 <= wave_rows &&
                          (double)n0 * n0 * (double)W <= kLoopTopWork;

    // the search's initial state, staged in pinned memory and copied asynchronously:
    // root flags, F1 counts, the top family record, its F list and its single job, rows,
    // F positions and row supports, the status record
    DFam top;
    top.slot = -1; top.item = -1; top.head_off = 0; top.head_len = 0; top.F_off = 0; top.nF = n0; top.nT = n0;
    top.sup = 0; top.next_row = top_loop ? 0 : n0; top.rows_done = 0; top.state = 0; top.top = 1;
    top.W = (int32_t)W; top.n = (int32_t)c->n_bits;
    ResStatus hs;
    memset(&hs, 0, sizeof hs);
    for (int k = 0; k < kPhases; k++) hs.ph_s[k] = ~0ull;
    hs.fam_n = 1;
    hs.item_n = n0;
    hs.jobs = 1;
    hs.rows = n0;
    hs.out_total = top_out;
    hs.max_cols = n0;
    if (top_loop) {
        hs.stack_n = 1;   // entry 0: the top family
    } else {
        hs.nodes = n0;
        hs.supports = (unsigned long long)top_out;
    }
    {
        SetupParts setup{};
        // the staging blob is the same for every mine of this database: built once, and the
        // parts (whose device pools may have moved) copied again on every mine
        const size_t nd = (size_t)std::max<int32_t>(c->info.n_dense, 1);
        struct Part { void* dst; size_t off, bytes; };
        std::vector<Part> parts;
        size_t total = 0;
        auto part = [&](void* dst, size_t bytes) {
            parts.push_back(Part{dst, total, bytes});
            total += (bytes + 15) & ~size_t(15);
            return parts.size() - 1;
        };
        const size_t p_root = part(R.is_root.p, is_root.size()), p_freq = part(R.dense_freq.p, c->dense_freq.size() * 4),
                     p_F = part(R.items.p, (size_t)n0 * 4),
                     p_dj = part(R.djobs.p, sizeof(DJob)), p_jd = part(R.jobs.p, sizeof(JobDesc)),
                     p_rows = part(R.rows.p, (size_t)n0 * sizeof(RowDesc)), p_rj = part(R.row_job.p, (size_t)n0 * 4),
                     p_rl = part(R.row_local.p, (size_t)n0 * 4), p_pos = part(R.top_pos.p, nd * 4),
                     p_diag = part(R.top_diag.p, (size_t)n0 * 4);
        unsigned char* h = nullptr;
        if (fresh_setup || !R.h_setup.p || R.setup_total != total) {
            TFIM_TRY(R.h_setup.reserve(total));
            h = R.h_setup.as<unsigned char>();
            auto at = [&](size_t k) { return (void*)(h + parts[k].off); };
            memcpy(at(p_root), is_root.data(), is_root.size());
            memcpy(at(p_freq), c->dense_freq.data(), c->dense_freq.size() * 4);
            memcpy(at(p_F), F0.data(), (size_t)n0 * 4);
            {
                DJob dj{};
                dj.kind = kJobFam; dj.nr = n0; dj.slot = -1; dj.log = -1; dj.sl3 = 1;
                *(DJob*)at(p_dj) = dj;
            }
            *(JobDesc*)at(p_jd) = JobDesc{-1, -1, n0, n0, 0, 0, 0, -1, (int32_t)W};
            RowDesc* rows = (RowDesc*)at(p_rows);
            int32_t* rj = (int32_t*)at(p_rj);
            int32_t* rl = (int32_t*)at(p_rl);
            int32_t* pos = (int32_t*)at(p_pos);
            int32_t* diag = (int32_t*)at(p_diag);
            std::fill(pos, pos + nd, -1);
            for (int32_t k = 0; k < n0; k++) {
                rows[k] = RowDesc{-1, F0[k]};
                rj[k] = 0;
                rl[k] = k;
                pos[F0[k]] = k;
                diag[k] = c->bit_support[F0[k]];
            }
            R.setup_uid = c->uid;
            R.setup_total = total;
        }
        h = R.h_setup.as<unsigned char>();
        for (const Part& q : parts)
            if (q.bytes) setup.part[setup.n++] = SetupPart{(const uint4*)(h + q.off), (uint4*)q.dst, (int64_t)(q.bytes + 15) / 16};
        // this mine's records: status, the top family, the stack's first entry
        const size_t o_top = (sizeof hs + 15) & ~size_t(15), o_stack = o_top + sizeof top;
        TFIM_TRY(R.h_first.reserve(o_stack + 16));
        TFIM_TRY(c->d_status.reserve(64));
        unsigned char* hf = R.h_first.as<unsigned char>();
        memcpy(hf, &hs, sizeof hs);
        memcpy(hf + o_top, &top, sizeof top);
        memset(hf + o_stack, 0, 16);
        setup.part[setup.n++] = SetupPart{(const uint4*)hf, (uint4*)R.status.p, (int64_t)o_top / 16};
        setup.part[setup.n++] = SetupPart{(const uint4*)(hf + o_top), (uint4*)R.fams.p, (int64_t)sizeof top / 16};
        setup.part[setup.n++] = SetupPart{(const uint4*)(hf + o_stack), (uint4*)R.stack.p, 1};
        setup.part[setup.n++] = SetupPart{(const uint4*)(hf + o_stack), (uint4*)c->d_status.p, 1};   // zeros too
        static_assert(sizeof(DFam) % 16 == 0, "a family record is whole 16-byte pieces");
        k_res_setup<<<dim3((unsigned)std::min<size_t>(16, (size_t)n0 / 512 + 1), (unsigned)setup.n), 256, 0, s>>>(setup);
        TFIM_CUDA(cudaGetLastError());
    }
    TFIM_TRY(R.h_status.reserve(sizeof(ResStatus)));
    ResStatus* hst = R.h_status.as<ResStatus>();

    double sync_ms = 0, kernel_ms = 0;
    int64_t launches = 0, count_launches = 0, bytes_alg = 0, waves = 0;
    int64_t path_launches[6] = {0, 0, 0, 0, 0, 0};
    bool used_tc = false;   // the tcgen05 family counter ran (its status is read at the end)
    const int64_t row_bytes = (c->n_bits + 7) / 8;
    ResStatus* d_st = (ResStatus*)R.status.p;

    ResPtrs P;
    auto refresh_ptrs = [&]() {
        P.fams = (DFam*)R.fams.p; P.items = (int32_t*)R.items.p; P.heads = (int32_t*)R.heads.p;
        P.stack = (int32_t*)R.stack.p; P.looks = (DLook*)R.looks.p; P.free_slots = (int32_t*)R.free_slots.p;
        P.defer = (int32_t*)R.defer.p; P.mfi_off = (int32_t*)R.mfi_off.p; P.mfi_len = (int32_t*)R.mfi_len.p;
        P.mfi_sup = (int32_t*)R.mfi_sup.p; P.mfi_items = (int32_t*)R.mfi_items.p;
        P.log_feat = (float*)R.log_feat.p; P.log_label = (float*)R.log_label.p;
        P.djobs = (DJob*)R.djobs.p; P.jobs = (JobDesc*)R.jobs.p; P.rows = (RowDesc*)R.rows.p;
        P.mjobs = (MaskJob*)R.mjobs.p;
        P.row_job = (int32_t*)R.row_job.p; P.row_local = (int32_t*)R.row_local.p;
        P.tiles_l3 = (TileDesc*)R.tiles_l3.p; P.tiles_b1 = (TileDesc*)R.tiles_b1.p; P.tiles_tc = (TileDesc*)R.tiles_tc.p;
        P.tiles_gr = (TileDesc*)R.tiles_gr.p;
        P.pk_list = (int32_t*)R.pk_list.p;
        P.counts = (int32_t*)R.counts.p;
        P.bitmap = c->d_bitmap; P.masks = c->d_masks.as<uint32_t>(); P.dense_freq = (const int32_t*)R.dense_freq.p;
        P.is_root = (const uint8_t*)R.is_root.p; P.st = (ResStatus*)R.status.p;
        P.W = W; P.n_bits = c->n_bits; P.min_count = minc; P.wave_rows = wave_rows;
        P.cap_out = cap_out; P.cap_tiles = cap_tiles; P.counter = o->counter; P.la_mode = la_mode;
        P.log_on = o->log_lookahead; P.proposal_threshold = c->proposal_threshold; P.kslice_min = 64; P.sm_count = sm_count;
        P.mlp_w = nullptr; P.mlp_p = nullptr;
        P.proj_list = (int32_t*)R.proj_list.p;
        P.avg_len = c->n_bits > 0 ? (float)((double)c->n_red_items / (double)c->n_bits) : 0.f;
        P.csr_ok = c->csr_exact ? 1 : 0;
        P.proj_auto = o->proj_auto >= 0 ? o->proj_auto : tn.proj_auto;
        P.b1_min_rows = tn.b1_min_rows;
        P.b1_min_cols = tn.b1_min_cols;
        P.l3_slices_per_sm = tn.l3_slices_per_sm;
        P.l3_dense_slices_per_sm = tn.l3_dense_slices_per_sm;
        P.b1_tiles_per_sm = tn.b1_tiles_per_sm;
        P.tc_min_work = tn.tc_min_work;
        P.tc_min_density = tn.tc_min_density;
        P.tc_tiles_per_sm = tn.tc_tiles_per_sm;
        P.gram_min_rows = tn.gram_min_rows;
        if (la_mode == 2 && c->proposal) {
            const void* wb = nullptr;
            const float* pp = nullptr;
            mlp_device_params(c->proposal, &wb, &pp);
            P.mlp_w = (const __nv_bfloat16*)wb;
            P.mlp_p = pp;
        }
        Caps& k = P.caps;
        k.fam = (int64_t)std::min(R.fams.bytes / sizeof(DFam), R.stack.bytes / 4);
        k.item = (int64_t)(R.items.bytes / 4);
        k.head = (int64_t)(R.heads.bytes / 4);
        k.mfi = (int64_t)std::min({R.mfi_off.bytes, R.mfi_len.bytes, R.mfi_sup.bytes}) / 4;
        k.mfi_items = (int64_t)(R.mfi_items.bytes / 4);
        k.looks = (int64_t)(R.looks.bytes / sizeof(DLook));
        k.slots = std::min<int64_t>(slot_cap, (int64_t)std::min(R.free_slots.bytes, R.defer.bytes) / 4);
        k.log = o->log_lookahead ? (int64_t)std::min(R.log_feat.bytes / 128, R.log_label.bytes / 4) : 0;
        k.rows = cap_rows;
        P.row_bytes = row_bytes;
        P.row_sum = nullptr;
        P.wave_limit = 0x7fffffff;
        P.launch_id = 0;
        P.max_launch_ns = small ? 1000ull : 2000000000ull;   // small_pools: every launch ends after one wave
        P.sup_index = sup_on ? (uint32_t*)R.sup_index.p : nullptr;
        P.sup_words = sup_words;
        P.sup_items = d;
        P.n_base = c->info.n_dense;
        P.vrows = (const uint32_t**)R.vrows.p;
        P.vitem = (int32_t*)R.vitem.p;
        P.pjobs = (PJob*)R.pjobs.p;
        P.pj_off = (int32_t*)R.pj_off.p;
        P.pj_pool = (uint32_t*)R.pj_pool.p;
        P.h_st = hst;
    };
    // capacity for the worst case of one expand over `rows` rows of at most `max_cols`
    // columns each and `out_total` counts
    auto ensure = [&](const ResStatus& h, int64_t rows, int64_t jobs, int64_t out_total, int64_t max_head,
                      int64_t max_cols) -> int {
        const int64_t list = max_head + 2 + max_cols;
        const int64_t need_fam = h.fam_n + rows + 1;
        const int64_t need_item = h.item_n + 2 * out_total + rows + 1;
        const int64_t need_head = h.head_n + rows * list + 1;
        const int64_t need_mfi = h.mfi_n + rows + jobs + 1;
        const int64_t need_mfi_items = h.mfi_item_n + (rows + jobs) * list + 1;
        const int64_t need_slots = h.slot_n + 2 * rows + 2;
        const int64_t need_log = h.log_n + rows + 1;
        TFIM_TRY(grow(R.fams, need_fam * sizeof(DFam), s));
        TFIM_TRY(grow(R.stack, need_fam * 4, s));
        TFIM_TRY(grow(R.items, need_item * 4, s));
        TFIM_TRY(grow(R.heads, need_head * 4, s));
        TFIM_TRY(grow(R.mfi_off, need_mfi * 4, s));
        TFIM_TRY(grow(R.mfi_len, need_mfi * 4, s));
        TFIM_TRY(grow(R.mfi_sup, need_mfi * 4, s));
        TFIM_TRY(grow(R.mfi_items, need_mfi_items * 4, s));
        TFIM_TRY(grow(R.looks, (rows + 1) * sizeof(DLook), s));
        TFIM_TRY(grow(R.free_slots, need_slots * 4, s));
        TFIM_TRY(grow(R.defer, need_slots * 4, s));
        if (o->log_lookahead) {
            TFIM_TRY(grow(R.log_feat, need_log * 32 * 4, s));
            TFIM_TRY(grow(R.log_label, need_log * 4, s));
        }
        if (need_slots > slot_cap) {
            DevBuf nb;
            nb.stream = s;
            const int64_t ncap = std::max<int64_t>(need_slots + need_slots / 2, 64);
            TFIM_TRY(nb.reserve((size_t)ncap * (size_t)W * 4));
            if (c->d_masks.p && slot_cap > 0)
                TFIM_CUDA(cudaMemcpyAsync(nb.p, c->d_masks.p, (size_t)slot_cap * (size_t)W * 4, cudaMemcpyDeviceToDevice, s));
            c->d_masks.release();
            c->d_masks = nb;
            slot_cap = ncap;
        }
        refresh_ptrs();
        return TFIM_OK;
    };
    // the pack declined a wave: grow what it asked for
    auto grow_for = [&](const ResStatus& h) -> int {
        if (h.starved) {
            // a single row does not fit the count buffer
            cap_out *= 4;
            TFIM_TRY(grow(R.counts, cap_out * 4, s));
        }
        if (h.grow) {
            if (h.g_out > cap_out) {
                cap_out = std::max<int64_t>(2 * cap_out, h.g_out);
                TFIM_TRY(grow(R.counts, cap_out * 4, s));
            }
            if (h.g_tiles > cap_tiles) {
                cap_tiles = std::max<int64_t>(2 * cap_tiles, h.g_tiles);
                TFIM_TRY(grow(R.tiles_l3, cap_tiles * sizeof(TileDesc), s));
                TFIM_TRY(grow(R.tiles_b1, cap_tiles * sizeof(TileDesc), s));
                TFIM_TRY(grow(R.tiles_tc, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.tiles_gr, cap_tiles * sizeof(TileDesc), s));
            }
            TFIM_TRY(ensure(h, h.g_rows, h.g_jobs, h.g_out, h.g_max_head, h.g_max_cols));
        }
        refresh_ptrs();   // the next pack clears the request
        return TFIM_OK;
    };

    auto project_families = [&]() -> int {
        const int64_t nt = W / kProjTile;
        P.pj_tm = nullptr;
        TFIM_TRY(grow(R.pjobs, (size_t)(n0 + 1) * sizeof(PJob), s));
        refresh_ptrs();
        k_proj_plan<<<1, kPackThreads, 0, s>>>(P);
        TFIM_CUDA(cudaGetLastError());
        TFIM_CUDA(cudaMemcpyAsync(hst, R.status.p, sizeof(ResStatus), cudaMemcpyDeviceToHost, s));
        TFIM_CUDA(cudaStreamSynchronize(s));
        launches++;
        const int32_t n_pj = hst->pj_n;
        const int64_t n_rows = hst->pj_rows, words = hst->pj_words;
        if (n_pj == 0) return TFIM_OK;
        const size_t row_bytes = (size_t)words * 4, off_bytes = (size_t)n_pj * (size_t)(nt + 1) * 4;
        // groups of 32 items, in chunks that shared memory holds; an odd number per chunk
        const int32_t groups = (n0 + 31) / 32;
        P.pj_chunks = (groups + kProjGroups - 1) / kProjGroups;
        P.pj_gc = ((groups + P.pj_chunks - 1) / P.pj_chunks) | 1;
        const int64_t n_g = (int64_t)P.pj_chunks * P.pj_gc;
        const size_t tm_bytes = (size_t)n_g * W * 128, inv_bytes = (size_t)n_pj * n_g * 64,
                     gb_bytes = (size_t)n_pj * P.pj_chunks * 4, extra = tm_bytes + inv_bytes + gb_bytes + (size_t)P.n_base * 4;
        bool by_row = n_rows >= kProjMinCols * hst->pj_groups && n0 <= 32767;
        size_t bytes = row_bytes + (by_row ? extra : 0);
        if (bytes > R.pj_pool.bytes) {   // its old contents are not needed
            dev_free(R.pj_pool.p, s);
            R.pj_pool = Pool{};
            // The compressed rows may take an eighth of the device's memory, and half of what is left
            // of it: later waves' pools grow beside them.  Without room for the transposed copy they
            // are made word by word, without room for them the families stay where they are.  The
            // driver is asked (slowly) only when the pool's own unused memory is not enough.
            const size_t side = off_bytes + (size_t)n_rows * 12;
            size_t left = dev_unused(c->device), room = left / 2;
            if (bytes + side > room || !R.mem_total) {
                size_t mem_free = 0;
                TFIM_CUDA(cudaMemGetInfo(&mem_free, &R.mem_total));
                room = (left + mem_free) / 2;
            }
            room = std::min(room, R.mem_total / 8);
            if (bytes + side > room) {
                by_row = false;
                bytes = row_bytes;
                if (bytes + side > room) return TFIM_OK;
            }
            if (dev_alloc(&R.pj_pool.p, bytes, s) != TFIM_OK) {
                R.pj_pool = Pool{};
                cudaGetLastError();
                return TFIM_OK;
            }
            R.pj_pool.bytes = bytes;
        }
        if (grow(R.vrows, (size_t)n_rows * 8, s) != TFIM_OK || grow(R.vitem, (size_t)n_rows * 4, s) != TFIM_OK ||
            grow(R.pj_off, off_bytes, s) != TFIM_OK) {
            cudaGetLastError();
            refresh_ptrs();
            return TFIM_OK;
        }
        refresh_ptrs();
        P.pj_pos = nullptr;
        if (by_row) {
            char* at = (char*)R.pj_pool.p + row_bytes;
            P.pj_tm = (uint32_t*)at;
            P.pj_inv = (int16_t*)(at + tm_bytes);
            P.pj_gbits = (uint32_t*)(at + tm_bytes + inv_bytes);
            P.pj_pos = (int32_t*)(at + tm_bytes + inv_bytes + gb_bytes);
        }
        k_proj_count<<<sm_count * 8, 256, 0, s>>>(P, n_pj);
        k_proj_scan<<<(n_pj + 7) / 8, 256, 0, s>>>(P, n_pj);
        k_proj_init<<<n_pj, 256, 0, s>>>(P);
        if (by_row) {
            // the limits are set for the widest chunk, the same from every thread
            TFIM_CUDA(cudaFuncSetAttribute(k_proj_tm, cudaFuncAttributeMaxDynamicSharedMemorySize, proj_tm_smem(kProjGroups)));
            TFIM_CUDA(cudaFuncSetAttribute(k_proj_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, proj_rows_smem(kProjGroups)));
            const int tm_smem = proj_tm_smem(P.pj_gc), smem = proj_rows_smem(P.pj_gc);
            k_proj_tm<<<dim3((unsigned)(W / 32), (unsigned)P.pj_chunks), 32 * P.pj_gc, tm_smem, s>>>(P);
            // a short database: several blocks per tile, each for a part of the families
            const int64_t units = nt * P.pj_chunks;
            const int32_t parts = (int32_t)std::max<int64_t>(
                1, std::min<int64_t>((4 * sm_count + units - 1) / units, (n_pj + kProjWarps - 1) / kProjWarps));
            k_proj_rows<<<(unsigned)std::min<int64_t>(units * parts, sm_count), 32 * kProjWarps, smem, s>>>(P, n_pj, parts);
        } else {
            k_proj_words<<<sm_count * 4, kProjThreads, 0, s>>>(P, n_pj);
        }
        k_proj_commit<<<n_pj, 128, 0, s>>>(P);
        TFIM_CUDA(cudaGetLastError());
        *projected = true;
        launches += by_row ? 6 : 5;
        return TFIM_OK;
    };

    // wave 1: the top family, counted whole
    *hst = hs;
    TFIM_TRY(ensure(hs, hs.rows, hs.jobs, hs.out_total, 0, hs.max_cols));
    if (top_loop) {
        stt->setup_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_entry).count();
    } else {
        std::vector<TileDesc> tl;
        bool top_wide = false;
        if (top_mode == 1) {
            if (top_i8) {
                top_wide = tiles_f4(0, n0, n0, W, sm_count, tl, true);
            } else if (top_b1) {
                const int64_t base = (int64_t)((n0 + kB1Rows - 1) / kB1Rows) * ((n0 + kB1Cols - 1) / kB1Cols);
                const int64_t want = (int64_t)(tn.b1_tiles_per_sm * sm_count);
                int64_t ks = std::min<int64_t>(std::max<int64_t>(1, (want + base - 1) / base), W / 64);
                const int64_t kslice = ((W / 64 + ks - 1) / ks) * 64;
                tiles_b1(0, n0, n0, W, kslice, tl, true);
            } else {
                const int64_t base = (int64_t)((n0 + kLop3Rows - 1) / kLop3Rows) * ((n0 + 63) / 64);
                const int64_t want = (int64_t)(tn.l3_slices_per_sm * sm_count);
                int64_t ws = std::min<int64_t>(std::max<int64_t>(1, (want + base - 1) / base), std::max<int64_t>(1, W / 256));
                const int64_t wslice = ((W / 64 + ws - 1) / ws) * 64;
                tiles_lop3(0, n0, n0, W, wslice, tl, true);
            }
        }
        if ((int64_t)tl.size() > cap_tiles) {
            cap_tiles = (int64_t)tl.size();
            TFIM_TRY(grow(R.tiles_l3, cap_tiles * sizeof(TileDesc), s));
            TFIM_TRY(grow(R.tiles_b1, cap_tiles * sizeof(TileDesc), s));
            TFIM_TRY(grow(R.tiles_tc, cap_tiles * sizeof(TileDesc), s));
    TFIM_TRY(grow(R.tiles_gr, cap_tiles * sizeof(TileDesc), s));
            refresh_ptrs();
        }
        if (!tl.empty()) {
            TFIM_TRY(R.h_tiles.reserve(tl.size() * sizeof(TileDesc)));
            memcpy(R.h_tiles.p, tl.data(), tl.size() * sizeof(TileDesc));
            TFIM_CUDA(cudaMemcpyAsync(top_b1 ? R.tiles_b1.p : R.tiles_l3.p, R.h_tiles.p, tl.size() * sizeof(TileDesc),
                                      cudaMemcpyHostToDevice, s));
        }
        TFIM_CUDA(cudaMemsetAsync(R.counts.p, 0, (size_t)top_out * 4, s));
        CountArgs a;
        a.bitmap = c->d_bitmap; a.W = W; a.masks = c->d_masks.as<uint32_t>(); a.jobs = P.jobs; a.rows = P.rows;
        a.cols = P.items; a.out = P.counts; a.status = c->d_status.as<int32_t>();
        stt->setup_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_entry).count();
        TFIM_CUDA(cudaEventRecord(c->ev0, s));
        if (top_mode == 2) {
            TFIM_TRY(launch_pair_count(c->d_red_off, c->d_red_items, c->n_bits, (const int32_t*)R.top_pos.p, n0, P.counts, s));
            bytes_alg += (c->n_bits + 1) * 8 + c->n_red_items * 4 + 4 * top_out;
        } else {
            a.tiles = top_b1 ? P.tiles_b1 : P.tiles_l3;
            a.n_tiles = (int32_t)tl.size();
            TFIM_TRY(top_i8 ? launch_count_f4(a, top_wide, s) : top_b1 ? launch_count_b1(a, s) : launch_count_lop3(a, s));
            bytes_alg += row_bytes * 2 * n0 + 4 * top_out;
        }
        TFIM_CUDA(cudaEventRecord(c->ev1, s));
        TFIM_TRY(grow(R.top_sum, (size_t)n0 * sizeof(RowSum), s));
        TFIM_CUDA(cudaMemsetAsync(R.top_sum.p, 0, (size_t)n0 * sizeof(RowSum), s));
        const unsigned nb = (unsigned)((n0 + 31) / 32);
        TFIM_CHECK(nb <= 65535, TFIM_E_INVALID, "family of %d items exceeds the grid", n0);
        k_top_finish<<<dim3(nb, nb), 256, 0, s>>>(P.counts, n0, (const int32_t*)R.top_diag.p, minc, (RowSum*)R.top_sum.p);
        TFIM_CUDA(cudaGetLastError());
        launches += 3;
        count_launches++;
        const int64_t threads = (int64_t)n0 * 32;
        ResPtrs Ptop = P;
        Ptop.row_sum = (const RowSum*)R.top_sum.p;
        k_res_expand<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(Ptop);
        TFIM_CUDA(cudaGetLastError());
        k_build_masks<<<sm_count * 8, 256, 0, s>>>(P);
        TFIM_CUDA(cudaGetLastError());
        if (project) TFIM_TRY(project_families());
        if (sup_on) {
            k_index_mfis<<<sm_count, 256, 0, s>>>(P);
            k_prune_stack<<<sm_count, 256, 0, s>>>(P);
            TFIM_CUDA(cudaGetLastError());
            launches += 2;
        }
        launches++;
        launches++;
        waves++;
    }
    // the counting path of the empty-prefix family, its work and (read at the end) its time
    const int top_path = top_mode == 2 ? TFIM_PATH_PAIRS : top_i8 ? TFIM_PATH_TC : top_b1 ? TFIM_PATH_B1 : TFIM_PATH_LOP3;
    if (!top_loop) path_launches[top_path]++;
    // following waves
    int64_t host_waves = 0;
    if (use_graph) {
        TFIM_TRY(grow(R.args, sizeof(ResArgs), s));
        TFIM_TRY(R.h_args.reserve(sizeof(ResArgs)));
        const bool with_proj = c->csr_exact && (o->counter == TFIM_COUNTER_PROJ || (o->counter == TFIM_COUNTER_AUTO && P.proj_auto));
        ResArgs* d_args = (ResArgs*)R.args.p;
        if (!R.graph.exec || R.graph.args != R.args.p || R.graph.status != R.status.p || R.graph.with_proj != (int)with_proj)
            TFIM_TRY(build_wave_graph(R.graph, d_args, (ResStatus*)R.status.p, with_proj, c->d_red_off, c->d_red_items, s));
        int64_t slices = 0;
        while (true) {
            ResArgs* ha = R.h_args.as<ResArgs>();
            ha->p = P;
            ha->p.launch_id = ++R.launch_id;
            ha->p.wave_limit = 0x7fffffff;
            CountArgs a;
            a.vrows = P.vrows; a.n_base = P.n_base; a.pk_list = P.pk_list; a.status = c->d_status.as<int32_t>();
            a.bitmap = c->d_bitmap; a.W = W; a.masks = P.masks; a.jobs = P.jobs; a.rows = P.rows;
            a.cols = P.items; a.out = P.counts; a.n_tiles = 0; a.job_list = P.proj_list;
            a.tiles = P.tiles_l3;
            a.ph_s = &d_st->ph_s[kPhLop3]; a.ph_e = &d_st->ph_e[kPhLop3];
            ha->a3 = a;
            a.tiles = P.tiles_b1;
            a.ph_s = &d_st->ph_s[kPhB1]; a.ph_e = &d_st->ph_e[kPhB1];
            ha->a1 = a;
            a.tiles = P.tiles_l3;
            a.ph_s = &d_st->ph_s[kPhProj]; a.ph_e = &d_st->ph_e[kPhProj];
            ha->ap = a;
            a.tiles = P.tiles_tc;
            a.ph_s = &d_st->ph_s[kPhTc]; a.ph_e = &d_st->ph_e[kPhTc];
            ha->atc = a;
            a.tiles = P.tiles_gr;
            a.ph_s = &d_st->ph_s[kPhGram]; a.ph_e = &d_st->ph_e[kPhGram];
            ha->agr = a;
            TFIM_CUDA(cudaMemcpyAsync(d_args, ha, sizeof(ResArgs), cudaMemcpyHostToDevice, s));
            TFIM_CUDA(cudaGraphLaunch(R.graph.exec, s));
            launches++;
            slices++;
            TFIM_CUDA(cudaMemcpyAsync(hst, R.status.p, sizeof(ResStatus), cudaMemcpyDeviceToHost, s));
            const double ts = std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
            TFIM_CUDA(cudaStreamSynchronize(s));
            sync_ms += (std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count() - ts) * 1e3;
            TFIM_TRY(check_search(c, hst->error));
            if (hst->starved || hst->grow) {
                TFIM_TRY(grow_for(*hst));
                continue;
            }
            if (hst->jobs == 0) break;   // the stack and the lookahead queue are empty
            TFIM_CHECK(slices < (1LL << 40), TFIM_E_STATE, "resident search did not finish");
        }
        // per wave: pack, zero, lop3, b1, [proj], tc, gram, expand, masks, index, prune, control
        launches += (int64_t)hst->waves * (11 + (with_proj ? 1 : 0));
        count_launches += (int64_t)hst->waves * (4 + (with_proj ? 1 : 0));
        path_launches[TFIM_PATH_GRAM] += hst->waves;
        path_launches[TFIM_PATH_LOP3] += hst->waves;
        path_launches[TFIM_PATH_B1] += hst->waves;
        path_launches[TFIM_PATH_TC] += hst->waves;
        used_tc = true;
        if (with_proj) path_launches[TFIM_PATH_PROJ] += hst->waves;
    }
    if (loop) TFIM_TRY(grow(R.loop_bar, 16, s));
    while (!use_graph) {
        if (loop) {
            uint32_t* bar = (uint32_t*)R.loop_bar.p;
            TFIM_CUDA(cudaMemsetAsync(bar, 0, 16, s));
            P.launch_id = ++R.launch_id;
            void* args[] = {&P, &bar};
            TFIM_CUDA(cudaLaunchCooperativeKernel((const void*)k_res_loop, dim3(sm_count), dim3(kLoopThreads), args, 0, s));
            count_launches++;
            path_launches[TFIM_PATH_LOP3]++;
        } else {
            k_res_pack<<<1, kPackThreads, 0, s>>>(P);
            TFIM_CUDA(cudaGetLastError());
        }
        launches++;
        const double ts = std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
        TFIM_CUDA(cudaStreamSynchronize(s));
        sync_ms += (std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count() - ts) * 1e3;
        TFIM_TRY(check_search(c, hst->error));
        if (hst->starved || hst->grow) {
            TFIM_TRY(grow_for(*hst));
            continue;
        }
        if (loop && hst->loop_go == 2) continue;   // the launch's time limit: go on
        if (hst->jobs == 0) break;
        TFIM_CUDA(cudaMemsetAsync(R.counts.p, 0, (size_t)hst->out_total * 4, s));
        CountArgs a;
        if (*projected) a.vrows = P.vrows, a.n_base = P.n_base;
        a.pk_list = P.pk_list; a.status = c->d_status.as<int32_t>();
        a.bitmap = c->d_bitmap; a.W = W; a.masks = c->d_masks.as<uint32_t>(); a.jobs = P.jobs; a.rows = P.rows;
        a.cols = P.items; a.out = P.counts; a.job_list = P.proj_list;
        if (hst->tiles_l3) {
            // dense families' tiles (the first tiles_l3d), then the zero-skipping ones
            a.ph_s = &d_st->ph_s[kPhLop3]; a.ph_e = &d_st->ph_e[kPhLop3];
            if (hst->tiles_l3d) {
                a.tiles = P.tiles_l3;
                a.n_tiles = hst->tiles_l3d;
                TFIM_TRY(launch_count_lop3_dense(a, s));
                launches++;
                count_launches++;
            }
            if (hst->tiles_l3 > hst->tiles_l3d) {
                a.tiles = P.tiles_l3 + hst->tiles_l3d;
                a.n_tiles = hst->tiles_l3 - hst->tiles_l3d;
                TFIM_TRY(launch_count_lop3(a, s));
                launches++;
                count_launches++;
            }
            path_launches[TFIM_PATH_LOP3]++;
        }
        if (hst->tiles_b1) {
            a.tiles = P.tiles_b1;
            a.n_tiles = hst->tiles_b1;
            a.ph_s = &d_st->ph_s[kPhB1]; a.ph_e = &d_st->ph_e[kPhB1];
            TFIM_TRY(launch_count_b1(a, s));
            launches++;
            count_launches++;
            path_launches[TFIM_PATH_B1]++;
        }
        if (hst->tiles_tc) {
            a.tiles = P.tiles_tc;
            a.n_tiles = hst->tiles_tc;
            a.ph_s = &d_st->ph_s[kPhTc]; a.ph_e = &d_st->ph_e[kPhTc];
            TFIM_TRY(launch_count_pk(a, sm_count, s));
            launches++;
            count_launches++;
            path_launches[TFIM_PATH_TC]++;
            used_tc = true;
        }
        if (hst->tiles_gr) {
            a.tiles = P.tiles_gr;
            a.n_tiles = hst->tiles_gr;
            a.ph_s = &d_st->ph_s[kPhGram]; a.ph_e = &d_st->ph_e[kPhGram];
            TFIM_TRY(launch_count_gram(a, s));
            launches++;
            count_launches++;
            path_launches[TFIM_PATH_GRAM]++;
        }
        if (hst->n_proj) {
            a.ph_s = &d_st->ph_s[kPhProj]; a.ph_e = &d_st->ph_e[kPhProj];
            TFIM_TRY(launch_count_proj(a, P.proj_list, hst->n_proj, c->d_red_off, c->d_red_items, s));
            launches++;
            count_launches++;
            path_launches[TFIM_PATH_PROJ]++;
        }
        const int64_t threads = (int64_t)hst->rows * 32;
        k_res_expand<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(P);
        TFIM_CUDA(cudaGetLastError());
        k_build_masks<<<sm_count * 8, 256, 0, s>>>(P);
        TFIM_CUDA(cudaGetLastError());
        if (sup_on) {
            k_index_mfis<<<sm_count, 256, 0, s>>>(P);
            k_prune_stack<<<sm_count, 256, 0, s>>>(P);
            TFIM_CUDA(cudaGetLastError());
            launches += 2;
        }
        launches++;
        launches++;
        host_waves++;
    }
    waves += host_waves + (int64_t)hst->waves;   // the graph's or the device loop's, and the host's
    // results
    const auto t_read0 = std::chrono::steady_clock::now();
    const ResStatus fin = *hst;
    // the MFIs in output order (sorted on the device) through one pinned staging buffer:
    // sort keys, lengths, supports, items
    const int32_t nm = fin.mfi_n;
    const int64_t ni = fin.mfi_item_n;
    TFIM_TRY(R.h_res.reserve(((size_t)nm * 4 + (size_t)ni + 8) * 4));   // (whole 16-byte pieces)
    uint64_t* hkey = R.h_res.as<uint64_t>();
    int32_t* hlen = (int32_t*)(hkey + nm);
    int32_t* hsup = hlen + nm;
    int32_t* hitems = hsup + nm;
    if (nm) {
        refresh_ptrs();
        TFIM_TRY(order_mfis(R, c, P, nm, ni, sm_count, s, hkey, hlen, hitems));
    }
    if (o->log_lookahead && fin.log_n) {
        c->la_feats.resize((size_t)fin.log_n * 32);
        c->la_labels.resize(fin.log_n);
        TFIM_CUDA(cudaMemcpyAsync(c->la_feats.data(), R.log_feat.p, (size_t)fin.log_n * 32 * 4, cudaMemcpyDeviceToHost, s));
        TFIM_CUDA(cudaMemcpyAsync(c->la_labels.data(), R.log_label.p, (size_t)fin.log_n * 4, cudaMemcpyDeviceToHost, s));
    }
    const bool used_f4 = top_i8 && top_mode == 1 && !top_loop;
    TFIM_TRY(c->h_status.reserve(64));
    int32_t* status = c->h_status.as<int32_t>();
    *status = 0;
    if (used_f4 || used_tc) TFIM_CUDA(cudaMemcpyAsync(status, c->d_status.p, 4, cudaMemcpyDeviceToHost, s));
    TFIM_CUDA(cudaStreamSynchronize(s));
    TFIM_TRY(tensor_status_check(*status));
    {
        MfiSet& M = c->mfis;
        const bool fresh = M.size() == 0;
        const size_t kbase = M.size();
        M.items.insert(M.items.end(), hitems, hitems + ni);
        M.sup.insert(M.sup.end(), hsup, hsup + nm);
        M.off.resize(kbase + 1 + (size_t)nm);
        for (int32_t k = 0; k < nm; k++) M.off[kbase + k + 1] = M.off[kbase + k] + hlen[k];
        if (fresh) {
            finish_mfi_order(M, hkey);
            M.ordered = true;
        } else {
            // appended to earlier results: long lists sorted here, the whole set by the caller
            for (size_t k = kbase; k < M.size(); k++)
                if (M.off[k + 1] - M.off[k] > 64)
                    std::sort(M.items.begin() + M.off[k], M.items.begin() + M.off[k + 1], std::greater<int32_t>());
            M.ordered = false;
        }
    }
    stt->nodes += (int64_t)fin.nodes;
    stt->supports += (int64_t)fin.supports;
    stt->lookaheads += (int64_t)fin.lookaheads;
    stt->lookahead_hits += (int64_t)fin.hits;
    stt->lookaheads_skipped += (int64_t)fin.skipped;
    stt->pruned_pep += (int64_t)fin.pep;
    stt->pruned_superset += (int64_t)fin.sup_pruned;
    // device times: the empty-prefix family's counting (events) and every later wave's phases
    // (stamps folded by the pack)
    {
        if (!top_loop) {
            float top_ms = 0;
            cudaEventElapsedTime(&top_ms, c->ev0, c->ev1);
            stt->top_ms += top_ms;
            kernel_ms += top_ms;
            stt->path_ms[top_path] += top_ms;
            stt->path_bytes[top_path] += bytes_alg;
            stt->path_bitops[top_path] += top_mode == 2 ? 0 : (int64_t)n0 * (n0 + 1) / 2 * c->n_bits;
            stt->path_supports[top_path] += top_out;
        }
        const double ns = 1e-6;
        const int ph_of_path[6] = {kPhLop3, kPhB1, kPhTc, -1, kPhProj, kPhGram};
        const int cls_of_path[6] = {kClsLop3, kClsB1, kClsTc, -1, kClsProj, kClsGram};
        for (int q = 0; q < 6; q++) {
            if (ph_of_path[q] >= 0) {
                const double ms = (double)fin.ph_ns[ph_of_path[q]] * ns;
                stt->path_ms[q] += ms;
                kernel_ms += ms;
            }
            if (cls_of_path[q] >= 0) {
                stt->path_bytes[q] += (int64_t)fin.cls_bytes[cls_of_path[q]];
                stt->path_bitops[q] += (int64_t)fin.cls_bitops[cls_of_path[q]];
                stt->path_supports[q] += (int64_t)fin.cls_sup[cls_of_path[q]];
                bytes_alg += (int64_t)fin.cls_bytes[cls_of_path[q]];
            }
            stt->path_launches[q] += path_launches[q];
        }
        stt->pack_ms += (double)fin.ph_ns[kPhPack] * ns;
        stt->zero_ms += (double)fin.ph_ns[kPhZero] * ns;
        stt->expand_ms += (double)fin.ph_ns[kPhExpand] * ns;
        stt->mask_ms += (double)fin.ph_ns[kPhMasks] * ns;
    }
    stt->waves += waves;
    stt->launches += launches;
    stt->count_launches += count_launches;
    stt->kernel_ms += kernel_ms;
    stt->sync_ms += sync_ms;
    stt->bytes_alg += bytes_alg;
    stt->bit_ops = stt->supports * c->n_bits;
    stt->readback_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_read0).count();
    return TFIM_OK;
}
}  // namespace

int mine_resident(tfim_ctx* c, const tfim_mine_opts* o, tfim_mine_stats* stt) {
    const tfim_mine_stats before = *stt;
    bool projected = false;
    int rc = search_resident(c, o, stt, true, &projected);
    if (rc == TFIM_E_NOMEM && projected) {
        // the search's pools found no room beside the projected rows: once more without these
        TFIM_CUDA(cudaStreamSynchronize(c->stream));
        dev_free(c->resident->pj_pool.p, c->stream);
        c->resident->pj_pool = Pool{};
        TFIM_CUDA(cudaStreamSynchronize(c->stream));
        dev_trim(c->device);
        c->mfis.clear();
        *stt = before;
        projected = false;
        rc = search_resident(c, o, stt, false, &projected);
    }
    return rc;
}

}  // namespace tfim
