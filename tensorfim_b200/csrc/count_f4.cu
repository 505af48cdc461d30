// Tensor-core wave counter on the 5th-generation tensor cores: tcgen05.mma kind::mxf4 on the
// bits expanded to 4-bit values.
//
// The AND+popc block of a count job, popc(A_r & B_c), is the dot product of the rows' 0/1
// vectors.  This counter expands bits to e2m1 values in shared memory and multiplies them
// with tcgen05.mma.cta_group::1.kind::mxf4 into a 128 x 256 accumulator in tensor memory.  The
// arithmetic is the reference's (a support is a popcount of ANDed bit rows,
// code/engine/src/kernel_bmma.cu:636-768, there computed by WMMA b1).  It is exact: every product
// is 0 or 1, the accumulator is FP32, and a tile covers at most 2^23 transactions, so every
// partial sum is an integer below 2^24; partial sums of different tiles meet in int32.
//
// Expansion without shifts per bit: the nibble masks 0x1, 0x2 and 0x4 of a word pick bits as
// the e2m1 values 0.5, 1 and 2, and (word >> 1) & 0x4 picks the last bit as 2.  All 16-byte
// chunks of one MMA (K = 64) hold the same value, and the block scale factors (2, 1, 1/2 on
// both operands) bring its products back to 0 or 1.  A scale region of tensor memory holds
// one value in every byte, so it does not depend on the scale factors' layout.
//
// Tile (TileDesc): columns [c0, c1) (at most 128, the accumulator's lanes, the A operand) x rows
// [r0, r0 + nr) (at most 256, its columns, the B operand) over words [w0, w1), one CTA.  A chunk is 512
// bits of K.
//
// Shared memory bounds the kernel: with both operands there, a 128 x 256 tile writes 12 KiB and
// the MMA reads 12 KiB per K = 64, beside what the loads return.  So a wide tile (more than 22
// units of 8 columns or rows) keeps only B in shared memory, two stages of a chunk each, and
// expands A into tensor memory (tcgen05.st; lane = column, 64 cells per chunk, two stages),
// which the MMA reads at no cost to shared memory.  A narrow tile keeps both in shared memory: its
// time is the hand-over of stages, so a stage is 2 or 4 chunks (8.4M transactions x 69 items x 1 row:
// 78 us with one chunk per stage, 55 us with four).  Operands in shared memory lie in the K-major
// 128-byte-swizzle layout, two K blocks of 256 bits per chunk.
// Measured: 2,048 x 512 x 8.4M 4.37 ms with A in shared memory, 3.51 ms so (2.5e15 bit-op/s);
// 300 x 6,162 x 1M 1.06 and 0.91 ms.
//
// Warp roles (544 threads):
//   warps 0..15: expansion.  Of B (narrow tiles: of both) a unit is 8 rows x 512 bits; a lane loads
//                one 16-byte piece (a warp's load covers 64 contiguous bytes of each row) two to
//                eight stages ahead into registers and stores its four words as four chunks;
//                lanes are placed so that the eight lanes of a store phase hit different banks.
//                In wide tiles warps 0..7 expand A and warps 8..15 B;
//   warp 16    : one lane issues the stage's MMAs and commits them to its `empty` barrier.
// Then all expansion warps read the accumulator (lane = column of the job, so the int32
// atomics of a row are coalesced).  Every mbarrier wait is bounded; on expiry the kernel
// records an error, stops issuing, drains what it issued and frees its tensor memory.
#include <algorithm>
#include <atomic>

#include "tfim_internal.h"
#include "tcgen05.cuh"

namespace tfim {
namespace {

constexpr int kQM = kF4Cols, kQN = kF4Rows;
constexpr int kQChunkWords = 16;                 // a chunk: 512 bits of K
constexpr int kQBlocks = 2;                      // K blocks (256 bits, 128 bytes of nibbles) per chunk
constexpr int kQExpWarps = 16;
constexpr int kQThreads = 32 * (kQExpWarps + 1);
constexpr int kQUnits = 3;                       // units of 8 rows per warp and stage, at most
constexpr int kQFlight = 8;                      // 16-byte loads in flight per lane: units x stages ahead
constexpr int kQMaxStages = 6;
constexpr int kQStaged = 2 * (kQM + kQN) * 128 * kQBlocks;   // two stages of the widest tile
// In shared memory the A operand spans 128 rows from its block's start whatever a narrow tile's width:
// past its columns it runs into the rows behind them (what it adds is not read), and past the
// last block into a guard of 16 KiB.  What shared memory leaves is the L1 cache that the loads in
// flight need, so launches of wide tiles alone take no more than their two stages.
constexpr int kQGuard = kQM * 128;
constexpr int kQNarrow = 22;
static_assert(2 * 2 * kQNarrow * 2048 + kQGuard <= kQStaged, "two stages of a narrow tile and the guard fit");
constexpr int kQSmem = kQStaged + 1024;
constexpr uint32_t kQTmemCols = 512;
constexpr uint32_t kQScale = 256;                // first scale column
constexpr uint32_t kQACol = kQScale + 3 * kScaleCols;   // wide tiles: the A stages, 64 columns per chunk
constexpr int kQWideStages = 2;                  // stages of a wide tile (B in shared memory, A in tensor memory)
constexpr int kQAWarps = 8;                      // wide tiles: warps that expand A
constexpr int kQWideSmem = kQWideStages * kQBlocks * kQN * 128 + 1024;
static_assert((kQM + kQN) / 8 <= kQUnits * kQExpWarps, "units fit the expansion warps");

// The expansion of one warp: U units of 8 rows (an A unit holds columns of the job, a B unit
// rows), kQFlight / U stages of raw words ahead.  Returns false when a wait expired.
template <int U, int NW = kQExpWarps>
__device__ __forceinline__ bool f4_expand(const CountArgs& a, const TileDesc& t, const JobDesc& j, int units_a, int units_b,
                                          int rb, int kc, uint32_t base, int S, int n_st, uint64_t* full, uint64_t* empty,
                                          int warp, int lane) {
    constexpr int kAhead = kQFlight / U;
    const int64_t W = a.W;
    const int units = units_a + units_b;
    const uint32_t kb_bytes = (uint32_t)(rb + units_b) * 1024u, stage_bytes = (uint32_t)kc * kQBlocks * kb_bytes;
    const int stage_words = kc * kQChunkWords;
    // Lane -> (row of the unit, 16-byte piece): the eight lanes of a store phase hold rows of one
    // parity and the two pieces of one K block, so chunk ^ row takes eight different values
    const int q = lane >> 3, i = lane & 7;
    const int row = 2 * (i >> 1) + (q >> 1), piece = 2 * (q & 1) + (i & 1);
    const uint32_t* src[U];
    uint32_t dst[U];
    bool on[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int ch = (warp + u * NW) / units, un = (warp + u * NW) - ch * units;
        on[u] = ch < kc;
        // rows past the tile repeat its last one: their results are not read
        const uint32_t* p = nullptr;   // null: all ones
        if (on[u]) {
            if (un < units_a) {
                const int c = min(t.c0 + un * 8 + row, t.c1 - 1);
                const int32_t col = c == j.self_col ? -1 : a.cols[j.col_off + c];
                if (col >= 0) p = a.bitmap + (int64_t)col * W;
            } else {
                const RowDesc rd = a.rows[j.row_off + t.r0 + min((un - units_a) * 8 + row, t.nr - 1)];
                if (rd.slot >= 0) p = a.masks + (int64_t)rd.slot * W;
                else if (rd.item >= 0) p = a.bitmap + (int64_t)rd.item * W;
            }
        }
        src[u] = p ? p + t.w0 + ch * kQChunkWords + piece * 4 : nullptr;
        dst[u] = base + (uint32_t)(ch * kQBlocks + (piece >> 1)) * kb_bytes +
                 (uint32_t)((un < units_a ? un : rb + un - units_a) * 8 + row) * 128u;
    }
    const uint32_t c0 = (uint32_t)(piece & 1), rx = (uint32_t)row;
    uint4 pf[kAhead][U];
    auto load = [&](int st, uint4 (&v)[U]) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            v[u] = make_uint4(~0u, ~0u, ~0u, ~0u);
            if (on[u] && src[u] && st < n_st)
                v[u] = __ldg(reinterpret_cast<const uint4*>(src[u] + (int64_t)st * stage_words));
        }
    };
#pragma unroll
    for (int d = 0; d < kAhead; d++) load(d, pf[d]);
    int s = 0;
    uint32_t ph = 1;   // parity to wait for on `empty`: the first pass over the stages waits for nothing
    bool ok = true;
    for (int st0 = 0; st0 < n_st && ok; st0 += kAhead) {
#pragma unroll
        for (int d = 0; d < kAhead; d++) {
            const int st = st0 + d;
            if (st >= n_st) break;
            if (st >= S) ok = mbar_wait(smem_u32(&empty[s]), ph);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t off = (uint32_t)s * stage_bytes;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!on[u]) continue;
                const uint4 x = pf[d][u];
                const uint32_t o = dst[u] + off;
                store_nibbles(o, c0, rx, x);
            }
            load(st + kAhead, pf[d]);
            // generic-proxy stores -> visible to the tensor cores' async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full[s]));
            if (++s == S) {
                s = 0;
                ph ^= 1u;
            }
        }
    }
    return ok;
}

// Expansion of a wide tile's A operand into tensor memory: warp w (0..7) holds lanes 32 (w % 4) .. + 32, a
// column of the job each, and fills stage w / 4 (every other chunk).  A warp load covers 64
// contiguous bytes of eight columns; the words reach their lanes through `raw`, 2 KiB of shared
// memory per warp (16-byte pieces swizzled so that both sides are free of bank conflicts), two of
// its chunks ahead in registers.
__device__ __forceinline__ bool f4_expand_a(const CountArgs& a, const TileDesc& t, const JobDesc& j, int n_st, uint32_t tmem,
                                            uint4* raw, uint64_t* full, uint64_t* empty, int warp, int lane) {
    static_assert(kQWideStages == 2 && kQAWarps == 8, "four warps per stage");
    constexpr int kAhead = 2;
    const int g = lane >> 2, piece = lane & 3, quad = warp & 3, s = warp >> 2;
    const uint32_t* src[4];   // null: all ones
#pragma unroll
    for (int i = 0; i < 4; i++) {
        // columns past the tile's last repeat it: their accumulator lanes are not read
        const int c = min(t.c0 + 32 * quad + 8 * i + g, t.c1 - 1);
        const int32_t col = c == j.self_col ? -1 : a.cols[j.col_off + c];
        src[i] = col >= 0 ? a.bitmap + (int64_t)col * a.W + t.w0 + s * kQChunkWords + piece * 4 : nullptr;
    }
    const int n_own = (n_st + 1 - s) / 2;   // this stage's chunks s, s + 2, ...
    uint4 pf[kAhead][4];
    auto load = [&](int k, uint4 (&v)[4]) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
            if (src[i] && k < n_own) v[i] = __ldg(reinterpret_cast<const uint4*>(src[i] + (int64_t)k * (2 * kQChunkWords)));
        }
    };
#pragma unroll
    for (int d = 0; d < kAhead; d++) load(d, pf[d]);
    bool ok = true;
    for (int k0 = 0; k0 < n_own && ok; k0 += kAhead) {
#pragma unroll
        for (int d = 0; d < kAhead; d++) {
            const int k = k0 + d;
            if (k >= n_own) break;
#pragma unroll
            for (int i = 0; i < 4; i++) raw[(8 * i + g) * 4 + (piece ^ ((g >> 1) & 3))] = pf[d][i];
            load(k + kAhead, pf[d]);
            __syncwarp();
            uint4 x[4];
#pragma unroll
            for (int q = 0; q < 4; q++) x[q] = raw[lane * 4 + (q ^ ((lane >> 1) & 3))];
            __syncwarp();
            if (k > 0) ok = mbar_wait(smem_u32(&empty[s]), (uint32_t)(k - 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t at = tmem + ((uint32_t)(32 * quad) << 16) + kQACol + 64u * (uint32_t)s;
#pragma unroll
            for (int kb = 0; kb < 2; kb++) {
                const uint32_t w[8] = {x[2 * kb].x,     x[2 * kb].y,     x[2 * kb].z,     x[2 * kb].w,
                                       x[2 * kb + 1].x, x[2 * kb + 1].y, x[2 * kb + 1].z, x[2 * kb + 1].w};
                uint32_t v[16];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    v[q] = w[q] & 0x11111111u;
                    v[8 + q] = w[q] & 0x22222222u;
                }
                tmem_st16(at + 32u * kb, v);
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    v[q] = w[q] & 0x44444444u;
                    v[8 + q] = (w[q] >> 1) & 0x44444444u;
                }
                tmem_st16(at + 32u * kb + 16u, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full[s]));
        }
    }
    return ok;
}

__global__ void __launch_bounds__(kQThreads, 1) k_count_f4(CountArgs a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kQMaxStages], empty[kQMaxStages], done;
    __shared__ uint32_t s_tmem;
    __shared__ int32_t s_abort;
    __shared__ __align__(16) uint4 s_raw[kQAWarps][128];
    const TileDesc t = a.tiles[blockIdx.x];
    const JobDesc j = a.jobs[t.job];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int N = (t.nr + 15) & ~15;
    // 8-row units of a K block: the columns', the rows'; rb: where the rows' units begin
    const int units_a = (t.c1 - t.c0 + 7) >> 3, units_b = N >> 3, units = units_a + units_b;
    const bool narrow = units <= kQNarrow;
    const int rb = narrow ? units_a : 0;   // wide tiles hold only rows in shared memory
    const int kc = units <= kQNarrow / 2 ? 4 : narrow ? 2 : 1;   // chunks per stage
    const uint32_t kb_bytes = (uint32_t)(rb + units_b) * 1024u;
    const uint32_t stage_bytes = (uint32_t)kc * kQBlocks * kb_bytes;
    const int S = narrow ? min(kQMaxStages, (kQStaged - kQGuard) / (int)stage_bytes) : kQWideStages;   // at least 2
    const int n_st = (t.w1 - t.w0) / (kc * kQChunkWords);      // word slices are multiples of 64 words

    if (tid == 0) {
        for (int s = 0; s < kQMaxStages; s++) {
            mbar_init(smem_u32(&full[s]), narrow ? kQExpWarps : kQExpWarps - kQAWarps / 2);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(&done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (warp == kQExpWarps) tmem_alloc(smem_u32(&s_tmem), kQTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (warp < 4) tmem_fill_scales(tmem + ((uint32_t)(32 * warp) << 16) + kQScale);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp == kQExpWarps) {
        if (lane == 0) {
            bool ok = true;
            const uint32_t idesc = idesc_mxf4(N);
            const uint32_t to_b = (uint32_t)rb * 1024u;
            auto chunk = [&](uint32_t blk, bool first) {
#pragma unroll
                for (int kb = 0; kb < kQBlocks; kb++) {
                    const uint32_t at = blk + (uint32_t)kb * kb_bytes;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        mma_mxf4(tmem, smem_desc(at + k * 32), smem_desc(at + to_b + k * 32), idesc,
                                 tmem + kQScale + kScaleCols * (uint32_t)min(k, 2), (!first || kb > 0 || k > 0) ? 1u : 0u);
                }
            };
            for (int st = 0; st < n_st; st++) {
                const int s = st % S;
                if (!mbar_wait(smem_u32(&full[s]), (uint32_t)(st / S) & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t stage = base + (uint32_t)s * stage_bytes;
                if (!narrow) {
                    const uint32_t ta = tmem + kQACol + 64u * (uint32_t)s;
#pragma unroll
                    for (int k = 0; k < 4 * kQBlocks; k++)
                        mma_mxf4_ta(tmem, ta + 8u * k, smem_desc(stage + (uint32_t)(k >> 2) * kb_bytes + (k & 3) * 32), idesc,
                                    tmem + kQScale + kScaleCols * (uint32_t)min(k & 3, 2), (st > 0 || k > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&empty[s]));
                    continue;
                }
                chunk(stage, st == 0);
                for (int c = 1; c < kc; c++) chunk(stage + (uint32_t)c * kQBlocks * kb_bytes, false);
                tc_commit(smem_u32(&empty[s]));
            }
            if (!ok) {
                atomicExch(&s_abort, 1);
                atomicExch(a.status, 1);
            }
            tc_commit(smem_u32(&done));   // tracks every MMA issued so far
        }
        __syncwarp();
    } else {
        bool ok;
        if (!narrow)
            ok = warp < kQAWarps
                     ? f4_expand_a(a, t, j, n_st, tmem, s_raw[warp], full, empty, warp, lane)
                     : f4_expand<4, kQExpWarps - kQAWarps>(a, t, j, 0, units_b, 0, 1, base, S, n_st, full, empty,
                                                           warp - kQAWarps, lane);
        else if (kc * units <= kQExpWarps) ok = f4_expand<1>(a, t, j, units_a, units_b, rb, kc, base, S, n_st, full, empty, warp, lane);
        else if (kc * units <= 2 * kQExpWarps)
            ok = f4_expand<2>(a, t, j, units_a, units_b, rb, kc, base, S, n_st, full, empty, warp, lane);
        else ok = f4_expand<3>(a, t, j, units_a, units_b, rb, kc, base, S, n_st, full, empty, warp, lane);
        if (!ok && lane == 0) {
            atomicExch(&s_abort, 1);
            atomicExch(a.status, 1);
        }
        // ---- epilogue: warp w reads lanes 32 * (w % 4) (columns of the job), accumulator columns
        // 16 * (w / 4) + 64 k (rows of the job)
        const bool fin = mbar_wait(smem_u32(&done), 0);
        tc_fence_after();
        const bool all_fin = __all_sync(0xffffffffu, fin);
        if (!all_fin && lane == 0) {
            atomicExch(&s_abort, 1);
            atomicExch(a.status, 1);
        }
        if (all_fin && !*(volatile int32_t*)&s_abort && n_st > 0) {
            const int quad = warp & 3, c = t.c0 + 32 * quad + lane;
            for (int n0 = 16 * (warp >> 2); n0 < N; n0 += 64) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)n0, v);
                if (c < t.c1) {
                    int32_t* out = a.out + j.out_off + (int64_t)(t.r0 + n0) * j.n_cols + c;
#pragma unroll
                    for (int k = 0; k < 16; k++) {
                        const int32_t n = __float2int_rn(__uint_as_float(v[k]));
                        if (n && n0 + k < t.nr) atomicAdd(out + (int64_t)k * j.n_cols, n);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kQExpWarps) tmem_free(tmem, kQTmemCols);
}

}  // namespace

// Tiles of one job of nr rows x nc columns.  The word slices are chosen so that the tiles fill
// whole waves of one CTA per SM: the cheapest count by (waves of CTAs) x (chunks per tile + the
// fixed cost of a tile, about 16 chunks' time: set-up, first loads and epilogue).  A slice holds
// at most 2^18 words (2^23 transactions), so that FP32 sums stay exact.  `upper`: rows and
// columns are the same list and tiles wholly below the diagonal are left out.
bool tiles_f4(int32_t job, int32_t nr, int32_t nc, int64_t W, int sms, std::vector<TileDesc>& out, bool upper) {
    bool wide = true;
    if (nr <= 0 || nc <= 0 || W <= 0) return false;
    std::vector<TileDesc> tl;
    // equal row groups of at most kF4Rows, multiples of 16
    const int32_t groups = (nr + kF4Rows - 1) / kF4Rows;
    const int32_t step = ((nr + groups - 1) / groups + 15) & ~15;
    for (int32_t r0 = 0; r0 < nr; r0 += step)
        for (int32_t c0 = 0; c0 < nc; c0 += kF4Cols) {
            const int32_t c1 = std::min(nc, c0 + kF4Cols);
            if (upper && c1 <= r0) continue;
            tl.push_back(TileDesc{job, r0, std::min(step, nr - r0), c0, c1, 0, 0, 0});
            wide &= (c1 - c0 + 7) / 8 + (std::min(step, nr - r0) + 15) / 16 * 2 > kQNarrow;
        }
    const int64_t blocks = W / kRowAlignWords, base = (int64_t)tl.size();
    int64_t best = 1;
    double best_cost = 1e300;
    const int64_t max_ks = std::min<int64_t>(blocks, std::max<int64_t>(1, 4 * sms / std::max<int64_t>(base, 1)) + (W >> 18) + 1);
    for (int64_t ks = 1; ks <= max_ks; ks++) {
        const int64_t per = (blocks + ks - 1) / ks;
        if (per * kRowAlignWords > (1 << 18)) continue;
        const int64_t n = (blocks + per - 1) / per;
        const double cost = (double)((base * n + sms - 1) / sms) * (double)(per * (kRowAlignWords / kQChunkWords) + 16);
        if (cost < best_cost) {
            best_cost = cost;
            best = per;
        }
    }
    if (best_cost == 1e300) best = (1 << 18) / kRowAlignWords;
    for (int64_t b0 = 0; b0 < blocks; b0 += best)
        for (TileDesc t : tl) {
            t.w0 = (int32_t)(b0 * kRowAlignWords);
            t.w1 = (int32_t)(std::min(blocks, b0 + best) * kRowAlignWords);
            out.push_back(t);
        }
    return wide;
}

int launch_count_f4(const CountArgs& a, bool wide, cudaStream_t s) {
    if (a.n_tiles <= 0) return TFIM_OK;
    static std::atomic<bool> configured[64];
    int dev = 0;
    TFIM_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev].load()) {
        TFIM_CUDA(cudaFuncSetAttribute(k_count_f4, cudaFuncAttributeMaxDynamicSharedMemorySize, kQSmem));
        configured[dev].store(true);
    }
    k_count_f4<<<a.n_tiles, kQThreads, wide ? kQWideSmem : kQSmem, s>>>(a);
    TFIM_CUDA(cudaGetLastError());
    return TFIM_OK;
}

int tensor_status_check(int32_t v) {
    TFIM_CHECK(v == 0, TFIM_E_TIMEOUT, "tensor-core counter: an mbarrier wait expired");
    return TFIM_OK;
}

}  // namespace tfim
