// Tensor-core counter for family jobs: packed Gram tiles on tcgen05.mma kind::mxf4.
//
// A family job counts popc(base & B[F[t]] & B[F[c]]) for the tail rows t (a run of F's
// entries) against every column c of F.  With the base ANDed into the columns,
// X_c = base & B[F[c]], the job is a Gram block of X: counts[t][c] = <X_t, X_c> over the
// transactions.  The arithmetic is the reference's (a support is a popcount of ANDed bit rows,
// code/engine/src/kernel_bmma.cu:636-768, there with WMMA b1).
//
// One tile holds the X rows of several jobs (their K ranges need not be the same transactions:
// only products within a job are read), expanded once to 4-bit values and used as both
// operands: A is all 128 rows, B the window of units that hold tail rows.  The expansion and
// its exactness are count_f4.cu's: nibble masks as the e2m1 values 0.5, 1 and 2, uniform block
// scales, FP32 sums of at most 2^23 transactions per tile.
//
// Layout: jobs of up to 8, 16, 24, 32, 40, 64 or 128 columns share a tile 16, 8, 5, 4, 3, 2 or 1
// at a time.  A unit is 8 columns of one job; unit u holds columns 8 (u / per) .. + 8 of the
// tile's job u % per, so the tail rows of all jobs, which are their first columns, lie in the first
// units and the B window is short.
//
// Why: per 64 transactions a tile of 128 columns moves 4 KiB of expanded rows into shared
// memory, the loads return 1 KiB and the MMA reads 4 KiB and the window, about 110 cycles of the
// shared-memory pipe whatever the number of tail rows (128 measured), while AND + popc spends
// rows x columns / 8 cycles: the two meet near eight tail rows per job.  Measured on the
// 6.3M-row dense database (267 items, minsup 6%): the families this kernel takes need 10.3 ms
// of a mine; the byte-expanding kind::i8 tiles of one family each that it replaces and the
// CUDA-core tiles needed 16.9 ms for the same.
//
// Warp roles (672 threads, one CTA per SM, tiles dealt round-robin):
//   warps 0..15 : expansion.  Per stage (1,024 transactions) a warp expands two units of 512
//                 bits; a lane loads one 16-byte piece of its row and of the job's base two
//                 stages ahead into registers;
//   warp 16     : one lane issues the stage's 16 MMAs and commits them to its `empty` barrier;
//   warps 17..20: read the finished accumulator (two of them, so that the next tile runs
//                 meanwhile) and add each job's block to its counts.
// Every mbarrier wait is bounded; on expiry the kernel records an error, stops, drains what it
// issued and frees its tensor memory.
#include <algorithm>
#include <atomic>

#include "tfim_internal.h"
#include "tcgen05.cuh"

namespace tfim {
namespace {

constexpr int kPUnits = 16;                      // units of 8 X rows
constexpr int kPChunks = 2;                      // chunks of 512 bits per stage
constexpr int kPStageWords = 16 * kPChunks;
constexpr int kPBlockBytes = kPUnits * 8 * 128;  // one K block (256 bits as nibbles) of 128 rows
constexpr int kPStageBytes = 2 * kPChunks * kPBlockBytes;   // 64 KiB
constexpr int kPStages = 3;
constexpr int kPExpWarps = 16;
constexpr int kPThreads = 32 * (kPExpWarps + 1 + 4);
constexpr int kPAhead = 2;
constexpr int kPSmem = kPStages * kPStageBytes + 1024;
constexpr uint32_t kPScale = 256;                // accumulators at columns 0 and 128, scales from here

struct PkShared {
    uint64_t full[kPStages], empty[kPStages], acc_full[2], acc_empty[2], drain;
    uint32_t tmem;
};

// The units [u0, u1) that hold the tile's tail rows (whole warp; the same on every lane).
__device__ __forceinline__ void pk_window(const CountArgs& a, const TileDesc& t, int per, int lane, int& u0, int& u1) {
    int lo = 1 << 20, hi = 0;
    if (lane < t.nr) {
        const JobDesc& j = a.jobs[a.pk_list[t.job + lane]];
        lo = j.r0 >> 3;
        hi = (j.r0 + j.n_rows + 7) >> 3;
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    u0 = (lo * per) & ~1;                     // N is a multiple of 16 rows
    u1 = min(kPUnits, (hi * per + 1) & ~1);
}

__global__ void __launch_bounds__(kPThreads, 1) k_count_pk(CountArgs a_val, const CountArgs* __restrict__ a_dev,
                                                           const int32_t* n_tiles_p, int32_t n_tiles_h) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) PkShared sh;
    const CountArgs a = a_dev ? *a_dev : a_val;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int32_t n_tiles = n_tiles_p ? *n_tiles_p : n_tiles_h;
    phase_begin(a.ph_s);
    if ((int32_t)blockIdx.x < n_tiles) {
        if (tid == 0) {
            for (int s = 0; s < kPStages; s++) {
                mbar_init(smem_u32(&sh.full[s]), kPExpWarps);
                mbar_init(smem_u32(&sh.empty[s]), 1);
            }
            for (int b = 0; b < 2; b++) {
                mbar_init(smem_u32(&sh.acc_full[b]), 1);
                mbar_init(smem_u32(&sh.acc_empty[b]), 4);
            }
            mbar_init(smem_u32(&sh.drain), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        if (warp == kPExpWarps) tmem_alloc(smem_u32(&sh.tmem), 512);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tmem = sh.tmem;
        if (warp < 4) tmem_fill_scales(tmem + ((uint32_t)(32 * warp) << 16) + kPScale);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();

        bool ok = true;
        if (warp == kPExpWarps) {
            // ---- MMA issue
            uint32_t it = 0;   // stages so far
            int i = 0;         // tiles so far
            for (int32_t ti = blockIdx.x; ti < n_tiles && ok; ti += gridDim.x, i++) {
                const TileDesc t = a.tiles[ti];
                int u0, u1;
                pk_window(a, t, t.c0, lane, u0, u1);
                const int n_st = (t.w1 - t.w0) / kPStageWords;
                if (lane == 0) {
                    const uint32_t idesc = idesc_mxf4(8 * (u1 - u0)), acc = tmem + 128u * (uint32_t)(i & 1);
                    if (i >= 2) ok = mbar_wait(smem_u32(&sh.acc_empty[i & 1]), (uint32_t)(i / 2 - 1) & 1u);
                    tc_fence_after();
                    for (int st = 0; st < n_st && ok; st++) {
                        const uint32_t s = (it + st) % kPStages;
                        ok = mbar_wait(smem_u32(&sh.full[s]), ((it + st) / kPStages) & 1u);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t stage = base + s * kPStageBytes;
#pragma unroll
                        for (int kb = 0; kb < 2 * kPChunks; kb++) {
                            const uint32_t blk = stage + (uint32_t)kb * kPBlockBytes;
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                mma_mxf4(acc, smem_desc(blk + k * 32), smem_desc(blk + (uint32_t)u0 * 1024u + k * 32), idesc,
                                         tmem + kPScale + kScaleCols * (uint32_t)min(k, 2), (st > 0 || kb > 0 || k > 0) ? 1u : 0u);
                        }
                        tc_commit(smem_u32(&sh.empty[s]));
                    }
                    if (ok) tc_commit(smem_u32(&sh.acc_full[i & 1]));
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                it += (uint32_t)n_st;
            }
            if (lane == 0) {   // every MMA issued is done before the tensor memory is freed
                tc_commit(smem_u32(&sh.drain));
                if (!mbar_wait(smem_u32(&sh.drain), 0)) ok = false;
            }
            __syncwarp();
        } else if (warp < kPExpWarps) {
            // ---- expansion.  Lane -> (row of the unit, 16-byte piece): the eight lanes of a store phase
            // hold rows of one parity and the two pieces of one K block, so chunk ^ row takes eight
            // different values
            const int q = lane >> 3, l8 = lane & 7;
            const int row = 2 * (l8 >> 1) + (q >> 1), piece = 2 * (q & 1) + (l8 & 1);
            const uint32_t c0 = (uint32_t)(piece & 1), rx = (uint32_t)row;
            const uint32_t dst = base + (uint32_t)(piece >> 1) * kPBlockBytes + (uint32_t)(warp * 8 + row) * 128u;
            uint32_t it = 0;
            for (int32_t ti = blockIdx.x; ti < n_tiles && ok; ti += gridDim.x) {
                const TileDesc t = a.tiles[ti];
                const int per = t.c0;
                const int n_st = (t.w1 - t.w0) / kPStageWords;
                // unit `warp` of the tile: 8 columns of one job (columns past its last repeat it)
                const int ji = warp % per, cb = warp / per;
                const uint32_t* src = nullptr;
                const uint32_t* bas = nullptr;
                int lim = 0;   // stages with words of this job
                if (ji < t.nr) {
                    const JobDesc j = a.jobs[a.pk_list[t.job + ji]];
                    if (8 * cb < j.n_cols) {
                        const int64_t w = t.w0 + piece * 4;
                        src = item_row(a, a.cols[j.col_off + min(8 * cb + row, j.n_cols - 1)]) + w;
                        if (j.base_slot >= 0) bas = a.masks + (int64_t)j.base_slot * a.W + w;
                        else if (j.base_item >= 0) bas = item_row(a, j.base_item) + w;
                        lim = min(n_st, max(0, (j.words - t.w0) / kPStageWords));
                    }
                }
                const bool on = src != nullptr;   // warp-uniform: whole units are absent
                uint4 px[kPAhead][kPChunks], pb[kPAhead][kPChunks];
                auto load = [&](int st, uint4 (&x)[kPChunks], uint4 (&b)[kPChunks]) {
#pragma unroll
                    for (int c = 0; c < kPChunks; c++) {
                        x[c] = make_uint4(0, 0, 0, 0);
                        b[c] = make_uint4(~0u, ~0u, ~0u, ~0u);
                        if (st < lim) {
                            x[c] = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)st * kPStageWords + c * 16));
                            if (bas) b[c] = __ldg(reinterpret_cast<const uint4*>(bas + (int64_t)st * kPStageWords + c * 16));
                        }
                    }
                };
#pragma unroll
                for (int d = 0; d < kPAhead; d++) load(d, px[d], pb[d]);
                for (int st0 = 0; st0 < n_st && ok; st0 += kPAhead) {
#pragma unroll
                    for (int d = 0; d < kPAhead; d++) {
                        const int st = st0 + d;
                        if (st >= n_st) break;
                        const uint32_t s = (it + st) % kPStages;
                        if (it + st >= kPStages) ok = mbar_wait(smem_u32(&sh.empty[s]), ((it + st) / kPStages - 1u) & 1u);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        if (on) {
#pragma unroll
                            for (int c = 0; c < kPChunks; c++) {
                                const uint4 x = make_uint4(px[d][c].x & pb[d][c].x, px[d][c].y & pb[d][c].y,
                                                           px[d][c].z & pb[d][c].z, px[d][c].w & pb[d][c].w);
                                store_nibbles(dst + s * kPStageBytes + (uint32_t)c * 2 * kPBlockBytes, c0, rx, x);
                            }
                        }
                        load(st + kPAhead, px[d], pb[d]);
                        // generic-proxy stores -> visible to the tensor cores' async proxy
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&sh.full[s]));
                    }
                }
                it += (uint32_t)n_st;
            }
        } else {
            // ---- epilogue: lane m of the accumulator is X row m, its column n row 8 u0 + n
            const int quad = warp & 3, m = 32 * quad + lane;
            int i = 0;
            for (int32_t ti = blockIdx.x; ti < n_tiles && ok; ti += gridDim.x, i++) {
                const TileDesc t = a.tiles[ti];
                const int per = t.c0;
                int u0, u1;
                pk_window(a, t, per, lane, u0, u1);
                const int ji = (m >> 3) % per, col = 8 * ((m >> 3) / per) + (m & 7);
                int32_t* out = nullptr;
                int r0 = 0, nr = 0, nc = 0;
                if (ji < t.nr) {
                    const JobDesc j = a.jobs[a.pk_list[t.job + ji]];
                    if (col < j.n_cols) {
                        out = a.out + j.out_off + col;
                        r0 = j.r0;
                        nr = j.n_rows;
                        nc = j.n_cols;
                    }
                }
                ok = mbar_wait(smem_u32(&sh.acc_full[i & 1]), (uint32_t)(i / 2) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                for (int u = u0; u < u1; u += 2) {
                    uint32_t v[16];
                    tmem_ld16(tmem + 128u * (uint32_t)(i & 1) + ((uint32_t)(32 * quad) << 16) + 8u * (uint32_t)(u - u0), v);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        if (!out || (u + h) % per != ji) continue;
                        const int t0 = 8 * ((u + h) / per) - r0;   // row of the job of the unit's first column
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const int32_t n = __float2int_rn(__uint_as_float(v[8 * h + k]));
                            if (n && t0 + k >= 0 && t0 + k < nr) atomicAdd(out + (int64_t)(t0 + k) * nc, n);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh.acc_empty[i & 1]));
            }
        }
        if (!ok && lane == 0) atomicExch(a.status, 1);
        tc_fence_before();
        __syncthreads();
        if (warp == kPExpWarps) tmem_free(tmem, 512);
    }
    phase_end(a.ph_e);
}

}  // namespace

int configure_pk_kernel() {
    static std::atomic<bool> configured[64];
    int dev = 0;
    TFIM_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev].load()) {
        TFIM_CUDA(cudaFuncSetAttribute(k_count_pk, cudaFuncAttributeMaxDynamicSharedMemorySize, kPSmem));
        configured[dev].store(true);
    }
    return TFIM_OK;
}

int launch_count_pk(const CountArgs& a, int32_t sms, cudaStream_t s) {
    if (a.n_tiles <= 0) return TFIM_OK;
    TFIM_TRY(configure_pk_kernel());
    k_count_pk<<<std::min(a.n_tiles, sms), kPThreads, kPSmem, s>>>(a, nullptr, nullptr, a.n_tiles);
    TFIM_CUDA(cudaGetLastError());
    return TFIM_OK;
}

int launch_count_pk_persistent(const CountArgs* d_args, const int32_t* d_n_tiles, int32_t grid, cudaStream_t s) {
    TFIM_TRY(configure_pk_kernel());
    CountArgs none;
    k_count_pk<<<grid, kPThreads, kPSmem, s>>>(none, d_args, d_n_tiles, 0);
    TFIM_CUDA(cudaGetLastError());
    return TFIM_OK;
}

}  // namespace tfim
