// Device ingest: F1 occurrence histogram, frequency compaction and the vertical bitmap.
//
// Semantics follow the reference's host pipeline (code/engine/src/kernel_bitmap.cu):
//   getItemsFrequenc :269-298   occurrence counts (a repeated id in one row counts twice)
//   main :806                   frequencyThreshold = transNum * supportThreshold (double)
//   reduceTransSet :692-703     drop ids with count < threshold, then empty rows
//   main :815-816               dimensionReduced: ids (0 included) with freq/transNum > thr
//   buildBitmap :342-380        survivors = ids 1..max with count >= threshold, dense ids in
//                               ascending original order; a frequent id 0 is parked after
//                               them; bit t of row x set iff reduced row t holds x
// The work is done on the GPU: one histogram pass, one pass that measures reduced rows,
// a scan that numbers the surviving rows, and one scatter pass that sets the bits.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <numeric>

#include <atomic>

#include "tfim_internal.h"
#include "wave_route.h"

namespace tfim {
namespace {

struct ScanStats {
    int32_t id_min, id_max;
    int32_t neg;        // any negative id seen
    int32_t bad_off;    // any decreasing offset seen
    long long len_min, len_max;
    unsigned long long len_sum;
    long long red_min, red_max;
    unsigned long long red_sum;
    unsigned long long red_sq_sum;   // sum of squared reduced lengths: pair-counting work
};

__global__ void k_item_minmax(const int32_t* __restrict__ items, int64_t nnz, ScanStats* st) {
    int32_t mn = INT_MAX, mx = INT_MIN, neg = 0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        int32_t v = items[j];
        mn = min(mn, v);
        mx = max(mx, v);
        neg |= (v < 0);
    }
    typedef cub::BlockReduce<int32_t, 256> BR;
    __shared__ typename BR::TempStorage t1;
    int32_t bmn = BR(t1).Reduce(mn, cub::Min());
    __syncthreads();
    int32_t bmx = BR(t1).Reduce(mx, cub::Max());
    __syncthreads();
    int32_t bneg = BR(t1).Reduce(neg, cub::Max());
    if (threadIdx.x == 0) {
        atomicMin(&st->id_min, bmn);
        atomicMax(&st->id_max, bmx);
        if (bneg) atomicExch(&st->neg, 1);
    }
}

__global__ void k_row_lengths(const int64_t* __restrict__ off, int64_t n_rows, ScanStats* st) {
    long long mn = LLONG_MAX, mx = 0;
    unsigned long long sum = 0;
    int bad = 0;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
        long long len = (long long)(off[r + 1] - off[r]);
        bad |= (len < 0);
        mn = min(mn, len);
        mx = max(mx, len);
        sum += (unsigned long long)(len > 0 ? len : 0);
    }
    typedef cub::BlockReduce<long long, 256> BR;
    typedef cub::BlockReduce<unsigned long long, 256> BRU;
    typedef cub::BlockReduce<int, 256> BRI;
    __shared__ typename BR::TempStorage t1;
    __shared__ typename BRU::TempStorage t2;
    __shared__ typename BRI::TempStorage t3;
    long long bmn = BR(t1).Reduce(mn, cub::Min());
    __syncthreads();
    long long bmx = BR(t1).Reduce(mx, cub::Max());
    unsigned long long bs = BRU(t2).Sum(sum);
    int bb = BRI(t3).Reduce(bad, cub::Max());
    if (threadIdx.x == 0) {
        atomicMin(&st->len_min, bmn);
        atomicMax(&st->len_max, bmx);
        atomicAdd(&st->len_sum, bs);
        if (bb) atomicExch(&st->bad_off, 1);
    }
}

__global__ void k_hist(const int32_t* __restrict__ items, int64_t nnz, int32_t* __restrict__ freq) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&freq[items[j]], 1);
}

// The same histogram when the id space fits in shared memory: every block counts a strided
// share of the items in a private shared histogram (no global atomics; the skewed ids of a
// long-tailed database collide only within a block) and writes it to partial[block]; the
// column sums are taken by k_hist_sum.
constexpr int kHistSmemBins = 48 * 1024;
__global__ void __launch_bounds__(1024) k_hist_smem(const int32_t* __restrict__ items, int64_t nnz, int32_t bins,
                                                    int32_t* __restrict__ partial) {
    extern __shared__ int32_t h[];
    for (int i = threadIdx.x; i < bins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&h[__ldg(items + j)], 1);
    __syncthreads();
    int32_t* out = partial + (int64_t)blockIdx.x * bins;
    for (int i = threadIdx.x; i < bins; i += blockDim.x) out[i] = h[i];
}
__global__ void k_hist_sum(const int32_t* __restrict__ partial, int32_t parts, int32_t bins, int32_t* __restrict__ freq) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bins) return;
    int32_t v = 0;
    for (int b = 0; b < parts; b++) v += partial[(int64_t)b * bins + i];
    freq[i] = v;
}

// Dense ids from the F1 histogram, one block: survivors (count >= min_count) of the ids 1..bins-1 in
// ascending order, then id 0 if it survives; map[id] = dense id or -1.  On the host the same loops
// over 40,000 ids and the two stable sorts below took 0.45 ms of a 300,000-row open.
struct DenseCounts {
    int32_t n_surv, n_dense, dimension, roots;
};
__global__ void __launch_bounds__(1024) k_dense_ids(const int32_t* __restrict__ freq, int32_t bins, int32_t min_count,
                                                    int32_t root_min, int32_t* __restrict__ map,
                                                    int32_t* __restrict__ dense_to_orig, int32_t* __restrict__ dense_freq,
                                                    DenseCounts* out) {
    typedef cub::BlockScan<int32_t, 1024> Scan;
    __shared__ typename Scan::TempStorage ts;
    __shared__ int32_t s_dim, s_roots;
    if (threadIdx.x == 0) s_dim = s_roots = 0;
    __syncthreads();
    int32_t base = 0;
    for (int64_t i0 = 0; i0 < bins; i0 += 4096) {
        int32_t f[4], on[4], at[4], total = 0, dim = 0, roots = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int64_t i = i0 + threadIdx.x * 4 + q;
            f[q] = i < bins ? freq[i] : 0;
            on[q] = i > 0 && i < bins && f[q] >= min_count;
            dim += f[q] != 0;
            roots += i < bins && f[q] >= root_min;
        }
        Scan(ts).ExclusiveSum(on, at, total);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int64_t i = i0 + threadIdx.x * 4 + q;
            if (i >= bins) break;
            map[i] = on[q] ? base + at[q] : -1;
            if (on[q]) {
                dense_to_orig[base + at[q]] = (int32_t)i;
                dense_freq[base + at[q]] = f[q];
            }
        }
        if (dim) atomicAdd(&s_dim, dim);
        if (roots) atomicAdd(&s_roots, roots);
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int32_t n = base;
        if (freq[0] >= min_count) {   // the parked id 0
            map[0] = n;
            dense_to_orig[n] = 0;
            dense_freq[n] = freq[0];
            n++;
        }
        *out = DenseCounts{base, n, s_dim, s_roots};
    }
}

// A stable order by rank: order[rank of i] = i, larger values first (or smaller first).  A block
// ranks 32 items: each of its 32 warps compares them with a 32nd of all items, and the ranks meet in
// shared memory.  n^2 comparisons, 38M for 6,156 items: 80 us for two orders of 4,000 with
// one thread per item, 14 us so.
constexpr int kRankItems = 32;
__global__ void __launch_bounds__(1024) k_rank_order(const int32_t* __restrict__ value, int32_t n, int descending,
                                                     int32_t* __restrict__ order) {
    __shared__ int32_t rank[kRankItems];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t i = blockIdx.x * kRankItems + lane;
    const int32_t flip = descending ? -1 : 0;   // ~v reverses the order
    const int32_t v = i < n ? value[i] ^ flip : 0;
    if (warp == 0) rank[lane] = 0;
    __syncthreads();
    int32_t r = 0;
    for (int32_t j0 = warp * 32; j0 < n; j0 += 1024) {
        const int32_t x = j0 + lane < n ? value[j0 + lane] ^ flip : INT_MAX;
        const int m = min(32, n - j0);
        for (int k = 0; k < m; k++) {
            const int32_t y = __shfl_sync(0xffffffffu, x, k);
            r += y < v || (y == v && j0 + k < i);
        }
    }
    atomicAdd(&rank[lane], r);
    __syncthreads();
    if (warp == 0 && i < n) order[rank[lane]] = i;
}
constexpr int32_t kRankMax = 1 << 15;   // beyond, the quadratic pass loses to the host's sort

// Row passes over the transaction list give a row to eight lanes: its ids come in 32-byte
// pieces, four rows per warp load, whether rows hold ten ids or a hundred (a thread per row read
// 784,000 rows of 74 ids at 1.9 TB/s in the first pass and 0.7 TB/s in the second).
constexpr int kRowLanes = 8;
__device__ __forceinline__ unsigned row_lanes_mask() { return 0xFFu << (threadIdx.x & 24); }

// Per row: the reduced length (occurrences of ids that survive the threshold, id 0
// included when frequent); 0 marks a row that reduction removes.
__global__ void k_reduced_rows(const int64_t* __restrict__ off, const int32_t* __restrict__ items, int64_t n_rows,
                               const int32_t* __restrict__ map, int32_t* __restrict__ red_len, ScanStats* st) {
    long long mn = LLONG_MAX, mx = 0;
    unsigned long long sum = 0, sq = 0;
    const int l = threadIdx.x & (kRowLanes - 1);
    const unsigned gm = row_lanes_mask();
    const int64_t step = (int64_t)gridDim.x * blockDim.x / kRowLanes;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kRowLanes; r < n_rows; r += step) {
        const int64_t e = off[r + 1];
        int32_t len = 0;
        for (int64_t j = off[r] + l; j < e; j += kRowLanes) len += __ldg(map + items[j]) >= 0;
#pragma unroll
        for (int o = kRowLanes / 2; o > 0; o >>= 1) len += __shfl_xor_sync(gm, len, o);
        if (l == 0) {
            red_len[r] = len;
            if (len > 0) {
                mn = min(mn, (long long)len);
                mx = max(mx, (long long)len);
                sum += (unsigned long long)len;
                sq += (unsigned long long)len * (unsigned long long)len;
            }
        }
    }
    typedef cub::BlockReduce<long long, 256> BR;
    typedef cub::BlockReduce<unsigned long long, 256> BRU;
    __shared__ typename BR::TempStorage t1;
    __shared__ typename BRU::TempStorage t2;
    long long bmn = BR(t1).Reduce(mn, cub::Min());
    __syncthreads();
    long long bmx = BR(t1).Reduce(mx, cub::Max());
    unsigned long long bs = BRU(t2).Sum(sum);
    __syncthreads();
    unsigned long long bq = BRU(t2).Sum(sq);
    if (threadIdx.x == 0) {
        atomicMin(&st->red_min, bmn);
        atomicMax(&st->red_max, bmx);
        atomicAdd(&st->red_sum, bs);
        atomicAdd(&st->red_sq_sum, bq);
    }
}

struct IsPositive {
    __host__ __device__ int32_t operator()(int32_t v) const { return v > 0; }
};

// The reduced transaction list in dense ids (reduced row rr = surviving row r).
__global__ void k_write_reduced(const int64_t* __restrict__ off, const int32_t* __restrict__ items, int64_t n_rows,
                                const int32_t* __restrict__ map, const int32_t* __restrict__ red_len,
                                const int64_t* __restrict__ red_idx, const int64_t* __restrict__ item_off,
                                int64_t* __restrict__ red_off, int32_t* __restrict__ red_items) {
    const int l = threadIdx.x & (kRowLanes - 1);
    const unsigned gm = row_lanes_mask(), below = gm & ((1u << (threadIdx.x & 31)) - 1u);
    const int64_t step = (int64_t)gridDim.x * blockDim.x / kRowLanes;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kRowLanes; r < n_rows; r += step) {
        if (red_len[r] == 0) continue;
        int64_t o = item_off[r];
        if (l == 0) red_off[red_idx[r]] = o;
        const int64_t e = off[r + 1];
        for (int64_t b = off[r]; b < e; b += kRowLanes) {
            const int32_t d = b + l < e ? __ldg(map + items[b + l]) : -1;
            const unsigned keep = __ballot_sync(gm, d >= 0) & gm;
            if (d >= 0) red_items[o + __popc(keep & below)] = d;
            o += __popc(keep);
        }
    }
}

// The bitmap from the reduced list, a block per 32 * wb consecutive reduced rows: their words of
// every item's row are formed in shared memory (n_dense x wb words) and leave whole, in pieces of
// at least a sector, zeros included, so that the bitmap is neither cleared first nor written
// by global atomics.  784,000 rows of 24 ids, 267 items: 543 us with warp-merged global atomics,
// 117 us so.
constexpr int kBitmapMaxDense = 6400;   // items whose 8-word pieces fit shared memory
__global__ void __launch_bounds__(1024) k_build_bitmap(const int64_t* __restrict__ red_off, const int32_t* __restrict__ red_items,
                                                       int64_t n_red, int32_t n_dense, int32_t wb_log,
                                                       uint32_t* __restrict__ bm, int64_t W) {
    extern __shared__ __align__(16) uint32_t tab[];
    const int n4 = n_dense << (wb_log - 2);
    for (int i = threadIdx.x; i < n4; i += blockDim.x) reinterpret_cast<uint4*>(tab)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x << (wb_log + 5), r1 = min(n_red, r0 + (32 << wb_log));
    const int l = threadIdx.x & (kRowLanes - 1);
    for (int64_t r = r0 + threadIdx.x / kRowLanes; r < r1; r += blockDim.x / kRowLanes) {
        const uint32_t bit = 1u << (r & 31), word = (uint32_t)(r - r0) >> 5;
        const int64_t e = red_off[r + 1];
        for (int64_t j = red_off[r] + l; j < e; j += kRowLanes) atomicOr(&tab[((uint32_t)red_items[j] << wb_log) + word], bit);
    }
    __syncthreads();
    const int q_log = wb_log - 2;   // 16-byte pieces per item
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        const int64_t d = i >> q_log;
        reinterpret_cast<uint4*>(bm + d * W + ((int64_t)blockIdx.x << wb_log))[i & ((1 << q_log) - 1)] =
            reinterpret_cast<const uint4*>(tab)[i];
    }
}

// One thread per reduced row: set the row's bit in the row of each of its items.  Rows
// of one warp are consecutive, so their bits for one item share a 32-bit word; the warp
// merges equal (item, word) targets before the atomic.
__global__ void k_scatter_bits(const int64_t* __restrict__ red_off, const int32_t* __restrict__ red_items, int64_t n_red,
                               uint32_t* __restrict__ bm, int64_t W) {
    for (int64_t r0 = blockIdx.x * (int64_t)blockDim.x; r0 < n_red; r0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t rr = r0 + threadIdx.x;
        const bool live = rr < n_red;
        int64_t j = live ? red_off[rr] : 0, je = live ? red_off[rr + 1] : 0;
        while (__any_sync(0xffffffffu, j < je)) {
            int32_t d = -1;
            if (j < je) { d = red_items[j]; j++; }
            const unsigned long long key = d >= 0 ? ((unsigned long long)(uint32_t)d << 32) | (unsigned long long)(rr >> 5) : ~0ull;
            const unsigned peers = __match_any_sync(0xffffffffu, key);
            const uint32_t bit = d >= 0 ? (1u << (rr & 31)) : 0u;
            uint32_t acc = bit;
            for (int k = 0; k < 32; k++) {
                const uint32_t v = __shfl_sync(0xffffffffu, bit, k);
                if ((peers >> k) & 1u) acc |= v;
            }
            const int leader = __ffs(peers) - 1;
            if (d >= 0 && (int)(threadIdx.x & 31) == leader) atomicOr(&bm[(int64_t)d * W + (rr >> 5)], acc);
        }
    }
}

__global__ void k_row_popc(const uint32_t* __restrict__ bm, int64_t W, int32_t n, int32_t* __restrict__ out) {
    const int row = blockIdx.x;
    if (row >= n) return;
    const uint4* p = reinterpret_cast<const uint4*>(bm + (int64_t)row * W);
    unsigned long long s = 0;
    for (int64_t w = threadIdx.x; w < W / 4; w += blockDim.x) {
        uint4 v = p[w];
        s += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    typedef cub::BlockReduce<unsigned long long, 256> BR;
    __shared__ typename BR::TempStorage t;
    unsigned long long b = BR(t).Sum(s);
    if (threadIdx.x == 0) out[row] = (int32_t)b;
}

int grid_for(int64_t n, int per = 256) {
    int64_t g = (n + per - 1) / per;
    if (g < 1) g = 1;
    if (g > 148 * 16) g = 148 * 16;
    return (int)g;
}

}  // namespace

int compute_bit_supports(tfim_ctx* c) {
    // popcount of every bitmap row (the counted ones are the bitmap supports); their sum
    // equals the reduced transaction list's length exactly when no row repeats an id
    const int32_t rows = c->from_db ? c->info.n_dense : c->n_counted;
    std::vector<int32_t> all(std::max<int32_t>(rows, 0), 0);
    if (rows > 0) {
        TFIM_TRY(c->d_scratch[7].reserve((size_t)rows * 8));
        k_row_popc<<<rows, 256, 0, c->stream>>>(c->d_bitmap, c->W, rows, c->d_scratch[7].as<int32_t>());
        TFIM_CUDA(cudaGetLastError());
        TFIM_CUDA(cudaMemcpyAsync(all.data(), c->d_scratch[7].p, (size_t)rows * 4, cudaMemcpyDeviceToHost, c->stream));
        // the counted rows in increasing support (the search's first family)
        c->support_order.clear();
        if (!c->sharded && c->n_counted > 0 && c->n_counted <= kRankMax) {
            c->support_order.resize(c->n_counted);
            int32_t* order = c->d_scratch[7].as<int32_t>() + rows;
            k_rank_order<<<(c->n_counted + kRankItems - 1) / kRankItems, 1024, 0, c->stream>>>(c->d_scratch[7].as<int32_t>(), c->n_counted, 0, order);
            TFIM_CUDA(cudaGetLastError());
            TFIM_CUDA(cudaMemcpyAsync(c->support_order.data(), order, (size_t)c->n_counted * 4, cudaMemcpyDeviceToHost, c->stream));
        }
        TFIM_CUDA(cudaStreamSynchronize(c->stream));
    }
    int64_t total = 0;
    for (int32_t v : all) total += v;
    c->csr_exact = c->from_db && c->d_red_off && total == c->n_red_items;
    if (c->sharded) {
        // row supports summed over the shards; the list counters are exact only if every shard's list is
        if (rows > 0) {
            TFIM_TRY(group_reduce(c, c->d_scratch[7].p, rows, TFIM_DT_I32, TFIM_RED_SUM, c->stream));
            TFIM_CUDA(cudaMemcpyAsync(all.data(), c->d_scratch[7].p, (size_t)rows * 4, cudaMemcpyDeviceToHost, c->stream));
            TFIM_CUDA(cudaStreamSynchronize(c->stream));
        }
        int64_t inexact = c->csr_exact ? 0 : 1;
        TFIM_TRY(group_reduce_host(c, &inexact, 1, TFIM_RED_MAX));
        c->csr_exact = inexact == 0;
    }
    c->bit_support.assign(all.begin(), all.begin() + std::min<int32_t>(rows, c->n_counted));
    c->empty_share = empty_pieces(c->bit_support.data(), (int64_t)c->bit_support.size(), c->sharded ? c->n_bits_total : c->n_bits);
    return TFIM_OK;
}

int ingest_csr(tfim_ctx* c, const int64_t* h_off, const int32_t* h_items, int64_t n_rows, double thr) {
    cudaStream_t s = c->stream;
    const int64_t base = n_rows > 0 ? h_off[0] : 0;
    TFIM_CHECK(base == 0, TFIM_E_INVALID, "row_offsets[0] must be 0");
    const int64_t nnz = n_rows > 0 ? h_off[n_rows] : 0;
    TFIM_CHECK(nnz >= 0, TFIM_E_INVALID, "row_offsets[n_rows] is negative");
    DevBuf d_off, d_items;
    d_off.stream = d_items.stream = s;
    int rc = TFIM_OK;
    if (!(rc = d_off.reserve((size_t)(n_rows + 1) * 8)) && !(rc = d_items.reserve((size_t)std::max<int64_t>(nnz, 1) * 4))) {
        if (cudaMemcpyAsync(d_off.p, h_off, (size_t)(n_rows + 1) * 8, cudaMemcpyHostToDevice, s) != cudaSuccess ||
            (nnz > 0 && cudaMemcpyAsync(d_items.p, h_items, (size_t)nnz * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)) {
            set_error("host-to-device copy of the transaction set failed");
            rc = TFIM_E_CUDA;
        } else {
            rc = ingest_device_csr(c, d_off.as<int64_t>(), d_items.as<int32_t>(), n_rows, nnz, thr);
        }
    }
    d_off.release();
    d_items.release();
    return rc;
}

int ingest_device_csr(tfim_ctx* c, const int64_t* d_off_p, const int32_t* d_items_p, int64_t n_rows, int64_t nnz,
                      double thr) {
    cudaStream_t s = c->stream;
    DevBuf d_stats, d_freq, d_map, d_flag, d_idx, d_tmp;
    for (DevBuf* b : {&d_stats, &d_freq, &d_map, &d_flag, &d_idx, &d_tmp}) b->stream = s;
    int rc = TFIM_OK;
    ScanStats hs{};
    int64_t id_max = 0, id_min = INT_MAX;
    // all device scratch below is released at the end of this function
    auto done = [&](int r) {
        d_stats.release(); d_freq.release();
        d_map.release(); d_flag.release(); d_idx.release(); d_tmp.release();
        return r;
    };
    if ((rc = d_stats.reserve(sizeof(ScanStats)))) return done(rc);
    hs.id_min = INT_MAX; hs.id_max = INT_MIN; hs.len_min = LLONG_MAX; hs.red_min = LLONG_MAX;
    cudaMemcpyAsync(d_stats.p, &hs, sizeof hs, cudaMemcpyHostToDevice, s);
    if (nnz > 0) k_item_minmax<<<grid_for(nnz), 256, 0, s>>>(d_items_p, nnz, d_stats.as<ScanStats>());
    if (n_rows > 0) k_row_lengths<<<grid_for(n_rows), 256, 0, s>>>(d_off_p, n_rows, d_stats.as<ScanStats>());
    cudaMemcpyAsync(&hs, d_stats.p, sizeof hs, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) { set_error("ingest statistics pass failed: %s", cudaGetErrorString(cudaGetLastError())); return done(TFIM_E_CUDA); }
    int64_t n_rows_all = n_rows, nnz_all = nnz;
    if (c->sharded) {
        // the whole database's statistics: errors, id range and row lengths (MIN as -MAX(-x))
        int64_t mx[6] = {hs.neg, hs.bad_off, nnz > 0 ? (int64_t)hs.id_max : -1, n_rows > 0 ? (int64_t)hs.len_max : 0,
                         nnz > 0 ? -(int64_t)hs.id_min : -(int64_t)INT_MAX, n_rows > 0 ? -(int64_t)hs.len_min : -(int64_t)LLONG_MAX};
        int64_t sm[3] = {n_rows, (int64_t)hs.len_sum, nnz};
        if ((rc = group_reduce_host(c, mx, 6, TFIM_RED_MAX)) || (rc = group_reduce_host(c, sm, 3, TFIM_RED_SUM))) return done(rc);
        hs.neg = (int32_t)mx[0];
        hs.bad_off = (int32_t)mx[1];
        n_rows_all = sm[0];
        nnz_all = sm[2];
        hs.len_sum = (unsigned long long)sm[1];
        if (sm[2] > 0) { id_max = mx[2]; id_min = -mx[4]; }
        hs.len_max = mx[3];
        hs.len_min = -mx[5];
    } else if (nnz > 0) {
        id_min = hs.id_min;
        id_max = hs.id_max;
    }
    if (hs.neg) { set_error("negative item id in the transaction set"); return done(TFIM_E_INVALID); }
    if (hs.bad_off) { set_error("row_offsets must be non-decreasing"); return done(TFIM_E_INVALID); }

    // F1 histogram over ids 0..id_max (kernel_bitmap.cu:269-275)
    if ((rc = d_freq.reserve((size_t)(id_max + 1) * 4))) return done(rc);
    {
        const int32_t bins = (int32_t)(id_max + 1);
        if (nnz > 0 && bins <= kHistSmemBins) {
            const int32_t parts = (int32_t)std::min<int64_t>(148, (nnz + 65535) / 65536);
            if ((rc = d_tmp.reserve((size_t)parts * bins * 4))) return done(rc);
            static std::atomic<bool> configured[64];
            int dev = 0;
            cudaGetDevice(&dev);
            if (dev >= 0 && dev < 64 && !configured[dev].load()) {
                cudaFuncSetAttribute(k_hist_smem, cudaFuncAttributeMaxDynamicSharedMemorySize, kHistSmemBins * 4);
                configured[dev].store(true);
            }
            k_hist_smem<<<parts, 1024, (size_t)bins * 4, s>>>(d_items_p, nnz, bins, d_tmp.as<int32_t>());
            k_hist_sum<<<(bins + 255) / 256, 256, 0, s>>>(d_tmp.as<int32_t>(), parts, bins, d_freq.as<int32_t>());
        } else {
            cudaMemsetAsync(d_freq.p, 0, (size_t)bins * 4, s);
            if (nnz > 0) k_hist<<<grid_for(nnz), 256, 0, s>>>(d_items_p, nnz, d_freq.as<int32_t>());
        }
    }
    if ((rc = group_reduce(c, d_freq.p, id_max + 1, TFIM_DT_I32, TFIM_RED_SUM, s))) return done(rc);
    const int32_t bins = (int32_t)(id_max + 1);
    const double fthr = (double)n_rows_all * thr;             // kernel_bitmap.cu:806
    const int32_t min_count = (int32_t)std::max(0.0, std::ceil(fthr));   // v >= fthr  <=>  v >= ceil(fthr) for integer v
    // the smallest count v with v / rows > thr (kernel_bitmap.cu:815-816), the quotient rounded as there
    int32_t root_min = INT_MAX;
    if (n_rows_all > 0) {
        int64_t lo = 0, hi = INT_MAX;
        while (lo < hi) {
            const int64_t mid = (lo + hi) / 2;
            if ((double)mid / (double)n_rows_all > thr) hi = mid; else lo = mid + 1;
        }
        root_min = (int32_t)lo;
    }
    // map, then dense_to_orig, dense_freq and the frequency order, then the counts
    // (an id survives with at least min_count of the nnz_all occurrences)
    const size_t tab = ((size_t)bins + 3) & ~size_t(3);
    const size_t cap = (std::min<size_t>(bins, (size_t)(nnz_all / std::max(min_count, 1)) + 1) + 4) & ~size_t(3);
    if ((rc = d_map.reserve((tab + 3 * cap) * 4 + sizeof(DenseCounts)))) return done(rc);
    int32_t* t_orig = d_map.as<int32_t>() + tab;
    int32_t* t_freq = t_orig + cap;
    int32_t* t_order = t_freq + cap;
    DenseCounts* t_counts = (DenseCounts*)(t_order + cap);
    k_dense_ids<<<1, 1024, 0, s>>>(d_freq.as<int32_t>(), bins, min_count, root_min, d_map.as<int32_t>(), t_orig, t_freq, t_counts);
    DenseCounts dc{};
    cudaMemcpyAsync(&dc, t_counts, sizeof dc, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) { set_error("F1 histogram failed: %s", cudaGetErrorString(cudaGetLastError())); return done(TFIM_E_CUDA); }

    tfim_db_info& I = c->info;
    memset(&I, 0, sizeof I);
    I.trans_num = n_rows_all;
    I.item_id_min = id_min;
    I.item_id_max = id_max;
    I.trans_len_min = n_rows_all > 0 ? hs.len_min : INT_MAX;
    I.trans_len_max = n_rows_all > 0 ? hs.len_max : 0;
    I.trans_len_mean = n_rows_all > 0 ? (double)hs.len_sum / (double)n_rows_all : 0.0;
    I.dimension = dc.dimension;
    I.support_threshold = thr;
    I.frequency_threshold = fthr;
    I.min_count = min_count;
    I.dimension_reduced = dc.roots;

    // dense ids (kernel_bitmap.cu:348-373); a frequent id 0 is parked last (:356, true for an empty
    // set: 0 >= 0.0)
    const int32_t n_surv = dc.n_surv, n_dense = dc.n_dense;
    I.n_survivors = n_surv;
    I.n_dense = n_dense;
    I.item_id_max_dense = n_dense - 1;
    c->n_counted = n_surv;
    c->dense_to_orig.assign(n_dense, 0);
    c->dense_freq.assign(n_dense, 0);
    c->items_in_freq_sort.assign(n_dense, 0);
    if (n_dense > 0) {
        // (waited for with the row reduction below)
        cudaMemcpyAsync(c->dense_to_orig.data(), t_orig, (size_t)n_dense * 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(c->dense_freq.data(), t_freq, (size_t)n_dense * 4, cudaMemcpyDeviceToHost, s);
        if (n_dense <= kRankMax) {
            k_rank_order<<<(n_dense + kRankItems - 1) / kRankItems, 1024, 0, s>>>(t_freq, n_dense, 1, t_order);
            cudaMemcpyAsync(c->items_in_freq_sort.data(), t_order, (size_t)n_dense * 4, cudaMemcpyDeviceToHost, s);
        }
    }

    // reduced rows, their numbering, and the reduced transaction list in dense ids
    if ((rc = d_flag.reserve((size_t)std::max<int64_t>(n_rows, 1) * 4)) ||
        (rc = d_idx.reserve((size_t)std::max<int64_t>(n_rows, 1) * 16)))
        return done(rc);
    int64_t n_red = 0, n_red_items = 0;
    int64_t* red_idx = d_idx.as<int64_t>();
    int64_t* item_off = red_idx + std::max<int64_t>(n_rows, 1);
    if (n_rows > 0) {
        int32_t* red_len = d_flag.as<int32_t>();
        k_reduced_rows<<<grid_for(n_rows * kRowLanes), 256, 0, s>>>(d_off_p, d_items_p, n_rows,
                                                         d_map.as<int32_t>(), red_len, d_stats.as<ScanStats>());
        cub::TransformInputIterator<int32_t, IsPositive, const int32_t*> flags(red_len, IsPositive());
        size_t tb1 = 0, tb2 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb1, flags, red_idx, n_rows, s);
        cub::DeviceScan::ExclusiveSum(nullptr, tb2, red_len, item_off, n_rows, s);
        if ((rc = d_tmp.reserve(std::max(tb1, tb2)))) return done(rc);
        cub::DeviceScan::ExclusiveSum(d_tmp.p, tb1, flags, red_idx, n_rows, s);
        cub::DeviceScan::ExclusiveSum(d_tmp.p, tb2, red_len, item_off, n_rows, s);
        int64_t last[2] = {0, 0};
        int32_t last_len = 0;
        cudaMemcpyAsync(&last[0], red_idx + (n_rows - 1), 8, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&last[1], item_off + (n_rows - 1), 8, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&last_len, red_len + (n_rows - 1), 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(&hs, d_stats.p, sizeof hs, cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) { set_error("row reduction failed: %s", cudaGetErrorString(cudaGetLastError())); return done(TFIM_E_CUDA); }
        n_red = last[0] + (last_len > 0);
        n_red_items = last[1] + last_len;
    } else if (cudaStreamSynchronize(s) != cudaSuccess) {
        set_error("dense ids failed: %s", cudaGetErrorString(cudaGetLastError()));
        return done(TFIM_E_CUDA);
    }
    if (n_dense > kRankMax) {
        std::iota(c->items_in_freq_sort.begin(), c->items_in_freq_sort.end(), 0);
        std::stable_sort(c->items_in_freq_sort.begin(), c->items_in_freq_sort.end(),
                         [&](int a, int b) { return c->dense_freq[a] > c->dense_freq[b]; });
    }
    const int64_t n_roots = std::min<int64_t>(dc.roots, n_dense);
    c->roots.assign(c->items_in_freq_sort.begin(), c->items_in_freq_sort.begin() + n_roots);
    int64_t n_red_all = n_red;
    if (c->sharded) {
        int64_t mx[2] = {n_red > 0 ? (int64_t)hs.red_max : 0, n_red > 0 ? -(int64_t)hs.red_min : -(int64_t)LLONG_MAX};
        int64_t sm[3] = {n_red, (int64_t)hs.red_sum, (int64_t)hs.red_sq_sum};
        if ((rc = group_reduce_host(c, mx, 2, TFIM_RED_MAX)) || (rc = group_reduce_host(c, sm, 3, TFIM_RED_SUM))) return done(rc);
        hs.red_max = mx[0];
        hs.red_min = -mx[1];
        n_red_all = sm[0];
        hs.red_sum = (unsigned long long)sm[1];
        hs.red_sq_sum = (unsigned long long)sm[2];
    }
    I.trans_num_reduced = n_red_all;
    I.trans_len_red_min = n_red_all > 0 ? hs.red_min : INT_MAX;
    I.trans_len_red_max = n_red_all > 0 ? hs.red_max : 0;
    I.trans_len_red_mean = (double)hs.red_sum / (double)n_red_all;   // 0/0 -> nan, as the reference
    c->red_pair_work = (double)hs.red_sq_sum;
    if ((rc = dev_alloc((void**)&c->d_red_off, (size_t)(n_red + 1) * 8, s)) ||
        (rc = dev_alloc((void**)&c->d_red_items, (size_t)std::max<int64_t>(n_red_items, 1) * 4, s)))
        return done(rc);
    c->n_red_items = n_red_items;
    cudaMemcpyAsync(c->d_red_off + n_red, &n_red_items, 8, cudaMemcpyHostToDevice, s);
    if (n_red > 0)
        k_write_reduced<<<grid_for(n_rows * kRowLanes), 256, 0, s>>>(d_off_p, d_items_p, n_rows, d_map.as<int32_t>(),
                                                          d_flag.as<int32_t>(), red_idx, item_off, c->d_red_off, c->d_red_items);

    // the bitmap: n_dense rows x W words, zero padded
    c->n_bits = n_red;
    c->n_bits_total = n_red_all;
    c->W = words_for_bits(n_red);
    if (c->sharded && c->W < kRowAlignWords) c->W = kRowAlignWords;   // an empty shard counts zeros
    I.words_per_row = (int32_t)c->W;
    const size_t bm_bytes = (size_t)std::max<int32_t>(n_dense, 1) * (size_t)std::max<int64_t>(c->W, 1) * 4;
    if ((rc = dev_alloc((void**)&c->d_bitmap, bm_bytes, s))) return done(rc);
    if (n_red > 0 && n_dense > 0 && n_dense <= kBitmapMaxDense) {
        static std::atomic<bool> configured[64];
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !configured[dev].load()) {
            cudaFuncSetAttribute(k_build_bitmap, cudaFuncAttributeMaxDynamicSharedMemorySize, kBitmapMaxDense * 32);
            configured[dev].store(true);
        }
        // 64-byte pieces while several blocks' tables fit an SM, else 32-byte ones
        const int32_t wb_log = n_dense <= 700 ? 4 : 3;
        const size_t smem = ((size_t)n_dense << wb_log) * 4;
        k_build_bitmap<<<(unsigned)(c->W >> wb_log), smem > (48 << 10) ? 1024 : 256, smem, s>>>(
            c->d_red_off, c->d_red_items, n_red, n_dense, wb_log, c->d_bitmap, c->W);
    } else {
        cudaMemsetAsync(c->d_bitmap, 0, bm_bytes, s);
        if (n_red > 0)
            k_scatter_bits<<<grid_for(n_red), 256, 0, s>>>(c->d_red_off, c->d_red_items, n_red, c->d_bitmap, c->W);
    }
    if (cudaGetLastError() != cudaSuccess) {
        set_error("bitmap scatter failed");
        return done(TFIM_E_CUDA);
    }
    c->from_db = true;
    rc = compute_bit_supports(c);
    return done(rc);
}

int ingest_bitmap(tfim_ctx* c, const uint32_t* rows, int32_t n_rows, int64_t n_bits, int32_t n_counted) {
    TFIM_CHECK(rows && n_rows > 0 && n_bits > 0 && n_counted >= 0 && n_counted <= n_rows, TFIM_E_INVALID,
               "tfim_open_bitmap: invalid arguments");
    const int64_t src_w = (n_bits + 31) / 32;
    c->n_bits = n_bits;
    c->n_bits_total = n_bits;
    if (c->sharded) TFIM_TRY(group_reduce_host(c, &c->n_bits_total, 1, TFIM_RED_SUM));
    c->W = words_for_bits(n_bits);
    c->n_counted = n_counted;
    memset(&c->info, 0, sizeof c->info);
    c->info.n_survivors = n_counted;
    c->info.n_dense = n_rows;
    c->info.trans_num_reduced = c->n_bits_total;
    c->info.words_per_row = (int32_t)c->W;
    const size_t bytes = (size_t)n_rows * (size_t)c->W * 4;
    TFIM_TRY(dev_alloc((void**)&c->d_bitmap, bytes, c->stream));
    TFIM_CUDA(cudaMemsetAsync(c->d_bitmap, 0, bytes, c->stream));
    TFIM_CUDA(cudaMemcpy2DAsync(c->d_bitmap, (size_t)c->W * 4, rows, (size_t)src_w * 4, (size_t)src_w * 4, n_rows,
                                cudaMemcpyHostToDevice, c->stream));
    // bits beyond n_bits in the last supplied word must not count: clear them
    if (n_bits % 32) {
        std::vector<uint32_t> last(n_rows);
        const uint32_t keep = (1u << (n_bits % 32)) - 1u;
        for (int32_t r = 0; r < n_rows; r++) last[r] = rows[(size_t)r * src_w + src_w - 1] & keep;
        TFIM_CUDA(cudaMemcpy2DAsync(c->d_bitmap + (src_w - 1), (size_t)c->W * 4, last.data(), 4, 4, n_rows,
                                    cudaMemcpyHostToDevice, c->stream));
    }
    TFIM_CUDA(cudaStreamSynchronize(c->stream));
    c->dense_to_orig.resize(n_rows);
    std::iota(c->dense_to_orig.begin(), c->dense_to_orig.end(), 0);
    return compute_bit_supports(c);
}

}  // namespace tfim
