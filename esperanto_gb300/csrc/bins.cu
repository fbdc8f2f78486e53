// bins.cu -- length-binned work list for the persistent DP kernels.
//
// Pairs are counting-sorted on the device by a 20-bit geometry key (columns
// per row, rows; both exact below 1023) in DESCENDING cost order, so that
// (a) the 32 pairs a warp takes from the queue share their loop trip counts,
// (b) the most expensive pairs start first (the tail of the launch is made
// of cheap pairs) and (c) neighbours in the list usually have identical band
// geometry, which the two-pairs-per-thread kernel needs.  Kernels:
// histogram, a three-phase scan, scatter; warp-aggregated atomics keep a
// single hot bin (uniform batches) cheap.
#include <cuda_runtime.h>

#include <cstdint>

#include "esp_internal.h"

namespace esp {

static constexpr int KEY_BITS = 10;
static constexpr int NBINS = 1 << (2 * KEY_BITS);
static constexpr int SCAN_TILE = 1024;  // counters per block of the scan
static constexpr int SCAN_BLOCKS = NBINS / SCAN_TILE;

// Key: larger = more expensive.  m = rows; w = columns per row (band
// width or window) in band mode and extend_hint's full-matrix attempt
// (mode 2); in its banded first attempt (mode 1) the window length instead:
// every first attempt has width 61 (or the window, up to 30), so the window
// length orders them as well and, with the rows, pins their geometry
// wherever the hint offset follows from the lengths (read + 2h windows at
// offset h, flank segments at offset 0, fixed-shape reads).
__device__ __forceinline__ uint32_t geometry_key(const esp_pair &P, int mode) {
    uint32_t m = P.read_len, n = P.win_len;
    uint32_t w;
    bool full = (mode == 0) ? (P.band_half < 0) : (mode == 2 || n <= 30);
    if (full || mode == 1) {
        w = n;
    } else {
        uint64_t bw = 2ull * (uint32_t)P.band_half + 1;
        w = (uint32_t)(bw < n ? bw : n);
    }
    const uint32_t top = (1u << KEY_BITS) - 1;
    return ((w < top ? w : top) << KEY_BITS) | (m < top ? m : top);
}

// Entry k of the pairs to bin: k itself, or list[k] over *count entries.
struct BinInput {
    const uint32_t *list;   // null: pairs 0 .. n-1
    const uint32_t *count;  // device count of list entries (list only)
    __device__ __forceinline__ uint64_t size(uint64_t n) const { return list ? *count : n; }
    __device__ __forceinline__ uint32_t at(uint64_t k) const { return list ? list[k] : (uint32_t)k; }
};

__device__ __forceinline__ void agg_add(uint32_t *ctr, uint32_t key, uint32_t *slot) {
    // warp-aggregated atomicAdd on ctr[key]; returns each lane's slot
    uint32_t active = __activemask();
    uint32_t peers = __match_any_sync(active, key);
    int leader = __ffs(peers) - 1;
    int lane = threadIdx.x & 31;
    uint32_t rank = __popc(peers & ((1u << lane) - 1));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(ctr + key, (uint32_t)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    if (slot) *slot = base + rank;
}

// Cells a pair's DP computes, near enough to weigh one pair against another.
__device__ __forceinline__ uint32_t cost_of(const esp_pair &P, int mode) {
    const uint32_t n = P.win_len;
    const bool full = mode == 0 ? P.band_half < 0 : (mode == 2 || n <= 30);
    const uint64_t band = 2ull * (mode == 0 ? (uint32_t)P.band_half : 30u) + 1;
    const uint64_t w = full || band > n ? n : band;
    const uint64_t c = w * P.read_len;
    return c < 0xffffffffull ? (uint32_t)c : 0xffffffffu;
}

// stats (optional, zeroed): the sum of the pairs' costs, the largest cost and
// the longest read.
struct BinStats {
    unsigned long long cost;
    uint32_t max_cost, max_m;
};

__global__ void bin_hist(const esp_pair *__restrict__ pairs, uint64_t n, BinInput in, int mode,
                         uint32_t *__restrict__ hist, BinStats *__restrict__ stats,
                         uint32_t *__restrict__ window_n) {
    const uint64_t cnt = in.size(n);
    uint32_t with_n = 0;
    unsigned long long cost = 0;
    uint32_t max_cost = 0, max_m = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t pi = in.at(i);
        if (pi >= n) continue;  // never index past the batch
        const esp_pair P = pairs[pi];
        agg_add(hist, NBINS - 1 - geometry_key(P, mode), nullptr);  // descending cost order
        with_n |= P.n_win;
        if (stats) {
            const uint32_t c = cost_of(P, mode);
            cost += c;
            max_cost = max(max_cost, c);
            max_m = max(max_m, P.read_len);
        }
    }
    if (__any_sync(0xffffffffu, with_n != 0) && (threadIdx.x & 31) == 0) *window_n = 1u;
    if (stats) {
        for (int o = 16; o; o >>= 1) cost += __shfl_down_sync(0xffffffffu, cost, o);
        max_cost = __reduce_max_sync(0xffffffffu, max_cost);
        max_m = __reduce_max_sync(0xffffffffu, max_m);
        if ((threadIdx.x & 31) == 0 && max_cost) {
            atomicAdd(&stats->cost, cost);
            atomicMax(&stats->max_cost, max_cost);
            atomicMax(&stats->max_m, max_m);
        }
    }
}

// Exclusive scan of the NBINS counters in three phases: tile sums, a scan of
// the tile sums (one block), tile scans offset by their prefix.  part[] holds
// SCAN_BLOCKS words after the counters.
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t *s_warp,
                                                       uint32_t &total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    uint32_t wpre = 0;
    total = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        uint32_t w = s_warp[k];
        if (k < wid) wpre += w;
        total += w;
    }
    return wpre + x - v;
}

// PAD: every bin's slot count rounded up to even, so that list positions
// 2k, 2k + 1 never straddle two bins; the spare slot of an odd bin holds
// NO_PAIR (the list is pre-filled with it).
__device__ __forceinline__ uint4 bin_counts(uint4 q, bool pad) {
    if (pad) {
        q.x += q.x & 1u;
        q.y += q.y & 1u;
        q.z += q.z & 1u;
        q.w += q.w & 1u;
    }
    return q;
}

template <bool PAD>
__global__ void __launch_bounds__(256) bin_scan_up(const uint32_t *__restrict__ hist,
                                                   uint32_t *__restrict__ part) {
    __shared__ uint32_t s_warp[8];
    uint4 q = bin_counts(
        reinterpret_cast<const uint4 *>(hist + (size_t)blockIdx.x * SCAN_TILE)[threadIdx.x], PAD);
    uint32_t total;
    block_excl_scan256(q.x + q.y + q.z + q.w, s_warp, total);
    if (threadIdx.x == 0) part[blockIdx.x] = total;
}

// Also writes the list length (the sum of all slots) to *total.
__global__ void __launch_bounds__(1024) bin_scan_top(uint32_t *__restrict__ part,
                                                     uint32_t *__restrict__ total) {
    __shared__ uint32_t s[1024];
    uint32_t v = threadIdx.x < SCAN_BLOCKS ? part[threadIdx.x] : 0;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        uint32_t y = threadIdx.x >= (unsigned)off ? s[threadIdx.x - off] : 0;
        __syncthreads();
        s[threadIdx.x] += y;
        __syncthreads();
    }
    if (threadIdx.x < SCAN_BLOCKS) part[threadIdx.x] = s[threadIdx.x] - v;
    if (threadIdx.x == 1023) *total = s[1023];
}

template <bool PAD>
__global__ void __launch_bounds__(256) bin_scan_down(uint32_t *__restrict__ hist,
                                                     const uint32_t *__restrict__ part) {
    __shared__ uint32_t s_warp[8];
    uint4 *tile = reinterpret_cast<uint4 *>(hist + (size_t)blockIdx.x * SCAN_TILE);
    uint4 q = bin_counts(tile[threadIdx.x], PAD);
    uint32_t total;
    uint32_t run = part[blockIdx.x] + block_excl_scan256(q.x + q.y + q.z + q.w, s_warp, total);
    uint4 r;
    r.x = run;
    r.y = r.x + q.x;
    r.z = r.y + q.y;
    r.w = r.z + q.z;
    tile[threadIdx.x] = r;
}

// First list position of bin b, after the scatter: the end of the bin before,
// rounded up to even.
__device__ __forceinline__ uint32_t bin_start(const uint32_t *cursor, uint32_t b) {
    const uint32_t end = b ? __ldcg(cursor + b - 1) : 0u;
    return end + (end & 1u);
}

// The plan of a batch that the mixed kernel may run, from the batch's costs (in
// cells; an item is two pairs): {list entries its groups run, log2 of a group's
// lanes (and 8 for pairs of about one cost), its list's length, the list's length for one pair per thread} -- one of the
// two lengths is 0.  For the paired kernel (no stats) the two lengths alone.
//
// A thread takes ~25 ns a row of 8 x 2 cells when its warp has the scheduler
// to itself (52 cycles, measured), the full chip 1.9 T cells/s: an item
// finishes with the rest of the batch when its cost is the mean cost times
// items / 23,700 (0.305 x the 77,824 resident threads).  Batches whose costliest
// item takes more than 1.1 times that give the items above half of it to
// groups: 65,536 mixed pairs (3.3 times it) 2.98 ms by threads, 1.43 split; a line
// at 1.5 or 2 costs 200,000 mixed pairs 4.0 ms, not 2.76.
// Lanes of a group from how far the costliest item is above the mean finish
// (the fastest of 4, 8, 16 and 32 lanes at 4,096 to 200,000 pairs of one shape
// and mixed).  Where nearly all pairs are among the costliest, groups wait for
// their empty lanes, not for the rest of the batch: then no more lanes than have
// work, unless the batch leaves schedulers without a warp, and one pair per
// thread where that is faster (group_shape, abi.cu), up to two warps a
// scheduler; above that two per thread: 36,000 pairs of 100 in 129 columns 0.52 ms
// one per thread, 0.61 two; 45,000 0.70 / 0.62; 45,000 of 100 to 150 in 65 0.64 in
// groups, 0.49 two per thread.
//
// Items whose two pairs differ in geometry (the bins know width and rows, not the
// band's offset) take both kernels of pairs twice the time, and with them every
// item of their warp.  So beyond one such item in UNLIKE the list goes to the
// one-pair kernel, unless its costliest pair alone takes a thread as long as the
// batch takes groups at half their rate (3.1 times the mean finish): 65,536 pairs of
// 150 x 214 at offsets of 12 to 52 1.68 -> 0.77 ms, 200,000 mixed pairs 7.1 -> 4.8;
// 4,096 mixed pairs stay with groups (0.83, one per thread 1.84; 65,536 3.5 /
// 3.6, about even).  In large batches one warp's second pass weighs less: 600,000
// pairs of which 0.5 % are at other offsets take 4.4 ms in pairs, 2 % 5.9, one per
// thread 5.2.
constexpr uint32_t UNLIKE = 256, UNLIKE_LARGE = 48, SAMPLE = 16;

__device__ void make_plan(const uint32_t *cursor, uint32_t n, const BinStats *stats, int mode,
                          const BinPlan &b) {
    const uint32_t unlike = __ldcg(b.unlike);
    if (!stats) {  // a list for the paired kernel
        const bool single = (uint64_t)unlike * SAMPLE * UNLIKE_LARGE > n / 2;
        b.plan[2] = single ? 0u : n;
        b.plan[3] = single ? n : 0u;
        return;
    }
    const float even = (float)stats->cost / (b.threads * 0.305f);  // of one pair of the item
    const float top = 2.0f * (float)stats->max_cost;
    const float above = even > 0.0f ? top / even : 0.0f;
    const float x = above / 0.4f;
    int lg = x < 5.0f ? 2 : (x < 11.0f ? 3 : (x < 60.0f ? 4 : 5));
    // (42,555 whole windows of 112 to 155 bases, 0.69 of their costliest, 1.51 ms
    // as alike, 1.34 not; 93,996 extend_hint pairs of 133 to 270 5.8, 4.36)
    const bool alike = (float)stats->cost > 0.8f * (float)stats->max_cost * (float)n;
    const bool filled = 2.0f * (float)n > b.threads;  // one per thread: over two warps a scheduler
    uint32_t split = 0;
    if (alike && filled && b.pairs_ok) {
        split = 0;
    } else if (b.all) {
        split = n;
    } else if (above > 1.1f) {
        // items of w columns a row and more: the list's order.  extend_hint's
        // first attempt has one width, its list goes by window length.
        const uint32_t cap = (1u << KEY_BITS) - 1;
        const float w = 0.55f * even / (float)max(stats->max_m, 1u);
        if (mode == 1) split = n;
        else split = w < 1.0f ? n : bin_start(cursor, NBINS - 1 - ((min((uint32_t)w, cap - 1u) << KEY_BITS) | cap));
    }
    if (alike) {
        // lanes that give each scheduler one warp: threads / 128 warps, 64 / lanes
        // entries a warp
        int idle = 2;
        while (idle < 5 && (float)n * (float)(4 << idle) <= b.threads) idle++;
        lg = min(lg, max(b.lanes_lg, idle));
    }
    const bool apart = (uint64_t)unlike * UNLIKE > n / 2 && above <= 3.1f;
    const bool single = b.single_ok && (apart || (alike && !filled && above <= b.single_line));
    b.plan[0] = single ? 0u : split;
    const bool same = (float)stats->cost > 0.9f * (float)stats->max_cost * (float)n;
    b.plan[1] = (uint32_t)max(lg, b.min_lg) | (same ? 8u : 0u);
    b.plan[2] = single ? 0u : n;
    b.plan[3] = single ? n : 0u;
}

// Whether two pairs have one band geometry, as two pairs of an item must to share
// its cells (process_item2 and group_section, gotoh.cu).
__device__ __forceinline__ bool same_band(const esp_pair &a, const esp_pair &b, int mode) {
    if (a.read_len != b.read_len || a.win_len != b.win_len) return false;
    if (mode == 2) return true;
    if (mode == 1) return a.win_len <= 30 || a.band_offset == b.band_offset;
    if (a.band_half < 0 || b.band_half < 0) return a.band_half < 0 && b.band_half < 0;
    return a.band_half == b.band_half && a.band_offset == b.band_offset;
}

// PLAN: also counts the items, list positions 2k and 2k + 1 (the list pre-filled
// with NO_PAIR), whose pairs do not have one geometry: an item's word takes each
// of them in one atomic, and the second finds the first there.  Large lists, which
// the paired kernel runs, count one item in SAMPLE (all of them: 4,194,304 mixed
// pairs 0.3 % longer).  The last block to end makes the plan (a launch of its
// own took 4 us).
template <bool PLAN>
__global__ void bin_scatter(const esp_pair *__restrict__ pairs, uint64_t n, BinInput in, int mode,
                            uint32_t *cursor, uint32_t *order, const uint32_t *total,
                            const BinStats *stats, BinPlan plan) {
    const uint64_t cnt = in.size(n);
    uint32_t found = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t pi = in.at(i);
        if (pi >= n) continue;
        const esp_pair P = pairs[pi];
        uint32_t slot;
        agg_add(cursor, NBINS - 1 - geometry_key(P, mode), &slot);
        if (PLAN && (stats || (slot >> 1) % SAMPLE == 0)) {
            const unsigned long long none = 0xffffffffull;
            const bool second = slot & 1u;
            const unsigned long long old =
                atomicAnd(reinterpret_cast<unsigned long long *>(order) + (slot >> 1),
                          second ? ((unsigned long long)pi << 32) | none : (none << 32) | pi);
            const uint32_t other = (uint32_t)(second ? old : old >> 32);
            if (other != (uint32_t)none && !same_band(P, pairs[other], mode)) found++;
        } else {
            order[slot] = pi;
        }
    }
    if (PLAN) {
        found = __reduce_add_sync(0xffffffffu, found);
        if ((threadIdx.x & 31) == 0 && found) atomicAdd(plan.unlike, found);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(plan.done, 1u) == gridDim.x - 1) {
            __threadfence();
            make_plan(cursor, *total, stats, mode, plan);
        }
    }
}

// Window width summed over rows 1..m (extend.rs:653-696).
__device__ uint64_t band_cells(uint32_t m, uint32_t n, int64_t off, int64_t half) {
    uint64_t cells = 0;
    for (uint32_t i = 1; i <= m; i++) {
        int64_t c = off + i;
        c = c < 1 ? 1 : (c > n ? n : c);
        int64_t lo = c - half > 1 ? c - half : 1;
        int64_t hi = c + half < (int64_t)n ? c + half : (int64_t)n;
        if (hi >= lo) cells += (uint64_t)(hi - lo + 1);
    }
    return cells;
}

__global__ void count_cells(const esp_pair *__restrict__ pairs,
                            const esp_extension *__restrict__ out, uint64_t n, int mode,
                            unsigned long long *cells) {
    uint64_t acc = 0;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const esp_pair P = pairs[k];
        uint32_t m = P.read_len, w = P.win_len;
        if (m == 0 || w == 0) continue;
        if (mode == 0) {
            acc += P.band_half < 0 ? (uint64_t)m * w : band_cells(m, w, P.band_offset, P.band_half);
        } else if (w <= 30) {
            acc += (uint64_t)m * w;
        } else {
            acc += band_cells(m, w, P.band_offset, 30);
            if (out[k].escalated) acc += (uint64_t)m * w;
        }
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(cells, (unsigned long long)acc);
}

cudaError_t launch_count_cells(const esp_pair *pairs, const esp_extension *out, uint64_t n,
                               int mode, unsigned long long *cells, int num_sms,
                               cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    uint64_t need = (n + 255) / 256;
    int grid = (int)(need < (uint64_t)num_sms * 8 ? need : (uint64_t)num_sms * 8);
    count_cells<<<grid, 256, 0, st>>>(pairs, out, n, mode, cells);
    return cudaGetLastError();
}

size_t bin_scratch_bytes() { return (size_t)(NBINS + SCAN_BLOCKS) * sizeof(uint32_t); }

uint64_t bin_pad_slots(uint64_t n) { return n < (uint64_t)NBINS ? n : (uint64_t)NBINS; }

// Length classes of the binned list (descending cost): band/window width
// w >= 196, [100, 196), [52, 100), < 52 columns.  bounds[s], bounds[s+1] is
// class s; read from the scanned histogram before the scatter moves it.
__global__ void class_bounds(const uint32_t *__restrict__ hist, const uint32_t *__restrict__ total,
                             uint32_t *__restrict__ bounds) {
    if (threadIdx.x == 0) {
        const uint32_t top = (1u << KEY_BITS) - 1;
        const uint32_t first_w[3] = {195u, 99u, 51u};  // widest width of classes 1..3
        bounds[0] = 0;
        for (int s = 0; s < 3; s++)
            bounds[s + 1] = hist[NBINS - 1 - ((first_w[s] << KEY_BITS) | top)];
        bounds[4] = *total;
    }
}

cudaError_t launch_binning(const esp_pair *pairs, uint64_t n, int mode, uint32_t *hist,
                           uint32_t *order, int num_sms, cudaStream_t st, uint32_t *total,
                           uint32_t *bounds, bool pad, uint32_t *window_n, const uint32_t *list,
                           const uint32_t *list_count, const BinPlan *plan) {
    const BinInput in{list, list_count};
    cudaError_t e = cudaMemsetAsync(hist, 0, bin_scratch_bytes(), st);
    if (e == cudaSuccess && pad)
        e = cudaMemsetAsync(order, 0xff, (n + bin_pad_slots(n)) * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    int grid = num_sms * 4;
    uint64_t need = (n + 255) / 256;
    if ((uint64_t)grid > need) grid = (int)(need ? need : 1);
    BinStats *stats = plan && plan->stats ? reinterpret_cast<BinStats *>(plan->stats) : nullptr;
    bin_hist<<<grid, 256, 0, st>>>(pairs, n, in, mode, hist, stats, window_n);
    if (pad) bin_scan_up<true><<<SCAN_BLOCKS, 256, 0, st>>>(hist, hist + NBINS);
    else bin_scan_up<false><<<SCAN_BLOCKS, 256, 0, st>>>(hist, hist + NBINS);
    bin_scan_top<<<1, 1024, 0, st>>>(hist + NBINS, total);
    if (pad) bin_scan_down<true><<<SCAN_BLOCKS, 256, 0, st>>>(hist, hist + NBINS);
    else bin_scan_down<false><<<SCAN_BLOCKS, 256, 0, st>>>(hist, hist + NBINS);
    if (bounds) class_bounds<<<1, 32, 0, st>>>(hist, total, bounds);
    if (plan)
        bin_scatter<true><<<grid, 256, 0, st>>>(pairs, n, in, mode, hist, order, total, stats, *plan);
    else
        bin_scatter<false><<<grid, 256, 0, st>>>(pairs, n, in, mode, hist, order, nullptr, nullptr, BinPlan{});
    return cudaGetLastError();
}

}  // namespace esp
