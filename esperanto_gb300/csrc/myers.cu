// myers.cu -- GB300 editing-aware bit-parallel Myers filters
// (crates/map/src/myers_ea.rs and crates/engine/src/myers.rs).
//
// One thread owns one read x text pair.  The pattern (m <= 256 bases) is a
// bit-vector of NW 32-bit limbs held in registers; the pattern-equality
// table Peq[limb][text code] lives in shared memory with a thread-private
// column per lane (conflict-free: limb w of code c of thread t is at
// (w * 4 + c) * MY_BLOCK + t).  Each text column advances the whole
// bit-vector as one wide word: the match-propagation addition ripples its
// carry across limbs in a single add.cc/addc chain and the horizontal deltas
// shift across limbs through funnel shifts.  This is the ripple-carry form of
// engine/src/myers.rs:179-208; the edlib block form of myers_ea.rs:64-91
// computes the same column scores, so one kernel serves both.
//
// EA equality (myers_ea.rs:28-56, engine/src/myers.rs:111-123): read A
// matches text {A}, C matches {C,T}, G matches {G,A}, T matches {T}; a read
// or text base that is not A/C/G/T matches nothing.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

#include "esp_device.cuh"
#include "esp_internal.h"

namespace esp {

// sum[k] = a[k] + b[k] + carry over k = 0..NW-1 in one PTX carry chain.
template <int NW>
__device__ __forceinline__ void add_chain(uint32_t (&s)[NW], const uint32_t (&a)[NW],
                                          const uint32_t (&b)[NW]);

template <>
__device__ __forceinline__ void add_chain<1>(uint32_t (&s)[1], const uint32_t (&a)[1],
                                             const uint32_t (&b)[1]) {
    s[0] = a[0] + b[0];
}
template <>
__device__ __forceinline__ void add_chain<2>(uint32_t (&s)[2], const uint32_t (&a)[2],
                                             const uint32_t (&b)[2]) {
    asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
        : "=r"(s[0]), "=r"(s[1])
        : "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]));
}
template <>
__device__ __forceinline__ void add_chain<3>(uint32_t (&s)[3], const uint32_t (&a)[3],
                                             const uint32_t (&b)[3]) {
    asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(b[0]), "r"(b[1]), "r"(b[2]));
}
template <>
__device__ __forceinline__ void add_chain<4>(uint32_t (&s)[4], const uint32_t (&a)[4],
                                             const uint32_t (&b)[4]) {
    asm("add.cc.u32 %0, %4, %8;\n\taddc.cc.u32 %1, %5, %9;\n\taddc.cc.u32 %2, %6, %10;\n\t"
        "addc.u32 %3, %7, %11;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]),
          "r"(b[3]));
}
template <>
__device__ __forceinline__ void add_chain<5>(uint32_t (&s)[5], const uint32_t (&a)[5],
                                             const uint32_t (&b)[5]) {
    asm("add.cc.u32 %0, %5, %10;\n\taddc.cc.u32 %1, %6, %11;\n\taddc.cc.u32 %2, %7, %12;\n\t"
        "addc.cc.u32 %3, %8, %13;\n\taddc.u32 %4, %9, %14;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(b[0]), "r"(b[1]),
          "r"(b[2]), "r"(b[3]), "r"(b[4]));
}
template <>
__device__ __forceinline__ void add_chain<6>(uint32_t (&s)[6], const uint32_t (&a)[6],
                                             const uint32_t (&b)[6]) {
    asm("add.cc.u32 %0, %6, %12;\n\taddc.cc.u32 %1, %7, %13;\n\taddc.cc.u32 %2, %8, %14;\n\t"
        "addc.cc.u32 %3, %9, %15;\n\taddc.cc.u32 %4, %10, %16;\n\taddc.u32 %5, %11, %17;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(b[0]),
          "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]));
}
template <>
__device__ __forceinline__ void add_chain<7>(uint32_t (&s)[7], const uint32_t (&a)[7],
                                             const uint32_t (&b)[7]) {
    asm("add.cc.u32 %0, %7, %14;\n\taddc.cc.u32 %1, %8, %15;\n\taddc.cc.u32 %2, %9, %16;\n\t"
        "addc.cc.u32 %3, %10, %17;\n\taddc.cc.u32 %4, %11, %18;\n\taddc.cc.u32 %5, %12, %19;\n\t"
        "addc.u32 %6, %13, %20;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]),
          "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]));
}
template <>
__device__ __forceinline__ void add_chain<8>(uint32_t (&s)[8], const uint32_t (&a)[8],
                                             const uint32_t (&b)[8]) {
    asm("add.cc.u32 %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\taddc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, %23;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
          "=r"(s[7])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]),
          "r"(a[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]),
          "r"(b[6]), "r"(b[7]));
}

constexpr int MY_BLOCK = 128;

// 16 text codes of one window in processing order: the code of the first
// column in bits 31:30, its N flag in bit 31 of `n`.
struct CodeWin {
    uint32_t c, n;
};

// Split 16 packed 2-bit codes (code k at bits 31-2k, 30-2k) into a high-bit
// and a low-bit mask with position k at bit k.
__device__ __forceinline__ void unshuffle16(uint32_t cw, uint32_t &hi, uint32_t &lo) {
    uint32_t x = __brev(cw);  // code k -> bits 2k (high), 2k+1 (low)
    uint32_t e = x & 0x55555555u, o = (x >> 1) & 0x55555555u;
    e = (e | (e >> 1)) & 0x33333333u;
    e = (e | (e >> 2)) & 0x0f0f0f0fu;
    e = (e | (e >> 4)) & 0x00ff00ffu;
    e = (e | (e >> 8)) & 0x0000ffffu;
    o = (o | (o >> 1)) & 0x33333333u;
    o = (o | (o >> 2)) & 0x0f0f0f0fu;
    o = (o | (o >> 4)) & 0x00ff00ffu;
    o = (o | (o >> 8)) & 0x0000ffffu;
    hi = e;
    lo = o;
}

// Pattern rows of 32 read positions starting at position `b` (may be
// negative: positions < 0 are absent): high/low code bits and the mask of
// real ACGT positions (bit k <-> position b + k).
__device__ __forceinline__ void read_limb(const MyersJob &job, const esp_myers_pair &P,
                                          const esp_n_interval *iv, int m, int b, uint32_t &hi,
                                          uint32_t &lo, uint32_t &real) {
    hi = lo = real = 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        int s = b + 16 * half;  // first position of this 16-position half
        if (s + 16 <= 0 || s >= m) continue;
        int start = s < 0 ? 0 : s;
        int skip = start - s;  // leading absent positions (s < 0)
        uint32_t cw = load16(job.arena, P.read_pos + (uint64_t)start);
        uint32_t nm = P.n_read ? nmask16(iv, P.n_read, start) : 0u;
        uint32_t h, l;
        unshuffle16(cw, h, l);
        uint32_t nb = __brev(nm) & 0xffffu;  // position start + k -> bit k
        int cnt = min(16 - skip, m - start);
        uint32_t v = (cnt >= 16 ? 0xffffu : ((1u << cnt) - 1u)) & ~nb;  // read N matches nothing
        int sh = 16 * half + skip;
        hi |= h << sh;
        lo |= l << sh;
        real |= v << sh;
    }
}

// EA Peq rows for text A, C, G, T from one limb's code bits.
__device__ __forceinline__ void ea_rows(uint32_t hi, uint32_t lo, uint32_t real,
                                        uint32_t (&rows)[4]) {
    uint32_t a = ~hi & ~lo & real, c = ~hi & lo & real, g = hi & ~lo & real,
             tt = hi & lo & real;
    rows[0] = a | g;   // text A: read A or G
    rows[1] = c;       // text C: read C
    rows[2] = g;       // text G: read G
    rows[3] = tt | c;  // text T: read T or C
}

// 16 text codes in processing order, the first column in bits 31:30 of `c`;
// its N flag in bit 31 of `n`.  `cnt` codes of the text from `at` on (reversed:
// the last of them first).
__device__ __forceinline__ CodeWin text_codes(const MyersJob &job, const esp_myers_pair &P,
                                              const esp_n_interval *iv, bool rev, int64_t at,
                                              int cnt) {
    CodeWin w;
    w.c = load16(job.arena, P.text_pos + (uint64_t)at);
    w.n = P.n_text ? nmask16(iv, P.n_text, at) : 0u;
    if (rev) {
        const uint32_t x = __brev(w.c >> (2 * (16 - cnt)));  // slot s -> bits 2s (high), 2s+1
        w.c = ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
        w.n = __brev(w.n >> (32 - cnt));
    }
    return w;
}

// One text column over all limbs; the horizontal delta of the last row is
// up - down.
template <int NW, bool GLOB>
__device__ __forceinline__ void myers_column(const uint32_t (&eq)[NW], uint32_t (&pv)[NW],
                                             uint32_t (&mv)[NW], uint32_t &up,
                                             uint32_t &down) {
    uint32_t xv[NW], s[NW], ph[NW], mh[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) {
        xv[w] = eq[w] | mv[w];
        s[w] = eq[w] & pv[w];
    }
    add_chain<NW>(s, s, pv);
#pragma unroll
    for (int w = 0; w < NW; w++) {
        const uint32_t xh = (s[w] ^ pv[w]) | xv[w];
        ph[w] = mv[w] | ~(xh | pv[w]);
        mh[w] = pv[w] & xh;
    }
    up = ph[NW - 1] >> 31;
    down = mh[NW - 1] >> 31;
#pragma unroll
    for (int w = NW - 1; w >= 0; w--) {
        const uint32_t phs = w ? __funnelshift_l(ph[w - 1], ph[w], 1) : ((ph[0] << 1) | (GLOB ? 1u : 0u));
        const uint32_t mhs = w ? __funnelshift_l(mh[w - 1], mh[w], 1) : (mh[0] << 1);
        pv[w] = mhs | ~(xv[w] | phs);
        mv[w] = phs & xv[w];
    }
}

// Virtual bits of limb w below a pattern whose row 0 is bit `off`.
__device__ __forceinline__ uint32_t virtual_bits(int off, int w) {
    const int vb = off - w * 32;  // bits [0, vb) of the limb
    return vb <= 0 ? 0u : (vb >= 32 ? 0xffffffffu : (1u << vb) - 1u);
}

// One pair.  flags: MYF_REVERSE (best start: read and text both reversed,
// myers_ea.rs:158-185), MYF_GLOBAL (engine global: leading column +1 per text
// base, engine/src/myers.rs:151-169).
//
// The m pattern rows occupy the TOP m bits of the NW*32-bit vector, so the last
// row is always bit 31 of limb NW-1.  The bits below are virtual rows with
// vertical delta 0 throughout.  In a search they match every text base: their
// horizontal deltas are 0, they never carry into the real rows and they shift
// 0 into real row 0, the semi-global boundary (hin = 0).  In a global
// alignment (GLOB) they match none: their horizontal deltas are +1, which they
// shift into row 0 (hin = +1).
//
// The loop is bound by the ALU (92 % busy): 10 operations a limb and column (the
// add with carry, seven three-input logic operations, two shifts), the rest
// counts a column.  Columns go 16 a chunk, after the text's first n % 16 (all
// lanes take that partial chunk together), so that a full chunk has constant
// shifts and no N test, and its best column is the least of score * 16 +
// column, one operation each; a column's Peq row is read a column ahead.
// 1,048,576 reads of 150 bases in texts of 200: 0.747 -> 0.687 ms; 12,000 of 200
// in 260 (few warps, latency) 37.6 -> 33.5 us.  Shifts as products with 2 (the
// multiply pipe) took fewer ALU operations and as long: their high halves
// stall the dispatch.
template <int NW, bool GLOB>
__device__ void myers_pair(const MyersJob &job, uint32_t k, uint32_t *__restrict__ peq) {
    const esp_myers_pair P = job.pairs[k];
    const int m = (int)P.read_len;
    const uint32_t n = P.text_len;
    const bool rev = job.flags & MYF_REVERSE;
    esp_myers_result res;
    res.dist = m;
    res.pos = 0;
    res.status = ESP_OK;
    if (m == 0 || m > NW * 32) {
        job.out[k] = res;  // the host routed m = 0 / m > 256 before launch
        if (m > NW * 32) job.out[k].status = ESP_EINVAL;
        return;
    }
    const esp_n_interval *iv = job.n_iv + P.n_first;
    uint32_t *col = peq + threadIdx.x;  // limb w of code c at (w * 4 + c) * MY_BLOCK
    const int off = NW * 32 - m;  // virtual rows below the pattern
    uint32_t pv[NW], mv[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) {
        // forward: bit k of limb w <-> read position w*32 + k - off.  Reversed:
        // position p <-> bit NW*32 - 1 - p, the forward limb NW-1-w with row 0
        // at bit 0 turned round; its padding above m lands in the virtual bits.
        uint32_t hi, lo, real, rows[4];
        read_limb(job, P, iv, m, rev ? (NW - 1 - w) * 32 : w * 32 - off, hi, lo, real);
        ea_rows(hi, lo, real, rows);
        const uint32_t virt = virtual_bits(off, w);
#pragma unroll
        for (int q = 0; q < 4; q++)
            col[(w * 4 + q) * MY_BLOCK] = (rev ? __brev(rows[q]) : rows[q]) | (GLOB ? 0u : virt);
        pv[w] = ~virt;  // pattern rows start with vertical delta +1 (D[i][0] = i)
        mv[w] = 0u;
    }
    constexpr int KEY = GLOB ? 1 : 16;  // score * 16 + column within 16
    int key = m * KEY, best = m;
    uint32_t best_at = 0;
    const esp_n_interval *tiv = iv + P.n_read;
    const char *rows = reinterpret_cast<const char *>(col);
    constexpr uint32_t ROW = MY_BLOCK * 4;  // bytes, a power of two
    uint32_t done = 0;
    for (uint32_t cnt = n & 15; done < n; done += cnt, cnt = 16) {
        if (cnt == 0) continue;
        CodeWin win = text_codes(job, P, tiv, rev, rev ? n - done - cnt : done, (int)cnt);
        int least = INT_MAX;
        if (cnt == 16 && win.n >> 16 == 0) {
            constexpr int STEP = 2;  // columns unrolled
            uint32_t next[NW];  // the next column's Peq row, read a column ahead
            const uint32_t *pe = reinterpret_cast<const uint32_t *>(rows + (win.c >> 30) * ROW);
#pragma unroll
            for (int w = 0; w < NW; w++) next[w] = pe[w * 4 * MY_BLOCK];
#pragma unroll 1
            for (int g = 0; g < 16; g += STEP) {
#pragma unroll
                for (int x = 0; x < STEP; x++) {
                    uint32_t eq[NW], up, down;
                    const uint32_t r = ((win.c >> (28 - 2 * x)) & 3u) * ROW;  // 0 after the last
                    pe = reinterpret_cast<const uint32_t *>(rows + r);
#pragma unroll
                    for (int w = 0; w < NW; w++) {
                        eq[w] = next[w];
                        next[w] = pe[w * 4 * MY_BLOCK];
                    }
                    myers_column<NW, GLOB>(eq, pv, mv, up, down);
                    key = (int)mad_u32(up, (uint32_t)KEY, (uint32_t)key);
                    key = (int)mad_u32(down, (uint32_t)-KEY, (uint32_t)key);
                    if (!GLOB) least = __viaddmin_s32(key, x, least);
                }
                win.c <<= 2 * STEP;
                if (!GLOB) key += STEP;
            }
            if (!GLOB) key -= 16;
        } else {  // a partial step, or N in the text: it matches virtual rows only
#pragma unroll 1
            for (int x = 0; x < (int)cnt; x++) {
                const uint32_t *pe = reinterpret_cast<const uint32_t *>(rows + (win.c >> 30) * ROW);
                uint32_t eq[NW], up, down;
                if ((int)win.n < 0) {
#pragma unroll
                    for (int w = 0; w < NW; w++) eq[w] = GLOB ? 0u : virtual_bits(off, w);
                } else {
#pragma unroll
                    for (int w = 0; w < NW; w++) eq[w] = pe[w * 4 * MY_BLOCK];
                }
                win.c <<= 2;
                win.n <<= 1;
                myers_column<NW, GLOB>(eq, pv, mv, up, down);
                key += (int)(up - down) * KEY;
                if (!GLOB) least = min(least, key + x);
            }
        }
        if (!GLOB && least < best * KEY) {  // the first column of a smaller score
            best = least >> 4;
            best_at = done + (uint32_t)(least & 15) + 1;
        }
    }
    if (GLOB) {
        res.dist = key > 0 ? key : 0;
        res.pos = 0;
    } else {
        res.dist = best;
        res.pos = rev ? (uint64_t)(n - best_at) : (uint64_t)best_at;
    }
    job.out[k] = res;
}

template <int NW, bool GLOB>
__device__ __noinline__ void myers_call(const MyersJob &job, uint32_t k, uint32_t *peq) {
    myers_pair<NW, GLOB>(job, k, peq);
}

// The limbs of the warp's longest read, 1..NW, choose its pairs' code.
template <int NW, bool GLOB>
__device__ __forceinline__ void myers_limbs(const MyersJob &job, uint32_t k, uint32_t *peq, int limbs) {
    if (limbs == NW) myers_call<NW, GLOB>(job, k, peq);
    else if constexpr (NW > 1) myers_limbs<NW - 1, GLOB>(job, k, peq, limbs);
}

template <int NW>
__device__ __forceinline__ int limbs_of(uint32_t m) {
    return m ? (int)min((m - 1) / 32 + 1, (uint32_t)NW) : 0;
}

// A block's warps are given its pairs in the order of their limbs: a warp's time
// is that of its longest read, and in the batch's order nearly every warp of a
// ragged batch has one near the longest, and all run the limbs of the batch's longest.
// Reads of 20 to 256 bases: 100,003 pairs, best start, 0.248 -> 0.168 ms; 262,144, best end,
// 0.48 -> 0.34, 400,000 0.72 -> 0.56.  Blocks of 256 order better (400,000 in 0.51)
// but fill the SMs unevenly: 131,072 reads of 150 bases took 107 us, in these 95,
// before 101.  Two columns unrolled: with 4 or 8 the code of several limb counts
// does not fit the instruction cache (a quarter slower).  A block whose reads all
// have NW limbs keeps the batch's order.
template <int NW, bool GLOB>
__global__ void __launch_bounds__(MY_BLOCK)
    myers_ordered_kernel(const __grid_constant__ MyersJob job) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_first[(NW + 1) * MY_BLOCK / 32];  // pairs of (class, warp), then those before
    __shared__ uint16_t s_order[MY_BLOCK];
    constexpr int WARPS = MY_BLOCK / 32, ENTRIES = (NW + 1) * WARPS;
    const uint64_t base = (uint64_t)blockIdx.x * MY_BLOCK;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t k = base + threadIdx.x;
    bool have = k < job.n_pairs;
    int limbs = have ? limbs_of<NW>(job.pairs[k].read_len) : 0;
    if (!__syncthreads_and(!have || limbs == NW)) {
        uint32_t mine = 0;
#pragma unroll
        for (int c = 0; c <= NW; c++) {
            const uint32_t b = __ballot_sync(0xffffffffu, limbs == c);
            if (limbs == c) mine = b;
            if (lane == 0) s_first[c * WARPS + warp] = (uint32_t)__popc(b);
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t before = 0;
            for (int e = 0; e < ENTRIES; e += 32) {
                const uint32_t v = e + lane < ENTRIES ? s_first[e + lane] : 0u;
                uint32_t x = v;
                for (int d = 1; d < 32; d *= 2) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= d) x += y;
                }
                if (e + lane < ENTRIES) s_first[e + lane] = before + x - v;
                before += __shfl_sync(0xffffffffu, x, 31);
            }
        }
        __syncthreads();
        s_order[s_first[limbs * WARPS + warp] + __popc(mine & ((1u << lane) - 1u))] =
            (uint16_t)threadIdx.x;
        __syncthreads();
        k = base + s_order[threadIdx.x];
        have = k < job.n_pairs;
        limbs = have ? limbs_of<NW>(job.pairs[k].read_len) : 0;
    }
    limbs = max(1, __reduce_max_sync(0xffffffffu, limbs));
    if (have) myers_limbs<NW, GLOB>(job, (uint32_t)k, smem, limbs);
}

// A thread a pair, in the batch's order.
template <int NW, bool GLOB>
__global__ void __launch_bounds__(MY_BLOCK) myers_kernel(const __grid_constant__ MyersJob job) {
    extern __shared__ uint32_t smem[];
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < job.n_pairs) myers_pair<NW, GLOB>(job, (uint32_t)k, smem);
}

template <int NW, bool GLOB>
static void launch_limbs(const MyersJob &job, bool ordered, cudaStream_t st) {
    const size_t smem = (size_t)4 * NW * MY_BLOCK * sizeof(uint32_t);
    const unsigned grid = (unsigned)((job.n_pairs + MY_BLOCK - 1) / MY_BLOCK);
    if (ordered) myers_ordered_kernel<NW, GLOB><<<grid, MY_BLOCK, smem, st>>>(job);
    else myers_kernel<NW, GLOB><<<grid, MY_BLOCK, smem, st>>>(job);
}

cudaError_t launch_myers(const MyersJob &job, int nw, int num_sms, cudaStream_t st) {
    if (job.n_pairs == 0) return cudaSuccess;
    // up to two warps a scheduler a launch lasts as long as its longest pair in
    // any order, and ordering costs 2 us: 12,000 reads of 60 bases 10.9 us, ordered
    // 12.5; 60,000 of 40 to 120 bases 51 us, ordered 41
    const bool ordered = job.n_pairs > (uint64_t)num_sms * 256;
    switch (nw) {
#define ESP_MY_CASE(W)                                                           \
    case W:                                                                      \
        if (job.flags & MYF_GLOBAL) launch_limbs<W, true>(job, ordered, st);     \
        else launch_limbs<W, false>(job, ordered, st);                           \
        break;
        ESP_MY_CASE(1) ESP_MY_CASE(2) ESP_MY_CASE(3) ESP_MY_CASE(4)
        ESP_MY_CASE(5) ESP_MY_CASE(6) ESP_MY_CASE(7) ESP_MY_CASE(8)
#undef ESP_MY_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace esp
