// gotoh.cu -- GB300 banded / full-matrix affine-gap (Gotoh) local alignment
// with traceback to CIGAR, bit-exact with the reference's scalar kernel
// (crates/map/src/extend.rs:606-1068).
//
// Execution model: one thread owns one read x window pair (inter-sequence
// parallelism).  A warp takes 32 consecutive entries of a length-sorted work
// list from a device queue (persistent kernel), so the lanes of a warp run the
// same loop trip counts and their scratch accesses coalesce.
//
// DP layout: the matrix is swept in strips of 8 rows.  Inside a strip the
// thread walks the strip's column range left to right and evaluates the 8
// cells of each column top to bottom, all in registers:
//   * H/F of column j-1 for each of the 8 rows ride in registers (left deps),
//   * H/E of the row above the strip come from a per-thread row buffer (one
//     packed int16x2 word per column) that the strip's last row rewrites in
//     place, so row-buffer traffic is 8 bytes per column per 8 cells,
//   * the 4 traceback bits of the 8 cells are packed into one 32-bit word
//     per (strip, column): 2 bits H source per row in the low half-word and
//     (E opened, F opened) per row in the high half-word.
//
// Scaled-key arithmetic (what makes the reference's tie cascade cheap):
// every score is held as 4*v plus a 2-bit tag so that a plain integer max
// performs both the value comparison and the reference's tie preference.
//   H is held as Hp = 4H + 2, E as E1 = 4E + 1, F as F4 = 4F.
//   Ho = Hp + 4*open_ext opens a gap from a cell, to the right and down: one
//          add serves both.
//   E key: max(E1_up + 4*ext, Ho_up): low bits 2 <=> opened, 1 <=> extended,
//          and an open/extend tie resolves to "open" as `better` (strict >)
//          does at extend.rs:731.
//   F key: max(F4_left + 4*ext, Ho_left): low bits 2 <=> opened, 0 <=>
//          extended; formed as soon as the left cell is (kF), so that a row
//          carries (Hp, kF) to the next column.
//   H key: max(4*diag + 2, E1, F4, 3): among equal values diag beats E beats
//          F (the cascade order of extend.rs:764-777), and the START tag 3
//          wins whenever the maximum is 0 (the zero-floor rewrite of
//          extend.rs:780-782).  hsrc = key & 3: 3 start, 2 diag, 1 E, 0 F.
//   Flags: (kE ^ kF) & 3 has bit 0 clear <=> E opened and bit 1 set <=>
//          exactly one of E, F opened.
// Out-of-window cells present H = 0, E = F = NEG to their neighbours exactly
// as the scalar kernel's margins do (extend.rs:718-759).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "esp_device.cuh"
#include "esp_internal.h"

namespace esp {

static constexpr int STRIP = 8;

struct Geo {
    int off, half, n;
    __device__ __forceinline__ int c(int i) const {
        int x = off + i;
        return x < 1 ? 1 : (x > n ? n : x);
    }
    __device__ __forceinline__ int lo(int i) const {
        int v = c(i) - half;
        return v > 1 ? v : 1;
    }
    __device__ __forceinline__ int hi(int i) const {
        int v = c(i) + half;
        return v < n ? v : n;
    }
};

struct Seq {
    const uint8_t *arena;
    uint64_t pos;
    const esp_n_interval *iv;
    uint32_t cnt;
    __device__ __forceinline__ uint32_t code(int64_t q) const {
        return code5(arena, pos, iv, cnt, q);
    }
};

// Row-max keys are Hp * 32768 + (32767 - j): 32 bits while Hp < 65536 (the
// int16 domain); the wide kernel keeps them in 64 bits.
template <bool WIDE>
struct StripT {
    using RK = typename std::conditional<WIDE, long long, int>::type;
    int Hl[STRIP], kF[STRIP];  // Hp of the column left of the next one; F key of the next one
    RK rk[STRIP];
    uint32_t l0[STRIP], l1[STRIP];
    int lo[STRIP], hi[STRIP];
};
using Strip = StripT<false>;

// a & m and (a & m) | o as opaque logic ops, so that the compiler keeps the
// differences below as adds instead of folding them back into logic.
__device__ __forceinline__ uint32_t and_u32(uint32_t a, uint32_t m) {
    uint32_t d;
    asm("and.b32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(m));
    return d;
}

// (a ^ b) & m in one LOP3
__device__ __forceinline__ uint32_t xor_and_u32(uint32_t a, uint32_t b, uint32_t m) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x28;" : "=r"(d) : "r"(a), "r"(b), "r"(m));
    return d;
}

__device__ __forceinline__ uint32_t and_or_u32(uint32_t a, uint32_t m, uint32_t o) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(m), "r"(o));
    return d;
}

// What a cell outside its row's window (or the matrix) shows to its
// neighbours: H = 0, and an E so low that opening from that H = 0 always
// wins, as it does against the scalar kernel's NEG.
__device__ __forceinline__ int absent_E(const GotohConst &K) { return K.oe4 + 1; }
__device__ __forceinline__ uint32_t absent_HE(const GotohConst &K) {
    return __byte_perm(2u, (uint32_t)absent_E(K), 0x5410);
}

// One column of one strip.  upH/upE enter as the row above the strip at
// column j and leave as the strip's last row at column j; `diag` is the row
// above at column j-1; cj = 32767 - j (row-max key tie order).  MASK = 1
// tests every cell against its row window (strip ramps); MASK = 0 is the
// strip interior where all 8 cells are in window.
template <int MASK, bool WIDE = false>
__device__ __forceinline__ uint32_t dp_column(StripT<WIDE> &S, const GotohConst &K, int j,
                                              uint32_t sel, uint32_t cj, int &upH, int &upE,
                                              int diag) {
    uint32_t wa = 0, wb = 0;
    int d = diag, upHo = upH + K.oe4;
#pragma unroll
    for (int r = 0; r < STRIP; r++) {
        int left = S.Hl[r];
        int kE = max(upE + K.ex4, upHo);
        int kF = S.kF[r];
        int E1 = (int)and_or_u32((uint32_t)kE, ~3u, 1u);
        int F4 = (int)and_u32((uint32_t)kF, ~3u);
        int kd = max(d + prmt_sx(S.l0[r], S.l1[r], sel), 3);  // START tag 3 folded in
        int key = max(max(kd, E1), F4);
        int Hp = (int)and_or_u32((uint32_t)key, ~3u, 2u);
        int Ho = Hp + K.oe4;
        // tags are accumulated as key - Hp = tag - 2 (adds and multiply-adds
        // issue off the saturated ALU pipe); the 2s are put back at the end
        wa = mad_u32(wa, 4u, (uint32_t)(key - Hp));
        wb = mad_u32(wb, 4u, xor_and_u32((uint32_t)kE, (uint32_t)kF, 3u));
        typename StripT<WIDE>::RK rkey;
        if constexpr (WIDE)
            rkey = ((long long)Hp << 15) | (long long)cj;
        else
            rkey = (int)mad_u32((uint32_t)Hp, 32768u, cj);
        kF = max(F4 + K.ex4, Ho);  // of the next column
        if (MASK) {
            // An out-of-window cell shows H = 0 and no E to the row below and
            // leaves its own row's state alone: before the window that is still
            // the start state, after it Hl keeps H at the window's last
            // column (the strip's bookkeeping reads it; the cells of the row
            // below that follow are out of their window too, as hi(i+1) <=
            // hi(i) + 1).
            const bool in = (j >= S.lo[r]) & (j <= S.hi[r]);
            if (in) {
                S.rk[r] = max(S.rk[r], rkey);
                S.Hl[r] = Hp;
                S.kF[r] = kF;
            }
            upHo = in ? Ho : 2 + K.oe4;
            upE = in ? E1 : absent_E(K);
        } else {
            S.rk[r] = max(S.rk[r], rkey);
            S.Hl[r] = Hp;
            S.kF[r] = kF;
            upHo = Ho;
            upE = E1;
        }
        d = left;
    }
    upH = upHo - K.oe4;
    return __byte_perm(wa + 0xAAAAu, wb, 0x5410);
}

struct FillResult {
    int bestHp, best_i, best_j;
    int last_j;  // the best cell is row best_i's first cell of value bestHp in [best_j, last_j]
    int trow;
    bool tleft, tclamp;
};

// Columns [a, b] of the current strip.  Window codes are fetched 16 at a
// time.  CHECK = true (strip ramps) tests the row-buffer read (the row above
// has a value only up to phi) and write (the strip's last row starts at
// lo7) per column; the interior needs neither test.
template <int MASK, bool CHECK, bool HASN>
__device__ __forceinline__ void dp_cols(Strip &S, const GotohConst &K, int a, int b, int &diag,
                                        const Seq &win, uint32_t *rb, int plo, int phi, int lo7,
                                        uint32_t *tbp) {
    uint32_t *rbr = rb + (size_t)(a - plo) * 32;
    uint32_t cj = 32767u - (uint32_t)a;
    // Interior: the row above is read two columns ahead of its use (the
    // L2 round trip of a row-buffer line is longer than one column of
    // arithmetic).  A slot is rewritten only at or after the column that
    // reads it, so the values fetched early are still the row above.
    uint32_t wn0 = 0, wn1 = 0;
    if (!CHECK) {
        wn0 = rbr[0];
        if (a + 1 <= b) wn1 = rbr[32];
    }
    for (int j = a; j <= b;) {
        uint32_t cw = load16(win.arena, win.pos + (uint64_t)(j - 1));
        uint32_t nm = HASN ? nmask16(win.iv, win.cnt, j - 1) : 0u;
        int cnt = min(16, b - j + 1);
#pragma unroll 1  // measured: the rolled loop beats unroll 2 (+13%) and 4
        for (int k = 0; k < cnt; k++, j++) {
            uint32_t code = HASN ? ((cw >> 30) | ((nm >> 29) & 4u)) : (cw >> 30);
            cw <<= 2;
            if (HASN) nm <<= 1;
            uint32_t sel = code * 0x1111u + 0x8880u;
            int bH = 2, bE = absent_E(K);
            if (!CHECK || j <= phi) {
                uint32_t w;
                if (CHECK) {
                    w = *rbr;
                } else {
                    w = wn0;
                    wn0 = wn1;
                    if (j + 2 <= b) wn1 = rbr[64];
                }
                bH = (int)(w & 0xffffu);
                bE = ((int)w) >> 16;
            }
            int upH = bH, upE = bE;
            uint32_t word = dp_column<MASK>(S, K, j, sel, cj, upH, upE, diag);
            diag = bH;
            uint32_t packed = __byte_perm((uint32_t)upH, (uint32_t)upE, 0x5410);
            if (CHECK) {
                if (j >= lo7) rb[(size_t)(j - lo7) * 32] = packed;
            } else {
                rbr[(ptrdiff_t)(plo - lo7) * 32] = packed;  // row-buffer slot j - lo7
            }
            *tbp = word;
            tbp += 32;
            rbr += 32;
            cj--;
        }
    }
}

// Fill the DP for one pair; traceback words land in tb (sw words per strip, 32
// words apart: the lanes of a warp interleave theirs).
// The row buffer holds sw words: strip 0 reads row 0 (H = 0, E = NEG on every
// column, extend.rs:664-681) from a prefilled copy, later strips read the last
// row of the previous strip, which each strip rewrites in place (a slot is
// always read at or before the column that overwrites it, since the strip's
// window start lo7 never precedes the previous row's start plo).
template <bool HASN>
__device__ FillResult dp_fill(const GotohConst &K, const uint32_t *__restrict__ s_lut, int m,
                              int n, const Geo &g, const Seq &read, const Seq &win,
                              uint32_t *tb, int sw, uint32_t *rb) {
    FillResult R;
    R.bestHp = 2;
    R.best_i = 0;
    R.best_j = R.last_j = 0;
    R.trow = 0;
    R.tleft = false;
    R.tclamp = false;
    int nstrips = (m + STRIP - 1) / STRIP;
    int plo = g.lo(1), phi = g.hi(min(STRIP, m));
    {
        const uint32_t row0 = absent_HE(K);
        for (int k = 0; k <= phi - plo; k++) rb[(size_t)k * 32] = row0;
    }
    Strip S;
    for (int s = 0; s < nstrips; s++) {
        int i0 = s * STRIP + 1;
        int nact = min(STRIP, m - i0 + 1);
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            S.lo[r] = g.lo(i0 + r);
            S.hi[r] = g.hi(i0 + r);
            S.Hl[r] = 2;
            S.kF[r] = 2 + K.oe4;  // F opened from H = 0
            S.rk[r] = -1;
        }
        int clo = S.lo[0];
        int chi = g.hi(i0 + nact - 1);
        int lo7 = S.lo[STRIP - 1];
        int hi0 = S.hi[0];
        // read codes of the strip's rows -> per-row substitution words
        uint32_t rw = load16(read.arena, read.pos + (uint64_t)(i0 - 1));
        uint32_t rn = read.cnt ? nmask16(read.iv, read.cnt, i0 - 1) : 0u;
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            uint32_t c = (rw >> (30 - 2 * r)) & 3u;
            if ((rn >> (31 - r)) & 1u) c = 4;
            S.l0[r] = s_lut[2 * c];
            S.l1[r] = s_lut[2 * c + 1];
        }
        int diag = 2;
        if (clo - 1 >= plo && clo - 1 <= phi)
            diag = (int)(rb[(size_t)(clo - 1 - plo) * 32] & 0xffffu);
        uint32_t *tbp = tb + (size_t)s * sw * 32;
        int a_end = min(lo7, chi);
        dp_cols<1, true, HASN>(S, K, clo, a_end, diag, win, rb, plo, phi, lo7, tbp);
        int b_beg = lo7 + 1, b_end = min(hi0 - 1, chi);
        if (b_beg <= b_end)
            dp_cols<0, false, HASN>(S, K, b_beg, b_end, diag, win, rb, plo, phi, lo7,
                                    tbp + (size_t)(b_beg - clo) * 32);
        int c_beg = max(lo7 + 1, hi0);
        // the row windows again rather than kept live across the interior
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            S.lo[r] = g.lo(i0 + r);
            S.hi[r] = g.hi(i0 + r);
        }
        if (c_beg <= chi)
            dp_cols<1, true, HASN>(S, K, c_beg, chi, diag, win, rb, plo, phi, lo7,
                                   tbp + (size_t)(c_beg - clo) * 32);
        // row bookkeeping in row order (extend.rs:795-827)
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            if (r < nact) {
                int rowHp = S.rk[r] >> 15;
                int argj = 32767 - (S.rk[r] & 32767);
                if (R.trow == 0) {
                    if (argj == S.lo[r]) {  // H at the left edge is the row max
                        R.trow = i0 + r;
                        R.tleft = true;
                        R.tclamp = S.lo[r] <= 1;
                    } else if (S.hi[r] < n && S.Hl[r] == rowHp) {
                        R.trow = i0 + r;
                        R.tleft = false;
                        R.tclamp = S.hi[r] >= n;
                    }
                }
                if (rowHp > R.bestHp) {
                    R.bestHp = rowHp;
                    R.best_i = i0 + r;
                    R.best_j = R.last_j = argj;
                }
            }
        }
        plo = lo7;
        phi = S.hi[STRIP - 1];
    }
    return R;
}

__device__ __forceinline__ bool neutral_col(uint32_t q, uint32_t r) {
    return q < 4 && r < 4 && (q == r || (r == 0 && q == 2) || (r == 3 && q == 1));
}

// Step kinds of a traceback walk: M with a match / mismatch / zero
// (editing-exempt) score, I or D opening a gap run (walk order), I or D
// extending it.
enum : int { K_MM = 0, K_MX = 1, K_MZ = 2, K_IO = 3, K_IE = 4, K_DO = 5, K_DE = 6 };
constexpr int REC_RUNS = 64;  // recorded runs of equal steps; walks with more walk twice
constexpr int RUNS_LOCAL = 16;  // CIGAR runs kept in the thread's own list

__device__ __forceinline__ int kind_op(int k) { return k < 3 ? ESP_OP_M : (k < 5 ? ESP_OP_I : ESP_OP_D); }

// The 32 bases ending at position q - 1 of a sequence, base q - 1 in bits
// 1:0, q - 2 in bits 3:2, ...; zeros above the sequence's first base.
// Reads no word past the one after the word that holds base q - 1.
__device__ __forceinline__ uint64_t tail32(const uint8_t *__restrict__ arena, uint64_t pos, int q) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(arena);
    const int q0 = q >= 32 ? q - 32 : 0;
    const uint64_t p0 = pos + (uint64_t)q0, wi = p0 >> 4, wl = (pos + (uint64_t)(q - 1)) >> 4;
    const uint32_t sh = (uint32_t)(p0 & 15) * 2;
    const uint32_t a = __byte_perm(__ldg(w + wi), 0, 0x0123);
    const uint32_t b = __byte_perm(__ldg(w + wi + 1), 0, 0x0123);
    const uint32_t c = __byte_perm(__ldg(w + (wi + 2 <= wl + 1 ? wi + 2 : wl + 1)), 0, 0x0123);
    const uint64_t v = ((uint64_t)__funnelshift_l(b, a, sh) << 32) | __funnelshift_l(c, b, sh);
    return v >> (2 * (32 - (q - q0)));
}

// Bases between position q and the nearest N below it (q itself when there
// is none): how far a run of matches ending at q - 1 may reach.
__device__ __forceinline__ int n_free(const esp_n_interval *iv, uint32_t cnt, int q) {
    int room = q;
    for (uint32_t k = 0; k < cnt; k++)
        if ((int)iv[k].start < q) room = min(room, q - min((int)iv[k].end, q));
    return room;
}

// Where a fill left the traceback word of (strip s, column j): sw words a
// strip from its first column on, STR words apart (the lanes of a warp
// interleave theirs; 1: a warp's own pair).
template <int STR>
struct StripTb {
    const uint32_t *tb;
    int sw;
    __device__ __forceinline__ uint32_t word(const Geo &g, int s, int j) const {
        // word indices fit 32 bits: a slot holds at most 4,096 strips of
        // 32,767 columns
        return tb[(size_t)(uint32_t)(s * sw + (j - g.lo(s * STRIP + 1))) * STR];
    }
};

// One traceback walk over the packed bits (extend.rs:884-930): state machine
// H/E/F from (best_i, best_j), stopping at i <= 0, j <= 0, outside the row
// window, or on an H START cell.
//
// A matching base in state H always steps along the diagonal, whatever the
// traceback word says, so the walk takes a run of matches in one move from
// the sequences alone and reads a word only at the other steps.  Why: with
// match the largest substitution score, match > 0 and gap costs >= 0, take
// an in-window cell (i, j) of equal bases whose predecessor (i-1, j-1) is in
// the window too.  A path into E(i, j) that leaves row i-k in H, shifted one
// column left, runs inside the window (row windows move right by 0 or 1
// columns a row) and shows H(i-1, j-1) >= E(i, j) - match; the same for
// F(i, j) and a path shifted up one row.  So the diagonal's value is >= E, F
// and > 0, and diagonal wins ties: hsrc is diag.  On the matrix border (i = 1
// or j = 1) E and F are at most match, and the same holds.  Only where the
// predecessor lies outside the window (the left edge of a band clamped at
// the window's end) is the word read for a match.  `skip` is K.match_skip.
//
// A read of a 2 % error rate so costs its ~4 mismatches and a 32-base
// compare per 32 bases instead of ~175 dependent word loads and state steps;
// measured when it came: 4,194,304 mixed pairs 49.8 -> 43.9 ms, one
// extend_hint call 146 -> 109 us.
template <class TB>
struct Walker {
    const Geo &g;
    const TB &tb;
    const Seq &read;
    const Seq &win;
    const GotohConst &K;
    int i, j, state;
    bool over = false;  // on an H START cell
    // the bases from (i, j) down, at bits 1:0 up, and how many are left
    uint64_t rv = 0, wv = 0;
    int rl = 0, wl = 0;

    __device__ Walker(const Geo &g_, const TB &tb_, const Seq &r_, const Seq &w_,
                      const GotohConst &K_, int bi, int bj)
        : g(g_), tb(tb_), read(r_), win(w_), K(K_), i(bi), j(bj), state(0) {}

    // Take a run of `len` matches (0..32) and then one step of `kind` (-1:
    // none this time).  Returns false when the walk stops (with len = 0).
    __device__ __forceinline__ bool next(int &len, int &kind) {
        len = 0;
        kind = -1;
        if (over || i <= 0 || j <= 0) return false;
        if (j < g.lo(i) || j > g.hi(i)) return false;
        uint32_t q = 4, rc = 4;  // base codes at the walk's position (state H)
        if (state == 0) {
            if (rl <= 0 || wl <= 0) {
                rv = tail32(read.arena, read.pos, i);
                wv = tail32(win.arena, win.pos, j);
                rl = min(i, 32);
                wl = min(j, 32);
            }
            uint64_t d = rv ^ wv;
            d = (d | (d >> 1)) & 0x5555555555555555ull;
            int room = min(rl, wl), rn = i, wn = j;
            if (read.cnt) rn = n_free(read.iv, read.cnt, i);
            if (win.cnt) wn = n_free(win.iv, win.cnt, j);
            const int known = room;
            room = min(room, min(rn, wn));
            int run = min(room, d ? (__ffsll((long long)d) - 1) >> 1 : 32);
            // every predecessor in the window: i - lo(i) - j grows upwards
            // along the diagonal, so the lowest one decides
            const int e = run == i || run == j ? run - 1 : run;
            if (!K.match_skip || (e > 0 && j - e < g.lo(i - e))) run = 0;
            if (run) {
                len = run;
                i -= run;
                j -= run;
                rl -= run;
                wl -= run;
                if (run == known || i <= 0 || j <= 0) return true;
                if (j < g.lo(i)) return true;  // the next call stops there
                rv >>= 2 * run;
                wv >>= 2 * run;
                rn -= run;
                wn -= run;
            }
            q = rn == 0 ? 4u : (uint32_t)rv & 3u;
            rc = wn == 0 ? 4u : (uint32_t)wv & 3u;
        }
        const int s = (i - 1) >> 3, r = (i - 1) & 7;
        const uint32_t w = tb.word(g, s, j);
        const int sh = 2 * (7 - r);
        const uint32_t hsrc = (w >> sh) & 3u;
        const uint32_t eo = ~(w >> (16 + sh)) & 1u;
        const uint32_t fo = ((w >> (17 + sh)) & 1u) ^ eo;
        // the step's source: the cell's H tag in state 0, else the gap it is in
        const uint32_t eff = state == 0 ? hsrc : (state == 1 ? 1u : 0u);
        if (eff == 3u) {  // H_START: the walk ends after the run just taken
            over = true;
            return len != 0;
        }
        const int open = state == 0;
        const int kdiag = (int)((K.dkind >> (2 * (q * 5 + rc))) & 3u);
        const int kvert = open ? K_IO : K_IE, khor = open ? K_DO : K_DE;
        kind = eff == 2u ? kdiag : (eff == 1u ? kvert : khor);
        state = eff == 2u ? 0 : (eff == 1u ? (eo ? 0 : 1) : (fo ? 0 : 2));
        if (eff != 0u) {
            i--;
            rv >>= 2;
            rl--;
        }
        if (eff != 1u) {
            j--;
            wv >>= 2;
            wl--;
        }
        return true;
    }
};

// Score of one traceback step.
__device__ __forceinline__ int delta_of(const GotohConst &K, int kind) {
    return kind < 3 ? (kind == K_MM ? K.match : (kind == K_MX ? (int)K.lut[1] : 0))
                    : ((kind & 1) ? K.open_ext : K.ext);
}

// The kept part of an alignment: its CIGAR runs in walk order, ends and score.
// Runs go to the thread's local list, so short CIGARs are written once, in
// final order, with no global read-back, and need only their final length in
// capacity; a long CIGAR moves the list to its slots cig[2..] (and needs them:
// it is reversed there in place).
struct Kept {
    uint32_t rr[RUNS_LOCAL];
    uint32_t runs;
    uint32_t read_start, ref_start, read_end, ref_end;
    int score;
    int first_op, last_op;  // forward order
    bool overflow;
    __device__ __forceinline__ void emit(uint32_t v, uint32_t *cig, uint32_t cap) {
        if (runs < RUNS_LOCAL) {
            rr[runs] = v;
        } else {
            if (2 + runs < cap) {
                if (runs == RUNS_LOCAL)
                    for (int k = 0; k < RUNS_LOCAL; k++) cig[2 + k] = rr[k];
                cig[2 + runs] = v;
            } else {
                overflow = true;
            }
        }
        runs++;
    }
};

// Walk the traceback from (F.best_i, j) and keep all of it.  Returns whether
// that is the alignment: its total is the best score T and the end trim
// (extend.rs:931-968) takes nothing off, i.e. the walk-order prefix sums stay
// positive and reach T with the last step only.  (They do for an optimal
// local alignment; the general rule is walk_trimmed.)
template <class TB>
__device__ __forceinline__ bool walk_whole(const GotohConst &K, const Geo &g, const TB &tb,
                                           const Seq &read, const Seq &win, int bi, int bj, int T,
                                           Kept &k, uint32_t *cig, uint32_t cap) {
    Walker<TB> W(g, tb, read, win, K, bi, bj);
    int P = 0, cur_op = ESP_OP_M, last_op = -1, len, kind;
    uint32_t cur_len = 0;
    bool whole = true;
    k.runs = 0;
    k.overflow = false;
    // no early way out: the lanes of a warp leave the loop together
    while (W.next(len, kind)) {
        const int op = kind < 0 ? ESP_OP_M : kind_op(kind);
        if (len) {
            whole = whole && P + (len - 1) * K.match < T;
            P += len * K.match;
            if (cur_op != ESP_OP_M) {
                k.emit((cur_len << 4) | (uint32_t)cur_op, cig, cap);
                cur_op = ESP_OP_M;
                cur_len = 0;
            }
            cur_len += (uint32_t)len;
            if (last_op < 0) last_op = ESP_OP_M;
        }
        if (kind >= 0) {
            whole = whole && P < T;
            P += delta_of(K, kind);
            whole = whole && P > 0;
            if (op != cur_op) {
                if (cur_len) k.emit((cur_len << 4) | (uint32_t)cur_op, cig, cap);
                cur_op = op;
                cur_len = 0;
            }
            cur_len++;
            if (last_op < 0) last_op = op;
        }
    }
    whole = whole && P == T && cur_len != 0;
    if (whole) k.emit((cur_len << 4) | (uint32_t)cur_op, cig, cap);
    k.first_op = cur_op;
    k.last_op = last_op;
    k.read_start = (uint32_t)W.i;
    k.ref_start = (uint32_t)W.j;
    k.read_end = (uint32_t)bi;
    k.ref_end = (uint32_t)bj;
    k.score = P;
    return whole;
}

// The same with the end trim: walk 1 records the walk as runs of equal steps
// (len << 3 | kind) and finds its number of steps N, its total T and trail
// (its steps up to and including the last non-positive prefix sum).
template <class TB>
__device__ __noinline__ void walk_trimmed(const GotohConst &K, const Geo &g, const TB &tb,
                                          const Seq &read, const Seq &win, int best_i, int best_j,
                                          Kept &kept, uint32_t *cig, uint32_t cap) {
    uint32_t rec[REC_RUNS];
    int n_rec = 0, N = 0, P = 0, trail = 0;
    {
        Walker<TB> W(g, tb, read, win, K, best_i, best_j);
        uint32_t open = 0;  // the run being extended (0: none yet)
        auto add = [&](int kind, int len) {
            if (open && (int)(open & 7u) == kind) {
                open += (uint32_t)len << 3;
            } else {
                if (open) {
                    if (n_rec < REC_RUNS) rec[n_rec] = open;
                    n_rec++;
                }
                open = ((uint32_t)len << 3) | (uint32_t)kind;
            }
        };
        int len, kind;
        while (W.next(len, kind)) {
            if (len) {  // match > 0 here: the prefix sums of the run rise
                if (P < 0) {
                    const int k = min(len, -P / K.match);
                    if (k) trail = N + k;
                }
                P += len * K.match;
                N += len;
                add(K_MM, len);
            }
            if (kind >= 0) {
                P += delta_of(K, kind);
                N++;
                if (P <= 0) trail = N;
                add(kind, 1);
            }
        }
        if (open) {
            if (n_rec < REC_RUNS) rec[n_rec] = open;
            n_rec++;
        }
    }
    const int T = P;
    kept.runs = 0;
    kept.overflow = false;
    kept.first_op = kept.last_op = -1;
    kept.score = 0;
    if (N == 0) {
        kept.read_start = (uint32_t)max(best_i, 0);
        kept.ref_start = (uint32_t)max(best_j, 0);
        kept.read_end = kept.read_start;
        kept.ref_end = kept.ref_start;
    } else {
        // With walk-order prefix sums P_t, the reference's forward lead is
        // N-1-u where u is the first index in [-1, N-2] with P_u >= T
        // (P_-1 = 0).  The kept steps are walk indices [trail, u] -- through
        // N-1 when no u exists -- and lead + trail >= N (the degenerate
        // keep-the-middle case, extend.rs:956-960) is exactly u < trail, or
        // T <= 0: then step tstar alone is kept, captured on the way.  A run
        // of equal steps crosses T at most once, and only rising.
        bool degenerate = T <= 0, done = false;
        const int tstar = N - 1 - N / 2;
        int i = best_i, j = best_j;
        int t0 = 0, P0 = 0, ptrail = 0;
        int ts_i = 0, ts_j = 0, ts_op = 0, ts_d = 0;
        int cur_op = -1;
        uint32_t cur_len = 0;
        auto take = [&](int kind, int len) {
            const int op = kind_op(kind), d = delta_of(K, kind);
            const int di = op != ESP_OP_D, dj = op != ESP_OP_I;
            if (tstar >= t0 && tstar < t0 + len) {
                ts_i = i - di * (tstar - t0);
                ts_j = j - dj * (tstar - t0);
                ts_op = op;
                ts_d = d;
            }
            int end = t0 + len - 1;
            if (!degenerate && d > 0 && P0 + d * len >= T) {  // P0 < T here
                const int u = t0 + (T - P0 + d - 1) / d - 1;
                if (u <= N - 2) {
                    end = u;
                    done = true;
                    degenerate = u < trail;
                }
            }
            if (!degenerate && end >= trail) {
                const int a = max(t0, trail);
                if (cur_op < 0) {  // the kept region's end (forward order)
                    kept.read_end = (uint32_t)(i - di * (a - t0));
                    kept.ref_end = (uint32_t)(j - dj * (a - t0));
                    ptrail = P0 + d * (a - t0);
                    kept.last_op = op;
                    cur_op = op;
                }
                if (op != cur_op) {
                    kept.emit((cur_len << 4) | (uint32_t)cur_op, cig, cap);
                    cur_op = op;
                    cur_len = 0;
                }
                cur_len += (uint32_t)(end - a + 1);
            }
            const int k = end - t0 + 1;
            i -= di * k;
            j -= dj * k;
            P0 += d * k;
            t0 += k;
            if (degenerate) {  // run on to tstar (it may lie past this end)
                i -= di * (len - k);
                j -= dj * (len - k);
                t0 += len - k;
                done = t0 > tstar;
            }
        };
        if (n_rec <= REC_RUNS) {
            for (int k = 0; k < n_rec && !done; k++) take((int)(rec[k] & 7u), (int)(rec[k] >> 3));
        } else {  // more runs than the record holds: walk again
            Walker<TB> W(g, tb, read, win, K, best_i, best_j);
            int len, kind;
            while (!done && W.next(len, kind)) {
                if (len) take(K_MM, len);
                if (kind >= 0 && !done) take(kind, 1);
            }
        }
        if (degenerate) {
            kept.read_end = (uint32_t)ts_i;
            kept.ref_end = (uint32_t)ts_j;
            kept.read_start = (uint32_t)(ts_i - (ts_op != ESP_OP_D));
            kept.ref_start = (uint32_t)(ts_j - (ts_op != ESP_OP_I));
            kept.score = ts_d;
            kept.runs = 0;
            kept.emit((1u << 4) | (uint32_t)ts_op, cig, cap);
            kept.first_op = kept.last_op = ts_op;
        } else {
            kept.emit((cur_len << 4) | (uint32_t)cur_op, cig, cap);
            kept.first_op = cur_op;
            kept.read_start = (uint32_t)i;
            kept.ref_start = (uint32_t)j;
            kept.score = P0 - ptrail;
        }
    }
}

// Traceback, end trimming, rebuild and neutral flanks (extend.rs:864-1068).
template <class TB>
__device__ void dp_finish(const GotohConst &K, const int8_t *__restrict__ lut, const Geo &g,
                          const TB &tb, int m, int n, const Seq &read, const Seq &win,
                          const FillResult &F, esp_extension &o, uint32_t *cig, uint32_t cap) {
    // When the best cell's column is known as a range, its columns are walked
    // in order until one's total is the best score: a walk's total is its
    // cell's H, and the first such cell is the best one.  (With mismatches
    // scoring <= 0 it ends on a match: a cell that equals the best by any
    // other step has an equal cell before it in row order.)
    Kept kept;
    const int T = (F.bestHp - 2) >> 2;
    bool done = false;
    int bj = F.best_j;
    if (T > 0) {
        const bool on_match = K.match_skip && K.lut[1] <= 0;
        do {
            while (on_match && bj < F.last_j && read.code(F.best_i - 1) != win.code(bj - 1)) bj++;
            done = walk_whole(K, g, tb, read, win, F.best_i, bj, T, kept, cig, cap);
        } while (!done && ++bj <= F.last_j);
        bj = min(bj, F.last_j);
    }
    if (!done) {
        // a trimmed alignment: the first column whose walk's total is T
        for (int j = F.best_j; j < F.last_j; j++) {
            Walker<TB> W(g, tb, read, win, K, F.best_i, j);
            int P = 0, len, kind;
            while (W.next(len, kind)) P += len * K.match + (kind >= 0 ? delta_of(K, kind) : 0);
            bj = j;
            if (P == T) break;
            bj = F.last_j;
        }
        walk_trimmed(K, g, tb, read, win, F.best_i, bj, kept, cig, cap);
    }
    uint32_t read_start = kept.read_start, ref_start = kept.ref_start;
    uint32_t read_end = kept.read_end;
    const uint32_t ref_end = kept.ref_end, K_runs = kept.runs;
    const int score = kept.score, first_op = kept.first_op, last_op = kept.last_op;
    // reverse the kept runs into forward order (a long CIGAR's, in place)
    if (!kept.overflow && K_runs > RUNS_LOCAL) {
        for (uint32_t a = 0, b = K_runs ? K_runs - 1 : 0; a < b; a++, b--) {
            uint32_t t = cig[2 + a];
            cig[2 + a] = cig[2 + b];
            cig[2 + b] = t;
        }
    }
    // neutral flanks (extend.rs:991-1049)
    uint32_t nl = 0, nr = 0;
    if (score > 0) {
        int delta = 0;
        uint32_t lim = min(read_start, ref_start);
        for (uint32_t k = 1; k <= lim; k++) {
            uint32_t q = read.code((int64_t)read_start - k), r = win.code((int64_t)ref_start - k);
            if (!neutral_col(q, r)) break;
            delta += lut[q * 5 + r];
            if (delta == 0) nl = k;
        }
        delta = 0;
        uint32_t av = min((uint32_t)m - read_end, (uint32_t)n - ref_end);
        for (uint32_t k = 0; k < av; k++) {
            uint32_t q = read.code((int64_t)read_end + k), r = win.code((int64_t)ref_end + k);
            if (!neutral_col(q, r)) break;
            delta += lut[q * 5 + r];
            if (delta == 0) nr = k + 1;
        }
        read_start -= nl;
        ref_start -= nl;
        read_end += nr;
    }
    // final CIGAR: S, M(neutral), kept runs, M(neutral), S (push_op merging)
    uint32_t total = K_runs;
    if (nl > 0 && first_op != ESP_OP_M) total++;
    if (nr > 0 && last_op != ESP_OP_M) total++;
    if (read_start > 0) total++;
    if (read_end < (uint32_t)m) total++;
    if (!kept.overflow && total <= cap) {
        uint32_t w = 0;
        int prev = -1;
        auto push = [&](uint32_t op, uint32_t len) {
            if ((int)op == prev) {
                cig[w - 1] += len << 4;
            } else {
                cig[w++] = (len << 4) | op;
                prev = (int)op;
            }
        };
        if (read_start > 0) push(ESP_OP_S, read_start);
        if (nl > 0) push(ESP_OP_M, nl);
        for (uint32_t k = 0; k < K_runs; k++) {
            uint32_t v = K_runs <= RUNS_LOCAL ? kept.rr[K_runs - 1 - k] : cig[2 + k];
            push(v & 15u, v >> 4);
        }
        if (nr > 0) push(ESP_OP_M, nr);
        if (read_end < (uint32_t)m) push(ESP_OP_S, (uint32_t)m - read_end);
        o.status = ESP_OK;
    } else {
        o.status = ESP_ECAP;
    }
    o.n_ops = total;
    o.read_start = read_start;
    o.read_end = read_end;
    o.ref_start = ref_start;
    o.score = score;
}

// A validated pair: geometry for the job's mode, sequences, output slot and
// the result record being built.
struct PairSetup {
    int m, n, sw;
    bool full;
    Geo g;
    Seq read, win;
    uint32_t *cig;
    esp_extension o;
};

// Validate pair pi and resolve its band geometry (extend.rs:392-428 for the
// extend_hint attempts).  Returns true when a DP is needed; otherwise the
// result (empty extension, or a refusal) has been written when `write`.
__device__ __forceinline__ bool setup_pair(const GotohJob &job, const GotohConst &K, uint32_t pi,
                                           uint64_t tb_cap, uint64_t rb_cap, bool write,
                                           PairSetup &S) {
    if (pi >= job.n_pairs) return false;  // corrupt work list: never index past the batch
    esp_pair P = job.pairs[pi];
    int m = (int)P.read_len, n = (int)P.win_len;
    esp_extension &o = S.o;
    o.read_start = o.read_end = o.ref_start = 0;
    o.score = 0;
    o.n_ops = 0;
    o.touch_row = 0;
    o.touched = o.touch_left = o.touch_clamped = 0;
    o.escalated = job.mode == 2 ? 1 : 0;
    o.status = ESP_OK;
    S.cig = job.cigar + (uint64_t)pi * job.cigar_stride;
    if (m == 0 || n == 0) {  // extend.rs:430-442 empty_extension
        if (m > 0) {
            o.n_ops = 1;
            if (job.cigar_stride >= 1) {
                if (write) S.cig[0] = ((uint32_t)m << 4) | ESP_OP_S;
            } else {
                o.status = ESP_ECAP;
            }
        }
        if (write) job.out[pi] = o;
        return false;
    }
    Geo g;
    bool full;
    // an offset past either end of the longest sequences puts every row's
    // centre on column 1 or n, however far past: sums with it stay in 32 bits
    const int offset = min(max(P.band_offset, -65536), 65536);
    if (job.mode == 0) {
        full = P.band_half < 0;
        g.off = full ? 0 : offset;
        g.half = full ? n : P.band_half;
    } else if (job.mode == 1) {
        full = 30 >= n;  // INITIAL_BAND >= window: full matrix, accepted directly
        g.off = full ? 0 : offset;
        g.half = full ? n : 30;
    } else {
        full = true;
        g.off = 0;
        g.half = n;
    }
    g.n = n;
    int sw = full ? n : min(2 * g.half + STRIP, n);
    uint64_t need_tb = (uint64_t)((m + STRIP - 1) / STRIP) * (uint64_t)sw;
    uint64_t need_rb = (uint64_t)sw;
    const uint8_t *warena = job.win_arena ? job.win_arena : job.arena;
    const uint64_t wbases = job.win_arena ? job.win_arena_bases : job.arena_bases;
    const bool outside = (uint64_t)P.n_first + P.n_read + P.n_win > job.n_iv_count ||
                         P.read_pos + (uint64_t)m > job.arena_bases ||
                         P.win_pos + (uint64_t)n > wbases || m > 32767 || n > 32767;
    if (!outside && m > K.max_m && !job.wide && job.wide_list) {
        // scores may leave the int16 domain: the wide kernel runs this pair
        if (write) job.wide_list[atomicAdd(job.wide_count, 1u)] = pi;
        return false;
    }
    if (need_tb > tb_cap || need_rb > rb_cap || outside || (m > K.max_m && !job.wide)) {
        // scratch sized too small by the host, or the pair lies outside its
        // tables: refuse, never overrun
        o.status = ESP_EINVAL;
        if (write) job.out[pi] = o;
        return false;
    }
    const esp_n_interval *iv = job.n_iv + P.n_first;
    S.read = Seq{job.arena, P.read_pos, iv, P.n_read};
    S.win = Seq{warena, P.win_pos, iv + P.n_read, P.n_win};
    S.m = m;
    S.n = n;
    S.sw = sw;
    S.full = full;
    S.g = g;
    return true;
}

// Traceback, CIGAR, TouchRec, extend_hint escalation (extend.rs:421-426),
// then the result record.  Returns whether attempt 1 escalates; the pair is
// appended to the escalation list when `queue` (the wide kernel runs its
// second attempt itself).
template <class TB>
__device__ __forceinline__ bool finish_pair(const GotohJob &job, const GotohConst &K,
                                            const int8_t *__restrict__ lut, uint32_t pi,
                                            PairSetup &S, const FillResult &F, const TB &tb,
                                            bool queue = true) {
    esp_extension &o = S.o;
    // A touched band escalates whatever its score: the second attempt writes
    // the pair's record and CIGAR, so the first one's are not built.
    if (job.mode == 1 && !S.full && F.trow != 0) {
        if (queue) job.esc_list[atomicAdd(job.esc_count, 1u)] = pi;
        return true;
    }
    dp_finish(K, lut, S.g, tb, S.m, S.n, S.read, S.win, F, o, S.cig,
                   job.cigar_stride);
    if (F.trow) {
        o.touched = 1;
        o.touch_row = F.trow;
        o.touch_left = F.tleft ? 1 : 0;
        o.touch_clamped = F.tclamp ? 1 : 0;
    }
    bool esc = false;
    if (job.mode == 1 && !S.full) {
        // escalate (on a band-edge touch, above, or) below 85% of perfect
        int perfect = S.m * K.match;
        if (o.score * 20 < perfect * 17) {
            if (queue) job.esc_list[atomicAdd(job.esc_count, 1u)] = pi;
            o.escalated = 1;
            esc = true;
        }
    }
    job.out[pi] = o;
    return esc;
}

// Whether a window of the batch may hold N (counted with the bins).
__device__ __forceinline__ bool windows_n(const GotohJob &job) {
    return job.window_n ? *job.window_n != 0 : job.n_iv_count != 0;
}

__device__ void process_pair(const GotohJob &job, const GotohConst &K,
                             const uint32_t *__restrict__ s_lut, const int8_t *__restrict__ lut,
                             uint32_t pi, uint32_t *tb, uint32_t *rb) {
    PairSetup S;
    if (!setup_pair(job, K, pi, job.tb_words, job.rb_words, true, S)) return;
    // one fill for the batch: lanes with N and lanes without would take turns
    FillResult F =
        windows_n(job) ? dp_fill<true>(K, s_lut, S.m, S.n, S.g, S.read, S.win, tb, S.sw, rb)
                  : dp_fill<false>(K, s_lut, S.m, S.n, S.g, S.read, S.win, tb, S.sw, rb);
    finish_pair(job, K, lut, pi, S, F, StripTb<32>{tb, S.sw});
}

template <int MINB>
__global__ void __launch_bounds__(128, MINB) gotoh_kernel(GotohJob job, GotohConst K) {
    if (job.list_count && *job.list_count == 0) return;  // the plan gave the list to another kernel
    __shared__ uint32_t s_lut[10];
    __shared__ int8_t s_lut25[32];
    if (threadIdx.x == 0) {  // static indices keep the parameter block out of local memory
#pragma unroll
        for (int k = 0; k < 10; k++) s_lut[k] = K.lut4[k >> 1][k & 1];
#pragma unroll
        for (int k = 0; k < 25; k++) s_lut25[k] = K.lut[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t warp_slot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t *tb = job.tb + warp_slot * job.tb_words * 32 + lane;
    uint32_t *rb = job.rb + warp_slot * job.rb_words * 32 + lane;
    uint64_t b0 = 0, total = job.list_count ? (uint64_t)(*job.list_count) : job.n_pairs;
    if (job.range) {  // one length class of the binned list
        b0 = job.range[0];
        total = job.range[1] > job.range[0] ? job.range[1] - job.range[0] : 0;
    }
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd((unsigned long long *)job.queue, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= total) break;
        uint64_t k = base + lane;
        if (k < total) {
            uint32_t pi = job.list ? job.list[b0 + k] : (uint32_t)(b0 + k);
            process_pair(job, K, s_lut, s_lut25, pi, tb, rb);
        }
        // lanes whose first attempt was touched are done early; without this the
        // warp takes its next pairs in two parts (200,000 extend_hint pairs of
        // 150 x 214 at several offsets 4.8 ms, so 3.7)
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Warp-per-pair DP (the per-call drop-in and small batches).  One pair's
// strips are taken in turn by the lanes of a warp (lane g has strips g, g + 32,
// ...) and swept as a wavefront, two columns a step: at step t lane g, in pass
// p, evaluates columns j and j + 1, j = base + 2 * (t - g - p * R), receiving the
// strip above's bottom row (H, E packed as int16 halves) at both by warp
// shuffles, one step after lane g - 1 produced it.  R, the steps from a lane's
// strip to its next one, is 32 where every lane is done with a strip by then
// (a band: lane 31's row reaches lane 0 by the same shuffle); else it is larger
// and the row crosses passes through a row buffer.  Lane 0 then walks the
// traceback.
//
// A lone warp is bound by latency: a row's five dependent steps (22 cycles)
// times the rows and columns on the wavefront's path.  Two columns a step let
// their rows overlap (column j + 1 follows one row behind column j), windows
// are applied by selects (a branch a row ends the overlap), and a third pass of
// strips no longer waits for the second.  Measured against one column a step,
// a pass at a time: one extend_hint call of 150 x 214 111 -> 104 us, with its
// second attempt 197 -> 172; 1,000 mixed pairs in bands 0.38 -> 0.277 ms, 2,000
// 0.54 ms.  Strips of 2 or 4 rows (more lanes at work in a band) were slower:
// 122 and 257 us, since a step's shuffles, windows and vote cost as before.
// ---------------------------------------------------------------------------

// One column of a strip for the int16 domain's warp kernel; `act` has a bit
// per row whose window holds the column (MASK), as in dp_column otherwise.
template <bool MASK>
__device__ __forceinline__ uint32_t warp_column(Strip &S, const GotohConst &K, uint32_t sel,
                                                int cj, uint32_t act, int upHo, int upE, int diag,
                                                uint32_t &bottom) {
    uint32_t wa = 0, wb = 0;
    int kd = __viaddmax_s32(diag, prmt_sx(S.l0[0], S.l1[0], sel), 3);
    int Hp = 2;
#pragma unroll
    for (int r = 0; r < STRIP; r++) {
        int kE = __viaddmax_s32(upE, K.ex4, upHo);
        if (MASK && r > 0) kE = (act & (1u << (r - 1))) ? kE : K.oe4 + 2;
        const int kF = S.kF[r];
        upE = (int)and_or_u32((uint32_t)kE, ~3u, 1u);
        const int F4 = (int)and_u32((uint32_t)kF, ~3u);
        const int key = __vimax3_s32(kd, upE, F4);
        if (r < STRIP - 1)
            kd = __viaddmax_s32(S.Hl[r], prmt_sx(S.l0[r + 1], S.l1[r + 1], sel), 3);
        Hp = (int)and_or_u32((uint32_t)key, ~3u, 2u);
        wa = mad_u32(wa, 4u, (uint32_t)(key - Hp));
        wb = mad_u32(wb, 4u, xor_and_u32((uint32_t)kE, (uint32_t)kF, 3u));
        upHo = Hp + K.oe4;
        const int nF = __viaddmax_s32(F4, K.ex4, upHo);
        const int nr = max(S.rk[r], (int)mad_u32((uint32_t)Hp, 32768u, (uint32_t)cj));
        const bool in = !MASK || (act & (1u << r));
        S.Hl[r] = in ? Hp : S.Hl[r];
        S.kF[r] = in ? nF : S.kF[r];
        S.rk[r] = in ? nr : S.rk[r];
    }
    bottom = __byte_perm((uint32_t)Hp, (uint32_t)upE, 0x5410);
    return __byte_perm(wa + 0xAAAAu, wb, 0x5410);
}

// R of a pair, and its number of steps.
__device__ __forceinline__ int warp_shift(const Geo &g, int m, int nstrips, int lane, int &steps) {
    const int base = g.lo(1);
    int r = 0;
    for (int s = lane; s + 32 < nstrips; s += 32)
        r = max(r, ((g.hi(min((s + 1) * STRIP, m)) - base) >> 1) -
                       ((g.lo((s + 32) * STRIP + 1) - base) >> 1) + 1);
    r = __reduce_max_sync(0xffffffffu, r);
    const int R = r <= 32 ? 32 : max(r, 36);  // a buffered pass runs behind its writes
    const int l = nstrips - 1;
    steps = ((g.hi(m) - base) >> 1) + (l & 31) + (l >> 5) * R + 1;
    return R;
}

__device__ FillResult warp_fill(const GotohConst &K, const uint32_t *__restrict__ s_lut,
                                const PairSetup &P, uint32_t *tb, uint32_t *rb, int lane) {
    constexpr uint32_t ALL = 0xffffffffu;
    const int m = P.m, n = P.n;
    const Geo g = P.g;
    const uint32_t ABSENT = absent_HE(K);
    const int base = g.lo(1), nstrips = (m + STRIP - 1) / STRIP;
    int steps;
    const int R = warp_shift(g, m, nstrips, lane, steps);
    const bool ring = R == 32;
    int bHp = 2, bi = 0, bj = 0, trow = 0;  // of this lane's strips
    bool tleft = false, tclamp = false;
    Strip S;
    int s = lane - 32, j = 0, clo = 1 << 30, chi = -1, plo = 0, phi = -1, lo7 = 0;
    uint32_t pub0 = ABSENT, pub1 = ABSENT, last = ABSENT;
    uint2 u0 = make_uint2(ABSENT, ABSENT), u1 = u0;
    uint32_t cw = 0, cn = 0;
    bool turn = true, open = false;
    auto codes = [&](int c) {
        cw = load16(P.win.arena, P.win.pos + (uint64_t)(c - 1));
        cn = P.win.cnt ? nmask16(P.win.iv, P.win.cnt, c - 1) : 0u;
    };
    // bottom row of the pass before, from the row buffer
    auto above = [&](int c) { return c >= plo && c <= phi ? rb[c - plo] : ABSENT; };
    for (int t = 0;; t++) {
        if (turn) {
            if (open) {  // row bookkeeping in row order (extend.rs:795-827)
                const int i0 = s * STRIP + 1;
#pragma unroll
                for (int r = 0; r < STRIP; r++) {
                    const int i = i0 + r;
                    if (i <= m) {
                        const int rowHp = S.rk[r] >> 15, argj = 32767 - (S.rk[r] & 32767);
                        if (trow == 0) {
                            if (argj == g.lo(i)) {
                                trow = i;
                                tleft = true;
                                tclamp = argj <= 1;
                            } else if (g.hi(i) < n && S.Hl[r] == rowHp) {
                                trow = i;
                            }
                        }
                        if (rowHp > bHp) {
                            bHp = rowHp;
                            bi = i;
                            bj = argj;
                        }
                    }
                }
            }
            turn = false;
            s += 32;
            open = s < nstrips;
            clo = 1 << 30;
            chi = -1;
            if (open) {
                const int i0 = s * STRIP + 1;
                clo = g.lo(i0);
                chi = g.hi(min(i0 + STRIP - 1, m));
                plo = s ? g.lo(i0 - 1) : 0;
                phi = s ? g.hi(i0 - 1) : -1;
                lo7 = g.lo(i0 + STRIP - 1);
                j = base + 2 * (t - lane - (s >> 5) * R);
                const uint32_t rw = load16(P.read.arena, P.read.pos + (uint64_t)(i0 - 1));
                const uint32_t rn = P.read.cnt ? nmask16(P.read.iv, P.read.cnt, i0 - 1) : 0u;
#pragma unroll
                for (int r = 0; r < STRIP; r++) {
                    uint32_t c = (rw >> (30 - 2 * r)) & 3u;
                    if ((rn >> (31 - r)) & 1u) c = 4;
                    S.l0[r] = s_lut[2 * c];
                    S.l1[r] = s_lut[2 * c + 1];
                    S.Hl[r] = 2;
                    S.kF[r] = 2 + K.oe4;  // F opened from H = 0
                    S.rk[r] = -1;
                }
                codes(base + (clo - base & ~1));
            }
        }
        if (t >= steps) break;
        const bool active = j + 1 >= clo && j <= chi;
        uint32_t w0 = __shfl_sync(ALL, pub0, (lane - 1) & 31);
        uint32_t w1 = __shfl_sync(ALL, pub1, (lane - 1) & 31);
        if (!ring && lane == 0 && s >= 32 && active) {
            if (j <= clo) {  // the strip's first step
                last = above(j - 1);
                u0 = make_uint2(above(j), above(j + 1));
                u1 = make_uint2(above(j + 2), above(j + 3));
            }
            w0 = u0.x;
            w1 = u0.y;
            u0 = u1;
            u1 = make_uint2(above(j + 4), above(j + 5));
        }
        // the row above: its cell at j - 1, j (diagonals) and j, j + 1
        const uint32_t d0 = j - 1 >= plo && j - 1 <= phi ? last : ABSENT;
        const uint32_t d1 = j >= plo && j <= phi ? w0 : ABSENT;
        const uint32_t a0 = j <= phi ? w0 : ABSENT, a1 = j + 1 <= phi ? w1 : ABSENT;
        last = w1;
        // rows inside their windows: lo(r) <= j <= hi(r) (Geo), a run of rows
        auto rows_at = [&](int c) {
            const int x = c - g.off - s * STRIP - 1;
            const int rl = c >= n - g.half ? STRIP - 1 : min(STRIP - 1, x + g.half);
            const int rf = c <= g.half + 1 ? 0 : max(0, x - g.half);
            return c >= clo && c <= chi ? ((2u << rl) - (1u << rf)) & 0xffu : 0u;
        };
        const uint32_t act0 = rows_at(j), act1 = rows_at(j + 1);
        const uint32_t code0 = (cw >> 30) | ((cn >> 29) & 4u);
        const uint32_t code1 = ((cw >> 28) & 3u) | ((cn >> 28) & 4u);
        const uint32_t sel0 = code0 * 0x1111u + 0x8880u, sel1 = code1 * 0x1111u + 0x8880u;
        const int h0 = (int)(a0 & 0xffffu) + K.oe4, e0 = (int)a0 >> 16;
        const int h1 = (int)(a1 & 0xffffu) + K.oe4, e1 = (int)a1 >> 16;
        uint32_t word0, word1;
        // a lane without a strip may compute what it likes
        if (__all_sync(ALL, !open || (act0 & act1) == 0xffu)) {
            word0 = warp_column<false>(S, K, sel0, 32767 - j, 0xffu, h0, e0, (int)(d0 & 0xffffu),
                                         pub0);
            word1 = warp_column<false>(S, K, sel1, 32766 - j, 0xffu, h1, e1, (int)(d1 & 0xffffu),
                                         pub1);
        } else {
            word0 = warp_column<true>(S, K, sel0, 32767 - j, act0, h0, e0, (int)(d0 & 0xffffu),
                                        pub0);
            word1 = warp_column<true>(S, K, sel1, 32766 - j, act1, h1, e1, (int)(d1 & 0xffffu),
                                        pub1);
        }
        if (active) {
            uint32_t *w = tb + (size_t)s * P.sw;
            if (act0) w[j - clo] = word0;
            if (act1) w[j + 1 - clo] = word1;
            if (!ring && lane == 31 && s + 1 < nstrips) {  // a full strip: its last row
                if (act0 & 0x80u) rb[j - lo7] = pub0;
                if (act1 & 0x80u) rb[j + 1 - lo7] = pub1;
            }
            turn = j + 1 >= chi;
            cw <<= 4;
            cn <<= 2;
        }
        j += 2;
        // new codes for all lanes at once, 16 columns after the last or sooner
        if ((t & 7) == 7 && j > clo && j <= chi) codes(j);
        __syncwarp();
    }
    // merge the lanes in row order: the largest H, its first row; the first
    // touching row
    FillResult F;
    const uint32_t key = ((uint32_t)bHp << 16) | (0xffffu - (uint32_t)bi);
    const uint32_t top = __reduce_max_sync(ALL, key);
    const int wl = __ffs(__ballot_sync(ALL, key == top)) - 1;
    F.bestHp = __shfl_sync(ALL, bHp, wl);
    F.best_i = __shfl_sync(ALL, bi, wl);
    F.best_j = F.last_j = __shfl_sync(ALL, bj, wl);
    const uint32_t row = __reduce_min_sync(ALL, trow ? (uint32_t)trow : 0xffffffffu);
    const int tl = __ffs(__ballot_sync(ALL, (uint32_t)trow == row)) - 1;
    F.trow = row == 0xffffffffu ? 0 : (int)row;
    F.tleft = F.trow && __shfl_sync(ALL, (int)tleft, tl & 31) != 0;
    F.tclamp = F.trow && __shfl_sync(ALL, (int)tclamp, tl & 31) != 0;
    return F;
}

__global__ void __launch_bounds__(128) gotoh_warp_kernel(GotohJob job, GotohConst K) {
    __shared__ uint32_t s_lut[10];
    __shared__ int8_t s_lut25[32];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 10; k++) s_lut[k] = K.lut4[k >> 1][k & 1];
#pragma unroll
        for (int k = 0; k < 25; k++) s_lut25[k] = K.lut[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t warp_slot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    uint32_t *tb = job.tb + warp_slot * (job.tb_words + job.rb_words);
    uint32_t *rb = tb + job.tb_words;
    const uint64_t total = job.list_count ? (uint64_t)(*job.list_count) : job.n_pairs;
    for (uint64_t k = warp_slot; k < total; k += n_warps) {
        const uint32_t pi = job.list ? job.list[k] : (uint32_t)k;
        PairSetup S;
        if (!setup_pair(job, K, pi, job.tb_words, job.rb_words, lane == 0, S)) continue;
        FillResult F = warp_fill(K, s_lut, S, tb, rb, lane);
        __syncwarp();  // traceback words of every lane are visible to lane 0
        if (lane == 0) finish_pair(job, K, s_lut25, pi, S, F, StripTb<1>{tb, S.sw});
        __syncwarp();
    }
}

cudaError_t launch_gotoh_warp(const GotohJob &job, const GotohConst &k, int warps,
                              cudaStream_t st) {
    int grid = (warps + 3) / 4;
    gotoh_warp_kernel<<<grid, 128, 0, st>>>(job, k);
    return cudaGetLastError();
}

// Pairs outside the int16 domain: passes of 32 strips (lane s owns rows
// 8s+1..8s+8 of the pass) swept one column a step, H and E of a strip's bottom
// row crossing lanes and passes as two int32 words (the row buffer holds 2
// words per column); lanes outside their windows publish H = 0 and no E.
__device__ FillResult wide_fill(const GotohConst &K, const uint32_t *__restrict__ s_lut,
                                const PairSetup &P, uint32_t *tb, uint32_t *rb, int lane) {
    const int m = P.m, n = P.n, sw = P.sw;
    const Geo &g = P.g;
    FillResult R;
    R.bestHp = 2;
    R.best_i = R.best_j = R.last_j = 0;
    R.trow = 0;
    R.tleft = R.tclamp = false;
    const int nstrips = (m + STRIP - 1) / STRIP;
    for (int base = 0; base < nstrips; base += 32) {
        const int s = base + lane;
        const bool act = s < nstrips;
        const int i0 = s * STRIP + 1;
        const int nact = act ? min(STRIP, m - i0 + 1) : 0;
        StripT<true> S;
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            S.lo[r] = g.lo(i0 + r);
            S.hi[r] = g.hi(i0 + r);
            S.Hl[r] = 2;
            S.kF[r] = 2 + K.oe4;  // F opened from H = 0
            S.rk[r] = -1;
        }
        const int clo = S.lo[0];
        const int chi = act ? g.hi(i0 + nact - 1) : 0;
        const int lo7 = S.lo[STRIP - 1];
        if (act) {
            uint32_t rw = load16(P.read.arena, P.read.pos + (uint64_t)(i0 - 1));
            uint32_t rn = P.read.cnt ? nmask16(P.read.iv, P.read.cnt, i0 - 1) : 0u;
#pragma unroll
            for (int r = 0; r < STRIP; r++) {
                uint32_t c = (rw >> (30 - 2 * r)) & 3u;
                if ((rn >> (31 - r)) & 1u) c = 4;
                S.l0[r] = s_lut[2 * c];
                S.l1[r] = s_lut[2 * c + 1];
            }
        }
        // the previous pass's last strip left its bottom row in rb, columns
        // [plo, phi] of row 8*base
        const int plo = base ? g.lo(base * STRIP) : 0, phi = base ? g.hi(base * STRIP) : -1;
        int t0 = act ? clo + lane : 0x7fffffff, t1 = act ? chi + lane : -1;
        t0 = __reduce_min_sync(0xffffffffu, t0);
        t1 = __reduce_max_sync(0xffffffffu, t1);
        // bottom row published at the end of a step
        int pubH = 2, pubE = absent_E(K);
        int diag = 2;           // H of the row above at the previous column
        if (lane == 0 && base && clo - 1 >= plo && clo - 1 <= phi)
            diag = (int)rb[2 * (clo - 1 - plo)];
        uint32_t *tbs = tb + (size_t)s * sw;
        const bool handoff = lane == 31 && s + 1 < nstrips;
        int cw_at = -1000000;  // first window position of the cached code word
        uint32_t cw = 0, cn = 0;
        int nx_at = -1000000;  // the word after it, loaded one word ahead
        uint32_t nx = 0, nxn = 0;
        for (int t = t0; t <= t1; t++) {
            const int j = t - lane;
            int inH = __shfl_up_sync(0xffffffffu, pubH, 1);
            int inE = __shfl_up_sync(0xffffffffu, pubE, 1);
            if (lane == 0) {
                const bool have = base && j >= plo && j <= phi;
                inH = have ? (int)rb[2 * (j - plo)] : 2;
                inE = have ? (int)rb[2 * (j - plo) + 1] : absent_E(K);
            }
            int outH = 2, outE = absent_E(K);
            if (act && j >= clo && j <= chi) {
                // window codes 16 at a time, each word loaded while the
                // one before is in use: a load that a lane waits for stalls
                // the whole wavefront, and the lanes reach their word
                // boundaries at different steps
                if (j - 1 >= cw_at + 16) {
                    if (j - 1 == nx_at) {
                        cw = nx;
                        cn = nxn;
                    } else {
                        cw = load16(P.win.arena, P.win.pos + (uint64_t)(j - 1));
                        cn = P.win.cnt ? nmask16(P.win.iv, P.win.cnt, j - 1) : 0u;
                    }
                    cw_at = j - 1;
                    nx_at = cw_at + 16;
                    if (nx_at < n) {
                        nx = load16(P.win.arena, P.win.pos + (uint64_t)nx_at);
                        nxn = P.win.cnt ? nmask16(P.win.iv, P.win.cnt, nx_at) : 0u;
                    }
                }
                const int sh = j - 1 - cw_at;
                uint32_t code = ((cn >> (31 - sh)) & 1u) ? 4u : ((cw >> (30 - 2 * sh)) & 3u);
                uint32_t sel = code * 0x1111u + 0x8880u;
                int upH = inH, upE = inE;
                uint32_t word = dp_column<1, true>(S, K, j, sel, 32767u - (uint32_t)j, upH, upE,
                                                   diag);
                tbs[j - clo] = word;
                outH = upH;
                outE = upE;
                if (handoff && j >= lo7) {
                    rb[2 * (j - lo7)] = (uint32_t)upH;
                    rb[2 * (j - lo7) + 1] = (uint32_t)upE;
                }
            }
            diag = inH;
            pubH = outH;
            pubE = outE;
        }
        __syncwarp();
        // this lane's rows, in row order (extend.rs:795-827)
        int bHp = -1, bi = 0, bj = 0, trow = 0;
        bool tleft = false, tclamp = false;
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            if (r < nact) {
                int rowHp = (int)(S.rk[r] >> 15);
                int argj = 32767 - (int)(S.rk[r] & 32767);
                if (trow == 0) {
                    if (argj == S.lo[r]) {
                        trow = i0 + r;
                        tleft = true;
                        tclamp = S.lo[r] <= 1;
                    } else if (S.hi[r] < n && S.Hl[r] == rowHp) {
                        trow = i0 + r;
                        tleft = false;
                        tclamp = S.hi[r] >= n;
                    }
                }
                if (rowHp > bHp) {
                    bHp = rowHp;
                    bi = i0 + r;
                    bj = argj;
                }
            }
        }
        // merge lanes in row order: the first strictly larger maximum wins,
        // the first touching row wins
        const int mx = __reduce_max_sync(0xffffffffu, bHp);
        const int wl = __ffs(__ballot_sync(0xffffffffu, bHp == mx)) - 1;
        const int wi = __shfl_sync(0xffffffffu, bi, wl), wj = __shfl_sync(0xffffffffu, bj, wl);
        if (mx > R.bestHp) {
            R.bestHp = mx;
            R.best_i = wi;
            R.best_j = R.last_j = wj;
        }
        const uint32_t tm = __ballot_sync(0xffffffffu, trow != 0);
        if (R.trow == 0 && tm) {
            const int tl = __ffs(tm) - 1;
            R.trow = __shfl_sync(0xffffffffu, trow, tl);
            R.tleft = __shfl_sync(0xffffffffu, (int)tleft, tl) != 0;
            R.tclamp = __shfl_sync(0xffffffffu, (int)tclamp, tl) != 0;
        }
    }
    return R;
}

// Pairs outside the int16 domain (reads longer than GotohConst::max_m), one
// warp per pair with int32 H / E / F and 64-bit row-max keys, otherwise the
// warp-per-pair fill and the same traceback: the same cells, words, maxima,
// touches and CIGARs as the reference's i32 flavour of run_band
// (extend.rs:462-528).  In hint mode the warp runs extend_hint's second
// attempt itself when the first escalates (extend.rs:421-426).
__global__ void __launch_bounds__(128) gotoh_wide_kernel(GotohJob job, GotohConst K) {
    __shared__ uint32_t s_lut[10];
    __shared__ int8_t s_lut25[32];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 10; k++) s_lut[k] = K.lut4[k >> 1][k & 1];
#pragma unroll
        for (int k = 0; k < 25; k++) s_lut25[k] = K.lut[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t warp_slot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    uint32_t *tb = job.tb + warp_slot * (job.tb_words + 2 * job.rb_words);
    uint32_t *rb = tb + job.tb_words;
    const uint64_t total = *job.list_count;
    for (uint64_t k = warp_slot; k < total; k += n_warps) {
        const uint32_t pi = job.list[k];
        PairSetup S;
        if (!setup_pair(job, K, pi, job.tb_words, job.rb_words, lane == 0, S)) continue;
        FillResult F = wide_fill(K, s_lut, S, tb, rb, lane);
        __syncwarp();
        int esc = 0;
        if (lane == 0) esc = finish_pair(job, K, s_lut25, pi, S, F, StripTb<1>{tb, S.sw}, false) ? 1 : 0;
        esc = __shfl_sync(0xffffffffu, esc, 0);
        __syncwarp();
        if (!esc) continue;
        GotohJob j2 = job;
        j2.mode = 2;
        if (!setup_pair(j2, K, pi, job.tb_words, job.rb_words, lane == 0, S)) continue;
        F = wide_fill(K, s_lut, S, tb, rb, lane);
        __syncwarp();
        if (lane == 0) finish_pair(j2, K, s_lut25, pi, S, F, StripTb<1>{tb, S.sw}, false);
        __syncwarp();
    }
}

cudaError_t launch_gotoh_wide(const GotohJob &job, const GotohConst &k, int warps,
                              cudaStream_t st) {
    GotohJob j = job;
    j.wide = 1;
    int grid = (warps + 3) / 4;
    gotoh_wide_kernel<<<grid, 128, 0, st>>>(j, k);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Two pairs per thread in 16x2 SIMD lanes.  Two pairs with identical band
// geometry and N-free windows share one thread: every register holds the
// scaled key of pair A in its low half and of pair B in its high half, and
// the half-word operations (add-max, 3-way max) evaluate both cells at once
// with the arithmetic above.  Keys carry a bias of BIAS2 a half, so that all
// of them are positive and a plain 32-bit add or subtract of two packed
// constants never carries across the halves (those adds may issue off the
// saturated ALU pipe): H <= 8191 by the score-range rule and gap costs <=
// 2,000 a side give keys in [384, 49,152] of an unsigned half.
// Substitution scores of both cells come from one PRMT over the two rows'
// LUT words.  Traceback words, row maxima and touches of each pair are
// exactly those of the thread-per-pair kernel, and each pair's traceback is
// walked by the same code (pair A's and B's words side by side, stride 64).
//
// A row's maximum is one max of keys H*S + (S - 1 - t), where t numbers the
// strip's columns (in blocks of 2^g columns where S of them do not reach):
// equal H keeps the first column, as the scalar kernel's strict > does, and
// the column comes with the maximum.  S, a multiple of 4, is as large as the
// read's highest score allows in 16 bits (H <= m * match: S = 216 for a
// 150-base read), and the key is one multiply-add of Hp, off the ALU pipe;
// keeping the column beside the maximum took three more ALU instructions.
// Where g > 0 the walk picks the block's column (FillResult::last_j).
//
// Strip shapes: where a strip's row windows move right by one column a row
// (a band away from the matrix edge) its two corners are unrolled as
// triangles, 28 and 36 cells with no test; where they stand still (the whole
// matrix, a band clamped at column 1 or n) that side has no corner at all;
// a strip in which clamping begins or ends tests every cell.  A band of 33
// columns so computes 272 cells a strip instead of 320, half of them masked.
//
// Bound by the ALU pipe (78 % busy in the fill, 13.5 ALU of 23.5 issued
// instructions a row of two cells; 28.9 ALU before these keys and corners).
// 4,194,304 mixed pairs: 43.9 -> 33.4 ms (38.0 without the two-column interior,
// its read-ahead and the one-pass walk).
// ---------------------------------------------------------------------------

constexpr uint32_t BIAS2 = 0x40004000u;
constexpr uint32_t KEEP2 = 0xFFFCFFFCu;
constexpr int PAIR_BLOCK = 128;  // threads of a paired block (stride of the shared first-cell keys)

struct Strip2 {
    uint32_t Hl[STRIP], kF[STRIP], rmax[STRIP];
    uint32_t la[STRIP], lb[STRIP];
};

struct Keys2 {
    uint32_t oe;     // 4*(gap_open + gap_ext) in both halves (subtracted)
    uint32_t ex;     // 4*ext in both halves (as 16-bit adds)
    uint32_t h0;     // H = 0
    uint32_t ho0;    // a gap opened from H = 0
    uint32_t e0;     // the E an out-of-window cell shows
    uint32_t ks;     // S / 4
    uint32_t ck0;    // row-max key of Hp at the strip's first column: Hp * ks + ck0
    int g;           // columns of a row-max key: blocks of 2^g
    uint32_t miss;   // 4 * (score against N) in both halves
};

__device__ __forceinline__ Keys2 keys2_of(const GotohConst &K, int m, int sw) {
    Keys2 c;
    c.oe = (uint32_t)(-K.oe4) * 0x10001u;
    c.ex = (uint32_t)(K.ex4 & 0xffff) * 0x10001u;
    c.h0 = BIAS2 + 0x00020002u;
    c.ho0 = c.h0 - c.oe;
    c.e0 = c.ho0 - 0x00010001u;
    c.ks = 16384u / (uint32_t)(m * K.smax + 1);
    c.ck0 = (4u * c.ks - 1u) * 0x10001u - c.h0 * c.ks;
    c.miss = (uint32_t)(4 * K.lut[4] & 0xffff) * 0x10001u;
    c.g = 0;
    while ((uint32_t)(sw - 1) >> c.g >= 4u * c.ks) c.g++;
    return c;
}

__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}

// One column as the rows see it.
struct Col2 {
    uint32_t sel;  // PRMT selector of both windows' codes
    uint32_t ck;   // row-max key of Hp: Hp * ks + ck
    uint32_t nkeep, nfill;  // N in a window: its half's score is nfill's
};

template <bool HASN>
__device__ __forceinline__ uint32_t sub2(uint32_t la, uint32_t lb, const Col2 &col) {
    const uint32_t x = prmt(la, lb, col.sel);
    return HASN ? and_or_u32(x, col.nkeep, col.nfill) : x;
}

// Rows R0..R1 of one column, top to bottom.  Enters with the row above R0:
// its Ho and E at this column and its Hp at the previous one (d); leaves with
// row R1's Ho and E.  Returns the column's traceback words (pair A, pair B).
template <int R0, int R1, bool HASN>
__device__ __forceinline__ uint2 dp_rows2(Strip2 &S, const Keys2 &c, const Col2 &col,
                                          uint32_t &upHo, uint32_t &upE, uint32_t d) {
    uint32_t wa = 0, wb = 0;
    uint32_t kd = __viaddmax_u16x2(d, sub2<HASN>(S.la[R0], S.lb[R0], col), BIAS2 + 0x00030003u);
#pragma unroll
    for (int r = R0; r <= R1; r++) {
        const uint32_t kE = __viaddmax_u16x2(upE, c.ex, upHo), kF = S.kF[r];
        upE = and_or_u32(kE, KEEP2, 0x00010001u);
        const uint32_t F4 = and_u32(kF, KEEP2);
        const uint32_t key = __vimax3_u16x2(kd, upE, F4);
        if (r < R1)  // the next row's diagonal, before this row's H is replaced
            kd = __viaddmax_u16x2(S.Hl[r], sub2<HASN>(S.la[r + 1], S.lb[r + 1], col),
                                  BIAS2 + 0x00030003u);
        const uint32_t Hp = and_or_u32(key, KEEP2, 0x00020002u);
        S.Hl[r] = Hp;
        wa = mad_u32(wa, 4u, key - Hp);
        wb = mad_u32(wb, 4u, xor_and_u32(kE, kF, 0x00030003u));
        upHo = Hp - c.oe;
        S.kF[r] = __viaddmax_u16x2(F4, c.ex, upHo);
        S.rmax[r] = __vmaxu2(S.rmax[r], mad_u32(Hp, c.ks, col.ck));
    }
    constexpr int SH = 2 * (STRIP - 1 - R1);
    wa += 0xAAAAAAAAu & ((0x10001u << (2 * (R1 - R0 + 1))) - 0x10001u);  // tags, not tag - 2
    wa <<= SH;
    wb <<= SH;
    return make_uint2(__byte_perm(wa, wb, 0x5410), __byte_perm(wa, wb, 0x7632));
}

// The same over all 8 rows with every cell tested against its row window
// (clamping strips): as dp_column's MASK.  hf: the rows' first-cell keys
// (stride PAIR_BLOCK).  Leaves the last row's Hp in botH.
template <bool HASN>
__device__ __forceinline__ uint2 dp_masked2(Strip2 &S, const Keys2 &c, const Geo &g, int i0, int j,
                                            const Col2 &col, uint32_t upHo, uint32_t &upE, uint32_t d,
                                            uint32_t &botH, uint32_t *hf) {
    uint32_t wa = 0, wb = 0;
#pragma unroll
    for (int r = 0; r < STRIP; r++) {
        const uint32_t left = S.Hl[r], kF = S.kF[r];
        const uint32_t kE = __viaddmax_u16x2(upE, c.ex, upHo);
        const uint32_t E1 = and_or_u32(kE, KEEP2, 0x00010001u);
        const uint32_t F4 = and_u32(kF, KEEP2);
        const uint32_t kd = __viaddmax_u16x2(d, sub2<HASN>(S.la[r], S.lb[r], col), BIAS2 + 0x00030003u);
        const uint32_t key = __vimax3_u16x2(kd, E1, F4);
        const uint32_t Hp = and_or_u32(key, KEEP2, 0x00020002u);
        wa = mad_u32(wa, 4u, key - Hp + 0x00020002u);
        wb = mad_u32(wb, 4u, xor_and_u32(kE, kF, 0x00030003u));
        const int lo = g.lo(i0 + r);
        const bool in = (j >= lo) & (j <= g.hi(i0 + r));
        if (in) {
            S.kF[r] = __viaddmax_u16x2(F4, c.ex, Hp - c.oe);
            S.rmax[r] = __vmaxu2(S.rmax[r], mad_u32(Hp, c.ks, col.ck));
            S.Hl[r] = Hp;
        }
        if (j == lo) hf[r * PAIR_BLOCK] = S.rmax[r];
        upHo = in ? Hp - c.oe : c.ho0;
        upE = in ? E1 : c.e0;
        d = left;
    }
    botH = upHo + c.oe;
    return make_uint2(__byte_perm(wa, wb, 0x5410), __byte_perm(wa, wb, 0x7632));
}

// The codes of both windows from column j on, 16 columns at a time.
template <bool HASN>
struct Codes2 {
    const Seq &wa, &wb;
    uint32_t a, b, na, nb;
    int t;  // columns taken so far in this strip
    __device__ __forceinline__ void load(int j) {
        a = load16(wa.arena, wa.pos + (uint64_t)(j - 1));
        b = load16(wa.arena, wb.pos + (uint64_t)(j - 1));  // one arena
        if (HASN) {
            na = wa.cnt ? nmask16(wa.iv, wa.cnt, j - 1) : 0u;
            nb = wb.cnt ? nmask16(wb.iv, wb.cnt, j - 1) : 0u;
        }
    }
    __device__ __forceinline__ Col2 here(const Keys2 &c) const {
        Col2 col;
        col.sel = (a >> 30) * 0x11u + (b >> 30) * 0x1100u + 0xC480u;
        col.ck = c.ck0 - (uint32_t)(t >> c.g) * 0x10001u;
        if (HASN) {
            col.nkeep = (na >> 31 ? 0u : 0xffffu) | (nb >> 31 ? 0u : 0xffff0000u);
            col.nfill = c.miss & ~col.nkeep;
        }
        return col;
    }
    // ... and on to the next column (whose row-max keys are 1 lower every 2^g
    // columns)
    __device__ __forceinline__ void step() {
        a <<= 2;
        b <<= 2;
        t++;
        if (HASN) {
            na <<= 1;
            nb <<= 1;
        }
    }
    __device__ __forceinline__ Col2 next(const Keys2 &c) {
        const Col2 col = here(c);
        step();
        return col;
    }
};

// The words of the row above at the next AHEAD columns, read ahead of their
// use: a column's arithmetic is ~200 cycles of dependent steps, an L2 round
// trip several times that when few warps share the scheduler.  A slot is
// rewritten only at or after the column that reads it.
constexpr int AHEAD = 4;
struct Above2 {
    uint2 q[AHEAD];
    const uint2 *p;  // the row above at the next column
    int left;        // columns of it from there on
    __device__ __forceinline__ uint2 at(int k, uint2 absent) const {
        return k < left ? p[k * 32] : absent;
    }
    __device__ __forceinline__ void start(const uint2 *p_, int left_, uint2 absent) {
        p = p_;
        left = left_;
#pragma unroll
        for (int k = 0; k < AHEAD; k++) q[k] = at(k, absent);
    }
    __device__ __forceinline__ uint2 next(uint2 absent) {
        const uint2 up = q[0];
#pragma unroll
        for (int k = 0; k + 1 < AHEAD; k++) q[k] = q[k + 1];
        q[AHEAD - 1] = at(AHEAD, absent);
        p += 32;
        left--;
        return up;
    }
};

// Columns clo + K of a sloped strip's left corner: rows 0..K.
template <int K, bool HASN>
__device__ __forceinline__ void head2(Strip2 &S, const Keys2 &c, Codes2<HASN> &w, Above2 &ab,
                                      uint2 absent, uint32_t &diag, uint2 *&tb, uint32_t *hf) {
    if constexpr (K < STRIP - 1) {
        const uint2 up = ab.next(absent);
        uint32_t upHo = up.x - c.oe, upE = up.y;
        __stcs(tb, dp_rows2<0, K, HASN>(S, c, w.next(c), upHo, upE, diag));
        hf[K * PAIR_BLOCK] = S.rmax[K];
        diag = up.x;
        tb += 32;
        head2<K + 1, HASN>(S, c, w, ab, absent, diag, tb, hf);
    }
}

// Columns hi0 + K of a sloped strip's right corner: rows K..7, the row above
// out of its window; up to column hi0 + last.
template <int K, bool HASN>
__device__ __forceinline__ void tail2(Strip2 &S, const Keys2 &c, Codes2<HASN> &w, int last, uint32_t &diag,
                                      uint2 *&rbw, uint2 *&tb) {
    if constexpr (K < STRIP) {
        if (K <= last) {
            uint32_t upHo = c.ho0, upE = c.e0;
            __stcs(tb, dp_rows2<K, STRIP - 1, HASN>(S, c, w.next(c), upHo, upE, diag));
            diag = S.Hl[K];  // row K's last cell: the next column's diagonal
            *rbw = make_uint2(upHo + c.oe, upE);
            rbw += 32;
            tb += 32;
            tail2<K + 1, HASN>(S, c, w, last, diag, rbw, tb);
        }
    }
}

// The best cells so far of both pairs: H (thr: the largest row-max key of
// that H), row, and the columns that hold the row's first cell of that H.
struct Best2 {
    uint32_t thr;
    int h[2], i[2], j0[2], j1[2];
};

// Fill the DP of two pairs with identical geometry (A's).  tb0, rb: the
// lane's traceback words and row buffer, 32 word pairs apart; hf: the keys of
// the strip's 8 first cells in shared memory (stride PAIR_BLOCK).
template <bool HASN>
__device__ void dp_fill2(const GotohConst &K, const uint32_t *__restrict__ s_lut,
                         const PairSetup &A, const PairSetup &B2, uint2 *tb0, uint2 *rb,
                         uint32_t *hf, FillResult &FA, FillResult &FB) {
    const int m = A.m, n = A.n, sw = A.sw;
    const Geo g = A.g;
    const Seq readA = A.read, readB = B2.read;
    const Keys2 c = keys2_of(K, m, sw);
    const uint32_t ksc = 4u * c.ks;                  // S
    const uint32_t inv_s = 0xffffffffu / ksc + 1u;  // key / S = mulhi(key, inv_s): key < 2^16, S <= 2^16
    Best2 B;
    B.thr = (ksc - 1u) * 0x10001u;
#pragma unroll
    for (int q = 0; q < 2; q++) B.h[q] = B.i[q] = B.j0[q] = B.j1[q] = 0;
    // the first touching row of each pair with its left / clamped flags, and
    // bit 15 of each half of open_halves while that pair has none
    uint32_t trow2 = 0u, tflags = 0u;  // touch rows (halves); left / clamped bits 0-1 (A), 2-3 (B)
    uint32_t open_halves = 0x80008000u;
    Strip2 S;
    const int nstrips = (m + STRIP - 1) / STRIP;
    int plo = g.lo(1), phi = g.hi(min(STRIP, m));
    for (int k = 0; k <= phi - plo; k++) rb[(size_t)k * 32] = make_uint2(c.h0, c.e0);
    for (int s = 0; s < nstrips; s++) {
        const int i0 = s * STRIP + 1;
        const int nact = min(STRIP, m - i0 + 1);
        const uint32_t rwA = load16(readA.arena, readA.pos + (uint64_t)(i0 - 1));
        const uint32_t rwB = load16(readA.arena, readB.pos + (uint64_t)(i0 - 1));  // one arena
        const uint32_t rnA = readA.cnt ? nmask16(readA.iv, readA.cnt, i0 - 1) : 0u;
        const uint32_t rnB = readB.cnt ? nmask16(readB.iv, readB.cnt, i0 - 1) : 0u;
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            S.Hl[r] = c.h0;
            S.kF[r] = c.ho0;
            S.rmax[r] = 0u;
            uint32_t ca = (rwA >> (30 - 2 * r)) & 3u, cb = (rwB >> (30 - 2 * r)) & 3u;
            if ((rnA >> (31 - r)) & 1u) ca = 4;
            if ((rnB >> (31 - r)) & 1u) cb = 4;
            S.la[r] = s_lut[2 * ca];
            S.lb[r] = s_lut[2 * cb];
        }
        const int clo = g.lo(i0), lo7 = g.lo(i0 + STRIP - 1);
        const int hi0 = g.hi(i0), chi = g.hi(i0 + nact - 1);
        // windows move by 0 or 1 columns a row, so the ends tell the shape
        const bool lslope = lo7 == clo + STRIP - 1 && hi0 >= lo7, lflat = lo7 == clo;
        const bool rslope = chi == hi0 + nact - 1, rflat = chi == hi0;
        uint32_t diag = c.h0;
        if (clo - 1 >= plo && clo - 1 <= phi) diag = rb[(size_t)(clo - 1 - plo) * 32].x;
        uint2 *tb = tb0 + (size_t)s * sw * 32;
        const uint2 *rbr = rb + (size_t)(clo - plo) * 32;  // the row above at the next column
        uint2 *rbw = rb;                                   // the last row from column lo7 on
        Codes2<HASN> w{A.win, B2.win};
        w.t = 0;
        if ((lslope | lflat) & (rslope | rflat)) {
            int jb = clo;  // first column with all 8 rows
            const uint2 absent = make_uint2(c.h0, c.e0);
            Above2 ab;
            ab.start(rbr, phi - clo + 1, absent);
            w.load(clo);
            if (lslope) {
                head2<0, HASN>(S, c, w, ab, absent, diag, tb, hf);
                jb = lo7;
            }
            // interior: all 8 rows in their windows, up to the first row's
            // last column, where the row above is out of its window if that
            // moved.  Two columns a turn: more of them, or a copy of the
            // column for the odd one, do not fit the instruction cache
            // beside the corners and the finish (four: no-instruction stalls
            // 0.1 -> 3.1 an issue, 5.7 -> 6.8 ms for 1,048,576 pairs).
            bool begins = true;  // rows begin in the next column
            for (int j = jb; j <= hi0;) {
                w.load(j);
                const int stop = min(j + 16, hi0 + 1);
#pragma unroll 1
                while (j < stop) {
                    const uint2 n0 = ab.at(AHEAD, absent), n1 = ab.at(AHEAD + 1, absent);
                    uint32_t upHo = ab.q[0].x - c.oe, upE = ab.q[0].y;
                    __stcs(tb, dp_rows2<0, STRIP - 1, HASN>(S, c, w.next(c), upHo, upE, diag));
                    *rbw = make_uint2(upHo + c.oe, upE);
                    diag = ab.q[0].x;
                    if (begins) {  // their first cells
#pragma unroll
                        for (int r = 0; r < STRIP; r++)
                            if (lflat | (r == STRIP - 1)) hf[r * PAIR_BLOCK] = S.rmax[r];
                        begins = false;
                    }
                    if (++j < stop) {
                        upHo = ab.q[1].x - c.oe;
                        upE = ab.q[1].y;
                        __stcs(tb + 32,
                               dp_rows2<0, STRIP - 1, HASN>(S, c, w.next(c), upHo, upE, diag));
                        rbw[32] = make_uint2(upHo + c.oe, upE);
                        diag = ab.q[1].x;
                        j++;
                        rbw += 32;
                        tb += 32;
                    }
                    ab.q[0] = ab.q[2];
                    ab.q[1] = ab.q[3];
                    ab.q[2] = n0;
                    ab.q[3] = n1;
                    ab.p += 64;
                    ab.left -= 2;
                    rbw += 32;
                    tb += 32;
                }
            }
            if (rslope && nact > 1) {
                w.load(hi0 + 1);
                diag = S.Hl[0];
                tail2<1, HASN>(S, c, w, nact - 1, diag, rbw, tb);
            }
        } else {
            // clamping begins or ends inside the strip
            for (int j = clo; j <= chi;) {
                w.load(j);
                const int cnt = min(16, chi - j + 1);
#pragma unroll 1
                for (int k = 0; k < cnt; k++, j++) {
                    const uint2 up = j <= phi ? *rbr : make_uint2(c.h0, c.e0);
                    uint32_t upE = up.y, botH;
                    __stcs(tb, dp_masked2<HASN>(S, c, g, i0, j, w.next(c), up.x - c.oe, upE, diag, botH,
                                                 hf));
                    diag = up.x;
                    if (j >= lo7) {
                        *rbw = make_uint2(botH, upE);
                        rbw += 32;
                    }
                    rbr += 32;
                    tb += 32;
                }
            }
        }
        // row bookkeeping (extend.rs:795-827); rows past the read do not count
        if (nact < STRIP) {
#pragma unroll
            for (int r = 1; r < STRIP; r++)
                if (r >= nact) S.rmax[r] = 0u;
        }
        // the best cell: a strictly larger row maximum, in row order, replaces it
        uint32_t smax = __vimax3_u16x2(S.rmax[0], S.rmax[1], S.rmax[2]);
        smax = __vimax3_u16x2(smax, S.rmax[3], S.rmax[4]);
        smax = __vimax3_u16x2(smax, S.rmax[5], __vmaxu2(S.rmax[6], S.rmax[7]));
        if (__vmaxu2(B.thr, smax) != B.thr) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const uint32_t v = (smax >> (16 * q)) & 0xffffu;
                if (v > ((B.thr >> (16 * q)) & 0xffffu)) {
                    const uint32_t h = __umulhi(v, inv_s), base = h * ksc;
                    int row = 0;
                    uint32_t key = 0;
#pragma unroll
                    for (int r = STRIP - 1; r >= 0; r--) {
                        const uint32_t x = (S.rmax[r] >> (16 * q)) & 0xffffu;
                        if (x >= base) {
                            row = i0 + r;
                            key = x;
                        }
                    }
                    const int j0 = clo + (int)((base + ksc - 1u - key) << c.g);
                    B.h[q] = (int)h;
                    B.i[q] = row;
                    B.j0[q] = max(j0, g.lo(row));
                    B.j1[q] = min(j0 + (1 << c.g) - 1, g.hi(row));
                    B.thr = (B.thr & (0xffff0000u >> (16 * q))) | ((base + ksc - 1u) << (16 * q));
                }
            }
        }
        // the first touching row, per pair, until both pairs have one: the
        // row's maximum is its first cell's key (left edge) or, when hi < n,
        // no larger than a key of its last cell's H (right edge).  (x - 0x10001) & ~x has bit 15 of a half
        // set for every zero half (and may set it in the half above one), so
        // a strip whose rows have none for a pair still without a touch skips
        // the exact per-row tests
        uint32_t zero_halves = 0u;
        if (open_halves) {
#pragma unroll
            for (int r = 0; r < STRIP; r++) {
                if (r < nact) {
                    const uint32_t zl = S.rmax[r] ^ hf[r * PAIR_BLOCK];
                    zero_halves |= (zl - 0x00010001u) & ~zl;
                    if (g.hi(i0 + r) < n) {
                        const uint32_t u = mad_u32(S.Hl[r], c.ks, c.ck0);
                        const uint32_t zr = __vmaxu2(S.rmax[r], u) ^ u;
                        zero_halves |= (zr - 0x00010001u) & ~zr;
                    }
                }
            }
        }
        if (zero_halves & open_halves) {
#pragma unroll
            for (int r = 0; r < STRIP; r++) {
                if (r < nact) {
                    const int lo = g.lo(i0 + r), hi = g.hi(i0 + r);
                    const uint32_t first = hf[r * PAIR_BLOCK];
                    const uint32_t last = mad_u32(S.Hl[r], c.ks, c.ck0);
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const uint32_t bit = 0x8000u << (16 * q);
                        if (open_halves & bit) {
                            const bool tl = (((S.rmax[r] ^ first) >> (16 * q)) & 0xffffu) == 0;
                            const bool tr = ((S.rmax[r] >> (16 * q)) & 0xffffu) <= ((last >> (16 * q)) & 0xffffu);
                            if (tl) {
                                trow2 |= (uint32_t)(i0 + r) << (16 * q);
                                tflags |= (1u | (lo <= 1 ? 2u : 0u)) << (2 * q);
                                open_halves &= ~bit;
                            } else if (hi < n && tr) {
                                trow2 |= (uint32_t)(i0 + r) << (16 * q);
                                open_halves &= ~bit;
                            }
                        }
                    }
                }
            }
        }
        plo = lo7;
        phi = g.hi(i0 + STRIP - 1);
    }
    auto put = [&](FillResult &F, int q) {
        F.bestHp = 4 * B.h[q] + 2;
        F.best_i = B.i[q];
        F.best_j = B.j0[q];
        F.last_j = B.j1[q];
        F.trow = (int)((trow2 >> (16 * q)) & 0xffffu);
        F.tleft = (tflags >> (2 * q)) & 1u;
        F.tclamp = (tflags >> (2 * q + 1)) & 1u;
    };
    put(FA, 0);
    put(FB, 1);
}

// Out-of-line fill, set-up and finish of the paired kernel: one copy of each in
// the kernel's code (the instruction cache holds the fill and little more),
// and their registers are not reserved across one another.
template <bool HASN>
__device__ __noinline__ void fill2_call(const GotohConst &K, const uint32_t *__restrict__ s_lut,
                                        const PairSetup &A, const PairSetup &B, uint32_t *tb,
                                        uint32_t *rb, uint32_t *hf, FillResult &FA, FillResult &FB) {
    dp_fill2<HASN>(K, s_lut, A, B, reinterpret_cast<uint2 *>(tb), reinterpret_cast<uint2 *>(rb), hf,
                   FA, FB);
}

__device__ __noinline__ void finish_call(const GotohJob &job, const GotohConst &K,
                                         const int8_t *__restrict__ lut, uint32_t pi,
                                         PairSetup &S, const FillResult &F, const uint32_t *tb) {
    finish_pair(job, K, lut, pi, S, F, StripTb<64>{tb, S.sw});
}

__device__ __noinline__ bool setup_call(const GotohJob &job, const GotohConst &K, uint32_t pi,
                                        bool write, PairSetup &S) {
    return setup_pair(job, K, pi, job.tb_words, job.rb_words, write, S);
}

// Work item (p[0], p[1]) of every lane (NO_PAIR: none): both pairs in one
// fill when their geometry matches; a pair without a partner of its geometry
// fills both halves, in the same pass over the lanes (lanes that took turns
// doubled a warp's time), and a second pass takes the other pair of a
// mismatched item.  N in a window costs one more instruction a row; a batch
// that has a window with N runs that fill for all its pairs, as the two fills do
// not fit the instruction cache together (1,000,003 mixed pairs, N in 0.5 % of
// the windows: 12.3 ms with the fill chosen per warp, 9.9 so; N in reads alone, which
// a row's score word takes care of, 7.8).  The descriptors are resolved again for
// the finish rather than kept live across the fill.
constexpr uint32_t NO_PAIR = 0xffffffffu;

template <bool MAYN>
__device__ void process_item2(const GotohJob &job, const GotohConst &K,
                              const uint32_t *__restrict__ s_lut, const int8_t *__restrict__ lut,
                              const uint32_t (&p)[2], uint32_t *tb, uint32_t *rb, uint32_t *hf) {
    int todo = 0;  // bit q: pair q has a DP
    bool together = false;
    for (int pass = 0; pass < 2; pass++) {
        FillResult F[2];
        int now = 0;  // pairs of this pass
        {
            PairSetup A, B;
            if (pass == 0) {
                const bool a = p[0] != NO_PAIR && setup_call(job, K, p[0], true, A);
                const bool b = p[1] != NO_PAIR && setup_call(job, K, p[1], true, B);
                todo = (a ? 1 : 0) | (b ? 2 : 0);
                together = todo == 3 && A.m == B.m && A.n == B.n && A.full == B.full &&
                           A.g.off == B.g.off && A.g.half == B.g.half;
                now = together ? 3 : (todo == 3 ? 1 : todo);
                if (now == 1) B = A;
                if (now == 2) A = B;
            } else {
                now = todo == 3 && !together ? 2 : 0;
                if (!__any_sync(0xffffffffu, now != 0)) break;
                if (now) {
                    setup_call(job, K, p[1], false, A);
                    B = A;
                }
            }
            if (now) {
                if (MAYN && windows_n(job)) fill2_call<true>(K, s_lut, A, B, tb, rb, hf, F[0], F[1]);
                else fill2_call<false>(K, s_lut, A, B, tb, rb, hf, F[0], F[1]);
            }
        }
#pragma unroll 1
        for (int q = 0; q < 2; q++) {
            if (now >> q & 1) {
                PairSetup S;
                setup_call(job, K, p[q], false, S);
                finish_call(job, K, lut, p[q], S, F[q], tb + q);
            }
        }
    }
}

// Work items of two list entries each, positions b0 + 2k and b0 + 2k + 1 below
// b1; neighbours in the binned list share their geometry key.
template <bool MAYN>
__device__ __forceinline__ void paired_section(const GotohJob &job, const GotohConst &K,
                                               const uint32_t *__restrict__ s_lut,
                                               const int8_t *__restrict__ lut, uint64_t b0,
                                               uint64_t b1, uint32_t *tb, uint32_t *rb, int lane,
                                               uint32_t *hf) {
    const uint64_t total = (b1 - b0 + 1) / 2;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd((unsigned long long *)job.queue, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= total) break;
        const uint64_t k = base + lane;
        uint32_t p[2] = {NO_PAIR, NO_PAIR};
        if (k < total) {
            const uint64_t x = b0 + 2 * k, y = x + 1;
            p[0] = job.list ? job.list[x] : (uint32_t)x;
            if (y < b1) p[1] = job.list ? job.list[y] : (uint32_t)y;
        }
        process_item2<MAYN>(job, K, s_lut, lut, p, tb, rb, hf);
    }
}

// How many of the launch's blocks began on this SM before this one.
__device__ __forceinline__ uint32_t sm_turn(const GotohJob &job) {
    __shared__ uint32_t s_turn;
    if (threadIdx.x == 0) {
        uint32_t sm;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
        s_turn = atomicAdd(job.sm_blocks + sm % (uint32_t)job.sms, 1u);
    }
    __syncthreads();
    return s_turn;
}

// The warps of a launch take chunks of work from one queue.  With fewer chunks
// than warps those that ask first get them, and they crowd: a scheduler with three
// busy warps takes 0.61 ms for pairs of 150 x 214, one with two 0.49, while others
// idle; and of a batch of unlike pairs the costliest chunks, the list's first, crowd
// too.  So an SM's second to fourth block (`turn` 1 to 3) wait 12,000 cycles (6 us)
// each for those before them, and blocks that find a chunk for every warp of those
// leave (false).  65,536 pairs (1,024 chunks on 608 schedulers) 0.86 ms when all ask
// at once, 0.54 so.  At 2 us an SM's blocks still overtake each other in some runs.
//
// The turn of a block in a batch of like pairs is its order on its SM: the first
// 152 blocks lie on 148 SMs, on which ones depends on the kernels before, and by
// block number 65,536 pairs take 0.53 or 0.65 ms.  For unlike pairs it is by block
// number: an SM then has chunks of all costs in each turn, not one warp a scheduler
// left with the costliest at the end (138,000 pairs of 129 to 244 bases with N 2.25
// ms, 2.4 by order on the SM).
__device__ __forceinline__ bool stagger(const GotohJob &job, uint64_t chunks, uint32_t turn) {
    if (chunks <= turn * (blockDim.x / 32ull) * (uint32_t)job.sms) return false;
    const long long t0 = clock64(), wait = 12000ll * min(turn, 3u);
    while (clock64() - t0 < wait) __nanosleep(200);
    return true;
}

// Persistent paired kernel over the (class range of the) list.  Scratch per
// warp: 2 x tb_words and 2 x rb_words words per lane.
template <int MINB>
__global__ void __launch_bounds__(PAIR_BLOCK, MINB) gotoh2_kernel(GotohJob job, GotohConst K) {
    __shared__ uint32_t s_lut[10];
    __shared__ int8_t s_lut25[32];
    __shared__ uint32_t s_first[STRIP * PAIR_BLOCK];
    if (threadIdx.x == 0) {  // static indices keep the parameter block out of local memory
#pragma unroll
        for (int k = 0; k < 10; k++) s_lut[k] = K.lut4[k >> 1][k & 1];
#pragma unroll
        for (int k = 0; k < 25; k++) s_lut25[k] = K.lut[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t warp_slot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t *tb = job.tb + warp_slot * (2 * job.tb_words) * 32 + 2 * lane;
    uint32_t *rb = job.rb + warp_slot * (2 * job.rb_words) * 32 + 2 * lane;
    uint64_t b0 = 0, b1 = job.list_count ? (uint64_t)(*job.list_count) : job.n_pairs;
    if (job.range) {  // one length class of the binned list
        b0 = job.range[0];
        b1 = job.range[1] > job.range[0] ? job.range[1] : b0;
    }
    const uint64_t chunks = (b1 - b0 + 63) / 64;
    if (chunks < gridDim.x * (PAIR_BLOCK / 32ull) && !stagger(job, chunks, sm_turn(job))) return;
    paired_section<true>(job, K, s_lut, s_lut25, b0, b1, tb, rb, lane, s_first + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Group kernel: G lanes (4, 8, 16 or 32) share a work item of one or two
// pairs.  Lane g of a group fills strips g, g + G, g + 2G, ... one after the
// other; all lanes step together, a strip one column behind the strip above
// it, whose bottom row (H, E) arrives by a warp shuffle one step after it
// was produced.  Strip s (lane g = s mod G, pass p = s / G) meets column j at
// time j + g + p*R; R is the smallest shift that lets every lane finish a
// strip before its next one begins.  Where R = G the last lane's bottom row
// reaches lane 0 by the same shuffle; otherwise it crosses passes through a
// row buffer of one word pair per column.
//
// Why: a thread that owns whole pairs needs the time of its largest pair
// whatever the batch's size (a 300 x 556 window: 5 ms), and with two pairs a
// thread the chip holds 155,648 pairs before it is full.  A group of G lanes
// takes 1/G of that time and holds 1/G of the pairs, so small and middling
// batches fill the chip; small groups waste fewer steps at a pair's ends,
// large ones finish it sooner (plan_dp in abi.cu and make_plan in bins.cu choose).
//
// Cells, keys and packing are the paired kernel's.  A row is computed only
// inside its window by predicates: `act` has a bit per row whose window holds
// the column.  A row below one that is outside its window takes the E that an
// absent cell gives; rows not yet begun or already ended keep their state.
// Steps in which every lane has all 8 rows inside skip the predicates.
// Traceback words of a step lie side by side (one 256-byte line a warp), at
// the step's time; the walks of the group's two pairs run on its first lanes.
// ---------------------------------------------------------------------------

// The traceback of a group's item: words of (strip, column) at their time.
struct GroupTb {
    const uint32_t *tb;  // the warp's region, already at the pair's word of an entry
    int lg, first, R, t0;  // log2 G, the group's first lane, pass shift, time of step 0
    __device__ __forceinline__ uint32_t word(const Geo &, int s, int j) const {
        const int gl = s & ((1 << lg) - 1), t = j + gl + (s >> lg) * R - t0;
        return tb[((size_t)(uint32_t)t * 32 + (uint32_t)(first + gl)) * 2];
    }
};

// One column of a strip, as dp_rows2 over all rows.  MASK: only the rows of
// `act` are inside their windows.  Selects, not branches: the rows' dependent
// steps overlap only within one basic block.
template <bool MASK, bool HASN>
__device__ __forceinline__ uint2 group_rows(Strip2 &S, const Keys2 &c, const Col2 &col,
                                            uint32_t act, uint32_t &upHo, uint32_t &upE,
                                            uint32_t d) {
    uint32_t wa = 0, wb = 0;
    uint32_t kd = __viaddmax_u16x2(d, sub2<HASN>(S.la[0], S.lb[0], col), BIAS2 + 0x00030003u);
#pragma unroll
    for (int r = 0; r < STRIP; r++) {
        const uint32_t kF = S.kF[r];
        uint32_t kE = __viaddmax_u16x2(upE, c.ex, upHo);
        if (MASK && r > 0) kE = (act & (1u << (r - 1))) ? kE : c.ho0;
        upE = and_or_u32(kE, KEEP2, 0x00010001u);
        const uint32_t F4 = and_u32(kF, KEEP2);
        const uint32_t key = __vimax3_u16x2(kd, upE, F4);
        if (r < STRIP - 1)
            kd = __viaddmax_u16x2(S.Hl[r], sub2<HASN>(S.la[r + 1], S.lb[r + 1], col),
                                  BIAS2 + 0x00030003u);
        const uint32_t Hp = and_or_u32(key, KEEP2, 0x00020002u);
        wa = mad_u32(wa, 4u, key - Hp);
        wb = mad_u32(wb, 4u, xor_and_u32(kE, kF, 0x00030003u));
        upHo = Hp - c.oe;
        const uint32_t nF = __viaddmax_u16x2(F4, c.ex, upHo);
        const uint32_t nr = __vmaxu2(S.rmax[r], mad_u32(Hp, c.ks, col.ck));
        const bool in = !MASK || (act & (1u << r));
        S.Hl[r] = in ? Hp : S.Hl[r];
        S.kF[r] = in ? nF : S.kF[r];
        S.rmax[r] = in ? nr : S.rmax[r];
    }
    wa += 0xAAAAAAAAu;  // tags, not tag - 2
    return make_uint2(__byte_perm(wa, wb, 0x5410), __byte_perm(wa, wb, 0x7632));
}

// What a lane knows of its pairs from the strips it has done: the best cell
// (thr, h, i, j0, j1 as in Best2) and the first touching row << 2 | clamped <<
// 1 | left (all ones: none) of each pair.  In shared memory (word w of thread
// t at w * GROUP_BLOCK + t): it is touched once a strip, and the fill needs
// the registers.
constexpr int GROUP_BLOCK = 128;
constexpr int TRACK_WORDS = 11;
enum : int { TR_THR = 0, TR_H = 1, TR_I = 3, TR_J0 = 5, TR_J1 = 7, TR_TOUCH = 9 };

// A strip's rows are done (extend.rs:795-827), as at the end of a strip in
// dp_fill2.  first: the keys of the rows' first cells (stride GROUP_BLOCK).
__device__ __forceinline__ void end_strip2(uint32_t *track, Strip2 &S, const Keys2 &c,
                                           const uint32_t *first, const Geo &g, int n, int i0,
                                           int nact, int clo) {
    const uint32_t ksc = 4u * c.ks;
    if (nact < STRIP) {  // rows past the read do not count
#pragma unroll
        for (int r = 1; r < STRIP; r++)
            if (r >= nact) S.rmax[r] = 0u;
    }
    uint32_t smax = __vimax3_u16x2(S.rmax[0], S.rmax[1], S.rmax[2]);
    smax = __vimax3_u16x2(smax, S.rmax[3], S.rmax[4]);
    smax = __vimax3_u16x2(smax, S.rmax[5], __vmaxu2(S.rmax[6], S.rmax[7]));
    uint32_t thr = track[TR_THR * GROUP_BLOCK];
    if (__vmaxu2(thr, smax) != thr) {
        const uint32_t inv_s = 0xffffffffu / ksc + 1u;  // key / S = mulhi(key, inv_s)
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t v = (smax >> (16 * q)) & 0xffffu;
            if (v > ((thr >> (16 * q)) & 0xffffu)) {
                const uint32_t h = __umulhi(v, inv_s), base = h * ksc;
                int row = 0;
                uint32_t key = 0;
#pragma unroll
                for (int r = STRIP - 1; r >= 0; r--) {
                    const uint32_t x = (S.rmax[r] >> (16 * q)) & 0xffffu;
                    if (x >= base) {
                        row = i0 + r;
                        key = x;
                    }
                }
                const int j0 = clo + (int)((base + ksc - 1u - key) << c.g);
                track[(TR_H + q) * GROUP_BLOCK] = h;
                track[(TR_I + q) * GROUP_BLOCK] = (uint32_t)row;
                track[(TR_J0 + q) * GROUP_BLOCK] = (uint32_t)max(j0, g.lo(row));
                track[(TR_J1 + q) * GROUP_BLOCK] = (uint32_t)min(j0 + (1 << c.g) - 1, g.hi(row));
                thr = (thr & (0xffff0000u >> (16 * q))) | ((base + ksc - 1u) << (16 * q));
            }
        }
        track[TR_THR * GROUP_BLOCK] = thr;
    }
    uint32_t touch[2] = {track[TR_TOUCH * GROUP_BLOCK], track[(TR_TOUCH + 1) * GROUP_BLOCK]};
    if ((touch[0] == ~0u) | (touch[1] == ~0u)) {
        uint32_t zero_halves = 0u;  // as in dp_fill2: no zero half, no touch
#pragma unroll
        for (int r = 0; r < STRIP; r++) {
            const uint32_t u = mad_u32(S.Hl[r], c.ks, c.ck0);
            const uint32_t zl = S.rmax[r] ^ first[r * GROUP_BLOCK], zr = __vmaxu2(S.rmax[r], u) ^ u;
            zero_halves |= ((zl - 0x00010001u) & ~zl) | ((zr - 0x00010001u) & ~zr);
        }
        if (zero_halves & 0x80008000u) {
#pragma unroll
            for (int r = 0; r < STRIP; r++) {
                if (r < nact) {
                    const int lo = g.lo(i0 + r), hi = g.hi(i0 + r);
                    const uint32_t u = mad_u32(S.Hl[r], c.ks, c.ck0), f = first[r * GROUP_BLOCK];
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const uint32_t x = (S.rmax[r] >> (16 * q)) & 0xffffu;
                        if (touch[q] == ~0u) {
                            if (x == ((f >> (16 * q)) & 0xffffu))
                                touch[q] = ((uint32_t)(i0 + r) << 2) | (lo <= 1 ? 3u : 1u);
                            else if (hi < n && x <= ((u >> (16 * q)) & 0xffffu))
                                touch[q] = (uint32_t)(i0 + r) << 2;
                        }
                    }
                }
            }
            track[TR_TOUCH * GROUP_BLOCK] = touch[0];
            track[(TR_TOUCH + 1) * GROUP_BLOCK] = touch[1];
        }
    }
}

// Pass shift of an item: lanes g of the group take the strips in turn.
__device__ __forceinline__ int group_shift(const Geo &g, int m, int nstrips, int lg, int gl) {
    const int G = 1 << lg;
    int r = 0;
    for (int s = gl; s + G < nstrips; s += G)  // chi(s) - clo(s + G) + 1
        r = max(r, g.hi(min((s + 1) * STRIP, m)) - g.lo((s + G) * STRIP + 1) + 1);
    for (int x = 1; x < G; x <<= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, x));
    // a buffered pass runs two columns behind its writes (read ahead)
    return r <= G ? G : max(r, G + 4);
}

// *p = v (shared memory) when x is not 0, as one predicated store: a branch a
// row cost as much as the row.
__device__ __forceinline__ void put_if(uint32_t *p, uint32_t v, uint32_t x) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.shared.u32 [%0], %1;\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(p)),
                 "r"(v), "r"(x)
                 : "memory");
}

// Fill the DP of every group's item (two pairs of one geometry, or one pair
// in both halves; nstrips = 0: none).  tb: the warp's traceback region, a
// word pair per step and lane; rb: the group's row buffer, a word pair per
// column 1..n; first, track: the thread's words in shared memory.
// Every lane of a group returns its item's results.
template <bool HASN>
__device__ __noinline__ void group_fill(const GotohConst &K, const uint32_t *__restrict__ s_lut,
                                        const PairSetup &A, const PairSetup &B, int nstrips, int R,
                                        int steps, uint2 *tb, uint2 *rb, int lane,
                                        int lg, uint32_t *first, uint32_t *track, FillResult &FA,
                                        FillResult &FB) {
    constexpr uint32_t ALL = 0xffffffffu;
    const int G = 1 << lg, gl = lane & (G - 1);
    const int src = (lane & ~(G - 1)) + ((gl - 1) & (G - 1));
    const int m = A.m, n = A.n;
    const Geo g = A.g;
    const Keys2 c = keys2_of(K, m, A.sw);
    const bool ring = R == G;
    const int nh = n - g.half, h1 = g.half + 1;  // c(i) clamped at n / at 1 (Geo)
    track[TR_THR * GROUP_BLOCK] = (4u * c.ks - 1u) * 0x10001u;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        track[(TR_H + q) * GROUP_BLOCK] = track[(TR_I + q) * GROUP_BLOCK] = 0u;
        track[(TR_J0 + q) * GROUP_BLOCK] = track[(TR_J1 + q) * GROUP_BLOCK] = 0u;
        track[(TR_TOUCH + q) * GROUP_BLOCK] = ~0u;
    }
    Strip2 S;
    uint32_t pubH = c.h0, pubE = c.e0, raw = c.h0, diag = c.h0;
    uint2 u0 = make_uint2(c.h0, c.e0), u1 = u0;
    Codes2<HASN> w{A.win, B.win};
    int s = gl - G, j = 0, clo = 1 << 30, chi = -1, phi = -1;
    int r0 = 0;        // off + i0: row r's window begins at j = r0 + r - half
    uint32_t was = 0;  // rows inside their windows one column before
    bool turn = nstrips > 0;  // the lane goes on to its next strip
    bool open = false;        // the lane has a strip, waiting, running or just ended
    for (int t = 0;; t++) {
        if (turn) {
            if (open) {
                const int i0 = s * STRIP + 1;
                end_strip2(track, S, c, first, g, n, i0, min(STRIP, m - i0 + 1), clo);
            }
            open = false;
            turn = false;
            s += G;
            if (s < nstrips) {
                const int i0 = s * STRIP + 1;
                clo = g.lo(i0);
                chi = g.hi(min(i0 + STRIP - 1, m));
                phi = s ? g.hi(i0 - 1) : -1;
                r0 = g.off + i0;
                j = t + g.lo(1) - gl - (s >> lg) * R;
                w.load(clo);
                w.t = 0;
                const uint32_t rwA = load16(A.read.arena, A.read.pos + (uint64_t)(i0 - 1));
                const uint32_t rwB = load16(A.read.arena, B.read.pos + (uint64_t)(i0 - 1));
                const uint32_t rnA = A.read.cnt ? nmask16(A.read.iv, A.read.cnt, i0 - 1) : 0u;
                const uint32_t rnB = B.read.cnt ? nmask16(B.read.iv, B.read.cnt, i0 - 1) : 0u;
#pragma unroll
                for (int r = 0; r < STRIP; r++) {
                    uint32_t ca = (rwA >> (30 - 2 * r)) & 3u, cb = (rwB >> (30 - 2 * r)) & 3u;
                    if ((rnA >> (31 - r)) & 1u) ca = 4;
                    if ((rnB >> (31 - r)) & 1u) cb = 4;
                    S.la[r] = s_lut[2 * ca];
                    S.lb[r] = s_lut[2 * cb];
                    S.Hl[r] = c.h0;
                    S.kF[r] = c.ho0;
                    S.rmax[r] = 0u;
                }
                was = 0;
                open = true;
            } else {
                clo = 1 << 30;
                chi = -1;
            }
        }
        if (t >= steps) break;
        const bool active = j >= clo && j <= chi;
        // the bottom row of the strip above at this column
        uint32_t upH = __shfl_sync(ALL, pubH, src), upE = __shfl_sync(ALL, pubE, src);
        if (!ring && gl == 0 && active && s) {
            if (j == clo) {
                if (clo > 1) raw = rb[clo - 1].x;
                u0 = rb[clo];
                if (clo + 1 <= phi) u1 = rb[clo + 1];
            }
            upH = u0.x;
            upE = u0.y;
            u0 = u1;
            if (j + 2 <= phi) u1 = rb[j + 2];
        }
        if (j == clo)  // the row above's last column left of this strip's
            diag = s && clo - 1 >= g.lo(s * STRIP) && clo - 1 <= phi ? raw : c.h0;
        raw = upH;
        upH = j > phi ? c.h0 : upH;
        upE = j > phi ? c.e0 : upE;
        // rows inside their windows: lo(r) <= j <= hi(r) (Geo), a run of rows
        const int x = j - r0;
        const int rb_ = j >= nh ? STRIP - 1 : min(STRIP - 1, x + g.half);
        const int ra = j <= h1 ? 0 : max(0, x - g.half);
        const uint32_t act = active ? ((2u << rb_) - (1u << ra)) & 0xffu : 0u;
        const uint32_t begin = act & ~was;
        was = act;
        uint32_t upHo = upH - c.oe;
        const Col2 col = w.here(c);
        uint2 words;
        // a lane without a strip may compute what it likes
        if (__all_sync(ALL, !open || act == 0xffu))
            words = group_rows<false, HASN>(S, c, col, act, upHo, upE, diag);
        else
            words = group_rows<true, HASN>(S, c, col, act, upHo, upE, diag);
#pragma unroll
        for (int r = 0; r < STRIP; r++)  // rows that met their first column
            put_if(first + r * GROUP_BLOCK, S.rmax[r], begin & (1u << r));
        pubH = upHo + c.oe;
        pubE = upE;
        diag = upH;
        if (active) {
            __stcs(tb + (size_t)t * 32 + lane, words);
            if (!ring && gl == G - 1) rb[j] = make_uint2(pubH, pubE);
            turn = j == chi && s + G < nstrips;
            w.step();
        }
        j++;
        // new codes for all lanes at once, 16 columns after the last ones or
        // sooner
        if ((t & 15) == 15 && j > clo && j <= chi) w.load(j);
        __syncwarp();
    }
    // the lanes' last strips, all at once
    if (open) {
        const int i0 = s * STRIP + 1;
        end_strip2(track, S, c, first, g, n, i0, min(STRIP, m - i0 + 1), clo);
    }
    // merge the lanes: the largest H, its first row; the first touching row
#pragma unroll
    for (int q = 0; q < 2; q++) {
        uint32_t key = (track[(TR_H + q) * GROUP_BLOCK] << 16) |
                       (0xffffu - track[(TR_I + q) * GROUP_BLOCK]);
        uint32_t j0 = track[(TR_J0 + q) * GROUP_BLOCK], j1 = track[(TR_J1 + q) * GROUP_BLOCK];
        uint32_t touch = track[(TR_TOUCH + q) * GROUP_BLOCK];
        for (int x = 1; x < G; x <<= 1) {
            const uint32_t ok = __shfl_xor_sync(ALL, key, x), ot = __shfl_xor_sync(ALL, touch, x);
            const uint32_t o0 = __shfl_xor_sync(ALL, j0, x), o1 = __shfl_xor_sync(ALL, j1, x);
            touch = min(touch, ot);
            if (ok > key) {
                key = ok;
                j0 = o0;
                j1 = o1;
            }
        }
        FillResult &F = q ? FB : FA;
        F.bestHp = 4 * (int)(key >> 16) + 2;
        F.best_i = key >> 16 ? (int)(0xffffu - (key & 0xffffu)) : 0;
        F.best_j = (int)j0;
        F.last_j = (int)j1;
        F.trow = touch == ~0u ? 0 : (int)(touch >> 2);
        F.tleft = touch != ~0u && (touch & 1u);
        F.tclamp = touch != ~0u && (touch & 2u);
    }
}

// Upper bound of the steps of an item of at most m rows, n columns and sw
// columns a strip.
uint64_t group_steps(uint64_t m, uint64_t n, uint64_t sw, int lg) {
    const uint64_t G = 1ull << lg, strips = (m + STRIP - 1) / STRIP, passes = (strips + G - 1) / G;
    return n + G + (passes ? passes - 1 : 0) * std::max<uint64_t>(sw, G + 4);
}

// A pair's set-up; the group section checks its own scratch.
__device__ __noinline__ bool setup_group(const GotohJob &job, const GotohConst &K, uint32_t pi,
                                         bool write, PairSetup &S) {
    return setup_pair(job, K, pi, ~0ull, ~0ull, write, S);
}

// Out of line for batches without intervals: inlined, the walk shares registers with
// all that the kernel keeps, and any change there moved extend_hint over 60,000
// pairs between 1.58 and 1.72 ms (so 1.47), over 45,000 of 50 to 150 bases between
// 1.14 and 1.24 (1.11).  Not so beside the N-taking fill, which loses more than the
// walk gains (9,718 whole windows with N 0.31 ms, 0.35 with the walk out of line).
__device__ __noinline__ void finish_group(const GotohJob &job, const GotohConst &K,
                                          const int8_t *__restrict__ lut, uint32_t pi, PairSetup &S,
                                          const FillResult &F, const GroupTb &tb) {
    finish_pair(job, K, lut, pi, S, F, tb);
}

// Items 0 .. items - 1 of the (padded, binned) list in groups of 1 << lg
// lanes; item k is positions 2k and 2k + 1.  A warp takes 32 >> lg items at a
// time.  Scratch: the warp's traceback region (group_tb_words word pairs per
// lane) and row buffers (group_rb_words word pairs per group).
template <bool MAYN>
__device__ void group_section(const GotohJob &job, const GotohConst &K,
                              const uint32_t *__restrict__ s_lut, const int8_t *__restrict__ lut,
                              uint64_t items, int lg, uint2 *tb, uint2 *rb0, int lane,
                              uint32_t *first, uint32_t *track) {
    const int G = 1 << lg, groups = 32 >> lg, gl = lane & (G - 1), grp = lane >> lg;
    uint2 *rb = rb0 + (uint64_t)grp * job.group_rb_words;
    const uint64_t total = items;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0)
            base = atomicAdd((unsigned long long *)job.group_queue, (unsigned long long)groups);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= total) break;
        const uint64_t k = base + grp;
        uint32_t p[2] = {NO_PAIR, NO_PAIR};
        if (k < total) {
            p[0] = job.list[2 * k];
            p[1] = job.list[2 * k + 1];
        }
        // both pairs at once when their geometry matches, else one by one
        int need = 0;  // bit q: pair q has a DP; bit 2: together
        {
            PairSetup A, B;
            const bool a = p[0] != NO_PAIR && setup_group(job, K, p[0], gl == 0, A);
            const bool b = p[1] != NO_PAIR && setup_group(job, K, p[1], gl == 0, B);
            need = (a ? 1 : 0) | (b ? 2 : 0);
            if (a && b && A.m == B.m && A.n == B.n && A.g.off == B.g.off && A.g.half == B.g.half)
                need = 4;
        }
        for (int round = 0; round < 2; round++) {
            // this round's first pair: the only one, or both
            const bool on = round == 0 ? need != 0 : need == 3;
            if (!__any_sync(0xffffffffu, on)) break;
            const int q = round == 0 ? (need == 2 ? 1 : 0) : 1;
            PairSetup A, B;
            int nstrips = 0, R = G, steps = -1;
            A.m = A.n = A.sw = 1;
            A.g = Geo{0, 1, 1};
            A.win.cnt = 0;
            if (on) {
                setup_group(job, K, p[q], false, A);
                nstrips = (A.m + STRIP - 1) / STRIP;
            }
            R = group_shift(A.g, A.m, nstrips, lg, gl);
            bool fits = on;
            if (on) {
                const int l = nstrips - 1;
                steps = A.g.hi(A.m) + (l & (G - 1)) + (l >> lg) * R - A.g.lo(1) + 1;
                if ((uint64_t)steps > job.group_tb_words || (uint64_t)A.n >= job.group_rb_words) {
                    // scratch sized too small by the host: refuse, never overrun
                    fits = false;
                    nstrips = 0;
                    steps = -1;
                    for (int x = 0; x < 2; x++)
                        if (gl == 0 && (need == 4 || x == q)) {
                            if (setup_group(job, K, p[x], false, B)) {
                                B.o.status = ESP_EINVAL;
                                job.out[p[x]] = B.o;
                            }
                        }
                }
            }
            B = A;
            if (need == 4 && fits) setup_group(job, K, p[1], false, B);
            const int all_steps = __reduce_max_sync(0xffffffffu, steps);
            FillResult FA, FB;
            if (MAYN && windows_n(job))  // as in process_item2
                group_fill<true>(K, s_lut, A, B, nstrips, R, all_steps, tb, rb, lane, lg, first, track, FA,
                                  FB);
            else
                group_fill<false>(K, s_lut, A, B, nstrips, R, all_steps, tb, rb, lane, lg, first, track, FA,
                                  FB);
            __syncwarp();  // traceback words of every lane are visible to the walks
            if (fits && gl < (need == 4 ? 2 : 1)) {
                const int gfirst = lane & ~(G - 1);
                PairSetup &S = gl ? B : A;
                const GroupTb view{reinterpret_cast<const uint32_t *>(tb) + gl, lg, gfirst, R, A.g.lo(1)};
                if (MAYN) finish_pair(job, K, lut, p[gl ? 1 : q], S, gl ? FB : FA, view);
                else finish_group(job, K, lut, p[gl ? 1 : q], S, gl ? FB : FA, view);
            }
            __syncwarp();
        }
    }
}

// Small and middling batches of the binned list: its costly front in groups
// (job.group_plan: list entries, log2 of a group's lanes), the rest two pairs
// per thread.  A thread's pair takes as long as it takes, so the items that
// would outlast the rest of the batch are the ones given to groups, and the
// others keep the paired kernel's higher throughput (make_plan, bins.cu).
//
// Two pairs a lane take several times a group's scratch.  With job.thread_warps
// set only that many of the warps an SM starts in one of a block's four places
// own it, the first to come, and the others as much as groups take (65,536 reads
// of at most 300 x 428: 6.4 GB, 10.1 with all warps the same).  Each SM uses its
// own part of the scratch, for groups and for pairs per thread one after the other:
// given out over the whole chip, or apart from the groups', the same work took up
// to a tenth longer (80,000 extend_hint pairs of 50 to 300 bases 3.5 ms, apart 3.8).
// MAYN: the batch has N intervals, in reads or windows.
template <bool MAYN>
__global__ void __launch_bounds__(GROUP_BLOCK, 4) gotoh_mixed_kernel(GotohJob job, GotohConst K) {
    static_assert(GROUP_BLOCK == PAIR_BLOCK, "one shared array serves both sections");
    __shared__ uint32_t s_lut[10];
    __shared__ int8_t s_lut25[32];
    __shared__ uint32_t s_words[(STRIP + TRACK_WORDS) * GROUP_BLOCK];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 10; k++) s_lut[k] = K.lut4[k >> 1][k & 1];
#pragma unroll
        for (int k = 0; k < 25; k++) s_lut25[k] = K.lut[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t total = *job.list_count;
    const uint64_t split = job.group_plan[0];
    const uint32_t lg = job.group_plan[1] & 7u;
    const uint64_t chunks = (split << lg) / 64 + (total - split + 63) / 64;
    const bool few = chunks < gridDim.x * (GROUP_BLOCK / 32ull), alike = job.group_plan[1] >> 3;
    // (a count that nothing needs would only change the order of the first chunks)
    const uint32_t turn = (few && alike) || job.thread_warps ? sm_turn(job) : 0u;
    if (few && !stagger(job, chunks, alike ? turn : blockIdx.x / (uint32_t)job.sms)) return;
    uint64_t tb, rb;      // the warp's words
    bool threads = true;  // it owns what pairs per thread take
    if (job.thread_warps) {
        uint32_t sm;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
        if (sm >= (uint32_t)job.sms || turn >= job.max_warps) return;  // no words for such a block
        const uint64_t unit = sm * 4ull + (threadIdx.x >> 5);
        threads = turn < job.thread_warps;
        const uint64_t early = min(turn, job.thread_warps), late = turn - early;
        tb = unit * job.unit_tb_words + early * job.warp_tb_words + late * 64 * job.group_tb_words;
        rb = unit * job.unit_rb_words + early * job.warp_rb_words + late * job.group_warp_rb;
    } else {
        const uint64_t warp_slot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        tb = warp_slot * job.warp_tb_words;
        rb = warp_slot * job.warp_rb_words;
    }
    group_section<MAYN>(job, K, s_lut, s_lut25, split / 2, (int)lg,
                  reinterpret_cast<uint2 *>(job.tb + tb), reinterpret_cast<uint2 *>(job.rb + rb), lane,
                  s_words + threadIdx.x, s_words + STRIP * GROUP_BLOCK + threadIdx.x);
    if (threads)
        paired_section<MAYN>(job, K, s_lut, s_lut25, split, total, job.tb + tb + 2 * lane,
                       job.rb + rb + 2 * lane, lane, s_words + threadIdx.x);
}

cudaError_t launch_gotoh_mixed(const GotohJob &job, const GotohConst &k, int warps,
                               cudaStream_t st) {
    if (job.n_iv_count) gotoh_mixed_kernel<true><<<(warps + 3) / 4, GROUP_BLOCK, 0, st>>>(job, k);
    else gotoh_mixed_kernel<false><<<(warps + 3) / 4, GROUP_BLOCK, 0, st>>>(job, k);
    return cudaGetLastError();
}

int make_gotoh_const(const esp_extend_params &p, GotohConst &k) {
    // Device domain: substitution scores fit the 4*s int8 PRMT table and the
    // scaled gap keys fit int16 in the row buffer.  The reference's own
    // parameter sets (defaults 2/-4/4/2 and the 400/400 rescue pass) are inside.
    auto in8 = [](int v) { return v >= -32 && v <= 31; };
    if (!in8(p.match_score) || !in8(p.mismatch) || p.gap_open < 0 || p.gap_ext < 0 ||
        4LL * (p.gap_open + p.gap_ext) > 8000 || p.edit_dir < 0 || p.edit_dir > 2)
        return ESP_EDOMAIN;
    k.open_ext = -(p.gap_open + p.gap_ext);
    k.ext = -p.gap_ext;
    k.oe4 = 4 * k.open_ext;
    k.ex4 = 4 * k.ext;
    k.match = p.match_score;
    k.edit_dir = p.edit_dir;
    // SubstLut (extend.rs:164-179): scores[read*5 + ref]
    int lut[25];
    for (int i = 0; i < 25; i++) lut[i] = (int16_t)p.mismatch;
    for (int c = 0; c < 4; c++) lut[c * 5 + c] = (int16_t)p.match_score;
    if (p.edit_dir == ESP_EDIT_AG) lut[10] = 0;  // read G / ref A
    if (p.edit_dir == ESP_EDIT_TC) lut[8] = 0;   // read C / ref T
    for (int i = 0; i < 25; i++) k.lut[i] = (int8_t)lut[i];
    // The row buffer keeps 4E (signed) and 4H + 2 in 16 bits, so every H and
    // E must stay <= 8191; H <= m * (largest substitution score).
    int smax = 0;
    for (int i = 0; i < 25; i++) smax = lut[i] > smax ? lut[i] : smax;
    k.max_m = smax > 0 ? 8191 / smax : 32767;
    k.smax = smax;
    // a walk may take matches without reading the traceback (Walker::next)
    k.match_skip = p.match_score > 0 && p.match_score == smax;
    // traceback kind of a diagonal step by read code * 5 + window code:
    // K_MM for equal ACGT codes, K_MZ for the edit-tolerated pair, K_MX
    // otherwise (a match and a tolerated pair exclude each other)
    k.dkind = 0;
    for (int q = 0; q < 5; q++)
        for (int c = 0; c < 5; c++) {
            const bool mz = (p.edit_dir == ESP_EDIT_AG && q == 2 && c == 0) ||
                            (p.edit_dir == ESP_EDIT_TC && q == 1 && c == 3);
            const int kd = (q == c && q < 4) ? K_MM : (mz ? K_MZ : K_MX);
            k.dkind |= (uint64_t)kd << (2 * (q * 5 + c));
        }
    for (int rc = 0; rc < 5; rc++) {
        uint32_t w[2] = {0, 0};
        for (int fc = 0; fc < 8; fc++) {
            int s = lut[rc * 5 + (fc < 4 ? fc : 4)];
            w[fc >> 2] |= (uint32_t)(uint8_t)(int8_t)(4 * s) << (8 * (fc & 3));
        }
        k.lut4[rc][0] = w[0];
        k.lut4[rc][1] = w[1];
    }
    return ESP_OK;
}

void gotoh_scratch_words(uint32_t m, uint32_t n, int32_t half, uint64_t &tb, uint64_t &rb) {
    bool full = half < 0;
    int64_t h = full ? n : half;
    int64_t sw = full ? n : (2 * h + STRIP < (int64_t)n ? 2 * h + STRIP : (int64_t)n);
    tb = (uint64_t)((m + STRIP - 1) / STRIP) * (uint64_t)sw;
    rb = (uint64_t)sw;
}

// Kernel variants: 0, 1 = one pair per thread at 3 / 4 resident blocks per
// SM; 2, 3 = two pairs per thread (16x2 lanes) at 3 / 4.  More blocks mean
// fewer registers per thread (spills) but more warps to hide latency; which
// wins depends on the band width, so the host picks per length class (the
// tuning in abi.cu).
int gotoh_blocks_per_sm(int block, int variant) {
    int nb = 0;
    cudaError_t e;
    switch (variant) {
    case 0: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, gotoh_kernel<3>, block, 0); break;
    case 2: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, gotoh2_kernel<3>, block, 0); break;
    case 3: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, gotoh2_kernel<4>, block, 0); break;
    default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, gotoh_kernel<4>, block, 0);
    }
    if (e != cudaSuccess) return 1;
    return nb > 0 ? nb : 1;
}

int gotoh_mixed_blocks_per_sm() {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, gotoh_mixed_kernel<true>, GROUP_BLOCK, 0) != cudaSuccess)
        return 1;
    return nb > 0 ? nb : 1;
}

cudaError_t launch_gotoh(const GotohJob &job, const GotohConst &k, int warps, int block,
                         cudaStream_t st, int variant) {
    int threads = warps * 32;
    int grid = (threads + block - 1) / block;
    switch (variant) {
    case 0: gotoh_kernel<3><<<grid, block, 0, st>>>(job, k); break;
    case 2: gotoh2_kernel<3><<<grid, block, 0, st>>>(job, k); break;
    case 3: gotoh2_kernel<4><<<grid, block, 0, st>>>(job, k); break;
    default: gotoh_kernel<4><<<grid, block, 0, st>>>(job, k);
    }
    return cudaGetLastError();
}

}  // namespace esp
