// swb_ext_skip.cuh -- the rows of an extension before its first mismatch,
// without computing them (BandedSWScalar.align,
// Sources/Alignment/BandedSWScalar.swift:21-191).
//
// While the query matches the target base for base from the start, every
// value is known: H(i, j) is max(0, h0 + a*(min(i, j) + 1) - gap(|i - j|)),
// since no path can have more matches or fewer gaps and the one along the
// diagonal and one gap reaches it; so is E on and left of the diagonal, the
// band (narrowing included), and the running results (the diagonal is each
// row's maximum and a new best, so max_off stays 0 and z-drop cannot stop).
// E right of the diagonal depends on chance matches there, but only through
// the last few rows: each row adds a + eIns + eDel to what a path through it
// can give, so after ext_lookback() rows a mismatch there (a + max(b, 1) less)
// still beats anything older.  A task therefore starts that many rows before
// its first mismatch with E = 0 there, in the state the reference would have.
// 30 % of the cells of 150-base reads with 1 % errors lie in these rows.
#pragma once

#include "swb_device.cuh"
#include "swb_internal.h"

namespace swb {
namespace {

// Rows after which the E words right of the diagonal are exact.
__device__ __forceinline__ int ext_lookback(const DevScoring &sc) {
    const int gain = sc.a + sc.e_ins + sc.e_del;
    return (sc.a + imax(sc.b, 1) + gain - 1) / gain;
}

// Eight bytes p[0..7] of a buffer, byte k of the result = p[k]: three aligned
// words, each holding one of the eight bytes at least.
__device__ __forceinline__ uint2 load8(const uint8_t *p) {
    const uintptr_t x = (uintptr_t)p;
    const uint32_t *w = (const uint32_t *)(x & ~(uintptr_t)3);
    const uint32_t sh = (uint32_t)(x & 3) * 8;
    const uint32_t w0 = w[0], w1 = w[1], w2 = sh ? w[2] : 0u;
    return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}

// Eight bases of the .pac strand from base b on, one per byte.
__device__ __forceinline__ uint2 load8_pac(const uint8_t *pac, uint64_t b) {
    const uint8_t *p = pac + (b >> 2);
    const uintptr_t x = (uintptr_t)p;
    const uint32_t *w = (const uint32_t *)(x & ~(uintptr_t)3);
    const uint32_t at = (uint32_t)(x & 3) * 4 + (uint32_t)(b & 3);             // base within the first word
    const uint32_t w0 = __byte_perm(w[0], 0u, 0x0123);                          // first base in the top bits
    const uint32_t w1 = at > 8 ? __byte_perm(w[1], 0u, 0x0123) : 0u;
    const uint32_t v = __funnelshift_l(w1, w0, 2 * at) >> 16;                   // 8 bases, the first at bits 15-14
    auto spread = [](uint32_t x4) {                                            // 4 bases, the first at bits 7-6
        return ((x4 >> 6) | (x4 << 4) | (x4 << 14) | (x4 << 24)) & 0x03030303u;
    };
    return make_uint2(spread(v >> 8), spread(v & 0xFFu));
}

__device__ __forceinline__ uint2 reverse8(uint2 v) {
    return make_uint2(__byte_perm(v.y, 0u, 0x0123), __byte_perm(v.x, 0u, 0x0123));
}

// Leading positions at which query and target hold the same base (not N).
// Eight at a time; loads stay within words that hold a byte of the spans.
__device__ __forceinline__ int ext_match_len(const swb_ext_task &tk, const uint8_t *__restrict__ bases,
                                             const uint8_t *__restrict__ pac) {
    const int m = imin(tk.qlen, tk.tlen);
    const bool qrev = tk.flags & SWB_Q_REVERSE, trev = tk.flags & SWB_T_REVERSE, tref = tk.flags & SWB_T_FROM_REF;
    const uint32_t comp = tk.flags & SWB_T_COMPLEMENT ? 0x03030303u : 0u;       // (an N becomes no base)
    int p = 0;
    for (; p + 8 <= m; p += 8) {
        uint2 q = load8(bases + tk.q_off + (uint64_t)(qrev ? tk.qlen - 8 - p : p));
        const uint64_t to = tk.t_off + (uint64_t)(trev ? tk.tlen - 8 - p : p);
        uint2 t = tref ? load8_pac(pac, to) : load8(bases + to);
        if (qrev) q = reverse8(q);
        if (trev) t = reverse8(t);
        const uint32_t d0 = (q.x ^ t.x ^ comp) | (q.x & 0xFCFCFCFCu), d1 = (q.y ^ t.y ^ comp) | (q.y & 0xFCFCFCFCu);
        if (d0 | d1) return p + (d0 ? (__ffs(d0) - 1) >> 3 : 4 + ((__ffs(d1) - 1) >> 3));
    }
    for (; p < m; ++p) {
        const uint32_t q = span_base(bases, pac, tk.q_off, p, tk.qlen, tk.flags, false);
        const uint32_t t = span_base(bases, pac, tk.t_off, p, tk.tlen, tk.flags, true);
        if (q != t || q > 3u) break;
    }
    return p;
}

// First rows a task leaves out: up to its first mismatch less the lookback.
__device__ __forceinline__ int ext_skip_rows(const swb_ext_task &tk, const DevScoring &sc,
                                             const uint8_t *__restrict__ bases, const uint8_t *__restrict__ pac) {
    constexpr int kMost = 1 << 20;   // keeps the sums below within int32
    if (sc.a <= 0 || tk.h0 <= 0 || tk.h0 > (1 << 29) || tk.w < 1 || tk.qlen <= 0 || tk.tlen <= 0 || sc.o_ins > kMost ||
        sc.e_ins > kMost || sc.o_del > kMost || sc.e_del > kMost)
        return 0;
    return imax(ext_match_len(tk, bases, pac) - ext_lookback(sc), 0);
}

// First column of row i0 > 0 (ExtStart::beg): the first nonzero word after row
// i0-1, within the band.
__device__ __forceinline__ int ext_start_col(const DevScoring &sc, int w, int h0, int i0) {
    const int num = sc.o_del + sc.e_del * i0 - h0 - sc.a;
    return imax(imax(i0 - 1 - w, 0), imin(num >= 0 ? num / (sc.a + sc.e_del) + 1 : 0, i0));
}

// The state after rows 0 .. i0-1 (i0 > 0).
struct ExtStart {
    int i0, beg, end;       // the next row's band before its clamps (:95-97)
    int b, e, eFirst;       // the last row's band [b, e), row 0's end
    int dLast;              // the last row's diagonal H, the best score
    int gScore, gTle;
    // Word j as the reference's h[j], e[j]: H of column j-1 of the last row and E of the next row.
    __device__ __forceinline__ void word(const DevScoring &sc, int h0, int j, int &hj, int &ej) const {
        ej = 0;
        if (j > e) {
            // Never reached (the first row's value, :65-77) or the zero tail.
            const long long v = (long long)h0 - sc.o_ins - (long long)sc.e_ins * j;
            hj = j > eFirst && v > 0 ? (int)v : 0;
        } else if (j > i0) {
            hj = imax(dLast - sc.o_ins - sc.e_ins * (j - i0), 0);
        } else if (j == i0) {
            hj = dLast;
        } else {
            // Left of the diagonal: one deletion from the column's diagonal cell.
            const int gap = sc.o_del + sc.e_del * (i0 - j), dj = h0 + sc.a * j;
            hj = (j == b && b > 0) || j < beg ? 0 : imax(dj - gap, 0);         // (b: the row began here)
            ej = j < beg ? 0 : imax(dj + sc.a - gap, 0);
        }
    }
};

// COUNT: adds the rows' cells as the reference computes them.
template <bool COUNT>
__device__ __forceinline__ ExtStart ext_start(const DevScoring &sc, int qlen, int w, int h0, int i0,
                                              unsigned long long &cells) {
    ExtStart s{i0, 0, qlen, 0, qlen, 0, h0 + sc.a * i0, -1, -1};
    for (int r = 0; r < i0; ++r) {
        s.b = imax(imax(s.beg, r - w), 0);
        s.e = imin(imin(s.end, r + w + 1), qlen);
        if (r == 0) s.eFirst = s.e;
        if (COUNT) cells += (unsigned long long)(s.e - s.b);
        const int d = h0 + sc.a * (r + 1);                                     // the row's diagonal H, its maximum
        if (s.e == qlen) {                                                     // :149-152 (it never falls from row to row)
            s.gTle = r;
            s.gScore = r == qlen - 1 ? d : imax(d - sc.o_ins - sc.e_ins * (qlen - 1 - r), 0);
        }
        const int right = imin(r + imax(d - sc.o_ins - 1, 0) / sc.e_ins, s.e - 1);   // last column with H > 0
        s.end = imin(right + 3, qlen);
        if (COUNT || r == i0 - 1) s.beg = imax(s.b, ext_start_col(sc, w, h0, r + 1));   // first nonzero word (:175-180)
    }
    return s;
}

}  // namespace
}  // namespace swb
