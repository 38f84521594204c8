// swb_local.cu -- kernel 3: local Smith-Waterman for mate rescue, bit-exact
// with LocalSWAligner.align (Sources/Alignment/LocalSWAligner.swift:42-493).
//
// The reference runs Farrar's striped algorithm on SIMD16<UInt8> (16 lanes,
// sn = ceil(qLen/16) stripes, lane l of stripe s holding query position
// s + l*sn) with a single-pass lazy-F correction and a per-stripe
// first-lane tie-break.  That is not the textbook SW recurrence, so a
// wavefront kernel would not match it.  Here 8 threads play the 16 SIMD
// lanes: thread t keeps lanes t and t + 8 of every stripe as the two 16-bit
// halves of one register (striped_pass), so one DPX s16x2 operation advances
// two lanes and a warp holds four tasks.
// The forward and the reverse pass (:106-131) are separate launches: the
// forward one takes the tasks by stripe count and target length, the reverse
// one by the stripe count and length that the forward hits leave, so the
// four tasks of a warp always have the same stripe count and nearly the same
// number of columns.
// Tasks the reference sends to its scalar int32 fallback (qLen*A > 250,
// u8 overflow, a zero forward score, or a failed reverse pass) are
// appended to a device list and finished by a one-thread-per-task kernel
// that restates scalarAlign/scalarSWPass (:327-492).
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <atomic>

#include "swb_device.cuh"
#include "swb_internal.h"

namespace swb {
namespace {

constexpr int kLT = 128;          // threads per block, striped kernels (16 tasks)
constexpr int kST = 64;           // threads per block, scalar fallback
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kMaxSn = 16;        // stripes: qLen * a <= 250 and a >= 1
// Stripe counts 1..kSnSplit run in one kernel instance, the others in a
// second one with more registers.
constexpr int kSnSplit = 10;

struct LocalArgs {
    DevScoring sc;
    const uint8_t *bases;
    const uint8_t *pac;
    const swb_local_task *tasks;
    swb_local_result *out;
    const uint32_t *order;       // sorted tasks of the pass
    const uint32_t *bin_start;   // 18 entries: bin 0 = scalar (forward) / nothing to do (reverse), bins 1..16 = stripes
    uint32_t *fallback;          // task indices for the scalar kernel
    unsigned int *fallback_n;
    unsigned long long *cells;
    uint32_t *claim;             // next unit of four tasks (zeroed per call)
    uint32_t *rkeys;             // forward pass: the reverse pass's sort key of each sorted position
    uint32_t *peaks;             // score2 peak lists, peak_stride entries per task in flight
    int peak_stride;
};

__device__ __forceinline__ int clamp_min_sub(int v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }

__device__ __forceinline__ uint32_t rep2(uint32_t v) { return v * 0x10001u; }

struct PassOut {
    int score, qEnd, tEnd, score2;
    bool nil;
};

// simdSWPass (:133-306) for one task per 8 threads; every active task of the
// warp has exactly SN stripes.
//
// Values are kept as 16-bit halves biased by kB, so the packed constants are
// added with one 32-bit add (no half ever goes below zero), and H is kept as
// G = H - gOE - gE, what both gap recurrences start from: the u8 saturating
// steps subs(max(subs(H, gOE), X), gE) are max(H - gOE - gE, X - gE, 0).
// Leaving E unclamped changes nothing, since H takes its maximum with F,
// which is clamped.  One stripe of two lanes is then a byte permute (both
// lanes' profile bytes), three adds, and three DPX operations: four half-rate
// and three full-rate instructions.  Bound by the ALU pipe and issue.  Against
// 16 threads a task with one lane each and 32-bit values (two tasks a warp,
// both passes in one launch per stripe count), 50k pairs of 150 x 700 went
// from 9.29 to 3.30 ms (forward launch 2.29 ms, issue 71 %).  Part of that is the
// reverse pass stopping early (rev_cap); its columns left out count as cells all
// the same.
//
// WRAP: H + profile may pass 255 while H <= 250, so the reference's UInt8
// wrap is applied; else it cannot happen (H > 250 ends the pass, :247).
//
// The position of the maximum is found once, at the end, from a copy of the
// stripes taken in shared memory at each column that raises the score.  The
// reference's stripe walk (:249-263) takes, at such a column, the first
// stripe whose lane maximum is the column's and the first real lane holding
// it there.  A padding lane never holds a new maximum: its diagonal term
// loses the bias (profile 0), its E and F descend from earlier columns or
// from a larger H of the same column, so its value stays at or below the old
// maximum or strictly below the column's real maximum.
//
// REV stops early once no later column can raise the score.  H at query
// position j is at most a*(j+1), so nothing passes a*qLen.  When the forward
// score is at least a*(qLen-1) - gOE - gE, no alignment with an insertion
// beats it (it would leave a query base unmatched and pay a gap), and every
// alignment without one is computed exactly by both passes (only F is subject
// to the striped shortcuts), so the reverse maximum is the forward score.
// (WRAP: the arithmetic may lose alignments, so only a*qLen bounds it.)
__device__ __forceinline__ int rev_cap(const DevScoring &sc, bool wrap, int qLen, int fwd_score) {
    const int gOEE = sc.o_ins + 2 * sc.e_ins;
    return !wrap && fwd_score >= sc.a * (qLen - 1) - gOEE ? fwd_score : sc.a * qLen;
}

template <int SN, bool WRAP, bool REV>
__device__ __forceinline__ PassOut striped_pass(const LocalArgs &a, const swb_local_task &tk, bool act, int qLen,
                                                int tLen, int minSub, int cap, uint32_t *peaks, uint4 *snap) {
    constexpr uint32_t kB = 0x1000u;                     // a multiple of 256
    const DevScoring &sc = a.sc;
    const int bias = sc.b & 0xFF;                        // UInt8(mismatchPenalty)
    const int gOE = (sc.o_ins + sc.e_ins) & 0xFF, gE = sc.e_ins & 0xFF;
    const uint32_t Z = rep2(kB);
    const uint32_t oee = rep2((uint32_t)(gOE + gE)), ge = rep2((uint32_t)gE);
    const uint32_t negGe = rep2((uint32_t)-gE & 0xFFFFu);   // lane-wise -gE for the DPX adds
    const uint32_t zeroG = Z - oee;
    const uint32_t cAdd = oee - rep2((uint32_t)bias);    // G + cAdd + profile = the biased diagonal term
    const uint32_t cBias = rep2(kB - (uint32_t)bias);
    const int t = threadIdx.x & 7;
    // Profile table of a target base: byte q = UInt8(clamping: mat[t][q] + bias)
    // for q in 0..4 (:153-167); byte 5 = 0 for padding lanes.
    auto cl = [](int v) -> uint32_t { return (uint32_t)(v < 0 ? 0 : (v > 255 ? 255 : v)); };
    const uint32_t pA = cl(sc.a + bias), pB = cl(-sc.b + bias), pN = cl(-1 + bias);
    const uint32_t rowB = pB * 0x01010101u, rowN = pN * 0x01010101u, dAB = pA - pB;
    uint32_t sel[SN], G[SN], E[SN];   // sel: prmt selector of both lanes' query codes
#pragma unroll
    for (int s = 0; s < SN; ++s) {
        auto code = [&](int j) -> uint32_t {
            return act && j < qLen
                       ? span_base(a.bases, a.pac, tk.q_off, REV ? (qLen - 1 - j) : j, tk.qlen, tk.flags, false) & 7u
                       : 5u;
        };
        sel[s] = code(s + t * SN) | 0x50u | (code(s + (t + 8) * SN) << 8) | 0x5000u;
        G[s] = zeroG;
        E[s] = Z;
    }
    const bool trackPeaks = !REV && minSub > 0;
    const int kNever = 0x3FFF;
    int maxScore = 0, maxI = -1;
    int nPeaks = 0, lastPeak = 0;                        // lastPeak = (score << 16) | col
    bool nil = false;
    // A column matters when its maximum passes thr: a new best score, a peak
    // (:266-286), or the u8 overflow limit (:247).
    const int peakThr = trackPeaks ? min(minSub - 1, 250) : 250;
    int thr = act ? 0 : kNever;
    int cols = act ? tLen : 0;
    cols = max(cols, __shfl_xor_sync(kFull, cols, 8));
    cols = max(cols, __shfl_xor_sync(kFull, cols, 16));
    // Row tables of the target, 8 columns per load: thread t holds column
    // c0 + t of its task, the next 8 are loaded a block ahead, and column i is
    // a shuffle from thread i % 8.
    auto tload = [&](int c) -> uint32_t {
        const uint32_t b = act && c < tLen
                               ? span_base(a.bases, a.pac, tk.t_off, REV ? (tLen - 1 - c) : c, tk.tlen, tk.flags, true)
                               : 4u;
        return b >= 4u ? rowN : rowB + (dAB << (8 * b));                       // :202
    };
    uint32_t tcur = tload(t), tnext = tload(8 + t);
    for (int i = 0; i < cols; ++i) {
        if (i > 0 && (i & 7) == 0) {   // warp-uniform
            tcur = tnext;
            tnext = tload(i + 8 + t);
        }
        if (i == tLen) thr = kNever;                     // the task's columns are done
        const uint32_t row = __shfl_sync(kFull, tcur, i & 7, 8);
        // shiftRight(hArr[sn-1]) (:206): lane l takes lane l-1, lane 0 zero;
        // lane 8 (thread 0's high half) takes lane 7 (thread 7's low half).
        uint32_t vG = __shfl_sync(kFull, G[SN - 1], (t - 1) & 7, 8);
        if (t == 0) vG = __byte_perm(vG, zeroG, 0x1054);
        uint32_t f = Z;
#pragma unroll
        for (int s = 0; s < SN; ++s) {                   // :209-231
            const uint32_t prof = prmt(row, pN, sel[s]);
            uint32_t d;
            if constexpr (WRAP) d = ((vG + oee + prof) & 0x00FF00FFu) + cBias;
            else d = vG + prof + cAdd;
            vG = G[s];
            E[s] = __viaddmax_s16x2(E[s], negGe, vG);
            G[s] = __vimax3_s16x2(d, E[s], f) - oee;
            f = __vimax3_s16x2(f - ge, G[s], Z);
        }
        uint32_t corrF = __shfl_sync(kFull, f, (t - 1) & 7, 8);   // lazy-F (:234-242)
        if (t == 0) corrF = __byte_perm(corrF, Z, 0x1054);
        // The correction runs until a stripe that it changes in no lane (:236-239).
        // Most columns of unrelated sequence change nothing at stripe 0 and skip
        // it; the others run the whole chain, note the stripes each thread
        // changes, and keep those before the first stripe that no lane of the
        // task changes (one exchange for the column instead of a vote per
        // stripe: 50k pairs of 150 x 700, 3.50 -> 3.30 ms).
        if (__any_sync(kFull, __vmaxs2(G[0], corrF - oee) != G[0])) {
            uint32_t nG[SN];
            unsigned ch = 0;
#pragma unroll
            for (int s = 0; s < SN; ++s) {
                nG[s] = __vmaxs2(G[s], corrF - oee);
                if (nG[s] != G[s]) ch |= 1u << s;
                corrF = __viaddmax_s16x2(corrF, negGe, nG[s]);
            }
            ch |= __shfl_xor_sync(kFull, ch, 4);
            ch |= __shfl_xor_sync(kFull, ch, 2);
            ch |= __shfl_xor_sync(kFull, ch, 1);
            ch = (ch ^ (ch + 1)) >> 1;                   // the ones below the first zero
#pragma unroll
            for (int s = 0; s < SN; ++s)
                if ((ch >> s) & 1u) G[s] = nG[s];
        }
        uint32_t m = G[0];                               // column max (:245-263)
#pragma unroll
        for (int s = 1; s + 1 < SN; s += 2) m = __vimax3_s16x2(m, G[s], G[s + 1]);
        if constexpr (SN % 2 == 0) m = __vmaxs2(m, G[SN - 1]);
        const uint32_t thrG = rep2((uint32_t)thr) + zeroG;
        if (!__any_sync(kFull, __vmaxs2(m, thrG) != thrG)) continue;
        m = __vmaxs2(m, __shfl_xor_sync(kFull, m, 4));
        m = __vmaxs2(m, __shfl_xor_sync(kFull, m, 2));
        m = __vmaxs2(m, __shfl_xor_sync(kFull, m, 1));
        const int colMax = (int)max(m & 0xFFFFu, m >> 16) - (int)(zeroG & 0xFFFFu);
        if (colMax > thr) {                              // group-uniform
            if (colMax > 250) {
                nil = true;
                thr = kNever;
            } else {
                if (colMax > maxScore) {
                    maxScore = colMax;
                    maxI = i;
#pragma unroll
                    for (int k = 0; k < (SN + 3) / 4; ++k)
                        snap[k * kLT] = make_uint4(G[4 * k], 4 * k + 1 < SN ? G[4 * k + 1 < SN ? 4 * k + 1 : 0] : 0u,
                                                   4 * k + 2 < SN ? G[4 * k + 2 < SN ? 4 * k + 2 : 0] : 0u,
                                                   4 * k + 3 < SN ? G[4 * k + 3 < SN ? 4 * k + 3 : 0] : 0u);
                }
                if (trackPeaks && colMax >= minSub) {    // :266-286
                    if (nPeaks == 0 || (lastPeak & 0xFFFF) + 1 != i) {
                        lastPeak = (colMax << 16) | i;
                        if (t == 0) peaks[nPeaks] = (uint32_t)lastPeak;
                        ++nPeaks;
                    } else if ((lastPeak >> 16) < colMax) {
                        lastPeak = (colMax << 16) | i;
                        if (t == 0) peaks[nPeaks - 1] = (uint32_t)lastPeak;
                    }
                }
                thr = REV && maxScore >= cap ? kNever : min(maxScore, peakThr);
            }
        }
        // Leave once every task of the warp has its answer.
        if (REV && __all_sync(kFull, thr == kNever)) break;
    }
    __syncwarp();
    // Position of the maximum in the copied stripes: the first stripe, then
    // the first lane, holding it.
    int at = 0x7FFF;                                     // stripe * 16 + lane
    if (act && maxScore > 0) {
        const uint32_t g = (uint32_t)maxScore + (zeroG & 0xFFFFu);
        for (int s = SN - 1; s >= 0; --s) {
            const uint32_t v = reinterpret_cast<const uint32_t *>(snap + (s >> 2) * kLT)[s & 3];
            if ((v >> 16) == g && s + (t + 8) * SN < qLen) at = s * 16 + t + 8;
            if ((v & 0xFFFFu) == g && s + t * SN < qLen) at = s * 16 + t;
        }
    }
    at = min(at, __shfl_xor_sync(kFull, at, 4));
    at = min(at, __shfl_xor_sync(kFull, at, 2));
    at = min(at, __shfl_xor_sync(kFull, at, 1));
    PassOut o{maxScore, at == 0x7FFF ? -1 : (at >> 4) + (at & 15) * SN, maxI, 0, nil || !act};
    if constexpr (!REV) {
        // score2 (:290-303): the 8 threads scan the peak list.
        int maxBase = 0;                                 // :192-199
        if (trackPeaks) {
            maxBase = (int)max(max(pA, pB), pN);
            maxBase = maxBase > bias ? maxBase - bias : 0;
        }
        int s2 = 0;
        const bool do2 = act && !nil && trackPeaks && nPeaks > 0 && maxScore > 0 && maxBase > 0;
        if (do2) {
            const int r = (maxScore + maxBase - 1) / maxBase;
            const int low = maxI - r, high = maxI + r;
            for (int k = t; k < nPeaks; k += 8) {
                const uint32_t e = peaks[k];
                const int col = (int)(e & 0xFFFFu), scv = (int)(e >> 16);
                if ((col < low || col > high) && scv > s2) s2 = scv;
            }
        }
        s2 = max(s2, __shfl_xor_sync(kFull, s2, 4));
        s2 = max(s2, __shfl_xor_sync(kFull, s2, 2));
        s2 = max(s2, __shfl_xor_sync(kFull, s2, 1));
        o.score2 = do2 ? s2 : 0;
    }
    return o;
}

template <bool WRAP, bool REV, int SN>
__device__ __forceinline__ PassOut pass_sn(int sn, const LocalArgs &a, const swb_local_task &tk, bool act, int qLen,
                                           int tLen, int minSub, int cap, uint32_t *peaks, uint4 *snap) {
    if constexpr (SN >= 1) {
        if (sn == SN) return striped_pass<SN, WRAP, REV>(a, tk, act, qLen, tLen, minSub, cap, peaks, snap);
        if constexpr (SN != 1 && SN != kSnSplit + 1)
            return pass_sn<WRAP, REV, SN - 1>(sn, a, tk, act, qLen, tLen, minSub, cap, peaks, snap);
    }
    return PassOut{0, -1, -1, 0, true};
}

// One launch per pass and stripe range (1..kSnSplit: HIGH = false, the rest:
// HIGH = true).  The grid is the device's resident blocks; each warp claims
// the next four tasks of one stripe count, longest stripes and targets first,
// so the launch ends with the work rather than on a last wave of fixed slices.
// Five blocks per SM (96 registers): 50k pairs 3.50 ms; four 3.71, six (which
// spill) 3.46, eight 3.85.  The larger stripe counts need four (128).
template <bool WRAP, bool REV, bool HIGH>
__global__ void __launch_bounds__(kLT, HIGH ? 4 : 5) local_striped_kernel(LocalArgs a) {
    __shared__ uint4 snaps[(kMaxSn / 4) * kLT];
    constexpr int kLo = HIGH ? kSnSplit + 1 : 1, kHi = HIGH ? kMaxSn : kSnSplit;
    const int g = (threadIdx.x >> 3) & 3, t = threadIdx.x & 7;
    uint32_t *peaks = a.peaks + ((size_t)blockIdx.x * (kLT / 8) + (threadIdx.x >> 3)) * a.peak_stride;
    unsigned long long cells = 0;
    for (;;) {
        uint32_t u = 0;
        if ((threadIdx.x & 31) == 0) u = atomicAdd(a.claim, 1u);
        u = __shfl_sync(kFull, u, 0);
        int sn = kHi;
        uint32_t lo = 0, hi = 0;
        for (; sn >= kLo; --sn) {                        // the stripe count that holds unit u
            lo = a.bin_start[sn];
            hi = a.bin_start[sn + 1];
            const uint32_t units = (hi - lo + 3) / 4;
            if (u < units) break;
            u -= units;
        }
        if (sn < kLo) break;
        const bool act = 4 * u + g < hi - lo;
        const uint32_t pos = act ? hi - 1 - (4 * u + g) : lo;
        const uint32_t ti = a.order[pos];
        const swb_local_task tk = a.tasks[ti];
        if constexpr (!REV) {
            const PassOut o = pass_sn<WRAP, false, kHi>(sn, a, tk, act, tk.qlen, tk.tlen, clamp_min_sub(tk.min_sub_score),
                                                        0, peaks, snaps + threadIdx.x);
            if (act && t == 0) {
                cells += (unsigned long long)tk.qlen * tk.tlen;
                const int revQ = o.qEnd + 1, revT = o.tEnd + 1;
                uint32_t key = 0;
                if (!o.nil && o.score > 0 && revQ > 0 && revT > 0) {
                    a.out[ti] = swb_local_result{o.score, 0, o.qEnd, 0, o.tEnd, o.score2};
                    // Columns the reverse pass will run: about the hit's length where it can stop there.
                    const bool stops = rev_cap(a.sc, WRAP, revQ, o.score) == o.score;
                    key = ((uint32_t)((revQ + 15) / 16) << 16) | (uint32_t)(stops ? min(revT, revQ + 8) : revT);
                } else {
                    a.fallback[atomicAdd(a.fallback_n, 1u)] = ti;
                }
                a.rkeys[pos] = key;
            }
        } else {
            const swb_local_result r = a.out[ti];
            const int revQ = r.qe + 1, revT = r.te + 1;
            const PassOut o = pass_sn<WRAP, true, kHi>(sn, a, tk, act, revQ, revT, 0, rev_cap(a.sc, WRAP, revQ, r.score),
                                                       nullptr, snaps + threadIdx.x);
            if (act && t == 0) {
                cells += (unsigned long long)revQ * revT;
                if (!o.nil)
                    a.out[ti] = swb_local_result{r.score, r.qe - o.qEnd, r.qe, r.te - o.tEnd, r.te, r.score2};
                else
                    a.fallback[atomicAdd(a.fallback_n, 1u)] = ti;
            }
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) cells += __shfl_down_sync(kFull, cells, o);
    if ((threadIdx.x & 31) == 0 && cells) atomicAdd(a.cells + kCntLocalStriped, cells);
}

// scalarSWPass (:383-492) over spans read through span_base.
struct ScalarPass {
    int score, qEnd, tEnd, score2;
};

__device__ ScalarPass scalar_pass(const LocalArgs &a, const swb_local_task &tk, int qLen, int tLen, bool rev,
                                  int minSub, int *h, int *e, unsigned long long *peaks, size_t stride) {
    const DevScoring &sc = a.sc;
    const int gapOE = sc.o_ins + sc.e_ins, gapE = sc.e_ins;
    for (int j = 0; j <= tLen; ++j) {
        h[(size_t)j * stride] = 0;
        e[(size_t)j * stride] = 0;
    }
    int best = 0, bq = -1, bt = -1;
    const bool trackPeaks = minSub > 0;
    int nPeaks = 0;
    unsigned long long last = 0;
    int maxBase = 0;
    if (trackPeaks) maxBase = max(max((int)(int8_t)sc.a, (int)(int8_t)(-sc.b)), max(-1, 0));
    for (int i = 0; i < qLen; ++i) {
        const uint32_t qb = min(span_base(a.bases, a.pac, tk.q_off, rev ? (qLen - 1 - i) : i, tk.qlen, tk.flags, false), 4u);
        const RowTable rt = row_table(sc, qb);   // mat is symmetric: row q, column t
        int f = 0, hPrev = 0, rowMax = 0;
        for (int j = 0; j < tLen; ++j) {
            const int j1 = j + 1;
            const uint32_t tb = min(span_base(a.bases, a.pac, tk.t_off, rev ? (tLen - 1 - j) : j, tk.tlen, tk.flags, true), 4u);
            int hCur = hPrev + row_score(rt, tb);
            const int hj1 = h[(size_t)j1 * stride];
            const int fOpen = hj1 - gapOE, fExt = f - gapE;
            f = fOpen > fExt ? fOpen : fExt;
            const int eOpen = h[(size_t)j * stride] - gapOE, eExt = e[(size_t)j1 * stride] - gapE;
            const int eVal = eOpen > eExt ? eOpen : eExt;
            e[(size_t)j1 * stride] = eVal;
            hCur = hCur > f ? hCur : f;
            hCur = hCur > eVal ? hCur : eVal;
            hCur = hCur > 0 ? hCur : 0;
            hPrev = hj1;
            h[(size_t)j1 * stride] = hCur;
            if (hCur > rowMax) rowMax = hCur;
            if (hCur > best) {
                best = hCur;
                bq = i;
                bt = j;
            }
        }
        if (trackPeaks && rowMax >= minSub) {
            const unsigned long long rm = (unsigned long long)(uint32_t)rowMax, iu = (unsigned long long)(uint32_t)i;
            if (nPeaks == 0 || (int)(uint32_t)(last & 0xFFFFFFFFull) + 1 != i) {
                last = (rm << 32) | iu;
                peaks[(size_t)nPeaks * stride] = last;
                ++nPeaks;
            } else if ((last >> 32) < rm) {
                last = (rm << 32) | iu;
                peaks[(size_t)(nPeaks - 1) * stride] = last;
            }
        }
    }
    int score2 = 0;
    if (trackPeaks && nPeaks > 0 && best > 0 && maxBase > 0) {
        const int r = (best + maxBase - 1) / maxBase;
        const int low = bq - r, high = bq + r;
        for (int k = 0; k < nPeaks; ++k) {
            const unsigned long long en = peaks[(size_t)k * stride];
            const int col = (int)(uint32_t)(en & 0xFFFFFFFFull), scv = (int)(en >> 32);
            if ((col < low || col > high) && scv > score2) score2 = scv;
        }
    }
    return ScalarPass{best, bq, bt, score2};
}

__global__ void __launch_bounds__(kST) local_scalar_kernel(LocalArgs a, int *hbuf, int *ebuf,
                                                           unsigned long long *pbuf, size_t nslots) {
    const size_t slot = blockIdx.x * (size_t)kST + threadIdx.x;
    const unsigned n = *a.fallback_n;
    unsigned long long cells = 0;
    for (size_t k = slot; k < n; k += nslots) {
        const uint32_t ti = a.fallback[k];
        const swb_local_task tk = a.tasks[ti];
        swb_local_result r{0, 0, 0, 0, 0, 0};
        const int qLen = tk.qlen, tLen = tk.tlen;
        if (qLen > 0 && tLen > 0) {
            const ScalarPass fw = scalar_pass(a, tk, qLen, tLen, false, clamp_min_sub(tk.min_sub_score), hbuf + slot,
                                              ebuf + slot, pbuf + slot, nslots);
            cells += (unsigned long long)qLen * tLen;
            // (the striped pass the reference runs first on what local_keys_kernel sends here directly)
            if (a.sc.a == 0 && qLen > 16 * kMaxSn) cells += (unsigned long long)qLen * tLen;
            if (fw.score > 0) {
                const int rq = fw.qEnd + 1, rt = fw.tEnd + 1;
                const ScalarPass rv = scalar_pass(a, tk, rq, rt, true, 0, hbuf + slot, ebuf + slot, pbuf + slot, nslots);
                cells += (unsigned long long)rq * rt;
                r = swb_local_result{fw.score, fw.qEnd - rv.qEnd, fw.qEnd, fw.tEnd - rv.tEnd, fw.tEnd, fw.score2};
            }
        }
        a.out[ti] = r;
    }
    for (int o = 16; o > 0; o >>= 1) cells += __shfl_down_sync(kFull, cells, o);
    if ((threadIdx.x & 31) == 0 && cells) atomicAdd(a.cells + kCntLocalScalar, cells);
}

// Bin: 0 = scalar (qLen*A > 250 or empty), else the stripe count.
__global__ void local_keys_kernel(const swb_local_task *__restrict__ tasks, size_t n, int a_score,
                                  uint32_t *__restrict__ keys, uint32_t *__restrict__ idx) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const swb_local_task t = tasks[i];
    int bin = 0;
    // (a_score = 0 would allow more stripes than the kernels have: every score
    // is then zero, which ends in the scalar fallback either way.)
    if (t.qlen > 0 && t.tlen > 0 && t.qlen <= 16 * kMaxSn && (long long)t.qlen * a_score <= 250) bin = (t.qlen + 15) / 16;
    keys[i] = ((uint32_t)bin << 16) | (uint32_t)min(max(t.tlen, 0), 0xFFFF);
    idx[i] = (uint32_t)i;
}

// bin_start[b] = first sorted position whose key's bin (key >> shift) is >= b,
// for b up to 17.  scalar: the tasks of bin 0 go straight to the fallback list.
__global__ void local_bounds_kernel(const uint32_t *__restrict__ sorted_keys, const uint32_t *__restrict__ order,
                                    size_t n, int shift, uint32_t *__restrict__ bin_start, bool scalar,
                                    uint32_t *__restrict__ fallback, unsigned int *__restrict__ fallback_n) {
    const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int b = (int)(sorted_keys[p] >> shift);
    const int bprev = p == 0 ? -1 : (int)(sorted_keys[p - 1] >> shift);
    for (int bb = bprev + 1; bb <= b; ++bb) bin_start[bb] = (uint32_t)p;
    if (p == n - 1)
        for (int bb = b + 1; bb <= 17; ++bb) bin_start[bb] = (uint32_t)n;
    if (scalar && b == 0) {
        const unsigned slot = atomicAdd(fallback_n, 1u);
        fallback[slot] = order[p];
    }
}

using StripedKernel = void (*)(LocalArgs);

template <bool REV, bool HIGH>
StripedKernel striped_kernel(bool wrap) {
    return wrap ? local_striped_kernel<true, REV, HIGH> : local_striped_kernel<false, REV, HIGH>;
}

// Launches one pass over one stripe range; *blocks: the grid (its resident
// blocks, fewer for small batches).
int striped_grid(swb_ctx *ctx, StripedKernel k, std::atomic<int> &occ, size_t n, size_t &blocks) {
    if (occ.load(std::memory_order_relaxed) == 0) {
        int b = 0;
        SWB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, kLT, 0));
        occ.store(b > 0 ? b : 1, std::memory_order_relaxed);
    }
    // At most one partly filled unit of four per stripe count.
    const size_t units = n / 4 + std::min<size_t>(n, kMaxSn);
    blocks = std::min((size_t)ctx->sm_count * occ.load(std::memory_order_relaxed), (units + kLT / 32 - 1) / (kLT / 32));
    return SWB_OK;
}

}  // namespace

int launch_local(swb_ctx *ctx, const DevScoring &sc, const uint8_t *d_bases, const swb_local_task *d_tasks,
                 size_t n, swb_local_result *d_out, unsigned long long *d_cells, cudaStream_t st, int max_q,
                 int max_t) {
    if (n == 0) return SWB_OK;
    if (n > 0x7FFFFFF0ull) return set_error(SWB_ERR_TOO_LARGE, "more than 2^31-16 tasks in one batch");
    int rc;
    if ((rc = ensure_dev(ctx, ctx->d_keys, n * 4)) || (rc = ensure_dev(ctx, ctx->d_keys2, n * 4)) ||
        (rc = ensure_dev(ctx, ctx->d_idx, n * 4)) || (rc = ensure_dev(ctx, ctx->d_idx2, n * 8)) ||
        (rc = ensure_dev(ctx, ctx->d_misc, 512)))
        return rc;
    uint32_t *keys = (uint32_t *)ctx->d_keys.p, *keys2 = (uint32_t *)ctx->d_keys2.p;
    uint32_t *idx = (uint32_t *)ctx->d_idx.p, *idx2 = (uint32_t *)ctx->d_idx2.p;
    uint32_t *fallback = idx2 + n;
    uint32_t *bin_start = (uint32_t *)ctx->d_misc.p, *rbin_start = bin_start + 64;   // 18 words each
    unsigned int *fallback_n = (unsigned int *)((char *)ctx->d_misc.p + 128);
    uint32_t *claim = (uint32_t *)((char *)ctx->d_misc.p + 160);   // one counter per striped launch
    SWB_CUDA(cudaMemsetAsync(fallback_n, 0, 64, st));               // fallback count and claim counters
    local_keys_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_tasks, n, sc.a, keys, idx);
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());
    size_t tmp = 0, tmp2 = 0;
    SWB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, keys, keys2, idx, idx2, (int)n, 0, 21, st));
    SWB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp2, keys, keys2, idx2, idx, (int)n, 0, 21, st));
    tmp = std::max(tmp, tmp2);
    if ((rc = ensure_dev(ctx, ctx->d_sort_tmp, tmp))) return rc;
    SWB_CUDA(cub::DeviceRadixSort::SortPairs(ctx->d_sort_tmp.p, tmp, keys, keys2, idx, idx2, (int)n, 0, 21, st));
    local_bounds_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(keys2, idx2, n, 16, bin_start, true, fallback,
                                                                     fallback_n);
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());

    // Stripe ranges that can occur for max_q, and their grids.
    const bool wrap = 250 + std::max(std::max(sc.a, -1), 0) + (sc.b & 0xFF) > 255;   // H + profile byte may pass 255
    static std::atomic<int> occ[2][2][2];   // [wrap][reverse][high] (the same on every sm_100 device)
    const StripedKernel fns[2][2] = {{striped_kernel<false, false>(wrap), striped_kernel<false, true>(wrap)},
                                     {striped_kernel<true, false>(wrap), striped_kernel<true, true>(wrap)}};
    const int ranges = max_q > 16 * kSnSplit ? 2 : 1;
    size_t grid[2][2] = {{0, 0}, {0, 0}}, slots = 1;
    for (int rev = 0; rev < 2; ++rev)
        for (int h = 0; h < ranges; ++h) {
            if ((rc = striped_grid(ctx, fns[rev][h], occ[wrap][rev][h], n, grid[rev][h]))) return rc;
            if (!rev) slots = std::max(slots, grid[rev][h] * (kLT / 8));
        }
    // Peak lists (score2) live in scratch, one window of max_t entries per task in flight.
    const int peak_stride = imax(max_t, 1);
    const size_t nsl = (size_t)ctx->sm_count * 4 * kST;
    const size_t scalar_bytes = nsl * ((size_t)(max_t + 2) * 8 + (size_t)(max_q + 1) * 8);
    const size_t peak_bytes = slots * (size_t)peak_stride * 4;
    if ((rc = ensure_dev(ctx, ctx->d_scratch, peak_bytes + scalar_bytes + 1024))) return rc;
    uint32_t *peaks = (uint32_t *)ctx->d_scratch.p;
    char *sp = (char *)ctx->d_scratch.p + ((peak_bytes + 255) & ~(size_t)255);
    int *hbuf = (int *)sp;
    int *ebuf = hbuf + (size_t)(max_t + 1) * nsl;
    unsigned long long *pbuf = (unsigned long long *)(ebuf + (size_t)(max_t + 1) * nsl);

    // Forward pass; the reverse keys go to `keys` (0 = nothing to do), then
    // the sort by them takes the forward order to the reverse one in `idx`.
    // The striped passes take the gap costs as their bytes hold them (mate rescue
    // allows more than 255), the scalar kernel as they are.
    LocalArgs a{sc, d_bases, ctx->d_pac, d_tasks, d_out, idx2, bin_start, fallback, fallback_n, d_cells, claim,
                keys, peaks, peak_stride};
    a.sc.e_ins = sc.e_ins & 0xFF;
    a.sc.o_ins = ((sc.o_ins + sc.e_ins) & 0xFF) - a.sc.e_ins;
    SWB_CUDA(cudaMemsetAsync(keys, 0, n * 4, st));
    for (int h = ranges - 1; h >= 0; --h) {
        ProfScope ps(ctx, st, "local_striped_fwd", kCntLocalStriped);
        a.claim = claim + h;
        fns[0][h]<<<(unsigned)grid[0][h], kLT, 0, st>>>(a);
        ctx->launches++;
        SWB_CUDA(cudaGetLastError());
    }
    SWB_CUDA(cub::DeviceRadixSort::SortPairs(ctx->d_sort_tmp.p, tmp, keys, keys2, idx2, idx, (int)n, 0, 21, st));
    local_bounds_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(keys2, idx, n, 16, rbin_start, false, nullptr, nullptr);
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());
    a.order = idx;
    a.bin_start = rbin_start;
    for (int h = ranges - 1; h >= 0; --h) {
        ProfScope ps(ctx, st, "local_striped_rev", kCntLocalStriped);
        a.claim = claim + 2 + h;
        fns[1][h]<<<(unsigned)grid[1][h], kLT, 0, st>>>(a);
        ctx->launches++;
        SWB_CUDA(cudaGetLastError());
    }
    {
        a.sc = sc;
        ProfScope ps(ctx, st, "local_scalar_i32", kCntLocalScalar);
        local_scalar_kernel<<<(unsigned)(nsl / kST), kST, 0, st>>>(a, hbuf, ebuf, pbuf, nsl);
    }
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());
    return SWB_OK;
}

}  // namespace swb
