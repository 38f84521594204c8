// swb_seed.cu -- SMEM seeding on the resident FM index, bit-exact with
// SMEMFinder.findAllSMEMs (Sources/FMIndex/SMEMFinder.swift:28-268) over
// BWT.occ (Sources/FMIndex/BWT.swift:68-84) and BackwardSearch.backwardExt
// (Sources/FMIndex/BackwardSearch.swift:21-77).
//
// Eight threads own one read and walk its start positions in the
// reference's order (each start's forward phase decides the next start), so
// the SMEMs, their order and their SA intervals are the reference's.  The
// work is a chain of rank queries into the checkpoint array: random reads
// over the resident index, so the kernel is bound by memory latency.  In the
// forward phase every extension depends on the one before it and the threads
// compute the same one; in the backward phase a row's candidate intervals are
// independent and each thread extends one of them, so a read waits for about
// one extension per forward base and one per eight candidates of a row
// instead of one per candidate.  The walk is a state machine whose every step
// is one round of extensions, so the reads of a warp run their rank queries
// together; a group claims its next read from a counter when its current one
// is done.  A read's candidate list (at most one entry per query base) keeps
// its first kShE entries in shared memory and the rest in the group's own row
// of global scratch.  A read's SMEMs go to its own window in the order found
// and are then sorted there (query begin, longer first), as the reference
// sorts its array; a scan of the counts and a gather pack the windows in read
// order, and only those entries are copied back to the host.
//
// The index is kept in 32-byte blocks (IndexBlock) when its length fits 32
// bits and its bitstrings are one-hot, as every BWT's are: one sector per
// rank query instead of two, half the footprint (100 MB for a 100 Mbp strand
// and its complement, which then fits the L2), and 32-bit interval
// arithmetic.  Otherwise the reference's 64-byte checkpoints are kept.
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <type_traits>

#include "swb_index.h"
#include "swb_internal.h"

namespace swb {
namespace {

constexpr int kSeedT = 128;   // threads per block
constexpr int kGrp = 8;       // threads per read
constexpr int kShE = 32;      // candidate entries per read in shared memory
constexpr unsigned kFullMask = 0xFFFFFFFFu;

// 64 BWT positions: before them, the number of bases >= 1, >= 2 and >= 3
// (C, G or T; G or T; T), and the high and low bits of their base codes (bit
// 63-y for position y; the sentinel's are 0, an A's).
struct __align__(32) IndexBlock {
    uint32_t above[3], unused;
    uint64_t hi, lo;
};

struct SeedArgs {
    const void *index;          // IndexBlock (compact) or swb_bwt_checkpoint (wide)
    int64_t count[5];
    int64_t sentinel;
    const uint8_t *bases;
    const uint64_t *read_off;
    const int32_t *read_len;
    uint32_t n_reads;
    int32_t min_seed_len;
    int64_t min_intv;
    int32_t split_len, split_width;   // internal re-seeding (split_len <= 0: off)
    uint32_t cap;
    swb_smem *out;
    uint32_t *n_out;
    uint32_t *claim;            // next unclaimed position of `order`
    const uint32_t *order;      // reads, tandem repeats (most work) first
    uint32_t *first_over;       // lowest read index with more SMEMs than cap (~0 = none)
    unsigned long long *exts;   // backward extensions (work counter)
    void *cand;                 // candidate entries past the first kShE: [group][entry - kShE]
    size_t entries;
};

// U: the type of BWT positions and interval sizes (uint32_t in the compact
// index, whose length is below 2^32 - 1; int64_t in the wide one).
template <class U>
struct Intv {
    U k, l, s;
};

// Ranks of the four bases before BWT position pos (BWT.occ for c = 0..3).
__device__ __forceinline__ void occ4(const SeedArgs &g, int64_t pos, int64_t o[4]) {
    const longlong2 *p = reinterpret_cast<const longlong2 *>((const swb_bwt_checkpoint *)g.index + (pos >> 6));
    const longlong2 c01 = __ldg(p), c23 = __ldg(p + 1), b01 = __ldg(p + 2), b23 = __ldg(p + 3);
    const int y = (int)(pos & 63);
    const unsigned long long mask = y == 0 ? 0ull : ~(~0ull >> y);   // oneHotMaskArray[y]: the top y bits
    o[0] = c01.x + __popcll((unsigned long long)b01.x & mask);
    o[1] = c01.y + __popcll((unsigned long long)b01.y & mask);
    o[2] = c23.x + __popcll((unsigned long long)b23.x & mask);
    o[3] = c23.y + __popcll((unsigned long long)b23.y & mask);
}

// BackwardSearch.backwardExt: the interval of base a prepended (a < 4).
// Branch-free, so the lanes of a warp stay together: both blocks are read
// even when sp and ep share one (the second read then hits the same cache
// line), and the base selects with conditional moves.
__device__ __forceinline__ Intv<int64_t> backward_ext(const SeedArgs &g, int64_t k, int64_t l, int64_t s, int a) {
    const int64_t sp = k, ep = k + s;
    int64_t osp[4], oep[4];
    occ4(g, sp, osp);
    occ4(g, ep, oep);
    const int64_t s0 = oep[0] - osp[0], s1 = oep[1] - osp[1], s2 = oep[2] - osp[2], s3 = oep[3] - osp[3];
    const int64_t l3 = l + (sp <= g.sentinel && ep > g.sentinel ? 1 : 0), l2 = l3 + s3, l1 = l2 + s2, l0 = l1 + s1;
    const int64_t c = a == 0 ? g.count[0] : a == 1 ? g.count[1] : a == 2 ? g.count[2] : g.count[3];
    const int64_t o = a == 0 ? osp[0] : a == 1 ? osp[1] : a == 2 ? osp[2] : osp[3];
    return {c + o, a == 0 ? l0 : a == 1 ? l1 : a == 2 ? l2 : l3, a == 0 ? s0 : a == 1 ? s1 : a == 2 ? s2 : s3};
}

// Positions before pos holding a base >= a (ge) and > a (gt), the sentinel
// counted as an A.
__device__ __forceinline__ void ranks(const SeedArgs &g, uint32_t pos, int a, uint32_t &ge, uint32_t &gt) {
    const uint4 *p = reinterpret_cast<const uint4 *>((const IndexBlock *)g.index + (pos >> 6));
    const uint4 c = __ldg(p), b = __ldg(p + 1);
    const unsigned long long rest = ~0ull >> (pos & 63u);                  // the positions from pos on
    const uint32_t m0 = ~(uint32_t)rest, m1 = ~(uint32_t)(rest >> 32);
    const uint32_t t1 = c.x + __popc((b.x | b.z) & m0) + __popc((b.y | b.w) & m1);
    const uint32_t t2 = c.y + __popc(b.x & m0) + __popc(b.y & m1);
    const uint32_t t3 = c.z + __popc(b.x & b.z & m0) + __popc(b.y & b.w & m1);
    ge = a == 0 ? pos : a == 1 ? t1 : a == 2 ? t2 : t3;
    gt = a == 0 ? t1 : a == 1 ? t2 : a == 2 ? t3 : 0u;
}

// The same extension from 32-byte blocks: the new interval's k needs the rank
// of a, its size the difference of a's ranks, and its l the bases above a
// (and the sentinel) between sp and ep.
__device__ __forceinline__ Intv<uint32_t> backward_ext(const SeedArgs &g, uint32_t k, uint32_t l, uint32_t s, int a) {
    const uint32_t sp = k, ep = k + s, sent = (uint32_t)g.sentinel;
    uint32_t ge0, gt0, ge1, gt1;
    ranks(g, sp, a, ge0, gt0);
    ranks(g, ep, a, ge1, gt1);
    const uint32_t after0 = sp > sent, after1 = ep > sent;
    const uint32_t o0 = ge0 - gt0 - (a == 0 ? after0 : 0u), o1 = ge1 - gt1 - (a == 0 ? after1 : 0u);
    const uint32_t c = (uint32_t)(a == 0 ? g.count[0] : a == 1 ? g.count[1] : a == 2 ? g.count[2] : g.count[3]);
    return {c + o0, l + (after1 - after0) + (gt1 - gt0), o1 - o0};
}

// Candidate entry (SMEMFinder.BidiInterval without its query begin, which all
// entries of a list share): 16 bytes compact, 32 wide.
struct EntryC {
    uint32_t k, l, s;
    int32_t n;
};
struct EntryW {
    int64_t k, l, s;
    int64_t n;
};

// A group's candidate list: the first kShE entries in shared memory.
template <class E>
struct List {
    E *sh, *row;
    static __device__ __forceinline__ void copy(E *d, const E *x) {
        const uint4 *p = reinterpret_cast<const uint4 *>(x);
        uint4 *q = reinterpret_cast<uint4 *>(d);
        q[0] = p[0];
        if constexpr (sizeof(E) == 32) q[1] = p[1];
    }
    __device__ __forceinline__ E get(int e) const {
        E x;
        if (e < kShE) copy(&x, sh + e);
        else copy(&x, row + (e - kShE));
        return x;
    }
    __device__ __forceinline__ void put(int e, const E &x) const {
        if (e < kShE) copy(sh + e, &x);
        else copy(row + (e - kShE), &x);
    }
};

__device__ __forceinline__ bool smem_before(const swb_smem &x, const swb_smem &y) {   // SMEMFinder.swift:53-58
    return x.qb < y.qb || (x.qb == y.qb && x.qe - x.qb > y.qe - y.qb);
}

// Sorts each group's window (n SMEMs; 0: nothing to do) by query begin, longer
// first; equal keys are equal SMEMs, so their order cannot differ from the
// reference's.  The whole warp calls it.  Up to kGrp SMEMs (nearly every read)
// each thread ranks one of them; more are insertion-sorted by one thread.
__device__ __forceinline__ void sort_smems(swb_smem *w, uint32_t n, int gl, int gbase) {
    const uint32_t ns = n <= (uint32_t)kGrp ? n : 0u;
    swb_smem x{};
    if ((uint32_t)gl < ns) x = w[gl];
    uint32_t rank = 0;
    for (int i = 0; i < kGrp; ++i) {
        swb_smem y;
        y.qb = __shfl_sync(kFullMask, x.qb, gbase + i);
        y.qe = __shfl_sync(kFullMask, x.qe, gbase + i);
        if ((uint32_t)i < ns && (smem_before(y, x) || (!smem_before(x, y) && i < gl))) ++rank;
    }
    if ((uint32_t)gl < ns) w[rank] = x;
    if (n > (uint32_t)kGrp && gl == 0) {
        for (uint32_t i = 1; i < n; ++i) {
            const swb_smem v = w[i];
            uint32_t j = i;
            while (j > 0 && smem_before(v, w[j - 1])) {
                w[j] = w[j - 1];
                --j;
            }
            w[j] = v;
        }
    }
    __syncwarp();
}

// SMEMFinder.findAllSMEMs for one read (SMEMFinder.swift:28-59; its
// findSMEMsAtPosition calls :89-268) followed by the internal re-seeding of
// BWAMemAligner (BWAMemAligner.swift:283-304), written as a state machine in
// which every step is one round of backward extensions.  The kernel runs the
// round and the two common outcomes (the next forward base, the next round or
// row of a backward phase) for all groups of the warp together, then the other
// transitions, which need no extension.  Everything but the thread's
// own candidate is the same in all threads of the group.
template <class U>
struct Walker {
    using E = typename std::conditional<sizeof(U) == 4, EntryC, EntryW>::type;
    // Below kRound: a transition is due.  kRound: a round is set up.  kNone: no read left.
    enum State : int { kSort, kClaim, kFwdEnd, kRow, kBwdDone, kNext, kRound, kNone };
    const uint8_t *q;
    int len;
    State st;
    bool fwd;             // the round is a forward step, else one of a backward row
    bool reseed;          // in the re-seeding pass (the first pass is sorted)
    bool phase2;          // backward row: past the first kept or emitted interval
    bool has_last;        // backward row: an earlier round had an interval of at least minIntv, of size last_s
    bool valid;           // backward row: this thread has a candidate in the round
    uint32_t r;           // the read
    int pos;              // first pass: the next start position
    uint32_t ri, n0;      // re-seeding: the next original SMEM, the originals' count
    U minIntv;            // of the current findSMEMsAtPosition call
    int startPos, nextPos, j, bj, p, numPrev, numCurr;
    int top;              // backward phase: entry p sits at list position top - p (:166: longest first)
    int m;                // query begin of the list's entries
    int nb;               // the query base after the round's: at j + 1, or at bj - 1 (4: none)
    U last_s;
    // The round's extension: interval and base.  A forward extension is a
    // backward one with k and l swapped and the complement base, so its
    // interval is held swapped (xk = l, xl = k).
    U xk, xl, xs;
    int xn, a;            // query end of the interval (inclusive)
    swb_smem *w;          // the read's window
    uint32_t n;           // its SMEMs so far

    // A threshold on interval sizes as U (sizes are in [0, length]).
    static __device__ __forceinline__ U threshold(int64_t v) {
        if constexpr (sizeof(U) == 4) return v < 0 ? 0u : v > 0xFFFFFFFFll ? 0xFFFFFFFFu : (U)v;
        else return v;
    }
    __device__ __forceinline__ int base(int x) const { return (unsigned)x < (unsigned)len ? q[x] : 4; }
    // Takes the read at position c of the claim order, if there is one.
    __device__ __forceinline__ void start(const SeedArgs &g, uint32_t c) {
        xk = xl = xs = 0;
        a = 0;
        valid = false;
        st = kNone;
        if (c >= g.n_reads) return;
        r = g.order[c];
        q = g.bases + g.read_off[r];
        len = g.read_len[r];
        st = kNext;
        reseed = false;
        pos = 0;
        w = g.out + (size_t)r * g.cap;
        n = 0;
    }
    __device__ __forceinline__ void emit(const SeedArgs &g, U k, U s, int qe, bool mine) {
        if (mine && n < g.cap) w[n] = swb_smem{(int64_t)k, (int64_t)k + (int64_t)s - 1, m, qe + 1};
        ++n;
    }
    // This thread's candidate of the round at p (its list is complete and visible).
    __device__ __forceinline__ void load_round(const List<E> &prev, int gl) {
        valid = p + gl < numPrev;
        xk = xl = xs = 0;
        if (valid) {
            const E e = prev.get(top - (p + gl));
            xk = e.k;
            xl = e.l;
            xs = e.s;
            xn = (int)e.n;
        }
    }
    __device__ __forceinline__ void begin_row() {
        p = 0;
        numCurr = 0;
        has_last = false;
        phase2 = false;
    }
    // One findSMEMsAtPosition call up to its first extension (:89-123).
    __device__ __forceinline__ void call(const SeedArgs &g, int sp, int64_t mi) {
        startPos = sp;
        minIntv = threshold(mi);
        nextPos = sp + 1;
        const int c = q[sp];
        if (c >= 4) {                                                        // :104-107
            if (!reseed) pos = nextPos;
            return;
        }
        xk = (U)g.count[3 - c];
        xl = (U)g.count[c];
        xs = (U)(g.count[c + 1] - g.count[c]);
        xn = sp;
        numPrev = 0;
        j = sp + 1;
        const int b = base(j);
        if (b >= 4) {
            if (j < len) nextPos = j + 1;
            st = kFwdEnd;
            return;
        }
        a = 3 - b;
        nb = base(j + 1);
        fwd = true;
        st = kRound;
    }
    // The end of a forward phase (:160-166); its candidates are read after a __syncwarp.
    __device__ __forceinline__ void fwd_end(const List<E> &prev, int gl) {
        if (xs >= minIntv) {
            E c;
            c.k = xl;
            c.l = xk;
            c.s = xs;
            c.n = xn;
            if (gl == 0) prev.put(numPrev, c);
            ++numPrev;
        }
        top = numPrev - 1;
        m = startPos;
        bj = startPos - 1;
        a = base(bj);
        nb = base(bj - 1);
        fwd = false;
        begin_row();
        st = a >= 4 || numPrev == 0 ? kBwdDone : kRow;
    }
    // The end of a call (:253-265) and the next one.
    __device__ __forceinline__ void next_call(const SeedArgs &g, const List<E> &prev, int gl) {
        if (st == kBwdDone) {
            if (numPrev != 0) {
                const E c = prev.get(top);
                if (((int)c.n - m + 1) >= g.min_seed_len) emit(g, c.k, c.s, (int)c.n, gl == 0);
            }
            if (!reseed) pos = nextPos;                                      // :41-51
            st = kNext;
        }
        if (!reseed) {
            if (pos < len) call(g, pos, g.min_intv);                         // :41-51
            else st = n <= g.cap ? kSort : kClaim;                           // :53-58; an overflowed window ends here
        } else {
            // Re-seeding: the first-pass SMEMs (w[0 .. n0), never overwritten:
            // new ones are appended behind them) that are long and rare enough.
            bool found = false;
            while (ri < n0 && !found) {
                const swb_smem sm = w[ri++];
                const int64_t cnt = sm.l - sm.k + 1;
                found = sm.qe - sm.qb >= g.split_len && cnt <= (int64_t)g.split_width;
                if (found) call(g, (sm.qb + sm.qe) / 2, cnt + 1);
            }
            if (!found) st = n > n0 && n <= g.cap ? kSort : kClaim;
        }
    }
};

// A read is a chain of about 240 dependent rounds (150 bp reads), each a
// random read of the index, so the kernel lives on many reads in flight and
// few instructions per round.  One thread per read needs 540 rounds on average
// and 7,000 for the worst tandem-repeat read, which alone held a 100k-read
// call at 12.8 ms; eight threads need 240 and 1,150.  Kernel time on a 100 Mbp
// index, 100k reads 12.8 -> 2.74 ms, 1M reads 39.9 -> 23.8 ms (four threads a
// read: 3.45 ms per 100k, sixteen: 3.77; ten blocks per SM 3.13, six 2.90).
// Bound by instruction issue (about 320 a round, 77 % of the issue slots).
// Control flow is uniform over the warp outside of short branches without
// synchronisation, so that its groups stay together (with a transition loop
// per group they ran the extension apart, 13.8 threads an instruction, 6.2 ms).
template <class U>
__global__ void __launch_bounds__(kSeedT, sizeof(U) == 4 ? 8 : 5) smem_kernel(const __grid_constant__ SeedArgs g) {
    using W = Walker<U>;
    using E = typename W::E;
    __shared__ __align__(16) E sh[(kSeedT / kGrp) * kShE];
    const int lane = threadIdx.x & 31, gl = lane & (kGrp - 1), gbase = lane & ~(kGrp - 1);
    const unsigned gm = (1u << kGrp) - 1u, lower = (1u << gl) - 1u;
    const size_t group = (size_t)blockIdx.x * (kSeedT / kGrp) + threadIdx.x / kGrp;
    const List<E> prev{sh + (threadIdx.x / kGrp) * kShE, (E *)g.cand + group * g.entries};
    uint32_t exts = 0;
    W w;
    w.st = W::kClaim;
    bool first_claim = true;
    for (;;) {
        // Transitions, until every group has a round or no read is left.
        if (__any_sync(kFullMask, w.st < W::kRound)) {
            do {
                if (__any_sync(kFullMask, w.st <= W::kClaim)) {
                    if (__any_sync(kFullMask, w.st == W::kSort)) {
                        const bool so = w.st == W::kSort;
                        sort_smems(w.w, so ? w.n : 0u, gl, gbase);
                        if (so) {
                            w.st = W::kClaim;
                            if (!w.reseed && g.split_len > 0) {
                                w.n0 = w.n;
                                w.ri = 0;
                                w.reseed = true;
                                w.st = W::kNext;
                            }
                        }
                    }
                    // Each group claims its next read as soon as its current one is done.
                    uint32_t c = 0;
                    if (w.st == W::kClaim && gl == 0) {
                        if (!first_claim) {
                            g.n_out[w.r] = w.n;
                            if (w.n > g.cap) atomicMin(g.first_over, w.r);
                        }
                        c = atomicAdd(g.claim, 1u);
                    }
                    c = __shfl_sync(kFullMask, c, gbase);
                    if (w.st == W::kClaim) w.start(g, c);
                    first_claim = false;
                }
                if (w.st == W::kBwdDone || w.st == W::kNext) w.next_call(g, prev, gl);
                if (w.st == W::kFwdEnd) w.fwd_end(prev, gl);
                __syncwarp();
                if (w.st == W::kRow) {
                    w.load_round(prev, gl);
                    w.st = W::kRound;
                }
            } while (__any_sync(kFullMask, w.st < W::kRound));
            if (!__any_sync(kFullMask, w.st == W::kRound)) break;
        }
        const Intv<U> ext = backward_ext(g, w.xk, w.xl, w.xs, w.a);
        const bool have = w.st == W::kRound, fwd = have && w.fwd, bwd = have && !w.fwd;
        const bool at_min = ext.s >= w.minIntv;
        // A round of a backward row (:177-246): among the row's candidates in
        // order, the first that is long enough but falls below minIntv
        // (emitted) or stays at minIntv (kept) decides phase2; then every one
        // of at least minIntv whose size differs from the last kept one's --
        // that is, from the previous one of at least minIntv -- is kept.
        const bool elig = bwd && w.valid && at_min;
        const bool over = bwd && w.valid && !at_min && (w.xn - w.m + 1) >= g.min_seed_len;
        const unsigned be = (__ballot_sync(kFullMask, elig) >> gbase) & gm;
        const unsigned bo = (__ballot_sync(kFullMask, over) >> gbase) & gm;
        const unsigned below = be & lower;
        const U s_prev = __shfl_sync(kFullMask, ext.s, gbase + (below ? 31 - __clz(below) : 0));
        const U s_last = __shfl_sync(kFullMask, ext.s, gbase + (be ? 31 - __clz(be) : 0));
        const bool same = below ? s_prev == ext.s : (w.has_last && w.last_s == ext.s);
        const bool kept = elig && !same;
        const unsigned bk = (__ballot_sync(kFullMask, kept) >> gbase) & gm;
        // What goes to the list: a kept candidate, or the forward interval
        // whose size the extension changed.
        const bool push = fwd && ext.s != w.xs;
        if (kept || (push && gl == 0)) {
            E x;
            x.k = fwd ? w.xl : ext.k;
            x.l = fwd ? w.xk : ext.l;
            x.s = fwd ? w.xs : ext.s;
            x.n = w.xn;
            prev.put(fwd ? w.numPrev : w.top - (w.numCurr + __popc(bk & lower)), x);
        }
        __syncwarp();
        if (fwd) {                                                           // :124-157
            w.numPrev += push ? 1 : 0;
            exts += gl == 0 ? 1 : 0;
            w.nextPos = w.j;
            if (at_min) {
                w.xk = ext.k;
                w.xl = ext.l;
                w.xs = ext.s;
                w.xn = w.j;
                ++w.j;
                w.nextPos = w.nb >= 4 && w.j < w.len ? w.j + 1 : w.j;        // N, or past the read
                w.a = 3 - w.nb;
            }
            if (!at_min || w.nb >= 4) w.st = W::kFwdEnd;
            w.nb = w.base(w.j + 1);   // for the next step, loaded while this one's extension waits
        }
        if (bwd) {
            exts += w.valid ? 1 : 0;
            if (!w.phase2 && (be | bo)) {
                const int first = __ffs(be | bo) - 1;
                if ((bo >> first) & 1u) w.emit(g, w.xk, w.xs, w.xn, gl == first);
                w.phase2 = true;
            }
            if (be) {
                w.has_last = true;
                w.last_s = s_last;
            }
            w.numCurr += __popc(bk);
            w.p += kGrp;
            if (w.p >= w.numPrev) {                                          // :248-249, the next row
                w.numPrev = w.numCurr;
                w.m = w.bj;
                if (w.numCurr == 0 || w.nb >= 4) w.st = W::kBwdDone;
                --w.bj;
                w.a = w.nb;
                w.nb = w.base(w.bj - 1);
                w.begin_row();
            }
            w.load_round(prev, gl);
        }
        __syncwarp();
    }
    unsigned long long sum = exts;
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(kFullMask, sum, o);
    if (lane == 0 && sum) atomicAdd(g.exts, sum);
}

// Claim order: reads of low complexity -- tandem repeats, whose SA intervals
// stay large and whose walks take many more extensions -- first, the others
// after them, so the launch ends on cheap reads.  A read is one when it has
// fewer than half of the distinct 3-mers it could have (of at most 64): 150
// random bases have 58, a tandem repeat with 1 % errors about 13.  Eight
// threads per read; the order within either part does not matter.
__global__ void seed_order_kernel(const uint8_t *__restrict__ bases, const uint64_t *__restrict__ read_off,
                                  const int32_t *__restrict__ read_len, uint32_t n_reads, uint32_t *__restrict__ fill,
                                  uint32_t *__restrict__ order) {
    const uint32_t r = (uint32_t)group_item(blockIdx.x, blockDim.x, threadIdx.x, kGrp);
    const int lane = threadIdx.x & 31, gl = lane & (kGrp - 1);
    unsigned long long seen = 0;
    int len = 0;
    if (r < n_reads) {
        const uint8_t *q = bases + read_off[r];
        len = read_len[r];
        for (int j = gl; j + 2 < len; j += kGrp) {
            const uint32_t a = q[j], b = q[j + 1], c = q[j + 2];
            if ((a | b | c) < 4) seen |= 1ull << (a * 16 + b * 4 + c);
        }
    }
    for (int o = kGrp / 2; o > 0; o >>= 1) seen |= __shfl_xor_sync(kFullMask, seen, o);
    const bool mine = gl == 0 && r < n_reads;
    const bool heavy = mine && 2 * __popcll(seen) < min(len - 2, 64);
    for (int part = 0; part < 2; ++part) {
        const bool in = mine && heavy == (part == 0);
        const unsigned m = __ballot_sync(kFullMask, in);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(fill + part, (uint32_t)__popc(m));
        at = __shfl_sync(kFullMask, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (in) order[part == 0 ? at : n_reads - 1 - at] = r;
    }
}

// 32-byte blocks of checkpoints [first, first + n) of the index; *bad is set
// when one cannot be kept that way: a count beyond 32 bits, counts that do not
// add up to the positions before the block, a position below `length` in no
// or several bitstrings, or a base at the sentinel.
__global__ void bwt_compact_kernel(const swb_bwt_checkpoint *__restrict__ cp, uint64_t first, uint64_t n,
                                   int64_t length, int64_t sentinel, IndexBlock *__restrict__ out,
                                   uint32_t *__restrict__ bad) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const swb_bwt_checkpoint c = cp[i];
    const uint64_t b = first + i;
    const int64_t left = length - (int64_t)(b << 6);          // positions of this block below length
    uint64_t want = left >= 64 ? ~0ull : left <= 0 ? 0ull : ~(~0ull >> left);
    const uint64_t sent = (uint64_t)(sentinel >> 6) == b ? 1ull << (63 - (sentinel & 63)) : 0ull;
    want &= ~sent;
    const uint64_t any = c.bits[0] | c.bits[1] | c.bits[2] | c.bits[3];
    const int sum = __popcll(c.bits[0]) + __popcll(c.bits[1]) + __popcll(c.bits[2]) + __popcll(c.bits[3]);
    bool ok = (any & want) == want && !(any & sent) && sum == __popcll(any);
    IndexBlock o;
    int64_t sum_above = 0;
    for (int x = 3; x >= 0; --x) {
        ok = ok && c.counts[x] >= 0 && c.counts[x] <= 0xFFFFFFFFll;
        sum_above += c.counts[x];
        if (x > 0) o.above[x - 1] = (uint32_t)sum_above;
    }
    o.unused = 0;
    // The A count is not kept: it is what is left of the positions before the block.
    ok = ok && sum_above == (int64_t)(b << 6) - (sentinel < (int64_t)(b << 6) ? 1 : 0);
    if (b > (uint64_t)(length >> 6)) ok = true;               // never read
    o.hi = c.bits[2] | c.bits[3];
    o.lo = c.bits[1] | c.bits[3];
    out[b] = o;
    if (!ok) atomicExch(bad, 1u);
}

// Packs every read's window into the output in read order: read r's first
// min(n[r], cap) SMEMs go to off[r] (off = exclusive sum of n).
__global__ void smem_pack_kernel(const swb_smem *__restrict__ win, const uint32_t *__restrict__ n,
                                 const unsigned long long *__restrict__ off, uint32_t n_reads, uint32_t cap,
                                 swb_smem *__restrict__ out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_reads) return;
    const uint32_t k = min(n[r], cap);
    const swb_smem *src = win + (size_t)r * cap;
    swb_smem *dst = out + off[r];
    for (uint32_t i = 0; i < k; ++i) dst[i] = src[i];
}

__global__ void u32_to_u64_kernel(const uint32_t *__restrict__ a, unsigned long long *__restrict__ b, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

}  // namespace
}  // namespace swb

using namespace swb;

namespace {

// Uploads the index as 32-byte blocks, the checkpoints passing through a
// chunk buffer that is freed again (the two together take the size of the
// 64-byte checkpoints and up to 288 bytes).  compact = false: the index or the
// budget does not allow it, nothing was kept.
int upload_compact(swb_ctx *ctx, const swb_bwt_checkpoint *cp, uint64_t n_cp, int64_t length, int64_t sentinel,
                   bool &compact) {
    compact = false;
    if (length >= 0xFFFFFFFFll || n_cp > 0xFFFFFFFFull) return SWB_OK;
    const uint64_t chunk = std::min<uint64_t>((n_cp + 1) / 2, 1u << 20);
    const size_t chunk_bytes = chunk * sizeof(swb_bwt_checkpoint) + 256;
    if (ensure_dev(ctx, ctx->d_bwt, n_cp * sizeof(IndexBlock)) != SWB_OK) return SWB_OK;
    if (ctx->allocated + chunk_bytes > ctx->budget) return SWB_OK;
    char *tmp = nullptr;
    if (cudaMalloc(&tmp, chunk_bytes) != cudaSuccess) {
        cudaGetLastError();
        return SWB_OK;
    }
    swb_bwt_checkpoint *d_cp = (swb_bwt_checkpoint *)tmp;
    uint32_t *d_bad = (uint32_t *)(tmp + chunk * sizeof(swb_bwt_checkpoint)), bad = 0;
    cudaError_t e = cudaMemsetAsync(d_bad, 0, 4, ctx->stream);
    for (uint64_t lo = 0; lo < n_cp && e == cudaSuccess; lo += chunk) {
        const uint64_t n = std::min(chunk, n_cp - lo);
        e = cudaMemcpyAsync(d_cp, cp + lo, n * sizeof(swb_bwt_checkpoint), cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) break;
        bwt_compact_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d_cp, lo, n, length, sentinel,
                                                                                (IndexBlock *)ctx->d_bwt.p, d_bad);
        ctx->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, 4, cudaMemcpyDeviceToHost, ctx->stream);
    const cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
    cudaFree(tmp);
    if (e != cudaSuccess || e2 != cudaSuccess) return check_cuda(e != cudaSuccess ? e : e2, "index upload");
    compact = bad == 0;
    return SWB_OK;
}

}  // namespace

extern "C" {

int swb_upload_bwt(swb_ctx *ctx, const swb_bwt_checkpoint *cp, uint64_t n_cp, const int64_t count[5], int64_t length,
                   int64_t sentinel) {
    if (!ctx || !count || (!cp && n_cp)) return set_error(SWB_ERR_INVALID_ARG, "NULL argument");
    if (length < 1 || n_cp < (uint64_t)(length >> 6) + 1 || sentinel < 0 || sentinel >= length || count[4] != length)
        return set_error(SWB_ERR_INVALID_ARG, "BWT: need length >= 1, (length >> 6) + 1 checkpoints, "
                                              "0 <= sentinel < length and count[4] == length");
    for (int c = 0; c < 4; ++c)
        if (count[c] < 0 || count[c] > count[c + 1]) return set_error(SWB_ERR_INVALID_ARG, "BWT: counts must ascend");
    std::lock_guard<std::mutex> lk(ctx->mu);
    SWB_CUDA(cudaSetDevice(ctx->device));
    // An index is accepted when the budget holds its 64-byte form, which either
    // form may need; a refused one leaves the index held so far alone.  From
    // here on that one is lost (its buffer is freed or overwritten), so no
    // later failure may leave it marked as there.
    const size_t wide = n_cp * sizeof(swb_bwt_checkpoint), others = ctx->allocated - ctx->d_bwt.cap;
    if (n_cp > SIZE_MAX / (2 * sizeof(swb_bwt_checkpoint)) || others + ((wide + 4095) & ~(size_t)4095) > ctx->budget)
        return set_error(SWB_ERR_OOM, "device memory budget exceeded (index of " + std::to_string(n_cp) + " checkpoints)");
    ctx->bwt_ncp = 0;
    int rc;
    bool compact = false;
    if ((rc = upload_compact(ctx, cp, n_cp, length, sentinel, compact))) return rc;
    if (!compact) {
        if ((rc = ensure_dev(ctx, ctx->d_bwt, wide))) return rc;
        SWB_CUDA(cudaMemcpy(ctx->d_bwt.p, cp, n_cp * sizeof(swb_bwt_checkpoint), cudaMemcpyHostToDevice));
    }
    ctx->bwt_compact = compact;
    for (int c = 0; c < 5; ++c) ctx->bwt_count[c] = count[c];
    ctx->bwt_length = length;
    ctx->bwt_sentinel = sentinel;
    ctx->bwt_ncp = n_cp;
    return SWB_OK;
}

int swb_smem_batch(swb_ctx *ctx, const uint8_t *bases, size_t n_bases, const uint64_t *read_off,
                   const int32_t *read_len, size_t n_reads, int32_t min_seed_len, int64_t min_intv,
                   int32_t split_len, int32_t split_width, uint32_t cap_per_read, swb_smem *out, size_t out_cap,
                   uint32_t *n_out, uint64_t *out_off) {
    if (!ctx || (n_reads && (!read_off || !read_len || !n_out || !out_off)) || (!out && out_cap) ||
        (!bases && n_bases))
        return set_error(SWB_ERR_INVALID_ARG, "NULL argument");
    // The offsets' scan takes int counts.
    if (n_reads > 0x7FFFFFF0ull) return set_error(SWB_ERR_TOO_LARGE, "more than 2^31-16 reads in one batch");
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->last_ms = 0;
    ctx->last_cells = 0;
    if (n_reads == 0) return SWB_OK;
    if (ctx->bwt_ncp == 0) return set_error(SWB_ERR_NO_REFERENCE, "no FM index uploaded (swb_upload_bwt)");
    int max_len = 0;
    for (size_t r = 0; r < n_reads; ++r) {
        if (read_len[r] < 0 || read_len[r] > kMaxLen)
            return set_error(SWB_ERR_TOO_LARGE, "read " + std::to_string(r) + ": length outside 0..65535");
        if (read_off[r] + (uint64_t)read_len[r] > n_bases)
            return set_error(SWB_ERR_INVALID_ARG, "read " + std::to_string(r) + ": span outside the bases buffer");
        max_len = std::max(max_len, read_len[r]);
    }
    SWB_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t b_bytes = al(n_bases), o_bytes = al(n_reads * 8), l_bytes = al(n_reads * 4);
    const size_t out_bytes = al(n_reads * (size_t)cap_per_read * sizeof(swb_smem)), n_bytes = al(n_reads * 4);
    const size_t off_bytes = al(n_reads * 8);
    size_t scan_bytes = 0;
    SWB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (unsigned long long *)nullptr,
                                           (unsigned long long *)nullptr, (int)n_reads, ctx->stream));
    int rc;
    if ((rc = work_acquire(ctx, st)) || (rc = ensure_dev(ctx, ctx->d_idx, n_reads * 4))) return rc;
    if ((rc = ensure_dev(ctx, ctx->d_bases, b_bytes + o_bytes + l_bytes + 256)) ||
        (rc = ensure_dev(ctx, ctx->d_out, out_bytes + n_bytes + 2 * off_bytes + al(scan_bytes) + 256)))
        return rc;
    char *in = (char *)ctx->d_bases.p;
    uint8_t *d_b = (uint8_t *)in;
    uint64_t *d_off = (uint64_t *)(in + b_bytes);
    int32_t *d_len = (int32_t *)(in + b_bytes + o_bytes);
    uint32_t *d_misc = (uint32_t *)(in + b_bytes + o_bytes + l_bytes);   // claim, order fill (2), first_over
    swb_smem *d_out = (swb_smem *)ctx->d_out.p;
    uint32_t *d_n = (uint32_t *)((char *)ctx->d_out.p + out_bytes);
    unsigned long long *d_n64 = (unsigned long long *)((char *)ctx->d_out.p + out_bytes + n_bytes);
    unsigned long long *d_off64 = d_n64 + off_bytes / 8;
    void *d_scan_tmp = (char *)ctx->d_out.p + out_bytes + n_bytes + 2 * off_bytes;
    // Persistent grid: resident blocks on every SM, each group of kGrp threads
    // with a candidate row of max_len entries past the kShE it keeps in
    // shared memory.
    const bool compact = ctx->bwt_compact;
    int per_sm = 0;
    if (compact) SWB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, smem_kernel<uint32_t>, kSeedT, 0));
    else SWB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, smem_kernel<int64_t>, kSeedT, 0));
    per_sm = std::max(per_sm, 1);
    constexpr size_t kGroups = kSeedT / kGrp;   // per block
    size_t blocks = std::min<size_t>((size_t)ctx->sm_count * per_sm, (n_reads + kGroups - 1) / kGroups);
    const size_t entries = (size_t)std::max(max_len - kShE, 1);
    const size_t per_slot = entries * (compact ? sizeof(EntryC) : sizeof(EntryW));
    const size_t avail = ctx->budget > ctx->allocated ? (ctx->budget - ctx->allocated) / 2 : 0;
    while (blocks > 1 && blocks * kGroups * per_slot > avail) blocks /= 2;
    const size_t nslots = blocks * kGroups;
    if ((rc = ensure_dev(ctx, ctx->d_seed, nslots * per_slot + 256))) return rc;
    char *sp = (char *)ctx->d_seed.p;
    SeedArgs g{};
    g.index = ctx->d_bwt.p;
    for (int c = 0; c < 5; ++c) g.count[c] = ctx->bwt_count[c];
    g.sentinel = ctx->bwt_sentinel;
    g.bases = d_b;
    g.read_off = d_off;
    g.read_len = d_len;
    g.n_reads = (uint32_t)n_reads;
    g.min_seed_len = min_seed_len;
    g.min_intv = min_intv;
    g.split_len = split_len;
    g.split_width = split_width;
    g.cap = cap_per_read;
    g.out = d_out;
    g.n_out = d_n;
    g.claim = d_misc;
    g.first_over = d_misc + 3;
    g.cand = sp;
    g.entries = entries;
    // Inputs: straight from the caller's buffers when all three are pinned,
    // else through the context's pinned staging buffer in the device layout
    // (host threads copy, then one transfer).
    if (is_pinned(bases) && is_pinned(read_off) && is_pinned(read_len)) {
        SWB_CUDA(cudaMemcpyAsync(in, bases, n_bases, cudaMemcpyHostToDevice, st));
        SWB_CUDA(cudaMemcpyAsync(in + b_bytes, read_off, n_reads * 8, cudaMemcpyHostToDevice, st));
        SWB_CUDA(cudaMemcpyAsync(in + b_bytes + o_bytes, read_len, n_reads * 4, cudaMemcpyHostToDevice, st));
    } else {
        if ((rc = ensure_host(ctx, ctx->h_in, b_bytes + o_bytes + l_bytes))) return rc;
        char *stage = (char *)ctx->h_in.p;
        par_copy(stage, bases, n_bases);
        par_copy(stage + b_bytes, read_off, n_reads * 8);
        par_copy(stage + b_bytes + o_bytes, read_len, n_reads * 4);
        SWB_CUDA(cudaMemcpyAsync(in, stage, b_bytes + o_bytes + l_bytes, cudaMemcpyHostToDevice, st));
    }
    SWB_CUDA(cudaMemsetAsync(d_misc, 0, 12, st));
    SWB_CUDA(cudaMemsetAsync(d_misc + 3, 0xFF, 4, st));
    SWB_CUDA(cudaMemsetAsync(ctx->d_counters, 0, sizeof(unsigned long long) * kNumCounters, st));
    g.exts = ctx->d_counters + kCntSeed;
    SWB_CUDA(cudaEventRecord(ctx->ev_start, st));
    {
        ProfScope ps(ctx, st, "seed_order", -1);
        uint32_t *order = (uint32_t *)ctx->d_idx.p;
        const unsigned ob = 256, per = ob / kGrp;
        seed_order_kernel<<<(unsigned)((n_reads + per - 1) / per), ob, 0, st>>>(d_b, d_off, d_len, (uint32_t)n_reads,
                                                                               d_misc + 1, order);
        ctx->launches++;
        SWB_CUDA(cudaGetLastError());
        g.order = order;
    }
    {
        ProfScope ps(ctx, st, compact ? "smem_search" : "smem_search_cp64", kCntSeed);
        if (compact) smem_kernel<uint32_t><<<(unsigned)blocks, kSeedT, 0, st>>>(g);
        else smem_kernel<int64_t><<<(unsigned)blocks, kSeedT, 0, st>>>(g);
    }
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());
    SWB_CUDA(cudaEventRecord(ctx->ev_stop, st));
    // Offsets: the running sum of every read's full count.
    const unsigned cb = 256, cg = (unsigned)((n_reads + cb - 1) / cb);
    u32_to_u64_kernel<<<cg, cb, 0, st>>>(d_n, d_n64, (uint32_t)n_reads);
    ctx->launches++;
    SWB_CUDA(cudaGetLastError());
    SWB_CUDA(cub::DeviceScan::ExclusiveSum(d_scan_tmp, scan_bytes, d_n64, d_off64, (int)n_reads, st));
    uint32_t first_over = 0;
    if ((rc = d2h_staged(ctx, st, {DevSpan{d_n, n_out, n_reads * 4}, DevSpan{d_off64, out_off, n_reads * 8},
                                   DevSpan{d_misc + 3, &first_over, 4}})))
        return rc;
    const uint64_t total = out_off[n_reads - 1] + n_out[n_reads - 1];
    if (total > out_cap)
        return set_error(SWB_ERR_TOO_LARGE, std::to_string(total) + " SMEMs, more than out_cap (" +
                                                std::to_string(out_cap) + ")");
    if (total) {
        // Pack the windows in read order, then copy just those entries back.
        if ((rc = ensure_dev(ctx, ctx->d_aux, total * sizeof(swb_smem)))) return rc;
        swb_smem *d_pack = (swb_smem *)ctx->d_aux.p;
        smem_pack_kernel<<<cg, cb, 0, st>>>(d_out, d_n, d_off64, (uint32_t)n_reads, cap_per_read, d_pack);
        ctx->launches++;
        SWB_CUDA(cudaGetLastError());
        if ((rc = d2h_staged(ctx, st, {DevSpan{d_pack, out, total * sizeof(swb_smem)}}))) return rc;
    }
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop) == cudaSuccess) ctx->last_ms = ms;
    unsigned long long exts = 0;
    if (cudaMemcpy(&exts, ctx->d_counters + kCntSeed, sizeof(exts), cudaMemcpyDeviceToHost) == cudaSuccess)
        ctx->last_cells = exts;
    if (first_over != 0xFFFFFFFFu)
        return set_error(SWB_ERR_TOO_LARGE, "read " + std::to_string(first_over) + ": " +
                                                std::to_string(n_out[first_over]) + " SMEMs, more than cap_per_read (" +
                                                std::to_string(cap_per_read) + ")");
    return SWB_OK;
}

}  // extern "C"
