// k_check.cu -- the exact smallest Goldbach prime p(n) of every even.
//
// The reference computes it on sampled segments (check30_xs* + check30_xb,
// goldbach.cl:2339-2418, 2880-3021), testing candidates over words of 32
// evens; here an even finds its smallest candidate in one or two 64-bit
// windows of the map (k_check below). Evens left without a witness <= 9781
// go to a list that k_retry settles on the GPU (the reference's CPU fallback
// cpu_min_goldbach_prime, src/primes.cpp:482-493, moved on device).
//
// Every kernel here is persistent: a fixed grid takes the "virtual CTAs"
// of all segments of the batch (per segment: vbx CTAs) from a
// work counter, each found through the batch descriptor's prefix arrays.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <utility>

#include "gbc_common.cuh"

namespace gbk {

__device__ __forceinline__ void append_leftover(gbc_segment_result *res, uint64_t n)
{
    const uint32_t slot = atomicAdd(&res->nleft, 1u);
    if (slot < GBC_LEFT_CAP) res->left_n[slot] = n;
    else atomicOr(&res->err, kErrLeftOverflow);
}

// (n, p(n)) of an even whose smallest witness reaches the ridge floor (the
// reference's ridge appends, include/ridge.hpp:116-165)
__device__ __forceinline__ void append_ridge(gbc_segment_result *res, uint64_t n, uint32_t p)
{
    const uint32_t slot = atomicAdd(&res->nridge, 1u);
    if (slot < GBC_RIDGE_CAP) {
        res->ridge_n[slot] = n;
        res->ridge_p[slot] = p;
    } else atomicOr(&res->err, kErrRidgeOverflow);
}

// ---- p(n) of every even of a sampled segment -----------------------------------
//
// Word form. In class bits of a run (base a multiple of 30) the even n = base +
// 30 T + r of class r and the candidate p = s + 30 d meet in bit T - o of array
// (r - s) mod 30, o = d + [r < s], so the evens T = 32 j .. 32 j + 31 of every
// class sit in word j. A lane takes word j of all eight arrays and settles the
// class's first candidates in ascending order, each a funnel shift and an AND
// over 32 evens; their counts are the differences of the evens still open after
// each: a popcount, two of them added to a counter in shared memory that two
// lanes of every warp share (a reduction over the warp for two, on the popcounts'
// own pipe, took 8.0 ms where this takes 6.5). Offsets and arrays are
// constants. A candidate settles 3.75 / ln q of the open evens: kCkFirst of them
// from 1e17 on (about 97 evens in a hundred settled), kCkFew below, where that
// many settle as much and the later ones are too rare to have been seen.
//
// Even form. The class arrays of a chunk are transposed to one byte per block
// of 30 (bit k: class k), where q ascends, and a 64-bit window of eight blocks
// ending at T is ANDed with the class's mask of the candidates it reaches: the
// largest q below n whose distance is a candidate is the witness of p(n), so the
// highest bit is it. The words the word form leaves open go to a queue of the
// warp and are taken from there, a word per lane, even by even through the
// windows from the class's next candidate on (kCkWindows in all, the candidates
// to 9781).
//
// An item's evens ascend from part to part (a few words, the rest of the first
// chunk, the other chunks), so a candidate seen before a part cannot come first
// in it. Words of classes with an unseen candidate among the first ones, the
// words at a segment's ends, and every word where p(n) or a low ridge floor
// wants each even, take the even form alone, a T per lane.
//
// Bound by issue and the popcounts' pipe. One GB300, p(n) of every even: 48
// segments of 467.5M at 4e18 6.5 ms (36 candidates in the word form 6.56, 44
// 6.59, 48 6.80; the even form alone, two windows a T, 11.8) against 17.6 for
// candidates tested over words of 32 evens until the last even of 4096 was
// settled; 195 segments of uneven windows 19.9 against 53.4; 5e8 evens at 1e12
// 0.31 against 0.69 (24 candidates there 0.32, 32 0.35, 40 1.04: the last ones
// are seen late); 1e7 with the p(n) array 0.10 against 1.45.
constexpr int kCkThreads = 512;
constexpr int kCkCtas = 2;                         // CTAs per SM
constexpr uint32_t kCkWarps = kCkThreads / 32;
constexpr uint32_t kCkHalo = 11;                   // words below a chunk: 41 windows of 8 blocks reach 335 back
constexpr uint32_t kCkWords = kCkThreads - kCkHalo;  // words of a full chunk: one word per thread staged
constexpr uint32_t kCkHist = 8;                    // windows counted in shared memory
constexpr uint32_t kCkHalf = 8;                    // classes settled at a time
constexpr uint32_t kCkQueue = 32 * kCkHalf;        // words of a warp's queue: a block's of that many classes
constexpr uint32_t kCkMaxChunks = 18;              // chunks of an item at most (check_split)
constexpr uint32_t kCkLanes = 16;                  // counters of a pair of candidates (lanes l and l + 16 share one)
static_assert(32 * kCkHalo >= 8 * kCkWindows + 7, "the last window is staged");
static_assert(kCkMaxChunks * kCkWarps * (32 / kCkLanes) * 32 < 65536, "a counter of 16 bits holds an item");
static_assert(kCkWords <= 512 && kCkFirst % 2 == 0 && kCkFew % 2 == 0, "queue entries and candidate pairs");

struct CkShared {
    uint32_t hist[GBC_NCLASS][64 * kCkHist];       // even form: marks by bit of the windows
    uint32_t open[GBC_NCLASS][kCkFirst + 1];       // word form: evens taken, and those open after each candidate,
    __align__(16) uint32_t part[GBC_NCLASS * kCkFirst / 2][kCkLanes];  // the latter of two candidates by lane until the item's end
    uint4 mask[GBC_NCLASS][kCkWindows];            // x, y: the window's candidates; z, w: those seen before the part
    uint32_t first[GBC_NCAND];
    uint32_t w0[GBC_NCLASS];                       // CheckTables::w0
    uint32_t slow;                                 // classes that take the even form alone
    uint32_t vb;
    uint32_t q_bits[kCkWarps][kCkQueue];           // open evens of a word ...
    uint16_t q_at[kCkWarps][kCkQueue];             // ... class << 9 | word in the chunk
    __align__(16) uint32_t bytes[8 * kCkThreads + 4];  // one byte per block, halo first; a window reads three words
};

namespace ckw {

struct Cand {
    uint32_t k, o, p;
};
// the i-th candidate of class r: ascending odd primes p with r - p a unit
constexpr Cand cand(uint32_t r, uint32_t i)
{
    for (uint32_t p = 3;; p += 2) {
        bool prime = true;
        for (uint32_t d = 3; d * d <= p; d += 2) prime = prime && p % d != 0;
        const uint32_t k = class_of((r + 30 - p % 30) % 30);
        if (prime && k < 8 && i-- == 0) return Cand{k, p / 30 + (r < p % 30 ? 1u : 0u), p};
    }
}
template <uint32_t R, uint32_t I>
struct Of {
    static constexpr Cand c = cand(R, I);
    static_assert(c.o <= 32, "the candidate reads words j - 1 and j");
};

// words j - 1 (x) and j (y) of the eight arrays (members, not an array: every
// access is by a constant, and an array went to local memory)
struct Words {
    uint2 a0, a1, a2, a3, a4, a5, a6, a7;
};
template <uint32_t K>
__device__ __forceinline__ uint2 words_of(const Words &w)
{
    if constexpr (K == 0) return w.a0;
    else if constexpr (K == 1) return w.a1;
    else if constexpr (K == 2) return w.a2;
    else if constexpr (K == 3) return w.a3;
    else if constexpr (K == 4) return w.a4;
    else if constexpr (K == 5) return w.a5;
    else if constexpr (K == 6) return w.a6;
    else return w.a7;
}

// the bits T - O of array K for the evens T of word j
template <uint32_t K, uint32_t O>
__device__ __forceinline__ uint32_t bits_at(const Words &w)
{
    const uint2 a = words_of<K>(w);
    if constexpr (O == 0) return a.y;
    else if constexpr (O == 32) return a.x;
    else return __funnelshift_l(a.x, a.y, O);
}

template <uint32_t R, uint32_t I>
__device__ __forceinline__ void two(const Words &w, uint32_t &un, uint32_t *part)
{
    un &= ~bits_at<Of<R, I>::c.k, Of<R, I>::c.o>(w);
    const uint32_t n = __popc(un);
    un &= ~bits_at<Of<R, I + 1>::c.k, Of<R, I + 1>::c.o>(w);
    atomicAdd(part + (R / 2 * kCkFirst + I) / 2 * kCkLanes, n + (__popc(un) << 16));
}

// class R's candidates From, ... over a word per lane; un: its evens, then those still open
template <uint32_t R, uint32_t From, size_t... H>
__device__ __forceinline__ void run(const Words &w, uint32_t &un, uint32_t *part, std::index_sequence<H...>)
{
    (two<R, From + 2 * H>(w, un, part), ...);
}

// the same for class C, and its words with open evens into the queue (place:
// the lane's word in the chunk)
template <uint32_t C>
__device__ __forceinline__ void one(const Words &w, bool inner, uint32_t taken, uint32_t slow, bool few, CkShared &sh,
                                     uint32_t *q_bits, uint16_t *q_at, uint32_t place,
                                    uint32_t lane, uint32_t &qn)
{
    if (slow >> C & 1u) return;
    uint32_t un = inner ? ~0u : 0u;
    if (lane == 0) atomicAdd(&sh.open[C][0], taken);
    uint32_t *const part = sh.part[0] + lane % kCkLanes;
    run<2 * C, 0>(w, un, part, std::make_index_sequence<kCkFew / 2>());
    if (!few) run<2 * C, kCkFew>(w, un, part, std::make_index_sequence<(kCkFirst - kCkFew) / 2>());
    const uint32_t bal = __ballot_sync(~0u, un != 0);
    if (un) {
        const uint32_t at = qn + __popc(bal & ((1u << lane) - 1u));
        q_bits[at] = un;
        q_at[at] = uint16_t((C << 9) | place);
    }
    qn += __popc(bal);
}

// classes From, ...
template <uint32_t From, size_t... C>
__device__ __forceinline__ void all(const Words &w, bool inner, uint32_t slow, bool few, CkShared &sh,
                                     uint32_t *q_bits, uint16_t *q_at, uint32_t place, uint32_t lane,
                                    uint32_t &qn, std::index_sequence<C...>)
{
    const uint32_t taken = 32 * __popc(__ballot_sync(~0u, inner));
    (one<From + C>(w, inner, taken, slow, few, sh, q_bits, q_at, place, lane, qn), ...);
}

}  // namespace ckw

// bytes at - 7 .. at of the staged blocks as two words (byte `at` topmost)
__device__ __forceinline__ void ck_window(const uint32_t *bytes, uint32_t at, uint32_t &lo, uint32_t &hi)
{
    const uint32_t a = at - 7, s = 8 * (a & 3u);
    const uint32_t *w = bytes + (a >> 2);
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
    lo = __funnelshift_r(w0, w1, s);
    hi = __funnelshift_r(w1, w2, s);
}

__global__ void __launch_bounds__(kCkThreads, kCkCtas) k_check(BatchDesc d, CheckTables ct)
{
    extern __shared__ __align__(16) uint8_t s_ck[];
    CkShared &sh = *reinterpret_cast<CkShared *>(s_ck);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t total = d.h->chk_vb, nseg = d.h->nseg;
    uint32_t *const q_bits = sh.q_bits[warp];
    uint16_t *const q_at = sh.q_at[warp];
    // (locals: the lambdas below would take the address of a copy of ct)
    const uint16_t *const ct_ci = ct.ci, *const ct_cand = ct.cand;
    const uint32_t ridge_w = ct.ridge_w, ridge_min = ct.ridge_min;
    const bool words = ct.word != 0;
    for (uint32_t i = tid; i < GBC_NCLASS * kCkWindows; i += kCkThreads) {
        const uint2 m = ct.mask[i];
        sh.mask[0][i] = make_uint4(m.x, m.y, 0u, 0u);
    }
    for (;;) {
        const uint32_t vb = next_item(d.work + kWorkCheck, &sh.vb);  // synchronizes the CTA
        if (vb >= total) break;
        const uint32_t si = find_prefix(d.chk_pref, nseg, vb);
        const SegParams &sp = d.segs[si];
        const BatchParams &bp = d.runs[sp.run];
        const uint32_t bx = vb - __ldg(d.chk_pref + si), cw = sp.cw;
        const uint32_t wpc = bp.wpc;
        const uint32_t *const map = bp.map;
        gbc_segment_result *const res = sp.res;
        uint16_t *const pn = sp.pn;
        // the segment's evens: T in [A, B] of every class, without A of the
        // classes below ra and B of those above rb; even (T, c) has index 15 T + c - D
        const uint64_t da = sp.seg_start - bp.base, db = sp.seg_end - bp.base;
        const uint32_t A = uint32_t(da / 30), ra = uint32_t(da % 30), B = uint32_t(db / 30), rb = uint32_t(db % 30);
        const uint32_t D = uint32_t(da / 2);
        const uint32_t jlo = A >> 5, jhi = B >> 5;
        const uint32_t nch = (jhi - jlo) / cw + 1;
        const uint32_t c0 = uint32_t(uint64_t(nch) * bx / sp.vbx), c1 = uint32_t(uint64_t(nch) * (bx + 1) / sp.vbx);
        const bool few = sp.ck_few != 0;
        if (tid < GBC_NCLASS) sh.w0[tid] = uint32_t((few ? ct.w0_few : ct.w0) >> (4 * tid)) & 15u;
        for (uint32_t i = tid; i < GBC_NCLASS * 64 * kCkHist; i += kCkThreads) sh.hist[0][i] = 0;
        const bool word_form = words && !pn;  // (else every class is slow)
        if (tid < GBC_NCLASS) sh.open[tid][0] = 0;
        if (word_form)
            for (uint32_t i = tid; i < sizeof sh.part / 16; i += kCkThreads)
                reinterpret_cast<uint4 *>(sh.part)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t i = tid; i < GBC_NCAND; i += kCkThreads) sh.first[i] = kNone;
        // everything of an even but its histogram mark: first occurrence, p(n), ridge
        auto note = [&](uint32_t c, uint32_t bit, uint32_t T) {
            const uint32_t ci = __ldg(ct_ci + c * (64 * kCkWindows) + bit), idx = 15 * T + c - D;
            if (sh.first[ci] > idx) atomicMin(&sh.first[ci], idx);
            if (pn || bit >= 64 * ridge_w) {
                const uint32_t p = __ldg(ct_cand + ci);
                if (pn) pn[idx] = uint16_t(p);
                if (p >= ridge_min) append_ridge(res, bp.base + 30ull * T + 2 * c, p);
            }
            return ci;
        };
        // The candidates of the counted windows seen before word j: theirs cannot
        // come first from j on (none where p(n) or a ridge wants each even). And
        // the classes not all of whose first candidates are. Between barriers.
        auto look = [&](uint32_t j) {
            if (tid == 0) sh.slow = 0;
            __syncthreads();
            const uint32_t idx0 = j == jlo ? 0u : 15 * 32 * j - D;  // no even from word j on has a smaller index
            for (uint32_t i = warp; i < GBC_NCLASS * kCkHist; i += kCkWarps) {
                const uint32_t c = i / kCkHist, w = i % kCkHist;
                const uint16_t *ci = ct_ci + c * (64 * kCkWindows) + 64 * w;
                const uint4 m = sh.mask[c][w];
                // lane l: bits l and 32 + l from the top
                const bool hi = (m.y >> (31 - lane) & 1u) && sh.first[__ldg(ci + lane)] < idx0;
                const bool lo = (m.x >> (31 - lane) & 1u) && sh.first[__ldg(ci + 32 + lane)] < idx0;
                const uint32_t sy = __brev(__ballot_sync(~0u, hi)), sx = __brev(__ballot_sync(~0u, lo));
                const bool all = pn || w >= ridge_w || !words;
                if (lane == 0) {
                    sh.mask[c][w].z = all ? 0u : sx;
                    sh.mask[c][w].w = all ? 0u : sy;
                    if (w <= sh.w0[c] && (all || sx != m.x || sy != m.y)) atomicOr(&sh.slow, 1u << c);
                }
            }
            __syncthreads();
        };
        for (uint32_t ch = c0; ch < c1; ++ch) {
            const uint32_t j0 = jlo + ch * cw, j1 = min(j0 + cw, jhi + 1);  // the chunk's words [j0, j1)
            __syncthreads();  // the last chunk's bytes read, the item's tables ready
            if (tid < j1 - j0 + kCkHalo) {
                // word j of the eight arrays as 32 bytes (no block below the map)
                const uint32_t j = j0 + tid - kCkHalo;
                uint32_t h[8];
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) h[k] = j < wpc ? __ldg(map + size_t(k) * wpc + j) : 0u;
                uint32_t t[8];
                transpose_word(h, t);
                uint4 *dst = reinterpret_cast<uint4 *>(sh.bytes + 8 * tid);
                dst[0] = make_uint4(t[0], t[1], t[2], t[3]);
                dst[1] = make_uint4(t[4], t[5], t[6], t[7]);
            }
            look(j0);
            // The queue's words, one per lane, even by even: the word's open evens
            // qm, its class and place, and for the highest open even the next
            // window from q0 (+ the class's first) on. A lane that is done takes
            // the queue's last word. Ends with the queue empty (words may stay
            // with lanes), or with all settled.
            uint32_t qn = 0, qm = 0, qc = 0, qj = 0, qw = 0;
            auto settle = [&](bool finish) {
                __syncwarp();
                for (;;) {
                    const uint32_t idle = __ballot_sync(~0u, qm == 0);
                    if (qn) {
                        const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
                        if (qm == 0 && rank < qn) {
                            const uint32_t at = q_at[qn - 1 - rank];
                            qm = q_bits[qn - 1 - rank];
                            qc = at >> 9;
                            qj = at & 511u;
                            qw = sh.w0[qc];
                        }
                        qn -= min(qn, uint32_t(__popc(idle)));
                    } else if (!finish || idle == ~0u) {
                        break;
                    }
                    // (an idle lane goes through the motions of its last even without a mark)
                    const bool busy = qm != 0;
                    const uint32_t eb = busy ? 31u - __clz(qm) : 0u, qt = 32 * qj + eb;
                    uint32_t lo, hi;
                    ck_window(sh.bytes, 32 * kCkHalo + qt - 8 * qw, lo, hi);
                    const uint4 m = sh.mask[qc][qw];
                    lo &= m.x;
                    hi &= m.y;
                    const uint32_t z = hi ? hi : lo, b = __clz(z);
                    const bool hit = busy && z;
                    const uint32_t bit = 64 * qw + b + (hi ? 0u : 32u);
                    if (hit && qw < kCkHist) atomicAdd(&sh.hist[qc][bit], 1u);
                    const bool seen = (hi ? m.w : m.z) << b >> 31;
                    const bool last = qw + 1 == kCkWindows;
                    if ((hit && !seen) || (busy && last)) {  // rare
                        if (hit) {
                            const uint32_t ci = note(qc, bit, 32 * j0 + qt);
                            if (qw >= kCkHist) atomicAdd(&res->hist[qc][ci], 1u);
                        } else {
                            append_leftover(res, bp.base + 30ull * (32 * j0 + qt) + 2 * qc);
                        }
                    }
                    __syncwarp();
                    const bool done = busy && (hit || last);
                    if (done) qm &= ~(1u << eb);
                    qw = done ? sh.w0[qc] : busy ? qw + 1 : qw;
                }
                __syncwarp();
            };
            // word j of the classes in `classes` in the even form, a T per lane:
            // the windows to the class's w0; the others' evens into the queue
            auto even_word = [&](uint32_t j, uint32_t classes) {
                const uint32_t T = 32 * j + lane, tl = T - 32 * j0;
#pragma unroll 1
                for (; classes; classes &= classes - 1u) {
                    const uint32_t c = __ffs(classes) - 1u;
                    bool open = T >= A + (2 * c < ra ? 1u : 0u) && T <= B - (2 * c > rb ? 1u : 0u);
                    for (uint32_t w = 0; w <= sh.w0[c]; ++w) {
                        uint32_t lo, hi;
                        ck_window(sh.bytes, 32 * kCkHalo + tl - 8 * w, lo, hi);
                        const uint4 m = sh.mask[c][w];
                        lo &= m.x;
                        hi &= m.y;
                        if (open && (lo | hi)) {
                            const uint32_t b = hi ? __clz(hi) : __clz(lo), bit = 64 * w + b + (hi ? 0u : 32u);
                            atomicAdd(&sh.hist[c][bit], 1u);
                            if (!((hi ? m.w : m.z) << b >> 31)) note(c, bit, T);
                            open = false;
                        }
                        __syncwarp();
                    }
                    const uint32_t left = __ballot_sync(~0u, open);
                    if (left) {
                        if (lane == 0) {
                            q_bits[qn] = left;
                            q_at[qn] = uint16_t((c << 9) | (j - j0));
                        }
                        ++qn;
                    }
                }
            };
            // the item's first chunk in two parts: a few words, after which the
            // first candidates have been seen, then the others
            const uint32_t jm = ch == c0 ? min(j0 + 3 * kCkWarps, j1) : j1;
            for (uint32_t part = 0, ja = j0, jb = jm; ja < jb; ++part, ja = jm, jb = part == 1 ? j1 : jm) {
                if (part) {
                    __syncthreads();
                    look(ja);
                }
                constexpr uint32_t kAll = (1u << GBC_NCLASS) - 1u;
                const uint32_t slow = sh.slow;
                if (slow == kAll) {
                    for (uint32_t j = ja + warp; j < jb; j += kCkWarps) {
                        even_word(j, kAll);
                        settle(false);
                    }
                } else {
                    for (uint32_t jw = ja + 32 * warp; jw < jb; jw += 32 * kCkWarps) {
                        // a word per lane; the segment's end words and slow classes apart
                        const uint32_t j = jw + lane;
                        const bool inner = j < jb && j > jlo && j < jhi;
                        const uint32_t *const at = map + (inner ? j : jlo + 1);
                        auto pair = [&](uint32_t k) {
                            return make_uint2(__ldg(at + size_t(k) * wpc - 1), __ldg(at + size_t(k) * wpc));
                        };
                        const ckw::Words w{pair(0), pair(1), pair(2), pair(3), pair(4), pair(5), pair(6), pair(7)};
                        ckw::all<0>(w, inner, slow, few, sh, q_bits, q_at, j - j0, lane, qn,
                                    std::make_index_sequence<kCkHalf>());
                        settle(false);
                        ckw::all<kCkHalf>(w, inner, slow, few, sh, q_bits, q_at, j - j0, lane, qn,
                                          std::make_index_sequence<GBC_NCLASS - kCkHalf>());
                        settle(false);
                        const uint32_t je = min(jw + 32, jb);
                        if (slow)
                            for (uint32_t i = jw; i < je; ++i)
                                if (i > jlo && i < jhi) {
                                    even_word(i, slow);
                                    settle(false);
                                }
                        if (jlo >= jw && jlo < je) even_word(jlo, kAll);
                        if (jhi >= jw && jhi < je && jhi != jlo) {
                            settle(false);
                            even_word(jhi, kAll);
                        }
                        settle(false);
                    }
                }
                settle(true);
            }
        }
        __syncthreads();
        for (uint32_t i = tid; word_form && i < GBC_NCLASS * kCkFirst / 2; i += kCkThreads) {
            const uint4 *v = reinterpret_cast<const uint4 *>(sh.part[i]);
            uint32_t a = 0, b = 0;
#pragma unroll
            for (uint32_t l = 0; l < kCkLanes / 4; ++l) {
                a += (v[l].x & 0xFFFFu) + (v[l].y & 0xFFFFu) + (v[l].z & 0xFFFFu) + (v[l].w & 0xFFFFu);
                b += (v[l].x >> 16) + (v[l].y >> 16) + (v[l].z >> 16) + (v[l].w >> 16);
            }
            uint32_t *const at = sh.open[i / (kCkFirst / 2)] + 2 * (i % (kCkFirst / 2)) + 1;
            at[0] = a;
            at[1] = b;
        }
        __syncthreads();
        for (uint32_t i = tid; i < GBC_NCLASS * 64 * kCkHist; i += kCkThreads) {
            const uint32_t v = sh.hist[0][i];
            if (!v) continue;
            const uint32_t c = i / (64 * kCkHist), bit = i % (64 * kCkHist);
            atomicAdd(&res->hist[c][__ldg(ct_ci + c * (64 * kCkWindows) + bit)], v);
        }
        for (uint32_t i = tid; word_form && i < GBC_NCLASS * kCkFirst; i += kCkThreads) {
            const uint32_t c = i / kCkFirst, at = i % kCkFirst;
            if (few && at >= kCkFew) continue;
            const uint32_t v = sh.open[c][at] - sh.open[c][at + 1];
            if (v) atomicAdd(&res->hist[c][__ldg(ct.rank + i)], v);
        }
        for (uint32_t i = tid; i < GBC_NCAND; i += kCkThreads)
            if (sh.first[i] != kNone) atomicMin(&res->first[i], sh.first[i]);
        __syncthreads();
    }
}

// Generic checker for segments that reach q < 7 (seg_start < 9788): one
// thread per even, every candidate ascending, q = 3 and q = 5 prime by
// definition (they are not in the class map), q < 3 ends the search.
__global__ void __launch_bounds__(256) k_check_low(BatchDesc d, const uint16_t *cand, uint32_t ridge_min)
{
    if (!d.h->nlow) return;
    const uint32_t nseg = d.h->nseg;
    for (uint32_t si = d.h->seg0; si < nseg; ++si) {
        const SegParams &sp = d.segs[si];
        if (!sp.low) continue;
        const BatchParams &bp = d.runs[sp.run];
        const uint64_t evens = (sp.seg_end - sp.seg_start) / 2 + 1;
        gbc_segment_result *res = sp.res;
        for (uint64_t e = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; e < evens;
             e += uint64_t(gridDim.x) * blockDim.x) {
            const uint64_t n = sp.seg_start + 2 * e;
            const uint32_t cr = uint32_t(n % 30) / 2;
            int ci = -1;
            for (int c = 0; c < GBC_NCAND; ++c) {
                const uint64_t p = cand[c];
                if (p + 3 > n) break;
                const uint64_t q = n - p;
                bool prime;
                if (q == 3 || q == 5) prime = true;
                else if (q % 3 == 0 || q % 5 == 0) prime = false;
                else {
                    const uint64_t t = (q - bp.base) / 30;
                    const uint32_t k = class_of(uint32_t(q % 30));
                    prime = (bp.map[size_t(k) * bp.wpc + (t >> 5)] >> (t & 31)) & 1u;
                }
                if (prime) {
                    ci = c;
                    break;
                }
            }
            if (ci >= 0) {
                atomicAdd(&res->hist[cr][ci], 1u);
                atomicMin(&res->first[ci], uint32_t(e));
                if (sp.pn) sp.pn[e] = cand[ci];
                if (cand[ci] >= ridge_min) append_ridge(res, n, cand[ci]);
            } else {
                append_leftover(res, n);
            }
        }
    }
}

// Evens without a witness <= 9781: ascending odd p > 9781 by Miller-Rabin on
// both p and n - p (n = 4: p = 2). A bounded search of at most max_tries
// candidates: one that runs out sets an error flag instead of looping. A
// CTA per segment.
__global__ void __launch_bounds__(64) k_retry(BatchDesc d, uint32_t ridge_min, uint32_t max_tries)
{
    const uint32_t nseg = d.h->nseg;
    for (uint32_t si = d.h->seg0 + blockIdx.x; si < nseg; si += gridDim.x) {
        const SegParams &sp = d.segs[si];
        gbc_segment_result *res = sp.res;
        const uint32_t nl = res->nleft < GBC_LEFT_CAP ? res->nleft : GBC_LEFT_CAP;
        for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) {
            const uint64_t n = res->left_n[i];
            uint64_t found = 0;
            if (n == 4) found = 2;
            else {
                uint32_t tries = 0;
                for (uint64_t p = GBC_MAX_CAND + 2; p <= n / 2; p += 2) {
                    if (++tries > max_tries) {
                        atomicOr(&res->err, kErrRetry);
                        break;
                    }
                    if (is_prime_u64_dev(p) && is_prime_u64_dev(n - p)) {
                        found = p;
                        break;
                    }
                }
            }
            res->left_p[i] = found;
            if (sp.pn) sp.pn[(n - sp.seg_start) / 2] = found < 65536 ? uint16_t(found) : 0;
            if (found && found >= ridge_min) append_ridge(res, n, uint32_t(found));
        }
    }
}

// Phase B (the reference's check30_b, kernels/goldbach.cl:2210-2306): the
// exact p(n) of every pending even, by the class's rest candidates in
// ascending order (every plan member already failed for it), one thread per
// pending word. The histogram and first occurrences of these evens hold
// every even with p(n) >= the plan bound; ridges above the floor are listed.
// The pending words of all segments of the batch form one index space (a
// prefix over the segments' counts), so the segments' words are settled
// side by side rather than one segment after another.
constexpr int kTailThreads = 256;
static_assert(kTailThreads >= 256, "one thread per segment of a batch for the prefix");

__global__ void __launch_bounds__(kTailThreads) k_tail(BatchDesc d, VerifyTables vt)
{
    __shared__ uint32_t s_pref[2][257];
    const uint32_t nseg = d.h->nseg, tid = threadIdx.x;
    // s_pref[.][s]: pending words of the segments before s (Hillis-Steele)
    {
        uint32_t c = 0;
        if (tid < nseg && tid >= d.h->seg0) {  // the segments of the window
            const SegParams &sp = d.segs[tid];
            const uint32_t np = sp.res->npend;
            c = sp.sampled ? 0u : (np < sp.pend_cap ? np : sp.pend_cap);
        }
        s_pref[0][tid + 1] = c;
        if (tid == 0) s_pref[0][0] = s_pref[1][0] = 0;
        __syncthreads();
        uint32_t src = 0;
        for (uint32_t o = 1; o < 256; o <<= 1, src ^= 1u) {
            uint32_t v = s_pref[src][tid + 1];
            if (tid >= o) v += s_pref[src][tid + 1 - o];
            s_pref[src ^ 1u][tid + 1] = v;
            __syncthreads();
        }
        if (src) {  // the result in s_pref[0]
            s_pref[0][tid + 1] = s_pref[1][tid + 1];
            __syncthreads();
        }
    }
    const uint32_t total = s_pref[0][nseg];
    for (uint32_t g = blockIdx.x * blockDim.x + tid; g < total; g += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nseg;  // s_pref[lo] <= g < s_pref[hi]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s_pref[0][mid] <= g) lo = mid;
            else hi = mid;
        }
        const uint32_t si = lo, i = g - s_pref[0][lo];
        const SegParams &sp = d.segs[si];
        const BatchParams &bp = d.runs[sp.run];
        gbc_segment_result *res = sp.res;
        const uint64_t seg_start = sp.seg_start, base = bp.base;
        {
            const uint2 e = sp.pend[i];
            const uint32_t cr = e.x >> 27, j = e.x & ((1u << 27) - 1), r = 2 * cr;
            uint32_t mask = e.y;
            const uint64_t n0 = seg_start + (r + 30 - uint32_t(seg_start % 30)) % 30;
            const uint32_t idx0 = uint32_t((n0 - seg_start) / 2);
            const uint32_t off = vt.rest_off[cr], cnt = vt.rest_cnt[cr];
            for (uint32_t c = 0; c < cnt && mask; ++c) {
                const uint32_t ci = vt.rest[off + c];
                const uint32_t p = vt.cand[ci];
                const uint32_t u = (r + 30 - p % 30) % 30;
                const uint32_t pos = uint32_t((n0 - base - p - u) / 30) + 32 * j;
                const uint32_t *wk = bp.map + size_t(class_of(u)) * bp.wpc + (pos >> 5);
                const uint32_t hit = mask & __funnelshift_r(__ldg(wk), __ldg(wk + 1), pos & 31);
                if (!hit) continue;
                atomicAdd(&res->hist[cr][ci], uint32_t(__popc(hit)));
                atomicMin(&res->first[ci], idx0 + 15u * (32u * j + __ffs(hit) - 1u));
                if (p >= vt.ridge_min)
                    for (uint32_t h = hit; h; h &= h - 1u)
                        append_ridge(res, n0 + 30ull * (32ull * j + __ffs(h) - 1u), p);
                mask &= ~hit;
            }
            for (; mask; mask &= mask - 1u) append_leftover(res, n0 + 30ull * (32ull * j + __ffs(mask) - 1u));
        }
    }
}

// Result areas of the batch's segments: zero, except the first-occurrence
// indices and the first prime (all ones: none yet); the slot's error word;
// a binned batch's tile-bin and overflow counts.
__global__ void __launch_bounds__(256) k_init(BatchDesc d)
{
    constexpr uint32_t kWords = sizeof(gbc_segment_result) / 4;
    constexpr uint32_t kF0 = offsetof(gbc_segment_result, first) / 4, kF1 = kF0 + GBC_NCAND;
    constexpr uint32_t kP0 = offsetof(gbc_segment_result, first_prime) / 4;
    const uint32_t nseg = d.h->nseg;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid == 0 && d.h->nrun) *d.runs[0].err = 0;
    if (d.h->nrun && hl_binned(d.runs[0])) {  // the tile bins' counts and the overflow count
        const BatchParams &bp = d.runs[0];
        for (uint32_t i = tid; i < 8 * bp.tb_tiles; i += gridDim.x * blockDim.x) bp.tb_cnt[i] = 0;
        if (tid == 0) *bp.ovf_cnt = 0;
    }
    for (uint32_t si = 0; si < nseg; ++si) {
        uint32_t *w = reinterpret_cast<uint32_t *>(d.segs[si].res);
        for (uint32_t i = tid; i < kWords; i += gridDim.x * blockDim.x)
            w[i] = ((i >= kF0 && i < kF1) || i == kP0 || i == kP0 + 1) ? ~0u : 0u;
    }
}

}  // namespace gbk

namespace gbh {

void launch_init(const gbk::BatchDesc &d, const Grids &g, cudaStream_t st)
{
    gbk::k_init<<<g.sm * 2, 256, 0, st>>>(d);
}

// words per chunk and items of a sampled segment: full chunks, up to 16 per
// item while the batch (words: of all its sampled segments) keeps three items
// per resident CTA (an item clears and flushes 31 KB of counts, and takes its
// first 48 words even by even); below that shorter chunks, down to a word per
// warp: 5e5 evens take 0.03 ms, against 0.06 on one CTA a class.
// A segment of eight CTAs' work or more in a batch of at most 48 chunks per CTA
// has a fixed number of items per CTA instead, all of the same chunks: one or
// two or three, the fewest with at most 16 chunks on the batch's mean (a
// segment's own, of 8 items or more, have an eighth more at most: kCkMaxChunks);
// two at least beside
// segments of less (smallest), whose items come between. p(n) of every even,
// one GB300, before the word form's counters: one segment of 467.5M at 4e18
// 0.30 ms (three items per CTA 0.43), two 0.46 (0.61), eight 1.51 (1.61); 1e9
// integers at 1e12 0.36 (0.45); sixteen windows of 2e4 to 5e8 0.71 (0.79, one
// item per CTA 0.87).
void check_split(uint64_t evens, uint64_t words, uint64_t smallest, int sm, uint32_t *cw, uint32_t *vbx)
{
    const uint64_t mine = evens / 15 / 32 + 2, want = uint64_t(sm) * gbk::kCkCtas;
    const uint64_t w = (words + want - 1) / want;
    const bool beside = 8 * words > smallest * want && w > 2 * gbk::kCkWords;
    const uint64_t k = std::max<uint64_t>((w + 16 * gbk::kCkWords - 1) / (16 * gbk::kCkWords), beside ? 2 : 1),
                   items = words ? mine * want * k / words : 0;  // (0: no segment of the batch is the checker's)
    if (items >= 8 * k && k <= 3) {
        const uint64_t m = (mine + gbk::kCkWords * items) / (gbk::kCkWords * items);
        const uint64_t each = (mine + m * items) / (m * items);
        if (each >= gbk::kCkWarps && m <= gbk::kCkMaxChunks) {
            *cw = uint32_t(each);
            *vbx = uint32_t(items);
            return;
        }
    }
    *cw = uint32_t(w < gbk::kCkWarps ? gbk::kCkWarps : w > gbk::kCkWords ? gbk::kCkWords : w);
    const uint64_t nch = (mine + *cw - 1) / *cw;
    const uint64_t per = std::min<uint64_t>(16, std::max<uint64_t>(1, words / *cw / (3 * want)));
    *vbx = uint32_t((nch + per - 1) / per);
}

// whether a segment takes the word form's kCkFew candidates
bool check_few(uint64_t seg_start) { return seg_start < 100000000000000000ull; }

void launch_check(const gbk::BatchDesc &d, const gbk::CheckTables &ct, const Grids &g, cudaStream_t st)
{
    gbk::k_check_low<<<g.sm * 16, 256, 0, st>>>(d, ct.cand, ct.ridge_min);
    gbk::k_check<<<g.sm * g.check, gbk::kCkThreads, sizeof(gbk::CkShared), st>>>(d, ct);
}

void launch_tail(const gbk::BatchDesc &d, const gbk::VerifyTables &vt, const Grids &g, cudaStream_t st)
{
    gbk::k_tail<<<g.sm * 2, gbk::kTailThreads, 0, st>>>(d, vt);
}

void launch_retry(const gbk::BatchDesc &d, uint32_t ridge_min, uint32_t tries, const Grids &g, cudaStream_t st)
{
    gbk::k_retry<<<g.max_seg < 1024 ? g.max_seg : 1024, 64, 0, st>>>(d, ridge_min, tries);
}

void query_check_grids(Grids &g)
{
    int n = 0;
    cudaFuncSetAttribute(gbk::k_check, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(gbk::CkShared)));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gbk::k_check, gbk::kCkThreads, sizeof(gbk::CkShared));
    g.check = n > 0 ? n : 1;
}

}  // namespace gbh
