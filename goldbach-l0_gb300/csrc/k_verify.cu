// k_verify.cu -- the funnel verify (phase A) of unsampled segments: a witness
// for every even, whichever candidate it is (the reference's check30_a,
// kernels/goldbach.cl:2029-2189).
//
// In class bits of a run (base a multiple of 30): the even n = base + 30 T +
// r of class r and the candidate p = s + 30 d' of residue s meet in q = n - p
// = base + 30 (T - d' - c) + u, u = (r - s) mod 30, c = 1 iff r < s. So the
// candidates of one residue s test bits T - o of the one class array u, o = d'
// + c, and the evens T = 32 j .. 32 j + 31 of every class r sit in word j.
//
// Word form. A funnel of residue s (all primes p0 .. p0 + 930 of the residue,
// about 20) over 32 evens is the OR of its array's words j - 1, j shifted by
// its offsets o <= 32. A thread takes word j of all eight arrays and settles
// word j of all fifteen even classes, three funnels a class: an array is read
// once for the five to seven funnels that use it, and the funnels share what
// they have in common, windows like W | W << 2 or W | W << 2 | W << 3, built
// once per array. The offsets are constants, so every funnel is straight-line
// code, covered by the windows' shifts at compile time (cover(): greedy;
// kArr's windows were found by a search that adds the window saving most).
// 40 ALU operations per class word (three funnels, windows included)
// where a funnel at a time, its members' shifts read from a table, takes 85.
//
// Even form. The funnel of one even is one 32-bit window of its class array
// ANDed with the member mask: about 20 instructions for about 20 candidates.
// After three funnels one class word in eight still has an open even (they
// cluster where primes are few), so those words go to a queue of the warp and
// are taken from there, a word per lane, even by even through the plan's other
// funnels.
//
// Plans without the word form's funnels take their few from a table, word by
// word (plan_words).
//
// Evens no plan funnel settles are pending: (class, word of the segment's
// evens of the class, bits) for k_tail.
//
// Bound by the ALU pipe (funnel shifts and three-input logic: 53 ALU of 90
// instructions per class word, issue 64%). One GB300, 127 verified segments
// of 467.5M at 4e18: 2.97 ms, 677 GB/s of map, against 8.78 ms for funnels
// from a table, class by class, each class staging its own windows of the
// map (233 instructions per class word). Words per lane and CTAs per SM: 4 / 4
// 2.97 ms, 3 / 5 3.01, 2 / 6 3.11, 2 / 5 3.17, 4 / 5 3.08; a queue taken 32
// words at a time until all are settled, 3.27.
#include <cuda_runtime.h>

#include <utility>

#include "gbc_common.cuh"

namespace gbk {

constexpr int kVerifyThreads = 128;
constexpr int kVerifyCtas = 4;             // CTAs per SM
constexpr uint32_t kVerifyWarps = kVerifyThreads / 32;
constexpr uint32_t kVW = 4;                // words per lane in a chunk
constexpr uint32_t kVChunk = 32 * kVW;     // words per warp chunk
constexpr uint32_t kVBack = 4;             // staged words below the chunk: a plan member is at most 100 bits back
constexpr uint32_t kVWin = kVChunk + 8;    // staged words per array: 4 below, the chunk, 1 above, a multiple of 4
constexpr uint32_t kVQueue = 32 * GBC_NCLASS + 32;  // words of the warp's queue (a step's), whole lines
constexpr uint32_t kVWarpWords = 2 * 8 * kVWin + kVQueue * 3 / 2;  // a warp's shared memory
constexpr size_t kVerifySmem = size_t(kVerifyWarps) * kVWarpWords * 4;
static_assert(GBC_TAIL_T / 30 + 1 < 32 * kVBack, "a plan member's window starts in the staged words");

// ---- the word form's program, at compile time --------------------------------
namespace vp {

constexpr bool is_prime(uint32_t p)
{
    for (uint32_t d = 2; d * d <= p; ++d)
        if (p % d == 0) return false;
    return p > 1;
}

// the smallest candidate of residue s (a unit mod 30)
constexpr uint32_t first_of(uint32_t s) { return s == 1 ? 31 : s; }

// residue of the i-th of the three funnels every word of class r takes: the
// residues s with r - s a unit, in the order a plan opens them (a plan of
// five funnels a class or more holds them all)
constexpr uint32_t residue(uint32_t r, uint32_t i)
{
    constexpr uint32_t order[8] = {7, 11, 13, 17, 19, 23, 29, 1};
    for (uint32_t k = 0; k < 8; ++k)
        if (class_of((r + 30 - order[k]) % 30) < 8 && i-- == 0) return order[k];
    return 0;
}

// offsets o <= 32 of the funnel (r, s), bit o
constexpr uint64_t offsets(uint32_t r, uint32_t s)
{
    uint64_t m = 0;
    for (uint32_t p = first_of(s); p <= first_of(s) + 930; p += 30) {
        const uint32_t o = p / 30 + (r < s ? 1 : 0);
        if (is_prime(p) && o <= 32) m |= 1ull << o;
    }
    return m;
}

// window i > 0 of an array: window x | window y << d (window 0: the array)
struct Window {
    uint8_t x, y, d;
};
constexpr uint32_t kWindows = 8;
struct Array {
    uint32_t n;
    Window w[kWindows];
};
constexpr Array kArr[8] = {
    {5, {{0, 0, 2}, {0, 1, 4}, {2, 1, 1}, {2, 2, 7}, {0, 1, 2}}},
    {6, {{0, 0, 2}, {1, 0, 1}, {2, 0, 4}, {0, 3, 5}, {0, 2, 13}, {3, 1, 9}}},
    {6, {{0, 0, 2}, {1, 0, 9}, {2, 1, 13}, {2, 0, 3}, {1, 0, 1}, {2, 4, 13}}},
    {6, {{0, 0, 2}, {1, 0, 1}, {2, 0, 4}, {0, 3, 5}, {0, 2, 13}, {3, 1, 9}}},
    {6, {{0, 0, 1}, {0, 1, 1}, {1, 0, 3}, {1, 2, 7}, {3, 1, 10}, {0, 2, 5}}},
    {5, {{0, 0, 2}, {1, 0, 1}, {2, 0, 4}, {0, 3, 6}, {0, 2, 2}}},
    {8, {{0, 0, 1}, {1, 1, 7}, {1, 0, 12}, {1, 3, 3}, {0, 0, 4}, {4, 0, 11}, {2, 1, 21}, {3, 0, 14}}},
    {7, {{0, 0, 1}, {1, 1, 7}, {1, 0, 12}, {1, 3, 3}, {2, 0, 5}, {3, 3, 3}, {4, 2, 18}}},
};

// the shifts of the windows whose OR is the funnel: window w[i] shifted by a[i]
struct Cover {
    uint32_t n = 0;
    uint8_t w[24] = {}, a[24] = {};
};
constexpr uint32_t bits(uint64_t m)
{
    uint32_t c = 0;
    for (; m; m &= m - 1) ++c;
    return c;
}
// k: the array's class; the shift covering most open offsets first, a shift
// by 0 or 32 (no operation) on ties
constexpr Cover cover(uint32_t k, uint64_t S)
{
    uint64_t pat[kWindows + 1] = {1};
    for (uint32_t i = 0; i < kArr[k].n; ++i)
        pat[i + 1] = pat[kArr[k].w[i].x] | (pat[kArr[k].w[i].y] << kArr[k].w[i].d);
    Cover c;
    uint64_t left = S;
    while (left) {
        uint32_t best = 0, bw = 0, ba = 0;
        bool bfree = false;
        uint64_t bm = 0;
        for (uint32_t i = 0; i <= kArr[k].n; ++i)
            for (uint32_t a = 0; (pat[i] << a) < (1ull << 33); ++a) {
                const uint64_t m = pat[i] << a;
                if (m & ~S) continue;
                const uint32_t g = bits(m & left);
                const bool free = a == 0 || a == 32;
                if (g > best || (g == best && g && free && !bfree)) {
                    best = g;
                    bw = i;
                    ba = a;
                    bfree = free;
                    bm = m;
                }
            }
        c.w[c.n] = uint8_t(bw);
        c.a[c.n++] = uint8_t(ba);
        left &= ~bm;
    }
    return c;
}

// window W shifted by A: bits [32 - A, 64 - A) of hi:lo
template <uint32_t W, uint32_t A>
__device__ __forceinline__ uint32_t back(const uint32_t *lo, const uint32_t *hi)
{
    if constexpr (A == 0) return hi[W];
    else if constexpr (A == 32) return lo[W];
    else return __funnelshift_l(lo[W], hi[W], A);
}

// class R's funnel on array K: its residue, whether it is one of the class's
// three, and its cover
template <uint32_t K, uint32_t R>
struct Funnel {
    static constexpr uint32_t s = (R + 30 - unit30(K)) % 30;
    static constexpr bool used = s == residue(R, 0) || s == residue(R, 1) || s == residue(R, 2);
    static constexpr Cover c = used ? cover(K, offsets(R, s)) : Cover{};
};

template <uint32_t K, uint32_t R, size_t... I>
__device__ __forceinline__ uint32_t funnel(const uint32_t *lo, const uint32_t *hi, std::index_sequence<I...>)
{
    return (back<Funnel<K, R>::c.w[I], Funnel<K, R>::c.a[I]>(lo, hi) | ...);
}

// clears from un[r / 2] what class r's funnel on array K settles, if it is one of the class's three
template <uint32_t K, uint32_t R>
__device__ __forceinline__ void class_funnel(const uint32_t *lo, const uint32_t *hi, uint32_t *un)
{
    if constexpr (Funnel<K, R>::used)
        un[R / 2] &= ~funnel<K, R>(lo, hi, std::make_index_sequence<Funnel<K, R>::c.n>());
}

// window W + 1 of array K
template <uint32_t K, size_t W>
__device__ __forceinline__ void window(uint32_t *lo, uint32_t *hi)
{
    constexpr Window x = kArr[K].w[W];
    hi[W + 1] = hi[x.x] | __funnelshift_l(lo[x.y], hi[x.y], x.d);
    lo[W + 1] = lo[x.x] | (lo[x.y] << x.d);
}

template <uint32_t K, size_t... W>
__device__ __forceinline__ void windows(uint32_t *lo, uint32_t *hi, std::index_sequence<W...>)
{
    (window<K, W>(lo, hi), ...);
}

// array K's words j - 1, j (w[-1], w[0]) through every funnel that reads it
template <uint32_t K, size_t... C>
__device__ __forceinline__ void array(const uint32_t *w, uint32_t *un, std::index_sequence<C...>)
{
    uint32_t lo[kWindows + 1], hi[kWindows + 1];
    lo[0] = w[-1];
    hi[0] = w[0];
    windows<K>(lo, hi, std::make_index_sequence<kArr[K].n>());
    (class_funnel<K, 2 * C>(lo, hi, un), ...);
}

template <size_t... K>
__device__ __forceinline__ void word(const uint32_t *w, uint32_t *un, std::index_sequence<K...>)
{
    (array<K>(w + K * kVWin, un, std::make_index_sequence<GBC_NCLASS>()), ...);
}

}  // namespace vp

// ---- the kernel -----------------------------------------------------------------

// one chunk's windows of the eight class arrays into a staging buffer: bulk
// copies of `bytes` each, completing on bar (issued by one lane)
__device__ __forceinline__ void stage_chunk(uint32_t *dst, uint64_t *bar, const uint32_t *src, uint32_t wpc)
{
    constexpr uint32_t bytes = kVWin * 4;
    mbar_arrive_expect_tx(bar, 8 * bytes);
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) bulk_copy_g2s(dst + k * kVWin, src + size_t(k) * wpc, bytes, bar);
}

// whether the even T of a class has a plan witness, from the map in memory
// (ev: the class's nf funnels)
__device__ __forceinline__ bool settled(const BatchParams &bp, const uint2 *ev, uint32_t nf, uint32_t T)
{
    for (uint32_t f = 0; f < nf; ++f) {
        const uint32_t pos = T - (ev[f].x >> 8);
        const uint32_t *a = bp.map + size_t(ev[f].x & 7u) * bp.wpc + (pos >> 5);
        if (__funnelshift_r(__ldg(a), __ldg(a + 1), pos) & ev[f].y) return true;
    }
    return false;
}

// The even T of class cr has no plan witness (rare): its word of the
// segment's evens of the class (evens T0 + 32 w .. of [T0, T1]) is appended
// by the thread that holds the word's first pending even.
__device__ __noinline__ void pend_word(const SegParams &sp, const BatchParams &bp, const uint2 *ev, uint32_t nf,
                                       uint32_t cr, uint32_t T, uint32_t T0, uint32_t T1)
{
    const uint32_t w = (T - T0) >> 5, first = T0 + 32 * w;
    uint32_t m = 0;
    for (uint32_t b = 0; b < 32 && first + b <= T1; ++b) {
        const bool open = first + b == T || !settled(bp, ev, nf, first + b);
        if (open && first + b < T) return;
        if (open) m |= 1u << b;
    }
    gbc_segment_result *res = sp.res;
    const uint32_t at = atomicAdd(&res->npend, 1u);
    if (at < sp.pend_cap) sp.pend[at] = make_uint2((cr << 27) | w, m);
    else atomicOr(&res->err, kErrPendOverflow);
    atomicAdd(reinterpret_cast<unsigned long long *>(&res->pending), (unsigned long long)__popc(m));
}

// The evens T .. T + 31 of a class that its plan settles, T the first even of
// a word plus s < 32, nf funnels read from the table a member at a time: two
// loads, a shift and an OR for 32 evens (w: the word of array 0 among the
// staged windows).
__device__ __forceinline__ uint32_t plan_word(const uint32_t *w, const uint2 *ev, uint32_t nf, uint32_t s)
{
    uint32_t v = 0;
    for (uint32_t f = 0; f < nf; ++f) {
        const uint2 e = ev[f];
        const uint32_t *const a = w + (e.x & 7u) * kVWin;
        for (uint32_t m = e.y; m; m &= m - 1u) {
            const int32_t o = int32_t(e.x >> 8) - (__ffs(m) - 1) - int32_t(s);  // below 0: up to s bits ahead
            const uint32_t *const x = a - (o >> 5);
            v |= __funnelshift_l(x[-1], x[0], uint32_t(o));
        }
    }
    return v;
}

// The plan's pending words among the warp's next 32 words of every class, jw ..
// of the run, by the table (win: the first one's among the staged windows): the
// words of the segment's evens of a class, a word per lane, are the pending list's.
__device__ __forceinline__ void plan_words(const SegParams &sp, const uint32_t *win, uint32_t jw,
                                           const uint2 (*ev)[kVerifyMaxFun], const uint32_t *nf, uint32_t A,
                                           uint32_t ra, uint32_t B, uint32_t rb)
{
    const uint32_t lane = threadIdx.x & 31u;
    gbc_segment_result *const res = sp.res;
#pragma unroll 1
    for (uint32_t c = 0; c < GBC_NCLASS; ++c) {
        const uint32_t T0 = A + (2 * c < ra ? 1u : 0u), T1 = B - (2 * c > rb ? 1u : 0u);
        const uint32_t t = 32 * (jw + lane) + (T0 & 31u);
        uint32_t m = 0;
        if (t >= T0 && t <= T1) m = (T1 - t >= 31 ? ~0u : (2u << (T1 - t)) - 1u) & ~plan_word(win + lane, ev[c], nf[c], T0 & 31u);
        const uint32_t bal = __ballot_sync(~0u, m != 0);
        if (!bal) continue;
        const uint32_t evens = __reduce_add_sync(~0u, __popc(m));
        uint32_t at = 0;
        if (lane == 0) {
            at = atomicAdd(&res->npend, uint32_t(__popc(bal)));
            atomicAdd(reinterpret_cast<unsigned long long *>(&res->pending), (unsigned long long)evens);
        }
        at = __shfl_sync(~0u, at, 0) + __popc(bal & ((1u << lane) - 1u));
        if (!m) continue;
        if (at < sp.pend_cap) sp.pend[at] = make_uint2((c << 27) | ((t - T0) >> 5), m);
        else atomicOr(&res->err, kErrPendOverflow);
    }
}

// kWord: the plan holds the word form's three funnels of every class. A plan
// of fewer than five funnels may not; all its funnels are then taken word by
// word from the table, and every even that is left is pending. One GB300, 1e7
// integers a call at 4e18, three and four funnels a class: 0.69 and 0.74 ms (9.31
// and 4.00 with every even by itself, 1.43 and 1.36 with class words staged
// class by class); five, in the word form, 0.75.
template <bool kWord>
__global__ void __launch_bounds__(kVerifyThreads, kVerifyCtas) k_verify(BatchDesc d, VerifyTables vt)
{
    __shared__ uint2 s_ev[GBC_NCLASS][kVerifyMaxFun];  // see VerifyTables::ev
    __shared__ uint32_t s_nf[GBC_NCLASS];
    __shared__ __align__(8) uint64_t s_bar[kVerifyWarps][2];
    __shared__ uint32_t s_vb;
    // per warp: two staging buffers of the eight arrays' windows, the queue's
    // words (open bits) and their places (class << 8 | word in the chunk)
    extern __shared__ __align__(16) uint32_t s_dyn[];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t *const stage = s_dyn + warp * kVWarpWords;
    uint32_t *const q_bits = stage + 2 * 8 * kVWin;
    uint16_t *const q_at = reinterpret_cast<uint16_t *>(q_bits + kVQueue);
    uint64_t *const bar = s_bar[warp];
    for (uint32_t i = tid; i < GBC_NCLASS * kVerifyMaxFun; i += blockDim.x) {
        const uint32_t cr = i / kVerifyMaxFun, f = i % kVerifyMaxFun;
        if (f < vt.fun_cnt[cr]) s_ev[cr][f] = vt.ev[vt.fun_off[cr] + f];
        if (f == 0) s_nf[cr] = vt.fun_cnt[cr];
    }
    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        mbar_init_fence();
    }
    uint32_t phase = 0;  // bit b: parity of buffer b's next completion
    const uint32_t total = d.h->ver_vb, nseg = d.h->nseg;
    for (;;) {
        const uint32_t vb = next_item(d.work + kWorkVerify, &s_vb);  // synchronizes the CTA
        if (vb >= total) break;
        const uint32_t si = find_prefix(d.ver_pref, nseg, vb);
        const SegParams &sp = d.segs[si];
        const BatchParams &bp = d.runs[sp.run];
        const uint32_t bx = vb - __ldg(d.ver_pref + si), step = sp.vbx * kVerifyWarps;
        const uint32_t wpc = bp.wpc;
        // the segment's evens: T in [A, B] of every class, without A of the
        // classes below ra and B of those above rb
        const uint64_t da = sp.seg_start - bp.base, db = sp.seg_end - bp.base;
        const uint32_t A = uint32_t(da / 30), ra = uint32_t(da % 30), B = uint32_t(db / 30), rb = uint32_t(db % 30);
        const uint32_t jlo = A >> 5, jhi = B >> 5, J0 = jlo & ~3u;  // chunks on 16-byte boundaries
        const uint32_t nch = (jhi - J0) / kVChunk + 1;
        const uint32_t *const src0 = bp.map + (J0 - kVBack);
        uint32_t ch = bx * kVerifyWarps + warp, buf = 0;
        if (ch < nch && lane == 0) {
            fence_proxy_async();
            stage_chunk(stage, bar, src0 + size_t(ch) * kVChunk, wpc);
        }
        for (; ch < nch; ch += step, buf ^= 1u) {
            if (ch + step < nch) {
                __syncwarp();  // every lane is done with the other buffer (the chunk before)
                if (lane == 0) {
                    fence_proxy_async();
                    stage_chunk(stage + (buf ^ 1u) * (8 * kVWin), bar + (buf ^ 1u),
                                src0 + size_t(ch + step) * kVChunk, wpc);
                }
            }
            if (!mbar_wait(bar + buf, (phase >> buf) & 1u, vt.spin0)) {
                atomicOr(&sp.res->err, kErrStaging);
                mbar_wait(bar + buf, (phase >> buf) & 1u);
            }
            phase ^= 1u << buf;
            const uint32_t Jc = J0 + ch * kVChunk;
            const uint32_t *const win = stage + buf * (8 * kVWin);
            if constexpr (!kWord) {
                for (uint32_t w = 0; w < kVW && Jc + 32 * w <= jhi; ++w)
                    plan_words(sp, win + kVBack + 32 * w, Jc + 32 * w, s_ev, s_nf, A, ra, B, rb);
                continue;
            }
            // The queue's words, one per lane, even by even; a lane whose word
            // is settled takes the queue's last one. Ends with the queue empty
            // (words may stay with lanes), or with every word settled.
            uint32_t qn = 0, m = 0, cr = 0, lw = 0, f = 0;
            auto settle = [&](bool finish) {
                for (;;) {
                    const uint32_t idle = __ballot_sync(~0u, m == 0);
                    if (qn) {
                        const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
                        if (m == 0 && rank < qn) {
                            const uint32_t at = q_at[qn - 1 - rank];
                            m = q_bits[qn - 1 - rank];
                            cr = at >> 8;
                            lw = at & 0xFFu;
                            f = 0;
                        }
                        qn -= min(qn, uint32_t(__popc(idle)));
                    } else if (!finish || idle == ~0u) {
                        break;
                    }
                    if (m) {
                        const uint32_t b = __ffs(m) - 1u, nf = s_nf[cr];
                        bool hit = false;
                        if (f < nf) {
                            const uint2 e = s_ev[cr][f];
                            const uint32_t pos = 32 * (lw + kVBack) + b - (e.x >> 8);
                            const uint32_t *a = win + (e.x & 7u) * kVWin + (pos >> 5);
                            hit = (__funnelshift_r(a[0], a[1], pos) & e.y) != 0;
                            ++f;
                        }
                        if (hit || f >= nf) {
                            if (!hit)
                                pend_word(sp, bp, s_ev[cr], nf, cr, 32 * (Jc + lw) + b, A + (2 * cr < ra ? 1u : 0u),
                                          B - (2 * cr > rb ? 1u : 0u));
                            m &= m - 1u;
                            f = 0;
                        }
                    }
                }
                __syncwarp();
            };
#pragma unroll 1
            for (uint32_t w = 0; w < kVW; ++w) {
                const uint32_t jw = Jc + 32 * w;  // the warp's first word
                if (jw > jhi) break;
                uint32_t un[GBC_NCLASS];
                if (jw > jlo && jw + 31 < jhi) {
#pragma unroll
                    for (uint32_t c = 0; c < GBC_NCLASS; ++c) un[c] = ~0u;
                } else {
                    const uint32_t t0 = 32 * (jw + lane);
#pragma unroll
                    for (uint32_t c = 0; c < GBC_NCLASS; ++c) {
                        // bits [lo, hi) of the word are evens of the segment
                        const uint32_t Ta = A + (2 * c < ra ? 1u : 0u), Tb = B + 1 - (2 * c > rb ? 1u : 0u);
                        const uint32_t lo = Ta > t0 ? min(Ta - t0, 32u) : 0u, hi = Tb > t0 ? min(Tb - t0, 32u) : 0u;
                        un[c] = hi > lo ? (0xFFFFFFFFu >> (32 - (hi - lo))) << lo : 0u;
                    }
                }
                vp::word(win + kVBack + 32 * w + lane, un, std::make_index_sequence<8>());
                // the words still open into the queue
#pragma unroll
                for (uint32_t c = 0; c < GBC_NCLASS; ++c) {
                    const uint32_t bal = __ballot_sync(~0u, un[c] != 0u);
                    if (un[c]) {
                        const uint32_t at = qn + __popc(bal & ((1u << lane) - 1u));
                        q_bits[at] = un[c];
                        q_at[at] = uint16_t((c << 8) | (32 * w + lane));
                    }
                    qn += __popc(bal);
                }
                __syncwarp();
                settle(w + 1 == kVW || jw + 32 > jhi);
            }
        }
        __syncthreads();
    }
}

}  // namespace gbk

namespace gbh {

// The plan funnel of residue s that class r takes word by word is the one
// that holds all its primes p0 .. p0 + 930; the word form needs all three of
// every class in the plan.
bool verify_word_funnel(uint32_t r, uint32_t p0, uint32_t members)
{
    const uint32_t s = p0 % 30;
    if (p0 != gbk::vp::first_of(s)) return false;
    for (uint32_t d = 0; d < 32; ++d)
        if (gbk::vp::is_prime(p0 + 30 * d) && !(members >> d & 1u)) return false;
    for (uint32_t i = 0; i < 3; ++i)
        if (gbk::vp::residue(r, i) == s) return true;
    return false;
}

// CTAs of an unsampled segment: eight chunks of words per warp, fewer where
// that leaves the device short of CTAs
uint32_t verify_vbx(uint64_t evens, int sm)
{
    const uint64_t chunks = (evens / 15 / 32 + 4) / gbk::kVChunk + 2;  // one chunk more where it straddles
    const uint64_t most = (chunks + gbk::kVerifyWarps - 1) / gbk::kVerifyWarps;
    const uint64_t few = (chunks + 8 * gbk::kVerifyWarps - 1) / (8 * gbk::kVerifyWarps);
    const uint64_t bx = few > uint64_t(sm) * 2 ? few : most < uint64_t(sm) * 2 ? most : uint64_t(sm) * 2;
    return uint32_t(bx);
}

void launch_verify(const gbk::BatchDesc &d, const gbk::VerifyTables &vt, const Grids &g, cudaStream_t st)
{
    if (vt.word) gbk::k_verify<true><<<g.sm * g.verify, gbk::kVerifyThreads, gbk::kVerifySmem, st>>>(d, vt);
    else gbk::k_verify<false><<<g.sm * g.verify, gbk::kVerifyThreads, gbk::kVerifySmem, st>>>(d, vt);
}

void query_verify_grids(Grids &g)
{
    int n = 0;
    cudaFuncSetAttribute(gbk::k_verify<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gbk::kVerifySmem));
    cudaFuncSetAttribute(gbk::k_verify<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gbk::kVerifySmem));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gbk::k_verify<true>, gbk::kVerifyThreads, gbk::kVerifySmem);
    g.verify = n > 0 ? n : 1;
}

}  // namespace gbh
