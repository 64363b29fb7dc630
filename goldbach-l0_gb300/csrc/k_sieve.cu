// k_sieve.cu -- builds the mod-30 class maps of a batch on the GPU.
//
// Stages (the reference's make_prime_map, mid_setup/mid_window and
// sieve_large_packed, kernels/goldbach.cl:1092-1608, 3528-3701, 1738-1849,
// re-designed for HBM-resident maps, one per run of consecutive segments,
// and persistent kernels that take every run of the batch in one launch):
//   k_xfirst  per tile-sieve prime, class and run: the first class bit of
//             the run that is a multiple of p and >= p^2 (mid_setup's job,
//             goldbach.cl:3528-3563; host_math.cpp:80-113).
//   k_tile    one CTA per (run, class, tile) item: up to tile_bits bits in
//             shared memory; the primes 7..67 by whole-word AND patterns of
//             seven prime groups, then every prime 71..p_mid by shared-memory
//             atomics (small primes warp-cooperatively, the rest one per
//             thread); one coalesced store of the finished tile.
//   k_large   primes in (p_mid, p_hl), streamed at one byte per prime and
//             decoded by warps, every run they reach: every multiple p m (m
//             coprime to 30) by a global atomic AND after a read
//             (read-before-mark, goldbach.cl:328-336), stepping over the
//             multipliers with a factor 7..43, whose multiples the pattern
//             stage clears (the 30030 wheel and the 17..43 skip of
//             goldbach.cl:638-748).
//   k_hitlist the primes above p_hl through the prime-multiplier table.
//   k_map_finish the marks that no bin held; in runs narrow for their height
//             primality tests of what the tiles leave, in place of every
//             prime past them.
// A thread reads its prime once and applies it to every run of the batch,
// so a batch of many short windows streams the sieving primes once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gbc_common.cuh"

namespace gbk {

// x mod p, exactly, for x < p * 2^32 and 3 <= p < 2^32, without a
// division: a float estimate of the quotient (error below 2^11 for these
// bounds), an exact 64-bit remainder r (negative when the estimate was
// high), a second float estimate of the now small quotient r / p (error
// below 1), and a final +-p correction. rp = 1/p rounded to nearest.
__device__ __forceinline__ uint32_t mod_below(uint64_t x, uint32_t p, float rp)
{
    // float(x) from its two 32-bit halves (32-bit conversions only: 64-bit
    // integer <-> float conversions are multi-instruction sequences)
    const float xf = fmaf(__uint2float_rz(uint32_t(x >> 32)), 4294967296.0f, __uint2float_rz(uint32_t(x)));
    const uint32_t qe = __float2uint_rz(xf * rp);
    int64_t r = int64_t(x - uint64_t(qe) * p);
    // |r| < 2^43: float(|r|) from its halves as above, then the sign (the
    // halves of a negative r would lose up to 2^8 in the low word's
    // conversion, too much for p below 2^9)
    const uint64_t m = r < 0 ? uint64_t(-r) : uint64_t(r);
    const float mf = fmaf(__uint2float_rz(uint32_t(m >> 32)), 4294967296.0f, __uint2float_rz(uint32_t(m)));
    const float rf = r < 0 ? -mf : mf;
    const int32_t q2 = __float2int_rn(rf * rp);
    r -= int64_t(q2) * p;
    if (r < 0) r += p;
    if (r >= int64_t(p)) r -= p;
    return uint32_t(r);
}

// x mod p for any 64-bit x (two base-2^32 digits)
__device__ __forceinline__ uint32_t mod_u64(uint64_t x, uint32_t p, float rp)
{
    const uint32_t hi = uint32_t(x >> 32);
    const uint32_t r = hi < p ? hi : mod_below(hi, p, rp);
    return mod_below((uint64_t(r) << 32) | uint32_t(x), p, rp);
}

// a + d mod p for a, d < p without overflow
__device__ __forceinline__ uint32_t addmod(uint32_t a, uint32_t d, uint32_t p)
{
    return a >= p - d ? a - (p - d) : a + d;
}

// First class bit, for each class k, of a multiple of p in the run with
// q >= p^2; kNone when the first one is at or past nblk. 29 < p < 2^31.
__device__ __forceinline__ void first_bits8(uint64_t base, uint32_t nblk, uint32_t p, uint32_t *out)
{
    const float rp = __frcp_rn(float(p));
    const uint32_t r = mod_u64(base, p, rp);
    const uint32_t iv = inv30_mod(p);
    const uint64_t pp = uint64_t(p) * p;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t u = unit30(k);
        uint32_t a = r + u;                                  // (base + u) mod p
        if (a >= p) a -= p;
        a = a ? p - a : 0;                                   // -(base + u) mod p
        uint64_t t = mod_below(uint64_t(a) * iv, p, rp);     // base + 30 t + u = 0 (mod p)
        const uint64_t q = base + 30 * t + u;
        if (q < pp) {                                        // p itself and smaller multiples stay unmarked
            const uint64_t tmin = (pp - base - u + 29) / 30;
            if (tmin > t) t += (tmin - t + p - 1) / p * p;
        }
        out[k] = t < nblk ? uint32_t(t) : kNone;
    }
}

// every run's first bits of the tile-sieve primes
__global__ void __launch_bounds__(256) k_xfirst(BatchDesc d)
{
    const uint32_t nrun = d.h->nrun, nmax = d.h->n_mid_max;
    if (!nrun) return;
    const uint32_t *primes = d.runs[0].primes;
    for (uint32_t i = d.runs[0].i0 + blockIdx.x * blockDim.x + threadIdx.x; i < nmax; i += gridDim.x * blockDim.x) {
        const uint32_t p = primes[i];
        for (uint32_t r = 0; r < nrun; ++r) {
            const BatchParams &bp = d.runs[r];
            const uint32_t n = bp.n_mid;
            if (i >= n) continue;
            uint32_t x[8];
            first_bits8(bp.base, bp.nblk, p, x);
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) bp.xfirst[size_t(k) * n + i] = x[k];
        }
    }
}

// the same for one run passed by value
__global__ void __launch_bounds__(256) k_xfirst1(BatchParams bp)
{
    const uint32_t n = bp.n_mid;
    for (uint32_t i = bp.i0 + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t x[8];
        first_bits8(bp.base, bp.nblk, bp.primes[i], x);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) bp.xfirst[size_t(k) * n + i] = x[k];
    }
}

// Tile-local first mark of a prime from its run-level first bit x.
__device__ __forceinline__ uint32_t local_start(uint32_t x, uint32_t t0, uint32_t p, uint32_t magic, uint32_t tb)
{
    if (x == kNone) return kNone;
    if (x >= t0) {
        const uint32_t d = x - t0;
        return d < tb ? d : kNone;
    }
    const uint32_t d = t0 - x;
    const uint32_t q = __umulhi(d, magic);  // floor(d / p) or one less
    uint32_t rem = d - q * p;
    if (rem >= p) rem -= p;
    return rem ? p - rem : 0;
}

// Tile-bin staging of the persistent tile kernel: the first `cap` offsets
// of an item's tile bin (cap: what the shared memory beside the tile holds,
// up to kTbStage, a multiple of kTbPiece, possibly 0) go into shared memory
// by bulk copies issued at the item's start (they land while the CTA
// sieves), the rest is prefetched into L2 by the TMA unit and read from
// there.
constexpr uint32_t kTbStage = 20480;       // offsets (80 KB), a multiple of kTbPiece
constexpr uint32_t kTbPiece = 4096;        // offsets per bulk copy (16 KB)

// thread 0 at an item's start: stages the first min(n, cap) offsets of the
// tile bin e (n offsets; the copy rounded up to 16 bytes, which stays in the
// bin: capacities are multiples of 32 offsets) into stg, completing on bar,
// and prefetches the rest into L2. Returns the offsets staged.
__device__ __forceinline__ uint32_t stage_tile_bin(uint32_t *stg, uint64_t *bar, const uint32_t *e, uint32_t n,
                                                   uint32_t cap)
{
    const uint32_t staged = min(n, cap);
    if (n > cap) bulk_prefetch_l2(e + cap, ((n - cap + 3u) & ~3u) * 4u);
    if (!staged) return 0;
    const uint32_t words = (staged + 3u) & ~3u;
    fence_proxy_async();  // the CTA's earlier reads of stg before the copies
    mbar_arrive_expect_tx(bar, words * 4u);
    for (uint32_t w0 = 0; w0 < words; w0 += kTbPiece)
        bulk_copy_g2s(stg + w0, e + w0, min(kTbPiece, words - w0) * 4u, bar);
    return staged;
}

// Bits of the shared-memory tile as the marks address them: bit b of the tile
// is b + 8 x (the tile's shared-memory address), so a mark's word address is
// that >> 3 without its low two bits and the base needs no addition of its own
// (the tile starts 16-byte aligned: the bit in the word is unchanged).
__device__ __forceinline__ uint32_t tile_bit0(const uint32_t *s) { return 8u * smem_addr(s); }

// Clears a bit so addressed: ~(1 << (b mod 32)) as one funnel-shift rotation of
// ~1. (128 segments of 467.5M on one GB300: the tile stage 10.62 -> 10.29 ms
// against an atomicAnd on a pointer; the kernel then waits for the shared
// memory's wavefronts, 71% of its cycles.)
__device__ __forceinline__ void clear_bit(uint32_t b)
{
    asm volatile("red.shared::cta.and.b32 [%0], %1;" ::"r"((b >> 3) & ~3u),
                 "r"(__funnelshift_l(0xFFFFFFFEu, 0xFFFFFFFEu, b))
                 : "memory");
}

// Clears bits b, b + st, b + 2 st, ... below end, four marks per bound check.
// b + 3 st < 2^32: a lane's own prime has b < end < 2^22 and st <=
// kMaxTilePrime, a prime of a whole warp b < end + st and st < 2^20.
static_assert(8u * (228u << 10) + 1835008u < 1u << 22, "bits of the largest tile in shared memory");
static_assert((1ull << 22) + 3ull * kMaxTilePrime <= 1ull << 32, "three strides past a tile's end");
__device__ __forceinline__ void clear_stride(uint32_t b, uint32_t st, uint32_t end)
{
    for (; b + 3u * st < end; b += 4u * st) {
        clear_bit(b);
        clear_bit(b + st);
        clear_bit(b + 2u * st);
        clear_bit(b + 3u * st);
    }
    for (; b < end; b += st) clear_bit(b);
}

// Sieves bits [t0, t0 + tl) of class array k of a run in shared memory s
// (the group patterns already in pat) and stores them: tile ti of the class
// array, tb bits per tile (the buffer s holds tb bits), tl <= tb a multiple
// of 128 bits. Ends with the CTA synchronized, s free for the next tile.
// kVec4: the context's own prime and reciprocal arrays (16-byte aligned,
// padded by 4 words), read four at a time, and the tile bin staged by
// stage_tile_bin (*nb offsets, the first min(*nb, cap) in stg once bar
// completes the phase of parity bit 0 of phase); otherwise any arrays and
// the tile bin read from global memory.
template <bool kVec4>
__device__ __forceinline__ void tile_body(const BatchParams &bp, const GroupInfo &gi, const uint32_t *pat,
                                          uint32_t *s, uint32_t k, uint32_t ti, uint32_t t0, uint32_t tl,
                                          uint32_t tb, const uint32_t *stg = nullptr, uint64_t *bar = nullptr,
                                          uint32_t *phase = nullptr, const uint32_t *nb = nullptr, uint32_t cap = 0)
{
    const uint32_t tid = threadIdx.x, bs = blockDim.x;
    const uint32_t tw = tl >> 5;
    const uint64_t q0 = bp.base + 30ull * t0 + unit30(k);

    // phase of this thread's first word in each group's canonical pattern:
    // local bit x is cleared by the group iff (x + c) mod P has a factor in
    // the group, c = (P - Y) mod P, Y = -q0 / 30 (mod P)
    uint32_t ph[kNumGroups], stp[kNumGroups];
#pragma unroll
    for (int g = 0; g < kNumGroups; ++g) {
        const uint32_t P = gi.P[g];
        const uint32_t qm = uint32_t(q0 % P);
        const uint32_t y = uint32_t(uint64_t((P - qm) % P) * gi.inv30[g] % P);
        const uint32_t c = (P - y) % P;
        ph[g] = uint32_t((32ull * tid + c) % P);
        stp[g] = uint32_t((32ull * bs) % P);
    }
    for (uint32_t w = tid; w < tw; w += bs) {
        uint32_t v = ~0u;
#pragma unroll
        for (int g = 0; g < kNumGroups; ++g) {
            const uint32_t *pg = pat + gi.off[g];
            const uint32_t x = ph[g];
            v &= __funnelshift_r(pg[x >> 5], pg[(x >> 5) + 1], x & 31);
            uint32_t nx = x + stp[g];
            if (nx >= gi.P[g]) nx -= gi.P[g];
            ph[g] = nx;
        }
        s[w] = v;
    }
    __syncthreads();
    if (tid == 0 && q0 < 4096) {
        // the pattern primes are prime themselves; 1 is not
        const uint32_t small[16] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67};
        for (int i = 0; i < 16; ++i) {
            const uint32_t p = small[i];
            if (p % 30 == unit30(k) && p >= q0) {
                const uint32_t b = uint32_t((p - q0) / 30);
                if (b < tl) s[b >> 5] |= 1u << (b & 31);
            }
        }
        if (q0 == 1) s[0] &= ~1u;
    }
    __syncthreads();

    const uint32_t lane = tid & 31, warp = tid >> 5, nw = bs >> 5, s0 = tile_bit0(s);
    const uint32_t *xk = bp.xfirst + size_t(k) * bp.n_mid;
    // small primes: a warp per prime, lanes take every 32nd multiple
    for (uint32_t i = bp.i0 + warp; i < bp.i_warp; i += nw) {
        const uint32_t p = bp.primes[i];
        const uint32_t l = local_start(xk[i], t0, p, bp.magic[i], tl);
        if (l >= tl) continue;
        clear_stride(s0 + l + lane * p, 32u * p, s0 + tl);
    }
    if constexpr (kVec4) {
        // the rest: four consecutive primes per thread and round, their
        // primes and reciprocals as one 16-byte load each and their first
        // bits as four loads, all issued before any of their marks (one L2
        // round trip per four primes)
        const uint32_t n = bp.n_mid, i_lo = bp.i_warp, c_lo = i_lo & ~3u;
        for (uint32_t i = c_lo + 4 * tid; i < n; i += 4 * bs) {
            const uint4 p4 = __ldg(reinterpret_cast<const uint4 *>(bp.primes + i));
            const uint4 m4 = __ldg(reinterpret_cast<const uint4 *>(bp.magic + i));
            uint32_t x4[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) x4[u] = i + u < n ? __ldg(xk + i + u) : kNone;
            const uint32_t pv[4] = {p4.x, p4.y, p4.z, p4.w}, mv[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (i + u < i_lo) continue;
                const uint32_t p = pv[u];
                const uint32_t l = local_start(x4[u], t0, p, mv[u], tl);
                if (l < tl) clear_stride(s0 + l, p, s0 + tl);
            }
        }
    } else {
        // the rest: four primes per thread and round, their loads all issued
        // before any of their marks
        const uint32_t n = bp.n_mid;
        for (uint32_t i = bp.i_warp + tid; i < n; i += 4 * bs) {
            uint32_t pv[4], xv[4], mv[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t j = min(i + u * bs, n - 1);
                pv[u] = __ldg(bp.primes + j);
                xv[u] = i + u * bs < n ? __ldg(xk + j) : kNone;
                mv[u] = __ldg(bp.magic + j);
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t l = local_start(xv[u], t0, pv[u], mv[u], tl);
                if (l < tl) clear_stride(s0 + l, pv[u], s0 + tl);
            }
        }
    }
    // a binned batch: the hit-list marks of this tile (offsets within it,
    // clamped to the tile buffer: a stale staged word or a damaged bin can
    // clear a wrong bit, never touch memory outside s)
    const uint32_t omax = tb - 1;
    if constexpr (kVec4) {
        const uint32_t n = *nb, staged = min(n, cap);
        if (staged) {
            bool ok = mbar_wait(bar, *phase & 1u, bp.spin0);
            if (!ok) {
                atomicOr(bp.err, kErrStaging);
                ok = mbar_wait(bar, *phase & 1u);
            }
            *phase ^= 1u;
            const uint4 *v4 = reinterpret_cast<const uint4 *>(stg);
            for (uint32_t i = tid; ok && 4 * i < staged; i += bs) {
                const uint4 v = v4[i];
                const uint32_t at = 4 * i;
                clear_bit(s0 + min(v.x, omax));
                if (at + 1 < staged) clear_bit(s0 + min(v.y, omax));
                if (at + 2 < staged) clear_bit(s0 + min(v.z, omax));
                if (at + 3 < staged) clear_bit(s0 + min(v.w, omax));
            }
        }
        if (n > cap) {
            // the rest from L2, four groups of four per thread in flight
            const uint32_t tile = k * bp.tb_tiles + bp.tb_vt0 + ti, m = n - cap;
            const uint4 *e = reinterpret_cast<const uint4 *>(bp.tb_buf + size_t(tile) * bp.tb_cap + cap);
            for (uint32_t i = tid; 4 * i < m; i += 4 * bs) {
                uint4 v[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t g = i + u * bs;
                    v[u] = 4 * g < m ? __ldcs(e + g) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t at = 4 * (i + u * bs);
                    if (at < m) clear_bit(s0 + min(v[u].x, omax));
                    if (at + 1 < m) clear_bit(s0 + min(v[u].y, omax));
                    if (at + 2 < m) clear_bit(s0 + min(v[u].z, omax));
                    if (at + 3 < m) clear_bit(s0 + min(v[u].w, omax));
                }
            }
        }
    } else if (bp.tb_cap && bp.hl_quota) {
        const uint32_t tile = k * bp.tb_tiles + bp.tb_vt0 + ti;
        const uint32_t n = min(__ldcg(bp.tb_cnt + tile), bp.tb_cap);
        const uint4 *e = reinterpret_cast<const uint4 *>(bp.tb_buf + size_t(tile) * bp.tb_cap);
        // four groups of four per thread in flight before their marks
        for (uint32_t i = tid; 4 * i < n; i += 4 * bs) {
            uint4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t g = i + u * bs;
                v[u] = 4 * g < n ? __ldcs(e + g) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t at = 4 * (i + u * bs);
                if (at < n) clear_bit(s0 + min(v[u].x, omax));
                if (at + 1 < n) clear_bit(s0 + min(v[u].y, omax));
                if (at + 2 < n) clear_bit(s0 + min(v[u].z, omax));
                if (at + 3 < n) clear_bit(s0 + min(v[u].w, omax));
            }
        }
    }
    __syncthreads();
    uint4 *dst = reinterpret_cast<uint4 *>(bp.map + size_t(k) * bp.wpc + (t0 >> 5));
    const uint4 *src = reinterpret_cast<const uint4 *>(s);
    for (uint32_t i = tid; i < tw / 4; i += bs) dst[i] = src[i];
    __syncthreads();
}

// Persistent tile kernel: CTAs take the batch's (run, class, tile) items
// from a work counter; tiles of tb bits (a multiple of 128), a run's last
// tile of a class ends at its class array's end; up to kCap offsets of each
// tile bin staged into shared memory. kCap is a compile-time constant: with
// it as a runtime parameter the kernel measured 3.7 times slower (47.9
// against 13.05 ms per 128-segment batch at 2^20-bit tiles, one GB300).
template <uint32_t kCap>
__global__ void __launch_bounds__(1024, 1) k_tile(BatchDesc d, GroupInfo gi, uint32_t tb)
{
    constexpr uint32_t cap = kCap;
    // shared memory: the tile, the tile-bin staging buffer, the patterns
    extern __shared__ __align__(16) uint32_t sm_tile[];
    uint32_t *s = sm_tile;
    uint32_t *stg = sm_tile + (tb >> 5);
    uint32_t *pat = stg + cap;
    const uint32_t nrun = d.h->nrun, items = d.h->tile_items;
    if (!nrun) return;
    __shared__ uint32_t s_j, s_nb;
    __shared__ uint64_t s_bar;
    if (threadIdx.x == 0) {
        mbar_init(&s_bar, 1);
        mbar_init_fence();
    }
    uint32_t phase = 0;
    for (uint32_t i = threadIdx.x; i < gi.words; i += blockDim.x) pat[i] = d.runs[0].pat[i];
    for (;;) {
        const uint32_t j = next_item(d.work + kWorkTile, &s_j);  // synchronizes the CTA
        if (j >= items) break;
        const uint32_t r = find_prefix(d.tile_pref, nrun, j);
        const BatchParams &bp = d.runs[r];
        // items tile-major within a run: a tile's eight classes side by side,
        // so the tiles of one segment are one range of items
        const uint32_t local = j - __ldg(d.tile_pref + r);
        const uint32_t k = local & 7u, ti = local >> 3, t0 = ti * tb;
        const uint32_t tl = min(tb, bp.wpc * 32 - t0);
        if (threadIdx.x == 0) {
            uint32_t n = 0;
            if (bp.tb_cap && bp.hl_quota) {
                const uint32_t tile = k * bp.tb_tiles + bp.tb_vt0 + ti;
                n = min(__ldcg(bp.tb_cnt + tile), bp.tb_cap);
                stage_tile_bin(stg, &s_bar, bp.tb_buf + size_t(tile) * bp.tb_cap, n, cap);
            }
            s_nb = n;
        }
        tile_body<true>(bp, gi, pat, s, k, ti, t0, tl, tb, stg, &s_bar, &phase, &s_nb, cap);
    }
}

// the staging capacities the host chooses from (the largest that fits)
constexpr uint32_t kTbStages[3] = {kTbStage, 2 * kTbPiece, 0};
template __global__ void k_tile<kTbStages[0]>(BatchDesc, GroupInfo, uint32_t);
template __global__ void k_tile<kTbStages[1]>(BatchDesc, GroupInfo, uint32_t);
template __global__ void k_tile<kTbStages[2]>(BatchDesc, GroupInfo, uint32_t);

// one run by value: grid (ceil(32 wpc / tile_bits), 8), the last tile of a class array cut short
__global__ void __launch_bounds__(1024, 1) k_tile1(BatchParams bp, GroupInfo gi)
{
    extern __shared__ uint32_t sm[];
    const uint32_t tb = bp.tile_bits, t0 = blockIdx.x * tb;
    uint32_t *pat = sm + (tb >> 5);
    for (uint32_t i = threadIdx.x; i < gi.words; i += blockDim.x) pat[i] = bp.pat[i];
    __syncthreads();
    tile_body<false>(bp, gi, pat, sm, blockIdx.y, blockIdx.x, t0, min(tb, bp.wpc * 32 - t0), tb);
}

// The packed large-prime tier (the reference's pack_large_primes,
// decode_large and large_packed_body, src/host_math.cpp:187-209,
// kernels/goldbach.cl:1678-1829 with the wheel walk of 638-748, in this
// repository's own form): the primes of [p_mid, p_hl) stream at one byte per
// prime, a half gap (p_i - p_{i-1}) / 2, with the first prime of every group
// of kPackGroup primes in a table of its own; a warp decodes a group (lane
// l: eight primes, its gap bytes as one 8-byte load, the group's running sum
// by a warp scan). Each prime then marks every run it reaches, class by
// class: the multiples q = p m of class k are the bits t0, t0 + p, t0 + 2 p,
// ... with m = m0 + 30 j. Multipliers with a factor 7, 11 or 13 are stepped
// over by a wheel mod 7 * 11 * 13 = 1001 (720 steps in 1001; inside one class
// array this is the reference's 30030 wheel, whose factor 30 the class
// layout already holds); multipliers with a factor 17..43 are skipped by a
// test of their residues, four 8-bit lanes per word. Either way q has a prime
// factor the pattern stage clears. A mark reads the word and clears the bit
// with an atomic AND only if it is still set.
constexpr uint32_t kWheelUnits = 720;          // residues mod 1001 coprime to it
constexpr uint32_t kSkipLanes1 = 0x1D171311u;  // 17, 19, 23, 29 as bytes
constexpr uint32_t kSkipLanes2 = 0x2B29251Fu;  // 31, 37, 41, 43
constexpr uint32_t kSkipBias1 = 0x63696D6Fu;   // 128 - 17, 128 - 19, 128 - 23, 128 - 29
constexpr uint32_t kSkipBias2 = 0x55575B61u;   // 128 - 31, 128 - 37, 128 - 41, 128 - 43

// per byte lane, (x + d) mod f for lanes x < f and d <= 4: add, then subtract
// f where the sum reached f (the bias 128 - f carries that into bit 7)
__device__ __forceinline__ uint32_t lanes_step(uint32_t x, uint32_t d, uint32_t f, uint32_t bias)
{
    x += d * 0x01010101u;
    const uint32_t ge = ((x + bias) >> 7) & 0x01010101u;
    return x - ((ge * 0xFFu) & f);
}

// nonzero iff some byte lane of x is zero
__device__ __forceinline__ uint32_t lanes_zero(uint32_t x) { return (x - 0x01010101u) & ~x & 0x80808080u; }

// Marks the multiples of p in one class array wk of nblk bits from bit t on.
// c = m0 / 30 mod 1001 and the lanes r1 (17..29), r2 (31..43) = m0 / 30 mod
// f for the multiplier m0 of bit t, so that m0 + 30 j has the factor f iff
// (c + j) or lane f of r + j is 0 mod f. wheel[x], x < 1001: the rank of the
// first unit >= x (wrapping) | its distance << 10; wheel[1001 + rank]: the
// gap from that unit to the next.
__device__ __forceinline__ void large_walk(uint32_t *wk, uint32_t nblk, uint32_t t, uint32_t p, uint32_t c,
                                           uint32_t r1, uint32_t r2, const uint16_t *wheel)
{
    const uint32_t e = wheel[c];
    uint32_t rank = e & 1023u;
    const uint32_t d0 = e >> 10;
    if (d0) {
        if (uint64_t(nblk - t) <= uint64_t(d0) * p) return;
        t += d0 * p;
        r1 = lanes_step(r1, d0, kSkipLanes1, kSkipBias1);
        r2 = lanes_step(r2, d0, kSkipLanes2, kSkipBias2);
    }
    for (;;) {
        if (!(lanes_zero(r1) | lanes_zero(r2))) {
            uint32_t *a = wk + (t >> 5);
            const uint32_t bit = 1u << (t & 31);
            if (__ldcg(a) & bit) atomicAnd(a, ~bit);
        }
        const uint32_t g = wheel[kWheelM + rank];
        if (uint64_t(nblk - t) <= uint64_t(g) * p) break;
        t += g * p;
        rank = rank + 1 == kWheelUnits ? 0u : rank + 1;
        r1 = lanes_step(r1, g, kSkipLanes1, kSkipBias1);
        r2 = lanes_step(r2, g, kSkipLanes2, kSkipBias2);
    }
}

// The packed large primes [n_mid, n_hl) of every run: a CTA per item of 32
// consecutive primes, a thread per (prime, class) walk, so that every walk of
// a batch (about eight per prime) runs side by side (the walks wait on
// global memory; a thread per prime walking its classes in turn measured
// about half the pipeline's speed with 46 K primes on this tier). Warp 0
// decodes the item's packing group (lane l: eight primes from one 8-byte
// load, the group's running sum by a warp scan) into shared memory.
constexpr uint32_t kLargeItem = 32;  // primes per CTA item; kPackGroup / kLargeItem items per group
__global__ void __launch_bounds__(256) k_large(BatchDesc d)
{
    __shared__ uint16_t s_wheel[kWheelTabWords];
    __shared__ uint32_t s_p[kLargeItem];
    const uint32_t nrun = d.h->nrun;
    if (!nrun) return;
    const BatchParams &b0 = d.runs[0];
    // runs whose large range is empty may have n_mid below the stream's start
    const uint32_t lo = max(d.h->n_mid_min, b0.pk_i0), hi = d.h->n_hl_max;
    if (lo >= hi) return;
    for (uint32_t i = threadIdx.x; i < kWheelTabWords; i += blockDim.x) s_wheel[i] = b0.wheel[i];
    const uint16_t *s_inv = s_wheel + kWheelM + kWheelUnits;  // x^-1 mod 1001 (0: none)
    const uint16_t *s_invf = s_inv + kWheelM;                  // x^-1 mod f, f = 17..43 back to back
    constexpr uint32_t kF[8] = {17, 19, 23, 29, 31, 37, 41, 43};
    constexpr uint32_t kFo[8] = {0, 17, 36, 59, 88, 119, 156, 197};
    const uint32_t tid = threadIdx.x, lane = tid & 31, i0 = b0.pk_i0;
    const uint32_t j_lo = (lo - i0) / kLargeItem, j_hi = (hi - i0 + kLargeItem - 1) / kLargeItem;
    const uint32_t k = tid & 7;        // this thread's class
    const uint32_t slot = tid >> 3;    // and prime of the item
    for (uint32_t j = j_lo + blockIdx.x; j < j_hi; j += gridDim.x) {
        __syncthreads();  // the wheel table loaded; the last item's primes read
        if (tid < 32) {
            const uint32_t g = j / (kPackGroup / kLargeItem), sl = j % (kPackGroup / kLargeItem);
            const uint2 gv = __ldg(reinterpret_cast<const uint2 *>(b0.pk_gap) + size_t(g) * (kPackGroup / 8) + lane);
            uint32_t sum = 0;
#pragma unroll
            for (uint32_t b = 0; b < 32; b += 8) sum += ((gv.x >> b) & 0xFFu) + ((gv.y >> b) & 0xFFu);
            uint32_t incl = sum;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(~0u, incl, o);
                if (lane >= o) incl += y;
            }
            uint32_t p = __ldg(b0.pk_base + g) + 2u * (incl - sum);
            const uint32_t first = sl * (kLargeItem / 8);  // the lanes of this item's slice of the group
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
                p += 2u * (((u < 4 ? gv.x : gv.y) >> (8 * (u & 3))) & 0xFFu);
                if (lane >= first && lane < first + kLargeItem / 8) s_p[(lane - first) * 8 + u] = p;
            }
        }
        __syncthreads();
        const uint32_t i = i0 + j * kLargeItem + slot;
        if (i < lo || i >= hi) continue;
        const uint32_t p = s_p[slot];
        const float rp = __frcp_rn(float(p));
        const uint32_t iv = inv30_mod(p);
        const uint32_t uk = unit30(k);
        const uint32_t ck = mod_below(uint64_t(uk) * iv, p, rp);  // u_k / 30 mod p
        // (30 p)^-1 mod 1001 and mod each skip prime f
        const uint32_t a1001 = s_inv[30u * (p % kWheelM) % kWheelM];
        uint32_t af[8];
#pragma unroll
        for (uint32_t jj = 0; jj < 8; ++jj) af[jj] = s_invf[kFo[jj] + 30u * (p % kF[jj]) % kF[jj]];
        for (uint32_t ri = 0; ri < nrun; ++ri) {
            const BatchParams &bp = d.runs[ri];
            if (i < bp.n_mid || i >= bp.n_hl) continue;
            // run 0's window (the plain form's per-segment launches):
            // bits [b0, b1), b0 a multiple of 32, as a run of its own
            const uint32_t w0 = ri ? 0u : d.h->win_b0, w1 = ri ? bp.nblk : min(bp.nblk, d.h->win_b1);
            if (w0 >= w1) continue;
            const uint64_t base = bp.base + 30ull * w0;
            const uint32_t nblk = w1 - w0;
            const uint32_t r = mod_u64(base, p, rp);
            // t_k = -(base + u_k) / 30 mod p = tb - c_k, tb = -base / 30
            const uint32_t tb = mod_below(uint64_t(r ? p - r : 0) * iv, p, rp);
            uint32_t tk = tb >= ck ? tb - ck : tb + (p - ck);
            if (uint64_t(p) * p > base) {  // only near the bottom of the range: q >= p^2
                const uint64_t pp = uint64_t(p) * p;
                const uint64_t q = base + 30ull * tk + uk;
                if (q < pp) {
                    const uint64_t tmin = (pp - base - uk + 29) / 30;
                    const uint64_t tt = tk + (tmin - tk + p - 1) / p * p;
                    tk = tt < nblk ? uint32_t(tt) : kNone;
                }
            }
            if (tk >= nblk) continue;
            // m0 = q0 / p with q0 = base + 30 tk + u_k, so m0 / 30 = q0 (30 p)^-1
            // mod 1001 and mod f (the run base's residues, moved to the window)
            const uint32_t bm1 = (bp.bm1 + 30u * (w0 % kWheelM)) % kWheelM;
            const uint32_t c = (bm1 + 30u * (tk % kWheelM) + uk) % kWheelM * a1001 % kWheelM;
            uint32_t r1 = 0, r2 = 0;
#pragma unroll
            for (uint32_t jj = 0; jj < 8; ++jj) {
                const uint32_t f = kF[jj];
                const uint32_t bf = (uint32_t(bp.bres[jj]) + 30u * (w0 % f)) % f;
                const uint32_t q = (bf + 30u * (tk % f) + uk) % f;
                const uint32_t rho = q * af[jj] % f;
                if (jj < 4) r1 |= rho << (8 * jj);
                else r2 |= rho << (8 * (jj - 4));
            }
            large_walk(bp.map + size_t(k) * bp.wpc + (w0 >> 5), nblk, tk, p, c, r1, r2, s_wheel);
        }
    }
}

// floor(2^64 / p), or up to four less, for a prime 3 <= p < 2^32: the hit lists'
// reciprocal. From 2^20 on without a division: a float estimate of 2^52 / p
// (error below 2^13 of it), scaled by 2^12 and corrected by the float estimate
// of what it leaves; the corrected value is within two of 2^64 / p, so two less
// never exceeds it.
__device__ __forceinline__ uint64_t recip64(uint32_t p, float rp)
{
    if (p < (1u << 20)) return 0xFFFFFFFFFFFFFFFFull / p;
    const uint32_t q1 = __float2uint_rz(rp * 4503599627370496.0f);  // 2^52 / p, saturated below 2^32
    const int64_t d = int64_t((1ull << 52) - uint64_t(q1) * p);     // |d| < 2^33
    const int32_t c = __float2int_rn(__int2float_rn(int32_t(d >> 2)) * (rp * 16384.0f));
    return (uint64_t(q1) << 12) + uint64_t(int64_t(c)) - 2;
}

// floor(2^64 / p) itself, from recip64
__device__ __forceinline__ uint64_t recip64_exact(uint32_t p, uint64_t inv)
{
    uint64_t e = 0 - inv * p;  // 2^64 - inv p < 5 p
#pragma unroll
    for (uint32_t step = 2; step; step >>= 1)
        if (e >= uint64_t(p) * step) {
            e -= uint64_t(p) * step;
            inv += step;
        }
    return e >= p ? inv + 1 : inv;
}

// floor(x / p) and x mod p for x < 2^60 and inv = recip64(p): the high half
// of x inv is the quotient or one less (x (2^64 / p - inv) / 2^64 < 1 / 2).
// The remainder before the correction is below 2 p: 32 bits hold it for
// p < 2^31.
__device__ __forceinline__ uint64_t divmod_recip(uint64_t x, uint32_t p, uint64_t inv, uint32_t &rem)
{
    const uint64_t q = __umul64hi(x, inv);
    uint32_t r = uint32_t(x) - uint32_t(q) * p;
    bool more;
    if (p >> 31) more = x - q * p >= p;
    else more = r >= p;
    if (more) r -= p;
    rem = r;
    return q + (more ? 1u : 0u);
}

// Hit lists through the prime-multiplier table (the reference's mt_build /
// hl_harvest_mt / hl_apply, kernels/goldbach.cl:3181-3471): for a prime
// p >= cbrt(q), a composite multiplier m of q = p m has a prime factor below
// p, which marks q already, so only prime m matter. One thread per prime
// p and run; each prime m of the run's multiplier range gives q = p m, whose
// class bit is cleared with an atomic AND. Every such q is a semiprime whose
// factors are both above the sieving bound of the other stages, so the bit
// is set and no read is needed.
//
// In class bits: with B = base / 30 (base a multiple of 30) and m = 30 b +
// u_k (byte b of the table, bit k), q = p m is bit p b + floor(p u_k / 30) -
// B of the class of p u_k mod 30. So one division per (prime, run), B = p b0
// + rho, places every mark: byte b holds the bits p (b - b0) + v_k - rho,
// v_k = floor(p u_k / 30) = (p / 30) u_k + floor((p mod 30) u_k / 30), in
// 32-bit arithmetic, and a mark belongs to the run iff its bit is below
// nblk (no masks over the end bytes). A run narrower than p / 4 bits holds a
// few multiples of p, from m = 30 b0 + j on, j the least with floor(p j / 30)
// >= rho (at most one where it is narrower than p / 32): a pair reads the table
// only for those that are units and inside the run, and most pairs of a narrow
// run end without a read.
__device__ __forceinline__ void ovf_push(const BatchParams &bp, uint32_t k, uint32_t t)
{
    const uint32_t slot = atomicAdd(bp.ovf_cnt, 1u);
    if (slot < bp.ovf_cap) bp.ovf_buf[slot] = make_uint2(k, t);
}

// Bound by issue (68% on one 467.5M segment) and, where p is below the run's
// width, by the table's random sectors. Measured against a pair that divided
// base and base + span apart, took byte bounds and masks with 64-bit divisions
// by 30 and placed each mark with 64-bit arithmetic (one GB300, harvest and
// sort): one segment 1.27 -> 0.66 ms, 8 segments 1.63 -> 1.14, 128 segments
// 8.13 -> 6.8, 292 segments of uneven windows 75.1 -> 36.9. Of that the units
// tested before the table is read (runs narrower than p / 4): one segment 0.75
// -> 0.70, 8 segments 1.40 -> 1.24, the windows 46.6 -> 42.5. Few, large CTAs: every CTA
// writes one stream per region bin, and the streams share the L2: 2 x 768
// threads 7.04 ms per 128 segments, 3 x 512 7.37, 4 x 384 8.17, 5 x 256
// 8.38, 1 x 1024 7.76.
constexpr int kHlThreads = 768, kHlCtas = 2;

// What the harvest reads of a run: of most pairs the first 16 bytes.
struct __align__(16) HlRun {
    uint64_t below;      // base - 1
    uint32_t span;       // 30 nblk - 1, or 2^32 - 1 where that is more
    uint32_t n_all;      // 0: no hit-listed prime
    uint64_t B;          // base / 30
    uint32_t nblk;
    uint32_t place;      // the run's first virtual bit (binned), or its number
};

// direct = 0: a binned batch's harvest (launched before the tiles); direct =
// 1: every other batch's direct marks (launched after the tiles)
__global__ void __launch_bounds__(kHlThreads, kHlCtas) k_hitlist(BatchDesc d, uint32_t direct)
{
    const uint32_t nrun = d.h->nrun;
    if (!nrun) return;
    const bool binned = hl_binned(d.runs[0]);
    if (binned == (direct != 0)) return;
    const BatchParams &run0 = d.runs[0];
    const uint32_t nhi = d.h->n_all_max;
    const uint32_t quota = binned ? run0.hl_quota : 0u;
    const uint32_t rlog = run0.hl_rlog, nreg = run0.hl_nreg, nbin = 8 * nreg;
    // per (class of p, class of m): u_m | floor((p mod 30) u_m / 30) << 8 |
    // the class kq of q = p m << 16 (kq * nreg, its first region bin, << 20);
    // the class of a residue
    __shared__ uint32_t s_cls[8][8];
    __shared__ uint8_t s_res[32];
    __shared__ uint32_t s_hcnt[kHlMaxBins];
    // the runs, those that most primes reach first
    __shared__ HlRun s_run[256];
    __shared__ uint32_t s_n[256];
    __shared__ uint32_t s_lo;
    if (threadIdx.x == 0) s_lo = kNone;
    __syncthreads();
    if (threadIdx.x < 64) {
        const uint32_t a = threadIdx.x >> 3, b = threadIdx.x & 7;
        const uint32_t x = unit30(a) * unit30(b), kq = class_of(x % 30);
        s_cls[a][b] = unit30(b) | (x / 30 << 8) | (kq << 16) | ((binned ? kq * nreg : 0u) << 20);
    } else if (threadIdx.x < 96) {
        s_res[threadIdx.x - 64] = uint8_t(class_of(threadIdx.x - 64));
    }
    if (threadIdx.x < kHlMaxBins) s_hcnt[threadIdx.x] = 0;
    if (threadIdx.x < nrun) {
        const BatchParams &bp = d.runs[threadIdx.x];
        s_n[threadIdx.x] = bp.n_hl < bp.n_all ? bp.n_all : 0u;
    }
    __syncthreads();
    if (threadIdx.x < nrun) {
        const BatchParams &bp = d.runs[threadIdx.x];
        const uint32_t n = s_n[threadIdx.x];
        uint32_t r = 0;  // the run's place
        for (uint32_t o = 0; o < nrun; ++o) r += s_n[o] > n || (s_n[o] == n && o < threadIdx.x) ? 1u : 0u;
        HlRun x{};
        x.below = bp.base - 1;  // (base 0: a run of a few small q, wide against every p)
        x.span = uint32_t(min(30ull * bp.nblk - 1, 0xFFFFFFFFull));
        x.n_all = n;
        x.B = bp.base / 30;
        x.nblk = bp.nblk;
        if (x.n_all) atomicMin(&s_lo, bp.n_hl);  // the same for every run that has some
        x.place = binned ? bp.tb_vt0 * run0.tile_bits : threadIdx.x;
        s_run[r] = x;
    }
    __syncthreads();
    const uint32_t i_lo = min(s_lo, nhi);
    // a binned batch files its marks in region bins (k_binsort takes them on)
    uint32_t *const hl_mine = quota ? run0.hl_buf + size_t(blockIdx.x) * nbin * quota : nullptr;
    const uint32_t rmask = (1u << rlog) - 1u;
    // the table: bytes [tb0, tb0 + tbn) of the multiplier line (the same for every run)
    const uint32_t *const mtab = run0.mtab;
    const uint64_t tb0 = run0.m0 / 30, tbn = (run0.m1 - run0.m0 + 1) / 30;
    // the mark of class e >> 16 of q at bit t of a run (t < nblk)
    auto mark = [&](uint32_t place, uint32_t e, uint32_t t) {
        if (quota) {
            const uint32_t v = place + t;
            const uint32_t bin = (e >> 20) + (v >> rlog);
            const uint32_t pos = atomicAdd(&s_hcnt[bin], 1u);
            if (pos < quota) hl_mine[bin * quota + pos] = v & rmask;
            else ovf_push(run0, (e >> 16) & 7u, v);
        } else {
            const BatchParams &bp = d.runs[place];
            atomicAnd(bp.map + size_t((e >> 16) & 7u) * bp.wpc + (t >> 5), ~(1u << (t & 31)));
        }
    };
    // the pair (prime p, run): every path of a lane ends here, so the
    // warp meets again before its next pair
    auto pair = [&](uint32_t p, float rp, uint64_t inv, uint32_t pq, uint32_t pr, const HlRun &run) {
        uint32_t rho;
        const uint64_t b = divmod_recip(run.B, p, inv, rho) - tb0;  // byte b0 in the table
        // m = 30 b0 + j from j = ceil(30 rho / p) on, the estimate lowered by
        // 0.01, far above its error
        if (run.nblk <= (p >> 5)) {
            // at most one multiple: when the estimate gives j - 1, the first
            // multiple is at least 0.99 p / 30 > nblk bits up, and j - 1
            // itself is below the run
            const uint32_t j = __float2uint_ru(fmaxf(__uint2float_rn(rho) * (30.0f * rp) - 0.01f, 0.0f));
            const uint32_t t = pq * j + ((pr * j * 2185u) >> 16) - rho;  // floor(pr j / 30): pr j < 900
            if (((kUnits30 >> j) & 1u) && t < run.nblk) {
                const uint32_t k = __popc(kUnits30 & ((1u << j) - 1u));
                if (b >= tbn) atomicOr(run0.err, kErrTable);
                else if ((__ldg(mtab + (b >> 2)) >> (8 * (uint32_t(b) & 3u) + k)) & 1u)
                    mark(run.place, s_cls[s_res[pr]][k], t);
            }
            return;
        }
        if (run.nblk <= (p >> 2) && !(p >> 31)) {
            // a few: the units among the next 30 nblk / p + 2 j (10 at most),
            // the table read only for one inside the run
            const float f30 = 30.0f * rp;
            const uint32_t j0 = __float2uint_ru(fmaxf(__uint2float_rn(rho) * f30 - 0.01f, 0.0f));
            const uint32_t n = __float2uint_rz(__uint2float_rn(run.nblk) * f30) + 3u;
            for (uint32_t v = uint32_t(kUnits60 >> j0) & ((1u << n) - 1u); v; v &= v - 1u) {
                uint32_t j = j0 + __ffs(v) - 1u;
                const bool next = j >= 30;  // a unit of the byte after b0
                j -= next ? 30u : 0u;
                const uint32_t t = (next ? p : 0u) + pq * j + ((pr * j * 2185u) >> 16) - rho;
                if (t < run.nblk) {
                    const uint64_t at = b + (next ? 1u : 0u);
                    const uint32_t k = __popc(kUnits30 & ((1u << j) - 1u));
                    if (b >= tbn || at >= tbn) atomicOr(run0.err, kErrTable);
                    else if ((__ldg(mtab + (at >> 2)) >> (8 * (uint32_t(at) & 3u) + k)) & 1u)
                        mark(run.place, s_cls[s_res[pr]][k], t);
                }
            }
            return;
        }
        const uint32_t *const cls = s_cls[s_res[pr]];
        if ((p >> 31) || p > ~run.nblk) {
            // p + nblk >= 2^32 (a run of 2^31 bits and the margin, p close to
            // 2^31) or p >= 2^31: at most three bytes, their bits in 64-bit
            // arithmetic
            const uint64_t x = uint64_t(rho) + run.nblk - 1;
            const uint32_t more = (x >= p ? 1u : 0u) + (x >= 2ull * p ? 1u : 0u);
            if (b >= tbn || b + more >= tbn) {
                atomicOr(run0.err, kErrTable);
                return;
            }
            for (uint32_t nb = 0; nb <= more; ++nb) {
                const uint64_t at = b + nb;
                uint32_t v = (__ldg(mtab + (at >> 2)) >> (8 * (uint32_t(at) & 3u))) & 0xFFu;
                for (; v; v &= v - 1u) {
                    const uint32_t e = cls[__ffs(v) - 1u];
                    const int64_t t = int64_t(uint64_t(nb) * p) + int64_t(pq * (e & 0xFFu) + ((e >> 8) & 0xFFu)) - rho;
                    if (t >= 0 && t < int64_t(run.nblk)) mark(run.place, e, uint32_t(t));
                }
            }
            return;
        }
        // bytes b .. b + nb, nb = floor((rho + nblk - 1) / p) (a float
        // estimate within one of it, corrected); bits in (-p, nblk + p):
        // one below zero is at least 2^31 as u32
        const uint32_t x = rho + run.nblk - 1;
        uint32_t nb = __float2uint_rz(__uint2float_rn(x) * rp);
        if (uint64_t(nb) * p > x) --nb;
        else if (x - nb * p >= p) ++nb;
        if (b >= tbn || b + nb >= tbn) {
            atomicOr(run0.err, kErrTable);
            return;
        }
        const uint32_t sh = uint32_t(b) & 3u, eb = sh + nb;  // the end byte from the first word's first
        const uint32_t *tw = mtab + (b >> 2);
        // the end bytes without most of the units outside the run: those below
        // 30 rho / p, and from 30 (x - nb p + 1) / p on (estimates that err by
        // 0.01 at most towards keeping one: a mark's own bit decides)
        const float f30 = 30.0f * rp;
        const uint32_t ja = __float2uint_ru(fmaxf(__uint2float_rn(rho) * f30 - 0.01f, 0.0f));
        const uint32_t jb = __float2uint_rz(__uint2float_rn(x - nb * p + 1) * f30 + 0.01f);
        const uint32_t lo8 = 0xFFu << __popc(kUnits30 & ((1u << ja) - 1u));
        const uint32_t hi8 = (1u << __popc(kUnits30 & ((2u << jb) - 1u))) - 1u;
        const uint32_t hi_mask = (0x00FFFFFFu >> (24 - 8 * (eb & 3u))) | (hi8 << (8 * (eb & 3u)));
        uint32_t left = eb >> 2;                             // words after the current one
        uint32_t tb = 0u - rho - p * sh;                     // bit of the word's byte 0, less its v_k
        uint32_t v = __ldg(tw) & ((0xFFFFFF00u | (lo8 & 0xFFu)) << (8 * sh));
        if (!left) v &= hi_mask;
        // the next table word loaded before this word's marks (its
        // latency hidden behind them); one mark per trip, whichever word
        // a lane is in, so a warp's trips follow its lanes' total marks
        // and not the fullest lane of every word
        uint32_t vn = left ? __ldg(tw + 1) : 0u;
        for (;;) {
            if (v) {
                const uint32_t j = __ffs(v) - 1u;
                v &= v - 1u;
                const uint32_t e = cls[j & 7u];
                const uint32_t t = tb + p * (j >> 3) + pq * (e & 0xFFu) + ((e >> 8) & 0xFFu);
                if (t < run.nblk) mark(run.place, e, t);
            }
            if (!v) {
                if (!left) break;
                --left;
                ++tw;
                tb += 4 * p;
                v = vn;
                if (left) vn = __ldg(tw + 1);
                else v &= hi_mask;
            }
        }
    };
    const uint32_t *primes = run0.primes;
    const uint32_t stride = gridDim.x * blockDim.x;
    // Warp-uniform loops: the warp's first prime bounds them.
    const uint32_t deal = d.h->hl_deal;
    // Of several runs only those that the warp's primes reach: 292 segments of
    // uneven windows at 1e15..5e18 39.3 -> 36.9 ms, 16 windows at 1e10..3e18 1.60
    // -> 0.73. One run apart (kMany), since that loop's bound, which the
    // compiler cannot tell to be the same for a warp's lanes, cost it 9%: one
    // segment 0.70 ms with a loop over all runs, 0.77 with this one, 0.66.
    auto harvest = [&](auto many) {
        constexpr bool kMany = decltype(many)::value;
        const uint32_t warp = threadIdx.x >> 5, off = (threadIdx.x & 31u) * (deal == kDealLanes ? gridDim.x : 1u);
        uint32_t first = i_lo + (deal == kDealBlocks  ? blockIdx.x * blockDim.x + warp * 32
                                 : deal == kDealWarps ? (warp * gridDim.x + blockIdx.x) * 32
                                                      : warp * 32 * gridDim.x + blockIdx.x);
        uint32_t p_next = first + off < nhi ? __ldg(primes + first + off) : 3u;
        uint32_t live = nrun, reach = 0;  // the runs that the warp's primes reach: all of them below reach
        for (; first < nhi; first += stride) {
            const uint32_t i = first + off, p = p_next;
            if (i + stride < nhi) p_next = __ldg(primes + i + stride);  // its latency behind this prime's work
            const float rp = __fdividef(1.0f, __uint2float_rn(p));
            uint64_t inv = recip64(p, rp);
            const uint32_t pq = p / 30, pr = p - 30 * pq;
            if constexpr (!kMany) {
                if (i < s_run[0].n_all) pair(p, rp, inv, pq, pr, s_run[0]);
                __syncwarp();
                continue;
            }
            if (first >= reach) {
                while (live && s_run[live - 1].n_all <= first) --live;
                reach = live ? s_run[live - 1].n_all : kNone;
            }
            // A run narrower than p / 64: a pair goes on only if one of its
            // integers is a multiple of p, which the remainder r of base - 1
            // tells (the next multiple is base + p - 1 - r), so most warps stop
            // there: 16 runs of 1e6 integers at 4e18..5e18 0.225 -> 0.146 ms a run.
            // (A run alone would pay the exact reciprocal for one remainder; p >=
            // 2^31: r takes 33 bits.)
            inv = recip64_exact(p, inv);
            const uint32_t narrow = p >> 31 ? 0u : p >> 6;
            for (uint32_t ri = 0; ri < live; ++ri) {
                const uint64_t below = s_run[ri].below;
                const uint32_t span = s_run[ri].span;
                bool go = i < s_run[ri].n_all;
                if (span < narrow) {
                    uint32_t r = uint32_t(below) - uint32_t(__umul64hi(below, inv)) * p;  // below 2 p
                    r = min(r, r - p);
                    go = go && r >= p - 1 - span;
                }
                if (go) {
                    const HlRun run = s_run[ri];  // in registers: the marks' atomics would have it read again
                    pair(p, rp, inv, pq, pr, run);
                }
                __syncwarp();
            }
        }
    };
    if (nrun > 1) harvest(std::true_type{});
    else harvest(std::false_type{});
    if (quota) {
        __syncthreads();
        for (uint32_t bi = threadIdx.x; bi < nbin; bi += blockDim.x) run0.hl_cnt[blockIdx.x * nbin + bi] = s_hcnt[bi];
    }
}

// exclusive prefix sums of in[0, n) into out (n <= 4 * 256; 256 threads;
// the caller synchronises before reading out or reusing s_wsum)
__device__ __forceinline__ void block_excl_scan4(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *s_wsum)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t v[4], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t idx = 4 * tid + j;
        v[j] = idx < n ? in[idx] : 0u;
        sum += v[j];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(~0u, x, o);
        if (lane >= uint32_t(o)) x += y;
    }
    if (lane == 31) s_wsum[warp] = x;
    __syncthreads();
    uint32_t run = x - sum;
    for (uint32_t i = 0; i < warp; ++i) run += s_wsum[i];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t idx = 4 * tid + j;
        if (idx < n) out[idx] = run;
        run += v[j];
    }
}

constexpr uint32_t kSortPer = 16;                   // offsets per thread and chunk (four uint4)
constexpr uint32_t kSortChunk = 256 * kSortPer;     // offsets a CTA sorts in shared memory at a time

// Binned hit lists, sorted by tile: every (harvest CTA, region bin) list,
// kSortChunk offsets at a time (read once, into registers), is counted per
// tile of its region, given room in each tile's bin by one atomic add per
// tile, sorted by tile in shared memory and stored tile run by tile run
// (consecutive threads, consecutive addresses). Offsets beyond a tile bin's
// capacity go to the overflow list. The lists start 16-byte aligned (the
// quota is a multiple of 32 words).
// Six CTAs per SM (40 registers): the hit-list stage takes 6.77 ms per
// 128-segment batch (four 6.85, five 6.73, eight 7.02; one wave of persistent CTAs).
__global__ void __launch_bounds__(256, 6) k_binsort(BatchDesc d)
{
    __shared__ uint32_t s_out[kSortChunk];
    __shared__ uint32_t s_cnt[kSortMaxTiles], s_start[kSortMaxTiles], s_gbase[kSortMaxTiles];
    __shared__ uint32_t s_wsum[8];
    __shared__ uint32_t s_j;
    if (!hl_binned(d.runs[0])) return;
    const BatchParams &bp = d.runs[0];
    const uint32_t tid = threadIdx.x, bs = blockDim.x;
    const uint32_t quota = bp.hl_quota, nreg = bp.hl_nreg, nbin = 8 * nreg, ctas = bp.hl_ctas;
    const uint32_t rlog = bp.hl_rlog, tb = bp.tile_bits, rcp = bp.tile_rcp;
    const uint32_t items = nbin * ctas, cap = bp.tb_cap;
    for (;;) {
        const uint32_t j = next_item(d.work + kWorkBinsort, &s_j);
        if (j >= items) break;
        const uint32_t bin = j / ctas, c = j - bin * ctas;
        const uint32_t k = bin / nreg, reg = bin - k * nreg;
        const uint32_t n = min(bp.hl_cnt[size_t(c) * nbin + bin], quota);
        const uint32_t *e = bp.hl_buf + (size_t(c) * nbin + bin) * quota;
        // the region's bits [rb, rb + 2^rlog) meet tiles ti0 .. ti0 + tpr - 1
        // of the class array (tiles may straddle regions: their bins are
        // filled by every region that meets them)
        const uint32_t rb = reg << rlog;
        const uint32_t ti0 = tile_of(rb, tb, rcp);
        const uint32_t tpr = tile_of(min(rb + ((1u << rlog) - 1u), bp.tb_tiles * tb - 1), tb, rcp) - ti0 + 1;
        const uint32_t tile0 = k * bp.tb_tiles + ti0;
        for (uint32_t cs = 0; cs < n; cs += kSortChunk) {
            const uint32_t m = min(n - cs, kSortChunk);
            for (uint32_t t = tid; t < tpr; t += bs) s_cnt[t] = 0;
            // this thread's offsets: groups of four at tid + 256 u (kNone past the end)
            uint32_t v[kSortPer];
            const uint4 *e4 = reinterpret_cast<const uint4 *>(e + cs);
#pragma unroll
            for (uint32_t u = 0; u < kSortPer / 4; ++u) {
                const uint32_t g = tid + bs * u;
                const uint4 q = 4 * g < m ? __ldcs(e4 + g) : make_uint4(kNone, kNone, kNone, kNone);
                v[4 * u] = q.x;
                v[4 * u + 1] = 4 * g + 1 < m ? q.y : kNone;
                v[4 * u + 2] = 4 * g + 2 < m ? q.z : kNone;
                v[4 * u + 3] = 4 * g + 3 < m ? q.w : kNone;
            }
            __syncthreads();
            // each offset as (tile of the region, bit in the tile): t - ti0 in
            // the top 11 bits, the bit (< tb <= 2^21) in the low 21
#pragma unroll
            for (uint32_t u = 0; u < kSortPer; ++u)
                if (v[u] != kNone) {
                    const uint32_t t = rb + v[u], ti = tile_of(t, tb, rcp);
                    v[u] = ((ti - ti0) << 21) | (t - ti * tb);
                    atomicAdd(&s_cnt[v[u] >> 21], 1u);
                }
            __syncthreads();
            block_excl_scan4(s_cnt, s_start, tpr, s_wsum);
            __syncthreads();
            for (uint32_t t = tid; t < tpr; t += bs) {
                const uint32_t cn = s_cnt[t];
                s_gbase[t] = cn ? atomicAdd(bp.tb_cnt + tile0 + t, cn) : 0u;
                s_cnt[t] = s_start[t];
            }
            __syncthreads();
#pragma unroll
            for (uint32_t u = 0; u < kSortPer; ++u)
                if (v[u] != kNone) s_out[atomicAdd(&s_cnt[v[u] >> 21], 1u)] = v[u];
            __syncthreads();
            for (uint32_t i = tid; i < m; i += bs) {
                const uint32_t off = s_out[i], t = off >> 21, bit = off & ((1u << 21) - 1u);
                const uint32_t pos = s_gbase[t] + (i - s_start[t]);
                if (pos < cap) bp.tb_buf[size_t(tile0 + t) * cap + pos] = bit;
                else ovf_push(bp, k, (ti0 + t) * tb + bit);
            }
            __syncthreads();
        }
    }
}

// The overflow list of a binned batch, cleared after the tiles.
__device__ __forceinline__ void overflow_marks(const BatchDesc &d, uint32_t nrun)
{
    const BatchParams &bp0 = d.runs[0];
    const uint32_t cnt = *bp0.ovf_cnt, tb = bp0.tile_bits;
    if (cnt > bp0.ovf_cap && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(bp0.err, kErrHlOverflow);
    const uint32_t n = min(cnt, bp0.ovf_cap);
    const uint32_t b0 = d.h->win_b0, b1 = d.h->win_b1;  // the plain form's window of run 0 (else everything)
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 e = bp0.ovf_buf[i];
        // the run of virtual bit e.y: the last one whose first virtual tile is at or below it
        const uint32_t vt = e.y / tb;
        uint32_t lo = 0, hi = nrun - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) / 2;
            if (d.runs[mid].tb_vt0 <= vt) lo = mid;
            else hi = mid - 1;
        }
        const BatchParams &bp = d.runs[lo];
        const uint32_t t = e.y - bp.tb_vt0 * tb;
        if (t < bp.nblk && t >= b0 && t < b1)
            atomicAnd(bp.map + size_t(e.x) * bp.wpc + (t >> 5), ~(1u << (t & 31)));
    }
}

// The primality test of one odd n, 2^33 < n < 2^64, without a prime factor
// below 128 (Baillie and Wagstaff, Mathematics of Computation 35, 1980): a
// strong probable prime to base 2, then an extra strong Lucas probable prime
// (Grantham, Mathematics of Computation 70, 2001; the first P from 3 on whose
// P^2 - 4 has Jacobi symbol -1, Q = 1). No composite below 2^64 is both: every
// base-2 pseudoprime of J. Feitsma's complete list fails the second. A square
// ends at base 2 (of a prime: only 1093^2 and 3511^2 pass, both below 2^33),
// so a P exists. Numbers are in Montgomery form, x 2^64 mod n.
struct Bpsw {
    uint64_t n, ninv, one;
    __device__ __forceinline__ explicit Bpsw(uint64_t q) : n(q)
    {
        ninv = n;  // n^-1 mod 2^64 (Newton: correct bits 3, 6, 12, ...)
#pragma unroll
        for (int i = 0; i < 5; ++i) ninv *= 2 - n * ninv;
        one = (0 - n) % n;  // 2^64 mod n
    }
    __device__ __forceinline__ uint64_t sub(uint64_t x, uint64_t y) const { return x >= y ? x - y : x - y + n; }
    __device__ __forceinline__ uint64_t twice(uint64_t x) const { return sub(x, n - x); }
    // x y / 2^64: the product less the multiple of n with the same low half
    __device__ __forceinline__ uint64_t mul(uint64_t x, uint64_t y) const
    {
        return sub(__umul64hi(x, y), __umul64hi(x * y * ninv, n));
    }

    // 2^d = 1, or 2^(d 2^r) = -1 for an r < s (n - 1 = d 2^s, d odd)
    __device__ __forceinline__ bool base2() const
    {
        const int s = __ffsll(static_cast<long long>(n - 1)) - 1;
        const uint64_t d = (n - 1) >> s, minus = n - one;
        uint64_t x = twice(one);
#pragma unroll 1
        for (int b = 62 - __clzll(static_cast<long long>(d)); b >= 0; --b) {
            x = mul(x, x);
            if (d >> b & 1) x = twice(x);
        }
        bool ok = x == one || x == minus;
        for (int r = 1; r < s && !ok; ++r) {
            x = mul(x, x);
            ok = x == minus;
        }
        return ok;
    }

    // the Jacobi symbol (a | n), 0 < a < 2^31
    __device__ __noinline__ static int jacobi(uint32_t a, uint64_t n)
    {
        bool neg = false;
        const int z = __ffs(a) - 1;
        if (z & 1) neg ^= (n & 7) == 3 || (n & 7) == 5;
        a >>= z;
        neg ^= (a & n & 3) == 3;
        uint32_t m = a;  // (n mod m | m)
        a = uint32_t(n % m);
        while (a) {
            const int y = __ffs(a) - 1;
            if (y & 1) neg ^= (m & 7) == 3 || (m & 7) == 5;
            a >>= y;
            neg ^= (a & m & 3) == 3;
            const uint32_t t = m % a;
            m = a;
            a = t;
        }
        return m > 1 ? 0 : neg ? -1 : 1;
    }

    // The first P, or 0 where P^2 - 4 has a factor of n before it (n > 2^33 is
    // then composite; not below P = 127, without a factor below 128): the
    // symbols of the primes up to 23 as a sign per k <= 24 give those of (P - 2)
    // (P + 2) up to P = 22; one n in a thousand or so needs more.
    template <uint32_t F>
    __device__ __forceinline__ static uint32_t signs(uint32_t r, uint64_t n)
    {
        constexpr uint32_t non = [] {
            uint32_t m = 0;
            for (uint32_t x = 1; x < F; ++x) m |= 1u << x;
            for (uint32_t x = 1; x < F; ++x) m &= ~(1u << (x * x % F));
            return m;
        }();
        constexpr uint32_t odd = [] {  // bit k: F divides k an odd number of times
            uint32_t m = 0;
            for (uint32_t k = F; k <= 24; ++k) {
                uint32_t v = 0, x = k;
                for (; x % F == 0; x /= F) ++v;
                m |= (v & 1u) << k;
            }
            return m;
        }();
        bool neg = non >> (r % F) & 1u;
        if ((F & 3) == 3) neg ^= (n & 3) == 3;
        return neg ? odd : 0u;
    }
    __device__ __forceinline__ uint32_t lucas_p() const
    {
        const uint32_t r = uint32_t(n % (3u * 5 * 7 * 11 * 13 * 17 * 19 * 23));
        uint32_t k = signs<3>(r, n) ^ signs<5>(r, n) ^ signs<7>(r, n) ^ signs<11>(r, n) ^ signs<13>(r, n) ^
                     signs<17>(r, n) ^ signs<19>(r, n) ^ signs<23>(r, n);
        if ((n & 7) == 3 || (n & 7) == 5) k ^= 1u << 2 | 1u << 6 | 1u << 8 | 1u << 10 | 1u << 14 | 1u << 18 | 1u << 22 | 1u << 24;
        const uint32_t p = (k ^ k >> 4) & 0x1FFFFEu;  // bit P - 2
        if (p) return uint32_t(__ffs(p)) + 1u;
        for (uint32_t x = 23; x < 30000; ++x) {
            const int j = jacobi(x * x - 4, n);
            if (j <= 0) return j ? x : 0u;
        }
        return 0;  // (a square)
    }

    // V_d = 2 and U_d = 0 (then V_(d+1) = P), the same with both signs turned,
    // or V_(d 2^r) = 0 for an r < s - 1 (n + 1 = d 2^s, d odd). V_d = 0 is taken
    // for s = 1 too, where no n has it: with x + 1 / x = P it says x^(n+1) = -1
    // modulo every prime q of n, so x has an order divisible by 4 there; the
    // order divides q - (P^2 - 4 | q), so the symbol is q mod 4 for every q, and
    // -1 for n makes n = 3 mod 4, which is s > 1.
    __device__ __forceinline__ bool lucas() const
    {
        const uint32_t p = lucas_p();
        uint64_t pm = 0;
#pragma unroll 1
        for (int b = 31 - __clz(p); b >= 0; --b) {
            pm = twice(pm);
            if (p >> b & 1) pm = sub(pm, n - one);
        }
        const int s = __ffsll(static_cast<long long>(n + 1)) - 1;
        const uint64_t d = (n + 1) >> s, two = twice(one);
        uint64_t v = pm, w = sub(mul(pm, pm), two);  // V_1, V_2
#pragma unroll 1
        for (int b = 62 - __clzll(static_cast<long long>(d)); b >= 0; --b) {
            const bool up = d >> b & 1;
            const uint64_t x = sub(mul(v, w), pm), y = up ? w : v, y2 = sub(mul(y, y), two);
            v = up ? x : y2;
            w = up ? y2 : x;
        }
        bool ok = v == 0 || (v == two && w == pm) || (v == n - two && w == n - pm);
        for (int r = 1; r < s - 1 && !ok; ++r) {
            v = sub(mul(v, v), two);
            ok = v == 0;
        }
        return ok && p;  // (a return at the start cost the test 6%)
    }
};

// Narrow runs (BatchParams::test): what the tiles leave has no factor up to
// p_mid, one integer in 25 or so, and each is settled by its own primality
// test instead of every larger sieving prime being divided into the run. A
// warp takes test_words words of a class array: their bits to a list, base 2
// for all, the Lucas test for those that pass (three in five, nearly all of
// them prime), 32 numbers at a time. Bound by the integer multipliers (11 of a
// product's 22 instructions, wide ones at a quarter of the issue rate): 13 ps
// an integer of the run at 4e18, where Miller-Rabin to seven bases takes 51.
// From kTestMinWords on a warp's first list has about 32 numbers: 16 runs of
// 1e4 integers at 4e18 take .23 ms with 6 words at least, .25 with 1 (2.59
// through the hit lists).
constexpr uint32_t kTestWords = 32, kTestMinWords = 6;
constexpr int kTestThreads = 128, kTestCtas = 8;

__device__ __forceinline__ void test_runs(const BatchDesc &d, uint32_t nrun)
{
    __shared__ uint16_t s_list[kTestThreads / 32][32 * kTestWords];
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5), tw = d.h->test_words;
    uint16_t *const list = s_list[threadIdx.x >> 5];
    uint32_t task = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    for (uint32_t r = 0; r < nrun; ++r) {
        const BatchParams &bp = d.runs[r];
        if (!bp.test) continue;
        const uint32_t nw = (bp.nblk + 31) / 32, per = (nw + tw - 1) / tw, tasks = 8 * per;
        for (; task < tasks; task += warps) {
            const uint32_t k = task / per, w0 = (task - k * per) * tw;
            uint32_t *const words = bp.map + size_t(k) * bp.wpc + w0;
            uint32_t v = lane < tw && w0 + lane < nw ? words[lane] : 0u;
            if (w0 + lane + 1 == nw && (bp.nblk & 31u)) v &= (1u << (bp.nblk & 31u)) - 1u;
            uint32_t at = __popc(v);
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(~0u, at, o);
                if (lane >= o) at += y;
            }
            uint32_t n = __shfl_sync(~0u, at, 31);
            at -= __popc(v);
            for (; v; v &= v - 1u) list[at++] = uint16_t(32 * lane + __ffs(v) - 1u);
            __syncwarp();
            const uint64_t q0 = bp.base + 30ull * 32 * w0 + unit30(k);
            for (uint32_t pass = 0; pass < 2; ++pass) {
                uint32_t kept = 0;
                for (uint32_t i = lane; i - lane < n; i += 32) {
                    const uint32_t bit = list[i < n ? i : 0u];
                    bool prime = false;
                    if (i < n) {
                        const Bpsw t(q0 + 30ull * bit);
                        prime = pass ? t.lucas() : t.base2();
                        if (!prime) atomicAnd(words + (bit >> 5), ~(1u << (bit & 31u)));
                    }
                    const uint32_t bal = __ballot_sync(~0u, prime);
                    if (prime) list[kept + __popc(bal & ((1u << lane) - 1u))] = uint16_t(bit);
                    kept += __popc(bal);
                    __syncwarp();
                }
                n = kept;
            }
        }
        task -= tasks;  // the next run's tasks go on from here
    }
}

// After the tiles: the overflow marks of a binned batch, and the narrow runs' tests.
__global__ void __launch_bounds__(kTestThreads) k_map_finish(BatchDesc d)
{
    const uint32_t nrun = d.h->nrun;
    if (!nrun) return;
    if (hl_binned(d.runs[0])) overflow_marks(d, nrun);
    if (d.h->test_words) test_runs(d, nrun);
}

// The class arrays of a sieved range, rewritten as one byte per block of 30
// (bit k = class k): one thread per class-array word, 32 bytes out.
__global__ void __launch_bounds__(256) k_wheel_bytes(BatchParams bp, uint32_t *out)
{
    const uint32_t nw = (bp.nblk + 31) / 32;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
        uint32_t a[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) a[k] = bp.map[size_t(k) * bp.wpc + w];
        const uint32_t valid = (w + 1) * 32 <= bp.nblk ? 32u : bp.nblk - w * 32;
#pragma unroll
        for (uint32_t o = 0; o < 8; ++o) {
            uint32_t word = 0;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t b = 4 * o + j;
                uint32_t byte = 0;
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) byte |= ((a[k] >> b) & 1u) << k;
                if (b >= valid) byte = 0;
                word |= byte << (8 * j);
            }
            out[size_t(w) * 8 + o] = word;
        }
    }
}

// Map self-check: every word of every run's class arrays in two batch
// descriptors of the same geometry (the maps built with and without hit
// lists); differing words are counted and flag the batch.
__global__ void __launch_bounds__(256) k_map_compare(BatchDesc a, BatchDesc b, uint32_t *count)
{
    const uint32_t nrun = a.h->nrun;
    for (uint32_t r = 0; r < nrun; ++r) {
        const BatchParams &ra = a.runs[r];
        const uint32_t *mb = b.runs[r].map;
        const size_t words = size_t(8) * ra.wpc;
        uint32_t bad = 0;
        for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < words; i += size_t(gridDim.x) * blockDim.x)
            bad += ra.map[i] != mb[i];
        bad = __reduce_add_sync(~0u, bad);
        if ((threadIdx.x & 31) == 0 && bad) {
            atomicAdd(count, bad);
            atomicOr(ra.err, kErrSelfCheck);
        }
    }
}

}  // namespace gbk

namespace gbh {

void launch_map_compare(const gbk::BatchDesc &a, const gbk::BatchDesc &b, uint32_t *count, const Grids &g,
                        cudaStream_t st)
{
    gbk::k_map_compare<<<g.sm * 8, 256, 0, st>>>(a, b, count);
}

static size_t tile_smem(uint32_t tile_bits, const gbk::GroupInfo &gi)
{
    return size_t((tile_bits >> 5) + gi.words) * 4;
}

// the persistent tile kernel adds the tile-bin staging buffer (stage offsets)
static size_t tile_smem_staged(uint32_t tile_bits, uint32_t stage, const gbk::GroupInfo &gi)
{
    return tile_smem(tile_bits, gi) + size_t(stage) * 4;
}

bool tile_attributes(uint32_t tile_bits, const gbk::GroupInfo &gi, int device, uint32_t *stage)
{
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, gbk::k_tile<gbk::kTbStages[0]>);
    const size_t room = size_t(optin) > fa.sharedSizeBytes ? size_t(optin) - fa.sharedSizeBytes : 0;
    const size_t base = tile_smem(tile_bits, gi);
    if (base > room) return false;
    // the largest staging buffer of the kernel's instantiations that fits
    uint32_t c = 0;
    while (c < 2 && base + size_t(gbk::kTbStages[c]) * 4 > room) ++c;
    *stage = gbk::kTbStages[c];
    const int bytes = int(tile_smem_staged(tile_bits, *stage, gi));
    if (c == 0) cudaFuncSetAttribute(gbk::k_tile<gbk::kTbStages[0]>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (c == 1) cudaFuncSetAttribute(gbk::k_tile<gbk::kTbStages[1]>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (c == 2) cudaFuncSetAttribute(gbk::k_tile<gbk::kTbStages[2]>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return true;
}

void launch_xfirst(const gbk::BatchDesc &d, const Grids &g, cudaStream_t st)
{
    gbk::k_xfirst<<<g.sm * 8, 256, 0, st>>>(d);
}

void launch_tile(const gbk::BatchDesc &d, const gbk::GroupInfo &gi, uint32_t tile_bits, uint32_t stage,
                 const Grids &g, cudaStream_t st)
{
    const size_t bytes = tile_smem_staged(tile_bits, stage, gi);
    if (stage == gbk::kTbStages[0]) gbk::k_tile<gbk::kTbStages[0]><<<g.sm, 1024, bytes, st>>>(d, gi, tile_bits);
    else if (stage == gbk::kTbStages[1]) gbk::k_tile<gbk::kTbStages[1]><<<g.sm, 1024, bytes, st>>>(d, gi, tile_bits);
    else gbk::k_tile<gbk::kTbStages[2]><<<g.sm, 1024, bytes, st>>>(d, gi, tile_bits);
}

void launch_large(const gbk::BatchDesc &d, const Grids &g, cudaStream_t st)
{
    gbk::k_large<<<g.sm * 8, 256, 0, st>>>(d);
}

void launch_hitlist(const gbk::BatchDesc &d, bool direct, const Grids &g, cudaStream_t st)
{
    gbk::k_hitlist<<<g.sm * g.hitlist, gbk::kHlThreads, 0, st>>>(d, direct ? 1u : 0u);
}

// the harvest's grid is one wave of resident CTAs: its primes are dealt out
// by CTA, so a second partial wave would run at a fraction of the occupancy
void query_sieve_grids(Grids &g)
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gbk::k_hitlist, gbk::kHlThreads, 0);
    g.hitlist = n > 0 ? n : 1;
}

void hl_shares(const uint32_t *primes, uint32_t n_lo, uint32_t n, uint32_t ctas, HlShares *out)
{
    for (uint32_t d = 0; d < 2; ++d) {
        const uint32_t block = d == gbk::kDealBlocks ? gbk::kHlThreads : 32;
        out->sum[d][0] = 0;
        for (uint32_t k = 0; k < kHlRounds; ++k) {
            const uint64_t i = n_lo + uint64_t(k) * block * ctas;
            out->sum[d][k + 1] = out->sum[d][k] + (i < n ? double(block) / primes[i] : 0.0);
        }
    }
}

// A CTA takes consecutive primes, whose table bytes are neighbours: dealt out
// warp by warp across the CTAs 128 segments took 7.55 ms, not 6.93. But every
// CTA has one quota a bin, the mean and 45% (hl_quota), and the first CTA's
// primes, the smallest of every round, have the most marks: 1.2 of the mean at
// 4e18 with the tile primes to 1.7e6, 1.42 at 1e15, 3.0 there with those to
// 2^18, above what the overflow list holds of a wide batch. So the primes are
// dealt out by warps where blocks would give the first CTA more than 1.40 (1 / p
// for a prime's marks: 3% above the marks themselves) or there are fewer than 8
// rounds, whose last is a part of one; and one by one where warps would (a few
// thousand primes, or primes from 2e4 on: 2.64 of the mean from 1e4 on at 1e12,
// 1.03 one by one).
uint32_t hl_deal(const HlShares *sh, const uint32_t *primes, uint32_t n_lo, uint32_t n_hi, uint32_t ctas, bool binned)
{
    constexpr double kMost = 1.40;
    const uint32_t n = n_hi - n_lo;
    const double lo = std::log(double(primes[n_lo])), hi = std::log(double(primes[n_hi - 1]));
    const double mean = std::max(std::log(hi / lo), double(n) / primes[n_hi - 1]) / ctas;
    auto first = [&](uint32_t d, uint32_t block) {  // the first CTA's share; past the summed rounds at most
        const uint32_t round = block * ctas, rounds = uint32_t((uint64_t(n) + round - 1) / round);
        if (rounds <= kHlRounds) return sh->sum[d][rounds];
        const double p = primes[n_lo + kHlRounds * round];
        return sh->sum[d][kHlRounds] + std::log(hi / std::log(p)) / ctas + block / p;
    };
    const bool few = n < 8ull * gbk::kHlThreads * ctas;
    if (!binned) return few ? gbk::kDealWarps : gbk::kDealBlocks;
    if (!few && first(gbk::kDealBlocks, gbk::kHlThreads) <= kMost * mean) return gbk::kDealBlocks;
    return first(gbk::kDealWarps, 32) <= kMost * mean ? gbk::kDealWarps : gbk::kDealLanes;
}

void launch_binsort(const gbk::BatchDesc &d, const Grids &g, cudaStream_t st)
{
    gbk::k_binsort<<<g.sm * 6, 256, 0, st>>>(d);
}

uint32_t test_words(uint64_t words, int sm)
{
    const uint64_t warps = uint64_t(sm) * gbk::kTestCtas * (gbk::kTestThreads / 32);
    const uint64_t share = std::max<uint64_t>((words + warps - 1) / warps, gbk::kTestMinWords);
    return words ? uint32_t(std::min<uint64_t>(share, gbk::kTestWords)) : 0u;
}

void launch_map_finish(const gbk::BatchDesc &d, const Grids &g, cudaStream_t st)
{
    gbk::k_map_finish<<<g.sm * gbk::kTestCtas, gbk::kTestThreads, 0, st>>>(d);
}

void launch_xfirst1(const gbk::BatchParams &bp, cudaStream_t st)
{
    if (bp.n_mid <= bp.i0) return;
    const uint32_t n = bp.n_mid - bp.i0;
    uint32_t blocks = (n + 255) / 256;
    if (blocks > 8192) blocks = 8192;
    gbk::k_xfirst1<<<blocks, 256, 0, st>>>(bp);
}

cudaError_t launch_tile1(const gbk::BatchParams &bp, uint32_t max_bits, const gbk::GroupInfo &gi, cudaStream_t st)
{
    // the attribute of the largest tile, whatever this call's: the same for every caller
    const cudaError_t e = cudaFuncSetAttribute(gbk::k_tile1, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(tile_smem(max_bits, gi)));
    if (e != cudaSuccess) return e;
    dim3 grid((bp.wpc * 32 + bp.tile_bits - 1) / bp.tile_bits, 8);
    gbk::k_tile1<<<grid, 1024, tile_smem(bp.tile_bits, gi), st>>>(bp, gi);
    return cudaSuccess;
}

void launch_wheel_bytes(const gbk::BatchParams &bp, uint32_t *out, cudaStream_t st)
{
    const uint32_t nw = (bp.nblk + 31) / 32;
    uint32_t blocks = (nw + 255) / 256;
    if (blocks > 65535) blocks = 65535;
    gbk::k_wheel_bytes<<<blocks, 256, 0, st>>>(bp, out);
}

}  // namespace gbh
