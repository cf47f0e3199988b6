// fz_encode.cuh -- the staged Lorenzo codes of an encode item (8 shuffle blocks, 16384
// consecutive elements) in 16-bit arithmetic.
//
// The dual-quantised value p = round(x * ebx2_r) of an element is an integer, and the Lorenzo
// delta is a sum of p over the element's corner neighbours.  While every partial sum stays
// below 2^24 the reference's float expression (lorenzo_var.cuh:79-295) is exact, so it equals
// the integer one in any order; while every difference below also fits 16 bits, two elements
// share one 32-bit word.  The path is taken where that is known before the item (a relative
// bound: from the field's range) or found while staging it (an absolute bound: from the item's range
// of x * ebx2_r); other items keep the float path (compute_block).
//
// 1. Staging, all threads of the CTA: 16-byte loads, p of each value, and of one difference --
//    along z in 3D, along y in 2D when rows are too long to stage the row above -- into shared
//    memory as 16-bit values D = p - p', biased by 0x8000.  The item's own elements and a halo
//    of one row before them are staged, so each value is quantised once (twice for the
//    difference) instead of once per neighbour it is.
// 2. Codes, lane g of a warp: the 64 consecutive elements of group g of the warp's block, the
//    words the bit transpose wants in that lane's registers.  T = D - D(row above), then
//    d = T - T(left), zero outside the tile, two elements per instruction.  The signs become
//    sign-magnitude after the transpose, a bit plane at a time.
//
// Blocks whose deltas fit 8 bits transpose bytes (byte_planes) instead of 16-bit words.
//
// What bounds it: the float path is bound by instruction issue (3D: 3690 warp instructions per
// 2048-element block, each value quantised for every stencil role it has); this one issues 1500 (2D
// 1390), in 38-46% of the cycles: a CTA waits for its item's loads and at the barrier before the
// images, and the 3-4 CTAs of an SM do not cover each other fully.  Encode launches on GB300, relative bound
// 1e-3, CUDA events around each launch, float path -> this one: 500x500x100 57.9 -> 33.0 us,
// 501x500x100 81.7 -> 38.3, 39200x388 26.9 -> 20.8, 8192x8192 97.1 -> 74.5, 3600x1800 16.4 ->
// 14.4, 3601x1801 19.6 -> 14.4, 2^25 46.9 -> 34.5 (the last at the DRAM's rate: field and slots
// exceed the L2).  Of that the byte planes gave 39200x388 23.6 -> 20.8, 500x500x100 37.2 -> 33.0.
// Items of 4 blocks, 5 CTAs an SM and deeper batches of loads measured the same or slower.
#pragma once

#include "fz_internal.h"

namespace fz {

constexpr uint32_t kItemCodes = 16384;  // elements of an encode item
// Staged element i (of a segment that starts at a multiple of 64 elements) is at byte
// 2 i + 8 (i / 64): the 8-byte pad per 64 elements spreads the lanes' reads, 64 elements apart,
// over all banks.
constexpr uint32_t kStageSlot = 136;  // bytes of 64 staged elements
// Longest row staged as a halo (about a quarter of an item is staged twice then, and 4 CTAs an SM
// still fit).  3D rows beyond it take the float path, 2D rows the difference along y while
// staging.
constexpr uint32_t kHaloRow = 4096;
constexpr uint32_t kBias2   = 0x80008000u;
constexpr uint32_t kBias2s  = 0x80808080u;  // of the deltas: a half's high byte is 0x80 where -128 <= d < 128
// Bound on the 16-bit path's magnitudes (a little below 2^15: the bounds are computed in
// float).
constexpr float kPackedMax = 32600.0f;

__host__ __device__ constexpr uint32_t stage_halo(uint32_t row) { return (row + 64u) & ~63u; }  // >= row + 1
__host__ __device__ constexpr uint32_t stage_bytes(uint32_t halo) { return (halo + kItemCodes) / 64 * kStageSlot; }

// p of two values as the low bits of two words: bits(round(fl(x r)) + magic), for
// |x r| < 2^22 and magic = 1.5 * 2^23 + an integer, two values per instruction
// (mul/add.f32x2).  Round half away from zero:
//   kPos (no value is negative): floor(v + 1/2), both additions rounded down -- the first may
//     drop bits but cannot cross an integer.
//   otherwise: a tie k + 1/2 below 2^22 has a zero last bit, so setting the last bit moves ties
//     (and only ties: a value one step short of a tie has that bit set already) past the
//     middle, and round-to-nearest does the rest.
__device__ __forceinline__ uint64_t pair2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t scale2(uint64_t x, uint64_t r)
{
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(x), "l"(r));
    return v;
}
template <bool kPos>
__device__ __forceinline__ void quant2(uint64_t v, uint64_t magic, uint32_t& p0, uint32_t& p1)
{
    uint64_t s;
    if (kPos) {
        asm("add.rm.f32x2 %0, %1, %2;" : "=l"(s) : "l"(v), "l"(0x3F0000003F000000ull));
        asm("add.rm.f32x2 %0, %0, %1;" : "+l"(s) : "l"(magic));
    } else {
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(s) : "l"(v | 0x0000000100000001ull), "l"(magic));
    }
    p0 = (uint32_t)s, p1 = (uint32_t)(s >> 32);
}
__device__ __forceinline__ float lo_of(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// Whether values of x r of this largest magnitude and within this range stay in 16 bits: a delta at
// a tile corner is a value itself, along an edge a difference of two, inside a difference of two
// (2D) or four (3D) such; the partial sums are smaller.  NaN: no.
template <int ND>
__device__ __forceinline__ bool packed_fits(float peak, float span)
{
    return fmax_nan(peak + 1.0f, (ND == 1 ? 1.0f : ND == 2 ? 2.0f : 4.0f) * (span + 2.0f)) < kPackedMax;
}
// The whole field, from its range.
template <int ND>
__device__ __forceinline__ bool packed_range(const EbInfo& e)
{
    return packed_fits<ND>(fmaxf(fabsf(e.vmin), fabsf(e.vmax)) * e.ebx2_r, (e.vmax - e.vmin) * e.ebx2_r);
}

// What is known of the values before an item is staged: that they fit, that none is negative too, or
// nothing.
enum class Range { Fits, Positive, Unknown };

// Least and largest of a thread's values of x r, both NaN where one is.  Range and peak instead of
// the peak alone (one instruction a pair of values more): a field far from zero under an absolute
// bound, 2 to 2.65 at 1e-4 (|x r| up to 13250), was staged, thrown away and encoded in the float
// path.  fz_compress on GB300, a pass among others: 39200x388 48.9 -> 35.3 us (float path without
// staging 38), 8192x8192 166 -> 111 (139), 500x500x100 87 -> 50 (72), 501x500x100 113 -> 54 (101); the same fields
// from zero up at 1e-3 31.0 -> 31.5, 102 -> 99, 46.1 -> 47.0, 49.4 -> 49.7.  An item that does not fit (its range past
// 16298 quanta in 2D, 8148 in 3D, or codes that overflow) is still staged first, which costs it 10 to 20%:
// skipping the CTA's next items after such a one, or sampling them, took 1 to 2% from the fields that fit.
struct Limits {
    float mn = INFINITY, mx = -INFINITY;
    __device__ __forceinline__ void add(uint64_t v)
    {
        mn = fmin3_nan(mn, lo_of(v), hi_of(v)), mx = fmax3_nan(mx, lo_of(v), hi_of(v));
    }
    // Whether the values of all threads of the CTA fit together (one CTA barrier); red: shared, two
    // words a warp.  f2ord's order holds for numbers only: a NaN goes as an infinity, which does
    // not fit either.
    template <int ND>
    __device__ __forceinline__ bool all_fit(uint32_t (*red)[8]) const
    {
        const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
        const uint32_t lo = __reduce_min_sync(kFull, f2ord(mn)), hi = __reduce_max_sync(kFull, f2ord(mx == mx ? mx : INFINITY));
        if (lane == 0) red[0][wid] = lo, red[1][wid] = hi;
        __syncthreads();
        const float l = ord2f(__reduce_min_sync(kFull, red[0][lane & 7u])), h = ord2f(__reduce_max_sync(kFull, red[1][lane & 7u]));
        return packed_fits<ND>(fmaxf(fabsf(l), fabsf(h)), h - l);
    }
};

constexpr uint32_t kStageStep = 256 * 4;  // elements a CTA stages with one group of 4 per thread

// How an item of the field is staged: `halo` elements before it, and with `shift` the
// difference to the element `shift` before, absent where (e / shift) % tile == 0.
struct StagePlan {
    uint32_t halo, shift, tmask;
    FastDiv  dshift;
};
template <int ND>
__device__ __forceinline__ bool stage_plan(uint32_t x, uint32_t xy, const FastDiv& dx, const FastDiv& dxy, StagePlan& p)
{
    if (ND == 1) {
        p.halo = 0, p.shift = 0, p.tmask = 0, p.dshift = dx;
        return true;
    }
    if (x < 8) return false;  // packed_deltas
    if (ND == 2) {
        const bool wide = x > kHaloRow;
        p.halo  = wide ? 64u : stage_halo(x);  // wide: only the last element's difference
        p.shift = wide ? x : 0u, p.tmask = 15u;
        p.dshift = dx;
        return true;
    }
    p.halo = stage_halo(x), p.shift = xy, p.tmask = 7u;
    p.dshift = dxy;
    return x <= kHaloRow;
}

// Which groups of an item have a neighbour `shift` before them: none (or no difference is
// staged), all, or some -- then also for groups of 4 that straddle two rows (planes).
enum class Diff { None, All, Some };

// Row (plane) of a group and its element in it, kStageStep elements at a time.
struct StageRow {
    uint32_t row, rem, drow, drem;
    __device__ __forceinline__ StageRow(uint32_t e, const StagePlan& p)
    {
        row  = fdiv(e, p.dshift), rem = e - row * p.shift;
        drow = fdiv(kStageStep, p.dshift), drem = kStageStep - drow * p.shift;
    }
    __device__ __forceinline__ void next(uint32_t shift)
    {
        row += drow, rem += drem;
        if (rem >= shift) rem -= shift, ++row;
    }
};

// kCnt groups of 4 elements, kStageStep elements apart, from element e on, to dst on.  kFull:
// all of them lie inside the field; otherwise groups past its last whole one read that one
// instead.  kAl: shift % 4 == 0, the neighbours' loads are aligned.  `mine`: whether the last
// group is stored.
template <bool k3D, uint32_t kCnt, Diff kDiff, bool kAl, Range kRange, bool kFull>
__device__ __forceinline__ void stage_groups(const float* __restrict__ in, uint32_t elast, uint32_t e,
                                             const StagePlan& p, StageRow& pos, float r, Limits& lim,
                                             uint8_t* dst, bool mine)
{
    const uint64_t rr    = pair2(r, r);
    const uint64_t magic = pair2(12582912.0f + 32768.0f, 12582912.0f + 32768.0f);  // bits: ...8000 + p
    const uint64_t magb  = pair2(12582912.0f, 12582912.0f);
    const float*   src   = in + e;
    const float*   bsrc  = src - p.shift;
    float4         v[kCnt], b[kDiff != Diff::None ? kCnt : 1];
    // 3D, Diff::Some: the elements without a neighbour, a bit each: the zero in its place is no value of
    // the item's.  (2D, where the difference is along y and few items hold such elements beside
    // others, tracks the zeros: the mask there costs 8192x8192 97.6 -> 113 us.)
    constexpr bool kOwn = k3D && kDiff == Diff::Some && kRange == Range::Unknown;
    uint32_t       own  = 0;
#pragma unroll
    for (uint32_t u = 0; u < kCnt; ++u) {
        const uint32_t at = kFull ? u * kStageStep : min(e + u * kStageStep, elast) - e;
        v[u]              = __ldg(reinterpret_cast<const float4*>(src + (int32_t)at));
        const float* bs   = bsrc + (int32_t)at;
        if (kDiff == Diff::All) {
            if (kAl) b[u] = __ldg(reinterpret_cast<const float4*>(bs));
            else b[u] = make_float4(__ldg(bs), __ldg(bs + 1), __ldg(bs + 2), __ldg(bs + 3));
        }
        if (kDiff == Diff::Some && kAl) {
            b[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (pos.row & p.tmask) b[u] = __ldg(reinterpret_cast<const float4*>(bs));
            else if (kOwn) own |= 15u << (4 * u);
            pos.next(p.shift);
        } else if (kDiff == Diff::Some) {
            const uint32_t left = p.shift - pos.rem;  // elements of the group in this row, if < 4
            const bool     r0 = (pos.row & p.tmask) != 0, r1 = ((pos.row + 1) & p.tmask) != 0;
            b[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r0) b[u].x = __ldg(bs);
            if (left > 1 ? r0 : r1) b[u].y = __ldg(bs + 1);
            if (left > 2 ? r0 : r1) b[u].z = __ldg(bs + 2);
            if (left > 3 ? r0 : r1) b[u].w = __ldg(bs + 3);
            if (kOwn) {
                const uint32_t in0 = left >= 4 ? 15u : (1u << left) - 1u;  // the group's elements of this row
                own |= ((r0 ? 0u : in0) | (r1 ? 0u : 15u & ~in0)) << (4 * u);
            }
            pos.next(p.shift);
        }
    }
#pragma unroll
    for (uint32_t u = 0; u < kCnt; ++u) {
        const uint64_t v0 = scale2(pair2(v[u].x, v[u].y), rr), v1 = scale2(pair2(v[u].z, v[u].w), rr);
        uint32_t       q0, q1, q2, q3;
        quant2<kRange == Range::Positive>(v0, magic, q0, q1);
        quant2<kRange == Range::Positive>(v1, magic, q2, q3);
        if (kRange == Range::Unknown) {
            lim.add(v0);
            lim.add(v1);
        }
        if (kDiff != Diff::None) {
            const uint64_t b0 = scale2(pair2(b[u].x, b[u].y), rr), b1 = scale2(pair2(b[u].z, b[u].w), rr);
            uint32_t       s0, s1, s2, s3;
            quant2<kRange == Range::Positive>(b0, magb, s0, s1);
            quant2<kRange == Range::Positive>(b1, magb, s2, s3);
            if (kRange == Range::Unknown) {
                const uint32_t o = own >> (4 * u);
                lim.add(kOwn ? pair2(o & 1u ? lo_of(v0) : lo_of(b0), o & 2u ? hi_of(v0) : hi_of(b0)) : b0);
                lim.add(kOwn ? pair2(o & 4u ? lo_of(v1) : lo_of(b1), o & 8u ? hi_of(v1) : hi_of(b1)) : b1);
            }
            // (the bias stays; the upper halves are dropped below)
            q0 -= s0, q1 -= s1, q2 -= s2, q3 -= s3;
        }
        if (u + 1 < kCnt || mine)
            *reinterpret_cast<uint2*>(dst + u * (kStageStep / 64 * kStageSlot)) =
                make_uint2(__byte_perm(q0, q1, 0x5410), __byte_perm(q2, q3, 0x5410));
    }
}

template <bool k3D, Diff kDiff, bool kAl, Range kRange, bool kFull>
__device__ __forceinline__ void stage_segment(const float* __restrict__ in, uint32_t n, uint32_t base,
                                              const StagePlan& p, float r, Limits& lim, uint8_t* st)
{
    const uint32_t     elast = (n & ~3u) - 4;
    constexpr uint32_t U    = kDiff != Diff::None ? 4 : 8;  // groups in flight per thread
    constexpr uint32_t kDst = kStageStep / 64 * kStageSlot;
    const uint32_t     t4   = 4 * threadIdx.x;
    uint8_t*           dst  = st + 2 * t4 + 8 * (t4 >> 6);
    uint32_t           e    = base + t4;
    if (p.halo && base) {
        uint32_t eh = e - p.halo, left = p.halo;
        StageRow pos(eh, p);
        uint8_t* dh = dst;
#pragma unroll 1
        for (; left > kStageStep; left -= min(left, 2 * kStageStep), eh += 2 * kStageStep, dh += 2 * kDst)
            stage_groups<k3D, 2, kDiff, kAl, kRange, kFull>(in, elast, eh, p, pos, r, lim, dh, t4 + kStageStep < left);
        if (t4 < left) stage_groups<k3D, 1, kDiff, kAl, kRange, kFull>(in, elast, eh, p, pos, r, lim, dh, true);
    }
    dst += p.halo / 64 * kStageSlot;
    StageRow pos(e, p);
#pragma unroll 1
    for (uint32_t k = 0; k < kItemCodes / kStageStep; k += U, e += U * kStageStep, dst += U * kDst)
        stage_groups<k3D, U, kDiff, kAl, kRange, kFull>(in, elast, e, p, pos, r, lim, dst, true);
    if (!kFull && (n & 3u)) {
        // the field's last, partial group: the thread that staged another in its place
        const uint32_t i = p.halo + (n & ~3u) - base;
        if (((n - base) & (kStageStep - 4)) == t4) {
            const uint32_t el = n & ~3u;
            StageRow       at(el, p);
            uint32_t       q[4] = {0, 0, 0, 0};
            for (uint32_t k = 0; k < (n & 3u); ++k) {
                uint32_t unused;
                uint64_t v = scale2(pair2(__ldg(in + el + k), 0.0f), pair2(r, r));
                quant2<kRange == Range::Positive>(v, pair2(12582912.0f + 32768.0f, 0.0f), q[k], unused);
                if (kRange == Range::Unknown) lim.add(pair2(lo_of(v), lo_of(v)));
                if (kDiff == Diff::All || (kDiff == Diff::Some && ((at.rem + k >= p.shift ? at.row + 1 : at.row) & p.tmask))) {
                    uint32_t b;
                    v = scale2(pair2(__ldg(in + el + k - p.shift), 0.0f), pair2(r, r));
                    quant2<kRange == Range::Positive>(v, pair2(12582912.0f, 0.0f), b, unused);
                    if (kRange == Range::Unknown) lim.add(pair2(lo_of(v), lo_of(v)));
                    q[k] -= b;
                }
            }
            *reinterpret_cast<uint2*>(st + 2 * i + 8 * (i >> 6)) =
                make_uint2(__byte_perm(q[0], q[1], 0x5410), __byte_perm(q[2], q[3], 0x5410));
        }
    }
}

// Staging of elements [base - halo, base + kItemCodes) at st; elements before the field are
// left unwritten and elements past it hold some other value (no code follows from either).
// n >= 8, and n >= 2 shift.  lim: takes every x r (Range::Unknown).
template <bool k3D, Range kRange, bool kFull>
__device__ __forceinline__ void stage_item(const float* __restrict__ in, uint32_t n, uint32_t base,
                                           const StagePlan& p, float r, Limits& lim, uint8_t* st)
{
    if (p.shift == 0) return stage_segment<k3D, Diff::None, true, kRange, kFull>(in, n, base, p, r, lim, st);
    // the rows (planes) the staged elements lie in
    const uint32_t r0 = fdiv(base - (base ? p.halo : 0u), p.dshift), r1 = fdiv(base + kItemCodes - 1, p.dshift);
    if (r0 == r1 && (r0 & p.tmask) == 0) return stage_segment<k3D, Diff::None, true, kRange, kFull>(in, n, base, p, r, lim, st);
    if ((r0 & p.tmask) && r1 - r0 <= p.tmask - (r0 & p.tmask)) {
        if (p.shift % 4 == 0) return stage_segment<k3D, Diff::All, true, kRange, kFull>(in, n, base, p, r, lim, st);
        return stage_segment<k3D, Diff::All, false, kRange, kFull>(in, n, base, p, r, lim, st);
    }
    if (p.shift % 4 == 0) return stage_segment<k3D, Diff::Some, true, kRange, kFull>(in, n, base, p, r, lim, st);
    return stage_segment<k3D, Diff::Some, false, kRange, kFull>(in, n, base, p, r, lim, st);
}

// Bits of a where m is set, of b elsewhere.
__device__ __forceinline__ uint32_t pick(uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); }

// Low `k` halves (of 4) set in the pair of words m0, m1; k <= 4.
__device__ __forceinline__ void low_halves(uint32_t k, uint32_t& m0, uint32_t& m1)
{
    m0 = k == 0 ? 0u : k == 1 ? 0xFFFFu : kFull;
    m1 = k <= 2 ? 0u : k == 3 ? 0xFFFFu : kFull;
}

// The 64 deltas of the lane's group of the block that starts at element e0 - 64 lane, two per
// word, biased, from the staged differences; i0 = staged index of e0.
// 1D: 256-element tiles, only the left neighbour; biased by 0x8000.
__device__ __forceinline__ void packed_deltas1(const uint8_t* st, uint32_t i0, uint32_t lane, uint32_t (&w)[32])
{
    const uint8_t* pc = st + (i0 >> 6) * kStageSlot;  // i0 % 64 == 0
    uint32_t       tp = kBias2;
    if (lane & 3u) tp = (uint32_t)*reinterpret_cast<const uint16_t*>(pc - 10) << 16;  // element e0 - 1
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint2 c = *reinterpret_cast<const uint2*>(pc + 8 * j);
        w[2 * j]      = c.x - __byte_perm(tp, c.x, 0x5432) + kBias2;
        w[2 * j + 1]  = c.y - __byte_perm(c.x, c.y, 0x5432) + kBias2;
        tp            = c.y;
    }
}

// 2D and 3D; biased by 0x8080; returns nonzero bits under 0xFF00FF00 where a delta does not fit 8
// bits.  kRow: subtract the row above (2D with the row staged, 3D).  kX: x % 4 where the row
// above is read (0, 2, or 1 for any odd x).  Rows of 64 elements and more end at most once in
// a lane's 64: that end, inside a group of 4, is behind a test of a warp-wide mask, and which
// elements start a tile row -- every 16th (8th) -- is kept as masks.  kNarrow (8 <= x < 64):
// both are found for each group.
template <int ND, bool kRow, int kX, bool kNarrow>
__device__ __forceinline__ uint32_t packed_deltas(const uint8_t* st, uint32_t i0, uint32_t e0, uint32_t x, uint32_t y,
                                              uint32_t xy, const FastDiv& dx, const FastDiv& dxy, uint32_t (&w)[32])
{
    constexpr uint32_t tw = ND == 2 ? 15u : 7u;  // tile width - 1
    constexpr int      kPer = (tw + 1) / 2;      // words of its period
    const uint8_t*     pc = st + (i0 >> 6) * kStageSlot;  // i0 % 64 == 0
    uint32_t           rw, col;  // row (3D: of the plane) and column of e0 (kNarrow: of the group)
    if (ND == 2) {
        rw = fdiv(e0, dx), col = e0 - rw * x;
    } else {
        const uint32_t rem = e0 - fdiv(e0, dxy) * xy;
        rw = fdiv(rem, dx), col = rem - rw * x;
    }
    const uint32_t q   = x - col;  // elements left in the row; the next row's first is element q (if < 64)
    uint32_t       rwn = ND == 3 && rw + 1 == y ? 0u : rw + 1;
    uint32_t       my  = (rw & tw) ? kFull : 0u;  // the row above lies in the tile
    uint32_t       myn = (rwn & tw) ? kFull : 0u;
    const uint32_t wu  = kNarrow ? 0u : __reduce_or_sync(kFull, q < 64 ? 1u << (q >> 2) : 0u);  // groups with a row's first element
    // halves of the words w, w + kPer, ... that start a tile row (kX == 0: low halves only)
    uint32_t sm[kPer];
    auto starts = [&](uint32_t k) {  // element k of the period starts one
#pragma unroll
        for (int i = 0; i < kPer; ++i) sm[i] = (k >> 1) == (uint32_t)i ? ((k & 1u) ? 0xFFFF0000u : 0xFFFFu) : 0u;
    };
    starts((0u - col) & tw);
    // the row above: halves h0 + k of the staging slots from ra on, h0 the same in every lane
    const uint32_t h0 = (0u - x) & 63u;
    uint32_t       last = 0, wide = 0, tp;  // tp: T of element e0 - 1 in the high half
    const uint8_t* ra = nullptr;
    auto word = [&](uint32_t h) { return *reinterpret_cast<const uint32_t*>(ra + 2 * h + ((h & 64u) >> 3)); };
    {
        uint32_t t = *reinterpret_cast<const uint16_t*>(pc - 10);
        if (kRow) {
            const uint32_t ir = i0 - x, il = ir - 1;  // ir >= halo - x > 0, ir % 64 == h0
            ra = st + (ir >> 6) * kStageSlot;
            const uint32_t tn = *reinterpret_cast<const uint16_t*>(st + 2 * il + 8 * (il >> 6));
            t = t - (my ? tn : 0x8000u) + 0x8000u;
            if (kX == 1) last = word(h0 - 1);  // h0 is odd
        }
        tp = t << 16;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint2 c   = *reinterpret_cast<const uint2*>(pc + 8 * j);
        uint32_t    t01 = c.x, t23 = c.y, m0 = my, m1 = my, s0 = sm[2 * j % kPer], s1 = sm[(2 * j + 1) % kPer];
        if (kNarrow) {
            const uint32_t k = (0u - col) & tw;  // element k starts a tile row (if < 4)
            s0 = k == 0 ? 0xFFFFu : k == 1 ? 0xFFFF0000u : 0u, s1 = k == 2 ? 0xFFFFu : k == 3 ? 0xFFFF0000u : 0u;
            col += 4;
            if (col >= x) {  // the group ends its row; its last col elements are in the next
                col -= x;
                uint32_t o0, o1, f0, f1;  // elements of the old row, and those and the new row's first
                low_halves(4 - col, o0, o1);
                low_halves(col ? 5 - col : 4u, f0, f1);
                m0 = pick(o0, my, myn), m1 = pick(o1, my, myn), my = myn;
                s0 = (s0 & o0) | (f0 & ~o0), s1 = (s1 & o1) | (f1 & ~o1);
                ++rwn;
                if (ND == 3 && rwn == y) rwn = 0;
                myn = (rwn & tw) ? kFull : 0u;
            }
        } else if (wu & (1u << j)) {  // (warp-uniform)
            if ((q >> 2) == (uint32_t)j) {
                uint32_t o0, o1;  // elements of the old row
                low_halves(q & 3u, o0, o1);
                m0 = pick(o0, my, myn), m1 = pick(o1, my, myn), my = myn;
                s0 &= o0, s1 &= o1;
                starts(q & tw);
                s0 |= sm[2 * j % kPer], s1 |= sm[(2 * j + 1) % kPer];
            }
        }
        if (kRow) {
            const uint32_t h = h0 + 4 * j;
            uint32_t       a0, a1;
            if (kX == 0) {
                const uint2 v = *reinterpret_cast<const uint2*>(ra + 2 * h + ((h & 64u) >> 3));
                a0 = v.x, a1 = v.y;
            } else if (kX == 2) {
                a0 = word(h), a1 = word(h + 2);
            } else {
                const uint32_t u = word(h + 1), v = word(h + 3);
                a0 = __byte_perm(last, u, 0x5432), a1 = __byte_perm(u, v, 0x5432);
                last = v;
            }
            t01 = t01 - pick(m0, a0, kBias2) + kBias2;
            t23 = t23 - pick(m1, a1, kBias2) + kBias2;
        }
        w[2 * j]     = t01 - pick(s0, kBias2, __byte_perm(tp, t01, 0x5432)) + kBias2s;
        w[2 * j + 1] = t23 - (kX == 0 ? __byte_perm(t01, t23, 0x5432) : pick(s1, kBias2, __byte_perm(t01, t23, 0x5432))) + kBias2s;
        wide |= (w[2 * j] ^ kBias2) | (w[2 * j + 1] ^ kBias2);
        tp = t23;
    }
    return wide;
}

// Bit planes of 32 words of two biased deltas (after the transpose: plane p of the low
// deltas in w[p], of the high ones in w[16 + p]) to the planes of their sign-magnitude codes:
// the sign is the inverted top plane, and where it is set the lower planes are negated with a
// rippling carry -- two three-input operations a plane, less than negating each word's
// halves before the transpose.  1D: codes at i % 4 != 0 (every high delta
// and the low ones of odd words) carry the magnitude only; the signs' planes are returned.
template <bool k1D>
__device__ __forceinline__ void sign_planes(uint32_t (&w)[32], uint32_t& slow, uint32_t& shigh)
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t s = ~w[16 * h + 15];
        uint32_t       c = s;
#pragma unroll
        for (int p = 0; p < 15; ++p) {
            const uint32_t b = w[16 * h + p];
            w[16 * h + p]    = b ^ s ^ c;
            c                = (b ^ s) & c;
        }
        w[16 * h + 15] = k1D ? (h ? 0u : s & 0x55555555u) : s;
        (h ? shigh : slow) = s;
    }
}

// Two biased deltas e as sign-magnitude codes (for a few words outside the transpose): for d < 0
// the code is -e in 16 bits, otherwise e ^ 0x8000.  neg: 1 in bit 0 (16) where the low (high)
// delta is negative.
__device__ __forceinline__ uint32_t sign_mag2(uint32_t e, uint32_t& neg)
{
    uint32_t pos;  // 0xFFFF where d >= 0: the top bit of each half, replicated (prmt mode 8 + byte)
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(pos) : "r"(e));
    neg = ~pos & 0x00010001u;
    return (e ^ (~pos | kBias2)) + neg;
}

// Deltas that all fit 8 bits (biased by 0x8080) to the planes of their sign-magnitude codes:
// gathered to bytes, 8x8 blocks transposed, half the work of the 32x32 transpose.  lo, hi: planes
// 0..7 of the low and high codes (7: magnitude 128), sl, sh: their signs.
__device__ __forceinline__ void byte_planes(const uint32_t (&w)[32], uint32_t (&lo)[8], uint32_t (&hi)[8], uint32_t& sl,
                                            uint32_t& sh)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // the low (high) codes of pairs i, 8 + i, 16 + i, 24 + i
        const uint32_t x = __byte_perm(w[i], w[8 + i], 0x6240), y = __byte_perm(w[16 + i], w[24 + i], 0x6240);
        lo[i] = __byte_perm(x, y, 0x5410), hi[i] = __byte_perm(x, y, 0x7632);
    }
    transpose8(lo);
    transpose8(hi);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t (&p)[8] = h ? hi : lo;
        const uint32_t s = ~p[7];
        uint32_t       c = s;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            const uint32_t b = p[i];
            p[i]             = b ^ s ^ c;
            c                = (b ^ s) & c;
        }
        p[7] = c;
        (h ? sh : sl) = s;
    }
}

// Bit k of v to bit 2 k (k < 16).
__device__ __forceinline__ uint32_t spread16(uint32_t v)
{
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u;
    return (v | (v << 1)) & 0x55555555u;
}

}  // namespace fz
