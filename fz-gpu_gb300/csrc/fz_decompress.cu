// fz_decompress.cu -- decompression kernels (the inverse of fz_compress.cuh).
//
//   k_decompress1d/2d/3d  fused decode + inverse bitshuffle + inverse Lorenzo, from the
//              stream straight into the field: each CTA decodes the 64-code groups its
//              rows (or 256-element blocks) need -- rank of every flagged chunk from the
//              bitmap and the block offset table, inverse 32x32 bit transposes -- then
//              runs the per-tile inclusive prefix sums (1D 256, 2D 16x16, 3D 8x8x8 -- the
//              tiling of x_lorenzo_{1d,2d,3d}, lorenzo_var.cuh:297-518) in 32-bit integers
//              (1D) or in floats that hold them exactly, and writes p * ebx2.
//   k_offsets  block offset table from the bitmap (COMPAT streams, which carry none).
//   k_recon{1,2,3}d  inverse Lorenzo of a code array (the stage-level API,
//              fz_lorenzo_reconstruct).
//
// The reference has no working FZ decompressor (its x_lorenzo kernels read a separate
// signum array that its compressor never writes), so this path is the exact inverse of
// the compressed format rather than a restatement.
#include <algorithm>
#include <atomic>

#include "fz_internal.h"

namespace fz {

// ------------------------------------------------------------- offsets --
// boff[b] = chunks of blocks 0..b-1 (the exclusive scan fz.cu:187-192 restricted to
// block granularity), boff[nb] = the total, checked against the header's nnz.  One
// thread per block (two 16-byte bitmap loads), CTAs of 256 chained by look-back.
constexpr uint32_t kOffThreads = 256;

__global__ void __launch_bounds__(kOffThreads) k_offsets(const uint8_t* __restrict__ st, uint64_t off_a,
                                                        uint32_t nb, uint64_t nnz, uint32_t* boff,
                                                        uint64_t* state, uint32_t* ticket,
                                                        uint32_t* status, uint32_t* epoch_word)
{
    __shared__ uint32_t s_w[kOffThreads / 32];
    __shared__ uint32_t cta_tile, s_excl, s_epoch;
    if (threadIdx.x == 0) {
        s_epoch = __ldcg(epoch_word);
        __threadfence();
        cta_tile = take_ticket(ticket, epoch_word, gridDim.x).tile;
    }
    __syncthreads();
    const uint32_t ct = cta_tile, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t epoch = s_epoch;
    const uint32_t b  = ct * kOffThreads + threadIdx.x;
    uint32_t       c  = 0;
    if (b < nb) {
        const uint4* A = reinterpret_cast<const uint4*>(st + off_a) + 2 * (size_t)b;
        const uint4  u = __ldg(A), v = __ldg(A + 1);
        c = __popc(u.x) + __popc(u.y) + __popc(u.z) + __popc(u.w) + __popc(v.x) + __popc(v.y) +
            __popc(v.z) + __popc(v.w);
    }
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, inc, o);
        if (lane >= (uint32_t)o) inc += u;
    }
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const uint32_t v = lane < kOffThreads / 32 ? s_w[lane] : 0u;
        uint32_t       vi = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(kFull, vi, o);
            if (lane >= (uint32_t)o) vi += u;
        }
        if (lane < kOffThreads / 32) s_w[lane] = vi - v;  // exclusive warp offsets
        const uint32_t tot  = __shfl_sync(kFull, vi, 31);
        uint32_t       excl = 0, povf = 0;
        if (ct == 0) {
            if (lane == 0) publish(state, 0, epoch, kFlagIncl, 0, tot);
        } else {
            if (lane == 0) publish(state, ct, epoch, kFlagAgg, 0, tot);
            lookback(state, ct, epoch, status, excl, povf);
            if (lane == 0) publish(state, ct, epoch, kFlagIncl, 0, excl + tot);
        }
        if (lane == 0) {
            s_excl = excl;
            if (ct == gridDim.x - 1) {
                boff[nb] = excl + tot;
                if (excl + tot != nnz) atomicOr(status, kStatusCorrupt);
            }
        }
    }
    __syncthreads();
    if (b < nb) boff[b] = s_excl + s_w[wid] + inc - c;
}

cudaError_t launch_offsets(const uint8_t* st, uint64_t off_a, uint32_t nb, uint32_t nwords, uint64_t nnz,
                           uint32_t* boff, uint64_t* state, uint32_t* ticket, uint32_t* status,
                           uint32_t* epoch, cudaStream_t s)
{
    (void)nwords;
    const uint32_t ctas = (uint32_t)std::max<uint64_t>(1, cdiv(nb, kOffThreads));
    k_offsets<<<ctas, kOffThreads, 0, s>>>(st, off_a, nb, nnz, boff, state, ticket, status, epoch);
    return cudaGetLastError();
}

// Gathers the shuffled image S of block t (words 4c..4c+3 of chunk c = lane + 32 i) into
// shared memory; flagged chunks come from Section B in order, the others are zero.
__device__ __forceinline__ void gather_block(const DecodeArgs& a, uint32_t t, uint32_t lane, uint32_t* sm)
{
    const uint4*   A4 = reinterpret_cast<const uint4*>(a.st + a.off_a) + 2 * (size_t)t;
    const uint4    b0 = __ldg(A4), b1 = __ldg(A4 + 1);
    const uint32_t bm[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    const uint4*   B   = reinterpret_cast<const uint4*>(a.st + a.off_b);
    const uint32_t lt  = lanemask_lt();
    uint32_t       pre = __ldg(a.boff + t);
    const uint32_t end = __ldg(a.boff + t + 1);
    bool           bad = false;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        uint4          v    = make_uint4(0, 0, 0, 0);
        const uint32_t rank = pre + __popc(bm[i] & lt);
        if ((bm[i] >> lane) & 1u) {
            if (rank < a.nnz) v = __ldg(B + rank);
            else bad = true;  // the bitmap claims more chunks than the stream holds
        }
        *reinterpret_cast<uint4*>(sm + (lane + 32 * i) * 4) = v;
        pre += __popc(bm[i]);
    }
    bad |= pre != end;  // bitmap and offset table disagree
    if (bad) atomicOr(a.status, kStatusCorrupt);
}

__device__ __forceinline__ uint32_t sm_decode(uint32_t c)
{
    const uint32_t mag = c & 0x7FFFu;
    return (c & 0x8000u) ? 0u - mag : mag;
}

// Both sign-magnitude codes of a word w = c0 | c1 << 16 as two's-complement deltas: the
// sign bit 15 (31) spread into an all-ones mask m, (mag ^ m) - m is -mag exactly when the
// sign is set -- sm_decode for both halves.
__device__ __forceinline__ void sm_decode2(uint32_t w, uint32_t& d0, uint32_t& d1)
{
    // m0, m1: byte permutes whose selectors replicate the sign bit of byte 1 (bit 15) and of
    // byte 3 (bit 31) into every byte (prmt's default mode, selector nibble 8 + byte)
    uint32_t m0, m1;
    asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(m0) : "r"(w));
    asm("prmt.b32 %0, %1, 0, 0xBBBB;" : "=r"(m1) : "r"(w));
    d0 = ((w & 0x7FFFu) ^ m0) - m0;
    d1 = ((__byte_perm(w, 0u, 0x4432) & 0x7FFFu) ^ m1) - m1;
}

// *p where cond is not 0, 0 elsewhere: a predicated load (the compiler makes a branch of the
// conditional expression).
__device__ __forceinline__ uint32_t ldg_if(const uint32_t* p, uint32_t cond)
{
    uint32_t v;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.u32 %0, 0; @q ld.global.nc.u32 %0, [%1]; }"
                 : "=r"(v)
                 : "l"(p), "r"(cond));
    return v;
}

// Bit planes of 32 words of two sign-magnitude codes (plane p of the low codes in w[p], of the
// high ones in w[16 + p]) to the planes of their deltas plus 0x8000: where the sign is set the
// magnitude is negated with a rippling carry, then the top bit inverted -- two three-input
// operations a plane, instead of several per code after the transpose.  (A set sign on a zero
// magnitude is zero, as in sm_decode.)
__device__ __forceinline__ void delta_planes(uint32_t (&w)[32])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t s = w[16 * h + 15];
        uint32_t       c = s;
#pragma unroll
        for (int p = 0; p < 15; ++p) {
            const uint32_t b = w[16 * h + p];
            w[16 * h + p]    = b ^ s ^ c;
            c                = (b ^ s) & c;
        }
        w[16 * h + 15] = ~(s ^ c);
    }
}

// Two sign-magnitude codes of a word as deltas plus 0x8000 (the few codes outside the shuffled
// blocks).
__device__ __forceinline__ uint32_t delta_word(uint32_t w)
{
    return ((sm_decode(w & 0xFFFFu) + 0x8000u) & 0xFFFFu) | ((sm_decode(w >> 16) + 0x8000u) << 16);
}

// A lane's group gg of block b is word r4 = gg % 4 of the 32 chunks (p, k = gg / 4): the ranks of
// those among the flagged chunks follow from the block's bitmap and its offset boff[b].  bm
// holds the bitmap (chunk (p, k) at bit 8 (p % 4) + k of word p / 4), all zero when the offset
// table disagrees with it or the block's chunks lie outside the stream (nothing is read then);
// W4 the word r4 of the block's first chunk.
struct GroupBits {
    uint32_t        bm[8], k;
    const uint32_t* W4;
};
__device__ __forceinline__ GroupBits group_bits(const DecodeArgs& a, uint32_t g)
{
    GroupBits      G;
    const uint32_t b = g >> 5;
    const uint4*   A4 = reinterpret_cast<const uint4*>(a.st + a.off_a) + 2 * (size_t)b;
    const uint4    b0 = __ldg(A4), b1 = __ldg(A4 + 1);
    const uint32_t base = __ldg(a.boff + b), end = __ldg(a.boff + b + 1);
    G.k  = (g & 31u) >> 2;
    G.W4 = reinterpret_cast<const uint32_t*>(a.st + a.off_b) + (g & 3u) + 4 * (size_t)base;
    // then every rank below is < nnz
    const bool bad = end - base != (uint32_t)(__popc(b0.x) + __popc(b0.y) + __popc(b0.z) + __popc(b0.w) +
                                              __popc(b1.x) + __popc(b1.y) + __popc(b1.z) + __popc(b1.w)) ||
                     end < base || end > a.nnz;
    const uint32_t live = bad ? 0u : kFull;
    G.bm[0] = b0.x & live, G.bm[1] = b0.y & live, G.bm[2] = b0.z & live, G.bm[3] = b0.w & live;
    G.bm[4] = b1.x & live, G.bm[5] = b1.y & live, G.bm[6] = b1.z & live, G.bm[7] = b1.w & live;
    if (bad) atomicOr(a.status, kStatusCorrupt);
    return G;
}
// Planes 4 i + q, q in [q0, q1), into w[4 i + q]; W4 moves past the word's chunks.
template <int i, int q0, int q1>
__device__ __forceinline__ void gather_planes(GroupBits& G, uint32_t* w)
{
#pragma unroll
    for (int q = q0; q < q1; ++q) {
        const uint32_t bit = 1u << (8 * q + G.k);
        w[q] = ldg_if(G.W4 + 4 * __popc(G.bm[i] & (bit - 1u)), G.bm[i] & bit);
    }
    G.W4 += 4 * __popc(G.bm[i]);
}

// Plane 4 i + 3 alone.
template <int i>
__device__ __forceinline__ void gather_sign(GroupBits& G, uint32_t& w)
{
    const uint32_t bit = 1u << (24 + G.k);
    w = ldg_if(G.W4 + 4 * __popc(G.bm[i] & (bit - 1u)), G.bm[i] & bit);
    G.W4 += 4 * __popc(G.bm[i]);
}

// The 64 codes of group g (codes g*64 .. g*64+63) as 32 words w[j] = code[2j] | code[2j+1] << 16.
// Groups past the last full block read the sidecar.
__device__ __forceinline__ void tail_group(const DecodeArgs& a, uint32_t g, uint32_t (&w)[32])
{
    const uint16_t* tc  = a.mode == 1 ? reinterpret_cast<const uint16_t*>(a.st + a.off_c) : nullptr;
    const uint32_t  e0  = g * 64;
    const uint32_t  tb  = a.nb * kBlockCodes;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const uint32_t e  = e0 + 2 * j;
        const uint32_t lo = (tc && e < a.n) ? tc[e - tb] : 0u;
        const uint32_t hi = (tc && e + 1 < a.n) ? tc[e + 1 - tb] : 0u;
        w[j] = lo | (hi << 16);
    }
}
__device__ __forceinline__ void gather_group(GroupBits& G, uint32_t (&w)[32])
{
    gather_planes<0, 0, 4>(G, w);
    gather_planes<1, 0, 4>(G, w + 4);
    gather_planes<2, 0, 4>(G, w + 8);
    gather_planes<3, 0, 4>(G, w + 12);
    gather_planes<4, 0, 4>(G, w + 16);
    gather_planes<5, 0, 4>(G, w + 20);
    gather_planes<6, 0, 4>(G, w + 24);
    gather_planes<7, 0, 4>(G, w + 28);
}
__device__ __forceinline__ void decode_group(const DecodeArgs& a, uint32_t g, uint32_t (&w)[32])
{
    if ((g >> 5) < a.nb) {
        GroupBits G = group_bits(a, g);
        gather_group(G, w);
        transpose32<true>(w);  // w[p] = S[p*32 + gg]  ->  w[j] = W[gg*32 + j]
    } else {
        tail_group(a, g, w);
    }
}

// Both deltas of byte c of the low and of the high word, sign-extended, plus 0x8000.
template <int c>
__device__ __forceinline__ uint32_t delta_bytes(uint32_t lo, uint32_t hi)
{
    uint32_t r;  // bytes c, its sign, 4 + c, its sign (prmt mode 8 + byte)
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "n"(0xC480 + 0x1111 * c));
    return r ^ 0x80008000u;
}

// The 64 deltas of group g plus 0x8000, two per word as decode_group's codes; all lanes of the
// warp call it, those without a group (valid false) get some values.  Where no lane of the warp
// has a magnitude of 2^7 or more -- most warps of a compressible stream: only tile corners
// hold values instead of differences -- planes 7..14 of either half are neither fetched nor
// transposed: 16 planes as bytes, widened at the end.
__device__ __forceinline__ void decode_deltas(const DecodeArgs& a, uint32_t g, bool valid, uint32_t (&w)[32])
{
    const bool in_block = valid && (g >> 5) < a.nb;
    GroupBits  G;
#pragma unroll
    for (int i = 0; i < 8; ++i) G.bm[i] = 0;
    G.k = 0, G.W4 = nullptr;
    if (in_block) G = group_bits(a, g);
    const uint32_t high = ((G.bm[1] & 0xFF000000u) | G.bm[2] | (G.bm[3] & 0x00FFFFFFu) | (G.bm[5] & 0xFF000000u) | G.bm[6] |
                           (G.bm[7] & 0x00FFFFFFu)) & (0x01010101u << G.k);
    if (!__any_sync(kFull, high != 0 || (valid && !in_block))) {
        uint32_t t[2][8], s[2];
        gather_planes<0, 0, 4>(G, t[0]);
        gather_planes<1, 0, 3>(G, t[0] + 4);
        gather_planes<2, 0, 0>(G, nullptr);
        gather_sign<3>(G, s[0]);
        gather_planes<4, 0, 4>(G, t[1]);
        gather_planes<5, 0, 3>(G, t[1] + 4);
        gather_planes<6, 0, 0>(G, nullptr);
        gather_sign<7>(G, s[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // as delta_planes, the sign plane kept
            uint32_t c = s[h];
#pragma unroll
            for (int p = 0; p < 7; ++p) {
                const uint32_t b = t[h][p];
                t[h][p]          = b ^ s[h] ^ c;
                c                = (b ^ s[h]) & c;
            }
            t[h][7] = s[h] ^ c;
            transpose8(t[h]);  // byte c of t[h][i]: the delta of pair 8 c + i
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            w[i]      = delta_bytes<0>(t[0][i], t[1][i]);
            w[8 + i]  = delta_bytes<1>(t[0][i], t[1][i]);
            w[16 + i] = delta_bytes<2>(t[0][i], t[1][i]);
            w[24 + i] = delta_bytes<3>(t[0][i], t[1][i]);
        }
        return;
    }
    if (in_block) {
        gather_group(G, w);
        delta_planes(w);
        transpose32<true>(w);
    } else if (valid) {
        tail_group(a, g, w);
#pragma unroll
        for (int j = 0; j < 32; ++j) w[j] = delta_word(w[j]);
    }
}

// Decoded row buffers (fused 2D/3D paths): a row of the field's window is held as 64-code slots
// (one decode group each) of 36 words: code e at word (e / 64) * 36 + (e % 64) / 2.  The
// 16-byte pad per slot puts neighbouring slots 4 banks apart, so the 16-byte stores of 8
// threads writing chunk tt of consecutive groups hit distinct banks; it repeats the next
// slot's first two words, so that 5 codes from anywhere are three words in a row.
constexpr uint32_t kSlotWords = 36;

// word holding code e: e / 2 + 4 (e / 64)
__device__ __forceinline__ uint32_t rb_word(uint32_t e) { return (e >> 1) + 4 * (e >> 6); }

// Group j's deltas into slot j; kPads: the first two words into the pad of the slot before too.
template <bool kPads>
__device__ __forceinline__ void rb_put_group(uint32_t* rb, uint32_t j, const uint32_t (&w)[32])
{
#pragma unroll
    for (uint32_t tt = 0; tt < 8; ++tt)
        *reinterpret_cast<uint4*>(rb + j * kSlotWords + 4 * tt) =
            make_uint4(w[4 * tt], w[4 * tt + 1], w[4 * tt + 2], w[4 * tt + 3]);
    if (kPads && j) *reinterpret_cast<uint2*>(rb + j * kSlotWords - 4) = make_uint2(w[0], w[1]);
}

// The deltas (plus 0x8000) of codes i..i+3 of a row buffer as two words of two.  kAl: i % 4 == 0.
template <bool kAl>
__device__ __forceinline__ void rb_read4(const uint32_t* rb, uint32_t i, uint32_t& x01, uint32_t& x23)
{
    const uint32_t* p = rb + rb_word(i);
    if (kAl) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        x01 = v.x, x23 = v.y;
    } else {
        const uint32_t u = p[0], v = p[1], w = p[2], sel = (i & 1u) ? 0x5432u : 0x3210u;
        x01 = __byte_perm(u, v, sel), x23 = __byte_perm(v, w, sel);
    }
}

// Prefix sums in float, two values per instruction (add/mul.f32x2).  Every partial sum is an
// integer of at most 512 deltas below 2^15 (an 8x8x8 tile; 256 in 2D), so below 2^24 and exact:
// the sums equal the 32-bit integer ones and their product with ebx2 is bit-identical.
struct Pair {
    float x, y;
};
__device__ __forceinline__ Pair add2(Pair a, Pair b)
{
    Pair r;
    asm("{ .reg .b64 s, t; mov.b64 s, {%2, %3}; mov.b64 t, {%4, %5}; add.rn.f32x2 s, s, t; mov.b64 {%0, %1}, s; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, float b)
{
    Pair r;
    asm("{ .reg .b64 s, t; mov.b64 s, {%2, %3}; mov.b64 t, {%4, %4}; mul.rn.f32x2 s, s, t; mov.b64 {%0, %1}, s; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b));
    return r;
}
// Both deltas of a word of two plus 0x8000: each half under the exponent of 2^23, less 2^23 + 2^15.
__device__ __forceinline__ Pair delta2(uint32_t x)
{
    const Pair f{__uint_as_float(__byte_perm(x, 0x4B000000u, 0x7410)), __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7432))};
    return add2(f, Pair{-8421376.0f, -8421376.0f});
}

// Stores min(live, 4) reconstructed values at out (none for live <= 0).  kAl: all 4, 16-byte
// aligned, as streaming stores: the field is written once and would push the stream out of the
// L2 (GB300: 39200x388 18.7 -> 17.6 us, 1100x200x100 44.3 -> 39.5, 500x500x100 31.2 -> 30.4).
// (Rows that start anywhere: gathering the aligned groups of 4 from neighbouring threads by
// shuffle took more instructions than its wider stores saved, 501x500x100 on GB300 46.6 -> 49.1
// us.)
template <bool kAl>
__device__ __forceinline__ void store_row(float* out, int32_t live, Pair a, Pair b, float ebx2)
{
    const Pair f = mul2(a, ebx2), g = mul2(b, ebx2);
    if (kAl) {
        if (live > 0) __stcs(reinterpret_cast<float4*>(out), make_float4(f.x, f.y, g.x, g.y));
    } else if (live >= 4) {
        if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
            *reinterpret_cast<float4*>(out) = make_float4(f.x, f.y, g.x, g.y);
        } else {
            out[0] = f.x, out[1] = f.y, out[2] = g.x, out[3] = g.y;
        }
    } else if (live > 0) {
        out[0] = f.x;
        if (live > 1) out[1] = f.y;
        if (live > 2) out[2] = g.x;
    }
}

// A thread's 4 deltas of a row to the sums along x up to its 4 columns: serially, then over the
// threads of the tile row (kQuads threads of 4 columns, q this one's place).
template <int kQuads>
__device__ __forceinline__ void sums_x(uint32_t x01, uint32_t x23, uint32_t q, Pair& a, Pair& b)
{
    a = delta2(x01), b = delta2(x23);
    a.y += a.x, b.x += a.y, b.y += b.x;
    float v = b.y, u = __shfl_up_sync(kFull, v, 1);
    if (kQuads == 2) {
        u = (q & 1u) ? u : 0.0f;
    } else {
        if (q >= 1) v += u;
        u = __shfl_up_sync(kFull, v, 2);
        if (q >= 2) v += u;
        u = v - b.y;
    }
    a = add2(a, Pair{u, u}), b = add2(b, Pair{u, u});
}

// ------------------------------------------------------ fused 2D decode --
// A CTA owns a 16-row tile band and a 960-column window (60 tile columns); the flat
// block index runs over windows fastest.  Phase 1: thread (row rr, j) decodes group
// glo(rr) + j of that row's span into the row buffer.  Phase 2: thread t owns columns
// 4t..4t+3; prefix along x (serial + quad shuffles), running sum along y, times ebx2,
// coalesced stores.  Traffic: the chunks once (plus the at most two groups a row shares
// with the next window) and the output once.
//
// Bound by instruction issue (70%), then by the tail of a last wave.  GB300, event-timed, with
// the signs undone in the bit planes, planes 7..14 left out where a warp has none, and the sums
// in float pairs, against a sign per code and integer sums: 39200x388 20.7 -> 18.5 us (17.6 with
// the streaming stores), 8192x8192 69.7 -> 57.5, 3601x1801 16.9 -> 14.6; 3600x1800 12.6 as with the separate kernel for
// x % 16 == 0 (12.3-13.0) that it replaces.  256 threads, 4 CTAs an SM (64 registers): 5 CTAs of
// 48 registers spill (3600x1800 13.5 us, 39200x388 18.8, 8192x8192 56.1); 128 threads with
// 448-column windows lose as much to the groups shared between windows (14.1, 19.0, 59.5).
constexpr uint32_t kT2 = 256;            // threads
constexpr uint32_t kW2 = 4 * kT2 - 64;   // columns of a window: their codes touch at most kT2 / 16 groups a row

// kAl: x % 4 == 0.  Windows start at multiples of kW2 columns, so every row's window then
// starts on a 4-code boundary: a thread's 4 codes are one 8-byte pair of row-buffer words,
// its 4 outputs one 16-byte store (c1 - c0 is a multiple of 4, so a live thread has all
// 4 columns), and nothing about alignment or width is decided per row.
template <bool kAl>
__global__ void __launch_bounds__(kT2, 4) k_decompress2d(const DecodeArgs a, uint32_t nwin)
{
    pdl_wait();
    pdl_trigger();
    constexpr uint32_t kG = kT2 / 16;  // groups per row
    __shared__ __align__(16) uint32_t rows[16][kG * kSlotWords];
    const uint32_t tid = threadIdx.x;
    const uint32_t bx = blockIdx.x % nwin, by = blockIdx.x / nwin;
    const uint32_t c0 = bx * kW2, c1 = min(c0 + kW2, a.x);
    const uint32_t r0 = by * 16;
    {
        const uint32_t rr = tid / kG, j = tid % kG, row = r0 + rr;
        const uint32_t lin0 = row * a.x + c0, g = (lin0 >> 6) + j;
        const bool     valid = row < a.y && g <= ((lin0 + (c1 - c0) - 1) >> 6);
        uint32_t       w[32];
        decode_deltas(a, g, valid, w);
        if (valid) rb_put_group<!kAl>(rows[rr], j, w);
    }
    __syncthreads();
    const uint32_t col  = c0 + 4 * tid;
    const bool     live = col < c1;
    const uint32_t q    = tid & 3u;
    Pair           s0{0.0f, 0.0f}, s1{0.0f, 0.0f};  // sums along y of the 4 columns
    const uint32_t nrows = min(16u, a.y - r0);
    uint32_t       lin0  = r0 * a.x + c0;  // first code of the window in row r0 + rr
    // threads past the window's end read the row's first codes (same alignment, in bounds; their
    // values reach only higher quad positions, past the end too, and are not stored)
    const uint32_t t4 = live ? 4 * tid : 0u;
#pragma unroll 4
    for (uint32_t rr = 0; rr < 16; ++rr) {
        if (rr >= nrows) break;  // uniform across the CTA
        uint32_t       x01, x23;
        const uint32_t i = (lin0 & 63u) + t4;
        rb_read4<kAl>(rows[rr], i, x01, x23);
        Pair d0, d1;
        sums_x<4>(x01, x23, q, d0, d1);
        s0 = add2(s0, d0), s1 = add2(s1, d1);
        store_row<kAl>(a.out + lin0 + 4 * tid, (int32_t)(c1 - col), s0, s1, a.ebx2);
        lin0 += a.x;
    }
}

// ------------------------------------------------------ fused 3D decode --
// A CTA owns `bands` 8-row tile bands x one 8-plane tile slab x a window of w columns
// (w a multiple of 8, at most 960); the flat block index runs over windows, then band
// groups, then slabs.  The slab is walked two planes at a time.  Phase 1 decodes the
// pass's codes into row buffers: when the window spans whole rows (x <= 960) a plane's
// rows are one contiguous range of codes, decoded group by group into one buffer of pg
// slots ("span" mode, no group decoded twice inside the CTA); otherwise each of the
// bands x 8 rows of a plane gets its own buffer of g slots.  Phase 2: thread (band, cq)
// owns columns 4cq..4cq+3 of its band; prefix along x within the 8-column tile row (pair
// shuffle), running sum along y within the plane, running sum along z in shared memory
// (one 16-byte slot per thread and row: in registers they would spill), then the
// stores.
//
// Bound by the latency of its phases at the 20 warps an SM the slabs leave (a thread per 4 columns
// and 8 rows), then by instruction issue (50%).  GB300, event-timed, with the decode and the sums
// of the 2D kernel and 128 threads a CTA, against a sign per code, integer sums and 256 threads:
// 500x500x100 41.2 -> 31.1 us, 256x256x256 38.9 -> 24.3, 501x500x100 55.3 -> 42.6, 64x64x64 24.1
// -> 14.4; with both planes of a pass in one loop over the rows 30.2 -> 28.5, 23.3 -> 22.4, 42.5 ->
// 39.5 and 14.4 -> 12.5.  Decoding plane p + 1 by half the warps while the others sum plane p: 37.1.
struct Brick3 {
    uint32_t w, q2, bands, g;  // window columns, column quads, bands per CTA, slots per row
    uint32_t nwin, nbgrp;      // windows along x, band groups along y
    uint32_t span, pg;         // span mode; slots per plane buffer
    uint32_t t;                // threads
};
constexpr uint32_t kW3 = 960;

// kAl: x % 4 == 0 (every group of 4 columns is whole and aligned, in the buffers and in the field).
// kT: threads.
template <bool kSpan, bool kAl, uint32_t kT>
__global__ void __launch_bounds__(kT, 768 / kT) k_decompress3d(const DecodeArgs a, const Brick3 k)
{
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint32_t rb3[];
    const uint32_t tid = threadIdx.x;
    const uint32_t bx = blockIdx.x % k.nwin, rest = blockIdx.x / k.nwin;
    const uint32_t by = rest % k.nbgrp, bz = rest / k.nbgrp;
    const uint32_t c0 = bx * k.w, c1 = min(c0 + k.w, a.x);
    const uint32_t yb0 = by * k.bands, z0 = bz * 8;
    const uint32_t ys = yb0 * 8, ye = min(ys + 8 * k.bands, a.y);  // the CTA's rows
    const uint32_t band = tid / k.q2, cq = tid - band * k.q2;
    const uint32_t col = c0 + 4 * cq, ybase = ys + band * 8;
    // rows of this thread's band that lie in the field (0: none, or past the window)
    const uint32_t nrow = band < k.bands && ybase < a.y && col < c1 ? min(8u, a.y - ybase) : 0u;
    // buffer words per plane (span) or per row
    const uint32_t rowwords = (kSpan ? k.pg : k.g) * kSlotWords;
    const uint32_t ntask    = kSpan ? 2 * k.pg : k.bands * 16 * k.g;
    // running sums along z, one 16-byte slot per thread and row of its band (after the row buffers)
    float4* zs = reinterpret_cast<float4*>(rb3 + (kSpan ? 2 : k.bands * 16) * rowwords) + tid;
#pragma unroll
    for (uint32_t yy = 0; yy < 8; ++yy) zs[yy * kT] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
    for (uint32_t pz = 0; pz < 8; pz += 2) {
        if (z0 + pz >= a.z) break;  // uniform across the CTA
        for (uint32_t t0 = 0; t0 < ntask; t0 += kT) {
            const uint32_t task = t0 + tid;
            uint32_t       r, j, zz, yv, len;
            if (kSpan) {
                r = task >= k.pg ? 1u : 0u, j = task - r * k.pg;
                zz = z0 + pz + r, yv = ys, len = (ye - ys) * a.x;
            } else {
                r = task / k.g, j = task - r * k.g;
                zz = z0 + pz + ((r >> 3) & 1u), yv = ys + (r >> 4) * 8 + (r & 7u), len = c1 - c0;
            }
            const uint32_t lin0 = (zz * a.y + yv) * a.x + c0, g = (lin0 >> 6) + j;
            const bool     valid = task < ntask && zz < a.z && yv < a.y && g <= ((lin0 + len - 1) >> 6);
            uint32_t       w[32];
            decode_deltas(a, g, valid, w);
            if (valid) rb_put_group<!kAl>(rb3 + r * rowwords, j, w);
        }
        __syncthreads();
        // both planes of the pass in one loop over the rows: two independent chains, and the sums
        // along z read and written once.  Threads without rows read the buffers' first codes, and
        // rows past the band's end repeat its last: neither is stored or reaches a thread or row
        // that is; a second plane past the slab's end is summed (nothing follows) and not stored
        const uint32_t  zz   = z0 + pz;
        const uint32_t  plane = a.x * a.y;
        const uint32_t  row0 = nrow ? (zz * a.y + ybase) * a.x + c0 : 0u;  // first code of the window
        const bool      two  = zz + 1 < a.z;
        float*          out  = a.out + row0 + 4 * cq;
        const uint32_t* rb   = rb3 + (kSpan ? 0u : (nrow ? band * 16 : 0u) * rowwords);
        const uint32_t* rc   = rb + (kSpan ? 1u : 8u) * rowwords;
        // span mode: from the planes' first slots
        const uint32_t f0 = (zz * a.y + ys) * a.x;
        uint32_t       i = kSpan ? row0 - (f0 & ~63u) : row0, k1 = kSpan ? row0 + plane - ((f0 + plane) & ~63u) : row0 + plane;
        if (!nrow) i = 0, k1 = 0;
        Pair s0{0.0f, 0.0f}, s1{0.0f, 0.0f}, t0{0.0f, 0.0f}, t1{0.0f, 0.0f};  // sums along y
#pragma unroll 8
        for (uint32_t yy = 0; yy < 8; ++yy) {
            uint32_t x01, x23, y01, y23;
            rb_read4<kAl>(rb, (kSpan ? i : i & 63u) + (nrow ? 4 * cq : 0u), x01, x23);
            rb_read4<kAl>(rc, (kSpan ? k1 : k1 & 63u) + (nrow ? 4 * cq : 0u), y01, y23);
            const float4 z4 = zs[yy * kT];
            Pair d0, d1, e0, e1;
            sums_x<2>(x01, x23, cq, d0, d1);
            sums_x<2>(y01, y23, cq, e0, e1);
            s0 = add2(s0, d0), s1 = add2(s1, d1);
            t0 = add2(t0, e0), t1 = add2(t1, e1);
            Pair q0 = add2(Pair{z4.x, z4.y}, s0), q1 = add2(Pair{z4.z, z4.w}, s1);
            store_row<kAl>(out, yy < nrow ? (int32_t)(c1 - col) : 0, q0, q1, a.ebx2);
            q0 = add2(q0, t0), q1 = add2(q1, t1);
            zs[yy * kT] = make_float4(q0.x, q0.y, q1.x, q1.y);
            store_row<kAl>(out + plane, two && yy < nrow ? (int32_t)(c1 - col) : 0, q0, q1, a.ebx2);
            if (yy + 1 < nrow) {
                i += a.x, k1 += a.x, out += a.x;
                if (!kSpan) rb += rowwords, rc += rowwords;
            }
        }
        __syncthreads();
    }
}

// Brick shape of the fused 3D path for a field of width x and height y, with t threads.  Span mode
// (whole rows) takes as many bands as keep both the compute threads (bands x q2) and the pass's
// decode tasks (2 pg) within the CTA's threads.
static Brick3 brick3(uint32_t x, uint32_t y, uint32_t t)
{
    Brick3 k{};
    k.t  = t;
    k.w  = std::min<uint32_t>(kW3, (x + 7) & ~7u);
    k.q2 = k.w / 4;
    k.g  = (k.w + 62) / 64 + 1;
    k.nwin = (uint32_t)cdiv(x, k.w);
    const uint32_t nbands = (uint32_t)cdiv(y, 8);
    k.span = k.nwin == 1;
    if (k.span) {
        k.bands = std::max(1u, std::min(t / k.q2, nbands));
        for (;;) {
            // a plane's span is at most 8 bands x rows of x codes, starting anywhere in a group;
            // rows' last quads read up to 3 codes past it.  x % 8 == 0: where bands start, a
            // group starts, in the first plane; planes of a multiple of 64 codes keep that
            const uint32_t n = 8 * k.bands * x;
            k.pg = x % 8 == 0 && (uint64_t)x * y % 64 == 0 ? (uint32_t)cdiv(n, 64) : (n + 66) / 64 + 1;
            if (k.bands == 1 || 2 * k.pg <= t) break;
            --k.bands;
        }
    } else {
        k.bands = std::max(1u, std::min({8u, t / k.q2, nbands}));
        while (k.bands > 1 && k.bands * 16 * k.g * kSlotWords * 4 > 48 * 1024) --k.bands;
    }
    k.nbgrp = (uint32_t)cdiv(nbands, k.bands);
    return k;
}

// 128 threads where they are used as well as 256 would be (within a tenth), since more and
// smaller CTAs decode and sum at different times: 500x500x100 on GB300 33.4 -> 31.3 us; 256
// where 128 leave a band's worth of threads idle (256x256x256 35.6 -> 31.0 us with 3 bands of 4).
static Brick3 brick3(uint32_t x, uint32_t y)
{
    const Brick3 big = brick3(x, y, 256);
    if (big.q2 > 128) return big;
    const Brick3 k = brick3(x, y, 128);
    return 2 * 10 * k.bands >= 9 * big.bands ? k : big;
}

// Dynamic shared memory of a k_decompress3d CTA: the row buffers (at most 48 KB) and the z sums
// (8 rows x 16 bytes per thread).
constexpr uint32_t kDecompress3dSmemMax = 48 * 1024 + 8 * 256 * 16;

static uint32_t brick3_smem(const Brick3& k)
{
    return (k.span ? 2 * k.pg : k.bands * 16 * k.g) * kSlotWords * 4 + 8 * k.t * 16;
}

using Decompress3d = void(const DecodeArgs, const Brick3);
template <uint32_t kT>
static Decompress3d* decompress3d(bool span, bool al)
{
    return span ? (al ? k_decompress3d<true, true, kT> : k_decompress3d<true, false, kT>)
                : (al ? k_decompress3d<false, true, kT> : k_decompress3d<false, false, kT>);
}

// Above 48 KB a kernel's dynamic shared memory needs an opt-in, which is per device.
static cudaError_t allow_decompress3d_smem()
{
    static std::atomic<uint64_t> done{0};  // bit d: opted in on device d
    int         dev = 0;
    cudaError_t e   = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    for (int v = 0; v < 8 && e == cudaSuccess; ++v) {
        Decompress3d* f = v & 4 ? decompress3d<128>(v & 1, v & 2) : decompress3d<256>(v & 1, v & 2);
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kDecompress3dSmemMax);
    }
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

// ------------------------------------------------------ fused 1D decode --
// One warp per shuffle block: lane g decodes its 64 codes (a quarter of one 256-element
// x_lorenzo block), prefix-sums them serially, adds the quad's carry, and writes 64
// floats through shared memory as coalesced 16-byte stores.  Codes at i%4 == 0 carry
// their sign; the others take it from the sidecar sign bits (or are non-negative).
//
// Bound by the latency of its one chain per warp (bitmap, chunks, sums, stores), so by the warps
// resident: 10 CTAs of 4 an SM, 48 registers and 4 KiB a warp.  GB300, event-timed, 2^25
// elements at 1e-3 / 1e-4: 46.7 / 51.7 us with 32-bit sums and 8 KiB a warp, 42.7 / 49.4 with the
// sums packed where they fit, 42.4 / 49.4, 38.7 / 45.1 and 37.0 / 43.4 with 6, 8 and 10 CTAs.
constexpr int kDecode1dWarps = 4;

// A warp's shared buffer of 32 words a lane: 16-byte chunk c (of 8) of lane l at position c ^ (l & 7),
// so that both the lanes' chunk stores and the output loops' loads (several lanes on one
// owner's chunks) spread over all 32 banks.
__device__ __forceinline__ uint32_t* chunk1d(uint32_t* sm, uint32_t l, uint32_t c) { return sm + 32 * l + 4 * (c ^ (l & 7u)); }

// Sums of the lane's deltas 32 h .. 32 h + 31 in 32 bits, from `acc` on; codes at i%4 == 0 carry
// their sign, the others take it from the sidecar word s.  kStore: each sum into the lane's
// words.  Only the run's first lim deltas count.
template <int h, bool kStore>
__device__ __forceinline__ uint32_t run1d(const uint32_t (&w)[32], uint32_t s, uint32_t lim, uint32_t lane, uint32_t acc,
                                          uint32_t* sm)
{
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int      j = 32 * h + i;
        const uint32_t c = (j & 1) ? (w[j >> 1] >> 16) : (w[j >> 1] & 0xFFFFu);
        const uint32_t d = (j & 3) == 0 ? sm_decode(c) : ((s >> i) & 1u ? 0u - c : c);
        acc += (uint32_t)j < lim ? d : 0u;
        q[i & 3] = acc;
        if (kStore && (i & 3) == 3) *reinterpret_cast<uint4*>(chunk1d(sm, lane, i >> 2)) = make_uint4(q[0], q[1], q[2], q[3]);
    }
    return acc;
}

// Bits 0, 2, 4 ... of v as the low 16 bits.
__device__ __forceinline__ uint32_t even_bits(uint32_t v)
{
    v &= 0x55555555u;
    v = (v | (v >> 1)) & 0x33333333u;
    v = (v | (v >> 2)) & 0x0F0F0F0Fu;
    v = (v | (v >> 4)) & 0x00FF00FFu;
    return (v | (v >> 8)) & 0xFFFFu;
}

// The packed path of k_decompress1d.  A lane's 64 deltas but the one that starts its tile (the
// tile's first value itself, which goes into the lane's base) are below 2^9: their running sums
// within the lane stay below 2^15, and two of them share a word.  w: the bit planes of the
// lane's codes (low codes in 0..15, high ones in 16..31); s0, s1: the sidecar's signs;
// base: the lane's first value's predecessor.  Leaves the sums plus 0x8000, two per word, in
// the lanes' words of `sm`; false, with nothing done, where a lane of the warp has a larger
// delta.
__device__ __forceinline__ bool sums1d_packed(uint32_t (&w)[32], uint32_t s0, uint32_t s1, uint32_t lane, uint32_t* sm,
                                              int32_t& base)
{
    const uint32_t first = (lane & 3u) == 0 ? 1u : 0u;  // low element 0 starts a tile
    // plane 15: the sign of low codes at even words (i % 4 == 0), a magnitude bit elsewhere
    const uint32_t big = ((w[9] | w[10] | w[11] | w[12] | w[13] | w[14] | (w[15] & 0xAAAAAAAAu)) & ~first) | w[25] | w[26] |
                         w[27] | w[28] | w[29] | w[30] | w[31];
    const uint32_t mid = ((w[7] | w[8]) & ~first) | w[23] | w[24];
    if (__any_sync(kFull, big != 0)) return false;
    uint32_t code = 0;  // the starting code
#pragma unroll
    for (int p = 15; p >= 0; --p) code = 2 * code + (w[p] & 1u);
    const int32_t start = first ? (int32_t)sm_decode(code) : 0;
    const uint32_t sl = ((w[15] & 0x55555555u) | ((even_bits(s0) | (even_bits(s1) << 16)) & 0xAAAAAAAAu)) & ~first;
    const uint32_t sh = even_bits(s0 >> 1) | (even_bits(s1 >> 1) << 16);
#pragma unroll
    for (int p = 0; p < 9; ++p) w[p] &= ~first;
    if (!__any_sync(kFull, mid != 0)) {  // below 2^7: as decode_deltas
        uint32_t t[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t s = h ? sh : sl;
            uint32_t       c = s;
#pragma unroll
            for (int p = 0; p < 7; ++p) {
                const uint32_t b = w[16 * h + p];
                t[h][p]          = b ^ s ^ c;
                c                = (b ^ s) & c;
            }
            t[h][7] = s ^ c;
            transpose8(t[h]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            w[i]      = delta_bytes<0>(t[0][i], t[1][i]) ^ 0x80000000u;
            w[8 + i]  = delta_bytes<1>(t[0][i], t[1][i]) ^ 0x80000000u;
            w[16 + i] = delta_bytes<2>(t[0][i], t[1][i]) ^ 0x80000000u;
            w[24 + i] = delta_bytes<3>(t[0][i], t[1][i]) ^ 0x80000000u;
        }
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t s = h ? sh : sl;
            uint32_t       c = s;
#pragma unroll
            for (int p = 0; p < 9; ++p) {
                const uint32_t b = w[16 * h + p];
                w[16 * h + p]    = b ^ s ^ c;
                c                = (b ^ s) & c;
            }
#pragma unroll
            for (int p = 9; p < 16; ++p) w[16 * h + p] = s ^ c;  // the sign extended
        }
        w[15] = ~w[15];
        transpose32<true>(w);
    }
    // w: deltas (d0 + 0x8000, d1) = d0 + 2^16 d1 + 0x8000 as an integer.  Times 2^16 + 1 that is
    // (d0, d0 + d1), both plus 0x8000; the sum so far goes in before.
    uint32_t h = 0x8000u;  // the sum so far plus 0x8000
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        w[j] = (w[j] + h - 0x8000u) * 65537u;
        h    = w[j] >> 16;
    }
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(chunk1d(sm, lane, c)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    const int32_t run = (int32_t)h - 0x8000;
    int32_t       v = run + start, u = __shfl_up_sync(kFull, v, 1);
    if (lane & 3u) v += u;
    u = __shfl_up_sync(kFull, v, 2);
    if ((lane & 3u) >= 2) v += u;
    base = v - run;
    return true;
}

__global__ void __launch_bounds__(kDecode1dWarps * 32, 10) k_decompress1d(const DecodeArgs a)
{
    pdl_wait();
    pdl_trigger();
    __shared__ __align__(16) uint32_t smem[kDecode1dWarps][kBlockWords];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t t    = blockIdx.x * kDecode1dWarps + wid;
    const uint32_t ntiles = a.nb + (a.tail ? 1u : 0u);
    if (t >= ntiles) return;  // warp-uniform
    uint32_t*       sm = smem[wid];
    uint32_t        w[32];
    const uint32_t  e0 = t * kBlockCodes + lane * 64;
    const uint32_t* sb = (a.mode == 1) ? reinterpret_cast<const uint32_t*>(a.st + a.off_sign) : nullptr;
    uint32_t        s0 = 0, s1 = 0;
    if (sb && e0 < a.n) {
        s0 = __ldg(sb + (e0 >> 5));
        s1 = (e0 + 32 < a.n) ? __ldg(sb + (e0 >> 5) + 1) : 0u;
    }
    if (t < a.nb) {
        gather_block(a, t, lane, sm);
        __syncwarp();
#pragma unroll
        for (uint32_t p = 0; p < 32; ++p) w[p] = sm[p * 32 + lane];
        __syncwarp();
        int32_t base;
        if ((t + 1) * kBlockCodes <= a.nl && sums1d_packed(w, s0, s1, lane, sm, base)) {
            // value = base + sum: each sum under the exponent of 2^23, less 2^23 + 2^15
            const float c = (float)base - 8421376.0f;
            __syncwarp();
            float* out = a.out + (size_t)t * kBlockCodes + lane * 4;
#pragma unroll 4
            for (uint32_t i = 0; i < 16; ++i) {  // elements 128 i + 4 lane .. + 3: of lane `ow`
                const uint32_t ow = 2 * i + (lane >> 4);
                const float    co = __shfl_sync(kFull, c, ow);
                const uint2    x  = *reinterpret_cast<const uint2*>(chunk1d(sm, ow, (lane & 15u) >> 1) + 2 * (lane & 1u));
                const Pair     f{__uint_as_float(__byte_perm(x.x, 0x4B000000u, 0x7410)), __uint_as_float(__byte_perm(x.x, 0x4B000000u, 0x7432))};
                const Pair     g{__uint_as_float(__byte_perm(x.y, 0x4B000000u, 0x7410)), __uint_as_float(__byte_perm(x.y, 0x4B000000u, 0x7432))};
                store_row<true>(out + 128 * i, 4, add2(f, Pair{co, co}), add2(g, Pair{co, co}), a.ebx2);
            }
            return;
        }
        transpose32<true>(w);
    } else {
        decode_group(a, t * 32 + lane, w);  // tail: sidecar codes
    }
    // elements of this lane's run inside x*y*z (all 64 except in the last block)
    const uint32_t lim  = a.nl > e0 ? a.nl - e0 : 0u;
    const uint32_t half = run1d<0, true>(w, s0, lim, lane, 0u, sm);
    const uint32_t acc  = run1d<1, false>(w, s1, lim, lane, half, sm);
    // carry across the 4 lanes of each 256-element block
    uint32_t v = acc, u = __shfl_up_sync(kFull, v, 1);
    if (lane & 3u) v += u;
    u = __shfl_up_sync(kFull, v, 2);
    if ((lane & 3u) >= 2) v += u;
    const uint32_t ex = v - acc;
    // write, half a run at a time: pass i covers 32 elements of the runs of lanes 4 i .. 4 i + 3
#pragma unroll 1
    for (uint32_t h = 0; h < 2; ++h) {
        __syncwarp();
        if (h) {
            run1d<1, true>(w, s1, lim, lane, half, sm);
            __syncwarp();
        }
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t ow  = 4 * i + (lane >> 3);
            const uint32_t exo = __shfl_sync(kFull, ex, ow);
            const uint4    pv  = *reinterpret_cast<const uint4*>(chunk1d(sm, ow, lane & 7u));
            const float    f[4] = {(float)(int32_t)(pv.x + exo) * a.ebx2, (float)(int32_t)(pv.y + exo) * a.ebx2,
                                   (float)(int32_t)(pv.z + exo) * a.ebx2, (float)(int32_t)(pv.w + exo) * a.ebx2};
            const uint32_t e = t * kBlockCodes + 64 * ow + 32 * h + 4 * (lane & 7u);
            if (e + 3 < a.nl) {
                __stcs(reinterpret_cast<float4*>(a.out + e), make_float4(f[0], f[1], f[2], f[3]));
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (e + k < a.nl) a.out[e + k] = f[k];
            }
        }
    }
}

cudaError_t launch_decompress_fused(const DecodeArgs& a, cudaStream_t s)
{
    const int nd = (a.z == 1 && a.y == 1) ? 1 : (a.z == 1 ? 2 : 3);
    if (nd == 2) {
        const uint32_t nwin = (uint32_t)cdiv(a.x, kW2);
        const uint32_t ctas = (uint32_t)(nwin * cdiv(a.y, 16));
        if (a.x % 4 == 0) return launch_pdl(k_decompress2d<true>, dim3(ctas), dim3(kT2), 0, s, a, nwin);
        return launch_pdl(k_decompress2d<false>, dim3(ctas), dim3(kT2), 0, s, a, nwin);
    }
    if (nd == 3) {
        const cudaError_t e = allow_decompress3d_smem();
        if (e != cudaSuccess) return e;
        const Brick3   k    = brick3(a.x, a.y);
        if (brick3_smem(k) > kDecompress3dSmemMax) return cudaErrorInvalidConfiguration;
        const uint64_t ctas = (uint64_t)k.nwin * k.nbgrp * cdiv(a.z, 8);
        Decompress3d*  f    = k.t == 128 ? decompress3d<128>(k.span != 0, a.x % 4 == 0)
                                        : decompress3d<256>(k.span != 0, a.x % 4 == 0);
        return launch_pdl(f, dim3((uint32_t)ctas), dim3(k.t), brick3_smem(k), s, a, k);
    }
    const uint32_t ntiles = a.nb + (a.tail ? 1u : 0u);
    return launch_pdl(k_decompress1d, dim3((uint32_t)cdiv(ntiles, kDecode1dWarps)), dim3(kDecode1dWarps * 32), 0, s,
                      a);
}

// ------------------------------------------------------------- recon --
// 2D: a CTA covers 16 rows x 512 columns; lane owns 4 consecutive columns, lanes 4k..4k+3
// one 16-column tile row.  Row prefix: serial over 4 + quad shuffle scan; column prefix:
// running sum over the 16 rows.  Bound by latency: 8 rows' codes are loaded at a time (one
// row at a time, 3600x1800 on GB300: 11.2 -> 8.1 us).
__global__ void __launch_bounds__(128) k_recon2d(const ReconArgs a, uint32_t nwin)
{
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t c0   = (blockIdx.x % nwin) * 512 + wid * 128 + lane * 4;
    const uint32_t r0   = (blockIdx.x / nwin) * 16;
    const uint32_t q    = lane & 3u, nrows = min(16u, a.y - r0);
    const bool     vec  = (a.x % 4 == 0) && (c0 + 3 < a.x);
    const size_t   base = (size_t)r0 * a.x + c0;
    uint32_t       acc[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (uint32_t h = 0; h < nrows; h += 8) {
        uint2 w[8];  // 4 codes of each row
#pragma unroll
        for (uint32_t rr = 0; rr < 8; ++rr) {
            w[rr] = make_uint2(0, 0);
            if (h + rr >= nrows) continue;  // uniform across the CTA
            const uint16_t* src = a.codes + base + (size_t)(h + rr) * a.x;
            if (vec) {
                w[rr] = __ldg(reinterpret_cast<const uint2*>(src));
            } else {
                if (c0 < a.x) w[rr].x = src[0];
                if (c0 + 1 < a.x) w[rr].x |= (uint32_t)src[1] << 16;
                if (c0 + 2 < a.x) w[rr].y = src[2];
                if (c0 + 3 < a.x) w[rr].y |= (uint32_t)src[3] << 16;
            }
        }
#pragma unroll
        for (uint32_t rr = 0; rr < 8; ++rr) {
            if (h + rr >= nrows) break;  // uniform across the CTA
            uint32_t d[4];
            sm_decode2(w[rr].x, d[0], d[1]);
            sm_decode2(w[rr].y, d[2], d[3]);
            d[1] += d[0], d[2] += d[1], d[3] += d[2];
            uint32_t v = d[3];
            uint32_t u = __shfl_up_sync(kFull, v, 1);
            if (q >= 1) v += u;
            u = __shfl_up_sync(kFull, v, 2);
            if (q >= 2) v += u;
            const uint32_t ex = v - d[3];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] += d[j] + ex;
            float* dst = a.out + base + (size_t)(h + rr) * a.x;
            if (vec) {
                *reinterpret_cast<float4*>(dst) =
                    make_float4((float)(int32_t)acc[0] * a.ebx2, (float)(int32_t)acc[1] * a.ebx2,
                                (float)(int32_t)acc[2] * a.ebx2, (float)(int32_t)acc[3] * a.ebx2);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c0 + j < a.x) dst[j] = (float)(int32_t)acc[j] * a.ebx2;
            }
        }
    }
}

// 3D: a warp covers 128 columns of one 8x8 (y, z) tile column; lane owns 4 columns, lane
// pairs one 8-column tile row.  zacc[y] keeps the running z-sum of each of the 8 rows.
// The flat block index runs over x windows, then groups of 4 bands, then z slabs.
__global__ void __launch_bounds__(128) k_recon3d(const ReconArgs a, uint32_t nwin, uint32_t nyg)
{
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t rest = blockIdx.x / nwin;
    const uint32_t c0   = (blockIdx.x % nwin) * 128 + lane * 4;
    const uint32_t y0   = ((rest % nyg) * 4 + wid) * 8;
    const uint32_t z0   = (rest / nyg) * 8;
    if (y0 >= a.y) return;  // warp-uniform
    const bool     vec = (a.x % 4 == 0) && (c0 + 3 < a.x);
    const size_t   xy  = (size_t)a.x * a.y;
    uint32_t       zacc[8][4];
#pragma unroll
    for (int yy = 0; yy < 8; ++yy) zacc[yy][0] = zacc[yy][1] = zacc[yy][2] = zacc[yy][3] = 0;
    for (uint32_t zz = 0; zz < 8; ++zz) {
        if (z0 + zz >= a.z) break;
        uint32_t colacc[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t yy = 0; yy < 8; ++yy) {
            const bool   live = y0 + yy < a.y;
            const size_t base = (size_t)(z0 + zz) * xy + (size_t)(y0 + yy) * a.x + c0;
            uint32_t     d[4] = {0, 0, 0, 0};
            if (live) {
                if (vec) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(a.codes + base));
                    sm_decode2(v.x, d[0], d[1]);
                    sm_decode2(v.y, d[2], d[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (c0 + j < a.x) d[j] = sm_decode(a.codes[base + j]);
                }
            }
            d[1] += d[0], d[2] += d[1], d[3] += d[2];
            const uint32_t u = __shfl_up_sync(kFull, d[3], 1);
            const uint32_t ex = (lane & 1u) ? u : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                colacc[j] += d[j] + ex;
                zacc[yy][j] += colacc[j];
            }
            if (!live) continue;
            if (vec) {
                *reinterpret_cast<float4*>(a.out + base) = make_float4(
                    (float)(int32_t)zacc[yy][0] * a.ebx2, (float)(int32_t)zacc[yy][1] * a.ebx2,
                    (float)(int32_t)zacc[yy][2] * a.ebx2, (float)(int32_t)zacc[yy][3] * a.ebx2);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c0 + j < a.x) a.out[base + j] = (float)(int32_t)zacc[yy][j] * a.ebx2;
            }
        }
    }
}

// 1D: one warp per 256-element block; lane owns 8 consecutive elements.  Codes at
// i%4 == 0 carry their sign in bit 15; the others take it from the sidecar sign bits
// (or the stage API's signum bytes), and are non-negative without either.
__global__ void __launch_bounds__(256) k_recon1d(const ReconArgs a)
{
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t blk  = blockIdx.x * 8 + wid;
    const uint32_t e0   = blk * 256 + lane * 8;
    if (blk * 256 >= a.nl) return;  // warp-uniform
    uint32_t c[8];
    if (e0 + 7 < a.nl) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.codes + e0));
        c[0] = v.x & 0xFFFFu, c[1] = v.x >> 16, c[2] = v.y & 0xFFFFu, c[3] = v.y >> 16;
        c[4] = v.z & 0xFFFFu, c[5] = v.z >> 16, c[6] = v.w & 0xFFFFu, c[7] = v.w >> 16;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = e0 + j < a.nl ? a.codes[e0 + j] : 0u;
    }
    uint32_t sb = 0;  // sign bits of the 8 elements
    if (a.signbits) {
        sb = (__ldg(a.signbits + (e0 >> 5)) >> (e0 & 31u)) & 0xFFu;
    } else if (a.signum) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sb |= (e0 + j < a.nl && a.signum[e0 + j]) ? (1u << j) : 0u;
    }
    uint32_t d[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if ((j & 3) == 0) {
            d[j] = sm_decode(c[j]);
        } else {
            d[j] = ((sb >> j) & 1u) ? 0u - c[j] : c[j];
        }
        if (j) d[j] += d[j - 1];
    }
    uint32_t v = d[7];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, v, o);
        if (lane >= (uint32_t)o) v += u;
    }
    const uint32_t ex = v - d[7];
    float          f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = (float)(int32_t)(d[j] + ex) * a.ebx2;
    if (e0 + 7 < a.nl) {
        float4* o = reinterpret_cast<float4*>(a.out + e0);
        o[0]      = make_float4(f[0], f[1], f[2], f[3]);
        o[1]      = make_float4(f[4], f[5], f[6], f[7]);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (e0 + j < a.nl) a.out[e0 + j] = f[j];
    }
}

// elements past x*y*z (fz.cu:117-118 lets the file be longer than the dims) decode to 0
__global__ void k_zero_tail(float* out, uint32_t from, uint32_t n)
{
    for (uint32_t i = from + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = 0.0f;
}

cudaError_t launch_zero_tail(float* out, uint32_t from, uint32_t n, cudaStream_t s)
{
    k_zero_tail<<<(uint32_t)std::min<uint64_t>(cdiv(n - from, 256), 1024), 256, 0, s>>>(out, from, n);
    return cudaGetLastError();
}

cudaError_t launch_reconstruct(const ReconArgs& a, cudaStream_t s)
{
    const int nd = (a.z == 1 && a.y == 1) ? 1 : (a.z == 1 ? 2 : 3);
    if (nd == 1) {
        k_recon1d<<<(uint32_t)cdiv(cdiv(a.nl, 256), 8), 256, 0, s>>>(a);
    } else if (nd == 2) {
        const uint32_t nwin = (uint32_t)cdiv(a.x, 512);
        k_recon2d<<<(uint32_t)(nwin * cdiv(a.y, 16)), 128, 0, s>>>(a, nwin);
    } else {
        const uint32_t nwin = (uint32_t)cdiv(a.x, 128), nyg = (uint32_t)cdiv(cdiv(a.y, 8), 4);
        k_recon3d<<<(uint32_t)((uint64_t)nwin * nyg * cdiv(a.z, 8)), 128, 0, s>>>(a, nwin, nyg);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && a.n > a.nl) {
        k_zero_tail<<<(uint32_t)std::min<uint64_t>(cdiv(a.n - a.nl, 256), 1024), 256, 0, s>>>(a.out, a.nl, a.n);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace fz
