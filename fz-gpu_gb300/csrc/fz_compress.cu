// fz_compress.cu -- launches of the compression kernels (fz_compress.cuh) and the stage-level kernels.
#include <algorithm>
#include <atomic>

#include "fz_compress.cuh"

namespace fz {

// --------------------------------------------------------------- range --
constexpr int kRangeUnroll = 8;
// max and min of the field (fz.cu:137) as order-preserving integers folded with one
// atomicMin/atomicMax per CTA into mm[0..1], which the consuming compress kernel resets
// to "empty" for the next call.  Each thread issues kRangeUnroll 16-byte loads at once
// (coalesced across the CTA); the grid covers the field in one batch per thread, so the
// block scheduler keeps every SM streaming until the last CTAs.  NaN/Inf raise
// kStatusNonfinite: the running min and max propagate NaN (min.NaN / max.NaN), so one
// test of each thread's final pair finds any NaN, -Inf or +Inf it has seen; the bit also
// goes to `callw` (a per-call word the header writer reads and resets), when given.
__global__ void __launch_bounds__(256) k_range(const float* __restrict__ in, uint32_t n, uint32_t* mm,
                                               uint32_t* status, uint32_t* callw)
{
    __shared__ uint32_t smn[8], smx[8], snf[8];
    float          mn = INFINITY, mx = -INFINITY;
    uint32_t       nonfinite = 0;
    const uint32_t n4        = n / 4;
    const uint32_t per       = blockDim.x * kRangeUnroll;
    for (uint32_t b = blockIdx.x * per + threadIdx.x; b < n4; b += gridDim.x * per) {
        float4 v[kRangeUnroll];
#pragma unroll
        for (int k = 0; k < kRangeUnroll; ++k)
            if (b + k * blockDim.x < n4) v[k] = ldg4(in + 4 * (size_t)(b + k * blockDim.x));
#pragma unroll
        for (int k = 0; k < kRangeUnroll; ++k) {
            if (b + k * blockDim.x >= n4) continue;
            mn = fmin_nan(fmin_nan(mn, v[k].x), fmin_nan(v[k].y, fmin_nan(v[k].z, v[k].w)));
            mx = fmax_nan(fmax_nan(mx, v[k].x), fmax_nan(v[k].y, fmax_nan(v[k].z, v[k].w)));
        }
    }
    // NaN leaves both NaN; -Inf shows in the min, +Inf in the max (the start values
    // +Inf / -Inf of a thread without elements stay on the other side)
    nonfinite = (mn != mn) | (mn == -INFINITY) | (mx == INFINITY);
    if (blockIdx.x == 0 && threadIdx.x < n - 4 * n4) {
        const float v = in[4 * n4 + threadIdx.x];
        mn = fminf(mn, v), mx = fmaxf(mx, v);
        nonfinite |= !isfinite(v);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    nonfinite = __reduce_or_sync(kFull, nonfinite);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) smn[w] = f2ord(mn), smx[w] = f2ord(mx), snf[w] = nonfinite;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t nw = blockDim.x >> 5;
        const uint32_t a  = __reduce_min_sync(kFull, lane < nw ? smn[lane] : 0xFFFFFFFFu);
        const uint32_t c  = __reduce_max_sync(kFull, lane < nw ? smx[lane] : 0u);
        const uint32_t f  = __reduce_or_sync(kFull, lane < nw ? snf[lane] : 0u);
        if (lane == 0) {
            atomicMin(mm, a);
            atomicMax(mm + 1, c);
            if (f) {
                atomicOr(status, kStatusNonfinite);
                if (callw) atomicOr(callw, kStatusNonfinite);
            }
        }
    }
}

void field_items(uint32_t n, uint32_t nb, uint32_t ntiles, bool rel, uint32_t& nr, uint32_t& ne, uint32_t& nc)
{
    nr = rel ? (uint32_t)std::max<uint64_t>(1, cdiv(n, kRangeItemElems)) : 0u;
    ne = (uint32_t)cdiv(ntiles, kCompressWarps);
    nc = (uint32_t)cdiv(nb, kCompactBlocks);  // none without full blocks (the encode launch writes the header)
}

// One warp looks back from tile 1 at tile 0, which nothing publishes in this epoch: the
// bounded wait must give up and raise kStatusTimeout (fz_selftest_wait_timeout).
__global__ void k_wait_selftest(const uint64_t* state, const uint32_t* epoch, uint32_t* status)
{
    // the current device epoch has not been used by any launch yet
    const uint32_t e    = __ldcg(epoch);
    uint32_t       excl = 0, ovf = 0;
    lookback(state, 1, e, status, excl, ovf);
}

cudaError_t launch_wait_selftest(const uint64_t* state, const uint32_t* epoch, uint32_t* status, cudaStream_t s)
{
    k_wait_selftest<<<1, 32, 0, s>>>(state, epoch, status);
    return cudaGetLastError();
}

// Resident CTAs of a kernel on the current device (SM count x CTAs per SM), after the
// device's opt-in to more than 48 KiB of dynamic shared memory where the kernel needs it;
// 0 when a query fails.
template <typename K>
static uint32_t resident_ctas(K kernel, int threads, int dyn_smem = 0)
{
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    // the opt-in is needed once static + dynamic shared memory passes 48 KiB; made for any
    // dynamic size (it only raises the kernel's limit)
    if (dyn_smem > 0 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_smem) != cudaSuccess)
        return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dyn_smem) != cudaSuccess) return 0;
    return (uint32_t)std::max(1, sms * std::max(per_sm, 1));
}

cudaError_t launch_range(const float* in, uint32_t n, uint32_t* mm, uint32_t* status, uint32_t* callw,
                         cudaStream_t s)
{
    const uint64_t want = cdiv(n / 4, 256ull * kRangeUnroll);  // n < 2^31: at most 2^18 CTAs
    const uint32_t ctas = (uint32_t)std::max<uint64_t>(1, want);
    k_range<<<ctas, 256, 0, s>>>(in, n, mm, status, callw);
    return cudaGetLastError();
}

static EncodeKernel* encode_kernel(int nd, bool list, bool rel)
{
    return rel ? pick_encode_kernel<true>(nd, list) : encode_kernel_abs(nd, list);
}
static WholeKernel* whole_kernel(int nd, bool scan, bool rel)
{
    return rel ? pick_whole_kernel<true>(nd, scan) : whole_kernel_abs(nd, scan);
}
static uint32_t encode_smem(int nd) { return nd == 1 ? encode_smem<1>() : nd == 2 ? encode_smem<2>() : encode_smem<3>(); }

// Resident CTAs of each list-compression kernel on the current device, cached per device
// (ordinals below 64): [0] range, [1..3] encode<1..3>, [4] compaction.
static uint32_t list_wave(int which, bool list, bool rel)
{
    static std::atomic<uint32_t> cache[64][2][2][5];
    int                          dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<uint32_t>* slot = (dev >= 0 && dev < 64) ? &cache[dev][rel][list][which] : nullptr;
    uint32_t               w    = slot ? slot->load(std::memory_order_acquire) : 0u;
    if (w) return w;
    constexpr int T = kCompressWarps * 32;
    // resident_ctas also opts the encode kernels in to their dynamic shared memory
    w = which == 0 ? resident_ctas(list ? k_range_fields<true> : k_range_fields<false>, T)
        : which == 4 ? resident_ctas(list ? k_compact_fields<true> : k_compact_fields<false>, T)
                     : resident_ctas(encode_kernel(which, list, rel), T, encode_smem(which));
    if (slot) slot->store(w, std::memory_order_release);
    return w;
}

cudaError_t launch_fields(FieldPhase phase, int nd, bool rel, const FieldJob* jobs, const Segment* segs, uint32_t nseg,
                          uint32_t total, const FieldJob& one, cudaStream_t s, uint32_t min_ctas)
{
    if (!total) return cudaSuccess;
    const bool list = jobs != nullptr;
    if (list && (!segs || !nseg)) return cudaErrorInvalidValue;
    const int      which = phase == FieldPhase::Range ? 0 : phase == FieldPhase::Encode ? nd : 4;
    const uint32_t wave  = list_wave(which, list, rel);
    if (!wave) return cudaErrorInvalidDevice;
    const dim3 grid(std::min(std::max(total, min_ctas), wave)), block(kCompressWarps * 32);
    // eager launches with programmatic stream serialization: each kernel's CTAs may start
    // as the previous kernel of the call (or of the previous call on the stream) retires
    if (phase == FieldPhase::Range) {
        if (list) return launch_pdl(k_range_fields<true>, grid, block, 0, s, jobs, segs, nseg, total, one);
        return launch_pdl(k_range_fields<false>, grid, block, 0, s, jobs, segs, nseg, total, one);
    }
    if (phase == FieldPhase::Compact) {
        if (list) return launch_pdl(k_compact_fields<true>, grid, block, 0, s, jobs, segs, nseg, total, one);
        return launch_pdl(k_compact_fields<false>, grid, block, 0, s, jobs, segs, nseg, total, one);
    }
    return launch_pdl(encode_kernel(nd, list, rel), grid, block, encode_smem(nd), s, jobs, segs, nseg, total, one);
}

// `query` on the current device, kept per device once it is not 0 (an error).
template <typename Q>
static uint32_t per_device(std::atomic<uint32_t> (&known)[64], Q query)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<uint32_t>* slot = dev < 64 ? &known[dev] : nullptr;
    uint32_t               v    = slot ? slot->load(std::memory_order_acquire) : 0;
    if (v) return v;
    v = query();
    if (slot) slot->store(v, std::memory_order_release);
    return v;
}

// CTAs of one resident wave of the one-launch kernel after a range launch on the current device (0:
// error), opted in to its dynamic shared memory.
static uint32_t whole_wave(int nd, bool rel)
{
    static std::atomic<uint32_t> waves[2][3][64];
    return per_device(waves[rel][nd - 1], [=] { return resident_ctas(whole_kernel(nd, true, rel), kCompressWarps * 32, encode_smem(nd)); });
}

// The largest cluster of the one-launch kernel, at most kSmallItems CTAs, that the current device can
// place (0: error), opted in to its dynamic shared memory and to clusters past 8 CTAs.
uint32_t small_items(int nd, bool rel)
{
    static std::atomic<uint32_t> sizes[2][3][64];
    return per_device(sizes[rel][nd - 1], [=] {
        WholeKernel* const k = whole_kernel(nd, false, rel);
        if (!resident_ctas(k, kCompressWarps * 32, encode_smem(nd))) return 0u;
        const bool wide = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        for (uint32_t c = wide ? kSmallItems : std::min(8u, kSmallItems); c > 1; --c) {
            cudaLaunchAttribute at{};
            at.id             = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim = {c, 1, 1};
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(c), cfg.blockDim = dim3(kCompressWarps * 32), cfg.dynamicSmemBytes = encode_smem(nd);
            cfg.attrs = &at, cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0) return c;
            (void)cudaGetLastError();  // a size that is refused leaves no error behind
        }
        return 1u;
    });
}

bool whole_field_fits(int nd, bool rel, uint32_t ne, bool waits)
{
    const uint32_t wave = whole_wave(nd, rel);
    return ne <= std::min(waits ? wave : wave / 2, 0xFFFFu);  // (wait_word counts in 16 bits)
}

cudaError_t launch_whole_field(int nd, const FieldJob& J, cudaStream_t s)
{
    const bool scan = J.ne > small_items(nd, J.rel != 0);
    return launch_pdl_cluster(whole_kernel(nd, scan, J.rel != 0), dim3(J.ne), dim3(kCompressWarps * 32), encode_smem(nd), s,
                              scan ? 1u : J.ne, J);
}

// One resident wave of k_compress<ND> on the current device.  The 64 KiB of dynamic shared
// memory needs a per-device opt-in, and the wave depends on the device's SM count, so
// both are done and cached per device (device ordinals below 64; others are computed on
// every call).
static uint32_t compress_wave(int nd)
{
    constexpr int                       kSmem = 2 * kCompressWarps * kBlockWords * 4;  // two tile buffers
    static std::atomic<uint32_t>        cache[64][3];
    int                                 dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<uint32_t>* slot = (dev >= 0 && dev < 64) ? &cache[dev][nd - 1] : nullptr;
    uint32_t               w    = slot ? slot->load(std::memory_order_acquire) : 0u;
    if (w) return w;
    w = nd == 1 ? resident_ctas(k_compress<1>, kCompressWarps * 32, kSmem)
        : nd == 2 ? resident_ctas(k_compress<2>, kCompressWarps * 32, kSmem)
                  : resident_ctas(k_compress<3>, kCompressWarps * 32, kSmem);
    if (slot) slot->store(w, std::memory_order_release);
    return w;
}

cudaError_t launch_compress(const CompressArgs& a, cudaStream_t s)
{
    // persistent: min(tiles, one resident wave) CTAs; a tile is 8 shuffle blocks
    constexpr int  kSmem = 2 * kCompressWarps * kBlockWords * 4;  // two tile buffers
    const uint32_t wave  = compress_wave((int)a.ndim);
    if (!wave) return cudaErrorInvalidDevice;
    const uint32_t nct  = (uint32_t)cdiv(a.ntiles, kCompressWarps);
    const uint32_t ctas = std::min(nct, wave);
    switch (a.ndim) {
    case 1: k_compress<1><<<ctas, kCompressWarps * 32, kSmem, s>>>(a); break;
    case 2: k_compress<2><<<ctas, kCompressWarps * 32, kSmem, s>>>(a); break;
    default: k_compress<3><<<ctas, kCompressWarps * 32, kSmem, s>>>(a); break;
    }
    return cudaGetLastError();
}

// =================================================== stage-level kernels ==
// fz_lorenzo_construct: codes of [0, x*y*z) into a u16 array (launch_construct_
// LorenzoI_var, lorenzo_var.cuh:520-597).  One warp per 128 consecutive elements.
template <int ND>
__global__ void __launch_bounds__(256) k_lorenzo_codes(const float* __restrict__ in, uint16_t* q,
                                                       uint8_t* signum, Geo g, float r)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t e0   = warp * 128 + lane * 4;
    if (warp * 128 >= g.nl) return;  // warp-uniform
    uint32_t c[4], ovf = 0, sgn = 0;
    codes4<ND>(in, g, e0, r, lane, c, ovf, sgn);
    if (e0 + 3 < g.nl) {
        *reinterpret_cast<uint2*>(q + e0) = make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e0 + j < g.nl) q[e0 + j] = (uint16_t)c[j];
    }
    if (ND == 1 && signum) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e0 + j < g.nl) signum[e0 + j] = (sgn >> j) & 1u;
    }
}

cudaError_t launch_lorenzo_construct(const float* in, uint16_t* q, uint8_t* signum, uint32_t x,
                                     uint32_t y, uint32_t z, float ebx2_r, cudaStream_t s)
{
    Geo g;
    g.x = x, g.y = y, g.xy = x * y, g.nl = x * y * z, g.lim = g.nl;
    g.dx = make_fastdiv(x), g.dxy = make_fastdiv(g.xy);
    g.al_x = (x % 4) == 0, g.al_xy = (g.xy % 4) == 0, g.al_xyx = ((g.xy + x) % 4) == 0;
    const int      nd    = (z == 1 && y == 1) ? 1 : (z == 1 ? 2 : 3);
    const uint32_t warps = (uint32_t)cdiv(g.nl, 128);
    const uint32_t ctas  = (uint32_t)cdiv(warps, 8);
    if (nd == 1) k_lorenzo_codes<1><<<ctas, 256, 0, s>>>(in, q, signum, g, ebx2_r);
    else if (nd == 2) k_lorenzo_codes<2><<<ctas, 256, 0, s>>>(in, q, signum, g, ebx2_r);
    else k_lorenzo_codes<3><<<ctas, 256, 0, s>>>(in, q, signum, g, ebx2_r);
    return cudaGetLastError();
}

// fz_bitshuffle_flag: bitshuffleAndBitflag over floor(n/2048) blocks (fz.cu:61-111)
// plus the raw tail copy (fz.cu:155) and zeroed flags past the last full block.
__global__ void __launch_bounds__(256) k_bitshuffle(const uint32_t* __restrict__ in, uint32_t* out,
                                                    uint32_t n_codes, uint32_t* bitflag,
                                                    uint32_t* byteflag)
{
    __shared__ __align__(16) uint32_t smem[8][kBlockWords];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t t    = blockIdx.x * 8 + wid;
    const uint32_t nb   = n_codes / kBlockCodes;
    const uint32_t nw   = (uint32_t)cdiv(n_codes, 256);
    uint32_t*      sm   = smem[wid];
    if (t < nb) {
        const uint4* src = reinterpret_cast<const uint4*>(in + (size_t)t * kBlockWords);
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t q = lane + 32 * i;
            *reinterpret_cast<uint4*>(sm + swz(q)) = src[q];
        }
        __syncwarp();
        uint32_t w[32];
#pragma unroll
        for (uint32_t tt = 0; tt < 8; ++tt) {
            const uint4 v = *reinterpret_cast<const uint4*>(sm + swz(lane * 8 + tt));
            w[4 * tt] = v.x, w[4 * tt + 1] = v.y, w[4 * tt + 2] = v.z, w[4 * tt + 3] = v.w;
        }
        transpose32(w);
        __syncwarp();
#pragma unroll
        for (uint32_t p = 0; p < 32; ++p) sm[p * 32 + lane] = w[p];
        __syncwarp();
        uint4* dst = reinterpret_cast<uint4*>(out + (size_t)t * kBlockWords);
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint4 v = *reinterpret_cast<const uint4*>(sm + (lane + 32 * i) * 4);
            dst[lane + 32 * i] = v;
            const bool f = (v.x | v.y | v.z | v.w) != 0;
            byteflag[(size_t)t * kChunks + lane + 32 * i] = f;
            const uint32_t b = __ballot_sync(kFull, f);
            if (lane == 0) bitflag[(size_t)t * 8 + i] = b;
        }
        return;
    }
    if (t == nb) {
        // tail: raw copy of the remaining bytes (2n total) and zero flags
        const uint8_t* s8 = reinterpret_cast<const uint8_t*>(in);
        uint8_t*       d8 = reinterpret_cast<uint8_t*>(out);
        for (uint64_t b = (uint64_t)nb * 4096 + lane; b < 2ull * n_codes; b += 32) d8[b] = s8[b];
        for (uint32_t i = nb * 8 + lane; i < nw; i += 32) bitflag[i] = 0;
        for (uint32_t i = nb * kChunks + lane; i < 32 * nw; i += 32) byteflag[i] = 0;
    }
}

cudaError_t launch_bitshuffle_flag(const uint32_t* in, uint32_t* out, uint32_t n_codes,
                                   uint32_t* bitflag, uint32_t* byteflag, cudaStream_t s)
{
    const uint32_t tiles = n_codes / kBlockCodes + 1;
    k_bitshuffle<<<(uint32_t)cdiv(tiles, 8), 256, 0, s>>>(in, out, n_codes, bitflag, byteflag);
    return cudaGetLastError();
}

// fz_scan_encode: exclusive scan of M u32 flags (cub::DeviceScan::ExclusiveSum,
// fz.cu:187-192) + total (fz.cu:194-201) + compaction (encodeDebug, fz.cu:49-59).
// One warp per 256 flags, 8 warps to a tile, one decoupled look-back per tile.  Bound by its
// round trips (flags, look-back, chunks).  A look-back per warp chained 8 times as many tiles:
// 3600x1800 codes on GB300 29.6 -> 16 us.
__global__ void __launch_bounds__(256) k_scan_encode(const uint8_t* __restrict__ shuffled,
                                                     const uint32_t* __restrict__ flags,
                                                     uint32_t n_codes, uint32_t m,
                                                     uint32_t* presum, uint8_t* out,
                                                     uint64_t* state, uint32_t* ticket,
                                                     uint32_t* status, uint32_t* total,
                                                     uint32_t* epoch_word)
{
    __shared__ uint32_t cta_tile, s_epoch, s_cnt[8], s_pre[8];
    const uint32_t      lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_epoch = __ldcg(epoch_word);
        __threadfence();
        cta_tile = take_ticket(ticket, epoch_word, gridDim.x).tile;
    }
    __syncthreads();
    const uint32_t epoch = s_epoch, tile = cta_tile;
    const uint32_t t     = tile * 8 + wid;  // the warp's 256 flags
    const uint32_t ntl   = (m + 255) / 256;
    uint32_t       bm[8], cnt = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t idx = t * 256 + 32 * i + lane;  // (m < 2^29)
        bm[i] = __ballot_sync(kFull, idx < m && flags[idx] != 0);
        cnt += __popc(bm[i]);
    }
    if (lane == 0) s_cnt[wid] = cnt;
    __syncthreads();
    if (wid == 0) {
        const uint32_t c   = lane < 8 ? s_cnt[lane] : 0u;
        const uint32_t tot = __reduce_add_sync(kFull, c);
        uint32_t       excl = 0, povf = 0;
        if (tile == 0) {
            if (lane == 0) publish(state, 0, epoch, kFlagIncl, 0, tot);
        } else {
            if (lane == 0) publish(state, tile, epoch, kFlagAgg, 0, tot);
            lookback(state, tile, epoch, status, excl, povf);
            if (lane == 0) publish(state, tile, epoch, kFlagIncl, 0, excl + tot);
        }
        uint32_t inc = c;
#pragma unroll
        for (uint32_t o = 1; o < 8; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane < 8) s_pre[lane] = excl + inc - c;
    }
    __syncthreads();
    if (t >= ntl) return;
    const uint32_t lt       = lanemask_lt();
    uint32_t       pre      = s_pre[wid];
    const uint64_t srcbytes = 2ull * n_codes;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t idx  = t * 256 + 32 * i + lane;
        const uint32_t rank = pre + __popc(bm[i] & lt);
        if (presum && idx < m) presum[idx] = rank;
        if ((bm[i] >> lane) & 1u && out) {
            const uint64_t b0 = 16ull * idx;
            if (b0 + 16 <= srcbytes) {
                reinterpret_cast<uint4*>(out)[rank] = reinterpret_cast<const uint4*>(shuffled)[idx];
            } else {
                for (int k = 0; k < 16; ++k) out[16ull * rank + k] = b0 + k < srcbytes ? shuffled[b0 + k] : 0;
            }
        }
        pre += __popc(bm[i]);
    }
    if (t == ntl - 1 && lane == 0) {
        if (presum) presum[m] = pre;
        *total = pre;
    }
}

cudaError_t launch_scan_encode(const uint8_t* shuffled, const uint32_t* byteflag,
                               uint32_t n_codes, uint32_t* presum, uint8_t* out,
                               uint64_t* state, uint32_t* ticket, uint32_t* status,
                               uint32_t* total, uint32_t* epoch, cudaStream_t s)
{
    const uint32_t m     = 32u * (uint32_t)cdiv(n_codes, 256);
    const uint32_t tiles = (uint32_t)cdiv(m, 256);
    k_scan_encode<<<(uint32_t)cdiv(tiles, 8), 256, 0, s>>>(shuffled, byteflag, n_codes, m, presum,
                                                           out, state, ticket, status, total, epoch);
    return cudaGetLastError();
}

}  // namespace fz
