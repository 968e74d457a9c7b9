// Float-center k-means and lookup.  No counterpart in the reference, whose centers are uint8
// (kmeans.cu:367); this mode generalises its assign and update (kmeans.cu:125-199, 356-372):
//
//   * centers are fp32: c = float(double(sum) / double(count)) from the exact integer sums,
//     kept when a center has no member (kmeans.cu:360-362);
//   * distances: score_b = |c_b|^2 - 2 x.c_b with x.c_b from the tensor core, in one of two forms:
//     centers in [0, 256) -- every build's, and most uploaded ones -- as 24-bit fixed point in three
//     bytes (assignKernelX, exact integer products); any others as hi = bf16(c) and lo = bf16(c - hi)
//     with x exact in bf16 (assignKernelF, fp32 accumulation);
//   * error bound: of the bf16 form, |score error| <= 4e-5 (|x||c| + |c|^2) (the split leaves
//     |c - hi - lo| <= 2^-18 |c|; the products are exact in fp32; at most 127 accumulation roundings
//     of <= 2^-23 each; |c|^2 and the final subtraction round once more); of the fixed-point form, see
//     assignKernelX; of few rows' lookups, which sum (x - c)^2 in fp32, see lookupDirectF.  A member whose
//     best-versus-second margin is at most kMarginScale (|x| max|c| + max|c|^2) -- six times the bf16
//     form's bound for both scores together -- plus the other forms' own terms is re-scored in FP64: the
//     warp computes its squared distance to every center within that margin of the best in the
//     oracle's fixed order (lane partials of four fused multiply-adds, then a butterfly of pairwise
//     sums) and keeps the lowest index on ties (kmeans.cu:131-135); every other center and member is
//     decided by more than the error;
//   * inertia: per node, sum_b (Q_b - 2 c_b.S_b + n_b |c_b|^2) in FP64 from the exact member
//     sums S_b, counts n_b and sums of squared norms Q_b, with the centers of the assignment.
#include "kmeans.cuh"
#include "timing.h"
#include "tuning.h"

#include <cuda_bf16.h>

#include <algorithm>

namespace rbw {
namespace {

constexpr float kMarginScale = 1.0f / 2048.0f;

__device__ __forceinline__ uint32_t packBf16x2(float a, float b)
{
    const __nv_bfloat16 ha = __float2bfloat16_rn(a), hb = __float2bfloat16_rn(b);
    return uint32_t(__bfloat16_as_ushort(ha)) | (uint32_t(__bfloat16_as_ushort(hb)) << 16);
}

// hi and lo bf16 parts of two values, packed as bf16x2 (first value in the low half).
__device__ __forceinline__ void splitPair(float a, float b, uint32_t& hi, uint32_t& lo)
{
    const __nv_bfloat16 ha = __float2bfloat16_rn(a), hb = __float2bfloat16_rn(b);
    hi = uint32_t(__bfloat16_as_ushort(ha)) | (uint32_t(__bfloat16_as_ushort(hb)) << 16);
    lo = packBf16x2(a - __bfloat162float(ha), b - __bfloat162float(hb));
}

// Split, |c|^2 and bound of one node (256 threads: thread t handles dims 8 (t % 16) .. +7 of
// center t / 16).  `red` is 16 floats of shared memory.  limbs: the fixed-point operand (centers in
// [0, 256)), else the bf16 one.
__device__ void prepareNode(const float* __restrict__ c, uint8_t* __restrict__ split, float* __restrict__ cn,
                            float2* __restrict__ bound, uint32_t B, bool limbs, float* red)
{
    const uint32_t t = threadIdx.x;
    const uint32_t j = t / 16, part = t % 16, d0 = part * 8;
    float v[8];
    double nrm = 0.0;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
        v[k] = j < B ? c[j * kDims + d0 + k] : 0.f;
        nrm = __fma_rn(double(v[k]), double(v[k]), nrm);
    }
    if (limbs) {
        // round(c * 2^16) in three bytes, the highest in rows 0-15, then 16-31 and 32-47; dims
        // 8 part .. + 7 are half of 16-byte chunk part / 2
        uint32_t w[3][2] = {};
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const uint32_t q = min(__float2uint_rn(v[k] * 65536.0f), 0xFFFFFFu);
#pragma unroll
            for (uint32_t l = 0; l < 3; l++) w[l][k / 4] |= ((q >> (16 - 8 * l)) & 0xFFu) << (8 * (k % 4));
        }
#pragma unroll
        for (uint32_t l = 0; l < 3; l++) {
            const uint32_t r = 16 * l + j;
            *reinterpret_cast<uint2*>(split + r * 128 + (((part / 2) ^ (r & 7u)) << 4) + (part % 2) * 8) =
                make_uint2(w[l][0], w[l][1]);
        }
    } else {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) splitPair(v[2 * k], v[2 * k + 1], hi[k], lo[k]);
        const uint32_t kb = d0 / 64, ch = (d0 % 64) / 8;
        uint8_t* base = split + kb * 4096;
        *reinterpret_cast<uint4*>(base + j * 128 + ((ch ^ (j & 7u)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        const uint32_t r = 16 + j;
        *reinterpret_cast<uint4*>(base + r * 128 + ((ch ^ (r & 7u)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
#pragma unroll
    for (uint32_t off = 8; off > 0; off >>= 1) nrm = __dadd_rn(nrm, __shfl_xor_sync(0xFFFFFFFFu, nrm, off));
    if (part == 0) {
        cn[j] = j < B ? __double2float_rn(nrm) : kPadNormF;
        red[j] = j < B ? __double2float_ru(nrm) : 0.f;
    }
    __syncthreads();
    if (t == 0) {
        float c2 = 0.f;
        for (uint32_t b = 0; b < B; b++) c2 = fmaxf(c2, red[b]);
        *bound = make_float2(__fsqrt_ru(c2), c2);
    }
}

__global__ void __launch_bounds__(256) centersToFloatKernel(KMeansLevelF lv)
{
    __shared__ float red[kMaxBranch];
    const uint32_t g = blockIdx.x;
    const uint8_t* u = lv.base.centers + uint64_t(g) * kMaxBranch * kDims;
    float* c = lv.centers + uint64_t(g) * kMaxBranch * kDims;
    for (uint32_t i = threadIdx.x; i < kMaxBranch * kDims; i += blockDim.x)
        c[i] = i / kDims < lv.base.B ? float(u[i]) : 0.f;
    __syncthreads();
    prepareNode(c, lv.split + uint64_t(g) * kSplitBytes, lv.cn + uint64_t(g) * kMaxBranch, lv.bound + g, lv.base.B,
                true, red);
}

__global__ void __launch_bounds__(256) prepareNodesKernel(const float* centers, uint8_t* split, float* cn,
                                                          float2* bound, uint32_t B, bool limbs)
{
    __shared__ float red[kMaxBranch];
    const uint64_t g = blockIdx.x;
    prepareNode(centers + g * kMaxBranch * kDims, split + g * kSplitBytes, cn + g * kMaxBranch, bound + g, B, limbs,
                red);
}

// The nearest of the centers in `cand` to the row whose dims 4 lane .. 4 lane + 3 are x0 .. x3, in FP64
// in the oracle's order (orc_dist64: lane partials of four fused multiply-adds, then a butterfly of
// pairwise sums), the lowest index on ties.  All lanes of the warp call it; cBase is their dims of
// center 0.  A distance that is no number is never the smallest, except that of center 0, where a scan of
// all centers starts (the oracle's).
__device__ __forceinline__ uint32_t nearestFp64(const float* cBase, uint32_t cand, double x0, double x1, double x2,
                                                double x3)
{
    auto partial = [&](const float4& c4) {
        double e = __dsub_rn(x0, double(c4.x));
        double p = __fma_rn(e, e, 0.0);
        e = __dsub_rn(x1, double(c4.y));
        p = __fma_rn(e, e, p);
        e = __dsub_rn(x2, double(c4.z));
        p = __fma_rn(e, e, p);
        e = __dsub_rn(x3, double(c4.w));
        return __fma_rn(e, e, p);
    };
    double bestD = 0.0;
    uint32_t bb = kMaxBranch;
    auto take = [&](double p, uint32_t b) {
        if (bb == kMaxBranch ? p == p || b == 0 : p < bestD) {
            bestD = p;
            bb = b;
        }
    };
    while (cand != 0) {
        const uint32_t b0 = __ffs(cand) - 1;
        cand &= cand - 1;
        const uint32_t b1 = cand ? __ffs(cand) - 1 : b0; // the same again if there is no other
        cand &= cand - 1;
        const float4 c0 = __ldg(reinterpret_cast<const float4*>(cBase + b0 * kDims));
        const float4 c1 = __ldg(reinterpret_cast<const float4*>(cBase + b1 * kDims));
        double p0 = partial(c0), p1 = partial(c1);
#pragma unroll
        for (uint32_t off = 16; off > 0; off >>= 1) {
            p0 = __dadd_rn(p0, __shfl_xor_sync(0xFFFFFFFFu, p0, off));
            p1 = __dadd_rn(p1, __shfl_xor_sync(0xFFFFFFFFu, p1, off));
        }
        take(p0, b0);
        take(p1, b1);
    }
    return bb == kMaxBranch ? 0u : bb;
}

// ------------------------------------------------------------------ assign, any fp32 centers
// Lookups through trees with centers outside [0, 256) (uploaded ones: centers of a build are means of
// bytes), for which the fixed-point operand of assignKernelX does not exist.
constexpr uint32_t kAfThreads = 128;
constexpr uint32_t kAfRows = 128;
constexpr uint32_t kAfTmemCols = 32;
constexpr uint32_t kAfCtasPerSm = 3;
constexpr uint32_t kAfTileWindow = kAfThreads; // one tile entry per thread per refill

struct AssignFSmem {
    uint8_t a[2][kAfRows * 128];     // members as bf16, two K-blocks of 64 dims, 128-byte swizzle
    uint8_t b[2][32 * 128];          // the node's hi (rows 0-15) and lo (rows 16-31) centers
    uint8_t x8[kAfRows * kDims];     // members as uint8, 128-byte swizzle (FP64 re-score)
    NodeTile win[kAfTileWindow];     // tiles [winBase, winBase + kAfTileWindow) of the CTA's range
    float cn[kMaxBranch];
    uint32_t xn[kAfRows];
    float2 bnd;
    uint64_t mmaBar;
    uint32_t tmemBase;
    uint32_t abortFlag;
    uint32_t refined;
    uint32_t visited;
};
constexpr size_t kAfSmemBytes = sizeof(AssignFSmem) + 1024;

// bf16 of the four bytes of w (exact: integers below 256), packed in two bf16x2 words.
__device__ __forceinline__ void bytesToBf16(uint32_t w, uint32_t& lo2, uint32_t& hi2)
{
    const float f0 = __int_as_float(int(__byte_perm(w, 0x4B000000u, 0x7540u))) - 8388608.0f;
    const float f1 = __int_as_float(int(__byte_perm(w, 0x4B000000u, 0x7541u))) - 8388608.0f;
    const float f2 = __int_as_float(int(__byte_perm(w, 0x4B000000u, 0x7542u))) - 8388608.0f;
    const float f3 = __int_as_float(int(__byte_perm(w, 0x4B000000u, 0x7543u))) - 8388608.0f;
    // the low 16 bits of these floats are zero, so the bf16 bits are the high halves
    lo2 = (__float_as_uint(f0) >> 16) | (__float_as_uint(f1) & 0xFFFF0000u);
    hi2 = (__float_as_uint(f2) >> 16) | (__float_as_uint(f3) & 0xFFFF0000u);
}

__global__ void __launch_bounds__(kAfThreads, kAfCtasPerSm) assignKernelF(KMeansLevelF lv, const NodeTile* tiles,
                                                                         const uint32_t* nTilesDev)
{
    extern __shared__ uint8_t smemRaw[];
    AssignFSmem& S = *reinterpret_cast<AssignFSmem*>(smemAligned(smemRaw));
    const KMeansLevel& L0 = lv.base;
    const uint32_t tid = threadIdx.x, lane = tid % 32;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, tid / 32, 0); // uniform
    const uint32_t B = L0.B;
    const uint32_t T = *nTilesDev;
    const uint32_t t0 = static_cast<uint32_t>(uint64_t(T) * blockIdx.x / gridDim.x);
    const uint32_t t1 = static_cast<uint32_t>(uint64_t(T) * (blockIdx.x + 1) / gridDim.x);
    volatile uint32_t* abortFlag = &S.abortFlag;
    if (tid == 0) {
        mbarInit(&S.mmaBar, 1);
        S.abortFlag = 0;
        S.refined = 0;
        S.visited = 0;
        fenceMbarInit();
    }
    if (warp == 0) {
        tmemAlloc(&S.tmemBase, kAfTmemCols);
        tmemRelinquish();
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = S.tmemBase;
    const bool issuer = warp == 0 && electOne(); // one thread issues and commits every MMA
    uint32_t curNode = 0xFFFFFFFFu, phase = 0;
    // The tile list is read a window of kAfTileWindow tiles at a time (one
    // load per thread, all in flight together), the member indices two tiles ahead and the member
    // rows one tile ahead of their use, into registers, so that no tile waits on a chain of
    // dependent global loads.  Every thread runs the same window refills (uniform).
    uint32_t winBase = t0;
    auto refill = [&](uint32_t base) {
        __syncthreads(); // nobody reads the old window any more
        if (base + tid < t1) {
            S.win[tid] = tiles[base + tid];
        }
        winBase = base;
        __syncthreads();
    };
    auto entry = [&](uint32_t t) -> NodeTile {
        if (t - winBase >= kAfTileWindow) refill(t);
        return S.win[t - winBase];
    };
    // rows past a tile's count repeat its first member (their results are not used)
    auto loadIndices = [&](const NodeTile& tn, uint32_t (&m)[kAfRows / 16]) {
#pragma unroll
        for (uint32_t k = 0; k < kAfRows / 16; k++) {
            const uint32_t row = 16u * k + tid / 8;
            m[k] = L0.members[uint64_t(tn.start) + (row < tn.count ? row : 0u)];
        }
    };
    const uint32_t c8 = tid % 8;
    auto loadRows = [&](const uint32_t (&m)[kAfRows / 16], uint4 (&v)[kAfRows / 16]) {
#pragma unroll
        for (uint32_t k = 0; k < kAfRows / 16; k++)
            v[k] = __ldg(reinterpret_cast<const uint4*>(L0.desc + uint64_t(m[k]) * kDims) + c8);
    };
    if (t0 < t1) refill(t0);
    uint32_t t = t0;
    NodeTile ti{}, tn1{};
    uint32_t mNext[kAfRows / 16];
    uint4 v[kAfRows / 16];
    if (t < t1) {
        ti = entry(t);
        loadIndices(ti, mNext);
        loadRows(mNext, v);
    }
    uint32_t n1 = min(t + 1, t1);
    if (n1 < t1) {
        tn1 = entry(n1);
        loadIndices(tn1, mNext);
    }
    while (t < t1) {
        if (tid == 0) S.visited += ti.count;
        if (ti.node != curNode) {
            __syncthreads(); // the previous node's centers are no longer read
            curNode = ti.node;
            const uint4* src = reinterpret_cast<const uint4*>(lv.split + uint64_t(curNode) * kSplitBytes);
#pragma unroll
            for (uint32_t k = 0; k < kSplitBytes / 16 / kAfThreads; k++)
                reinterpret_cast<uint4*>(&S.b[0][0])[tid + kAfThreads * k] = src[tid + kAfThreads * k];
            if (tid < kMaxBranch) {
                S.cn[tid] = lv.cn[uint64_t(curNode) * kMaxBranch + tid];
            }
            if (tid == 0) S.bnd = lv.bound[curNode];
        }
        {
            // Eight threads per row, 16 rows per round: thread c8 = tid % 8 stages dims
            // 16 c8 .. 16 c8 + 15 of its row as uint8 and as bf16 (K-block c8 / 4, 16-byte chunks
            // 2 (c8 % 4) and 2 (c8 % 4) + 1 of the 128-byte row, swizzled by the row's low bits),
            // and the eight threads add up the row's |x|^2.
#pragma unroll
            for (uint32_t k = 0; k < kAfRows / 16; k++) {
                const uint32_t row = 16u * k + tid / 8;
                *reinterpret_cast<uint4*>(S.x8 + row * kDims + ((c8 ^ (row & 7u)) << 4)) = v[k];
                uint32_t w[8];
                bytesToBf16(v[k].x, w[0], w[1]);
                bytesToBf16(v[k].y, w[2], w[3]);
                bytesToBf16(v[k].z, w[4], w[5]);
                bytesToBf16(v[k].w, w[6], w[7]);
                uint8_t* rowBase = S.a[c8 / 4] + row * 128;
                const uint32_t j0 = (c8 % 4) * 2;
                *reinterpret_cast<uint4*>(rowBase + ((j0 ^ (row & 7u)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<uint4*>(rowBase + (((j0 + 1) ^ (row & 7u)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
                uint32_t xn = __dp4a(v[k].x, v[k].x, 0u);
                xn = __dp4a(v[k].y, v[k].y, xn);
                xn = __dp4a(v[k].z, v[k].z, xn);
                xn = __dp4a(v[k].w, v[k].w, xn);
                xn += __shfl_xor_sync(0xFFFFFFFFu, xn, 1);
                xn += __shfl_xor_sync(0xFFFFFFFFu, xn, 2);
                xn += __shfl_xor_sync(0xFFFFFFFFu, xn, 4);
                if (c8 == 0) S.xn[row] = xn;
            }
        }
        // the next live tile's rows into registers (its indices were loaded one tile ago), the
        // indices of the one after it; both land while this tile is scored
        uint32_t n2 = t1;
        NodeTile tn2{};
        if (n1 < t1) {
            loadRows(mNext, v);
            n2 = n1 + 1;
            if (n2 < t1) {
                tn2 = entry(n2);
                loadIndices(tn2, mNext);
            }
        }
        const uint32_t row = tid;
        const bool valid = row < ti.count;
        // generic-proxy shared-memory writes read by the tensor core
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            tcFenceAfter();
            const uint64_t aDesc = smemDescSw128(smemAddr(&S.a[0][0])), bDesc = smemDescSw128(smemAddr(&S.b[0][0]));
#pragma unroll
            for (uint32_t k = 0; k < 8; k++)
                if (issuer)
                    mmaBf16(tmem, aDesc + (((k >> 2) * (kAfRows * 128) + 32u * (k & 3u)) >> 4),
                            bDesc + (((k >> 2) * (32 * 128) + 32u * (k & 3u)) >> 4), idescBf16(32), k > 0 ? 1u : 0u);
            if (issuer) mmaCommit(&S.mmaBar);
        }
        if (!mbarWait(&S.mmaBar, phase, abortFlag, L0.err, 50)) break;
        phase ^= 1u;
        tcFenceAfter();
        uint32_t rh[16], rl[16];
        tmemLoad16(tmem + ((warp * 32u) << 16), rh);
        tmemLoad16(tmem + ((warp * 32u) << 16) + 16u, rl);
        tmemWaitTie(rh);
        tmemWaitTie(rl);
        tcFenceBefore(); // the next tile's MMA overwrites these columns after the barriers below
        float best = __int_as_float(0x7F800000), second = best;
        uint32_t bi = 0;
#pragma unroll
        for (uint32_t b = 0; b < kMaxBranch; b++) {
            if (b < B) {
                const float dot = __fadd_rn(__uint_as_float(rh[b]), __uint_as_float(rl[b]));
                const float s = __fmaf_rn(-2.f, dot, S.cn[b]);
                if (s < best) {
                    second = best;
                    best = s;
                    bi = b;
                } else if (s < second) {
                    second = s;
                }
            }
        }
        const float thr = kMarginScale * __fmaf_rn(__fsqrt_ru(float(S.xn[row])), S.bnd.x, S.bnd.y);
        const bool refine = valid && !(second - best > thr);
        uint32_t mask = __ballot_sync(0xFFFFFFFFu, refine);
        if (mask != 0) {
            // FP64 re-score of the flagged rows of this warp, one row at a time, every lane on
            // dims 4 lane .. 4 lane + 3 (the oracle's orc_dist64 order) -- of the centers whose
            // score is within the margin of the best, two at a time: by the margin's definition
            // every other center is farther than the best in FP64 too.
            uint32_t near = 0;
#pragma unroll
            for (uint32_t b = 0; b < kMaxBranch; b++) {
                const float dot = __fadd_rn(__uint_as_float(rh[b]), __uint_as_float(rl[b]));
                const float s = __fmaf_rn(-2.f, dot, S.cn[b]);
                if (b < B && !(s - best > thr)) near |= 1u << b;
            }
            if (lane == 0) atomicAdd(&S.refined, uint32_t(__popc(mask)));
            const float* cBase = lv.centers + uint64_t(curNode) * kMaxBranch * kDims + 4u * lane;
            while (mask != 0) {
                const uint32_t src = __ffs(mask) - 1;
                mask &= mask - 1;
                const uint32_t cand = __shfl_sync(0xFFFFFFFFu, near, src);
                const uint32_t xw = *reinterpret_cast<const uint32_t*>(
                    S.x8 + (warp * 32u + src) * kDims + (((lane >> 2) ^ (src & 7u)) << 4) + ((lane & 3u) << 2));
                const double x0 = double(xw & 0xFFu), x1 = double((xw >> 8) & 0xFFu);
                const double x2 = double((xw >> 16) & 0xFFu), x3 = double(xw >> 24);
                const uint32_t bb = nearestFp64(cBase, cand, x0, x1, x2, x3);
                if (lane == src) bi = bb;
            }
        }
        if (valid) {
            const uint64_t at = uint64_t(ti.start) + row;
            if (L0.leaf) L0.leaf[L0.members[at]] = curNode * B + bi;
            else L0.assign[at] = static_cast<uint8_t>(bi);
        }
        __syncthreads(); // the tiles and xn are rewritten by the next step
        t = n1;
        ti = tn1;
        n1 = n2;
        tn1 = tn2;
    }
    if (tid == 0) {
        if (S.refined) atomicAdd(lv.refined, (unsigned long long)S.refined);
        if (S.visited) atomicAdd(lv.refined + 1, (unsigned long long)S.visited);
    }
    if (warp == 0) {
        tcFenceAfter();
        tmemDealloc(tmem, kAfTmemCols);
    }
}

// ------------------------------------------------------------------ assign, centers in [0, 256)
// The build's Lloyd step and lookups: assignKernel's tiles with fp32 centers.  A center is
// round(c * 2^16), three bytes, so the distances are one u8 x u8 -> s32 product of the tile as it was
// gathered (no conversion of the rows) with N = 48: x.c = 2^-16 (65536 D2 + 256 D1 + D0), D exact.
//   * |x.c - that| <= 2^-17 sum(x) <= 8.7e-5 |x|; forming D2 + 2^-8 (D1 + floor(D0 / 2^8)) loses less
//     than 2^-8 and rounds once, |c|^2 and the score round once: two scores are off by less than
//     2^-21 (|x||c| + |c|^2) + 3.6e-4 |x| + 0.02 together, which the margin covers twice
//     (kMarginScale's part alone: 256 times the first term).
//   * Members within the margin go to a queue; the warps settle them in FP64 together, each row's
//     near centers two at a time (oracle's orc_dist64 order), when the queue fills and at the end of
//     the CTA's tiles: about 1 % of the rows, whose 1,200-cycle chains would otherwise hold up
//     nearly every tile.  Their counts and sums go to global memory directly.
// 300,007 members, one Lloyd step: 23-28 us, 33-40 us by bf16 halves (rows converted to bf16 in shared
// memory, two K-blocks, the queue's work inside each tile); a lookup level of 200,003: 15.6, 21.5 us.
constexpr uint32_t kAxThreads = 128;
constexpr uint32_t kAxRows = 128;
constexpr uint32_t kAxTmemCols = 64;    // three limbs' distances | sums
constexpr uint32_t kAxSumCol = 48;
constexpr uint32_t kAxCtasPerSm = 4;    // by shared memory (~49 KB each)
constexpr uint32_t kAxFlushTiles = 65536; // 65,536 x 128 x 255 < 2^31
constexpr uint32_t kAxQueue = 256;      // queued members; a tile adds at most 128
constexpr uint32_t kAxFrozen = 0x80000000u;

struct AssignXSmem {
    uint8_t tile[2][kAxRows * kDims];     // member rows, 128-byte swizzle
    uint8_t cen[48 * kDims];              // the node's limbs, same layout
    uint8_t oh[kAxRows * kMaxBranch];     // [member][center] one-hot
    NodeTile win[kAxThreads];             // tiles [winBase, winBase + 128) of the CTA's range
    uint4 queue[kAxQueue];                // member position, node, near centers | previous << 16, |x|^2
    unsigned long long q[kMaxBranch];
    float cn[kMaxBranch];
    uint32_t cnt[kMaxBranch];
    float2 bnd;
    uint64_t mmaBar, sumBar;
    uint32_t tmemBase, abortFlag, chg, nQueue, nFold, refined, visited;
};
constexpr size_t kAxSmemBytes = sizeof(AssignXSmem) + 1024;

__global__ void __launch_bounds__(kAxThreads, kAxCtasPerSm) assignKernelX(KMeansLevelF lv, const NodeTile* tiles,
                                                                         const uint32_t* nTilesDev)
{
    extern __shared__ uint8_t smemRaw[];
    AssignXSmem& S = *reinterpret_cast<AssignXSmem*>(smemAligned(smemRaw));
    const KMeansLevel& L0 = lv.base;
    const uint32_t tid = threadIdx.x, lane = tid % 32;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, tid / 32, 0); // uniform
    const uint32_t B = L0.B;
    const bool build = lv.lookupOnly == 0;
    if (build && blockIdx.x == 0 && tid == 0) *L0.activeCount = 0; // counted by the update that follows
    const uint32_t T = *nTilesDev;
    const uint32_t t0 = static_cast<uint32_t>(uint64_t(T) * blockIdx.x / gridDim.x);
    const uint32_t t1 = static_cast<uint32_t>(uint64_t(T) * (blockIdx.x + 1) / gridDim.x);
    if (t0 == t1) return; // uniform: fewer tiles than CTAs
    volatile uint32_t* abortFlag = &S.abortFlag;
    if (tid == 0) {
        mbarInit(&S.mmaBar, 1);
        mbarInit(&S.sumBar, 1);
        S.abortFlag = 0;
        S.nQueue = 0;
        S.refined = 0;
        S.visited = 0;
        fenceMbarInit();
    }
    if (warp == 0) {
        tmemAlloc(&S.tmemBase, kAxTmemCols);
        tmemRelinquish();
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = S.tmemBase;
    const bool issuer = warp == 0 && electOne(); // one thread issues and commits every MMA
    uint32_t curNode = 0xFFFFFFFFu, phase = 0, sumPhase = 0, accTiles = 0, buf = 0;
    uint32_t myCnt = 0, myChg = 0;   // lane c < 16: this warp's rows that chose center c, and the
    unsigned long long myQ = 0;      // sum of their |x|^2
    bool curExclusive = false;       // every tile of the current node is in this CTA's range
    bool ok = true;
    uint32_t winBase = t0;
    auto refill = [&](uint32_t base) {
        __syncthreads(); // nobody reads the old window any more
        if (base + tid < t1) {
            NodeTile x = tiles[base + tid];
            if (build && L0.lastChanged[x.node] == 0) x.count |= kAxFrozen; // frozen node (kmeans.cu:238-240)
            S.win[tid] = x;
        }
        winBase = base;
        __syncthreads();
    };
    auto entry = [&](uint32_t t) -> NodeTile {
        if (t - winBase >= kAxThreads) refill(t);
        return S.win[t - winBase];
    };
    auto nextLive = [&](uint32_t t) -> uint32_t {
        for (; t < t1; t++)
            if (!(entry(t).count & kAxFrozen)) return t;
        return t1;
    };
    auto loadIndices = [&](const NodeTile& tn, uint32_t (&m)[kAxRows / 16]) {
#pragma unroll
        for (uint32_t k = 0; k < kAxRows / 16; k++) {
            const uint32_t row = 16u * k + tid / 8;
            m[k] = L0.members[uint64_t(tn.start) + (row < tn.count ? row : 0u)];
        }
    };
    auto gatherRows = [&](const uint32_t (&m)[kAxRows / 16], uint32_t b) {
        const uint32_t c = tid % 8;
#pragma unroll
        for (uint32_t k = 0; k < kAxRows / 16; k++) {
            const uint32_t row = 16u * k + tid / 8;
            cpAsync16(S.tile[b] + row * kDims + ((c ^ (row & 7u)) << 4), L0.desc + uint64_t(m[k]) * kDims + (c << 4));
        }
        cpAsyncCommit();
    };
    // Settles the queued members, one per warp at a time; their counts and sums go to global memory
    // atomically.  At the end of the CTA's tiles (`last`) those of the current node, which are all of
    // them where a node has many tiles, form one more tile for the sums MMA instead: 4,000 queued
    // members of one node are half a million atomics on 1,280 addresses.
    auto drain = [&](bool last) {
        const bool fold = last && build && accTiles > 0;
        if (fold) {
            if (issuer) mmaCommit(&S.sumBar);
            ok = mbarWait(&S.sumBar, sumPhase, abortFlag, L0.err, 57) && ok;
            sumPhase ^= 1u;
            tcFenceAfter();
            *reinterpret_cast<uint4*>(S.oh + tid * kMaxBranch) = make_uint4(0, 0, 0, 0);
            if (tid == 0) S.nFold = 0;
        }
        __syncthreads(); // the queue is complete
        const uint32_t nq = S.nQueue;
        for (uint32_t e = warp; e < nq; e += kAxThreads / 32) {
            const uint4 en = S.queue[e];
            const uint32_t member = L0.members[en.x];
            const uint32_t xw = __ldg(reinterpret_cast<const uint32_t*>(L0.desc + uint64_t(member) * kDims) + lane);
            const float* cBase = lv.centers + uint64_t(en.y) * kMaxBranch * kDims + 4u * lane;
            const double x0 = double(xw & 0xFFu), x1 = double((xw >> 8) & 0xFFu);
            const double x2 = double((xw >> 16) & 0xFFu), x3 = double(xw >> 24);
            const uint32_t bi = nearestFp64(cBase, en.z & 0xFFFFu, x0, x1, x2, x3);
            if (!build) {
                if (lane == 0) {
                    if (L0.leaf) L0.leaf[member] = en.y * B + bi;
                    else L0.assign[en.x] = static_cast<uint8_t>(bi);
                    if (L0.counts) atomicAdd(L0.counts + uint64_t(en.y) * kMaxBranch + bi, 1u);
                }
                continue;
            }
            if (lane == 0) L0.assign[en.x] = static_cast<uint8_t>(bi);
            uint32_t slot = kAxRows;
            if (fold && en.y == curNode) {
                if (lane == 0) slot = atomicAdd(&S.nFold, 1u);
                slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
            }
            if (slot < kAxRows) {
                *reinterpret_cast<uint32_t*>(S.tile[buf] + slot * kDims + (((lane >> 2) ^ (slot & 7u)) << 4) +
                                             ((lane & 3u) << 2)) = xw;
                if (lane == 0) {
                    S.oh[slot * kMaxBranch + bi] = 1;
                    atomicAdd(&S.cnt[bi], 1u);
                    atomicAdd(&S.q[bi], (unsigned long long)en.w);
                    if (en.z >> 16 != bi) atomicAdd(&S.chg, 1u);
                }
            } else {
                if (en.y == curNode) curExclusive = false; // a plain-store flush would overwrite these
                unsigned long long* sum = L0.sums + (uint64_t(en.y) * kMaxBranch + bi) * kDims + 4u * lane;
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) atomicAdd(sum + k, (unsigned long long)((xw >> (8 * k)) & 0xFFu));
                if (lane == 0) {
                    atomicAdd(L0.counts + uint64_t(en.y) * kMaxBranch + bi, 1u);
                    atomicAdd(lv.q + uint64_t(en.y) * kMaxBranch + bi, (unsigned long long)en.w);
                    if (en.z >> 16 != bi) atomicAdd(L0.changed + en.y, 1u);
                }
            }
        }
        if (fold) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        curExclusive = __syncthreads_and(curExclusive) != 0; // and the queue has been read
        if (fold && warp == 0) {
            tcFenceAfter();
            mmaU8x4(issuer, tmem + kAxSumCol, smemDescSw128(smemAddr(S.tile[buf])), 4096u, smemDescMn16(smemAddr(S.oh)),
                    512u, idescU8(16) | kIdescMnMajorAB, 1u);
        }
        if (tid == 0) {
            S.refined += nq;
            S.nQueue = 0;
        }
        __syncthreads();
    };
    auto flush = [&]() {
        if (curNode != 0xFFFFFFFFu && (build || L0.counts)) {
            if (lane < kMaxBranch && myCnt) atomicAdd(&S.cnt[lane], myCnt);
            if (build && lane < kMaxBranch && myQ) atomicAdd(&S.q[lane], myQ);
            if (lane == 0 && myChg) atomicAdd(&S.chg, myChg);
            if (accTiles > 0) {
                if (issuer) mmaCommit(&S.sumBar); // nothing was committed yet for the last sums MMA
                ok = ok && mbarWait(&S.sumBar, sumPhase, abortFlag, L0.err, 55);
                sumPhase ^= 1u;
                tcFenceAfter();
                uint32_t r[16];
                tmemLoad16(tmem + kAxSumCol + ((warp * 32u) << 16), r); // lane = dimension tid
                tmemWaitTie(r);
                tcFenceBefore();
#pragma unroll
                for (uint32_t b = 0; b < kMaxBranch; b++) {
                    if (r[b] == 0) continue;
                    unsigned long long* dst = L0.sums + (uint64_t(curNode) * kMaxBranch + b) * kDims + tid;
                    if (curExclusive) *dst = r[b];
                    else atomicAdd(dst, (unsigned long long)r[b]);
                }
            }
            __syncthreads(); // S.cnt, S.q and S.chg complete
            if (tid < kMaxBranch && S.cnt[tid]) {
                uint32_t* c = L0.counts + uint64_t(curNode) * kMaxBranch + tid;
                unsigned long long* qd = lv.q + uint64_t(curNode) * kMaxBranch + tid;
                if (build && curExclusive) {
                    *c = S.cnt[tid];
                    *qd = S.q[tid];
                } else {
                    atomicAdd(c, S.cnt[tid]);
                    if (build) atomicAdd(qd, S.q[tid]);
                }
            }
            if (build && tid == 0 && S.chg) {
                if (curExclusive) L0.changed[curNode] = S.chg;
                else atomicAdd(L0.changed + curNode, S.chg);
            }
        }
        accTiles = 0;
        myCnt = 0;
        myChg = 0;
        myQ = 0;
        __syncthreads();
    };
    refill(t0);
    uint32_t t = nextLive(t0);
    NodeTile ti{}, tn1{};
    uint32_t mNext[kAxRows / 16];
    if (t < t1) {
        ti = entry(t);
        loadIndices(ti, mNext);
        gatherRows(mNext, buf);
    }
    uint32_t n1 = t < t1 ? nextLive(t + 1) : t1;
    if (n1 < t1) {
        tn1 = entry(n1);
        loadIndices(tn1, mNext);
    }
    while (ok && t < t1) {
        if (tid == 0) S.visited += ti.count;
        if (ti.node != curNode) {
            flush();
            curNode = ti.node;
            curExclusive = ti.first >= t0 && uint64_t(ti.first) + (L0.nodeCnt[curNode] + kAxRows - 1) / kAxRows <= t1;
            const uint4* src = reinterpret_cast<const uint4*>(lv.split + uint64_t(curNode) * kSplitBytes);
#pragma unroll
            for (uint32_t k = 0; k < 3; k++) reinterpret_cast<uint4*>(S.cen)[tid + kAxThreads * k] = src[tid + kAxThreads * k];
            if (tid < kMaxBranch) {
                S.cn[tid] = lv.cn[uint64_t(curNode) * kMaxBranch + tid];
                S.cnt[tid] = 0;
                S.q[tid] = 0;
            }
            if (tid == 0) {
                S.bnd = lv.bound[curNode];
                S.chg = 0;
            }
        } else if (accTiles == kAxFlushTiles) {
            // keep each s32 sum below 2^31: this node's partial results go out, later flushes add
            curExclusive = false;
            flush();
            if (tid < kMaxBranch) {
                S.cnt[tid] = 0;
                S.q[tid] = 0;
            }
            if (tid == 0) S.chg = 0;
        }
        const uint32_t row = tid;
        const bool valid = row < ti.count;
        const uint64_t at = uint64_t(ti.start) + row;
        const uint32_t prevAssign = build && valid ? L0.assign[at] : 0u;
        cpAsyncWait<0>(); // this tile's rows
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            tcFenceAfter();
            mmaU8x4(issuer, tmem, smemDescSw128(smemAddr(S.tile[buf])), 32u, smemDescSw128(smemAddr(S.cen)), 32u,
                    idescU8(48), 0u);
            if (issuer) mmaCommit(&S.mmaBar);
        }
        // |x|^2 of this thread's row while the product runs
        uint32_t xn = 0;
#pragma unroll
        for (uint32_t c = 0; c < 8; c++) {
            const uint4 x = *reinterpret_cast<const uint4*>(S.tile[buf] + row * kDims + ((c ^ (row & 7u)) << 4));
            xn = __dp4a(x.x, x.x, xn);
            xn = __dp4a(x.y, x.y, xn);
            xn = __dp4a(x.z, x.z, xn);
            xn = __dp4a(x.w, x.w, xn);
        }
        const float xLen = __fsqrt_ru(float(xn));
        const float thr = __fmaf_rn(kMarginScale, __fmaf_rn(xLen, S.bnd.x, S.bnd.y), __fmaf_rn(xLen, 7.2e-4f, 0.04f));
        if (!mbarWait(&S.mmaBar, phase, abortFlag, L0.err, 54)) {
            ok = false;
            break;
        }
        phase ^= 1u;
        tcFenceAfter();
        // The commit also covers the previous tile's sums MMAs: the other tile buffer and the one-hot
        // rows are free.
        uint32_t n2 = t1;
        NodeTile tn2{};
        if (n1 < t1) {
            gatherRows(mNext, buf ^ 1u);
            n2 = nextLive(n1 + 1);
            if (n2 < t1) {
                tn2 = entry(n2);
                loadIndices(tn2, mNext);
            }
        }
        float score[kMaxBranch];
        {
            uint32_t d2[16], d1[16], d0[16];
            const uint32_t at0 = tmem + ((warp * 32u) << 16);
            tmemLoad16(at0, d2);
            tmemLoad16(at0 + 16u, d1);
            tmemLoad16(at0 + 32u, d0);
            tmemWaitTie(d2);
            tmemWaitTie(d1);
            tmemWaitTie(d0);
            tcFenceBefore(); // the next tile's MMA overwrites these columns after the barriers below
#pragma unroll
            for (uint32_t b = 0; b < kMaxBranch; b++) {
                // both integers are below 2^23: placed in the mantissa of 2^23 and freed of it
                const float hi = __uint_as_float(d2[b] | 0x4B000000u) - 8388608.0f;
                const float lo = __uint_as_float((d1[b] + (d0[b] >> 8)) | 0x4B000000u) - 8388608.0f;
                score[b] = __fmaf_rn(-2.f, __fmaf_rn(lo, 0x1p-8f, hi), S.cn[b]);
            }
        }
        float best = __int_as_float(0x7F800000), second = best;
        uint32_t bi = 0;
#pragma unroll
        for (uint32_t b = 0; b < kMaxBranch; b++) {
            if (b < B) {
                const float s = score[b];
                if (s < best) {
                    second = best;
                    best = s;
                    bi = b;
                } else if (s < second) {
                    second = s;
                }
            }
        }
        const bool refine = valid && !(second - best > thr);
        if (refine) {
            uint32_t near = 0;
#pragma unroll
            for (uint32_t b = 0; b < kMaxBranch; b++)
                if (b < B && !(score[b] - best > thr)) near |= 1u << b;
            S.queue[atomicAdd(&S.nQueue, 1u)] = make_uint4(static_cast<uint32_t>(at), curNode, near | (prevAssign << 16), xn);
        }
        const bool settled = valid && !refine;
        if (settled) {
            if (L0.leaf) L0.leaf[L0.members[at]] = curNode * B + bi;
            else L0.assign[at] = static_cast<uint8_t>(bi);
        }
        if (build || L0.counts) {
            uint32_t chose = __ballot_sync(0xFFFFFFFFu, settled);
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t bits = __ballot_sync(0xFFFFFFFFu, (bi >> k) & 1u);
                chose &= (lane >> k) & 1u ? bits : ~bits;
            }
            myCnt += __popc(chose); // used of lanes below kMaxBranch
        }
        if (build) {
            const uint32_t word = settled ? 1u << (8u * (bi & 3u)) : 0u, quad = bi >> 2;
            *reinterpret_cast<uint4*>(S.oh + row * kMaxBranch) =
                make_uint4(quad == 0 ? word : 0u, quad == 1 ? word : 0u, quad == 2 ? word : 0u, quad == 3 ? word : 0u);
            myChg += __popc(__ballot_sync(0xFFFFFFFFu, settled && prevAssign != bi));
            const uint32_t xs = settled ? xn : 0u; // below 2^23: 32 of them fit 32 bits
            for (uint32_t b = 0; b < B; b++) {
                const uint32_t part = __reduce_add_sync(0xFFFFFFFFu, bi == b ? xs : 0u);
                if (lane == b) myQ += part;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads(); // one-hot rows and queue entries are in, every warp has read its distances
        if (build) {
            if (warp == 0) {
                tcFenceAfter();
                mmaU8x4(issuer, tmem + kAxSumCol, smemDescSw128(smemAddr(S.tile[buf])), 4096u, smemDescMn16(smemAddr(S.oh)),
                        512u, idescU8(16) | kIdescMnMajorAB, accTiles);
            }
            accTiles++;
        }
        if (S.nQueue > kAxQueue - kAxRows) drain(false); // uniform
        buf ^= 1u;
        t = n1;
        ti = tn1;
        n1 = n2;
        tn1 = tn2;
    }
    cpAsyncWait<0>(); // a prefetch of a tile that was not scored (abort) must land before exit
    if (ok) {
        drain(true);
        flush();
    } else {
        // MMAs may still be in flight: the TMEM is freed after them (a bounded wait)
        if (issuer) mmaCommit(&S.sumBar);
        mbarWait(&S.sumBar, sumPhase, abortFlag, L0.err, 56);
        __syncthreads();
    }
    if (tid == 0) {
        if (S.refined) atomicAdd(lv.refined, (unsigned long long)S.refined);
        if (S.visited) atomicAdd(lv.refined + 1, (unsigned long long)S.visited);
    }
    if (warp == 0) {
        tcFenceAfter();
        tmemDealloc(tmem, kAxTmemCols);
    }
}

// ------------------------------------------------------------------ update
__global__ void __launch_bounds__(256) updateKernelF(KMeansLevelF lv)
{
    __shared__ uint32_t ch, ran;
    __shared__ uint32_t cnt[kMaxBranch];
    __shared__ double term[kMaxBranch];
    __shared__ float red[kMaxBranch];
    const KMeansLevel& L0 = lv.base;
    const uint32_t g = blockIdx.x, t = threadIdx.x, B = L0.B;
    if (t == 0) {
        const uint32_t prev = L0.lastChanged[g];
        ch = L0.changed[g];
        ran = prev != 0 ? 1u : 0u; // the assign step visited this node
        L0.lastChanged[g] = ch;
        L0.changed[g] = 0;
        if (ch != 0) atomicAdd(L0.activeCount, 1u);
    }
    if (t < kMaxBranch) cnt[t] = L0.counts[uint64_t(g) * kMaxBranch + t];
    __syncthreads();
    // A node frozen before this step was skipped by the assign (ch is 0 then): nothing was
    // accumulated, every counter is zero and its inertia is that of its last assignment.
    if (!ran) return;
    float* c = lv.centers + uint64_t(g) * kMaxBranch * kDims;
    unsigned long long* sums = L0.sums + uint64_t(g) * kMaxBranch * kDims;
    unsigned long long* q = lv.q + uint64_t(g) * kMaxBranch;
    if (ran) {
        // inertia of the assignment just made, with the centers it was made against
        const uint32_t j = t / 16, part = t % 16;
        double cs = 0.0, cc = 0.0;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const uint32_t d = part * 8 + k;
            const double cv = double(c[j * kDims + d]);
            cs = __fma_rn(cv, double(sums[j * kDims + d]), cs);
            cc = __fma_rn(cv, cv, cc);
        }
#pragma unroll
        for (uint32_t off = 8; off > 0; off >>= 1) {
            cs = __dadd_rn(cs, __shfl_xor_sync(0xFFFFFFFFu, cs, off));
            cc = __dadd_rn(cc, __shfl_xor_sync(0xFFFFFFFFu, cc, off));
        }
        if (part == 0)
            term[j] = j < B ? __fma_rn(double(cnt[j]), cc, __fma_rn(-2.0, cs, double(q[j]))) : 0.0;
        __syncthreads();
        if (t == 0) {
            double s = 0.0;
            for (uint32_t b = 0; b < B; b++) s = __dadd_rn(s, term[b]);
            lv.inertiaNode[g] = s;
        }
    }
    __syncthreads();
    if (ch != 0) {
        for (uint32_t i = t; i < kMaxBranch * kDims; i += blockDim.x) {
            const uint32_t b = i / kDims;
            if (b < B && cnt[b] != 0) c[i] = __double2float_rn(__ddiv_rn(double(sums[i]), double(cnt[b])));
        }
    }
    for (uint32_t i = t; i < B * kDims; i += blockDim.x) sums[i] = 0ull; // centers b >= B have none
    __syncthreads();
    if (t < B) {
        L0.counts[uint64_t(g) * kMaxBranch + t] = 0;
        q[t] = 0ull;
    }
    if (ch != 0)
        prepareNode(c, lv.split + uint64_t(g) * kSplitBytes, lv.cn + uint64_t(g) * kMaxBranch, lv.bound + g, B, true, red);
}

__global__ void __launch_bounds__(1024) inertiaSumKernel(const double* in, uint32_t n, double* out)
{
    __shared__ double part[1024];
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < n; i += 1024) s = __dadd_rn(s, in[i]);
    part[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 512; off > 0; off >>= 1) {
        if (threadIdx.x < off) part[threadIdx.x] = __dadd_rn(part[threadIdx.x], part[threadIdx.x + off]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = part[0];
}

// ------------------------------------------------------------------ lookups
// Few descriptors: a warp per descriptor takes it through every level.  Lane l holds dims 4 l .. + 3 and
// sums (x - c)^2 over them in fp32 for every center; the 16 sums are reduced over the lanes together,
// each step halving the centers a lane keeps.  All terms are positive, so a distance is off by less
// than 2^-20 of itself (eleven roundings: the difference counts twice, then four products and five sums
// over the lanes), whatever the centers' length: unlike |c|^2 - 2 x.c it holds |x|^2, which for centers
// much shorter than the row is far more than kMarginScale's part.  Two distances within 2^-18 of the
// smaller one are therefore left to FP64 too, and what the squares of tiny differences lose by
// underflow (2^-142 over all dims) by the constant.
// Bound by the node reads (512 bytes per center, row and level).
constexpr uint32_t kDirectFThreads = 128;
__global__ void __launch_bounds__(kDirectFThreads) lookupDirectF(const float* __restrict__ centers,
                                                                 const float2* __restrict__ bound, uint32_t B,
                                                                 uint32_t L, const uint8_t* __restrict__ desc,
                                                                 uint64_t n, uint32_t* __restrict__ leaf,
                                                                 unsigned long long* refined)
{
    const uint64_t row = uint64_t(blockIdx.x) * (kDirectFThreads / 32) + threadIdx.x / 32;
    if (row >= n) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t xw = __ldg(reinterpret_cast<const uint32_t*>(desc + row * kDims) + lane);
    const float x0 = float(xw & 0xFFu), x1 = float((xw >> 8) & 0xFFu);
    const float x2 = float((xw >> 16) & 0xFFu), x3 = float(xw >> 24);
    const float xLen = __fsqrt_ru(float(__reduce_add_sync(0xFFFFFFFFu, __dp4a(xw, xw, 0u))));
    // the center whose distance this lane ends up with (two lanes hold each)
    const uint32_t mine = ((lane >> 4) & 1u) * 8u + ((lane >> 3) & 1u) * 4u + ((lane >> 2) & 1u) * 2u + ((lane >> 1) & 1u);
    uint64_t idx = 0, lb = 0;
    uint32_t settled = 0;
    for (uint32_t level = 0; level < L; level++) {
        const float* c = centers + (lb + idx) * kMaxBranch * kDims + 4u * lane;
        float acc[kMaxBranch];
#pragma unroll
        for (uint32_t b = 0; b < kMaxBranch; b++) {
            acc[b] = 1e30f;
            if (b < B) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(c + b * kDims));
                const float e0 = x0 - v.x, e1 = x1 - v.y, e2 = x2 - v.z, e3 = x3 - v.w;
                acc[b] = fmaf(e3, e3, fmaf(e2, e2, fmaf(e1, e1, e0 * e0)));
            }
        }
#pragma unroll
        for (uint32_t half = 8; half >= 1; half >>= 1) {
            const bool up = (lane & (2u * half)) != 0;
#pragma unroll
            for (uint32_t b = 0; b < half; b++) {
                const float give = up ? acc[b] : acc[b + half];
                acc[b] = (up ? acc[b + half] : acc[b]) + __shfl_xor_sync(0xFFFFFFFFu, give, 2u * half);
            }
        }
        const float dist = acc[0] + __shfl_xor_sync(0xFFFFFFFFu, acc[0], 1);
        // non-negative floats order like their bits
        const uint32_t bits = __float_as_uint(dist);
        const uint32_t least = __reduce_min_sync(0xFFFFFFFFu, bits);
        uint32_t bi = __reduce_min_sync(0xFFFFFFFFu, bits == least ? mine : kMaxBranch);
        const uint32_t next = __reduce_min_sync(0xFFFFFFFFu, mine == bi ? 0x7F800000u : bits);
        const float best = __uint_as_float(least);
        const float2 bnd = __ldg(bound + lb + idx);
        const float thr = __fmaf_rn(kMarginScale, __fmaf_rn(xLen, bnd.x, bnd.y), __fmaf_rn(best, 0x1p-18f, 0x1p-100f));
        if (!(__uint_as_float(next) - best > thr)) {
            const uint32_t near = __reduce_or_sync(0xFFFFFFFFu, mine < B && !(dist - best > thr) ? 1u << mine : 0u);
            bi = nearestFp64(c, near, double(x0), double(x1), double(x2), double(x3));
            settled++;
        }
        idx = idx * B + bi;
        lb = lb * B + 1;
    }
    if (lane == 0) {
        leaf[row] = static_cast<uint32_t>(idx);
        if (settled) atomicAdd(refined, (unsigned long long)settled);
        atomicAdd(refined + 1, (unsigned long long)L);
    }
}

// More descriptors: per level one assign launch (which also counts the children), one scan of the
// counts, and one launch that moves the members to their children and lists the next level's tiles.
// The order of a node's members does not matter to a lookup, so a warp takes its slots from the
// children's cursors.
__global__ void lookupInitKernel(uint32_t n, uint32_t* members, uint32_t* nodeCnt, uint32_t* nodeOff, NodeTile* tiles,
                                 uint32_t* totals, uint32_t* counts)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) members[i] = i;
    const uint32_t T = (n + 127) / 128;
    if (i < T) tiles[i] = NodeTile{0u, i * 128u, min(128u, n - i * 128u), 0u};
    if (i < kMaxBranch) counts[i] = 0;
    if (i == 0) {
        nodeCnt[0] = n;
        nodeOff[0] = 0;
        totals[0] = T;
    }
}

constexpr uint32_t kLookupScanChildren = 32768; // one CTA scans this many
__global__ void __launch_bounds__(1024) lookupScanKernel(const uint32_t* counts, uint32_t nbNodes, uint32_t B,
                                                         uint32_t* childCnt, uint32_t* childOff, uint32_t* cursor,
                                                         uint32_t* tileOff, uint32_t* totals)
{
    __shared__ uint32_t wa[32], wb[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    const uint32_t nc = nbNodes * B, per = (nc + 1023) / 1024;
    const uint32_t c0 = min(nc, tid * per), c1 = min(nc, c0 + per);
    uint32_t a = 0, t = 0;
    for (uint32_t c = c0; c < c1; c++) {
        const uint32_t v = counts[(c / B) * kMaxBranch + c % B];
        a += v;
        t += (v + 127) / 128;
    }
    uint32_t ia = a, it = t;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t xa = __shfl_up_sync(0xFFFFFFFFu, ia, off), xt = __shfl_up_sync(0xFFFFFFFFu, it, off);
        if (lane >= off) {
            ia += xa;
            it += xt;
        }
    }
    if (lane == 31) {
        wa[w] = ia;
        wb[w] = it;
    }
    __syncthreads();
    if (w == 0) {
        uint32_t va = wa[lane], vb = wb[lane];
#pragma unroll
        for (uint32_t off = 1; off < 32; off <<= 1) {
            const uint32_t xa = __shfl_up_sync(0xFFFFFFFFu, va, off), xb = __shfl_up_sync(0xFFFFFFFFu, vb, off);
            if (lane >= off) {
                va += xa;
                vb += xb;
            }
        }
        wa[lane] = va;
        wb[lane] = vb;
    }
    __syncthreads();
    uint32_t ra = (w ? wa[w - 1] : 0u) + ia - a, rt = (w ? wb[w - 1] : 0u) + it - t;
    for (uint32_t c = c0; c < c1; c++) {
        const uint32_t v = counts[(c / B) * kMaxBranch + c % B];
        childCnt[c] = v;
        childOff[c] = ra;
        cursor[c] = ra;
        tileOff[c] = rt;
        ra += v;
        rt += (v + 127) / 128;
    }
    if (tid == 1023) totals[0] = wb[31];
}

// A CTA takes eight quarter tiles, a warp each, and the warps whose quarters belong to one node claim
// their places in its children together: one atomic per child, node and CTA.  With one per warp the
// ten cursors of the first level took 62,000 for 200,003 rows: the three levels' launches 24 us, 17 us
// now (17.5 with 16 warps; 23 with 32, of which an SM holds one).
constexpr uint32_t kMoveWarps = 8;
__global__ void __launch_bounds__(32 * kMoveWarps) lookupMoveKernel(KMeansLevel lv, const NodeTile* tiles, const uint32_t* nTiles,
                                                        uint32_t* cursor, uint32_t* childMembers,
                                                        const uint32_t* childCnt, const uint32_t* childOff,
                                                        const uint32_t* tileOff, const uint32_t* nextTotals,
                                                        NodeTile* nextTiles, uint32_t* nextCounts)
{
    const uint32_t lane = threadIdx.x & 31u, threads = gridDim.x * blockDim.x;
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x, nc = lv.nbNodes * lv.B;
    for (uint32_t i = gid; i < nc * kMaxBranch; i += threads) nextCounts[i] = 0;
    const uint32_t nt = *nextTotals;
    for (uint32_t t = gid; t < nt; t += threads) {
        uint32_t lo = 0, hi = nc; // the last child whose first tile is at most t
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (tileOff[mid] <= t) lo = mid + 1;
            else hi = mid;
        }
        const uint32_t g = lo - 1, k = t - tileOff[g];
        nextTiles[t] = NodeTile{g, childOff[g] + k * 128u, min(128u, childCnt[g] - k * 128u), tileOff[g]};
    }
    __shared__ uint32_t cnt[kMoveWarps][kMaxBranch]; // rows per child, then the first one's place
    __shared__ uint32_t node[kMoveWarps + 1];
    const uint32_t warp = threadIdx.x / 32;
    const uint32_t T4 = *nTiles * 4;
    for (uint32_t q0 = blockIdx.x * kMoveWarps; q0 < T4; q0 += gridDim.x * kMoveWarps) {
        const uint32_t q = q0 + warp;
        const NodeTile ti = q < T4 ? tiles[q / 4] : NodeTile{0xFFFFFFFFu, 0u, 0u, 0u};
        const uint32_t r = 32 * (q % 4) + lane;
        const bool valid = r < ti.count;
        const uint32_t b = valid ? lv.assign[uint64_t(ti.start) + r] : 0xFFu;
        const uint32_t member = valid ? lv.members[uint64_t(ti.start) + r] : 0u;
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, b);
        const uint32_t rank = __popc(same & ((1u << lane) - 1u));
        if (lane < kMaxBranch) cnt[warp][lane] = 0;
        if (lane == 0) node[warp] = ti.node;
        if (threadIdx.x == 0) node[kMoveWarps] = 0xFFFFFFFFu;
        __syncwarp();
        if (valid && rank == 0) cnt[warp][b] = __popc(same);
        __syncthreads();
        if (threadIdx.x < kMoveWarps * kMaxBranch) {
            const uint32_t w0 = threadIdx.x / kMaxBranch, c = threadIdx.x % kMaxBranch, g = node[w0];
            if (g != 0xFFFFFFFFu && c < lv.B && (w0 == 0 || node[w0 - 1] != g)) { // the first warp of the node
                uint32_t sum = 0;
                for (uint32_t w = w0; node[w] == g; w++) sum += cnt[w][c];
                uint32_t at = sum ? atomicAdd(cursor + g * lv.B + c, sum) : 0u;
                for (uint32_t w = w0; node[w] == g; w++) {
                    const uint32_t own = cnt[w][c];
                    cnt[w][c] = at;
                    at += own;
                }
            }
        }
        __syncthreads();
        if (valid) childMembers[cnt[warp][b] + rank] = member;
        __syncthreads(); // the tables are rewritten
    }
}

} // namespace

void launchCentersToFloat(const KMeansLevelF& lv, cudaStream_t s)
{
    if (lv.base.nbNodes == 0) return;
    centersToFloatKernel<<<lv.base.nbNodes, 256, 0, s>>>(lv);
    RBW_CUDA(cudaGetLastError());
}

void launchPrepareFloatNodes(const float* centers, uint8_t* split, float* cn, float2* bound, uint64_t nbNodes,
                             uint32_t B, bool limbs, cudaStream_t s)
{
    for (uint64_t off = 0; off < nbNodes; off += 0x7FFFFFFFull) {
        const uint64_t m = std::min<uint64_t>(nbNodes - off, 0x7FFFFFFFull);
        prepareNodesKernel<<<static_cast<uint32_t>(m), 256, 0, s>>>(centers + off * kMaxBranch * kDims,
                                                                     split + off * kSplitBytes, cn + off * kMaxBranch,
                                                                     bound + off, B, limbs);
        RBW_CUDA(cudaGetLastError());
    }
}

void launchAssignF(const KMeansLevelF& lv, const NodeTile* tiles, const uint32_t* nTilesDev, uint32_t maxTiles,
                   cudaStream_t s)
{
    static_assert(kAfCtasPerSm * kAfTmemCols <= 512 && kAxCtasPerSm * kAxTmemCols <= 512, "TMEM columns");
    static_assert(kAfCtasPerSm * kAfSmemBytes <= 227 * 1024, "shared memory of the resident CTAs");
    static_assert(kAxCtasPerSm * (kAxSmemBytes + 1024) <= 228 * 1024, "shared memory of the resident CTAs");
    static std::atomic<uint64_t> attrF{0}, attrX{0};
    const uint32_t tuned = tunedValue(kTuneAssignFCtasPerSm, lv.base.B, 0, lv.base.nbMembers);
    const uint32_t sms = static_cast<uint32_t>(currentSmCount());
    ScopedKernelTimer timer(kTimedAssign, s);
    if (lv.limbs) {
        const uint32_t perSm = std::min(kAxCtasPerSm, tuned);
        setMaxDynamicSmemOncePerDevice(reinterpret_cast<const void*>(assignKernelX), int(kAxSmemBytes), attrX);
        assignKernelX<<<std::max(1u, std::min(maxTiles, sms * perSm)), kAxThreads, kAxSmemBytes, s>>>(lv, tiles, nTilesDev);
    } else {
        if (lv.lookupOnly == 0) throw Error(kInternal, "builds use fixed-point centers");
        setMaxDynamicSmemOncePerDevice(reinterpret_cast<const void*>(assignKernelF), int(kAfSmemBytes), attrF);
        assignKernelF<<<std::max(1u, std::min(maxTiles, sms * std::min(kAfCtasPerSm, tuned))), kAfThreads, kAfSmemBytes,
                        s>>>(lv, tiles, nTilesDev);
    }
    RBW_CUDA(cudaGetLastError());
}

void launchUpdateF(const KMeansLevelF& lv, cudaStream_t s)
{
    if (lv.base.nbNodes == 0) return;
    ScopedKernelTimer timer(kTimedUpdate, s);
    updateKernelF<<<lv.base.nbNodes, 256, 0, s>>>(lv);
    RBW_CUDA(cudaGetLastError());
}

void launchInertiaSum(const double* inertiaNode, uint32_t nbNodes, double* out, cudaStream_t s)
{
    inertiaSumKernel<<<1, 1024, 0, s>>>(inertiaNode, nbNodes, out);
    RBW_CUDA(cudaGetLastError());
}

uint32_t launchLookupDirectF(const KMeansLevelF& tree, uint32_t L, uint64_t n, uint32_t* leaf, cudaStream_t s)
{
    const uint64_t perBlock = kDirectFThreads / 32;
    ScopedKernelTimer timer(kTimedAssign, s);
    lookupDirectF<<<static_cast<uint32_t>((n + perBlock - 1) / perBlock), kDirectFThreads, 0, s>>>(
        tree.centers, tree.bound, tree.base.B, L, tree.base.desc, n, leaf, tree.refined);
    RBW_CUDA(cudaGetLastError());
    return 1;
}

bool lookupCountsChildren(uint32_t B, uint32_t L) { return ipow(B, L - 1) <= kLookupScanChildren; }

void launchLookupInit(uint32_t n, const LookupLevel& lvl, uint32_t* members, cudaStream_t s)
{
    lookupInitKernel<<<std::max(1u, (n + 255) / 256), 256, 0, s>>>(n, members, lvl.nodeCnt, lvl.nodeOff, lvl.tiles,
                                                                  lvl.totals, lvl.counts);
    RBW_CUDA(cudaGetLastError());
}

void launchLookupNextLevel(const KMeansLevel& lv, const LookupLevel& from, const LookupLevel& to, uint32_t* cursor,
                           uint32_t* tileOff, uint32_t* childMembers, cudaStream_t s)
{
    lookupScanKernel<<<1, 1024, 0, s>>>(from.counts, lv.nbNodes, lv.B, to.nodeCnt, to.nodeOff, cursor, tileOff, to.totals);
    const uint64_t warps = lv.nbMembers / 32 + lv.nbNodes + 1;
    const uint32_t blocks = static_cast<uint32_t>(
        std::min<uint64_t>((warps + kMoveWarps - 1) / kMoveWarps, uint64_t(currentSmCount()) * (64 / kMoveWarps)));
    lookupMoveKernel<<<blocks, 32 * kMoveWarps, 0, s>>>(lv, from.tiles, from.totals, cursor, childMembers, to.nodeCnt, to.nodeOff,
                                            tileOff, to.totals, to.tiles, to.counts);
    RBW_CUDA(cudaGetLastError());
}

} // namespace rbw
