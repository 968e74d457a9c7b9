// Hierarchical k-means kernels.  Distances are exact integers: score_b = |c_b|^2 - 2 x.c_b with
// x.c_b from the tensor core (tcgen05.mma.kind::i8, u8 x u8 -> s32) in the assign step and from
// dp4a in k-means++, argmin with the lowest index on ties (kmeans.cu:131-135).
// Center sums are exact (s32 in tensor memory, u64 in global memory).
#include "kmeans.cuh"
#include "timing.h"
#include "tuning.h"

#include <algorithm>

namespace rbw {
namespace {

constexpr uint32_t kScanBlock = 1024;
constexpr uint32_t kScanPerThread = 4;
constexpr uint32_t kScanTile = kScanBlock * kScanPerThread;

__device__ __forceinline__ uint32_t blockExclusiveScan(uint32_t v, uint32_t* warpSums, uint32_t& total)
{
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warpSums[w] = x;
    __syncthreads();
    if (w == 0) {
        const uint32_t nw = blockDim.x / 32;
        uint32_t s = lane < nw ? warpSums[lane] : 0u;
#pragma unroll
        for (uint32_t off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, off);
            if (lane >= off) s += y;
        }
        warpSums[lane] = s;
    }
    __syncthreads();
    total = warpSums[blockDim.x / 32 - 1];
    const uint32_t r = (w ? warpSums[w - 1] : 0u) + x - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanBlock) scanBlockSums(const uint32_t* in, uint64_t n, uint32_t* blockSums)
{
    __shared__ uint32_t ws[32];
    const uint64_t base = uint64_t(blockIdx.x) * kScanTile + threadIdx.x * kScanPerThread;
    uint32_t s = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanPerThread; k++)
        if (base + k < n) s += in[base + k];
    uint32_t total;
    blockExclusiveScan(s, ws, total);
    if (threadIdx.x == 0) blockSums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanBlock) scanSingle(uint32_t* data, uint32_t n)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += kScanBlock) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < n ? data[i] : 0u;
        uint32_t total;
        const uint32_t e = blockExclusiveScan(v, ws, total);
        if (i < n) data[i] = e + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

// kOwnSums: blockOff holds the blocks' sums (at most kScanBlock of them), each block adds up those
// before it; else their scan.
template <bool kOwnSums>
__global__ void __launch_bounds__(kScanBlock) scanApply(const uint32_t* in, uint64_t n, const uint32_t* blockOff,
                                                        uint32_t* out)
{
    __shared__ uint32_t ws[32];
    uint32_t before = 0;
    if (kOwnSums) blockExclusiveScan(threadIdx.x < blockIdx.x ? blockOff[threadIdx.x] : 0u, ws, before);
    else before = blockOff[blockIdx.x];
    const uint64_t base = uint64_t(blockIdx.x) * kScanTile + threadIdx.x * kScanPerThread;
    uint32_t v[kScanPerThread];
    uint32_t s = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanPerThread; k++) {
        v[k] = base + k < n ? in[base + k] : 0u;
        s += v[k];
    }
    uint32_t total;
    uint32_t e = blockExclusiveScan(s, ws, total) + before;
#pragma unroll
    for (uint32_t k = 0; k < kScanPerThread; k++) {
        if (base + k < n) out[base + k] = e;
        e += v[k];
    }
}

__global__ void ceilDivKernel(const uint32_t* cnt, uint32_t n, uint32_t d, uint32_t* out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (cnt[i] + d - 1) / d;
}

__global__ void tilesTotal(const uint32_t* cnt, const uint32_t* tileOff, uint32_t n, uint32_t d, uint32_t* totals)
{
    if (n == 0) {
        totals[0] = 0;
        return;
    }
    totals[0] = tileOff[n - 1] + (cnt[n - 1] + d - 1) / d;
}

__global__ void fillNodeTiles(const uint32_t* cnt, const uint32_t* off, const uint32_t* tileOff, uint32_t nbNodes,
                              uint32_t d, const uint32_t* totals, uint32_t maxTiles, NodeTile* tiles)
{
    const uint32_t nTiles = totals[0];
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nTiles && t < maxTiles;
         t += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nbNodes;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (tileOff[mid] <= t) lo = mid + 1; else hi = mid;
        }
        const uint32_t g = lo - 1;
        const uint32_t k = t - tileOff[g];
        const uint32_t c = cnt[g] - k * d;
        tiles[t] = NodeTile{g, off[g] + k * d, c < d ? c : d, tileOff[g]};
    }
}

// The whole tile list in one launch where a CTA can scan the nodes' tile counts by itself: each does,
// then fills its share of the list; the first also writes the offsets and the total.
constexpr uint32_t kTileListNodes = kScanTile;
__global__ void __launch_bounds__(kScanBlock) nodeTilesKernel(const uint32_t* cnt, const uint32_t* off, uint32_t nbNodes,
                                                              uint32_t d, uint32_t maxTiles, uint32_t* tileOff,
                                                              uint32_t* totals, NodeTile* tiles)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t first[kTileListNodes];
    uint32_t v[kScanPerThread], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanPerThread; k++) {
        const uint32_t g = threadIdx.x * kScanPerThread + k;
        v[k] = g < nbNodes ? (cnt[g] + d - 1) / d : 0u;
        sum += v[k];
    }
    uint32_t total;
    uint32_t e = blockExclusiveScan(sum, ws, total);
#pragma unroll
    for (uint32_t k = 0; k < kScanPerThread; k++) {
        const uint32_t g = threadIdx.x * kScanPerThread + k;
        first[g] = e;
        if (blockIdx.x == 0 && g < nbNodes) tileOff[g] = e;
        e += v[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) totals[0] = total;
    __syncthreads();
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total && t < maxTiles; t += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nbNodes;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (first[mid] <= t) lo = mid + 1; else hi = mid;
        }
        const uint32_t g = lo - 1, k = t - first[g], c = cnt[g] - k * d;
        tiles[t] = NodeTile{g, off[g] + k * d, c < d ? c : d, first[g]};
    }
}

// ------------------------------------------------------------------ centers
__global__ void initCentersKernel(KMeansLevel lv, const uint32_t* pos, uint64_t nbDescTotal, int posIsDesc)
{
    // thread per (node, slot, 16-byte chunk)
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t total = uint64_t(lv.nbNodes) * kMaxBranch * 8;
    if (i >= total) return;
    const uint32_t chunk = i % 8;
    const uint32_t b = (i / 8) % kMaxBranch;
    const uint32_t g = static_cast<uint32_t>(i / (8 * kMaxBranch));
    uint4 v = make_uint4(0, 0, 0, 0);
    if (b < lv.B) {
        const uint32_t p = pos[uint64_t(g) * lv.B + b];
        const uint64_t at = posIsDesc ? uint64_t(p) : uint64_t(lv.nodeOff[g]) + p;
        if (p != kInvalidIdx && at < (posIsDesc ? nbDescTotal : lv.nbMembers)) {
            const uint32_t d = posIsDesc ? p : lv.members[at];
            v = reinterpret_cast<const uint4*>(lv.desc + uint64_t(d) * kDims)[chunk];
        } else {
            v = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        }
    }
    reinterpret_cast<uint4*>(lv.centers + (uint64_t(g) * kMaxBranch + b) * kDims)[chunk] = v;
}

__global__ void centerNormsKernel(KMeansLevel lv)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= uint64_t(lv.nbNodes) * kMaxBranch) return;
    const uint32_t b = i % kMaxBranch;
    if (b >= lv.B) {
        lv.cnorm[i] = kPadNorm;
        return;
    }
    const uint4* c = reinterpret_cast<const uint4*>(lv.centers + i * kDims);
    uint32_t acc = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint4 v = c[k];
        acc = __dp4a(v.x, v.x, acc);
        acc = __dp4a(v.y, v.y, acc);
        acc = __dp4a(v.z, v.z, acc);
        acc = __dp4a(v.w, v.w, acc);
    }
    lv.cnorm[i] = static_cast<int32_t>(acc);
}

// ------------------------------------------------------------------ k-means++ init
// SplitMix64 (Steele, Lea, Flood 2014): the output for state z; the generator adds
// kSplitMixGamma to the state before each output, so draw i (from 0) of a stream started at s
// is splitMixOut(s + (i + 1) * kSplitMixGamma).
constexpr uint64_t kSplitMixGamma = 0x9E3779B97F4A7C15ull;
__device__ __forceinline__ uint64_t splitMixOut(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t splitmix64(uint64_t& s)
{
    s += kSplitMixGamma;
    return splitMixOut(s);
}

constexpr uint32_t kPPSample = 256;
constexpr uint32_t kPPWarps = kPPSample / 32;
constexpr uint32_t kPPCtasPerSm = 6; // by shared memory: 32 KB of candidate rows per CTA

// One CTA (256 threads) per node.  Same specification as the oracle's orc_kmeanspp_init:
// SplitMix64 stream seeded by (seed, level, node); Floyd sampling of min(n, 256) member
// positions (sorted); first center uniform; then D^2 sampling with exact integer weights.
// Floyd's draws do not depend on the set, so thread m makes draw m, t_m = out_m % (j_m + 1) with
// j_m = n - 256 + m, directly from the counter-based stream.  Step m inserts j_m when t_m is
// already in the set, else t_m; with base = n - 256:
//   - t_m < base: t_m is in the set iff an earlier draw equals it (values below base enter only
//     as themselves, and the first equal draw did enter);
//   - t_m = base + m: not yet in the set (every earlier value is below j_m);
//   - t_m = j_r, r < m: in the set iff step r inserted j_r (found_r) or a draw t_q, r <= q < m,
//     equals it;
// so found_m = local_m || found_r along links m -> r < m, an OR over a chain of at most 256
// steps, resolved by eight rounds of pointer jumping.  The distinct positions are then sorted by
// rank (each thread counts the smaller ones).  The candidate rows sit in shared memory and thread
// i holds candidate i's D^2 weight; each pick's prefix sums are warp scans plus one pass over the
// eight warp totals, and every thread draws the same random numbers, so a pick costs two
// barriers.  Registers stay low enough for six CTAs per SM (deep levels have 10^5 nodes).
//
// Distances are |x|^2 + |p|^2 - 2 x.p by dp4a (exact), each row's norm taken once.
struct PPSmem {
    // candidate rows, chunk c of row i at [i][c ^ (i & 7)] (a quarter-warp reading its own rows
    // hits 32 different banks)
    uint4 rowS[kPPSample][kDims / 16];
    uint32_t pos[kPPSample];
    uint32_t cand[kPPSample];
    uint32_t draw[kPPSample]; // later the rows' |x|^2
    uint32_t link[kPPSample];
    uint8_t found[kPPSample];
    uint32_t warpSum[kPPWarps];
    uint32_t chosen[kMaxBranch];
};
__device__ __forceinline__ uint32_t dot16(const uint4& x, const uint4& y, uint32_t acc)
{
    return __dp4a(x.w, y.w, __dp4a(x.z, y.z, __dp4a(x.y, y.y, __dp4a(x.x, y.x, acc))));
}

__device__ __forceinline__ void kmeansPPNode(const KMeansLevel& lv, uint64_t seed, uint32_t level, uint32_t g,
                                             uint32_t* nValidOut, PPSmem& sm)
{
    auto& rowS = sm.rowS;
    auto& pos = sm.pos;
    auto& cand = sm.cand;
    auto& draw = sm.draw;
    auto& link = sm.link;
    auto& found = sm.found;
    auto& warpSum = sm.warpSum;
    auto& chosen = sm.chosen;
    const uint32_t n = lv.nodeCnt[g];
    const uint32_t tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const uint32_t S = n < kPPSample ? n : kPPSample;
    if (n == 0) {
        if (tid == 0) nValidOut[g] = 0;
        for (uint32_t i = tid; i < kMaxBranch * 8; i += blockDim.x) {
            reinterpret_cast<uint4*>(lv.centers + uint64_t(g) * kMaxBranch * kDims)[i] =
                make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        }
        return;
    }
    uint64_t s = seed ^ (uint64_t(level) * 0x9E3779B97F4A7C15ull) ^ (uint64_t(g) * 0xD1B54A32D192ED03ull);
    if (n > kPPSample) {
        constexpr uint32_t kNone = 0xFFFFFFFFu;
        const uint32_t base = n - kPPSample;
        const uint32_t t = static_cast<uint32_t>(splitMixOut(s + uint64_t(tid + 1) * kSplitMixGamma) %
                                                 (uint64_t(base) + tid + 1));
        draw[tid] = t;
        __syncthreads();
        bool f = false;
        uint32_t lk = kNone, q0 = 0;
        if (t >= base) {
            const uint32_t r = t - base;
            q0 = r < tid ? r : tid; // r == tid: nothing to compare, no link
            if (r < tid) lk = r;
        }
        for (uint32_t q = q0; q < tid; q++) f |= draw[q] == t;
        found[tid] = f ? 1 : 0;
        link[tid] = lk;
        __syncthreads();
#pragma unroll 1
        for (uint32_t round = 0; round < 8; round++) {
            bool nf = f;
            uint32_t nl = lk;
            if (lk != kNone) {
                nf = f || found[lk] != 0;
                nl = link[lk];
            }
            __syncthreads();
            f = nf;
            lk = nl;
            found[tid] = f ? 1 : 0;
            link[tid] = lk;
            __syncthreads();
        }
        pos[tid] = f ? base + tid : t;
        s += uint64_t(kPPSample) * kSplitMixGamma; // the stream after the 256 draws
        __syncthreads();
        // ascending order: the positions are distinct, so each one's rank is its slot
        const uint32_t v = pos[tid];
        uint32_t rk = 0;
#pragma unroll 4
        for (uint32_t q = 0; q < kPPSample / 4; q++) {
            const uint4 x = reinterpret_cast<const uint4*>(pos)[q];
            rk += (x.x < v ? 1u : 0u) + (x.y < v ? 1u : 0u) + (x.z < v ? 1u : 0u) + (x.w < v ? 1u : 0u);
        }
        cand[rk] = lv.members[lv.nodeOff[g] + v];
    } else if (tid < S) {
        cand[tid] = lv.members[lv.nodeOff[g] + tid];
    }
    __syncthreads();
    const bool mine = tid < S;
    // eight threads per row, 32 rows per round
#pragma unroll
    for (uint32_t k = 0; k < kPPSample / 32; k++) {
        const uint32_t r = 32u * k + tid / 8, c = tid % 8;
        if (r < S) rowS[r][c ^ (r & 7u)] = reinterpret_cast<const uint4*>(lv.desc + uint64_t(cand[r]) * kDims)[c];
    }
    const uint32_t pick = static_cast<uint32_t>(splitmix64(s) % S);
    if (tid == 0) chosen[0] = pick;
    __syncthreads();
    uint32_t norm = 0;
    if (mine) {
#pragma unroll
        for (uint32_t c = 0; c < kDims / 16; c++) norm = dot16(rowS[tid][c ^ (tid & 7u)], rowS[tid][c ^ (tid & 7u)], norm);
    }
    draw[tid] = norm;
    __syncthreads();
    // the squared distance of this thread's row to row p
    auto distTo = [&](uint32_t p) -> uint32_t {
        uint32_t dot = 0;
#pragma unroll
        for (uint32_t c = 0; c < kDims / 16; c++) dot = dot16(rowS[tid][c ^ (tid & 7u)], rowS[p][c ^ (p & 7u)], dot);
        return norm + draw[p] - 2 * dot;
    };
    uint32_t d2 = mine ? distTo(pick) : 0u;
    uint32_t nv = 1;
    for (uint32_t k = 1; k < lv.B; k++) {
        // inclusive prefix of d2 over the candidates: warp scan, then the earlier warps' totals
        uint32_t incl = d2;
#pragma unroll
        for (uint32_t off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += v;
        }
        if (lane == 31) warpSum[warp] = incl;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < kPPWarps; w++) {
            const uint32_t v = warpSum[w];
            before += w < warp ? v : 0u;
            total += v;
        }
        if (total == 0) break; // uniform across the CTA
        incl += before;
        const uint32_t t = static_cast<uint32_t>(splitmix64(s) % total);
        // smallest i with prefix[i] > t: exactly one candidate has prefix > t >= prefix - d2
        const bool hit = mine && incl > t && incl - d2 <= t;
        if (hit) chosen[k] = tid;
        nv = k + 1;
        __syncthreads();
        if (mine) {
            d2 = min(d2, distTo(chosen[k]));
        }
        __syncthreads(); // warpSum is rewritten by the next pick
    }
    if (tid == 0) nValidOut[g] = nv;
    for (uint32_t i = tid; i < kMaxBranch * 8; i += blockDim.x) {
        const uint32_t b = i / 8, chunk = i % 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (b < lv.B) {
            const uint32_t c = cand[chosen[b < nv ? b : nv - 1]];
            v = reinterpret_cast<const uint4*>(lv.desc + uint64_t(c) * kDims)[chunk];
        }
        reinterpret_cast<uint4*>(lv.centers + (uint64_t(g) * kMaxBranch + b) * kDims)[chunk] = v;
    }
}

// list: nullptr (every node), or a count and the nodes to take.
__global__ void __launch_bounds__(kPPSample, kPPCtasPerSm) kmeansPPKernel(KMeansLevel lv, uint64_t seed, uint32_t level,
                                                                          const uint32_t* list, uint32_t* nValidOut)
{
    __shared__ PPSmem sm;
    if (list == nullptr) {
        kmeansPPNode(lv, seed, level, blockIdx.x, nValidOut, sm);
        return;
    }
    const uint32_t count = list[0];
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        kmeansPPNode(lv, seed, level, list[1 + i], nValidOut, sm);
        __syncthreads();
    }
}

// A warp per node for nodes of at most kPPSmall members, the larger ones listed for kmeansPPKernel.
// The same specification; lane l holds candidates l, l + 32, ..  Bound by instructions, like the kernel
// above, whose eight warps all run the picks' scans, divisions and barriers for a hundred rows.  100,000
// nodes of 100 members on average, B = 10: 2,400 us there, 540 us here and 850 us there for the quarter
// with more than 128 (a warp per node of 256 candidates has too little shared memory to share an SM: no
// faster).
constexpr uint32_t kPPSmall = 128;
constexpr uint32_t kPPSmallNodes = 1024;
constexpr uint32_t kPer = kPPSmall / 32; // candidates of a lane
static_assert(uint64_t(kPPSample) * kDims * 255 * 255 < (uint64_t(1) << 32), "sums of the weights fit 32 bits");
__global__ void __launch_bounds__(32) kmeansPPSmallKernel(KMeansLevel lv, uint64_t seed, uint32_t level, uint32_t* list,
                                                          uint32_t* nValidOut)
{
    __shared__ uint4 rowS[kPPSmall][kDims / 16]; // as in PPSmem
    const uint32_t g = blockIdx.x, lane = threadIdx.x;
    const uint32_t n = lv.nodeCnt[g];
    uint4* centers = reinterpret_cast<uint4*>(lv.centers + uint64_t(g) * kMaxBranch * kDims);
    if (n > kPPSmall) {
        if (lane == 0) list[1 + atomicAdd(list, 1u)] = g;
        return;
    }
    if (n == 0) {
        if (lane == 0) nValidOut[g] = 0;
        for (uint32_t i = lane; i < kMaxBranch * 8; i += 32)
            centers[i] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        return;
    }
    uint32_t m[kPer];
#pragma unroll
    for (uint32_t j = 0; j < kPer; j++) {
        const uint32_t r = 32 * j + lane;
        m[j] = r < n ? lv.members[lv.nodeOff[g] + r] : 0u;
    }
    // eight lanes per row
#pragma unroll
    for (uint32_t j = 0; j < kPer; j++) {
        if (32 * j >= n) break; // uniform
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            const uint32_t r = 32 * j + 4 * k + lane / 8, c = lane % 8;
            const uint32_t id = __shfl_sync(0xFFFFFFFFu, m[j], 4 * k + lane / 8);
            if (r < n) cpAsync16(&rowS[r][c ^ (r & 7u)], lv.desc + uint64_t(id) * kDims + (c << 4));
        }
    }
    cpAsyncCommit();
    uint64_t s = seed ^ (uint64_t(level) * 0x9E3779B97F4A7C15ull) ^ (uint64_t(g) * 0xD1B54A32D192ED03ull);
    uint32_t pick = static_cast<uint32_t>(splitmix64(s) % n);
    cpAsyncWait<0>();
    __syncwarp();
    uint32_t norm[kPer], d2[kPer];
#pragma unroll
    for (uint32_t j = 0; j < kPer; j++) {
        const uint32_t r = 32 * j + lane;
        norm[j] = 0;
        if (r < n) {
#pragma unroll
            for (uint32_t c = 0; c < kDims / 16; c++) norm[j] = dot16(rowS[r][c ^ (r & 7u)], rowS[r][c ^ (r & 7u)], norm[j]);
        }
        d2[j] = r < n ? 0xFFFFFFFFu : 0u;
    }
    uint32_t mine = 0, nv = 0; // lane k: the k-th pick
    for (uint32_t k = 0;; k++) {
        if (lane == k) mine = pick;
        nv = k + 1;
        if (nv == lv.B) break;
        // weights against the pick, their sums per 32 candidates
        uint32_t pn = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) pn = pick / 32 == j ? norm[j] : pn;
        pn = __shfl_sync(0xFFFFFFFFu, pn, pick % 32);
        uint4 p[kDims / 16];
#pragma unroll
        for (uint32_t c = 0; c < kDims / 16; c++) p[c] = rowS[pick][c ^ (pick & 7u)];
        uint32_t incl[kPer], total = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) {
            const uint32_t r = 32 * j + lane;
            if (r < n) {
                uint32_t dot = 0;
#pragma unroll
                for (uint32_t c = 0; c < kDims / 16; c++) dot = dot16(rowS[r][c ^ (r & 7u)], p[c], dot);
                d2[j] = min(d2[j], norm[j] + pn - 2 * dot);
            }
            incl[j] = d2[j];
            if (32 * j < n) { // uniform
#pragma unroll
                for (uint32_t off = 1; off < 32; off <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl[j], off);
                    if (lane >= off) incl[j] += v;
                }
            }
            incl[j] += total;
            total = __shfl_sync(0xFFFFFFFFu, incl[j], 31);
        }
        if (total == 0) break; // uniform
        const uint32_t t = static_cast<uint32_t>(splitmix64(s) % total);
        // smallest candidate with prefix > t: exactly one has prefix > t >= prefix - d2
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) {
            const uint32_t hit = __ballot_sync(0xFFFFFFFFu, incl[j] > t && incl[j] - d2[j] <= t);
            if (hit) pick = 32 * j + __ffs(hit) - 1;
        }
    }
    if (lane == 0) nValidOut[g] = nv;
#pragma unroll
    for (uint32_t i = 0; i < kMaxBranch * 8 / 32; i++) {
        const uint32_t b = 4 * i + lane / 8, chunk = lane % 8;
        const uint32_t c = __shfl_sync(0xFFFFFFFFu, mine, b < nv ? b : nv - 1);
        centers[32 * i + lane] = b < lv.B ? rowS[c][chunk ^ (c & 7u)] : make_uint4(0, 0, 0, 0);
    }
}

// ------------------------------------------------------------------ assign
// One step handles one 128-member tile of one node (the reference's DescTile groups,
// kmeans.cu:62-211), both contractions on the tensor core:
//   1. the members' rows are gathered into shared memory in the 128-byte swizzled layout (eight
//      threads per row), next to the node's 16 centers in the same layout;
//   2. distances: one thread issues four tcgen05.mma.kind::i8 (M = 128 members, N = 16 centers,
//      K = 4 x 32 dims, u8 x u8 -> s32, exact) into TMEM columns [0, 16); warp w reads rows
//      32 w .. 32 w + 31 and takes the argmin of |c_b|^2 - 2 x.c_b, lowest index on ties
//      (kmeans.cu:131-135);
//   3. center sums: D[dim][center] += X[member][dim] * OH[member][center] over the tile's
//      members, four more MMAs (M = 128 dims, N = 16, K = 4 x 32 members) into columns [16, 32),
//      accumulated over the node's tiles in this CTA.  X is the gathered tile as it lies (read
//      MN-major: K = members), OH one 16-byte row per member, a single 1 at its center (zeros
//      for rows past the tile's count).
// Counts, change counts and sums go to global memory when the CTA moves to another node (or every
// kAssignFlushTiles tiles, which keeps each s32 below 2^31: 65,536 x 128 x 255 < 2^31).
//
// A tile costs the SM 8 x 45 cycles of tensor pipe and its 16 KB of gathered rows, which is more
// (0.37 us per tile at HBM speed); the wait -> MMA -> read -> MMA chain of a tile (~1 us) is hidden
// by five CTAs per SM, each gathering its next tile while one is scored.  10M members, B = 10: 0.22 ms
// per step against 0.20 ms to read the rows (0.30 ms where the nodes are small and their sums as many
// bytes as the rows: those stay on chip, see kmeans_lloyd.cu).  The 60 steps of a build took 39.6 ms with
// the sums by shared atomics (128 per member), 35.3 ms by MMAs over a tile transposed in shared
// memory, 18.2 ms with these.
constexpr uint32_t kAssignThreads = 128;
constexpr uint32_t kAssignRows = 128;
constexpr uint32_t kAssignTmemCols = 32; // the smallest allocation: distances | sums
constexpr uint32_t kAssignCtasPerSm = 5; // by shared memory (~40 KB each)
constexpr uint32_t kAssignFlushTiles = 65536;
constexpr uint32_t kTileWindow = kAssignThreads; // one tile entry per thread per refill
constexpr uint32_t kTileFrozen = 0x80000000u;

struct AssignSmem {
    uint8_t tile[2][kAssignRows * kDims]; // member rows, 128-byte swizzle (1024-byte aligned)
    uint8_t cen[kMaxBranch * kDims];      // node centers, same layout
    uint8_t oh[kAssignRows * kMaxBranch]; // [member][center] one-hot
    NodeTile win[kTileWindow];            // tiles [winBase, winBase + kTileWindow) of the CTA's
                                          // range, count | kTileFrozen for a frozen node
    int32_t cnk[kMaxBranch];              // 16 |c_b|^2 + b, INT_MAX for padding slots
    uint32_t cnt[kMaxBranch];
    uint64_t mmaBar, sumBar;
    uint32_t tmemBase;
    uint32_t chg;
    uint32_t abortFlag;
};
constexpr size_t kAssignSmemBytes = sizeof(AssignSmem) + 1024;

__global__ void __launch_bounds__(kAssignThreads, kAssignCtasPerSm) assignKernel(KMeansLevel lv, const NodeTile* tiles,
                                                                  const uint32_t* nTilesDev)
{
    extern __shared__ uint8_t smemRaw[];
    AssignSmem& S = *reinterpret_cast<AssignSmem*>(smemAligned(smemRaw));
    const uint32_t tid = threadIdx.x, lane = tid % 32;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, tid / 32, 0); // uniform
    const uint32_t T = *nTilesDev;
    const uint32_t t0 = static_cast<uint32_t>(uint64_t(T) * blockIdx.x / gridDim.x);
    const uint32_t t1 = static_cast<uint32_t>(uint64_t(T) * (blockIdx.x + 1) / gridDim.x);
    if (lv.activeCount && blockIdx.x == 0 && tid == 0) *lv.activeCount = 0; // counted by the update that follows
    if (t0 == t1) return; // uniform: fewer tiles than CTAs
    volatile uint32_t* abortFlag = &S.abortFlag;
    if (tid == 0) {
        mbarInit(&S.mmaBar, 1);
        mbarInit(&S.sumBar, 1);
        S.abortFlag = 0;
        fenceMbarInit();
    }
    if (warp == 0) {
        tmemAlloc(&S.tmemBase, kAssignTmemCols);
        tmemRelinquish();
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmem = S.tmemBase;
    const bool issuer = warp == 0 && electOne(); // one thread issues and commits every MMA
    uint32_t curNode = 0xFFFFFFFFu, phase = 0, sumPhase = 0, accTiles = 0, buf = 0;
    uint32_t myCnt = 0, myChg = 0; // lane c < 16: members of this warp's rows that chose center c
    bool curExclusive = false;     // every tile of the current node is in this CTA's range
    bool ok = true;
    // The tile list and the frozen flags are read a window of kTileWindow tiles at a time (one
    // load per thread, all in flight together), so that finding the next live tile costs no
    // global round trip; the member indices of the next tile are loaded into registers one
    // tile ahead of its row copies.  Every thread runs the same window refills (uniform).
    uint32_t winBase = t0;
    auto refill = [&](uint32_t base) {
        __syncthreads(); // nobody reads the old window any more
        if (base + tid < t1) {
            NodeTile x = tiles[base + tid];
            if (lv.lastChanged[x.node] == 0) x.count |= kTileFrozen; // frozen node (kmeans.cu:238-240)
            S.win[tid] = x;
        }
        winBase = base;
        __syncthreads();
    };
    auto entry = [&](uint32_t t) -> NodeTile {
        if (t - winBase >= kTileWindow) refill(t);
        return S.win[t - winBase];
    };
    // the first live tile at or after t, or t1
    auto nextLive = [&](uint32_t t) -> uint32_t {
        for (; t < t1; t++)
            if (!(entry(t).count & kTileFrozen)) return t;
        return t1;
    };
    auto loadIndices = [&](const NodeTile& tn, uint32_t (&m)[kAssignRows / 16]) {
#pragma unroll
        for (uint32_t k = 0; k < kAssignRows / 16; k++) {
            const uint32_t row = 16u * k + tid / 8;
            m[k] = lv.members[uint64_t(tn.start) + (row < tn.count ? row : 0u)];
        }
    };
    // eight threads per row, 16 rows per round; rows past the tile's count repeat its first
    // member (their results are not used); one copy group per tile
    auto gatherRows = [&](const uint32_t (&m)[kAssignRows / 16], uint32_t b) {
        const uint32_t c = tid % 8;
#pragma unroll
        for (uint32_t k = 0; k < kAssignRows / 16; k++) {
            const uint32_t row = 16u * k + tid / 8;
            cpAsync16(S.tile[b] + row * kDims + ((c ^ (row & 7u)) << 4), lv.desc + uint64_t(m[k]) * kDims + (c << 4));
        }
        cpAsyncCommit();
    };
    // writes the node's partial sums (TMEM), counts and change count
    auto flush = [&]() {
        if (curNode != 0xFFFFFFFFu) {
            if (lane < kMaxBranch && myCnt) atomicAdd(&S.cnt[lane], myCnt);
            if (lane == 0 && myChg) atomicAdd(&S.chg, myChg);
            if (accTiles > 0) {
                // nothing was committed yet for the last sums MMA
                if (issuer) mmaCommit(&S.sumBar);
                ok = ok && mbarWait(&S.sumBar, sumPhase, abortFlag, lv.err, 42);
                sumPhase ^= 1u;
                tcFenceAfter();
                uint32_t r[16];
                tmemLoad16(tmem + 16u + ((warp * 32u) << 16), r); // lane = dimension tid
                tmemWaitTie(r);
                tcFenceBefore();
                // A node no other CTA touches in this launch is written with plain stores (its
                // global accumulators are zero on entry); a shared node is added atomically.
#pragma unroll
                for (uint32_t b = 0; b < kMaxBranch; b++) {
                    if (r[b] == 0) continue;
                    unsigned long long* dst = lv.sums + (uint64_t(curNode) * kMaxBranch + b) * kDims + tid;
                    if (curExclusive) *dst = r[b];
                    else atomicAdd(dst, (unsigned long long)r[b]);
                }
            }
            __syncthreads(); // S.cnt and S.chg complete
            if (tid < kMaxBranch && S.cnt[tid]) {
                uint32_t* dst = lv.counts + uint64_t(curNode) * kMaxBranch + tid;
                if (curExclusive) *dst = S.cnt[tid];
                else atomicAdd(dst, S.cnt[tid]);
            }
            if (tid == 0 && S.chg) {
                if (curExclusive) lv.changed[curNode] = S.chg;
                else atomicAdd(lv.changed + curNode, S.chg);
            }
        }
        accTiles = 0;
        myCnt = 0;
        myChg = 0;
        __syncthreads();
    };
    refill(t0);
    uint32_t t = nextLive(t0);
    NodeTile ti{}, tn1{};
    uint32_t mNext[kAssignRows / 16];
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
        if (ti.node != curNode) {
            flush();
            curNode = ti.node;
            curExclusive = ti.first >= t0 && uint64_t(ti.first) + (lv.nodeCnt[curNode] + kAssignRows - 1) / kAssignRows <= t1;
            {
                // thread i copies chunk i % 8 of center i / 8 (16 centers x 8 chunks)
                const uint32_t b = tid / 8, c = tid % 8;
                const uint4 v = reinterpret_cast<const uint4*>(lv.centers + (uint64_t(curNode) * kMaxBranch + b) * kDims)[c];
                *reinterpret_cast<uint4*>(S.cen + b * kDims + ((c ^ (b & 7u)) << 4)) = v;
            }
            if (tid < kMaxBranch) {
                S.cnk[tid] = tid < lv.B ? lv.cnorm[uint64_t(curNode) * kMaxBranch + tid] * 16 + int32_t(tid) : 0x7FFFFFFF;
                S.cnt[tid] = 0;
            }
            if (tid == 0) S.chg = 0;
        } else if (accTiles == kAssignFlushTiles) {
            // keep each s32 sum below 2^31: add this node's partial results to global memory and
            // go on from zero (its later flushes add too)
            curExclusive = false;
            flush();
            if (tid < kMaxBranch) S.cnt[tid] = 0;
            if (tid == 0) S.chg = 0;
        }
        const uint32_t row = tid; // warp w reads TMEM lanes 32w .. 32w + 31
        const bool valid = row < ti.count;
        const uint64_t at = uint64_t(ti.start) + row;
        const uint32_t prevAssign = valid ? lv.assign[at] : 0u;
        cpAsyncWait<0>(); // this tile's rows
        // the copies, the center stores and the one-hot rows are generic-proxy writes read by the
        // tensor core
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            tcFenceAfter();
            mmaU8x4(issuer, tmem, smemDescSw128(smemAddr(S.tile[buf])), 32u, smemDescSw128(smemAddr(S.cen)), 32u,
                    idescU8(16), 0u);
            if (issuer) mmaCommit(&S.mmaBar);
        }
        if (!mbarWait(&S.mmaBar, phase, abortFlag, lv.err, 41)) {
            ok = false;
            break;
        }
        phase ^= 1u;
        tcFenceAfter();
        // The commit also covers the previous tile's sums MMAs: the other tile buffer and the
        // one-hot rows are free.  The next live tile's rows go into that buffer (its indices were
        // loaded one tile ago), the indices of the one after it into registers.
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
        uint32_t r[16];
        tmemLoad16(tmem + ((warp * 32u) << 16), r);
        tmemWaitTie(r);
        tcFenceBefore(); // the next tile's MMA overwrites these columns after the barriers below
        // |c|^2 - 2 x.c lies in (-2^24, 2^23]: 16 times it plus the center fits 32 bits, and the
        // minimum is the lowest center of the lowest score
        int32_t best = 0x7FFFFFFF;
#pragma unroll
        for (uint32_t b = 0; b < kMaxBranch; b++) best = min(best, S.cnk[b] - 32 * static_cast<int32_t>(r[b]));
        const uint32_t bi = static_cast<uint32_t>(best) & 15u;
        if (valid) lv.assign[at] = static_cast<uint8_t>(bi);
        {
            const uint32_t word = valid ? 1u << (8u * (bi & 3u)) : 0u;
            const uint32_t q = bi >> 2;
            *reinterpret_cast<uint4*>(S.oh + row * kMaxBranch) =
                make_uint4(q == 0 ? word : 0u, q == 1 ? word : 0u, q == 2 ? word : 0u, q == 3 ? word : 0u);
        }
        {
            const uint32_t live = __ballot_sync(0xFFFFFFFFu, valid);
            uint32_t mask = live;
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t bits = __ballot_sync(0xFFFFFFFFu, (bi >> k) & 1u);
                mask &= (lane >> k) & 1u ? bits : ~bits;
            }
            myCnt += __popc(mask); // used of lanes below kMaxBranch
            myChg += __popc(__ballot_sync(0xFFFFFFFFu, valid && prevAssign != bi));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads(); // every row's one-hot is in, every warp has read its distances
        if (warp == 0) {
            tcFenceAfter();
            mmaU8x4(issuer, tmem + 16u, smemDescSw128(smemAddr(S.tile[buf])), 4096u, smemDescMn16(smemAddr(S.oh)), 512u,
                    idescU8(16) | kIdescMnMajorAB, accTiles);
        }
        accTiles++;
        buf ^= 1u;
        t = n1;
        ti = tn1;
        n1 = n2;
        tn1 = tn2;
    }
    cpAsyncWait<0>(); // a prefetch of a tile that was not scored (abort) must land before exit
    if (ok) {
        flush();
    } else {
        // MMAs may still be in flight: the TMEM is freed after them (a bounded wait)
        if (issuer) mmaCommit(&S.sumBar);
        mbarWait(&S.sumBar, sumPhase, abortFlag, lv.err, 43);
        __syncthreads();
    }
    if (warp == 0) {
        tcFenceAfter();
        tmemDealloc(tmem, kAssignTmemCols);
    }
}

// ------------------------------------------------------------------ regroup
constexpr uint32_t kRegroupRows = 32;

__global__ void regroupHistKernel(KMeansLevel lv, const NodeTile* tiles, const uint32_t* nTilesDev, uint32_t maxTiles,
                                  uint32_t* tileHist)
{
    // warp per 32-member tile: lane q < B writes how many members chose center q
    const uint32_t T = *nTilesDev;
    const uint32_t warpsTotal = gridDim.x * (blockDim.x / 32);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t t = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; t < T; t += warpsTotal) {
        const NodeTile ti = tiles[t];
        const uint32_t b = lane < ti.count ? lv.assign[ti.start + lane] : 0xFFu;
        uint32_t c = 0;
        for (uint32_t q = 0; q < lv.B; q++) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, b == q);
            if (lane == q) c = __popc(m);
        }
        if (lane < lv.B) tileHist[uint64_t(lane) * maxTiles + t] = c;
    }
}

// Warp per 32-member tile.  A node's children lie in center order from its own offset
// (Vocabulary.cpp:83-98): lane q takes the size of child q from the scan over the node's tiles (of
// which only differences within a row are used), a scan over the lanes gives their offsets, and the
// warp of a node's first tile writes both.
__global__ void regroupScatterKernel(KMeansLevel lv, const NodeTile* tiles, const uint32_t* nTilesDev,
                                     uint32_t maxTiles, const uint32_t* tileHist, const uint32_t* tileScan,
                                     uint32_t* childCnt, uint32_t* childOff, uint32_t* childMembers)
{
    const uint32_t T = *nTilesDev;
    const uint32_t warpsTotal = gridDim.x * (blockDim.x / 32);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t t = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; t < T; t += warpsTotal) {
        const NodeTile ti = tiles[t];
        const bool valid = lane < ti.count;
        const uint32_t b = valid ? lv.assign[ti.start + lane] : 0xFFu;
        const uint32_t member = valid ? lv.members[ti.start + lane] : 0u;
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, b);
        const uint32_t rank = __popc(same & ((1u << lane) - 1u));
        uint32_t size = 0, within = 0; // of child `lane`: its members, and those before this tile
        if (lane < lv.B) {
            const uint32_t lastT = ti.first + (lv.nodeCnt[ti.node] + kRegroupRows - 1) / kRegroupRows - 1;
            const uint64_t row = uint64_t(lane) * maxTiles;
            const uint32_t base = tileScan[row + ti.first];
            size = tileScan[row + lastT] - base + tileHist[row + lastT];
            within = tileScan[row + t] - base;
        }
        uint32_t off = size;
#pragma unroll
        for (uint32_t k = 1; k < kMaxBranch; k <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, off, k);
            if (lane >= k) off += x;
        }
        off += lv.nodeOff[ti.node] - size;
        if (t == ti.first && lane < lv.B) {
            childCnt[uint64_t(ti.node) * lv.B + lane] = size;
            childOff[uint64_t(ti.node) * lv.B + lane] = off;
        }
        const uint32_t at = __shfl_sync(0xFFFFFFFFu, off + within, b & 31u);
        if (valid) childMembers[at + rank] = member;
    }
    // nodes without members have no tile
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < lv.nbNodes; g += gridDim.x * blockDim.x) {
        if (lv.nodeCnt[g] != 0) continue;
        for (uint32_t b = 0; b < lv.B; b++) {
            childCnt[uint64_t(g) * lv.B + b] = 0;
            childOff[uint64_t(g) * lv.B + b] = lv.nodeOff[g];
        }
    }
}

} // namespace

size_t scanTempWords(uint64_t n)
{
    const uint64_t blocks = (n + kScanTile - 1) / kScanTile;
    return blocks + 32;
}

void exclusiveScanU32(const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* tmp, cudaStream_t s)
{
    if (n == 0) return;
    const uint32_t blocks = static_cast<uint32_t>((n + kScanTile - 1) / kScanTile);
    scanBlockSums<<<blocks, kScanBlock, 0, s>>>(in, n, tmp);
    if (blocks <= kScanBlock) {
        scanApply<true><<<blocks, kScanBlock, 0, s>>>(in, n, tmp, out);
    } else {
        scanSingle<<<1, kScanBlock, 0, s>>>(tmp, blocks);
        scanApply<false><<<blocks, kScanBlock, 0, s>>>(in, n, tmp, out);
    }
    RBW_CUDA(cudaGetLastError());
}

void buildNodeTiles(const uint32_t* nodeCnt, const uint32_t* nodeOff, uint32_t nbNodes, uint32_t tileRows,
                    uint32_t* tileOff, uint32_t* tmp, NodeTile* tiles, uint32_t maxTiles, uint32_t* totals,
                    cudaStream_t s)
{
    // Six launches of ~4 us each with their gaps against one of ~4 us (with a level's other launches
    // halved as well, a build of 200,000 rows takes 745 us and not 826).
    if (nbNodes <= kTileListNodes) {
        const uint32_t blocks = std::max(1u, std::min<uint32_t>((maxTiles + kScanBlock - 1) / kScanBlock, 296));
        nodeTilesKernel<<<blocks, kScanBlock, 0, s>>>(nodeCnt, nodeOff, nbNodes, tileRows, maxTiles, tileOff, totals, tiles);
        RBW_CUDA(cudaGetLastError());
        return;
    }
    ceilDivKernel<<<(nbNodes + 255) / 256, 256, 0, s>>>(nodeCnt, nbNodes, tileRows, tileOff);
    exclusiveScanU32(tileOff, tileOff, nbNodes, tmp, s);
    tilesTotal<<<1, 1, 0, s>>>(nodeCnt, tileOff, nbNodes, tileRows, totals);
    const uint32_t blocks = std::min<uint32_t>((maxTiles + 255) / 256, 8192);
    fillNodeTiles<<<std::max(blocks, 1u), 256, 0, s>>>(nodeCnt, nodeOff, tileOff, nbNodes, tileRows, totals, maxTiles,
                                                      tiles);
    RBW_CUDA(cudaGetLastError());
}

void launchInitCenters(const KMeansLevel& lv, const uint32_t* pos, uint64_t nbDescTotal, cudaStream_t s)
{
    const uint64_t total = uint64_t(lv.nbNodes) * kMaxBranch * 8;
    initCentersKernel<<<static_cast<uint32_t>((total + 255) / 256), 256, 0, s>>>(lv, pos, nbDescTotal, 0);
    RBW_CUDA(cudaGetLastError());
}

void launchInitCentersFromDesc(const KMeansLevel& lv, const uint32_t* descIdx, uint64_t nbDescTotal, cudaStream_t s)
{
    const uint64_t total = uint64_t(lv.nbNodes) * kMaxBranch * 8;
    initCentersKernel<<<static_cast<uint32_t>((total + 255) / 256), 256, 0, s>>>(lv, descIdx, nbDescTotal, 1);
    RBW_CUDA(cudaGetLastError());
}

void launchCenterNorms(const KMeansLevel& lv, cudaStream_t s)
{
    const uint64_t total = uint64_t(lv.nbNodes) * kMaxBranch;
    centerNormsKernel<<<static_cast<uint32_t>((total + 255) / 256), 256, 0, s>>>(lv);
    RBW_CUDA(cudaGetLastError());
}

void launchKMeansPPInit(const KMeansLevel& lv, uint64_t seed, uint32_t level, uint32_t* nValid, uint32_t* list,
                        cudaStream_t s)
{
    // A CTA per node, or, where the nodes have at most kPPSmall members on average and are many, a warp
    // per node and a CTA for each larger one.
    if (lv.nbNodes >= kPPSmallNodes && lv.nbMembers <= uint64_t(kPPSmall) * lv.nbNodes) {
        RBW_CUDA(cudaMemsetAsync(list, 0, 4, s));
        kmeansPPSmallKernel<<<lv.nbNodes, 32, 0, s>>>(lv, seed, level, list, nValid);
        kmeansPPKernel<<<currentSmCount() * kPPCtasPerSm, kPPSample, 0, s>>>(lv, seed, level, list, nValid);
    } else {
        kmeansPPKernel<<<lv.nbNodes, kPPSample, 0, s>>>(lv, seed, level, nullptr, nValid);
    }
    RBW_CUDA(cudaGetLastError());
}

void launchAssign(const KMeansLevel& lv, const NodeTile* tiles, const uint32_t* nTilesDev, uint32_t maxTiles,
                  cudaStream_t s)
{
    int dev = 0, sms = 0;
    RBW_CUDA(cudaGetDevice(&dev));
    RBW_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // A fixed grid (the occupancy query gave one CTA per SM on some launches, 3-4x slower) of
    // up to kAssignCtasPerSm CTAs per SM, or fewer where the autotuner chose so for this workload.
    static_assert(kAssignCtasPerSm * kAssignTmemCols <= 512, "TMEM columns of the resident CTAs");
    static_assert(kAssignCtasPerSm * (kAssignSmemBytes + 1024) <= 228 * 1024, "shared memory of the resident CTAs");
    const uint32_t perSm = std::min(kAssignCtasPerSm, tunedValue(kTuneAssignCtasPerSm, lv.B, 0, lv.nbMembers));
    const uint32_t grid = std::max(1u, std::min<uint32_t>(maxTiles, static_cast<uint32_t>(sms) * perSm));
    ScopedKernelTimer timer(kTimedAssign, s);
    static std::atomic<uint64_t> attr{0};
    setMaxDynamicSmemOncePerDevice(reinterpret_cast<const void*>(assignKernel), int(kAssignSmemBytes), attr);
    assignKernel<<<grid, kAssignThreads, kAssignSmemBytes, s>>>(lv, tiles, nTilesDev);
    RBW_CUDA(cudaGetLastError());
}

void launchRegroup(const KMeansLevel& lv, const RegroupScratch& rs, uint32_t* childMembers, uint32_t* childCnt,
                   uint32_t* childOff, cudaStream_t s)
{
    buildNodeTiles(lv.nodeCnt, lv.nodeOff, lv.nbNodes, kRegroupRows, rs.tileOff, rs.scanTmp, rs.tiles, rs.maxTiles,
                   rs.totals, s);
    // Entries past the last tile of each row are not written: they add the same to every scan value
    // of the later rows.
    const uint32_t warpsPerBlock = 8;
    const uint32_t blocks = std::max(1u, std::min<uint32_t>((rs.maxTiles + warpsPerBlock - 1) / warpsPerBlock, 16384));
    regroupHistKernel<<<blocks, 32 * warpsPerBlock, 0, s>>>(lv, rs.tiles, rs.totals, rs.maxTiles, rs.tileHist);
    exclusiveScanU32(rs.tileHist, rs.tileScan, uint64_t(lv.B) * rs.maxTiles, rs.scanTmp, s);
    regroupScatterKernel<<<blocks, 32 * warpsPerBlock, 0, s>>>(lv, rs.tiles, rs.totals, rs.maxTiles, rs.tileHist,
                                                               rs.tileScan, childCnt, childOff, childMembers);
    RBW_CUDA(cudaGetLastError());
}

} // namespace rbw
