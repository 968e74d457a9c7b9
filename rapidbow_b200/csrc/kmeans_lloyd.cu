// Lloyd loops of small nodes, whole in one CTA: the node's rows stay in shared memory from its
// first assignment to its last center update (kmeans.cpp:118-133, kmeans.cu:62-384).  This
// translation unit is compiled with --use_fast_math like kmeans_update.cu, so that
// float(sum) / float(count) is the reference's quotient (kmeans.cu:367); everything else here is
// integer arithmetic.
#include "kmeans.cuh"
#include "timing.h"

#include <algorithm>

namespace rbw {
namespace {

constexpr uint32_t kRows = 128;     // members per tile
constexpr uint32_t kTileBytes = kRows * kDims;
constexpr uint32_t kOneHotBytes = kRows * kMaxBranch;

// Sorts the level's nodes by the room they need: lists of nodes of at most lloydTiles(c) tiles
// for each resident class c, and streamCnt / lastChanged for the nodes that stay with the
// streaming assign (0 members, frozen, for all others).
__global__ void __launch_bounds__(256) classifyNodesKernel(const uint32_t* nodeCnt, uint32_t nbNodes,
                                                           LloydClasses cls, uint32_t* lastChanged)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const uint32_t n = g < nbNodes ? nodeCnt[g] : 0u;
    uint32_t c = kLloydClasses + 1; // empty: nothing to do
    if (n > 0) {
        c = kLloydClasses;          // streamed
#pragma unroll
        for (uint32_t k = kLloydClasses; k-- > 0;)
            if (n <= lloydTiles(k) * kRows) c = k;
    }
    if (c == kLloydClasses) {
        const uint32_t tiles = (n + kRows - 1) / kRows, most = lloydTiles(kLloydClasses - 1);
        atomicAdd(cls.counters + kLloydShareCtas, (tiles + most - 1) / most);
    }
    if (g < nbNodes) {
        cls.streamCnt[g] = c == kLloydClasses ? n : 0u;
        lastChanged[g] = c == kLloydClasses ? 0xFFFFFFFFu : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k <= kLloydClasses; k++) {
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, c == k);
        if (mask == 0) continue;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(cls.counters + k, uint32_t(__popc(mask)));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (c == k) cls.lists[uint64_t(k) * nbNodes + base + __popc(mask & ((1u << lane) - 1u))] = g;
    }
}

// One CTA per node at a time, kTiles x 128 rows of shared memory, kGroups groups of 128 threads.
// Per step:
//   1. group q takes tiles q, q + kGroups, ...: its first warp issues their distance MMAs (M = 128
//      members, N = 16 centers, see assignKernel), one commit per tile;
//   2. a thread per row takes the argmin of |c|^2 - 2 x.c (lowest center on ties) and writes the
//      row's one-hot; then the group's first warp issues the tile's sums MMAs (A = the tile read
//      MN-major) into the group's own 16 TMEM columns;
//   3. the thread of dimension d adds the groups' sums and writes the new byte of each center
//      with members (kmeans.cu:356-372), and the norms follow by warp sums.
// A node stops after the step that changes no assignment (kmeans.cu:238-240, 341-343).
//
// The streaming assign reads a node's rows from memory in every step and passes its sums through
// global memory to the update; for nodes of about 100 members those sums are as many bytes as the
// rows.  Here a step is bound by its chain (MMA -> argmin -> MMA -> update, ~2 us) with as many
// nodes in flight per SM as fit.
template <uint32_t kTiles, uint32_t kGroups>
struct LloydSmem {
    uint8_t tile[kTiles][kTileBytes];  // member rows, 128-byte swizzle
    uint8_t cen[kMaxBranch * kDims];   // centers, same layout
    uint8_t oh[kTiles][kOneHotBytes];  // [member][center] one-hot
    int32_t cnk[kMaxBranch];           // 16 |c_b|^2 + b, INT_MAX for padding slots
    uint32_t cnt[kMaxBranch];
    uint32_t normPart[4][kMaxBranch];
    uint64_t distBar[kTiles];
    uint64_t sumBar;
    uint32_t tmemBase, abortFlag, chg, slot;
};
template <uint32_t kTiles, uint32_t kGroups>
constexpr size_t lloydSmemBytes() { return sizeof(LloydSmem<kTiles, kGroups>) + 1024; }

template <uint32_t kTiles, uint32_t kGroups>
__host__ __device__ constexpr uint32_t lloydTmemCols()
{
    const uint32_t need = 16 * (kTiles + kGroups);
    return need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : 256;
}

// 32 lanes x N columns of 32-bit accumulators, waited for.
template <uint32_t N>
__device__ __forceinline__ void tmemLoadN(uint32_t taddr, uint32_t (&r)[N])
{
    if constexpr (N == 16) {
        tmemLoad16(taddr, r);
        tmemWaitTie(r);
    } else if constexpr (N == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr)
                     : "memory");
    } else {
        static_assert(N == 4, "4, 8 or 16 columns");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(taddr)
                     : "memory");
    }
}

// Barrier of one group's 128 threads.  Barrier numbers are constants: with a number in a register
// the compiler reserves all 16 of the CTA, and an SM has barriers for four such CTAs only.
template <uint32_t kGroups>
__device__ __forceinline__ void groupBarrier(uint32_t group)
{
    static_assert(kGroups == 1 || kGroups == 2 || kGroups == 4, "one, two or four groups");
    if (kGroups == 1 || group == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
    else if (kGroups == 2 || group == 1) asm volatile("bar.sync 2, 128;" ::: "memory");
    else if (group == 2) asm volatile("bar.sync 3, 128;" ::: "memory");
    else asm volatile("bar.sync 4, 128;" ::: "memory");
}

// What a CTA's threads carry from node to node.
struct LloydThread {
    uint32_t tid, lane, warp;
    uint32_t group, row;            // row of a tile; dimension in the update
    uint32_t laneQuarter, tmem;
    bool issuer;                    // one thread per group issues and commits its MMAs
    uint32_t distPhase, sumPhase;   // distPhase: bit j for this group's tile j
    bool failed;
};

template <uint32_t kTiles, uint32_t kGroups>
__device__ __forceinline__ LloydThread lloydSetup(LloydSmem<kTiles, kGroups>& S)
{
    LloydThread th{};
    th.tid = threadIdx.x;
    th.lane = threadIdx.x % 32;
    th.warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x / 32, 0); // uniform
    th.group = th.warp / 4;
    th.row = threadIdx.x % kRows;
    th.laneQuarter = ((th.warp % 4) * 32u) << 16;
    if (th.tid == 0) {
        for (uint32_t i = 0; i < kTiles; i++) mbarInit(&S.distBar[i], 1);
        mbarInit(&S.sumBar, kGroups);
        S.abortFlag = 0;
        fenceMbarInit();
    }
    if (th.warp == 0) {
        tmemAlloc(&S.tmemBase, lloydTmemCols<kTiles, kGroups>());
        tmemRelinquish();
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    th.tmem = S.tmemBase;
    th.issuer = th.warp % 4 == 0 && electOne();
    return th;
}

template <uint32_t kTiles, uint32_t kGroups>
__device__ __forceinline__ void lloydTeardown(LloydSmem<kTiles, kGroups>& S, LloydThread& th, DeviceErrors* err)
{
    if (th.failed) {
        // a wait ran out: MMAs may still be in flight, the TMEM is freed after them (bounded)
        if (th.issuer) mmaCommit(&S.sumBar);
        mbarWait(&S.sumBar, th.sumPhase, &S.abortFlag, err, 52);
    }
    __syncthreads();
    if (th.warp == 0) {
        tcFenceAfter();
        tmemDealloc(th.tmem, lloydTmemCols<kTiles, kGroups>());
    }
}

// A node whose rows are spread over several CTAs of one cooperative launch: the CTAs add their
// partial sums, counts and change counts of step s into buffer s % 3, meet, and each computes the
// same new centers from the totals.  Buffer (s + 2) % 3 was last read in step s - 1, before its
// reader arrived in step s, and is next added to after the meeting of step s + 1: the leader clears
// it in between.
constexpr uint32_t kShareSums = kMaxBranch * kDims;      // then 16 counts and the change count
constexpr uint32_t kShareBufWords = kShareSums + 32;
constexpr uint32_t kShareArrive = 3 * kShareBufWords;    // CTAs that have arrived, all steps
constexpr uint32_t kShareNodeWords = kShareArrive + 32;
struct LloydShare {
    uint32_t* node;     // [kShareNodeWords], zero at first
    uint32_t* abortAll; // a CTA of the launch gave up
    uint32_t ctas;
    bool leader;
};

__device__ __forceinline__ uint32_t loadAcquire(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One thread: waits (bounded) until every CTA of the node has arrived in this step.
__device__ __forceinline__ bool shareMeet(const LloydShare& sh, uint32_t step, DeviceErrors* err)
{
    __threadfence(); // the CTA's additions, which came before its barrier
    atomicAdd(sh.node + kShareArrive, 1u);
    const uint32_t want = sh.ctas * (step + 1u);
    const uint64_t t0 = globalTimerNs();
    for (uint32_t spin = 1;; spin++) {
        if (loadAcquire(sh.node + kShareArrive) >= want) return true;
        if ((spin & 63u) == 0) {
            if (loadAcquire(sh.abortAll) != 0) return false;
            if (globalTimerNs() - t0 > kWaitLimitNs) {
                if (err != nullptr && atomicCAS(&err->code, 0u, 1u) == 0u) {
                    err->where = 53;
                    err->block = blockIdx.x;
                    err->detail = step;
                }
                return false;
            }
        }
    }
}

// The Lloyd loop of node g, or of this CTA's part of it (kShared): members [off, off + n).
template <bool kShared, uint32_t kTiles, uint32_t kGroups>
__device__ __forceinline__ void lloydNode(LloydSmem<kTiles, kGroups>& S, LloydThread& th, const KMeansLevel& lv,
                                          uint32_t g, uint64_t off, uint32_t n, uint32_t maxIterations,
                                          uint32_t* maxSteps, const LloydShare& share)
{
    constexpr uint32_t kThreads = kRows * kGroups;
    constexpr uint32_t kPerGroup = kTiles / kGroups;       // tiles of a group
    constexpr uint32_t kOwnCenters = kMaxBranch / kGroups; // centers a group updates
    constexpr uint32_t kSumCol = 16 * kTiles;
    static_assert(kTiles % kGroups == 0 && kMaxBranch % kGroups == 0, "whole tiles and centers per group");
    const uint32_t tid = th.tid, lane = th.lane, warp = th.warp, group = th.group, row = th.row;
    const uint32_t laneQuarter = th.laneQuarter, tmem = th.tmem;
    const bool issuer = th.issuer;
    bool failed = th.failed;
    volatile uint32_t* abortFlag = &S.abortFlag;
    const uint32_t T = (n + kRows - 1) / kRows;
    // rows: eight threads per row; rows past n keep whatever the buffer holds (their one-hot is
    // zero and their assignment is not written)
    for (uint32_t r0 = tid / 8; r0 < n; r0 += 8 * (kThreads / 8)) {
        uint32_t m[8];
#pragma unroll
        for (uint32_t u = 0; u < 8; u++) {
            const uint32_t r = r0 + u * (kThreads / 8);
            m[u] = r < n ? lv.members[off + r] : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 8; u++) {
            const uint32_t r = r0 + u * (kThreads / 8), c = tid % 8;
            if (r < n)
                cpAsync16(&S.tile[0][0] + r * kDims + ((c ^ (r & 7u)) << 4),
                          lv.desc + uint64_t(m[u]) * kDims + (c << 4));
        }
    }
    cpAsyncCommit();
    if (tid < kMaxBranch * 8) {
        const uint32_t b = tid / 8, c = tid % 8;
        *reinterpret_cast<uint4*>(S.cen + b * kDims + ((c ^ (b & 7u)) << 4)) =
            reinterpret_cast<const uint4*>(lv.centers + (uint64_t(g) * kMaxBranch + b) * kDims)[c];
    }
    if (tid < kMaxBranch) {
        S.cnk[tid] = tid < lv.B ? lv.cnorm[uint64_t(g) * kMaxBranch + tid] * 16 + int32_t(tid) : 0x7FFFFFFF;
        S.cnt[tid] = 0;
    }
    if (tid == 0) S.chg = 0;
    cpAsyncWait<0>();
    uint32_t mine[kPerGroup]; // this thread's rows' centers (zero at first, as fresh assignment memory)
#pragma unroll
    for (uint32_t j = 0; j < kPerGroup; j++) mine[j] = 0;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    uint32_t step = 0;
    for (;;) {
        if (warp % 4 == 0) {
            tcFenceAfter();
            for (uint32_t i = group; i < T; i += kGroups) {
                mmaU8x4(issuer, tmem + 16u * i, smemDescSw128(smemAddr(S.tile[i])), 32u,
                        smemDescSw128(smemAddr(S.cen)), 32u, idescU8(16), 0u);
                if (issuer) mmaCommit(&S.distBar[i]);
            }
        }
        uint32_t myCnt = 0, myChg = 0; // lane c < 16: rows of this warp that chose center c
#pragma unroll
        for (uint32_t j = 0; j < kPerGroup; j++) {
            const uint32_t i = group + kGroups * j;
            if (i < T) { // uniform in the group
                failed |= !mbarWait(&S.distBar[i], (th.distPhase >> j) & 1u, abortFlag, lv.err, 50);
                th.distPhase ^= 1u << j;
                tcFenceAfter();
                uint32_t r[16];
                tmemLoad16(tmem + 16u * i + laneQuarter, r);
                tmemWaitTie(r);
                // 16 (|c|^2 - 2 x.c) + b fits 32 bits: the minimum is the lowest center of the
                // lowest score
                int32_t best = 0x7FFFFFFF;
#pragma unroll
                for (uint32_t b = 0; b < kMaxBranch; b++)
                    best = min(best, S.cnk[b] - 32 * static_cast<int32_t>(r[b]));
                const uint32_t bi = static_cast<uint32_t>(best) & 15u;
                const bool valid = kRows * i + row < n;
                const uint32_t word = valid ? 1u << (8u * (bi & 3u)) : 0u, q = bi >> 2;
                *reinterpret_cast<uint4*>(S.oh[i] + row * kMaxBranch) =
                    make_uint4(q == 0 ? word : 0u, q == 1 ? word : 0u, q == 2 ? word : 0u, q == 3 ? word : 0u);
                uint32_t mask = __ballot_sync(0xFFFFFFFFu, valid);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {
                    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, (bi >> k) & 1u);
                    mask &= (lane >> k) & 1u ? bits : ~bits;
                }
                myCnt += __popc(mask);
                myChg += __popc(__ballot_sync(0xFFFFFFFFu, valid && mine[j] != bi));
                mine[j] = bi;
                tcFenceBefore();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                groupBarrier<kGroups>(group);
                if (warp % 4 == 0) {
                    tcFenceAfter();
                    mmaU8x4(issuer, tmem + kSumCol + 16u * group, smemDescSw128(smemAddr(S.tile[i])), 4096u,
                            smemDescMn16(smemAddr(S.oh[i])), 512u, idescU8(16) | kIdescMnMajorAB, j);
                }
            }
        }
        if (issuer) {
            if (group < T) mmaCommit(&S.sumBar);
            else mbarArrive(&S.sumBar);
        }
        if (lane < kMaxBranch && myCnt) atomicAdd(&S.cnt[lane], myCnt);
        if (lane == 0 && myChg) atomicAdd(&S.chg, myChg);
        failed |= !mbarWait(&S.sumBar, th.sumPhase, abortFlag, lv.err, 51);
        th.sumPhase ^= 1u;
        tcFenceAfter();
        failed = __syncthreads_or(failed) != 0; // and cnt, chg are complete
        if (!kShared) {
            step++;
            if (failed || S.chg == 0) break; // uniform
        }
        // centers b0 .. b0 + kOwnCenters - 1, dimension `row`
        const uint32_t b0 = group * kOwnCenters;
        uint32_t sum[kOwnCenters];
        tmemLoadN<kOwnCenters>(tmem + kSumCol + b0 + laneQuarter, sum);
#pragma unroll
        for (uint32_t q = 1; q < kGroups; q++) {
            if (q < T) {
                uint32_t more[kOwnCenters];
                tmemLoadN<kOwnCenters>(tmem + kSumCol + 16u * q + b0 + laneQuarter, more);
#pragma unroll
                for (uint32_t k = 0; k < kOwnCenters; k++) sum[k] += more[k];
            }
        }
        tcFenceBefore();
        uint32_t cnt[kOwnCenters];
        if (kShared) {
            uint32_t* buf = share.node + (step % 3u) * kShareBufWords;
#pragma unroll
            for (uint32_t k = 0; k < kOwnCenters; k++)
                if (sum[k]) atomicAdd(buf + (b0 + k) * kDims + row, sum[k]);
            if (tid < kMaxBranch && S.cnt[tid]) atomicAdd(buf + kShareSums + tid, S.cnt[tid]);
            if (tid == kMaxBranch && S.chg) atomicAdd(buf + kShareSums + kMaxBranch, S.chg);
            __syncthreads();
            bool met = true;
            if (tid == 0) {
                met = !failed && shareMeet(share, step, lv.err);
                if (!met) atomicExch(share.abortAll, 1u);
            }
            failed = __syncthreads_or(!met || failed) != 0;
            step++;
            if (failed) break; // uniform
#pragma unroll
            for (uint32_t k = 0; k < kOwnCenters; k++) sum[k] = __ldcg(buf + (b0 + k) * kDims + row);
            // one warp fetches the counts: they are one line, which all CTAs of the node read now (with
            // every thread reading them a step of 50,000 rows over 131 CTAs took 6.3 us, not 4.8)
            if (tid < kMaxBranch) S.cnt[tid] = __ldcg(buf + kShareSums + tid);
            if (tid == kMaxBranch) S.chg = __ldcg(buf + kShareSums + kMaxBranch);
            __syncthreads();
            if (S.chg == 0) break; // uniform in all CTAs of the node
#pragma unroll
            for (uint32_t k = 0; k < kOwnCenters; k++) cnt[k] = S.cnt[b0 + k];
            if (share.leader) { // step was counted: (step + 1) % 3 is the buffer after the next
                uint32_t* next = share.node + ((step + 1u) % 3u) * kShareBufWords;
                for (uint32_t i = tid; i < kShareBufWords; i += kThreads) next[i] = 0;
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < kOwnCenters; k++) cnt[k] = S.cnt[b0 + k];
        }
#pragma unroll
        for (uint32_t k = 0; k < kOwnCenters; k++) {
            const uint32_t b = b0 + k, c = cnt[k];
            uint8_t* at = S.cen + b * kDims + (((row >> 4) ^ (b & 7u)) << 4) + (row & 15u);
            uint32_t v = *at;
            if (c != 0) {
                const float quot =
                    lv.ieeeDivision ? __fdiv_rn(float(sum[k]), float(c)) : float(sum[k]) / float(c);
                v = static_cast<uint8_t>(roundf(quot));
                *at = static_cast<uint8_t>(v);
            }
            const uint32_t part = __reduce_add_sync(0xFFFFFFFFu, v * v);
            if (lane == 0) S.normPart[warp % 4][b] = part;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads(); // centers and norm parts written, cnt read
        if (tid < kMaxBranch) {
            if (tid < lv.B)
                S.cnk[tid] = int32_t(S.normPart[0][tid] + S.normPart[1][tid] + S.normPart[2][tid] +
                                     S.normPart[3][tid]) * 16 + int32_t(tid);
            S.cnt[tid] = 0;
        }
        if (tid == 0) S.chg = 0;
        if (step >= maxIterations) break; // uniform
        __syncthreads();
    }
    __syncthreads(); // cnk is final
#pragma unroll
    for (uint32_t j = 0; j < kPerGroup; j++) {
        const uint32_t r = kRows * (group + kGroups * j) + row;
        if (r < n) lv.assign[off + r] = static_cast<uint8_t>(mine[j]);
    }
    th.failed = failed;
    if (kShared && !share.leader) return;
    if (tid < kMaxBranch * 8) {
        const uint32_t b = tid / 8, c = tid % 8;
        reinterpret_cast<uint4*>(lv.centers + (uint64_t(g) * kMaxBranch + b) * kDims)[c] =
            *reinterpret_cast<const uint4*>(S.cen + b * kDims + ((c ^ (b & 7u)) << 4));
    }
    if (tid < lv.B) lv.cnorm[uint64_t(g) * kMaxBranch + tid] = S.cnk[tid] >> 4;
    if (tid == 0) atomicMax(maxSteps, step);
}

template <uint32_t kTiles, uint32_t kGroups, uint32_t kCtasPerSm>
__global__ void __launch_bounds__(kRows * kGroups, kCtasPerSm)
    lloydResidentKernel(KMeansLevel lv, const uint32_t* list, const uint32_t* listCount, uint32_t* cursor,
                        uint32_t maxIterations, uint32_t* maxSteps)
{
    using Smem = LloydSmem<kTiles, kGroups>;
    extern __shared__ uint8_t smemRaw[];
    Smem& S = *reinterpret_cast<Smem*>(smemAligned(smemRaw));
    LloydThread th = lloydSetup(S);
    const uint32_t nList = *listCount;
    while (!th.failed) {
        if (th.tid == 0) S.slot = atomicAdd(cursor, 1u);
        __syncthreads(); // the previous node's shared memory is no longer read
        const uint32_t slot = S.slot;
        if (slot >= nList) break;
        const uint32_t g = list[slot];
        lloydNode<false>(S, th, lv, g, lv.nodeOff[g], lv.nodeCnt[g], maxIterations, maxSteps, LloydShare{});
    }
    lloydTeardown(S, th, lv.err);
}

// One cooperative launch, a CTA per SM: the larger nodes are spread over the CTAs (every node's
// tiles in parts of at most t tiles, with the smallest t whose parts fit the grid and leave CTAs for
// the resident nodes), and CTAs that are done, or had no part, take those (`tail`), the largest class
// first.  For levels
// whose streamed rows fit the SMs' shared memory together (220,000 rows): a step is two MMA chains,
// 2,048 atomic adds per CTA and one meeting of the node's CTAs, where the streaming path takes two
// launches, a cleared counter and, every few steps, a read-back of it.
constexpr uint32_t kShareTiles = 12, kShareGroups = 4;
__global__ void __launch_bounds__(kRows * kShareGroups, 1)
    lloydSharedKernel(KMeansLevel lv, LloydClasses cls, uint32_t* shareMem, uint32_t maxIterations, uint32_t tail)
{
    using Smem = LloydSmem<kShareTiles, kShareGroups>;
    extern __shared__ uint8_t smemRaw[];
    Smem& S = *reinterpret_cast<Smem*>(smemAligned(smemRaw));
    LloydThread th = lloydSetup(S);
    const uint32_t m = cls.counters[kLloydClasses]; // at most one node per CTA
    if (m > 0) {
        const uint32_t* list = cls.lists + uint64_t(kLloydClasses) * lv.nbNodes;
        uint32_t* tiles = reinterpret_cast<uint32_t*>(S.tile[0]); // [m] tiles of node i
        uint32_t* total = tiles + gridDim.x;                      // [kShareTiles] parts for t = 1 ..
        uint32_t* job = total + kShareTiles;                      // node, part, parts, or job[2] = 0
        for (uint32_t i = th.tid; i < m; i += blockDim.x) tiles[i] = (lv.nodeCnt[list[i]] + kRows - 1) / kRows;
        if (th.tid == 0) job[2] = 0;
        __syncthreads();
        if (th.warp < kShareTiles) {
            uint32_t sum = 0;
            for (uint32_t i = th.lane; i < m; i += 32) sum += (tiles[i] + th.warp) / (th.warp + 1u);
            sum = __reduce_add_sync(0xFFFFFFFFu, sum);
            if (th.lane == 0) total[th.warp] = sum;
        }
        __syncthreads();
        // The most CTAs (fewest tiles each) that leave enough for the small nodes: a small node's step
        // takes about half the time of a shared one, so as many CTAs as half those nodes finish them
        // meanwhile.  (200,000 rows, 256 nodes: 103 us with all CTAs on the few large ones first, 75 us
        // with a third of them; with no small nodes fewer CTAs are slower, 276 -> 383 us.)
        uint32_t small = 0;
        for (uint32_t c = 0; tail && c < kLloydClasses; c++) small += cls.counters[c];
        const uint32_t most = gridDim.x - min(small / 2, gridDim.x);
        uint32_t t = 1;
        while (t < kShareTiles && total[t - 1] > most) t++;
        for (uint32_t i = th.tid; i < m; i += blockDim.x) {
            uint32_t first = 0;
            for (uint32_t j = 0; j < i; j++) first += (tiles[j] + t - 1u) / t;
            const uint32_t parts = (tiles[i] + t - 1u) / t;
            if (blockIdx.x >= first && blockIdx.x < first + parts) {
                job[0] = i;
                job[1] = blockIdx.x - first;
                job[2] = parts;
            }
        }
        __syncthreads();
        const uint32_t i = job[0], part = job[1], parts = job[2];
        const uint32_t nTiles = parts ? tiles[i] : 0u;
        __syncthreads(); // the tile buffer is overwritten by the rows
        if (parts) {
            const uint32_t g = list[i], n = lv.nodeCnt[g];
            const uint32_t r0 = uint32_t(uint64_t(nTiles) * part / parts) * kRows;
            const uint32_t r1 = min(n, uint32_t(uint64_t(nTiles) * (part + 1) / parts) * kRows);
            const LloydShare share{shareMem + uint64_t(i) * kShareNodeWords, shareMem + uint64_t(m) * kShareNodeWords,
                                   parts, part == 0};
            lloydNode<true>(S, th, lv, g, uint64_t(lv.nodeOff[g]) + r0, r1 - r0, maxIterations,
                            cls.counters + kLloydMaxSteps, share);
        }
    }
    for (uint32_t c = tail ? kLloydClasses : 0u; c-- > 0;) {
        while (!th.failed) {
            __syncthreads(); // the previous node's shared memory is no longer read
            if (th.tid == 0) S.slot = atomicAdd(cls.counters + kLloydCursor + c, 1u);
            __syncthreads();
            const uint32_t slot = S.slot;
            if (slot >= cls.counters[c]) break;
            const uint32_t g = cls.lists[uint64_t(c) * lv.nbNodes + slot];
            lloydNode<false>(S, th, lv, g, lv.nodeOff[g], lv.nodeCnt[g], maxIterations, cls.counters + kLloydMaxSteps,
                             LloydShare{});
        }
    }
    lloydTeardown(S, th, lv.err);
}

template <uint32_t kTiles, uint32_t kGroups, uint32_t kCtasPerSm>
void launchClass(const KMeansLevel& lv, const LloydClasses& cls, uint32_t c, uint32_t count, uint32_t maxIterations,
                 cudaStream_t s)
{
    if (count == 0) return;
    constexpr size_t smem = lloydSmemBytes<kTiles, kGroups>();
    static_assert(kCtasPerSm * (smem + 1024) <= 228 * 1024, "shared memory of the resident CTAs");
    static_assert(kCtasPerSm * lloydTmemCols<kTiles, kGroups>() <= 512, "TMEM columns of the resident CTAs");
    static std::atomic<uint64_t> attr{0};
    const auto kernel = lloydResidentKernel<kTiles, kGroups, kCtasPerSm>;
    setMaxDynamicSmemOncePerDevice(reinterpret_cast<const void*>(kernel), int(smem), attr);
    const uint32_t grid = std::min(count, uint32_t(currentSmCount()) * kCtasPerSm);
    kernel<<<grid, kRows * kGroups, smem, s>>>(lv, cls.lists + uint64_t(c) * lv.nbNodes, cls.counters + c,
                                               cls.counters + kLloydCursor + c, maxIterations,
                                               cls.counters + kLloydMaxSteps);
    RBW_CUDA(cudaGetLastError());
}

} // namespace

void launchClassifyNodes(const KMeansLevel& lv, const LloydClasses& cls, cudaStream_t s)
{
    classifyNodesKernel<<<(lv.nbNodes + 255) / 256, 256, 0, s>>>(lv.nodeCnt, lv.nbNodes, cls, lv.lastChanged);
    RBW_CUDA(cudaGetLastError());
}

void launchLloydResident(const KMeansLevel& lv, const LloydClasses& cls, const uint32_t* hostCounts,
                         uint32_t maxIterations, cudaStream_t s)
{
    ScopedKernelTimer timer(kTimedAssign, s);
    // the longest nodes first, so that the short ones fill the last wave
    launchClass<lloydTiles(3), 4, 1>(lv, cls, 3, hostCounts[3], maxIterations, s);
    launchClass<lloydTiles(2), 2, 2>(lv, cls, 2, hostCounts[2], maxIterations, s);
    launchClass<lloydTiles(1), 1, 5>(lv, cls, 1, hostCounts[1], maxIterations, s);
    launchClass<lloydTiles(0), 1, 8>(lv, cls, 0, hostCounts[0], maxIterations, s);
}

size_t lloydShareBytes(uint32_t nbShared) { return (uint64_t(nbShared) * kShareNodeWords + 32) * 4; }

bool launchLloydShared(const KMeansLevel& lv, const LloydClasses& cls, uint32_t nbShared, void* shareMem, bool tail,
                       uint32_t maxIterations, cudaStream_t s)
{
    ScopedKernelTimer timer(kTimedAssign, s);
    constexpr size_t smem = lloydSmemBytes<kShareTiles, kShareGroups>();
    static std::atomic<uint64_t> attr{0};
    setMaxDynamicSmemOncePerDevice(reinterpret_cast<const void*>(lloydSharedKernel), int(smem), attr);
    RBW_CUDA(cudaMemsetAsync(shareMem, 0, lloydShareBytes(nbShared), s));
    KMeansLevel lvArg = lv;
    LloydClasses clsArg = cls;
    uint32_t* mem = static_cast<uint32_t*>(shareMem);
    uint32_t tailArg = tail ? 1u : 0u;
    void* args[] = {&lvArg, &clsArg, &mem, &maxIterations, &tailArg};
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(lloydSharedKernel),
                                                      dim3(currentSmCount()), dim3(kRows * kShareGroups), args, smem, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError(); // answered here
        return false;
    }
    RBW_CUDA(e);
    return true;
}

} // namespace rbw
