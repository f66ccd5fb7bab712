/*
 * ryoanji-b200: interaction lists, the form of the traversal for launches of few groups and for groups far longer than
 * the others. walkKernel walks the tree and writes every group's approximated cells and direct leaves to items, pieces
 * of bounded cost; an evaluation kernel (traverse.cu, traverse64.cu) sums the items in any order; finishKernel adds a
 * group's items in a fixed order. The time of a small solve is then that of its total work and not of its longest
 * group's. The walk follows the reference's rule (ryoanji/src/ryoanji/nbody/traversal_gpu.cu:210-237).
 *
 * What bounds it: the walk of many groups is bound by instruction issue and the L1 (a step of 32 cells takes about 170
 * instructions with the list's writing; 5% of the evaluation's time), that of few groups by the latency of its longest
 * part. The parts of a divided walk load two steps' cells at once: 60,001 Plummer bodies 132 -> 112 us. A whole walk
 * does not, which costs it up to a fifth of its time (2^20 bodies 430 against 340 us, 1% of the solve): it is the walk
 * whose depth the caller sees. Divided ones have theirs taken beside the evaluation (walkDepth), at 1 to 3% of a solve.
 * The lists take 6-15 KB per group and stay in the L2 between the two kernels.
 */
#pragma once

#include <type_traits>

#include "internal.hpp"

namespace ryo
{

constexpr int kTravWarps    = 4;
constexpr int kTravThreads  = kTravWarps * kWarp;
constexpr int kM2PCap       = 64;  // pending approximated cells (flushed at 64, or 32 for dipole expansions)
constexpr int kRootOnly     = -2;  // stack marker: the root itself is the only cell (single-leaf tree); a marker
                                   // -(r + 2) stands for the single cell r

constexpr int kSegLeafCap   = kWarp; // direct leaves per list segment
// segment header of an interaction list: kind in the low two bits, entry count above
constexpr uint32_t kSegCells = 0, kSegLeaves = 1, kSegReplica = 2, kSegImages = 3;
constexpr int kReplicaWords  = 4;

//! a list walk's pending entries: a segment leaves fewer than a segment's, and one walk step adds at most kWarp
struct WalkSmem
{
    int m2p[kM2PCap + kWarp];
    uint32_t image[kM2PCap + kWarp]; // of periodic groups: the image each pending cell is seen in
    int2 leaves[kSegLeafCap + kWarp];
};

//! a periodic image (ix, iy, iz), each in [-kMaxImage, kMaxImage), in one word, and its components
constexpr int kMaxImage = 512;
__device__ __forceinline__ uint32_t packImage(int ix, int iy, int iz)
{
    return uint32_t(ix + kMaxImage) | (uint32_t(iy + kMaxImage) << 10) | (uint32_t(iz + kMaxImage) << 20);
}
__device__ __forceinline__ float imageShift(uint32_t image, int d)
{
    return float(int((image >> (10 * d)) & 1023u) - kMaxImage);
}

//! the tree root and periodic images of a group: the launch's, or its system's in a batched solve (float only)
template<class R>
struct GroupFrame
{
    int rootEntry, shells;
    R boxL[3];
    uint32_t sys;

    __device__ __forceinline__ void set(const TraverseLaunch& P, unsigned g)
    {
        rootEntry = P.numNodes == 1 ? kRootOnly : P.initNode;
        shells    = P.numShells;
        sys       = 0;
        if constexpr (std::is_same_v<R, double>)
        {
#pragma unroll
            for (int d = 0; d < 3; ++d)
                boxL[d] = P.boxL64[d];
            return;
        }
        if (P.groupSys)
        {
            sys               = P.groupSys[g];
            const SysTrav& st = P.systems[sys];
            rootEntry         = st.entry;
            shells            = st.numShells;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                boxL[d] = st.boxL[d];
        }
        else
        {
#pragma unroll
            for (int d = 0; d < 3; ++d)
                boxL[d] = P.boxL[d];
        }
    }
};

// ------------------------------------------------------------------------------------------------ lists

/*! the interaction list under construction, in items of P.itemWords words taken from the launch's pool as they are
 *  needed. What an item holds depends on the walk alone, never on the order in which warps take items. */
struct ListWriter
{
    int item;        // current item, -1 before the first
    int count;       // items of the task
    bool replicaSet; // the item knows the current replica
    bool starved;    // the pool ran out
    uint32_t pos;    // words used in the item
    unsigned cost;   // interactions in the item: direct bodies + 2 x cells

    //! room for a segment of @p payload words and @p segCost interactions (all lanes call it); false if starved
    __device__ __forceinline__ bool room(const TraverseLaunch& P, unsigned g, uint32_t payload, unsigned segCost)
    {
        if (item < 0 || pos + 1 + kReplicaWords + payload > P.itemWords || (cost > 0 && cost + segCost > P.itemCost))
        {
            int next = 0;
            if (laneId() == 0)
            {
                const unsigned at = atomicAdd(&P.ctl->itemCount, 1u);
                next              = at < P.itemCapacity ? int(at) : -1;
                if (next >= 0)
                {
                    if (item >= 0) P.items[item].words = pos;
                    P.items[next] = ListItem{g, 0u, item, 0u};
                }
            }
            next = __shfl_sync(0xffffffffu, next, 0);
            if (next < 0)
            {
                starved = true;
                return false;
            }
            item = next;
            ++count;
            replicaSet = false;
            pos        = 0;
            cost       = 0;
        }
        cost += segCost;
        return true;
    }

    __device__ __forceinline__ uint32_t* at(const TraverseLaunch& P) const
    {
        return P.lists + size_t(item) * P.itemWords + pos;
    }

    //! the segments that follow are seen from the targets moved by replica @p rep
    __device__ __forceinline__ void markReplica(const TraverseLaunch& P, const int rep[3])
    {
        if (replicaSet) return;
        uint32_t* w = at(P);
        if (laneId() == 0) w[0] = kSegReplica | (3u << 2);
        if (laneId() < 3) w[1 + laneId()] = uint32_t(laneId() == 0 ? rep[0] : laneId() == 1 ? rep[1] : rep[2]);
        pos += kReplicaWords;
        replicaSet = true;
    }

    //! the first @p n (<= kM2PCap) pending cells as a segment; with @p images each cell's image follows, so that
    //! cells of several replicas share a batch, which is seen from the targets where they are
    __device__ __forceinline__ void cells(const TraverseLaunch& P, unsigned g, const WalkSmem& W, int n, bool images,
                                          const int* rep)
    {
        const uint32_t payload = unsigned(images ? 2 * n : n);
        if (!room(P, g, payload, 2u * unsigned(n))) return;
        if (rep) markReplica(P, rep);
        if (images) replicaSet = false;
        uint32_t* w = at(P);
        if (laneId() == 0) w[0] = (images ? kSegImages : kSegCells) | (uint32_t(n) << 2);
        for (int k = int(laneId()); k < n; k += kWarp)
        {
            w[1 + k] = uint32_t(W.m2p[k]);
            if (images) w[1 + n + k] = W.image[k];
        }
        pos += 1 + payload;
    }

    //! the first @p n (<= kSegLeafCap) pending leaves as a segment of (first body, body count) pairs
    __device__ __forceinline__ void leaves(const TraverseLaunch& P, unsigned g, const WalkSmem& W, int n,
                                           const int* rep)
    {
        const unsigned mine   = int(laneId()) < n ? unsigned(W.leaves[laneId()].y) : 0u;
        const unsigned bodies = __reduce_add_sync(0xffffffffu, mine);
        if (!room(P, g, 2u * unsigned(n), bodies)) return;
        if (rep) markReplica(P, rep);
        uint32_t* w    = at(P);
        const int* src = reinterpret_cast<const int*>(W.leaves);
        if (laneId() == 0) w[0] = kSegLeaves | (uint32_t(n) << 2);
        for (int k = int(laneId()); k < 2 * n; k += kWarp)
            w[1 + k] = uint32_t(src[k]);
        pos += 1 + 2 * unsigned(n);
    }
};

//! centre and half extent of the bounding box of group @p g
template<class R, class Targets>
__device__ __forceinline__ void groupBox(const TraverseLaunch& P, const Targets& tgt, unsigned g, R tc[3], R ts[3])
{
    using F     = Fp<R>;
    const int b = int(P.groupStart[g]), e = int(P.groupEnd[g]);
    R u[3], v[3];
    tgt.position(min(b + int(laneId()), e - 1), u);
    tgt.position(min(b + kWarp + int(laneId()), e - 1), v);
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        const R l = warpMin(fmin(u[d], v[d])), h = warpMax(fmax(u[d], v[d]));
        tc[d]     = F::mul(F::add(h, l), R(0.5));
        ts[d]     = F::mul(F::sub(h, l), R(0.5));
    }
}

/*! the most entries that the undivided walk of group @p g holds, four taken per step: the depth that a caller's stack
 *  capacity bounds and that the statistics report. The parts of a divided walk have other depths, since each starts
 *  lower and takes two steps at once. Every replica's walk starts anew: part @p sub of @p parts takes its share of them.
 *  False if a walk passes P.stackCapacity. */
template<class Nodes, class Targets>
__device__ __forceinline__ bool walkDepth(const TraverseLaunch& P, const Nodes& nodes, const Targets& tgt, unsigned g,
                                          unsigned sub, unsigned parts, int* stack, int& maxStack)
{
    const int lane    = laneId();
    const unsigned lt = lanemaskLt();
    using R = typename Nodes::Real;
    using F = Fp<R>;
    R tc[3], ts[3];
    groupBox(P, tgt, g, tc, ts);
    GroupFrame<R> G;
    G.set(P, g);
    maxStack      = 0;
    unsigned turn = parts - sub; // the replicas at multiples of parts are walked
    for (int iz = -G.shells; iz <= G.shells; ++iz)
        for (int iy = -G.shells; iy <= G.shells; ++iy)
            for (int ix = -G.shells; ix <= G.shells; ++ix)
            {
                const R sh[3] = {F::mul(R(ix), G.boxL[0]), F::mul(R(iy), G.boxL[1]), F::mul(R(iz), G.boxL[2])};
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    tc[d] = F::add(tc[d], sh[d]);
                int sp = turn % parts == 0 ? 1 : 0;
                ++turn;
                __syncwarp();
                if (lane == 0) stack[0] = G.rootEntry;
                __syncwarp();
                while (sp > 0)
                {
                    const int k     = min(4, sp), at = k - 4 + (lane >> 3);
                    sp -= k;
                    const int entry = at >= 0 ? stack[sp + at] : -1;
                    int cell        = -1;
                    if (entry <= kRootOnly) cell = (lane & 7) == 0 ? kRootOnly - entry : -1;
                    else if (entry >= 0) cell = entry + (lane & 7);
                    __syncwarp();
                    typename Nodes::Center c = {};
                    int4 link                = {};
                    if (cell >= 0) nodes.load(cell, c, link);
                    const bool split  = cell >= 0 && macFails(c, tc, ts) && link.x != 0;
                    const unsigned bs = __ballot_sync(0xffffffffu, split);
                    if (sp + __popc(bs) > P.stackCapacity) return false;
                    if (split) stack[sp + __popc(bs & lt)] = link.x;
                    sp += __popc(bs);
                    maxStack = max(maxStack, sp);
                    __syncwarp();
                }
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    tc[d] = F::sub(tc[d], sh[d]);
            }
    return true;
}

/*! the depths of the launch's groups whose walks were divided, taken by the evaluation's warps before its items; a
 *  group that passes the stack's capacity has failed. @p stack holds P.stackCapacity entries. */
template<class Nodes, class Targets>
__device__ __forceinline__ void depthTasks(const TraverseLaunch& P, const Nodes& nodes, const Targets& tgt, int* stack)
{
    // replicas are shared out where the groups alone do not occupy the warps: 128 groups with 729 replicas 0.78 -> 0.74
    // ms a solve, but 4,096 groups with 27 replicas 1.90 -> 1.96 ms (of batched systems some may be periodic)
    const unsigned parts = P.numGroups <= 512 && (P.numShells > 0 || P.groupSys) ? P.subWalks : 1u;
    while (true)
    {
        unsigned task = 0;
        if (laneId() == 0) task = atomicAdd(&P.ctl->depthHead, 1u);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= unsigned(P.numGroups) * parts) return;
        const unsigned i = task / parts, g = P.groupList ? P.groupList[i] : i;
        int depth;
        const bool ok = walkDepth(P, nodes, tgt, g, task % parts, parts, stack, depth);
        __syncwarp();
        if (laneId() != 0) continue;
        atomicMax(&P.ctl->stats[kMaxStack], (unsigned long long)depth);
        if (!ok && atomicCAS(&P.groupState[g], 0u, kGroupFailed) == 0u)
            P.failedGroups[atomicAdd(&P.ctl->failedCount, 1u)] = g;
    }
}

//! the depths before any walk, for a capacity that some groups may pass: they are neither walked nor evaluated
template<class Nodes, class Targets>
__global__ void __launch_bounds__(kTravThreads) depthKernel(TraverseLaunch P, Nodes nodes, Targets tgt)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    depthTasks(P, nodes, tgt, reinterpret_cast<int*>(smemRaw) + threadIdx.x / kWarp * P.stackCapacity);
}

/*! walks the tree for one task and writes the interaction list to @p L: a group's whole walk, or part @p sub of
 *  P.subWalks parts. False if the walk overflowed the stack or was starved. */
template<class Nodes, class Targets>
__device__ __forceinline__ bool walkTask(const TraverseLaunch& P, const Nodes& nodes, const Targets& tgt, unsigned g,
                                         unsigned sub, WalkSmem& W, int* stack, ListWriter& L, unsigned& numM2P,
                                         unsigned& numP2P, int& maxStack)
{
    const int lane    = laneId();
    const unsigned lt = lanemaskLt();
    using R = typename Nodes::Real;
    using F = Fp<R>;
    // steps whose cells are loaded at once; in double a second one costs more registers than the latency is worth (the
    // walk of 120,001 Plummer bodies 88 -> 100 us)
    constexpr int kSteps = std::is_same_v<R, float> ? 2 : 1;
    R tc[3], ts[3];
    groupBox(P, tgt, g, tc, ts);
    GroupFrame<R> G;
    G.set(P, g);
    // a part takes one child of the root, or in a periodic group every subWalks-th replica; a single-cell tree belongs
    // to the first part
    const int shells    = G.shells;
    const bool replicas = shells > 0;
    const bool images   = replicas && shells < kMaxImage;
    const bool byChild  = P.subWalks > 1 && !replicas && G.rootEntry >= 0;
    const int start     = byChild ? kRootOnly - (G.rootEntry + int(sub)) : G.rootEntry;
    unsigned turn       = byChild ? 0u : P.subWalks - sub; // the replicas at multiples of subWalks are walked

    L = ListWriter{-1, 0, false, false, 0u, 0u};
    unsigned nM2P = 0, nP2P = 0; // of this lane
    maxStack      = 0;
    int nM        = 0;
    bool overflow = false;
    for (int iz = -shells; iz <= shells && !overflow; ++iz)
        for (int iy = -shells; iy <= shells && !overflow; ++iy)
            for (int ix = -shells; ix <= shells && !overflow; ++ix)
            {
                // the replica shift is added to and later subtracted from the group centre, as in the
                // reference (traversal_gpu.cu:484-505), so the MAC decisions are the reference's. The targets
                // are the original positions plus the shift: shifting them back and forth as the reference
                // does leaves rounding residues, and a target then meets itself at about one float ulp of the
                // box coordinates, which a softening below that turns into a large spurious force.
                const R sh[3]    = {F::mul(R(ix), G.boxL[0]), F::mul(R(iy), G.boxL[1]), F::mul(R(iz), G.boxL[2])};
                const int rep[3] = {ix, iy, iz};
                L.replicaSet     = false;
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    tc[d] = F::add(tc[d], sh[d]);

                int sp = turn % P.subWalks == 0 ? 1 : 0, nL = 0;
                ++turn;
                const uint32_t image = packImage(ix, iy, iz);
                __syncwarp();
                if (lane == 0) stack[0] = start;
                __syncwarp();
                while (sp > 0 && !L.starved && !overflow)
                {
                    // four stack entries, 32 cells, per step; the next step's cells are loaded with them, so that two
                    // steps wait for the L2 once
                    const int k = min(kSteps > 1 ? P.walkEntries : 4, sp);
                    sp -= k;
                    const int slot = lane >> 3;
                    int cells[kSteps];
                    typename Nodes::Center centers[kSteps] = {};
                    int4 links[kSteps]                     = {};
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
                    {
                        const int at    = k - 4 * (u + 1) + slot; // from the top down
                        const int entry = at >= 0 && at < k - 4 * u ? stack[sp + at] : -1;
                        cells[u]        = -1;
                        if (entry <= kRootOnly) cells[u] = (lane & 7) == 0 ? kRootOnly - entry : -1;
                        else if (entry >= 0) cells[u] = entry + (lane & 7);
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
                        if (cells[u] >= 0) nodes.load(cells[u], centers[u], links[u]);
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
                    {
                        if (4 * u >= k) break;
                        const int cell                 = cells[u];
                        const bool valid               = cell >= 0;
                        const typename Nodes::Center c = centers[u];
                        const int4 link                = links[u];
                        bool close  = valid && macFails(c, tc, ts);
                        bool isNode = link.x != 0;
                        bool split  = close && isNode;
                        unsigned bs = __ballot_sync(0xffffffffu, split);
                        int nsplit  = __popc(bs);
                        if (sp + nsplit > P.walkCapacity)
                        {
                            overflow = true;
                            break;
                        }
                        if (split) stack[sp + __popc(bs & lt)] = link.x;
                        sp += nsplit;
                        maxStack = max(maxStack, sp);

                        bool direct = close && !isNode;
                        bool remote = direct && link.z == 0 && c.w != R(0);
                        bool approx = valid && (!close || remote);
                        nM2P += approx ? 1u : 0u;

                        bool evalM  = approx && c.w != R(0); // massless cells contribute exactly zero
                        unsigned bm = __ballot_sync(0xffffffffu, evalM);
                        if (evalM)
                        {
                            W.m2p[nM + __popc(bm & lt)] = cell;
                            if (images) W.image[nM + __popc(bm & lt)] = image;
                        }
                        nM += __popc(bm);

                        bool hasB   = direct && link.z > 0;
                        unsigned bl = __ballot_sync(0xffffffffu, hasB);
                        if (hasB)
                        {
                            W.leaves[nL + __popc(bl & lt)] = make_int2(link.y, link.z);
                            nP2P += unsigned(link.z);
                        }
                        nL += __popc(bl);
                        __syncwarp();
                        if (nM >= kM2PCap)
                        {
                            L.cells(P, g, W, kM2PCap, images, replicas && !images ? rep : nullptr);
                            nM -= kM2PCap; // fewer than kWarp cells remain: one move per lane
                            __syncwarp();
                            if (lane < nM)
                            {
                                W.m2p[lane] = W.m2p[kM2PCap + lane];
                                if (images) W.image[lane] = W.image[kM2PCap + lane];
                            }
                            __syncwarp();
                        }
                        if (nL >= kSegLeafCap)
                        {
                            L.leaves(P, g, W, kSegLeafCap, replicas ? rep : nullptr);
                            nL -= kSegLeafCap;
                            __syncwarp();
                            if (lane < nL) W.leaves[lane] = W.leaves[kSegLeafCap + lane];
                            __syncwarp();
                        }
                    }
                }
                overflow |= L.starved;
                if (nM > 0 && replicas && !images && !overflow)
                {
                    L.cells(P, g, W, nM, false, rep);
                    nM = 0;
                }
                if (nL > 0 && !overflow) L.leaves(P, g, W, nL, replicas ? rep : nullptr);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    tc[d] = F::sub(tc[d], sh[d]);
            }
    if (nM > 0 && !overflow) L.cells(P, g, W, nM, images, nullptr);
    numM2P = __reduce_add_sync(0xffffffffu, nM2P);
    numP2P = __reduce_add_sync(0xffffffffu, nP2P);
    return !overflow && !L.starved;
}

/*! walks the tree and writes the interaction lists. Warps take tasks from the queue: a group each, or one of P.subWalks
 *  parts of a group's walk, so that a launch of few groups still fills the GPU. */
template<class Nodes, class Targets>
__global__ void __launch_bounds__(kTravThreads) walkKernel(TraverseLaunch P, Nodes nodes, Targets tgt)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int warp = threadIdx.x / kWarp, lane = laneId();
    WalkSmem& W    = reinterpret_cast<WalkSmem*>(smemRaw)[warp];
    int* stack     = reinterpret_cast<int*>(smemRaw + sizeof(WalkSmem) * kTravWarps) + warp * P.walkCapacity;
    const unsigned numTasks = unsigned(P.numGroups) * P.subWalks;
    while (true)
    {
        unsigned task = 0;
        if (lane == 0) task = atomicAdd(&P.ctl->workCounter, 1u);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= numTasks) return;
        const unsigned sub = task % P.subWalks;
        const unsigned g   = P.groupList ? P.groupList[task / P.subWalks] : task / P.subWalks;
        if (P.depthFirst && P.groupState[g] != 0u) continue;
        ListWriter L;
        unsigned nM2P, nP2P;
        int maxStack;
        const bool ok = walkTask(P, nodes, tgt, g, sub, W, stack, L, nM2P, nP2P, maxStack);
        __syncwarp();
        if (lane != 0) continue;
        P.taskLast[task] = L.item;
        if (!L.starved && P.subWalks == 1) atomicMax(&P.ctl->stats[kMaxStack], (unsigned long long)maxStack);
        if (!ok)
        {
            // nothing of this group is evaluated: it goes back to the host, to be walked again when the pool is free,
            // or to be split when it overflowed the stack
            if (atomicCAS(&P.groupState[g], 0u, L.starved ? kGroupUnserved : kGroupFailed) == 0u)
            {
                unsigned at = atomicAdd(L.starved ? &P.ctl->unservedCount : &P.ctl->failedCount, 1u);
                (L.starved ? P.unservedGroups : P.failedGroups)[at] = g;
            }
            continue;
        }
        if (L.item >= 0)
        {
            P.items[L.item].words = L.pos;
            P.items[L.item].only  = P.subWalks == 1 && L.count == 1 ? 1u : 0u;
        }
        if (P.subWalks > 1)
        {
            atomicAdd(&P.countM2P[g], nM2P);
            atomicAdd(&P.countP2P[g], nP2P);
        }
        else
        {
            P.countM2P[g] = nM2P;
            P.countP2P[g] = nP2P;
        }
    }
}

constexpr int kFinishThreads = 256;
constexpr int kWalkParts     = kFinishThreads / kWarp; // parts of a divided walk

/*! every group of the launch: interaction counts and statistics, and the results of the groups whose list became items
 *  (or is empty): the items' sums added in FP64, each part of the walk from its last item to its first, then the parts.
 *  @p sink reads the items' sums and stores a target's results, returning its m phi. Bound by the latency of the chains
 *  of items: a warp follows those of a group's parts one after the other, with kParts the warps of a block at once. The
 *  order of the additions is the same, so a launch may take either. */
template<bool kParts, class Sink>
__global__ void __launch_bounds__(kFinishThreads) finishKernel(TraverseLaunch P, Sink sink)
{
    const int lane = laneId(), warp = threadIdx.x / kWarp;
    const unsigned stride = kParts ? gridDim.x : gridDim.x * (kFinishThreads / kWarp);
    __shared__ double sPart[kParts ? kWalkParts : 1][4][2 * kWarp];
    unsigned long long sumP = 0, sumM = 0, maxP = 0, maxM = 0;
    for (unsigned i = kParts ? blockIdx.x : (blockIdx.x * kFinishThreads + threadIdx.x) / kWarp;
         i < unsigned(P.numGroups); i += stride)
    {
        const unsigned g = P.groupList ? P.groupList[i] : i;
        if (P.groupState[g] != 0u) continue;
        const int b = int(P.groupStart[g]), e = int(P.groupEnd[g]);
        if (!kParts || warp == 0)
        {
            const unsigned nM = P.countM2P[g], nP = P.countP2P[g];
            sumP += (unsigned long long)nP * unsigned(e - b);
            sumM += (unsigned long long)nM * unsigned(e - b);
            maxP = max(maxP, (unsigned long long)nP);
            maxM = max(maxM, (unsigned long long)nM);
            if (lane == 0 && P.groupM2P) P.groupM2P[g] = nM;
            if (lane == 0 && P.groupP2P) P.groupP2P[g] = nP;
        }
        double sum[2][4] = {};
        if (!kParts)
        {
            const int last = P.taskLast[i * P.subWalks];
            if (last >= 0 && P.items[last].only) continue;
        }
        for (unsigned sub = kParts ? warp : 0; sub < P.subWalks; sub += kParts ? kWalkParts : 1)
        {
            double part[2][4] = {};
            for (int it = P.taskLast[i * P.subWalks + sub]; it >= 0; it = P.items[it].prev)
            {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                {
                    const auto v = sink.part(P, size_t(it) * (2 * kWarp) + t * kWarp + lane);
                    part[t][0] += v.x;
                    part[t][1] += v.y;
                    part[t][2] += v.z;
                    part[t][3] += v.w;
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    sum[t][k] += part[t][k];
        }
        if constexpr (kParts)
        {
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    sPart[warp][k][t * kWarp + lane] = sum[t][k];
            __syncthreads();
            if (warp < 2) // 32 targets each
            {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    sum[0][k] = 0.0;
#pragma unroll
                    for (int w = 0; w < kWalkParts; ++w)
                        sum[0][k] += sPart[w][k][warp * kWarp + lane];
                }
            }
            __syncthreads();
            if (warp >= 2) continue;
        }
        double pot = 0.0;
#pragma unroll
        for (int t = 0; t < (kParts ? 1 : 2); ++t)
        {
            const int idx = b + (kParts ? warp : t) * kWarp + lane;
            if (idx < e) pot += sink.store(P, idx, sum[t]);
        }
        pot = warpSum(pot);
        if (lane == 0 && pot != 0.0)
        {
            atomicAdd(&P.ctl->potential, pot);
            if (P.sysPotential) atomicAdd(P.sysPotential + (P.groupSys ? P.groupSys[g] : 0u), pot);
        }
    }
    // every lane of a warp holds the same counts; one set of atomics per block
    __shared__ unsigned long long sh[4][kFinishThreads / kWarp];
    if (lane == 0) sh[0][warp] = sumP, sh[1][warp] = sumM, sh[2][warp] = maxP, sh[3][warp] = maxM;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int k = 1; k < kFinishThreads / kWarp; ++k)
    {
        sumP += sh[0][k];
        sumM += sh[1][k];
        maxP = max(maxP, sh[2][k]);
        maxM = max(maxM, sh[3][k]);
    }
    if (sumP == 0 && sumM == 0) return;
    atomicAdd(&P.ctl->stats[kSumP2P], sumP);
    atomicMax(&P.ctl->stats[kMaxP2P], maxP);
    atomicAdd(&P.ctl->stats[kSumM2P], sumM);
    atomicMax(&P.ctl->stats[kMaxM2P], maxM);
}

//! blocks of @p kernel that are resident at once, at most those for @p warps warps
template<class Kernel>
unsigned residentBlocks(Kernel kernel, size_t smem, size_t warps, int smCount)
{
    int perSm = 0;
    // the limit is the kernel's, for all threads and contexts: always the same value, with room for the deepest stacks
    if (smem > 48 * 1024)
        RYO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    RYO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kTravThreads, smem));
    return unsigned(std::min((warps + kTravWarps - 1) / kTravWarps, size_t(std::max(perSm, 1)) * smCount));
}

template<class Nodes, class Targets>
void launchWalk(const TraverseLaunch& t, const Nodes& nodes, const Targets& tgt, int smCount, cudaStream_t s)
{
    if (t.depthFirst)
    {
        auto depth        = depthKernel<Nodes, Targets>;
        const size_t smem = sizeof(int) * size_t(t.stackCapacity) * kTravWarps;
        depth<<<residentBlocks(depth, smem, size_t(t.numGroups), smCount), kTravThreads, smem, s>>>(t, nodes, tgt);
        RYO_LAUNCH_CHECK();
    }
    auto walk         = walkKernel<Nodes, Targets>;
    const size_t smem = (sizeof(int) * size_t(t.walkCapacity) + sizeof(WalkSmem)) * kTravWarps;
    walk<<<residentBlocks(walk, smem, size_t(t.numGroups) * t.subWalks, smCount), kTravThreads, smem, s>>>(t, nodes,
                                                                                                          tgt);
    RYO_LAUNCH_CHECK();
}

template<class Sink>
void launchFinish(const TraverseLaunch& t, const Sink& sink, int smCount, cudaStream_t s)
{
    // a block per group for as many groups as two rounds of eight blocks per SM take: the chains are long there
    // (100,003 bodies at theta 0.2, 1,563 groups: 81 -> 22 us, and 45 us since the items' sums are doubles; 60,001
    // Plummer bodies: 32 -> 17 us, now 21), but with 3,907 groups of a cube, whose parts are an item or two, it took 34
    // instead of 20 us
    const size_t numGroups = size_t(t.numGroups);
    if (t.subWalks == kWalkParts && numGroups <= size_t(16) * smCount)
        finishKernel<true><<<unsigned(std::min(numGroups, size_t(8) * smCount)), kFinishThreads, 0, s>>>(t, sink);
    else
    {
        const size_t blocks = ceilDiv(numGroups * kWarp, kFinishThreads);
        finishKernel<false><<<unsigned(std::min(blocks, size_t(8) * smCount)), kFinishThreads, 0, s>>>(t, sink);
    }
    RYO_LAUNCH_CHECK();
}

} // namespace ryo
