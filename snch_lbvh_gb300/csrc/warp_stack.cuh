// What the one-query-per-warp searches of 3D (coop.cuh) and 2D scenes (scene2d.cu)
// share: the warp's stack, and the list of queries that one launch leaves to the next.
#pragma once
#include "common.cuh"

namespace snch
{

// Queries that a launch leaves to the next one, which finishes them one per warp
// (coop.cuh) from the candidate each has: the long packets at the end of a batch
// (leave_packet) and the long searches of a mid-sized batch (kDefer below).
struct DeferArgs
{
    uint4 *list = nullptr;      // (query, candidate's distance bits, rank or key, triangle or edge); nullptr: off
    uint32_t *count = nullptr;  // entries reserved; may pass capacity, by entries that are not in the list
    uint32_t capacity = 0;
};
// lists the entry of every lane with `add` set; called by any subset of a warp
SNCH_DEV void defer_query(const DeferArgs &d, bool add, uint4 entry)
{
    const uint32_t active = __activemask(), mask = __ballot_sync(active, add);
    if (!add)
        return;
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader)
        base = atomicAdd(d.count, (uint32_t)__popc(mask));
    base = __shfl_sync(mask, base, leader);
    d.list[base + __popc(mask & ((1u << lane) - 1u))] = entry;
}
// stack entries of a warp. A step that takes k entries adds at most k (2k
// children), so a warp takes fewer than 32 when fewer than 32 places are left
// below kCoopWide; one at a time adds one entry a level, and a tree over 64-bit
// keys is at most 65 levels deep.
constexpr int kCoopStack = 512, kCoopWide = kCoopStack - 72;
constexpr int kCoopWarps = 2;  // per block: a block's slot is freed by its slower warp
// Until a first candidate bounds the search, wide steps would mostly read nodes
// that the bound then rules out, so the first steps (one per bit of the triangle
// count, about a descent) take kCoopNarrow entries. 64,000 queries of the
// 2M-triangle scene, nearest / silhouette: 0.44 / 0.93 ms, against 0.52 / 1.14 ms
// with wide steps from the start; 2 or 4 entries: the same there, but small closed
// meshes lose (1,280 triangles, silhouette, 0.57 -> 0.62 / 0.68 ms).
constexpr int kCoopNarrow = 8;

struct CoopStack
{
    uint32_t node[kCoopStack];
    float md[kCoopStack];
};
// entries the next step takes from a stack of sp entries
SNCH_DEV int coop_take(uint32_t leaves, int sp, bool bounded, int step)
{
    const int width = bounded || step >= 32 - __clz(leaves) ? 32 : kCoopNarrow;
    return min(min(sp, width), max(1, kCoopWide - sp));
}

// pushes the children that pass (far ones first, then the near ones, lane 0's
// near child on top); false: the stack is full
SNCH_DEV bool coop_push(CoopStack &s, int &sp, bool pL, bool pR, uint32_t L, uint32_t R, float Lmd, float Rmd)
{
    const unsigned full = 0xffffffffu;
    const bool two = pL && pR, any = pL || pR;
    const bool l_near = two ? Lmd <= Rmd : pL;
    const uint32_t mf = __ballot_sync(full, two), mn = __ballot_sync(full, any);
    const int nf = __popc(mf), nn = __popc(mn);
    if (sp + nf + nn > kCoopStack)
        return false;
    uint32_t above;
    asm("mov.u32 %0, %%lanemask_gt;" : "=r"(above));
    __syncwarp();  // every lane has read its entry
    if (two)
    {
        const int at = sp + __popc(mf & above);
        s.node[at] = l_near ? R : L;
        s.md[at] = l_near ? Rmd : Lmd;
    }
    if (any)
    {
        const int at = sp + nf + __popc(mn & above);
        s.node[at] = l_near ? L : R;
        s.md[at] = l_near ? Lmd : Rmd;
    }
    sp += nf + nn;
    __syncwarp();
    return true;
}

// The list's entries for this warp (count[0] entries, count[1] those handed out beyond the
// first of each warp): the first is the warp's own place in the grid, for a list is often
// short, and thousands of warps that only ask for an entry would queue at the counter (30,000
// nearest queries at the surface of a 1,280-triangle sphere 44 -> 40 us).
SNCH_DEV uint32_t first_deferred() { return blockIdx.x * kCoopWarps + (threadIdx.x >> 5); }
SNCH_DEV uint32_t next_deferred(const DeferArgs &d)
{
    uint32_t i = 0;
    if ((threadIdx.x & 31) == 0)
        i = gridDim.x * kCoopWarps + atomicAdd(d.count + 1, 1u);
    return __shfl_sync(0xffffffffu, i, 0);
}
// entry i, or false past the end; an unused place comes back as query kInvalid
SNCH_DEV bool take_deferred(const DeferArgs &d, uint32_t i, uint4 &e)
{
    if (i >= min(__ldcg(d.count), d.capacity))
        return false;
    e = __ldcg(d.list + i);
    return true;
}

}  // namespace snch
