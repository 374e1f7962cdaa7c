// Cooperative searches: one nearest / silhouette query per warp.
//
// A per-lane search visits its nodes one after the other, and the longest
// search of a batch decides when a small batch ends: a point deep inside a
// closed mesh visits thousands of nodes (20,480-triangle sphere, 20,011
// silhouette queries: mean 589 visits, longest 6,216) while the rest of the GPU
// idles. Here the 32 lanes of a warp expand up to 32 nodes of ONE query's
// frontier per step: the warp's stack of (node, mindist) entries lives in
// shared memory, lane i takes the i-th entry from the top, tests both children
// of its node and evaluates its own leaves, the best candidate is reduced over
// the warp, and the children that pass go back on the stack, nearest on top.
// What bounds it: the latency of one record read per step (a chain of visits /
// 32 steps instead of visits), and for many queries the L1 requests of 32
// different records per step.
//
// Same answers as the per-lane near-first searches: every child test is the
// same, the answer is the minimum over the leaves reached, and exact ties are
// resolved by leaf rank (edge key), so the order of the visits is free.
#pragma once
#include "warp_stack.cuh"

// The edges of a step's leaves as (EdgeRec slot, tie key) items, so that lane i
// tests the i-th edge of the warp instead of each lane looping over its own: a
// step of 32 nodes has about 13 edges to test, in one round of loads instead of
// the four or five of its longest lane.
constexpr int kCoopEdges = 32 * 6;
struct CoopEdges
{
    uint32_t slot[kCoopEdges], key[kCoopEdges];
};

// one query, all 32 lanes with the same arguments; (best, best_rank, nearest) is
// the candidate the search starts with and then its answer. false: stack overflow
SNCH_DEV bool nearest_coop(const TreeView &t, f3 p, uint32_t root, float &best, uint32_t &best_rank, uint32_t &nearest,
                           CoopStack &s)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t ni = t.num_tris - 1;
    if (root == kInvalid)
        return true;
    if (root >= ni)  // a one-triangle tree or mesh
    {
        leaf_nearest_fast(t, root - ni, p, best, best_rank, nearest);
        return true;
    }
    const float rmd = mindist(load_root_box(t.aabbs + root), p);
    if (rmd > best)
        return true;
    __syncwarp();  // the previous query's last reads
    if (lane == 0)
    {
        s.node[0] = root;
        s.md[0] = rmd;
    }
    int sp = 1;
    __syncwarp();
    for (int step = 0; sp > 0; ++step)
    {
        const int k = coop_take(t.num_tris, sp, best < INFINITY, step);
        uint32_t node = 0;
        bool act = false;
        if (lane < k)
        {
            node = s.node[sp - 1 - lane];
            act = !(s.md[sp - 1 - lane] > best);
        }
        sp -= k;
        if (__ballot_sync(full, act) == 0u)
            continue;
        uint32_t L = kInvalid, R = kInvalid;
        float Lmd = INFINITY, Rmd = INFINITY;
        float cb = best;
        uint32_t cr = best_rank, cn = nearest;
        if (act)
        {
            Box lb, rb;
            unpack_inner(load_inner(t.inner + node), lb, rb, L, R);
            Lmd = mindist(lb, p);
            Rmd = mindist(rb, p);
            if (L >= ni && Lmd <= cb)
                leaf_nearest_fast(t, L - ni, p, cb, cr, cn);
            if (R >= ni && Rmd <= cb)
                leaf_nearest_fast(t, R - ni, p, cb, cr, cn);
        }
        // the best of the lanes' new candidates: smallest distance, then the larger rank
        const bool found = cn != nearest;
        if (__ballot_sync(full, found))
        {
            const uint32_t d = __reduce_min_sync(full, found ? __float_as_uint(cb) : 0xffffffffu);
            const bool tie = found && __float_as_uint(cb) == d;
            const uint32_t r = __reduce_max_sync(full, tie ? cr : 0u);
            const int src = __ffs(__ballot_sync(full, tie && cr == r)) - 1;
            best = __uint_as_float(d);
            best_rank = r;
            nearest = __shfl_sync(full, cn, src);
        }
        if (!coop_push(s, sp, L < ni && Lmd <= best, R < ni && Rmd <= best, L, R, Lmd, Rmd))
            return false;
    }
    return true;
}

// the search and the results of query q
SNCH_DEV void nearest_coop_query(const TreeView &t, const float *__restrict__ pts, uint32_t *__restrict__ out_idx,
                                 float *__restrict__ out_dist, const SeedArgs &seed, int64_t q, float r0, float best,
                                 uint32_t best_rank, uint32_t nearest, CoopStack &s)
{
    const QueryRoot qr = query_root(t, q);
    if (!nearest_coop(t, load_point(pts, q), qr.node, best, best_rank, nearest, s))
    {
        if ((threadIdx.x & 31) == 0)
            atomicOr(t.status, kStatusStackOverflow);
        nearest = kInvalid;
        best = NAN;
    }
    if ((threadIdx.x & 31) != 0)
        return;
    const bool failed = seed.radius && nearest == kInvalid && r0 < INFINITY;
    if (seed.radius && nearest == kInvalid)
        best = INFINITY;  // nothing within the seed radius: the fallback pass answers it
    st_out(out_idx + q, nearest == kInvalid ? kInvalid : nearest - qr.tri_off);
    st_out(out_dist + q, sqrtf(best));
    if (seed.fail_flag)
        seed.fail_flag[q] = failed ? 1u : 0u;
}

__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    nearest_coop_kernel(TreeView t, const float *__restrict__ pts, int64_t n, uint32_t *__restrict__ out_idx,
                        float *__restrict__ out_dist, SeedArgs seed)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    const int w = threadIdx.x >> 5;
    const int64_t qi = blockIdx.x * (int64_t)kCoopWarps + w;
    if (qi >= n)
        return;
    const int64_t q = query_index(t, qi);
    const float r0 = seed.radius ? __ldg(seed.radius + q) : INFINITY;
    nearest_coop_query(t, pts, out_idx, out_dist, seed, q, r0, r0 * r0, 0u, kInvalid, s_stack[w]);
}

// the queries that the packets of a batch left (DeferArgs), one per warp, each from
// the candidate it had
__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    nearest_finish_kernel(TreeView t, const float *__restrict__ pts, uint32_t *__restrict__ out_idx,
                          float *__restrict__ out_dist, SeedArgs seed, DeferArgs d)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    uint4 e;
    for (uint32_t i = first_deferred(); take_deferred(d, i, e); i = next_deferred(d))
        if (e.x != kInvalid)
            nearest_coop_query(t, pts, out_idx, out_dist, seed, (int64_t)e.x,
                               seed.radius ? __ldg(seed.radius + e.x) : INFINITY, __uint_as_float(e.y), e.z, e.w,
                               s_stack[threadIdx.x >> 5]);
}

// one silhouette query, as nearest_coop
SNCH_DEV bool silhouette_coop(const TreeView &t, f3 p, bool flip, uint32_t root, float &best, uint32_t &best_key,
                              int32_t &best_edge, CoopStack &s, CoopEdges &items)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t ni = t.num_tris - 1;
    if (root == kInvalid)
        return true;
    if (root >= ni)
    {
        uint32_t n_edge = 0;
        leaf_silhouette_fast(t, root - ni, p, flip, best, best_key, best_edge, n_edge);
        return true;
    }
    const float rmd = mindist(load_root_box(t.aabbs + root), p);
    if (rmd > best * best)
        return true;
    __syncwarp();
    if (lane == 0)
    {
        s.node[0] = root;
        s.md[0] = rmd;
    }
    int sp = 1;
    __syncwarp();
    for (int step = 0; sp > 0; ++step)
    {
        const int k = coop_take(t.num_tris, sp, best < INFINITY, step);
        const float b2 = best * best;
        uint32_t node = 0;
        bool act = false;
        if (lane < k)
        {
            node = s.node[sp - 1 - lane];
            act = !(s.md[sp - 1 - lane] > b2);
        }
        sp -= k;
        if (__ballot_sync(full, act) == 0u)
            continue;
        uint32_t L = kInvalid, R = kInvalid;
        float Lmd = INFINITY, Rmd = INFINITY;
        bool hitL = false, hitR = false;
        float cb = best;
        uint32_t ck = best_key;
        int32_t ce = best_edge;
        uint32_t Linfo = 0, Rinfo = 0, nL = 0, nR = 0;
        if (act)
        {
            Box lb, rb;
            const InnerRec rec = load_inner(t.inner + node);
            const float4 *cr = reinterpret_cast<const float4 *>(t.inner_cones + node);
            InnerConeRec icr;
            icr.a = __ldg(cr);
            icr.b = __ldg(cr + 1);
            icr.c = __ldg(cr + 2);
            unpack_inner(rec, lb, rb, L, R);
            unpack_leaf_info(rec, Linfo, Rinfo);
            Cone lc, rc;
            unpack_cones(icr, lc, rc);
            Lmd = mindist(lb, p);
            Rmd = mindist(rb, p);
            hitL = Lmd <= b2 && lc.half_angle >= 0.0f && cone_test(lc, p, lb, Lmd);
            hitR = Rmd <= b2 && rc.half_angle >= 0.0f && cone_test(rc, p, rb, Rmd);
            nL = hitL && L >= ni ? Linfo >> 30 : 0u;
            nR = hitR && R >= ni ? Rinfo >> 30 : 0u;
        }
        // the leaf children's edges, listed for the whole warp
        uint32_t at = nL + nR;
        if (__ballot_sync(full, at != 0u))
        {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t y = __shfl_up_sync(full, at, o);
                if (lane >= o)
                    at += y;
            }
            const uint32_t edges = __shfl_sync(full, at, 31);
            at -= nL + nR;
            for (uint32_t e = 0; e < nL; ++e, ++at)
            {
                items.slot[at] = 3u * (L - ni) + e;
                items.key[at] = (Linfo & kLeafRankMask) * 4u + e;
            }
            for (uint32_t e = 0; e < nR; ++e, ++at)
            {
                items.slot[at] = 3u * (R - ni) + e;
                items.key[at] = (Rinfo & kLeafRankMask) * 4u + e;
            }
            __syncwarp();
            for (uint32_t i = lane; i < edges; i += 32)
                edge_record_candidate<true>(t, items.slot[i], items.key[i], p, flip, cb, ck, ce);
            __syncwarp();  // the next step's items overwrite these
        }
        // the best of the lanes' new candidates: smallest distance, then the larger
        // key, at distance 0 the smaller one
        const bool found = ce != best_edge;
        if (__ballot_sync(full, found))
        {
            const uint32_t d = __reduce_min_sync(full, found ? __float_as_uint(cb) : 0xffffffffu);
            const bool tie = found && __float_as_uint(cb) == d;
            const uint32_t order = __uint_as_float(d) > 0.0f ? ck : ~ck;
            const uint32_t o = __reduce_max_sync(full, tie ? order : 0u);
            const int src = __ffs(__ballot_sync(full, tie && order == o)) - 1;
            best = __uint_as_float(d);
            best_key = __shfl_sync(full, ck, src);
            best_edge = __shfl_sync(full, ce, src);
        }
        const float b2n = best * best;
        if (!coop_push(s, sp, hitL && L < ni && Lmd <= b2n, hitR && R < ni && Rmd <= b2n, L, R, Lmd, Rmd))
            return false;
    }
    return true;
}

// the search and the results of query q
SNCH_DEV void silhouette_coop_query(const TreeView &t, const float *__restrict__ pts, const uint8_t *__restrict__ flips,
                                    float *__restrict__ out_dist, int32_t *__restrict__ out_edge, const SeedArgs &seed,
                                    int64_t q, float r0, float best, uint32_t best_key, int32_t best_edge,
                                    CoopStack &s, CoopEdges &items)
{
    const bool flip = flips ? ld_in(flips + q) != 0 : false;
    const QueryRoot qr = query_root(t, q);
    if (!silhouette_coop(t, load_point(pts, q), flip, qr.node, best, best_key, best_edge, s, items))
    {
        if ((threadIdx.x & 31) == 0)
            atomicOr(t.status, kStatusStackOverflow);
        best = NAN;
        best_edge = -1;
    }
    if ((threadIdx.x & 31) != 0)
        return;
    const bool failed = seed.radius && best_edge < 0 && r0 < INFINITY;
    if (seed.radius && best_edge < 0)
        best = INFINITY;  // nothing within the seed radius: the fallback pass answers it
    st_out(out_dist + q, best);
    if (out_edge)
        st_out(out_edge + q, best_edge < 0 ? best_edge : best_edge - qr.edge_off);
    if (seed.fail_flag)
        seed.fail_flag[q] = failed ? 1u : 0u;
}

__global__ void __launch_bounds__(32 * kCoopWarps, 14)
    silhouette_coop_kernel(TreeView t, const float *__restrict__ pts, const uint8_t *__restrict__ flips, int64_t n,
                           float *__restrict__ out_dist, int32_t *__restrict__ out_edge, SeedArgs seed)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    __shared__ CoopEdges s_items[kCoopWarps];
    const int w = threadIdx.x >> 5;
    const int64_t qi = blockIdx.x * (int64_t)kCoopWarps + w;
    if (qi >= n)
        return;
    const int64_t q = query_index(t, qi);
    const float r0 = seed.radius ? __ldg(seed.radius + q) : INFINITY;
    silhouette_coop_query(t, pts, flips, out_dist, out_edge, seed, q, r0, r0, 0u, -1, s_stack[w], s_items[w]);
}

// (16 blocks, 64 registers: at 66 only 14 fit, and a finish takes 5 % longer)
__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    silhouette_finish_kernel(TreeView t, const float *__restrict__ pts, const uint8_t *__restrict__ flips,
                             float *__restrict__ out_dist, int32_t *__restrict__ out_edge, SeedArgs seed, DeferArgs d)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    __shared__ CoopEdges s_items[kCoopWarps];
    const int w = threadIdx.x >> 5;
    uint4 e;
    for (uint32_t i = first_deferred(); take_deferred(d, i, e); i = next_deferred(d))
        if (e.x != kInvalid)
            silhouette_coop_query(t, pts, flips, out_dist, out_edge, seed, (int64_t)e.x,
                                  seed.radius ? __ldg(seed.radius + e.x) : INFINITY, __uint_as_float(e.y), e.z,
                                  (int32_t)e.w, s_stack[w], s_items[w]);
}
