// Silhouette topology on the device: the reference does this on the host with
// std::map / std::unordered_map (include/snch_lbvh/scene.cuh:1135-1225).
//
// Every (triangle i, corner j) is an edge occurrence k = 3i+j of the edge
// (v_j, v_{j+1}). The occurrences are inserted into an open-addressing hash
// table keyed by (min vertex, max vertex); per distinct edge the table keeps
//   * the first occurrence (atomicMin)            -> edge ids in first-seen
//     order (assign_edge_indices, 1135-1166) and ownership (build_bvh, 1207-1225:
//     the first triangle that meets an edge owns it);
//   * the last occurrence of each orientation (atomicMax) -> the 4-vertex
//     record {opp0, min, max, opp1} that compute_silhouettes (1167-1204)
//     leaves after its in-order overwrites.
// All of these are order-independent reductions, so the result is
// deterministic and identical to the reference's host loop.
//
// An edge's entry is one 32-byte sector (EdgeSlot), so the compare-and-swap and the
// three reductions of an occurrence, and later its reads, touch one sector, and the
// table is laid out along the vertices: an edge starts at one of the places of its
// smaller vertex, so neighbouring triangles, which share vertices, work on
// neighbouring sectors that stay in L2 (most meshes number their vertices along
// their surface). After kLocalProbes taken places the probes jump by hashes of the whole
// key: a vertex with a million edges costs a few more probes (1M triangles 0.45 ms).
// One table each for keys, first and last occurrences, by a hash of the key: 2M
// triangles, insert + flags + scan + finalise 410 + 40 + 60 + 264 us, bound by random
// sectors, against 160 + 44 + 9 + 68 us (and a smaller table to clear) here.
#include "common.cuh"
#include "internal.h"

namespace snch
{
namespace
{

constexpr unsigned long long kEmpty = ~0ull;
constexpr uint32_t kLocalProbes = 4, kJumps = 64;

// all bits set = empty; last occurrences as kInvalid - (k + 1), so that every field's
// reduction is a minimum from the same initial value (kInvalid: none)
struct alignas(32) EdgeSlot
{
    unsigned long long key;  // smaller vertex << 32 | larger vertex
    uint32_t first, last_pos, last_neg;
    uint32_t pad[3];
};

// 1.5 slots per occurrence: a closed mesh fills a third of them, separate triangles two thirds
inline uint32_t table_capacity(uint32_t num_tris)
{
    const uint64_t c = 9ull * num_tris / 2 + 64;
    return (uint32_t)(c < 0xFFFFFFF0ull ? c : 0xFFFFFFF0ull);
}

struct Table
{
    EdgeSlot *slots;
    uint32_t cap;
    uint32_t stride;  // places per vertex (0: more vertices than slots, hash at once)
};

// the 64-bit finaliser of MurmurHash3 (A. Appleby, public domain)
__device__ __forceinline__ unsigned long long mix64(unsigned long long k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

// the slot of the edge (found or claimed), kInvalid if the table is full. Places of
// consecutive vertices with many edges each fill up into runs of thousands of full
// slots, so the probes after the local ones jump (a walk along such a run took 0.7 ms
// for a sphere of 10,000 triangles); at two thirds full, 64 jumps all fail once in 1e11,
// and the walk over the whole table after them only makes the search complete.
__device__ __forceinline__ uint32_t find_or_claim(const Table &t, uint32_t lo, uint32_t hi)
{
    const unsigned long long key = ((unsigned long long)lo << 32) | hi;
    unsigned long long h64 = mix64(key);
    uint32_t h = t.stride ? lo * t.stride + (uint32_t)((h64 & 0xFFFFFFFFull) * t.stride >> 32)
                          : (uint32_t)(((h64 >> 32) * t.cap) >> 32);
    for (uint64_t probe = 0; probe < kLocalProbes + kJumps + (uint64_t)t.cap; ++probe)
    {
        // a key never changes once set, so a cached read may only be late, seeing the
        // slot still empty; other keys are passed without an atomic (a fan of 1M
        // triangles queued 10 ms on its centre's few slots)
        unsigned long long prev = *reinterpret_cast<const unsigned long long *>(&t.slots[h].key);
        if (prev == kEmpty)
            prev = atomicCAS(&t.slots[h].key, kEmpty, key);
        if (prev == kEmpty || prev == key)
            return h;
        if (probe + 1 >= kLocalProbes && probe + 1 < kLocalProbes + kJumps)
        {
            h64 = mix64(h64 + 0x9E3779B97F4A7C15ull);
            h = (uint32_t)(((h64 >> 32) * t.cap) >> 32);
        }
        else
            h = h + 1 < t.cap ? h + 1 : 0;
    }
    return kInvalid;
}

// one thread per triangle: its three edges' probes are in flight together
__global__ void __launch_bounds__(256) edge_insert_kernel(const int32_t *__restrict__ tris, uint32_t num_tris, Table t,
                                                          uint32_t *__restrict__ slot_of, uint32_t *status)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_tris)
        return;
    const int32_t v[3] = {tris[3 * (uint64_t)i], tris[3 * (uint64_t)i + 1], tris[3 * (uint64_t)i + 2]};
    uint32_t slot[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        // compute_silhouettes swaps (J, K) only when v_J > v_K (orientation -1)
        const int32_t vj = v[j], vk = v[(j + 1) % 3];
        slot[j] = find_or_claim(t, (uint32_t)min(vj, vk), (uint32_t)max(vj, vk));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        const uint32_t k = 3 * i + j;
        slot_of[k] = slot[j];
        if (slot[j] == kInvalid)
        {
            atomicOr(status, kStatusHashFull);
            continue;
        }
        EdgeSlot *e = t.slots + slot[j];
        atomicMin(&e->first, k);
        atomicMin(v[j] > v[(j + 1) % 3] ? &e->last_neg : &e->last_pos, kInvalid - (k + 1));
    }
}

// "This occurrence is its edge's first", a bit per occurrence, and each word's count. An
// edge's id is the number of first occurrences before its own first one: the scanned
// counts of the words before it and the bits below it in its word. (One kernel that
// scanned the flags itself, by look-back, and stored each id in its slot took 112 us for
// 2M triangles, this and the scan of the words 44 + 9 us: the stores of the ids and the
// idle warps during the scan are gone.)
__global__ void __launch_bounds__(256) edge_first_kernel(Table t, const uint32_t *__restrict__ slot_of, uint32_t num_occ,
                                                         uint32_t *__restrict__ bits, uint32_t *__restrict__ counts)
{
    constexpr int kPer = 4;  // words per warp: their reads are in flight together
    const int lane = threadIdx.x & 31;
    const uint64_t w0 = (blockIdx.x * 8ull + (threadIdx.x >> 5)) * kPer;
    uint32_t slot[kPer], first[kPer];
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        const uint64_t k = 32 * (w0 + r) + lane;
        slot[r] = k < num_occ ? slot_of[k] : kInvalid;
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r)
        first[r] = slot[r] != kInvalid ? t.slots[slot[r]].first : kInvalid;
#pragma unroll
    for (int r = 0; r < kPer; ++r)
    {
        const uint32_t m = __ballot_sync(0xffffffffu, slot[r] != kInvalid && first[r] == (uint32_t)(32 * (w0 + r)) + lane);
        if (lane == 0 && 32 * (w0 + r) < num_occ)
        {
            bits[w0 + r] = m;
            counts[w0 + r] = (uint32_t)__popc(m);
        }
    }
}
// first occurrence -> edge id
struct EdgeIds
{
    const uint32_t *bits, *before;  // before: first occurrences in the words before
    __device__ __forceinline__ int32_t of(uint32_t first) const
    {
        const uint32_t w = first >> 5;
        return (int32_t)(__ldg(before + w) + __popc(__ldg(bits + w) & ((1u << (first & 31u)) - 1u)));
    }
};

__device__ __forceinline__ int32_t opposite_vertex(const int32_t *tris, uint32_t k)
{
    const uint32_t i = k / 3, j = k - 3 * i;
    return __ldg(tris + 3 * (uint64_t)i + (j + 2) % 3);
}

__device__ __forceinline__ void finalize_triangle(const int32_t *__restrict__ tris, uint32_t i, const Table &t,
                                                  const EdgeIds &ids, const uint32_t *__restrict__ slot_of,
                                                  int32_t *__restrict__ tri_edges,
                                                  int32_t *__restrict__ tri_owned, int32_t *__restrict__ edge_verts,
                                                  const float *verts, snch_triangle &obj,
                                                  snch_silhouette_edge *ref_edges)
{
    int32_t owned[3] = {-1, -1, -1};
    int p = 0;
    uint4 lo[3];
    uint32_t hi[3], slot[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        slot[j] = slot_of[3 * (uint64_t)i + j];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (slot[j] != kInvalid)
        {
            const uint4 *q = reinterpret_cast<const uint4 *>(t.slots + slot[j]);
            lo[j] = __ldg(q);      // key (low word: larger vertex), first, last_pos
            hi[j] = __ldg(&t.slots[slot[j]].last_neg);
        }
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        const uint32_t k = 3 * i + j;
        if (slot[j] == kInvalid)  // only after a full hash table (status bit set)
        {
            tri_edges[k] = -1;
            continue;
        }
        const int32_t e = ids.of(lo[j].z);
        tri_edges[k] = e;
        if (lo[j].z == k)
        {
#pragma unroll
            for (int o = 0; o < 3; ++o)
                if (o == p)
                    owned[o] = e;
            ++p;
            const uint32_t lp = kInvalid - lo[j].w, ln = kInvalid - hi[j];  // occurrence + 1, 0 = none
            int4 rec;
            rec.x = lp ? opposite_vertex(tris, lp - 1) : -1;
            rec.y = (int32_t)lo[j].y;
            rec.z = (int32_t)lo[j].x;
            rec.w = ln ? opposite_vertex(tris, ln - 1) : -1;
            reinterpret_cast<int4 *>(edge_verts)[e] = rec;
            snch_silhouette_edge se;
            se.indices[0] = rec.x;
            se.indices[1] = rec.y;
            se.indices[2] = rec.z;
            se.indices[3] = rec.w;
            se.vertices = verts;
            se.pad_ = 0;
            ref_edges[e] = se;
        }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        tri_owned[3 * (uint64_t)i + j] = owned[j];
        obj.vertex_indices[j] = tris[3 * (uint64_t)i + j];
        obj.silhouette_indices[j] = owned[j];
    }
    obj.vertices = verts;
    obj.silhouettes = ref_edges;
}


// Edge ids and ownership per triangle, the 4-vertex record per edge, and both in the
// reference's device layout (scene.cuh:708-722 silhouette_edge, 826-840 triangle) for the
// byte-compatible view: they depend on the topology alone, so a build over moved
// vertices does not write them again, and here the values are at hand (a kernel of their
// own per build took 87 us for 2M triangles). The 40-byte triangles are staged in shared
// memory and stored 16 bytes a lane.
__global__ void __launch_bounds__(256) edge_finalize_kernel(const int32_t *__restrict__ tris, uint32_t num_tris, Table t,
                                                            EdgeIds ids, const uint32_t *__restrict__ slot_of,
                                                            int32_t *__restrict__ tri_edges,
                                                            int32_t *__restrict__ tri_owned,
                                                            int32_t *__restrict__ edge_verts, const float *verts,
                                                            snch_triangle *objs, snch_silhouette_edge *ref_edges)
{
    __shared__ __align__(16) snch_triangle s_obj[256];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < num_tris)
        finalize_triangle(tris, i, t, ids, slot_of, tri_edges, tri_owned, edge_verts, verts, s_obj[threadIdx.x], ref_edges);
    __syncthreads();
    const uint32_t first = blockIdx.x * 256u, here = min(256u, num_tris - first);  // 256 triangles = 640 x 16 bytes
    const uint4 *from = reinterpret_cast<const uint4 *>(s_obj);
    uint4 *to = reinterpret_cast<uint4 *>(objs + first);
    const uint32_t vecs = here * (uint32_t)sizeof(snch_triangle) / 16u;
    for (uint32_t x = threadIdx.x; x < vecs; x += 256)
        to[x] = from[x];
    if (threadIdx.x == 0 && (here & 1u))  // 40 x odd: the last 8 bytes
        reinterpret_cast<uint2 *>(to + vecs)[0] = reinterpret_cast<const uint2 *>(from + vecs)[0];
}
inline uint32_t flag_words(uint32_t num_tris) { return (3 * num_tris + 31) / 32; }
struct Layout
{
    size_t slots, slot_of, bits, counts, before, scan, total;
};
inline Layout layout(uint32_t num_tris)
{
    Layout l;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t words = al(4 * (size_t)flag_words(num_tris));
    l.slots = 0;
    l.slot_of = l.slots + al(sizeof(EdgeSlot) * (size_t)table_capacity(num_tris));
    l.bits = l.slot_of + al(4 * 3 * (size_t)num_tris);
    l.counts = l.bits + words;
    l.before = l.counts + words;
    l.scan = l.before + words;
    l.total = l.scan + al(scan_flags_scratch_bytes(flag_words(num_tris)));
    // up to a quarter of a power of two, so that scenes of about the same size share
    // cached blocks
    size_t step = 256;
    while (8 * step <= l.total)
        step <<= 1;
    l.total = (l.total + step - 1) / step * step;
    return l;
}

}  // namespace

size_t topology_scratch_bytes(uint32_t num_tris) { return layout(num_tris).total; }

cudaError_t compute_topology(const int32_t *tris, uint32_t num_tris, uint32_t num_verts, int32_t *tri_edges,
                             int32_t *tri_owned, int32_t *edge_verts, uint32_t *num_edges, const float *verts,
                             snch_triangle *objs, snch_silhouette_edge *ref_edges, void *scratch, uint32_t *status,
                             cudaStream_t st)
{
    if (num_tris == 0)
        return cudaMemsetAsync(num_edges, 0, 4, st);
    const Layout l = layout(num_tris);
    char *base = static_cast<char *>(scratch);
    Table t;
    t.slots = reinterpret_cast<EdgeSlot *>(base + l.slots);
    t.cap = table_capacity(num_tris);
    t.stride = num_verts ? t.cap / num_verts : 0;
    uint32_t *slot_of = reinterpret_cast<uint32_t *>(base + l.slot_of);
    uint32_t *bits = reinterpret_cast<uint32_t *>(base + l.bits), *counts = reinterpret_cast<uint32_t *>(base + l.counts),
             *before = reinterpret_cast<uint32_t *>(base + l.before);
    cudaError_t e;
    if ((e = cudaMemsetAsync(t.slots, 0xff, sizeof(EdgeSlot) * (size_t)t.cap, st)) != cudaSuccess)
        return e;
    const int tb = 256;
    const uint32_t grid = (num_tris + tb - 1) / tb, words = flag_words(num_tris);
    edge_insert_kernel<<<grid, tb, 0, st>>>(tris, num_tris, t, slot_of, status);
    edge_first_kernel<<<(words + 31) / 32, tb, 0, st>>>(t, slot_of, 3 * num_tris, bits, counts);
    note_launch(2);
    if ((e = scan_flags(counts, before, words, num_edges, base + l.scan, status, st)) != cudaSuccess)
        return e;
    edge_finalize_kernel<<<grid, tb, 0, st>>>(tris, num_tris, t, EdgeIds{bits, before}, slot_of, tri_edges, tri_owned,
                                              edge_verts, verts, objs, ref_edges);
    note_launch();
    return cudaGetLastError();
}

}  // namespace snch
