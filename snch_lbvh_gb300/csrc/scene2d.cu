// 2D scenes: the reference's scene<2> (include/snch_lbvh/scene.cuh:287-703) on
// the GPU -- line segments with silhouette VERTICES, the LBVH over 2D boxes and
// normal cones (bvh.cuh with aabb<float,2>, cone<float,2>), and the nearest /
// silhouette / ray / circle-sample queries (query.cuh, sample.cuh over the 2D
// functors), behind the snch_scene2_* C ABI.
//
// Compiled with -fmad=false: every + - * / is one binary32 operation in the
// reference's expression order, so topology, Morton codes, tree and boxes are
// bit-identical to the reference's; acosf / asinf / atan2f / logf / sinf / cosf
// are CUDA's. Rays and circle samples replay the reference's traversal order; the
// nearest and silhouette searches go near-first where that gives its answers, and replay
// it where it may not (settled2).
#include <algorithm>
#include <string>

#include "internal.h"
#include "warp_stack.cuh"

namespace snch
{
namespace
{

constexpr float kBvhOffset = 1e-3f;  // bvh_offset scene.cuh:12

struct B2  // aabb<float,2>, upper first
{
    float2 upper, lower;
};
struct C2  // cone<float,2>
{
    float2 axis;
    float half_angle, radius;
};

SNCH_DEV float2 f2(float x, float y) { return make_float2(x, y); }
SNCH_DEV float2 sub2(float2 a, float2 b) { return f2(a.x - b.x, a.y - b.y); }
SNCH_DEV float dot2(float2 a, float2 b) { return a.x * b.x + a.y * b.y; }
SNCH_DEV float len2(float2 a) { return sqrtf(a.x * a.x + a.y * a.y); }
SNCH_DEV float2 norm2(float2 v)
{
    const float n = len2(v);
    return f2(v.x / n, v.y / n);
}
SNCH_DEV float2 vload2(const float *__restrict__ v, int32_t i) { return f2(__ldg(v + 2 * i), __ldg(v + 2 * i + 1)); }
SNCH_DEV float2 centroid2(const B2 &b)
{
    return f2((b.upper.x + b.lower.x) * 0.5f, (b.upper.y + b.lower.y) * 0.5f);
}
SNCH_DEV B2 load_b2(const float4 *p)
{
    const float4 v = __ldcg(p);
    B2 b;
    b.upper = f2(v.x, v.y);
    b.lower = f2(v.z, v.w);
    return b;
}
SNCH_DEV C2 load_c2(const float4 *p)
{
    const float4 v = __ldcg(p);
    C2 c;
    c.axis = f2(v.x, v.y);
    c.half_angle = v.z;
    c.radius = v.w;
    return c;
}
SNCH_DEV float4 pack_b2(const B2 &b) { return make_float4(b.upper.x, b.upper.y, b.lower.x, b.lower.y); }
SNCH_DEV float4 pack_c2(const C2 &c) { return make_float4(c.axis.x, c.axis.y, c.half_angle, c.radius); }

// ------------------------------------------------------------------ topology
// compute_silhouettes scene.cuh:642-664: silhouette vertex v = {prev, v, next, -1}
// where later segments overwrite earlier ones (the last segment starting at v
// gives next, the last ending at v gives prev); build_bvh scene.cuh:666-683: a
// segment owns the endpoints no earlier segment touched, in (x, y) order.
__global__ void topo2_init_kernel(int64_t nv, int32_t *last_start, int32_t *last_end, int32_t *first_ref)
{
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v < nv)
    {
        last_start[v] = -1;
        last_end[v] = -1;
        first_ref[v] = 0x7FFFFFFF;
    }
}
__global__ void topo2_scan_kernel(const int32_t *__restrict__ segs, int64_t n, int32_t *last_start, int32_t *last_end,
                                  int32_t *first_ref)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int32_t a = segs[2 * i], b = segs[2 * i + 1];
    atomicMax(last_start + a, (int32_t)i);
    atomicMax(last_end + b, (int32_t)i);
    atomicMin(first_ref + a, (int32_t)i);
    atomicMin(first_ref + b, (int32_t)i);
}
__global__ void topo2_vertex_kernel(const int32_t *__restrict__ segs, int64_t nv, const int32_t *last_start,
                                    const int32_t *last_end, int4 *sv)
{
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nv)
        return;
    const int32_t s0 = last_start[v], s1 = last_end[v];
    int4 r = make_int4(-1, -1, -1, -1);
    // the later of the two writers of index 1 writes v either way
    if (s0 >= 0 || s1 >= 0)
        r.y = (int32_t)v;
    if (s0 >= 0)
        r.z = segs[2 * s0 + 1];
    if (s1 >= 0)
        r.x = segs[2 * s1];
    sv[v] = r;
}
__global__ void topo2_owned_kernel(const int32_t *__restrict__ segs, int64_t n, const int32_t *first_ref,
                                   int2 *seg_owned)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int32_t a = segs[2 * i], b = segs[2 * i + 1];
    int32_t own[2] = {-1, -1}, k = 0;
    if (first_ref[a] == (int32_t)i)
        own[k++] = a;
    if (b != a && first_ref[b] == (int32_t)i)
        own[k++] = b;
    seg_owned[i] = make_int2(own[0], own[1]);
}

// silhouette_vertex scene.cuh:291-384
SNCH_DEV bool sv_has_face(const int4 &sv, int f) { return f == 0 ? sv.z != -1 : sv.x != -1; }
SNCH_DEV float2 sv_face_normal(const float *verts, const int4 &sv, int f, bool do_normalize)
{
    const float2 pa = f == 0 ? vload2(verts, sv.y) : vload2(verts, sv.x);
    const float2 pb = f == 0 ? vload2(verts, sv.z) : vload2(verts, sv.y);
    const float2 s = sub2(pb, pa);
    const float2 nn = f2(s.y, -s.x);
    return do_normalize ? norm2(nn) : nn;
}
SNCH_DEV float2 sv_normal(const float *verts, const int4 &sv)
{
    float2 nn = f2(0.0f, 0.0f);
    if (sv_has_face(sv, 0))
    {
        const float2 a = sv_face_normal(verts, sv, 0, false);
        nn = f2(nn.x + a.x, nn.y + a.y);
    }
    if (sv_has_face(sv, 1))
    {
        const float2 a = sv_face_normal(verts, sv, 1, false);
        nn = f2(nn.x + a.x, nn.y + a.y);
    }
    return norm2(nn);
}

// Traversal records of the nearest and silhouette searches, written by the refit and
// the rank pass: expanding a node reads 48 consecutive bytes (80 with the cones)
// instead of its node, two boxes and, per child, a node again (144 bytes in six
// places); a leaf's segment and silhouette vertices are gathered in sorted order.
struct alignas(16) Inner2
{
    float4 lb, rb;  // child boxes
    uint4 ch;       // L, R, leaf info of L, of R: DFS rank | owned vertices << 30
};
struct Cones2
{
    float4 l, r;
};
// silhouette vertex of a leaf's segment: a = (position, unit normal of face 0),
// b = (unit normal of face 1, bits has_face(0) | has_face(1) << 1, vertex id)
struct Vert2
{
    float4 a, b;
};

// ------------------------------------------------------------------ build
struct Build2
{
    uint32_t n;
    const float *verts;
    const int32_t *segs;
    const int4 *sv;
    const int2 *seg_owned;
    uint32_t *scene_box;  // ordered uints: upper.xy (max), lower.xy (min)
    float4 *leaf_box, *leaf_cone;  // original order
    uint32_t *keys, *vals;
    NodeRec *nodes;
    float4 *aabbs, *cones;  // 2N-1 each
    uint32_t *flags, *sizes;
    Inner2 *inner;          // N-1
    Cones2 *inner_cones;    // N-1
    float4 *leaf_seg;       // N, sorted: both endpoints
    Vert2 *leaf_verts;      // 2N: slot 2 x position + k
};

// aabb_getter scene.cuh:420-432
SNCH_DEV B2 seg_box(float2 p0, float2 p1)
{
    B2 b;
    b.upper = f2(fmaxf(p0.x, p1.x) + kBvhOffset, fmaxf(p0.y, p1.y) + kBvhOffset);
    b.lower = f2(fminf(p0.x, p1.x) - kBvhOffset, fminf(p0.y, p1.y) - kBvhOffset);
    return b;
}
// cone_getter scene.cuh:434-494
SNCH_DEV C2 seg_cone(const Build2 &a, const B2 &bb, int2 owned)
{
    const float2 bc = centroid2(bb);
    C2 r;
    r.axis = f2(0.0f, 0.0f);
    r.half_angle = kPi;
    r.radius = 0.0f;
    bool any = false, all_two = true;
    const int32_t ow[2] = {owned.x, owned.y};
    for (int i = 0; i < 2; ++i)
    {
        if (ow[i] == -1)
            continue;
        const int4 sv = a.sv[ow[i]];
        const float2 nn = sv_normal(a.verts, sv);
        r.axis.x += nn.x;
        r.axis.y += nn.y;
        const float2 c = vload2(a.verts, sv.y);
        r.radius = smax(r.radius, len2(f2(c.x - bc.x, c.y - bc.y)));
        all_two = all_two && sv_has_face(sv, 0) && sv_has_face(sv, 1);
        any = true;
    }
    if (!any)
        r.half_angle = -kPi;
    else if (!all_two)
        r.half_angle = kPi;
    else
    {
        const float an = len2(r.axis);
        if (an > kEps)
        {
            r.axis.x /= an;
            r.axis.y /= an;
            r.half_angle = 0.0f;
            for (int i = 0; i < 2; ++i)
            {
                if (ow[i] == -1)
                    continue;
                const int4 sv = a.sv[ow[i]];
                float2 fn[2];
                fn[0] = sv_has_face(sv, 0) ? sv_face_normal(a.verts, sv, 0, true) : f2(0.0f, 0.0f);
                fn[1] = sv_has_face(sv, 1) ? sv_face_normal(a.verts, sv, 1, true) : f2(0.0f, 0.0f);
                for (int j = 0; j < 2; ++j)
                    r.half_angle = smax(r.half_angle, acosf(smax(-1.0f, smin(1.0f, dot2(r.axis, fn[j])))));
            }
        }
    }
    return r;
}

__global__ void init2_kernel(uint32_t *scene_box)
{
    if (threadIdx.x < 2)
        scene_box[threadIdx.x] = float_to_ordered(-INFINITY);
    else if (threadIdx.x < 4)
        scene_box[threadIdx.x] = float_to_ordered(INFINITY);
}
// leaf boxes and cones in original order, and the scene box (bvh.cuh:423-432), reduced in
// each block first (an atomic per warp and side: 1M segments 88 us, against 24 us here)
__global__ void __launch_bounds__(256) leaf2_kernel(Build2 a)
{
    __shared__ uint32_t s_box[4];
    if (threadIdx.x < 4)
        s_box[threadIdx.x] = float_to_ordered(threadIdx.x < 2 ? -INFINITY : INFINITY);
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    B2 b{f2(-INFINITY, -INFINITY), f2(INFINITY, INFINITY)};
    if (i < a.n)
    {
        const float2 p0 = vload2(a.verts, a.segs[2 * i]), p1 = vload2(a.verts, a.segs[2 * i + 1]);
        b = seg_box(p0, p1);
        a.leaf_box[i] = pack_b2(b);
        a.leaf_cone[i] = pack_c2(seg_cone(a, b, a.seg_owned[i]));
    }
    const uint32_t side[4] = {__reduce_max_sync(0xffffffffu, float_to_ordered(b.upper.x)),
                              __reduce_max_sync(0xffffffffu, float_to_ordered(b.upper.y)),
                              __reduce_min_sync(0xffffffffu, float_to_ordered(b.lower.x)),
                              __reduce_min_sync(0xffffffffu, float_to_ordered(b.lower.y))};
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 4; ++k)
            k < 2 ? atomicMax(s_box + k, side[k]) : atomicMin(s_box + k, side[k]);
    __syncthreads();
    if (threadIdx.x < 4)
        threadIdx.x < 2 ? atomicMax(a.scene_box + threadIdx.x, s_box[threadIdx.x])
                        : atomicMin(a.scene_box + threadIdx.x, s_box[threadIdx.x]);
}
// expand_bits morton_code.cuh:19-38; morton_code(float2) 83-91: the 3D spreading, x * 2 + y
SNCH_DEV uint32_t spread3(uint32_t v)
{
    v = (v | (v << 16)) & 0x070000FFu;
    v = (v | (v << 8)) & 0x0700F00Fu;
    v = (v | (v << 4)) & 0x430C30C3u;
    v = (v | (v << 2)) & 0x49249249u;
    return v;
}
// default_morton_code_calculator<Real,2> bvh.cuh:257-279
__global__ void __launch_bounds__(256) morton2_kernel(Build2 a)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n)
        return;
    const float4 lb = a.leaf_box[i];
    const float ux = ordered_to_float(a.scene_box[0]), uy = ordered_to_float(a.scene_box[1]);
    const float lx = ordered_to_float(a.scene_box[2]), ly = ordered_to_float(a.scene_box[3]);
    float px = (lb.x + lb.z) * 0.5f, py = (lb.y + lb.w) * 0.5f;
    px -= lx;
    py -= ly;
    px /= (ux - lx);
    py /= (uy - ly);
    const float res = 1024.0f;
    px = fminf(fmaxf(px * res, 0.0f), res - 1.0f);
    py = fminf(fmaxf(py * res, 0.0f), res - 1.0f);
    a.keys[i] = spread3((uint32_t)px) * 2 + spread3((uint32_t)py);
    a.vals[i] = i;
}

// rotate(float2) cone.cuh:266-275
SNCH_DEV float2 rotate2(float2 u, float2 v, float theta)
{
    const float det = u.x * v.y - u.y * v.x;
    theta *= copysignf(1.0f, det);
    const float ct = cosf(theta), st = sinf(theta);
    return f2(ct * u.x - st * u.y, st * u.x + ct * u.y);
}
// merge(cone<float,2>) cone.cuh:320-371; pi where the reference leaves the half
// angle unassigned (o_theta >= pi, lines 347-351), zeros for the axis / radius
// of a merge of two invalid cones (unset there)
SNCH_DEV C2 cone_merge2(const C2 &a, const C2 &b, float2 oa, float2 ob, float2 on)
{
    C2 r;
    r.axis = f2(0.0f, 0.0f);
    r.half_angle = 0.0f;
    r.radius = 0.0f;
    const bool va = a.half_angle >= 0.0f, vb = b.half_angle >= 0.0f;
    if (va && vb)
    {
        float2 axis_a = a.axis, axis_b = b.axis;
        float ha = a.half_angle, hb = b.half_angle;
        const float2 da = sub2(on, oa), db = sub2(on, ob);
        r.radius = sqrtf(smax(a.radius * a.radius + (da.x * da.x + da.y * da.y),
                              b.radius * b.radius + (db.x * db.x + db.y * db.y)));
        if (hb > ha)
        {
            const float2 t = axis_a;
            axis_a = axis_b;
            axis_b = t;
            const float h = ha;
            ha = hb;
            hb = h;
        }
        const float theta = acosf(smax(-1.0f, smin(1.0f, dot2(axis_a, axis_b))));
        if (smin(theta + hb, kPi) <= ha)
        {
            r.axis = axis_a;
            r.half_angle = ha;
            return r;
        }
        const float o_theta = (ha + theta + hb) / 2.0f;
        if (o_theta >= kPi)
        {
            r.axis = axis_a;
            r.half_angle = kPi;
            return r;
        }
        r.axis = rotate2(axis_a, axis_b, o_theta - ha);
        r.half_angle = o_theta;
    }
    else if (va)
        r = a;
    else if (vb)
        r = b;
    else
        r.half_angle = -kPi;
    return r;
}

// Leaf j's position in the reference's full depth-first order (leaf children of an
// expanded node left then right, then the right subtree, then the left one), into its
// parent's record; the near-first searches resolve exact ties with it.
SNCH_DEV void rank2(const Build2 &a, uint32_t j)
{
    const uint32_t n = a.n, ni = n - 1;
    if (j < ni)  // the child ids of internal node j
    {
        const uint4 rec = __ldg(reinterpret_cast<const uint4 *>(a.nodes + j));  // parent, left, right, object
        *reinterpret_cast<uint2 *>(&a.inner[j].ch) = make_uint2(rec.y, rec.z);
    }
    const uint32_t parent = a.nodes[ni + j].parent;
    uint32_t node = ni + j, p = parent, r = 0, slot = 0;
    for (int level = 0; level < 96 && p < ni; ++level)
    {
        const uint4 rec = __ldg(reinterpret_cast<const uint4 *>(a.nodes + p));
        const uint32_t lleaf = rec.y >= ni ? 1u : 0u, rleaf = rec.z >= ni ? 1u : 0u;
        if (node == rec.y)
            r += lleaf ? 0u : rleaf + (rleaf ? 0u : __ldg(a.sizes + rec.z));
        else
            r += lleaf;
        if (level == 0)
            slot = node == rec.y ? 2u : 3u;
        node = p;
        p = rec.x;
    }
    if (parent >= ni)
        return;
    const uint32_t orig = a.vals[j];
    const int2 own = orig < n ? a.seg_owned[orig] : make_int2(-1, -1);
    const uint32_t info = (r & kLeafRankMask) | (uint32_t)((own.x != -1) + (own.y != -1)) << 30;
    reinterpret_cast<uint32_t *>(&a.inner[parent].ch)[slot] = info;
}

// bottom-up AABB + cone refit with arrival counters (bvh.cuh:517-604, one pass), bound by
// the chain of arrivals; the blocks from refit_blocks on rank the leaves meanwhile, which
// needs the nodes alone. Builds of 20,000 / 180,000 / 1M segments, us: 150 / 199 / 495 with
// the ranks in a launch after it, two fences around each arrival and a clear before it, 130 /
// 157 / 377 here (this kernel 40 / 51 / 193).
__global__ void __launch_bounds__(128) refit2_kernel(Build2 a, uint32_t refit_blocks)
{
    const uint32_t n = a.n, ni = n - 1;
    const bool ranks = blockIdx.x >= refit_blocks;
    const uint32_t j = (blockIdx.x - (ranks ? refit_blocks : 0u)) * blockDim.x + threadIdx.x;
    if (j >= n)
        return;
    if (ranks)
    {
        rank2(a, j);
        return;
    }
    const uint32_t orig = a.vals[j];
    if (orig >= n)
        return;
    const uint32_t leaf = ni + j;
    a.aabbs[leaf] = a.leaf_box[orig];
    a.cones[leaf] = a.leaf_cone[orig];
    const float2 p0 = vload2(a.verts, a.segs[2 * orig]), p1 = vload2(a.verts, a.segs[2 * orig + 1]);
    a.leaf_seg[j] = make_float4(p0.x, p0.y, p1.x, p1.y);
    const int2 own = a.seg_owned[orig];
    for (int k = 0; k < 2; ++k)
    {
        const int32_t v = k ? own.y : own.x;
        if (v == -1)
            continue;
        const int4 sv = a.sv[v];
        const bool h0 = sv_has_face(sv, 0), h1 = sv_has_face(sv, 1);
        const float2 pv = vload2(a.verts, sv.y);
        const float2 n0 = h0 ? sv_face_normal(a.verts, sv, 0, true) : f2(0.0f, 0.0f);
        const float2 n1 = h1 ? sv_face_normal(a.verts, sv, 1, true) : f2(0.0f, 0.0f);
        Vert2 r;
        r.a = make_float4(pv.x, pv.y, n0.x, n0.y);
        r.b = make_float4(n1.x, n1.y, __uint_as_float((h0 ? 1u : 0u) | (h1 ? 2u : 0u)), __int_as_float(v));
        a.leaf_verts[2 * (uint64_t)j + k] = r;
    }
    if (n == 1)
        return;
    uint32_t p = a.nodes[leaf].parent;
    for (int level = 0; level < 96 && p < ni; ++level)
    {
        const uint4 rec = __ldg(reinterpret_cast<const uint4 *>(a.nodes + p));  // parent, left, right, object
        if (arrive_acq_rel(a.flags + p) == 0u)
            return;
        const uint32_t L = rec.y, R = rec.z;
        const B2 lb = load_b2(a.aabbs + L), rb = load_b2(a.aabbs + R);
        const C2 lc = load_c2(a.cones + L), rc = load_c2(a.cones + R);
        B2 m;
        m.upper = f2(fmaxf(lb.upper.x, rb.upper.x), fmaxf(lb.upper.y, rb.upper.y));
        m.lower = f2(fminf(lb.lower.x, rb.lower.x), fminf(lb.lower.y, rb.lower.y));
        a.aabbs[p] = pack_b2(m);
        a.cones[p] = pack_c2(cone_merge2(lc, rc, centroid2(lb), centroid2(rb), centroid2(m)));
        a.inner[p].lb = pack_b2(lb);
        a.inner[p].rb = pack_b2(rb);
        a.inner_cones[p] = Cones2{pack_c2(lc), pack_c2(rc)};
        p = rec.x;
    }
}

// ------------------------------------------------------------------ queries
struct Tree2
{
    uint32_t n;
    const float *verts;
    const int32_t *segs;
    const int4 *sv;
    const int2 *seg_owned;
    const NodeRec *nodes;
    const float4 *aabbs, *cones;
    const Inner2 *inner;
    const Cones2 *inner_cones;
    const float4 *leaf_seg;
    const Vert2 *leaf_verts;
    const uint32_t *order;  // original segment of each sorted position
    uint32_t *status;
};
SNCH_DEV B2 unpack_b2(float4 v)
{
    B2 b;
    b.upper = f2(v.x, v.y);
    b.lower = f2(v.z, v.w);
    return b;
}
SNCH_DEV C2 unpack_c2(float4 v)
{
    C2 c;
    c.axis = f2(v.x, v.y);
    c.half_angle = v.z;
    c.radius = v.w;
    return c;
}
SNCH_DEV B2 node_box2(const Tree2 &t, uint32_t i)
{
    const float4 v = __ldg(t.aabbs + i);
    B2 b;
    b.upper = f2(v.x, v.y);
    b.lower = f2(v.z, v.w);
    return b;
}
// mindist / minmaxdist aabb.cuh:130-135, 161-180
SNCH_DEV float mindist2(const B2 &b, float2 p)
{
    const float dx = fminf(b.upper.x, fmaxf(b.lower.x, p.x)) - p.x;
    const float dy = fminf(b.upper.y, fmaxf(b.lower.y, p.y)) - p.y;
    return dx * dx + dy * dy;
}
SNCH_DEV float minmaxdist2(const B2 &b, float2 p)
{
    float rmx = (b.lower.x - p.x) * (b.lower.x - p.x), rmy = (b.lower.y - p.y) * (b.lower.y - p.y);
    float rMx = (b.upper.x - p.x) * (b.upper.x - p.x), rMy = (b.upper.y - p.y) * (b.upper.y - p.y);
    float t;
    if ((b.upper.x + b.lower.x) * 0.5f < p.x)
    {
        t = rmx;
        rmx = rMx;
        rMx = t;
    }
    if ((b.upper.y + b.lower.y) * 0.5f < p.y)
    {
        t = rmy;
        rmy = rMy;
        rMy = t;
    }
    return fminf(rmx + rMy, rMx + rmy);
}
// find_closest_point_line_segment(float2) scene.cuh:176-199: the squared length whose
// square root is the distance
SNCH_DEV float closest_point_segment2_sq(float2 pa, float2 pb, float2 x)
{
    const float2 u = sub2(pb, pa), v = sub2(x, pa);
    const float c1 = dot2(u, v);
    if (c1 <= 0.0f)
        return dot2(v, v);
    const float c2 = dot2(u, u);
    if (c2 <= c1)
    {
        const float2 w = sub2(x, pb);
        return dot2(w, w);
    }
    const float t = c1 / c2;
    const float2 pt = f2(pa.x + u.x * t, pa.y + u.y * t);
    const float2 w = f2(x.x - pt.x, x.y - pt.y);
    return dot2(w, w);
}
SNCH_DEV float2 load_pt2(const float *p, int64_t q) { return f2(__ldg(p + 2 * q), __ldg(p + 2 * q + 1)); }

// ---- where near-first gives the reference's answers
// The reference takes its stack in a fixed order and prunes stack entries by the best so
// far, but evaluates every leaf child of a node that it expands. Its child tests (nearest:
// mindist against the sibling's minmaxdist; silhouette: the cone) depend on the node and
// the query alone; the near-first searches keep them (a 2D box is inflated by 1e-3, so that
// the sibling test can cut off a nearer segment: dropping it would change answers). Its
// answer is the minimum over the leaves that those tests reach, the last one visited among
// equals, if no leaf at the minimum is ever pruned; any order then gives the same, with
// equals resolved by leaf rank. A leaf's box (and so each of its ancestors', which contain
// it) is never pruned while its mindist, as computed, is at most the square of its distance
// d, as computed. Exactly, the inflation keeps the box 1e-3 nearer than the element. With u
// = 2^-24, every coordinate (also the query's) at most M, the rounding can take away at most
//   box corner u M, mindist 2 u d, d and its square 3.5 u d, and for a segment the closest
//   point on it sqrt(2) u M + 2 u |segment| <= 7.1 u M
// so 8.1 u M + 5.5 u d < 1e-3 suffices for segments, u M + 5.5 u d < 1e-3 for vertices (1e-3
// / u = 16777): M to 1,700 and 8,000. Near-first against the reference's order: 180,000
// segments, 200k queries, nearest 0.18 / 2.26 ms, silhouettes 0.49 / 46.8 ms.
// Beyond (a scene at 1e5 from the origin, or a query as far from it, where two segments of
// one vertex tie as a rule) a lane goes near-first once more, pruning only what the same
// bounds leave no doubt of (reach2): so it sees every leaf at the minimum D. The reference
// sees such a leaf for certain if its parent's mindist, which it prunes by, is at most D
// (then so is that of every ancestor, whose box is no smaller, and its best is never below
// D). If one leaf at D is not certain in that way, the query replays the reference's order.
// 200k queries of a scene 2,000 across, nearest 195 us (replayed 1,403), of one 8,000 across,
// silhouettes 1.08 ms (replayed 38 ms); at 1e5 from the origin most warps hold a query that is
// in doubt: 1.7 and 22 ms.
constexpr float kMarginUlps = 16000.0f, kNearestUlps = 9.0f, kSilhouetteUlps = 2.0f, kDistanceUlps = 6.0f;
// what the coordinates (root box b, which holds them all, and p) take of the margin
SNCH_DEV float coordinate_ulps(float4 b, float2 p, float per_unit)
{
    return per_unit * fmaxf(fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))),
                            fmaxf(fabsf(p.x), fabsf(p.y)));
}
// an answer at distance d found near-first is the reference's
SNCH_DEV bool settled2(float used, float d) { return used + kDistanceUlps * d <= kMarginUlps; }
// a box at a squared mindist beyond this holds nothing at a distance of d or less
SNCH_DEV float reach2(float used, float d)
{
    const float r = d + (used + kDistanceUlps * d) * 5.9604644775390625e-8f;  // 2^-24
    return beyond_sq(r * r);
}

SNCH_DEV void leaf_nearest2(const Tree2 &t, uint32_t pos, uint32_t rank, float2 p, float &best, uint32_t &best_rank,
                            uint32_t &best_pos)
{
    const float4 g = __ldg(t.leaf_seg + pos);
    const float sq = closest_point_segment2_sq(f2(g.x, g.y), f2(g.z, g.w), p);
    if (sq > beyond_sq(best))
        return;  // d > best
    float d = sqrtf(sq);
    d *= d;
    if (d < best || (d == best && (best_pos == kInvalid || rank > best_rank)))
    {
        best = d;
        best_rank = rank;
        best_pos = pos;
    }
}
// The reference's order (query.cuh:239-318), one lane; t.n > 1. A call of its own, so that
// the near-first searches keep their registers.
struct Found2
{
    float best;   // nearest: squared distance; silhouette: distance
    uint32_t id;  // sorted position of the segment; silhouette: vertex
};
__device__ __noinline__ Found2 nearest2_in_order(Tree2 t, float2 p)
{
    const uint32_t ni = t.n - 1;
    uint32_t sn[kStackDepth];
    float sd[kStackDepth];
    Found2 f{INFINITY, kInvalid};
    int sp = 0;
    sn[sp] = 0;
    sd[sp++] = mindist2(node_box2(t, 0), p);
    while (sp > 0)
    {
        --sp;
        if (sd[sp] > f.best)
            continue;
        const Inner2 *rec = t.inner + sn[sp];
        const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
        const uint4 ch = __ldg(&rec->ch);
        const float Lmd = mindist2(lb, p), Rmd = mindist2(rb, p);
        const bool aL = Lmd <= minmaxdist2(rb, p), aR = Rmd <= minmaxdist2(lb, p);
        for (int k = 0; k < 2; ++k)
        {
            if (!(k ? aR : aL))
                continue;
            const uint32_t child = k ? ch.y : ch.x;
            if (child >= ni)
            {
                const float4 g = __ldg(t.leaf_seg + (child - ni));
                float d = sqrtf(closest_point_segment2_sq(f2(g.x, g.y), f2(g.z, g.w), p));
                d *= d;
                if (d <= f.best)
                    f = Found2{d, child - ni};
                continue;
            }
            if (sp >= kStackDepth)
            {
                atomicOr(t.status, kStatusStackOverflow);
                return Found2{NAN, kInvalid};
            }
            sn[sp] = child;
            sd[sp++] = k ? Rmd : Lmd;
        }
    }
    return f;
}
// A query that is not settled near-first: near-first within reach2, or in the reference's order
__device__ __noinline__ Found2 nearest2_unsettled(Tree2 t, float2 p)
{
    const uint32_t ni = t.n - 1;
    const float4 root = __ldg(t.aabbs);
    const float used = coordinate_ulps(root, p, kNearestUlps);
    uint32_t sn[kStackDepth];
    float sd[kStackDepth];
    Found2 f{INFINITY, kInvalid};
    uint32_t rank = 0, node = 0;
    float nd = mindist2(unpack_b2(root), p), lim = INFINITY;
    bool doubt = false;
    int sp = 0;
    for (;;)
    {
        const Inner2 *rec = t.inner + node;
        const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
        const uint4 ch = __ldg(&rec->ch);
        const float md[2] = {mindist2(lb, p), mindist2(rb, p)};
        const bool ok[2] = {md[0] <= minmaxdist2(rb, p), md[1] <= minmaxdist2(lb, p)};
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            const uint32_t child = k ? ch.y : ch.x, info = (k ? ch.w : ch.z) & kLeafRankMask;
            if (!ok[k] || child < ni || md[k] > lim)
                continue;
            const float4 g = __ldg(t.leaf_seg + (child - ni));
            float d = sqrtf(closest_point_segment2_sq(f2(g.x, g.y), f2(g.z, g.w), p));
            d *= d;
            if (!(d <= f.best))
                continue;
            const bool first = d < f.best || f.id == kInvalid;
            doubt = (first ? false : doubt) || !(nd <= d);
            if (first || info > rank)
            {
                f = Found2{d, child - ni};
                rank = info;
                lim = reach2(used, sqrtf(d));
            }
        }
        const bool pL = ok[0] && ch.x < ni && !(md[0] > lim), pR = ok[1] && ch.y < ni && !(md[1] > lim);
        if (pL || pR)
        {
            const bool left = pL && (!pR || md[0] <= md[1]);
            if (pL && pR)
            {
                if (sp >= kStackDepth)
                {
                    doubt = true;
                    break;
                }
                sn[sp] = left ? ch.y : ch.x;
                sd[sp++] = left ? md[1] : md[0];
            }
            node = left ? ch.x : ch.y;
            nd = left ? md[0] : md[1];
            continue;
        }
        while (sp > 0 && sd[sp - 1] > lim)
            --sp;
        if (sp == 0)
            break;
        --sp;
        node = sn[sp];
        nd = sd[sp];
    }
    return doubt ? nearest2_in_order(t, p) : f;
}
// what a nearest query of this point takes of the margin; unsettled from the start if the
// coordinates, or the distance to the scene, take all of it (or for a NaN point)
SNCH_DEV float nearest2_ulps(const Tree2 &t, float2 p)
{
    const float4 b = __ldg(t.aabbs);
    const float used = coordinate_ulps(b, p, kNearestUlps);
    return settled2(used, sqrtf(mindist2(unpack_b2(b), p))) ? used : INFINITY;
}
SNCH_DEV void store_nearest2(const Tree2 &t, int64_t q, float best, uint32_t pos, uint32_t *__restrict__ out_idx,
                             float *__restrict__ out_dist)
{
    out_idx[q] = pos == kInvalid ? kInvalid : __ldg(t.order + pos);
    out_dist[q] = sqrtf(best);
}
__global__ void __launch_bounds__(128) nearest2_kernel(Tree2 t, const float *__restrict__ pts, int64_t n,
                                                       uint32_t *__restrict__ out_idx, float *__restrict__ out_dist)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const float2 p = load_pt2(pts, q);
    uint32_t best_pos = kInvalid, best_rank = 0;
    float best = INFINITY;
    const uint32_t ni = t.n - 1;
    const float used = t.n > 1 ? nearest2_ulps(t, p) : 0.0f;
    if (t.n == 1)
        leaf_nearest2(t, 0u, 0u, p, best, best_rank, best_pos);
    else if (t.n > 1 && used < INFINITY)
    {
        uint32_t sn[kStackDepth];
        float sd[kStackDepth];
        int sp = 0;
        uint32_t node = 0;
        bool live = true;
        while (live)
        {
            const Inner2 *rec = t.inner + node;
            const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
            const uint4 ch = __ldg(&rec->ch);
            const uint32_t L = ch.x, R = ch.y;
            const float Lmd = mindist2(lb, p), Rmd = mindist2(rb, p);
            const bool aL = Lmd <= minmaxdist2(rb, p), aR = Rmd <= minmaxdist2(lb, p);
            if (aL && L >= ni && Lmd <= best)
                leaf_nearest2(t, L - ni, ch.z & kLeafRankMask, p, best, best_rank, best_pos);
            if (aR && R >= ni && Rmd <= best)
                leaf_nearest2(t, R - ni, ch.w & kLeafRankMask, p, best, best_rank, best_pos);
            const bool pL = aL && L < ni && Lmd <= best, pR = aR && R < ni && Rmd <= best;
            if (pL && pR)
            {
                if (sp > kStackDepth - 2)
                {
                    atomicOr(t.status, kStatusStackOverflow);
                    best_pos = kInvalid;
                    best = NAN;
                    break;
                }
                const bool l_first = Lmd <= Rmd;
                sn[sp] = l_first ? R : L;
                sd[sp] = l_first ? Rmd : Lmd;
                ++sp;
                node = l_first ? L : R;
                continue;
            }
            if (pL || pR)
            {
                node = pL ? L : R;
                continue;
            }
            live = false;
            while (sp > 0)
            {
                --sp;
                if (!(sd[sp] > best))
                {
                    node = sn[sp];
                    live = true;
                    break;
                }
            }
        }
    }
    if (t.n > 1 && (used == INFINITY || (best_pos != kInvalid && !settled2(used, sqrtf(best)))))
    {
        const Found2 f = nearest2_unsettled(t, p);
        best = f.best;
        best_pos = f.id;
    }
    store_nearest2(t, q, best, best_pos, out_idx, out_dist);
}

// is_silhouette_vertex scene.cuh:112-141
SNCH_DEV bool is_silhouette_vertex(float2 n0, float2 n1, float2 view_dir, float d, bool flip)
{
    const float precision = 1e-3f;
    const float sign = flip ? 1.0f : -1.0f;
    if (d <= precision)
        return sign * (n0.x * n1.y - n0.y * n1.x) > precision;
    const float2 vu = f2(view_dir.x / d, view_dir.y / d);
    const float dot0 = dot2(vu, n0), dot1 = dot2(vu, n1);
    if (fabsf(dot0) <= precision)
        return sign * dot1 > precision;
    if (fabsf(dot1) <= precision)
        return sign * dot0 > precision;
    return dot0 * dot1 < 0.0f;
}
// silhouette_distance_calculator scene.cuh:512-532 with
// find_closest_silhouette_point scene.cuh:354-381 for one owned vertex; key = rank * 4 +
// slot orders candidates like the reference's visits: among equal distances the last
// one, except at distance 0, after which no vertex is accepted (the first)
SNCH_DEV void vertex_candidate2(const Tree2 &t, uint64_t slot, uint32_t key, float2 o, bool flip, float &best,
                                uint32_t &best_key, int32_t &best_vert)
{
    const Vert2 *r = t.leaf_verts + slot;
    const float4 a = __ldg(&r->a), b = __ldg(&r->b);
    const float2 vd = f2(o.x - a.x, o.y - a.y);
    const float sq = dot2(vd, vd);
    if (sq > beyond_sq(best * best))
        return;  // d > best
    const float d = sqrtf(sq);
    if (!(d <= best))
        return;
    const bool is_sil = __float_as_uint(b.z) != 3u ||
                        is_silhouette_vertex(f2(a.z, a.w), f2(b.x, b.y), vd, d, flip);
    if (!is_sil)
        return;
    if (d < best || best_vert < 0 || (d > 0.0f ? key > best_key : key < best_key))
    {
        best = d;
        best_key = key;
        best_vert = __float_as_int(b.w);
    }
}
// overlap(cone<float,2>) cone.cuh:78-120 with project_to_plane(float2) 44-49
SNCH_DEV bool cone_overlap2(const C2 &bc, float2 o, const B2 &b, float dist_to_box)
{
    if (bc.half_angle >= kPi2 || dist_to_box < kEps)
        return true;
    const float2 c = centroid2(b);
    float2 v = f2(c.x - o.x, c.y - o.y);
    const float l = len2(v);
    v.x /= l;
    v.y /= l;
    const float dax = acosf(smax(-1.0f, smin(1.0f, dot2(bc.axis, v))));
    if (kPi2 >= dax - bc.half_angle && kPi2 <= dax + bc.half_angle)
        return true;
    if (l > bc.radius)
    {
        const float hs = bc.half_angle + asinf(bc.radius / l);
        return hs >= kPi2 ? true : (kPi2 >= dax - hs && kPi2 <= dax + hs);
    }
    const float2 e = f2(b.upper.x - c.x, b.upper.y - c.y);
    float d = dot2(e, f2(fabsf(v.x), fabsf(v.y)));
    const float s = l - d;
    if (s <= 0.0f)
        return true;
    d = fabsf(dot2(e, f2(fabsf(-v.y), fabsf(v.x))));
    const float hs = bc.half_angle + atan2f(d, s);
    return hs >= kPi2 ? true : (kPi2 >= dax - hs && kPi2 <= dax + hs);
}
// the same decision from the filter (cone_filter): 1 / 0, -1: left to the exact test
SNCH_DEV int cone_overlap2_fast(const C2 &bc, float2 o, const B2 &b, float dist_to_box)
{
    if (bc.half_angle >= kPi2 || dist_to_box < kEps)
        return 1;
    const float2 c = centroid2(b);
    const float2 v = f2(c.x - o.x, c.y - o.y);
    return cone_filter(bc.half_angle, bc.radius, __fmaf_rn(v.x, v.x, v.y * v.y),
                       __fmaf_rn(bc.axis.x, v.x, bc.axis.y * v.y));
}
SNCH_DEV bool cone_test2(const C2 &bc, float2 o, const B2 &b, float dist_to_box)
{
    const int f = cone_overlap2_fast(bc, o, b, dist_to_box);
    return f >= 0 ? f == 1 : cone_overlap2(bc, o, b, dist_to_box);
}
// Self-check, as cone_filter_check_kernel: random boxes, cones and points, half of them
// within 1e-3 rad of the decision. counts[0] agree, [1] disagree, [2] left to the exact test.
__global__ void cone_filter2_check_kernel(int64_t n, uint64_t seed, unsigned long long *counts)
{
    __shared__ unsigned long long s_c[3];
    if (threadIdx.x < 3)
        s_c[threadIdx.x] = 0;
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n)
    {
        uint64_t st = check_mix(seed ^ (0x632BE59BD9B4E019ull * (uint64_t)(i + 1)));
        const float2 c = f2(2.f * unit_rand(st) - 1.f, 2.f * unit_rand(st) - 1.f);
        const float2 h = f2(exp2f(-12.f + 11.f * unit_rand(st)), exp2f(-12.f + 11.f * unit_rand(st)));
        const B2 b{f2(c.x + h.x, c.y + h.y), f2(c.x - h.x, c.y - h.y)};
        C2 k;
        const float ph = 6.2831853f * unit_rand(st);
        k.axis = f2(cosf(ph), sinf(ph));
        k.half_angle = unit_rand(st) < 0.5f ? 0.3f * unit_rand(st) : kPi2 * unit_rand(st);
        k.radius = len2(h) * (0.5f + unit_rand(st));
        const float l = k.radius * exp2f(-1.f + 6.f * unit_rand(st));
        // direction at a chosen angle to the axis: random, or near the decision boundary
        float theta = 6.2831853f * unit_rand(st);
        if (unit_rand(st) < 0.5f)
        {
            const float hs = k.half_angle + (l > k.radius ? asinf(k.radius / l) : 0.f);
            theta = kPi2 + (unit_rand(st) < 0.5f ? -hs : hs) + 1e-3f * (2.f * unit_rand(st) - 1.f);
        }
        const float2 o = f2(c.x - l * cosf(ph + theta), c.y - l * sinf(ph + theta));
        const float md = mindist2(b, o);
        const int f = cone_overlap2_fast(k, o, b, md);
        atomicAdd(&s_c[f < 0 ? 2 : ((f == 1) == cone_overlap2(k, o, b, md) ? 0 : 1)], 1ull);
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_c[threadIdx.x])
        atomicAdd(counts + threadIdx.x, s_c[threadIdx.x]);
}
// The reference's order (query.cuh:326-423), one lane; t.n > 1
__device__ __noinline__ Found2 silhouette2_in_order(Tree2 t, float2 p, bool flip)
{
    const uint32_t ni = t.n - 1;
    uint32_t sn[kStackDepth];
    float sd[kStackDepth];
    Found2 f{INFINITY, (uint32_t)-1};
    int sp = 0;
    sn[sp] = 0;
    sd[sp++] = mindist2(node_box2(t, 0), p);
    while (sp > 0)
    {
        --sp;
        if (sd[sp] > f.best * f.best)
            continue;
        const uint32_t node = sn[sp];
        const uint4 ch = __ldg(&t.inner[node].ch);
        for (int k = 0; k < 2; ++k)
        {
            const B2 b = unpack_b2(__ldg(k ? &t.inner[node].rb : &t.inner[node].lb));
            const C2 c = unpack_c2(__ldg(k ? &t.inner_cones[node].r : &t.inner_cones[node].l));
            const float md = mindist2(b, p);
            if (!(c.half_angle >= 0.0f && cone_overlap2(c, p, b, md)))
                continue;
            const uint32_t child = k ? ch.y : ch.x;
            if (child >= ni)
            {
                // the owned vertices in turn, by the squared bound of the leaf so far
                float bound = f.best * f.best, d = INFINITY;
                uint32_t id = f.id;
                bool found = false;
                for (uint32_t e = 0; e < (k ? ch.w : ch.z) >> 30 && bound > 0.0f; ++e)
                {
                    const Vert2 *r = t.leaf_verts + 2 * (uint64_t)(child - ni) + e;
                    const float4 va = __ldg(&r->a), vb = __ldg(&r->b);
                    const float2 vd = f2(p.x - va.x, p.y - va.y);
                    const float l = len2(vd);
                    if (l * l <= bound && (__float_as_uint(vb.z) != 3u ||
                                           is_silhouette_vertex(f2(va.z, va.w), f2(vb.x, vb.y), vd, l, flip)))
                    {
                        d = l;
                        bound = l * l;
                        id = __float_as_uint(vb.w);
                        found = true;
                    }
                }
                if (found && d <= f.best)
                    f = Found2{d, id};
                continue;
            }
            if (sp >= kStackDepth)
            {
                atomicOr(t.status, kStatusStackOverflow);
                return Found2{NAN, (uint32_t)-1};
            }
            sn[sp] = child;
            sd[sp++] = md;
        }
    }
    return f;
}
// as nearest2_unsettled
__device__ __noinline__ Found2 silhouette2_unsettled(Tree2 t, float2 p, bool flip)
{
    const uint32_t ni = t.n - 1;
    const float4 root = __ldg(t.aabbs);
    const float used = coordinate_ulps(root, p, kSilhouetteUlps);
    uint32_t sn[kStackDepth];
    float sd[kStackDepth];
    Found2 f{INFINITY, (uint32_t)-1};
    uint32_t key = 0, node = 0;
    float nd = mindist2(unpack_b2(root), p), lim = INFINITY;
    bool doubt = false;
    int sp = 0;
    for (;;)
    {
        const Inner2 *rec = t.inner + node;
        const Cones2 *cr = t.inner_cones + node;
        const B2 box[2] = {unpack_b2(__ldg(&rec->lb)), unpack_b2(__ldg(&rec->rb))};
        const C2 cone[2] = {unpack_c2(__ldg(&cr->l)), unpack_c2(__ldg(&cr->r))};
        const uint4 ch = __ldg(&rec->ch);
        float md[2];
        bool ok[2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            md[k] = mindist2(box[k], p);
            ok[k] = !(md[k] > lim) && cone[k].half_angle >= 0.0f && cone_test2(cone[k], p, box[k], md[k]);
            const uint32_t child = k ? ch.y : ch.x, info = k ? ch.w : ch.z;
            for (uint32_t e = 0; ok[k] && child >= ni && e < info >> 30; ++e)
            {
                const Vert2 *r = t.leaf_verts + 2 * (uint64_t)(child - ni) + e;
                const float4 va = __ldg(&r->a), vb = __ldg(&r->b);
                const float2 vd = f2(p.x - va.x, p.y - va.y);
                const float d = len2(vd);
                if (!(d <= f.best) || (__float_as_uint(vb.z) == 3u &&
                                       !is_silhouette_vertex(f2(va.z, va.w), f2(vb.x, vb.y), vd, d, flip)))
                    continue;
                const bool first = d < f.best || f.id == (uint32_t)-1;
                const uint32_t ek = (info & kLeafRankMask) * 4u + e;
                doubt = (first ? false : doubt) || !(nd <= d * d);
                if (first || (d > 0.0f ? ek > key : ek < key))
                {
                    f = Found2{d, __float_as_uint(vb.w)};
                    key = ek;
                    lim = reach2(used, d);
                }
            }
        }
        const bool pL = ok[0] && ch.x < ni && !(md[0] > lim), pR = ok[1] && ch.y < ni && !(md[1] > lim);
        if (pL || pR)
        {
            const bool left = pL && (!pR || md[0] <= md[1]);
            if (pL && pR)
            {
                if (sp >= kStackDepth)
                {
                    doubt = true;
                    break;
                }
                sn[sp] = left ? ch.y : ch.x;
                sd[sp++] = left ? md[1] : md[0];
            }
            node = left ? ch.x : ch.y;
            nd = left ? md[0] : md[1];
            continue;
        }
        while (sp > 0 && sd[sp - 1] > lim)
            --sp;
        if (sp == 0)
            break;
        --sp;
        node = sn[sp];
        nd = sd[sp];
    }
    return doubt ? silhouette2_in_order(t, p, flip) : f;
}
SNCH_DEV float silhouette2_ulps(const Tree2 &t, float2 p)  // as nearest2_ulps
{
    const float4 b = __ldg(t.aabbs);
    const float used = coordinate_ulps(b, p, kSilhouetteUlps);
    return settled2(used, sqrtf(mindist2(unpack_b2(b), p))) ? used : INFINITY;
}
// query_device(nearest_silhouette) query.cuh:326-423 over segments, near-first; also the
// silhouette vertex (mesh vertex id) of the answer. kDefer: a query that is not done after
// kLaneTurns2 expansions is left to the next launch.
constexpr uint32_t kLaneTurns2 = 64;  // 48: 160,000 queries 389 -> 460 us; 96 the same
template <bool kDefer>
__global__ void __launch_bounds__(128) silhouette2_kernel(Tree2 t, const float *__restrict__ pts,
                                                          const uint8_t *__restrict__ flips, int64_t n,
                                                          float *__restrict__ out_dist, int32_t *__restrict__ out_vid,
                                                          DeferArgs defer)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const float2 p = load_pt2(pts, q);
    const bool flip = flips ? __ldg(flips + q) != 0 : false;
    float best = INFINITY;
    uint32_t best_key = 0;
    int32_t best_vert = -1;
    bool deferred = false;
    const uint32_t ni = t.n - 1;
    if (t.n == 1)
    {
        const int2 own = t.seg_owned[t.nodes[0].object];
        for (uint32_t k = 0; k < 2; ++k)
            if ((k ? own.y : own.x) != -1)
                vertex_candidate2(t, k, k, p, flip, best, best_key, best_vert);
    }
    else if (t.n > 1)
    {
        uint32_t sn[kStackDepth];
        float sd[kStackDepth];
        int sp = 0;
        uint32_t node = 0;
        bool live = true;
        uint32_t turns = kDefer ? kLaneTurns2 : 0xFFFFFFFFu;
        while (live)
        {
            if (kDefer && turns-- == 0)
            {
                deferred = true;
                break;
            }
            const Inner2 *rec = t.inner + node;
            const Cones2 *cr = t.inner_cones + node;
            const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
            const uint4 ch = __ldg(&rec->ch);
            const C2 lc = unpack_c2(__ldg(&cr->l)), rc = unpack_c2(__ldg(&cr->r));
            const uint32_t L = ch.x, R = ch.y;
            const float Lmd = mindist2(lb, p), Rmd = mindist2(rb, p);
            const float b2 = best * best;
            const bool hitL = Lmd <= b2 && lc.half_angle >= 0.0f && cone_test2(lc, p, lb, Lmd);
            const bool hitR = Rmd <= b2 && rc.half_angle >= 0.0f && cone_test2(rc, p, rb, Rmd);
            const uint32_t nL = hitL && L >= ni ? ch.z >> 30 : 0u, nR = hitR && R >= ni ? ch.w >> 30 : 0u;
            for (uint32_t k = 0; k < nL + nR; ++k)
            {
                const bool right = k >= nL;
                const uint32_t slot = right ? k - nL : k;
                vertex_candidate2(t, 2 * (uint64_t)(right ? R - ni : L - ni) + slot,
                                  ((right ? ch.w : ch.z) & kLeafRankMask) * 4u + slot, p, flip, best, best_key,
                                  best_vert);
            }
            const float b2n = best * best;
            const bool pL = hitL && L < ni && Lmd <= b2n, pR = hitR && R < ni && Rmd <= b2n;
            if (pL && pR)
            {
                if (sp > kStackDepth - 2)
                {
                    atomicOr(t.status, kStatusStackOverflow);
                    best = NAN;
                    best_vert = -1;
                    break;
                }
                const bool l_first = Lmd <= Rmd;
                sn[sp] = l_first ? R : L;
                sd[sp] = l_first ? Rmd : Lmd;
                ++sp;
                node = l_first ? L : R;
                continue;
            }
            if (pL || pR)
            {
                node = pL ? L : R;
                continue;
            }
            live = false;
            while (sp > 0)
            {
                --sp;
                if (!(sd[sp] > best * best))
                {
                    node = sn[sp];
                    live = true;
                    break;
                }
            }
        }
    }
    if (kDefer)
    {
        defer_query(defer, deferred, make_uint4((uint32_t)q, __float_as_uint(best), best_key, (uint32_t)best_vert));
        if (deferred)
            return;
    }
    out_dist[q] = best;
    if (out_vid)
        out_vid[q] = best_vert;
}

// The same searches, one query per warp: 32 nodes of its frontier a step (coop.cuh tells
// why; the tests are those above, the best candidate is reduced over the warp). One lane
// ends with its longest search: 20,000 silhouette queries of 180,000 segments take as long
// as 100,000.
SNCH_DEV bool nearest2_coop(const Tree2 &t, float2 p, float &best, uint32_t &best_rank, uint32_t &best_pos, CoopStack &s)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t ni = t.n - 1;
    __syncwarp();  // the previous query's last reads
    if (lane == 0)
    {
        s.node[0] = 0;
        s.md[0] = 0.0f;
    }
    int sp = 1;
    __syncwarp();
    for (int step = 0; sp > 0; ++step)
    {
        const int k = coop_take(t.n, sp, best < INFINITY, step);
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
        float Lmd = INFINITY, Rmd = INFINITY, cb = best;
        bool aL = false, aR = false;
        uint32_t cr = best_rank, cp = best_pos;
        if (act)
        {
            const Inner2 *rec = t.inner + node;
            const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
            const uint4 ch = __ldg(&rec->ch);
            L = ch.x;
            R = ch.y;
            Lmd = mindist2(lb, p);
            Rmd = mindist2(rb, p);
            aL = Lmd <= minmaxdist2(rb, p);
            aR = Rmd <= minmaxdist2(lb, p);
            if (aL && L >= ni && Lmd <= cb)
                leaf_nearest2(t, L - ni, ch.z & kLeafRankMask, p, cb, cr, cp);
            if (aR && R >= ni && Rmd <= cb)
                leaf_nearest2(t, R - ni, ch.w & kLeafRankMask, p, cb, cr, cp);
        }
        const bool found = cp != best_pos;
        if (__ballot_sync(full, found))
        {
            const uint32_t d = __reduce_min_sync(full, found ? __float_as_uint(cb) : 0xffffffffu);
            const bool tie = found && __float_as_uint(cb) == d;
            const uint32_t r = __reduce_max_sync(full, tie ? cr : 0u);
            const int src = __ffs(__ballot_sync(full, tie && cr == r)) - 1;
            best = __uint_as_float(d);
            best_rank = r;
            best_pos = __shfl_sync(full, cp, src);
        }
        if (!coop_push(s, sp, aL && L < ni && Lmd <= best, aR && R < ni && Rmd <= best, L, R, Lmd, Rmd))
            return false;
    }
    return true;
}
// The first lane_blocks blocks: a lane per query, for those that are unsettled from the start
// (a warp gains nothing on the reference's order).
__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    nearest2_coop_kernel(Tree2 t, const float *__restrict__ pts, int64_t n, uint32_t *__restrict__ out_idx,
                         float *__restrict__ out_dist, unsigned lane_blocks)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    if (blockIdx.x < lane_blocks)
    {
        const int64_t q = blockIdx.x * (int64_t)(32 * kCoopWarps) + threadIdx.x;
        if (q >= n)
            return;
        const float2 p = load_pt2(pts, q);
        if (nearest2_ulps(t, p) < INFINITY)
            return;
        const Found2 f = nearest2_unsettled(t, p);
        store_nearest2(t, q, f.best, f.id, out_idx, out_dist);
        return;
    }
    const int w = threadIdx.x >> 5;
    const int64_t q = (blockIdx.x - lane_blocks) * (int64_t)kCoopWarps + w;
    if (q >= n)
        return;
    const float2 p = load_pt2(pts, q);
    float best = INFINITY;
    uint32_t best_rank = 0, best_pos = kInvalid;
    if (!nearest2_coop(t, p, best, best_rank, best_pos, s_stack[w]))
    {
        if ((threadIdx.x & 31) == 0)
            atomicOr(t.status, kStatusStackOverflow);
        best_pos = kInvalid;
        best = NAN;
    }
    if ((threadIdx.x & 31) != 0)
        return;
    const float used = nearest2_ulps(t, p);
    if (used == INFINITY)
        return;
    if (best_pos != kInvalid && !settled2(used, sqrtf(best)))
    {
        const Found2 f = nearest2_unsettled(t, p);
        best = f.best;
        best_pos = f.id;
    }
    store_nearest2(t, q, best, best_pos, out_idx, out_dist);
}

SNCH_DEV bool silhouette2_coop(const Tree2 &t, float2 p, bool flip, float &best, uint32_t &best_key, int32_t &best_vert,
                               CoopStack &s)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t ni = t.n - 1;
    __syncwarp();
    if (lane == 0)
    {
        s.node[0] = 0;
        s.md[0] = 0.0f;
    }
    int sp = 1;
    __syncwarp();
    for (int step = 0; sp > 0; ++step)
    {
        const int k = coop_take(t.n, sp, best < INFINITY, step);
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
        uint32_t L = kInvalid, R = kInvalid, ck = best_key;
        float Lmd = INFINITY, Rmd = INFINITY, cb = best;
        bool hitL = false, hitR = false;
        int32_t cv = best_vert;
        if (act)
        {
            const Inner2 *rec = t.inner + node;
            const Cones2 *cr = t.inner_cones + node;
            const B2 lb = unpack_b2(__ldg(&rec->lb)), rb = unpack_b2(__ldg(&rec->rb));
            const uint4 ch = __ldg(&rec->ch);
            const C2 lc = unpack_c2(__ldg(&cr->l)), rc = unpack_c2(__ldg(&cr->r));
            L = ch.x;
            R = ch.y;
            Lmd = mindist2(lb, p);
            Rmd = mindist2(rb, p);
            hitL = Lmd <= b2 && lc.half_angle >= 0.0f && cone_test2(lc, p, lb, Lmd);
            hitR = Rmd <= b2 && rc.half_angle >= 0.0f && cone_test2(rc, p, rb, Rmd);
            const uint32_t nL = hitL && L >= ni ? ch.z >> 30 : 0u, nR = hitR && R >= ni ? ch.w >> 30 : 0u;
            for (uint32_t i = 0; i < nL + nR; ++i)
            {
                const bool right = i >= nL;
                const uint32_t slot = right ? i - nL : i;
                vertex_candidate2(t, 2 * (uint64_t)(right ? R - ni : L - ni) + slot,
                                  ((right ? ch.w : ch.z) & kLeafRankMask) * 4u + slot, p, flip, cb, ck, cv);
            }
        }
        const bool found = cv != best_vert || ck != best_key;
        if (__ballot_sync(full, found))
        {
            const uint32_t d = __reduce_min_sync(full, found ? __float_as_uint(cb) : 0xffffffffu);
            const bool tie = found && __float_as_uint(cb) == d;
            const uint32_t order = __uint_as_float(d) > 0.0f ? ck : ~ck;
            const uint32_t o = __reduce_max_sync(full, tie ? order : 0u);
            const int src = __ffs(__ballot_sync(full, tie && order == o)) - 1;
            best = __uint_as_float(d);
            best_key = __shfl_sync(full, ck, src);
            best_vert = __shfl_sync(full, cv, src);
        }
        const float b2n = best * best;
        if (!coop_push(s, sp, hitL && L < ni && Lmd <= b2n, hitR && R < ni && Rmd <= b2n, L, R, Lmd, Rmd))
            return false;
    }
    return true;
}
// kSettle: the answer is settled here (silhouette2_coop_kernel), not by the pass after
template <bool kSettle>
SNCH_DEV void silhouette2_coop_query(const Tree2 &t, const float *__restrict__ pts, const uint8_t *__restrict__ flips,
                                     float *__restrict__ out_dist, int32_t *__restrict__ out_vid, int64_t q, float best,
                                     uint32_t best_key, int32_t best_vert, CoopStack &s)
{
    const bool flip = flips ? __ldg(flips + q) != 0 : false;
    const float2 p = load_pt2(pts, q);
    if (!silhouette2_coop(t, p, flip, best, best_key, best_vert, s))
    {
        if ((threadIdx.x & 31) == 0)
            atomicOr(t.status, kStatusStackOverflow);
        best = NAN;
        best_vert = -1;
    }
    if ((threadIdx.x & 31) != 0)
        return;
    if (kSettle)
    {
        const float used = silhouette2_ulps(t, p);
        if (used == INFINITY)
            return;  // answered by a lane of its own
        if (best_vert >= 0 && !settled2(used, best))
        {
            const Found2 f = silhouette2_unsettled(t, p, flip);
            best = f.best;
            best_vert = (int32_t)f.id;
        }
    }
    out_dist[q] = best;
    if (out_vid)
        out_vid[q] = best_vert;
}
__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    silhouette2_coop_kernel(Tree2 t, const float *__restrict__ pts, const uint8_t *__restrict__ flips, int64_t n,
                            float *__restrict__ out_dist, int32_t *__restrict__ out_vid, unsigned lane_blocks)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    if (blockIdx.x < lane_blocks)  // as nearest2_coop_kernel
    {
        const int64_t q = blockIdx.x * (int64_t)(32 * kCoopWarps) + threadIdx.x;
        if (q >= n)
            return;
        const float2 p = load_pt2(pts, q);
        if (silhouette2_ulps(t, p) < INFINITY)
            return;
        const Found2 f = silhouette2_unsettled(t, p, flips ? __ldg(flips + q) != 0 : false);
        out_dist[q] = f.best;
        if (out_vid)
            out_vid[q] = (int32_t)f.id;
        return;
    }
    const int w = threadIdx.x >> 5;
    const int64_t q = (blockIdx.x - lane_blocks) * (int64_t)kCoopWarps + w;
    if (q < n)
        silhouette2_coop_query<true>(t, pts, flips, out_dist, out_vid, q, INFINITY, 0u, -1, s_stack[w]);
}
__global__ void __launch_bounds__(32 * kCoopWarps, 16)
    silhouette2_finish_kernel(Tree2 t, const float *__restrict__ pts, const uint8_t *__restrict__ flips,
                              float *__restrict__ out_dist, int32_t *__restrict__ out_vid, DeferArgs d)
{
    __shared__ CoopStack s_stack[kCoopWarps];
    uint4 e;
    for (uint32_t i = first_deferred(); take_deferred(d, i, e); i = next_deferred(d))
        silhouette2_coop_query<false>(t, pts, flips, out_dist, out_vid, (int64_t)e.x, __uint_as_float(e.y), e.z,
                                      (int32_t)e.w, s_stack[threadIdx.x >> 5]);
}

// After the lanes' silhouette searches: the queries that are not settled, a lane each. (The
// call in the search's own kernel took it from 48 registers to 54, 200k queries 481 -> 559 us;
// this pass takes 4 us.)
__global__ void __launch_bounds__(128) silhouette2_settle_kernel(Tree2 t, const float *__restrict__ pts,
                                                                 const uint8_t *__restrict__ flips, int64_t n,
                                                                 float *__restrict__ out_dist,
                                                                 int32_t *__restrict__ out_vid)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const float2 p = load_pt2(pts, q);
    const float d = out_dist[q];  // infinite: none found, so nothing was pruned
    if (settled2(coordinate_ulps(__ldg(t.aabbs), p, kSilhouetteUlps), d < INFINITY ? d : 0.0f))
        return;
    const Found2 f = silhouette2_unsettled(t, p, flips ? __ldg(flips + q) != 0 : false);
    out_dist[q] = f.best;
    if (out_vid)
        out_vid[q] = (int32_t)f.id;
}

// intersects_d(ray<float,2>) aabb.cuh:366-390
SNCH_DEV bool ray_box2(float2 o, float2 inv, const B2 &b, float max_dist, float &dist)
{
    float t1 = (b.lower.x - o.x) * inv.x, t2 = (b.upper.x - o.x) * inv.x;
    float tmin = fminf(t1, t2), tmax = fmaxf(t1, t2);
    t1 = (b.lower.y - o.y) * inv.y;
    t2 = (b.upper.y - o.y) * inv.y;
    tmin = fmaxf(tmin, fminf(t1, t2));
    tmax = fminf(tmax, fmaxf(t1, t2));
    if (tmax >= tmin && tmax >= 0.0f && tmin <= max_dist)
    {
        dist = tmin >= 0.0f ? tmin : 0.0f;
        return true;
    }
    return false;
}
// scene<2>::intersect_test scene.cuh:555-583
SNCH_DEV bool ray_segment(float2 o, float2 dir, float2 p0, float2 p1, float &t, float &s)
{
    const float2 sd = sub2(p1, p0);
    const float D = dir.x * (-sd.y) + dir.y * sd.x;
    if (fabsf(D) < kEps)
        return false;
    const float inv = __frcp_rn(D);
    const float tt = ((p0.x - o.x) * (-sd.y) - (p0.y - o.y) * (-sd.x)) * inv;
    const float ss = (dir.x * (p0.y - o.y) - dir.y * (p0.x - o.x)) * inv;
    if (ss >= -1e-3f && ss <= 1.0f + 1e-3f && tt >= 0.0f)
    {
        t = tt;
        s = ss;
        return true;
    }
    return false;
}
// query_device(ray_intersect) query.cuh:82-169 over segments, the reference's order;
// kAny: TestOnly = true (query.cuh:117-121), stop at the first accepted hit and
// write only the hit flag
template <bool kAny = false>
__global__ void __launch_bounds__(128) ray2_kernel(Tree2 t, const float *__restrict__ origins,
                                                   const float *__restrict__ dirs, const float *__restrict__ tmaxs,
                                                   int64_t n, uint8_t *__restrict__ out_hit, float *__restrict__ out_t,
                                                   float *__restrict__ out_s, uint32_t *__restrict__ out_idx)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const float2 o = load_pt2(origins, q), dir = load_pt2(dirs, q);
    const float2 inv = f2(1.0f / dir.x, 1.0f / dir.y);
    const float max_dist = __ldg(tmaxs + q);
    float min_dist = INFINITY, bs = 0.0f;
    bool found = false;
    uint32_t nearest = kInvalid;
    if (t.n > 0)
    {
        uint32_t sn[kStackDepth];
        float sd[kStackDepth];
        int sp = 0;
        sn[sp] = 0;
        sd[sp++] = INFINITY;
        do
        {
            --sp;
            const uint32_t node = sn[sp];
            if (sd[sp] > min_dist)
                continue;
            const uint32_t obj = t.nodes[node].object;
            if (obj != kInvalid)
            {
                float tt, ss;
                if (ray_segment(o, dir, vload2(t.verts, t.segs[2 * obj]), vload2(t.verts, t.segs[2 * obj + 1]), tt,
                                ss) &&
                    tt < max_dist && tt < min_dist)
                {
                    min_dist = tt;
                    found = true;
                    bs = ss;
                    nearest = obj;
                    if (kAny)
                        break;
                }
                continue;
            }
            const uint32_t L = t.nodes[node].left, R = t.nodes[node].right;
            float Ld = 0.0f, Rd = 0.0f;
            const bool Lh = ray_box2(o, inv, node_box2(t, L), max_dist, Ld);
            const bool Rh = ray_box2(o, inv, node_box2(t, R), max_dist, Rd);
            if (sp > kStackDepth - 2)
            {
                atomicOr(t.status, kStatusStackOverflow);
                found = false;
                nearest = kInvalid;
                min_dist = NAN;
                break;
            }
            if (Lh && Rh)
            {
                uint32_t closer = L, other = R;
                if (Rd < Ld)
                {
                    const float tmp = Ld;
                    Ld = Rd;
                    Rd = tmp;
                    closer = R;
                    other = L;
                }
                sn[sp] = other;
                sd[sp++] = Rd;
                sn[sp] = closer;
                sd[sp++] = Ld;
            }
            else if (Lh)
            {
                sn[sp] = L;
                sd[sp++] = Ld;
            }
            else if (Rh)
            {
                sn[sp] = R;
                sd[sp++] = Rd;
            }
        } while (sp > 0);
    }
    out_hit[q] = found ? 1 : 0;
    if (kAny)
        return;
    out_t[q] = min_dist;
    out_s[q] = bs;
    out_idx[q] = nearest;
}

// intersect_sphere(sphere<float,2>, aabb) aabb.cuh:433-449
SNCH_DEV bool circle_box(float2 c, float r, const B2 &b)
{
    const float cx = smax(b.lower.x, smin(c.x, b.upper.x)), cy = smax(b.lower.y, smin(c.y, b.upper.y));
    const float dx = cx - c.x, dy = cy - c.y;
    return dx * dx + dy * dy <= (r * r);
}
// scene<2>::intersect_sphere scene.cuh:585-608
SNCH_DEV bool circle_segment(float2 c, float radius, float2 p1, float2 p2)
{
    const float2 d = sub2(p2, p1);
    const float len_sq = d.x * d.x + d.y * d.y;
    float t = ((c.x - p1.x) * d.x + (c.y - p1.y) * d.y) / len_sq;
    t = smax(0.0f, smin(1.0f, t));
    const float dx = (p1.x + t * d.x) - c.x, dy = (p1.y + t * d.y) - c.y;
    return dx * dx + dy * dy <= (radius * radius);
}
// scene<2>::green_weight scene.cuh:610-617
SNCH_DEV float green_weight2(float2 x, float2 y)
{
    const float r = smax(len2(f2(x.x - y.x, x.y - y.y)), 1e-2f);
    return fabsf(logf(r) / (3.14159265358979323846f * 2.0f));
}
// sample_object_in_sphere sample.cuh:23-91 over segments (measurement_getter:
// segment length); pdf 0 where the reference leaves it unset
__global__ void __launch_bounds__(128) sample2_kernel(Tree2 t, const float *__restrict__ centers,
                                                      const float *__restrict__ radii, const float *__restrict__ us,
                                                      int64_t n, int32_t *__restrict__ out_idx,
                                                      float *__restrict__ out_pdf)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const float2 ctr = load_pt2(centers, q);
    const float rad = __ldg(radii + q);
    float u = __ldg(us + q);
    int32_t oi = -1;
    float opdf = 0.0f;
    if (t.n > 0)
    {
        uint32_t node = 0;
        float npdf = 1.0f;
        for (int level = 0; level < 128; ++level)
        {
            const uint32_t obj = t.nodes[node].object;
            if (obj != kInvalid)
            {
                const float2 p0 = vload2(t.verts, t.segs[2 * obj]), p1 = vload2(t.verts, t.segs[2 * obj + 1]);
                if (circle_segment(ctr, rad, p0, p1))
                {
                    oi = (int32_t)obj;
                    opdf = npdf;
                    opdf /= len2(f2(p0.x - p1.x, p0.y - p1.y));
                }
                break;
            }
            const uint32_t L = t.nodes[node].left, R = t.nodes[node].right;
            const B2 lb = node_box2(t, L), rb = node_box2(t, R);
            const float Lw = circle_box(ctr, rad, lb) ? green_weight2(ctr, centroid2(lb)) : 0.0f;
            const float Rw = circle_box(ctr, rad, rb) ? green_weight2(ctr, centroid2(rb)) : 0.0f;
            const float tw = Lw + Rw;
            if (!(tw > 0.0f))
                break;
            const float Lp = Lw / tw;
            if (u < Lp)
            {
                u /= Lp;
                node = L;
                npdf = Lp * npdf;
            }
            else
            {
                const float Rp = 1.0f - Lp;
                u = (u - Lp) / Rp;
                node = R;
                npdf = Rp * npdf;
            }
        }
    }
    out_idx[q] = oi;
    out_pdf[q] = opdf;
}
// sample_on_object scene.cuh:619-623 -> sample_line scene.cuh:29-32
__global__ void sample_point2_kernel(const float *verts, const int32_t *segs, uint32_t ns, const int32_t *idx,
                                     const float *u, int64_t n, float *out)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    const int32_t i = idx[q];
    if (i < 0 || (uint32_t)i >= ns)
    {
        out[2 * q] = NAN;
        out[2 * q + 1] = NAN;
        return;
    }
    const float2 pa = vload2(verts, segs[2 * i]), pb = vload2(verts, segs[2 * i + 1]);
    const float uu = u[q];
    out[2 * q] = pa.x + uu * (pb.x - pa.x);
    out[2 * q + 1] = pa.y + uu * (pb.y - pa.y);
}

inline unsigned blocks(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace
}  // namespace snch

using namespace snch;

struct snch_scene2_s
{
    uint32_t nv = 0, n = 0;
    float *verts = nullptr;
    int32_t *segs = nullptr;
    int4 *sv = nullptr;
    int2 *seg_owned = nullptr;
    int32_t *topo = nullptr;  // 3 x nv: last segment starting / ending at, first touching each vertex
    float4 *leaf_box = nullptr, *leaf_cone = nullptr, *aabbs = nullptr, *cones = nullptr;
    uint32_t *keys = nullptr, *vals = nullptr, *keys_tmp = nullptr, *vals_tmp = nullptr, *flags = nullptr,
             *sizes = nullptr, *small = nullptr;
    NodeRec *nodes = nullptr;
    Inner2 *inner = nullptr;
    Cones2 *inner_cones = nullptr;
    float4 *leaf_seg = nullptr;
    Vert2 *leaf_verts = nullptr;
    void *scratch = nullptr;
    bool built = false;
    Tree2 tree() const
    {
        return Tree2{n, verts, segs, sv, seg_owned, nodes, aabbs, cones, inner, inner_cones, leaf_seg, leaf_verts,
                     vals, small + 8};
    }
};

namespace
{
#define SNCH2_CUDA(expr)                                                                                 \
    do                                                                                                   \
    {                                                                                                    \
        cudaError_t e_ = (expr);                                                                         \
        if (e_ != cudaSuccess)                                                                           \
            return report_error(e_ == cudaErrorMemoryAllocation ? SNCH_ERR_OUT_OF_MEMORY : SNCH_ERR_CUDA, \
                                std::string(#expr) + ": " + cudaGetErrorString(e_));                     \
    } while (0)

inline cudaStream_t S2(snch_stream_t s) { return static_cast<cudaStream_t>(s); }

void free2(snch_scene2_s *s)
{
    void *ptrs[] = {s->verts, s->segs, s->sv, s->seg_owned, s->topo, s->leaf_box, s->leaf_cone, s->aabbs,
                    s->cones, s->keys, s->vals, s->keys_tmp, s->vals_tmp, s->flags, s->sizes, s->small,
                    s->nodes, s->inner, s->inner_cones, s->leaf_seg, s->leaf_verts, s->scratch};
    for (void *p : ptrs)
        if (p)
            cudaFree(p);
    delete s;
}
template <typename T>
cudaError_t dalloc2(T **p, size_t count)
{
    return cudaMalloc(reinterpret_cast<void **>(p), sizeof(T) * (count ? count : 1));
}
int check2(snch_scene2_t s, int64_t n, std::initializer_list<const void *> ptrs)
{
    if (!s)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "scene is NULL");
    if (!s->built)
        return report_error(SNCH_ERR_NOT_BUILT, "BVH is not built yet.");
    if (n < 0)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "negative query count");
    if (n > 0)
        for (const void *p : ptrs)
            if (!p)
                return report_error(SNCH_ERR_INVALID_ARGUMENT, "NULL query buffer");
    return SNCH_OK;
}
}  // namespace

namespace
{
// Batches of up to kCoopDirect2 queries are searched a warp each, so that they do not wait
// for the longest search of one lane; silhouette batches of up to kLanesFirst2 a lane each
// at first, and the long ones then a warp each; larger ones keep the chip busy with a lane
// each. Measured, a lane each / as chosen, us: nearest, 20,000 queries of 180,000 segments
// 128 / 113, 26,000 of 1,800 143 / 89; silhouettes 394 / 166, 218 / 133, 130,000 of 180,000
// 460 / 361 (200,000: 516 / 547; nearest with lanes first, 130,000: 179 / 195).
constexpr int64_t kCoopDirect2 = 24576, kLanesFirst2 = 131072;
// launch(d): the lanes, finish(d, blocks): the warps that finish their list; without memory
// for the list, or under capture (no allocation in the graph), direct(): a warp each (180,000
// segments, a lane / a warp each: 30,000 queries 2,391 / 320 us, 130,000 2,906 / 1,003)
template <typename Launch, typename Finish, typename Direct>
cudaError_t launch_lanes_first2(int64_t n, cudaStream_t st, Launch launch, Finish finish, Direct direct)
{
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess)
        return e;
    DeferArgs d;
    char *scratch = optional_scratch(256 + 16 * (size_t)n, st, false);
    if (!scratch)
    {
        direct();
        note_launch();
        return cudaGetLastError();
    }
    d.count = reinterpret_cast<uint32_t *>(scratch);
    d.list = reinterpret_cast<uint4 *>(scratch + 256);
    d.capacity = (uint32_t)n;
    e = cudaMemsetAsync(scratch, 0, 8, st);
    if (e == cudaSuccess)
    {
        launch(d);
        finish(d, 16 * (unsigned)sms);
        note_launch(2);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(scratch, st);
    return e != cudaSuccess ? e : f;
}
}  // namespace

extern "C" {

int snch_scene2_create(const float *verts_xy, int64_t nv, const int32_t *segs, int64_t ns, snch_scene2_t *out)
{
    if (!out)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "out_scene is NULL");
    *out = nullptr;
    if (nv < 0 || ns < 0 || (nv > 0 && !verts_xy) || (ns > 0 && !segs))
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "bad vertex or segment buffer");
    if (ns >= (int64_t(1) << 30) || nv >= (int64_t(1) << 31))
        return report_error(SNCH_ERR_TOO_LARGE, "at most 2^30 - 1 segments and 2^31 - 1 vertices are supported");
    for (int64_t i = 0; i < 2 * ns; ++i)
        if (segs[i] < 0 || segs[i] >= nv)
            return report_error(SNCH_ERR_INVALID_ARGUMENT,
                                "segment vertex index out of range at segment " + std::to_string(i / 2));
    snch_scene2_s *s = new snch_scene2_s();
    s->nv = (uint32_t)nv;
    s->n = (uint32_t)ns;
    const size_t n = s->n, nn = n ? 2 * n - 1 : 1;
    cudaError_t e = cudaSuccess;
    auto A = [&](cudaError_t x) {
        if (e == cudaSuccess)
            e = x;
    };
    A(dalloc2(&s->verts, 2 * (size_t)nv));
    A(dalloc2(&s->segs, 2 * n));
    A(dalloc2(&s->sv, (size_t)nv));
    A(dalloc2(&s->seg_owned, n));
    A(dalloc2(&s->topo, 3 * (size_t)nv));
    A(dalloc2(&s->leaf_box, n));
    A(dalloc2(&s->leaf_cone, n));
    A(dalloc2(&s->aabbs, nn));
    A(dalloc2(&s->cones, nn));
    A(dalloc2(&s->keys, n));
    A(dalloc2(&s->vals, n));
    A(dalloc2(&s->keys_tmp, n));
    A(dalloc2(&s->vals_tmp, n));
    A(dalloc2(&s->flags, n));
    A(dalloc2(&s->sizes, n));
    A(dalloc2(&s->small, 1056));
    A(dalloc2(&s->nodes, nn));
    A(dalloc2(&s->inner, n));
    A(dalloc2(&s->inner_cones, n));
    A(dalloc2(&s->leaf_seg, n));
    A(dalloc2(&s->leaf_verts, 2 * n));
    if (e == cudaSuccess)
        e = cudaMalloc(&s->scratch, std::max<size_t>(sort_scratch_bytes((uint32_t)std::max<size_t>(n, 1), 30), 256));
    if (e == cudaSuccess)
        e = cudaMemset(s->small, 0, 1056 * 4);
    if (e == cudaSuccess && nv)
        e = cudaMemcpy(s->verts, verts_xy, 8 * (size_t)nv, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n)
        e = cudaMemcpy(s->segs, segs, 8 * n, cudaMemcpyHostToDevice);
    if (e != cudaSuccess)
    {
        free2(s);
        return report_error(e == cudaErrorMemoryAllocation ? SNCH_ERR_OUT_OF_MEMORY : SNCH_ERR_CUDA,
                            std::string("2D scene: ") + cudaGetErrorString(e));
    }
    *out = s;
    return SNCH_OK;
}

int snch_scene2_destroy(snch_scene2_t s)
{
    if (!s)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "scene is NULL");
    free2(s);
    return SNCH_OK;
}

int snch_scene2_build(snch_scene2_t s, snch_stream_t stream)
{
    if (!s)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "scene is NULL");
    cudaStream_t st = S2(stream);
    const uint32_t n = s->n, nv = s->nv;
    int32_t *last_start = s->topo, *last_end = s->topo + nv, *first_ref = s->topo + 2 * (size_t)nv;
    if (nv)
    {
        topo2_init_kernel<<<blocks(nv, 256), 256, 0, st>>>(nv, last_start, last_end, first_ref);
        note_launch();
    }
    if (n)
    {
        topo2_scan_kernel<<<blocks(n, 256), 256, 0, st>>>(s->segs, n, last_start, last_end, first_ref);
        topo2_owned_kernel<<<blocks(n, 256), 256, 0, st>>>(s->segs, n, first_ref, s->seg_owned);
        note_launch(2);
    }
    if (nv)
    {
        topo2_vertex_kernel<<<blocks(nv, 256), 256, 0, st>>>(s->segs, nv, last_start, last_end, s->sv);
        note_launch();
    }
    SNCH2_CUDA(cudaGetLastError());
    if (n)
    {
        Build2 a{n, s->verts, s->segs, s->sv, s->seg_owned, s->small, s->leaf_box, s->leaf_cone, s->keys, s->vals,
                 s->nodes, s->aabbs, s->cones, s->flags, s->sizes, s->inner, s->inner_cones, s->leaf_seg,
                 s->leaf_verts};
        init2_kernel<<<1, 32, 0, st>>>(s->small);
        leaf2_kernel<<<blocks(n, 256), 256, 0, st>>>(a);
        const bool ranks = n <= kRankSortMax;
        if (ranks)
        {
            a.keys = s->keys_tmp;
            a.vals = s->vals_tmp;
        }
        morton2_kernel<<<blocks(n, 256), 256, 0, st>>>(a);
        note_launch(3);
        SNCH2_CUDA(cudaGetLastError());
        if (ranks)
            SNCH2_CUDA(rank_sort_pairs(a.keys, a.vals, s->keys, s->vals, n, st));
        else
            SNCH2_CUDA(radix_sort_pairs(s->keys, s->vals, s->keys_tmp, s->vals_tmp, n, 30, nullptr, s->scratch,
                                        s->small + 8, st));
        a.keys = s->keys;
        a.vals = s->vals;
        BuildArgs k{};
        k.num_tris = n;
        k.keys = s->keys;
        k.vals = s->vals;
        k.nodes = s->nodes;
        k.sizes = s->sizes;
        k.flags = s->flags;
        SNCH2_CUDA(launch_karras(k, st));
        refit2_kernel<<<2 * blocks(n, 128), 128, 0, st>>>(a, blocks(n, 128));
        note_launch();
        SNCH2_CUDA(cudaGetLastError());
    }
    s->built = true;
    return SNCH_OK;
}

int snch_scene2_get_device_status(snch_scene2_t s, uint32_t *out_bits, int reset, snch_stream_t stream)
{
    if (!s || !out_bits)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "scene and out_bits are required");
    SNCH2_CUDA(cudaMemcpyAsync(out_bits, s->small + 8, 4, cudaMemcpyDeviceToHost, S2(stream)));
    SNCH2_CUDA(cudaStreamSynchronize(S2(stream)));
    if (reset)
        SNCH2_CUDA(cudaMemsetAsync(s->small + 8, 0, 4, S2(stream)));
    return SNCH_OK;
}

int snch_scene2_export(snch_scene2_t s, int32_t *sv, int32_t *seg_owned, uint32_t *sorted_morton,
                       uint32_t *sorted_idx, uint32_t *nodes, float *aabbs, float *cones, snch_stream_t stream)
{
    int rc = check2(s, 0, {});
    if (rc != SNCH_OK)
        return rc;
    cudaStream_t st = S2(stream);
    const size_t n = s->n, nn = n ? 2 * n - 1 : 0;
    const auto cp = [&](void *dst, const void *src, size_t bytes) {
        return dst && bytes ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st) : cudaSuccess;
    };
    SNCH2_CUDA(cp(sv, s->sv, 16 * (size_t)s->nv));
    SNCH2_CUDA(cp(seg_owned, s->seg_owned, 8 * n));
    SNCH2_CUDA(cp(sorted_morton, s->keys, 4 * n));
    SNCH2_CUDA(cp(sorted_idx, s->vals, 4 * n));
    SNCH2_CUDA(cp(nodes, s->nodes, 16 * nn));
    SNCH2_CUDA(cp(aabbs, s->aabbs, 16 * nn));
    SNCH2_CUDA(cp(cones, s->cones, 16 * nn));
    return SNCH_OK;
}

int snch_scene2_query_nearest(snch_scene2_t s, const float *pts, int64_t n, uint32_t *idx, float *dist,
                              snch_stream_t stream)
{
    int rc = check2(s, n, {pts, idx, dist});
    if (rc != SNCH_OK || n == 0)
        return rc;
    const Tree2 t = s->tree();
    cudaStream_t st = S2(stream);
    if (t.n > 1 && n <= kCoopDirect2)
    {
        const unsigned lanes = blocks(n, 32 * kCoopWarps);
        nearest2_coop_kernel<<<lanes + blocks(n, kCoopWarps), 32 * kCoopWarps, 0, st>>>(t, pts, n, idx, dist, lanes);
    }
    else
        nearest2_kernel<<<blocks(n, 128), 128, 0, st>>>(t, pts, n, idx, dist);
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_scene2_query_silhouette(snch_scene2_t s, const float *pts, const uint8_t *flip, int64_t n, float *dist,
                                 int32_t *vertex, snch_stream_t stream)
{
    int rc = check2(s, n, {pts, dist});
    if (rc != SNCH_OK || n == 0)
        return rc;
    const Tree2 t = s->tree();
    cudaStream_t st = S2(stream);
    const auto settle = [&] {
        silhouette2_settle_kernel<<<blocks(n, 128), 128, 0, st>>>(t, pts, flip, n, dist, vertex);
        note_launch();
    };
    const auto direct = [&] {  // a warp per query
        const unsigned lanes = blocks(n, 32 * kCoopWarps);
        silhouette2_coop_kernel<<<lanes + blocks(n, kCoopWarps), 32 * kCoopWarps, 0, st>>>(t, pts, flip, n, dist,
                                                                                          vertex, lanes);
    };
    if (t.n > 1 && n > kCoopDirect2 && n <= kLanesFirst2)
    {
        SNCH2_CUDA(launch_lanes_first2(
            n, st,
            [&](const DeferArgs &d) {
                silhouette2_kernel<true><<<blocks(n, 128), 128, 0, st>>>(t, pts, flip, n, dist, vertex, d);
            },
            [&](const DeferArgs &d, unsigned g) {
                silhouette2_finish_kernel<<<g, 32 * kCoopWarps, 0, st>>>(t, pts, flip, dist, vertex, d);
                settle();
            },
            direct));
        return SNCH_OK;
    }
    if (t.n > 1 && n <= kCoopDirect2)
        direct();
    else
    {
        silhouette2_kernel<false><<<blocks(n, 128), 128, 0, st>>>(t, pts, flip, n, dist, vertex, DeferArgs());
        if (t.n > 1)
            settle();
    }
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_scene2_query_ray(snch_scene2_t s, const float *origins, const float *dirs, const float *tmax, int64_t n,
                          uint8_t *hit, float *t, float *seg_param, uint32_t *idx, snch_stream_t stream)
{
    int rc = check2(s, n, {origins, dirs, tmax, hit, t, seg_param, idx});
    if (rc != SNCH_OK || n == 0)
        return rc;
    ray2_kernel<<<blocks(n, 128), 128, 0, S2(stream)>>>(s->tree(), origins, dirs, tmax, n, hit, t, seg_param, idx);
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_scene2_query_ray_test(snch_scene2_t s, const float *origins, const float *dirs, const float *tmax,
                               int64_t n, uint8_t *hit, snch_stream_t stream)
{
    int rc = check2(s, n, {origins, dirs, tmax, hit});
    if (rc != SNCH_OK || n == 0)
        return rc;
    ray2_kernel<true><<<blocks(n, 128), 128, 0, S2(stream)>>>(s->tree(), origins, dirs, tmax, n, hit, nullptr,
                                                               nullptr, nullptr);
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_scene2_sample_in_circle(snch_scene2_t s, const float *centers, const float *radii, const float *u, int64_t n,
                                 int32_t *idx, float *pdf, snch_stream_t stream)
{
    int rc = check2(s, n, {centers, radii, u, idx, pdf});
    if (rc != SNCH_OK || n == 0)
        return rc;
    sample2_kernel<<<blocks(n, 128), 128, 0, S2(stream)>>>(s->tree(), centers, radii, u, n, idx, pdf);
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_scene2_sample_on_object(snch_scene2_t s, const int32_t *idx, const float *u, int64_t n, float *pts,
                                 snch_stream_t stream)
{
    int rc = check2(s, n, {idx, u, pts});
    if (rc != SNCH_OK || n == 0)
        return rc;
    sample_point2_kernel<<<blocks(n, 256), 256, 0, S2(stream)>>>(s->verts, s->segs, s->n, idx, u, n, pts);
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

int snch_selfcheck_cone_filter2(int64_t n, uint64_t seed, uint64_t *device_counts, snch_stream_t stream)
{
    if (n < 0 || !device_counts)
        return report_error(SNCH_ERR_INVALID_ARGUMENT, "bad count or NULL counts");
    if (n == 0)
        return SNCH_OK;
    cone_filter2_check_kernel<<<blocks(n, 256), 256, 0, S2(stream)>>>(
        n, seed, reinterpret_cast<unsigned long long *>(device_counts));
    note_launch();
    SNCH2_CUDA(cudaGetLastError());
    return SNCH_OK;
}

}  // extern "C"
