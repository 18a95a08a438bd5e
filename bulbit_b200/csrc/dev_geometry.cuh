// BVH traversal and ray-primitive tests on the device.
//
// Restates, operation for operation, BVH::RayCast (include/bulbit/bvh.h:102-155),
// BoundingBox3::TestRay (include/bulbit/bounding_box.h:443-483), the
// Möller-Trumbore test of Triangle::Intersect (src/geometry/triangle.cpp:55-110)
// and Sphere::Intersect (src/geometry/sphere.cpp:35-85), so closest-hit
// primitive ids and t agree bit for bit with the reference, including its
// last-visited-wins rule for equal t.
//
// Layout in HBM (see bbg_internal.h):
//   nodes: 32 B each = two float4 (min.xyz, max.x) (max.yz, offset, count|axis<<16)
//   slots: 48 B each = three float4 per leaf slot, primitives in leaf order
#pragma once

#include "bbg_internal.h"
#include "dev_math.cuh"
#include "wide8_build.cuh"

#include <cuda_fp16.h>

namespace bbg
{

struct AccelView
{
    const float4* nodes;  // reference layout: 2 per node
    const float4* slots;  // 3 per slot
    const float4* wide;   // child-box layout: 4 per interior node
    const int2* leaves;   // (first slot, count) per leaf
    int32_t root;         // child-box layout root reference
    int32_t ordered;      // 1: nearest-first traversal over the child-box layout
    const float4* wide8 = nullptr; // 8-wide layout: 6 per node, the root first (null: not built)
};

struct RayQ
{
    V3 o, d;          // ray as given
    V3 inv_dir;       // 1 / d per component (the reference's slab test)
    V3 inv_box;       // finite 1 / d of the ordered and 8-wide box tests (BoxInverse)
    V3 dn;            // d after Vector3::Normalize (triangle test)
    float l;          // length returned by that Normalize
    V3 o_near, o_far; // o * inv_box moved outward, for the fused slab test of the ordered traversal
    int neg[3];       // inv_dir < 0
};

// 1 / d for box tests in fused form, plane * (1/d) - o * (1/d): a component
// that is zero (or below 1e-18 of the largest one) counts as 1e-18 of the
// largest, with its own sign, so that its reciprocal is finite. With an
// infinite one both planes of that axis come out as inf - inf = NaN, which
// the three-way minimum ignores: the axis never culls, and a ray parallel to
// a coordinate plane opens every box along its projection. On the
// 1,310,734-triangle Cornell scene one such ray opened 3,200 wide nodes and
// tested 13,553 triangles (the mean ray: 13 and 21) and kept its launch alive
// long after the other rays had finished (2^21 incoherent rays: 8.4 ms, now
// 2.05 ms). The ray strays less than 1e-18 of its length from the given one;
// where it runs in a box's face, which the reference's NaN never culls, the
// tests move their planes outward by more than the face's distance comes out
// at (SlabMargin, IntersectNode8), so no primitive that the reference reaches
// is culled; a direction of length zero keeps its infinities.
__device__ __forceinline__ float BoxInverse(float d, float least)
{
    return 1 / (fabsf(d) < least ? copysignf(least, d) : d);
}

// How far the ordered traversal's slab test, plane * inv - o_inv with o_inv =
// o * inv rounded, moves its planes outward. At a plane through the origin's
// own coordinate all that is left is the rounding of o_inv (half an ulp, and
// as much again where the margin is added), of either sign and, with a
// reciprocal of 1e18, larger than any distance along the ray: without a
// margin the box of a face at coordinate 100 was culled for half of the rays
// that run in it (below 32 the boxes' padding of 10 epsilon hid it). The first
// term is twice that rounding; the second, half an epsilon of length, keeps
// the interval open at coordinate 0, where boxes without padding (spheres')
// have faces and the first term vanishes.
__device__ __forceinline__ float SlabMargin(float o_inv, float inv)
{
    return __fmaf_rn(fabsf(o_inv), 0x1p-22f, fabsf(inv) * 0x1p-24f);
}

__device__ __forceinline__ RayQ MakeRayQ(V3 o, V3 d)
{
    RayQ q;
    q.o = o;
    q.d = d;
    q.inv_dir = V3{ 1 / d.x, 1 / d.y, 1 / d.z };
    q.neg[0] = q.inv_dir.x < 0;
    q.neg[1] = q.inv_dir.y < 0;
    q.neg[2] = q.inv_dir.z < 0;
    q.dn = d;
    q.l = NormalizeInPlace(q.dn);
    const float least = 1e-18f * fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
    q.inv_box = V3{ BoxInverse(d.x, least), BoxInverse(d.y, least), BoxInverse(d.z, least) };
    const V3 oi{ o.x * q.inv_box.x, o.y * q.inv_box.y, o.z * q.inv_box.z };
    const V3 m{ SlabMargin(oi.x, q.inv_box.x), SlabMargin(oi.y, q.inv_box.y), SlabMargin(oi.z, q.inv_box.z) };
    q.o_near = oi + m;
    q.o_far = oi - m;
    return q;
}

// BoundingBox3::TestRay: x and y slabs narrow [t_min, t_max], z only tests.
__device__ __forceinline__ bool TestRay(const float4& a, const float4& b, const RayQ& q, float t_min, float t_max)
{
    // a = (min.x, min.y, min.z, max.x), b = (max.y, max.z, ., .)
    float lo_x = q.neg[0] ? a.w : a.x, hi_x = q.neg[0] ? a.x : a.w;
    float lo_y = q.neg[1] ? b.x : a.y, hi_y = q.neg[1] ? a.y : b.x;
    float lo_z = q.neg[2] ? b.y : a.z, hi_z = q.neg[2] ? a.z : b.y;

    float t_min_x = (lo_x - q.o.x) * q.inv_dir.x;
    float t_max_x = (hi_x - q.o.x) * q.inv_dir.x;
    if (t_min > t_max_x || t_max < t_min_x)
    {
        return false;
    }
    if (t_min_x > t_min) t_min = t_min_x;
    if (t_max_x < t_max) t_max = t_max_x;

    float t_min_y = (lo_y - q.o.y) * q.inv_dir.y;
    float t_max_y = (hi_y - q.o.y) * q.inv_dir.y;
    if (t_min > t_max_y || t_max < t_min_y)
    {
        return false;
    }
    if (t_min_y > t_min) t_min = t_min_y;
    if (t_max_y < t_max) t_max = t_max_y;

    float t_min_z = (lo_z - q.o.z) * q.inv_dir.z;
    float t_max_z = (hi_z - q.o.z) * q.inv_dir.z;
    if (t_min > t_max_z || t_max < t_min_z)
    {
        return false;
    }
    return true;
}

// Möller-Trumbore on the normalised direction (src/geometry/triangle.cpp:55-94).
// The edges e1 = p1 - p0 and e2 = p2 - p0 are stored precomputed (the same
// float values the reference computes per test). Returns true and (t, u, v)
// on a hit in [t_min, t_max].
__device__ __forceinline__ bool IntersectTriangle(V3 p0, V3 e1, V3 e2, V3 o, V3 dn, float l, float t_min, float t_max,
                                                  float* t_out, float* u_out, float* v_out)
{
    V3 pvec = Cross(dn, e2);
    float det = Dot(e1, pvec);
    if (fabsf(det) < kEpsilon)
    {
        return false;
    }
    float invDet = 1 / det;
    V3 tvec = o - p0;
    const float du = Dot(tvec, pvec);
    float u = du * invDet;
    if (u < 0 || u > 1)
    {
        return false;
    }
    V3 qvec = Cross(tvec, e1);
    float v = Dot(dn, qvec) * invDet;
    if (v < 0 || u + v > 1)
    {
        return false;
    }
    float t = Dot(e2, qvec) * invDet / l;
    if (t < t_min || t > t_max)
    {
        return false;
    }
    *t_out = t;
    *u_out = u;
    *v_out = v;
    return true;
}

// Quat::RotateInv / Rotate (include/bulbit/quaternion.h:140-170).
__device__ __forceinline__ V3 QuatRotateInv(float4 q, V3 v)
{
    float vx = 2 * v.x, vy = 2 * v.y, vz = 2 * v.z;
    float w2 = q.w * q.w - 0.5f;
    float dot2 = (q.x * vx + q.y * vy + q.z * vz);
    return V3{ (vx * w2 - (q.y * vz - q.z * vy) * q.w + q.x * dot2),
               (vy * w2 - (q.z * vx - q.x * vz) * q.w + q.y * dot2),
               (vz * w2 - (q.x * vy - q.y * vx) * q.w + q.z * dot2) };
}

__device__ __forceinline__ V3 QuatRotate(float4 q, V3 v)
{
    float vx = 2 * v.x, vy = 2 * v.y, vz = 2 * v.z;
    float w2 = q.w * q.w - 0.5f;
    float dot2 = (q.x * vx + q.y * vy + q.z * vz);
    return V3{ (vx * w2 + (q.y * vz - q.z * vy) * q.w + q.x * dot2),
               (vy * w2 + (q.z * vx - q.x * vz) * q.w + q.y * dot2),
               (vz * w2 + (q.x * vy - q.y * vx) * q.w + q.z * dot2) };
}

// Sphere::Intersect (src/geometry/sphere.cpp:35-61) in object space:
// MulT(transform, ray) then the half-b quadratic; near root first.
__device__ __forceinline__ bool IntersectSphere(V3 p, float4 rot, V3 s, float radius, V3 o, V3 d, float t_min,
                                                float t_max, float* t_out)
{
    V3 ro = QuatRotateInv(rot, o - p) / s;
    V3 rd = QuatRotateInv(rot, d / s);
    V3 oc = ro;
    float a = Length2(rd);
    float half_b = Dot(oc, rd);
    float c = Length2(oc) - radius * radius;
    float discriminant = half_b * half_b - a * c;
    if (discriminant < 0)
    {
        return false;
    }
    float sqrt_d = sqrtf(discriminant);
    float root = (-half_b - sqrt_d) / a;
    if (root < t_min || t_max < root)
    {
        root = (-half_b + sqrt_d) / a;
        if (root < t_min || t_max < root)
        {
            return false;
        }
    }
    *t_out = root;
    return true;
}

struct TraceResult
{
    int32_t prim; // primitive index, -1 on a miss
    float t, u, v;
};

// One leaf slot: the primitive's test with the current [t_min, t_max].
__device__ __forceinline__ bool TestSlot(const AccelView& a, int32_t slot, const RayQ& q, float t_min, float t_max,
                                         TraceResult* res)
{
    const float4* s = a.slots + 3 * size_t(slot);
    float4 s0 = __ldg(s);
    float4 s1 = __ldg(s + 1);
    float4 s2 = __ldg(s + 2);
    uint32_t tag = __float_as_uint(s0.w);
    float t, u = 0, v = 0;
    bool hit;
    if (tag & kSphereBit)
    {
        hit = IntersectSphere(V3{ s0.x, s0.y, s0.z }, s1, V3{ s2.x, s2.y, s2.z }, s2.w, q.o, q.d, t_min, t_max, &t);
    }
    else
    {
        hit = IntersectTriangle(V3{ s0.x, s0.y, s0.z }, V3{ s1.x, s1.y, s1.z }, V3{ s2.x, s2.y, s2.z }, q.o, q.dn,
                                q.l, t_min, t_max, &t, &u, &v);
    }
    if (hit)
    {
        res->prim = int32_t(tag & ~kSphereBit);
        res->t = t;
        res->u = u;
        res->v = v;
    }
    return hit;
}

// Stack traversal of BVH::RayCast over the reference's own node order. ANY =
// IntersectAny semantics (stop at the first hit); otherwise Intersect
// semantics (shrink t_max; a hit at exactly the current t_max replaces the
// previous one). COUNT accumulates nodes popped and primitive tests.
template <bool ANY, bool COUNT>
__device__ __forceinline__ TraceResult TraceReference(const AccelView& a, const RayQ& q, float t_min, float t_max,
                                                      uint32_t* nodes_visited = nullptr,
                                                      uint32_t* prims_tested = nullptr)
{
    TraceResult res{ -1, t_max, 0, 0 };
    int32_t stack[kStackCapacity];
    int sp = 0;
    stack[sp++] = 0;

    while (sp > 0)
    {
        int32_t index = stack[--sp];
        float4 na = __ldg(a.nodes + 2 * index);
        float4 nb = __ldg(a.nodes + 2 * index + 1);
        if (COUNT) ++*nodes_visited;
        if (!TestRay(na, nb, q, t_min, t_max))
        {
            continue;
        }
        int32_t offset = __float_as_int(nb.z);
        uint32_t packed = __float_as_uint(nb.w);
        int32_t count = int32_t(packed & 0xffffu);
        if (count > 0)
        {
            for (int32_t i = 0; i < count; ++i)
            {
                if (COUNT) ++*prims_tested;
                // The callback's return value: t_min after an any-hit, the
                // hit's t after a closest hit, the running t_max on a miss;
                // RayCast stops when it is <= t_min, else takes it as t_max.
                if (TestSlot(a, offset + i, q, t_min, t_max, &res))
                {
                    if (ANY)
                    {
                        return res;
                    }
                    t_max = res.t;
                }
                if (t_max <= t_min)
                {
                    return res;
                }
            }
        }
        else
        {
            int32_t child1 = index + 1;
            int32_t child2 = offset;
            int axis = int((packed >> 16) & 0xffu);
            if (q.neg[axis])
            {
                stack[sp++] = child1;
                stack[sp++] = child2;
            }
            else
            {
                stack[sp++] = child2;
                stack[sp++] = child1;
            }
        }
    }
    return res;
}

// Slab test of one child box: [entry, exit] of the ray within the box and
// within [t_min, t_max] (include/bulbit/bounding_box.h:448-480).
__device__ __forceinline__ bool SlabTest(float lx, float ly, float lz, float hx, float hy, float hz, const RayQ& q,
                                         float t_min, float t_max, float* entry)
{
    // bound * (1/d) - o * (1/d) in one fused multiply-add per plane. It rounds
    // differently from the reference's (bound - o) * (1/d); it only decides
    // which boxes are opened, and the planes are moved outward by more than
    // o * (1/d) can be off (SlabMargin).
    float x0 = __fmaf_rn(q.neg[0] ? hx : lx, q.inv_box.x, -q.o_near.x);
    float x1 = __fmaf_rn(q.neg[0] ? lx : hx, q.inv_box.x, -q.o_far.x);
    float y0 = __fmaf_rn(q.neg[1] ? hy : ly, q.inv_box.y, -q.o_near.y);
    float y1 = __fmaf_rn(q.neg[1] ? ly : hy, q.inv_box.y, -q.o_far.y);
    float z0 = __fmaf_rn(q.neg[2] ? hz : lz, q.inv_box.z, -q.o_near.z);
    float z1 = __fmaf_rn(q.neg[2] ? lz : hz, q.inv_box.z, -q.o_far.z);
    float t0 = fmaxf(fmaxf(x0, y0), fmaxf(z0, t_min));
    float t1 = fminf(fminf(x1, y1), fminf(z1, t_max));
    *entry = t0;
    return t0 <= t1;
}


// Persistent warp-cooperative traversal over the child-box layout (the
// while-while scheme of Aila & Laine, "Understanding the efficiency of ray
// traversal on GPUs", HPG 2009, with dynamic ray fetch):
//   * a warp takes batches of work items from a global counter whenever fewer
//     than kRefill of its lanes still hold a ray, so lanes that finish early
//     get new rays instead of idling until the slowest ray of the batch ends;
//   * each round first walks interior nodes until every busy lane has found a
//     leaf (a lane that reaches a leaf postpones it and keeps walking), then
//     tests leaves together, so node and leaf work do not serialise the warp.
// Per ray: nearest child first over the child-box layout (each interior node
// holds both children's boxes, so one 64-byte fetch tests two), the farther
// child pushed with its entry distance and skipped on pop once a closer hit
// is known; the same primitive tests as BVH::RayCast in a different order, so
// the closest hit is the same except between hits at exactly equal t.
// Src supplies Load(item, RayQ*, t_min*, t_max*) and Store(item, result).
constexpr int32_t kNoNode = int32_t(0x80000000);
// 28 of 32 measured best for both layouts (16: -9 %, 24: -2.5 %, 32: -9 % on
// the 1M-triangle soup's closest + any-hit rays; path tracing unchanged).
#ifndef BBG_REFILL
#define BBG_REFILL 28
#endif
#ifndef BBG_SHORT_STACK
#define BBG_SHORT_STACK 16
#endif
// A warp fetches new rays when fewer than kRefill of its lanes are busy.
constexpr int kRefill = BBG_REFILL;
// Kernels calling TracePersistent run blocks of this many threads.
constexpr int kTraversalBlock = 128;
// Stack entries kept in shared memory per thread; deeper ones go to local
// memory. The shared part is laid out [depth][thread], so a warp's lanes hit
// distinct banks whatever depth each lane is at.
constexpr int kShortStack = BBG_SHORT_STACK;

// BLOCK: threads per block of the launch; SHORT: stack entries kept in
// shared memory per thread (0: the whole stack in local memory).
template <bool ANY, class Src, int BLOCK = kTraversalBlock, int SHORT = kShortStack>
__device__ __forceinline__ void TracePersistent(const AccelView& a, int32_t n, int32_t* next, Src& src)
{
    const unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int tid = threadIdx.x;
    int32_t item = -1;
    bool exhausted = false;
    RayQ q;
    float t_min = 0, t_max = 0;
    TraceResult res{ -1, 0, 0, 0 };
    __shared__ int32_t s_ref[(SHORT > 0 ? SHORT : 1) * BLOCK];
    __shared__ float s_entry[(SHORT > 0 ? SHORT : 1) * BLOCK];
    int2 spill[kStackCapacity - SHORT];
    int sp = 0;
    int32_t node = kNoNode, leaf = kNoNode;
    // The tree a ray is traced in: the one given, or, when the work source
    // names one per item (several scenes in one launch), that one.
    AccelView av = a;

    auto push = [&](int32_t ref, float entry) {
        if (sp < SHORT)
        {
            s_ref[sp * BLOCK + tid] = ref;
            s_entry[sp * BLOCK + tid] = entry;
        }
        else
        {
            spill[sp - SHORT] = make_int2(ref, __float_as_int(entry));
        }
        ++sp;
    };
    auto pop = [&]() -> int32_t {
        while (sp > 0)
        {
            --sp;
            int32_t ref;
            float entry;
            if (sp < SHORT)
            {
                ref = s_ref[sp * BLOCK + tid];
                entry = s_entry[sp * BLOCK + tid];
            }
            else
            {
                int2 e = spill[sp - SHORT];
                ref = e.x;
                entry = __int_as_float(e.y);
            }
            if (entry <= t_max)
            {
                return ref;
            }
        }
        return kNoNode;
    };

    while (true)
    {
        __syncwarp();
        bool busy = item >= 0;
        unsigned have = __ballot_sync(kFull, busy);
        if (!exhausted && __popc(have) < kRefill)
        {
            unsigned need = ~have;
            int32_t cnt = __popc(need);
            int32_t base = 0;
            if (lane == 0)
            {
                base = atomicAdd(next, cnt);
            }
            base = __shfl_sync(kFull, base, 0);
            exhausted = base + cnt >= n;
            if (!busy)
            {
                int32_t r = base + __popc(need & ((1u << lane) - 1u));
                if (r < n)
                {
                    item = r;
                    src.Load(r, &q, &t_min, &t_max);
                    if constexpr (requires { src.View(r); })
                    {
                        av = src.View(r);
                    }
                    res = TraceResult{ -1, t_max, 0, 0 };
                    sp = 0;
                    node = av.root;
                    leaf = kNoNode;
                    busy = true;
                }
            }
            have = __ballot_sync(kFull, busy);
        }
        if (have == 0)
        {
            break;
        }
        if (busy)
        {
            if (node < 0 && node != kNoNode && leaf == kNoNode)
            {
                leaf = node;
                node = pop();
            }
            // Node phase.
            while (node >= 0)
            {
                const float4* nd = av.wide + 4 * size_t(node);
                float4 f0 = __ldg(nd);
                float4 f1 = __ldg(nd + 1);
                float4 f2 = __ldg(nd + 2);
                int4 f3 = __ldg(reinterpret_cast<const int4*>(nd + 3));
                float e0, e1;
                bool h0 = SlabTest(f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, q, t_min, t_max, &e0);
                bool h1 = SlabTest(f1.z, f1.w, f2.x, f2.y, f2.z, f2.w, q, t_min, t_max, &e1);
                if (h0 && h1)
                {
                    bool swap = e1 < e0;
                    push(swap ? f3.x : f3.y, swap ? e0 : e1);
                    node = swap ? f3.y : f3.x;
                }
                else if (h0 || h1)
                {
                    node = h0 ? f3.x : f3.y;
                }
                else
                {
                    node = pop();
                }
                if (node < 0 && node != kNoNode && leaf == kNoNode)
                {
                    leaf = node;
                    node = pop();
                }
                if (__all_sync(__activemask(), leaf != kNoNode))
                {
                    break;
                }
            }
            // Leaf phase.
            while (leaf != kNoNode)
            {
                int2 lf = __ldg(av.leaves + (~leaf));
                bool stop = false;
                for (int32_t i = 0; i < lf.y; ++i)
                {
                    if (TestSlot(av, lf.x + i, q, t_min, t_max, &res))
                    {
                        if (ANY)
                        {
                            stop = true;
                            break;
                        }
                        t_max = res.t;
                    }
                    if (t_max <= t_min)
                    {
                        stop = true;
                        break;
                    }
                }
                leaf = kNoNode;
                if (stop)
                {
                    node = kNoNode;
                    sp = 0;
                    break;
                }
                if (node < 0 && node != kNoNode)
                {
                    leaf = node;
                    node = pop();
                }
            }
            if (node == kNoNode && leaf == kNoNode)
            {
                src.Store(item, res);
                item = -1;
            }
        }
    }
}

// ---------------------------------------------------------------- 8-wide layout
//
// The reference's binary SAH tree collapsed into nodes of up to eight
// children (the compressed wide BVH of Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017).
// 96 bytes per node, six float4:
//   [0]   origin p (the node box's lower corner), meta = biased exponents
//         e_x | e_y << 8 | e_z << 16 of the per-axis scales s = 2^e, and
//         << 24 the mask of interior-child slots
//   [1-3] child boxes as bytes, child k in byte k & 3 of word k >> 2:
//         qlo_x, qlo_y, qlo_z, qhi_x, qhi_y, qhi_z (two words each)
//   [4-5] child references: >= 0 node, < 0 a leaf ~(first slot << 5 |
//         count); an empty slot is a leaf of no primitives with an inverted
//         box
// Child k's box is [p + qlo s, p + qhi s], rounded outward when built, so it
// contains the binary node it stands for and no ray that reaches a leaf in
// the binary tree is culled here. Slots are assigned so that, for a ray whose
// direction signs form the octant code o (bit a set for a negative axis),
// visiting slots in the order k ^ o for k = 0..7 is roughly front to back.

// Blocks per SM that a traversal kernel's registers must leave room for: 1,024
// threads (64 registers) over the 8-wide layout, where 72 (7 blocks of 128)
// made frames 2.5 % slower and 56 (9 blocks) as well; no bound otherwise.
constexpr int TraceMinBlocks(int block, bool wide) { return wide ? 1024 / block : 1; }

// Bytes 2 pair and 2 pair + 1 of w, each plus 1024, as floats: one byte
// permute assembles the half2 (1024 + b0, 1024 + b1) (bits 0x64bb), which
// converts exactly; the planes' constants take the 1024 off again.
__device__ __forceinline__ float2 BytePairPlus1024(uint32_t w, int pair)
{
    uint32_t h = __byte_perm(w, 0x64646464u, pair ? 0x4342u : 0x4140u);
    __half2 v = *reinterpret_cast<__half2*>(&h);
    return __half22float2(v);
}

// Two fused multiply-adds in one instruction (the same roundings).
__device__ __forceinline__ float2 Fma2(float2 q, float b, float c)
{
    float2 r;
    asm("{\n\t.reg .b64 q, b, c, r;\n\tmov.b64 q, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
        "fma.rn.f32x2 r, q, b, c;\n\tmov.b64 {%0, %1}, r;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(q.x), "f"(q.y), "f"(b), "f"(c));
    return r;
}

// Three-input minimum / maximum (PTX min.f32 / max.f32 with three sources;
// a NaN source is ignored as by fminf / fmaxf).
__device__ __forceinline__ float Max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float Min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Moves bit k of each byte of m to bit k ^ oct (oct in 0..7).
__device__ __forceinline__ uint32_t PermuteByOctant(uint32_t m, uint32_t oct)
{
    if (oct & 1u) m = ((m & 0x55555555u) << 1) | ((m >> 1) & 0x55555555u);
    if (oct & 2u) m = ((m & 0x33333333u) << 2) | ((m >> 2) & 0x33333333u);
    if (oct & 4u) m = ((m & 0x0f0f0f0fu) << 4) | ((m >> 4) & 0x0f0f0f0fu);
    return m;
}

// The first 64 bytes of a node (box, scales, child planes) in two 32-byte
// loads: a warp's lanes read different nodes, and each load instruction costs
// the L1 one tag lookup per distinct line, whatever its width.
__device__ __forceinline__ void LoadNode64(const float4* nd, float4* h, uint4* w1, uint4* w2, uint4* w3)
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(h->x), "=f"(h->y), "=f"(h->z), "=f"(h->w), "=r"(w1->x), "=r"(w1->y), "=r"(w1->z), "=r"(w1->w)
        : "l"(nd));
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w2->x), "=r"(w2->y), "=r"(w2->z), "=r"(w2->w), "=r"(w3->x), "=r"(w3->y), "=r"(w3->z), "=r"(w3->w)
        : "l"(nd + 2));
}

// Tests the ray against a node's eight child boxes. Bits of *inner / *leaf
// are visit positions (slot ^ octant) of the hit interior / leaf children;
// order maps a mask of slots to the mask of their visit positions.
// The traversal is bound by instruction issue, and this is most of it, so it
// is written for few instructions: planes over 1024 + q (no subtraction per
// plane), two planes to a fused multiply-add, misses collected by shifting
// sign bits, and a table for the visit order (without which the soup's rays
// take 1.47 ms instead of 1.37). All of it took 2^21 soup rays from 1.61 to
// 1.47 ms and a 512 x 512, 64-sample Cornell frame from 110.9 to 106.0 ms.
__device__ __forceinline__ void IntersectNode8(const float4* nd, V3 o, V3 inv_box, float t_min, float t_max,
                                               const uint8_t* order, uint32_t* inner, uint32_t* leaf)
{
    float4 h;
    uint4 w1, w2, w3;
    LoadNode64(nd, &h, &w1, &w2, &w3);
    uint32_t meta = __float_as_uint(h.w);
    // Plane k of axis a sits at p_a + q s_a: t = q (s_a / d_a) + (p_a - o_a) / d_a.
    float bx = __uint_as_float((meta & 0xffu) << 23) * inv_box.x;
    float by = __uint_as_float(((meta >> 8) & 0xffu) << 23) * inv_box.y;
    float bz = __uint_as_float(((meta >> 16) & 0xffu) << 23) * inv_box.z;
    // (p - o) / d in the reference's slab form; the ray's signs from 1/d
    // (kept in predicates rather than per-ray registers).
    float ax = (h.x - o.x) * inv_box.x;
    float ay = (h.y - o.y) * inv_box.y;
    float az = (h.z - o.z) * inv_box.z;
    // Constants of the entry and exit planes over 1024 + q, apart by what the
    // 1024 and the larger sum cost in rounding (2^-14 |b| + 2^-24 |a| each),
    // and more, so that a box never comes out smaller than over q itself.
    const float wx = __fmaf_rn(fabsf(bx), 0x1p-13f, fabsf(ax) * 0x1p-22f);
    const float wy = __fmaf_rn(fabsf(by), 0x1p-13f, fabsf(ay) * 0x1p-22f);
    const float wz = __fmaf_rn(fabsf(bz), 0x1p-13f, fabsf(az) * 0x1p-22f);
    const float cx = __fmaf_rn(bx, -1024.0f, ax), cy = __fmaf_rn(by, -1024.0f, ay), cz = __fmaf_rn(bz, -1024.0f, az);
    const float nx = cx - wx, ny = cy - wy, nz = cz - wz, fx = cx + wx, fy = cy + wy, fz = cz + wz;
    const bool negx = inv_box.x < 0, negy = inv_box.y < 0, negz = inv_box.z < 0;
    // Entry planes are the low bounds on a positive axis, the high ones on a negative axis.
    uint32_t nx0 = negx ? w2.z : w1.x, nx1 = negx ? w2.w : w1.y;
    uint32_t fx0 = negx ? w1.x : w2.z, fx1 = negx ? w1.y : w2.w;
    uint32_t ny0 = negy ? w3.x : w1.z, ny1 = negy ? w3.y : w1.w;
    uint32_t fy0 = negy ? w1.z : w3.x, fy1 = negy ? w1.w : w3.y;
    uint32_t nz0 = negz ? w3.z : w2.x, nz1 = negz ? w3.w : w2.y;
    uint32_t fz0 = negz ? w2.x : w3.z, fz1 = negz ? w2.y : w3.w;
    uint32_t miss = 0;
#pragma unroll
    for (int j = 3; j >= 0; --j) // children 2j + 1 and 2j
    {
        const int pair = j & 1;
        const bool hi = j >= 2;
        float2 qnx = BytePairPlus1024(hi ? nx1 : nx0, pair), qfx = BytePairPlus1024(hi ? fx1 : fx0, pair);
        float2 qny = BytePairPlus1024(hi ? ny1 : ny0, pair), qfy = BytePairPlus1024(hi ? fy1 : fy0, pair);
        float2 qnz = BytePairPlus1024(hi ? nz1 : nz0, pair), qfz = BytePairPlus1024(hi ? fz1 : fz0, pair);
        const float2 pnx = Fma2(qnx, bx, nx), pny = Fma2(qny, by, ny), pnz = Fma2(qnz, bz, nz);
        const float2 pfx = Fma2(qfx, bx, fx), pfy = Fma2(qfy, by, fy), pfz = Fma2(qfz, bz, fz);
        float t0a = Max3(pnx.x, pny.x, fmaxf(pnz.x, t_min));
        float t1a = Min3(pfx.x, pfy.x, fminf(pfz.x, t_max));
        float t0b = Max3(pnx.y, pny.y, fmaxf(pnz.y, t_min));
        float t1b = Min3(pfx.y, pfy.y, fminf(pfz.y, t_max));
        // A child is missed where exit - entry is negative: its sign bit is
        // shifted in (a NaN, of an unbounded interval, counts as a hit).
        miss = __funnelshift_l(__float_as_uint(t1b - t0b), miss, 1);
        miss = __funnelshift_l(__float_as_uint(t1a - t0a), miss, 1);
    }
    // Slot-order masks (interior slots from the header), then visit positions.
    const uint32_t imask = meta >> 24;
    *inner = order[imask & ~miss];
    *leaf = order[~(imask | miss) & 0xffu];
}

__device__ __forceinline__ int32_t ChildRef8(const float4* wide8, int32_t node, uint32_t slot)
{
    return __ldg(reinterpret_cast<const int32_t*>(wide8 + 6 * size_t(node) + 4) + slot);
}

// Persistent traversal of the 8-wide layout (same work-source protocol as
// TracePersistent), one ray per lane. Each iteration opens one node per lane,
// the nearest unopened child (by the octant order) of the lane's current
// group, a group being the hit interior children of one node (node << 8 |
// visit positions left). A node with hit interior children makes them the
// current group and pushes what is left of the old one; every push is one
// tree level deeper than the last, so the tree depth bounds the stack. The
// next node is picked and its reference fetched right after a node's test, so
// that the fetch runs beside the queueing of the leaves.
//
// The primitives of the hit leaves are not tested by the lane that found them
// but by the whole warp: a hit leaf goes into a queue of the warp in shared
// memory as lane << 26 | node << 3 | slot, and as soon as 32 leaves wait there
// their primitives are dealt out, one to a lane, each tested against its
// leaf's ray (origin and direction are kept in shared memory). A ray's
// primitives are tested in the order in which a loop of its own would test
// them and a hit is taken by the same rule, so the results are that loop's; a
// leaf waiting in the queue only means that t_max shrinks a few nodes later,
// and a node opened meanwhile holds no primitive at or before the nearest
// hit. The queue is emptied before it holds 32 when kWaitFlush lanes have
// nothing left to do but wait for their leaves, when no lane has a node to
// open, or when leaves have waited kLeafAge iterations: a warp with few rays
// left would otherwise fill it too slowly and open nodes behind a hit that it
// does not know of yet.
//
// The nearest hit of each ray stands in shared memory, written by the lane
// that tested the primitive, and the closest-hit kernels read the origin from
// there too: both would otherwise be registers that live through the node
// test, and at 64 registers a single spilled one costs 3 to 5 %.
//
// Measured on one B200 against a loop per lane over its own leaves (which ran
// with 8 to 16 of a warp's 32 threads active, 20 to 23 here), both with the
// memset of the work counter: 2^21 incoherent closest-hit rays in the
// 1,310,734-triangle Cornell box 2.05 -> 1.30 ms, the any-hit rays 1.03 -> 0.67
// ms, a 512 x 512, 64-sample frame 151.9 -> 104.0 ms; in the 1,048,576-triangle
// soup (7 primitives per ray against 28 nodes) 1.60 -> 1.35 ms and 0.32 -> 0.30
// ms, 20,000 rays there 161 -> 142 us and 100 -> 96 us; 1,024 rays in a
// 20,000-triangle soup 79.8 -> 75.8 us; a frame of a 34-triangle box 2.24 -> 2.06
// ms. Dearer than the loop: small any-hit batches that meet few leaves (20,000
// small triangles; 300, 1,024 and 20,000 rays 20.8 -> 22.7, 24.4 -> 26.1 and 29.1
// -> 30.3 us), where a warp has its scheduler to itself and the ballots around
// the queue lengthen every iteration; in the larger soup the same batches gain
// (1,024 rays 61.8 -> 57.3 us), so the batch's size does not tell them apart,
// and emptying the queue sooner, by age or by the share of rays that wait,
// made them no faster and the large batches 2 to 15 % slower. Queueing single
// primitives instead of leaves, in a step per primitive, had cost the soup
// 13 %: the queueing steps were half of all instructions. Without kLeafAge
// 20,000 closest-hit rays in the large soup took 1.45 times as long.
constexpr int kWarpQueue = 64; // at most 31 waiting leaves + 32 new ones
constexpr int kWaitFlush = 4;  // 1 to 10 measure alike
constexpr int kLeafAge = 8;    // 3 to 12 measure alike

template <bool ANY, class Src, int BLOCK = kTraversalBlock, int SHORT = kShortStack, bool SPHERES = true>
__device__ __forceinline__ void TracePersistentWide(const AccelView& a, int32_t n, int32_t* work, Src& src)
{
    const unsigned kFull = 0xffffffffu;
    constexpr bool kPerItemView = requires { src.View(0); };
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    __shared__ int32_t s_stack[(SHORT > 0 ? SHORT : 1) * BLOCK];
    __shared__ uint32_t s_leaves[BLOCK / 32 * kWarpQueue];
    __shared__ uint32_t s_order[8 * 64];          // octant, slot mask -> visit-position mask (a byte each)
    __shared__ float4 s_org[BLOCK];               // ray origin, t_min
    __shared__ float4 s_dir[BLOCK];               // normalised direction, its length before
    __shared__ float4 s_raw[SPHERES ? BLOCK : 1]; // direction as given (sphere test)
    __shared__ float4 s_best[ANY ? 1 : BLOCK];    // nearest hit so far: primitive, t, u, v
    __shared__ const float4* s_slots[kPerItemView ? BLOCK : 1];
    __shared__ const float4* s_wide8[kPerItemView ? BLOCK : 1];
    const int warp0 = tid & ~31; // the warp's rays in s_org and s_dir
    uint32_t* const leaves = s_leaves + (tid >> 5) * kWarpQueue;
    int32_t spill[kStackCapacity - SHORT];
    if (int64_t(blockIdx.x) * BLOCK >= n)
    {
        return; // fewer rays than lanes in the launch: the first blocks take them
    }
    for (int i = tid; i < 8 * 64; i += BLOCK) // four masks to a word
    {
        s_order[i] = PermuteByOctant(uint32_t(i & 63) * 0x04040404u + 0x03020100u, uint32_t(i >> 6));
    }
    __syncthreads();

    int32_t item = -1;
    bool exhausted = false;
    V3 inv_box{};
    float t_max = 0;
    int32_t found = -1; // ANY: 0 once something is hit
    int sp = 0;
    uint32_t oct = 0;
    int32_t next = -1;           // node to open, -1: none left
    uint32_t group = 0;          // current group, without it
    const float4* wide8 = a.wide8;
    uint32_t lm = 0;             // hit leaves of the node just opened, not queued yet
    uint32_t head = 0, tail = 0; // queue positions: tested, filled (warp-uniform)
    uint32_t last = 0;           // the queue position after the lane's last leaf
    int age = 0;                 // iterations that leaves have waited (warp-uniform)

    auto push = [&](uint32_t e) {
        if (sp < SHORT)
        {
            s_stack[sp * BLOCK + tid] = int32_t(e);
        }
        else
        {
            spill[sp - SHORT] = int32_t(e);
        }
        ++sp;
    };
    auto pop = [&]() -> uint32_t {
        --sp;
        return uint32_t(sp < SHORT ? s_stack[sp * BLOCK + tid] : spill[sp - SHORT]);
    };

    // Tests the primitives of the queue's first min(32, tail - head) leaves
    // and hands the hits to their rays' lanes in queue order.
    auto test_leaves = [&]() {
        __syncwarp();
        const uint32_t waiting = min(32u, tail - head);
        const uint32_t entry = leaves[(head + lane) & (kWarpQueue - 1)];
        __syncwarp(); // read before new leaves are written there
        int owner = int(entry >> 26);
        int32_t first = -1, count = 1;
        if (uint32_t(lane) < waiting)
        {
            const float4* nodes = kPerItemView ? s_wide8[kPerItemView ? warp0 + owner : 0] : a.wide8;
            const uint32_t lf = ~uint32_t(ChildRef8(nodes, int32_t((entry >> 3) & 0x7fffffu), entry & 7u));
            count = int32_t(lf & ((1u << kWide8LeafCountBits) - 1u));
            first = count > 0 ? int32_t(lf >> kWide8LeafCountBits) : -1;
            count = max(count, 1);
        }
        head += waiting;
        // Leaves of one primitive each: one to a lane as they are. Else the
        // primitives are numbered through the leaves (start: the number of a
        // leaf's first one) and dealt out 32 at a time.
        const bool single = !__any_sync(kFull, count != 1);
        uint32_t start = uint32_t(lane), total = waiting;
        if (!single)
        {
            uint32_t sum = uint32_t(lane) < waiting ? uint32_t(count) : 0u;
            const uint32_t mine = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const uint32_t below_sum = __shfl_up_sync(kFull, sum, off);
                sum += lane >= off ? below_sum : 0u;
            }
            start = sum - mine;
            total = __shfl_sync(kFull, sum, 31);
        }
        for (uint32_t round = 0; round < total; round += 32)
        {
            int32_t slot = first;
            int ray = owner;
            bool leading = true; // the leaf's first primitive
            if (!single)
            {
                // Leaf k starts at bit start - round; the leaf a lane works on
                // is the last one that starts at or before its number.
                const bool here = uint32_t(lane) < waiting && start >= round && start < round + 32;
                const uint32_t starts = __reduce_or_sync(kFull, here ? 1u << (start - round) : 0u);
                const int before = __popc(__ballot_sync(kFull, uint32_t(lane) < waiting && start < round));
                const int leaf = before + __popc(starts & (below | (1u << lane))) - 1;
                const uint32_t at = __shfl_sync(kFull, start, leaf);
                slot = __shfl_sync(kFull, first, leaf);
                ray = __shfl_sync(kFull, owner, leaf);
                leading = round + lane == at;
                slot = slot < 0 ? slot : slot + int32_t(round + lane - at);
            }
            const float ray_t_max = __shfl_sync(kFull, t_max, ray);
            bool hit = false;
            float t = 0, u = 0, v = 0;
            int32_t prim = -1;
            if (round + lane < total && slot >= 0)
            {
                const float4* s = (kPerItemView ? s_slots[kPerItemView ? warp0 + ray : 0] : a.slots) + 3 * size_t(slot);
                const float4 s0 = __ldg(s), s1 = __ldg(s + 1), s2 = __ldg(s + 2);
                const float4 ro = s_org[warp0 + ray], rd = s_dir[warp0 + ray];
                const uint32_t tag = __float_as_uint(s0.w);
                prim = int32_t(tag & ~kSphereBit);
                if (SPHERES && (tag & kSphereBit))
                {
                    const float4 raw = s_raw[SPHERES ? warp0 + ray : 0];
                    hit = IntersectSphere(V3{ s0.x, s0.y, s0.z }, s1, V3{ s2.x, s2.y, s2.z }, s2.w,
                                          V3{ ro.x, ro.y, ro.z }, V3{ raw.x, raw.y, raw.z }, ro.w, ray_t_max, &t);
                }
                else
                {
                    hit = IntersectTriangle(V3{ s0.x, s0.y, s0.z }, V3{ s1.x, s1.y, s1.z }, V3{ s2.x, s2.y, s2.z },
                                            V3{ ro.x, ro.y, ro.z }, V3{ rd.x, rd.y, rd.z }, rd.w, ro.w, ray_t_max, &t,
                                            &u, &v);
                }
                // An interval of no length: only the first primitive counts.
                if (hit && ray_t_max <= ro.w)
                {
                    hit = leading && (ANY || __float_as_int(s_best[ANY ? 0 : warp0 + ray].x) < 0);
                }
            }
            if constexpr (ANY)
            {
                // One hit is enough: the ray is done.
                if ((__reduce_or_sync(kFull, hit ? 1u << ray : 0u) >> lane) & 1u)
                {
                    found = 0;
                    next = -1;
                    sp = 0;
                    lm = 0;
                }
            }
            else
            {
                // The hits' lanes write the records, all at once where no ray
                // has two (handing them over one by one instead cost closed
                // scenes, where most lanes hit, 5 to 10 %), else in the order of
                // the queue by the rule of a loop over the ray's own leaves:
                // nothing farther than the nearest hit (the primitive's test
                // has seen to that for a ray's first), and nothing more once
                // that is at t_min.
                const unsigned hits = __ballot_sync(kFull, hit);
                if (hits != 0)
                {
                    const unsigned rays = __reduce_or_sync(kFull, hit ? 1u << ray : 0u);
                    const float4 record = make_float4(__int_as_float(prim), t, u, v);
                    if (__popc(rays) == __popc(hits))
                    {
                        if (hit)
                        {
                            s_best[ANY ? 0 : warp0 + ray] = record;
                        }
                    }
                    else
                    {
                        for (unsigned left = hits; left != 0; left &= left - 1)
                        {
                            if (lane == __ffs(left) - 1)
                            {
                                const float4 best = s_best[ANY ? 0 : warp0 + ray];
                                if (!(t > best.y) &&
                                    (__float_as_int(best.x) < 0 || !(best.y <= s_org[warp0 + ray].w)))
                                {
                                    s_best[ANY ? 0 : warp0 + ray] = record;
                                }
                            }
                            __syncwarp();
                        }
                    }
                    __syncwarp();
                    if ((rays >> lane) & 1u)
                    {
                        t_max = s_best[ANY ? 0 : tid].y;
                        if (t_max <= s_org[tid].w)
                        {
                            next = -1;
                            sp = 0;
                            lm = 0;
                        }
                    }
                    __syncwarp(); // read before the next round writes there
                }
            }
        }
    };

    while (true)
    {
        __syncwarp();
        unsigned have = __ballot_sync(kFull, item >= 0);
        if (!exhausted && __popc(have) < kRefill)
        {
            unsigned need = ~have;
            int32_t cnt = __popc(need);
            int32_t base = 0;
            if (lane == 0)
            {
                base = atomicAdd(work, cnt);
            }
            base = __shfl_sync(kFull, base, 0);
            exhausted = base + cnt >= n;
            if (item < 0)
            {
                int32_t r = base + __popc(need & below);
                if (r < n)
                {
                    item = r;
                    RayQ q;
                    float t_min;
                    src.Load(r, &q, &t_min, &t_max);
                    inv_box = q.inv_box;
                    s_org[tid] = make_float4(q.o.x, q.o.y, q.o.z, t_min);
                    s_dir[tid] = make_float4(q.dn.x, q.dn.y, q.dn.z, q.l);
                    if (SPHERES)
                    {
                        s_raw[SPHERES ? tid : 0] = make_float4(q.d.x, q.d.y, q.d.z, 0.0f);
                    }
                    if constexpr (kPerItemView)
                    {
                        const AccelView av = src.View(r);
                        wide8 = av.wide8;
                        s_wide8[tid] = av.wide8;
                        s_slots[tid] = av.slots;
                    }
                    found = -1;
                    if (!ANY)
                    {
                        s_best[ANY ? 0 : tid] = make_float4(__int_as_float(-1), t_max, 0.0f, 0.0f);
                    }
                    sp = 0;
                    oct = uint32_t(inv_box.x < 0) | (uint32_t(inv_box.y < 0) << 1) | (uint32_t(inv_box.z < 0) << 2);
                    next = 0; // the root
                    group = 0;
                    last = head;
                }
            }
            have = __ballot_sync(kFull, item >= 0);
        }
        if (have == 0)
        {
            break;
        }
        uint32_t entry = 0;
        if (next >= 0)
        {
            const int32_t node = next;
            uint32_t im;
            const float4 ro = s_org[tid];
            IntersectNode8(wide8 + 6 * size_t(node), V3{ ro.x, ro.y, ro.z }, inv_box, ro.w, t_max,
                           reinterpret_cast<const uint8_t*>(s_order) + (oct << 8), &im, &lm);
            if (im != 0)
            {
                if ((group & 0xffu) != 0)
                {
                    push(group);
                }
                group = (uint32_t(node) << 8) | im;
            }
            // The next node: its reference is under way while the leaves queue.
            if ((group & 0xffu) == 0 && sp > 0)
            {
                group = pop();
            }
            next = -1;
            if ((group & 0xffu) != 0)
            {
                next = ChildRef8(wide8, int32_t(group >> 8), uint32_t(__ffs(group) - 1) ^ oct);
                group &= group - 1;
            }
            entry = (uint32_t(lane) << 26) | (uint32_t(node) << 3);
        }
        // The nodes' hit leaves into the queue, one per lane and step, in
        // each lane's visit order.
        while (true)
        {
            const unsigned adding = __ballot_sync(kFull, lm != 0);
            if (lm != 0)
            {
                const uint32_t pos = uint32_t(__ffs(lm) - 1);
                lm &= lm - 1;
                last = tail + uint32_t(__popc(adding & below));
                leaves[last & (kWarpQueue - 1)] = entry | (pos ^ oct);
                ++last;
                if (t_max <= s_org[tid].w)
                {
                    // An interval of no length: the first leaf is the last one.
                    next = -1;
                    sp = 0;
                    lm = 0;
                }
            }
            tail += uint32_t(__popc(adding));
            bool flush = tail - head >= 32;
            if (adding == 0 && head != tail)
            {
                // Lanes with no node left wait for their leaves.
                const bool walking = next >= 0;
                const unsigned walk = __ballot_sync(kFull, walking);
                const unsigned wait = __ballot_sync(kFull, !walking && item >= 0 && int32_t(last - head) > 0);
                flush = walk == 0 || __popc(wait) >= kWaitFlush || ++age >= kLeafAge;
            }
            if (flush)
            {
                test_leaves();
                age = 0;
            }
            if (adding == 0)
            {
                break;
            }
        }
        if (item >= 0 && next < 0 && int32_t(last - head) <= 0)
        {
            const float4 b = ANY ? make_float4(__int_as_float(found), t_max, 0.0f, 0.0f) : s_best[ANY ? 0 : tid];
            src.Store(item, TraceResult{ __float_as_int(b.x), b.y, b.z, b.w });
            item = -1;
        }
    }
}


} // namespace bbg
