// Closest-hit traversal of the reference's two-level SAH BVH on sm_103a.
//
// Bit-exact restatement of Scene::hit (src/Scene.cpp:154-189) ->
// CacheBVHNode_world::hit (src/BVH/BVH_world.cpp:267-283) -> Mesh::hit
// (src/mesh.cpp:70-105) -> CacheBVHNode_mesh::hit (src/BVH/BVH_mesh.cpp:265-283) ->
// aabb::hit (src/aabb.cpp:6-41) and Triangle::hit (src/Triangle.cpp:20-88):
//  * stack DFS, right child pushed before left, so the left subtree is visited first;
//  * every box is tested against the current closest distance of its own level (the
//    passes test both children's boxes at their parent and keep the right one's entry
//    distance on the stack: mesh_traverse_children says why that is the same test);
//  * a world leaf starts a fresh record (distance = inf) and, if any of its meshes is
//    hit, OVERWRITES the running result - so the answer is the last hit world leaf's
//    closest triangle, exactly as the reference returns it;
//  * ties keep the first triangle found (strict t < closest).
// Vertices are pre-transformed on upload with the reference's operation order, which
// gives the same floats the reference recomputes per test.
#pragma once
#include "dev_math.cuh"

namespace rc {

// Device view of the scene.  Nodes: two float4 per node (min.xyz|w0, max.xyz|w1), the
// mesh nodes interleaved in one array (node i at nodes[2i], nodes[2i+1]: one 32-byte
// sector per visit).  Mesh-level inner nodes hold global child indices; mesh-level
// leaves hold (0x80000000|count, first triangle slot).  World leaves hold
// (0x80000000|count, first slot in world_mesh).  Triangles are stored in leaf order,
// the three records a test reads interleaved (slot j at tris[3j .. 3j+2]).
struct SceneView {
    const float4* __restrict__ nodes;       // mesh BVH nodes, 2 per node
    const float4* __restrict__ wnode_lo;
    const float4* __restrict__ wnode_hi;
    const int* __restrict__ world_mesh;     // mesh id per world-leaf slot
    const int* __restrict__ mesh_root;      // global root node per mesh
    const float4* __restrict__ tris;        // 3 per triangle: v0.xyz | global triangle id,
                                            // (v1 - v0).xyz | material, (v2 - v0).xyz | mesh id
    const float4* __restrict__ tri_n0;      // vertex normals (normalised, world space)
    const float4* __restrict__ tri_n1;
    const float4* __restrict__ tri_n2;
    int num_world_nodes;
    int num_meshes;
};

constexpr int kStackSize = 64;   // BVH_STACK_SIZE in the reference

// Traversal stacks.  LocalStack / LocalPairStack: per-thread arrays (local memory),
// declared by each mesh traversal when the caller passes the CallStack tag, so that
// their lifetime is the traversal.  (Stacks kept in shared memory as
// [kStackSize][block] columns measured 1.5-3.6x slower on the water workload.)  Any
// type with int& operator[] can serve as the stack of mesh_traverse_impl.
struct LocalStack {
    int s[kStackSize];
    __device__ __forceinline__ int& operator[](int i) { return s[i]; }
};
// CallStack: the tag of the persistent passes' traversal (mesh_traverse_children).
struct CallStack {};
// Its per-traversal stack: node index and box entry distance (float bits) per entry.
struct LocalPairStack {
    int2 s[kStackSize];
    __device__ __forceinline__ int2& operator[](int i) { return s[i]; }
};

struct HitRec {
    float t, u, v;
    int slot;       // triangle slot (leaf order) of the reported hit, -1 if none
};

// aabb::hit with the per-ray reciprocals (1/d computed once: the same division the
// reference repeats per box).  NaN and -0 behaviour follows the ternaries as written.
__device__ __forceinline__ bool box_hit(float4 lo, float4 hi, F3 o, F3 inv, float tmin, float tmax) {
    float t0 = (lo.x - o.x) * inv.x, t1 = (hi.x - o.x) * inv.x;
    if (inv.x < 0) { float s = t0; t0 = t1; t1 = s; }
    tmin = t0 > tmin ? t0 : tmin;
    tmax = t1 < tmax ? t1 : tmax;
    if (tmax < tmin) return false;
    t0 = (lo.y - o.y) * inv.y; t1 = (hi.y - o.y) * inv.y;
    if (inv.y < 0) { float s = t0; t0 = t1; t1 = s; }
    tmin = t0 > tmin ? t0 : tmin;
    tmax = t1 < tmax ? t1 : tmax;
    if (tmax < tmin) return false;
    t0 = (lo.z - o.z) * inv.z; t1 = (hi.z - o.z) * inv.z;
    if (inv.z < 0) { float s = t0; t0 = t1; t1 = s; }
    tmin = t0 > tmin ? t0 : tmin;
    tmax = t1 < tmax ? t1 : tmax;
    if (tmax < tmin) return false;
    return true;
}

// The traversal's constants of a ray, in the form the box test reads them: (x, y) pairs
// for the packed two-lane FP32 instructions.
struct RayBox {
    unsigned long long noxy, ixy;   // (-o.x, -o.y), (1/d.x, 1/d.y)
    float noz, iz;
    bool sx, sy, sz;                // 1/d < 0: the high plane is the near one
};

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// (a - o) * inv of two coordinates at once, each lane rounded as the scalar operations
// round (a + (-o) is a - o)
__device__ __forceinline__ void slab2(float ax, float ay, unsigned long long no, unsigned long long inv, float& tx,
                                      float& ty) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(ax, ay)), "l"(no));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(r), "l"(inv));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(tx), "=f"(ty) : "l"(r));
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ RayBox ray_box(F3 o, F3 inv) {
    return {pack2(-o.x, -o.y), pack2(inv.x, inv.y), -o.z, inv.z, inv.x < 0, inv.y < 0, inv.z < 0};
}

// box_hit in two parts: the same slab arithmetic, with the box's entry distance n
// (tmin and the three near-slab distances, NaNs skipped, as box_hit folds them) kept.
// box_hit's early exits never change its answer (the interval only narrows), so it
// equals !(far < near) over all three slabs: box_entry returns exactly box_hit(tmax),
// and for any tmax' <= tmax, box_hit(tmax') == box_entry(tmax) && !(tmax' < n).
// box_hit's folds `t > a ? t : a` and `t < b ? t : b` skip a NaN t, as the max and min
// instructions do (a and b are never NaN), and the order of the folds does not matter;
// the two differ only in the sign of a zero, which no comparison sees.
// The traversal is issue- and latency-bound, and compares and selects run at half the
// FP32 rate, so the test is kept to 8 packed or scalar FP32 operations, 6 selects, 6
// (three-input) maxima and minima and one compare per box, against 12 + 6 + 12 + 3 with
// the folds written as compare-and-select: light pass 12.97 -> 12.02 ms (water pool,
// 16.7M paths), 40.9 -> 36.5 ms (2,000 gems, 4.2M paths).
__device__ __forceinline__ bool box_entry(float4 lo, float4 hi, const RayBox& r, float tmin, float tmax, float& n) {
    float lx, ly, hx, hy;
    slab2(lo.x, lo.y, r.noxy, r.ixy, lx, ly);
    slab2(hi.x, hi.y, r.noxy, r.ixy, hx, hy);
    const float lz = (lo.z + r.noz) * r.iz, hz = (hi.z + r.noz) * r.iz;
    const float near = max3f(r.sx ? hx : lx, r.sy ? hy : ly, r.sz ? hz : lz);
    const float far = min3f(r.sx ? lx : hx, r.sy ? ly : hy, r.sz ? lz : hz);
    n = fmaxf(near, tmin);
    return !(fminf(far, tmax) < n);
}

// Möller-Trumbore as src/Triangle.cpp:44-66 computes it.
__device__ __forceinline__ bool tri_hit(const SceneView& s, int slot, F3 o, F3 d, float tmin, float tmax,
                                        float& t_out, float& u_out, float& v_out) {
    float4 a = __ldg(&s.tris[3 * slot]);
    float4 b = __ldg(&s.tris[3 * slot + 1]);
    float4 c = __ldg(&s.tris[3 * slot + 2]);
    F3 v0 = xyz(a), e1 = xyz(b), e2 = xyz(c);
    F3 pvec = cross(d, e2);
    float det = dot(e1, pvec);
    if (fabsf(det) < 0.0000001f) return false;
    float inv_det = 1.0f / det;
    F3 tvec = o - v0;
    float u = dot(tvec, pvec) * inv_det;
    if (u < 0.0f || u > 1.0f) return false;
    F3 qvec = cross(tvec, e1);
    float v = dot(d, qvec) * inv_det;
    if (v < 0.0f || u + v > 1.0f) return false;
    float t = dot(e2, qvec) * inv_det;
    if (t > tmin && t < tmax) {
        t_out = t; u_out = u; v_out = v;
        return true;
    }
    return false;
}

// Mesh::hit on one mesh with the running record of the current world leaf.
// Returns false (and sets *overflow) if the stack would exceed kStackSize.
template <class Stack>
__device__ __forceinline__ bool mesh_traverse(const SceneView& s, int mesh, F3 o, F3 d, F3 inv, float tmin,
                                              HitRec& rec, bool& any, int* overflow, Stack& stack);

template <class Stack>
__device__ __forceinline__ bool mesh_traverse_impl(const SceneView& s, int mesh, F3 o, F3 d, F3 inv, float tmin,
                                                   HitRec& rec, bool& any, int* overflow, Stack& stack) {
    int sp = 0;
    stack[sp++] = __ldg(&s.mesh_root[mesh]);
    while (sp) {
        int id = stack[--sp];
        float4 lo = __ldg(&s.nodes[2 * id]);
        float4 hi = __ldg(&s.nodes[2 * id + 1]);
        if (!box_hit(lo, hi, o, inv, tmin, rec.t)) continue;
        uint32_t w0 = __float_as_uint(lo.w), w1 = __float_as_uint(hi.w);
        if (w0 & 0x80000000u) {
            int cnt = (int)(w0 & 0x7fffffffu);
            for (int k = 0; k < cnt; ++k) {
                int slot = (int)w1 + k;
                float t, u, v;
                if (tri_hit(s, slot, o, d, tmin, rec.t, t, u, v)) {
                    rec.t = t; rec.u = u; rec.v = v; rec.slot = slot;
                    any = true;
                }
            }
        } else {
            if (sp + 2 > kStackSize) { *overflow = 1; return false; }
            stack[sp++] = (int)w1;   // right first ...
            stack[sp++] = (int)w0;   // ... so the left child is popped first
        }
    }
    return true;
}

// Mesh::hit (src/mesh.cpp:70-105) visits nodes in left-first DFS order and tests each
// box when it is popped, against the running distance then.  mesh_traverse_children
// (the persistent passes, one lane per ray) and search_run (the staged passes, a warp's
// lanes in phases) test both children's boxes at their parent instead, with the same
// outcome: the left child is the node the reference pops next, with the same distance, so
// its test is the reference's; the right child is popped only after the left subtree, when
// the distance may have shrunk.  The distance never grows, so a right box that fails now
// fails then too (box_hit is monotone in tmax) and is not pushed; one that passes is
// pushed with its entry distance n, and at its pop the reference's test is
// !(distance < n) (box_entry).  Same nodes, same triangles, same order.
// Measured on the water pool (light pass per iteration): pop-and-test
// (mesh_traverse_impl) 13.3 ms, children tested at the parent 11.9 ms, four-wide records
// of grandchildren tested at the grandparent 14.7 ms.
template <class Stack>
__device__ __forceinline__ bool mesh_traverse_children(const SceneView& s, int mesh, F3 o, F3 d, F3 inv,
                                                       float tmin, HitRec& rec, bool& any, int* overflow,
                                                       Stack& stack) {
    const int root = __ldg(&s.mesh_root[mesh]);
    float4 lo = __ldg(&s.nodes[2 * root]);
    float4 hi = __ldg(&s.nodes[2 * root + 1]);
    const RayBox rb = ray_box(o, inv);
    float n;
    bool active = box_entry(lo, hi, rb, tmin, rec.t, n);
    int sp = 0;
    while (active) {
        const uint32_t w0 = __float_as_uint(lo.w), w1 = __float_as_uint(hi.w);
        bool descend = false;
        if (!(w0 & 0x80000000u)) {
            // both children's boxes (two independent loads in flight) at the distance now;
            // the left one is the reference's next test exactly, the right one waits with
            // its entry distance
            const float4 llo = __ldg(&s.nodes[2 * w0]), lhi = __ldg(&s.nodes[2 * w0 + 1]);
            const float4 rlo = __ldg(&s.nodes[2 * w1]), rhi = __ldg(&s.nodes[2 * w1 + 1]);
            float nl, nr;
            const bool hl = box_entry(llo, lhi, rb, tmin, rec.t, nl);
            const bool hr = box_entry(rlo, rhi, rb, tmin, rec.t, nr);
            if (hl && hr) {
                if (sp >= kStackSize) { *overflow = 1; return false; }
                stack[sp++] = make_int2((int)w1, __float_as_int(nr));
            }
            descend = hl || hr;
            lo = hl ? llo : rlo;
            hi = hl ? lhi : rhi;
        } else {
            const int cnt = (int)(w0 & 0x7fffffffu);
            for (int k = 0; k < cnt; ++k) {
                const int slot = (int)w1 + k;
                float t, u, v;
                if (tri_hit(s, slot, o, d, tmin, rec.t, t, u, v)) {
                    rec.t = t; rec.u = u; rec.v = v; rec.slot = slot;
                    any = true;
                }
            }
        }
        if (!descend) {
            // pop pending right children until one whose box the current distance reaches
            int next = -1;
            while (sp > 0 && next < 0) {
                const int2 e = stack[--sp];
                if (!(rec.t < __int_as_float(e.y))) next = e.x;
            }
            active = next >= 0;
            if (active) {
                lo = __ldg(&s.nodes[2 * next]);
                hi = __ldg(&s.nodes[2 * next + 1]);
            }
        }
    }
    return true;
}

template <class Stack>
__device__ __forceinline__ bool mesh_traverse(const SceneView& s, int mesh, F3 o, F3 d, F3 inv, float tmin,
                                              HitRec& rec, bool& any, int* overflow, Stack& stack) {
    return mesh_traverse_impl(s, mesh, o, d, inv, tmin, rec, any, overflow, stack);
}
template <>
__device__ __forceinline__ bool mesh_traverse<CallStack>(const SceneView& s, int mesh, F3 o, F3 d, F3 inv,
                                                         float tmin, HitRec& rec, bool& any, int* overflow,
                                                         CallStack&) {
    LocalPairStack st;
    return mesh_traverse_children(s, mesh, o, d, inv, tmin, rec, any, overflow, st);
}

// Scene::hit.  `out` is the reported record (t = inf when nothing was hit).  `stack`
// serves the mesh levels; the world level (several world leaves only) uses its own.
template <class Stack>
__device__ __forceinline__ bool scene_hit(const SceneView& s, F3 o, F3 d, float tmin, HitRec& out, int* overflow,
                                          Stack& stack) {
    F3 inv = {1.0f / d.x, 1.0f / d.y, 1.0f / d.z};
    out.t = INFINITY; out.u = 0.0f; out.v = 0.0f; out.slot = -1;
    bool hit = false;
    if (s.num_world_nodes == 1) {
        // single world leaf (a scene of one mesh)
        float4 lo = __ldg(&s.wnode_lo[0]);
        float4 hi = __ldg(&s.wnode_hi[0]);
        if (!box_hit(lo, hi, o, inv, tmin, out.t)) return false;
        uint32_t w0 = __float_as_uint(lo.w), w1 = __float_as_uint(hi.w);
        int cnt = (int)(w0 & 0x7fffffffu);
        HitRec leaf = {INFINITY, 0.0f, 0.0f, -1};
        bool any = false;
        for (int k = 0; k < cnt; ++k) {
            int mesh = __ldg(&s.world_mesh[w1 + k]);
            bool mesh_any = false;
            if (!mesh_traverse(s, mesh, o, d, inv, tmin, leaf, mesh_any, overflow, stack)) return false;
            any |= mesh_any;
        }
        if (any) out = leaf;
        return any;
    }
    int wstack[kStackSize];
    int sp = 0;
    wstack[sp++] = 0;
    while (sp) {
        int id = wstack[--sp];
        float4 lo = __ldg(&s.wnode_lo[id]);
        float4 hi = __ldg(&s.wnode_hi[id]);
        if (!box_hit(lo, hi, o, inv, tmin, out.t)) continue;
        uint32_t w0 = __float_as_uint(lo.w), w1 = __float_as_uint(hi.w);
        if (w0 & 0x80000000u) {
            int cnt = (int)(w0 & 0x7fffffffu);
            HitRec leaf = {INFINITY, 0.0f, 0.0f, -1};   // fresh Isect temp_rec
            bool any = false;
            for (int k = 0; k < cnt; ++k) {
                int mesh = __ldg(&s.world_mesh[w1 + k]);
                bool mesh_any = false;
                if (!mesh_traverse(s, mesh, o, d, inv, tmin, leaf, mesh_any, overflow, stack)) return false;
                any |= mesh_any;
            }
            if (any) { out = leaf; hit = true; }   // unconditional overwrite (world-leaf quirk)
        } else {
            if (sp + 2 > kStackSize) { *overflow = 1; return false; }
            wstack[sp++] = (int)w1;
            wstack[sp++] = (int)w0;
        }
    }
    return hit;
}

// Scene::hit as a state machine: one lane's search, put down and taken up between nodes,
// so that a warp can run its lanes' searches in phases (search_run) and lanes whose
// search has ended can shade and start new rays while the others' searches wait.  Each
// search visits the nodes and triangles that scene_hit visits, in the same order, with
// the same tests.
constexpr uint32_t kLeafFlag = 0x80000000u;     // as in the node words
constexpr uint32_t kSearchIdle = 0xffffffffu;
struct SearchStack {
    int2 s[kStackSize];    // waiting right children: node, entry distance
    int w[kStackSize];     // waiting world nodes
};
struct Search {
    RayBox rb;             // the ray's (negated) origin and reciprocals
    HitRec rec, out;       // the current world leaf's record; the reported hit so far
    uint32_t w0, w1;       // current node: child indices, or kLeafFlag | triangles left, next slot;
                           // kLeafFlag alone: between meshes; kSearchIdle: no search
    int sp;                // waiting right children
    int mesh, mesh_end;    // rest of the current leaf's mesh list
    int wsp;               // waiting world nodes
    __device__ __forceinline__ F3 origin() const {
        float nx, ny;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(nx), "=f"(ny) : "l"(rb.noxy));
        return {-nx, -ny, -rb.noz};
    }
};

__device__ __forceinline__ void search_begin(Search& q, SearchStack& st, F3 o, F3 d) {
    q.rb = ray_box(o, F3{1.0f / d.x, 1.0f / d.y, 1.0f / d.z});
    q.rec = q.out = HitRec{INFINITY, 0.0f, 0.0f, -1};
    q.w0 = kLeafFlag;
    q.sp = 0;
    q.mesh = q.mesh_end = 0;
    st.w[0] = 0;
    q.wsp = 1;
}

// Between meshes: on to the next mesh whose root box the ray enters, or idle: the search has
// ended and q.out is the reported hit.  A world leaf starts a fresh record and overwrites
// the reported one if any of its meshes was hit.
__device__ __forceinline__ void search_world(const SceneView& s, Search& q, SearchStack& st, float tmin,
                                             int* overflow) {
    for (;;) {
        float n;
        if (q.mesh < q.mesh_end) {
            const int root = __ldg(&s.mesh_root[__ldg(&s.world_mesh[q.mesh++])]);
            const float4 lo = __ldg(&s.nodes[2 * root]), hi = __ldg(&s.nodes[2 * root + 1]);
            if (!box_entry(lo, hi, q.rb, tmin, q.rec.t, n)) continue;
            q.w0 = __float_as_uint(lo.w);
            q.w1 = __float_as_uint(hi.w);
            return;
        }
        if (q.rec.slot >= 0) q.out = q.rec;
        q.rec = HitRec{INFINITY, 0.0f, 0.0f, -1};
        if (q.wsp == 0) { q.w0 = kSearchIdle; return; }
        const int id = st.w[--q.wsp];
        const float4 lo = __ldg(&s.wnode_lo[id]), hi = __ldg(&s.wnode_hi[id]);
        if (!box_entry(lo, hi, q.rb, tmin, q.out.t, n)) continue;
        const uint32_t w0 = __float_as_uint(lo.w), w1 = __float_as_uint(hi.w);
        if (w0 & kLeafFlag) {
            q.mesh = (int)w1;
            q.mesh_end = (int)(w1 + (w0 & ~kLeafFlag));
        } else {
            if (q.wsp + 2 > kStackSize) { *overflow = 1; q.out.slot = -1; q.w0 = kSearchIdle; return; }
            st.w[q.wsp++] = (int)w1;
            st.w[q.wsp++] = (int)w0;
        }
    }
}

// The next waiting right child that the current distance reaches, or between meshes.
__device__ __forceinline__ void search_pop(const SceneView& s, Search& q, SearchStack& st) {
    q.w0 = kLeafFlag;
    while (q.sp > 0) {
        const int2 e = st.s[--q.sp];
        if (q.rec.t < __int_as_float(e.y)) continue;
        q.w0 = __float_as_uint(__ldg(&s.nodes[2 * e.x].w));
        q.w1 = __float_as_uint(__ldg(&s.nodes[2 * e.x + 1].w));
        break;
    }
}

// A warp's searches (every lane of the warp calls it), until at most `keep` lanes still
// search.  Per round, the lanes at inner nodes test their two children, or the lanes at
// leaves test their next triangle, or the lanes between meshes go on to their next one,
// whichever are the most; lanes that have nothing left below take their next waiting node.
// (A lane per ray in a plain loop runs a warp's inner, leaf and between-mesh code in turn
// for the few lanes that need each: 9.4 lanes active on average on the water pool, 15.4 in
// phases.  Up to kInnerSteps node steps go between two votes: 1, 2, 3 steps 9.8, 9.8, 9.6
// ms of light pass.)
constexpr int kInnerSteps = 3;
__device__ __forceinline__ void search_run(const SceneView& s, Search& q, SearchStack& st, F3 d, float tmin, int keep,
                                           int* overflow) {
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, q.w0 == kSearchIdle);
        if (32 - __popc(idle) <= keep) break;
        const unsigned inner = __ballot_sync(0xffffffffu, (int)q.w0 >= 0);
        const unsigned between = __ballot_sync(0xffffffffu, q.w0 == kLeafFlag);
        const int ni = __popc(inner), nb = __popc(between), nl = 32 - __popc(idle | inner | between);
        if (ni >= nl && ni >= nb) {
#pragma unroll 1
            for (int k = 0; k < kInnerSteps; ++k)
                if ((int)q.w0 >= 0) {
                    const float4 llo = __ldg(&s.nodes[2 * q.w0]), lhi = __ldg(&s.nodes[2 * q.w0 + 1]);
                    const float4 rlo = __ldg(&s.nodes[2 * q.w1]), rhi = __ldg(&s.nodes[2 * q.w1 + 1]);
                    float el, er;
                    const bool hl = box_entry(llo, lhi, q.rb, tmin, q.rec.t, el);
                    const bool hr = box_entry(rlo, rhi, q.rb, tmin, q.rec.t, er);
                    const bool push = hl && hr, full = q.sp >= kStackSize;
                    if (push && !full) st.s[q.sp++] = make_int2((int)q.w1, __float_as_int(er));
                    q.w0 = __float_as_uint(hl ? llo.w : rlo.w);
                    q.w1 = __float_as_uint(hl ? lhi.w : rhi.w);
                    if (!(hl || hr)) search_pop(s, q, st);
                    if (push && full) { *overflow = 1; q.out.slot = -1; q.w0 = kSearchIdle; }
                }
        } else if (nl >= nb) {
            if ((int)q.w0 < 0 && q.w0 != kLeafFlag && q.w0 != kSearchIdle) {
                float t, u, v;
                if (tri_hit(s, (int)q.w1, q.origin(), d, tmin, q.rec.t, t, u, v)) q.rec = HitRec{t, u, v, (int)q.w1};
                --q.w0;
                ++q.w1;
                if (q.w0 == kLeafFlag) search_pop(s, q, st);
            }
        } else if (q.w0 == kLeafFlag) {
            search_world(s, q, st, tmin, overflow);
        }
    }
}

// Scene::hit with per-traversal local-memory stacks.
__device__ __forceinline__ bool scene_hit(const SceneView& s, F3 o, F3 d, float tmin, HitRec& out, int* overflow) {
    CallStack st;
    return scene_hit(s, o, d, tmin, out, overflow, st);
}

// Attributes Triangle::hit fills in (src/Triangle.cpp:68-80), for the reported triangle.
struct Isect {
    F3 ng, ns, pos, dir;
    float t, u, v;
    bool front;
    int material;
    int tri;     // global triangle id
    int mesh;
};

__device__ __forceinline__ void fill_isect(const SceneView& s, const HitRec& h, F3 o, F3 d, Isect& is) {
    float4 a = __ldg(&s.tris[3 * h.slot]);
    float4 b = __ldg(&s.tris[3 * h.slot + 1]);
    float4 c = __ldg(&s.tris[3 * h.slot + 2]);
    F3 e1 = xyz(b), e2 = xyz(c);
    is.t = h.t; is.u = h.u; is.v = h.v;
    is.ng = normalize(cross(e1, e2));
    F3 n0 = xyz(__ldg(&s.tri_n0[h.slot]));
    F3 n1 = xyz(__ldg(&s.tri_n1[h.slot]));
    F3 n2 = xyz(__ldg(&s.tri_n2[h.slot]));
    float w = 1 - h.u - h.v;
    is.ns = n0 * w + n1 * h.u + n2 * h.v;
    is.front = dot(is.ns, d) < 0;
    is.pos = o + d * h.t;
    is.dir = d;
    is.tri = (int)__float_as_uint(a.w);
    is.material = (int)__float_as_uint(b.w);
    is.mesh = (int)__float_as_uint(c.w);
}

}  // namespace rc
