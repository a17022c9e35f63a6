// Radius gather at the camera vertices (Path_Vertices::get_contrib,
// src/Path_Vertices.h:46-68, over KD_Tree::find_closest_in_radius,
// src/KD_Tree.cpp:217-280).
//
// The photons the reference's query returns for a camera vertex q are exactly
// { p : ((dx*dx + dy*dy) + dz*dz) < r^2 } in FP32 without contraction: its descent
// prunes a side only when (q[axis] - split)^2 >= r^2, and every photon beyond that
// plane has a squared distance at least as large (rounding is monotonic), so pruning
// never drops a photon the predicate accepts.  The set does not depend on the tree's
// shape, so the gather may walk the photons in any order, as long as it skips only
// boxes that provably hold no accepted photon and tests every other photon with the
// reference's predicate.
//
// Layout (launch_photon_order).  The photons, sorted along a Hilbert curve, are cut into
// 2^Lc runs of at most 32 (chunks), Lc being the shallowest level whose runs hold at most
// 31 where the cut is even.  Each chunk has its photons' bounding box, with its first
// position and count in the spare .w words; every node above has the union of its
// children's boxes.
//
// Work split (k_gather).  Queries are sorted in space too (launch_query_order) and a
// warp owns G consecutive ones (a group), one per lane.  The warp descends the box hierarchy
// once for the whole group, E levels per step (lane j tests descendant j's box against
// the group's bounding box grown by the radius), down to the candidate chunks.  At a
// chunk each lane tests its own query's sphere against the chunk box (a ballot names the
// overlapping queries), each lane loads one of the chunk's photons, and for every
// overlapping query the warp tests all of the chunk's photons at once: a query x photon
// cross product, one photon per lane, the query broadcast from shared memory.  Accepted
// (query slot, photon) pairs collect in a per-warp pending list, and every 32 of them
// go to the sink with all lanes busy.  The render's sink evaluates the merges (the
// camera vertex's BSDF at the photon's direction, MIS weight, photon throughput) from
// per-query BSDF state staged in shared memory when the group starts, sums them per
// query in shared memory, and adds each query's sum into its FP64 pixel once.  The
// parity hook's sink records photon ids instead; both are the same kernel template.
#include <algorithm>
#include "vm.cuh"
#include "bsdf.cuh"

namespace rc {

namespace {

constexpr int kWarpsPerBlock = 8;
// DFS stack of subtree roots per warp.  Lc <= 24 for n < 2^28 photons, so a path from
// the root crosses at most ceil(24 / E) expansion steps, the last of which reaches the
// chunks (processed at once, never pushed): at most 4 x 31 + 1 = 125 (E = 5) or
// 5 x 15 + 1 = 76 (E = 4) pending roots.
constexpr int kRootStack = 128;
constexpr unsigned kFull = 0xffffffffu;

struct ChunkTree {
    const float4* __restrict__ lo;    // node boxes, heap order, levels [0, lc]; chunk level: .w = first position
    const float4* __restrict__ hi;    //                                          chunk level: .w = photon count
    const float4* __restrict__ pos;   // sorted photon positions (TreePhotons::t0)
    int lc;                           // chunk level (-1: no photons)
};

// Squared distance from q to a box, formed like the acceptance test, so that it never
// exceeds the squared distance to any photon inside the box (rounding is monotonic).
__device__ __forceinline__ bool box_outside(F3 q, float4 lo, float4 hi, float r2) {
    const float dx = q.x < lo.x ? lo.x - q.x : (q.x > hi.x ? q.x - hi.x : 0.0f);
    const float dy = q.y < lo.y ? lo.y - q.y : (q.y > hi.y ? q.y - hi.y : 0.0f);
    const float dz = q.z < lo.z ? lo.z - q.z : (q.z > hi.z ? q.z - hi.z : 0.0f);
    return !(dx * dx + dy * dy + dz * dz < r2);
}

// The same bound between two boxes: never more than the squared distance from any
// point of the first (a query of the group) to any point of the second (a photon).
__device__ __forceinline__ bool gap_outside(float4 glo, float4 ghi, float4 lo, float4 hi, float r2) {
    const float dx = lo.x > ghi.x ? lo.x - ghi.x : (glo.x > hi.x ? glo.x - hi.x : 0.0f);
    const float dy = lo.y > ghi.y ? lo.y - ghi.y : (glo.y > hi.y ? glo.y - hi.y : 0.0f);
    const float dz = lo.z > ghi.z ? lo.z - ghi.z : (glo.z > hi.z ? glo.z - hi.z : 0.0f);
    return !(dx * dx + dy * dy + dz * dz < r2);
}

// Bounding box of the queries of the lanes with `in` set (all lanes call it).
__device__ __forceinline__ void warp_box(bool in, F3 q, float4& lo, float4& hi) {
    float lx = in ? q.x : INFINITY, ly = in ? q.y : INFINITY, lz = in ? q.z : INFINITY;
    float hx = in ? q.x : -INFINITY, hy = in ? q.y : -INFINITY, hz = in ? q.z : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o)); ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
        lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o)); hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
        hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o)); hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
    }
    lo = make_float4(lx, ly, lz, 0.0f);
    hi = make_float4(hx, hy, hz, 0.0f);
}

// Lane holding the largest value (the lowest such lane on ties).
__device__ __forceinline__ int warp_argmax(float v) {
    int at = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ov > v || (ov == v && oa < at)) { v = ov; at = oa; }
    }
    return at;
}

// Surface of a box grown by `g` on every side (a proxy for how many chunk boxes it meets).
__device__ __forceinline__ float box_surface(float4 lo, float4 hi, float g) {
    const float ex = hi.x - lo.x + 2.0f * g, ey = hi.y - lo.y + 2.0f * g, ez = hi.z - lo.z + 2.0f * g;
    return ex * ey + ey * ez + ex * ez;
}

// The reference's acceptance test (src/KD_Tree.cpp:217-280): ((dx*dx + dy*dy) + dz*dz) < r2.
__device__ __forceinline__ bool in_radius(F3 q, float px, float py, float pz, float r2) {
    const float dx = q.x - px, dy = q.y - py, dz = q.z - pz;
    return dx * dx + dy * dy + dz * dz < r2;
}

// Camera-vertex state a merge evaluation needs, staged once per query.  29 words: an
// odd stride, so lanes reading different queries' fields hit different banks.
struct QState {
    int kind;
    float R[3], ior, a2, s;
    float fx[3], fy[3], fz[3];   // shading frame
    float wo[3];                 // local direction towards the previous camera vertex
    float ng[3];
    float wo_ng, fwo, dvm;       // dot(to_world(wo), Ng), plastic Fresnel at wo, camera dVM
    float tp[3];                 // camera throughput x VM normalisation
    float pad;
};
static_assert(sizeof(QState) == 29 * 4, "QState must keep an odd word stride");

// Parking (the last two shapes).  A caustic's focus meets the spheres of a few groups with
// most of the photons, and the warps of those groups are then the gather's time.  A warp that
// has done kParkWork (chunks tested and eighths of accepted pairs: 32 pairs take as long as 4
// chunks) leaves the rest to a second launch: the current step's untested chunks one by one,
// its pending subtrees in kParkParts parts each (every kParkParts-th chunk).  An item is
// (group, first | end << 8 of its sub-group's lanes, root, part) at parked[1 + i],
// parked[0].x of them; void items have root 0.  216k queries and 20k photons behind a glass
// ball under a point light: 783 us, parked 120 (102 with kParkWork 16; 258 with subtrees
// only).  The list has to hold what the focus parks: the warps that find it full do their
// rest alone, and are the gather's time again.  With 65,535 items, against a render's list of
// 2^20 - 1 (kParkedItems), 512x512 queries behind the ball take 15.3 and 1.1 ms with 580k
// photons, 12.5 and 3.1 with 18k and 20 times the radius (2^18: 12.5); 1920x1080 with 145k
// photons 4.5 and 1.2.  Where 65,535 were enough the longer list costs nothing.
// Without a focus the second launch costs more than it gives (3.7M queries on a water
// pool's floor 1.79 ms against 2.17), so the autotuner chooses.
constexpr unsigned kParkWork = 64, kParkParts = 16;

template <bool Eval> struct GroupExtra {};
template <> struct GroupExtra<true> {
    QState qs[32];
    float acc[32][3];            // per-query merge sums (word stride 3: conflict-free)
};

template <bool Eval> struct WarpSmem {
    float4 qp[32];               // query positions (broadcast in the cross product)
    uint32_t qidx[32];           // query indices of the group's slots
    uint32_t pend_pos[64];       // accepted pairs: tree position ...
    uint8_t pend_slot[64];       // ... and query slot
    uint32_t stk[kRootStack];
    GroupExtra<Eval> g;
};

// The render's sink: merge evaluation (Path_Vertices::get_contrib, src/Path_Vertices.h:46-68)
// and FP64 pixel accumulation.
struct EvalSink {
    static constexpr bool kEval = true;
    VMParams P;
    QueryBuf qb;
    TreePhotons tp;
    const uint32_t* tree_id;
    double* accum;

    __device__ __forceinline__ void setup(WarpSmem<true>& sm, int lane, bool active, uint32_t qi) const {
        if (active) {
            const float dvm = qb.q0[qi].w;
            const float4 b = qb.q1[qi], c = qb.q2[qi], e = qb.q4[qi], g = qb.q3[qi];
            const DevMaterial& qm = P.materials[__float_as_int(b.w)];
            const int channel = __float_as_int(e.w);   // the camera path's dispersion channel
            Bsdf bs;
            bs.init(qm, xyz(b), xyz(e), true, (qm.disp > 0.0f && channel >= 0) ? (float)(channel - 1) * qm.disp : 0.0f);
            QState& st = sm.g.qs[lane];
            st.kind = bs.kind;
            st.R[0] = bs.R.x; st.R[1] = bs.R.y; st.R[2] = bs.R.z;
            st.ior = bs.ior; st.a2 = bs.a2; st.s = bs.s;
            st.fx[0] = bs.fr.x.x; st.fx[1] = bs.fr.x.y; st.fx[2] = bs.fr.x.z;
            st.fy[0] = bs.fr.y.x; st.fy[1] = bs.fr.y.y; st.fy[2] = bs.fr.y.z;
            st.fz[0] = bs.fr.z.x; st.fz[1] = bs.fr.z.y; st.fz[2] = bs.fr.z.z;
            st.wo[0] = bs.wo.x; st.wo[1] = bs.wo.y; st.wo[2] = bs.wo.z;
            st.ng[0] = c.x; st.ng[1] = c.y; st.ng[2] = c.z;
            st.wo_ng = dot(bs.fr.to_world(bs.wo), xyz(c));
            st.fwo = (bs.kind == BSDF_K_PLASTIC_GGX || bs.kind == BSDF_K_PLASTIC_SMOOTH)
                         ? fresnel_reflectance(fabsf(bs.wo.z), bs.s) : 0.0f;
            st.dvm = dvm;
            st.tp[0] = g.x * P.merge_scale; st.tp[1] = g.y * P.merge_scale; st.tp[2] = g.z * P.merge_scale;
        }
        sm.g.acc[lane][0] = 0.0f; sm.g.acc[lane][1] = 0.0f; sm.g.acc[lane][2] = 0.0f;
    }

    // Evaluate the first `count` pending pairs (lane j: pair j); sum each run of one
    // query's pairs across the lanes and add it to that query's shared sum.
    __device__ __forceinline__ void flush(WarpSmem<true>& sm, int lane, int count) const {
        F3 c = f3(0.0f);
        int s = -1;
        if (lane < count) {
            const uint32_t p = sm.pend_pos[lane];
            s = sm.pend_slot[lane];
            const QState& st = sm.g.qs[s];
            Bsdf bs;
            bs.kind = st.kind;
            bs.R = f3(st.R[0], st.R[1], st.R[2]);
            bs.ior = st.ior; bs.a2 = st.a2; bs.s = st.s; bs.cont = 0.0f;
            bs.fr.x = f3(st.fx[0], st.fx[1], st.fx[2]);
            bs.fr.y = f3(st.fy[0], st.fy[1], st.fy[2]);
            bs.fr.z = f3(st.fz[0], st.fz[1], st.fz[2]);
            bs.wo = f3(st.wo[0], st.wo[1], st.wo[2]);
            bs.radiance = true;
            const float4 p0 = __ldg(&tp.t0[p]);
            const float4 p1 = __ldg(&tp.t1[p]);
            const float2 p2 = __ldg(&tp.t2[p]);
            F3 ev;
            float fwd, rev;
            bs.eval_pdf(xyz(p1), f3(st.ng[0], st.ng[1], st.ng[2]), st.wo_ng, st.fwo, ev, fwd, rev);
            const float weight = 1.0f / (1.0f + st.dvm * rev + p0.w * fwd);
            c = ev * f3(p1.w, p2.x, p2.y) * weight;
            if (P.path_contrib) {
                // learned-proposal training signal: the squared luminance this merge adds
                // to its pixel, summed per light path
                const F3 img = f3(st.tp[0], st.tp[1], st.tp[2]) * c;
                const float lum = (fabsf(img.x) + fabsf(img.y) + fabsf(img.z)) * (1.0f / 3.0f);
                if (lum > 0.0f) atomicAdd(&P.path_contrib[__ldg(&P.photon_path[__ldg(&tree_id[p])])], lum * lum);
            }
        }
        // runs of equal slot, numbered by their heads (one query can form two runs in a
        // flush: its pairs from two chunks with another query's between them)
        const int sprev = __shfl_up_sync(kFull, s, 1);
        const unsigned heads = __ballot_sync(kFull, lane == 0 || sprev != s);
        const int run = __popc(heads & ((2u << lane) - 1u));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float x = __shfl_up_sync(kFull, c.x, o);
            const float y = __shfl_up_sync(kFull, c.y, o);
            const float z = __shfl_up_sync(kFull, c.z, o);
            const int ro = __shfl_up_sync(kFull, run, o);
            if (lane >= o && ro == run) { c.x += x; c.y += y; c.z += z; }
        }
        const int snext = __shfl_down_sync(kFull, s, 1);
        if (s >= 0 && (lane == 31 || snext != s) && !is_zero(c)) {
            atomicAdd(&sm.g.acc[s][0], c.x);
            atomicAdd(&sm.g.acc[s][1], c.y);
            atomicAdd(&sm.g.acc[s][2], c.z);
        }
    }

    __device__ __forceinline__ void finish(WarpSmem<true>& sm, int lane, bool active, uint32_t qi) const {
        if (!active) return;
        const QState& st = sm.g.qs[lane];
        const F3 r = f3(st.tp[0], st.tp[1], st.tp[2]) * f3(sm.g.acc[lane][0], sm.g.acc[lane][1], sm.g.acc[lane][2]);
        if (is_zero(r)) return;
        const long long pixel = __float_as_int(qb.q2[qi].w);
        atomicAdd(&accum[3 * pixel + 0], (double)r.x);
        atomicAdd(&accum[3 * pixel + 1], (double)r.y);
        atomicAdd(&accum[3 * pixel + 2], (double)r.z);
    }
};

// The parity hook's sink: per query, the ids of the photons it accepts.  Without
// `offsets` it counts (counts[] zeroed by the caller), with them it writes the ids at
// offsets[q] + cursor[q]++ (cursor zeroed by the caller).
struct SetSink {
    static constexpr bool kEval = false;
    const uint32_t* tree_id;
    int* counts;
    const long long* offsets;
    int* cursor;
    int* idx;

    __device__ __forceinline__ void setup(WarpSmem<false>&, int, bool, uint32_t) const {}
    __device__ __forceinline__ void flush(WarpSmem<false>& sm, int lane, int count) const {
        if (lane >= count) return;
        const uint32_t qi = sm.qidx[sm.pend_slot[lane]];
        const uint32_t p = sm.pend_pos[lane];
        if (!offsets) atomicAdd(&counts[qi], 1);
        else idx[offsets[qi] + atomicAdd(&cursor[qi], 1)] = (int)__ldg(&tree_id[p]);
    }
    __device__ __forceinline__ void finish(WarpSmem<false>&, int, bool, uint32_t) const {}
};

// One group of G queries per warp (stage 0; 1: and it may park subtrees; 2: one parked item
// at a time).  MinBlocks
// (resident blocks per SM the register allocation must allow), G and E (levels per
// expansion step) are the launch shape the autotuner picks.  counters (optional, 4 u64
// accumulated): accepted pairs, photon tests (chunk photons x overlapping queries), chunks
// tested, boxes tested.
template <int kStage, int MinBlocks, int G, int E, class Sink>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MinBlocks)
    k_gather(const ChunkTree t, const float* __restrict__ qpos, int qstride, const uint32_t* __restrict__ order,
             long long nq, const unsigned long long* __restrict__ nq_dev, const int* __restrict__ skip, float r2,
             const Sink sink, uint4* parked, uint32_t room, unsigned long long* __restrict__ counters,
             int* __restrict__ err) {
    constexpr bool kRest = kStage == 2;
    static_assert(G == 16 || G == 32, "a group is a half or a whole warp of queries");
    static_assert(E >= 1 && E <= 5, "an expansion step tests at most 32 descendants");
    // device-side count (bounded by the capacity nq) and an iteration-wide skip flag,
    // for iterations enqueued without a host round trip
    if (skip && *skip) return;
    if (nq_dev) nq = (long long)min(*nq_dev, (unsigned long long)nq);
    __shared__ WarpSmem<Sink::kEval> smem[kWarpsPerBlock];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    WarpSmem<Sink::kEval>& sm = smem[warp];
    if (t.lc < 0) return;
    const uint32_t items = kRest ? min(parked[0].x, room) : 0u;
    for (long long w = (long long)blockIdx.x * kWarpsPerBlock + warp;; w += (long long)gridDim.x * kWarpsPerBlock) {
    uint4 item = make_uint4((uint32_t)w, 0u, 1u, 0u);
    if (kRest) {
        if (w >= items) return;
        item = parked[1 + w];
        if (item.z == 0u) continue;
    }
    const long long first = (long long)item.x * G;
    if (first >= nq) return;
    const int nslots = (int)min((long long)G, nq - first);
    const bool active = lane < nslots;
    uint32_t qi = 0;
    F3 q = f3(0.0f);
    if (active) {
        qi = __ldg(&order[first + lane]);
        const float* qp = qpos + (long long)qstride * qi;
        q = f3(qp[0], qp[1], qp[2]);
        sm.qidx[lane] = qi;
        sm.qp[lane] = make_float4(q.x, q.y, q.z, 0.0f);
    }
    sink.setup(sm, lane, active, qi);
    __syncwarp();
    // The group is traversed as one or more sub-groups (lane ranges [a, b) of the sorted
    // queries, `in` = this lane's query belongs to the current one, glo/ghi its box).
    bool in = false;
    float4 glo, ghi;

    bool park = kStage == 1 && t.lc > 0;
    int np = 0;
    unsigned n_acc = 0, n_tests = 0, n_chunks = 0, n_boxes = 0;

    // Append one chunk's accepted pairs: this lane's photon (tree position p) is accepted
    // by the queries whose bits are set in `am`.  Pairs go in query by query (runs of one
    // query), every 32 to the sink.
    auto emit = [&](uint32_t am, uint32_t p) {
        unsigned qa = __reduce_or_sync(kFull, am);
        while (qa) {
            const int s = __ffs(qa) - 1;
            qa &= qa - 1u;
            const bool acc = (am >> s) & 1u;
            const unsigned m = __ballot_sync(kFull, acc);
            if (acc) {
                const int at = np + __popc(m & lt);
                sm.pend_pos[at] = p;
                sm.pend_slot[at] = (uint8_t)s;
            }
            np += __popc(m);
            __syncwarp();
            if (np >= 32) {
                sink.flush(sm, lane, 32);
                n_acc += 32;
                __syncwarp();
                const int rest = np - 32;
                uint32_t vp = 0;
                uint8_t vs = 0;
                if (lane < rest) { vp = sm.pend_pos[32 + lane]; vs = sm.pend_slot[32 + lane]; }
                __syncwarp();
                if (lane < rest) { sm.pend_pos[lane] = vp; sm.pend_slot[lane] = vs; }
                np = rest;
                __syncwarp();
            }
        }
    };

    // The candidate chunks of one expansion step: lane j holds chunk j's box (blo, bhi;
    // .w = first position, count) and bm names the chunks that met the group box.  First
    // each candidate's mask of the group's queries whose sphere meets its box (kept by
    // lane j), then the photon tests chunk by chunk, the next chunk's photons loaded
    // while the current one's are tested; the queries of a chunk are tested two at a
    // time into a per-photon mask of accepting queries.
    // Returns the candidates it left (to park) because the warp's share of work was done.
    auto chunks = [&](unsigned bm, float4 blo, float4 bhi) -> unsigned {
        uint32_t my_qm = 0;
        while (bm) {
            const int j = __ffs(bm) - 1;
            bm &= bm - 1u;
            const float4 lo = make_float4(__shfl_sync(kFull, blo.x, j), __shfl_sync(kFull, blo.y, j),
                                          __shfl_sync(kFull, blo.z, j), 0.0f);
            const float4 hi = make_float4(__shfl_sync(kFull, bhi.x, j), __shfl_sync(kFull, bhi.y, j),
                                          __shfl_sync(kFull, bhi.z, j), 0.0f);
            const unsigned qm = __ballot_sync(kFull, in && !box_outside(q, lo, hi, r2));
            if (lane == j) my_qm = qm;
        }
        unsigned cm = __ballot_sync(kFull, my_qm != 0u);
        if (!cm) return 0u;
        int j = __ffs(cm) - 1;
        uint32_t start = __shfl_sync(kFull, __float_as_uint(blo.w), j);
        uint32_t cnt = __shfl_sync(kFull, __float_as_uint(bhi.w), j);
        float4 pp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if ((uint32_t)lane < cnt) pp = __ldg(&t.pos[start + lane]);
        for (;;) {
            if (kStage == 1 && park && n_chunks + n_acc / 8 >= kParkWork) return cm;
            const uint32_t qm = __shfl_sync(kFull, my_qm, j);
            cm &= cm - 1u;
            int jn = 0;
            uint32_t sn = 0, cn = 0;
            float4 pn = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (cm) {
                jn = __ffs(cm) - 1;
                sn = __shfl_sync(kFull, __float_as_uint(blo.w), jn);
                cn = __shfl_sync(kFull, __float_as_uint(bhi.w), jn);
                if ((uint32_t)lane < cn) pn = __ldg(&t.pos[sn + lane]);
            }
            ++n_chunks;
            n_tests += cnt * (unsigned)__popc(qm);
            uint32_t am = 0, qq = qm;
            while (qq) {
                const int s0 = __ffs(qq) - 1;
                qq &= qq - 1u;
                const int s1 = qq ? __ffs(qq) - 1 : s0;
                qq &= qq - 1u;
                const float4 a = sm.qp[s0], b = sm.qp[s1];
                if (in_radius(xyz(a), pp.x, pp.y, pp.z, r2)) am |= 1u << s0;
                if (in_radius(xyz(b), pp.x, pp.y, pp.z, r2)) am |= 1u << s1;
            }
            if ((uint32_t)lane >= cnt) am = 0u;
            emit(am, start + (uint32_t)lane);
            if (!cm) return 0u;
            j = jn; start = sn; cnt = cn; pp = pn;
        }
    };

    // Room for `add` parked items, from `at`; without it the items given below the end are
    // void and the warp parks no more.  A full list is not asked again: the count stays
    // below `room` and one request of every warp in flight, however many groups the
    // launch has (counted for all of them it wraps at 2^32: 3.6M groups of some 1,200).
    auto reserve_items = [&](uint32_t add) -> uint32_t {
        uint32_t at = room;
        if (lane == 0 && __ldcg(&parked[0].x) < room) at = atomicAdd(&parked[0].x, add);
        at = __shfl_sync(kFull, at, 0);
        park = at + add <= room;
        return at;
    };
    auto write_item = [&](uint32_t at, int a, int b, uint32_t root, uint32_t which) {
        if (at < room)
            parked[1 + at] = make_uint4(item.x, (uint32_t)a | ((uint32_t)b << 8), park ? root : 0u, which);
    };

    const int lc = t.lc;
    const float4 rlo = __ldg(&t.lo[1]), rhi = __ldg(&t.hi[1]);
    // Sub-groups.  Consecutive queries of the curve can straddle a jump of the
    // curve, and a group holding two distant clusters would walk every chunk between
    // them.  A range is therefore split at its largest gap between consecutive queries
    // when the two parts' boxes, grown by 4 radii, have less than half the surface of the
    // whole range's; the parts are traversed one after another.
    const float grow = 4.0f * sqrtf(r2);
    int a = kRest ? (int)(item.y & 255u) : 0;
    const int end = kRest ? (int)(item.y >> 8) : nslots;
    while (a < end) {
        int b = end;
        warp_box(lane >= a && lane < b, q, glo, ghi);
        while (!kRest && b - a >= 4) {
            const F3 qp = f3(__shfl_up_sync(kFull, q.x, 1), __shfl_up_sync(kFull, q.y, 1), __shfl_up_sync(kFull, q.z, 1));
            const float gap = (lane > a && lane < b) ? length_sq(q - qp) : -1.0f;
            const int c = warp_argmax(gap);
            float4 llo, lhi, rlo2, rhi2;
            warp_box(lane >= a && lane < c, q, llo, lhi);
            warp_box(lane >= c && lane < b, q, rlo2, rhi2);
            if (!(box_surface(llo, lhi, grow) + box_surface(rlo2, rhi2, grow) < 0.5f * box_surface(glo, ghi, grow)))
                break;
            b = c;
            glo = llo;
            ghi = lhi;
        }
        in = lane >= a && lane < b;
        ++n_boxes;
        if (kRest || !gap_outside(glo, ghi, rlo, rhi, r2)) {
        if (lc == 0) {
            chunks(1u, rlo, rhi);
        } else {
            if (lane == 0) sm.stk[0] = item.z;
            __syncwarp();
            int sp = 1;
            while (sp > 0) {
                if (kStage == 1 && park && n_chunks + n_acc / 8 >= kParkWork) {
                    // this warp has done its share: the subtrees left, in kParkParts parts
                    // each, to the second launch
                    const uint32_t add = (uint32_t)sp * kParkParts, at = reserve_items(add);
                    for (uint32_t i = lane; i < add; i += 32) write_item(at + i, a, b, sm.stk[i / kParkParts], i % kParkParts);
                    if (park) break;
                }
                --sp;
                const uint32_t e = sm.stk[sp];
                __syncwarp();
                const int L = 31 - __clz(e);
                const int k = (lc - L) < E ? (lc - L) : E;
                const uint32_t m = 1u << k;
                const uint32_t ce = (e << k) + (uint32_t)lane;
                bool keep = false;
                float4 blo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), bhi = blo;
                if ((uint32_t)lane < m) {
                    blo = __ldg(&t.lo[ce]);
                    bhi = __ldg(&t.hi[ce]);
                    keep = (!kRest || L + k < lc || ce % kParkParts == item.w) && !gap_outside(glo, ghi, blo, bhi, r2);
                }
                n_boxes += m;
                const unsigned bm = __ballot_sync(kFull, keep);
                if (L + k == lc) {
                    unsigned left = chunks(bm, blo, bhi);
                    while (kStage == 1 && left) {
                        const uint32_t at = reserve_items((uint32_t)__popc(left));
                        if ((left >> lane) & 1u) write_item(at + __popc(left & lt), a, b, ce, ce % kParkParts);
                        if (park) break;
                        left = chunks(left, blo, bhi);
                    }
                } else {
                    const int add = __popc(bm);
                    if (sp + add > kRootStack) {   // cannot happen (bound above); flagged, not silent
                        if (lane == 0 && err) atomicOr(err, 1);
                        break;
                    }
                    if (keep) sm.stk[sp + __popc(bm & lt)] = ce;
                    sp += add;
                    __syncwarp();
                }
            }
        }
        }
        a = b;
    }
    if (np > 0) {
        __syncwarp();
        sink.flush(sm, lane, np);
        n_acc += (unsigned)np;
    }
    __syncwarp();
    sink.finish(sm, lane, active, qi);
    if (counters && lane == 0) {
        atomicAdd(&counters[0], (unsigned long long)n_acc);
        atomicAdd(&counters[1], (unsigned long long)n_tests);
        atomicAdd(&counters[2], (unsigned long long)n_chunks);
        atomicAdd(&counters[3], (unsigned long long)n_boxes);
    }
    if (!kRest) return;
    __syncwarp();
    }
}

ChunkTree chunk_tree(const PhotonTree& tree, const float4* t0) {
    return ChunkTree{tree.box_lo, tree.box_hi, t0, photon_chunk_level(tree.n)};
}

// Launch shapes: resident blocks per SM, queries per group, levels per expansion step, parking.
constexpr int kNumShapes = 10;
constexpr int kDefaultShape = 1;

int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}

template <int MB, int G, int E, bool kPark, class Sink>
void launch_shape(const ChunkTree& t, const float* qpos, int qstride, const uint32_t* order, long long nq,
                  const unsigned long long* nq_dev, const int* skip, float r2, const Sink& sink,
                  const ParkedList& list, unsigned long long* counters, int* err, cudaStream_t s) {
    const long long warps = (nq + G - 1) / G;
    const unsigned blocks = (unsigned)((warps + kWarpsPerBlock - 1) / kWarpsPerBlock);
    uint4* const parked = static_cast<uint4*>(list.p);
    if (kPark) cudaMemsetAsync(parked, 0, sizeof(uint4), s);
    k_gather<kPark ? 1 : 0, MB, G, E, Sink><<<blocks, 32 * kWarpsPerBlock, 0, s>>>(
        t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, parked, list.items, counters, err);
    if (kPark)
        k_gather<2, MB, G, E, Sink><<<MB * sm_count(), 32 * kWarpsPerBlock, 0, s>>>(
            t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, parked, list.items, counters, err);
}

template <class Sink>
void launch_variant(int v, const ChunkTree& t, const float* qpos, int qstride, const uint32_t* order, long long nq,
                    const unsigned long long* nq_dev, const int* skip, float r2, const Sink& sink,
                    const ParkedList& list, unsigned long long* counters, int* err, cudaStream_t s) {
    switch (v) {
    case 0: launch_shape<2, 32, 5, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 2: launch_shape<4, 32, 5, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 3: launch_shape<3, 32, 4, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 4: launch_shape<4, 32, 4, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 5: launch_shape<3, 16, 5, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 6: launch_shape<4, 16, 4, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 7: launch_shape<4, 16, 5, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 8: launch_shape<3, 16, 5, true>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    case 9: launch_shape<3, 32, 5, true>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    default: launch_shape<3, 32, 5, false>(t, qpos, qstride, order, nq, nq_dev, skip, r2, sink, list, counters, err, s); break;
    }
}

}  // namespace

size_t gather_parked_bytes(uint32_t items) { return sizeof(uint4) * ((size_t)items + 1); }
int gather_variants() { return kNumShapes; }
bool gather_parks(int variant) { return variant >= 8 && variant < kNumShapes; }
int gather_default_variant() { return kDefaultShape; }

const char* gather_variant_name(int v) {
    static const char* names[kNumShapes] = {
        "blocks/SM>=2, 32 queries/group, 5-level steps", "blocks/SM>=3, 32 queries/group, 5-level steps",
        "blocks/SM>=4, 32 queries/group, 5-level steps", "blocks/SM>=3, 32 queries/group, 4-level steps",
        "blocks/SM>=4, 32 queries/group, 4-level steps", "blocks/SM>=3, 16 queries/group, 5-level steps",
        "blocks/SM>=4, 16 queries/group, 4-level steps", "blocks/SM>=4, 16 queries/group, 5-level steps",
        "blocks/SM>=3, 16 queries/group, 5-level steps, parking", "blocks/SM>=3, 32 queries/group, 5-level steps, parking"};
    return (v >= 0 && v < kNumShapes) ? names[v] : "?";
}

void launch_gather(const VMParams& p, const PhotonTree& tree, TreePhotons tp, QueryBuf qb, const uint32_t* order,
                   long long nq, double* accum, const ParkedList& parked, unsigned long long* counters, cudaStream_t s,
                   int variant, const unsigned long long* nq_dev, const int* skip) {
    if (nq <= 0 || tree.n <= 0) return;
    const EvalSink sink{p, qb, tp, tree.id, accum};
    launch_variant(variant, chunk_tree(tree, tp.t0), reinterpret_cast<const float*>(qb.q0), 4, order, nq, nq_dev,
                   skip, p.radius_sqr, sink, parked, counters, p.error + ERR_GATHER, s);
}

void launch_gather_sets(const PhotonTree& tree, const float4* t0, const float* qpos, int qstride, const uint32_t* order,
                        long long nq, float r2, int* counts, const long long* offsets, int* cursor, int* idx,
                        int variant, const ParkedList& parked, unsigned long long* counters, int* err, cudaStream_t s) {
    if (nq <= 0 || tree.n <= 0) return;
    const SetSink sink{tree.id, counts, offsets, cursor, idx};
    launch_variant(variant, chunk_tree(tree, t0), qpos, qstride, order, nq, nullptr, nullptr, r2, sink,
                   parked, counters, err, s);
}

}  // namespace rc
