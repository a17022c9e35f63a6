// Light pass, camera pass and the closest-hit parity kernel.
#include <algorithm>

#include "vm.cuh"
#include "bsdf.cuh"
#include "lights.cuh"
#include "rng.cuh"

namespace rc {

namespace {

// Warp-aggregated append: one atomic per converged group of lanes.  kGrouped: the
// lanes may append to different counters (the batch passes, where a warp's lanes can
// hold paths of several scenes): one atomic per group of lanes sharing a counter.
template <bool kGrouped = false>
__device__ __forceinline__ unsigned long long warp_append(unsigned long long* counter) {
    unsigned m = __activemask();
    if (kGrouped) m = __match_any_sync(m, (unsigned long long)counter);
    int lane = threadIdx.x & 31;
    int leader = __ffs(m) - 1;
    unsigned lower = m & ((1u << lane) - 1u);
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(m));
    base = __shfl_sync(m, base, leader);
    return base + __popc(lower);
}

// Persistent light pass with path regeneration: each loop iteration advances every
// live path by one bounce; lanes whose path ended fetch the next unstarted light path
// (one atomic per warp), so a warp's lanes stay busy until the pool is empty instead of
// waiting for the warp's longest path.  Photons, their order within a path and every
// random number are the same as one-thread-per-path execution (counter-based samples).
struct LightPath {
    F3 o, d, tp;
    float dVM;
    int diffuse, last, len;
    int channel;      // dispersion channel, -1 until a dispersive material is met
    long long idx;
    PathRng rng;
};

// Emission: the light's own direction sampling, or the learned proposal's direction
// with throughput factor p_light / q (0 when the direction leaves no emission).
__device__ __forceinline__ bool light_path_start(const VMParams& P, long long pidx, LightPath& s) {
    s.idx = pidx;
    s.rng.init(P.seed, (uint64_t)pidx, P.iteration, STREAM_LIGHT);
    U4 b0 = s.rng.block(0), b1 = s.rng.block(1);
    const LightSample ls = light_position(P.lights, u01(b0.a), u01(b0.b), u01(b0.c));
    s.o = ls.o;
    if (P.proposal) {
        const float4 pr = __ldg(&P.proposal[pidx]);
        if (!(pr.w > 0.0f)) return false;
        s.d = f3(pr.x, pr.y, pr.z);
        s.tp = ls.tp * pr.w;
    } else {
        s.d = light_direction(P.lights.lights[ls.idx], u01(b0.d), u01(b1.a));
        s.tp = ls.tp;
    }
    s.diffuse = 0;
    s.last = EV_DIFFUSE;
    s.dVM = 0.0f;
    s.len = 0;
    s.channel = -1;
    return true;
}

// One bounce of Vertex_Merging::trace_light_path (src/Vertex_Merging.cpp:140-194), in
// two halves: the closest hit of the path's next segment (false: the path ends), then
// the shading at that hit - photon store, BSDF sample, Russian roulette, dVM update -
// which returns false when the path ends.  The persistent pass runs both per bounce,
// the staged pass searches for a whole warp at a time (search_run).  ro: the ray's origin.
template <bool kGrouped = false>
__device__ __forceinline__ bool light_path_shade(const VMParams& P, const PhotonBuf& ph, LightPath& s,
                                                 const HitRec& h, F3 ro) {
    Isect is;
    fill_isect(P.scene, h, ro, s.d, is);
    if ((unsigned)is.material >= (unsigned)P.num_materials) { atomicOr(P.error + ERR_MATERIAL, 1); return false; }
    const DevMaterial& mat = P.materials[is.material];
    const float shift = mat.disp > 0.0f
        ? dispersion_shift(mat, s.channel, s.tp, u01(s.rng.block(kChannelBlock + s.len).a)) : 0.0f;
    Bsdf b;
    b.init(mat, is.ns, is.dir, false, shift);
    if (!b.valid()) return false;
    s.dVM /= fabsf(b.cos_theta_in());
    bool stored = false;
    if (!b.is_delta() && (s.last & EV_GLOSSY)) {
        unsigned long long slot = warp_append<kGrouped>(ph.count);
        if (slot < (unsigned long long)ph.capacity) {
            ph.pos[slot] = make_float4(is.pos.x, is.pos.y, is.pos.z, s.dVM);
            ph.dir[slot] = make_float4(-is.dir.x, -is.dir.y, -is.dir.z, s.tp.x);
            ph.tp[slot] = make_float2(s.tp.y, s.tp.z);
            ph.path[slot] = (uint32_t)s.idx;
        }
        stored = true;
    }
    if (s.len > P.max_path_length || s.diffuse > kMaxDiffuse) return false;
    U4 bb = s.rng.block(2 + s.len);
    BsdfSample smp = b.sample(u01(bb.a), u01(bb.b), u01(bb.c), is.ng);
    if (is_zero(smp.f)) return false;
    F3 f = smp.f;
    if (s.len > kRRDepth) {
        if (u01(bb.d) > smp.cont) return false;
        f = div_each(f, smp.cont);
    }
    s.o = is.pos;
    s.d = smp.wi;
    if (smp.event & EV_DIFFUSE) s.diffuse++;
    s.tp = s.tp * f;
    s.last = smp.event;
    if (!stored) s.dVM *= (smp.cos_out / smp.fwd) * smp.rev;
    else s.dVM = (smp.cos_out / smp.fwd) * (1.0f + smp.rev * s.dVM);
    s.len++;
    return true;
}

template <bool kGrouped = false, class Stack>
__device__ __forceinline__ bool light_path_bounce(const VMParams& P, const PhotonBuf& ph, LightPath& s,
                                                  Stack& stack) {
    const F3 ro = s.o + s.d * kRayEps;
    HitRec h;
    if (!scene_hit(P.scene, ro, s.d, kRayEps, h, P.error + ERR_STACK, stack)) return false;
    return light_path_shade<kGrouped>(P, ph, s, h, ro);
}

// Light-path order: 4D Morton key of a path's emission samples (the same Philox draws
// light_path_start reads; with the learned proposal, the area samples and the proposed
// direction), counting-sorted.
constexpr int kOrderBits = 5;                      // cells per axis: 32
constexpr int kOrderCells = 1 << (4 * kOrderBits);

__global__ void k_light_keys(const VMParams P, uint32_t* __restrict__ keys, uint32_t* __restrict__ counts) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= P.num_light_paths) return;
    PathRng g;
    g.init(P.seed, (uint64_t)i, P.iteration, STREAM_LIGHT);
    const U4 b0 = g.block(0), b1 = g.block(1);
    float u[4] = {u01(b0.b), u01(b0.c), u01(b0.d), u01(b1.a)};
    if (P.proposal_table) {
        // emission about to be drawn from the tabulated proposal (mlp_proposal, in this
        // order): area cell, mixture component sample and the first direction sample, so
        // that a warp's lanes read the same table cells and lobes
        u[2] = u01(b1.b);
        u[3] = u01(b0.d);
    } else if (P.proposal) {
        // the learned proposal gives the direction: its octahedral coordinates instead
        const float4 pr = __ldg(&P.proposal[i]);
        const float l1 = fabsf(pr.x) + fabsf(pr.y) + fabsf(pr.z);
        float ox = l1 > 0.0f ? pr.x / l1 : 0.0f, oy = l1 > 0.0f ? pr.y / l1 : 0.0f;
        if (pr.z < 0.0f) {
            const float tx = (1.0f - fabsf(oy)) * (ox < 0.0f ? -1.0f : 1.0f);
            oy = (1.0f - fabsf(ox)) * (oy < 0.0f ? -1.0f : 1.0f);
            ox = tx;
        }
        u[2] = 0.5f * (ox + 1.0f);
        u[3] = 0.5f * (oy + 1.0f);
    }
    uint32_t key = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t c = min((uint32_t)(u[k] * (float)(1 << kOrderBits)), (uint32_t)((1 << kOrderBits) - 1));
#pragma unroll
        for (int bit = 0; bit < kOrderBits; ++bit) key |= ((c >> bit) & 1u) << (4 * bit + k);
    }
    keys[i] = key;
    atomicAdd(&counts[key], 1u);
}

__global__ void k_light_scatter(const uint32_t* __restrict__ keys, long long n, uint32_t* __restrict__ cursor,
                                uint32_t* __restrict__ order) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    order[atomicAdd(&cursor[keys[i]], 1u)] = (uint32_t)i;
}

constexpr int kRefillLanes = 24;
__device__ __forceinline__ int refill_lanes(int lanes) { return (kRefillLanes * lanes + 31) / 32; }

// kMinBlocks caps the registers per thread (resident blocks per SM the allocation must
// allow); traversal stacks are per-traversal local-memory arrays.
template <int kBlock, int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_light_pass_persistent(const VMParams P, PhotonBuf ph, int lanes,
                                                                               unsigned long long* __restrict__ next_path,
                                                                               unsigned long long* __restrict__ rays) {
    CallStack stk;
    const int lane = threadIdx.x & 31;
    LightPath s;
    bool alive = false;
    bool pool_left = true;
    unsigned traced = 0;      // closest-hit queries of this lane (one per bounce)
    const int refill = refill_lanes(lanes);
    while (true) {
        // refill lanes without a path, once at least kRefillLanes are free (or none has
        // a path): lanes refilled together take consecutive, coherent paths (the order
        // sorts paths by their emission samples), so a warp keeps groups of coherent
        // paths together for several bounces (measured on the water pool: refilling at
        // any free lane 14.2 ms, at 16 free 13.6, at 20-24 free 13.4, at 32 free 14.5;
        // with the children tested at the parent, per iteration at 20 / 24 / 28 / 32
        // free: 20.49 / 20.48 / 20.82 / 21.13 ms)
        const unsigned need = __ballot_sync(0xffffffffu, !alive && lane < lanes);
        if (pool_left && __popc(need) >= refill) {
            unsigned long long base = 0;
            if (lane == __ffs(need) - 1) base = atomicAdd(next_path, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, __ffs(need) - 1);
            if (!alive && lane < lanes) {
                const unsigned long long mine = base + __popc(need & ((1u << lane) - 1u));
                if (mine < (unsigned long long)P.num_light_paths)
                    alive = light_path_start(P, P.path_order ? (long long)__ldg(&P.path_order[mine]) : (long long)mine,
                                             s);
            }
            if (base + __popc(need) >= (unsigned long long)P.num_light_paths) pool_left = false;
        }
        if (!__any_sync(0xffffffffu, alive)) break;
        if (alive) { alive = light_path_bounce(P, ph, s, stk); ++traced; }
    }
    const unsigned w = __reduce_add_sync(0xffffffffu, traced);
    if (rays && lane == 0) atomicAdd(rays, (unsigned long long)w);
}

// Persistent camera pass with path regeneration (same scheme as the light pass).
struct CameraPath {
    F3 o, d, tp;
    float dVM;
    int len;
    int channel;      // dispersion channel, -1 until a dispersive material is met
    int target;       // pixel the path adds to: the one its jittered sample falls in
    uint32_t pix;     // the path's index
    int step;         // 1: the sample falls one column on, 2: one row on
    PathRng rng;
};

__device__ __forceinline__ int camera_target(const VMParams& P, int X, int row) {
    return (int)((long long)X + (long long)(P.camera.height - row) * P.camera.width);
}

// Generate_camera_sample + Image_Buffer::add_color's row mapping; false when the
// sample falls outside the image buffer (camera row 0, src/Image_Buffer.h:28-31).
__device__ __forceinline__ bool camera_path_start(const VMParams& P, long long pix, CameraPath& s) {
    const int W = P.camera.width, H = P.camera.height;
    s.rng.init(P.camera_seed, (uint64_t)pix, P.iteration, STREAM_CAMERA);
    U4 b1 = s.rng.block(1);
    const float x = (float)(int)(pix % W);
    const float y = (float)(int)(pix / W);
    const float sx = x + u01(b1.b), sy = y + u01(b1.c);
    if (sx < 0 || sx >= (float)W || sy < 0 || sy >= (float)H) return false;
    const int X = (int)sx, Y = H - (int)sy;
    const long long target = (long long)X + (long long)Y * W;
    if (target > (long long)W * H - 1) return false;
    F3 dir = ld3(P.camera.bottom_left) + ld3(P.camera.horizontal) * (sx / (float)W) +
             ld3(P.camera.vertical) * (sy / (float)H);
    dir = dir - ld3(P.camera.origin);
    s.o = ld3(P.camera.origin);
    s.d = normalize(dir);
    s.tp = f3(1.0f);
    s.dVM = 0.0f;
    s.len = 0;
    s.channel = -1;
    s.target = (int)target;
    s.pix = (uint32_t)pix;
    s.step = (X != (int)x ? 1 : 0) | ((int)sy != (int)y ? 2 : 0);
    return true;
}

template <bool kGrouped = false>
__device__ __forceinline__ bool camera_path_shade(const VMParams& P, const QueryBuf& qb, CameraPath& s,
                                                  const HitRec& h, F3 ro) {
    Isect is;
    fill_isect(P.scene, h, ro, s.d, is);
    if ((unsigned)is.material >= (unsigned)P.num_materials) { atomicOr(P.error + ERR_MATERIAL, 1); return false; }
    const DevMaterial& mat = P.materials[is.material];
    const float shift = mat.disp > 0.0f
        ? dispersion_shift(mat, s.channel, s.tp, u01(s.rng.block(kChannelBlock + s.len).a)) : 0.0f;
    Bsdf b;
    b.init(mat, is.ns, is.dir, true, shift);
    if (!b.valid()) return false;
    s.dVM /= fabsf(b.cos_theta_in());
    if (!b.is_delta()) {
        unsigned long long slot = warp_append<kGrouped>(qb.count);
        if (slot < (unsigned long long)qb.capacity) {
            F3 w = s.tp * P.vm_norm;
            qb.q0[slot] = make_float4(is.pos.x, is.pos.y, is.pos.z, s.dVM);
            qb.q1[slot] = make_float4(is.ns.x, is.ns.y, is.ns.z, __int_as_float(is.material));
            qb.q2[slot] = make_float4(is.ng.x, is.ng.y, is.ng.z, __int_as_float(s.target));
            qb.q3[slot] = make_float4(w.x, w.y, w.z, 0.0f);
            qb.q4[slot] = make_float4(is.dir.x, is.dir.y, is.dir.z, __int_as_float(s.channel));
        }
    }
    if (s.len > P.max_path_length) return false;
    U4 bb = s.rng.block(2 + s.len);
    BsdfSample smp = b.sample(u01(bb.a), u01(bb.b), u01(bb.c), is.ng);
    if (is_zero(smp.f)) return false;
    F3 f = smp.f;
    if (s.len > kRRDepth) {
        if (u01(bb.d) > smp.cont) return false;
        f = div_each(f, smp.cont);
    }
    s.o = is.pos;
    s.d = smp.wi;
    s.tp = s.tp * f;
    if (smp.event & EV_SPECULAR) s.dVM *= (smp.cos_out / smp.fwd) * smp.rev;
    else s.dVM = (smp.cos_out / smp.fwd) * (1.0f + smp.rev * s.dVM);
    s.len++;
    return true;
}

template <bool kGrouped = false, class Stack>
__device__ __forceinline__ bool camera_path_bounce(const VMParams& P, const QueryBuf& qb, CameraPath& s,
                                                   Stack& stack) {
    const F3 ro = s.o + s.d * kRayEps;
    HitRec h;
    if (!scene_hit(P.scene, ro, s.d, kRayEps, h, P.error + ERR_STACK, stack)) return false;
    return camera_path_shade<kGrouped>(P, qb, s, h, ro);
}

template <int kBlock, int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_camera_pass_persistent(const VMParams P, QueryBuf qb, int lanes,
                                                                                unsigned long long* __restrict__ next_pixel) {
    CallStack stk;
    const int lane = threadIdx.x & 31;
    const long long npix = (long long)P.camera.width * P.camera.height;
    CameraPath s;
    bool alive = false;
    bool pool_left = true;
    const int refill = refill_lanes(lanes);
    while (true) {
        // refill as in the light pass: once kRefillLanes lanes are free (2.43 -> 2.35 ms on
        // the water pool), drawing again for samples that fall outside the buffer
        unsigned need = __ballot_sync(0xffffffffu, !alive && lane < lanes);
        while (pool_left && __popc(need) >= refill) {
            unsigned long long base = 0;
            if (lane == __ffs(need) - 1) base = atomicAdd(next_pixel, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, __ffs(need) - 1);
            if (!alive && lane < lanes) {
                const unsigned long long mine = base + __popc(need & ((1u << lane) - 1u));
                if (mine < (unsigned long long)npix) alive = camera_path_start(P, (long long)mine, s);
            }
            if (base + __popc(need) >= (unsigned long long)npix) pool_left = false;
            need = __ballot_sync(0xffffffffu, !alive && lane < lanes);   // samples outside the buffer: draw again
        }
        if (!__any_sync(0xffffffffu, alive)) break;
        if (alive) alive = camera_path_bounce(P, qb, s, stk);
    }
}

// Batch passes: the persistent light and camera passes over the paths (pixels) of
// several resident scenes in one launch.  Work index g runs over the scenes' paths laid
// end to end (prefix[i] = first index of scene i, prefix[n] = total); a lane that takes
// index g finds its scene by binary search and runs that scene's path with the scene's
// own parameters and buffers (read from global memory: every lane of a warp that holds
// paths of one scene reads the same words).  Each path's samples, bounces and photons
// are those of the scene's own pass.
__device__ __forceinline__ int batch_scene_of(const long long* __restrict__ prefix, int n, long long g) {
    int lo = 0, hi = n - 1;   // the last scene whose range starts at or before g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&prefix[mid]) <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int kBlock, int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_light_pass_batch(const BatchScene* __restrict__ B,
                                                                         const long long* __restrict__ prefix, int n,
                                                                         unsigned long long* __restrict__ next_path) {
    CallStack stk;
    const int lane = threadIdx.x & 31;
    const unsigned long long total = (unsigned long long)__ldg(&prefix[n]);
    LightPath s;
    int sid = 0;
    bool alive = false;
    bool pool_left = true;
    while (true) {
        const unsigned need = __ballot_sync(0xffffffffu, !alive);
        if (need && pool_left && (__popc(need) >= kRefillLanes || need == 0xffffffffu)) {
            unsigned long long base = 0;
            if (lane == __ffs(need) - 1) base = atomicAdd(next_path, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, __ffs(need) - 1);
            if (!alive) {
                const unsigned long long mine = base + __popc(need & ((1u << lane) - 1u));
                if (mine < total) {
                    sid = batch_scene_of(prefix, n, (long long)mine);
                    const VMParams& P = B[sid].p;
                    const long long local = (long long)mine - __ldg(&prefix[sid]);
                    alive = light_path_start(P, P.path_order ? (long long)__ldg(&P.path_order[local]) : local, s);
                }
            }
            if (base + __popc(need) >= total) pool_left = false;
        }
        if (!__any_sync(0xffffffffu, alive)) break;
        if (alive) alive = light_path_bounce<true>(B[sid].p, B[sid].ph, s, stk);
    }
}

template <int kBlock, int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_camera_pass_batch(const BatchScene* __restrict__ B,
                                                                          const long long* __restrict__ prefix, int n,
                                                                          unsigned long long* __restrict__ next_pixel) {
    CallStack stk;
    const int lane = threadIdx.x & 31;
    const unsigned long long total = (unsigned long long)__ldg(&prefix[n]);
    CameraPath s;
    int sid = 0;
    bool alive = false;
    bool pool_left = true;
    while (true) {
        unsigned need = __ballot_sync(0xffffffffu, !alive);
        while (need && pool_left && (__popc(need) >= kRefillLanes || need == 0xffffffffu)) {
            unsigned long long base = 0;
            if (lane == __ffs(need) - 1) base = atomicAdd(next_pixel, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, __ffs(need) - 1);
            if (!alive) {
                const unsigned long long mine = base + __popc(need & ((1u << lane) - 1u));
                if (mine < total) {
                    sid = batch_scene_of(prefix, n, (long long)mine);
                    alive = camera_path_start(B[sid].p, (long long)mine - __ldg(&prefix[sid]), s);
                }
            }
            if (base + __popc(need) >= total) pool_left = false;
            need = __ballot_sync(0xffffffffu, !alive);
        }
        if (!__any_sync(0xffffffffu, alive)) break;
        if (alive) alive = camera_path_bounce<true>(B[sid].p, B[sid].qb, s, stk);
    }
}

// Staged passes: a pass in two launches.  k_pass_first takes fresh paths, 32 at a time per
// warp, through their first kSegs segments, all lanes together: they start coherent (the
// light-path order; the pixels of a row), and mixing them with paths further on costs more
// than the idle lanes do.  The paths that go on are parked, packed (48 bytes each).
// k_pass_rest takes the parked paths to their ends; these are incoherent, so lanes shade as
// soon as at most kKeep lanes of the warp still search, and ended paths are replaced once
// kFree lanes are free.  Paths, samples and stored records are the persistent passes'.
//
// What bounds the passes is the instruction issue of the closest-hit search (repeating the
// search doubles k_pass_first's time); a step of 32 lanes at different places of the tree
// had 9 to 10 of them active.  With the search by phases (search_run) k_pass_first has 21,
// k_pass_rest 13 (960x540 water pool, 4.2M paths).  Measured
// against the best persistent shape: light pass of the 1080p water pool (16.7M paths)
// 11.3 -> 9.6 ms, of 2,000 gems (4.2M paths) 35.9 -> 21.1 ms.  Tried and lost: one
// kernel that holds the continuing paths back per warp in global memory and switches
// between the two modes (11.4 ms on the pool); the state a search needs rarely in shared
// memory (9.7 ms); four-wide nodes with 8-bit child boxes, conservative with an exact test
// per leaf (10.2 ms; 17.7 ms on the gems).
// Small passes end with a few long paths whatever the order; there the persistent shapes
// stay ahead (518,400 paths: 0.59 against 0.79 ms), and the autotuner keeps one of them.
struct Parked {
    float4* a;   // origin | dVM
    float4* b;   // direction | throughput.r
    float4* c;   // throughput.gb | path index | meta, scene << 16
    unsigned long long* count;   // [0] parked paths, [1], [2] next path of the two launches
};
constexpr long long kParkChunk = 1LL << 24;   // paths per pair of launches (800 MB parked at most)

struct LightKind {
    using Path = LightPath;
    using Out = PhotonBuf;
    static __device__ __forceinline__ bool start(const VMParams& P, uint32_t i, Path& s) {
        return light_path_start(P, P.path_order ? (long long)__ldg(&P.path_order[i]) : (long long)i, s);
    }
    static __device__ __forceinline__ uint32_t index(const Path& s) { return (uint32_t)s.idx; }
    static __device__ __forceinline__ uint32_t meta(const Path& s) {
        return (uint32_t)s.last | ((uint32_t)s.len << 5) | ((uint32_t)s.diffuse << 11) | ((uint32_t)(s.channel + 1) << 14);
    }
    static __device__ __forceinline__ void restore(const VMParams& P, uint32_t idx, uint32_t m, Path& s) {
        s.idx = (long long)idx;
        s.last = (int)(m & 31u);
        s.len = (int)((m >> 5) & 63u);
        s.diffuse = (int)((m >> 11) & 7u);
        s.channel = (int)((m >> 14) & 3u) - 1;
        s.rng.init(P.seed, (uint64_t)idx, P.iteration, STREAM_LIGHT);
    }
    template <bool kGrouped>
    static __device__ __forceinline__ bool shade(const VMParams& P, const Out& out, Path& s, const HitRec& h, F3 ro) {
        return light_path_shade<kGrouped>(P, out, s, h, ro);
    }
};
static_assert(2 * EV_SPECULAR - 1 == 31 && kMaxDiffuse + 1 <= 7, "LightKind::meta's fields");

struct CameraKind {
    using Path = CameraPath;
    using Out = QueryBuf;
    static __device__ __forceinline__ bool start(const VMParams& P, uint32_t i, Path& s) {
        return camera_path_start(P, (long long)i, s);
    }
    static __device__ __forceinline__ uint32_t index(const Path& s) { return s.pix; }
    static __device__ __forceinline__ uint32_t meta(const Path& s) {
        return (uint32_t)s.len | ((uint32_t)(s.channel + 1) << 6) | ((uint32_t)s.step << 8);
    }
    static __device__ __forceinline__ void restore(const VMParams& P, uint32_t idx, uint32_t m, Path& s) {
        s.pix = idx;
        s.len = (int)(m & 63u);
        s.channel = (int)((m >> 6) & 3u) - 1;
        s.step = (int)((m >> 8) & 3u);
        const int W = P.camera.width, y = (int)idx / W, x = (int)idx - y * W;
        s.target = camera_target(P, x + (s.step & 1), y + (s.step >> 1));
        s.rng.init(P.camera_seed, (uint64_t)idx, P.iteration, STREAM_CAMERA);
    }
    template <bool kGrouped>
    static __device__ __forceinline__ bool shade(const VMParams& P, const Out& out, Path& s, const HitRec& h, F3 ro) {
        return camera_path_shade<kGrouped>(P, out, s, h, ro);
    }
};

// The scenes of a pass: one, its parameters in the kernel's, or the batch's.  Work indices
// run from first to first + count.
template <class Kind> struct OneScene {
    static constexpr bool kMany = false;
    VMParams p;
    typename Kind::Out out;
    unsigned long long first, count;
    __device__ __forceinline__ const VMParams& params(int) const { return p; }
    __device__ __forceinline__ const typename Kind::Out& buffers(int) const { return out; }
    __device__ __forceinline__ int locate(unsigned long long g, uint32_t& local) const {
        local = (uint32_t)g;
        return 0;
    }
};
__device__ __forceinline__ const PhotonBuf& batch_buffers(const BatchScene& b, const LightKind*) { return b.ph; }
__device__ __forceinline__ const QueryBuf& batch_buffers(const BatchScene& b, const CameraKind*) { return b.qb; }
template <class Kind> struct ManyScenes {
    static constexpr bool kMany = true;
    const BatchScene* b;
    const long long* prefix;
    int n;
    unsigned long long first, count;
    __device__ __forceinline__ const VMParams& params(int sid) const { return b[sid].p; }
    __device__ __forceinline__ const typename Kind::Out& buffers(int sid) const {
        return batch_buffers(b[sid], (const Kind*)nullptr);
    }
    __device__ __forceinline__ int locate(unsigned long long g, uint32_t& local) const {
        const int sid = batch_scene_of(prefix, n, (long long)g);
        local = (uint32_t)((long long)g - __ldg(&prefix[sid]));
        return sid;
    }
};

template <class Kind, class Scenes, int kMinBlocks, int kSegs>
__global__ void __launch_bounds__(128, kMinBlocks) k_pass_first(const Scenes S, const Parked park,
                                                                unsigned long long* __restrict__ rays) {
    SearchStack st;
    Search q;
    const int lane = threadIdx.x & 31;
    unsigned traced = 0;   // closest-hit queries of this lane
    while (true) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(park.count + 1, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= S.count) break;
        typename Kind::Path s;
        bool alive = false;
        int sid = 0;
        if (base + lane < S.count) {
            uint32_t local;
            sid = S.locate(S.first + base + lane, local);
            alive = Kind::start(S.params(sid), local, s);
        }
        const VMParams& P = S.params(sid);
#pragma unroll 1
        for (int k = 0; k < kSegs; ++k) {
            q.w0 = kSearchIdle;
            if (alive) {
                search_begin(q, st, s.o + s.d * kRayEps, s.d);
                ++traced;
            }
            __syncwarp();
            search_run(P.scene, q, st, s.d, kRayEps, 0, P.error + ERR_STACK);
            if (alive)
                alive = q.out.slot >= 0 && Kind::template shade<Scenes::kMany>(P, S.buffers(sid), s, q.out, q.origin());
            __syncwarp();
        }
        if (alive) {
            const unsigned long long j = warp_append(park.count);
            park.a[j] = make_float4(s.o.x, s.o.y, s.o.z, s.dVM);
            park.b[j] = make_float4(s.d.x, s.d.y, s.d.z, s.tp.x);
            park.c[j] = make_float4(s.tp.y, s.tp.z, __uint_as_float(Kind::index(s)),
                                    __uint_as_float(Kind::meta(s) | ((uint32_t)sid << 16)));
        }
        __syncwarp();
    }
    const unsigned w = __reduce_add_sync(0xffffffffu, traced);
    if (rays && lane == 0) atomicAdd(rays, (unsigned long long)w);
}

template <class Kind, class Scenes, int kMinBlocks, int kKeep, int kFree>
__global__ void __launch_bounds__(128, kMinBlocks) k_pass_rest(const Scenes S, const Parked park,
                                                               unsigned long long* __restrict__ rays) {
    SearchStack st;
    Search q;
    q.w0 = kSearchIdle;
    const int lane = threadIdx.x & 31;
    const unsigned long long total = park.count[0];
    typename Kind::Path s;
    int sid = 0;
    bool alive = false, left = true;
    unsigned traced = 0;
    while (true) {
        const unsigned need = __ballot_sync(0xffffffffu, !alive);
        if (left && (__popc(need) >= kFree || need == 0xffffffffu)) {
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(park.count + 2, (unsigned long long)__popc(need));
            base = __shfl_sync(0xffffffffu, base, leader);
            const unsigned long long mine = base + __popc(need & ((1u << lane) - 1u));
            if (!alive && mine < total) {
                const float4 a = park.a[mine], b = park.b[mine], c = park.c[mine];
                const uint32_t m = __float_as_uint(c.w);
                sid = Scenes::kMany ? (int)(m >> 16) : 0;
                s.o = f3(a.x, a.y, a.z); s.dVM = a.w;
                s.d = f3(b.x, b.y, b.z); s.tp = f3(b.w, c.x, c.y);
                Kind::restore(S.params(sid), __float_as_uint(c.z), m & 0xffffu, s);
                alive = true;
            }
            if (base + __popc(need) >= total) left = false;
        }
        const int n = __popc(__ballot_sync(0xffffffffu, alive));
        if (n == 0) {
            if (!left) break;
            continue;
        }
        if (alive && q.w0 == kSearchIdle) {
            search_begin(q, st, s.o + s.d * kRayEps, s.d);
            ++traced;
        }
        __syncwarp();
        const VMParams& P = S.params(sid);
        search_run(P.scene, q, st, s.d, kRayEps, min(kKeep, n - 1), P.error + ERR_STACK);
        if (alive && q.w0 == kSearchIdle)
            alive = q.out.slot >= 0 && Kind::template shade<Scenes::kMany>(P, S.buffers(sid), s, q.out, q.origin());
        __syncwarp();
    }
    const unsigned w = __reduce_add_sync(0xffffffffu, traced);
    if (rays && lane == 0) atomicAdd(rays, (unsigned long long)w);
}

// Closest hits of given rays by the staged passes' search.
__global__ void __launch_bounds__(128) k_trace_search(const SceneView S, int n, const float* __restrict__ o,
                                                      const float* __restrict__ d, float tmin,
                                                      HitRec* __restrict__ hits, int* err) {
    SearchStack st;
    Search q;
    q.w0 = kSearchIdle;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    F3 rd = f3(0.0f);
    if (i < n) {
        rd = f3(d[3 * i], d[3 * i + 1], d[3 * i + 2]);
        search_begin(q, st, f3(o[3 * i], o[3 * i + 1], o[3 * i + 2]), rd);
    }
    __syncwarp();
    search_run(S, q, st, rd, tmin, 0, err);
    if (i < n) hits[i] = q.out;
}

// The hit records of given rays: `found` (k_trace_search), or searched here with Stack:
// CallStack (the persistent passes' traversal: children tested at the parent) or
// LocalStack (pop-and-test, the reference's own form).
template <class Stack>
__global__ void k_trace_rays(const SceneView S, int n, const float* __restrict__ o, const float* __restrict__ d,
                             float tmin, const HitRec* __restrict__ found, float* out_full, unsigned* out_words,
                             int* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    F3 ro = f3(o[3 * i], o[3 * i + 1], o[3 * i + 2]);
    F3 rd = f3(d[3 * i], d[3 * i + 1], d[3 * i + 2]);
    HitRec h;
    bool hit;
    if (found) {
        h = found[i];
        hit = h.slot >= 0;
    } else {
        Stack stk;
        hit = scene_hit(S, ro, rd, tmin, h, err, stk);
    }
    Isect is;
    if (hit) fill_isect(S, h, ro, rd, is);
    if (out_words) {
        unsigned* w = out_words + 8 * i;
        w[0] = hit ? 1u : 0u;
        w[1] = __float_as_uint(h.t);
        w[2] = __float_as_uint(h.u);
        w[3] = __float_as_uint(h.v);
        w[4] = hit ? (unsigned)is.tri : 0xffffffffu;
        w[5] = hit ? (unsigned)is.material : 0xffffffffu;
        w[6] = hit ? (unsigned)is.mesh : 0xffffffffu;
        w[7] = 0u;
    }
    if (out_full) {
        float* f = out_full + 16 * i;
        f[0] = hit ? 1.0f : 0.0f;
        f[1] = h.t; f[2] = h.u; f[3] = h.v;
        if (hit) {
            f[4] = is.ng.x; f[5] = is.ng.y; f[6] = is.ng.z;
            f[7] = is.ns.x; f[8] = is.ns.y; f[9] = is.ns.z;
            f[10] = is.pos.x; f[11] = is.pos.y; f[12] = is.pos.z;
            f[13] = is.front ? 1.0f : 0.0f;
            f[14] = (float)is.material;
            f[15] = __int_as_float(is.tri);
        } else {
            for (int k = 4; k < 16; ++k) f[k] = 0.0f;
            f[14] = -1.0f;
            f[15] = __int_as_float(-1);
        }
    }
}

// Persistent grid for one shape: resident blocks per SM (occupancy with its dynamic
// shared memory) x SMs, capped by the work.
template <class K>
unsigned persistent_grid(K kernel, int block, size_t smem, long long work_items) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
    const long long blocks = (long long)sms * (per_sm > 0 ? per_sm : 1);
    const long long need = (work_items + block - 1) / block;
    return (unsigned)(need < blocks ? need : blocks);
}

// Paths that a warp of the persistent passes holds.  A pass too small to give 12 warps per
// SM 32 paths each is spread over the warps of the whole GPU: its time is then the longest
// warp, and a warp of few paths executes fewer of the others' steps (sphere of 5k triangles,
// light / camera pass in us: 6,144 paths 248 / 237 with 32 lanes, 191 / 163 with 4; 19,200:
// 261 / 274 with 32, 193 / 223 with 8; 49,152: 306 / 299 with 32, 265 / 256 with 16).  12 warps
// leave room for the other pass beside it: an update of 6,144 paths and pixels takes 566 us
// with 32 lanes, 502 / 495 / 497 / 500 / 515 with 8 / 12 / 16 / 24 / 32 warps per SM.
int path_lanes(long long n) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long warps = 12LL * std::max(sms, 1);
    return (int)std::min(std::max((n + warps / 2) / warps, 1LL), 32LL);
}

template <int B, int MB>
void launch_light_t(const VMParams& p, PhotonBuf ph, unsigned long long* next_path, unsigned long long* rays,
                    cudaStream_t s) {
    // per host thread: contexts on different threads launch concurrently
    static thread_local unsigned grid_cache = 0;
    static thread_local long long grid_for = -1;
    static thread_local int lanes = 32;
    if (grid_for != p.num_light_paths) {
        lanes = path_lanes(p.num_light_paths);
        grid_cache = persistent_grid(k_light_pass_persistent<B, MB>, B, 0, p.num_light_paths * 32 / lanes);
        grid_for = p.num_light_paths;
    }
    cudaMemsetAsync(next_path, 0, sizeof(unsigned long long), s);
    if (rays) cudaMemsetAsync(rays, 0, sizeof(unsigned long long), s);
    k_light_pass_persistent<B, MB><<<grid_cache, B, 0, s>>>(p, ph, lanes, next_path, rays);
}

template <int B, int MB>
void launch_camera_t(const VMParams& p, QueryBuf qb, unsigned long long* next_pixel, cudaStream_t s) {
    const long long n = (long long)p.camera.width * p.camera.height;
    // per host thread: contexts on different threads launch concurrently
    static thread_local unsigned grid_cache = 0;
    static thread_local long long grid_for = -1;
    static thread_local int lanes = 32;
    if (grid_for != n) {
        lanes = path_lanes(n);
        grid_cache = persistent_grid(k_camera_pass_persistent<B, MB>, B, 0, n * 32 / lanes);
        grid_for = n;
    }
    cudaMemsetAsync(next_pixel, 0, sizeof(unsigned long long), s);
    k_camera_pass_persistent<B, MB><<<grid_cache, B, 0, s>>>(p, qb, lanes, next_pixel);
}

template <int B, int MB>
void launch_light_batch_t(const BatchScene* scenes, const long long* prefix, int n, long long total,
                          unsigned long long* next, cudaStream_t s) {
    static thread_local unsigned grid_cache = 0;
    static thread_local long long grid_for = -1;
    if (grid_for != total) {
        grid_cache = persistent_grid(k_light_pass_batch<B, MB>, B, 0, total);
        grid_for = total;
    }
    cudaMemsetAsync(next, 0, sizeof(unsigned long long), s);
    k_light_pass_batch<B, MB><<<grid_cache, B, 0, s>>>(scenes, prefix, n, next);
}

template <int B, int MB>
void launch_camera_batch_t(const BatchScene* scenes, const long long* prefix, int n, long long total,
                           unsigned long long* next, cudaStream_t s) {
    static thread_local unsigned grid_cache = 0;
    static thread_local long long grid_for = -1;
    if (grid_for != total) {
        grid_cache = persistent_grid(k_camera_pass_batch<B, MB>, B, 0, total);
        grid_for = total;
    }
    cudaMemsetAsync(next, 0, sizeof(unsigned long long), s);
    k_camera_pass_batch<B, MB><<<grid_cache, B, 0, s>>>(scenes, prefix, n, next);
}

}  // namespace

size_t light_order_scratch_bytes(long long n) {
    return 4 * (size_t)(n > 0 ? n : 1) + 4 * (size_t)kOrderCells + 4 * scan_scratch_words(kOrderCells) + 512;
}

bool light_order_pays(long long n) { return path_lanes(n) >= 32; }

void launch_light_order(const VMParams& p, void* scratch, uint32_t* order, cudaStream_t s) {
    const long long n = p.num_light_paths;
    if (n <= 0) return;
    uint32_t* keys = static_cast<uint32_t*>(scratch);
    uint32_t* counts = keys + ((n + 63) & ~63LL);
    cudaMemsetAsync(counts, 0, 4 * (size_t)kOrderCells, s);
    const unsigned g = (unsigned)((n + 255) / 256);
    k_light_keys<<<g, 256, 0, s>>>(p, keys, counts);
    launch_scan_counts(counts, kOrderCells, counts + kOrderCells, s);
    k_light_scatter<<<g, 256, 0, s>>>(keys, n, counts, order);
}

int pass_variants() { return 7; }
bool pass_is_staged(int v) { return v >= 4 && v < 7; }
size_t pass_park_bytes(long long n) { return 48 * (size_t)std::min(std::max(n, 1LL), kParkChunk) + 256; }

const char* pass_variant_name(int v) {
    static const char* names[7] = {"256 threads, >= 3 blocks/SM (<= 85 registers)",
                                   "128 threads, >= 7 blocks/SM (<= 73 registers)",
                                   "128 threads, >= 8 blocks/SM (<= 64 registers)",
                                   "128 threads, >= 9 blocks/SM (<= 56 registers)",
                                   "staged: 2 segments, then 8 lanes kept, 8 freed",
                                   "staged: 2 segments, then 12 lanes kept, 4 freed",
                                   "staged: 1 segment, then 12 lanes kept, 4 freed"};
    return (v >= 0 && v < 7) ? names[v] : "?";
}

namespace {

template <class Kind, int kSegs, int kMinFirst, int kMinRest, int kKeep, int kFree, class Scenes>
void launch_staged(Scenes S, long long n, long long most, void* scratch, unsigned long long* rays, cudaStream_t s) {
    const long long chunk = std::min(n, most);
    float4* const m = static_cast<float4*>(scratch);
    const Parked park{m, m + chunk, m + 2 * chunk, reinterpret_cast<unsigned long long*>(m + 3 * chunk)};
    auto* const first = k_pass_first<Kind, Scenes, kMinFirst, kSegs>;
    auto* const rest = k_pass_rest<Kind, Scenes, kMinRest, kKeep, kFree>;
    // per host thread: contexts on different threads launch concurrently
    static thread_local unsigned full_first = 0, full_rest = 0;
    if (!full_first) {
        full_first = persistent_grid(first, 128, 0, 1LL << 40);
        full_rest = persistent_grid(rest, 128, 0, 1LL << 40);
    }
    if (rays) cudaMemsetAsync(rays, 0, sizeof(unsigned long long), s);
    for (long long lo = 0; lo < n; lo += chunk) {
        const long long c = std::min(chunk, n - lo);
        const unsigned need = (unsigned)((c + 127) / 128);
        S.first = (unsigned long long)lo;
        S.count = (unsigned long long)c;
        cudaMemsetAsync(park.count, 0, 3 * sizeof(unsigned long long), s);
        first<<<std::min(need, full_first), 128, 0, s>>>(S, park, rays);
        rest<<<std::min(need, full_rest), 128, 0, s>>>(S, park, rays);
    }
}

template <class Kind, class Scenes>
void launch_staged_variant(const Scenes& S, long long n, long long most, void* scratch, unsigned long long* rays,
                           cudaStream_t s, int variant) {
    if (most <= 0 || most > kParkChunk) most = kParkChunk;
    switch (variant) {
    case 5: launch_staged<Kind, 2, 9, 9, 12, 4>(S, n, most, scratch, rays, s); break;
    case 6: launch_staged<Kind, 1, 10, 8, 12, 4>(S, n, most, scratch, rays, s); break;
    default: launch_staged<Kind, 2, 8, 8, 8, 8>(S, n, most, scratch, rays, s); break;
    }
}

}  // namespace

void launch_light_pass(const VMParams& p, PhotonBuf ph, unsigned long long* next_path, cudaStream_t s, int variant,
                       unsigned long long* rays, void* park, long long chunk) {
    const long long n = p.num_light_paths;
    if (n <= 0) return;
    if (!next_path) return;
    if (pass_is_staged(variant) && park && n < (1LL << 32)) {
        launch_staged_variant<LightKind>(OneScene<LightKind>{p, ph, 0, 0}, n, chunk, park, rays, s, variant);
        return;
    }
    switch (variant) {
    case 1: launch_light_t<128, 7>(p, ph, next_path, rays, s); break;
    case 2: launch_light_t<128, 8>(p, ph, next_path, rays, s); break;
    case 3: launch_light_t<128, 9>(p, ph, next_path, rays, s); break;
    default: launch_light_t<256, 3>(p, ph, next_path, rays, s); break;
    }
}

void launch_camera_pass(const VMParams& p, QueryBuf qb, unsigned long long* next_pixel, cudaStream_t s, int variant,
                        void* park, long long chunk) {
    const long long n = (long long)p.camera.width * p.camera.height;
    if (n <= 0) return;
    if (!next_pixel) return;
    if (pass_is_staged(variant) && park && n < (1LL << 31)) {
        launch_staged_variant<CameraKind>(OneScene<CameraKind>{p, qb, 0, 0}, n, chunk, park, nullptr, s, variant);
        return;
    }
    switch (variant) {
    case 1: launch_camera_t<128, 7>(p, qb, next_pixel, s); break;
    case 2: launch_camera_t<128, 8>(p, qb, next_pixel, s); break;
    case 3: launch_camera_t<128, 9>(p, qb, next_pixel, s); break;
    default: launch_camera_t<256, 3>(p, qb, next_pixel, s); break;
    }
}

// (a parked path names its scene in 16 bits; a scene's own indices fit 32)
void launch_light_pass_batch(const BatchScene* scenes, const long long* path_prefix, int n, long long total_paths,
                             unsigned long long* next_path, cudaStream_t s, int variant, void* park, long long chunk) {
    if (n <= 0 || total_paths <= 0 || !next_path) return;
    if (pass_is_staged(variant) && park && n < (1 << 16)) {
        launch_staged_variant<LightKind>(ManyScenes<LightKind>{scenes, path_prefix, n, 0, 0}, total_paths, chunk, park,
                                         nullptr, s, variant);
        return;
    }
    switch (variant) {
    case 1: launch_light_batch_t<128, 7>(scenes, path_prefix, n, total_paths, next_path, s); break;
    case 2: launch_light_batch_t<128, 8>(scenes, path_prefix, n, total_paths, next_path, s); break;
    case 3: launch_light_batch_t<128, 9>(scenes, path_prefix, n, total_paths, next_path, s); break;
    default: launch_light_batch_t<256, 3>(scenes, path_prefix, n, total_paths, next_path, s); break;
    }
}

void launch_camera_pass_batch(const BatchScene* scenes, const long long* pixel_prefix, int n, long long total_pixels,
                              unsigned long long* next_pixel, cudaStream_t s, int variant, void* park, long long chunk) {
    if (n <= 0 || total_pixels <= 0 || !next_pixel) return;
    if (pass_is_staged(variant) && park && n < (1 << 16)) {
        launch_staged_variant<CameraKind>(ManyScenes<CameraKind>{scenes, pixel_prefix, n, 0, 0}, total_pixels, chunk, park,
                                          nullptr, s, variant);
        return;
    }
    switch (variant) {
    case 1: launch_camera_batch_t<128, 7>(scenes, pixel_prefix, n, total_pixels, next_pixel, s); break;
    case 2: launch_camera_batch_t<128, 8>(scenes, pixel_prefix, n, total_pixels, next_pixel, s); break;
    case 3: launch_camera_batch_t<128, 9>(scenes, pixel_prefix, n, total_pixels, next_pixel, s); break;
    default: launch_camera_batch_t<256, 3>(scenes, pixel_prefix, n, total_pixels, next_pixel, s); break;
    }
}

// Debug views (src/Debug_scene.cpp:21-214, dispatched by src/main.cpp:172-180): one
// unjittered primary ray per pixel corner, closest hit with tmin 1e-4 from the camera
// origin, the colour added to the pixel Image_Buffer::add_color picks (row 0 dropped).
__global__ void __launch_bounds__(256) k_debug_view(const VMParams P, int mode, float ior, double* accum) {
    const long long pix = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int W = P.camera.width, H = P.camera.height;
    if (pix >= (long long)W * H) return;
    const float x = (float)(int)(pix % W);
    const float y = (float)(int)(pix / W);
    F3 dir = ld3(P.camera.bottom_left) + ld3(P.camera.horizontal) * (x / (float)W) +
             ld3(P.camera.vertical) * (y / (float)H);
    dir = dir - ld3(P.camera.origin);
    const F3 o = ld3(P.camera.origin);
    const F3 d = normalize(dir);
    HitRec h;
    if (!scene_hit(P.scene, o, d, 0.0001f, h, P.error + ERR_STACK)) return;
    Isect is;
    fill_isect(P.scene, h, o, d, is);
    F3 c;
    if (mode == 2) {
        c = is.ns;                                            // run_debug_normals
    } else if (mode == 3) {                                   // run_debug_facing
        const F3 base = is.front ? f3(0.0f, 0.0f, 1.0f) : f3(1.0f, 0.0f, 0.0f);
        c = base * fabsf(dot(d, is.ns));
    } else {                                                  // run_debug_materials
        Frame fr;
        fr.set_from_z(is.ns);
        const F3 dl = fr.to_local(-is.dir);
        float eta = ior;
        if (dl.z > 0.0f) eta = 1.0f / ior;
        c = f3(fresnel_eta(fabsf(dl.z), eta));
    }
    const int X = (int)x, Y = H - (int)y;
    const long long target = (long long)X + (long long)Y * W;
    if (target > (long long)W * H - 1) return;
    accum[3 * target] += (double)c.x;
    accum[3 * target + 1] += (double)c.y;
    accum[3 * target + 2] += (double)c.z;
}

void launch_debug_view(const VMParams& p, int mode, float ior, double* accum, cudaStream_t s) {
    const long long n = (long long)p.camera.width * p.camera.height;
    if (n <= 0) return;
    k_debug_view<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(p, mode, ior, accum);
}

// Running FP64 sum -> FP32 mean image (Vertex_Merging::run's final scale,
// src/Vertex_Merging.cpp:367-379, done at readback).
__global__ void k_image_mean(const double* __restrict__ acc, float* __restrict__ out, long long n, double scale) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)(acc[i] * scale);
}

void launch_image_mean(const double* acc, float* out, long long n, double scale, cudaStream_t s) {
    if (n <= 0) return;
    k_image_mean<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(acc, out, n, scale);
}

__global__ void k_pad_photons(float4* __restrict__ pos, const unsigned long long* __restrict__ count, long long cap,
                              float4 pad) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= cap || (unsigned long long)i < *count) return;
    pos[i] = pad;
}

__global__ void k_check_counts(const unsigned long long* photons, long long pcap, const unsigned long long* queries,
                               long long qcap, int* flag) {
    *flag = (*photons > (unsigned long long)pcap || *queries > (unsigned long long)qcap) ? 1 : 0;
}

void launch_pad_photons(float4* pos, const unsigned long long* count, long long capacity, float4 pad, cudaStream_t s) {
    if (capacity <= 0) return;
    k_pad_photons<<<(unsigned)((capacity + 255) / 256), 256, 0, s>>>(pos, count, capacity, pad);
}

void launch_check_counts(const unsigned long long* photons, long long photon_cap, const unsigned long long* queries,
                         long long query_cap, int* flag, cudaStream_t s) {
    k_check_counts<<<1, 1, 0, s>>>(photons, photon_cap, queries, query_cap, flag);
}

void launch_trace_rays(const SceneView& sv, int n, const float* o, const float* d, float tmin, HitRec* found,
                       float* out_full, unsigned* out_words, int* err, cudaStream_t st, int shape) {
    if (n <= 0) return;
    const unsigned g = (unsigned)((n + 127) / 128);
    if (shape == 0) k_trace_search<<<g, 128, 0, st>>>(sv, n, o, d, tmin, found, err);
    if (shape == 2)
        k_trace_rays<LocalStack><<<g, 128, 0, st>>>(sv, n, o, d, tmin, nullptr, out_full, out_words, err);
    else
        k_trace_rays<CallStack><<<g, 128, 0, st>>>(sv, n, o, d, tmin, shape == 0 ? found : nullptr, out_full, out_words,
                                                   err);
}

}  // namespace rc
