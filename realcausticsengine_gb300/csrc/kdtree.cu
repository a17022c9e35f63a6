// GPU photon KD-tree build by parallel median splits (see kdtree.cuh for the tree).
//
// Levels whose nodes hold more than kSmemSeg photons are split with global passes,
// one pass per step over all photons (SoA x/y/z/id, double buffered):
//   hist x4   8-bit radix select of the rank-count/2 key along the node's axis (its box's
//             largest extent; the leading digits the box fixes are skipped)
//   partition photons below / equal / above the median key to their halves, and the halves'
//             boxes (the next level's nodes)
// Each pass first picks the previous digit: every CTA does it for its own nodes, from the
// finished histogram, and the histograms, boxes and cursors of the next level are cleared by
// the passes of this one, so a level is 5 launches, each started while the one before ends.
// At a few hundred thousand photons a pass is mostly its launch and one chain of loads: with
// the box, its axis and each digit's choice in launches of their own (12 a level) 300,001
// photons took 750 us, with 5 a level 519, started early 395 (472 without loading the
// photons before the wait).
// A CTA covers T x kItems consecutive positions (T = 256 threads on levels whose nodes
// hold more than 2048 photons, else 128); because nodes on these levels hold more
// than that many photons, a chunk meets at most two nodes (and one ancestor median
// between them), so histograms and counters stay in shared memory and only their
// totals go to global memory.
// From the first level with at most kSmemSeg photons per node, one CTA per node
// loads its photons into shared memory and finishes the whole subtree there: one
// sort along x, y and z (key, then local index), then stable splits of the three
// lists per level, writing nodes and final order.
#include "kdtree.cuh"
#include "dev_once.h"
#include "early_launch.cuh"
#include <cmath>
#include <cstdio>
#include <mutex>
#include <utility>

namespace rc {

namespace {

constexpr int kSmemSeg = 1024;      // largest node finished in shared memory (~66 KB: 3 CTAs per SM)
constexpr int kItems = 8;           // positions per thread in the global passes
constexpr int kThreads = 128;       // CTA size of the global passes (kThreads x kItems <= kSmemSeg)
constexpr int kWideThreads = 256;   // CTA size on levels whose nodes hold more than its positions
constexpr int kSmemThreads = 256;
constexpr float kSplitBias = 1.175494e-38f;   // src/KD_Tree.cpp:150

__device__ __forceinline__ uint32_t f2key(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}
// order-preserving int encoding for atomicMin/Max on floats
__device__ __forceinline__ int f2ord(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : (i ^ 0x7fffffff);
}
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : (i ^ 0x7fffffff)); }

__device__ __forceinline__ uint32_t odd_mask(int axis) { return axis == 0 ? 0x90000000u : (axis == 1 ? 0xb0000000u : 0xf0000000u); }
__device__ __forceinline__ uint32_t even_mask(int axis) { return axis == 0 ? 0x80000000u : (axis == 1 ? 0xa0000000u : 0xe0000000u); }

// aproximate_biggest_axis's final choice (src/KD_Tree.cpp:90-94)
__device__ __forceinline__ int biggest_axis(float ex, float ey, float ez) {
    float b = fmaxf(fmaxf(ex, ey), ez);
    return b == ex ? 0 : (b == ey ? 1 : 2);
}

// Node on `level` whose range holds position i; returns 0 if i is the median photon
// of an ancestor.  *start receives the node's first position.
__device__ __forceinline__ long long locate(long long i, int level, long long n, long long* start) {
    long long e = 1, s = 0, c = n;
    for (int j = 0; j < level; ++j) {
        long long half = c >> 1, odd = c & 1;
        if (i < s + half) { e = 2 * e; }
        else if (odd && i == s + half) { *start = 0; return 0; }
        else { e = 2 * e + 1; s += half + odd; }
        c = half;
    }
    *start = s;
    return e;
}

// The global passes' state.  Levels alternate between two box and two cursor arrays.
struct LevelState {
    int* box;          // 6 per node of this level: min xyz, max xyz (f2ord)
    int* cnt;          // 3 per node of this level: partition cursors (below / equal / above)
    int* next_box;     // the next level's
    int* next_cnt;
    uint32_t* hist;    // [pass][node][256]
    uint2* sel;        // [pass][node]: (selected high bits of the median key, rank left) after the pass
    long long nodes;   // nodes the arrays hold
};

// A node's selection before `pass` (4: complete).
struct NodeSel {
    uint32_t prefix;   // selected high bits of the median key
    int krem;          // remaining rank inside the selected bin
    int eq;            // photons whose key equals the median key (pass 4)
    int axis;
    int first;         // first digit pass that runs (earlier digits fixed by the node's box)
};

struct Buffers {
    float* x[2]; float* y[2]; float* z[2]; uint32_t* id[2];
};

// One half of the double buffer, picked with selects: indexing the kernel parameter
// with a runtime value would copy all of it to local memory in every thread.
struct Side {
    float* x; float* y; float* z; uint32_t* id;
};
__device__ __forceinline__ Side side(const Buffers& B, int k) {
    return k ? Side{B.x[1], B.y[1], B.z[1], B.id[1]} : Side{B.x[0], B.y[0], B.z[0], B.id[0]};
}

// Chunk -> at most two nodes A, B on `level`.
struct ChunkNodes {
    long long eA, sA, eB, sB, c;
};

__device__ __forceinline__ void chunk_nodes(long long a, long long chunk, int level, long long n, ChunkNodes& cn) {
    long long c = n >> level;
    long long s;
    long long e = locate(a, level, n, &s);
    if (e == 0) e = locate(a + 1, level, n, &s);
    cn.eA = e; cn.sA = s; cn.c = c;
    long long endA = s + c;
    cn.eB = 0; cn.sB = -1;
    if (endA < a + chunk && endA < n) {
        long long s2;
        long long e2 = locate(endA, level, n, &s2);
        if (e2 == 0 && endA + 1 < n) e2 = locate(endA + 1, level, n, &s2);
        if (e2) { cn.eB = e2; cn.sB = s2; }
    }
}

// 0 = node A, 1 = node B, -1 = not inside a node on this level
__device__ __forceinline__ int which(long long i, const ChunkNodes& cn) {
    if (i >= cn.sA && i < cn.sA + cn.c) return 0;
    if (cn.eB && i >= cn.sB && i < cn.sB + cn.c) return 1;
    return -1;
}

// The root's box (the partition computes the other nodes').
__global__ void __launch_bounds__(kWideThreads) k_root_box(Buffers B, long long n, int* box) {
    __shared__ int sb[6];
    if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : (int)0x80000000;
    const long long a = blockIdx.x * (long long)(kWideThreads * kItems);
    int mn[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff};
    int mx[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
#pragma unroll
    for (int it = 0; it < kItems; ++it) {   // (past the end: the chunk's first photon again)
        const long long i = a + it * kWideThreads + threadIdx.x, j = i < n ? i : a;
        const int v[3] = {f2ord(B.x[0][j]), f2ord(B.y[0][j]), f2ord(B.z[0][j])};
#pragma unroll
        for (int k = 0; k < 3; ++k) { mn[k] = min(mn[k], v[k]); mx[k] = max(mx[k], v[k]); }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int v = __reduce_min_sync(0xffffffffu, mn[k]), u = __reduce_max_sync(0xffffffffu, mx[k]);
        if ((threadIdx.x & 31) == 0) { atomicMin(&sb[k], v); atomicMax(&sb[3 + k], u); }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&box[threadIdx.x], sb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&box[threadIdx.x], sb[threadIdx.x]);
}

// One warp: node t's selection before `pass`.  Every key of the node
// lies between the keys of its box's ends along its axis (both orders are IEEE total
// order), so the whole leading digits those two keys share are the median's digits too:
// they go into the prefix, and the radix-select passes over them are skipped (the last pass
// always runs: it gives the split and the count of keys equal to the median).  Otherwise
// the digit of pass - 1 is the bin of its histogram that holds rank krem.  `keep` (one CTA
// per node) stores the result for the next passes.
__device__ __forceinline__ NodeSel node_select(const LevelState& S, long long t, int count, int pass, bool keep,
                                               int* err) {
    const int lane = threadIdx.x & 31;
    const int* b = S.box + 6 * t;
    const int b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3], b4 = b[4], b5 = b[5];
    // (all loads in flight together, used or not)
    uint2 prev = make_uint2(0u, 0u);
    uint4 h0 = make_uint4(0u, 0u, 0u, 0u), h1 = h0;
    if (pass >= 2) prev = S.sel[(pass - 2) * S.nodes + t];
    if (pass >= 1) {
        const uint4* h = reinterpret_cast<const uint4*>(S.hist + ((pass - 1) * S.nodes + t) * 256) + 2 * lane;
        h0 = h[0];
        h1 = h[1];
    }
    NodeSel s;
    s.axis = biggest_axis(ord2f(b3) - ord2f(b0), ord2f(b4) - ord2f(b1), ord2f(b5) - ord2f(b2));
    const uint32_t lo = f2key(ord2f(s.axis == 0 ? b0 : (s.axis == 1 ? b1 : b2)));
    const uint32_t hi = f2key(ord2f(s.axis == 0 ? b3 : (s.axis == 1 ? b4 : b5)));
    s.first = min(__clz(lo ^ hi) >> 3, 3);
    s.prefix = lo & ~(0xffffffffu >> (8 * s.first));
    s.krem = count >> 1;
    s.eq = 0;
    if (pass <= s.first) return s;
    if (pass - 1 > s.first) {
        s.prefix = prev.x;
        s.krem = (int)prev.y;
    }
    const uint32_t v[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += v[k];
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    uint32_t cum = incl - sum;
    // lane whose range [cum, incl) contains krem
    const unsigned bal = __ballot_sync(0xffffffffu, (uint32_t)s.krem >= cum && (uint32_t)s.krem < incl);
    if (!bal) {
        if (lane == 0) atomicOr(err, 1);   // histogram does not hold rank krem
        return s;
    }
    int bin = lane * 8 + 7;
    uint32_t at = cum, eq = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (eq == 0 && (uint32_t)s.krem < at + v[k]) { bin = lane * 8 + k; cum = at; eq = v[k]; }
        at += v[k];
    }
    const int owner = __ffs(bal) - 1;
    s.krem -= (int)__shfl_sync(0xffffffffu, cum, owner);
    s.prefix |= (uint32_t)__shfl_sync(0xffffffffu, bin, owner) << (24 - 8 * (pass - 1));
    s.eq = (int)__shfl_sync(0xffffffffu, eq, owner);
    if (keep && lane == 0 && pass < 4) S.sel[(pass - 1) * S.nodes + t] = make_uint2(s.prefix, (uint32_t)s.krem);
    return s;
}

// Grid-wide clear of histogram `pass` for `nodes` nodes.
__device__ __forceinline__ void clear_hist(const LevelState& S, int pass, long long nodes) {
    uint4* h = reinterpret_cast<uint4*>(S.hist + pass * S.nodes * 256);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 64 * nodes; i += (long long)gridDim.x * blockDim.x)
        h[i] = make_uint4(0u, 0u, 0u, 0u);
}

// next: nodes of the next level (0: there is none).
template <int T>
__global__ void __launch_bounds__(T) k_hist(Buffers B, int cur, int level, long long n, long long first, LevelState S,
                                            long long next, int pass, int* err) {
    __shared__ ChunkNodes cn;
    __shared__ uint32_t sh[2][256];
    __shared__ uint32_t pre[2];
    __shared__ int ax[2];
    __shared__ bool live[2];   // the node's digit for this pass is not fixed by its box
    long long a = blockIdx.x * (long long)(T * kItems);
    // the chunk's coordinates, loaded before the wait: the level's partition wrote them, at
    // least two launches ago (pass 0: one, so it loads them after)
    const Side P = side(B, cur);
    float px[kItems], py[kItems], pz[kItems];
    auto load = [&]() {
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const long long i = a + it * T + threadIdx.x, j = i < n ? i : a;
            px[it] = __ldcg(&P.x[j]); py[it] = __ldcg(&P.y[j]); pz[it] = __ldcg(&P.z[j]);
        }
    };
    if (pass > 0) load();
    if (threadIdx.x == 0) chunk_nodes(a, T * kItems, level, n, cn);
    for (int k = threadIdx.x; k < 512; k += T) (&sh[0][0])[k] = 0;
    early_launch_wait();
    if (pass == 0) load();
    if (pass == 0) {
        clear_hist(S, 3, first);
        for (long long t = blockIdx.x * (long long)T + threadIdx.x; t < next; t += (long long)gridDim.x * T) {
            for (int k = 0; k < 6; ++k) S.next_box[6 * t + k] = k < 3 ? 0x7fffffff : (int)0x80000000;
            for (int k = 0; k < 3; ++k) S.next_cnt[3 * t + k] = 0;
        }
    } else if (pass >= 2) {
        clear_hist(S, pass - 2, next);
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        const int w = threadIdx.x >> 5;
        const long long e = w ? cn.eB : cn.eA, s = w ? cn.sB : cn.sA;
        if (e) {
            const NodeSel q = node_select(S, e - first, (int)cn.c, pass, s >= a, err);
            if ((threadIdx.x & 31) == 0) { ax[w] = q.axis; pre[w] = q.prefix; live[w] = pass >= q.first; }
        } else if ((threadIdx.x & 31) == 0) {
            live[w] = false;
        }
    }
    __syncthreads();
    if (!live[0] && !live[1]) return;
    const int shift = 24 - 8 * pass;
    float val[kItems];
    int wh[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        long long i = a + it * T + threadIdx.x;
        const int w = i < n ? which(i, cn) : -1;
        wh[it] = w >= 0 && live[w] ? w : -1;
        const int axis = wh[it] >= 0 ? ax[wh[it]] : 0;
        val[it] = axis == 0 ? px[it] : (axis == 1 ? py[it] : pz[it]);
    }
#pragma unroll
    for (int it = 0; it < kItems; ++it) {   // every lane runs every round (full-warp match)
        unsigned slot = 0xffffffffu;
        const int w = wh[it];
        if (w >= 0) {
            uint32_t key = f2key(val[it]);
            if (pass == 0 || (key >> (shift + 8)) == (pre[w] >> (shift + 8)))
                slot = (unsigned)w * 256u + ((key >> shift) & 255u);
        }
        // lanes with the same bin add once (the top digits of nearby coordinates
        // coincide, so per-lane atomics would serialise on a few bins)
        const unsigned peers = __match_any_sync(0xffffffffu, slot);
        if (slot != 0xffffffffu && (threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1))
            atomicAdd(&(&sh[0][0])[slot], (uint32_t)__popc(peers));
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 512; k += T) {
        int q = k >> 8;
        uint32_t v = (&sh[0][0])[k];
        long long e = q == 0 ? cn.eA : cn.eB;
        if (v && e) atomicAdd(&S.hist[(pass * S.nodes + e - first) * 256 + (k & 255)], v);
    }
}

template <int T>
__global__ void __launch_bounds__(T) k_partition(Buffers B, int cur, int level, long long n, long long first,
                                                 LevelState L, long long next, uint2* nodes, int* err) {
    __shared__ ChunkNodes cn;
    __shared__ int ax[2], krem[2], eq[2];
    __shared__ uint32_t med[2];
    __shared__ int base[6];
    __shared__ int woff[kItems][T / 32][6];
    __shared__ int sb[4][6];   // boxes of the halves: node A left, right, node B left, right
    long long a = blockIdx.x * (long long)(T * kItems);
    if (threadIdx.x == 0) chunk_nodes(a, T * kItems, level, n, cn);
    if (threadIdx.x < 24) sb[threadIdx.x / 6][threadIdx.x % 6] = (threadIdx.x % 6) < 3 ? 0x7fffffff : (int)0x80000000;
    // the chunk's photons, loaded before the wait (the partition before wrote them)
    float px[kItems], py[kItems], pz[kItems];
    uint32_t pid[kItems];
    const Side S = side(B, cur);
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const long long i = a + it * T + threadIdx.x, j = i < n ? i : a;
        px[it] = __ldcg(&S.x[j]); py[it] = __ldcg(&S.y[j]); pz[it] = __ldcg(&S.z[j]); pid[it] = __ldcg(&S.id[j]);
    }
    early_launch_wait();
    clear_hist(L, 2, next);
    __syncthreads();
    if (threadIdx.x < 64) {
        const int w = threadIdx.x >> 5;
        const long long e = w ? cn.eB : cn.eA, s = w ? cn.sB : cn.sA;
        if (e) {
            const NodeSel q = node_select(L, e - first, (int)cn.c, 4, false, err);
            if ((threadIdx.x & 31) == 0) {
                ax[w] = q.axis; krem[w] = q.krem; eq[w] = q.eq; med[w] = q.prefix;
                if (s >= a) {   // the node's split, written by the CTA its range starts in
                    const float m = key2f(q.prefix);
                    nodes[e].y = __float_as_uint((cn.c & 1) ? m : m + kSplitBias);
                    if (!(cn.c & 1)) nodes[e].x = even_mask(q.axis);
                }
            }
        }
    }
    __syncthreads();
    const int dst = cur ^ 1;
    // coalesced rounds of T consecutive positions; the rank of a photon in its
    // class (node A/B x below/equal/above) follows position order inside the CTA:
    // ballots within a warp, then per-(round, warp) offsets
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    // position past n: -2, ancestor median (stays in place): -1
    int cls[kItems], rank[kItems];
    const Side D = side(B, dst);
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const long long i = a + it * T + threadIdx.x;
        cls[it] = i < n ? which(i, cn) : -2;
    }
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const int w = cls[it];   // node A (0) / B (1), or -1 / -2 as above
        int q = w;
        if (w >= 0) {
            const int axw = ax[w];
            const uint32_t key = f2key(axw == 0 ? px[it] : (axw == 1 ? py[it] : pz[it]));
            q = w * 3 + (key < med[w] ? 0 : (key == med[w] ? 1 : 2));
        }
        cls[it] = q;
        rank[it] = 0;
#pragma unroll
        for (int cq = 0; cq < 6; ++cq) {
            const unsigned m = __ballot_sync(0xffffffffu, q == cq);
            if (q == cq) rank[it] = __popc(m & lt_mask);
            if (lane == 0) woff[it][wid][cq] = __popc(m);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int q = threadIdx.x;
        int run = 0;
        for (int it = 0; it < kItems; ++it)
            for (int w = 0; w < T / 32; ++w) {
                const int v = woff[it][w][q];
                woff[it][w][q] = run;
                run += v;
            }
        long long e = q < 3 ? cn.eA : cn.eB;
        base[q] = (e && run) ? atomicAdd(&L.cnt[3 * (e - first) + q % 3], run) : 0;
    }
    __syncthreads();
    const long long c = cn.c;
    const long long k = c >> 1, odd = c & 1;
    int half[kItems];   // the half the photon goes to (2 w + right), -1: none
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        long long i = a + it * T + threadIdx.x;
        int q = cls[it];
        half[it] = -1;
        if (q == -2) continue;
        const float xv = px[it], yv = py[it], zv = pz[it];
        const uint32_t idv = pid[it];
        long long d;
        if (q < 0) {
            d = i;   // ancestor median: stays in place
        } else {
            int w = q / 3, cl = q % 3;
            long long s = w == 0 ? cn.sA : cn.sB;
            long long r = base[q] + woff[it][wid][q] + rank[it];
            long long kl = krem[w];
            long long lt = k - kl;
            if (cl == 0) d = s + r;
            else if (cl == 1) {
                if (r < kl) d = s + lt + r;
                else if (odd && r == kl) {
                    d = s + k;
                    long long e = w == 0 ? cn.eA : cn.eB;
                    nodes[e].x = idv | odd_mask(ax[w]);
                } else d = s + k + odd + (r - kl - odd);
            } else d = s + k + odd + (eq[w] - kl - odd) + r;
            if (d < s || d >= s + c) { atomicOr(err, 2); continue; }   // inconsistent counts
            if (!(odd && d == s + k)) half[it] = 2 * w + (d >= s + k);
        }
        D.x[d] = xv; D.y[d] = yv; D.z[d] = zv; D.id[d] = idv;
    }
    if (!next) return;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        if (h >= 2 && !cn.eB) break;
        int mn[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff};
        int mx[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            if (half[it] != h) continue;
            const int vx = f2ord(px[it]), vy = f2ord(py[it]), vz = f2ord(pz[it]);
            mn[0] = min(mn[0], vx); mn[1] = min(mn[1], vy); mn[2] = min(mn[2], vz);
            mx[0] = max(mx[0], vx); mx[1] = max(mx[1], vy); mx[2] = max(mx[2], vz);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int v = __reduce_min_sync(0xffffffffu, mn[j]), u = __reduce_max_sync(0xffffffffu, mx[j]);
            if (lane == 0) { atomicMin(&sb[h][j], v); atomicMax(&sb[h][3 + j], u); }
        }
    }
    __syncthreads();
    if (threadIdx.x < 24) {
        const int h = threadIdx.x / 6, j = threadIdx.x % 6;
        const long long e = h < 2 ? cn.eA : cn.eB;
        if (e) {
            int* dst2 = L.next_box + 6 * (2 * (e - first) + (h & 1)) + j;
            if (j < 3) atomicMin(dst2, sb[h][j]); else atomicMax(dst2, sb[h][j]);
        }
    }
}

__global__ void k_load(const float4* __restrict__ pos4, long long n, Buffers B, LevelState S) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (S.nodes > 0 && i < 6) S.box[i] = i < 3 ? 0x7fffffff : (int)0x80000000;
    if (S.nodes > 0 && i < 3) S.cnt[i] = 0;
    if (i >= n) return;
    float4 p = pos4[i];
    B.x[0][i] = p.x; B.y[0][i] = p.y; B.z[0][i] = p.z; B.id[0][i] = (uint32_t)i;
}

// Copy the median photons of levels < level0 from buffer `src` to buffer 0.
__global__ void k_copy_medians(Buffers B, int src, int level0, long long n) {
    long long e = 1 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (1LL << level0)) return;
    int lv = 63 - __clzll(e);
    long long c = n >> lv;
    if (!(c & 1)) return;
    long long p = kd_node_start(e, lv, n) + (c >> 1);
    const Side S = side(B, src);
    B.x[0][p] = S.x[p]; B.y[0][p] = S.y[p]; B.z[0][p] = S.z[p]; B.id[0][p] = S.id[p];
}

// Shared-memory subtree builder: one CTA per node on level0 (at most kSmemSeg photons).
// The photons are sorted once along x, y and z (three index lists; bitonic on the key
// (coordinate, local index)).  Every level then reads each sub-node's extents (first
// and last entry of each list) and its median (middle entry of the chosen axis's list)
// off the lists, and splits all three lists stably into left / median / right.  A
// sub-node of c photons has exactly c/2 photons on each side, so the rank of a photon
// inside its sub-node's class is a block-wide prefix count minus s * (c/2).
struct SmemLayout {
    static constexpr size_t xs = 0;                                  // photons by local index
    static constexpr size_t ys = xs + 4 * kSmemSeg;
    static constexpr size_t zs = ys + 4 * kSmemSeg;
    static constexpr size_t ids = zs + 4 * kSmemSeg;
    static constexpr size_t v = ids + 4 * kSmemSeg;                  // 3 x kSmemSeg uint64 sort keys,
    static constexpr size_t lists = v;                               // then 3 x kSmemSeg uint32 lists
    static constexpr size_t temp = v + 4 * 3 * kSmemSeg;             // and 3 x kSmemSeg uint32 split output
    static constexpr size_t cls = v + 8 * 3 * kSmemSeg;              // class per photon (0 left, 1 median, 2 right)
    static constexpr size_t segs = cls + 4 * kSmemSeg;               // sub-node starts (up to kSmemSeg)
    static constexpr size_t axes = segs + 4 * kSmemSeg;              // split axis per sub-node (up to kSmemSeg / 2)
    static constexpr size_t warp = axes + 4 * (kSmemSeg / 2);        // block scan scratch
    static constexpr size_t total = warp + 4 * 6 * (kSmemThreads / 32);
};

__device__ __forceinline__ float axis_coord(const float* X, const float* Y, const float* Z, int a, uint32_t q) {
    return a == 0 ? X[q] : (a == 1 ? Y[q] : Z[q]);
}

// Compare-exchange of a thread's keys E0 < E1 (positions 4t + E0, 4t + E1) in all three
// lists, ascending where bit k of the position is clear.
template <int E0, int E1>
__device__ __forceinline__ void sort_pair(unsigned long long (&key)[3][4], int tid, int k) {
    const bool up = ((4 * tid + E0) & k) == 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const unsigned long long lo = key[a][E0], hi = key[a][E1];
        const bool swap = (lo > hi) == up;
        key[a][E0] = swap ? hi : lo;
        key[a][E1] = swap ? lo : hi;
    }
}

__global__ void __launch_bounds__(kSmemThreads) k_smem_build(Buffers B, int src, int level0, long long n, uint2* nodes) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* X = (float*)(smem + SmemLayout::xs);
    float* Y = (float*)(smem + SmemLayout::ys);
    float* Z = (float*)(smem + SmemLayout::zs);
    uint32_t* I = (uint32_t*)(smem + SmemLayout::ids);
    unsigned long long* V = (unsigned long long*)(smem + SmemLayout::v);
    uint32_t* L = (uint32_t*)(smem + SmemLayout::lists);   // current lists: L[a * kSmemSeg + p]
    uint32_t* T = (uint32_t*)(smem + SmemLayout::temp);    // split output (swapped with L per level)
    int* cls = (int*)(smem + SmemLayout::cls);
    int* segs = (int*)(smem + SmemLayout::segs);
    int* axes = (int*)(smem + SmemLayout::axes);
    int (*wsum)[6] = (int (*)[6])(smem + SmemLayout::warp);

    const long long e0 = (1LL << level0) + blockIdx.x;
    const long long s0 = kd_node_start(e0, level0, n);
    const int c0 = (int)(n >> level0);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31, wid = tid >> 5;
    const Side S = side(B, src);
    early_launch_wait();
    for (int i = tid; i < c0; i += nt) {
        X[i] = S.x[s0 + i]; Y[i] = S.y[s0 + i]; Z[i] = S.z[s0 + i]; I[i] = S.id[s0 + i];
    }
    __syncthreads();
    // three sorted lists: a bitonic network over kSmemSeg keys (coordinate key, local
    // index) per list, padding keys ~0 sorting last.  Thread t holds keys 4t..4t+3 of
    // every list in registers: strides 1 and 2 are exchanged in registers, 4..64 with
    // warp shuffles (partner lane t ^ stride/4), 128 and up through shared memory.
    static_assert(kSmemSeg == 4 * kSmemThreads, "four keys per thread and list");
    unsigned long long key[3][4];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int p = 4 * tid + e;
            key[a][e] = p < c0 ? ((unsigned long long)f2key(axis_coord(X, Y, Z, a, p)) << 32) | (unsigned)p : ~0ull;
        }
    for (int k = 2; k <= kSmemSeg; k <<= 1) {
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            if (jj >= 4) {
                const bool smem_stage = jj >= 128;
                if (smem_stage) {
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int e = 0; e < 4; ++e) V[a * kSmemSeg + 4 * tid + e] = key[a][e];
                    __syncthreads();
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = 4 * tid + e;
                    // the lower index of a pair keeps the minimum in an ascending run
                    const bool keep_min = ((i & jj) == 0) == ((i & k) == 0);
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const unsigned long long other =
                            smem_stage ? V[a * kSmemSeg + (i ^ jj)]
                                       : (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)key[a][e], jj >> 2);
                        const unsigned long long mine = key[a][e];
                        key[a][e] = keep_min ? (mine < other ? mine : other) : (mine < other ? other : mine);
                    }
                }
                if (smem_stage) __syncthreads();
            } else if (jj == 2) {
                sort_pair<0, 2>(key, tid, k);
                sort_pair<1, 3>(key, tid, k);
            } else {
                sort_pair<0, 1>(key, tid, k);
                sort_pair<2, 3>(key, tid, k);
            }
        }
    }
    // keys -> index lists (the lists overlay the keys; the last shared-memory stage
    // ended with a barrier)
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int p = 4 * tid + e;
            if (p < c0) L[a * kSmemSeg + p] = (uint32_t)(key[a][e] & 0xffffffffu);
        }
    __syncthreads();
    for (int j = 0;; ++j) {
        const int c = c0 >> j;
        const int nsub = 1 << j;
        for (int s = tid; s < nsub; s += nt) {
            int st = 0, cc = c0;
            for (int b = j - 1; b >= 0; --b) {
                int half = cc >> 1;
                if ((s >> b) & 1) st += half + (cc & 1);
                cc = half;
            }
            segs[s] = st;
        }
        __syncthreads();
        if (c <= 1) {
            for (int s = tid; s < nsub; s += nt) nodes[(e0 << j) + s] = make_uint2(I[L[segs[s]]], 0u);
            break;
        }
        const int k = c >> 1, odd = c & 1;
        // node records: extents and median read off the lists
        for (int s = tid; s < nsub; s += nt) {
            const int st = segs[s];
            const float ex = X[L[st + c - 1]] - X[L[st]];
            const float ey = Y[L[kSmemSeg + st + c - 1]] - Y[L[kSmemSeg + st]];
            const float ez = Z[L[2 * kSmemSeg + st + c - 1]] - Z[L[2 * kSmemSeg + st]];
            const int a = biggest_axis(ex, ey, ez);
            const uint32_t q = L[a * kSmemSeg + st + k];
            const float m = axis_coord(X, Y, Z, a, q);
            const long long e = (e0 << j) + s;
            if (odd) nodes[e] = make_uint2(I[q] | odd_mask(a), __float_as_uint(m));
            else nodes[e] = make_uint2(even_mask(a), __float_as_uint(m + kSplitBias));
            axes[s] = a;
        }
        __syncthreads();
        // class of every photon (0 left, 1 median, 2 right) from its place in its
        // sub-node's axis list
        const int nv = nsub * c;
        for (int v = tid; v < nv; v += nt) {
            const int s = v / c, off = v - s * c;
            cls[L[axes[s] * kSmemSeg + segs[s] + off]] = off < k ? 0 : ((odd && off == k) ? 1 : 2);
        }
        __syncthreads();
        // stable split of the three lists: thread t takes positions v = 4t..4t+3 of the
        // level's index space v -> (sub-node s = v / c, offset v % c)
        int cnt[6] = {0, 0, 0, 0, 0, 0};
        int cl[3][4];
        uint32_t qq[3][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int v = 4 * tid + r;
            const int s = v / c, off = v - s * c;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                cl[a][r] = -1;
                if (v < nv) {
                    const uint32_t q = L[a * kSmemSeg + segs[s] + off];
                    qq[a][r] = q;
                    cl[a][r] = cls[q];
                    cnt[2 * a] += cl[a][r] == 0;
                    cnt[2 * a + 1] += cl[a][r] == 2;
                }
            }
        }
        // block-wide exclusive prefix of the 6 counters
        int excl[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) {
            int x = cnt[u];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            excl[u] = x - cnt[u];
            if (lane == 31) wsum[wid][u] = x;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 6; ++u) {
            int before = 0;
            for (int w = 0; w < wid; ++w) before += wsum[w][u];
            excl[u] += before;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int v = 4 * tid + r;
            if (v >= nv) break;
            const int s = v / c;
            const int st = segs[s];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int c2 = cl[a][r];
                int dst;
                if (c2 == 0) dst = st + (excl[2 * a]++ - s * k);
                else if (c2 == 1) dst = st + k;
                else dst = st + k + odd + (excl[2 * a + 1]++ - s * k);
                T[a * kSmemSeg + dst] = qq[a][r];
                // a median keeps its place for good, outside every later sub-node: it
                // goes into both buffers (this level's reads of L ended at the barrier)
                if (c2 == 1) L[a * kSmemSeg + dst] = qq[a][r];
            }
        }
        __syncthreads();
        uint32_t* const done = L;   // the split lists become the current ones
        L = T;
        T = done;
    }
    __syncthreads();
    for (int i = tid; i < c0; i += nt) {
        const uint32_t q = L[i];
        B.x[0][s0 + i] = X[q]; B.y[0][s0 + i] = Y[q]; B.z[0][s0 + i] = Z[q]; B.id[0][s0 + i] = I[q];
    }
}

int first_smem_level(long long n) {
    int l = 0;
    while ((n >> l) > kSmemSeg) ++l;
    return l;
}

}  // namespace

long long kd_node_array_len(long long n) {
    if (n <= 0) return 0;
    // kdtree.resize(std::pow(2, (int)(std::log2f(size) + 1)))  (src/KD_Tree.cpp:186)
    long long ref = (long long)std::pow(2.0, (int)(std::log2f((float)n) + 1));
    int L = 63 - __builtin_clzll((unsigned long long)n);
    long long need = 1LL << (L + 1);
    return ref > need ? ref : need;
}

size_t kd_scratch_bytes(long long n) {
    if (n <= 0) return 256;
    int l0 = first_smem_level(n);
    long long maxnodes = l0 > 0 ? (1LL << (l0 - 1)) : 1;
    size_t b = 0;
    b += 16 * (size_t)n;                      // second buffer x/y/z/id
    b += 2 * 36 * (size_t)maxnodes;           // boxes and cursors of two levels
    b += 3 * 8 * (size_t)maxnodes;            // selection state after passes 0 .. 2
    b += 4 * 1024 * (size_t)maxnodes;         // histograms of the four passes
    return b + 1024;
}

int kd_build(const float4* pos4, long long n, KdTree& tree, void* scratch, size_t scratch_bytes,
             cudaStream_t stream, int* launches, int* err) {
    int nl = 0;
    tree.n = n;
    if (n <= 0) { tree.levels = 0; tree.num_nodes = 0; if (launches) *launches = 0; return 0; }
    tree.levels = 63 - __builtin_clzll((unsigned long long)n);
    tree.num_nodes = kd_node_array_len(n);
    if (scratch_bytes < kd_scratch_bytes(n)) return -1;
    int l0 = first_smem_level(n);
    long long maxnodes = l0 > 0 ? (1LL << (l0 - 1)) : 1;
    char* p = (char*)scratch;
    Buffers B;
    B.x[0] = tree.x; B.y[0] = tree.y; B.z[0] = tree.z; B.id[0] = tree.id;
    B.x[1] = (float*)p; p += 4 * (size_t)n;
    B.y[1] = (float*)p; p += 4 * (size_t)n;
    B.z[1] = (float*)p; p += 4 * (size_t)n;
    B.id[1] = (uint32_t*)p; p += 4 * (size_t)n;
    p = (char*)(((uintptr_t)p + 255) & ~(uintptr_t)255);
    LevelState S{};
    S.nodes = l0 > 0 ? maxnodes : 0;
    S.hist = (uint32_t*)p; p += 4 * 1024 * (size_t)maxnodes;
    S.sel = (uint2*)p; p += 3 * 8 * (size_t)maxnodes;
    S.box = (int*)p; p += 24 * (size_t)maxnodes;
    S.next_box = (int*)p; p += 24 * (size_t)maxnodes;
    S.cnt = (int*)p; p += 12 * (size_t)maxnodes;
    S.next_cnt = (int*)p;

    cudaMemsetAsync(tree.nodes, 0, sizeof(uint2) * (size_t)tree.num_nodes, stream);
    k_load<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(pos4, n, B, S);
    nl++;
    int cur = 0;
    if (l0 > 0) {
        // the root's histograms; the passes clear those of the levels below
        for (int pass = 0; pass < 4; ++pass)
            cudaMemsetAsync(S.hist + pass * maxnodes * 256, 0, 1024, stream);
        const long long span = (long long)kWideThreads * kItems;
        k_root_box<<<(unsigned)((n + span - 1) / span), kWideThreads, 0, stream>>>(B, n, S.box);
        nl++;
    }
    for (int l = 0; l < l0; ++l) {
        const long long first = 1LL << l, next = l + 1 < l0 ? 2 * first : 0;
        // half as many CTAs, each twice as wide, while a wide chunk still meets at most
        // two nodes: the passes' per-CTA fixed cost (chunk location, shared-memory
        // reduction) is paid half as often
        const bool wide = (n >> l) > (long long)kWideThreads * kItems;
        const long long span = (long long)(wide ? kWideThreads : kThreads) * kItems;
        const unsigned chunks = (unsigned)((n + span - 1) / span);
        for (int pass = 0; pass < 4; ++pass, ++nl) {
            if (wide) launch_early(k_hist<kWideThreads>, chunks, kWideThreads, 0, stream, B, cur, l, n, first, S, next, pass, err);
            else launch_early(k_hist<kThreads>, chunks, kThreads, 0, stream, B, cur, l, n, first, S, next, pass, err);
        }
        if (wide) launch_early(k_partition<kWideThreads>, chunks, kWideThreads, 0, stream, B, cur, l, n, first, S, next, tree.nodes, err);
        else launch_early(k_partition<kThreads>, chunks, kThreads, 0, stream, B, cur, l, n, first, S, next, tree.nodes, err);
        nl++;
        cur ^= 1;
        std::swap(S.box, S.next_box);
        std::swap(S.cnt, S.next_cnt);
    }
    if (cur == 1 && l0 > 0) {
        long long cnt = (1LL << l0) - 1;
        k_copy_medians<<<(unsigned)((cnt + 255) / 256), 256, 0, stream>>>(B, 1, l0, n);
        nl++;
    }
    size_t smem = SmemLayout::total;
    // once per device: later builds may be recorded into a CUDA graph, and contexts on
    // several threads build concurrently
    static std::once_flag attr_set[kOnceDevices];
    once_per_device(attr_set, [&] { cudaFuncSetAttribute(k_smem_build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
    launch_early(k_smem_build, (unsigned)(1LL << l0), kSmemThreads, smem, stream, B, cur, l0, n, tree.nodes);
    nl++;
    if (launches) *launches = nl;
    return 0;
}

}  // namespace rc
