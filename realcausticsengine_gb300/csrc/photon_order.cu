// Spatial orders of the iteration's photons and merge queries, and the gather's box tree.
//
// Photons are sorted along a Hilbert curve over a grid of the scene's box (Skilling,
// "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004), so that any run of consecutive
// ones is compact: unlike the Morton curve the Hilbert curve has no jumps.  Queries are
// sorted along either (launch_query_order says which and why).
// The gather's photon sets do not depend on how the photons are stored (gather.cu), so its
// chunks are simply runs of the sorted photons, cut evenly into 2^Lc.  (They were the leaves
// of the reference's median-split KD tree, built with four radix-select passes and a
// partition per level: 4.4 ms for the 7.7M photons of the 1080p water pool, where the
// sort, the records and the boxes take 0.74 ms; the query order and gather went from 2.16
// to 1.69 ms.)
//
// The sort is a stable LSD radix sort, 10-bit digits.  A pass reads 4096 keys per block:
// digit counts (k_rs_hist), one scan of all blocks' counts (digit-major), then ranks and
// scatter (k_rs_scatter).  It is bound by the scattered writes (four keys of a digit per
// block on average); its arrays stay in L2.
#include <algorithm>
#include <cmath>

#include "vm.cuh"

namespace rc {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBits = 10, kBins = 1 << kBits;          // digit of a radix pass
constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kPerLane = 16;                           // keys per lane
constexpr int kPerWarp = 32 * kPerLane;
constexpr long long kTile = kWarps * kPerWarp;         // keys per block
constexpr long long kScanTile = 8192;                  // counters per scan block
constexpr long long kChunkNode = 31;                   // photons per chunk, one more where the cut is uneven
constexpr int kBoxLevels = 10;                         // levels of the box tree per launch

size_t round_up(size_t b) { return (b + 255) & ~(size_t)255; }
long long tiles_of(long long n) { return (n + kTile - 1) / kTile; }

// ---------------------------------------------------------------- scan

// Exclusive scan of one 8192-counter tile per block, in place, and the tile's total.
__global__ void __launch_bounds__(1024) k_scan_tile(uint32_t* counts, long long m, uint32_t* tile_sums) {
    __shared__ uint32_t warp_sums[32];
    const long long base = blockIdx.x * kScanTile;
    uint32_t v[8];
    uint32_t sum = 0;
    const long long i0 = base + (long long)threadIdx.x * 8;
    for (int k = 0; k < 8; ++k) { v[k] = (i0 + k < m) ? counts[i0 + k] : 0u; sum += v[k]; }
    uint32_t incl = sum;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = warp_sums[lane], wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(kFull, wi, o);
            if (lane >= o) wi += y;
        }
        warp_sums[lane] = wi - w;
        if (lane == 31) tile_sums[blockIdx.x] = wi;
    }
    __syncthreads();
    uint32_t run = warp_sums[wid] + incl - sum;
    for (int k = 0; k < 8; ++k) {
        if (i0 + k < m) counts[i0 + k] = run;
        run += v[k];
    }
}

// Exclusive scan of the tile totals in one block.
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* sums, long long m) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (long long base = 0; base < m; base += 1024) {
        const long long i = base + threadIdx.x;
        const uint32_t v = i < m ? sums[i] : 0u;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sums[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            uint32_t w = warp_sums[lane], wi = w;
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t y = __shfl_up_sync(kFull, wi, o);
                if (lane >= o) wi += y;
            }
            warp_sums[lane] = wi - w;
        }
        __syncthreads();
        const uint32_t before = carry + warp_sums[wid] + incl - v;
        if (i < m) sums[i] = before;
        __syncthreads();
        if (threadIdx.x == 1023) carry = before + v;
        __syncthreads();
    }
}

__global__ void k_scan_add(uint32_t* counts, long long m, const uint32_t* __restrict__ tile_offsets) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < m) counts[i] += tile_offsets[i / kScanTile];
}

// ---------------------------------------------------------------- curve

__device__ __forceinline__ uint32_t cell_of(float v, float cells) {
    return v > 0.0f ? (v < cells - 1.0f ? (uint32_t)v : (uint32_t)(cells - 1.0f)) : 0u;   // NaN -> 0
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {   // bit b of v (10 bits) to bit 3 b
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}

// Index along the Hilbert curve of cell (x, y, z) of a 2^bits grid: the coordinates' bits
// transformed in place (Skilling's AxestoTranspose), then interleaved, x's the highest.
// Issue-bound: with masks for branches, the 10-bit loops unrolled and the bits spread by
// shifts, the keys of 7.8M photons take 79 us (124 bit by bit;
// four points per thread no faster).
__device__ __forceinline__ void hilbert_step(uint32_t& x, uint32_t& y, uint32_t& z, int b) {
    const uint32_t p = (1u << b) - 1u;
    x ^= p & (0u - ((x >> b) & 1u));
    uint32_t m = 0u - ((y >> b) & 1u), t = (x ^ y) & p;
    x ^= (p & m) | (t & ~m);
    y ^= t & ~m;
    m = 0u - ((z >> b) & 1u);
    t = (x ^ z) & p;
    x ^= (p & m) | (t & ~m);
    z ^= t & ~m;
}
__device__ __forceinline__ void hilbert_gray(uint32_t& x, uint32_t& y, uint32_t& z) {
    y ^= x;
    z ^= y;
    uint32_t t = z >> 1;   // bit b: the parity of z's bits above it
    t ^= t >> 1; t ^= t >> 2; t ^= t >> 4; t ^= t >> 8; t ^= t >> 16;
    x ^= t; y ^= t; z ^= t;
}
__device__ __forceinline__ void hilbert_index(uint32_t x, uint32_t y, uint32_t z, int, uint32_t& key) {   // 10 bits
#pragma unroll
    for (int b = 9; b >= 1; --b) hilbert_step(x, y, z, b);
    hilbert_gray(x, y, z);
    key = (spread3(x) << 2) | (spread3(y) << 1) | spread3(z);
}
__device__ __forceinline__ void hilbert_index(uint32_t x, uint32_t y, uint32_t z, int bits, unsigned long long& key) {
    for (int b = bits - 1; b >= 1; --b) hilbert_step(x, y, z, b);
    hilbert_gray(x, y, z);
    key = ((unsigned long long)((spread3(x >> 10) << 2) | (spread3(y >> 10) << 1) | spread3(z >> 10)) << 30) |
          ((spread3(x & 1023u) << 2) | (spread3(y & 1023u) << 1) | spread3(z & 1023u));
}

// Keys of the points at pos + stride * i, i < n: along the Hilbert curve, or (kMorton, 10
// bits) the Morton curve.  count (optional): the number of points on the device; the ones
// from there to n sort last (kPadLast) or get no key.
template <class Key, bool kPadLast, bool kMorton>
__global__ void k_curve_keys(const float* __restrict__ pos, int stride, long long n,
                             const unsigned long long* __restrict__ count, CurveFrame f, Key* __restrict__ keys) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (count && (unsigned long long)i >= *count) {
        if (kPadLast) keys[i] = ~(Key)0;
        return;
    }
    const float* p = pos + (long long)stride * i;
    const float cells = (float)(1 << f.bits);
    const uint32_t x = cell_of((p[0] - f.lo[0]) * f.scale[0], cells);
    const uint32_t y = cell_of((p[1] - f.lo[1]) * f.scale[1], cells);
    const uint32_t z = cell_of((p[2] - f.lo[2]) * f.scale[2], cells);
    if (kMorton) keys[i] = spread3(x) | (spread3(y) << 1) | (spread3(z) << 2);
    else hilbert_index(x, y, z, f.bits, keys[i]);
}

// ---------------------------------------------------------------- radix sort

// Digit counts per block, digit-major (hist[d * blocks + b]), so that one exclusive scan of
// the whole array gives every (digit, block) its first output position.
template <class Key>
__global__ void __launch_bounds__(kThreads) k_rs_hist(const Key* __restrict__ keys, long long n,
                                                      const unsigned long long* __restrict__ count, int shift,
                                                      uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[kBins];
    for (int d = threadIdx.x; d < kBins; d += kThreads) cnt[d] = 0;
    __syncthreads();
    if (count) n = (long long)min(*count, (unsigned long long)n);
    const long long base = (long long)blockIdx.x * kTile;
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
        const long long i = base + k * kThreads + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(uint32_t)(keys[i] >> shift) & (kBins - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kBins; d += kThreads) hist[(long long)d * gridDim.x + blockIdx.x] = cnt[d];
}

// Stable scatter of one block's keys: warp w ranks its 512 consecutive keys round by round
// (lanes of one digit find each other with a match, the digit's running count is in shared
// memory), and a prefix over the warps and the digits gives each key its place in the
// sorted tile.  kFirst: the values are the keys' own indices; kLast: the sorted keys are not
// needed any more.  Latency-bound (loads, the rounds' chain through shared memory, scattered
// sectors), so 5 blocks share an SM at 48 registers although a few spill (4 with 64-bit
// keys); and where 32-bit keys and
// values are both written the tile is first put in order in shared memory, so that the ~4
// keys of a digit leave together (values alone leave faster from the ranking lanes).  7.8M
// photons, three passes: 153 + 125 + 77 us at 80-112 registers without the reordering, 102 + 99
// + 75 with it and 3 blocks, 94 + 90 + 63 with 4, 93 + 88 + 53 with 5.
template <class Key, bool kFirst, bool kLast>
__global__ void __launch_bounds__(kThreads, sizeof(Key) == 4 ? 5 : 4) k_rs_scatter(const Key* __restrict__ keys_in,
                                                         const uint32_t* __restrict__ vals_in,
                                                         Key* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                                         long long n, const unsigned long long* __restrict__ count,
                                                         int shift, const uint32_t* __restrict__ offsets,
                                                         const uint32_t* __restrict__ tile_offsets) {
    constexpr bool kInOrder = !kLast && sizeof(Key) == 4;   // the tile goes through shared memory
    // the warps' counts, then (the ranks known) the sorted tile's keys
    __shared__ union __align__(16) { uint16_t wc[kWarps][kBins]; Key key[kInOrder ? kTile : 1]; } u;
    __shared__ uint32_t val[kInOrder ? kTile : 1];
    __shared__ __align__(16) uint32_t first[kBins];    // a digit's output position (kInOrder: less its place in the tile)
    __shared__ __align__(16) uint32_t inside[kInOrder ? kBins : 4];   // its place in the tile
    __shared__ uint32_t warp_sum[kWarps];
    static_assert(kBins == 4 * kThreads, "four digits per thread");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    for (int k = threadIdx.x; k < kWarps * kBins / 2; k += kThreads) reinterpret_cast<uint32_t*>(&u.wc[0][0])[k] = 0u;
    if (count) n = (long long)min(*count, (unsigned long long)n);
    const long long tile = (long long)blockIdx.x * kTile, base = tile + (long long)warp * kPerWarp + lane;
    Key key[kPerLane];
    uint32_t place[kPerLane];   // digit, rank among the warp's keys of the digit << 16; then the place in the tile
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) key[r] = base + r * 32 < n ? keys_in[base + r * 32] : (Key)0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        const bool valid = base + r * 32 < n;
        const uint32_t d = valid ? (uint32_t)(key[r] >> shift) & (kBins - 1) : kBins;
        const unsigned peers = __match_any_sync(kFull, d);
        uint32_t before = 0;
        if (valid) before = u.wc[warp][d];
        __syncwarp();
        if (valid && (peers & lt) == 0u) u.wc[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        place[r] = d | ((before + __popc(peers & lt)) << 16);
    }
    __syncthreads();
    if (!kInOrder) {
        for (int d = threadIdx.x; d < kBins; d += kThreads) {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = u.wc[w][d];
                u.wc[w][d] = (uint16_t)run;
                run += c;
            }
            const long long o = (long long)d * gridDim.x + blockIdx.x;
            first[d] = offsets[o] + tile_offsets[o / kScanTile];
        }
    } else {
        // four digits per thread, in order
        uint32_t at[4], run[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const long long o = (long long)(4 * threadIdx.x + j) * gridDim.x + blockIdx.x;
            at[j] = offsets[o] + tile_offsets[o / kScanTile];
        }
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            uint2* const c = reinterpret_cast<uint2*>(&u.wc[w][0]) + threadIdx.x;
            const uint2 q = *c;
            *c = make_uint2(run[0] | (run[1] << 16), run[2] | (run[3] << 16));
            run[0] += q.x & 0xffffu; run[1] += q.x >> 16; run[2] += q.y & 0xffffu; run[3] += q.y >> 16;
        }
        const uint32_t sum = run[0] + run[1] + run[2] + run[3];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        uint32_t in = incl - sum;
        for (int w = 0; w < warp; ++w) in += warp_sum[w];
        const uint4 place4 = make_uint4(in, in + run[0], in + run[0] + run[1], in + run[0] + run[1] + run[2]);
        reinterpret_cast<uint4*>(inside)[threadIdx.x] = place4;
        reinterpret_cast<uint4*>(first)[threadIdx.x] =
            make_uint4(at[0] - place4.x, at[1] - place4.y, at[2] - place4.z, at[3] - place4.w);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        const long long i = base + r * 32;
        if (i >= n) continue;
        const uint32_t d = place[r] & 0xffffu;
        const uint32_t among = u.wc[warp][d] + (place[r] >> 16);
        if (kInOrder) {
            place[r] = inside[d] + among;
        } else {
            if (!kLast) keys_out[first[d] + among] = key[r];
            vals_out[first[d] + among] = kFirst ? (uint32_t)i : vals_in[i];
        }
    }
    if (!kInOrder) return;
    __syncthreads();   // the counts are read: their memory takes the keys
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        const long long i = base + r * 32;
        if (i >= n) continue;
        u.key[place[r]] = key[r];
        val[place[r]] = kFirst ? (uint32_t)i : vals_in[i];
    }
    __syncthreads();
    const int held = (int)min((long long)kTile, n - tile);
    for (int k = threadIdx.x; k < held; k += kThreads) {
        const Key q = u.key[k];
        const uint32_t to = first[(uint32_t)(q >> shift) & (kBins - 1)] + (uint32_t)k;
        keys_out[to] = q;
        vals_out[to] = val[k];
    }
}

// The sort's working memory, cut from one block.
template <class Key> struct SortSpace {
    Key* keys[2];
    uint32_t* vals;
    uint32_t* hist;
    uint32_t* tiles;
    SortSpace(void* scratch, long long n) {
        char* p = (char*)scratch;
        keys[0] = (Key*)p; p += round_up(sizeof(Key) * (size_t)n);
        keys[1] = (Key*)p; p += round_up(sizeof(Key) * (size_t)n);
        vals = (uint32_t*)p; p += round_up(4 * (size_t)n);
        hist = (uint32_t*)p; p += round_up(4 * (size_t)(tiles_of(n) * kBins));
        tiles = (uint32_t*)p;
    }
};

// order = the indices 0 .. n - 1 sorted by keys[0] (3 * bits bits).
template <class Key>
void sort_keys(const SortSpace<Key>& sp, long long n, const unsigned long long* count, int bits, uint32_t* order,
               cudaStream_t s, int* launches) {
    const long long blocks = tiles_of(n), m = blocks * kBins, scans = (m + kScanTile - 1) / kScanTile;
    const int passes = (3 * bits + kBits - 1) / kBits;
    const uint32_t* in = nullptr;
    for (int p = 0; p < passes; ++p) {
        const Key* kin = sp.keys[p & 1];
        Key* kout = sp.keys[(p & 1) ^ 1];
        uint32_t* out = ((passes - 1 - p) & 1) ? sp.vals : order;
        const int shift = p * kBits;
        const unsigned g = (unsigned)blocks;
        k_rs_hist<Key><<<g, kThreads, 0, s>>>(kin, n, count, shift, sp.hist);
        k_scan_tile<<<(unsigned)scans, 1024, 0, s>>>(sp.hist, m, sp.tiles);
        k_scan_sums<<<1, 1024, 0, s>>>(sp.tiles, scans);
        if (p == 0 && passes == 1)
            k_rs_scatter<Key, true, true><<<g, kThreads, 0, s>>>(kin, in, kout, out, n, count, shift, sp.hist, sp.tiles);
        else if (p == 0)
            k_rs_scatter<Key, true, false><<<g, kThreads, 0, s>>>(kin, in, kout, out, n, count, shift, sp.hist, sp.tiles);
        else if (p == passes - 1)
            k_rs_scatter<Key, false, true><<<g, kThreads, 0, s>>>(kin, in, kout, out, n, count, shift, sp.hist, sp.tiles);
        else
            k_rs_scatter<Key, false, false><<<g, kThreads, 0, s>>>(kin, in, kout, out, n, count, shift, sp.hist, sp.tiles);
        in = out;
    }
    if (launches) *launches += 4 * passes;
}

template <class Key, bool kPadLast, bool kMorton>
void order_points(const float* pos, int stride, long long n, const unsigned long long* count, const CurveFrame& f,
                  void* scratch, uint32_t* order, cudaStream_t s, int* launches) {
    const SortSpace<Key> sp(scratch, n);
    k_curve_keys<Key, kPadLast, kMorton><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pos, stride, n, count, f, sp.keys[0]);
    if (launches) *launches += 1;
    sort_keys<Key>(sp, n, kPadLast ? nullptr : count, f.bits, order, s, launches);
}

// ---------------------------------------------------------------- records and boxes

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// One warp per chunk: the chunk's photons gathered into sorted order (positions only when
// ph.dir is null) and its box.
__global__ void __launch_bounds__(256) k_chunks(const PhotonBuf ph, const uint32_t* __restrict__ id, long long n, int lc,
                                                TreePhotons tp, float4* __restrict__ lo, float4* __restrict__ hi) {
    const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long m = 1LL << lc;
    if (w >= m) return;
    const long long start = (w * n) >> lc, c = (((w + 1) * n) >> lc) - start;   // <= 32
    float4 a = make_float4(INFINITY, INFINITY, INFINITY, 0.0f), b = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
    if (lane < c) {
        const uint32_t i = id[start + lane];
        a = b = ph.pos[i];
        tp.t0[start + lane] = a;
        if (ph.dir) {
            tp.t1[start + lane] = ph.dir[i];
            tp.t2[start + lane] = ph.tp[i];
        }
    }
    a = make_float4(warp_min(a.x), warp_min(a.y), warp_min(a.z), __uint_as_float((uint32_t)start));
    b = make_float4(warp_max(b.x), warp_max(b.y), warp_max(b.z), __uint_as_float((uint32_t)c));
    if (lane == 0) {
        lo[m + w] = a;
        hi[m + w] = b;
    }
}

// Boxes of the nodes on levels [top, bottom), bottom-up, one block per node of level `top`:
// each the union of its children's.
__global__ void __launch_bounds__(256) k_box_levels(int top, int bottom, float4* lo, float4* hi) {
    for (int l = bottom - 1; l >= top; --l) {
        const int count = 1 << (l - top);
        for (int i = threadIdx.x; i < count; i += 256) {
            const long long e = (1LL << l) + (long long)blockIdx.x * count + i;
            const float4 a = lo[2 * e], b = lo[2 * e + 1], c = hi[2 * e], d = hi[2 * e + 1];
            lo[e] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f);
            hi[e] = make_float4(fmaxf(c.x, d.x), fmaxf(c.y, d.y), fmaxf(c.z, d.z), 0.0f);
        }
        __syncthreads();
    }
}

}  // namespace

size_t scan_scratch_words(long long m) { return (size_t)(m / kScanTile + 2); }

void launch_scan_counts(uint32_t* counts, long long m, uint32_t* tile_scratch, cudaStream_t s) {
    if (m <= 0) return;
    const long long tiles = (m + kScanTile - 1) / kScanTile;
    k_scan_tile<<<(unsigned)tiles, 1024, 0, s>>>(counts, m, tile_scratch);
    k_scan_sums<<<1, 1024, 0, s>>>(tile_scratch, tiles);
    k_scan_add<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(counts, m, tile_scratch);
}

CurveFrame curve_frame(const float lo[3], const float hi[3], float radius) {
    CurveFrame f;
    float ext = 0.0f;
    for (int k = 0; k < 3; ++k) ext = std::max(ext, hi[k] - lo[k]);
    // A cell should not be wider than the merge spheres it is searched with: the photons of
    // a cell keep their storage order, and a query tests whole chunks.  10 bits per axis
    // (three passes) reach 2 radii in a scene up to 2048 radii wide, as rendered scenes are;
    // wider ones take more bits, in 64-bit keys.
    f.bits = 10;
    while (f.bits < 20 && ext > 2.0f * radius * (float)(1 << f.bits)) ++f.bits;
    const float cells = (float)(1 << f.bits) - 0.01f;
    for (int k = 0; k < 3; ++k) {
        const float e = hi[k] - lo[k];
        f.lo[k] = lo[k];
        f.scale[k] = e > 0.0f && e < INFINITY ? cells / e : 0.0f;
    }
    return f;
}

size_t order_scratch_bytes(long long n) {
    n = std::max(n, 1LL);
    const long long m = tiles_of(n) * kBins;
    return 2 * round_up(8 * (size_t)n) + round_up(4 * (size_t)n) + round_up(4 * (size_t)m) +
           round_up(4 * scan_scratch_words(m));
}

void launch_query_order(const float* qpos, int stride, long long nq, const CurveFrame& frame, bool parks, void* scratch,
                        uint32_t* order, int* launches, cudaStream_t s, const unsigned long long* nq_dev) {
    if (nq <= 0) return;
    if (!parks) {
        CurveFrame f = frame;   // 10 bits per axis
        for (float& k : f.scale) k *= 1023.99f / ((float)(1 << frame.bits) - 0.01f);
        f.bits = 10;
        order_points<uint32_t, false, true>(qpos, stride, nq, nq_dev, f, scratch, order, s, launches);
    } else if (frame.bits <= 10) {
        order_points<uint32_t, false, false>(qpos, stride, nq, nq_dev, frame, scratch, order, s, launches);
    } else {
        order_points<unsigned long long, false, false>(qpos, stride, nq, nq_dev, frame, scratch, order, s, launches);
    }
}

int photon_chunk_level(long long n) {
    if (n <= 0) return -1;
    int l = 0;
    while ((n >> l) > kChunkNode) ++l;
    return l;
}

void launch_photon_order(const PhotonBuf& ph, long long n, const unsigned long long* count, const CurveFrame& frame,
                         void* scratch, const PhotonTree& tree, TreePhotons tp, int* launches, cudaStream_t s) {
    if (n <= 0) return;
    const float* pos = reinterpret_cast<const float*>(ph.pos);
    if (frame.bits <= 10) order_points<uint32_t, true, false>(pos, 4, n, count, frame, scratch, tree.id, s, launches);
    else order_points<unsigned long long, true, false>(pos, 4, n, count, frame, scratch, tree.id, s, launches);
    const int lc = photon_chunk_level(n);
    k_chunks<<<(unsigned)(((32LL << lc) + 255) / 256), 256, 0, s>>>(ph, tree.id, n, lc, tp, tree.box_lo, tree.box_hi);
    int nl = 1;
    for (int bottom = lc; bottom > 0; ++nl) {
        const int top = std::max(bottom - kBoxLevels, 0);
        k_box_levels<<<1u << top, 256, 0, s>>>(top, bottom, tree.box_lo, tree.box_hi);
        bottom = top;
    }
    if (launches) *launches += nl;
}

}  // namespace rc
