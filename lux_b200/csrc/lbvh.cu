// LBVH construction and refit for sm_100a.
//
// Pipeline (one stream, no host synchronisation):
//   1. k_root_reduce   per-primitive boxes -> union (order-free atomics on ordered ints)
//   2. k_morton_hist   30-/63-bit Morton code of each box centroid, and the digit
//                      histograms of every sort pass from the same pass over the codes
//   3. radix sort      stable LSD sort of (code, input index), 8-bit digits: one
//                      k_onesweep launch per digit (local ranking, then the tile's digit
//                      offsets by a decoupled look-back over the earlier tiles)
//   4. k_climb         leaf boxes + triangle records in sorted order, then one bottom-up
//                      climb per leaf through the binary radix tree of the codes (Karras's
//                      hierarchy and node numbers), each node written once with both its
//                      child boxes: within a block's own leaves through shared memory
//      k_climb_top     the levels above the blocks, through global memory
//      k_build_small   1 to 3 in one block for few primitives, all of it for fewer
// A refit (k_refit) climbs the known hierarchy with new geometry.
//
// Reference counterparts (src/): bvh/gpu_bvh.cu:135-149 (codes), 582-584 (sort),
// 151-180 (hierarchy), 182-214 (bottom-up boxes), 535-613 (build/refit drivers);
// bvh/cpu_lbvh_builder.h:163-259 (the host builder the results are bit-exact with).
// The reference's separate subtree-size, preorder and escape passes (gpu_bvh.cu:216-363)
// have no counterpart: traversal walks the Karras nodes directly.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "../../include/lux_gpu.h"
#include "lux_internal.h"

namespace lux {
namespace {

// Launch shapes; the LUX_* macros exist so that other shapes can be built and timed
// against these defaults (results do not depend on them).
#ifndef LUX_CLIMB_THREADS
#define LUX_CLIMB_THREADS 256
#endif
#ifndef LUX_CLIMB_BLOCKS
#define LUX_CLIMB_BLOCKS 6
#endif
#ifndef LUX_LOOKBACK_BATCH
#define LUX_LOOKBACK_BATCH 8
#endif
#ifndef LUX_SORT_THREADS
#define LUX_SORT_THREADS 512
#endif

constexpr int kThreads = 256;
constexpr int kRadix = 256;
constexpr int kSortThreads = LUX_SORT_THREADS;      // threads of a k_onesweep block
// The allocation-free sort's tiles (its scratch size is part of the ABI): fixed.
constexpr int kStaticItems = 16;
constexpr int kStaticTile = kThreads * kStaticItems;
constexpr int kScanThreads = 1024;
constexpr int kClimbBound = 160;                 // > max tree depth (64 + 96 bits)
constexpr int kMaxPasses = 8;                    // 8-bit digits of a 63-bit key
constexpr int kClimbThreads = LUX_CLIMB_THREADS; // leaves per climb block
constexpr long long kLookbackSpins = 1ll << 22;  // bound of one look-back wait

// Relaxed device-scope accesses of the look-back words (each word carries its own value,
// so no other ordering is needed) and an acquire-release add for the climb's flags.
LUX_D unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
LUX_D void st_relaxed(unsigned* p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
LUX_D unsigned atomic_add_acq_rel(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
                 : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

LUX_D unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <int Kind>
LUX_D void load_prim(const float* prims, int i, f3& v0, f3& v1, f3& v2, box3& b) {
    if (Kind == LUX_PRIM_TRIANGLES) {
        const float* t = prims + static_cast<size_t>(i) * 9;
        v0 = make_f3(t[0], t[1], t[2]);
        v1 = make_f3(t[3], t[4], t[5]);
        v2 = make_f3(t[6], t[7], t[8]);
        b = triangle_box(v0, v1, v2);
    } else {
        const float* t = prims + static_cast<size_t>(i) * 6;
        b = box3{make_f3(t[0], t[1], t[2]), make_f3(t[3], t[4], t[5])};
        v0 = v1 = v2 = make_f3(0, 0, 0);
    }
}

// load_prim through 16-byte loads: the aligned window of three float4 (triangles, 36 B at
// any 4-byte offset) or two (boxes, 24 B at an 8-byte offset) that holds the primitive,
// the primitive's floats then selected from it.  Three load instructions instead of nine
// (two instead of six), each lane's bytes in at most three sectors.  Used when the
// buffer is 16-byte aligned and the window ends inside it; the scalar loads otherwise.
template <int Kind>
LUX_D void load_prim_vec(const float* prims, int n, int i, bool aligned, f3& v0, f3& v1,
                         f3& v2, box3& b) {
    constexpr int kFloats = Kind == LUX_PRIM_TRIANGLES ? 9 : 6;
    constexpr int kWindow = Kind == LUX_PRIM_TRIANGLES ? 12 : 8;
    const size_t off = static_cast<size_t>(i) * kFloats;
    const size_t base = off & ~size_t(3);
    if (!aligned || base + kWindow > static_cast<size_t>(n) * kFloats) {
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        return;
    }
    const int r = static_cast<int>(off & 3);
    const float4* p = reinterpret_cast<const float4*>(prims + base);
    float w[kWindow];
#pragma unroll
    for (int q = 0; q < kWindow / 4; ++q) {
        const float4 x = __ldg(p + q);
        w[4 * q] = x.x; w[4 * q + 1] = x.y; w[4 * q + 2] = x.z; w[4 * q + 3] = x.w;
    }
    float t[kFloats];
#pragma unroll
    for (int j = 0; j < kFloats; ++j) {
        if (Kind == LUX_PRIM_TRIANGLES)
            t[j] = r == 0 ? w[j] : r == 1 ? w[j + 1] : r == 2 ? w[j + 2] : w[j + 3];
        else
            t[j] = r == 0 ? w[j] : w[j + 2];
    }
    if (Kind == LUX_PRIM_TRIANGLES) {
        v0 = make_f3(t[0], t[1], t[2]);
        v1 = make_f3(t[3], t[4], t[5]);
        v2 = make_f3(t[6], t[7], t[8]);
        b = triangle_box(v0, v1, v2);
    } else {
        b = box3{make_f3(t[0], t[1], t[2]), make_f3(t[3], t[4], t[5])};
        v0 = v1 = v2 = make_f3(0, 0, 0);
    }
}

LUX_D bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---------------------------------------------------------------- 1. root box

template <int Kind>
__global__ void __launch_bounds__(kThreads) k_root_reduce(const float* prims, int n,
                                                          unsigned* root_ord) {
    float lo[3] = {INFINITY, INFINITY, INFINITY};
    float hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        lo[0] = fminf(lo[0], b.lo.x); lo[1] = fminf(lo[1], b.lo.y); lo[2] = fminf(lo[2], b.lo.z);
        hi[0] = fmaxf(hi[0], b.hi.x); hi[1] = fmaxf(hi[1], b.hi.y); hi[2] = fmaxf(hi[2], b.hi.z);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    // The block's warps meet in shared memory; one atomic per block and value (the
    // atomics of every warp on six words serialised in L2).
    __shared__ float part[kThreads / 32][6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            part[warp][a] = lo[a];
            part[warp][3 + a] = hi[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int a = threadIdx.x;
        float v = part[0][a];
        for (int w = 1; w < kThreads / 32; ++w) v = a < 3 ? fminf(v, part[w][a]) : fmaxf(v, part[w][a]);
        // Maxima of ordered integers (of the complement for the lower corner): zero is their
        // identity.
        atomicMax(root_ord + a, a < 3 ? ~float_to_ordered(v) : float_to_ordered(v));
    }
}

LUX_D box3 decode_root(const unsigned* root_ord) {
    return box3{make_f3(ordered_to_float(~root_ord[0]), ordered_to_float(~root_ord[1]),
                        ordered_to_float(~root_ord[2])),
                make_f3(ordered_to_float(root_ord[3]), ordered_to_float(root_ord[4]),
                        ordered_to_float(root_ord[5]))};
}

// ---------------------------------------------------------------- 2. Morton codes

template <int Kind, typename Key>
__global__ void __launch_bounds__(kThreads) k_morton(const float* prims, int n,
                                                     const unsigned* root_ord, Key* codes) {
    box3 root = decode_root(root_ord);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        if (sizeof(Key) == 4) {
            codes[i] = static_cast<Key>(morton30(b, root));
        } else {
            codes[i] = static_cast<Key>(morton63(b, root));
        }
    }
}

// ---------------------------------------------------------------- 3. radix sort

template <typename Key>
LUX_D unsigned digit_of(Key k, int shift) {
    return static_cast<unsigned>(k >> shift) & (kRadix - 1);
}

// Morton codes (as k_morton) plus, for every sort pass p, the count of each 8-bit digit
// of the codes: hist[p * kRadix + d], accumulated in shared memory (one copy per warp
// for 30-bit keys, two for the 63-bit keys' eight passes, to stay within 48 KB) and added
// to the global counts once per block.
template <int Kind, typename Key, int Passes>
__global__ void __launch_bounds__(kThreads) k_morton_hist(const float* prims, int n,
                                                          const unsigned* root_ord,
                                                          Key* codes, unsigned* hist) {
    constexpr int kCopies = Passes <= 4 ? kThreads / 32 : 2;
    __shared__ unsigned h[kCopies][Passes][kRadix];
    for (int i = threadIdx.x; i < kCopies * Passes * kRadix; i += kThreads) (&h[0][0][0])[i] = 0;
    __syncthreads();
    const int warp = (threadIdx.x >> 5) % kCopies;
    box3 root = decode_root(root_ord);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        Key c = sizeof(Key) == 4 ? static_cast<Key>(morton30(b, root))
                                 : static_cast<Key>(morton63(b, root));
        codes[i] = c;
#pragma unroll
        for (int p = 0; p < Passes; ++p) atomicAdd(&h[warp][p][digit_of(c, 8 * p)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < Passes * kRadix; i += kThreads) {
        unsigned v = 0;
#pragma unroll
        for (int w = 0; w < kCopies; ++w) v += (&h[w][0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
}

// Lanes of the warp whose digit (and validity) equal this lane's: a validity ballot and
// one ballot per digit bit, ANDed (cheaper than a general match on sm_100a).
LUX_D unsigned digit_peers(unsigned d, bool valid) {
    unsigned peers = __ballot_sync(0xffffffffu, valid);
    if (!valid) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Look-back words, 32 bits: 0 while not yet published; kTileAggregate | this tile's own
// count (at most the tile's keys); kTilePrefix | the count over tiles 0..t (at most 2^30, the
// primitive limit, so it fits below the flag bit).
constexpr unsigned kTileAggregate = 1u << 30;
constexpr unsigned kTilePrefix = 1u << 31;
constexpr int kLookbackBatch = LUX_LOOKBACK_BATCH;   // earlier tiles' words loaded together

// One stable LSD pass over all keys.  Tiles of kSortTile keys are taken in launch order
// (an atomic counter), ranked inside the tile as k_sort_downsweep ranks them (per-warp
// digit counts in input order, so equal digits keep input order), and placed at
// (keys of smaller digits) + (digit d's count in earlier tiles) + the rank in the tile.  The count in
// earlier tiles comes from a decoupled look-back: each tile publishes its per-digit
// count, then walks back over the earlier tiles' words until one holds an inclusive
// prefix, and publishes its own inclusive prefix.  A tile waits only on tiles that were
// handed out before it (and so are running or done); each wait is bounded and a wait
// that runs out reports through `error`.
//
// The scatter goes through shared memory: the tile's keys and values are first placed in
// digit order there, so that consecutive threads store runs of a digit at consecutive
// addresses (stored straight from the ranking order, a warp's 32 stores met 32 sectors).
template <typename Key, int Items>
constexpr int onesweep_smem() {
    return kSortThreads * Items * static_cast<int>(sizeof(Key) + sizeof(int));
}

template <typename Key, bool First, int kSortItems>
__global__ void __launch_bounds__(kSortThreads) k_onesweep(const Key* keys_in,
                                                           const int* vals_in, Key* keys_out,
                                                           int* vals_out, int n, int shift,
                                                           const unsigned* hist,
                                                           unsigned* lookback,
                                                           unsigned* tile_counter, int* error) {
    static_assert(kSortThreads >= kRadix, "one thread per digit in the look-back");
    constexpr int kSortTile = kSortThreads * kSortItems;
    constexpr int kWarps = kSortThreads / 32;
    constexpr int kWarpSpan = kSortTile / kWarps;
    extern __shared__ __align__(16) unsigned char sort_smem[];
    Key* skeys = reinterpret_cast<Key*>(sort_smem);
    int* svals = reinterpret_cast<int*>(skeys + kSortTile);
    __shared__ unsigned wcount[kWarps][kRadix];
    __shared__ unsigned loff[kRadix], gbase[kRadix];
    __shared__ uint2 warp_sums[kRadix / 32];
    __shared__ int tile_s;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) tile_s = static_cast<int>(atomicAdd(tile_counter, 1u));
    const unsigned all = threadIdx.x < kRadix ? hist[threadIdx.x] : 0u;
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kSortThreads) (&wcount[0][0])[i] = 0;
    __syncthreads();
    const int tile = tile_s;

    const unsigned lt = lanemask_lt();
    const int base = tile * kSortTile + warp * kWarpSpan;
    Key k[kSortItems];
    int v[kSortItems];
    unsigned rank[kSortItems];
    // All of the warp's keys and values are loaded before the ranking starts, so their
    // loads are in flight together rather than one per ranking round.
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        int idx = base + j * 32 + lane;
        bool valid = idx < n;
        k[j] = valid ? keys_in[idx] : Key(0);
        v[j] = First ? idx : (valid ? vals_in[idx] : 0);
    }
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        int idx = base + j * 32 + lane;
        bool valid = idx < n;
        unsigned d = valid ? digit_of(k[j], shift) : 0u;
        unsigned peers = digit_peers(d, valid);
        unsigned before = valid ? wcount[warp][d] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcount[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[j] = valid ? before + __popc(peers & lt) : 0xffffffffu;
    }
    __syncthreads();
    // Exclusive sums over the digits: of the tile's counts (the keys' places in it) and of
    // all keys' counts (the digits' places in the output).
    unsigned total = 0;
    uint2 incl = make_uint2(0, 0);
    unsigned* mine = lookback + static_cast<size_t>(tile) * kRadix + threadIdx.x;
    if (threadIdx.x < kRadix) {
        const int d = threadIdx.x;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            unsigned c = wcount[w][d];
            wcount[w][d] = total;
            total += c;
        }
        st_relaxed(mine, tile == 0 ? kTilePrefix | total : kTileAggregate | total);
        incl = make_uint2(total, all);
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned x = __shfl_up_sync(0xffffffffu, incl.x, off);
            const unsigned y = __shfl_up_sync(0xffffffffu, incl.y, off);
            if (lane >= off) {
                incl.x += x;
                incl.y += y;
            }
        }
        if (lane == 31) warp_sums[warp] = incl;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
        uint2 before = make_uint2(0, 0);
        for (int w = 0; w < warp; ++w) {
            before.x += warp_sums[w].x;
            before.y += warp_sums[w].y;
        }
        loff[threadIdx.x] = before.x + incl.x - total;
        gbase[threadIdx.x] = before.y + incl.y - all;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        if (rank[j] == 0xffffffffu) continue;
        const unsigned d = digit_of(k[j], shift);
        const unsigned at = loff[d] + wcount[warp][d] + rank[j];   // < the tile's keys
        skeys[at] = k[j];
        svals[at] = v[j];
    }
    if (threadIdx.x < kRadix) {
        const int d = threadIdx.x;
        unsigned prefix = 0;
        if (tile > 0) {
            // Walk back kLookbackBatch tiles at a time (their words are loaded together,
            // so a run of aggregates costs one load latency per batch): take every
            // published word up to the nearest inclusive prefix, and re-read from the
            // first word not yet published.
            int t = tile - 1;
            long long spins = 0;
            bool found = false;
            while (!found && t >= 0) {
                unsigned w[kLookbackBatch];
#pragma unroll
                for (int j = 0; j < kLookbackBatch; ++j)
                    w[j] = t - j >= 0 ? ld_relaxed(lookback + static_cast<size_t>(t - j) * kRadix + d)
                                      : 0u;
                int taken = 0;
                bool blocked = false;
#pragma unroll
                for (int j = 0; j < kLookbackBatch; ++j) {
                    if (found || blocked || t - j < 0) continue;
                    if (w[j] == 0) {          // not published yet: resume at this tile
                        blocked = true;
                        continue;
                    }
                    found = (w[j] & kTilePrefix) != 0;
                    prefix += w[j] & (found ? ~kTilePrefix : ~kTileAggregate);
                    taken = j + 1;
                }
                t -= taken;
                if (blocked && ++spins > kLookbackSpins) {
                    atomicOr(error, kErrLoopBound);
                    break;
                }
            }
            st_relaxed(mine, kTilePrefix | (prefix + total));
        }
        gbase[d] += prefix - loff[d];
    }
    __syncthreads();
    const int count = min(kSortTile, n - tile * kSortTile);
    for (int j = threadIdx.x; j < count; j += kSortThreads) {
        const Key key = skeys[j];
        const unsigned pos = gbase[digit_of(key, shift)] + j;
        if (pos >= static_cast<unsigned>(n)) {  // cannot happen for consistent counts
            atomicOr(error, kErrLoopBound);
            continue;
        }
        keys_out[pos] = key;
        vals_out[pos] = svals[j];
    }
}

// Per-tile digit counts, stored digit-major: hist[d * tiles + tile].
template <typename Key>
__global__ void __launch_bounds__(kThreads) k_sort_upsweep(const Key* keys, int n, int shift,
                                                           unsigned* hist, int tiles) {
    __shared__ unsigned counts[kRadix];
    counts[threadIdx.x] = 0;
    __syncthreads();
    int base = blockIdx.x * kStaticTile;
#pragma unroll 4
    for (int j = 0; j < kStaticItems; ++j) {
        int idx = base + j * kThreads + threadIdx.x;
        bool valid = idx < n;
        unsigned d = valid ? digit_of(keys[idx], shift) : kRadix;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        if (valid && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&counts[d], __popc(peers));
    }
    __syncthreads();
    hist[threadIdx.x * tiles + blockIdx.x] = counts[threadIdx.x];
}

// Exclusive scan of `count` words in place, one block.  count is a multiple of 4 and
// data 16-byte aligned: each pass covers 4096 words with one coalesced uint4 per
// thread, a warp-shuffle scan of the per-thread sums and a carry into the next pass.
__global__ void __launch_bounds__(kScanThreads) k_scan_exclusive(unsigned* data, int count) {
    constexpr int kWarps = kScanThreads / 32;
    __shared__ unsigned warp_sums[kWarps];
    __shared__ unsigned carry_s;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry_s = 0;
    uint4* data4 = reinterpret_cast<uint4*>(data);
    const int count4 = count >> 2;
    for (int base = 0; base < count4; base += kScanThreads) {
        int i = base + threadIdx.x;
        uint4 v = i < count4 ? data4[i] : make_uint4(0, 0, 0, 0);
        unsigned s = v.x + v.y + v.z + v.w;
        unsigned incl = s;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            unsigned o = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += o;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            unsigned w = warp_sums[lane];
            unsigned wi = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                unsigned o = __shfl_up_sync(0xffffffffu, wi, off);
                if (lane >= off) wi += o;
            }
            warp_sums[lane] = wi - w;  // exclusive prefix of warp totals
        }
        __syncthreads();
        unsigned carry = carry_s;
        unsigned run = carry + warp_sums[warp] + incl - s;
        if (i < count4) {
            uint4 o;
            o.x = run;
            o.y = run + v.x;
            o.z = o.y + v.y;
            o.w = o.z + v.z;
            data4[i] = o;
        }
        __syncthreads();
        if (threadIdx.x == kScanThreads - 1) carry_s = run + s;
        __syncthreads();
    }
}

// Stable scatter of one tile.  Warp w owns tile keys [w*512, w*512+512), visited in
// rounds of 32 consecutive keys; a key's rank is (count of its digit in this warp's
// earlier rounds) + (peers with the same digit in lower lanes), then offset by the same
// digit's counts in earlier warps and earlier tiles, so equal digits keep input order.
template <typename Key, bool First>
__global__ void __launch_bounds__(kThreads) k_sort_downsweep(const Key* keys_in,
                                                             const int* vals_in, Key* keys_out,
                                                             int* vals_out, int n, int shift,
                                                             const unsigned* scanned,
                                                             int tiles, int* error) {
    constexpr int kWarps = kThreads / 32;
    constexpr int kWarpSpan = kStaticTile / kWarps;
    __shared__ unsigned wcount[kWarps][kRadix];
    __shared__ unsigned gbase[kRadix];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kWarps * kRadix; i += kThreads) (&wcount[0][0])[i] = 0;
    gbase[threadIdx.x] = scanned[threadIdx.x * tiles + blockIdx.x];
    __syncthreads();

    const unsigned lt = lanemask_lt();
    const int base = blockIdx.x * kStaticTile + warp * kWarpSpan;
    Key k[kStaticItems];
    int v[kStaticItems];
    unsigned rank[kStaticItems];
#pragma unroll
    for (int j = 0; j < kStaticItems; ++j) {
        int idx = base + j * 32 + lane;
        bool valid = idx < n;
        k[j] = valid ? keys_in[idx] : Key(0);
        v[j] = First ? idx : (valid ? vals_in[idx] : 0);
        unsigned d = valid ? digit_of(k[j], shift) : kRadix;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        unsigned before = valid ? wcount[warp][d] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcount[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[j] = valid ? before + __popc(peers & lt) : 0xffffffffu;
    }
    __syncthreads();
    {
        unsigned run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            unsigned c = wcount[w][threadIdx.x];
            wcount[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kStaticItems; ++j) {
        if (rank[j] == 0xffffffffu) continue;
        unsigned d = digit_of(k[j], shift);
        unsigned pos = gbase[d] + wcount[warp][d] + rank[j];
        if (pos >= static_cast<unsigned>(n)) {  // cannot happen for a consistent histogram
            atomicOr(error, kErrLoopBound);
            continue;
        }
        keys_out[pos] = k[j];
        vals_out[pos] = v[j];
    }
}

// ---------------------------------------------------------------- 4. Karras hierarchy

LUX_D int clz64(unsigned long long x) { return __clzll(static_cast<long long>(x)); }

// Common-prefix length of sorted keys i and j.  30-bit codes: the reference's merged
// key (code << 32) | index (bvh/gpu_bvh.cu:66-74).  63-bit codes: the code prefix, and
// the index prefix beyond it when the codes are equal.
template <typename Key>
LUX_D int delta(const Key* codes, int i, int j) {
    if (sizeof(Key) == 4) {
        unsigned long long ki = (static_cast<unsigned long long>(codes[i]) << 32) | unsigned(i);
        unsigned long long kj = (static_cast<unsigned long long>(codes[j]) << 32) | unsigned(j);
        return clz64(ki ^ kj);
    } else {
        unsigned long long x = static_cast<unsigned long long>(codes[i] ^ codes[j]);
        if (x) return clz64(x);
        return 64 + __clz(static_cast<int>(unsigned(i) ^ unsigned(j)));
    }
}

// One subtree on its way up: its box, its sorted leaves [first, last], and the common
// prefix lengths with the neighbours outside it (-1 at the ends of the array).
struct Subtree {
    box3 b;
    int first, last;
    int dl, dr;
    // The parent splits its range after this leaf: the subtree joins the neighbour it shares
    // more bits with (the two lengths never agree: the keys with their indices are distinct).
    LUX_D bool is_left() const { return dr > dl; }
    LUX_D bool is_root() const { return dl < 0 && dr < 0; }
    // Karras node number: a left child is numbered by its last leaf, a right child by its
    // first, the root 0 (bvh/gpu_bvh.cu:151-180 numbers its nodes so).
    LUX_D int id() const { return is_root() ? 0 : is_left() ? last : first; }
};

// Joins left = [.., s] and right = [s + 1, ..] and writes the new node's record and its
// children's parent links.  ch.z, ch.w of the record: the other end of its leaves and, until
// the node is joined itself, the prefix length beyond it, which the sibling that meets this
// node in global memory reads; then its parent link (-1 for the root, as its prefix length).
LUX_D Subtree join(const Subtree& left, const Subtree& right, BvhNode* nodes, int* leaf_parent) {
    Subtree t;
    t.b = box_union(left.b, right.b);
    t.first = left.first;
    t.last = right.last;
    t.dl = left.dl;
    t.dr = right.dr;
    const int id = t.id(), s = left.last;
    const bool ll = left.first == left.last, rl = right.first == right.last;
    const box3 &l = left.b, &r = right.b;
    const bool side = t.is_left();
    float4* o = reinterpret_cast<float4*>(nodes + id);
    stg8(o, make_float4(l.lo.x, l.lo.y, l.lo.z, l.hi.x),
         make_float4(l.hi.y, l.hi.z, r.lo.x, r.lo.y));
    stg8(o + 2, make_float4(r.lo.z, r.hi.x, r.hi.y, r.hi.z),
         make_float4(__int_as_float(ll ? ~s : s), __int_as_float(rl ? ~(s + 1) : s + 1),
                     __int_as_float(side ? t.first : t.last),
                     __int_as_float(side ? t.dl : t.dr)));
    *(ll ? leaf_parent + s : &nodes[s].ch.w) = id << 1;
    *(rl ? leaf_parent + s + 1 : &nodes[s + 1].ch.w) = (id << 1) | 1;
    return t;
}

LUX_D void store_root(float* root, const box3& b) {
    root[0] = b.lo.x; root[1] = b.lo.y; root[2] = b.lo.z;
    root[3] = b.hi.x; root[4] = b.hi.y; root[5] = b.hi.z;
}

// Few primitives, by one block: scene box, Morton codes and their stable sort with the keys
// and (16-bit) input indices in shared memory over all passes; and, up to kWholeBuild, the
// hierarchy too (Whole).  A chain of kernels over so few keys is launch, look-back and atomic
// latency and nothing else: the chain took 33 us for 257 triangles, 38 us for 1,000 and 49 us
// for 2,000, the whole build by one block takes 16, 28 and 46 us.  It climbs with one SM's
// issue slots, 18 us per 1,024 leaves, so beyond that k_climb's many blocks are faster (4,000
// triangles: 61 against 84 us), and one SM's sort is faster than the chain of sort kernels up
// to kSmallSort (4,000: 61 against 67 us, with 63-bit codes 76 against 99; 6,144: 74 against
// 74, 96 against 104).
constexpr int kWholeBuild = 2048;
constexpr int kSmallSort = 6144;
constexpr int kSmallThreads = 1024;

template <typename Key, bool Whole>
constexpr int small_build_smem() {
    constexpr int kMax = Whole ? kWholeBuild : kSmallSort;
    const int sort = 2 * kMax * static_cast<int>(sizeof(Key) + sizeof(unsigned short)) +
                     (kSmallThreads / 32) * kRadix * static_cast<int>(sizeof(unsigned));
    const int climb = kWholeBuild * static_cast<int>(6 * sizeof(float) + sizeof(unsigned) +
                                                     sizeof(unsigned short));
    return sort > climb || !Whole ? sort : climb;
}

template <int Kind, typename Key, bool Whole>
__global__ void __launch_bounds__(kSmallThreads) k_build_small(
        const float* prims, int n, Key* codes, int* sorted_ids, TriRecord* tris, BvhNode* nodes,
        int* leaf_parent, float* root_box) {
    constexpr int kWarps = kSmallThreads / 32;
    constexpr int kPasses = sizeof(Key) == 4 ? 4 : 8;
    constexpr int kMax = Whole ? kWholeBuild : kSmallSort;
    constexpr int kEach = kMax / kSmallThreads;
    extern __shared__ __align__(16) unsigned char small_smem[];
    Key* keys[2];
    unsigned short* ids[2];
    keys[0] = reinterpret_cast<Key*>(small_smem);
    keys[1] = keys[0] + kMax;
    unsigned (*wcount)[kRadix] = reinterpret_cast<unsigned (*)[kRadix]>(keys[1] + kMax);
    ids[0] = reinterpret_cast<unsigned short*>(wcount + kWarps);
    ids[1] = ids[0] + kMax;
    __shared__ float part[kWarps][6];
    __shared__ unsigned loff[kRadix], warp_sums[kRadix / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The scene box (min and max are order-free).
    float lo[3] = {INFINITY, INFINITY, INFINITY};
    float hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        lo[0] = fminf(lo[0], b.lo.x); lo[1] = fminf(lo[1], b.lo.y); lo[2] = fminf(lo[2], b.lo.z);
        hi[0] = fmaxf(hi[0], b.hi.x); hi[1] = fmaxf(hi[1], b.hi.y); hi[2] = fmaxf(hi[2], b.hi.z);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            part[warp][a] = lo[a];
            part[warp][3 + a] = hi[a];
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = part[lane][a];
        hi[a] = part[lane][3 + a];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    const box3 root{make_f3(lo[0], lo[1], lo[2]), make_f3(hi[0], hi[1], hi[2])};
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, i, v0, v1, v2, b);
        keys[0][i] = sizeof(Key) == 4 ? static_cast<Key>(morton30(b, root))
                                      : static_cast<Key>(morton63(b, root));
        ids[0][i] = static_cast<unsigned short>(i);
    }
    // Each warp ranks a run of `rounds` * 32 consecutive keys, as k_onesweep's warps do.
    const unsigned lt = lanemask_lt();
    const int rounds = (n + kSmallThreads - 1) / kSmallThreads;
    const int base = warp * rounds * 32;
    int cur = 0;
    for (int p = 0; p < kPasses; ++p) {
        const int shift = 8 * p;
        for (int i = threadIdx.x; i < kWarps * kRadix; i += kSmallThreads) (&wcount[0][0])[i] = 0;
        __syncthreads();
        unsigned rank[kEach];
#pragma unroll
        for (int j = 0; j < kEach; ++j) {
            if (j >= rounds) break;
            const int idx = base + j * 32 + lane;
            const bool valid = idx < n;
            const unsigned d = valid ? digit_of(keys[cur][idx], shift) : 0u;
            const unsigned peers = digit_peers(d, valid);
            const unsigned before = valid ? wcount[warp][d] : 0u;
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) wcount[warp][d] = before + __popc(peers);
            __syncwarp();
            rank[j] = before + __popc(peers & lt);
        }
        __syncthreads();
        unsigned total = 0, incl = 0;
        if (threadIdx.x < kRadix) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const unsigned c = wcount[w][threadIdx.x];
                wcount[w][threadIdx.x] = total;
                total += c;
            }
            incl = total;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned o = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += o;
            }
            if (lane == 31) warp_sums[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < kRadix) {
            unsigned before = 0;
            for (int w = 0; w < warp; ++w) before += warp_sums[w];
            loff[threadIdx.x] = before + incl - total;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kEach; ++j) {
            if (j >= rounds) break;
            const int idx = base + j * 32 + lane;
            if (idx >= n) break;
            const Key key = keys[cur][idx];
            const unsigned d = digit_of(key, shift);
            const unsigned at = loff[d] + wcount[warp][d] + rank[j];   // < n
            keys[cur ^ 1][at] = key;
            ids[cur ^ 1][at] = ids[cur][idx];
        }
        cur ^= 1;
        __syncthreads();
    }
    if (!Whole) {
        for (int i = threadIdx.x; i < n; i += kSmallThreads) {
            codes[i] = keys[cur][i];
            sorted_ids[i] = ids[cur][i];
        }
        return;
    }
    // The hierarchy, as k_climb's blocks build it, of all leaves.  What it needs of the sort
    // is kept in registers (its ids) and in place (the prefix lengths), the rest of the shared
    // memory is taken anew.
    __shared__ signed char sdelta[Whole ? kMax + 1 : 1];   // prefix length of leaves j - 1 and j
    int pid[kEach];
#pragma unroll
    for (int r = 0; r < kEach; ++r) {
        const int k = r * kSmallThreads + static_cast<int>(threadIdx.x);
        pid[r] = -1;
        if (k < n) {
            pid[r] = ids[cur][k];
            codes[k] = keys[cur][k];
            sorted_ids[k] = pid[r];
            sdelta[k] = static_cast<signed char>(k > 0 ? delta(keys[cur], k - 1, k) : -1);
        }
    }
    if (threadIdx.x == 0) sdelta[n] = -1;
    __syncthreads();
    float* sbox = reinterpret_cast<float*>(small_smem);                   // [6][kMax]
    unsigned* sflag = reinterpret_cast<unsigned*>(sbox + 6 * kMax);   // per split
    unsigned short* send = reinterpret_cast<unsigned short*>(sflag + kMax);
    auto put_box = [&](int j, const box3& b) {
        sbox[j] = b.lo.x; sbox[kMax + j] = b.lo.y; sbox[2 * kMax + j] = b.lo.z;
        sbox[3 * kMax + j] = b.hi.x; sbox[4 * kMax + j] = b.hi.y;
        sbox[5 * kMax + j] = b.hi.z;
    };
    auto get_box = [&](int j) {
        return box3{make_f3(sbox[j], sbox[kMax + j], sbox[2 * kMax + j]),
                    make_f3(sbox[3 * kMax + j], sbox[4 * kMax + j],
                            sbox[5 * kMax + j])};
    };
#pragma unroll
    for (int r = 0; r < kEach; ++r) {
        const int k = r * kSmallThreads + static_cast<int>(threadIdx.x);
        if (pid[r] < 0) continue;
        f3 v0, v1, v2;
        box3 b;
        load_prim<Kind>(prims, pid[r], v0, v1, v2, b);
        if (Kind == LUX_PRIM_TRIANGLES) {
            TriRecord t;
            t.p0 = make_float4(v0.x, v0.y, v0.z, __int_as_float(pid[r]));
            t.p1 = make_float4(v1.x, v1.y, v1.z, 0.0f);
            t.p2 = make_float4(v2.x, v2.y, v2.z, 0.0f);
            tris[k] = t;
        }
        put_box(k, b);
        send[k] = static_cast<unsigned short>(k);
        sflag[k] = 0;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = threadIdx.x; k < n; k += kSmallThreads) {
        Subtree t;
        t.b = get_box(k);
        t.first = t.last = k;
        t.dl = sdelta[k];
        t.dr = sdelta[k + 1];
        for (;;) {   // at most n - 1 joins in all
            if (t.is_root()) {
                store_root(root_box, t.b);
                break;
            }
            const bool left = t.is_left();
            const int s = left ? t.last : t.first - 1;
            const int own = left ? s : s + 1, sib = left ? s + 1 : s;
            if (t.first != t.last) {
                put_box(own, t.b);
                send[own] = static_cast<unsigned short>(left ? t.first : t.last);
            }
            __threadfence_block();
            if (atomicAdd(&sflag[s], 1u) == 0) break;   // the sibling joins them
            __threadfence_block();
            Subtree o;
            o.b = get_box(sib);
            o.first = left ? sib : send[sib];
            o.last = left ? send[sib] : sib;
            o.dl = left ? t.dr : sdelta[o.first];
            o.dr = left ? sdelta[o.last + 1] : t.dl;
            t = left ? join(t, o, nodes, leaf_parent) : join(o, t, nodes, leaf_parent);
        }
    }
}

// Hierarchy and boxes in one bottom-up pass over the sorted codes, in two kernels.  The tree
// is Karras's (the binary radix tree of the codes), node numbers included, without his
// searches: the codes are read once.
//
// k_climb: one thread per sorted leaf.  The leaf's box (and, for triangles, its sorted
// record) is formed; then the thread climbs: from the prefix lengths at the two ends of its
// subtree it knows the leaf after which the parent splits, where the two children meet at a
// counter in shared memory, and the second to arrive joins them, writes the node and goes
// on.  A subtree whose sibling reaches beyond the block waits there for nobody: when the
// block has come to rest, every subtree that is left is listed for k_climb_top.
//
// Bound by latency: the gather of the primitives (one random record per leaf), then a chain
// of some tens of shared-memory steps.
template <int Kind, typename Key>
__global__ void __launch_bounds__(kClimbThreads, LUX_CLIMB_BLOCKS) k_climb(
        const float* prims, int n, const Key* codes, const int* sorted_ids, TriRecord* tris,
        BvhNode* nodes, int* leaf_parent, int2* open, int* open_count, float* root,
        int* error) {
    constexpr int T = kClimbThreads;
    // By the subtree's number within the block (a left child: its last leaf, a right child:
    // its first): box and other end.  The number is free again once the sibling has read it.
    __shared__ float sbox[6][T];
    __shared__ int send[T];
    __shared__ unsigned sflag[T];     // per split: 1 the left child arrived, 2 the right one
    __shared__ int sdelta[T + 1];     // prefix length of leaves lo + j - 1 and lo + j
    __shared__ int left_over;
    const int tid = threadIdx.x;
    const int lo = blockIdx.x * T;
    const int k = lo + tid;
    sflag[tid] = 0;
    if (tid == 0) {
        left_over = 0;
        sdelta[T] = lo + T < n ? delta(codes, lo + T - 1, lo + T) : -1;
    }
    sdelta[tid] = k > 0 && k < n ? delta(codes, k - 1, k) : -1;
    Subtree t{};
    bool climbing = k < n;
    if (climbing) {
        const int pid = sorted_ids[k];
        if (pid < 0 || pid >= n) {  // cannot happen for a consistent sort
            atomicOr(error, kErrLoopBound);
            climbing = false;
        } else {
            f3 v0, v1, v2;
            load_prim_vec<Kind>(prims, n, pid, aligned16(prims), v0, v1, v2, t.b);
            if (Kind == LUX_PRIM_TRIANGLES) {
                TriRecord r;
                r.p0 = make_float4(v0.x, v0.y, v0.z, __int_as_float(pid));
                r.p1 = make_float4(v1.x, v1.y, v1.z, 0.0f);
                r.p2 = make_float4(v2.x, v2.y, v2.z, 0.0f);
                tris[k] = r;
            }
            t.first = t.last = k;
        }
    }
    __syncthreads();
    auto leave = [&](int first, int last) {
        // Fewer than T: the subtrees are disjoint runs of the block's leaves.
        open[lo + atomicAdd(&left_over, 1)] = make_int2(first, last);
    };
    if (climbing) {
        t.dl = sdelta[tid];
        t.dr = sdelta[tid + 1];
    }
    while (climbing) {   // at most T - 1 joins in the block
        if (t.is_root()) {
            store_root(root, t.b);
            break;
        }
        const bool left = t.is_left();
        const int s = (left ? t.last : t.first - 1) - lo;   // split, within the block
        if (s < 0 || s >= T - 1) {
            leave(t.first, t.last);
            break;
        }
        const int own = left ? s : s + 1, sib = left ? s + 1 : s;
        sbox[0][own] = t.b.lo.x; sbox[1][own] = t.b.lo.y; sbox[2][own] = t.b.lo.z;
        sbox[3][own] = t.b.hi.x; sbox[4][own] = t.b.hi.y; sbox[5][own] = t.b.hi.z;
        send[own] = left ? t.first : t.last;
        // The block fences order these stores before the counter's add, and the add before
        // the sibling's values are read (they are also compiler barriers).
        __threadfence_block();
        if (atomicAdd(&sflag[s], left ? 1u : 2u) == 0) break;   // the sibling joins them
        __threadfence_block();
        Subtree o;
        o.b = box3{make_f3(sbox[0][sib], sbox[1][sib], sbox[2][sib]),
                   make_f3(sbox[3][sib], sbox[4][sib], sbox[5][sib])};
        if (left) {
            o.first = lo + s + 1;
            o.last = send[sib];
            o.dl = t.dr;
            o.dr = sdelta[o.last + 1 - lo];
            t = join(t, o, nodes, leaf_parent);
        } else {
            o.first = send[sib];
            o.last = lo + s;
            o.dl = sdelta[o.first - lo];
            o.dr = t.dl;
            t = join(o, t, nodes, leaf_parent);
        }
    }
    __syncthreads();
    const unsigned arrived = sflag[tid];   // split lo + tid: one child came, the other is outside
    if (arrived == 1u) leave(send[tid], lo + tid);
    else if (arrived == 2u) leave(lo + tid + 1, send[tid + 1]);
    __syncthreads();
    if (tid == 0) open_count[blockIdx.x] = left_over;
}

// Box of a finished subtree from what it wrote: its node's record, or its leaf.
template <int Kind>
LUX_D box3 finished_box(bool leaf, int at, const float* prims, int n, const int* sorted_ids,
                        const TriRecord* tris, const BvhNode* nodes, int4& ch) {
    box3 b;
    if (!leaf) {
        const float4* p = reinterpret_cast<const float4*>(nodes + at);
        const float4 x = __ldcg(p), y = __ldcg(p + 1), z = __ldcg(p + 2);
        ch = __ldcg(reinterpret_cast<const int4*>(p + 3));
        b = box_union(box3{make_f3(x.x, x.y, x.z), make_f3(x.w, y.x, y.y)},
                      box3{make_f3(y.z, y.w, z.x), make_f3(z.y, z.z, z.w)});
    } else if (Kind == LUX_PRIM_TRIANGLES) {
        const float4* p = reinterpret_cast<const float4*>(tris + at);
        const float4 x = __ldcg(p), y = __ldcg(p + 1), z = __ldcg(p + 2);
        b = triangle_box(make_f3(x.x, x.y, x.z), make_f3(y.x, y.y, y.z), make_f3(z.x, z.y, z.z));
    } else {
        f3 v0, v1, v2;
        load_prim<Kind>(prims, min(max(sorted_ids[at], 0), n - 1), v0, v1, v2, b);
    }
    return b;
}

// The climb above k_climb's blocks: one warp per block of leaves takes the subtrees that it
// listed.  The children of a split meet at a counter in global memory (acquire-release,
// zeroed again by the second arrival), which publishes the first one's record; the second
// reads it for the box, the other end and the prefix length there.  Some fifteen levels,
// each one atomic and one dependent load.
constexpr int kTopThreads = 256;
template <int Kind, typename Key>
__global__ void __launch_bounds__(kTopThreads) k_climb_top(
        const float* prims, int n, const Key* codes, const int* sorted_ids,
        const TriRecord* tris, BvhNode* nodes, int* leaf_parent, const int2* open,
        const int* open_count, int blocks, unsigned* flags, float* root, int* error) {
    const int block = (blockIdx.x * kTopThreads + threadIdx.x) >> 5;
    if (block >= blocks) return;
    const int count = min(open_count[block], kClimbThreads);
    for (int e = threadIdx.x & 31; e < count; e += 32) {
        const int2 range = open[block * kClimbThreads + e];
        Subtree t;
        t.first = range.x;
        t.last = range.y;
        if (t.first < 0 || t.last >= n || t.first > t.last) {  // cannot happen
            atomicOr(error, kErrLoopBound);
            return;
        }
        t.dl = t.first > 0 ? delta(codes, t.first - 1, t.first) : -1;
        t.dr = t.last + 1 < n ? delta(codes, t.last, t.last + 1) : -1;
        int4 ch;
        t.b = finished_box<Kind>(t.first == t.last, t.first == t.last ? t.first : t.id(), prims,
                                 n, sorted_ids, tris, nodes, ch);
        bool climbing = true;
        for (int level = 0; climbing; ++level) {
            const bool left = t.is_left();
            const int s = left ? t.last : t.first - 1;
            if (level >= kClimbBound || s < 0 || s >= n - 1) {   // cannot happen for sorted codes
                atomicOr(error, kErrClimbBound);
                return;
            }
            // 1: arrived, 2: and is a leaf.
            const unsigned prior = atomic_add_acq_rel(flags + s, t.first == t.last ? 3u : 1u);
            if (prior == 0) break;            // the sibling joins them
            flags[s] = 0;
            const int sib = left ? s + 1 : s;
            Subtree o;
            const bool leaf = (prior & 2u) != 0;
            o.b = finished_box<Kind>(leaf, sib, prims, n, sorted_ids, tris, nodes, ch);
            const int end = leaf ? sib : ch.z;
            if (end < 0 || end >= n) {        // cannot happen for a consistent record
                atomicOr(error, kErrClimbBound);
                return;
            }
            if (left) {
                o.first = sib;
                o.last = end;
                o.dl = t.dr;
                o.dr = !leaf ? ch.w : sib + 1 < n ? delta(codes, sib, sib + 1) : -1;
                t = join(t, o, nodes, leaf_parent);
            } else {
                o.first = end;
                o.last = sib;
                o.dl = !leaf ? ch.w : sib > 0 ? delta(codes, sib - 1, sib) : -1;
                o.dr = t.dl;
                t = join(o, t, nodes, leaf_parent);
            }
            if (t.is_root()) {
                store_root(root, t.b);
                climbing = false;
            }
        }
    }
}

LUX_D void store_slot(BvhNode* node, int slot, const box3& b) {
    float* f = reinterpret_cast<float*>(node);
    if (slot == 0) {
        __stcg(reinterpret_cast<float4*>(f), make_float4(b.lo.x, b.lo.y, b.lo.z, b.hi.x));
        __stcg(reinterpret_cast<float2*>(f + 4), make_float2(b.hi.y, b.hi.z));
    } else {
        __stcg(reinterpret_cast<float2*>(f + 6), make_float2(b.lo.x, b.lo.y));
        __stcg(reinterpret_cast<float4*>(f + 8), make_float4(b.lo.z, b.hi.x, b.hi.y, b.hi.z));
    }
}

LUX_D box3 load_slot_cg(const BvhNode* node, int slot) {
    const float* f = reinterpret_cast<const float*>(node);
    if (slot == 0) {
        float4 a = __ldcg(reinterpret_cast<const float4*>(f));
        float2 b = __ldcg(reinterpret_cast<const float2*>(f + 4));
        return box3{make_f3(a.x, a.y, a.z), make_f3(a.w, b.x, b.y)};
    }
    float2 a = __ldcg(reinterpret_cast<const float2*>(f + 6));
    float4 b = __ldcg(reinterpret_cast<const float4*>(f + 8));
    return box3{make_f3(a.x, a.y, b.x), make_f3(b.y, b.z, b.w)};
}

// Refit: one thread per sorted leaf.  The leaf box (and, for triangles, the sorted triangle
// record) is written; then the thread climbs: it hands its box to the parent, and the
// second of the two children to arrive (a counter) unions both and continues upward, so
// every node box is the union of its children's boxes (merge_bounds_kernel,
// bvh/gpu_bvh.cu:182-214).  A node whose leaf range lies inside this block's leaves
// [lo, lo + kClimbThreads) has both its children climbing in this block and an index in
// that range too (a Karras node is numbered by one end of its range), so the hand-over
// goes through shared memory; above that through the node's slot in global memory with
// an acquire-release counter, which the second arrival resets to zero.  One 16-byte load
// per level, of the last words of the node's record, gives its range and its parent link
// (from a table of their own 113 us instead of 105 for 1,048,576 triangles, and 15 us to make
// it after every build).  The topology being known, this is one kernel (105 us for 1,048,576
// triangles, 20 us for 5,000), where a build's climb and its top take 124 and 30 us.
template <int Kind>
__global__ void __launch_bounds__(kClimbThreads) k_refit(const float* prims, int n,
                                                              const int* sorted_ids,
                                                              TriRecord* tris, BvhNode* nodes,
                                                              const int* leaf_parent,
                                                              unsigned* flags, float* root,
                                                              int* error) {
    // Per node of the block: each child's box (three float2) and an arrival counter.
    __shared__ float2 sbox[kClimbThreads][2][3];
    __shared__ unsigned sflag[kClimbThreads];
    const int lo = blockIdx.x * kClimbThreads;
    sflag[threadIdx.x] = 0;
    __syncthreads();
    int k = lo + threadIdx.x;
    if (k >= n) return;
    // The leaf's id, its parent link and the parent's record are fetched before the
    // primitive, so the two dependent chains overlap.
    const int pid = sorted_ids[k];
    int code = n > 1 ? leaf_parent[k] : -1;
    int4 info = make_int4(0, 0, -1, -1);   // the last words of the parent's record
    if (code >= 0 && (code >> 1) < n - 1) info = nodes[code >> 1].ch;
    if (pid < 0 || pid >= n) {  // cannot happen for a consistent sort
        atomicOr(error, kErrLoopBound);
        return;
    }
    f3 v0, v1, v2;
    box3 b;
    load_prim_vec<Kind>(prims, n, pid, aligned16(prims), v0, v1, v2, b);
    if (Kind == LUX_PRIM_TRIANGLES) {
        TriRecord r;
        r.p0 = make_float4(v0.x, v0.y, v0.z, __int_as_float(pid));
        r.p1 = make_float4(v1.x, v1.y, v1.z, 0.0f);
        r.p2 = make_float4(v2.x, v2.y, v2.z, 0.0f);
        tris[k] = r;
    }
    if (n == 1) {
        root[0] = b.lo.x; root[1] = b.lo.y; root[2] = b.lo.z;
        root[3] = b.hi.x; root[4] = b.hi.y; root[5] = b.hi.z;
        return;
    }
    for (int level = 0; level < kClimbBound; ++level) {
        int p = code >> 1;
        int slot = code & 1;
        if (code < 0 || p >= n - 1) break;  // parent links out of range: report below
        // The grandparent's record is requested now, before the hand-over, so its load
        // overlaps this level's (for the half of the threads that go on).
        const int up = info.w;
        int4 next = make_int4(0, 0, -1, -1);
        if (up >= 0 && (up >> 1) < n - 1) next = nodes[up >> 1].ch;
        // Both ends of the node's leaves: its number and ch.z.
        const int s = p - lo, other = info.z - lo;
        if (s >= 0 && s < kClimbThreads && other >= 0 && other < kClimbThreads) {
            // The block fences order the box's stores before the counter's add, and the
            // add before the sibling's box is read (they are also compiler barriers).
            float2* mine = &sbox[s][slot][0];
            mine[0] = make_float2(b.lo.x, b.lo.y);
            mine[1] = make_float2(b.lo.z, b.hi.x);
            mine[2] = make_float2(b.hi.y, b.hi.z);
            __threadfence_block();
            unsigned prior = atomicAdd(&sflag[s], 1u);
            if (prior == 0) return;  // the sibling finishes this node
            __threadfence_block();
            const float2* o = &sbox[s][slot ^ 1][0];
            const float2 o0 = o[0], o1 = o[1], o2 = o[2];
            box3 sib{make_f3(o0.x, o0.y, o1.x), make_f3(o1.y, o2.x, o2.y)};
            const box3 left = slot ? sib : b;
            const box3 right = slot ? b : sib;
            store_slot(nodes + p, 0, left);
            store_slot(nodes + p, 1, right);
            b = box_union(left, right);
        } else {
            store_slot(nodes + p, slot, b);
            unsigned prior = atomic_add_acq_rel(flags + p, 1u);
            if (prior == 0) return;  // the sibling finishes this node
            flags[p] = 0;
            box3 sib = load_slot_cg(nodes + p, slot ^ 1);
            b = slot ? box_union(sib, b) : box_union(b, sib);
        }
        if (p == 0) {
            root[0] = b.lo.x; root[1] = b.lo.y; root[2] = b.lo.z;
            root[3] = b.hi.x; root[4] = b.hi.y; root[5] = b.hi.z;
            return;
        }
        code = up;
        info = next;
    }
    atomicOr(error, kErrClimbBound);
}

// ---------------------------------------------------------------- export

// Host tree layout (bvh/cpu_bvh.h:15-32): internal i, then leaf k at n-1+k.
template <typename Key>
__global__ void k_export(BvhView v, const Key* codes, unsigned long long* codes64, int* left,
                         int* right, float* bounds) {
    int n = v.n;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && codes64) codes64[i] = static_cast<unsigned long long>(codes[i]);
    if (i >= 2 * n - 1) return;
    box3 b;
    int l = -1, r = -1;
    if (i < n - 1) {
        BvhNode nd = load_node(v.nodes, i);
        b = box_union(node_left_box(nd), node_right_box(nd));
        l = nd.ch.x < 0 ? n - 1 + ~nd.ch.x : nd.ch.x;
        r = nd.ch.y < 0 ? n - 1 + ~nd.ch.y : nd.ch.y;
    } else {
        b = leaf_box(v, i - (n - 1));
    }
    if (left) left[i] = l;
    if (right) right[i] = r;
    if (bounds) {
        float* o = bounds + static_cast<size_t>(i) * 6;
        o[0] = b.lo.x; o[1] = b.lo.y; o[2] = b.lo.z;
        o[3] = b.hi.x; o[4] = b.hi.y; o[5] = b.hi.z;
    }
}

int grid_for(int count, int threads = kThreads) { return (count + threads - 1) / threads; }

// Launches one kernel of the build chain on ctx's stream and counts it.
template <typename... Params, typename... Args>
cudaError_t chain_launch(lux_ctx* ctx, void (*kernel)(Params...), int grid, int block,
                         size_t smem, Args... args) {
    ctx->launches += 1;
    kernel<<<grid, block, smem, ctx->stream>>>(static_cast<Params>(args)...);
    return cudaGetLastError();
}

int stride_grid(const lux_ctx* ctx, int count) {
    return std::max(1, std::min(grid_for(count), ctx->sm_count * 8));
}

// More than 48 KB of dynamic shared memory has to be asked for, once per device and kernel
// (asking again changes nothing, so calls from several threads are harmless).
template <typename Kernel>
cudaError_t allow_smem(Kernel kernel, int bytes) {
    if (bytes <= 24 * 1024) return cudaSuccess;   // with the static part within 48 KB
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Device scratch of a build: the sort's alternate keys and values; then the words that start
// at zero (the scene box's ordered words, every pass's digit counts, the tile counters and
// the look-back words).
struct SortScratch {
    size_t key_bytes, val_bytes, zero_bytes, lookback_bytes;
    size_t total() const { return key_bytes + val_bytes + zero_bytes + lookback_bytes; }
    // Word offsets within the zeroed part.
    static constexpr int kRoot = 0, kCounters = 8, kHist = 64;
    static constexpr int kLookback = kHist + kMaxPasses * kRadix;
};

// Keys per thread of a k_onesweep block: the more the fewer tiles look back, but the longer
// each tile's chain of ranking rounds.  Builds with 4, 8 and 16 keys a thread, in us, of 30-bit
// codes: 262,144 triangles 118, 118, 134; 393,216 139, 139, 147; 524,288 158, 150, 160; 1,048,576
// 235, 219, 218; 1,310,720 276, 266, 270; 4,194,304 722, 681, 696; of 63-bit codes: 262,144 159,
// 176, 198; 393,216 188, 189, 217; 524,288 219, 205, 235; 1,048,576 337, 296, 302; 4,194,304 1035,
// 897, 941.
constexpr int kFewKeys = 3 << 17;
int sort_items(int n) {
#ifdef LUX_SORT_ITEMS
    return LUX_SORT_ITEMS;
#endif
    return n > kFewKeys ? 8 : 4;
}

SortScratch sort_scratch(int n, size_t key_size, int passes) {
    // Tiles of any count up to n (a smaller one may take smaller tiles), so that a rebuild of
    // fewer primitives never needs more room.
    size_t tiles = 0;
    for (int m : {n, std::min(n, kFewKeys)}) {
        const int tile = kSortThreads * sort_items(m);
        tiles = std::max(tiles, static_cast<size_t>((m + tile - 1) / tile));
    }
    SortScratch s;
    s.key_bytes = (static_cast<size_t>(n) * key_size + 255) & ~size_t(255);
    s.val_bytes = (static_cast<size_t>(n) * sizeof(int) + 255) & ~size_t(255);
    s.zero_bytes = sizeof(unsigned) * SortScratch::kLookback;
    s.lookback_bytes = sizeof(unsigned) * kRadix * tiles * passes;
    return s;
}

// Morton codes of the primitives into `codes` and their stable sort with the input
// indices into (codes, vals): k_morton_hist, then one k_onesweep per
// 8-bit digit (an even count, so the result lands back in the caller's arrays).
template <int Kind, typename Key>
int morton_and_sort(lux_ctx* ctx, const float* prims, Key* codes, int* vals, int n) {
    constexpr int kPasses = sizeof(Key) == 4 ? 4 : 8;   // 30 bits: 4 digits; 63 bits: 8
    const int items = sort_items(n);
    const int tiles = grid_for(n, kSortThreads * items);
    const SortScratch layout = sort_scratch(n, sizeof(Key), kPasses);
    int st = ensure_scratch(ctx, layout.total());
    if (st) return st;
    char* s = static_cast<char*>(ctx->scratch);
    Key* keys_alt = reinterpret_cast<Key*>(s);
    int* vals_alt = reinterpret_cast<int*>(s + layout.key_bytes);
    unsigned* zeroed = reinterpret_cast<unsigned*>(s + layout.key_bytes + layout.val_bytes);
    const unsigned* root_ord = zeroed + SortScratch::kRoot;
    unsigned* hist = zeroed + SortScratch::kHist;
    unsigned* counters = zeroed + SortScratch::kCounters;
    unsigned* lookback = zeroed + SortScratch::kLookback;
    // Counts, tile counters and look-back words start at zero (reset by the caller
    // before the chain's first kernel, reset_sort_scratch).
    const int hist_grid = std::max(1, std::min(grid_for(n), ctx->sm_count * 2));
    cudaError_t err = chain_launch(ctx, k_morton_hist<Kind, Key, kPasses>, hist_grid, kThreads,
                                   0, prims, n, root_ord, codes, hist);
    Key* kin = codes;
    int* vin = vals;
    Key* kout = keys_alt;
    int* vout = vals_alt;
    for (int p = 0; p < kPasses && err == cudaSuccess; ++p) {
        unsigned* words = lookback + static_cast<size_t>(p) * tiles * kRadix;
        auto pass = [&](auto first, auto rest, int smem) {
            err = allow_smem(p == 0 ? first : rest, smem);
            if (err == cudaSuccess)
                err = chain_launch(ctx, p == 0 ? first : rest, tiles, kSortThreads, smem, kin,
                                   vin, kout, vout, n, 8 * p, hist + p * kRadix, words,
                                   counters + p, ctx->d_error);
        };
        if (items == 8)
            pass(k_onesweep<Key, true, 8>, k_onesweep<Key, false, 8>, onesweep_smem<Key, 8>());
        else
            pass(k_onesweep<Key, true, 4>, k_onesweep<Key, false, 4>, onesweep_smem<Key, 4>());
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return cuda_fail(err, "radix sort");
}

// Zeroes the words of ctx's scratch that start at zero (laid out as morton_and_sort lays it
// out); grows the scratch first.  *root_ord: the scene box's words.
template <typename Key>
int reset_sort_scratch(lux_ctx* ctx, int n, unsigned** root_ord) {
    constexpr int kPasses = sizeof(Key) == 4 ? 4 : 8;
    const SortScratch layout = sort_scratch(n, sizeof(Key), kPasses);
    if (int st = ensure_scratch(ctx, layout.total())) return st;
    unsigned* zeroed = reinterpret_cast<unsigned*>(static_cast<char*>(ctx->scratch) +
                                                   layout.key_bytes + layout.val_bytes);
    *root_ord = zeroed + SortScratch::kRoot;
    const size_t tiles = static_cast<size_t>(grid_for(n, kSortThreads * sort_items(n)));
    return cuda_fail(cudaMemsetAsync(zeroed, 0,
                                     layout.zero_bytes + sizeof(unsigned) * kRadix * kPasses * tiles,
                                     ctx->stream),
                     "sort scratch reset");
}

template <int Kind, typename Key>
int climb(lux_ctx* ctx, lux_bvh* bvh, const float* prims) {
    const int blocks = grid_for(bvh->n, kClimbThreads);
    const Key* codes = static_cast<const Key*>(bvh->codes);
    cudaError_t err = chain_launch(ctx, k_climb<Kind, Key>, blocks, kClimbThreads, 0, prims,
                                   bvh->n, codes, bvh->sorted_ids, bvh->tris, bvh->nodes,
                                   bvh->leaf_parent, bvh->open, bvh->open_count, bvh->root,
                                   ctx->d_error);
    if (err == cudaSuccess && blocks > 1)
        err = chain_launch(ctx, k_climb_top<Kind, Key>, grid_for(blocks, kTopThreads / 32),
                           kTopThreads, 0, prims, bvh->n, codes, bvh->sorted_ids, bvh->tris,
                           bvh->nodes, bvh->leaf_parent, bvh->open, bvh->open_count, blocks,
                           bvh->flags, bvh->root, ctx->d_error);
    return cuda_fail(err, "climb");
}

template <int Kind>
int refit(lux_ctx* ctx, lux_bvh* bvh, const float* prims) {
    return cuda_fail(chain_launch(ctx, k_refit<Kind>, grid_for(bvh->n, kClimbThreads),
                                  kClimbThreads, 0, prims, bvh->n, bvh->sorted_ids, bvh->tris,
                                  bvh->nodes, bvh->leaf_parent, bvh->flags, bvh->root,
                                  ctx->d_error),
                     "refit");
}

template <int Kind, typename Key>
int build_typed(lux_ctx* ctx, lux_bvh* bvh, const float* prims) {
    int n = bvh->n;
    Key* codes = static_cast<Key*>(bvh->codes);
    cudaError_t err = cudaSuccess;
    if (n == 1)
        // A lone leaf has no parent (the storage may hold a larger earlier tree).
        err = cudaMemsetAsync(bvh->leaf_parent, 0xff, sizeof(int), ctx->stream);
    if (err != cudaSuccess) return cuda_fail(err, "memset leaf parent");
    if (n <= kSmallSort) {
        const bool whole = n <= kWholeBuild;
        const auto kernel = whole ? k_build_small<Kind, Key, true> : k_build_small<Kind, Key, false>;
        const int smem = whole ? small_build_smem<Key, true>() : small_build_smem<Key, false>();
        err = allow_smem(kernel, smem);
        if (err == cudaSuccess)
            err = chain_launch(ctx, kernel, 1, kSmallThreads, smem, prims, n, codes,
                               bvh->sorted_ids, bvh->tris, bvh->nodes, bvh->leaf_parent,
                               bvh->root);
        if (err != cudaSuccess) return cuda_fail(err, "k_build_small");
        return whole ? LUX_OK : climb<Kind, Key>(ctx, bvh, prims);
    }
    unsigned* root_ord = nullptr;
    if (int st = reset_sort_scratch<Key>(ctx, n, &root_ord)) return st;
    err = chain_launch(ctx, k_root_reduce<Kind>, stride_grid(ctx, n), kThreads, 0, prims, n,
                       root_ord);
    if (err != cudaSuccess) return cuda_fail(err, "k_root_reduce");
    int st = morton_and_sort<Kind, Key>(ctx, prims, codes, bvh->sorted_ids, n);
    if (st) return st;
    return climb<Kind, Key>(ctx, bvh, prims);
}

}  // namespace

size_t lbvh_scratch_bytes(int n, int morton_bits) {
    return morton_bits == 63 ? sort_scratch(n, 8, 8).total() : sort_scratch(n, 4, 4).total();
}

int lbvh_alloc(lux_ctx* ctx, lux_bvh* bvh) {
    const int capacity = std::max(bvh->capacity, std::max(bvh->n, 1));
    const size_t n = static_cast<size_t>(capacity);
    const size_t inner = std::max<size_t>(n - 1, 1);
    const size_t key = bvh->morton_bits == 63 ? 8 : 4;
    // One allocation for every array (each cudaMalloc of a build is time on the host).
    struct Req {
        void** ptr;
        size_t bytes;
    } reqs[] = {
        {reinterpret_cast<void**>(&bvh->nodes), sizeof(BvhNode) * inner},
        {reinterpret_cast<void**>(&bvh->tris), sizeof(TriRecord) * n},
        {reinterpret_cast<void**>(&bvh->sorted_ids), sizeof(int) * n},
        {reinterpret_cast<void**>(&bvh->leaf_parent), sizeof(int) * n},
        {reinterpret_cast<void**>(&bvh->flags), sizeof(unsigned) * inner},
        {reinterpret_cast<void**>(&bvh->open), sizeof(int2) * n},
        {reinterpret_cast<void**>(&bvh->open_count),
         sizeof(int) * static_cast<size_t>(grid_for(capacity, kClimbThreads))},
        {&bvh->codes, key * n},
        {reinterpret_cast<void**>(&bvh->root), sizeof(float) * 16},
    };
    size_t total = 0;
    for (const auto& r : reqs) total += (r.bytes + 255) & ~size_t(255);
    // Triangles are built to be traced: their 4-wide nodes have their place from the start,
    // unless only the other arrays fit (the first ray query then asks for it).
    size_t wide_bytes = bvh->kind == LUX_PRIM_TRIANGLES ? sizeof(WideNode) * inner : 0;
    char* base = nullptr;
    cudaError_t got = cudaMalloc(reinterpret_cast<void**>(&base), total + wide_bytes);
    if (got != cudaSuccess && wide_bytes) {
        cudaGetLastError();
        wide_bytes = 0;
        got = cudaMalloc(reinterpret_cast<void**>(&base), total);
    }
    if (got != cudaSuccess) {
        cudaGetLastError();
        lbvh_free(bvh);
        return fail(LUX_ERR_OUT_OF_MEMORY, "lbvh allocation failed");
    }
    bvh->arena = base;
    bvh->capacity = capacity;   // only now: a BVH without arrays has room for nothing
    for (const auto& r : reqs) {
        *r.ptr = base;
        base += (r.bytes + 255) & ~size_t(255);
    }
    if (wide_bytes) {
        bvh->wide = reinterpret_cast<WideNode*>(base);
        bvh->wide_capacity = static_cast<int>(inner);
        bvh->wide_in_arena = true;
    }
    // On the context's stream: one on the default stream has no order with the build that
    // follows on a non-blocking stream.
    cudaError_t err = cudaMemsetAsync(bvh->flags, 0, sizeof(unsigned) * inner, ctx->stream);
    if (err == cudaSuccess)
        err = cudaMemsetAsync(bvh->leaf_parent, 0xff, sizeof(int) * n, ctx->stream);
    if (err != cudaSuccess) lbvh_free(bvh);
    return cuda_fail(err, "lbvh init");
}

void lbvh_free(lux_bvh* bvh) {
    if (bvh->wide && !bvh->wide_in_arena) cudaFree(bvh->wide);
    if (bvh->arena) cudaFree(bvh->arena);
    bvh->arena = nullptr;
    bvh->capacity = 0;
    bvh->wide = nullptr;
    bvh->wide_capacity = 0;
    bvh->wide_in_arena = false;
    bvh->wide_current = false;
    bvh->nodes = nullptr;
    bvh->tris = nullptr;
    bvh->sorted_ids = nullptr;
    bvh->leaf_parent = nullptr;
    bvh->flags = nullptr;
    bvh->open = nullptr;
    bvh->open_count = nullptr;
    bvh->codes = nullptr;
    bvh->root = nullptr;
}

int lbvh_build(lux_ctx* ctx, lux_bvh* bvh, const float* prims) {
    bvh->wide_current = false;
    if (bvh->n <= 0) return LUX_OK;
    bool wide = bvh->morton_bits == 63;
    if (bvh->kind == LUX_PRIM_TRIANGLES) {
        return wide ? build_typed<LUX_PRIM_TRIANGLES, unsigned long long>(ctx, bvh, prims)
                    : build_typed<LUX_PRIM_TRIANGLES, unsigned>(ctx, bvh, prims);
    }
    return wide ? build_typed<LUX_PRIM_AABBS, unsigned long long>(ctx, bvh, prims)
                : build_typed<LUX_PRIM_AABBS, unsigned>(ctx, bvh, prims);
}

namespace {

// Triangle records in sorted order from triangles given in input order.
__global__ void k_attach(const float* tris, int n, const int* sorted_ids, TriRecord* out,
                         int* error) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int pid = sorted_ids[k];
    if (pid < 0 || pid >= n) {
        atomicOr(error, kErrLoopBound);
        return;
    }
    f3 v0, v1, v2;
    box3 b;
    load_prim<LUX_PRIM_TRIANGLES>(tris, pid, v0, v1, v2, b);
    TriRecord r;
    r.p0 = make_float4(v0.x, v0.y, v0.z, __int_as_float(pid));
    r.p1 = make_float4(v1.x, v1.y, v1.z, 0.0f);
    r.p2 = make_float4(v2.x, v2.y, v2.z, 0.0f);
    out[k] = r;
}

}  // namespace

int lbvh_attach_triangles(lux_ctx* ctx, lux_bvh* bvh, const float* tris) {
    if (bvh->n <= 0) return LUX_OK;
    k_attach<<<grid_for(bvh->n), kThreads, 0, ctx->stream>>>(tris, bvh->n, bvh->sorted_ids,
                                                              bvh->tris, ctx->d_error);
    ctx->launches += 1;
    return cuda_fail(cudaGetLastError(), "k_attach");
}

int lbvh_refit(lux_ctx* ctx, lux_bvh* bvh, const float* prims) {
    bvh->wide_current = false;
    if (bvh->n <= 0) return LUX_OK;
    return bvh->kind == LUX_PRIM_TRIANGLES ? refit<LUX_PRIM_TRIANGLES>(ctx, bvh, prims)
                                           : refit<LUX_PRIM_AABBS>(ctx, bvh, prims);
}

namespace {

// Grid of one axis of a wide node whose children span [lo, hi]: the smallest exponent e
// whose grid, starting at k * 2^e with k * 2^e <= lo - kWideMargin * 2^e, holds hi and the
// margin within 255 steps.  False when no exponent within the range does.
LUX_D bool wide_axis(float lo, float hi, float* scale, float* inv_scale, float* origin,
                     float* c) {
    const float extent = sub(hi, lo);
    int e = -kWideMaxExp;
    if (extent > 0.0f) {
        int ex;
        frexpf(extent / 255.0f, &ex);
        e = max(ex, -kWideMaxExp);
    }
    for (; e <= kWideMaxExp; ++e) {
        const float s = wide_scale(e);
        const float inv = wide_scale(-e);
        const float x = mul(lo, inv);           // exact: a power of two
        float k = floorf(x);
        if (!(fabsf(k) < 4194304.0f)) continue;  // 2^22
        if (sub(x, k) < kWideMargin) k = sub(k, 1.0f);
        const float o = mul(k, s);              // exact
        if (!(add(mul(sub(hi, o), inv), kWideMargin) <= 255.0f)) continue;
        *scale = s;
        *inv_scale = inv;
        *origin = o;
        *c = mul(sub(k, 32768.0f), s);          // exact
        return true;
    }
    return false;
}

// Grid coordinates of [lo, hi], at least kWideMargin (less the rounding of the difference,
// 2^-16 of a step) outside it.
LUX_D void wide_quantize(float origin, float inv, float lo, float hi, unsigned& qlo,
                         unsigned& qhi) {
    const float a = floorf(sub(mul(sub(lo, origin), inv), kWideMargin));
    const float b = ceilf(add(mul(sub(hi, origin), inv), kWideMargin));
    qlo = static_cast<unsigned>(fminf(fmaxf(a, 0.0f), 255.0f));
    qhi = static_cast<unsigned>(fminf(fmaxf(b, 0.0f), 255.0f));
}

LUX_D float half_area(const box3& b) {
    const f3 d = b.hi - b.lo;
    return add(add(mul(d.x, d.y), mul(d.y, d.z)), mul(d.z, d.x));
}

// Wide node i from binary node i and the nodes below it (see WideNode).
__global__ void __launch_bounds__(kThreads) k_widen(const BvhNode* nodes, int n,
                                                    WideNode* wide, int* error) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const BvhNode nd = load_node(nodes, i);
    if (nd.ch.x >= n - 1 || nd.ch.y >= n - 1) {  // cannot happen for a consistent hierarchy
        atomicOr(error, kErrLoopBound);
        return;
    }
    box3 box[4];
    int ch[4];
    int count;
    if (nd.ch.x >= 0 && nd.ch.y >= 0) {
        const BvhNode l = load_node(nodes, nd.ch.x), r = load_node(nodes, nd.ch.y);
        box[0] = node_left_box(l); ch[0] = l.ch.x;
        box[1] = node_right_box(l); ch[1] = l.ch.y;
        box[2] = node_left_box(r); ch[2] = r.ch.x;
        box[3] = node_right_box(r); ch[3] = r.ch.y;
        count = 4;
    } else if (nd.ch.x < 0 && nd.ch.y < 0) {
        box[0] = node_left_box(nd); ch[0] = nd.ch.x;
        box[1] = node_right_box(nd); ch[1] = nd.ch.y;
        count = 2;
    } else {
        // One leaf and one internal child: the leaf, the child's children, and one of
        // those opened (the larger box first).
        const bool leaf_first = nd.ch.x < 0;
        const BvhNode m = load_node(nodes, leaf_first ? nd.ch.y : nd.ch.x);
        const box3 lb = leaf_first ? node_left_box(nd) : node_right_box(nd);
        const int lh = leaf_first ? nd.ch.x : nd.ch.y;
        box3 b3[3] = {node_left_box(m), node_right_box(m), box3{}};
        int c3[3] = {m.ch.x, m.ch.y, kNoNode};
        int c3n = 2;
        int open = -1;
        if (m.ch.x >= 0 && (m.ch.y < 0 || half_area(b3[0]) >= half_area(b3[1]))) open = 0;
        else if (m.ch.y >= 0) open = 1;
        if (open >= 0 && c3[open] < n - 1) {
            const BvhNode g = load_node(nodes, open ? m.ch.y : m.ch.x);
            if (open == 0) {
                b3[2] = b3[1]; c3[2] = c3[1];
                b3[0] = node_left_box(g); c3[0] = g.ch.x;
                b3[1] = node_right_box(g); c3[1] = g.ch.y;
            } else {
                b3[1] = node_left_box(g); c3[1] = g.ch.x;
                b3[2] = node_right_box(g); c3[2] = g.ch.y;
            }
            c3n = 3;
        }
        count = c3n + 1;
        if (leaf_first) {
            box[0] = lb; ch[0] = lh;
            box[1] = b3[0]; ch[1] = c3[0];
            box[2] = b3[1]; ch[2] = c3[1];
            box[3] = b3[2]; ch[3] = c3[2];
        } else {
            box[0] = b3[0]; ch[0] = c3[0];
            box[1] = b3[1]; ch[1] = c3[1];
            box[2] = c3n == 3 ? b3[2] : lb; ch[2] = c3n == 3 ? c3[2] : lh;
            box[3] = lb; ch[3] = lh;
        }
    }
    const box3 u = box_union(node_left_box(nd), node_right_box(nd));
    const float o[3] = {u.lo.x, u.lo.y, u.lo.z};
    const float top[3] = {u.hi.x, u.hi.y, u.hi.z};
    bool fits = true;
    float scale[3] = {1.0f, 1.0f, 1.0f}, inv[3], origin[3], cgrid[3];
    for (int a = 0; a < 3 && fits; ++a)
        fits = isfinite(o[a]) && isfinite(top[a]) &&
               wide_axis(o[a], top[a], &scale[a], &inv[a], &origin[a], &cgrid[a]);
    unsigned lo_w[3] = {0, 0, 0}, hi_w[3] = {0, 0, 0};
    if (fits) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c >= count) break;
            const float lo[3] = {box[c].lo.x, box[c].lo.y, box[c].lo.z};
            const float hi[3] = {box[c].hi.x, box[c].hi.y, box[c].hi.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                unsigned ql, qh;
                wide_quantize(origin[a], inv[a], lo[a], hi[a], ql, qh);
                lo_w[a] |= ql << (8 * c);
                hi_w[a] |= qh << (8 * c);
            }
        }
    } else {
        for (int a = 0; a < 3; ++a) {
            cgrid[a] = __int_as_float(0x7fffffff);
            scale[a] = 1.0f;
        }
    }
    if (count < 4) ch[3] = kNoNode;
    if (count < 3) ch[2] = kNoNode;
    WideNode w;
    w.q0 = make_float4(cgrid[0], cgrid[1], cgrid[2], scale[2]);
    w.q1 = make_float4(__uint_as_float(lo_w[0]), __uint_as_float(lo_w[1]),
                       __uint_as_float(lo_w[2]), __uint_as_float(hi_w[0]));
    w.q2 = make_float4(__uint_as_float(hi_w[1]), __uint_as_float(hi_w[2]), __int_as_float(ch[0]),
                       __int_as_float(ch[1]));
    w.q3 = make_float4(__int_as_float(ch[2]), __int_as_float(ch[3]), scale[0], scale[1]);
    wide[i] = w;
}

}  // namespace

int lbvh_ensure_wide(lux_ctx* ctx, lux_bvh* bvh) {
    if (bvh->wide_current || bvh->n <= 1) return LUX_OK;
    int need = std::max(bvh->capacity - 1, 1);
    if (bvh->wide_capacity < need) {
        // Nodes in the arena have its capacity: what is freed here is an allocation of its own.
        if (bvh->wide) cudaFree(bvh->wide);
        bvh->wide = nullptr;
        bvh->wide_capacity = 0;
        cudaError_t err = cudaMalloc(&bvh->wide, sizeof(WideNode) * size_t(need));
        if (err != cudaSuccess) {
            cudaGetLastError();
            bvh->wide = nullptr;
            return fail(LUX_ERR_OUT_OF_MEMORY, "wide node allocation failed");
        }
        bvh->wide_capacity = need;
    }
    k_widen<<<grid_for(bvh->n - 1), kThreads, 0, ctx->stream>>>(bvh->nodes, bvh->n, bvh->wide,
                                                                 ctx->d_error);
    ctx->launches += 1;
    int st = cuda_fail(cudaGetLastError(), "k_widen");
    if (!st) bvh->wide_current = true;
    return st;
}

int lbvh_export(lux_ctx* ctx, const lux_bvh* bvh, uint64_t* codes64, int* left, int* right,
                float* bounds) {
    int n = bvh->n;
    if (n <= 0) return LUX_OK;
    int count = 2 * n - 1;
    auto* c64 = reinterpret_cast<unsigned long long*>(codes64);
    if (bvh->morton_bits == 63) {
        k_export<unsigned long long><<<grid_for(count), kThreads, 0, ctx->stream>>>(
            bvh->view(), static_cast<const unsigned long long*>(bvh->codes), c64, left, right,
            bounds);
    } else {
        k_export<unsigned><<<grid_for(count), kThreads, 0, ctx->stream>>>(
            bvh->view(), static_cast<const unsigned*>(bvh->codes), c64, left, right, bounds);
    }
    ctx->launches += 1;
    return cuda_fail(cudaGetLastError(), "k_export");
}

}  // namespace lux

// ---------------------------------------------------------------- no-allocation sort
// lux_lbvh_morton_sort_static keeps every temporary of the Morton sort in this array
// instead of context scratch, so that a call allocates no device memory.  The module
// holds it on every GPU it is loaded on until the process exits.  Layout in bytes:
//   [0, 24)      six ordered-int root words (start at zero: the identity of max)
//   [64, 68)     device error word (starts at zero)
//   [256, ...)   digit histograms, kRadix x tiles words (fully rewritten every pass)
//   then keys    LUX_STATIC_SORT_MAX_PRIMS x 8 bytes: 63-bit alternate keys, or both
//                30-bit key buffers
//   then values  LUX_STATIC_SORT_MAX_PRIMS x 4 bytes: alternate primitive ids
namespace lux {
namespace {

constexpr int kStaticMaxPrims = LUX_STATIC_SORT_MAX_PRIMS;
constexpr int kStaticMaxTiles = (kStaticMaxPrims + kStaticTile - 1) / kStaticTile;
constexpr size_t kStaticHeaderBytes = 256;
constexpr size_t kStaticHistBytes = size_t(kRadix) * kStaticMaxTiles * sizeof(unsigned);
constexpr size_t kStaticKeyBytes = size_t(kStaticMaxPrims) * 8;
constexpr size_t kStaticValBytes = size_t(kStaticMaxPrims) * 4;
constexpr size_t kStaticBytes = kStaticHeaderBytes + kStaticHistBytes + kStaticKeyBytes +
                                kStaticValBytes;
static_assert(kStaticBytes == LUX_STATIC_SORT_SCRATCH_BYTES, "static sort array size");
static_assert(kStaticHistBytes % 256 == 0 && kStaticKeyBytes % 256 == 0, "region alignment");
constexpr int kMaxDevices = 64;

}  // namespace
}  // namespace lux

static __device__ __align__(256) unsigned char lux_static_sort_scratch[lux::kStaticBytes];

namespace lux {
namespace {

// Device address of the array on `device`, which must be current.  Looked up once per
// device (the first call on it), then reused.
int static_sort_scratch(int device, unsigned char** out) {
    static std::mutex mu;
    static unsigned char* address[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices)
        return fail(LUX_ERR_INVALID_ARGUMENT, "device ordinal out of range for the static sort");
    std::lock_guard<std::mutex> lk(mu);
    if (!address[device]) {
        void* p = nullptr;
        cudaError_t err = cudaGetSymbolAddress(&p, lux_static_sort_scratch);
        if (err != cudaSuccess) return cuda_fail(err, "cudaGetSymbolAddress(static sort array)");
        address[device] = static_cast<unsigned char*>(p);
    }
    *out = address[device];
    return LUX_OK;
}

__global__ void k_widen_codes(const unsigned* codes, int n, unsigned long long* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = codes[i];
}

// Root box, Morton codes and the LSD sort over explicit buffers: the even pass count
// leaves the result in (keys, vals).
template <int Kind, typename Key>
int morton_sort_into(lux_ctx* ctx, const float* prims, int n, Key* keys, Key* keys_alt,
                     int* vals, int* vals_alt, unsigned* hist, unsigned* root_ord, int* error) {
    cudaStream_t stream = ctx->stream;
    k_root_reduce<Kind><<<stride_grid(ctx, n), kThreads, 0, stream>>>(prims, n, root_ord);
    k_morton<Kind, Key><<<stride_grid(ctx, n), kThreads, 0, stream>>>(prims, n, root_ord, keys);
    ctx->launches += 2;
    const int tiles = grid_for(n, kStaticTile);
    int passes = (sizeof(Key) == 4 ? 30 + 7 : 63 + 7) / 8;
    if (passes & 1) ++passes;
    Key* kin = keys;
    Key* kout = keys_alt;
    int* vin = vals;
    int* vout = vals_alt;
    for (int p = 0; p < passes; ++p) {
        int shift = 8 * p;
        k_sort_upsweep<Key><<<tiles, kThreads, 0, stream>>>(kin, n, shift, hist, tiles);
        k_scan_exclusive<<<1, kScanThreads, 0, stream>>>(hist, kRadix * tiles);
        if (p == 0) {
            k_sort_downsweep<Key, true><<<tiles, kThreads, 0, stream>>>(
                kin, vin, kout, vout, n, shift, hist, tiles, error);
        } else {
            k_sort_downsweep<Key, false><<<tiles, kThreads, 0, stream>>>(
                kin, vin, kout, vout, n, shift, hist, tiles, error);
        }
        ctx->launches += 3;
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return cuda_fail(cudaGetLastError(), "static morton sort");
}

}  // namespace

int lbvh_morton_sort_static(lux_ctx* ctx, const float* prims, int n, int kind, int morton_bits,
                            uint64_t* sorted_codes, int* sorted_ids) {
    if (n < 0 || n > kStaticMaxPrims)
        return fail(LUX_ERR_INVALID_ARGUMENT,
                    "static morton sort: n = " + std::to_string(n) + " is outside 0.." +
                        std::to_string(kStaticMaxPrims) + " (the static array's limit)");
    unsigned char* base = nullptr;
    if (int st = static_sort_scratch(ctx->device, &base)) return st;
    if (n == 0) return LUX_OK;
    unsigned* root_ord = reinterpret_cast<unsigned*>(base);
    int* error = reinterpret_cast<int*>(base + 64);
    unsigned* hist = reinterpret_cast<unsigned*>(base + kStaticHeaderBytes);
    unsigned char* keys = base + kStaticHeaderBytes + kStaticHistBytes;
    int* vals_alt = reinterpret_cast<int*>(keys + kStaticKeyBytes);
    auto* codes64 = reinterpret_cast<unsigned long long*>(sorted_codes);
    cudaStream_t stream = ctx->stream;
    // The array keeps the previous call's contents: reset the words that must start at a
    // fixed value.  Histograms, keys and values are fully written before they are read.
    cudaError_t err = cudaMemsetAsync(root_ord, 0, 6 * sizeof(unsigned), stream);
    if (err == cudaSuccess) err = cudaMemsetAsync(error, 0, sizeof(int), stream);
    if (err != cudaSuccess) return cuda_fail(err, "static sort reset");
    int st;
    if (morton_bits == 63) {
        auto* alt = reinterpret_cast<unsigned long long*>(keys);
        st = kind == LUX_PRIM_TRIANGLES
                 ? morton_sort_into<LUX_PRIM_TRIANGLES>(ctx, prims, n, codes64, alt, sorted_ids,
                                                        vals_alt, hist, root_ord, error)
                 : morton_sort_into<LUX_PRIM_AABBS>(ctx, prims, n, codes64, alt, sorted_ids,
                                                    vals_alt, hist, root_ord, error);
    } else {
        auto* k30 = reinterpret_cast<unsigned*>(keys);
        auto* alt = k30 + kStaticMaxPrims;
        st = kind == LUX_PRIM_TRIANGLES
                 ? morton_sort_into<LUX_PRIM_TRIANGLES>(ctx, prims, n, k30, alt, sorted_ids,
                                                        vals_alt, hist, root_ord, error)
                 : morton_sort_into<LUX_PRIM_AABBS>(ctx, prims, n, k30, alt, sorted_ids,
                                                    vals_alt, hist, root_ord, error);
        if (!st) {
            k_widen_codes<<<stride_grid(ctx, n), kThreads, 0, stream>>>(k30, n, codes64);
            ctx->launches += 1;
            st = cuda_fail(cudaGetLastError(), "k_widen_codes");
        }
    }
    if (st) return st;
    err = cudaStreamSynchronize(stream);
    if (err != cudaSuccess) return cuda_fail(err, "static morton sort");
    int word = 0;
    err = cudaMemcpy(&word, error, sizeof(int), cudaMemcpyDeviceToHost);
    if (err != cudaSuccess) return cuda_fail(err, "static sort error word");
    if (word) return fail(LUX_ERR_DEVICE_CHECK, "static morton sort: device check failed");
    return LUX_OK;
}

}  // namespace lux
