// Stable LSD radix sort of (u32 key, u32 value) pairs.
//
// Replaces the comparison sort of whole 108-byte particle records in the reference
// (thrust::sort with a.hash < b.hash, NeighbourSearchCUDA.cu:167-170).  Only keys and a u32
// payload move; particle state is gathered once afterwards.  Stability makes equal keys keep their
// incoming order — for the cell-hash sort that is the previous step's sorted order, which is what
// the reference's merge sort yields for equal hashes.
//
// A sort of `bits`-bit keys runs ceil(bits / 10) passes of equal digit width (8..10 bits).  Each
// pass: per-tile digit counts, a scan of the (tile, digit) count matrix over the tiles (for inputs of
// few tiles in the scatter itself), and a stable scatter in which warps rank their keys by ballots and
// per-warp running digit counters, order the tile in shared memory and store it in runs.  Inputs of
// at most kClusterMax pairs take one launch per pass, with digits of up to 9 or 11 bits
// (make_cluster_plan).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dependent_launch.cuh"

namespace akua {
namespace radix {

constexpr int MAX_BITS = 10;
constexpr int MAX_RADIX = 1 << MAX_BITS;
constexpr int BLOCK = 256;
constexpr int WARPS = BLOCK / 32;
constexpr int ROUNDS = 16;                // keys per lane
constexpr int WARP_ITEMS = ROUNDS * 32;   // 512
constexpr int TILE = WARPS * WARP_ITEMS;  // 4096 keys per tile
constexpr int MAX_PASSES = 4;
// Tiles up to which the scatters add up the counts themselves.  Three passes in us without and with
// the scan's launch: 100,000 keys 27 / 32, 262,144 (64 tiles) 33 / 37, 300,000 40 / 36.
constexpr int kFusedTiles = 64;

inline int num_tiles(int n) { return (n + TILE - 1) / TILE; }

// Digit width per pass for keys of `bits` significant bits.
struct Plan {
    bool cluster = false;  // passes of one cluster each (make_cluster_plan)
    bool fused = false;    // the scatters scan the counts themselves (at most kFusedTiles tiles)
    int passes = 0;
    int width[MAX_PASSES] = {0, 0, 0, 0};
    int shift[MAX_PASSES] = {0, 0, 0, 0};
};

inline Plan make_plan(int bits) {
    Plan p;
    if (bits < 1) bits = 1;
    p.passes = (bits + MAX_BITS - 1) / MAX_BITS;
    int shift = 0, left = bits;
    for (int k = 0; k < p.passes; ++k) {
        const int w0 = (left + (p.passes - k) - 1) / (p.passes - k);
        const int w = w0 < 8 ? (left < 8 ? left : 8) : w0;  // widths below 8 gain nothing
        p.width[k] = w;
        p.shift[k] = shift;
        shift += w;
        left -= w;
        if (left <= 0) { p.passes = k + 1; break; }
    }
    return p;
}

inline int bits_for(uint64_t bound) {  // keys are < bound
    int bits = 0;
    uint64_t b = bound > 0 ? bound - 1 : 0;
    while (b) { ++bits; b >>= 1; }
    return bits < 1 ? 1 : bits;
}

// The lanes whose digit equals this lane's, of the lanes with `live`.  One ballot per bit: match.any
// takes a warp's distinct values one after another (2^20 random keys, 27 bits: 68 us with it, 54 with
// ballots; a pass over 8M particles' keys 65 against 58).
template <int BITS>
__device__ __forceinline__ uint32_t same_digit(uint32_t digit, bool live) {
    uint32_t peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        const bool one = (digit >> b) & 1u;
        const uint32_t ones = __ballot_sync(0xffffffffu, one);
        peers &= one ? ones : ~ones;
    }
    return peers;
}

// A kernel launched with `after` is set up while the stream's previous kernel ends, and waits for its
// stores (dependent_launch.cuh).  No kernel lets the next one start before its own blocks are done:
// blocks that wait take the room of blocks that work (2^20 pairs launched one by one: 68 us without,
// 58 with an early start, 47 like this; replayed from a graph 48, 55, 46).
template <class... Params, class... Args>
inline cudaError_t launch(bool after, void (*kernel)(Params...), int grid, int block, size_t smem,
                          cudaStream_t st, int cluster, Args... args) {
    cudaLaunchAttribute attr[2] = {};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    if (after) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// counts[tile * RADIX + d] = keys of `tile` with digit d.  A key's digit is (key >> shift) &
// digit_mask; digit_mask < RADIX narrows a pass to fewer bits than BITS.  (One row per tile: stores
// and the scatter's reads are contiguous.  One row per digit, with the digits' totals added up by
// atomics, cost 26 us against 12 over 8M keys and 54 against 48 for three passes over 2^20.)
template <int BITS>
__global__ void __launch_bounds__(BLOCK) upsweep(const uint32_t* __restrict__ keys, int n, int shift,
                                                 uint32_t digit_mask,
                                                 uint32_t* __restrict__ counts) {
    constexpr int RADIX = 1 << BITS;
    __shared__ uint32_t hist[WARPS][RADIX];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < WARPS * RADIX; t += BLOCK) (&hist[0][0])[t] = 0;
    __syncthreads();
    pdl::wait_for_previous(keys);
    const int base = blockIdx.x * TILE + warp * WARP_ITEMS + lane;
    uint32_t key[ROUNDS];  // all loads in flight at once: 14.4 -> 8.8 us at 1M, launch included
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int idx = base + r * 32;
        key[r] = idx < n ? keys[idx] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
        if (base + r * 32 < n) atomicAdd(&hist[warp][(key[r] >> shift) & digit_mask], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += BLOCK) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) s += hist[w][d];
        counts[(size_t)blockIdx.x * RADIX + d] = s;
    }
}

// counts[t][d] becomes the sum of counts[0..t)[d], totals[d] the sum over all tiles.  A block takes 8
// digits (one 32-byte sector of a row), its warps a run of tiles each, a quarter of the run per lane.
constexpr int SCAN_WARPS = 32;
constexpr int SCAN_DIGITS = 8;
template <int BITS>
__global__ void __launch_bounds__(32 * SCAN_WARPS)
    scan_tiles(uint32_t* __restrict__ counts, uint32_t* __restrict__ totals, int tiles) {
    constexpr int RADIX = 1 << BITS;
    constexpr int PARTS = 32 / SCAN_DIGITS;
    __shared__ uint32_t sums[SCAN_WARPS][SCAN_DIGITS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int digit = lane % SCAN_DIGITS, part = lane / SCAN_DIGITS;
    const int per = (tiles + SCAN_WARPS * PARTS - 1) / (SCAN_WARPS * PARTS);
    const int t0 = min((warp * PARTS + part) * per, tiles), t1 = min(t0 + per, tiles);
    pdl::wait_for_previous(counts);
    uint32_t* col = counts + blockIdx.x * SCAN_DIGITS + digit;
    uint32_t sum = 0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) sum += col[(size_t)t * RADIX];
    uint32_t run = 0, warp_sum = 0;  // the lower parts of this warp's run, and all of it
#pragma unroll
    for (int q = 0; q < PARTS; ++q) {
        const uint32_t c = __shfl_sync(0xffffffffu, sum, q * SCAN_DIGITS + digit);
        run += q < part ? c : 0u;
        warp_sum += c;
    }
    if (part == 0) sums[warp][digit] = warp_sum;
    __syncthreads();
    uint32_t all = 0;
#pragma unroll
    for (int w = 0; w < SCAN_WARPS; ++w) {
        const uint32_t c = sums[w][digit];
        run += w < warp ? c : 0u;
        all += c;
    }
    if (warp == 0 && part == 0) totals[blockIdx.x * SCAN_DIGITS + digit] = all;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) {
        const uint32_t c = col[(size_t)t * RADIX];
        col[(size_t)t * RADIX] = run;
        run += c;
    }
}

// Exclusive prefix sum of `v` over the block's threads (threads a multiple of 32); sums: one word per
// warp.  Ends with a barrier the caller can rely on for its own shared stores before the call.
template <int WARPS_>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    uint32_t lower = 0;
#pragma unroll
    for (int w = 0; w < WARPS_; ++w) lower += w < warp ? sums[w] : 0u;
    return lower + incl - v;
}

// Shared memory of a scatter: the per-warp digit counters, whose space the tile's pairs take once
// every pair knows its place in the tile, and two words per digit.
__host__ __device__ constexpr size_t scatter_smem(int warps, int radix, int pairs) {
    const size_t a = sizeof(uint32_t) * warps * radix, b = sizeof(uint2) * pairs;
    return (a > b ? a : b) + 2 * sizeof(uint32_t) * radix;
}

// Stable scatter of one tile.  `vals_in == nullptr` means the payload is the key's index.  With
// `rank_out`, rank_out[payload] = the pair's output position too (the inverse permutation).
// The tile is first ordered in shared memory, so that a warp's stores go to a few runs of
// consecutive addresses: an SM issues one 32-byte sector per two cycles, and pairs stored straight
// from their input order touch one each.
// 2^20 random pairs of 27 bits, three passes: 92 -> 54 us (with the upsweep's loads and the ballots,
// 73 without the ordering); a pass over 8M particles' keys 73 -> 53 us, over 1M 13.3 -> 13.5 (their
// runs of equal keys make short runs of stores by themselves).
// FUSED: `counts` holds the tiles' counts themselves and every block adds up what it needs; there are
// then few blocks, and all the registers they ask for are theirs (three blocks per SM otherwise: a
// pass over 8M particles' keys 53 us, with two 58, with one 88).
template <int BITS, bool FUSED>
__global__ void __launch_bounds__(BLOCK, FUSED ? 1 : 3)
    downsweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
              uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n, int shift,
              uint32_t digit_mask, const uint32_t* __restrict__ counts,
              const uint32_t* __restrict__ totals, int tiles, uint32_t* __restrict__ rank_out) {
    constexpr int RADIX = 1 << BITS;
    constexpr int PER = RADIX / BLOCK;  // digits per thread in the scan
    static_assert(RADIX % BLOCK == 0, "the scan gives every thread the same number of digits");
    extern __shared__ __align__(16) uint8_t scatter_raw[];
    uint32_t(*count)[RADIX] = reinterpret_cast<uint32_t(*)[RADIX]>(scatter_raw);  // [WARPS]
    uint2* pair = reinterpret_cast<uint2*>(scatter_raw);                          // [TILE], later
    uint32_t* start = reinterpret_cast<uint32_t*>(
        scatter_raw + scatter_smem(WARPS, RADIX, TILE) - 2 * sizeof(uint32_t) * RADIX);
    uint32_t* to = start + RADIX;  // digit's first output position minus its place in the tile
    __shared__ uint32_t sums[WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < WARPS * RADIX; t += BLOCK) (&count[0][0])[t] = 0;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const int tile0 = blockIdx.x * TILE;
    pdl::wait_for_previous(counts, totals);
    const int base = tile0 + warp * WARP_ITEMS + lane;
    uint32_t key[ROUNDS], val[ROUNDS], pos[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int idx = base + r * 32;
        const bool valid = idx < n;
        key[r] = valid ? keys_in[idx] : 0u;
        val[r] = valid ? (vals_in ? vals_in[idx] : (uint32_t)idx) : 0u;
    }
    // this thread's digits: the keys of the tiles before this one, and of all
    uint32_t first[PER], all[PER];
    if (FUSED) {
#pragma unroll
        for (int k = 0; k < PER; ++k) first[k] = all[k] = 0u;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t)
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const uint32_t c = counts[(size_t)t * RADIX + threadIdx.x * PER + k];
                first[k] += t < (int)blockIdx.x ? c : 0u;
                all[k] += c;
            }
    } else {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            first[k] = counts[(size_t)blockIdx.x * RADIX + threadIdx.x * PER + k];
            all[k] = totals[threadIdx.x * PER + k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool valid = base + r * 32 < n;
        const uint32_t d = (key[r] >> shift) & digit_mask;
        const uint32_t peers = same_digit<BITS>(d, valid);
        uint32_t before = 0;
        if (valid) before = count[warp][d];
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) count[warp][d] = before + __popc(peers);
        __syncwarp();
        pos[r] = before + __popc(peers & lt_mask);
    }
    __syncthreads();
    uint32_t total = 0, mine[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int d = threadIdx.x * PER + k;
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const uint32_t c = count[w][d];
            count[w][d] = run;
            run += c;
        }
        mine[k] = run;
        total += run;
    }
    uint32_t below = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) below += all[k];
    uint32_t at = block_exclusive<WARPS>(total, sums);
    __syncthreads();  // `sums` again
    below = block_exclusive<WARPS>(below, sums);  // the keys of all lower digits
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        start[threadIdx.x * PER + k] = at;
        to[threadIdx.x * PER + k] = below + first[k] - at;
        at += mine[k];
        below += all[k];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const uint32_t d = (key[r] >> shift) & digit_mask;
        pos[r] += start[d] + count[warp][d];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
        if (base + r * 32 < n) pair[pos[r]] = make_uint2(key[r], val[r]);
    __syncthreads();
    const int here = min(TILE, n - tile0);
#pragma unroll
    for (int r = 0; r < TILE / BLOCK; ++r) {
        const int k = r * BLOCK + threadIdx.x;
        if (k < here) {
            const uint2 p = pair[k];
            const uint32_t dst = to[(p.x >> shift) & digit_mask] + k;
            keys_out[dst] = p.x;
            vals_out[dst] = p.y;
            if (rank_out) rank_out[p.y] = dst;
        }
    }
}

// One pass over the digit (key >> shift) & digit_mask; digit_mask defaults to all BITS bits.
// `after`: the stream's previous kernel is this sort's previous pass.  `fused`: no scan launch, for
// inputs of few tiles (the scatters then read tiles x tiles rows).
template <int BITS, class Mark>
inline void run_pass(cudaStream_t s, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                     uint32_t* vout, uint32_t* counts, uint32_t* totals, int n, int shift,
                     uint32_t* rank_out, Mark& mark, bool fused, bool after,
                     uint32_t digit_mask = (1u << BITS) - 1u) {
    const int tiles = num_tiles(n);
    constexpr int RADIX = 1 << BITS;
    constexpr size_t smem = scatter_smem(WARPS, RADIX, TILE);
    digit_mask &= RADIX - 1;  // the kernels' shared-memory tables hold RADIX digits
    launch(after, upsweep<BITS>, tiles, BLOCK, 0, s, 1, kin, n, shift, digit_mask, counts);
    mark("radix_upsweep");
    if (!fused) {
        launch(true, scan_tiles<BITS>, RADIX / SCAN_DIGITS, 32 * SCAN_WARPS, 0, s, 1, counts, totals,
               tiles);
        mark("radix_scan");
        launch(true, downsweep<BITS, false>, tiles, BLOCK, smem, s, 1, kin, vin, kout, vout, n, shift,
               digit_mask, counts, totals, tiles, rank_out);
    } else {
        launch(true, downsweep<BITS, true>, tiles, BLOCK, smem, s, 1, kin, vin, kout, vout, n, shift,
               digit_mask, counts, nullptr, tiles, rank_out);
    }
    mark("radix_downsweep");
}

// ---- Sorts of up to kClusterMax pairs: a pass in one kernel, on one cluster of blocks.
//
// A tiled pass over a small input is three launches, each a few microseconds of latency for next to
// no work.  Here one cluster holds all pairs in registers: a block ranks its own (ballots or match.any,
// and per-warp digit counters), reads the other blocks' digit totals through distributed shared memory,
// scans them and scatters to global memory.
// Sorts of random keys in three passes: 27,000 pairs 56 -> 16.7 us, 65,536 34 -> 24.3; in two, 4,096:
// 39 -> 7.4.  The step of 27,000 particles went from 158 to 129 us with it.  (With 32-bit counters 27,000
// took 17.9 us and 4,096 7.8: the scan over the warps' counters and their zeroing are twice the shared
// memory.)
constexpr int kClusterThreads = 512;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterMax = 16 * kClusterThreads * 8;         // 65,536: eight rounds of 16 blocks
constexpr int kClusterPortableMax = 8 * kClusterThreads * 4;  // 16,384: four rounds of 8 blocks

// Digits of up to 9 bits (one per thread in the scans), or of up to 11 (four) where that saves a pass
// of 8 blocks and two or four rounds: 8,192 pairs of 19 bits 13.0 -> 10.6 us, 16,384 of 20 16.1 ->
// 14.8.  16 blocks read twice the counts from one another (27,000 of 21 bits 17.8 -> 19.6, 65,536 of
// 32 32.6 -> 35.3).  One round would gain 0.8 us of a step of 80 (4,096 of 20 bits 11.2 -> 10.4).
inline Plan make_cluster_plan(int bits, int n) {
    Plan p;
    p.cluster = true;
    if (bits < 1) bits = 1;
    const bool wide = n > 8 * kClusterThreads && n <= kClusterPortableMax;
    const int most = wide && (bits + 8) / 9 > (bits + 10) / 11 ? 11 : 9;
    p.passes = (bits + most - 1) / most;
    for (int k = 0, shift = 0; k < p.passes; ++k) {
        p.shift[k] = shift;
        p.width[k] = (bits - shift + (p.passes - k) - 1) / (p.passes - k);
        shift += p.width[k];
    }
    return p;
}

// Counts of up to 4,096 pairs, 16 bits each: a thread's PER neighbouring digits in one access.
template <int PER>
struct Counts;
template <>
struct Counts<1> {
    uint16_t w;
    __device__ __forceinline__ uint32_t operator[](int) const { return w; }
    __device__ __forceinline__ void operator+=(Counts o) { w += o.w; }
};
template <>
struct __align__(8) Counts<4> {
    uint32_t w[2];
    __device__ __forceinline__ uint32_t operator[](int k) const {
        return (k & 1) ? w[k >> 1] >> 16 : w[k >> 1] & 0xffffu;
    }
    __device__ __forceinline__ void operator+=(Counts o) {  // no half overflows
        w[0] += o.w[0];
        w[1] += o.w[1];
    }
};
__device__ __forceinline__ Counts<1> ld_remote(const Counts<1>* p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    Counts<1> c;
    asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(c.w) : "r"(a) : "memory");
    return c;
}
__device__ __forceinline__ Counts<4> ld_remote(const Counts<4>* p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    Counts<4> c;
    asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("ld.shared::cluster.v2.u32 {%0,%1}, [%2];"
                 : "=r"(c.w[0]), "=r"(c.w[1])
                 : "r"(a)
                 : "memory");
    return c;
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// Dynamic shared memory of a block: the per-warp counters, whose space its pairs take once every pair
// knows its place in the block, two words per digit, and the block's counts for the others.
__host__ __device__ constexpr size_t cluster_smem(int bits, int pairs) {
    const size_t a = (sizeof(uint16_t) * kClusterWarps) << bits, b = sizeof(uint2) * pairs;
    return (a > b ? a : b) + ((2 * sizeof(uint32_t) + sizeof(uint16_t)) << bits);
}

// One pass over the digit (key >> shift) & digit_mask, digit_mask < 1 << BITS.  Block b holds the
// pairs from b * 512 * ROUNDS on; warp w of it 32 * ROUNDS of them, in rounds of 32.
template <int BITS, int BLOCKS, int ROUNDS, bool RUNS>
__global__ void __launch_bounds__(kClusterThreads)
    cluster_pass(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                 uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n, int shift,
                 uint32_t digit_mask, uint32_t* __restrict__ rank_out) {
    constexpr int kPairs = kClusterThreads * ROUNDS;
    constexpr int RADIX = 1 << BITS;
    constexpr int PER = RADIX / kClusterThreads;  // digits per thread in the scans
    static_assert(kPairs <= 4096, "a block's counts fit 16 bits");
    extern __shared__ __align__(16) uint8_t scatter_raw[];
    uint16_t(*count)[RADIX] = reinterpret_cast<uint16_t(*)[RADIX]>(scatter_raw);
    uint2* pair = reinterpret_cast<uint2*>(scatter_raw);  // [kPairs], once the counters are done with
    uint32_t* start = reinterpret_cast<uint32_t*>(
        scatter_raw + cluster_smem(BITS, kPairs) - (2 * sizeof(uint32_t) + sizeof(uint16_t)) * RADIX);
    uint32_t* to = start + RADIX;  // digit's output position minus its place in the block
    // this block's pairs per digit, read by the others
    Counts<PER>* total = reinterpret_cast<Counts<PER>*>(to + RADIX);
    __shared__ uint32_t sums[kClusterWarps];
    const uint32_t rank = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int first = (int)rank * kPairs + warp * (32 * ROUNDS) + lane;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t key[ROUNDS], val[ROUNDS], pos[ROUNDS];
    uint4* zero = reinterpret_cast<uint4*>(&count[0][0]);
#pragma unroll
    for (int k = 0; k < kClusterWarps * RADIX / 8 / kClusterThreads; ++k)
        zero[k * kClusterThreads + t] = make_uint4(0u, 0u, 0u, 0u);
    pdl::wait_for_previous(keys_in, vals_in);
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int at = first + 32 * r;
        key[r] = at < n ? keys_in[at] : 0u;
        val[r] = at < n ? (vals_in ? vals_in[at] : (uint32_t)at) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool live = first + 32 * r < n;
        const uint32_t d = (key[r] >> shift) & digit_mask;
        const uint32_t peers = RUNS ? __match_any_sync(0xffffffffu, live ? d : 0xffffffffu)
                                    : same_digit<BITS>(d, live);
        uint32_t before = 0;
        if (live) before = count[warp][d];
        __syncwarp();
        if (live && lane == __ffs(peers) - 1) count[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        pos[r] = before + __popc(peers & below);
    }
    __syncthreads();
    Counts<PER> sum{};  // this thread's digits: exclusive over the warps, then the block's total
#pragma unroll
    for (int w = 0; w < kClusterWarps; ++w) {
        Counts<PER>* at = reinterpret_cast<Counts<PER>*>(count[w]) + t;
        const Counts<PER> c = *at;
        *at = sum;
        sum += c;
    }
    total[t] = sum;
    cluster_arrive();
    cluster_wait();
    // the pairs of all blocks, and of the blocks before this one
    uint32_t all[PER], before[PER], mine = 0, every = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) all[k] = before[k] = 0;
#pragma unroll
    for (uint32_t b = 0; b < BLOCKS; ++b) {
        const Counts<PER> c = ld_remote(&total[t], b);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            all[k] += c[k];
            before[k] += b < rank ? c[k] : 0u;
        }
    }
    cluster_arrive();  // this block is done with the others' totals
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        mine += sum[k];
        every += all[k];
    }
    uint32_t at = block_exclusive<kClusterWarps>(mine, sums);
    __syncthreads();  // `sums` again
    uint32_t lower = block_exclusive<kClusterWarps>(every, sums);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        start[t * PER + k] = at;
        to[t * PER + k] = lower + before[k] - at;
        at += sum[k];
        lower += all[k];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const uint32_t d = (key[r] >> shift) & digit_mask;
        pos[r] += start[d] + count[warp][d];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
        if (first + 32 * r < n) pair[pos[r]] = make_uint2(key[r], val[r]);
    __syncthreads();
    const int here = n - (int)rank * kPairs;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int k = r * kClusterThreads + t;
        if (k < here) {
            const uint2 p = pair[k];
            const uint32_t dst = to[(p.x >> shift) & digit_mask] + k;
            keys_out[dst] = p.x;
            vals_out[dst] = p.y;
            if (rank_out) rank_out[p.y] = dst;
        }
    }
    cluster_wait();  // no block exits while another may still read its totals
}

// One pass of a sort of n <= kClusterMax pairs.  RUNS: neighbouring pairs mostly have equal digits
// (a scene's particles, which come in the previous step's order), so a warp's match.any finds few
// distinct values; it then beats a ballot per bit (27,000 particles 110.5 against 111.6 us a step,
// 60,000 143 against 146, but 19.5 against 16.7 us for a sort of 27,000 random keys).
template <bool RUNS, class Mark>
inline void run_cluster_pass(cudaStream_t s, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                             uint32_t* vout, int n, int shift, int width, uint32_t* rank_out,
                             Mark& mark, bool after) {
    constexpr int kRound = 8 * kClusterThreads;
    const uint32_t mask = (1u << width) - 1u;
    auto go = [&](auto kernel, int bits, int blocks, int rounds) {
        const size_t smem = cluster_smem(bits, kClusterThreads * rounds);
        if (smem > 48 * 1024)  // above the default limit of dynamic shared memory
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        launch(after, kernel, blocks, kClusterThreads, smem, s, blocks, kin, vin, kout, vout, n, shift,
               mask, rank_out);
    };
    // 8 blocks wait for one another sooner, 16 spread the pairs and their scattered stores over more
    // SMs.  A step with 8 and with 16: 6,000 particles 85.3 and 86.3 us, 12,000 91.1 and 91.8, 27,000
    // 115.5 and 113.9, 40,000 136.3 and 132.1, 60,000 151.5 and 147.0.
    if (n <= kRound) {
        go(cluster_pass<9, 8, 1, RUNS>, 9, 8, 1);
    } else if (n <= 2 * kRound) {
        if (width > 9) go(cluster_pass<11, 8, 2, RUNS>, 11, 8, 2);
        else go(cluster_pass<9, 8, 2, RUNS>, 9, 8, 2);
    } else if (n <= 4 * kRound) {
        if (width > 9) go(cluster_pass<11, 8, 4, RUNS>, 11, 8, 4);
        else go(cluster_pass<9, 8, 4, RUNS>, 9, 8, 4);
    } else if (n <= 8 * kRound) {
        go(cluster_pass<9, 16, 4, RUNS>, 9, 16, 4);
    } else {
        go(cluster_pass<9, 16, 8, RUNS>, 9, 16, 8);
    }
    mark("radix_cluster_pass");
}

// Whether the current device places clusters of 16 blocks (beyond the portable 8, so the kernels must
// be allowed them first).
template <bool RUNS>
inline bool places_16() {
    cudaError_t e = cudaSuccess;
    auto allow = [&](auto kernel) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    };
    allow(cluster_pass<9, 16, 4, RUNS>);
    allow(cluster_pass<9, 16, 8, RUNS>);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 16;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem(9, kClusterThreads * 8);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveClusters(&clusters, cluster_pass<9, 16, 8, RUNS>, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && clusters > 0;
}

// Whether a sort of n pairs takes a cluster's passes; `places` is asked only where 16 blocks would run.
template <class Places>
inline bool takes_cluster(int n, Places&& places) {
    return n <= kClusterPortableMax || (n <= kClusterMax && places());
}

// Scratch words the sort needs for n keys: the count matrix and a pass's digit totals.
inline size_t scratch_words(int n) {
    return (size_t)MAX_RADIX * num_tiles(n) + MAX_RADIX;
}

// Sorts (k0, v0) by the low plan bits, ping-ponging with (k1, v1); all four buffers hold n words (a
// cluster plan: takes_cluster(n)).  With `index_payload` the input payload is each key's index and v0
// is not read.  The result buffers are returned through keys_out / vals_out.  With `rank_out` (n
// words), the last pass also writes rank_out[payload] = output position.  `mark(name)` is called after
// every kernel.
template <class Mark>
inline void sort_pairs(cudaStream_t s, const Plan& plan, uint32_t* k0, uint32_t* v0, uint32_t* k1,
                       uint32_t* v1, bool index_payload, uint32_t* scratch, int n,
                       uint32_t** keys_out, uint32_t** vals_out, Mark& mark,
                       uint32_t* rank_out = nullptr) {
    uint32_t* counts = scratch;
    uint32_t* totals = scratch + (size_t)MAX_RADIX * num_tiles(n);
    const uint32_t* kin = k0;
    const uint32_t* vin = index_payload ? nullptr : v0;
    uint32_t* kout = k1;
    uint32_t* vout = v1;
    for (int p = 0; p < plan.passes; ++p) {
        const bool last = p + 1 == plan.passes;
        // a digit narrower than 8 bits only occurs in the last pass, where the key's higher
        // bits are zero, so the 8-bit kernel sorts it correctly
        if (plan.cluster)
            run_cluster_pass<true>(s, kin, vin, kout, vout, n, plan.shift[p], plan.width[p],
                             last ? rank_out : nullptr, mark, p > 0);
        else if (plan.width[p] <= 8)
            run_pass<8>(s, kin, vin, kout, vout, counts, totals, n, plan.shift[p],
                        last ? rank_out : nullptr, mark, plan.fused, p > 0);
        else if (plan.width[p] == 9)
            run_pass<9>(s, kin, vin, kout, vout, counts, totals, n, plan.shift[p],
                        last ? rank_out : nullptr, mark, plan.fused, p > 0);
        else
            run_pass<10>(s, kin, vin, kout, vout, counts, totals, n, plan.shift[p],
                        last ? rank_out : nullptr, mark, plan.fused, p > 0);
        if (kout == k1) {
            kin = k1; vin = v1; kout = k0; vout = v0;
        } else {
            kin = k0; vin = v0; kout = k1; vout = v1;
        }
    }
    *keys_out = const_cast<uint32_t*>(kin);
    *vals_out = const_cast<uint32_t*>(vin);
}

}  // namespace radix
}  // namespace akua
