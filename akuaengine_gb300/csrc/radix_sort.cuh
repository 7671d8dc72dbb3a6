// Stable LSD radix sort of (u32 key, u32 value) pairs.
//
// Replaces the comparison sort of whole 108-byte particle records in the reference
// (thrust::sort with a.hash < b.hash, NeighbourSearchCUDA.cu:167-170).  Only keys and a u32
// payload move; particle state is gathered once afterwards.  Stability makes equal keys keep their
// incoming order — for the cell-hash sort that is the previous step's sorted order, which is what
// the reference's merge sort yields for equal hashes.
//
// A sort of `bits`-bit keys runs ceil(bits / 10) passes of equal digit width (8..10 bits).  Each
// pass: per-tile digit counts (also accumulated into per-digit totals), one block per digit that
// turns its row of the (digit, tile) count matrix into global offsets, and a stable scatter in
// which warps rank their keys by ballots and per-warp running digit counters, order the tile in
// shared memory and store it in runs.  Inputs of at most kClusterMax pairs take one launch per pass.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace akua {
namespace radix {

constexpr int MAX_BITS = 10;
constexpr int MAX_RADIX = 1 << MAX_BITS;
constexpr int BLOCK = 256;
constexpr int WARPS = BLOCK / 32;
constexpr int ROUNDS = 16;                // keys per lane
constexpr int WARP_ITEMS = ROUNDS * 32;   // 512
constexpr int TILE = WARPS * WARP_ITEMS;  // 4096 keys per tile
constexpr int SCAN_BLOCK = 256;
constexpr int MAX_PASSES = 4;

inline int num_tiles(int n) { return (n + TILE - 1) / TILE; }

// Digit width per pass for keys of `bits` significant bits.
struct Plan {
    bool cluster = false;  // passes of one cluster each (make_cluster_plan)
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

// counts[d * tiles + tile] = keys of `tile` with digit d; totals[d] += the same.  A key's digit
// is (key >> shift) & digit_mask; digit_mask < RADIX narrows a pass to fewer bits than BITS.
template <int BITS>
__global__ void __launch_bounds__(BLOCK) upsweep(const uint32_t* __restrict__ keys, int n, int shift,
                                                 uint32_t digit_mask, uint32_t* __restrict__ counts,
                                                 uint32_t* __restrict__ totals, int tiles) {
    constexpr int RADIX = 1 << BITS;
    __shared__ uint32_t hist[WARPS][RADIX];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < WARPS * RADIX; t += BLOCK) (&hist[0][0])[t] = 0;
    __syncthreads();
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
        counts[(size_t)d * tiles + blockIdx.x] = s;
        if (s) atomicAdd(&totals[d], s);
    }
}

// Block d: offsets[d][t] = sum of totals[0..d) + sum of counts[d][0..t).
__global__ void __launch_bounds__(SCAN_BLOCK) scan_rows(uint32_t* __restrict__ counts,
                                                        const uint32_t* __restrict__ totals,
                                                        int tiles) {
    __shared__ uint32_t red[SCAN_BLOCK / 32];
    __shared__ uint32_t carry_s;
    const int d = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t part = 0;
    for (int k = threadIdx.x; k < d; k += SCAN_BLOCK) part += totals[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t b = 0;
        for (int w = 0; w < SCAN_BLOCK / 32; ++w) b += red[w];
        carry_s = b;
    }
    __syncthreads();
    uint32_t* row = counts + (size_t)d * tiles;
    for (int chunk = 0; chunk < tiles; chunk += SCAN_BLOCK) {
        const int t = chunk + threadIdx.x;
        const uint32_t v = t < tiles ? row[t] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        __syncthreads();  // red[] reuse
        if (lane == 31) red[warp] = incl;
        __syncthreads();
        uint32_t wpre = 0;
        for (int w = 0; w < warp; ++w) wpre += red[w];
        const uint32_t carry = carry_s;
        if (t < tiles) row[t] = carry + wpre + incl - v;
        __syncthreads();
        if (threadIdx.x == SCAN_BLOCK - 1) carry_s = carry + wpre + incl;
        __syncthreads();
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
// 73 without the ordering); a pass over 8M particles' keys 73 -> 58 us, over 1M 13.3 -> 13.5 (their
// runs of equal keys make short runs of stores by themselves).
template <int BITS>
__global__ void __launch_bounds__(BLOCK)
    downsweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
              uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n, int shift,
              uint32_t digit_mask, const uint32_t* __restrict__ offsets, int tiles,
              uint32_t* __restrict__ rank_out) {
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
    const int base = tile0 + warp * WARP_ITEMS + lane;
    uint32_t key[ROUNDS], val[ROUNDS], pos[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int idx = base + r * 32;
        const bool valid = idx < n;
        key[r] = valid ? keys_in[idx] : 0u;
        val[r] = valid ? (vals_in ? vals_in[idx] : (uint32_t)idx) : 0u;
    }
    uint32_t first[PER];  // this thread's digits: output position of the tile's first key
#pragma unroll
    for (int k = 0; k < PER; ++k)
        first[k] = offsets[(size_t)(threadIdx.x * PER + k) * tiles + blockIdx.x];
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
    uint32_t at = block_exclusive<WARPS>(total, sums);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        start[threadIdx.x * PER + k] = at;
        to[threadIdx.x * PER + k] = first[k] - at;
        at += mine[k];
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
template <int BITS, class Mark>
inline void run_pass(cudaStream_t s, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                     uint32_t* vout, uint32_t* counts, uint32_t* totals, int n, int shift,
                     uint32_t* rank_out, Mark& mark, uint32_t digit_mask = (1u << BITS) - 1u) {
    const int tiles = num_tiles(n);
    constexpr int RADIX = 1 << BITS;
    digit_mask &= RADIX - 1;  // the kernels' shared-memory tables hold RADIX digits
    upsweep<BITS><<<tiles, BLOCK, 0, s>>>(kin, n, shift, digit_mask, counts, totals, tiles);
    mark("radix_upsweep");
    scan_rows<<<RADIX, SCAN_BLOCK, 0, s>>>(counts, totals, tiles);
    mark("radix_scan");
    downsweep<BITS><<<tiles, BLOCK, scatter_smem(WARPS, RADIX, TILE), s>>>(
        kin, vin, kout, vout, n, shift, digit_mask, counts, tiles, rank_out);
    mark("radix_downsweep");
}

// ---- Sorts of up to kClusterMax pairs: a pass in one kernel, on one cluster of 8 blocks.
//
// A tiled pass over a small input is three launches, each a few microseconds of latency for next to
// no work.  Here one cluster holds all pairs in registers: a block ranks its own (match.any and
// per-warp digit counters, as downsweep does), reads the other blocks' digit totals through
// distributed shared memory, scans them and scatters to global memory.
// Three passes over 27,000 random keys: 56 -> 22 us, 4,096: 39 -> 8; at 65,536 32 us, where the tiled
// passes take 34 (eight SMs against sixteen).  The step of 27,000 particles: 158 -> 133 us.
constexpr int kClusterBlocks = 8;
constexpr int kClusterThreads = 512;  // one thread per digit in the scans
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterBits = 9;
constexpr int kClusterRadix = 1 << kClusterBits;
constexpr int kClusterMaxRounds = 16;
constexpr int kClusterMax = kClusterBlocks * kClusterThreads * kClusterMaxRounds;  // 65,536 pairs
static_assert(kClusterRadix == kClusterThreads, "thread d scans digit d");

inline Plan make_cluster_plan(int bits) {
    Plan p;
    p.cluster = true;
    if (bits < 1) bits = 1;
    p.passes = (bits + kClusterBits - 1) / kClusterBits;
    for (int k = 0, shift = 0; k < p.passes; ++k) {
        p.shift[k] = shift;
        p.width[k] = (bits - shift + (p.passes - k) - 1) / (p.passes - k);
        shift += p.width[k];
    }
    return p;
}

__device__ __forceinline__ uint32_t ld_remote(const uint32_t* p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), v;
    asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// One pass over the digit (key >> shift) & digit_mask, digit_mask < kClusterRadix.  Block b holds
// the pairs from b * 512 * ROUNDS on; warp w of it 32 * ROUNDS of them, in rounds of 32.
template <int ROUNDS, bool RUNS>
__global__ void __cluster_dims__(kClusterBlocks, 1, 1) __launch_bounds__(kClusterThreads)
    cluster_pass(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                 uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n, int shift,
                 uint32_t digit_mask, uint32_t* __restrict__ rank_out) {
    constexpr int kPer = kClusterThreads * ROUNDS;
    extern __shared__ __align__(16) uint8_t scatter_raw[];
    uint32_t(*count)[kClusterRadix] = reinterpret_cast<uint32_t(*)[kClusterRadix]>(scatter_raw);
    uint2* pair = reinterpret_cast<uint2*>(scatter_raw);  // [kPer], once the counters are done with
    uint32_t* start = reinterpret_cast<uint32_t*>(
        scatter_raw + scatter_smem(kClusterWarps, kClusterRadix, kPer) -
        2 * sizeof(uint32_t) * kClusterRadix);
    uint32_t* to = start + kClusterRadix;  // digit's output position minus its place in the block
    __shared__ uint32_t total[kClusterRadix];  // this block's pairs per digit, read by the others
    __shared__ uint32_t sums[kClusterWarps];
    const uint32_t rank = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int first = (int)rank * kPer + warp * (32 * ROUNDS) + lane;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t key[ROUNDS], val[ROUNDS], pos[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int at = first + 32 * r;
        key[r] = at < n ? keys_in[at] : 0u;
        val[r] = at < n ? (vals_in ? vals_in[at] : (uint32_t)at) : 0u;
    }
    uint4* zero = reinterpret_cast<uint4*>(&count[0][0]);
#pragma unroll
    for (int k = 0; k < kClusterWarps * kClusterRadix / 4 / kClusterThreads; ++k)
        zero[k * kClusterThreads + t] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool live = first + 32 * r < n;
        const uint32_t d = (key[r] >> shift) & digit_mask;
        const uint32_t peers = RUNS ? __match_any_sync(0xffffffffu, live ? d : 0xffffffffu)
                                    : same_digit<kClusterBits>(d, live);
        uint32_t before = 0;
        if (live) before = count[warp][d];
        __syncwarp();
        if (live && lane == __ffs(peers) - 1) count[warp][d] = before + __popc(peers);
        __syncwarp();
        pos[r] = before + __popc(peers & below);
    }
    __syncthreads();
    uint32_t sum = 0;  // digit t: exclusive over the warps, then the block's total
#pragma unroll
    for (int w = 0; w < kClusterWarps; ++w) {
        const uint32_t c = count[w][t];
        count[w][t] = sum;
        sum += c;
    }
    total[t] = sum;
    cluster_arrive();
    cluster_wait();
    // digit t: the pairs of all blocks, and of the blocks before this one
    uint32_t all = 0, before = 0;
#pragma unroll
    for (uint32_t b = 0; b < kClusterBlocks; ++b) {
        const uint32_t c = ld_remote(&total[t], b);
        all += c;
        before += b < rank ? c : 0u;
    }
    cluster_arrive();  // this block is done with the others' totals
    const uint32_t at = block_exclusive<kClusterWarps>(sum, sums);
    __syncthreads();  // `sums` again
    start[t] = at;
    to[t] = block_exclusive<kClusterWarps>(all, sums) + before - at;
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
    const int here = n - (int)rank * kPer;
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
// distinct values; it then beats a ballot per bit (27,000 particles: 136 against 140 us a step, but
// 27 against 22 us for a sort of as many random keys).
template <bool RUNS, class Mark>
inline void run_cluster_pass(cudaStream_t s, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                             uint32_t* vout, int n, int shift, int width, uint32_t* rank_out,
                             Mark& mark) {
    constexpr int kRound = kClusterBlocks * kClusterThreads;
    const uint32_t mask = (1u << width) - 1u;
    auto go = [&](auto kernel, int rounds) {
        const size_t smem = scatter_smem(kClusterWarps, kClusterRadix, kClusterThreads * rounds);
        if (smem > 48 * 1024)  // above the default limit of dynamic shared memory
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<kClusterBlocks, kClusterThreads, smem, s>>>(kin, vin, kout, vout, n, shift, mask,
                                                             rank_out);
    };
    if (n <= kRound) go(cluster_pass<1, RUNS>, 1);
    else if (n <= 2 * kRound) go(cluster_pass<2, RUNS>, 2);
    else if (n <= 4 * kRound) go(cluster_pass<4, RUNS>, 4);
    else if (n <= 8 * kRound) go(cluster_pass<8, RUNS>, 8);
    else go(cluster_pass<16, RUNS>, 16);
    mark("radix_cluster_pass");
}

// Scratch words the sort needs for n keys: the count matrix plus per-pass digit totals.
inline size_t scratch_words(int n) {
    return (size_t)MAX_RADIX * num_tiles(n) + (size_t)MAX_PASSES * MAX_RADIX;
}

// Sorts (k0, v0) by the low plan bits (a cluster plan: n <= kClusterMax), ping-ponging with (k1, v1); all four buffers hold n words.
// With `index_payload` the input payload is each key's index and v0 is not read.  The result
// buffers are returned through keys_out / vals_out.  With `rank_out` (n words), the last pass
// also writes rank_out[payload] = output position.  `mark(name)` is called after every kernel.
template <class Mark>
inline void sort_pairs(cudaStream_t s, const Plan& plan, uint32_t* k0, uint32_t* v0, uint32_t* k1,
                       uint32_t* v1, bool index_payload, uint32_t* scratch, int n,
                       uint32_t** keys_out, uint32_t** vals_out, Mark& mark,
                       uint32_t* rank_out = nullptr) {
    uint32_t* counts = scratch;
    uint32_t* totals = scratch + (size_t)MAX_RADIX * num_tiles(n);
    if (!plan.cluster) cudaMemsetAsync(totals, 0, sizeof(uint32_t) * MAX_PASSES * MAX_RADIX, s);
    const uint32_t* kin = k0;
    const uint32_t* vin = index_payload ? nullptr : v0;
    uint32_t* kout = k1;
    uint32_t* vout = v1;
    for (int p = 0; p < plan.passes; ++p) {
        uint32_t* tot = totals + (size_t)p * MAX_RADIX;
        const bool last = p + 1 == plan.passes;
        // a digit narrower than 8 bits only occurs in the last pass, where the key's higher
        // bits are zero, so the 8-bit kernel sorts it correctly
        if (plan.cluster)
            run_cluster_pass<true>(s, kin, vin, kout, vout, n, plan.shift[p], plan.width[p],
                             last ? rank_out : nullptr, mark);
        else if (plan.width[p] <= 8)
            run_pass<8>(s, kin, vin, kout, vout, counts, tot, n, plan.shift[p], last ? rank_out : nullptr, mark);
        else if (plan.width[p] == 9)
            run_pass<9>(s, kin, vin, kout, vout, counts, tot, n, plan.shift[p], last ? rank_out : nullptr, mark);
        else
            run_pass<10>(s, kin, vin, kout, vout, counts, tot, n, plan.shift[p], last ? rank_out : nullptr, mark);
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
