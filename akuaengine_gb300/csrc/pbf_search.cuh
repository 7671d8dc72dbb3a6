// Neighbour walk of the PBF step (NeighbourSearchCUDA.cu:72-130).
//
// The reference's walk: for the 27 cells around a particle's cell (dx outer, dz inner), look up
// the bucket of the cell's hash — a run of the hash-sorted (reference) order — and walk it in that
// order, skipping self, accepting |x_i - x_j|^2 < h^2, until maxNeighbours entries are found.  A
// bucket shared by two of the 27 cells is walked twice.
//
// The internal order sorts particles by the Morton code of their cell and, inside a cell, by
// reference rank.  A bucket that holds one cell is therefore a contiguous run of internal slots in
// the same order the reference walks it: a candidate's slot is directly its list entry.  Buckets
// flagged as mixed (several cells on one hash, or cells sharing a clamped Morton key) are walked in
// reference order, their ranks mapped to slots.  Both give the reference's list, entry for entry.
//
// Warp-cooperative walk.  A warp takes 32 consecutive particles (fewer in small scenes, see
// search_per_warp); consecutive particles of the same cell (a run) share one candidate sequence: the
// concatenation of the 27 buckets in walk order.
//
//   stage    lanes 0..26 look up one bucket each (the next run's lookups are in flight meanwhile),
//            a warp scan gives each bucket's offset, and the lanes write the sequence's slots into
//            the warp's pool of shared memory;
//   cull     candidates out of reach of the box around the run's particles leave the sequence (the
//            rest keep their order): half of them, as a run is about seven particles that fill
//            part of a cell.  The test is the pair test at the box's nearest point; rounding is
//            monotonic, so nothing a particle could accept is dropped.  A round takes 128, four per
//            lane: a quarter of the latencies of rounds of 32, even where those load a round ahead
//            (walk at 1M: 275 us with 32, 265 with 64, 253 with 128, 262 with 160, whose records no
//            longer fit the registers);
//   test     64 candidates at a time, two per lane, against the run's particles, two per round in
//            packed FP32x2.  A round's four ballots are all it leaves behind (hit masks in the
//            pool): no counts, no placement and no self test, two shared loads, twelve packed
//            operations, four compares and ballots and one store per 128 pairs.  A particle's
//            own slot is cleared from its mask by the lane that holds it as a candidate;
//   extract  once the pool is full or the warp's runs are staged, every lane turns its own
//            particle's masks into its list, all 32 lanes at once (a run alone would keep a fifth
//            of them busy): four set bits at a time become a tile, written as one coalesced uint4,
//            and its four candidates feed the first Jacobi iteration's density and lambda (same
//            terms, same order as k_density_lambda), so the list is not read back.
//
// What bounds it is instruction issue (70% of the issue slots at 32 warps per SM; 207 M warp
// instructions at 1M particles with 35 neighbours, against 319 M for a walk that placed every hit
// as it was found): the distance tests (210-270 candidates a particle before the cull) and the
// extraction.  Measured on that scene, 394 us before: hit masks and extraction 358 us, with one
// pool for masks and candidates 316, 64 candidates per round 279, masks with hits named by a bit
// and the reach tests of list entries dropped 265, the next run's lookup in flight 262; the cull
// makes the pool a third smaller and the walk's chain shorter (2,196 against 2,231 at 8M, 30 against
// 36 at 27k), and in rounds of 128: 253 at 1M, 2,060 at 8M.
//
// A run whose sequence does not fit the pool (pile-ups, or a walk cell much wider than h) goes
// through the same stages in segments of the sequence and stops once every list is full; its
// lists are placed entry by entry and read back for the density.
//
// The block size and STAGE (the walk's tile shape: a pool of 32 x STAGE words per warp) are
// template parameters; the solver's autotuner picks them by measurement (lists do not depend on
// them).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pbf_device.cuh"
#include "pbf_learned.cuh"
#include "pbf_pairs.cuh"

namespace akua {

// Default tile shape.  With culls of 32 the walk takes 273 us at 1M particles with 64 or 128 threads
// and 32 x 32 words, 294 with 32 x 48 (fewer warps fit an SM) and 404 with 32 x 16 (a warp's runs no
// longer fit the pool at once, so the extraction runs several times with few lanes).
constexpr int kSearchBlock = 128;
constexpr int kListStage = 32;

// Particles per warp.  32 keep every lane of the extraction busy, but a warp works through its runs
// one after another, so with few warps the walk lasts as long as one warp: a scene that would not
// fill the chip takes fewer per warp.  In exact math 8, 16 or 24 where those warps still all fit (24
// per SM at 80 registers; past that a second wave starts: 100,000 particles 63 us with 24, 53 with
// 32; 66,000 54 with 16, 40 with 24).  In fast math 8 to 28 up to 20 to 28 warps per SM (32 fit; us
// with w - 4 and w at the lines: 23,000 particles 22.0 with 8 and 22.8 with 12, 29,000 24.2 / 23.1,
// 33,000 26.2 / 24.8; 40,000 27.0 with 12 and 26.7 with 16; 50,000 29.3 / 29.2 and 60,000 31.6 / 30.9
// with 16 and 20; 78,000 35.3 / 35.0 with 20 and 24; 100,000 38.8 / 38.6 with 24 and 28 and 40.4 with
// 32; 122,000 44.8 / 43.7 with 28 and 32).  Fewer than 8 up to 12 warps per SM: with 1, 2, 4 and 8
// particles per warp 1,000 take 13.9 / 14.2 / 14.6 / 16.3 us, 4,000 - / 16.0 / 15.9 / 16.4, 9,000 (4, 6
// and 8) 17.8 / 17.5 / 18.1, 16,000 22.3 / 20.2 / 20.2.
//
// FEW (exact math, at most 8 particles per warp): four lanes turn a particle's masks into its list,
// which then lies in the pool, and evaluate its terms as the pair kernels do with four lanes.  Exact
// terms take the longest part of such a walk, a list's one after another (us before and after:
// 1,000 particles 20.5 and 15.5, 9,000 24.1 and 20.1, 27,000 30.0 and 24.9).  In fast math the
// longer code costs what the lanes gain (1,000: 13.9 and 14.2, 27,000: 23.3 and 23.9).
constexpr int kFewPerWarp = 8;
inline int search_per_warp(int n, int sms, bool exact) {
    const int most = 12 * sms;  // warps
    if (n <= kFewPerWarp * most) return (n + most - 1) / most;
    for (int w = 8; w < 32; w += exact ? 8 : 4) {
        const int per_sm = exact ? 24 : w < 24 ? 16 + w / 2 : 28;
        if (n <= w * per_sm * sms) return w;
    }
    return 32;
}
constexpr int kPairWords = 3 * 32;  // a run's positions, two particles interleaved
// Words of shared memory per warp: the pool of candidates and hit masks, then the positions.
__host__ __device__ constexpr int search_words(int stage) { return 32 * stage + kPairWords; }
__host__ __device__ constexpr size_t search_smem(int block, int stage) {
    return sizeof(uint32_t) * (block / 32) * search_words(stage);
}
constexpr uint32_t kRunMax = 32 * 32;  // candidates whose chunks one 32-bit mask can name
constexpr uint32_t kFullWarp = 0xffffffffu;
constexpr uint32_t kMixedBucket = 0x80000000u;  // bucket table: y bit for a mixed bucket

// The smallest value of a warp's lanes (NaN is ignored).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

template <bool EXACT, int BLOCK, int STAGE, bool FEW>
__global__ void __launch_bounds__(BLOCK, (EXACT ? 768 : 1024) / BLOCK)
    k_search(const StepParams* __restrict__ P, const float4* __restrict__ ps,
             const uint2* __restrict__ table, const uint32_t* __restrict__ r2i,
             uint32_t* __restrict__ nbr, uint32_t* __restrict__ cnt, float* __restrict__ rho_out,
             float* __restrict__ lam_out, uint32_t* __restrict__ flags, int density,
             const float* __restrict__ speed, const float* __restrict__ lprev,
             float* __restrict__ lacc, float* __restrict__ feat, float4* __restrict__ psl,
             int per_warp) {
    extern __shared__ __align__(16) uint32_t smem[];
    const StepParams& p = *P;
    const int n = p.n;
    const int lane = threadIdx.x & 31;
    // this warp's first particle (at most n plus a block's particles)
    const int base = (blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5)) * per_warp;
    if (base >= n) return;  // uniform over the warp
    const int i = base + lane;
    const int nvalid = min(per_warp, n - base);
    const bool valid = lane < nvalid;
    constexpr uint32_t kPool = 32 * STAGE;
    uint32_t* pool = smem + (threadIdx.x >> 5) * search_words(STAGE);
    float* pairs = reinterpret_cast<float*>(pool + kPool);
    const float4* pair_xy = reinterpret_cast<const float4*>(pairs);  // (xa, xb, ya, yb)
    const float2* pair_z = reinterpret_cast<const float2*>(pairs + 64);

    const float4 xi = valid ? ps[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int cx = cell_coord(xi.x, p.search_cell);
    const int cy = cell_coord(xi.y, p.search_cell);
    const int cz = cell_coord(xi.z, p.search_cell);
    // a run: consecutive particles of one scene in one cell
    const int sid = (valid && p.scene_of) ? (int)p.scene_of[i] : 0;
    const int px = __shfl_up_sync(kFullWarp, cx, 1);
    const int py = __shfl_up_sync(kFullWarp, cy, 1);
    const int pz = __shfl_up_sync(kFullWarp, cz, 1);
    const int ps_ = __shfl_up_sync(kFullWarp, sid, 1);
    uint32_t starts = __ballot_sync(
        kFullWarp, valid && (lane == 0 || px != cx || py != cy || pz != cz || ps_ != sid));

    const float h2 = p.h2;
    const int cap = p.cap;
    const uint32_t below = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7f800000);
    uint4* out4 = reinterpret_cast<uint4*>(nbr);

    // the bucket of the walk this lane looks up (dx = b/9 - 1, dy = b/3%3 - 1, dz = b%3 - 1)
    const int bdx = lane / 9 - 1, bdy = lane / 3 % 3 - 1, bdz = lane % 3 - 1;
    auto lookup = [&](uint32_t runs) {  // for the run starting at the lowest bit of `runs`
        const int q = __ffs(runs) - 1;
        const int rx = __shfl_sync(kFullWarp, cx, q);
        const int ry = __shfl_sync(kFullWarp, cy, q);
        const int rz = __shfl_sync(kFullWarp, cz, q);
        const StepParams& pr = P[__shfl_sync(kFullWarp, sid, q)];  // the run's scene
        uint2 e = make_uint2(0u, 0u);
        if (lane < 27)
            e = __ldg(table + pr.table_offset +
                      cell_hash(rx + bdx, ry + bdy, rz + bdz, pr.table_size, pr.table_magic));
        return e;
    };

    // Culls `total` staged candidates at `seq` (the first word of an even offset) against the run
    // of particles [q0, q0 + m) and tests the rest: returns their number; their masks follow them,
    // [64 candidates][particle][2 words], from the next even word.
    auto test = [&](uint32_t* seq, uint32_t total, int q0, int m) {
        const bool own = lane >= q0 && lane < q0 + m;
        if (own) {
            const int r = lane - q0;
            pairs[4 * (r >> 1) + (r & 1)] = xi.x;
            pairs[4 * (r >> 1) + 2 + (r & 1)] = xi.y;
            pairs[64 + r] = xi.z;
        }
        __syncwarp();
        uint32_t kept = total;
        if (total > 64u) {  // one round of tests takes no more than that as they are
            const float lx = warp_min(own ? xi.x : inf), hx = warp_min(own ? -xi.x : inf);
            const float ly = warp_min(own ? xi.y : inf), hy = warp_min(own ? -xi.y : inf);
            const float lz = warp_min(own ? xi.z : inf), hz = warp_min(own ? -xi.z : inf);
            kept = 0;
            auto reach = [&](float4 c) {
                const float dx = fmaxf(fmaxf(lx - c.x, c.x + hx), 0.f);
                const float dy = fmaxf(fmaxf(ly - c.y, c.y + hy), 0.f);
                const float dz = fmaxf(fmaxf(lz - c.z, c.z + hz), 0.f);
                return len2(dx, dy, dz) < h2;
            };
            constexpr int kCull = 4;  // candidates per lane and round: their loads are in flight at once
            for (uint32_t c0 = 0; c0 < total; c0 += 32 * kCull) {
                uint32_t j[kCull];
                float4 c[kCull];
#pragma unroll
                for (int q = 0; q < kCull; ++q) {
                    const uint32_t at = c0 + 32 * q + lane;
                    j[q] = at < total ? seq[at] : 0u;
                    c[q] = __ldg(ps + j[q]);
                }
                __syncwarp();  // what is kept goes where this round's candidates were read
#pragma unroll
                for (int q = 0; q < kCull; ++q) {
                    if (c0 + 32 * q >= total) break;
                    const bool keep = c0 + 32 * q + lane < total && reach(c[q]);
                    const uint32_t bal = __ballot_sync(kFullWarp, keep);
                    if (keep) seq[kept + __popc(bal & below)] = j[q];
                    kept += __popc(bal);
                }
            }
            __syncwarp();
        }
        uint2* put = reinterpret_cast<uint2*>(seq + ((kept + 1u) & ~1u));
        auto fetch = [&](uint32_t at, uint32_t& j) {
            j = at < kept ? seq[at] : 0xffffffffu;
            return at < kept ? __ldg(ps + j) : make_float4(inf, inf, inf, 0.f);
        };
        for (uint32_t c0 = 0; c0 < kept; c0 += 64, put += m) {
            uint32_t j0, j1;
            const float4 c = fetch(c0 + lane, j0), d = fetch(c0 + 32 + lane, j1);
            const float2 cx2 = f2(-c.x), cy2 = f2(-c.y), cz2 = f2(-c.z);
            const float2 dx2 = f2(-d.x), dy2 = f2(-d.y), dz2 = f2(-d.z);
            for (int r = 0; r < m; r += 2) {
                const float4 a = pair_xy[r >> 1];
                const float2 z = pair_z[r >> 1];
                const float2 ax = make_float2(a.x, a.y), ay = make_float2(a.z, a.w);
                const float2 rc = len2_2(add2(ax, cx2), add2(ay, cy2), add2(z, cz2));
                const float2 rd = len2_2(add2(ax, dx2), add2(ay, dy2), add2(z, dz2));
                const uint32_t ca = __ballot_sync(kFullWarp, rc.x < h2);
                const uint32_t cb = __ballot_sync(kFullWarp, rc.y < h2);
                const uint32_t da = __ballot_sync(kFullWarp, rd.x < h2);
                const uint32_t db = __ballot_sync(kFullWarp, rd.y < h2);
                if (lane < min(2, m - r))  // lanes 0 and 1 store a particle's masks each
                    put[r + lane] = lane ? make_uint2(cb, db) : make_uint2(ca, da);
            }
            __syncwarp();
            const uint32_t s0 = j0 - (uint32_t)(base + q0), s1 = j1 - (uint32_t)(base + q0);
            if (s0 < (uint32_t)m) atomicAnd(&put[s0].x, ~(1u << lane));
            if (s1 < (uint32_t)m) atomicAnd(&put[s1].y, ~(1u << lane));
        }
        __syncwarp();
        return kept;
    };

    // This lane's hits, in order: its masks at `mask` (chunk pair k at mask[k * stride]), its
    // candidates at `seq`.
    struct Hits {
        const uint2* mask;
        const uint32_t* seq;
        const uint32_t* at;  // the current chunk's candidates
        int stride, count;
        uint32_t left, bits;  // chunks with hits still to come, hits of the current chunk
        __device__ __forceinline__ Hits(const uint32_t* s, uint32_t kept, int r, int m)
            : mask(reinterpret_cast<const uint2*>(s + ((kept + 1u) & ~1u)) + r), seq(s), at(s),
              stride(m), count(0), left(0u), bits(0u) {
            for (uint32_t k = 0; 64 * k < kept; ++k) {
                const uint2 w = mask[k * stride];
                count += __popc(w.x) + __popc(w.y);
                left |= ((w.x ? 1u : 0u) | (w.y ? 2u : 0u)) << (2 * k);
            }
        }
        __device__ __forceinline__ uint32_t next() {  // only called while hits remain
            if (bits == 0u) {
                const int k = __ffs(left) - 1;
                left &= left - 1;
                bits = reinterpret_cast<const uint32_t*>(mask + (k >> 1) * stride)[k & 1];
                at = seq + 32 * k;
            }
            const uint32_t j = at[__ffs(bits) - 1];
            bits &= bits - 1;
            return j;
        }
    };
    // Density, lambda and the network's features of a particle's finished list.
    auto finish = [&](const DensityLambda2<EXACT>& acc, int count, int i, float4 xi) {
        rho_out[i] = acc.rho;
        const float l = acc.lambda(p);
        lam_out[i] = l;
        psl[i] = make_float4(xi.x, xi.y, xi.z, l);
        if (feat) {  // learned modes: the lambda sum starts; the network's features
            lacc[i] = l;
            write_features(params_for(P, i), acc, l, count, lprev[i], speed[i],
                           feat + (size_t)kFeatures * i);
        }
    };

    uint2 e_next = lookup(starts);
    while (starts) {
        uint32_t used = 0;       // words of the pool in use (even)
        uint32_t my_seq = 0;     // this lane's run: its candidates' place in the pool,
        uint32_t my_kept = 0;    // how many they are,
        int my_q0 = -1;          // its first lane (-1: this lane's run is not in the pool)
        int my_m = 0;            // and its particles
        while (starts) {
            const int q0 = __ffs(starts) - 1;
            const uint32_t rest = starts & (starts - 1);
            const int q1 = rest ? __ffs(rest) - 1 : nvalid;
            const int m = q1 - q0;
            const uint2 e = e_next;
            const uint32_t blen = e.y & ~kMixedBucket;
            // A lone particle whose only candidate is itself has an empty list.  (A bucket of one is
            // never mixed: e.x is its slot.  With a walk cell that is not the smoothing radius the only
            // candidate may be another particle, which then counts as two.)  Warps of spray have a run
            // per particle and end last, so a run that needs nothing more than its lookup counts
            // (300,000 particles between obstacles: walk 101 -> 96 us).
            const uint32_t others = blen == 1u && e.x != (uint32_t)(base + q0) ? 2u : blen;
            if (m == 1 && __reduce_add_sync(kFullWarp, others) == 1u) {
                if (lane == q0) {
                    my_seq = used;
                    my_q0 = q0;
                    my_m = 1;
                }
                if (rest) e_next = lookup(rest);
                starts = rest;
                continue;
            }
            uint32_t incl = blen;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(kFullWarp, incl, o);
                if (lane >= o) incl += v;
            }
            const uint32_t off = incl - blen;  // lanes 27..31: the sequence length
            const uint32_t total = __shfl_sync(kFullWarp, incl, 31);
            const uint32_t words = ((total + 1u) & ~1u) + 2u * ((total + 63u) >> 6) * m;

            // a dense run: segments of its sequence, the pool to itself
            if (words > kPool || total > kRunMax) {
                if (used) break;
                constexpr uint32_t kSegment = kPool / 2;  // its masks take as much again at most
                static_assert(kSegment <= kRunMax, "a segment's chunks must fit Hits::left");
                int count = 0;
                for (uint32_t s0 = 0; s0 < total; s0 += kSegment) {
                    // later hits of full lists are neither stored nor needed for the overflow flag
                    if (__all_sync(kFullWarp, lane < q0 || lane >= q1 || count >= cap)) break;
                    const uint32_t len = min(kSegment, total - s0);
                    for (uint32_t c0 = 0; c0 < len; c0 += 32) {
                        const uint32_t at = s0 + c0 + lane;
                        int b = 0;  // the last bucket starting at or before `at`
#pragma unroll
                        for (int step = 16; step; step >>= 1)
                            if (__shfl_sync(kFullWarp, off, b + step) <= at) b += step;
                        const uint32_t bx = __shfl_sync(kFullWarp, e.x, b);
                        const uint32_t by = __shfl_sync(kFullWarp, e.y, b);
                        const uint32_t t = bx + (at - __shfl_sync(kFullWarp, off, b));
                        if (c0 + lane < len)
                            pool[c0 + lane] = (by & kMixedBucket) ? __ldg(r2i + t) : t;
                    }
                    __syncwarp();
                    const uint32_t kept = test(pool, len, q0, m);
                    if (lane >= q0 && lane < q1) {
                        Hits hits(pool, kept, lane - q0, m);
                        for (int k = 0; k < hits.count && count + k < cap; ++k) {
                            const int pos = count + k;
                            nbr[4 * ((size_t)(pos >> 2) * n + i) + (pos & 3)] = hits.next();
                        }
                        count += hits.count;
                    }
                    __syncwarp();
                }
                if (lane >= q0 && lane < q1) {
                    if (count >= cap) atomicOr(flags, 1u);
                    count = min(count, cap);
                    cnt[i] = (uint32_t)count;
                    if (density) {
                        DensityLambda2<EXACT> acc;
                        acc.init(xi.w, p);
                        for (int g = 0; 4 * g < count; ++g) {
                            const uint4 t = out4[(size_t)g * n + i];
                            const int left = count - 4 * g;
                            acc.template add2<true>(p, xi, __ldg(ps + t.x),
                                                    __ldg(ps + (left >= 2 ? t.y : t.x)), left >= 2);
                            if (left > 2)
                                acc.template add2<true>(p, xi, __ldg(ps + t.z),
                                                        __ldg(ps + (left >= 4 ? t.w : t.z)),
                                                        left >= 4);
                        }
                        finish(acc, count, i, xi);
                    }
                }
                if (rest) e_next = lookup(rest);
                starts = rest;
                continue;
            }
            if (used + words > kPool) break;  // extract first
            if (rest) e_next = lookup(rest);

            uint32_t* seq = pool + used;
            const uint32_t longest = __reduce_max_sync(kFullWarp, blen);
            const uint32_t tag = e.y & kMixedBucket;
            for (uint32_t k = 0; k < longest; ++k)
                if (k < blen) seq[off + k] = (e.x + k) | tag;
            // Ranks -> slots over the whole sequence, four loads of a lane in flight: where walk cells are
            // not hash cells every bucket is mixed, and 27 of them one after another were slower than
            // a walk without a pool (200,000 particles, cells of h / 2: a step 343 us, 184 like this).
            if (__any_sync(kFullWarp, tag != 0u)) {
                __syncwarp();
                constexpr int kMap = 4;
                for (uint32_t c0 = lane; c0 < total; c0 += 32 * kMap) {
                    uint32_t t[kMap];
#pragma unroll
                    for (int q = 0; q < kMap; ++q) {
                        const uint32_t at = c0 + 32 * q;
                        t[q] = at < total ? seq[at] : 0u;
                        if (t[q] & kMixedBucket) t[q] = __ldg(r2i + (t[q] & ~kMixedBucket));
                    }
#pragma unroll
                    for (int q = 0; q < kMap; ++q)
                        if (c0 + 32 * q < total) seq[c0 + 32 * q] = t[q];
                }
            }
            const uint32_t kept = test(seq, total, q0, m);  // synchronises before it reads
            if (lane >= q0 && lane < q1) {
                my_seq = used;
                my_kept = kept;
                my_q0 = q0;
                my_m = m;
            }
            used += ((kept + 1u) & ~1u) + 2u * ((kept + 63u) >> 6) * m;
            starts = rest;
        }

        if constexpr (FEW) {  // four lanes per particle, through lists in the pool
            const int src = lane >> 2, role = lane & 3;
            const int q0 = __shfl_sync(kFullWarp, my_q0, src);
            const uint32_t kept = __shfl_sync(kFullWarp, my_kept, src);  // 0 without a run in the pool
            const int m = __shfl_sync(kFullWarp, my_m, src);
            const uint32_t* seq = pool + __shfl_sync(kFullWarp, my_seq, src);
            const uint2* mask = reinterpret_cast<const uint2*>(seq + ((kept + 1u) & ~1u)) + (src - q0);
            int total = 0;
            for (uint32_t k = 0; 64 * k < kept; ++k) {
                const uint2 w = mask[k * m];
                total += __popc(w.x) + __popc(w.y);
            }
            const int count = min(total, cap);
            const int room = (int)((__reduce_max_sync(kFullWarp, (unsigned)count) + 3u) & ~3u);
            const int lists = (int)((used + 3u) & ~3u);
            if (lists + 8 * room <= (int)kPool) {
                uint32_t* list = pool + lists + src * room;
                int at = 0;
                for (uint32_t k = 0; 64 * k < kept; ++k) {  // a lane places every fourth chunk's hits
                    const uint2 w = mask[k * m];
                    const uint32_t first = role == (int)(2 * k & 3) ? w.x : 0u;
                    const uint32_t second = role == (int)(2 * k + 1 & 3) ? w.y : 0u;
                    uint32_t bits = first | second;
                    const uint32_t* from = seq + 64 * k + (first ? 0 : 32);
                    for (int to = first ? at : at + __popc(w.x); bits; bits &= bits - 1, ++to)
                        if (to < count) list[to] = from[__ffs(bits) - 1];
                    at += __popc(w.x) + __popc(w.y);
                }
                __syncwarp();
                const int ip = min(base + src, n - 1);
                for (int g = role; 4 * g < count; g += 4) {
                    uint4 t = *reinterpret_cast<const uint4*>(list + 4 * g);
                    const int left = count - 4 * g;  // a partial last tile repeats its last entry
                    if (left < 2) t.y = t.x;
                    if (left < 3) t.z = t.y;
                    if (left < 4) t.w = t.z;
                    out4[(size_t)g * n + ip] = t;
                }
                const float4 xp = make_float4(
                    __shfl_sync(kFullWarp, xi.x, src), __shfl_sync(kFullWarp, xi.y, src),
                    __shfl_sync(kFullWarp, xi.z, src), __shfl_sync(kFullWarp, xi.w, src));
                const bool writes = role == 0 && q0 >= 0;
                if (writes) {
                    if (total >= cap) atomicOr(flags, 1u);
                    cnt[ip] = (uint32_t)count;
                }
                if (density) {
                    DensityLambda2<EXACT> acc;
                    acc.init(xp.w, p);
                    lanes_add<4, 6>(
                        ip, count,
                        [&](int e) { return *reinterpret_cast<const uint2*>(list + e); },
                        [&](uint32_t j) { return __ldg(ps + j); },
                        [&](float4 a, float4 b) {
                            return DensityLambda2<EXACT>::template terms<true>(p, xp, a, b);
                        },
                        acc);
                    if (writes) finish(acc, count, ip, xp);
                }
                __syncwarp();
                continue;
            }
        }
        // extract the lists of the runs in the pool, one lane per particle
        if (my_q0 >= 0) {
            Hits hits(pool + my_seq, my_kept, lane - my_q0, my_m);
            if (hits.count >= cap) atomicOr(flags, 1u);
            const int count = min(hits.count, cap);
            cnt[i] = (uint32_t)count;
            DensityLambda2<EXACT> acc;
            acc.init(xi.w, p);
            for (int g = 0; 4 * g < count; ++g) {
                const int left = count - 4 * g;
                uint4 t;
                t.x = hits.next();
                t.y = t.x;
                if (left >= 2) t.y = hits.next();
                t.z = t.y;
                if (left >= 3) t.z = hits.next();
                t.w = t.z;
                if (left >= 4) t.w = hits.next();
                out4[(size_t)g * n + i] = t;  // a partial last tile repeats its last entry
                if (density) {
                    const float4 a = __ldg(ps + t.x), b = __ldg(ps + t.y);
                    const float4 c = __ldg(ps + t.z), d = __ldg(ps + t.w);
                    acc.template add2<true>(p, xi, a, b, left >= 2);
                    if (left > 2) acc.template add2<true>(p, xi, c, d, left >= 4);
                }
            }
            if (density) finish(acc, count, i, xi);
        }
        __syncwarp();
    }
}

}  // namespace akua
