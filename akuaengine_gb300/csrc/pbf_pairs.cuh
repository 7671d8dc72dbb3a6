// Neighbour-pair passes of the PBF step, evaluated two neighbours at a time with Blackwell's packed
// FP32 instructions (__fadd2_rn / __fmul2_rn / __ffma2_rn: two IEEE round-to-nearest operations in
// one instruction).  Each lane of a packed operation rounds exactly like the scalar operation, so a
// pair term is bit-identical to its scalar evaluation; the per-particle sums stay scalar and run
// in list order.
//
// Neighbour lists are stored as uint4 tiles: nbr4[g * n + i] holds entries 4g..4g+3 of particle i,
// so one coalesced 16-byte load per lane fetches four neighbour indices.  Entries at or beyond a
// particle's count are never dereferenced.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pbf_device.cuh"

namespace akua {

// The neighbour-pair kernels run with a block size chosen per kernel (64, 128 or 256 threads; the
// solver's autotuner picks them by measurement); results do not depend on it.
constexpr int kMaxPairBlock = 256;

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a - b: fma(b, -1, a) is the exact difference rounded once, i.e. the IEEE subtraction.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// Differences and products with one operand shared, written as two scalar operations: gathered
// components lie in different registers of their records, and moving them together for a packed
// operation costs more instructions than it saves.
__device__ __forceinline__ float2 diff2(float a, float b, float c) {  // (a - b, a - c)
    return make_float2(a - b, a - c);
}
__device__ __forceinline__ float2 rdiff2(float b, float c, float a) {  // (b - a, c - a)
    return make_float2(b - a, c - a);
}
__device__ __forceinline__ float2 scale2(float a, float b, float c) {  // (a b, a c)
    return make_float2(a * b, a * c);
}
__device__ __forceinline__ float2 plus2(float a, float b, float c) {  // (a + b, a + c)
    return make_float2(a + b, a + c);
}
// dot3 of each lane (same contraction as the scalar dot3)
__device__ __forceinline__ float2 len2_2(float2 x, float2 y, float2 z) {
    return fma2(z, z, fma2(x, x, mul2(y, y)));
}

// IN_REACH: the caller knows r2 <= h2 (a list's entries at the positions that made the list).
template <bool IN_REACH = false>
__device__ __forceinline__ float2 poly6_2(const StepParams& p, float2 r2) {
    const float2 d = sub2(f2(p.h2), r2);
    const float2 w = mul2(f2(p.kp), mul2(mul2(d, d), d));
    if (IN_REACH) return w;
    return make_float2(r2.x > p.h2 ? 0.0f : w.x, r2.y > p.h2 ? 0.0f : w.y);
}

// 1 / sqrt(x).  Subnormal arguments, which rsqrtf would scale first, only occur below the distance at
// which spiky2 drops the result.
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Spiky gradient coefficient c with grad W = c * r (per lane).
template <bool EXACT, bool IN_REACH = false>
__device__ __forceinline__ void spiky2(const StepParams& p, float2 sx, float2 sy, float2 sz,
                                       float2 r2, float2& gx, float2& gy, float2& gz) {
    if constexpr (EXACT) {
        const float rx = __fsqrt_rn(r2.x), ry = __fsqrt_rn(r2.y);
        const float2 q = sub2(f2(p.h), make_float2(rx, ry));
        const float2 c = mul2(f2(p.ks), mul2(q, q));
        const float2 ax = mul2(c, sx), ay = mul2(c, sy), az = mul2(c, sz);
        const bool zx = rx > p.h || rx < 1e-5f, zy = ry > p.h || ry < 1e-5f;
        gx = make_float2(zx ? 0.f : __fdiv_rn(ax.x, rx), zy ? 0.f : __fdiv_rn(ax.y, ry));
        gy = make_float2(zx ? 0.f : __fdiv_rn(ay.x, rx), zy ? 0.f : __fdiv_rn(ay.y, ry));
        gz = make_float2(zx ? 0.f : __fdiv_rn(az.x, rx), zy ? 0.f : __fdiv_rn(az.y, ry));
    } else {
        const float2 ir = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
        const float2 r = mul2(r2, ir);
        const float2 q = sub2(f2(p.h), r);
        float2 c = mul2(mul2(f2(p.ks), mul2(q, q)), ir);
        if ((!IN_REACH && r2.x > p.h2) || r2.x < 1e-10f) c.x = 0.f;
        if ((!IN_REACH && r2.y > p.h2) || r2.y < 1e-10f) c.y = 0.f;
        gx = mul2(c, sx);
        gy = mul2(c, sy);
        gz = mul2(c, sz);
    }
}

// One tile of four list entries.  A pass reads each list once, so the tile takes no room in the L1
// that its gathers live on (1M particles: density 69.2 -> 65.8 us, delta 68.4 -> 65.1, XSPH 101 ->
// 98).
__device__ __forceinline__ uint4 ld_tile(const uint4* p) {
    uint4 t;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(t.x), "=r"(t.y), "=r"(t.z), "=r"(t.w)
                 : "l"(p));
    return t;
}

// Calls f(load(j0), load(j1), two) for consecutive neighbour pairs of one particle in list order;
// `two` is false only for a trailing single entry, in which case j1 == j0 and must not be
// accumulated.  The next tile of indices is loaded while the current one is processed.  With
// WHOLE_TILE all four records of a tile are loaded before the first pair is processed: fewer
// latencies in a row, more registers.  It pays in the density pass (65.8 -> 63.5 us at 1M) and in
// scenes that do not fill the chip (step of 60,000 particles 188 -> 182 us) and not where the
// records are wide or the registers short (vorticity 103 -> 107 us, confinement 76 -> 78).
template <bool WHOLE_TILE, class L, class F>
__device__ __forceinline__ void for_each_pair(const uint4* __restrict__ col, int n, int c, L&& load,
                                              F&& f) {
    const int ng = (c + 3) >> 2;
    if (ng == 0) return;
    uint4 cur = ld_tile(col);
    for (int g = 0; g < ng; ++g) {
        const int left = c - 4 * g;
        if (WHOLE_TILE) {
            const auto r0 = load(cur.x), r1 = load(left >= 2 ? cur.y : cur.x);
            auto r2 = r0, r3 = r0;
            if (left > 2) {
                r2 = load(cur.z);
                r3 = load(left >= 4 ? cur.w : cur.z);
            }
            if (g + 1 < ng) cur = ld_tile(col + (size_t)(g + 1) * n);
            f(r0, r1, left >= 2);
            if (left > 2) f(r2, r3, left >= 4);
        } else {
            uint4 nxt = cur;
            if (g + 1 < ng) nxt = ld_tile(col + (size_t)(g + 1) * n);
            f(load(cur.x), load(left >= 2 ? cur.y : cur.x), left >= 2);
            if (left > 2) f(load(cur.z), load(left >= 4 ? cur.w : cur.z), left >= 4);
            cur = nxt;
        }
    }
}

// What a pair of neighbours adds to a particle's sums: N values of each.
template <int N>
struct Terms {
    float2 v[N];
};

// for_each_neighbour with 2, 4 or 8 lanes per particle: entries(e) gives the list's entries e and e + 1
// (e even and below c).
template <int LANES, int N, class E, class L, class T, class A>
__device__ __forceinline__ void lanes_add(int i, int c, E&& entries, L&& load, T&& term, A&& add) {
    constexpr int kStep = 2 * LANES;  // entries per step
    const int role = threadIdx.x & (LANES - 1);
    const int group = (threadIdx.x & 31) & ~(LANES - 1);
    const int steps = __reduce_max_sync(0xffffffffu, (unsigned)((c + kStep - 1) / kStep));
    auto pair = [&](int s, uint32_t& j0, uint32_t& j1) {  // this lane's entries of step s
        const int e = kStep * s + 2 * role;
        j0 = j1 = (uint32_t)i;
        if (e < c) {
            const uint2 t = entries(e);
            j0 = t.x;
            j1 = e + 1 < c ? t.y : t.x;
        }
    };
    uint32_t j0, j1;
    pair(0, j0, j1);
    auto ra = load(j0), rb = load(j1);
    pair(1, j0, j1);
    for (int s = 0; s < steps; ++s) {
        const Terms<N> t = term(ra, rb);
        if (s + 1 < steps) {
            ra = load(j0);
            rb = load(j1);
            pair(s + 2, j0, j1);
        }
#pragma unroll
        for (int k = 0; k < kStep; ++k) {
            float one[N];
#pragma unroll
            for (int q = 0; q < N; ++q)
                one[q] = __shfl_sync(0xffffffffu, (k & 1) ? t.v[q].y : t.v[q].x, group + (k >> 1));
            if (kStep * s + k < c) add(one);
        }
    }
}

// Calls add(t, k) with the N terms t[] of each neighbour of particle i, in list order: load(j)
// gathers a neighbour's record, term(a, b) evaluates two of them.  With LANES = 1 a thread works
// through its particle's list by itself.  With 2, 4 or 8 lanes per particle each lane gathers
// and evaluates its own pair of every 4, 8 or 16 entries, the next one's records in flight, and the
// lanes hand their terms round by shuffles, so that every lane adds all of them in list order (the
// sums are the same bit for bit) and a list takes a half, a quarter or an eighth of the steps.  All
// lanes of a warp call it (c = 0 for lanes without a particle).
template <int LANES, bool WHOLE_TILE, int N, class L, class T, class A>
__device__ __forceinline__ void for_each_neighbour(const uint4* __restrict__ nbr4, int n, int i, int c,
                                                   L&& load, T&& term, A&& add) {
    if constexpr (LANES == 1) {
        for_each_pair<WHOLE_TILE>(nbr4 + i, n, c, load, [&](auto a, auto b, bool two) {
            const Terms<N> t = term(a, b);
            float one[N];
#pragma unroll
            for (int q = 0; q < N; ++q) one[q] = t.v[q].x;
            add(one);
            if (two) {
#pragma unroll
                for (int q = 0; q < N; ++q) one[q] = t.v[q].y;
                add(one);
            }
        });
    } else {
        lanes_add<LANES, N>(
            i, c,
            [&](int e) {
                const uint2* at = reinterpret_cast<const uint2*>(nbr4 + (size_t)(e >> 2) * n + i);
                return at[(e >> 1) & 1];
            },
            load, term, add);
    }
}

// Lanes per particle of the pair kernels.  A scene too small to fill the chip is as slow as the chain
// of gathers of one list, which more lanes shorten, until the shuffles cost more issue slots than the
// chain costs time: about 10 warps per SM with 8 lanes (22 with exact math, whose terms are longer)
// and 18 with 4 or 2 (24 with exact math: all that fit of its kernels of up to 80 registers).  Steps in us with 4 / 8 / 16 lanes: 1,000
// particles 70 / 66 / 68, 4,000 80 / 77 / 84, 6,000 82.6 / 82.2 / 92, 8,000 85 / 87; exact 1,000
// 88 / 75 / 72, 4,000 105 / 89 / 92, 12,000 118 / 109, 16,000 124 / 132.  With 1 / 2 / 4: 20,000 116 /
// 110 / 105, 27,000 120 / 111 / 114, 45,000 134 / 132, 52,000 140 / 144; exact 27,000 183 / 160 / 139,
// 36,000 195 / 179 / 180, 52,000 210 / 196, 60,000 214 / 230.
inline int pair_lanes(int n, int sms, bool exact) {
    const long long warps = 32ll * sms;  // threads of one warp per SM
    if (8ll * n <= (exact ? 22 : 10) * warps) return 8;
    if (4ll * n <= (exact ? 24 : 18) * warps) return 4;
    return 2ll * n <= (exact ? 24 : 18) * warps ? 2 : 1;
}

// sum += s * (x, y, z) of each neighbour's terms (s, x, y, z), one rounding per component.
struct Sum3 {
    float x = 0.f, y = 0.f, z = 0.f;
    __device__ __forceinline__ void operator()(const float (&t)[4]) {
        x = __fmaf_rn(t[0], t[1], x);
        y = __fmaf_rn(t[0], t[2], y);
        z = __fmaf_rn(t[0], t[3], z);
    }
};

// A particle's two-float4 record (x.xyz, w0 | v.xyz, w1) read in one 256-bit load (32-byte
// aligned: record j starts at float4 2j of a cudaMalloc'd array).
struct Rec8 {
    float4 x, v;
};
__device__ __forceinline__ Rec8 ld_rec8(const float4* __restrict__ rec, uint32_t j) {
    Rec8 r;
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r.x.x), "=f"(r.x.y), "=f"(r.x.z), "=f"(r.x.w), "=f"(r.v.x), "=f"(r.v.y),
                   "=f"(r.v.z), "=f"(r.v.w)
                 : "l"(rec + 2 * (size_t)j));
    return r;
}

// Density and lambda accumulators (ConstraintSolverCUDA.cu:16-97) and the terms of two neighbours:
// mass, poly6, the spiky gradient, |grad_j C_i|^2.
template <bool EXACT>
struct DensityLambda2 {
    float rho, gx, gy, gz, sum;
    __device__ __forceinline__ void init(float mi, const StepParams& p) {
        rho = mi * p.w0;
        gx = gy = gz = sum = 0.f;
    }
    template <bool IN_REACH = false>
    static __device__ __forceinline__ Terms<6> terms(const StepParams& p, float4 xi, float4 a,
                                                     float4 b) {
        const float2 sx = diff2(xi.x, a.x, b.x);
        const float2 sy = diff2(xi.y, a.y, b.y);
        const float2 sz = diff2(xi.z, a.z, b.z);
        const float2 r2 = len2_2(sx, sy, sz);
        Terms<6> t;
        t.v[0] = make_float2(a.w, b.w);
        t.v[1] = poly6_2<IN_REACH>(p, r2);
        spiky2<EXACT, IN_REACH>(p, sx, sy, sz, r2, t.v[2], t.v[3], t.v[4]);
        const float2 s = scale2(-p.inv_rho0, a.w, b.w);
        t.v[5] = len2_2(mul2(s, t.v[2]), mul2(s, t.v[3]), mul2(s, t.v[4]));
        return t;
    }
    __device__ __forceinline__ void operator()(const float (&t)[6]) {
        rho = __fmaf_rn(t[0], t[1], rho);
        gx = __fmaf_rn(t[0], t[2], gx);
        gy = __fmaf_rn(t[0], t[3], gy);
        gz = __fmaf_rn(t[0], t[4], gz);
        sum = sum + t[5];
    }
    template <bool IN_REACH = false>
    __device__ __forceinline__ void add2(const StepParams& p, float4 xi, float4 a, float4 b,
                                         bool two) {
        const Terms<6> t = terms<IN_REACH>(p, xi, a, b);
        (*this)({t.v[0].x, t.v[1].x, t.v[2].x, t.v[3].x, t.v[4].x, t.v[5].x});
        if (two) (*this)({t.v[0].y, t.v[1].y, t.v[2].y, t.v[3].y, t.v[4].y, t.v[5].y});
    }
    __device__ __forceinline__ float lambda(const StepParams& p) const {
        const float ax = gx * p.inv_rho0, ay = gy * p.inv_rho0, az = gz * p.inv_rho0;
        const float c = __fmaf_rn(rho, p.inv_rho0, -1.0f);
        const float den = (sum + len2(ax, ay, az)) + p.relaxation;
        return EXACT ? __fdiv_rn(-c, den) : __fdividef(-c, den);
    }
};

// The particle of this thread (LANES threads each) and whether there is one; threads beyond the last
// particle leave, except where their warp's lanes work together.
template <int LANES>
__device__ __forceinline__ bool particle_of_thread(int n, int& i) {
    i = (int)((blockIdx.x * blockDim.x + threadIdx.x) / LANES);
    const bool live = i < n;
    if (LANES > 1 && !live) i = n - 1;
    return live;
}
// Whether this thread writes its particle's results.
template <int LANES>
__device__ __forceinline__ bool writes(bool live) {
    return live && (threadIdx.x & (LANES - 1)) == 0;
}

template <bool EXACT, int LANES>
__global__ void __launch_bounds__(kMaxPairBlock)
    k_density_lambda(const StepParams* __restrict__ P, const float4* __restrict__ ps,
                     const uint4* __restrict__ nbr4, const uint32_t* __restrict__ cnt,
                     float* __restrict__ rho_out, float* __restrict__ lam_out,
                     float* __restrict__ lacc, float4* __restrict__ psl) {
    const int n = P->n;
    int i;
    const bool live = particle_of_thread<LANES>(n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(ps);
    const float4 xi = ps[i];
    DensityLambda2<EXACT> acc;
    acc.init(xi.w, p);
    for_each_neighbour<LANES, true, 6>(
        nbr4, n, i, live ? (int)cnt[i] : 0, [&](uint32_t j) { return ps[j]; },
        [&](float4 a, float4 b) { return DensityLambda2<EXACT>::terms(p, xi, a, b); }, acc);
    if (!writes<LANES>(live)) return;
    rho_out[i] = acc.rho;
    const float l = acc.lambda(p);
    lam_out[i] = l;
    psl[i] = make_float4(xi.x, xi.y, xi.z, l);
    if (lacc) lacc[i] += l;  // learned modes: the step's accumulated lambda
}

// (W(r2) / W(dq^2))^n of two pairs: the power in s_corr = -k * (...)^n (ConstraintSolverCUDA.cu:124).
template <bool EXACT, bool FOUR>
__device__ __forceinline__ float2 scorr_pow2(const StepParams& p, float2 r2) {
    const float2 w = poly6_2(p, r2);
    float2 ratio;
    if (EXACT) ratio = make_float2(__fdiv_rn(w.x, p.wdq), __fdiv_rn(w.y, p.wdq));
    else ratio = mul2(w, f2(p.inv_wdq));
    float2 pw;
    if (FOUR || p.corr_n_int == 4) {
        const float2 q = mul2(ratio, ratio);
        pw = mul2(q, q);
    } else if (p.corr_n_int >= 0) {
        pw = make_float2(pown(ratio.x, p.corr_n_int), pown(ratio.y, p.corr_n_int));
    } else {
        pw = make_float2(powf(ratio.x, p.corr_n), powf(ratio.y, p.corr_n));
    }
    return pw;
}

// A particle's position and mass with one more value of it.
struct Rec5 {
    float4 x;
    float l;
};

// Position delta with artificial pressure (ConstraintSolverCUDA.cu:99-130).
template <bool EXACT, int LANES>
__device__ __forceinline__ float3 position_delta(const StepParams& p, float4 xi, float li,
                                                 const float4* __restrict__ ps,
                                                 const float* __restrict__ lam,
                                                 const uint4* __restrict__ nbr4, int i, int c) {
    Sum3 d;
    auto load = [&](uint32_t j) { return Rec5{ps[j], lam[j]}; };
    auto term = [&](const Rec5& ra, const Rec5& rb) {
        const float4 a = ra.x, b = rb.x;
        const float2 lj = make_float2(ra.l, rb.l);
        const float2 sx = diff2(xi.x, a.x, b.x);
        const float2 sy = diff2(xi.y, a.y, b.y);
        const float2 sz = diff2(xi.z, a.z, b.z);
        const float2 r2 = len2_2(sx, sy, sz);
        // (lambda_i + lambda_j + s_corr) * m_j with s_corr = -k * pw: the product feeds the sum
        // and is contracted into it, as the CUDA compiler does with the reference's expression
        // (ConstraintSolverCUDA.cu:124-126).
        const float2 pw = scorr_pow2<EXACT, false>(p, r2);
        Terms<4> t;
        t.v[0] = mul2(fma2(f2(p.neg_k), pw, add2(f2(li), lj)), make_float2(a.w, b.w));
        spiky2<EXACT>(p, sx, sy, sz, r2, t.v[1], t.v[2], t.v[3]);
        return t;
    };
    for_each_neighbour<LANES, false, 4>(nbr4, p.n, i, c, load, term, d);
    return make_float3(d.x * p.inv_rho0, d.y * p.inv_rho0, d.z * p.inv_rho0);
}

// The same sum when every particle has mass `m`: positions and lambdas come from one 16-byte
// gather of psl[j] = (x*_j, lambda_j), and (lambda_i + lambda_j + s_corr) * m is the same product.
// FOUR: the power is 4 (the reference's), known before the loop: without the per-pair branch to
// powf the parameters stay in registers (1M particles: 75.1 -> 69.9 us).
template <bool EXACT, bool FOUR, int LANES>
__device__ __forceinline__ float3 position_delta_uniform(const StepParams& p,
                                                         const float4* __restrict__ psl, float m,
                                                         const uint4* __restrict__ nbr4, int i,
                                                         int c) {
    const float4 xl = psl[i];
    Sum3 d;
    auto load = [&](uint32_t j) { return psl[j]; };
    auto term = [&](float4 a, float4 b) {
        const float2 sx = diff2(xl.x, a.x, b.x);
        const float2 sy = diff2(xl.y, a.y, b.y);
        const float2 sz = diff2(xl.z, a.z, b.z);
        const float2 r2 = len2_2(sx, sy, sz);
        const float2 pw = scorr_pow2<EXACT, FOUR>(p, r2);
        Terms<4> t;
        t.v[0] = mul2(fma2(f2(p.neg_k), pw, plus2(xl.w, a.w, b.w)), f2(m));
        spiky2<EXACT>(p, sx, sy, sz, r2, t.v[1], t.v[2], t.v[3]);
        return t;
    };
    for_each_neighbour<LANES, true, 4>(nbr4, p.n, i, c, load, term, d);
    return make_float3(d.x * p.inv_rho0, d.y * p.inv_rho0, d.z * p.inv_rho0);
}

// Delta of particle i: the single-gather form when the step's masses all have one bit pattern
// (mass_bits = {0 when they do, that pattern}, from k_gather), else the general one.
template <bool EXACT, int LANES>
__device__ __forceinline__ float3 delta_of(const StepParams& p, int i, float4 xi,
                                           const float4* __restrict__ ps_in,
                                           const float* __restrict__ lam,
                                           const float4* __restrict__ psl,
                                           const uint32_t* __restrict__ mass_bits,
                                           const uint4* __restrict__ nbr4, int c) {
    if (mass_bits[0] == 0u) {
        const float m = __uint_as_float(mass_bits[1]);
        return p.corr_n_int == 4
                   ? position_delta_uniform<EXACT, true, LANES>(p, psl, m, nbr4, i, c)
                   : position_delta_uniform<EXACT, false, LANES>(p, psl, m, nbr4, i, c);
    }
    return position_delta<EXACT, LANES>(p, xi, lam[i], ps_in, lam, nbr4, i, c);
}

// Soft box clamp of one coordinate (ConstraintSolverCUDA.cu:136-157).
__device__ __forceinline__ float clamp_axis(float x, float lo_wall, float hi_wall) {
    const float lo = lo_wall + 0.025f, hi = hi_wall - 0.025f;
    float c = 0.f;
    if (x < lo) c = __fmaf_rn(0.5f, lo - x, c);
    if (x > hi) c = __fmaf_rn(0.5f, hi - x, c);
    return x + c;
}

template <bool EXACT, int LANES>
__global__ void __launch_bounds__(kMaxPairBlock)
    k_delta_correct(const StepParams* __restrict__ P, const float4* __restrict__ ps_in,
                    const float* __restrict__ lam, const uint4* __restrict__ nbr4,
                    const uint32_t* __restrict__ cnt, float4* __restrict__ ps_out,
                    float4* __restrict__ dp4, const float4* __restrict__ psl,
                    const uint32_t* __restrict__ mass_bits) {
    int i;
    const bool live = particle_of_thread<LANES>(P->n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(lam, psl, nbr4, cnt);
    const float4 xi = ps_in[i];
    const float3 d = delta_of<EXACT, LANES>(p, i, xi, ps_in, lam, psl, mass_bits, nbr4,
                                            live ? (int)cnt[i] : 0);
    if (!writes<LANES>(live)) return;
    dp4[i] = make_float4(d.x, d.y, d.z, 0.f);
    float nx = clamp_axis(xi.x + d.x, p.box_min[0], p.box_max[0]);
    float ny = clamp_axis(xi.y + d.y, p.box_min[1], p.box_max[1]);
    float nz = clamp_axis(xi.z + d.z, p.box_min[2], p.box_max[2]);
    sdf_correct(p, nx, ny, nz);
    ps_out[i] = make_float4(nx, ny, nz, xi.w);
}

// resolve_collision against one axis-aligned plane (IntegrationCUDA.cu:51-73), with the plane
// given as the reference builds it (IntegrationCUDA.cu:90-97): point on one axis, unit normal.
__device__ __forceinline__ void damp_plane(const StepParams& p, float px, float py, float pz,
                                           float qx, float qy, float qz, float nx, float ny, float nz,
                                           float& vx, float& vy, float& vz) {
    const float dist = dot3(px - qx, py - qy, pz - qz, nx, ny, nz);
    const float appr = dot3(vx, vy, vz, nx, ny, nz);
    if (dist < 0.025f) {
        const float vnx = appr * nx, vny = appr * ny, vnz = appr * nz;
        const float tx = vx - vnx, ty = vy - vny, tz = vz - vnz;
        if (appr < 0.0f) {
            vx = __fmaf_rn(p.neg_restitution, vnx, p.keep * tx);
            vy = __fmaf_rn(p.neg_restitution, vny, p.keep * ty);
            vz = __fmaf_rn(p.neg_restitution, vnz, p.keep * tz);
        } else if (fabsf(appr) < 1e-5f) {
            vx = p.keep * tx;
            vy = p.keep * ty;
            vz = p.keep * tz;
        }
    }
}

// Last Jacobi iteration fused with update (IntegrationCUDA.cu:38-49) and boundary damping
// (IntegrationCUDA.cu:75-102).  With `has_delta == 0` (zero iterations) the predicted positions
// go straight to the update and the carried density/lambda/delta move into the state.  Also moves
// the gathered origin and reference rank into the state arrays.
template <bool EXACT, int LANES>
__global__ void __launch_bounds__(kMaxPairBlock)
    k_delta_final(const StepParams* __restrict__ P, const float4* __restrict__ ps_in,
                  const float* __restrict__ lam, const uint4* __restrict__ nbr4,
                  const uint32_t* __restrict__ cnt, const float4* __restrict__ x_old,
                  float4* __restrict__ x4, float4* __restrict__ v4, float4* __restrict__ vstar4,
                  float4* __restrict__ dp4, const uint32_t* __restrict__ origing,
                  uint32_t* __restrict__ origin, const uint32_t* __restrict__ rref_new,
                  uint32_t* __restrict__ rref, const float* __restrict__ rho_c,
                  const float* __restrict__ lam_c, const float4* __restrict__ dp_c,
                  float* __restrict__ rho, float* __restrict__ lam_out, int has_delta,
                  const float4* __restrict__ psl, const uint32_t* __restrict__ mass_bits,
                  float4* __restrict__ xv8) {
    int i;
    const bool live = particle_of_thread<LANES>(P->n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(lam, psl, nbr4, cnt);
    const float4 xi = ps_in[i];
    float nx = xi.x, ny = xi.y, nz = xi.z;
    float3 d = make_float3(0.f, 0.f, 0.f);
    if (has_delta)
        d = delta_of<EXACT, LANES>(p, i, xi, ps_in, lam, psl, mass_bits, nbr4,
                                   live ? (int)cnt[i] : 0);
    if (!writes<LANES>(live)) return;
    if (has_delta) {
        dp4[i] = make_float4(d.x, d.y, d.z, 0.f);
        nx = clamp_axis(xi.x + d.x, p.box_min[0], p.box_max[0]);
        ny = clamp_axis(xi.y + d.y, p.box_min[1], p.box_max[1]);
        nz = clamp_axis(xi.z + d.z, p.box_min[2], p.box_max[2]);
        sdf_correct(p, nx, ny, nz);
    } else {
        rho[i] = rho_c[i];
        lam_out[i] = lam_c[i];
        dp4[i] = dp_c[i];
    }
    const float4 xo = x_old[i];
    const float vx0 = __fdiv_rn(nx - xo.x, p.dt);
    const float vy0 = __fdiv_rn(ny - xo.y, p.dt);
    const float vz0 = __fdiv_rn(nz - xo.z, p.dt);
    vstar4[i] = make_float4(vx0, vy0, vz0, 0.f);
    float vx = vx0, vy = vy0, vz = vz0;
    damp_plane(p, nx, ny, nz, p.box_min[0], 0.f, 0.f, 1.f, 0.f, 0.f, vx, vy, vz);
    damp_plane(p, nx, ny, nz, p.box_max[0], 0.f, 0.f, -1.f, 0.f, 0.f, vx, vy, vz);
    damp_plane(p, nx, ny, nz, 0.f, p.box_min[1], 0.f, 0.f, 1.f, 0.f, vx, vy, vz);
    damp_plane(p, nx, ny, nz, 0.f, p.box_max[1], 0.f, 0.f, -1.f, 0.f, vx, vy, vz);
    damp_plane(p, nx, ny, nz, 0.f, 0.f, p.box_min[2], 0.f, 0.f, 1.f, vx, vy, vz);
    damp_plane(p, nx, ny, nz, 0.f, 0.f, p.box_max[2], 0.f, 0.f, -1.f, vx, vy, vz);
    // the same damping against each obstacle, along its SDF gradient (plain dot products)
    for (int k = 0; k < p.num_shapes; ++k) {
        float g[3];
        const float dist = sdf_eval(p.shapes[k], nx, ny, nz, g);
        const float appr = vx * g[0] + vy * g[1] + vz * g[2];
        if (dist < p.sdf_min_dist) {
            const float vnx = appr * g[0], vny = appr * g[1], vnz = appr * g[2];
            const float tx = vx - vnx, ty = vy - vny, tz = vz - vnz;
            if (appr < 0.0f) {
                vx = __fmaf_rn(p.neg_restitution, vnx, p.keep * tx);
                vy = __fmaf_rn(p.neg_restitution, vny, p.keep * ty);
                vz = __fmaf_rn(p.neg_restitution, vnz, p.keep * tz);
            } else if (fabsf(appr) < 1e-5f) {
                vx = p.keep * tx;
                vy = p.keep * ty;
                vz = p.keep * tz;
            }
        }
    }
    const float4 xn = make_float4(nx, ny, nz, xi.w), vn = make_float4(vx, vy, vz, 0.f);
    x4[i] = xn;
    v4[i] = vn;
    xv8[2 * (size_t)i] = xn;  // (x, m | v) for vorticity's single gather
    xv8[2 * (size_t)i + 1] = vn;
    origin[i] = origing[i];
    rref[i] = rref_new[i];
}

// omega_i = sum_j -m_j (v_j - v_i) x grad W(x_i - x_j)  (IntegrationCUDA.cu:104-128).
// om4.w = |omega_i| for the confinement pass.
template <bool EXACT, int LANES>
__global__ void __launch_bounds__(kMaxPairBlock)
    k_vorticity(const StepParams* __restrict__ P, const float4* __restrict__ x4,
                const float4* __restrict__ v4, const float4* __restrict__ xv8,
                const uint4* __restrict__ nbr4, const uint32_t* __restrict__ cnt,
                float4* __restrict__ om4, float4* __restrict__ xw4) {
    const int n = P->n;
    int i;
    const bool live = particle_of_thread<LANES>(n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(x4, v4, xv8);
    const float4 xi = x4[i], vi = v4[i];
    Sum3 w;
    auto load = [&](uint32_t j) { return ld_rec8(xv8, j); };
    auto term = [&](const Rec8& ra, const Rec8& rb) {
        const float4 a = ra.x, b = rb.x, va = ra.v, vb = rb.v;
        const float2 sx = diff2(xi.x, a.x, b.x);
        const float2 sy = diff2(xi.y, a.y, b.y);
        const float2 sz = diff2(xi.z, a.z, b.z);
        float2 gx, gy, gz;
        spiky2<EXACT>(p, sx, sy, sz, len2_2(sx, sy, sz), gx, gy, gz);
        const float2 ux = rdiff2(va.x, vb.x, vi.x);
        const float2 uy = rdiff2(va.y, vb.y, vi.y);
        const float2 uz = rdiff2(va.z, vb.z, vi.z);
        // cross(u, g) contracted as fma(u.y, g.z, -(u.z * g.y)), ...
        Terms<4> t;
        t.v[0] = make_float2(-a.w, -b.w);
        t.v[1] = fma2(uy, gz, mul2(f2(-1.0f), mul2(uz, gy)));
        t.v[2] = fma2(uz, gx, mul2(f2(-1.0f), mul2(ux, gz)));
        t.v[3] = fma2(ux, gy, mul2(f2(-1.0f), mul2(uy, gx)));
        return t;
    };
    for_each_neighbour<LANES, EXACT, 4>(nbr4, n, i, live ? (int)cnt[i] : 0, load, term, w);
    if (!writes<LANES>(live)) return;
    const float wx = w.x, wy = w.y, wz = w.z;
    const float wn = __fsqrt_rn(len2(wx, wy, wz));
    om4[i] = make_float4(wx, wy, wz, wn);
    xw4[i] = make_float4(xi.x, xi.y, xi.z, wn);  // (x, |omega|) for confinement's single gather
}

// Vorticity confinement (IntegrationCUDA.cu:130-165); writes the confined velocity to the
// particle records (x, m_i / rho_i | v) for the XSPH pass.
// Capped at 48 registers (five 256-thread blocks per SM; 40 bytes spill, 60 in exact math), which slowed
// vorticity and the last delta pass.  1M particles capped and not: exact math 114 and 117 us, fast math
// 74 and 70 (80 and 84 before the pair loop took fewer instructions).
template <bool EXACT, int LANES>
__global__ void __launch_bounds__(kMaxPairBlock, LANES == 1 ? 5 : 1)
    k_confine(const StepParams* __restrict__ P, const float4* __restrict__ x4,
              const float4* __restrict__ v4, const float4* __restrict__ om4,
              const float* __restrict__ rho, const uint4* __restrict__ nbr4,
              const uint32_t* __restrict__ cnt, float4* __restrict__ xv8,
              const float4* __restrict__ xw4, const uint32_t* __restrict__ mass_bits) {
    const int n = P->n;
    int i;
    const bool live = particle_of_thread<LANES>(n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(om4, xw4);
    const float4 xi = x4[i], vi = v4[i], wi = om4[i];
    const float rho_i = rho[i];
    const int c = live ? (int)cnt[i] : 0;
    Sum3 eta;
    // m_j (|omega_i| - |omega_j|) and grad W, given positions, masses and |omega_j|
    auto pair = [&](float4 a, float4 b, float2 mj, float2 wj) {
        const float2 sx = diff2(xi.x, a.x, b.x);
        const float2 sy = diff2(xi.y, a.y, b.y);
        const float2 sz = diff2(xi.z, a.z, b.z);
        Terms<4> t;
        spiky2<EXACT>(p, sx, sy, sz, len2_2(sx, sy, sz), t.v[1], t.v[2], t.v[3]);
        t.v[0] = mul2(mj, sub2(f2(wi.w), wj));
        return t;
    };
    if (mass_bits[0] == 0u) {  // one mass: (x, |omega|) in one gather, the same products
        const float m = __uint_as_float(mass_bits[1]);
        auto load = [&](uint32_t j) { return xw4[j]; };
        auto term = [&](float4 a, float4 b) { return pair(a, b, f2(m), make_float2(a.w, b.w)); };
        for_each_neighbour<LANES, false, 4>(nbr4, n, i, c, load, term, eta);
    } else {
        auto load = [&](uint32_t j) { return Rec5{x4[j], om4[j].w}; };
        auto term = [&](const Rec5& a, const Rec5& b) {
            return pair(a.x, b.x, make_float2(a.x.w, b.x.w), make_float2(a.l, b.l));
        };
        for_each_neighbour<LANES, false, 4>(nbr4, n, i, c, load, term, eta);
    }
    if (!writes<LANES>(live)) return;
    float ex = eta.x, ey = eta.y, ez = eta.z;
    const float inv_d = __fdiv_rn(1.0f, rho_i);
    ex = ex * inv_d;
    ey = ey * inv_d;
    ez = ez * inv_d;
    float vx = vi.x, vy = vi.y, vz = vi.z;
    const float el = __fsqrt_rn(len2(ex, ey, ez));
    if (!(el < 1e-5f)) {
        float nx, ny, nz;
        if (EXACT) {
            nx = __fdiv_rn(ex, el); ny = __fdiv_rn(ey, el); nz = __fdiv_rn(ez, el);
        } else {
            const float inv = __fdividef(1.0f, el);
            nx = ex * inv; ny = ey * inv; nz = ez * inv;
        }
        const float3 cr = cross3(nx, ny, nz, wi.x, wi.y, wi.z);
        vx = __fmaf_rn(p.dt, p.vort_eps * cr.x, vx);
        vy = __fmaf_rn(p.dt, p.vort_eps * cr.y, vy);
        vz = __fmaf_rn(p.dt, p.vort_eps * cr.z, vz);
    }
    // (x, m_i / rho_i | confined v) for XSPH's single gather; vorticity, the only other reader of
    // these records, has finished, and no thread here reads another particle's record
    xv8[2 * (size_t)i] = make_float4(xi.x, xi.y, xi.z, __fdiv_rn(xi.w, rho_i));
    xv8[2 * (size_t)i + 1] = make_float4(vx, vy, vz, 0.f);
}

// XSPH viscosity (IntegrationCUDA.cu:167-195) from the confined-velocity snapshot in the records
// (x, m / rho | v).  Also leaves the bucket table all-empty for the next step.
template <bool EXACT, int LANES>  // the same in both modes
__global__ void __launch_bounds__(kMaxPairBlock)
    k_xsph(const StepParams* __restrict__ P, const float4* __restrict__ xv8,
           const uint4* __restrict__ nbr4, const uint32_t* __restrict__ cnt,
           float4* __restrict__ v4, const uint32_t* __restrict__ kr, uint2* __restrict__ table) {
    const int n = P->n;
    int i;
    const bool live = particle_of_thread<LANES>(n, i);
    if (LANES == 1 && !live) return;
    const StepParams& p = params_for(P, i);
    pdl::wait_for_previous(xv8);
    if (writes<LANES>(live)) {
        // the walk is done: empty this step's bucket entries (particle i: the bucket starting at
        // rank i)
        const uint32_t k = kr[i];
        if (i == 0 || kr[i - 1] != k) table[k] = make_uint2(0u, 0u);
    }
    const Rec8 ri = ld_rec8(xv8, (uint32_t)i);
    const float4 xi = ri.x, vi = ri.v;
    Sum3 sum;
    auto load = [&](uint32_t j) { return ld_rec8(xv8, j); };
    auto term = [&](const Rec8& ra, const Rec8& rb) {
        const float4 a = ra.x, b = rb.x, va = ra.v, vb = rb.v;
        const float2 sx = diff2(xi.x, a.x, b.x);
        const float2 sy = diff2(xi.y, a.y, b.y);
        const float2 sz = diff2(xi.z, a.z, b.z);
        const float2 s = make_float2(a.w, b.w);  // m_j / rho_j
        Terms<4> t;
        t.v[0] = poly6_2(p, len2_2(sx, sy, sz));
        t.v[1] = mul2(s, rdiff2(va.x, vb.x, vi.x));
        t.v[2] = mul2(s, rdiff2(va.y, vb.y, vi.y));
        t.v[3] = mul2(s, rdiff2(va.z, vb.z, vi.z));
        return t;
    };
    for_each_neighbour<LANES, true, 4>(nbr4, n, i, live ? (int)cnt[i] : 0, load, term, sum);
    if (!writes<LANES>(live)) return;
    const float ax = sum.x, ay = sum.y, az = sum.z;
    v4[i] = make_float4(__fmaf_rn(p.visc, ax, vi.x), __fmaf_rn(p.visc, ay, vi.y),
                        __fmaf_rn(p.visc, az, vi.z), 0.f);
}

}  // namespace akua
