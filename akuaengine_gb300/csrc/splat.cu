// Headless point-splat renderer of the particle records: the consumer of the reference's interop
// buffer, restated as CUDA kernels writing an RGBA8 image (no graphics API).
//
// What it computes is the reference's particle pass (assets/shaders/fluidParticle.vert/.frag,
// src/Rendering/Renderer.cpp:29-50, src/Application/Application.cpp:72,112-113):
//   vertex   world = position (the particle object's model matrix is the identity,
//            SceneObject.cpp:61-62); point size = size / |world - camera|;
//            clip = (projection * view) * world
//   raster   a non-antialiased point: the pixels whose centres lie in the square of that side
//            around the window position; points whose vertex is outside the clip volume vanish
//   fragment offset = pointCoord - 0.5 (pointCoord's origin at the upper left); discarded when
//            |offset| > 0.5; colour = particle colour * exp(-|offset|^2 * 3)
//   output   depth test LESS against a cleared depth of 1, no blending, clear colour
//            (0.15, 0.15, 0.18, 1); equal depths keep the first particle drawn (lowest index)
// view = lookAt(eye, eye + gaze, up) and projection = perspective(fovy, aspect, near, far) are the
// right-handed, [-1, 1]-depth conventions of the reference's camera (Camera.cpp:32,74-87,
// Renderer.cpp:30).
//
// Pass 1 projects each particle and resolves visibility per pixel with one 64-bit atomicMin of
// (depth bits, particle index) -- non-negative float depths order like their bit patterns, and the
// index breaks ties as draw order does; pass 2 shades each pixel from its winning particle, projected
// again, and leaves the depth buffer empty for the next frame.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <new>

#include "akua_pbf.h"
#include "dependent_launch.cuh"

namespace {

struct SplatParams {
    float vp[16];   // projection * view, column-major (vp[4 * col + row])
    float eye[3];
    int width, height;
};

constexpr unsigned long long kEmpty = ~0ull;
constexpr float kMaxPointSize = 2047.0f;  // a typical implementation's point size range

__device__ __forceinline__ float frag_alpha(float ox, float oy, float* dist_out) {
    const float dist = sqrtf(ox * ox + oy * oy);
    *dist_out = dist;
    return expf(-dist * dist * 3.0f);
}

// (window x, window y, window depth, point size) of a record; size 0 marks a clipped point.
__device__ __forceinline__ float4 project(const SplatParams& P, const float* __restrict__ r) {
    const float x = r[0], y = r[1], z = r[2];
    const float dx = x - P.eye[0], dy = y - P.eye[1], dz = z - P.eye[2];
    const float dist = sqrtf(dx * dx + dy * dy + dz * dz);
    float size = r[26] / dist;  // Particle::size follows colour (offset 104 bytes)
    size = fminf(fmaxf(size, 1.0f), kMaxPointSize);
    float c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = P.vp[k] * x + P.vp[4 + k] * y + P.vp[8 + k] * z + P.vp[12 + k];
    const float w = c[3];
    const bool inside = w > 0.0f && fabsf(c[0]) <= w && fabsf(c[1]) <= w && fabsf(c[2]) <= w;
    const float nx = c[0] / w, ny = c[1] / w, nz = c[2] / w;
    const float xw = (nx + 1.0f) * 0.5f * (float)P.width;
    const float yw = (ny + 1.0f) * 0.5f * (float)P.height;
    const float zw = (nz + 1.0f) * 0.5f;
    return make_float4(xw, yw, zw, inside ? size : 0.0f);
}

// Pixel span of a point: centres px + 0.5 in [xw - s/2, xw + s/2).
__device__ __forceinline__ void span(float c, float s, int limit, int* lo, int* hi) {
    *lo = max(0, (int)ceilf(c - 0.5f * s - 0.5f));
    *hi = min(limit - 1, (int)ceilf(c + 0.5f * s - 0.5f) - 1);
}

// Whether a fragment whose centre is (dx, dy) off the point's centre lies in the disc: the test of
// pass 2's distance, |(dx, dy) / size| <= 0.5, decided from the product with 1 / size unless that is
// within its rounding (a few 1e-7) of the edge.
__device__ __forceinline__ bool in_disc(float dx, float dy, float size, float inv) {
    const float ax = dx * inv, ay = dy * inv;
    const float a2 = ax * ax + ay * ay;
    if (a2 < 0.25f - 1e-6f) return true;
    if (a2 > 0.25f + 1e-6f) return false;
    const float ox = dx / size, oy = -dy / size;
    float dist;
    frag_alpha(ox, oy, &dist);
    return !(dist > 0.5f);
}

// The pixel's nearest key so far, possibly an older one (this SM's L1): keys only fall within a
// pass, so a fragment that is not nearer than an older key is not nearer than the current one.
__device__ __forceinline__ unsigned long long seen(const unsigned long long* z) {
    unsigned long long v;
    asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(z));
    return v;
}

// A warp takes `per_warp` particles.  A sprite of at most `lane_pixels` is drawn by its own lane, which
// reads a pixel's key before it sends an atomic (there are most particles, and most hidden ones, where
// sprites are small); a larger one by the whole warp, one sprite after another, with plain atomics:
// 32 in flight at once wait for nothing, where a read first made each 32 pixels wait for L2 (30,000
// sprites of 13 pixels across 47 us with reads, 35 without, 25 across 118 and 70).  A sprite of more
// than `warp_pixels` is queued, in parts, for k_splat_large: particles near the eye come cell by cell,
// and warps that draw all of theirs keep the frame waiting.
// 32 particles per warp keep the lanes of a large scene busy; a scene too small to fill the chip that
// way has fewer per warp (splat_per_warp), or its sprites would wait for each other (1,000 particles of
// 40 pixels across: 171 us against 17).
// Frames of 1280 x 720 in us with a warp per particle, a projection pass and a cleared depth buffer, and
// like this: 1M particles with sprites of 1 to 4 pixels 176 and 37, of 12 across 628 and 424; 30,000
// with sprites of 5, 13 and 25 across 23, 37, 75 and 18, 35, 70; the eye among 27,000 particles 1,396 and
// 54, among 1M 836 and 164, in front of 100,000 with small sprites 33 and 35; 4M particles 657 and 93.
struct Shape {
    int per_warp;     // particles
    int lane_pixels;  // most pixels of a lane's sprite
    int warp_pixels;  // most pixels of a warp's sprite
};
constexpr int kPartPixels = 1024;      // of a queued sprite per part, at least
constexpr int kMaxParts = 64;          // of a sprite
constexpr uint32_t kQueue = 1u << 20;  // parts; a frame with more draws the rest by their warps
// Parts a frame may want before its sprites get at most 16, and 4: 30,000 sprites of half the image,
// which want 1.9M parts, 14.9 ms where the first half of the queue went to sprites in 64 parts 20.4.
constexpr unsigned long long kWantedFew = kQueue / 4, kWantedMany = kQueue;
constexpr unsigned long long kNoPart = ~0ull;
struct Queue {
    unsigned long long count;   // parts asked for, 0 between frames
    unsigned long long wanted;  // parts wanted at kMaxParts a sprite, 0 between frames
    unsigned long long part[kQueue];  // particle | part << 32 | parts << 40
};

// The next kernel of the stream may start once every block has got here, and waits for this one's
// completion itself (dependent_launch.cuh).
__device__ __forceinline__ void let_next_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct Sprite {
    float4 q;
    unsigned long long key;
    int x0, y0, nx, ny;
    __device__ __forceinline__ Sprite(const SplatParams& P, float4 q_, int i) : q(q_) {
        int x1 = -1, y1 = -1;
        x0 = y0 = 0;
        if (q.w > 0.0f && q.z < 1.0f) {  // else clipped, or not nearer than the cleared depth
            span(q.x, q.w, P.width, &x0, &x1);
            span(q.y, q.w, P.height, &y0, &y1);
        }
        nx = max(0, x1 - x0 + 1);  // at most 2048 each
        ny = max(0, y1 - y0 + 1);
        key = ((unsigned long long)__float_as_uint(fmaxf(q.z, 0.0f)) << 32) | (unsigned)i;
    }
    __device__ __forceinline__ uint32_t parts(int most) const {
        return (uint32_t)min(most, (nx * ny + kPartPixels - 1) / kPartPixels);
    }
    // The place of pixel k in the depth buffer, if it lies in the disc.
    __device__ __forceinline__ bool pixel(const SplatParams& P, int k, float inv, size_t& at) const {
        const int row = k / nx, px = x0 + (k - row * nx), py = y0 + row;
        at = (size_t)py * P.width + px;
        return in_disc(((float)px + 0.5f) - q.x, ((float)py + 0.5f) - q.y, q.w, inv);
    }
    // Draws the pixels first, first + step, ...
    __device__ __forceinline__ void draw(const SplatParams& P, unsigned long long* zbuf, int first,
                                         int step) const {
        const float inv = 1.0f / q.w;
        const int count = nx * ny;
        for (int k = first; k < count; k += step) {
            size_t at;
            if (pixel(P, k, inv, at)) atomicMin(zbuf + at, key);
        }
    }
    // Draws all pixels where the key read is farther; the reads of two are in flight at once.
    __device__ __forceinline__ void draw_nearer(const SplatParams& P, unsigned long long* zbuf) const {
        const float inv = 1.0f / q.w;
        const int count = nx * ny;
        for (int k = 0; k < count; k += 2) {
            size_t at[2];
            unsigned long long z[2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
                z[u] = k + u < count && pixel(P, k + u, inv, at[u]) ? seen(zbuf + at[u]) : 0ull;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (key < z[u]) atomicMin(zbuf + at[u], key);
        }
    }
};

constexpr int kRasterWarps = 8;

// Sum of `v` over the lower threads of the block; sums[kRasterWarps] becomes the block's.
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t upto = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
    }
    __syncthreads();  // `sums` may still be read from an earlier call
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
        for (int w = 0; w < kRasterWarps; ++w) {
            const uint32_t x = sums[w];
            sums[w] = all;
            all += x;
        }
        sums[kRasterWarps] = all;
    }
    __syncthreads();
    return sums[warp] + (upto - v);
}

// Six blocks per SM (40 registers; with 44 and five blocks 4M particles take 98 us instead of 93).
__global__ void __launch_bounds__(32 * kRasterWarps, 6)
    k_splat_raster(SplatParams P, const char* __restrict__ aos, uint64_t stride, int n, Shape shape,
                   unsigned long long* __restrict__ zbuf, Queue* __restrict__ queue) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * kRasterWarps + (threadIdx.x >> 5)) * shape.per_warp + lane;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane < shape.per_warp && i < n)
        q = project(P, reinterpret_cast<const float*>(aos + (uint64_t)i * stride));
    Sprite me(P, q, (int)i);
    const int count = me.nx * me.ny;
    bool whole = count > shape.lane_pixels;
    const bool large = count > shape.warp_pixels;
    if (__syncthreads_or(large)) {  // one reservation per block: 1 ns each on one address
        __shared__ uint32_t sums[kRasterWarps + 1];
        __shared__ unsigned long long wanted, from;
        uint32_t parts = large ? me.parts(kMaxParts) : 0u;
        uint32_t below = block_prefix(parts, sums);
        if (threadIdx.x == 0)
            wanted = atomicAdd(&queue->wanted, (unsigned long long)sums[kRasterWarps]);
        __syncthreads();
        if (wanted >= kWantedFew) {
            parts = large ? me.parts(wanted < kWantedMany ? 16 : 4) : 0u;
            below = block_prefix(parts, sums);
        }
        if (threadIdx.x == 0) from = atomicAdd(&queue->count, (unsigned long long)sums[kRasterWarps]);
        __syncthreads();
        const unsigned long long at = from + below;
        if (large) whole = at + parts > kQueue;  // no room: the slots that exist hold nothing
        for (uint32_t k = 0; k < parts && at + k < kQueue; ++k)
            queue->part[at + k] =
                whole ? kNoPart : (unsigned long long)(parts << 8 | k) << 32 | (uint32_t)i;
    }
    if (count <= shape.lane_pixels) me.draw_nearer(P, zbuf);
    unsigned big = __ballot_sync(0xffffffffu, whole);
    while (big) {
        const int src = __ffs(big) - 1;
        big &= big - 1;
        Sprite other = me;
        other.q.x = __shfl_sync(0xffffffffu, me.q.x, src);
        other.q.y = __shfl_sync(0xffffffffu, me.q.y, src);
        other.q.w = __shfl_sync(0xffffffffu, me.q.w, src);
        other.key = __shfl_sync(0xffffffffu, me.key, src);
        other.x0 = __shfl_sync(0xffffffffu, me.x0, src);
        other.y0 = __shfl_sync(0xffffffffu, me.y0, src);
        other.nx = __shfl_sync(0xffffffffu, me.nx, src);
        other.ny = __shfl_sync(0xffffffffu, me.ny, src);
        other.draw(P, zbuf, lane, 32);
    }
    let_next_start();
}

// The queued parts, a warp each (pass 2 empties the queue).
__global__ void __launch_bounds__(256)
    k_splat_large(SplatParams P, const char* __restrict__ aos, uint64_t stride,
                  unsigned long long* __restrict__ zbuf, const Queue* __restrict__ queue) {
    akua::pdl::wait_for_previous(aos, zbuf, queue);
    let_next_start();
    const uint32_t count = (uint32_t)min(__ldcg(&queue->count), (unsigned long long)kQueue);
    const uint32_t warps = gridDim.x * (blockDim.x / 32);
    const int lane = threadIdx.x & 31;
    for (uint32_t e = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); e < count; e += warps) {
        const unsigned long long part = __ldcg(&queue->part[e]);
        if (part == kNoPart) continue;
        const uint32_t i = (uint32_t)part;
        const int k = (int)(part >> 32) & 0xff, parts = (int)(part >> 40);  // parts is at least 1
        const Sprite s(P, project(P, reinterpret_cast<const float*>(aos + (uint64_t)i * stride)), (int)i);
        s.draw(P, zbuf, 32 * k + lane, 32 * parts);
    }
}

__device__ __forceinline__ uint32_t to_u8(float v) {
    return (uint32_t)(fminf(fmaxf(v, 0.0f), 1.0f) * 255.0f + 0.5f);
}

// Row 0 of the image is the top of the window (window y = height - 1).
__global__ void __launch_bounds__(256)
    k_splat_resolve(SplatParams P, const char* __restrict__ aos, uint64_t stride,
                    unsigned long long* __restrict__ zbuf, Queue* __restrict__ queue,
                    uint32_t* __restrict__ rgba) {
    akua::pdl::wait_for_previous(aos, zbuf, queue);
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) queue->count = queue->wanted = 0ull;  // for the next frame
    if (p >= P.width * P.height) return;
    const int px = p % P.width, py = p / P.width;
    const unsigned long long key = __ldcg(zbuf + p);  // not an older one in this SM's L1
    float c[4] = {0.15f, 0.15f, 0.18f, 1.0f};
    if (key != kEmpty) {
        zbuf[p] = kEmpty;  // for the next frame
        const uint32_t i = (uint32_t)(key & 0xFFFFFFFFull);
        const float* r = reinterpret_cast<const float*>(aos + (uint64_t)i * stride);
        const float4 q = project(P, r);
        const float ox = (((float)px + 0.5f) - q.x) / q.w;   // pointCoord.s - 0.5
        const float oy = -(((float)py + 0.5f) - q.y) / q.w;  // pointCoord.t - 0.5 (t downwards)
        float dist;
        const float a = frag_alpha(ox, oy, &dist);
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = r[22 + k] * a;
    }
    rgba[(size_t)(P.height - 1 - py) * P.width + px] =
        to_u8(c[0]) | (to_u8(c[1]) << 8) | (to_u8(c[2]) << 16) | (to_u8(c[3]) << 24);
}

// Particles per warp: the most (a power of two, at most 32) at which the warps still fill the chip
// once, 32 of them per SM.  (64 of them: 100,000 particles with small sprites 20.5 us against 16.5, 120,000
// with sprites of 5 pixels across 31 against 33.)
int splat_per_warp(int n, int sms) {
    int w = 1;
    while (w < 32 && (int64_t)n >= 2ll * w * 32 * sms) w *= 2;
    return w;
}

// Up to 64 warps of 32 particles per SM a frame lasts as long as its warps' chains, so few pixels go
// one after another and sprites go to the queue early; beyond that it is bound by atomics, and a lane's
// reads save them.  us with 9 and 64 pixels per lane: 120,000 sprites of 5 across 33 and 45, 300,000 of
// 9 across 90 and 118, but 1M of 3 to 5 132 and 92.  With 96 and 256 pixels per warp: the eye in front
// of 100,000 particles 33 and 41, among 300,000 35 and 45, but 1M sprites of 12 across 551 (128 pixels)
// and 424.
Shape splat_shape(int n, int sms) {
    const int w = splat_per_warp(n, sms);
    const bool crowded = n > 64ll * 32 * sms;
    const int lane = std::min(2 * w, crowded ? 64 : 9);
    return {w, lane, std::max(lane, crowded ? 256 : 96)};
}

// A launch that may begin while the stream's previous kernel ends (the kernel waits for it).
template <class... Args>
void launch_after(void (*kernel)(Args...), unsigned blocks, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

int status_of(cudaError_t e) {
    if (e == cudaSuccess) return AKUA_OK;
    if (e == cudaErrorMemoryAllocation) return AKUA_ERR_OUT_OF_MEMORY;
    return AKUA_ERR_CUDA;
}

// column-major 4x4 helpers in double
void mat_mul(const double* a, const double* b, double* out) {  // out = a * b
    for (int c = 0; c < 4; ++c)
        for (int r = 0; r < 4; ++r) {
            double s = 0.0;
            for (int k = 0; k < 4; ++k) s += a[4 * k + r] * b[4 * c + k];
            out[4 * c + r] = s;
        }
}

void normalize3(double* v) {
    const double l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    for (int k = 0; k < 3; ++k) v[k] /= l;
}

void cross3(const double* a, const double* b, double* out) {
    out[0] = a[1] * b[2] - a[2] * b[1];
    out[1] = a[2] * b[0] - a[0] * b[2];
    out[2] = a[0] * b[1] - a[1] * b[0];
}

bool finite_camera(const akua_camera* c) {
    for (int k = 0; k < 3; ++k)
        if (!std::isfinite(c->position[k]) || !std::isfinite(c->gaze[k]) || !std::isfinite(c->up[k]))
            return false;
    return std::isfinite(c->fovDegrees) && c->fovDegrees > 0.0f && c->fovDegrees < 180.0f &&
           c->nearZ > 0.0f && c->farZ > c->nearZ;
}

}  // namespace

struct akua_splat {
    int device = 0;
    int sms = 1;
    int width = 0, height = 0;
    unsigned long long* zbuf = nullptr;  // empty between frames
    Queue* queue = nullptr;
    bool dirty = false;  // a frame was not launched whole: they may not be
};

extern "C" {

void akua_camera_default(akua_camera* c) {
    if (!c) return;
    // CameraConfig.h:8-16 (yaw -90, pitch 0: gaze (0, 0, -1)); Application.cpp:17-18
    c->position[0] = 3.0f; c->position[1] = 2.0f; c->position[2] = 6.0f;
    c->gaze[0] = 0.0f; c->gaze[1] = 0.0f; c->gaze[2] = -1.0f;
    c->up[0] = 0.0f; c->up[1] = 1.0f; c->up[2] = 0.0f;
    c->fovDegrees = 45.0f;
    c->nearZ = 0.1f;
    c->farZ = 160.0f;
}

int akua_camera_matrices(const akua_camera* cam, float aspect, float* view, float* projection,
                         float* viewProjection) {
    if (!cam || !finite_camera(cam) || !(aspect > 0.0f)) return AKUA_ERR_INVALID_ARGUMENT;
    double f[3] = {cam->gaze[0], cam->gaze[1], cam->gaze[2]};
    normalize3(f);
    double wu[3] = {cam->up[0], cam->up[1], cam->up[2]};
    double s[3], u[3];
    cross3(f, wu, s);
    normalize3(s);
    cross3(s, f, u);
    const double e[3] = {cam->position[0], cam->position[1], cam->position[2]};
    double V[16] = {0};
    for (int k = 0; k < 3; ++k) {
        V[4 * k + 0] = s[k];
        V[4 * k + 1] = u[k];
        V[4 * k + 2] = -f[k];
    }
    V[12] = -(s[0] * e[0] + s[1] * e[1] + s[2] * e[2]);
    V[13] = -(u[0] * e[0] + u[1] * e[1] + u[2] * e[2]);
    V[14] = f[0] * e[0] + f[1] * e[1] + f[2] * e[2];
    V[15] = 1.0;
    const double t = std::tan(0.5 * (double)cam->fovDegrees * 3.14159265358979323846 / 180.0);
    const double zn = cam->nearZ, zf = cam->farZ;
    double Pm[16] = {0};
    Pm[0] = 1.0 / ((double)aspect * t);
    Pm[5] = 1.0 / t;
    Pm[10] = -(zf + zn) / (zf - zn);
    Pm[11] = -1.0;
    Pm[14] = -(2.0 * zf * zn) / (zf - zn);
    double VP[16];
    mat_mul(Pm, V, VP);
    for (int k = 0; k < 16; ++k) {
        if (view) view[k] = (float)V[k];
        if (projection) projection[k] = (float)Pm[k];
        if (viewProjection) viewProjection[k] = (float)VP[k];
    }
    return AKUA_OK;
}

int akua_splat_create(int32_t width, int32_t height, akua_splat** out) {
    if (!out || width <= 0 || height <= 0 || (int64_t)width * height > (1ll << 28))
        return AKUA_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    akua_splat* r = new (std::nothrow) akua_splat();
    if (!r) return AKUA_ERR_OUT_OF_MEMORY;
    r->width = width;
    r->height = height;
    cudaGetDevice(&r->device);
    cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, r->device);
    const size_t bytes = sizeof(unsigned long long) * (size_t)width * height;
    cudaError_t e = cudaMalloc(&r->zbuf, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&r->queue, sizeof(Queue));
    if (e == cudaSuccess) e = cudaMemset(r->zbuf, 0xFF, bytes);
    if (e == cudaSuccess) e = cudaMemset(r->queue, 0, offsetof(Queue, part));
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // any stream may render next
    if (e != cudaSuccess) {
        cudaFree(r->zbuf);
        cudaFree(r->queue);
        delete r;
        cudaGetLastError();
        return status_of(e);
    }
    *out = r;
    return AKUA_OK;
}

int akua_splat_destroy(akua_splat* r) {
    if (!r) return AKUA_ERR_INVALID_ARGUMENT;
    cudaDeviceSynchronize();
    cudaFree(r->zbuf);
    cudaFree(r->queue);
    delete r;
    return AKUA_OK;
}

int akua_splat_render(akua_splat* r, const void* particles, size_t stride, int32_t n,
                      const akua_camera* camera, uint32_t* rgba, void* stream) {
    if (!r || !camera || !rgba || n < 0 || (n > 0 && !particles) ||
        stride < sizeof(akua_particle) || stride % 4 != 0)
        return AKUA_ERR_INVALID_ARGUMENT;
    SplatParams P{};
    P.width = r->width;
    P.height = r->height;
    int rc = akua_camera_matrices(camera, (float)r->width / (float)r->height, nullptr, nullptr,
                                  P.vp);
    if (rc != AKUA_OK) return rc;
    for (int k = 0; k < 3; ++k) P.eye[k] = camera->position[k];
    cudaStream_t st = (cudaStream_t)stream;
    const size_t pixels = (size_t)r->width * r->height;
    if (r->dirty) {  // the last frame failed between its first and its last launch
        cudaError_t e = cudaMemsetAsync(r->zbuf, 0xFF, sizeof(unsigned long long) * pixels, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(r->queue, 0, offsetof(Queue, part), st);
        if (e != cudaSuccess) return status_of(e);
    }
    const char* aos = static_cast<const char*>(particles);
    if (n > 0) {
        const Shape shape = splat_shape(n, r->sms);
        const int per_block = kRasterWarps * shape.per_warp;
        k_splat_raster<<<(unsigned)((n + (int64_t)per_block - 1) / per_block), 32 * kRasterWarps, 0, st>>>(
            P, aos, stride, n, shape, r->zbuf, r->queue);
        launch_after(k_splat_large, 8 * r->sms, st, P, aos, (uint64_t)stride, r->zbuf,
                     static_cast<const Queue*>(r->queue));
    }
    launch_after(k_splat_resolve, (unsigned)((pixels + 255) / 256), st, P, aos, (uint64_t)stride,
                 r->zbuf, r->queue, rgba);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        r->dirty = true;
    } else if (r->dirty) {  // cleared now, unless the stream is being captured and nothing has run
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
        if (cudaStreamIsCapturing(st, &capture) == cudaSuccess)
            r->dirty = capture != cudaStreamCaptureStatusNone;
    }
    return status_of(e);
}

}  // extern "C"
