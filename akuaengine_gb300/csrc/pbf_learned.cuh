// Learned warm start of the Jacobi loop: per-particle features for the lambda network.
//
// The warm start replaces iteration 1's lambda (the one-step Jacobi estimate) by the network's
// prediction of the lambda a 20-iteration solve accumulates over the step (the sum of its
// iterations' lambdas, which is what drives the total position correction since delta-p is linear
// in lambda), blended with iteration 1's lambda by a calibrated factor.  Later iterations run the
// reference's update unchanged, so the plain iterated solver still corrects whatever the
// prediction leaves.
//
// Features of particle i at the start of the step, all by-products of iteration 1's density and
// lambda over the step's neighbour list (the walk writes them; no extra neighbour pass):
//   0 C_i = rho_i / rho0 - 1              4 the previous step's accumulated lambda
//   1 neighbour count / 32                5 |grad_i C_i| (large at the free surface)
//   2 S_i = sum_j |grad_j C_i|^2 + |grad_i C_i|^2 (the lambda denominator without epsilon)
//   3 lambda_i of iteration 1             6 grad_i C_i along gravity (which side is open)
//                                         7 |predicted velocity|
// All of them are functions of the state the step starts from, the same in plain and in
// warm-started runs (the record's own `lambda` field is not: it holds the last iteration's value).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pbf_device.cuh"

namespace akua {

constexpr int kFeatures = 8;

// `acc`: iteration 1's density/lambda accumulator of particle i (rho, sum of |grad_j C_i|^2 and
// sum_j m_j grad W_ij in gx, gy, gz).
template <class Acc>
__device__ __forceinline__ void write_features(const StepParams& p, const Acc& acc, float lam0,
                                               int count, float lprev, float speed, float* out) {
    const float ax = acc.gx * p.inv_rho0, ay = acc.gy * p.inv_rho0, az = acc.gz * p.inv_rho0;
    const float a2 = ax * ax + ay * ay + az * az;
    const float g2 = p.gravity[0] * p.gravity[0] + p.gravity[1] * p.gravity[1] +
                     p.gravity[2] * p.gravity[2];
    const float ig = g2 > 0.f ? rsqrtf(g2) : 0.f;
    const float along = (ax * p.gravity[0] + ay * p.gravity[1] + az * p.gravity[2]) * ig;
    float4* o = reinterpret_cast<float4*>(out);
    o[0] = make_float4(acc.rho * p.inv_rho0 - 1.0f, (float)count * (1.0f / 32.0f), acc.sum + a2,
                       lam0);
    o[1] = make_float4(lprev, sqrtf(a2), along, speed);
}

}  // namespace akua
