// Scalar pieces of the FP32 pair kernels (pair.cu, pair_small.cu).
#pragma once

#include <cstdint>

#include "tile_sums.cuh"

namespace khrr {
namespace {

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// A partial (FP32) as a fixed-point integer: times the power of two s,
// rounded to the nearest integer (exact for |v s| >= 2^24).
__device__ __forceinline__ long long to_fx(float v, double s) {
    return __double2ll_rn(static_cast<double>(v) * s);
}

// Integer atomic add without return (red.global.add.u64): two's complement
// makes the unsigned add a signed one.
__device__ __forceinline__ void fx_add(unsigned long long* p, long long v) {
    atomicAdd(p, static_cast<unsigned long long>(v));
}

// Kernel features (template bit mask).
constexpr unsigned kUnif = 1;   // every body has the same softening: no h array
constexpr unsigned kAcc = 2;    // accumulate accelerations
constexpr unsigned kPhi = 4;    // accumulate potentials
constexpr unsigned kBMass = 8;  // one mass per block: masses factored out

}  // namespace
}  // namespace khrr
