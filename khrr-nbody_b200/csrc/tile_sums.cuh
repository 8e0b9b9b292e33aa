// Compensated FP32 sums of the force kernels (force.cu, pair.cu, pair_small.cu)
// and of the one-sided kernel's partials per tile (integrate.cu, force.cu).
#pragma once

namespace khrr {
namespace {

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void two_sum_into(float& hi, float& lo, float p) {
    const float s = hi + p;
    const float bp = s - hi;
    const float e = (hi - (s - bp)) + (p - bp);
    hi = s;
    lo += e;
}

// The same of the product m p, which is not rounded on its own.
__device__ __forceinline__ void two_sum_into(float& hi, float& lo, float m, float p) {
    const float s = __fmaf_rn(m, p, hi);
    const float bp = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fmaf_rn(m, p, -bp));
    hi = s;
    lo = __fadd_rn(lo, e);
}

// One body's sums from its tiles' partials (ForceArgs::tiles): `chains` runs of
// consecutive tiles, each a compensated FP32 sum as one item's, the runs' FP64
// values added in order.
template <int AHEAD>
__device__ __forceinline__ double4 sum_tile_chains(const float4* __restrict__ tiles, long long npad, long long i,
                                                   int ntiles, int chains, const float* __restrict__ tile_mass) {
    double4 total = make_double4(0.0, 0.0, 0.0, 0.0);
    float h[4] = {0.f, 0.f, 0.f, 0.f}, l[4] = {0.f, 0.f, 0.f, 0.f};
    int chain = 0, end = ntiles / chains;  // the run's last tile + 1 (ntiles >= chains)
    for (int t0 = 0; t0 < ntiles; t0 += AHEAD) {
        float4 p[AHEAD];
        float m[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (t0 + k < ntiles) {
                p[k] = tiles[(t0 + k) * npad + i];
                m[k] = tile_mass ? tile_mass[t0 + k] : 1.0f;
            }
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if (t0 + k >= ntiles) break;
            const float v[4] = {p[k].x, p[k].y, p[k].z, p[k].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) two_sum_into(h[c], l[c], m[k], v[c]);
            if (t0 + k + 1 == end) {
                double d[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    d[c] = static_cast<double>(h[c]) + static_cast<double>(l[c]);
                    h[c] = l[c] = 0.f;
                }
                total.x += d[0];
                total.y += d[1];
                total.z += d[2];
                total.w += d[3];
                ++chain;
                end = (chain + 1) * ntiles / chains;
            }
        }
    }
    return total;
}

}  // namespace
}  // namespace khrr
