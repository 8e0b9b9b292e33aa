// The symmetric pair kernel's sums (pair.cu) for layouts of few block pairs.
//
// One CTA per pair of 1024-body blocks takes a CTA 110-140 us whatever the
// rest of the chip does: 10,007 bodies are 55 of them, and two thirds of the
// SMs have none.  Here the two sides of a block pair are formed separately,
// one-sided, each by many CTAs, with the partial sums of the pair kernel: every
// FP32 chain has the pair kernel's terms in its order, so the results agree
// with it to the rounding of the fixed-point sums, and a layout that grows
// across the line between the two kernels keeps its numbers.
//
//   * i side (kind 0): NT x KI bodies of a block against one later block (or
//     their own), two chains per body (the even and the odd 32-body
//     sub-chunks) over the block's tiles, lane l starting each sub-chunk at
//     its body l: pair_tile's i-side sums without the reactions.
//   * j side (kind 1): the reactions of one earlier block on a 128-body tile.
//     Warp w of four forms the chain of that warp's 256 i bodies on the four
//     bodies of lane l: at step s the i bodies of lane (l - s) mod 32, k =
//     0..7, in the order in which pair_tile hands a reaction from lane to
//     lane.  The four warps' sums meet in shared memory and add up in order.
//
// Every pair of different blocks is then evaluated twice (22 packed FMA-pipe
// operations for the two instead of 14), which is why larger layouts, whose
// block pairs fill the chip, run the pair kernel.  Bound by the latency of a
// CTA's chains at the small end (512 packed steps, 20 us, with one body per
// thread), by shared-memory loads (6-10 per step for one or two bodies) and
// the FP32 pipe at the large one.  us per acceleration pass, pair kernel ->
// this (events around the call): 117 -> 25 at 3,072 bodies, 117 -> 33 at 6,144,
// 139 -> 63 at 10,007 (masses and softenings per body; 68 without the forms of
// one mass and softening per tile), 148 -> 97 at 12,500, 115 -> 96 at 13,312,
// 219 -> 189 at 20,000; the planner has the lines.
#include <cstdint>

#include "khrr_internal.h"
#include "pair_math.cuh"

namespace khrr {
namespace {

constexpr int NT = kPairThreads;   // 128
constexpr int K = kPairBodies;     // i bodies per thread of the pair kernel
constexpr int JT = kPairTile;      // 128
constexpr int W = NT / 32;

// One block's bodies in shared memory: x, y, z, [m], [h].
template <unsigned F>
struct SmallShape {
    static constexpr bool UNIF = F & kUnif, ACC = F & kAcc, PHI = F & kPhi, BMASS = F & kBMass;
    static constexpr int NC = (ACC ? 3 : 0) + (PHI ? 1 : 0);
    static constexpr int NCOMP = 3 + (BMASS ? 0 : 1) + (UNIF ? 0 : 1);
    static constexpr int kOffM = 3, kOffH = BMASS ? 3 : 4;
};

// The pair term of packed j bodies (X2, ...) and one i body (negated
// coordinates, duplicated): d, r^-1 and r^-3, operation for operation as in
// pair_tile.
template <bool UNIF>
__device__ __forceinline__ void pair_term(float2 X2, float2 Y2, float2 Z2, float2 H2, float2 nx, float2 ny, float2 nz,
                                          float2 hi, float2 e2, float2& dx, float2& dy, float2& dz, float2& inv,
                                          float2& i3) {
    dx = __fadd2_rn(X2, nx);
    dy = __fadd2_rn(Y2, ny);
    dz = __fadd2_rn(Z2, nz);
    float2 r2 = UNIF ? e2 : __fadd2_rn(H2, hi);
    r2 = __ffma2_rn(dx, dx, r2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    inv = f2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    i3 = __fmul2_rn(inv, __fmul2_rn(inv, inv));
}

// One tile of the i side (kind 0).  ONE: the tile's masses are all mt and its
// softenings with the warp's bodies' add up to e2; the same numbers as the
// general form without reading and adding them per pair.
template <unsigned F, int KI, bool ONE>
__device__ __forceinline__ void side_tile(const float (&sb)[SmallShape<F>::NCOMP][kPairBlock], int t0, int lane,
                                          const float2 (&nx)[KI], const float2 (&ny)[KI], const float2 (&nz)[KI],
                                          const float2 (&hi)[KI], float2 e2, float2 mt,
                                          float2 (&ai)[SmallShape<F>::NC][KI]) {
    using S = SmallShape<F>;
    constexpr bool UNIF = S::UNIF || ONE, ACC = S::ACC, PHI = S::PHI, BMASS = S::BMASS;
    constexpr int CP = S::NC - 1;
    constexpr int kU = 4 / KI;  // steps in flight: the chains leave only the last FMA serial
#pragma unroll 1
    for (int c0 = 0; c0 < JT; c0 += 64) {
#pragma unroll kU
        for (int s = 0; s < 32; ++s) {
            const int ja = t0 + c0 + ((lane + s) & 31), jb = ja + 32;
            const float2 X2 = f2(sb[0][ja], sb[0][jb]), Y2 = f2(sb[1][ja], sb[1][jb]);
            const float2 Z2 = f2(sb[2][ja], sb[2][jb]);
            const float2 M2 = BMASS ? f2(1.f, 1.f) : ONE ? mt : f2(sb[S::kOffM][ja], sb[S::kOffM][jb]);
            const float2 H2 = UNIF ? f2(0.f, 0.f) : f2(sb[S::kOffH][ja], sb[S::kOffH][jb]);
#pragma unroll
            for (int k = 0; k < KI; ++k) {
                float2 dx, dy, dz, inv, i3;
                pair_term<UNIF>(X2, Y2, Z2, H2, nx[k], ny[k], nz[k], hi[k], e2, dx, dy, dz, inv, i3);
                if (ACC) {
                    const float2 fi = BMASS ? i3 : __fmul2_rn(M2, i3);
                    ai[0][k] = __ffma2_rn(dx, fi, ai[0][k]);
                    ai[1][k] = __ffma2_rn(dy, fi, ai[1][k]);
                    ai[2][k] = __ffma2_rn(dz, fi, ai[2][k]);
                }
                if (PHI) ai[CP][k] = BMASS ? __fadd2_rn(ai[CP][k], inv) : __ffma2_rn(M2, inv, ai[CP][k]);
            }
        }
    }
}

// The chains of the j side (kind 1): the block's n bodies (the warp's 32 of
// every 128) on the lane's four.  ONE as above, mt the block's mass.
template <unsigned F, bool ONE>
__device__ __forceinline__ void reaction_chains(const float (&sb)[SmallShape<F>::NCOMP][kPairBlock], int n, int lane,
                                                int warp, const float2 (&X2)[2], const float2 (&Y2)[2],
                                                const float2 (&Z2)[2], const float2 (&H2)[2], float2 e2, float2 mt,
                                                float2 (&r)[SmallShape<F>::NC][2]) {
    using S = SmallShape<F>;
    constexpr bool UNIF = S::UNIF || ONE, ACC = S::ACC, PHI = S::PHI, BMASS = S::BMASS;
    constexpr int CP = S::NC - 1;
#pragma unroll 1
    for (int s = 0; s < 32; ++s) {
        const int li = warp * 32 + ((lane - s) & 31);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int q = k * NT + li;
            if (k * NT >= n) break;  // blocks are whole tiles
            const float2 nx = f2(sb[0][q], sb[0][q]), ny = f2(sb[1][q], sb[1][q]), nz = f2(sb[2][q], sb[2][q]);
            const float2 mi = BMASS ? f2(1.f, 1.f) : ONE ? mt : f2(sb[S::kOffM][q], sb[S::kOffM][q]);
            const float2 hi = UNIF ? f2(0.f, 0.f) : f2(sb[S::kOffH][q], sb[S::kOffH][q]);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float2 dx, dy, dz, inv, i3;
                pair_term<UNIF>(X2[p], Y2[p], Z2[p], H2[p], nx, ny, nz, hi, e2, dx, dy, dz, inv, i3);
                if (ACC) {
                    const float2 fj = BMASS ? i3 : __fmul2_rn(mi, i3);
                    r[0][p] = __ffma2_rn(dx, fj, r[0][p]);
                    r[1][p] = __ffma2_rn(dy, fj, r[1][p]);
                    r[2][p] = __ffma2_rn(dz, fj, r[2][p]);
                }
                if (PHI) r[CP][p] = BMASS ? __fadd2_rn(r[CP][p], inv) : __ffma2_rn(mi, inv, r[CP][p]);
            }
        }
    }
}

template <unsigned F, int KI>
__global__ void __launch_bounds__(NT) pair_small_kernel(const PairArgs a, const SmallItem* __restrict__ items) {
    using S = SmallShape<F>;
    constexpr bool UNIF = S::UNIF, ACC = S::ACC, PHI = S::PHI, BMASS = S::BMASS;
    constexpr int NC = S::NC, CP = NC - 1;
    static_assert(NC > 0, "nothing to accumulate");
    __shared__ float sb[S::NCOMP][kPairBlock];
    __shared__ float jw[W][NC][JT];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SmallItem w = items[blockIdx.x];
    const float2 e2 = f2(a.h_uniform + a.h_uniform, a.h_uniform + a.h_uniform);

    // The block that streams past: the j block (kind 0) or the i block (kind
    // 1, negated coordinates; bodies past its end have no mass, and are not
    // visited in the block-mass form).
    const int sbeg = w.kind ? w.i_begin : w.j_begin, n = (w.kind ? w.i_end : w.j_end) - sbeg;
    for (int q = tid; q < n; q += NT) {
        const float x = a.sh.x[sbeg + q], y = a.sh.y[sbeg + q], z = a.sh.z[sbeg + q];
        sb[0][q] = w.kind ? -x : x;
        sb[1][q] = w.kind ? -y : y;
        sb[2][q] = w.kind ? -z : z;
        if (!BMASS) sb[S::kOffM][q] = a.sh.m[sbeg + q];
        if (!UNIF) sb[S::kOffH][q] = a.sh.h[sbeg + q];
    }
    __syncthreads();

    if (w.kind == 0) {
        float2 nx[KI], ny[KI], nz[KI], hi[KI], ai[NC][KI];
        float rh[PHI ? NC : 1][KI], rl[PHI ? NC : 1][KI];
#pragma unroll
        for (int k = 0; k < KI; ++k) {
            const int i = w.i_begin + k * NT + tid;
            const bool in = i < w.i_end;
            const float x = in ? -a.sh.x[i] : 0.f, y = in ? -a.sh.y[i] : 0.f, z = in ? -a.sh.z[i] : 0.f;
            const float h = UNIF ? 0.f : (in ? a.sh.h[i] : 1.f);
            nx[k] = f2(x, x);
            ny[k] = f2(y, y);
            nz[k] = f2(z, z);
            hi[k] = f2(h, h);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                ai[c][k] = f2(0.f, 0.f);
                if (PHI) rh[c][k] = rl[c][k] = 0.f;
            }
        }
        const float mt = BMASS ? a.tile_mass[w.j_begin / JT] : 1.f;
        const float h0 = __shfl_sync(0xffffffffu, hi[0].x, 0);
        bool one = true;  // the warp's bodies share a softening (lanes past the end have none)
#pragma unroll
        for (int k = 0; k < KI; ++k) one = one && w.i_begin + k * NT + tid < w.i_end && hi[k].x == h0;
        one = __all_sync(0xffffffffu, one);
        for (int t0 = 0; t0 < n; t0 += JT) {
            // One mass and one softening in the tile?
            float ht = 0.f, m1 = 1.f;
            bool t_one = one && !(UNIF && BMASS);
            if (t_one) {
                if (!UNIF) ht = sb[S::kOffH][t0];
                if (!BMASS) m1 = sb[S::kOffM][t0];
#pragma unroll
                for (int q = 0; q < JT; q += 32) {
                    if (!UNIF) t_one = t_one && sb[S::kOffH][t0 + q + lane] == ht;
                    if (!BMASS) t_one = t_one && sb[S::kOffM][t0 + q + lane] == m1;
                }
                t_one = __all_sync(0xffffffffu, t_one);
            }
            if (t_one)
                side_tile<F, KI, true>(sb, t0, lane, nx, ny, nz, hi, UNIF ? e2 : __fadd2_rn(f2(ht, ht), hi[0]),
                                       f2(m1, m1), ai);
            else
                side_tile<F, KI, false>(sb, t0, lane, nx, ny, nz, hi, e2, f2(1.f, 1.f), ai);
            if (PHI) {  // the potential variants fold every tile
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int k = 0; k < KI; ++k) {
                        const float v = ai[c][k].x + ai[c][k].y;
                        two_sum_into(rh[c][k], rl[c][k], BMASS ? mt * v : v);
                        ai[c][k] = f2(0.f, 0.f);
                    }
            }
        }
#pragma unroll
        for (int k = 0; k < KI; ++k) {
            const int i = w.i_begin + k * NT + tid;
            if (i >= w.i_end || i >= w.real_end) continue;
            const FxScale sc = a.scale[i / JT];
            auto sum = [&](int c, double scale) {
                if (PHI) return to_fx(rh[c][k], scale) + to_fx(rl[c][k], scale);
                const float v = ai[c][k].x + ai[c][k].y;
                if (!BMASS) return to_fx(v, scale);
                // The pair kernel's first fold: the product and its rounding.
                const float hi = __fmul_rn(mt, v);
                return to_fx(hi, scale) + to_fx(fmaf(mt, v, -hi), scale);
            };
            if (ACC) {
                fx_add(a.fx + i, sum(0, sc.acc));
                fx_add(a.fx + a.npad + i, sum(1, sc.acc));
                fx_add(a.fx + 2 * a.npad + i, sum(2, sc.acc));
            }
            if (PHI) fx_add(a.fx + 3 * a.npad + i, sum(CP, sc.phi));
        }
        return;
    }

    // The lane's bodies lane, lane + 32 (pair 0) and lane + 64, lane + 96 (1).
    float2 X2[2], Y2[2], Z2[2], H2[2], r[NC][2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const int ja = w.j_begin + 64 * p + lane, jb = ja + 32;
        X2[p] = f2(a.sh.x[ja], a.sh.x[jb]);
        Y2[p] = f2(a.sh.y[ja], a.sh.y[jb]);
        Z2[p] = f2(a.sh.z[ja], a.sh.z[jb]);
        H2[p] = UNIF ? f2(0.f, 0.f) : f2(a.sh.h[ja], a.sh.h[jb]);
#pragma unroll
        for (int c = 0; c < NC; ++c) r[c][p] = f2(0.f, 0.f);
    }
    // One softening among the tile's bodies and the warp's of the block, and one
    // mass among the latter?  (A block is whole tiles.)
    float hb = 0.f, m1 = 1.f;
    bool one = !(UNIF && BMASS);
    if (one) {
        const float hj = __shfl_sync(0xffffffffu, H2[0].x, 0);
        if (!UNIF) hb = sb[S::kOffH][warp * 32];
        if (!BMASS) m1 = sb[S::kOffM][warp * 32];
        if (!UNIF) one = H2[0].x == hj && H2[0].y == hj && H2[1].x == hj && H2[1].y == hj;
        for (int q = warp * 32 + lane; q < n; q += NT) {
            if (!UNIF) one = one && sb[S::kOffH][q] == hb;
            if (!BMASS) one = one && sb[S::kOffM][q] == m1;
        }
        one = __all_sync(0xffffffffu, one);
    }
    if (one)
        reaction_chains<F, true>(sb, n, lane, warp, X2, Y2, Z2, H2, UNIF ? e2 : __fadd2_rn(H2[0], f2(hb, hb)), f2(m1, m1),
                                 r);
    else
        reaction_chains<F, false>(sb, n, lane, warp, X2, Y2, Z2, H2, e2, f2(1.f, 1.f), r);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            jw[warp][c][64 * p + lane] = r[c][p].x;
            jw[warp][c][64 * p + lane + 32] = r[c][p].y;
        }
    __syncthreads();
    const int j = w.j_begin + tid;
    if (j >= w.real_end) return;
    const float mI = BMASS ? a.tile_mass[w.i_begin / JT] : 1.f;
    const FxScale sc = a.scale[w.j_begin / JT];
    auto total = [&](int c) {
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < W; ++q) v += jw[q][c][tid];
        return v;
    };
    if (ACC) {
        fx_add(a.fx + j, to_fx(-mI * total(0), sc.acc));
        fx_add(a.fx + a.npad + j, to_fx(-mI * total(1), sc.acc));
        fx_add(a.fx + 2 * a.npad + j, to_fx(-mI * total(2), sc.acc));
    }
    if (PHI) fx_add(a.fx + 3 * a.npad + j, to_fx(mI * total(CP), sc.phi));
}

template <unsigned F>
cudaError_t launch(const PairArgs& a, const SmallItem* items, int n, int ki, cudaStream_t s) {
    if (ki == 1) pair_small_kernel<F, 1><<<n, NT, 0, s>>>(a, items);
    else pair_small_kernel<F, 2><<<n, NT, 0, s>>>(a, items);
    return cudaGetLastError();
}

template <unsigned BASE>
cudaError_t launch_outputs(const ForceVariant* v, const PairArgs& a, const SmallItem* items, int n, int ki,
                           cudaStream_t s) {
    if (v->acc && v->phi) return launch<BASE | kAcc | kPhi>(a, items, n, ki, s);
    return v->acc ? launch<BASE | kAcc>(a, items, n, ki, s) : launch<BASE | kPhi>(a, items, n, ki, s);
}

}  // namespace

cudaError_t launch_pair_small(const ForceVariant* v, const PairArgs& a, const SmallItem* items, int n, int ki,
                              cudaStream_t s) {
    if (n < 1) return cudaSuccess;
    if (v->tile_mass)
        return v->uniform_eps ? launch_outputs<kUnif | kBMass>(v, a, items, n, ki, s)
                              : launch_outputs<kBMass>(v, a, items, n, ki, s);
    return v->uniform_eps ? launch_outputs<kUnif>(v, a, items, n, ki, s) : launch_outputs<0>(v, a, items, n, ki, s);
}

}  // namespace khrr
