// FP64 direct-sum gravity on sm_100a: the reference's own precision for
// ACCEL_kernel (nbody-kernel.cuh:89-142) and PHI_kernel (nbody-kernel.cuh:43-86),
// behind the state API (KHRR_FP64).  Every run reports its FP32 forces and
// its energy drift against this path.
//
// Two forms.  fp64_pair_kernel (the default; below) evaluates each unordered
// pair once for both bodies on the tapered plan of single tiles.  fp64_force_kernel
// (KHRR_FP64_ONESIDED=1) evaluates every ordered pair: the one-sided
// kernel's queue of WorkItems (system, i tile of 512 bodies, j chunk),
// pulled by a persistent grid with one atomic per item; each item writes its
// FP64 sums to its partial slot, which the corrector adds in FP64.
//
// Per item: 128 threads hold 4 i bodies each (FP64 position, softening and
// sums in registers); the chunk's j bodies pass through a double-buffered
// shared-memory tile of 128 (x, y, z, m, eps^2/2 as doubles), the next tile
// loaded into registers while the current one is evaluated, one barrier per
// tile.  Per pair: d (3 sub), r^2 = h_i + h_j + d.d (1 add, 3 fma), r^-1 =
// rsqrt (CUDA's double-precision function), m r^-3 (3 mul), the sums (3 fma,
// + 1 fma for the potential).  FP64-pipe bound: B200 runs FP64 at half the
// FP32 rate.
//
// Terms: the softening enters as (eps2_i + eps2_j) / 2, the self pair gives
// zero acceleration and m / eps to the potential, ghosts (zero mass) give
// nothing: the reference's sums, evaluated in IEEE double.
#include <cstdint>

#include "khrr_internal.h"

namespace khrr {
namespace {

#ifndef KHRR_F64_NT
#define KHRR_F64_NT 128
#endif
constexpr int NT = KHRR_F64_NT;   // threads per CTA
constexpr int K = kF64ITile / NT;  // i bodies per thread
constexpr int JT = 128;            // j bodies per shared-memory tile
constexpr int FP = (JT + NT - 1) / NT;  // j bodies each thread stages per tile
static_assert(NT * K == kF64ITile && JT == kPad && (JT % NT == 0 || NT % JT == 0), "tile shapes");

constexpr int kMinCtas = NT >= 128 ? 512 / NT : 4;  // resident CTAs per SM the registers aim at

template <bool ACC, bool PHI>
__global__ void __launch_bounds__(NT, kMinCtas) fp64_force_kernel(const F64Args a) {
    __shared__ double sx[2][JT], sy[2][JT], sz[2][JT], sm[2][JT], sh[2][JT];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_item = static_cast<int>(atomicAdd(a.queue, 1u));
        __syncthreads();
        const int it = s_item;
        if (it >= a.n_items) break;
        const WorkItem w = a.items[it];

        double xi[K], yi[K], zi[K], hi[K], ax[K], ay[K], az[K], ph[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = w.i_begin + k * NT + tid;
            const bool in = i < w.i_end;
            xi[k] = in ? a.pos[3 * static_cast<int64_t>(i)] : 0.0;
            yi[k] = in ? a.pos[3 * static_cast<int64_t>(i) + 1] : 0.0;
            zi[k] = in ? a.pos[3 * static_cast<int64_t>(i) + 2] : 0.0;
            hi[k] = in ? 0.5 * a.eps2[i] : 1.0;
            ax[k] = ay[k] = az[k] = ph[k] = 0.0;
        }

        const int ntiles = (w.j_end - w.j_begin) / JT;
        // Register copy of the next tile's bodies tid, tid + NT, ... (< JT).
        double nx[FP], ny[FP], nz[FP], nm[FP], nh[FP];
        auto fetch = [&](int t) {
#pragma unroll
            for (int q = 0; q < FP; ++q) {
                const int jj = tid + q * NT;
                if (jj >= JT) break;
                const int64_t j = w.j_begin + static_cast<int64_t>(t) * JT + jj;
                nx[q] = a.pos[3 * j];
                ny[q] = a.pos[3 * j + 1];
                nz[q] = a.pos[3 * j + 2];
                nm[q] = a.mass[j];
                nh[q] = 0.5 * a.eps2[j];
            }
        };
        fetch(0);
        for (int t = 0; t < ntiles; ++t) {
            const int b = t & 1;
#pragma unroll
            for (int q = 0; q < FP; ++q) {
                const int jj = tid + q * NT;
                if (jj >= JT) break;
                sx[b][jj] = nx[q];
                sy[b][jj] = ny[q];
                sz[b][jj] = nz[q];
                sm[b][jj] = nm[q];
                sh[b][jj] = nh[q];
            }
            __syncthreads();
            if (t + 1 < ntiles) fetch(t + 1);
#pragma unroll 2
            for (int jj = 0; jj < JT; ++jj) {
                const double xj = sx[b][jj], yj = sy[b][jj], zj = sz[b][jj], mj = sm[b][jj], hj = sh[b][jj];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const double dx = xj - xi[k], dy = yj - yi[k], dz = zj - zi[k];
                    double r2 = hi[k] + hj;
                    r2 = fma(dx, dx, r2);
                    r2 = fma(dy, dy, r2);
                    r2 = fma(dz, dz, r2);
                    const double inv = rsqrt(r2);
                    if (ACC) {
                        const double k3 = mj * (inv * inv * inv);
                        ax[k] = fma(dx, k3, ax[k]);
                        ay[k] = fma(dy, k3, ay[k]);
                        az[k] = fma(dz, k3, az[k]);
                    }
                    if (PHI) ph[k] = fma(mj, inv, ph[k]);
                }
            }
        }
        double4* out = a.part + static_cast<long long>(w.slot) * a.npad;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = w.i_begin + k * NT + tid;
            if (i < w.i_end) out[i] = make_double4(ax[k], ay[k], az[k], ph[k]);
        }
        // Every thread is done with the item (and s_item) before the next pull.
        __syncthreads();
    }
}

// The symmetric form of the same sums (the default FP64 pass): every
// unordered pair of a system evaluated once for both bodies, on a plan of its
// own (plan_pair_tiles: 1024-body blocks, a block row cut into chunks of
// 128-body tiles that taper to single ones, the block's own tiles one-sided).
// A CTA holds its i block in registers (128 threads x 8 bodies) and streams the
// chunk's j tiles of 128 bodies through a double-buffered shared-memory tile; the
// reaction on a j body is summed across a warp by handing it from lane to lane (lane l
// evaluates body (l + s) mod 32 of a 32-body sub-chunk at step s and passes
// its running reaction to lane l - 1), then across the 4 warps in shared
// memory, and added with FP64 atomics into the body's sums, as are the i
// block's sums every eighth tile and at the item's end.  The sums are FP64
// throughout; their order differs from the reference's j loop only at the
// level of FP64 rounding.
//
// A body's sum over the partials is kept in two doubles: every partial is cut
// at a multiple of the body's grid, coarse enough (2^-51 of the bound on its
// force) that the upper parts add up without rounding, and the lower parts, below 2^-52 of that bound, add up in the
// second.  So the number of partials, and the order the atomics land in, do
// not show in the result: relative RMS error against 80-bit sums 2.4e-16 with
// one double and chunks of eight tiles, 3.5e-16 with one double and these
// chunks, 1.0e-16 cut, at 49,152 bodies (5.3e-16, 1.9e-16, 1.6e-16 at 3,072).
//
// The kernel is bound by the FP64 pipe (64 lanes per SM and clock), so what
// counts is FP64 instructions per unordered pair:
//   * r^-3 from the hardware's reciprocal-square-root seed y0 (one XU
//     instruction on the upper word, relative error 2^-20) and the binomial
//     series of (1 - e)^(-3/2) in e = 1 - r2 y0^2 (y0^2 is exact, y0 having 21
//     significant bits), cut after e^2: the term left out is 35/16 e^3, below
//     2^-55 for |e| < 2^-19.  Six operations, and r^-1 = r2 r^-3 where the
//     potential is wanted too, instead of rsqrt() with its range handling and
//     two multiplies.
//   * where the i block has one mass and one softening and so has the j tile
//     (all but the tiles at a component's border and a ragged end), the
//     masses leave the pair term (applied once per sum) and h_i + h_j is a
//     constant: 18 operations per unordered pair (3 sub, 3 fma, 6, 6 fma)
//     against 21 with per-body masses and softenings.
// Per pass: 2.24 -> 1.57 ms at 49,152 bodies, 370 -> 130 us at 10,007 (the
// tapered plan: 55 block pairs left most SMs idle).
// The series needs r2 well inside the exponent range: tiles whose h or
// coordinates leave [2^-600, 2^580] and 2^290 in magnitude (or are not
// numbers) take rsqrt(), which handles every operand.
// Shape, measured (ms per pass at 131,072 bodies, accelerations / with the
// potential): 128 threads x 8 bodies, two CTAs per SM, step loop unrolled 8
// times 10.5 / 14.1, 4 times 10.8 / 13.0, twice 11.1 / 12.9, once 11.5 / 13.0;
// three CTAs (168 registers) 11.0 / 13.7 (before the cut sums); 256 x 4 11.3 /
// 12.6.  The kernel before, rsqrt() and per-body masses throughout: 14.5 /
// 16.0.  What bounds it: DFMA reads three 64-bit registers, and the register
// file delivers one a cycle (3.05 cycles for three different operands
// against 2.05 for two, measured on plain chains), so a pair costs 43
// register-read cycles where its 18 operations would issue in 36; the pass
// above takes 45.
constexpr int PNT = 128;                  // threads per CTA
constexpr int kF64PUnroll = 8, kF64PUnrollPhi = 2;
constexpr int PK = kPairBlock / PNT;      // i bodies per thread (8)
constexpr int PJT = kPairTile;            // j bodies per tile (128)
constexpr int PW = PNT / 32;              // warps (4)
static_assert(PNT * PK == kPairBlock && PJT == 128 && PJT % 32 == 0 && PNT >= PJT, "pair shapes");

constexpr double kSafePos = 0x1p290, kSafeHMin = 0x1p-600, kSafeHMax = 0x1p580;

__device__ __forceinline__ bool safe_body(double x, double y, double z, double h) {
    return fabs(x) < kSafePos && fabs(y) < kSafePos && fabs(z) < kSafePos && h > kSafeHMin && h < kSafeHMax;
}

__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// r^-3, and r^-1 where the potential needs it, of a normal r2 (see above).
template <bool PHI>
__device__ __forceinline__ void inverse_powers(double r2, double& inv, double& i3) {
    const double y0 = rsqrt_seed(r2);
    const double s = y0 * y0;
    const double e = fma(-r2, s, 1.0);
    const double c = s * y0;
    i3 = fma(c * e, fma(1.875, e, 1.5), c);
    if (PHI) inv = r2 * i3;
}

// Adds v into the pair of sums, cut at the grid 2^-52 c / 1.5.
__device__ __forceinline__ void add_cut(double* upper, int64_t lower, double v, double c) {
    const double u = (v + c) - c;
    const double l = v - u;
    atomicAdd(upper, u);
    atomicAdd(upper + lower, fabs(v) < 0x1p1000 ? l : 0.0);  // an infinite or overlarge v stays what it is
}
constexpr double kCutGrid = 0x1.8p62;  // times a tile's 2^-E (FxScale): 1.5 x 2^52 grids of 2^(10-E)

struct F64Tiles {
    double x[2][PJT], y[2][PJT], z[2][PJT], m[2][PJT], h[2][PJT];
};

// One staged tile against the thread's PK bodies.  SYM adds the reactions
// (jw[c][body] of the warp).  UNI: one mass and softening on either side, the
// sums without their masses, H = h_i + h_j.  SAFE: the series above.
template <bool ACC, bool PHI, bool SYM, bool UNI, bool SAFE>
__device__ __forceinline__ void fp64_pair_tile(const F64Tiles& T, int b, double H, double (*__restrict__ jw)[PJT],
                                               const double (&xi)[PK], const double (&yi)[PK], const double (&zi)[PK],
                                               const double (&hi)[PK], const double (&mi)[PK],
                                               double (&ai)[(ACC ? 3 : 0) + (PHI ? 1 : 0)][PK], int lane) {
    constexpr int NC = (ACC ? 3 : 0) + (PHI ? 1 : 0), CP = NC - 1;
    constexpr int kU = PHI ? kF64PUnrollPhi : kF64PUnroll;
    const int src = (lane + 1) & 31;
#pragma unroll 1
    for (int c0 = 0; c0 < PJT; c0 += 32) {
        double r[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) r[c] = 0.0;
#pragma unroll kU
        for (int s = 0; s < 32; ++s) {
            const int j = c0 + ((lane + s) & 31);
            const double xj = T.x[b][j], yj = T.y[b][j], zj = T.z[b][j];
            const double mj = UNI ? 1.0 : T.m[b][j], hj = UNI ? 0.0 : T.h[b][j];
#pragma unroll
            for (int k = 0; k < PK; ++k) {
                const double dx = xj - xi[k], dy = yj - yi[k], dz = zj - zi[k];
                double r2 = UNI ? H : hi[k] + hj;
                r2 = fma(dx, dx, r2);
                r2 = fma(dy, dy, r2);
                r2 = fma(dz, dz, r2);
                double inv = 0.0, i3 = 0.0;
                if (SAFE) {
                    inverse_powers<PHI>(r2, inv, i3);
                } else {
                    inv = rsqrt(r2);
                    i3 = inv * inv * inv;
                }
                if (ACC) {
                    const double fi = UNI ? i3 : mj * i3;
                    const double fj = UNI ? i3 : (SYM ? mi[k] * i3 : 0.0);
                    ai[0][k] = fma(dx, fi, ai[0][k]);
                    if (SYM) r[0] = fma(dx, fj, r[0]);
                    ai[1][k] = fma(dy, fi, ai[1][k]);
                    if (SYM) r[1] = fma(dy, fj, r[1]);
                    ai[2][k] = fma(dz, fi, ai[2][k]);
                    if (SYM) r[2] = fma(dz, fj, r[2]);
                }
                if (PHI) {
                    ai[CP][k] = UNI ? ai[CP][k] + inv : fma(mj, inv, ai[CP][k]);
                    if (SYM) r[CP] = UNI ? r[CP] + inv : fma(mi[k], inv, r[CP]);
                }
            }
            if (SYM) {
#pragma unroll
                for (int c = 0; c < NC; ++c) r[c] = __shfl_sync(0xffffffffu, r[c], src);
            }
        }
        if (SYM) {
#pragma unroll
            for (int c = 0; c < NC; ++c) jw[c][c0 + lane] = r[c];
        }
    }
}

template <bool ACC, bool PHI>
__global__ void __launch_bounds__(PNT, 2) fp64_pair_kernel(const F64PairArgs a) {
    constexpr int NC = (ACC ? 3 : 0) + (PHI ? 1 : 0), CP = NC - 1;
    __shared__ F64Tiles T;
    __shared__ double jw[PW][NC][PJT];
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t lower = 4 * a.npad;  // from a sum's upper part to its lower one
    for (;;) {
        if (tid == 0) s_item = static_cast<int>(atomicAdd(a.queue, 1u));
        __syncthreads();
        const int it = s_item;
        if (it >= a.n_items) break;
        const PairItem w = a.items[it];
        // The i bodies (index i_begin + k PNT + tid); lanes past the block's
        // end have no mass (and a positive softening term).
        double xi[PK], yi[PK], zi[PK], ai[NC][PK];
        bool safe_i = true;
#pragma unroll
        for (int k = 0; k < PK; ++k) {
            const int64_t i = w.i_begin + k * PNT + tid;
            const bool in = i < w.i_end;
            xi[k] = in ? a.pos[3 * i] : 0.0;
            yi[k] = in ? a.pos[3 * i + 1] : 0.0;
            zi[k] = in ? a.pos[3 * i + 2] : 0.0;
            safe_i = safe_i && safe_body(xi[k], yi[k], zi[k], in ? 0.5 * a.eps2[i] : 1.0);
#pragma unroll
            for (int c = 0; c < NC; ++c) ai[c][k] = 0.0;
        }
        // Whether the block is 1024 real bodies of one mass and softening.
        const double2 ci = a.tile_class[w.i_begin / PJT];
        bool uni_i = w.i_end - w.i_begin == kPairBlock && ci.y > 0.0;
        for (int q = 1; uni_i && q < kPairBlock / PJT; ++q) {
            const double2 cq = a.tile_class[w.i_begin / PJT + q];
            uni_i = cq.x == ci.x && cq.y == ci.y;
        }
        double scale_i = 1.0;  // the mass left out of the sums in ai
        // The sums so far, times the mass left out of them, into the bodies'
        // accumulators.
        auto flush = [&]() {
#pragma unroll
            for (int k = 0; k < PK; ++k) {
                const int64_t i = w.i_begin + k * PNT + tid;
                if (i < w.i_end && i < w.real_end) {
                    const FxScale sc = a.scale[i / PJT];
                    double* u = a.sums + i;
                    if (ACC) {
                        const double c = kCutGrid * sc.inv_acc;
                        add_cut(u, lower, scale_i * ai[0][k], c);
                        add_cut(u + a.npad, lower, scale_i * ai[1][k], c);
                        add_cut(u + 2 * a.npad, lower, scale_i * ai[2][k], c);
                    }
                    if (PHI) add_cut(u + 3 * a.npad, lower, scale_i * ai[CP][k], kCutGrid * sc.inv_phi);
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) ai[c][k] = 0.0;
            }
        };
        const int ntiles = (w.j_end - w.j_begin) / PJT;
        // Register copy of the next tile's body tid (threads < PJT).
        double nx = 0.0, ny = 0.0, nz = 0.0, nm = 0.0, nh = 1.0;
        auto fetch = [&](int t) {
            if (tid < PJT) {
                const int64_t j = w.j_begin + static_cast<int64_t>(t) * PJT + tid;
                nx = a.pos[3 * j];
                ny = a.pos[3 * j + 1];
                nz = a.pos[3 * j + 2];
                nm = a.mass[j];
                nh = 0.5 * a.eps2[j];
            }
        };
        fetch(0);
        for (int t = 0; t < ntiles; ++t) {
            const int b = t & 1;
            if (tid < PJT) {
                T.x[b][tid] = nx;
                T.y[b][tid] = ny;
                T.z[b][tid] = nz;
                T.m[b][tid] = nm;
                T.h[b][tid] = nh;
            }
            // The tile is staged; the last tile's reactions were read.
            const bool safe = !__syncthreads_or(!(safe_i && safe_body(nx, ny, nz, nh)));
            if (t + 1 < ntiles) fetch(t + 1);
            const int jt0 = w.j_begin + t * PJT;
            const bool sym = jt0 >= w.diag_end;
            const double2 cj = a.tile_class[jt0 / PJT];
            const bool uni = uni_i && safe && cj.y > 0.0;
            const double scale = uni ? cj.x : 1.0;
            if (scale != scale_i || (t > 0 && (t & 7) == 0)) {
                flush();
                scale_i = scale;
            }
            if (uni) {
                const double none[PK] = {};
                const double H = ci.y + cj.y;
                if (sym)
                    fp64_pair_tile<ACC, PHI, true, true, true>(T, b, H, jw[warp], xi, yi, zi, none, none, ai, lane);
                else
                    fp64_pair_tile<ACC, PHI, false, true, true>(T, b, H, jw[warp], xi, yi, zi, none, none, ai, lane);
            } else {
                double hi[PK], mi[PK];
#pragma unroll
                for (int k = 0; k < PK; ++k) {
                    const int64_t i = w.i_begin + k * PNT + tid;
                    hi[k] = i < w.i_end ? 0.5 * a.eps2[i] : 1.0;
                    mi[k] = i < w.i_end ? a.mass[i] : 0.0;
                }
                if (safe)
                    if (sym) fp64_pair_tile<ACC, PHI, true, false, true>(T, b, 0.0, jw[warp], xi, yi, zi, hi, mi, ai, lane);
                    else fp64_pair_tile<ACC, PHI, false, false, true>(T, b, 0.0, jw[warp], xi, yi, zi, hi, mi, ai, lane);
                else if (sym)
                    fp64_pair_tile<ACC, PHI, true, false, false>(T, b, 0.0, jw[warp], xi, yi, zi, hi, mi, ai, lane);
                else
                    fp64_pair_tile<ACC, PHI, false, false, false>(T, b, 0.0, jw[warp], xi, yi, zi, hi, mi, ai, lane);
            }
            if (sym) {
                __syncthreads();  // every warp's reactions of the tile are in jw
                if (tid < PJT) {
                    const int64_t j = jt0 + tid;
                    if (j < w.real_end) {
                        double s4[NC];
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            double v = 0.0;
#pragma unroll
                            for (int q = 0; q < PW; ++q) v += jw[q][c][tid];
                            s4[c] = uni ? ci.x * v : v;
                        }
                        // The reaction on j is minus the sum of m_i d / r^3
                        // (d = x_j - x_i); the potential's sum keeps its sign.
                        const FxScale sc = a.scale[jt0 / PJT];
                        double* u = a.sums + j;
                        if (ACC) {
                            const double c = kCutGrid * sc.inv_acc;
                            add_cut(u, lower, -s4[0], c);
                            add_cut(u + a.npad, lower, -s4[1], c);
                            add_cut(u + 2 * a.npad, lower, -s4[2], c);
                        }
                        if (PHI) add_cut(u + 3 * a.npad, lower, s4[CP], kCutGrid * sc.inv_phi);
                    }
                }
            }
        }
        flush();
        // Every thread is done with the item (and s_item) before the next pull.
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_fp64_force(const F64Args& a, bool acc, bool phi, int grid, cudaStream_t s) {
    if (a.n_items < 1) return cudaSuccess;
    if (acc && phi) fp64_force_kernel<true, true><<<grid, NT, 0, s>>>(a);
    else if (acc) fp64_force_kernel<true, false><<<grid, NT, 0, s>>>(a);
    else fp64_force_kernel<false, true><<<grid, NT, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_fp64_pair(const F64PairArgs& a, bool acc, bool phi, int grid, cudaStream_t s) {
    if (a.n_items < 1) return cudaSuccess;
    if (acc && phi) fp64_pair_kernel<true, true><<<grid, PNT, 0, s>>>(a);
    else if (acc) fp64_pair_kernel<true, false><<<grid, PNT, 0, s>>>(a);
    else fp64_pair_kernel<false, true><<<grid, PNT, 0, s>>>(a);
    return cudaGetLastError();
}

int fp64_pair_ctas(int sm_count) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fp64_pair_kernel<true, true>, PNT, 0) != cudaSuccess ||
        occ < 1)
        occ = 1;
    return occ * sm_count;
}

int fp64_force_ctas(int sm_count) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fp64_force_kernel<true, true>, NT, 0) != cudaSuccess ||
        occ < 1)
        occ = 1;
    return occ * sm_count;
}

}  // namespace khrr
