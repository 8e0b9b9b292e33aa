// FP64 predictor-corrector, external field and conservation sums on sm_100a.
//
// Replaces kernelNbody_integTime (nbody-kernel.cuh:144-193) with dev_fex
// (nbody-kernel.cuh:8-40), the reference's step sequencing
// (nbody/src/nbody.cu:1525-1582) and the host FP64 loop of result()
// (nbody/src/nbody.cu:797-833).  All of it is HBM-bound FP64 work.
//
// The time step is  predictor -> force -> corrector.  Because the corrector
// leaves x(t+dt) = x* and the next predictor only needs x(t+dt), v(t+dt) and
// a(t+dt) (plus fex at the same x), the corrector of step k and the predictor
// of step k+1 are fused into one pass ("kick-drift"), which also writes the
// FP32 shadow (x*, m) the next force pass reads.  The arithmetic is the
// reference's, operation for operation; this file is built with FMA
// contraction off so the results equal the reference's expressions evaluated
// in IEEE double.
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "khrr_internal.h"
#include "tile_sums.cuh"

namespace khrr {

FieldConsts make_field(double Mh, double a, double Rh, double Mb, double b, double Rb) {
    // Host constants as nbody/src/nbody.cu:1111-1120 derives them.
    FieldConsts f{};
    const double Rh2 = 3.0 * Rh;
    const double rcore1 = Rh / a;
    const double rbcore1 = 1.0 / b;
    const double rbcore2 = rbcore1 * rbcore1;
    const double root1 = std::sqrt(1.0 + (Rb * Rb) * rbcore2);
    f.a = a;
    f.b = b;
    f.Rb = Rb;
    f.Mb = Mb;
    f.Rh2 = Rh2;
    f.con = Mh / (rcore1 - std::atan(rcore1));
    f.const1 = Mb / (b * std::log(Rb * rbcore1 + root1) - Rb / root1);
    f.Mh_inf = Mh * (Rh2 / a - std::atan(Rh2 / a)) / (rcore1 - std::atan(rcore1));
    f.enabled = 1;
    return f;
}

namespace {

struct d3 {
    double x, y, z;
};

__device__ __forceinline__ d3 ld3(const double* p, int64_t i) {
    return d3{p[3 * i], p[3 * i + 1], p[3 * i + 2]};
}

__device__ __forceinline__ void st3(double* p, int64_t i, const d3& v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}

// dev_fex (nbody-kernel.cuh:8-40): static halo + bulge acceleration at p.
__device__ d3 fex(const FieldConsts& F, const d3& p) {
    if (!F.enabled) return d3{0.0, 0.0, 0.0};
    const double rr = sqrt(p.x * p.x + p.y * p.y + p.z * p.z);
    if (!(rr > 0.0)) return d3{0.0, 0.0, 0.0};
    const double rr3 = rr * rr * rr;
    const double rrcore = rr / F.a;
    const double rrbcore1 = rr / F.b;
    const double root1 = sqrt(1.0 + rrbcore1 * rrbcore1);
    const double forcehalo = rr < F.Rh2 ? -F.con * (rrcore - atan(rrcore)) / rr3 : -F.Mh_inf / rr3;
    const double forceblg1 =
        rr < F.Rb ? -F.const1 * (F.b * log(rrbcore1 + root1) - rr / root1) / rr3 : -F.Mb / rr3;
    const double s = forceblg1 + forcehalo;
    return d3{s * p.x, s * p.y, s * p.z};
}

// Positions of the FP32 shadow (its masses and softenings never change).
__device__ __forceinline__ void write_shadow(const Shadow& sh, int64_t i, const d3& p) {
    sh.x[i] = static_cast<float>(p.x);
    sh.y[i] = static_cast<float>(p.y);
    sh.z[i] = static_cast<float>(p.z);
}

// Predictor (istep 0): v* = v + dt f, x* = x + dt/2 (v + v*), f = a + fex(x).
__device__ __forceinline__ void predict(const StepArgs& a, int64_t i, const d3& r, const d3& v,
                                        const d3& f) {
    d3 vt, pt;
    vt.x = v.x + a.dt * f.x;
    vt.y = v.y + a.dt * f.y;
    vt.z = v.z + a.dt * f.z;
    pt.x = r.x + 0.5 * a.dt * (v.x + vt.x);
    pt.y = r.y + 0.5 * a.dt * (v.y + vt.y);
    pt.z = r.z + 0.5 * a.dt * (v.z + vt.z);
    st3(a.post, i, pt);
    st3(a.velt, i, vt);
    write_shadow(a.shadow, i, pt);
}

__global__ void predictor_kernel(const StepArgs a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const d3 r = ld3(a.pos, i), v = ld3(a.vel, i), ac = ld3(a.acc, i);
        const d3 fe = fex(a.field, r);
        const d3 f{ac.x + fe.x, ac.y + fe.y, ac.z + fe.z};
        predict(a, i, r, v, f);
    }
}

// Where a pass left its sums: the pair kernel's fixed-point words, the symmetric
// FP64 pass's two parts, the one-sided kernel's partial per tile, or its slots.
// The kernels that read them are compiled for each: in one kernel the partials'
// loads ahead set the registers of all (214, one block per SM where there were
// four), and the corrector of 393,216 bodies with one slot took 31.5 us where it takes 18.7
// now, a collect 21.8 and 7.0.
enum class Src { kFx, kF64, kTiles, kSlots, kFewSlots };

// The sums of body i; the accumulating kernels' (fx, f64) are left zero for
// the next pass, and so is its queue: two memsets less per step (about 2 us
// each between small kernels).
template <Src S>
__device__ __forceinline__ void sum_partials(const StepArgs& a, int64_t i, d3& s, double& sp) {
    s = d3{0.0, 0.0, 0.0};
    sp = 0.0;
    if (a.queue)
        for (int64_t q = i; q < kQueueWords; q += a.n) a.queue[q] = 0u;
    if constexpr (S == Src::kFx) {
        // The pair kernel's fixed-point sums (zero for ghosts).
        const FxScale sc = a.fx_scale[i / kPad];
        s.x = static_cast<double>(static_cast<long long>(a.fx[i])) * sc.inv_acc;
        s.y = static_cast<double>(static_cast<long long>(a.fx[a.npad + i])) * sc.inv_acc;
        s.z = static_cast<double>(static_cast<long long>(a.fx[2 * a.npad + i])) * sc.inv_acc;
        sp = static_cast<double>(static_cast<long long>(a.fx[3 * a.npad + i])) * sc.inv_phi;
#pragma unroll
        for (int c = 0; c < kFxComps; ++c) a.fx[c * a.npad + i] = 0ull;
    } else if constexpr (S == Src::kF64) {
        double *u = a.f64 + i, *l = u + 4 * a.npad;
        s = d3{u[0] + l[0], u[a.npad] + l[a.npad], u[2 * a.npad] + l[2 * a.npad]};
        sp = u[3 * a.npad] + l[3 * a.npad];
#pragma unroll
        for (int c = 0; c < 8; ++c) u[c * a.npad] = 0.0;
    } else if constexpr (S == Src::kTiles) {
        if (a.nsplit[i] == 0) return;
        const double4 t = sum_tile_chains<16>(a.tiles, a.npad, i, a.ntiles, a.chains, a.tile_mass);
        s = d3{t.x, t.y, t.z};
        sp = t.w;
    } else {
        // Slots in order, eight loads in flight where the bodies are few (a
        // small system's 24 slots one after the other took most of the
        // corrector's 8 us) and the other warps cannot cover them.
        const int ns = a.nsplit[i];
        constexpr int kAhead = S == Src::kFewSlots ? 8 : 1;
        for (int k0 = 0; k0 < ns; k0 += kAhead) {
            double4 p[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (k0 + k < ns) p[k] = a.part[(k0 + k) * a.npad + i];
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (k0 + k < ns) {
                    s.x += p[k].x;
                    s.y += p[k].y;
                    s.z += p[k].z;
                    sp += p[k].w;
                }
        }
    }
}

// Corrector (istep 1) fused with the next predictor.
template <Src S>
__global__ void corrector_kernel(const StepArgs a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        d3 an;
        double sp;
        sum_partials<S>(a, i, an, sp);
        if (a.compat_accumulate) {
            // The reference adds each step's force onto acct_ (never zeroed).
            d3 prev = ld3(a.acct, i);
            an = d3{prev.x + an.x, prev.y + an.y, prev.z + an.z};
            st3(a.acct, i, an);
        }
        const d3 xs = ld3(a.post, i), vs = ld3(a.velt, i), vo = ld3(a.vel, i);
        const d3 fe = fex(a.field, xs);
        const d3 f{an.x + fe.x, an.y + fe.y, an.z + fe.z};
        d3 vn;
        vn.x = 0.5 * (vo.x + vs.x + a.dt * f.x);
        vn.y = 0.5 * (vo.y + vs.y + a.dt * f.y);
        vn.z = 0.5 * (vo.z + vs.z + a.dt * f.z);
        st3(a.pos, i, xs);
        st3(a.vel, i, vn);
        st3(a.acc, i, an);
        if (a.want_phi) a.phi[i] = 0.0 - sp;
        if (a.predict_next) predict(a, i, xs, vn, f);
    }
}

// Partials -> state acc/phi (khrr_forces).
template <Src S>
__global__ void collect_kernel(const StepArgs a, int want_acc, int accumulate) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        d3 s;
        double sp;
        sum_partials<S>(a, i, s, sp);
        if (want_acc) {
            if (accumulate) {
                const d3 prev = ld3(a.acc, i);
                s = d3{prev.x + s.x, prev.y + s.y, prev.z + s.z};
            }
            st3(a.acc, i, s);
        }
        if (a.want_phi) a.phi[i] = 0.0 - sp;
    }
}

// kernelNbody_integTime (nbody-kernel.cuh:144-193) with its argument roles.
__global__ void integ_time_kernel(const double* acc, double* pos_t, double* vel_t, const double* pos,
                                  const double* vel, double dt, int istep, double* acc0, int64_t n,
                                  const FieldConsts F) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const d3 v = ld3(vel, i), r = ld3(pos, i), ac = ld3(acc, i);
        const d3 fe = fex(F, r);
        const d3 f{ac.x + fe.x, ac.y + fe.y, ac.z + fe.z};
        if (istep == 0) {
            d3 vt, pt;
            vt.x = v.x + dt * f.x;
            vt.y = v.y + dt * f.y;
            vt.z = v.z + dt * f.z;
            pt.x = r.x + 0.5 * dt * (v.x + vt.x);
            pt.y = r.y + 0.5 * dt * (v.y + vt.y);
            pt.z = r.z + 0.5 * dt * (v.z + vt.z);
            st3(pos_t, i, pt);
            st3(vel_t, i, vt);
        } else {
            const d3 vt = ld3(vel_t, i);
            d3 vtt;
            vtt.x = 0.5 * (vt.x + v.x + dt * f.x);
            vtt.y = 0.5 * (vt.y + v.y + dt * f.y);
            vtt.z = 0.5 * (vt.z + v.z + dt * f.z);
            st3(pos_t, i, r);
            st3(vel_t, i, vtt);
            st3(acc0, i, ac);
        }
    }
}

// ---- conservation sums (result(), nbody/src/nbody.cu:797-833) ---------------
// 8 sums (Lx Ly Lz Ix Iy Iz Ek Ep) + 5 maxima (R Z |Vr| Vfi |Vz|) per block;
// the block that finishes last folds the block results, a warp per field and
// every lane its own stride of blocks: the order is fixed by the block count,
// so the result is deterministic.  (One thread folding 592 blocks in a second
// launch took 324 us of a pass whose blocks take 15; now 16 us in all.)
constexpr int kConsThreads = 256;
constexpr int kConsFields = 13, kConsSums = 8;

__device__ __forceinline__ double cons_fold(double a, double b, bool sum) { return sum ? a + b : fmax(a, b); }

__global__ void __launch_bounds__(kConsThreads) conservation_kernel(const double* pos, const double* vel,
                                                                    const double* mass, const double* phi, int64_t n,
                                                                    double* block_out, unsigned* done, const unsigned* err,
                                                                    double* out16) {
    double v[kConsFields];
#pragma unroll
    for (int k = 0; k < kConsFields; ++k) v[k] = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
        const double vx = vel[3 * i], vy = vel[3 * i + 1], vz = vel[3 * i + 2];
        const double m = mass[i];
        const double r = sqrt(x * x + y * y);
        double vr = 0.0, vfi = 0.0;
        if (r > 0.0) {
            vr = (vx * x + vy * y) / r;
            vfi = (vy * x - vx * y) / r;
        }
        v[0] += (vz * y - vy * z) * m;
        v[1] += (vx * z - vz * x) * m;
        v[2] += (vy * x - vx * y) * m;
        v[3] += m * vx;
        v[4] += m * vy;
        v[5] += m * vz;
        v[6] += m * (vx * vx + vy * vy + vz * vz);
        v[7] += m * phi[i];
        v[8] = fmax(v[8], r);
        v[9] = fmax(v[9], fabs(z));
        v[10] = fmax(v[10], fabs(vr));
        v[11] = fmax(v[11], vfi);
        v[12] = fmax(v[12], fabs(vz));
    }
    constexpr int kWarps = kConsThreads / 32;
    __shared__ double sh[kConsFields][kWarps];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kConsFields; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = cons_fold(v[k], __shfl_xor_sync(0xffffffffu, v[k], o), k < kConsSums);
        if (lane == 0) sh[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < kConsFields) {
        const int k = threadIdx.x;
        double r = sh[k][0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) r = cons_fold(r, sh[k][w], k < kConsSums);
        block_out[static_cast<int64_t>(blockIdx.x) * kConsFields + k] = r;
        __threadfence();
    }
    __syncthreads();
    // The counter wraps to zero with the last block, ready for the next call.
    if (threadIdx.x == 0) last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = warp; k < kConsFields; k += kWarps) {
        double r = 0.0;
        for (unsigned b = lane; b < gridDim.x; b += 32)
            r = cons_fold(r, __ldcg(block_out + static_cast<int64_t>(b) * kConsFields + k), k < kConsSums);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r = cons_fold(r, __shfl_xor_sync(0xffffffffu, r, o), k < kConsSums);
        if (lane == 0) sh[k][0] = r;
    }
    __syncthreads();
    // Layout of khrr_lie: L[3], Imp[3], Ek, Ep, E, R_max, Z_max, Vr_max, Vfi_max, Vz_max,
    // then a free word and the error flag.  Straight into the host's
    // page-locked words: with the flag's copy gone too, a call at 3,072
    // bodies takes 17 us instead of 41.
    if (threadIdx.x < 16) {
        const int k = threadIdx.x;
        if (k < 14) out16[k] = k < 8 ? sh[k][0] : (k == 8 ? 0.5 * (sh[6][0] + sh[7][0]) : sh[k - 1][0]);
        else out16[k] = k == 15 ? static_cast<double>(__ldcg(err)) : 0.0;
    }
}

// Threads per block of the per-body kernels: 256, or 64 where that leaves SMs
// without a block.
constexpr int64_t kFewBodies = 148 * 256;
int step_block(int64_t n) { return n < kFewBodies ? 64 : 256; }

// Calls f with the place of a's sums as a template argument.
template <class F>
void with_source(const StepArgs& a, F f) {
    if (a.fx) f(std::integral_constant<Src, Src::kFx>{});
    else if (a.f64) f(std::integral_constant<Src, Src::kF64>{});
    else if (a.tiles) f(std::integral_constant<Src, Src::kTiles>{});
    else if (a.n < kFewBodies) f(std::integral_constant<Src, Src::kFewSlots>{});
    else f(std::integral_constant<Src, Src::kSlots>{});
}

int grid_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    if (g > 148 * 16) g = 148 * 16;
    if (g < 1) g = 1;
    return static_cast<int>(g);
}

}  // namespace

cudaError_t launch_predictor(const StepArgs& a, cudaStream_t s) {
    const int b = step_block(a.n);
    predictor_kernel<<<grid_for(a.n, b), b, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_corrector(const StepArgs& a, cudaStream_t s) {
    const int b = step_block(a.n);
    with_source(a, [&](auto src) { corrector_kernel<decltype(src)::value><<<grid_for(a.n, b), b, 0, s>>>(a); });
    return cudaGetLastError();
}

cudaError_t launch_collect(const StepArgs& a, bool want_acc, bool accumulate, cudaStream_t s) {
    const int b = step_block(a.n);
    with_source(a, [&](auto src) {
        collect_kernel<decltype(src)::value><<<grid_for(a.n, b), b, 0, s>>>(a, want_acc ? 1 : 0, accumulate ? 1 : 0);
    });
    return cudaGetLastError();
}

cudaError_t launch_integ_time(const double* acc, double* pos_t, double* vel_t, const double* pos,
                              const double* vel, double dt, int istep, double* acc0, int64_t n,
                              const FieldConsts& f, cudaStream_t s) {
    integ_time_kernel<<<grid_for(n, 256), 256, 0, s>>>(acc, pos_t, vel_t, pos, vel, dt, istep, acc0,
                                                       n, f);
    return cudaGetLastError();
}

int conservation_blocks(int64_t n) {
    int64_t b = (n + kConsThreads - 1) / kConsThreads;
    if (b > 148 * 4) b = 148 * 4;
    if (b < 1) b = 1;
    return static_cast<int>(b);
}

cudaError_t launch_conservation(const double* pos, const double* vel, const double* mass,
                                const double* phi, int64_t n, double* block_out, int nblocks, unsigned* done,
                                const unsigned* err, double* out16, cudaStream_t s) {
    conservation_kernel<<<nblocks, kConsThreads, 0, s>>>(pos, vel, mass, phi, n, block_out, done, err, out16);
    return cudaGetLastError();
}

}  // namespace khrr
