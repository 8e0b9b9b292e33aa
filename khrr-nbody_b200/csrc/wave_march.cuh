// The damped-wave stencil marched along z: wave_diss_iteration
// (wave-kernel.cuh:5-103) in FP64, and the FP32 form of the step.
//
// A thread owns V consecutive x cells of one row (16 bytes where the rows
// allow it) and walks a range of z planes: the column's phi values stay in
// registers for the two planes around them, so a plane costs one new 16-byte
// load each of phi, phi_old and the mass (issued one plane ahead), the two y
// rows and the two x neighbours (just read by neighbouring threads: L1), and
// one store.  Rows are laid out one after the other over the threads of a
// block (any nx fills its warps), and the z ranges are cut so that the whole
// grid is resident at once: no last wave, and a column is re-read at range
// borders only.
//
// The step's coefficients depend on x, y and z through the sponge alone,
// whose z term is zero over the lower 45 % of the planes: they are kept and
// recomputed only where the z term changes.
//
// What bounds it, measured at 256^3 (FP32 / FP64): the kernels before spent
// 86 / 249 instructions a cell on addresses, repeated coefficients and single
// loads, issue slots 62 / 69 % busy at 59 / 54 % of the copy bandwidth.
#pragma once

#include <cstdint>

#include "khrr_internal.h"

namespace khrr {
namespace {

template <class T, int V>
struct alignas(sizeof(T) * V) Pack {
    T v[V];
};

template <class T, int V>
__device__ __forceinline__ Pack<T, V> load_pack(const T* __restrict__ p) {
    Pack<T, V> r;
    if constexpr (V == 1) r.v[0] = *p;
    else *reinterpret_cast<int4*>(&r) = *reinterpret_cast<const int4*>(p);
    return r;
}

template <class T, int V>
__device__ __forceinline__ void store_pack(T* __restrict__ p, const Pack<T, V>& r) {
    if constexpr (V == 1) *p = r.v[0];
    else *reinterpret_cast<int4*>(p) = *reinterpret_cast<const int4*>(&r);
}

// a / b, correctly rounded, from y = RN(1/b): Markstein's correction step
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Develop. 34(1), 1990; see also
// Muller et al., "Handbook of Floating-Point Arithmetic", ch. 4): q = RN(a y)
// is within an ulp of a/b, r = a - b q is exact in one fma, and RN(q + r y)
// is RN(a/b).  Several quotients over one denominator then share one
// correctly rounded reciprocal (__drcp_rn).  Checked bitwise against the IEEE
// division on 1.7e10 quotients (the stencil's operand ranges and random
// operands over 64 binary orders of magnitude): no difference.
__device__ __forceinline__ double div_rn(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    const double r = fma(-b, q, a);
    return fma(r, y, q);
}

// The FP32 step.  The sponge is separable, diss = base + sx[ix] + sy[iy] +
// sz[iz] (per-axis tables built in FP64 on the host); per cell: Q = diss c dt
// / 2, w = 1 / (1 + Q), and
//   phi_new = nb K w + phi (2 (1 - 3K)) w + phi_old (Q - 1) w + mass S w,
// with nb the six-neighbour sum and S = -c^2 dt^2 4 pi / dx^3.
template <int V>
struct StepF32 {
    using T = float;
    const WaveF32 W;
    float sxy[V], kw[V], aw[V], ow[V], sw[V];
    __device__ __forceinline__ void column(int ix, int iy) {
#pragma unroll
        for (int k = 0; k < V; ++k) sxy[k] = (W.diss_base + W.sx[ix + k]) + W.sy[iy];
    }
    __device__ __forceinline__ float plane_term(int z) const { return W.sz[z]; }
    __device__ __forceinline__ void coefficients(float sz) {
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const float diss = sxy[k] + sz;
            const float Q = diss * W.cdt_half;
            const float w = __frcp_rn(1.0f + Q);  // correctly rounded: the bits of 1.0f / (1.0f + Q)
            kw[k] = W.K * w;
            aw[k] = W.A * w;
            ow[k] = (Q - 1.0f) * w;
            sw[k] = W.S * w;
        }
    }
    __device__ __forceinline__ float cell(int k, float xm, float xp, float ym, float yp, float zm, float zp, float c,
                                          float po, float ms) const {
        const float nb = ((xm + xp) + (ym + yp)) + (zm + zp);
        return fmaf(nb, kw[k], fmaf(c, aw[k], fmaf(po, ow[k], ms * sw[k])));
    }
};

// The reference's FP64 expression term for term (same bits as its literal
// evaluation): the sponge of wave-kernel.cuh:32-60 (coordinates ix*dx, not
// centred; the x test compares against -(L - bc)), added axis by axis, and
// the five divisions through shared correctly rounded reciprocals.
template <int V>
struct StepF64 {
    using T = double;
    WaveConsts W;
    double L, D3, yD3, K, KFn, KAn;
    double sxy[V], km[V], ka[V], ko[V], kf[V];
    __device__ __forceinline__ double term(double p, bool above, bool below) const {
        if (above) return W.diss_extra * fabs(p - L) * fabs(p - L);
        if (below) return W.diss_extra * fabs(p + L) * fabs(p + L);
        return 0.0;
    }
    __device__ __forceinline__ void column(int ix, int iy) {
        L = W.sim_l - W.bc_l;
        D3 = W.dx * W.dx * W.dx;
        yD3 = __drcp_rn(D3);
        K = W.c * W.c * (W.dt * W.dt) / (W.dx * W.dx);
        KFn = -(W.c * W.c) * (W.dt * W.dt);
        KAn = 2 * (1. - 3 * K);
        const double y = iy * W.dx, sy = term(y, y > L, y < -L);
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const double x = (ix + k) * W.dx;
            sxy[k] = (W.diss_base + term(x, x > -L, x < -L)) + sy;
        }
    }
    __device__ __forceinline__ double plane_term(int z) const {
        const double p = z * W.dx;
        return term(p, p > L, p < -L);
    }
    __device__ __forceinline__ void coefficients(double sz) {
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const double diss = sxy[k] + sz;
            const double Q = diss * W.c * W.dt * 0.5;
            const double Wt = 1 + Q;
            const double yW = __drcp_rn(Wt);
            km[k] = div_rn(K, Wt, yW);
            kf[k] = div_rn(KFn, Wt, yW);
            ka[k] = div_rn(KAn, Wt, yW);
            ko[k] = div_rn(Q - 1., Wt, yW);
        }
    }
    __device__ __forceinline__ double cell(int k, double xm, double xp, double ym, double yp, double zm, double zp,
                                           double c, double po, double ms) const {
        const double rho = div_rn(ms, D3, yD3);
        const double f = 4 * 3.14159265358979 * 1.0 * rho;  // the reference's PI (common.cuh:7)
        return xm * km[k] + xp * km[k] + ym * km[k] + yp * km[k] + zm * km[k] + zp * km[k] + c * ka[k] + po * ko[k] +
               f * kf[k];
    }
};

// One step over the mesh: block (b, r) owns cells b * NT * V .. of each plane
// and the planes [r nx / gridDim.y, (r + 1) nx / gridDim.y).  nx % V == 0;
// with V > 1 the arrays are 16-byte aligned.  RESID: sum (phi_new - phi)^2 and
// sum phi_new^2 in FP64 are added into resid[0..1].
template <class S, int V, int NT, int MINB, bool RESID, class W>
__global__ void __launch_bounds__(NT, MINB) wave_march_kernel(typename S::T* __restrict__ phi_new,
                                                              const typename S::T* __restrict__ phi,
                                                              const typename S::T* __restrict__ phi_old,
                                                              const typename S::T* __restrict__ mass, const W w,
                                                              int nx, double* __restrict__ resid) {
    using T = typename S::T;
    using P = Pack<T, V>;
    // Programmatic dependent launch: the next step's grid may be scheduled
    // while this one drains; every grid waits here until the previous one
    // has completed and its writes are visible (a no-op without a
    // programmatic dependency).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int rowp = nx / V;  // packs per row
    const int64_t t = static_cast<int64_t>(blockIdx.x) * NT + threadIdx.x;
    const int iy = static_cast<int>(t / rowp), ix = static_cast<int>(t - static_cast<int64_t>(iy) * rowp) * V;
    const int z0 = static_cast<int>(static_cast<int64_t>(blockIdx.y) * nx / gridDim.y);
    const int z1 = static_cast<int>(static_cast<int64_t>(blockIdx.y + 1) * nx / gridDim.y);
    double d2 = 0.0, n2 = 0.0;
    S s{w};
    const bool in = iy < nx;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (in) {
        s.column(ix, iy);
        const int64_t sz = static_cast<int64_t>(nx) * nx;
        int64_t at = z0 * sz + static_cast<int64_t>(iy) * nx + ix;
        // Neighbour offsets clamped into the mesh, so every load is in bounds
        // (face cells discard their values).
        const int64_t dym = iy > 0 ? nx : 0, dyp = iy < nx - 1 ? nx : 0;
        const int dxm = ix > 0 ? 1 : 0, dxp = ix + V < nx ? V : V - 1;
        const bool edge_y = iy == 0 || iy == nx - 1;
        P zm = load_pack<T, V>(phi + at - (z0 > 0 ? sz : 0)), c = load_pack<T, V>(phi + at);
        P zp = load_pack<T, V>(phi + at + (z0 + 1 < nx ? sz : 0));
        P po = load_pack<T, V>(phi_old + at), ms = load_pack<T, V>(mass + at);
        T sz_last = s.plane_term(z0);
        s.coefficients(sz_last);
        for (int z = z0; z < z1; ++z) {
            P zp_next = zp, po_next = po, ms_next = ms;
            if (z + 1 < z1) {
                zp_next = load_pack<T, V>(phi + at + (z + 2 < nx ? 2 * sz : sz));
                po_next = load_pack<T, V>(phi_old + at + sz);
                ms_next = load_pack<T, V>(mass + at + sz);
            }
            const P ym = load_pack<T, V>(phi + at - dym), yp = load_pack<T, V>(phi + at + dyp);
            const T xl = phi[at - dxm], xr = phi[at + dxp];
            const T sz_now = s.plane_term(z);
            if (sz_now != sz_last) {  // the same for the whole grid row
                sz_last = sz_now;
                s.coefficients(sz_now);
            }
            const bool edge = edge_y || z == 0 || z == nx - 1;
            P out;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const T xm = k == 0 ? xl : c.v[k > 0 ? k - 1 : 0], xp = k == V - 1 ? xr : c.v[k < V - 1 ? k + 1 : k];
                const T o = s.cell(k, xm, xp, ym.v[k], yp.v[k], zm.v[k], zp.v[k], c.v[k], po.v[k], ms.v[k]);
                out.v[k] = edge || ix + k == 0 || ix + k == nx - 1 ? T(0) : o;
                if (RESID) {
                    const double dd = static_cast<double>(out.v[k]) - static_cast<double>(c.v[k]);
                    d2 += dd * dd;
                    n2 += static_cast<double>(out.v[k]) * static_cast<double>(out.v[k]);
                }
            }
            store_pack<T, V>(phi_new + at, out);
            at += sz;
            zm = c;
            c = zp;
            zp = zp_next;
            po = po_next;
            ms = ms_next;
        }
    }
    if (RESID) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d2 += __shfl_xor_sync(0xffffffffu, d2, o);
            n2 += __shfl_xor_sync(0xffffffffu, n2, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&resid[0], d2);
            atomicAdd(&resid[1], n2);
        }
    }
}

template <class S, int V, int NT, int MINB, bool RESID, class W>
cudaError_t launch_march(typename S::T* phi_new, const typename S::T* phi, const typename S::T* phi_old,
                         const typename S::T* mass, const W& w, int nx, double* resid, cudaStream_t s) {
    // Launched with programmatic stream serialization: a chain of steps
    // overlaps each grid's launch with the previous grid's tail.
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(NT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int64_t per_plane = (static_cast<int64_t>(nx) * (nx / V) + NT - 1) / NT;
    // The z ranges: rounds of resident blocks times the planes of one (and the
    // start of its march, about one and a half more).
    const int64_t resident = 148 * MINB;
    int ranges = 1;
    double best = 1e300;
    for (int r = 1; r <= nx && r <= 256; ++r) {
        const double t = static_cast<double>((per_plane * r + resident - 1) / resident) * ((nx + r - 1) / r + 1.5);
        if (t < best) {
            best = t;
            ranges = r;
        }
    }
    cfg.gridDim = dim3(static_cast<unsigned>(per_plane), static_cast<unsigned>(ranges));
    return cudaLaunchKernelEx(&cfg, wave_march_kernel<S, V, NT, MINB, RESID, W>, phi_new, phi, phi_old, mass, w, nx,
                              resid);
}

}  // namespace
}  // namespace khrr
