// The FP64 step of wave_march.cuh with its planes streamed through shared
// memory.
//
// A block owns `seg` consecutive cells of a plane (rows one after the other)
// and a range of z planes.  Those cells, and the row before and after them, are
// one contiguous piece of every plane, so a plane's phi (with both rows),
// phi_old and mass are three bulk copies of some kilobytes each, into a ring of
// ST planes.  The neighbours in y and x come from shared memory, the ones in z
// from registers and from the next stage.
//
// What it is for: from 178^3 on the march waits for memory with 30 KB an SM on
// the way (640 threads, 48 bytes each); the ring keeps 50 to 100 KB on the way.
// us per iteration, march / this: 200^3 52.1 / 45.3 (5.7 TB/s of 32 bytes a
// cell), 240^3 85.6 / 73.8, 256^3 103.6 / 91.2, 320^3 200 / 180.  Below, where the
// field stays in L2, the march is faster (160^3 27.3 / 31.5).  FP32 gained
// nothing (256^3 49.1 / 49.3).  Dealing the planes out as equal runs over the
// grid, so that blocks of neighbouring cells are at different planes, loses the
// shared rows in L2: 50.3 at 200^3, 82.8 at 240^3.
#pragma once

#include <algorithm>

#include "async_copy.cuh"
#include "wave_march.cuh"

namespace khrr {
namespace {

// nx and seg are even and the arrays 16-byte aligned, so every copy starts on a
// 16-byte boundary and its length is a multiple of 16.  A thread owns U pairs of
// cells.
template <int NT, int U, int MINB, int ST>
__global__ void __launch_bounds__(NT, MINB) wave_stream_kernel(double* __restrict__ phi_new,
                                                               const double* __restrict__ phi,
                                                               const double* __restrict__ phi_old,
                                                               const double* __restrict__ mass, const WaveConsts w,
                                                               int nx, int seg, unsigned* __restrict__ err) {
    constexpr int V = 2;
    using P = Pack<double, V>;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem);
    const int stage_cells = 3 * seg + 2 * nx;
    double* const ring = reinterpret_cast<double*>(smem + 64);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tid = threadIdx.x;
    const int plane = nx * nx;
    const int q0 = static_cast<int>(blockIdx.x) * seg, len = min(seg, plane - q0);
    const int z0 = static_cast<int>(static_cast<int64_t>(blockIdx.y) * nx / gridDim.y);
    const int z1 = static_cast<int>(static_cast<int64_t>(blockIdx.y + 1) * nx / gridDim.y);
    const int K = z1 - z0, stages = K + (z1 < nx ? 1 : 0);  // the plane after the range: its phi only
    if (tid == 0) {
#pragma unroll
        for (int k = 0; k < ST; ++k) mbar_init(bar + k, 1);
        fence_mbar_init();
    }
    __syncthreads();
    // Stage k: plane z0 + k; cell q of the plane at phi index q - (q0 - nx).
    auto fetch = [&](int k) {
        const int64_t at = static_cast<int64_t>(z0 + k) * plane;
        const int lo = k < K ? max(q0 - nx, 0) : q0, hi = k < K ? min(q0 + len + nx, plane) : q0 + len;
        double* const st = ring + (k % ST) * stage_cells;
        uint64_t* const b = bar + k % ST;
        const unsigned pb = static_cast<unsigned>((hi - lo) * sizeof(double)), lb = static_cast<unsigned>(len * sizeof(double));
        mbar_arrive_expect_tx(b, k < K ? pb + 2 * lb : pb);
        bulk_copy_g2s(st + (lo - (q0 - nx)), phi + at + lo, pb, b);
        if (k < K) {
            bulk_copy_g2s(st + seg + 2 * nx, phi_old + at + q0, lb, b);
            bulk_copy_g2s(st + 2 * seg + 2 * nx, mass + at + q0, lb, b);
        }
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tid == 0)
        for (int k = 0; k < min(ST, stages); ++k) fetch(k);

    StepF64<V> s[U];
    P zm[U], c[U];
    bool in[U], edge_y[U];
    int ix[U];
    double sz_last = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int j = (u * NT + tid) * V;
        in[u] = j < len;
        const int q = in[u] ? q0 + j : q0, iy = q / nx;
        ix[u] = q - iy * nx;
        edge_y[u] = iy == 0 || iy == nx - 1;
        s[u].W = w;
        s[u].column(ix[u], iy);
        sz_last = s[u].plane_term(z0);
        s[u].coefficients(sz_last);
        zm[u] = load_pack<double, V>(phi + static_cast<int64_t>(max(z0 - 1, 0)) * plane + q);
    }
    bool lost = !mbar_wait_bounded(bar, 0);
    if (!lost) {
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = load_pack<double, V>(ring + nx + (in[u] ? (u * NT + tid) * V : 0));
    }
    for (int k = 0; k < K; ++k) {
        const int z = z0 + k;
        const double* const st = ring + (k % ST) * stage_cells;
        const double* const next = ring + ((k + 1) % ST) * stage_cells + nx;
        if (!lost && k + 1 < stages)
            lost = !mbar_wait_bounded(bar + (k + 1) % ST, ((k + 1) / ST) & 1);
        const double sz_now = s[0].plane_term(z);
        if (sz_now != sz_last) {  // the same for the whole grid row
            sz_last = sz_now;
#pragma unroll
            for (int u = 0; u < U; ++u) s[u].coefficients(sz_now);
        }
        if (!lost) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!in[u]) continue;
                const int j = (u * NT + tid) * V;
                const P zp = k + 1 < stages ? load_pack<double, V>(next + j) : c[u];
                const P ym = load_pack<double, V>(st + j), yp = load_pack<double, V>(st + j + 2 * nx);
                const double xl = st[j + nx - 1], xr = st[j + nx + V];
                const P po = load_pack<double, V>(st + seg + 2 * nx + j), ms = load_pack<double, V>(st + 2 * seg + 2 * nx + j);
                const bool edge = edge_y[u] || z == 0 || z == nx - 1;
                P out;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const double xm = v == 0 ? xl : c[u].v[0], xp = v == V - 1 ? xr : c[u].v[V - 1];
                    const double o = s[u].cell(v, xm, xp, ym.v[v], yp.v[v], zm[u].v[v], zp.v[v], c[u].v[v], po.v[v], ms.v[v]);
                    out.v[v] = edge || ix[u] + v == 0 || ix[u] + v == nx - 1 ? 0.0 : o;
                }
                store_pack<double, V>(phi_new + static_cast<int64_t>(z) * plane + q0 + j, out);
                zm[u] = c[u];
                c[u] = zp;
            }
        }
        // Every thread is done with stage k; one that gave up its wait ends the block.
        if (__syncthreads_or(lost)) {
            if (tid == 0) {
                atomicOr(err, kErrTimeout);
                for (int f = k; f < min(k + ST, stages); ++f)
                    mbar_wait_bounded(bar + f % ST, (f / ST) & 1);
            }
            return;
        }
        if (tid == 0 && k + ST < stages) {
            fence_proxy_async();
            fetch(k + ST);
        }
    }
}

// The cut of the mesh: blocks per plane, cells of one (a multiple of 128 bytes,
// at most what the block's threads and `smem` bytes of ring hold; 0: nothing
// fits), z ranges.  cost: rounds of `resident` blocks times the planes of one
// (and two more to start) times what a plane brings in.
struct StreamCut {
    int seg = 0, blocks = 0, ranges = 0;
    double cost = 1e300;
};

inline StreamCut stream_cut(int nx, int max_cells, int smem, int stages, int resident) {
    constexpr int kLine = 16;
    const int plane = nx * nx, room = (smem - 64) / (stages * static_cast<int>(sizeof(double))) - 2 * nx;
    const int cap = std::min(max_cells, room / 3) / kLine * kLine;
    StreamCut best;
    if (cap < kLine) return best;
    for (int r = 1; r <= nx; ++r) {
        const int want = std::max((plane + cap - 1) / cap, resident / r);
        const int seg = std::min(cap, ((plane + want - 1) / want + kLine - 1) / kLine * kLine);
        const int blocks = (plane + seg - 1) / seg;
        const int64_t rounds = (static_cast<int64_t>(blocks) * r + resident - 1) / resident;
        const double cost = static_cast<double>(rounds) * ((nx + r - 1) / r + 2) * (3.0 * seg + 2.0 * nx);
        if (cost < best.cost) best = StreamCut{seg, blocks, r, cost};
    }
    return best;
}

template <int NT, int U, int MINB, int ST>
struct StreamShape {
    static constexpr int kSmem = (227 * 1024) / MINB - 1024;
    static StreamCut cut(int nx) { return stream_cut(nx, 2 * NT * U, kSmem, ST, 148 * MINB); }
    static cudaError_t launch(const StreamCut& cut, double* phi_new, const double* phi, const double* phi_old,
                              const double* mass, const WaveConsts& w, unsigned* err, cudaStream_t s) {
        const auto kernel = wave_stream_kernel<NT, U, MINB, ST>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(cut.blocks), static_cast<unsigned>(cut.ranges));
        cfg.blockDim = dim3(NT);
        cfg.dynamicSmemBytes = 64 + ST * (3 * cut.seg + 2 * w.nx) * sizeof(double);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kernel, phi_new, phi, phi_old, mass, w, w.nx, cut.seg, err);
    }
};

}  // namespace
}  // namespace khrr
