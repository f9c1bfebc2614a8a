// fft_x.cu — the x pass fused with the Green's function, and the gradient.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

template <int NG>
__global__ void __launch_bounds__(512, 2) xpot_wide_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                                           int ncols, size_t rs, size_t ps,
                                                           const float2* __restrict__ tw, PotentialOp op) {
    xone_body<NG, 512, PotentialOp, XW<NG>::C>(in, out, ncols, rs, ps, tw, op, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------------------
// Force grid from the potential phi (real, [ng][ng][ng], z fastest):
// F_d(x) = (phi(x - e_d) - phi(x + e_d)) / 2, periodic, written as float4
// (F_x, F_y, F_z, 0) per cell.  With the unnormalised transforms used here
// this is exactly the reference's -i sin(k_d) G rho_k followed by the inverse
// FFT (kspace_solver.cu:55-90, solver.cpp:144-170): the central difference
// multiplies mode k by -i sin(2 pi k_d / ng), it is real, so it commutes with
// taking the real part, and it annihilates the Nyquist mode of its own axis
// as the reference's real part does.  blockIdx.y = slot.
// ---------------------------------------------------------------------------
// 256-bit (8 x f32) global accesses, sm_100: 32-byte aligned addresses.
struct F8 {
    float v[8];
};
__device__ __forceinline__ F8 ldg8(const float* p) {
    F8 r;
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]),
                   "=f"(r.v[7])
                 : "l"(p));
    return r;
}
// two float4 cells, streaming (evict-first)
__device__ __forceinline__ void stcs8(float4* p, float4 a, float4 b) {
    asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

// A thread makes 8 z-consecutive cells at XR consecutive x: 256-bit loads of
// phi and of its y neighbours, the x neighbours carried from the previous x
// (one new row per x), 256-bit stores of two cells each (whole sectors).
template <int XR, int MINB = 1, int U = 1>
__global__ void __launch_bounds__(256, MINB) gradient_kernel(const float* __restrict__ phi, float4* __restrict__ f, int ng,
                                                       Slots sl) {
    if (slot_idle(sl, blockIdx.y)) return;
    phi += (size_t)blockIdx.y * sl.s0;
    f += (size_t)blockIdx.y * sl.s1;
    const int n8 = ng / 8;
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    // the launcher makes (ng / XR) ng^2 / 8 a whole number of warps, so this
    // exit takes whole warps and the shuffles below see all 32 lanes
    if (q >= (size_t)(ng / XR) * ng * n8) return;
    const int z0 = (int)(q % n8) * 8;
    const int r = (int)(q / n8);
    const int y = r % ng;
    int x = (r / ng) * XR;
    const int ym = y == 0 ? ng - 1 : y - 1, yp = y + 1 == ng ? 0 : y + 1;
    const size_t plane = (size_t)ng * ng;
    const size_t oy = (size_t)y * ng + z0, oym = (size_t)ym * ng + z0, oyp = (size_t)yp * ng + z0;
    const int lane = threadIdx.x & 31;
    F8 a = ldg8(phi + (size_t)(x == 0 ? ng - 1 : x - 1) * plane + oy);
    F8 c = ldg8(phi + (size_t)x * plane + oy);
#pragma unroll U
    for (int k = 0; k < XR; ++k, ++x) {
        const size_t px = (size_t)x * plane;
        const F8 b = ldg8(phi + (size_t)(x + 1 == ng ? 0 : x + 1) * plane + oy);
        const F8 d = ldg8(phi + px + oym);
        const F8 e = ldg8(phi + px + oyp);
        // the z neighbours of the run's ends are the adjacent lanes' end cells
        // (same row); the warp's end lanes and the row's periodic wrap load them
        float zm = __shfl_up_sync(0xffffffffu, c.v[7], 1);
        float zp = __shfl_down_sync(0xffffffffu, c.v[0], 1);
        if (lane == 0 || z0 == 0) zm = __ldg(phi + px + oy - z0 + (z0 == 0 ? ng - 1 : z0 - 1));
        if (lane == 31 || z0 + 8 == ng) zp = __ldg(phi + px + oy - z0 + (z0 + 8 == ng ? 0 : z0 + 8));
        float4 o[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const float lo = m == 0 ? zm : c.v[m - 1];
            const float hi = m == 7 ? zp : c.v[m + 1];
            o[m] = make_float4(0.5f * (a.v[m] - b.v[m]), 0.5f * (d.v[m] - e.v[m]), 0.5f * (lo - hi), 0.f);
        }
        float4* dst = f + px + oy;
#pragma unroll
        for (int m = 0; m < 8; m += 2) stcs8(dst + m, o[m], o[m + 1]);
        a = c;
        c = b;
    }
}

cudaError_t launch_gradient(int ng, const float* phi, float4* f, cudaStream_t s, const Slots& sl, int nslots) {
    if (!fft_size_supported(ng)) return cudaErrorInvalidValue;
    // eight x per thread from 64^3 (the thread count, ng^3 / 64, is then a
    // whole number of warps for ng a multiple of 16); one on smaller grids,
    // which need every thread they can get (ng^3 / 8 threads, ng a multiple
    // of 8).  Measured at 512^3: x runs of 4, 8 or 16 within 1 %, 0.04 ms
    // faster than one x per thread.
#define GV(XR, MB, U)                                                                      \
    {                                                                                      \
        const size_t nq = (size_t)(ng / XR) * ng * (ng / 8);                               \
        gradient_kernel<XR, MB, U><<<dim3(cdiv(nq, 256), nslots), 256, 0, s>>>(phi, f, ng, sl); \
    }
    if (ng % 16 == 0 && ng >= 64) GV(8, 3, 2)
    else GV(1, 1, 1)
#undef GV
    return cudaGetLastError();
}

cudaError_t launch_xpotential(int ng, const float2* in, float2* out, int ncols, size_t rs, size_t ps, int nplanes,
                              const float2* tw, const double* cosq, double coeff, cudaStream_t s, const Slots& sl,
                              int nslots) {
    PotentialOp op{cosq, coeff};
    switch (ng) {
#define X(n) \
    case n: return xfused_impl<n, PotentialOp>(in, out, ncols, rs, ps, nplanes, 0, tw, op, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

template <int NG>
static cudaError_t xpot_wide_impl(const float2* in, float2* out, int ncols, size_t rs, size_t ps, int nplanes,
                                  const float2* tw, const PotentialOp& op, cudaStream_t s) {
    constexpr int C = XW<NG>::C, SMEM = NG * C * 8;
    auto k = xpot_wide_kernel<NG>;
    cudaError_t e = ensure_smem(k, SMEM);
    if (e != cudaSuccess) return e;
    k<<<dim3(cdiv(ncols, C), nplanes), 512, SMEM, s>>>(in, out, ncols, rs, ps, tw, op);
    return cudaGetLastError();
}

cudaError_t launch_xpotential_wide(int ng, const float2* in, float2* out, int ncols, size_t rs, size_t ps, int nplanes,
                                   const float2* tw, const double* cosq, double coeff, cudaStream_t s) {
    PotentialOp op{cosq, coeff};
    switch (ng) {
#define X(n) \
    case n: return xpot_wide_impl<n>(in, out, ncols, rs, ps, nplanes, tw, op, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
