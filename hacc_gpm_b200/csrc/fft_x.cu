// fft_x.cu — the x pass fused with the Green's function, and the gradient.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// The x pass: forward x transform, the Green's function, inverse x transform
// of the potential's spectrum, line tiles in register groups.  Bound by issue
// and latency (at 512^3 before: 138 instructions an element at 63 % of the
// issue slots, DRAM at 29 %): the quotient of the Green's function (green())
// takes a third of the instructions a division took, and the tile crosses
// shared memory 4 times instead of 6 (8 at 1024).  us a pass, against tiles
// staged through shared memory for every radix and a division per mode: 256^3
// 52 / 66, 200^3 33 / 43, 512^3 395 / 430, 1024^3 3780 / 4300.
// Tile size: large enough for 16 columns (whole 128-byte lines) up to 512
// and 8 above, 2 or more CTAs an SM; small grids take small tiles, so that
// they spread over the GPU (64^3: 8.7 us in 2^10-element tiles, 10.7 in
// 2^11); 320 takes 16 columns (104 us; 122 with 8).
template <int NG>
using XT = LineTile<NG, NG <= 64 ? 1024 : NG <= 128 ? 2048 : NG <= 256 ? 4096 : NG < 384 ? 6144 : 8192>;

template <int NG>
__global__ void __launch_bounds__(XT<NG>::NT, XT<NG>::MINB) xpot_kernel(const float2* __restrict__ in,
                                                                        float2* __restrict__ out, int zs,
                                                                        const float2* __restrict__ tw, PotentialOp op,
                                                                        Slots sl) {
    using T = XT<NG>;
    if (slot_idle(sl, blockIdx.y)) return;
    in += (size_t)blockIdx.y * sl.s0;
    out += (size_t)blockIdx.y * sl.s1;
    const LineCols<T, NG> cols{(int)blockIdx.x};
    const size_t rs = (size_t)NG * zs;
    fft_lines_fwd_op_inv<NG, T::C, T::NT>(
        reinterpret_cast<float2*>(hgpm_smem), tw,
        [&](int e, int c) {
            int iy, iz;
            bool ok;
            cols.at(c, iy, iz, ok);
            return ok ? __ldcs(in + (size_t)e * rs + (size_t)iy * zs + iz) : make_float2(0.f, 0.f);
        },
        [&](int e, int c, float2 v) {
            int iy, iz;
            bool ok;
            cols.at(c, iy, iz, ok);
            if (ok) __stcs(out + (size_t)e * rs + (size_t)iy * zs + iz, v);
        },
        [&](int ix, int c, float2 v) {
            int iy, iz;
            bool ok;
            cols.at(c, iy, iz, ok);
            if (!ok) iy = iz = 0;  // an empty line of zeros
            return op.apply(__ldg(&op.cosq[ix]), __ldg(&op.cosq[iy]) + __ldg(&op.cosq[iz]), v);
        });
}

template <int NG>
static cudaError_t xpot_impl(const float2* in, float2* out, int zs, const float2* tw, const PotentialOp& op,
                             cudaStream_t s, const Slots& sl, int nslots) {
    using T = XT<NG>;
    auto k = xpot_kernel<NG>;
    cudaError_t e = ensure_smem(k, T::SMEM, T::NT);
    if (e != cudaSuccess) return e;
    k<<<dim3(T::TILES, nslots), T::NT, T::SMEM, s>>>(in, out, zs, tw, op, sl);
    return cudaGetLastError();
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

cudaError_t launch_xpotential(int ng, const float2* in, float2* out, int zs, const float2* tw, const double* cosq,
                              double coeff, cudaStream_t s, const Slots& sl, int nslots) {
    PotentialOp op{cosq, coeff};
    switch (ng) {
#define X(n) \
    case n: return xpot_impl<n>(in, out, zs, tw, op, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

// Over every sum of three entries of cosq: how many of green()'s floats are not
// the division's (out[0]), and the most float steps between the two (out[1]).
__global__ void green_check_kernel(int ng, const double* __restrict__ cosq, double coeff,
                                   unsigned long long* __restrict__ out) {
    const int iz = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y;
    if (iz >= ng) return;
    const double cyz = cosq[iy] + cosq[iz];
    unsigned long long n = 0, most = 0;
    for (int ix = 0; ix < ng; ++ix) {
        const double s = cosq[ix] + cyz;
        const int a = __float_as_int(green(s, coeff)), b = __float_as_int(s == 0.0 ? 0.f : (float)(coeff / s));
        const unsigned long long d = a > b ? (unsigned long long)((long long)a - b) : (unsigned long long)((long long)b - a);
        n += d != 0;
        most = d > most ? d : most;
    }
    if (n) {
        atomicAdd(&out[0], n);
        atomicMax(&out[1], most);
    }
}

cudaError_t launch_green_check(int ng, const double* cosq, double coeff, unsigned long long* out, cudaStream_t s) {
    green_check_kernel<<<dim3(cdiv(ng, 128), ng), 128, 0, s>>>(ng, cosq, coeff, out);
    return cudaGetLastError();
}

}  // namespace hgpm
