// fft_z.cu — the z passes: R2C, C2R (real and paired).
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// R2C: tiles of about 4096 elements, 16 a thread, smaller on small grids, so
// that they spread over the GPU.  At its traffic's HBM time where the line's
// radices are powers of two (512^3: 0.44 ms for the 20 bytes a cell read,
// zeroed and written); elsewhere bound by issue, and by spills when it staged a
// tile at 256 threads whatever the side: us a pass, against that, 200^3 40 / 49,
// 320^3 134 / 215, 480^3 486 / 818, 768^3 2047 / 3191, 1000^3 4690 / 7378.
// (The C2R pass loses in this form, 0.40 against 0.28 ms at 512^3: every mode
// is read twice for the mirrored pairs.)
template <int NG> using ZT = ZTile<NG, NG <= 32 ? 256 : NG <= 48 ? 512 : NG <= 64 ? 1024 : NG <= 128 ? 2048 : 4096>;

// The density accumulator's z pass, and a real grid's.
template <int NG>
__global__ void __launch_bounds__(ZT<NG>::NT, ZT<NG>::MINB)
    zpass_rho_kernel(unsigned long long* __restrict__ rho, float2* __restrict__ out, int nlines, int zs, double mean, const float2* __restrict__ tw,
                     Slots sl) {
    using T = ZT<NG>;
    if (slot_idle(sl, blockIdx.y)) return;
    z_rho<NG, T::L, T::NT>(reinterpret_cast<float2*>(hgpm_smem), rho + (size_t)blockIdx.y * sl.s0,
                           out + (size_t)blockIdx.y * sl.s1, blockIdx.x * T::L, nlines, zs, mean, tw);
}

template <int NG>
__global__ void __launch_bounds__(ZT<NG>::NT, ZT<NG>::MINB)
    zpass_r2c_kernel(const float* __restrict__ in, float2* __restrict__ out, int nlines, int zs,
                     const float2* __restrict__ tw) {
    using T = ZT<NG>;
    z_r2c<NG, T::L, T::NT>(reinterpret_cast<float2*>(hgpm_smem), out, blockIdx.x * T::L, nlines, zs, tw,
                           [&](int line, int m) { return __ldcs(reinterpret_cast<const float2*>(in + (size_t)line * NG) + m); });
}

template <int NG>
__global__ void __launch_bounds__(kThreads) zpass_c2r_pair_kernel(const float2* __restrict__ in,
                                                                  float* __restrict__ out, int nlines, int zs,
                                                                  const float2* __restrict__ tw, Slots sl) {
    if (slot_idle(sl, blockIdx.y)) return;
    in += (size_t)blockIdx.y * sl.s0;
    out += (size_t)blockIdx.y * sl.s1;
    zpass_c2r_body<NG, true>(in, out, nlines, zs, 1.0f, tw, blockIdx.x);
}

template <int NG>
__global__ void __launch_bounds__(kThreads) zpass_c2r_kernel(const float2* __restrict__ in, float* __restrict__ out,
                                                             int nlines, int zs, size_t in_cs, size_t out_cs,
                                                             float scale, const float2* __restrict__ tw, int ncomp,
                                                             Slots sl) {
    const int slot = blockIdx.y / ncomp, comp = blockIdx.y % ncomp;
    if (slot_idle(sl, slot)) return;
    in += (size_t)slot * sl.s0 + (size_t)comp * in_cs;
    out += (size_t)slot * sl.s1 + (size_t)comp * out_cs;
    zpass_c2r_body<NG>(in, out, nlines, zs, scale, tw, blockIdx.x);
}

template <int NG>
static cudaError_t zfwd_impl(const float* in, float2* out, int nlines, int zs, const float2* tw, cudaStream_t s) {
    using T = ZT<NG>;
    auto k = zpass_r2c_kernel<NG>;
    cudaError_t e = ensure_smem(k, T::SMEM, T::NT);
    if (e != cudaSuccess) return e;
    k<<<cdiv(nlines, T::L), T::NT, T::SMEM, s>>>(in, out, nlines, zs, tw);
    return cudaGetLastError();
}

template <int NG>
static cudaError_t zrho_impl(unsigned long long* rho, float2* out, int zs, double mean, const float2* tw, cudaStream_t s,
                             const Slots& sl, int nslots) {
    using T = ZT<NG>;
    auto k = zpass_rho_kernel<NG>;
    cudaError_t e = ensure_smem(k, T::SMEM, T::NT);
    if (e != cudaSuccess) return e;
    k<<<dim3(cdiv(NG * NG, T::L), nslots), T::NT, T::SMEM, s>>>(rho, out, NG * NG, zs, mean, tw, sl);
    return cudaGetLastError();
}

template <int NG>
static cudaError_t zinv_impl(const float2* in, float* out, int nlines, int zs, size_t in_cs, size_t out_cs,
                             int ncomp, float scale, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    using G = Cfg<NG>;
    auto k = zpass_c2r_kernel<NG>;
    cudaError_t e = ensure_smem(k, G::ZSMEM, kThreads);
    if (e != cudaSuccess) return e;
    dim3 grid(cdiv(nlines, G::L), ncomp * nslots);
    k<<<grid, kThreads, G::ZSMEM, s>>>(in, out, nlines, zs, in_cs, out_cs, scale, tw, ncomp, sl);
    return cudaGetLastError();
}

template <int NG>
static cudaError_t zinv_pair_impl(const float2* in, float* out, int nlines, int zs, const float2* tw, cudaStream_t s,
                                  const Slots& sl, int nslots) {
    using G = Cfg<NG>;
    auto k = zpass_c2r_pair_kernel<NG>;
    cudaError_t e = ensure_smem(k, G::ZSMEM, kThreads);
    if (e != cudaSuccess) return e;
    k<<<dim3(cdiv(nlines, G::L), nslots), kThreads, G::ZSMEM, s>>>(in, out, nlines, zs, tw, sl);
    return cudaGetLastError();
}

bool fft_size_supported(int ng) {
    switch (ng) {
#define X(n) case n:
        HGPM_SIZES(X)
#undef X
        return true;
        default:
            return false;
    }
}

cudaError_t launch_zfwd(int ng, const float* in, float2* out, int nlines, int zs, const float2* tw, cudaStream_t s) {
    switch (ng) {
#define X(n) \
    case n: return zfwd_impl<n>(in, out, nlines, zs, tw, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_zfwd_rho(int ng, unsigned long long* rho, float2* out, int zs, double mean, const float2* tw,
                            cudaStream_t s, const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return zrho_impl<n>(rho, out, zs, mean, tw, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_zinv(int ng, const float2* in, float* out, int nlines, int zs, size_t in_cs, size_t out_cs,
                        int ncomp, float scale, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return zinv_impl<n>(in, out, nlines, zs, in_cs, out_cs, ncomp, scale, tw, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_zinv_pair(int ng, const float2* in, float* out, int zs, const float2* tw, cudaStream_t s,
                             const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return zinv_pair_impl<n>(in, out, n * n, zs, tw, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
