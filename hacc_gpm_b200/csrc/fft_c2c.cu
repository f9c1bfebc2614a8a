// fft_c2c.cu — the 3D complex transform of a caller's grid.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// ---------------------------------------------------------------------------
// z pass of a complex-to-complex transform of a caller's [ng][ng][ng] grid
// (forward_fft / backward_fft on a cufftComplex grid, ffts.cu:244-294,
// 397-445), in place: a CTA transforms CZ<NG>::L contiguous z lines, 16
// elements a thread, in register groups (fft_rows).
template <int NG> struct CZ {
    static constexpr int L0 = 4096 / NG, L = L0 > 32 ? 32 : L0;  // lines a CTA
    static constexpr int NT0 = (NG * L / 16 + 31) / 32 * 32, NT = NT0;
    static constexpr int SMEM = L * RowTile<NG>::LS * 8;
};

template <int NG, bool INV>
__global__ void __launch_bounds__(CZ<NG>::NT, 1024 / CZ<NG>::NT > 16 ? 16 : 1024 / CZ<NG>::NT)
    zpass_c2c_kernel(float2* __restrict__ data, int nlines, const float2* __restrict__ tw) {
    constexpr int L = CZ<NG>::L;
    const int line0 = blockIdx.x * L;
    data += (size_t)line0 * NG;
    fft_rows<NG, L, CZ<NG>::NT, INV>(
        reinterpret_cast<float2*>(hgpm_smem), tw,
        [&](int l, int e) { return line0 + l < nlines ? __ldcs(data + l * NG + e) : make_float2(0.f, 0.f); },
        [&](int l, int e, float2 v) {
            if (line0 + l < nlines) __stcs(data + l * NG + e, v);
        });
}

template <int NG>
static cudaError_t c2c_impl(float2* data, bool inv, const float2* tw, cudaStream_t s) {
    constexpr int L = CZ<NG>::L;
    const int nlines = NG * NG;
    auto kz = inv ? zpass_c2c_kernel<NG, true> : zpass_c2c_kernel<NG, false>;
    cudaError_t e = ensure_smem(kz, CZ<NG>::SMEM, CZ<NG>::NT);
    if (e != cudaSuccess) return e;
    kz<<<cdiv(nlines, L), CZ<NG>::NT, CZ<NG>::SMEM, s>>>(data, nlines, tw);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // y lines (stride ng, planes x at ng^2), then x lines (stride ng^2,
    // planes y at ng); the z index is the contiguous column in both
    e = launch_strided(NG, inv, data, NG, (size_t)NG, (size_t)NG * NG, NG, 0, 1, tw, s, Slots{}, 1);
    if (e != cudaSuccess) return e;
    return launch_strided(NG, inv, data, NG, (size_t)NG * NG, (size_t)NG, NG, 0, 1, tw, s, Slots{}, 1);
}

cudaError_t launch_fft_c2c(int ng, float2* data, bool inv, const float2* tw, cudaStream_t s) {
    switch (ng) {
#define X(n) \
    case n: return c2c_impl<n>(data, inv, tw, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
