// fft_strided.cu — the plain strided passes (y lines, x lines).
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

template <int NG, bool INV>
__global__ void __launch_bounds__(Cfg<NG>::NTS, 2) strided_kernel(float2* __restrict__ data, int ncols, size_t rs,
                                                               size_t ps, size_t cs, const float2* __restrict__ tw,
                                                               int ncomp, Slots sl) {
    const int slot = blockIdx.z / ncomp, comp = blockIdx.z % ncomp;
    if (slot_idle(sl, slot)) return;
    strided_body<NG, INV, Cfg<NG>::NTS>(data + (size_t)slot * sl.s0 + (size_t)comp * cs, ncols, rs, ps, tw,
                                        blockIdx.x, blockIdx.y);
}

template <int NG>
static cudaError_t strided_impl(bool inv, float2* data, int ncols, size_t rs, size_t ps, int nplanes, size_t cs,
                                int ncomp, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    using G = Cfg<NG>;
    dim3 grid(cdiv(ncols, G::CS), nplanes, ncomp * nslots);
    if (inv) {
        auto k = strided_kernel<NG, true>;
        cudaError_t e = ensure_smem(k, G::SSMEM);
        if (e != cudaSuccess) return e;
        k<<<grid, G::NTS, G::SSMEM, s>>>(data, ncols, rs, ps, cs, tw, ncomp, sl);
    } else {
        auto k = strided_kernel<NG, false>;
        cudaError_t e = ensure_smem(k, G::SSMEM);
        if (e != cudaSuccess) return e;
        k<<<grid, G::NTS, G::SSMEM, s>>>(data, ncols, rs, ps, cs, tw, ncomp, sl);
    }
    return cudaGetLastError();
}

cudaError_t launch_strided(int ng, bool inv, float2* data, int ncols, size_t rs, size_t ps, int nplanes, size_t cs,
                           int ncomp, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return strided_impl<n>(inv, data, ncols, rs, ps, nplanes, cs, ncomp, tw, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
