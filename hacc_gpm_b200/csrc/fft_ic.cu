// fft_ic.cu — the x pass fused with the IC displacement operator.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

cudaError_t launch_xic(int n, const float2* in, float2* out, int ncols, size_t rs, size_t ps, int nplanes,
                       size_t out_cs, const float2* tw, const double* table, int nbins, double k_delta,
                       double pkscale, double inv_delta, const float* kf, int* err, cudaStream_t s) {
    ICOp op{table, nbins, k_delta, pkscale, inv_delta, kf, err, n / 2};
    switch (n) {
#define X(m) \
    case m: return xfused_impl<m, ICOp>(in, out, ncols, rs, ps, nplanes, out_cs, tw, op, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
