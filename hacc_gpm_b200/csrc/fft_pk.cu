// fft_pk.cu — the x pass fused with P(k).
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// ---------------------------------------------------------------------------
// x pass fused with P(k): forward x FFT, |delta|^2 * scale * CIC window, and
// deterministic per-warp FP64 shell sums.  Persistent CTAs take tiles
// blockIdx.x, +gridDim.x, ... and write one partial histogram each.
// ---------------------------------------------------------------------------
template <int NG>
__global__ void __launch_bounds__(kThreads) xpk_kernel(const float2* __restrict__ in, int ncols, size_t rs,
                                                       size_t ps, int nchunks, const float2* __restrict__ tw,
                                                       PkArgs a, double* __restrict__ part_sum,
                                                       unsigned long long* __restrict__ part_cnt) {
    constexpr int C = Cfg<NG>::CX;
    constexpr int M = NG / 2;
    constexpr int NW = kThreads / 32;
    float2* tile = reinterpret_cast<float2*>(hgpm_smem);
    double* hs = reinterpret_cast<double*>(tile + NG * C);
    unsigned long long* hc = reinterpret_cast<unsigned long long*>(hs + NW * a.nbins);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < NW * a.nbins; i += kThreads) {
        hs[i] = 0.0;
        hc[i] = 0ull;
    }
    const int ntiles = nchunks * NG;
    for (int tile_id = blockIdx.x; tile_id < ntiles; tile_id += gridDim.x) {
        const int chunk = tile_id % nchunks, iy = tile_id / nchunks;
        const int col0 = chunk * C;
        const int nvalid = ncols - col0;
        __syncthreads();
        load_tile<NG, C>(tile, in + (size_t)iy * ps + col0, rs, nvalid);
        __syncthreads();
        fft_tile<NG, C, C, false, kThreads>(tile, tw);
        // each warp walks its own cells in a fixed order
        for (int base = warp * 32; base < NG * C; base += kThreads) {
            const int i = base + lane;
            int bin = -1;
            double val = 0.0;
            int wgt = 0;
            if (i < NG * C) {
                const int ix = i / C, c = i % C, iz = col0 + c;
                const bool dc = (ix == 0 && iy == 0 && iz == 0);
                const bool corner = (ix == M && iy == M && iz == M);
                if (c < nvalid && !dc && !corner) {
                    const float kx = __ldg(&a.kf[ix]), ky = __ldg(&a.kf[iy]), kz = __ldg(&a.kf[iz]);
                    const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky)), __fmul_rn(kz, kz));
                    const float kmag = __fsqrt_rn(s2);
                    double fb;
                    if (a.log_bins) {
                        fb = log((double)kmag / a.min_k) / a.bin_delta;
                    } else {
                        fb = ((double)kmag - a.min_k) / a.bin_delta;
                    }
                    // (int) truncates, as calc_power_bins does (bin_power.cu:12-13):
                    // a mode just below minK lands in bin 0; further below
                    // the reference indexes before the array, here it is dropped
                    const int b = (int)fb;
                    if (b >= 0 && b < a.nbins) {
                        const float2 v = tile[i];
                        wgt = (iz == 0 || iz == M) ? 1 : 2;
                        const double p = ((double)v.x * v.x + (double)v.y * v.y) * a.scale *
                                         __ldg(&a.filt[ix]) * __ldg(&a.filt[iy]) * __ldg(&a.filt[iz]);
                        val = p * wgt;
                        bin = b;
                    }
                }
            }
            const unsigned grp = __match_any_sync(0xffffffffu, bin);
            const int leader = __ffs(grp) - 1;
            double s = 0.0;
            unsigned long long n = 0;
            unsigned m = grp;
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1;
                const double vv = __shfl_sync(grp, val, src);
                const int ww = __shfl_sync(grp, wgt, src);
                s += vv;
                n += (unsigned long long)ww;
            }
            if (lane == leader && bin >= 0) {
                hs[warp * a.nbins + bin] += s;
                hc[warp * a.nbins + bin] += n;
            }
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.nbins; b += kThreads) {
        double s = 0.0;
        unsigned long long n = 0;
        for (int w = 0; w < NW; ++w) {
            s += hs[w * a.nbins + b];
            n += hc[w * a.nbins + b];
        }
        part_sum[(size_t)blockIdx.x * a.nbins + b] = s;
        part_cnt[(size_t)blockIdx.x * a.nbins + b] = n;
    }
}

// Bin b's partial sums: one warp per bin, lane l adding partials l, l + 32,
// ... in order, then the 32 lane sums combined by a fixed shuffle tree (a
// fixed order: deterministic run to run).
__global__ void pk_reduce_kernel(const double* __restrict__ part_sum, const unsigned long long* __restrict__ part_cnt,
                                 int nparts, int nbins, double* __restrict__ sum, unsigned long long* __restrict__ cnt) {
    const int b = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (b >= nbins) return;  // whole warps
    double s = 0.0;
    unsigned long long n = 0;
    for (int p = lane; p < nparts; p += 32) {
        s += part_sum[(size_t)p * nbins + b];
        n += part_cnt[(size_t)p * nbins + b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        n += __shfl_down_sync(0xffffffffu, n, o);
    }
    if (lane == 0) {
        sum[b] = s;
        cnt[b] = n;
    }
}

template <int NG>
static cudaError_t xpk_impl(const float2* in, int ncols, size_t rs, size_t ps, const float2* tw, const PkArgs& a,
                            double* part_sum, unsigned long long* part_cnt, int nparts, double* sum,
                            unsigned long long* cnt, cudaStream_t s) {
    using G = Cfg<NG>;
    constexpr int NW = kThreads / 32;
    const int smem = NG * G::CX * 8 + NW * a.nbins * 16;
    auto k = xpk_kernel<NG>;
    cudaError_t e = smem_attr_once((const void*)k, smem, kThreads);
    if (e != cudaSuccess) return e;
    const int nchunks = cdiv(ncols, G::CX);
    k<<<nparts, kThreads, smem, s>>>(in, ncols, rs, ps, nchunks, tw, a, part_sum, part_cnt);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    pk_reduce_kernel<<<cdiv((size_t)a.nbins * 32, 256), 256, 0, s>>>(part_sum, part_cnt, nparts, a.nbins, sum, cnt);
    return cudaGetLastError();
}

cudaError_t launch_xpk(int ng, const float2* in, int ncols, size_t rs, size_t ps, const float2* tw, const PkArgs& a,
                       double* part_sum, unsigned long long* part_cnt, int nparts, double* sum,
                       unsigned long long* cnt, cudaStream_t s) {
    switch (ng) {
#define X(n) \
    case n: return xpk_impl<n>(in, ncols, rs, ps, tw, a, part_sum, part_cnt, nparts, sum, cnt, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

int pk_max_bins() { return 1024; }

}  // namespace hgpm
