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
// Bound by issue: 28 instructions an element went to the bin's double division
// and about as many to summing a warp's equal bins one lane after the other.
// The bin is now found in single precision and settled in double only within
// 1e-3 of an edge (its error is below 3e-4 of a bin for the 1024 bins allowed:
// the same bins, mode for mode), equal bins are summed in five rounds of
// pointer jumping, and what depends on a line's column alone is formed once a
// tile: P(k) of 256^3 in 221 bins 519 -> 385 us (this kernel 222 -> 88), 1024^3
// cells 25.7 -> 15.0 ms.
template <int NG> using PT = LineTile<NG, NG <= 512 ? 4096 : 8192>;
// (at most 256 threads: 8 histograms of 1024 bins fit beside the tile)
template <int NG> constexpr int pk_threads() { return PT<NG>::NT < 128 ? 128 : PT<NG>::NT > 256 ? 256 : PT<NG>::NT; }

// What a tile's line contributes to every mode on it.
struct PkLine {
    double g;         // scale times the CIC window of ky and kz
    float ky2, kz2;
    int iy, iz;       // iz < 0: an empty line
};

__device__ __forceinline__ int pk_bin(const PkArgs& a, float min_k, float inv, float kmag) {
    const float f = a.log_bins ? logf(kmag * min_k) * inv : (kmag - min_k) * inv;
    if (fabsf(f - rintf(f)) > 1e-3f) return (int)f;
    // (int) truncates, as calc_power_bins does (bin_power.cu:12-13): a mode
    // just below minK lands in bin 0; further below the reference indexes
    // before the array, here it is dropped
    const double fb = a.log_bins ? log((double)kmag / a.min_k) / a.bin_delta : ((double)kmag - a.min_k) / a.bin_delta;
    return (int)fb;
}

template <int NG>
__global__ void __launch_bounds__(pk_threads<NG>(), (NG & (NG - 1)) == 0 && NG <= 512 ? 768 / pk_threads<NG>() : 2) xpk_kernel(const float2* __restrict__ in, int zs,
                                                               const float2* __restrict__ tw, PkArgs a,
                                                               double* __restrict__ part_sum,
                                                               unsigned long long* __restrict__ part_cnt) {
    using T = PT<NG>;
    constexpr int C = T::C, NT = pk_threads<NG>(), NW = NT / 32, M = NG / 2;
    float2* tile = reinterpret_cast<float2*>(hgpm_smem);
    double* hs = reinterpret_cast<double*>(tile + NG * C);
    unsigned long long* hc = reinterpret_cast<unsigned long long*>(hs + NW * a.nbins);
    __shared__ PkLine line[C];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < NW * a.nbins; i += NT) {
        hs[i] = 0.0;
        hc[i] = 0ull;
    }
    const float min_k = a.log_bins ? (float)(1.0 / a.min_k) : (float)a.min_k, inv = (float)(1.0 / a.bin_delta);
    const size_t rs = (size_t)NG * zs;
    for (int t = blockIdx.x; t < T::TILES; t += gridDim.x) {
        const LineCols<T, NG> cols{t};
        __syncthreads();  // the last tile's modes are binned
        for (int c = threadIdx.x; c < C; c += NT) {
            int iy, iz;
            bool ok;
            cols.at(c, iy, iz, ok);
            PkLine l{0.0, 0.f, 0.f, 0, -1};
            if (ok) {
                const float ky = __ldg(&a.kf[iy]), kz = __ldg(&a.kf[iz]);
                l = PkLine{a.scale * __ldg(&a.filt[iy]) * __ldg(&a.filt[iz]), __fmul_rn(ky, ky), __fmul_rn(kz, kz), iy, iz};
            }
            line[c] = l;
        }
        run_groups<NG, C, NT, false, 1, 1, true, false, true>(
            tile, tw,
            [&](int e, int c) {
                int iy, iz;
                bool ok;
                cols.at(c, iy, iz, ok);
                return ok ? __ldcs(in + (size_t)e * rs + (size_t)iy * zs + iz) : make_float2(0.f, 0.f);
            },
            [](int, int, float2) {}, GroupPlan<NG>{});
        // each warp walks its own cells in a fixed order (NG C is a multiple of 32)
        for (int base = warp * 32; base < NG * C; base += NT) {
            const int i = base + lane;
            const int ix = i / C, c = i % C;
            const PkLine l = line[c];
            int bin = -1;
            double val = 0.0;
            const bool dc = ix == 0 && l.iy == 0 && l.iz == 0;
            const bool corner = ix == M && l.iy == M && l.iz == M;
            const bool twice = l.iz != 0 && l.iz != M;
            if (l.iz >= 0 && !dc && !corner) {
                const float kx = __ldg(&a.kf[ix]);
                const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(kx, kx), l.ky2), l.kz2);
                const int b = pk_bin(a, min_k, inv, __fsqrt_rn(s2));
                if (b >= 0 && b < a.nbins) {
                    const float2 v = tile[tile_at<C>(ix, c)];
                    val = ((double)v.x * v.x + (double)v.y * v.y) * l.g * __ldg(&a.filt[ix]);
                    if (twice) val += val;
                    bin = b;
                }
            }
            // the warp's equal bins: each lane adds the next member's sum, then
            // the sum of the one after what that covered, and so on; the lowest
            // lane ends with the whole group's (a fixed order)
            const unsigned grp = __match_any_sync(0xffffffffu, bin);
            const unsigned pairs = __ballot_sync(0xffffffffu, twice);
            const unsigned above = grp & (0xfffffffeu << lane);
            int nxt = above ? __ffs(above) - 1 : lane;
#pragma unroll
            for (int r = 0; r < 5; ++r) {
                const double vv = __shfl_sync(0xffffffffu, val, nxt);
                const int nn = __shfl_sync(0xffffffffu, nxt, nxt);
                // a lane at the end of its chain points at itself
                if (nxt != lane) val += vv;
                nxt = nxt == lane || nn == nxt ? lane : nn;
            }
            if (bin >= 0 && lane == __ffs(grp) - 1) {
                hs[warp * a.nbins + bin] += val;
                hc[warp * a.nbins + bin] += (unsigned long long)(__popc(grp) + __popc(grp & pairs));
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.nbins; b += NT) {
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
static cudaError_t xpk_impl(const float2* in, int zs, const float2* tw, const PkArgs& a, double* part_sum,
                            unsigned long long* part_cnt, int nparts, double* sum, unsigned long long* cnt,
                            cudaStream_t s) {
    constexpr int NT = pk_threads<NG>();
    const int smem = PT<NG>::SMEM + NT / 32 * a.nbins * 16;
    auto k = xpk_kernel<NG>;
    cudaError_t e = smem_attr_once((const void*)k, smem, NT);
    if (e != cudaSuccess) return e;
    // as many CTAs as are resident at once (the histograms' size is the caller's)
    int dev = 0, sms = 0, per_sm = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, NT, smem);
    if (e != cudaSuccess) return e;
    if (per_sm > 0 && sms * per_sm < nparts) nparts = sms * per_sm;
    if (PT<NG>::TILES < nparts) nparts = PT<NG>::TILES;
    k<<<nparts, NT, smem, s>>>(in, zs, tw, a, part_sum, part_cnt);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    pk_reduce_kernel<<<cdiv((size_t)a.nbins * 32, 256), 256, 0, s>>>(part_sum, part_cnt, nparts, a.nbins, sum, cnt);
    return cudaGetLastError();
}

cudaError_t launch_xpk(int ng, const float2* in, int zs, const float2* tw, const PkArgs& a, double* part_sum,
                       unsigned long long* part_cnt, int nparts, double* sum, unsigned long long* cnt,
                       cudaStream_t s) {
    switch (ng) {
#define X(n) \
    case n: return xpk_impl<n>(in, zs, tw, a, part_sum, part_cnt, nparts, sum, cnt, s);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

int pk_max_bins() { return 1024; }

}  // namespace hgpm
