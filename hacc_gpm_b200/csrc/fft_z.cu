// fft_z.cu — the z passes: R2C, C2R (real and paired).
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// The single-class kernel: zpass_r2c_body's code with the slot prologue
// written out (as a kernel with its own restrict-qualified parameters it
// compiles without the body's 76 bytes of spills at 512^3).
template <int NG, bool FIX>
__global__ void __launch_bounds__(kThreads, 4) zpass_r2c_kernel(void* __restrict__ in_, float2* __restrict__ out,
                                                             int nlines, int zs, double mean,
                                                             const float2* __restrict__ tw, Slots sl) {
    constexpr int M = NG / 2, L = Cfg<NG>::L, ES = L + 1;
    float2* buf = reinterpret_cast<float2*>(hgpm_smem);
    if (slot_idle(sl, blockIdx.y)) return;
    // slot stride s0 counts input elements (int64 when FIX, float otherwise)
    in_ = FIX ? (void*)(reinterpret_cast<unsigned long long*>(in_) + (size_t)blockIdx.y * sl.s0)
              : (void*)(reinterpret_cast<float*>(in_) + (size_t)blockIdx.y * sl.s0);
    out += (size_t)blockIdx.y * sl.s1;
    const int line0 = blockIdx.x * L;
    constexpr int TOT = L * M;
    constexpr int PER = (TOT + kThreads - 1) / kThreads;
    if (FIX) {
        ulonglong2 q[PER];
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * kThreads;
            const int l = i / M, m = i % M;
            q[t] = make_ulonglong2(0ull, 0ull);
            if (((TOT % kThreads) == 0 || i < TOT) && line0 + l < nlines)
                q[t] = __ldcs(reinterpret_cast<const ulonglong2*>(reinterpret_cast<unsigned long long*>(in_) +
                                                                  (size_t)(line0 + l) * NG) + m);
        }
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * kThreads;
            const int l = i / M, m = i % M;
            if (((TOT % kThreads) == 0 || i < TOT)) {
                if (line0 + l < nlines)
                    __stcs(reinterpret_cast<ulonglong2*>(reinterpret_cast<unsigned long long*>(in_) +
                                                         (size_t)(line0 + l) * NG) + m, make_ulonglong2(0ull, 0ull));
                buf[m * ES + l] = make_float2((float)((double)(long long)q[t].x * kFixInv - mean),
                                              (float)((double)(long long)q[t].y * kFixInv - mean));
            }
        }
    } else {
        float2 z[PER];
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * kThreads;
            const int l = i / M, m = i % M;
            z[t] = make_float2(0.f, 0.f);
            if (((TOT % kThreads) == 0 || i < TOT) && line0 + l < nlines)
                z[t] = reinterpret_cast<const float2*>(reinterpret_cast<const float*>(in_) + (size_t)(line0 + l) * NG)[m];
        }
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * kThreads;
            if ((TOT % kThreads) == 0 || i < TOT) buf[(i % M) * ES + i / M] = z[t];
        }
    }
    __syncthreads();
    fft_tile<M, L, ES, false, kThreads, 2>(buf, tw);
    constexpr int H = M / 2 + 1;
    for (int i = threadIdx.x; i < L * H; i += kThreads) {
        const int l = i / H, k = i % H;
        const int line = line0 + l;
        if (line >= nlines) continue;
        const float2 zk = buf[k * ES + l];
        const float2 zm = buf[((M - k) % M) * ES + l];
        const float2 w = __ldg(&tw[k]);
        // E = (Zk + conj Zm)/2, O = -i (Zk - conj Zm)/2, X[k] = E + w O,
        // X[M-k] = conj(E - w O)
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
        const float2 wo = cmul(w, o);
        float2* dst = out + (size_t)line * zs;
        dst[k] = cadd(e, wo);
        if (k != M - k) {
            const float2 xm = csub(e, wo);
            dst[M - k] = make_float2(xm.x, -xm.y);
        }
    }
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
static cudaError_t zfwd_impl(void* in, bool fixed, float2* out, int nlines, int zs, double mean,
                             const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    using G = Cfg<NG>;
    const dim3 grid(cdiv(nlines, G::L), nslots);
    if (fixed) {
        auto k = zpass_r2c_kernel<NG, true>;
        cudaError_t e = ensure_smem(k, G::ZSMEM, kThreads);
        if (e != cudaSuccess) return e;
        k<<<grid, kThreads, G::ZSMEM, s>>>(in, out, nlines, zs, mean, tw, sl);
    } else {
        auto k = zpass_r2c_kernel<NG, false>;
        cudaError_t e = ensure_smem(k, G::ZSMEM, kThreads);
        if (e != cudaSuccess) return e;
        k<<<grid, kThreads, G::ZSMEM, s>>>(in, out, nlines, zs, mean, tw, sl);
    }
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

cudaError_t launch_zfwd(int ng, void* in, bool fixed, float2* out, int nlines, int zs, double mean,
                        const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return zfwd_impl<n>(in, fixed, out, nlines, zs, mean, tw, s, sl, nslots);
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
