// fft_small.cu — the whole Poisson solve of a small box in one cluster.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// Density to paired potential with the half spectrum kept in the shared memory
// of a cluster of 8 CTAs, P planes of x each: the five passes of a small box
// are five kernels of 2.6 us that move at most 0.8 MB, bound by their launches
// and ramps.  A thread holds a whole line in registers (two radices, one
// group), so a pass is a read of the line, the butterflies and a write back of
// the same cells; the x lines are read and written across the cluster.  The
// butterflies are those of the separate passes, bit for bit.  us a step of one
// box back to back, after / before: 16^3 16 / 32, 24^3 22 / 32, 32^3 24 / 34,
// 40^3 36 / 39 (one CTA for the whole box: 20, 27, 44); three 32^3 boxes on
// streams of their own 9 / 20 a step.
template <int NG> struct SmallBox {
    static constexpr int M = NG / 2, H = M + 1;  // H odd: rows start on different banks
    static constexpr int CS = 8, P = NG / CS;
    static constexpr int YL = P * H, ZL = P * NG;  // y (and x) and z lines of a CTA
    static constexpr int NT = 128;
    static_assert(YL <= NT, "a thread for every y line");
};

template <int NG>
__global__ void __cluster_dims__(SmallBox<NG>::CS, 1, 1) __launch_bounds__(SmallBox<NG>::NT)
    solve_small_kernel(unsigned long long* __restrict__ rho, float* __restrict__ out, double mean,
                       const float2* __restrict__ tw, PotentialOp op) {
    using B = SmallBox<NG>;
    constexpr int M = B::M, H = B::H, NT = B::NT, P = B::P, ZL = B::ZL, YL = B::YL;
    using ZPlan = typename Plan<M>::type;
    using LPlan = typename Plan<NG>::type;
    static_assert(SeqProd<ZPlan>::value == M && SeqProd<LPlan>::value == NG, "a line is one group");
    __shared__ float2 s[P * NG * H];  // [x of this CTA][y][kz]
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = blockIdx.x;
    rho += (size_t)rank * P * NG * NG;
    out += (size_t)rank * P * NG * NG * 2;
    // the density less its mean, pairs of cells as complex; zeroed for the
    // next deposit
#pragma unroll 8
    for (int i = threadIdx.x; i < ZL * M; i += NT) {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(rho) + i;
        const ulonglong2 v = *q;
        *q = make_ulonglong2(0ull, 0ull);
        s[i / M * H + i % M] = make_float2((float)((double)(long long)v.x * kFixInv - mean),
                                           (float)((double)(long long)v.y * kFixInv - mean));
    }
    __syncthreads();
    // z lines, real to half spectrum (zpass_rho_kernel's split)
    for (int l = threadIdx.x; l < ZL; l += NT) {
        float2* row = s + l * H;
        float2 v[M];
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] = row[m];
        GroupRun<M, 1, false, 2, true, ZPlan>::run(v, 0, tw);
#pragma unroll
        for (int k = 0; k <= M / 2; ++k) {
            const float2 zk = v[k], zm = v[k ? M - k : 0];
            const float2 w = __ldg(&tw[k]);
            const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
            const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
            const float2 wo = cmul(w, o);
            row[k] = cadd(e, wo);
            if (k != M - k) {
                const float2 xm = csub(e, wo);
                row[M - k] = make_float2(xm.x, -xm.y);
            }
        }
    }
    __syncthreads();
    float2 v[NG];
    const bool mine = threadIdx.x < YL;
    const int x = threadIdx.x / H, kz = threadIdx.x % H;  // the y line's
    if (mine) {
#pragma unroll
        for (int e = 0; e < NG; ++e) v[e] = s[(x * NG + e) * H + kz];
        GroupRun<NG, 1, false, 1, true, LPlan>::run(v, 0, tw);
#pragma unroll
        for (int e = 0; e < NG; ++e) s[(x * NG + e) * H + kz] = v[e];
    }
    cl.sync();
    if (mine) {
        const int line = rank * YL + threadIdx.x, y = line / H, kx = line % H;  // the x line's y and kz
        float2* at[B::CS];
#pragma unroll
        for (int r = 0; r < B::CS; ++r) at[r] = cl.map_shared_rank(s, r) + y * H + kx;
#pragma unroll
        for (int e = 0; e < NG; ++e) v[e] = at[e / P][e % P * NG * H];
        GroupRun<NG, 1, false, 1, true, LPlan>::run(v, 0, tw);
        const double cyz = __ldg(&op.cosq[y]) + __ldg(&op.cosq[kx]);
#pragma unroll
        for (int e = 0; e < NG; ++e) v[e] = op.apply(__ldg(&op.cosq[e]), cyz, v[e]);
        GroupRun<NG, 1, true, 1, true, typename SeqRev<LPlan>::type>::run(v, 0, tw);
#pragma unroll
        for (int e = 0; e < NG; ++e) at[e / P][e % P * NG * H] = v[e];
    }
    cl.sync();
    if (mine) {
#pragma unroll
        for (int e = 0; e < NG; ++e) v[e] = s[(x * NG + e) * H + kz];
        GroupRun<NG, 1, true, 1, true, LPlan>::run(v, 0, tw);
#pragma unroll
        for (int e = 0; e < NG; ++e) s[(x * NG + e) * H + kz] = v[e];
    }
    __syncthreads();
    // z lines, half spectrum to real (zpass_c2r_body's split)
    for (int l = threadIdx.x; l < ZL; l += NT) {
        float2* row = s + l * H;
        float2 z[M];
#pragma unroll
        for (int k = 0; k <= M / 2; ++k) {
            float2 xk = row[k], xm = row[M - k];
            if (k == 0) {
                xk.y = 0.f;
                xm.y = 0.f;
            }
            const float2 w = __ldg(&tw[k]);
            const float2 p = make_float2(xk.x + xm.x, xk.y - xm.y);
            const float2 d = make_float2(xk.x - xm.x, xk.y + xm.y);
            const float2 cd = cmulc(d, w);
            const float2 tt = make_float2(-cd.y, cd.x);
            z[k] = cadd(p, tt);
            if (k != 0 && k != M - k) {
                const float2 zm = csub(p, tt);
                z[M - k] = make_float2(zm.x, -zm.y);
            }
        }
        GroupRun<M, 1, true, 2, true, ZPlan>::run(z, 0, tw);
#pragma unroll
        for (int m = 0; m < M; ++m) row[m] = z[m];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ZL * M; i += NT) {
        const int l = i / M, m = i % M;
        const float2 z = s[l * H + m];
        reinterpret_cast<float4*>(out)[i] = make_float4(z.x, z.y, z.y, s[l * H + (m + 1 == M ? 0 : m + 1)].x);
    }
}

// The sides whose lines are two radices (one group of registers).  40 gains
// least (36 against 39 us a step), so 64, the next such side, with four times
// its cells for each of the 8 CTAs, is left to the passes.
bool solve_small_supported(int ng) { return ng == 16 || ng == 24 || ng == 32 || ng == 40; }

cudaError_t launch_solve_small(int ng, unsigned long long* rho, float* out, double mean, const float2* tw,
                               const double* cosq, double coeff, cudaStream_t s) {
    const PotentialOp op{cosq, coeff};
    switch (ng) {
#define X(n)                                                                                     \
    case n:                                                                                      \
        solve_small_kernel<n><<<SmallBox<n>::CS, SmallBox<n>::NT, 0, s>>>(rho, out, mean, tw, op); \
        return cudaGetLastError();
        X(16) X(24) X(32) X(40)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
