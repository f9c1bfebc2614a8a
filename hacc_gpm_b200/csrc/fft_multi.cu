// ===========================================================================
// Multi-class FFT passes (multi_class.h): one launch per pass over the work
// units of every class and slot, one CTA of 256 threads per unit.  The inverse
// z pass runs the single-class kernel's body; the forward z pass and the flat y
// and x tiles are this file's own.  The bits are the single-class passes' all
// the same: a butterfly's arithmetic does not depend on which thread does it.
// ===========================================================================
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"
#include "multi_class.h"

namespace hgpm {

namespace {

// Threads and minimum CTAs per SM of each pass.  z passes: 256 threads, 3
// CTAs per SM (80 registers; the forward pass with half-height tiles from
// 192 up, kZLines, which bounds its register staging: 0.283 against 0.326 ms
// per ensemble step at 2 CTAs of 128 registers; the inverse 0.156 against
// 0.184).  y and x passes: 256 threads, 4 CTAs per SM.
constexpr int kMCThreads = 256;
template <int PASS> constexpr int mc_minb() { return PASS == 0 || PASS == 4 ? 3 : 4; }

// The y and x passes' tiles: 4096 elements whatever the side, 16 a thread, the
// box's lines (NG planes of NG/2 + 1 columns) taken as they come, so that
// every thread of every CTA has work on every side (a plane's columns alone
// fill a small side's tile to a fourth, and its Nyquist column none).
template <int NG> struct FlatTile {
    static constexpr int H = NG / 2 + 1, C = 4096 / NG, TILES = (NG * H + C - 1) / C;
    int t;
    __device__ __forceinline__ void at(int c, int& plane, int& col, bool& ok) const {
        const int f = t * C + c;
        plane = f / H;
        col = f - plane * H;
        ok = plane < NG;
    }
};
// z lines per forward z tile: half the single-class count from 192 up
template <int NG> constexpr int kZLines = NG >= 192 ? Cfg<NG>::L / 2 : Cfg<NG>::L;

// One unit of each pass for one grid side.
template <int NG>
__device__ __forceinline__ void mc_zfwd_unit(const MCClass& c, int slot, int lu) {
    zpass_rho_body<NG, kZLines<NG>>(c.rho64 + (size_t)slot * c.ncell, c.spec + (size_t)slot * c.spec_elems, NG * NG,
                                    c.zs, c.mean, c.tw, lu);
}
template <int NG, bool INV>
__device__ __forceinline__ void mc_ypass_unit(const MCClass& c, int slot, int lu) {
    float2* data = INV ? c.fspec + (size_t)slot * 3 * c.spec_elems : c.spec + (size_t)slot * c.spec_elems;
    const FlatTile<NG> cols{lu};
    const int zs = c.zs;
    fft_lines<NG, FlatTile<NG>::C, kMCThreads, INV>(
        reinterpret_cast<float2*>(hgpm_smem), c.tw,
        [&](int e, int l) {
            int ix, iz;
            bool ok;
            cols.at(l, ix, iz, ok);
            return ok ? __ldcs(data + (ix * NG + e) * zs + iz) : make_float2(0.f, 0.f);
        },
        [&](int e, int l, float2 v) {
            int ix, iz;
            bool ok;
            cols.at(l, ix, iz, ok);
            if (ok) __stcs(data + (ix * NG + e) * zs + iz, v);
        });
}
template <int NG>
__device__ __forceinline__ void mc_xpot_unit(const MCClass& c, int slot, int lu) {
    const PotentialOp op{c.cosq, 0.5 / ((double)NG * NG * NG)};
    const float2* in = c.spec + (size_t)slot * c.spec_elems;
    float2* out = c.fspec + (size_t)slot * 3 * c.spec_elems;
    const FlatTile<NG> cols{lu};
    const int zs = c.zs;
    fft_lines_fwd_op_inv<NG, FlatTile<NG>::C, kMCThreads>(
        reinterpret_cast<float2*>(hgpm_smem), c.tw,
        [&](int e, int l) {
            int iy, iz;
            bool ok;
            cols.at(l, iy, iz, ok);
            return ok ? __ldcs(in + (e * NG + iy) * zs + iz) : make_float2(0.f, 0.f);
        },
        [&](int e, int l, float2 v) {
            int iy, iz;
            bool ok;
            cols.at(l, iy, iz, ok);
            if (ok) __stcs(out + (e * NG + iy) * zs + iz, v);
        },
        [&](int ix, int l, float2 v) {
            int iy, iz;
            bool ok;
            cols.at(l, iy, iz, ok);
            if (!ok) iy = iz = 0;
            return op.apply(__ldg(&op.cosq[ix]), __ldg(&op.cosq[iy]) + __ldg(&op.cosq[iz]), v);
        });
}
template <int NG>
__device__ __forceinline__ void mc_zinv_unit(const MCClass& c, int slot, int lu) {
    zpass_c2r_body<NG, true>(c.fspec + (size_t)slot * 3 * c.spec_elems, c.force + (size_t)slot * c.force_elems,
                             NG * NG, c.zs, 1.0f, c.tw, lu);
}

// PASS: 0 z forward, 1 y forward, 2 x with the Green's function, 3 y
// inverse, 4 z inverse.  One CTA per unit: CTA u of the launch is unit u -
// u0[k] of class k (slot (u - u0[k]) / per[k]).  (A persistent grid whose CTAs
// each serve one class ran 1.7-2.2x slower at the 96-box ensemble: CTAs
// shared out by points per unit starve the small sides, whose tiles cost
// nearly as much as large ones; the block scheduler balances by itself.)
template <int PASS>
__global__ void __launch_bounds__(kMCThreads, mc_minb<PASS>()) mc_fft_kernel(const __grid_constant__ MCTable t) {
    const int u = blockIdx.x;
    int k = 0;
    while (k + 1 < t.n && u >= t.u0[k + 1]) ++k;
    const MCClass& c = t.c[k];
    const int r = u - t.u0[k], slot = r / t.per[k], lu = r - slot * t.per[k];
    if (c.active && !c.active[slot]) return;
    switch (c.ng) {
#define X(n)                                                     \
    case n:                                                      \
        if (PASS == 0) mc_zfwd_unit<n>(c, slot, lu);             \
        else if (PASS == 1) mc_ypass_unit<n, false>(c, slot, lu); \
        else if (PASS == 2) mc_xpot_unit<n>(c, slot, lu);        \
        else if (PASS == 3) mc_ypass_unit<n, true>(c, slot, lu); \
        else mc_zinv_unit<n>(c, slot, lu);                       \
        break;
        HGPM_MC_SIZES(X)
#undef X
    }
}

// Per-size unit counts and shared memory of the passes (host).
struct MCPassGeom {
    int zfunits, zunits, yunits;  // per slot (z forward, z inverse, y and x)
    int zsmem, ysmem;
};
MCPassGeom mc_geom(int ng) {
    switch (ng) {
#define X(n)                                                                                           \
    case n:                                                                                            \
        return MCPassGeom{(n * n + kZLines<n> - 1) / kZLines<n>, (n * n + Cfg<n>::L - 1) / Cfg<n>::L, \
                          FlatTile<n>::TILES, Cfg<n>::ZSMEM, n * FlatTile<n>::C * 8};
        HGPM_MC_SIZES(X)
#undef X
    }
    return MCPassGeom{0, 0, 0, 0, 0};
}

// One launch of `kern` (`threads` per CTA, `smem` bytes), one CTA per unit
// of every class's slots.
cudaError_t mc_launch(const void* kern, MCTable t, const int* units, int threads, int smem, cudaStream_t s) {
    t.u0[0] = 0;
    for (int k = 0; k < t.n; ++k) {
        t.per[k] = units[k];
        t.u0[k + 1] = t.u0[k] + units[k] * t.c[k].nslots;
    }
    if (t.u0[t.n] == 0) return cudaSuccess;
    cudaError_t e = smem_attr_once(kern, smem, threads);
    if (e != cudaSuccess) return e;
    void* args[] = {&t};
    return cudaLaunchKernel(kern, dim3(t.u0[t.n]), dim3(threads), args, smem, s);
}

}  // namespace

cudaError_t mc_launch_fft_passes(const MCTable& base, cudaStream_t s) {
    int zf[kMaxMC], zu[kMaxMC], yu[kMaxMC];
    int zs = 0, ys = 0;
    for (int k = 0; k < base.n; ++k) {
        const MCPassGeom g = mc_geom(base.c[k].ng);
        if (!g.zunits) return cudaErrorInvalidValue;
        zf[k] = g.zfunits;
        zu[k] = g.zunits;
        yu[k] = g.yunits;
        zs = g.zsmem > zs ? g.zsmem : zs;
        ys = g.ysmem > ys ? g.ysmem : ys;
    }
    cudaError_t e = mc_launch((const void*)mc_fft_kernel<0>, base, zf, kMCThreads, zs, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<1>, base, yu, kMCThreads, ys, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<2>, base, yu, kMCThreads, ys, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<3>, base, yu, kMCThreads, ys, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<4>, base, zu, kMCThreads, zs, s);
    return e;
}

}  // namespace hgpm
