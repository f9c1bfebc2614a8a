// ===========================================================================
// Multi-class FFT passes (multi_class.h): one launch per pass over the work
// units of every class and slot, one CTA per unit.  The body is the one the
// single-class kernel runs (the z passes with 256 threads, the y and x passes
// with 512, for every size: a butterfly's arithmetic does not depend on which
// thread does it).
// ===========================================================================
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"
#include "multi_class.h"

namespace hgpm {

namespace {

// Threads and minimum CTAs per SM of each pass.  z passes: 256 threads, 3
// CTAs per SM (80 registers; the forward pass with half-height tiles from
// 192 up, MCCols::ZL, which bounds its register staging: 0.283 against
// 0.326 ms per ensemble step at 2 CTAs of 128 registers; the inverse 0.156
// against 0.184).  y and x passes: 512 x 2 (62 / 64 registers;
// the single-class configuration at 128^3 and above; 256 x 2 at 101 / 104
// registers measured the same at the 96-box ensemble).
constexpr int kMCYX = 512;
template <int PASS> constexpr int mc_threads() { return PASS == 0 || PASS == 4 ? 256 : kMCYX; }
template <int PASS> constexpr int mc_minb() { return PASS == 0 || PASS == 4 ? 3 : 2; }

// Columns per y / x tile.  Up to 128 a plane's ng/2 + 1 columns are split
// into the fewest even-width tiles that keep a stage at about two radix-8
// butterflies per thread (NG C <= 8192): the Nyquist column gets no tile of
// its own, which left most of a last tile empty (at 64: 33 columns in tiles
// of 16 or 32).  Larger sides keep the single-class widths.
template <int NG> struct MCCols {
    static constexpr int NC = NG / 2 + 1;
    static constexpr int TILES = ((NC + 1) / 2 * 2 * NG + 8191) / 8192;
    static constexpr int EVEN = ((NC + TILES - 1) / TILES + 1) / 2 * 2;
    static constexpr int Y = NG <= 128 ? EVEN : Cfg<NG>::CS;
    static constexpr int X = NG <= 128 ? EVEN : XW<NG>::C;
    // z lines per forward z tile: half the single-class count from 192 up,
    // which bounds the pass's register staging by the smaller sides'
    static constexpr int ZL = NG >= 192 ? Cfg<NG>::L / 2 : Cfg<NG>::L;
};

// One unit of each pass for one grid side.
template <int NG>
__device__ __forceinline__ void mc_zfwd_unit(const MCClass& c, int slot, int lu) {
    zpass_r2c_body<NG, true, MCCols<NG>::ZL>(c.rho64 + (size_t)slot * c.ncell, c.spec + (size_t)slot * c.spec_elems,
                                             NG * NG, c.zs, c.mean, c.tw, lu);
}
template <int NG, bool INV>
__device__ __forceinline__ void mc_ypass_unit(const MCClass& c, int slot, int lu) {
    float2* data = INV ? c.fspec + (size_t)slot * 3 * c.spec_elems : c.spec + (size_t)slot * c.spec_elems;
    constexpr int ncols = NG / 2 + 1, nch = (ncols + MCCols<NG>::Y - 1) / MCCols<NG>::Y;
    strided_body<NG, INV, kMCYX, MCCols<NG>::Y>(data, ncols, (size_t)c.zs, (size_t)NG * c.zs, c.tw, lu % nch,
                                                 lu / nch);
}
template <int NG>
__device__ __forceinline__ void mc_xpot_unit(const MCClass& c, int slot, int lu) {
    constexpr int ncols = NG / 2 + 1, nch = (ncols + MCCols<NG>::X - 1) / MCCols<NG>::X;
    const PotentialOp op{c.cosq, 0.5 / ((double)NG * NG * NG)};
    xone_body<NG, kMCYX, PotentialOp, MCCols<NG>::X>(c.spec + (size_t)slot * c.spec_elems, c.fspec + (size_t)slot * 3 * c.spec_elems, ncols,
                       (size_t)NG * c.zs, (size_t)c.zs, c.tw, op, lu % nch, lu / nch);
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
__global__ void __launch_bounds__(mc_threads<PASS>(), mc_minb<PASS>()) mc_fft_kernel(const __grid_constant__ MCTable t) {
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
    int zfunits, zunits, yunits, xunits;  // per slot (z forward, z inverse, y, x)
    int zsmem, ysmem, xsmem;
};
MCPassGeom mc_geom(int ng) {
    switch (ng) {
#define X(n)                                                                                            \
    case n: {                                                                                           \
        const int ncols = n / 2 + 1;                                                                    \
        return MCPassGeom{(n * n + MCCols<n>::ZL - 1) / MCCols<n>::ZL, (n * n + Cfg<n>::L - 1) / Cfg<n>::L,  \
                          (ncols + MCCols<n>::Y - 1) / MCCols<n>::Y * n,                                 \
                          (ncols + MCCols<n>::X - 1) / MCCols<n>::X * n, Cfg<n>::ZSMEM,                   \
                          n * MCCols<n>::Y * 8, n * MCCols<n>::X * 8};                                   \
    }
        HGPM_MC_SIZES(X)
#undef X
    }
    return MCPassGeom{0, 0, 0, 0, 0, 0, 0};
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
    int zf[kMaxMC], zu[kMaxMC], yu[kMaxMC], xu[kMaxMC];
    int zs = 0, ys = 0, xs = 0;
    for (int k = 0; k < base.n; ++k) {
        const MCPassGeom g = mc_geom(base.c[k].ng);
        if (!g.zunits) return cudaErrorInvalidValue;
        zf[k] = g.zfunits;
        zu[k] = g.zunits;
        yu[k] = g.yunits;
        xu[k] = g.xunits;
        zs = g.zsmem > zs ? g.zsmem : zs;
        ys = g.ysmem > ys ? g.ysmem : ys;
        xs = g.xsmem > xs ? g.xsmem : xs;
    }
    cudaError_t e = mc_launch((const void*)mc_fft_kernel<0>, base, zf, mc_threads<0>(), zs, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<1>, base, yu, mc_threads<1>(), ys, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<2>, base, xu, mc_threads<2>(), xs, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<3>, base, yu, mc_threads<3>(), ys, s);
    if (e == cudaSuccess) e = mc_launch((const void*)mc_fft_kernel<4>, base, zu, mc_threads<4>(), zs, s);
    return e;
}

}  // namespace hgpm
