// fft_strided.cu — the strided passes (y lines, x lines) in line tiles.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_tiles.cuh"

namespace hgpm {

// The strided pass in line tiles: ALL, every one of NG columns (a caller's
// complex grid), else a half spectrum's.  One CTA a tile: a tile's loads, its
// exchanges (one fewer than the plan's register groups) and its stores, other
// CTAs of the SM in between.
template <int NG, bool ALL>
using YT = LineTile<NG, NG <= 64 ? 1024 : NG <= 128 ? 2048 : NG <= 256 ? 4096 : NG < 384 ? 6144 : 8192,
                    ALL ? NG : NG / 2 + 1>;

// The y passes of a half spectrum, TMA-fed persistent (tma_passes.cu) against
// line tiles, us forward / inverse: 120: 13 / 13 against 11 / 11; 160: 18 / 17,
// 15 / 15; 192: 23 / 23, 23 / 23; 200: 26 / 26, 23 / 23; 240: 41 / 41, 37 / 37;
// 256: 35 / 36, 35 / 38; 320: 75 / 76, 74 / 81; 384: 125 / 126, 126 / 137; 400:
// 222 / 225, 157 / 166; 480: 254 / 257, 280 / 289; 512: 209 / 217, 280 / 293;
// 640: 616 / 617, 539 / 537; 768: 973 / 979, 1047 / 1013; 800: 1773 / 1762,
// 1549 / 1525; 960: 2309 / 1957, 2384 / 2363; 1000: 6951 / 6927, 2609 / 2625;
// 1024: 2242 / 2247, 2182 / 2132; 128: 12 / 12, 15 / 15; below alike, and line
// tiles need no tensor map.  The list is these measurements, not a rule in the
// side: the TMA-fed pass overlaps a tile's transform with the next one's load,
// the line tiles exchange less and, at long lines, have rows twice as wide.
// They win by most with two or three radix-5 stages (200, 400, 800, 1000), by
// a tenth at 120, 160, 240 and 640; at 320, 768, 960 and 1024 the two are close.
bool ypass_tma_default(int ng) {
    switch (ng) {
        case 128: case 192: case 256: case 320: case 384: case 480: case 512: case 768: case 960:
            return true;
        default:
            return false;
    }
}

template <int NG, bool INV, bool ALL>
__global__ void __launch_bounds__(YT<NG, ALL>::NT, YT<NG, ALL>::MINB)
    strided_kernel(float2* __restrict__ data, size_t rs, size_t ps, size_t cs, const float2* __restrict__ tw, Slots sl) {
    using T = YT<NG, ALL>;
    if (slot_idle(sl, blockIdx.z)) return;
    data += (size_t)blockIdx.z * sl.s0 + (size_t)blockIdx.y * cs;
    const LineCols<T, NG> cols{(int)blockIdx.x};
    fft_lines<NG, T::C, T::NT, INV>(
        reinterpret_cast<float2*>(hgpm_smem), tw,
        [&](int e, int c) {
            int plane, col;
            bool ok;
            cols.at(c, plane, col, ok);
            return ok ? __ldcs(data + (size_t)e * rs + (size_t)plane * ps + col) : make_float2(0.f, 0.f);
        },
        [&](int e, int c, float2 v) {
            int plane, col;
            bool ok;
            cols.at(c, plane, col, ok);
            if (ok) __stcs(data + (size_t)e * rs + (size_t)plane * ps + col, v);
        });
}

template <int NG, bool INV, bool ALL>
static cudaError_t strided_impl(float2* data, size_t rs, size_t ps, size_t cs, int ncomp, const float2* tw,
                                cudaStream_t s, const Slots& sl, int nslots) {
    using T = YT<NG, ALL>;
    auto k = strided_kernel<NG, INV, ALL>;
    cudaError_t e = ensure_smem(k, T::SMEM, T::NT);
    if (e != cudaSuccess) return e;
    k<<<dim3(T::TILES, ncomp, nslots), T::NT, T::SMEM, s>>>(data, rs, ps, cs, tw, sl);
    return cudaGetLastError();
}

template <int NG>
static cudaError_t strided_any(bool inv, float2* data, int ncols, size_t rs, size_t ps, int nplanes, size_t cs,
                               int ncomp, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    if (nplanes != NG) return cudaErrorInvalidValue;
    if (ncols == NG)
        return inv ? strided_impl<NG, true, true>(data, rs, ps, cs, ncomp, tw, s, sl, nslots)
                   : strided_impl<NG, false, true>(data, rs, ps, cs, ncomp, tw, s, sl, nslots);
    if (ncols != NG / 2 + 1) return cudaErrorInvalidValue;
    return inv ? strided_impl<NG, true, false>(data, rs, ps, cs, ncomp, tw, s, sl, nslots)
               : strided_impl<NG, false, false>(data, rs, ps, cs, ncomp, tw, s, sl, nslots);
}

cudaError_t launch_strided(int ng, bool inv, float2* data, int ncols, size_t rs, size_t ps, int nplanes, size_t cs,
                           int ncomp, const float2* tw, cudaStream_t s, const Slots& sl, int nslots) {
    switch (ng) {
#define X(n) \
    case n: return strided_any<n>(inv, data, ncols, rs, ps, nplanes, cs, ncomp, tw, s, sl, nslots);
        HGPM_SIZES(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

}  // namespace hgpm
