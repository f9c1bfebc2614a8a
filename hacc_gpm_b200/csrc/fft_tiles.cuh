// fft_tiles.cuh — the device bodies of the 3D R2C/C2R FFT passes of the PM step
// (fft_z.cu, fft_strided.cu, fft_x.cu, fft_pk.cu, fft_plane.cu, fft_multi.cu).
//
// Layouts (row-major, z fastest, as get_index in src/haccgpm.hpp:423-429):
//   real grid      float  [ng][ng][ng]
//   half spectrum  float2 [ng][ng][zs]   kz in [0, ng/2], zs = padded row
// The forward 3D transform is: z pass (R2C along contiguous rows) ->
// y pass (strided, in place) -> x pass (strided).  The inverse runs the
// passes in reverse order with a C2R z pass.  The step never materialises
// the forward x output: the x pass is fused with the Green's function and
// gradient (Poisson), with the IC displacement operator, or with P(k)
// binning, all of which act on one x-line tile while it is in shared memory.
#include <cuda_runtime.h>
#pragma once
#include <stdint.h>
#include <math.h>


#include "fft_engine.cuh"
#include "hgpm_device.cuh"
#include "hgpm_internal.h"
#include "kspace_ops.cuh"

namespace hgpm {

extern __shared__ float4 hgpm_smem[];

// ---------------------------------------------------------------------------
// per-size tile configuration
// ---------------------------------------------------------------------------
template <int NG> struct Cfg {
    static constexpr int M = NG / 2;                       // complex length of z lines
    static constexpr int L = M >= 512 ? 8 : (M >= 256 ? 16 : (M >= 96 ? 32 : 64));  // z lines per CTA
    static constexpr int CX = NG >= 768 ? 4 : (NG >= 384 ? 8 : 16);  // fused x-pass columns
    static constexpr int ZSMEM = M * (L + 1) * 8;
    static constexpr int XSMEM = 2 * NG * CX * 8;
    // threads per CTA of the fused x pass: 512 halves the per-thread register
    // staging so two CTAs (32 warps) fit per SM
    static constexpr int NTX = NG >= 128 ? 512 : 256;
};

// ---------------------------------------------------------------------------
// tile load/store between global strided lines and shared [N][C]
// ---------------------------------------------------------------------------
// Rows e in [0, N) at g + e*rs; columns [0, nvalid) valid (nvalid may be < C).
// All of a thread's global loads are issued before any shared store
// (register staging) so each CTA keeps its whole tile in flight.  CG: loads
// from L2 (ld.global.cg), for data other CTAs of the same kernel wrote.
template <int N, int C, int NT = kThreads, bool CG = false>
__device__ __forceinline__ void load_tile(float2* __restrict__ tile, const float2* __restrict__ g,
                                          size_t rs, int nvalid) {
    constexpr int TPR = C / 2;  // float4 (two complex) per row chunk
    constexpr int TOT = N * TPR;
    constexpr int PER = (TOT + NT - 1) / NT;
    float4 v[PER];
    if (nvalid >= C) {
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * NT;
            if ((TOT % NT) == 0 || i < TOT) {
                const int e = i / TPR, c = 2 * (i % TPR);
                const float4* src = reinterpret_cast<const float4*>(g + (size_t)e * rs + c);
                v[t] = CG ? __ldcg(src) : __ldcs(src);
            }
        }
    } else {
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int i = threadIdx.x + t * NT;
            v[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            if ((TOT % NT) == 0 || i < TOT) {
                const int e = i / TPR, c = 2 * (i % TPR);
                const float2* src = g + (size_t)e * rs + c;
                if (c + 1 < nvalid) {
                    v[t] = CG ? __ldcg(reinterpret_cast<const float4*>(src)) : *reinterpret_cast<const float4*>(src);
                } else if (c < nvalid) {
                    const float2 s = CG ? __ldcg(src) : src[0];
                    v[t] = make_float4(s.x, s.y, 0.f, 0.f);
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * NT;
        if ((TOT % NT) == 0 || i < TOT) {
            const int e = i / TPR, c = 2 * (i % TPR);
            *reinterpret_cast<float4*>(&tile[e * C + c]) = v[t];
        }
    }
}

// WB: write-back stores (kept in L2 for a read later in the same kernel)
// instead of streaming ones.
template <int N, int C, int NT = kThreads, bool WB = false>
__device__ __forceinline__ void store_tile(const float2* __restrict__ tile, float2* __restrict__ g,
                                           size_t rs, int nvalid) {
    constexpr int TPR = C / 2;
    constexpr int TOT = N * TPR;
    constexpr int PER = (TOT + NT - 1) / NT;
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * NT;
        if ((TOT % NT) == 0 || i < TOT) {
            const int e = i / TPR, c = 2 * (i % TPR);
            float2* dst = g + (size_t)e * rs + c;
            const float4 v = *reinterpret_cast<const float4*>(&tile[e * C + c]);
            if (c + 1 < nvalid) {
                if (WB) *reinterpret_cast<float4*>(dst) = v;
                else __stcs(reinterpret_cast<float4*>(dst), v);
            } else if (c < nvalid) {
                dst[0] = make_float2(v.x, v.y);
            }
        }
    }
}

// store_tile with a per-column operator applied on the way out:
// g[e][c] = op.comp(d, 0, iy, col0 + c, tile[e][c]) (components d >= 1 of the
// fused x pass, whose factor depends on the plane and column only).
template <int N, int C, int NT, class Op>
__device__ __forceinline__ void store_tile_comp(const float2* __restrict__ tile, float2* __restrict__ g, size_t rs,
                                                int nvalid, const Op& op, int d, int iy, int col0) {
    constexpr int TPR = C / 2;
    constexpr int TOT = N * TPR;
    constexpr int PER = (TOT + NT - 1) / NT;
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * NT;
        if ((TOT % NT) == 0 || i < TOT) {
            const int e = i / TPR, c = 2 * (i % TPR);
            float2* dst = g + (size_t)e * rs + c;
            const float4 v = *reinterpret_cast<const float4*>(&tile[e * C + c]);
            const float2 a = op.comp(d, 0, iy, col0 + c, make_float2(v.x, v.y));
            const float2 b = op.comp(d, 0, iy, col0 + c + 1, make_float2(v.z, v.w));
            if (c + 1 < nvalid) {
                __stcs(reinterpret_cast<float4*>(dst), make_float4(a.x, a.y, b.x, b.y));
            } else if (c < nvalid) {
                dst[0] = a;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// z pass, forward R2C, of the int64 fixed-point density: converted to float
// delta = rho - mean in FP64 and zeroed for the next deposit.
// ---------------------------------------------------------------------------
// The multi-class pass: the lines of group bx of one box.  (The register groups
// of z_rho below lose there, 64 against 58 us a step of the five sides.)
template <int NG, int L>
__device__ __forceinline__ void zpass_rho_body(unsigned long long* __restrict__ in, float2* __restrict__ out, int nlines,
                                               int zs, double mean, const float2* __restrict__ tw, int bx) {
    constexpr int M = NG / 2, ES = L + 1;
    float2* buf = reinterpret_cast<float2*>(hgpm_smem);
    const int line0 = bx * L;
    constexpr int TOT = L * M;
    constexpr int PER = (TOT + kThreads - 1) / kThreads;
    ulonglong2 q[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * kThreads;
        const int l = i / M, m = i % M;
        q[t] = make_ulonglong2(0ull, 0ull);
        if (((TOT % kThreads) == 0 || i < TOT) && line0 + l < nlines)
            q[t] = __ldcs(reinterpret_cast<const ulonglong2*>(in + (size_t)(line0 + l) * NG) + m);
    }
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * kThreads;
        const int l = i / M, m = i % M;
        if (((TOT % kThreads) == 0 || i < TOT)) {
            if (line0 + l < nlines)
                __stcs(reinterpret_cast<ulonglong2*>(in + (size_t)(line0 + l) * NG) + m, make_ulonglong2(0ull, 0ull));
            buf[m * ES + l] = make_float2((float)((double)(long long)q[t].x * kFixInv - mean),
                                          (float)((double)(long long)q[t].y * kFixInv - mean));
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

// ---------------------------------------------------------------------------
// R2C z pass: L contiguous lines of NG reals, as NG/2 complex each, in register
// groups (fft_rows), NT threads.  The first group takes its elements from
// global memory.
// ---------------------------------------------------------------------------
template <int NG, int ELEMS> struct ZTile {
    static constexpr int M = NG / 2;
    static constexpr int L0 = ELEMS / M, L = L0 < 1 ? 1 : L0;
    static constexpr int EPT = NG <= 96 ? 8 : 16;
    static constexpr int NT0 = (M * L / EPT + 31) / 32 * 32, NT = NT0 < L ? (L + 31) / 32 * 32 : NT0;
    static constexpr int MINB = 1024 / NT > 16 ? 16 : 1024 / NT;
    static constexpr int SMEM = L * RowTile<M>::LS * 8;
};

// R2C of lines [line0, line0 + L): ld(line, m) gives cells (2m, 2m + 1).
// Leaves the tile being read.
template <int NG, int L, int NT, class Ld>
__device__ __forceinline__ void z_r2c(float2* __restrict__ tile, float2* __restrict__ out, int line0, int nlines, int zs,
                                      const float2* __restrict__ tw, const Ld& ld) {
    constexpr int M = NG / 2, H = M / 2 + 1;
    using R = RowTile<M>;
    fft_rows_to_tile<M, L, NT, false, 2>(tile, tw, [&](int l, int e) {
        return line0 + l < nlines ? ld(line0 + l, e) : make_float2(0.f, 0.f);
    });
    for (int i = threadIdx.x; i < L * H; i += NT) {
        const int l = i / H, k = i % H;
        const int line = line0 + l;
        if (line >= nlines) continue;
        const float2 zk = tile[R::at(l, k)];
        const float2 zm = tile[R::at(l, k ? M - k : 0)];
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

// R2C of the int64 fixed-point density less the mean (formed in FP64); the
// lines are zeroed for the next deposit.
template <int NG, int L, int NT>
__device__ __forceinline__ void z_rho(float2* __restrict__ tile, unsigned long long* __restrict__ rho,
                                      float2* __restrict__ out, int line0, int nlines, int zs, double mean,
                                      const float2* __restrict__ tw) {
    z_r2c<NG, L, NT>(tile, out, line0, nlines, zs, tw, [&](int line, int m) {
        const ulonglong2 q = __ldcs(reinterpret_cast<const ulonglong2*>(rho + (size_t)line * NG) + m);
        return make_float2((float)((double)(long long)q.x * kFixInv - mean), (float)((double)(long long)q.y * kFixInv - mean));
    });
    // every line has been read (the transform's barriers)
    const int n = (nlines - line0 < L ? nlines - line0 : L) * (NG / 2);
    ulonglong2* q = reinterpret_cast<ulonglong2*>(rho + (size_t)line0 * NG);
    for (int i = threadIdx.x; i < n; i += NT) __stcs(q + i, make_ulonglong2(0ull, 0ull));
}

// ---------------------------------------------------------------------------
// z pass, inverse C2R, ncomp components, unnormalised * scale;
// blockIdx.y = slot * ncomp + component.
// X[0] and X[ng/2] are taken as real (Hermitian extension), which makes the
// result equal to the real part of the reference's full C2C inverse.
// ---------------------------------------------------------------------------
// PAIR: out holds nlines * NG pairs, cell z of a line (phi(z), phi(z+1 mod
// NG)) (the paired potential the pair-gathering kick reads).
// CG: the spectrum is read from L2 (written earlier in the same kernel).
template <int NG, bool PAIR = false, bool CG = false>
__device__ __forceinline__ void zpass_c2r_body(const float2* __restrict__ in, float* __restrict__ out, int nlines,
                                               int zs, float scale, const float2* __restrict__ tw, int bx) {
    constexpr int M = NG / 2, L = Cfg<NG>::L, ES = L + 1;
    float2* buf = reinterpret_cast<float2*>(hgpm_smem);
    const int line0 = bx * L;
    constexpr int H = M / 2 + 1;
    constexpr int TOT = L * H;
    constexpr int PER = (TOT + kThreads - 1) / kThreads;
    // register-staged: every (X[k], X[M-k]) pair of the thread is in flight
    // before the first use
    float2 rk[PER], rm[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * kThreads;
        const int l = i / H, k = i % H;
        rk[t] = make_float2(0.f, 0.f);
        rm[t] = make_float2(0.f, 0.f);
        if (i < TOT && line0 + l < nlines) {
            const float2* src = in + (size_t)(line0 + l) * zs;
            rk[t] = CG ? __ldcg(&src[k]) : __ldcs(&src[k]);
            rm[t] = CG ? __ldcg(&src[M - k]) : __ldcs(&src[M - k]);
        }
    }
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        const int i = threadIdx.x + t * kThreads;
        if (i >= TOT) break;
        const int l = i / H, k = i % H;
        float2 xk = rk[t], xm = rm[t];
        if (k == 0) {
            xk.y = 0.f;
            xm.y = 0.f;
        }
        const float2 w = __ldg(&tw[k]);
        // S = X[k] + conj X[M-k], D = X[k] - conj X[M-k], T = i conj(w) D
        // Z[k] = S + T, Z[M-k] = conj(S - T)
        const float2 s = make_float2(xk.x + xm.x, xk.y - xm.y);
        const float2 d = make_float2(xk.x - xm.x, xk.y + xm.y);
        const float2 cd = cmulc(d, w);                  // conj(w) * d
        const float2 tt = make_float2(-cd.y, cd.x);     // i * conj(w) * d
        buf[k * ES + l] = cadd(s, tt);
        if (k != 0 && k != M - k) {
            const float2 zm = csub(s, tt);
            buf[(M - k) * ES + l] = make_float2(zm.x, -zm.y);
        }
    }
    __syncthreads();
    fft_tile<M, L, ES, true, kThreads, 2>(buf, tw);
    for (int i = threadIdx.x; i < L * M; i += kThreads) {
        const int l = i / M, m = i % M;
        const int line = line0 + l;
        if (line >= nlines) continue;
        const float2 z = buf[m * ES + l];
        if (PAIR) {
            // cells 2m and 2m+1: (phi(2m), phi(2m+1)), (phi(2m+1), phi(2m+2))
            const float nx = buf[(m + 1 == M ? 0 : m + 1) * ES + l].x * scale;
            reinterpret_cast<float4*>(out + (size_t)line * NG * 2)[m] =
                make_float4(z.x * scale, z.y * scale, z.y * scale, nx);
        } else {
            reinterpret_cast<float2*>(out + (size_t)line * NG)[m] = make_float2(z.x * scale, z.y * scale);
        }
    }
}

// ---------------------------------------------------------------------------
// Strided lines (along y or x) in register groups (fft_lines): a tile is C
// neighbouring columns, C a multiple of 8 (rows of 64 bytes or more), of about
// ELEMS elements.
// ---------------------------------------------------------------------------
template <int NG, int ELEMS, int NCOL = NG / 2 + 1> struct LineTile {
    static constexpr int C0 = ELEMS / NG / 8 * 8, C1 = C0 > 32 ? 32 : (C0 < 8 ? 8 : C0);
    static constexpr int C = C1 > NCOL / 8 * 8 ? NCOL / 8 * 8 : C1;
    static constexpr int EPT = NG <= 96 ? 8 : 16;  // elements a thread
    static constexpr int NT0 = (NG * C / EPT + 31) / 32 * 32;
    static constexpr int NT = NT0 > 512 ? 512 : NT0;
    static constexpr int MINB = 1024 / NT > 16 ? 16 : 1024 / NT;
    static constexpr int SMEM = NG * C * 8;
    // a plane's NCOL columns: FULL whole tiles and REM left over, which go
    // into tiles of their own, PPT planes in each (a tile of one plane's
    // Nyquist column alone would leave C - 1 of its lines empty)
    static constexpr int FULL = NCOL / C, REM = NCOL - FULL * C, PPT = REM ? C / REM : 1;
    static constexpr int TILES = FULL * NG + (REM ? (NG + PPT - 1) / PPT : 0);
};

// Line c of tile t of a box of NG planes: its plane, its column; valid.
template <class T, int NG>
struct LineCols {
    int t;
    __device__ __forceinline__ void at(int c, int& plane, int& col, bool& ok) const {
        if (t < T::FULL * NG) {
            plane = t / T::FULL;
            col = t % T::FULL * T::C + c;
            ok = true;
        } else {
            constexpr int R = T::REM ? T::REM : 1;
            plane = (t - T::FULL * NG) * T::PPT + c / R;
            col = T::FULL * T::C + c % R;
            ok = c / R < T::PPT && plane < NG;
        }
    }
};

// ---------------------------------------------------------------------------
// host helpers of the launchers
// ---------------------------------------------------------------------------
template <class K>
static inline cudaError_t ensure_smem(K kernel, int bytes, int threads) {
    return smem_attr_once((const void*)kernel, bytes, threads);
}

static inline unsigned cdiv(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

// ---------------------------------------------------------------------------
// x pass fused with a k-space operator producing 3 components:
//   forward x FFT of the (z,y)-transformed tile -> t = op.pre(k, rho_k) ->
//   out[0] = IFFT_x(op.comp(0, k, t));  T = IFFT_x(t) ->
//   out[1] = op.comp(1, ky, kz, T), out[2] = op.comp(2, ky, kz, T).
// The y and z components' operators (e.g. -i sin(k_y)) are constant along an
// x line, so they commute with the inverse x transform: two inverse FFTs per
// tile instead of three.
// plane = ky index, rows = kx index, columns = kz index; blockIdx.z = slot.
// ---------------------------------------------------------------------------
template <int NG, class Op>
__global__ void __launch_bounds__(Cfg<NG>::NTX) xfused_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                                              int ncols, size_t rs, size_t ps, size_t out_cs,
                                                              const float2* __restrict__ tw, Op op, Slots sl) {
    constexpr int C = Cfg<NG>::CX, NT = Cfg<NG>::NTX;
    float2* tile = reinterpret_cast<float2*>(hgpm_smem);
    float2* work = tile + NG * C;
    if (slot_idle(sl, blockIdx.z)) return;
    in += (size_t)blockIdx.z * sl.s0;
    out += (size_t)blockIdx.z * sl.s1;
    const int col0 = blockIdx.x * C;
    const int iy = blockIdx.y;
    const size_t off = (size_t)iy * ps + col0;
    const int nvalid = ncols - col0;
    load_tile<NG, C, NT>(tile, in + off, rs, nvalid);
    __syncthreads();
    // the three-output IC pass, whose registers are tight, reads every
    // twiddle from the table
    fft_tile<NG, C, C, false, NT, 1, false>(tile, tw);
    for (int i = threadIdx.x; i < NG * C; i += NT) {
        const int ix = i / C, c = i % C;
        tile[i] = op.pre(ix, iy, col0 + c, tile[i]);
    }
    // (fft_tile ended with a barrier; pre() only touches the thread's own cells)
    for (int i = threadIdx.x; i < NG * C; i += NT) {
        const int ix = i / C, c = i % C;
        work[i] = op.comp(0, ix, iy, col0 + c, tile[i]);
    }
    __syncthreads();
    fft_tile<NG, C, C, true, NT, 1, false>(work, tw);
    store_tile<NG, C, NT>(work, out + off, rs, nvalid);
    // (no thread writes tile between the barrier above and this transform)
    fft_tile<NG, C, C, true, NT, 1, false>(tile, tw);
    store_tile_comp<NG, C, NT>(tile, out + out_cs + off, rs, nvalid, op, 1, iy, col0);
    store_tile_comp<NG, C, NT>(tile, out + 2 * out_cs + off, rs, nvalid, op, 2, iy, col0);
}

template <int NG, class Op>
static inline cudaError_t xfused_impl(const float2* in, float2* out, int ncols, size_t rs, size_t ps, int nplanes,
                               size_t out_cs, const float2* tw, const Op& op, cudaStream_t s, const Slots& sl = Slots{},
                               int nslots = 1) {
    using G = Cfg<NG>;
    auto k = xfused_kernel<NG, Op>;
    cudaError_t e = ensure_smem(k, G::XSMEM, G::NTX);
    if (e != cudaSuccess) return e;
    dim3 grid(cdiv(ncols, G::CX), nplanes, nslots);
    k<<<grid, G::NTX, G::XSMEM, s>>>(in, out, ncols, rs, ps, out_cs, tw, op, sl);
    return cudaGetLastError();
}

}  // namespace hgpm
