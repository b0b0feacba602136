// kernels_fft2l.cuh -- the Poisson transforms for lengths with a two-level split (fft_reg.cuh).
//
// Same operations, inputs and outputs as the Stockham kernels of kernels_poisson.cuh (k_fwd_x, k_col_fft, k_inv_x):
// only the transform itself is organised differently.  Step 1 of the z transforms reads its operands straight from
// global memory and their step 2 writes straight to global memory, so a column crosses shared memory once.  The forward x
// transform fills shared memory first, with coalesced loads of the divergence, and forms the modes k and M-k together; the
// inverse one forms the packed half-length spectrum in registers straight from global memory (staged through shared memory
// the same way it took 32 us at 256 x 192 x 256 cells in FP32, and 29 us like this).
#pragma once

#include "fft_reg.cuh"
#include "kernels_poisson.cuh"

namespace dfdm {

template <typename T> struct Vec2;
template <> struct Vec2<float> { typedef float2 type; };
template <> struct Vec2<double> { typedef double2 type; };

// lanes that share a line of Q vectors in the loader: the largest power of two up to 32 that divides Q
template <int Q> struct RowGroup {
    static constexpr int value = Q % 32 == 0 ? 32 : Q % 16 == 0 ? 16 : Q % 8 == 0 ? 8 : Q % 4 == 0 ? 4 : Q % 2 == 0 ? 2 : 1;
};

// ---- div u* (or a real field) + forward real-to-complex x transform, line length Nx = 2M ----------------------
// Phase A forms the packed half-length line z_n = x_2n + i x_2n+1 in shared memory from 16-byte loads (every two-level
// length makes Nx a multiple of 16, so rows and vectors are aligned); the two register steps follow in place.  It is bound
// by the latency of its phases more than by bandwidth: pairs of cells with per-pair indexing and two buffers (fewer lines
// per block) took 62 us at 256 x 192 x 256 cells in FP32 and 145 us in FP64, this form 46 to 49 and 110 us (202 MB in FP32:
// 0.62 to 0.67 of the measured copy bandwidth).
template <typename T, bool FROM_DIV, int M, bool TR = false, class BC>
__device__ __forceinline__ void k_fwd_x2_body(const BC &bc, const PoissonArgs<T> &a, int lx, const T *__restrict__ U, const T *__restrict__ V,
                                                const T *__restrict__ W_, const T *__restrict__ src,
                                                typename cplx_t<T>::type *__restrict__ spec,
                                                const typename cplx_t<T>::type *__restrict__ tw,
                                                const typename cplx_t<T>::type *__restrict__ twr) {
    typedef typename cplx_t<T>::type C;
    constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, Nx = 2 * M;
    constexpr int LD = TR ? RowLayout<M>::LDT : RowLayout<M>::LD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *buf = (C *)smem_raw;
    const Dims &d = a.d;
    const int Ny = d.Ny, Nz = d.Nz, plane = Nx * Ny;
    // blocks run roughly in index order: the first take the highest lines (top z planes), which the stage kernel
    // wrote last and which are the likeliest to still be in L2
    const int line0 = (bc.dim().x - 1 - bc.idx().x) * lx;
    const int nl = min(lx, Ny * Nz - line0);
    // 16-byte vectors of W cells; G lanes (a power of two that divides the line's vector count) share a line, so the
    // line's indices, metrics and row pointers are formed once per lane and line
    constexpr int W = 16 / (int)sizeof(T), Q = Nx / W, G = RowGroup<Q>::value, NQ = Q / G, UNR = NQ % 2 == 0 ? 2 : 1;
    struct alignas(16) Vec { T x[W]; };
    auto put = [](C *p, const Vec &z) {   // lines of the TR form start on 8-byte boundaries only (FP32)
        if constexpr (TR && W == 4) { p[0] = mkc<T>(z.x[0], z.x[1]); p[1] = mkc<T>(z.x[2], z.x[3]); }
        else *reinterpret_cast<Vec *>(p) = z;
    };
    const int lane = threadIdx.x % G;
    for (int ll = threadIdx.x / G; ll < nl; ll += blockDim.x / G) {
        const int line = line0 + ll;
        C *zl = buf + ll * LD + lane * (W / 2);
        if constexpr (FROM_DIV) {
            const int k = (int)fdiv((unsigned)line, a.fNy), j = line - k * Ny;
            const bool vzero = (j == 0) && !d.yper;
            const T riy = a.my.idc[j], riz = a.mz.idc[k];
            const T *Ur = U + (size_t)line * Nx, *Vr = V + (size_t)line * Nx, *Wr = W_ + (size_t)line * Nx;
            const T *Vm = Vr + (vzero ? 0 : (j > 0 ? -Nx : (Ny - 1) * Nx)), *Wm = Wr + (k == 0 ? (Nz - 1) * plane : -plane);
#pragma unroll 1
            for (int c0 = 0; c0 < NQ; c0 += UNR) {
                Vec u[UNR], v[UNR], vm[UNR], w[UNR], wm[UNR];   // all loads of UNR vectors first
                T um[UNR];
#pragma unroll
                for (int q = 0; q < UNR; ++q) {
                    const int i = ((c0 + q) * G + lane) * W;
                    u[q] = *reinterpret_cast<const Vec *>(Ur + i);
                    um[q] = __ldg(Ur + (i == 0 ? Nx - 1 : i - 1));
                    v[q] = *reinterpret_cast<const Vec *>(Vr + i);
                    vm[q] = *reinterpret_cast<const Vec *>(Vm + i);
                    w[q] = *reinterpret_cast<const Vec *>(Wr + i);
                    wm[q] = *reinterpret_cast<const Vec *>(Wm + i);
                }
#pragma unroll
                for (int q = 0; q < UNR; ++q) {
                    Vec z;
#pragma unroll
                    for (int x = 0; x < W; ++x) {
                        const T vb = vzero ? T(0) : vm[q].x[x];
                        z.x[x] = (u[q].x[x] - (x == 0 ? um[q] : u[q].x[x - 1])) * a.inv_dx + (v[q].x[x] - vb) * riy +
                                 (w[q].x[x] - wm[q].x[x]) * riz;
                    }
                    put(zl + (c0 + q) * G * (W / 2), z);
                }
            }
        } else {
            const T *row = src + (size_t)line * Nx + lane * W;
#pragma unroll
            for (int c = 0; c < NQ; ++c) put(zl + c * G * (W / 2), *reinterpret_cast<const Vec *>(row + c * G * W));
        }
    }
    __syncthreads();
    // both steps in place: a thread's items (one of step 1, R2 of step 2; blockDim.x == lx N2) are all in registers before
    // the barrier that precedes their stores
    {
        const int ll = threadIdx.x / N2, n2 = threadIdx.x - ll * N2;
        C v[N1];
        if (ll < nl) {
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) v[n1] = buf[ll * LD + n1 * N2 + n2];
        }
        __syncthreads();
        if (ll < nl) row_step1<T, false, M>(v, buf + ll * LD, n2, tw);
    }
    __syncthreads();
    {
        constexpr int R2 = (N1 + N2 - 1) / N2;
        C v[R2][N2];
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int b = threadIdx.x + r * blockDim.x, ll = b / N1, k1 = b - ll * N1;
            if (ll < nl) {
#pragma unroll
                for (int n2 = 0; n2 < N2; ++n2) v[r][n2] = buf[ll * LD + k1 * (N2 + 1) + n2];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int b = threadIdx.x + r * blockDim.x, ll = b / N1, k1 = b - ll * N1;
            if (ll < nl) {
                Codelet<T, false, N2>::run(v[r]);
#pragma unroll
                for (int k2 = 0; k2 < N2; ++k2) buf[ll * LD + k1 + N1 * k2] = v[r][k2];
            }
        }
    }
    __syncthreads();
    const int Nxc = d.Nxc;
    // modes k and M-k together: with E, O as k_fwd_x forms them, X_k = E + W^k O and X_{M-k} = conj(E - W^k O).  Consecutive
    // threads take consecutive modes of a line, or (TR) one mode of consecutive lines: the spectrum's contiguous index
    constexpr int H = M / 2 + 1;
    const size_t nlines = (size_t)Ny * Nz;
    for (int e = threadIdx.x; e < (TR ? lx : nl) * H; e += blockDim.x) {
        const int ll = TR ? e & (lx - 1) : e / H, k = TR ? e / lx : e - ll * H;   // lx is a power of two
        if (TR && ll >= nl) continue;
        const C *res = buf + ll * LD;
        const C Zk = res[k], Zm = res[k == 0 ? 0 : M - k];
        const T Er = T(0.5) * (Zk.x + Zm.x), Ei = T(0.5) * (Zk.y - Zm.y);
        const T Dr = T(0.5) * (Zk.x - Zm.x), Di = T(0.5) * (Zk.y + Zm.y);
        const T Or = Di, Oi = -Dr;
        const C w = __ldg(twr + k);
        const T Pr = w.x * Or - w.y * Oi, Pi = w.x * Oi + w.y * Or;
        C *row = TR ? spec + line0 + ll : spec + (size_t)(line0 + ll) * Nxc;
        const size_t ks = TR ? nlines : 1;
        row[k * ks] = mkc<T>(Er + Pr, Ei + Pi);
        if (2 * k != M) row[(M - k) * ks] = mkc<T>(Er - Pr, Pi - Ei);
    }
}
template <typename T, bool FROM_DIV, int M, bool TR>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) k_fwd_x2(PoissonArgs<T> a, int lx, const T *__restrict__ U, const T *__restrict__ V,
                                                const T *__restrict__ W, const T *__restrict__ src,
                                                typename cplx_t<T>::type *__restrict__ spec,
                                                const typename cplx_t<T>::type *__restrict__ tw,
                                                const typename cplx_t<T>::type *__restrict__ twr) {
    pdl_enter();
    k_fwd_x2_body<T, FROM_DIV, M, TR>(HwBlock(), a, lx, U, V, W, src, spec, tw, twr);
}

// ---- inverse complex-to-real x transform, writes phi = x / (nxp*nzp) -----------------------------------------
template <typename T, int M, bool TR = false, class BC>
__device__ __forceinline__ void k_inv_x2_body(const BC &bc, const PoissonArgs<T> &a, int lx, const typename cplx_t<T>::type *__restrict__ spec,
                                                T *__restrict__ phi, const typename cplx_t<T>::type *__restrict__ tw,
                                                const typename cplx_t<T>::type *__restrict__ twr) {
    typedef typename cplx_t<T>::type C;
    typedef typename Vec2<T>::type T2;
    constexpr int N1 = Split<M>::N1, N2 = Split<M>::N2, Nx = 2 * M;
    constexpr int LD = TR ? RowLayout<M>::LDT : RowLayout<M>::LD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bt = (C *)smem_raw;
    const Dims &d = a.d;
    const int Nxc = d.Nxc;
    const int line0 = bc.idx().x * lx;
    const int nl = min(lx, d.Ny * d.Nz - line0);
    const size_t ks = TR ? (size_t)d.Ny * d.Nz : 1;   // between modes; TR: consecutive threads on consecutive lines
    for (int b = threadIdx.x; b < (TR ? lx : nl) * N2; b += blockDim.x) {
        const int ll = TR ? b & (lx - 1) : b / N2, n2 = TR ? b / lx : b - ll * N2;   // lx is a power of two
        if (TR && ll >= nl) continue;
        const C *row = TR ? spec + line0 + ll : spec + (size_t)(line0 + ll) * Nxc;
        C v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) {
            const int kx = n1 * N2 + n2;
            C X = row[kx * ks], Xm = row[(M - kx) * ks];
            if (kx == 0) { X.y = T(0); Xm.y = T(0); }
            T E2r = X.x + Xm.x, E2i = X.y - Xm.y;
            T D2r = X.x - Xm.x, D2i = X.y + Xm.y;
            C w = __ldg(twr + kx);
            T O2r = D2r * w.x + D2i * w.y, O2i = D2i * w.x - D2r * w.y;
            v[n1].x = E2r - O2i;
            v[n1].y = E2i + O2r;
        }
        row_step1<T, true, M>(v, bt + ll * LD, n2, tw);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nl * N1; b += blockDim.x) {
        const int ll = b / N1, k1 = b - ll * N1;
        C v[N2];
        const C *tl = bt + ll * LD + k1 * (N2 + 1);
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) v[n2] = tl[n2];
        Codelet<T, true, N2>::run(v);
        T2 *out = reinterpret_cast<T2 *>(phi + (size_t)(line0 + ll) * Nx);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            T2 o;
            if (sizeof(T) == 8) {
                o.x = (T)div_by((double)v[k2].x, a.norm, a.rnorm);
                o.y = (T)div_by((double)v[k2].y, a.norm, a.rnorm);
            } else {
                o.x = v[k2].x * (T)a.rnorm;
                o.y = v[k2].y * (T)a.rnorm;
            }
            out[k1 + N1 * k2] = o;
        }
    }
}
template <typename T, int M, bool TR>
__global__ void __launch_bounds__(256) k_inv_x2(PoissonArgs<T> a, int lx, const typename cplx_t<T>::type *__restrict__ spec,
                                                T *__restrict__ phi, const typename cplx_t<T>::type *__restrict__ tw,
                                                const typename cplx_t<T>::type *__restrict__ twr) {
    pdl_enter();
    k_inv_x2_body<T, M, TR>(HwBlock(), a, lx, spec, phi, tw, twr);
}

// ---- z transforms (MODE 0 forward, 1 inverse) and the periodic-y solve (MODE 2) on tiles of NL columns ----
// Columns are consecutive in the flattened (j, kx) index (MODE 2: (kz, kx)), as in k_col_fft: no idle columns but in the
// last block, and 128-byte tile rows that start on 128-byte boundaries where Ny (Nx/2 + 1) is a multiple of 16.  Against
// one block per (kx tile, j), a step went from 260 to 245 us at 128 x 96 x 128 cells and from 1237 to 1206 us at
// 256 x 192 x 256 (FP32).
// MODE 2: forward FFT along y, division by kxx+kyy+kzz with the (0,0,0) mode set to zero, inverse FFT, division
// by nyp (src/projection.f90:246-273).
template <typename T, int MODE, int NL, int L>
__global__ void __launch_bounds__(256) k_col2(Dims d, typename cplx_t<T>::type *__restrict__ spec,
                                              const typename cplx_t<T>::type *__restrict__ tw,
                                              const double *__restrict__ kxx, const double *__restrict__ kyy,
                                              const double *__restrict__ kzz) {
    pdl_enter();
#define DFDM_BLOCK_IDX blockIdx
#include "k_col2_body.inc"
#undef DFDM_BLOCK_IDX
}

}  // namespace dfdm
