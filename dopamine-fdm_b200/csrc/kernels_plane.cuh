// kernels_plane.cuh -- the spectral part of a wall-bounded pressure solve between the x transforms, one kx plane per pair
// of blocks.
//
// For every kx the forward z transform, the tridiagonal y solves and the inverse z transform touch only that kx's Ny x Nz
// plane.  Where half a plane and its pivots fit in a block's shared memory this kernel does all three in one launch: a
// cluster of two blocks reads the plane once, each block its half of the y rows, keeps it in shared memory through the
// passes and writes it once, in place of three launches that each read and write the whole spectrum (k_col2 / k_ysolve3 /
// k_col2).  It is bound by the latency of its passes (at 128 x 96 x 128 cells in FP32 6.4 MB of spectrum in and out and 6.4 MB
// of pivots in 16.6 us, the blocks issuing in 31 % of their SMs' active cycles), so it pays where the three launches are
// latency-bound too (plane_wins in dfdm_api.cu has the rule and the timings).  One block per plane sweeping top to bottom took
// 21.6 us there against 32 for the three launches; the pair of blocks brought the step from 197 to 182 us more.
//
// Layout.  The spectrum of a context that runs this kernel is plane-major, spec[kx][line] with line = k*Ny + j, so a plane is
// contiguous; the x transforms read and write it that way (their TR form).  In shared memory row `slot` holds one kz (or
// one z before the transform) at slot*RS, RS odd: the z passes run with lanes along j, the sweeps with lanes along the
// rows, and both are free of bank conflicts.
//
// Transforms in place.  With L = N1 N2, step 1 of a two-level transform (fft_reg.cuh) for one n2 reads the elements n1*N2+n2
// and its outputs take the same slots, k1*N2+n2; step 2 for one k1 reads k1*N2+n2 and its outputs take the same slots,
// k1*N2+k2, which hold kz = k1+N1*k2.  The solve does not care about the order, and the inverse runs the two steps backwards
// (over k2, the twiddle, over k1) from the same slots into natural order.  No pass moves an element another thread holds, so
// one buffer and one barrier per pass suffice.
//
// The y solve.  (Dyy + kxx + kzz) x = b by elimination from both ends (the twisted factorisation: D from the top as
// k_ysolve2, E from the bottom), so that each block sweeps its own rows and the two meet once, at the row M that the first
// block ends with:
//   b'(r) = b(r) - lo(r) b'(r-1)/D(r-1) down to M-1,   c'(r) = b(r) - up(r) c'(r+1)/E(r+1) up to M+1,
//   x(M) = (b(M) - lo(M) b'(M-1)/D(M-1) - up(M) c'(M+1)/E(M+1)) / F,
//   x(r) = (b'(r) - up(r) x(r+1))/D(r) above M,        x(r) = (c'(r) - lo(r) x(r-1))/E(r) below.
// The table holds 1/D, 1/F and 1/E by row.  The operator is similar to a symmetric negative-definite matrix (k_ysolve2), so
// elimination from either end is stable.  The two blocks exchange one double per system through distributed shared memory.
#pragma once

#include "fft_reg.cuh"
#include "kernels_poisson.cuh"

namespace dfdm {

constexpr int PLANE_THREADS = 512;   // most threads of a block
__host__ __device__ constexpr int plane_rows(int ny) { return (ny + 1) / 2; }   // y rows of the first block; M is its last
__host__ __device__ constexpr int plane_rs(int ny) { return plane_rows(ny) | 1; }
// shared memory of a block: half the plane, its pivots, the operator's off-diagonals, the exchanged doubles
template <typename T> __host__ __device__ constexpr size_t plane_smem(int ny, int nz) {
    return (size_t)plane_rows(ny) * nz * sizeof(double) + (size_t)2 * plane_rows(ny) * sizeof(double) +
           (size_t)2 * nz * sizeof(double) + (size_t)plane_rs(ny) * nz * 2 * sizeof(T);
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();   // the aligned forms want whole warps
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// a double into the same shared-memory location of block `rank` of the cluster
__device__ __forceinline__ void cluster_store(double *p, unsigned rank, double v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(ra), "d"(v) : "memory");
}

// The pivot tables of every (kx, kz) system, set up once per context: rpiv (unless null) in the layout (kz, row, kx) of
// k_ysolve2, 1/D of the elimination from the top; rpivp (unless null) as above.  One thread per system, the operations
// rounded one by one.  The (0,0) system's first diagonal entry is scaled by 3/2 (src/projection.f90:284-295); *bad is set
// where a pivot vanishes.  A host loop over both tables took 25 ms at 128 x 96 x 128 cells.
__global__ void __launch_bounds__(128) k_pivots(Dims d, int n1, int n2, const double *__restrict__ kxx,
                                                const double *__restrict__ kzz, const double *__restrict__ lo,
                                                const double *__restrict__ di, const double *__restrict__ up,
                                                double *__restrict__ rpiv, double *__restrict__ rpivp, int *__restrict__ bad) {
    pdl_enter();
    const int kx = blockIdx.x * blockDim.x + threadIdx.x, kz = blockIdx.y;
    if (kx >= d.Nxc) return;
    const double lam = __dadd_rn(kxx[kx], kzz[kz]);
    const int M = plane_rows(d.Ny) - 1;
    double *o = rpiv ? rpiv + (size_t)kz * d.Ny * d.Nxc + kx : nullptr;
    double *op = rpivp ? rpivp + (size_t)kx * d.Ny * d.Nz + (kz % n1) * n2 + kz / n1 : nullptr;
    double D = __dadd_rn(di[0], lam), DM = 0.0;   // DM: the pivot of row M - 1
    if (kx == 0 && kz == 0) D = __dmul_rn(1.5, D);
    bool zero = D == 0.0;
    for (int r = 0; r < d.Ny; ++r) {
        if (r > 0) {
            D = __dsub_rn(__dadd_rn(di[r], lam), __dmul_rn(__ddiv_rn(lo[r], D), up[r - 1]));
            zero = zero || D == 0.0;
        }
        const double inv = __drcp_rn(D);
        if (o) o[(size_t)r * d.Nxc] = inv;
        if (op && r < M) op[(size_t)r * d.Nz] = inv;
        if (r == M - 1) DM = D;
        if (!o && r == M - 1) break;
    }
    if (op) {
        double E = __dadd_rn(di[d.Ny - 1], lam);
        for (int r = d.Ny - 1; r > M; --r) {
            if (r < d.Ny - 1) E = __dsub_rn(__dadd_rn(di[r], lam), __dmul_rn(__ddiv_rn(up[r], E), lo[r + 1]));
            zero = zero || E == 0.0;
            op[(size_t)r * d.Nz] = __drcp_rn(E);
        }
        const double F = __dsub_rn(__dsub_rn(__dadd_rn(di[M], lam), __dmul_rn(__ddiv_rn(lo[M], DM), up[M - 1])),
                                   __dmul_rn(__ddiv_rn(up[M], E), lo[M + 1]));
        zero = zero || F == 0.0;
        op[(size_t)M * d.Nz] = __drcp_rn(F);
    }
    if (zero) *bad = 1;
}

// lo, up: the operator's off-diagonals by y row.  blockDim.x >= 2 L (two sweep threads per system).
template <typename T, int L>
__global__ void __launch_bounds__(PLANE_THREADS) __cluster_dims__(2, 1, 1)
    k_plane(Dims d, typename cplx_t<T>::type *__restrict__ spec, const typename cplx_t<T>::type *__restrict__ twz,
            const double *__restrict__ rpiv, const double *__restrict__ lo, const double *__restrict__ up) {
    pdl_enter();
    cluster_arrive();   // waited for before the exchange: the other block has started by then
    typedef typename cplx_t<T>::type C;
    constexpr int N1 = Split<L>::N1, N2 = Split<L>::N2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int rows = plane_rows(d.Ny), RS = plane_rs(d.Ny), nt = blockDim.x;
    const int rank = (int)cluster_rank(), kx = blockIdx.x >> 1, j0 = rank ? rows : 0, ny = rank ? d.Ny - rows : rows;
    double *piv = reinterpret_cast<double *>(smem_raw);   // [row][slot]
    double *hand = piv + (size_t)rows * L;                // [2 slot + part]: from the other block
    double *sco = hand + 2 * L;                           // lo at [0, rows), up at [rows, 2 rows)
    C *s = reinterpret_cast<C *>(sco + 2 * rows);
    C *g = spec + (size_t)kx * d.Ny * L + j0;
    const double *rp = rpiv + ((size_t)kx * d.Ny + j0) * L;
    // the pivots travel while the transform runs (16-byte copies: L is even)
    for (int e = threadIdx.x; e < ny * L / 2; e += nt) cp_async16(piv + 2 * e, rp + 2 * e);
    cp_async_commit();
    for (int r = threadIdx.x; r < ny; r += nt) { sco[r] = lo[j0 + r]; sco[rows + r] = up[j0 + r]; }
    // ---- forward z: step 1 from global memory, step 2 in place ----
    for (int b = threadIdx.x; b < ny * N2; b += nt) {
        const int n2 = b / ny, j = b - n2 * ny;
        C v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) v[n1] = g[(n1 * N2 + n2) * d.Ny + j];
        Codelet<T, false, N1>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) s[(k1 * N2 + n2) * RS + j] = k1 == 0 ? v[0] : cmul(v[k1], __ldg(twz + n2 * k1));
    }
    __syncthreads();
    for (int b = threadIdx.x; b < ny * N1; b += nt) {
        const int k1 = b / ny, j = b - k1 * ny;
        C v[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) v[n2] = s[(k1 * N2 + n2) * RS + j];
        Codelet<T, false, N2>::run(v);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) s[(k1 * N2 + k2) * RS + j] = v[k2];
    }
    cp_async_wait_all();
    __syncthreads();
    // ---- one tridiagonal system per kz, its real and imaginary parts in two threads ----
    const bool sweeps = threadIdx.x < 2 * L;
    const int slot = threadIdx.x >> 1;
    T *x = reinterpret_cast<T *>(s + slot * RS) + (threadIdx.x & 1);
    const double *pv = piv + slot, *slo = sco, *sup = sco + rows;
    double mine = 0.0, rF = 0.0, upM = 0.0;
    if (sweeps) {
        if (rank == 0) {
            const int M = rows - 1;
            double b = (double)x[0], rprev = pv[0];
#pragma unroll 8
            for (int r = 1; r < M; ++r) {
                const double m = slo[r] * rprev;
                b = (double)x[2 * r] - m * b;
                x[2 * r] = (T)b;
                rprev = pv[r * L];
            }
            rF = pv[M * L];
            upM = sup[M];
            mine = (double)x[2 * M] - (slo[M] * rprev) * b;
        } else {
            const int last = ny - 1;
            double c = (double)x[2 * last], rprev = pv[last * L];
            rF = __ldg(rp - L + slot);
            upM = __ldg(up + rows - 1);
#pragma unroll 8
            for (int r = last - 1; r >= 0; --r) {
                const double m = sup[r] * rprev;
                c = (double)x[2 * r] - m * c;
                x[2 * r] = (T)c;
                rprev = pv[r * L];
            }
            mine = c * rprev;
        }
    }
    cluster_wait();
    if (sweeps) cluster_store(hand + threadIdx.x, rank ^ 1, mine);
    cluster_arrive();
    cluster_wait();
    if (sweeps) {
        const double other = hand[threadIdx.x];
        double y = (rank == 0 ? mine - upM * other : other - upM * mine) * rF;   // x(M)
        if (rank == 0) {
            const int M = rows - 1;
            x[2 * M] = (T)y;
#pragma unroll 8
            for (int r = M - 1; r >= 0; --r) {
                const double p = pv[r * L];
                y = (double)x[2 * r] * p - (sup[r] * p) * y;
                x[2 * r] = (T)y;
            }
        } else {
#pragma unroll 8
            for (int r = 0; r < ny; ++r) {
                const double p = pv[r * L];
                y = (double)x[2 * r] * p - (slo[r] * p) * y;
                x[2 * r] = (T)y;
            }
        }
    }
    __syncthreads();
    // ---- inverse z: over k2 in place, over k1 to global memory ----
    for (int b = threadIdx.x; b < ny * N1; b += nt) {
        const int k1 = b / ny, j = b - k1 * ny;
        C v[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) v[k2] = s[(k1 * N2 + k2) * RS + j];
        Codelet<T, true, N2>::run(v);
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2)
            s[(k1 * N2 + n2) * RS + j] = k1 == 0 || n2 == 0 ? v[n2] : cmulc(v[n2], __ldg(twz + n2 * k1));
    }
    __syncthreads();
    for (int b = threadIdx.x; b < ny * N2; b += nt) {
        const int n2 = b / ny, j = b - n2 * ny;
        C v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) v[k1] = s[(k1 * N2 + n2) * RS + j];
        Codelet<T, true, N1>::run(v);
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) g[(n1 * N2 + n2) * d.Ny + j] = v[n1];
    }
}

}  // namespace dfdm
