// kernels_step.cuh -- eddy viscosity, wall model and the fused RHS + RK3 stage kernel.
#pragma once

#include "dfdm_common.cuh"
#include "f32x2.cuh"

namespace dfdm {

// Elementwise arithmetic of the right-hand sides for double, float and packed pairs: one fused multiply-add where the
// formulas below say mad / nmad.
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ F2 mad(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
template <typename T> __device__ __forceinline__ T nmad(T a, T b, T c) { return mad(-a, b, c); }   // c - a b
__device__ __forceinline__ double mulv(double a, double b) { return a * b; }
__device__ __forceinline__ float mulv(float a, float b) { return a * b; }
__device__ __forceinline__ F2 mulv(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }

// The constants of the right-hand sides.  FP32 keeps each twice, so that a packed kernel reads a pair with one load.
template <typename D> struct RhsConst {
    D inv_dx, cx, nu, nu2, n2x, two_inv_dx2, dPdx, dPdz;   // 1/dx, -1/(2 dx), nu, 2 nu, 2 nu/dx^2, 2/dx^2
    D wd, p, q, hwd, hp, hq;                   // the blend outside the wall band: wd = 1 - wa, p = 1 - wa/2, q = wa/2, halves
    D half, m2;                                // 0.5, -2
};
template <typename T> struct RhsDup;
template <> struct RhsDup<double> { typedef double type; };
template <> struct RhsDup<float> { typedef float2 type; };
template <typename T> __device__ __forceinline__ T bcast(double x) { return T(x); }
template <typename T> __device__ __forceinline__ T bcast(float2 x);
template <> __device__ __forceinline__ float bcast<float>(float2 x) { return x.x; }
template <> __device__ __forceinline__ F2 bcast<F2>(float2 x) { return F2(x); }

// Base-profile terms of one row (FP32; the profile is zero in FP64), from ub of rows j-1, j, j+1 (mirrored on wall ghost
// rows).  f: the profile at the y face j; df: its step from face j-1, f - fm with w0 + w1 = 1, formed from the steps dp and dm
// across the two faces; x: (1 + wd) ub; c: its diffusion's flux difference.
template <typename T> struct RowProfile {
    T u, f, df, x, c, dp, dm;
    template <typename Y> __device__ __forceinline__ void load(const T *ubr, const Y &y, T wd) {
        u = ubr[1];
        f = mad(y.w1(), ubr[2], mulv(y.w0(), ubr[1]));
        x = mad(wd, ubr[1], ubr[1]);
        dp = ubr[2] - ubr[1];
        dm = ubr[1] - ubr[0];
        df = mad(y.w0m(), dm, mulv(y.w1(), dp));
        c = nmad(y.invfm(), dm, mulv(y.invf(), dp));
    }
};
template <> struct RowProfile<double> {
    template <typename Y> __device__ __forceinline__ void load(const double *, const Y &, double) {}
};

// Everything a step kernel reads besides the fields.  Metric arrays are offset so index -1 is valid.
template <typename T> struct StepArgs {
    Dims d;
    Metric1D<T> my, mz;          // y and z metrics in the storage type
    T inv_dx, dx2;
    int nwl;                     // divergence-form wall band (adv_wall_layers)
    int wm;                      // flat-wall EQWM on both no-slip walls
    int sgs_model;               // 1 Vreman, 2 AMD
    T C_amd, c_V;
    double nu_d, Ly, yg2, ygtop; // wall distances of the first centres: yg(2), Ly - yg(nyg-1)
    // Streamwise base profile: U is stored as U - ub(j) (FP32-mixed; all zeros in FP64).  ub is exactly
    // representable in the storage type; ubd is the same profile in double.
    const T *ub;
    const double *ubd;
    // advection_scheme = 2: the dissipative terms of k_adv_hybrid_faces (u, v, w blocks of `cells`), added to the
    // right-hand sides; null otherwise
    const T *adv;
    // fused correction of the previous stage (CORR kernels): its potential phi; the plane loads then hold u* and
    // the loader forms u = u* - grad(phi) exactly as k_correct does
    const T *phi;
    RhsConst<typename RhsDup<T>::type> rc;
    // FP32: the eight z metrics of every plane in AxisLocal<F2>::load_pairs order, each twice: ZPAIRS consecutive values
    // per plane (copied to shared memory with the plane); null in FP64
    const float *zm8;
    // FP64: the same eight values per z plane and per y row, once each; null in FP32
    const double *zmd, *ymd;
    // LES with the wall model: the first-cell gradient factor of every wall cell, (iw*Nz + k)*Nx + i, written by
    // k_wall_sgs from the velocity the eddy viscosity is computed from (NaN where the override does not apply);
    // null: nut_at solves for it in place
    const double *wfac;
};

// ---------------------------------------------------------------------------------------------------------------
// Reichardt law and the Newton solve for u_tau (src/wallmodel.f90:29-74), always in double.
__device__ __forceinline__ void reichardt_uplus(double yplus, double &uplus, double &duplus) {
    const double kappa = 0.41, A1 = 11.0, A2 = 0.33;
    const double c_buf = 5.2 - log(kappa) / kappa;
    const double a1i = 1.0 / A1, rkappa = 1.0 / kappa;
    double e1 = exp(-yplus * a1i);
    double e2 = exp(-A2 * yplus);
    uplus = div_by(log(1.0 + kappa * yplus), kappa, rkappa) + c_buf * (1.0 - e1 - yplus * a1i * e2);
    duplus = 1.0 / (1.0 + kappa * yplus) + c_buf * (a1i * e1 - a1i * e2 + yplus * a1i * A2 * e2);
}
__device__ __forceinline__ double solve_u_tau(double u_ref, double y_ref, double nu_l) {
    const double rnu = 1.0 / nu_l;
    double u_tau = fmax(1e-3 * u_ref, sqrt(nu_l * u_ref / fmax(y_ref, 1e-14)));
    for (int iter = 1; iter <= 20; ++iter) {   // n_iter_wm = 20, bounded
        double yplus = div_by(u_tau * y_ref, nu_l, rnu), uplus, duplus;
        reichardt_uplus(yplus, uplus, duplus);
        double f = u_ref / fmax(u_tau, 1e-20) - uplus;
        double fp = -u_ref / fmax(u_tau * u_tau, 1e-20) - div_by(duplus * y_ref, nu_l, rnu);
        double u_tau_new = u_tau - f / (fp + copysign(1e-14, fp));
        u_tau_new = fmin(fmax(u_tau_new, 0.1 * u_tau), 10.0 * u_tau);
        if (fabs(u_tau_new - u_tau) < 1e-6 * u_tau_new) { u_tau = u_tau_new; break; }
        u_tau = u_tau_new;
    }
    return u_tau;
}

// The wall-modelled first-cell gradient override of compute_vreman (src/sgs_model.f90:158-172): the factor
// u_tau/(kappa y_w |u|) (signed by the wall) that replaces du/dy and dw/dy by fac*u_c and fac*w_c, with u_tau from the
// Reichardt law at the first-cell velocity magnitude; NaN where |u| <= 1e-14 and the gradients are kept.
__device__ __forceinline__ double wall_gradient_factor(double u_c, double w_c, bool lower, double y_w, double nu) {
    double u_mag = sqrt(u_c * u_c + w_c * w_c);
    if (!(u_mag > 1e-14)) return __longlong_as_double(0x7ff8000000000000LL);
    double u_tau = solve_u_tau(u_mag, y_w, nu);
    return (lower ? 1.0 : -1.0) * u_tau / (0.41 * y_w * u_mag);
}

// ---------------------------------------------------------------------------------------------------------------
// Eddy viscosity at one cell centre: compute_vreman pass 1 (src/sgs_model.f90:118-223) with the AMD
// (Rozema et al. 2015) or Vreman (2004) closure and the wall-modelled first-cell gradient override (:158-172).
// Ghost values come from the neighbourhood accessor (sgs_fill_ghosts' rules, :458-531).
template <typename T, typename Q>
__device__ __forceinline__ T nut_at(const StepArgs<T> &a, const Q &q, int i, int j, int k) {
    const Dims &d = a.d;
    const Metric1D<T> &my = a.my, &mz = a.mz;
    T dz_c = mz.dc[k], dz2 = dz_c * dz_c;
    T inv_dz_k = mz.idc[k], inv_zg_km = mz.idf[k - 1], inv_zg_kp = mz.idf[k];
    T dy_c = my.dc[j], dy2_c = dy_c * dy_c;
    T inv_yg_jm = my.idf[j - 1], inv_yg_jp = my.idf[j], inv_dy_j = my.idc[j];
    T inv_dx = a.inv_dx, dx2 = a.dx2;
    T Uc = q.U(0, 0, 0), Um = q.U(-1, 0, 0);
    T a11 = (Uc - Um) * inv_dx;
    T a21 = T(0.5) * ((Uc - q.U(0, -1, 0)) * inv_yg_jm + (q.U(0, 1, 0) - Uc) * inv_yg_jp);
    T a31 = T(0.5) * ((Uc - q.U(0, 0, -1)) * inv_zg_km + (q.U(0, 0, 1) - Uc) * inv_zg_kp);
    T Vc = q.V(0, 0, 0);
    T a12 = T(0.5) * ((Vc - q.V(-1, 0, 0)) + (q.V(1, 0, 0) - Vc)) * inv_dx;
    T a22 = (Vc - q.V(0, -1, 0)) * inv_dy_j;
    T a32 = T(0.5) * ((Vc - q.V(0, 0, -1)) * inv_zg_km + (q.V(0, 0, 1) - Vc) * inv_zg_kp);
    T Wc = q.W(0, 0, 0), Wkm = q.W(0, 0, -1);
    T a13 = T(0.5) * ((Wc - q.W(-1, 0, 0)) + (q.W(1, 0, 0) - Wc)) * inv_dx;
    T a23 = T(0.5) * ((Wc - q.W(0, -1, 0)) * inv_yg_jm + (q.W(0, 1, 0) - Wc) * inv_yg_jp);
    T a33 = (Wc - Wkm) * inv_dz_k;
    if (a.wm && (j == 0 || j == d.Ny - 1)) {
        double u_c = 0.5 * ((double)Um + (double)Uc);
        double w_c = 0.5 * ((double)Wkm + (double)Wc);
        double fac_w;
        if (a.wfac) {
            fac_w = a.wfac[((j == 0 ? 0 : d.Nz) + k) * d.Nx + i];   // NaN: no override
        } else {
            fac_w = wall_gradient_factor(u_c, w_c, j == 0, (j == 0) ? a.yg2 : a.ygtop, a.nu_d);
        }
        if (!isnan(fac_w)) {
            a21 = (T)(fac_w * u_c);
            a23 = (T)(fac_w * w_c);
        }
    }
    T b11 = dx2 * (a11 * a11) + dy2_c * (a21 * a21) + dz2 * (a31 * a31);
    T b22 = dx2 * (a12 * a12) + dy2_c * (a22 * a22) + dz2 * (a32 * a32);
    T b33 = dx2 * (a13 * a13) + dy2_c * (a23 * a23) + dz2 * (a33 * a33);
    T b12 = dx2 * (a11 * a12) + dy2_c * (a21 * a22) + dz2 * (a31 * a32);
    T b13 = dx2 * (a11 * a13) + dy2_c * (a21 * a23) + dz2 * (a31 * a33);
    T b23 = dx2 * (a12 * a13) + dy2_c * (a22 * a23) + dz2 * (a32 * a33);
    T alpha_sq = a11 * a11 + a12 * a12 + a13 * a13 + a21 * a21 + a22 * a22 + a23 * a23 + a31 * a31 + a32 * a32 + a33 * a33;
    T nu_t = T(0);
    if (a.sgs_model == 2) {
        T amd_num = -(b11 * a11 + b22 * a22 + b33 * a33 + b12 * (a12 + a21) + b13 * (a13 + a31) + b23 * (a23 + a32));
        if (alpha_sq > T(1e-20) && amd_num > T(1e-12) * (dx2 + dy2_c + dz2) * alpha_sq * sqrt(alpha_sq))
            nu_t = a.C_amd * amd_num / alpha_sq;
    } else {
        T B_beta = b11 * b22 - b12 * b12 + b11 * b33 - b13 * b13 + b22 * b33 - b23 * b23;
        if (alpha_sq > T(1e-20) && B_beta > T(0)) nu_t = a.c_V * sqrt(B_beta / alpha_sq);
    }
    return nu_t;
}

// ---------------------------------------------------------------------------------------------------------------
// Flat-wall EQWM state, one plane per wall (iw = 0 bottom, 1 top), index (iw*Nz + k)*Nx + i.
struct WallState {
    double *tau_x, *tau_z;                       // wall shear at U faces / W faces
    double *ux, *wx, *tx, *uz, *wz, *tz;         // filtered velocity and u_tau (wmf_* of src/global.f90:343)
};

// update_wm_filter (src/wallmodel.f90:397-439; filter != 0, seeding it with seed != 0) and compute_flat_wall_eqwm
// (:442-583), smooth Reichardt law, matching height = first centre.  One thread per wall face of one set: blockIdx.z is
// 2 iw + set, wall iw 0 lower or 1 upper, set 0 the U faces or 1 the W faces, so that every face's Newton solve (a serial
// chain of FP64 logarithms, exponentials and divisions) runs in a thread of its own.  With one thread per (i, k) taking all
// four solves in turn, behind a separate filter kernel, the two launches took 23 us at 96 x 96 columns; this one takes
// 8 us.
constexpr int WALL_THREADS = 64;
template <typename T>
__global__ void __launch_bounds__(WALL_THREADS) k_wall_model(StepArgs<T> a, WallState ws, const T *__restrict__ U,
                                                             const T *__restrict__ W, int filter, int seed, double dt_fixed,
                                                             const double *__restrict__ dtp, double Tf_fac) {
    pdl_enter();
    const Dims &d = a.d;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y, iw = blockIdx.z >> 1;
    const bool wface = blockIdx.z & 1;
    if (i >= d.Nx) return;
    const int im = wrap(i - 1, d.Nx), km = wrap(k - 1, d.Nz), jw = iw ? d.Ny - 1 : 0;
    const double y_match = fmax(iw ? a.ygtop : a.yg2, 1e-14), ubw = a.ubd[jw];
    const long long p = ((long long)iw * d.Nz + k) * d.Nx + i;
    // the velocity at the face
    double u = (double)U[idx3(d, i, jw, k)] + ubw, w = (double)W[idx3(d, i, jw, k)];
    if (wface) u = 0.5 * (((double)U[idx3(d, im, jw, k)] + ubw) + u);
    else w = 0.5 * ((double)W[idx3(d, i, jw, km)] + w);
    double *ut = wface ? ws.tz : ws.tx;
    if (filter) {
        double *uf = wface ? ws.uz : ws.ux, *wf = wface ? ws.wz : ws.wx;
        const double dt = dtp ? *dtp : dt_fixed;   // adaptive time step: from device memory
        double eps = 1.0;
        if (!seed && ut[p] > 0.0) eps = fmin(1.0, dt * 0.41 * ut[p] / (Tf_fac * y_match));
        u = (1.0 - eps) * uf[p] + eps * u;
        w = (1.0 - eps) * wf[p] + eps * w;
        uf[p] = u;
        wf[p] = w;
    }
    const double u_ref = sqrt(u * u + w * w);
    const double u_tau = solve_u_tau(u_ref, y_match, a.nu_d);
    ut[p] = u_tau;
    const double tv = u_tau * u_tau * (wface ? w : u) / fmax(u_ref, 1e-30);
    (wface ? ws.tau_z : ws.tau_x)[p] = iw ? -tv : tv;
}

// ---------------------------------------------------------------------------------------------------------------
// Metric values around one index p of an axis: weights of faces p-1 and p, widths and spacings at p-1, p, p+1.
// FP32 reads them once per thread (y) or once per plane (z) and keeps them in registers; FP64 reads them where
// they are used (its registers are taken by the double-precision stencil), k_tiled from shared memory.
constexpr int ZPAIRS = 16;   // floats of one plane's z metrics in load_pairs order
template <typename T> struct AxisLocal;
template <> struct AxisLocal<float> {
    float w0m_, w1m_, w0_, w1_, idc_, idcp_, idfm_, idf_;
    __device__ __forceinline__ void load(const Metric1D<float> &m, int p) {
        w0m_ = __ldg(m.w0 + p - 1); w1m_ = __ldg(m.w1 + p - 1); w0_ = __ldg(m.w0 + p); w1_ = __ldg(m.w1 + p);
        idc_ = __ldg(m.idc + p); idcp_ = __ldg(m.idc + p + 1); idfm_ = __ldg(m.idf + p - 1); idf_ = __ldg(m.idf + p);
    }
    __device__ __forceinline__ float w0m() const { return w0m_; }
    __device__ __forceinline__ float w1m() const { return w1m_; }
    __device__ __forceinline__ float w0() const { return w0_; }
    __device__ __forceinline__ float w1() const { return w1_; }
    __device__ __forceinline__ float invc() const { return idc_; }
    __device__ __forceinline__ float invcp() const { return idcp_; }
    __device__ __forceinline__ float invf() const { return idf_; }
    __device__ __forceinline__ float invfm() const { return idfm_; }
};
template <> struct AxisLocal<F2> {   // packed pairs: the same metrics broadcast to both lanes, read once
    F2 w0m_, w1m_, w0_, w1_, idc_, idcp_, idfm_, idf_;
    __device__ __forceinline__ void load(const Metric1D<float> &m, int p) {
        w0m_ = F2(__ldg(m.w0 + p - 1)); w1m_ = F2(__ldg(m.w1 + p - 1)); w0_ = F2(__ldg(m.w0 + p)); w1_ = F2(__ldg(m.w1 + p));
        idc_ = F2(__ldg(m.idc + p)); idcp_ = F2(__ldg(m.idc + p + 1)); idfm_ = F2(__ldg(m.idf + p - 1)); idf_ = F2(__ldg(m.idf + p));
    }
    // the same eight values, each twice (w0, w1 at p-1 and p; idc at p, p+1; idf at p-1, p), from 16-byte aligned storage
    __device__ __forceinline__ void load_pairs(const float *z) {
        const float4 *z4 = reinterpret_cast<const float4 *>(z);
        const float4 a = z4[0], b = z4[1], c = z4[2], e = z4[3];
        w0m_ = F2::pair(a.x, a.y); w1m_ = F2::pair(a.z, a.w); w0_ = F2::pair(b.x, b.y); w1_ = F2::pair(b.z, b.w);
        idc_ = F2::pair(c.x, c.y); idcp_ = F2::pair(c.z, c.w); idfm_ = F2::pair(e.x, e.y); idf_ = F2::pair(e.z, e.w);
    }
    __device__ __forceinline__ F2 w0m() const { return w0m_; }
    __device__ __forceinline__ F2 w1m() const { return w1m_; }
    __device__ __forceinline__ F2 w0() const { return w0_; }
    __device__ __forceinline__ F2 w1() const { return w1_; }
    __device__ __forceinline__ F2 invc() const { return idc_; }
    __device__ __forceinline__ F2 invcp() const { return idcp_; }
    __device__ __forceinline__ F2 invf() const { return idf_; }
    __device__ __forceinline__ F2 invfm() const { return idfm_; }
};
template <> struct AxisLocal<double> {
    const double *v;   // the eight values of load_pairs' order, once each (shared memory in k_tiled, else StepArgs::zmd, ymd)
    __device__ __forceinline__ double w0m() const { return v[0]; }
    __device__ __forceinline__ double w1m() const { return v[1]; }
    __device__ __forceinline__ double w0() const { return v[2]; }
    __device__ __forceinline__ double w1() const { return v[3]; }
    __device__ __forceinline__ double invc() const { return v[4]; }
    __device__ __forceinline__ double invcp() const { return v[5]; }
    __device__ __forceinline__ double invfm() const { return v[6]; }
    __device__ __forceinline__ double invf() const { return v[7]; }
};

// The gradient factor of the eddy viscosity's wall override for every wall cell (wall_gradient_factor), from the
// velocity the eddy viscosity is then computed from: U and W as stored, or (CORR) the previous stage's u* with its
// projection applied exactly as the stage kernels' loaders apply it.  One thread per
// wall cell (blockIdx.z: the wall): the Reichardt solve runs once per wall cell here instead of on the critical path of
// every tile that holds the cell.  One thread for both walls took 9.5 us at 96 x 96 columns, this form 5.9 us.
template <typename T, bool CORR>
__global__ void __launch_bounds__(WALL_THREADS) k_wall_sgs(StepArgs<T> a, const T *__restrict__ U, const T *__restrict__ W, const T *__restrict__ phi,
                           double *__restrict__ wfac) {
    pdl_enter();
    const Dims &d = a.d;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i >= d.Nx) return;
    const int im = wrap(i - 1, d.Nx), ip = wrap(i + 1, d.Nx), km = wrap(k - 1, d.Nz), kp = wrap(k + 1, d.Nz);
    const int iw = blockIdx.z, j = iw ? d.Ny - 1 : 0;
    T u0 = U[idx3(d, im, j, k)], u1 = U[idx3(d, i, j, k)], w0 = W[idx3(d, i, j, km)], w1 = W[idx3(d, i, j, k)];
    if constexpr (CORR) {
        const T pm = phi[idx3(d, im, j, k)], pc = phi[idx3(d, i, j, k)], pp = phi[idx3(d, ip, j, k)];
        const T pkm = phi[idx3(d, i, j, km)], pkp = phi[idx3(d, i, j, kp)];
        u0 = u0 - (pc - pm) * a.inv_dx;
        u1 = u1 - (pp - pc) * a.inv_dx;
        w0 = w0 - (pc - pkm) * a.mz.idf[km];
        w1 = w1 - (pkp - pc) * a.mz.idf[k];
    }
    const T ubj = a.ub[j];
    const T Um = u0 + ubj, Uc = u1 + ubj;   // as TileQ::U forms them
    const double u_c = 0.5 * ((double)Um + (double)Uc);
    const double w_c = 0.5 * ((double)w0 + (double)w1);
    wfac[((long long)iw * d.Nz + k) * d.Nx + i] = wall_gradient_factor(u_c, w_c, iw == 0, iw ? a.ygtop : a.yg2, a.nu_d);
}

// Wall-model flux of the cell at t (plain types) or of the cells at t and t+1 (packed pairs), from double.
template <typename T> __device__ __forceinline__ T wall_flux(const double *t) { return (T)t[0]; }
template <> __device__ __forceinline__ F2 wall_flux<F2>(const double *t) { return F2::pair((float)t[0], (float)t[1]); }

// The right-hand sides of u, v and w (src/equations.f90:25-721) at one index (i, j, k), from the neighbourhood accessor q
// (q.Ud: U as stored, the deviation from the row's base profile; equal to U in FP64).  Every boundary rule is applied in q
// and the profile terms, so the formulas see the values the reference reads from its ghosted arrays.
//
// The reference writes each convective term as wd (a1 b1 - a0 b0) + wa b (a1 - a0), a the advected and b the advecting
// velocity on the two faces, b = (b0 + b1)/2 and wa + wd = 1 (wa = 1/2 skew-symmetric, 0 divergence form and in the wall
// band).  It is evaluated here in the equivalent forms with the fewest operations:
//   a1 (wd b1 + m) - a0 (wd b0 + m), m = wa (b0 + b1)/2              for vw and wv, which have no mean part,
//   (wd b1 or a's total) (b1 - b0) + (a1 - a0)(p b0 + q b1)           where U takes part: FP32 then takes a1 - a0 from the
//     stored deviations and the profile's own steps, without the cancellation of the mean flow.  On a smooth channel flow
//     with 96 rows the u equation is 2.2e-7 from 64 bits that way; with the first form for uv it was 8.5e-7, no faster,
//   (a1 - a0) (wd (a1 + a0) + wa a)                                  for uu, vv, ww,
// interpolations to the y face j and the z face k are shared by two equations each, with constant viscosity the two terms of
// a flux are collected before its metric, and with an eddy viscosity each edge's shear flux is formed once.  About 160
// operations per cell against 240 for the term by term form (which in FP64 had 24 divisions besides), and in FP64 with a
// smaller error against 80-bit arithmetic (relative to a noisy channel's right-hand sides: u 1.8e-15 -> 1.4e-16, v and w
// 1.7e-16 -> 1.6e-16; a smooth one's: u 7.2e-15 -> 2.4e-16), since fewer terms are rounded.  The stage kernels are bound by
// instruction issue at 16 warps per SM: 256 x 192 x 256 cells went from 172 to 146 us (stage 1) and from 223 to 187 us (fused
// stage) in FP32, and the FP64 step from 2.74 to 2.41 ms; the LES kernels on 96 x 64 x 96 cells take 20 us as before in FP32,
// 90 x 53 x 60 cells step in 195 against 224 us in FP64.
template <typename T, bool LES, bool WM, typename Q, typename SA, typename ZM>
__device__ __forceinline__ void rhs_at(const SA &a, const Q &q, const AxisLocal<T> &Y, const RowProfile<T> &R, const ZM &Z,
                                       const double *__restrict__ tau_x, const double *__restrict__ tau_z, int i, int j,
                                       int k, bool vrow, T &ru, T &rv, T &rw) {
    constexpr bool PROF = Fp32Forms<T>::value;
    const Dims &d = a.d;
    const auto &K = a.rc;
    const T inv_dx = bcast<T>(K.inv_dx), half = bcast<T>(K.half), m2 = bcast<T>(K.m2), nu = bcast<T>(K.nu);
    const T wd0 = bcast<T>(K.wd), q0 = bcast<T>(K.q), hwd0 = bcast<T>(K.hwd), p0 = bcast<T>(K.p);   // v: never banded
    T wd = wd0, hwd = hwd0, pp = p0, qq = q0, hp = bcast<T>(K.hp), hq = bcast<T>(K.hq);
    if (WM && a.wm && (j < a.nwl || j >= d.Ny - a.nwl)) {   // divergence form in the wall band
        wd = T(1); hwd = T(0.5); pp = T(1); qq = T(0); hp = T(0.5); hq = T(0);
    }
    const bool wall_lo = WM && a.wm && j == 0, wall_hi = WM && a.wm && j == d.Ny - 1;
    const bool in_lo = d.yper != 0 || j != 0, in_hi = d.yper != 0 || j != d.Ny - 1;   // LES: nu_t reaches the face
    (void)wall_lo; (void)wall_hi; (void)in_lo; (void)in_hi;
    auto N = [&](int di, int dj, int dk) { return q.N(di, dj, dk); };

    // Values that two equations share are written out in both: the compiler keeps them in registers, except in the LES
    // kernels, where SEP makes it read the shared planes again instead (their registers are full: it would spill).
    auto SEP = [] { if constexpr (LES) asm volatile("" ::: "memory"); };
    // LES: the shear fluxes through the upper edges, (nu + nu_t)(dU_a/dx_b + dU_b/dx_a), serve two equations each
    T fxy = T(0), fxz = T(0), fyz = T(0);
    (void)fxy; (void)fxz; (void)fyz;
    // ---- u ----
    {
        const T Uc = q.Ud(0, 0, 0), Vc = q.V(0, 0, 0), Wc = q.W(0, 0, 0), Ujp = q.Ud(0, 1, 0), Ukp = q.Ud(0, 0, 1);
        const T V10 = q.V(1, 0, 0), W10 = q.W(1, 0, 0);
        const T uy = mad(Y.w1(), Ujp, mulv(Y.w0(), Uc)), uz = mad(Z.w1(), Ukp, mulv(Z.w0(), Uc));   // to y face j, z face k
        const T dUy = Ujp - Uc, dUz = Ukp - Uc, dVx = V10 - Vc, dWx = W10 - Wc;
        const T Um = q.Ud(-1, 0, 0), Up = q.Ud(1, 0, 0), s = Up + Um;
        T e;
        if constexpr (PROF) e = mad(hwd, s, Uc + R.x); else e = mad(hwd, s, Uc);
        T r = mad(mulv(bcast<T>(K.cx), Up - Um), e, bcast<T>(K.dPdx));
        const T V0m = q.V(0, -1, 0), V1m = q.V(1, -1, 0), Ujm = q.Ud(0, -1, 0);
        const T W0m = q.W(0, 0, -1), W1m = q.W(1, 0, -1), Ukm = q.Ud(0, 0, -1);
        // y
        const T vs1 = Vc + V10, vs0 = V0m + V1m;
        T u1 = uy, duy = uy - mad(Y.w1m(), Uc, mulv(Y.w0m(), Ujm));
        if constexpr (PROF) { u1 = u1 + R.f; duy = duy + R.df; }
        const T cy = mad(duy, mad(hq, vs1, mulv(hp, vs0)), mulv(mulv(hwd, u1), vs1 - vs0));
        // z
        const T ws1 = Wc + W10, ws0 = W0m + W1m, uzm = mad(Z.w1m(), Uc, mulv(Z.w0m(), Ukm)), du = uz - uzm;
        T ut;
        if constexpr (PROF) ut = uz + R.u; else ut = uz;
        const T cz = mad(du, mad(hq, ws1, mulv(hp, ws0)), mulv(mulv(hwd, ut), ws1 - ws0));
        if constexpr (LES || WM) {
            T nx1 = nu, nx2 = nu, ny1 = nu, ny2 = nu, nz1 = nu, nz2 = nu;
            if constexpr (LES) {
                const T n0 = N(0, 0, 0), n1 = N(1, 0, 0), ns = n0 + n1;
                nx1 = nu + n0; nx2 = nu + n1;
                if (in_lo) ny1 = mad(half, mad(Y.w0m(), N(0, -1, 0) + N(1, -1, 0), mulv(Y.w1m(), ns)), nu);
                if (in_hi) ny2 = mad(half, mad(Y.w1(), N(0, 1, 0) + N(1, 1, 0), mulv(Y.w0(), ns)), nu);
                nz1 = mad(half, mad(Z.w0m(), N(0, 0, -1) + N(1, 0, -1), mulv(Z.w1m(), ns)), nu);
                nz2 = mad(half, mad(Z.w1(), N(0, 0, 1) + N(1, 0, 1), mulv(Z.w0(), ns)), nu);
            }
            T sp = dUy, sm = Uc - Ujm;
            if constexpr (PROF) { sp = sp + R.dp; sm = sm + R.dm; }
            T fy2 = mulv(ny2, mad(Y.invf(), sp, mulv(inv_dx, dVx)));
            T fy1 = mulv(ny1, mad(Y.invfm(), sm, mulv(inv_dx, V1m - V0m)));
            const T fz2 = mulv(nz2, mad(Z.invf(), dUz, mulv(inv_dx, dWx)));
            fxy = fy2; fxz = fz2;
            if (wall_lo) fy1 = wall_flux<T>(tau_x + k * d.Nx + i);
            if (wall_hi) fy2 = wall_flux<T>(tau_x + (d.Nz + k) * d.Nx + i);
            const T fz1 = mulv(nz1, mad(Z.invfm(), Uc - Ukm, mulv(inv_dx, W1m - W0m)));
            const T fx = nmad(nx1, Uc - Um, mulv(nx2, Up - Uc));
            r = mad(bcast<T>(K.two_inv_dx2), fx, r);
            r = mad(Y.invc(), (fy2 - fy1) - cy, r);
            ru = mad(Z.invc(), (fz2 - fz1) - cz, r);
        } else {
            r = mad(bcast<T>(K.n2x), mad(m2, Uc, s), r);
            T F;
            if constexpr (PROF) F = mad(Y.invf(), dUy, R.c); else F = mulv(Y.invf(), dUy);
            F = mad(inv_dx, dVx - (V1m - V0m), nmad(Y.invfm(), Uc - Ujm, F));
            r = mad(Y.invc(), mad(nu, F, -cy), r);
            F = nmad(Z.invfm(), Uc - Ukm, mulv(Z.invf(), dUz));
            F = mad(inv_dx, dWx - (W1m - W0m), F);
            ru = mad(Z.invc(), mad(nu, F, -cz), r);
        }
    }
    // ---- v ----
    rv = T(0);
    if (vrow) {
        SEP();
        const T Uc = q.Ud(0, 0, 0), Vc = q.V(0, 0, 0), Wc = q.W(0, 0, 0), Ujp = q.Ud(0, 1, 0), Wjp = q.W(0, 1, 0);
        const T V10 = q.V(1, 0, 0), Vkp = q.V(0, 0, 1);
        const T uy = mad(Y.w1(), Ujp, mulv(Y.w0(), Uc)), wy = mad(Y.w1(), Wjp, mulv(Y.w0(), Wc));   // to y face j
        const T vz = mad(Z.w1(), Vkp, mulv(Z.w0(), Vc));                                             // to z face k
        const T dUy = Ujp - Uc, dWy = Wjp - Wc, dVx = V10 - Vc, dVz = Vkp - Vc;
        const T Vjp = q.V(0, 1, 0), Vjm = q.V(0, -1, 0), Vm = q.V(-1, 0, 0), Vkm = q.V(0, 0, -1);
        const T Um = q.Ud(-1, 0, 0), Ump = q.Ud(-1, 1, 0), Wkm = q.W(0, 0, -1), Wkmjp = q.W(0, 1, -1);
        // y
        const T ey = mulv(mulv(half, Vjp - Vjm), mad(hwd0, Vjp + Vjm, Vc));
        // x
        const T um = mad(Y.w1(), Ump, mulv(Y.w0(), Um)), du = uy - um, vs = Vm + Vc;
        T g;
        if constexpr (PROF) g = mad(q0, um, mad(p0, uy, R.f)); else g = mad(q0, um, mulv(p0, uy));
        const T cx = mad(mulv(hwd0, vs), du, mulv(mulv(half, V10 - Vm), g));
        // z
        const T vzm = mad(Z.w1m(), Vc, mulv(Z.w0m(), Vkm)), wym = mad(Y.w1(), Wkmjp, mulv(Y.w0(), Wkm));
        const T m = mulv(q0, wym + wy);
        const T cz = nmad(vzm, mad(wd0, wym, m), mulv(vz, mad(wd0, wy, m)));
        if constexpr (LES) {
            const T n0 = N(0, 0, 0), np = N(0, 1, 0), w0 = Y.w0(), w1 = Y.w1(), ny = mad(w1, np, mulv(w0, n0));
            const T nx1 = mad(half, mad(w1, N(-1, 1, 0), mad(w0, N(-1, 0, 0), ny)), nu);
            const T nz1 = mad(Z.w0m(), mad(w1, N(0, 1, -1), mulv(w0, N(0, 0, -1))), mad(Z.w1m(), ny, nu));
            const T nz2 = mad(Z.w1(), mad(w1, N(0, 1, 1), mulv(w0, N(0, 0, 1))), mad(Z.w0(), ny, nu));
            T un = Ump - Um;   // the total across the y face (with constant viscosity the profile's step cancels)
            if constexpr (PROF) un = un + R.dp;
            const T fx1 = mulv(nx1, mad(inv_dx, Vc - Vm, mulv(Y.invf(), un)));
            const T fz2 = mulv(nz2, mad(Z.invf(), dVz, mulv(Y.invf(), dWy)));
            fyz = fz2;
            const T fz1 = mulv(nz1, mad(Z.invfm(), Vc - Vkm, mulv(Y.invf(), Wkmjp - Wkm)));
            const T fy = nmad(nu + n0, mulv(Y.invc(), Vc - Vjm), mulv(nu + np, mulv(Y.invcp(), Vjp - Vc)));
            T r = mulv(Y.invf(), mad(fy, T(2), -ey));
            r = mad(inv_dx, (fxy - fx1) - cx, r);
            rv = mad(Z.invc(), (fz2 - fz1) - cz, r);
        } else {
            T F = nmad(Y.invc(), Vc - Vjm, mulv(Y.invcp(), Vjp - Vc));
            T r = mulv(Y.invf(), mad(bcast<T>(K.nu2), F, -ey));
            F = mad(Y.invf(), dUy - (Ump - Um), mulv(inv_dx, mad(m2, Vc, V10 + Vm)));
            r = mad(inv_dx, mad(nu, F, -cx), r);
            F = nmad(Z.invfm(), Vc - Vkm, mulv(Z.invf(), dVz));
            F = mad(Y.invf(), dWy - (Wkmjp - Wkm), F);
            rv = mad(Z.invc(), mad(nu, F, -cz), r);
        }
    }
    // ---- w ----
    {
        SEP();
        const T Uc = q.Ud(0, 0, 0), Vc = q.V(0, 0, 0), Wc = q.W(0, 0, 0), Ukp = q.Ud(0, 0, 1), Wjp = q.W(0, 1, 0);
        const T W10 = q.W(1, 0, 0), Vkp = q.V(0, 0, 1);
        const T uz = mad(Z.w1(), Ukp, mulv(Z.w0(), Uc)), vz = mad(Z.w1(), Vkp, mulv(Z.w0(), Vc));   // to z face k
        const T wy = mad(Y.w1(), Wjp, mulv(Y.w0(), Wc));                                             // to y face j
        const T dUz = Ukp - Uc, dVz = Vkp - Vc, dWy = Wjp - Wc, dWx = W10 - Wc;
        const T Wkp = q.W(0, 0, 1), Wkm = q.W(0, 0, -1), Wm = q.W(-1, 0, 0), Wjm = q.W(0, -1, 0);
        const T Um = q.Ud(-1, 0, 0), Umkp = q.Ud(-1, 0, 1), Vjm = q.V(0, -1, 0), Vjmkp = q.V(0, -1, 1);
        // z
        const T ez = mulv(mulv(half, Wkp - Wkm), mad(hwd, Wkp + Wkm, Wc));
        // x
        const T um = mad(Z.w1(), Umkp, mulv(Z.w0(), Um)), du = uz - um, ws = Wm + Wc;
        T g;
        if constexpr (PROF) g = mad(qq, um, mad(pp, uz, R.u)); else g = mad(qq, um, mulv(pp, uz));
        const T cx = mad(mulv(hwd, ws), du, mulv(mulv(half, W10 - Wm), g));
        // y
        const T vzm = mad(Z.w1(), Vjmkp, mulv(Z.w0(), Vjm)), wym = mad(Y.w1m(), Wc, mulv(Y.w0m(), Wjm));
        const T m = mulv(qq, vzm + vz);
        const T cy = nmad(wym, mad(wd, vzm, m), mulv(wy, mad(wd, vz, m)));
        if constexpr (LES || WM) {
            T nx1 = nu, ny1 = nu, nz1 = nu, nz2 = nu, fx2, fy2;
            if constexpr (LES) {
                const T n0 = N(0, 0, 0), np = N(0, 0, 1), z0 = Z.w0(), z1 = Z.w1(), nz = mad(z1, np, mulv(z0, n0));
                nx1 = mad(half, mad(z1, N(-1, 0, 1), mad(z0, N(-1, 0, 0), nz)), nu);
                if (in_lo) ny1 = mad(Y.w0m(), mad(z1, N(0, -1, 1), mulv(z0, N(0, -1, 0))), mad(Y.w1m(), nz, nu));
                nz1 = nu + n0;
                nz2 = nu + np;
                fx2 = fxz;
                fy2 = vrow ? fyz : mulv(nu, mad(Y.invf(), dWy, mulv(Z.invf(), dVz)));   // the top wall: nu_t does not reach it
            } else {
                fx2 = mulv(nu, mad(inv_dx, dWx, mulv(Z.invf(), dUz)));
                fy2 = mulv(nu, mad(Y.invf(), dWy, mulv(Z.invf(), dVz)));
            }
            T fy1 = mulv(ny1, mad(Y.invfm(), Wc - Wjm, mulv(Z.invf(), Vjmkp - Vjm)));
            if (wall_lo) fy1 = wall_flux<T>(tau_z + k * d.Nx + i);
            if (wall_hi) fy2 = wall_flux<T>(tau_z + (d.Nz + k) * d.Nx + i);
            const T fx1 = mulv(nx1, mad(inv_dx, Wc - Wm, mulv(Z.invf(), Umkp - Um)));
            const T fz = nmad(nz1, mulv(Z.invc(), Wc - Wkm), mulv(nz2, mulv(Z.invcp(), Wkp - Wc)));
            T r = mad(Z.invf(), mad(fz, T(2), -ez), bcast<T>(K.dPdz));
            r = mad(inv_dx, (fx2 - fx1) - cx, r);
            rw = mad(Y.invc(), (fy2 - fy1) - cy, r);
        } else {
            T F = nmad(Z.invc(), Wc - Wkm, mulv(Z.invcp(), Wkp - Wc));
            T r = mad(Z.invf(), mad(bcast<T>(K.nu2), F, -ez), bcast<T>(K.dPdz));
            F = mad(Z.invf(), dUz - (Umkp - Um), mulv(inv_dx, mad(m2, Wc, W10 + Wm)));
            r = mad(inv_dx, mad(nu, F, -cx), r);
            F = nmad(Y.invfm(), Wc - Wjm, mulv(Y.invf(), dWy));
            F = mad(Z.invf(), dVz - (Vjmkp - Vjm), F);
            rw = mad(Y.invc(), mad(nu, F, -cy), r);
        }
    }
}

// wd of row j: 1 in the wall band of the wall model, else the blend's
template <typename T, bool WM, typename SA> __device__ __forceinline__ T row_wd(const SA &a, int j) {
    if (WM && a.wm && (j < a.nwl || j >= a.d.Ny - a.nwl)) return T(1);
    return bcast<T>(a.rc.wd);
}

// Stage coefficients of the Butcher-form RK3 update (src/time_integration.f90:255-259, :393-397, :525-532):
//   s = 1: u* = uo + (dt a11) F1                 (F1 = rhs, uo = u)
//   s = 2: u* = uo + dt (a21 F1 + a22 rhs)
//   s = 3: u* = uo + dt (a31 F1 + a33 rhs)        (a32 = 0, so F2 is never needed)
struct StageCoef {
    int stage;       // 1, 2 or 3
    double dt_a11;   // dt*rk_coef(1,1), stage 1
    double dt;       // dt, stages 2 and 3
    double c1, c2;   // rk_coef(s,1) and rk_coef(s,s), stages 2 and 3
    int incr;        // store the increment du = dt (c1 F1 + c2 rhs) instead of u* = uo + du; uo is not read
    const double *dtp = nullptr;   // adaptive time step: dt is dtp[0] (device memory) and dt_a11, dt are not used
    int no_uo = 0;                 // stage 1: the step-start velocity stays in U (fused corrections), uo is not written
};

// Shared-memory neighbourhood of one thread: three z-planes (k-1, k, k+1) of each field, each plane a
// (TX+2) x (TY+2) tile with a one-cell halo in x and y.
template <typename T, int PX> struct TileQ {
    const T *u[3], *v[3], *w[3], *n[3];
    int c;       // local index of the centre cell
    T ub[3];     // streamwise base profile of rows j-1, j, j+1 (mirrored on wall ghost rows)
    // U (total) and Ud (stored deviation from the base profile; equal to U in FP64, where the profile is zero)
    __device__ __forceinline__ T U(int di, int dj, int dk) const { return u[dk + 1][c + dj * PX + di] + ub[dj + 1]; }
    __device__ __forceinline__ T Ud(int di, int dj, int dk) const { return u[dk + 1][c + dj * PX + di]; }
    __device__ __forceinline__ T V(int di, int dj, int dk) const { return v[dk + 1][c + dj * PX + di]; }
    __device__ __forceinline__ T W(int di, int dj, int dk) const { return w[dk + 1][c + dj * PX + di]; }
    __device__ __forceinline__ T N(int di, int dj, int dk) const { return n[dk + 1][c + dj * PX + di]; }
};

// The same neighbourhood for a pair of x-neighbour cells (c, c+1) in FP32 shared planes; c is even and so is the
// row pitch PX, so a pair at an even x-offset is one 8-byte shared load.
template <int PX> struct TileQ2 {
    const float *u[3], *v[3], *w[3], *n[3];
    int c;
    static __device__ __forceinline__ F2 ld(const float *pl, int off) {
        if ((off & 1) == 0) return F2(*reinterpret_cast<const float2 *>(pl + off));
        return F2::pair(pl[off], pl[off + 1]);
    }
    __device__ __forceinline__ F2 Ud(int di, int dj, int dk) const { return ld(u[dk + 1] + c, dj * PX + di); }
    __device__ __forceinline__ F2 V(int di, int dj, int dk) const { return ld(v[dk + 1] + c, dj * PX + di); }
    __device__ __forceinline__ F2 W(int di, int dj, int dk) const { return ld(w[dk + 1] + c, dj * PX + di); }
    __device__ __forceinline__ F2 N(int di, int dj, int dk) const { return ld(n[dk + 1] + c, dj * PX + di); }
};



// One thread's cell (i, j, k) from the shared-memory neighbourhood q: the three right-hand sides and the RK3 stage
// update (or, with rhs_only, the right-hand sides themselves).  Shared by the one-cell stage kernels.
template <typename T, bool LES, bool WM, bool HYB, typename Q>
__device__ __forceinline__ void stage_cell(const StepArgs<T> &a, const Q &q, const AxisLocal<T> &Y,
                                           const RowProfile<T> &R, const T *zm, const double *__restrict__ tau_x,
                                           const double *__restrict__ tau_z, const StageCoef &sc, int i, int j, int k, T *__restrict__ uo,
                                           T *__restrict__ vo, T *__restrict__ wo, T *__restrict__ f1u,
                                           T *__restrict__ f1v, T *__restrict__ f1w, T *__restrict__ us,
                                           T *__restrict__ vs, T *__restrict__ wsf, T *__restrict__ rhs_only) {
    const Dims &d = a.d;
    const int p = k * (d.Nx * d.Ny) + j * d.Nx + i;
    const bool vrow = j < d.NyV;
    const bool upd = !rhs_only && sc.stage != 1;
    T ou = T(0), ov = T(0), ow = T(0), fu = T(0), fv = T(0), fw = T(0);
    if (upd) {   // issue the base-state and F1 loads before the arithmetic
        if (!sc.incr) { ou = uo[p]; ow = wo[p]; if (vrow) ov = vo[p]; }
        fu = f1u[p]; fw = f1w[p];
        if (vrow) fv = f1v[p];
    }
    AxisLocal<T> Z;
    if constexpr (sizeof(T) == 8) Z.v = zm; else Z.load(a.mz, k);
    T ru, rv, rw;
    rhs_at<T, LES, WM>(a, q, Y, R, Z, tau_x, tau_z, i, j, k, vrow, ru, rv, rw);
    if constexpr (HYB) {
        ru = ru + a.adv[p]; rw = rw + a.adv[2 * d.cells + p];
        if (vrow) rv = rv + a.adv[d.cells + p];
    }
    if (rhs_only) {
        rhs_only[p] = ru; rhs_only[d.cells + p] = rv; rhs_only[2 * d.cells + p] = rw;
    } else if (sc.stage == 1) {
        T c = (T)(sc.dtp ? *sc.dtp * (8.0 / 15.0) : sc.dt_a11);
        T u0 = q.Ud(0, 0, 0), w0 = q.W(0, 0, 0);   // U as stored (deviation from the base profile)
        f1u[p] = ru; us[p] = u0 + c * ru;
        f1w[p] = rw; wsf[p] = w0 + c * rw;
        if (!sc.no_uo) { uo[p] = u0; wo[p] = w0; }
        if (vrow) {
            T v0 = q.V(0, 0, 0);
            f1v[p] = rv; vs[p] = v0 + c * rv;
            if (!sc.no_uo) vo[p] = v0;
        }
    } else {
        T c1 = (T)sc.c1, c2 = (T)sc.c2, dtt = (T)(sc.dtp ? *sc.dtp : sc.dt);   // with sc.incr the base stays zero: du
        us[p] = ou + dtt * (c1 * fu + c2 * ru);
        wsf[p] = ow + dtt * (c1 * fw + c2 * rw);
        if (vrow) vs[p] = ov + dtt * (c1 * fv + c2 * rv);
    }
}

// Tiled kernels (KIND 0: fused stage, KIND 1: eddy viscosity, KIND 2: fused stage adding the dissipative terms of
// advection_scheme = 2 from StepArgs::adv), 2.5-D blocked: a block owns a TX x TY column of
// (i,j) cells and marches through a chunk of kc z-planes.  Each z-plane of U, V, W (and nu_t) is copied from HBM
// once per block, with its one-cell halo, into one of four rotating shared planes by cp.async: the copies of
// plane k+2 are in flight while the cells of plane k are evaluated, and one barrier per plane suffices.  After
// its copies land, each thread adds the streamwise base profile to the U elements it copied and applies the wall
// rules (no-slip mirror of U and W, zero V and nu_t on the ghost rows).  Every thread then evaluates the three
// right-hand sides of its cell from shared memory and writes the RK3 update (or, with rhs_only, the right-hand
// sides themselves for the unit entry point; with KIND 1, nu_t).
// WM = false compiles the flat-wall model out.
// CORR (stages 2 and 3 of a step whose stage kernel is the only reader of the corrected velocity): U, V, W are the
// previous stage's u*, and the loader applies that stage's projection, u = u* - grad(phi) with StepArgs::phi, to
// every plane element it copies, before the wall rules -- the arithmetic of k_correct, so the values are the ones
// k_correct would have stored.  phi planes rotate through five more shared planes and are copied two planes ahead
// of the velocity planes (a plane's w correction needs phi of the plane above), so they have landed, and passed a
// barrier, before the plane that needs them is corrected.
template <typename T, bool LES, bool WM, int TX, int TY, int KIND, bool CORR = false, class BC>
__device__ __forceinline__ void k_tiled_body(const BC &bc, const StepArgs<T> &a, const T *__restrict__ U, const T *__restrict__ V,
                                                  const T *__restrict__ W, const T *__restrict__ NU,
                                                  const double *__restrict__ tau_x, const double *__restrict__ tau_z,
                                                  const StageCoef &sc, const int kc, T *__restrict__ uo, T *__restrict__ vo,
                                                  T *__restrict__ wo, T *__restrict__ f1u, T *__restrict__ f1v,
                                                  T *__restrict__ f1w, T *__restrict__ us, T *__restrict__ vs,
                                                  T *__restrict__ wsf, T *__restrict__ rhs_only, T *__restrict__ nut_out) {
    constexpr int PX = TX + 2, PY = TY + 2, PS = PX * PY, NT = TX * TY;
    constexpr int NF = LES ? 4 : 3;
    constexpr int PER = (PS + NT - 1) / NT;   // plane elements per thread
    __shared__ __align__(16) T sm[NF][4][PS];
    constexpr int PXP = PX + 1, PSP = PXP * (PY + 1), PERP = (PSP + NT - 1) / NT;   // phi tile: one more column, row
    __shared__ __align__(16) T smp[CORR ? 5 : 1][CORR ? PSP : 1];
    // FP64: the metrics of the tile's rows and, in a ring, of planes k .. k+2.  A thread reads each value several times per
    // cell, and read from the global tables they were the kernel's longest stall: a step took 2296 us at 256 x 192 x 256
    // (2166 from shared memory) and 301 us at 128 x 94 x 128 (285)
    constexpr bool MS = sizeof(T) == 8 && KIND != 1;
    __shared__ double ymr[MS ? TY * 8 : 1], zmr[MS ? 4 : 1][8];
    const Dims &d = a.d;
    const int Nx = d.Nx, Ny = d.Ny, Nz = d.Nz;
    const int i0 = bc.idx().x * TX, j0 = bc.idx().y * TY;
    const int k0 = bc.idx().z * kc, kend = min(k0 + kc, Nz);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    auto issue_z = [&](int k) {   // the z metrics of plane k (k0 <= k < kend) into zmr[(k - k0) & 3]
        if constexpr (MS)
            if (threadIdx.x < 8 && k < kend) cp_async<8>(&zmr[(k - k0) & 3][threadIdx.x], a.zmd + 8 * k + threadIdx.x);
    };
    const int i = i0 + tx, j = j0 + ty;
    const bool active = i < Nx && j < Ny;
    const int plane = Nx * Ny;

    // This thread's share of a plane: offsets within the plane (or -1), the wall rule and the base profile.
    int off[PER];
    bool ghost[PER];   // wall ghost row: mirror U/W, zero V/nu_t
    int pix[CORR ? PER : 1];    // CORR: phi-tile index of the element
    T iyq[CORR ? PER : 1];      // CORR: 1/(centre spacing) of its row for the v correction, 0 where v is not corrected
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        int e = threadIdx.x + q * NT;
        off[q] = -1; ghost[q] = false;
        if (e < PS) {
            int jj = e / PX, ii = e - jj * PX;
            int gi = i0 - 1 + ii;
            gi = gi < 0 ? gi + Nx : gi;
            while (gi >= Nx) gi -= Nx;
            int gj = j0 - 1 + jj, g;
            if (d.yper) {
                g = gj < 0 ? gj + Ny : gj;
                while (g >= Ny) g -= Ny;
            } else {
                g = gj < 0 ? 0 : (gj >= Ny ? Ny - 1 : gj);
                ghost[q] = (gj < 0 || gj >= Ny);
            }
            off[q] = g * Nx + gi;
            if constexpr (CORR) {
                pix[q] = jj * PXP + ii;
                iyq[q] = (ghost[q] || g >= d.NyV) ? T(0) : a.my.idf[g];
            }
        }
    }
    int offp[CORR ? PERP : 1];   // CORR: this thread's share of a phi plane (same row and column rules)
    if constexpr (CORR) {
#pragma unroll
        for (int q = 0; q < PERP; ++q) {
            int e = threadIdx.x + q * NT;
            offp[q] = -1;
            if (e < PSP) {
                int jj = e / PXP, ii = e - jj * PXP;
                int gi = i0 - 1 + ii;
                gi = gi < 0 ? gi + Nx : gi;
                while (gi >= Nx) gi -= Nx;
                int gj = j0 - 1 + jj, g;
                if (d.yper) { g = gj < 0 ? gj + Ny : gj; while (g >= Ny) g -= Ny; }
                else g = gj < 0 ? 0 : (gj >= Ny ? Ny - 1 : gj);
                offp[q] = g * Nx + gi;
            }
        }
    }
    auto issue_phi = [&](int k) {   // phi plane k into phi slot (k - k0 + 1) % 5
        if constexpr (CORR) {
            const int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k), slot = (k - k0 + 1) % 5;
#pragma unroll
            for (int q = 0; q < PERP; ++q)
                if (offp[q] >= 0) cp_async<sizeof(T)>(&smp[slot][threadIdx.x + q * NT], a.phi + kw * plane + offp[q]);
        }
    };
    auto issue = [&](int slot, int k) {
        int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k);
        const int kb = kw * plane;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (off[q] < 0) continue;
            const int o = kb + off[q], e = threadIdx.x + q * NT;
            cp_async<sizeof(T)>(&sm[0][slot][e], U + o);
            cp_async<sizeof(T)>(&sm[2][slot][e], W + o);
            if (!ghost[q]) {
                cp_async<sizeof(T)>(&sm[1][slot][e], V + o);
                if (LES) cp_async<sizeof(T)>(&sm[NF - 1][slot][e], NU + o);
            }
        }
    };
    auto fix = [&](int slot, int k) {   // after the copies of plane k (and, CORR, phi k and k+1) have landed
        if constexpr (CORR) {   // project_velocity of the previous stage (k_correct's arithmetic)
            const int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k);
            const int p0 = (k - k0 + 1) % 5, p1 = (k - k0 + 2) % 5;
            const T iz = a.mz.idf[kw];
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                if (off[q] < 0) continue;
                const int e = threadIdx.x + q * NT;
                const T pc = smp[p0][pix[q]], pxp = smp[p0][pix[q] + 1], pzp = smp[p1][pix[q]];
                sm[0][slot][e] = sm[0][slot][e] - (pxp - pc) * a.inv_dx;
                sm[2][slot][e] = sm[2][slot][e] - (pzp - pc) * iz;
                if (iyq[q] != T(0)) sm[1][slot][e] = sm[1][slot][e] - (smp[p0][pix[q] + PXP] - pc) * iyq[q];
            }
        }
#pragma unroll
        for (int q = 0; q < PER; ++q) {   // wall ghost rows
            if (off[q] < 0 || !ghost[q]) continue;
            const int e = threadIdx.x + q * NT;
            sm[0][slot][e] = -sm[0][slot][e];   // deviation mirrored; the row profile is mirrored in TileQ::ub
            sm[2][slot][e] = -sm[2][slot][e];
            sm[1][slot][e] = T(0);
            if (LES) sm[NF - 1][slot][e] = T(0);
        }
    };
    // base profile of the thread's rows j-1, j, j+1 (a wall ghost row carries minus its mirror row's profile)
    T ubr[3];
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj) {
        int gj = min(j, Ny - 1) + dj;
        T sgn = T(1);
        if (d.yper) { gj = gj < 0 ? gj + Ny : (gj >= Ny ? gj - Ny : gj); }
        else if (gj < 0 || gj >= Ny) { gj = gj < 0 ? 0 : Ny - 1; sgn = T(-1); }
        ubr[dj + 1] = sgn * __ldg(a.ub + gj);
    }

    AxisLocal<T> Y;   // this thread's y metrics (FP32: read here once for every plane)
    if constexpr (sizeof(T) == 8 && KIND != 1) {
        for (int e = threadIdx.x; e < TY * 8; e += NT) ymr[e] = a.ymd[min(j0 + e / 8, Ny - 1) * 8 + e % 8];
        Y.v = reinterpret_cast<const double *>(ymr) + 8 * ty;
    } else if constexpr (sizeof(T) == 4) {
        Y.load(a.my, min(j, Ny - 1));
    }
    RowProfile<T> R;
    R.load(ubr, Y, row_wd<T, WM>(a, j));

    // planes k0-1, k0, k0+1 into slots 0, 1, 2; plane k lives in slot (k - k0 + 1) & 3 (CORR: phi k0-1 .. k0+2)
    issue(0, k0 - 1); issue(1, k0); issue(2, k0 + 1);
    issue_phi(k0 - 1); issue_phi(k0); issue_phi(k0 + 1); issue_phi(k0 + 2); issue_phi(k0 + 3);
    issue_z(k0); issue_z(k0 + 1);
    cp_async_commit();
    cp_async_wait_all();
    if (CORR) __syncthreads();   // phi elements copied by other threads
    fix(0, k0 - 1); fix(1, k0); fix(2, k0 + 1);
    __syncthreads();
    const int cloc = (ty + 1) * PX + tx + 1;
    for (int k = k0; k < kend; ++k) {
        const bool more = k + 2 <= kend;
        const int snext = (k - k0 + 3) & 3;
        if (more) { issue(snext, k + 2); issue_phi(k + 4); }
        issue_z(k + 2);
        cp_async_commit();
        const int sm_ = (k - k0) & 3, s0 = (k - k0 + 1) & 3, sp = (k - k0 + 2) & 3;
        if (active) {
            const int p = k * plane + j * Nx + i;
            TileQ<T, PX> q;
            q.c = cloc;
            q.ub[0] = ubr[0]; q.ub[1] = ubr[1]; q.ub[2] = ubr[2];
            q.u[0] = sm[0][sm_]; q.u[1] = sm[0][s0]; q.u[2] = sm[0][sp];
            q.v[0] = sm[1][sm_]; q.v[1] = sm[1][s0]; q.v[2] = sm[1][sp];
            q.w[0] = sm[2][sm_]; q.w[1] = sm[2][s0]; q.w[2] = sm[2][sp];
            q.n[0] = sm[NF - 1][sm_]; q.n[1] = sm[NF - 1][s0]; q.n[2] = sm[NF - 1][sp];
            if (KIND == 1) {
                nut_out[p] = nut_at<T>(a, q, i, j, k);
            } else {
                const T *zm = nullptr;
                if constexpr (MS) zm = zmr[(k - k0) & 3];
                stage_cell<T, LES, WM, KIND == 2>(a, q, Y, R, zm, tau_x, tau_z, sc, i, j, k, uo, vo, wo, f1u, f1v, f1w, us, vs,
                                                  wsf, rhs_only);
            }
        }
        cp_async_wait_all();
        if (more) fix(snext, k + 2);   // CORR: phi k+2 and k+3 were copied one and two iterations ago
        __syncthreads();
    }
}
template <typename T, bool LES, bool WM, int TX, int TY, int KIND, bool CORR = false>
__global__ void __launch_bounds__(TX *TY, sizeof(T) == 4 ? 3 : 2) k_tiled(StepArgs<T> a, const T *__restrict__ U, const T *__restrict__ V,
                                                  const T *__restrict__ W, const T *__restrict__ NU,
                                                  const double *__restrict__ tau_x, const double *__restrict__ tau_z,
                                                  StageCoef sc, int kc, T *__restrict__ uo, T *__restrict__ vo,
                                                  T *__restrict__ wo, T *__restrict__ f1u, T *__restrict__ f1v,
                                                  T *__restrict__ f1w, T *__restrict__ us, T *__restrict__ vs,
                                                  T *__restrict__ wsf, T *__restrict__ rhs_only, T *__restrict__ nut_out) {
    pdl_enter();
    k_tiled_body<T, LES, WM, TX, TY, KIND, CORR>(HwBlock(), a, U, V, W, NU, tau_x, tau_z, sc, kc, uo, vo, wo, f1u, f1v, f1w, us, vs, wsf, rhs_only, nut_out);
}


// One thread's pair of cells (i, i+1) of plane k from the shared-memory neighbourhood q: the three right-hand sides
// and the RK3 stage update (or, with rhs_only, the right-hand sides themselves).  zm holds the z metrics of
// plane k (AxisLocal<F2>::load_pairs order).  Shared by the packed stage kernels.
template <bool LES, bool WM, bool HYB, int PX>
__device__ __forceinline__ void stage_pair(const StepArgs<float> &a, const TileQ2<PX> &q, const AxisLocal<F2> &Y,
                                           const RowProfile<F2> &R, const float *zm, const double *__restrict__ tau_x,
                                           const double *__restrict__ tau_z, const StageCoef &sc, int i, int j, int k,
                                           float *__restrict__ uo, float *__restrict__ vo, float *__restrict__ wo,
                                           float *__restrict__ f1u, float *__restrict__ f1v, float *__restrict__ f1w,
                                           float *__restrict__ us, float *__restrict__ vs, float *__restrict__ wsf,
                                           float *__restrict__ rhs_only) {
    const Dims &d = a.d;
    const int p = k * (d.Nx * d.Ny) + j * d.Nx + i;
    const bool vrow = j < d.NyV;
    const bool upd = !rhs_only && sc.stage != 1;
    auto ld2 = [&](const float *b) { return F2(*reinterpret_cast<const float2 *>(b + p)); };
    auto st2 = [&](float *b, F2 x) { *reinterpret_cast<float2 *>(b + p) = x.v; };
    F2 ou(0.0f), ov(0.0f), ow(0.0f), fu(0.0f), fv(0.0f), fw(0.0f);
    if (upd) {
        if (!sc.incr) { ou = ld2(uo); ow = ld2(wo); if (vrow) ov = ld2(vo); }
        fu = ld2(f1u); fw = ld2(f1w);
        if (vrow) fv = ld2(f1v);
    }
    AxisLocal<F2> Z;
    Z.load_pairs(zm);
    F2 ru, rv, rw;
    rhs_at<F2, LES, WM>(a, q, Y, R, Z, tau_x, tau_z, i, j, k, vrow, ru, rv, rw);
    if constexpr (HYB) {
        ru = ru + ld2(a.adv); rw = rw + ld2(a.adv + 2 * d.cells);
        if (vrow) rv = rv + ld2(a.adv + d.cells);
    }
    if (rhs_only) {
        st2(rhs_only, ru); st2(rhs_only + d.cells, rv); st2(rhs_only + 2 * d.cells, rw);
    } else if (sc.stage == 1) {
        const F2 c = F2(sc.dtp ? *sc.dtp * (8.0 / 15.0) : sc.dt_a11);
        F2 u0 = q.Ud(0, 0, 0), w0 = q.W(0, 0, 0);
        st2(f1u, ru); st2(us, u0 + c * ru);
        st2(f1w, rw); st2(wsf, w0 + c * rw);
        if (!sc.no_uo) { st2(uo, u0); st2(wo, w0); }
        if (vrow) {
            F2 v0 = q.V(0, 0, 0);
            st2(f1v, rv); st2(vs, v0 + c * rv);
            if (!sc.no_uo) st2(vo, v0);
        }
    } else {
        const F2 c1 = F2(sc.c1), c2 = F2(sc.c2), dtt = F2(sc.dtp ? *sc.dtp : sc.dt);
        st2(us, ou + dtt * (c1 * fu + c2 * ru));
        st2(wsf, ow + dtt * (c1 * fw + c2 * rw));
        if (vrow) st2(vs, ov + dtt * (c1 * fv + c2 * rv));
    }
}

// FP32 stage kernel with two x-neighbour cells per thread, computed with the packed FP32x2 instructions (F2).  Same
// loader, ghost rules and RK3 epilogue as k_tiled<float, LES, WM, ..., 0>; a block owns 64 x TY cells, one warp
// per row of 32 cell pairs; HYB adds the dissipative terms of advection_scheme = 2 (StepArgs::adv); CORR fuses
// the previous stage's correction into the loader as k_tiled does.  It needs ~118 registers: capping it at 96 or 80 (for more resident warps) spills
// 170-300 bytes, so it runs 2 blocks of 256 threads per SM.  Shared rows hold cells i0-2 .. i0+65 (pitch 68), so every pair starts at an even index.
template <bool LES, bool WM, int TY = 8, bool HYB = false, bool CORR = false, class BC>
__device__ __forceinline__ void k_tiled2_body(const BC &bc, const StepArgs<float> &a, const float *__restrict__ U, const float *__restrict__ V,
                                                   const float *__restrict__ W, const float *__restrict__ NU,
                                                   const double *__restrict__ tau_x, const double *__restrict__ tau_z,
                                                   const StageCoef &sc, const int kc, float *__restrict__ uo, float *__restrict__ vo,
                                                   float *__restrict__ wo, float *__restrict__ f1u, float *__restrict__ f1v,
                                                   float *__restrict__ f1w, float *__restrict__ us, float *__restrict__ vs,
                                                   float *__restrict__ wsf, float *__restrict__ rhs_only) {
    constexpr int TXC = 64, NT = 32 * TY;
    constexpr int PX = TXC + 4, PY = TY + 2, PS = PX * PY;
    constexpr int NF = LES ? 4 : 3;
    // the loader moves element pairs (columns 2m, 2m+1 of a tile row: even global x, so one 8-byte copy)
    constexpr int PS2 = PS / 2, PER = (PS2 + NT - 1) / NT;
    __shared__ __align__(16) float sm[NF][4][PS];
    // CORR phi tile: two more columns (an even pitch keeps pairs aligned) and one more row
    constexpr int PXP = PX + 2, PSP2 = PXP * (PY + 1) / 2, PERP = (PSP2 + NT - 1) / NT;
    __shared__ __align__(16) float smp[CORR ? 5 : 1][CORR ? 2 * PSP2 : 2];
    // the z metrics of planes k .. k+2 (AxisLocal<F2>::load_pairs order), copied with the planes: under the streaming
    // tile copies the metric tables do not stay in L1, and every thread needs them at the start of its plane
    __shared__ __align__(16) float zmr[4][ZPAIRS];
    const Dims &d = a.d;
    const int Nx = d.Nx, Ny = d.Ny, Nz = d.Nz;
    const int i0 = bc.idx().x * TXC, j0 = bc.idx().y * TY;
    const int k0 = bc.idx().z * kc, kend = min(k0 + kc, Nz);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i = i0 + 2 * tx, j = j0 + ty;
    const bool active = i < Nx && j < Ny;   // Nx is even: the pair's second cell is in range too
    const int plane = Nx * Ny;

    int off[PER];       // global offset of the pair's first element within a plane, or -1
    bool ghost[PER];
    int pix[CORR ? PER : 1];      // CORR: phi-tile index of the pair
    float iyq[CORR ? PER : 1];    // CORR: 1/(centre spacing) of its row for the v correction, 0 where v is not corrected
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        int e2 = threadIdx.x + q * NT;
        off[q] = -1; ghost[q] = false;
        if (e2 < PS2) {
            int jj = e2 / (PX / 2), ii = 2 * (e2 - jj * (PX / 2));
            int gi = i0 - 2 + ii;
            gi = gi < 0 ? gi + Nx : gi;
            while (gi >= Nx) gi -= Nx;
            int gj = j0 - 1 + jj, g;
            if (d.yper) {
                g = gj < 0 ? gj + Ny : gj;
                while (g >= Ny) g -= Ny;
            } else {
                g = gj < 0 ? 0 : (gj >= Ny ? Ny - 1 : gj);
                ghost[q] = (gj < 0 || gj >= Ny);
            }
            off[q] = g * Nx + gi;
            if constexpr (CORR) {
                pix[q] = jj * PXP + ii;
                iyq[q] = (ghost[q] || g >= d.NyV) ? 0.0f : a.my.idf[g];
            }
        }
    }
    int offp[CORR ? PERP : 1];   // CORR: this thread's pairs of a phi plane (same row and column rules)
    if constexpr (CORR) {
#pragma unroll
        for (int q = 0; q < PERP; ++q) {
            int e2 = threadIdx.x + q * NT;
            offp[q] = -1;
            if (e2 < PSP2) {
                int jj = e2 / (PXP / 2), ii = 2 * (e2 - jj * (PXP / 2));
                int gi = i0 - 2 + ii;
                gi = gi < 0 ? gi + Nx : gi;
                while (gi >= Nx) gi -= Nx;
                int gj = j0 - 1 + jj, g;
                if (d.yper) { g = gj < 0 ? gj + Ny : gj; while (g >= Ny) g -= Ny; }
                else g = gj < 0 ? 0 : (gj >= Ny ? Ny - 1 : gj);
                offp[q] = g * Nx + gi;
            }
        }
    }
    auto issue_phi = [&](int k) {   // phi plane k into phi slot (k - k0 + 1) % 5
        if constexpr (CORR) {
            const int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k), slot = (k - k0 + 1) % 5;
#pragma unroll
            for (int q = 0; q < PERP; ++q)
                if (offp[q] >= 0) cp_async<8>(&smp[slot][2 * (threadIdx.x + q * NT)], a.phi + kw * plane + offp[q]);
        }
    };
    auto issue_z = [&](int k) {   // the z metrics of plane k (k0 <= k < kend) into zmr[(k - k0) & 3]
        if (threadIdx.x < ZPAIRS / 2) cp_async<8>(&zmr[(k - k0) & 3][2 * threadIdx.x], a.zm8 + ZPAIRS * k + 2 * threadIdx.x);
    };
    auto issue = [&](int slot, int k) {
        int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k);
        const int kb = kw * plane;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (off[q] < 0) continue;
            const int o = kb + off[q], e = 2 * (threadIdx.x + q * NT);
            cp_async<8>(&sm[0][slot][e], U + o);
            cp_async<8>(&sm[2][slot][e], W + o);
            if (!ghost[q]) {
                cp_async<8>(&sm[1][slot][e], V + o);
                if (LES) cp_async<8>(&sm[NF - 1][slot][e], NU + o);
            }
        }
    };
    auto fix = [&](int slot, int k) {
        if constexpr (CORR) {   // project_velocity of the previous stage (k_correct's arithmetic, lane by lane)
            const int kw = k < 0 ? k + Nz : (k >= Nz ? k - Nz : k);
            const int p0 = (k - k0 + 1) % 5, p1 = (k - k0 + 2) % 5;
            const float iz = a.mz.idf[kw];
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                if (off[q] < 0) continue;
                const int e = 2 * (threadIdx.x + q * NT);
                const float2 pc = *reinterpret_cast<const float2 *>(&smp[p0][pix[q]]);
                const float pn = smp[p0][pix[q] + 2];
                const float2 pz = *reinterpret_cast<const float2 *>(&smp[p1][pix[q]]);
                float2 *u2 = reinterpret_cast<float2 *>(&sm[0][slot][e]), *w2 = reinterpret_cast<float2 *>(&sm[2][slot][e]);
                float2 u = *u2, w = *w2;
                u.x = u.x - (pc.y - pc.x) * a.inv_dx; u.y = u.y - (pn - pc.y) * a.inv_dx;
                w.x = w.x - (pz.x - pc.x) * iz; w.y = w.y - (pz.y - pc.y) * iz;
                *u2 = u; *w2 = w;
                if (iyq[q] != 0.0f) {
                    const float2 py = *reinterpret_cast<const float2 *>(&smp[p0][pix[q] + PXP]);
                    float2 *v2 = reinterpret_cast<float2 *>(&sm[1][slot][e]);
                    float2 v = *v2;
                    v.x = v.x - (py.x - pc.x) * iyq[q]; v.y = v.y - (py.y - pc.y) * iyq[q];
                    *v2 = v;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (off[q] < 0 || !ghost[q]) continue;
            const int e = 2 * (threadIdx.x + q * NT);
            float2 *u2 = reinterpret_cast<float2 *>(&sm[0][slot][e]), *w2 = reinterpret_cast<float2 *>(&sm[2][slot][e]);
            const float2 u = *u2, w = *w2;
            *u2 = make_float2(-u.x, -u.y);
            *w2 = make_float2(-w.x, -w.y);
            *reinterpret_cast<float2 *>(&sm[1][slot][e]) = make_float2(0.0f, 0.0f);
            if (LES) *reinterpret_cast<float2 *>(&sm[NF - 1][slot][e]) = make_float2(0.0f, 0.0f);
        }
    };
    F2 ubr[3];
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj) {
        int gj = min(j, Ny - 1) + dj;
        float sgn = 1.0f;
        if (d.yper) { gj = gj < 0 ? gj + Ny : (gj >= Ny ? gj - Ny : gj); }
        else if (gj < 0 || gj >= Ny) { gj = gj < 0 ? 0 : Ny - 1; sgn = -1.0f; }
        ubr[dj + 1] = F2(sgn * __ldg(a.ub + gj));
    }
    AxisLocal<F2> Y;
    Y.load(a.my, min(j, Ny - 1));
    RowProfile<F2> R;
    R.load(ubr, Y, row_wd<F2, WM>(a, j));

    issue(0, k0 - 1); issue(1, k0); issue(2, k0 + 1);
    issue_phi(k0 - 1); issue_phi(k0); issue_phi(k0 + 1); issue_phi(k0 + 2); issue_phi(k0 + 3);
    issue_z(k0);
    if (k0 + 1 < kend) issue_z(k0 + 1);
    cp_async_commit();
    cp_async_wait_all();
    if (CORR) __syncthreads();   // phi elements copied by other threads
    fix(0, k0 - 1); fix(1, k0); fix(2, k0 + 1);
    __syncthreads();
    const int cloc = (ty + 1) * PX + 2 + 2 * tx;
    for (int k = k0; k < kend; ++k) {
        const bool more = k + 2 <= kend;
        const int snext = (k - k0 + 3) & 3;
        if (more) { issue(snext, k + 2); issue_phi(k + 4); }
        if (k + 2 < kend) issue_z(k + 2);
        cp_async_commit();
        const int sm_ = (k - k0) & 3, s0 = (k - k0 + 1) & 3, sp = (k - k0 + 2) & 3;
        if (active) {
            TileQ2<PX> q;
            q.c = cloc;
            q.u[0] = sm[0][sm_]; q.u[1] = sm[0][s0]; q.u[2] = sm[0][sp];
            q.v[0] = sm[1][sm_]; q.v[1] = sm[1][s0]; q.v[2] = sm[1][sp];
            q.w[0] = sm[2][sm_]; q.w[1] = sm[2][s0]; q.w[2] = sm[2][sp];
            q.n[0] = sm[NF - 1][sm_]; q.n[1] = sm[NF - 1][s0]; q.n[2] = sm[NF - 1][sp];
            stage_pair<LES, WM, HYB>(a, q, Y, R, zmr[(k - k0) & 3], tau_x, tau_z, sc, i, j, k, uo, vo, wo, f1u, f1v, f1w,
                                     us, vs, wsf, rhs_only);
        }
        cp_async_wait_all();
        if (more) fix(snext, k + 2);   // CORR: phi k+2 and k+3 were copied one and two iterations ago
        __syncthreads();
    }
}
template <bool LES, bool WM, int TY = 8, bool HYB = false, bool CORR = false>
__global__ void __launch_bounds__(32 * TY, 512 / (32 * TY)) k_tiled2(StepArgs<float> a, const float *__restrict__ U, const float *__restrict__ V,
                                                   const float *__restrict__ W, const float *__restrict__ NU,
                                                   const double *__restrict__ tau_x, const double *__restrict__ tau_z,
                                                   StageCoef sc, int kc, float *__restrict__ uo, float *__restrict__ vo,
                                                   float *__restrict__ wo, float *__restrict__ f1u, float *__restrict__ f1v,
                                                   float *__restrict__ f1w, float *__restrict__ us, float *__restrict__ vs,
                                                   float *__restrict__ wsf, float *__restrict__ rhs_only) {
    pdl_enter();
    k_tiled2_body<LES, WM, TY, HYB, CORR>(HwBlock(), a, U, V, W, NU, tau_x, tau_z, sc, kc, uo, vo, wo, f1u, f1v, f1w, us, vs, wsf, rhs_only);
}

}  // namespace dfdm
