// FP64 per-particle and per-node physics of the step: Kirchhoff stress,
// trial p/q, failure surface, Drucker-Prager return map. Each function names
// the reference lines (simulation/mpm_kernels.cuh) whose mathematics it
// carries out.
#pragma once

#include "device_common.cuh"
#include "svd3.cuh"

namespace icempm {

__device__ __forceinline__ double det3(const double a[3][3]) {
    return a[0][0] * (a[1][1] * a[2][2] - a[2][1] * a[1][2])
         - a[1][0] * (a[0][1] * a[2][2] - a[2][1] * a[0][2])
         + a[2][0] * (a[0][1] * a[1][2] - a[1][1] * a[0][2]);
}

// b = F F^T
__device__ __forceinline__ void ffT(const double F[3][3], double b[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) b[i][j] = F[i][0] * F[j][0] + F[i][1] * F[j][1] + F[i][2] * F[j][2];
}

// KirchhoffStress_Wolper (mpm_kernels.cuh:547-557):
// tau = mu J^(-2/3) dev(F F^T) + kappa/2 (J^2 - 1) I
__device__ __forceinline__ void kirchhoff_wolper(const DevParams& P, const double F[3][3], double tau[3][3]) {
    double Je = det3(F);
    double b[3][3];
    ffT(F, b);
    double tr3 = (b[0][0] + b[1][1] + b[2][2]) / 3;
    double s = P.mu * rcbrt(Je * Je);
    double hyd = P.kappa * 0.5 * (Je * Je - 1.);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) tau[i][j] = s * (b[i][j] - (i == j ? tr3 : 0.0)) + (i == j ? hyd : 0.0);
}

// Water (mpm_kernels.cuh:559-566): kappa (1 - J^-3), times I
__device__ __forceinline__ double water_pressure(const DevParams& P, double J) {
    return P.kappa * (1. - pow(J, -3.0));
}

// ComputePQ (mpm_kernels.cuh:477-484); PP: DevParams or DPParams
template <class PP>
__device__ __forceinline__ void trial_pq(const PP& P, const double F[3][3], double& Je, double& p_tr,
                                         double& q_tr) {
    Je = det3(F);
    double Jsq = Je * Je;
    p_tr = -(0.5 * P.kappa) * (Jsq - 1.);
    double b[3][3];
    ffT(F, b);
    double tr3 = (b[0][0] + b[1][1] + b[2][2]) / 3;
    double sq = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double d = b[i][j] - (i == j ? tr3 : 0.0);
            sq += d * d;
        }
    q_tr = kCoeff1 * P.mu * rcbrt(Jsq) * sqrt(sq);
}

// GetParametersForGrain + CheckIfPointIsInsideFailureSurface
// (mpm_kernels.cuh:434-474). True if the point crushes now.
__device__ __forceinline__ bool outside_failure_surface(const DevParams& P, short grain, double p_tr, double q_tr) {
    const double var2 = 1.0 + P.grain_var * 0.033 * (-15 + (grain + 3) % 30);
    const double var3 = 1.0 + P.grain_var * 0.1 * (-10 + (grain + 4) % 11);
    const double pmax = P.pmax;
    const double pmin = -P.tensile;
    const double qmax = P.shear * var3;
    const double pmin2 = -P.tensile2 * var2;
    const double beta = P.beta;
    if (p_tr < 0) {
        if (p_tr < pmin2) return true;
        double q0 = 2 * sqrt(-pmax * pmin) * qmax / (pmax - pmin);
        double k = -q0 / pmin2;
        return q_tr > k * (p_tr - pmin2);
    }
    const double mSq = (4 * qmax * qmax * (1 + 2 * beta)) / ((pmax - pmin) * (pmax - pmin));
    double y = (1. + 2. * beta) * q_tr * q_tr + mSq * (p_tr + beta * pmax) * (p_tr - pmax);
    return y > 0;
}

// F = U diag(d) V^T
__device__ __forceinline__ void compose_usv(const double U[3][3], const double d[3], const double V[3][3],
                                            double F[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            F[i][j] = U[i][0] * d[0] * V[j][0] + U[i][1] * d[1] * V[j][1] + U[i][2] * d[2] * V[j][2];
}

// The material constants the return map reads (a small by-value copy for
// out-of-line callers).
struct DPParams {
    double mu, kappa, pmax, tensile, shear, tan_phi;
};

__device__ __forceinline__ DPParams dp_params(const DevParams& P) {
    DPParams d;
    d.mu = P.mu; d.kappa = P.kappa; d.pmax = P.pmax; d.tensile = P.tensile; d.shear = P.shear; d.tan_phi = P.tan_phi;
    return d;
}

// ------------------------------------------- return map without an SVD
//
// The projected deformation gradient is an isotropic function of b = F F^T:
// with F = U diag(s) V^T, the map's U diag(s') V^T equals B R, where R = U V^T
// is the rotation of F's polar decomposition and B = U diag(s') U^T:
//   apex:   B = c I                          (all s' = c)
//   yield:  B = sqrt(alpha dev(b) + mean I)  (s'^2 = alpha (s^2 - mean) + mean)
// R and the square root come from Newton iterations (Higham, "Computing the
// polar decomposition - with applications", 1986; Denman and Beavers, "The
// matrix sign function and computations in systems", 1976), which converge
// quadratically: 3-4 steps for the strains of crushed ice, each one 3x3
// inverse. The SVD of the same matrix is 24 Jacobi rotations and 3 Givens
// rotations, each with a square root and a division in a serial chain, and
// that chain is the kernel's time (the crushed points rarely fill the chip):
// 0.7 % of 500,000 points crushed, mixed return map with its launch 16.4 ->
// 12.5 us per substep; a 3,001-point block's substep 31 -> 27 us. Error of F
// against the map in 40 digits, strains of 1e-6 to 0.4, apex and yield: at most
// 5e-16, the 64-bit SVD form's 1.8e-15.

__device__ __forceinline__ double tval(double x) { return x; }

template <class T>
__device__ __forceinline__ T cof_det(const T X[3][3], T cof[3][3]) {
    cof[0][0] = X[1][1] * X[2][2] - X[1][2] * X[2][1];
    cof[0][1] = X[1][2] * X[2][0] - X[1][0] * X[2][2];
    cof[0][2] = X[1][0] * X[2][1] - X[1][1] * X[2][0];
    cof[1][0] = X[0][2] * X[2][1] - X[0][1] * X[2][2];
    cof[1][1] = X[0][0] * X[2][2] - X[0][2] * X[2][0];
    cof[1][2] = X[0][1] * X[2][0] - X[0][0] * X[2][1];
    cof[2][0] = X[0][1] * X[1][2] - X[0][2] * X[1][1];
    cof[2][1] = X[0][2] * X[1][0] - X[0][0] * X[1][2];
    cof[2][2] = X[0][0] * X[1][1] - X[0][1] * X[1][0];
    return X[0][0] * cof[0][0] + X[0][1] * cof[0][1] + X[0][2] * cof[0][2];
}

// A step that moved the iterate by less than this leaves an error of its
// square, below the last bit; EXTRA more steps let a derivative that is
// carried along converge too.
constexpr double kNewtonDelta2 = 1e-18;
constexpr int kNewtonSteps = 12;

// R of F = S R (S symmetric positive); false if the iteration has not converged.
template <int EXTRA, class T>
__device__ __forceinline__ bool polar_rotation(const T F[3][3], T R[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) R[i][j] = F[i][j];
    int left = EXTRA;
    bool ok = false;
#pragma unroll 1
    for (int it = 0; it < kNewtonSteps; it++) {
        T cof[3][3];
        const T det = cof_det(R, cof);
        const T s = T(0.5) / det;
        double d2 = 0;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const T x = T(0.5) * R[i][j] + s * cof[i][j];
                const double d = tval(x) - tval(R[i][j]);
                d2 += d * d;
                R[i][j] = x;
            }
        if (d2 < kNewtonDelta2) {
            ok = true;
            if (left-- == 0) break;
        }
    }
    return ok;
}

// Inverse of the symmetric matrix {00, 01, 02, 11, 12, 22}, halved.
template <class T>
__device__ __forceinline__ void half_inv_sym(const T a[6], T r[6]) {
    const T c0 = a[3] * a[5] - a[4] * a[4], c1 = a[2] * a[4] - a[1] * a[5], c2 = a[1] * a[4] - a[2] * a[3];
    const T s = T(0.5) / (a[0] * c0 + a[1] * c1 + a[2] * c2);
    r[0] = s * c0; r[1] = s * c1; r[2] = s * c2;
    r[3] = s * (a[0] * a[5] - a[2] * a[2]);
    r[4] = s * (a[1] * a[2] - a[0] * a[4]);
    r[5] = s * (a[0] * a[3] - a[1] * a[1]);
}

// Square root of the symmetric positive matrix a (six entries as above).
template <int EXTRA, class T>
__device__ __forceinline__ bool sqrt_sym(const T a[6], T Y[6]) {
    T Z[6];
#pragma unroll
    for (int k = 0; k < 6; k++) { Y[k] = a[k]; Z[k] = T((k == 0 || k == 3 || k == 5) ? 1.0 : 0.0); }
    int left = EXTRA;
    bool ok = false;
#pragma unroll 1
    for (int it = 0; it < kNewtonSteps; it++) {
        T yi[6], zi[6];
        half_inv_sym(Y, yi);
        half_inv_sym(Z, zi);
        double d2 = 0;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const T y = T(0.5) * Y[k] + zi[k];
            const double d = tval(y) - tval(Y[k]);
            d2 += d * d;
            Y[k] = y;
            Z[k] = T(0.5) * Z[k] + yi[k];
        }
        if (d2 < kNewtonDelta2) {
            ok = true;
            if (left-- == 0) break;
        }
    }
    return ok && tval(Y[0]) > 0;
}

// F <- B R with B = c I (apex), or B^2 = alpha dev(b) + mean I. False (F
// unchanged) for a strongly compressed or inverted F and where an iteration
// does not converge: the caller then takes the SVD.
constexpr double kPolarMinDet = 0.05;
template <int EXTRA, class T>
__device__ __forceinline__ bool project_polar(T F[3][3], double J, bool apex, T c, T alpha, const T b[3][3], T mean) {
    if (!(J > kPolarMinDet)) return false;
    T R[3][3];
    if (!polar_rotation<EXTRA>(F, R)) return false;
    if (apex) {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) F[i][j] = c * R[i][j];
        return true;
    }
    const T a[6] = {alpha * (b[0][0] - mean) + mean, alpha * b[0][1], alpha * b[0][2],
                    alpha * (b[1][1] - mean) + mean, alpha * b[1][2], alpha * (b[2][2] - mean) + mean};
    T Y[6];
    if (!sqrt_sym<EXTRA>(a, Y)) return false;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        F[0][j] = Y[0] * R[0][j] + Y[1] * R[1][j] + Y[2] * R[2][j];
        F[1][j] = Y[1] * R[0][j] + Y[3] * R[1][j] + Y[4] * R[2][j];
        F[2][j] = Y[2] * R[0][j] + Y[4] * R[1][j] + Y[5] * R[2][j];
    }
    return true;
}

// ComputeSVD (mpm_kernels.cuh:486-492) + Wolper_Drucker_Prager (:494-544)
// for a crushed point. p0 is the apex shift (DP_threshold_p, or the
// per-particle cohesion / tan(phi)). K selects the arithmetic: SvdF32 the
// reference's 32-bit SVD, bit for bit; SvdF64 the polar form above, with the
// 64-bit SVD for the deformations it leaves.
template <class K, class PP>
__device__ __forceinline__ void drucker_prager_return(const PP& P, double F[3][3], double& Jp_inv,
                                                      double Je_tr, double p_tr, double q_tr, double p0) {
    typedef typename K::T T;
    const double mu = P.mu, kappa = P.kappa;
    const bool apex = p_tr < -p0 || Jp_inv < 1;
    const double Je_tr_sq = Je_tr * Je_tr;
    double c = 0, coef = 0;
    if (apex) {
        // tension cut-off / recompaction: project to the apex
        const double p_new = -p0;
        const double Je_new = sqrt(-2. * p_new / kappa + 1.);
        c = cbrt(Je_new);
        Jp_inv *= Je_new / Je_tr;
    } else {
        double q_n_1;
        if (p_tr > P.pmax) {
            q_n_1 = 0;
        } else {
            const double q_from_dp = (p_tr + p0) * P.tan_phi;
            const double pmin = -P.tensile;
            const double q_from_failure_surface = 2 * sqrt((P.pmax - p_tr) * (p_tr - pmin)) * P.shear / (P.pmax - pmin);
            q_n_1 = fmin(q_from_failure_surface, q_from_dp);
        }
        if (!(q_tr >= q_n_1)) return;
        coef = (q_n_1 * kCoeff1Inv) * cbrt(Je_tr_sq) / mu;
    }
    if (sizeof(T) == sizeof(double)) {
        double b[3][3];
        ffT(F, b);
        const double mean = (b[0][0] + b[1][1] + b[2][2]) / 3;
        const double d0 = b[0][0] - mean, d1 = b[1][1] - mean, d2 = b[2][2] - mean;
        const double dn = sqrt(d0 * d0 + d1 * d1 + d2 * d2 +
                               2 * (b[0][1] * b[0][1] + b[0][2] * b[0][2] + b[1][2] * b[1][2]));
        if (project_polar<0>(F, Je_tr, apex, c, dn > 0 ? coef / dn : 0.0, b, mean)) return;
    }
    T A[3][3], Uk[3][3], Sk[3], Vk[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) A[i][j] = (T)F[i][j];
    svd3x3<K>(A, Uk, Sk, Vk);
    double U[3][3], V[3][3], sig2[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double s = (double)Sk[i];
        sig2[i] = s * s;
#pragma unroll
        for (int j = 0; j < 3; j++) { U[i][j] = (double)Uk[i][j]; V[i][j] = (double)Vk[i][j]; }
    }
    double sig[3] = {c, c, c};
    if (!apex) {
        const double mean = (sig2[0] + sig2[1] + sig2[2]) / 3;
        const double sfac = mu * rcbrt(Je_tr_sq);
        double sh[3];
#pragma unroll
        for (int i = 0; i < 3; i++) sh[i] = sfac * (sig2[i] - mean);      // v_s_hat_tr
        const double nrm = sqrt(sh[0] * sh[0] + sh[1] * sh[1] + sh[2] * sh[2]);
#pragma unroll
        for (int i = 0; i < 3; i++) sig[i] = sqrt(coef * (nrm > 0 ? sh[i] / nrm : 0.0) + mean);
    }
    compose_usv(U, sig, V, F);
}

}  // namespace icempm
