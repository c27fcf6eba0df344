// adi_device.cuh -- device-side building blocks of the ADI time step.
//
// The arithmetic policy `X` selects between
//   X = true : every +,-,*,/ is an explicitly rounded IEEE operation (__dadd_rn, ...), so
//              the compiler cannot fuse a*b+c, and each expression keeps the reference's
//              left-to-right order -> results bit-identical to the reference's host code;
//   X = false: plain operators, the compiler contracts into FMA (rounding-level changes).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace lss_gb300 {

template <bool X> struct ar;
template <> struct ar<true> {
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};
template <> struct ar<false> {
    template <typename T> static __device__ __forceinline__ T mul(T a, T b) { return a * b; }
    template <typename T> static __device__ __forceinline__ T add(T a, T b) { return a + b; }
    template <typename T> static __device__ __forceinline__ T sub(T a, T b) { return a - b; }
    template <typename T> static __device__ __forceinline__ T div(T a, T b) { return a / b; }
};

// Device view of one instance's time-invariant data (all arrays row-major, i*ny + j).
template <typename T> struct dev_instance {
    int nx, ny;
    T theta, zeta, gamma, delta, ni, rho, h1;
    const T *M, *P, *Z, *Mt, *Pt, *W, *C; // nx*ny each
    const T *D0, *E0, *F0;                 // nx each: D, E, F on the v = v_lo line
    const T *s_lo, *s_hi_neu, *v_hi;       // ny, ny, nx
    const int *imap, *jmap;                // nx, ny
    int ds;                                // 1: double-sweep line solves, 0: Thomas LU
};

// Stage selectors of the S-direction sweeps.
enum s_stage : int {
    S_STAGE1 = 1,    // rhs_intermed_1: explicit 9-point operator (all schemes)
    S_STAGE3_CS = 3, // Craig-Sneyd rhs_intermed_3
    S_STAGE3_MCS = 4,// modified Craig-Sneyd rhs_intermed_3
    S_STAGE4_HV = 5  // Hundsdorfer-Verwer rhs_intermed_4
};

// Right-hand side of an S-line at row t of line j, reference operation order.
//   S_STAGE1    : A = U
//   S_STAGE3_*  : A = U, B = Y1, Cc = Y2
//   S_STAGE4_HV : A = Y2, B = Y3
template <typename T, bool X, int STAGE>
__device__ __forceinline__ T s_rhs(const dev_instance<T> &d, int t, int j, const T *A, const T *B, const T *Cc,
                                    T a_low, T theta_z, T theta_p)
{
    using R = ar<X>;
    const int ny = d.ny;
    const int o = t * ny + j;
    const T one = T(1);
    if constexpr (STAGE == S_STAGE1) {
        // lss_heat_douglas_rachford_method.hpp:56-67
        const T gC = R::mul(d.gamma, d.C[o]);
        const T omt = R::sub(one, d.theta);
        const T *U = A;
        const T t1 = R::mul(gC, U[o - ny - 1]);
        const T t2 = R::mul(R::mul(omt, d.M[o]), U[o - ny]);
        const T t3 = R::mul(gC, U[o - ny + 1]);
        const T t4 = R::mul(d.Mt[o], U[o - 1]);
        const T t5 = R::mul(R::sub(R::sub(one, d.W[o]), R::mul(omt, d.Z[o])), U[o]);
        const T t6 = R::mul(d.Pt[o], U[o + 1]);
        const T t7 = R::mul(gC, U[o + ny - 1]);
        const T t8 = R::mul(R::mul(omt, d.P[o]), U[o + ny]);
        const T t9 = R::mul(gC, U[o + ny + 1]);
        return R::add(R::add(R::sub(R::add(R::add(R::add(R::sub(R::add(t1, t2), t3), t4), t5), t6), t7), t8), t9);
    } else if constexpr (STAGE == S_STAGE3_CS || STAGE == S_STAGE3_MCS) {
        // lss_heat_craig_sneyd_method.hpp:144-155; lss_heat_modified_craig_sneyd_method.hpp:147-164
        const T *U = A, *Y1 = B, *Y2 = Cc;
        T s = R::add(R::sub(R::add(R::mul(a_low, U[o - ny]), R::mul(theta_z, U[o])), R::mul(theta_p, U[o + ny])), Y1[o]);
        const T d1 = R::sub(Y2[o + ny + 1], U[o + ny + 1]);
        const T d2 = R::sub(Y2[o + ny - 1], U[o + ny - 1]);
        const T d3 = R::sub(Y2[o - ny + 1], U[o - ny + 1]);
        const T d4 = R::sub(Y2[o - ny - 1], U[o - ny - 1]);
        const T mix = R::add(R::sub(R::sub(d1, d2), d3), d4);
        s = R::add(s, R::mul(R::mul(R::mul(d.zeta, d.gamma), d.C[o]), mix));
        if constexpr (STAGE == S_STAGE3_MCS) {
            const T e1 = R::mul(d.M[o], R::sub(Y2[o - ny], U[o - ny]));
            const T e2 = R::mul(R::add(d.Z[o], d.W[o]), R::sub(Y2[o], U[o]));
            const T e3 = R::mul(d.P[o], R::sub(Y2[o + ny], U[o + ny]));
            const T e4 = R::mul(d.Mt[o], R::sub(Y2[o - 1], U[o - 1]));
            const T e5 = R::mul(d.Pt[o], R::sub(Y2[o + 1], U[o + 1]));
            s = R::add(s, R::mul(R::sub(d.zeta, d.theta), R::add(R::add(R::sub(R::sub(e1, e2), e3), e4), e5)));
        }
        return s;
    } else {
        // lss_heat_hundsdorfer_verwer_method.hpp:187-193
        const T *Y2 = A, *Y3 = B;
        return R::add(R::sub(R::add(R::mul(a_low, Y2[o - ny]), R::mul(theta_z, Y2[o])), R::mul(theta_p, Y2[o + ny])),
                      Y3[o]);
    }
}

// Weight of U_t in the explicit operator with differences along the S line, (M + P - Z) - W times ib, for
// the neighbours' weights ws = M~ ib and wn = P~ ib as they are stored: the row's sum is the reaction
// term r = (M + P - Z) + ((M~ + P~) - W), and the weight is formed from it.  Written as -W plus the reaction it is rounded by the same
// amount wherever W has the same exponent (W is a multiple of its last place, the reaction a constant), a
// reaction of up to eps W that adds up over the steps: SABR 12 x 3000 (W = 1.3e4) was 6.7e-12 off extended
// precision after 10 steps, so 1.5e-13.  A reaction of less than 2^20 last places does not get different
// roundings from the change of ib along the line; there the weight is rounded up or down in proportion (a
// hash of row t and column j is added below the last place of T).
template <typename T>
__device__ __forceinline__ T center_weight(double r, double ib, T ws, T wn, int t, int j)
{
    constexpr int digits = sizeof(T) == 8 ? 52 : 23;
    const double sum = static_cast<double>(ws) + static_cast<double>(wn);
    auto exponent = [](double x) { return (__double2hiint(x) >> 20) & 0x7ff; };
    const int last = exponent(sum) - digits; // exponent field of the last place of the sum in T
    if (exponent(r) + exponent(ib) - 1023 >= last + 20 || last <= 0) return static_cast<T>(fma(r, ib, -sum));
    unsigned h = static_cast<unsigned>(t) * 0x9e3779b1u + static_cast<unsigned>(j);
    h = (h ^ (h >> 16)) * 0x85ebca6bu;
    h = (h ^ (h >> 13)) * 0xc2b2ae35u;
    h ^= h >> 16;
    const double frac = __hiloint2double(0x3ff00000 | static_cast<int>(h >> 12), static_cast<int>(h << 20)) - 1.5; // [-1/2, 1/2)
    return static_cast<T>(fma(r, ib, frac * __hiloint2double(last << 20, 0)) - sum);
}

// ------------------------------------------------------------------------------------------
// boundary#1: explicit_heston_boundary_scheme::rhs (explicit_boundary.hpp:39-84) + v_hi column
// ------------------------------------------------------------------------------------------
// Results go to bcol0[i * stride], bcolN[i * stride]: the boundary columns of the v lines
// (stride 1) or, for the explicit Euler step, columns 0 and ny-1 of the next state (stride ny).
template <typename T, bool X>
__device__ __forceinline__ void boundary1_row(const dev_instance<T> &d, const T *U, int i, T *bcol0, T *bcolN, int stride)
{
    using R = ar<X>;
    const int nx = d.nx, ny = d.ny, N = nx - 1;
    const T one = T(1), two = T(2), three = T(3), four = T(4);
    const long long w = static_cast<long long>(i) * stride;
    if (i == 0) {
        bcol0[0] = d.s_lo[0];
    } else if (i == N) {
        const T D = d.D0[N], E = d.E0[N], F = d.F0[N];
        const T dlt = R::mul(R::mul(two, d.h1), d.s_hi_neu[0]);
        const T t1 = R::mul(R::add(R::sub(one, R::mul(R::mul(three, d.ni), E)), R::mul(d.rho, F)), U[N * ny]);
        const T t2 = R::mul(R::mul(R::mul(four, d.ni), E), U[N * ny + 1]);
        const T t3 = R::mul(R::mul(d.ni, E), U[N * ny + 2]);
        const T t4 = R::mul(R::mul(d.delta, dlt), D);
        bcol0[w] = R::sub(R::sub(R::add(t1, t2), t3), t4);
    } else {
        const T D = d.D0[i], E = d.E0[i], F = d.F0[i];
        const T t1 = R::mul(R::mul(-d.delta, D), U[(i - 1) * ny]);
        const T t2 = R::mul(R::add(R::sub(one, R::mul(R::mul(three, d.ni), E)), R::mul(d.rho, F)), U[i * ny]);
        const T t3 = R::mul(R::mul(d.delta, D), U[(i + 1) * ny]);
        const T t4 = R::mul(R::mul(d.ni, E), U[i * ny + 2]);
        const T t5 = R::mul(R::mul(R::mul(four, d.ni), E), U[i * ny + 1]);
        bcol0[w] = R::add(R::sub(R::add(R::add(t1, t2), t3), t4), t5);
    }
    bcolN[w] = d.v_hi[i];
}

// ------------------------------------------------------------------------------------------
// HV full-grid stage rhs_intermed_3 (lss_heat_hundsdorfer_verwer_method.hpp:146-171).
// ------------------------------------------------------------------------------------------
template <typename T, bool X>
__device__ __forceinline__ T hv3_value(const dev_instance<T> &d, const T *U, const T *Y1, const T *Y2, int o)
{
    using R = ar<X>;
    const int ny = d.ny;
    const T one = T(1);
    const T th = d.theta;
    const T M = d.M[o], Z = d.Z[o], P = d.P[o], W = d.W[o];
    const T t1 = R::mul(R::mul(-th, M), Y1[o - ny]);
    const T t2 = R::mul(R::add(one, R::mul(th, Z)), Y1[o]);
    const T t3 = R::mul(R::mul(th, P), Y1[o + ny]);
    const T t4 = R::mul(R::mul(th, M), U[o - ny]);
    const T t5 = R::mul(R::mul(th, Z), U[o]);
    const T t6 = R::mul(R::mul(th, P), U[o + ny]);
    const T d1 = R::sub(Y2[o + ny + 1], U[o + ny + 1]);
    const T d2 = R::sub(Y2[o + ny - 1], U[o + ny - 1]);
    const T d3 = R::sub(Y2[o - ny + 1], U[o - ny + 1]);
    const T d4 = R::sub(Y2[o - ny - 1], U[o - ny - 1]);
    const T t7 = R::mul(R::mul(R::mul(d.zeta, d.gamma), d.C[o]), R::add(R::sub(R::sub(d1, d2), d3), d4));
    const T e1 = R::mul(M, R::sub(Y2[o - ny], U[o - ny]));
    const T e2 = R::mul(R::add(W, Z), R::sub(Y2[o], U[o]));
    const T e3 = R::mul(P, R::sub(Y2[o + ny], U[o + ny]));
    const T e4 = R::mul(d.Mt[o], R::sub(Y2[o - 1], U[o - 1]));
    const T e5 = R::mul(d.Pt[o], R::sub(Y2[o + 1], U[o + 1]));
    const T t8 = R::mul(d.zeta, R::add(R::add(R::add(R::sub(e1, e2), e3), e4), e5));
    return R::add(R::add(R::add(R::sub(R::add(R::sub(R::add(t1, t2), t3), t4), t5), t6), t7), t8);
}

// ------------------------------------------------------------------------------------------
// boundary#2 (explicit_boundary.hpp:202-238): row 0 Dirichlet, row nx-1 from the
// one-sided Neumann extrapolation with the index_of-remapped column.
// ------------------------------------------------------------------------------------------
template <typename T, bool X> __device__ __forceinline__ void boundary2_column(const dev_instance<T> &d, T *V, int j)
{
    using R = ar<X>;
    const int nx = d.nx, ny = d.ny;
    const T two = T(2), three = T(3), four = T(4);
    V[j] = d.s_lo[j];
    const int jj = d.jmap[j];
    const int lri = nx - 1;
    V[lri * ny + j] = R::div(R::sub(R::sub(R::mul(four, V[(lri - 1) * ny + jj]), V[(lri - 2) * ny + jj]),
                                    R::mul(R::mul(two, d.h1), d.s_hi_neu[j])),
                             three);
}

} // namespace lss_gb300
