// heat1d.cu -- batched 1-D implicit heat / Black-Scholes theta scheme (include/lss_heat1d.h).
//
// Reference path (MichalSara99/linear_system_solvers):
//   heat_time_loop::run / run_with_stepping  (pde_solvers/one_dimensional/heat_type/
//                                             lss_1d_general_heat_equation_implicit_kernel.hpp:83-251)
//   heat_implicit_solver_method::solve        (.../solver_method/lss_heat_implicit_solver_method.hpp:245-262)
//     implicit_heat_scheme::rhs / rhs_source  (same file :37-176), split (:200-211)
//   thomas_lu_solver::kernel                  (sparse_solvers/tridiagonal/thomas_lu_solver/
//                                             lss_thomas_lu_solver.hpp:125-191, lss_thomas_lu_boundary.hpp:114-236)
//   double_sweep_solver::kernel               (sparse_solvers/tridiagonal/double_sweep_solver/
//                                             lss_double_sweep_solver.hpp:112-155, lss_double_sweep_boundary.hpp:88-190)
//
// Layout.  Instances are sorted by size and cut into groups of 32 of equal n; a group's arrays
// are interleaved (element t of lane l at t*32 + l), so each load of a warp (one thread per
// instance, all walking their line in step) is one 256-byte (FP64) line.  Slots of a group's
// point block (n*32 elements each):
//   REFERENCE: 0 A_, 1 B_, 2 D_ (scheme coefficients), 4 gamma / L, 5 sol / K, 6 U
//   FAST:      1 WB, 2 WD (right-hand-side weights of u_t, u_{t+1} scaled by the pivot reciprocal;
//              the weight of u_{t-1} is -(1-theta)/theta * M), 3 M (a_t / beta_t), 4 G (gamma_t),
//              5 KR (k / beta_t), 6 U, 7 Y (forward sweep); slot 0 keeps A_ (unused)
//   FAST, FP64, groups whose sweep is in registers (k_h1_reg; up to 512 points): 3 l, 4 g, 5 q (h1_setup_reg), 6 final U
// Per-step boundary values (2 per step) and source rows are interleaved the same way.  The
// whole time loop of an instance runs in one launch, on one thread (through memory) or on the
// lanes of one warp (in registers): there is no exchange between instances and no per-step
// launch.  A batch with lines for both sweeps has one launch of each, side by side.
#include "lss_heat1d.h"

#include "adi_common.hpp"
#include "adi_device.cuh"
#include "adi_threads.hpp"
#include "heat1d_schedule.hpp"

#include <algorithm>
#include <cmath>
#include <memory>
#include <numeric>
#include <thread>
#include <type_traits>
#include <vector>

namespace lss_gb300 {
namespace heat1d {

constexpr int LANES = 32;
constexpr int NSLOT = 8;
// Warps per CTA of the factorised sweep, one CTA per SM: 16 in FP32 (at most 128 registers per
// thread), 8 in FP64, whose 16-point rings take ~200 registers per thread (the deeper ring
// keeps more loads in flight in each warp, which is what the longest instances, running alone
// at the end of a batch, are bound by)
template <typename T> __host__ __device__ constexpr int h1_warps() { return sizeof(T) == 4 ? 16 : 8; }
// prefetch distance (points) of the forward sweep and of the back substitution.  At most 16:
// the loads past the last row stay in H1_PAD, those below row 0 in the group's block.
constexpr int H1_PF = 16;
constexpr int H1_PFB = 16;
// elements after the last group: the sweeps may load up to the prefetch distance + 1 points past a row
constexpr long long H1_PAD = (H1_PF + 2) * LANES;
enum { S_A = 0, S_B = 1, S_D = 2, S_M = 3, S_G = 4, S_K = 5, S_U = 6, S_Y = 7 };

// One instance (device).  Solver-type scalars are stored as double (exact).
struct h1lane {
    int inst;          // creation index
    int steps;         // nt - 1
    int lo_kind, hi_kind;
    int start, end;    // first / last solved row (FAST: filled by the set-up kernel)
    int has_src;
    int forward;
    int eval_i;        // value = (1 - eval_w) U[eval_i] + eval_w U[eval_i + 1]
    int pad;
    double eval_w;
    double theta, h, k; // theta, grid step 1/(n-1), time step
    double lo_lin, hi_lin; // transformed Robin linear values (constant in time)
    double bl, bh;      // FAST: coefficients of the boundary values in the first / last row
    double kb_lo, kb_hi; // FAST in registers: weight of the old boundary value (Dirichlet ends, see k_h1_setup_reg)
    long long init_off; // offset of the instance's initial condition (contiguous)
};

struct h1group {
    int n, lanes, steps;
    int reg;        // 1: the factorised sweep runs in registers (k_h1_reg); 2: in registers, row after row (k_h1_relay)
    long long pt;   // point block: slot s, point t, lane l at pt + (s*n + t)*32 + l
    long long bnd;  // boundary values: step s, side q (0 lower, 1 upper) at bnd + (s*2 + q)*32 + l
    long long src;  // source rows (steps + 1) x n, or -1
    long long all;  // every time level (steps + 1) x n, or -1
};

// One warp of the factorised sweep in registers: `sub` instances (lanes lane0 .. lane0 + sub - 1 of
// group g), W = 32 / 2^k lanes each, R rows per lane (W * R >= the solved rows), up to `steps` steps.
struct h1unit {
    int g, lane0, sub, W, R, steps;
};

template <typename T> struct h1params {
    const h1group *groups;
    h1lane *lanes;
    int ngroups;
    T *pt;
    const T *bnd;
    const T *src;
    T *all;
    const T *init;
    double *values;
    int *status;
    const h1unit *units;   // factorised sweep in registers: one warp per unit
    const int *warp_first; // factorised sweep through memory: the groups of warp w are
    const int *warp_group; // warp_group[warp_first[w] .. warp_first[w + 1])
    int nwarps, warps_per_cta; // (a CTA is launched with the warps that have groups)
};

__device__ __forceinline__ long long el(int t) { return static_cast<long long>(t) * LANES; }
__device__ __forceinline__ double h1_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float h1_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// ------------------------------------------------------------------------------------------
// Reference order (bit-identical to the reference's host policies)
// ------------------------------------------------------------------------------------------
// implicit_heat_scheme::rhs / rhs_source at row t (lss_heat_implicit_solver_method.hpp:37-176),
// `um, uc, up` the previous solution at t-1, t, t+1 and `s0, s1` the source at time and next
// time (has_src only).  Rows 0 and N are only formed for Neumann / Robin ends.
template <typename T>
__device__ __forceinline__ T ref_rhs(int t, int N, int lo_kind, int hi_kind, T A, T B, T D, T um, T uc, T up, T th,
                                     T h, T k, T lv, T ll, T hv, T hl, bool has_src, T s0, T s1)
{
    using R = ar<true>;
    const T one = T(1), two = T(2);
    const T omt = R::sub(one, th);
    T f;
    if (t == 0) {
        const T beta = R::mul(R::mul(two, h), lv);
        const T t1 = R::mul(R::mul(omt, beta), A);
        T t2;
        if (lo_kind == LSS_HEAT1D_ROBIN) {
            const T alpha = R::mul(R::mul(two, h), ll);
            t2 = R::mul(R::sub(one, R::mul(omt, R::sub(R::mul(two, B), R::mul(alpha, A)))), uc);
        } else {
            t2 = R::mul(R::sub(one, R::mul(R::mul(two, omt), B)), uc);
        }
        const T t3 = R::mul(R::mul(omt, R::add(A, D)), up);
        f = R::add(R::add(t1, t2), t3);
        if (has_src) f = R::add(R::add(f, R::mul(R::mul(th, k), s1)), R::mul(R::mul(omt, k), s0));
    } else if (t == N) {
        const T delta = R::mul(R::mul(two, h), hv);
        const T t1 = R::mul(R::mul(omt, R::add(A, D)), um);
        T t2;
        if (hi_kind == LSS_HEAT1D_ROBIN) {
            const T gamma = R::mul(R::mul(two, h), hl);
            t2 = R::mul(R::sub(one, R::mul(omt, R::add(R::mul(two, B), R::mul(gamma, D)))), uc);
        } else {
            t2 = R::mul(R::sub(one, R::mul(R::mul(two, omt), B)), uc);
        }
        const T t3 = R::mul(R::mul(omt, delta), D);
        f = R::sub(R::add(t1, t2), t3);
        if (has_src) f = R::add(R::add(f, R::mul(R::mul(th, k), s1)), R::mul(R::mul(omt, k), s0));
    } else {
        const T t1 = R::mul(R::mul(D, omt), up);
        const T t2 = R::mul(R::sub(one, R::mul(R::mul(two, B), omt)), uc);
        const T t3 = R::mul(R::mul(A, omt), um);
        f = R::add(R::add(t1, t2), t3);
        if (has_src) f = R::add(f, R::mul(k, R::add(R::mul(th, s1), R::mul(omt, s0))));
    }
    return f;
}

// split (lss_heat_implicit_solver_method.hpp:200-211)
template <typename T> __device__ __forceinline__ void ref_split(T th, T A, T B, T D, T &a, T &b, T &c)
{
    using R = ar<true>;
    a = R::mul(-th, A);
    b = R::add(T(1), R::mul(R::mul(T(2), th), B));
    c = R::mul(-th, D);
}

template <typename T, bool DS, int PF> __device__ __forceinline__ void h1_ref_body(const h1params<T> &p)
{
    using R = ar<true>;
    const int g = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
    const int lane = threadIdx.x % LANES;
    if (g >= p.ngroups) return;
    const h1group G = p.groups[g];
    if (lane >= G.lanes) return;
    const h1lane L = p.lanes[static_cast<long long>(g) * LANES + lane];
    const int n = G.n, N = n - 1;
    const long long NS = static_cast<long long>(n) * LANES;
    T *base = p.pt + G.pt + lane;
    const T *A = base + S_A * NS, *B = base + S_B * NS, *D = base + S_D * NS;
    T *GM = base + S_G * NS, *SL = base + S_K * NS, *U = base + S_U * NS;
    const T *BND = p.bnd + G.bnd + lane;
    const bool has_src = L.has_src != 0;
    const T *SRC = has_src ? p.src + G.src + lane : nullptr;
    T *ALL = G.all >= 0 ? p.all + G.all + lane : nullptr;
    const T th = T(L.theta), h = T(L.h), k = T(L.k), ll = T(L.lo_lin), hl = T(L.hi_lin);
    const T two = T(2), one = T(1);
    const int lo_kind = L.lo_kind, hi_kind = L.hi_kind;
    const int steps = L.steps;

    for (int t = 0; t < n; ++t) U[el(t)] = p.init[L.init_off + t];
    int row = L.forward ? 0 : steps;
    if (ALL)
        for (int t = 0; t < n; ++t) ALL[(static_cast<long long>(row) * n + t) * LANES] = U[el(t)];

    for (int s = 0; s < steps; ++s) {
        const T lv = BND[el(2 * s)], hv = BND[el(2 * s + 1)];
        const T *S0 = has_src ? SRC + static_cast<long long>(s) * NS : nullptr;
        const T *S1 = has_src ? S0 + NS : nullptr;
        auto rhs_v = [&](int t, T Av, T Bv, T Dv, T um, T uc, T up) -> T {
            return ref_rhs<T>(t, N, lo_kind, hi_kind, Av, Bv, Dv, um, uc, up, th, h, k, lv, ll, hv, hl, has_src,
                              has_src ? S0[el(t)] : T(0), has_src ? S1[el(t)] : T(0));
        };
        auto rhs = [&](int t, T um, T uc, T up) -> T { return rhs_v(t, A[el(t)], B[el(t)], D[el(t)], um, uc, up); };
        // rings of PF points: the loads of point t + PF are issued before point t is computed
        T ra[PF], rb[PF], rd[PF], ru[PF];
        auto load_pt = [&](int j, int t) {
            ra[j] = A[el(t)];
            rb[j] = B[el(t)];
            rd[j] = D[el(t)];
            ru[j] = t < N ? U[el(t + 1)] : T(0);
        };
        if (!DS) {
            // thomas_lu_solver::kernel: init_coefficients, forward loops (fused: each value is
            // computed as in the reference's separate beta/gamma and solution loops), back substitution
            const int start = lo_kind == LSS_HEAT1D_DIRICHLET ? 1 : 0;
            const int end = hi_kind == LSS_HEAT1D_DIRICHLET ? n - 2 : n - 1;
            T um = start ? U[el(0)] : T(0), uc = U[el(start)], up = U[el(start + 1)];
            T a, b, c;
            ref_split(th, A[el(start)], B[el(start)], D[el(start)], a, b, c);
            const T f0 = rhs(start, um, uc, up);
            T beta, gam, z;
            if (lo_kind == LSS_HEAT1D_DIRICHLET) {
                beta = b;
                gam = R::div(c, beta);
                z = R::div(R::sub(f0, R::mul(a, lv)), beta);
            } else {
                const T cst = R::mul(R::mul(two, h), lv);
                beta = lo_kind == LSS_HEAT1D_ROBIN ? R::add(b, R::mul(a, R::mul(R::mul(two, h), ll))) : b;
                gam = R::div(R::add(a, c), beta);
                z = R::div(R::sub(f0, R::mul(a, cst)), beta);
            }
            GM[el(start)] = gam;
            SL[el(start)] = z;
            T sol = z;
#pragma unroll
            for (int j = 0; j < PF; ++j)
                if (start + 1 + j < end) load_pt(j, start + 1 + j);
            for (int tb = start + 1; tb < end; tb += PF) {
#pragma unroll
                for (int j = 0; j < PF; ++j) {
                    const int t = tb + j;
                    if (t < end) {
                        const T Av = ra[j], Bv = rb[j], Dv = rd[j], un = ru[j];
                        if (t + PF < end) load_pt(j, t + PF);
                        um = uc;
                        uc = up;
                        up = un;
                        ref_split(th, Av, Bv, Dv, a, b, c);
                        const T f = rhs_v(t, Av, Bv, Dv, um, uc, up);
                        beta = R::sub(b, R::mul(a, gam));
                        gam = R::div(c, beta);
                        sol = R::div(R::sub(f, R::mul(a, sol)), beta);
                        GM[el(t)] = gam;
                        SL[el(t)] = sol;
                    }
                }
            }
            // final_coefficients at the last solved row
            um = uc;
            uc = up;
            up = end < N ? U[el(end + 1)] : T(0);
            ref_split(th, A[el(end)], B[el(end)], D[el(end)], a, b, c);
            const T fe = rhs(end, um, uc, up);
            T an, bn, rn;
            if (hi_kind == LSS_HEAT1D_DIRICHLET) {
                an = a;
                bn = b;
                rn = R::sub(fe, R::mul(c, hv));
            } else {
                const T cst = R::mul(R::mul(two, h), hv);
                an = R::add(a, c);
                bn = hi_kind == LSS_HEAT1D_ROBIN ? R::sub(b, R::mul(c, R::mul(R::mul(two, h), hl))) : b;
                rn = R::add(fe, R::mul(c, cst));
            }
            const T beta_e = R::sub(bn, R::mul(an, gam));
            T x = R::div(R::sub(rn, R::mul(an, sol)), beta_e);
            U[el(end)] = x;
#pragma unroll
            for (int j = 0; j < PF; ++j)
                if (end - 1 - j >= start) {
                    ra[j] = SL[el(end - 1 - j)];
                    rb[j] = GM[el(end - 1 - j)];
                }
            for (int tb = end - 1; tb >= start; tb -= PF) {
#pragma unroll
                for (int j = 0; j < PF; ++j) {
                    const int t = tb - j;
                    if (t >= start) {
                        const T sv = ra[j], gv = rb[j];
                        if (t - PF >= start) {
                            ra[j] = SL[el(t - PF)];
                            rb[j] = GM[el(t - PF)];
                        }
                        x = R::sub(sv, R::mul(gv, x));
                        U[el(t)] = x;
                    }
                }
            }
            if (start == 1) U[el(0)] = lv;
            if (end == N - 1) U[el(N)] = hv;
        } else {
            // double_sweep_solver::kernel
            const int start = lo_kind == LSS_HEAT1D_DIRICHLET ? 1 : 0;
            const int end = hi_kind == LSS_HEAT1D_DIRICHLET ? n - 2 : n - 1;
            T Kp, Lp;
            T um = U[el(0)], uc = U[el(0)], up = U[el(1)];
            T a, b, c;
            if (lo_kind == LSS_HEAT1D_DIRICHLET) {
                Kp = lv;
                Lp = T(0);
            } else {
                ref_split(th, A[el(0)], B[el(0)], D[el(0)], a, b, c);
                const T f0 = rhs(0, T(0), uc, up);
                const T den = lo_kind == LSS_HEAT1D_ROBIN ? R::add(b, R::mul(R::mul(R::mul(a, h), two), ll)) : b;
                Kp = R::div(R::sub(f0, R::mul(R::mul(R::mul(a, h), two), lv)), den);
                Lp = R::div(R::mul(T(-1), R::add(a, c)), den);
            }
            SL[el(0)] = Kp;
            GM[el(0)] = Lp;
            T Kq = T(0), Lq = T(0); // K_{N-1}, L_{N-1} when the loop ends at N
#pragma unroll
            for (int j = 0; j < PF; ++j)
                if (1 + j <= end) load_pt(j, 1 + j);
            for (int tb = 1; tb <= end; tb += PF) {
#pragma unroll
                for (int j = 0; j < PF; ++j) {
                    const int t = tb + j;
                    if (t <= end) {
                        const T Av = ra[j], Bv = rb[j], Dv = rd[j], un = ru[j];
                        if (t + PF <= end) load_pt(j, t + PF);
                        um = uc;
                        uc = up;
                        up = un;
                        ref_split(th, Av, Bv, Dv, a, b, c);
                        const T f = rhs_v(t, Av, Bv, Dv, um, uc, up);
                        const T tmp = R::add(b, R::mul(a, Lp));
                        const T Ln = R::div(R::mul(T(-1), c), tmp);
                        const T Kn = R::div(R::sub(f, R::mul(a, Kp)), tmp);
                        Kq = Kp;
                        Lq = Lp;
                        Kp = Kn;
                        Lp = Ln;
                        SL[el(t)] = Kn;
                        GM[el(t)] = Ln;
                    }
                }
            }
            T x;
            if (hi_kind == LSS_HEAT1D_DIRICHLET) {
                x = hv;
            } else {
                // loop ended at t = N: (Kp, Lp) = (K_N, L_N), (Kq, Lq) = (K_{N-1}, L_{N-1})
                const T cst = R::mul(R::mul(two, h), hv);
                const T den = hi_kind == LSS_HEAT1D_ROBIN
                                  ? R::sub(one, R::mul(Lp, R::sub(Lq, R::mul(R::mul(two, h), hl))))
                                  : R::sub(one, R::mul(Lp, Lq));
                x = R::div(R::add(R::mul(Lp, R::sub(Kq, cst)), Kp), den);
            }
            U[el(N)] = x;
#pragma unroll
            for (int j = 0; j < PF; ++j)
                if (N - 1 - j >= start) {
                    ra[j] = SL[el(N - 1 - j)];
                    rb[j] = GM[el(N - 1 - j)];
                }
            for (int tb = N - 1; tb >= start; tb -= PF) {
#pragma unroll
                for (int j = 0; j < PF; ++j) {
                    const int t = tb - j;
                    if (t >= start) {
                        const T kv = ra[j], lv2 = rb[j];
                        if (t - PF >= start) {
                            ra[j] = SL[el(t - PF)];
                            rb[j] = GM[el(t - PF)];
                        }
                        x = R::add(R::mul(lv2, x), kv);
                        U[el(t)] = x;
                    }
                }
            }
            if (start == 1) U[el(0)] = lv;
        }
        row += L.forward ? 1 : -1;
        if (ALL)
            for (int t = 0; t < n; ++t) ALL[(static_cast<long long>(row) * n + t) * LANES] = U[el(t)];
    }
    // value at the evaluation point and finiteness of the final solution
    int bad = 0;
    for (int t = 0; t < n; ++t) bad |= !isfinite(static_cast<double>(U[el(t)]));
    const int i = L.eval_i;
    p.values[L.inst] = (1.0 - L.eval_w) * static_cast<double>(U[el(i)]) + L.eval_w * static_cast<double>(U[el(i + 1)]);
    p.status[L.inst] = bad;
}
// FP64 asks for two CTAs per SM: with 168 registers, the compiler's own choice, its spills cost 16 %
// (65536 Black-Scholes calls 1346 ms against 1164).
template <typename T, bool DS, int PF> __global__ void __launch_bounds__(128) k_h1_ref(const h1params<T> p) { h1_ref_body<T, DS, PF>(p); }
template <bool DS, int PF> __global__ void __launch_bounds__(128, 2) k_h1_ref64(const h1params<double> p) { h1_ref_body<double, DS, PF>(p); }

// ------------------------------------------------------------------------------------------
// FAST: one factorisation per instance (set-up), then per step one fused right-hand-side +
// forward sweep y_t = WB u_t + WD u_{t+1} + M (kap u_{t-1} - y_{t-1}) (+ boundary / source
// terms; kap = -(1-theta)/theta) and one back substitution x_t = y_t - G x_{t+1}.  Four loads,
// one store and four FP64 operations per point forward; two loads, one store and one FMA per
// point backward: 64 bytes per point-step in FP64.
// ------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ void h1_setup_reg(const h1params<T> &p, const h1group &G, h1lane &L, int lane);

template <typename T> __global__ void __launch_bounds__(128) k_h1_setup_fast(const h1params<T> p)
{
    const int g = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;
    const int lane = threadIdx.x % LANES;
    if (g >= p.ngroups) return;
    const h1group G = p.groups[g];
    if (lane >= G.lanes) return;
    h1lane &L = p.lanes[static_cast<long long>(g) * LANES + lane];
    if (G.reg == 1) {
        h1_setup_reg<T>(p, G, L, lane);
        return;
    }
    const int n = G.n, N = n - 1;
    const long long NS = static_cast<long long>(n) * LANES;
    T *base = p.pt + G.pt + lane;
    T *WA = base + S_A * NS, *WB = base + S_B * NS, *WD = base + S_D * NS;
    T *M = base + S_M * NS, *GG = base + S_G * NS, *KR = base + S_K * NS;
    const T th = T(L.theta), h2 = T(2) * T(L.h), k = T(L.k), ll = T(L.lo_lin), hl = T(L.hi_lin);
    const T one = T(1), omt = one - th;
    const int start = L.lo_kind == LSS_HEAT1D_DIRICHLET ? 1 : 0;
    const int end = L.hi_kind == LSS_HEAT1D_DIRICHLET ? N - 1 : N;
    T gam = T(0), bl = T(0), bh = T(0);
    for (int t = 0; t < n; ++t) {
        const T A = WA[el(t)], B = WB[el(t)], D = WD[el(t)];
        if (t < start || t > end) {
            WB[el(t)] = WD[el(t)] = M[el(t)] = GG[el(t)] = KR[el(t)] = T(0);
            continue;
        }
        const T a = -th * A, b = one + T(2) * th * B, c = -th * D;
        T beta, wa, wb, wd, m;
        if (t == start && start == 0) { // Neumann / Robin lower row
            beta = L.lo_kind == LSS_HEAT1D_ROBIN ? b + a * (h2 * ll) : b;
            gam = (a + c) / beta;
            const T rb = one / beta;
            wa = T(0);
            wb = (L.lo_kind == LSS_HEAT1D_ROBIN ? one - omt * (T(2) * B - h2 * ll * A) : one - T(2) * omt * B) * rb;
            wd = omt * (A + D) * rb;
            m = T(0);
            bl = (omt * h2 * A - a * h2) * rb;
            KR[el(t)] = k * rb;
        } else if (t == end && end == N) { // Neumann / Robin upper row
            const T an = a + c;
            const T bn = L.hi_kind == LSS_HEAT1D_ROBIN ? b - c * (h2 * hl) : b;
            beta = bn - an * gam;
            const T rb = one / beta;
            wa = omt * (A + D) * rb;
            wb = (L.hi_kind == LSS_HEAT1D_ROBIN ? one - omt * (T(2) * B + h2 * hl * D) : one - T(2) * omt * B) * rb;
            wd = T(0);
            m = an * rb;
            bh = (c * h2 - omt * h2 * D) * rb;
            gam = T(0);
            KR[el(t)] = k * rb;
        } else { // interior row (the first one after a Dirichlet end uses y_0 = lower value)
            beta = t == start ? b : b - a * gam;
            gam = c / beta;
            const T rb = one / beta;
            wa = omt * A * rb;
            wb = (one - T(2) * omt * B) * rb;
            wd = omt * D * rb;
            m = a * rb;
            if (t == end) bh = -c * rb; // Dirichlet upper end: - c_{N-1} v_hi / beta_{N-1}
            KR[el(t)] = k * rb;
        }
        (void)wa; // = kap * m, formed by the sweep
        WB[el(t)] = wb;
        WD[el(t)] = wd;
        M[el(t)] = m;
        GG[el(t)] = gam;
    }
    L.start = start;
    L.end = end;
    L.bl = static_cast<double>(bl);
    L.bh = static_cast<double>(bh);
}

// Time loop of group g in one warp.  Per step: the first solved row, the interior rows in
// blocks of PF (the loads of point t + PF are issued before point t is computed, from a ring of
// PF registers per array; loads past the last row stay inside the group's block and are never
// used), the last solved row, then the back substitution the same way downwards.  SRC: the
// batch has heat sources; KEEP: every time level is written out.
template <typename T, int PF, bool SRC, bool KEEP>
__device__ __forceinline__ void h1_fast_group(const h1params<T> p, const int g, const int lane)
{
    const h1group G = p.groups[g];
    if (lane >= G.lanes) return;
    const h1lane L = p.lanes[static_cast<long long>(g) * LANES + lane];
    const int n = G.n, N = n - 1;
    const int NS = n * LANES;
    T *base = p.pt + G.pt + lane;
    const T *__restrict__ WB = base + S_B * NS;
    const T *__restrict__ WD = base + S_D * NS;
    const T *__restrict__ M = base + S_M * NS;
    const T *__restrict__ GG = base + S_G * NS;
    const T *__restrict__ KR = base + S_K * NS;
    T *__restrict__ U = base + S_U * NS;
    T *__restrict__ Y = base + S_Y * NS;
    const T *BND = p.bnd + G.bnd + lane;
    const bool has_src = SRC && L.has_src != 0;
    const T *SRCP = has_src ? p.src + G.src + lane : nullptr;
    T *ALL = KEEP ? p.all + G.all + lane : nullptr;
    const T th = T(L.theta), omt = T(1) - th, bl = T(L.bl), bh = T(L.bh);
    const T kap = -omt / th; // -1 (Crank-Nicolson) or 0 (Euler), exact
    const bool cn = kap != T(0);
    const int start = L.start, end = L.end, steps = L.steps;
    const int S = LANES;

    for (int t = 0; t < n; ++t) U[t * S] = p.init[L.init_off + t];
    int row = L.forward ? 0 : steps;
    if (KEEP)
        for (int t = 0; t < n; ++t) ALL[(static_cast<long long>(row) * n + t) * S] = U[t * S];

    for (int s = 0; s < steps; ++s) {
        const T lv = BND[(2 * s) * S], hv = BND[(2 * s + 1) * S];
        const T *S0 = has_src ? SRCP + static_cast<long long>(s) * NS : nullptr;
        auto src_term = [&](int t) -> T {
            return has_src ? KR[t * S] * (th * S0[NS + t * S] + omt * S0[t * S]) : T(0);
        };
        // first solved row.  Every row's weight of u_{t-1} is kap * M_t (a_t = -theta A_t, so
        // (1 - theta) A_t / beta_t = kap a_t / beta_t, also in the Neumann / Robin end rows):
        // y_t = WB u_t + WD u_{t+1} + M (kap u_{t-1} - y_{t-1}), four loads per point
        T um = start ? U[0] : T(0);
        T uc = U[start * S];
        T up = U[(start + 1) * S];
        T yp = WB[start * S] * uc + WD[start * S] * up + M[start * S] * (kap * um - (start ? lv : T(0)));
        if (start == 0) yp += bl * lv;
        yp += src_term(start);
        Y[start * S] = yp;
        um = uc;
        uc = up;
        // interior rows start+1 .. end-1 as y_t = c_t - M_t y_{t-1}, c_t = WB u_t + WD u_{t+1}
        // - [CN] M_t u_{t-1} (+ source): c_t does not depend on the recurrence, so the dependent
        // chain through y is one FMA per point
        T rwb[PF], rwd[PF], rm[PF], rup[PF];
        int t = start + 1;
#pragma unroll
        for (int j = 0; j < PF; ++j) {
            const int q = (t + j) * S;
            rwb[j] = WB[q];
            rwd[j] = WD[q];
            rm[j] = M[q];
            rup[j] = U[q + S];
        }
        for (; t + PF <= end; t += PF) {
#pragma unroll
            for (int j = 0; j < PF; ++j) {
                const T wb = rwb[j], wd = rwd[j], m = rm[j], u1 = rup[j];
                const int q = (t + j + PF) * S;
                rwb[j] = WB[q];
                rwd[j] = WD[q];
                rm[j] = M[q];
                rup[j] = U[q + S];
                T c = h1_fma(-m, cn ? um : T(0), h1_fma(wd, u1, wb * uc));
                if (SRC) c += src_term(t + j);
                const T y = h1_fma(-m, yp, c);
                Y[(t + j) * S] = y;
                yp = y;
                um = uc;
                uc = u1;
            }
        }
#pragma unroll
        for (int j = 0; j < PF; ++j) {
            if (t + j < end) {
                T c = h1_fma(-rm[j], cn ? um : T(0), h1_fma(rwd[j], rup[j], rwb[j] * uc));
                if (SRC) c += src_term(t + j);
                const T y = h1_fma(-rm[j], yp, c);
                Y[(t + j) * S] = y;
                yp = y;
                um = uc;
                uc = rup[j];
            }
        }
        // last solved row
        T x = yp;
        if (end > start) {
            const int q = end * S;
            const T u1 = end < N ? U[q + S] : T(0);
            x = WB[q] * uc + WD[q] * u1 + M[q] * (kap * um - yp) + bh * hv;
            x += src_term(end);
        }
        U[end * S] = x;
        // back substitution end-1 .. start (loads down to PFB <= 16 rows below row start - 1 stay
        // inside the group's block: G and Y have at least 4n >= 16 rows of other slots below them)
        constexpr int PFB = H1_PFB;
        T ry[PFB], rg[PFB];
        t = end - 1;
#pragma unroll
        for (int j = 0; j < PFB; ++j) {
            const int q = (t - j) * S;
            ry[j] = Y[q];
            rg[j] = GG[q];
        }
        for (; t - PFB >= start - 1; t -= PFB) {
#pragma unroll
            for (int j = 0; j < PFB; ++j) {
                const T yv = ry[j], gv = rg[j];
                const int q = (t - j - PFB) * S;
                ry[j] = Y[q];
                rg[j] = GG[q];
                x = yv - gv * x;
                U[(t - j) * S] = x;
            }
        }
#pragma unroll
        for (int j = 0; j < PFB; ++j) {
            if (t - j >= start) {
                x = ry[j] - rg[j] * x;
                U[(t - j) * S] = x;
            }
        }
        if (start == 1) U[0] = lv;
        if (end == N - 1) U[N * S] = hv;
        row += L.forward ? 1 : -1;
        if (KEEP)
            for (int q = 0; q < n; ++q) ALL[(static_cast<long long>(row) * n + q) * S] = U[q * S];
    }
    int bad = 0;
    for (int q = 0; q < n; ++q) bad |= !isfinite(static_cast<double>(U[q * S]));
    const int i = L.eval_i;
    p.values[L.inst] = (1.0 - L.eval_w) * static_cast<double>(U[i * S]) + L.eval_w * static_cast<double>(U[(i + 1) * S]);
    p.status[L.inst] = bad;
}

// One CTA of h1_warps<T>() warps per SM (the register file holds one CTA); warp w runs the groups warp_group[warp_first[w] .. warp_first[w + 1]) placed by
// schedule_groups.
template <typename T, int PF, bool SRC, bool KEEP>
__global__ void __launch_bounds__(h1_warps<T>() * LANES, 1) k_h1_fast(const h1params<T> p)
{
    const int w = blockIdx.x * p.warps_per_cta + threadIdx.x / LANES;
    const int lane = threadIdx.x % LANES;
    asm volatile("griddepcontrol.launch_dependents;"); // the sweep in registers of the same run may start
    if (w >= p.nwarps) return;
    const int q1 = p.warp_first[w + 1];
    for (int q = p.warp_first[w]; q < q1; ++q) h1_fast_group<T, PF, SRC, KEEP>(p, p.warp_group[q], lane);
}

// ------------------------------------------------------------------------------------------
// FAST, FP64 instances whose rows fit a warp's registers (at most 512 points).
//
// With A = I - theta k L (the step's matrix) the theta scheme is
//   x = (1/theta) A^{-1} u - ((1-theta)/theta) u   (CN: 2 A^{-1} u - u; Euler: A^{-1} u),
// so the right-hand side needs no operator application: y_t = u_t - l_t y_{t-1},
// xi_t = y_t - g_t xi_{t+1}, x_t = q_t xi_t - kap u_t with l_t = a_t / beta_{t-1},
// g_t = c_t / beta_{t+1}, q_t = 1 / (theta beta_t): three operations per point.  The boundary
// values enter as the chain's incoming values: l of the first row times (new + kb old) (Dirichlet:
// l = theta a, kb = (1-theta)/theta; Neumann / Robin: l = -theta h2 A, kb = 0), likewise g of the
// last row.
//
// W lanes share an instance, R consecutive rows each, and keep l, g, q and u in registers for the
// whole time loop: no memory traffic per step but the two boundary values.  Each recurrence is run
// twice per lane (from zero for the lane's end value, then from the incoming value that a scan of
// the affine end maps over the lanes gives); the scan's products do not change with time and lie
// in shared memory.  FP64 cost per point and step: 5 + (2 log2 W + 1) / R warp instructions.
//
// What bounds it: the FP64 pipe (one warp instruction per 64 cycles and SM sub-partition, latency
// the same, so two warps per sub-partition saturate it).  Measured on 4096 uneven Black-Scholes
// calls (6.1e8 point-steps): 7.8 ms = 7.9e10 point-steps/s, 0.75 of the pipe at 6 instructions a
// point; the sweep through memory took 104 ms, the time of its longest line walked by one thread.
// ------------------------------------------------------------------------------------------
constexpr int H1_SCAN = 5; // log2(32)
constexpr int H1_RMAX = 16;    // rows per lane that fit the registers (l, g, u and the sweep's values)

// Launched behind the sweep through memory, a sweep in registers runs beside it (the two share no instance);
// it ends after it, so that its end is the run's.
__device__ __forceinline__ void end_of_run() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Factors of one instance per thread, in double, written over the group's slots: l -> S_M,
// g -> S_G, q -> S_K (zero on rows that are not solved).  Groups of larger lines keep k_h1_setup_fast.
template <typename T> __device__ __forceinline__ void h1_setup_reg(const h1params<T> &p, const h1group &G, h1lane &L, int lane)
{
    const int n = G.n, N = n - 1;
    const long long NS = static_cast<long long>(n) * LANES;
    T *base = p.pt + G.pt + lane;
    const T *A = base + S_A * NS, *B = base + S_B * NS, *D = base + S_D * NS;
    T *LF = base + S_M * NS, *GF = base + S_G * NS, *Q = base + S_K * NS;
    const double th = L.theta, h2 = 2.0 * L.h;
    const int start = L.lo_kind == LSS_HEAT1D_DIRICHLET ? 1 : 0;
    const int end = L.hi_kind == LSS_HEAT1D_DIRICHLET ? N - 1 : N;
    double ib = 0.0, c_prev = 0.0; // 1 / beta and c of the row before
    for (int t = 0; t < n; ++t) {
        if (t < start || t > end) {
            LF[el(t)] = GF[el(t)] = Q[el(t)] = T(0);
            continue;
        }
        const double At = A[el(t)], Bt = B[el(t)], Dt = D[el(t)];
        double a = -th * At, b = 1.0 + 2.0 * th * Bt, c = -th * Dt;
        if (t == 0) {
            if (L.lo_kind == LSS_HEAT1D_ROBIN) b += a * h2 * L.lo_lin;
            c += a;
            LF[el(t)] = static_cast<T>(-th * At * h2);
        }
        if (t == N) {
            if (L.hi_kind == LSS_HEAT1D_ROBIN) b -= c * h2 * L.hi_lin;
            GF[el(t)] = static_cast<T>(th * Dt * h2);
            a += c;
        }
        const double beta = t == start ? b : b - a * ib * c_prev;
        if (t > start) {
            LF[el(t)] = static_cast<T>(a * ib);
            GF[el(t - 1)] = static_cast<T>(c_prev / beta);
        } else if (start) {
            LF[el(t)] = static_cast<T>(th * a);
        }
        ib = 1.0 / beta;
        c_prev = c;
        Q[el(t)] = static_cast<T>(ib / th);
        if (t == end && end < N) GF[el(t)] = static_cast<T>(th * c);
    }
    L.start = start;
    L.end = end;
    L.kb_lo = start ? (1.0 - th) / th : 0.0;
    L.kb_hi = end < N ? (1.0 - th) / th : 0.0;
}

template <typename T, int R, bool SRC, bool KEEP>
__device__ __forceinline__ void h1_reg_unit(const h1params<T> &p, const h1unit un, T (*__restrict__ scan)[LANES],
                                            T (*__restrict__ sq)[LANES])
{
    const int wl = threadIdx.x & 31, W = un.W, li = wl & (W - 1), sub = wl / W;
    const unsigned all = 0xffffffffu;
    const h1group G = p.groups[un.g];
    const bool act = sub < un.sub;
    const int lane = un.lane0 + (act ? sub : 0); // idle sub-warps shadow the first instance and store nothing
    const h1lane L = p.lanes[static_cast<long long>(un.g) * LANES + lane];
    const int n = G.n, N = n - 1;
    const long long NS = static_cast<long long>(n) * LANES;
    T *base = p.pt + G.pt + lane;
    T *U = base + S_U * NS;
    const T *BND = p.bnd + G.bnd + lane;
    const bool has_src = SRC && L.has_src != 0;
    const T *SRCP = has_src ? p.src + G.src + lane : nullptr;
    T *ALL = KEEP ? p.all + G.all + lane : nullptr;
    const int start = L.start, end = L.end, steps = act ? L.steps : 0;
    const int t0 = start + li * R; // first row of this lane
    const bool low = li == 0, high = li == W - 1;
    const T s1w = T(L.theta * L.theta * L.k), s0w = T(L.theta * (1.0 - L.theta) * L.k); // A z = u + theta k (theta s1 + (1-theta) s0)
    const bool cn = L.theta != 1.0; // kap = 1 (Crank-Nicolson) or 0 (Euler)
    const T *init = p.init + L.init_off;

    T l[R], g[R], u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int t = t0 + r;
        const bool in = t <= end;
        l[r] = in ? base[S_M * NS + el(t)] : T(0);
        g[r] = in ? base[S_G * NS + el(t)] : T(-1); // rows past the last pass the upper value down
        u[r] = in ? init[t] : T(0);
        sq[r][wl] = in ? base[S_K * NS + el(t)] : T(0);
    }
    // products of the scan: level d multiplies the value of lane li -/+ 2^d by the product of the
    // end maps of the lanes li - 2^d + 1 .. li (li .. li + 2^d - 1)
    {
        T hf = T(1), hb = T(1);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            hf *= -l[r];
            hb *= -g[r];
        }
#pragma unroll
        for (int d = 0; d < H1_SCAN; ++d) {
            scan[d][wl] = hf;
            scan[H1_SCAN + d][wl] = hb;
            const T pf = __shfl_up_sync(all, hf, 1 << d, W), pb = __shfl_down_sync(all, hb, 1 << d, W);
            if (li >= (1 << d)) hf *= pf;
            if (li + (1 << d) < W) hb *= pb;
        }
    }
    __syncwarp();
    // boundary values: lane 0 of the instance carries the lower one, every other lane the upper one
    const int side = low ? 0 : 1;
    const T kb = T(low ? L.kb_lo : L.kb_hi);
    T bold = init[low ? 0 : N];
    T bnew = steps > 0 ? BND[side * LANES] : T(0);
    int row = L.forward ? 0 : L.steps;
    if (KEEP && act) {
        for (int t = li; t < n; t += W) ALL[(static_cast<long long>(row) * n + t) * LANES] = init[t];
    }
    for (int s = 0; s < un.steps; ++s) {
        const bool live = s < steps;
        const T bin = h1_fma(kb, bold, bnew);
        bold = live ? bnew : bold;
        const T bcur = bold; // the value stored on the boundary row of this level
        if (s + 1 < steps) bnew = BND[(2 * (s + 1) + side) * LANES];
        T f[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            f[r] = u[r];
            if (SRC) {
                const int t = t0 + r;
                if (has_src && live && t <= end) {
                    const T *S0 = SRCP + static_cast<long long>(s) * NS;
                    f[r] += s1w * S0[NS + el(t)] + s0w * S0[el(t)];
                }
            }
        }
        // forward recurrence
        T y = low ? bin : T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) y = h1_fma(-l[r], y, f[r]);
#pragma unroll
        for (int d = 0; d < H1_SCAN; ++d) {
            if ((1 << d) < W) {
                const T o = __shfl_up_sync(all, y, 1 << d, W);
                if (li >= (1 << d)) y = h1_fma(scan[d][wl], o, y);
            }
        }
        y = __shfl_up_sync(all, y, 1, W);
        if (low) y = bin;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            y = h1_fma(-l[r], y, f[r]);
            f[r] = y;
        }
        // back substitution
        T x = high ? bin : T(0);
#pragma unroll
        for (int r = R - 1; r >= 0; --r) x = h1_fma(-g[r], x, f[r]);
#pragma unroll
        for (int d = 0; d < H1_SCAN; ++d) {
            if ((1 << d) < W) {
                const T o = __shfl_down_sync(all, x, 1 << d, W);
                if (li + (1 << d) < W) x = h1_fma(scan[H1_SCAN + d][wl], o, x);
            }
        }
        x = __shfl_down_sync(all, x, 1, W);
        if (high) x = bin;
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            x = h1_fma(-g[r], x, f[r]);
            const T v = h1_fma(sq[r][wl], x, cn ? -u[r] : T(0));
            u[r] = live ? v : u[r];
        }
        if (KEEP && live) {
            row += L.forward ? 1 : -1;
            T *A1 = ALL + static_cast<long long>(row) * NS;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (t0 + r <= end) A1[el(t0 + r)] = u[r];
            if (low && start == 1) A1[0] = bcur;
            if (high && end < N) A1[el(N)] = bcur;
        }
    }
    int bad = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (act && t0 + r <= end) {
            U[el(t0 + r)] = u[r];
            bad |= !isfinite(static_cast<double>(u[r]));
        }
    if (act && low && start == 1) {
        U[0] = bold;
        bad |= !isfinite(static_cast<double>(bold));
    }
    if (act && high && end < N) {
        U[el(N)] = bold;
        bad |= !isfinite(static_cast<double>(bold));
    }
    const unsigned b = __ballot_sync(all, bad);
    const unsigned mine = (W == 32 ? all : ((1u << W) - 1u) << (sub * W));
    __syncwarp();
    if (act && low) {
        const int i = L.eval_i;
        p.values[L.inst] = (1.0 - L.eval_w) * static_cast<double>(U[el(i)]) + L.eval_w * static_cast<double>(U[el(i + 1)]);
        p.status[L.inst] = (b & mine) != 0;
    }
    __syncwarp();
}

// One warp per unit (units costliest first: CTAs are dispatched in order, so the longest start
// first), two warps per SM sub-partition.
template <bool SRC, bool KEEP> __global__ void __launch_bounds__(LANES, 8) k_h1_reg(const h1params<double> p)
{
    __shared__ double scan[2 * H1_SCAN][LANES];
    __shared__ double sq[H1_RMAX][LANES];
    const h1unit un = p.units[blockIdx.x];
    switch (un.R) {
    case 4: h1_reg_unit<double, 4, SRC, KEEP>(p, un, scan, sq); break;
    case 5: h1_reg_unit<double, 5, SRC, KEEP>(p, un, scan, sq); break;
    case 6: h1_reg_unit<double, 6, SRC, KEEP>(p, un, scan, sq); break;
    case 7: h1_reg_unit<double, 7, SRC, KEEP>(p, un, scan, sq); break;
    case 8: h1_reg_unit<double, 8, SRC, KEEP>(p, un, scan, sq); break;
    case 9: h1_reg_unit<double, 9, SRC, KEEP>(p, un, scan, sq); break;
    case 10: h1_reg_unit<double, 10, SRC, KEEP>(p, un, scan, sq); break;
    case 11: h1_reg_unit<double, 11, SRC, KEEP>(p, un, scan, sq); break;
    case 12: h1_reg_unit<double, 12, SRC, KEEP>(p, un, scan, sq); break;
    case 13: h1_reg_unit<double, 13, SRC, KEEP>(p, un, scan, sq); break;
    case 14: h1_reg_unit<double, 14, SRC, KEEP>(p, un, scan, sq); break;
    case 15: h1_reg_unit<double, 15, SRC, KEEP>(p, un, scan, sq); break;
    default: h1_reg_unit<double, H1_RMAX, SRC, KEEP>(p, un, scan, sq); break;
    }
    end_of_run();
}

// ------------------------------------------------------------------------------------------
// FAST, FP32 instances whose rows fit a warp's registers: the operations of the sweep through memory in
// its order (same bits), with W lanes of R rows per instance as above.  The first and the last solved
// row are scalars of the lowest and highest lane, the rows between them fill the lanes from the upper
// end; places below them pass a value through (slope -1 on -0: exact for every value) and hold the first
// row's u.  Right-hand sides are evaluated by all lanes at once.  A recurrence is run W times by every
// lane, each time from the value that the lane before ended with: after k rounds the lanes below k
// are final.
//
// What bounds it: 2 W rounds of R dependent multiply-adds and a shuffle (about 90 cycles at R = 16, 3.3 ms
// for 512 points and 1000 steps) for the longest instances, the issue slots of those rounds for a
// full GPU.  8192 Black-Scholes calls of 101..512 points and 100..1000 steps: 4.7 ms; the sweep through
// memory took 22.2 ms, 85 cycles per row of its longest line.
// ------------------------------------------------------------------------------------------
constexpr int H1_RELAY_MIN = 8; // points: at least two rows between first and last solved one

template <int R, bool KEEP> __device__ __forceinline__ void h1_relay_unit(const h1params<float> &p, const h1unit un)
{
    using T = float;
    const unsigned all = 0xffffffffu;
    const int wl = threadIdx.x & 31, W = un.W, li = wl & (W - 1), sub = wl / W;
    const h1group G = p.groups[un.g];
    const bool act = sub < un.sub;
    const int lane = un.lane0 + (act ? sub : 0); // idle sub-warps shadow the first instance and store nothing
    const h1lane L = p.lanes[static_cast<long long>(un.g) * LANES + lane];
    const int n = G.n, N = n - 1;
    const long long NS = static_cast<long long>(n) * LANES;
    T *base = p.pt + G.pt + lane;
    const T *WB = base + S_B * NS, *WD = base + S_D * NS, *M = base + S_M * NS, *GG = base + S_G * NS;
    T *U = base + S_U * NS;
    const T *BND = p.bnd + G.bnd + lane;
    T *ALL = KEEP ? p.all + G.all + lane : nullptr;
    const T th = T(L.theta), omt = T(1) - th, bl = T(L.bl), bh = T(L.bh);
    const T kap = -omt / th;
    const bool cn = kap != T(0);
    const int start = L.start, end = L.end, steps = act ? L.steps : 0;
    const bool low = li == 0, high = li == W - 1;
    const T *init = p.init + L.init_off;
    const int pad = W * R - (end - start - 1);    // places below the rows
    const int t0 = start + 1 - pad + li * R;      // row of this lane's first place
    const int pr = min(max(pad - li * R, 0), R);  // places of this lane below the rows

    T wb[R], wd[R], m[R], g[R], u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool in = r >= pr;
        const int t = in ? t0 + r : start;
        wb[r] = in ? WB[el(t)] : T(0);
        wd[r] = in ? WD[el(t)] : T(0);
        m[r] = in ? M[el(t)] : T(-1);
        g[r] = in ? GG[el(t)] : T(-1);
        u[r] = init[t];
    }
    // the end row of this lane's side (lane 0: the first, others: the last one)
    const int te = low ? start : end;
    const T ewb = WB[el(te)], ewd = WD[el(te)], em = M[el(te)], eg = GG[el(start)];
    T ue = init[te];
    T nb = init[low ? start + 1 : end - 1];                                     // its neighbour inside
    T ob = low ? (start ? init[0] : T(0)) : (end < N ? init[N] : T(0));          // and outside
    const int side = low ? 0 : 1;
    T bnew = steps > 0 ? BND[side * LANES] : T(0);
    T bcur = init[low ? 0 : N];
    int row = L.forward ? 0 : L.steps;
    if (KEEP && act) {
        for (int t = li; t < n; t += W) ALL[(static_cast<long long>(row) * n + t) * LANES] = init[t];
    }
    for (int s = 0; s < un.steps; ++s) {
        const bool live = s < steps;
        const T bv = bnew;
        if (s + 1 < steps) bnew = BND[(2 * (s + 1) + side) * LANES];
        // right-hand sides
        T c[R];
        const T first_u = __shfl_sync(all, ue, 0, W), last_u = __shfl_sync(all, ue, W - 1, W);
        T um = __shfl_up_sync(all, u[R - 1], 1, W), un1 = __shfl_down_sync(all, u[0], 1, W);
        if (low) um = first_u;
        if (high) un1 = last_u;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const T u1 = r + 1 < R ? u[r + 1 < R ? r + 1 : 0] : un1;
            const T v = h1_fma(-m[r], cn ? um : T(0), h1_fma(wd[r], u1, wb[r] * u[r]));
            c[r] = r >= pr ? v : T(-0.0f);
            um = u[r];
        }
        // first row (lane 0); the order of the sums is that of the sweep through memory
        T yf;
        {
            const T uc = ue, up = nb;
            yf = h1_fma(em, h1_fma(kap, ob, start ? -bv : T(0)), h1_fma(ewb, uc, ewd * up));
            if (start == 0) yf = h1_fma(bl, bv, yf);
            yf += T(0);
        }
        // forward recurrence
        T y = yf;
        for (int k = 1; k < W; ++k) {
            T z = y;
#pragma unroll
            for (int r = 0; r < R; ++r) z = h1_fma(-m[r], z, c[r]);
            z = __shfl_up_sync(all, z, 1, W);
            y = low ? yf : z;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            y = h1_fma(-m[r], y, c[r]);
            c[r] = y;
        }
        // last row (lane W - 1: y is the row before)
        T xl;
        {
            const T uc = ue, u1 = ob, um2 = nb;
            xl = h1_fma(bh, bv, h1_fma(em, h1_fma(kap, um2, -y), h1_fma(ewb, uc, ewd * u1)));
            xl += T(0);
        }
        // back substitution
#pragma unroll
        for (int r = 0; r < R; ++r) c[r] = r >= pr ? c[r] : T(-0.0f);
        T x = xl;
        for (int k = 1; k < W; ++k) {
            T z = x;
#pragma unroll
            for (int r = R - 1; r >= 0; --r) z = h1_fma(-g[r], z, c[r]);
            z = __shfl_down_sync(all, z, 1, W);
            x = high ? xl : z;
        }
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            x = h1_fma(-g[r], x, c[r]);
            c[r] = x;
        }
        // x of lane 0: row start + 1; the first row
        const T xf = h1_fma(-eg, x, yf);
        const T fill = __shfl_sync(all, xf, 0, W);
        if (live) {
#pragma unroll
            for (int r = 0; r < R; ++r) u[r] = r >= pr ? c[r] : fill;
            ue = low ? xf : xl;
            nb = low ? x : c[R - 1];
            ob = (low ? start == 1 : end < N) ? bv : T(0);
            bcur = bv;
        }
        if (KEEP && live) {
            row += L.forward ? 1 : -1;
            T *A1 = ALL + static_cast<long long>(row) * NS;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r >= pr) A1[el(t0 + r)] = u[r];
            if (low) A1[el(start)] = ue;
            if (high) A1[el(end)] = ue;
            if (low && start == 1) A1[0] = bcur;
            if (high && end < N) A1[el(N)] = bcur;
        }
    }
    int bad = 0;
    if (act) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r >= pr) {
                U[el(t0 + r)] = u[r];
                bad |= !isfinite(u[r]);
            }
        if (low || high) {
            U[el(te)] = ue;
            bad |= !isfinite(ue);
            if (low ? start == 1 : end < N) {
                U[el(low ? 0 : N)] = bcur;
                bad |= !isfinite(bcur);
            }
        }
    }
    const unsigned b = __ballot_sync(all, bad);
    const unsigned mine = (W == 32 ? all : ((1u << W) - 1u) << (sub * W));
    __syncwarp();
    if (act && low) {
        const int i = L.eval_i;
        p.values[L.inst] = (1.0 - L.eval_w) * static_cast<double>(U[el(i)]) + L.eval_w * static_cast<double>(U[el(i + 1)]);
        p.status[L.inst] = (b & mine) != 0;
    }
}

template <bool KEEP> __global__ void __launch_bounds__(LANES, 16) k_h1_relay(const h1params<float> p)
{
    const h1unit un = p.units[blockIdx.x];
    switch (un.R) {
    case 4: h1_relay_unit<4, KEEP>(p, un); break;
    case 5: h1_relay_unit<5, KEEP>(p, un); break;
    case 6: h1_relay_unit<6, KEEP>(p, un); break;
    case 7: h1_relay_unit<7, KEEP>(p, un); break;
    case 8: h1_relay_unit<8, KEEP>(p, un); break;
    case 9: h1_relay_unit<9, KEEP>(p, un); break;
    case 10: h1_relay_unit<10, KEEP>(p, un); break;
    case 11: h1_relay_unit<11, KEEP>(p, un); break;
    case 12: h1_relay_unit<12, KEEP>(p, un); break;
    case 13: h1_relay_unit<13, KEEP>(p, un); break;
    case 14: h1_relay_unit<14, KEEP>(p, un); break;
    case 15: h1_relay_unit<15, KEEP>(p, un); break;
    default: h1_relay_unit<H1_RMAX, KEEP>(p, un); break;
    }
    end_of_run();
}

// scatter of per-instance contiguous tables into the interleaved group layout (the instance of
// a flat position found by binary search over the instances' offsets)
// coef (3 rows of n) -> slots 0..2
template <typename T>
__global__ void k_h1_scatter_coef(const h1group *groups, const int *ig, const int *il, const long long *off,
                                  const int *nn, int count, const T *flat, T *pt, long long total)
{
    for (long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; q < total;
         q += static_cast<long long>(gridDim.x) * blockDim.x) {
        // locate the instance by binary search over offsets (3n elements each)
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (off[mid] <= q) lo = mid; else hi = mid - 1;
        }
        const int inst = lo;
        const long long r = q - off[inst];
        const int n = nn[inst];
        const int slot = static_cast<int>(r / n), t = static_cast<int>(r % n);
        const h1group G = groups[ig[inst]];
        pt[G.pt + (static_cast<long long>(slot) * n + t) * LANES + il[inst]] = flat[q];
    }
}

// rows x len per instance (boundary values: len 2, source: len n) -> interleaved at `field`
template <typename T>
__global__ void k_h1_scatter_rows(const h1group *groups, const int *ig, const int *il, const long long *off,
                                  const int *len, int count, const T *flat, T *dst, int field, long long total)
{
    for (long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; q < total;
         q += static_cast<long long>(gridDim.x) * blockDim.x) {
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (off[mid] <= q) lo = mid; else hi = mid - 1;
        }
        const int inst = lo;
        const long long r = q - off[inst];
        const h1group G = groups[ig[inst]];
        const long long base = field == 0 ? G.bnd : G.src;
        dst[base + r * LANES + il[inst]] = flat[q];
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
struct inst_info {
    int n, nt, lo_kind, hi_kind, has_src, forward, theta_scheme;
    double t_lo, t_hi, lo_lin, hi_lin;
    int eval_i;
    double eval_w;
};

template <typename T> struct host_tables {
    std::vector<T> coef, init, bnd, src; // coef 3n, init n, bnd 2*steps, src (steps+1)*n
    std::vector<T> x;                    // physical grid (Black-Scholes)
};

struct batch_base {
    virtual ~batch_base() = default;
    int precision = LSS_ADI_FP64, arith = LSS_ADI_ARITH_FAST, options = 0, count = 0;
    double point_steps = 0;
    virtual int launches() const = 0; // kernels of one run
};

template <typename T> struct batch_t : batch_base {
    std::vector<inst_info> info;
    std::vector<h1group> groups;
    std::vector<h1lane> lanes;
    std::vector<int> inst_group, inst_lane;
    std::vector<long long> init_off;
    std::vector<std::vector<T>> grids;
    long long total_init = 0;
    dbuf<h1group> d_groups;
    dbuf<h1lane> d_lanes;
    dbuf<T> d_pt, d_bnd, d_src, d_all, d_init;
    dbuf<double> d_values;
    dbuf<int> d_status;
    dbuf<h1unit> d_units;         // factorised sweep in registers
    int nunits = 0;
    warp_schedule sched;          // placement of the groups for the factorised sweep through memory
    dbuf<int> d_wfirst, d_wgroup;
    bool ds = false;

    h1params<T> params()
    {
        h1params<T> p{};
        p.groups = d_groups.p;
        p.lanes = d_lanes.p;
        p.ngroups = static_cast<int>(groups.size());
        p.pt = d_pt.p;
        p.bnd = d_bnd.p;
        p.src = d_src.p;
        p.all = d_all.p;
        p.init = d_init.p;
        p.values = d_values.p;
        p.status = d_status.p;
        p.units = d_units.p;
        p.warp_first = d_wfirst.p;
        p.warp_group = d_wgroup.p;
        p.nwarps = sched.ctas * sched.warps_per_cta;
        p.warps_per_cta = sched.warps_per_cta;
        return p;
    }
    // most rows that an instance of a group solves in registers (k_h1_relay: between its first and last)
    int group_rows(size_t g) const
    {
        int rows = 0;
        for (int l = 0; l < groups[g].lanes; ++l) {
            const h1lane &L = lanes[g * LANES + l];
            rows = std::max(rows, L.end - L.start + 1);
        }
        return groups[g].reg == 2 ? rows - 2 : rows;
    }
    int build(std::vector<inst_info> &&inf, std::vector<host_tables<T>> &tabs);
    int run(cudaStream_t s);
    int launches() const override { return arith == LSS_ADI_ARITH_FAST ? (nunits > 0) + (sched.ctas > 0) : 1; }
};

static int check_theta(int th)
{
    return th == LSS_ADI_EULER || th == LSS_ADI_CRANK_NICOLSON;
}

template <typename T> int batch_t<T>::build(std::vector<inst_info> &&inf, std::vector<host_tables<T>> &tabs)
{
    info = std::move(inf);
    count = static_cast<int>(info.size());
    // sort by size (desc), then steps (desc): equal-size groups of 32 with similar time loops
    std::vector<int> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        if (info[a].n != info[b].n) return info[a].n > info[b].n;
        return info[a].nt > info[b].nt;
    });
    inst_group.assign(count, 0);
    inst_lane.assign(count, 0);
    long long pt = 0, bnd = 0, src = 0, all = 0;
    const bool keep_all = (options & LSS_HEAT1D_OPT_ALL_STEPS) != 0;
    for (int q = 0; q < count;) {
        const int n = info[order[q]].n;
        h1group G{};
        G.n = n;
        int l = 0, steps = 0, gsrc = 0;
        while (q + l < count && l < LANES && info[order[q + l]].n == n) {
            steps = std::max(steps, info[order[q + l]].nt - 1);
            gsrc |= info[order[q + l]].has_src;
            ++l;
        }
        G.lanes = l;
        G.steps = steps;
        // FP64 lines that fit a warp's registers (but see memory_limit).  Against the sweep through memory (a
        // thread per instance): 4096 Black-Scholes calls of 101..512 points, 100..1000 steps 104 ms -> 7.7 ms.
        // FP32 lines without sources keep that sweep's operations and their order (k_h1_relay): 8192 calls
        // of the same sizes 22.2 ms -> 4.7 ms.  Sources and longer lines stay in memory.
        G.reg = 0;
        if (arith == LSS_ADI_ARITH_FAST && n <= LANES * H1_RMAX) {
            if (std::is_same<T, double>::value) G.reg = 1;
            else if (!gsrc && n >= H1_RELAY_MIN) G.reg = 2;
        }
        G.pt = pt;
        pt += static_cast<long long>(NSLOT) * n * LANES;
        G.bnd = bnd;
        bnd += 2LL * steps * LANES;
        G.src = gsrc ? src : -1;
        if (gsrc) src += static_cast<long long>(steps + 1) * n * LANES;
        G.all = keep_all ? all : -1;
        if (keep_all) all += static_cast<long long>(steps + 1) * n * LANES;
        const int gi = static_cast<int>(groups.size());
        for (int j = 0; j < l; ++j) {
            inst_group[order[q + j]] = gi;
            inst_lane[order[q + j]] = j;
        }
        groups.push_back(G);
        q += l;
    }
    // lanes and contiguous initial conditions
    lanes.assign(groups.size() * LANES, h1lane{});
    for (auto &L : lanes) L.inst = -1;
    init_off.assign(count, 0);
    total_init = 0;
    point_steps = 0;
    for (int i = 0; i < count; ++i) {
        init_off[i] = total_init;
        total_init += info[i].n;
        point_steps += static_cast<double>(info[i].n) * (info[i].nt - 1);
        const inst_info &f = info[i];
        h1lane &L = lanes[static_cast<size_t>(inst_group[i]) * LANES + inst_lane[i]];
        L.inst = i;
        L.steps = f.nt - 1;
        L.lo_kind = f.lo_kind;
        L.hi_kind = f.hi_kind;
        L.start = f.lo_kind == LSS_HEAT1D_DIRICHLET ? 1 : 0;
        L.end = f.hi_kind == LSS_HEAT1D_DIRICHLET ? f.n - 2 : f.n - 1;
        L.has_src = f.has_src;
        L.forward = f.forward;
        L.eval_i = f.eval_i;
        L.eval_w = f.eval_w;
        const T one = T(1.0);
        L.theta = f.theta_scheme == LSS_ADI_EULER ? 1.0 : 0.5;
        L.h = static_cast<double>(one / static_cast<T>(static_cast<size_t>(f.n - 1)));
        L.k = static_cast<double>((static_cast<T>(f.t_hi) - static_cast<T>(f.t_lo)) / static_cast<T>(static_cast<size_t>(f.nt - 1)));
        L.lo_lin = f.lo_lin;
        L.hi_lin = f.hi_lin;
        L.init_off = init_off[i];
    }
    // FP64 groups of short lines in a book that fills the GPU go back to the sweep through memory
    {
        int dev = 0, sms = 0;
        LSS_CUDA_TRY(cudaGetDevice(&dev), "heat1d: device");
        LSS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "heat1d: SM count");
        std::vector<group_cost> cost;
        for (size_t g = 0; g < groups.size(); ++g)
            if (groups[g].reg == 1) cost.push_back({groups[g].n, group_rows(g), groups[g].lanes, groups[g].steps});
        const int limit = memory_limit(cost, sms, H1_RMAX);
        for (h1group &G : groups)
            if (G.reg == 1 && G.n <= limit) G.reg = 0;
    }
    // flat host arrays in creation order
    std::vector<T> coef_flat, init_flat(total_init), bnd_flat, src_flat;
    std::vector<long long> coef_off(count), bnd_off(count), src_off(count);
    std::vector<int> nn(count);
    long long cpos = 0, bpos = 0, spos = 0;
    for (int i = 0; i < count; ++i) {
        coef_off[i] = cpos;
        cpos += 3LL * info[i].n;
        bnd_off[i] = bpos;
        bpos += 2LL * (info[i].nt - 1);
        src_off[i] = spos;
        if (info[i].has_src) spos += static_cast<long long>(info[i].nt) * info[i].n;
        nn[i] = info[i].n;
    }
    coef_flat.resize(cpos);
    bnd_flat.resize(bpos);
    src_flat.resize(spos);
    for (int i = 0; i < count; ++i) {
        std::copy(tabs[i].coef.begin(), tabs[i].coef.end(), coef_flat.begin() + coef_off[i]);
        std::copy(tabs[i].init.begin(), tabs[i].init.end(), init_flat.begin() + init_off[i]);
        std::copy(tabs[i].bnd.begin(), tabs[i].bnd.end(), bnd_flat.begin() + bnd_off[i]);
        if (info[i].has_src) std::copy(tabs[i].src.begin(), tabs[i].src.end(), src_flat.begin() + src_off[i]);
        if (!tabs[i].x.empty()) grids.push_back(std::move(tabs[i].x));
        std::vector<T>().swap(tabs[i].coef);
        std::vector<T>().swap(tabs[i].bnd);
        std::vector<T>().swap(tabs[i].src);
    }
    LSS_CUDA_TRY(d_groups.alloc(groups.size()), "heat1d: allocating groups");
    LSS_CUDA_TRY(d_groups.upload(groups.data(), groups.size()), "heat1d: uploading groups");
    LSS_CUDA_TRY(d_lanes.alloc(lanes.size()), "heat1d: allocating lanes");
    LSS_CUDA_TRY(d_lanes.upload(lanes.data(), lanes.size()), "heat1d: uploading lanes");
    LSS_CUDA_TRY(d_pt.alloc(pt + H1_PAD), "heat1d: allocating point arrays");
    LSS_CUDA_TRY(cudaMemset(d_pt.p, 0, (pt + H1_PAD) * sizeof(T)), "heat1d: clearing point arrays");
    LSS_CUDA_TRY(d_bnd.alloc(std::max(1LL, bnd)), "heat1d: allocating boundary values");
    LSS_CUDA_TRY(cudaMemset(d_bnd.p, 0, d_bnd.n * sizeof(T)), "heat1d: clearing boundary values");
    if (src > 0) {
        LSS_CUDA_TRY(d_src.alloc(src), "heat1d: allocating source rows");
        LSS_CUDA_TRY(cudaMemset(d_src.p, 0, src * sizeof(T)), "heat1d: clearing source rows");
    }
    if (all > 0) LSS_CUDA_TRY(d_all.alloc(all), "heat1d: allocating time levels");
    LSS_CUDA_TRY(d_init.alloc(total_init), "heat1d: allocating initial conditions");
    LSS_CUDA_TRY(d_init.upload(init_flat.data(), total_init), "heat1d: uploading initial conditions");
    LSS_CUDA_TRY(d_values.alloc(count), "heat1d: allocating values");
    LSS_CUDA_TRY(d_status.alloc(count), "heat1d: allocating status");
    {
        dbuf<int> d_ig, d_il, d_nn, d_len;
        dbuf<long long> d_off;
        dbuf<T> d_flat;
        LSS_CUDA_TRY(d_ig.alloc(count), "heat1d: set-up");
        LSS_CUDA_TRY(d_ig.upload(inst_group.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_il.alloc(count), "heat1d: set-up");
        LSS_CUDA_TRY(d_il.upload(inst_lane.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_nn.alloc(count), "heat1d: set-up");
        LSS_CUDA_TRY(d_nn.upload(nn.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_off.alloc(count), "heat1d: set-up");
        // coefficient tables
        LSS_CUDA_TRY(d_off.upload(coef_off.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_flat.alloc(cpos), "heat1d: set-up");
        LSS_CUDA_TRY(d_flat.upload(coef_flat.data(), cpos), "heat1d: set-up");
        k_h1_scatter_coef<T><<<std::min(grid_for(cpos, 256), 65535), 256>>>(d_groups.p, d_ig.p, d_il.p, d_off.p,
                                                                           d_nn.p, count, d_flat.p, d_pt.p, cpos);
        LSS_CUDA_TRY(cudaGetLastError(), "heat1d: scattering coefficients");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "heat1d: scattering coefficients");
        // boundary values (2 per step)
        std::vector<int> len(count);
        for (int i = 0; i < count; ++i) len[i] = 2;
        LSS_CUDA_TRY(d_len.alloc(count), "heat1d: set-up");
        LSS_CUDA_TRY(d_len.upload(len.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_off.upload(bnd_off.data(), count), "heat1d: set-up");
        LSS_CUDA_TRY(d_flat.alloc(std::max(1LL, bpos)), "heat1d: set-up");
        LSS_CUDA_TRY(d_flat.upload(bnd_flat.data(), bpos), "heat1d: set-up");
        k_h1_scatter_rows<T><<<std::min(grid_for(bpos, 256), 65535), 256>>>(d_groups.p, d_ig.p, d_il.p, d_off.p,
                                                                           d_len.p, count, d_flat.p, d_bnd.p, 0, bpos);
        LSS_CUDA_TRY(cudaGetLastError(), "heat1d: scattering boundary values");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "heat1d: scattering boundary values");
        if (spos > 0) {
            // instances without a source own no rows: give them an offset past the end so
            // that the search never lands on them for a position they do not own
            std::vector<long long> so(count);
            std::vector<int> sidx;
            for (int i = 0; i < count; ++i)
                if (info[i].has_src) sidx.push_back(i);
            std::vector<long long> soff(sidx.size());
            std::vector<int> sig(sidx.size()), sil(sidx.size()), sn(sidx.size());
            for (size_t j = 0; j < sidx.size(); ++j) {
                soff[j] = src_off[sidx[j]];
                sig[j] = inst_group[sidx[j]];
                sil[j] = inst_lane[sidx[j]];
                sn[j] = info[sidx[j]].n;
            }
            const int sc = static_cast<int>(sidx.size());
            LSS_CUDA_TRY(d_off.upload(soff.data(), sc), "heat1d: set-up");
            LSS_CUDA_TRY(d_ig.upload(sig.data(), sc), "heat1d: set-up");
            LSS_CUDA_TRY(d_il.upload(sil.data(), sc), "heat1d: set-up");
            LSS_CUDA_TRY(d_len.upload(sn.data(), sc), "heat1d: set-up");
            LSS_CUDA_TRY(d_flat.alloc(spos), "heat1d: set-up");
            LSS_CUDA_TRY(d_flat.upload(src_flat.data(), spos), "heat1d: set-up");
            k_h1_scatter_rows<T><<<std::min(grid_for(spos, 256), 65535), 256>>>(
                d_groups.p, d_ig.p, d_il.p, d_off.p, d_len.p, sc, d_flat.p, d_src.p, 1, spos);
            LSS_CUDA_TRY(cudaGetLastError(), "heat1d: scattering source rows");
            LSS_CUDA_TRY(cudaDeviceSynchronize(), "heat1d: scattering source rows");
        }
    }
    if (arith == LSS_ADI_ARITH_FAST) {
        int dev = 0, sms = 0;
        LSS_CUDA_TRY(cudaGetDevice(&dev), "heat1d: device");
        LSS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "heat1d: SM count");
        // lines that fit a warp's registers: one unit per 32 / W instances of a group, costliest first
        std::vector<h1unit> units;
        std::vector<int> mem_groups;
        double warps = 0.0; // of the FP64 groups on the fewest lanes
        for (size_t g = 0; g < groups.size(); ++g)
            if (groups[g].reg == 1) {
                int W = 0, R = 0;
                register_shape(group_rows(g), 4, H1_RMAX, W, R);
                warps += (groups[g].lanes * W + 31) / 32;
            }
        const bool idle = warps <= 8.0 * sms; // two warps per SM sub-partition
        for (size_t g = 0; g < groups.size(); ++g) {
            const h1group &G = groups[g];
            if (!G.reg) {
                mem_groups.push_back(static_cast<int>(g));
                continue;
            }
            int W = 0, R = 0;
            const int rows = group_rows(g);
            int least = G.reg == 1 ? 4 : 2;
            if (G.reg == 1 && idle) register_shape(G.n, 4, H1_RMAX, least, R);
            register_shape(rows, least, H1_RMAX, W, R);
            for (int l = 0; l < G.lanes; l += 32 / W) {
                h1unit u{static_cast<int>(g), l, std::min(32 / W, G.lanes - l), W, R, 0};
                for (int q = 0; q < u.sub; ++q) u.steps = std::max(u.steps, lanes[g * LANES + l + q].steps);
                units.push_back(u);
            }
        }
        std::stable_sort(units.begin(), units.end(), [](const h1unit &a, const h1unit &b) {
            return static_cast<long long>(a.R) * a.steps > static_cast<long long>(b.R) * b.steps;
        });
        nunits = static_cast<int>(units.size());
        LSS_CUDA_TRY(d_units.alloc(units.size()), "heat1d: allocating the warp units");
        LSS_CUDA_TRY(d_units.upload(units.data(), units.size()), "heat1d: uploading the warp units");
        std::vector<double> work(mem_groups.size());
        for (size_t g = 0; g < mem_groups.size(); ++g)
            work[g] = static_cast<double>(groups[mem_groups[g]].n) * groups[mem_groups[g]].steps;
        sched = schedule_groups(work, sms, h1_warps<T>());
        for (int &g : sched.group) g = mem_groups[g];
        LSS_CUDA_TRY(d_wfirst.alloc(sched.first.size()), "heat1d: allocating the warp schedule");
        LSS_CUDA_TRY(d_wfirst.upload(sched.first.data(), sched.first.size()), "heat1d: uploading the warp schedule");
        LSS_CUDA_TRY(d_wgroup.alloc(sched.group.size()), "heat1d: allocating the warp schedule");
        LSS_CUDA_TRY(d_wgroup.upload(sched.group.data(), sched.group.size()), "heat1d: uploading the warp schedule");
        const h1params<T> p = params();
        k_h1_setup_fast<T><<<grid_for(static_cast<long long>(groups.size()) * LANES, 128), 128>>>(p);
        LSS_CUDA_TRY(cudaGetLastError(), "heat1d: launching the factorisation");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "heat1d: factorisation");
    }
    return LSS_ADI_OK;
}

template <typename T> int batch_t<T>::run(cudaStream_t s)
{
    const h1params<T> p = params();
    const int blocks = grid_for(static_cast<long long>(groups.size()) * LANES, 128);
    const bool keep = d_all.p != nullptr, src = d_src.p != nullptr;
    if (arith == LSS_ADI_ARITH_FAST) {
        const int ctas = sched.ctas, th = sched.warps_used() * LANES;
        if (ctas) {
            if (keep && src) k_h1_fast<T, H1_PF, true, true><<<ctas, th, 0, s>>>(p);
            else if (keep) k_h1_fast<T, H1_PF, false, true><<<ctas, th, 0, s>>>(p);
            else if (src) k_h1_fast<T, H1_PF, true, false><<<ctas, th, 0, s>>>(p);
            else k_h1_fast<T, H1_PF, false, false><<<ctas, th, 0, s>>>(p);
            LSS_CUDA_TRY(cudaGetLastError(), "heat1d: launching the time loop");
        }
        if (!nunits) return LSS_ADI_OK;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(nunits);
        cfg.blockDim = dim3(LANES);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = ctas ? 1 : 0;
        void (*k)(const h1params<T>);
        if constexpr (std::is_same<T, double>::value)
            k = keep && src ? k_h1_reg<true, true> : keep ? k_h1_reg<false, true> : src ? k_h1_reg<true, false> : k_h1_reg<false, false>;
        else
            k = keep ? k_h1_relay<true> : k_h1_relay<false>;
        LSS_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, p), "heat1d: launching the time loop");
        return LSS_ADI_OK;
    }
    if constexpr (std::is_same<T, double>::value) {
        if (ds) k_h1_ref64<true, 4><<<blocks, 128, 0, s>>>(p);
        else k_h1_ref64<false, 4><<<blocks, 128, 0, s>>>(p);
    } else {
        if (ds) k_h1_ref<T, true, 4><<<blocks, 128, 0, s>>>(p);
        else k_h1_ref<T, false, 4><<<blocks, 128, 0, s>>>(p);
    }
    LSS_CUDA_TRY(cudaGetLastError(), "heat1d: launching the time loop");
    return LSS_ADI_OK;
}

// ---- Black-Scholes tables in the reference's arithmetic (host) ----------------------------
// grid_config_1d (discretization/lss_grid_config.hpp:21-52), grid_transform_config<One>
// (discretization/lss_grid_transform_config.hpp:32-87), heat_data_transform<One>
// (pde_solvers/transformation/lss_heat_data_transform.hpp:34-131), general_heat_equation_coefficients
// (implicit_coefficients/lss_1d_general_heat_equation_coefficients.hpp:34-64); user lambdas as in
// unit_tests/pde_solvers/one_dimensional/lss_black_scholes_equation_t.hpp:854-880 (double).
template <typename T> static void bs_tables(const lss_heat1d_bs &q, host_tables<T> &tb, inst_info &f)
{
    const int n = q.n, steps = q.nt - 1;
    const T one = T(1.0), two = T(2.0), half = T(0.5);
    const T step = one / static_cast<T>(static_cast<size_t>(n - 1));
    const T k = (static_cast<T>(q.maturity) - T(0.0)) / static_cast<T>(static_cast<size_t>(q.nt - 1));
    const T h = one / static_cast<T>(static_cast<size_t>(n - 1));
    const T lambda = k / (h * h), gamma = k / (two * h), delta = half * k;
    const T low = static_cast<T>(q.s_lo), high = static_cast<T>(q.s_hi), point = static_cast<T>(q.acc_point);
    T alpha = high - low;
    if (q.nonuniform) alpha = (point - low) / static_cast<T>(q.alpha_scale);
    const T c0 = std::asinh((high - point) / alpha), c1 = std::asinh((low - point) / alpha);
    const T cdiff = c0 - c1;
    auto arg = [&](T z) { return c0 * z + c1 * (one - z); };
    auto xval = [&](T z) { return point + alpha * std::sinh(arg(z)); };
    auto ader = [&](T z) { return alpha * cdiff * std::cosh(arg(z)); };
    auto bder = [&](T z) { return alpha * cdiff * cdiff * std::sinh(arg(z)); };
    const double sig = q.sigma, rate = q.rate, strike = q.strike, maturity = q.maturity, s_hi = q.s_hi;
    auto ua = [&](T x) -> T { return static_cast<T>(0.5 * sig * sig * x * x); };
    auto ub = [&](T x) -> T { return static_cast<T>(rate * x); };
    auto uc = [&](T x) -> T { (void)x; return static_cast<T>(-rate); };
    tb.coef.resize(3 * static_cast<size_t>(n));
    tb.init.resize(n);
    tb.x.resize(n);
    for (int i = 0; i < n; ++i) {
        const T zeta = step * static_cast<T>(static_cast<size_t>(i));
        const T x = xval(zeta);
        const T av = ader(zeta);
        const T ta = ua(x) / (ader(zeta) * ader(zeta));
        const T first = ub(x) / av;
        const T second = (ua(x) * bder(zeta)) / (av * av * av);
        const T tbv = first - second;
        const T tc = uc(x);
        tb.coef[i] = lambda * ta - gamma * tbv;
        tb.coef[n + i] = lambda * ta - delta * tc;
        tb.coef[2 * n + i] = lambda * ta + gamma * tbv;
        const T v = q.put ? static_cast<T>(strike - static_cast<double>(x)) : static_cast<T>(static_cast<double>(x) - strike);
        tb.init[i] = (T(0.0) < v) ? v : T(0.0);
        tb.x[i] = x;
    }
    // boundary values at the times of the backward loop: t = maturity - k, then -= k
    tb.bnd.resize(2 * static_cast<size_t>(steps));
    T time = static_cast<T>(q.maturity) - k;
    for (int s = 0; s < steps; ++s) {
        const double disc = strike * std::exp(-rate * (maturity - static_cast<double>(time)));
        tb.bnd[2 * s] = q.put ? static_cast<T>(disc) : T(0.0);
        tb.bnd[2 * s + 1] = q.put ? T(0.0) : static_cast<T>(s_hi - disc);
        time -= k;
    }
    f.n = n;
    f.nt = q.nt;
    f.lo_kind = f.hi_kind = LSS_HEAT1D_DIRICHLET;
    f.has_src = 0;
    f.forward = 0;
    f.theta_scheme = q.theta_scheme;
    f.t_lo = 0.0;
    f.t_hi = q.maturity;
    f.lo_lin = f.hi_lin = 0.0;
    // linear interpolation weight of eval_s
    int i0 = 0;
    while (i0 + 2 < n && static_cast<double>(tb.x[i0 + 1]) <= q.eval_s) ++i0;
    const double x0 = static_cast<double>(tb.x[i0]), x1 = static_cast<double>(tb.x[i0 + 1]);
    f.eval_i = i0;
    f.eval_w = x1 > x0 ? std::min(1.0, std::max(0.0, (q.eval_s - x0) / (x1 - x0))) : 0.0;
}

} // namespace heat1d
} // namespace lss_gb300

using namespace lss_gb300;
using namespace lss_gb300::heat1d;

struct lss_heat1d_batch {
    std::unique_ptr<batch_base> impl;
    cudaStream_t last = nullptr;
};

template <typename T> static batch_t<T> *as(lss_heat1d_batch *b) { return static_cast<batch_t<T> *>(b->impl.get()); }

static int valid_common(int count, int precision, int arith, int options, lss_heat1d_batch **b)
{
    if (!b) return set_error(LSS_ADI_EINVAL, "heat1d: batch pointer is NULL");
    *b = nullptr;
    if (count < 1) return set_error(LSS_ADI_EINVAL, "heat1d: count must be >= 1");
    if (precision != LSS_ADI_FP64 && precision != LSS_ADI_FP32) return set_error(LSS_ADI_EINVAL, "heat1d: precision");
    if (arith != LSS_ADI_ARITH_FAST && arith != LSS_ADI_ARITH_REFERENCE) return set_error(LSS_ADI_EINVAL, "heat1d: arith");
    if (options & ~(LSS_HEAT1D_OPT_ALL_STEPS | LSS_HEAT1D_OPT_DOUBLE_SWEEP))
        return set_error(LSS_ADI_EINVAL, "heat1d: unknown option bits");
    return LSS_ADI_OK;
}

template <typename T>
static int create_tab(const lss_heat1d_tables *ps, int count, int arith, int options, lss_heat1d_batch **b)
{
    std::vector<inst_info> info(count);
    std::vector<host_tables<T>> tabs(count);
    for (int i = 0; i < count; ++i) {
        const lss_heat1d_tables &q = ps[i];
        if (q.n < 4 || q.nt < 2) return set_error(LSS_ADI_EINVAL, "heat1d: n must be >= 4 and nt >= 2");
        if (!check_theta(q.theta_scheme))
            return set_error(LSS_ADI_EINVAL, "heat1d: the implicit 1-D kernel accepts Euler and Crank-Nicolson only");
        if (q.lo_kind < 0 || q.lo_kind > 2 || q.hi_kind < 0 || q.hi_kind > 2)
            return set_error(LSS_ADI_EINVAL, "heat1d: unknown boundary kind");
        if (!q.coef || !q.initial || !q.boundary) return set_error(LSS_ADI_EINVAL, "heat1d: table pointer is NULL");
        if (!(q.t_hi > q.t_lo)) return set_error(LSS_ADI_EINVAL, "heat1d: t_hi must exceed t_lo");
        const int n = q.n, steps = q.nt - 1;
        const T *coef = static_cast<const T *>(q.coef), *init = static_cast<const T *>(q.initial);
        const T *bnd = static_cast<const T *>(q.boundary);
        host_tables<T> &tb = tabs[i];
        tb.coef.assign(coef, coef + 3 * static_cast<size_t>(n));
        tb.init.assign(init, init + n);
        tb.bnd.resize(2 * static_cast<size_t>(steps));
        for (int s = 0; s < steps; ++s) {
            if (bnd[4 * s + 1] != bnd[1] || bnd[4 * s + 3] != bnd[3])
                return set_error(LSS_ADI_EUNSUPPORTED, "heat1d: Robin linear values must not change in time");
            tb.bnd[2 * s] = bnd[4 * s];
            tb.bnd[2 * s + 1] = bnd[4 * s + 2];
        }
        if (q.source) {
            const T *src = static_cast<const T *>(q.source);
            tb.src.assign(src, src + static_cast<size_t>(q.nt) * n);
        }
        inst_info &f = info[i];
        f.n = n;
        f.nt = q.nt;
        f.lo_kind = q.lo_kind;
        f.hi_kind = q.hi_kind;
        f.has_src = q.source ? 1 : 0;
        f.forward = q.forward ? 1 : 0;
        f.theta_scheme = q.theta_scheme;
        f.t_lo = q.t_lo;
        f.t_hi = q.t_hi;
        f.lo_lin = q.lo_kind == LSS_HEAT1D_ROBIN ? static_cast<double>(bnd[1]) : 0.0;
        f.hi_lin = q.hi_kind == LSS_HEAT1D_ROBIN ? static_cast<double>(bnd[3]) : 0.0;
        f.eval_i = n / 2; // value = the solution's middle point (n >= 4: n/2 + 1 < n)
        f.eval_w = 0.0;
    }
    auto bt = std::make_unique<batch_t<T>>();
    bt->precision = std::is_same<T, double>::value ? LSS_ADI_FP64 : LSS_ADI_FP32;
    bt->arith = arith;
    bt->options = options;
    bt->ds = (options & LSS_HEAT1D_OPT_DOUBLE_SWEEP) != 0;
    int rc = bt->build(std::move(info), tabs);
    if (rc != LSS_ADI_OK) return rc;
    auto *h = new (std::nothrow) lss_heat1d_batch;
    if (!h) return set_error(LSS_ADI_ENOMEM, "heat1d: host allocation");
    h->impl = std::move(bt);
    *b = h;
    return LSS_ADI_OK;
}

template <typename T>
static int create_bs(const lss_heat1d_bs *ps, int count, int arith, int options, lss_heat1d_batch **b)
{
    for (int i = 0; i < count; ++i) {
        const lss_heat1d_bs &q = ps[i];
        if (q.n < 4 || q.nt < 2) return set_error(LSS_ADI_EINVAL, "heat1d: n must be >= 4 and nt >= 2");
        if (!check_theta(q.theta_scheme))
            return set_error(LSS_ADI_EINVAL, "heat1d: the implicit 1-D kernel accepts Euler and Crank-Nicolson only");
        if (!(q.s_hi > q.s_lo) || !(q.maturity > 0.0) || !(q.sigma > 0.0))
            return set_error(LSS_ADI_EINVAL, "heat1d: invalid Black-Scholes problem (ranges, maturity, sigma)");
        if (q.nonuniform && !(q.alpha_scale > 0.0)) return set_error(LSS_ADI_EINVAL, "heat1d: alpha_scale must be > 0");
    }
    std::vector<inst_info> info(count);
    std::vector<host_tables<T>> tabs(count);
    const unsigned hw = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    const int nthr = static_cast<int>(std::min<long long>(hw, count));
    run_shares(static_cast<unsigned>(nthr), [&](unsigned w) {
        for (int i = static_cast<int>(w); i < count; i += nthr) bs_tables<T>(ps[i], tabs[i], info[i]);
    });
    auto bt = std::make_unique<batch_t<T>>();
    bt->precision = std::is_same<T, double>::value ? LSS_ADI_FP64 : LSS_ADI_FP32;
    bt->arith = arith;
    bt->options = options;
    bt->ds = (options & LSS_HEAT1D_OPT_DOUBLE_SWEEP) != 0;
    int rc = bt->build(std::move(info), tabs);
    if (rc != LSS_ADI_OK) return rc;
    auto *h = new (std::nothrow) lss_heat1d_batch;
    if (!h) return set_error(LSS_ADI_ENOMEM, "heat1d: host allocation");
    h->impl = std::move(bt);
    *b = h;
    return LSS_ADI_OK;
}

template <typename T> static int run_host_t(lss_heat1d_batch *b, const void *initials, double *values, int *status,
                                            cudaStream_t s)
{
    batch_t<T> *bt = as<T>(b);
    if (initials)
        LSS_CUDA_TRY(cudaMemcpyAsync(bt->d_init.p, initials, bt->total_init * sizeof(T), cudaMemcpyHostToDevice, s),
                     "heat1d: uploading initial conditions");
    int rc = bt->run(s);
    if (rc) return rc;
    if (values)
        LSS_CUDA_TRY(cudaMemcpyAsync(values, bt->d_values.p, bt->count * sizeof(double), cudaMemcpyDeviceToHost, s),
                     "heat1d: downloading values");
    if (status)
        LSS_CUDA_TRY(cudaMemcpyAsync(status, bt->d_status.p, bt->count * sizeof(int), cudaMemcpyDeviceToHost, s),
                     "heat1d: downloading status");
    LSS_CUDA_TRY(cudaStreamSynchronize(s), "heat1d: end-to-end step");
    return LSS_ADI_OK;
}

template <typename T> static int solution_t(lss_heat1d_batch *b, int index, void *out)
{
    batch_t<T> *bt = as<T>(b);
    const int gi = bt->inst_group[index], lane = bt->inst_lane[index];
    const h1group &G = bt->groups[gi];
    const inst_info &f = bt->info[index];
    const bool all = (bt->options & LSS_HEAT1D_OPT_ALL_STEPS) != 0;
    const long long rows = all ? f.nt : 1;
    const long long src_off = all ? G.all : G.pt + static_cast<long long>(S_U) * G.n * LANES;
    const T *src = all ? bt->d_all.p : bt->d_pt.p;
    // strided copy: element t of row r at src_off + (r*n + t)*32 + lane
    LSS_CUDA_TRY(cudaMemcpy2D(out, sizeof(T), src + src_off + lane, LANES * sizeof(T), sizeof(T), rows * f.n,
                              cudaMemcpyDeviceToHost),
                 "heat1d: downloading a solution");
    return LSS_ADI_OK;
}

extern "C" {

int lss_heat1d_batch_create(const lss_heat1d_tables *problems, int count, int precision, int arith, int options,
                            lss_heat1d_batch **b)
{
    clear_error();
    int rc = valid_common(count, precision, arith, options, b);
    if (rc) return rc;
    if (!problems) return set_error(LSS_ADI_EINVAL, "heat1d: problems is NULL");
    try {
        return precision == LSS_ADI_FP64 ? create_tab<double>(problems, count, arith, options, b)
                                         : create_tab<float>(problems, count, arith, options, b);
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "heat1d: host allocation failed");
    }
}

int lss_heat1d_batch_create_bs(const lss_heat1d_bs *problems, int count, int precision, int arith, int options,
                               lss_heat1d_batch **b)
{
    clear_error();
    int rc = valid_common(count, precision, arith, options, b);
    if (rc) return rc;
    if (!problems) return set_error(LSS_ADI_EINVAL, "heat1d: problems is NULL");
    try {
        return precision == LSS_ADI_FP64 ? create_bs<double>(problems, count, arith, options, b)
                                         : create_bs<float>(problems, count, arith, options, b);
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "heat1d: host allocation failed");
    }
}

int lss_heat1d_batch_run(lss_heat1d_batch *b, void *stream)
{
    if (!b) return set_error(LSS_ADI_EINVAL, "heat1d: batch is NULL");
    clear_error();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    b->last = s;
    return b->impl->precision == LSS_ADI_FP64 ? as<double>(b)->run(s) : as<float>(b)->run(s);
}

int lss_heat1d_batch_run_host(lss_heat1d_batch *b, const void *initials, double *values, int *status, void *stream)
{
    if (!b) return set_error(LSS_ADI_EINVAL, "heat1d: batch is NULL");
    clear_error();
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    b->last = s;
    return b->impl->precision == LSS_ADI_FP64 ? run_host_t<double>(b, initials, values, status, s)
                                              : run_host_t<float>(b, initials, values, status, s);
}

int lss_heat1d_batch_results(lss_heat1d_batch *b, double *values, int *status)
{
    if (!b) return set_error(LSS_ADI_EINVAL, "heat1d: batch is NULL");
    clear_error();
    LSS_CUDA_TRY(cudaStreamSynchronize(b->last), "heat1d: waiting for the run");
    const int count = b->impl->count;
    if (b->impl->precision == LSS_ADI_FP64) {
        auto *bt = as<double>(b);
        if (values) LSS_CUDA_TRY(cudaMemcpy(values, bt->d_values.p, count * sizeof(double), cudaMemcpyDeviceToHost), "heat1d: values");
        if (status) LSS_CUDA_TRY(cudaMemcpy(status, bt->d_status.p, count * sizeof(int), cudaMemcpyDeviceToHost), "heat1d: status");
    } else {
        auto *bt = as<float>(b);
        if (values) LSS_CUDA_TRY(cudaMemcpy(values, bt->d_values.p, count * sizeof(double), cudaMemcpyDeviceToHost), "heat1d: values");
        if (status) LSS_CUDA_TRY(cudaMemcpy(status, bt->d_status.p, count * sizeof(int), cudaMemcpyDeviceToHost), "heat1d: status");
    }
    return LSS_ADI_OK;
}

int lss_heat1d_batch_solution(lss_heat1d_batch *b, int index, void *out)
{
    if (!b || !out) return set_error(LSS_ADI_EINVAL, "heat1d: NULL argument");
    if (index < 0 || index >= b->impl->count) return set_error(LSS_ADI_EINVAL, "heat1d: index out of range");
    clear_error();
    LSS_CUDA_TRY(cudaStreamSynchronize(b->last), "heat1d: waiting for the run");
    return b->impl->precision == LSS_ADI_FP64 ? solution_t<double>(b, index, out) : solution_t<float>(b, index, out);
}

int lss_heat1d_batch_grid(const lss_heat1d_batch *b, int index, void *x)
{
    if (!b || !x) return set_error(LSS_ADI_EINVAL, "heat1d: NULL argument");
    if (index < 0 || index >= b->impl->count) return set_error(LSS_ADI_EINVAL, "heat1d: index out of range");
    if (b->impl->precision == LSS_ADI_FP64) {
        auto *bt = static_cast<const batch_t<double> *>(b->impl.get());
        if (bt->grids.size() != static_cast<size_t>(bt->count)) return set_error(LSS_ADI_EINVAL, "heat1d: not a Black-Scholes batch");
        std::copy(bt->grids[index].begin(), bt->grids[index].end(), static_cast<double *>(x));
    } else {
        auto *bt = static_cast<const batch_t<float> *>(b->impl.get());
        if (bt->grids.size() != static_cast<size_t>(bt->count)) return set_error(LSS_ADI_EINVAL, "heat1d: not a Black-Scholes batch");
        std::copy(bt->grids[index].begin(), bt->grids[index].end(), static_cast<float *>(x));
    }
    return LSS_ADI_OK;
}

int lss_heat1d_batch_launch_count(const lss_heat1d_batch *b)
{
    if (!b) return 0;
    return b->impl->launches();
}

double lss_heat1d_batch_point_steps(const lss_heat1d_batch *b) { return b ? b->impl->point_steps : 0.0; }

void lss_heat1d_batch_destroy(lss_heat1d_batch *b) { delete b; }

} // extern "C"
