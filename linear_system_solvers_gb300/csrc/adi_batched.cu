// adi_batched.cu -- many uneven ADI instances advanced by one persistent kernel.
//
// Each CTA is cut into warp groups of 1-4 warps; a group pulls an instance index from its
// class's device counter (instances sorted longest first), runs that instance's whole time
// loop with the group's own barrier between the sweeps, then pulls the next one.  The
// time-invariant line systems of every instance are
// factorised once on the device (k_setup_s_lines / k_setup_v_lines): the time loop only
// does the pre-scaled right-hand side, one FMA of forward recurrence and one of back
// substitution per point, because GB300's FP64 pipe (~1.25 TFLOP/s measured) and not HBM
// is the binding resource.  Same time-step structure as the reference
// (implicit_heston_time_loop::run, lss_2d_general_heston_equation_implicit_kernel.hpp:150-207).
#include <algorithm>
#include <cmath>
#include <memory>
#include <numeric>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "adi_batched.hpp"
#include "adi_index.hpp"
#include "adi_threads.hpp"

namespace lss_gb300 {

// slots of the FP32 S-line tables ([t][slot][j], pitch ld)
enum {
    SL_LA = 0, SL_G, SL_WG, SL_WW, SL_WS, SL_WC, SL_WN, SL_WE,
    SL_S2SC, SL_S2SE, SL_S2IB, SL_S2MZ, SL_X1, SL_X2, SL_X3, SL_X4, SL_X5, SL_IB, SL_COUNT
};
// and v-line tables ([t][slot][i]: i fastest)
enum { VL_LA = 0, VL_G, VL_VC, VL_VN, VL_IB, VL_COUNT };
// slots of the FP64 line tables: S lines [t][slot][j] (pitch ld), v lines [t][slot][i] (pitch nx)
enum { DS_LA = 0, DS_G, DS_WG, DS_WW, DS_WS, DS_WQ, DS_WN, DS_WE, DS_IB, DS_WC, DS_COUNT };
enum { DV_L = 0, DV_U, DV_IB, DV_COUNT };
template <typename T> __host__ __device__ constexpr int s_slots() { return sizeof(T) == 8 ? static_cast<int>(DS_COUNT) : static_cast<int>(SL_COUNT); }
template <typename T> __host__ __device__ constexpr int v_slots() { return sizeof(T) == 8 ? static_cast<int>(DV_COUNT) : static_cast<int>(VL_COUNT); }
// per-instance 1-D arrays along S (nx each).  Adjoint only, coefficient derivatives split into
// S and v factors: X_HX = S/A (dd^/dr), X_HC = S-factor of c^ (Heston S/A, SABR F^beta/A),
// X_HA = F^(2 beta)/A^2 and X_HDD = F^(2 beta) A''/A^3 (SABR D(t) terms of a^ and d^)
enum { XB_M = 0, XB_C, XB_P, XB_2, XB_1, X_VHI, X_CHV, X_HX, X_HC, X_HA, X_HDD, X_COUNT };
// per-instance 1-D arrays along v (ny each).  Adjoint only: Y_HY = v-factor of c^ (Heston v/B,
// SABR v^2/B), Y_BS = db^/dsigma, Y_EK = de^/dkappa, Y_ET = de^/dtheta, Y_ES = de^/dsigma,
// Y_HV2 = v^2/2 (SABR D(t) terms)
enum { Y_SLO = 0, Y_B2C, Y_CHS, Y_HY, Y_BS, Y_EK, Y_ET, Y_ES, Y_HV2, Y_COUNT };

struct bdesc {
    int nx, ny, steps, scheme;
    int ld, pad0_; // row pitch of the state and the S-line tables (a multiple of 32 bytes)
    long long o2;  // offset of the instance in the nx*ld arenas
    long long op;  // offset in the nx*ny arena of initial conditions
    int ox, oy;    // offsets in the nx- and ny-sized arenas
    double bnc;    // constant of the Neumann-corner boundary row
    int i0, j0;    // bilinear cell of (eval_s, eval_v)
    double w00, w10, w01, w11;
    int ck;        // checkpoint interval of the adjoint (steps)
    int pad_;
    // scalars of the parameter derivatives: delta, k/2, ni, beta~, sigma, rho, theta, zeta, gamma, k
    double a_delta, a_halfk, a_ni, a_betat, a_sigma, a_rho, a_theta, a_zeta, a_gamma, a_k;
    // SABR (r = 0): dD^p/dr = -p tau with tau = T - t = a_tau0 + a_dtau * step; alpha~, 1 - beta
    int model, pad2_;
    double a_alphat, a_omb, a_tau0, a_dtau;
};

// Instances are split into classes by the number of warps that work on one of them (1..4 for
// the persistent kernels: about one thread per S line).  Class c's instances are
// order[cls_start[c] .. cls_start[c] + cls_count[c]), longest first, pulled through counter[c].
constexpr int MAX_GROUP_WARPS = 4;

template <typename T> struct bparams {
    const bdesc *desc;
    const int *order;
    int count;
    int *counter;                     // one work counter per class (index 1..4)
    int cls_start[MAX_GROUP_WARPS + 1], cls_count[MAX_GROUP_WARPS + 1];
    long long cls_need[MAX_GROUP_WARPS + 1]; // largest adjoint workspace (doubles) of a class's instances
    const int *layout;                // per CTA: sizes of its warp groups, one hex digit each, lowest first
    T *U, *V, *Y1, *Y2, *Y3;          // state arenas (sum nx*ny each)
    T *B0;                            // nx arena: the explicit v = v_lo boundary column of a step
    const T *S, *Vt;                  // S- and v-direction tables (inst_view)
    const T *X[X_COUNT];              // nx arenas
    const T *Yv[Y_COUNT];             // ny arenas
    const int *imap, *jmap;           // nx / ny arenas
    double *values;                   // count
    int *status;                      // count
    int *final_in_v;                  // count: 1 if the final surface is in V
    // forward + adjoint (mode 1, FP64 only)
    double *grads;                    // 5 * count: d value / d(kappa, theta, sigma, rho, r)
    double *ws;                       // adjoint workspace: a slice of ws_per_warp doubles per warp
    long long ws_per_warp;            // a group of w warps owns w consecutive slices
    const T *payoff;                  // sum nx*ny initial conditions
};

// The warps of one CTA that work on one instance together, synchronised by their own named
// barrier (a one-warp group by __syncwarp), so that the groups of a CTA run independently.
struct grp {
    int t;      // thread index in the group
    int n;      // threads in the group (a multiple of 32)
    int gi;     // group index in the CTA (barrier 1 + gi)
    int warp0;  // first warp of the group in the CTA
    __device__ __forceinline__ void sync() const
    {
        // constant barrier ids: a run-time id makes the compiler reserve all 16 of the CTA's
        // named barriers, which would cap the CTAs per SM at 4
        if (n == 32) {
            __syncwarp();
        } else {
            switch (gi) {
            case 0: __barrier_sync_count(1, n); break;
            case 1: __barrier_sync_count(2, n); break;
            case 2: __barrier_sync_count(3, n); break;
            default: __barrier_sync_count(4, n); break;
            }
        }
    }
};

// This thread's group from the CTA's layout word (group sizes in warps, one hex digit each).
__device__ __forceinline__ grp make_grp(int layout)
{
    const int w = threadIdx.x >> 5;
    int first = 0, gi = 0, size = layout & 15;
    while (size > 0 && w >= first + size) {
        first += size;
        layout >>= 4;
        size = layout & 15;
        ++gi;
    }
    grp g;
    g.gi = gi;
    g.warp0 = first;
    g.n = 32 * (size > 0 ? size : 1);
    g.t = threadIdx.x - 32 * first;
    return g;
}

// Next instance for a group whose home class is `cls` (updated in place as classes run dry):
// its own class first, then the classes of fewer warps per instance; with max_need >= 0 only
// classes whose instances' workspace fits max_need doubles.  Called by the group's thread 0.
template <typename T>
__device__ __forceinline__ int next_instance(const bparams<T> &p, int &cls, long long max_need)
{
    while (cls >= 1) {
        if (p.cls_count[cls] > 0 && (max_need < 0 || p.cls_need[cls] <= max_need)) {
            const int q = atomicAdd(p.counter + cls, 1);
            if (q < p.cls_count[cls]) return p.order[p.cls_start[cls] + q];
        }
        --cls;
    }
    return -1;
}

// ------------------------------------------------------------------------------------------
// set-up: factorise the S-lines and v-lines of every instance once (double arithmetic)
// ------------------------------------------------------------------------------------------
struct setup_params {
    const bdesc *desc;
    const long long *line_start; // prefix of line counts per instance
    int count;
    long long total_lines;
    const double *base;          // 7 * sum(n): M, P, Z, Mt, Pt, W, C (each arena sum(n))
    long long total_n;
    const double *scal;          // per instance: theta, zeta, gamma
};

// The 18 S-line slots of one point from its coefficients, 1/beta and gamma (double arithmetic).
template <typename T>
__device__ __forceinline__ void s_line_slots(T *s, long long slot_stride, int scheme, double th, double ze, double gm,
                                             double M, double P, double Z, double Mt, double Pt, double W, double C,
                                             double ib, double gam)
{
    const double a = -th * M, c = -th * P;
    s[SL_LA * slot_stride] = static_cast<T>(a * ib);
    s[SL_G * slot_stride] = static_cast<T>(gam);
    s[SL_WG * slot_stride] = static_cast<T>(gm * C * ib);
    s[SL_WW * slot_stride] = static_cast<T>((1.0 - th) * M * ib);
    s[SL_WS * slot_stride] = static_cast<T>(Mt * ib);
    s[SL_WC * slot_stride] = static_cast<T>((1.0 - W - (1.0 - th) * Z) * ib);
    s[SL_WN * slot_stride] = static_cast<T>(Pt * ib);
    s[SL_WE * slot_stride] = static_cast<T>((1.0 - th) * P * ib);
    const double sc = th * Z * ib, se = c * ib;
    if (scheme == LSS_ADI_HUNDSDORFER_VERWER) {
        // fused HV stage: rhs4 + rhs_intermed_3 expressed in Delta = Y2 - U and Y1
        s[SL_S2SC * slot_stride] = static_cast<T>(sc + ib);
        s[SL_S2SE * slot_stride] = static_cast<T>(se);
        s[SL_S2IB * slot_stride] = static_cast<T>(0.0);
        s[SL_S2MZ * slot_stride] = static_cast<T>(ze * gm * C * ib);
        s[SL_X1 * slot_stride] = static_cast<T>(a * ib + ze * M * ib);
        s[SL_X2 * slot_stride] = static_cast<T>(sc - ze * (W + Z) * ib);
        s[SL_X3 * slot_stride] = static_cast<T>(se + ze * P * ib);
        s[SL_X4 * slot_stride] = static_cast<T>(ze * Mt * ib);
        s[SL_X5 * slot_stride] = static_cast<T>(ze * Pt * ib);
    } else {
        const double zt = (scheme == LSS_ADI_MODIFIED_CRAIG_SNEYD) ? (ze - th) : 0.0;
        s[SL_S2SC * slot_stride] = static_cast<T>(sc);
        s[SL_S2SE * slot_stride] = static_cast<T>(se);
        s[SL_S2IB * slot_stride] = static_cast<T>(ib);
        s[SL_S2MZ * slot_stride] = static_cast<T>(ze * gm * C * ib);
        s[SL_X1 * slot_stride] = static_cast<T>(zt * M * ib);
        s[SL_X2 * slot_stride] = static_cast<T>(-zt * (Z + W) * ib);
        s[SL_X3 * slot_stride] = static_cast<T>(-zt * P * ib);
        s[SL_X4 * slot_stride] = static_cast<T>(zt * Mt * ib);
        s[SL_X5 * slot_stride] = static_cast<T>(zt * Pt * ib);
    }
    s[SL_IB * slot_stride] = static_cast<T>(ib);
}

template <typename T>
__global__ void k_setup_s_lines(setup_params sp, T *S0, T *chS_arena)
{
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= sp.total_lines) return;
    int inst = 0;
    { // binary search the instance owning global line g
        int lo = 0, hi = sp.count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sp.line_start[mid] <= g) lo = mid; else hi = mid - 1;
        }
        inst = lo;
    }
    const bdesc d = sp.desc[inst];
    const int j = 1 + static_cast<int>(g - sp.line_start[inst]);
    const int ld = d.ld, e = d.nx - 2;
    const double th = sp.scal[3 * inst], ze = sp.scal[3 * inst + 1], gm = sp.scal[3 * inst + 2];
    const long long N = sp.total_n;
    const double *__restrict__ bM = sp.base, *__restrict__ bP = sp.base + N, *__restrict__ bZ = sp.base + 2 * N,
                 *__restrict__ bMt = sp.base + 3 * N, *__restrict__ bPt = sp.base + 4 * N,
                 *__restrict__ bW = sp.base + 5 * N, *__restrict__ bC = sp.base + 6 * N;
    // the next point's coefficients are loaded before this point's eighteen stores, so that one
    // DRAM latency per point overlaps the work of the point before (the loop is serial along the
    // line, and an instance has few lines; made once, for FP32 batches and FP32 instances with a
    // thread per line)
    long long o1 = d.o2 + ld + j;
    double nM = bM[o1], nP = bP[o1], nZ = bZ[o1], nMt = bMt[o1], nPt = bPt[o1], nW = bW[o1], nC = bC[o1];
    double gam = 0.0;
    for (int t = 1; t <= e; ++t) {
        const long long o = d.o2 + (long long)t * ld + j;
        const double M = nM, P = nP, Z = nZ, Mt = nMt, Pt = nPt, W = nW, C = nC;
        if (t < e) {
            o1 = o + ld;
            nM = bM[o1]; nP = bP[o1]; nZ = bZ[o1]; nMt = bMt[o1]; nPt = bPt[o1]; nW = bW[o1]; nC = bC[o1];
        }
        const double a = -th * M, b = 1.0 + th * Z, c = -th * P;
        const double beta = (t == 1) ? b : b - a * gam;
        const double ib = 1.0 / beta;
        if (t < e) gam = c / beta;
        s_line_slots<T>(S0 + d.o2 * SL_COUNT + (long long)t * SL_COUNT * ld + j, ld, d.scheme, th, ze, gm, M, P, Z, Mt, Pt, W, C, ib, t < e ? gam : 0.0);
        if (t == e) chS_arena[d.oy + j] = static_cast<T>(c * ib);
    }
}

template <typename T>
__global__ void k_setup_v_lines(setup_params sp, T *V0, T *chV_arena)
{
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= sp.total_lines) return;
    int lo = 0, hi = sp.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sp.line_start[mid] <= g) lo = mid; else hi = mid - 1;
    }
    const int inst = lo;
    const bdesc d = sp.desc[inst];
    const int i = 1 + static_cast<int>(g - sp.line_start[inst]);
    const int nx = d.nx, e = d.ny - 2;
    const double th = sp.scal[3 * inst];
    const long long N = sp.total_n;
    const double *bMt = sp.base + 3 * N, *bPt = sp.base + 4 * N, *bW = sp.base + 5 * N;
    double gam = 0.0;
    for (int t = 1; t <= e; ++t) {
        const long long ob = d.o2 + (long long)i * d.ld + t;  // base tables are [i][j]
        const double a = -th * bMt[ob], b = 1.0 + th * bW[ob], c = -th * bPt[ob];
        const double beta = (t == 1) ? b : b - a * gam;
        const double ib = 1.0 / beta;
        if (t < e) gam = c / beta;
        T *s = V0 + d.o2 * VL_COUNT + (long long)t * VL_COUNT * nx + i; // v tables are [t][slot][i]
        s[VL_LA * nx] = static_cast<T>(a * ib);
        s[VL_G * nx] = static_cast<T>(t < e ? gam : 0.0);
        s[VL_VC * nx] = static_cast<T>(th * bW[ob] * ib);
        s[VL_VN * nx] = static_cast<T>(c * ib);
        s[VL_IB * nx] = static_cast<T>(ib);
        if (t == e) chV_arena[d.ox + i] = static_cast<T>(c * ib);
    }
}

// The same in delta form (FP64; the tables of adi_wide.cuh, v lines transposed to [t][i]).
__device__ __forceinline__ int setup_instance(const setup_params &sp, long long g)
{
    int lo = 0, hi = sp.count - 1; // the instance owning global line g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sp.line_start[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}
static __global__ void k_setup_s_delta(setup_params sp, double *S0);
static __global__ void k_setup_v_delta(setup_params sp, double *V0);

// ------------------------------------------------------------------------------------------
// the persistent time-loop kernel
// ------------------------------------------------------------------------------------------
// One instance's view of the arenas.  The arena base pointers stay in the kernel's parameter
// space (__grid_constant__), so they cost no registers; only the offsets are carried.
// FAR: FP32 rows of any length (adi_index.hpp).
template <typename T, bool FAR = false> struct inst_view {
    const bparams<T> *p;
    int nx, ny, ld, e_s, e_v;
    long long o2;
    int ox, oy;
    long long so, vo; // line tables
    table_index<s_slots<T>(), FAR> si;
    table_index<v_slots<T>(), FAR> vi;
    // line tables of the instance: row t of the S lines holds all its slots, column t of the v lines too (a
    // row's operands lie within a few KB instead of ten arenas: 5 to 15 % where a GPU full of 256 x 128
    // instances reads them from HBM)
    __device__ __forceinline__ const T *S(int k, int t, int j) const { return p->S + so + si.at(t, k, j); }
    __device__ __forceinline__ const T *Vt(int k, int t, int i) const { return p->Vt + vo + vi.at(t, k, i); }
    __device__ __forceinline__ const T *X(int k) const { return p->X[k] + ox; }
    __device__ __forceinline__ const T *Yv(int k) const { return p->Yv[k] + oy; }
    __device__ __forceinline__ const int *imap() const { return p->imap + ox; }
    __device__ __forceinline__ const int *jmap() const { return p->jmap + oy; }
};

template <typename T> __device__ __forceinline__ T ldg(const T *p) { return __ldg(p); }

// Explicitly rounded products and fused multiply-adds: the FP32 stages, whose results keep their bits,
// round the same way whatever the compiler would contract.
__device__ __forceinline__ float mul_x(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma_x(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// One point of the v-line forward recurrence: y_t = la a0 + vc a1 + vn a2 + ib h - la y_{t-1}
// (a0, a1, a2: `in` at t-1, t, t+1; h: `inh` at t).
__device__ __forceinline__ float v_point(float la, float vc, float vn, float ib, float a0, float a1, float a2, float h, float y)
{
    float f = mul_x(la, a0);
    f = fma_x(vc, a1, f);
    f = fma_x(vn, a2, f);
    f = fma_x(ib, h, f);
    return fma_x(-la, y, f);
}

// boundary#1: the v = v_lo column, explicit (explicit_boundary.hpp:39-84); result in smem
// Work distribution of every stage: items l0, l0 + ls, ... (threads of one CTA in the
// batched kernel; all threads of a grid in the per-stage kernels of the wide path).
template <typename T, bool FAR>
__device__ __forceinline__ void b1_stage(const inst_view<T, FAR> &v, const T *__restrict__ U, T *__restrict__ sb0, double bnc,
                                         int l0, int ls)
{
    const int nx = v.nx, ld = v.ld, N = nx - 1;
    for (int i = l0; i < nx; i += ls) {
        T r;
        if (i == 0) {
            r = ldg(v.Yv(Y_SLO));
        } else if (i == N) {
            r = ldg(v.X(XB_C) + i) * U[(long long)N * ld] + ldg(v.X(XB_1) + i) * U[(long long)N * ld + 1] +
                ldg(v.X(XB_2) + i) * U[(long long)N * ld + 2] + static_cast<T>(bnc);
        } else {
            const long long o = (long long)i * ld;
            r = ldg(v.X(XB_M) + i) * U[o - ld] + ldg(v.X(XB_C) + i) * U[o] + ldg(v.X(XB_P) + i) * U[o + ld] +
                ldg(v.X(XB_2) + i) * U[o + 2] + ldg(v.X(XB_1) + i) * U[o + 1];
        }
        sb0[i] = r;
    }
}

// boundary#2: row S_lo and the S_max extrapolation row (explicit_boundary.hpp:202-238)
template <typename T, bool FAR> __device__ __forceinline__ void b2_stage(const inst_view<T, FAR> &v, T *Vn, int l0, int ls)
{
    const int nx = v.nx, ny = v.ny, ld = v.ld, lri = nx - 1;
    const T four3 = T(4.0 / 3.0), third = T(1.0 / 3.0);
    for (int j = l0; j < ny; j += ls) {
        Vn[j] = ldg(v.Yv(Y_SLO) + j);
        const int jj = ldg(v.jmap() + j);
        Vn[(long long)lri * ld + j] =
            four3 * Vn[(long long)(lri - 1) * ld + jj] - third * Vn[(long long)(lri - 2) * ld + jj] - ldg(v.Yv(Y_B2C) + j);
    }
}

// Rows that a thread of the batched kernels loads ahead: AH of the right-hand sides, blocks of BK in the
// one-instruction passes, VB4 blocks of four columns in the v lines' scaled passes (FP64), two blocks of
// eight columns or none (FP32).
struct deep {
    static constexpr int AH = 5, BK = 16, VB4 = 4;
    static constexpr bool FAR = false;
};
// FP32 rows of tables beyond NEAR_PITCH (the kernels of one instance with a thread per line always take it)
struct deep_far : deep {
    static constexpr bool FAR = true;
};
struct shallow {
    static constexpr int AH = 1, BK = 4, VB4 = 1;
    static constexpr bool FAR = false;
};

// Stages of the FP32 instances, written on Y1, Y2, Y3 (their values keep that form's rounding; FP64
// runs in delta form, adi_delta.cuh).
//
// S-line sweeps.  KIND 1: explicit operator on U (Y1).  KIND 2: second S stage of CS/MCS/HV
// (scheme SCH) on U, Y1, Y2.  Thread per line j; every access of a warp is one coalesced row
// segment.  The mixed difference (x(t-1,j-1) - x(t-1,j+1)) - (x(t+1,j-1) - x(t+1,j+1)) is formed
// from a rolling window of the per-row differences x(r,j-1) - x(r,j+1): one subtraction per row.
//
// The next rows' operands are loaded before the current ones are used (five rows ahead, 16 in the back
// substitution); the fused multiply-adds are written out, so the rounding hangs on no contraction.
template <int KIND, int SCH, typename DEPTH = deep, bool FAR>
__device__ __forceinline__ void s_stage(const inst_view<float, FAR> &v, const float *U, const float *Y1, const float *Y2, float *Y, int l0, int ls)
{
    constexpr bool xt = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD || SCH == LSS_ADI_HUNDSDORFER_VERWER;
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER;
    constexpr int FA = DEPTH::AH, FK = DEPTH::BK;
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = v.e_s, last = (nx - 1) * ld;
    struct row { // tables of row t, state of row t + 1
        float la, w[10];
        float um, uc, up;  // KIND 1: U; else Y2 - U (side columns; centre: xt) and
        float uu, y1;      // U, Y1 at the centre
    };
    for (int j = 1 + l0; j <= ny - 2; j += ls) {
        const int jj = ldg(v.jmap() + j);
        const float lo = U[jj], hi = U[last + jj];
        auto load = [&](int t) -> row {
            const int o2 = (t + 1) * ld + j;
            row r;
            r.la = ldg(v.S(SL_LA, t, j));
            if constexpr (KIND == 1) {
                r.w[0] = ldg(v.S(SL_WG, t, j));
                r.w[1] = ldg(v.S(SL_WW, t, j));
                r.w[2] = ldg(v.S(SL_WS, t, j));
                r.w[3] = ldg(v.S(SL_WC, t, j));
                r.w[4] = ldg(v.S(SL_WN, t, j));
                r.w[5] = ldg(v.S(SL_WE, t, j));
                r.um = U[o2 - 1];
                r.uc = U[o2];
                r.up = U[o2 + 1];
            } else {
                r.w[0] = ldg(v.S(SL_S2SC, t, j));
                r.w[1] = ldg(v.S(SL_S2SE, t, j));
                r.w[2] = ldg(v.S(SL_S2MZ, t, j));
                if constexpr (!hv) r.w[3] = ldg(v.S(SL_S2IB, t, j));
                if constexpr (xt) {
                    r.w[4] = ldg(v.S(SL_X1, t, j));
                    r.w[5] = ldg(v.S(SL_X2, t, j));
                    r.w[6] = ldg(v.S(SL_X3, t, j));
                    r.w[7] = ldg(v.S(SL_X4, t, j));
                    r.w[8] = ldg(v.S(SL_X5, t, j));
                }
                r.uu = U[o2];
                r.um = Y2[o2 - 1] - U[o2 - 1];
                r.up = Y2[o2 + 1] - U[o2 + 1];
                if constexpr (xt) r.uc = Y2[o2] - r.uu;
                r.y1 = Y1[o2];
            }
            return r;
        };
        // rows t-1, t of the centre columns, side columns at row t, per-row differences of them
        float u0c, u1c, u1m, u1p, q0, q1, c0 = 0.0f, c1 = 0.0f, y10 = 0.0f, y11 = 0.0f;
        if constexpr (KIND == 1) {
            u0c = U[j];
            u1c = U[ld + j];
            u1m = U[ld + j - 1];
            u1p = U[ld + j + 1];
            q0 = U[j - 1] - U[j + 1];
        } else {
            c0 = U[j];
            c1 = U[ld + j];
            y10 = Y1[j];
            y11 = Y1[ld + j];
            u0c = Y2[j] - c0;
            u1c = Y2[ld + j] - c1;
            u1m = Y2[ld + j - 1] - U[ld + j - 1];
            u1p = Y2[ld + j + 1] - U[ld + j + 1];
            q0 = (Y2[j - 1] - U[j - 1]) - (Y2[j + 1] - U[j + 1]);
        }
        q1 = u1m - u1p;
        const float chs = ldg(v.Yv(Y_CHS) + j);
        float y = lo;
        auto point = [&](const row &r, int t) {
            const float q2 = r.um - r.up, mix = q0 - q2;
            float f;
            if constexpr (KIND == 1) {
                f = fma_x(r.w[0], mix, mul_x(r.w[1], u0c));
                f = fma_x(r.w[2], u1m, f);
                f = fma_x(r.w[3], u1c, f);
                f = fma_x(r.w[4], u1p, f);
                f = fma_x(r.w[5], r.uc, f);
            } else {
                if constexpr (hv) {
                    f = fma_x(r.la, y10, mul_x(r.w[0], y11));
                    f = fma_x(r.w[1], r.y1, f);
                } else {
                    f = fma_x(r.la, c0, mul_x(r.w[0], c1));
                    f = fma_x(r.w[1], r.uu, f);
                    f = fma_x(r.w[3], y11, f);
                }
                f = fma_x(r.w[2], mix, f);
                if constexpr (xt) {
                    f = fma_x(r.w[4], u0c, f);
                    f = fma_x(r.w[5], u1c, f);
                    f = fma_x(r.w[6], r.uc, f);
                    f = fma_x(r.w[7], u1m, f);
                    f = fma_x(r.w[8], u1p, f);
                }
                c0 = c1; c1 = r.uu;
                y10 = y11; y11 = r.y1;
            }
            y = fma_x(-r.la, y, f);
            if (t == e) y = fma_x(-chs, hi, y);
            Y[t * ld + j] = y;
            u0c = u1c; u1c = r.uc;
            u1m = r.um; u1p = r.up;
            q0 = q1; q1 = q2;
        };
        row ring[FA];
#pragma unroll
        for (int k = 0; k < FA; ++k) ring[k] = load(min(1 + k, e));
        int t = 1;
        for (; t + FA - 1 <= e; t += FA)
#pragma unroll
            for (int k = 0; k < FA; ++k) {
                const row next = load(min(t + k + FA, e));
                point(ring[k], t + k);
                ring[k] = next;
            }
#pragma unroll
        for (int k = 0; k < FA - 1; ++k)
            if (t + k <= e) point(ring[k], t + k);
        float x = y, yb[FK], gb[FK], yn[FK], gn[FK];
        auto block = [&](int t, float *yo, float *go) {
#pragma unroll
            for (int z = 0; z < FK; ++z) {
                const int r = max(t - z, 1);
                yo[z] = Y[r * ld + j];
                go[z] = ldg(v.S(SL_G, r, j));
            }
        };
        block(e - 1, yb, gb);
        for (t = e - 1; t >= 1; t -= FK) {
            block(t - FK, yn, gn);
#pragma unroll
            for (int z = 0; z < FK; ++z) {
                if (t - z >= 1) {
                    x = fma_x(-gb[z], x, yb[z]);
                    Y[(t - z) * ld + j] = x;
                }
                yb[z] = yn[z];
                gb[z] = gn[z];
            }
        }
        Y[j] = lo;
        Y[last + j] = hi;
    }
}

// The scheme as a template argument: calls f(std::integral_constant<int, SCH>{}).
template <typename F> __device__ __forceinline__ void with_scheme(int scheme, F &&f)
{
    switch (scheme) {
    case LSS_ADI_DOUGLAS_RACHFORD: f(std::integral_constant<int, LSS_ADI_DOUGLAS_RACHFORD>{}); break;
    case LSS_ADI_CRAIG_SNEYD: f(std::integral_constant<int, LSS_ADI_CRAIG_SNEYD>{}); break;
    case LSS_ADI_MODIFIED_CRAIG_SNEYD: f(std::integral_constant<int, LSS_ADI_MODIFIED_CRAIG_SNEYD>{}); break;
    default: f(std::integral_constant<int, LSS_ADI_HUNDSDORFER_VERWER>{}); break;
    }
}

// v-line sweep: line i reads row i of `in` (t-1, t, t+1) and `inh` (t); tables are [t][slot][i].  A lane walks
// its row eight columns at a time (256-bit loads and stores, rows padded to a multiple of eight: whole
// 32-byte sectors; with half of a sector per access a full GPU ran at half the speed), the next
// 16 columns and eight columns of tables ahead.
__device__ __forceinline__ void ldv(const float *p, float *o)
{
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
                 : "l"(p));
}
__device__ __forceinline__ void stv(float *p, const float *o)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(o[0]), "f"(o[1]), "f"(o[2]), "f"(o[3]), "f"(o[4]),
                 "f"(o[5]), "f"(o[6]), "f"(o[7])
                 : "memory");
}
template <typename DEPTH = deep, bool FAR>
__device__ __forceinline__ void v_stage(const inst_view<float, FAR> &v, const float *in, const float *inh, const float *sb0, float *out, int l0, int ls)
{
    constexpr bool ahead = DEPTH::VB4 > 1;
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = v.e_v;
    struct cols {
        float a[8], h[8];
    };
    struct tabs {
        float la[4], vc[4], vn[4], ib[4];
    };
    struct bbk {
        float y[8], g[8];
    };
    for (int i = 1 + l0; i <= nx - 2; i += ls) {
        const int ii = ldg(v.imap() + i), row = i * ld;
        const float lo = sb0[ii], hi = ldg(v.X(X_VHI) + ii), chv = ldg(v.X(X_CHV) + i);
        auto columns = [&](int t) -> cols { // columns t .. t + 7
            cols b;
            const int at = row + min(t, ld - 8);
            ldv(in + at, b.a);
            ldv(inh + at, b.h);
            return b;
        };
        auto tables = [&](int t) -> tabs { // of columns t .. t + 3
            tabs b;
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                const int c = min(max(t + z, 1), e);
                b.la[z] = ldg(v.Vt(VL_LA, c, i));
                b.vc[z] = ldg(v.Vt(VL_VC, c, i));
                b.vn[z] = ldg(v.Vt(VL_VN, c, i));
                b.ib[z] = ldg(v.Vt(VL_IB, c, i));
            }
            return b;
        };
        float y = lo, a0 = 0.0f;
        cols b, b2;
        tabs qr[2];
        if constexpr (ahead) {
            b = columns(0);
            b2 = columns(8);
            qr[0] = tables(0);
            qr[1] = tables(4);
        }
        for (int t = 0; t <= e; t += 8) {
            cols nb;
            if constexpr (ahead) {
                nb = b2;
                b2 = columns(t + 16);
            } else {
                b = columns(t);
                nb.a[0] = in[row + min(t + 8, ld - 1)];
            }
            float o[8];
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
                if constexpr (!ahead) qr[h / 4] = tables(t + h);
                const tabs q = qr[h / 4];
                if constexpr (ahead) qr[h / 4] = tables(t + h + 8);
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const int w = h + z, c = t + w;
                    const float a2 = w < 7 ? b.a[w < 7 ? w + 1 : 0] : nb.a[0];
                    if (c >= 1 && c <= e) {
                        y = v_point(q.la[z], q.vc[z], q.vn[z], q.ib[z], a0, b.a[w], a2, b.h[w], y);
                        if (c == e) y = fma_x(-chv, hi, y);
                    }
                    o[w] = y;
                    a0 = b.a[w];
                }
            }
            stv(out + row + t, o);
            if constexpr (ahead) b = nb;
        }
        float x = y;
        auto back = [&](int t) -> bbk {
            bbk k;
            ldv(out + row + max(t, 0), k.y);
#pragma unroll
            for (int z = 0; z < 8; ++z) k.g[z] = ldg(v.Vt(VL_G, min(max(t + z, 1), e), i));
            return k;
        };
        const int tl = (ny - 1) / 8 * 8;
        bbk k = back(tl), k2;
        if constexpr (ahead) k2 = back(tl - 8);
        for (int t = tl; t >= 0; t -= 8) {
            bbk nk;
            if constexpr (ahead) {
                nk = k2;
                k2 = back(t - 16);
            } else if (t >= 8) {
                nk = back(t - 8);
            }
            float o[8];
#pragma unroll
            for (int z = 7; z >= 0; --z) {
                const int c = t + z;
                if (c >= 1 && c < e) x = fma_x(-k.g[z], x, k.y[z]);
                o[z] = c >= 1 && c <= e ? x : c == 0 ? lo : c == ny - 1 ? hi : 0.0f;
            }
            stv(out + row + t, o);
            k = nk;
        }
    }
}

template <bool FAR, typename T> __device__ __forceinline__ inst_view<T, FAR> make_view(const bparams<T> &p, const bdesc &d)
{
    inst_view<T, FAR> v;
    v.p = &p;
    v.nx = d.nx;
    v.ny = d.ny;
    v.ld = d.ld;
    v.e_s = d.nx - 2;
    v.e_v = d.ny - 2;
    v.o2 = d.o2;
    v.si = table_index<s_slots<T>(), FAR>(d.ld);
    v.vi = table_index<v_slots<T>(), FAR>(d.nx);
    v.so = d.o2 * s_slots<T>() + v.si.base();
    v.vo = d.o2 * v_slots<T>() + v.vi.base();
    v.ox = d.ox;
    v.oy = d.oy;
    return v;
}

#include "adi_delta.cuh"

// One time step U -> Vn of scheme SCH with stage outputs in Y1, Y2, Y3; ends with a group barrier.
template <int SCH, typename DEPTH>
__device__ __forceinline__ void fwd_step(const inst_view<float, DEPTH::FAR> &v, const float *U, float *Y1, float *Y2, float *Y3, float *Vn, float *sb0,
                                         double bnc, const grp &g)
{
    const int l0 = g.t, ls = g.n;
    b1_stage<float>(v, U, sb0, bnc, l0, ls);
    s_stage<1, SCH, DEPTH>(v, U, nullptr, nullptr, Y1, l0, ls);
    g.sync();
    if constexpr (SCH == LSS_ADI_DOUGLAS_RACHFORD) {
        v_stage<DEPTH>(v, U, Y1, sb0, Vn, l0, ls);
    } else {
        v_stage<DEPTH>(v, U, Y1, sb0, Y2, l0, ls);
        g.sync();
        s_stage<2, SCH, DEPTH>(v, U, Y1, Y2, Y3, l0, ls);
        g.sync();
        if constexpr (SCH == LSS_ADI_HUNDSDORFER_VERWER)
            v_stage<DEPTH>(v, Y2, Y3, sb0, Vn, l0, ls);
        else
            v_stage<DEPTH>(v, U, Y3, sb0, Vn, l0, ls);
    }
    g.sync();
    b2_stage<float>(v, Vn, l0, ls);
    g.sync();
}

// Persistent forward kernel of the instances of scheme SCH: CTAs of 4 warps split into groups
// (the layout word of the CTA), each group pulling instances of its class (warps per instance)
// from the class counter.  FP64: two CTAs per SM, whose threads hold the rows that the sweeps load ahead
// (adi_delta.cuh).  FP32: three, 168 registers (768 uneven calls 49.9 ms with five rows ahead, 51.8 with
// four, 71 with six; two rows ahead with four CTAs of 128 registers 64.7 ms, a GPU full of equal 256 x 128
// instances alone 301 against 367 us a step).
constexpr int BATCH_CTA = 32 * MAX_GROUP_WARPS;

// value at (eval_s, eval_v), corner o of its cell
template <typename T> __device__ __forceinline__ double bilinear_value(const bdesc &d, const T *U, long long o)
{
    const double a = U[o], b = U[o + d.ld], c = U[o + 1], e = U[o + d.ld + 1];
    if (sizeof(T) == 8) return fma(d.w11, e, fma(d.w01, c, fma(d.w10, b, d.w00 * a)));
    return d.w00 * a + d.w10 * b + d.w01 * c + d.w11 * e;
}
// initial condition into the pitched state
template <typename T> __device__ __forceinline__ void load_payoff(const bparams<T> &p, const bdesc &d, T *U, const grp &g)
{
    for (int i = g.t / 32; i < d.nx; i += g.n / 32)
        for (int j = g.t & 31; j < d.ny; j += 32) U[i * d.ld + j] = p.payoff[d.op + (long long)i * d.ny + j];
}

template <typename T, int SCH, typename DEPTH>
__global__ void __launch_bounds__(BATCH_CTA, sizeof(T) == 8 && DEPTH::AH == deep::AH ? 2 : 3) k_batch_forward(const __grid_constant__ bparams<T> p)
{
    __shared__ int s_idx[MAX_GROUP_WARPS];
    __shared__ int s_bad[MAX_GROUP_WARPS];
    const grp g = make_grp(p.layout[blockIdx.x]);
    int cls = g.n / 32;
    while (true) {
        if (g.t == 0) s_idx[g.gi] = next_instance(p, cls, -1);
        g.sync();
        const int inst = s_idx[g.gi];
        g.sync();
        if (inst < 0) break;
        const bdesc d = p.desc[inst];
        const auto v = make_view<DEPTH::FAR>(p, d);
        T *U = p.U + d.o2, *Vn = p.V + d.o2, *Y1 = p.Y1 + d.o2, *Y2 = p.Y2 + d.o2, *Y3 = p.Y3 + d.o2;
        T *sb0 = p.B0 + d.ox;
        load_payoff(p, d, U, g);
        g.sync();
        for (int step = 0; step < d.steps; ++step) {
            if constexpr (sizeof(T) == 8) delta_step<SCH, DEPTH>(v, d, U, Y1, Y2, Y3, Vn, sb0, g);
            else fwd_step<SCH, DEPTH>(v, U, Y1, Y2, Y3, Vn, sb0, d.bnc, g);
            T *tmp = U;
            U = Vn;
            Vn = tmp;
        }
        // value at (eval_s, eval_v) and a finiteness check of the final surface
        if (g.t == 0) s_bad[g.gi] = 0;
        g.sync();
        const long long n = (long long)d.nx * d.ld; // the pitch's padding is zero
        int bad = 0;
        for (long long q = g.t; q < n; q += g.n) bad |= !isfinite(static_cast<double>(U[q]));
        if (bad) atomicOr(&s_bad[g.gi], 1);
        g.sync();
        if (g.t == 0) {
            const long long o = (long long)d.i0 * d.ld + d.j0;
            p.values[inst] = bilinear_value(d, U, o);
            p.status[inst] = s_bad[g.gi];
            p.final_in_v[inst] = d.steps & 1;
        }
        g.sync();
    }
}

// Forward + adjoint of each instance of scheme SCH by one warp group: forward pass keeping a checkpoint every
// d.ck steps (and the stage values of every step of the last segment), then per segment (last
// first) a forward recomputation that keeps the stage values of every step (not needed for the
// last segment), followed by the adjoint steps of the segment in reverse order.
// Results: value, the 5 parameter sensitivities, the final surface (state U arena) and
// dV/d(initial condition) (state V arena).  A group of w warps works in w consecutive workspace
// slices.  Two CTAs of 4 warps per SM, as the forward kernel.
template <int SCH>
__global__ void __launch_bounds__(BATCH_CTA, 2) k_batch_fwdadj(const __grid_constant__ bparams<double> p)
{
    __shared__ int s_idx[MAX_GROUP_WARPS];
    __shared__ int s_bad[MAX_GROUP_WARPS];
    __shared__ double red[MAX_GROUP_WARPS][5];
    const grp g = make_grp(p.layout[blockIdx.x]);
    const int gw = g.n / 32;
    double *ws = p.ws + (long long)(blockIdx.x * MAX_GROUP_WARPS + g.warp0) * p.ws_per_warp;
    int cls = gw;
    while (true) {
        if (g.t == 0) s_idx[g.gi] = next_instance(p, cls, gw * p.ws_per_warp);
        g.sync();
        const int inst = s_idx[g.gi];
        g.sync();
        if (inst < 0) break;
        const bdesc d = p.desc[inst];
        const inst_view<double> v = make_view<false>(p, d);
        const int nx = d.nx, ny = d.ny;
        const long long n = (long long)nx * d.ld;
        const int c = d.ck;
        const int nseg = (d.steps + c - 1) / c;
        double *sb0 = p.B0 + d.ox;
        // workspace carve-up
        double *CK = ws;                                  // nseg * n
        double *SEG = CK + (long long)nseg * n;           // (c + 1) * 4 * n: U, D1, D2, D3 of a step
        double *W0 = SEG + (long long)(c + 1) * 4 * n;    // n
        double *W1 = W0 + n;                              // n
        double *VB = W1 + n, *DB = VB + n, *FB = DB + n, *MU = FB + n, *DV = MU + n, *D2B = DV + n;
        double *LV = D2B + n, *LS = LV + nx, *HS = LS + ny;
        auto slot = [&](int m, int a) -> double * { return SEG + ((long long)m * 4 + a) * n; };

        // FB's boundary rows and columns are read as zeros
        for (long long q = g.t; q < n; q += g.n) FB[q] = VB[q] = 0.0;
        load_payoff(p, d, CK, g);
        g.sync();
        // forward pass with checkpoints; the steps of the last segment keep their stage increments in
        // the segment slots, so the reverse sweep starts without recomputing that segment
        const double *cur = CK;
        const int n0_last = (nseg - 1) * c;
        for (int step = 0; step < d.steps; ++step) {
            const bool keep = step >= n0_last;
            const int m = keep ? step - n0_last : 0;
            double *next = keep ? slot(m + 1, 0)
                                : (step + 1) % c == 0 ? CK + (long long)((step + 1) / c) * n : ((step & 1) ? W1 : W0);
            delta_step<SCH>(v, d, cur, slot(m, 1), slot(m, 2), slot(m, 3), next, sb0, g);
            cur = next;
        }
        // value, finiteness, final surface
        if (g.t == 0) s_bad[g.gi] = 0;
        g.sync();
        int bad = 0;
        double *outU = p.U + d.o2;
        for (int i = g.t / 32; i < nx; i += g.n / 32)
            for (int j = g.t & 31; j < ny; j += 32) {
                const double val = cur[i * d.ld + j];
                bad |= !isfinite(val);
                outU[i * d.ld + j] = val;
            }
        if (bad) atomicOr(&s_bad[g.gi], 1);
        g.sync();
        if (g.t == 0) {
            const long long o = (long long)d.i0 * d.ld + d.j0;
            p.values[inst] = bilinear_value(d, cur, o);
            p.status[inst] = s_bad[g.gi];
            p.final_in_v[inst] = 0;
            VB[o] = d.w00;
            VB[o + d.ld] = d.w10;
            VB[o + 1] = d.w01;
            VB[o + d.ld + 1] = d.w11;
        }
        g.sync();
        // reverse sweep over the segments
        adj_acc acc = {{0.0, 0.0, 0.0, 0.0, 0.0}};
        for (int sgi = nseg - 1; sgi >= 0; --sgi) {
            const int n0 = sgi * c;
            const int L = min(c, d.steps - n0);
            const double *u0 = CK + (long long)sgi * n;
            for (int m = 0; m < L && sgi < nseg - 1; ++m)
                delta_step<SCH>(v, d, m == 0 ? u0 : slot(m, 0), slot(m, 1), slot(m, 2), slot(m, 3), slot(m + 1, 0), sb0, g);
            for (int m = L - 1; m >= 0; --m)
                delta_adjoint<SCH>(v, d, m == 0 ? u0 : slot(m, 0), slot(m, 1), slot(m, 2), slot(m, 3), slot(m + 1, 0), VB, DB, FB, MU, DV,
                                   D2B, LV, LS, HS, acc, d.a_tau0 + d.a_dtau * (n0 + m), g);
        }
        // VB = adjoint of the initial condition
        double *outL = p.V + d.o2;
        for (long long q = g.t; q < n; q += g.n) outL[q] = VB[q];
        // order in the output: kappa, theta, sigma, rho, r
        double gr[5] = {acc.s[1], acc.s[2], acc.s[3], acc.s[4], acc.s[0]};
        // sum over the group: within each warp by shuffles, then the warps in order
        for (int q = 0; q < 5; ++q)
            for (int off = 16; off > 0; off >>= 1) gr[q] += __shfl_down_sync(0xffffffffu, gr[q], off);
        for (int w = 0; w < gw; ++w) {
            if (g.t == 32 * w)
                for (int q = 0; q < 5; ++q) red[g.gi][q] = (w == 0 ? 0.0 : red[g.gi][q]) + gr[q];
            g.sync();
        }
        if (g.t < 5) p.grads[5LL * inst + g.t] = red[g.gi][g.t];
        g.sync();
    }
}

// ------------------------------------------------------------------------------------------
// wide path: one instance, a thread per line and one kernel per stage over all threads of the grid,
// the batched kernel's stage arithmetic (bit-identical results; LSS_ADI_OPT_LINE_PER_THREAD)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int gtid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int gstride() { return gridDim.x * blockDim.x; }

template <typename T> __global__ void k_wide_b1(const __grid_constant__ bparams<T> p, const T *U, T *b0, T *Y2)
{
    const bdesc d = p.desc[0];
    const auto v = make_view<sizeof(T) == 4>(p, d);
    if constexpr (sizeof(T) == 8) {
        db1_stage(v, d, U, b0, gtid(), gstride());
        d2_edges(v, U, Y2, gtid(), gstride());
    } else {
        b1_stage<T>(v, U, b0, d.bnc, gtid(), gstride());
    }
}
template <typename T, int KIND>
__global__ void k_wide_s(const __grid_constant__ bparams<T> p, const T *U, const T *Y1, const T *Y2, T *Y)
{
    const bdesc d = p.desc[0];
    const auto v = make_view<sizeof(T) == 4>(p, d);
    with_scheme(d.scheme, [&](auto sch) {
        if constexpr (sizeof(T) == 8) ds_stage<KIND, decltype(sch)::value>(v, d, U, KIND == 1 ? U : Y2, Y1, Y, gtid(), gstride());
        else s_stage<KIND, decltype(sch)::value>(v, U, Y1, Y2, Y, gtid(), gstride());
    });
}
// the v stage after the S stage with result `s` (LAST: the step's last one)
template <typename T, bool LAST>
__global__ void k_wide_v(const __grid_constant__ bparams<T> p, const T *U, const T *Y1, const T *Y2, const T *s, const T *b0, T *out)
{
    const bdesc d = p.desc[0];
    const auto v = make_view<sizeof(T) == 4>(p, d);
    const bool hv = LAST && d.scheme == LSS_ADI_HUNDSDORFER_VERWER;
    if constexpr (sizeof(T) == 4) v_stage(v, hv ? Y2 : U, s, b0, out, gtid(), gstride());
    else if constexpr (!LAST) dv_stage<V_FIRST>(v, U, s, nullptr, nullptr, b0, out, gtid(), gstride());
    else if (hv) dv_stage<V_LAST_HV>(v, U, Y1, s, Y2, b0, out, gtid(), gstride());
    else dv_stage<V_LAST>(v, U, s, nullptr, nullptr, b0, out, gtid(), gstride());
}
template <typename T> __global__ void k_wide_b2(const __grid_constant__ bparams<T> p, T *Vn)
{
    const bdesc d = p.desc[0];
    const auto v = make_view<sizeof(T) == 4>(p, d);
    if constexpr (sizeof(T) == 8) db2_stage(v, Vn, gtid(), gstride());
    else b2_stage<T>(v, Vn, gtid(), gstride());
}
// value, finiteness flag and final-array flag of the single instance
// value at the evaluation point and finiteness of the final surface, grid-wide (the status word
// is cleared before the time loop; any block that sees a non-finite point sets it)
template <typename T> __global__ void k_wide_finish(const __grid_constant__ bparams<T> p, const T *U)
{
    const bdesc d = p.desc[0];
    const long long n = (long long)d.nx * d.ld;
    int b = 0;
    for (long long q = gtid(); q < n; q += gstride()) b |= !isfinite(static_cast<double>(U[q]));
    b = __syncthreads_or(b);
    if (b && threadIdx.x == 0) atomicOr(p.status, 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const long long o = (long long)d.i0 * d.ld + d.j0;
        p.values[0] = bilinear_value(d, U, o);
        p.final_in_v[0] = d.steps & 1;
    }
}

static __global__ void k_setup_s_delta(setup_params sp, double *S0)
{
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= sp.total_lines) return;
    const int inst = setup_instance(sp, g);
    const bdesc d = sp.desc[inst];
    const int j = 1 + static_cast<int>(g - sp.line_start[inst]);
    const int ld = d.ld, e = d.nx - 2;
    const double th = sp.scal[3 * inst], gm = sp.scal[3 * inst + 2];
    const long long N = sp.total_n;
    // the next row's coefficients are loaded before this row's stores
    double gam = 0.0, nv[7];
    long long o = d.o2 + ld + j;
    for (int k = 0; k < 7; ++k) nv[k] = sp.base[k * N + o];
    for (int t = 1; t <= e; ++t, o += ld) {
        const double M = nv[0], P = nv[1], Z = nv[2], Mt = nv[3], Pt = nv[4], W = nv[5], C = nv[6];
        if (t < e)
            for (int k = 0; k < 7; ++k) nv[k] = sp.base[k * N + o + ld];
        const double a = -th * M, b = 1.0 + th * Z, c = -th * P;
        const double ib = 1.0 / fma(-a, gam, b);
        gam = c * ib;
        const table_index<DS_COUNT> si(ld);
        double *tab = S0 + d.o2 * DS_COUNT + si.base();
        auto slot = [&](int k) -> double & { return tab[si.at(t, k, j)]; };
        slot(DS_LA) = a * ib;
        slot(DS_G) = gam;
        slot(DS_WG) = gm * C * ib;
        slot(DS_WW) = M * ib;
        const double ws = Mt * ib, wn = Pt * ib;
        slot(DS_WS) = ws;
        slot(DS_WQ) = center_weight<double>((M + P - Z) + ((Mt + Pt) - W), ib, ws, wn, t, j);
        slot(DS_WC) = -(Z + W) * ib;
        slot(DS_WN) = wn;
        slot(DS_WE) = P * ib;
        slot(DS_IB) = ib;
    }
}
static __global__ void k_setup_v_delta(setup_params sp, double *V0)
{
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= sp.total_lines) return;
    const int inst = setup_instance(sp, g);
    const bdesc d = sp.desc[inst];
    const int i = 1 + static_cast<int>(g - sp.line_start[inst]);
    const int nx = d.nx, e = d.ny - 2;
    const double th = sp.scal[3 * inst];
    const long long N = sp.total_n, row = d.o2 + (long long)i * d.ld;
    const double *Mt = sp.base + 3 * N + row, *Pt = sp.base + 4 * N + row, *W = sp.base + 5 * N + row;
    double *L = V0 + d.o2 * DV_COUNT + i, *U = L + DV_U * nx, *IB = L + DV_IB * nx;
    const long long row_t = (long long)DV_COUNT * nx;
    double ib = 0.0, cp = 0.0;
    for (int t = 1; t <= e; ++t) {
        const double a = -th * Mt[t], b = 1.0 + th * W[t], c = -th * Pt[t];
        const double l = t == 1 ? a : a * ib;
        ib = 1.0 / (t == 1 ? b : fma(-l, cp, b));
        L[t * row_t] = l;
        IB[t * row_t] = ib;
        if (t > 1) U[(t - 1) * row_t] = cp * ib;
        cp = c;
    }
    U[e * row_t] = cp;
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
template <typename T> struct batch_typed {
    // line tables: delta form (FP64) or the stages on Y1, Y2, Y3 (FP32)
    static constexpr bool DELTA = std::is_same<T, double>::value;
    static constexpr int S_SLOTS = s_slots<T>(), V_SLOTS = v_slots<T>();
    static constexpr int PITCH = 32 / sizeof(T); // rows of the state start on 32-byte sectors
    int count = 0;
    std::vector<bdesc> desc;
    std::vector<int> order;
    std::vector<long long> gps;
    long long total_n = 0, total_flat = 0, total_x = 0, total_y = 0; // sums of nx*ld, nx*ny, nx, ny
    dbuf<bdesc> d_desc;
    dbuf<int> d_order, d_counter, d_status, d_final, d_imap, d_jmap;
    dbuf<double> d_values;
    dbuf<T> state, stab, vtab, xarena, yarena;
    dbuf<T> d_payoff; // concatenated initial conditions (sum n)
    long long launches = 0;
    // forward + adjoint
    bool adjoint_ok = false;      // FP64, Heston and SABR with r = 0
    std::string adjoint_why;
    int ck_override = 0;          // checkpoint interval (0 = planned from the workspace cap)
    double ws_cap = 0.0;          // adjoint workspace cap in bytes (0 = a quarter of the device memory)
    dbuf<double> d_grads, d_ws;
    dbuf<T> b0arena;              // nx arena: boundary column of the step (persistent kernels)
    // warp-group plan of a persistent kernel (per mode): instance classes, class queues, CTA
    // layouts and, for mode 1, the workspace slices and checkpoint intervals
    // (one launch per scheme present: each specialisation gets its own register allocation)
    struct group_plan {
        int grid = 0;
        bool small = false; // forward: every instance has small lines
        bool far = false;   // FP32: rows of tables that need 64-bit offsets (adi_index.hpp)
        int start[MAX_GROUP_WARPS + 1] = {}, cnt[MAX_GROUP_WARPS + 1] = {};
        long long need[MAX_GROUP_WARPS + 1] = {};
        std::vector<int> order, layout;
        dbuf<int> d_order, d_layout;
    };
    static constexpr int NSCHEMES = 4; // LSS_ADI_DOUGLAS_RACHFORD .. LSS_ADI_HUNDSDORFER_VERWER
    struct mode_plan {
        bool valid = false;
        int gcap = 0, override_ck = -1;
        double cap = -1.0;
        long long per_warp = 0;
        group_plan sch[NSCHEMES];
    } plan[2];
    int sms = 0;
    cudaGraphExec_t graph = nullptr;
    int graph_mode = -1;

    ~batch_typed()
    {
        if (graph) cudaGraphExecDestroy(graph);
        if (wide_graph) cudaGraphExecDestroy(wide_graph);
    }

    bparams<T> params()
    {
        bparams<T> p{};
        p.desc = d_desc.p;
        p.order = d_order.p;
        p.count = count;
        p.counter = d_counter.p;
        p.B0 = b0arena.p;
        p.U = state.p;
        p.V = state.p + total_n;
        p.Y1 = state.p + 2 * total_n;
        p.Y2 = state.p + 3 * total_n;
        p.Y3 = state.p + 4 * total_n;
        p.S = stab.p;
        p.Vt = vtab.p;
        for (int s = 0; s < X_COUNT; ++s) p.X[s] = xarena.p + s * total_x;
        for (int s = 0; s < Y_COUNT; ++s) p.Yv[s] = yarena.p + s * total_y;
        p.imap = d_imap.p;
        p.jmap = d_jmap.p;
        p.values = d_values.p;
        p.status = d_status.p;
        p.final_in_v = d_final.p;
        p.grads = d_grads.p;
        p.ws = d_ws.p;
        p.payoff = d_payoff.p;
        return p;
    }
    // params() with the class queues and layouts of mode m's plan for scheme sc
    bparams<T> params_for(int m, int sc)
    {
        bparams<T> p = params();
        const group_plan &g = plan[m].sch[sc];
        p.order = g.d_order.p;
        p.layout = g.d_layout.p;
        p.counter = d_counter.p + sc * (MAX_GROUP_WARPS + 1);
        for (int c = 0; c <= MAX_GROUP_WARPS; ++c) {
            p.cls_start[c] = g.start[c];
            p.cls_count[c] = g.cnt[c];
            p.cls_need[c] = g.need[c];
        }
        p.ws_per_warp = plan[m].per_warp;
        return p;
    }

    int create(const lss_adi_problem *ps, int n);
    int prepare_adjoint(cudaStream_t s);
    double ws_bytes_allowed();
    // most threads per instance (32 x warps of a group) of the persistent kernels, per mode;
    // chosen by autotune()
    int bs_mode[2] = {BATCH_CTA, BATCH_CTA};
    int make_plan(int mode); // (re)plans mode's groups when its inputs changed
    int launch_forward(cudaStream_t s);
    int launch_fwdadj(cudaStream_t s);
    int autotune(int mode, int *chosen, cudaStream_t s);
    // wide path (count == 1)
    dbuf<T> d_b0;
    cudaGraphExec_t wide_graph = nullptr;
    void enqueue_wide_step(cudaStream_t s, const bparams<T> &p, const T *U, T *Y1, T *Y2, T *Y3, T *V);
    int enqueue_wide(cudaStream_t s);
    int run_wide(cudaStream_t s, bool use_graph);
    int enqueue(int mode, cudaStream_t s);
    int run(int mode, cudaStream_t s, bool use_graph);
};

template <typename T> int batch_typed<T>::create(const lss_adi_problem *ps, int n)
{
    count = n;
    desc.resize(n);
    gps.resize(n);
    long long on = 0, of = 0, ox = 0, oy = 0;
    for (int k = 0; k < n; ++k) {
        desc[k].nx = ps[k].nx;
        desc[k].ny = ps[k].ny;
        desc[k].steps = ps[k].nt - 1;
        desc[k].scheme = ps[k].scheme;
        desc[k].ld = (ps[k].ny + PITCH - 1) / PITCH * PITCH;
        desc[k].o2 = on;
        desc[k].op = of;
        desc[k].ox = static_cast<int>(ox);
        desc[k].oy = static_cast<int>(oy);
        gps[k] = static_cast<long long>(ps[k].nx) * ps[k].ny * (ps[k].nt - 1);
        on += static_cast<long long>(ps[k].nx) * desc[k].ld;
        of += static_cast<long long>(ps[k].nx) * ps[k].ny;
        ox += ps[k].nx;
        oy += ps[k].ny;
    }
    total_n = on;
    total_flat = of;
    total_x = ox;
    total_y = oy;
    if (ox > (1LL << 31) || oy > (1LL << 31)) return set_error(LSS_ADI_EINVAL, "batch too large");

    // host tables in the reference arithmetic, in parallel over instances
    std::vector<double> base(7 * static_cast<size_t>(total_n));
    std::vector<T> xh(X_COUNT * static_cast<size_t>(total_x)), yh(Y_COUNT * static_cast<size_t>(total_y));
    std::vector<int> imh(total_x), jmh(total_y);
    std::vector<double> scal(3 * static_cast<size_t>(n));
    std::vector<T> pay(static_cast<size_t>(total_flat));
    const unsigned nthr = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
    run_shares(nthr, [&](unsigned w) {
        for (int k = static_cast<int>(w); k < n; k += static_cast<int>(nthr)) {
            instance_tables<T> tt;
            build_tables_for<T>(ps[k], tt);
            const bdesc &d = desc[k];
            const size_t nn = static_cast<size_t>(d.nx) * d.ny;
            for (int s = 0; s < 7; ++s)
                for (int i = 0; i < d.nx; ++i) {
                    double *dst = base.data() + s * static_cast<size_t>(total_n) + d.o2 + static_cast<size_t>(i) * d.ld;
                    const T *src = tt.coef.data() + s * nn + static_cast<size_t>(i) * d.ny;
                    for (int j = 0; j < d.ny; ++j) dst[j] = static_cast<double>(src[j]);
                }
            std::copy(tt.payoff.begin(), tt.payoff.end(), pay.begin() + d.op);
            const double th = tt.sc.theta, ni = tt.sc.ni, dl = tt.sc.delta, rk = tt.sc.rho;
            scal[3 * k] = th;
            scal[3 * k + 1] = static_cast<double>(tt.sc.zeta);
            scal[3 * k + 2] = static_cast<double>(tt.sc.gamma);
            for (int i = 0; i < d.nx; ++i) {
                const double D = tt.coef_v0[i], E = tt.coef_v0[d.nx + i], F = tt.coef_v0[2 * d.nx + i];
                xh[XB_M * total_x + d.ox + i] = static_cast<T>(-dl * D);
                xh[XB_C * total_x + d.ox + i] = static_cast<T>(1.0 - 3.0 * ni * E + rk * F);
                xh[XB_P * total_x + d.ox + i] = static_cast<T>(dl * D);
                xh[XB_2 * total_x + d.ox + i] = static_cast<T>(-ni * E);
                xh[XB_1 * total_x + d.ox + i] = static_cast<T>(4.0 * ni * E);
                xh[X_VHI * total_x + d.ox + i] = tt.v_hi[i];
                imh[d.ox + i] = tt.imap[i];
            }
            const double h1 = tt.sc.h1;
            {
                // coefficient derivatives (adjoint), double
                sinh_map<double> g;
                g.init(ps[k]);
                const double sg = ps[k].sigma, bt = ps[k].sabr_beta;
                for (int i = 0; i < d.nx; ++i) {
                    const s_factors q = derivative_s(ps[k], g, static_cast<double>(tt.sc.h1) * i);
                    xh[X_HX * total_x + d.ox + i] = static_cast<T>(q.hx);
                    xh[X_HC * total_x + d.ox + i] = static_cast<T>(q.hc);
                    xh[X_HA * total_x + d.ox + i] = static_cast<T>(q.ha);
                    xh[X_HDD * total_x + d.ox + i] = static_cast<T>(q.hdd);
                }
                for (int j = 0; j < d.ny; ++j) {
                    const v_factors q = derivative_v(ps[k], g, static_cast<double>(tt.sc.h2) * j);
                    yh[Y_HY * total_y + d.oy + j] = static_cast<T>(q.hy);
                    yh[Y_BS * total_y + d.oy + j] = static_cast<T>(q.bs);
                    yh[Y_EK * total_y + d.oy + j] = static_cast<T>(q.ek);
                    yh[Y_ET * total_y + d.oy + j] = static_cast<T>(q.et);
                    yh[Y_ES * total_y + d.oy + j] = static_cast<T>(q.es);
                    yh[Y_HV2 * total_y + d.oy + j] = static_cast<T>(q.hv2);
                }
                desc[k].model = ps[k].model;
                desc[k].a_alphat = static_cast<double>(tt.sc.alpha);
                desc[k].a_omb = 1.0 - bt;
                const double kk = static_cast<double>(tt.sc.k);
                desc[k].a_tau0 = ps[k].forward ? ps[k].maturity - kk : kk;
                desc[k].a_dtau = ps[k].forward ? -kk : kk;
                desc[k].a_delta = static_cast<double>(tt.sc.delta);
                desc[k].a_halfk = 0.5 * static_cast<double>(tt.sc.k);
                desc[k].a_ni = static_cast<double>(tt.sc.ni);
                desc[k].a_betat = static_cast<double>(tt.sc.beta);
                desc[k].a_sigma = sg;
                desc[k].a_rho = ps[k].rho;
                desc[k].a_theta = static_cast<double>(tt.sc.theta);
                desc[k].a_zeta = static_cast<double>(tt.sc.zeta);
                desc[k].a_gamma = static_cast<double>(tt.sc.gamma);
                desc[k].a_k = static_cast<double>(tt.sc.k);
                desc[k].ck = std::max(1, static_cast<int>(std::ceil(std::sqrt(static_cast<double>(d.steps)))));
            }
            for (int j = 0; j < d.ny; ++j) {
                yh[Y_SLO * total_y + d.oy + j] = tt.s_lo[j];
                yh[Y_B2C * total_y + d.oy + j] = static_cast<T>(2.0 * h1 * static_cast<double>(tt.s_hi_neu[j]) / 3.0);
                jmh[d.oy + j] = tt.jmap[j];
            }
            // modified Craig-Sneyd with zeta == theta adds (zeta - theta) * (...) = 0: it is
            // Craig-Sneyd (the reference's surfaces are bit-identical), so run the CS stencil
            if (ps[k].scheme == LSS_ADI_MODIFIED_CRAIG_SNEYD && tt.sc.zeta == tt.sc.theta)
                desc[k].scheme = LSS_ADI_CRAIG_SNEYD;
            const double DN = tt.coef_v0[d.nx - 1];
            desc[k].bnc = -dl * (2.0 * h1 * static_cast<double>(tt.s_hi_neu[0])) * DN;
            const bilinear b = make_bilinear(tt.x.data(), d.nx, tt.y.data(), d.ny, ps[k].eval_s, ps[k].eval_v);
            desc[k].i0 = b.i0;
            desc[k].j0 = b.j0;
            desc[k].w00 = b.w00;
            desc[k].w10 = b.w10;
            desc[k].w01 = b.w01;
            desc[k].w11 = b.w11;
        }
    });

    // longest instances first
    order.resize(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return gps[a] > gps[b]; });

    LSS_CUDA_TRY(d_desc.alloc(n), "batch: allocating descriptors");
    LSS_CUDA_TRY(d_desc.upload(desc.data(), n), "batch: uploading descriptors");
    LSS_CUDA_TRY(d_order.alloc(n), "batch: allocating order");
    LSS_CUDA_TRY(d_order.upload(order.data(), n), "batch: uploading order");
    LSS_CUDA_TRY(d_counter.alloc(4 * (MAX_GROUP_WARPS + 1)), "batch: allocating counters");
    LSS_CUDA_TRY(b0arena.alloc(total_x), "batch: allocating boundary columns");
    LSS_CUDA_TRY(d_status.alloc(n), "batch: allocating status");
    LSS_CUDA_TRY(d_final.alloc(n), "batch: allocating flags");
    LSS_CUDA_TRY(d_values.alloc(n), "batch: allocating values");
    LSS_CUDA_TRY(d_imap.alloc(total_x), "batch: allocating remaps");
    LSS_CUDA_TRY(d_imap.upload(imh.data(), total_x), "batch: uploading remaps");
    LSS_CUDA_TRY(d_jmap.alloc(total_y), "batch: allocating remaps");
    LSS_CUDA_TRY(d_jmap.upload(jmh.data(), total_y), "batch: uploading remaps");
    LSS_CUDA_TRY(xarena.alloc(X_COUNT * total_x), "batch: allocating S boundary arrays");
    LSS_CUDA_TRY(yarena.alloc(Y_COUNT * total_y), "batch: allocating v boundary arrays");
    LSS_CUDA_TRY(state.alloc(5 * total_n), "batch: allocating state");
    LSS_CUDA_TRY(cudaMemset(state.p, 0, state.n * sizeof(T)), "batch: clearing state");
    LSS_CUDA_TRY(d_payoff.alloc(total_flat), "batch: allocating initial conditions");
    LSS_CUDA_TRY(d_payoff.upload(pay.data(), total_flat), "batch: uploading initial conditions");
    LSS_CUDA_TRY(stab.alloc(S_SLOTS * total_n), "batch: allocating S-line tables");
    LSS_CUDA_TRY(vtab.alloc(V_SLOTS * total_n), "batch: allocating v-line tables");
    // boundary rows/columns of the line tables are read (as zeros) by the adjoint's gather
    LSS_CUDA_TRY(cudaMemset(stab.p, 0, stab.n * sizeof(T)), "batch: clearing S-line tables");
    LSS_CUDA_TRY(cudaMemset(vtab.p, 0, vtab.n * sizeof(T)), "batch: clearing v-line tables");
    LSS_CUDA_TRY(d_grads.alloc(5 * static_cast<size_t>(n)), "batch: allocating gradients");
    LSS_CUDA_TRY(cudaMemset(d_grads.p, 0, d_grads.n * sizeof(double)), "batch: clearing gradients");
    adjoint_ok = std::is_same<T, double>::value;
    adjoint_why = adjoint_ok ? "" : "the adjoint is FP64 only";

    // factorise on the device from the base tables
    {
        dbuf<double> d_base, d_scal;
        dbuf<long long> d_ls;
        dbuf<bdesc> dd;
        LSS_CUDA_TRY(d_base.alloc(base.size()), "batch: allocating base tables");
        LSS_CUDA_TRY(d_base.upload(base.data(), base.size()), "batch: uploading base tables");
        LSS_CUDA_TRY(d_scal.alloc(scal.size()), "batch: allocating scalars");
        LSS_CUDA_TRY(d_scal.upload(scal.data(), scal.size()), "batch: uploading scalars");
        LSS_CUDA_TRY(cudaMemcpy(xarena.p, xh.data(), xh.size() * sizeof(T), cudaMemcpyHostToDevice), "batch: x arena");
        LSS_CUDA_TRY(cudaMemcpy(yarena.p, yh.data(), yh.size() * sizeof(T), cudaMemcpyHostToDevice), "batch: y arena");
        LSS_CUDA_TRY(d_ls.alloc(n), "batch: line offsets");
        setup_params sp{};
        sp.desc = d_desc.p;
        sp.count = n;
        sp.base = d_base.p;
        sp.total_n = total_n;
        sp.scal = d_scal.p;
        sp.line_start = d_ls.p;
        // S lines: ny - 2 per instance
        std::vector<long long> ls(n);
        long long acc = 0;
        for (int k = 0; k < n; ++k) { ls[k] = acc; acc += desc[k].ny - 2; }
        LSS_CUDA_TRY(d_ls.upload(ls.data(), n), "batch: line offsets");
        sp.total_lines = acc;
        if constexpr (DELTA) k_setup_s_delta<<<grid_for(acc, 128), 128>>>(sp, stab.p);
        else k_setup_s_lines<T><<<grid_for(acc, 128), 128>>>(sp, stab.p, yarena.p + Y_CHS * total_y);
        LSS_CUDA_TRY(cudaGetLastError(), "batch: launching S-line set-up");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: S-line set-up");
        acc = 0;
        for (int k = 0; k < n; ++k) { ls[k] = acc; acc += desc[k].nx - 2; }
        LSS_CUDA_TRY(d_ls.upload(ls.data(), n), "batch: line offsets");
        sp.total_lines = acc;
        if constexpr (DELTA) k_setup_v_delta<<<grid_for(acc, 128), 128>>>(sp, vtab.p);
        else k_setup_v_lines<T><<<grid_for(acc, 128), 128>>>(sp, vtab.p, xarena.p + X_CHV * total_x);
        LSS_CUDA_TRY(cudaGetLastError(), "batch: launching v-line set-up");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: v-line set-up");
    }
    int dev = 0, sms = 0; // local
    LSS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
    LSS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    this->sms = sms;
    if (n == 1) LSS_CUDA_TRY(d_b0.alloc(desc[0].nx), "batch: allocating the boundary column");
    return LSS_ADI_OK;
}

template <typename T> int batch_typed<T>::prepare_adjoint(cudaStream_t s)
{
    (void)s;
    if (!adjoint_ok) return set_error(LSS_ADI_EUNSUPPORTED, "batch: " + adjoint_why);
    return make_plan(1);
}

// Instances that run with `shallow`, where no instance of their scheme is larger: most of what `deep` loads
// ahead lies past the ends of their lines, and its registers leave fewer instances on an SM.  Forward,
// 50 steps, ms with deep / shallow (and with the kernels before rows were loaded ahead): FP64 DR 20000 of
// 8 x 8 8.2 / 6.7 (7.0), 1000 of 8 x 100 4.9 / 3.6 (4.3), 20000 of 64 x 16 53 / 46, but 1000 Craig-Sneyd of
// 64 x 16 7.0 / 7.2; FP32 DR 20000 of 8 x 8 3.0 / 1.8 (1.4), of 16 x 16 4.5 / 3.8 (4.2), but 1000
// Craig-Sneyd of 24 x 16 0.93 / 1.0.
template <typename T> static bool small_lines(const bdesc &d) { return static_cast<long long>(d.nx) * d.ny <= (sizeof(T) == 8 ? 900 : 256); }

// Workspace (doubles) of one instance checkpointed every c steps: nseg checkpoints, the stage
// increments of one segment (4 arrays per step plus the segment's end), two scratch states, six
// adjoint arrays and three line-end vectors.
static long long adj_ws_need(const bdesc &d, int c)
{
    const long long nn = static_cast<long long>(d.nx) * d.ld;
    const long long nseg = (d.steps + c - 1) / c;
    return (nseg + 4LL * (c + 1) + 2 + 6) * nn + d.nx + 2LL * d.ny;
}

// Bytes the adjoint workspace may take: the cap set by lss_adi_batch_set_workspace, by default
// a quarter of the device memory, and never more than half of what is free (counting the
// workspace already held, which a new plan replaces).
template <typename T> double batch_typed<T>::ws_bytes_allowed()
{
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return ws_cap > 0.0 ? ws_cap : 0.0;
    }
    // the default (a quarter of the device) leaves at least half of what is free to the caller;
    // a cap the caller sets is honoured up to 90 % of what is free
    const double held = d_ws.p ? static_cast<double>(d_ws.n) * sizeof(double) : 0.0;
    const double avail = static_cast<double>(free_b) + held;
    if (ws_cap > 0.0) return std::min(ws_cap, 0.9 * avail);
    return std::min(0.25 * static_cast<double>(total_b), 0.5 * avail);
}

// CTA layouts (warp-group sizes, one hex digit per group) for `grid` CTAs of MAX_GROUP_WARPS
// warps: each CTA in turn takes the layout that covers the most of the classes' remaining
// shares of the warps (class c's share: its grid-point-steps over all, times the warps); the
// groups' stealing of smaller instances evens out what the rounding leaves.
static std::vector<int> plan_layouts(int grid, const double work[MAX_GROUP_WARPS + 1], int gcap)
{
    struct lay { int code; int w[MAX_GROUP_WARPS + 1]; };
    const lay all[] = {{0x4, {0, 0, 0, 0, 1}}, {0x13, {0, 1, 0, 1, 0}}, {0x22, {0, 0, 2, 0, 0}},
                       {0x112, {0, 2, 1, 0, 0}}, {0x1111, {0, 4, 0, 0, 0}}};
    std::vector<lay> cand;
    for (const lay &l : all) {
        bool ok = true;
        for (int c = gcap + 1; c <= MAX_GROUP_WARPS; ++c) ok = ok && l.w[c] == 0;
        if (ok) cand.push_back(l);
    }
    double tot = 0.0;
    for (int c = 1; c <= MAX_GROUP_WARPS; ++c) tot += work[c];
    double want[MAX_GROUP_WARPS + 1] = {};
    for (int c = 1; c <= MAX_GROUP_WARPS; ++c)
        want[c] = tot > 0.0 ? work[c] / tot * MAX_GROUP_WARPS * grid : 0.0;
    // the first CTA holds a group as large as the largest class that has work, so that every
    // class has a group able to take its instances
    int top = 0;
    for (int c = 1; c <= MAX_GROUP_WARPS; ++c)
        if (work[c] > 0.0) top = c;
    std::vector<int> out(grid);
    for (int b = 0; b < grid; ++b) {
        int best = 0;
        double best_score = -1.0;
        if (b == 0 && top > 0) {
            for (size_t q = 0; q < cand.size(); ++q) {
                bool fits = cand[q].w[top] > 0;
                for (int c = top + 1; c <= MAX_GROUP_WARPS; ++c) fits = fits && cand[q].w[c] == 0;
                if (fits) { best = static_cast<int>(q); break; }
            }
            out[b] = cand[best].code;
            for (int c = 1; c <= MAX_GROUP_WARPS; ++c) want[c] -= cand[best].w[c] * c;
            continue;
        }
        for (size_t q = 0; q < cand.size(); ++q) {
            double score = 0.0;
            for (int c = 1; c <= MAX_GROUP_WARPS; ++c)
                score += std::min(static_cast<double>(cand[q].w[c] * c), std::max(0.0, want[c]));
            if (score > best_score + 1e-9) { best_score = score; best = static_cast<int>(q); }
        }
        out[b] = cand[best].code;
        for (int c = 1; c <= MAX_GROUP_WARPS; ++c) want[c] -= cand[best].w[c] * c;
    }
    return out;
}

// Warp-group plan of mode `mode`: class (warps per instance) of every instance -- one warp per 32
// S lines, at most bs_mode/32 -- and, per scheme present (one launch each), the class queues
// longest first and the CTA layouts; for mode 1 the workspace slices (per warp, within the cap,
// shared by the schemes' launches) and every instance's checkpoint interval: at least
// ceil(sqrt(steps)) (or the fixed interval), else the longest whose workspace fits the slices of
// its class's group.  A cap too small for the minimal slices of every resident CTA runs fewer CTAs.
template <typename T> int batch_typed<T>::make_plan(int mode)
{
    mode_plan &mp = plan[mode];
    const int gcap = std::max(1, std::min(MAX_GROUP_WARPS, bs_mode[mode] / 32));
    if (mp.valid && mp.gcap == gcap && (mode == 0 || (mp.override_ck == ck_override && mp.cap == ws_cap))) return LSS_ADI_OK;
    if (graph && graph_mode == mode) { // a captured launch holds the old plan
        cudaGraphExecDestroy(graph);
        graph = nullptr;
        graph_mode = -1;
    }
    mp.valid = false;
    std::vector<int> cls(count);
    double work[NSCHEMES][MAX_GROUP_WARPS + 1] = {};
    int warps_wanted[NSCHEMES] = {};
    for (int k = 0; k < count; ++k) {
        const int nx = desc[k].nx, ny = desc[k].ny, sc = desc[k].scheme;
        cls[k] = std::max(1, std::min(gcap, (ny - 2 + 31) / 32));
        // the group's threads that have a line, over its threads, per S / v sweep: the class's
        // warps are shared out by work over that efficiency
        const int th = 32 * cls[k];
        const double lines = static_cast<double>(nx - 2) * (ny - 2);
        const double slots = static_cast<double>(nx - 2) * ((ny - 2 + th - 1) / th) * th +
                             static_cast<double>(ny - 2) * ((nx - 2 + th - 1) / th) * th;
        work[sc][cls[k]] += static_cast<double>(gps[k]) * slots / (2.0 * lines);
        warps_wanted[sc] += cls[k];
    }
    int per_sm = 0, per_sm_small = 0;
    if constexpr (std::is_same<T, double>::value) {
        if (mode == 1)
            LSS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_fwdadj<LSS_ADI_CRAIG_SNEYD>, BATCH_CTA, 0),
                         "occupancy");
    }
    if (mode == 0) {
        LSS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_forward<T, LSS_ADI_CRAIG_SNEYD, deep>, BATCH_CTA, 0),
                     "occupancy");
        LSS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_small, k_batch_forward<T, LSS_ADI_CRAIG_SNEYD, shallow>, BATCH_CTA, 0),
                     "occupancy");
    }
    int grid[NSCHEMES];
    for (int sc = 0; sc < NSCHEMES; ++sc) {
        bool &small = mp.sch[sc].small;
        small = mode == 0;
        mp.sch[sc].far = false;
        for (int k = 0; k < count; ++k) {
            small = small && (desc[k].scheme != sc || small_lines<T>(desc[k]));
            mp.sch[sc].far = mp.sch[sc].far || (desc[k].scheme == sc && desc[k].ld > NEAR_PITCH);
        }
        const int resident = sms * std::max(1, small ? per_sm_small : per_sm);
        grid[sc] = std::max(1, std::min(resident, (warps_wanted[sc] + MAX_GROUP_WARPS - 1) / MAX_GROUP_WARPS));
    }
    mp.per_warp = 0;
    for (int sc = 0; sc < NSCHEMES; ++sc)
        for (int c = 0; c <= MAX_GROUP_WARPS; ++c) mp.sch[sc].need[c] = 0;
    if (mode == 1) {
        std::vector<int> c0(count);
        long long base_w = 1, full_w = 1; // doubles per warp: minimal and no-recomputation slices
        for (int k = 0; k < count; ++k) {
            const bdesc &d = desc[k];
            c0[k] = ck_override > 0 ? std::min(ck_override, d.steps)
                                    : std::max(1, static_cast<int>(std::ceil(std::sqrt(static_cast<double>(d.steps)))));
            base_w = std::max(base_w, (adj_ws_need(d, c0[k]) + cls[k] - 1) / cls[k]);
            full_w = std::max(full_w, (adj_ws_need(d, d.steps) + cls[k] - 1) / cls[k]);
        }
        base_w = (base_w + 31) / 32 * 32;
        const double allowed = ws_bytes_allowed() / sizeof(double);
        const long long fit = static_cast<long long>(allowed / (static_cast<double>(base_w) * MAX_GROUP_WARPS));
        if (fit < 1)
            return set_error(LSS_ADI_ENOMEM, "batch: the adjoint workspace cap (" + std::to_string(allowed * 8.0 / 1e6) +
                                                 " MB) does not hold the checkpoints of the largest instance");
        int gmax = 1;
        for (int sc = 0; sc < NSCHEMES; ++sc) {
            grid[sc] = static_cast<int>(std::min<long long>(grid[sc], fit));
            gmax = std::max(gmax, grid[sc]);
        }
        long long per_warp = base_w;
        if (ck_override <= 0)
            per_warp = std::max(base_w, std::min((full_w + 31) / 32 * 32,
                                                 static_cast<long long>(allowed / (static_cast<double>(gmax) * MAX_GROUP_WARPS)) / 32 * 32));
        bool changed = false;
        for (int k = 0; k < count; ++k) {
            bdesc &d = desc[k];
            int c = c0[k];
            if (ck_override <= 0)
                for (int cc = d.steps; cc > c0[k]; --cc)
                    if (adj_ws_need(d, cc) <= per_warp * cls[k]) { c = cc; break; }
            if (c != d.ck) { d.ck = c; changed = true; }
            long long &nd = mp.sch[d.scheme].need[cls[k]];
            nd = std::max(nd, adj_ws_need(d, c));
        }
        if (changed)
            LSS_CUDA_TRY(cudaMemcpy(d_desc.p, desc.data(), count * sizeof(bdesc), cudaMemcpyHostToDevice), "batch: descriptors");
        mp.per_warp = per_warp;
        const size_t want = static_cast<size_t>(per_warp) * MAX_GROUP_WARPS * gmax;
        if (d_ws.n != want) {
            d_ws.release();
            LSS_CUDA_TRY(d_ws.alloc(want), "batch: allocating adjoint workspace");
        }
    }
    for (int sc = 0; sc < NSCHEMES; ++sc) {
        group_plan &g = mp.sch[sc];
        // class queues, longest first within a class
        g.order.clear();
        for (int c = 0; c <= MAX_GROUP_WARPS; ++c) g.start[c] = g.cnt[c] = 0;
        for (int c = 1; c <= MAX_GROUP_WARPS; ++c) {
            g.start[c] = static_cast<int>(g.order.size());
            for (int k : order)
                if (cls[k] == c && desc[k].scheme == sc) g.order.push_back(k);
            g.cnt[c] = static_cast<int>(g.order.size()) - g.start[c];
        }
        g.grid = g.order.empty() ? 0 : grid[sc];
        if (!g.grid) continue;
        g.layout = plan_layouts(g.grid, work[sc], gcap);
        LSS_CUDA_TRY(g.d_order.alloc(g.order.size()), "batch: allocating class queues");
        LSS_CUDA_TRY(g.d_order.upload(g.order.data(), g.order.size()), "batch: uploading class queues");
        LSS_CUDA_TRY(g.d_layout.alloc(g.grid), "batch: allocating CTA layouts");
        LSS_CUDA_TRY(g.d_layout.upload(g.layout.data(), g.grid), "batch: uploading CTA layouts");
    }
    LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: plan upload");
    mp.gcap = gcap;
    mp.override_ck = ck_override;
    mp.cap = ws_cap;
    mp.valid = true;
    return LSS_ADI_OK;
}

template <typename T> int batch_typed<T>::launch_forward(cudaStream_t s)
{
    for (int sc = 0; sc < NSCHEMES; ++sc) {
        const group_plan &g = plan[0].sch[sc];
        if (!g.grid) continue;
        const bparams<T> p = params_for(0, sc);
        auto launch = [&](auto depth) {
            using D = decltype(depth);
            switch (sc) {
            case LSS_ADI_DOUGLAS_RACHFORD: k_batch_forward<T, LSS_ADI_DOUGLAS_RACHFORD, D><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            case LSS_ADI_CRAIG_SNEYD: k_batch_forward<T, LSS_ADI_CRAIG_SNEYD, D><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            case LSS_ADI_MODIFIED_CRAIG_SNEYD: k_batch_forward<T, LSS_ADI_MODIFIED_CRAIG_SNEYD, D><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            default: k_batch_forward<T, LSS_ADI_HUNDSDORFER_VERWER, D><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            }
        };
        bool far = false;
        if constexpr (sizeof(T) == 4) {
            far = g.far;
            if (far) launch(deep_far{});
        }
        if (!far && g.small) launch(shallow{});
        else if (!far) launch(deep{});
        LSS_CUDA_TRY(cudaGetLastError(), "batch: launching k_batch_forward");
        ++launches;
    }
    return LSS_ADI_OK;
}

template <typename T> int batch_typed<T>::launch_fwdadj(cudaStream_t s)
{
    if constexpr (std::is_same<T, double>::value) {
        for (int sc = 0; sc < NSCHEMES; ++sc) {
            const group_plan &g = plan[1].sch[sc];
            if (!g.grid) continue;
            const bparams<double> p = params_for(1, sc);
            switch (sc) {
            case LSS_ADI_DOUGLAS_RACHFORD: k_batch_fwdadj<LSS_ADI_DOUGLAS_RACHFORD><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            case LSS_ADI_CRAIG_SNEYD: k_batch_fwdadj<LSS_ADI_CRAIG_SNEYD><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            case LSS_ADI_MODIFIED_CRAIG_SNEYD: k_batch_fwdadj<LSS_ADI_MODIFIED_CRAIG_SNEYD><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            default: k_batch_fwdadj<LSS_ADI_HUNDSDORFER_VERWER><<<g.grid, BATCH_CTA, 0, s>>>(p); break;
            }
            LSS_CUDA_TRY(cudaGetLastError(), "batch: launching k_batch_fwdadj");
            ++launches;
        }
        return LSS_ADI_OK;
    } else {
        (void)s;
        return set_error(LSS_ADI_EUNSUPPORTED, "batch: the adjoint is FP64 only");
    }
}

template <typename T> int batch_typed<T>::enqueue(int mode, cudaStream_t s)
{
    int rc = make_plan(mode == 1 ? 1 : 0);
    if (rc) return rc;
    LSS_CUDA_TRY(cudaMemsetAsync(d_counter.p, 0, d_counter.n * sizeof(int), s), "batch: counter reset");
    launches = 0;
    if (mode == 1) {
        rc = launch_fwdadj(s);
    } else {
        rc = launch_forward(s);
    }
    return rc;
}

// Times one run per cap on the warps per instance (32, 64 and 128 threads: groups of at most 1,
// 2 or 4 warps) and keeps the fastest for `mode`; with *chosen > 0 on entry (32, 64, 96 or 128),
// sets that cap without timing.
template <typename T> int batch_typed<T>::autotune(int mode, int *chosen, cudaStream_t s)
{
    const int m = mode == 1 ? 1 : 0;
    if (mode == 1 && !adjoint_ok) return set_error(LSS_ADI_EUNSUPPORTED, "batch: " + adjoint_why);
    if (chosen && *chosen > 0) {
        if (*chosen != 32 && *chosen != 64 && *chosen != 96 && *chosen != 128)
            return set_error(LSS_ADI_EINVAL, "autotune: threads per instance must be 32, 64, 96 or 128");
        bs_mode[m] = *chosen;
        int rc = make_plan(m);
        if (rc) return rc;
    } else {
        const int cand[3] = {32, 64, 128};
        float best = 1e30f;
        int best_bs = bs_mode[m];
        cudaEvent_t e0, e1;
        LSS_CUDA_TRY(cudaEventCreate(&e0), "autotune: event");
        LSS_CUDA_TRY(cudaEventCreate(&e1), "autotune: event");
        for (int c : cand) {
            bs_mode[m] = c;
            int rc = make_plan(m);
            if (rc == LSS_ADI_ENOMEM) { // a plan whose workspace does not fit is skipped
                clear_error();
                continue;
            }
            if (!rc) {
                cudaEventRecord(e0, s);
                rc = enqueue(mode, s);
                cudaEventRecord(e1, s);
            }
            if (rc) {
                cudaEventDestroy(e0);
                cudaEventDestroy(e1);
                return rc;
            }
            LSS_CUDA_TRY(cudaEventSynchronize(e1), "autotune: run");
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                best_bs = c;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        bs_mode[m] = best_bs;
        int rc = make_plan(m);
        if (rc) return rc;
    }
    if (chosen) *chosen = bs_mode[m];
    return LSS_ADI_OK;
}

// One time step U -> V of the wide path (stage outputs in Y1, Y2, Y3).
template <typename T>
void batch_typed<T>::enqueue_wide_step(cudaStream_t s, const bparams<T> &p, const T *U, T *Y1, T *Y2, T *Y3, T *V)
{
    const bdesc &d = desc[0];
    T *b0 = d_b0.p;
    const int gs = grid_for(d.ny - 2, 32), gv = grid_for(d.nx - 2, 32);
    k_wide_b1<T><<<grid_for(std::max(d.nx, d.ny), 128), 128, 0, s>>>(p, U, b0, Y2);
    k_wide_s<T, 1><<<gs, 32, 0, s>>>(p, U, nullptr, nullptr, Y1);
    if (d.scheme == LSS_ADI_DOUGLAS_RACHFORD) {
        k_wide_v<T, true><<<gv, 32, 0, s>>>(p, U, Y1, Y2, Y1, b0, V);
    } else {
        k_wide_v<T, false><<<gv, 32, 0, s>>>(p, U, Y1, Y2, Y1, b0, Y2);
        k_wide_s<T, 2><<<gs, 32, 0, s>>>(p, U, Y1, Y2, Y3);
        k_wide_v<T, true><<<gv, 32, 0, s>>>(p, U, Y1, Y2, Y3, b0, V);
    }
    k_wide_b2<T><<<grid_for(d.ny, 128), 128, 0, s>>>(p, V);
}

template <typename T> int batch_typed<T>::enqueue_wide(cudaStream_t s)
{
    const bdesc &d = desc[0];
    bparams<T> p = params();
    T *U = p.U, *V = p.V, *Y1 = p.Y1, *Y2 = p.Y2, *Y3 = p.Y3;
    LSS_CUDA_TRY(cudaMemcpy2DAsync(U, d.ld * sizeof(T), d_payoff.p, d.ny * sizeof(T), d.ny * sizeof(T), d.nx,
                                   cudaMemcpyDeviceToDevice, s), "wide: initial state");
    LSS_CUDA_TRY(cudaMemsetAsync(d_status.p, 0, sizeof(int), s), "wide: clearing the status");
    long long nl = 0;
    for (int step = 0; step < d.steps; ++step) {
        enqueue_wide_step(s, p, U, Y1, Y2, Y3, V);
        nl += d.scheme == LSS_ADI_DOUGLAS_RACHFORD ? 4 : 6;
        std::swap(U, V);
    }
    k_wide_finish<T><<<grid_for(total_n, 256), 256, 0, s>>>(p, U);
    LSS_CUDA_TRY(cudaGetLastError(), "wide: launching the time loop");
    launches = nl + 1;
    return LSS_ADI_OK;
}

template <typename T> int batch_typed<T>::run_wide(cudaStream_t s, bool use_graph)
{
    if (count != 1) return set_error(LSS_ADI_EINVAL, "wide path: one instance only");
    if (!use_graph) return enqueue_wide(s);
    if (!wide_graph) {
        cudaStream_t cs;
        LSS_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "wide: capture stream");
        LSS_CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "wide: begin capture");
        const int rc = enqueue_wide(cs);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(cs, &g);
        cudaStreamDestroy(cs);
        if (rc) return rc;
        LSS_CUDA_TRY(e, "wide: end capture");
        e = cudaGraphInstantiate(&wide_graph, g, 0);
        cudaGraphDestroy(g);
        LSS_CUDA_TRY(e, "wide: instantiate graph");
    }
    LSS_CUDA_TRY(cudaGraphLaunch(wide_graph, s), "wide: graph launch");
    return LSS_ADI_OK;
}

template <typename T> int batch_typed<T>::run(int mode, cudaStream_t s, bool use_graph)
{
    { // plans (allocations, uploads) happen here, never inside a stream capture
        int rc = mode == 1 ? prepare_adjoint(s) : make_plan(0);
        if (rc) return rc;
    }
    if (!use_graph) return enqueue(mode, s);
    if (!graph || graph_mode != mode) {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        cudaStream_t cs;
        LSS_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "batch: capture stream");
        LSS_CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "batch: begin capture");
        int rc = enqueue(mode, cs);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(cs, &g);
        cudaStreamDestroy(cs);
        if (rc) return rc;
        LSS_CUDA_TRY(e, "batch: end capture");
        e = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        LSS_CUDA_TRY(e, "batch: instantiate graph");
        graph_mode = mode;
    }
    LSS_CUDA_TRY(cudaGraphLaunch(graph, s), "batch: graph launch");
    return LSS_ADI_OK;
}

// One thread per line (LSS_ADI_OPT_LINE_PER_THREAD).
template <typename T> struct wide_solver : wide_solver_base {
    batch_typed<T> b;
    lss_adi_problem prob{};
    std::vector<T> x, y, pay0;
    std::unique_ptr<wide_solver_base> parts; // partitioned, once lss_adi_line_chunks asks for it

    int init(const lss_adi_problem &p)
    {
        prob = p;
        instance_tables<T> tt;
        build_tables_for<T>(p, tt);
        x = tt.x;
        y = tt.y;
        pay0 = tt.payoff;
        return b.create(&p, 1);
    }
    int forward(const void *payoff, void *out_surface, double *out_value, int flags, void *stream, bool use_graph) override
    {
        if (parts) return parts->forward(payoff, out_surface, out_value, flags, stream, use_graph);
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const bool dev = (flags & LSS_ADI_DEVICE_POINTERS) != 0;
        const size_t n = static_cast<size_t>(b.total_flat);
        const void *src = payoff ? payoff : static_cast<const void *>(pay0.data());
        LSS_CUDA_TRY(cudaMemcpyAsync(b.d_payoff.p, src, n * sizeof(T),
                                     (payoff && dev) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s),
                     "wide: copying the terminal condition");
        int rc = b.run_wide(s, use_graph);
        if (rc) return rc;
        if (out_value)
            LSS_CUDA_TRY(cudaMemcpyAsync(out_value, b.d_values.p, sizeof(double), cudaMemcpyDeviceToHost, s), "wide: value");
        if (out_surface) {
            const T *fin = b.state.p + ((b.desc[0].steps & 1) ? b.total_n : 0);
            const bdesc &d = b.desc[0];
            LSS_CUDA_TRY(cudaMemcpy2DAsync(out_surface, d.ny * sizeof(T), fin, d.ld * sizeof(T), d.ny * sizeof(T), d.nx,
                                           dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s),
                         "wide: surface");
        }
        if (!dev || out_value) LSS_CUDA_TRY(cudaStreamSynchronize(s), "wide: time loop");
        return LSS_ADI_OK;
    }
    int grid(void *gx, void *gy) const override
    {
        std::copy(x.begin(), x.end(), static_cast<T *>(gx));
        std::copy(y.begin(), y.end(), static_cast<T *>(gy));
        return LSS_ADI_OK;
    }
    int chunks(int s_chunks, int v_chunks, int *out_s, int *out_v, void *stream) override
    {
        if (!parts) {
            std::unique_ptr<wide_solver_base> w;
            int rc = make_partitioned_solver(prob, w);
            if (!rc) rc = w->chunks(s_chunks, v_chunks, out_s, out_v, stream);
            if (!rc) parts = std::move(w);
            return rc;
        }
        return parts->chunks(s_chunks, v_chunks, out_s, out_v, stream);
    }
    bool asked_chunks(int &s_chunks, int &v_chunks) const override { return parts && parts->asked_chunks(s_chunks, v_chunks); }
};

int make_wide_solver(const lss_adi_problem &p, std::unique_ptr<wide_solver_base> &out)
{
    // time-dependent coefficients (no batched kernel to agree with) run partitioned; where a thread per
    // line is asked for, in relay order: the chunks of a line one after the other, with a thread per
    // line's operations
    if (!(p.options & LSS_ADI_OPT_LINE_PER_THREAD) || time_dependent(p)) return make_partitioned_solver(p, out);
    try {
        if (p.precision == LSS_ADI_FP64) {
            std::unique_ptr<wide_solver<double>> w(new wide_solver<double>());
            int rc = w->init(p);
            if (rc) return rc;
            out = std::move(w);
        } else {
            std::unique_ptr<wide_solver<float>> w(new wide_solver<float>());
            int rc = w->init(p);
            if (rc) return rc;
            out = std::move(w);
        }
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "wide: host allocation failed");
    }
    return LSS_ADI_OK;
}

template <typename T> static int set_workspace_t(batch_typed<T> &bt, double max_bytes, int checkpoint_every)
{
    bt.ws_cap = max_bytes;
    bt.ck_override = checkpoint_every;
    if (bt.graph && bt.graph_mode == 1) { // a captured launch holds the old workspace and plan
        cudaGraphExecDestroy(bt.graph);
        bt.graph = nullptr;
        bt.graph_mode = -1;
    }
    return LSS_ADI_OK;
}

template <typename T> static int payoff_grad_t(batch_typed<T> &bt, int index, void *out)
{
    if (index < 0 || index >= bt.count) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_payoff_gradient: index out of range");
    if (!std::is_same<T, double>::value) return set_error(LSS_ADI_EUNSUPPORTED, "lss_adi_batch_payoff_gradient: FP64 only");
    LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: synchronising");
    const bdesc &d = bt.desc[index];
    LSS_CUDA_TRY(cudaMemcpy2D(out, d.ny * sizeof(T), bt.state.p + bt.total_n + d.o2, d.ld * sizeof(T), d.ny * sizeof(T), d.nx,
                              cudaMemcpyDeviceToHost),
                 "batch: payoff gradient");
    return LSS_ADI_OK;
}

} // namespace lss_gb300

using namespace lss_gb300;

struct lss_adi_batch {
    int precision = LSS_ADI_FP64;
    std::unique_ptr<batch_typed<double>> b64;
    std::unique_ptr<batch_typed<float>> b32;
    cudaStream_t last_stream = nullptr;
};

template <typename T>
static int run_host_t(batch_typed<T> &bt, int mode, const void *payoffs, double *values, double *grads, cudaStream_t s)
{
    if (payoffs)
        LSS_CUDA_TRY(cudaMemcpyAsync(bt.d_payoff.p, payoffs, bt.total_flat * sizeof(T), cudaMemcpyHostToDevice, s),
                     "batch: uploading payoffs");
    int rc = bt.run(mode, s, true);
    if (rc) return rc;
    if (values)
        LSS_CUDA_TRY(cudaMemcpyAsync(values, bt.d_values.p, bt.count * sizeof(double), cudaMemcpyDeviceToHost, s),
                     "batch: reading values");
    if (grads && mode == 1)
        LSS_CUDA_TRY(cudaMemcpyAsync(grads, bt.d_grads.p, 5 * bt.count * sizeof(double), cudaMemcpyDeviceToHost, s),
                     "batch: reading gradients");
    LSS_CUDA_TRY(cudaStreamSynchronize(s), "batch: run");
    return LSS_ADI_OK;
}

template <typename T> static int results_t(batch_typed<T> &bt, double *values, double *grads, int *status)
{
    LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: synchronising");
    if (values) LSS_CUDA_TRY(cudaMemcpy(values, bt.d_values.p, bt.count * sizeof(double), cudaMemcpyDeviceToHost), "batch: values");
    if (status) LSS_CUDA_TRY(cudaMemcpy(status, bt.d_status.p, bt.count * sizeof(int), cudaMemcpyDeviceToHost), "batch: status");
    if (grads) LSS_CUDA_TRY(cudaMemcpy(grads, bt.d_grads.p, 5 * bt.count * sizeof(double), cudaMemcpyDeviceToHost), "batch: grads");
    return LSS_ADI_OK;
}

template <typename T> static int surface_t(batch_typed<T> &bt, int index, void *out)
{
    if (index < 0 || index >= bt.count) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_surface: index out of range");
    LSS_CUDA_TRY(cudaDeviceSynchronize(), "batch: synchronising");
    int fin = 0;
    LSS_CUDA_TRY(cudaMemcpy(&fin, bt.d_final.p + index, sizeof(int), cudaMemcpyDeviceToHost), "batch: flag");
    const bdesc &d = bt.desc[index];
    const T *src = bt.state.p + (fin ? bt.total_n : 0) + d.o2;
    LSS_CUDA_TRY(cudaMemcpy2D(out, d.ny * sizeof(T), src, d.ld * sizeof(T), d.ny * sizeof(T), d.nx, cudaMemcpyDeviceToHost),
                 "batch: surface");
    return LSS_ADI_OK;
}

extern "C" {

int lss_adi_batch_create(const lss_adi_problem *problems, int count, lss_adi_batch **b)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_create: null output");
    *b = nullptr;
    if (!problems || count <= 0) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_create: empty batch");
    const int prec = problems[0].precision;
    for (int k = 0; k < count; ++k) {
        std::string why;
        int rc = validate_problem(problems[k], why);
        if (rc) return set_error(rc, "lss_adi_batch_create: instance " + std::to_string(k) + ": " + why);
        if (problems[k].precision != prec) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_create: mixed precisions");
        if (problems[k].scheme == LSS_ADI_EXPLICIT_EULER)
            return set_error(LSS_ADI_EUNSUPPORTED, "lss_adi_batch_create: instance " + std::to_string(k) +
                                                       ": the explicit Euler scheme runs on lss_adi_create");
        if (time_dependent(problems[k]))
            return set_error(LSS_ADI_EUNSUPPORTED, "lss_adi_batch_create: instance " + std::to_string(k) +
                                                       ": SABR with r != 0 has time-dependent coefficients (use lss_adi_create)");
    }
    std::unique_ptr<lss_adi_batch> h(new (std::nothrow) lss_adi_batch());
    if (!h) return set_error(LSS_ADI_ENOMEM, "host allocation failed");
    h->precision = prec;
    int rc;
    try {
        if (prec == LSS_ADI_FP64) {
            h->b64.reset(new batch_typed<double>());
            rc = h->b64->create(problems, count);
        } else {
            h->b32.reset(new batch_typed<float>());
            rc = h->b32->create(problems, count);
        }
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "lss_adi_batch_create: host allocation failed");
    }
    if (rc) return rc;
    *b = h.release();
    return LSS_ADI_OK;
}

static int batch_run(lss_adi_batch *b, int mode, void *stream, bool graph)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_run: null batch");
    if (mode != 0 && mode != 1) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_run: mode must be 0 or 1");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    b->last_stream = s;
    return b->b64 ? b->b64->run(mode, s, graph) : b->b32->run(mode, s, graph);
}

int lss_adi_batch_run(lss_adi_batch *b, int mode, void *stream) { return batch_run(b, mode, stream, false); }
int lss_adi_batch_graph_launch(lss_adi_batch *b, int mode, void *stream) { return batch_run(b, mode, stream, true); }


int lss_adi_batch_run_host(lss_adi_batch *b, int mode, const void *payoffs, double *values, double *grads, void *stream)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_run_host: null batch");
    if (mode != 0 && mode != 1) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_run_host: mode must be 0 or 1");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    b->last_stream = s;
    return b->b64 ? run_host_t(*b->b64, mode, payoffs, values, grads, s)
                  : run_host_t(*b->b32, mode, payoffs, values, grads, s);
}


int lss_adi_batch_results(lss_adi_batch *b, double *values, double *grads, int *status)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_results: null batch");
    return b->b64 ? results_t(*b->b64, values, grads, status) : results_t(*b->b32, values, grads, status);
}


int lss_adi_batch_surface(lss_adi_batch *b, int index, void *out_surface)
{
    clear_error();
    if (!b || !out_surface) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_surface: null argument");
    return b->b64 ? surface_t(*b->b64, index, out_surface) : surface_t(*b->b32, index, out_surface);
}

int lss_adi_batch_payoff_gradient(lss_adi_batch *b, int index, void *out)
{
    clear_error();
    if (!b || !out) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_payoff_gradient: null argument");
    return b->b64 ? payoff_grad_t(*b->b64, index, out) : payoff_grad_t(*b->b32, index, out);
}

int lss_adi_batch_autotune(lss_adi_batch *b, int mode, int *threads_per_instance, void *stream)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_autotune: null batch");
    if (mode != 0 && mode != 1) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_autotune: mode must be 0 or 1");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return b->b64 ? b->b64->autotune(mode, threads_per_instance, s) : b->b32->autotune(mode, threads_per_instance, s);
}

int lss_adi_batch_launch_count(const lss_adi_batch *b)
{
    if (!b) return 0;
    return static_cast<int>(b->b64 ? b->b64->launches : b->b32->launches);
}

int lss_adi_batch_checkpoints(const lss_adi_batch *b, int *intervals)
{
    if (!b || !intervals) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_checkpoints: null argument");
    const int count = b->b64 ? b->b64->count : b->b32->count;
    for (int k = 0; k < count; ++k) intervals[k] = b->b64 ? b->b64->desc[k].ck : b->b32->desc[k].ck;
    return LSS_ADI_OK;
}

int lss_adi_batch_set_workspace(lss_adi_batch *b, double max_bytes, int checkpoint_every)
{
    clear_error();
    if (!b) return set_error(LSS_ADI_EINVAL, "lss_adi_batch_set_workspace: null batch");
    if (!(max_bytes >= 0.0) || checkpoint_every < 0)
        return set_error(LSS_ADI_EINVAL, "lss_adi_batch_set_workspace: negative cap or interval");
    return b->b64 ? set_workspace_t(*b->b64, max_bytes, checkpoint_every)
                  : set_workspace_t(*b->b32, max_bytes, checkpoint_every);
}

double lss_adi_batch_workspace_bytes(const lss_adi_batch *b)
{
    if (!b) return 0.0;
    return b->b64 ? static_cast<double>(b->b64->d_ws.n) * sizeof(double) : 0.0;
}

void lss_adi_batch_destroy(lss_adi_batch *b) { delete b; }

} // extern "C"
