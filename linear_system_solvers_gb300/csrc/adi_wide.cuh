// adi_wide.cuh -- partitioned line solves of one instance over the whole GPU (device side).
//
// Delta form.  With A1, A2, A0 the S, v and mixed parts of the scheme's operator times k, F = A0 +
// A1 + A2, S = (I - theta A1)^-1 per S line and V = (I - theta A2)^-1 per v line, the stages of
// lss_heat_*_method.hpp are solved for their increments (same equations, boundary values moved
// accordingly):
//   D1 = S F(U)                                   (= Y1 - U)
//   Douglas-Rachford:       next = U + V(D1)
//   others:                 D2 = V(D1)            (= Y2 - U; rows 0 and nx-1 of Y2 are zero: D2 = -U there)
//   Craig-Sneyd, modified:  D3 = S(D1 + zeta A0 D2 + (zeta - theta) G(D2)),   next = U + V(D3)
//   Hundsdorfer-Verwer:     E = S(zeta F(D2) - D2),                           next = U + D2 + V(D1 + E)
// (G: the modified scheme's extra terms with the reference's sign of the P term).  A v solve then
// needs its right-hand side and three tables instead of two right-hand-side arrays and five
// tables, every S stage reads the same six right-hand-side tables, and a time step takes about
// two thirds of the FP64 operations of the stages written on Y1, Y2, Y3.  F is evaluated with
// differences along the S line, M (U_{t-1} - U_t) + P (U_{t+1} - U_t) + (M + P - Z - W) U_t + ...: the
// terms of size k / h^2 U cancel exactly (the rounding of F, not of the whole solve, is 10 to 300
// times below that of the operator written out; the centre weight: center_weight).
//
// Line solves.  S lines in row-scaled factors (tables already divided by the pivot):
//   y_t = f_t - la_t y_{t-1},  x_t = y_t - g_t x_{t+1}          (x_0 = lo, x_{nx-1} = hi)
// v lines unscaled, l_t = a_t / beta_{t-1}, u_t = c_t / beta_{t+1}, ib_t = 1 / beta_t:
//   y_t = d_t - l_t y_{t-1},   xi_t = y_t - u_t xi_{t+1},  x_t = ib_t xi_t
// with identity rows (l = u = 0, ib = 1) at t = 0 and t = ny-1 that carry the boundary values.
//
// Partition.  A line's rows are cut into PC chunks of R rows, one thread each, solved concurrently
// by one CTA (L lines x PC chunks).  A chunk's rows stay in registers: a first pass of the recurrence
// from zero gives its end value, the chunks' affine end maps are composed through shared memory,
// and the recurrence is run again from the true incoming value.  The products of the maps do not
// change with time (k_wide_products).  Lines longer than PC R rows take several such tiles one
// after the other, the carry passed on in a register.
//
// What bounds it: one FP64 instruction of a warp takes 64 cycles of its SM sub-partition, and a
// dependent one no longer than that, so large instances are bound by the number of FP64
// instructions (two extra per point and solve for the second pass), small ones by the launch
// (programmatic dependent launches overlap the next stage's start with this one's end), the
// length R of a chunk, one memory latency per pass and the composition.
#pragma once

#include "adi_split.hpp"

namespace lss_gb300 {
namespace wide {

// chunk products of one sweep: chunk tile * PC + c of line l at [(tile * PC + c) * ls + l], in the
// sweep's order (the back sweeps run the chunks from the last to the first)
template <typename T> struct carry_tab {
    const T *A;    // product of the chunk
    const T *PreG; // of the chunks before it in its group
    const T *GA;   // of a group: [(tile * groups + group) * ls + l]
};

template <typename T> struct wparams {
    int nx, ny, ld;     // ld: row pitch (a multiple of 4)
    int tdep;           // S tables change before every step: nothing of them may be read before the wait
    T zeta, zt;         // zt: zeta - theta (modified Craig-Sneyd)
    T bnc;              // constant of the Neumann-corner boundary row
    const T *S[10];     // S-line tables ([i][j], pitch ld)
    const T *V[3];      // v-line tables ([i][t], pitch ld)
    const T *xbm, *xbc, *xbp, *xb2, *xb1, *xvhi; // nx
    const T *yslo, *yb2c;                        // ny
    const int *imap, *jmap;
    carry_tab<T> sf, sb, vf, vb; // S forward / back, v forward / back
    int ls;                      // line stride of the S carry tables
    split s, v;
    int lv;                      // line stride of the v carry tables
};

enum { W_LA = 0, W_G, W_WG, W_WW, W_WS, W_WQ, W_WN, W_WE, W_IB, W_WC, W_COUNT };
enum { W_VL = 0, W_VU, W_VIB };
enum { V_FIRST = 0, V_LAST = 1, V_LAST_HV = 2 };

__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ double wfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float wfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// four consecutive elements (32-byte aligned doubles, 16-byte aligned floats); volatile, so that no
// load of the state moves above the wait for the stage before
__device__ __forceinline__ void ld4(const double *p, double *o)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3]) : "l"(p));
}
__device__ __forceinline__ void ld4(const float *p, float *o)
{
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "l"(p));
}
__device__ __forceinline__ void st4(double *p, const double *o)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(o[0]), "d"(o[1]), "d"(o[2]), "d"(o[3]) : "memory");
}
__device__ __forceinline__ void st4(float *p, const float *o)
{
    *reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
}

// Composition of the chunks' end maps: shared arrays of one sweep (b: end values, then the values
// entering the chunks from inside their group; a: the chunks' products; gb, ga: the same of groups).
template <typename T> struct carry {
    T *b, *a, *gb, *ga;
    int L, PC, gs, ng, lane, c;
};
template <typename T> __device__ __forceinline__ carry<T> make_carry(T *raw, const split &s, int sweep, int lane, int c)
{
    carry<T> k;
    k.L = s.L; k.PC = s.PC; k.gs = s.gs; k.ng = s.groups();
    k.b = raw + sweep * carry_words(s);
    k.a = k.b + s.L * s.PC;
    k.gb = k.a + s.L * s.PC;
    k.ga = k.gb + s.L * k.ng;
    k.lane = lane; k.c = c;
    return k;
}
// The recurrence over the chunks one after the other, each from the value that the one before ended
// with (run(y): this thread's rows from the incoming y, returning the last): the operations of a
// thread that solves the whole line, so the same bits, while right-hand sides and everything
// that does not hang on the recurrence stay spread over the chunks' threads.
template <typename T, bool FWD, typename F> __device__ __forceinline__ void relay(const carry<T> &k, T &in, F run)
{
    for (int q = 0; q < k.PC; ++q) {
        if (k.c == (FWD ? q : k.PC - 1 - q)) {
            const T y = q == 0 ? in : k.gb[k.lane];
            k.gb[k.lane] = run(y);
        }
        __syncthreads();
    }
    in = k.gb[k.lane]; // every thread: the value entering the next tile
    __syncthreads();
}
// Products of this thread's chunk into shared memory; preg: of those before it in its group.
template <typename T>
__device__ __forceinline__ void carry_load(const carry<T> &k, const carry_tab<T> &t, int ls, int tile, int l, T &preg)
{
    const long long g = (long long)(tile * k.PC + k.c) * ls + l;
    k.a[k.c * k.L + k.lane] = t.A[g];
    preg = t.PreG[g];
    if (k.c < k.ng) k.ga[k.c * k.L + k.lane] = t.GA[(long long)(tile * k.ng + k.c) * ls + l];
}
// Incoming value of this thread's chunk.  FWD: chunks run 0, 1, 2, ... (the sweep's order is
// reversed otherwise).  `in` (threads of chunk 0): value entering the tile, replaced by the value
// entering the next.  A thread per group runs the group's chunks, a thread per line the groups:
// about 2 sqrt(PC) multiply-adds of latency on few warps, then one by every thread (in FP64 a
// warp's instruction costs the same whatever its active lanes, so the serial part must not run
// on every warp).
template <typename T, bool FWD> __device__ __forceinline__ T compose(const carry<T> &k, T end, T preg, T &in)
{
    const int PC = k.PC, L = k.L, lane = k.lane;
    const int at = FWD ? k.c : PC - 1 - k.c; // position in the sweep's order
    k.b[k.c * L + lane] = end;
    __syncthreads();
    if (k.c < k.ng) { // this thread's group: k.c
        T s = T(0);
        const int q1 = min((k.c + 1) * k.gs, PC);
        for (int q = k.c * k.gs; q < q1; ++q) {
            const int z = (FWD ? q : PC - 1 - q) * L + lane;
            const T v = k.b[z], w = k.a[z];
            k.b[z] = s;
            s = wfma(w, s, v);
        }
        k.gb[k.c * L + lane] = s;
    }
    __syncthreads();
    if (k.c == 0) {
        T y = in;
        for (int q = 0; q < k.ng; ++q) {
            const T v = k.gb[q * L + lane], w = k.ga[q * L + lane];
            k.gb[q * L + lane] = y;
            y = wfma(w, y, v);
        }
        in = y;
    }
    __syncthreads();
    return wfma(preg, k.gb[at / k.gs * L + lane], k.b[k.c * L + lane]);
}

// ------------------------------------------------------------------------------------------
// S stages.  KIND 1: D1 = S F(U) (A = U).  KIND 2: D3 or E (A = D2; D1: the first stage's increment).
// SER: the recurrences in relay order (a thread-per-line solve's bits).
// ------------------------------------------------------------------------------------------
template <typename T, int R, int KIND, int SCH, bool SER>
__global__ void __launch_bounds__(MAX_CTA) k_wide_s(const __grid_constant__ wparams<T> p, const T *U, const T *A, const T *D1, T *Y)
{
    extern __shared__ __align__(16) unsigned char raw[];
    const split &sp = p.s;
    const int L = sp.L, lane = threadIdx.x % L, c = threadIdx.x / L;
    const int nx = p.nx, ny = p.ny, ld = p.ld, e = nx - 2;
    const int jl = blockIdx.x * L + lane;
    const bool act = jl >= 1 && jl <= ny - 2;
    const int j = min(max(jl, 1), ny - 2);
    const carry<T> kf = make_carry(reinterpret_cast<T *>(raw), sp, 0, lane, c);
    const carry<T> kb = make_carry(reinterpret_cast<T *>(raw), sp, 1, lane, c);
    pdl_launch();
    if (p.tdep) pdl_wait();
    T preg, bpreg;
    carry_load(kf, p.sf, p.ls, 0, j, preg);
    carry_load(kb, p.sb, p.ls, sp.tiles - 1, j, bpreg);
    const int jj = p.jmap[j];
    if (!p.tdep) pdl_wait();
    const long long last = (long long)(nx - 1) * ld;
    T lo, hi;
    if constexpr (KIND == 2 && SCH == LSS_ADI_HUNDSDORFER_VERWER) {
        lo = U[j]; // E = Y4 - Y1 - D2 with D2 = -U on rows 0 and nx-1
        hi = U[last + j];
    } else {
        lo = U[jj] - U[j];
        hi = U[last + jj] - U[last + j];
    }
    if (act && c == 0) {
        Y[j] = lo;
        Y[last + j] = hi;
    }
    // Rows past the last one are read at row nx-1, whose tables are zero: they hold the upper
    // value (f = hi) and pass it down (g = 0), so no row needs a branch and the loads of a chunk
    // are issued together.
    T f[R], q[R], g[R];
    T in = lo;
    for (int tile = 0; tile < sp.tiles; ++tile) {
        const int t0 = 1 + (tile * sp.PC + c) * R;
        if (tile > 0) {
            __syncthreads(); // the tile before is done with the shared arrays
            carry_load(kf, p.sf, p.ls, tile, j, preg);
        }
        auto row = [&](int t) -> long long { return (long long)min(t, nx - 1) * ld + j; };
        T y = T(0);
        // rows t-1, t, t+1 of the centre column, side columns and their differences
        T a0c = A[row(t0 - 1)], a1c = A[row(t0)], a1m = A[row(t0) - 1], a1p = A[row(t0) + 1];
        T q0 = A[row(t0 - 1) - 1] - A[row(t0 - 1) + 1], q1 = a1m - a1p, dw = a0c - a1c;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long long o = row(t0 + r), o2 = row(t0 + r + 1);
            const T a2m = A[o2 - 1], a2c = A[o2], a2p = A[o2 + 1];
            const T q2 = a2m - a2p, mix = q0 - q2;
            T v;
            if constexpr (KIND == 1 || SCH == LSS_ADI_HUNDSDORFER_VERWER) {
                v = p.S[W_WG][o] * mix;
                v = wfma(p.S[W_WW][o], dw, v);
                v = wfma(p.S[W_WS][o], a1m, v);
                v = wfma(p.S[W_WQ][o], a1c, v);
                v = wfma(p.S[W_WN][o], a1p, v);
                dw = a1c - a2c;
                v = wfma(p.S[W_WE][o], -dw, v);
                if constexpr (KIND == 2) v = wfma(p.zeta, v, -p.S[W_IB][o] * a1c);
            } else {
                v = p.S[W_IB][o] * D1[o];
                v = wfma(p.zeta * p.S[W_WG][o], mix, v);
                if constexpr (SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD) {
                    T z = p.S[W_WW][o] * a0c;
                    z = wfma(p.S[W_WS][o], a1m, z);
                    z = wfma(p.S[W_WC][o], a1c, z);
                    z = wfma(p.S[W_WN][o], a1p, z);
                    z = wfma(-p.S[W_WE][o], a2c, z);
                    v = wfma(p.zt, z, v);
                }
            }
            if (t0 + r > e) v = hi;
            f[r] = v;
            q[r] = p.S[W_LA][o];
            if constexpr (R <= 8) g[r] = p.S[W_G][o];
            if constexpr (!SER) y = wfma(-q[r], y, v);
            a0c = a1c; a1c = a2c;
            a1m = a2m; a1p = a2p;
            q0 = q1; q1 = q2;
        }
        const bool more = tile + 1 < sp.tiles;
        auto sweep = [&](T z) -> T {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                z = wfma(-q[r], z, f[r]);
                f[r] = z;
                if (more && act && t0 + r <= e) Y[(long long)(t0 + r) * ld + j] = z;
            }
            return z;
        };
        if constexpr (SER) relay<T, true>(kf, in, sweep);
        else sweep(compose<T, true>(kf, y, preg, in));
    }
    in = hi;
    for (int tile = sp.tiles - 1; tile >= 0; --tile) {
        const int t0 = 1 + (tile * sp.PC + c) * R;
        const bool again = tile + 1 < sp.tiles;
        if (again) {
            __syncthreads();
            carry_load(kb, p.sb, p.ls, tile, j, bpreg);
        }
        T x = T(0);
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            const int t = t0 + r;
            const long long o = (long long)min(t, nx - 1) * ld + j;
            if (again) f[r] = t <= e ? Y[o] : hi;
            if (R > 8 || again) g[r] = p.S[W_G][o];
            if constexpr (!SER) x = wfma(-g[r], x, f[r]);
        }
        auto sweep = [&](T z) -> T {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) {
                z = wfma(-g[r], z, f[r]);
                if (act && t0 + r <= e) Y[(long long)(t0 + r) * ld + j] = z;
            }
            return z;
        };
        if constexpr (SER) relay<T, false>(kb, in, sweep);
        else sweep(compose<T, false>(kb, x, bpreg, in));
    }
}

// explicit v = v_lo boundary value of row i (explicit_boundary.hpp:39-84)
template <typename T> __device__ __forceinline__ T boundary1(const wparams<T> &p, const T *U, int i)
{
    const int N = p.nx - 1;
    const T *u = U + (long long)i * p.ld;
    if (i == 0) return p.yslo[0];
    const T r = wfma(p.xb2[i], u[2], wfma(p.xb1[i], u[1], p.xbc[i] * u[0]));
    if (i == N) return r + p.bnc;
    return wfma(p.xbp[i], u[p.ld], wfma(p.xbm[i], u[-p.ld], r));
}

// ------------------------------------------------------------------------------------------
// v stages.  KIND V_FIRST: D2 = V(D1).  V_LAST: next = U + V(D).  V_LAST_HV: next = U + D2 + V(D + E).
// Block 0 holds the last rows, so that the extrapolated row nx-1 (explicit_boundary.hpp:202-238)
// follows in the same CTA.
// ------------------------------------------------------------------------------------------
template <typename T, int R, int KIND, bool SER>
__global__ void __launch_bounds__(MAX_CTA) k_wide_v(const __grid_constant__ wparams<T> p, const T *U, const T *D, const T *E,
                                                    const T *D2, T *out)
{
    extern __shared__ __align__(16) unsigned char raw[];
    const split &sp = p.v;
    const int L = sp.L, lane = threadIdx.x % L, c = threadIdx.x / L;
    const int nx = p.nx, ny = p.ny, ld = p.ld;
    const int il = nx - 2 - ((int)blockIdx.x * L + lane);
    const bool act = il >= 1;
    const int i = max(il, 1);
    const long long row = (long long)i * ld;
    const carry<T> kf = make_carry(reinterpret_cast<T *>(raw), sp, 0, lane, c);
    const carry<T> kb = make_carry(reinterpret_cast<T *>(raw), sp, 1, lane, c);
    pdl_launch();
    T preg, bpreg;
    carry_load(kf, p.vf, p.lv, 0, i, preg);
    carry_load(kb, p.vb, p.lv, sp.tiles - 1, i, bpreg);
    const int ii = p.imap[i];
    const T hi = p.xvhi[ii];
    // columns past the row's end are read at its last four, with the tables taken as zero there
    auto col = [&](int t) -> long long { return row + min(t, ld - 4); };
    T f[R], q[R], g[R], ib[R];
    auto tables = [&](int t0) {
#pragma unroll
        for (int r = 0; r < R; r += 4) {
            ld4(p.V[W_VL] + col(t0 + r), q + r);
            ld4(p.V[W_VU] + col(t0 + r), g + r);
            if (R <= 8) ld4(p.V[W_VIB] + col(t0 + r), ib + r);
            if (t0 + r >= ld) {
#pragma unroll
                for (int z = 0; z < 4; ++z) q[r + z] = g[r + z] = T(0);
            }
        }
    };
    if (R <= 8) tables(c * R); // constant: loaded while the stage before finishes
    pdl_wait();
    T in = T(0), lo = T(0);
    if (c == 0) lo = boundary1(p, U, ii);
    const T u0 = U[row], un = U[row + ny - 1];
    for (int tile = 0; tile < sp.tiles; ++tile) {
        const int t0 = (tile * sp.PC + c) * R;
        if (tile > 0) {
            __syncthreads();
            carry_load(kf, p.vf, p.lv, tile, i, preg);
        }
        if (R > 8 || tile > 0) tables(t0);
#pragma unroll
        for (int r = 0; r < R; r += 4) {
            ld4(D + col(t0 + r), f + r);
            if constexpr (KIND == V_LAST_HV) {
                T ev[4];
                ld4(E + col(t0 + r), ev);
#pragma unroll
                for (int z = 0; z < 4; ++z) f[r + z] += ev[z];
            }
        }
        T y = T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int t = t0 + r;
            if (t == 0) f[r] = KIND == V_LAST_HV ? T(0) : lo - u0;
            if (t == ny - 1) f[r] = KIND == V_LAST_HV ? T(0) : hi - un;
            if (t >= ny) f[r] = T(0);
            if constexpr (!SER) y = wfma(-q[r], y, f[r]);
        }
        const bool more = tile + 1 < sp.tiles;
        auto sweep = [&](T z) -> T {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                z = wfma(-q[r], z, f[r]);
                f[r] = z;
                if ((r & 3) == 3 && more && act && t0 + r < ld) st4(out + row + t0 + r - 3, f + r - 3);
            }
            return z;
        };
        if constexpr (SER) relay<T, true>(kf, in, sweep);
        else sweep(compose<T, true>(kf, y, preg, in));
    }
    in = T(0);
    for (int tile = sp.tiles - 1; tile >= 0; --tile) {
        const int t0 = (tile * sp.PC + c) * R;
        const bool again = tile + 1 < sp.tiles;
        if (again) {
            __syncthreads();
            carry_load(kb, p.vb, p.lv, tile, i, bpreg);
            tables(t0);
#pragma unroll
            for (int r = 0; r < R; r += 4) ld4(out + col(t0 + r), f + r);
        }
        T x = T(0);
        if constexpr (!SER) {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) x = wfma(-g[r], x, f[r]);
        }
        // what the output needs is loaded before the composition waits
        T u[R];
        if constexpr (KIND != V_FIRST) {
#pragma unroll
            for (int r = 0; r < R; r += 4) {
                ld4(U + col(t0 + r), u + r);
                if constexpr (KIND == V_LAST_HV) {
                    T d2[4];
                    ld4(D2 + col(t0 + r), d2);
#pragma unroll
                    for (int z = 0; z < 4; ++z) u[r + z] += d2[z];
                }
            }
        }
        auto sweep = [&](T z) -> T {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) {
                z = wfma(-g[r], z, f[r]);
                f[r] = z;
            }
            return z;
        };
        if constexpr (SER) relay<T, false>(kb, in, sweep);
        else sweep(compose<T, false>(kb, x, bpreg, in));
#pragma unroll
        for (int r = R - 4; r >= 0; r -= 4) {
            if (R > 8) ld4(p.V[W_VIB] + col(t0 + r), ib + r);
            T o[4];
#pragma unroll
            for (int z = 3; z >= 0; --z) {
                const int t = t0 + r + z;
                if constexpr (KIND == V_FIRST) o[z] = ib[r + z] * f[r + z];
                else o[z] = wfma(ib[r + z], f[r + z], u[r + z]);
                if constexpr (KIND != V_FIRST) {
                    if (t == 0) o[z] = lo;
                    if (t == ny - 1) o[z] = hi;
                }
            }
            if (act && t0 + r < ld) st4(out + row + t0 + r, o);
        }
    }
    if (blockIdx.x == 0) {
        const int w = threadIdx.x, ws = blockDim.x;
        const long long lr = (long long)(nx - 1) * ld;
        if constexpr (KIND == V_FIRST) {
            for (int t = w; t < ny; t += ws) {
                out[t] = -U[t];
                out[lr + t] = -U[lr + t];
            }
        } else {
            __syncthreads();
            const T four3 = T(4.0 / 3.0), third = T(1.0 / 3.0);
            for (int t = w; t < ny; t += ws) {
                out[t] = p.yslo[t];
                const int tt = p.jmap[t];
                out[lr + t] = wfma(four3, __ldcg(out + lr - ld + tt), wfma(-third, __ldcg(out + lr - 2 * ld + tt), -p.yb2c[t]));
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// set-up
// ------------------------------------------------------------------------------------------
// Products of the chunks' end maps, in the shape of the solve: one CTA of L lines x PC chunks per
// tile and block of lines.  -fac of row t is the map's slope; rows outside first..last are
// identity rows of the boundary (slope 0).  Element t of line l at fac[t * ts + l * st]; the transposed
// solves of the adjoint take their row's factor from the row `shift` away.
template <typename T>
__global__ void __launch_bounds__(MAX_CTA) k_wide_products(const T *fac, long long ts, long long st, int lines, int first, int last,
                                                           int base, int shift, split sp, bool fwd, carry_tab<T> out, int ls)
{
    extern __shared__ __align__(16) unsigned char raw[];
    T *a = reinterpret_cast<T *>(raw);
    const int lane = threadIdx.x % sp.L, c = threadIdx.x / sp.L;
    const int tile = blockIdx.x % sp.tiles, l = blockIdx.x / sp.tiles * sp.L + lane;
    const bool act = l < lines;
    pdl_launch();
    pdl_wait();
    T pr = T(1);
    const int G = tile * sp.PC + c, t0 = base + G * sp.R;
    if (act)
        for (int r = 0; r < sp.R; ++r) {
            const int t = t0 + r;
            pr *= (t >= first && t <= last) ? -fac[(t + shift) * ts + l * st] : T(0);
        }
    a[c * sp.L + lane] = pr;
    __syncthreads();
    if (!act) return;
    const int at = fwd ? c : sp.PC - 1 - c, g0 = at / sp.gs * sp.gs;
    auto prod = [&](int from, int to) {
        T x = T(1);
        for (int q = from; q < to; ++q) x *= a[(fwd ? q : sp.PC - 1 - q) * sp.L + lane];
        return x;
    };
    const T in_group = prod(g0, at);
    const_cast<T *>(out.A)[(long long)G * ls + l] = pr;
    const_cast<T *>(out.PreG)[(long long)G * ls + l] = in_group;
    if (at == min(g0 + sp.gs, sp.PC) - 1)
        const_cast<T *>(out.GA)[(long long)(tile * sp.groups() + at / sp.gs) * ls + l] = in_group * pr;
}

// S-line tables of one line per thread (double arithmetic), from M, P, Z, Mt, Pt, W, C (pitch ld) and mpz, M + P - Z
template <typename T>
__device__ __forceinline__ void s_slots(T *s, long long n, double M, double P, double Z, double mpz, double Mt, double Pt, double W,
                                        double C, double gm, double ib, int t, int j)
{
    const T ws = static_cast<T>(Mt * ib), wn = static_cast<T>(Pt * ib);
    s[W_WG * n] = static_cast<T>(gm * C * ib);
    s[W_WW * n] = static_cast<T>(M * ib);
    s[W_WS * n] = ws;
    s[W_WQ * n] = center_weight<T>(mpz + ((Mt + Pt) - W), ib, ws, wn, t, j);
    s[W_WC * n] = static_cast<T>(-(Z + W) * ib);
    s[W_WN * n] = wn;
    s[W_WE * n] = static_cast<T>(P * ib);
}
template <typename T>
__global__ void k_wide_setup_s(const double *base, long long n, int nx, int ny, int ld, double th, double gm, T *S)
{
    const int j = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (j > ny - 2) return;
    const int e = nx - 2;
    double gam = 0.0;
    // the next row's coefficients are loaded before this row's stores: one latency per row
    // overlaps the divisions of the row before
    long long o = ld + j;
    double nv[7];
    for (int k = 0; k < 7; ++k) nv[k] = base[k * n + o];
    for (int t = 1; t <= e; ++t, o += ld) {
        double v[7];
        for (int k = 0; k < 7; ++k) v[k] = nv[k];
        if (t < e)
            for (int k = 0; k < 7; ++k) nv[k] = base[k * n + o + ld];
        const double a = -th * v[0], b = 1.0 + th * v[2], c = -th * v[1];
        const double ib = 1.0 / fma(-a, gam, b);
        gam = c * ib;
        T *s = S + o;
        s[W_LA * n] = static_cast<T>(a * ib);
        s[W_G * n] = static_cast<T>(gam);
        s[W_IB * n] = static_cast<T>(ib);
        s_slots(s, n, v[0], v[1], v[2], v[0] + v[1] - v[2], v[3], v[4], v[5], v[6], gm, ib, t, j);
    }
}
template <typename T>
__global__ void k_wide_setup_v(const double *base, long long n, int nx, int ny, int ld, double th, T *V)
{
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nx - 2) return;
    const double *Mt = base + 3 * n, *Pt = base + 4 * n, *W = base + 5 * n;
    const long long row = (long long)i * ld;
    T *L = V + row, *Uf = V + n + row, *IB = V + 2 * n + row;
    double ib = 0.0, cp = 0.0;
    IB[0] = T(1);
    for (int t = 1; t <= ny - 2; ++t) {
        const double a = -th * Mt[row + t], b = 1.0 + th * W[row + t], c = -th * Pt[row + t];
        const double l = t == 1 ? a : a * ib;
        ib = 1.0 / (t == 1 ? b : fma(-l, cp, b));
        L[t] = static_cast<T>(l);
        IB[t] = static_cast<T>(ib);
        if (t > 1) Uf[t - 1] = static_cast<T>(cp * ib);
        cp = c;
    }
    Uf[ny - 2] = static_cast<T>(cp);
    IB[ny - 1] = T(1);
}

// Time-dependent coefficients (SABR with r != 0): a and c carry da = D(t)^(2(1-beta)) and dc =
// D(t)^(1-beta), so that at a step's time
//   M = da ma + mb,  P = da pa - mb,  Z = da (ma + pa) + z0,  C = dc cs
// with ma, pa, cs per point and mb per row (general_heston_equation_coefficients, coefficients.hpp:89-98,
// on the transformed data of lss_heat_data_transform.hpp:174-214).
struct tdep_tab {
    const double *ma, *pa, *cs, *mt, *pt, *w; // pitch ld
    const double *mb;                         // nx
    const double *am, *bm;                    // nx: boundary weights XB_M = -(da am + bm), XB_P = da am + bm
    double z0, th, gm;
    int nx, ny, ld;
    long long n;
};
// One step's set of tables among those of a group: S-line tables, boundary weights, chunk products.
struct tdep_set {
    double *S, *xb;                // of the group's first step: W_COUNT n; XB_M and XB_P, nx each
    carry_tab<double> sf, sb, sz, sw; // (sz, sw: the transposed solves', null A without them)
    long long stride;              // doubles from one step's set to the next
};
constexpr int TDEP_STEPS = 16;
struct tdep_steps {
    double da[TDEP_STEPS], dc[TDEP_STEPS];
};
// 2^-e of the largest of four magnitudes (1 for zero): the exponent field's arithmetic, no FP64
__device__ __forceinline__ double pow2_inverse(double a, double b, double c, double d)
{
    const int top = 0x7fffffff;
    const int m = max(max(__double2hiint(a) & top, __double2hiint(b) & top), max(__double2hiint(c) & top, __double2hiint(d) & top)) >> 20;
    return m == 0 || m > 2044 ? 1.0 : __hiloint2double((2046 - m) << 20, 0);
}
// All S-line tables of a group of steps (blockIdx.y: the step) in the shape of the S stages' split: a
// CTA factorises its lines, writes factors and right-hand-side slots and composes the chunks' products.
// beta_t = b_t - a_t c_{t-1} / beta_{t-1} is the Moebius map of the matrix [[b_t, -a_t c_{t-1}], [1, 0]]
// applied to beta_{t-1}: each chunk forms the product of its rows' matrices (scaled by powers of two:
// only the ratio matters), the chunks' maps are composed like the solves' end maps, a chunk then runs
// its own rows' recurrence from its incoming beta.
// What bounds it: FP64 instructions (about 45 per point, one division among them) as long as the grid
// fills the GPU, which the steps of a group are there for.  A launch per step of 32 CTAs, followed by
// one for the slots and one for each sweep's products, took 115 to 240 us of a 512 x 256 step.
template <int R>
__global__ void __launch_bounds__(MAX_CTA) k_wide_tdep(const __grid_constant__ tdep_tab q, const __grid_constant__ tdep_steps steps,
                                                       const __grid_constant__ tdep_set set, const __grid_constant__ split sp, int ls)
{
    extern __shared__ __align__(16) unsigned char raw[];
    const int L = sp.L, PC = sp.PC, ng = sp.groups(), gs = sp.gs, lane = threadIdx.x % L, c = threadIdx.x / L;
    const int j = 1 + blockIdx.x * L + lane, e = q.nx - 2, w = L * PC, at = c * L + lane;
    const bool act = j <= q.ny - 2;
    double *sm = reinterpret_cast<double *>(raw), *gm = sm + 4 * w; // chunks' maps (later products), groups' maps
    const double th = q.th, da = steps.da[blockIdx.y], dc = steps.dc[blockIdx.y];
    const long long off = blockIdx.y * set.stride;
    double *S = set.S + off;
    pdl_launch();
    double in = 1.0; // beta of the row before the tile: row 1's map ignores it (a_1 c_0 = 0)
    bool waited = false;
    for (int tile = 0; tile < sp.tiles; ++tile) {
        const int G = tile * PC + c, t0 = 1 + G * R;
        double m[R], pp[R];
        double cin = 0.0; // c of the row before the chunk
        if (act) {
            if (t0 > 1 && t0 <= e + 1) cin = -th * fma(da, q.pa[(long long)(t0 - 1) * q.ld + j], -q.mb[t0 - 1]);
            double m11 = 1.0, m12 = 0.0, m21 = 0.0, m22 = 1.0, cp = cin;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int t = t0 + r;
                m[r] = pp[r] = 0.0;
                if (t > e) continue;
                const long long o = (long long)t * q.ld + j;
                m[r] = fma(da, q.ma[o], q.mb[t]);
                pp[r] = fma(da, q.pa[o], -q.mb[t]);
                const double b = fma(th, m[r] + pp[r] + q.z0, 1.0), ac = (-th * m[r]) * cp;
                cp = -th * pp[r];
                const double n11 = b * m11 - ac * m21, n12 = b * m12 - ac * m22;
                m21 = m11; m22 = m12; m11 = n11; m12 = n12;
                if ((r & 7) == 7 || r == R - 1 || t == e) {
                    const double sc = pow2_inverse(m11, m12, m21, m22);
                    m11 *= sc; m12 *= sc; m21 *= sc; m22 *= sc;
                }
            }
            sm[at] = m11; sm[w + at] = m12; sm[2 * w + at] = m21; sm[3 * w + at] = m22;
        }
        __syncthreads();
        if (act && c < ng) { // this thread's group: maps of the chunks before each one in the group
            double m11 = 1.0, m12 = 0.0, m21 = 0.0, m22 = 1.0;
            const int q1 = min((c + 1) * gs, PC);
            for (int k = c * gs; k < q1; ++k) {
                const int z = k * L + lane;
                const double a11 = sm[z], a12 = sm[w + z], a21 = sm[2 * w + z], a22 = sm[3 * w + z];
                sm[z] = m11; sm[w + z] = m12; sm[2 * w + z] = m21; sm[3 * w + z] = m22;
                const double n11 = a11 * m11 + a12 * m21, n12 = a11 * m12 + a12 * m22;
                const double n21 = a21 * m11 + a22 * m21, n22 = a21 * m12 + a22 * m22;
                const double sc = pow2_inverse(n11, n12, n21, n22);
                m11 = n11 * sc; m12 = n12 * sc; m21 = n21 * sc; m22 = n22 * sc;
            }
            const int z = 4 * (c * L + lane);
            gm[z] = m11; gm[z + 1] = m12; gm[z + 2] = m21; gm[z + 3] = m22;
        }
        __syncthreads();
        if (act && c == 0) { // beta as a ratio x / y through the groups
            double x = in, y = 1.0;
            for (int k = 0; k < ng; ++k) {
                double *g = gm + 4 * (k * L + lane);
                const double a11 = g[0], a12 = g[1], a21 = g[2], a22 = g[3];
                g[0] = x; g[1] = y;
                const double nx = a11 * x + a12 * y, ny = a21 * x + a22 * y;
                const double sc = pow2_inverse(nx, ny, 0.0, 0.0);
                x = nx * sc; y = ny * sc;
            }
            in = x / y;
        }
        __syncthreads();
        double prl = 1.0, prb = 1.0, prz = 1.0; // products of this chunk's slopes (prl: la without its first row's)
        double la1 = 0.0;                       // la of the chunk's first row
        double gam = 0.0, la_next = 0.0;
        if (act) {
            const double x = gm[4 * (c / gs * L + lane)], y = gm[4 * (c / gs * L + lane) + 1];
            // incoming beta; gamma of the row before the chunk
            const double bx = sm[at] * x + sm[w + at] * y, by = sm[2 * w + at] * x + sm[3 * w + at] * y;
            gam = cin != 0.0 ? cin * by / bx : 0.0;
        }
        if (!waited) pdl_wait(); // the stages that read the sets before are done
        waited = true;
        if (act) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int t = t0 + r;
                prz *= t <= e ? -gam : 0.0;
                if (t > e) {
                    prl = prb = 0.0;
                    continue;
                }
                const long long o = (long long)t * q.ld + j;
                const double z = m[r] + pp[r] + q.z0;
                const double ib = 1.0 / fma(th * m[r], gam, fma(th, z, 1.0));
                const double la = (-th * m[r]) * ib;
                gam = (-th * pp[r]) * ib;
                S[W_IB * q.n + o] = ib;
                S[W_G * q.n + o] = gam;
                S[W_LA * q.n + o] = la;
                s_slots(S + o, q.n, m[r], pp[r], z, -q.z0, q.mt[o], q.pt[o], q.w[o], dc * q.cs[o], q.gm, ib, t, j);
                if (r == 0) la1 = la;
                else prl *= -la;
                prb *= -gam;
            }
            // la of the row after the tile (the tile's last chunk): pivot from its own row
            if (c == PC - 1 && t0 + R <= e) {
                const long long o = (long long)(t0 + R) * q.ld + j;
                const double mm = fma(da, q.ma[o], q.mb[t0 + R]), p1 = fma(da, q.pa[o], -q.mb[t0 + R]);
                la_next = (-th * mm) / fma(th * mm, gam, fma(th, mm + p1 + q.z0, 1.0));
            }
        }
        __syncthreads(); // every thread has its incoming beta: the maps' arrays become the products'
        if (act) {
            sm[at] = -la1 * prl;
            sm[w + at] = prb;
            sm[2 * w + at] = prz;
            gm[at] = la1;
        }
        __syncthreads();
        if (act && set.sw.A) { // slopes of the transposed back sweep: la of the row after
            sm[3 * w + at] = -(c < PC - 1 ? gm[at + L] : la_next) * prl;
        }
        __syncthreads();
        // products of the chunks before each in its group, of the groups; sweep u / ng, group u % ng
        const int sweeps = set.sw.A ? 4 : 2;
        for (int u = c; act && u < sweeps * ng; u += PC) {
            const int sw = u / ng, g = u % ng;
            const carry_tab<double> &t = sw == 0 ? set.sf : sw == 1 ? set.sb : sw == 2 ? set.sz : set.sw;
            const bool fwd = (sw & 1) == 0;
            double pr = 1.0;
            for (int k = g * gs; k < min((g + 1) * gs, PC); ++k) {
                const int ch = fwd ? k : PC - 1 - k;
                const long long o = (long long)(tile * PC + ch) * ls + j + off;
                const double a = sm[sw * w + ch * L + lane];
                const_cast<double *>(t.A)[o] = a;
                const_cast<double *>(t.PreG)[o] = pr;
                pr *= a;
            }
            const_cast<double *>(t.GA)[(long long)(tile * ng + g) * ls + j + off] = pr;
        }
        __syncthreads();
    }
    // the boundary column's weights
    if (blockIdx.x == 0) {
        double *xb = set.xb + off;
        for (int i = threadIdx.x; i < q.nx; i += blockDim.x) {
            const double d = fma(da, q.am[i], q.bm[i]);
            xb[i] = -d;
            xb[q.nx + i] = d;
        }
    }
}

// initial condition into the pitched state; final surface out of it, with its value and finiteness
template <typename T> __global__ void k_wide_begin(const T *pay, T *U, int nx, int ny, int ld, int *status)
{
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q == 0) *status = 0;
    if (q >= (long long)nx * ny) return;
    const int i = static_cast<int>(q / ny), j = static_cast<int>(q % ny);
    U[(long long)i * ld + j] = pay[q];
}
template <typename T>
__global__ void k_wide_end(const T *U, int nx, int ny, int ld, bilinear b, T *surface, double *value, int *status)
{
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int bad = 0;
    if (q < (long long)nx * ny) {
        const int i = static_cast<int>(q / ny), j = static_cast<int>(q % ny);
        const T v = U[(long long)i * ld + j];
        surface[q] = v;
        bad = !isfinite(static_cast<double>(v));
    }
    bad = __syncthreads_or(bad);
    if (bad && threadIdx.x == 0) atomicOr(status, 1);
    if (q == 0) {
        const long long o = (long long)b.i0 * ld + b.j0;
        *value = fma(b.w11, static_cast<double>(U[o + ld + 1]),
                     fma(b.w01, static_cast<double>(U[o + 1]), fma(b.w10, static_cast<double>(U[o + ld]), b.w00 * static_cast<double>(U[o]))));
    }
}

// ------------------------------------------------------------------------------------------
// Adjoint of a time step (FP64).  The transposed solve of an S line, given xbar:
//   z_t = xbar_t - g_{t-1} z_{t-1},  w_t = z_t - la_{t+1} w_{t+1};  fbar = w, lobar = -la_1 w_1, hibar = -g_e z_e
// and of a v line z_t = ib_t xbar_t - u_{t-1} z_{t-1}, w_t = z_t - l_{t+1} w_{t+1}, dbar = w (the
// identity rows give the boundary values' adjoints w_0, w_{ny-1}).  In delta form the state's
// adjoint passes through the step unchanged but for its ends and F's transpose, so one array VB
// is updated in place.  Parameter sensitivities of an S solve (I - theta A1) Y = rhs(X) are
// mu . (d rhs X + theta dA1 Y), mu = ib w; of a v solve w . theta dA2 x.  Both are accumulated by the
// S kernels, where the coefficient derivatives' v factors are constant along a thread's line (in relay
// order by k_wadj_lines, for a run of steps).
// ------------------------------------------------------------------------------------------
struct adj_params {
    const double *hx, *hc, *ha, *hdd;          // nx
    const double *hy, *bs, *ek, *et, *es, *hv2; // ny
    double delta, halfk, ni, betat, sigma, rho, theta, zeta, gamma, k, alphat, omb;
    double dw;                                  // weight of the D2 terms: zeta - theta (modified), zeta (HV)
    int sabr;
    carry_tab<double> sz, sw, vz, vw;
};

template <int R, int KIND, bool SER>
__global__ void __launch_bounds__(MAX_CTA) k_wadj_v(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params q,
                                                    const double *XB, double *VB, double *DB, double *LV, int add_lv)
{
    extern __shared__ __align__(16) unsigned char raw[];
    const split &sp = p.v;
    const int L = sp.L, lane = threadIdx.x % L, c = threadIdx.x / L;
    const int nx = p.nx, ny = p.ny, ld = p.ld;
    const int il = nx - 2 - ((int)blockIdx.x * L + lane);
    const bool act = il >= 1;
    const int i = max(il, 1);
    const long long row = (long long)i * ld, lr = (long long)(nx - 1) * ld;
    const carry<double> kf = make_carry(reinterpret_cast<double *>(raw), sp, 0, lane, c);
    const carry<double> kb = make_carry(reinterpret_cast<double *>(raw), sp, 1, lane, c);
    pdl_launch();
    double preg, bpreg;
    carry_load(kf, q.vz, p.lv, 0, i, preg);
    carry_load(kb, q.vw, p.lv, sp.tiles - 1, i, bpreg);
    auto col = [&](int t) -> long long { return row + min(t, ld - 4); };
    // b2^T: rows nx-2 and nx-3 take the extrapolated row's adjoint
    const double fold = KIND == V_FIRST ? 0.0 : il == nx - 2 ? 4.0 / 3.0 : il == nx - 3 ? -1.0 / 3.0 : 0.0;
    double f[R], g[R];
    double in = 0.0;
    pdl_wait();
    for (int tile = 0; tile < sp.tiles; ++tile) {
        const int t0 = (tile * sp.PC + c) * R;
        if (tile > 0) {
            __syncthreads();
            carry_load(kf, q.vz, p.lv, tile, i, preg);
        }
        double ib[R];
#pragma unroll
        for (int r = 0; r < R; r += 4) {
            ld4(XB + col(t0 + r), f + r);
            ld4(p.V[W_VIB] + col(t0 + r), ib + r);
            double u[4];
            ld4(p.V[W_VU] + col(t0 + r), u);
            g[r] = t0 + r > 0 ? p.V[W_VU][row + min(t0 + r - 1, ld - 1)] : 0.0;
#pragma unroll
            for (int z = 1; z < 4; ++z) g[r + z] = u[z - 1];
        }
        if (fold != 0.0) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int t = t0 + r;
                if (t < ny) {
                    double a = p.jmap[t] == t ? XB[lr + t] : 0.0;
                    if (t + 1 < ny && p.jmap[t + 1] == t) a += XB[lr + t + 1];
                    f[r] = fma(fold, a, f[r]);
                    VB[row + t] = f[r];
                }
            }
        }
        double z = 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            f[r] = t0 + r < ny ? ib[r] * f[r] : 0.0;
            if (t0 + r >= ny) g[r] = 0.0;
            if constexpr (!SER) z = fma(-g[r], z, f[r]);
        }
        const bool more = tile + 1 < sp.tiles;
        auto sweep = [&](double y) -> double {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                y = fma(-g[r], y, f[r]);
                f[r] = y;
                if ((r & 3) == 3 && more && act && t0 + r < ld) st4(DB + row + t0 + r - 3, f + r - 3);
            }
            return y;
        };
        if constexpr (SER) relay<double, true>(kf, in, sweep);
        else sweep(compose<double, true>(kf, z, preg, in));
    }
    in = 0.0;
    for (int tile = sp.tiles - 1; tile >= 0; --tile) {
        const int t0 = (tile * sp.PC + c) * R;
        if (tile + 1 < sp.tiles) {
            __syncthreads();
            carry_load(kb, q.vw, p.lv, tile, i, bpreg);
#pragma unroll
            for (int r = 0; r < R; r += 4) ld4(DB + col(t0 + r), f + r);
        }
#pragma unroll
        for (int r = 0; r < R; r += 4) { // l of the row after
            double l[4];
            ld4(p.V[W_VL] + col(t0 + r), l);
#pragma unroll
            for (int z = 1; z < 4; ++z) g[r + z - 1] = l[z];
            g[r + 3] = t0 + r + 4 < ld ? p.V[W_VL][row + t0 + r + 4] : 0.0;
            if (t0 + r >= ld) {
#pragma unroll
                for (int z = 0; z < 4; ++z) f[r + z] = g[r + z] = 0.0;
            }
        }
        double w = 0.0;
        if constexpr (!SER) {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) w = fma(-g[r], w, f[r]);
        }
        auto sweep = [&](double y) -> double {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) {
                y = fma(-g[r], y, f[r]);
                f[r] = y;
            }
            return y;
        };
        if constexpr (SER) relay<double, false>(kb, in, sweep);
        else sweep(compose<double, false>(kb, w, bpreg, in));
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            const int t = t0 + r;
            w = f[r];
            if constexpr (KIND != V_LAST_HV) {
                if (act && t == ny - 1) VB[row + t] -= w;
                if (act && t == 0) {
                    VB[row] -= w;
                    LV[i] = add_lv ? LV[i] + w : w;
                }
            }
            if ((r & 3) == 0 && act && t < ld) st4(DB + row + t, f + r);
        }
    }
    if (KIND != V_FIRST && blockIdx.x == 0) { // rows 0 and nx-1 of the state do not reach the step's input
        __syncthreads();
        for (int t = threadIdx.x; t < ny; t += blockDim.x) VB[t] = VB[lr + t] = 0.0;
    }
}

// Parameter sums of one thread (rows of one line) of an S kernel, before the line's v factors.
struct s_acc {
    double A, Y, E, B, C, Q, S, Aa, Ya, Dd, Yd, v0, vm, vd;
};

template <int R, int KIND, int SCH, bool SER>
__global__ void __launch_bounds__(MAX_CTA) k_wadj_s(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params q,
                                                const double *U, const double *Vn, const double *D1, const double *D2, const double *Y,
                                                const double *XB, const double *DV, double *VB, double *FB, double *MU, double *LS,
                                                double *HS, double *acc, long long nacc, double tau, double da, double dc)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD, dr = SCH == LSS_ADI_DOUGLAS_RACHFORD;
    constexpr bool xt = KIND == 2 && (hv || mcs); // D2 terms besides the mixed one
    extern __shared__ __align__(16) unsigned char raw[];
    const split &sp = p.s;
    const int L = sp.L, lane = threadIdx.x % L, c = threadIdx.x / L;
    const int nx = p.nx, ny = p.ny, ld = p.ld, e = nx - 2;
    const int jl = blockIdx.x * L + lane;
    const bool act = jl >= 1 && jl <= ny - 2;
    const int j = min(max(jl, 1), ny - 2);
    const carry<double> kf = make_carry(reinterpret_cast<double *>(raw), sp, 0, lane, c);
    const carry<double> kb = make_carry(reinterpret_cast<double *>(raw), sp, 1, lane, c);
    pdl_launch();
    if (p.tdep) pdl_wait();
    double preg, bpreg;
    carry_load(kf, q.sz, p.ls, 0, j, preg);
    carry_load(kb, q.sw, p.ls, sp.tiles - 1, j, bpreg);
    if (!p.tdep) pdl_wait();
    auto at = [&](int t) -> long long { return (long long)min(t, nx - 1) * ld + j; };
    double f[R], g[R];
    double in = 0.0;
    for (int tile = 0; tile < sp.tiles; ++tile) {
        const int t0 = 1 + (tile * sp.PC + c) * R;
        if (tile > 0) {
            __syncthreads();
            carry_load(kf, q.sz, p.ls, tile, j, preg);
        }
        double z = 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long long o = at(t0 + r);
            double x = XB[o];
            if constexpr (KIND == 1 && !dr) x += DV[o];
            f[r] = t0 + r <= e ? x : 0.0;
            g[r] = t0 + r <= e ? p.S[W_G][o - ld] : 0.0; // row 0 of the table is zero
            if constexpr (!SER) z = fma(-g[r], z, f[r]);
        }
        const bool more = tile + 1 < sp.tiles;
        auto sweep = [&](double y) -> double {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                y = fma(-g[r], y, f[r]);
                f[r] = y;
            }
            return y;
        };
        if constexpr (SER) relay<double, true>(kf, in, sweep);
        else sweep(compose<double, true>(kf, z, preg, in));
#pragma unroll
        for (int r = 0; r < R; ++r) {
            z = f[r];
            if (more && act && t0 + r <= e) FB[at(t0 + r)] = z;
            if (act && t0 + r == e) { // adjoint of the upper value
                const double h = -p.S[W_G][at(e)] * z;
                if constexpr (KIND == 2 && hv) VB[at(nx - 1)] += h;
                else HS[j] = KIND == 1 && !dr && !hv ? HS[j] + h : h;
            }
        }
    }
    in = 0.0;
    s_acc s = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int tile = sp.tiles - 1; tile >= 0; --tile) {
        const int t0 = 1 + (tile * sp.PC + c) * R;
        const bool again = tile + 1 < sp.tiles;
        if (again) {
            __syncthreads();
            carry_load(kb, q.sw, p.ls, tile, j, bpreg);
        }
        double w = 0.0;
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            if (again) f[r] = t0 + r <= e ? FB[at(t0 + r)] : 0.0;
            g[r] = t0 + r < e ? p.S[W_LA][at(t0 + r + 1)] : 0.0;
            if constexpr (!SER) w = fma(-g[r], w, f[r]);
        }
        auto sweep = [&](double y) -> double {
#pragma unroll
            for (int r = R - 1; r >= 0; --r) {
                y = fma(-g[r], y, f[r]);
                f[r] = y;
            }
            return y;
        };
        if constexpr (SER) relay<double, false>(kb, in, sweep);
        else sweep(compose<double, false>(kb, w, bpreg, in));
        auto store = [&](int t, long long o, double w, double mu) {
            if (!act) return;
            FB[o] = w;
            if constexpr (KIND == 2 && !hv) MU[o] = mu; // adjoint of D1
            if (t == 1) {
                const double l = -p.S[W_LA][o] * w;
                if constexpr (KIND == 2 && hv) VB[j] += l;
                else LS[j] = KIND == 1 && !dr && !hv ? LS[j] + l : l;
            }
        };
        if (acc == nullptr) { // the sums: k_wadj_lines
#pragma unroll
            for (int r = R - 1; r >= 0; --r) {
                const long long o = at(t0 + r);
                if (t0 + r <= e) store(t0 + r, o, f[r], p.S[W_IB][o] * f[r]);
            }
            continue;
        }
        // X: the operand of the explicit terms (U, or D2), Y: the stage's result; rows t+1, t, t-1
        const double *X = KIND == 1 ? U : D2;
        double xh = X[at(t0 + R)], xc = X[at(t0 + R - 1)], yh = Y[at(t0 + R)], yc = Y[at(t0 + R - 1)];
        double ddh = X[at(t0 + R) - 1] - X[at(t0 + R) + 1];
        double ss = X[at(t0 + R - 1) - 1];
        double ddc = ss - X[at(t0 + R - 1) + 1];
#pragma unroll
        for (int r = R - 1; r >= 0; --r) {
            const int t = t0 + r;
            const long long o = at(t), ol = at(t - 1);
            w = f[r];
            const double xl = X[ol], yl = Y[ol], sl = X[ol - 1], ddl = sl - X[ol + 1];
            if (t <= e) {
                const double mu = p.S[W_IB][o] * w;
                store(t, o, w, mu);
                const double mx = mu * q.hx[t], mc = q.sabr ? mu * q.hc[t] : mx;
                const double dy = yh - yl;
                s.Y = fma(mx, dy, s.Y);
                s.B = fma(mu, yc, s.B);
                s.E = fma(mc, ddl - ddh, s.E);
                double dx = 0.0;
                if constexpr (KIND == 1 || xt) {
                    dx = KIND == 2 && mcs ? -xh - xl : xh - xl;
                    s.A = fma(mx, dx, s.A);
                    s.C = fma(mu, xc, s.C);
                    s.Q = fma(mu, ddc, s.Q);
                    s.S = fma(mu, ss - xc, s.S);
                }
                if (q.sabr) {
                    const double ma = mu * q.ha[t], md = mu * q.hdd[t];
                    s.Ya = fma(ma, yl + yh - 2.0 * yc, s.Ya);
                    s.Yd = fma(md, dy, s.Yd);
                    if constexpr (KIND == 1 || xt) {
                        s.Aa = fma(ma, xl + (KIND == 2 && mcs ? -xh : xh) - 2.0 * xc, s.Aa);
                        s.Dd = fma(md, dx, s.Dd);
                    }
                }
                // v solve whose right-hand side this stage produced (DR, last v stage), or whose
                // result is D2 (first v stage)
                double m, x0, x1, x2;
                if constexpr (KIND == 1 && !dr) {
                    m = DV[o];
                    x0 = D2[o - 1]; x1 = D2[o]; x2 = D2[o + 1];
                } else {
                    m = XB[o];
                    x0 = Vn[o - 1] - U[o - 1]; x1 = Vn[o] - U[o]; x2 = Vn[o + 1] - U[o + 1];
                    if constexpr (hv) { x0 -= D2[o - 1]; x1 -= D2[o]; x2 -= D2[o + 1]; }
                }
                s.vd = fma(m, x2 - x0, s.vd);
                s.v0 = fma(m, x1, s.v0);
                s.vm = fma(m, x0 - x1, s.vm);
            }
            xh = xc; xc = xl;
            yh = yc; yc = yl;
            ddh = ddc; ddc = ddl;
            ss = sl;
        }
    }
    if (!act || acc == nullptr) return;
    // the line's sums: theta weighs the terms in Y, dw (1 for the first stage) those in X
    const double th = q.theta, wx = KIND == 1 ? 1.0 : q.dw, we = KIND == 1 ? 1.0 : q.zeta;
    const double A = th * s.Y + wx * s.A;
    const double B = -(th * s.B + 2.0 * wx * s.C);
    const double Q = -wx * s.Q, D = wx * (2.0 * s.S - s.Q), E = we * q.gamma * dc * s.E;
    const double ek = q.ek[j], et = q.et[j], es = q.es[j], bs = q.bs[j], hy = q.hy[j];
    double g0 = q.delta * A + q.halfk * B;
    if (q.sabr) {
        const double Aa = da * (th * s.Ya + wx * s.Aa), Dd = da * (th * s.Yd + wx * s.Dd);
        g0 += tau * q.omb * (q.hv2[j] * (2.0 * q.delta * Dd - 2.0 * q.alphat * Aa) - q.rho * q.sigma * hy * E);
    }
    const double vq = th * q.ni * s.vd, vs = th * q.betat * (2.0 * s.vm + s.vd);
    g0 -= q.halfk * th * s.v0;
    const double g1 = ek * (q.ni * Q + vq), g2 = et * (q.ni * Q + vq);
    const double g3 = es * (q.ni * Q + vq) + bs * (q.betat * D + vs) + q.rho * hy * E, g4 = q.sigma * hy * E;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    acc[t] += g0;
    acc[nacc + t] += g1;
    acc[2 * nacc + t] += g2;
    acc[3 * nacc + t] += g3;
    acc[4 * nacc + t] += g4;
}

// Cross-line adjoints of an S stage, one thread per grid point (p, q).  KIND 2: adjoint of D2 (for HV
// on top of the state's adjoint, next = U + D2 + ...; rows 0 and nx-1 are -U).  KIND 1: F^T into the
// state's adjoint, the S lines' boundary values (index_of remap) and the explicit v = v_lo column
// with its parameter sensitivities (acc slots of the rows; without acc k_wadj_rows has them).
template <int KIND, int SCH>
__global__ void __launch_bounds__(256) k_wadj_gather(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params a,
                                                     const double *U, const double *FB, double *D2B, double *VB, const double *LS,
                                                     const double *HS, const double *LV, double *acc, long long nacc, double tau, double da)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD;
    const int nx = p.nx, ny = p.ny, ld = p.ld;
    const long long n = (long long)nx * ny, id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_launch();
    pdl_wait();
    if (id >= n) return;
    const int r = static_cast<int>(id / ny), q = static_cast<int>(id % ny);
    const long long o = (long long)r * ld + q;
    // Row t contributes down (to t-1), up (to t+1) and mid (to t) terms from FB and the tables at
    // columns q-1, q, q+1 (the operations of da_gather, in its order); FB and the tables are zero on
    // boundary rows and columns, only points outside need a guard.
    constexpr bool six = KIND == 1 || hv || mcs;
    const bool lf = q >= 1, rt = q + 1 < ny;
    auto F = [&](long long at, bool ok) { return ok ? FB[at] : 0.0; };
    auto W = [&](int slot, long long at, bool ok) { return ok ? p.S[slot][at] : 0.0; };
    auto mixed = [&](long long t) { return fma(W(W_WG, t + 1, rt), F(t + 1, rt), -W(W_WG, t - 1, lf) * F(t - 1, lf)); };
    double dn = 0.0, up = 0.0, mid = 0.0;
    if (r + 1 < nx) {
        const long long t = o + ld;
        const double g = mixed(t);
        dn = !six ? g : KIND == 2 && mcs ? fma(p.zeta, g, p.zt * (p.S[W_WW][t] * FB[t])) : fma(p.S[W_WW][t], FB[t], g);
    }
    if (r > 0) {
        const long long t = o - ld;
        const double g = mixed(t);
        up = !six ? -g : KIND == 2 && mcs ? -fma(p.zeta, g, p.zt * (p.S[W_WE][t] * FB[t])) : fma(p.S[W_WE][t], FB[t], -g);
    }
    double x = dn + up;
    if constexpr (six) {
        mid = fma(W(W_WS, o + 1, rt), F(o + 1, rt), fma(W(W_WN, o - 1, lf), F(o - 1, lf), p.S[W_WC][o] * FB[o]));
        x += KIND == 2 && mcs ? __dmul_rn(p.zt, mid) : mid; // rounded by itself, as there
    }
    if constexpr (KIND == 2) {
        const double d = hv ? fma(p.zeta, x, -(p.S[W_IB][o] * FB[o])) : mcs ? x : p.zeta * x;
        if (r == 0 || r == nx - 1) VB[o] -= d;
        else D2B[o] = hv ? VB[o] + d : d;
    } else {
        if (r == 0 || r == nx - 1) {
            const double *E = r == 0 ? LS : HS;
            double s = q >= 1 && q <= ny - 2 && p.jmap[q] != q ? -E[q] : 0.0;
            if (q + 1 <= ny - 2 && p.jmap[q + 1] == q) s += E[q + 1];
            x += s;
        }
        double v = VB[o] + x;
        if (q <= 2) {
            auto B0 = [&](int i) -> double { // adjoint of the boundary value of row i
                if (i < 1 || i > nx - 2) return 0.0;
                double sum = p.imap[i] == i ? LV[i] : 0.0;
                if (i + 1 <= nx - 2 && p.imap[i + 1] == i) sum += LV[i + 1];
                return sum;
            };
            const double bb = B0(r);
            if (q == 1) v = fma(p.xb1[r], bb, v);
            else if (q == 2) v = fma(p.xb2[r], bb, v);
            else {
                const double below = r >= 1 ? p.xbp[r - 1] : 0.0, above = r + 1 <= nx - 2 ? p.xbm[r + 1] : 0.0;
                v += fma(below, B0(r - 1), fma(p.xbc[r], bb, above * B0(r + 1)));
                if (acc != nullptr && bb != 0.0) {
                    const double u0 = U[o], u1 = U[o + 1], u2 = U[o + 2];
                    const double ee = a.ni * bb * (4.0 * u1 - 3.0 * u0 - u2);
                    double hd = a.hx[r];
                    if (a.sabr) hd += 2.0 * a.omb * tau * a.hv2[0] * a.hdd[r] * da;
                    acc[r] += bb * (a.delta * hd * (U[o + ld] - U[o - ld]) - a.k * u0);
                    acc[nacc + r] += ee * a.ek[0];
                    acc[2 * nacc + r] += ee * a.et[0];
                    acc[3 * nacc + r] += ee * a.es[0];
                }
            }
        }
        VB[o] = v;
    }
}

// Parameter sums of an adjoint in relay order, from the arrays of a run of steps of a checkpoint segment: with the
// operations of the batched kernel (da_s, da_b1) in its order, so that the gradients have the bits of the
// same instance in a batch, on a warp group of its own class.  They are small against their terms where the
// scheme has growing modes: with a thread per chunk and its own partial sums, 4 of 240 small calls came out
// more than 1e-13 from the batch's.  The stages, where the sums were a chain of every step, are left with
// the solves (k_wadj_s without acc), and the sums of many steps are made at once: 128 x 64 x
// 200 Craig-Sneyd 23.4 ms with sensitivities, 26.1 ms with the sums in the stages.
struct line_sums {
    const double *u0, *seg;                     // state of the first step; U, D1, D2, D3 of step k at seg + 4 k n
    const double *FB, *DB, *DV, *LV;            // FB: stages 2 and 1 of step k at FB + 2 k n
    double *terms, *rows, *acc;                 // terms of line l: [step][stage][4][lp]; of row p: [step][3][rp]
    long long n;
    int len, lp, rp, threads;                   // steps; lines, rows of a multiple of 32; threads of the batch's group
    int n0;                                     // number of the first of them
    double tau, dtau;                           // time of step 0, of a step
    __device__ __forceinline__ const double *U(int k) const { return k == 0 ? u0 : seg + 4LL * k * n; }
};

// What bounds it: a line's FP64 instructions (25 per row); a thread per line and step, so the whole GPU has work.
template <int KIND, int SCH>
__global__ void __launch_bounds__(128) k_wadj_lines(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params q,
                                                    const __grid_constant__ line_sums g)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD, dr = SCH == LSS_ADI_DOUGLAS_RACHFORD;
    constexpr bool xt = KIND == 2 && (hv || mcs); // D2 terms besides the mixed one
    constexpr bool first_v = KIND == 1 && !dr;
    const int nx = p.nx, ny = p.ny, ld = p.ld, e = nx - 2;
    const long long last = (nx - 1LL) * ld, id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = static_cast<int>(id / g.lp), l = static_cast<int>(id % g.lp), j = l + 1;
    if (k >= g.len || j > ny - 2) return;
    const bool sabr = q.sabr;
    const double *U = g.U(k), *Vn = g.U(k + 1), *D1 = g.seg + (4LL * k + 1) * g.n, *D2 = D1 + g.n, *D3 = D2 + g.n;
    const double *X = KIND == 1 ? U : D2, *Y = KIND == 1 ? D1 : D3;
    const double *FB = g.FB + (2LL * k + (KIND == 1 ? 1 : 0)) * g.n, *M = (first_v ? g.DV : g.DB) + k * g.n;
    double sY = 0, sB = 0, sE = 0, sA = 0, sC = 0, sQ = 0, sS = 0, sYa = 0, sYd = 0, sAa = 0, sDd = 0, vd = 0, v0 = 0, vm = 0;
    double xh = X[last + j], xc = X[last - ld + j], yh = Y[last + j], yc = Y[last - ld + j];
    double ddh = X[last + j - 1] - X[last + j + 1], ss = X[last - ld + j - 1], ddc = ss - X[last - ld + j + 1];
#pragma unroll 4
    for (int t = e; t >= 1; --t) {
        const long long o = (long long)t * ld + j, ol = o - ld;
        const double mu = p.S[W_IB][o] * FB[o];
        const double xl = X[ol], sl = X[ol - 1], yl = Y[ol], ddl = sl - X[ol + 1], m = M[o];
        double x0, x1, x2;
        if constexpr (first_v) {
            x0 = D2[o - 1]; x1 = D2[o]; x2 = D2[o + 1];
        } else {
            x0 = Vn[o - 1] - U[o - 1]; x1 = Vn[o] - U[o]; x2 = Vn[o + 1] - U[o + 1];
            if constexpr (hv) { x0 -= D2[o - 1]; x1 -= D2[o]; x2 -= D2[o + 1]; }
        }
        const double mx = mu * q.hx[t], mc = sabr ? mu * q.hc[t] : mx;
        const double dy = yh - yl;
        sY = fma(mx, dy, sY);
        sB = fma(mu, yc, sB);
        sE = fma(mc, ddl - ddh, sE);
        double dx = 0.0;
        if constexpr (KIND == 1 || xt) {
            dx = KIND == 2 && mcs ? -xh - xl : xh - xl;
            sA = fma(mx, dx, sA);
            sC = fma(mu, xc, sC);
            sQ = fma(mu, ddc, sQ);
            sS = fma(mu, ss - xc, sS);
        }
        if (sabr) {
            const double ma = mu * q.ha[t], md = mu * q.hdd[t];
            sYa = fma(ma, yl + yh - 2.0 * yc, sYa);
            sYd = fma(md, dy, sYd);
            if constexpr (KIND == 1 || xt) {
                sAa = fma(ma, xl + (KIND == 2 && mcs ? -xh : xh) - 2.0 * xc, sAa);
                sDd = fma(md, dx, sDd);
            }
        }
        vd = fma(m, x2 - x0, vd);
        v0 = fma(m, x1, v0);
        vm = fma(m, x0 - x1, vm);
        xh = xc; xc = xl;
        yh = yc; yc = yl;
        ddh = ddc; ddc = ddl;
        ss = sl;
    }
    const double th = q.theta, wx = KIND == 1 ? 1.0 : hv ? q.zeta : q.zeta - q.theta, we = KIND == 1 ? 1.0 : q.zeta;
    const double A = th * sY + wx * sA, B = -(th * sB + 2.0 * wx * sC), Q = -wx * sQ, D = wx * (2.0 * sS - sQ);
    const double E = we * q.gamma * sE;
    const double es = q.es[j], bs = q.bs[j], hy = q.hy[j], tau = g.tau + g.dtau * (g.n0 + k);
    double g0 = q.delta * A + q.halfk * B;
    if (sabr)
        g0 += tau * q.omb * (q.hv2[j] * (2.0 * q.delta * (th * sYd + wx * sDd) - 2.0 * q.alphat * (th * sYa + wx * sAa)) -
                             q.rho * q.sigma * hy * E);
    const double nq = q.ni * (Q + th * vd);
    double *o = g.terms + (2LL * k + (KIND == 1 ? 1 : 0)) * 4 * g.lp + l;
    o[0] = g0 - q.halfk * th * v0;
    o[g.lp] = nq;
    o[2 * g.lp] = es * nq + q.betat * bs * (D + th * (2.0 * vm + vd)) + q.rho * hy * E;
    o[3 * g.lp] = E;
}

// Terms of the explicit v = v_lo column (da_b1), a thread per row and step.
static __global__ void __launch_bounds__(128) k_wadj_rows(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params q,
                                                          const __grid_constant__ line_sums g)
{
    const int nx = p.nx, ld = p.ld;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = static_cast<int>(id / g.rp), i = static_cast<int>(id % g.rp);
    if (k >= g.len) return;
    const double *U = g.U(k) + (long long)i * ld, *LV = g.LV + (long long)k * nx;
    double bb = 0.0, x = 0.0, ee = 0.0;
    if (i >= 1 && i <= nx - 2) {
        bb = p.imap[i] == i ? LV[i] : 0.0;
        if (i + 1 <= nx - 2 && p.imap[i + 1] == i) bb += LV[i + 1];
    }
    if (bb != 0.0) {
        const double u0 = U[0], tau = g.tau + g.dtau * (g.n0 + k);
        ee = q.ni * bb * (4.0 * U[1] - 3.0 * u0 - U[2]);
        double hd = q.hx[i];
        if (q.sabr) hd += 2.0 * q.omb * tau * q.hv2[0] * q.hdd[i];
        x = q.delta * hd * (U[ld] - U[-ld]) - q.k * u0;
    }
    double *o = g.rows + 3LL * k * g.rp + i;
    o[0] = bb;
    o[g.rp] = x;
    o[2 * g.rp] = ee;
}

// The terms added up over the steps, last step first, as the batch's group does: thread l0 has the lines 1 + l0,
// 1 + l0 + threads, ... of stage 2, those of stage 1, then the rows l0, l0 + threads, ...  A CTA per sum
// (r, kappa, theta, sigma, rho).  What bounds it: one chain of
// additions, and L2 latency.
template <bool DR> __global__ void __launch_bounds__(128) k_wadj_fold(const __grid_constant__ wparams<double> p, const __grid_constant__ adj_params q,
                                                                      const __grid_constant__ line_sums g, bool end, double *grads)
{
    __shared__ double red[4];
    const int what = blockIdx.x, l0 = threadIdx.x, ls = g.threads, lines = p.ny - 2, nx = p.nx;
    // what each line's term is: added, or times a factor of the line
    const int term = what == 0 ? 0 : what == 3 ? 2 : what == 4 ? 3 : 1;
    const double *col = what == 1 ? q.ek : what == 2 ? q.et : q.es;
    const double sh = q.sigma;
    double acc = g.acc[128 * what + l0];
    for (int k = g.len - 1; k >= 0; --k) {
        for (int st = DR ? 1 : 0; st < 2; ++st) {
            const double *t = g.terms + ((2LL * k + st) * 4 + term) * g.lp;
            for (int l = l0; l < lines; l += ls) {
                if (what == 0 || what == 3) acc += t[l];
                else acc = fma(what == 4 ? sh * q.hy[l + 1] : col[l + 1], t[l], acc);
            }
        }
        const double *b = g.rows + 3LL * k * g.rp;
        if (what < 4)
            for (int i = l0; i < nx; i += ls)
                if (b[i] != 0.0) acc = what == 0 ? fma(b[i], b[g.rp + i], acc) : fma(b[2 * g.rp + i], col[0], acc);
    }
    g.acc[128 * what + l0] = acc;
    if (!end) return;
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if (l0 % 32 == 0) red[l0 / 32] = acc;
    __syncthreads();
    if (l0 == 0) {
        double sum = 0.0;
        for (int w = 0; w < ls / 32; ++w) sum += red[w];
        grads[what == 0 ? 4 : what - 1] = sum;
    }
}

// adjoint seed: the bilinear weights of the value
static __global__ void k_wadj_seed(double *VB, int ld, bilinear b)
{
    const long long o = (long long)b.i0 * ld + b.j0;
    VB[o] = b.w00;
    VB[o + ld] = b.w10;
    VB[o + 1] = b.w01;
    VB[o + ld + 1] = b.w11;
}
// sums of the per-thread parameter sums (output order kappa, theta, sigma, rho, r) and the pitched
// adjoint of the initial condition in the caller's layout
static __global__ void __launch_bounds__(1024) k_wadj_reduce(const double *acc, long long nacc, double *grads)
{
    __shared__ double red[1024];
    const int out[5] = {4, 0, 1, 2, 3};
    double sum = 0.0;
    for (long long t = threadIdx.x; t < nacc; t += 1024) sum += acc[blockIdx.x * nacc + t];
    red[threadIdx.x] = sum;
    __syncthreads();
    for (int h = 512; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) grads[out[blockIdx.x]] = red[0];
}
static __global__ void k_wadj_unpitch(const double *src, double *dst, int nx, int ny, int ld)
{
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q < (long long)nx * ny) dst[q] = src[q / ny * ld + q % ny];
}

} // namespace wide
} // namespace lss_gb300
