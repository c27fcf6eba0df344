// adi_exact.cuh -- the reference's operation order with everything off the serial chain (device side).
//
// The line solves of one instance in the reference's arithmetic, y_t = (f_t - a_t y_{t-1}) / beta_t and
// x_t = y_t - gamma_t x_{t+1}, rounded operation by operation like lss_thomas_lu_solver.hpp:161-190.
// With tables that do not change with time beta and gamma are the same in every step: they are
// computed once, in the reference's order, with 1 / beta rounded to nearest beside them.  A CTA takes
// L lines: all its threads evaluate the right-hand sides of all rows into shared memory, one warp
// then runs the chains (one line per lane), all threads write the result.
//
// The division by a divisor known in advance is one multiplication and two fused multiply-adds,
//   q0 = RN(x r),  rem = RN(x - q0 beta),  q = RN(q0 + rem r),      r = RN(1 / beta)
// which is the correctly rounded quotient for all x and beta as long as nothing underflows or overflows
// (Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division when the divisor
// is known in advance", IEEE Trans. Computers 53(8), 2004).  The range of beta is checked when
// the tables are made, that of x on its exponent field; x outside (zeros, tiny and huge values, NaN)
// takes the division itself.
//
// What bounds it: the chain.  A dependent FP64 operation takes 64 cycles, five of them a row forward and
// two backward (39 us of a 100 x 50 Douglas-Rachford step at 1.9 GHz), and the chain warp has its FP64
// pipe to itself: every other operand comes from one 32-byte record per row or from shared memory,
// loaded ahead, and comparisons are integer ones.  Douglas-Rachford, 100 x 50: 297 us a step with a
// thread per line that did all of it (two divisions and a factorisation per row and sweep, four
// launches), 100 us with separate tables, a bounds test per row and a branch per division, 54 us so.
#pragma once

#include "adi_device.cuh"

namespace lss_gb300 {
namespace exact {

__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ bool in_range(double x) { return ((static_cast<unsigned>(__double2hiint(x)) >> 20 & 0x7ffu) - 123u) < 1800u; }
__device__ __forceinline__ bool in_range(float x) { return ((__float_as_uint(x) >> 23 & 0xffu) - 31u) < 192u; }
__device__ __forceinline__ bool divisor_ok(double b) { return ((static_cast<unsigned>(__double2hiint(b)) >> 20 & 0x7ffu) - 959u) < 128u; }
__device__ __forceinline__ bool divisor_ok(float b) { return ((__float_as_uint(b) >> 23 & 0xffu) - 103u) < 48u; }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

template <typename T> struct record {
    T a, b, r, g;
};
__device__ __forceinline__ record<double> load(const double *p)
{
    record<double> q;
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(q.a), "=d"(q.b), "=d"(q.r), "=d"(q.g) : "l"(p));
    return q;
}
__device__ __forceinline__ record<float> load(const float *p)
{
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    return {v.x, v.y, v.z, v.w};
}

// One row forward; ok: cleared if the quotient needs the division itself.
template <typename T> __device__ __forceinline__ T row_fast(const record<T> &q, T f, T y, bool &ok)
{
    using R = ar<true>;
    const T x = R::sub(f, R::mul(q.a, y));
    ok = ok && in_range(x);
    const T q0 = R::mul(x, q.r);
    return fma_rn(fma_rn(-q.b, q0, x), q.r, q0);
}
template <typename T> __device__ __forceinline__ T row_slow(const record<T> &q, T f, T y)
{
    using R = ar<true>;
    return R::div(R::sub(f, R::mul(q.a, y)), q.b);
}

// One line: right-hand sides f[0..e-1] (shared memory) become the solution; row k's record at rec + k * st.
// f[e-1] has the upper boundary's term already.  Four rows at a time: their operands are loaded while the
// four before run, and one branch repeats them with divisions where a numerator was out of range.
template <typename T> __device__ __forceinline__ void chain(T *f, const T *rec, int st, int e, T lo)
{
    using R = ar<true>;
    constexpr int W = 4;
    record<T> nq[W];
    T nf[W];
    const int head = e % W, blocks = e / W;
    T y = lo;
    const T *p = rec + static_cast<long long>(head) * st;
    auto ahead = [&](const T *at, const T *fa) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            nq[w] = load(at + static_cast<long long>(w) * st);
            nf[w] = fa[w];
        }
    };
    if (blocks > 0) ahead(p, f + head);
    for (int t = 0; t < head; ++t) {
        const record<T> q = load(rec + static_cast<long long>(t) * st);
        bool ok = true;
        T z = row_fast(q, f[t], y, ok);
        if (!ok) z = row_slow(q, f[t], y);
        y = z;
        f[t] = y;
    }
    T *fo = f + head;
    for (int k = 0; k < blocks; ++k) {
        record<T> q[W];
        T cf[W], z[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            q[w] = nq[w];
            cf[w] = nf[w];
        }
        const int step = k + 1 < blocks ? W : 0;
        p += static_cast<long long>(step) * st;
        ahead(p, fo + step);
        bool ok = true;
#pragma unroll
        for (int w = 0; w < W; ++w) z[w] = row_fast(q[w], cf[w], w ? z[w - 1] : y, ok);
        if (!ok) {
#pragma unroll 1
            for (int w = 0; w < 1; ++w) {
                z[0] = row_slow(q[0], cf[0], y);
                z[1] = row_slow(q[1], cf[1], z[0]);
                z[2] = row_slow(q[2], cf[2], z[1]);
                z[3] = row_slow(q[3], cf[3], z[2]);
            }
        }
#pragma unroll
        for (int w = 0; w < W; ++w) fo[w] = z[w];
        y = z[W - 1];
        fo += W;
    }
    // back: rows e-2 .. 0
    constexpr int B = 8;
    T ng[B], nv[B];
    T x = y;
    const int tail = (e - 1) % B, back = (e - 1) / B;
    const T *g = rec + 3 + static_cast<long long>(e - 2 - tail) * st;
    T *fb = f + e - 2 - tail;
    auto behind = [&](const T *at, const T *fa) {
#pragma unroll
        for (int w = 0; w < B; ++w) {
            ng[w] = __ldg(at - static_cast<long long>(w) * st);
            nv[w] = fa[-w];
        }
    };
    if (back > 0) behind(g, fb);
    for (int t = e - 2; t > e - 2 - tail; --t) {
        x = R::sub(f[t], R::mul(__ldg(rec + 3 + static_cast<long long>(t) * st), x));
        f[t] = x;
    }
    for (int k = 0; k < back; ++k) {
        T cg[B], cv[B];
#pragma unroll
        for (int w = 0; w < B; ++w) {
            cg[w] = ng[w];
            cv[w] = nv[w];
        }
        const int step = k + 1 < back ? B : 0;
        g -= static_cast<long long>(step) * st;
        behind(g, fb - step);
#pragma unroll
        for (int w = 0; w < B; ++w) {
            x = R::sub(cv[w], R::mul(cg[w], x));
            fb[-w] = x;
        }
        fb -= B;
    }
}

// S stage: lines j = 1..ny-2, L per CTA; with bcol0 the grid has one more CTA, which evaluates the boundary
// columns of the v lines from the state.
template <typename T, int STAGE>
__global__ void k_exact_s(const __grid_constant__ dev_instance<T> d, const T *rec, int L, const T *Ub, const T *A,
                          const T *B, const T *Cc, T *Y, T *bcol0, T *bcolN)
{
    using R = ar<true>;
    extern __shared__ __align__(16) unsigned char raw[];
    T *f = reinterpret_cast<T *>(raw);
    const int nx = d.nx, ny = d.ny, e = nx - 2, pitch = e | 1;
    pdl_launch();
    if (bcol0 && blockIdx.x == gridDim.x - 1) {
        pdl_wait();
        for (int i = threadIdx.x; i < nx; i += blockDim.x) boundary1_row<T, true>(d, Ub, i, bcol0, bcolN, 1);
        return;
    }
    const int j0 = 1 + static_cast<int>(blockIdx.x) * L, lines = min(L, ny - 1 - j0);
    const int ln = threadIdx.x, jl = min(j0 + ln, ny - 2), jj = d.jmap[jl];
    pdl_wait();
    const T top = Ub[jj], bot = Ub[(nx - 1) * ny + jj]; // (threads below `lines`: their line's ends)
    for (int k = threadIdx.x; k < e * L; k += blockDim.x) {
        const int l = k % L, t = 1 + k / L, j = j0 + l;
        if (l >= lines) continue;
        const int o = t * ny + j;
        const T a = R::mul(-d.theta, d.M[o]);
        const T tz = R::mul(d.theta, d.Z[o]);
        const T tp = R::mul(d.theta, d.P[o]);
        T v;
        if constexpr (STAGE == S_STAGE4_HV) // A = Y2, B = Y1; rhs_intermed_3 is wanted at this point only
            v = R::add(R::sub(R::add(R::mul(a, A[o - ny]), R::mul(tz, A[o])), R::mul(tp, A[o + ny])), hv3_value<T, true>(d, Ub, B, A, o));
        else
            v = s_rhs<T, true, STAGE>(d, t, j, A, B, Cc, a, tz, tp);
        if (t == e && e > 1) v = R::sub(v, R::mul(-tp, Ub[(nx - 1) * ny + d.jmap[j]]));
        f[l * pitch + t - 1] = v;
    }
    __syncthreads();
    if (ln < lines) {
        const long long o = ny + j0 + ln;
        chain(f + ln * pitch, rec + 4 * o, 4 * ny, e, top);
        Y[j0 + ln] = top;
        Y[(nx - 1) * ny + j0 + ln] = bot;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < e * L; k += blockDim.x) {
        const int l = k % L, t = 1 + k / L;
        if (l < lines) Y[t * ny + j0 + l] = f[l * pitch + t - 1];
    }
}

// v stage: lines i = nx-2 .. 1 in descending order, L (at least 2) per CTA.  `last`: the result is the
// next state, whose rows 0 and nx-1 the first CTA (it has rows nx-2 and nx-3) writes.
template <typename T>
__global__ void k_exact_v(const __grid_constant__ dev_instance<T> d, const T *rec, int L, const T *in, const T *inh,
                          const T *bcol0, const T *bcolN, T *out, int last)
{
    using R = ar<true>;
    extern __shared__ __align__(16) unsigned char raw[];
    T *f = reinterpret_cast<T *>(raw);
    const int nx = d.nx, ny = d.ny, e = ny - 2, pitch = e | 1;
    const int i0 = nx - 2 - static_cast<int>(blockIdx.x) * L, lines = min(L, i0), ln = threadIdx.x; // line l: row i0 - l
    pdl_launch();
    const int ii = d.imap[max(i0 - min(ln, lines - 1), 1)];
    pdl_wait();
    const T lo = bcol0[ii], hi = bcolN[ii];
    for (int k = threadIdx.x; k < e * lines; k += blockDim.x) {
        const int l = k / e, t = 1 + k % e, i = i0 - l;
        const int o = i * ny + t;
        const T a = R::mul(-d.theta, d.Mt[o]);
        const T tw = R::mul(d.theta, d.W[o]);
        const T tp = R::mul(d.theta, d.Pt[o]);
        T v = R::add(R::sub(R::add(R::mul(a, in[o - 1]), R::mul(tw, in[o])), R::mul(tp, in[o + 1])), inh[o]);
        if (t == e && e > 1) v = R::sub(v, R::mul(-tp, bcolN[d.imap[i]]));
        f[l * pitch + t - 1] = v;
    }
    __syncthreads();
    if (ln < lines) {
        const long long o = static_cast<long long>(i0 - ln) * ny + 1;
        chain(f + ln * pitch, rec + 4 * o, 4, e, lo);
        out[o - 1] = lo;
        out[o + e] = hi;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < e * lines; k += blockDim.x) {
        const int l = k / e, t = 1 + k % e;
        out[(i0 - l) * ny + t] = f[l * pitch + t - 1];
    }
    if (last && blockIdx.x == 0) {
        __syncthreads();
        for (int j = threadIdx.x; j < ny; j += blockDim.x) boundary2_column<T, true>(d, out, j);
    }
}

// Records -theta M, beta, 1 / beta, gamma of one line, in the order of k_s_sweep and k_v_sweep.  S lines: low = M, diag =
// Z, up = P, st = ny; v lines: Mt, W, Pt, st = 1.
template <typename T>
__global__ void k_exact_setup(const T *low, const T *diag, const T *up, T theta, int lines, long long first, long long next, long long st,
                              int e, T *rec, int *bad)
{
    using R = ar<true>;
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= lines) return;
    T gam = T(0);
    int out = 0;
    long long o = first + l * next;
    T nl = low[o], nd = diag[o], nu = up[o]; // the next row's coefficients, loaded before this row's division
    for (int t = 1; t <= e; ++t, o += st) {
        const T av = R::mul(-theta, nl);
        const T bv = R::add(T(1), R::mul(theta, nd));
        const T cv = -R::mul(theta, nu);
        if (t < e) {
            nl = low[o + st];
            nd = diag[o + st];
            nu = up[o + st];
        }
        const T beta = t == 1 ? bv : R::sub(bv, R::mul(av, gam));
        const T r = R::div(T(1), beta);
        const bool ok = divisor_ok(beta);
        if (ok && in_range(cv)) {
            const T q0 = R::mul(cv, r);
            gam = fma_rn(fma_rn(-beta, q0, cv), r, q0);
        } else {
            gam = R::div(cv, beta);
        }
        out |= !ok;
        rec[4 * o] = av;
        rec[4 * o + 1] = beta;
        rec[4 * o + 2] = r;
        rec[4 * o + 3] = gam;
    }
    if (out) atomicOr(bad, 1);
}

} // namespace exact
} // namespace lss_gb300
