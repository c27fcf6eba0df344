// adi_delta.cuh -- time step and adjoint step of one FP64 instance with a thread per line, in delta
// form: the stage functions of the batched persistent kernels and of the thread-per-line path.
//
// The stages are solved for their increments (adi_wide.cuh derives them):
//   D1 = S F(U);  DR: next = U + V(D1);  else D2 = V(D1) (rows 0 and nx-1: -U);
//   CS / MCS: D3 = S(D1 + zeta A0 D2 + (zeta - theta) G(D2)), next = U + V(D3);
//   HV: E = S(zeta F(D2) - D2), next = U + D2 + V(D1 + E)
// with S lines in row-scaled factors, y_t = f_t - la_t y_{t-1}, x_t = y_t - g_t x_{t+1}, and v lines
// unscaled, y_t = d_t - l_t y_{t-1}, xi_t = y_t - u_t xi_{t+1}, x_t = ib_t xi_t.  Per grid point and
// step 23 FP64 instructions for Craig-Sneyd (32 when written on Y1, Y2, Y3), ten S and three v
// tables (instead of 18 and five).  F is evaluated with differences along the S line,
//   F(U) = M (U_{t-1} - U_t) + P (U_{t+1} - U_t) + M~ U_{j-1} + P~ U_{j+1} + (M + P - Z - W) U_t + mixed,
// one subtraction more than with the weight -(Z + W): the terms of size k / h^2 U cancel exactly.  The
// rounding of F itself, against extended precision, is 10 to 300 times below that of the operator
// written out on grids of 100 x 50 to 2050 x 9 (the state is still rounded once a step, which bounds
// what a whole solve gains); the centre weight is formed from the row's reaction term, by center_weight.
//
// What bounds them: an FP64 instruction of a warp takes 64 cycles of its SM sub-partition, whether
// or not it depends on the one before, so a warp that has its operands in registers saturates its
// sub-partition alone.  A batch's time is that of its largest instances while the GPU is full: their
// operands come from HBM (about 1 us), which the rows in flight of one warp have to cover.  So a thread
// takes 255 registers (two CTAs per SM) and holds the next rows: five of the right-hand sides, 16 to
// 32 of the passes with one instruction per row.  1024 uneven calls (Craig-Sneyd, up to 256 x 128):
// 187 ms; with two and eight rows at 128 registers and four CTAs per SM 245 ms; sensitivities of 768
// calls 437 against 552 ms (GPU filled with equal 256 x 128 instances alone: 1.75e10 against 1.95e10
// point-steps/s).  L2 prefetch instructions instead cost more than they gave (257 ms: their issue
// slots add to the FP64 chain's).  The v sweeps walk the rows of the row-major state, a lane per row:
// they move four columns per access (256-bit loads and stores, rows padded to a multiple of four),
// 8 L1 wavefronts per column and array instead of 32.
#pragma once
// Included by adi_batched.cu inside namespace lss_gb300, after inst_view.

__device__ __forceinline__ void ld4(const double *p, double *o)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3]) : "l"(p));
}
__device__ __forceinline__ void st4(double *p, const double *o)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(o[0]), "d"(o[1]), "d"(o[2]), "d"(o[3]) : "memory");
}

enum { V_FIRST = 0, V_LAST = 1, V_LAST_HV = 2 };

constexpr int BK = deep::BK, VB4 = deep::VB4; // of the adjoint's passes

// The explicit v = v_lo column and the rows of S_lo and S_max (b1_stage, b2_stage) in the order of
// adi_wide.cuh: a single instance in relay order has the same bits.
__device__ __forceinline__ void db1_stage(const inst_view<double> &v, const bdesc &d, const double *U, double *sb0, int l0, int ls)
{
    const int nx = v.nx, ld = v.ld;
    for (int i = l0; i < nx; i += ls) {
        const double *u = U + i * ld;
        double r = fma(__ldg(v.X(XB_2) + i), u[2], fma(__ldg(v.X(XB_1) + i), u[1], __ldg(v.X(XB_C) + i) * u[0]));
        if (i == 0) r = __ldg(v.Yv(Y_SLO));
        else if (i == nx - 1) r += d.bnc;
        else r = fma(__ldg(v.X(XB_P) + i), u[ld], fma(__ldg(v.X(XB_M) + i), u[-ld], r));
        sb0[i] = r;
    }
}
__device__ __forceinline__ void db2_stage(const inst_view<double> &v, double *Vn, int l0, int ls)
{
    const int ny = v.ny, ld = v.ld, last = (v.nx - 1) * ld;
    for (int j = l0; j < ny; j += ls) {
        Vn[j] = __ldg(v.Yv(Y_SLO) + j);
        const int jj = __ldg(v.jmap() + j);
        Vn[last + j] = fma(4.0 / 3.0, Vn[last - ld + jj], fma(-1.0 / 3.0, Vn[last - 2 * ld + jj], -__ldg(v.Yv(Y_B2C) + j)));
    }
}

// One S stage.  KIND 1: A = U.  KIND 2: A = D2.  Y: the increment, rows 0 and nx-1 included.
template <int KIND, int SCH, typename DEPTH = deep>
__device__ __forceinline__ void ds_stage(const inst_view<double> &v, const bdesc &d, const double *U, const double *A, const double *D1,
                                         double *Y, int l0, int ls)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD;
    constexpr bool six = KIND == 1 || hv || mcs; // the six-point operator enters
    constexpr int AH = DEPTH::AH, BK = DEPTH::BK;
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = nx - 2, last = (nx - 1) * ld;
    const double zeta = d.a_zeta, zt = d.a_zeta - d.a_theta;
    struct row {
        double la, wg, ww, ws, wc, wn, we, ib, d1, am, ac, ap; // tables and D1 at row t, A at row t+1 (wc: MCS -(Z + W), else M + P - Z - W)
    };
    for (int j = 1 + l0; j <= ny - 2; j += ls) {
        const int jj = __ldg(v.jmap() + j);
        double lo, hi;
        if constexpr (KIND == 2 && hv) {
            lo = U[j];
            hi = U[last + j];
        } else {
            lo = U[jj] - U[j];
            hi = U[last + jj] - U[last + j];
        }
        auto load = [&](int t) -> row {
            const int o = t * ld + j;
            row r;
            r.la = __ldg(v.S(DS_LA, t, j));
            r.wg = __ldg(v.S(DS_WG, t, j));
            if constexpr (six) {
                r.ww = __ldg(v.S(DS_WW, t, j));
                r.ws = __ldg(v.S(DS_WS, t, j));
                r.wc = __ldg(v.S(KIND == 2 && mcs ? DS_WC : DS_WQ, t, j));
                r.wn = __ldg(v.S(DS_WN, t, j));
                r.we = __ldg(v.S(DS_WE, t, j));
            }
            if constexpr (KIND == 2) r.ib = __ldg(v.S(DS_IB, t, j));
            if constexpr (KIND == 2 && !hv) r.d1 = D1[o];
            r.am = A[o + ld - 1];
            r.ac = A[o + ld];
            r.ap = A[o + ld + 1];
            return r;
        };
        double a0c = A[j], a1c = A[ld + j], a1m = A[ld + j - 1], a1p = A[ld + j + 1];
        double q0 = A[j - 1] - A[j + 1], q1 = a1m - a1p;
        double dw = a0c - a1c; // difference to the row before
        double y = lo;
        auto point = [&](const row &r, int t) {
            const double q2 = r.am - r.ap, mix = q0 - q2;
            double f;
            if constexpr (KIND == 1 || hv) {
                f = r.wg * mix;
                f = fma(r.ww, dw, f);
                f = fma(r.ws, a1m, f);
                f = fma(r.wc, a1c, f);
                f = fma(r.wn, a1p, f);
                dw = a1c - r.ac;
                f = fma(r.we, -dw, f);
                if constexpr (KIND == 2) f = fma(zeta, f, -r.ib * a1c);
            } else {
                f = r.ib * r.d1;
                f = fma(zeta * r.wg, mix, f);
                if constexpr (mcs) {
                    double z = r.ww * a0c;
                    z = fma(r.ws, a1m, z);
                    z = fma(r.wc, a1c, z);
                    z = fma(r.wn, a1p, z);
                    z = fma(-r.we, r.ac, z);
                    f = fma(zt, z, f);
                }
            }
            y = fma(-r.la, y, f);
            Y[t * ld + j] = y;
            a0c = a1c; a1c = r.ac;
            a1m = r.am; a1p = r.ap;
            q0 = q1; q1 = q2;
        };
        row ring[AH];
#pragma unroll
        for (int k = 0; k < AH; ++k) ring[k] = load(min(1 + k, e));
        int t = 1;
        for (; t + AH - 1 <= e; t += AH)
#pragma unroll
            for (int k = 0; k < AH; ++k) {
                const row next = load(min(t + k + AH, e));
                point(ring[k], t + k);
                ring[k] = next;
            }
#pragma unroll
        for (int k = 0; k < AH - 1; ++k)
            if (t + k <= e) point(ring[k], t + k);
        // back substitution, blocks of BK rows loaded one block ahead
        double x = hi, yb[BK], gb[BK], yn[BK], gn[BK];
        auto block = [&](int t, double *yo, double *go) {
#pragma unroll
            for (int z = 0; z < BK; ++z) {
                const int r = max(t - z, 1);
                yo[z] = Y[r * ld + j];
                go[z] = __ldg(v.S(DS_G, r, j));
            }
        };
        block(e, yb, gb);
        for (t = e; t >= 1; t -= BK) {
            block(t - BK, yn, gn);
#pragma unroll
            for (int z = 0; z < BK; ++z) {
                if (t - z >= 1) {
                    x = fma(-gb[z], x, yb[z]);
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

// One v stage (KIND, see adi_wide.cuh): right-hand side D (+ E), boundary column sb0.
template <int KIND, typename DEPTH = deep>
__device__ __forceinline__ void dv_stage(const inst_view<double> &v, const double *U, const double *D, const double *E, const double *D2,
                                         const double *sb0, double *out, int l0, int ls)
{
    constexpr int BK = DEPTH::BK, VB4 = DEPTH::VB4;
    static_assert(BK % 4 == 0, "columns move four at a time");
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = ny - 2;
    for (int i = 1 + l0; i <= nx - 2; i += ls) {
        const int row = i * ld;
        const int ii = __ldg(v.imap() + i);
        const double lo = sb0[ii], hi = __ldg(v.X(X_VHI) + ii);
        const double d0 = KIND == V_LAST_HV ? 0.0 : lo - U[row], dn = KIND == V_LAST_HV ? 0.0 : hi - U[row + ny - 1];
        double db[BK], lb[BK], dx[BK], lx[BK];
        auto block = [&](int t, double *dd, double *ll) { // columns t .. t + BK - 1 (t a multiple of BK)
#pragma unroll
            for (int z = 0; z < BK; z += 4) {
                const int c = row + min(t + z, ld - 4);
                ld4(D + c, dd + z);
                if constexpr (KIND == V_LAST_HV) {
                    double ev[4];
                    ld4(E + c, ev);
#pragma unroll
                    for (int w = 0; w < 4; ++w) dd[z + w] += ev[w];
                }
            }
#pragma unroll
            for (int z = 0; z < BK; ++z) ll[z] = __ldg(v.Vt(DV_L, min(t + z, e), i));
        };
        double y = d0;
        block(0, db, lb);
        for (int t = 0; t <= e; t += BK) {
            block(t + BK, dx, lx);
#pragma unroll
            for (int z = 0; z < BK; ++z) {
                if (t + z >= 1 && t + z <= e) y = fma(-lb[z], y, db[z]);
                db[z] = y;
                if ((z & 3) == 3 && t + z - 3 < ld) st4(out + row + t + z - 3, db + z - 3);
            }
#pragma unroll
            for (int z = 0; z < BK; ++z) {
                db[z] = dx[z];
                lb[z] = lx[z];
            }
        }
        // back substitution and the stage's result, blocks of four columns
        double x = dn;
        struct blk {
            double y[4], u[4], ib[4], s[4];
        };
        auto back = [&](int t) -> blk {
            blk b;
            const int c = row + max(t, 0);
            ld4(out + c, b.y);
            if constexpr (KIND != V_FIRST) {
                ld4(U + c, b.s);
                if constexpr (KIND == V_LAST_HV) {
                    double w[4];
                    ld4(D2 + c, w);
#pragma unroll
                    for (int z = 0; z < 4; ++z) b.s[z] += w[z];
                }
            }
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                const int c = min(max(t, 0) + z, ny - 1);
                b.u[z] = __ldg(v.Vt(DV_U, c, i));
                b.ib[z] = __ldg(v.Vt(DV_IB, c, i));
            }
            return b;
        };
        const int tl = (ny - 1) / 4 * 4;
        blk ring[VB4];
#pragma unroll
        for (int k = 0; k < VB4; ++k) ring[k] = back(tl - 4 * k);
        for (int t0 = tl; t0 >= 0; t0 -= 4 * VB4)
#pragma unroll
            for (int k = 0; k < VB4; ++k) {
                const int t = t0 - 4 * k;
                if (t < 0) break;
                const blk nb = back(t - 4 * VB4), b = ring[k];
                double o[4];
#pragma unroll
                for (int z = 3; z >= 0; --z) {
                    const int c = t + z;
                    if (c >= 1 && c <= e) {
                        x = fma(-b.u[z], x, b.y[z]);
                        o[z] = KIND == V_FIRST ? b.ib[z] * x : fma(b.ib[z], x, b.s[z]);
                    } else {
                        o[z] = c == 0 ? (KIND == V_FIRST ? d0 : lo) : c == ny - 1 ? (KIND == V_FIRST ? dn : hi) : 0.0;
                    }
                }
                st4(out + row + t, o);
                ring[k] = nb;
            }
    }
}

// rows 0 and nx-1 of D2 (the reference reads Y2 as zero there)
__device__ __forceinline__ void d2_edges(const inst_view<double> &v, const double *U, double *D2, int l0, int ls)
{
    const int last = (v.nx - 1) * v.ld;
    for (int q = l0; q < v.ny; q += ls) {
        D2[q] = -U[q];
        D2[last + q] = -U[last + q];
    }
}

// ------------------------------------------------------------------------------------------
// adjoint (adi_wide.cuh: the state's adjoint VB is updated in place)
// ------------------------------------------------------------------------------------------
// b2^T: the extrapolated row's adjoint into rows nx-2 and nx-3
__device__ __forceinline__ void da_b2(const inst_view<double> &v, double *VB, int l0, int ls)
{
    const int ny = v.ny, ld = v.ld, last = (v.nx - 1) * ld;
    for (int q = l0; q < ny; q += ls) {
        double add = __ldg(v.jmap() + q) == q ? VB[last + q] : 0.0;
        if (q + 1 < ny && __ldg(v.jmap() + q + 1) == q) add += VB[last + q + 1];
        VB[last - ld + q] = fma(4.0 / 3.0, add, VB[last - ld + q]);
        VB[last - 2 * ld + q] = fma(-1.0 / 3.0, add, VB[last - 2 * ld + q]);
    }
}
// rows 0 and nx-1 of a step's output do not depend on its input
__device__ __forceinline__ void da_edges(const inst_view<double> &v, double *VB, int l0, int ls)
{
    const int last = (v.nx - 1) * v.ld;
    for (int q = l0; q < v.ny; q += ls) VB[q] = VB[last + q] = 0.0;
}

// Transposed v solve: XB the adjoint of the solve's result, DB receives that of its right-hand side.
template <int KIND>
__device__ __forceinline__ void da_v(const inst_view<double> &v, const double *XB, double *VB, double *DB, double *LV, bool add, int l0,
                                     int ls)
{
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = ny - 2;
    for (int i = 1 + l0; i <= nx - 2; i += ls) {
        const int row = i * ld;
        struct blk {
            double x[4], ib[4], u[4];
        };
        auto fwd = [&](int t) -> blk { // u of the column before
            blk b;
            ld4(XB + row + min(t, ld - 4), b.x);
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                b.ib[z] = __ldg(v.Vt(DV_IB, min(t + z, ny - 1), i));
                b.u[z] = __ldg(v.Vt(DV_U, min(max(t + z - 1, 0), ny - 1), i));
            }
            return b;
        };
        double z_ = 0.0, zn = 0.0, z0 = 0.0;
        blk ring[VB4];
#pragma unroll
        for (int k = 0; k < VB4; ++k) ring[k] = fwd(4 * k);
        for (int t0 = 0; t0 < ny; t0 += 4 * VB4)
#pragma unroll
            for (int k = 0; k < VB4; ++k) {
                const int t = t0 + 4 * k;
                if (t >= ny) break;
                const blk nb = fwd(t + 4 * VB4), b = ring[k];
                double o[4];
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const int c = t + z;
                    if (c >= 1 && c <= e) z_ = fma(-b.u[z], z_, b.ib[z] * b.x[z]);
                    if (c == 0) z0 = b.x[z];
                    if (c == ny - 1) zn = fma(-b.u[z], z_, b.x[z]);
                    o[z] = c <= e ? z_ : 0.0;
                }
                st4(DB + row + t, o);
                ring[k] = nb;
            }
        double w = 0.0, zb[BK], lb[BK], zx[BK], lx[BK];
        auto back = [&](int t, double *zz, double *ll) { // columns t .. t + BK - 1; l of the column after
#pragma unroll
            for (int z = 0; z < BK; z += 4) ld4(DB + row + min(max(t + z, 0), ld - 4), zz + z);
#pragma unroll
            for (int z = 0; z < BK; ++z) ll[z] = __ldg(v.Vt(DV_L, min(max(t + z + 1, 0), ny - 1), i));
        };
        const int tl = (ny - 1) / BK * BK;
        back(tl, zb, lb);
        for (int t = tl; t >= 0; t -= BK) {
            back(t - BK, zx, lx);
#pragma unroll
            for (int z = BK - 1; z >= 0; --z) {
                const int c = t + z;
                if (c >= 1 && c <= e) w = fma(-lb[z], w, zb[z]);
                zb[z] = w;
                if (c == 0) z0 = fma(-lb[z], w, z0);
                if ((z & 3) == 0 && c < ld) st4(DB + row + c, zb + z);
            }
#pragma unroll
            for (int z = 0; z < BK; ++z) {
                zb[z] = zx[z];
                lb[z] = lx[z];
            }
        }
        if constexpr (KIND != V_LAST_HV) {
            VB[row] -= z0;
            VB[row + ny - 1] -= zn;
            LV[i] = add ? LV[i] + z0 : z0;
        }
    }
}

// the five parameter sums of a thread (r, kappa, theta, sigma, rho)
struct adj_acc {
    double s[5];
};

// Transposed S solve with the parameter sums of the stage and of the v solve that it feeds or reads
// (adi_wide.cuh, k_wadj_s).  XB (+ DV): adjoint of the stage's increment; Y: the increment.
template <int KIND, int SCH>
__device__ __forceinline__ void da_s(const inst_view<double> &v, const bdesc &d, const double *U, const double *Vn, const double *D2,
                                     const double *Y, const double *XB, const double *DV, double *VB, double *FB, double *MU, double *LS,
                                     double *HS, adj_acc &acc, double tau, int l0, int ls)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD, dr = SCH == LSS_ADI_DOUGLAS_RACHFORD;
    constexpr bool xt = KIND == 2 && (hv || mcs);  // D2 terms besides the mixed one
    constexpr bool first_v = KIND == 1 && !dr;     // the v solve with result D2, right-hand-side adjoint DV
    const int nx = v.nx, ny = v.ny, ld = v.ld, e = nx - 2, last = (nx - 1) * ld;
    const bool sabr = d.model == LSS_ADI_SABR;
    const double *X = KIND == 1 ? U : D2;
    for (int j = 1 + l0; j <= ny - 2; j += ls) {
        // z_t = xbar_t - g_{t-1} z_{t-1} (the table's row 0 is zero)
        double z = 0.0, xb[BK], gb[BK], xn[BK], gn[BK];
        auto block = [&](int t, double *xo, double *go) {
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                const int r = min(t + k, e), o = r * ld + j;
                xo[k] = XB[o];
                if constexpr (first_v) xo[k] += DV[o];
                go[k] = __ldg(v.S(DS_G, r - 1, j));
            }
        };
        block(1, xb, gb);
        for (int t = 1; t <= e; t += BK) {
            block(t + BK, xn, gn);
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                if (t + k <= e) {
                    z = fma(-gb[k], z, xb[k]);
                    FB[(t + k) * ld + j] = z;
                }
                xb[k] = xn[k];
                gb[k] = gn[k];
            }
        }
        const double hib = -__ldg(v.S(DS_G, e, j)) * z;
        // w_t = z_t - la_{t+1} w_{t+1} with the sums, rows t+1, t, t-1 of X and Y in a window
        struct row {
            double z, la, ib, xc, ss, sn, y, m, x0, x1, x2; // z, la_{t+1}, ib, m, x of row t; X, Y of row t-1
        };
        auto load = [&](int t) -> row {
            const int o = t * ld + j, ol = o - ld;
            row r;
            r.z = FB[o];
            r.la = __ldg(v.S(DS_LA, t + 1, j)); // the table's row nx-1 is zero
            r.ib = __ldg(v.S(DS_IB, t, j));
            r.xc = X[ol];
            r.ss = X[ol - 1];
            r.sn = X[ol + 1];
            r.y = Y[ol];
            if constexpr (first_v) {
                r.m = DV[o];
                r.x0 = D2[o - 1]; r.x1 = D2[o]; r.x2 = D2[o + 1];
            } else {
                r.m = XB[o];
                r.x0 = Vn[o - 1] - U[o - 1]; r.x1 = Vn[o] - U[o]; r.x2 = Vn[o + 1] - U[o + 1];
                if constexpr (hv) { r.x0 -= D2[o - 1]; r.x1 -= D2[o]; r.x2 -= D2[o + 1]; }
            }
            return r;
        };
        double sY = 0, sB = 0, sE = 0, sA = 0, sC = 0, sQ = 0, sS = 0, sYa = 0, sYd = 0, sAa = 0, sDd = 0, vd = 0, v0 = 0, vm = 0;
        double xh = X[last + j], xc = X[last - ld + j], yh = Y[last + j], yc = Y[last - ld + j];
        double ddh = X[last + j - 1] - X[last + j + 1], ss = X[last - ld + j - 1], ddc = ss - X[last - ld + j + 1];
        double w = 0.0;
        row nr = load(e), nr2 = load(max(e - 1, 1));
        for (int t = e; t >= 1; --t) {
            const row r = nr;
            nr = nr2;
            nr2 = load(max(t - 2, 1));
            const int o = t * ld + j;
            w = fma(-r.la, w, r.z);
            const double mu = r.ib * w, ddl = r.ss - r.sn;
            FB[o] = w;
            if constexpr (KIND == 2 && !hv) MU[o] = mu; // adjoint of D1
            const double mx = mu * __ldg(v.X(X_HX) + t);
            const double mc = sabr ? mu * __ldg(v.X(X_HC) + t) : mx;
            const double dy = yh - r.y;
            sY = fma(mx, dy, sY);
            sB = fma(mu, yc, sB);
            sE = fma(mc, ddl - ddh, sE);
            double dx = 0.0;
            if constexpr (KIND == 1 || xt) {
                dx = KIND == 2 && mcs ? -xh - r.xc : xh - r.xc;
                sA = fma(mx, dx, sA);
                sC = fma(mu, xc, sC);
                sQ = fma(mu, ddc, sQ);
                sS = fma(mu, ss - xc, sS);
            }
            if (sabr) {
                const double ma = mu * __ldg(v.X(X_HA) + t), md = mu * __ldg(v.X(X_HDD) + t);
                sYa = fma(ma, r.y + yh - 2.0 * yc, sYa);
                sYd = fma(md, dy, sYd);
                if constexpr (KIND == 1 || xt) {
                    sAa = fma(ma, r.xc + (KIND == 2 && mcs ? -xh : xh) - 2.0 * xc, sAa);
                    sDd = fma(md, dx, sDd);
                }
            }
            vd = fma(r.m, r.x2 - r.x0, vd);
            v0 = fma(r.m, r.x1, v0);
            vm = fma(r.m, r.x0 - r.x1, vm);
            xh = xc; xc = r.xc;
            yh = yc; yc = r.y;
            ddh = ddc; ddc = ddl;
            ss = r.ss;
        }
        const double lob = -__ldg(v.S(DS_LA, 1, j)) * w;
        if constexpr (KIND == 2 && hv) { // E's boundary values are U's rows 0 and nx-1
            VB[j] += lob;
            VB[last + j] += hib;
        } else if constexpr (first_v && !hv) {
            LS[j] += lob;
            HS[j] += hib;
        } else {
            LS[j] = lob;
            HS[j] = hib;
        }
        // the line's sums: theta weighs the terms in Y, wx those in X
        const double th = d.a_theta, wx = KIND == 1 ? 1.0 : hv ? d.a_zeta : d.a_zeta - d.a_theta, we = KIND == 1 ? 1.0 : d.a_zeta;
        const double A = th * sY + wx * sA, B = -(th * sB + 2.0 * wx * sC), Q = -wx * sQ, D = wx * (2.0 * sS - sQ);
        const double E = we * d.a_gamma * sE;
        const double ek = __ldg(v.Yv(Y_EK) + j), et = __ldg(v.Yv(Y_ET) + j), es = __ldg(v.Yv(Y_ES) + j), bs = __ldg(v.Yv(Y_BS) + j);
        const double hy = __ldg(v.Yv(Y_HY) + j);
        double g0 = d.a_delta * A + d.a_halfk * B;
        if (sabr)
            g0 += tau * d.a_omb * (__ldg(v.Yv(Y_HV2) + j) * (2.0 * d.a_delta * (th * sYd + wx * sDd) - 2.0 * d.a_alphat * (th * sYa + wx * sAa)) -
                                   d.a_rho * d.a_sigma * hy * E);
        const double nq = d.a_ni * (Q + th * vd);
        acc.s[0] += g0 - d.a_halfk * th * v0;
        acc.s[1] += ek * nq;
        acc.s[2] += et * nq;
        acc.s[3] += es * nq + d.a_betat * bs * (D + th * (2.0 * vm + vd)) + d.a_rho * hy * E;
        acc.s[4] += d.a_sigma * hy * E;
    }
}

// Cross-line adjoints of an S stage, a thread per column walking down with a window of rows.  Row r
// contributes down (to r-1), up (to r+1) and mid (to r) terms from FB and the tables at columns
// q-1, q, q+1; FB and the tables are zero on the boundary rows and columns.  KIND 2: adjoint of D2
// (HV: on top of the state's; rows 0 and nx-1 are -U).  KIND 1: F^T and the S lines' boundary
// values into VB (the explicit boundary column follows in da_b1).
template <int KIND, int SCH>
__device__ __forceinline__ void da_gather(const inst_view<double> &v, const bdesc &d, const double *FB, const double *LS, const double *HS,
                                          double *VB, double *D2B, int l0, int ls)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, mcs = SCH == LSS_ADI_MODIFIED_CRAIG_SNEYD;
    constexpr bool six = KIND == 1 || hv || mcs;
    const int nx = v.nx, ny = v.ny, ld = v.ld;
    const double zeta = d.a_zeta, zt = d.a_zeta - d.a_theta;
    struct raw {
        double f0, fm, fp, gm, gp, wd, wu, wm, wr, wl, ib, vb;
    };
    for (int q = l0; q < ny; q += ls) {
        const bool lf = q >= 1, rt = q + 1 <= ny - 1;
        auto load = [&](int r) -> raw {
            const int t = min(max(r, 0), nx - 1), o = t * ld + q;
            raw a;
            a.f0 = FB[o];
            a.fm = lf ? FB[o - 1] : 0.0;
            a.fp = rt ? FB[o + 1] : 0.0;
            a.gm = lf ? __ldg(v.S(DS_WG, t, q - 1)) : 0.0;
            a.gp = rt ? __ldg(v.S(DS_WG, t, q + 1)) : 0.0;
            if constexpr (six) {
                a.wd = __ldg(v.S(DS_WW, t, q));
                a.wu = __ldg(v.S(DS_WE, t, q));
                a.wm = __ldg(v.S(DS_WC, t, q));
                a.wr = rt ? __ldg(v.S(DS_WS, t, q + 1)) : 0.0;
                a.wl = lf ? __ldg(v.S(DS_WN, t, q - 1)) : 0.0;
            }
            if constexpr (KIND == 2 && hv) a.ib = __ldg(v.S(DS_IB, t, q));
            if constexpr (KIND == 1 || hv) a.vb = VB[o];
            return a;
        };
        // down, up, mid of a row: mixed part g, five-point part
        struct part {
            double g, dn, up, mid, e;
        };
        auto parts = [&](const raw &a) -> part {
            part p;
            p.g = fma(a.gp, a.fp, -a.gm * a.fm);
            p.e = 0.0;
            if constexpr (mcs && KIND == 2) {
                p.dn = fma(zeta, p.g, zt * (a.wd * a.f0));
                p.up = -fma(zeta, p.g, zt * (a.wu * a.f0));
                p.mid = zt * fma(a.wr, a.fp, fma(a.wl, a.fm, a.wm * a.f0));
            } else if constexpr (six) {
                p.dn = fma(a.wd, a.f0, p.g);
                p.up = fma(a.wu, a.f0, -p.g);
                p.mid = fma(a.wr, a.fp, fma(a.wl, a.fm, a.wm * a.f0));
                if constexpr (KIND == 2) p.e = a.ib * a.f0;
            } else {
                p.dn = p.g;
                p.up = -p.g;
                p.mid = 0.0;
            }
            return p;
        };
        double lsum = 0.0, hsum = 0.0;
        if constexpr (KIND == 1) {
            if (q >= 1 && q <= ny - 2) {
                const bool own = __ldg(v.jmap() + q) == q;
                lsum = own ? 0.0 : -LS[q];
                hsum = own ? 0.0 : -HS[q];
            }
            if (q + 1 <= ny - 2 && __ldg(v.jmap() + q + 1) == q) {
                lsum += LS[q + 1];
                hsum += HS[q + 1];
            }
        }
        double up_m = 0.0;
        raw a0 = load(0), an = load(1), an2 = load(2);
        part pc = parts(a0);
        double vbc = a0.vb;
        for (int r = 0; r < nx; ++r) {
            const raw a = an;
            an = an2;
            an2 = load(r + 3);
            part pn;
            if (r + 1 < nx) pn = parts(a);
            else pn.g = pn.dn = pn.up = pn.mid = pn.e = 0.0;
            double x = pn.dn + up_m;
            if constexpr (six) x += pc.mid;
            const int o = r * ld + q;
            if constexpr (KIND == 2) {
                double db = x;
                if constexpr (hv) db = fma(zeta, x, -pc.e);
                else if constexpr (!mcs) db = zeta * x;
                if (r == 0 || r == nx - 1) VB[o] = (hv ? vbc : VB[o]) - db;
                else D2B[o] = hv ? vbc + db : db;
            } else {
                if (r == 0) x += lsum;
                if (r == nx - 1) x += hsum;
                VB[o] = vbc + x;
            }
            up_m = pc.up;
            pc = pn;
            vbc = a.vb;
        }
    }
}

// b1^T of columns 0..2: the explicit v = v_lo column, whose values are the lo ends of the v lines,
// with its parameter sensitivities, a thread per row.
__device__ __forceinline__ void da_b1(const inst_view<double> &v, const bdesc &d, const double *U, const double *LV, double *VB, adj_acc &acc,
                                      double tau, int l0, int ls)
{
    const int nx = v.nx, ld = v.ld;
    auto B0 = [&](int i) -> double {
        if (i < 1 || i > nx - 2) return 0.0;
        double sum = __ldg(v.imap() + i) == i ? LV[i] : 0.0;
        if (i + 1 <= nx - 2 && __ldg(v.imap() + i + 1) == i) sum += LV[i + 1];
        return sum;
    };
    for (int p = l0; p < nx; p += ls) {
        const int o = p * ld;
        const double bb = B0(p);
        const double below = p >= 1 ? __ldg(v.X(XB_P) + p - 1) : 0.0, above = p + 1 <= nx - 2 ? __ldg(v.X(XB_M) + p + 1) : 0.0;
        VB[o] += fma(below, B0(p - 1), fma(__ldg(v.X(XB_C) + p), bb, above * B0(p + 1)));
        VB[o + 1] = fma(__ldg(v.X(XB_1) + p), bb, VB[o + 1]);
        VB[o + 2] = fma(__ldg(v.X(XB_2) + p), bb, VB[o + 2]);
        if (bb != 0.0) {
            const double u0 = U[o], u1 = U[o + 1], u2 = U[o + 2];
            const double ee = d.a_ni * bb * (4.0 * u1 - 3.0 * u0 - u2);
            double hd = __ldg(v.X(X_HX) + p);
            if (d.model == LSS_ADI_SABR) hd += 2.0 * d.a_omb * tau * __ldg(v.Yv(Y_HV2)) * __ldg(v.X(X_HDD) + p);
            acc.s[0] += bb * (d.a_delta * hd * (U[o + ld] - U[o - ld]) - d.a_k * u0);
            acc.s[1] += ee * __ldg(v.Yv(Y_EK));
            acc.s[2] += ee * __ldg(v.Yv(Y_ET));
            acc.s[3] += ee * __ldg(v.Yv(Y_ES));
        }
    }
}

// One forward step U -> Vn by group g, stage increments in D1, D2, D3; ends with a group barrier.
template <int SCH, typename DEPTH = deep>
__device__ __forceinline__ void delta_step(const inst_view<double> &v, const bdesc &d, const double *U, double *D1, double *D2, double *D3,
                                           double *Vn, double *sb0, const grp &g)
{
    const int l0 = g.t, ls = g.n;
    db1_stage(v, d, U, sb0, l0, ls);
    ds_stage<1, SCH, DEPTH>(v, d, U, U, nullptr, D1, l0, ls);
    if constexpr (SCH != LSS_ADI_DOUGLAS_RACHFORD) d2_edges(v, U, D2, l0, ls);
    g.sync();
    if constexpr (SCH == LSS_ADI_DOUGLAS_RACHFORD) {
        dv_stage<V_LAST, DEPTH>(v, U, D1, nullptr, nullptr, sb0, Vn, l0, ls);
    } else {
        dv_stage<V_FIRST, DEPTH>(v, U, D1, nullptr, nullptr, sb0, D2, l0, ls);
        g.sync();
        ds_stage<2, SCH, DEPTH>(v, d, U, D2, D1, D3, l0, ls);
        g.sync();
        if constexpr (SCH == LSS_ADI_HUNDSDORFER_VERWER) dv_stage<V_LAST_HV, DEPTH>(v, U, D1, D3, D2, sb0, Vn, l0, ls);
        else dv_stage<V_LAST, DEPTH>(v, U, D3, nullptr, nullptr, sb0, Vn, l0, ls);
    }
    g.sync();
    db2_stage(v, Vn, l0, ls);
    g.sync();
}

// Adjoint of one time step by group g: VB in place from the step's output to its input.
template <int SCH>
__device__ __forceinline__ void delta_adjoint(const inst_view<double> &v, const bdesc &d, const double *U, const double *D1, const double *D2,
                                              const double *D3, const double *Vn, double *VB, double *DB, double *FB, double *MU, double *DV,
                                              double *D2B, double *LV, double *LS, double *HS, adj_acc &acc, double tau, const grp &g)
{
    constexpr bool hv = SCH == LSS_ADI_HUNDSDORFER_VERWER, dr = SCH == LSS_ADI_DOUGLAS_RACHFORD;
    const int l0 = g.t, ls = g.n;
    da_b2(v, VB, l0, ls);
    g.sync();
    da_edges(v, VB, l0, ls);
    da_v<hv ? V_LAST_HV : V_LAST>(v, VB, VB, DB, LV, false, l0, ls);
    g.sync();
    if constexpr (dr) {
        da_s<1, SCH>(v, d, U, Vn, D2, D1, DB, DV, VB, FB, MU, LS, HS, acc, tau, l0, ls);
    } else {
        da_s<2, SCH>(v, d, U, Vn, D2, D3, DB, DV, VB, FB, MU, LS, HS, acc, tau, l0, ls);
        g.sync();
        da_gather<2, SCH>(v, d, FB, LS, HS, VB, D2B, l0, ls);
        g.sync();
        da_v<V_FIRST>(v, D2B, VB, DV, LV, !hv, l0, ls);
        g.sync();
        da_s<1, SCH>(v, d, U, Vn, D2, D1, hv ? DB : MU, DV, VB, FB, MU, LS, HS, acc, tau, l0, ls);
    }
    g.sync();
    da_gather<1, SCH>(v, d, FB, LS, HS, VB, D2B, l0, ls);
    g.sync();
    da_b1(v, d, U, LV, VB, acc, tau, l0, ls);
    g.sync();
}
