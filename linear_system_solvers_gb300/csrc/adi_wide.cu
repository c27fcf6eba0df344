// adi_wide.cu -- one instance in the factorised ("fast") arithmetic over the whole GPU: host side of
// the partitioned line solves (adi_wide.cuh).  Per time step two kernels (Douglas-Rachford) or
// four (the other schemes); the boundary column of the step is evaluated by the v stages, the
// extrapolated boundary row by the last one.  Launched with programmatic stream serialisation,
// directly or as a captured graph.
#include <algorithm>
#include <cmath>
#include <memory>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "adi_batched.hpp"
#include "adi_threads.hpp"
#include "adi_wide.cuh"

namespace lss_gb300 {
namespace wide {

template <typename T> struct line_solver {
    int nx = 0, ny = 0, ld = 0, steps = 0, scheme = 0, sms = 0;
    long long n = 0;
    dbuf<T> state, stab, vtab, xy, carry_mem, pay, surf;
    dbuf<int> maps, status;
    dbuf<double> value;
    bilinear bil{};
    wparams<T> wp{};
    bool serial = false; // recurrences in relay order (FP64)
    T *U = nullptr, *Vn = nullptr, *D1 = nullptr, *D2 = nullptr, *D3 = nullptr;
    long long launches = 0;
    // time-dependent coefficients (FP64)
    bool tdep = false;
    dbuf<double> td_mem;
    tdep_tab td{};
    std::vector<double> td_da, td_dc;
    dbuf<double> td_sets;
    tdep_set td_set{};
    int td_group = 1, td_have = -1; // steps per set-up launch; the group whose tables are held
    bool td_adjoint = false;
    cudaGraphExec_t graph = nullptr;

    ~line_solver()
    {
        if (graph) cudaGraphExecDestroy(graph);
    }

    int init(const lss_adi_problem &p, const instance_tables<T> &tt)
    {
        nx = tt.nx;
        ny = tt.ny;
        ld = (ny + 3) / 4 * 4;
        steps = tt.steps;
        scheme = tt.scheme;
        // zeta == theta: the modified scheme's extra term has weight 0 (bit-identical in the reference)
        if (scheme == LSS_ADI_MODIFIED_CRAIG_SNEYD && tt.sc.zeta == tt.sc.theta) scheme = LSS_ADI_CRAIG_SNEYD;
        n = static_cast<long long>(nx) * ld;
        int dev = 0;
        LSS_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
        LSS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
        const size_t flat = static_cast<size_t>(nx) * ny;
        LSS_CUDA_TRY(state.alloc(5 * n), "wide: allocating state");
        LSS_CUDA_TRY(cudaMemset(state.p, 0, state.n * sizeof(T)), "wide: clearing state");
        U = state.p; Vn = U + n; D1 = U + 2 * n; D2 = U + 3 * n; D3 = U + 4 * n;
        const bool td_case = time_dependent(p); // (S-line tables in sets: set_chunks)
        if (!td_case) LSS_CUDA_TRY(stab.alloc(W_COUNT * n), "wide: allocating S-line tables");
        LSS_CUDA_TRY(vtab.alloc(3 * n), "wide: allocating v-line tables");
        if (!td_case) LSS_CUDA_TRY(cudaMemset(stab.p, 0, stab.n * sizeof(T)), "wide: clearing S-line tables");
        LSS_CUDA_TRY(cudaMemset(vtab.p, 0, vtab.n * sizeof(T)), "wide: clearing v-line tables");
        LSS_CUDA_TRY(pay.alloc(flat), "wide: allocating the initial condition");
        LSS_CUDA_TRY(surf.alloc(flat), "wide: allocating the surface");
        LSS_CUDA_TRY(status.alloc(1), "wide: allocating status");
        LSS_CUDA_TRY(value.alloc(1), "wide: allocating value");
        // boundary arrays
        const double dl = tt.sc.delta, ni = tt.sc.ni, rk = tt.sc.rho, h1 = tt.sc.h1;
        std::vector<T> h(6 * static_cast<size_t>(nx) + 2 * static_cast<size_t>(ny));
        for (int i = 0; i < nx; ++i) {
            const double D = tt.coef_v0[i], E = tt.coef_v0[nx + i], F = tt.coef_v0[2 * nx + i];
            h[i] = static_cast<T>(-dl * D);
            h[nx + i] = static_cast<T>(1.0 - 3.0 * ni * E + rk * F);
            h[2 * nx + i] = static_cast<T>(dl * D);
            h[3 * nx + i] = static_cast<T>(-ni * E);
            h[4 * nx + i] = static_cast<T>(4.0 * ni * E);
            h[5 * nx + i] = tt.v_hi[i];
        }
        for (int j = 0; j < ny; ++j) {
            h[6 * nx + j] = tt.s_lo[j];
            h[6 * nx + ny + j] = static_cast<T>(2.0 * h1 * static_cast<double>(tt.s_hi_neu[j]) / 3.0);
        }
        LSS_CUDA_TRY(xy.alloc(h.size()), "wide: allocating boundary arrays");
        LSS_CUDA_TRY(xy.upload(h.data(), h.size()), "wide: uploading boundary arrays");
        std::vector<int> mp(tt.imap);
        mp.insert(mp.end(), tt.jmap.begin(), tt.jmap.end());
        LSS_CUDA_TRY(maps.alloc(mp.size()), "wide: allocating remaps");
        LSS_CUDA_TRY(maps.upload(mp.data(), mp.size()), "wide: uploading remaps");
        bil = make_bilinear(tt.x.data(), nx, tt.y.data(), ny, p.eval_s, p.eval_v);
        // coefficient tables, pitched, in double
        const double th = tt.sc.theta, gm = tt.sc.gamma;
        dbuf<double> base;
        LSS_CUDA_TRY(base.alloc(7 * n), "wide: allocating coefficient tables");
        {
            std::vector<double> hb(7 * static_cast<size_t>(n), 0.0);
            const unsigned nthr = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
            auto fill = [&](unsigned w, unsigned of) {
                for (int k = 0; k < 7; ++k)
                    for (int i = static_cast<int>(w); i < nx; i += static_cast<int>(of)) {
                        const T *src = tt.coef.data() + k * flat + static_cast<size_t>(i) * ny;
                        double *dst = hb.data() + k * static_cast<size_t>(n) + static_cast<size_t>(i) * ld;
                        for (int j = 0; j < ny; ++j) dst[j] = static_cast<double>(src[j]);
                    }
            };
            const unsigned shares = flat < 100000 ? 1 : nthr;
            run_shares(shares, [&](unsigned w) { fill(w, shares); });
            LSS_CUDA_TRY(base.upload(hb.data(), hb.size()), "wide: uploading coefficient tables");
        }
        if (!td_case) k_wide_setup_s<T><<<grid_for(ny - 2, 32), 32>>>(base.p, n, nx, ny, ld, th, gm, stab.p);
        k_wide_setup_v<T><<<grid_for(nx - 2, 32), 32>>>(base.p, n, nx, ny, ld, th, vtab.p);
        LSS_CUDA_TRY(cudaGetLastError(), "wide: launching the set-up");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "wide: set-up");
        wp.nx = nx; wp.ny = ny; wp.ld = ld;
        wp.zeta = static_cast<T>(tt.sc.zeta);
        wp.zt = static_cast<T>(static_cast<double>(tt.sc.zeta) - static_cast<double>(tt.sc.theta));
        wp.bnc = static_cast<T>(-dl * (2.0 * h1 * static_cast<double>(tt.s_hi_neu[0])) * static_cast<double>(tt.coef_v0[nx - 1]));
        for (int k = 0; k < W_COUNT && !td_case; ++k) wp.S[k] = stab.p + k * n;
        for (int k = 0; k < 3; ++k) wp.V[k] = vtab.p + k * n;
        const T *x = xy.p;
        wp.xbm = x; wp.xbc = x + nx; wp.xbp = x + 2 * nx; wp.xb2 = x + 3 * nx; wp.xb1 = x + 4 * nx; wp.xvhi = x + 5 * nx;
        wp.yslo = x + 6 * nx; wp.yb2c = wp.yslo + ny;
        wp.imap = maps.p; wp.jmap = maps.p + nx;
        if (td_case) {
            int rc = init_tdep(tt);
            if (rc) return rc;
        }
        return set_chunks(0, 0);
    }

    int init_tdep(const instance_tables<T> &tt)
    {
        if constexpr (!std::is_same<T, double>::value) {
            (void)tt;
            return set_error(LSS_ADI_EUNSUPPORTED, "wide: time-dependent coefficients are FP64 only");
        } else {
            std::vector<double> h(6 * static_cast<size_t>(n) + 3 * static_cast<size_t>(nx), 0.0);
            double *ma = h.data(), *pa = ma + n, *cs = pa + n, *mt = cs + n, *pt = mt + n, *w = pt + n, *mb = w + n, *am = mb + nx, *bm = am + nx;
            const size_t flat = static_cast<size_t>(nx) * ny;
            const double alpha = tt.sc.alpha, delta = tt.sc.delta;
            for (int i = 0; i < nx; ++i) {
                const double aval = tt.per_i[i], aa = tt.per_i[nx + i], aaa = tt.per_i[2 * nx + i], gc = tt.per_i[3 * nx + i],
                             ud = tt.per_i[4 * nx + i];
                mb[i] = -delta * (ud / aval);
                for (int j = 0; j < ny; ++j) {
                    const size_t o = static_cast<size_t>(i) * ny + j, q = static_cast<size_t>(i) * ld + j;
                    const double as = tt.a_static[o];
                    ma[q] = alpha * (as / aa) + delta * ((as * gc) / aaa);
                    pa[q] = alpha * (as / aa) - delta * ((as * gc) / aaa);
                    cs[q] = tt.c_static[o] / tt.ab[o];
                    mt[q] = tt.coef[3 * flat + o];
                    pt[q] = tt.coef[4 * flat + o];
                    w[q] = tt.coef[5 * flat + o];
                    if (j == 0) {
                        am[i] = -delta * ((as * gc) / aaa);
                        bm[i] = delta * (ud / aval);
                    }
                }
            }
            LSS_CUDA_TRY(td_mem.alloc(h.size()), "wide: allocating time-dependent tables");
            LSS_CUDA_TRY(td_mem.upload(h.data(), h.size()), "wide: uploading time-dependent tables");
            LSS_CUDA_TRY(cudaDeviceSynchronize(), "wide: time-dependent tables");
            td.ma = td_mem.p; td.pa = td.ma + n; td.cs = td.pa + n; td.mt = td.cs + n; td.pt = td.mt + n; td.w = td.pt + n;
            td.mb = td.w + n; td.am = td.mb + nx; td.bm = td.am + nx;
            td.z0 = -tt.half_rho_f;
            td.th = tt.sc.theta;
            td.gm = tt.sc.gamma;
            td.nx = nx; td.ny = ny; td.ld = ld; td.n = n;
            td_da = tt.step_da;
            td_dc = tt.step_dc;
            tdep = true;
            wp.tdep = 1;
            return LSS_ADI_OK;
        }
    }

    // chunk products of both sweeps of both directions
    long long carry_need() const
    {
        return 2 * (carry_table(wp.s, wp.ls) + carry_table(wp.v, wp.lv));
    }
    template <typename Q> static void carve(carry_tab<Q> &c, const split &sp, int stride, Q *&q)
    {
        const long long chunks = static_cast<long long>(sp.tiles) * sp.PC * stride;
        c.A = q; q += chunks;
        c.PreG = q; q += chunks;
        c.GA = q; q += static_cast<long long>(sp.tiles) * sp.groups() * stride;
    }
    // Partition: `ps`, `pv` chunks per S / v line (0: chosen by choose_split).  The products and the cleared
    // table sets are on the device when it returns: no stream of the caller is ordered behind the set-up's.
    int set_chunks(int ps, int pv)
    {
        wp.s = choose_split(nx - 2, ny - 2, false, ps, sms, sizeof(T));
        wp.v = choose_split(ny, nx - 2, true, pv, sms, sizeof(T));
        wp.ls = ld;
        wp.lv = nx;
        const long long need = carry_need();
        if (static_cast<long long>(carry_mem.n) < need) LSS_CUDA_TRY(carry_mem.alloc(need), "wide: allocating chunk products");
        T *q = carry_mem.p;
        for (carry_tab<T> *c : {&wp.sf, &wp.sb}) carve(*c, wp.s, wp.ls, q);
        for (carry_tab<T> *c : {&wp.vf, &wp.vb}) carve(*c, wp.v, wp.lv, q);
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        if (tdep) {
            const int rc = set_groups();
            if (rc) return rc;
        } else {
            products(nullptr, true);
        }
        products(nullptr, false);
        LSS_CUDA_TRY(cudaGetLastError(), "wide: chunk products");
        LSS_CUDA_TRY(cudaStreamSynchronize(nullptr), "wide: chunk products");
        return LSS_ADI_OK;
    }

    // one launch with programmatic stream serialisation
    template <typename... P, typename... A>
    void launch(cudaStream_t s, void (*k)(P...), dim3 grid, dim3 block, size_t smem, A &&...args)
    {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k, P(std::forward<A>(args))...);
        ++launches;
    }

    // products of the sweep `out` of a direction's factors fac, rows first..last (k_wide_products)
    void product(cudaStream_t s, bool s_lines, const T *fac, int first, int last, int shift, bool fwd, const carry_tab<T> &out)
    {
        const split &sp = s_lines ? wp.s : wp.v;
        const int lines = s_lines ? ny : nx, grid = grid_for(lines, sp.L) * sp.tiles;
        const long long ts = s_lines ? ld : 1, st = s_lines ? 1 : ld;
        launch(s, k_wide_products<T>, grid, dim3(sp.L * sp.PC), sizeof(T) * sp.L * sp.PC, fac, ts, st, lines, first, last,
               s_lines ? 1 : 0, shift, sp, fwd, out, s_lines ? wp.ls : wp.lv);
    }
    void products(cudaStream_t s, bool s_lines)
    {
        if (s_lines) {
            product(s, true, wp.S[W_LA], 1, nx - 2, 0, true, wp.sf);
            product(s, true, wp.S[W_G], 1, nx - 2, 0, false, wp.sb);
        } else {
            product(s, false, wp.V[W_VL], 0, ny - 1, 0, true, wp.vf);
            product(s, false, wp.V[W_VU], 0, ny - 1, 0, false, wp.vb);
        }
    }

    // Sets of S-line tables of a time-dependent instance: as many steps to a launch as keep its grid at
    // four CTAs per SM, while the sets stay within 56 MB of L2 (SABR 512 x 256 forward and adjoint: 11.70 ms with
    // four steps of 12.3 MB, 11.97 with five, 12.50 with three).
    int set_groups()
    {
        const long long words = (W_COUNT * n + 2 * nx + (td_adjoint ? 4 : 2) * carry_table(wp.s, wp.ls) + 3) / 4 * 4;
        const long long fit = (56LL << 20) / (words * static_cast<long long>(sizeof(double))), ctas = grid_for(ny - 2, wp.s.L);
        const long long fill = (4LL * sms + ctas - 1) / ctas;
        td_group = static_cast<int>(std::max(1LL, std::min({fit, fill, static_cast<long long>(TDEP_STEPS), static_cast<long long>(steps)})));
        LSS_CUDA_TRY(td_sets.alloc(td_group * words), "wide: allocating time-dependent tables");
        LSS_CUDA_TRY(cudaMemset(td_sets.p, 0, td_sets.n * sizeof(double)), "wide: clearing time-dependent tables");
        td_set = tdep_set{};
        td_set.S = td_sets.p;
        td_set.xb = td_sets.p + W_COUNT * n;
        td_set.stride = words;
        double *q = td_set.xb + 2 * nx;
        carve(td_set.sf, wp.s, wp.ls, q);
        carve(td_set.sb, wp.s, wp.ls, q);
        if (td_adjoint) {
            carve(td_set.sz, wp.s, wp.ls, q);
            carve(td_set.sw, wp.s, wp.ls, q);
        }
        return LSS_ADI_OK;
    }
    static carry_tab<double> shifted(const carry_tab<double> &c, long long o) { return {c.A + o, c.PreG + o, c.GA + o}; }

    // Points wp (and an adjoint's sz, sw) at the S-line tables of time step `step`, made for its group
    // of steps when they are not at hand.
    void refresh(cudaStream_t s, int step, adj_params *ap = nullptr)
    {
        if constexpr (std::is_same<T, double>::value) {
            const int group = step / td_group, first = group * td_group;
            if (group != td_have) {
                tdep_steps st{};
                const int len = std::min(td_group, steps - first);
                for (int k = 0; k < len; ++k) {
                    st.da[k] = td_da[first + k];
                    st.dc[k] = td_dc[first + k];
                }
                const split &sp = wp.s;
                const size_t smem = sizeof(double) * sp.L * (4 * sp.PC + std::max(4 * sp.groups(), sp.PC));
                const dim3 grid(grid_for(ny - 2, sp.L), len), block(sp.L * sp.PC);
                if (sp.R == 5) launch(s, k_wide_tdep<5>, grid, block, smem, td, st, td_set, sp, wp.ls);
                else if (sp.R == 8) launch(s, k_wide_tdep<8>, grid, block, smem, td, st, td_set, sp, wp.ls);
                else launch(s, k_wide_tdep<16>, grid, block, smem, td, st, td_set, sp, wp.ls);
                td_have = group;
            }
            const long long o = (step - first) * td_set.stride;
            for (int k = 0; k < W_COUNT; ++k) wp.S[k] = td_set.S + o + k * n;
            wp.xbm = td_set.xb + o;
            wp.xbp = wp.xbm + nx;
            wp.sf = shifted(td_set.sf, o);
            wp.sb = shifted(td_set.sb, o);
            if (ap) {
                ap->sz = shifted(td_set.sz, o);
                ap->sw = shifted(td_set.sw, o);
            }
        }
    }

    // f(R, SER) with the rows per chunk of a split and the order of the recurrences as constants
    template <bool S_LINES, typename F> void shaped(F &&f)
    {
        const int R = S_LINES ? wp.s.R : wp.v.R;
        auto with = [&](auto ser) {
            if (R == 8) f(std::integral_constant<int, 8>{}, ser);
            else if (R == 16) f(std::integral_constant<int, 16>{}, ser);
            else f(std::integral_constant<int, S_LINES ? 5 : 4>{}, ser);
        };
        if constexpr (std::is_same<T, double>::value) {
            if (serial) return with(std::true_type{});
        }
        with(std::false_type{});
    }
    template <int KIND, int SCH> void s_stage(cudaStream_t s, const T *u, const T *a, const T *d1, T *y)
    {
        const split &sp = wp.s;
        shaped<true>([&](auto r, auto ser) {
            launch(s, k_wide_s<T, decltype(r)::value, KIND, SCH, decltype(ser)::value>, grid_for(ny - 1, sp.L), dim3(sp.L * sp.PC),
                   2 * sizeof(T) * carry_words(sp), wp, u, a, d1, y);
        });
    }
    template <int KIND> void v_stage(cudaStream_t s, const T *u, const T *d, const T *e, const T *d2, T *out)
    {
        const split &sp = wp.v;
        shaped<false>([&](auto r, auto ser) {
            launch(s, k_wide_v<T, decltype(r)::value, KIND, decltype(ser)::value>, grid_for(nx - 2, sp.L), dim3(sp.L * sp.PC),
                   2 * sizeof(T) * carry_words(sp), wp, u, d, e, d2, out);
        });
    }
    // one time step u -> next, stage increments in d1, d2, d3
    void step(cudaStream_t s, const T *u, T *d1, T *d2, T *d3, T *next)
    {
        s_stage<1, LSS_ADI_DOUGLAS_RACHFORD>(s, u, u, nullptr, d1);
        if (scheme == LSS_ADI_DOUGLAS_RACHFORD) {
            v_stage<V_LAST>(s, u, d1, nullptr, nullptr, next);
            return;
        }
        v_stage<V_FIRST>(s, u, d1, nullptr, nullptr, d2);
        if (scheme == LSS_ADI_HUNDSDORFER_VERWER) {
            s_stage<2, LSS_ADI_HUNDSDORFER_VERWER>(s, u, d2, d1, d3);
            v_stage<V_LAST_HV>(s, u, d1, d3, d2, next);
        } else {
            if (scheme == LSS_ADI_MODIFIED_CRAIG_SNEYD) s_stage<2, LSS_ADI_MODIFIED_CRAIG_SNEYD>(s, u, d2, d1, d3);
            else s_stage<2, LSS_ADI_CRAIG_SNEYD>(s, u, d2, d1, d3);
            v_stage<V_LAST>(s, u, d3, nullptr, nullptr, next);
        }
    }

    // the same at time step m (time-dependent tables rebuilt first)
    void forward_step(cudaStream_t s, int m, const T *u, T *d1, T *d2, T *d3, T *next)
    {
        if (tdep) refresh(s, m);
        step(s, u, d1, d2, d3, next);
    }

    int enqueue(cudaStream_t s)
    {
        launches = 0;
        td_have = -1;
        const long long flat = static_cast<long long>(nx) * ny;
        k_wide_begin<T><<<grid_for(flat, 256), 256, 0, s>>>(pay.p, U, nx, ny, ld, status.p);
        const T *u = U;
        for (int m = 0; m < steps; ++m) {
            T *next = u == U ? Vn : U;
            forward_step(s, m, u, D1, D2, D3, next);
            u = next;
        }
        k_wide_end<T><<<grid_for(flat, 256), 256, 0, s>>>(u, nx, ny, ld, bil, surf.p, value.p, status.p);
        launches += 2;
        LSS_CUDA_TRY(cudaGetLastError(), "wide: launching the time loop");
        return LSS_ADI_OK;
    }

    int run(cudaStream_t s, bool use_graph)
    {
        if (!use_graph) return enqueue(s);
        if (!graph) {
            cudaStream_t cs;
            LSS_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "wide: capture stream");
            LSS_CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "wide: begin capture");
            const int rc = enqueue(cs);
            cudaGraph_t g = nullptr;
            cudaError_t e = cudaStreamEndCapture(cs, &g);
            cudaStreamDestroy(cs);
            if (rc) return rc;
            LSS_CUDA_TRY(e, "wide: end capture");
            e = cudaGraphInstantiate(&graph, g, 0);
            cudaGraphDestroy(g);
            LSS_CUDA_TRY(e, "wide: instantiate graph");
        }
        LSS_CUDA_TRY(cudaGraphLaunch(graph, s), "wide: graph launch");
        return LSS_ADI_OK;
    }
};

template <typename T> struct line_front : wide_solver_base {
    line_solver<T> w;
    std::vector<T> x, y, pay0;
    int ask_s = 0, ask_v = 0;
    bool asked = false;

    int init(const lss_adi_problem &p)
    {
        instance_tables<T> tt;
        build_tables_for<T>(p, tt);
        int rc = w.init(p, tt);
        if (p.options & LSS_ADI_OPT_LINE_PER_THREAD) w.serial = 1;
        x = std::move(tt.x);
        y = std::move(tt.y);
        pay0 = std::move(tt.payoff);
        return rc;
    }
    int forward(const void *payoff, void *out_surface, double *out_value, int flags, void *stream, bool use_graph) override
    {
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const bool dev = (flags & LSS_ADI_DEVICE_POINTERS) != 0;
        const size_t bytes = w.pay.n * sizeof(T);
        const void *src = payoff ? payoff : static_cast<const void *>(pay0.data());
        LSS_CUDA_TRY(cudaMemcpyAsync(w.pay.p, src, bytes, (payoff && dev) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s),
                     "wide: copying the terminal condition");
        int rc = w.run(s, use_graph);
        if (rc) return rc;
        if (out_value)
            LSS_CUDA_TRY(cudaMemcpyAsync(out_value, w.value.p, sizeof(double), cudaMemcpyDeviceToHost, s), "wide: value");
        if (out_surface)
            LSS_CUDA_TRY(cudaMemcpyAsync(out_surface, w.surf.p, bytes, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s),
                         "wide: surface");
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
        if (s_chunks < 0 || v_chunks < 0) return set_error(LSS_ADI_EINVAL, "lss_adi_line_chunks: negative chunk count");
        auto ok = [](int P, int e) { return P <= MAX_CHUNKS && (P <= 1 || e >= 4 * P); };
        if (!ok(s_chunks, w.nx - 2) || !ok(v_chunks, w.ny - 2)) return set_error(LSS_ADI_EINVAL, "wide: chunk count out of range");
        LSS_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "lss_adi_line_chunks");
        w.serial = 0; // chunk counts ask for partitioned solves
        int rc = w.set_chunks(s_chunks, v_chunks);
        if (rc) return rc;
        ask_s = s_chunks;
        ask_v = v_chunks;
        asked = true;
        if (out_s) *out_s = w.wp.s.PC;
        if (out_v) *out_v = w.wp.v.PC;
        return LSS_ADI_OK;
    }
    bool asked_chunks(int &s_chunks, int &v_chunks) const override
    {
        s_chunks = ask_s;
        v_chunks = ask_v;
        return asked;
    }
};

// Forward + adjoint of one FP64 instance: forward pass keeping a checkpoint every c steps (and the
// stage increments of the last segment), then per segment (last first) a recomputation that keeps
// every step's increments (not for the last one) and the adjoint steps in reverse order.
struct line_adjoint : wide_adjoint_base {
    line_solver<double> w;
    dbuf<double> ws, factors, carry_adj, grads;
    adj_params ap{};
    long long nacc = 0;
    int planned = 0; // interval of checkpoint_every = 0, kept while its workspace is held

    int init(const lss_adi_problem &p)
    {
        instance_tables<double> tt;
        build_tables<double>(p, tt);
        w.td_adjoint = true;
        int rc = w.init(p, tt);
        if (rc) return rc;
        LSS_CUDA_TRY(cudaMemcpy(w.pay.p, tt.payoff.data(), tt.payoff.size() * sizeof(double), cudaMemcpyHostToDevice),
                     "wide adjoint: initial condition");
        LSS_CUDA_TRY(grads.alloc(5), "wide adjoint: allocating gradients");
        const int nx = w.nx, ny = w.ny;
        sinh_map<double> g;
        g.init(p);
        std::vector<double> h(4 * static_cast<size_t>(nx) + 6 * static_cast<size_t>(ny));
        for (int i = 0; i < nx; ++i) {
            const s_factors d = derivative_s(p, g, tt.sc.h1 * i);
            h[i] = d.hx; h[nx + i] = d.hc; h[2 * nx + i] = d.ha; h[3 * nx + i] = d.hdd;
        }
        double *y = h.data() + 4 * nx;
        for (int j = 0; j < ny; ++j) {
            const v_factors d = derivative_v(p, g, tt.sc.h2 * j);
            y[j] = d.hy; y[ny + j] = d.bs; y[2 * ny + j] = d.ek; y[3 * ny + j] = d.et; y[4 * ny + j] = d.es; y[5 * ny + j] = d.hv2;
        }
        LSS_CUDA_TRY(factors.alloc(h.size()), "wide adjoint: allocating coefficient derivatives");
        LSS_CUDA_TRY(factors.upload(h.data(), h.size()), "wide adjoint: uploading coefficient derivatives");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "wide adjoint: coefficient derivatives");
        const double *x = factors.p, *yv = x + 4 * nx;
        ap.hx = x; ap.hc = x + nx; ap.ha = x + 2 * nx; ap.hdd = x + 3 * nx;
        ap.hy = yv; ap.bs = yv + ny; ap.ek = yv + 2 * ny; ap.et = yv + 3 * ny; ap.es = yv + 4 * ny; ap.hv2 = yv + 5 * ny;
        ap.delta = tt.sc.delta; ap.halfk = 0.5 * tt.sc.k; ap.ni = tt.sc.ni; ap.betat = tt.sc.beta; ap.sigma = p.sigma; ap.rho = p.rho;
        ap.theta = tt.sc.theta; ap.zeta = tt.sc.zeta; ap.gamma = tt.sc.gamma; ap.k = tt.sc.k; ap.alphat = tt.sc.alpha;
        ap.omb = 1.0 - p.sabr_beta;
        ap.dw = w.scheme == LSS_ADI_MODIFIED_CRAIG_SNEYD ? tt.sc.zeta - tt.sc.theta : w.scheme == LSS_ADI_HUNDSDORFER_VERWER ? tt.sc.zeta : 0.0;
        ap.sabr = p.model == LSS_ADI_SABR;
        tau0 = p.forward ? p.maturity - ap.k : ap.k;
        dtau = p.forward ? -ap.k : ap.k;
        // Up to 256 x 160 points the recurrences run in relay order: value and gradients have the bits of
        // the same instance in a batch (gradients: see line_sums).  (One warp group of the batched kernel took 119 ms for a 128 x 64 x 200
        // Craig-Sneyd call with sensitivities.)  Larger ones, and those of LSS_ADI_OPT_WIDE_ADJOINT, are
        // partitioned; LINE_PER_THREAD asks for relay order at any size.
        small = p.nx <= 256 && static_cast<long long>(p.nx) * p.ny <= 40960 && !time_dependent(p) && !(p.options & LSS_ADI_OPT_WIDE_ADJOINT);
        w.serial = small || (p.options & LSS_ADI_OPT_LINE_PER_THREAD);
        return partition(0, 0);
    }
    double tau0 = 0.0, dtau = 0.0;
    bool small = false; // relay order whatever chunk counts the forward solve was given

    // Counts set for the forward solve ask for partitioned solves here too, of instances that are not small.
    int set_chunks(int ps, int pv, void *stream) override
    {
        LSS_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "lss_adi_adjoint: chunk counts");
        w.serial = small;
        return partition(small ? 0 : ps, small ? 0 : pv);
    }
    // Partition of both passes.  Counts of 0 give the adjoint the lines per CTA of choose_split as well (handing
    // it the forward's counts as set ones gave tiled lines 4 instead of 8 lines per S stage).
    int partition(int ps, int pv)
    {
        int rc = w.set_chunks(ps, pv);
        if (rc) return rc;
        const long long need = w.carry_need();
        if (static_cast<long long>(carry_adj.n) < need) LSS_CUDA_TRY(carry_adj.alloc(need), "wide adjoint: allocating chunk products");
        double *q = carry_adj.p;
        for (carry_tab<double> *c : {&ap.sz, &ap.sw}) w.carve(*c, w.wp.s, w.wp.ls, q);
        for (carry_tab<double> *c : {&ap.vz, &ap.vw}) w.carve(*c, w.wp.v, w.wp.lv, q);
        if (!w.tdep) s_products(nullptr);
        w.product(nullptr, false, w.wp.V[W_VU], 1, w.ny - 1, -1, true, ap.vz);
        w.product(nullptr, false, w.wp.V[W_VL], 0, w.ny - 2, 1, false, ap.vw);
        LSS_CUDA_TRY(cudaGetLastError(), "wide adjoint: chunk products");
        LSS_CUDA_TRY(cudaDeviceSynchronize(), "wide adjoint: chunk products");
        return LSS_ADI_OK;
    }
    void s_products(cudaStream_t s)
    {
        w.product(s, true, w.wp.S[W_G], 1, w.nx - 2, -1, true, ap.sz);
        w.product(s, true, w.wp.S[W_LA], 1, w.nx - 2, 1, false, ap.sw);
    }

    template <int KIND> void adj_v(cudaStream_t s, const double *XB, double *VB, double *DB, double *LV, int add)
    {
        const split &sp = w.wp.v;
        w.shaped<false>([&](auto r, auto ser) {
            w.launch(s, k_wadj_v<decltype(r)::value, KIND, decltype(ser)::value>, grid_for(w.nx - 2, sp.L), dim3(sp.L * sp.PC),
                     2 * sizeof(double) * carry_words(sp), w.wp, ap, XB, VB, DB, LV, add);
        });
    }
    struct arrays {
        double *VB, *DB, *FB[2], *MU, *DV, *D2B, *LV, *LS, *HS, *ACC; // FB: first and second S stage
    };
    template <int KIND, int SCH>
    void adj_s(cudaStream_t s, const arrays &a, const double *U, const double *Vn, const double *D1, const double *D2, const double *Y,
               const double *XB, double tau, double da, double dc)
    {
        const split &sp = w.wp.s;
        w.shaped<true>([&](auto r, auto ser) {
            w.launch(s, k_wadj_s<decltype(r)::value, KIND, SCH, decltype(ser)::value>, grid_for(w.ny - 1, sp.L), dim3(sp.L * sp.PC),
                     2 * sizeof(double) * carry_words(sp), w.wp, ap, U, Vn, D1, D2, Y, XB, a.DV, a.VB, a.FB[KIND - 1], a.MU, a.LS, a.HS,
                     a.ACC, nacc, tau, da, dc);
        });
    }
    template <int KIND, int SCH> void gather(cudaStream_t s, const arrays &a, const double *U, double tau, double da)
    {
        const int grid = grid_for(static_cast<long long>(w.nx) * w.ny, 256);
        w.launch(s, k_wadj_gather<KIND, SCH>, grid, dim3(256), 0, w.wp, ap, U, a.FB[KIND - 1], a.D2B, a.VB, a.LS, a.HS, a.LV, a.ACC, nacc, tau, da);
    }
    template <int SCH>
    void adjoint_step(cudaStream_t s, const arrays &a, int m, const double *U, const double *D1, const double *D2, const double *D3,
                      const double *Vn)
    {
        double da = 1.0, dc = 1.0;
        if (w.tdep) {
            w.refresh(s, m, &ap);
            da = w.td_da[m];
            dc = w.td_dc[m];
        }
        const double tau = tau0 + dtau * m;
        if constexpr (SCH == LSS_ADI_DOUGLAS_RACHFORD) {
            adj_v<V_LAST>(s, a.VB, a.VB, a.DB, a.LV, 0);
            adj_s<1, SCH>(s, a, U, Vn, D1, D2, D1, a.DB, tau, da, dc);
        } else {
            if constexpr (SCH == LSS_ADI_HUNDSDORFER_VERWER) adj_v<V_LAST_HV>(s, a.VB, a.VB, a.DB, a.LV, 0);
            else adj_v<V_LAST>(s, a.VB, a.VB, a.DB, a.LV, 0);
            adj_s<2, SCH>(s, a, U, Vn, D1, D2, D3, a.DB, tau, da, dc);
            gather<2, SCH>(s, a, U, tau, da);
            adj_v<V_FIRST>(s, a.D2B, a.VB, a.DV, a.LV, SCH != LSS_ADI_HUNDSDORFER_VERWER);
            adj_s<1, SCH>(s, a, U, Vn, D1, D2, D1, SCH == LSS_ADI_HUNDSDORFER_VERWER ? a.DB : a.MU, tau, da, dc);
        }
        gather<1, SCH>(s, a, U, tau, da);
    }

    // Relay order: the parameter sums are made from the arrays of a run of steps of a segment (k_wadj_lines).
    bool by_lines() const { return w.serial && !w.tdep; }
    // Steps of a run: 256 MB of arrays, at least 32 steps (128 x 64 x 200 24.4 ms with runs of 32, 23.4 with one).
    int run_of(int c) const { return static_cast<int>(std::min<long long>(c, std::max(32LL, (1LL << 23) / w.n))); }
    static int padded(int k) { return (k + 31) / 32 * 32; }
    // Workspace (doubles) at checkpoint interval c
    long long need(int c) const
    {
        const long long nseg = (w.steps + c - 1) / c;
        const long long base = (nseg + 4LL * (c + 1) + 2) * w.n + 2LL * w.ny;
        if (by_lines()) return base + (3 + 4LL * run_of(c)) * w.n + run_of(c) * (w.nx + 8LL * padded(w.ny - 2) + 3LL * padded(w.nx)) + 5 * 128;
        return base + 6 * w.n + w.nx + 5 * nacc;
    }
    template <int SCH> void sum_lines(cudaStream_t s, const line_sums &g, bool end)
    {
        const int lines = grid_for(static_cast<long long>(g.len) * g.lp, 128);
        constexpr bool dr = SCH == LSS_ADI_DOUGLAS_RACHFORD;
        if constexpr (!dr) k_wadj_lines<2, SCH><<<lines, 128, 0, s>>>(w.wp, ap, g);
        k_wadj_lines<1, SCH><<<lines, 128, 0, s>>>(w.wp, ap, g);
        k_wadj_rows<<<grid_for(static_cast<long long>(g.len) * g.rp, 128), 128, 0, s>>>(w.wp, ap, g);
        k_wadj_fold<dr><<<5, g.threads, 0, s>>>(w.wp, ap, g, end, grads.p);
    }

    // Checkpoint interval and workspace of a run.  every = 0: the longest interval within a sixteenth of the
    // device and half of what is free (no step is recomputed when one segment holds the whole time
    // loop), at least ceil(sqrt(steps)).  It is chosen once and kept: what other users of the device hold
    // does not make a call allocate again.  Where its workspace cannot be had after all, the shortest is taken.
    int reserve(int every, int &c)
    {
        const int steps = w.steps, least = std::max(1, static_cast<int>(std::ceil(std::sqrt(static_cast<double>(steps)))));
        const bool keep = every <= 0 && planned > 0 && static_cast<long long>(ws.n) == need(planned);
        c = every > 0 ? std::min(every, steps) : keep ? planned : least;
        if (every <= 0 && !keep) {
            size_t free_b = 0, total_b = 0;
            LSS_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b), "wide adjoint: device memory");
            const double held_b = static_cast<double>(ws.n) * sizeof(double);
            const double most = std::min(static_cast<double>(total_b) / 16, 0.5 * (static_cast<double>(free_b) + held_b));
            for (int k = steps; k > c; --k)
                if (static_cast<double>(need(k)) * sizeof(double) <= most) {
                    c = k;
                    break;
                }
        }
        cudaError_t e = static_cast<long long>(ws.n) == need(c) ? cudaSuccess : ws.alloc(need(c));
        if (e == cudaErrorMemoryAllocation && every <= 0 && c > least) {
            (void)cudaGetLastError();
            c = least;
            e = ws.alloc(need(c));
        }
        LSS_CUDA_TRY(e, "wide adjoint: allocating workspace");
        if (every <= 0) planned = c;
        return LSS_ADI_OK;
    }

    int run(const void *payoff, double *out_value, double *dv_dparams, void *dv_dpayoff, int checkpoint_every, int flags,
            void *stream) override
    {
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const bool dev = (flags & LSS_ADI_DEVICE_POINTERS) != 0;
        const long long n = w.n;
        const int steps = w.steps;
        const size_t bytes = w.pay.n * sizeof(double);
        if (payoff)
            LSS_CUDA_TRY(cudaMemcpyAsync(w.pay.p, payoff, bytes, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s),
                         "lss_adi_adjoint: copying the terminal condition");
        nacc = std::max<long long>(static_cast<long long>(grid_for(w.ny - 1, w.wp.s.L)) * w.wp.s.L * w.wp.s.PC, w.nx);
        int c = 0;
        int rc = reserve(checkpoint_every, c);
        if (rc) return rc;
        const int nseg = (steps + c - 1) / c;
        double *CK = ws.p, *SEG = CK + nseg * n, *W0 = SEG + 4LL * (c + 1) * n, *W1 = W0 + n;
        const bool lines = by_lines();
        const int each = lines ? run_of(c) : 1; // steps whose adjoint arrays are kept
        line_sums ls{};
        arrays a;
        a.MU = W1 + n; a.D2B = a.MU + n;
        double *DB = a.D2B + n, *DV = DB + each * n;
        ls.terms = DV + each * n;
        ls.lp = lines ? padded(w.ny - 2) : 0;
        ls.rp = lines ? padded(w.nx) : 0;
        ls.rows = ls.terms + 8LL * ls.lp * each;
        a.VB = ls.rows + 3LL * ls.rp * each;
        double *FB = a.VB + n, *LV = FB + (lines ? 2 * each : 1) * n;
        a.LS = LV + static_cast<long long>(each) * w.nx; a.HS = a.LS + w.ny; a.ACC = a.HS + w.ny;
        ls.FB = FB; ls.DB = DB; ls.DV = DV; ls.LV = LV; ls.acc = a.ACC; ls.n = n; ls.tau = tau0; ls.dtau = dtau;
        ls.threads = 32 * std::max(1, std::min(4, (w.ny - 2 + 31) / 32)); // of the batch's warp groups
        if (lines) a.ACC = nullptr;
        auto arrays_of = [&](int k) { // of step k of a segment
            const long long at = k % each;
            a.DB = DB + at * n; a.DV = DV + at * n; a.LV = LV + at * w.nx;
            a.FB[1] = FB + (lines ? 2 * at : 0) * n;
            a.FB[0] = lines ? a.FB[1] + n : FB;
        };
        // read where no kernel writes: VB and FB (boundary rows and columns) and the sums.  The states and
        // increments are written wherever they are read, so the checkpoints need no clearing.
        LSS_CUDA_TRY(cudaMemsetAsync(a.VB, 0, (need(c) - (a.VB - ws.p)) * sizeof(double), s), "wide adjoint: clearing");
        auto slot = [&](int m, int k) { return SEG + (4LL * m + k) * n; };
        const long long flat = static_cast<long long>(w.nx) * w.ny;
        w.launches = 0;
        w.td_have = -1;
        k_wide_begin<double><<<grid_for(flat, 256), 256, 0, s>>>(w.pay.p, CK, w.nx, w.ny, w.ld, w.status.p);
        const double *cur = CK;
        const int n0_last = (nseg - 1) * c;
        for (int m = 0; m < steps; ++m) {
            if (m >= n0_last) {
                const int k = m - n0_last;
                w.forward_step(s, m, cur, slot(k, 1), slot(k, 2), slot(k, 3), slot(k + 1, 0));
                cur = slot(k + 1, 0);
            } else {
                double *next = (m + 1) % c == 0 ? CK + (m + 1) / c * n : (m & 1) ? W1 : W0;
                w.forward_step(s, m, cur, slot(0, 1), slot(0, 2), slot(0, 3), next);
                cur = next;
            }
        }
        k_wide_end<double><<<grid_for(flat, 256), 256, 0, s>>>(cur, w.nx, w.ny, w.ld, w.bil, w.surf.p, w.value.p, w.status.p);
        k_wadj_seed<<<1, 1, 0, s>>>(a.VB, w.ld, w.bil);
        for (int g = nseg - 1; g >= 0; --g) {
            const int n0 = g * c, len = std::min(c, steps - n0);
            const double *u0 = CK + g * n;
            for (int k = 0; k < len && g < nseg - 1; ++k)
                w.forward_step(s, n0 + k, k == 0 ? u0 : slot(k, 0), slot(k, 1), slot(k, 2), slot(k, 3), slot(k + 1, 0));
            for (int k = len - 1; k >= 0; --k) {
                arrays_of(k);
                const double *U = k == 0 ? u0 : slot(k, 0), *D1 = slot(k, 1), *D2 = slot(k, 2), *D3 = slot(k, 3), *Vn = slot(k + 1, 0);
                switch (w.scheme) {
                case LSS_ADI_DOUGLAS_RACHFORD: adjoint_step<LSS_ADI_DOUGLAS_RACHFORD>(s, a, n0 + k, U, D1, D2, D3, Vn); break;
                case LSS_ADI_CRAIG_SNEYD: adjoint_step<LSS_ADI_CRAIG_SNEYD>(s, a, n0 + k, U, D1, D2, D3, Vn); break;
                case LSS_ADI_MODIFIED_CRAIG_SNEYD: adjoint_step<LSS_ADI_MODIFIED_CRAIG_SNEYD>(s, a, n0 + k, U, D1, D2, D3, Vn); break;
                default: adjoint_step<LSS_ADI_HUNDSDORFER_VERWER>(s, a, n0 + k, U, D1, D2, D3, Vn); break;
                }
                if (!lines || k % each != 0) continue;
                ls.u0 = U; ls.seg = slot(k, 0); ls.len = std::min(each, len - k); ls.n0 = n0 + k;
                const bool end = ls.n0 == 0;
                switch (w.scheme) {
                case LSS_ADI_DOUGLAS_RACHFORD: sum_lines<LSS_ADI_DOUGLAS_RACHFORD>(s, ls, end); break;
                case LSS_ADI_CRAIG_SNEYD: sum_lines<LSS_ADI_CRAIG_SNEYD>(s, ls, end); break;
                case LSS_ADI_MODIFIED_CRAIG_SNEYD: sum_lines<LSS_ADI_MODIFIED_CRAIG_SNEYD>(s, ls, end); break;
                default: sum_lines<LSS_ADI_HUNDSDORFER_VERWER>(s, ls, end); break;
                }
            }
        }
        if (!lines) k_wadj_reduce<<<5, 1024, 0, s>>>(a.ACC, nacc, grads.p);
        LSS_CUDA_TRY(cudaGetLastError(), "wide adjoint: launching");
        if (out_value)
            LSS_CUDA_TRY(cudaMemcpyAsync(out_value, w.value.p, sizeof(double), cudaMemcpyDeviceToHost, s), "lss_adi_adjoint: value");
        if (dv_dparams)
            LSS_CUDA_TRY(cudaMemcpyAsync(dv_dparams, grads.p, 5 * sizeof(double), cudaMemcpyDeviceToHost, s), "lss_adi_adjoint: gradients");
        if (dv_dpayoff) {
            k_wadj_unpitch<<<grid_for(flat, 256), 256, 0, s>>>(a.VB, w.surf.p, w.nx, w.ny, w.ld);
            LSS_CUDA_TRY(cudaGetLastError(), "wide adjoint: payoff gradient");
            LSS_CUDA_TRY(cudaMemcpyAsync(dv_dpayoff, w.surf.p, bytes, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s),
                         "lss_adi_adjoint: payoff gradient");
        }
        LSS_CUDA_TRY(cudaStreamSynchronize(s), "lss_adi_adjoint: run");
        return LSS_ADI_OK;
    }
};

template <typename T> static int make_line(const lss_adi_problem &p, std::unique_ptr<wide_solver_base> &out)
{
    std::unique_ptr<line_front<T>> w(new line_front<T>());
    int rc = w->init(p);
    if (rc) return rc;
    out = std::move(w);
    return LSS_ADI_OK;
}

} // namespace wide

int make_partitioned_solver(const lss_adi_problem &p, std::unique_ptr<wide_solver_base> &out)
{
    try {
        return p.precision == LSS_ADI_FP64 ? wide::make_line<double>(p, out) : wide::make_line<float>(p, out);
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "wide: host allocation failed");
    }
}

int make_wide_adjoint(const lss_adi_problem &p, std::unique_ptr<wide_adjoint_base> &out)
{
    try {
        std::unique_ptr<wide::line_adjoint> a(new wide::line_adjoint());
        int rc = a->init(p);
        if (rc) return rc;
        out = std::move(a);
    } catch (const std::bad_alloc &) {
        return set_error(LSS_ADI_ENOMEM, "wide adjoint: host allocation failed");
    }
    return LSS_ADI_OK;
}

} // namespace lss_gb300
