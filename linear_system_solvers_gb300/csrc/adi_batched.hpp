// adi_batched.hpp -- batched persistent-kernel solver and the adjoint solver.
#pragma once

#include <memory>
#include <vector>

#include "adi_common.hpp"
#include "adi_device.cuh"
#include "adi_tables.hpp"

namespace lss_gb300 {

// Single instance on the factorised ("fast") arithmetic: one kernel per stage over the whole
// GPU, graph-replayed time loop (behind lss_adi_create with LSS_ADI_ARITH_FAST).
struct wide_solver_base {
    virtual ~wide_solver_base() = default;
    virtual int forward(const void *payoff, void *out_surface, double *out_value, int flags, void *stream,
                        bool use_graph) = 0;
    virtual int grid(void *x, void *y) const = 0;
    virtual int chunks(int s_chunks, int v_chunks, int *out_s, int *out_v, void *stream) = 0;
    // true once lss_adi_line_chunks has set counts (0: chosen by the line's length)
    virtual bool asked_chunks(int &s_chunks, int &v_chunks) const = 0;
};
int make_wide_solver(const lss_adi_problem &p, std::unique_ptr<wide_solver_base> &out);
// the same with the line solves partitioned over the whole GPU (adi_wide.cu)
int make_partitioned_solver(const lss_adi_problem &p, std::unique_ptr<wide_solver_base> &out);

// Forward + adjoint of one parametric FP64 instance (behind lss_adi_adjoint, adi_wide.cu).
struct wide_adjoint_base {
    virtual ~wide_adjoint_base() = default;
    virtual int set_chunks(int s_chunks, int v_chunks, void *stream) = 0; // counts of lss_adi_line_chunks
    virtual int run(const void *payoff, double *out_value, double *dv_dparams, void *dv_dpayoff, int checkpoint_every, int flags,
                    void *stream) = 0;
};
int make_wide_adjoint(const lss_adi_problem &p, std::unique_ptr<wide_adjoint_base> &out);

// Most chunks per line that lss_adi_line_chunks sets.
constexpr int MAX_CHUNKS = 128;

} // namespace lss_gb300
