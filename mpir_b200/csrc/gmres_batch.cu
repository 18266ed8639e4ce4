// Several GMRES-IR solves with one factor in lockstep.
//
// Each right-hand side runs exactly the control flow of GmresLDLIR::Solve
// (gmres_ir.hpp:536-634) and PrecondGmres (gmres_ir.hpp:636-741) that
// Solver::solve_device runs for one: its own Arnoldi basis, Hessenberg
// matrix, Givens rotations, stop tests and refinement steps.  The vectors of
// the batch sit side by side (vector k at k*n inside blocks of n*width
// doubles), so every vector kernel takes the whole batch in one launch
// (gridDim.y = vectors, finished ones masked), and every preconditioner
// application is one several-vector triangular solve (solve_multi.cu) that
// reads L once for all of them.  Per vector the arithmetic outside the
// preconditioner is that of the single solve; the several-vector triangular
// solve sums in another order, so results agree with one-at-a-time solves to
// rounding, and each vector stops on its own tests.
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "solver.hpp"

namespace mpir {

size_t Solver::batch_growth(int width) const {
  if (!plan_ || width <= 1) return 0;
  const int64_t n = std::max<int64_t>(plan_->S.n, 1);
  const int64_t m = std::max<int64_t>(std::min(gmres_iter, n), 1);
  if (bw_ == width && bm_ == m) return 0;
  const size_t want = MultiSolveWorkspace::bytes_for(*plan_, width) +
                      static_cast<size_t>(m + 1 + 6) * n * width * sizeof(double) +
                      Arnoldi::bytes_for(m, width);
  size_t have = bar_.bytes();
  for (const DeviceBuffer *d : {&bV_, &bbs_, &bbp_, &bx_, &br_, &bin_, &bout_, &mws_.vals, &mws_.sync,
                                &mws_.err, &vecb_.infbits})
    have += d->bytes();
  return want > have ? want - have : 0;
}

void Solver::ensure_batch(int width) {
  ensure_vectors();
  const int64_t n = plan_->S.n, m = std::max<int64_t>(std::min(gmres_iter, n), 1);
  if (bw_ == width && bm_ == m) return;
  bw_ = 0;  // until all of it is there
  const size_t blk = static_cast<size_t>(std::max<int64_t>(n, 1)) * width * sizeof(double);
  bV_.resize(blk * (m + 1));
  bbs_.resize(blk);
  bbp_.resize(blk);
  bx_.resize(blk);
  br_.resize(blk);
  bin_.resize(blk);
  bout_.resize(blk);
  bar_.allocate(n, m, width);
  // Columns that no vector of a call uses stay zero (the several-vector
  // solve reads all width columns).
  MPIR_CUDA(cudaMemsetAsync(bV_.as<void>(), 0, blk * (m + 1), stream_));
  for (DeviceBuffer *b : {&bbs_, &bbp_, &bx_, &br_})
    MPIR_CUDA(cudaMemsetAsync(b->as<void>(), 0, blk, stream_));
  if (mws_.nr != width) {
    mws_.allocate(*plan_, width);
    MPIR_CUDA(cudaMemcpy(mws_.err.as<int32_t>() + 1, wait_ctl_, sizeof wait_ctl_,
                         cudaMemcpyHostToDevice));
  }
  vecb_.allocate(n, width);
  bw_ = width;
  bm_ = m;
}

void Solver::precond_device(int nrhs, double *d_X) {
  if (!plan_ || !num_.valid) throw std::logic_error("no valid factor");
  MPIR_CUDA(cudaSetDevice(device));
  const int64_t n = plan_->S.n;
  if (nrhs < 1 || nrhs > kMaxBatch) throw std::invalid_argument("1 <= nrhs <= 16");
  if (nrhs == 1) {
    ldlt_solve(*plan_, num_, d_X, ws_, stream_);
  } else {
    const int width = multi_width(nrhs);
    ensure_batch(width);
    double *blk = bin_.as<double>();
    MPIR_CUDA(cudaMemsetAsync(blk, 0, n * width * sizeof(double), stream_));
    MPIR_CUDA(cudaMemcpyAsync(blk, d_X, n * nrhs * sizeof(double), cudaMemcpyDeviceToDevice,
                              stream_));
    apply(nrhs, width, blk, ActiveFlags());
    MPIR_CUDA(cudaMemcpyAsync(d_X, blk, n * nrhs * sizeof(double), cudaMemcpyDeviceToDevice,
                              stream_));
  }
  MPIR_CUDA(cudaStreamSynchronize(stream_));
  int32_t e0 = 0, e1 = 0;
  MPIR_CUDA(cudaMemcpy(&e0, ws_.err.as<void>(), sizeof e0, cudaMemcpyDeviceToHost));
  if (mws_.nr) MPIR_CUDA(cudaMemcpy(&e1, mws_.err.as<void>(), sizeof e1, cudaMemcpyDeviceToHost));
  if (e0 || e1) {
    device_zero(ws_.err.as<void>(), sizeof(int32_t));
    if (mws_.nr) device_zero(mws_.err.as<void>(), sizeof(int32_t));
    throw WaitTimeout();
  }
}

// GmresLDLIR::Solve (gmres_ir.hpp:536-634) for nrhs right-hand sides.
int Solver::solve_batch_device(int nrhs, const double *d_B, double *d_X, Report *reps) {
  if (!plan_) throw std::logic_error("solve before analyze");
  if (!num_.valid) throw std::logic_error("solve before a successful factor");
  if (nrhs < 1 || nrhs > kMaxBatch) throw std::invalid_argument("1 <= nrhs <= 16");
  MPIR_CUDA(cudaSetDevice(device));
  const int64_t n = plan_->S.n;
  if (n == 0) {
    for (int k = 0; k < nrhs && reps; k++) reps[k] = Report{};
    return kOk;
  }
  const int W = multi_width(nrhs);
  ensure_batch(W);
  const int    nb = nrhs;
  const Plan  &P  = *plan_;
  cudaStream_t s  = stream_;
  MPIR_CUDA(cudaEventRecord(ev0_, s));
  const int64_t *Kp = P.Kp.as<int64_t>();
  const int32_t *Kj = P.Kj.as<int32_t>();
  const double  *Kv = num_.Kval.as<double>();
  double *bs = bbs_.as<double>(), *x = bx_.as<double>(), *r = br_.as<double>();
  double *V = bV_.as<double>(), *ADp = ADp_.as<double>(), *inf = box_->inf;
  const bool dd = ur == kDD;
  std::vector<Report> st(nb);
  for (Report &r : st) r.factor_prec = applied_prec();
  const auto t_outer  = std::chrono::steady_clock::now();
  auto       ms_since = [](std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0)
        .count();
  };
  VecFactors fac{}, scale{};
  for (int k = 0; k < nb; k++) fac.v[k] = 1.0;
  uint32_t act = (1u << nb) - 1u;
  vecb_.rhs_in(nb, P.perm.as<int64_t>(), num_.AD.as<double>(), d_B, bs, ADp, bbp_.as<double>(), s);
  inner(nb, W, act, bs, fac, V, bar_, vecb_, x, false, fac);
  vecb_.residual(nb, act, Kp, Kj, Kv, x, bs, r, dd, true, s);
  vecb_.read_inf(nb, inf, s);
  count_inner(nb, act, bar_.mail(), st.data());
  std::vector<double> bs_inf(nb), r_inf(nb), r_prev(nb, DBL_MAX), r_norm(nb);
  std::vector<IrEvent> evs(nb);
  for (int k = 0; k < nb; k++) {
    st[k].spmv_count++;
    bs_inf[k]               = inf[8 * k + 3];
    r_inf[k]                = inf[8 * k];
    r_norm[k]               = r_inf[k] / bs_inf[k];
    evs[k].initial_residual = r_inf[k];
  }
  const double eps_w = eps_of(uw);
  for (int64_t iter = 1; iter <= ir_iter; iter++) {
    for (int k = 0; k < nb; k++) {
      if (!(act >> k & 1u)) continue;
      if (r_inf[k] == 0.0) {  // exact: nothing left to refine
        st[k].stop_reason = 3;
        act &= ~(1u << k);
      } else if (!std::isfinite(r_inf[k]) || num_.nonfinite) {
        st[k].stop_reason = 4;
        act &= ~(1u << k);
      } else {
        fac.v[k]   = 1.0 / r_inf[k];
        scale.v[k] = r_inf[k];
      }
    }
    if (act == 0) break;
    const auto t_inner = std::chrono::steady_clock::now();
    inner(nb, W, act, r, fac, V, bar_, vecb_, x, true, scale);
    vecb_.residual(nb, act, Kp, Kj, Kv, x, bs, r, dd, false, s);
    vecb_.read_inf(nb, inf, s);
    count_inner(nb, act, bar_.mail(), st.data());
    const double inner_ms = ms_since(t_inner);
    for (int k = 0; k < nb; k++) {
      if (!(act >> k & 1u)) continue;
      const double nrm0 = inf[8 * k + 1], nrm1 = inf[8 * k + 2];
      st[k].spmv_count++;
      r_inf[k]            = inf[8 * k];
      r_norm[k]           = r_inf[k] / bs_inf[k];
      st[k].ir_iterations = static_cast<int32_t>(iter);
      evs[k].iterations.push_back({iter, r_norm[k], nrm0, ms_since(t_outer), inner_ms});
      if (nrm0 <= nrm1 * (10 * eps_w)) {
        st[k].stop_reason = 1;
        act &= ~(1u << k);
      } else if (std::fabs(r_norm[k] - r_prev[k]) < tol) {
        st[k].stop_reason = 2;
        act &= ~(1u << k);
      } else {
        r_prev[k] = r_norm[k];
      }
    }
  }
  vecb_.sol_out(nb, P.perm.as<int64_t>(), ADp, x, d_X, s);
  vecb_.backward_terms(nb, Kp, Kj, num_.Korig.as<double>(), x, ADp, bbp_.as<double>(), s);
  MPIR_CUDA(cudaEventRecord(ev1_, s));
  MPIR_CUDA(cudaMemcpyAsync(&box_->err, mws_.err.as<void>(), sizeof box_->err, cudaMemcpyDeviceToHost, s));
  vecb_.read_inf(nb, inf, s);
  float ms = 0;
  MPIR_CUDA(cudaEventElapsedTime(&ms, ev0_, ev1_));
  for (int k = 0; k < nb; k++) {
    const double *be  = inf + 8 * k + 4;
    const double  den = be[1] * be[2] + be[3];
    st[k].backward_error = den > 0 ? be[0] / den : be[0];
    st[k].residual_norm  = r_norm[k];
    st[k].solve_ms       = ms;
    st[k].factor_ms      = last_factor_ms;
    evs[k].stop_reason      = st[k].stop_reason;
    evs[k].total_iterations = st[k].ir_iterations;
    evs[k].total_time_ms    = ms_since(t_outer);
    log_.push_back(std::move(evs[k]));
  }
  const int rc = box_->err != 0 ? -5 : kOk;
  if (rc != kOk) device_zero(mws_.err.as<void>(), sizeof(int32_t));
  for (int k = 0; k < nb; k++) {
    if (rc != kOk) st[k].status = rc;
    if (reps) reps[k] = st[k];
  }
  return rc;
}

int Solver::solve_batch(int nrhs, const double *B, double *X, Report *reps) {
  if (!plan_) throw std::logic_error("solve before analyze");
  if (nrhs < 1 || nrhs > kMaxBatch) throw std::invalid_argument("1 <= nrhs <= 16");
  MPIR_CUDA(cudaSetDevice(device));
  const int64_t n = plan_->S.n;
  ensure_batch(multi_width(nrhs));
  MPIR_CUDA(cudaMemcpyAsync(bin_.as<void>(), B, n * nrhs * sizeof(double), cudaMemcpyHostToDevice,
                            stream_));
  const int rc = solve_batch_device(nrhs, bin_.as<double>(), bout_.as<double>(), reps);
  MPIR_CUDA(cudaMemcpyAsync(X, bout_.as<void>(), n * nrhs * sizeof(double),
                            cudaMemcpyDeviceToHost, stream_));
  MPIR_CUDA(cudaStreamSynchronize(stream_));
  return rc;
}

}  // namespace mpir
