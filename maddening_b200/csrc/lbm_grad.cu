// Differentiated rollout: checkpointed (or moment-keeping) forward pass and the
// reverse sweep over the adjoint kernels.
#include <cuda_runtime.h>

#include <utility>

#include "lbm_adjoint.cuh"
#include "lbm_host.h"

// Forward pass that keeps (rho^n, u^n) of every step (AdjLayout::full).
template <int Q, class S>
int adj_forward_full(cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
                     const AdjLayout& L, char* ws) {
  char* cur = ws + L.A;
  char* nxt = ws + L.B;
  lbm::StepArgs m = a;
  m.prs = nullptr;
  m.mflags = lbm::kMomRawVelocity;
  m.f_in = f_in;
  auto keep = [&](int64_t n) {
    m.rho = ws + L.hist + static_cast<size_t>(n) * L.slot;
    m.vel = static_cast<char*>(m.rho) + L.rho_bytes;
  };
  keep(0);
  m.pout = cur;
  int rc = launch_prepare<Q, S>(m, s);
  if (rc) return rc;
  for (int64_t n = 1; n < L.T; ++n) {
    keep(n);
    m.pin = cur;
    m.pout = nxt;
    rc = launch_step<Q, S>(m, false, s);
    if (rc) return rc;
    std::swap(cur, nxt);
  }
  // the moments of f^T, raw in walls
  keep(L.T);
  m.pin = cur;
  rc = launch_step_moments_only<Q, S>(m, s);
  if (rc) return rc;
  a.pin = cur;
  a.f_out = f_out;
  return launch_step<Q, S>(a, true, s);
}

template <int Q, class S>
int adj_forward(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
                const AdjLayout& L, char* ws) {
  if (L.full) return adj_forward_full<Q, S>(s, a, f_in, f_out, L, ws);
  char* AB[2] = {ws + L.A, ws + L.B};
  auto slot = [&](int64_t j) { return ws + L.ck + static_cast<size_t>(j - 1) * L.sb; };
  // Producer of p^m writes into checkpoint j = (m+1)/K when m+1 is a segment start.
  auto out_for = [&](int64_t m, char* cur) -> char* {
    if ((m + 1) % L.K == 0 && m + 1 < L.T) return slot((m + 1) / L.K);
    return cur == AB[0] ? AB[1] : AB[0];
  };
  lbm::StepArgs m = a;
  m.rho = m.vel = m.prs = nullptr;
  m.f_in = f_in;
  char* cur = out_for(0, nullptr);
  m.pout = cur;
  int rc = launch_prepare<Q, S>(m, s);
  if (rc) return rc;
  for (int64_t n = 1; n < L.T; ++n) {
    char* nxt = out_for(n, cur);
    m.pin = cur;
    m.pout = nxt;
    rc = launch_state_step<Q, S>(p, m, s);
    if (rc) return rc;
    cur = nxt;
  }
  a.pin = cur;
  a.f_out = f_out;
  return launch_step<Q, S>(a, true, s);
}

template <int Q, class S>
int adj_backward(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in,
                 const void* g_rho, const void* g_vel, const void* g_f, double* grad_force,
                 void* grad_f_in, const AdjLayout& L, char* ws) {
  char* AB[2] = {ws + L.A, ws + L.B};
  char* MU[2] = {ws + L.mu0, ws + L.mu1};
  auto slot = [&](int64_t j) { return ws + L.ck + static_cast<size_t>(j - 1) * L.sb; };
  auto hist_rho = [&](int64_t j) { return ws + L.hist + static_cast<size_t>(j) * L.slot; };
  auto hist_vel = [&](int64_t j) { return hist_rho(j) + L.rho_bytes; };
  double* dF = reinterpret_cast<double*>(ws + L.dF);
  const unsigned grid = grid_for(p->g.ncell);

  lbm::AdjArgs q{};
  q.g = p->g;
  q.omega = a.omega;
  q.guo_c = a.guo_c;
  q.force_mode = a.force_mode;
  for (int d = 0; d < 3; ++d) q.force[d] = a.force[d];
  q.force_field = a.force_field;
  q.wall = a.wall;
  q.dF = grad_force != nullptr ? dF : nullptr;
  const bool force = a.force_mode != 0;

  lbm::StepArgs m = a;  // recompute steps: moments into the history, raw velocity
  m.prs = nullptr;
  m.mflags = lbm::kMomRawVelocity;
  m.f_in = f_in;
  int mu = 0;  // MU[mu] holds mu^{n+1}
  int rc = LBM_OK;
  const int64_t segments = L.full ? 1 : L.S;
  for (int64_t sg = segments - 1; sg >= 0; --sg) {
    const int64_t n0 = sg * L.K;
    const int64_t n1 = L.full || n0 + L.K > L.T ? L.T : n0 + L.K;
    if (!L.full) {
      // (rho^n, u^n) for n in [n0, n1): recompute from the segment's checkpoint
      char* cur = AB[0];
      m.rho = hist_rho(0);
      m.vel = hist_vel(0);
      m.pout = cur;
      if (sg == 0) {
        rc = launch_prepare<Q, S>(m, s);
      } else {
        m.pin = slot(sg);
        rc = launch_step<Q, S>(m, false, s);
      }
      if (rc) return rc;
      for (int64_t n = n0 + 1; n < n1; ++n) {
        char* nxt = cur == AB[0] ? AB[1] : AB[0];
        m.rho = hist_rho(n - n0);
        m.vel = hist_vel(n - n0);
        m.pin = cur;
        m.pout = nxt;
        rc = launch_step<Q, S>(m, false, s);
        if (rc) return rc;
        cur = nxt;
      }
      if (sg == L.S - 1) {  // moments of f^T
        m.rho = hist_rho(n1 - n0);
        m.vel = hist_vel(n1 - n0);
        m.pin = cur;
        rc = launch_step_moments_only<Q, S>(m, s);
        if (rc) return rc;
      }
    }
    if (sg == segments - 1) {
      // lambda^T from the output gradients
      q.rho = hist_rho(n1 - n0);
      q.vel = hist_vel(n1 - n0);
      q.g_rho = g_rho;
      q.g_vel = g_vel;
      q.g_f = g_f;
      q.mout = MU[mu];
      lbm::k_adj_init<Q, S><<<grid, lbm::kBlock, 0, s>>>(q);
      rc = cuda_check(cudaGetLastError(), "k_adj_init launch");
      if (rc) return rc;
    }
    for (int64_t n = n1 - 1; n >= n0; --n) {
      q.rho = hist_rho(n - n0);
      q.vel = hist_vel(n - n0);
      q.min = MU[mu];
      q.mout = MU[1 - mu];
      const bool aos = n == 0 && grad_f_in != nullptr;
      q.grad_f0 = grad_f_in;
      if (aos) {
        if (force) launch_after(lbm::k_adj_step<Q, S, true, lbm::kAdjOutAoS>, grid, lbm::kBlock, s, q);
        else launch_after(lbm::k_adj_step<Q, S, false, lbm::kAdjOutAoS>, grid, lbm::kBlock, s, q);
      } else {
        if (force) launch_after(lbm::k_adj_step<Q, S, true, lbm::kAdjOutState>, grid, lbm::kBlock, s, q);
        else launch_after(lbm::k_adj_step<Q, S, false, lbm::kAdjOutState>, grid, lbm::kBlock, s, q);
      }
      rc = cuda_check(cudaGetLastError(), "k_adj_step launch");
      if (rc) return rc;
      mu = 1 - mu;
    }
  }
  if (grad_force != nullptr) {
    if (a.force_mode == LBM_FORCE_UNIFORM) {
      double* part = reinterpret_cast<double*>(ws + L.part);
      if (p->D == 3)
        lbm::k_field_sum_part<3><<<kReduceBlocks, lbm::kReduceThreads, 0, s>>>(dF, p->g.ncell, part);
      else
        lbm::k_field_sum_part<2><<<kReduceBlocks, lbm::kReduceThreads, 0, s>>>(dF, p->g.ncell, part);
      lbm::k_field_sum_final<<<1, lbm::kReduceThreads, 0, s>>>(part, kReduceBlocks, p->D,
                                                              grad_force);
      rc = cuda_check(cudaGetLastError(), "k_field_sum launch");
    } else {
      rc = cuda_check(cudaMemcpyAsync(grad_force, dF,
                                      static_cast<size_t>(p->g.ncell) * p->D * sizeof(double),
                                      cudaMemcpyDeviceToDevice, s),
                      "cudaMemcpyAsync");
    }
  }
  return rc;
}

#define LBM_GRAD_INST(Q, S)                                                                    \
  template int adj_forward<Q, S>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*,    \
                                 void*, const AdjLayout&, char*);                              \
  template int adj_backward<Q, S>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*,   \
                                  const void*, const void*, const void*, double*, void*,       \
                                  const AdjLayout&, char*);
LBM_GRAD_INST(19, float)
LBM_GRAD_INST(19, double)
LBM_GRAD_INST(9, float)
LBM_GRAD_INST(9, double)
