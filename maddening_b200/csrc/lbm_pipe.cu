// Rollouts of the pipe node: single phase with its tracer, Shan-Chen two-phase.
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>
#include <utility>

#include "lbm_host.h"
#include "lbm_multiphase.cuh"
#include "lbm_pipe.cuh"

// Single-phase pipe rollout: one fused launch per step (k_pipe_step: D3Q19
// pull step + the tracer of the same cell), tracer populations ping-ponged
// between two plane sets.  A single step (the call a graph manager makes) runs
// its fluid half in one pass over the reference layout instead, then the
// tracer with the velocity that pass wrote: 173 + 69 + 60 B per cell for 496
// (256 x 128 x 128 FP32: 351 -> 271 us).
template <class S>
int run_pipe(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
             const void* t_in, void* t_out, int64_t n, double tau_tracer, void* tracer_out,
             char* ws) {
  using IO = typename lbm::StoreT<S>::IO;
  const size_t cells = p->g.ncell;
  const size_t sb = align256(state_bytes(p)), tb = align256(7 * cells * p->io);
  char* A = ws;
  char* B = ws + sb;
  char* T[2] = {ws + 2 * sb, ws + 2 * sb + tb};
  const unsigned grid = grid_for(p->g.ncell);
  lbm::TracerArgs t{};
  t.g = p->g;
  t.wall = a.wall;
  t.inv_tau = 1.0 / tau_tracer;
  t.f7_in = t_in;
  t.tout = T[0];
  a.f_in = f_in;
  a.f_out = f_out;
  a.prs = nullptr;
  int rc;
  bool done = false;
  if constexpr (std::is_same<S, float>::value) {
    if (n == 1 && tiled_form<S>(p, a, ws, true) == kTiledBulk) {
      lbm::StepArgs m = a;
      m.mflags &= ~lbm::kMomRawVelocity;
      if (m.vel == nullptr) m.vel = ws + 2 * sb + 2 * tb;
      m.status = reinterpret_cast<int*>(ws);
      rc = cuda_check(cudaMemsetAsync(m.status, 0, sizeof(int), s), "cudaMemsetAsync");
      if (rc) return rc;
      rc = launch_tiled_pipe<19, S>(p, m, s);
      if (rc) return rc;
      t.vel = m.vel;
      lbm::k_tracer_step<IO><<<grid, lbm::kBlock, 0, s>>>(t);
      rc = cuda_check(cudaGetLastError(), "k_tracer_step launch");
      if (rc) return rc;
      done = true;
    }
  }
  int cur = 0;
  if (!done) {
    lbm::StepArgs m = a;
    m.rho = m.vel = nullptr;
    m.pout = A;
    rc = launch_prepare<19, S>(m, s);
    if (rc) return rc;
    for (int64_t i = 1; i < n; ++i) {
      m.pin = A;
      m.pout = B;
      if (i == 1) launch_after(lbm::k_pipe_step<S, true, false>, grid, lbm::kBlock, s, m, t);
      else launch_after(lbm::k_pipe_step<S, false, false>, grid, lbm::kBlock, s, m, t);
      rc = cuda_check(cudaGetLastError(), "k_pipe_step launch");
      if (rc) return rc;
      std::swap(A, B);
      t.tin = T[cur];
      cur = 1 - cur;
      t.tout = T[cur];
    }
    a.pin = A;
    a.mflags &= ~lbm::kMomRawVelocity;
    if (n == 1) launch_after(lbm::k_pipe_step<S, true, true>, grid, lbm::kBlock, s, a, t);
    else launch_after(lbm::k_pipe_step<S, false, true>, grid, lbm::kBlock, s, a, t);
    rc = cuda_check(cudaGetLastError(), "k_pipe_step launch");
    if (rc) return rc;
  }
  t.tin = T[cur];
  t.f7_out = t_out;
  t.tracer_out = tracer_out;
  launch_after(lbm::k_tracer_final<IO>, grid, lbm::kBlock, s, t);
  return cuda_check(cudaGetLastError(), "k_tracer_final launch");
}

// Multiphase pipe step (G != 0): two passes per step over pre-collision
// population planes (lbm_multiphase.cuh); the workspace holds two population
// sets and the psi plane, inside the single-phase layout.
template <class R>
int run_pipe_mp(const lbm_plan* p, cudaStream_t s, const lbm::StepArgs& a,
                const lbm_pipe_args* pa, const void* f_in, void* f_out, const void* t_in,
                void* t_out, int64_t n, const lbm_moments* out, void* tracer_out, char* ws) {
  const size_t cells = p->g.ncell;
  const size_t sb = align256(state_bytes(p));
  char* A = ws;
  char* B = ws + sb;
  lbm::MPArgs m{};
  m.s = a;
  m.G = pa->G;
  m.rho0 = pa->rho_0;
  m.psi_wall = pa->rho_0 * (1.0 - std::exp(-pa->rho_wall / pa->rho_0));
  m.rho_gas = pa->rho_gas;
  m.drho = pa->rho_liquid - pa->rho_gas;
  m.psi = ws + 2 * sb;
  m.f_aos_in = f_in;
  const unsigned grid = grid_for(p->g.ncell);
  // step 1: psi of the reference f, then its collide into A
  launch_after(lbm::k_mp_density<R, lbm::kMPFirst>, grid, lbm::kBlock, s, m);
  int rc = cuda_check(cudaGetLastError(), "k_mp_density launch");
  if (rc) return rc;
  m.fout = A;
  launch_after(lbm::k_mp_collide<R, true>, grid, lbm::kBlock, s, m);
  rc = cuda_check(cudaGetLastError(), "k_mp_collide launch");
  if (rc) return rc;
  // steps 2..n: both passes pull from the post-collision planes
  for (int64_t i = 1; i < n; ++i) {
    m.fin = A;
    m.fout = B;
    launch_after(lbm::k_mp_density<R, lbm::kMPStep>, grid, lbm::kBlock, s, m);
    rc = cuda_check(cudaGetLastError(), "k_mp_density launch");
    if (rc) return rc;
    launch_after(lbm::k_mp_collide<R, false>, grid, lbm::kBlock, s, m);
    rc = cuda_check(cudaGetLastError(), "k_mp_collide launch");
    if (rc) return rc;
    std::swap(A, B);
  }
  m.fin = A;
  m.f_aos_out = f_out;
  m.rho_out = out != nullptr ? out->density : nullptr;
  m.vel_out = out != nullptr ? out->velocity : nullptr;
  m.tracer_out = tracer_out;
  launch_after(lbm::k_mp_density<R, lbm::kMPLast>, grid, lbm::kBlock, s, m);
  rc = cuda_check(cudaGetLastError(), "k_mp_density launch");
  if (rc) return rc;
  // tracer_f is not evolved in multiphase mode (lbm_pipe.py:858-860)
  return cuda_check(cudaMemcpyAsync(t_out, t_in, 7 * cells * sizeof(R), cudaMemcpyDeviceToDevice, s),
                    "tracer_f copy");
}

#define LBM_PIPE_INST(R)                                                                      \
  template int run_pipe<R>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*, void*,  \
                           const void*, void*, int64_t, double, void*, char*);                \
  template int run_pipe_mp<R>(const lbm_plan*, cudaStream_t, const lbm::StepArgs&,            \
                              const lbm_pipe_args*, const void*, void*, const void*, void*,   \
                              int64_t, const lbm_moments*, void*, char*);
LBM_PIPE_INST(float)
LBM_PIPE_INST(double)
