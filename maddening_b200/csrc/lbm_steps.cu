// Launches and rollouts of the step kernels for one lattice and storage: the
// build compiles this file once per pair (LBM_UNIT_Q, LBM_UNIT_S), so that the
// units are compiled in parallel and each as a whole.
#include <cuda_runtime.h>

#include "lbm_host.h"
#include "lbm_kernels.cuh"
#include "lbm_pair.cuh"

namespace {

// AFTER: as a step of a rollout on one stream (launch_after).
template <int Q, class S, int MODE, bool AFTER = true>
void launch_step_mode(const lbm::StepArgs& a, cudaStream_t s) {
  const unsigned grid = grid_for(a.cell_end - a.cell0);
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  auto launch = [&](void (*kern)(const lbm::StepArgs)) {
    if constexpr (AFTER) launch_after(kern, grid, lbm::kBlock, s, a);
    else kern<<<grid, lbm::kBlock, 0, s>>>(a);
  };
  if (faces) {
    if (force) launch(lbm::k_step<Q, S, MODE, true, true>);
    else launch(lbm::k_step<Q, S, MODE, true, false>);
  } else {
    if (force) launch(lbm::k_step<Q, S, MODE, false, true>);
    else launch(lbm::k_step<Q, S, MODE, false, false>);
  }
}

// Paired-cell state step (lbm_pair.cuh): the default for 16-bit storage; for FP32
// without faces, or on lattices large enough that the faces' own code is few
// warps' work; always with LBM_PLAN_PAIRED_CELLS, never with
// LBM_PLAN_SINGLE_CELLS.  FP32 us a step of a 20-step rollout with two cells / one
// cell per thread: without faces 64^3 5.7 / 6.5, 96^3 21.3 / 23.3, 256^3 396 / 424,
// 512^2 3.8 / 4.5, 1024^2 9.5 / 11.9.  With faces, D3Q19: 64^3 9.5 / 8.5, 80^3 14.0 /
// 13.3, 96^3 24.6 / 25.1, 112^3 40.1 / 39.2, 128^3 57.1 / 56.9, 144^3 79.1 / 78.5, 160^3
// 105 / 107, 176^3 140 / 143, 200^3 197 / 204, 256^3 404 / 428: 2 % either way between
// 96^3 and 160^3, a gain beyond.  D2Q9: 362^2 5.1 / 4.4, 512^2 5.6 / 5.5, 600^2 6.4 /
// 6.4, 700^2 7.3 / 7.8, 800^2 8.4 / 9.4, 960^2 10.7 / 12.3, 1024^2 11.4 / 13.8.
// Rows of even length; state planes and the wall mask aligned for the pair width.
template <int Q, class S>
bool pair_ok(const lbm_plan* p, const lbm::StepArgs& a) {
  if constexpr (sizeof(S) == 8) {
    return false;
  } else {
    if (p->flags & LBM_PLAN_SINGLE_CELLS) return false;
    if (sizeof(S) == 4 && !(p->flags & LBM_PLAN_PAIRED_CELLS)) {
      const bool faces =
          a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
      if (faces && p->g.ncell < (Q == 9 ? 1u << 19 : 1u << 22)) return false;
    }
    const uintptr_t al = 2 * sizeof(S);
    return p->g.n2 % 2 == 0 && reinterpret_cast<uintptr_t>(a.pin) % al == 0 &&
           reinterpret_cast<uintptr_t>(a.pout) % al == 0 &&
           reinterpret_cast<uintptr_t>(a.wall) % 2 == 0;
  }
}

template <int Q, class S, int W>
void launch_pair_w(const lbm::StepArgs& a, cudaStream_t s) {
  const dim3 grid(a.g.n0 * a.g.n1, a.g.n2 / (64 * W));
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  if (faces) {
    if (force) launch_after(lbm::k_step_pair<Q, S, true, true, W>, grid, 32 * W, s, a);
    else launch_after(lbm::k_step_pair<Q, S, true, false, W>, grid, 32 * W, s, a);
  } else {
    if (force) launch_after(lbm::k_step_pair<Q, S, false, true, W>, grid, 32 * W, s, a);
    else launch_after(lbm::k_step_pair<Q, S, false, false, W>, grid, 32 * W, s, a);
  }
}

template <int Q, class S, int W>
void launch_quad_w(const lbm::StepArgs& a, cudaStream_t s) {
  const dim3 grid(a.g.n0 * a.g.n1, a.g.n2 / (128 * W));
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  if (faces) {
    if (force) launch_after(lbm::k_step_quad<Q, S, true, true, W>, grid, 32 * W, s, a);
    else launch_after(lbm::k_step_quad<Q, S, true, false, W>, grid, 32 * W, s, a);
  } else {
    if (force) launch_after(lbm::k_step_quad<Q, S, false, true, W>, grid, 32 * W, s, a);
    else launch_after(lbm::k_step_quad<Q, S, false, false, W>, grid, 32 * W, s, a);
  }
}

// The four-cell form (16-bit storage): rows of a multiple of 128 cells,
// unpadded state rows, 8-byte aligned planes and a 4-byte aligned wall mask.
// D3Q19 also takes it (a B200 sweep at 256^3 with one-wide arithmetic: 79.2k MLUPS
// FP16 against 71.7k for pairs; register budgets at quad_min_warps) on rows of a
// multiple of 256 cells: with one-warp blocks (rows of 128) it keeps 15 warps resident and
// loses to pairs.
#ifndef LBM_QUAD_Q19
#define LBM_QUAD_Q19 1
#endif
template <int Q, class S>
bool quad_ok(const lbm::StepArgs& a) {
  return (Q == 9 || (LBM_QUAD_Q19 && Q == 19)) && sizeof(S) == 2 &&
         a.g.n2 % (Q == 19 ? 256 : 128) == 0 && a.g.rstride == a.g.n2 &&
         a.g.pstride % 4 == 0 && reinterpret_cast<uintptr_t>(a.pin) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a.pout) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a.wall) % 4 == 0;
}

template <int Q, class S>
void launch_gquad(const lbm::StepArgs& a, cudaStream_t s) {
  const unsigned grid = grid_for(a.g.ncell / 4);
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  if (faces) {
    if (force) launch_after(lbm::k_step_gquad<Q, S, true, true>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_gquad<Q, S, true, false>, grid, lbm::kBlock, s, a);
  } else {
    if (force) launch_after(lbm::k_step_gquad<Q, S, false, true>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_gquad<Q, S, false, false>, grid, lbm::kBlock, s, a);
  }
}

// The instance-wide four-cell form: D2Q9 with 16-bit storage, rows of a
// multiple of 4 cells (a quad never spans two rows), the same alignment as the
// row form (4000^2 channel: 148.9k MLUPS against 114.4k for pairs).  D3Q19
// keeps pairs there: with per-lane rows its 96-register budget spills and it
// lost (48.3k against 61.9k at 160^3; 56.4k at 128 registers and 16 warps).
template <int Q, class S>
bool gquad_ok(const lbm::StepArgs& a) {
  return Q == 9 && sizeof(S) == 2 && a.g.n2 % 4 == 0 &&
         a.g.rstride == a.g.n2 && a.g.pstride % 4 == 0 &&
         reinterpret_cast<uintptr_t>(a.pin) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a.pout) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a.wall) % 4 == 0;
}

template <int Q, class S, bool PAD>
void launch_gpair(const lbm::StepArgs& a, cudaStream_t s) {
  const unsigned grid = grid_for(a.g.pstride / 2);
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  if (faces) {
    if (force) launch_after(lbm::k_step_gpair<Q, S, true, true, PAD>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_gpair<Q, S, true, false, PAD>, grid, lbm::kBlock, s, a);
  } else {
    if (force) launch_after(lbm::k_step_gpair<Q, S, false, true, PAD>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_gpair<Q, S, false, false, PAD>, grid, lbm::kBlock, s, a);
  }
}

template <int Q, class S>
int launch_pair(const lbm::StepArgs& a, cudaStream_t s) {
  if constexpr (sizeof(S) == 8) {
    return fail(LBM_ERR_UNSUPPORTED, "paired step has no FP64 form");
  } else {
    if constexpr ((Q == 9 || (LBM_QUAD_Q19 && Q == 19)) && sizeof(S) == 2) {
      if (quad_ok<Q, S>(a)) {
        if (a.g.n2 % 512 == 0) launch_quad_w<Q, S, 4>(a, s);
        else if (a.g.n2 % 256 == 0) launch_quad_w<Q, S, 2>(a, s);
        else launch_quad_w<Q, S, 1>(a, s);
        return cuda_check(cudaGetLastError(), "k_step_quad launch");
      }
    }
    if constexpr (Q == 9 && sizeof(S) == 2) {
      if (gquad_ok<Q, S>(a)) {
        launch_gquad<Q, S>(a, s);
        return cuda_check(cudaGetLastError(), "k_step_gquad launch");
      }
    }
    // row segments in blocks of two or four warps, else instance-wide pairs (192^3
    // FP16 107 us a step against 122 in one-warp blocks, 320^3 482 / 552)
    if (a.g.n2 % 256 == 0) launch_pair_w<Q, S, 4>(a, s);
    else if (a.g.n2 % 128 == 0) launch_pair_w<Q, S, 2>(a, s);
    else launch_gpair<Q, S, false>(a, s);
    return cuda_check(cudaGetLastError(), "k_step_pair launch");
  }
}

template <int Q, class S>
int launch_step_padded(const lbm::StepArgs& a, cudaStream_t s) {
  const unsigned grid = grid_for(a.g.ncell);
  const bool faces = a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone;
  const bool force = a.force_mode != 0;
  if (faces) {
    if (force) launch_after(lbm::k_step_padded<Q, S, true, true>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_padded<Q, S, true, false>, grid, lbm::kBlock, s, a);
  } else {
    if (force) launch_after(lbm::k_step_padded<Q, S, false, true>, grid, lbm::kBlock, s, a);
    else launch_after(lbm::k_step_padded<Q, S, false, false>, grid, lbm::kBlock, s, a);
  }
  return cuda_check(cudaGetLastError(), "k_step_padded launch");
}

}  // namespace

template <int Q, class S>
int launch_prepare(const lbm::StepArgs& a, cudaStream_t s) {
  const unsigned grid = grid_for(a.g.ncell);
  if (a.force_mode != 0)
    lbm::k_prepare<Q, S, true><<<grid, lbm::kBlock, 0, s>>>(a);
  else
    lbm::k_prepare<Q, S, false><<<grid, lbm::kBlock, 0, s>>>(a);
  return cuda_check(cudaGetLastError(), "k_prepare launch");
}

template <int Q, class S>
int launch_step(const lbm::StepArgs& a, bool final_aos, cudaStream_t s) {
  if (final_aos) launch_step_mode<Q, S, lbm::kOutAoS>(a, s);
  else launch_step_mode<Q, S, lbm::kOutState>(a, s);
  return cuda_check(cudaGetLastError(), "k_step launch");
}

template <int Q, class S>
int launch_step_moments_only(const lbm::StepArgs& a, cudaStream_t s) {
  launch_step_mode<Q, S, lbm::kOutMoments>(a, s);
  return cuda_check(cudaGetLastError(), "k_step launch");
}

// One state-to-state step (p in -> p out, no moments): paired or one-cell.
template <int Q, class S>
int launch_state_step(const lbm_plan* p, const lbm::StepArgs& m, cudaStream_t s) {
  if constexpr (sizeof(S) == 2) {
    if (m.g.rstride != m.g.n2) {  // padded odd rows
      launch_gpair<Q, S, true>(m, s);
      return cuda_check(cudaGetLastError(), "k_step_gpair launch");
    }
  }
  if (pair_ok<Q, S>(p, m)) return launch_pair<Q, S>(m, s);
  return launch_step<Q, S>(m, false, s);
}

// Collide the whole padded block into the workspace, then the padded step.
template <int Q, class S>
int run_padded(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in,
               void* f_out, char* ws) {
  (void)p;
  lbm::StepArgs m = a;
  m.rho = m.vel = m.prs = nullptr;  // halo moments stay the caller's
  m.f_in = f_in;
  m.pout = ws;
  int rc = launch_prepare<Q, S>(m, s);
  if (rc) return rc;
  a.pin = ws;
  a.f_in = f_in;
  a.f_out = f_out;
  return launch_step_padded<Q, S>(a, s);
}

// Runs the first step (one-pass tiled kernel, or prepare + a state step),
// the state steps and the final step; ws holds 1 or 2 state copies (with n > 1
// also the status word after them).
template <int Q, class S>
int run_steps(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
              int64_t n, char* ws, size_t ws_bytes) {
  size_t sb = align256(state_bytes(p));
  if (n > 1 && ws_bytes >= rollout_bytes(p) && reinterpret_cast<uintptr_t>(ws) % 4 == 0 &&
      p->odd_rows_padded(a.face[0].kind != lbm::kFaceNone || a.face[1].kind != lbm::kFaceNone)) {
    // 16-bit state with odd rows: a padding cell per row lets the steps run two
    // cells per thread.  A workspace without room for the padding, or off the 4-byte
    // boundaries that a pair's accesses need, keeps one cell.
    a.g = p->gpad;
    sb = align256(padded_state_bytes(p));
  }
  char* A = ws;
  char* B = ws + sb;
  a.f_in = f_in;
  a.f_out = f_out;
  int rc;
  if constexpr (sizeof(typename lbm::StoreT<S>::IO) == 4) {
    const TiledForm form = n == 1 ? tiled_form<S>(p, a, ws, true) : kTiledNone;
    if (form != kTiledNone) {
      // the whole update in one pass; the workspace holds only the status word
      a.status = reinterpret_cast<int*>(ws);
      rc = cuda_check(cudaMemsetAsync(a.status, 0, sizeof(int), s), "cudaMemsetAsync");
      if (rc) return rc;
      return form == kTiledBulk ? launch_tiled<Q, S, lbm::kOutAoS>(p, a, s)
                                : launch_tiled_words<Q, S>(p, a, s);
    }
  }
  a.pout = A;
  lbm::StepArgs m = a;  // the first pass and intermediate steps write no moments
  m.rho = m.vel = m.prs = nullptr;
  const bool tiled = n > 1 && tiled_form<S>(p, a, ws + 2 * sb, false) == kTiledBulk;
  if (tiled) {
    m.status = reinterpret_cast<int*>(ws + 2 * sb);
    rc = cuda_check(cudaMemsetAsync(m.status, 0, sizeof(int), s), "cudaMemsetAsync");
    if (rc) return rc;
  }
  if (tiled) {
    // step 1 straight from the reference layout (p after one step into A)
    if constexpr (sizeof(typename lbm::StoreT<S>::IO) == 4)
      rc = launch_tiled<Q, S, lbm::kOutState>(p, m, s);
    --n;
  } else {
    rc = launch_prepare<Q, S>(m, s);
  }
  if (rc) return rc;
  for (int64_t i = 0; i + 1 < n; ++i) {
    m.pin = A;
    m.pout = B;
    rc = launch_state_step<Q, S>(p, m, s);
    if (rc) return rc;
    char* t = A;
    A = B;
    B = t;
  }
  a.pin = A;
  a.f_out = f_out;
  return launch_step<Q, S>(a, true, s);
}

// Rollout that also records the reference state after every `every`-th step
// (record r = after step (r + 1) every): recorded state steps write f and the
// moments into the history slots as they collide; the last step's outputs are
// copied into its slot when it is recorded.
template <int Q, class S>
int run_history(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in,
                void* f_out, int64_t n, int64_t every, const lbm_history* h, char* ws) {
  const size_t sb = align256(state_bytes(p));
  const size_t cells = p->g.ncell;
  const size_t fb = cells * p->Q * p->io, rb = cells * p->io, vb = cells * p->D * p->io;
  auto slot = [](void* base, size_t bytes, int64_t r) -> void* {
    return base == nullptr ? nullptr : static_cast<char*>(base) + static_cast<size_t>(r) * bytes;
  };
  char* A = ws;
  char* B = ws + sb;
  lbm::StepArgs m = a;
  m.rho = m.vel = m.prs = nullptr;
  m.f_in = f_in;
  m.pout = A;
  int rc = launch_prepare<Q, S>(m, s);
  if (rc) return rc;
  for (int64_t i = 1; i < n; ++i) {
    m.pin = A;
    m.pout = B;
    if (i % every == 0) {
      const int64_t r = i / every - 1;
      lbm::StepArgs rec = m;
      rec.f_out = slot(h->f, fb, r);
      rec.rho = slot(h->density, rb, r);
      rec.vel = slot(h->velocity, vb, r);
      rec.prs = slot(h->pressure, rb, r);
      launch_step_mode<Q, S, lbm::kOutRecord>(rec, s);
      rc = cuda_check(cudaGetLastError(), "k_step launch");
    } else {
      rc = launch_state_step<Q, S>(p, m, s);
    }
    if (rc) return rc;
    char* t = A;
    A = B;
    B = t;
  }
  const bool last = n % every == 0;
  const int64_t r = n / every - 1;
  a.pin = A;
  a.f_out = f_out;
  // the last step's moments go to the caller's buffers, or straight to the
  // history slot when the caller wants none
  if (last && a.rho == nullptr) a.rho = slot(h->density, rb, r);
  if (last && a.vel == nullptr) a.vel = slot(h->velocity, vb, r);
  if (last && a.prs == nullptr) a.prs = slot(h->pressure, rb, r);
  rc = launch_step<Q, S>(a, true, s);
  if (rc || !last) return rc;
  struct { void* dst; const void* src; size_t bytes; } copies[4] = {
      {slot(h->f, fb, r), f_out, fb},
      {slot(h->density, rb, r), a.rho, rb},
      {slot(h->velocity, vb, r), a.vel, vb},
      {slot(h->pressure, rb, r), a.prs, rb}};
  for (const auto& c : copies) {
    if (c.dst == nullptr || c.dst == c.src) continue;
    rc = cuda_check(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToDevice, s),
                    "cudaMemcpyAsync");
    if (rc) return rc;
  }
  return LBM_OK;
}

template <int Q, class S>
int state_op(StateOp op, const lbm::StepArgs& a, cudaStream_t s) {
  if (op == kFromF) return launch_prepare<Q, S>(a, s);
  // One cell per thread, any storage.  Ordinary launches: the caller orders these
  // steps against exchanges on other streams, and across such a wait a launch
  // ahead of the step before has nothing to hide.
  if (op == kStep) launch_step_mode<Q, S, lbm::kOutState, false>(a, s);
  else launch_step_mode<Q, S, lbm::kOutAoS, false>(a, s);
  return cuda_check(cudaGetLastError(), "k_step launch");
}

#define LBM_UNIT(Q, S)                                                                        \
  template int launch_prepare<Q, S>(const lbm::StepArgs&, cudaStream_t);                      \
  template int launch_step<Q, S>(const lbm::StepArgs&, bool, cudaStream_t);                   \
  template int launch_step_moments_only<Q, S>(const lbm::StepArgs&, cudaStream_t);            \
  template int launch_state_step<Q, S>(const lbm_plan*, const lbm::StepArgs&, cudaStream_t);  \
  template int run_padded<Q, S>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*,    \
                                void*, char*);                                                \
  template int run_steps<Q, S>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*,     \
                               void*, int64_t, char*, size_t);                                \
  template int run_history<Q, S>(const lbm_plan*, cudaStream_t, lbm::StepArgs, const void*,   \
                                 void*, int64_t, int64_t, const lbm_history*, char*);         \
  template int state_op<Q, S>(StateOp, const lbm::StepArgs&, cudaStream_t);
LBM_UNIT(LBM_UNIT_Q, LBM_UNIT_S)
