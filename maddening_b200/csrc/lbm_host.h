// Host-side pieces shared by the translation units of liblbm_b200.so: the plan,
// the error helpers behind lbm_last_error, and the launchers that live in
// their own units (compiled in parallel).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "../../include/lbm_b200.h"
#include "lbm_kernels.cuh"

struct lbm_plan {
  int Q = 0, D = 0, storage = 0;
  int64_t shape[3] = {0, 0, 0};  // reference grid_shape
  lbm::Geo g{};                  // internal geometry
  double tau = 0;
  size_t elem = 4;               // bytes per stored population
  size_t io = 4;                 // bytes per f / force / moment element
  uint32_t flags = 0;            // LBM_PLAN_* bits
  lbm::Geo gpad{};               // the geometry with state rows of n2 + 1 cells
  bool gpad_ok = false;          // ... indexes below 2^32

  // 16-bit states with odd rows are kept padded inside a rollout where two cells per
  // thread gain more than the padding cell costs (faces: whether the call has face
  // conditions; without them the plan's workspace is sized for it), and wherever the
  // plan asks for pairs.  us of 20 steps, padded pairs / one cell per thread, FP16:
  // without faces 24^3 45.8 / 44.8, 33^3 50.5 / 54.9, 48 x 48 x 49 73 / 91, 200 x 200 x
  // 199 2538 / 3212, 999^2 178 / 229, 200 x 200 x 5 89 / 108, 512 x 512 x 5 525 / 526,
  // 1024 x 1024 x 3 1337 / 1233, 512 x 512 x 1 153 / 128; with faces, whose own code
  // runs for both cells of a pair, 33^3 138 / 101, 64 x 64 x 63 192 / 180, 80 x 80 x 81
  // 269 / 281, 700 x 701 156 / 167, 300 x 300 x 15 627 / 616, 300 x 300 x 31 1138 / 1191.
  bool odd_rows_padded(bool faces) const {
    if (elem != 2 || g.n2 % 2 == 0 || !gpad_ok || (flags & LBM_PLAN_SINGLE_CELLS)) return false;
    if (flags & LBM_PLAN_PAIRED_CELLS) return true;
    if (faces) return g.n2 > 16 && g.ncell >= (3u << 17);
    return g.n2 >= 3 && g.ncell >= (1u << 15) && (g.n2 >= 7 || g.ncell < (1u << 20));
  }
};

// Records the message for lbm_last_error (calling thread) and returns code.
int fail(int code, const char* fmt, ...);
// LBM_OK, or fail(LBM_ERR_CUDA, "<what>: <CUDA message>").
int cuda_check(cudaError_t e, const char* what);

inline size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

inline size_t state_bytes(const lbm_plan* p) {
  return static_cast<size_t>(p->Q) * static_cast<size_t>(p->g.ncell) * p->elem;
}

inline size_t padded_state_bytes(const lbm_plan* p) {
  return static_cast<size_t>(p->Q) * static_cast<size_t>(p->gpad.pstride) * p->elem;
}
// Workspace of a rollout of more than one step: two state copies, a status word.
inline size_t rollout_bytes(const lbm_plan* p) {
  const size_t sb = p->odd_rows_padded(false) ? padded_state_bytes(p) : state_bytes(p);
  return 2 * align256(sb) + 256;
}

inline unsigned grid_for(uint64_t n) { return static_cast<unsigned>((n + lbm::kBlock - 1) / lbm::kBlock); }

// Launches a kernel whose blocks may start while the kernel before it in the
// stream is still finishing (programmatic stream serialisation): only for
// kernels that call grid_wait_previous() before their first memory access.
template <class... KA, class... A>
cudaError_t launch_after(void (*kern)(KA...), dim3 grid, unsigned block, cudaStream_t s,
                         const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// ---- Launchers, one unit per lattice and storage (lbm_steps.cu) ----------
// p = C(f) of the reference state a.f_in into a.pout.
template <int Q, class S>
int launch_prepare(const lbm::StepArgs& a, cudaStream_t s);
// One step, one cell per thread: the next state, or (final_aos) f_bc and moments.
template <int Q, class S>
int launch_step(const lbm::StepArgs& a, bool final_aos, cudaStream_t s);
template <int Q, class S>
int launch_step_moments_only(const lbm::StepArgs& a, cudaStream_t s);
template <int Q, class S>
int run_padded(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
               char* ws);
template <int Q, class S>
int run_steps(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
              int64_t n, char* ws, size_t ws_bytes);
template <int Q, class S>
int run_history(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in,
                void* f_out, int64_t n, int64_t every, const lbm_history* h, char* ws);
enum StateOp { kFromF, kStep, kToF };
template <int Q, class S>
int state_op(StateOp op, const lbm::StepArgs& a, cudaStream_t s);
// One state-to-state step in the form the plan and the storage take.
template <int Q, class S>
int launch_state_step(const lbm_plan* p, const lbm::StepArgs& m, cudaStream_t s);

// ---- Differentiated rollout (lbm_grad.cu) -----------------------------------
constexpr int kReduceBlocks = 148 * 4;
struct AdjLayout {
  int64_t T = 0, K = 0, S = 0;  // steps, checkpoint interval, segments
  size_t sb = 0;                // bytes of one population copy
  size_t rho_bytes = 0, slot = 0;
  size_t A = 0, B = 0, ck = 0, hist = 0, mu0 = 0, mu1 = 0, dF = 0, part = 0, total = 0;
  bool full = false;  // the moments of every step are kept: no checkpoints, no recompute
};

template <int Q, class S>
int adj_forward(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
                const AdjLayout& L, char* ws);
template <int Q, class S>
int adj_backward(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in,
                 const void* g_rho, const void* g_vel, const void* g_f, double* grad_force,
                 void* grad_f_in, const AdjLayout& L, char* ws);

// ---- Batched ensemble (lbm_batch.cu) ----------------------------------------
// A contiguous range [t0, t1) of the tile list whose instances are stepped
// together; grid = blocks of the persistent launch for that range; pair = its
// state steps run the paired kernel (16-bit storage, even rows).
struct TileRange {
  uint32_t t0, t1;  // reference-layout tiles (prepare, one-cell steps, last step)
  uint32_t s0, s1;  // state-layout tiles (paired state steps)
  unsigned grid, sgrid;
  bool pair;        // state steps paired
  bool pad;         // ... with padded state rows
};

template <int Q, class S>
int batched_run(const lbm::StepArgs* args, const lbm::BatchTile* tiles,
                const lbm::BatchTile* stiles, uint32_t ntiles, unsigned grid_all,
                const std::vector<TileRange>& groups, int64_t n, cudaStream_t s,
                cudaStream_t side, bool use_graph, int spec);

// ---- Pipe node (lbm_pipe.cu) -------------------------------------------------
template <class S>
int run_pipe(const lbm_plan* p, cudaStream_t s, lbm::StepArgs a, const void* f_in, void* f_out,
             const void* t_in, void* t_out, int64_t n, double tau_tracer, void* tracer_out,
             char* ws);
template <class R>
int run_pipe_mp(const lbm_plan* p, cudaStream_t s, const lbm::StepArgs& a,
                const lbm_pipe_args* pa, const void* f_in, void* f_out, const void* t_in,
                void* t_out, int64_t n, const lbm_moments* out, void* tracer_out, char* ws);

// One-pass tiled step (lbm_tiled.cuh, launched from lbm_tiled.cu) for 32-bit
// IO: MODE lbm::kOutAoS (a whole update) or lbm::kOutState (the first step of a
// rollout).  Instantiated for Q in {9, 19}, S in {float, __half, __nv_bfloat16}.
template <int Q, class S, int MODE>
int launch_tiled(const lbm_plan* p, const lbm::StepArgs& a, cudaStream_t s);

// The fluid half of one pipe-node step (force mode 3) in one pass: f_bc and the
// moments (D3Q19 FP32).
template <int Q, class S>
int launch_tiled_pipe(const lbm_plan* p, const lbm::StepArgs& a, cudaStream_t s);

// The one-pass update without any alignment of rows and buffers (D2Q9).
template <int Q, class S>
int launch_tiled_words(const lbm_plan* p, const lbm::StepArgs& a, cudaStream_t s);

// Where a D2Q9 lattice takes the one-pass step: it must fill the tiles (rows of
// kTiledRow9 cells) and be long enough for the ring's latency to hide.  Short or
// just-over-a-tile rows leave the lanes idle and small lattices are a few planes
// per block, one after the other, while the two passes then run from the L2.
// One pass / two passes, us a call (FP32, chained calls in a recorded graph):
// bulk copies 4096 x 256 34 / 25, 4096 x 128 120 / 108 (8e6 cells: 199 / 208),
// 1024^2 25 / 26, 1000 x 1048 23 / 25, 1000 x 2097 40 / 56, 512 x 2048 28 / 25,
// 512 x 4096 48 / 56, 300 x 6990 52 / 57, 256^2 10 / 5; word copies 3 x 21845 73 /
// 5, 3 x 349525 1045 / 26, 100 x 10485 38 / 25, 301 x 13934 118 / 109, 999 x 1049
// 27 / 26, 999 x 1574 38 / 43, 1023 x 1537 42 / 43, 1023 x 2050 53 / 57.  Queued
// calls of the smaller ones cost the same 23 us to issue either way.
constexpr uint32_t kTiledRow9 = 252;
inline bool tiled_pays9(const lbm::Geo& g, bool words) {
  const uint64_t n2 = g.n2, held = (n2 + kTiledRow9 - 1) / kTiledRow9 * kTiledRow9;
  const uint64_t used = uint64_t(g.ncell) * n2;  // cells x share of the tiles' lanes x held
  return words ? 3 * n2 >= 2 * held && used >= (uint64_t(5) << 18) * held
               : 9 * n2 >= 5 * held && used >= (uint64_t(1) << 20) * held;
}

// How the one-pass step takes the call: not at all (FP64, a plan that asked for
// two passes, padded rows, f_out overlapping f_in, which other blocks still read,
// a D2Q9 lattice on which two passes are faster unless the plan asked for one),
// by bulk copies (rows of a multiple of 4 cells and 16-byte aligned
// reference-layout buffers), else for D2Q9 by word copies.  A D3Q19 plane is 250
// warp-wide word copies and lost: 255^3 1.66 ms with one producer warp, 1.02 with
// four, 0.85 in two passes.  status: where its status word goes.
enum TiledForm { kTiledNone, kTiledWords, kTiledBulk };
template <class S>
TiledForm tiled_form(const lbm_plan* p, const lbm::StepArgs& a, const void* status, bool aos_out) {
  if constexpr (sizeof(typename lbm::StoreT<S>::IO) != 4) {
    return kTiledNone;
  } else {
    if (p->flags & LBM_PLAN_TWO_PASS) return kTiledNone;
    if (a.g.rstride != a.g.n2 || a.face_inset != 0) return kTiledNone;
    const uintptr_t fi = reinterpret_cast<uintptr_t>(a.f_in);
    const uintptr_t fo = reinterpret_cast<uintptr_t>(a.f_out);
    if (fi % 4 != 0 || reinterpret_cast<uintptr_t>(status) % 4 != 0) return kTiledNone;
    if (aos_out) {
      const uintptr_t bytes = static_cast<uintptr_t>(p->g.ncell) * p->Q * 4;
      if (fo % 4 != 0 || (fo < fi + bytes && fi < fo + bytes)) return kTiledNone;
    }
    const bool aligned = p->g.n2 % 4 == 0 && fi % 16 == 0 && (!aos_out || fo % 16 == 0);
    if (p->Q == 9 && !(p->flags & (LBM_PLAN_ONE_PASS | LBM_PLAN_TEST_WAIT_TIMEOUT)) &&
        !tiled_pays9(p->g, !aligned))
      return kTiledNone;
    return aligned ? kTiledBulk : (p->Q == 9 ? kTiledWords : kTiledNone);
  }
}
