// Batched ensemble: the step sequence over the tile list, for one lattice and
// storage (compiled once per pair, like lbm_steps.cu).
#include <cuda_runtime.h>

#include <vector>

#include "lbm_host.h"
#include "lbm_kernels.cuh"
#include "lbm_pair.cuh"

// Prepare pass over all tiles, then for each instance group its n - 1 state
// steps and its last step.  A group whose two population copies fit in L2
// stays there for all of its steps.
template <int Q, class S, int MODE, int SPEC>
void batched_launch(bool pair, bool pad, const lbm::StepArgs* args, const lbm::BatchTile* t,
                    uint32_t nt, unsigned grid, int which, cudaStream_t s) {
  if constexpr (MODE == lbm::kOutState && sizeof(S) == 2) {
    if (pair) {
      if (pad) lbm::k_batched_pair<Q, S, SPEC, true><<<grid, lbm::kBlock, 0, s>>>(args, t, nt, which);
      else lbm::k_batched_pair<Q, S, SPEC, false><<<grid, lbm::kBlock, 0, s>>>(args, t, nt, which);
      return;
    }
  }
  lbm::k_batched_step<Q, S, MODE, SPEC><<<grid, lbm::kBlock, 0, s>>>(args, t, nt, which);
}

// spec: 0 = per-tile run-time choice, else 1 + 2 FACES + FORCE shared by all members
template <int Q, class S, int MODE>
void batched_step(int spec, bool pair, bool pad, const lbm::StepArgs* args,
                  const lbm::BatchTile* t, uint32_t nt, unsigned grid, int which, cudaStream_t s) {
  switch (spec) {
    case 1: batched_launch<Q, S, MODE, 1>(pair, pad, args, t, nt, grid, which, s); break;
    case 2: batched_launch<Q, S, MODE, 2>(pair, pad, args, t, nt, grid, which, s); break;
    case 3: batched_launch<Q, S, MODE, 3>(pair, pad, args, t, nt, grid, which, s); break;
    case 4: batched_launch<Q, S, MODE, 4>(pair, pad, args, t, nt, grid, which, s); break;
    default: batched_launch<Q, S, MODE, 0>(pair, pad, args, t, nt, grid, which, s); break;
  }
}

template <int Q, class S>
int batched_run(const lbm::StepArgs* args, const lbm::BatchTile* tiles,
                const lbm::BatchTile* stiles, uint32_t ntiles, unsigned grid_all,
                const std::vector<TileRange>& groups, int64_t n, cudaStream_t s,
                cudaStream_t side, bool use_graph, int spec) {
  lbm::k_batched_prepare<Q, S><<<grid_all, lbm::kBlock, 0, s>>>(args, tiles, ntiles);
  int rc = cuda_check(cudaGetLastError(), "k_batched_prepare launch");
  if (rc) return rc;
  cudaStream_t ls = s;
  cudaGraph_t graph = nullptr;
  if (use_graph) {
    // The step sequence is recorded on the batch's own stream (capture only
    // records, nothing runs there) and replayed on the caller's stream, after
    // the work already queued on it.
    rc = cuda_check(cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal),
                    "cudaStreamBeginCapture");
    if (rc) return rc;
    ls = side;
  }
  for (const TileRange& r : groups) {
    const lbm::BatchTile* t = tiles + r.t0;
    const uint32_t nt = r.t1 - r.t0;
    for (int64_t k = 1; k < n; ++k) {
      if (r.pair)
        batched_step<Q, S, lbm::kOutState>(spec, true, r.pad, args, stiles + r.s0, r.s1 - r.s0,
                                           r.sgrid, static_cast<int>(k % 2), ls);
      else
        batched_step<Q, S, lbm::kOutState>(spec, false, false, args, t, nt, r.grid,
                                           static_cast<int>(k % 2), ls);
    }
    batched_step<Q, S, lbm::kOutAoS>(spec, false, false, args, t, nt, r.grid, 2, ls);
  }
  rc = cuda_check(cudaGetLastError(), "k_batched_step launch");
  if (use_graph) {
    const int rc2 = cuda_check(cudaStreamEndCapture(side, &graph), "cudaStreamEndCapture");
    if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (rc2) return rc2;
    cudaGraphExec_t exec = nullptr;
    rc = cuda_check(cudaGraphInstantiate(&exec, graph, 0), "cudaGraphInstantiate");
    cudaGraphDestroy(graph);
    if (rc) return rc;
    rc = cuda_check(cudaGraphLaunch(exec, s), "cudaGraphLaunch");
    cudaGraphExecDestroy(exec);  // released once the launched graph completes
  }
  return rc;
}

#define LBM_UNIT(Q, S)                                                                       \
  template int batched_run<Q, S>(const lbm::StepArgs*, const lbm::BatchTile*,                \
                                 const lbm::BatchTile*, uint32_t, unsigned,                  \
                                 const std::vector<TileRange>&, int64_t, cudaStream_t,       \
                                 cudaStream_t, bool, int);
LBM_UNIT(LBM_UNIT_Q, LBM_UNIT_S)
