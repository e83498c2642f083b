// One-pass step from the reference layout: LBMNode.update in a single launch.
//
// The reference's update (src/maddening/nodes/lbm.py:899-986) reads f in its
// own layout (*grid, Q), collides every cell, streams, applies the wall swap
// and the faces and returns f_bc with the moments.  Done as two passes
// (k_prepare: f -> p = C(f) into the state planes; k_step: pull p -> f_bc) it
// moves 76 + 76 + 76 + 96 = 324 B per cell.  This kernel moves f once:
//
//   * A block owns a column of the lattice: a tile of TY x TZ cells across
//     the two inner axes, swept along the outer axis plane by plane (D3Q19:
//     tiles over (a1, a2), sweep along a0; D2Q9: row segments of TZ cells
//     along a2, sweep along a1).
//   * Each plane of the column, with a one-cell halo on every side, is moved
//     from the reference layout into a ring of shared-memory slots by the copy
//     engine (1-D bulk asynchronous copies, cp.async.bulk, completion on an
//     mbarrier); the periodic wrap along a row is a copy of its own.
//   * Warps have one role each and meet only at mbarriers, never at a block
//     barrier: a producer warp issues the copies of plane P once the slot's
//     previous plane is consumed; collide warps collide plane P in place
//     (every tile and halo cell, k_prepare's arithmetic, two cells per lane
//     with two-wide FP32 arithmetic) once it has landed and keep the wall
//     bits of its cells beside it; output warps, each over 32 or 64 cells of
//     the tile, pull the collided populations of plane P from slots P - 1, P,
//     P + 1 once P + 1 is collided, apply the wall swap and the faces, take
//     the moments and write f_bc (kOutAoS: staged per warp in shared memory
//     and written by a bulk asynchronous store) or collide again and write
//     the next state planes (kOutState: the first step of a rollout).
//     Collide warps run up to a few planes ahead of the output warps.
//   * A persistent grid walks work items (column, chunk of planes along the
//     sweep); blocks take items with a grid stride in chunk-major order, so
//     neighbouring columns are swept at the same time and the halo rows they
//     share are served by L2.  Each item costs two extra (halo) planes.
//
// Bytes per cell from HBM: 76 (f) + 76 (f_bc) + 20 (moments) + 1 (wall) for
// D3Q19 FP32; the halo re-reads hit L2.  The arithmetic is the two-pass
// path's operation for operation, so the outputs are bit-identical to it.
//
// Requirements (checked on the host): 32-bit IO (FP32, FP16 or BF16 storage),
// f_in and f_out not overlapping, no halo-padded block; the bulk copies want an
// a2 extent that is a multiple of 4 and f_in (and f_out for kOutAoS) 16-byte
// aligned, the word-copy form (D2Q9 update) neither.  Every wait is bounded in
// time and also ends when another warp has given up; then the block sets bit 0 of
// *status, waits (bounded) for its own copies in flight, fills its output cells
// with NaN and returns.
#pragma once

#include <type_traits>

#include "lbm_kernels.cuh"
#include "lbm_pair.cuh"
#include "lbm_staged.cuh"

namespace lbm {

// Tile shape, warp roles and sweep mapping per lattice.
//
// What bounds the kernel is the chain of dependent instructions in the collide
// and output warps, at the few warps that one ring of planes leaves room for:
// both are busy for 0.8-0.9 of the launch, which issues on 0.58 of the cycles
// with DRAM at 0.43 (160^2 x 128).  One update, measured side by side:
//   D3Q19, 256^3 with spheres and faces / channel with a force: 0.59 / 0.66 ms
//   (0.68 / 0.68 before, with five slots of 37 KB -- whole groups of four halo
//   cells -- and collide lanes that run one cell after the other).  The ring
//   takes six planes of 10 + 2 rows at 31 KB: three read, one collided, two
//   landing.  Two cells per output lane: 0.70 / 0.62 (half the warps); the same
//   in two groups of warps on alternate planes of 8 rows: 0.65 / 0.69; 12 rows in
//   five slots: 0.69 / 0.71; 13 collide warps of one cell per lane: 0.73 / 0.61
//   (80 registers, spills).
//   D2Q9, 4096^2: 0.276 ms (0.41 before): its planes are small, so three blocks
//   of nine warps share an SM.  252 cells per row: the 254 collided cells fill
//   four warps.  124 cells in six blocks: 0.293; 252 in two or four: 0.32, 0.31.
template <int Q>
struct Sweep;
template <>
struct Sweep<19> {
  static constexpr int TY = 10, TZ = 32;    // tile rows (a1) x row cells (a2)
  static constexpr int HR = 1;              // halo rows
  static constexpr int CPO = 1;             // cells per output lane
  static constexpr int OZ = 0;              // its second cell: that many cells further
  static constexpr int NOW = 10;            // output warps
  static constexpr int SLOTS = 6;           // plane slots
  static constexpr int MINB = 1;            // resident blocks per SM
  __host__ __device__ static constexpr int cs(int q) { return Lat<19>::c0(q); }  // sweep
  __host__ __device__ static constexpr int cr(int q) { return Lat<19>::c1(q); }  // rows
};
template <>
struct Sweep<9> {
  static constexpr int TY = 1, TZ = 252;
  static constexpr int HR = 0;
  static constexpr int CPO = 2;
  static constexpr int OZ = 128;
  static constexpr int NOW = 4;
  static constexpr int SLOTS = 6;
  static constexpr int MINB = 3;
  __host__ __device__ static constexpr int cs(int q) { return Lat<9>::c1(q); }
  __host__ __device__ static constexpr int cr(int) { return 0; }
};

template <int Q>
struct TileShape {
  static constexpr int TY = Sweep<Q>::TY, TZ = Sweep<Q>::TZ, HR = Sweep<Q>::HR;
  static constexpr int RP = TY + 2 * HR;              // buffered rows per plane
  static constexpr int CW = TZ + 2;                   // buffered (= collided) cells per row
  // A buffered row: the halo cell before the tile, the tile's cells, the halo
  // cell after it, copied in whole 16-byte units.  Tile rows start on groups of
  // four cells (4 Q x 4 B is a multiple of 16), so the cell before the tile ends
  // on a 16-byte boundary and the cell after it starts on one.
  static constexpr int LCH = (Q + 3) / 4 * 4;         // words of either halo cell's copy
  static constexpr int RW = LCH + TZ * Q + LCH;       // words per buffered row
  static constexpr int PLANE = RP * RW;               // words per plane slot
  static constexpr int NCW = (RP * CW + 63) / 64;     // collide warps, two cells per lane
  static constexpr int NOW = Sweep<Q>::NOW, CPO = Sweep<Q>::CPO, OZ = Sweep<Q>::OZ;
  static constexpr int NT = 32 * (1 + NCW + NOW);     // + the producer warp
  static_assert(TZ % 4 == 0, "tile rows start on 16-byte boundaries");
  static_assert(RP <= 32, "one producer lane per buffered row");
  static_assert(CPO == 1 ? NOW == TY && TZ == 32
                         : TY == 1 && OZ == 32 * NOW && TZ <= 2 * OZ,
                "the output lanes' cells cover the tile");
};

// Barriers and flags of a block, after the slots and the staging rows.
template <int Q>
struct TileSync {
  static constexpr int S = Sweep<Q>::SLOTS;
  uint64_t full[S];      // plane landed (producer arrive + copy bytes)
  uint64_t collided[S];  // plane collided (one arrive per collide warp)
  uint64_t consumed[S];  // plane read for the last time (one per output warp)
  uint32_t wall[S][2 * TileShape<Q>::NCW];  // wall bits of the collided cells
  int abort;             // a wait gave up
  uint32_t issued;       // planes copied by the producer
};

template <int Q, int MODE>
__host__ __device__ constexpr size_t tiled_stage_bytes() {
  return MODE == kOutAoS
             ? static_cast<size_t>(TileShape<Q>::NOW) * 32 * TileShape<Q>::CPO * Q * 4
             : 0;
}
// Shared memory: the ring, the staging rows, kIdleWords words, TileSync.
constexpr uint32_t kIdleWords = 32;
template <int Q, int MODE>
__host__ __device__ constexpr uint32_t tiled_idle_word() {
  return Sweep<Q>::SLOTS * TileShape<Q>::PLANE +
         static_cast<uint32_t>(tiled_stage_bytes<Q, MODE>() / 4);
}
template <int Q, int MODE>
__host__ __device__ constexpr size_t tiled_smem_bytes() {
  return static_cast<size_t>(tiled_idle_word<Q, MODE>() + kIdleWords) * 4 + sizeof(TileSync<Q>);
}

// Place of collide cell m (row m / CW, cell m % CW of a plane's buffered cells) in
// a tile of tyv x tzv cells: its word in slot 0 and the words from a slot to the
// next.  Without such a cell in the tile the lane reads the idle words instead,
// the same in every slot, which nothing writes once the block has started: the
// value is thrown away, but any cell of the plane is one that another warp may be
// overwriting.
struct CollidePlace {
  uint32_t word, step;
};
template <int Q, int MODE>
__host__ __device__ constexpr CollidePlace collide_place(uint32_t m, uint32_t tyv, uint32_t tzv) {
  using T = TileShape<Q>;
  static_assert(Q <= static_cast<int>(kIdleWords), "the idle words hold one cell");
  const uint32_t rr = m / T::CW, cc = m % T::CW;
  if (rr < tyv + 2 * T::HR && cc < tzv + 2)
    return {rr * T::RW + (T::LCH - Q) + cc * Q, static_cast<uint32_t>(T::PLANE)};
  return {tiled_idle_word<Q, MODE>(), 0u};
}

// Host-computed geometry of the sweep.
struct TileGeo {
  uint32_t NS, NR;        // planes along the sweep axis; rows per plane
  uint32_t SS, SR;        // cell strides of the sweep and row axes
  uint32_t ncolz, ncol;   // tiles along a2; tiles per plane
  uint32_t chunk, items;  // planes per work item; work items = ncol x chunks
  uint64_t wait_ns;       // a wait gives up after this long (global timer)
  uint32_t no_copy;       // test hook: barriers armed, no copies issued
};

// One plane of a work item: j = 0 and j = nv + 1 are the halo planes.  The
// item's position is cached when the item starts.
struct PlaneRef {
  uint32_t item, j, nv;
  uint32_t k0;        // first plane of the chunk (sweep coordinate of j = 1)
  uint32_t y0, z0;    // first tile row / cell
  uint32_t tyv, tzv;  // tile rows / cells inside the lattice
};

template <int Q>
__device__ __forceinline__ void plane_first(const StepArgs& a, const TileGeo& t, uint32_t item,
                                            PlaneRef& p) {
  using T = TileShape<Q>;
  p.item = item;
  p.j = 0;
  if (item >= t.items) return;
  const uint32_t col = item % t.ncol;
  p.k0 = (item / t.ncol) * t.chunk;
  p.nv = t.NS - p.k0 < t.chunk ? t.NS - p.k0 : t.chunk;
  p.y0 = (col / t.ncolz) * T::TY;
  p.z0 = (col % t.ncolz) * T::TZ;
  p.tyv = t.NR - p.y0 < static_cast<uint32_t>(T::TY) ? t.NR - p.y0 : T::TY;
  p.tzv = a.g.n2 - p.z0 < static_cast<uint32_t>(T::TZ) ? a.g.n2 - p.z0 : T::TZ;
}
template <int Q>
__device__ __forceinline__ void plane_next(const StepArgs& a, const TileGeo& t, PlaneRef& p) {
  if (p.item >= t.items) return;
  if (++p.j == p.nv + 2) plane_first<Q>(a, t, p.item + gridDim.x, p);
}
// Sweep coordinate of the plane (periodic wrap for the halo planes).
__device__ __forceinline__ uint32_t plane_s(const TileGeo& t, const PlaneRef& p) {
  return wrapu(static_cast<int>(p.k0 + p.j) - 1, t.NS);
}

// Producer warp: lane 0 arms `bar` with the bytes of one plane (tile rows with
// their halo cells), then lane rr copies buffered row rr into buf, so the
// copies of a plane are issued together rather than one after another.
template <int Q>
__device__ __forceinline__ void tiled_issue(const StepArgs& a, const TileGeo& t,
                                            const PlaneRef& p, float* buf, uint64_t* bar,
                                            uint32_t lane) {
  using T = TileShape<Q>;
  const uint32_t ps = plane_s(t, p);
  const uint32_t nrow = p.tyv + 2 * T::HR;
  if (lane == 0) mbar_arrive_expect_tx(bar, nrow * (p.tzv * Q + 2 * T::LCH) * 4);
  __syncwarp();
  const uint32_t rr = lane;
  if (t.no_copy || rr >= nrow) return;
  const uint32_t n2 = a.g.n2;
  const uint32_t r = wrapu(static_cast<int>(p.y0 + rr) - T::HR, t.NR);
  const float* row = static_cast<const float*>(a.f_in) +
                     (static_cast<size_t>(ps) * t.SS + static_cast<size_t>(r) * t.SR) * Q;
  float* dst = buf + static_cast<size_t>(rr) * T::RW;
  // words [b, e) of the row around the tile; either end may wrap
  const bool wrap_l = p.z0 == 0, wrap_r = p.z0 + p.tzv == n2;
  const uint32_t b = p.z0 * Q - (wrap_l ? 0u : T::LCH);
  const uint32_t e = (p.z0 + p.tzv) * Q + (wrap_r ? 0u : T::LCH);
  if (wrap_l) bulk_copy_g2s(dst, row + n2 * Q - T::LCH, T::LCH * 4, bar);
  bulk_copy_g2s(dst + (wrap_l ? T::LCH : 0), row + b, (e - b) * 4, bar);
  if (wrap_r) bulk_copy_g2s(dst + T::LCH + p.tzv * Q, row, T::LCH * 4, bar);
}

// p = C(f) of the reference state of cell c (k_prepare's arithmetic), with the
// 16-bit storage rounding applied and undone: d holds the values the state
// planes would return.
template <int Q, class S, bool FORCE>
__device__ __forceinline__ void collide_ref(const StepArgs& a, uint32_t c, float (&d)[Q]) {
  using R = float;
  R F[3] = {0, 0, 0};
  if (FORCE) {
    if (a.force_mode == 2) load_force<Q, float>(a.force_field, c, F);
    else uniform_force<Q, R>(a, F);
  }
  const Mom<R> m = moments<Q, R, FORCE>(d, F, true);
  collide<Q, R, FORCE>(d, m, F, static_cast<R>(a.omega), static_cast<R>(a.guo_c));
  if constexpr (sizeof(S) == 2) {
    const uint32_t seed = sr_seed(c, m.u[0], m.u[1], m.u[2], m.rd);
#pragma unroll
    for (int q = 0; q < Q; ++q) d[q] = to_r(sr_one<S>(d[q], sr_bits(seed, d[q])));
  }
}

// The same without any alignment (rows that are not groups of four cells, an
// f_in off 16-byte boundaries), for one-row tiles: the warp copies the buffered
// row word by word, the wrapped halo cells as pieces of their own, into the same
// places.
template <int Q>
__device__ __forceinline__ void tiled_issue_words(const StepArgs& a, const TileGeo& t,
                                                  const PlaneRef& p, float* buf, uint64_t* bar,
                                                  uint32_t lane) {
  using T = TileShape<Q>;
  static_assert(T::RP == 1, "one buffered row per plane");
  if (t.no_copy) return;
  const uint32_t n2 = a.g.n2;
  const bool wrap_l = p.z0 == 0, wrap_r = p.z0 + p.tzv == n2;
  const uint32_t b = p.z0 * Q - (wrap_l ? 0u : Q);
  const uint32_t e = (p.z0 + p.tzv) * Q + (wrap_r ? 0u : Q);
  const float* row = static_cast<const float*>(a.f_in) +
                     static_cast<size_t>(plane_s(t, p)) * t.SS * Q;
  float* dst = buf + (T::LCH - Q);  // the cell before the tile
  if (wrap_l && lane < Q) word_copy_g2s(dst + lane, row + (n2 - 1) * Q + lane);
  if (wrap_r && lane < Q) word_copy_g2s(dst + (1 + p.tzv) * Q + lane, row + lane);
  const float* const src = row + b + lane;
  float* const dl = dst + (wrap_l ? Q : 0) + lane;
#pragma unroll 8
  for (uint32_t i = 0; i < (T::CW * Q + 31) / 32; ++i)
    if (lane + i * 32 < e - b) word_copy_g2s(dl + i * 32, src + i * 32);
  word_copies_arrive(bar);
}

// collide_ref for the two cells of a lane (c0, c1), two-wide arithmetic.
template <int Q, class S, bool FORCE>
__device__ __forceinline__ void collide_ref2(const StepArgs& a, uint32_t c0, uint32_t c1,
                                             F2 (&d)[Q]) {
  F2 F[3] = {0, 0, 0};
  if (FORCE) {
    float G0[3], G1[3];
    if (a.force_mode == 2) {
      load_force<Q, float>(a.force_field, c0, G0);
      load_force<Q, float>(a.force_field, c1, G1);
#pragma unroll
      for (int k = 0; k < 3; ++k) F[k] = F2(G0[k], G1[k]);
    } else {
      uniform_force<Q, float>(a, G0);
#pragma unroll
      for (int k = 0; k < 3; ++k) F[k] = F2(G0[k]);
    }
  }
  const Mom<F2> m = moments<Q, F2, FORCE>(d, F, true);
  collide<Q, F2, FORCE>(d, m, F, F2(a.omega), F2(a.guo_c));
  if constexpr (sizeof(S) == 2) {
    const uint32_t s2 =
        sr_pair(sr_seed(c0, m.u[0].v.x, m.u[1].v.x, m.u[2].v.x, m.rd.v.x),
                sr_seed(c1, m.u[0].v.y, m.u[1].v.y, m.u[2].v.y, m.rd.v.y));
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const uint32_t w = sr_two<S>(d[q].v.x, d[q].v.y, s2);
      d[q] = F2(PairT<S>::lo(w), PairT<S>::hi(w));
    }
  }
}

// The pipe node's collide of a lane's two cells (k_prepare's with force mode 3):
// no half-force step in the moments; w0, w1: wall cells.  i0: the cells' plane.
__device__ __forceinline__ void collide_pipe2(const StepArgs& a, uint32_t i0, uint32_t c0,
                                              uint32_t c1, bool w0, bool w1, F2 (&d)[19]) {
  float f0 = 0, f1 = 0;
  if (i0 == a.prop_x) {
    const uint32_t base = i0 * a.g.plane;
    if (__ldg(a.prop_mask + (c0 - base)) != 0) f0 = static_cast<float>(a.force[0]);
    if (__ldg(a.prop_mask + (c1 - base)) != 0) f1 = static_cast<float>(a.force[0]);
  }
  const float gz = static_cast<float>(a.force[2]);
  const F2 F[3] = {F2(f0, f1), F2(0.0f), F2(w0 ? 0.0f : gz, w1 ? 0.0f : gz)};
  const Mom<F2> m = moments<19, F2, true>(d, F, false);
  collide<19, F2, true>(d, m, F, F2(a.omega), F2(a.guo_c));
}

// Population qs of p = C(f) at cell c, from the reference state in global
// memory (zero-gradient faces reach cells outside the buffered planes).
template <int Q, class S, bool FORCE>
__device__ __noinline__ float collided_pop(const StepArgs& a, uint32_t c, int qs) {
  const float* fi = static_cast<const float*>(a.f_in) + static_cast<size_t>(c) * Q;
  float d[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) d[q] = to_offset<Q, float>(__ldg(fi + q), q);
  collide_ref<Q, S, FORCE>(a, c, d);
  float v = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (q == qs) v = d[q];
  return v;
}

// Zero-gradient face of the one-pass step: unknown q <- f_bc of the cell one
// inwards, its pulled (or wall-swapped) population recomputed from f_in.
template <int Q, class S, bool FORCE>
__device__ __forceinline__ void face_zero_gradient_ref(float (&d)[Q], const StepArgs& a, int fi,
                                                       const Cell& x) {
  const Geo& g = a.g;
  const FaceK& fc = a.face[fi];
  const int ax = fc.axis;
  const int st = fc.side == 0 ? 1 : -1;
  const int n0 = static_cast<int>(x.i0) + (ax == 0 ? st : 0);
  const int n1 = static_cast<int>(x.i1) + (ax == 1 ? st : 0);
  const int n2 = static_cast<int>(x.k) + (ax == 2 ? st : 0);
  const bool wl =
      a.wall != nullptr && a.wall[(static_cast<uint32_t>(n0) * g.n1 + n1) * g.n2 + n2] != 0;
  const int s = wl ? 1 : -1;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int cq = comp<Q>(q, ax);
    const bool unknown = fc.side == 0 ? (cq > 0) : (cq < 0);
    if (!unknown) continue;
    const uint32_t j0 = wrapu(n0 + s * Lat<Q>::c0(q), g.n0);
    const uint32_t j1 = wrapu(n1 + s * Lat<Q>::c1(q), g.n1);
    const uint32_t j2 = wrapu(n2 + s * Lat<Q>::c2(q), g.n2);
    d[q] = collided_pop<Q, S, FORCE>(a, (j0 * g.n1 + j1) * g.n2 + j2, wl ? Lat<Q>::opp(q) : q);
  }
}

// Faces `on` of a cell: inlet, then outlet, the zero-gradient neighbour taken
// from the reference state.
template <int Q, class S, bool FORCE>
__device__ __forceinline__ void faces_ref(const StepArgs& a, const Cell& x, uint32_t on,
                                          float (&d)[Q]) {
#pragma unroll
  for (int fi = 0; fi < 2; ++fi) {
    if (!((on >> fi) & 1u)) continue;
    const FaceK& fc = a.face[fi];
    if (fc.kind == kFacePressure) face_pressure<Q, float>(d, a, fi);
    else if (fc.kind == kFaceVelocity) face_velocity<Q, float>(d, a, fi);
    else face_zero_gradient_ref<Q, S, FORCE>(d, a, fi, x);
  }
}
// ... of one of a lane's two cells (HI: the high half).
template <int Q, class S, bool FORCE, bool HI>
__device__ __forceinline__ void faces_ref2(const StepArgs& a, const Cell& x, uint32_t on,
                                           F2 (&d)[Q]) {
  float t[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) t[q] = HI ? d[q].v.y : d[q].v.x;
  faces_ref<Q, S, FORCE>(a, x, on, t);
#pragma unroll
  for (int q = 0; q < Q; ++q) d[q] = HI ? F2(d[q].v.x, t[q]) : F2(t[q], d[q].v.y);
}

// Cell J of a lane's one or two cells.
template <int J>
__device__ __forceinline__ float cell_of(float v) { return v; }
template <int J>
__device__ __forceinline__ float cell_of(F2 v) { return J == 0 ? v.v.x : v.v.y; }

// A wall byte, loaded where the source places it: the collide warps fetch the
// bytes of their cells ahead of the wait for the plane, and a volatile load is
// neither moved towards its use nor repeated there by the compiler.
__device__ __forceinline__ uint8_t ld_wall(const uint8_t* p) {
  uint16_t v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=h"(v) : "l"(p));
  return static_cast<uint8_t>(v);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// try_wait that suspends the thread until the phase completes or about 20 us
// pass (a hint: the hardware may return earlier), so a waiting warp takes few
// issue slots from the working ones.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
      : "memory");
  return ok != 0;
}

// Wait bounded by wall time (limit_ns of the global timer) that also ends when
// another warp of the block has given up (*abort set); a wait that runs out
// sets *abort itself.  Between polls the warp is suspended by the barrier's own
// wait, so it takes few issue slots.
__device__ __forceinline__ bool tile_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns,
                                          volatile int* abort) {
  if (mbar_try_wait_sleep(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 8; ++i)
      if (mbar_try_wait_sleep(bar, parity)) return true;
    if (*abort) return false;
    if (globaltimer_ns() - t0 > limit_ns) break;
  }
  *abort = 1;
  return false;
}

// Place of the current plane in the ring: slot and parity of its barriers.
template <int Q>
struct Ring {
  uint32_t s = 0, par = 0;
  __device__ __forceinline__ void next() {
    if (++s == static_cast<uint32_t>(Sweep<Q>::SLOTS)) {
      s = 0;
      par ^= 1u;
    }
  }
};

// NaN in every output cell of this block's work items: what a block writes whose
// waits ran out, so that an incomplete result shows in the results themselves
// and in what later steps make of them, with no status to ask for.
template <int Q, class S, int MODE>
__device__ __noinline__ void tiled_mark_failed(const StepArgs& a, const TileGeo& t) {
  constexpr int D = Lat<Q>::D;
  const float nan = __uint_as_float(0x7fffffffu);
  PlaneRef p;
  for (uint32_t item = blockIdx.x; item < t.items; item += gridDim.x) {
    plane_first<Q>(a, t, item, p);
    for (uint32_t i = threadIdx.x; i < p.nv * p.tyv * p.tzv; i += blockDim.x) {
      const uint32_t r = i / p.tzv;
      const uint32_t c = (p.k0 + r / p.tyv) * t.SS + (p.y0 + r % p.tyv) * t.SR + p.z0 + i % p.tzv;
      for (int q = 0; q < Q; ++q) {
        if constexpr (MODE == kOutAoS) {
          static_cast<float*>(a.f_out)[static_cast<size_t>(c) * Q + q] = nan;
        } else if constexpr (sizeof(S) == 2) {  // NaN in both 16-bit formats
          static_cast<unsigned short*>(a.pout)[static_cast<uint32_t>(q) * a.g.pstride + c] = 0x7fffu;
        } else {
          static_cast<float*>(a.pout)[static_cast<uint32_t>(q) * a.g.pstride + c] = nan;
        }
      }
      if (a.rho != nullptr) static_cast<float*>(a.rho)[c] = nan;
      if (a.prs != nullptr) static_cast<float*>(a.prs)[c] = nan;
      if (a.vel != nullptr)
        for (int d = 0; d < D; ++d) static_cast<float*>(a.vel)[static_cast<size_t>(c) * D + d] = nan;
    }
  }
}

// PIPE: the pipe node's force (force mode 3), f_bc and moments out, no faces.
// WORDS: no alignment of rows and buffers -- planes come in word by word
// (tiled_issue_words) and f_bc leaves the staging rows by plain stores.
template <int Q, class S, int MODE, bool FACES, bool FORCE, bool PIPE = false, bool WORDS = false>
__global__ void __launch_bounds__(TileShape<Q>::NT, Sweep<Q>::MINB)
    k_tiled(const __grid_constant__ StepArgs a, const __grid_constant__ TileGeo t) {
  using T = TileShape<Q>;
  using R = float;
  static_assert(MODE == kOutAoS || MODE == kOutState, "f_bc out or the next state out");
  static_assert(!PIPE || (Q == 19 && sizeof(S) == 4 && MODE == kOutAoS && !FACES && !FORCE),
                "the pipe node's update");
  constexpr uint32_t S_ = Sweep<Q>::SLOTS;
  static_assert(Sweep<Q>::SLOTS >= 5, "ring depth: three planes read, one collided, one landing");
  extern __shared__ __align__(128) unsigned char smem[];
  float* planes = reinterpret_cast<float*>(smem);
  float* stage = planes + static_cast<size_t>(S_) * T::PLANE;
  TileSync<Q>* sync = reinterpret_cast<TileSync<Q>*>(
      smem + static_cast<size_t>(tiled_idle_word<Q, MODE>() + kIdleWords) * 4);
  volatile int* abort = &sync->abort;
  const Geo& g = a.g;
  const uint32_t tid = threadIdx.x;
  const uint32_t lane = tid & 31u, warp = tid >> 5;

  if (tid == 0) {
    for (uint32_t s = 0; s < S_; ++s) {
      mbar_init(&sync->full[s], WORDS ? 32 : 1);
      mbar_init(&sync->collided[s], T::NCW);
      mbar_init(&sync->consumed[s], T::NOW);
    }
    sync->abort = 0;
    sync->issued = 0;
    fence_mbar_init();
  }
  if (tid < kIdleWords) planes[tiled_idle_word<Q, MODE>() + tid] = 0.0f;
  __syncthreads();

  if (warp == 0) {
    // ---- producer: copy plane P into its slot once the slot's last plane is consumed
    PlaneRef L;
    plane_first<Q>(a, t, blockIdx.x, L);
    Ring<Q> r;
    uint32_t P = 0;
    for (; L.item < t.items; plane_next<Q>(a, t, L), ++P, r.next()) {
      const bool ok =
          P < S_ || tile_wait(&sync->consumed[r.s], r.par ^ 1u, t.wait_ns, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      fence_proxy_async_smem();
      float* buf = planes + static_cast<size_t>(r.s) * T::PLANE;
      if constexpr (WORDS) tiled_issue_words<Q>(a, t, L, buf, &sync->full[r.s], lane);
      else tiled_issue<Q>(a, t, L, buf, &sync->full[r.s], lane);
    }
    if (lane == 0) sync->issued = P;
  } else if (warp <= static_cast<uint32_t>(T::NCW)) {
    // ---- collide warps: plane P in place once it has landed, two cells per
    // lane; the wall bits of its cells go to the plane's words
    const uint32_t j = warp - 1;
    uint32_t rz[2] = {0, 0};
    CollidePlace at[2] = {};
    PlaneRef C;
    plane_first<Q>(a, t, blockIdx.x, C);
    Ring<Q> r;
    uint32_t item = ~0u;
    for (; C.item < t.items; plane_next<Q>(a, t, C), r.next()) {
      if (C.item != item) {  // a new work item: the lane cells' rows and columns
        item = C.item;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint32_t m = (2 * j + k) * 32 + lane;
          at[k] = collide_place<Q, MODE>(m, C.tyv, C.tzv);
          // a lane without a cell takes the index of the plane's first one
          const bool mine = at[k].step != 0;
          const uint32_t ry = mine ? m / T::CW : 0u, cz = mine ? m % T::CW : 0u;
          rz[k] = wrapu(static_cast<int>(C.y0 + ry) - T::HR, t.NR) * t.SR +
                  wrapu(static_cast<int>(C.z0 + cz) - 1, g.n2);
        }
      }
      const uint32_t cs0 = plane_s(t, C) * t.SS;
      uint8_t wb[2] = {0, 0};
      if (a.wall != nullptr) {  // fetched ahead of the wait for the plane
        wb[0] = ld_wall(a.wall + cs0 + rz[0]);
        wb[1] = ld_wall(a.wall + cs0 + rz[1]);
      }
      const bool ok = tile_wait(&sync->full[r.s], r.par, t.wait_ns, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      float* const c0 = planes + (at[0].word + r.s * at[0].step);
      float* const c1 = planes + (at[1].word + r.s * at[1].step);
      // No branch around this body: given one per cell, the compiler splits it
      // by which cells a lane owns and a warp runs it up to three times.
      F2 d[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) d[q] = F2(c0[q], c1[q]);
#pragma unroll
      for (int q = 0; q < Q; ++q) d[q] = to_offset<Q, F2>(d[q], q);
      if constexpr (PIPE)
        collide_pipe2(a, plane_s(t, C), cs0 + rz[0], cs0 + rz[1], wb[0] != 0, wb[1] != 0, d);
      else
        collide_ref2<Q, S, FORCE>(a, cs0 + rz[0], cs0 + rz[1], d);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (at[0].step != 0) c0[q] = d[q].v.x;
        if (at[1].step != 0) c1[q] = d[q].v.y;
      }
      const uint32_t w0 = __ballot_sync(0xffffffffu, wb[0] != 0);
      const uint32_t w1 = __ballot_sync(0xffffffffu, wb[1] != 0);
      fence_proxy_async_smem();  // before the slot is refilled by a copy
      __syncwarp();
      if (lane == 0) {
        sync->wall[r.s][2 * j] = w0;
        sync->wall[r.s][2 * j + 1] = w1;
        mbar_arrive(&sync->collided[r.s]);
      }
    }
  } else {
    // ---- output warps: plane P once P + 1 is collided; one cell (ty, tz) per
    // lane, or two (tz and tz + OZ)
    constexpr bool kTwo = T::CPO == 2;
    using V = typename std::conditional<kTwo, F2, float>::type;
    constexpr int kSA = Lat<Q>::D == 3 ? 0 : 1;  // the internal axis of the sweep
    const uint32_t ow = warp - 1 - T::NCW;
    const uint32_t ty = kTwo ? 0u : ow, tz = (kTwo ? ow * 32 : 0u) + lane;
    float* const wst = stage + static_cast<size_t>(ow) * 32 * T::CPO * Q;  // staging rows
    // the places of its cells among the collided ones (wall bits)
    const uint32_t m0 = (ty + T::HR) * T::CW + tz + 1, m1 = m0 + T::OZ;
    bool act0 = false, act1 = false;  // its cells lie inside the lattice
    uint32_t off = 0, off1 = 0, col = 0, face0 = 0, face1 = 0;
    Cell x{};
    PlaneRef O;
    plane_first<Q>(a, t, blockIdx.x, O);
    Ring<Q> r, rn;  // plane P, plane P + 1
    rn.next();
    uint32_t sm = S_ - 1;  // slot of plane P - 1
    uint32_t item = ~0u;
    for (; O.item < t.items; plane_next<Q>(a, t, O), sm = r.s, r.next(), rn.next()) {
      if (O.item != item) {  // a new work item: the lane cells' column
        item = O.item;
        act0 = ty < O.tyv && tz < O.tzv;
        act1 = kTwo && act0 && tz + T::OZ < O.tzv;
        // A lane without a first cell runs the tile's first one, a lane without a
        // second cell its first one again; neither stores it (no branch around
        // the body, as above).
        const uint32_t tye = act0 ? ty : 0u, tze = act0 ? tz : 0u;
        off = ((tye + T::HR) * T::RW + T::LCH) + tze * Q;
        off1 = act1 ? T::OZ * Q : 0u;
        x.i1 = O.y0 + tye;  // D3Q19; the sweep's own coordinate with D2Q9
        x.k = O.z0 + tze;
        col = (O.y0 + tye) * t.SR + x.k;
        // faces along the axes across the sweep
        face0 = face1 = 0;
        if constexpr (FACES) {
#pragma unroll
          for (int fi = 0; fi < 2; ++fi) {
            const FaceK& fc = a.face[fi];
            if (fc.kind == kFaceNone || fc.axis == kSA) continue;
            const uint32_t last = (fc.axis == 1 ? g.n1 : g.n2) - 1;
            const uint32_t at = fc.side == 0 ? 0u : last;
            if (act0 && (fc.axis == 1 ? x.i1 : x.k) == at) face0 |= 1u << fi;
            if (act1 && x.k + T::OZ == at) face1 |= 1u << fi;
          }
        }
      }
      if (O.j < 1 || O.j > O.nv) continue;
      const bool ok = tile_wait(&sync->collided[rn.s], rn.par, t.wait_ns, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint32_t ps = plane_s(t, O);
      if (Lat<Q>::D == 3) x.i0 = ps;
      else x.i1 = ps;
      x.c = ps * t.SS + col;
      x.row = x.c - x.k;
      x.srow = x.row;
      const uint32_t* wbits = sync->wall[r.s];
      const bool wall0 = act0 && ((wbits[m0 >> 5] >> (m0 & 31u)) & 1u) != 0;
      const bool wall1 = act1 && ((wbits[m1 >> 5] >> (m1 & 31u)) & 1u) != 0;
      V d[Q];
      {
        // the three planes of the pull: x - e_q lies in plane P - c_s(q)
        const float* pm = planes + static_cast<size_t>(sm) * T::PLANE + off;
        const float* p0 = planes + static_cast<size_t>(r.s) * T::PLANE + off;
        const float* pp = planes + static_cast<size_t>(rn.s) * T::PLANE + off;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int cs = Sweep<Q>::cs(q);
          const float* base = (cs > 0 ? pm : (cs < 0 ? pp : p0)) +
                              (-Sweep<Q>::cr(q) * T::RW - Lat<Q>::c2(q) * Q + q);
          if constexpr (kTwo) d[q] = F2(base[0], base[off1]);
          else d[q] = base[0];
        }
      }
      V F[3] = {0, 0, 0};
      if (FORCE) {
        float G0[3], G1[3];
        if (a.force_mode == 2) {
          load_force<Q, float>(a.force_field, x.c, G0);
          if constexpr (kTwo)
            load_force<Q, float>(a.force_field, act1 ? x.c + T::OZ : x.c, G1);
        } else {
          uniform_force<Q, R>(a, G0);
#pragma unroll
          for (int k = 0; k < 3; ++k) G1[k] = G0[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if constexpr (kTwo) F[k] = F2(G0[k], G1[k]);
          else F[k] = G0[k];
        }
      }
      // obstacles are clustered: most warps hold no wall cell
      if (__any_sync(0xffffffffu, wall0 || wall1)) {
        if constexpr (kTwo) {
          wall_swap2<Q>(d, wall0, wall1);
        } else {
#pragma unroll
          for (int q = 1; q < Q; ++q) {
            const int o = Lat<Q>::opp(q);
            if (q > o) continue;
            const float u = d[q], v = d[o];
            d[q] = wall0 ? v : u;
            d[o] = wall0 ? u : v;
          }
        }
      }
      if constexpr (FACES) {
        uint32_t on0 = face0, on1 = face1;
#pragma unroll
        for (int fi = 0; fi < 2; ++fi) {
          const FaceK& fc = a.face[fi];
          if (fc.kind != kFaceNone && fc.axis == kSA && ps == (fc.side == 0 ? 0u : t.NS - 1)) {
            on0 |= 1u << fi;
            on1 |= 1u << fi;
          }
        }
        if (__any_sync(0xffffffffu, (on0 | on1) != 0)) {
          // wall face cells keep the swapped populations
          if constexpr (kTwo) {
            Cell x1 = x;
            x1.k += T::OZ;
            if (act0 && !wall0 && on0) faces_ref2<Q, S, FORCE, false>(a, x, on0, d);
            if (act1 && !wall1 && on1) faces_ref2<Q, S, FORCE, true>(a, x1, on1, d);
          } else if (act0 && !wall0 && on0) {
            faces_ref<Q, S, FORCE>(a, x, on0, d);
          }
          __syncwarp();
        }
      }
      const Mom<V> mo = moments<Q, V, FORCE>(d, F, true);
      if constexpr (MODE == kOutAoS) {
        // this warp's earlier store has read the staging rows
        if (!WORDS && lane == 0) bulk_wait_read();
        __syncwarp();
        float* row = wst + lane * Q;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const V v = from_offset<Q, V>(d[q], q);
          row[q] = cell_of<0>(v);
          if constexpr (kTwo) row[32 * Q + q] = cell_of<1>(v);
        }
        // The warp's cells are prefixes of one or two contiguous runs of the
        // output.  The proxy fence comes before this warp's global stores of the
        // moments, so that it waits only for the staging writes.
        const uint32_t n0 = __popc(__ballot_sync(0xffffffffu, act0));
        const uint32_t n1 = kTwo ? __popc(__ballot_sync(0xffffffffu, act1)) : 0u;
        if constexpr (WORDS) {
          __syncwarp();
          // (lane 0 has the run's first cell where there is one)
          float* out = static_cast<float*>(a.f_out) +
                       static_cast<size_t>(__shfl_sync(0xffffffffu, x.c, 0)) * Q;
#pragma unroll
          for (uint32_t i = 0; i < Q; ++i) {
            const uint32_t w = i * 32 + lane;
            if (w < n0 * Q) out[w] = wst[w];
            if (kTwo && w < n1 * Q) out[T::OZ * Q + w] = wst[32 * Q + w];
          }
          __syncwarp();
        } else {
          fence_proxy_async_smem();
          __syncwarp();
        }
        if (!WORDS && lane == 0 && n0 > 0) {
          float* out = static_cast<float*>(a.f_out) + static_cast<size_t>(x.c) * Q;
          bulk_store2_s2g(out, wst, n0 * Q * 4, out + T::OZ * Q, wst + 32 * Q, n1 * Q * 4);
        }
      }
      if (act0) {
        Mom<R> v0, v1;
        v0.rd = cell_of<0>(mo.rd), v1.rd = cell_of<1>(mo.rd);
        v0.rho = cell_of<0>(mo.rho), v1.rho = cell_of<1>(mo.rho);
#pragma unroll
        for (int k = 0; k < 3; ++k) v0.u[k] = cell_of<0>(mo.u[k]), v1.u[k] = cell_of<1>(mo.u[k]);
        store_moments<Q, float>(a, x.c, v0, wall0);
        if (act1) store_moments<Q, float>(a, x.c + T::OZ, v1, wall1);
        if constexpr (MODE == kOutState) {
          collide<Q, V, FORCE>(d, mo, F, static_cast<V>(a.omega), static_cast<V>(a.guo_c));
          S* out = static_cast<S*>(a.pout) + x.c;
          if constexpr (sizeof(S) == 2) {
            const uint32_t s2 = sr_pair(sr_seed(x.c, v0.u[0], v0.u[1], v0.u[2], v0.rd),
                                        sr_seed(x.c + T::OZ, v1.u[0], v1.u[1], v1.u[2], v1.rd));
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              S* o = out + static_cast<uint32_t>(q) * g.pstride;
              if constexpr (kTwo) {
                const uint32_t w = sr_two<S>(cell_of<0>(d[q]), cell_of<1>(d[q]), s2);
                reinterpret_cast<unsigned short*>(o)[0] = static_cast<unsigned short>(w & 0xffffu);
                if (act1)
                  reinterpret_cast<unsigned short*>(o)[T::OZ] = static_cast<unsigned short>(w >> 16);
              } else {
                o[0] = sr_one<S>(d[q], sr_bits(s2, d[q]));
              }
            }
          } else {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              S* o = out + static_cast<uint32_t>(q) * g.pstride;
              o[0] = cell_of<0>(d[q]);
              if (act1) o[T::OZ] = cell_of<1>(d[q]);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) {
        // plane P - 1 has had its last reader; at the end of an item, P and P + 1 too
        mbar_arrive(&sync->consumed[sm]);
        if (O.j == O.nv) {
          mbar_arrive(&sync->consumed[r.s]);
          mbar_arrive(&sync->consumed[rn.s]);
        }
      }
    }
    if constexpr (MODE == kOutAoS && !WORDS) {
      if (lane == 0) bulk_wait_all();
    }
  }

  // (the warp that gave up sees its own flag, so every thread learns of it here)
  if (__syncthreads_or(*abort)) {
    if (tid == 0) {
      atomicOr(a.status, 1);
      // the last copies issued may be in flight: wait for them (bounded) before exit
      sync->abort = 0;
      const uint32_t n = sync->issued;
      for (uint32_t P = n > S_ ? n - S_ : 0; P < n; ++P)
        if (!tile_wait(&sync->full[P % S_], (P / S_) & 1u, t.wait_ns, abort)) break;
    }
    tiled_mark_failed<Q, S, MODE>(a, t);
  }
}

}  // namespace lbm
