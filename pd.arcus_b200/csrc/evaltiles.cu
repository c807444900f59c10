// One GB evaluation on the cluster-pair tiles.
//
// FF_GeneralizedBorn_Still::calcForces in FastMode (gbff.cpp:168-180) has
// three passes over the pairs with a global dependency between each:
//   A  Born-radius sums (calcBornRadii_PairwiseApprox, gbff.cpp:415-466);
//      every pair term must be in before a radius can be formed
//   B  GB + LJ + Coulomb (calcForcesIncludingVacuo loop 1, :1529-1736);
//      needs every radius, and leaves each atom's dE/da complete only when
//      every pair is in
//   C  Born-radius chain rule (loop 2, :1751-1818); needs every dE/da.
// They run as three launches of persistent grids, each a dependent launch
// that loads its first tiles' older records before it waits for the phase
// before, or as the phases of one cooperative launch (every block resident)
// with two grid barriers (pdgpu_eval_mode 1).  The per-atom steps between
// them are folded into the phases: phase B forms each atom's Born radius
// from its fixed-point sum when it stages the atom (the FP64 expression of
// k_born_finish, so the same bits), and phase C forms each atom's chain
// weight gpi * dE/da the same way.  The per-atom outputs (Born radii, the
// per-atom energies) are written by grid-stride epilogues that nothing in
// the same phase reads.
//
// Every phase has its own build (the template's PH), because what bounds the
// phases includes fetching their instructions: the one kernel that held all
// three was 126 KB of code, a warp of a small system runs each part of it
// once per launch, and a quarter of its stalls were on instruction fetch
// (ncu, 985 atoms).  The builds are 32, 55 and 43 KB and get the registers
// their phase needs (no spills in A and B).  Measured, one launch of all
// three / three launches of it / three builds: MD at 20,566 atoms - / 65.4 /
// 63.8 us a step, 64 OPLS peptides - / 219 / 212 us a step; a call of
// pdgpu_calc_forces 52 / 49 / 46 us at 985 atoms, 92 / - / 82 at 20,566,
// 907 / - / 888 for 512 peptides.  So every caller uses the three launches;
// the cooperative form stays for callers that ask for it.
//
// Every warp keeps one contiguous tile range for phases A and B (an equal
// share of the pack's tiles).  Phase A also notes the tiles that hold a
// pair inside the Still cutoff (within the guard band); phase C runs over
// that compacted list only, in equal shares.  As in the separate passes
// (tiles.cu), a tile's sums depend on the tile alone and are added in
// 64-bit fixed point, so results do not depend on how the tiles are spread
// over warps, on the grid, or on the batch a system sits in.
//
// The barriers spin with a bounded number of naps; a barrier that runs out
// sets F_BARRIER, and every block then returns (the host reports it and
// clears the counter).  PDGPU_FUSED=0 turns the cooperative form off.
//
// Pair arithmetic: the phase-A Born terms are those of the row and tile
// passes (born_term_noV, explicit roundings: the same Born radii bit for
// bit); phases B and C follow gb_pair_term and chain_term with every
// selection branch-free except the GB cross term and the rare FP64
// re-decisions.  The j records of a tile are stored twice in shared memory
// (slots 0-7 and 8-15) so lane a reads j atom (a + t) mod 8 at slot a + t
// with a fixed offset per step.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "tilecommon.cuh"

namespace pdgpu {

constexpr int kEvWarps = 4;  // warps per block
// resident blocks per SM the register allocation must allow (up to 128
// registers a thread).  With five for phases A and C 64 OPLS peptides ran 1 %
// faster a step and 985 atoms 1.4 % slower; with six or eight every size was
// slower, phase B with five 6 % slower.
constexpr int kEvBlocks = 4;
constexpr unsigned kBarrierNaps = 1u << 22;  // about half a second of 100 ns naps

// ------------------------------------------------------------- barrier
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned x;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
  return x;
}
// The wait of a programmatic dependent launch: every earlier kernel of the
// stream has completed and its memory is visible; then the next kernel may
// be scheduled (PDGPU_DEP_ENTRY's two steps, after a launch's static loads).
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Grid barrier over a counter that counts arrivals; every block waits for
// `target` arrivals.  False when the wait ran out (the flag is set).  The
// arrival releases what the block wrote (ordered before it by the block
// barrier) and returns nothing, and a poll that sees the target acquires what
// the others wrote: the last block to arrive passes after one poll (2,700
// cycles with fences around an atomic that returned its value, 2,000 now).
__device__ __forceinline__ bool grid_barrier(unsigned *ctr, unsigned target, int *flags) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    int ok = 1;
    unsigned naps = 0;
    while (ld_acquire_u32(ctr) < target) {
      if (++naps > kBarrierNaps) {
        ok = 0;
        atomicExch(&flags[F_BARRIER], 1);
        break;
      }
      if (naps > 64) __nanosleep(100);  // (a phase's tail is short: the first polls are back to back)
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// Blocks of the launch that take part: one warp per tile at most, enough
// threads for one atom each.  The grid is sized for the pack's worst case
// (1,984 warps at 985 atoms, which has 347 tiles); the blocks past the active
// ones leave at once, so the barriers and the exit count fewer arrivals.
__device__ __forceinline__ int ev_active(const PackView &v) {
  const int need = max((v.tile_count[0] + kEvWarps - 1) / kEvWarps, (v.n_atoms + 32 * kEvWarps - 1) / (32 * kEvWarps));
  return min((int)gridDim.x, max(need, 1));
}
// This warp's share [e0, e1) of T work items, over `blocks` blocks.
__device__ __forceinline__ void ev_range(long long T, int blocks, int warp, int &e0, int &e1) {
  const long long G = (long long)blocks * kEvWarps;
  const long long g = (long long)blockIdx.x * kEvWarps + warp;
  e0 = (int)(T * g / G);
  e1 = (int)(T * (g + 1) / G);
}

// Born radius of atom i from its fixed-point sum (k_born_finish's FP64
// expression, gbff.cpp:463-465).
__device__ __forceinline__ double born_radius(const PackView &v, const SysParams &P, int i) {
  const double Gpol = v.terms123[i] + (double)v.bsum[i] * kInvBornScale;
  return -P.halfeconv_d / Gpol + P.born_offset_d;
}

// A lane's bond-order rows rotated so bit t is j atom (a + t) mod 8.
__device__ __forceinline__ unsigned rot8(unsigned row, int a) {
  row &= 0xffu;
  return ((row >> a) | (row << (8 - a))) & 0xffu;
}

// Tile staging shared by the phases: the tile's metadata, this lane's row
// bits and bond-order rows and, in lanes 0..7, the j atom's records and the
// per-atom inputs the phase forms from them.  Records are loaded one tile
// ahead of their use and the metadata two tiles ahead (the records' address
// depends on it), so no tile waits for a load chain.
struct EvStage {
  int4 m;
  unsigned row, x0, x1;  // list bits; bond order <= 2 rows; == 3 rows
  float4 a, b, c;
  double u;              // phase B: terms123[j]; phase C: born_d[j]
  long long w;           // phase B: bsum[j]; phase C: the dE/da sum of j
};
// PH: the phase (1 A, 2 B, 4 C) the stage is for.  The static part reads
// only what the list build and the integrator wrote (the tile records,
// coordinates, per-atom parameters); the dynamic part what the evaluation's
// earlier phases wrote (the Born sums; the Born radii and dE/da sums).
// (Of the static part, what the integrator did not write comes first: phase A
// of a step without a rebuild reads that much before its wait.)
template <int PH>
__device__ __forceinline__ void ev_stage_old(const PackView &v, int t, int lane, EvStage &q) {
  q.row = tile_row(v, t, lane);
  q.x0 = q.x1 = 0;
  if (q.m.y >= 0) {
    q.x0 = spec_row(v, q.m.y, 0, lane);
    if (PH == 2) q.x1 = spec_row(v, q.m.y, 1, lane);
  }
  if (lane <= (q.m.w & 7)) {
    const int j = q.m.x + lane;
    q.c = v.prm[j];
    if (PH == 2) q.u = v.terms123[j];
  }
}
__device__ __forceinline__ void ev_stage_xyz(const PackView &v, int lane, EvStage &q) {
  if (lane <= (q.m.w & 7)) {
    const int j = q.m.x + lane;
    q.a = v.pq[2 * (size_t)j];
    q.b = v.pq[2 * (size_t)j + 1];
  }
}
template <int PH>
__device__ __forceinline__ void ev_stage_dyn(const PackView &v, int lane, EvStage &q) {
  if (lane <= (q.m.w & 7)) {
    const int j = q.m.x + lane;
    if (PH == 2) q.w = v.bsum[j];
    if (PH == 4) {
      q.u = v.born_d[j];
      q.w = v.ej[(size_t)3 * v.n_atoms + j];
    }
  }
}
template <int PH>
__device__ __forceinline__ void ev_stage(const PackView &v, int t, int lane, EvStage &q) {
  ev_stage_old<PH>(v, t, lane, q);
  ev_stage_xyz(v, lane, q);
  ev_stage_dyn<PH>(v, lane, q);
}
// Walks a warp's tiles [e, e1) (PH 1, 2) or still-list entries (PH 4) with
// the two-deep prefetch: next() returns the stage of the current tile and
// its index, and issues the loads for the tiles after it.  The start is in
// parts: the loads of the first items that a launch may issue before the
// launches before it are done, then the rest of the first item's stage.
template <int PH>
struct EvWalk {
  int e, e1;
  int t0, t1, t2;  // tiles of items e, e+1, e+2
  int4 m1;         // metadata of item e+1
  EvStage nx;      // stage of item e
  __device__ __forceinline__ int tile_of(const PackView &v, int k) const {
    return PH == 4 ? v.still_list[k] : k;
  }
  __device__ __forceinline__ void start_old(const PackView &v, int lane, int b, int end) {
    e = b;
    e1 = end;
    t0 = t1 = t2 = 0;
    if (e < e1) {
      t0 = tile_of(v, e);
      nx.m = v.tile_meta[t0];
      ev_stage_old<PH>(v, t0, lane, nx);
    }
    if (e + 1 < e1) {
      t1 = tile_of(v, e + 1);
      m1 = v.tile_meta[t1];
    }
    if (e + 2 < e1) t2 = tile_of(v, e + 2);
  }
  __device__ __forceinline__ void start_xyz(const PackView &v, int lane) {
    if (e < e1) ev_stage_xyz(v, lane, nx);
  }
  __device__ __forceinline__ void start_dyn(const PackView &v, int lane) {
    if (e < e1) ev_stage_dyn<PH>(v, lane, nx);
  }
  // the current item's stage and tile; advances the prefetch by one item
  __device__ __forceinline__ EvStage next(const PackView &v, int lane, int &tile) {
    const EvStage cur = nx;
    tile = t0;
    if (e + 1 < e1) {
      nx.m = m1;
      ev_stage<PH>(v, t1, lane, nx);
    }
    if (e + 2 < e1) m1 = v.tile_meta[t2];
    t0 = t1;
    t1 = t2;
    if (e + 3 < e1) t2 = tile_of(v, e + 3);
    e++;
    return cur;
  }
};
// One tile staged on its own (the deferred tiles' second pass).
template <int PH>
__device__ __forceinline__ EvStage ev_stage_one(const PackView &v, int t, int lane) {
  EvStage q;
  q.m = v.tile_meta[t];
  ev_stage<PH>(v, t, lane, q);
  return q;
}

// A tile with a pair at a decision edge (the Still cutoff's, or the
// exp-approximation range's) is not added in a phase's main loop: its index
// goes to the warp's slots of defer_list ([first, first + n) for a warp
// whose items start at `first`), and the warp redoes those tiles in the
// careful form after its main loop, adding their sums then.  A tile's
// result therefore depends on the tile alone, and the main loop carries
// neither the FP64 decisions nor the registers they need.
__device__ __forceinline__ void defer_tile(const PackView &v, int lane, int first, int &n, int t) {
  if (lane == 0) v.defer_list[first + n] = t;
  n++;
}

// ============================================================= phase A
// Born sums.  Each term is converted to fixed point and added exactly
// (the row and tile passes' arithmetic).  Tiles with a pair inside the
// Still cutoff's guard band are appended to the still list in runs of up
// to 32 (per-warp order inside a run).
//
// One tile's terms: the i side's sum (this lane's i atom) and the j side's
// (lane (g,a): j atom a, this group's i atoms).  A pair in the guard band
// of the Still cutoff is decided by its FP64 distance: the fast form
// (CAREFUL false) leaves such pairs out and reports them in `band`, and the
// caller then redoes the tile in the careful form, which decides them; a
// tile's result therefore depends on the tile alone.
// The FP64 inputs of the guard-band decisions (passed by value to the
// careful forms, which are out of line).
struct ExactIn {
  const double *x, *y, *z;
  const double *terms123;
  const long long *bsum;
};
__device__ __forceinline__ ExactIn exact_in(const PackView &v) {
  ExactIn x;
  x.x = v.x;
  x.y = v.y;
  x.z = v.z;
  x.terms123 = v.terms123;
  x.bsum = v.bsum;
  return x;
}
struct BornTileIn {
  float4 ia, ib;
  float Ri, Vi, s_lo, s_hi, invP5, piP5, P4s;
  double still2_d;
  int i, b0;
};
struct BornTileOut {
  long long tile_i, jacc;
  bool any;
};
// born_term_noV's value with every step taken on every lane and the
// results selected (the same bits; no divergent branches, so the eight
// steps of a tile interleave).
__device__ __forceinline__ float born_term_sel(const Dx &d, float Ri, float Rj, float invP5, float piP5,
                                               float P4scaled) {
  const float Rs = __fadd_rn(Ri, Rj);
  const float ir2 = __fdividef(1.f, d.r2);
  const float term = __fmul_rn(__fmul_rn(P4scaled, ir2), ir2);
  const float rdivR = __fdividef(d.r2, __fmul_rn(Rs, Rs));
  const float sh = __sinf(__fmul_rn(__fmul_rn(0.5f, piP5), rdivR));
  const float c = __fmul_rn(sh, sh);
  const float tc = __fmul_rn(term, __fmul_rn(c, c));
  return rdivR > invP5 ? term : tc;
}
template <bool CAREFUL>
__device__ __forceinline__ BornTileOut born_tile(const ExactIn &v, const BornTileIn &q, const float4 *sA,
                                                 const float4 *sB, const float4 *sC, unsigned rows, int a, int g8,
                                                 bool &band) {
  long long tile_i = 0, jacc = 0;
  bool any = false;
#pragma unroll(CAREFUL ? 1 : 8)
  for (int t = 0; t < 8; t++) {
    const bool row = (rows >> t) & 1u;
    const float4 ja = sA[a + t], jb = sB[a + t], jc = sC[a + t];
    const Dx d = diff(q.ia, q.ib, ja, jb);
    bool ok = row && d.r2 <= q.s_lo;
    const bool edge = row && !(d.r2 <= q.s_lo) && d.r2 <= q.s_hi;
    if (CAREFUL) {
      if (edge) {
        const int j = q.b0 + ((a + t) & 7), i = q.i;
        ok = !(ref_d2(v.x[i], v.y[i], v.z[i], v.x[j], v.y[j], v.z[j]) > q.still2_d);
      }
    } else {
      band |= edge;
    }
    any |= row && d.r2 <= q.s_hi;
    const float term = born_term_sel(d, q.Ri, jc.x, q.invP5, q.piP5, q.P4s);
    // the j side's term is made fixed point by the lane that owns j (the same bits)
    const float tJ = ok ? __fmul_rn(term, q.Vi) : 0.f;
    tile_i += __float2ll_rn(ok ? __fmul_rn(term, jc.y) : 0.f);
    jacc += __float2ll_rn(t == 0 ? tJ : __shfl_sync(0xffffffffu, tJ, g8 | ((a - t) & 7)));
  }
  BornTileOut o;
  o.tile_i = tile_i;
  o.jacc = jacc;
  o.any = any;
  return o;
}
// The i-side inputs of atom i of the tile's i-cluster (this lane's): the
// parameters, then the position.
__device__ __forceinline__ void born_i_old(const PackView &v, const TileInfo &ti, int lane, BornTileIn &q) {
  q.i = ti.a0 + (lane < ti.na ? lane : 0);
  const float4 pi = v.prm[q.i];
  q.Ri = pi.z;
  q.Vi = pi.w;
  const SysParams &P = v.sp[ti.s];
  q.s_hi = P.still2 * (1.f + 4e-6f);
  q.s_lo = P.still2 * (1.f - 4e-6f);
  q.invP5 = P.invP5;
  q.piP5 = P.piP5;
  q.P4s = P.P4 * (float)kBornScale;
  q.still2_d = P.still2_d;
}
__device__ __forceinline__ void born_i_xyz(const PackView &v, BornTileIn &q) {
  q.ia = v.pq[2 * (size_t)q.i];
  q.ib = v.pq[2 * (size_t)q.i + 1];
}
// A tile's j records into this warp's slots.
__device__ __forceinline__ void born_stage_j(const TileInfo &ti, const EvStage &cur, int lane, float4 *sA,
                                             float4 *sB, float4 *sC) {
  if (lane < ti.nb) {
    sA[lane] = sA[lane + 8] = cur.a;
    sB[lane] = sB[lane + 8] = cur.b;
    sC[lane] = sC[lane + 8] = make_float4(cur.c.z, cur.c.w, 0.f, 0.f);
  }
}
// The j side's sums of a tile over the i groups, added to the Born sums.
__device__ __forceinline__ void born_add_j(const PackView &v, const TileInfo &ti, int lane, long long jacc) {
  jacc += __shfl_xor_sync(0xffffffffu, jacc, 8);
  jacc += __shfl_xor_sync(0xffffffffu, jacc, 16);
  if (lane < ti.nb && jacc) atomicAdd((unsigned long long *)&v.bsum[ti.b0 + lane], (unsigned long long)jacc);
}

// `wait` runs after the loads of what is older than the launch before (with
// ZF_OLD_TILES: the tiles and the parameters).
template <class Wait>
__device__ __forceinline__ void phase_born(const PackView &v, int blocks, int warp, int lane, float4 (*sA)[16],
                                           float4 (*sB)[16], float4 (*sC)[16], Wait wait) {
  int e, e1;
  ev_range(v.tile_count[0], blocks, warp, e, e1);
  const int first = e;
  const int g8 = lane & ~7, a = lane & 7;
  int a0 = -1, na = 0, nd = 0;
  BornTileIn q;
  q.ia = q.ib = make_float4(0, 0, 0, 0);
  q.Ri = q.Vi = q.s_lo = q.s_hi = q.invP5 = q.piP5 = q.P4s = 0.f;
  q.still2_d = 0.0;
  q.i = 0;
  long long acc_i = 0;
  unsigned near = 0;
  int run0 = e;
  const ExactIn xin = exact_in(v);
  EvWalk<1> walk;
  walk.start_old(v, lane, e, e1);
  if (e < e1) {
    const TileInfo ti = tile_info(walk.nx.m);
    born_i_old(v, ti, lane, q);
    a0 = ti.a0;
    na = ti.na;
  }
  wait();
  walk.start_xyz(v, lane);
  if (e < e1) born_i_xyz(v, q);
  auto flush_near = [&](int upto) {
    // tiles [run0, upto) with their bits in `near`
    const int cnt = __popc(near);
    if (cnt) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&v.tile_count[2], cnt);
      base = __shfl_sync(0xffffffffu, base, 0);
      if ((near >> lane) & 1u) v.still_list[base + __popc(near & ((1u << lane) - 1u))] = run0 + lane;
    }
    near = 0;
    run0 = upto;
  };
#pragma unroll 1
  for (; e < e1; e++) {
    int te;
    const EvStage cur = walk.next(v, lane, te);
    const TileInfo ti = tile_info(cur.m);
    if (ti.a0 != a0) {
      if (lane < na && acc_i) atomicAdd((unsigned long long *)&v.bsum[a0 + lane], (unsigned long long)acc_i);
      acc_i = 0;
      a0 = ti.a0;
      na = ti.na;
      born_i_old(v, ti, lane, q);
      born_i_xyz(v, q);
    }
    q.b0 = ti.b0;
    born_stage_j(ti, cur, lane, sA[warp], sB[warp], sC[warp]);
    const unsigned rows = rot8(cur.row & ~cur.x0, a);  // bond order > 2 only
    __syncwarp();
    bool band = false;  // a pair whose inclusion the FP64 distance decides
    const BornTileOut o = born_tile<false>(xin, q, sA[warp], sB[warp], sC[warp], rows, a, g8, band);
    // a pair inside the Still cutoff's guard band: the tile goes to the chain-rule phase
    const bool any = __any_sync(0xffffffffu, o.any);
    if (any) near |= 1u << (e - run0);
    if (__any_sync(0xffffffffu, band)) {
      defer_tile(v, lane, first, nd, e);
    } else {
      acc_i += o.tile_i;
      if (any) born_add_j(v, ti, lane, o.jacc);  // no pair inside the cutoff: no j terms
    }
    if (e - run0 == 31) flush_near(e + 1);
    __syncwarp();
  }
  if (lane < na && acc_i) atomicAdd((unsigned long long *)&v.bsum[a0 + lane], (unsigned long long)acc_i);
  flush_near(e1);
  if (v.defer_stats && lane == 0 && nd) atomicAdd(&v.defer_stats[0], nd);
  // the deferred tiles in the careful form
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < nd; k++) {
    const int t = v.defer_list[first + k];
    const EvStage cur = ev_stage_one<1>(v, t, lane);
    const TileInfo ti = tile_info(cur.m);
    born_i_old(v, ti, lane, q);
    born_i_xyz(v, q);
    q.b0 = ti.b0;
    born_stage_j(ti, cur, lane, sA[warp], sB[warp], sC[warp]);
    const unsigned rows = rot8(cur.row & ~cur.x0, a);
    __syncwarp();
    bool band = false;
    const BornTileOut o = born_tile<true>(xin, q, sA[warp], sB[warp], sC[warp], rows, a, g8, band);
    if (lane < ti.na && o.tile_i) atomicAdd((unsigned long long *)&v.bsum[q.i], (unsigned long long)o.tile_i);
    born_add_j(v, ti, lane, o.jacc);
    __syncwarp();
  }
}

// ============================================================= phase B
// GB + LJ + Coulomb for one pair (gb_pair_term's expressions), every
// output zero unless `in`.  Selections are branch-free except the GB cross
// term (skipped by a warp with no pair inside the exp-approximation range)
// and the FP64 re-decision of that range's edge.
struct PairOut {
  float fscal, epol, dedal, vdw, elec;
};
// The exp-approximation range's edge is decided by the FP64 predicate: the
// fast form (CAREFUL false) takes the FP32 decision and reports a pair
// inside the edge's guard band in `band` (the caller then redoes the tile
// in the careful form).
// LEAN: every system of the pack runs FastMode and switches LJ with the
// GB/Coulomb switch (the same parameters, so the same values): the slow
// branch and the second switch are left out.  Both builds give the same
// bits for such a system.
template <bool CAREFUL, bool LEAN>
__device__ __forceinline__ PairOut pair_gb(const GbSettings &g, float r2, bool in, bool nb, bool b14, float ai,
                                           float aj, float qiqj, float radsum, float epsij, const ExactIn &v,
                                           int i, int j, double ai_d, const SysParams *P, bool &band) {
  const float invr = rsqrtf(r2);
  const float r = r2 * invr;
  const float aiaj = ai * aj;
  const float u = __fdividef(-0.25f * r2, aiaj);
  bool gb = u > g.thr;
  const bool edge = in && fabsf(u - g.thr) <= g.band;
  if (CAREFUL) {
    if (edge) {
      // the FP64 predicate of gbff.cpp:1553-1575 with both radii formed
      // from their sums (the same values the epilogue stores)
      const double aj_d = -P->halfeconv_d / (v.terms123[j] + (double)v.bsum[j] * kInvBornScale) + P->born_offset_d;
      const double srij = ref_d2(v.x[i], v.y[i], v.z[i], v.x[j], v.y[j], v.z[j]);
      gb = -srij * 0.25 / (ai_d * aj_d) > g.thr_d;
    }
  } else {
    band |= edge;
  }
  gb = gb && in;
  const float dr = r - g.rin;
  const bool on = r >= g.rin;
  const float sw = 1.f - g.inv_sw2 * dr * dr;
  const float S = on ? sw * sw : 1.f;
  const float dSdd = on ? -4.f * g.inv_sw2 * dr * sw : 0.f;
  float dedr = 0.f, epol = 0.f, dedal = 0.f;
  if (gb) {
    const float tg = __expf(u);
    const float fgb = rsqrtf(r2 + tg * aiaj);
    const float l = fgb * fgb;
    const float epol0 = g.premul * qiqj * fgb;
    const float dedr0 = -epol0 * (r - 0.25f * r * tg) * l;
    const float dedal0 = -epol0 * tg * (1.f - u) * l;
    epol = epol0 * S;
    dedr = S * dedr0 + dSdd * epol0;
    dedal = dedal0 * S;
  } else if (!LEAN && g.slow && in) {
    // FastMode off (calcBornForces, gbff.cpp:1292-1324): the GB term's
    // t = 0 limit q_i q_j / r beyond the exp-approximation range
    const float epol0 = g.premul * qiqj * invr;
    epol = epol0 * S;
    dedr = S * (-epol0 * invr) + dSdd * epol0;
  }
  if (!LEAN) nb = nb && !g.slow;  // FastMode off: the vacuum terms come from FF_NonBonded::calcForces
  const float ec = (gb ? g.econv_in : g.econv_out) * (b14 ? g.elec14 : 1.f) * qiqj * invr;
  const float elf = S * (-ec * invr) + ec * dSdd;
  // Lennard-Jones 12-6 with its own switch
  const float rr = radsum * invr;
  const float rr2 = rr * rr;
  const float B = rr2 * rr2 * rr2;
  const float A = B * B;
  const float eps = epsij * (b14 ? g.vdw14 : 1.0f);
  float vdw = (2.f * eps) * (0.5f * A - B);
  float vdwf = -(12.f * eps * invr) * (A - B);
  float vS = S, vdS = dSdd;
  if (!LEAN) {
    const float vd = r - g.vdw_rin;
    const float vs = 1.f - g.vdw_inv_sw2 * vd * vd;
    const bool von = r > g.vdw_rin;
    vS = von ? vs * vs : 1.f;
    vdS = von ? -4.f * g.vdw_inv_sw2 * vd * vs : 0.f;
  }
  vdwf = vS * vdwf + vdw * vdS;
  vdw *= vS;
  const bool lj = in && nb && r < g.vdw_rc;
  const bool el = in && nb;
  vdw = lj ? vdw : 0.f;
  vdwf = lj ? vdwf : 0.f;
  PairOut o;
  o.elec = el ? ec * S : 0.f;
  const float fel = el ? elf : 0.f;
  o.fscal = in ? dedr * 2.f * invr + (vdwf + fel) * invr : 0.f;
  o.epol = epol;
  o.dedal = dedal;
  o.vdw = vdw;
  return o;
}

// The i side of a tile is converted to fixed point per tile (so its sums
// depend on the tile alone) and kept in this lane's shared-memory slots
// while the warp's range stays in one i-cluster; the sums go to memory when
// the range moves to the next cluster.  Exact integer sums: the same bits
// as adding every tile's share to memory at once.
struct ISide {
  long long (*f)[32];  // [7][32]: this warp's slots
  int lane;
  bool bad;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int q = 0; q < 7; q++) f[q][lane] = 0;
    bad = false;
  }
  __device__ __forceinline__ void add(int q, float x) {
    bad |= !(fabsf(x) <= 3.0e38f);
    f[q][lane] += to_fixed_j(x);
  }
  __device__ __forceinline__ void flush(const PackView &v, int i, int N) {
    long long *dst[7] = {v.hx + i, v.hy + i, v.hz + i, v.ej + i, v.ej + (size_t)N + i, v.ej + (size_t)2 * N + i,
                         v.ej + (size_t)3 * N + i};
#pragma unroll
    for (int q = 0; q < 7; q++) {
      const long long x = f[q][lane];
      if (x) atomicAdd((unsigned long long *)dst[q], (unsigned long long)x);
    }
  }
};
// A non-finite partial (coincident atoms) marks its system.
__device__ __forceinline__ void flush_bad(const PackView &v, bool bad, int s) {
  if (bad) atomicOr(&(v.ebuf ? v.sys_flags_alt : v.sys_flags)[s], SF_NONFINITE);
}

// One tile's GB + LJ + Coulomb terms: the i side's sums of this lane's i
// atom (io: force x, y, z, vdw, elec, pol, dE/da) and the j side's (jo,
// lane (g,a): j atom a, this group's i atoms, before the sum over groups).
struct PairTileIn {
  float4 ia, ib, ip;
  double ai_d;
  int i, b0;
};
struct PairTileOut {
  float io[7], jo[7];
};
template <bool CAREFUL, bool LEAN>
__device__ __forceinline__ PairTileOut pair_tile(const ExactIn &v, const GbSettings &gs, const SysParams *P,
                                                 const PairTileIn &q, const float4 *sA, const float4 *sB,
                                                 const float4 *sP, unsigned rows, unsigned xrows, unsigned brows,
                                                 int a, int g8, bool &band) {
  float io[7], jo[7];
#pragma unroll
  for (int k = 0; k < 7; k++) io[k] = jo[k] = 0.f;
#pragma unroll(CAREFUL ? 1 : 8)
  for (int t = 0; t < 8; t++) {
    const float4 ja = sA[a + t], jb = sB[a + t], jp = sP[a + t];
    const Dx d = diff(q.ia, q.ib, ja, jb);
    const bool in = ((rows >> t) & 1u) && d.r2 <= gs.rc2;
    const bool nb3 = !((xrows >> t) & 1u);
    const bool b14 = (brows >> t) & 1u;
    const PairOut o = pair_gb<CAREFUL, LEAN>(gs, d.r2, in, nb3, b14, q.ib.w, jb.w, q.ia.w * ja.w, q.ip.x + jp.x,
                                       q.ip.y * jp.y, v, q.i, q.b0 + ((a + t) & 7), q.ai_d, P, band);
    io[5] += o.epol;
    io[6] += o.dedal * jb.w;
    io[3] += o.vdw;
    io[4] += o.elec;
    const float cx = o.fscal * d.x, cy = o.fscal * d.y, cz = o.fscal * d.z;
    io[0] -= cx;
    io[1] -= cy;
    io[2] -= cz;
    const float c[7] = {cx, cy, cz, o.vdw, o.elec, o.epol, o.dedal * q.ib.w};
    // (at t = 0 the source is this lane; plain additions, never contracted
    // with the product a term may be)
    const int src = g8 | ((a - t) & 7);
#pragma unroll
    for (int k = 0; k < 7; k++) jo[k] = __fadd_rn(jo[k], t == 0 ? c[k] : __shfl_sync(0xffffffffu, c[k], src));
  }
  PairTileOut o;
#pragma unroll
  for (int k = 0; k < 7; k++) {
    o.io[k] = io[k];
    o.jo[k] = jo[k];
  }
  return o;
}
// The i-side inputs of this lane's atom of the tile's i-cluster: what the
// list build and the integrator wrote (with the fixed Born terms, kept in
// ai_d), then the Born radius from the sum of the earlier phase.
__device__ __forceinline__ void pair_i_static(const PackView &v, const TileInfo &ti, int lane, PairTileIn &q) {
  q.i = ti.a0 + (lane < ti.na ? lane : 0);
  q.ia = v.pq[2 * (size_t)q.i];
  q.ib = v.pq[2 * (size_t)q.i + 1];
  q.ip = v.prm[q.i];
  q.ai_d = v.terms123[q.i];
}
__device__ __forceinline__ void pair_i_dyn(const PackView &v, double hec, double boff, PairTileIn &q) {
  // k_born_finish's expression (born_radius; hec is -halfeconv)
  q.ai_d = hec / (q.ai_d + (double)v.bsum[q.i] * kInvBornScale) + boff;
  q.ib.w = (float)q.ai_d;
}
// A tile's j records into this warp's slots, with each j atom's Born
// radius formed from its staged sum: -halfeconv / G + offset with 1/G from
// the FP32 reciprocal and one Newton step in FP64 (about 48 bits, so the
// FP32 radius is born_radius's rounded in all but tie cases; decisions at
// the exp-approximation edge use the FP64 radii themselves).
__device__ __forceinline__ void pair_stage_j(const TileInfo &ti, const EvStage &cur, int lane, double hec,
                                             double boff, float4 *sA, float4 *sB, float4 *sP) {
  if (lane < ti.nb) {
    float4 b = cur.b;
    const double G = cur.u + (double)cur.w * kInvBornScale;
    const double r0 = (double)__frcp_rn((float)G);
    const double r1 = fma(r0, fma(-G, r0, 1.0), r0);
    b.w = (float)fma(hec, r1, boff);
    sA[lane] = sA[lane + 8] = cur.a;
    sB[lane] = sB[lane + 8] = b;
    sP[lane] = sP[lane + 8] = cur.c;
  } else if (lane < 8) {
    // a j-cluster shorter than 8 atoms: its empty slots hold zero records,
    // so the masked-out terms of those slots multiply finite numbers
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    sA[lane] = sA[lane + 8] = z;
    sB[lane] = sB[lane + 8] = z;
    sP[lane] = sP[lane + 8] = z;
  }
}
// Adds one FP32 partial of this lane to the fixed-point sum at p[at] when
// `mine` (add_fixed without its branches: a zero adds nothing either way).
__device__ __forceinline__ void add_fixed_if(bool mine, long long *p, float x, bool &bad) {
  bad |= mine && !(fabsf(x) <= 3.0e38f);
  const long long f = to_fixed_j(x);
  if (mine && f) atomicAdd((unsigned long long *)p, (unsigned long long)f);
}
// The j side's sums of a tile over the i groups, added to the j atoms.  The
// sums are (g0 + g1) + (g2 + g3) of the four groups' partials whichever group
// forms them, so each exchange halves the quantities a group goes on with
// (even groups keep 0-3, odd 4-6; then groups 0 and 2, 1 and 3 share those)
// and a lane converts and adds two of its j atom's seven sums, not all seven
// in the first group: 6 shuffles and 2 conversions a lane instead of 14 and 7.
__device__ __forceinline__ void pair_add_j(const PackView &v, const TileInfo &ti, int lane, const float (&j)[7],
                                           bool &bad) {
  const int g = lane >> 3;
  const bool odd = g & 1, high = g & 2;
  float x[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float lo = j[k], hi = k < 3 ? j[4 + k] : 0.f;
    const float other = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 8);
    x[k] = __fadd_rn(odd ? hi : lo, other);
  }
  float y[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const float other = __shfl_xor_sync(0xffffffffu, high ? x[k] : x[2 + k], 16);
    y[k] = __fadd_rn(high ? x[2 + k] : x[k], other);
  }
  // group g holds quantities 4 odd + 2 high + {0, 1} (force x, y, z, vdw, elec,
  // pol, dE/da; the eighth does not exist)
  const int at = ti.b0 + (lane & 7);
  const size_t N = (size_t)v.n_atoms;
  long long *p0 = odd ? (high ? v.ej + 3 * N : v.ej + N) : (high ? v.hz : v.hx);
  long long *p1 = odd ? v.ej + 2 * N : (high ? v.ej : v.hy);
  const bool mine = (lane & 7) < ti.nb;
  add_fixed_if(mine, p0 + at, y[0], bad);
  add_fixed_if(mine && !(odd && high), p1 + at, y[1], bad);
}

// `wait` runs between the static loads of the first tile (its records, its
// i side, the system's settings) and the first read of what the earlier
// phase wrote; false ends the phase.
template <bool LEAN, class Wait>
__device__ __forceinline__ bool phase_pair(const PackView &v, int blocks, int warp, int lane, float4 (*sA)[16],
                                           float4 (*sB)[16], float4 (*sP)[16], long long (*sI)[7][32], Wait wait) {
  int e, e1;
  ev_range(v.tile_count[0], blocks, warp, e, e1);
  const int first = e;
  const int N = v.n_atoms;
  const int g8 = lane & ~7, a = lane & 7;
  int a0 = -1, s_cur = -1, na = 0, s_i = 0, nd = 0;
  bool jbad = false;  // a non-finite sum of a j atom
  ISide acc;
  acc.f = sI[warp];
  acc.lane = lane;
  acc.clear();
  PairTileIn q;
  q.ia = q.ib = q.ip = make_float4(0, 0, 0, 0);
  q.ai_d = 0.0;
  q.i = 0;
  const SysParams *P = nullptr;
  double hec = 0.0, boff = 0.0;  // -halfeconv and the Born radius offset
  GbSettings gs;
  auto settings = [&](int s) {
    s_cur = s;
    P = &v.sp[s];
    gs.load(*P);
    hec = -P->halfeconv_d;
    boff = P->born_offset_d;
  };
  const ExactIn xin = exact_in(v);
  EvWalk<2> walk;
  walk.start_old(v, lane, e, e1);
  walk.start_xyz(v, lane);
  if (e < e1) {
    const TileInfo ti = tile_info(walk.nx.m);
    pair_i_static(v, ti, lane, q);
    settings(ti.s);
    a0 = ti.a0;
    na = ti.na;
    s_i = ti.s;
  }
  if (!wait()) return false;
  walk.start_dyn(v, lane);
  if (e < e1) pair_i_dyn(v, hec, boff, q);
#pragma unroll 1
  for (; e < e1; e++) {
    int te;
    const EvStage cur = walk.next(v, lane, te);
    const TileInfo ti = tile_info(cur.m);
    if (ti.a0 != a0) {
      flush_bad(v, jbad || (lane < na && acc.bad), s_i);
      if (lane < na) acc.flush(v, q.i, N);
      acc.clear();
      jbad = false;
      a0 = ti.a0;
      na = ti.na;
      s_i = ti.s;
      pair_i_static(v, ti, lane, q);
      if (ti.s != s_cur) settings(ti.s);
      pair_i_dyn(v, hec, boff, q);
    }
    q.b0 = ti.b0;
    pair_stage_j(ti, cur, lane, hec, boff, sA[warp], sB[warp], sP[warp]);
    const unsigned rows = rot8(cur.row, a);
    const unsigned xrows = rot8(cur.x0, a), brows = rot8(cur.x1, a);  // bond order <= 2, == 3
    __syncwarp();
    bool band = false;
    PairTileOut o = pair_tile<false, LEAN>(xin, gs, P, q, sA[warp], sB[warp], sP[warp], rows, xrows, brows, a, g8, band);
    if (__any_sync(0xffffffffu, band)) {
      defer_tile(v, lane, first, nd, e);
    } else {
      pair_add_j(v, ti, lane, o.jo, jbad);
#pragma unroll
      for (int k = 0; k < 7; k++) acc.add(k, o.io[k]);
    }
    __syncwarp();
  }
  flush_bad(v, jbad || (lane < na && acc.bad), s_i);
  if (lane < na) acc.flush(v, q.i, N);
  if (v.defer_stats && lane == 0 && nd) atomicAdd(&v.defer_stats[1], nd);
  // the deferred tiles in the careful form; their i sums go to memory at once
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < nd; k++) {
    const int t = v.defer_list[first + k];
    const EvStage cur = ev_stage_one<2>(v, t, lane);
    const TileInfo ti = tile_info(cur.m);
    settings(ti.s);
    pair_i_static(v, ti, lane, q);
    pair_i_dyn(v, hec, boff, q);
    q.b0 = ti.b0;
    pair_stage_j(ti, cur, lane, hec, boff, sA[warp], sB[warp], sP[warp]);
    const unsigned rows = rot8(cur.row, a);
    const unsigned xrows = rot8(cur.x0, a), brows = rot8(cur.x1, a);
    __syncwarp();
    bool band = false;
    PairTileOut o = pair_tile<true, LEAN>(xin, gs, P, q, sA[warp], sB[warp], sP[warp], rows, xrows, brows, a, g8, band);
    acc.clear();
    jbad = false;
    pair_add_j(v, ti, lane, o.jo, jbad);
#pragma unroll
    for (int c = 0; c < 7; c++) acc.add(c, o.io[c]);
    flush_bad(v, jbad || (lane < ti.na && acc.bad), ti.s);
    if (lane < ti.na) acc.flush(v, q.i, N);
    __syncwarp();
  }
  return true;
}

// ============================================================= phase C
// Chain-rule weight of an atom: gpi * dE/da with gpi = a^2 / 166.0 (the
// literal of gbff.cpp:1755) and dE/da = the pair sum - Eself / a, Eself =
// premul q^2 / a (gbff.cpp:1731-1757; k_gb_finish's expression), here as
// (a^2 * sum - premul q^2) / 166 in FP64: one rounding apart, and the
// weight is used in FP32.
__device__ __forceinline__ float chain_weight(const SysParams &P, double ai_d, long long dsum, float q) {
  const double dd = (double)dsum * kInvJScale;
  const double qd = (double)q;
  return (float)((ai_d * ai_d * dd - P.premul_d * qd * qd) * (1.0 / 166.0));
}

// One tile's chain-rule terms: the i side's force on this lane's i atom
// (io) and the j side's (jo, lane (g,a): j atom a, this group's i atoms,
// before the sum over groups); the Still cutoff's guard band as in phase A.
struct ChainTileIn {
  float4 ia, ib, ic;  // ic: R, V, the chain weight
  float s_lo, s_hi, invP5, piP5, P4;
  double still2_d;
  int i, b0;
};
struct ChainTileOut {
  float io[3], jo[3];
};
// chain_term's value with every step taken on every lane and the results
// selected (no divergent branches, so the eight steps of a tile interleave).
__device__ __forceinline__ float chain_term_sel(const Dx &d, float Ri, float Rj, float Vi, float Vj, float wi,
                                                float wj, float invP5, float piP5, float P4) {
  const float Rs = Ri + Rj;
  const float rdivR = __fdividef(d.r2, Rs * Rs);
  const float th = rdivR * piP5;
  float sn, cs;
  __sincosf(th, &sn, &cs);
  const float sq = 0.5f - 0.5f * cs;
  const float Xc = 4.f * sq * sq - 2.f * sq * sn * th;
  const float X = rdivR > invP5 ? 4.f : Xc;
  const float ir2 = __fdividef(1.f, d.r2);  // the fast reciprocal: deterministic, ~1 ulp
  const float ir6 = ir2 * ir2 * ir2;
  return P4 * X * ir6 * (wi * Vj + wj * Vi);
}
template <bool CAREFUL>
__device__ __forceinline__ ChainTileOut chain_tile(const ExactIn &v, const ChainTileIn &q, const float4 *sA,
                                                   const float4 *sB, const float4 *sC, unsigned rows, int a, int g8,
                                                   bool &band) {
  float io[3], jo[3];
#pragma unroll
  for (int k = 0; k < 3; k++) io[k] = jo[k] = 0.f;
#pragma unroll(CAREFUL ? 1 : 8)
  for (int t = 0; t < 8; t++) {
    const float4 ja = sA[a + t], jb = sB[a + t], jc = sC[a + t];
    const Dx d = diff(q.ia, q.ib, ja, jb);
    const bool row = (rows >> t) & 1u;
    bool ok = row && d.r2 <= q.s_lo;
    const bool edge = row && !ok && d.r2 <= q.s_hi;
    if (CAREFUL) {
      if (edge) {
        const int j = q.b0 + ((a + t) & 7), i = q.i;
        ok = !(ref_d2(v.x[i], v.y[i], v.z[i], v.x[j], v.y[j], v.z[j]) > q.still2_d);
      }
    } else {
      band |= edge;
    }
    // selected, not multiplied by zero: a lane without a pair may hold a
    // stale j slot of any value
    const float tt = chain_term_sel(d, q.ic.x, jc.x, q.ic.y, jc.y, q.ic.z, jc.z, q.invP5, q.piP5, q.P4);
    const float cx = ok ? tt * d.x : 0.f, cy = ok ? tt * d.y : 0.f, cz = ok ? tt * d.z : 0.f;
    io[0] += cx;
    io[1] += cy;
    io[2] += cz;
    const int src = g8 | ((a - t) & 7);
    jo[0] = __fadd_rn(jo[0], t == 0 ? -cx : __shfl_sync(0xffffffffu, -cx, src));
    jo[1] = __fadd_rn(jo[1], t == 0 ? -cy : __shfl_sync(0xffffffffu, -cy, src));
    jo[2] = __fadd_rn(jo[2], t == 0 ? -cz : __shfl_sync(0xffffffffu, -cz, src));
  }
  ChainTileOut o;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    o.io[k] = io[k];
    o.jo[k] = jo[k];
  }
  return o;
}
// The i-side inputs of this lane's atom of the tile's i-cluster: what is older
// than the evaluation, then the chain weight from the earlier phases' sums.
__device__ __forceinline__ const SysParams *chain_i_static(const PackView &v, const TileInfo &ti, int lane,
                                                           ChainTileIn &q) {
  q.i = ti.a0 + (lane < ti.na ? lane : 0);
  q.ia = v.pq[2 * (size_t)q.i];
  q.ib = v.pq[2 * (size_t)q.i + 1];
  const float4 pi = v.prm[q.i];
  q.ic = make_float4(pi.z, pi.w, 0.f, 0.f);
  const SysParams *P = &v.sp[ti.s];
  q.s_hi = P->still2 * (1.f + 4e-6f);
  q.s_lo = P->still2 * (1.f - 4e-6f);
  q.invP5 = P->invP5;
  q.piP5 = P->piP5;
  q.P4 = P->P4;
  q.still2_d = P->still2_d;
  return P;
}
__device__ __forceinline__ void chain_i_dyn(const PackView &v, const SysParams *P, ChainTileIn &q) {
  q.ic.z = chain_weight(*P, v.born_d[q.i], v.ej[(size_t)3 * v.n_atoms + q.i], q.ia.w);
}
// A tile's j records (with each j atom's chain weight) into this warp's slots.
__device__ __forceinline__ void chain_stage_j(const TileInfo &ti, const EvStage &cur, const SysParams *P, int lane,
                                              float4 *sA, float4 *sB, float4 *sC) {
  if (lane < ti.nb) {
    const float4 c = make_float4(cur.c.z, cur.c.w, chain_weight(*P, cur.u, cur.w, cur.a.w), 0.f);
    sA[lane] = sA[lane + 8] = cur.a;
    sB[lane] = sB[lane + 8] = cur.b;
    sC[lane] = sC[lane + 8] = c;
  }
}
// The j side's forces of a tile, summed over the i groups as in pair_add_j
// (even groups x and y, odd groups z; then group 0 x, group 2 y) and added to
// the j atoms, one component a lane.
__device__ __forceinline__ void chain_add_j(const PackView &v, const TileInfo &ti, int lane, const float (&j)[3],
                                            bool &bad) {
  const int g = lane >> 3;
  const bool odd = g & 1, high = g & 2;
  const float a = __fadd_rn(odd ? j[2] : j[0], __shfl_xor_sync(0xffffffffu, odd ? j[0] : j[2], 8));
  const float b = __fadd_rn(j[1], __shfl_xor_sync(0xffffffffu, j[1], 8));
  // an odd group holds z in a: both odd groups form the same sum
  const float keep = odd ? a : (high ? b : a), give = odd ? a : (high ? a : b);
  const float y = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16));
  long long *p = odd ? v.hz : (high ? v.hy : v.hx);
  add_fixed_if((lane & 7) < ti.nb && g != 3, p + ti.b0 + (lane & 7), y, bad);
}
// The i side's forces, fixed point per tile and added to memory when the
// warp's range leaves the i-cluster (exact sums: the same bits).
struct ChainISide {
  long long f[3];
  bool bad;
  __device__ __forceinline__ void clear() {
    f[0] = f[1] = f[2] = 0;
    bad = false;
  }
  __device__ __forceinline__ void add(const float (&io)[3]) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      bad |= !(fabsf(io[c]) <= 3.0e38f);
      f[c] += to_fixed_j(io[c]);
    }
  }
  __device__ __forceinline__ void flush(const PackView &v, int i) {
    if (f[0]) atomicAdd((unsigned long long *)&v.hx[i], (unsigned long long)f[0]);
    if (f[1]) atomicAdd((unsigned long long *)&v.hy[i], (unsigned long long)f[1]);
    if (f[2]) atomicAdd((unsigned long long *)&v.hz[i], (unsigned long long)f[2]);
  }
};

template <class Wait>
__device__ __forceinline__ bool phase_chain(const PackView &v, int blocks, int warp, int lane, float4 (*sA)[16],
                                            float4 (*sB)[16], float4 (*sC)[16], Wait wait) {
  int q0, q1;
  ev_range(v.tile_count[2], blocks, warp, q0, q1);  // (the still list is phase A's: complete)
  const int g8 = lane & ~7, a = lane & 7;
  int a0 = -1, na = 0, s_i = 0, nd = 0;
  bool jbad = false;
  ChainISide acc;
  acc.clear();
  ChainTileIn q;
  q.ia = q.ib = q.ic = make_float4(0, 0, 0, 0);
  q.s_hi = q.s_lo = q.invP5 = q.piP5 = q.P4 = 0.f;
  q.still2_d = 0.0;
  q.i = 0;
  const SysParams *P = nullptr;
  const ExactIn xin = exact_in(v);
  EvWalk<4> walk;
  walk.start_old(v, lane, q0, q1);
  walk.start_xyz(v, lane);
  if (q0 < q1) {
    const TileInfo ti = tile_info(walk.nx.m);
    P = chain_i_static(v, ti, lane, q);
    a0 = ti.a0;
    na = ti.na;
    s_i = ti.s;
  }
  if (!wait()) return false;
  walk.start_dyn(v, lane);
  if (q0 < q1) chain_i_dyn(v, P, q);
#pragma unroll 1
  for (int k = q0; k < q1; k++) {
    int t;
    const EvStage cur = walk.next(v, lane, t);
    const TileInfo ti = tile_info(cur.m);
    if (ti.a0 != a0) {
      flush_bad(v, jbad || (lane < na && acc.bad), s_i);
      if (lane < na) acc.flush(v, q.i);
      acc.clear();
      jbad = false;
      a0 = ti.a0;
      na = ti.na;
      s_i = ti.s;
      P = chain_i_static(v, ti, lane, q);
      chain_i_dyn(v, P, q);
    }
    q.b0 = ti.b0;
    chain_stage_j(ti, cur, P, lane, sA[warp], sB[warp], sC[warp]);
    const unsigned rows = rot8(cur.row & ~cur.x0, a);  // bond order > 2 only
    __syncwarp();
    bool band = false;
    const ChainTileOut o = chain_tile<false>(xin, q, sA[warp], sB[warp], sC[warp], rows, a, g8, band);
    if (__any_sync(0xffffffffu, band)) {
      defer_tile(v, lane, q0, nd, t);
    } else {
      chain_add_j(v, ti, lane, o.jo, jbad);
      acc.add(o.io);
    }
    __syncwarp();
  }
  flush_bad(v, jbad || (lane < na && acc.bad), s_i);
  if (lane < na) acc.flush(v, q.i);
  if (v.defer_stats && lane == 0 && nd) atomicAdd(&v.defer_stats[2], nd);
  // the deferred tiles in the careful form
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < nd; k++) {
    const int t = v.defer_list[q0 + k];
    const EvStage cur = ev_stage_one<4>(v, t, lane);
    const TileInfo ti = tile_info(cur.m);
    P = chain_i_static(v, ti, lane, q);
    chain_i_dyn(v, P, q);
    q.b0 = ti.b0;
    chain_stage_j(ti, cur, P, lane, sA[warp], sB[warp], sC[warp]);
    const unsigned rows = rot8(cur.row & ~cur.x0, a);
    __syncwarp();
    bool band = false;
    const ChainTileOut o = chain_tile<true>(xin, q, sA[warp], sB[warp], sC[warp], rows, a, g8, band);
    acc.clear();
    jbad = false;
    chain_add_j(v, ti, lane, o.jo, jbad);
    acc.add(o.io);
    flush_bad(v, jbad || (lane < ti.na && acc.bad), ti.s);
    if (lane < ti.na) acc.flush(v, q.i);
    __syncwarp();
  }
  return true;
}

// ============================================================= per-atom steps
// Before phase A: zero what phase B adds into (and, first in an
// evaluation, the forces and the record; ZeroFlags), as k_born_finish did.
__device__ __forceinline__ void prologue_zero(const PackView &v, int blocks, int zero) {
  const int N = v.n_atoms;
  const int stride = blocks * blockDim.x;
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    for (int q = 0; q < 4; q++) v.ej[(size_t)q * N + i] = 0;
    if (zero & ZF_PAIRS) {
      if (zero & ZF_BONDED) {
        v.fx[i] = 0;
        v.fy[i] = 0;
        v.fz[i] = 0;
      }
      v.gx[i] = 0.0;
      v.gy[i] = 0.0;
      v.gz[i] = 0.0;
      v.hx[i] = 0;
      v.hy[i] = 0;
      v.hz[i] = 0;
      const int s = v.sys_of[i];
      if ((zero & ZF_RECORD) && i == v.atom_off[s]) {
        for (int k = 0; k < E_COUNT; k++)
          if (k != E_EKIN) v.ene[(size_t)s * E_COUNT + k] = 0.0;
        v.sys_flags[s] = 0;
        v.sys_flags_alt[s] = 0;
      }
    }
  }
}
// After phase B (no phase-B reader of these): the Born radii.
__device__ __forceinline__ void epilogue_radii(const PackView &v, int blocks) {
  const int N = v.n_atoms;
  const int stride = blocks * blockDim.x;
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    const double a = born_radius(v, v.sp[v.sys_of[i]], i);
    v.born_d[i] = a;
    reinterpret_cast<float *>(&v.pq[2 * (size_t)i + 1])[3] = (float)a;
  }
}
// After phase C: the per-atom energies (k_gb_finish's values) and the
// Born sums cleared for the next evaluation.
__device__ __forceinline__ void epilogue_energies(const PackView &v, int blocks) {
  const int N = v.n_atoms;
  const int stride = blocks * blockDim.x;
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
    const SysParams &P = v.sp[v.sys_of[i]];
    const double dv = (double)v.ej[i] * kInvJScale;
    const double de = (double)v.ej[(size_t)N + i] * kInvJScale;
    const double dp = (double)v.ej[(size_t)2 * N + i] * kInvJScale;
    const double ai_d = v.born_d[i];
    const double qd = (double)v.pq[2 * (size_t)i].w;
    double *ep = v.ebuf ? v.e_pair_alt : v.e_atom;  // the pair slots of this energy buffer
    ep[(size_t)AE_VDW * N + i] = 0.5 * dv;
    ep[(size_t)AE_ELEC * N + i] = 0.5 * de;
    ep[(size_t)AE_POL * N + i] = dp;
    ep[(size_t)AE_POL_SELF * N + i] = P.premul_d * qd * qd / ai_d;
    v.bsum[i] = 0;
  }
}

// ============================================================= the kernel
// PH: which phases (1 A, 2 B, 4 C); more than one needs a cooperative
// launch.  tile_count[2] is the still-list length, tile_count[3] the barrier /
// exit counter; the last block out clears both.
template <bool LEAN, int PH>
__global__ void __launch_bounds__(32 * kEvWarps, kEvBlocks) k_eval_tiles(PackView v, int zero) {
  // a launch of phase B or C alone follows the launch of the phase before
  // it: it stages its first tiles while that one still runs, and waits for
  // it (griddep_wait) before it reads anything the evaluation writes
  constexpr int ph = PH;
  constexpr bool early = ph == 2 || ph == 4;
  const bool old_tiles = ph == 1 && (zero & ZF_OLD_TILES);
  if (!early && !old_tiles) PDGPU_DEP_ENTRY();
  const int G = ev_active(v);
  if (v.flags[F_NL_OVERFLOW] || (int)blockIdx.x >= G) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ float4 s0[kEvWarps][16], s1[kEvWarps][16], s2[kEvWarps][16];
  __shared__ long long si[kEvWarps][7][32];  // phase B's i-side sums
  unsigned *ctr = reinterpret_cast<unsigned *>(&v.tile_count[3]);
  unsigned passed = 0;  // barriers this launch has crossed
  if (ph & 1) {
    phase_born(v, G, warp, lane, s0, s1, s2, [&] {
      if (old_tiles) griddep_wait();
      prologue_zero(v, G, zero);
    });
  }
  // phases B and C load their first tiles' older records, then wait for the
  // phase before: a grid barrier in the cooperative launch, the previous
  // launch's end otherwise
  auto wait = [&](bool barrier) {
    if (barrier) return grid_barrier(ctr, (unsigned)G * ++passed, v.flags);
    if (early) griddep_wait();
    return true;
  };
  if (ph & 2) {
    if (!phase_pair<LEAN>(v, G, warp, lane, s0, s1, s2, si, [&] { return wait(ph & 1); })) return;
    epilogue_radii(v, G);
  }
  if (ph & 4) {
    if (!phase_chain(v, G, warp, lane, s0, s1, s2, [&] { return wait(ph & 2); })) return;
    epilogue_energies(v, G);
    // the last block out clears the still list and the counter
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned prev = atomicAdd(ctr, 1u);
      if (prev == (unsigned)G * (passed + 1) - 1) {
        v.tile_count[2] = 0;
        atomicExch(ctr, 0u);
      }
    }
  }
}

// ============================================================= host side
static int fused_wanted() {
  static int w = -1;
  if (w < 0) {
    const char *s = getenv("PDGPU_FUSED");
    w = (s && s[0] == '0') ? 0 : 1;
  }
  return w;
}

// PDGPU_EV_LEAN=0 runs the general build for every pack (the lean build
// gives the same bits where it applies; tested)
static int lean_allowed() {
  static int w = -1;
  if (w < 0) {
    const char *s = getenv("PDGPU_EV_LEAN");
    w = (s && s[0] == '0') ? 0 : 1;
  }
  return w;
}

// Resident blocks of the evaluation kernel on this device (the grid of its
// launches; the one-phase builds keep at least as many resident), and no more
// warps than a pack can have tiles.
int eval_tiles_grid(long long tile_cap) {
  int dev = 0, sms = 148, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_eval_tiles<false, 7>, 32 * kEvWarps, 0);
  const long long need = (tile_cap + kEvWarps - 1) / kEvWarps;
  return (int)std::max(1LL, std::min((long long)std::max(occ, 1) * sms, need));
}

static cudaError_t launch_ev(int ph, const PackView &v, cudaStream_t st, int zero, bool coop) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(v.ev_blocks);
  cfg.blockDim = dim3(32 * kEvWarps);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (coop) {
    attr[na].id = cudaLaunchAttributeCooperative;
    attr[na].val.cooperative = 1;
    na++;
  }
  // programmatic dependent launch for the one-phase launches (a
  // cooperative launch waits for the kernel before it in the stream)
  if (!coop && pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e;
  const bool lean = v.ev_lean && lean_allowed();
  auto go = [&](auto kernel) { return cudaLaunchKernelEx(&cfg, kernel, v, zero); };
  switch (ph) {
    case 1: e = lean ? go(k_eval_tiles<true, 1>) : go(k_eval_tiles<false, 1>); break;
    case 2: e = lean ? go(k_eval_tiles<true, 2>) : go(k_eval_tiles<false, 2>); break;
    case 4: e = lean ? go(k_eval_tiles<true, 4>) : go(k_eval_tiles<false, 4>); break;
    default: e = lean ? go(k_eval_tiles<true, 7>) : go(k_eval_tiles<false, 7>); break;
  }
  count_launch();
  return e;
}

// The three GB passes on the tiles: one cooperative launch when allowed,
// else three launches of the same phases.
bool eval_tiles_split(const PackView &v, bool coop) {
  return v.n_sc && v.ev_blocks > 0 && !(coop && fused_wanted());
}
cudaError_t launch_eval_tiles(const PackView &v, cudaStream_t st, int zero, bool coop, cudaEvent_t behind_a) {
  if (!v.n_sc || v.ev_blocks <= 0) return cudaSuccess;
  if (!eval_tiles_split(v, coop)) return launch_ev(7, v, st, zero, true);
  cudaError_t e = launch_ev(1, v, st, zero, false);
  if (behind_a) cudaEventRecord(behind_a, st);
  if (e == cudaSuccess) e = launch_ev(2, v, st, 0, false);
  if (e == cudaSuccess) e = launch_ev(4, v, st, 0, false);
  return e;
}

cudaError_t launch_born_phase_only(const PackView &v, cudaStream_t st) {
  if (!v.n_sc || v.ev_blocks <= 0) return cudaSuccess;
  return launch_ev(1, v, st, 0, false);
}

// One evaluation (three launches) that counts the tiles each phase
// deferred to its careful form into stats[0..2] (device memory, zeroed by
// the caller).
cudaError_t count_deferred_tiles(const PackView &v, cudaStream_t st, int *stats) {
  if (!v.n_sc || v.ev_blocks <= 0) return cudaSuccess;
  PackView w = v;
  w.defer_stats = stats;
  return launch_eval_tiles(w, st, ZF_PAIRS, false);
}

// Device times of the evaluation: the three phases as three launches
// (ms[0..2]), then the one cooperative launch (ms[3]); averages over reps.
// The forces of the timed evaluations are left in the accumulators.
cudaError_t profile_eval_tiles(const PackView &v, cudaStream_t st, int reps, double *ms) {
  cudaEvent_t ev[5];
  for (int q = 0; q < 5; q++) cudaEventCreate(&ev[q]);
  double acc[4] = {0, 0, 0, 0};
  cudaError_t e = cudaSuccess;
  for (int it = 0; it < reps && e == cudaSuccess; it++) {
    cudaEventRecord(ev[0], st);
    e = launch_ev(1, v, st, ZF_PAIRS, false);
    cudaEventRecord(ev[1], st);
    if (e == cudaSuccess) e = launch_ev(2, v, st, 0, false);
    cudaEventRecord(ev[2], st);
    if (e == cudaSuccess) e = launch_ev(4, v, st, 0, false);
    cudaEventRecord(ev[3], st);
    if (e == cudaSuccess) e = launch_ev(7, v, st, ZF_PAIRS, true);
    cudaEventRecord(ev[4], st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    for (int q = 0; q < 4 && e == cudaSuccess; q++) {
      float t = 0;
      cudaEventElapsedTime(&t, ev[q], ev[q + 1]);
      acc[q] += t;
    }
  }
  for (int q = 0; q < 5; q++) cudaEventDestroy(ev[q]);
  for (int q = 0; q < 4; q++) ms[q] = reps > 0 ? acc[q] / reps : 0.0;
  return e;
}

}  // namespace pdgpu
