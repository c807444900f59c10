// Cluster-pair tiles: the neighbour pair set re-cut into 32 x 8 blocks so
// the three pair passes read their partners once per block with coalesced
// loads and evaluate each unordered pair once.
//
// Atoms of a system are cut, in their own order (residue order: bonded and
// spatially close atoms are neighbours in memory), into i-clusters of 32
// (one per lane of a warp) and j-clusters of 8.  The tiles of an i-cluster
// are the j-clusters at or after it that hold a list partner of one of its
// atoms; they are read off the neighbour list itself (built with the
// reference's FP64 predicate, neighbourlist.cpp:263-266), so a tile's bits
// are exactly list pairs: every unordered list pair sits in one tile (the
// pair with j > i where the j-cluster lies inside the i-cluster).  A tile
// stores, per i lane, one byte of bits over its 8 j atoms; tiles with 1-2,
// 1-3 or 1-4 partners (bond orders from the list entries) carry two more
// byte rows: bond order <= 2 and bond order == 3.
//
// Each pass runs a persistent grid of G warps over the pack's T tiles
// (every system's clusters, the tiles of a cluster consecutive): warp g
// takes the contiguous range [T g / G, T (g+1) / G), so every warp gets the
// same number of tiles, give or take one, however unequal the clusters'
// tile counts are.  A warp prefetches the next tile's 8 j atoms while it
// works on the current one, and reloads its i atoms when the range enters
// the next cluster.  Lane l = 8g + a (one i atom) walks the tile's j atoms
// in the order (a+t) mod 8: the i side accumulates in registers, the j
// side goes with one shuffle to the lane of its group that owns the j
// atom; after the 8 steps the four groups' j sums meet with two xor
// shuffles.  Both sides of each tile are then added to their atoms with
// 64-bit fixed-point atomics.  A tile's sums depend on the tile alone, and
// fixed-point sums do not depend on the order of the additions, so every
// result is bit-identical run to run, however the tiles are spread over
// the warps and whatever other systems share the pack.  Pass results:
//   K2 k_born_tile   Born sums, fixed point 2^40 (exact per term);
//                    k_born_finish inverts them (FP64) and zeroes the
//                    accumulators of the next passes
//   K3 k_gb_tile     forces, per-atom LJ / Coulomb / GB energies and dE/da,
//                    fixed point 2^24; k_gb_finish forms the reference's
//                    per-atom values and the chain-rule weights
//   K4 k_chain_tile  chain-rule forces, fixed point 2^24
// The per-pair arithmetic is the row kernels' (pairmath.cuh).
#include <cuda_runtime.h>

#include <algorithm>

#include "tilecommon.cuh"

namespace pdgpu {

constexpr int kTileWarps = 4;    // warps per block
// resident blocks per SM the register allocation must allow, per pass
#ifndef PDGPU_K2_BLOCKS
#define PDGPU_K2_BLOCKS 6
#endif
#ifndef PDGPU_K3_BLOCKS
#define PDGPU_K3_BLOCKS 5
#endif
#ifndef PDGPU_K4_BLOCKS
#define PDGPU_K4_BLOCKS 6
#endif
constexpr int kBuildChunk = 128; // tiles assembled in shared memory at a time

// --------------------------------------------------------------- tile list
// One block per i-cluster.  (1) A bitmap over the system's j-clusters at or
// after the i-cluster marks those holding a half-list partner; (2) its set
// bits, in order, are the cluster's tiles (deterministic order); (3) the
// rows are scanned again to set the pair bits and the bond-order bits of
// each tile, kBuildChunk tiles at a time in shared memory.
__device__ __forceinline__ bool half_pair(int i, int j, int a0) {
  // j in a later j-cluster, or in this i-cluster with j > i
  return j >= a0 && (j >= a0 + 32 || j > i);
}

__global__ void __launch_bounds__(128) k_tile_build(PackView v) {
  extern __shared__ unsigned sm[];
  const int sc = blockIdx.x;
  if (v.flags[F_NL_OVERFLOW]) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s = v.sc_sys[sc];
  const int a0 = v.sc_atom0[sc];
  const int end = v.atom_off[s + 1];
  const int na = min(32, end - a0);
  const int nbits = (end - a0 + 7) / 8;  // j-clusters at or after a0
  const int W = (nbits + 31) / 32;
  unsigned *bm = sm;                                // [W]
  unsigned *pre = bm + W;                           // [W+1]
  int *cb0 = (int *)(pre + W + 1);                  // [chunk] first j atom
  unsigned *rw = (unsigned *)(cb0 + kBuildChunk);   // [chunk*8] pair bits: byte l of word l/4
  unsigned *xw = rw + kBuildChunk * 8;              // bond order <= 2
  unsigned *bw = xw + kBuildChunk * 8;              // bond order == 3
  __shared__ int base_s;
  for (int w = tid; w < W; w += blockDim.x) bm[w] = 0;
  __syncthreads();
  for (int q = warp; q < na; q += kTileWarps) {
    const int i = a0 + q;
    const long long b = v.row_start[i], e = v.row_start[i + 1];
    for (long long k = b + lane; k < e; k += 32) {
      const int j = (int)(v.nl[k] >> 3);
      if (half_pair(i, j, a0)) {
        const int p = (j - a0) >> 3;
        atomicOr(&bm[p >> 5], 1u << (p & 31));
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    int c = 0;
    for (int w = 0; w < W; w++) {
      pre[w] = c;
      c += __popc(bm[w]);
    }
    pre[W] = c;
    base_s = atomicAdd(&v.tile_count[0], c);
  }
  __syncthreads();
  const int ncand = pre[W];
  const int base = base_s;
  if ((long long)base + ncand > v.tile_cap) {  // cannot happen: the capacity is the worst case
    if (tid == 0) atomicExch(&v.flags[F_NL_OVERFLOW], 1);
    return;
  }
  for (int c0 = 0; c0 < ncand; c0 += kBuildChunk) {
    for (int w = tid; w < kBuildChunk * 8 * 3; w += blockDim.x) rw[w] = 0;
    for (int w = tid; w < W; w += blockDim.x) {
      unsigned bits = bm[w];
      while (bits) {
        const int b = __ffs(bits) - 1;
        bits &= bits - 1;
        const int r = pre[w] + __popc(bm[w] & ((1u << b) - 1u)) - c0;
        if (r >= 0 && r < kBuildChunk) cb0[r] = a0 + 8 * (32 * w + b);
      }
    }
    __syncthreads();
    for (int q = warp; q < na; q += kTileWarps) {
      const int i = a0 + q;
      const long long b = v.row_start[i], e = v.row_start[i + 1];
      for (long long k = b + lane; k < e; k += 32) {
        const unsigned ent = v.nl[k];
        const int j = (int)(ent >> 3);
        if (!half_pair(i, j, a0)) continue;
        const int p = (j - a0) >> 3;
        const int r = pre[p >> 5] + __popc(bm[p >> 5] & ((1u << (p & 31)) - 1u)) - c0;
        if (r < 0 || r >= kBuildChunk) continue;
        const unsigned bit = 1u << ((q & 3) * 8 + ((j - a0) & 7));
        const int wi = r * 8 + (q >> 2);
        atomicOr(&rw[wi], bit);
        const unsigned bo = ent & 7u;
        if (bo <= 2u) atomicOr(&xw[wi], bit);
        if (bo == 3u) atomicOr(&bw[wi], bit);
      }
    }
    __syncthreads();
    const int nr = min(kBuildChunk, ncand - c0);
    for (int r = tid; r < nr; r += blockDim.x) {
      const int et = base + c0 + r;
      unsigned spec_any = 0;
      for (int w = 0; w < 8; w++) {
        v.tile_rows[8 * (size_t)et + w] = rw[r * 8 + w];
        spec_any |= xw[r * 8 + w] | bw[r * 8 + w];
      }
      int spec = -1;
      if (spec_any) {
        spec = atomicAdd(&v.tile_count[1], 1);
        if (spec < v.spec_cap) {
          for (int w = 0; w < 8; w++) {
            v.spec_rows[16 * (size_t)spec + w] = xw[r * 8 + w];
            v.spec_rows[16 * (size_t)spec + 8 + w] = bw[r * 8 + w];
          }
        } else {
          atomicExch(&v.flags[F_NL_OVERFLOW], 1);
          spec = -1;
        }
      }
      const int nb = min(8, end - cb0[r]);
      v.tile_meta[et] = make_int4(cb0[r], spec, a0, (s << 8) | ((na - 1) << 3) | (nb - 1));
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------- tile search
// The tiles straight from the positions, without the list.  The pair test
// is the list's (the reference's FP64 expression without contraction,
// neighbourlist.cpp:263-266, and j != i) and the bond orders come from the
// same band and off-diagonal tables, so the tiles hold exactly the pairs a
// list build at these positions would give them.
//
// (1) k_cluster_boxes: eight lanes per j-cluster fold its atoms into an FP32
// box rounded outward (a cluster with a NaN coordinate gets an infinite box:
// its pairs are decided by the distance test alone), save the positions of
// this rebuild (for a later list build at the same positions) and clear the
// tile counters.
// (2) k_tile_search: one block per i-cluster.  Its threads take the system's
// j-clusters at or after the i-cluster, one each, and put those whose box
// may lie within the list cutoff of the i-cluster's box on a list in shared
// memory (gaps rounded down, so the cull drops no pair); its warps then take
// the list's entries in turn, test the 32 x 8 atom pairs (lane = i atom)
// with the positions of the next entry already loading, and stage a tile
// when any pair is in.
//
// What bounds it: latency (the pair tests of a 20,566-atom search are 3 us of
// FP64 issue).  Chain neighbours sit next to one another, so of the groups
// of 32 j-clusters that warps used to take whole, the first held nearly all
// the candidates and one warp walked them one pair of loads at a time; with
// the shared list the four warps get equal shares.  The FP32 boxes replace a
// per-atom FP64 cull: they pass 11,140 candidates for 9,479 tiles on the
// 16 x 80-residue system, 368 for 346 on a 64-residue peptide.
// Measured (launch, ncu): 985 atoms 45 -> 8 us, 20,566 atoms 62 -> 15 us,
// 64 OPLS peptides 150 -> 33 us, 512 peptides 671 -> 150 us.
__global__ void __launch_bounds__(128) k_cluster_boxes(PackView v) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW] == kGateShut) return;  // (k_tile_search returns on the flag too)
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 2) v.tile_count[t] = 0;
  const int jc = t >> 3, k = t & 7;
  const int q = min(jc, v.n_jc - 1);  // whole warps take part in the shuffles
  const int a0 = v.jc_atom0[q];
  const int n = min(8, v.atom_off[v.sys_of[a0] + 1] - a0);
  const int N = v.n_atoms;
  const int i = a0 + (k < n ? k : 0);
  const double p[3] = {v.x[i], v.y[i], v.z[i]};
  float lo[3], hi[3];
  bool wild = false;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    wild |= !(p[c] == p[c]);
    lo[c] = __double2float_rd(p[c]);
    hi[c] = __double2float_ru(p[c]);
    if (jc < v.n_jc && k < n) v.xs[(size_t)c * N + i] = p[c];
  }
  const unsigned g = 0xffu << (threadIdx.x & 24);  // this cluster's lanes
  wild = (__ballot_sync(0xffffffffu, wild) & g) != 0;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  if (jc >= v.n_jc || k > 1) return;
  const float w = k ? INFINITY : -INFINITY;
  const float b[3] = {k ? hi[0] : lo[0], k ? hi[1] : lo[1], k ? hi[2] : lo[2]};
  v.cbox[2 * (size_t)jc + k] = wild ? make_float4(w, w, w, 0.f) : make_float4(b[0], b[1], b[2], 0.f);
}

constexpr int kSearchWarps = 4;      // warps per i-cluster block of the tile search
constexpr int kSearchThreads = 32 * kSearchWarps;
// candidates held in shared memory: the cull takes that many j-clusters
// between two rounds of pair tests, so the list cannot run over and the cull
// has no barrier inside
constexpr int kSearchCand = 1024;

// Lower bound of the squared distance of two boxes (NaN gaps, from infinite
// boxes, count as 0).
__device__ __forceinline__ float box_gap2(const float4 &alo, const float4 &ahi, const float4 &blo,
                                          const float4 &bhi) {
  const float x = fmaxf(0.f, fmaxf(__fsub_rd(blo.x, ahi.x), __fsub_rd(alo.x, bhi.x)));
  const float y = fmaxf(0.f, fmaxf(__fsub_rd(blo.y, ahi.y), __fsub_rd(alo.y, bhi.y)));
  const float z = fmaxf(0.f, fmaxf(__fsub_rd(blo.z, ahi.z), __fsub_rd(alo.z, bhi.z)));
  return __fadd_rd(__fadd_rd(__fmul_rd(x, x), __fmul_rd(y, y)), __fmul_rd(z, z));
}

// The bond-order bits (<= 2, == 3) of one candidate's pairs in `row` (some
// lane's row is not empty, so the system has a band).  The eight band entries
// load together, whether in the row or not: with a load under each bit's
// branch a near-diagonal tile waited for eight of them in turn.
__device__ __forceinline__ void search_orders(const PackView &v, unsigned row, int i, int li, int jb0, int o, int mid,
                                              const signed char *band, bool has_off, unsigned &xr, unsigned &br) {
  int bo[8];
  unsigned inb = 0;
#pragma unroll
  for (int t = 0; t < 8; t++) {
    const int delta = jb0 + t - o - li;  // j > i wherever the row has a bit
    const bool in = ((row >> t) & 1u) && delta < mid;
    inb |= (unsigned)in << t;
    bo[t] = band[in ? (long long)li * mid + (delta - 1) : 0];
  }
#pragma unroll
  for (int t = 0; t < 8; t++) {
    if (((inb >> t) & 1u) && bo[t] <= 2) xr |= 1u << t;
    if (((inb >> t) & 1u) && bo[t] == 3) br |= 1u << t;
  }
  if (has_off) {
    const unsigned rest = row & ~inb;  // beyond the band: the off-diagonal partners
    for (int k = v.off_ptr[i], e = v.off_ptr[i + 1]; k < e; k++) {
      const int2 q = v.off_data[k];
      const int t = q.x - jb0;
      if (t < 0 || t > 7 || !((rest >> t) & 1u)) continue;
      if ((q.y & 7) <= 2) xr |= 1u << t;
      if ((q.y & 7) == 3) br |= 1u << t;
    }
  }
}
// A search block's tiles (and their bond-order rows) are staged in shared
// memory and written to the tile store as one contiguous range, so the tiles
// of an i-cluster sit together and a pass that walks contiguous tile ranges
// meets few i-cluster changes (each one a reload of the i side), and one
// atomic per block and counter reserves the space.  What does not fit the
// stage goes to the store one at a time.
constexpr int kSearchStage = 256, kSearchSpec = 24;
struct SearchStage {
  int n, nspec;                        // emitted (may pass the capacities)
  int base, sbase;                     // first slots in the store
  int4 meta[kSearchStage];             // y: -1, the staged rows' index, or -2 - the store's index
  unsigned rows[kSearchStage * 8];     // byte l of tile k's 32 bytes = i lane l's bits
  unsigned spec[kSearchSpec * 16];
};
// Store one tile that holds a pair; false when a capacity ran out (cannot
// happen: the capacities are worst cases).
__device__ __forceinline__ bool search_emit(const PackView &v, int lane, unsigned row, unsigned xr, unsigned br,
                                            int jb0, int a0, int s, int na, int nb, SearchStage &stage) {
  const bool special = __any_sync(0xffffffffu, (xr | br) != 0);
  int k = 0, spec = -1;
  if (lane == 0) {
    k = atomicAdd(&stage.n, 1);
    if (special && k < kSearchStage) spec = atomicAdd(&stage.nspec, 1);
  }
  k = __shfl_sync(0xffffffffu, k, 0);
  spec = __shfl_sync(0xffffffffu, spec, 0);
  const bool staged = k < kSearchStage;
  int e = k;  // a tile past the stage: its slot in the store
  if (!staged) {
    if (lane == 0) e = atomicAdd(&v.tile_count[0], 1);
    e = __shfl_sync(0xffffffffu, e, 0);
    if (e >= v.tile_cap) {
      if (lane == 0) atomicExch(&v.flags[F_NL_OVERFLOW], 1);
      return false;
    }
  }
  if (special) {
    unsigned char *to = reinterpret_cast<unsigned char *>(stage.spec) + 64 * spec;
    if (!staged || spec >= kSearchSpec) {
      int se = 0;
      if (lane == 0) se = atomicAdd(&v.tile_count[1], 1);
      se = __shfl_sync(0xffffffffu, se, 0);
      if (se >= v.spec_cap) {
        if (lane == 0) atomicExch(&v.flags[F_NL_OVERFLOW], 1);
        return false;
      }
      spec = staged ? -2 - se : se;
      to = reinterpret_cast<unsigned char *>(v.spec_rows) + 64 * (size_t)se;
    }
    to[lane] = (unsigned char)xr;
    to[32 + lane] = (unsigned char)br;
  }
  unsigned char *rows = staged ? reinterpret_cast<unsigned char *>(stage.rows)
                               : reinterpret_cast<unsigned char *>(v.tile_rows);
  rows[32 * (size_t)e + lane] = (unsigned char)row;
  if (lane == 0) (staged ? stage.meta : v.tile_meta)[e] = make_int4(jb0, spec, a0, (s << 8) | ((na - 1) << 3) | (nb - 1));
  return true;
}

__global__ void __launch_bounds__(kSearchThreads) k_tile_search(PackView v) {
  // everything but the boxes and the counters is older than k_cluster_boxes:
  // it is read while that kernel still runs
  const int sc = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = v.sc_sys[sc];
  const int a0 = v.sc_atom0[sc];
  const int end = v.atom_off[s + 1];
  const int na = min(32, end - a0);
  const int jc0 = v.sc_jc0[sc], jcs = v.jc_off[s], jc_end = v.jc_off[s + 1];
  const double lim = v.sp[s].nl_lim2_d;
  const float cull = __double2float_ru(lim);
  const bool live = lane < na;
  const int i = a0 + (live ? lane : 0);
  const double xi = v.x[i], yi = v.y[i], zi = v.z[i];
  const int o = v.atom_off[s], mid = v.mid[s], li = i - o;
  const signed char *band = reinterpret_cast<const signed char *>(v.band) + v.band_off[s];
  const bool has_off = v.off_ptr[i + 1] > v.off_ptr[i];
  const bool any_off = __any_sync(0xffffffffu, has_off);
  __shared__ SearchStage stage;
  __shared__ int cand[kSearchCand];
  __shared__ int ncand, stop_s;  // stop_s: an earlier overflow, read once so every thread agrees
  __shared__ double sj[kSearchWarps][3][8];
  __shared__ float4 ilo_s[32], ihi_s[32];  // the i atoms, rounded down and up
  if (warp == 0) {
    ilo_s[lane] = make_float4(__double2float_rd(xi), __double2float_rd(yi), __double2float_rd(zi), 0.f);
    ihi_s[lane] = make_float4(__double2float_ru(xi), __double2float_ru(yi), __double2float_ru(zi), 0.f);
  }
  if (threadIdx.x == 0) {
    stage.n = stage.nspec = 0;
    ncand = 0;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) stop_s = v.flags[F_NL_OVERFLOW];
  // the i-cluster's box: its (up to four) j-clusters' boxes
  float4 ilo = v.cbox[2 * (size_t)jc0], ihi = v.cbox[2 * (size_t)jc0 + 1];
  for (int q = 1; q < 4 && jc0 + q < jc_end; q++) {
    const float4 l = v.cbox[2 * (size_t)(jc0 + q)], h = v.cbox[2 * (size_t)(jc0 + q) + 1];
    ilo = make_float4(fminf(ilo.x, l.x), fminf(ilo.y, l.y), fminf(ilo.z, l.z), 0.f);
    ihi = make_float4(fmaxf(ihi.x, h.x), fmaxf(ihi.y, h.y), fmaxf(ihi.z, h.z), 0.f);
  }
  // An i-cluster across the end of one chain and the start of the next has a
  // box as long as the chains (647 j-clusters passed it on the 16 x 80-residue
  // system, and that block took 88 us).  Where the box is wider than the
  // cutoff, one of the i-cluster's j-cluster boxes must also lie within the
  // cutoff of the candidate's, and for one of those that is as wide, one of
  // its atoms.  Ordinary clusters (10-12 A) pass about as many either way.
  const float reach = sqrtf(cull);
  const bool wide = !(ihi.x - ilo.x <= reach && ihi.y - ilo.y <= reach && ihi.z - ilo.z <= reach);
  __syncthreads();
  if (stop_s) return;
  bool ok = true;  // false once a capacity ran out (warp-uniform)
  const int axis = min(lane >> 3, 2);  // lanes 0-23 load a candidate's x, y, z
  const double *src = axis == 0 ? v.x : (axis == 1 ? v.y : v.z);
  for (int base = jc0; base < jc_end; base += kSearchCand) {
    // cull: one j-cluster per thread and turn, the next turn's boxes loading
    const int stop = min(base + kSearchCand, jc_end);
    const int first = base + (int)threadIdx.x;
    float4 nlo = v.cbox[2 * (size_t)min(first, jc_end - 1)], nhi = v.cbox[2 * (size_t)min(first, jc_end - 1) + 1];
    for (int j0 = base + 32 * warp; j0 < stop; j0 += kSearchThreads) {
      const int jc = j0 + lane, jn = min(jc + kSearchThreads, jc_end - 1);
      const float4 jlo = nlo, jhi = nhi;
      nlo = v.cbox[2 * (size_t)jn];
      nhi = v.cbox[2 * (size_t)jn + 1];
      bool in = jc < stop && !(box_gap2(ilo, ihi, jlo, jhi) > cull);
      if (wide && in) {
        in = false;
        for (int q = 0; q < 4 && jc0 + q < jc_end; q++) {
          const float4 l = v.cbox[2 * (size_t)(jc0 + q)], h = v.cbox[2 * (size_t)(jc0 + q) + 1];
          bool near = !(box_gap2(l, h, jlo, jhi) > cull);
          if (near && !(h.x - l.x <= reach && h.y - l.y <= reach && h.z - l.z <= reach)) {
            near = false;
#pragma unroll
            for (int k = 0; k < 8; k++) near |= !(box_gap2(ilo_s[8 * q + k], ihi_s[8 * q + k], jlo, jhi) > cull);
          }
          in |= near;
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (m) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&ncand, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (in) cand[at + __popc(m & ((1u << lane) - 1u))] = jc;
      }
    }
    __syncthreads();
    const int n = ncand;
    // the pair tests: a candidate per warp, the next two's positions loading
    // (a j-cluster's first atom follows from its index: no load before them)
    auto fetch = [&](int c, int &jb0) {
      jb0 = o + 8 * (cand[min(c, n - 1)] - jcs);
      return src[min(jb0 + (lane & 7), end - 1)];
    };
    int jb1 = 0, jb2 = 0;
    double p1 = 0.0, p2 = 0.0;
    if (warp < n) {
      p1 = fetch(warp, jb1);
      p2 = fetch(warp + kSearchWarps, jb2);
    }
    for (int c = warp; ok && c < n; c += kSearchWarps) {
      __syncwarp();
      if (lane < 24) sj[warp][axis][lane & 7] = p1;
      __syncwarp();
      const int jb = jb1, nj = min(8, end - jb);
      p1 = p2;
      jb1 = jb2;
      p2 = fetch(c + 2 * kSearchWarps, jb2);
      unsigned row = 0;
#pragma unroll
      for (int t = 0; t < 8; t++)
        if (!(ref_d2(xi, yi, zi, sj[warp][0][t], sj[warp][1][t], sj[warp][2][t]) > lim)) row |= 1u << t;
      row &= (1u << nj) - 1u;
      // the half list: j > i inside the i-cluster
      if (jb < a0 + 32 && i >= jb) row &= i - jb >= 7 ? 0u : ~((2u << (i - jb)) - 1u);
      if (!live) row = 0;
      if (__any_sync(0xffffffffu, row != 0)) {
        unsigned xr = 0, br = 0;
        if (any_off || jb - (a0 + na - 1) < mid) search_orders(v, row, i, li, jb, o, mid, band, has_off, xr, br);
        ok = search_emit(v, lane, row, xr, br, jb, a0, s, na, nj, stage);
      }
    }
    __syncthreads();  // the list has been read
    if (threadIdx.x == 0) ncand = 0;
    if (stop < jc_end) __syncthreads();
  }
  const int n = min(stage.n, kSearchStage), ns = min(stage.nspec, kSearchSpec);
  if (n == 0) return;
  if (threadIdx.x == 0) stage.base = atomicAdd(&v.tile_count[0], n);
  if (threadIdx.x == 32) stage.sbase = ns ? atomicAdd(&v.tile_count[1], ns) : 0;
  __syncthreads();
  const long long b0 = stage.base, s0 = stage.sbase;
  if (b0 + n > v.tile_cap || s0 + ns > v.spec_cap) {
    if (threadIdx.x == 0) atomicExch(&v.flags[F_NL_OVERFLOW], 1);
    return;
  }
  for (int w = threadIdx.x; w < 8 * n; w += kSearchThreads) v.tile_rows[8 * b0 + w] = stage.rows[w];
  for (int w = threadIdx.x; w < 16 * ns; w += kSearchThreads) v.spec_rows[16 * s0 + w] = stage.spec[w];
  for (int k = threadIdx.x; k < n; k += kSearchThreads) {
    int4 m = stage.meta[k];
    if (m.y >= 0)
      m.y += (int)s0;
    else if (m.y < -1)
      m.y = -2 - m.y;
    v.tile_meta[b0 + k] = m;
  }
}

// --------------------------------------------------------------- tile passes
// Staging of a tile: its metadata and this lane's row bits, and in lanes
// 0..7 three records of their j atom, held in registers (prefetched one
// tile ahead) and written to the warp's shared slots before the tile is
// processed.
struct JStage {
  float4 a, b, c;
  int4 m;
  unsigned row;
};
template <int REC>  // third record: 0 chainp (radius R, volume V, chain weight w), 1 prm (LJ radius, eps)
__device__ __forceinline__ void stage_load(const PackView &v, int e, int lane, JStage &q) {
  q.m = v.tile_meta[e];
  q.row = tile_row(v, e, lane);
  if (lane <= (q.m.w & 7)) {
    const int j = q.m.x + lane;
    q.a = v.pq[2 * (size_t)j];
    q.b = v.pq[2 * (size_t)j + 1];
    q.c = REC == 0 ? v.chainp[j] : v.prm[j];
  }
}

// This warp's tile range [e0, e1): an equal share of the pack's tiles.
__device__ __forceinline__ void warp_range(const PackView &v, int warp, int &e0, int &e1) {
  const long long T = v.tile_count[0];
  const long long G = (long long)gridDim.x * kTileWarps;
  const long long g = (long long)blockIdx.x * kTileWarps + warp;
  e0 = (int)(T * g / G);
  e1 = (int)(T * (g + 1) / G);
}

// --------------------------------------------------------------- K2 tiles
// (register bounds: five blocks per SM)
__global__ void __launch_bounds__(32 * kTileWarps, PDGPU_K2_BLOCKS) k_born_tile(PackView v) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW]) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g8 = lane & ~7, a = lane & 7;
  __shared__ float4 sA[kTileWarps][8], sB[kTileWarps][8], sC[kTileWarps][8];
  int e, e1;
  warp_range(v, warp, e, e1);
  if (e >= e1) return;
  JStage nx;
  stage_load<0>(v, e, lane, nx);
  int a0 = -1, na = 0, i = 0;
  float4 ia, ib, ic;
  float s_hi = 0.f, s_lo = 0.f, invP5 = 0.f, piP5 = 0.f, P4s = 0.f;
  double still2_d = 0.0;
  long long acc_i = 0;  // exact per term: added when the range leaves the cluster
  for (; e < e1; e++) {
    const JStage cur = nx;
    const TileInfo ti = tile_info(cur.m);
    if (e + 1 < e1) stage_load<0>(v, e + 1, lane, nx);
    if (ti.a0 != a0) {
      if (lane < na && acc_i) atomicAdd((unsigned long long *)&v.bsum[a0 + lane], (unsigned long long)acc_i);
      acc_i = 0;
      a0 = ti.a0;
      na = ti.na;
      i = a0 + (lane < na ? lane : 0);
      ia = v.pq[2 * (size_t)i];
      ib = v.pq[2 * (size_t)i + 1];
      ic = v.chainp[i];
      const SysParams &P = v.sp[ti.s];
      s_hi = P.still2 * (1.f + 4e-6f);
      s_lo = P.still2 * (1.f - 4e-6f);
      invP5 = P.invP5;
      piP5 = P.piP5;
      P4s = P.P4 * (float)kBornScale;
      still2_d = P.still2_d;
    }
    if (lane < ti.nb) {
      sA[warp][lane] = cur.a;
      sB[warp][lane] = cur.b;
      sC[warp][lane] = cur.c;
    }
    unsigned rows = cur.row;
    if (ti.spec >= 0) rows &= ~spec_row(v, ti.spec, 0, lane);  // bond order > 2 only
    __syncwarp();
    long long jacc = 0;  // lane (g,a): j atom a, this group's i atoms
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int jt = (a + t) & 7;
      long long tI = 0, tJ = 0;
      if ((rows >> jt) & 1u) {
        const float4 ja = sA[warp][jt], jb = sB[warp][jt], jc = sC[warp][jt];
        const Dx d = diff(ia, ib, ja, jb);
        bool ok = d.r2 <= s_lo;
        if (!ok && d.r2 <= s_hi) {
          const int j = ti.b0 + jt;
          ok = !(ref_d2(v.x[i], v.y[i], v.z[i], v.x[j], v.y[j], v.z[j]) > still2_d);
        }
        if (ok) {
          const float term = born_term_noV(d, ic.x, jc.x, invP5, piP5, P4s);
          tI = __float2ll_rn(__fmul_rn(term, jc.y));
          tJ = __float2ll_rn(__fmul_rn(term, ic.y));
        }
      }
      acc_i += tI;
      jacc += __shfl_sync(0xffffffffu, tJ, g8 | ((a - t) & 7));
    }
    jacc += __shfl_xor_sync(0xffffffffu, jacc, 8);
    jacc += __shfl_xor_sync(0xffffffffu, jacc, 16);
    if (lane < ti.nb && jacc) atomicAdd((unsigned long long *)&v.bsum[ti.b0 + lane], (unsigned long long)jacc);
    __syncwarp();
  }
  if (lane < na && acc_i) atomicAdd((unsigned long long *)&v.bsum[a0 + lane], (unsigned long long)acc_i);
}

// a_i = -halfeconv / (terms123_i + sum) (FP64); zero the accumulators the
// following passes add into (and, first in an evaluation, the forces)
__global__ void k_born_finish(PackView v, int zero_first) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW]) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  const int s = v.sys_of[i];
  const SysParams &P = v.sp[s];
  long long sum = v.bsum[i];
  v.bsum[i] = 0;
  double Gpol = v.terms123[i] + (double)sum * kInvBornScale;
  double a = -P.halfeconv_d / Gpol + P.born_offset_d;
  v.born_d[i] = a;
  reinterpret_cast<float *>(&v.pq[2 * (size_t)i + 1])[3] = (float)a;
  const int N = v.n_atoms;
  for (int q = 0; q < 4; q++) v.ej[(size_t)q * N + i] = 0;
  if (zero_first) {
    if (zero_first & ZF_BONDED) {
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
    if ((zero_first & ZF_RECORD) && i == v.atom_off[s]) {
      for (int k = 0; k < E_COUNT; k++)
        if (k != E_EKIN) v.ene[(size_t)s * E_COUNT + k] = 0.0;
      v.sys_flags[s] = 0;
    }
  }
}

// --------------------------------------------------------------- K3 tiles
__global__ void __launch_bounds__(32 * kTileWarps, PDGPU_K3_BLOCKS) k_gb_tile(PackView v) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW]) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g8 = lane & ~7, a = lane & 7;
  __shared__ float4 sA[kTileWarps][8], sB[kTileWarps][8], sP[kTileWarps][8];
  int e, e1;
  warp_range(v, warp, e, e1);
  if (e >= e1) return;
  const int N = v.n_atoms;
  JStage nx;
  stage_load<1>(v, e, lane, nx);
  int a0 = -1, i = 0;
  float4 ia, ib, ip;
  GbSettings gs;
  for (; e < e1; e++) {
    const JStage cur = nx;
    const TileInfo ti = tile_info(cur.m);
    if (e + 1 < e1) stage_load<1>(v, e + 1, lane, nx);
    if (ti.a0 != a0) {
      a0 = ti.a0;
      i = a0 + (lane < ti.na ? lane : 0);
      ia = v.pq[2 * (size_t)i];
      ib = v.pq[2 * (size_t)i + 1];
      ip = v.prm[i];
      gs.load(v.sp[ti.s]);
    }
    if (lane < ti.nb) {
      sA[warp][lane] = cur.a;
      sB[warp][lane] = cur.b;
      sP[warp][lane] = cur.c;
    }
    const unsigned rows = cur.row;
    unsigned xrows = 0, brows = 0;  // bond order <= 2, == 3
    if (ti.spec >= 0) {
      xrows = spec_row(v, ti.spec, 0, lane);
      brows = spec_row(v, ti.spec, 1, lane);
    }
    __syncwarp();
    float fx = 0.f, fy = 0.f, fz = 0.f, e_vdw = 0.f, e_el = 0.f, e_pol = 0.f, deda = 0.f;
    float jacc[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int t = 0; t < 8; t++) {
      const int jt = (a + t) & 7;
      const float4 ja = sA[warp][jt], jb = sB[warp][jt], jp = sP[warp][jt];
      const Dx d = diff(ia, ib, ja, jb);
      const bool in = ((rows >> jt) & 1u) && d.r2 <= gs.rc2;
      float c[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (in) {
        const bool nb3 = !((xrows >> jt) & 1u);
        const bool b14 = (brows >> jt) & 1u;
        const GbPair gp = gb_pair_term(gs, d, nb3, b14, ib.w, jb.w, ia.w, ja.w, ip.x, jp.x, ip.y, jp.y, v, i,
                                       ti.b0 + jt);
        e_pol += gp.epol;
        deda += gp.dedal * jb.w;
        e_vdw += gp.vdw;
        e_el += gp.elec;
        fx -= gp.fscal * d.x;
        fy -= gp.fscal * d.y;
        fz -= gp.fscal * d.z;
        c[0] = gp.fscal * d.x;
        c[1] = gp.fscal * d.y;
        c[2] = gp.fscal * d.z;
        c[3] = gp.vdw;
        c[4] = gp.elec;
        c[5] = gp.epol;
        c[6] = gp.dedal * ib.w;
      }
      const int src = g8 | ((a - t) & 7);
#pragma unroll
      for (int q = 0; q < 7; q++) jacc[q] += __shfl_sync(0xffffffffu, c[q], src);
    }
#pragma unroll
    for (int q = 0; q < 7; q++) {
      jacc[q] += __shfl_xor_sync(0xffffffffu, jacc[q], 8);
      jacc[q] += __shfl_xor_sync(0xffffffffu, jacc[q], 16);
    }
    if (lane < ti.nb) {
      const int j = ti.b0 + lane;
      add_fixed(v, &v.hx[j], jacc[0], ti.s);
      add_fixed(v, &v.hy[j], jacc[1], ti.s);
      add_fixed(v, &v.hz[j], jacc[2], ti.s);
#pragma unroll
      for (int q = 0; q < 4; q++) add_fixed(v, &v.ej[(size_t)q * N + j], jacc[3 + q], ti.s);
    }
    if (lane < ti.na) {
      add_fixed(v, &v.hx[i], fx, ti.s);
      add_fixed(v, &v.hy[i], fy, ti.s);
      add_fixed(v, &v.hz[i], fz, ti.s);
      add_fixed(v, &v.ej[i], e_vdw, ti.s);
      add_fixed(v, &v.ej[(size_t)N + i], e_el, ti.s);
      add_fixed(v, &v.ej[(size_t)2 * N + i], e_pol, ti.s);
      add_fixed(v, &v.ej[(size_t)3 * N + i], deda, ti.s);
    }
    __syncwarp();
  }
}

// Per-atom values of the fused pass, as the row kernel leaves them: LJ and
// Coulomb halves, the GB pair sum, the self term, and the chain-rule
// weight gpi * dE/da_i (gbff.cpp:1731-1757).
__global__ void k_gb_finish(PackView v) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW]) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  const int N = v.n_atoms;
  const SysParams &P = v.sp[v.sys_of[i]];
  double dv = (double)v.ej[i] * kInvJScale;
  double de = (double)v.ej[(size_t)N + i] * kInvJScale;
  double dp = (double)v.ej[(size_t)2 * N + i] * kInvJScale;
  double dd = (double)v.ej[(size_t)3 * N + i] * kInvJScale;
  double ai_d = v.born_d[i];
  double qd = (double)v.pq[2 * (size_t)i].w;
  double eself = P.premul_d * qd * qd / ai_d;
  v.e_atom[(size_t)AE_VDW * N + i] = 0.5 * dv;
  v.e_atom[(size_t)AE_ELEC * N + i] = 0.5 * de;
  v.e_atom[(size_t)AE_POL * N + i] = dp;
  v.e_atom[(size_t)AE_POL_SELF * N + i] = eself;
  double deda_i = dd - eself / ai_d;
  double gpi = ai_d * ai_d / 166.0;  // gbff.cpp:1755 uses the literal 166.0
  reinterpret_cast<float *>(&v.chainp[i])[2] = (float)(gpi * deda_i);
}

// --------------------------------------------------------------- K4 tiles
__global__ void __launch_bounds__(32 * kTileWarps, PDGPU_K4_BLOCKS) k_chain_tile(PackView v) {
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW]) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g8 = lane & ~7, a = lane & 7;
  __shared__ float4 sA[kTileWarps][8], sB[kTileWarps][8], sC[kTileWarps][8];
  int e, e1;
  warp_range(v, warp, e, e1);
  if (e >= e1) return;
  JStage nx;
  stage_load<0>(v, e, lane, nx);
  int a0 = -1, i = 0;
  float4 ia, ib, ic;
  float s_hi = 0.f, s_lo = 0.f, invP5 = 0.f, piP5 = 0.f, P4 = 0.f;
  double still2_d = 0.0;
  for (; e < e1; e++) {
    const JStage cur = nx;
    const TileInfo ti = tile_info(cur.m);
    if (e + 1 < e1) stage_load<0>(v, e + 1, lane, nx);
    if (ti.a0 != a0) {
      a0 = ti.a0;
      i = a0 + (lane < ti.na ? lane : 0);
      ia = v.pq[2 * (size_t)i];
      ib = v.pq[2 * (size_t)i + 1];
      ic = v.chainp[i];
      const SysParams &P = v.sp[ti.s];
      s_hi = P.still2 * (1.f + 4e-6f);
      s_lo = P.still2 * (1.f - 4e-6f);
      invP5 = P.invP5;
      piP5 = P.piP5;
      P4 = P.P4;
      still2_d = P.still2_d;
    }
    if (lane < ti.nb) {
      sA[warp][lane] = cur.a;
      sB[warp][lane] = cur.b;
      sC[warp][lane] = cur.c;
    }
    unsigned rows = cur.row;
    if (ti.spec >= 0) rows &= ~spec_row(v, ti.spec, 0, lane);  // bond order > 2 only
    __syncwarp();
    float fx = 0.f, fy = 0.f, fz = 0.f, j0 = 0.f, j1 = 0.f, j2 = 0.f;
#pragma unroll 2
    for (int t = 0; t < 8; t++) {
      const int jt = (a + t) & 7;
      float c0 = 0.f, c1 = 0.f, c2 = 0.f;
      if ((rows >> jt) & 1u) {
        const float4 ja = sA[warp][jt], jb = sB[warp][jt], jc = sC[warp][jt];
        const Dx d = diff(ia, ib, ja, jb);
        bool ok = d.r2 <= s_lo;
        if (!ok && d.r2 <= s_hi) {
          const int j = ti.b0 + jt;
          ok = !(ref_d2(v.x[i], v.y[i], v.z[i], v.x[j], v.y[j], v.z[j]) > still2_d);
        }
        if (ok) {
          const float tt = chain_term(d, ic.x, jc.x, ic.y, jc.y, ic.z, jc.z, invP5, piP5, P4);
          fx += tt * d.x;
          fy += tt * d.y;
          fz += tt * d.z;
          c0 = -tt * d.x;
          c1 = -tt * d.y;
          c2 = -tt * d.z;
        }
      }
      const int src = g8 | ((a - t) & 7);
      j0 += __shfl_sync(0xffffffffu, c0, src);
      j1 += __shfl_sync(0xffffffffu, c1, src);
      j2 += __shfl_sync(0xffffffffu, c2, src);
    }
    j0 += __shfl_xor_sync(0xffffffffu, j0, 8);
    j1 += __shfl_xor_sync(0xffffffffu, j1, 8);
    j2 += __shfl_xor_sync(0xffffffffu, j2, 8);
    j0 += __shfl_xor_sync(0xffffffffu, j0, 16);
    j1 += __shfl_xor_sync(0xffffffffu, j1, 16);
    j2 += __shfl_xor_sync(0xffffffffu, j2, 16);
    if (lane < ti.nb) {
      const int j = ti.b0 + lane;
      add_fixed(v, &v.hx[j], j0, ti.s);
      add_fixed(v, &v.hy[j], j1, ti.s);
      add_fixed(v, &v.hz[j], j2, ti.s);
    }
    if (lane < ti.na) {
      add_fixed(v, &v.hx[i], fx, ti.s);
      add_fixed(v, &v.hy[i], fy, ti.s);
      add_fixed(v, &v.hz[i], fz, ti.s);
    }
    __syncwarp();
  }
}

// instrumentation: out[0] += list pairs held by the tiles, out[1] += tiles
__global__ void k_tile_counts(PackView v, unsigned long long *out) {
  const int n = v.tile_count[0];
  unsigned long long p = 0, t = 0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    for (int w = 0; w < 8; w++) p += __popc(v.tile_rows[8 * (size_t)e + w]);
    t++;
  }
  p = group_sum<32>(p);
  t = group_sum<32>(t);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], p);
    atomicAdd(&out[1], t);
  }
}
void launch_tile_counts(const PackView &v, cudaStream_t st, unsigned long long *out) {
  PDGPU_LAUNCH(k_tile_counts, 296, 256, 0, st, v, out);
}

// --------------------------------------------------------------- launchers
size_t tile_build_smem(int max_sys_atoms) {
  int nbits = (max_sys_atoms + 7) / 8;
  int W = (nbits + 31) / 32;
  return sizeof(unsigned) * (2 * (size_t)W + 1 + kBuildChunk + 3 * 8 * (size_t)kBuildChunk);
}
// Persistent grids: the blocks one wave holds, and no more warps than the
// pack can have tiles.
void tile_launch_shapes(PackView &v) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int occ[3] = {1, 1, 1};
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[0], k_born_tile, 32 * kTileWarps, 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[1], k_gb_tile, 32 * kTileWarps, 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[2], k_chain_tile, 32 * kTileWarps, 0);
  const long long need = (v.tile_cap + kTileWarps - 1) / kTileWarps;
  for (int p = 0; p < 3; p++)
    v.tile_blocks[p] = (int)std::max(1LL, std::min((long long)std::max(occ[p], 1) * sms, need));
  v.ev_blocks = eval_tiles_grid(v.tile_cap);
}
void launch_tiles_build(const PackView &v, cudaStream_t st, bool filled) {
  if (!v.n_sc) return;
  if (!filled) cudaMemsetAsync(v.tile_count, 0, 2 * sizeof(int), st);
  size_t smem = tile_build_smem(v.max_sys_atoms);
  static size_t opted = 0;  // dynamic shared memory above 48 KB needs an opt-in
  if (smem > 48 * 1024 && smem > opted) {
    cudaFuncSetAttribute(k_tile_build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    opted = smem;
  }
  PDGPU_LAUNCH(k_tile_build, v.n_sc, 128, smem, st, v);
}
void launch_tiles_search(const PackView &v, cudaStream_t st) {
  if (!v.n_sc) return;
  PDGPU_LAUNCH_DEP(k_cluster_boxes, (v.n_jc + 15) / 16, 128, 0, st, v);
  PDGPU_LAUNCH_DEP(k_tile_search, v.n_sc, kSearchThreads, 0, st, v);
}
void launch_born_radii_tile(const PackView &v, cudaStream_t st, int zero_first) {
  if (!v.n_sc) return;
  PDGPU_LAUNCH_DEP(k_born_tile, v.tile_blocks[0], 32 * kTileWarps, 0, st, v);
  PDGPU_LAUNCH_DEP(k_born_finish, (v.n_atoms + 63) / 64, 64, 0, st, v, zero_first);
}
void launch_gb_pair_tile(const PackView &v, cudaStream_t st) {
  if (!v.n_sc) return;
  PDGPU_LAUNCH_DEP(k_gb_tile, v.tile_blocks[1], 32 * kTileWarps, 0, st, v);
  PDGPU_LAUNCH_DEP(k_gb_finish, (v.n_atoms + 63) / 64, 64, 0, st, v);
}
void launch_gb_chain_tile(const PackView &v, cudaStream_t st) {
  if (!v.n_sc) return;
  PDGPU_LAUNCH_DEP(k_chain_tile, v.tile_blocks[2], 32 * kTileWarps, 0, st, v);
}

}  // namespace pdgpu
