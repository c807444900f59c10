// Energy record (Hamiltonian, workspace/hamiltonian.h:23-49) from the
// per-atom and per-term energies the force kernels write.
//
// One kernel, two stages, both in a fixed order so every total is
// bit-reproducible: each block of the grid (chunks, systems) sums one
// kReduceChunk-item chunk of each range of one system (per-atom terms and the
// bond / angle / dihedral term arrays); the last block of a system to finish
// adds the chunk partials in chunk order, applies them to the record with
// the reference's semantics (the GB and stand-alone LJ/Coulomb components
// assign epot_vdw / epot_elec, everything else accumulates), and in a step
// loop records the step's energies and advances the step.
//
// What bounds it: on a single system the chain of loads, barriers and one
// atomic between its two stages; on a batch the reduction's instructions.  A
// system of up to 4,096 items a range (about 1,500 atoms) is one block and
// skips the second stage; a thread holds eight items of a range in flight;
// the record is read beside them; and the block's sums cross shared memory
// once (warp w adds slot w, sixteen values a lane and one shuffle tree)
// instead of a five-step shuffle tree of every slot in every warp.  The grid is as deep as the
// largest system; a smaller system's blocks past its own chunks leave at
// once.  Measured (launch, against 256 items and 384 threads a block): 985
// atoms 7.0 -> 5.7 us, 64 peptides 21.7 -> 10.9, 512 peptides 149 -> 22;
// 20,566 atoms 8.9 -> 9.5 (14 blocks; with 1,024 items 8.8, but 985 atoms
// 8.0, and it is the small systems' steps that wait for this record).
#include <cuda_runtime.h>

#include "minstep.cuh"

namespace pdgpu {

constexpr int kChunk = kReduceChunk;
constexpr int kEnergyThreads = 512;
constexpr int kEnergyWarps = kEnergyThreads / 32;
constexpr int kItems = kChunk / kEnergyThreads;  // of a range, per thread
static_assert(kChunk % kEnergyThreads == 0, "whole items per thread");
// partial slots
enum { P_VDW = 0, P_ELEC, P_POL, P_SELF, P_NBVIR, P_KIN, P_BOND, P_BVIR, P_ANGLE, P_DIH, P_SURF, P_COUNT };
static_assert(P_COUNT <= kPartSlots, "partials fit the reduction buffer");

// this thread's items of [b, e) (at most kChunk of them), loaded together
__device__ __forceinline__ double chunk_sum(const double *p, int b, int e) {
  double x[kItems];
#pragma unroll
  for (int q = 0; q < kItems; q++) {
    const int i = b + (int)threadIdx.x + q * kEnergyThreads;
    x[q] = i < e ? p[i] : 0.0;
  }
  double t = x[0];
#pragma unroll
  for (int q = 1; q < kItems; q++) t += x[q];
  return t;
}

// hist: [step][sys][3] (epot, ekin, etot); step_dev: StepSlot.
__global__ void __launch_bounds__(kEnergyThreads) k_energy(PackView v, int mode, int C, double J2kcalmol,
                                                           double *hist, int *step_dev, MinCtl ctl) {
  // the ranges are fixed with the pack: read before the wait
  const int c = blockIdx.x, s = blockIdx.y, N = v.n_atoms;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S1 = v.n_sys + 1;
  const int *off = v.bt.term_off;
  int lo[5], hi[5], most = 1;  // atoms, bonds, angles, torsions, impropers
#pragma unroll
  for (int r = 0; r < 5; r++) {
    lo[r] = r == 0 ? v.atom_off[s] : off ? off[(r - 1) * S1 + s] : 0;
    hi[r] = r == 0 ? v.atom_off[s + 1] : off ? off[(r - 1) * S1 + s + 1] : 0;
    most = max(most, hi[r] - lo[r]);
    lo[r] += c * kChunk;
    hi[r] = min(hi[r], lo[r] + kChunk);
  }
  const int mine = min(C, (most + kChunk - 1) / kChunk);  // this system's chunks
  PDGPU_DEP_ENTRY();
  if (c >= mine) return;
  const int overflow = v.flags[F_NL_OVERFLOW];  // (waited for after the loads)
  __shared__ double sh[P_COUNT][kEnergyThreads];
  __shared__ double tot[P_COUNT];
  __shared__ int last;
  const bool pair = mode & (EM_PAIR_GB | EM_PAIR_NB), pol = mode & (EM_PAIR_GB | EM_BORN_ENERGY | EM_PAIR_GB_SLOW);
  const bool nb = mode & EM_PAIR_NB, bonded = mode & EM_BONDED, surf = mode & EM_SURF, kin = mode & EM_KINETIC;
  const unsigned slots = (pair ? 1u << P_VDW | 1u << P_ELEC : 0u) | (pol ? 1u << P_POL | 1u << P_SELF : 0u) |
                         (nb ? 1u << P_NBVIR : 0u) | (kin ? 1u << P_KIN : 0u) | (surf ? 1u << P_SURF : 0u) |
                         (bonded ? 1u << P_BOND | 1u << P_BVIR | 1u << P_ANGLE | 1u << P_DIH : 0u);
  const double *ep = v.ebuf ? v.e_pair_alt : v.e_atom;  // the pair slots of this energy buffer
  int *sflags = v.ebuf ? v.sys_flags_alt : v.sys_flags;
  double *E = v.ene + (size_t)s * E_COUNT;
  const int x = threadIdx.x;
  // the record, the step counter and the system's flags, read beside the
  // ranges (nothing else writes them meanwhile)
  __shared__ double sE[E_COUNT];
  __shared__ int sflag, sk;
  static_assert(E_COUNT <= 30, "one lane per record slot");
  if (warp == kEnergyWarps - 1) {
    if (lane < E_COUNT) sE[lane] = __ldcg(E + lane);
    if (lane == 30) sflag = __ldcg(sflags + s);
    if (lane == 31 && (mode & EM_RECORD)) sk = __ldcg(step_dev + SD_STEP) - __ldcg(step_dev + SD_FIRST);
  }
  if (pair) {
    sh[P_VDW][x] = chunk_sum(ep + (size_t)AE_VDW * N, lo[0], hi[0]);
    sh[P_ELEC][x] = chunk_sum(ep + (size_t)AE_ELEC * N, lo[0], hi[0]);
  }
  if (pol) {
    sh[P_POL][x] = chunk_sum(ep + (size_t)AE_POL * N, lo[0], hi[0]);
    sh[P_SELF][x] = chunk_sum(ep + (size_t)AE_POL_SELF * N, lo[0], hi[0]);
  }
  if (nb) sh[P_NBVIR][x] = chunk_sum(v.e_atom + (size_t)AE_VIR * N, lo[0], hi[0]);
  if (surf) sh[P_SURF][x] = chunk_sum(v.e_atom + (size_t)AE_SURF * N, lo[0], hi[0]);
  if (kin) sh[P_KIN][x] = chunk_sum(v.e_atom + (size_t)AE_KIN * N, lo[0], hi[0]);
  if (bonded) {
    const BondedTerms &t = v.bt;
    const size_t alt = v.ebuf ? 1 : 0;
    sh[P_BOND][x] = chunk_sum(t.e_bond + alt * t.nb, lo[1], hi[1]);
    sh[P_BVIR][x] = chunk_sum(t.vir_bond + alt * t.nb, lo[1], hi[1]);
    sh[P_ANGLE][x] = chunk_sum(t.e_angle + alt * t.na, lo[2], hi[2]);
    // torsions and impropers share the dihedral array: two ranges
    const double *dih = t.e_dih + alt * (t.nt + t.ni);
    sh[P_DIH][x] = chunk_sum(dih, lo[3], hi[3]) + chunk_sum(dih, lo[4], hi[4]);
  }
  if (overflow) return;
  __syncthreads();
  double *part = v.e_part + (size_t)s * C * P_COUNT;
  for (int k = warp; k < P_COUNT; k += kEnergyWarps) {
    double t = 0.0;
    if ((slots >> k) & 1u) {
#pragma unroll
      for (int q = 0; q < kEnergyWarps; q++) t += sh[k][32 * q + lane];
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (lane == 0) {
      if (mine == 1)
        tot[k] = t;
      else
        part[(size_t)c * P_COUNT + k] = t;
    }
  }
  if (mine > 1) {
    // the last block of this system to finish forms the record: warp w adds
    // slot w (of P_COUNT) over the chunks, lane l the chunks l, l + 32, ...
    // (loads in parallel), then a fixed shuffle tree
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&v.e_done[s], 1) == mine - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = warp; k < P_COUNT; k += kEnergyWarps) {
      double t = 0.0;
      if ((slots >> k) & 1u) {
        for (int q = lane; q < mine; q += 32) t += __ldcg(part + (size_t)q * P_COUNT + k);
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      if (lane == 0) tot[k] = t;
    }
    if (threadIdx.x == 0) v.e_done[s] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double R[E_COUNT];  // in registers: the sums below are a chain
#pragma unroll
    for (int k = 0; k < E_COUNT; k++) R[k] = sE[k];
    if (mode & EM_ASSIGN)  // as WorkSpace::zeroForces left it
#pragma unroll
      for (int k = 0; k < E_COUNT; k++)
        if (k != E_EKIN) R[k] = 0.0;
    if (mode & (EM_PAIR_GB | EM_PAIR_NB)) {
      R[E_VDW] = tot[P_VDW];
      R[E_ELEC] = tot[P_ELEC];
      R[E_EPOT] += tot[P_VDW] + tot[P_ELEC];
    }
    if (mode & EM_PAIR_GB) {
      R[E_POL] += tot[P_POL] + tot[P_SELF];
      R[E_POL_CROSS] += tot[P_POL];
      R[E_POL_SELF] += tot[P_SELF];
      R[E_EPOT] += tot[P_POL] + tot[P_SELF];
    }
    if (mode & EM_PAIR_NB) R[E_VIRIAL] += tot[P_NBVIR];
    if (mode & EM_PAIR_GB_SLOW) {
      // calcBornForces adds its energy to epot alone (gbff.cpp:1340); the
      // component's own totals go to the extra slots
      R[E_EPOT] += tot[P_POL] + tot[P_SELF];
      R[E_GB_COMPONENT] = tot[P_POL] + tot[P_SELF];
      R[E_GB_COMPONENT + 1] = tot[P_POL];
      R[E_GB_COMPONENT + 2] = tot[P_SELF];
    }
    if (mode & EM_BORN_ENERGY) {
      // the energy-only path adds the Born energy to epot alone
      // (gbff.cpp:574-578); the component's own totals go to extra slots
      R[E_EPOT] += tot[P_POL] + tot[P_SELF];
      R[E_GB_COMPONENT] = tot[P_POL] + tot[P_SELF];
      R[E_GB_COMPONENT + 1] = tot[P_POL];
      R[E_GB_COMPONENT + 2] = tot[P_SELF];
    }
    if (mode & EM_BONDED) {
      R[E_BOND] += tot[P_BOND];
      R[E_ANGLE] += tot[P_ANGLE];
      R[E_TORSION] += tot[P_DIH];
      R[E_VIRIAL] += tot[P_BVIR];
      R[E_EPOT] += tot[P_BOND] + tot[P_ANGLE] + tot[P_DIH];
    }
    if (mode & EM_SURF) {  // FF_SASA_LCPO adds epot_cav to epot and epot_surf
      R[E_SURF] += tot[P_SURF];
      R[E_EPOT] += tot[P_SURF];
    }
    if (mode & EM_KINETIC) {
      R[E_EKIN] = tot[P_KIN] * J2kcalmol;
      R[E_ETOT] = R[E_EPOT] + R[E_EKIN];
    }
    if (sflag & SF_NONFINITE) R[E_EPOT] = __longlong_as_double(0x7ff8000000000000LL);  // NaN
    if (!(R[E_EPOT] == R[E_EPOT])) atomicExch(&v.flags[F_NAN], 1);
    if (ctl.ms) min_control(v, ctl.ms[s], ctl, R[E_EPOT]);
#pragma unroll
    for (int k = 0; k < E_COUNT; k++) sE[k] = R[k];
  }
  __syncthreads();
  if (warp == 0) {
    if (lane < E_COUNT) E[lane] = sE[lane];
    if (lane == 31) sflags[s] = 0;  // consumed
    if ((mode & EM_RECORD) && lane < 3) {
      double *h = hist + ((size_t)sk * v.n_sys + s) * 3;
      h[lane] = sE[lane == 0 ? E_EPOT : lane == 1 ? E_EKIN : E_ETOT];
    }
    // the last system to finish advances the step (every block has read
    // SD_STEP before it counts itself finished)
    if ((mode & EM_RECORD) && lane == 0) {
      __threadfence();
      int done = atomicAdd(&step_dev[SD_DONE], 1);
      if (done == v.n_sys - 1) {
        step_dev[SD_DONE] = 0;
        if (mode & EM_GATE) {
          step_dev[SD_BLOCK] = __ldcg(step_dev + SD_STEP) + 1;
          if (__ldcg(&v.flags[F_NAN]) || __ldcg(&v.flags[F_LCPO_CAND]))
            atomicExch(&v.flags[F_NL_OVERFLOW], kGateShut);
        }
        __threadfence();
        atomicAdd(&step_dev[SD_STEP], 1);
      }
    }
  }
}

void launch_energy(const PackView &v, cudaStream_t st, int mode, double *hist, int *step_dev, const MinCtl *ctl) {
  if (!v.n_sys) return;
  const Consts &k = consts();
  int C = v.e_chunks;
  PDGPU_LAUNCH_DEP(k_energy, dim3(C, v.n_sys), kEnergyThreads, 0, st, v, mode, C, k.J2kcal * k.Na, hist, step_dev,
                   ctl ? *ctl : MinCtl());
}

}  // namespace pdgpu
