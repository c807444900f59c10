// MD integrators, kinetic energy, velocity initialisation and the
// minimiser's device-side control flow.
//
//   Langevin        MolecularDynamics::applyForces_LangevinIntegration (md.cpp:906-1042)
//   Langevin non-H  applyForces_LangevinIntegration_NonHydrogens        (md.cpp:1048-1218)
//   VelocityVerlet  applyForces_VelocityVerletIntegration               (md.cpp:788-838)
//   Beeman          applyForces_BeemanIntegration                       (md.cpp:841-902)
//   Verlet          applyForces_VerletIntegration                       (md.cpp:748-786)
//   KE              calcKineticEnergy                                   (md.cpp:504-539)
//   init velocities setInitialSpeeds                                    (md.cpp:342-363)
//   SD / CG         Minimisation::doSteepestDescentStep / doConjugateGradientStep
//                   (minimise.cpp:181-318) and the runcore bookkeeping (:99-179)
//
// State is FP64 (positions in Angstrom, velocities in m/s, forces converted
// from the fixed-point accumulators to N), as in the reference.  Random
// normals come from a counter-based Philox4x32-10 generator keyed by the
// system's seed and indexed by (system-local atom, step), so a system's
// trajectory does not depend on which other systems share its launch.
// Roofline: HBM-bound, 152 B/atom/step algorithmic traffic.
#include <cuda_runtime.h>
#include <cstddef>

#include "mdatom.cuh"
#include "minstep.cuh"

namespace pdgpu {

// One integrator step for every atom of the pack.  KE per atom goes to
// e_atom[AE_KIN] and is reduced per system afterwards.
// The thermostat's normals depend on the step, the atom and its system's key
// only, so they are drawn before the wait for the force passes (under a
// programmatic dependent launch, beside the last pass's tail).  The step is the
// block's first one, which stays while the block runs, and the number of this
// launch in it: the counter itself is advanced by the previous step's record,
// which may still run (in a graph every edge into this launch is programmatic,
// the one from that record too).  The atom's mass, velocity and position (the
// previous step's, complete before this step's first phase passed its own
// wait) and the noise widths of its mass are ready before the wait too; after
// it come the nine force loads and the update.
__global__ void k_md_step(PackView v, MDDev d, const double *normals, const int *step_dev) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < v.n_atoms;
  const int step = !live ? 0 : step_dev ? step_dev[SD_BLOCK] + d.c.step : d.c.step;
  double nr[6];
  const bool pre = live && !normals && md_draws_normals(v, d, step, i);
  MDIn in;
  if (live) md_load(v, d, i, in);
  if (pre) md_normals(v, d, step, i, nr);
  PDGPU_DEP_ENTRY();
  if (!live || v.flags[F_NL_OVERFLOW]) return;  // forces incomplete: keep the state, host re-plans
  v.e_atom[(size_t)AE_KIN * v.n_atoms + i] = md_atom(v, d, normals, step, i, in, pre ? nr : nullptr);  // J
}

// Kinetic energies from the current velocities: every atom's (J) and each
// system's total into its record, as an energy record with kinetic energies
// alone would leave it.  The total scales the initial velocities, so its order
// of addition is part of every trajectory: 256-atom chunks (a shuffle tree per
// 32 atoms, the eight in order), then lane l of a warp the chunks l, l + 32,
// ... and a shuffle tree.  A block takes 16 chunks, four atoms a thread at
// once; a larger system's blocks leave their chunks' sums to its last one.
// Bound by latency.  A call of pdgpu_md_init_velocities (four kernels and a
// synchronisation), one block walking a system / this form: 2,972 atoms 31 / 30
// us, 20,566 57 / 32, 97,336 183 / 33, 512,000 850 / 50; 256 peptides 36 / 35.
constexpr int kKinChunk = 256, kKinThreads = 1024;
constexpr int kKinChunks = kReduceChunk / kKinChunk, kKinItems = kReduceChunk / kKinThreads;
static_assert(kKinChunks <= kPartSlots && kKinChunks <= 32, "a block's sums fit its partials and a warp");
__global__ void __launch_bounds__(kKinThreads) k_kinetic_record(PackView v, double J2kcalmol, int C) {
  __shared__ double sh[kReduceChunk / 32];
  const int s = blockIdx.y, a1 = v.atom_off[s + 1], a0 = v.atom_off[s], b = a0 + blockIdx.x * kReduceChunk;
  const int mine = (a1 - a0 + kReduceChunk - 1) / kReduceChunk;  // this system's blocks
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool skip = v.flags[F_NL_OVERFLOW];  // the record keeps its state
  if ((int)blockIdx.x >= mine) return;
  double ke[kKinItems];
#pragma unroll
  for (int r = 0; r < kKinItems; r++) {
    const int i = b + r * kKinThreads + (int)threadIdx.x;
    ke[r] = 0.0;
    if (i < a1) {
      const double vx = v.vx[i], vy = v.vy[i], vz = v.vz[i];
      ke[r] = 0.5 * v.mass_si[i] * (vx * vx + vy * vy + vz * vz);
      v.e_atom[(size_t)AE_KIN * v.n_atoms + i] = ke[r];
    }
  }
#pragma unroll
  for (int r = 0; r < kKinItems; r++) {
    for (int o = 16; o > 0; o >>= 1) ke[r] += __shfl_xor_sync(0xffffffffu, ke[r], o);
    if (lane == 0) sh[r * (kKinThreads / 32) + warp] = ke[r];
  }
  __syncthreads();
  if (warp != 0) return;
  double acc = 0.0;
  if (lane < kKinChunks)
    for (int w = 0; w < kKinChunk / 32; w++) acc += sh[lane * (kKinChunk / 32) + w];  // (past the end: zeros)
  if (mine > 1) {
    double *part = v.e_part + (size_t)s * C * kKinChunks;
    if (lane < kKinChunks) part[(size_t)blockIdx.x * kKinChunks + lane] = acc;
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(&v.e_done[s], 1) == mine - 1;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    acc = 0.0;
#pragma unroll 4
    for (int q = lane; q < mine * kKinChunks; q += 32) acc += __ldcg(part + q);
    if (lane == 0) v.e_done[s] = 0;
  }
  if (skip) return;
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane) return;
  double *E = v.ene + (size_t)s * E_COUNT;
  E[E_EKIN] = acc * J2kcalmol;
  E[E_ETOT] = E[E_EPOT] + E[E_EKIN];
  if (v.sys_flags[s] & SF_NONFINITE) E[E_EPOT] = __longlong_as_double(0x7ff8000000000000LL);  // NaN
  if (!(E[E_EPOT] == E[E_EPOT])) atomicExch(&v.flags[F_NAN], 1);
  v.sys_flags[s] = 0;  // consumed
}

// setInitialSpeeds: Boltzmann draw (two nrand pairs, the second overwriting
// vy as the reference does, md.cpp:353-356); then rescale to 3/2 N kB T.
__global__ void k_vel_init(PackView v, double kB, double temp, const unsigned long long *sys_seed) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  int s = v.sys_of[i];
  double nr[6];
  six_normals(sys_seed[s] ^ 0x5EEDull, i - v.atom_off[s], -1, nr);
  double sigma = sqrt(kB * temp / v.mass_si[i]);
  double vx = nr[0] * sigma, vy = nr[1] * sigma;
  vy = nr[2] * sigma;  // nrand(vy, vz): second pair overwrites vy
  double vz = nr[3] * sigma;
  v.vx[i] = vx;
  v.vy[i] = vy;
  v.vz[i] = vz;
}
__global__ void k_vel_scale(PackView v, double kB, double temp, double kcal2J_per_mol) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  int s = v.sys_of[i];
  int n = v.atom_off[s + 1] - v.atom_off[s];
  double ekin = v.ene[(size_t)s * E_COUNT + E_EKIN] * kcal2J_per_mol;  // J
  double edes = 3 * n * kB * temp / 2;
  double chi = sqrt(edes / ekin);
  v.vx[i] *= chi;
  v.vy[i] *= chi;
  v.vz[i] *= chi;
}

// --------------------------------------------------------------- minimiser
// CG dot products: per (256-atom chunk, system) partials of fmagold = sum of
// of.of and fmagnew = sum of (of-f).f; the last block of each system to finish
// adds them in a fixed order into its state, before the energy record whose
// last block takes the step's decision (min_control).  An atom per thread: a
// step waits for this launch and its blocks for twelve loads an atom, which
// the record's 4,096-item chunks made sixteen times in a row.  A step's share
// (CG step minus SD step), 4,096 items -> 256: 985 atoms 7.2 -> 4.0 us, 2,972
// 14.2 -> 3.6, 20,566 17.2 -> 5.5.  A system of one chunk needs no second stage.
constexpr int kDotChunk = 256;
static_assert(2 * (kReduceChunk / kDotChunk) <= kPartSlots, "two partials a chunk fit the reduction buffer");
__global__ void __launch_bounds__(kDotChunk) k_min_dots(PackView v, MinState *ms, double N_per_unit, int C) {
  const int c = blockIdx.x, s = blockIdx.y;
  const int i = v.atom_off[s] + c * kDotChunk + threadIdx.x, end = v.atom_off[s + 1];
  const int mine = (end - v.atom_off[s] + kDotChunk - 1) / kDotChunk;  // this system's chunks
  PDGPU_DEP_ENTRY();
  if (v.flags[F_NL_OVERFLOW] || c >= mine) return;
  __shared__ double sa[kDotChunk], sb[kDotChunk];
  double A = 0, B = 0;
  if (i < end) {
    double f[3] = {force_N(v.fx[i], v.gx[i], v.hx[i]) * N_per_unit, force_N(v.fy[i], v.gy[i], v.hy[i]) * N_per_unit,
                   force_N(v.fz[i], v.gz[i], v.hz[i]) * N_per_unit};
    double of[3] = {v.fox[i], v.foy[i], v.foz[i]};
    A += of[0] * of[0] + of[1] * of[1] + of[2] * of[2];
    B += (of[0] - f[0]) * f[0] + (of[1] - f[1]) * f[1] + (of[2] - f[2]) * f[2];
  }
  sa[threadIdx.x] = A;
  sb[threadIdx.x] = B;
  __syncthreads();
  for (int w = kDotChunk / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      sa[threadIdx.x] += sa[threadIdx.x + w];
      sb[threadIdx.x] += sb[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (mine == 1) {
    if (threadIdx.x == 0) {
      ms[s].fmagold = sa[0];
      ms[s].fmagnew = sb[0];
    }
    return;
  }
  double *part = v.e_part + (size_t)s * C * 2;
  if (threadIdx.x == 0) {
    part[2 * (size_t)c] = sa[0];
    part[2 * (size_t)c + 1] = sb[0];
  }
  // the last block of the system adds the chunk partials (lanes strided over
  // the chunks, then a fixed shuffle tree)
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&v.e_done[s], 1) == mine - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 2) {
    double t = 0.0;
    for (int q = lane; q < mine; q += 32) t += __ldcg(part + 2 * (size_t)q + warp);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) (warp == 0 ? ms[s].fmagold : ms[s].fmagnew) = t;
  }
  if (threadIdx.x == 0) v.e_done[s] = 0;
}

// The step of every atom by its system's decision.  Positions and forces are
// older than the energy record this launch follows (the forces were complete
// before it), so they are read before the wait and only the decision after it.
__global__ void k_min_update(PackView v, const MinState *ms, double N_per_unit, double step_size) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  int s = v.sys_of[i];
  double f[3] = {force_N(v.fx[i], v.gx[i], v.hx[i]) * N_per_unit, force_N(v.fy[i], v.gy[i], v.hy[i]) * N_per_unit,
                 force_N(v.fz[i], v.gz[i], v.hz[i]) * N_per_unit};
  double p[3] = {v.x[i], v.y[i], v.z[i]};
  PDGPU_DEP_ENTRY();
  const MinState &m = ms[s];
  const int a = m.action;
  if (a < 0 || v.flags[F_NL_OVERFLOW]) return;  // (no valid forces: nothing moves, the host retries)
  double sc = step_size * m.mult;
  if (a == 0) {  // SD accept (or first step): save p, f; step along f
    v.ox[i] = p[0];
    v.oy[i] = p[1];
    v.oz[i] = p[2];
    v.fox[i] = f[0];
    v.foy[i] = f[1];
    v.foz[i] = f[2];
    for (int k = 0; k < 3; k++) p[k] += f[k] * sc;
  } else if (a == 1) {  // SD reject: restore p (the restored force is recomputed next step)
    p[0] = v.ox[i];
    p[1] = v.oy[i];
    p[2] = v.oz[i];
  } else if (a == 2) {  // CG reject: restore p, step along the current direction
    p[0] = v.ox[i] + v.dirx[i] * sc;
    p[1] = v.oy[i] + v.diry[i] * sc;
    p[2] = v.oz[i] + v.dirz[i] * sc;
  } else {  // 3: CG accept (new direction), 4: first CG step
    double d[3];
    if (a == 3) {
      d[0] = v.odx[i] * m.gamma + f[0];
      d[1] = v.ody[i] * m.gamma + f[1];
      d[2] = v.odz[i] * m.gamma + f[2];
    } else {
      d[0] = f[0];
      d[1] = f[1];
      d[2] = f[2];
    }
    v.dirx[i] = d[0];
    v.diry[i] = d[1];
    v.dirz[i] = d[2];
    v.odx[i] = d[0];
    v.ody[i] = d[1];
    v.odz[i] = d[2];
    v.ox[i] = p[0];
    v.oy[i] = p[1];
    v.oz[i] = p[2];
    v.fox[i] = f[0];
    v.foy[i] = f[1];
    v.foz[i] = f[2];
    for (int k = 0; k < 3; k++) p[k] += d[k] * sc;
  }
  store_pos(v, i, p[0], p[1], p[2]);
}

// end of runcore: cur = old (the last accepted positions)
__global__ void k_min_restore_best(PackView v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.n_atoms) return;
  store_pos(v, i, v.ox[i], v.oy[i], v.oz[i]);
}

// --------------------------------------------------------------- launchers
void launch_md_step_impl(const PackView &v, cudaStream_t st, const MDCoef &c, const double *normals,
                         const int *step_dev, const unsigned char *is_h, const unsigned long long *seeds,
                         double *frames, int frame_every, int frame_cap) {
  MDDev d = make_md_dev(c, is_h, seeds);
  d.frames = frames;
  d.frame_every = frames ? frame_every : 0;
  d.frame_cap = frame_cap;
  // 64-thread blocks: a 20k-atom system spreads over every SM
  if (v.n_atoms) PDGPU_LAUNCH_DEP(k_md_step, (v.n_atoms + 63) / 64, 64, 0, st, v, d, normals, step_dev);
}

std::atomic<long long> &launch_counter() {
  static std::atomic<long long> n{0};
  return n;
}
static thread_local long long tl_captured = -1;  // -1: this thread is not capturing
void count_launch() {
  if (tl_captured >= 0)
    tl_captured++;
  else
    launch_counter()++;
}
bool pdl_enabled() {
  static const bool on = [] {
    const char *e = getenv("PDGPU_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}
void begin_capture_count() { tl_captured = 0; }
long long end_capture_count() {
  long long n = tl_captured;
  tl_captured = -1;
  return n;
}
void launch_ke_from_velocities(const PackView &v, cudaStream_t st) {
  if (!v.n_atoms) return;
  const Consts &k = consts();
  const int C = (v.max_sys_atoms + kReduceChunk - 1) / kReduceChunk;
  PDGPU_LAUNCH(k_kinetic_record, dim3(C, v.n_sys), kKinThreads, 0, st, v, k.J2kcal * k.Na, C);
}
void launch_vel_init_impl(const PackView &v, cudaStream_t st, double temp, const unsigned long long *seeds) {
  const Consts &k = consts();
  if (!v.n_atoms) return;
  PDGPU_LAUNCH(k_vel_init, (v.n_atoms + 255) / 256, 256, 0, st, v, k.kB, temp, seeds);
  launch_ke_from_velocities(v, st);
  PDGPU_LAUNCH(k_vel_scale, (v.n_atoms + 255) / 256, 256, 0, st, v, k.kB, temp, k.kcal2J / k.Na);
  launch_ke_from_velocities(v, st);
}
MinCtl min_ctl(void *ms, int algorithm, double slope_kcal, double strict_kcal, int nsteps) {
  const Consts &k = consts();
  MinCtl c;
  c.ms = (MinState *)ms;
  c.algorithm = algorithm;
  c.nsteps = nsteps;
  c.slope_kcal = slope_kcal;
  c.strict_kcal = strict_kcal;
  c.J_unit = k.J2kcal * k.Na;
  return c;
}
void launch_min_dots(const PackView &v, cudaStream_t st, const MinCtl &c) {
  if (c.algorithm != PDGPU_MIN_CONJUGATE_GRADIENTS) return;
  const int C = (v.max_sys_atoms + kDotChunk - 1) / kDotChunk;
  if (C) PDGPU_LAUNCH_DEP(k_min_dots, dim3(C, v.n_sys), kDotChunk, 0, st, v, c.ms, consts().N_per_kcalmolA, C);
}
void launch_min_update(const PackView &v, cudaStream_t st, const MinCtl &c, double step_size) {
  if (v.n_atoms)
    PDGPU_LAUNCH_DEP(k_min_update, (v.n_atoms + 63) / 64, 64, 0, st, v, c.ms, consts().N_per_kcalmolA, step_size);
}
void launch_min_finish(const PackView &v, cudaStream_t st) {
  if (v.n_atoms) PDGPU_LAUNCH(k_min_restore_best, (v.n_atoms + 255) / 256, 256, 0, st, v);
}
size_t min_state_size() { return sizeof(MinState); }
int min_state_last(const void *host_buf, int s) { return ((const MinState *)host_buf)[s].last; }
StepSrc min_step_src(const void *ms, bool last) {
  static_assert(sizeof(MinState) % sizeof(int) == 0, "MinState is a whole number of ints");
  StepSrc r;
  r.p = (const int *)((const char *)ms + (last ? offsetof(MinState, last) : offsetof(MinState, step)));
  r.stride = (int)(sizeof(MinState) / sizeof(int));
  return r;
}
void min_state_init(void *host_buf, int n) {
  MinState *m = (MinState *)host_buf;
  for (int s = 0; s < n; s++) {
    m[s] = MinState{};
    m[s].mult = 1.0;
  }
}
void min_state_read(const void *host_buf, int s, int *taken, int *nan, double *mult) {
  const MinState *m = (const MinState *)host_buf;
  *taken = m[s].taken;
  *nan = m[s].nan;
  *mult = m[s].mult;
}

}  // namespace pdgpu
