// The minimiser's per-system control (Minimisation::runcore and its steps,
// minimise.cpp:99-318): the accept / restore decision of a step, taken by the
// energy record's last block where the step's energy is formed (energy.cu).
#pragma once
#include "internal.cuh"

namespace pdgpu {

struct MinState {
  double mult, old_energy, local_old, gamma, fmagold, fmagnew;
  int step, breakcount, done, action;  // action: 0 step, 1 restore-and-skip, 2 restore-then-step
  int taken, nan;
  int last;  // the last step the loop evaluated (WorkSpace::Step when the loop ends)
};

// The decision for one system on its potential energy (kcal/mol); one joule
// per molecule (the reference's "m_OldEnergy += 1" after a rejected SD step)
// is J_unit kcal/mol.
__device__ __forceinline__ void min_control(const PackView &v, MinState &m, const MinCtl &c, double epot) {
  if (m.done) {
    m.action = -1;
    return;
  }
  m.last = m.step;
  if (!(epot == epot)) {
    m.nan = 1;
    m.done = 1;
    m.action = -1;
    atomicExch(&v.flags[F_NAN], 1);
    return;
  }
  if (m.step == 0) m.local_old = epot;
  if (m.step > 0 && c.slope_kcal > 0.0) {
    double d = m.local_old - epot;
    if (d >= 0.0 && d < c.slope_kcal) m.breakcount++;
    m.local_old = epot;
  }
  if (m.breakcount > 10) {
    m.done = 1;
    m.action = -1;
    return;
  }
  if (c.algorithm == PDGPU_MIN_STEEPEST_DESCENT) {
    if (m.step != 0) {
      if (epot <= m.old_energy) {
        m.mult *= 1.2;
        m.old_energy = epot;
        m.action = 0;  // save then step
      } else {
        m.mult *= 0.5 / 1.2;
        m.old_energy += c.J_unit;
        m.action = 1;  // restore, no step
      }
    } else {
      m.old_energy = epot;
      m.action = 0;
    }
  } else {
    if (m.step != 0) {
      if ((m.mult < 0.05 && (epot - m.old_energy) < c.strict_kcal) || epot < m.old_energy) {
        m.mult *= 1.2;
        double g = m.fmagold != 0 ? m.fmagnew / m.fmagold : 0.0;
        if (g < 0) g = 0;
        m.gamma = g;
        m.old_energy = epot;
        m.action = 3;  // new direction, save, step
      } else {
        m.mult *= 0.5 / 1.2;
        m.action = 2;  // restore positions, step along the old direction
      }
    } else {
      m.old_energy = epot;
      m.action = 4;  // first step: direction = force
    }
  }
  m.step++;
  m.taken = m.step;
  if (m.step >= c.nsteps) m.done = 1;
}

}  // namespace pdgpu
