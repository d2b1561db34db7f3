// Nodal update and time-step logic of one node / one instance, shared by the nodal kernels
// (dnl_host.cu) and the batch's persistent step kernel (dnl_elem.cu):
//   node_update  the CSR gather of the element forces + ExplicitSolverCH::computePredictions
//                (ExplicitSolverCH.C:387-431), explicitSolve (:490-545), updateGrid (:555-567) and
//                the constant boundary conditions (Boundary.C:478-525, 636-665), in the
//                reference's operation order, products added by fma;
//   dt_update    Solver::computeTimeStep (Solver.C:220-267), ExplicitSolverCH::initStep
//                (:434-447), updateTime and Solver::betweenTimeBounds.
// Every product and sum is written with an explicit rounding intrinsic or fma, so the code rounds
// the same in every translation unit whatever its contraction flags.
#pragma once

#include "dnl_common.cuh"

namespace dnl {

// ----------------------------------------------------------------------------- nodal update
// The step's products of the update: dt (1/2 - beta), dt (1 - gamma), dt gamma, dt^2 beta
struct NodeDt {
  double dt, c1, c2, cg, cb;
};
__device__ __forceinline__ NodeDt node_dt(double dt, const NodeConst &p)
{
  return {dt, __dmul_rn(dt, p.hb), __dmul_rn(dt, p.hg), __dmul_rn(dt, p.gamma), __dmul_rn(__dmul_rn(dt, dt), p.beta)};
}
// the same for a block that shares one time step, four lanes of its first warp one product each (two
// FP64 instructions of the pipe instead of five); contains a barrier
__device__ __forceinline__ NodeDt node_dt_block(double dt, const NodeConst &p)
{
  __shared__ double c[4];
  if (threadIdx.x < 4) {
    const int l = threadIdx.x;
    const double f = l == 0 ? p.hb : l == 1 ? p.hg : l == 2 ? p.gamma : p.beta;
    const double dt2 = __dmul_rn(dt, dt);
    c[l] = __dmul_rn(l == 3 ? dt2 : dt, f);
  }
  __syncthreads();
  return {dt, c[0], c[1], c[2], c[3]};
}

// sum of the element forces' component fe over a node's slots, in ascending element order; eight
// slots' loads are in flight at a time (one by one, each add waited for two dependent loads)
__device__ __forceinline__ double gather_sum(const double *fe, const int *entry, int b, int e)
{
  double f = 0.0;
  for (int q = b; q < e; q += 8) {
    int ent[8];
    double v[8];
    const int n = e - q;
#pragma unroll
    for (int k = 0; k < 8; k++) ent[k] = __ldg(entry + q + (k < n ? k : 0));
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = fe[ent[k]];
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (k < n) f = __dadd_rn(f, v[k]);
  }
  return f;
}

// Component c of node n of the Chung-Hulbert update.  One thread per component: the FP64 pipe bounds
// this kernel (22 FP64 instructions per component of a node with eight elements, 64 cycles each), and
// on small meshes its latency, which is a third or half per thread that way.  In 2D the third
// components of the nodal fields stay 0 (nothing writes them).  Products are added by fma, with one
// rounding.  Against one thread per node, loads and adds of the gather alternating, masses inverted
// here: 539,000 nodes of hexahedra 108 -> 96 us, a step of 306 nodes and 250 quads 30.5 -> 26.4 us,
// a step of a tetrahedral bar, 24 elements to a node, 47 -> 37 us.  The two divisions of the
// corrector, F/M and (. - alphaM a)/(1 - alphaM), go through a reciprocal (the mass's is stored
// beside it) and one residual correction (quot).
template <int DIM>
__device__ __forceinline__ void node_update(const NodeArgs &g, int n, int c, const NodeConst &p, const NodeDt &k)
{
  double cv = g.cur.v[c][n], ca = g.cur.a[c][n];
  const double cd = g.cur.disp[c][n], x = g.x[c][n];
  const double m = g.mass[n], rm = g.mass[(long)g.N + n];
  const int bc = g.bcIdx[n];
  const int act = bc >= 0 ? (g.bcCode[bc] >> (2 * c)) & 3 : 0;  // 1 restrained, 2 imposed speed
  // computePredictions
  double ndu = __dmul_rn(fma(ca, k.c1, cv), k.dt);
  double nv = fma(ca, k.c2, cv);
  if (act) ca = 0.;
  // assembled internal forces
  const double f = gather_sum(g.fe + (long)c * g.EN, g.entry, g.start[n], g.start[n + 1]);
  if (g.fint) g.fint[(long)n * DIM + c] = f;
  // explicitSolve
  double na = quot(f, m, rm);
  na = quot(fma(-p.alphaM, ca, na), p.oma, p.roma);
  nv = fma(k.cg, na, nv);
  ndu = fma(k.cb, na, ndu);
  if (act) {
    const double s = act == 2 ? g.bcSpeed[3 * bc + c] : 0.;
    na = 0.;
    nv = s;
    ndu = act == 2 ? __dmul_rn(s, k.dt) : 0.;
  }
  g.nxt.du[c][n] = ndu;
  g.nxt.v[c][n] = nv;
  g.nxt.a[c][n] = na;
  g.nxt.disp[c][n] = __dadd_rn(cd, ndu);
  g.x[c][n] = __dadd_rn(x, ndu);
}

enum { DT_FORCE = 1, DT_POST = 2, DT_PRE = 4 };


__device__ __forceinline__ bool in_bounds(const DevTime *tm)
{
  const double up = tm->endTime < tm->upTime ? tm->endTime : tm->upTime;
  return tm->currentTime >= tm->startTime && tm->currentTime < up;
}

static __device__ void recompute_dt(DevTime *tm, int method, double safetyOmega, double Cs)
{
  double fmax;
  if (method == DNL_COURANT) {
    const double crit = __longlong_as_double((long long)tm->lenMinBits) / Cs;
    fmax = 2.0 / crit;
    tm->lenMinBits = 0x7ff0000000000000ull;  // +inf for the next reduction
  } else {
    fmax = tm->fmax;
  }
  tm->timeStep = safetyOmega / fmax;
  tm->lastTsDate = tm->tsDate;
  tm->lastTimeStep = tm->computedTimeStep;
  tm->tsDate = tm->currentTime;
  tm->computedTimeStep = tm->timeStep;
}

static __device__ void dt_update(DevTime *tm, int mode, int freq, int method, double safetyOmega, double Cs)
{
  if (tm->status) return;
  if (mode & DT_FORCE) recompute_dt(tm, method, safetyOmega, Cs);
  if ((mode & DT_POST) && !tm->done) {
    tm->currentTime = __dadd_rn(tm->currentTime, tm->timeStep);  // ExplicitSolverCH::updateTime
    if (!in_bounds(tm)) {
      tm->done = 1;
    } else if (tm->increment % freq == 0) {
      recompute_dt(tm, method, safetyOmega, Cs);
    } else if (tm->tsDate != tm->lastTsDate) {  // LINEARdbl extrapolation (Math.h:91)
      const double dx = __dsub_rn(tm->currentTime, tm->lastTsDate) / __dsub_rn(tm->tsDate, tm->lastTsDate);
      tm->timeStep = __dadd_rn(__dmul_rn(dx, tm->computedTimeStep), __dmul_rn(__dsub_rn(1.0, dx), tm->lastTimeStep));
    }
  }
  if ((mode & DT_PRE) && !tm->done) {
    if (!in_bounds(tm)) {
      tm->done = 1;
    } else {
      if (__dadd_rn(tm->currentTime, tm->timeStep) > tm->upTime) tm->timeStep = __dsub_rn(tm->upTime, tm->currentTime);
      tm->nextTime = __dadd_rn(tm->currentTime, tm->timeStep);
      tm->increment++;
    }
  }
  if (!tm->done && !(tm->timeStep > 0. && tm->timeStep < 1e300)) {
    tm->status = DNL_ERR_DT;
    tm->badElem = -1;
  }
}

// scheduled steps (dnl_sens_run, dnl_adjoint): phase 0 initStep with the scheduled step, 1
// updateTime, 2 both (updateTime of one step then initStep of the next)
static __device__ void sched_update(DevTime *tm, const double *dts, int phase)
{
  if (tm->status) return;
  if (phase != 0) tm->currentTime = __dadd_rn(tm->currentTime, tm->timeStep);
  if (phase != 1) {
    const double dt = dts[tm->increment];
    tm->timeStep = dt;
    tm->nextTime = __dadd_rn(tm->currentTime, dt);
    tm->increment++;
  }
}

// Called by every thread of every block of a kernel once its work is done: the block that arrives
// last runs the step's time logic, for which every other block has read the time record and written
// its part.  Saves a launch and the gap before it (about 3.5 us of a step) against a kernel of one
// thread.  The arrival counter is back at 0 afterwards, so every block must arrive, also where the run
// is over or has failed (the time logic looks at that itself).  Warp 0 of each block must not have left.
static __device__ void step_tail(const StepTail &t, DevTime *tm)
{
  if (!t.mode && !t.sched) return;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  unsigned last = 0;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&tm->arrived, 1u) + 1u == gridDim.x * gridDim.y;
    __threadfence();
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  __syncwarp();  // lane 0's fences order memory for the other lanes through this (a shuffle orders none)
  if (threadIdx.x == 0) tm->arrived = 0u;
  if (t.count) {
    for (int i = threadIdx.x; i < t.count; i += 32) {
      const InstParams &p = t.prm[i];
      dt_update(t.tms + i, t.mode, p.freq, p.method, p.safetyOmega, p.Cs);
    }
  } else if (threadIdx.x == 0) {
    if (t.sched)
      sched_update(tm, t.dts, t.sched);
    else
      dt_update(tm, t.mode, t.freq, t.method, t.safetyOmega, t.Cs);
  }
}

}  // namespace dnl
