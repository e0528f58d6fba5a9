// wg_kernels.cu -- kernels of the GB300 WaterGAP2 daily step (sm_103a).
//
//  k_vertical      one thread per cell: calcNewDay for one day (daily.cpp:94-1257),
//                  the reference's per-day call granularity.
//  k_pipeline      persistent cooperative kernel: routing through the drainage
//                  tree as a wavefront over drainage levels.  With FUSED it also
//                  runs the vertical balance and pipelines days: cell n computes
//                  day d at step d + offset(n), offset = longest flow path -
//                  distance of n to its outlet.  Every upstream cell of n then
//                  has offset(n) - 1 and delivers day d's outflow exactly one step
//                  earlier.  A cell waits for these outflows themselves (one
//                  member, FP64 or FP32; rows of the outflow buffer per step), or
//                  all cells for a grid barrier per step (ensembles, GLWD units,
//                  runs with skipped cells) or, optionally, for per-warp step
//                  flags.  Cells
//                  without a water body take their vertical balance from the ring
//                  that k_vertical_ahead filled; the monthly output aggregates are
//                  accumulated in its epilogue.  With ENS the cells carry
//                  `members` independent states (ensemble members), innermost in
//                  memory.  With VAW (one FP64 member) each block's idle warp, any
//                  further warps it has room for and the routing warps that are
//                  done run k_vertical_ahead's work for the next chunk; with WT
//                  every cell also gets
//                  its water temperature (calcWTemp), the river temperature
//                  travelling downstream beside the outflow.
//  k_pet           potential evapotranspiration of a run's days, side by side,
//                  into the ring.
//  k_vertical_ahead  the vertical balance of the cells without a water body for
//                  a chunk of days, state in registers, into the ring.
//  k_state_rows / k_rows   state, output grids, water use and water temperature
//                  into cell order for reading.
//  k_fetch_row / k_keep_outflow / k_clear_skipped   the outflow rows that lie
//                  between the calls of a run.
//  k_math_eval     the FP64 path's exp/log/pow/reciprocal on arrays (tests).
//  k_unf_forcing / k_gather_forcing  forcing uploads into the slot layout.
//  k_volume / k_balance_sum   compensated (Neumaier) FP64 water-balance sums.
//
// Precision: R = double is the plain FP64 path; R = float keeps state and
// fluxes in FP32 while confluence sums, the outflow buffer and all balance
// sums stay FP64.  The grid barrier and the waits for outflows spin with an
// iteration limit: on timeout they raise the context's error word and every block
// returns (no trap).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "wg_device.h"
#include "wg_kernels.h"
#include "wg_physics.cuh"
#include "wg_volume.cuh"
#include "wg_wtemp.cuh"

namespace wg {

#define WG_BARRIER_SPIN_LIMIT (1u << 24)

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid-wide barrier for a cooperative launch (all blocks co-resident).  The
// counter only grows; round r completes when it reaches (r+1)*gridDim.x.
// Block-level part of the grid barrier: all threads of the block, or (nthr <
// blockDim.x) the first nthr threads only, on hardware barrier 1, while the
// block's other warps do independent work.
__device__ __forceinline__ void block_sync(int nthr) {
  if (nthr == (int)blockDim.x) __syncthreads();
  else asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
}

__device__ __forceinline__ bool grid_barrier(const DevSync &sync, unsigned round, int nthr) {
  block_sync(nthr);
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    const unsigned target = (round + 1u) * gridDim.x + sync.extra_arrivals;
    __threadfence();
    atomicAdd(sync.counter, 1u);
    unsigned it = 0;
    int ok = 1;
    while (ld_acquire(sync.counter) < target) {
      if (*(volatile int *)sync.error) { ok = 0; break; }
      if (++it > WG_BARRIER_SPIN_LIMIT) {
        atomicExch(sync.error, 1);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  block_sync(nthr);
  return s_ok != 0;
}

// An outflow (or river temperature) of the step before, which another thread writes.
// With sync.data it is its own signal: one 64-bit word, written and read with
// relaxed gpu-scope accesses, so that no ordering between words matters and no
// acquire empties the SM's L1 cache (the grid barrier's did, and every constant and
// state of the next step came back from L2).  The wait is bounded like the grid
// barrier's: when it runs out the error word is set and the caller stops.
#define WG_DATA_SPIN_LIMIT (1u << 20)
#ifndef WG_POLL_NS
#define WG_POLL_NS 100
#endif

__device__ __forceinline__ double ld_relaxed(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_outflow(double *p, double v) {
  if ((unsigned long long)__double_as_longlong(v) == kNoOutflow) v = __longlong_as_double(0x7ff8000000000000ll);
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ bool is_outflow(const DevSync &sync, double v) {
  return (unsigned long long)__double_as_longlong(v) != kNoOutflow && !sync.extra_arrivals;
}
__device__ __forceinline__ bool has_outflow(const DevSync &sync, const double *p) { return is_outflow(sync, ld_relaxed(p)); }

// One more poll of a warp (converged) or thread: true when the wait has run out, here
// or elsewhere in the grid.
__device__ __forceinline__ bool wait_ran_out(const DevSync &sync, unsigned &it) {
  if (++it <= WG_DATA_SPIN_LIMIT && ((it & 255u) != 0u || !*(volatile int *)sync.error)) return false;
  atomicExch(sync.error, 2);
  return true;
}

// The outflow itself.  WAIT (the per-day routing call, whose lanes each route one
// cell once): waiting for it if need be, failed when the wait runs out.  Else it is
// there, or belongs to an upstream cell that does not run.
template <bool WAIT>
__device__ __forceinline__ double upstream_value(const DevSync &sync, const double *p, bool &failed) {
  double v = ld_relaxed(p);
  if constexpr (WAIT) {
    unsigned it = 0;
    while (sync.data && !failed && ((unsigned long long)__double_as_longlong(v) == kNoOutflow || sync.extra_arrivals)) {
      failed = wait_ran_out(sync, it);
      v = ld_relaxed(p);
    }
  }
  return (unsigned long long)__double_as_longlong(v) == kNoOutflow ? 0. : v;
}

__device__ __forceinline__ int ld_acquire_int(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release_int(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Step flags: wait until every warp this warp depends on has completed step
// `need` (relative).  The lanes share the dependency list; bounded like the grid
// barrier (a wait that runs out sets the error word; the caller then stops).
__device__ __forceinline__ bool wait_deps(const DevSync &sync, int w, int need) {
  bool ok = true;
  const int k0 = sync.dep_ptr[w], k1 = sync.dep_ptr[w + 1];
  for (int k = k0 + (int)(threadIdx.x & 31); k < k1; k += 32) {
    const int *flag = sync.wstep + sync.dep_idx[k];
    unsigned it = 0;
    while (ld_acquire_int(flag) < need) {
      if (*(volatile int *)sync.error || ++it > WG_BARRIER_SPIN_LIMIT) {
        atomicExch(sync.error, 1);
        ok = false;
        break;
      }
      __nanosleep(32);
    }
    if (!ok) break;
  }
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void neumaier_add(double *acc, size_t k_sum, size_t k_comp, double x) {
  const double s = acc[k_sum];
  const double t = s + x;
  double c = acc[k_comp];
  if (fabs(s) >= fabs(x)) c += (s - t) + x;
  else c += (x - t) + s;
  acc[k_sum] = t;
  acc[k_comp] = c;
}

__device__ __forceinline__ void record_routing_balance(const DevBalance &b, size_t N, size_t i, double up,
                                                       double out, double leak) {
  neumaier_add(b.acc, 2 * N + i, 7 * N + i, out);
  neumaier_add(b.acc, 3 * N + i, 8 * N + i, up);
  neumaier_add(b.acc, 4 * N + i, 9 * N + i, leak);
}

__device__ __forceinline__ void record_balance(const DevBalance &b, size_t N, size_t i, double in, double evap,
                                               double up, double out, double leak) {
  neumaier_add(b.acc, 0 * N + i, 5 * N + i, in);
  neumaier_add(b.acc, 1 * N + i, 6 * N + i, evap);
  neumaier_add(b.acc, 2 * N + i, 7 * N + i, out);
  neumaier_add(b.acc, 3 * N + i, 8 * N + i, up);
  neumaier_add(b.acc, 4 * N + i, 9 * N + i, leak);
}

template <class R>
__device__ __forceinline__ RState<R> load_rstate(const DevStateT<R> &s, size_t i, uint32_t fl) {
  RState<R> r;
  r.gw = s.gw[i];
  r.river = s.river[i];
  r.loclake = (fl & F_LOCLAKE) ? s.loclake[i] : R(0);
  r.rf_loclake = (fl & F_LOCLAKE) ? s.rf_loclake[i] : R(0);
  r.locwetl = (fl & F_LOCWETL) ? s.locwetl[i] : R(0);
  r.rf_locwetl = (fl & F_LOCWETL) ? s.rf_locwetl[i] : R(0);
  r.glolake = (fl & F_GLOLAKE) ? s.glolake[i] : R(0);
  r.rf_glolake = (fl & F_GLOLAKE) ? s.rf_glolake[i] : R(0);
  r.glowetl = (fl & F_GLOWETL) ? s.glowetl[i] : R(0);
  r.rf_glowetl = (fl & F_GLOWETL) ? s.rf_glowetl[i] : R(0);
  r.res = (fl & F_RES) ? s.res[i] : R(0);
  r.rf_res = (fl & F_RES) ? s.rf_res[i] : R(0);
  r.k_release = (fl & F_RES) ? s.k_release[i] : R(0);
  return r;
}

// Store only what the cell's water bodies can have changed.
template <class R>
__device__ __forceinline__ void store_rstate(const DevStateT<R> &s, size_t i, const RState<R> &r, uint32_t fl) {
  s.gw[i] = r.gw;
  s.river[i] = r.river;
  if (fl & F_LOCLAKE) { s.loclake[i] = r.loclake; s.rf_loclake[i] = r.rf_loclake; }
  if (fl & F_LOCWETL) { s.locwetl[i] = r.locwetl; s.rf_locwetl[i] = r.rf_locwetl; }
  if (fl & F_GLOLAKE) { s.glolake[i] = r.glolake; s.rf_glolake[i] = r.rf_glolake; }
  if (fl & F_GLOWETL) { s.glowetl[i] = r.glowetl; s.rf_glowetl[i] = r.rf_glowetl; }
  if (fl & F_RES) { s.res[i] = r.res; s.rf_res[i] = r.rf_res; s.k_release[i] = r.k_release; }
}

// One cell-day of the vertical balance on state index si (slot s); rad: the
// radiation terms, for the output grids.
template <class R>
__device__ __forceinline__ void vertical_at(const DevCellsT<R> &c, const DevStateT<R> &st, size_t N, int s,
                                            size_t si, R Pin, R gamma_soil, float Tf, const Pet<R> &pet, R laf, R prev,
                                            VOut<R> &o, const VSink *vs = nullptr, const Radiation<R> *rad = nullptr,
                                            R ext_rad = R(0)) {
  if (c.flags[s] & F_NOCONT) {   // no vertical balance: the terms stay 0, the state as it is
    o.rs = R(0); o.gwr = R(0); o.transfer = R(0); o.owp = R(0); o.owpet = R(0);
    o.land_in = R(0); o.land_evap = R(0); o.land_leak = R(0);
    return;
  }
  R canopy = st.canopy[si], soil = st.soil[si], gsnow = st.snow[si], psum = st.lai_precsum[si];
  int days = st.lai_days[si], status = st.lai_status[si];
  if (vs)   // the output grids (FP64 single member)
    vertical_cell<R, std::is_same<R, double>::value>(c, s, gamma_soil, canopy, soil, gsnow, st.snow_band + si, N,
                                                      days, status, psum, laf, prev, Pin, Tf, pet, o, vs, rad, ext_rad);
  else
    vertical_cell<R>(c, s, gamma_soil, canopy, soil, gsnow, st.snow_band + si, N, days, status, psum, laf, prev, Pin,
                     Tf, pet, o);
  st.canopy[si] = canopy; st.soil[si] = soil; st.snow[si] = gsnow; st.lai_precsum[si] = psum;
  st.lai_days[si] = days; st.lai_status[si] = status;
}

// The radiation terms of slot s on a day of the year.
template <class R>
__device__ __forceinline__ Radiation<R> radiation_at(const DevCellsT<R> &c, int s, int doy, float Tf, float SWf) {
  const size_t ti = (size_t)(doy - 1) * c.nrow + c.ext_row[s];
  return radiation<R>(c, s, Tf, SWf, c.ext_rad[ti], c.inv_s0[ti]);
}

// Row of the ring for day d (a division only where the run is longer than the ring).
template <class R>
__device__ __forceinline__ size_t ring_row(const DevRingT<R> &ring, int d) {
  return (size_t)(d < ring.ring_days ? d : d % ring.ring_days);
}

template <class R>
__device__ __forceinline__ Pet<R> ring_pet(const DevRingT<R> &ring, size_t k) {
  return Pet<R>{ring.pet[k], ring.pet_snow[k], ring.pet_water[k]};
}

// Potential evapotranspiration of the days that the wavefront steps [t_b, t_e) will
// route, every cell, into the ring: it depends on the forcing alone, not on the
// state or the member, so it is taken out of the day-after-day chains of the
// vertical balance (which two thirds of its FP64 and integer instructions then
// leave) into a launch that runs all cell-days side by side.  A thread runs
// kPetDays days of its slot; the ring's rows are written coalesced where a warp's
// cells share their wavefront offset.  Bound by the integer pipe (fixed point): 1.2 ms
// per year of the global grid, where k_vertical_ahead went from 396 to 356 us and
// k_pipeline from 731 to 619 us per 20 days; 64 FP32 members for 90 days, which
// shared nothing of it before, 31.2 -> 29.0 ms.
constexpr int kPetDays = 8;
template <class R>
__global__ void __launch_bounds__(256) k_pet(DevCellsT<R> c, DevForcing f, DevRingT<R> ring, int doy0, int fday0,
                                             int ndays, int t_b, int t_e) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.n || (c.active && !c.active[s]) || (c.flags[s] & F_NOCONT)) return;
  const int kd = ring.days_per_step;
  const long long first = (long long)kd * (t_b - c.offset[s]) + (long long)blockIdx.y * kPetDays;
  const int d0 = (int)max(0ll, first);
  const int d1 = (int)min(min(first + kPetDays, (long long)kd * (t_e - c.offset[s])), (long long)ndays);
  for (int d = d0; d < d1; ++d) {
    const size_t fo = (size_t)(fday0 + d) * c.n + s, k = ring_row(ring, d) * c.n + s;
    const Pet<R> p = pet_of<R>(c, s, radiation_at<R>(c, s, (doy0 - 1 + d) % 365 + 1, f.temp[fo], f.swrad[fo]));
    ring.pet[k] = p.land;
    ring.pet_snow[k] = p.snow;
    ring.pet_water[k] = p.water;
  }
}

template <class R>
__global__ void __launch_bounds__(256) k_vertical(DevCellsT<R> c, DevStateT<R> st, DevVertT<R> v, DevForcing f,
                                                  int doy, int fday) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c.n || (c.active && !c.active[s])) return;
  const size_t fo = (size_t)fday * c.n + s;
  VOut<R> o;
  const R laf = st.laf[s];
  const R prev = (st.laf_started[s] == 1) ? st.laf_prev[s] : laf;   // daily.cpp:159-169
  const float Tf = f.temp[fo];
  const Pet<R> pet = pet_of<R>(c, s, radiation_at<R>(c, s, doy, Tf, f.swrad[fo]));
  vertical_at<R>(c, st, (size_t)c.n, s, (size_t)s, R(f.prec[fo]), c.gamma[s], Tf, pet, laf, prev, o);
  v.rs[s] = o.rs; v.gwr[s] = o.gwr; v.transfer[s] = o.transfer; v.owp[s] = o.owp; v.owpet[s] = o.owpet;
  v.land_in[s] = o.land_in; v.land_evap[s] = o.land_evap; v.land_leak[s] = o.land_leak;
}

// Vertical balance ahead of routing for the cells whose land fraction and open-water
// fluxes do not depend on routing (no water body): each thread takes one
// (cell, member) through the days the pipeline steps [t_b, t_e) will route, with
// the vertical state in registers, and leaves surface runoff and recharge in the
// ring buffer.  Results equal the in-wavefront computation: the vertical balance of
// such a cell reads nothing routing writes.
// One (cell, member) state index i of the vertical balance run ahead: the days
// the wavefront steps [t_b, t_e) will route, vertical state in registers, surface
// runoff and recharge into the ring; balance terms into arrays 0, 1 and 10.
// The output grids of state si for output day od: its entry in the vertical
// balance's monthly grids (the month of the output calendar, as the routing
// aggregates count it) and in the daily grids, each null when the grids are off
// or the day is outside them.  False: no grid takes the day.
__device__ __forceinline__ bool vert_sink(const DevMonthly &mon, int od, size_t si, size_t N, VSink &vs) {
  vs.mo = nullptr;
  vs.dd = nullptr;
  if (mon.vert) {
    const int yd = mon.doy_day0 - 1 + od;
    const int mi = (yd / 365) * 12 + month_of(yd % 365 + 1) - mon.month0;
    if (mi >= 0 && mi < mon.nmonths) vs.mo = mon.vert + (size_t)mi * N + si;
  }
  if (mon.dvert && od >= 0 && od < mon.dvert_days) vs.dd = mon.dvert + (size_t)od * N + si;
  vs.mos = (size_t)mon.nmonths * N;
  vs.dds = (size_t)mon.dvert_days * N;
  vs.vk = mon.vconst + si;
  vs.vks = N;
  return vs.mo || vs.dd;
}

template <class R, bool ENS>
__device__ __forceinline__ void va_cell(const DevCellsT<R> &c, const DevStateT<R> &st, const DevForcing &f,
                                        const DevMembers &mem, const DevBalance &b, const DevRingT<R> &ring,
                                        int doy0, int fday0, int ndays, int t_b, int t_e, size_t i, size_t N,
                                        const DevMonthly *mon = nullptr, int oday0 = 0) {
  const int n = c.n;
  const int M = ENS ? mem.members : 1;
  const int s = ENS ? (int)(i / M) : (int)i;
  const int mm = ENS ? (int)(i - (size_t)s * M) : 0;
  if ((c.flags[s] & F_VINLINE) || (c.active && !c.active[s])) return;
  const int off = c.offset[s];
  const int kd = ring.days_per_step;   // step t routes days kd*(t-off) .. kd*(t-off)+kd-1
  const int d0 = max(0, kd * (t_b - off)), d1 = min(ndays, kd * (t_e - off));
  if (d0 >= d1) return;
  R canopy = st.canopy[i], soil = st.soil[i], gsnow = st.snow[i], psum = st.lai_precsum[i];
  int days = st.lai_days[i], status = st.lai_status[i];
  const R laf = st.laf[i];   // constant for these cells (no water body)
  R pf = R(1), gam = c.gamma[s];
  if (ENS) {
    pf = R(mem.prec_factor[mm]);
    gam *= R(mem.gamma_factor[mm]);
  }
  double acc_in = 0., acc_ev = 0., acc_lk = 0.;
  const double land_f = (double)c.area_f[s] * (double)laf;
  for (int d = d0; d < d1; ++d) {
    const int doy = (doy0 - 1 + d) % 365 + 1;
    const size_t fo = (size_t)(fday0 + d) * n + s;
    const float Tf = f.temp[fo];
    const Pet<R> pet = ring_pet(ring, ring_row(ring, d) * n + s);
    VOut<R> o;
    VSink vs;
    if (!ENS && mon && vert_sink(*mon, oday0 + d, i, N, vs)) {   // the output grids (FP64 single member)
      const Radiation<R> rad = radiation_at<R>(c, s, doy, Tf, f.swrad[fo]);
      vertical_cell<R, std::is_same<R, double>::value, true>(c, s, gam, canopy, soil, gsnow, st.snow_band + i, N, days,
                                                        status, psum, laf, laf, R(f.prec[fo]) * pf, Tf, pet, o, &vs,
                                                        &rad, c.ext_rad[(size_t)(doy - 1) * c.nrow + c.ext_row[s]]);
    } else {
      vertical_cell<R, false, true>(c, s, gam, canopy, soil, gsnow, st.snow_band + i, N, days, status, psum, laf, laf,
                       R(f.prec[fo]) * pf, Tf, pet, o);
    }
    const size_t ri = ring_row(ring, d) * N + i;
    ring.rs[ri] = o.rs;
    ring.gwr[ri] = o.gwr;
    if (ring.owp) ring.owp[ri] = o.owp;   // the river's, for the water temperature
    if (b.enabled) {
      acc_in += (double)o.land_in * land_f;
      acc_ev += (double)o.land_evap * land_f;
      acc_lk += (double)o.land_leak * land_f;
    }
  }
  st.canopy[i] = canopy; st.soil[i] = soil; st.snow[i] = gsnow; st.lai_precsum[i] = psum;
  st.lai_days[i] = days; st.lai_status[i] = status;
  if (b.enabled) {
    neumaier_add(b.acc, 0 * N + i, 5 * N + i, acc_in);
    neumaier_add(b.acc, 1 * N + i, 6 * N + i, acc_ev);
    neumaier_add(b.acc, 10 * N + i, 11 * N + i, acc_lk);
  }
}

// Vertical balance ahead of routing for the cells whose land fraction and open-water
// fluxes do not depend on routing (no water body): each thread takes one
// (cell, member) through the days the pipeline steps [t_b, t_e) will route, with
// the vertical state in registers, and leaves surface runoff and recharge in the
// ring buffer.  Results equal the in-wavefront computation: the vertical balance of
// such a cell reads nothing routing writes.
// OUT: the vertical balance's monthly output grids too (DevMonthly::vert, FP64 single member).
// BLOCKS: of 256 threads an SM holds; an ensemble of many states per thread the GPU holds
// gains more from the third (80 registers instead of 110, 92 bytes of spills) than it
// loses: 67k cells x 64 members, 90 days 8.7 -> 7.7 ms, 67k x 12 the same, 67k x 2, 40 days 0.71 -> 0.78.
template <class R, bool ENS, bool OUT = false, int BLOCKS = VaBounds<R, ENS>::min_blocks>
__global__ void __launch_bounds__(VaBounds<R, ENS>::threads, BLOCKS) k_vertical_ahead(DevCellsT<R> c, DevStateT<R> st, DevForcing f,
                                                        DevMembers mem, DevBalance b, DevRingT<R> ring, int doy0,
                                                        int fday0, int ndays, int t_b, int t_e, DevMonthly mon,
                                                        int oday0) {
  const size_t N = (size_t)c.n * (ENS ? mem.members : 1);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
    va_cell<R, ENS>(c, st, f, mem, b, ring, doy0, fday0, ndays, t_b, t_e, i, N, OUT ? &mon : nullptr, oday0);
}

// X: what each cell computes after its routing, bit 0 the water temperature,
// bit 1 the water use, bit 2 (with bit 1) the water use of GLWD units' riparian
// cells met by their outflow cell, bit 3 the vertical balance's monthly output
// grids (FP64 single member, alone).
template <class R, bool FUSED, bool ENS, bool VAW, int X>
__global__ void __launch_bounds__(WaveBounds<R, ENS, VAW>::threads, WaveBounds<R, ENS, VAW>::min_blocks) k_pipeline(DevCellsT<R> c, DevStateT<R> st, DevVertT<R> v, DevForcing f,
                                                  DevMembers mem, DevBalance b, DevRingT<R> ring, DevSync sync,
                                                  double *outq, double *qst, int doy0, int fday0, int oday0,
                                                  int ndays, int t_b, int t_e, int cell_warps, int idle_warp,
                                                  DevMonthly mon, DevVaWork vw, DevWaterTemp wtp, DevWaterUse wu) {
  constexpr bool WT = (X & 1) != 0;
  constexpr bool WU = (X & 2) != 0;
  constexpr bool GL = (X & 4) != 0;   // water use with GLWD units (aggrNUsGloLakResOpt = 1)
  constexpr bool VO = (X & 8) != 0;   // the vertical balance's output grids
  constexpr bool RO = (X & 16) != 0;  // routing's further output grids (always with VO)
  const int n = c.n;
  const int M = ENS ? mem.members : 1;
  const size_t N = (size_t)n * M;
  // the block's last vw.warps warps run no routing
  const bool va_only = VAW && (int)(threadIdx.x >> 5) >= (int)(blockDim.x >> 5) - vw.warps;
  const int route_threads = VAW ? (int)blockDim.x - 32 * vw.warps : (int)blockDim.x;

  const int kd = FUSED ? ring.days_per_step : 1;   // days per step (the per-day routing call: one)
  // thread -> first state index and stride: plain (i mod the grid), or the
  // single-member layout with one idle warp per block (cell_warps warps of cells)
  long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long gstride = (long long)gridDim.x * blockDim.x;
  int wpos = -1;   // this warp's position (flow mode): slots 32*wpos .. 32*wpos+31
  if (!ENS && idle_warp >= 0) {
    const int warp = threadIdx.x >> 5;
    const int weff = warp - (warp > idle_warp ? 1 : 0);
    gtid = warp == idle_warp ? (long long)N : ((long long)blockIdx.x * cell_warps + weff) * 32 + (threadIdx.x & 31);
    gstride = (long long)gridDim.x * cell_warps * 32;
    if (warp != idle_warp) wpos = blockIdx.x * cell_warps + weff;
  }
  // flow mode: every cell warp owns exactly its 32 slots (one cell per thread)
  const bool flow = !ENS && !VAW && !GL && sync.flow && idle_warp >= 0 && gstride >= (long long)N;
  if (flow && (wpos < 0 || wpos >= sync.nwarps)) return;   // no cells: nothing to wait for or publish
  // A cell's routing state and land fractions are read and written each day
  // (mostly L2 hits: the state of the grid is a few MB).  Holding them in
  // registers for the whole launch instead takes ~32 more of a thread's registers,
  // which the wavefront launch with vertical-balance warps pays in spills.
  // waiting for outflows, one cell per thread and one day per step (the shape of every
  // single-member FP64 run): what the wait reads of the topology stays in registers,
  // the day's ring values are loaded before the wait and the outflows it has seen are
  // the day's inflow, so that one trip to L2 lies between two steps instead of three
  const bool one = FUSED && !ENS && !GL && sync.data && kd == 1 && gstride >= (long long)N;
  int one_off = 0, one_u = 0, one_ue = 0, one_up = 0;
  if (one && gtid < (long long)N) {
    one_off = c.offset[gtid];
    one_u = c.up_ptr[gtid];
    one_ue = c.up_ptr[gtid + 1];
    if (one_ue > one_u) one_up = c.up_idx[one_u];
  }
  // Ensembles that fill the GPU (blocks of more than 128 threads): the warps of a block
  // take its states 32 at a time from a shared counter, in slot order, which puts the
  // cells with the most water bodies first. Dealt out to the warps in advance a third of
  // the time went by in waiting at the steps' barriers for the one whose states took
  // longest (67k cells x 64 members, 90 days: 20.5 -> 16.5 ms; 9k x 33, 40 days: 1.72 ->
  // 1.49). 64 states go to each block in turn: 128 or 512 in a row spread the active part
  // of a class unevenly (with blocks of 512 and no class first 18.9 as 64, 21.6 ms), 32
  // halve the use of a fetched sector (19.3).
  // A block's states stay its own, so that what one of its warps wrote in a step the
  // others read after the barrier. The counter only grows: each warp of the block takes
  // one number past a step's. Smaller ensembles, about a state a thread, have nothing to
  // share out and keep the plain mapping.
  const bool take = ENS && blockDim.x > 128;
  [[maybe_unused]] __shared__ unsigned s_taken;
  [[maybe_unused]] unsigned step_base = 0, block_items = 0;
  if (take) {
    const size_t groups = (N + 63) / 64;
    block_items = 2 * (unsigned)(groups / gridDim.x + (blockIdx.x < groups % gridDim.x ? 1 : 0));
    if (threadIdx.x == 0) s_taken = 0;
    __syncthreads();
  }
  // this lane's next state of the step after state i (-1: its first), -1 when there is none;
  // N and more: none for this lane, but the warp has one
  auto next_state = [&](long long i) -> long long {
    if (!take) {
      i = i < 0 ? gtid : i + gstride;
      return i < (long long)N ? i : -1;
    }
    unsigned k = 0;
    if ((threadIdx.x & 31) == 0) k = atomicAdd(&s_taken, 1u) - step_base;
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k >= block_items) return -1;
    return ((((long long)(k >> 1) * gridDim.x + blockIdx.x) * 2 + (k & 1)) << 5) + (threadIdx.x & 31);
  };
  int row_t = t_b % sync.rows;   // t % sync.rows
  for (int t = va_only ? t_e : t_b; t < t_e; ++t, row_t = row_t + 1 == sync.rows ? 0 : row_t + 1) {
    if (flow && t > t_b) {
      if (!wait_deps(sync, wpos, t - t_b - 1)) return;
      __syncwarp();   // the lanes that acquired the flags order the others' loads
    }
    if (kd * (t - c.nlevel + 1) < ndays) {   // some cell still has a day to compute
      const size_t row = (size_t)row_t * kd * N, prev_row = (size_t)(row_t ? row_t - 1 : sync.rows - 1) * kd * N;
      double *q_now0 = outq + row;
      const double *q_prev0 = outq + prev_row;
      double *t_now0 = WT ? wtp.outt + row : nullptr;   // river temperature, same slots
      const double *t_prev0 = WT ? wtp.outt + prev_row : nullptr;
      [[maybe_unused]] R pre_rs = R(0), pre_gwr = R(0);
      [[maybe_unused]] double pre_up = 0., pre_e = 0.;
      if (one) {
        int k = 0, k_e = 0;
        const int d = t - one_off;
        if (gtid < (long long)N && d >= 0 && d < ndays) {
          const size_t ri = ring_row(ring, d) * N + (size_t)gtid;
          pre_rs = ring.rs[ri];
          pre_gwr = ring.gwr[ri];
          k = one_u;
          k_e = one_ue;
        }
        unsigned it = 0;
        for (;;) {
          while (k < k_e) {
            const size_t ui = k == one_u ? one_up : c.up_idx[k];
            const double q = ld_relaxed(q_prev0 + ui);
            double tq = 0.;
            if constexpr (WT) tq = ld_relaxed(t_prev0 + ui);
            if (!is_outflow(sync, q) || (WT && !is_outflow(sync, tq))) break;
            pre_up += q;
            if constexpr (WT) pre_e += q * (tq + WT_CONV_K);
            ++k;
          }
          if (__all_sync(0xffffffffu, k >= k_e)) break;
          if (wait_ran_out(sync, it)) return;
          __nanosleep(WG_POLL_NS);
        }
      } else if (VAW && !GL && sync.data) {
        // the whole warp waits here, converged, for the outflows its cells need: a
        // wait lane by lane inside the cell's routing split the warps, and each part
        // then ran the rest of the step by itself (global grid, one year: 32 ms)
        for (long long i = gtid; __any_sync(0xffffffffu, i < (long long)N); i += gstride) {
          int u = 0, u_e = 0, left = 0;
          const double *p = q_prev0, *pt = t_prev0;
          if (i < (long long)N) {
            const int dbase = kd * (t - c.offset[i]);
            if (dbase >= 0 && dbase < ndays) {
              u = c.up_ptr[i];
              u_e = c.up_ptr[i + 1];
              left = u_e > u ? min(kd, ndays - dbase) : 0;
            }
          }
          unsigned it = 0;
          int k = u;
          for (;;) {   // day by day of the step, upstream cell by upstream cell
            while (left > 0 && has_outflow(sync, p + c.up_idx[k]) && (!WT || has_outflow(sync, pt + c.up_idx[k]))) {
              if (++k == u_e) {
                k = u;
                p += N;
                if constexpr (WT) pt += N;
                --left;
              }
            }
            if (__all_sync(0xffffffffu, left == 0)) break;
            if (wait_ran_out(sync, it)) return;
            __nanosleep(WG_POLL_NS);
          }
        }
      }
      // several cells per thread, or days per step: the same wait before each of its cells,
      // the outflows seen summed to a day's inflow where a step has one day (true: ran out).
      // As a pass over all of a thread's cells before the first, as above, it read the
      // topology and the outflows twice: FP32, 275,000 cells, 500 days 25.9 -> 22.9 ms,
      // 550,000 cells, 365 days 32.1 -> 29.0; FP64, 275,000 cells, 200 days 28.0 -> 26.1.
      // The launches with vertical balance have one cell per thread and keep the pass: in
      // their loop the wait cost 0.7 % on the global grid.
      const bool each = FUSED && !ENS && !VAW && !GL && sync.data && !one;
      [[maybe_unused]] auto wait_for = [&](long long i) -> bool {
        int u = 0, u_e = 0, left = 0;
        const double *p = q_prev0, *pt = t_prev0;
        if (i < (long long)N) {
          const int db = kd * (t - c.offset[i]);
          if (db >= 0 && db < ndays) {
            u = c.up_ptr[i];
            u_e = c.up_ptr[i + 1];
            left = u_e > u ? min(kd, ndays - db) : 0;
          }
        }
        pre_up = pre_e = 0.;
        unsigned it = 0;
        int k = u;
        for (;;) {   // day by day of the step, upstream cell by upstream cell
          while (left > 0) {
            const size_t ui = c.up_idx[k];
            const double q = ld_relaxed(p + ui);
            double tq = 0.;
            if constexpr (WT) tq = ld_relaxed(pt + ui);
            if (!is_outflow(sync, q) || (WT && !is_outflow(sync, tq))) break;
            if (kd == 1) {
              pre_up += q;
              if constexpr (WT) pre_e += q * (tq + WT_CONV_K);
            }
            if (++k == u_e) {
              k = u;
              p += N;
              if constexpr (WT) pt += N;
              --left;
            }
          }
          if (__all_sync(0xffffffffu, left == 0)) return false;
          if (wait_ran_out(sync, it)) return true;
          __nanosleep(WG_POLL_NS);
        }
      };
      // an ensemble's state index belongs to one block's warps, any other to one thread, so
      // that what a step left of a state is there for the next; only upstream outflows
      // cross threads (read via L2)
      for (long long i = ENS ? next_state(-1) : gtid;
           ENS ? i >= 0 : each ? __any_sync(0xffffffffu, i < (long long)N) != 0 : i < (long long)N;
           i = ENS ? next_state(i) : i + gstride) {
        if (each && wait_for(i)) return;
        if ((ENS || each) && i >= (long long)N) continue;
        const int s0 = !ENS ? (int)i : N >> 32 ? (int)(i / M) : (int)((unsigned)i / (unsigned)M);
        const int mm = ENS ? (int)(i - (long long)s0 * M) : 0;
        const int dbase = kd * (t - (one ? one_off : c.offset[s0]));
        if (dbase < 0 || dbase >= ndays) continue;   // this cell's wavefront has not reached it yet / is done
        // a GLWD unit whose riparian cells' use its outflow cell meets (GL) is routed
        // by the thread of its first cell in routing order, cell by cell in that
        // order each day (its cells share one wavefront offset): a riparian cell
        // after the outflow cell sees the unmet share of the same day, one before
        // it that of the day before, as in the reference's sweep
        int unit = -1, m_b = 0, m_e = 1;
        if constexpr (GL) {
          const int u = wu.unit_of[s0];
          if (u >= 0) {
            if (wu.unit_mem[wu.unit_ptr[u]] != s0) continue;   // routed by the unit's first cell
            unit = u;
            m_b = wu.unit_ptr[u];
            m_e = wu.unit_ptr[u + 1];
          }
        }
        if (unit < 0 && c.active && !c.active[s0]) continue;
        // the step's kd days of this cell, in order; the upstream cells routed the
        // same days one step earlier (their offset is one less)
        for (int kk = 0; kk < kd && dbase + kk < ndays; ++kk) {
         for (int m = m_b; m < m_e; ++m) {
          const int s = unit >= 0 ? wu.unit_mem[m] : s0;
          const size_t si = unit >= 0 ? (size_t)s : (size_t)i;
          if (unit >= 0 && c.active && !c.active[s]) continue;
          const int d = dbase + kk;
          double *q_now = q_now0 + (size_t)kk * N;
          const double *q_prev = q_prev0 + (size_t)kk * N;
          const int doy = (doy0 - 1 + d) % 365 + 1;
          const int month = month_of(doy);
          const uint32_t fl = c.flags[s];
          VOut<R> o;
          const R laf = st.laf[si];
          const R laf_prev = st.laf_prev[si];
          if (FUSED && !(fl & F_VINLINE)) {
            const size_t ri = ring_row(ring, d) * N + si;
            o.rs = one ? pre_rs : ring.rs[ri];
            o.gwr = one ? pre_gwr : ring.gwr[ri];
            o.transfer = R(0); o.owp = R(0); o.owpet = R(0);
            o.land_in = R(0); o.land_evap = R(0); o.land_leak = R(0);   // accounted ahead
            if constexpr (WT) {
              o.owp = ring.owp[ri];
              o.owpet = ring.pet_water[ri];   // one member: the same index
            }
          } else if (FUSED) {
            const size_t fo = (size_t)(fday0 + d) * n + s;
            R Pin = R(f.prec[fo]);
            R gam = c.gamma[s];
            if (ENS) {
              Pin *= R(mem.prec_factor[mm]);
              gam *= R(mem.gamma_factor[mm]);
            }
            const int started = st.laf_started[si];
            VSink vs;
            const bool vo = VO && vert_sink(mon, oday0 + d, si, N, vs);
            if (VO && doy == 1 && started == 1 && (fl & F_LOCLAKE) && mon.vconst) {
              // total PET's freshwater share after the first year: the local lakes'
              // share at the year's start (routing.cpp:1249-1259, 5045-5048)
              double *vk = mon.vconst + si;
              const double rf = (double)st.rf_loclake[si], ll = (double)c.ll100[s];   // G_loc_lake / 100
              const double fll = (ll > 0. && rf > 0.) ? rf * ll : 0.;              // G_fLocLake
              vk[3 * N] = vk[4 * N] + fll * 100. + vk[5 * N];
            }
            const float Tf = f.temp[fo];
            // (with one member the ring's runoff and recharge slots hold the land's PETs)
            const size_t rk = ring_row(ring, d) * n + s;
            const Pet<R> pet = one ? Pet<R>{pre_rs, pre_gwr, ring.pet_water[rk]} : ring_pet(ring, rk);
            const R prev = started == 1 ? laf_prev : laf;   // daily.cpp:159-169
            if (VO && vo) {
              const Radiation<R> rad = radiation_at<R>(c, s, doy, Tf, f.swrad[fo]);
              vertical_at<R>(c, st, N, s, si, Pin, gam, Tf, pet, laf, prev, o, &vs, &rad,
                             c.ext_rad[(size_t)(doy - 1) * c.nrow + c.ext_row[s]]);
            } else {
              vertical_at<R>(c, st, N, s, si, Pin, gam, Tf, pet, laf, prev, o);
            }
          } else {
            o.rs = v.rs[s]; o.gwr = v.gwr[s]; o.transfer = v.transfer[s]; o.owp = v.owp[s]; o.owpet = v.owpet[s];
            o.land_in = v.land_in[s]; o.land_evap = v.land_evap[s]; o.land_leak = v.land_leak[s];
          }
          // upstream inflow, summed in FP64 in the reference's push order
          // (routing.cpp:3955-3958), when routing asks for it
          double up = 0., e_up = 0.;
          bool failed = false;
          const bool seen = one || (each && kd == 1);
          const int u0 = seen ? 0 : c.up_ptr[s], u1 = seen ? 0 : c.up_ptr[s + 1];
          if (seen) {
            up = pre_up;
            e_up = pre_e;
          }
          auto inflow_up = [&]() -> double {
            for (int k = u0; k < u1; ++k) {
              const size_t ui = (size_t)c.up_idx[k] * M + mm;
              // an upstream cell of the same unit was routed this step, earlier in this loop
              const double qu = (GL && unit >= 0 && wu.unit_of[c.up_idx[k]] == unit)
                                    ? q_now[ui]
                                    : ENS ? __ldcg(q_prev + ui) : upstream_value<!FUSED>(sync, q_prev + ui, failed);
              up += qu;
              if constexpr (WT)   // the energy the inflow carries (calcWaterTemp.cpp:76-83)
                e_up += qu * (upstream_value<!FUSED>(sync, t_prev0 + (size_t)kk * N + ui, failed) + WT_CONV_K);
            }
            return up;
          };
          // the water temperature's day begins with the inflow; an ensemble's 64
          // registers hold it rather than the routing state before it
          if constexpr (WT || ENS) inflow_up();
          RState<R> rs = load_rstate(st, si, fl);
          RTerms<R> rt;
          // the water temperature (routing.cpp:4241-4513) body by body inside
          // routing_cell, the river after it
          wt::WtDay wtd;
          if constexpr (WT) {
            const size_t fo = (size_t)(fday0 + d) * n + s;
            const float g = wtp.gwt[s];
            wtd.begin(&wtp, s, si, N, fl, (double)f.temp[fo], (double)f.swrad[fo], (double)wtp.lw[fo], (double)o.owp,
                      (double)c.area[s], g < 0.f ? 0. : (double)g, up, e_up);
            if (mon.wtemp) {   // the monthly mean temperatures of the day's month
              const int yd = mon.doy_day0 - 1 + oday0 + d;
              const int mi = (yd / 365) * 12 + month_of(yd % 365 + 1) - mon.month0;
              if (mi >= 0 && mi < mon.nmonths) {
                wtd.msum = mon.wtemp + (size_t)mi * N + si;
                wtd.ms = (size_t)mon.nmonths * N;
              }
            }
          }
          const size_t wrow = WU ? (size_t)wu.row_of_fday[fday0 + d] * WU_FIELDS * (size_t)n : 0;
          R tv;
          [[maybe_unused]] RoutOut ro;   // the output grids' routing terms (RO)
          const bool nocont = (fl & F_NOCONT) != 0;
          if (nocont) {
            // the reference routes only continental cells (routing.cpp:1878-4518): the
            // storages stay, nothing flows on, and the inflow stays behind in
            // G_riverInflow, i.e. leaves the system (a negative leak: the leak
            // counts water the model adds)
            if constexpr (!WT && !ENS) inflow_up();
            tv = R(0);
            rt.p_ow = R(0); rt.e_ow = R(0); rt.leak = R(-up); rt.velocity = R(0);
          } else {
            tv = routing_cell<R, WT, WU, GL, RO>(c, s, rs, doy, month, laf, laf_prev, o,
                                                 [&]() { return WT || ENS ? up : inflow_up(); }, rt, &wtd, &wu, wrow, si, N, &ro);
            if (!FUSED && failed) return;
            store_rstate(st, si, rs, fl);
          }
          if (ENS) q_now[si] = (double)tv;
          else st_outflow(q_now + si, (double)tv);
          if constexpr (WT) {
            // a cell without continental area keeps the reference's initial 15 degrees (routing.cpp:174)
            const double tr = nocont ? 15. : wtd.river((double)rs.river, (double)c.rlen[s], (double)c.cfa[s],
                                                       (double)o.owpet);
            st_outflow(t_now0 + (size_t)kk * N + si, tr);
            const int stw = c.station[s];
            if (stw >= 0) wtp.qst_t[(size_t)(oday0 + d) * c.nstation + stw] = tr;
          }
          if (b.enabled) {
            const double land_f = (double)c.area_f[s] * (double)laf;
            if (!FUSED || (fl & F_VINLINE))
              record_balance(b, N, si, (double)o.land_in * land_f + (double)rt.p_ow,
                             (double)o.land_evap * land_f + (double)rt.e_ow, up, (double)tv,
                             (double)o.land_leak * land_f + (double)rt.leak);
            else {   // vertical ran ahead: its land terms are in arrays 0, 1 and 10
              record_routing_balance(b, N, si, up, (double)tv, (double)rt.leak);
              if constexpr (WU) neumaier_add(b.acc, 12 * N + si, 13 * N + si, (double)rt.e_ow);
            }
          }
          // land-area fraction for the next day (routing.cpp:5034-5188, 5343-5352)
          if (fl & (F_LOCLAKE | F_LOCWETL | F_GLOWETL)) {
            R fswb = st.fswb_next[si];
            st.laf[si] = fraction_next<R>(fl, rs, c.ll100[s], c.lw100[s], c.gw100[s], laf, fswb);
            st.fswb_next[si] = fswb;
          }
          st.laf_prev[si] = laf;
          st.laf_started[si] = 1;
          const int stn = c.station[s];
          if (stn >= 0) qst[((size_t)(oday0 + d) * c.nstation + stn) * M + mm] = (double)tv;
          if (mon.daily_storage && oday0 + d < mon.daily_days) {   // the state file's daily storages
            double *ds = mon.daily_storage + (size_t)(oday0 + d) * 7 * N + si;
            ds[0] = (double)rs.loclake;
            ds[N] = (double)rs.locwetl;
            ds[2 * N] = (double)rs.glolake;
            ds[3 * N] = (double)rs.glowetl;
            ds[4 * N] = (double)rs.res;
            ds[5 * N] = (double)rs.river;
            ds[6 * N] = (double)rs.gw;
          }
          if (mon.enabled) {
            // monthly epilogue: this thread owns the cell, so no atomics
            const int od = oday0 + d;
            const int yd = mon.doy_day0 - 1 + od;
            const int mi = (yd / 365) * 12 + month_of(yd % 365 + 1) - mon.month0;
            if (mi >= 0 && mi < mon.nmonths) {
              const size_t k = (size_t)mi * N + si;
              const double q = (double)tv;
              // the flux grids of continental cells (routing.cpp:1878-4518), river
              // availability outside inland sinks (routing.cpp:4010-4037)
              if (!(fl & (F_SINK | F_NOCONT))) {
                mon.river_avail[k] += q;
                mon.min_avail[k] = fmin(mon.min_avail[k], q);
                mon.max_avail[k] = fmax(mon.max_avail[k], q);
              }
              mon.storage[k] += (double)rs.gw + (double)rs.river + (double)rs.loclake + (double)rs.locwetl +
                                (double)rs.glolake + (double)rs.glowetl + (double)rs.res;
              if (!(fl & F_NOCONT)) {
                // CellRunoff (routing.cpp:3933-3939): in inland sinks the transported
                // volume leaves the cell as evaporation
                mon.cell_runoff[k] += ((fl & F_SINK) ? 0. : q) - up;
                mon.velocity[k] += (double)rt.velocity / 86.4;   // km/d -> m/s
              }
            }
          }
          if constexpr (RO) {
            // routing's further output grids (routing.cpp:3964-4238, 4525-4737,
            // 5183-5186); the flux terms of continental cells only (routing.cpp:1878-4518)
            const int od = oday0 + d;
            const double q = (double)tv;
            const double cr = ((fl & F_SINK) ? 0. : q) - up;   // CellRunoff [km3]
            double owe = 0., csr = 0., crmm = 0., cp = 0.;
            if (!nocont && (mon.rext || mon.drout)) {
              const double cf = (double)c.contfreq[s], area = (double)c.area[s];
              const double rc = 1e8 * fm::rcp_pos(area * cf);   // km3 -> mm over the continental area
              // open-water evaporation, with an inland sink's transported volume (routing.cpp:4549-4560)
              owe = (ro.owe + ((fl & F_SINK) ? q : 0.)) * rc;
              csr = (cr - ro.gw_runoff) * rc;                  // routing.cpp:3998-4001
              crmm = cr * rc;
              const double *vk = mon.vconst + si;
              double lwe = cf - vk[4 * N] - vk[5 * N];          // G_landWaterExclGloLakAreaFrac (routing.cpp:1187-1196)
              if (lwe < 0.) lwe = 0.;
              const double owp = (double)(c.mprec[s] * R(f.prec[(size_t)(fday0 + d) * n + s]));
              cp = owp * lwe * area * 1e-8 + ro.p_lake;       // consistent precipitation (routing.cpp:3973-3977)
            }
            if (mon.rext) {
              const int yd = mon.doy_day0 - 1 + od;
              const int mi = (yd / 365) * 12 + month_of(yd % 365 + 1) - mon.month0;
              if (mi >= 0 && mi < mon.nmonths) {
                double *r = mon.rext + (size_t)mi * N + si;
                const size_t k = (size_t)mon.nmonths * N;
                if (!nocont) {
                  r[0] += owe;
                  r[k] += csr;
                  r[2 * k] += ro.gw_runoff;
                  r[4 * k] += ro.lw_ext;
                  r[5 * k] += ro.gw_ext;
                  // the reference adds the reservoir's flows twice a day, in the cell
                  // loop and after it (routing.cpp:4049-4050, 4653-4655)
                  r[6 * k] += 2. * ro.res_in;
                  r[7 * k] += 2. * ro.res_out;
                  r[8 * k] += cp;
                }
                r[3 * k] += (double)laf;
                r[9 * k] = (double)rs.loclake + (double)rs.locwetl + (double)rs.glolake + (double)rs.glowetl +
                           (double)rs.river + (double)rs.res;
                if constexpr (WU) {
                  if (!nocont) {   // routing.cpp:3744-3747
                    r[10 * k] += ro.actual_use;
                    r[11 * k] += ro.nug;
                  }
                }
              }
            }
            if (mon.drout && !nocont && od < mon.drout_days) {
              double *r = mon.drout + (size_t)od * N + si;
              const size_t k = (size_t)mon.drout_days * N;
              r[0] = (fl & F_SINK) ? 0. : q;
              r[k] = (double)rt.velocity / 86.4;
              r[2 * k] = cr;
              r[3 * k] = crmm;
              r[4 * k] = csr;
              r[5 * k] = ro.gw_runoff;
              r[6 * k] = (double)laf;
              r[7 * k] = cp;
              r[8 * k] = owe;
            }
          }
         }   // cells of the unit
        }   // days of the step
      }
      if (take) step_base += block_items + blockDim.x / 32;
    }
    if (flow) {
      // publish step t: every lane's writes of this step (fence, one instruction for
      // the warp), then the flag (release)
      __threadfence();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) st_release_int(sync.wstep + wpos, t - t_b);
    } else if (!sync.data && t + 1 < t_e) {
      if (!grid_barrier(sync, (unsigned)(t - t_b), route_threads)) return;
    }
  }
  if constexpr (VAW) {
    // vertical balance ahead for the next launch's steps, 32 slots at a time from a
    // shared counter: by the block's vw.warps warps from the start, filling the FP64
    // pipe while the routing warps wait, and by the routing warps once their steps
    // are done (global grid, one year: five warps that do nothing else 17.5 ms, one
    // such warp, the idle warp and this help 17.2 ms)
    const unsigned lane = threadIdx.x & 31;
    for (;;) {
      unsigned g = 0;
      if (lane == 0) g = atomicAdd(vw.next, 1u);
      g = __shfl_sync(0xffffffffu, g, 0);
      if (g >= (unsigned)vw.nitems) break;
      const size_t i = (size_t)g * 32 + lane;
      if (i < N) va_cell<R, ENS>(c, st, f, mem, b, ring, doy0, fday0, ndays, vw.t_b, vw.t_e, i, N, VO ? &mon : nullptr,
                                 oday0);
    }
  }
}

template <class R>
__global__ void k_volume(DevCellsT<R> c, DevStateT<R> st, int M, double *vol) {
  const size_t N = (size_t)c.n * M;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) vol[i] = cell_volume<R>(c, st, N, (int)(i / M), i);
}

// Block-level Neumaier reduction; partial[blockIdx.x*8 + k] sums of
//   0 storage, 1 in, 2 evap, 3 outflow at outlets and sinks, 4 leak,
//   5 largest closure residual of a cell relative to its throughput.
template <class R>
__global__ void __launch_bounds__(256) k_balance_sum(DevCellsT<R> c, DevStateT<R> st, int M, DevBalance b,
                                                     const double *vol0, double *partial) {
  __shared__ double sh[6][256];
  __shared__ double shc[5][256];
  const size_t N = (size_t)c.n * M;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double val[6] = {0, 0, 0, 0, 0, 0};
  if (i < N) {
    const int s = (int)(i / M);
    const double vnow = cell_volume<R>(c, st, N, s, i);
    const double in = b.acc[0 * N + i] + b.acc[5 * N + i];
    const double ev = (b.acc[1 * N + i] + b.acc[6 * N + i]) + (b.acc[12 * N + i] + b.acc[13 * N + i]);
    const double out = b.acc[2 * N + i] + b.acc[7 * N + i];
    const double up = b.acc[3 * N + i] + b.acc[8 * N + i];
    const double lk = (b.acc[4 * N + i] + b.acc[9 * N + i]) + (b.acc[10 * N + i] + b.acc[11 * N + i]);
    val[0] = vnow;
    val[1] = in;
    val[2] = ev;
    val[3] = (c.flags[s] & F_OUTLET) ? out : 0.;
    val[4] = lk;
    const double resid = (vnow - vol0[i]) - (in - ev + up - out + lk);
    const double scale = fmax(fmax(fabs(vnow), fabs(vol0[i])), fmax(fmax(in, ev), fmax(up, out)));
    val[5] = scale > 0. ? fabs(resid) / scale : 0.;
  }
  for (int k = 0; k < 6; ++k) sh[k][threadIdx.x] = val[k];
  for (int k = 0; k < 5; ++k) shc[k][threadIdx.x] = 0.;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      for (int k = 0; k < 5; ++k) {
        const double a = sh[k][threadIdx.x], x = sh[k][threadIdx.x + w];
        const double tsum = a + x;
        const double e = (fabs(a) >= fabs(x)) ? (a - tsum) + x : (x - tsum) + a;
        sh[k][threadIdx.x] = tsum;
        shc[k][threadIdx.x] += shc[k][threadIdx.x + w] + e;
      }
      sh[5][threadIdx.x] = fmax(sh[5][threadIdx.x], sh[5][threadIdx.x + w]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 6; ++k) partial[blockIdx.x * 8 + k] = sh[k][0] + (k < 5 ? shc[k][0] : 0.);
}

// forcing arrives day-major in cell order; the device keeps it in slot order
__global__ void k_gather_forcing(const float *__restrict__ src, float *__restrict__ dst,
                                 const int32_t *__restrict__ cell_of_slot, int n, int ndays) {
  const size_t total = (size_t)n * ndays;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    const size_t d = k / n;
    const int s = (int)(k - d * n);
    dst[k] = src[d * n + cell_of_slot[s]];
  }
}

// Forcing as the reference's yearly files hold it (`.365.UNF0`: big-endian float,
// cell-major [cell][nd_file], climateYear.cpp:38-79, grid_io_adapters.h:91-129):
// days [d_first, d_first + nd) of the file into dst [day][slot].  32 x 32 tiles
// through shared memory: a warp reads 32 days of one cell (contiguous) and writes
// 32 slots of one day (contiguous); the byte swap is one byte permute.
__global__ void __launch_bounds__(256) k_unf_forcing(const uint32_t *__restrict__ raw, float *__restrict__ dst,
                                                     const int32_t *__restrict__ cell_of_slot, int n, int nd_file,
                                                     int d_first, int nd, unsigned swap) {
  __shared__ float tile[32][33];
  const int s0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8) {
    const int s = s0 + r, d = d0 + tx;
    if (s < n && d < nd) {
      const uint32_t v = raw[(size_t)cell_of_slot[s] * nd_file + d_first + d];
      tile[r][tx] = __uint_as_float(__byte_perm(v, 0u, swap));   // 0x0123: big-endian file bytes
    }
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int d = d0 + r, s = s0 + tx;
    if (s < n && d < nd) dst[(size_t)d * n + s] = tile[tx][r];
  }
}

cudaError_t launch_unf_forcing(const uint32_t *raw, float *dst, const int32_t *cell_of_slot, int n, int nd_file,
                               int d_first, int nd, cudaStream_t st, bool big_endian) {
  const dim3 grid((unsigned)((n + 31) / 32), (unsigned)((nd + 31) / 32));
  k_unf_forcing<<<grid, 256, 0, st>>>(raw, dst, cell_of_slot, n, nd_file, d_first, nd,
                                      big_endian ? 0x0123u : 0x3210u);
  return cudaGetLastError();
}

// Reads in cell order: writes are contiguous, the slots' values come from L2 (a field
// of the global grid is 0.5 MB).
__global__ void __launch_bounds__(256) k_state_rows(StateRows rows, char *out, const int32_t *__restrict__ slot_of_cell,
                                                    int n, size_t N, int members, int member) {
  const StateRow r = rows.row[blockIdx.y];
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (size_t)n * r.per) return;
  const size_t cell = k / r.per, b = k - cell * r.per;
  const size_t i = b * N + (size_t)slot_of_cell[cell] * members + member;
  if (r.kind == 0) ((double *)(out + r.offset))[k] = ((const double *)r.src)[i];
  else if (r.kind == 1) ((double *)(out + r.offset))[k] = (double)((const float *)r.src)[i];
  else ((int32_t *)(out + r.offset))[k] = ((const int32_t *)r.src)[i];
}

cudaError_t launch_state_rows(const StateRows &rows, char *out, const int32_t *slot_of_cell, int n, size_t N,
                              int members, int member, cudaStream_t st) {
  int per = 1;
  for (int k = 0; k < rows.count; ++k) per = std::max(per, rows.row[k].per);
  const dim3 grid((unsigned)(((size_t)n * per + 255) / 256), (unsigned)rows.count);
  k_state_rows<<<grid, 256, 0, st>>>(rows, out, slot_of_cell, n, N, members, member);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_rows(const double *__restrict__ src, const double *__restrict__ land,
                                              double *__restrict__ out, const int32_t *__restrict__ slot_of_cell,
                                              int n, int members, size_t rows, bool no_inf) {
  const size_t per = (size_t)n * members, total = rows * per;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    const size_t r = k / per, q = k - r * per, cell = q / members;
    const size_t i = r * per + (size_t)slot_of_cell[cell] * members + (q - cell * members);
    double v = src[i];
    if (land) v += land[i];
    out[k] = (no_inf && isinf(v)) ? 0. : v;
  }
}

cudaError_t launch_rows(const double *src, const double *land, double *out, const int32_t *slot_of_cell, int n,
                        int members, size_t rows, bool no_inf, cudaStream_t st) {
  const size_t total = rows * n * members;
  if (total == 0) return cudaSuccess;
  k_rows<<<(unsigned)std::min<size_t>((total + 255) / 256, 152 * 32), 256, 0, st>>>(src, land, out, slot_of_cell, n,
                                                                                 members, rows, no_inf);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_clear_skipped(double *rows, double *rows_t, const uint8_t *__restrict__ active,
                                                       int members, size_t row, size_t total) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    if (active[i % row / members]) continue;
    rows[i] = 0.;
    if (rows_t) rows_t[i] = 0.;
  }
}

cudaError_t launch_clear_skipped(double *rows, double *rows_t, const uint8_t *active, int n, int members, int nrows,
                                 cudaStream_t st) {
  const size_t row = (size_t)n * members, total = row * nrows;
  k_clear_skipped<<<(unsigned)std::min<size_t>((total + 255) / 256, 152 * 32), 256, 0, st>>>(rows, rows_t, active, members,
                                                                                           row, total);
  return cudaGetLastError();
}

// One row of outflows (2.7 MB on the global grid at five days per step), before a call
// that goes on with a run: a launch costs 3 us of the stream where a copy costs 9.
__global__ void __launch_bounds__(256) k_fetch_row(double *dst, const double *src, double *dst_t, const double *src_t, size_t n) {
  double *d = blockIdx.y ? dst_t : dst;
  const double *s = blockIdx.y ? src_t : src;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) d[i] = s[i];
}

cudaError_t launch_fetch_row(double *dst, const double *src, double *dst_t, const double *src_t, size_t n, cudaStream_t st) {
  const dim3 grid((unsigned)std::min<size_t>((n + 255) / 256, 152 * 32), dst_t ? 2 : 1);
  k_fetch_row<<<grid, 256, 0, st>>>(dst, src, dst_t, src_t, n);
  return cudaGetLastError();
}

// What a wavefront of two rows (one member, a grid barrier per step) holds of steps [a,
// b): per cell and day of the step the last two steps that had such a day.
__global__ void __launch_bounds__(256) k_keep_outflow(const double *rows, const double *rows_t, double *kept, double *kept_t,
                                                      const int32_t *__restrict__ offset, int n, int kd, int nrows,
                                                      int ndays, int a, int b) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, row = (size_t)kd * n;
  if (i >= row) return;
  const int s = (int)(i % n), left = ndays - 1 - (int)(i / n);   // from this place in the first step to the last day
  if (left < 0) return;
  const int first = max(a, offset[s]), last = min(b - 1, offset[s] + left / kd);
  for (int t = max(first, last - 1); t <= last; ++t) {
    kept[(t & 1) * row + i] = rows[t % nrows * row + i];
    if (rows_t) kept_t[(t & 1) * row + i] = rows_t[t % nrows * row + i];
  }
}

cudaError_t launch_keep_outflow(const double *rows, const double *rows_t, double *kept, double *kept_t,
                                const int32_t *offset, int n, int kd, int nrows, int ndays, int a, int b,
                                cudaStream_t st) {
  k_keep_outflow<<<(unsigned)(((size_t)kd * n + 255) / 256), 256, 0, st>>>(rows, rows_t, kept, kept_t, offset, n, kd,
                                                                          nrows, ndays, a, b);
  return cudaGetLastError();
}

__global__ void k_fill(double *p, size_t n, double v) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

cudaError_t launch_fill(double *p, size_t n, double v, cudaStream_t st) {
  k_fill<<<(unsigned)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, st>>>(p, n, v);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- launchers
// The day step's FP64 math functions on arrays (numerics tests): 0 exp, 1 log,
// 2 pow, 3 the refined reciprocal, 4 the hardware's approximate reciprocal alone.
__global__ void k_math_eval(int fn, const double *x, const double *y, double *out, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i];
  double r = 0.;
  switch (fn) {
    case 0: r = fm::exp(a); break;
    case 1: r = fm::log(a); break;
    case 2: r = fm::pow(a, y[i]); break;
    case 3: r = fm::rcp_pos(a); break;
    default: asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a)); break;
  }
  out[i] = r;
}

cudaError_t launch_math_eval(int fn, const double *x, const double *y, double *out, size_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_math_eval<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(fn, x, y, out, n);
  return cudaGetLastError();
}

cudaError_t upload_fastmath_tables(const unsigned long long exp2_tab[256], const ulonglong2 log2_tab[256]) {
  cudaError_t e = cudaMemcpyToSymbol(fm::g_exp2_tab, exp2_tab, 256 * sizeof(exp2_tab[0]));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(fm::g_log2_tab, log2_tab, 256 * sizeof(log2_tab[0]));
  return e;
}

cudaError_t launch_gather_forcing(const float *src, float *dst, const int32_t *cell_of_slot, int n, int ndays,
                                  cudaStream_t st) {
  const size_t total = (size_t)n * ndays;
  const int threads = 256;
  const int blocks = (int)std::min<size_t>((total + threads - 1) / threads, 152 * 16);
  k_gather_forcing<<<blocks, threads, 0, st>>>(src, dst, cell_of_slot, n, ndays);
  return cudaGetLastError();
}

template <class R>
cudaError_t launch_vertical(const DevCellsT<R> &c, const DevStateT<R> &s, const DevVertT<R> &v, const DevForcing &f,
                            int doy, int fday, cudaStream_t st) {
  const int threads = 256, blocks = (c.n + threads - 1) / threads;
  k_vertical<R><<<blocks, threads, 0, st>>>(c, s, v, f, doy, fday);
  return cudaGetLastError();
}

template <class R>
cudaError_t launch_vertical_ahead(const DevCellsT<R> &c, const DevStateT<R> &s, const DevForcing &f,
                                  const DevMembers &mem, const DevBalance &b, const DevRingT<R> &ring, int doy0,
                                  int fday0, int ndays, int t_b, int t_e, int blocks, int threads, cudaStream_t st,
                                  const DevMonthly &mon, int oday0, bool dense) {
  if constexpr (std::is_same<R, float>::value) {
    if (mem.members > 1 && dense) {
      k_vertical_ahead<R, true, false, VaBounds<R, true>::min_blocks + 1><<<blocks, threads, 0, st>>>(
          c, s, f, mem, b, ring, doy0, fday0, ndays, t_b, t_e, mon, oday0);
      return cudaGetLastError();
    }
  }
  if (mem.members > 1)
    k_vertical_ahead<R, true><<<blocks, threads, 0, st>>>(c, s, f, mem, b, ring, doy0, fday0, ndays, t_b, t_e, mon,
                                                          oday0);
  else if ((mon.vert || mon.dvert) && std::is_same<R, double>::value)
    k_vertical_ahead<R, false, true><<<blocks, threads, 0, st>>>(c, s, f, mem, b, ring, doy0, fday0, ndays, t_b, t_e,
                                                                 mon, oday0);
  else
    k_vertical_ahead<R, false><<<blocks, threads, 0, st>>>(c, s, f, mem, b, ring, doy0, fday0, ndays, t_b, t_e, mon,
                                                           oday0);
  return cudaGetLastError();
}

template <class R>
cudaError_t launch_pet(const DevCellsT<R> &c, const DevForcing &f, const DevRingT<R> &ring, int doy0, int fday0,
                       int ndays, int t_b, int t_e, cudaStream_t st) {
  const int most = 65535 * kPetDays / ring.days_per_step;   // steps that the grid's second dimension holds
  for (int a = t_b; a < t_e; a += most) {
    const int b = std::min(t_e, a + most);
    const long long days = (long long)ring.days_per_step * (b - a);
    const dim3 grid((unsigned)((c.n + 255) / 256), (unsigned)((days + kPetDays - 1) / kPetDays));
    k_pet<R><<<grid, 256, 0, st>>>(c, f, ring, doy0, fday0, ndays, a, b);
  }
  return cudaGetLastError();
}

template <class R, int X>
static const void *pipeline_fn_x(bool fused, bool vaw) {
  return vaw ? (fused ? (const void *)k_pipeline<R, true, false, true, X> : nullptr)
             : (fused ? (const void *)k_pipeline<R, true, false, false, X>
                      : (const void *)k_pipeline<R, false, false, false, X>);
}

template <class R>
static const void *pipeline_fn(bool fused, bool ens, bool vaw, bool wt = false, bool wu = false, bool gl = false,
                               bool vo = false, bool ro = false) {
  if (gl && (ens || wt || !wu || !std::is_same<R, double>::value)) return nullptr;   // GLWD units: FP64, one member
  if (vo || ro) {   // the output grids: FP64, one member
    if constexpr (std::is_same<R, double>::value) {
      if (ens) return nullptr;
      if (wt) return (wu || ro) ? nullptr : pipeline_fn_x<R, 9>(fused, vaw);   // the vertical balance's with the water temperature
      if (gl) return pipeline_fn_x<R, 30>(fused, vaw);   // water use over GLWD units: all outputs in one variant
      if (wu) return pipeline_fn_x<R, 26>(fused, vaw);   // with water use: all outputs in one variant
      return ro ? pipeline_fn_x<R, 24>(fused, vaw) : pipeline_fn_x<R, 8>(fused, vaw);
    } else {
      return nullptr;
    }
  }
  if (ens) return wt ? nullptr
                     : (wu ? (const void *)k_pipeline<R, true, true, false, 2> : (const void *)k_pipeline<R, true, true, false, 0>);
  if constexpr (std::is_same<R, double>::value) {   // FP64 single member only
    if (gl) return pipeline_fn_x<R, 6>(fused, vaw);
    if (wt && wu) return pipeline_fn_x<R, 3>(fused, vaw);
    if (wt) return pipeline_fn_x<R, 1>(fused, vaw);
    if (wu) return pipeline_fn_x<R, 2>(fused, vaw);
    if (vaw) return (const void *)k_pipeline<R, true, false, true, 0>;
  } else {   // FP32: no vertical-balance warps, no water temperature
    if (vaw || wt) return nullptr;
    if (wu) return fused ? (const void *)k_pipeline<R, true, false, false, 2> : (const void *)k_pipeline<R, false, false, false, 2>;
  }
  return fused ? (const void *)k_pipeline<R, true, false, false, 0>
               : (const void *)k_pipeline<R, false, false, false, 0>;
}

template <class R>
int pipeline_max_blocks(bool fused, bool ens, int threads, bool vaw, bool wt, bool wu) {
  int dev = 0, nsm = 0, per = 0;
  const void *fn = pipeline_fn<R>(fused, ens, vaw, wt, wu);
  if (!fn) return 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, 0) != cudaSuccess) return 0;
  return per * nsm;
}

template <class R>
int vertical_ahead_max_blocks(bool ens, int threads) {
  int dev = 0, nsm = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const void *fn = ens ? (const void *)k_vertical_ahead<R, true> : (const void *)k_vertical_ahead<R, false>;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, 0) != cudaSuccess) return 0;
  return per * nsm;
}

template <class R>
cudaError_t launch_pipeline(bool fused, const DevCellsT<R> &c, const DevStateT<R> &s, const DevVertT<R> &v,
                            const DevForcing &f, const DevMembers &mem, const DevBalance &b, const DevRingT<R> &ring,
                            const DevSync &sync, double *outq, double *qst, int doy0, int fday0, int oday0, int ndays,
                            int t_b, int t_e, int blocks, int threads, const WarpLayout &lay, const DevMonthly &mon,
                            const DevVaWork &vw, const DevWaterTemp &wtp, const DevWaterUse &wu, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (sync.data) {   // the rows of this launch's steps: no outflow yet
    const size_t row = (size_t)(fused ? ring.days_per_step : 1) * c.n * sizeof(double);
    const int steps = std::min(t_e - t_b, sync.rows), first = t_b % sync.rows, head = std::min(steps, sync.rows - first);
    for (char *p : {(char *)outq, (char *)(wtp.enabled ? wtp.outt : nullptr)}) {
      if (!p) continue;
      if (e == cudaSuccess) e = cudaMemsetAsync(p + first * row, 0xff, head * row, st);
      if (e == cudaSuccess && steps > head) e = cudaMemsetAsync(p, 0xff, (steps - head) * row, st);
    }
  } else {
    e = cudaMemsetAsync(sync.counter, 0, sizeof(unsigned), st);
  }
  if (e == cudaSuccess && sync.flow && sync.wstep)
    e = cudaMemsetAsync(sync.wstep, 0xff, (size_t)sync.nwarps * sizeof(int), st);   // -1: no step done yet
  const bool vaw = fused && vw.nitems > 0;
  if (e == cudaSuccess && vaw) e = cudaMemsetAsync(vw.next, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  int cell_warps = lay.cell_warps, idle_warp = mem.members > 1 ? -1 : lay.idle_warp;
  if (idle_warp >= 0 && (threads != lay.threads || (long long)blocks * cell_warps * 32 < (long long)c.n))
    idle_warp = -1;   // the layout does not describe this launch: plain mapping
  // vertical-balance warps only on the single-member layout they were sized for
  if (vaw && (idle_warp < 0 || mem.members > 1 || vw.warps != lay.va_warps)) return cudaErrorInvalidConfiguration;
  DevVaWork vwk = vw;
  if (!vaw) vwk.warps = vwk.nitems = 0;
  if (mem.members > 1 && lay.join > 1 && blocks % lay.join == 0) {
    blocks /= lay.join;
    threads *= lay.join;
  }
  void *args[] = {(void *)&c,    (void *)&s,    (void *)&v,     (void *)&f,     (void *)&mem,   (void *)&b,
                  (void *)&ring, (void *)&sync, (void *)&outq,  (void *)&qst,   (void *)&doy0,  (void *)&fday0,
                  (void *)&oday0, (void *)&ndays, (void *)&t_b, (void *)&t_e, (void *)&cell_warps,
                  (void *)&idle_warp, (void *)&mon, (void *)&vwk, (void *)&wtp, (void *)&wu};
  const bool ens = mem.members > 1;
  const void *fn = pipeline_fn<R>(fused, ens, vaw, wtp.enabled != 0, wu.enabled != 0, wu.enabled && wu.glwd,
                                  mon.vert != nullptr || mon.dvert != nullptr,
                                  mon.rext != nullptr || mon.drout != nullptr);
  if (!fn) return cudaErrorInvalidConfiguration;
  if (vaw) threads += 32 * vw.warps;
  // cooperative (all blocks resident, or the launch fails) through the launch
  // attribute, which stream capture records into a graph kernel node
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

template <class R>
cudaError_t launch_volume(const DevCellsT<R> &c, const DevStateT<R> &s, int M, double *vol, cudaStream_t st) {
  const size_t N = (size_t)c.n * M;
  const int threads = 256, blocks = (int)((N + threads - 1) / threads);
  k_volume<R><<<blocks, threads, 0, st>>>(c, s, M, vol);
  return cudaGetLastError();
}

template <class R>
cudaError_t launch_balance_sum(const DevCellsT<R> &c, const DevStateT<R> &s, int M, const DevBalance &b,
                               const double *vol0, double *partial, int *nblocks, cudaStream_t st) {
  const size_t N = (size_t)c.n * M;
  const int threads = 256, blocks = (int)((N + threads - 1) / threads);
  *nblocks = blocks;
  k_balance_sum<R><<<blocks, threads, 0, st>>>(c, s, M, b, vol0, partial);
  return cudaGetLastError();
}

#define WG_INSTANTIATE(R)                                                                                          \
  template cudaError_t launch_vertical<R>(const DevCellsT<R> &, const DevStateT<R> &, const DevVertT<R> &,        \
                                          const DevForcing &, int, int, cudaStream_t);                             \
  template cudaError_t launch_pet<R>(const DevCellsT<R> &, const DevForcing &, const DevRingT<R> &, int, int, int,  \
                                     int, int, cudaStream_t);                                                      \
  template int pipeline_max_blocks<R>(bool, bool, int, bool, bool, bool);                                        \
  template int vertical_ahead_max_blocks<R>(bool, int);                                                           \
  template cudaError_t launch_pipeline<R>(bool, const DevCellsT<R> &, const DevStateT<R> &, const DevVertT<R> &,  \
                                          const DevForcing &, const DevMembers &, const DevBalance &,             \
                                          const DevRingT<R> &, const DevSync &, double *, double *, int, int,     \
                                          int, int, int, int, int, int, const WarpLayout &, const DevMonthly &,    \
                                          const DevVaWork &, const DevWaterTemp &, const DevWaterUse &,           \
                                          cudaStream_t);                                                          \
  template cudaError_t launch_vertical_ahead<R>(const DevCellsT<R> &, const DevStateT<R> &, const DevForcing &,   \
                                                const DevMembers &, const DevBalance &, const DevRingT<R> &, int,  \
                                                int, int, int, int, int, int, cudaStream_t, const DevMonthly &,   \
                                                int, bool);                                                              \
  template cudaError_t launch_volume<R>(const DevCellsT<R> &, const DevStateT<R> &, int, double *, cudaStream_t); \
  template cudaError_t launch_balance_sum<R>(const DevCellsT<R> &, const DevStateT<R> &, int, const DevBalance &,  \
                                             const double *, double *, int *, cudaStream_t);
WG_INSTANTIATE(double)
WG_INSTANTIATE(float)

}  // namespace wg
