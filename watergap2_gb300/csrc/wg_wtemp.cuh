// wg_wtemp.cuh -- water temperature of one cell and day on the GPU: the
// reference's calcWaterTempClass::calcWTemp (source/calcWaterTemp.cpp:48-1324),
// the energy balance of Beek et al. (2012) with the thermocline depth of
// Wanders et al. (2019), for the river and the five kinds of surface water
// body, with ice cover.  FP64, branch for branch as the reference.  Its FP64 pipe
// bounds the wavefront (68 cycles per warp and operation, taken or predicated off), so:
// - energies are in units of the heat capacity of a km3 of water, K km3, so that rho c
//   leaves every term but the fluxes', and a temperature is one quotient of energy and
//   volume;
// - quotients and the square root run in fixed point (fm::rcp_pos, fm::div, fm::sqrt),
//   comparisons are those of integers;
// - what depends on the cell alone (areas from percentages, the thermocline volumes, the
//   river bed's terms) is laid out at setup.
// A few ulp of rounding against the oracle, which keeps the reference's expression
// order. 67k cells, 181 days, every kind of water body: the wavefront
// 18.2 -> 13.9 ms.
//
// calcWTemp runs after a cell's routing (routing.cpp:4241-4513) and visits the
// water bodies in routing's own order (local lake, local wetland, global lake,
// reservoir, global wetland, river), each reading what its own routing left
// and what the bodies before it computed.  WtDay therefore runs each body as
// soon as routing_cell has finished it: the body's temperature and ice are
// written to the state at once, and only what the later bodies read (the
// local runoff, the temperature and volume of the next body's inflow) is
// carried on -- a few values instead of calcWTemp's sixty-odd arguments, so
// that the routing kernel holds them in registers.
#pragma once
#include "wg_compare.cuh"
#include "wg_device.h"
#include "wg_fastmath.cuh"

namespace wg {
namespace wt {

typedef Cn<double> W;   // false with a NaN on either side
__device__ __forceinline__ bool wt_lt(double a, double b) { return W::gt(b, a); }
__device__ __forceinline__ bool wt_ge0(double a) { return !C<double>::lt0(a) && !W::nan(a); }
__device__ __forceinline__ double wt_max(double a, double b) { return wt_lt(a, b) ? b : a; }   // std::max
__device__ __forceinline__ double wt_min(double a, double b) { return wt_lt(b, a) ? b : a; }   // std::min
__device__ __forceinline__ double pow4(double x) { const double x2 = x * x; return x2 * x2; }

/* constants, calcWaterTemp.cpp:24-32 (the two exchange coefficients are ints there) */
#define WT_CONV_K 273.15
#define WT_HEAT_CAP_W 4180.
#define WT_RHO_W (1000. * 1.e9)
#define WT_K_H 20
#define WT_K_H_ICE 8
#define WT_PRECIP_T_CORR 1.5
#define WT_LAMBDA_F (333.4 * 1.e3)
#define WT_ALBEDO_W 0.08
#define WT_ALBEDO_I 0.6
#define WT_NO_TEMP (-9999.)
__device__ __forceinline__ bool no_temp(double t) { return __double_as_longlong(t) == __double_as_longlong(WT_NO_TEMP); }
// folded constants of the device version (the oracle keeps the reference's
// separate factors): rho c [J/(km3 K)], a day's W/m2 over a km2 and a mm of evaporation's
// latent heat in K km3, and the day's ice growth per W/m2
#define WT_RC (WT_RHO_W * WT_HEAT_CAP_W)
#define WT_FLUX (1.e6 * 86400. / WT_RC)
#define WT_ICE_PER_FLUX (86400. / 1000. / (WT_LAMBDA_F * WT_RHO_W / 1.e9))

// What every water body of the cell reads on the day (calcWaterTempClass::transfer,
// calcWaterTemp.h:23-95, without the per-body entries).
struct WtCommon {
  double air;       // air temperature [degC]
  double prec;      // open-water precipitation [mm/d]
  double area;      // cell area [km2]
  double rain_k;    // temperature of precipitation and surface runoff [K]
  double gw_k;      // groundwater temperature [K]
  double nr_water;  // net radiation over water [W/m2]
  double lat;       // latent heat of evaporation [K km3 per km3]
  double ice0;      // ice growth's part that the water bodies share [W/m2]
  // runoff into the cell's water bodies, and past them into the river (fractional routing)
  double local_runoff, local_gw_runoff, runoff_into_river, gw_runoff_into_river;
  bool keep_runoff;   // no outflow and no river (river length 55): the runoff stays in the water bodies
  int gw_used;        // an earlier water body took the local runoff
};

/* growth of the ice cover over one day [km] (same expression in every water body;
 * the river passes its storage where the others pass their temperature) */
__device__ __forceinline__ double ice_growth(double prev, const WtCommon &t) {
  return (t.ice0 - WT_K_H_ICE * prev) * WT_ICE_PER_FLUX;
}

/* the clamps every water body ends with (calcWaterTemp.cpp:400-411 and the others) */
__device__ __forceinline__ void finish(const WtCommon &t, double *temp, double *ice, double ice_floor) {
  if (W::gt(*temp, 60.)) *temp = t.air;
  if (wt_lt(*temp, 1.e-10) && !no_temp(*temp)) *temp = 0.;
  if (wt_lt(*ice, ice_floor)) *ice = 0.;
}

/* the energy balance of an open water body once its total energy (without the
 * sensible heat flux) and volume are known: the sensible heat flux may only
 * bring the temperature to the air temperature (calcWaterTemp.cpp:376-395) */
__device__ __forceinline__ double open_water_temp(const WtCommon &t, double energy, double sens, double vol) {
  if (!W::gt0(vol)) return WT_NO_TEMP;
  const double inv = fm::rcp_pos(vol);   // vol > 0
  const bool cools = W::ge(energy * inv - WT_CONV_K, t.air);
  const double temp = (energy - sens) * inv - WT_CONV_K;
  return (cools ? wt_lt(temp, t.air) : W::gt(temp, t.air)) ? t.air : temp;
}

/* the water under an ice cover: stored energy minus the heat to the ice, mixed
 * with the day's inflows of volume in_vol and energy in_e */
__device__ __forceinline__ double under_ice_temp(double stor, double flux_area, double temp_prev, double ice,
                                                 double area, double in_vol, double in_e) {
  double temp = (temp_prev + WT_CONV_K) - fm::div(WT_K_H_ICE * temp_prev * flux_area, stor) - WT_CONV_K;
  if (wt_lt(temp, 0.)) temp = 0.;
  if (W::gt0(in_vol)) {
    const double under = stor - ice * area;
    double e = in_e, v = in_vol;
    if (W::gt0(under)) {
      e += under * (temp + WT_CONV_K);
      v += under;
    }
    temp = fm::div(e, v) - WT_CONV_K;
  }
  return temp;
}

/* the inflows' energy where the body before has no temperature (calcWaterTemp.cpp:683-686):
 * the mean of precipitation and runoff over the whole volume */
__device__ __noinline__ double mean_energy(double e, double vol, double in_vol, double in_temp) {
  return in_temp < 0. ? e / vol * in_vol : in_temp;   // (a NaN goes on)
}

/* local lake, calcWaterTemp.cpp:258-407: share its part of the cell, stor_prev
 * its storage before the day plus its capacity, evapo [mm] after any reduction,
 * rf its reduction factor; ice in *ice (in and out) */
__device__ __forceinline__ double loclake_temp(const WtCommon &t, double share, double stor_prev, double temp_prev,
                                               double evapo, double rf, double *ice_io) {
  double gw = t.local_gw_runoff;
  double ice = *ice_io;
  double temp = 0.;
  int ice_max = 0;
  const double area = t.area * share * rf;
  const double precip = t.prec * 1.e-6 * area;
  double surf = t.local_runoff - t.local_gw_runoff;
  if (t.keep_runoff) {
    surf += t.runoff_into_river - t.gw_runoff_into_river;
    gw += t.gw_runoff_into_river;
  }
  const double flux_area = WT_FLUX * area;
  if (W::le0(t.air) || W::gt0(ice)) {
    ice += ice_growth(temp_prev, t);
    if (W::ge(ice * area, stor_prev)) {
      ice = fm::div(stor_prev, area);
      if (W::le0(precip + surf + t.local_gw_runoff)) ice_max = 1;
    }
  }
  if (!ice_max) {
    if (W::gt0(ice)) {
      const double in_vol = precip + surf + t.local_gw_runoff;
      temp = under_ice_temp(stor_prev, flux_area, temp_prev, ice, area, in_vol,
                            (precip + surf) * t.rain_k + t.local_gw_runoff * t.gw_k);
    } else {
      const double evap = evapo * 1.e-6 * area;
      const double energy = stor_prev * (temp_prev + WT_CONV_K) + (precip + surf) * t.rain_k + gw * t.gw_k +
                            t.nr_water * flux_area - t.lat * evap;
      const double sens = WT_K_H * (temp_prev - t.air) * flux_area;
      temp = open_water_temp(t, energy, sens, stor_prev + precip + surf + t.local_gw_runoff - evap);
    }
  } else {
    temp = W::gt0(ice) ? 0. : WT_NO_TEMP;
  }
  finish(t, &temp, &ice, 0.);
  *ice_io = ice;
  return temp;
}

/* local runoff into the first water body of the cell when no earlier one took it
 * (calcWaterTemp.cpp:447-457 and the same block of the others) */
__device__ __forceinline__ void take_runoff(const WtCommon &t, double *surf, double *gw) {
  if (t.keep_runoff) {
    *surf += t.runoff_into_river - t.gw_runoff_into_river;
    *gw += t.gw_runoff_into_river;
  }
  *surf += t.local_runoff - t.local_gw_runoff;
  *gw += t.local_gw_runoff;
}

/* local wetland (calcWaterTemp.cpp:420-568), global lake, reservoir and global wetland
 * (585-745, 761-915, 931-1081): area [km2], stor_prev the storage that exchanges heat,
 * inflow the volume that comes from the body before and in_temp its temperature (used
 * where with_temp) */
__device__ __forceinline__ double body_temp(const WtCommon &t, double area, double stor_prev, double temp_prev,
                                            double evapo, double inflow, double in_temp, bool with_temp, double *ice_io) {
  double surf = 0., gw = 0.;
  double ice = *ice_io;
  double temp = 0.;
  int ice_max = 0;
  const double precip = t.prec * 1.e-6 * area;
  const double flux_area = WT_FLUX * area;
  if (!t.gw_used) take_runoff(t, &surf, &gw);
  const double own = precip + (surf + gw), in_vol = own + inflow;
  if (W::le0(t.air) || W::gt0(ice)) {
    ice += ice_growth(temp_prev, t);
    if (W::ge(ice * area, stor_prev)) {
      ice = fm::div(stor_prev, area);
      if (W::le0(in_vol)) ice_max = 1;
    }
  }
  if (!ice_max) {
    double in_e = (precip + surf) * t.rain_k + gw * t.gw_k;
    if (with_temp) in_e += inflow * (in_temp + WT_CONV_K);
    if (W::gt0(ice)) {
      if (!with_temp && !C<double>::is_zero(inflow)) in_e = mean_energy(in_e, own, in_vol, in_temp);
      temp = under_ice_temp(stor_prev, flux_area, temp_prev, ice, area, in_vol, in_e);
    } else {
      const double evap = evapo * 1.e-6 * area;
      const double energy = stor_prev * (temp_prev + WT_CONV_K) + in_e + t.nr_water * flux_area - t.lat * evap;
      const double sens = WT_K_H * (temp_prev - t.air) * flux_area;
      temp = open_water_temp(t, energy, sens, stor_prev + in_vol - evap);
    }
  } else {
    temp = W::gt0(ice) ? 0. : WT_NO_TEMP;
  }
  finish(t, &temp, &ice, 0.);
  *ice_io = ice;
  return temp;
}

/* the volume above the thermocline [km3] (calcWaterTemp.cpp:1313-1324) depends on the
 * area alone and is laid out at setup */

/* river, calcWaterTemp.cpp:1097-1298: river_stor its storage after routing,
 * own_prev its temperature of the previous day, inflow the volume of the last
 * water body's outflow (or the upstream inflow) and mix_temp its temperature;
 * power-plant cooling (options.calc_wtemp = 2, calcWaterTemp.cpp:1263-1285) with
 * the day's withdrawal and consumption when calc_pp */
__device__ __forceinline__ double river_temp(const WtCommon &t, double river_stor, double bed, double bed2,
                                             double river_length, double cfa, double ow_pet, double own_prev,
                                             double inflow, double mix_temp, bool calc_pp, double pp_withdrawal,
                                             double pp_consumption, double *ice_io) {
  double area = 0., depth = 0.;
  double gw = t.runoff_into_river;   /* the reference starts its groundwater term from this field */
  double ice = *ice_io;
  int ice_max = 0;
  double temp = 0., vol = 0.;
  const double csa = fm::div(river_stor, river_length);
  if (W::gt0(csa)) {
    depth = -bed + fm::sqrt(bed2 + 0.5 * csa);
    area = fm::div(river_stor, depth);
  }
  const double precip = t.prec * area * 1.e-6;
  const double flux_area = WT_FLUX * area;
  double surf = t.runoff_into_river - t.gw_runoff_into_river;
  if (!t.gw_used) {
    surf += (t.local_runoff - t.local_gw_runoff);
    gw += t.local_gw_runoff;
  }
  const double own = precip + surf + gw, in_vol = own + inflow;
  if (W::le0(t.air) || W::ge(ice, 5.e-6)) {
    if (W::gt0(area)) {
      ice += ice_growth(river_stor, t);
      if (W::ge(ice * area, river_stor)) {
        ice = fm::div(river_stor, area);
        if (W::le0(in_vol)) ice_max = 1;
      }
    } else {
      ice = 0.;
    }
  }
  if (!ice_max) {
    double in_e = (precip + surf) * t.rain_k + gw * t.gw_k;
    const bool with_temp = wt_ge0(mix_temp);
    if (with_temp) in_e += inflow * (mix_temp + WT_CONV_K);
    if (W::ge(ice, 5.e-6)) {
      vol = river_stor;
      if (!with_temp && !C<double>::is_zero(inflow)) in_e = mean_energy(in_e, own, in_vol, mix_temp);
      temp = under_ice_temp(river_stor, flux_area, own_prev, ice, area, in_vol, in_e);
    } else {
      const double evapo = ((1.0 - cfa) * t.prec + (cfa * ow_pet)) * area * 1.e-6;
      if (W::ge(evapo, river_stor + in_vol)) {
        *ice_io = 0.;   /* everything evaporates; the ice record is reset */
        return WT_NO_TEMP;
      }
      const double energy = river_stor * (own_prev + WT_CONV_K) + in_e + t.nr_water * flux_area - t.lat * evapo;
      const double sens = WT_K_H * (own_prev - t.air) * flux_area;
      vol = river_stor + in_vol - evapo;
      temp = open_water_temp(t, energy, sens, vol);
    }
    if (temp >= 0. && pp_withdrawal > 0. && calc_pp) {
      if (ice >= 5.e-6) vol -= ice * area;
      if (vol > 0.) {
        const double wd = vol < pp_withdrawal ? vol : pp_withdrawal;
        const double ret = wd > pp_consumption ? wd - pp_consumption : 0.;
        if (ret > 0.)
          temp = (((vol - wd) * (temp + WT_CONV_K) + ret * (temp + 3. + WT_CONV_K)) / (vol - wd + ret)) - WT_CONV_K;
      }
    }
  } else {
    temp = W::gt0(ice) ? 0. : WT_NO_TEMP;
  }
  finish(t, &temp, &ice, 5.e-6);
  *ice_io = ice;
  return temp;
}

/* mixing temperature of the cell's river inflow (its energy e_in) and its local wetland
 * (or local lake) outflow: the block calcWTemp repeats before each global water body and
 * the river where no global water body came before */
__device__ __forceinline__ double local_mix(double tot_in, double e_in, double loclake_t, double locwetl_t,
                                            double locwetl_inflow, double locwetl_outflow) {
  const bool wetl = wt_ge0(tot_in) && W::gt0(locwetl_outflow);
  if (wetl || W::gt0(tot_in)) {
    const double v = wetl ? locwetl_outflow : locwetl_inflow;
    const double mix = fm::div(e_in + ((wetl ? locwetl_t : loclake_t) + WT_CONV_K) * v, tot_in + v) - WT_CONV_K;
    return wt_lt(mix, 0.) ? 0. : mix;
  }
  return W::gt0(locwetl_inflow) ? loclake_t : WT_NO_TEMP;
}

// One cell's calcWTemp on one day, driven by routing_cell: begin() with the day's
// inputs, runoff() once the runoff is split, one call per water body right after
// its routing (locals_done() between the local and the global ones), river() at
// the end.  Temperatures and ice go to the state [6][N] (index k * N + si; 0
// river, 1 local lake, 2 local wetland, 3 global lake, 4 reservoir, 5 global
// wetland); a water body without a temperature keeps the air temperature (at
// least 0), one the cell does not have gets no ice record (-9999).
struct WtDay {
  const DevWaterTemp *w;   // the state (temp/ice [k * N + si]) and the water-body areas (slot s)
  size_t si, N;
  int s;
  uint32_t fl;          // the cell's flag bits (which water bodies it has)
  WtCommon t;
  double tot_in, e_in;   // upstream river inflow [km3] and its energy [K km3] (calcWaterTemp.cpp:76-90)
  double loclake_t, locwetl_t, ll_out, lw_out;   // the local bodies' temperatures and outflows
  double mix, chain_in;     // temperature and volume of the next global body's (or the river's) inflow
  double last;              // the temperature calcWTemp reports for the cell (its last water body's)
  // the monthly mean temperatures (routing.cpp:4375-4458): sums (k) and day
  // counts (6 + k) of the day's month at msum[k * ms], or null
  double *msum = nullptr;
  size_t ms = 0;
  __device__ __forceinline__ void file(int k, double tk) {
    if (msum && wt_ge0(tk)) {   // a computed temperature (calcWTempReturns[k] >= 0)
      msum[k * ms] += tk;
      msum[(6 + k) * ms] += 1.;
    }
  }

  // tot_in/e_in: the upstream cells' river outflow of the day, summed, and the
  // energy it carries (sum of volume x (T + 273.15))
  __device__ __forceinline__ void begin(const DevWaterTemp *w_, int s_, size_t si_, size_t N_, uint32_t fl_, double air,
                                        double sw, double lw, double prec, double area, double gw_temp,
                                        double tot_in_, double e_in_) {
    w = w_; si = si_; N = N_; fl = fl_; s = s_;
    t.air = air;
    t.prec = prec;
    t.area = area;
    t.rain_k = wt_max(air - WT_PRECIP_T_CORR, 0.) + WT_CONV_K;
    t.gw_k = gw_temp + WT_CONV_K;
    t.lat = W::gt0(air) ? (2.501 - 0.002361 * air) * (1.e6 / WT_HEAT_CAP_W) : 0.;
    const double net_long = lw - 1. * 0.00000005670374419 * pow4(air + WT_CONV_K);
    t.nr_water = (sw * (1. - WT_ALBEDO_W) + net_long);
    t.ice0 = WT_K_H * (-air) - (sw * (1. - WT_ALBEDO_I) + net_long);
    t.keep_runoff = (fl & F_OUTLET) && __double_as_longlong(w->len_check[s]) == __double_as_longlong(55.);
    t.gw_used = 0;
    tot_in = tot_in_;
    e_in = W::gt0(tot_in) ? e_in_ : tot_in * WT_CONV_K;   // (no inflow: 0 degrees)
    loclake_t = 0.; locwetl_t = 0.; ll_out = 0.; lw_out = 0.;
    last = WT_NO_TEMP;
  }
  __device__ __forceinline__ void runoff(double local_runoff, double local_gw_runoff, double into_river,
                                         double gw_into_river) {
    t.local_runoff = local_runoff;
    t.local_gw_runoff = local_gw_runoff;
    t.runoff_into_river = into_river;
    t.gw_runoff_into_river = gw_into_river;
  }
  __device__ __forceinline__ double &temp(int k) const { return w->temp[(size_t)k * N + si]; }
  __device__ __forceinline__ double &ice(int k) const { return w->ice[(size_t)k * N + si]; }
  __device__ __forceinline__ double keep() const { return wt_lt(t.air, 0.) ? 0. : t.air; }
  __device__ __forceinline__ void absent(int k) {
    temp(k) = keep();
    ice(k) = WT_NO_TEMP;
  }
  __device__ __forceinline__ void put(int k, double temp_k, double ice_k) {
    temp(k) = no_temp(temp_k) ? keep() : temp_k;
    ice(k) = ice_k;
    last = temp_k;
    file(k, temp_k);
  }
  // local lake: storage before the day plus capacity, evaporation after any
  // reduction, reduction factor, outflow
  __device__ __forceinline__ void loclake(double stor_prev, double evapo, double rf, double outflow) {
    double ic = ice(1);
    loclake_t = loclake_temp(t, w->ll_part[s], stor_prev, temp(1), evapo, rf, &ic);
    t.gw_used = 1;
    ll_out = outflow;
    put(1, loclake_t, ic);
  }
  __device__ __forceinline__ void locwetl(double stor_prev, double evapo, double rf, double outflow) {
    double ic = ice(2);
    locwetl_t = body_temp(t, t.area * w->lw_part[s] * rf, stor_prev, temp(2), evapo, ll_out, loclake_t,
                          (fl & F_LOCLAKE) != 0, &ic);
    t.gw_used = 1;
    lw_out = outflow;
    put(2, locwetl_t, ic);
  }
  // after the local water bodies: the inflow of the first global one (or of the
  // river) and its temperature
  __device__ __forceinline__ void locals_done() {
    mix = local_mix(tot_in, e_in, loclake_t, locwetl_t, ll_out, lw_out);
    chain_in = tot_in;
    if (fl & F_LOCWETL) chain_in += lw_out;
    else if (fl & F_LOCLAKE) chain_in += ll_out;
  }
  // a global lake (k 3), reservoir (4) or global wetland (5): area [km2], the
  // storage that exchanges heat, evaporation after any reduction, outflow;
  // glolake and res take their storage before the day (with the global lake's
  // capacity added), glowetl also its reduction factor
  __device__ __forceinline__ void global_body(int k, double area, double stor_prev, double evapo, double outflow) {
    double ic = ice(k);
    const double tk = body_temp(t, area, stor_prev, temp(k), evapo, chain_in, mix, wt_ge0(mix), &ic);
    t.gw_used = 1;
    mix = tk;
    chain_in = outflow;
    put(k, tk, ic);
  }
  __device__ __forceinline__ void glolake(double stor_prev, double evapo, double outflow) {
    global_body(3, w->lake_km2[s], wt_min(stor_prev, w->lake_therm[s]), evapo, outflow);
  }
  __device__ __forceinline__ void res(double stor_prev, double evapo, double outflow) {
    global_body(4, w->res_km2[s], wt_min(stor_prev, w->res_therm[s]), evapo, outflow);
  }
  __device__ __forceinline__ void glowetl(double stor_prev, double evapo, double rf, double outflow) {
    global_body(5, t.area * w->gw_part[s] * rf, stor_prev, evapo, outflow);
  }
  // the river (where the cell has an outflow or a river), the water bodies the
  // cell does not have, and the river temperature the downstream cell reads
  __device__ __forceinline__ double river(double river_stor, double river_length, double cfa, double ow_pet) {
    double ice0 = WT_NO_TEMP;
    if (!t.keep_runoff) {
      double ic = ice(0);
      // no power-plant cooling in this path (calc_wtemp = 1)
      last = river_temp(t, river_stor, w->bed[s], w->bed2[s], river_length, cfa, ow_pet, temp(0), chain_in, mix, false, 0., 0.,
                        &ic);
      ice0 = ic;
    }
    file(0, last);   // the cell's reported temperature (calcWTempReturns[0])
    if (!(fl & F_LOCLAKE)) absent(1);
    if (!(fl & F_LOCWETL)) absent(2);
    if (!(fl & F_GLOLAKE)) absent(3);
    if (!(fl & F_RES)) absent(4);
    if (!(fl & F_GLOWETL)) absent(5);
    const double tr = no_temp(last) ? keep() : last;
    temp(0) = tr;
    ice(0) = ice0;
    return tr;
  }
};

}  // namespace wt
}  // namespace wg
