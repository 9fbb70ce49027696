// sc_pass64.cu -- the plain FP64 form: neighbour-list build and force passes.
//
// Compiled with -fmad=false: together with the operation order of sc_pair.cuh and
// the explicit Heun arithmetic below, every pair contribution and every position
// update is the reference's own sequence of IEEE operations
// (tmarschall/spherocyls src/cpp/strain_dynamics.cpp:17-235,
// src/cpp/resize_dynamics.cpp:164-243, src/cpp/spherocyl_box.cpp:303-355).
//
// A pass is two kernels.  k_pairs64 screens every list entry in FP32 and evaluates
// each pair that may touch once, in FP64, with the lower particle index as the
// reference's "p"; k_step64 sums each particle's contributions in list order and runs
// the Heun predictor or corrector.  k_pass64 does both in one thread per particle
// (each pair from both sides): it serves lists longer than a mask word and handles
// whose pair buffers could not be had, with the same bits.
#include "sc_internal.hpp"
#include "sc_pair.cuh"
#include "sc_rebuild.cuh"

namespace sc {

namespace {

// check_neighbors, src/cpp/spherocyl_box.cpp:303-318, with p the lower index.
__device__ __forceinline__ bool nbr_criterion(double2 pp, double2 pq, double sig, double pad,
                                              double gamma, double Lx, double Ly) {
  double dY = pp.y - pq.y;
  dY += Ly * (double)((dY < -0.5 * Ly) - (dY > 0.5 * Ly));
  if (fabs(dY) < sig + pad) {
    double dX = pp.x - pq.x;
    dX += Lx * (double)((dX < -0.5 * Lx) - (dX > 0.5 * Lx));
    double dXmax = dX + 0.5 * dY;  // dX at the largest gamma of the list lifetime
    dX += gamma * dY;
    if (fabs(dX) < sig + pad || fabs(dXmax) < sig + pad) return true;
  }
  return false;
}

// The padded list of slot i (system s): the reference's criterion in FP64, decided in
// FP32 wherever that is certain.  The FP32 copies of the positions move |dX|, |dX + dY/2|
// and |dY| by less than `slack` (see Screen64), so a candidate outside the bound by more
// is out and one inside it by more is in; about one in a thousand is evaluated in FP64.
// Boxes so small that a candidate at the image boundary (|d| = L/2), where FP32 might
// choose the other image, can be in reach evaluate all in FP64.  The FP64 pipe
// bounded the build: 14 operations for each of about 33 candidates a particle took 191 us
// at 131072 particles (a/R 0.25 to 2), the FP32 test takes 26 us.
// GL = 8 threads (sub: which) take the candidates side by side; the list keeps the order of
// the scan.  With one thread a slot small systems wait for 33 loads in turn: 17 us at 1024
// particles, 5 with eight.
template <int GL>
__device__ __forceinline__ void build_nbrs(const Dev& d, const StepScalars* __restrict__ tab,
                                           int row, int i, int s, int sub, unsigned lanes,
                                           Candidates* table) {
  const SysGeom& g = d.geom[s];
  const StepScalars& ts = tab[row * d.nsys + s];
  const float4 ri = d.rec[i];
  const float si = d.rsf[i];
  const int idi = d.id[i];
  const float gam = (float)ts.gamma_p, fLx = (float)ts.Lx_p, fLy = (float)ts.Ly_p;
  const float pad = g.fpad;
  const float slack = 5e-7f * (fmaxf(fLx, fabsf(ri.x)) + fmaxf(fLy, fabsf(ri.y))) *
                          (1.f + fabsf(gam)) +
                      1e-6f * (2.f * g.smax + pad);
  const float reach = g.smax + pad + slack;
  const bool small = !(0.5f * fLx > reach * (1.f + fmaxf(fabsf(gam), 0.5f)) &&
                       0.5f * fLy > reach);
  int col, rw;
  cell_colrow(g, d.cell[i] - g.c0, &col, &rw);
  int cnt = 0;
  // whether candidate j is listed, and which of the two has the lower index
  auto test = [&](int j, bool* ip) {
    const float4 rj = d.rec[j];
    float dx = ri.x - rj.x, dy = ri.y - rj.y;
    dx += fLx * (float)((dx < -0.5f * fLx) - (dx > 0.5f * fLx));
    dy += fLy * (float)((dy < -0.5f * fLy) - (dy > 0.5f * fLy));
    const float near = fminf(fabsf(fmaf(gam, dy, dx)), fabsf(fmaf(0.5f, dy, dx)));
    const float over = fmaxf(fabsf(dy), near) - (si + d.rsf[j] + pad);
    if (!small && over > slack) return false;
    *ip = idi < d.id[j];
    if (small || !(over < -slack)) {
      const double2 pi = d.xy[i], pj = d.xy[j], rai = d.ra[i], raj = d.ra[j];
      // S = R_p + A_p + R_q + A_q summed in the reference's order
      double sig = *ip ? rai.x + rai.y + raj.x + raj.y : raj.x + raj.y + rai.x + rai.y;
      return *ip ? nbr_criterion(pi, pj, sig, g.pad, ts.gamma_p, ts.Lx_p, ts.Ly_p)
                 : nbr_criterion(pj, pi, sig, g.pad, ts.gamma_p, ts.Lx_p, ts.Ly_p);
    }
    return true;
  };
  if (GL == 1) {
    // 3x3 block of cells; a dimension with fewer than three cells is scanned once
    // per distinct cell (the reference would list such cells twice).
    const int ncx = g.cols < 3 ? g.cols : 3, ncy = g.rows < 3 ? g.rows : 3;
    for (int a = 0; a < ncy; a++) {
      const int r2 = ncy == 3 ? wrap_index(rw + a - 1, g.rows) : a;
      for (int b = 0; b < ncx; b++) {
        const int c2 = ncx == 3 ? wrap_index(col + b - 1, g.cols) : b;
        const int cc = g.c0 + cell_local(g, c2, r2);
        const int st = d.cell_start[cc], en = st + d.cell_count[cc];
        for (int j = st; j < en; j++) {
          bool ip = false;
          if (j == i || !test(j, &ip)) continue;
          if (cnt < d.maxn)
            d.nbr[(size_t)cnt * d.ntot + i] = (int)((unsigned)j | (ip ? kOwner64 : 0u));
          cnt++;
        }
      }
    }
  } else {
    const int n = list_candidates(d, g, col, rw, *table, sub, lanes);
    for (int k0 = 0, q = 0; k0 < n; k0 += GL) {
      const int k = k0 + sub;
      bool ip = false, hit = false;
      int j = 0;
      if (k < n) {
        while (k >= table->off[q + 1]) q++;
        j = table->first[q] + k - table->off[q];
        hit = j != i && test(j, &ip);
      }
      const unsigned all = __ballot_sync(lanes, hit) & lanes;
      const int at = cnt + __popc(all & ((1u << (threadIdx.x & 31)) - 1u));
      cnt += __popc(all);
      if (hit && at < d.maxn)
        d.nbr[(size_t)at * d.ntot + i] = (int)((unsigned)j | (ip ? kOwner64 : 0u));
    }
  }
  if (sub != 0) return;
  d.nbr_n[i] = cnt;
  if (cnt > d.maxn) atomicOr(d.status, ST_NBR_OVERFLOW);
}

// The rebuild of the FP64 form (sc_rebuild.cuh): cells, shaft vectors and FP32 copies, lists.
template <int BS>
__global__ void __launch_bounds__(BS, 1024 / BS) k_rebuild64(Dev d,
                                                             const StepScalars* __restrict__ tab,
                                                             int row, int moved) {
  if (!rebuild_pending(d)) return;
  GridBarrier bar(d.gbar);
  const rb::Work<BS> work(d);
  const bool ok = rb::sort_cells<false, BS>(
      d, work, tab, row, moved != 0, bar,
      [&](int i, int, double2 p, double, double2 ra, double2, int, int) {
        const double2 n = d.s_nxy[i];
        d.nxy[i] = n;
        // the records take the memory of this slot's scratch, as other types: no store of
        // theirs before the loads of put_back
        asm volatile("" ::: "memory");
        d.rec[i] = screen_record(p, n);
        d.rf[i] = (float)ra.x;
        d.rsf[i] = (float)(ra.x + ra.y);
        if (d.iaa) d.iaa[i] = shared_rcp(ra.y * ra.y);
      });
  if (!ok) {
    bar.leave();
    return;
  }
  if (work.items > kLaneItems) {
    work.each(d, [&](int i, int s) { build_nbrs<1>(d, tab, row, i, s, 0, 0u, nullptr); });
  } else {
    __shared__ Candidates table[BS / 8];
    const unsigned lanes = 0xffu << (threadIdx.x & 24);
    for (int g = (blockIdx.x * BS + threadIdx.x) / 8; g < work.items; g += gridDim.x * BS / 8) {
      int i, s;
      if (work.at(d, g, &i, &s))
        build_nbrs<8>(d, tab, row, i, s, threadIdx.x & 7, lanes, &table[threadIdx.x / 8]);
    }
  }
  rb::finish(d, bar);
}

// ---- the FP32 screen ----
//
// Each particle keeps (x, y, A cos phi, A sin phi) of the state and of the predictor
// copy rounded to FP32 (Dev::rec, rec_t) and R (rf); 20 bytes a neighbour instead of 48,
// and no instruction of the FP64 pipe, which bounds the pass.  The rounding moves a
// displacement by less than 3.5e-7 X per axis, X the larger of L and the particle's own
// coordinate (that coordinate, a partner's within L and the reach of it, their difference, the
// image shift), by up to 1 + |gamma| of it after the shear: `slack` covers both axes, on top
// of the margins of may_touch_fp32.  (A long step takes particles many boxes out, where the
// pair's own displacement may still be a contact.)  Where a pair at
// the image boundary (|d| = L/2) is out of reach the image may be chosen in FP32; smaller
// boxes take the FP64 displacement.
struct Screen64 {
  double Lx, Ly, gamma;
  float fLx, fLy, fgamma, slack;
  bool small;
};
// of a particle with FP32 record ri
__device__ __forceinline__ Screen64 screen_of(const SysGeom& g, const StepScalars& ts, bool pred,
                                              float4 ri) {
  Screen64 c;
  c.gamma = pred ? ts.gamma_c : ts.gamma_p;
  c.Lx = pred ? ts.Lx_c : ts.Lx_p;
  c.Ly = pred ? ts.Ly_c : ts.Ly_p;
  c.fLx = (float)c.Lx;
  c.fLy = (float)c.Ly;
  c.fgamma = (float)c.gamma;
  c.slack = 5e-7f * (fmaxf(c.fLx, fabsf(ri.x)) + fmaxf(c.fLy, fabsf(ri.y))) *
            (1.f + fabsf(c.fgamma));
  const float reach = g.smax + c.slack;
  c.small = !(0.5f * c.fLx > reach * (1.f + fabsf(c.fgamma)) && 0.5f * c.fLy > reach);
  return c;
}
// whether the pair (i, j), with FP32 records ri, rj and radius sum sig, may touch
__device__ __forceinline__ bool screen_pair(const Screen64& c, const double2* __restrict__ XY,
                                            int i, int j, float4 ri, float4 rj, float sig) {
  float dx, dy;
  if (!c.small) {
    dx = ri.x - rj.x;
    dy = ri.y - rj.y;
    dx += c.fLx * (float)((dx < -0.5f * c.fLx) - (dx > 0.5f * c.fLx));
    dy += c.fLy * (float)((dy < -0.5f * c.fLy) - (dy > 0.5f * c.fLy));
    dx = fmaf(c.fgamma, dy, dx);
  } else {
    const double2 pi = XY[i], pj = XY[j];
    double dX = pi.x - pj.x, dY = pi.y - pj.y;
    dX += c.Lx * (double)((dX < -0.5 * c.Lx) - (dX > 0.5 * c.Lx));
    dY += c.Ly * (double)((dY < -0.5 * c.Ly) - (dY > 0.5 * c.Ly));
    dX += c.gamma * dY;
    dx = (float)dX;
    dy = (float)dY;
  }
  return may_touch_fp32(dx, dy, ri.z, ri.w, rj.z, rj.w, sig + c.slack);
}

// The reference rebuilds inside its corrector loop as soon as particle i has
// moved more than pad/2 (strain_dynamics.cpp:220-225, resize_dynamics.cpp:222-227);
// the lowest such index per system is kept so the rebuild can reproduce which
// particles the reference wrapped before, and which after, their update.
__device__ __forceinline__ void flag_moved(const Dev& d, int s, int id, double2 m, double pad) {
  if (m.x > 0.5 * pad || m.x < -0.5 * pad || m.y > 0.5 * pad || m.y < -0.5 * pad) {
    atomicMin(&d.istar[s], id);
    request_rebuild(d, s);
  }
}

// The Heun step of slot i after its forces (fx, fy, tq) at the pass's positions are
// known: predictor, corrector with the rebuild test, or (PASS_FORCE) the forces alone.
// rot: rot64<MODE> of the slot, which needs no force.
template <int MODE>
__device__ __forceinline__ double rot64(const Dev& d, int i) {
  if (MODE == PASS_PRED_STRAIN) return iso_rot64(d.irc[i].y, d.ph[i]);
  if (MODE == PASS_CORR_STRAIN) return iso_rot64(d.irc[i].y, d.ph_t[i]);
  return 0.0;
}
template <int MODE>
__device__ __forceinline__ void step64_slot(const Dev& d, const StepScalars& ts, const SysGeom& g,
                                            int s, int i, double2 rai, int idi, double gamma,
                                            double rot, double fx, double fy, double tq) {
  const double2 irc = d.irc[i];  // (I, RC)
  const double dt = ts.step;
  if (MODE == PASS_FORCE) {
    d.fx[i] = fx;
    d.fy[i] = fy;
    d.tau[i] = tq;
  } else if (MODE == PASS_PRED_STRAIN) {
    // strain_step predictor, strain_dynamics.cpp:187-199
    d.fx[i] = fx;
    d.fy[i] = fy;
    d.tau[i] = tq;
    double phi = d.ph[i];
    double v0x = fx - gamma * fy;
    double v0y = fy;
    double v0p = tq / irc.x - ts.rate * rot;
    d.v0x[i] = v0x;
    d.v0y[i] = v0y;
    d.v0p[i] = v0p;
    double2 p = d.xy[i];
    double2 pt = make_double2(p.x + dt * v0x, p.y + dt * v0y);
    double pht = phi + dt * v0p;
    d.xy_t[i] = pt;
    d.ph_t[i] = pht;
    double sn, cs;
    sincos(pht, &sn, &cs);
    const double2 nt = make_double2(rai.y * cs, rai.y * sn);
    d.nxy_t[i] = nt;
    d.rec_t[i] = screen_record(pt, nt);
  } else if (MODE == PASS_CORR_STRAIN) {
    // strain_step corrector, strain_dynamics.cpp:203-219
    double v1x = fx - gamma * fy;
    double v1y = fy;
    double v1p = tq / irc.x - ts.rate * rot;
    double ddx = 0.5 * dt * (d.v0x[i] + v1x);
    double ddy = 0.5 * dt * (d.v0y[i] + v1y);
    double ddp = 0.5 * dt * (d.v0p[i] + v1p);
    double2 p = d.xy[i];
    const double2 p0 = p;
    const double phi0 = d.ph[i];
    p.x += ddx;
    p.y += ddy;
    double phi = phi0 + ddp;
    d.xy[i] = p;
    d.ph[i] = phi;
    // pre-step state and increments, for a rebuild that follows this step
    d.s_xy[i] = p0;
    d.s_ph[i] = phi0;
    d.v0x[i] = ddx;
    d.v0y[i] = ddy;
    d.v0p[i] = ddp;
    double2 m = d.moved[i];
    m.x += ddx;
    m.y += ddy;
    d.moved[i] = m;
    double sn, cs;
    sincos(phi, &sn, &cs);
    const double2 n1 = make_double2(rai.y * cs, rai.y * sn);
    d.nxy[i] = n1;
    d.rec[i] = screen_record(p, n1);
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(phi))) atomicOr(d.status, ST_NAN);
    flag_moved(d, s, idi, m, g.pad);
  } else if (MODE == PASS_PRED_RESIZE) {
    // resize_step predictor, resize_dynamics.cpp:172-191
    d.fx[i] = fx;
    d.fy[i] = fy;
    d.tau[i] = tq;
    d.v0x[i] = fx;
    d.v0y[i] = fy;
    d.v0p[i] = tq;
    double2 p = d.xy[i];
    double2 pt;
    double pht;
    if (ts.mode == 3) {
      // pure-shear predictor (pure_euler_est_2p, src/cuda/2point_dynamics.cu:1882-1891,
      // with unit drag and the torque over I): the affine flow (+x/2, -y/2) times the
      // strain rate, and the isolated rotation -RC sin(2 phi)/2, by an Euler step
      const double phi = d.ph[i];
      pt = make_double2(p.x + dt * (fx + 0.5 * ts.rate * p.x),
                        p.y + dt * (fy - 0.5 * ts.rate * p.y));
      pht = phi + dt * (tq / irc.x + ts.rate * (-0.5 * irc.y * sin(2 * phi)));
    } else {
      pt = make_double2(p.x + dt * fx, p.y + dt * fy);
      pht = d.ph[i] + dt * tq / irc.x;
      if (ts.mode == 1) {
        pt.x *= ts.scale;
        pt.y *= ts.scale;
      } else if (ts.mode == 2) {
        pt.x /= ts.scale;
        pt.y /= ts.scale;
      }
    }
    d.xy_t[i] = pt;
    d.ph_t[i] = pht;
    double sn, cs;
    sincos(pht, &sn, &cs);
    const double2 nt = make_double2(rai.y * cs, rai.y * sn);
    d.nxy_t[i] = nt;
    d.rec_t[i] = screen_record(pt, nt);
  } else if (MODE == PASS_CORR_RESIZE) {
    double2 p0 = d.xy[i];
    const double phi0 = d.ph[i];
    double2 p;
    double phi, ddx, ddy, ddp;
    if (ts.mode == 3) {
      // pure-shear corrector (pure_heun_corr_2p, src/cuda/2point_dynamics.cu:2140-2173):
      // the predicted state plus dt/2 times the change of the contact forces
      ddx = 0.5 * dt * (fx - d.v0x[i]);
      ddy = 0.5 * dt * (fy - d.v0y[i]);
      ddp = 0.5 * dt * (tq / irc.x - d.v0p[i] / irc.x);
      const double2 pt = d.xy_t[i];
      p = make_double2(pt.x + ddx, pt.y + ddy);
      phi = d.ph_t[i] + ddp;
    } else {
      // resize_step corrector, resize_dynamics.cpp:194-218
      ddx = 0.5 * dt * (d.v0x[i] + fx);
      ddy = 0.5 * dt * (d.v0y[i] + fy);
      ddp = 0.5 * dt * (d.v0p[i] + tq) / irc.x;
      p = make_double2(p0.x + ddx, p0.y + ddy);
      phi = phi0 + ddp;
      if (ts.mode == 1) {
        p.x *= ts.scale;
        p.y *= ts.scale;
      } else if (ts.mode == 2) {
        p.x /= ts.scale;
        p.y /= ts.scale;
      }
    }
    d.xy[i] = p;
    d.ph[i] = phi;
    d.s_xy[i] = p0;
    d.s_ph[i] = phi0;
    d.v0x[i] = ddx;
    d.v0y[i] = ddy;
    d.v0p[i] = ddp;
    double2 m = d.moved[i];
    m.x += p.x - p0.x;
    m.y += p.y - p0.y;
    d.moved[i] = m;
    double sn, cs;
    sincos(phi, &sn, &cs);
    const double2 n1 = make_double2(rai.y * cs, rai.y * sn);
    d.nxy[i] = n1;
    d.rec[i] = screen_record(p, n1);
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(phi))) atomicOr(d.status, ST_NAN);
    flag_moved(d, s, idi, m, g.pad);
  }
}

// The FP64 pass of one slot: its pairs over its full list, then the Heun epilogue.
template <int MODE, bool SE, bool TWO, bool FAST = false>
__device__ __forceinline__ void pass64_slot(const Dev& d, const StepScalars* __restrict__ tab,
                                            int row, int i) {
  constexpr bool kPred =
      (MODE == PASS_CORR_STRAIN || MODE == PASS_CORR_RESIZE || MODE == PASS_ENERGY_T);
  int s = d.psys[i];
  if (d.skip && d.skip[s]) return;  // a converged minimiser system
  const SysGeom& g = d.geom[s];
  const StepScalars ts = tab[row * d.nsys + s];
  const double2* __restrict__ XY = kPred ? d.xy_t : d.xy;
  const double2* __restrict__ NXY = kPred ? d.nxy_t : d.nxy;
  const double gamma = kPred ? ts.gamma_c : ts.gamma_p;
  const double Lx = kPred ? ts.Lx_c : ts.Lx_p;
  const double Ly = kPred ? ts.Ly_c : ts.Ly_p;
  const bool virial = d.stress_mode == STRESS_VIRIAL;
  constexpr bool two_point = TWO;
  const double two_n = 2.0 * g.n;

  double2 pi = XY[i];
  double2 ni = NXY[i];
  double2 rai = d.ra[i];
  int idi = d.id[i];
  double fx = 0.0, fy = 0.0, tq = 0.0;
  double se0 = 0.0, se1 = 0.0, se2 = 0.0, se3 = 0.0, se4 = 0.0;
  int cnt = d.nbr_n[i];
  if (cnt > d.maxn) cnt = d.maxn;
  const float4* __restrict__ REC = kPred ? d.rec_t : d.rec;
  const float4 ri = REC[i];
  const Screen64 scr = screen_of(g, ts, kPred, ri);
  const float Ri = d.rf[i];
  for (int k0 = 0; k0 < cnt; k0 += 64) {
    // FP32 screen of up to 64 entries: the FP64 contact code then runs only for the
    // entries that may touch, in list order, so the sums are unchanged bit for bit
    unsigned long long cand = 0ull;
    const int kend = cnt - k0 < 64 ? cnt : k0 + 64;
    for (int k = k0; k < kend; k++) {
      const int j = d.nbr[(size_t)k * d.ntot + i] & kSlot64Mask;
      if (screen_pair(scr, XY, i, j, ri, REC[j], Ri + d.rf[j])) cand |= 1ull << (k - k0);
    }
    while (cand) {
      const int k = k0 + __ffsll((long long)cand) - 1;
      cand &= cand - 1ull;
      const unsigned e = (unsigned)d.nbr[(size_t)k * d.ntot + i];
      const int j = (int)(e & kSlot64Mask);
      double2 pj = XY[j];
      double2 nj = NXY[j];
      double2 raj = d.ra[j];
      // the lower particle index plays the reference's "p": select the operands (one
      // copy of the pair code per warp) rather than branch into two
      const bool ip = (e & kOwner64) != 0u;
      const double2 pP = ip ? pi : pj, pQ = ip ? pj : pi;
      const double2 nP = ip ? ni : nj, nQ = ip ? nj : ni;
      const double2 rP = ip ? rai : raj, rQ = ip ? raj : rai;
      const double ivi = d.iaa ? d.iaa[i] : 0.0, ivj = d.iaa ? d.iaa[j] : 0.0;
      PairF64 o;
      const bool hit =
          two_point ? pair2_fp64<SE, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x,
                                           nQ.y, rQ.y, rP.x + rQ.x, gamma, Lx, Ly, two_n, o,
                                           ip ? ivi : ivj, ip ? ivj : ivi)
                    : pair_fp64<SE, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x, nQ.y,
                                          rQ.y, rP.x + rQ.x, gamma, Lx, Ly, virial, two_n, o,
                                          ip ? ivi : ivj, ip ? ivj : ivi);
      if (hit) {
        if (ip) {
          fx += o.fx;
          fy += o.fy;
          tq += o.tp;
          if (SE) {
            se0 += o.e;
            se1 += o.pxx;
            se2 += o.pyy;
            se3 += o.pxy;
            se4 += o.pyx;
          }
        } else {
          fx -= o.fx;
          fy -= o.fy;
          tq += o.tq;
        }
      }
    }
  }
  if (SE) {
    d.se_part[i] = se0;
    d.se_part[(size_t)d.ntot + i] = se1;
    d.se_part[(size_t)2 * d.ntot + i] = se2;
    d.se_part[(size_t)3 * d.ntot + i] = se3;
    d.se_part[(size_t)4 * d.ntot + i] = se4;
  }

  step64_slot<MODE>(d, ts, g, s, i, rai, idi, gamma, rot64<MODE>(d, i), fx, fy, tq);
}

template <int MODE, bool SE, bool TWO, bool FAST = false>
__global__ void __launch_bounds__(128) k_pass64(Dev d, const StepScalars* __restrict__ tab,
                                               int row) {
  if (MODE == PASS_CORR_STRAIN || MODE == PASS_CORR_RESIZE) mark_pending_rebuilds(d, tab, row);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ntot) return;
  pass64_slot<MODE, SE, TWO, FAST>(d, tab, row, i);
}

// ---- a pass with each pair evaluated once ----
//
// k_pairs64, one block of kPairBlock threads per window of pr_win slots.  Phase 1: TPS
// threads per slot screen its list in FP32 and leave the mask of the entries that may
// touch; the pairs the slot owns (its index is the lower one) become the block's jobs,
// in slot and list order.  Phase 2: one thread per job evaluates it in FP64, on full
// warps whatever the lists' lengths, and writes the force and both torques to the
// window's results.  With SE the owners then add their pairs' stress and energy, 128
// jobs at a time, in list order (2: the energy alone).  RES false: no results wanted.
//
// The FP64 pipe (two lanes a cycle and SM) bounds it: about 115 operations a contact
// (sc_pair.cuh keeps comparisons, clamps and repeated divisors off the pipe; with them on
// it, 0.50 ms at 2^20 particles instead of 0.40).  With one thread per particle, each pair
// evaluated from both sides and the screen's displacement in FP64, a shear pass took 2.66
// ms at 2^20 particles and 65 us at 1024 (8 blocks, the rest of the GPU idle); here 0.40 +
// 0.25 ms (k_pairs64 + k_step64) and 7 + 8 us.
constexpr int kPairBlock = 128;

template <int SE, bool RES, bool TWO, bool FAST, int TPS>
__global__ void __launch_bounds__(kPairBlock) k_pairs64(Dev d, const StepScalars* __restrict__ tab,
                                                       int row, int pred) {
  constexpr int S = kPairBlock / TPS;
  __shared__ unsigned short job[S * 64];  // slot in the window << 6 | list entry
  __shared__ int wsum[kPairBlock / 32];
  __shared__ double res[SE == 1 ? 5 : 1][SE ? kPairBlock : 1];
  const int t = threadIdx.x, l = t / TPS, sub = t % TPS;
  const int i0 = blockIdx.x * S, i = i0 + l;
  const double2* __restrict__ XY = pred ? d.xy_t : d.xy;
  const double2* __restrict__ NXY = pred ? d.nxy_t : d.nxy;
  const float4* __restrict__ REC = pred ? d.rec_t : d.rec;
  const size_t ntot = d.ntot;

  unsigned long long m = 0ull, mo = 0ull;
  bool live = i < d.ntot;
  if (live) {
    const int s = d.psys[i];
    live = !(d.skip && d.skip[s]);  // converged minimiser systems have no jobs
    if (live) {
      const float4 ri = REC[i];
      const Screen64 scr = screen_of(d.geom[s], tab[row * d.nsys + s], pred != 0, ri);
      const float Ri = d.rf[i];
      const int cnt = min(d.nbr_n[i], d.maxn);
      for (int k = sub; k < cnt; k += TPS) {
        const unsigned e = (unsigned)d.nbr[k * ntot + i];
        // a pass without results has no use for the entries it does not own
        if (!RES && !(e & kOwner64)) continue;
        const int j = (int)(e & kSlot64Mask);
        if (screen_pair(scr, XY, i, j, ri, REC[j], Ri + d.rf[j])) {
          m |= 1ull << k;
          if (e & kOwner64) mo |= 1ull << k;
        }
      }
    }
  }
  for (int o = 1; o < TPS; o <<= 1) {
    m |= __shfl_xor_sync(0xffffffffu, m, o);
    mo |= __shfl_xor_sync(0xffffffffu, mo, o);
  }
  // exclusive scan of the slots' job counts over the block
  const int c = sub == 0 ? __popcll(mo) : 0;
  int v = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if ((t & 31) >= o) v += u;
  }
  if ((t & 31) == 31) wsum[t >> 5] = v;
  __syncthreads();
  int off = v - c, total = 0;
  for (int w = 0; w < kPairBlock / 32; w++) {
    if (w < (t >> 5)) off += wsum[w];
    total += wsum[w];
  }
  const bool fits = total <= S * kPairCap;
  if (sub == 0 && live) {
    if (RES) {
      d.pr_mask[i] = m;
      d.pr_info[i] = fits ? (unsigned)off | (unsigned)c << 16 : kPairsOver;
    }
    int q = off;
    for (unsigned long long b = mo; b; b &= b - 1ull)
      job[q++] = (unsigned short)(l << 6 | (__ffsll((long long)b) - 1));
  }
  __syncthreads();

  double acc[SE == 1 ? 5 : 1] = {};
  const size_t base = (size_t)i0 * kPairCap;
  for (int b0 = 0; b0 < total; b0 += kPairBlock) {
    const int p = b0 + t;
    if (p < total) {
      const int io = i0 + (job[p] >> 6), k = job[p] & 63;
      const int j = (int)((unsigned)d.nbr[k * ntot + io] & kSlot64Mask);
      const int s = d.psys[io];
      const StepScalars& ts = tab[row * d.nsys + s];
      const double gamma = pred ? ts.gamma_c : ts.gamma_p;
      const double Lx = pred ? ts.Lx_c : ts.Lx_p, Ly = pred ? ts.Ly_c : ts.Ly_p;
      const double two_n = SE ? 2.0 * d.geom[s].n : 0.0;
      const double2 pP = XY[io], pQ = XY[j], nP = NXY[io], nQ = NXY[j], rP = d.ra[io], rQ = d.ra[j];
      const double iP = FAST ? 0.0 : d.iaa[io], iQ = FAST ? 0.0 : d.iaa[j];
      PairF64 o;
      const bool hit =
          TWO ? pair2_fp64<SE != 0, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x, nQ.y,
                                          rQ.y, rP.x + rQ.x, gamma, Lx, Ly, two_n, o, iP, iQ)
              : pair_fp64<SE != 0, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x, nQ.y,
                                         rQ.y, rP.x + rQ.x, gamma, Lx, Ly,
                                         d.stress_mode == STRESS_VIRIAL, two_n, o, iP, iQ);
      if (RES && fits) {
        d.pr_who[base + p] = hit ? j : -1;
        if (hit) {
          double4_16a r;
          r.x = o.fx;
          r.y = o.fy;
          r.z = o.tp;
          r.w = o.tq;
          d.pr_res[base + p] = r;
        }
      }
      if (SE) res[0][t] = hit ? o.e : 0.0;
      if (SE == 1) {
        res[1][t] = hit ? o.pxx : 0.0;
        res[2][t] = hit ? o.pyy : 0.0;
        res[3][t] = hit ? o.pxy : 0.0;
        res[4][t] = hit ? o.pyx : 0.0;
      }
    }
    if (SE) {
      __syncthreads();
      const int q0 = max(off, b0), q1 = min(off + c, b0 + kPairBlock);
      for (int q = q0; q < q1; q++)
        for (int comp = 0; comp < (SE == 1 ? 5 : 1); comp++) acc[comp] += res[comp][q - b0];
      __syncthreads();
    }
  }
  if (SE && live && sub == 0)
    for (int comp = 0; comp < (SE == 1 ? 5 : 1); comp++) d.se_part[comp * ntot + i] = acc[comp];
}

// One pair of a window whose results did not fit, evaluated where it is needed (the same
// operations, so the same bits); out of line, since it hardly ever runs.
template <bool TWO, bool FAST>
__device__ __noinline__ bool pair_again64(const double2* XY, const double2* NXY,
                                          const double2* ra, const double* iaa, int iP, int iQ,
                                          double gamma, double Lx, double Ly, double4_16a* r) {
  const double2 pP = XY[iP], pQ = XY[iQ], nP = NXY[iP], nQ = NXY[iQ], rP = ra[iP], rQ = ra[iQ];
  PairF64 o;
  const bool hit =
      TWO ? pair2_fp64<false, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x, nQ.y, rQ.y,
                                    rP.x + rQ.x, gamma, Lx, Ly, 0.0, o, iaa[iP], iaa[iQ])
          : pair_fp64<false, FAST>(pP.x - pQ.x, pP.y - pQ.y, nP.x, nP.y, rP.y, nQ.x, nQ.y, rQ.y,
                                   rP.x + rQ.x, gamma, Lx, Ly, false, 0.0, o, iaa[iP], iaa[iQ]);
  if (hit) {
    r->x = o.fx;
    r->y = o.fy;
    r->z = o.tp;
    r->w = o.tq;
  }
  return hit;
}

// The contribution of entry e of slot i's list (info: its pr_info, rank: the owned entries
// before e that may touch) to its force and torque; zero where there is no contact.
template <int MODE, bool TWO, bool FAST>
__device__ __forceinline__ void pair_result64(const Dev& d, const StepScalars& ts, double gamma,
                                              int i, unsigned info, unsigned e, int rank,
                                              double& x, double& y, double& q) {
  constexpr bool kCorr = MODE == PASS_CORR_STRAIN || MODE == PASS_CORR_RESIZE;
  const int win = d.pr_win;
  const int j = (int)(e & kSlot64Mask);
  const bool ip = (e & kOwner64) != 0u;
  const int o = ip ? i : j;  // the owner
  const unsigned inf = ip ? info : d.pr_info[j];
  double4_16a r;
  bool hit = false;
  if (inf == kPairsOver) {
    const double Lx = kCorr ? ts.Lx_c : ts.Lx_p, Ly = kCorr ? ts.Ly_c : ts.Ly_p;
    hit = pair_again64<TWO, FAST>(kCorr ? d.xy_t : d.xy, kCorr ? d.nxy_t : d.nxy, d.ra, d.iaa, o,
                                  ip ? j : i, gamma, Lx, Ly, &r);
  } else {
    const size_t q0 = (size_t)(o / win) * win * kPairCap + (inf & 0xffffu);
    if (ip) {
      hit = d.pr_who[q0 + rank] >= 0;
      if (hit) r = d.pr_res[q0 + rank];
    } else {
      const int n = (int)(inf >> 16);
      for (int k = 0; k < n; k++)
        if (d.pr_who[q0 + k] == i) {
          hit = true;
          r = d.pr_res[q0 + k];
          break;
        }
    }
  }
  x = hit ? (ip ? r.x : -r.x) : 0.0;
  y = hit ? (ip ? r.y : -r.y) : 0.0;
  q = hit ? (ip ? r.z : r.w) : 0.0;
}

// k_step64: a slot's contributions from the pair results, in list order (its own pairs
// follow each other in its window; a pair it does not own is looked up among its partner's
// two or three), then the Heun epilogue.  GL = 1: a thread does all of it for its slot.
// GL = 8, for small systems, where the gather's chain of dependent loads (four or five
// contacts of three loads each) is what the kernel waits for: eight threads of a slot
// fetch a contribution each (the last sixteen of the block take the cosine of the rotation
// first, beside the other warps' fetches), and one thread a slot sums and steps.
constexpr int kStepBlock = 128;

template <int MODE, bool TWO, bool FAST, int GL>
__global__ void __launch_bounds__(kStepBlock) k_step64(Dev d, const StepScalars* __restrict__ tab,
                                                      int row) {
  constexpr bool kCorr = MODE == PASS_CORR_STRAIN || MODE == PASS_CORR_RESIZE;
  constexpr int S = kStepBlock / GL;
  if (kCorr) mark_pending_rebuilds(d, tab, row);
  const int t = threadIdx.x, l = t / GL, sub = t % GL;
  const int i = blockIdx.x * S + l;
  int s = 0;
  bool live = i < d.ntot;
  if (live) {
    s = d.psys[i];
    live = !(d.skip && d.skip[s]);  // not a converged minimiser system
  }
  if (GL == 1 && !live) return;
  const StepScalars& ts = tab[row * d.nsys + s];
  const double gamma = kCorr ? ts.gamma_c : ts.gamma_p;
  double fx = 0.0, fy = 0.0, tq = 0.0;
  if constexpr (GL == 1) {
    const unsigned info = d.pr_info[i];
    int rank = 0;
    for (unsigned long long m = d.pr_mask[i]; m; m &= m - 1ull) {
      const unsigned e = (unsigned)d.nbr[(size_t)(__ffsll((long long)m) - 1) * d.ntot + i];
      double x, y, q;
      pair_result64<MODE, TWO, FAST>(d, ts, gamma, i, info, e, rank, x, y, q);
      rank += (e & kOwner64) != 0u;
      fx += x;
      fy += y;
      tq += q;
    }
    step64_slot<MODE>(d, ts, d.geom[s], s, i, d.ra[i], d.id[i], gamma, rot64<MODE>(d, i), fx, fy,
                      tq);
  } else {
    __shared__ double part[3][kStepBlock], rot[S];
    __shared__ int left[S];
    // the last S threads: the rotation of the block's slots
    const int ir = blockIdx.x * S + t - (kStepBlock - S);
    if (t >= kStepBlock - S && ir < d.ntot) rot[t - (kStepBlock - S)] = rot64<MODE>(d, ir);
    unsigned long long m = live ? d.pr_mask[i] : 0ull;
    const unsigned info = live ? d.pr_info[i] : 0u;
    int rank = 0, more;
    do {
      // this thread's entry: the sub-th of the mask's remaining ones
      unsigned long long b = m;
      for (int k = 0; k < sub; k++) b &= b - 1ull;
      unsigned e = 0u;
      if (b) e = (unsigned)d.nbr[(size_t)(__ffsll((long long)b) - 1) * d.ntot + i];
      const unsigned group = (__ballot_sync(0xffffffffu, (e & kOwner64) != 0u) >>
                              ((t & 31) / GL * GL)) & ((1u << GL) - 1u);
      double x = 0.0, y = 0.0, q = 0.0;
      if (b)
        pair_result64<MODE, TWO, FAST>(d, ts, gamma, i, info, e,
                                       rank + __popc(group & ((1u << sub) - 1u)), x, y, q);
      rank += __popc(group);
      part[0][t] = x;
      part[1][t] = y;
      part[2][t] = q;
      if (sub == 0) left[l] = __popcll(m);
      for (int k = 0; k < GL; k++) m &= m - 1ull;
      more = __syncthreads_or(m != 0ull);
      if (t < S) {
        const int n = min(left[t], GL);
        for (int k = 0; k < n; k++) {
          fx += part[0][t * GL + k];
          fy += part[1][t * GL + k];
          tq += part[2][t * GL + k];
        }
      }
      if (more) __syncthreads();
    } while (more);
    const int io = blockIdx.x * S + t;
    if (t >= S || io >= d.ntot) return;
    const int so = d.psys[io];
    if (d.skip && d.skip[so]) return;
    const StepScalars& to = tab[row * d.nsys + so];
    step64_slot<MODE>(d, to, d.geom[so], so, io, d.ra[io], d.id[io],
                      kCorr ? to.gamma_c : to.gamma_p, rot[t], fx, fy, tq);
  }
}

// ---- stress and energy of the mixed form, in FP64 ----
//
// The mixed form advances with FP32 pair forces, but the stress tensor and the
// energy it reports are those of the FP64 form at its state: on the steps that
// record them, the compensated state (FP32 value plus FP32 compensation, about
// 48 bits) is widened to FP64 relative to each particle's cell centre, the shaft
// vectors are recomputed in FP64, and every listed pair is evaluated by the FP64
// pair code (the reference's operation order, lower particle index as "p") with
// the sums of calc_se (src/cpp/spherocyl_box.cpp:425-522).  The quantities then
// differ from the FP64 form's only through the states themselves.

// FP64 local positions and shaft vectors of the state (scratch: the FP64 predictor
// arrays, which the mixed form does not use)
__global__ void k_mx_se_prep(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ntot) return;
  const float4 r = d.rec[i];
  const float4 c = d.mc[i];
  const double phi = widen(c.z) + widen(c.w);
  const double A = d.ra[i].y;
  double sn, cs;
  sincos(phi, &sn, &cs);
  d.xy_t[i] = make_double2(widen(r.x) + widen(c.x), widen(r.y) + widen(c.y));
  d.nxy_t[i] = make_double2(A * cs, A * sn);
}

// The mixed form's FP64 stress and energy of the state, one block per window of
// kPairBlock / TPS slots, in the phases of k_pairs64: TPS threads per slot screen the mixed
// list (entries: slot | cell offset code) with the FP32 records and mark the pairs that
// the slot owns (its index is the lower one) and that may touch; one thread a pair evaluates
// them, 128 at a time, in FP64 with shared reciprocals (FAST: this stress is the mixed
// form's, checked against the FP64 form to 1e-9, not the reference's rounding); each
// owner adds the results of its own pairs in list order, so the sums are deterministic.
// Systems whose grid has under three cells a side evaluate every pair they own: their
// image is chosen in FP64.
// With the screen's displacements in FP64 and one thread a slot it took 35 us at 16384
// particles and 942 us at 2^20; now 18 and 446.
template <bool TWO, bool FAST, int TPS>
__global__ void __launch_bounds__(kPairBlock) k_mx_se64(Dev d, const StepScalars* __restrict__ tab,
                                                       int row) {
  constexpr int S = kPairBlock / TPS;
  __shared__ unsigned short job[S * 64];  // slot in the window << 6 | entry of the 64
  __shared__ int wsum[kPairBlock / 32];
  __shared__ int longest;
  __shared__ double res[5][kPairBlock];
  const int t = threadIdx.x, l = t / TPS, sub = t % TPS;
  const int i0 = blockIdx.x * S, i = i0 + l;
  const bool valid = i < d.ntot;
  const size_t ntot = d.ntot;
  int cnt = 0, idi = 0;
  float4 ri = make_float4(0.f, 0.f, 0.f, 0.f);
  float Ri = 0.f, W = 0.f, H = 0.f, gam = 0.f;
  bool small = false;
  if (valid) {
    const int s = d.psys[i];
    const SysGeom& g = d.geom[s];
    const StepScalars& ts = tab[row * d.nsys + s];
    W = ts.f_Wp;
    H = ts.f_Hp;
    gam = ts.f_gamma_p;
    small = g.cols < 3 || g.rows < 3;
    ri = d.rec[i];
    // with what the rounding of local positions (up to a cell) and shaft vectors may add
    Ri = d.rf[i] + 1e-6f * g.smax * (1.f + fabsf(gam));
    idi = d.id[i];
    cnt = min(d.nbr_n[i], d.maxn);
  }
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (t == 0) longest = 0;
  __syncthreads();
  if (cnt > 64) atomicMax(&longest, cnt);  // more than one window of 64 entries: rare
  for (int k0 = 0;; k0 += 64) {
    unsigned long long m = 0ull;
    const int kend = min(cnt, k0 + 64);
    for (int k = k0 + sub; k < kend; k += TPS) {
      const unsigned e = (unsigned)d.nbr[k * ntot + i];
      const int j = (int)(e & kSlotMask);
      if (!(idi < d.id[j])) continue;
      const float4 rj = d.rec[j];
      const float dx = ri.x - rj.x + (float)(1 - (int)((e >> 28) & 3u)) * W;
      const float dy = ri.y - rj.y + (float)(1 - (int)(e >> 30)) * H;
      if (small || may_touch_fp32(fmaf(gam, dy, dx), dy, ri.z, ri.w, rj.z, rj.w, Ri + d.rf[j]))
        m |= 1ull << (k - k0);
    }
    for (int o = 1; o < TPS; o <<= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
    // exclusive scan of the slots' job counts over the block
    const int c = sub == 0 ? __popcll(m) : 0;
    int v = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if ((t & 31) >= o) v += u;
    }
    if ((t & 31) == 31) wsum[t >> 5] = v;
    __syncthreads();
    int off = v - c, total = 0;
    for (int w = 0; w < kPairBlock / 32; w++) {
      if (w < (t >> 5)) off += wsum[w];
      total += wsum[w];
    }
    if (sub == 0) {
      int q = off;
      for (unsigned long long b = m; b; b &= b - 1ull)
        job[q++] = (unsigned short)(l << 6 | (__ffsll((long long)b) - 1));
    }
    __syncthreads();
    for (int b0 = 0; b0 < total; b0 += kPairBlock) {
      const int p = b0 + t;
      if (p < total) {
        const int io = i0 + (job[p] >> 6), k = k0 + (job[p] & 63);
        const unsigned e = (unsigned)d.nbr[k * ntot + io];
        const int j = (int)(e & kSlotMask);
        const int s = d.psys[io];
        const SysGeom& g = d.geom[s];
        const StepScalars& ts = tab[row * d.nsys + s];
        const double2 pi = d.xy_t[io], pj = d.xy_t[j], ni = d.nxy_t[io], nj = d.nxy_t[j];
        const double2 rai = d.ra[io], raj = d.ra[j];
        const double dX = (pi.x - pj.x) + (double)(1 - (int)((e >> 28) & 3u)) * ts.W_p;
        const double dY = (pi.y - pj.y) + (double)(1 - (int)(e >> 30)) * ts.H_p;
        const double two_n = 2.0 * g.n, i2n = 0.5 * g.inv_n;
        PairF64 r;
        const bool hit =
            TWO ? pair2_fp64<true, FAST>(dX, dY, ni.x, ni.y, rai.y, nj.x, nj.y, raj.y,
                                         rai.x + raj.x, ts.gamma_p, ts.Lx_p, ts.Ly_p, two_n, r,
                                         0.0, 0.0, ts.inv_area, i2n)
                : pair_fp64<true, FAST>(dX, dY, ni.x, ni.y, rai.y, nj.x, nj.y, raj.y,
                                        rai.x + raj.x, ts.gamma_p, ts.Lx_p, ts.Ly_p,
                                        d.stress_mode == STRESS_VIRIAL, two_n, r, 0.0, 0.0,
                                        ts.inv_area, i2n);
        res[0][t] = hit ? r.e : 0.0;
        res[1][t] = hit ? r.pxx : 0.0;
        res[2][t] = hit ? r.pyy : 0.0;
        res[3][t] = hit ? r.pxy : 0.0;
        res[4][t] = hit ? r.pyx : 0.0;
      }
      __syncthreads();
      // each owner adds its pairs of this batch, in list order (a pair that does
      // not touch adds zeros)
      const int q0 = max(off, b0), q1 = min(off + c, b0 + kPairBlock);
      for (int q = q0; q < q1; q++)
        for (int comp = 0; comp < 5; comp++) acc[comp] += res[comp][q - b0];
      __syncthreads();
    }
    __syncthreads();  // longest is complete, the jobs are done with
    if (k0 + 64 >= longest) break;
  }
  if (valid && sub == 0)
    for (int comp = 0; comp < 5; comp++) d.se_part[comp * ntot + i] = acc[comp];
}

template <int MODE, bool SE, bool FAST = false>
void launch_whole(const Dev& d, const StepScalars* tab, int row, cudaStream_t st) {
  const int block = 128, grid = (d.ntot + block - 1) / block;
  if (d.contact_model == 1)
    k_pass64<MODE, SE, true, FAST><<<grid, block, 0, st>>>(d, tab, row);
  else
    k_pass64<MODE, SE, false, FAST><<<grid, block, 0, st>>>(d, tab, row);
}

template <int SE, bool RES, bool FAST, int TPS>
void launch_pairs_of(const Dev& d, const StepScalars* tab, int row, int pred, cudaStream_t st) {
  const int grid = (d.ntot + d.pr_win - 1) / d.pr_win;
  if (d.contact_model == 1)
    k_pairs64<SE, RES, true, FAST, TPS><<<grid, kPairBlock, 0, st>>>(d, tab, row, pred);
  else
    k_pairs64<SE, RES, false, FAST, TPS><<<grid, kPairBlock, 0, st>>>(d, tab, row, pred);
}

template <int SE, bool RES, bool FAST>
void launch_pairs(const Dev& d, const StepScalars* tab, int row, bool pred, cudaStream_t st) {
  switch (kPairBlock / d.pr_win) {
    case 1: launch_pairs_of<SE, RES, FAST, 1>(d, tab, row, pred, st); break;
    case 4: launch_pairs_of<SE, RES, FAST, 4>(d, tab, row, pred, st); break;
    case 16: launch_pairs_of<SE, RES, FAST, 16>(d, tab, row, pred, st); break;
  }
}

template <int MODE, bool FAST, int GL>
void launch_step_of(const Dev& d, const StepScalars* tab, int row, cudaStream_t st) {
  const int grid = (d.ntot + kStepBlock / GL - 1) / (kStepBlock / GL);
  if (d.contact_model == 1)
    k_step64<MODE, true, FAST, GL><<<grid, kStepBlock, 0, st>>>(d, tab, row);
  else
    k_step64<MODE, false, FAST, GL><<<grid, kStepBlock, 0, st>>>(d, tab, row);
}

template <int MODE, bool FAST = false>
void launch_step(const Dev& d, const StepScalars* tab, int row, cudaStream_t st) {
  // eight threads a slot against one, a shear step in us: 43 and 56 at 1024 particles, 53
  // and 66 at 8192, 77 and 77 at 16384, 109 and 97 at 32768
  if (d.ntot <= 8192)
    launch_step_of<MODE, FAST, 8>(d, tab, row, st);
  else
    launch_step_of<MODE, FAST, 1>(d, tab, row, st);
}

// the pass of one mode through the pair buffers, or in one kernel without them
template <int MODE>
int launch_mode(const Dev& d, bool se, const StepScalars* tab, int row, cudaStream_t st) {
  constexpr bool corr = MODE == PASS_CORR_STRAIN || MODE == PASS_CORR_RESIZE;
  if (d.pr_win == 0) {
    if constexpr (corr)
      launch_whole<MODE, false>(d, tab, row, st);
    else
      se ? launch_whole<MODE, true>(d, tab, row, st) : launch_whole<MODE, false>(d, tab, row, st);
    return 1;
  }
  if (!corr && se)
    launch_pairs<1, true, false>(d, tab, row, corr, st);
  else
    launch_pairs<0, true, false>(d, tab, row, corr, st);
  launch_step<MODE>(d, tab, row, st);
  return 2;
}

}  // namespace

// Slots per window of the pair results: small systems take small windows, several threads
// screening a slot, which puts the pairs on more SMs.  A shear step in us with windows of
// 8, 32 and 128 slots: 43, 46 and 72 at 1024 particles, 48, 49 and 76 at 4096, 88, 77 and 91
// at 16384, 210, 145 and 149 at 65536, 365, 236 and 224 at 131072.
int pair_window(int ntot) {
  return ntot <= 4096 ? kPairBlock / 16 : ntot <= 65536 ? kPairBlock / 4 : kPairBlock;
}

int launch_pass_fp64(const Dev& d, int mode, bool se, const StepScalars* tab, int row,
                     cudaStream_t st, bool fast) {
  if (fast && !d.odd_shapes && mode == PASS_FORCE && !se) {
    // the minimiser's force evaluation (shared reciprocals, see qdiv)
    if (d.pr_win == 0) {
      launch_whole<PASS_FORCE, false, true>(d, tab, row, st);
      return 1;
    }
    launch_pairs<0, true, true>(d, tab, row, false, st);
    launch_step<PASS_FORCE, true>(d, tab, row, st);
    return 2;
  }
  switch (mode) {
    case PASS_FORCE: return launch_mode<PASS_FORCE>(d, se, tab, row, st);
    case PASS_CORR_STRAIN: return launch_mode<PASS_CORR_STRAIN>(d, false, tab, row, st);
    case PASS_PRED_STRAIN: return launch_mode<PASS_PRED_STRAIN>(d, se, tab, row, st);
    case PASS_CORR_RESIZE: return launch_mode<PASS_CORR_RESIZE>(d, false, tab, row, st);
    case PASS_PRED_RESIZE: return launch_mode<PASS_PRED_RESIZE>(d, se, tab, row, st);
    case PASS_ENERGY_T:
      if (d.pr_win == 0)
        launch_whole<PASS_ENERGY_T, true>(d, tab, row, st);
      else
        launch_pairs<2, false, false>(d, tab, row, true, st);
      return 1;
  }
  return 0;
}

template <int TPS>
static void launch_mx_se64_of(const Dev& d, const StepScalars* tab, int row, cudaStream_t st) {
  const int grid = (d.ntot + kPairBlock / TPS - 1) / (kPairBlock / TPS);
  if (d.contact_model == 1)
    (d.odd_shapes ? k_mx_se64<true, false, TPS> : k_mx_se64<true, true, TPS>)<<<
        grid, kPairBlock, 0, st>>>(d, tab, row);
  else
    (d.odd_shapes ? k_mx_se64<false, false, TPS> : k_mx_se64<false, true, TPS>)<<<
        grid, kPairBlock, 0, st>>>(d, tab, row);
}

void launch_mx_se64(const Dev& d, const StepScalars* tab, int row, cudaStream_t st) {
  k_mx_se_prep<<<(d.ntot + 127) / 128, 128, 0, st>>>(d);
  switch (kPairBlock / pair_window(d.ntot)) {
    case 1: launch_mx_se64_of<1>(d, tab, row, st); break;
    case 4: launch_mx_se64_of<4>(d, tab, row, st); break;
    case 16: launch_mx_se64_of<16>(d, tab, row, st); break;
  }
}

int launch_rebuild_fp64(const Dev& d, const StepScalars* tab, int row, bool moved,
                        cudaStream_t st) {
  int mv = moved ? 1 : 0;
  void* args[] = {(void*)&d, (void*)&tab, &row, &mv};
  if (d.ntot <= kSmallRebuild) {
    const void* fn = (const void*)k_rebuild64<128>;
    cudaLaunchCooperativeKernel(fn, coop_blocks<0>(fn, 128, (d.ntot + 15) / 16), 128, args, 0, st);
  } else {
    const void* fn = (const void*)k_rebuild64<512>;
    cudaLaunchCooperativeKernel(fn, coop_blocks<1>(fn, 512, (d.ntot + 63) / 64), 512, args, 0,
                                st);
  }
  return 1;
}

}  // namespace sc
