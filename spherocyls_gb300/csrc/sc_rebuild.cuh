// sc_rebuild.cuh -- the cell rebuild as the phases of one cooperative kernel (device code).
//
// The rebuild follows the reference's find_cells / find_neighbors
// (tmarschall/spherocyls src/cpp/spherocyl_box.cpp:270-355): positions are wrapped
// into the box, each particle is hashed to its cell (col + row*cols in the
// reference; here numbered tile by tile, see cell_local), and the cell lists
// hold particles in increasing particle index.  On the GPU the lists are a
// counting sort of the particle arrays themselves into cell order:
//
//   hash (set-back, wrap, an arrival rank inside the cell) | cell starts | the indices of
//   each cell side by side | every particle to its place (its rank by index among its
//   cell's) in scratch | back, with the records the passes read | neighbour lists
//
// with a grid barrier at each bar.  Every step carries the kernel; without a pending
// rebuild it returns at once.  That costs 1.3 us a step.  The chain of 13 kernels it
// replaces sat in a conditional graph node, which cost 7 us a step when it was not taken
// and 32 to 39 us before its first kernel when it was.
//
// The phases take the slots of the flagged systems, so that a rebuild of a few systems of a
// large batch costs in proportion to them: every block lists those systems in its shared
// memory and finds a work item's system by binary search there.
//
// The mixed form compiles this with fused multiply-adds, the FP64 form without: what both
// compute is written so that the flag makes no difference.
#pragma once

#include <atomic>

#include "sc_internal.hpp"
#include "sc_pair.cuh"

namespace sc {
namespace rb {

constexpr double kRefPi = 3.14159265358979;  // src/cpp/spherocyl_box.cpp:12

// The reference's wrap loops (while v > hi: v -= period; while v < lo: v += period).
// A runaway value would make them spin for ever; after 64 periods the wrap
// finishes with floor() and flags the state as non-finite instead.
__device__ __forceinline__ double wrap_bounded(double v, double lo, double hi, double period,
                                               int* status) {
  int it = 0;
  while (v > hi && it < 64) {
    v -= period;
    it++;
  }
  while (v < lo && it < 64) {
    v += period;
    it++;
  }
  if (it >= 64) {
    v = __dsub_rn(v, __dmul_rn(period, floor((v - lo) / period)));
    atomicOr(status, ST_NAN);
  }
  return v;
}

// The same for a value that hardly ever needs it: within [0, hi], or within [-hi, hi],
// decided on its bits (the comparisons run on the FP64 pipe).
__device__ __forceinline__ double wrap_side(double v, double L, int* status) {
  if ((unsigned long long)__double_as_longlong(v) <= (unsigned long long)__double_as_longlong(L))
    return v;
  return wrap_bounded(v, 0.0, L, L, status);
}
__device__ __forceinline__ double wrap_angle(double v, int* status) {
  if (abs_bits(v) <= (unsigned long long)__double_as_longlong(kRefPi)) return v;
  return wrap_bounded(v, -kRefPi, kRefPi, 2 * kRefPi, status);
}

// The flagged systems of a handle, listed by each block for itself: first work item of each
// and its slot, in shared memory.  More than kMaxWork of them: every slot is a work item,
// and those of other systems are passed over.
constexpr int kMaxWork = 1024;
template <int BS>
struct Work {
  int count, items;  // listed systems (-1: all slots are items), work items
  int windows;       // windows of kOrderWindow slots that hold any of them
  const int* off;    // [count] first item
  const int* sys;    // [count] system
  const int* woff;   // [count] first window item

  __device__ __forceinline__ explicit Work(const Dev& d) {
    __shared__ int s_off[kMaxWork], s_sys[kMaxWork], s_win[kMaxWork], sums[3][BS / 32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    off = s_off;
    sys = s_sys;
    woff = s_win;
    count = items = windows = 0;
    const int all = (d.ntot + kOrderWindow - 1) / kOrderWindow;
    if (d.nsys == 1) {
      if (t == 0) s_off[0] = s_sys[0] = s_win[0] = 0;
      count = 1;
      items = d.ntot;
      windows = all;
      __syncthreads();
      return;
    }
    for (int s0 = 0; s0 < d.nsys; s0 += BS) {
      const int s = s0 + t;
      const bool on = s < d.nsys && d.flags[s] != 0;
      const int n = on ? d.geom[s].n : 0;
      const int nw = on ? window_count(d, s) : 0;
      int a = on, b = n, c = nw;
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o),
                  z = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) {
          a += x;
          b += y;
          c += z;
        }
      }
      if (lane == 31) {
        sums[0][w] = a;
        sums[1][w] = b;
        sums[2][w] = c;
      }
      __syncthreads();
      int at = count + a - on, first = items + b - n, win = windows + c - nw;
      for (int q = 0; q < BS / 32; q++) {
        if (q < w) {
          at += sums[0][q];
          first += sums[1][q];
          win += sums[2][q];
        }
        count += sums[0][q];
        items += sums[1][q];
        windows += sums[2][q];
      }
      if (on && at < kMaxWork) {
        s_off[at] = first;
        s_sys[at] = s;
        s_win[at] = win;
      }
      __syncthreads();
    }
    if (count > kMaxWork) {
      count = -1;
      items = d.ntot;
      windows = all;
    }
  }
  // the first window of a flagged system that is its own, and how many it has: a window it
  // shares with a flagged system before it is that one's (a system with a window between
  // two others has none)
  __device__ __forceinline__ static int first_window(const Dev& d, int s) {
    const int p0 = d.geom[s].p0, w = p0 / kOrderWindow;
    for (int i = w * kOrderWindow; i < p0; i += d.geom[d.psys[i]].n + d.geom[d.psys[i]].p0 - i)
      if (d.flags[d.psys[i]] != 0) return w + 1;
    return w;
  }
  __device__ __forceinline__ static int window_count(const Dev& d, int s) {
    const int last = (d.geom[s].p0 + d.geom[s].n - 1) / kOrderWindow;
    return last + 1 - first_window(d, s);
  }
  // the listed system of item g by its first items
  __device__ __forceinline__ int find(const int* first, int g) const {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first[mid] <= g)
        lo = mid;
      else
        hi = mid - 1;
    }
    return lo;
  }
  // the slot of item g and its system; false: nothing to do
  __device__ __forceinline__ bool at(const Dev& d, int g, int* i, int* s) const {
    if (count < 0) {
      *i = g;
      *s = d.psys[g];
      return d.flags[*s] != 0;
    }
    const int q = find(off, g);
    *s = sys[q];
    *i = d.geom[*s].p0 + (g - off[q]);
    return true;
  }
  // the window of window item g
  __device__ __forceinline__ int window(const Dev& d, int g) const {
    if (count < 0 || d.nsys == 1) return g;
    const int q = find(woff, g);
    return first_window(d, sys[q]) + (g - woff[q]);
  }
  // f(slot, system) over the work items
  template <class F>
  __device__ __forceinline__ void each(const Dev& d, F&& f) const {
    for (int g = blockIdx.x * BS + threadIdx.x; g < items; g += gridDim.x * BS) {
      int i, s;
      if (at(d, g, &i, &s)) f(i, s);
    }
  }
};

// set_back_gamma, spherocyl_box.cpp:524-545 (positions; gamma itself is advanced on
// the host), for a system whose table row says so
__device__ __forceinline__ double2 set_back(double2 p, double Lx, double Ly, int* status) {
  if (p.y < 0)
    p.y += Ly;
  else if (p.y > Ly)
    p.y -= Ly;
  p.x = __dadd_rn(p.x, __dmul_rn(Lx / Ly, p.y));  // x + y in a square box (Lx / Ly == 1)
  if (p.x < 0)
    p.x += Lx;
  else
    p.x = wrap_bounded(p.x, -1.0, Lx, Lx, status);  // only the "> Lx" loop applies
  return p;
}

// FP64 position of a mixed record: its cell's centre plus the compensated local position
__device__ __forceinline__ double2 mixed_position(const Dev& d, const StepScalars& ts, int i,
                                                  float4 r, float4 c) {
  const int cp = d.cellp[i];
  return make_double2(fma(widen((float)(cp & 0xffff) + 0.5f), ts.W_p, widen(r.x) + widen(c.x)),
                      fma(widen((float)(cp >> 16) + 0.5f), ts.H_p, widen(r.y) + widen(c.y)));
}

// The column (row) of x in cells of side w, (int)(x / w) as the reference divides: by an
// FP32 quotient unless that is too near a whole number to tell (about one in a thousand;
// the quotient is below 65536 and off by less than 1e-6 of itself).
__device__ __forceinline__ int cell_index(double x, double w) {
  const float q = __fdividef(narrow(x), narrow(w));
  const float f = q - floorf(q), near = 1e-6f * q + 1e-6f;
  if (f > near && f < 1.f - near) return (int)q;
  return (int)(x / w);
}

// find_cells, spherocyl_box.cpp:270-301: wrap, then hash.  moved: the mixed form's state is
// in its records, the FP64 form's shaft vectors are those of its angles (else they are made
// here, as for the angles that wrap).
//
// A displacement-triggered rebuild happens in the reference inside the corrector
// loop, at the first particle i* whose accumulated displacement exceeds pad/2:
// particles up to i* are wrapped after their update, the others before it, and
// the displacement counters of the latter restart from this step's move.  The
// reference wraps with the box length of the loop (before a resize shrinks it).
// Reproducing that matters under resize, where the reference's predictor pass
// uses the pre-resize box for the minimum image and so depends on which image a
// particle sits at.  Forced rebuilds and set-back steps wrap every particle.
template <bool MIXED, int BS>
__device__ __forceinline__ void hash_cells(const Dev& d, const Work<BS>& work,
                                           const StepScalars* __restrict__ tab, int row,
                                           bool moved) {
  work.each(d, [&](int i, int s) {
    const SysGeom& g = d.geom[s];
    const StepScalars& ts = tab[row * d.nsys + s];
    // pure shear rebuilds after the box update (pure_strain_step_2p,
    // src/cuda/2point_dynamics.cu:2255-2282), so it wraps with the new box
    const double Lx = ts.mode == 3 ? ts.Lx_p : ts.Lx_c, Ly = ts.mode == 3 ? ts.Ly_p : ts.Ly_c;
    double2 p;
    double phi;
    if (MIXED && moved) {
      const float4 r = d.rec[i], c = d.mc[i];
      p = mixed_position(d, ts, i, r, c);
      phi = widen(c.z) + widen(c.w);
    } else {
      p = d.xy[i];
      phi = d.ph[i];
    }
    const double phi0 = phi;
    double2 mv = make_double2(0.0, 0.0);
    const int istar = MIXED ? kNoTrigger : d.istar[s];
    if (!MIXED && istar != kNoTrigger && !ts.setback && ts.mode != 3 && d.id[i] > istar) {
      double2 p0 = d.s_xy[i];
      p0.x = wrap_side(p0.x, Lx, d.status);
      p0.y = wrap_side(p0.y, Ly, d.status);
      double ph0 = wrap_angle(d.s_ph[i], d.status);
      p = make_double2(p0.x + d.v0x[i], p0.y + d.v0y[i]);
      phi = ph0 + d.v0p[i];
      if (ts.mode == 1) {
        p.x *= ts.scale;
        p.y *= ts.scale;
      } else if (ts.mode == 2) {
        p.x /= ts.scale;
        p.y /= ts.scale;
      }
      mv = make_double2(p.x - p0.x, p.y - p0.y);
    } else {
      if (ts.setback) p = set_back(p, ts.Lx_p, ts.Ly_p, d.status);
      p.x = wrap_side(p.x, Lx, d.status);
      p.y = wrap_side(p.y, Ly, d.status);
      phi = wrap_angle(phi, d.status);
    }
    d.xy[i] = p;
    d.ph[i] = phi;
    if (!MIXED) {
      d.nxy_t[i] = mv;  // displacement counter to carry into the new slot
      if (!moved || phi != phi0) {
        const double A = d.ra[i].y;
        double sn, cs;
        sincos(phi, &sn, &cs);
        d.nxy[i] = make_double2(A * cs, A * sn);
      }
    }
    // the FP64 form divides as the reference does (find_cells); the mixed form,
    // whose records are relative to whatever cell it is given, takes the FP32
    // quotient (two FP64 divisions per particle dominate this phase on GB300; a
    // particle a rounding error outside its cell is still well inside the 3x3 block
    // its list search covers, whose cells are 0.24 (R + A) wider than the reach)
    int col, rw;
    if (MIXED) {
      col = (int)__fdividef(narrow(p.x), ts.f_Wp);
      rw = (int)__fdividef(narrow(p.y), ts.f_Hp);
    } else {
      col = cell_index(p.x, ts.W_p);
      rw = cell_index(p.y, ts.H_p);
    }
    // a coordinate at (or, after a resize, just past) the box edge stays on the grid
    if (col >= g.cols) col = g.cols - 1;
    if (rw >= g.rows) rw = g.rows - 1;
    if (col < 0) col = 0;
    if (rw < 0) rw = 0;
    const int c = cell_local(g, col, rw);
    d.cell_tmp[i] = g.c0 + c;
    // one atomic per cell, and one per scan chunk, among the converged lanes: the slots
    // arrive in cell order, so neighbouring lanes mostly share both (the order inside a
    // cell is settled by its indices)
    const int lane = threadIdx.x & 31;
    const unsigned act = __activemask();
    const unsigned peers = __match_any_sync(act, g.c0 + c);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&d.cell_fill[g.c0 + c], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    d.rank[i] = base + __popc(peers & ((1u << lane) - 1u));
    const int ch = g.chunk0 + c / kScanChunk;
    const unsigned same = __match_any_sync(act, ch);
    if (lane == __ffs(same) - 1) atomicAdd(&d.chunk_sum[ch], __popc(same));
  });
}

// Cell starts and counts: the block of a scan chunk sums the chunks of its system before
// it, then scans its own cells.  The fill counters are cleared for the next rebuild.
template <int BS>
__device__ __forceinline__ void scan_cells(const Dev& d) {
  constexpr int kPer = kScanChunk / BS;
  __shared__ int sh[BS / 32 + 1];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int ch = blockIdx.x; ch < d.nchunks; ch += gridDim.x) {
    const int s = d.chunk_sys[ch];
    if (d.flags[s] == 0) continue;  // the whole block
    const SysGeom& g = d.geom[s];
    int before = 0;
    for (int k = g.chunk0 + t; k < ch; k += BS) before += d.chunk_sum[k];
    for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    const int c0 = d.chunk_c0[ch], nc = d.chunk_nc[ch];
    int v[kPer], sum = 0;
    for (int q = 0; q < kPer; q++) {
      const int k = t * kPer + q;
      v[q] = k < nc ? d.cell_fill[c0 + k] : 0;
      sum += v[q];
    }
    int x = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();  // sh is free
    if (lane == 0) sh[w] = before;
    __syncthreads();
    int at = g.p0;
    for (int q = 0; q < BS / 32; q++) at += sh[q];
    __syncthreads();
    if (lane == 31) sh[w] = x;
    __syncthreads();
    at += x - sum;
    int all = 0;
    for (int q = 0; q < BS / 32; q++) {
      if (q < w) at += sh[q];
      all += sh[q];
    }
    for (int q = 0; q < kPer; q++) {
      const int k = t * kPer + q;
      if (k < nc) {
        d.cell_start[c0 + k] = at;
        d.cell_count[c0 + k] = v[q];
        d.cell_fill[c0 + k] = 0;
        at += v[q];
      }
    }
    if (t == BS - 1 && ch == g.chunk0 + g.nchunks - 1 && at != g.p0 + g.n)
      atomicOr(d.status, ST_CELL_OVERFLOW);
  }
}

// The indices of each cell's particles side by side, in order of arrival.
template <int BS>
__device__ __forceinline__ void list_indices(const Dev& d, const Work<BS>& work) {
  work.each(d, [&](int i, int) {
    d.perm[d.cell_start[d.cell_tmp[i]] + d.rank[i]] = d.id[i];
  });
  for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < d.nchunks;
       ch += gridDim.x * blockDim.x)
    d.chunk_sum[ch] = 0;
}

// Each particle to its place, in scratch: cells hold their particles in increasing index
// (the reference's cell lists are filled in particle order, spherocyl_box.cpp:277-298).
template <bool MIXED, int BS>
__device__ __forceinline__ void place(const Dev& d, const Work<BS>& work) {
  work.each(d, [&](int src, int) {
    const int c = d.cell_tmp[src], id = d.id[src];
    const int st = d.cell_start[c], n = d.cell_count[c];
    int i = st;
    for (int k = 0; k < n; k++) i += d.perm[st + k] < id;
    d.s_xy[i] = d.xy[src];
    d.s_ph[i] = d.ph[src];
    d.s_ra[i] = d.ra[src];
    d.s_irc[i] = d.irc[src];
    d.s_id[i] = id;
    d.s_cell[i] = c;
    if (!MIXED) {
      // nobody reads the counters themselves here, and the predictor's velocities (s_nxy) are
      // made anew after a rebuild
      d.moved[i] = d.nxy_t[src];
      d.s_nxy[i] = d.nxy[src];
    }
    if (d.fvx) {  // minimiser velocities travel with their particles (predictor copy is dead here)
      d.xy_t[i] = make_double2(d.fvx[src], d.fvy[src]);
      d.ph_t[i] = d.fvp[src];
    }
    if (d.cg0x) {  // and the minimiser's previous forces (stress partials are dead here)
      d.se_part[i] = d.cg0x[src];
      d.se_part[(size_t)d.ntot + i] = d.cg0y[src];
      d.se_part[2 * (size_t)d.ntot + i] = d.cg0p[src];
    }
  });
}

// Back from scratch; f(slot, system, position, angle, (R, A), (I, RC), index, cell) then
// makes the records that the form's passes read (the FP64 form's in the scratch that the same
// slot has just been read from).  records: the state is in them alone
// (the FP64 positions and angles are not read before they are next made).
template <int BS, class F>
__device__ __forceinline__ void put_back(const Dev& d, const Work<BS>& work, bool records, F&& f) {
  work.each(d, [&](int i, int s) {
    const double2 p = d.s_xy[i], ra = d.s_ra[i], irc = d.s_irc[i];
    const double phi = d.s_ph[i];
    const int id = d.s_id[i], c = d.s_cell[i];
    if (!records) {
      d.xy[i] = p;
      d.ph[i] = phi;
    }
    d.ra[i] = ra;
    d.irc[i] = irc;
    d.id[i] = id;
    d.cell[i] = c;
    if (d.fvx) {
      const double2 v = d.xy_t[i];
      d.fvx[i] = v.x;
      d.fvy[i] = v.y;
      d.fvp[i] = d.ph_t[i];
    }
    if (d.cg0x) {
      d.cg0x[i] = d.se_part[i];
      d.cg0y[i] = d.se_part[(size_t)d.ntot + i];
      d.cg0p[i] = d.se_part[2 * (size_t)d.ntot + i];
    }
    f(i, s, p, phi, ra, irc, id, c);
  });
}

// The end of a rebuild: the last block out takes back the flags and counts it, unless a
// barrier timed out on the way.
__device__ __forceinline__ void finish(const Dev& d, GridBarrier& bar) {
  if (!bar.leave()) return;
  for (int s = threadIdx.x; s < d.nsys; s += blockDim.x) {
    d.flags[s] = 0;
    d.istar[s] = kNoTrigger;
  }
  __syncthreads();
  if (threadIdx.x == 0 && !timed_out(d)) {
    *d.any = 0;
    d.status[1] += 1;  // rebuilds executed
  }
}

// The phases up to the records; false when a barrier timed out.
template <bool MIXED, int BS, class F>
__device__ __forceinline__ bool sort_cells(const Dev& d, const Work<BS>& work,
                                           const StepScalars* __restrict__ tab, int row,
                                           bool moved, GridBarrier& bar, F&& records) {
  hash_cells<MIXED>(d, work, tab, row, moved);
  if (!bar.wait(d.status)) return false;
  scan_cells<BS>(d);
  if (!bar.wait(d.status)) return false;
  list_indices(d, work);
  if (!bar.wait(d.status)) return false;
  place<MIXED>(d, work);
  if (!bar.wait(d.status)) return false;
  put_back(d, work, MIXED && moved, records);
  return bar.wait(d.status);
}

}  // namespace rb

// Blocks of the cooperative kernel `fn`: as many as are resident at once (asked of the
// runtime once per device and kernel), and no more than `need`.
template <int TAG>
int coop_blocks(const void* fn, int block, int need) {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  int most = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
  if (most == 0) {
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, 0) != cudaSuccess)
      return 0;
    most = sms * per_sm;
    if (dev < 64) known[dev].store(most, std::memory_order_relaxed);
  }
  return most < need ? most : need;
}

// The candidates of a slot, taken by eight threads: the cells of its 3x3 block (a dimension
// with fewer than three cells once per distinct cell) with the first candidate of each in
// the scan order, in shared memory.
struct Candidates {
  int first[9], off[10];
  unsigned code[9];
};
// the table for column col, row rw, filled by the group `lanes` (sub: which of them);
// returns the number of candidates
__device__ __forceinline__ int list_candidates(const Dev& d, const SysGeom& g, int col, int rw,
                                               Candidates& c, int sub, unsigned lanes) {
  const int ncx = g.cols < 3 ? g.cols : 3, ncy = g.rows < 3 ? g.rows : 3, nc = ncx * ncy;
  __syncwarp(lanes);
  for (int q = sub; q < nc; q += 8) {
    const int a = q / ncx, b = q - a * ncx;
    const int dr = ncy < 3 ? a - rw : a - 1, dc = ncx < 3 ? b - col : b - 1;
    const int r2 = ncy < 3 ? a : wrap_index(rw + dr, g.rows);
    const int c2 = ncx < 3 ? b : wrap_index(col + dc, g.cols);
    const int cc = g.c0 + cell_local(g, c2, r2);
    c.first[q] = d.cell_start[cc];
    c.off[q + 1] = d.cell_count[cc];
    c.code[q] = ((unsigned)(dc + 1) << 28) | ((unsigned)(dr + 1) << 30);
  }
  __syncwarp(lanes);
  if (sub == 0) {
    c.off[0] = 0;
    for (int q = 0; q < nc; q++) c.off[q + 1] += c.off[q];
  }
  __syncwarp(lanes);
  return c.off[nc];
}

// Small handles rebuild in blocks of 128 threads, large ones in blocks of 512 (the fewer
// blocks, the cheaper a barrier); eight threads a slot where there are that many, up to the
// blocks that are resident.  Up to kLaneItems work items, eight threads list a slot's
// neighbours, at most two and a half rounds of them.  A forced rebuild with its call, us,
// with eight and with one thread a slot: FP64 52 and 64 at 8192 particles, 60 and 76 at
// 16384, 64 and 76 at 30000, 67 and 76 at 45000, 77 and 77 at 70000; mixed 52 and 54, 53
// and 64, 64 and 64, 66 and 66, 77 and 66.
constexpr int kSmallRebuild = 4096;
constexpr int kLaneItems = 49152;

}  // namespace sc
