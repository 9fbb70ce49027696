// sc_cells.cu -- the rebuild's flags, stress/energy reductions, the gradient-descent
// update, and the particle arrays' ingest and output.  (The rebuild itself:
// sc_rebuild.cuh.)
// Compiled with -fmad=false: the wrap arithmetic is the reference's IEEE operations.
#include "sc_internal.hpp"
#include "sc_pair.cuh"

namespace sc {

namespace {

constexpr double kRefPi = 3.14159265358979;  // src/cpp/spherocyl_box.cpp:12

__global__ void k_rb_clear(Dev d) {
  if (!rebuild_pending(d)) return;
  for (int s = threadIdx.x; s < d.nsys; s += blockDim.x) {
    d.flags[s] = 0;
    d.istar[s] = kNoTrigger;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *d.any = 0;
    d.status[1] += 1;  // rebuilds executed
  }
}

__global__ void k_force_all(Dev d) {
  for (int s = threadIdx.x; s < d.nsys; s += blockDim.x) d.flags[s] = 2;
  if (threadIdx.x == 0) *d.any = 1;
}

// gradient_relax_step, src/cpp/relaxation_dynamics.cpp:11-31
__global__ void k_gd_update(Dev d, const StepScalars* __restrict__ tab, int row) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ntot) return;
  int s = d.psys[i];
  const SysGeom& g = d.geom[s];
  const double step = tab[row * d.nsys + s].step;
  if (step == 0.0) return;
  double ddx = step * d.fx[i];
  double ddy = step * d.fy[i];
  double ddp = step * d.tau[i] / d.irc[i].x;
  const double2 p0 = d.xy[i];
  const double phi0 = d.ph[i];
  double2 p = make_double2(p0.x + ddx, p0.y + ddy);
  double phi = phi0 + ddp;
  d.xy[i] = p;
  d.ph[i] = phi;
  d.s_xy[i] = p0;
  d.s_ph[i] = phi0;
  d.v0x[i] = ddx;
  d.v0y[i] = ddy;
  d.v0p[i] = ddp;
  double2 m = d.moved[i];
  m.x += ddx;
  m.y += ddy;
  d.moved[i] = m;
  double2 ra = d.ra[i];
  double sn, cs;
  sincos(phi, &sn, &cs);
  const double2 n = make_double2(ra.y * cs, ra.y * sn);
  d.nxy[i] = n;
  d.rec[i] = screen_record(p, n);
  if (!(isfinite(p.x) && isfinite(p.y) && isfinite(phi))) atomicOr(d.status, ST_NAN);
  // the reference tests and rebuilds inside the update loop
  if (m.x > 0.5 * g.pad || m.x < -0.5 * g.pad || m.y > 0.5 * g.pad || m.y < -0.5 * g.pad) {
    if (d.flags[s] == 0) atomicOr(&d.flags[s], 1);
    atomicMin(&d.istar[s], d.id[i]);
    if (*d.any == 0) atomicExch(d.any, 1);
  }
}

// Stress/energy: deterministic two-level reduction of the per-slot contributions, one
// block per chunk and component; the block that finishes a system's last one sums its
// chunks, each thread its strided share in order, then a fixed tree, and stores the record
// (dst, may be null).  The sums run at the FP64 pipe's rate, so the components are on
// different SMs.  Systems with d.skip set keep their sums.  As three kernels (chunks with
// the components in turn, systems, records) it took 15 us at 16384 particles, here 8.
constexpr int kSeThreads = 256;

__global__ void __launch_bounds__(kSeThreads) k_se_reduce(Dev d, double* __restrict__ dst) {
  constexpr int kPer = kSeChunk / kSeThreads, kWarps = kSeThreads / 32;
  __shared__ double sh[5][kWarps];
  __shared__ int last;
  const int ch = blockIdx.x, comp = blockIdx.y, nc = gridDim.y;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int p0 = d.pchunk_p0[ch], np = d.pchunk_np[ch], s = d.pchunk_sys[ch];
  if (d.skip && d.skip[s]) return;
  double v[kPer];
  for (int q = 0; q < kPer; q++) {
    const int k = t + q * kSeThreads;
    v[q] = k < np ? d.se_part[(size_t)comp * d.ntot + p0 + k] : 0.0;
  }
  double x = 0.0;
  for (int q = 0; q < kPer; q++) x += v[q];
  for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (lane == 0) sh[0][w] = x;
  __syncthreads();
  const SysGeom& g = d.geom[s];
  const int nch = pchunk_count(g);
  if (w == 0) {
    x = lane < kWarps ? sh[0][lane] : 0.0;
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) {
      d.se_chunk[(size_t)comp * d.npchunks + ch] = x;
      __threadfence();
      last = atomicAdd(&d.se_done[s], 1) == nch * nc - 1;
      __threadfence();
    }
  }
  __syncthreads();
  if (!last) return;
  for (int c = 0; c < nc; c++) {
    x = 0.0;
    for (int k = t; k < nch; k += kSeThreads)
      x += __ldcg(&d.se_chunk[(size_t)c * d.npchunks + g.pch0 + k]);
    if (w * 32 < nch)
      for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[c][w] = x;
  }
  __syncthreads();
  if (t < nc) {
    x = 0.0;
    for (int k = 0; k < kWarps; k++) x += sh[t][k];
    d.se_sys[(size_t)t * d.nsys + s] = x;
    if (dst) dst[5 * s + t] = x;
  }
  if (t == 0) d.se_done[s] = 0;
}

// set_particle's wrap loop (src/cpp/spherocyl_box.cpp:204-215) for the input state:
// the reference's repeated subtraction, finished by a floor for a value more than
// 64 periods out (where the loop would take that long; not an error here).
__device__ __forceinline__ double wrap_input(double v, double lo, double hi, double period) {
  int it = 0;
  while (v > hi && it < 64) {
    v -= period;
    it++;
  }
  while (v < lo && it < 64) {
    v += period;
    it++;
  }
  if (it >= 64) v -= period * floor((v - lo) / period);
  return v;
}

// Per-particle state of a new handle (set_particle, src/cpp/spherocyl_box.cpp:188-221):
// the wrapped position and angle, (R, A), the moment of inertia I and the rotation
// coefficient RC in the reference's operation order, the particle index and system
// of each slot.  x..A are the caller's arrays: host memory that the GPU reads in
// place where it can address pageable memory, else a device copy.  sys_p0 holds the
// first slot of each system and ntot at [nsys]; sys_L the (Lx, Ly) pairs.
__global__ void k_ingest(Dev d, const double* __restrict__ x, const double* __restrict__ y,
                         const double* __restrict__ phi, const double* __restrict__ R,
                         const double* __restrict__ A, const int* __restrict__ sys_p0,
                         const double* __restrict__ sys_L, int* __restrict__ psys) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.ntot; i += stride) {
    int lo = 0, hi = d.nsys - 1;  // the system whose slot range holds i
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sys_p0[mid] <= i)
        lo = mid;
      else
        hi = mid - 1;
    }
    const int s = lo;
    const double Lx = sys_L[2 * s], Ly = sys_L[2 * s + 1];
    const double r = R[i], a = A[i];
    const double al = a / r;
    const double C = (3 * kRefPi + 24 * al + 6 * kRefPi * al * al + 8 * al * al * al);
    const double area = r * (kRefPi * r + 4 * a);
    d.irc[i] = make_double2(r * r * r * r * C / (6 * area),
                            (8 * al + 6 * kRefPi * al * al + 8 * al * al * al) / C);
    d.ra[i] = make_double2(r, a);
    d.xy[i] = make_double2(wrap_input(x[i], 0.0, Lx, Lx), wrap_input(y[i], 0.0, Ly, Ly));
    d.ph[i] = wrap_input(phi[i], -kRefPi, kRefPi, 2 * kRefPi);
    d.id[i] = i - sys_p0[s];
    psys[i] = s;
  }
}

// Output in the caller's particle order: slot i holds particle p0 + id[i] of its
// system, so each value goes to out[k * ntot + p0 + id[i]].
__global__ void k_unsort_state(Dev d, double* __restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ntot) return;
  const size_t o = (size_t)d.geom[d.psys[i]].p0 + d.id[i];
  const double2 p = d.xy[i];
  out[o] = p.x;
  out[(size_t)d.ntot + o] = p.y;
  out[(size_t)2 * d.ntot + o] = d.ph[i];
}

__global__ void k_unsort_forces(Dev d, double* __restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.ntot) return;
  const size_t o = (size_t)d.geom[d.psys[i]].p0 + d.id[i];
  out[o] = d.fx[i];
  out[(size_t)d.ntot + o] = d.fy[i];
  out[(size_t)2 * d.ntot + o] = d.tau[i];
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

int launch_rebuild(const Dev& d, bool mixed, const StepScalars* tab, int row, bool moved,
                   cudaStream_t st) {
  return mixed ? launch_rebuild_mixed(d, tab, row, moved, st)
               : launch_rebuild_fp64(d, tab, row, moved, st);
}

void launch_force_rebuild_all(const Dev& d, cudaStream_t st) { k_force_all<<<1, 256, 0, st>>>(d); }

void launch_clear_flags(const Dev& d, cudaStream_t st) { k_rb_clear<<<1, 256, 0, st>>>(d); }

void launch_gd_update(const Dev& d, bool mixed, const StepScalars* tab, int row, cudaStream_t st) {
  (void)mixed;  // the CPU-compatible gradient descent is a plain FP64 protocol
  k_gd_update<<<nblk(d.ntot, 256), 256, 0, st>>>(d, tab, row);
}

void launch_ingest(const Dev& d, const double* x, const double* y, const double* phi,
                   const double* R, const double* A, const int* sys_p0, const double* sys_L,
                   int* psys, cudaStream_t st) {
  const int blocks = nblk(d.ntot, 256) < 152 * 8 ? nblk(d.ntot, 256) : 152 * 8;
  k_ingest<<<blocks, 256, 0, st>>>(d, x, y, phi, R, A, sys_p0, sys_L, psys);
}

void launch_unsort_state(const Dev& d, double* out, cudaStream_t st) {
  k_unsort_state<<<nblk(d.ntot, 256), 256, 0, st>>>(d, out);
}

void launch_unsort_forces(const Dev& d, double* out, cudaStream_t st) {
  k_unsort_forces<<<nblk(d.ntot, 256), 256, 0, st>>>(d, out);
}

void launch_se_reduce(const Dev& d, double* dst, bool energy, cudaStream_t st) {
  k_se_reduce<<<dim3(d.npchunks, energy ? 1 : 5), kSeThreads, 0, st>>>(d, dst);
}

}  // namespace sc
