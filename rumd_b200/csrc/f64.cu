// Double-precision engine: the per-step path of RUMD (neighbour list, LJ pair
// forces, Nose-Hoover leap-frog, energy/virial/kinetic sums) computed in FP64
// throughout.  It is the analogue of RUMD rebuilt after changeToDouble.sh
// (changeToDouble.sh:1-189, which turns every float of the sources into a
// double) and serves as the accuracy oracle on the GPU for the FP32 engine:
// the same potential and integrator, evaluated without FP32 rounding.
//
// Algorithm, step by step (the order of Simulation.Run, Simulation.py:585-610,
// with IntegratorNVT::Integrate, IntegratorNVT.cu:64-92, 364-437):
//   1. every reset_interval steps: centre-of-mass velocity removed
//      (IntegratorNVT::SetMomentumToZero, IntegratorNVT.cu:176-183);
//   2. if a particle moved more than skin/2 since the last build: cell list
//      and full neighbour list within (rc_ij + skin)^2
//      (NeighborList::UpdateNBlist, NeighborList.cu:583-690);
//   3. pair forces, u_i (halved) and w_i = sum d^2 s (fij, PairPotential.h:1198-1244;
//      Pot_IPL_12_6::ComputeInteraction, PairPotential.h:161-168);
//   4. Nose-Hoover leap-frog with PBC wrap and image count, FP64 kinetic sums
//      (integrateNVTAlgorithm, IntegratorNVT.cu:364-418);
//   5. thermostat update xi += dt * omega^2 * min(KE2/(DOF T) - 1, 10)
//      (updateNVTThermostatState, IntegratorNVT.cu:426-437).
// The pair constants: rc, A12 and A6 come from the RUMD parameter table; the
// shifted-force / shifted-potential constants s(rc) rc and u(rc) are
// recomputed here in FP64 from them, as the double build's CopyParamsToGPU
// (PairPotential.cu:82-125) would.
//
// Layout: at every list build the particles are sorted by (cell, place), so
// that a warp's neighbours share cache lines; uid holds each place's particle
// in the caller's order, which get and set use.  Cells are at least
// rc_max + skin wide (27-cell stencil); boxes with fewer than three cells
// along a side use all pairs.  Lists and sums have a fixed order: runs are
// deterministic.  All sums are FP64 with a fixed tree (block partials added in
// block order).
//
// A step is three launches: the list build (one cooperative kernel that
// returns at once unless a build is due), the forces, and the integration
// with the step's totals.  What bounds a step is the latency of dependent
// FP64 arithmetic and of the neighbour gathers, so 4 to 32 lanes share a
// particle, the more the fewer particles there are.  At LJ N=32000 a step takes
// 49 to 51 us; one thread per particle, in the caller's order, with ten launches
// a step took 121.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/rumd_b200.h"

namespace b2md_internal {
void set_last_error(const char* msg);
}

namespace {

constexpr int kB = 256;        // threads per block
constexpr int kMaxT = 16;      // particle types
constexpr int kNPartF64 = 4;   // per-block partials of the momentum: P, M
constexpr unsigned kPolls = 1u << 22;  // grid-barrier polls before a wait gives up

struct F64Pair {
  double rc, rc2, a12, a6, cs, cu, nb2;  // cs = s(rc) rc, cu = u(rc), nb2 = (rc + skin)^2
};

struct F64Dev {  // device-resident scalars
  double xi, P[3], M, pe, W, ke_t, ke2;
  long long rebuilds, steps;
  int need, overflow;
  unsigned arrive, gen;  // grid barrier of the list build
  unsigned done;         // blocks of the list build / integration finished
  int err;               // a grid-barrier wait gave up
};

struct F64Args {
  int n, ntypes, cutoff, max_nbrs, ncell, allpairs, thermo, fblocks;
  int nc[3];
  double L[3], invL[3], ilim[3], dt, skin2_4, T, omega2, dof;
  double4 *r, *v, *f, *last_r;
  int4 *im, *im2;          // (im2, uid2: the sort's copies; f and last_r serve for r and v)
  unsigned *uid, *uid2;    // the caller's particle of each place
  int *cell, *rank, *order, *cnt, *cstart, *ctot;
  unsigned *nn, *nbl;      // entry k of place i at nbl[((k / 4) n + i) 4 + k % 4]
  double *part, *part_f;   // per-block sums of the integration (and momentum); of the forces
  F64Dev* st;
  const F64Pair* par;
};

// d - L rint(d / L); adding and subtracting 1.5 2^52 rounds |x| < 2^51 to an
// integer, ties to even, in two additions.
__device__ __forceinline__ double mi64(double d, double L, double iL) {
  const double M = 6755399441055744.0;
  return d - L * __dsub_rn(__dadd_rn(d * iL, M), M);
}

__device__ __forceinline__ int type_of(const double4& r) { return (int)r.w; }

// Block sum of K doubles per thread (warp butterfly, then warps in order);
// the result is valid in s_out after the call.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double* s_warp, double* s_out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) s_warp[wid * K + k] = x;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += s_warp[w * K + threadIdx.x];
    s_out[threadIdx.x] = s;
  }
  __syncthreads();
}

// Sums the K columns of `nblocks` rows of partials (row stride K) in a fixed
// order: thread t adds rows t, t+kB, ...; then the block adds the threads in
// order.  Read past L1: other blocks of the same launch may have written them.
template <int K>
__device__ __forceinline__ void sum_partials(const double* part, int nblocks, double* s_warp, double* s_out) {
  double v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] += __ldcg(part + (size_t)b * K + k);
  block_sum<K>(v, s_warp, s_out);
}

// ---- 1. momentum reset ----
__global__ void __launch_bounds__(kB) k64_momentum_part(F64Args a) {
  __shared__ double s_warp[(kB / 32) * 4], s_out[4];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < a.n) {
    const double4 vi = a.v[i];
    const double m = 1.0 / vi.w;
    v[0] = m * vi.x; v[1] = m * vi.y; v[2] = m * vi.z; v[3] = m;
  }
  block_sum<4>(v, s_warp, s_out);
  if (threadIdx.x < 4) a.part[(size_t)blockIdx.x * kNPartF64 + threadIdx.x] = s_out[threadIdx.x];
}

__global__ void __launch_bounds__(kB) k64_momentum_total(F64Args a, int nblocks) {
  __shared__ double s_warp[(kB / 32) * 4], s_out[4];
  sum_partials<4>(a.part, nblocks, s_warp, s_out);
  if (threadIdx.x == 0) {
    a.st->P[0] = s_out[0]; a.st->P[1] = s_out[1]; a.st->P[2] = s_out[2]; a.st->M = s_out[3];
  }
}

__global__ void __launch_bounds__(kB) k64_momentum_apply(F64Args a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n || !(a.st->M > 0.0)) return;
  const double iM = 1.0 / a.st->M;
  double4 v = a.v[i];
  v.x -= a.st->P[0] * iM; v.y -= a.st->P[1] * iM; v.z -= a.st->P[2] * iM;
  a.v[i] = v;
}

// ---- 2. neighbour list (each kernel returns at once unless a build is due) ----
__device__ __forceinline__ int cell_of(const F64Args& a, const double4& r) {
  int c[3];
  const double x[3] = {r.x, r.y, r.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int k = (int)floor((x[d] * a.invL[d] + 0.5) * a.nc[d]);
    c[d] = k < 0 ? 0 : (k >= a.nc[d] ? a.nc[d] - 1 : k);
  }
  return c[0] + a.nc[0] * (c[1] + a.nc[1] * c[2]);
}

// Grid barrier of the list build (every block resident: cooperative launch);
// false, in every thread, when the wait gave up.
__device__ bool grid_barrier(F64Dev* st) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_ok = 1;
    volatile unsigned* gen = &st->gen;
    const unsigned g = *gen;
    __threadfence();
    if (atomicAdd(&st->arrive, 1u) == gridDim.x - 1) {
      st->arrive = 0u;
      __threadfence();
      *gen = g + 1u;
    } else {
      unsigned it = 0;
      while (*gen == g && it < kPolls) {
        __nanosleep(32);
        ++it;
      }
      if (it >= kPolls) {
        atomicExch(&st->err, 1);
        s_ok = 0;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return s_ok != 0;
}

// Appends the accepted candidates [b, e) (places) of particle i to its list;
// the particle's 8 lanes test 8 consecutive ones a round, in order.  All lanes
// of the warp call it (others with an empty range).
__device__ __forceinline__ unsigned list_run(const F64Args& a, int i, const double4& ri, const F64Pair* row, int b,
                                             int e, unsigned count) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u, l8 = lane & 7u, shift = lane & 24u;
  const int rounds = __reduce_max_sync(FULL, e > b ? (e - b + 7) >> 3 : 0);
  for (int k = 0; k < rounds; ++k) {
    const int j = b + 8 * k + (int)l8;
    bool in = false;
    if (j < e && j != i) {
      const double4 rj = a.r[j];
      const double dx = mi64(ri.x - rj.x, a.L[0], a.invL[0]);
      const double dy = mi64(ri.y - rj.y, a.L[1], a.invL[1]);
      const double dz = mi64(ri.z - rj.z, a.L[2], a.invL[2]);
      in = dx * dx + dy * dy + dz * dz < row[type_of(rj)].nb2;
    }
    const unsigned m = (__ballot_sync(FULL, in) >> shift) & 0xffu;
    if (in) {
      const unsigned pos = count + __popc(m & ((1u << l8) - 1u));
      if (pos < (unsigned)a.max_nbrs) a.nbl[((size_t)(pos >> 2) * a.n + i) * 4 + (pos & 3u)] = (unsigned)j;
    }
    count += __popc(m);
  }
  return count;
}

// The list build: one cooperative launch whose blocks meet between the phases
// of the sort; it returns at once unless a build is due.
__global__ void __launch_bounds__(kB) k64_rebuild(F64Args a) {
  F64Dev* st = a.st;
  if (!st->need || st->err) return;
  __shared__ int s_w[kB / 32 + 1];
  const int tid = threadIdx.x, gid = blockIdx.x * blockDim.x + tid, gsz = gridDim.x * blockDim.x;
  const int lane = tid & 31, wid = tid >> 5;
  for (int c = gid; c < a.ncell; c += gsz) a.cnt[c] = 0;
  if (!grid_barrier(st)) return;  // (also: every block has seen that a build is due)
  if (!a.allpairs) {
    for (int i = gid; i < a.n; i += gsz) {
      const int c = cell_of(a, a.r[i]);
      a.cell[i] = c;
      a.rank[i] = atomicAdd(&a.cnt[c], 1);
    }
    if (!grid_barrier(st)) return;
    // exclusive scan of the counts: block b owns a run of cells; first the
    // runs' totals, then every block adds the totals before its own
    const int run = (a.ncell + gridDim.x - 1) / gridDim.x;
    const int c0 = min(a.ncell, (int)blockIdx.x * run), c1 = min(a.ncell, c0 + run);
    auto block_total = [&](int x) -> int {
      x = __reduce_add_sync(0xffffffffu, x);
      __syncthreads();
      if (lane == 0) s_w[wid] = x;
      __syncthreads();
      int t = 0;
      for (int w = 0; w < kB / 32; ++w) t += s_w[w];
      return t;
    };
    {
      int x = 0;
      for (int c = c0 + tid; c < c1; c += kB) x += __ldcg(a.cnt + c);
      x = block_total(x);
      if (tid == 0) a.ctot[blockIdx.x] = x;
    }
    if (!grid_barrier(st)) return;
    {
      int x = 0;
      for (int b = tid; b < (int)blockIdx.x; b += kB) x += __ldcg(a.ctot + b);
      int first = block_total(x);
      for (int cb = c0; cb < c1; cb += kB) {
        const int c = cb + tid;
        const int m = c < c1 ? __ldcg(a.cnt + c) : 0;
        int incl = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        __syncthreads();
        if (lane == 31) s_w[wid] = incl;
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < kB / 32; ++w) {
          if (w < wid) before += s_w[w];
          all += s_w[w];
        }
        if (c < c1) a.cstart[c] = first + before + incl - m;
        first += all;
      }
    }
    if (!grid_barrier(st)) return;
    for (int i = gid; i < a.n; i += gsz) a.order[__ldcg(a.cstart + a.cell[i]) + a.rank[i]] = i;
    if (!grid_barrier(st)) return;
    // each bucket by place (members counted against each other), state copied
    // in that order
    for (int s = gid; s < a.n; s += gsz) {
      const int i = __ldcg(a.order + s), c = __ldcg(a.cell + i), b = __ldcg(a.cstart + c), m = __ldcg(a.cnt + c);
      int place = b;
      for (int k = 0; k < m; ++k) place += __ldcg(a.order + b + k) < i;
      a.f[place] = a.r[i];
      a.last_r[place] = a.v[i];
      a.im2[place] = a.im[i];
      a.uid2[place] = a.uid[i];
    }
    if (!grid_barrier(st)) return;
    for (int i = gid; i < a.n; i += gsz) {
      const double4 r = a.f[i];
      a.v[i] = a.last_r[i];
      a.r[i] = r;
      a.last_r[i] = r;
      a.im[i] = a.im2[i];
      a.uid[i] = a.uid2[i];
    }
    if (!grid_barrier(st)) return;
  } else {
    for (int i = gid; i < a.n; i += gsz) a.last_r[i] = a.r[i];
  }
  // the lists: 8 lanes per particle, four particles per warp
  const int nwarps = gsz >> 5;
  for (int i0 = (gid >> 5) * 4; i0 < a.n; i0 += nwarps * 4) {
    const int i = i0 + (lane >> 3);
    const bool valid = i < a.n;
    const double4 ri = a.r[valid ? i : 0];
    const F64Pair* row = a.par + type_of(ri) * a.ntypes;
    unsigned count = 0;
    if (a.allpairs) {
      count = list_run(a, i, ri, row, 0, valid ? a.n : 0, count);
    } else {
      const int c = cell_of(a, ri);
      const int cx = c % a.nc[0], cy = (c / a.nc[0]) % a.nc[1], cz = c / (a.nc[0] * a.nc[1]);
      for (int k = 0; k < 9; ++k) {
        const int oy = (cy + k % 3 - 1 + a.nc[1]) % a.nc[1], oz = (cz + k / 3 - 1 + a.nc[2]) % a.nc[2];
        const int base = a.nc[0] * (oy + a.nc[1] * oz);
        // x cells cx-1 .. cx+1: one run of places, or two when the row wraps
        const int lo = max(cx - 1, 0), hi = min(cx + 1, a.nc[0] - 1);
        const int b = a.cstart[base + lo], e = a.cstart[base + hi] + a.cnt[base + hi];
        count = list_run(a, i, ri, row, b, valid ? e : b, count);
        const int o = cx == 0 ? base + a.nc[0] - 1 : base;  // the wrapped cell
        const bool two = valid && (cx == 0 || cx == a.nc[0] - 1);
        count = list_run(a, i, ri, row, two ? a.cstart[o] : 0, two ? a.cstart[o] + a.cnt[o] : 0, count);
      }
    }
    if (valid && (lane & 7) == 0) {
      a.nn[i] = min(count, (unsigned)a.max_nbrs);
      if ((int)count > a.max_nbrs) st->overflow = 1;
    }
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&st->done, 1u) == gridDim.x - 1) {
      st->done = 0u;
      st->need = 0;
      st->rebuilds += 1;
    }
  }
}

// ---- 3. pair forces: TP lanes per particle, lane t takes entries t, t + TP, ... ----
template <int TP>
__global__ void __launch_bounds__(kB) k64_forces(F64Args a) {
  __shared__ double s_warp[(kB / 32) * 2], s_out[2];
  constexpr unsigned FULL = 0xffffffffu;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / TP, t = threadIdx.x % TP;
  const bool valid = i < a.n;
  const double4 ri = a.r[valid ? i : 0];
  const F64Pair* row = a.par + type_of(ri) * a.ntypes;
  // a particle farther than rc_max + 2 skin from both faces of a dimension has
  // its listed neighbours at their minimum image in it, when these are inside
  // the box (ilim < 0 until a state given with other coordinates has been
  // wrapped by a step)
  const bool wx = __any_sync(FULL, !(fabs(ri.x) < a.ilim[0])), wy = __any_sync(FULL, !(fabs(ri.y) < a.ilim[1])),
             wz = __any_sync(FULL, !(fabs(ri.z) < a.ilim[2]));
  double fx = 0.0, fy = 0.0, fz = 0.0, u = 0.0, w = 0.0;
  const unsigned nn = valid ? a.nn[i] : 0u;
  const unsigned* list = a.nbl + (size_t)i * 4;
  auto entry = [&](unsigned k) { return k < nn ? __ldg(list + (size_t)(k >> 2) * a.n * 4 + (k & 3u)) : 0u; };
  unsigned j = entry(t);
  for (unsigned k = t; k < nn; k += TP) {
    const double4 rj = a.r[j];
    j = entry(k + TP);
    double dx = ri.x - rj.x, dy = ri.y - rj.y, dz = ri.z - rj.z;
    if (wx) dx = mi64(dx, a.L[0], a.invL[0]);
    if (wy) dy = mi64(dy, a.L[1], a.invL[1]);
    if (wz) dz = mi64(dz, a.L[2], a.invL[2]);
    const double d2 = dx * dx + dy * dy + dz * dz;
    const F64Pair& p = row[type_of(rj)];
    if (d2 < p.rc2) {
      const double i2 = 1.0 / d2, i6 = i2 * i2 * i2, q = p.a12 * i6;
      double s = i6 * i2 * (12.0 * q + 6.0 * p.a6);
      double uu = i6 * (q + p.a6);
      if (a.cutoff == B2MD_CUTOFF_SF) {
        const double y = rsqrt(d2);
        s -= p.cs * y;
        uu += p.cs * (d2 * y - p.rc) - p.cu;
      } else if (a.cutoff == B2MD_CUTOFF_SP) {
        uu -= p.cu;
      }
      fx += dx * s; fy += dy * s; fz += dz * s;
      u += uu; w += d2 * s;
    }
  }
#pragma unroll
  for (int o = TP / 2; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(FULL, fx, o);
    fy += __shfl_xor_sync(FULL, fy, o);
    fz += __shfl_xor_sync(FULL, fz, o);
    u += __shfl_xor_sync(FULL, u, o);
    w += __shfl_xor_sync(FULL, w, o);
  }
  double acc[2] = {0.0, 0.0};
  if (valid && t == 0) {
    a.f[i] = make_double4(fx, fy, fz, 0.5 * u);
    acc[0] = 0.5 * u;
    acc[1] = w;
  }
  block_sum<2>(acc, s_warp, s_out);
  if (threadIdx.x < 2) a.part_f[(size_t)blockIdx.x * 2 + threadIdx.x] = s_out[threadIdx.x];
}

// ---- 4. Nose-Hoover leap-frog; the last block adds up the step: totals,
// thermostat, energy log ----
__global__ void __launch_bounds__(kB) k64_integrate(F64Args a, double* elog) {
  __shared__ double s_warp[(kB / 32) * 2], s_out[2], s_for[2];
  __shared__ int s_last;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[2] = {0.0, 0.0};
  if (i < a.n) {
    const double factor = a.thermo ? 0.5 * a.st->xi * a.dt : 0.0;
    const double plus = 1.0 / (1.0 + factor), minus = 1.0 - factor;
    const double4 f = a.f[i];
    double4 v = a.v[i], r = a.r[i];
    int4 im = a.im[i];
    const double vb = v.x * v.x + v.y * v.y + v.z * v.z;
    v.x = plus * (minus * v.x + v.w * f.x * a.dt);
    v.y = plus * (minus * v.y + v.w * f.y * a.dt);
    v.z = plus * (minus * v.z + v.w * f.z * a.dt);
    r.x += v.x * a.dt; r.y += v.y * a.dt; r.z += v.z * a.dt;
    const double kx = rint(r.x * a.invL[0]), ky = rint(r.y * a.invL[1]), kz = rint(r.z * a.invL[2]);
    r.x -= a.L[0] * kx; r.y -= a.L[1] * ky; r.z -= a.L[2] * kz;
    im.x += (int)kx; im.y += (int)ky; im.z += (int)kz;
    a.v[i] = v; a.r[i] = r; a.im[i] = im;
    const double vf = v.x * v.x + v.y * v.y + v.z * v.z;
    const double m = 1.0 / v.w;
    acc[0] = 0.25 * m * (vb + vf);
    acc[1] = m * vf;
    const double4 lr = a.last_r[i];
    const double ex = mi64(r.x - lr.x, a.L[0], a.invL[0]), ey = mi64(r.y - lr.y, a.L[1], a.invL[1]);
    const double ez = mi64(r.z - lr.z, a.L[2], a.invL[2]);
    if (ex * ex + ey * ey + ez * ez > a.skin2_4) a.st->need = 1;
  }
  block_sum<2>(acc, s_warp, s_out);
  if (threadIdx.x < 2) a.part[(size_t)blockIdx.x * 2 + threadIdx.x] = s_out[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.st->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  sum_partials<2>(a.part_f, a.fblocks, s_warp, s_for);
  sum_partials<2>(a.part, gridDim.x, s_warp, s_out);
  if (threadIdx.x != 0) return;
  F64Dev* S = a.st;
  S->done = 0u;
  S->pe = s_for[0];
  S->W = s_for[1] / 6.0;
  S->ke_t = s_out[0];
  S->ke2 = s_out[1];
  if (a.thermo) {
    double dev = s_out[1] / (a.dof * a.T) - 1.0;
    if (dev > 10.0) dev = 10.0;
    S->xi += a.dt * a.omega2 * dev;
  }
  S->steps += 1;
  if (elog) {
    elog[0] = S->pe;
    elog[1] = S->W;
    elog[2] = S->ke_t;
    elog[3] = S->xi;
  }
}

// ---- 5. the force evaluation's totals alone (b2md_f64_calc_f) ----
__global__ void __launch_bounds__(kB) k64_finish(F64Args a) {
  __shared__ double s_warp[(kB / 32) * 2], s_out[2];
  sum_partials<2>(a.part_f, a.fblocks, s_warp, s_out);
  if (threadIdx.x != 0) return;
  a.st->pe = s_out[0];
  a.st->W = s_out[1] / 6.0;
}

// A field in the caller's order in the list build's scratch arrays (idle
// between builds): 32-byte vectors, or images as 3 ints.
__global__ void __launch_bounds__(kB) k64_unsort(F64Args a, const double4* src, double4* out, int* images) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const size_t o = a.uid[i];
  if (src) {
    out[o] = src[i];
  } else {
    const int4 im = a.im[i];
    images[3 * o] = im.x; images[3 * o + 1] = im.y; images[3 * o + 2] = im.z;
  }
}

__global__ void __launch_bounds__(kB) k64_iota(unsigned* ids, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ids[i] = (unsigned)i;
}

}  // namespace

struct b2md_f64 {
  int device = 0;
  cudaStream_t stream = nullptr;
  F64Args a = {};
  F64Dev* st = nullptr;
  F64Pair* par = nullptr;
  int reset_interval = 100;
  bool have_state = false;
  double ilim[3];       // k64_forces' limits for coordinates inside the box
  double inside[3];     // largest |coordinate| that counts as inside: half a box and half a skin, by which a
                        // listed neighbour still is at its minimum image (see k64_forces)
  int tp = 4;           // lanes per particle of the force kernel
  int rb_grid = 1;      // blocks of the list build, all resident at once
  double* elog = nullptr;  // energies of a run, kept for the next
  long long elog_cap = 0;
  std::vector<void*> bufs;
  double4* scratch = nullptr;  // the list build's per-particle scratch: im2, uid2, cell, rank, order
};

namespace {

std::string f64_errmsg;

// Page-locked staging of the read-backs, a piece for each that is under way
// (page-locking one costs milliseconds, which every engine would pay for its
// first read-back): taken from the free pieces of the process, allocated when
// there is none, and given back; freed with the last engine.  The lock is held
// for the taking and giving only, so that engines on several threads or GPUs
// read back at the same time.
constexpr size_t kStageBytes = (size_t)1 << 20;
constexpr int kMaxFree = 8;  // free pieces kept
std::mutex g_stage_mu;
void* g_free[kMaxFree];
int g_nfree = 0, g_engines = 0;

void* take_stage() {
  {
    std::lock_guard<std::mutex> lock(g_stage_mu);
    if (g_nfree > 0) return g_free[--g_nfree];
  }
  void* p = nullptr;
  if (cudaHostAlloc(&p, kStageBytes, cudaHostAllocPortable) == cudaSuccess) return p;
  (void)cudaGetLastError();
  return nullptr;
}

void give_stage(void* p) {
  {
    std::lock_guard<std::mutex> lock(g_stage_mu);
    if (g_nfree < kMaxFree) {
      g_free[g_nfree++] = p;
      return;
    }
  }
  cudaFreeHost(p);
}

int f64_fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  f64_errmsg = buf;
  b2md_internal::set_last_error(f64_errmsg.c_str());
  return code;
}

#define F64_CK(x)                                                                       \
  do {                                                                                  \
    cudaError_t err_ = (x);                                                             \
    if (err_ != cudaSuccess)                                                            \
      return f64_fail(B2MD_ERR_CUDA, "%s: %s", #x, cudaGetErrorString(err_));           \
  } while (0)

template <class T>
int f64_alloc(b2md_f64* h, T*& p, size_t count) {
  void* q = nullptr;
  cudaError_t err = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
  if (err != cudaSuccess) return f64_fail(B2MD_ERR_NOMEM, "b2md_f64: cudaMalloc of %zu bytes failed: %s",
                                          count * sizeof(T), cudaGetErrorString(err));
  h->bufs.push_back(q);
  p = static_cast<T*>(q);
  return B2MD_OK;
}

int nblocks(const b2md_f64* h) { return (h->a.n + kB - 1) / kB; }

// step 2 + 3: list (when due) and forces
int launch_forces(b2md_f64* h) {
  F64Args a = h->a;
  cudaStream_t s = h->stream;
  void* args[] = {&a};
  F64_CK(cudaLaunchCooperativeKernel((const void*)k64_rebuild, dim3(h->rb_grid), dim3(kB), args, 0, s));
  switch (h->tp) {
    case 32: k64_forces<32><<<a.fblocks, kB, 0, s>>>(a); break;
    case 8: k64_forces<8><<<a.fblocks, kB, 0, s>>>(a); break;
    default: k64_forces<4><<<a.fblocks, kB, 0, s>>>(a); break;
  }
  F64_CK(cudaGetLastError());
  return B2MD_OK;
}

int read_dev(b2md_f64* h, F64Dev* out) {
  F64_CK(cudaMemcpyAsync(out, h->st, sizeof(F64Dev), cudaMemcpyDeviceToHost, h->stream));
  F64_CK(cudaStreamSynchronize(h->stream));
  return B2MD_OK;
}

int check_overflow(b2md_f64* h) {
  F64Dev d;
  int rc = read_dev(h, &d);
  if (rc) return rc;
  if (d.err) return f64_fail(B2MD_ERR_CUDA, "b2md_f64: a grid-barrier wait of the list build gave up");
  if (d.overflow)
    return f64_fail(B2MD_ERR_OVERFLOW, "b2md_f64: a particle has more than %d neighbours within rc + skin; "
                                       "the run is invalid (create the engine with a larger max_nbrs)",
                    h->a.max_nbrs);
  return B2MD_OK;
}

}  // namespace

extern "C" {

int b2md_f64_create(int device, int n, int ntypes, const double* box3, const float* params, int cutoff_method,
                    double skin, int max_nbrs, b2md_f64** out) {
  if (!out || !box3 || !params) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: null argument");
  *out = nullptr;
  if (n < 2) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: n must be >= 2");
  if (ntypes < 1 || ntypes > kMaxT) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: ntypes must be 1..%d", kMaxT);
  if (cutoff_method < 0 || cutoff_method > 2)
    return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: cut-off method must be NS, SP or SF");
  if (!(skin >= 0.0)) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: skin must be >= 0");
  for (int d = 0; d < 3; ++d)
    if (!(box3[d] > 0.0)) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: box lengths must be positive");
  // pair constants in FP64 from rc = p0, A12 = p1, A6 = p2 of the RUMD table
  std::vector<F64Pair> pars((size_t)ntypes * ntypes);
  double rc_max = 0.0;
  for (int k = 0; k < ntypes * ntypes; ++k) {
    const float* p = params + (size_t)k * 12;
    F64Pair& q = pars[k];
    q.rc = p[0]; q.a12 = p[1]; q.a6 = p[2];
    if (!(q.rc > 0.0)) return f64_fail(B2MD_ERR_ARG, "b2md_f64_create: pair %d has no positive cut-off", k);
    q.rc2 = q.rc * q.rc;
    const double i2 = 1.0 / q.rc2, i6 = i2 * i2 * i2;
    q.cu = i6 * (q.a12 * i6 + q.a6);
    q.cs = i6 * i2 * (12.0 * q.a12 * i6 + 6.0 * q.a6) * q.rc;
    q.nb2 = (q.rc + skin) * (q.rc + skin);
    rc_max = std::max(rc_max, q.rc);
  }
  b2md_f64* h = new b2md_f64();
  {
    std::lock_guard<std::mutex> lock(g_stage_mu);
    ++g_engines;
  }
  h->device = device;
  F64Args& a = h->a;
  a.n = n; a.ntypes = ntypes; a.cutoff = cutoff_method;
  a.allpairs = 0;
  a.ncell = 1;
  for (int d = 0; d < 3; ++d) {
    a.L[d] = box3[d];
    a.invL[d] = 1.0 / box3[d];
    a.nc[d] = (int)std::floor(box3[d] / (rc_max + skin));
    if (a.nc[d] < 3) a.allpairs = 1;
    a.ncell *= std::max(a.nc[d], 1);
    h->ilim[d] = a.ilim[d] = 0.5 * box3[d] - (rc_max + 2.0 * skin) - 1e-9 * box3[d];
    h->inside[d] = 0.5 * (box3[d] + skin);
  }
  // lanes per particle: about as many threads as the GPU holds.  us per step, LJ,
  // with 4 / 8 / 16 / 32 lanes: N=4000 34 / 27 / 27 / 26, 8192 32 / 28 / 27 / 30,
  // 32000 48 / 49 / 52 / 62, 65536 72 / 72 / 79 / 100, 200000 174 / 186 / 214 / 281
  h->tp = n < 8192 ? 32 : n < 65536 ? 8 : 4;
  a.fblocks = (int)(((long long)n * h->tp + kB - 1) / kB);
  const double vol = box3[0] * box3[1] * box3[2];
  const double est = n / vol * 4.0 / 3.0 * M_PI * std::pow(rc_max + skin, 3.0);
  a.max_nbrs = max_nbrs > 0 ? max_nbrs : (int)std::min<double>(n - 1, 1.6 * est + 32.0);
  a.skin2_4 = 0.25 * skin * skin;
  a.dt = 0.005; a.T = 1.0; a.omega2 = 4.0 * M_PI * M_PI / (0.2 * 0.2); a.thermo = 1;
  a.dof = 3.0 * n - 3.0;
  int rc = B2MD_OK;
  auto done = [&](int code) {
    if (code) { b2md_f64_destroy(h); return code; }
    *out = h;
    return B2MD_OK;
  };
  if (cudaSetDevice(device) != cudaSuccess) return done(f64_fail(B2MD_ERR_CUDA, "b2md_f64_create: bad device %d", device));
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
    return done(f64_fail(B2MD_ERR_CUDA, "b2md_f64_create: stream creation failed"));
  int sms = 0, per_sm = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k64_rebuild, kB, 0) != cudaSuccess || per_sm < 1)
    return done(f64_fail(B2MD_ERR_CUDA, "b2md_f64_create: the list build does not fit on the device"));
  // the list build's blocks: enough for 8 lanes per particle, two per SM at
  // most (its barriers cost more the more blocks meet)
  h->rb_grid = (int)std::max(1LL, std::min((long long)sms * std::min(per_sm, 2), (8LL * n + kB - 1) / kB));
  const size_t nb = (size_t)((n + kB - 1) / kB), rows = ((size_t)a.max_nbrs + 3) / 4 * 4;
  if ((rc = f64_alloc(h, a.r, n)) || (rc = f64_alloc(h, a.v, n)) || (rc = f64_alloc(h, a.f, n)) ||
      (rc = f64_alloc(h, a.last_r, n)) || (rc = f64_alloc(h, a.im, n)) || (rc = f64_alloc(h, h->scratch, n)) ||
      (rc = f64_alloc(h, a.uid, n)) || (rc = f64_alloc(h, a.cnt, a.ncell)) ||
      (rc = f64_alloc(h, a.cstart, a.ncell)) || (rc = f64_alloc(h, a.ctot, h->rb_grid)) ||
      (rc = f64_alloc(h, a.nn, n)) || (rc = f64_alloc(h, a.nbl, rows * n)) ||
      (rc = f64_alloc(h, a.part, nb * kNPartF64)) || (rc = f64_alloc(h, a.part_f, (size_t)a.fblocks * 2)) ||
      (rc = f64_alloc(h, h->st, 1)) || (rc = f64_alloc(h, h->par, pars.size())))
    return done(rc);
  a.st = h->st;
  a.par = h->par;
  a.im2 = reinterpret_cast<int4*>(h->scratch);
  a.uid2 = reinterpret_cast<unsigned*>(a.im2 + n);
  a.cell = reinterpret_cast<int*>(a.uid2 + n);
  a.rank = a.cell + n;
  a.order = a.rank + n;
  static_assert(sizeof(double4) == sizeof(int4) + 4 * sizeof(int), "the scratch arrays of a particle");
  if (cudaMemcpy(h->par, pars.data(), pars.size() * sizeof(F64Pair), cudaMemcpyHostToDevice) != cudaSuccess)
    return done(f64_fail(B2MD_ERR_CUDA, "b2md_f64_create: parameter upload failed"));
  F64Dev d0 = {};
  d0.need = 1;
  if (cudaMemcpy(h->st, &d0, sizeof d0, cudaMemcpyHostToDevice) != cudaSuccess)
    return done(f64_fail(B2MD_ERR_CUDA, "b2md_f64_create: state upload failed"));
  return done(B2MD_OK);
}

int b2md_f64_destroy(b2md_f64* h) {
  if (!h) return B2MD_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (void* p : h->bufs) cudaFree(p);
  if (h->elog) cudaFree(h->elog);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  std::lock_guard<std::mutex> lock(g_stage_mu);
  if (--g_engines == 0)
    while (g_nfree > 0) cudaFreeHost(g_free[--g_nfree]);
  return B2MD_OK;
}

int b2md_f64_set_state(b2md_f64* h, const double* pos4, const double* vel4, const int* im3) {
  if (!h || !pos4 || !vel4) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_state: null argument");
  const int n = h->a.n;
  std::vector<double4> r(n), v(n);
  std::vector<int4> im(n);
  bool inside = true;
  for (int i = 0; i < n; ++i) {
    const double t = pos4[4 * i + 3];
    if (!(t >= 0.0 && t < h->a.ntypes && t == std::floor(t)))
      return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_state: particle %d has type %g (want 0..%d)", i, t,
                      h->a.ntypes - 1);
    if (!(vel4[4 * i + 3] > 0.0)) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_state: particle %d: 1/m must be > 0", i);
    r[i] = make_double4(pos4[4 * i], pos4[4 * i + 1], pos4[4 * i + 2], t);
    v[i] = make_double4(vel4[4 * i], vel4[4 * i + 1], vel4[4 * i + 2], vel4[4 * i + 3]);
    im[i] = im3 ? make_int4(im3[3 * i], im3[3 * i + 1], im3[3 * i + 2], 0) : make_int4(0, 0, 0, 0);
    inside = inside && std::fabs(r[i].x) <= h->inside[0] && std::fabs(r[i].y) <= h->inside[1] &&
             std::fabs(r[i].z) <= h->inside[2];
  }
  F64_CK(cudaSetDevice(h->device));
  if (h->have_state) {
    // the last forces stay readable: into the caller's order, as the new state is
    k64_unsort<<<nblocks(h), kB, 0, h->stream>>>(h->a, h->a.f, h->scratch, nullptr);
    F64_CK(cudaGetLastError());
    F64_CK(cudaMemcpyAsync(h->a.f, h->scratch, n * sizeof(double4), cudaMemcpyDeviceToDevice, h->stream));
  }
  F64_CK(cudaMemcpyAsync(h->a.r, r.data(), n * sizeof(double4), cudaMemcpyHostToDevice, h->stream));
  F64_CK(cudaMemcpyAsync(h->a.v, v.data(), n * sizeof(double4), cudaMemcpyHostToDevice, h->stream));
  F64_CK(cudaMemcpyAsync(h->a.im, im.data(), n * sizeof(int4), cudaMemcpyHostToDevice, h->stream));
  k64_iota<<<nblocks(h), kB, 0, h->stream>>>(h->a.uid, n);
  F64_CK(cudaGetLastError());
  const int one = 1;
  F64_CK(cudaMemcpyAsync(&h->st->need, &one, sizeof(int), cudaMemcpyHostToDevice, h->stream));
  F64_CK(cudaStreamSynchronize(h->stream));
  for (int d = 0; d < 3; ++d) h->a.ilim[d] = inside ? h->ilim[d] : -1.0;
  h->have_state = true;
  return B2MD_OK;
}

int b2md_f64_set_integrator(b2md_f64* h, double dt, double target_T, double tau, int thermostat_on,
                            int reset_interval) {
  if (!h) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_integrator: null engine");
  if (!(dt > 0.0)) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_integrator: dt must be > 0");
  if (thermostat_on && !(target_T > 0.0 && tau > 0.0))
    return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_integrator: thermostat needs T > 0 and tau > 0");
  if (reset_interval < 0) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_integrator: reset_interval must be >= 0");
  h->a.dt = dt;
  h->a.T = target_T;
  h->a.thermo = thermostat_on ? 1 : 0;
  h->a.omega2 = thermostat_on ? 4.0 * M_PI * M_PI / (tau * tau) : 0.0;
  h->reset_interval = reset_interval;
  return B2MD_OK;
}

int b2md_f64_set_xi(b2md_f64* h, double xi) {
  if (!h) return f64_fail(B2MD_ERR_ARG, "b2md_f64_set_xi: null engine");
  F64_CK(cudaSetDevice(h->device));
  F64_CK(cudaMemcpyAsync(&h->st->xi, &xi, sizeof(double), cudaMemcpyHostToDevice, h->stream));
  F64_CK(cudaStreamSynchronize(h->stream));
  return B2MD_OK;
}

int b2md_f64_calc_f(b2md_f64* h) {
  if (!h) return f64_fail(B2MD_ERR_ARG, "b2md_f64_calc_f: null engine");
  if (!h->have_state) return f64_fail(B2MD_ERR_STATE, "b2md_f64_calc_f: no state set");
  F64_CK(cudaSetDevice(h->device));
  int rc = launch_forces(h);
  if (rc) return rc;
  k64_finish<<<1, kB, 0, h->stream>>>(h->a);
  F64_CK(cudaGetLastError());
  return check_overflow(h);
}

int b2md_f64_run(b2md_f64* h, long long nsteps, double* energies) {
  if (!h) return f64_fail(B2MD_ERR_ARG, "b2md_f64_run: null engine");
  if (nsteps < 0) return f64_fail(B2MD_ERR_ARG, "b2md_f64_run: nsteps must be >= 0");
  if (!h->have_state) return f64_fail(B2MD_ERR_STATE, "b2md_f64_run: no state set");
  F64_CK(cudaSetDevice(h->device));
  double* d_log = nullptr;
  if (energies && nsteps > 0) {
    if (nsteps > h->elog_cap) {
      F64_CK(cudaStreamSynchronize(h->stream));
      if (h->elog) cudaFree(h->elog);
      h->elog = nullptr;
      h->elog_cap = 0;
      F64_CK(cudaMalloc(&h->elog, (size_t)nsteps * 4 * sizeof(double)));
      h->elog_cap = nsteps;
    }
    d_log = h->elog;
  }
  const int B = nblocks(h);
  int rc = B2MD_OK;
  for (long long k = 0; k < nsteps && rc == B2MD_OK; ++k) {
    if (h->reset_interval > 0 && k % h->reset_interval == 0) {
      k64_momentum_part<<<B, kB, 0, h->stream>>>(h->a);
      k64_momentum_total<<<1, kB, 0, h->stream>>>(h->a, B);
      k64_momentum_apply<<<B, kB, 0, h->stream>>>(h->a);
    }
    rc = launch_forces(h);
    if (rc) break;
    k64_integrate<<<B, kB, 0, h->stream>>>(h->a, d_log ? d_log + 4 * k : nullptr);
    for (int d = 0; d < 3; ++d) h->a.ilim[d] = h->ilim[d];  // the step wraps what a state gave unwrapped
    if (cudaGetLastError() != cudaSuccess) rc = f64_fail(B2MD_ERR_CUDA, "b2md_f64_run: launch failed");
    if (rc == B2MD_OK && (k + 1) % 256 == 0) rc = check_overflow(h);
  }
  if (rc == B2MD_OK) rc = check_overflow(h);
  if (rc == B2MD_OK && d_log) {
    if (cudaMemcpy(energies, d_log, (size_t)nsteps * 4 * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = f64_fail(B2MD_ERR_CUDA, "b2md_f64_run: energy copy failed");
  }
  // (a log of more than 64 MB is not kept)
  if (h->elog_cap > (1LL << 21)) {
    cudaFree(h->elog);
    h->elog = nullptr;
    h->elog_cap = 0;
  }
  return rc;
}

int b2md_f64_get(b2md_f64* h, int field, void* out) {
  if (!h || !out) return f64_fail(B2MD_ERR_ARG, "b2md_f64_get: null argument");
  const int n = h->a.n;
  F64_CK(cudaSetDevice(h->device));
  if (field >= B2MD_F64_POS && field <= B2MD_F64_IMAGES) {
    // (the order of the caller's particles comes with the state)
    if (!h->have_state) return f64_fail(B2MD_ERR_STATE, "b2md_f64_get: no state set");
    const double4* src = field == B2MD_F64_POS ? h->a.r : field == B2MD_F64_VEL ? h->a.v : field == B2MD_F64_FORCE ? h->a.f : nullptr;
    const size_t bytes = (size_t)n * (src ? sizeof(double4) : 3 * sizeof(int));
    k64_unsort<<<nblocks(h), kB, 0, h->stream>>>(h->a, src, h->scratch, reinterpret_cast<int*>(h->scratch));
    F64_CK(cudaGetLastError());
    void* stage = take_stage();
    cudaError_t err = cudaSuccess;
    if (!stage) {  // no page-locked memory to be had
      err = cudaMemcpyAsync(out, h->scratch, bytes, cudaMemcpyDeviceToHost, h->stream);
      if (err == cudaSuccess) err = cudaStreamSynchronize(h->stream);
    }
    for (size_t b = 0; stage && b < bytes && err == cudaSuccess; b += kStageBytes) {
      const size_t m = std::min(kStageBytes, bytes - b);
      err = cudaMemcpyAsync(stage, reinterpret_cast<const char*>(h->scratch) + b, m, cudaMemcpyDeviceToHost, h->stream);
      if (err == cudaSuccess) err = cudaStreamSynchronize(h->stream);
      if (err == cudaSuccess) std::memcpy(static_cast<char*>(out) + b, stage, m);
    }
    if (stage) give_stage(stage);
    F64_CK(err);
    return B2MD_OK;
  }
  return f64_fail(B2MD_ERR_ARG, "b2md_f64_get: unknown field %d", field);
}

int b2md_f64_stats(b2md_f64* h, double* out) {
  if (!h || !out) return f64_fail(B2MD_ERR_ARG, "b2md_f64_stats: null argument");
  F64_CK(cudaSetDevice(h->device));
  F64Dev d;
  int rc = read_dev(h, &d);
  if (rc) return rc;
  out[0] = d.pe; out[1] = d.W; out[2] = d.ke_t; out[3] = d.ke2; out[4] = d.xi;
  out[5] = (double)d.rebuilds; out[6] = (double)d.steps;
  return B2MD_OK;
}

}  // extern "C"
