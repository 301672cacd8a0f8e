// LJ forces, potential energy and virial of one configuration without any
// device allocation.
//
// Some callers cannot allocate device memory when they call this library:
// a host application that owns every device buffer and hands a plugin only
// pointers to its own buffers, or a real-time loop that must not call
// cudaMalloc/cudaFree because those may synchronise the device and take
// unbounded time.  b2md_forces_noalloc serves them: the caller passes device
// pointers to its own inputs and outputs, and the only scratch memory (the
// particles binned in cells, the per-block FP64 partial sums of the energy and
// virial and a completion counter) is a fixed, statically allocated array in
// this library's device image, sized for at most kNoAllocMaxParticles
// particles.
//
// The array exists once per GPU that loads the library and lives until the
// process exits.  Every call shares it, so calls whose kernels overlap on the
// GPU (different streams, no ordering between them) race on it; order them on
// one stream or with events.  Their results are then undefined, but nothing
// outside the scratch and the calls' own outputs is touched: every index that
// comes from the scratch is held to the call's particles.  The completion
// counter and the cell counts are cleared at the start of every call; the rest
// is overwritten before it is read.
//
// Host code cannot use the array's name as a device address (it names a
// host-side stand-in).  The first call on a device, with that device current,
// looks the address up with cudaGetSymbolAddress and keeps it together with
// the device's current CUDA context; a later call in another context (after
// cudaDeviceReset, say, which unloads the module and so moves the array)
// looks it up again.  Make the first call on a device before any stream
// capture, since the lookup is not a stream operation.
//
// The pair sum uses the minimum-image convention, which counts each pair once;
// that equals the periodic sum only while every cut-off is at most half of
// every box length, so larger cut-offs are rejected.
//
// Its results match b2md_calc_f for the same configuration: the same pair
// function (shifted-force / shifted-potential / plain LJ), all pairs within
// the cut-off under the minimum-image convention, per-particle energies halved.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <mutex>

#include "../../include/rumd_b200.h"
#include "pbc_math.cuh"

namespace {

constexpr int kNoAllocMaxParticles = 65536;
constexpr int kNoAllocBlock = 128;
constexpr int kNoAllocWarps = kNoAllocBlock / 32;
constexpr int kNoAllocMaxBlocks = 2048;
constexpr int kNoAllocMaxCells = 65536;
constexpr int kNoAllocMaxTypes = 8;
constexpr int kRow = 8;    // rc^2, A12, A6, c_s, c_u0, 6 A6, unused x2
constexpr int kRows = 25;  // (dz, dy) rows of a cell's 5x5x5 neighbourhood

struct NoAllocScratch {
  unsigned counter;            // blocks finished in this call; cleared with cnt
  int dense;                   // a cell is too crowded (crowd_limit): all pairs instead
  unsigned pad[62];
  int cnt[kNoAllocMaxCells];   // particles per cell
  int start[kNoAllocMaxCells]; // first sorted place of each cell
  int key[kNoAllocMaxParticles], rank[kNoAllocMaxParticles], order[kNoAllocMaxParticles];
  float4 pos[kNoAllocMaxParticles];   // sorted by (cell, index), wrapped into the box
  unsigned id[kNoAllocMaxParticles];  // the particle of each sorted place; kBadType set: unknown type
  double part[kNoAllocMaxBlocks][2];  // per-block sums of u_i and w_i
};
constexpr unsigned kBadType = 0x80000000u;
constexpr unsigned kNoParticle = 0xffffffffu;  // a group's place without a particle: past every n
// One warp works on a cell's particles, so a few crowded cells (a cluster in a
// much larger box) would leave the work to a few warps: then the all-pairs form
// runs, which spreads evenly.  A round of 32 candidates takes a warp about
// 0.5 us in both, so their longest chains are compared: the fullest cell's
// groups of four against 125 cells as full, and a warp's share of all pairs.
// The first is three to four times what the fullest cell of an even liquid
// has, whose neighbours hold the mean, hence the factor.  With the number in a
// cell as the only bound, a droplet of density 0.06 in a box of 400 took
// 1297 us at N=8000 and 747 at N=3500, now 172 and 94 (one thread per particle
// against all, before there were cells: 673 and 302).
constexpr int kDense = 64;
constexpr int kResidentWarps = 148 * 7 * kNoAllocWarps;  // k_forces_noalloc

// The largest number of particles in a cell for which the cells are used.
int crowd_limit(int n) {
  const long long all = (long long)(((n + 3) / 4 + kResidentWarps - 1) / kResidentWarps) * n;
  int most = kDense;
  while (most > 1 && (long long)((most + 3) / 4) * std::min(n, 125 * most) > 4 * all) --most;
  return most;
}

// The scratch: a fixed array in the library's device image (no allocation).
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

struct PairTable {
  float p[kNoAllocMaxTypes * kNoAllocMaxTypes * kRow];
};

// Device address of g_noalloc_scratch per device, looked up once per device
// and context (the context the address was found in is kept beside it).
std::mutex g_mu;
NoAllocScratch* g_scratch_ptr[64] = {};
void* g_scratch_ctx[64] = {};

struct Grid3 {
  int nx, ny, nz;
};

// ---- particles binned in cells: sorted by (cell, index), so that every sum
// below has a fixed order ----
__device__ __forceinline__ float wrapped(float x, float L, float iL) {
  return __fmaf_rn(-L, rintf(x * iL), x);  // x itself inside the box
}
__device__ __forceinline__ int cell_of(float x, float iL, int nc) {
  const int c = __float2int_rz(__fmaf_rn(x, iL, 0.5f) * (float)nc);  // 0 for NaN
  return min(max(c, 0), nc - 1);
}

__global__ void __launch_bounds__(256) k_na_count(const float4* __restrict__ pos, int n, float3 L, float3 iL, Grid3 g,
                                                  NoAllocScratch* scr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 r = pos[i];
  const int c = cell_of(wrapped(r.x, L.x, iL.x), iL.x, g.nx) +
                g.nx * (cell_of(wrapped(r.y, L.y, iL.y), iL.y, g.ny) + g.ny * cell_of(wrapped(r.z, L.z, iL.z), iL.z, g.nz));
  scr->key[i] = c;
  scr->rank[i] = atomicAdd(&scr->cnt[c], 1);
}

// exclusive scan of the cell counts (and the largest) by one block: thread t
// owns a run of cells
__global__ void __launch_bounds__(1024) k_na_scan(int ncell, int limit, NoAllocScratch* scr) {
  __shared__ int s_w[32], s_m[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int run = ((ncell + 1023) / 1024 + 3) & ~3;  // whole int4 loads
  const int c0 = threadIdx.x * run, c1 = min(ncell, c0 + run);
  int tot = 0, most = 0;
  for (int c = c0; c < c1; c += 4) {  // counts past ncell are zero
    const int4 x = *reinterpret_cast<const int4*>(scr->cnt + c);
    tot += x.x + x.y + x.z + x.w;
    most = max(max(most, max(x.x, x.y)), max(x.z, x.w));
  }
  most = __reduce_max_sync(0xffffffffu, most);
  int incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) {
    s_w[wid] = incl;
    s_m[wid] = most;
  }
  __syncthreads();
  int first = incl - tot;
  for (int w = 0; w < wid; ++w) first += s_w[w];
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) most = max(most, s_m[w]);
    scr->dense = most > limit;
  }
  for (int c = c0; c < c1; c += 4) {
    const int4 x = *reinterpret_cast<const int4*>(scr->cnt + c);
    const int4 o = make_int4(first, first + x.x, first + x.x + x.y, first + x.x + x.y + x.z);
    *reinterpret_cast<int4*>(scr->start + c) = o;
    first = o.w + x.w;
  }
}

__global__ void __launch_bounds__(256) k_na_scatter(int n, NoAllocScratch* scr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) scr->order[min(scr->start[scr->key[i]] + scr->rank[i], n - 1)] = i;
}

// Each bucket by index (its members counted against each other; a few per
// cell), positions wrapped into the box.  A particle of unknown type gets a
// NaN position: no pair with it is in range.
__global__ void __launch_bounds__(256) k_na_gather(const float4* __restrict__ pos, int n, float3 L, float3 iL,
                                                   int ntypes, NoAllocScratch* scr) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n || scr->dense) return;
  const int i = min(scr->order[s], n - 1), c = scr->key[i], b = min(scr->start[c], n), m = min(scr->cnt[c], n - b);
  int place = b;
  for (int k = 0; k < m; ++k) place += scr->order[b + k] < i;
  place = min(place, n - 1);
  float4 r = pos[i];
  const int t = __float_as_int(r.w);
  const bool ok = t >= 0 && t < ntypes;
  r.x = ok ? wrapped(r.x, L.x, iL.x) : __int_as_float(0x7fc00000);
  r.y = wrapped(r.y, L.y, iL.y);
  r.z = wrapped(r.z, L.z, iL.z);
  r.w = ok ? r.w : 0.f;
  scr->pos[place] = r;
  scr->id[place] = (unsigned)i | (ok ? 0u : kBadType);
}

// ---- pair sums ----
struct Sum5 {
  float fx = 0.f, fy = 0.f, fz = 0.f, u = 0.f, w = 0.f;
};

// The warp's sums of G particles' values: lane q 32/G holds particle q's
// total (fixed tree; halving exchanges while more than one particle is left).
template <int G>
__device__ __forceinline__ float warp_sum(const float (&v)[G]) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float x;
  int o = 16;
  if constexpr (G == 4) {
    float a[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float keep = lane & 16 ? v[k + 2] : v[k], give = lane & 16 ? v[k] : v[k + 2];
      a[k] = keep + __shfl_xor_sync(FULL, give, 16);
    }
    x = (lane & 8 ? a[1] : a[0]) + __shfl_xor_sync(FULL, lane & 8 ? a[0] : a[1], 8);
    o = 4;
  } else if constexpr (G == 2) {
    x = (lane & 16 ? v[1] : v[0]) + __shfl_xor_sync(FULL, lane & 16 ? v[0] : v[1], 16);
    o = 8;
  } else {
    x = v[0];
  }
#pragma unroll
  for (; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
  return x;
}

// Candidate j of every lane (a NaN position where the lane has none) against
// the warp's G particles.  wrap: the dimensions (1, 2, 4) that need the
// minimum-image step; uniform in the warp.
template <int G, bool SF>
__device__ __forceinline__ void add_candidate(Sum5 (&A)[G], const float4 (&rp)[G], int p0, int j, const float4& rj,
                                              unsigned wrap, const float* s_tab, int ntypes, const float3& L,
                                              const float3& iL) {
  const int tj = __float_as_int(rj.w);
  float dx[G], dy[G], dz[G];
#pragma unroll
  for (int q = 0; q < G; ++q) {
    dx[q] = rp[q].x - rj.x;
    dy[q] = rp[q].y - rj.y;
    dz[q] = rp[q].z - rj.z;
  }
  if (wrap & 1u)
#pragma unroll
    for (int q = 0; q < G; ++q) dx[q] = b2md::mi_comp(dx[q], L.x, iL.x);
  if (wrap & 2u)
#pragma unroll
    for (int q = 0; q < G; ++q) dy[q] = b2md::mi_comp(dy[q], L.y, iL.y);
  if (wrap & 4u)
#pragma unroll
    for (int q = 0; q < G; ++q) dz[q] = b2md::mi_comp(dz[q], L.z, iL.z);
#pragma unroll
  for (int q = 0; q < G; ++q) {
    const float d2 = b2md::dist2_ref(dx[q], dy[q], dz[q]);
    const float* row = s_tab + (__float_as_int(rp[q].w) * ntypes + tj) * kRow;
    const float4 c = *reinterpret_cast<const float4*>(row);  // rc^2, A12, A6, c_s
    const bool in = d2 < c.x && j != p0 + q;
    if (!__any_sync(0xffffffffu, in)) continue;
    // the engine's pair function (pair_add of the step kernels), with 1/r^2 the
    // hardware reciprocal of d^2 (one unit in the last place; the energies'
    // error against 64-bit sums is a tenth of that with the square of 1/r) and
    // 1/r, which only the shifted-force term uses, refined as there
    const float2 e = *reinterpret_cast<const float2*>(row + 4);  // c_u0, 6 A6
    const float i2 = b2md::rcp_approx(d2), i6 = i2 * i2 * i2, t = c.y * i6;
    float s = i6 * i2 * __fmaf_rn(12.f, t, e.y), u0 = e.x;
    if constexpr (SF) {
      float y = b2md::rsqrt_approx(d2);
      y = y * __fmaf_rn(-0.5f * d2 * y, y, 1.5f);
      s = __fmaf_rn(-c.w, y, s);
      u0 = __fmaf_rn(c.w, d2 * y, u0);
    }
    if (in) {  // (dx is NaN in lanes without a candidate)
      A[q].u += __fmaf_rn(i6, t + c.z, u0);
      A[q].fx = __fmaf_rn(dx[q], s, A[q].fx);
      A[q].fy = __fmaf_rn(dy[q], s, A[q].fy);
      A[q].fz = __fmaf_rn(dz[q], s, A[q].fz);
      A[q].w = __fmaf_rn(d2, s, A[q].w);
    }
  }
}

// Forces of particles p0 .. p0 + G - 1 from the sums, by the lanes that hold
// them; their energies and virials are added to u, w.
template <int G>
__device__ __forceinline__ void store_forces(const Sum5 (&A)[G], const unsigned (&id)[G], int n,
                                             float4* __restrict__ force, double& u, double& w) {
  float v[5][G];
#pragma unroll
  for (int q = 0; q < G; ++q) {
    v[0][q] = A[q].fx; v[1][q] = A[q].fy; v[2][q] = A[q].fz; v[3][q] = A[q].u; v[4][q] = A[q].w;
  }
  const float fx = warp_sum<G>(v[0]), fy = warp_sum<G>(v[1]), fz = warp_sum<G>(v[2]), uu = warp_sum<G>(v[3]),
              ww = warp_sum<G>(v[4]);
  const int lane = threadIdx.x & 31;
  if (lane % (32 / G) == 0) {
    unsigned me = id[0];
#pragma unroll
    for (int q = 1; q < G; ++q) me = lane / (32 / G) == q ? id[q] : me;
    if ((me & ~kBadType) >= (unsigned)n) {
    } else if (me & kBadType) {
      const float nanf_ = __int_as_float(0x7fc00000);
      force[me & ~kBadType] = make_float4(nanf_, nanf_, nanf_, nanf_);
    } else {
      force[me] = make_float4(fx, fy, fz, 0.5f * uu);
      u += 0.5 * (double)uu;
      w += (double)ww;
    }
  }
}

// The m <= G particles of a cell from p0 on (a missing one has a NaN position,
// which is in range of nothing).  The next round's candidates are loaded while
// the current one's pairs are computed.
template <int G, bool SF>
__device__ __forceinline__ void cell_group(NoAllocScratch* scr, int n, const int4* tab, int off, int len, int total,
                                           int p0, int m, unsigned wrap, const float* s_tab, int ntypes, const float3& L,
                                           const float3& iL, float4* __restrict__ force, double& u, double& w) {
  const int lane = threadIdx.x & 31;
  const float nan = __int_as_float(0x7fc00000);
  const float4* __restrict__ sp = scr->pos;
  Sum5 A[G];
  float4 rp[G];
  unsigned id[G];
#pragma unroll
  for (int q = 0; q < G; ++q) {
    rp[q] = q < m ? sp[p0 + q] : make_float4(nan, nan, nan, 0.f);
    id[q] = q < m ? scr->id[p0 + q] : kNoParticle;
  }
  int rows = 0;  // non-empty rows that start before the round
  auto candidate = [&](int ch) -> int {
    const int v = ch + lane;
    const unsigned rel = (unsigned)(off - ch);
    const unsigned st = __reduce_or_sync(0xffffffffu, len > 0 && rel < 32u ? 1u << rel : 0u);
    const int4 t = tab[rows + __popc(st & ((2u << lane) - 1u)) - 1];
    rows += __popc(st);
    return v < total ? v + (v < t.z ? t.y : t.w) : p0;
  };
  int jn = candidate(0);
  float4 rn = sp[jn];
#pragma unroll 1
  for (int ch = 0; ch < total; ch += 32) {
    const int j = jn;
    float4 rj = rn;
    if (ch + 32 < total) {
      jn = candidate(ch + 32);
      rn = sp[jn];
    }
    if (ch + lane >= total) rj.x = nan;
    add_candidate<G, SF>(A, rp, p0, j, rj, wrap, s_tab, ntypes, L, iL);
  }
  store_forces<G>(A, id, n, force, u, w);
}

template <int G, bool SF>
__device__ __forceinline__ void all_pairs_group(const float4* __restrict__ pos, int n, int p0, const float* s_tab,
                                                int ntypes, const float3& L, const float3& iL,
                                                float4* __restrict__ force, double& u, double& w) {
  const int lane = threadIdx.x & 31;
  Sum5 A[G];
  float4 rp[G];
  unsigned id[G];
#pragma unroll
  for (int q = 0; q < G; ++q) {
    rp[q] = pos[p0 + q];
    const int t = __float_as_int(rp[q].w);
    const bool ok = t >= 0 && t < ntypes;
    id[q] = (unsigned)(p0 + q) | (ok ? 0u : kBadType);
    if (!ok) rp[q].w = 0.f;
  }
#pragma unroll 2
  for (int ch = 0; ch < n; ch += 32) {
    const int j = ch + lane;
    float4 rj = pos[min(j, n - 1)];
    const int t = __float_as_int(rj.w);
    if (j >= n || t < 0 || t >= ntypes) {
      rj.x = __int_as_float(0x7fc00000);
      rj.w = 0.f;
    }
    add_candidate<G, SF>(A, rp, p0, j, rj, 7u, s_tab, ntypes, L, iL);
  }
  store_forces<G>(A, id, n, force, u, w);
}

// One warp works on up to four particles at a time, 32 candidates a round, one
// per lane: of a cell's particles against its 5x5x5 neighbourhood (CELLS), or
// of G consecutive particles against all.  Units go to warps in a fixed order.
// What bounds the cell form is the pair arithmetic: about 300 candidates per
// particle at KA density, of which a quarter is in range, and the chain to the
// candidates' positions.  Held to 72 registers for seven blocks per SM (KA
// N=65521: 109 us a call with 96 registers, 112 with 80, 106 with 72, before 1/r
// was refined).  Calls back to back, shifted force, all pairs by one thread per
// particle before: N=65521 7275 -> 111 us (shifted potential 108), N=16384
// 1388 -> 51, N=4000 369 -> 37, N=1000 109 -> 16 (the last three mostly
// launches).
template <int G, bool CELLS, bool SF>
__global__ void __launch_bounds__(kNoAllocBlock, 7)
    k_forces_noalloc(const float4* __restrict__ pos, int n, float3 L, float3 iL, Grid3 g, int ntypes, PairTable tab,
                     float4* __restrict__ force, double* __restrict__ sums, NoAllocScratch* scr) {
  __shared__ __align__(16) float s_tab[kNoAllocMaxTypes * kNoAllocMaxTypes * kRow];
  __shared__ int4 s_rows[kNoAllocWarps * kRows];
  __shared__ double s_red[kNoAllocBlock][2];
  __shared__ int s_last, s_cells;
  if (threadIdx.x == 0) s_cells = CELLS && !scr->dense;
  for (int k = threadIdx.x; k < ntypes * ntypes * kRow; k += blockDim.x) s_tab[k] = tab.p[k];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = gridDim.x * kNoAllocWarps;
  double u = 0.0, w = 0.0;
  if (s_cells) {
    int4* rowtab = s_rows + warp * kRows;
    const int ncell = g.nx * g.ny * g.nz;
    for (int c = blockIdx.x * kNoAllocWarps + warp; c < ncell; c += stride) {
      const int p0 = __shfl_sync(0xffffffffu, min(scr->start[c], n), 0);
      const int p1 = __shfl_sync(0xffffffffu, min(p0 + scr->cnt[c], n), 0);
      if (p0 >= p1) continue;
      const int cx = c % g.nx, cy = (c / g.nx) % g.ny, cz = c / (g.nx * g.ny);
      // with at least 7 cells and none of the five wrapped, candidates are
      // within 3/7 of a box length: the minimum-image step is the identity
      const unsigned wrap = (g.nx >= 7 && cx >= 2 && cx < g.nx - 2 ? 0u : 1u) |
                            (g.ny >= 7 && cy >= 2 && cy < g.ny - 2 ? 0u : 2u) |
                            (g.nz >= 7 && cz >= 2 && cz < g.nz - 2 ? 0u : 4u);
      int b0 = 0, l0 = 0, b1 = 0, l1 = 0;  // lane r < 25: row (dz, dy) as one or two runs of places
      if (lane < kRows) {
        int z = cz + lane / 5 - 2, y = cy + lane % 5 - 2;
        z += ((z < 0) - (z >= g.nz)) * g.nz;
        y += ((y < 0) - (y >= g.ny)) * g.ny;
        const int row = g.nx * (y + g.ny * z), lo = cx - 2, hi = cx + 2;
        const int ca = row + (lo < 0 ? lo + g.nx : lo), cb = row + (hi >= g.nx ? hi - g.nx : hi);
        const bool two = lo < 0 || hi >= g.nx;
        const int ce = two ? row + g.nx - 1 : cb;  // last cell of the first run
        b0 = min(scr->start[ca], n);
        l0 = max(min(scr->start[ce] + scr->cnt[ce], n) - b0, 0);
        if (two) {
          b1 = min(scr->start[row], n);
          l1 = max(min(scr->start[cb] + scr->cnt[cb], n) - b1, 0);
        }
      }
      const int len = l0 + l1;
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int off = incl - len, total = __shfl_sync(0xffffffffu, incl, 31);
      if (total == 0) continue;  // (only beside an overlapping call: a cell is its own neighbour)
      const unsigned ne = __ballot_sync(0xffffffffu, len > 0);
      __syncwarp();
      if (len > 0) rowtab[__popc(ne & ((1u << lane) - 1u))] = make_int4(off, b0 - off, off + l0, b1 - off - l0);
      __syncwarp();
      for (int p = p0; p < p1; p += 4) {
        const int m = min(4, p1 - p);
#define CG(K) cell_group<K, SF>(scr, n, rowtab, off, len, total, p, m, wrap, s_tab, ntypes, L, iL, force, u, w)
        if (m > 2) CG(4);
        else CG(2);
#undef CG
      }
    }
  } else {
    const int units = (n + G - 1) / G;
    for (int k = blockIdx.x * kNoAllocWarps + warp; k < units; k += stride) {
      const int p = k * G;
      if (p + G <= n) {
        all_pairs_group<G, SF>(pos, n, p, s_tab, ntypes, L, iL, force, u, w);
      } else {
        for (int r = p; r < n; ++r) all_pairs_group<1, SF>(pos, n, r, s_tab, ntypes, L, iL, force, u, w);
      }
    }
  }
  // FP64 block sums; the last block adds the blocks in a fixed order
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    u += __shfl_xor_sync(0xffffffffu, u, o);
    w += __shfl_xor_sync(0xffffffffu, w, o);
  }
  if (lane == 0) {
    s_red[warp][0] = u;
    s_red[warp][1] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double bu = 0.0, bw = 0.0;
    for (int k = 0; k < kNoAllocWarps; ++k) {
      bu += s_red[k][0];
      bw += s_red[k][1];
    }
    scr->part[blockIdx.x][0] = bu;
    scr->part[blockIdx.x][1] = bw;
    __threadfence();
    s_last = atomicAdd(&scr->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double su = 0.0, sw = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kNoAllocBlock) {
    su += __ldcg(&scr->part[b][0]);
    sw += __ldcg(&scr->part[b][1]);
  }
  s_red[threadIdx.x][0] = su;
  s_red[threadIdx.x][1] = sw;
  __syncthreads();
  for (int h = kNoAllocBlock / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      s_red[threadIdx.x][0] += s_red[threadIdx.x + h][0];
      s_red[threadIdx.x][1] += s_red[threadIdx.x + h][1];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    sums[0] = s_red[0][0];        // potential energy, sum of u_i
    sums[1] = s_red[0][1] / 6.0;  // virial W = sum w_i / 6
    scr->counter = 0u;
  }
}

// Cells of half the largest cut-off (5x5x5 then covers it), made larger where
// there would be more than the scratch holds; false when a dimension has
// fewer than five, so that the neighbourhood would count a cell twice.
bool cell_grid(const float* box, float rcmax, Grid3* g) {
  double nc[3];
  for (int d = 0; d < 3; ++d) {
    // a cell is wider than rc/2 by more than the rounding of positions to cells
    // (2e-7 of a box length, which is at most 1400 cut-offs in cells this small)
    nc[d] = std::floor(2.0 * (double)box[d] / ((double)rcmax * 1.001));
    if (!(nc[d] >= 5.0)) return false;
    nc[d] = std::min(nc[d], 1048576.0);
  }
  while (nc[0] * nc[1] * nc[2] > (double)kNoAllocMaxCells) {
    const int d = nc[0] >= nc[1] && nc[0] >= nc[2] ? 0 : (nc[1] >= nc[2] ? 1 : 2);
    if (nc[d] <= 5.0) return false;
    nc[d] = std::max(5.0, std::floor(nc[d] * 0.9));
  }
  *g = Grid3{(int)nc[0], (int)nc[1], (int)nc[2]};
  return true;
}

// The current CUDA context (driver call cuCtxGetCurrent, fetched through the
// runtime so that the library needs no link to the driver library); null
// when it cannot be read.
void* current_context() {
  typedef int (*CtxGetCurrent)(void**);
  static CtxGetCurrent fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<CtxGetCurrent>(f);
  }();
  void* ctx = nullptr;
  if (!fn || fn(&ctx) != 0) return nullptr;
  return ctx;
}

// Looks up (once per device and context, with that device current) the
// device address of the scratch array; host code may not use the symbol
// itself as a pointer.
NoAllocScratch* scratch_for_current_device(int* err) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    *err = B2MD_ERR_CUDA;
    return nullptr;
  }
  void* ctx = current_context();
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_ptr[dev] || !ctx || ctx != g_scratch_ctx[dev]) {
    // the lookup also makes the device's primary context current on this
    // thread when none was, so the context is read again after it
    NoAllocScratch* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_noalloc_scratch) != cudaSuccess || !p) {
      *err = B2MD_ERR_CUDA;
      return nullptr;
    }
    g_scratch_ptr[dev] = p;
    g_scratch_ctx[dev] = current_context();
  }
  return g_scratch_ptr[dev];
}

}  // namespace

namespace b2md_internal {
void set_last_error(const char* msg);
}

namespace {
int noalloc_fail(int code, const char* msg) {
  b2md_internal::set_last_error(msg);
  return code;
}
}  // namespace

extern "C" int b2md_forces_noalloc(const float* pos4, int n, const float* box, int ntypes, const float* params,
                                   int cutoff_method, float* force4, double* sums, void* stream) {
  if (n < 2 || n > kNoAllocMaxParticles)
    return noalloc_fail(B2MD_ERR_ARG, "b2md_forces_noalloc: n must be between 2 and 65536 (the size of its "
                                      "fixed scratch array)");
  if (!pos4 || !box || !params || !force4 || !sums) return noalloc_fail(B2MD_ERR_ARG, "b2md_forces_noalloc: null pointer");
  if (ntypes < 1 || ntypes > kNoAllocMaxTypes) return noalloc_fail(B2MD_ERR_ARG, "b2md_forces_noalloc: ntypes must be 1..8");
  if (cutoff_method < 0 || cutoff_method > 2)
    return noalloc_fail(B2MD_ERR_ARG, "b2md_forces_noalloc: cutoff method must be NS, SP or SF");
  if (!(box[0] > 0.f) || !(box[1] > 0.f) || !(box[2] > 0.f))
    return noalloc_fail(B2MD_ERR_ARG, "b2md_forces_noalloc: box lengths must be positive");
  // minimum image counts one image per pair: exact only for rc <= L/2
  float rcmax = 0.f;
  for (int k = 0; k < ntypes * ntypes; ++k) rcmax = params[k * 12] > rcmax ? params[k * 12] : rcmax;
  const float lmin = fminf(box[0], fminf(box[1], box[2]));
  if (rcmax > 0.5f * lmin) {
    char msg[200];
    snprintf(msg, sizeof(msg),
             "b2md_forces_noalloc: cut-off %g exceeds half the smallest box length %g (the minimum-image sum "
             "would miss periodic images)", (double)rcmax, (double)lmin);
    return noalloc_fail(B2MD_ERR_ARG, msg);
  }
  // an error left by an earlier runtime call on this thread is not this
  // call's: clear it so that the launch check below sees only this launch
  (void)cudaGetLastError();
  int err = B2MD_OK;
  NoAllocScratch* scr = scratch_for_current_device(&err);
  if (!scr) return noalloc_fail(err, "b2md_forces_noalloc: cannot find the device address of the scratch array");
  // pack the RUMD table (T*T*12) into the kernel's rows, by value
  PairTable tab = {};
  for (int k = 0; k < ntypes * ntypes; ++k) {
    const float* p = params + k * 12;
    float* q = tab.p + k * kRow;
    const float rc = p[0], sc = p[10], uc = p[11];
    const bool sf = cutoff_method == B2MD_CUTOFF_SF, sp = cutoff_method == B2MD_CUTOFF_SP;
    q[0] = rc * rc;
    q[1] = p[1];
    q[2] = p[2];
    q[3] = sf ? sc : 0.f;
    q[4] = sf ? -(sc * rc + uc) : (sp ? -uc : 0.f);
    q[5] = 6.f * p[2];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // Cells pay from about 3000 particles (us a call with cells / all pairs, one
  // particle per warp: KA N=2400 33 / 27, 3000 35 / 32, 3500 37 / 37, 4000
  // 37 / 41; LJ 2400 31 / 27, 3000 32 / 31, 3500 34 / 36) and where a cell's
  // neighbourhood is a third of the box or less.  Otherwise every warp tests one,
  // two or four particles against all: one while the GPU's warps hold them all
  // in one wave, and more where that would take several (KA with one / two /
  // four: N=2400 27 / 31 / 44 us, 4000 41 / 50 / 70, 4800 81 / 58 / 83, 8000
  // 135 / 101 / 142, 16000 491 / 364 / 354).  The lines at 2400 and 4800 lie
  // before the crossings: only boxes without cells reach the larger sizes.
  Grid3 g{1, 1, 1};
  float reach = 0.f;  // (a pair's range is its cut-off squared, whatever its sign)
  for (int k = 0; k < ntypes * ntypes; ++k) reach = std::max(reach, fabsf(params[k * 12]));
  const bool cells = n >= 3000 && cell_grid(box, reach, &g) && g.nx * g.ny * g.nz >= 3 * 125;
  const int ncell = cells ? g.nx * g.ny * g.nz : 0;
  // the completion counter and the cell counts must start at zero for every
  // call (the counts rounded up to whole int4 loads of the scan)
  const size_t clear = cells ? offsetof(NoAllocScratch, cnt) + ((size_t)ncell + 3) / 4 * 4 * sizeof(int) : sizeof(unsigned);
  const cudaError_t me = cudaMemsetAsync(scr, 0, clear, s);
  if (me != cudaSuccess) {
    char msg[200];
    snprintf(msg, sizeof(msg), "b2md_forces_noalloc: clearing the scratch counter failed: %s",
             cudaGetErrorName(me));
    return noalloc_fail(B2MD_ERR_CUDA, msg);
  }
  const float3 L = make_float3(box[0], box[1], box[2]);
  const float3 iL = make_float3(1.f / box[0], 1.f / box[1], 1.f / box[2]);
  const float4* p4 = reinterpret_cast<const float4*>(pos4);
  float4* f4 = reinterpret_cast<float4*>(force4);
  const int tb = (n + 255) / 256;
  const bool sf = cutoff_method == B2MD_CUTOFF_SF;
#define NA(G, C, UNITS)                                                                                     \
  {                                                                                                         \
    const auto kernel = sf ? k_forces_noalloc<G, C, true> : k_forces_noalloc<G, C, false>;                  \
    kernel<<<std::min(((UNITS) + kNoAllocWarps - 1) / kNoAllocWarps, kNoAllocMaxBlocks), kNoAllocBlock, 0, s>>>( \
        p4, n, L, iL, g, ntypes, tab, f4, sums, scr);                                                       \
  }
  if (cells) {
    k_na_count<<<tb, 256, 0, s>>>(p4, n, L, iL, g, scr);
    k_na_scan<<<1, 1024, 0, s>>>(ncell, crowd_limit(n), scr);
    k_na_scatter<<<tb, 256, 0, s>>>(n, scr);
    k_na_gather<<<tb, 256, 0, s>>>(p4, n, L, iL, ntypes, scr);
    // (a warp per cell, and warps enough for all pairs, four particles each,
    // should the cells turn out crowded)
    NA(4, true, std::max(ncell, (n + 3) / 4))
  } else if (n <= 2400) {
    NA(1, false, n)
  } else if (n <= 4800) {
    NA(2, false, (n + 1) / 2)
  } else {
    NA(4, false, (n + 3) / 4)
  }
#undef NA
  const cudaError_t le = cudaGetLastError();
  if (le != cudaSuccess) {
    char msg[200];
    snprintf(msg, sizeof(msg), "b2md_forces_noalloc: launch failed: %s (%s)", cudaGetErrorName(le),
             cudaGetErrorString(le));
    return noalloc_fail(B2MD_ERR_CUDA, msg);
  }
  return B2MD_OK;
}
