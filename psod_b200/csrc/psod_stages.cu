// psod_stages.cu -- cell-sorted cube, CIC density and seed order.
//
//  stage_cellsort  the linked list of spherover (main:1564-1604) as a
//                  counting sort of the particles into nx^3 SOD cells.
//                  Each particle becomes one 16-byte float4 record, so every
//                  later gather is a coalesced stream of whole cells.
//  stage_cic       cic (main:1077-1265) on the 2nx-per-side periodic grid,
//                  deposited as int64 fixed point (integer atomics are
//                  associative, so the grid is the same on every run).
//  stage_cicm1     cicm1 (main:1268-1390): 8-node gather per particle in the
//                  reference's term order, FP64 without contraction.
//  stage_tri_cic   tri_cic (main:998-1037): 1/rho < 0.01 compaction and a
//                  stable radix sort of the seeds, ties by input index.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "psod_internal.cuh"

namespace psod {

namespace {

constexpr double FIX_ONE = 1099511627776.0;  // 2^40

// ---------------------------------------------------------------------------
// cell sort
// ---------------------------------------------------------------------------
// Slab partition.  The particles arrive in random order, so a direct
// counting sort into nx^3 cells spreads its atomics and its record writes
// over the whole cube.  A first pass groups them by slab (a run of z-planes
// of cells, at most SLAB_MAX slabs) with coalesced writes: each CTA orders a
// tile of SLAB_TILE particles by slab in shared memory and writes one run
// per slab.  The counting sort then reads the records slab after slab, so at
// any moment its atomics and record writes fall into the few slabs that the
// running CTAs hold, which stay in L2.
constexpr int SLAB_MAX = 512;
constexpr int SLAB_TILE = 4096;
constexpr int SLAB_THREADS = 256;
constexpr int SLAB_PER = SLAB_TILE / SLAB_THREADS;

__device__ __forceinline__ bool in_unit_box(float x, float y, float z) {
  return x >= 0.f && x <= 1.f && y >= 0.f && y <= 1.f && z >= 0.f && z <= 1.f;
}

// slab of a position in the unit box: its z cell scaled to the slab count
// (slabs are runs of whole z-planes, so runs of cell indices).  A position
// outside the box has no cell (sod_cell_axis wraps once): k_slab_count sets
// *bad for one, and no pass computes a slab or a cell once it is set.
__device__ __forceinline__ unsigned slab_of(float z, float nxf, double xs, int nx, int nslab) {
  const int k = sod_cell_axis(to_grid(z, nxf), xs, nx);
  return (unsigned)(((long long)k * nslab) / nx);
}

__global__ void __launch_bounds__(SLAB_THREADS) k_slab_count(const float *pos, long long n, float nxf, double xs,
                                                             int nx, int nslab, unsigned *hist, int *bad) {
  __shared__ unsigned h[SLAB_MAX];
  for (int k = threadIdx.x; k < nslab; k += SLAB_THREADS) h[k] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * SLAB_TILE;
  int badl = 0;
  for (int u = 0; u < SLAB_PER; u++) {
    const long long i = base + (long long)u * SLAB_THREADS + threadIdx.x;
    if (i >= n) break;
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    if (!in_unit_box(x, y, z)) {
      badl = 1;
      continue;
    }
    atomicAdd(&h[slab_of(z, nxf, xs, nx, nslab)], 1u);
  }
  if (badl) atomicOr(bad, 1);
  __syncthreads();
  for (int k = threadIdx.x; k < nslab; k += SLAB_THREADS)
    if (h[k]) atomicAdd(&hist[k], h[k]);
}

// exclusive scan of the slab counts into the write cursors (one CTA)
__global__ void k_slab_scan(const unsigned *hist, int nslab, unsigned *cursor) {
  __shared__ unsigned s[SLAB_MAX];
  for (int k = threadIdx.x; k < SLAB_MAX; k += blockDim.x) s[k] = k < nslab ? hist[k] : 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned run = 0;
    for (int k = 0; k < nslab; k++) {
      const unsigned v = s[k];
      cursor[k] = run;
      run += v;
    }
  }
}

// records (x, y, z, input index) grouped by slab; the order inside a slab
// carries no meaning
__global__ void __launch_bounds__(SLAB_THREADS) k_slab_scatter(const float *pos, long long n, float nxf, double xs,
                                                               int nx, int nslab, const int *bad, unsigned *cursor,
                                                               float4 *rec, unsigned *at_of) {
  if (*bad) return;
  __shared__ unsigned cnt[SLAB_MAX], start[SLAB_MAX], gbase[SLAB_MAX], wsum[SLAB_THREADS / 32];
  extern __shared__ __align__(16) unsigned char slab_smem[];
  float4 *stage = reinterpret_cast<float4 *>(slab_smem);                                // SLAB_TILE records
  unsigned short *sdig = reinterpret_cast<unsigned short *>(stage + SLAB_TILE);          // their slabs
  for (int k = threadIdx.x; k < nslab; k += SLAB_THREADS) cnt[k] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * SLAB_TILE;
  const int m = (int)min((long long)SLAB_TILE, n - base);
  unsigned d[SLAB_PER], r[SLAB_PER];
#pragma unroll
  for (int u = 0; u < SLAB_PER; u++) {
    const int j = u * SLAB_THREADS + threadIdx.x;
    if (j < m) {
      d[u] = slab_of(pos[3 * (base + j) + 2], nxf, xs, nx, nslab);
      r[u] = atomicAdd(&cnt[d[u]], 1u);
    }
  }
  __syncthreads();
  // exclusive scan of the slab counts, two slabs a thread (one thread in turn
  // over all of them: the pass took 298 us at 256^3, 276 now with inv written too)
  static_assert(SLAB_MAX == 2 * SLAB_THREADS, "two slabs a thread");
  {
    const int k = 2 * threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned a = k < nslab ? cnt[k] : 0u, b = k + 1 < nslab ? cnt[k + 1] : 0u;
    if (a) gbase[k] = atomicAdd(&cursor[k], a);
    if (b) gbase[k + 1] = atomicAdd(&cursor[k + 1], b);
    unsigned x = a + b;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    x -= a + b;
    for (int q = 0; q < w; q++) x += wsum[q];
    start[k] = x;
    start[k + 1] = x + a;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < SLAB_PER; u++) {
    const int j = u * SLAB_THREADS + threadIdx.x;
    if (j < m) {
      const long long i = base + j;
      const unsigned at = start[d[u]] + r[u];
      stage[at] = make_float4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], __uint_as_float((unsigned)i));
      sdig[at] = (unsigned short)d[u];
      at_of[i] = gbase[d[u]] + r[u];
    }
  }
  __syncthreads();
  // consecutive threads write consecutive records of each slab's run
  for (int j = threadIdx.x; j < m; j += SLAB_THREADS) {
    const unsigned k = sdig[j];
    rec[gbase[k] + (j - start[k])] = stage[j];
  }
}

// The count, the sub-cell count and the scatter below wait for chains of
// dependent L2 reads and atomics at scattered addresses, so each thread
// carries CELL_PER records, the loads of all before the use of any
// (256^3, us a pass: count 215 -> 180, sub-cell count 147 -> 103, scatter
// with its own writes alone 300 with one record a thread, 270 with four).
constexpr int CELL_PER = 4;
constexpr int CELL_TILE = 256 * CELL_PER;

__global__ void __launch_bounds__(256) k_cell_count(const float4 *rec, long long n, float nxf, double3 xs, int nx,
                                                    const int *bad, unsigned *cell, unsigned *count) {
  if (*bad) return;
  const long long i0 = (long long)blockIdx.x * CELL_TILE + threadIdx.x;
  float4 v[CELL_PER];
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const long long i = i0 + u * 256;
    v[u] = i < n ? rec[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const long long i = i0 + u * 256;
    unsigned c = 0xffffffffu;
    if (i < n) {
      const int ci = sod_cell_axis(to_grid(v[u].x, nxf), xs.x, nx);
      const int cj = sod_cell_axis(to_grid(v[u].y, nxf), xs.y, nx);
      const int ck = sod_cell_axis(to_grid(v[u].z, nxf), xs.z, nx);
      c = (unsigned)ci + (unsigned)nx * ((unsigned)cj + (unsigned)nx * (unsigned)ck);
      cell[i] = c;
    }
    // one atomic per distinct cell in the warp
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    if (c != 0xffffffffu && __ffs(peers) - 1 == (int)(threadIdx.x & 31)) atomicAdd(&count[c], __popc(peers));
  }
}

// Cells holding at least SUB_MIN particles are ordered inside by a 4x4x4
// sub-cell key (Morton order), so that consecutive records of a dense cell lie
// close together.  Records inside a cell carry no order of their own (every
// later result is ordered by input index), so this changes no output; it lets
// the refinement hand a warp 32 nearby candidates.
constexpr unsigned SUB_MIN = 64;
constexpr unsigned SUB_N = 64;
constexpr unsigned BIG_FLAG = 0x80000000u;

__device__ __forceinline__ unsigned sub_axis(float xg, double xs) {
  const double d = dsub((double)xg, xs);
  const int s = (int)(dsub(d, floor(d)) * 4.0);
  return (unsigned)min(max(s, 0), 3);
}

__device__ __forceinline__ unsigned sub_key(const float4 &p, float nxf, double3 xs) {
  const unsigned a = sub_axis(to_grid(p.x, nxf), xs.x), b = sub_axis(to_grid(p.y, nxf), xs.y),
                 c = sub_axis(to_grid(p.z, nxf), xs.z);
  return (a & 1u) | ((b & 1u) << 1) | ((c & 1u) << 2) | ((a >> 1) << 3) | ((b >> 1) << 4) | ((c >> 1) << 5);
}

// count[c] becomes BIG_FLAG | table index for cells of SUB_MIN or more
// particles, else the cell's first slot start[c] (the fill cursor of the
// scatter, so that one atomic gives the slot; start < n < 2^31 keeps the
// flag bit clear).  bigcell has room for every cell that can be dense, so no
// pass counts them first (a zone of a 512^3 grid: 1.05 -> 0.64 ms).
__global__ void k_mark_big(unsigned *count, unsigned long long ncell, unsigned *nbig, unsigned *bigcell,
                           const unsigned *start) {
  const unsigned long long c = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool big = c < ncell && count[c] >= SUB_MIN;
  const unsigned m = __ballot_sync(0xffffffffu, big);
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (lane == 0 && m) base = atomicAdd(nbig, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (c >= ncell) return;
  if (big) {
    const unsigned idx = base + __popc(m & ((1u << lane) - 1u));
    bigcell[idx] = (unsigned)c;
    count[c] = BIG_FLAG | idx;
  } else {
    count[c] = start[c];
  }
}

__global__ void __launch_bounds__(256) k_sub_count(const float4 *rec, long long n, const unsigned *cell,
                                                   const unsigned *count, float nxf, double3 xs, unsigned *tab) {
  const long long i0 = (long long)blockIdx.x * CELL_TILE + threadIdx.x;
  unsigned v[CELL_PER];
  float4 r[CELL_PER];
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const long long i = i0 + u * 256;
    v[u] = i < n ? cell[i] : 0xffffffffu;
  }
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) v[u] = i0 + u * 256 < n ? count[v[u]] : 0u;
#pragma unroll
  for (int u = 0; u < CELL_PER; u++)
    if (v[u] & BIG_FLAG) r[u] = rec[i0 + u * 256];
#pragma unroll
  for (int u = 0; u < CELL_PER; u++)
    if (v[u] & BIG_FLAG)
      atomicAdd(&tab[(unsigned long long)(v[u] & ~BIG_FLAG) * SUB_N + sub_key(r[u], nxf, xs)], 1u);
}

// one warp per dense cell: sub-cell counts -> absolute start slots
__global__ void k_sub_scan(unsigned *tab, const unsigned *bigcell, unsigned nbig, const unsigned *start) {
  const unsigned b = (unsigned)(((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (b >= nbig) return;
  unsigned *t = tab + (unsigned long long)b * SUB_N;
  const unsigned a0 = t[2 * lane], a1 = t[2 * lane + 1];
  unsigned x = a0 + a1;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const unsigned excl = start[bigcell[b]] + x - (a0 + a1);
  t[2 * lane] = excl;
  t[2 * lane + 1] = excl + a0;
}

__global__ void __launch_bounds__(256) k_cell_scatter(const float4 *rec, long long n, unsigned *cell,
                                                      unsigned *fill, unsigned *tab, float nxf, double3 xs,
                                                      float4 *cube) {
  const long long i0 = (long long)blockIdx.x * CELL_TILE + threadIdx.x;
  const int lane = threadIdx.x & 31;
  unsigned c[CELL_PER], v[CELL_PER], base[CELL_PER], peers[CELL_PER];
  float4 r[CELL_PER];
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const long long i = i0 + u * 256;
    c[u] = i < n ? cell[i] : 0xffffffffu;
    r[u] = i < n ? rec[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the flag bit never changes under the atomics below
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) v[u] = i0 + u * 256 < n ? fill[c[u]] : 0u;
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const bool in = i0 + u * 256 < n, big = (v[u] & BIG_FLAG) != 0;
    const unsigned sub = big ? sub_key(r[u], nxf, xs) : 0u;
    // records of one cell, and of one sub-cell where the cell is dense
    peers[u] = __match_any_sync(0xffffffffu, in ? c[u] : 0xffffffffu);
    if (__any_sync(0xffffffffu, big)) peers[u] &= __match_any_sync(0xffffffffu, sub);
    base[u] = 0;
    if (in && lane == __ffs(peers[u]) - 1)
      base[u] = big ? atomicAdd(&tab[(unsigned long long)(v[u] & ~BIG_FLAG) * SUB_N + sub], __popc(peers[u]))
                    : atomicAdd(&fill[c[u]], __popc(peers[u]));
  }
#pragma unroll
  for (int u = 0; u < CELL_PER; u++) {
    const unsigned slot =
        __shfl_sync(0xffffffffu, base[u], __ffs(peers[u]) - 1) + __popc(peers[u] & ((1u << lane) - 1u));
    if (i0 + u * 256 < n) {
      cube[slot] = r[u];
      cell[i0 + u * 256] = slot;
    }
  }
}

// Slot of each input record: inv holds its place among the slab records
// (written by the partition in input order), slot the cube slot of each of
// those.  A tile's records lie in one short run per slab, so the sectors that
// a CTA gathers from are read whole; writing inv from the scatter instead
// takes a sector per record, spread over all of inv (256^3: scatter 565 us,
// now 270 and 53 here; 512^3: 7.6 ms, now 2.7 and 1.0).
__global__ void __launch_bounds__(SLAB_THREADS) k_slot_of_input(unsigned *inv, long long n, const unsigned *slot) {
  const long long i0 = (long long)blockIdx.x * SLAB_TILE + threadIdx.x;
  unsigned v[SLAB_PER];
#pragma unroll
  for (int u = 0; u < SLAB_PER; u++) {
    const long long i = i0 + u * SLAB_THREADS;
    v[u] = i < n ? inv[i] : 0u;
  }
#pragma unroll
  for (int u = 0; u < SLAB_PER; u++) v[u] = slot[v[u]];
#pragma unroll
  for (int u = 0; u < SLAB_PER; u++) {
    const long long i = i0 + u * SLAB_THREADS;
    if (i < n) inv[i] = v[u];
  }
}

// Dense sub-cells are then ordered by a finer Morton key inside the
// sub-cell: 4, 8 or 16 bins per axis for sub-cells of at least 32, 128 or
// 1024 records, so a bin holds about one record and 64 consecutive records
// of a dense cell span a box a few bins wide.  This is what lets the
// refinement's group boxes stay small in halo cores (tens of thousands of
// particles per cell), where the 4x4x4 order alone leaves a 64-record group
// spread over a whole sub-cell.  Like the sub-cell order it changes no
// output.
constexpr unsigned FINE_MIN = 32, FINE_BINS_MAX = 4096;

__device__ __forceinline__ unsigned fine_axis(float xg, double xs, int bits) {
  const double d = dsub((double)xg, xs);
  const int q = (int)(dsub(d, floor(d)) * (double)(4 << bits));
  return (unsigned)q & ((1u << bits) - 1u);
}

__device__ __forceinline__ unsigned fine_key(const float4 &p, float nxf, double3 xs, int bits) {
  const unsigned a = fine_axis(to_grid(p.x, nxf), xs.x, bits), b = fine_axis(to_grid(p.y, nxf), xs.y, bits),
                 c = fine_axis(to_grid(p.z, nxf), xs.z, bits);
  unsigned k = 0;
  for (int j = 0; j < bits; j++)
    k |= (((a >> j) & 1u) << (3 * j)) | (((b >> j) & 1u) << (3 * j + 1)) | (((c >> j) & 1u) << (3 * j + 2));
  return k;
}

// one CTA per dense cell, its 64 sub-cells in turn: a counting sort of each
// sub-cell of FINE_MIN or more records by its fine key, through tmp (the
// same slots of a spare record array), then back into the cube with inv
// updated.  tab holds the sub-cells' end slots (the scatter's cursors).
__global__ void __launch_bounds__(256) k_sub_fine(float4 *cube, unsigned *inv, float4 *tmp, const unsigned *tab,
                                                  const unsigned *bigcell, const unsigned *start, float nxf,
                                                  double3 xs) {
  __shared__ unsigned hist[FINE_BINS_MAX];
  __shared__ unsigned wtot[8];
  const unsigned b = blockIdx.x;
  const unsigned *t = tab + (unsigned long long)b * SUB_N;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  unsigned a = start[bigcell[b]];
  for (unsigned s = 0; s < SUB_N; s++) {
    const unsigned e = t[s], m = e - a;
    if (m >= FINE_MIN) {
      const int bits = m >= 1024u ? 4 : (m >= 128u ? 3 : 2);
      const unsigned nb = 1u << (3 * bits), per = (nb + 255u) / 256u;  // nb <= 4096: per <= 16
      for (unsigned i = tid; i < nb; i += 256u) hist[i] = 0u;
      __syncthreads();
      for (unsigned i = a + tid; i < e; i += 256u) atomicAdd(&hist[fine_key(cube[i], nxf, xs, bits)], 1u);
      __syncthreads();
      // exclusive scan: thread tid owns bins [tid*per, tid*per + per)
      const unsigned lo = min(nb, (unsigned)tid * per), hi = min(nb, lo + per);
      unsigned own = 0;
      for (unsigned i = lo; i < hi; i++) own += hist[i];
      unsigned x = own;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wtot[wid] = x;
      __syncthreads();
      unsigned wbase = 0;
      for (int q = 0; q < wid; q++) wbase += wtot[q];
      unsigned run = wbase + x - own;
      for (unsigned i = lo; i < hi; i++) {
        const unsigned h = hist[i];
        hist[i] = run;
        run += h;
      }
      __syncthreads();
      for (unsigned i = a + tid; i < e; i += 256u) {
        const float4 v = cube[i];
        tmp[a + atomicAdd(&hist[fine_key(v, nxf, xs, bits)], 1u)] = v;
      }
      __syncthreads();
      for (unsigned i = a + tid; i < e; i += 256u) {
        const float4 v = tmp[i];
        cube[i] = v;
        inv[__float_as_uint(v.w)] = i;
      }
      __syncthreads();
    }
    a = e;
  }
}

__global__ void k_set_range(unsigned *a, unsigned long long lo, unsigned long long hi, unsigned v) {
  unsigned long long i = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < hi) a[i] = v;
}

// ---------------------------------------------------------------------------
// CIC along one axis (main:1154-1190): returns the two node indices and the
// weights ddx (upper node) and dex (lower node).
// ---------------------------------------------------------------------------
struct CicConst {
  double xxmin[3], xxmax[3];  // zone with buffer per axis, box units
  double dx, kc;
  double inv_dx;  // 1/dx when it is exact (dx a power of two), else 0
  int nc;
  int zone_test;  // 1: particles outside the zone with buffer are skipped (main:1138-1146)
};

// CIC along one axis (main:1154-1190): the two node indices and the weights
// ddx (upper node) and dex (lower node).  (x - xxmin)/dx is formed as a
// product when 1/dx is exact, which gives the same double.
__device__ __forceinline__ void cic_axis(float xf, const CicConst &k, int a, int &i0, int &i1, double &dd, double &de) {
  const double diff = dsub((double)xf, k.xxmin[a]);
  double d = k.inv_dx != 0.0 ? dmul(diff, k.inv_dx) : ddiv(diff, k.dx);
  int ix = (int)d;  // Fortran int(): truncation
  if (d < 0.0) ix = ix - 1;
  d = dsub(d, (double)ix);
  const double e = dsub(1.0, d);
  int ixp1 = ix + 1;
  const int nc = k.nc;
  if (ixp1 < 0) ixp1 += nc;
  if (ix < 0) ix += nc;
  if (ixp1 >= nc) ixp1 -= nc;
  if (ix >= nc) ix -= nc;
  i0 = ix;
  i1 = ixp1;
  dd = d;
  de = e;
}

__device__ __forceinline__ bool in_zone_periodic(double x, double lo, double hi) {
  return (x >= lo && x <= hi) || (x >= dadd(lo, 1.0) && x <= dadd(hi, 1.0)) ||
         (x >= dsub(lo, 1.0) && x <= dsub(hi, 1.0));
}

// the particle selection of cic and cicm1 (main:1138-1146, 1309-1317)
__device__ __forceinline__ bool in_cic_zone(const float4 &p, const CicConst &k) {
  return in_zone_periodic(p.x, k.xxmin[0], k.xxmax[0]) && in_zone_periodic(p.y, k.xxmin[1], k.xxmax[1]) &&
         in_zone_periodic(p.z, k.xxmin[2], k.xxmax[2]);
}

// deposit: 8 int64 atomics per particle, weights quantised to 2^-40
__global__ void k_cic_deposit(const float4 *cube, long long n, CicConst k, unsigned long long *grid) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = cube[i];
  if (!in_cic_zone(p, k)) return;
  int ix, ixp, iy, iyp, iz, izp;
  double ddx, dex, ddy, dey, ddz, dez;
  cic_axis(p.x, k, 0, ix, ixp, ddx, dex);
  cic_axis(p.y, k, 1, iy, iyp, ddy, dey);
  cic_axis(p.z, k, 2, iz, izp, ddz, dez);
  const long long nc = k.nc;
  const int cx[2] = {ix, ixp}, cy[2] = {iy, iyp}, cz[2] = {iz, izp};
  const double wx[2] = {dex, ddx}, wy[2] = {dey, ddy}, wz[2] = {dez, ddz};
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int a = c & 1, b = (c >> 1) & 1, e = c >> 2;
    double w = dmul(dmul(wx[a], wy[b]), wz[e]);
    unsigned long long q = (unsigned long long)__double2ll_rn(dmul(w, FIX_ONE));
    long long node = (long long)cx[a] + nc * ((long long)cy[b] + nc * (long long)cz[e]);
    atomicAdd(&grid[node], q);
  }
}

// interpolation: rho in the reference's term order (main:1368-1383)
__global__ void k_cic_interp(const float4 *cube, long long n, CicConst k, const unsigned long long *grid,
                             double *rho) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = cube[i];
  unsigned idx = __float_as_uint(p.w) & PSOD_IDX_MASK;
  if (!in_cic_zone(p, k)) {
    rho[idx] = 0.0;
    return;
  }
  int ix, ixp, iy, iyp, iz, izp;
  double ddx, dex, ddy, dey, ddz, dez;
  cic_axis(p.x, k, 0, ix, ixp, ddx, dex);
  cic_axis(p.y, k, 1, iy, iyp, ddy, dey);
  cic_axis(p.z, k, 2, iz, izp, ddz, dez);
  const long long nc = k.nc;
  const int cx[2] = {ix, ixp}, cy[2] = {iy, iyp}, cz[2] = {iz, izp};
  const double wx[2] = {dex, ddx}, wy[2] = {dey, ddy}, wz[2] = {dez, ddz};
  double r = 0.0;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int a = c & 1, b = (c >> 1) & 1, e = c >> 2;
    long long node = (long long)cx[a] + nc * ((long long)cy[b] + nc * (long long)cz[e]);
    double g = dmul((double)(long long)grid[node], k.kc);
    r = dadd(r, dmul(dmul(dmul(g, wx[a]), wy[b]), wz[e]));
  }
  rho[idx] = r;
}

// Tile-fused CIC: one CTA owns a tile of up to CT^3 SOD cells, its fine cells
// [0, w) per axis (w = twice its cells).  It deposits into a shared-memory
// window of nodes [0, w] every particle that touches them -- those of the
// tile and of the adjacent fine cells, all filed in the tile's cells and a
// one-cell halo -- then interpolates rho for the particles of its fine cells.
// Every node they read receives all its contributions inside the window, so
// the integer node sums, and therefore rho, equal the global grid's exactly.
//
// Bound: latency inside a tile (a tile of a mean-density box holds 512
// particles: the range look-ups, the barriers and the shared atomics are its
// time, not HBM and not FP64), so what counts is how many tiles an SM holds
// and how few steps one takes.  A window of 17^3 nodes, not of the whole halo's
// 21^3, lets four CTAs run instead of three (64 registers a thread and 42 KB:
// both limits are four) and drops 27 % of the deposits; a
// tile of at most SPLIT_MAX particles adds each weight as two 20-bit halves
// with 32-bit atomics that return nothing; a tile without particles leaves at
// once, unless the load has a foreign-filed particle, which any tile may hold;
// a record number finds its range from a table (walking the ranges took
// 40 % of the instructions).  512^3 box: 17.0 -> 10.4 ms; one 4^3 zone of it,
// mostly empty tiles, without that particle 4.3 -> 2.1 ms; 150^3 (was the global
// grid) 0.44 -> 0.39 ms.
constexpr int CT = 8;             // SOD cells per tile side
constexpr int CW = 2 * CT + 1;    // window nodes per side
constexpr int CW3 = CW * CW * CW;
constexpr unsigned DEP_BATCH = 4;     // record loads in flight per thread in the deposit
constexpr unsigned SPLIT_MAX = 4095;  // particles whose 20-bit halves a 32-bit sum holds

constexpr int CRNG = 2 * (CT + 2) * (CT + 2);  // record ranges of a tile plus halo (two where x wraps)

// exclusive prefix of s_len[0..n) into s_pre[0..n], n <= 32 * 8, by warp 0
__device__ __forceinline__ void range_prefix(const unsigned *s_len, unsigned *s_pre, int n) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x, per = (n + 31) / 32, lo = lane * per;
  unsigned t = 0;
  for (int i = lo; i < min(n, lo + per); i++) t += s_len[i];
  unsigned x = t;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  unsigned run = x - t;
  for (int i = lo; i < min(n, lo + per); i++) {
    s_pre[i] = run;
    run += s_len[i];
  }
  if (lane == 31) s_pre[n] = x;
}

// Range of a record number: s_first[b] is the range holding record b << shift,
// so a look-up starts there and steps over the few ranges of one block (a
// strided walk over all ranges took most of the deposit's instructions).
constexpr unsigned NFIRST = 128;

__device__ __forceinline__ int first_shift(unsigned total) {
  int sh = 4;
  while ((total >> sh) >= NFIRST) sh++;
  return sh;
}

__device__ __forceinline__ void range_first(const unsigned *s_pre, int n, int sh, unsigned char *s_first) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const unsigned a = s_pre[t], e = s_pre[t + 1];
    for (unsigned b = (a + (1u << sh) - 1u) >> sh; (b << sh) < e; b++) s_first[b] = (unsigned char)t;
  }
}

__device__ __forceinline__ unsigned record_slot(const unsigned *s_rb, const unsigned *s_pre, const unsigned char *s_first,
                                                int sh, unsigned f) {
  int r = s_first[f >> sh];
  while (s_pre[r + 1] <= f) r++;
  return s_rb[r] + (f - s_pre[r]);
}

// ZONE: particles outside the zone with buffer are skipped (zone contexts;
// the test costs registers, so one-zone contexts run without it).
// RAGGED: nx is not a power of two (or the zone's corner no multiple of the
// cell), so a particle at a cell edge may be filed, by the rounding of its
// grid coordinate, in the cell beside the one its CIC coordinate lies in.  The
// tile holding its fine cell interpolates it, whatever cell lists it: every
// loaded record is looked at, not only those of the tile's own cells.
template <bool ZONE, bool RAGGED>
__global__ void __launch_bounds__(256, 4) k_cic_tile(const float4 *cube, const unsigned *cs, int nx, CicConst k,
                                                     double *rho, int *bad, unsigned quirk_pos) {
  extern __shared__ __align__(16) unsigned long long win[];
  unsigned *win32 = reinterpret_cast<unsigned *>(win);  // split sums: [low 20 bits | high 20 bits] of CW3 each
  __shared__ unsigned s_rb[CRNG], s_len[CRNG], s_pre[CRNG + 1];
  __shared__ unsigned char s_first[NFIRST];
  static_assert(CRNG <= 256, "a range number is a byte");
  const int ntile = (nx + CT - 1) / CT;
  const int x0 = (int)(blockIdx.x % (unsigned)ntile) * CT, y0 = (int)((blockIdx.x / (unsigned)ntile) % (unsigned)ntile) * CT,
            z0 = (int)(blockIdx.x / (unsigned)(ntile * ntile)) * CT;
  const int xe = min(x0 + CT, nx), ye = min(y0 + CT, nx), ze = min(z0 + CT, nx);
  const int wx_ = 2 * (xe - x0), wy_ = 2 * (ye - y0), wz_ = 2 * (ze - z0);  // fine cells; nodes 0..w
  const int nc = k.nc;
  const int ox = 2 * x0, oy = 2 * y0, oz = 2 * z0;
  auto rel = [&](int f, int o) {  // fine index from the tile's first, in [-1, nc - 2]
    int d = f - o;
    if (d < -1) d += nc;
    if (d > nc - 2) d -= nc;
    return d;
  };
  struct Pt {
    int fx, fy, fz;      // fine cell relative to the tile
    double wx[2], wy[2], wz[2];
  };
  auto locate = [&](const float4 &v, Pt &q) {
    int i0, i1;
    cic_axis(v.x, k, 0, i0, i1, q.wx[1], q.wx[0]);
    q.fx = rel(i0, ox);
    cic_axis(v.y, k, 1, i0, i1, q.wy[1], q.wy[0]);
    q.fy = rel(i0, oy);
    cic_axis(v.z, k, 2, i0, i1, q.wz[1], q.wz[0]);
    q.fz = rel(i0, oz);
  };
  const bool has_q = quirk_pos != 0xffffffffu;
  // the tile's own records; without any (and without the quirk particle,
  // which another cell's run may hold) there is nothing to do
  unsigned own = 0;
  for (int row = threadIdx.x; row < (ye - y0) * (ze - z0); row += blockDim.x) {
    const int yy = y0 + row % (ye - y0), zz = z0 + row / (ye - y0);
    const unsigned long long base = (unsigned long long)nx * ((unsigned)yy + (unsigned long long)nx * (unsigned)zz);
    const unsigned rb = cs[base + (unsigned)x0];
    unsigned len = cs[base + (unsigned)xe] - rb;
    if (len && rb + len - 1u == quirk_pos) len--;  // handled below, by its own fine cell
    own += len;
  }
  // (a ragged tile may interpolate records filed beside it: its halo counts)
  if (!RAGGED && !has_q && !__syncthreads_or(own != 0)) return;
  // record ranges of the rows of the tile plus halo; the particles are then
  // dealt to all threads of the CTA evenly, whatever their spread over rows
  const int ny = ye - y0 + 2, nrow = ny * (ze - z0 + 2);
  unsigned any = 0;
  for (int row = threadIdx.x; row < CRNG / 2; row += blockDim.x) {
    unsigned rb[2] = {0, 0}, len[2] = {0, 0};
    if (row < nrow) {
      const int yy = (y0 - 1 + row % ny + nx) % nx, zz = (z0 - 1 + row / ny + nx) % nx;
      const unsigned long long base = (unsigned long long)nx * ((unsigned)yy + (unsigned long long)nx * (unsigned)zz);
      const int xa = x0 - 1, xb = xe;  // inclusive, may wrap
      int pa[2] = {0, 0}, pb[2] = {-1, -1};
      if (xa < 0) { pa[0] = xa + nx; pb[0] = nx - 1; pa[1] = 0; pb[1] = xb; }
      else if (xb >= nx) { pa[0] = xa; pb[0] = nx - 1; pa[1] = 0; pb[1] = xb - nx; }
      else { pa[0] = xa; pb[0] = xb; }
      for (int q = 0; q < 2; q++)
        if (pb[q] >= pa[q]) {
          rb[q] = cs[base + (unsigned)pa[q]];
          len[q] = cs[base + (unsigned)pb[q] + 1] - rb[q];
          // the quirk particle is the cube's last record, at the end of its listed cell's run
          if (len[q] && rb[q] + len[q] - 1u == quirk_pos) len[q]--;
        }
    }
    for (int q = 0; q < 2; q++) {
      s_rb[2 * row + q] = rb[q];
      s_len[2 * row + q] = len[q];
      any |= len[q];
    }
  }
  if (!__syncthreads_or(any != 0) && !has_q) return;
  for (int i = threadIdx.x; i < CW3; i += blockDim.x) win[i] = 0ull;
  range_prefix(s_len, s_pre, CRNG);
  __syncthreads();
  const unsigned total = s_pre[CRNG];
  const bool split = total < SPLIT_MAX;  // the quirk particle makes one more
  // quantised weight: (w 2^40) rounded to an integer; 2^40 goes into one axis
  // weight (an exact scaling), and adding 1.5 2^52 leaves the rounded integer
  // in the low bits
  auto quant = [&](double w) {
    return (unsigned long long)(__double_as_longlong(dadd(w, 6755399441055744.0)) - 0x4338000000000000ll);
  };
  auto node = [&](const Pt &q, int c) { return (q.fx + (c & 1)) + CW * ((q.fy + ((c >> 1) & 1)) + CW * (q.fz + (c >> 2))); };
  auto touches = [&](const Pt &q, int c) {
    const int a = q.fx + (c & 1), b = q.fy + ((c >> 1) & 1), e = q.fz + (c >> 2);
    return a >= 0 && a <= wx_ && b >= 0 && b <= wy_ && e >= 0 && e <= wz_;
  };
  auto deposit_split = [&](const float4 &v) {
    if (ZONE && !in_cic_zone(v, k)) return;
    Pt q;
    locate(v, q);
    if (q.fx > wx_ || q.fy > wy_ || q.fz > wz_) return;
    const double wx[2] = {dmul(q.wx[0], FIX_ONE), dmul(q.wx[1], FIX_ONE)};
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if (!touches(q, c)) continue;
      const unsigned long long w = quant(dmul(dmul(wx[c & 1], q.wy[(c >> 1) & 1]), q.wz[c >> 2]));
      const int at = node(q, c);
      atomicAdd(&win32[at], (unsigned)w & 0xfffffu);
      atomicAdd(&win32[CW3 + at], (unsigned)(w >> 20));
    }
  };
  int sh = first_shift(total);
  if (split) {
    range_first(s_pre, CRNG, sh, s_first);
    __syncthreads();
    for (unsigned f = threadIdx.x; f < total; f += 2 * blockDim.x) {
      const unsigned g = f + blockDim.x;
      const float4 va = cube[record_slot(s_rb, s_pre, s_first, sh, f)];
      const float4 vb = g < total ? cube[record_slot(s_rb, s_pre, s_first, sh, g)] : va;
      deposit_split(va);
      if (g < total) deposit_split(vb);
    }
  } else {
    // Each thread deposits one contiguous share of the tile's particles
    // (all threads busy, whatever the tile's count).  Dense cells are
    // sub-cell ordered, so consecutive particles mostly share a fine cell
    // and its 8 nodes: their fixed-point weights are summed in registers and
    // written with one atomic per node when the fine cell changes (integer
    // sums, so the grid is the same).  Records are loaded DEP_BATCH at a
    // time before any is used.
    const unsigned per = (total + blockDim.x - 1) / blockDim.x;
    const unsigned f0 = min(total, threadIdx.x * per), f1 = min(total, f0 + per);
    int r = 0;  // last range with s_pre[r] <= f0
    {
      int hi = CRNG;
      while (hi - r > 1) {
        const int mid = (r + hi) >> 1;
        if (s_pre[mid] <= f0) r = mid;
        else hi = mid;
      }
    }
    unsigned long long acc[8];
    Pt run;  // fine cell of the accumulated run
    run.fx = -2;
    auto flush = [&]() {
      if (run.fx < -1) return;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (touches(run, c) && acc[c]) atomicAdd(&win[node(run, c)], acc[c]);
      run.fx = -2;
    };
    for (unsigned fb = f0; fb < f1; fb += DEP_BATCH) {
      float4 vb[DEP_BATCH];
#pragma unroll
      for (unsigned u = 0; u < DEP_BATCH; u++) {
        const unsigned f = fb + u;
        if (f < f1) {
          while (s_pre[r + 1] <= f) r++;
          vb[u] = cube[s_rb[r] + (f - s_pre[r])];
        }
      }
#pragma unroll
      for (unsigned u = 0; u < DEP_BATCH; u++) {
        if (fb + u >= f1) break;
        if (ZONE && !in_cic_zone(vb[u], k)) continue;
        Pt q;
        locate(vb[u], q);
        if (q.fx > wx_ || q.fy > wy_ || q.fz > wz_) continue;
        if (q.fx != run.fx || q.fy != run.fy || q.fz != run.fz) {
          flush();
          run.fx = q.fx;
          run.fy = q.fy;
          run.fz = q.fz;
#pragma unroll
          for (int c = 0; c < 8; c++) acc[c] = 0ull;
        }
        const double wx[2] = {dmul(q.wx[0], FIX_ONE), dmul(q.wx[1], FIX_ONE)};
#pragma unroll
        for (int c = 0; c < 8; c++) acc[c] += quant(dmul(dmul(wx[c & 1], q.wy[(c >> 1) & 1]), q.wz[c >> 2]));
      }
    }
    flush();
  }
  // The run scan files a single particle of the last cell under the
  // previous cell's run (the linked-list quirk), which may lie in another
  // tile.  Its CIC weights belong to its own cell: every tile it touches
  // deposits it, and the tile holding its fine cell interpolates it.
  float4 vq = make_float4(0.f, 0.f, 0.f, 0.f);
  Pt pq;
  bool own_q = false;
  if (has_q && threadIdx.x == 0) {
    vq = cube[quirk_pos];
    locate(vq, pq);
    const bool sel = !(ZONE && !in_cic_zone(vq, k));
    own_q = pq.fx >= 0 && pq.fx < wx_ && pq.fy >= 0 && pq.fy < wy_ && pq.fz >= 0 && pq.fz < wz_;
    if (sel && pq.fx <= wx_ && pq.fy <= wy_ && pq.fz <= wz_) {
#pragma unroll
      for (int c = 0; c < 8; c++) {
        if (!touches(pq, c)) continue;
        const unsigned long long w =
            quant(dmul(dmul(dmul(pq.wx[c & 1], FIX_ONE), pq.wy[(c >> 1) & 1]), pq.wz[c >> 2]));
        if (split) {
          atomicAdd(&win32[node(pq, c)], (unsigned)w & 0xfffffu);
          atomicAdd(&win32[CW3 + node(pq, c)], (unsigned)(w >> 20));
        } else {
          atomicAdd(&win[node(pq, c)], w);
        }
      }
    }
  }
  __syncthreads();
  // the tile's particles: rho in the reference's term order (main:1368-1383)
  auto interp = [&](const float4 &v) {
    Pt q;
    locate(v, q);
    const bool mine = q.fx >= 0 && q.fx < wx_ && q.fy >= 0 && q.fy < wy_ && q.fz >= 0 && q.fz < wz_;
    if (!mine) {
      if (!RAGGED) atomicOr(bad, 1);
      return;
    }
    const unsigned idx = __float_as_uint(v.w) & PSOD_IDX_MASK;
    if (ZONE && !in_cic_zone(v, k)) {  // not selected by cicm1: rho stays 0
      rho[idx] = 0.0;
      return;
    }
    double rr = 0.0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int at = node(q, c);
      // a split sum is below 2^53: exact
      const double sum = split ? dadd(dmul((double)win32[CW3 + at], 1048576.0), (double)win32[at]) : (double)(long long)win[at];
      rr = dadd(rr, dmul(dmul(dmul(dmul(sum, k.kc), q.wx[c & 1]), q.wy[(c >> 1) & 1]), q.wz[c >> 2]));
    }
    rho[idx] = rr;
  };
  unsigned nown = total;
  if (!RAGGED) {
    // only the tile's own cells
    __syncthreads();
    for (int row = threadIdx.x; row < CT * CT; row += blockDim.x) {
      unsigned rb = 0, len = 0;
      if (row < (ye - y0) * (ze - z0)) {
        const int yy = y0 + row % (ye - y0), zz = z0 + row / (ye - y0);
        const unsigned long long base = (unsigned long long)nx * ((unsigned)yy + (unsigned long long)nx * (unsigned)zz);
        rb = cs[base + (unsigned)x0];
        len = cs[base + (unsigned)xe] - rb;
        if (len && rb + len - 1u == quirk_pos) len--;
      }
      s_rb[row] = rb;
      s_len[row] = len;
    }
    __syncthreads();
    range_prefix(s_len, s_pre, CT * CT);
    __syncthreads();
    nown = s_pre[CT * CT];
  }
  sh = first_shift(nown);
  range_first(s_pre, RAGGED ? CRNG : CT * CT, sh, s_first);
  __syncthreads();
  // two records per thread and step, both loaded before either is used
  for (unsigned fa = threadIdx.x; fa < nown; fa += 2 * blockDim.x) {
    const unsigned fb = fa + blockDim.x;
    const float4 va = cube[record_slot(s_rb, s_pre, s_first, sh, fa)];
    const float4 vb = fb < nown ? cube[record_slot(s_rb, s_pre, s_first, sh, fb)] : va;
    interp(va);
    if (fb < nown) interp(vb);
  }
  if (own_q) interp(vq);
}

__global__ void k_grid_to_double(const unsigned long long *grid, long long nnode, double kc, double *out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nnode) out[i] = dmul((double)(long long)grid[i], kc);
}

// ---------------------------------------------------------------------------
// seeds
// ---------------------------------------------------------------------------
// Seeds are the particles with 1/rho < 0.01 (main:1029), i.e. rho >= rho_seed,
// the smallest double whose quotient is below (the rounded quotient falls as
// rho grows).  Two passes over rho: the counts per tile of SEED_TILE particles
// with the extreme keys, then the compaction in input order.  (Flags, their
// scan over all particles and separate passes for the extremes moved 44 bytes a
// particle; these move 16.  256^3: 0.32 -> 0.10 ms.)
constexpr int SEED_TILE = 2048, SEED_PER = SEED_TILE / 256;

__global__ void __launch_bounds__(256) k_seed_count(const double *rho, long long n, double rho_seed, unsigned *count,
                                                    unsigned long long *seed_min, unsigned long long *other_min) {
  __shared__ unsigned s_cnt[8];
  __shared__ unsigned long long s_seed[8], s_other[8];
  const long long base = (long long)blockIdx.x * SEED_TILE;
  unsigned cnt = 0;
  double top = 0.0, below = 0.0;  // largest rho among the seeds and among the others
  bool any = false;
#pragma unroll
  for (int u = 0; u < SEED_PER; u++) {
    const long long i = base + u * 256 + threadIdx.x;
    if (i >= n) break;
    const double r = rho[i];
    if (r >= rho_seed) {
      cnt++;
      top = fmax(top, r);
    } else {
      below = any ? fmax(below, r) : r;
      any = true;
    }
  }
  // keys: bits of 1/rho, which falls as rho grows
  unsigned long long ks = cnt ? dbits(ddiv(1.0, top)) : ~0ull, ko = any ? dbits(ddiv(1.0, below)) : ~0ull;
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    const unsigned long long a = __shfl_down_sync(0xffffffffu, ks, o), b = __shfl_down_sync(0xffffffffu, ko, o);
    ks = a < ks ? a : ks;
    ko = b < ko ? b : ko;
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_cnt[w] = cnt;
    s_seed[w] = ks;
    s_other[w] = ko;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < 8; q++) {
      cnt += s_cnt[q];
      ks = s_seed[q] < ks ? s_seed[q] : ks;
      ko = s_other[q] < ko ? s_other[q] : ko;
    }
    count[blockIdx.x] = cnt;
    // the running minima only fall: a tile that does not lower them writes nothing
    if (ks < *(volatile unsigned long long *)seed_min) atomicMin(seed_min, ks);
    if (ko < *(volatile unsigned long long *)other_min) atomicMin(other_min, ko);
  }
}

// the seeds in input order with their keys: K = unsigned, the 32 bits of (bits
// - kmin) from bit `shift` up, or the full bits (shift 0, kmin 0); and the
// lowest index of a particle with the others' smallest key
template <typename K>
__global__ void __launch_bounds__(256) k_seed_compact(const double *rho, long long n, double rho_seed,
                                                      const unsigned *tile_pos, unsigned long long kmin, int shift,
                                                      double rho_other, unsigned long long other_min, unsigned *minidx,
                                                      K *keys, unsigned *vals) {
  __shared__ unsigned s_cnt[SEED_PER][8];
  const long long base = (long long)blockIdx.x * SEED_TILE;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double r[SEED_PER];
  unsigned m[SEED_PER];
#pragma unroll
  for (int u = 0; u < SEED_PER; u++) {
    const long long i = base + u * 256 + threadIdx.x;
    r[u] = i < n ? rho[i] : -1.0;
  }
#pragma unroll
  for (int u = 0; u < SEED_PER; u++) {
    m[u] = __ballot_sync(0xffffffffu, r[u] >= rho_seed);
    if (lane == 0) s_cnt[u][w] = (unsigned)__popc(m[u]);
    const long long i = base + u * 256 + threadIdx.x;
    if (i < n && !(r[u] >= rho_seed) && r[u] >= rho_other && dbits(ddiv(1.0, r[u])) == other_min)
      atomicMin(minidx, (unsigned)i);
  }
  __syncthreads();
  unsigned at = tile_pos[blockIdx.x];
#pragma unroll
  for (int u = 0; u < SEED_PER; u++) {
    unsigned mine = at;
    for (int q = 0; q < 8; q++) {
      if (q < w) mine += s_cnt[u][q];
      at += s_cnt[u][q];
    }
    if (r[u] >= rho_seed) {
      const unsigned o = mine + __popc(m[u] & ((1u << lane) - 1u));
      keys[o] = (K)((dbits(ddiv(1.0, r[u])) - kmin) >> shift);
      vals[o] = (unsigned)(base + u * 256 + threadIdx.x);
    }
  }
}

// After the sort on the truncated keys: each run of equal ones is put in (full
// key, input index) order by the thread at its start.  A run longer than
// TIE_MAX sets *redo (the caller sorts the full keys instead).
constexpr unsigned TIE_MAX = 64;

__global__ void k_seed_ties(const unsigned *key, unsigned *val, unsigned n, const double *rho, unsigned *redo) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 >= n) return;
  const unsigned k = key[i];
  if (key[i + 1] != k || (i > 0 && key[i - 1] == k)) return;
  unsigned e = i + 2;
  while (e < n && e - i <= TIE_MAX && key[e] == k) e++;
  if (e - i > TIE_MAX) {
    *redo = 1;
    return;
  }
  auto full = [&](unsigned v) { return dbits(ddiv(1.0, rho[v])); };
  for (unsigned a = i + 1; a < e; a++) {
    const unsigned v = val[a];
    const unsigned long long fk = full(v);
    unsigned b = a;
    while (b > i) {
      const unsigned u = val[b - 1];
      const unsigned long long fu = full(u);
      if (fu < fk || (fu == fk && u < v)) break;
      val[b] = u;
      b--;
    }
    val[b] = v;
  }
}

__global__ void k_widen_seeds(const unsigned *in, long long n, long long *out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (long long)in[i];
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ---------------------------------------------------------------------------
int stage_cellsort(psod_ctx *c, const float *dpos) {
  const long long n = c->n;
  const int nx = c->nx;
  c->ncell = (unsigned long long)nx * nx * nx;
  int st;
  unsigned *cell = nullptr, *count = nullptr, *slabs = nullptr;
  float4 *rec = nullptr;
  int *bad = nullptr;
  if ((st = scratch(c, SLOT_PART_U32, (size_t)n, &cell))) return st;
  if ((st = scratch(c, SLOT_SLAB_REC, (size_t)n, &rec))) return st;
  if ((st = scratch(c, SLOT_SLABS, 2 * SLAB_MAX, &slabs))) return st;
  if ((st = scratch(c, SLOT_CELL_U32, (size_t)c->ncell + 1, &count))) return st;
  if ((st = scratch(c, SLOT_LOAD_FLAGS, 2, &bad))) return st;
  if ((st = ensure(c, &c->d_cell_start, &c->cs_cap, (size_t)c->ncell + 1))) return st;
  if ((st = ensure(c, &c->d_cube, &c->cube_cap, (size_t)n))) return st;
  if ((st = ensure(c, &c->d_inv, &c->inv_cap, (size_t)n))) return st;
  PSOD_CUDA(c, cudaMemsetAsync(count, 0, sizeof(unsigned) * (c->ncell + 1), c->stream));
  PSOD_CUDA(c, cudaMemsetAsync(bad, 0, 2 * sizeof(int), c->stream));
  // xxmin*scale per axis (main:1565); slabs follow the z axis
  const double3 xs = make_double3(c->xxmin[0] * c->scale, c->xxmin[1] * c->scale, c->xxmin[2] * c->scale);
  // records grouped by slab first (see k_slab_scatter)
  const int nslab = std::min(nx, SLAB_MAX);
  PSOD_CUDA(c, cudaMemsetAsync(slabs, 0, sizeof(unsigned) * SLAB_MAX, c->stream));
  const unsigned ntile = nblk(n, SLAB_TILE);
  k_slab_count<<<ntile, SLAB_THREADS, 0, c->stream>>>(dpos, n, (float)nx, xs.z, nx, nslab, slabs, bad);
  k_slab_scan<<<1, 32, 0, c->stream>>>(slabs, nslab, slabs + SLAB_MAX);
  const int slab_smem = SLAB_TILE * (int)(sizeof(float4) + sizeof(unsigned short));
  PSOD_CUDA(c, cudaFuncSetAttribute(k_slab_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, slab_smem));
  k_slab_scatter<<<ntile, SLAB_THREADS, slab_smem, c->stream>>>(dpos, n, (float)nx, xs.z, nx, nslab, bad,
                                                                slabs + SLAB_MAX, rec, c->d_inv);
  k_cell_count<<<nblk(n, CELL_TILE), 256, 0, c->stream>>>(rec, n, (float)nx, xs, nx, bad, cell, count);
  if ((st = scan_u32(c, count, c->d_cell_start, (long long)c->ncell, true))) return st;
  unsigned *nbig = reinterpret_cast<unsigned *>(bad + 1);
  const long long ncell = (long long)c->ncell;
  // the dense cells are listed in the cube's memory, which the scatter fills
  // later, so that their tables are allocated for as many as there are
  unsigned *tab = nullptr, *bigcell = nullptr, *found = reinterpret_cast<unsigned *>(c->d_cube);
  static_assert(SUB_MIN * sizeof(float4) >= sizeof(unsigned), "room in the cube for the dense cells");
  k_mark_big<<<nblk(ncell, 256), 256, 0, c->stream>>>(count, c->ncell, nbig, found, c->d_cell_start);
  int hflags[2] = {0, 0};
  PSOD_CUDA(c, cudaMemcpyAsync(hflags, bad, sizeof(hflags), cudaMemcpyDeviceToHost, c->stream));
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  const int hbad = hflags[0];
  const unsigned hnbig = (unsigned)hflags[1];
  if (!hbad) {
    if ((st = scratch(c, SLOT_BIG_TAB, (size_t)hnbig * SUB_N + 1, &tab))) return st;
    if ((st = scratch(c, SLOT_BIG_CELL, (size_t)hnbig + 1, &bigcell))) return st;
    PSOD_CUDA(c, cudaMemcpyAsync(bigcell, found, sizeof(unsigned) * hnbig, cudaMemcpyDeviceToDevice, c->stream));
    PSOD_CUDA(c, cudaMemsetAsync(tab, 0, sizeof(unsigned) * (size_t)hnbig * SUB_N, c->stream));
    if (hnbig) {
      k_sub_count<<<nblk(n, CELL_TILE), 256, 0, c->stream>>>(rec, n, cell, count, (float)nx, xs, tab);
      k_sub_scan<<<nblk((long long)hnbig * 32, 256), 256, 0, c->stream>>>(tab, bigcell, hnbig, c->d_cell_start);
    }
    k_cell_scatter<<<nblk(n, CELL_TILE), 256, 0, c->stream>>>(rec, n, cell, count, tab, (float)nx, xs, c->d_cube);
    k_slot_of_input<<<ntile, SLAB_THREADS, 0, c->stream>>>(c->d_inv, n, cell);
    // rec is free once the scatter has read it
    if (hnbig)
      k_sub_fine<<<hnbig, 256, 0, c->stream>>>(c->d_cube, c->d_inv, rec, tab, bigcell, c->d_cell_start, (float)nx, xs);
    PSOD_CUDA(c, cudaGetLastError());
    PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  if (hbad) return set_err(c, PSOD_ERR_ARG, "particle positions must lie in [0,1] (box units)");

  // The reference's run scan (main:1591-1604) files a final cell holding a
  // single particle under the previous run.  Reproduce that by extending the
  // previous cell's range over it.
  c->has_quirk = 0;
  c->quirk_pos = 0xffffffffu;
  if (n >= 2) {
    float4 last2[2];
    PSOD_CUDA(c, cudaMemcpyAsync(last2, c->d_cube + (n - 2), sizeof(last2), cudaMemcpyDeviceToHost, c->stream));
    PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
    auto host_cell = [&](const float4 &p) {
      const float v[3] = {p.x, p.y, p.z};
      unsigned idx[3];
      for (int a = 0; a < 3; a++) {
        float xg = v[a] * (float)nx;  // exact product rounded once, as on the device
        int i = (int)std::floor((double)xg - (a == 0 ? xs.x : a == 1 ? xs.y : xs.z));
        if (i < 0) i += nx;
        if (i >= nx) i -= nx;
        idx[a] = (unsigned)i;
      }
      return idx[0] + (unsigned)nx * (idx[1] + (unsigned)nx * idx[2]);
    };
    unsigned ca = host_cell(last2[0]), cl = host_cell(last2[1]);
    if (ca != cl) {
      c->has_quirk = 1;
      c->quirk_pos = (unsigned)(n - 1);
      c->quirk_listed = ca;
      c->quirk_phys = cl;
      unsigned long long lo = (unsigned long long)ca + 1, hi = (unsigned long long)cl + 1;
      k_set_range<<<nblk((long long)(hi - lo), 256), 256, 0, c->stream>>>(c->d_cell_start, lo, hi, (unsigned)n);
    }
  }
  PSOD_CUDA(c, cudaGetLastError());
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  return PSOD_OK;
}

static CicConst make_cic_const(const psod_ctx *c) {
  CicConst k;
  k.nc = 2 * c->nx;                                 // main:667
  k.dx = 1.0 / (double)k.nc;                        // main:1126
  k.inv_dx = ((k.nc & (k.nc - 1)) == 0) ? (double)k.nc : 0.0;
  for (int a = 0; a < 3; a++) {
    k.xxmin[a] = c->xxmin[a];                       // main:665
    k.xxmax[a] = c->xxmax[a];                       // zone + buffer upper edge
  }
  // one zone covers the box: every particle is selected
  k.zone_test = c->nxcpu > 1 ? 1 : 0;
  const double vol = (k.dx * k.dx) * k.dx;          // main:1263
  k.kc = ((double)c->mpf / FIX_ONE) / vol;
  return k;
}

int stage_cic(psod_ctx *c, double *grid_out) {
  CicConst k = make_cic_const(c);
  const long long nnode = (long long)k.nc * k.nc * k.nc;
  int st;
  if (!c->d_rho || c->rho_cap < c->n) {
    if ((st = dalloc(c, &c->d_rho, (size_t)c->n))) return st;
    c->rho_cap = c->n;
  }
  // fused tile path (no global grid); boxes of fewer than CT + 2 cells a side
  // would meet their own halo
  bool tiled = false;
  if (c->nx >= CT + 2) {
    int *bad = nullptr;
    if ((st = scratch(c, SLOT_CIC_FLAG, 1, &bad))) return st;
    PSOD_CUDA(c, cudaMemsetAsync(bad, 0, sizeof(int), c->stream));
    const int smem = CW3 * (int)sizeof(unsigned long long);
    const int nt = (c->nx + CT - 1) / CT;
    const unsigned ntiles = (unsigned)nt * (unsigned)nt * (unsigned)nt;
    const unsigned qpos = c->has_quirk ? c->quirk_pos : 0xffffffffu;
    auto launch = [&](auto *kern) -> int {
      PSOD_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      kern<<<ntiles, 256, smem, c->stream>>>(c->d_cube, c->d_cell_start, c->nx, k, c->d_rho, bad, qpos);
      return PSOD_OK;
    };
    if ((st = k.zone_test ? launch(k_cic_tile<true, true>)
                          : (k.inv_dx != 0.0 ? launch(k_cic_tile<false, false>) : launch(k_cic_tile<false, true>))))
      return st;
    int hbad = 0;
    PSOD_CUDA(c, cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
    tiled = (hbad == 0);
  }
  if (!tiled || grid_out) {
    if ((st = dalloc(c, &c->d_grid, (size_t)nnode))) return st;
    PSOD_CUDA(c, cudaMemsetAsync(c->d_grid, 0, sizeof(unsigned long long) * nnode, c->stream));
    k_cic_deposit<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->d_cube, c->n, k, c->d_grid);
    if (!tiled) k_cic_interp<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->d_cube, c->n, k, c->d_grid, c->d_rho);
  }
  c->cic_tiled = tiled;
  PSOD_CUDA(c, cudaGetLastError());
  if (grid_out) {
    double *tmp = nullptr;
    if (is_device_ptr(grid_out)) {
      tmp = grid_out;
    } else if ((st = dalloc(c, &tmp, (size_t)nnode))) {
      return st;
    }
    k_grid_to_double<<<nblk(nnode, 256), 256, 0, c->stream>>>(c->d_grid, nnode, k.kc, tmp);
    if (tmp != grid_out) {
      st = copy_out(c, grid_out, tmp, sizeof(double) * nnode);
      dfree(&tmp);
      if (st) return st;
    }
  }
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  dfree(&c->d_grid);
  c->cic_done = true;
  c->rho_done = true;
  return PSOD_OK;
}

int stage_cicm1(psod_ctx *c, double *rho_out) {
  if (!c->rho_done) return set_err(c, PSOD_ERR_STATE, "psod_cicm1 needs psod_cic first");
  if (rho_out) return copy_out(c, rho_out, c->d_rho, sizeof(double) * c->n);
  return PSOD_OK;
}

int stage_tri_cic(psod_ctx *c, int64_t *isort_out) {
  if (!c->rho_done) return set_err(c, PSOD_ERR_STATE, "psod_tri_cic needs psod_cic first");
  const long long n = c->n;
  int st;
  // the smallest rho whose 1/rho rounds below 0.01
  double rho_seed = 100.0;
  while (!(1.0 / rho_seed < 0.01)) rho_seed = std::nextafter(rho_seed, 1e300);
  while (1.0 / std::nextafter(rho_seed, 0.0) < 0.01) rho_seed = std::nextafter(rho_seed, 0.0);
  unsigned *tiles = nullptr;
  unsigned long long *mins = nullptr;  // smallest key of the seeds, of the others; index of the latter, tie flag
  const long long ntile = nblk(n, SEED_TILE);
  if ((st = scratch(c, SLOT_PART_U32, (size_t)std::max<long long>(n, ntile + 1), &tiles))) return st;
  if ((st = scratch(c, SLOT_TRI_MIN, 3, &mins))) return st;
  unsigned *minidx = reinterpret_cast<unsigned *>(mins + 2), *redo = minidx + 1;
  PSOD_CUDA(c, cudaMemsetAsync(mins, 0xff, 3 * sizeof(unsigned long long), c->stream));
  k_seed_count<<<(unsigned)ntile, 256, 0, c->stream>>>(c->d_rho, n, rho_seed, tiles, mins, mins + 1);
  if ((st = scan_u32(c, tiles, tiles, ntile, true))) return st;
  unsigned nd = 0;
  unsigned long long hm[2] = {0, 0};
  PSOD_CUDA(c, cudaMemcpyAsync(&nd, tiles + ntile, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
  PSOD_CUDA(c, cudaMemcpyAsync(hm, mins, sizeof(hm), cudaMemcpyDeviceToHost, c->stream));
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  const bool has_extra = hm[1] != ~0ull;
  const long long nseed = (long long)nd + (has_extra ? 1 : 0);
  // densities that can have the others' smallest key
  double rho_other = 0.0;
  if (has_extra) {
    double pd;
    memcpy(&pd, &hm[1], sizeof(pd));
    rho_other = (1.0 / pd) * (1.0 - 1e-14);
  }
  if ((st = scratch(c, SLOT_SEED_IDX, (size_t)nseed + 1, &c->d_seed_idx))) return st;
  // Seeds arrive in input order; a stable sort on 1/rho leaves ties in input
  // order.  The keys are sorted by their top 32 varying bits (four digit passes
  // of 8 bytes a seed instead of seven of 12), then the few equal ones are put
  // in full order.
  const double edge = 0.01;
  unsigned long long kmax;
  memcpy(&kmax, &edge, sizeof(kmax));
  int shift = 0;
  while (nd && ((kmax - hm[0]) >> shift) > 0xffffffffull) shift++;
  unsigned *keys = nullptr;
  if ((st = scratch(c, SLOT_TRI_KEYS, (size_t)nd + 1, &keys))) return st;
  k_seed_compact<unsigned><<<(unsigned)ntile, 256, 0, c->stream>>>(c->d_rho, n, rho_seed, tiles, nd ? hm[0] : 0ull, shift,
                                                                   rho_other, hm[1], minidx, keys, c->d_seed_idx);
  if ((st = radix_sort_u32(c, keys, c->d_seed_idx, (long long)nd, 32))) return st;
  PSOD_CUDA(c, cudaMemsetAsync(redo, 0, sizeof(unsigned), c->stream));
  if (nd > 1 && shift > 0) k_seed_ties<<<nblk(nd, 256), 256, 0, c->stream>>>(keys, c->d_seed_idx, nd, c->d_rho, redo);
  unsigned hredo = 0;
  PSOD_CUDA(c, cudaMemcpyAsync(&hredo, redo, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  if (hredo) {
    // long runs of nearly equal densities: sort the full keys
    unsigned long long *keys64 = nullptr;
    if ((st = scratch(c, SLOT_TRI_KEYS, (size_t)nd + 1, &keys64))) return st;
    k_seed_compact<unsigned long long><<<(unsigned)ntile, 256, 0, c->stream>>>(
        c->d_rho, n, rho_seed, tiles, 0ull, 0, rho_other, hm[1], minidx, keys64, c->d_seed_idx);
    if ((st = radix_sort_u64(c, keys64, c->d_seed_idx, (long long)nd, 64))) return st;
  }
  if (has_extra)
    PSOD_CUDA(c, cudaMemcpyAsync(c->d_seed_idx + nd, minidx, sizeof(unsigned), cudaMemcpyDeviceToDevice, c->stream));
  PSOD_CUDA(c, cudaGetLastError());
  PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  c->nseed_dense = nd;
  c->npart_new = nseed;  // main:1032 (clamped to n when every particle is dense)
  if (isort_out && nseed > 0) {
    // widened on the device (through host vectors a 256^3 box took 13 ms of its
    // 22; the kernel takes 20 us): in place where the destination is this
    // device's memory, else in pieces through the tile counts' slot, which are
    // read by now
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, isort_out) == cudaSuccess;
    if (!known) cudaGetLastError();
    const bool here = known && reinterpret_cast<uintptr_t>(isort_out) % sizeof(int64_t) == 0 &&
                      (at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == c->device));
    long long *stage = here ? reinterpret_cast<long long *>(isort_out) : reinterpret_cast<long long *>(tiles);
    const long long piece = here ? nseed : std::max<long long>(n, ntile + 1) / 2;
    for (long long i = 0; i < nseed; i += piece) {
      const long long m = std::min(piece, nseed - i);
      k_widen_seeds<<<nblk(m, 256), 256, 0, c->stream>>>(c->d_seed_idx + i, m, stage);
      PSOD_CUDA(c, cudaGetLastError());
      if (!here && (st = copy_out(c, isort_out + i, stage, sizeof(int64_t) * m))) return st;
    }
    PSOD_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  c->seeds_done = true;
  return PSOD_OK;
}

}  // namespace psod
