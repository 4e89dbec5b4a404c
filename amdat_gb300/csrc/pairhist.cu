// Pair histograms: the radial distribution function's per-frame pair loop
// (Radial_Distribution_Function::listkernel2 + bin,
// src/radial_distribution_function.cpp:233-253) and the distinct van Hove
// pair loop over time pairs (Van_Hove_Distinct::listkernel2,
// src/van_hove_distinct.cpp:200-213, with the distance the reference meant to
// bin: the minimum-image |r_j(t1) - r_i(t0)|).
//
// Every bin is the reference's FP32 chain exactly - Coordinate::length_unwrapped
// (src/coordinate.cpp:126-137): per axis d = r_j - r_i, m = min(|d|, L - |d|);
// length = sqrtf((mx*mx + my*my) + mz*mz); bin = int(length / bin_size) - with
// correctly rounded, uncontracted operations, so the integer counts equal the
// reference's bit for bit.  A pair's bin is first estimated (contracted square sum,
// hardware square root, reciprocal bin size: within 1e-6 relative of the exact
// quotient) and counted at once unless the estimate lies within its error bound of a
// bin edge; those pairs (about one in a thousand) take the correctly rounded chain.
// Pairs whose squared length is safely beyond the last bin are dropped before that.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <utility>
#include <vector>

#include "engine.h"
#include "f32x2.cuh"

namespace amdat {

constexpr int PH_THREADS = 256;
constexpr int PH_WARPS = PH_THREADS / 32;
constexpr int PH_JT = 1024;  // list-2 members staged at a time

struct PHList {
  int32_t n;
  int32_t first;
  const int32_t* idx;
};

static PHList phview(const ListEntry& e) {
  return PHList{e.n, e.first, e.contiguous ? nullptr : e.idx.ptr};
}

__device__ __forceinline__ int member(const PHList& l, int a) {
  return l.idx ? l.idx[a] : l.first + a;
}

__device__ __forceinline__ float min_image(float d, float L) {
  const float a = fabsf(d);
  const float b = __fsub_rn(L, a);
  return a < b ? a : b;
}

struct PHParams {
  const float* w;
  int64_t n_pad;
  PHList l1, l2;
  const int32_t* frame_a;  // [n_rows] frame of list-1 positions
  const int32_t* frame_b;  // [n_rows] frame of list-2 positions
  const int32_t* row_of;   // [n_rows] output row (frame index or gap)
  float3 box;
  float bin_size;
  float inv_bin;  // 1 / bin_size (the bin estimate)
  float lim;      // 1/2 - the estimate's error bound, in bins
  float s2_cut;
  int32_t n_bins;
  unsigned long long* counts;  // [rows][n_bins]
};

// the reference's chain of one pair, for estimates near a bin edge
__device__ __noinline__ int exact_bin(float dx, float dy, float dz, float3 box, float bin_size) {
  const float mx = min_image(dx, box.x), my = min_image(dy, box.y), mz = min_image(dz, box.z);
  const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(mx, mx), __fmul_rn(my, my)), __fmul_rn(mz, mz));
  return (int)__fdiv_rn(__fsqrt_rn(s2), bin_size);
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two pairs at once (packed FP32): minimum-image square sums s and bin estimates
// x = sqrt(s) * inv_bin - 1/2, rounded to integers by adding 1.5 * 2^23: the low bits of
// y hold the bin (PH_MAGIC_BITS + bin), r = x - bin is in [-1/2, 1/2] and its ends are
// the bin's edges.
constexpr float PH_MAGIC = 12582912.0f;
constexpr uint32_t PH_MAGIC_BITS = 0x4B400000u;
__device__ __forceinline__ void pair_estimate2(const PHParams& p, uint64_t dx, uint64_t dy, uint64_t dz, float* s,
                                               float* y, float* r) {
  const uint64_t d[3] = {dx, dy, dz};
  const float L[3] = {p.box.x, p.box.y, p.box.z};
  uint64_t s2 = 0ull;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float d0, d1;
    upk2(d[a], d0, d1);
    const float m0 = fminf(fabsf(d0), __fsub_rn(L[a], fabsf(d0)));
    const float m1 = fminf(fabsf(d1), __fsub_rn(L[a], fabsf(d1)));
    const uint64_t m = pk2(m0, m1);
    s2 = a == 0 ? mul2(m, m) : fma2(m, m, s2);
  }
  upk2(s2, s[0], s[1]);
  const uint64_t magic = pk2(PH_MAGIC, PH_MAGIC);
  const uint64_t x2 = fma2(pk2(sqrt_approx(s[0]), sqrt_approx(s[1])), pk2(p.inv_bin, p.inv_bin), pk2(-0.5f, -0.5f));
  const uint64_t y2 = add2(x2, magic);
  upk2(sub2(x2, sub2(y2, magic)), r[0], r[1]);
  upk2(y2, y[0], y[1]);
}

// counts a pair with s < cut into the slot its estimate names; hist is the histogram's
// shared-memory address less 4 * PH_MAGIC_BITS.  Predicated, not branched around: most
// warps have lanes on both sides.
__device__ __forceinline__ void count_if(float s, float cut, float y, uint32_t hist, uint32_t inc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b32 a;\n\t"
      "setp.lt.f32 p, %0, %1;\n\t"
      "shl.b32 a, %2, 2;\n\t"
      "add.u32 a, a, %3;\n\t"
      "@p red.shared.add.u32 [a], %4;\n\t}"
      :: "f"(s), "f"(cut), "r"(__float_as_uint(y)), "r"(hist), "r"(inc));
}

// how an atom's own pair is left out
enum { PH_SELF_ZERO, PH_SELF_IDS, PH_SELF_LATER };  // one frame: the pair at zero distance; by index; by the caller

// One list-1 member (x, y, z duplicated in packed pairs) against the four staged list-2
// members at sx[0..3], ...: every pair within the cut is counted into its estimated
// slot, then the counts of estimates within their error bound of a bin edge are put
// right by the exact chain.
template <int SELF>
__device__ __forceinline__ void count4(const PHParams& p, uint64_t xi, uint64_t yi, uint64_t zi, int ai, float4 X, float4 Y,
                                       float4 Z, const float* sx, const float* sy, const float* sz, const int* sid,
                                       uint32_t hist, unsigned int* whist, uint32_t inc) {
  float s[4], y[4], r[4];
  pair_estimate2(p, sub2(pk2(X.x, X.y), xi), sub2(pk2(Y.x, Y.y), yi), sub2(pk2(Z.x, Z.y), zi), s, y, r);
  pair_estimate2(p, sub2(pk2(X.z, X.w), xi), sub2(pk2(Y.z, Y.w), yi), sub2(pk2(Z.z, Z.w), zi), s + 2, y + 2, r + 2);
  if (SELF == PH_SELF_IDS) {
    const int4 id = *reinterpret_cast<const int4*>(sid);
    const float nan = __int_as_float(0x7fffffff);
    if (id.x == ai) s[0] = nan;
    if (id.y == ai) s[1] = nan;
    if (id.z == ai) s[2] = nan;
    if (id.w == ai) s[3] = nan;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) count_if(s[e], p.s2_cut, y[e], hist, inc);
  if (fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fmaxf(fabsf(r[2]), fabsf(r[3]))) >= p.lim) {
    const float xs = __uint_as_float((uint32_t)xi), ys = __uint_as_float((uint32_t)yi), zs = __uint_as_float((uint32_t)zi);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (!(s[e] < p.s2_cut) || fabsf(r[e]) < p.lim) continue;
      const int est = (int)(__float_as_uint(y[e]) - PH_MAGIC_BITS);
      const int b = exact_bin(__fsub_rn(sx[e], xs), __fsub_rn(sy[e], ys), __fsub_rn(sz[e], zs), p.box, p.bin_size);
      const bool self = SELF == PH_SELF_ZERO && sid[e] == ai;
      if (b == est && !self) continue;
      atomicSub(whist + est, inc);
      if (!self && b >= 0 && b < p.n_bins) atomicAdd(whist + b, inc);
    }
  }
}

// a block's per-warp histograms added to the row's counts
__device__ __forceinline__ void flush_counts(const PHParams& p, const unsigned int* hist, int row) {
  unsigned long long* dst = p.counts + (int64_t)row * p.n_bins;
  for (int b = threadIdx.x; b < p.n_bins; b += PH_THREADS) {
    unsigned long long s = 0;
    for (int w = 0; w < PH_WARPS; ++w) s += hist[w * (p.n_bins + 1) + b];
    if (s) atomicAdd(dst + b, s);
  }
}

// one unit of the all-pairs pass: members [i0, i0 + 256 I) of list 1 against
// members [j0, j1) of list 2, each pair counted inc times
struct PHUnit {
  int32_t i0, j0, j1, inc;
};

// All-pairs pass.  A thread holds I members of list 1 in registers; list 2 streams
// through shared memory as planes, so one 16-byte load per axis brings four members
// for 4 I pairs.  Units are rectangles, so the work per block is even; in the
// symmetric pass (one list, one frame) the squares on the diagonal take every ordered
// pair once and the rectangles above it count twice (|d| is symmetric to the bit).
// Bound: instruction issue, 23 per pair and warp at 69 % of the issue slots; the
// histogram's shared-memory atomics take 2.5 wavefronts per 32 pairs (half the pairs in
// range).  g(r) of 64,000 atoms to half the box, 50 frames: 70.6 ms, against 163 ms with
// 35 instructions per pair (scalar chain, a branch around every count) over blocks of a
// triangle.
template <int I, int SELF>
__global__ void __launch_bounds__(PH_THREADS)
    pair_hist_kernel(PHParams p, const PHUnit* __restrict__ units) {
  extern __shared__ unsigned int sh_hist[];  // [8 warps][n_bins + 1], the last slot past the end
  __shared__ __align__(16) float sx[PH_JT], sy[PH_JT], sz[PH_JT];
  __shared__ __align__(16) int sid[PH_JT];
  const PHUnit U = units[blockIdx.x];
  const int q = blockIdx.y, nb1 = p.n_bins + 1;
  const float* A = p.w + (int64_t)p.frame_a[q] * 3 * p.n_pad;
  const float* B = p.w + (int64_t)p.frame_b[q] * 3 * p.n_pad;
  unsigned int* whist = sh_hist + (threadIdx.x >> 5) * nb1;
  const uint32_t hist = (uint32_t)__cvta_generic_to_shared(whist) - 4u * PH_MAGIC_BITS;
  for (int b = threadIdx.x; b < PH_WARPS * nb1; b += PH_THREADS) sh_hist[b] = 0u;
  const float nan = __int_as_float(0x7fffffff);  // members past the end: never within the cut
  uint64_t xi[I], yi[I], zi[I];
  int ai[I];
#pragma unroll
  for (int k = 0; k < I; ++k) {
    const int i = U.i0 + k * PH_THREADS + threadIdx.x;
    const bool live = i < p.l1.n;
    ai[k] = live ? member(p.l1, i) : -1;
    const float x = live ? A[ai[k]] : nan, y = live ? A[p.n_pad + ai[k]] : nan, z = live ? A[2 * p.n_pad + ai[k]] : nan;
    xi[k] = pk2(x, x), yi[k] = pk2(y, y), zi[k] = pk2(z, z);
  }
  for (int jt = U.j0; jt < U.j1; jt += PH_JT) {
    const int nj = min(PH_JT, U.j1 - jt);
    __syncthreads();
    for (int t = threadIdx.x; t < ((nj + 3) & ~3); t += PH_THREADS) {
      const bool live = t < nj;
      const int aj = live ? member(p.l2, jt + t) : -1;
      sx[t] = live ? B[aj] : nan;
      sy[t] = live ? B[p.n_pad + aj] : nan;
      sz[t] = live ? B[2 * p.n_pad + aj] : nan;
      sid[t] = aj;
    }
    __syncthreads();
    for (int t = 0; t < nj; t += 4) {
      const float4 X = *reinterpret_cast<const float4*>(sx + t), Y = *reinterpret_cast<const float4*>(sy + t),
                   Z = *reinterpret_cast<const float4*>(sz + t);
#pragma unroll
      for (int k = 0; k < I; ++k)
        count4<SELF>(p, xi[k], yi[k], zi[k], ai[k], X, Y, Z, sx + t, sy + t, sz + t, sid + t, hist, whist, (uint32_t)U.inc);
    }
  }
  __syncthreads();
  flush_counts(p, sh_hist, p.row_of[q]);
}

// ---------------------------------------------------------------------------
// cell pass for short-range ordered pair loops (the distinct van Hove pass and RDFs
// of two different lists), when every box axis holds at least three cutoffs.  Per
// frame each list's atoms are counted into cells, the counts scanned and the atoms
// scattered in cell order as (x, y, z, atom index bits).
// List 1 is ordered along pencils: (y, z) squares about as wide as 32 atoms' cube,
// filled with thin x cells, neighbouring pencils run in opposite directions; 32
// consecutive atoms then fill a compact box.  A warp takes such a group.
// List 2 is ordered in narrower pencils of x cells.  Of every pencil whose distance to
// the group's bounding box is within the cutoff, the warp gathers the run of x cells
// the cutoff reaches, keeps the atoms within the cutoff of the box in shared memory, and
// each lane goes through them (count4).  A pair within the last bin's edge is visited
// exactly once, so the counts equal the all-pairs pass's.
// Bound: instruction issue, as the all-pairs pass; a visited pair in three or so is
// within the cutoff.  G_d of 64,000 atoms over 1226 time pairs to 5.0 in a box of 42.3:
// 93.7 ms; 118 ms with every atom of the runs visited; 331 ms with one atom per thread
// walking its own 27 cells of the cutoff's width.
// ---------------------------------------------------------------------------
struct PHGrid {
  int3 n;
  float3 lo, cell, inv;
  int32_t n_cells;
  int32_t snake;  // x runs back in every other row of cells, rows run back in every other layer
  float tol;      // atoms further than this outside the box flag the call
};

__device__ __forceinline__ int wrap_index(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// the cell of a coordinate; outside the box its image's (wrap) or the nearest one
__device__ __forceinline__ int ph_cell_axis(float x, float lo, float inv_cell, int n, bool wrap) {
  const int c = (int)floorf((x - lo) * inv_cell);
  return min(max(wrap ? wrap_index(c, n) : c, 0), n - 1);
}

// members of list l at frame frames[s] counted into the cells of slot s
__global__ void ph_cell_count_kernel(const float* __restrict__ w, int64_t n_pad, PHList l,
                                     const int32_t* __restrict__ frames, PHGrid g,
                                     int32_t* __restrict__ cell_of, int32_t* __restrict__ count, int32_t* __restrict__ out) {
  const int s = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= l.n) return;
  const float* P = w + (int64_t)frames[s] * 3 * n_pad;
  const int a = member(l, i);
  const float x = P[a], y = P[n_pad + a], z = P[2 * n_pad + a];
  // list 1 (snake) keeps an atom beside its neighbours, list 2 is looked up by image
  const bool wrap = !g.snake;
  int cx = ph_cell_axis(x, g.lo.x, g.inv.x, g.n.x, wrap), cy = ph_cell_axis(y, g.lo.y, g.inv.y, g.n.y, wrap);
  const int cz = ph_cell_axis(z, g.lo.z, g.inv.z, g.n.z, wrap);
  if (g.snake) {
    if (cz & 1) cy = g.n.y - 1 - cy;
    if ((cz * g.n.y + cy) & 1) cx = g.n.x - 1 - cx;
  }
  const int c = (cz * g.n.y + cy) * g.n.x + cx;
  cell_of[(int64_t)s * l.n + i] = c;
  atomicAdd(count + (int64_t)s * g.n_cells + c, 1);
  const float ex = fmaxf(g.lo.x - x, x - g.lo.x - g.cell.x * g.n.x), ey = fmaxf(g.lo.y - y, y - g.lo.y - g.cell.y * g.n.y),
              ez = fmaxf(g.lo.z - z, z - g.lo.z - g.cell.z * g.n.z);
  if (!(fmaxf(ex, fmaxf(ey, ez)) <= g.tol)) *out = 1;
}

// exclusive scan of one slot's cell counts (one block per slot) into start and
// the scatter cursors: four cells per thread, shuffle scans of a warp and of the warps
// (50,000 cells: 15 us; a scan over 1,024 cells at a time in shared memory, ten barriers
// each, 110)
constexpr int PS_THREADS = 1024, PS_ITEMS = 4;
__device__ __forceinline__ int32_t warp_scan(int32_t v, int lane) {  // inclusive
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t u = __shfl_up_sync(0xffffffffu, v, off);
    if (lane >= off) v += u;
  }
  return v;
}
__global__ void __launch_bounds__(PS_THREADS) ph_cell_scan_kernel(const int32_t* __restrict__ count, int32_t n_cells,
                                                                  int32_t* __restrict__ start, int32_t* __restrict__ cursor) {
  __shared__ int32_t s_warp[2][32];
  const int s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t* C = count + (int64_t)s * n_cells;
  int32_t* S = start + (int64_t)s * (n_cells + 1);
  int32_t* U = cursor + (int64_t)s * n_cells;
  int32_t carry = 0;
  for (int base = 0, it = 0; base < n_cells; base += PS_THREADS * PS_ITEMS, ++it) {
    const int i0 = base + PS_ITEMS * threadIdx.x;
    int32_t v[PS_ITEMS], sum = 0;
#pragma unroll
    for (int j = 0; j < PS_ITEMS; ++j) {
      v[j] = i0 + j < n_cells ? C[i0 + j] : 0;
      sum += v[j];
    }
    const int32_t incl = warp_scan(sum, lane);
    int32_t* T = s_warp[it & 1];  // written again after the next iteration's barrier
    if (lane == 31) T[warp] = incl;
    __syncthreads();
    const int32_t totals = warp_scan(T[lane], lane);  // every warp scans the warps' totals
    int32_t excl = carry + incl - sum + (warp ? __shfl_sync(0xffffffffu, totals, warp - 1) : 0);
    carry += __shfl_sync(0xffffffffu, totals, 31);
#pragma unroll
    for (int j = 0; j < PS_ITEMS; ++j)
      if (i0 + j < n_cells) {
        S[i0 + j] = excl;
        U[i0 + j] = excl;
        excl += v[j];
      }
  }
  if (threadIdx.x == 0) S[n_cells] = carry;
}

__global__ void ph_cell_scatter_kernel(const float* __restrict__ w, int64_t n_pad, PHList l,
                                       const int32_t* __restrict__ frames, int32_t n_cells,
                                       const int32_t* __restrict__ cell_of, int32_t* __restrict__ cursor,
                                       float4* __restrict__ pos) {
  const int s = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= l.n) return;
  const float* P = w + (int64_t)frames[s] * 3 * n_pad;
  const int a = member(l, i);
  const int k = atomicAdd(cursor + (int64_t)s * n_cells + cell_of[(int64_t)s * l.n + i], 1);
  pos[(int64_t)s * l.n + k] = make_float4(P[a], P[n_pad + a], P[2 * n_pad + a], __int_as_float(a));
}

// group minimum and maximum of a coordinate (lanes without an atom pass NaN)
__device__ __forceinline__ void warp_range(float v, float& lo, float& hi) {
  lo = hi = v;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
  }
}

constexpr int PG_TILE = 128;           // gathered list-2 members gone through at a time
constexpr int PG_BUF = PG_TILE + 32;

struct PHGroups {
  const float4* pos1;     // [slot][n1]: list-1 members in pencil order
  int32_t n1, per_warp;   // groups per warp
  const float4* pos2;     // [slot][n2]
  const int32_t* start2;  // [slot][n_cells + 1]
  int32_t n2;
  PHGrid g2;
  const int32_t* slot_a;  // slots of each row
  const int32_t* slot_b;
  float reach;            // cutoff with its margin
  int32_t same;           // one list: each atom's own pair is taken out at the end
  const int32_t* outside;  // set: some atom lies far outside the box, nothing is counted
};

template <int SELF>
__global__ void __launch_bounds__(PH_THREADS) pair_hist_groups_kernel(PHParams p, PHGroups G) {
  extern __shared__ unsigned int sh_hist[];  // [8 warps][n_bins + 1]
  __shared__ __align__(16) float sbuf[PH_WARPS][3][PG_BUF];
  __shared__ __align__(16) int sids[PH_WARPS][SELF == PH_SELF_IDS ? PG_BUF : 4];
  if (*G.outside) return;  // cell indexes would not wrap into the grid
  const int q = blockIdx.y, nb1 = p.n_bins + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned int* whist = sh_hist + warp * nb1;
  const uint32_t hist = (uint32_t)__cvta_generic_to_shared(whist) - 4u * PH_MAGIC_BITS;
  for (int b = threadIdx.x; b < PH_WARPS * nb1; b += PH_THREADS) sh_hist[b] = 0u;
  __syncthreads();
  const float4* P1 = G.pos1 + (int64_t)G.slot_a[q] * G.n1;
  const float4* P2 = G.pos2 + (int64_t)G.slot_b[q] * G.n2;
  const int32_t* S2 = G.start2 + (int64_t)G.slot_b[q] * (G.g2.n_cells + 1);
  const PHGrid& g = G.g2;
  const float nan = __int_as_float(0x7fffffff);
  float *bx = sbuf[warp][0], *by = sbuf[warp][1], *bz = sbuf[warp][2];
  int* bid = sids[warp];
  for (int gi = 0; gi < G.per_warp; ++gi) {
    const int i0 = 32 * ((blockIdx.x * G.per_warp + gi) * PH_WARPS + warp);
    if (i0 >= G.n1) break;
    const bool live = i0 + lane < G.n1;
    const float4 pi = live ? P1[i0 + lane] : make_float4(nan, nan, nan, __int_as_float(-1));
    const int ai = __float_as_int(pi.w);
    const uint64_t xi = pk2(pi.x, pi.x), yi = pk2(pi.y, pi.y), zi = pk2(pi.z, pi.z);
    // the group's box, relative to the periodic box's origin (as every length below that
    // only selects members: the origin may lie at any distance, and coordinates far from
    // zero round by more than the cutoff's margin)
    float x0, x1, y0, y1, z0, z1;
    warp_range(pi.x - g.lo.x, x0, x1);
    warp_range(pi.y - g.lo.y, y0, y1);
    warp_range(pi.z - g.lo.z, z0, z1);
    // the pencils the cutoff reaches (all of an axis once when it reaches around)
    int ya = (int)floorf((y0 - G.reach) * g.inv.y), ny = (int)floorf((y1 + G.reach) * g.inv.y) - ya + 1;
    int za = (int)floorf((z0 - G.reach) * g.inv.z), nz = (int)floorf((z1 + G.reach) * g.inv.z) - za + 1;
    const bool all_y = ny >= g.n.y, all_z = nz >= g.n.z;
    if (all_y) ya = 0, ny = g.n.y;
    if (all_z) za = 0, nz = g.n.z;
    // the box's centre as members' coordinates round, and its half edges from there
    const float xm = g.lo.x + 0.5f * (x0 + x1), ym = g.lo.y + 0.5f * (y0 + y1), zm = g.lo.z + 0.5f * (z0 + z1);
    const float xh = fmaxf(x1 - (xm - g.lo.x), xm - g.lo.x - x0), yh = fmaxf(y1 - (ym - g.lo.y), ym - g.lo.y - y0),
                zh = fmaxf(z1 - (zm - g.lo.z), zm - g.lo.z - z0);
    int cnt = 0;  // gathered members
    auto go = [&](int n) {  // lanes against the first n gathered members (a multiple of four)
      __syncwarp();
      for (int t = 0; t < n; t += 4)
        count4<SELF>(p, xi, yi, zi, ai, *reinterpret_cast<const float4*>(bx + t), *reinterpret_cast<const float4*>(by + t),
                     *reinterpret_cast<const float4*>(bz + t), bx + t, by + t, bz + t, bid + (SELF == PH_SELF_IDS ? t : 0),
                     hist, whist, 1u);
      __syncwarp();
    };
    auto gather = [&](int k0, int k1) {
      for (int k = k0; k < k1; k += 32) {
        // only members within reach of the group's box are kept
        const float4 c = k + lane < k1 ? __ldg(P2 + k + lane) : make_float4(nan, nan, nan, 0.f);
        const float gx = fmaxf(0.f, fabsf(min_image(c.x - xm, p.box.x)) - xh), gy = fmaxf(0.f, fabsf(min_image(c.y - ym, p.box.y)) - yh),
                    gz = fmaxf(0.f, fabsf(min_image(c.z - zm, p.box.z)) - zh);
        const bool keep = k + lane < k1 && fmaf(gz, gz, fmaf(gy, gy, gx * gx)) <= G.reach * G.reach;
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int at = cnt + __popc(kept & ((1u << lane) - 1u));
          bx[at] = c.x;
          by[at] = c.y;
          bz[at] = c.z;
          if (SELF == PH_SELF_IDS) bid[at] = __float_as_int(c.w);
        }
        cnt += __popc(kept);
        if (cnt >= PG_TILE) {
          go(PG_TILE);
          cnt -= PG_TILE;
          float cx = 0.f, cy = 0.f, cz = 0.f;
          int ci = 0;
          if (lane < cnt) {
            cx = bx[PG_TILE + lane], cy = by[PG_TILE + lane], cz = bz[PG_TILE + lane];
            if (SELF == PH_SELF_IDS) ci = bid[PG_TILE + lane];
            bx[lane] = cx, by[lane] = cy, bz[lane] = cz;
            if (SELF == PH_SELF_IDS) bid[lane] = ci;
          }
          __syncwarp();
        }
      }
    };
    for (int t0 = 0; t0 < ny * nz; t0 += 32) {
      // one pencil per lane: its run of cells, in two parts when it crosses the box's end
      int a0 = 0, a1 = 0, b0 = 0, b1 = 0;
      if (t0 + lane < ny * nz) {
        const int jz = za + (t0 + lane) / ny, jy = ya + (t0 + lane) % ny;
        const float fy = (float)jy * g.cell.y, fz = (float)jz * g.cell.z;
        const float gy = all_y ? 0.f : fmaxf(0.f, fmaxf(fy - y1, y0 - (fy + g.cell.y)));
        const float gz = all_z ? 0.f : fmaxf(0.f, fmaxf(fz - z1, z0 - (fz + g.cell.z)));
        const float rem = G.reach * G.reach - gy * gy - gz * gz;
        if (rem >= 0.f) {
          const float h = sqrtf(rem);
          const int32_t* S = S2 + (wrap_index(jz, g.n.z) * g.n.y + wrap_index(jy, g.n.y)) * g.n.x;
          const int xa = (int)floorf((x0 - h) * g.inv.x), nx = (int)floorf((x1 + h) * g.inv.x) - xa + 1;
          if (nx >= g.n.x) {
            a0 = S[0], a1 = S[g.n.x];
          } else {
            const int w = wrap_index(xa, g.n.x), e = w + nx;
            a0 = S[w], a1 = S[min(e, g.n.x)];
            if (e > g.n.x) b0 = S[0], b1 = S[e - g.n.x];
          }
        }
      }
      for (unsigned m = __ballot_sync(0xffffffffu, a1 > a0 || b1 > b0); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        gather(__shfl_sync(0xffffffffu, a0, src), __shfl_sync(0xffffffffu, a1, src));
        const int k0 = __shfl_sync(0xffffffffu, b0, src), k1 = __shfl_sync(0xffffffffu, b1, src);
        if (k1 > k0) gather(k0, k1);
      }
    }
    if (cnt & 3) {
      if (lane < 4 - (cnt & 3)) {
        bx[cnt + lane] = by[cnt + lane] = bz[cnt + lane] = nan;
        if (SELF == PH_SELF_IDS) bid[cnt + lane] = -1;
      }
      cnt = (cnt + 3) & ~3;
    }
    go(cnt);
    if (G.same && live) {
      // this atom's own pair was counted when it lies within the last bin
      const float* B = p.w + (int64_t)p.frame_b[q] * 3 * p.n_pad;
      const float dx = __fsub_rn(B[ai], pi.x), dy = __fsub_rn(B[p.n_pad + ai], pi.y), dz = __fsub_rn(B[2 * p.n_pad + ai], pi.z);
      const float mx = min_image(dx, p.box.x), my = min_image(dy, p.box.y), mz = min_image(dz, p.box.z);
      if (fmaf(mz, mz, fmaf(my, my, mx * mx)) < p.s2_cut) {
        const int b = exact_bin(dx, dy, dz, p.box, p.bin_size);
        if (b >= 0 && b < p.n_bins) atomicSub(whist + b, 1u);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  flush_counts(p, sh_hist, p.row_of[q]);
}

// The walk: list-1 members too sparse for compact groups (a few atoms of a solute, cutoffs
// below the atoms' spacing).  PARTS lanes per list-1 member go through the 27 cells around
// its own, cells at least as wide as the cutoff, a cell per lane at a time; every pair takes
// the exact chain.  Bound by the latency of its scattered loads.
struct PHWalk {
  const float4* pos1;     // [slot][n1] in cell order
  int32_t n1;
  const float4* pos2;     // [slot][n2]
  const int32_t* start2;  // [slot][n_cells + 1]
  int32_t n2;
  PHGrid g;
  const int32_t* slot_a;
  const int32_t* slot_b;
  const int32_t* outside;
};

template <int PARTS>
__global__ void __launch_bounds__(PH_THREADS) pair_hist_walk_kernel(PHParams p, PHWalk W) {
  extern __shared__ unsigned int sh_hist[];  // [8 warps][n_bins + 1]
  if (*W.outside) return;
  const int q = blockIdx.y, nb1 = p.n_bins + 1;
  unsigned int* whist = sh_hist + (threadIdx.x >> 5) * nb1;
  for (int b = threadIdx.x; b < PH_WARPS * nb1; b += PH_THREADS) sh_hist[b] = 0u;
  __syncthreads();
  const int i = blockIdx.x * (PH_THREADS / PARTS) + threadIdx.x / PARTS;
  if (i < W.n1) {
    const PHGrid& g = W.g;
    const float4 pi = W.pos1[(int64_t)W.slot_a[q] * W.n1 + i];
    const int32_t* S2 = W.start2 + (int64_t)W.slot_b[q] * (g.n_cells + 1);
    const float4* P2 = W.pos2 + (int64_t)W.slot_b[q] * W.n2;
    const int cx = ph_cell_axis(pi.x, g.lo.x, g.inv.x, g.n.x, true), cy = ph_cell_axis(pi.y, g.lo.y, g.inv.y, g.n.y, true),
              cz = ph_cell_axis(pi.z, g.lo.z, g.inv.z, g.n.z, true);
    for (int off = threadIdx.x % PARTS; off < 27; off += PARTS) {
      const int x = wrap_index(cx + off % 3 - 1, g.n.x), y = wrap_index(cy + off / 3 % 3 - 1, g.n.y),
                z = wrap_index(cz + off / 9 - 1, g.n.z);
      const int c = (z * g.n.y + y) * g.n.x + x;
      const int k1 = __ldg(S2 + c + 1);
      for (int k = __ldg(S2 + c); k < k1; ++k) {
        const float4 cj = __ldg(P2 + k);
        const float mx = min_image(__fsub_rn(cj.x, pi.x), p.box.x), my = min_image(__fsub_rn(cj.y, pi.y), p.box.y),
                    mz = min_image(__fsub_rn(cj.z, pi.z), p.box.z);
        const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(mx, mx), __fmul_rn(my, my)), __fmul_rn(mz, mz));
        if (s2 < p.s2_cut && __float_as_int(cj.w) != __float_as_int(pi.w)) {
          const int b = (int)__fdiv_rn(__fsqrt_rn(s2), p.bin_size);
          if (b < p.n_bins) atomicAdd(whist + b, 1u);
        }
      }
    }
  }
  __syncthreads();
  flush_counts(p, sh_hist, p.row_of[q]);
}

// cells of about edge_x x edge_yz x edge_yz over the box, at most 2^20
static PHGrid make_grid(amdat_ctx* ctx, double edge_x, double edge_yz, bool snake, float tol) {
  auto cells = [](double L, double e, int most) { return (int)std::min<double>(most, std::max(1.0, std::floor(L / e))); };
  PHGrid g;
  g.n = make_int3(cells(ctx->box[0], edge_x, 1024), cells(ctx->box[1], edge_yz, 1024), cells(ctx->box[2], edge_yz, 1024));
  while ((int64_t)g.n.x * g.n.y * g.n.z > (1 << 20)) {
    int& m = g.n.x >= g.n.y && g.n.x >= g.n.z ? g.n.x : (g.n.y >= g.n.z ? g.n.y : g.n.z);
    m = (m + 1) / 2;
  }
  g.n_cells = g.n.x * g.n.y * g.n.z;
  g.lo = make_float3(ctx->box_lo[0], ctx->box_lo[1], ctx->box_lo[2]);
  g.cell = make_float3(ctx->box[0] / g.n.x, ctx->box[1] / g.n.y, ctx->box[2] / g.n.z);
  g.inv = make_float3((float)g.n.x / ctx->box[0], (float)g.n.y / ctx->box[1], (float)g.n.z / ctx->box[2]);
  g.snake = snake ? 1 : 0;
  g.tol = tol;
  return g;
}

// units of the all-pairs pass, 256 I members by up to seg list-2 members: wide ones while
// they fill the chip six times over, then fewer members per thread and shorter segments
static std::vector<PHUnit> pair_units(const amdat_ctx* ctx, int n1, int n2, bool symmetric, int64_t n_q, int* per_thread) {
  const int64_t want = 6 * (int64_t)ctx->n_sm;
  auto count_units = [&](int I, int seg) {
    const int64_t ib = ceil_div(n1, 256 * I), js = ceil_div(n2, seg);
    return (symmetric ? (ib * js + ib) / 2 : ib * js) * n_q;
  };
  int I = 4, seg = 8192;
  while (seg > 1024 && count_units(I, seg) < want) seg /= 2;
  while (I > 1 && count_units(I, seg) < want) I /= 2;
  while (seg > 128 && count_units(I, seg) < want) seg /= 2;
  std::vector<PHUnit> units;
  for (int i0 = 0; i0 < n1; i0 += 256 * I) {
    const int i1 = std::min(n1, i0 + 256 * I);
    if (symmetric)
      for (int j = i0; j < i1; j += seg) units.push_back(PHUnit{i0, j, std::min(i1, j + seg), 1});
    for (int j = symmetric ? i1 : 0; j < n2; j += seg) units.push_back(PHUnit{i0, j, std::min(n2, j + seg), symmetric ? 2 : 1});
  }
  *per_thread = I;
  return units;
}

// Cell tables of all frames of both sides stay within this many bytes (AMDAT_PAIR_SCRATCH_MB);
// beyond, the rows run in batches of frames.
constexpr size_t PH_TABLE_BYTES = (size_t)4 << 30;

// rows [row0, row0 + rows) of the reordered row tables: their frames are the distinct frames
// f0[s] .. f0[s] + nf[s] of each side
struct PHBatch {
  int32_t f0[2], nf[2];
  size_t row0, rows;
};

static void run_pair_hist(amdat_ctx* ctx, const ListEntry& l1, const ListEntry& l2, bool symmetric,
                          const std::vector<int32_t>& fa, const std::vector<int32_t>& fb,
                          const std::vector<int32_t>& row, int32_t n_rows_out, float max_distance,
                          int32_t n_bins, int32_t out_flags, int64_t* counts) {
  AMDAT_REQUIRE(n_bins >= 1 && n_bins <= 4096, "n_bins must be in [1, 4096]");
  AMDAT_REQUIRE(max_distance > 0.0f, "max_distance must be positive");
  AMDAT_REQUIRE(counts != nullptr, "null output");
  const size_t n_q = fa.size();
  const size_t n_out = (size_t)n_rows_out * n_bins;
  const bool any = n_q && l1.n > 0 && l2.n > 0;
  AMDAT_REQUIRE(!any || n_q <= 65535, "at most 65535 frames or time pairs per call");
  // cell lists for the ordered pass when the box holds at least three cutoffs per axis
  const float cell_edge = (float)((double)max_distance * (1.0 + 1e-4));
  const int3 nc = make_int3((int)std::floor(ctx->box[0] / cell_edge), (int)std::floor(ctx->box[1] / cell_edge),
                            (int)std::floor(ctx->box[2] / cell_edge));
  const int64_t n_cells = (int64_t)nc.x * nc.y * nc.z;
  const char* pc = std::getenv("AMDAT_PAIR_CELLS");  // "off": the all-pairs pass
  const bool cells = !symmetric && any && l2.n >= 1024 && nc.x >= 3 && nc.y >= 3 && nc.z >= 3 &&
                     n_cells <= (1 << 20) && !(pc && std::strcmp(pc, "off") == 0);
  // the host's tables go to the device in one copy
  auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
  std::vector<unsigned char> host;
  auto table = [&](const auto& v) {
    const size_t at = host.size(), bytes = v.size() * sizeof(v[0]);
    host.resize(align(at + bytes));
    if (bytes) std::memcpy(host.data() + at, v.data(), bytes);
    return at;
  };
  std::vector<int32_t> qa = fa, qb = fb, qrow = row;  // the rows, in the batches' order
  std::vector<int32_t> fr[2], slot[2];  // the distinct frames of each side and each row's place among them
  size_t o_fr[2] = {0, 0}, o_slot[2] = {0, 0}, o_units = 0;
  std::vector<PHUnit> units;
  int per_thread = 1;
  std::vector<PHBatch> batches;
  const ListEntry* lists[2] = {&l1, &l2};
  PHGrid grid[2];
  bool walk = false;
  int lanes = 1;  // of the walk, per list-1 member
  const double edge = (double)std::max(ctx->box[0], std::max(ctx->box[1], ctx->box[2]));
  const bool same = &l1 == &l2;
  int sides = 2;
  if (cells) {
    // list 1: pencils as wide as the cube of 32 atoms, x cells an eighth of that (a quarter
    // leaves the groups longer: 2 % slower); list 2: pencils of half the cutoff (a third:
    // 5 % slower, more runs; the whole: 2 %), but wide enough for runs of about 16 atoms,
    // x cells of half a pencil or two atoms
    const double vol = (double)ctx->box[0] * ctx->box[1] * ctx->box[2];
    const double w1 = std::cbrt(32.0 * vol / l1.n), rho2 = l2.n / vol;
    const double f2 = std::max((double)max_distance / 2.0, std::sqrt(16.0 / (rho2 * (1.6 * max_distance + w1))));
    // wrapped coordinates need not lie in the box (read from a file so, or rounded there
    // from far unwrapped ones).  Up to an eighth of it the cells wrap and L - |d| is still
    // the distance to the nearest image; beyond, the all-pairs pass gives the chain's value
    const float tol = 0.125f * std::min(ctx->box[0], std::min(ctx->box[1], ctx->box[2]));
    grid[0] = make_grid(ctx, 0.125 * w1, w1, true, tol);
    grid[1] = make_grid(ctx, std::max(0.5 * f2, 2.0 / (f2 * f2 * rho2)), f2, false, tol);
    // The walk instead of the groups where these would gather far more members.  Gathered
    // for a group: the members of its box (as the cube of its atoms) widened by the cutoff.
    // Walked for an atom: the members of 27 cells, each cell costing as much as 0.7 of them.
    // G_d of n1 atoms to n2, groups / walk: 10 to 64,000 (r 3.0, 12 frames) 3,677 / 122 us
    // (428 with a thread per atom, as before the groups), 1,000 to 200,000 (2.0, 2 frames)
    // 1,706 / 166; 16,000 to 200,000 (2.0, 12 frames) 1,942 / 900.  At the line: 64,000 to
    // 200,000 (2.0, 12 frames) 2,723 / 2,547 at 2.4 times the walk's members, 64,000 to
    // themselves (2.0, 12 frames) 1,606 / 2,138 at 1.4; few atoms, 32 lanes each: 1,000 to 3,000 (3.0,
    // 12 frames) 209 / 217 at 1.3, 1,000 to 20,000 (5.0) 649 / 778 at 1.2.
    const double ew = std::max((double)max_distance * (1.0 + 1e-4) + 1e-6 * edge, std::cbrt(2.0 / rho2));
    const PHGrid gw = make_grid(ctx, ew, ew, false, tol);
    const double c = max_distance, w = l1.n > 1 ? std::min(w1, std::cbrt(vol)) : 0.0;
    const double by_group = std::min<double>(l2.n, rho2 * (w * w * w + 6.0 * w * w * c + 9.42 * w * c * c + 4.19 * c * c * c));
    const double by_walk = 27.0 * ((double)l2.n / gw.n_cells + 0.7);
    // lanes per atom while there are too few to fill the chip (10 to 64,000 as above: 427 /
    // 169 / 122 us with 1, 8 and 32; 4,000 to 64,000: 374 / 332 / 367)
    const int64_t members = (int64_t)l1.n * (int64_t)n_q;
    lanes = members <= 512 * (int64_t)ctx->n_sm ? 32 : (members <= 2048 * (int64_t)ctx->n_sm ? 8 : 1);
    walk = gw.n.x >= 3 && gw.n.y >= 3 && gw.n.z >= 3 && by_group > (lanes == 32 ? 1.2 : 2.4) * by_walk;
    if (walk) grid[0] = grid[1] = gw;
    auto per_frame = [&](int s) { return (size_t)lists[s]->n * 20 + (size_t)grid[s].n_cells * 12 + 4; };
    auto distinct = [](std::vector<int32_t> f) {
      std::sort(f.begin(), f.end());
      f.erase(std::unique(f.begin(), f.end()), f.end());
      return f;
    };
    const char* mb = std::getenv("AMDAT_PAIR_SCRATCH_MB");
    const size_t most = mb ? (size_t)std::max(0, std::atoi(mb)) << 20 : PH_TABLE_BYTES;
    fr[0] = distinct(fa), fr[1] = distinct(fb);
    if (walk && same) {  // the walk of one list has one set of tables
      std::vector<int32_t> both = fr[0];
      both.insert(both.end(), fr[1].begin(), fr[1].end());
      both = distinct(both);
      if (both.size() * per_frame(0) <= most) sides = 1, fr[0] = fr[1] = both;
    }
    for (int s = 0; s < 2; ++s)
      for (int32_t x : s ? fb : fa)
        slot[s].push_back((int32_t)(std::lower_bound(fr[s].begin(), fr[s].end(), x) - fr[s].begin()));
    // frames per batch and side: all, or what half of the limit holds
    int32_t step[2] = {(int32_t)fr[0].size(), (int32_t)fr[1].size()};
    if (sides == 2 && fr[0].size() * per_frame(0) + fr[1].size() * per_frame(1) > most) {
      for (int s = 0; s < 2; ++s) step[s] = (int32_t)std::max<size_t>(1, std::min<size_t>(fr[s].size(), most / 2 / per_frame(s)));
      std::vector<int32_t> order(n_q);
      std::iota(order.begin(), order.end(), 0);
      auto batch = [&](int32_t q) { return std::make_pair(slot[0][q] / step[0], slot[1][q] / step[1]); };
      std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return batch(x) < batch(y); });
      auto reorder = [&](std::vector<int32_t>& v) {
        const std::vector<int32_t> old = v;
        for (size_t i = 0; i < n_q; ++i) v[i] = old[order[i]];
      };
      for (std::vector<int32_t>* v : {&qa, &qb, &qrow, &slot[0], &slot[1]}) reorder(*v);
    }
    for (size_t i = 0; i < n_q; ++i) {
      const int32_t f0[2] = {slot[0][i] / step[0] * step[0], slot[1][i] / step[1] * step[1]};
      if (batches.empty() || batches.back().f0[0] != f0[0] || batches.back().f0[1] != f0[1]) {
        PHBatch B{{f0[0], f0[1]}, {0, 0}, i, 0};
        for (int s = 0; s < 2; ++s) B.nf[s] = std::min<int32_t>(step[s], (int32_t)fr[s].size() - f0[s]);
        batches.push_back(B);
      }
      ++batches.back().rows;
      for (int s = 0; s < 2; ++s) slot[s][i] -= f0[s];
    }
    for (int s = 0; s < 2; ++s) {
      o_fr[s] = table(fr[s]);
      o_slot[s] = table(slot[s]);
    }
  } else if (any) {
    units = pair_units(ctx, l1.n, l2.n, symmetric, (int64_t)n_q, &per_thread);
    o_units = table(units);
  }
  const size_t o_fa = table(qa), o_fb = table(qb), o_row = table(qrow);
  const size_t o_flag = host.size(), o_cnt = align(o_flag + 4);
  unsigned char* base = ctx->scratch.reserve(o_cnt + n_out * 8);
  if (!host.empty()) AMDAT_CUDA(cudaMemcpyAsync(base, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream));
  AMDAT_CUDA(cudaMemsetAsync(base + o_flag, 0, o_cnt - o_flag + n_out * 8, ctx->stream));
  PHParams p{};
  p.w = ctx->w.ptr;
  p.n_pad = ctx->n_pad;
  p.l1 = phview(l1);
  p.l2 = phview(l2);
  p.frame_a = (const int32_t*)(base + o_fa);
  p.frame_b = (const int32_t*)(base + o_fb);
  p.row_of = (const int32_t*)(base + o_row);
  p.box = make_float3(ctx->box[0], ctx->box[1], ctx->box[2]);
  p.bin_size = max_distance / (float)n_bins;
  p.inv_bin = 1.0f / p.bin_size;
  // the estimate's error, in bins: the square sums differ by 6 roundings of 2^-24 (3 after
  // the root), the root by 2^-23 and 2^-24 (the chain's), the quotient by the chain's
  // 2^-24, the reciprocal's 2^-24 and the product's 2^-24: 9 roundings of the bin number
  p.lim = 0.5f - 9.0f * 5.9604645e-8f * (float)(n_bins + 1) - 1e-6f;
  // squared lengths at or above this are past the last bin for sure
  const double cut = (double)max_distance * (1.0 + 1e-5);
  p.s2_cut = (float)(cut * cut);
  p.n_bins = n_bins;
  p.counts = (unsigned long long*)(base + o_cnt);
  if (cells) {
    size_t need = 0;
    size_t off[2][5];
    for (int s = 0; s < sides; ++s) {
      size_t nf = 0;
      for (const PHBatch& B : batches) nf = std::max(nf, (size_t)B.nf[s]);
      const size_t n = (size_t)lists[s]->n, nc1 = (size_t)grid[s].n_cells;
      off[s][0] = need; need = align(need + nf * n * 4);           // cell_of
      off[s][1] = need; need = align(need + nf * nc1 * 4);         // count
      off[s][2] = need; need = align(need + nf * (nc1 + 1) * 4);   // start
      off[s][3] = need; need = align(need + nf * nc1 * 4);         // cursor
      off[s][4] = need; need = align(need + nf * n * sizeof(float4));  // pos
    }
    unsigned char* cb = ctx->scratch2.reserve(need);
    cudaStream_t st = ctx->stream;
    int32_t *far = (int32_t*)(base + o_flag), at[2] = {-1, -1};  // at: first frame of the tables in place
    auto build = [&](int s, const PHBatch& B) {
      if (at[s] == B.f0[s]) return;
      at[s] = B.f0[s];
      const int nf = B.nf[s];
      const PHList l = phview(*lists[s]);
      const PHGrid& gs = grid[s];
      const int32_t* frames = (const int32_t*)(base + o_fr[s]) + B.f0[s];
      AMDAT_CUDA(cudaMemsetAsync(cb + off[s][1], 0, (size_t)nf * gs.n_cells * 4, st));
      const dim3 gn((unsigned)ceil_div(l.n, 256), (unsigned)nf);
      ph_cell_count_kernel<<<gn, 256, 0, st>>>(p.w, p.n_pad, l, frames, gs, (int32_t*)(cb + off[s][0]),
                                               (int32_t*)(cb + off[s][1]), far);
      ph_cell_scan_kernel<<<(unsigned)nf, PS_THREADS, 0, st>>>((const int32_t*)(cb + off[s][1]), gs.n_cells,
                                                               (int32_t*)(cb + off[s][2]), (int32_t*)(cb + off[s][3]));
      ph_cell_scatter_kernel<<<gn, 256, 0, st>>>(p.w, p.n_pad, l, frames, gs.n_cells, (const int32_t*)(cb + off[s][0]),
                                                 (int32_t*)(cb + off[s][3]), (float4*)(cb + off[s][4]));
      check_launch("pair cell lists");
      count_launch(ctx, 3);
    };
    const size_t shm = (size_t)PH_WARPS * (n_bins + 1) * 4;
    const int t = sides - 1;  // list 2's tables
    const float4 *pos1 = (const float4*)(cb + off[0][4]), *pos2 = (const float4*)(cb + off[t][4]);
    const int32_t* start2 = (const int32_t*)(cb + off[t][2]);
    const float reach = (float)(max_distance * (1.0 + 1e-5) + 2.0 * std::max(1e-4 * max_distance, 2e-6 * edge));
    // lists that may share atoms tell an atom's own pair by its index
    const bool apart = l1.contiguous && l2.contiguous && (l1.first + l1.n <= l2.first || l2.first + l2.n <= l1.first);
    for (const PHBatch& B : batches) {
      for (int s = 0; s < sides; ++s) build(s, B);
      PHParams pb = p;
      pb.frame_a += B.row0, pb.frame_b += B.row0, pb.row_of += B.row0;
      const int32_t *slot_a = (const int32_t*)(base + o_slot[0]) + B.row0, *slot_b = (const int32_t*)(base + o_slot[1]) + B.row0;
      auto launch = [&](auto kern, const auto& view, int64_t blocks) {
        if (shm > 24 * 1024)
          AMDAT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
        KernelTimer kt(ctx, "pair_hist_cells_kernel");
        kern<<<dim3((unsigned)blocks, (unsigned)B.rows), PH_THREADS, shm, st>>>(pb, view);
        check_launch("pair_hist_cells_kernel");
        count_launch(ctx);
      };
      if (walk) {
        KernelTimer kt(ctx, "pair_hist_walk_kernel");
        const PHWalk W{pos1, l1.n, pos2, start2, l2.n, grid[1], slot_a, slot_b, far};
        const int64_t blocks = ceil_div(l1.n, PH_THREADS / lanes);
        if (lanes == 32) launch(pair_hist_walk_kernel<32>, W, blocks);
        else if (lanes == 8) launch(pair_hist_walk_kernel<8>, W, blocks);
        else launch(pair_hist_walk_kernel<1>, W, blocks);
      } else {
        // up to eight groups per warp (one flush of the histograms for them) while the blocks
        // fill the chip twice over
        const int64_t groups = ceil_div(l1.n, 32);
        const int per_warp = (int)std::max<int64_t>(1, std::min<int64_t>(8, groups * (int64_t)B.rows / ((int64_t)ctx->n_sm * 8 * PH_WARPS)));
        const PHGroups G{pos1, l1.n, per_warp, pos2, start2, l2.n, grid[1], slot_a, slot_b, reach, same ? 1 : 0, far};
        const int64_t blocks = ceil_div(groups, (int64_t)PH_WARPS * per_warp);
        if (same || apart) launch(pair_hist_groups_kernel<PH_SELF_LATER>, G, blocks);
        else launch(pair_hist_groups_kernel<PH_SELF_IDS>, G, blocks);
      }
    }
  }
  auto all_pairs = [&](const PHUnit* d_units) {
    const bool ids = fa != fb;
    const size_t shm = (size_t)PH_WARPS * (n_bins + 1) * 4;
    auto launch = [&](auto kern) {
      if (shm > 32 * 1024)
        AMDAT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
      KernelTimer kt(ctx, "pair_hist_kernel");
      kern<<<dim3((unsigned)units.size(), (unsigned)n_q), PH_THREADS, shm, ctx->stream>>>(p, d_units);
      check_launch("pair_hist_kernel");
      count_launch(ctx);
    };
    const int I = per_thread;
    if (ids) I == 4 ? launch(pair_hist_kernel<4, PH_SELF_IDS>) : I == 2 ? launch(pair_hist_kernel<2, PH_SELF_IDS>) : launch(pair_hist_kernel<1, PH_SELF_IDS>);
    else I == 4 ? launch(pair_hist_kernel<4, PH_SELF_ZERO>) : I == 2 ? launch(pair_hist_kernel<2, PH_SELF_ZERO>) : launch(pair_hist_kernel<1, PH_SELF_ZERO>);
  };
  auto read = [&] {
    AMDAT_CUDA(cudaMemcpyAsync(counts, base + o_cnt, n_out * 8,
                               out_flags == AMDAT_OUT_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                               ctx->stream));
    AMDAT_CUDA(cudaStreamSynchronize(ctx->stream));
  };
  if (any && !cells) all_pairs((const PHUnit*)(base + o_units));
  int32_t here = 0, *outside = ctx->result ? (int32_t*)ctx->result : &here;
  *outside = 0;
  if (cells) AMDAT_CUDA(cudaMemcpyAsync(outside, base + o_flag, 4, cudaMemcpyDeviceToHost, ctx->stream));
  read();
  if (*outside) {
    // atoms far outside the box: the all-pairs pass instead
    units = pair_units(ctx, l1.n, l2.n, symmetric, (int64_t)n_q, &per_thread);
    PHUnit* d_units = (PHUnit*)ctx->scratch2.reserve(units.size() * sizeof(PHUnit));
    AMDAT_CUDA(cudaMemcpyAsync(d_units, units.data(), units.size() * sizeof(PHUnit), cudaMemcpyHostToDevice, ctx->stream));
    AMDAT_CUDA(cudaMemsetAsync(base + o_cnt, 0, n_out * 8, ctx->stream));
    all_pairs(d_units);
    read();
  }
}

}  // namespace amdat

using namespace amdat;

extern "C" {

amdat_status amdat_rdf_run(amdat_ctx* ctx, int32_t list1, int32_t list2, const int32_t* frames,
                           int32_t n_frames, float max_distance, int32_t n_bins, int32_t out_flags,
                           int64_t* counts) {
  return guarded([&] {
    check_ctx(ctx);
    if (!ctx->have_traj) throw Error(AMDAT_ERR_STATE, "no trajectory uploaded");
    AMDAT_REQUIRE(frames != nullptr && n_frames >= 1, "need >= 1 frame");
    for (int f = 0; f < n_frames; ++f)
      AMDAT_REQUIRE(frames[f] >= 0 && frames[f] < ctx->n_frames, "frame index out of range");
    const ListEntry& a = list_entry(ctx, list1);
    const ListEntry& b = list_entry(ctx, list2);
    std::vector<int32_t> fa(frames, frames + n_frames), row(n_frames);
    for (int f = 0; f < n_frames; ++f) row[f] = f;
    run_pair_hist(ctx, a, b, list1 == list2, fa, fa, row, n_frames, max_distance, n_bins,
                  out_flags, counts);
  });
}

amdat_status amdat_vhd_run(amdat_ctx* ctx, int32_t list1, int32_t list2, int32_t fullblock,
                           float max_distance, int32_t n_bins, int32_t out_flags, int64_t* counts) {
  return guarded([&] {
    check_ctx(ctx);
    if (!ctx->have_traj) throw Error(AMDAT_ERR_STATE, "no trajectory uploaded");
    const ListEntry& a = list_entry(ctx, list1);
    const ListEntry& b = list_entry(ctx, list2);
    const PairTable& P = pair_table(ctx, fullblock != 0, false);
    Pairs hp = scheme_pairs(ctx->scheme, fullblock != 0, false);
    // time pairs with t0 == t1 (gap 0) are the same-time pair loop: symmetric counting
    // applies only when t0 == t1; keep the general ordered loop for every pair.
    run_pair_hist(ctx, a, b, false, hp.t0, hp.t1, hp.gap, P.n_gaps, max_distance, n_bins,
                  out_flags, counts);
  });
}

}  // extern "C"
