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
// IDS: frames differ, so an atom's own pair has to be told by its index; within one
// frame it is the pair at zero distance, which the exact path checks.
// Bound: instruction issue, 23 per pair and warp at 69 % of the issue slots; the
// histogram's shared-memory atomics take 2.5 wavefronts per 32 pairs (half the pairs in
// range).  g(r) of 64,000 atoms to half the box, 50 frames: 70.6 ms, against 163 ms with
// 35 instructions per pair (scalar chain, a branch around every count) over blocks of a
// triangle.
template <int I, bool IDS>
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
      const uint64_t xj[2] = {pk2(X.x, X.y), pk2(X.z, X.w)}, yj[2] = {pk2(Y.x, Y.y), pk2(Y.z, Y.w)},
                     zj[2] = {pk2(Z.x, Z.y), pk2(Z.z, Z.w)};
      int4 id = make_int4(0, 0, 0, 0);
      if (IDS) id = *reinterpret_cast<const int4*>(sid + t);
      const int ids[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
      for (int k = 0; k < I; ++k) {
        float s[4], y[4], r[4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          pair_estimate2(p, sub2(xj[h], xi[k]), sub2(yj[h], yi[k]), sub2(zj[h], zi[k]), s + 2 * h, y + 2 * h, r + 2 * h);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (IDS && ids[e] == ai[k]) s[e] = nan;
          count_if(s[e], p.s2_cut, y[e], hist, (uint32_t)U.inc);
        }
        // estimates within their error bound of a bin edge: the counts are put right
        // (and an atom's own pair, at zero distance, taken out)
        if (fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fmaxf(fabsf(r[2]), fabsf(r[3]))) >= p.lim) {
          const float x = __uint_as_float((uint32_t)xi[k]), yy = __uint_as_float((uint32_t)yi[k]), z = __uint_as_float((uint32_t)zi[k]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (!(s[e] < p.s2_cut) || fabsf(r[e]) < p.lim) continue;
            const int est = (int)(__float_as_uint(y[e]) - PH_MAGIC_BITS);
            const int b = exact_bin(__fsub_rn(sx[t + e], x), __fsub_rn(sy[t + e], yy), __fsub_rn(sz[t + e], z), p.box, p.bin_size);
            const bool self = sid[t + e] == ai[k];
            if (b == est && !self) continue;
            atomicSub(whist + est, (unsigned int)U.inc);
            if (!self && b >= 0 && b < p.n_bins) atomicAdd(whist + b, (unsigned int)U.inc);
          }
        }
      }
    }
  }
  __syncthreads();
  unsigned long long* dst = p.counts + (int64_t)p.row_of[q] * p.n_bins;
  for (int b = threadIdx.x; b < p.n_bins; b += PH_THREADS) {
    unsigned long long s = 0;
    for (int w = 0; w < PH_WARPS; ++w) s += sh_hist[w * nb1 + b];
    if (s) atomicAdd(dst + b, s);
  }
}

// ordered pairs of the cell pass: the short exact branch
__device__ __forceinline__ void pair_term(const PHParams& p, float4 c, float xi, float yi, float zi,
                                          unsigned int* hist) {
  const float mx = min_image(__fsub_rn(c.x, xi), p.box.x);
  const float my = min_image(__fsub_rn(c.y, yi), p.box.y);
  const float mz = min_image(__fsub_rn(c.z, zi), p.box.z);
  const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(mx, mx), __fmul_rn(my, my)), __fmul_rn(mz, mz));
  if (s2 < p.s2_cut) {
    const int b = (int)__fdiv_rn(__fsqrt_rn(s2), p.bin_size);
    if (b >= 0 && b < p.n_bins) atomicAdd(hist + b, 1u);
  }
}

// ---------------------------------------------------------------------------
// cell lists for short-range ordered pair loops (the distinct van Hove pass and
// RDFs of two different lists): when every box axis holds at least three cells
// no narrower than the last bin edge, a pair that can fall in a bin has its
// atoms in the same or neighbouring cells (periodic).  Per frame the list's
// atoms are counted into cells, the counts scanned and the atoms scattered in
// cell order as (x, y, z, atom index bits); a thread takes one list-1 member in
// cell order at t0 and visits the 27 cells around it in the list-2 cells at t1.
// Distances and bins are the exact chain of pair_term, counts are integer
// atomics, so the counts equal the all-pairs kernel's bit for bit.
// ---------------------------------------------------------------------------
struct PHCells {
  int3 nc;
  float3 lo, inv_cell;
  int32_t n_cells;
  const int32_t* start;  // [slot][n_cells + 1]
  const float4* pos;     // [slot][n]: members in cell order
  int32_t n;             // members per slot
};

__device__ __forceinline__ int ph_cell_axis(float x, float lo, float inv_cell, int n) {
  const int c = (int)((x - lo) * inv_cell);
  return min(max(c, 0), n - 1);
}

// members of list l at frame frames[s] counted into the cells of slot s
__global__ void ph_cell_count_kernel(const float* __restrict__ w, int64_t n_pad, PHList l,
                                     const int32_t* __restrict__ frames, int3 nc, float3 lo, float3 inv_cell,
                                     int32_t* __restrict__ cell_of, int32_t* __restrict__ count) {
  const int s = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= l.n) return;
  const float* P = w + (int64_t)frames[s] * 3 * n_pad;
  const int a = member(l, i);
  const int c = (ph_cell_axis(P[2 * n_pad + a], lo.z, inv_cell.z, nc.z) * nc.y +
                 ph_cell_axis(P[n_pad + a], lo.y, inv_cell.y, nc.y)) * nc.x +
                ph_cell_axis(P[a], lo.x, inv_cell.x, nc.x);
  cell_of[(int64_t)s * l.n + i] = c;
  atomicAdd(count + (int64_t)s * nc.x * nc.y * nc.z + c, 1);
}

// exclusive scan of one slot's cell counts (one block per slot) into start and
// the scatter cursors
__global__ void __launch_bounds__(1024) ph_cell_scan_kernel(const int32_t* __restrict__ count, int32_t n_cells,
                                                            int32_t* __restrict__ start, int32_t* __restrict__ cursor) {
  __shared__ int32_t s_part[1024];
  __shared__ int32_t s_carry;
  const int s = blockIdx.x;
  const int32_t* C = count + (int64_t)s * n_cells;
  int32_t* S = start + (int64_t)s * (n_cells + 1);
  int32_t* U = cursor + (int64_t)s * n_cells;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int base = 0; base < n_cells; base += 1024) {
    const int i = base + threadIdx.x;
    s_part[threadIdx.x] = i < n_cells ? C[i] : 0;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
      const int v = threadIdx.x >= off ? s_part[threadIdx.x - off] : 0;
      __syncthreads();
      s_part[threadIdx.x] += v;
      __syncthreads();
    }
    if (i < n_cells) {
      const int excl = s_carry + s_part[threadIdx.x] - C[i];
      S[i] = excl;
      U[i] = excl;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_carry += s_part[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) S[n_cells] = s_carry;
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

// ordered pairs (i at t0 from list 1, j != i at t1 from list 2) within the 27
// cells around i; slot_a / slot_b give each row's cell slots
__global__ void __launch_bounds__(PH_THREADS)
    pair_hist_cells_kernel(PHParams p, PHCells C1, PHCells C2, const int32_t* __restrict__ slot_a,
                           const int32_t* __restrict__ slot_b) {
  extern __shared__ unsigned int sh_hist[];  // [8 warps][n_bins]
  const int q = blockIdx.y;
  const int warp = threadIdx.x >> 5;
  unsigned int* hist = sh_hist + warp * p.n_bins;
  for (int b = threadIdx.x; b < 8 * p.n_bins; b += blockDim.x) sh_hist[b] = 0u;
  __syncthreads();
  const int i = blockIdx.x * PH_THREADS + threadIdx.x;
  if (i < C1.n) {
    const float4 pi = C1.pos[(int64_t)slot_a[q] * C1.n + i];
    const int ai = __float_as_int(pi.w);
    const int32_t* S2 = C2.start + (int64_t)slot_b[q] * (C2.n_cells + 1);
    const float4* P2 = C2.pos + (int64_t)slot_b[q] * C2.n;
    const int cx = ph_cell_axis(pi.x, C2.lo.x, C2.inv_cell.x, C2.nc.x);
    const int cy = ph_cell_axis(pi.y, C2.lo.y, C2.inv_cell.y, C2.nc.y);
    const int cz = ph_cell_axis(pi.z, C2.lo.z, C2.inv_cell.z, C2.nc.z);
    for (int dz = -1; dz <= 1; ++dz) {
      int z = cz + dz;
      z += z < 0 ? C2.nc.z : (z >= C2.nc.z ? -C2.nc.z : 0);
      for (int dy = -1; dy <= 1; ++dy) {
        int y = cy + dy;
        y += y < 0 ? C2.nc.y : (y >= C2.nc.y ? -C2.nc.y : 0);
        for (int dx = -1; dx <= 1; ++dx) {
          int x = cx + dx;
          x += x < 0 ? C2.nc.x : (x >= C2.nc.x ? -C2.nc.x : 0);
          const int c = (z * C2.nc.y + y) * C2.nc.x + x;
          const int k1 = __ldg(S2 + c + 1);
          for (int k = __ldg(S2 + c); k < k1; ++k) {
            const float4 cj = __ldg(P2 + k);
            if (__float_as_int(cj.w) != ai) pair_term(p, cj, pi.x, pi.y, pi.z, hist);
          }
        }
      }
    }
  }
  __syncthreads();
  unsigned long long* dst = p.counts + (int64_t)p.row_of[q] * p.n_bins;
  for (int b = threadIdx.x; b < p.n_bins; b += blockDim.x) {
    unsigned long long s = 0;
    for (int w = 0; w < 8; ++w) s += sh_hist[w * p.n_bins + b];
    if (s) atomicAdd(dst + b, s);
  }
}

static void run_pair_hist(amdat_ctx* ctx, const ListEntry& l1, const ListEntry& l2, bool symmetric,
                          const std::vector<int32_t>& fa, const std::vector<int32_t>& fb,
                          const std::vector<int32_t>& row, int32_t n_rows_out, float max_distance,
                          int32_t n_bins, int32_t out_flags, int64_t* counts) {
  AMDAT_REQUIRE(n_bins >= 1 && n_bins <= 4096, "n_bins must be in [1, 4096]");
  AMDAT_REQUIRE(max_distance > 0.0f, "max_distance must be positive");
  AMDAT_REQUIRE(counts != nullptr, "null output");
  const size_t n_q = fa.size();
  const size_t n_out = (size_t)n_rows_out * n_bins;
  auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
  size_t o = 0;
  const size_t o_fa = o; o = align(o + std::max<size_t>(n_q, 1) * 4);
  const size_t o_fb = o; o = align(o + std::max<size_t>(n_q, 1) * 4);
  const size_t o_row = o; o = align(o + std::max<size_t>(n_q, 1) * 4);
  const size_t o_cnt = o; o = align(o + n_out * 8);
  unsigned char* base = ctx->scratch.reserve(o);
  std::vector<unsigned char> host(o_cnt, 0);
  if (n_q) {
    std::memcpy(host.data() + o_fa, fa.data(), n_q * 4);
    std::memcpy(host.data() + o_fb, fb.data(), n_q * 4);
    std::memcpy(host.data() + o_row, row.data(), n_q * 4);
  }
  AMDAT_CUDA(cudaMemcpyAsync(base, host.data(), o_cnt, cudaMemcpyHostToDevice, ctx->stream));
  AMDAT_CUDA(cudaMemsetAsync(base + o_cnt, 0, n_out * 8, ctx->stream));
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
  // cell lists for the ordered pass when the box holds at least three cells per
  // axis no narrower than the last bin edge (with a 1e-4 margin over the
  // in-range cut, so a rounding of a cell index never splits an in-range pair)
  const float cell_edge = (float)((double)max_distance * (1.0 + 1e-4));
  const int3 nc = make_int3((int)std::floor(ctx->box[0] / cell_edge), (int)std::floor(ctx->box[1] / cell_edge),
                            (int)std::floor(ctx->box[2] / cell_edge));
  const int64_t n_cells = (int64_t)nc.x * nc.y * nc.z;
  const char* pc = std::getenv("AMDAT_PAIR_CELLS");  // "off": the all-pairs pass
  const bool cells = !symmetric && n_q && l1.n > 0 && l2.n >= 1024 && nc.x >= 3 && nc.y >= 3 && nc.z >= 3 &&
                     n_cells <= (1 << 20) && !(pc && std::strcmp(pc, "off") == 0);
  if (cells) {
    // frame slots: the distinct frames of each side; one structure when both
    // sides are the same list
    const bool same = &l1 == &l2;
    std::vector<int32_t> fr1, fr2;
    auto slots = [](const std::vector<int32_t>& f, std::vector<int32_t>& uniq, std::vector<int32_t>& slot_of) {
      uniq = f;
      std::sort(uniq.begin(), uniq.end());
      uniq.erase(std::unique(uniq.begin(), uniq.end()), uniq.end());
      slot_of.resize(f.size());
      for (size_t i = 0; i < f.size(); ++i)
        slot_of[i] = (int32_t)(std::lower_bound(uniq.begin(), uniq.end(), f[i]) - uniq.begin());
    };
    std::vector<int32_t> sa, sb;
    if (same) {
      std::vector<int32_t> both(fa);
      both.insert(both.end(), fb.begin(), fb.end());
      std::vector<int32_t> tmp;
      slots(both, fr1, tmp);
      sa.assign(tmp.begin(), tmp.begin() + (std::ptrdiff_t)n_q);
      sb.assign(tmp.begin() + (std::ptrdiff_t)n_q, tmp.end());
      fr2 = fr1;
    } else {
      slots(fa, fr1, sa);
      slots(fb, fr2, sb);
    }
    const int n_sides = same ? 1 : 2;
    const ListEntry* lists[2] = {&l1, &l2};
    const std::vector<int32_t>* frs[2] = {&fr1, &fr2};
    size_t need = 0;
    size_t off[2][6];
    for (int s = 0; s < n_sides; ++s) {
      const size_t nf = frs[s]->size(), n = (size_t)lists[s]->n;
      off[s][0] = need; need = align(need + nf * 4);                           // frames
      off[s][1] = need; need = align(need + nf * n * 4);                       // cell_of
      off[s][2] = need; need = align(need + nf * (size_t)n_cells * 4);         // count
      off[s][3] = need; need = align(need + nf * (size_t)(n_cells + 1) * 4);   // start
      off[s][4] = need; need = align(need + nf * (size_t)n_cells * 4);         // cursor
      off[s][5] = need; need = align(need + nf * n * sizeof(float4));          // pos
    }
    const size_t o_sa = need; need = align(need + n_q * 4);
    const size_t o_sb = need; need = align(need + n_q * 4);
    unsigned char* cb = ctx->scratch2.reserve(need);
    cudaStream_t st = ctx->stream;
    AMDAT_CUDA(cudaMemcpyAsync(cb + o_sa, sa.data(), n_q * 4, cudaMemcpyHostToDevice, st));
    AMDAT_CUDA(cudaMemcpyAsync(cb + o_sb, sb.data(), n_q * 4, cudaMemcpyHostToDevice, st));
    PHCells C[2];
    for (int s = 0; s < n_sides; ++s) {
      const int nf = (int)frs[s]->size();
      const PHList l = phview(*lists[s]);
      PHCells& c = C[s];
      c.nc = nc;
      c.lo = make_float3(ctx->box_lo[0], ctx->box_lo[1], ctx->box_lo[2]);
      c.inv_cell = make_float3((float)nc.x / ctx->box[0], (float)nc.y / ctx->box[1], (float)nc.z / ctx->box[2]);
      c.n_cells = (int32_t)n_cells;
      c.start = (const int32_t*)(cb + off[s][3]);
      c.pos = (const float4*)(cb + off[s][5]);
      c.n = l.n;
      AMDAT_CUDA(cudaMemcpyAsync(cb + off[s][0], frs[s]->data(), (size_t)nf * 4, cudaMemcpyHostToDevice, st));
      AMDAT_CUDA(cudaMemsetAsync(cb + off[s][2], 0, (size_t)nf * n_cells * 4, st));
      AMDAT_REQUIRE(nf <= 65535, "at most 65535 frames per call");
      const dim3 g((unsigned)ceil_div(l.n, 256), (unsigned)nf);
      ph_cell_count_kernel<<<g, 256, 0, st>>>(p.w, p.n_pad, l, (const int32_t*)(cb + off[s][0]), nc, c.lo,
                                              c.inv_cell, (int32_t*)(cb + off[s][1]), (int32_t*)(cb + off[s][2]));
      ph_cell_scan_kernel<<<(unsigned)nf, 1024, 0, st>>>((const int32_t*)(cb + off[s][2]), (int32_t)n_cells,
                                                          (int32_t*)(cb + off[s][3]), (int32_t*)(cb + off[s][4]));
      ph_cell_scatter_kernel<<<g, 256, 0, st>>>(p.w, p.n_pad, l, (const int32_t*)(cb + off[s][0]), (int32_t)n_cells,
                                                (const int32_t*)(cb + off[s][1]), (int32_t*)(cb + off[s][4]),
                                                (float4*)(cb + off[s][5]));
      check_launch("pair cell lists");
      count_launch(ctx, 3);
    }
    if (same) C[1] = C[0];
    const size_t shm = (size_t)8 * n_bins * 4;
    if (shm > 48 * 1024)
      AMDAT_CUDA(cudaFuncSetAttribute(pair_hist_cells_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
    AMDAT_REQUIRE(n_q <= 65535, "at most 65535 frames or time pairs per call");
    dim3 grid((unsigned)ceil_div(l1.n, PH_THREADS), (unsigned)n_q);
    KernelTimer kt(ctx, "pair_hist_cells_kernel");
    pair_hist_cells_kernel<<<grid, PH_THREADS, shm, st>>>(p, C[0], C[1], (const int32_t*)(cb + o_sa),
                                                          (const int32_t*)(cb + o_sb));
    check_launch("pair_hist_cells_kernel");
    count_launch(ctx);
  } else if (n_q && l1.n > 0 && l2.n > 0) {
    AMDAT_REQUIRE(n_q <= 65535, "at most 65535 frames or time pairs per call");
    // units of 256 I members by up to seg list-2 members: wide ones while they fill
    // the chip six times over, then fewer members per thread and shorter segments
    const bool ids = fa != fb;
    const int64_t want = 6 * (int64_t)ctx->n_sm;
    auto count_units = [&](int I, int seg) {
      const int64_t ib = ceil_div(l1.n, 256 * I), js = ceil_div(l2.n, seg);
      return (symmetric ? (ib * js + ib) / 2 : ib * js) * (int64_t)n_q;
    };
    int I = 4, seg = 8192;
    while (seg > 1024 && count_units(I, seg) < want) seg /= 2;
    while (I > 1 && count_units(I, seg) < want) I /= 2;
    while (seg > 128 && count_units(I, seg) < want) seg /= 2;
    std::vector<PHUnit> units;
    for (int i0 = 0; i0 < l1.n; i0 += 256 * I) {
      const int i1 = std::min(l1.n, i0 + 256 * I);
      if (symmetric)
        for (int j = i0; j < i1; j += seg) units.push_back(PHUnit{i0, j, std::min(i1, j + seg), 1});
      for (int j = symmetric ? i1 : 0; j < l2.n; j += seg)
        units.push_back(PHUnit{i0, j, std::min(l2.n, j + seg), symmetric ? 2 : 1});
    }
    PHUnit* d_units = (PHUnit*)ctx->scratch2.reserve(units.size() * sizeof(PHUnit));
    AMDAT_CUDA(cudaMemcpyAsync(d_units, units.data(), units.size() * sizeof(PHUnit), cudaMemcpyHostToDevice, ctx->stream));
    const size_t shm = (size_t)PH_WARPS * (n_bins + 1) * 4;
    auto launch = [&](auto kern) {
      if (shm > 32 * 1024)
        AMDAT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
      KernelTimer kt(ctx, "pair_hist_kernel");
      kern<<<dim3((unsigned)units.size(), (unsigned)n_q), PH_THREADS, shm, ctx->stream>>>(p, d_units);
      check_launch("pair_hist_kernel");
      count_launch(ctx);
    };
    if (ids) I == 4 ? launch(pair_hist_kernel<4, true>) : I == 2 ? launch(pair_hist_kernel<2, true>) : launch(pair_hist_kernel<1, true>);
    else I == 4 ? launch(pair_hist_kernel<4, false>) : I == 2 ? launch(pair_hist_kernel<2, false>) : launch(pair_hist_kernel<1, false>);
  }
  AMDAT_CUDA(cudaMemcpyAsync(counts, base + o_cnt, n_out * 8,
                             out_flags == AMDAT_OUT_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                             ctx->stream));
  AMDAT_CUDA(cudaStreamSynchronize(ctx->stream));
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
