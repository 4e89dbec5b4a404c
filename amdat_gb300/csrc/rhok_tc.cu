// Tensor-core (tcgen05) Fourier densities over the whole half-space lattice.
//
// rho[(nx,ny), nz] = sum_j W_j(nx,ny) Z_j(nz), W = X(nx) Y(ny), is a complex
// GEMM with the atoms as the reduction axis, and W(-nx,-ny) = conj W(nx,ny): the
// rows of half the (nx, ny) plane serve the other half against conj Z.  As a real
// GEMM per tile of 64 complex rows (8 nx >= 0 x 8 ny) and n consecutive nz:
//   A (128 x 2J): of complex row (nx0 + m, ny0 + y), k = 2j, 2j+1 per atom j:
//                 lane 16 y + m = [Wr, -Wi], lane 16 y + 8 + m = [Wi,  Wr]
//   B ( 2n x 2J): rows 0..n-1 [Zr, Zi], rows n..2n-1 [Zr, -Zi] of the n nz
//   D = A B^T  (128 x 2n): lane 16 y + m = Re, lane 16 y + 8 + m = Im of
//                rho(nx, ny, nz) in the first n columns; Re and -Im of
//                rho(-nx, -ny, nz) in the others.
// One built A so serves two lattice rows, and the MMAs are twice as wide: at the
// benchmark's lattice (|n| <= 106) MMA N = 2 x 81 on average runs at the full
// rate, where N = 81 is bound by the operand fetch (M = 128, K = 16: 32 + N/4
// cycles against N/2).  Every product, split and accumulation is the one a
// full-plane tile would do, so the densities do not depend on the tiling.
// A builder thread forms W of two rows for four atoms and writes both lanes of each
// row (16 x 128-bit tensor-memory stores: a thread holds rows t / 4 and t / 4 + 8,
// columns t % 4 of every four), so a product is formed and split once for its two
// lanes and the X and Y factors are read from shared memory once for four lanes.
// With one lane per thread the kernel was bound by shared-memory bandwidth: per
// 32-atom chunk 633 wavefronts of factor loads beside ~490 of MMA operand reads and
// ~370 of copies in 1510 cycles; now 192.
// Operands are FP16 split into hi + lo parts (hi = x rounded to a multiple of
// 2^-11, exact in FP16; lo = x - hi to ~2^-24), and each chunk of 32 atoms
// runs three tcgen05.mma passes, hi*lo + lo*hi + hi*hi (small terms first),
// accumulating in FP32 tensor memory.  The tensor core's FP32 accumulation
// drops low bits as the accumulator grows, so an accumulation never spans more
// than TC_GROUP chunks (64 atoms): the drain warps then add the accumulator
// into compensated sums held in their registers (Fast2Sum) and write the
// rounding residual back into the accumulator, where the next accumulation on
// it starts.  The phases are the exact fixed-point phases of the FP32 kernels
// (fraction of the box in units of 2^-31 turns).
//
// What bounds it: the MMAs.  Back to back, an M = 128, K = 16 tcgen05.mma takes
// N / 2 + 10 cycles (1.13 ms per frame of the benchmark lattice: 32,000 atoms,
// 2.56 M vectors), the kernel 1.55 ms; with the builders off 1.27 ms, with the drains
// off 1.41 ms, with the copies off 1.43 ms.  Before (one lane row per thread, separate
// tiles for the two half planes, one-lane waits): 2.58 ms.
//
// Per frame batch, zgen_kernel precomputes the B operands (Z and conj Z, hi/lo, in
// the K-major 128-byte-swizzled layout, one blob per (frame, chunk)) and
// xygen_kernel the X and Y phase tables.  The main kernel is warp-specialised,
// one CTA per SM, 512 tensor-memory columns (two accumulators of 2n columns, then
// A stages of 64 columns):
//   warps 0-7    drain: accumulator -> register sums (lane quadrant warp % 4,
//                16-column blocks 2 i + warp / 4), then the epilogue
//   warp 8       producer: bulk copies (cp.async.bulk) of the Z parts and the X/Y
//                tables of each chunk into a shared-memory ring
//   warps 9-10   MMA issuers, one per accumulator (even and odd groups of chunks): 12
//                tcgen05.mma per chunk, A read from tensor memory
//   warps 12-19  builders: the A operand of the chunk (W products, FP16 split)
//                stored into tensor memory (lane quadrant warp % 4; warps 12-15 the
//                even, 16-19 the odd chunks)
// Hand-offs are mbarriers (bulk-copy transactions, tcgen05.commit, thread
// arrivals).  A waiting warp waits with all its lanes and one elected lane issues:
// an mbarrier hand-off and back between two warps takes 227 cycles so, and 713
// when one lane waits and the warp then reconverges.  Every wait is bounded, and a
// timeout makes every role stop, wait for its own copies and MMAs, free tensor
// memory and report through an error word.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.h"
#include "f32x2.cuh"
#include "tc_tiles.h"
#include "umma.cuh"

namespace amdat {

constexpr int TC_J = 32;                      // atoms per chunk
constexpr int TC_K = 2 * TC_J;                // real K per chunk
constexpr int TC_ROWS = 64;                   // complex rows (8 nx x 8 ny)
constexpr int TC_NZMAX = 96;                  // widest nz window (MMA N = 192)
constexpr int TC_M = 2 * TC_ROWS;             // MMA M = 128
constexpr int TC_GROUP = 2;                   // chunks per tensor-memory accumulation
constexpr int TC_ZS = 4;                      // shared-memory ring stages: Z, X, Y
constexpr int TC_AS_MAX = 4;                  // A stages in tensor memory at most
constexpr uint32_t TC_HDR = 1024;             // barrier header ahead of the ring
constexpr uint32_t TC_SMEM_MAX = 227 * 1024;  // dynamic shared memory per block
constexpr int TC_DRAIN_WARPS = 8;             // warps 0-7
constexpr int TC_DRAIN_PAR = TC_DRAIN_WARPS / 4;  // drain warps per lane quadrant
constexpr int TC_PRODUCER_WARP = 8;
constexpr int TC_MMA_WARP = 9;                // warps 9 and 10: one per accumulator
constexpr int TC_MMA_WARPS = 2;
constexpr int TC_BUILD_WARP0 = 12;            // a multiple of 4: lane quadrant = warp % 4
constexpr int TC_BUILD_WARPS = 8;
constexpr int TC_THREADS = 32 * (TC_BUILD_WARP0 + TC_BUILD_WARPS);  // 640
// registers: 96 a thread at launch (61440), moved to the drain warps' sums
constexpr int TC_REG_DRAIN = 152, TC_REG_MISC = 48, TC_REG_BUILD = 64;
static_assert(256 * TC_REG_DRAIN + 128 * TC_REG_MISC + 256 * TC_REG_BUILD <= TC_THREADS * 96, "register split");
constexpr uint32_t TC_XB = TC_J * 8 * sizeof(float2);         // 2 KB: cos and sin of 32 atoms x 8 lattice indices
constexpr uint32_t TC_XYB = 2 * TC_XB;
constexpr uint32_t TC_ZROW = TC_K * 2;                        // 128 bytes: one nz of a Z part
constexpr uint32_t TC_WAIT = 1u << 19;                        // try_wait calls of <= 1 us (~0.5 s bound)
// tensor-memory columns of a tile of n nz: accumulators at 0 and 2n, A stages from
// 4n; an A stage holds per 16-atom half u [hi (16 columns) | lo (16 columns)] at 32 u
constexpr uint32_t TC_A_COLS = 2 * (TC_K / 2);
constexpr uint32_t TC_TMEM_COLS = 512;
static_assert(4 * TC_NZMAX + 2 * TC_A_COLS <= TC_TMEM_COLS, "accumulators and two A stages must fit tensor memory");

struct TcHdr {
  uint64_t full_z[TC_ZS];       // the stage's copies landed
  uint64_t full_a[2 * TC_GROUP];  // A(c) built, barrier c % 4: each belongs to one MMA issuer
  uint64_t half_done[2];        // the MMAs of a group's first chunk finished (groups alternate)
  uint64_t full_acc[2];         // the MMAs of the whole group finished: accumulator full, its chunks' stages free
  uint64_t empty_acc[2];        // the accumulator drained
  uint64_t mma_done;
  uint32_t tmem;
  volatile int bad;  // any role gave up
  int z_issued;      // chunks whose copies were issued
};
static_assert(sizeof(TcHdr) <= TC_HDR, "the barrier header must fit its slot");
// the Z operands use the 128-byte-swizzled K-major layout: 128-byte rows, 1024-byte aligned tiles
static_assert(TC_K * 2 == 128, "one chunk's K must fill a 128-byte swizzle row");

// shared-memory ring stage bytes for tiles of at most nzw nz: hi and lo parts of
// 2 nzw rows (Z, conj Z) of 128 bytes each, X, Y
__host__ __device__ constexpr uint32_t tc_zstage(int nzw) { return 2u * 2u * (uint32_t)nzw * TC_ZROW + TC_XYB; }

__device__ __forceinline__ void tc_split(float x, __half& hi, __half& lo) {
  hi = __float2half_rn(x);
  lo = __float2half_rn(__fsub_rn(x, __half2float(hi)));
}

__device__ __forceinline__ void tc_phase(int32_t ph, float* s, float* c) {
  sincospif(__fmul_rn((float)ph, 9.313225746154785e-10f), s, c);  // ph * 2^-30 * pi
}

// hi and lo parts of a pair with |x| <= 1: hi = round to a multiple of 2^-11 (6144 =
// 1.5 * 2^12 has a 2^-11 ulp, so (x + 6144) - 6144 rounds x to that grid; every such
// value in [-1, 1] is exact in FP16), lo = x - hi exactly in FP32 (|lo| <= 2^-12)
__device__ __forceinline__ void tc_split2(uint64_t w, float (&hi)[2], float (&lo)[2]) {
  const uint64_t c = pk2(6144.0f, 6144.0f);
  const uint64_t h = sub2(add2(w, c), c);
  upk2(h, hi[0], hi[1]);
  upk2(sub2(w, h), lo[0], lo[1]);
}
__device__ __forceinline__ uint32_t tc_half2(float a, float b) {  // (a: low half, b: high half)
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Z operands of one frame batch: blob (f, chunk) = [Z hi][conj Z hi][Z lo][conj Z lo],
// each an nzr (nz) x 64 (k) K-major tile; k = 2j -> Re Z_j, 2j+1 -> Im Z_j.  A thread
// forms four atoms of one nz: one 16-byte word of each part.
__global__ void __launch_bounds__(256)
    zgen_kernel(const int4* __restrict__ fx, int32_t n_list, int32_t n_chunks, int32_t nzr,
                unsigned char* __restrict__ zbuf) {
  __shared__ int32_t qz[TC_J];
  const int c = blockIdx.x, f = blockIdx.y;
  const int live = n_list - c * TC_J;  // atoms of this chunk
  if (threadIdx.x < TC_J) qz[threadIdx.x] = (int)threadIdx.x < live ? fx[(int64_t)f * n_list + c * TC_J + threadIdx.x].z : 0;
  __syncthreads();
  const size_t part = (size_t)nzr * TC_ZROW;
  unsigned char* out = zbuf + ((size_t)f * n_chunks + c) * 4 * part;
  for (int e = threadIdx.x; e < nzr * (TC_J / 4); e += blockDim.x) {
    const int z = e >> 3, j0 = 4 * (e & 7);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float s = 0.f, co = 0.f;
      if (j0 + i < live) tc_phase((int32_t)((uint32_t)z * (uint32_t)qz[j0 + i]), &s, &co);
      __half rh, rl, ih, il;
      tc_split(co, rh, rl);
      tc_split(s, ih, il);
      const __half2 h = __halves2half2(rh, ih), l = __halves2half2(rl, il);
      hi[i] = *reinterpret_cast<const uint32_t*>(&h);
      lo[i] = *reinterpret_cast<const uint32_t*>(&l);
    }
    unsigned char* o = out + umma::kmajor_sw128_offset(z, 2 * j0);
    constexpr uint32_t S = 0x80000000u;  // the sign of the imaginary half
    *reinterpret_cast<uint4*>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(o + part) = make_uint4(hi[0] ^ S, hi[1] ^ S, hi[2] ^ S, hi[3] ^ S);
    *reinterpret_cast<uint4*>(o + 2 * part) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(o + 3 * part) = make_uint4(lo[0] ^ S, lo[1] ^ S, lo[2] ^ S, lo[3] ^ S);
  }
}

// X and Y phase tables of one frame batch, exp(i 2 pi n q_j) of 32 atoms and eight
// lattice indices (X: n = 8 b + m, Y: n = -nmax + 8 b + m) in TC_XB bytes per (block,
// chunk): float4 ((2 u + i) * 8 + m) * 4 + c = (cos, cos', sin, sin') of the atoms
// 16 u + 8 i + c and 4 on, in the order the builder threads read them
__global__ void __launch_bounds__(256)
    xygen_kernel(const int4* __restrict__ fx, int32_t n_list, int32_t n_chunks, int32_t n_xb, int32_t n_yb,
                 int32_t nmax, float4* __restrict__ xbuf, float4* __restrict__ ybuf) {
  __shared__ int2 qxy[TC_J];
  const int c = blockIdx.x, f = blockIdx.y;
  const int live = n_list - c * TC_J;
  if (threadIdx.x < TC_J) {
    const int4 q = (int)threadIdx.x < live ? fx[(int64_t)f * n_list + c * TC_J + threadIdx.x] : make_int4(0, 0, 0, 0);
    qxy[threadIdx.x] = make_int2(q.x, q.y);
  }
  __syncthreads();
  constexpr int PER = TC_XB / 16;  // float4 of a block
  for (int e = threadIdx.x; e < PER * (n_xb + n_yb); e += blockDim.x) {
    const int blk = e / PER, w = e % PER, m = (w >> 2) & 7, j = 8 * (w >> 5) + (w & 3);
    const bool is_x = blk < n_xb;
    const int b = is_x ? blk : blk - n_xb;
    const int32_t n = is_x ? 8 * b + m : 8 * b + m - nmax;
    float s[2] = {0.f, 0.f}, co[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int2 q = qxy[j + 4 * i];
      if (j + 4 * i < live) tc_phase((int32_t)((uint32_t)n * (uint32_t)(is_x ? q.x : q.y)), &s[i], &co[i]);
    }
    float4* out = is_x ? xbuf + (((size_t)f * n_xb + b) * n_chunks + c) * PER : ybuf + (((size_t)f * n_yb + b) * n_chunks + c) * PER;
    out[w] = make_float4(co[0], co[1], s[0], s[1]);
  }
}

// bounded wait of a whole warp (false: give up); the block's error flag is read only
// when the phase is not complete yet
__device__ __forceinline__ bool warp_wait(uint64_t* mbar, uint32_t parity, volatile int* bad) {
  if (__all_sync(0xffffffffu, umma::mbar_try_wait(mbar, parity, 1000))) return true;
  bool ok = false;
  for (uint32_t i = 0; i < TC_WAIT && !ok && !*bad; ++i) ok = umma::mbar_try_wait(mbar, parity, 1000);
  return __all_sync(0xffffffffu, ok) != 0;
}

static_assert(TC_GROUP == 2 && TC_ZS == 2 * TC_GROUP, "a ring cycle holds one group of each accumulator");
// position in the ring and the parity of its current use.  A parity wait is sound
// only for a waiter that saw the barrier's phase before and that the barrier cannot
// run two phases ahead of: every barrier here has its phases seen in turn by each
// of its waiters, and its next phase but one needs the waiter's own progress
struct TcSlot {
  int s = 0;
  uint32_t ph;
  __device__ explicit TcSlot(uint32_t first) : ph(first) {}
  __device__ void next(int n) {
    if (++s == n) {
      s = 0;
      ph ^= 1u;
    }
  }
};

// the barrier that completes (phase c / 4) when the MMAs of chunk c have finished
__device__ __forceinline__ uint64_t* chunk_done(TcHdr& S, int c) {
  return c & 1 ? &S.full_acc[(c >> 1) & 1] : &S.half_done[(c >> 1) & 1];
}

__global__ void __launch_bounds__(TC_THREADS, 1)
    rhok_tc_kernel(int32_t n_chunks, int32_t nzr, int32_t nzw, int32_t n_xb, int32_t n_yb, int32_t nmax,
                   const HalfTile* __restrict__ tiles, const int2* __restrict__ entry_k,
                   const unsigned char* __restrict__ zbuf, const float4* __restrict__ xbuf,
                   const float4* __restrict__ ybuf, int32_t frame0, int32_t n_k, float2* __restrict__ rho,
                   int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                         ~(uintptr_t)1023);
  TcHdr& S = *reinterpret_cast<TcHdr*>(base);
  unsigned char* ring = base + TC_HDR;  // TC_ZS stages of zstage bytes
  const HalfTile T = tiles[blockIdx.x];
  const int fl = blockIdx.y;  // frame within the batch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = T.n, n2 = 2 * T.n;
  const uint32_t zhalf = 2u * (uint32_t)nzw * TC_ZROW, zstage = tc_zstage(nzw);
  // A stages: two or four (even, so that the chunk a stage was used for last was built by
  // the same warpgroup, which therefore sees that chunk's barrier phases in turn)
  const int n_as = 2 * n2 + TC_AS_MAX * (int)TC_A_COLS <= (int)TC_TMEM_COLS ? TC_AS_MAX : 2;
  const int n_groups = (n_chunks + TC_GROUP - 1) / TC_GROUP;

  if (tid == 0) {
    for (int s = 0; s < TC_ZS; ++s) umma::mbar_init(&S.full_z[s], 1);
    for (int s = 0; s < 2 * TC_GROUP; ++s) umma::mbar_init(&S.full_a[s], TC_BUILD_WARPS / 2);
    for (int b = 0; b < 2; ++b) {
      umma::mbar_init(&S.half_done[b], 1);
      umma::mbar_init(&S.full_acc[b], 1);
      umma::mbar_init(&S.empty_acc[b], TC_DRAIN_WARPS);
    }
    umma::mbar_init(&S.mma_done, TC_MMA_WARPS);
    umma::fence_mbarrier_init();
    S.bad = 0;
    S.z_issued = 0;
  }
  if (warp == 0) {
    umma::tmem_alloc(&S.tmem, TC_TMEM_COLS);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = S.tmem;
  const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;  // this warp's tensor-memory lane quadrant
  const uint32_t col_a = 2u * (uint32_t)n2;                  // first column of the A stages

  if (warp >= TC_BUILD_WARP0) {
    umma::reg_dec<TC_REG_BUILD>();
    // ---- builders: A(c) = the chunk's W products into tensor-memory stage c % n_as.
    // Thread t of the warp: nx offset m = t / 4, ny offsets 2 (warp % 4) + h (h = 0, 1),
    // atoms 16 u + 4 i + t % 4 (u < 2, i < 4); packed FP32 over the atom pairs i = 0, 1
    // and 2, 3.  The two warpgroups take alternate chunks, so one's hand-offs overlap
    // the other's products
    const int first = (warp - TC_BUILD_WARP0) >> 2;  // even or odd chunks
    for (int c = first; c < n_chunks; c += 2) {
      const int zs = c % TC_ZS;
      if (!warp_wait(&S.full_z[zs], (c / TC_ZS) & 1, &S.bad)) {
        S.bad = 1;
        break;
      }
      const unsigned char* st = ring + (size_t)zs * zstage + 2 * zhalf;
      const float4* X4 = reinterpret_cast<const float4*>(st) + lane;
      const float4* Y4 = reinterpret_cast<const float4*>(st + TC_XB) + 8 * (warp & 3) + (lane & 3);
      const uint32_t col = tmem + lanes + col_a + (uint32_t)(c % n_as) * TC_A_COLS;
      bool ok = true;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        // per ny offset: columns i (hi) and 4 + i (lo) of [Wr, -Wi] (even) and [Wi, Wr] (odd)
        uint32_t a[2][16];
#pragma unroll
        for (int ip = 0; ip < 2; ++ip) {
          const float4 x = X4[64 * u + 32 * ip];
          const uint64_t xc = pk2(x.x, x.y), xs = pk2(x.z, x.w), xn = pk2(-x.z, -x.w);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 y = Y4[64 * u + 32 * ip + 4 * h];
            const uint64_t yc = pk2(y.x, y.y), ys = pk2(y.z, y.w);
            float rh[2], rl[2], ih[2], il[2];
            tc_split2(fma2(xc, yc, mul2(xn, ys)), rh, rl);  // Wr = xc yc - xs ys
            tc_split2(fma2(xs, yc, mul2(xc, ys)), ih, il);  // Wi = xs yc + xc ys
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int i = 2 * ip + k;
              const uint32_t hi = tc_half2(rh[k], ih[k]), lo = tc_half2(rl[k], il[k]);
              a[h][2 * i] = hi ^ 0x80000000u;
              a[h][2 * i + 1] = __byte_perm(hi, 0, 0x1032);
              a[h][8 + 2 * i] = lo ^ 0x80000000u;
              a[h][9 + 2 * i] = __byte_perm(lo, 0, 0x1032);
            }
          }
        }
        if (u == 0) {
          // the stores wait for the MMAs of the chunk that used the stage last
          const int pc = c - n_as;
          ok = pc < 0 || warp_wait(chunk_done(S, pc), (pc >> 2) & 1, &S.bad);
          if (!ok) break;
          umma::fence_after_sync();
        }
        umma::tmem_st_16x128b_x8(col + 32u * u, a[0]);
        umma::tmem_st_16x128b_x8(col + 32u * u + (16u << 16), a[1]);
      }
      if (!ok) {
        S.bad = 1;
        break;
      }
      umma::tmem_st_wait();
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&S.full_a[zs]);
    }
  } else if (warp >= TC_DRAIN_WARPS) {
    umma::reg_dec<TC_REG_MISC>();
    if (warp == TC_PRODUCER_WARP) {
      // ---- producer: Z(c), X(c), Y(c) into a ring stage once the MMAs of its last chunk are done
      const size_t part = (size_t)nzr * TC_ZROW;
      const unsigned char* Z = zbuf + (size_t)fl * n_chunks * 4 * part + (size_t)T.z0 * TC_ZROW;
      const unsigned char* XT =
          reinterpret_cast<const unsigned char*>(xbuf) + ((size_t)fl * n_xb + T.nx0 / 8) * (size_t)n_chunks * TC_XB;
      const unsigned char* YT = reinterpret_cast<const unsigned char*>(ybuf) +
                                ((size_t)fl * n_yb + (T.ny0 + nmax) / 8) * (size_t)n_chunks * TC_XB;
      const uint32_t zb = (uint32_t)n * TC_ZROW;
      TcSlot z(0);
      int c = 0;
      for (; c < n_chunks; ++c) {
        // the stage is free once the MMAs of its last chunk are done
        if (c >= TC_ZS && !warp_wait(chunk_done(S, c - TC_ZS), ((c - TC_ZS) >> 2) & 1, &S.bad)) {
          S.bad = 1;
          break;
        }
        if (umma::elect_one()) {
          unsigned char* dst = ring + (size_t)z.s * zstage;
          const unsigned char* src = Z + (size_t)c * 4 * part;
          uint64_t* full = &S.full_z[z.s];
          umma::mbar_expect_tx(full, 4u * zb + TC_XYB);
          umma::bulk_g2s(dst + 2 * zhalf, XT + (size_t)c * TC_XB, TC_XB, full);
          umma::bulk_g2s(dst + 2 * zhalf + TC_XB, YT + (size_t)c * TC_XB, TC_XB, full);
          umma::bulk_g2s(dst, src, zb, full);
          umma::bulk_g2s(dst + zb, src + part, zb, full);
          umma::bulk_g2s(dst + zhalf, src + 2 * part, zb, full);
          umma::bulk_g2s(dst + zhalf + zb, src + 3 * part, zb, full);
        }
        __syncwarp();
        z.next(TC_ZS);
      }
      S.z_issued = c;
    } else if (warp < TC_MMA_WARP + TC_MMA_WARPS) {
      // ---- MMA issuers: warp TC_MMA_WARP + b issues the groups of accumulator b
      // (even / odd groups): one waits for its operands while the other's MMAs run
      const int mine = warp - TC_MMA_WARP;
      const uint32_t idesc = umma::idesc_f16_f32(TC_M, n2);
      // the B descriptor's address field is the byte address >> 4 (14 bits, all
      // of shared memory), so the ring stage, the lo half (both 1024-byte
      // aligned) and the k-step (32 B inside the swizzled 128-byte rows) add to
      // it; k-step ks (atoms 8 ks .. 8 ks + 7) of the A stage is column
      // 32 (ks / 2) + 8 (ks % 2), its lo part 16 columns on
      const uint64_t b_desc0 = umma::smem_desc_sw128(umma::smem_addr(ring));
      const uint32_t b_lo16 = zhalf >> 4;
      TcSlot z(0);
      int as = 0;
      bool ok = true;
      for (int c = 0; c < n_chunks; ++c) {
        const int g = c / TC_GROUP, buf = g & 1;
        if (buf != mine) {
          z.next(TC_ZS);
          if (++as == n_as) as = 0;
          continue;
        }
        if ((c % TC_GROUP == 0 && !warp_wait(&S.empty_acc[buf], ((g >> 1) & 1) ^ 1, &S.bad)) ||
            !warp_wait(&S.full_z[z.s], z.ph, &S.bad) || !warp_wait(&S.full_a[z.s], z.ph, &S.bad)) {
          ok = false;
          break;
        }
        umma::fence_after_sync();
        const uint32_t d = tmem + (uint32_t)(buf * n2);
        const uint32_t a = tmem + col_a + (uint32_t)as * TC_A_COLS;
        const uint64_t bd = b_desc0 + (uint64_t)((uint32_t)z.s * (zstage >> 4));
        // small cross terms first, then hi*hi, so the accumulator is still small
        // while the 2^-11-sized terms are added; an accumulator's first group
        // starts from zero, later ones from the residual the drain left
        const uint32_t first = c < TC_GROUP * 2 && c % TC_GROUP == 0 ? 0u : 1u;
        if (umma::elect_one()) {
#pragma unroll
          for (int pass = 0; pass < 3; ++pass)
#pragma unroll
            for (int ks = 0; ks < TC_K / 16; ++ks)
              umma::mma_f16_tmem_a(d, a + (uint32_t)((pass == 1 ? 16 : 0) + 32 * (ks / 2) + 8 * (ks % 2)),
                                   bd + (uint64_t)((pass == 0 ? b_lo16 : 0u) + 2u * ks), idesc,
                                   (pass == 0 && ks == 0) ? first : 1u);
          // a commit costs the pipe ~50 cycles: one per chunk
          umma::mma_commit(c % TC_GROUP == TC_GROUP - 1 || c == n_chunks - 1 ? &S.full_acc[buf] : &S.half_done[buf]);
        }
        __syncwarp();
        z.next(TC_ZS);
        if (++as == n_as) as = 0;
      }
      if (!ok) S.bad = 1;
      // every MMA the warp's lane issued has finished once mma_done completes
      if (umma::elect_one()) umma::mma_commit(&S.mma_done);
      __syncwarp();
      if (!umma::mbar_wait(&S.mma_done, 0, TC_WAIT)) S.bad = 1;
    }
  } else {
    umma::reg_inc<TC_REG_DRAIN>();
    // ---- drain: accumulator of group g -> compensated register sums.  Warp w
    // owns lane quadrant w % 4 and the 16-column blocks TC_DRAIN_PAR i + w / 4:
    // s += acc by Fast2Sum on packed FP32 pairs, the rounding residual goes back
    // into the accumulator
    const int par = warp >> 2;
    constexpr int NB = 2 * TC_NZMAX / 16 / TC_DRAIN_PAR;  // column blocks per warp
    uint64_t sp[NB][8];  // column pairs of the sums
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int k = 0; k < 8; ++k) sp[i][k] = 0ull;
    bool ok = true;
    for (int g = 0; g < n_groups; ++g) {
      const int buf = g & 1;
      if (!warp_wait(&S.full_acc[buf], (g >> 1) & 1, &S.bad)) {
        ok = false;
        break;
      }
      umma::fence_after_sync();
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int cb = 16 * (TC_DRAIN_PAR * i + par);
        if (cb < n2) {
          uint32_t v[16];  // accumulator in, residual out
          const uint32_t col = tmem + lanes + (uint32_t)(buf * n2 + cb);
          umma::tmem_ld_32x32b_x16(col, v);
          umma::tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            // Fast2Sum: t = s + a, e = a - (t - s), exact while |s| >= |a|; when
            // a 64-atom partial outweighs the running sum the residual may lose
            // about an ulp of the partial (~1e-6), far inside the error bounds
            const uint64_t s2 = sp[i][k];
            const uint64_t a2 = pk2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
            const uint64_t t2 = add2(s2, a2);
            const uint64_t e2 = sub2(a2, sub2(t2, s2));
            sp[i][k] = t2;
            float e0, e1;
            upk2(e2, e0, e1);
            v[2 * k] = __float_as_uint(e0);
            v[2 * k + 1] = __float_as_uint(e1);
          }
          umma::tmem_st_32x32b_x16(col, v);
        }
      }
      umma::tmem_st_wait();
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&S.empty_acc[buf]);
    }
    if (ok && n_groups > 0) {
      // epilogue: the sums into the D staging area, rows of n2 + 1 floats (the
      // ring is idle: every copy was consumed by an MMA that completed before
      // the last group's commit)
      float* D = reinterpret_cast<float*>(ring) + (size_t)(32 * (warp & 3) + lane) * (n2 + 1);
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int cb = 16 * (TC_DRAIN_PAR * i + par);
        if (cb < n2)
#pragma unroll
          for (int k = 0; k < 8; ++k) upk2(sp[i][k], D[cb + 2 * k], D[cb + 2 * k + 1]);
      }
    }
    if (!ok) S.bad = 1;
  }

  __syncthreads();
  if (S.bad) {
    // copies still in flight land before the block exits
    // (the last copy issued into each stage; earlier ones were waited for)
    if (tid == 32 * TC_PRODUCER_WARP)
      for (int c = std::max(0, S.z_issued - TC_ZS); c < S.z_issued; ++c)
        umma::mbar_wait(&S.full_z[c % TC_ZS], (c / TC_ZS) & 1, TC_WAIT);
    if (tid == 0) atomicExch(err, 1);
  } else if (n_groups > 0) {
    const int DP = n2 + 1;
    const float* D = reinterpret_cast<const float*>(ring);
    const int2* E = entry_k + T.entry0;
    float2* out = rho + (int64_t)(frame0 + fl) * n_k;
    for (int e = tid; e < TC_ROWS * n; e += TC_THREADS) {
      const int2 k = E[e];
      if ((k.x & k.y) == -1) continue;  // no vector here
      const int r = e / n, col = e - r * n;
      const float* R = D + (size_t)(16 * (r >> 3) + (r & 7)) * DP + col;
      if (k.x >= 0) out[k.x] = make_float2(R[0], R[8 * DP]);
      if (k.y >= 0) out[k.y] = make_float2(R[n], -R[8 * DP + n]);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, TC_TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// host: tile plan over the shell-sorted vector list, launches per frame batch
// ---------------------------------------------------------------------------
HalfPlan* half_plan_build(amdat_ctx* ctx, const std::vector<int32_t>& kvec) {
  // the register split draws on what the block is launched with: a kernel compiled to fewer
  // would wait for registers that never come
  cudaFuncAttributes attr;
  AMDAT_CUDA(cudaFuncGetAttributes(&attr, rhok_tc_kernel));
  if (attr.numRegs * TC_THREADS < 256 * TC_REG_DRAIN + 128 * TC_REG_MISC + 256 * TC_REG_BUILD)
    throw Error(AMDAT_ERR_CUDA, "rhok_tc_kernel was compiled to too few registers for its split");
  int nmax = 0;
  for (int v : kvec) nmax = std::max(nmax, std::abs(v));
  const LatticeIndex index(kvec, nmax);
  std::vector<HalfTile> tiles;
  std::vector<int2> entries;
  int nzw = 8;
  for (int x0 = 0; x0 <= nmax; x0 += 8)
    for (int y0 = -nmax; y0 <= nmax; y0 += 8) {
      auto images = [&](int r, int nz) { return index.images(x0 + (r & 7), y0 + (r >> 3), nz); };
      int ext = 0;  // nz extent of the 64 rows
      for (int z = nmax; z >= 0 && !ext; --z)
        for (int r = 0; r < TC_ROWS && !ext; ++r) {
          const int2 k = images(r, z);
          if (k.x >= 0 || k.y >= 0) ext = z + 1;
        }
      if (!ext) continue;
      // equal nz windows of at most TC_NZMAX, multiples of 8
      const int nw = (ext + TC_NZMAX - 1) / TC_NZMAX;
      const int w = (int)ceil_div(ceil_div(ext, nw), 8) * 8;
      for (int z0 = 0; z0 < ext; z0 += w) {
        const int n = std::min(w, (int)ceil_div(ext - z0, 8) * 8);
        nzw = std::max(nzw, n);
        tiles.push_back(HalfTile{x0, y0, z0, n, (int32_t)entries.size()});
        for (int r = 0; r < TC_ROWS; ++r)
          for (int c = 0; c < n; ++c) entries.push_back(images(r, z0 + c));
        AMDAT_REQUIRE(entries.size() < (size_t)INT32_MAX, "lattice too large for the tensor-core tiling");
      }
    }
  // the widest tiles first: the last wave of a launch ends on short ones
  std::stable_sort(tiles.begin(), tiles.end(), [](const HalfTile& a, const HalfTile& b) { return a.n > b.n; });
  auto* p = new HalfPlan();
  try {
    p->n_tiles = (int32_t)tiles.size();
    p->nzw = nzw;
    p->nmax = nmax;
    p->tiles.reserve(std::max<size_t>(tiles.size(), 1));
    p->entry_k.reserve(std::max<size_t>(entries.size(), 1));
    upload_tables(ctx, {{p->tiles.ptr, tiles.data(), tiles.size() * sizeof(HalfTile)},
                        {p->entry_k.ptr, entries.data(), entries.size() * sizeof(int2)}});
  } catch (...) {
    delete p;
    throw;
  }
  return p;
}

void half_plan_free(HalfPlan* p) { delete p; }

// rho[f][k] for frames 0..n_frames-1 of fx ([n_frames][n_list] fixed-point phases)
void rhok_tc_run(amdat_ctx* ctx, const HalfPlan& P, const int4* fx, int32_t n_list, int32_t n_frames,
                 int32_t n_k, float2* rho) {
  if (P.n_tiles == 0 || n_list == 0 || n_frames == 0) return;
  const int32_t n_chunks = (int32_t)ceil_div(n_list, TC_J);
  const int32_t n_xb = P.nmax / 8 + 1, n_yb = 2 * P.nmax / 8 + 1;  // 8-index blocks from 0 and from -nmax
  // nz rows of a Z part: every tile's window lies inside (windows end at a multiple of 8 of their start)
  const int32_t nzr = (int32_t)ceil_div(P.nmax + 1, 8) * 8 + 8;
  const size_t z_frame = (size_t)n_chunks * 4 * nzr * TC_ZROW;
  const size_t x_frame = (size_t)n_xb * n_chunks * TC_XB, y_frame = (size_t)n_yb * n_chunks * TC_XB;
  const size_t per_frame = z_frame + x_frame + y_frame;
  // frame batches bound the operand buffers to ~1 GB
  const int32_t batch = (int32_t)std::max<size_t>(1, std::min<size_t>(n_frames, (size_t)(1u << 30) / per_frame));
  unsigned char* zbuf = ctx->scratch.reserve(per_frame * batch + 256);
  float4* xbuf = reinterpret_cast<float4*>(zbuf + z_frame * batch);
  float4* ybuf = reinterpret_cast<float4*>(zbuf + (z_frame + x_frame) * batch);
  int* d_err = (int*)(zbuf + per_frame * batch);
  AMDAT_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
  // the ring beside the barrier header (1024 bytes of alignment slack); the
  // epilogue stages D (128 rows of 2n + 1 floats) in the idle ring
  const size_t ring = (size_t)TC_ZS * tc_zstage(P.nzw);
  const size_t shm = 1024 + TC_HDR + ring;
  AMDAT_REQUIRE(P.nzw <= TC_NZMAX && shm <= TC_SMEM_MAX, "nz window too wide for the tensor-core ring");
  AMDAT_REQUIRE(ring >= sizeof(float) * TC_M * (2 * P.nzw + 1), "ring too small for the D staging");
  AMDAT_REQUIRE(n_chunks <= INT32_MAX / 4 && batch <= 65535, "too many atoms or frames for one launch");
  AMDAT_CUDA(cudaFuncSetAttribute(rhok_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  for (int32_t f0 = 0; f0 < n_frames; f0 += batch) {
    const int32_t nb = std::min(batch, n_frames - f0);
    const dim3 gen((unsigned)n_chunks, (unsigned)nb);
    zgen_kernel<<<gen, 256, 0, ctx->stream>>>(fx + (int64_t)f0 * n_list, n_list, n_chunks, nzr, zbuf);
    check_launch("zgen_kernel");
    count_launch(ctx);
    xygen_kernel<<<gen, 256, 0, ctx->stream>>>(fx + (int64_t)f0 * n_list, n_list, n_chunks, n_xb, n_yb, P.nmax,
                                               xbuf, ybuf);
    check_launch("xygen_kernel");
    count_launch(ctx);
    KernelTimer kt(ctx, "rhok_tc_kernel");
    dim3 grid((unsigned)P.n_tiles, (unsigned)nb);
    rhok_tc_kernel<<<grid, TC_THREADS, shm, ctx->stream>>>(n_chunks, nzr, P.nzw, n_xb, n_yb, P.nmax, P.tiles.ptr,
                                                          P.entry_k.ptr, zbuf, xbuf, ybuf, f0, n_k, rho, d_err);
    check_launch("rhok_tc_kernel");
    count_launch(ctx);
  }
  int h_err = 0;
  AMDAT_CUDA(cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  AMDAT_CUDA(cudaStreamSynchronize(ctx->stream));
  if (h_err) throw Error(AMDAT_ERR_TIMEOUT, "tensor-core rho_k: a bounded wait timed out");
}

}  // namespace amdat
