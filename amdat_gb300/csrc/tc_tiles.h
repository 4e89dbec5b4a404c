// Tilings of a half-space lattice for the tensor-core kernels.  Both cut half the
// (nx, ny) plane into squares of 8 nx >= 0 x 8 ny, a row standing for (nx, ny) and
// (-nx, -ny): the forward rho_k kernel's tiles cover nz windows trimmed to a multiple
// of 8, the S(k) adjoint's nz windows trimmed to a multiple of 16.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "engine.h"

namespace amdat {

// (nx, ny, nz) -> position in a half-space vector list, -1 when it is not listed
struct LatticeIndex {
  int nmax;
  std::vector<int32_t> at;
  LatticeIndex(const std::vector<int32_t>& kvec, int nmax_) : nmax(nmax_) {
    const size_t W = 2 * (size_t)nmax + 1, H = (size_t)nmax + 1;
    at.assign(W * W * H, -1);
    for (size_t k = 0; k < kvec.size() / 3; ++k) {
      const int x = kvec[3 * k], y = kvec[3 * k + 1], z = kvec[3 * k + 2];
      AMDAT_REQUIRE(z > 0 || (z == 0 && (y > 0 || (y == 0 && x > 0))), "lattice vector outside the half space");
      at[((size_t)(x + nmax) * W + (size_t)(y + nmax)) * H + (size_t)z] = (int32_t)k;
    }
  }
  int32_t operator()(int x, int y, int z) const {
    if (x < -nmax || x > nmax || y < -nmax || y > nmax || z < 0 || z > nmax) return -1;
    const size_t W = 2 * (size_t)nmax + 1, H = (size_t)nmax + 1;
    return at[((size_t)(x + nmax) * W + (size_t)(y + nmax)) * H + (size_t)z];
  }
  // the vectors (x, y, z) and (-x, -y, z) of a half-plane row x >= 0 (of x = 0 the rows y >= 0 carry both)
  int2 images(int x, int y, int z) const {
    if (x == 0 && y < 0) return make_int2(-1, -1);
    return make_int2((*this)(x, y, z), x || y ? (*this)(-x, -y, z) : -1);
  }
};

// one half-plane tile: rows (nx0 + r % 8, ny0 + r / 8), r < 64, nz = z0 + c, c < n
struct HalfTile {
  int32_t nx0, ny0, z0;
  int32_t n;       // nz columns of this tile (multiple of 8, <= 96)
  int32_t entry0;  // entry map: 64 rows x n int2 from entry0: the vectors (nx, ny, nz) and (-nx, -ny, nz), or -1
};

struct HalfPlan {
  DevBuf<HalfTile> tiles;
  DevBuf<int2> entry_k;
  int32_t n_tiles = 0, nzw = 0, nmax = 0;  // nzw: the widest tile's n
};

HalfPlan* half_plan_build(amdat_ctx* ctx, const std::vector<int32_t>& kvec);
void half_plan_free(HalfPlan* p);

struct TcTile {
  int32_t nx0, ny0, zblk, entry0;  // entry map: 64 rows x n int2 from entry0, as HalfTile's
  int32_t n;                       // nz columns of this tile (multiple of 16, <= 128)
};

struct TcPlan {
  DevBuf<TcTile> tiles;
  DevBuf<int2> entry_k;
  std::vector<TcTile> host_tiles;
  int32_t n_tiles = 0, n_zblk = 0, nzw = 0, nmax = 0;
};

TcPlan* tc_plan_build(amdat_ctx* ctx, const std::vector<int32_t>& kvec);
void tc_plan_free(TcPlan* p);
// the tensor-core tiling of a lattice density's plan (built at first use)
TcPlan* lattice_tc_plan(amdat_ctx* ctx, const std::string& lattice_key);
// whether the tensor-core kernels run (compute capability 10.x and not
// disabled through AMDAT_RHOK_KERNEL=fp32)
bool tc_enabled(amdat_ctx* ctx);

}  // namespace amdat
