/*
 * fdtd_tile.cuh -- what the TMA pipelines over x-y tiles share
 * (fdtd_tma.cu's half-step kernels, fdtd_flow.cu's multi-step kernel): the
 * warps of a block, the tile geometries with their stage layouts, the
 * batched stages' descriptor slots and the thread-to-cell map.
 */
#pragma once
#include <cuda.h>
#include <stdint.h>

#include <type_traits>

#include "fdtd_internal.h"

namespace fdtd_tile {

constexpr int NCW = 8;                       // consumer warps
constexpr int NT = (NCW + 1) * 32;           // + one producer warp
// Tile geometry: a work item is a BX x BY tile of cells over a run of
// z-planes.  The single-grid kernels use 64 x 8; the batched ones 32 x 16,
// since their grids are narrow (32..128 cells in x) and a 64-wide tile of a
// 70-cell axis leaves most lanes of its second tile idle.  Both have the
// same stage byte sizes.
template <int BX_, int BY_>
struct Geo {
  static constexpr int BX = BX_, BY = BY_;
  static constexpr int LX = BX == 32 ? 5 : (BX == 64 ? 6 : 7), LY = 9 - LX;  // log2
  static constexpr int HW = BX + 4;                   // halo box row (floats)
  static constexpr int HH = BY + 1;                   // halo box rows
  static constexpr int TILE_B = BX * BY * 4;          // 2048 B
  static constexpr int HALO_B = HW * HH * 4;          // bytes transferred
  static constexpr int HALO_SLOT = (HALO_B + 127) / 128 * 128;  // 128-byte aligned slot
  static constexpr int MAT_B = BX * BY * 2;           // 1024 B
  static constexpr int E_OFF_H = 3 * TILE_B;
  static constexpr int E_OFF_M = E_OFF_H + 3 * HALO_SLOT;
  static constexpr int E_STAGE = E_OFF_M + MAT_B;
  static constexpr int H_OFF_H = 3 * HALO_SLOT;
  static constexpr int H_STAGE = H_OFF_H + 3 * TILE_B;
  static_assert(BX % 32 == 0 && (256 / 32) % (BX / 32) == 0 && BX * BY == 512,
                "8 consumer warps, two cells per thread");
  static_assert(E_STAGE % 128 == 0 && H_STAGE % 128 == 0, "stage alignment");
  static_assert((HW * 4) % 16 == 0 && (BX * 4) % 16 == 0 && (BX * 2) % 16 == 0,
                "TMA inner box extents must be multiples of 16 bytes");
};
using GS = Geo<64, 8>;   // single-grid kernels (tile 0, the default)
using GB = Geo<32, 16>;  // batched kernels; single-grid tile 1 (narrow grids)
using GW = Geo<128, 4>;  // single-grid tile 2 (wide grids)
// The single-grid tile geometry by index (fdtd_dev::tile_e / tile_h).
template <int T>
using TileGeo = typename std::conditional<T == 0, GS,
                                          typename std::conditional<T == 1, GB, GW>::type>::type;
constexpr int kSmemTabMax = 512;             // coefficient ids staged in shared memory
constexpr int CTRL_B = 512;                  // barriers + stage metadata
// Batch mode: every stage also carries its grid's descriptor and op (bulk
// copies completing on the stage's barrier), so the per-cell code reads
// them from shared memory instead of global memory; E stages also carry
// the grid's coefficient table when it has at most kStageTabMax ids.
constexpr int DESC_B = 1536;                 // >= sizeof(fdtd_dev), 128-aligned
constexpr int OPSLOT_B = 128;                // >= sizeof(fdtd_op)
constexpr int kStageTabMax = 64;
constexpr int TAB_B = kStageTabMax * 6 * 4;  // 1536 B
static_assert(sizeof(fdtd_dev) <= DESC_B && sizeof(fdtd_dev) % 16 == 0, "descriptor slot");
static_assert(sizeof(fdtd_op) <= OPSLOT_B && sizeof(fdtd_op) % 16 == 0, "op slot");
struct Maps {
  CUtensorMap m[FDTD_NUM_MAPS];
};

// Thread -> cell map of the consumer warps: warp w covers one 32-cell x run
// (run w % (BX/32) of the tile's row) of rows r0 = w / (BX/32) and
// r0 + BY/2, so that whole warps fall inside or outside the CPML x slabs and
// TF/SF x faces.
template <class G>
__device__ __forceinline__ void cell_map(int tid, int &xo, int &r0) {
  constexpr int WPR = G::BX / 32;  // warps per tile row
  const int w = tid >> 5;
  xo = 32 * (w % WPR) + (tid & 31);
  r0 = w / WPR;
}

}  // namespace fdtd_tile
