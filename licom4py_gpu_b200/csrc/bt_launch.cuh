// bt_launch.cuh - host-side launch interface of the barotropic kernels (internal C++).
#pragma once

#include <string>

#include "bt_common.cuh"
#include "bt_stencil.cuh"

namespace bt {

// Record the thread-local message returned by bt_last_error(); returns code.
int set_error(int code, const std::string& msg);

struct TileCfg {
  int ti, tj;
};

// Tile shapes compiled into the library (rows x columns of interior cells).
bool tile_cfg_supported(TileCfg c);
// Tile constant blocks (Geo::cblk) for tile shape c (even: the even split):
// elements needed, and a stream-ordered build from the constant arrays of g.
size_t const_block_elems(TileCfg c, int n);
template <typename T>
cudaError_t launch_const_blocks(const Geo<T>& g, TileCfg c, bool even, T* out, cudaStream_t s);
// Elements of the momentum terms of one member at n cells per face edge in a
// type of esize bytes: enough for every supported tile shape (the plan's tile
// can change later), and for the planes of the 8 x 16 tiles alone.
size_t terms_elems(int n, size_t esize);
inline size_t terms_plane_elems(int n, size_t esize) { return (esize == 8 ? 6 : 2) * (size_t)6 * n * n; }
// Elements of the bands of one member (velocity: 3 planes, h: 2, or 3 with the fused stage kernel).
inline size_t band_elems(int n, bool fused = false) { return (fused ? 6 : 5) * (size_t)72 * n; }
Tiling make_tiling(TileCfg c, int n);
Tiling make_even_tiling(TileCfg c, int n);

// Set kernel attributes (dynamic shared memory opt-in) for the current device.
template <typename T>
cudaError_t prime_kernels();
// Phase kernels of one stage.  full_tiles selects the kernel: 1 = the one with
// the full-interior-tile path, 0 = edge path only, -1 = by size (the edge-only
// kernel when the launch's CTAs all fit on the device at once).  Results are
// the same either way.
template <typename T>
cudaError_t launch_phase_h(const Geo<T>& g, const StageIO<T>& io, TileCfg cfg, cudaStream_t s, int full_tiles = -1,
                           bool overlap = true);
// Which kernels those launches take at n: bit 0 set = phase H runs the full-tile
// kernel, bit 1 = phase UV (-1: unsupported tile shape).
template <typename T>
int phase_full_paths(TileCfg cfg, int n, int full_tiles);
template <typename T>
cudaError_t launch_phase_uv(const Geo<T>& g, const StageIO<T>& io, TileCfg cfg, cudaStream_t s, int full_tiles = -1);
// The fused stage kernel (bt_fused.cuh), the tile shape of the phases around it (and of its own tiles, except
// where fused_tile gives a wider one), and the tables of decoded work it reads (built once per plan, stream
// ordered).  alone: rounds of other plans are not expected beside this one (spread_smem).
constexpr TileCfg kFusedTile{8, 16};
TileCfg fused_tile(int n);
template <typename T>
struct FusedIO;
size_t stage_table_bytes(int n, size_t esize);
template <typename T>
cudaError_t launch_stage_tables(const Geo<T>& g, void* out, cudaStream_t s);
template <typename T>
cudaError_t launch_stage(const Geo<T>& g, const FusedIO<T>& p, const void* tables, bool alone, cudaStream_t s);
// Persistent cooperative launch of a whole round (phases of all substeps);
// max_ctas > 0 caps the grid.  The grid size used is returned in *grid_out.
template <typename T>
cudaError_t launch_round(const RoundArgs<T>& a, TileCfg cfg, int max_ctas, cudaStream_t s, int* grid_out);
// Tile-resident round (one CTA per tile, neighbour flags; bt_resident.cuh).
bool resident_tile_supported(TileCfg c);
template <typename T>
cudaError_t prime_resident();
// CTAs of the resident kernel for tile shape c that fit on the current device at once.
template <typename T>
cudaError_t resident_capacity(TileCfg c, int* ctas);
template <typename T>
cudaError_t launch_resident(const RoundArgs<T>& a, const ResSync& rs, TileCfg cfg, cudaStream_t s);
// Materialise the halo cells of h (scalar) and/or (u, v) (vector) from their interiors.
template <typename T>
cudaError_t launch_fill_halo(const Geo<T>& g, T* h, T* u, T* v, cudaStream_t s);
template <typename T>
cudaError_t launch_diag(const Geo<T>& g, const T* h, const T* u, const T* v, const DiagOut<T>& d,
                        cudaStream_t s);

}  // namespace bt
