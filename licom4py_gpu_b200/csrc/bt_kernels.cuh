// bt_kernels.cuh - sm_100a kernels of the barotropic duogrid solver and their launchers.
//
// Included by bt_kernels_f64.cu (float64 drop-in, compiled with -fmad=false so
// the arithmetic rounds like the reference term by term) and bt_kernels_f32.cu
// (float32 precision form, FMA contraction allowed), each instantiating one type.
//
// Per RK stage two tile kernels run back to back (phase H, phase UV); each CTA
// stages one tile of one face plus its 3-cell stencil halo in shared memory
// (cross-shaped region, corners skipped), computes the C/D-grid face
// quantities once per face and the cell updates from them.  The whole
// member (6 faces) is one launch; halos across face edges are gathered
// inside the tile loader (bt_stencil.cuh), so no separate exchange kernel
// runs between phases.

#pragma once

#include <algorithm>
#include <atomic>

#include "bt_fused.cuh"
#include "bt_launch.cuh"

namespace bt {

constexpr int kThreads = 256;  // of the element-wise kernels
// SMs of a B200, which the tile rules below (fused_tile, spread_smem, late launches) are measured on: they choose
// between forms of equal results, also where a part of the GPU has fewer.
constexpr int kSms = 148;

// FP: the full-interior-tile path compiled in (multi-wave launches), else
// every tile runs the edge path (one-wave launches: half the code to fetch).
template <typename T, int TI, int TJ, bool FP>
__global__ void __launch_bounds__(kTileThreads, PhaseBlocksH<T, FP>::value) k_phase_h(Geo<T> g, StageIO<T> io, Tiling t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  if (!t.late) release_dependents();
  const TileBox b = tile_box(t, g.n, blockIdx.x);
  tile_h<T, TI, TJ, FP>(g, io, b, reinterpret_cast<T*>(smraw), t.late);
}

template <typename T, int TI, int TJ, bool FP>
__global__ void __launch_bounds__(kTileThreads, PhaseBlocksUV<T, TileShape<TI, TJ>::KP, FP>::value) k_phase_uv(Geo<T> g, StageIO<T> io, Tiling t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  if (!t.late) release_dependents();
  const TileBox b = tile_box(t, g.n, blockIdx.x);
  tile_uv<T, TI, TJ, FP>(g, io, b, reinterpret_cast<T*>(smraw), t.late);
}

// One whole round of one member in a single cooperative launch: every CTA
// walks its tiles of a phase, then all CTAs meet at a grid barrier.  Before
// waiting at the barrier a CTA already issues the next phase's prologue for
// its first tile (constants by cp.async, halo descriptors), so those loads
// overlap the barrier.  The loop runs per RK stage (phase H, barrier, phase
// UV, barrier) so the two phases' gather states are never live together.
// float64 runs two CTAs per SM (96 registers: at three the prologue's values, held
// across the barrier, spill 344-1364 bytes; C96 8 x 16 31.8 -> 28.6 us per substep,
// C192 16 x 32 75.5 -> 59.3), float32 three (C192 16 x 32 35.2 against 38.2 with two).
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(kTileThreads, sizeof(T) == 8 ? 2 : 3) k_round(RoundArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ StageIO<T> s_io[2];  // stage pointers, alternating between consecutive stages
  T* sm = reinterpret_cast<T*>(smraw);
  const int ntiles = 6 * a.t.tiles_per_face();
  const int nst = a.rk == 2 ? 2 : 3;
  const int nstage = a.nbb * nst;
  const int t0 = blockIdx.x;
  unsigned gen = 0;
  for (int sg = 0; sg < nstage; ++sg) {
    if (threadIdx.x == 0) s_io[sg & 1] = round_stage(a, a.step0 + sg / nst, sg % nst);
    __syncthreads();
    const StageIO<T>& io = s_io[sg & 1];
    {
      HPre<T, TI, TJ> pre{};
      if (t0 < ntiles) tile_h_pro<T, TI, TJ>(a.g, io, tile_box(a.t, a.g.n, t0), sm, pre);
      if (sg > 0 && !grid_barrier(a.bar, gen, a.err, a.spin_limit)) {
        cp_async_wait_all();  // no copy may be left in flight when the CTA leaves
        return;
      }
      int k = 0;
      for (int tile = t0; tile < ntiles; tile += gridDim.x, ++k) {
        const TileBox b = tile_box(a.t, a.g.n, tile);
        if (k > 0) tile_h_pro<T, TI, TJ>(a.g, io, b, sm, pre);
        tile_h_main<T, TI, TJ, true, true>(a.g, io, b, sm, pre);
        __syncthreads();
      }
    }
    UvPre<T, TI, TJ> pre{};
    if (t0 < ntiles) tile_uv_pro<T, TI, TJ>(a.g, tile_box(a.t, a.g.n, t0), pre);
    if (!grid_barrier(a.bar, gen, a.err, a.spin_limit)) return;
    int k = 0;
    for (int tile = t0; tile < ntiles; tile += gridDim.x, ++k) {
      const TileBox b = tile_box(a.t, a.g.n, tile);
      if (k > 0) tile_uv_pro<T, TI, TJ>(a.g, b, pre);
      tile_uv_main<T, TI, TJ, true, true>(a.g, io, b, sm, pre);
      __syncthreads();
    }
  }
}

// Tile constant blocks (TileShape::cW words per tile): rda, rdx, rdy, a_f of
// the tile's cells, c_dy of its x faces, d_dx of its y faces, dzph_x of its x
// faces and dzph_y of its y faces, the image of phase H's shared-memory
// constant area.  Positions outside a partial tile and the padding are zero.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(kThreads) k_const_blocks(Geo<T> g, Tiling t, T* out) {
  using S = TileShape<TI, TJ>;
  const long total = 6L * t.nti * t.ntj * S::cW;
  const int m = g.m;
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < total; k += (long)gridDim.x * blockDim.x) {
    const int tile = (int)(k / S::cW), w = (int)(k - (long)tile * S::cW);
    const TileBox b = tile_box_at(t, g.n, tile);
    T v = T(0);
    if (w < S::bCDY) {
      const int arr = w / S::C, e = w % S::C, a = e / TJ, q = e % TJ;
      if (a < b.ni && q < b.nj) {
        const long c = cell(b.f, b.i0 + a, b.j0 + q, m);
        v = arr == 0 ? g.rda[c] : arr == 1 ? g.rdx[c] : arr == 2 ? g.rdy[c] : g.a_f[c];
      }
    } else {
      const bool xf = w < S::bDDX || (w >= S::bDZX && w < S::bDZY);
      const T* src = w < S::bDDX ? g.c_dy : w < S::bDZX ? g.d_dx : w < S::bDZY ? g.dzph_x : g.dzph_y;
      const int e = w - (w < S::bDDX ? S::bCDY : w < S::bDZX ? S::bDDX : w < S::bDZY ? S::bDZX : S::bDZY);
      const int W = xf ? TJ : TJ + 1, a = e / W, q = e % W;
      if (xf ? (a <= b.ni && q < b.nj) : (a < b.ni && q <= b.nj)) v = src[cell(b.f, b.i0 + a, b.j0 + q, m)];
    }
    out[k] = v;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_fill_halo(Geo<T> g, T* h, T* u, T* v) {
  wait_prior_grid();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < 6 * g.nh) fill_halo_cell(g, h, u, v, k);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_diag(Geo<T> g, const T* h, const T* u, const T* v,
                                                   DiagOut<T> d) {
  wait_prior_grid();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = g.m;
  if (k >= 6 * m * m) return;
  const int f = k / (m * m);
  const int r = k - f * m * m;
  diag_cell(g, h, u, v, d, f, r / m, r % m);
}

#ifdef BT_DEFINE_COMMON
bool tile_cfg_supported(TileCfg c) {
  return (c.tj == 32 && (c.ti == 7 || c.ti == 8 || c.ti == 15 || c.ti == 16)) ||
         (c.tj == 16 && (c.ti == 8 || c.ti == 16));
}

size_t terms_elems(int n, size_t esize) {
  size_t most = terms_plane_elems(n, esize);
  for (TileCfg c : {TileCfg{7, 32}, TileCfg{8, 32}, TileCfg{15, 32}, TileCfg{16, 32}, TileCfg{16, 16}}) {
    const size_t tiles = (size_t)6 * ((n + c.ti - 1) / c.ti) * ((n + c.tj - 1) / c.tj);
    most = std::max(most, tiles * c.ti * c.tj * (esize == 8 ? 6 : 2));
  }
  return most;
}

namespace {
template <int TI, int TJ>
size_t const_block_elems_tile(int n) {
  const size_t nti = (n + TI - 1) / TI, ntj = (n + TJ - 1) / TJ;
  return 6 * nti * ntj * (size_t)TileShape<TI, TJ>::cW;
}
}  // namespace

size_t const_block_elems(TileCfg c, int n) {
  if (c.ti == 7 && c.tj == 32) return const_block_elems_tile<7, 32>(n);
  if (c.ti == 8 && c.tj == 32) return const_block_elems_tile<8, 32>(n);
  if (c.ti == 15 && c.tj == 32) return const_block_elems_tile<15, 32>(n);
  if (c.ti == 16 && c.tj == 32) return const_block_elems_tile<16, 32>(n);
  if (c.ti == 8 && c.tj == 16) return const_block_elems_tile<8, 16>(n);
  if (c.ti == 12 && c.tj == 16) return const_block_elems_tile<12, 16>(n);
  if (c.ti == 16 && c.tj == 16) return const_block_elems_tile<16, 16>(n);
  return 0;
}

Tiling make_tiling(TileCfg c, int n) {
  Tiling t;
  t.ti = c.ti;
  t.tj = c.tj;
  t.nti = (n + c.ti - 1) / c.ti;
  t.ntj = (n + c.tj - 1) / c.tj;
  t.bi = t.ri = t.bj = t.rj = t.late = 0;
  return t;
}

Tiling make_even_tiling(TileCfg c, int n) {
  Tiling t = make_tiling(c, n);
  t.bi = n / t.nti;
  t.ri = n % t.nti;
  t.bj = n / t.ntj;
  t.rj = n % t.ntj;
  return t;
}

// Tile shape of the fused stage kernel: 8 x 16, and 12 x 16 (416 threads, two CTAs
// per SM) where that makes three tiles per SM two: it evaluates 1.9 velocities per
// cell against 2.1, and two tiles of 13 warps spread evenly.  us per substep, 8 x
// 16 / 12 x 16: float64 C80 13.5 / 12.0, C96 14.25 / 13.2; float32 C80 8.00 / 7.93,
// C96 8.31 / 8.17, C90 RK3 14.6 / 14.3.
TileCfg fused_tile(int n) {
  const auto tiles = [n](TileCfg c) { return 6 * make_even_tiling(c, n).tiles_per_face(); };
  const TileCfg wide{12, 16};
  return tiles(kFusedTile) > 2 * kSms && tiles(wide) <= 2 * kSms ? wide : kFusedTile;
}

size_t stage_table_bytes(int n, size_t esize) {
  const TileCfg c = fused_tile(n);
  return (size_t)6 * make_even_tiling(c, n).tiles_per_face() * tile_threads(c.ti) * (3 * sizeof(int4) + 2 * esize);
}
#endif

namespace {

template <typename T, int TI, int TJ, bool UV>
size_t tile_smem() {
  using S = TileShape<TI, TJ>;
  return sizeof(T) * (UV ? S::kWordsUV : S::kWordsH);
}

// Shared memory a one-wave float64 launch of up to two tiles per SM asks for at
// least, so that no SM takes more than two of its tiles -- or one, if there is one
// per SM at most and nothing else to run beside it (``alone``): the CTAs start as
// those of the kernel before leave, and without the limit the SMs that are done
// first take three while others get one.  us per substep without / with it: fused
// kernel C24 8.5 / 7.7, C48 9.1 / 8.4, C64 12.2 / 9.8, C72 14.4 / 10.2; phase
// kernels C64 14.2 / 13.6, C72 14.5 / 13.1.  The request stays just above the
// limit, which leaves the rest to L1 (C72 11.7 with all of it).  With three tiles
// per SM the registers set the limit already and the larger request only costs
// (C96 14.2 / 14.6, C128 16 x 16 20.9 / 21.8); phase launches of up to one tile per
// SM are late (launch_tile) and lose with it (C48 12.1 / 12.9); float32 tiles are
// short enough for the start of the next kernel's tiles beside them to be worth
// more (C64 6.99 / 7.11).
// One tile per SM leaves the rounds of other plans on other streams no room beside
// the CTAs that wait for the kernel ahead.  Graph rounds, which several streams can
// run at once from one thread, allow two: four C48 plans 15.6 us per substep against
// 23.6, four C36 plans 12.3 / 19.0 (phase kernels 16.3 and 16.0), one C48 plan 8.9 /
// 8.4.  Stream rounds of one thread are launched too slowly to fill the GPU (four
// C48 plans 26.2 with one, 24.3 with two; phase kernels 45.7) and keep one: a C48
// plan 8.3 against 9.6.
template <typename T>
size_t spread_smem(int tiles, bool alone) {
  constexpr size_t per_sm = 228 * 1024, per_cta = 1024;  // sm_100: shared memory of an SM, reserved by each CTA
  if (sizeof(T) == 4 || tiles > 2 * kSms) return 0;
  return per_sm / (tiles <= kSms && alone ? 2 : 3) - per_cta + 256;
}

// The persistent kernel runs both phases in one allocation: the larger of the two.
template <typename T, int TI, int TJ>
size_t round_smem() {
  return std::max(tile_smem<T, TI, TJ, false>(), tile_smem<T, TI, TJ, true>());
}

// CTAs of one phase kernel (edge-only build) that fit on each device at once,
// recorded by prime_tile at plan creation (0 = not recorded yet).
constexpr int kMaxDevices = 64;
template <typename T, int TI, int TJ, bool UV>
std::atomic<int>* wave_slots() {  // relaxed: plans on several host threads may record them at once
  static std::atomic<int> slots[kMaxDevices];
  return slots;
}

template <typename T, int TI, int TJ, bool UV>
cudaError_t record_wave_slots() {
  int dev, sms, per_sm;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaSuccess;  // the launch then keeps the full-tile path
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  auto kern = UV ? k_phase_uv<T, TI, TJ, false> : k_phase_h<T, TI, TJ, false>;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kTileThreads, tile_smem<T, TI, TJ, UV>())) !=
      cudaSuccess)
    return e;
  wave_slots<T, TI, TJ, UV>()[dev].store(sms * per_sm, std::memory_order_relaxed);
  return cudaSuccess;
}

// Opt in to more than 48 KB of dynamic shared memory and record the wave slots
// (done at plan creation, never during stream capture).
template <typename T, int TI, int TJ>
cudaError_t prime_tile() {
  cudaError_t e;
  const size_t spread = spread_smem<T>(1, true);  // the most it asks for
  for (auto k : {k_phase_h<T, TI, TJ, true>, k_phase_h<T, TI, TJ, false>})
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::max(tile_smem<T, TI, TJ, false>(), spread))) != cudaSuccess)
      return e;
  for (auto k : {k_phase_uv<T, TI, TJ, true>, k_phase_uv<T, TI, TJ, false>})
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::max(tile_smem<T, TI, TJ, true>(), spread))) != cudaSuccess)
      return e;
  e = cudaFuncSetAttribute(k_round<T, TI, TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)round_smem<T, TI, TJ>());
  if (e != cudaSuccess) return e;
  if constexpr (TI == 8 && TJ == 16) {
    e = cudaFuncSetAttribute(k_stage<T, TI, TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)std::max(sizeof(T) * FusedShape<TI, TJ>::kWords, spread));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_stage<T, 12, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)std::max(sizeof(T) * FusedShape<12, 16>::kWords, spread));
    if (e != cudaSuccess) return e;
  }
  if ((e = record_wave_slots<T, TI, TJ, false>()) != cudaSuccess) return e;
  return record_wave_slots<T, TI, TJ, true>();
}

// Co-resident grid for the persistent kernel (at most one CTA per tile).
template <typename T, int TI, int TJ>
cudaError_t launch_round_tile(RoundArgs<T> a, int max_ctas, cudaStream_t s, int* grid_out) {
  const size_t smem = round_smem<T, TI, TJ>();
  int dev, sms, per_sm;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_round<T, TI, TJ>, kTileThreads, smem)) !=
      cudaSuccess)
    return e;
  a.t = make_tiling({TI, TJ}, a.g.n);
  int grid = std::min(per_sm * sms, 6 * a.t.tiles_per_face());
  if (max_ctas > 0) grid = std::min(grid, max_ctas);
  if (grid < 1) return cudaErrorInvalidConfiguration;
  if (grid_out) *grid_out = grid;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel((const void*)k_round<T, TI, TJ>, dim3(grid), dim3(kTileThreads), args, smem, s);
}

// Whether a phase launch at n cells per face edge runs the full-tile kernel:
// forced by full_tiles >= 0, else by size (the edge-only kernel when the
// launch's CTAs all fit on the current device at once).
template <typename T, int TI, int TJ, bool UV>
bool full_path(int n, int full_tiles) {
  if (full_tiles >= 0) return full_tiles != 0;
  int dev = -1;
  int slots = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices)
    slots = wave_slots<T, TI, TJ, UV>()[dev].load(std::memory_order_relaxed);
  return !(slots > 0 && 6 * make_tiling({TI, TJ}, n).tiles_per_face() <= slots);
}

template <typename T, int TI, int TJ, bool UV>
cudaError_t launch_tile(const Geo<T>& g, const StageIO<T>& io, cudaStream_t s, int full_tiles, bool overlap) {
  const size_t smem = tile_smem<T, TI, TJ, UV>();
  Tiling t = make_tiling({TI, TJ}, g.n);
  // up to one tile per SM the next kernel starts only when this one runs: its CTAs, and those of the kernels
  // after it, would otherwise share SMs with this kernel's while other SMs idle (C48 8 x 16 float64 12.9 -> 12.0
  // us per substep); with more, the early start is the faster (C384 16 x 16 float64 137 against 165)
  t.late = 6 * t.tiles_per_face() <= kSms ? 1 : 0;
  const bool fp = full_path<T, TI, TJ, UV>(g.n, full_tiles);
  auto kern = UV ? (fp ? k_phase_uv<T, TI, TJ, true> : k_phase_uv<T, TI, TJ, false>)
                 : (fp ? k_phase_h<T, TI, TJ, true> : k_phase_h<T, TI, TJ, false>);
  // programmatic dependent launch (overlap): the kernel's constant prologue overlaps the
  // previous kernel's tail; it waits (griddepcontrol.wait) before reading state
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(6 * t.tiles_per_face());
  cfg.blockDim = dim3(kTileThreads);
  cfg.dynamicSmemBytes = fp || t.late ? smem : std::max(smem, spread_smem<T>(6 * t.tiles_per_face(), false));
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, g, io, t);
}

template <typename T, bool UV>
cudaError_t dispatch(const Geo<T>& g, const StageIO<T>& io, TileCfg c, cudaStream_t s, int full_tiles, bool overlap) {
  if (c.ti == 7 && c.tj == 32) return launch_tile<T, 7, 32, UV>(g, io, s, full_tiles, overlap);
  if (c.ti == 8 && c.tj == 32) return launch_tile<T, 8, 32, UV>(g, io, s, full_tiles, overlap);
  if (c.ti == 15 && c.tj == 32) return launch_tile<T, 15, 32, UV>(g, io, s, full_tiles, overlap);
  if (c.ti == 16 && c.tj == 32) return launch_tile<T, 16, 32, UV>(g, io, s, full_tiles, overlap);
  if (c.ti == 8 && c.tj == 16) return launch_tile<T, 8, 16, UV>(g, io, s, full_tiles, overlap);
  if (c.ti == 16 && c.tj == 16) return launch_tile<T, 16, 16, UV>(g, io, s, full_tiles, overlap);
  return cudaErrorInvalidValue;
}

}  // namespace

template <typename T>
cudaError_t launch_round(const RoundArgs<T>& a, TileCfg c, int max_ctas, cudaStream_t s, int* grid_out) {
  if (c.ti == 7 && c.tj == 32) return launch_round_tile<T, 7, 32>(a, max_ctas, s, grid_out);
  if (c.ti == 8 && c.tj == 32) return launch_round_tile<T, 8, 32>(a, max_ctas, s, grid_out);
  if (c.ti == 15 && c.tj == 32) return launch_round_tile<T, 15, 32>(a, max_ctas, s, grid_out);
  if (c.ti == 16 && c.tj == 32) return launch_round_tile<T, 16, 32>(a, max_ctas, s, grid_out);
  if (c.ti == 8 && c.tj == 16) return launch_round_tile<T, 8, 16>(a, max_ctas, s, grid_out);
  if (c.ti == 16 && c.tj == 16) return launch_round_tile<T, 16, 16>(a, max_ctas, s, grid_out);
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t prime_kernels() {
  cudaError_t e;
  if ((e = prime_tile<T, 7, 32>()) != cudaSuccess) return e;
  if ((e = prime_tile<T, 8, 32>()) != cudaSuccess) return e;
  if ((e = prime_tile<T, 15, 32>()) != cudaSuccess) return e;
  if ((e = prime_tile<T, 16, 32>()) != cudaSuccess) return e;
  if ((e = prime_tile<T, 8, 16>()) != cudaSuccess) return e;
  return prime_tile<T, 16, 16>();
}

template <typename T>
int phase_full_paths(TileCfg c, int n, int full_tiles) {
#define BT_FP_BITS(TI, TJ) \
  if (c.ti == TI && c.tj == TJ) \
    return (full_path<T, TI, TJ, false>(n, full_tiles) ? 1 : 0) | (full_path<T, TI, TJ, true>(n, full_tiles) ? 2 : 0);
  BT_FP_BITS(7, 32)
  BT_FP_BITS(8, 32)
  BT_FP_BITS(15, 32)
  BT_FP_BITS(16, 32)
  BT_FP_BITS(8, 16)
  BT_FP_BITS(16, 16)
#undef BT_FP_BITS
  return -1;
}

template <typename T>
cudaError_t launch_phase_h(const Geo<T>& g, const StageIO<T>& io, TileCfg cfg, cudaStream_t s, int full_tiles,
                           bool overlap) {
  return dispatch<T, false>(g, io, cfg, s, full_tiles, overlap);
}

template <typename T>
cudaError_t launch_phase_uv(const Geo<T>& g, const StageIO<T>& io, TileCfg cfg, cudaStream_t s, int full_tiles) {
  return dispatch<T, true>(g, io, cfg, s, full_tiles, true);
}

template <typename T, int TI, int TJ>
static cudaError_t launch_stage_tables_tile(const Geo<T>& g, void* out, cudaStream_t s) {
  constexpr int kT = TileShape<TI, TJ>::kT;
  const Tiling t = make_even_tiling({TI, TJ}, g.n);
  const int tiles = 6 * t.tiles_per_face();
  int4* const rec = (int4*)out;
  k_stage_tables<T, TI, TJ><<<tiles, kT, 0, s>>>(g, t, rec, (T*)(rec + (size_t)tiles * 3 * kT));
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_stage_tables(const Geo<T>& g, void* out, cudaStream_t s) {
  return fused_tile(g.n).ti == 8 ? launch_stage_tables_tile<T, 8, 16>(g, out, s)
                                            : launch_stage_tables_tile<T, 12, 16>(g, out, s);
}

template <typename T, int TI, int TJ>
static cudaError_t launch_stage_tile(const Geo<T>& g, const FusedIO<T>& p, const void* tables, bool alone,
                                     cudaStream_t s) {
  using F = FusedShape<TI, TJ>;
  const Tiling t = make_even_tiling({TI, TJ}, g.n);
  const int4* const rec = (const int4*)tables;
  const T* const weights = (const T*)(rec + (size_t)6 * t.tiles_per_face() * 3 * F::kT);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(6 * t.tiles_per_face());
  cfg.blockDim = dim3(F::kT);
  cfg.dynamicSmemBytes = std::max(sizeof(T) * (p.beta_prev != T(0) ? F::kWords : F::kHP),
                                  spread_smem<T>(6 * t.tiles_per_face(), alone));
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_stage<T, TI, TJ>, g, p, t, rec, weights);
}

template <typename T>
cudaError_t launch_stage(const Geo<T>& g, const FusedIO<T>& p, const void* tables, bool alone, cudaStream_t s) {
  return fused_tile(g.n).ti == 8 ? launch_stage_tile<T, 8, 16>(g, p, tables, alone, s)
                                 : launch_stage_tile<T, 12, 16>(g, p, tables, alone, s);
}

template <typename T, int TI, int TJ>
cudaError_t launch_const_blocks_tile(const Geo<T>& g, bool even, T* out, cudaStream_t s) {
  const Tiling t = even ? make_even_tiling({TI, TJ}, g.n) : make_tiling({TI, TJ}, g.n);
  const long total = 6L * t.nti * t.ntj * TileShape<TI, TJ>::cW;
  const int grid = (int)std::min<long>((total + kThreads - 1) / kThreads, 148L * 16);
  k_const_blocks<T, TI, TJ><<<grid, kThreads, 0, s>>>(g, t, out);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_const_blocks(const Geo<T>& g, TileCfg c, bool even, T* out, cudaStream_t s) {
  if (c.ti == 7 && c.tj == 32) return launch_const_blocks_tile<T, 7, 32>(g, even, out, s);
  if (c.ti == 8 && c.tj == 32) return launch_const_blocks_tile<T, 8, 32>(g, even, out, s);
  if (c.ti == 15 && c.tj == 32) return launch_const_blocks_tile<T, 15, 32>(g, even, out, s);
  if (c.ti == 16 && c.tj == 32) return launch_const_blocks_tile<T, 16, 32>(g, even, out, s);
  if (c.ti == 8 && c.tj == 16) return launch_const_blocks_tile<T, 8, 16>(g, even, out, s);
  if (c.ti == 12 && c.tj == 16) return launch_const_blocks_tile<T, 12, 16>(g, even, out, s);
  if (c.ti == 16 && c.tj == 16) return launch_const_blocks_tile<T, 16, 16>(g, even, out, s);
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_fill_halo(const Geo<T>& g, T* h, T* u, T* v, cudaStream_t s) {
  const int total = 6 * g.nh;
  k_fill_halo<T><<<(total + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, h, u, v);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_diag(const Geo<T>& g, const T* h, const T* u, const T* v, const DiagOut<T>& d,
                        cudaStream_t s) {
  const int total = 6 * g.m * g.m;
  k_diag<T><<<(total + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, h, u, v, d);
  return cudaGetLastError();
}

#define BT_INSTANTIATE(T)                                                                           \
  template cudaError_t prime_kernels<T>();                                                          \
  template int phase_full_paths<T>(TileCfg, int, int);                                              \
  template cudaError_t launch_phase_h<T>(const Geo<T>&, const StageIO<T>&, TileCfg, cudaStream_t, int, bool); \
  template cudaError_t launch_phase_uv<T>(const Geo<T>&, const StageIO<T>&, TileCfg, cudaStream_t, int); \
  template cudaError_t launch_fill_halo<T>(const Geo<T>&, T*, T*, T*, cudaStream_t);                \
  template cudaError_t launch_const_blocks<T>(const Geo<T>&, TileCfg, bool, T*, cudaStream_t);         \
  template cudaError_t launch_stage_tables<T>(const Geo<T>&, void*, cudaStream_t);                     \
  template cudaError_t launch_stage<T>(const Geo<T>&, const FusedIO<T>&, const void*, bool, cudaStream_t); \
  template cudaError_t launch_round<T>(const RoundArgs<T>&, TileCfg, int, cudaStream_t, int*);      \
  template cudaError_t launch_diag<T>(const Geo<T>&, const T*, const T*, const T*, const DiagOut<T>&, \
                                      cudaStream_t);

}  // namespace bt
