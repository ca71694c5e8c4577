// bt_plan.cuh - the plan object behind bt_plan_t (host side, internal to libbt.so).
//
// A plan holds one resolution's geometry (the caller's constant arrays and
// the halo gather tables built from them), the member scratch of the
// single-integration entry points, launch options and the graph cache.

#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "bt_fused.cuh"
#include "bt_launch.cuh"
#include "licom_bt.h"

using namespace bt;

// The kernels read the 2x2 matrix arrays (a_c2l, a_l2c, a_gct: four values
// per cell) with 16-byte copies and vector loads, so each must start on a
// 16-byte boundary.
inline bool matrices_aligned(const bt_grid_desc* d) {
  return (((uintptr_t)d->a_c2l | (uintptr_t)d->a_l2c | (uintptr_t)d->a_gct) & 15) == 0;
}

struct bt_plan;
namespace bt {
// Build what rounds and stages of plan p with tiles of shape t read, if it is not there yet (bt_capi.cu).
int prepare_tile(bt_plan* p, TileCfg t, cudaStream_t s);
}  // namespace bt

struct bt_plan {
  int n = 0, m = 0, nh = 0, dtype = BT_F64, device = 0;
  TileCfg tile{8, 32};
  int mode = BT_MODE_STREAM;
  const void* c[17] = {};
  int route[24] = {};
  void* d_hw = nullptr;    // T[6*nh*2]; the halo tables are one allocation, d_hsrc and d_bsrc point into it
  void* d_hsrc = nullptr;  // int2[6*nh]
  int* d_bsrc = nullptr;   // int[72*n]
  void* scratch = nullptr; // Y (3 fields) + Z (3 fields) + edge lines + bands + momentum terms
  size_t field_elems = 0;
  cudaStream_t cap_stream = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  // graph cache
  cudaGraphExec_t gexec = nullptr;
  std::vector<uintptr_t> gkey;
  // tile constant blocks, one buffer per tile shape used (built on first use, see ensure_const_blocks):
  // the plan's own rounds use the plan's tile, batched rounds the batch's
  struct ConstBlocks {
    TileCfg tile{0, 0};
    void* ptr = nullptr;
  };
  ConstBlocks cblks[6];
  const ConstBlocks* cblk_for(TileCfg t) const {
    for (const ConstBlocks& c : cblks)
      if (c.ptr && c.tile.ti == t.ti && c.tile.tj == t.tj) return &c;
    return nullptr;
  }
  // host copy of the halo gather sources (the resident mode's dependency lists are built from it)
  std::vector<int2> h_src;
  // resident mode: dependency lists and progress flags of the tile shape res_tile, one device block:
  // dep_off [tiles + 1], dep_idx [ndep], flags [tiles], abort word
  TileCfg res_tile{0, 0};
  int* d_res = nullptr;
  int res_tiles = 0, res_ndep = 0;
  // persistent mode: barrier counter + device error flag, options
  unsigned* d_flags = nullptr;  // [0] barrier counter, [1] error bits
  int max_ctas = 0;
  long long spin_limit = 1ll << 24;
  int full_tiles = -1;  // BT_OPT_FULL_TILES
  bool fused = false;   // the scratch and the halo tables allow the fused stage kernel
  bool stage_ready = false;  // its tables and constant blocks are built (prepare_tile)
  bool fused_rk3 = false;  // whether RK3 rounds use it too
  int last_grid = 0;
  // optional kernel timing: event pairs on the launch stream around the round
  // kernel (persistent mode) or each phase kernel (stream mode), with their kind
  int timing = 0;
  mutable std::vector<cudaEvent_t> tev;
  mutable std::vector<int> tkind;
  mutable size_t tev_used = 0;

  // Record the start event of a timed kernel of the given kind (nullptr if timing is off).
  cudaError_t time_begin(int kind, cudaStream_t s, cudaEvent_t* stop) const {
    *stop = nullptr;
    if (!timing || mode == BT_MODE_GRAPH) return cudaSuccess;  // an event in a captured round times nothing
    if (tev_used + 2 > tev.size()) {
      for (int k = 0; k < 2; ++k) {
        cudaEvent_t ev;
        cudaError_t e = cudaEventCreate(&ev);
        if (e != cudaSuccess) return e;
        tev.push_back(ev);
      }
    }
    tkind.resize(tev.size() / 2);
    tkind[tev_used / 2] = kind;
    cudaEvent_t start = tev[tev_used];
    *stop = tev[tev_used + 1];
    tev_used += 2;
    return cudaEventRecord(start, s);
  }

  size_t esize() const { return dtype == BT_F64 ? 8 : 4; }
  // scratch layout: 6 stage fields, edge lines (24 n), bands, then on a 256-byte boundary the
  // momentum terms
  size_t terms_offset() const {
    return ((6 * field_elems + 24 * (size_t)n + band_elems(n, fused)) * esize() + 255) & ~(size_t)255;
  }
  // with the fused stage kernel: a second set of terms, its tables, the constant blocks of its even split
  size_t stage_offset() const {
    return (terms_offset() + (fused ? 2 : 1) * terms_elems(n, esize()) * esize() + 255) & ~(size_t)255;
  }
  size_t even_offset() const { return (stage_offset() + stage_table_bytes(n, esize()) + 255) & ~(size_t)255; }
  size_t scratch_bytes() const {
    return fused ? even_offset() + const_block_elems(fused_tile(n), n) * esize() : stage_offset();
  }
  void* stage_tables() const { return (char*)scratch + stage_offset(); }
  void* even_blocks() const { return (char*)scratch + even_offset(); }
  void* scratch_field(int k) const { return (char*)scratch + (size_t)k * field_elems * esize(); }
  void* edge_lines() const { return scratch_field(6); }
  void* bands() const { return (char*)edge_lines() + 24 * (size_t)n * esize(); }
  void* terms(int k = 0) const { return (char*)scratch + terms_offset() + (size_t)k * terms_elems(n, esize()) * esize(); }

  // geometry for kernels of tile shape t (its constant blocks if built)
  template <typename T>
  Geo<T> geo_tile(TileCfg t) const {
    Geo<T> g = geo_arrays<T>();
    const ConstBlocks* c = cblk_for(t);
    g.cblk = c ? (const T*)c->ptr : nullptr;
    g.cblk_ti = c ? t.ti : 0;
    g.cblk_tj = c ? t.tj : 0;
    return g;
  }
  template <typename T>
  Geo<T> geo() const {
    return geo_tile<T>(tile);
  }
  // geometry for the fused stage kernel
  template <typename T>
  Geo<T> geo_fused() const {
    Geo<T> g = geo_arrays<T>();
    g.cblk = (const T*)even_blocks();
    const TileCfg c = fused_tile(n);
    g.cblk_ti = c.ti;
    g.cblk_tj = c.tj;
    return g;
  }
  // geometry without constant blocks (the arrays only)
  template <typename T>
  Geo<T> geo_arrays() const {
    Geo<T> g;
    g.n = n;
    g.m = m;
    g.nh = nh;
    g.dzph_x = (const T*)c[0];
    g.dzph_y = (const T*)c[1];
    g.rdx = (const T*)c[2];
    g.rdy = (const T*)c[3];
    g.a_f = (const T*)c[4];
    g.c2l = (const T*)c[8];
    g.l2c = (const T*)c[9];
    g.gct = (const T*)c[12];
    g.sina = (const T*)c[13];
    g.rda = (const T*)c[14];
    g.c_dy = (const T*)c[15];
    g.d_dx = (const T*)c[16];
    g.hsrc = (const int2*)d_hsrc;
    g.hw = (const T*)d_hw;
    g.bsrc = d_bsrc;
    g.cblk = nullptr;
    g.cblk_ti = g.cblk_tj = 0;
    std::memcpy(g.route, route, sizeof(route));
    return g;
  }
};
