// bt_resident.cuh - the tile-resident round kernel (BT_MODE_RESIDENT).
//
// The reference runs a round as one XLA while loop of nbb substeps
// (src/licom/momentum/barotr.py:41-87, lax.fori_loop at :61).  For grids whose
// tiles all fit on the GPU at once (C48, C96), this kernel runs the whole
// round in one cooperative launch with ONE CTA PER TILE, and each CTA keeps
// everything that does not change during the round on chip:
//
//   * the tile's cell and face constants (depths, spacings) are staged into
//     shared memory once, at launch, and for the 8 x 16 tiles, whose threads
//     have one region point each, the points' metric, halo sources and weights
//     (ResHeld; the larger shapes read those again in each phase's prologue,
//     ahead of its wait);
//   * phase H leaves the momentum terms of the tile's cells in shared memory,
//     so phase UV reads only the new h of its region and the base velocities.
//
// Tiles synchronise with their neighbours only: after each phase a CTA
// publishes the number of phases it has completed (release store of its own
// flag), and before a phase it waits until every tile it depends on has
// completed the previous phase.  The dependency list of a tile (built on the
// host, bt_resident_deps) holds every tile owning a cell the tile reads in
// either phase -- its 3-cell stencil region, halo cells resolved to their
// gather sources, the neighbour face's 6-point lines along the face edges it
// touches -- and is made symmetric, so a tile is never more than one phase
// ahead of a tile it reads from or that reads from it: no buffer is
// overwritten while a neighbour may still read it.  Every wait is bounded by
// the plan's spin limit; a tile that gives up raises kErrNeighbourTimeout and
// an abort word that ends every other tile's wait, and all CTAs return.
//
// The arithmetic is the tile phases' own (bt_stencil.cuh, RES = true), so the
// results are bitwise identical to the stream, graph and persistent modes.

#pragma once

#include "bt_launch.cuh"

namespace bt {

// Resident CTAs per SM the kernel is compiled for (register cap 65536 / (288 *
// blocks)).  The float64 layouts of the larger tiles (16 x 16: 73 KB, 8 x 32: 83 KB)
// fit only two CTAs per SM anyway, so they get the registers of two.
template <typename T, int TI, int TJ>
struct ResBlocks {
  static constexpr int value = (sizeof(T) == 8 && TI * TJ > 128) ? 2 : 3;
};

// Shared-memory layout of a resident CTA (words of T): phase H layout, momentum
// terms, then with one region point per thread what HPre holds of it (ResHeld;
// phase UV's region h takes the place of phase H's, dead by then, so that three
// float64 CTAs fit an SM), else phase UV's layout.
template <typename T, int TI, int TJ>
struct ResLayout {
  using S = TileShape<TI, TJ>;
  static_assert(S::kWordsUV <= S::hUC, "phase UV's region fits phase H's");
  static constexpr int kTermsAt = up4(S::kWordsH), kHeldAt = up4(kTermsAt + kTerms<T> * S::C);
  static constexpr int kHeldPlanes = HPre<T, TI, TJ>::kLineHeld ? 14 : 13, kHeldInts = 3 * S::kT * (int)sizeof(int) / (int)sizeof(T);
  static constexpr int kUV = S::kHeld ? 0 : kHeldAt;
  static constexpr int kWords = up4(kHeldAt + (S::kHeld ? kHeldPlanes * S::kT + kHeldInts : S::kWordsUV));
  static constexpr size_t kBytes = sizeof(T) * kWords;
};

// What HPre holds of a thread's region point and line point, kept in shared memory
// for the whole round where a thread has one of each (TileShape::kHeld): planes
// of one word per thread -- metric (4), sina, l2c (4), halo weights (2), then the
// line point's metric (kLineHeld) or weights -- and ints: the numbers of the first
// halo sources (complemented where the second is the one before) and the line slot.
// With them read from memory in every phase, as the larger shapes do: C48 float64
// 19.4 against 17.0 us per substep, C96 float64 21.3 / 19.0, float32 18.1 / 15.6.
template <typename T, int TI, int TJ>
struct ResHeld {
  using S = TileShape<TI, TJ>;
  using H = HPre<T, TI, TJ>;
  T* p;
  int* b;
  __device__ __forceinline__ explicit ResHeld(T* sm)
      : p(sm + ResLayout<T, TI, TJ>::kHeldAt + threadIdx.x),
        b(reinterpret_cast<int*>(sm + ResLayout<T, TI, TJ>::kHeldAt + ResLayout<T, TI, TJ>::kHeldPlanes * S::kT) +
          threadIdx.x) {}
  __device__ __forceinline__ void put(const HaloRef<T>& r, int w, int z) const {
    p[w * S::kT] = r.w0;
    p[(w + 1) * S::kT] = r.w1;
    b[z * S::kT] = r.d < 0 ? ~r.b0 : r.b0;
  }
  __device__ __forceinline__ void get(HaloRef<T>& r, int w, int z) const {
    const int e = b[z * S::kT];
    r.w0 = p[w * S::kT];
    r.w1 = p[(w + 1) * S::kT];
    r.b0 = e < 0 ? ~e : e;
    r.d = e < 0 ? -1 : 1;
  }
  __device__ __forceinline__ void store(const H& h) const {
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      p[z * S::kT] = h.g[z];
      p[(5 + z) * S::kT] = h.halo.l2[z];
    }
    p[4 * S::kT] = h.sn;
    put(h.halo.ref, 9, 0);
    b[S::kT] = h.slot;
    if (H::kLineHeld) {
      p[11 * S::kT] = h.halo.g0;
      p[12 * S::kT] = h.halo.g1;
      p[13 * S::kT] = h.halo.sn;
    } else {
      put(h.lref, 11, 2);
    }
  }
  __device__ __forceinline__ void load(const Geo<T>& g, const TileBox& box, int stored_halo, H& h) const {
    h.P = edge_count(box, g.m, g.route, h.cnt);
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      h.g[z] = p[z * S::kT];
      h.halo.l2[z] = p[(5 + z) * S::kT];
    }
    h.sn = p[4 * S::kT];
    get(h.halo.ref, 9, 0);
    h.slot = stored_halo ? -1 : b[S::kT];
    if (H::kLineHeld) {
      h.halo.g0 = p[11 * S::kT];
      h.halo.g1 = p[12 * S::kT];
      h.halo.sn = p[13 * S::kT];
    } else {
      get(h.lref, 11, 2);
    }
  }
  // phase UV: the thread's cell and region point (c_block: the tile's cell constants)
  __device__ __forceinline__ void load(const Geo<T>& g, const TileBox& box, const T* c_block,
                                       UvPre<T, TI, TJ>& u) const {
    const int c = threadIdx.x, a = c / TJ, q = c % TJ;
    get(u.ref[0], 9, 0);
    if (a < box.ni && q < box.nj) {
      u.rdx[0] = c_block[S::C + c];
      u.rdy[0] = c_block[2 * S::C + c];
      if (in_bands(box.i0 + a, box.j0 + q, g.n)) {
        ld_quad(g.c2l + 4 * (long)cell32(box.f, box.i0 + a, box.j0 + q, g.m), u.c2);
        const T* const r = p - c + (a + kHalo) * TJ + q;  // the cell's region point
#pragma unroll
        for (int z = 0; z < 4; ++z) u.g[z] = r[z * S::kT];
        u.sn = r[4 * S::kT];
      }
    }
  }
};

// Publish that this CTA has completed ``phases`` phases: every thread's global
// stores are ordered before the flag by the barrier and the (cumulative)
// release store.
__device__ __forceinline__ void res_publish(int* flag, int phases) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(flag), "r"(phases) : "memory");
}

// Wait until every dependency of ``tile`` has completed ``need`` phases.  The
// lanes of warp 0 poll one dependency each (relaxed loads, a fence after the
// last one), at most ``limit`` polls per dependency; the abort word is
// checked every 64 polls.  Returns false when the round must stop.
__device__ __forceinline__ bool res_wait(const ResSync& s, int tile, int need, int* err, long long limit) {
  __shared__ int s_ok;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int b = s.dep_off[tile], e = s.dep_off[tile + 1];
    int ok = 1;
    for (int k = b + lane; k < e && ok; k += 32) {
      const int* fp = s.flags + s.dep_idx[k] * kResFlagStride;
      long long polls = 0;
      while (true) {
        int seen;
        asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(fp) : "memory");
        if (seen >= need) break;
        ++polls;
        if ((polls & 63) == 0) {
          int ab;
          asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(ab) : "l"(s.abort) : "memory");
          if (ab) {
            ok = 0;
            break;
          }
        }
        if (polls > limit) {
          atomicOr(err, kErrNeighbourTimeout);
          atomicExch(s.abort, 1);
          ok = 0;
          break;
        }
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Phase H then phase UV of one stage for a tile of kind FULL.
template <typename T, int TI, int TJ, bool FULL>
__device__ __forceinline__ bool res_stage(const RoundArgs<T>& a, const ResSync& rsy, const StageIO<T>& io,
                                          const TileBox& b, T* sm, const ResSm<T>& rs, int tile, int done) {
  constexpr bool kHeld = TileShape<TI, TJ>::kHeld;
  {
    HPre<T, TI, TJ> pre{};
    if constexpr (kHeld)
      ResHeld<T, TI, TJ>(sm).load(a.g, b, io.stored_halo, pre);
    else
      tile_h_points<T, TI, TJ, FULL>(a.g, io, b, sm, pre);
    if (done > 0 && !res_wait(rsy, tile, done, a.err, a.spin_limit)) return false;
    tile_h_main_t<T, TI, TJ, FULL, true, true>(a.g, io, b, sm, pre, rs);
    res_publish(rsy.flags + tile * kResFlagStride, done + 1);
  }
  {
    UvPre<T, TI, TJ> pre{};
    if constexpr (kHeld)
      ResHeld<T, TI, TJ>(sm).load(a.g, b, sm + LayoutH<T, TI, TJ>::S::hC, pre);
    else
      tile_uv_pro_t<T, TI, TJ, FULL>(a.g, b, pre);
    if (!res_wait(rsy, tile, done + 1, a.err, a.spin_limit)) return false;
    tile_uv_main_t<T, TI, TJ, FULL, true, true>(a.g, io, b, sm + ResLayout<T, TI, TJ>::kUV, pre, rs);
    res_publish(rsy.flags + tile * kResFlagStride, done + 2);
  }
  return true;
}

// One CTA per tile (face-major order); the grid is exactly the tile count.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(kTileThreads, ResBlocks<T, TI, TJ>::value) k_resident(RoundArgs<T> a, ResSync rsy) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ StageIO<T> s_io;
  T* const sm = reinterpret_cast<T*>(smraw);
  ResSm<T> rs;
  rs.terms = sm + ResLayout<T, TI, TJ>::kTermsAt;
  const int tile = blockIdx.x;
  const TileBox b = tile_box_at(a.t, a.g.n, tile);
  const bool full = tile_full(b, a.g.m, TI, TJ);
  // the constants, once per round (awaited by the first phase's barrier)
  tile_consts<T, TI, TJ>(a.g, b, LayoutH<T, TI, TJ>(sm));
  if constexpr (TileShape<TI, TJ>::kHeld) {  // with the lines' depths
    if (threadIdx.x == 0) {
      s_io.stored_halo = 0;
      s_io.last = 1;
    }
    __syncthreads();
    HPre<T, TI, TJ> pre{};
    tile_h_points<T, TI, TJ, false>(a.g, s_io, b, sm, pre);
    ResHeld<T, TI, TJ>(sm).store(pre);
    __syncthreads();
  }
  const int nst = a.rk == 2 ? 2 : 3;
  const int nstage = a.nbb * nst;
  for (int sg = 0; sg < nstage; ++sg) {
    if (threadIdx.x == 0) s_io = round_stage(a, a.step0 + sg / nst, sg % nst);
    __syncthreads();
    const bool ok = full ? res_stage<T, TI, TJ, true>(a, rsy, s_io, b, sm, rs, tile, 2 * sg)
                         : res_stage<T, TI, TJ, false>(a, rsy, s_io, b, sm, rs, tile, 2 * sg);
    if (!ok) {
      cp_async_wait_all();  // no copy may be left in flight when the CTA leaves
      return;
    }
  }
}

}  // namespace bt

namespace bt {
namespace {

template <typename T, int TI, int TJ>
cudaError_t prime_resident_tile() {
  return cudaFuncSetAttribute(k_resident<T, TI, TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)ResLayout<T, TI, TJ>::kBytes);
}

template <typename T, int TI, int TJ>
cudaError_t resident_capacity_tile(int* ctas) {
  int dev, sms, per_sm;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = prime_resident_tile<T, TI, TJ>()) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resident<T, TI, TJ>, kTileThreads,
                                                    ResLayout<T, TI, TJ>::kBytes);
  if (e != cudaSuccess) return e;
  *ctas = per_sm * sms;
  return cudaSuccess;
}

template <typename T, int TI, int TJ>
cudaError_t launch_resident_tile(RoundArgs<T> a, ResSync rs, cudaStream_t s) {
  a.t = make_tiling({TI, TJ}, a.g.n);
  void* args[] = {&a, &rs};
  return cudaLaunchCooperativeKernel((const void*)k_resident<T, TI, TJ>, dim3(6 * a.t.tiles_per_face()),
                                     dim3(kTileThreads), args, ResLayout<T, TI, TJ>::kBytes, s);
}

}  // namespace

#ifdef BT_DEFINE_COMMON
bool resident_tile_supported(TileCfg c) {
  return (c.ti == 8 && c.tj == 16) || (c.ti == 16 && c.tj == 16) || (c.ti == 8 && c.tj == 32);
}
#endif

template <typename T>
cudaError_t prime_resident() {
  cudaError_t e = prime_resident_tile<T, 8, 16>();
  if (e == cudaSuccess) e = prime_resident_tile<T, 16, 16>();
  if (e == cudaSuccess) e = prime_resident_tile<T, 8, 32>();
  return e;
}

template <typename T>
cudaError_t resident_capacity(TileCfg c, int* ctas) {
  if (c.ti == 8 && c.tj == 16) return resident_capacity_tile<T, 8, 16>(ctas);
  if (c.ti == 16 && c.tj == 16) return resident_capacity_tile<T, 16, 16>(ctas);
  if (c.ti == 8 && c.tj == 32) return resident_capacity_tile<T, 8, 32>(ctas);
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_resident(const RoundArgs<T>& a, const ResSync& rs, TileCfg c, cudaStream_t s) {
  if (c.ti == 8 && c.tj == 16) return launch_resident_tile<T, 8, 16>(a, rs, s);
  if (c.ti == 16 && c.tj == 16) return launch_resident_tile<T, 16, 16>(a, rs, s);
  if (c.ti == 8 && c.tj == 32) return launch_resident_tile<T, 8, 32>(a, rs, s);
  return cudaErrorInvalidValue;
}

#define BT_INSTANTIATE_RESIDENT(T)                                                           \
  template cudaError_t prime_resident<T>();                                                  \
  template cudaError_t resident_capacity<T>(TileCfg, int*);                                  \
  template cudaError_t launch_resident<T>(const RoundArgs<T>&, const ResSync&, TileCfg, cudaStream_t);

}  // namespace bt
