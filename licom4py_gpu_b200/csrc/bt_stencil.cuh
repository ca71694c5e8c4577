// bt_stencil.cuh - device functions of the barotropic RK stage on the duogrid.
//
// One RK stage (src/licom/momentum/barotr_pure.py:100-168) is split at its two
// global dependencies into two tile phases:
//
//   phase H  (tile_h):  everything that depends on the stage input alone:
//            celerity, A->C remap, C-grid edge average, D-grid upwind,
//            velocity viscosity, mass flux (+ flux edge average on the last
//            stage), divergence, new h = h_base - div*dt, and the momentum
//            terms other than the pressure gradient (vorticity / kinetic
//            energy advection, Coriolis, celerity viscosity) of each cell.
//   phase UV (tile_uv): what needs the new h: its pressure gradient, and the
//            momentum update from that and phase H's terms.
//
// Everything local to the stage input runs in phase H, so that phase UV reads 11
// words per cell in float64 (7 in float32) instead of the 26 it took when it
// recomputed the advection from the faces' cache, and gathers only h at the
// face edges.  Both are bound by latency at one-wave sizes (loads, two to four
// barriers, one float64 face chain) and by issue and memory latency at
// C384.  Measured before and after this split with the band gathers, 16-byte
// constant copies and 288 threads (us per substep): float64 C96 8 x 16 15.2 /
// 14.0, C192 8 x 32 39.5 / 36.1, C384 16 x 16 149 / 137, 16 x 32 184 / 155;
// float32 C96 8 x 16 11.9 / 10.8, C192 16 x 32 24.3 / 22.1, C384 16 x 32 70.0 / 65.9.
//
// The ext_scalar / ext_vector halo fills of the reference (cube.py:130-153)
// are computed by whoever reads a halo cell.  Both of a halo cell's sources
// lie on one of the three interior lines next to the shared edge, side by
// side; each phase therefore also writes what the halo remap reads -- the new
// h, or the lon/lat velocity -- of those lines into band buffers ordered along
// the edge, so that the reads of neighbouring halo cells are runs of
// consecutive words whatever the two faces' orientation.  The
// boundary_communication edge averages (communication.py:504-570) are computed
// in place by recomputing the neighbouring face's edge value from that face's
// data.
//
// Every arithmetic expression keeps the reference's operand order; with
// -fmad=false the float64 instantiation rounds exactly like the NumPy run of
// the reference.

#pragma once

#include "bt_common.cuh"

namespace bt {

// 3rd-order reconstruction coefficients, src/licom/operators/poly.py:29-37
#define BT_EP23 (-1.0 / 20.0)
#define BT_EP13 (9.0 / 20.0)
#define BT_EP03 (47.0 / 60.0)
#define BT_EM13 (-13.0 / 60.0)
#define BT_EM23 (1.0 / 30.0)
#define BT_M13 (37.0 / 60.0)
#define BT_M23 (-2.0 / 15.0)
#define BT_M33 (1.0 / 60.0)

// a x + b y.  float32 names the product that is fused into the sum: left to the
// compiler the choice differs from kernel to kernel, and with it the last bits of
// a stage that one kernel or two compute.
template <typename T>
__device__ __forceinline__ T lin2(T a, T x, T b, T y) {
  if constexpr (sizeof(T) == 4)
    return __fmaf_rn(a, x, __fmul_rn(b, y));
  else
    return a * x + b * y;
}
// a x + c, one rounding in float32: named for the same reason.  (The reconstructions
// below are written out for each type: nested calls load and form float64 values in
// another order, batches in one launch per phase 3 % slower; statements do that to
// float32, C384 62.1 -> 63.5 us per substep.)
template <typename T>
__device__ __forceinline__ T mad(T a, T x, T c) {
  if constexpr (sizeof(T) == 4)
    return __fmaf_rn(a, x, c);
  else
    return a * x + c;
}
// Value at the + face of the centre point of p[0], p[s], .., p[4s] (poly.py:50-56)
template <typename T>
__device__ __forceinline__ T rplus(const T* p, int s) {
  if constexpr (sizeof(T) == 4)
    return mad(T(BT_EP23), p[4 * s],
               mad(T(BT_EP13), p[3 * s], mad(T(BT_EP03), p[2 * s], lin2(T(BT_EM23), p[0], T(BT_EM13), p[s]))));
  else
    return lin2(T(BT_EM23), p[0], T(BT_EM13), p[s]) + T(BT_EP03) * p[2 * s] + T(BT_EP13) * p[3 * s] +
           T(BT_EP23) * p[4 * s];
}
// Value at the - face of the centre point (poly.py:57-63)
template <typename T>
__device__ __forceinline__ T rminus(const T* p, int s) {
  if constexpr (sizeof(T) == 4)
    return mad(T(BT_EM23), p[4 * s],
               mad(T(BT_EM13), p[3 * s], mad(T(BT_EP03), p[2 * s], lin2(T(BT_EP23), p[0], T(BT_EP13), p[s]))));
  else
    return lin2(T(BT_EP23), p[0], T(BT_EP13), p[s]) + T(BT_EP03) * p[2 * s] + T(BT_EM13) * p[3 * s] +
           T(BT_EM23) * p[4 * s];
}
// 6-point centred face value between p[2s] and p[3s] (poly.py:120-124)
template <typename T>
__device__ __forceinline__ T mid6(const T* p, int s) {
  if constexpr (sizeof(T) == 4)
    return mad(T(BT_M33), p[0] + p[5 * s], lin2(T(BT_M13), p[2 * s] + p[3 * s], T(BT_M23), p[s] + p[4 * s]));
  else
    return lin2(T(BT_M13), p[2 * s] + p[3 * s], T(BT_M23), p[s] + p[4 * s]) + T(BT_M33) * (p[0] + p[5 * s]);
}
// Gravity-wave speed with the 10 m/s floor (barotr_pure.py:21-26); NaN propagates like jnp.maximum.
template <typename T>
__device__ __forceinline__ T celerity(T hface, T dz) {
  T c = sqrt(T(9.8) * (hface + dz));
  return (c < T(10.0)) ? T(10.0) : c;
}

// ---------------------------------------------------------------------------
// Halo values on the fly
// ---------------------------------------------------------------------------
// Scalar value at (f, i, j).  Interior cells (and every cell when the stored
// halo is valid) are read directly; a halo cell is the kinked->extended linear
// interpolation of two interior cells of a neighbouring face (cube.py:40-134).
template <typename T>
__device__ __forceinline__ T fetch_s(const T* F, const Geo<T>& g, int f, int i, int j, int stored) {
  const int m = g.m;
  if (stored || is_interior(i, j, m)) return F[cell(f, i, j, m)];
  const int k = f * g.nh + halo_id(i, j, m);
  const int2 s = g.hsrc[k];
  const T w0 = g.hw[2 * k], w1 = g.hw[2 * k + 1];
  return lin2(w0, F[s.x], w1, F[s.y]);
}

// Vector (covariant u, v) at (f, i, j): the halo value is rotated to lon/lat at
// the two source cells with c2l, interpolated, and rotated back with the
// target's l2c (ext_vector, cube.py:137-153; the inner/outer masks are 1/0 there).
template <typename T>
__device__ __forceinline__ void fetch_v(const T* U, const T* V, const Geo<T>& g, int f, int i, int j,
                                        int stored, T& u, T& v) {
  const int m = g.m;
  const long o = cell(f, i, j, m);
  if (stored || is_interior(i, j, m)) {
    u = U[o];
    v = V[o];
    return;
  }
  const int k = f * g.nh + halo_id(i, j, m);
  const int2 s = g.hsrc[k];
  const T w0 = g.hw[2 * k], w1 = g.hw[2 * k + 1];
  const T* C0 = g.c2l + 4 * (long)s.x;
  const T* C1 = g.c2l + 4 * (long)s.y;
  const T u0 = U[s.x], v0 = V[s.x], u1 = U[s.y], v1 = V[s.y];
  const T ull0 = lin2(C0[0], u0, C0[1], v0), vll0 = lin2(C0[2], u0, C0[3], v0);
  const T ull1 = lin2(C1[0], u1, C1[1], v1), vll1 = lin2(C1[2], u1, C1[3], v1);
  const T ull = lin2(w0, ull0, w1, ull1);
  const T vll = lin2(w0, vll0, w1, vll1);
  const T* L = g.l2c + 4 * o;
  u = lin2(L[0], ull, L[1], vll);
  v = lin2(L[2], ull, L[3], vll);
}

// Contravariant component along axis -2 (x) or axis -1 (y) (remap.py:34-39)
template <typename T>
__device__ __forceinline__ T contra(const Geo<T>& g, long o, T u, T v, int y) {
  const T* G = g.gct + 4 * o;
  return y ? lin2(G[2], u, G[3], v) * g.sina[o] : lin2(G[0], u, G[1], v) * g.sina[o];
}

// ---------------------------------------------------------------------------
// The neighbouring face's side of a C-grid edge
// ---------------------------------------------------------------------------
// k-th of the 6 points (k = 0..5) on the line normal to ``side`` of a face that
// straddles that side's C-grid edge face, at along-edge position kk.  The
// edge face itself sits between points 2 and 3.
__host__ __device__ __forceinline__ void edge_point(int side, int kk, int k, int m, int& i, int& j) {
  switch (side) {
    case kS: i = k; j = kHalo + kk; break;
    case kN: i = m - 6 + k; j = kHalo + kk; break;
    case kW: i = kHalo + kk; j = k; break;
    default: i = kHalo + kk; j = m - 6 + k; break;
  }
}

// The neighbour's C-grid normal velocity before averaging, at the edge shared
// with side ``side`` of face f, position k along our edge
// (communication.py:226-235 pack + remap.py:41-55 on the neighbour).
template <typename T>
__device__ T nb_normal_raw(const Geo<T>& g, const T* U, const T* V, int stored, int f, int side,
                           int k) {
  const int r = g.route[f * 4 + side];
  const int nb = route_nb(r), ns = route_side(r);
  const int kk = route_rev(r) ? g.n - 1 - k : k;
  const int y = (ns == kE || ns == kW);
  T p[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    int i, j;
    edge_point(ns, kk, q, g.m, i, j);
    T u, v;
    fetch_v(U, V, g, nb, i, j, stored, u, v);
    p[q] = contra(g, cell(nb, i, j, g.m), u, v, y);
  }
  return T(0.5) * (rplus(p, 1) + rminus(p + 1, 1));
}

// Side of a face whose C-grid edge lies at x-face index i (or y-face index j).
__device__ __forceinline__ int xface_side(int i, int m) {
  return i == kHalo ? kS : (i == m - kHalo ? kN : -1);
}
__device__ __forceinline__ int yface_side(int j, int m) {
  return j == kHalo ? kW : (j == m - kHalo ? kE : -1);
}

// ---------------------------------------------------------------------------
// Tile phases
// ---------------------------------------------------------------------------
// A CTA of kTileThreads threads computes one TI x TJ tile of one face, as lists
// of independent items spread over the CTA: the points of the tile's stencil
// region, its faces, its cells.  (Below, "C96 8 x 16" and the like name a grid and a
// tile shape; times are us per RK2 substep of a graph round.)  The lists are row-major, so every global
// access of a warp is a run of consecutive cells and the shared-memory reads
// are conflict-free or nearly so.
//
// The stencil region of a tile is a cross: the tile's columns extended by 3
// rows on each side (the "vertical bar", read along i by the x faces) and
// the tile's rows extended by 3 columns on each side (the "horizontal bar",
// read along j by the y faces).  A region point is loaded, or gathered from
// the neighbouring face's bands where it lies in the halo, by one thread, which
// stores what the stencils read: h, the contravariant velocity normal to the
// faces that read the point, and the raw velocity tangential to them.  Cell
// and face constants are staged with cp.async in a prologue that does not
// depend on the state.
//
// 288 threads: with 8 x 16 tiles (the one-wave sizes) the 272 region points,
// the 280 faces and the edge items each fit one pass, so a CTA runs one face
// chain, not two; 8 x 32 and 16 x 16 tiles need two (552 and 544 faces; three
// with 256 threads), 16 x 32 four (1072).
constexpr int kTileThreads = 288;
// Threads of a TI x TJ tile's CTA: 416 for the fused kernel's 12 x 16 tiles (360
// region points, 412 faces).
constexpr int tile_threads(int ti) { return ti == 12 ? 416 : kTileThreads; }


// Resident CTAs per SM the phase kernels are compiled for (registers 65536 /
// (288 * blocks), rounded down to a multiple of 8).  A tile spends more than half
// of its time waiting (loads, barriers, the face chain), so what counts in
// multi-wave launches (FP) is how many tiles share the SM.  Phase H: float32 has
// the registers for 4 (56; C384 16 x 32 66.6 -> 62.4 us per substep; 5 with 52
// bytes spilled 61.2 against 59.4, with phase UV at 5), float64 for 3 (72; C384
// 16 x 16 141.3, with 4 and 60 bytes spilled 153.1).  One-wave launches keep 3:
// no more tiles are there to share.
template <typename T, bool FP>
struct PhaseBlocksH {
  static constexpr int value = sizeof(T) == 4 && FP ? 4 : 3;
};
template <typename T, int KP, bool FP>
struct PhaseBlocksUV {
  // float64 tiles of two region points per thread in multi-wave launches: 4 (C384 16 x 16 136.7 us per
  // substep against 144.3 at 3, 8 x 32 151.5 against 156.4); in one-wave launches (C96 8 x 32 21.2 at 4
  // against 19.5) and with one point (C48 8 x 16 14.4 against 12.9) or three (C384 16 x 32 156.5
  // against 154.0): 3.  float32 multi-wave: 5 (40 registers; C384 16 x 32 62.4 -> 59.4; 6 with 8 bytes
  // spilled 59.7).
  static constexpr int value = sizeof(T) == 4 ? (FP ? 5 : 3) : KP == 2 && FP ? 4 : 3;
};

constexpr int up4(int x) { return (x + 3) & ~3; }  // shared-memory offsets in words, 16-byte aligned

template <int TI, int TJ>
struct TileShape {
  static_assert(TJ == 16 || TJ == 32, "tile columns must be 16 or 32");
  static constexpr int kT = tile_threads(TI);
  static constexpr int RI = TI + 6, RJ = TJ + 6;    // stencil region
  static constexpr int VB = RI * TJ;                // vertical-bar points (r * TJ + q)
  static constexpr int NP = VB + 6 * TI;            // region points: vertical bar, then 3 W + 3 E columns per tile row
  static constexpr int FX = (TI + 1) * TJ;          // x faces (a * TJ + q)
  static constexpr int FY = TI * (TJ + 1);          // y faces (r * (TJ + 1) + q)
  static constexpr int C = TI * TJ;                 // cells (a * TJ + q)
  static constexpr int EW = TI > TJ ? TI : TJ;
  static constexpr int NE = 4 * EW;                 // edge slots: 4 kinds x max(TI, TJ) positions
  static constexpr int KP = (NP + kT - 1) / kT;  // region points per thread
  static constexpr int KC = (C + kT - 1) / kT;   // cells per thread
  // with one region point per thread its constants (metric, halo weights) are held in registers
  // across the wait for the previous phase; with more they are staged in shared memory
  static constexpr bool kHeld = KP == 1;
  // tile constant block (words): cells rda, rdx, rdy, a_f [C] each; x faces c_dy, y faces d_dx, x
  // faces dzph_x, y faces dzph_y
  static constexpr int FXP = up4(FX), FYP = up4(FY);
  static constexpr int bCDY = 4 * C, bDDX = bCDY + FXP, bDZX = bDDX + FYP, bDZY = bDZX + FXP, cW = bDZY + FYP;
  // phase H (words): s_h [RI][RJ], contravariant s_uc [VB] / s_vc [TI][RJ], raw s_v [VB] /
  // s_u [TI][RJ] (tangential reconstructions), face results x [4][FXP] and y [4][FYP] (sharing
  // memory with the staged region metric s_g [NP][4], s_sn [NP], dead by then), the constant
  // block, neighbour lines
  static constexpr int kFaceWords = 4 * (FXP + FYP), kMetricWords = kHeld ? 0 : 5 * NP;
  static constexpr int hH = 0, hUC = up4(hH + RI * RJ), hVC = up4(hUC + VB), hV = up4(hVC + TI * RJ),
                       hU = up4(hV + VB), hFX = up4(hU + TI * RJ), hFY = hFX + 4 * FXP,
                       hC = up4(hFX + (kFaceWords > kMetricWords ? kFaceWords : kMetricWords)), hNP = up4(hC + cW),
                       hNH = hNP + 6 * NE, hNDZ = hNH + 6 * NE, kWordsH = up4(hNDZ + NE);
  // phase UV (words): s_hn [RI][RJ], the (blended) new h of the region
  static constexpr int kWordsUV = up4(RI * RJ);
};

// Momentum terms of a cell handed from phase H to phase UV, kTerms planes.
// float64 keeps the three terms of each component apart, because the reference
// adds them to the pressure gradient one by one (barotr_pure.py:149-150); float32
// sums them.  The 8 x 16 tiles, whose terms the fused stage kernel reads beyond
// its own tile, keep planes over the interior cells of the faces, (6, N, N) each;
// the other shapes a block of planes [TI][TJ] per tile, at offsets known when the
// kernel is compiled (C384 float64 16 x 16 139.5 -> 137 us per substep, 16 x 32 163
// -> 155).
template <typename T>
constexpr int kTerms = sizeof(T) == 8 ? 6 : 2;

// Gradient of h along one axis at the centre of 7 values (agrid.py:55-69).
template <typename T>
__device__ __forceinline__ T gradient(T rd, const T* h) {
  return rd * (mid6(h + 1, 1) - mid6(h, 1));
}
// New velocity component (Y: along j) of a cell: the base, and dt times the
// pressure gradient (barotr_pure.py:57-60) of its h gradient ``gr`` plus the
// cell's momentum terms (barotr_pure.py:149-150).
template <typename T, bool Y>
__device__ __forceinline__ T momentum(T base, T gr, const T* tm, T dt) {
  if constexpr (kTerms<T> == 6) {
    const T pg = T(-9.80) * gr;
    return base + (Y ? pg + tm[3] - tm[4] + tm[5] : pg + tm[0] + tm[1] + tm[2]) * dt;
  } else {
    return mad(mad(T(-9.80), gr, tm[Y ? 1 : 0]), dt, base);
  }
}

struct TileBox {
  int f, i0, j0, ni, nj;
  int idx;  // number of the tile in face-major, row-major order
};

// a / b for 0 <= a < 2^24, b >= 1, without the integer division's long
// sequence (the quotient by reciprocal is off by one at most).
__device__ __forceinline__ int div24(int a, int b) {
  int q = __float2int_rz(__int2float_rn(a) * __frcp_rn(__int2float_rn(b)));
  const int r = a - q * b;
  if (r < 0) --q;
  if (r >= b) ++q;
  return q;
}

__device__ __forceinline__ TileBox tile_box_rc(const Tiling& t, int n, int f, int ti, int tj) {
  TileBox b;
  b.f = f;
  if (t.bi > 0) {  // even split
    b.i0 = kHalo + ti * t.bi + min(ti, t.ri);
    b.j0 = kHalo + tj * t.bj + min(tj, t.rj);
    b.ni = t.bi + (ti < t.ri ? 1 : 0);
    b.nj = t.bj + (tj < t.rj ? 1 : 0);
  } else {
    b.i0 = kHalo + ti * t.ti;
    b.j0 = kHalo + tj * t.tj;
    b.ni = min(t.ti, n - ti * t.ti);
    b.nj = min(t.tj, n - tj * t.tj);
  }
  b.idx = (f * t.nti + ti) * t.ntj + tj;
  return b;
}

// Tile number ``tile`` in face-major, row-major order.
__device__ __forceinline__ TileBox tile_box_at(const Tiling& t, int n, int tile) {
  const int f = div24(tile, t.nti * t.ntj), r = tile - f * (t.nti * t.ntj), ti = div24(r, t.ntj);
  return tile_box_rc(t, n, f, ti, r - ti * t.ntj);
}

// The tile that work item ``item`` (a CTA of a phase launch, or a step of a
// persistent CTA's tile loop) computes.  The tiles on the ring of each face's
// tile grid (those touching a face edge: halo gathers and edge averages make
// them the slowest) come first, the interior tiles after them, so that the
// long tiles start in the first wave instead of finishing a launch alone
// (largest work first); the faces take turns.  The batched phase kernels keep
// the face-major order instead (tile_box_at): with many members in one launch
// the last wave is short anyway, and neighbouring tiles running together share
// their halo rows in L2 (2.7 % faster there).
__device__ __forceinline__ TileBox tile_box(const Tiling& t, int n, int item) {
  const int nti = t.nti, ntj = t.ntj, f = item % 6;
  int r = item / 6, ti, tj;
  if (nti < 3 || ntj < 3) {  // every tile touches a face edge
    ti = div24(r, ntj);
    tj = r - ti * ntj;
  } else if (r < ntj) {
    ti = 0;
    tj = r;
  } else if ((r -= ntj) < ntj) {
    ti = nti - 1;
    tj = r;
  } else if ((r -= ntj) < nti - 2) {
    ti = 1 + r;
    tj = 0;
  } else if ((r -= nti - 2) < nti - 2) {
    ti = 1 + r;
    tj = ntj - 1;
  } else {
    r -= nti - 2;
    const int k = div24(r, ntj - 2);
    ti = 1 + k;
    tj = 1 + r - k * (ntj - 2);
  }
  return tile_box_rc(t, n, f, ti, tj);
}

// A full interior tile: TI x TJ cells whose whole stencil region (3 cells
// beyond each side) lies inside the face.  Such a tile needs no halo gather,
// no edge average and no bounds checks, so the tile phases are compiled
// separately for it (FULL = true) with its extents as constants.
__device__ __forceinline__ bool tile_full(const TileBox& b, int m, int ti, int tj) {
  return b.ni == ti && b.nj == tj && b.i0 >= 2 * kHalo && b.i0 + b.ni + kHalo <= m - kHalo &&
         b.j0 >= 2 * kHalo && b.j0 + b.nj + kHalo <= m - kHalo;
}

// 32-bit offset of cell (i, j) of face f (fields of up to 2^31 elements).
__device__ __forceinline__ int cell32(int f, int i, int j, int m) { return (f * m + i) * m + j; }

// Where a tile's momentum terms are.
template <typename T, int TI, int TJ, bool PLANAR>
struct TermsAt {
  T* p;
  int n;
  __device__ __forceinline__ TermsAt(T* fx, const TileBox& b, int n_)
      : p(PLANAR ? fx + (b.f * n_ + b.i0 - kHalo) * n_ + b.j0 - kHalo : fx + (long)b.idx * (kTerms<T> * TI * TJ)),
        n(n_) {}
  __device__ __forceinline__ explicit TermsAt(T* block) : p(block), n(0) {}  // a tile's block in shared memory
  __device__ __forceinline__ T& at(int z, int a, int q) const {
    return PLANAR ? p[z * (6 * n * n) + a * n + q] : p[z * (TI * TJ) + a * TJ + q];
  }
};
template <int TI, int TJ>
constexpr bool kPlanarTerms = TI == 8 && TJ == 16;

// ---- asynchronous global -> shared copies ---------------------------------
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  else if (BYTES == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_t(T* dst, const T* src) {
  cp_async<sizeof(T)>(dst, src);
}
template <typename T>
__device__ __forceinline__ void cp_async_mat(T* dst, const T* src) {  // 4 consecutive T
  if (sizeof(T) == 8) {
    cp_async<16>(dst, src);
    cp_async<16>(dst + 2, src + 2);
  } else {
    cp_async<16>(dst, src);
  }
}

// N (2 or 4) consecutive values from an address aligned to two values.
template <int N, typename T>
__device__ __forceinline__ void cp_async_pairs(T* dst, const T* src) {
#pragma unroll
  for (int k = 0; k < N; k += 2) cp_async<2 * sizeof(T)>(dst + k, src + k);
}

// One 2x2 matrix (four consecutive values) or one row of it with vector
// loads: bt_plan_create and bt_round_noalloc require the matrix arrays
// (a_c2l, a_l2c, a_gct) to start on a 16-byte boundary.
__device__ __forceinline__ void ld_quad(const float* p, float* q) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  q[0] = v.x;
  q[1] = v.y;
  q[2] = v.z;
  q[3] = v.w;
}
__device__ __forceinline__ void ld_quad(const double* p, double* q) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  q[0] = a.x;
  q[1] = a.y;
  q[2] = b.x;
  q[3] = b.y;
}
__device__ __forceinline__ void ld_pair(const float* p, float& a, float& b) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  a = v.x;
  b = v.y;
}
__device__ __forceinline__ void ld_pair(const double* p, double& a, double& b) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  a = v.x;
  b = v.y;
}

// ---- the tile's face-edge positions ----------------------------------------
// Item q of a tile's edge list: kind 0/1 = x faces of side S/N (position along
// the tile's columns), kind 2/3 = y faces of side W/E (along the tile's rows).
struct EdgeItem {
  int kind, pos, side, k;
};
// Edge positions of a tile per kind (S, N, W, E) and the routes of the
// tile's face across its four sides (8 bits each, kind order).  Scalars, not
// arrays: a dynamically indexed array would live in local memory, and each
// decode would wait on it.
struct EdgeCnt {
  int s, n, w, e, routes;
};
__device__ __forceinline__ int edge_count(const TileBox& b, int m, const int* route, EdgeCnt& c) {
  c.s = b.i0 == kHalo ? b.nj : 0;
  c.n = b.i0 + b.ni == m - kHalo ? b.nj : 0;
  c.w = b.j0 == kHalo ? b.ni : 0;
  c.e = b.j0 + b.nj == m - kHalo ? b.ni : 0;
  c.routes = route[b.f * 4 + kS] | (route[b.f * 4 + kN] << 8) | (route[b.f * 4 + kW] << 16) |
             (route[b.f * 4 + kE] << 24);
  return c.s + c.n + c.w + c.e;
}
__device__ __forceinline__ EdgeItem edge_item(const TileBox& b, const EdgeCnt& c, int q) {
  EdgeItem e;
  int kind;
  if (q < c.s) {
    kind = 0;
  } else if ((q -= c.s) < c.n) {
    kind = 1;
  } else if ((q -= c.n) < c.w) {
    kind = 2;
  } else {
    q -= c.w;
    kind = 3;
  }
  e.kind = kind;
  e.pos = q;
  e.side = kind == 0 ? kS : (kind == 1 ? kN : (kind == 2 ? kW : kE));
  e.k = kind < 2 ? (b.j0 + q - kHalo) : (b.i0 + q - kHalo);
  return e;
}

// ---- halo values from the bands ---------------------------------------------
// Band order: cell k along side s of face f, line c (0..2, increasing i or j)
// has number ((f * 4 + s) * 3 + c) * n + k, for the halo cells outside the side
// and for the interior cells inside it alike.
__device__ __forceinline__ int band_no(int f, int s, int c, int k, int n) { return ((f * 4 + s) * 3 + c) * n + k; }

// A point of a face by its coordinates: interior, or line c, position k of the
// halo band outside ``side`` (the corner blocks are never asked for).
struct PointKind {
  int side, c, k;  // side -1: interior
  __device__ __forceinline__ PointKind(int i, int j, int m) {
    side = -1;
    c = k = 0;
    if (i < kHalo) {
      side = kS;
      c = i;
      k = j - kHalo;
    } else if (i >= m - kHalo) {
      side = kN;
      c = i - (m - kHalo);
      k = j - kHalo;
    } else if (j < kHalo) {
      side = kW;
      c = j;
      k = i - kHalo;
    } else if (j >= m - kHalo) {
      side = kE;
      c = j - (m - kHalo);
      k = i - kHalo;
    }
  }
};

// The two band cells and weights a halo cell is interpolated from (cube.py:40-127).
template <typename T>
struct HaloRef {
  int b0, d;  // the second source is number b0 + d (added at use: the first is still in flight here)
  T w0, w1;
  __device__ __forceinline__ void load(const Geo<T>& g, int f, int side, int c, int k) {
    b0 = g.bsrc[band_no(f, side, c, k, g.n)];
    d = route_rev(g.route[f * 4 + side]) ? -1 : 1;  // the next along our edge
    ld_pair(g.hw + 2 * (f * g.nh + halo_word(g, side, c, k)), w0, w1);
  }
  // halo_id of a band cell
  __device__ __forceinline__ static int halo_word(const Geo<T>& g, int side, int c, int k) {
    return side == kS   ? c * g.m + kHalo + k
           : side == kN ? (3 + c) * g.m + kHalo + k
                        : 6 * g.m + (side == kE ? 3 * g.n : 0) + 3 * k + c;
  }
  __device__ __forceinline__ T lerp(const T* band) const { return lin2(w0, band[b0], w1, band[b0 + d]); }
};

// Halo velocity (ext_vector, cube.py:137-153) from the bands' lon/lat velocity
// and the target's l2c.
template <typename T>
__device__ __forceinline__ void halo_uv(const StageIO<T>& io, const HaloRef<T>& r, int plane, const T* l2, T& u, T& v) {
  const T ull = r.lerp(io.band_uv), vll = r.lerp(io.band_uv + plane);
  u = lin2(l2[0], ull, l2[1], vll);
  v = lin2(l2[2], ull, l2[3], vll);
}

// Words of one band plane.
__host__ __device__ __forceinline__ int band_plane(int n) { return 72 * n; }

// Whether a cell lies on one of the three lines next to a side of its face.
__device__ __forceinline__ bool in_bands(int i, int j, int n) {
  return min(i, j) < 2 * kHalo || max(i, j) >= n;
}

// Run fn(side, band number) for every side whose three interior lines hold cell (i, j) of face f.
template <typename F>
__device__ __forceinline__ void for_bands(int f, int i, int j, int n, F fn) {
  const int a = i - kHalo, b = j - kHalo;
  if (a < kHalo) fn((int)kS, band_no(f, kS, a, b, n));
  if (a >= n - kHalo) fn((int)kN, band_no(f, kN, a - (n - kHalo), b, n));
  if (b < kHalo) fn((int)kW, band_no(f, kW, b, a, n));
  if (b >= n - kHalo) fn((int)kE, band_no(f, kE, b - (n - kHalo), a, n));
}

// Shared-memory pointers of the tile-resident round kernel.
template <typename T>
struct ResSm {
  T* terms;  // momentum terms [kTerms][TI][TJ]
};

// Normal velocity of the neighbour's line (6 contravariant values) before averaging.
template <typename T>
__device__ __forceinline__ T line_raw(const T* np) {
  return T(0.5) * (rplus(np, 1) + rminus(np + 1, 1));
}

// Wait for the previous kernel of the stream (programmatic dependent launch);
// a no-op when the kernel was launched without a programmatic dependency.
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// Allow the next kernel of the stream to start its prologue.
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Celerity sqrt(g (h + dz)) with the 10 m/s floor and the viscosity
// coefficient 4.9 / celerity (barotr_pure.py:21-33).  float64 keeps IEEE
// sqrt and division like the reference; the float32 form takes the
// reciprocal square root once (sqrt = x * rsqrt(x)), with the same floor and
// NaN propagation.
template <typename T>
__device__ __forceinline__ void celerity_coef(T hface, T dz, T& c, T& coef) {
  if constexpr (sizeof(T) == 8) {
    c = celerity(hface, dz);
    coef = T(4.9) / c;
  } else {
    const float x = 9.8f * (hface + dz);
    if (x > 0.0f) {
      const float r = rsqrtf(x);
      c = x * r;
      coef = 4.9f * r;
      if (c < 10.0f) {
        c = 10.0f;
        coef = 0.49f;
      }
    } else {  // zero, negative depth or NaN: the exact path
      c = celerity(hface, dz);
      coef = 4.9f / c;
    }
  }
}

// Values of a thread's items that only some threads have, or only some items:
// assigned under a condition and read under the same one.  In a kernel that loops
// over tiles or stages (LOOP) such a variable would stay live around the whole
// loop, because on the other path the register still holds what the iteration
// before left there; there it is set first.  (k_batch_round float64 16 x 32: 924
// bytes spilled without, 76 with; a mixed ensemble of 8 C48, 6 C96 and 2 C192
// members 352 -> 246 us per substep; k_round C192 16 x 32 101 -> 74.5; k_resident
// C96 8 x 16 27.8 -> 21.3.)  Kernels of one tile have no use for it (float32
// batch of that ensemble, one launch per phase: 100.8 without, 104.2 with).
template <bool LOOP, typename V>
__device__ __forceinline__ void begin_items(V& v) {
  if constexpr (LOOP) v = V{};
}
template <bool LOOP, typename V, int N>
__device__ __forceinline__ void begin_items(V (&v)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) begin_items<LOOP>(v[k]);
}

// ---- phase H ----------------------------------------------------------------
template <typename T, int TI, int TJ>
struct LayoutH {
  using S = TileShape<TI, TJ>;
  static constexpr int kSlotS = 0, kSlotN = S::EW, kSlotW = 2 * S::EW, kSlotE = 3 * S::EW;  // neighbour lines
  T *s_h, *s_uc, *s_vc, *s_v, *s_u, *s_g, *s_sn, *s_fx, *s_fy, *s_cell, *s_cdy, *s_ddx, *s_dzx, *s_dzy, *s_np, *s_nh,
      *s_ndz;
  __device__ __forceinline__ explicit LayoutH(T* sm) {
    s_h = sm + S::hH;
    s_uc = sm + S::hUC;
    s_vc = sm + S::hVC;
    s_v = sm + S::hV;
    s_u = sm + S::hU;
    s_g = sm + S::hFX;
    s_sn = s_g + 4 * S::NP;
    s_fx = sm + S::hFX;
    s_fy = sm + S::hFY;
    s_cell = sm + S::hC;
    s_cdy = s_cell + S::bCDY;
    s_ddx = s_cell + S::bDDX;
    s_dzx = s_cell + S::bDZX;
    s_dzy = s_cell + S::bDZY;
    s_np = sm + S::hNP;
    s_nh = sm + S::hNH;
    s_ndz = sm + S::hNDZ;
  }
};

// Region point number p of a tile: region row r and column c, and whether the
// tile has it (partial tiles).
template <int TI, int TJ, bool FULL>
struct RegionPoint {
  int r, c;
  bool on, vbar, hbar;  // on the vertical bar (tile columns) / horizontal bar (tile rows)
  __device__ __forceinline__ RegionPoint(const TileBox& b, int p) {
    using S = TileShape<TI, TJ>;
    const int ni = FULL ? TI : b.ni, nj = FULL ? TJ : b.nj;
    if (p < S::VB) {
      r = p / TJ;
      c = p % TJ + kHalo;
      vbar = true;
      hbar = r >= kHalo && r < ni + kHalo;
      on = r < ni + 6 && c < nj + kHalo;
    } else {
      const int s = p - S::VB, a = s / 6, d = s - 6 * a;
      r = a + kHalo;
      c = d < 3 ? d : nj + d;
      vbar = false;
      hbar = true;
      on = a < ni;
    }
  }
};

// Depth d (0..2) of the neighbour's lines normal to the shared edge: a line has
// six points at edge position e of the tile, three inside the neighbouring face
// nb (line d inside its side ns) and three in its halo (line d outside), at
// position kk along that side; slots of the two points in the tile's line
// arrays, and which of them is the first point past the edge face (the depth
// is read there).
struct LinePoint {
  int nb, ns, kk, d, slot_in, slot_out;
  bool low, y;  // low: the halo points come first; y: the lines run along axis -1
  __device__ __forceinline__ LinePoint(const TileBox& b, const EdgeCnt& cnt, int P, int t, int n, int EW) {
    d = div24(t, P);
    const EdgeItem e = edge_item(b, cnt, t - d * P);
    const int r = (cnt.routes >> (8 * e.kind)) & 0xff;
    nb = route_nb(r);
    ns = route_side(r);
    kk = route_rev(r) ? n - 1 - e.k : e.k;
    low = ns == kS || ns == kW;
    y = ns == kE || ns == kW;
    const int base = (e.kind * EW + e.pos) * 6;
    slot_in = base + (low ? 3 + d : d);
    slot_out = base + (low ? d : 3 + d);
  }
  __device__ __forceinline__ int offset(bool out, int m) const {  // cell offset of the halo / inside point
    int i, j;
    edge_point(ns, kk, out == low ? d : 3 + d, m, i, j);
    return cell32(nb, i, j, m);
  }
};

// Constants of one halo value: its two sources and l2c, and for a line's halo
// point the metric row along the line.
template <typename T>
struct HaloWork {
  HaloRef<T> ref;
  T l2[4], g0, g1, sn;
  __device__ __forceinline__ void line_constants(const Geo<T>& g, const LinePoint& p) {
    const int o = p.offset(true, g.m);
    ld_quad(g.l2c + 4 * (long)o, l2);
    ld_pair(g.gct + 4 * (long)o + (p.y ? 2 : 0), g0, g1);
    sn = g.sina[o];
  }
};

// The lines' inside points (and depths) of an edge tile, line point t: the
// contravariant velocity along the line and, on the last stage, h come from the
// neighbour's bands as they are (cp.async).
template <typename T, int TI, int TJ>
__device__ __forceinline__ void line_inside(const Geo<T>& g, const StageIO<T>& io, const LinePoint& p,
                                            const LayoutH<T, TI, TJ>& L) {
  const int e = band_no(p.nb, p.ns, p.d, p.kk, g.n);
  cp_async_t(L.s_np + p.slot_in, (const T*)io.band_uv + 2 * band_plane(g.n) + e);
  if (io.last) cp_async_t(L.s_nh + p.slot_in, io.band_h + e);
}
template <typename T, int TI, int TJ>
__device__ __forceinline__ void line_depth(const Geo<T>& g, const LinePoint& p, const LayoutH<T, TI, TJ>& L) {
  if (p.d == 0) {  // point 3 of the line: the first past the edge face
    const int slot = (p.slot_in < p.slot_out ? p.slot_in : p.slot_out) / 6;
    cp_async_t(L.s_ndz + slot, (p.y ? g.dzph_y : g.dzph_x) + p.offset(!p.low, g.m));
  }
}
// The lines' halo points: line point t, its value gathered like a halo point's.
template <typename T, int TI, int TJ>
__device__ __forceinline__ void line_outside(const StageIO<T>& io, int slot, const HaloWork<T>& w, int plane,
                                             const LayoutH<T, TI, TJ>& L) {
  T u, v;
  halo_uv(io, w.ref, plane, w.l2, u, v);
  L.s_np[slot] = lin2(w.g0, u, w.g1, v) * w.sn;  // remap.py:34-39
  if (io.last) L.s_nh[slot] = w.ref.lerp(io.band_h);
}
// Both points of a line read directly (first stage of a round: the halo cells are stored).
template <typename T, int TI, int TJ>
__device__ __forceinline__ void line_stored(const Geo<T>& g, const StageIO<T>& io, const LinePoint& p,
                                            const LayoutH<T, TI, TJ>& L) {
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const int o = p.offset(k != 0, g.m), slot = k ? p.slot_out : p.slot_in;
    L.s_np[slot] = contra(g, (long)o, io.u[o], io.v[o], p.y);
    if (io.last) L.s_nh[slot] = io.h[o];
  }
}

// On the last stage the mass flux of an edge face is averaged with the
// neighbour's: from the gathered 6-point lines (slot = edge kind x EW +
// position) the neighbour's reconstructed face h values and celerity viscosity
// coefficient replace the line's first three h values, and its raw C-grid
// normal velocity (line_raw) the first velocity value.  Run between two
// barriers, one edge position per thread, so that the face pass of an edge
// face carries one square root and division chain instead of two; on the other
// stages the face pass forms line_raw itself and the extra barrier is saved.
template <typename T, int EW>
__device__ __forceinline__ void edge_lines(const TileBox& b, const EdgeCnt& cnt, int P, T* s_np, T* s_nh,
                                           const T* s_ndz) {
#pragma unroll 1
  for (int k = threadIdx.x; k < P; k += kTileThreads) {
    const EdgeItem e = edge_item(b, cnt, k);
    const int slot = e.kind * EW + e.pos;
    T* np = s_np + 6 * slot;
    T* nh = s_nh + 6 * slot;
    const T lr = line_raw(np);
    const T nhe = rplus(nh, 1), nhw = rminus(nh + 1, 1);
    T nc, ncoef;
    celerity_coef(mid6(nh, 1), s_ndz[slot], nc, ncoef);
    nh[0] = nhe;
    nh[1] = nhw;
    nh[2] = ncoef;
    np[0] = lr;
  }
}

// Phase H of one x face or y face: C-grid normal velocity (remap.py:41-55)
// and its edge average (communication.py:504-570), upwind mass flux with the
// celerity-based velocity viscosity (barotr_pure.py:21-49) and its edge
// average on the last stage, upwind tangential component (remap.py:73-95),
// kinetic energy (barotr_pure.py:91-92) and celerity-viscosity flux
// (barotr_pure.py:68-69).  ph / pu / pt: the 6 h / contravariant / raw
// tangential values along the face normal (strides sh / su / su); len: c_dy or
// d_dx of the face; side, slot: the face edge it lies on (-1: none) and its
// staged line.  Writes four planes ``plane`` words apart: mass flux x len,
// kinetic energy, tangential velocity x len, celerity-viscosity flux.
template <typename T>
__device__ __forceinline__ void face_h(const StageIO<T>& io, const T* ph, int sh, const T* pu, const T* pt, int su,
                                       int side, int slot, T dz, T len, const T* s_np, const T* s_nh, const T* s_ndz,
                                       T* fo, int plane) {
  T hh[6], uu[6], tt[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    hh[k] = ph[k * sh];
    uu[k] = pu[k * su];
    tt[k] = pt[k * su];
  }
  const T ue = rplus(uu, 1), uw = rminus(uu + 1, 1);
  T bc = T(0.5) * (ue + uw);
  if (side >= 0)  // with the neighbour's raw normal velocity
    bc = (bc + (io.last ? s_np[6 * slot] : line_raw(s_np + 6 * slot))) / T(2.0);
  const T he = rplus(hh, 1), hw = rminus(hh + 1, 1);
  T cc, coef;
  celerity_coef(mid6(hh, 1), dz, cc, coef);
  const T vis = mad(coef, he - hw, bc);
  T fl = lin2(dz, vis, vis > T(0.0) ? he : hw, vis);
  if (io.last && side >= 0) {  // the neighbour's flux at the same edge face (barotr_pure.py:29-49)
    const T* nh = s_nh + 6 * slot;
    const T ndz = s_ndz[slot];
    const T nvis = mad(nh[2], nh[0] - nh[1], bc);
    fl = (fl + lin2(ndz, nvis, nvis > T(0.0) ? nh[0] : nh[1], nvis)) / T(2.0);
  }
  const T vt = bc > T(0.0) ? rplus(tt, 1) : rminus(tt + 1, 1);
  fo[0] = fl * len;
  fo[plane] = T(0.5) * lin2(vis, vis, vt, vt);
  fo[2 * plane] = vt * len;
  fo[3 * plane] = T(0.5) * cc * (ue - uw);
}

// The tile's cell and face constants (cp.async, not yet awaited): its prepared
// block with 16-byte copies when the plan has one for this tile shape, else
// element by element from the constant arrays.
template <typename T, int TI, int TJ, typename LAY>
__device__ __forceinline__ void tile_consts(const Geo<T>& g, const TileBox& b, const LAY& L) {
  using S = TileShape<TI, TJ>;
  if (g.cblk != nullptr && g.cblk_ti == TI && g.cblk_tj == TJ) {
    constexpr int V = 16 / sizeof(T);
    const T* blk = g.cblk + (long)b.idx * S::cW;
#pragma unroll
    for (int w = 0; w < S::cW; w += S::kT * V) {
      const int e = w + (int)threadIdx.x * V;
      if (w + S::kT * V <= S::cW || e < S::cW) cp_async<16>(L.s_cell + e, blk + e);
    }
    return;
  }
  const int m = g.m, o0 = cell32(b.f, b.i0, b.j0, m);
#pragma unroll 1
  for (int e = threadIdx.x; e < S::FX; e += S::kT) {
    const int a = e / TJ, q = e % TJ, o = o0 + a * m + q;
    if (a > b.ni || q >= b.nj) continue;
    cp_async_t(L.s_dzx + e, g.dzph_x + o);
    cp_async_t(L.s_cdy + e, g.c_dy + o);
    if (a == b.ni) continue;
    cp_async_t(L.s_cell + e, g.rda + o);
    cp_async_t(L.s_cell + S::C + e, g.rdx + o);
    cp_async_t(L.s_cell + 2 * S::C + e, g.rdy + o);
    cp_async_t(L.s_cell + 3 * S::C + e, g.a_f + o);
  }
#pragma unroll 1
  for (int e = threadIdx.x; e < S::FY; e += S::kT) {
    const int r = e / (TJ + 1), q = e - r * (TJ + 1), o = o0 + r * m + q;
    if (r >= b.ni || q > b.nj) continue;
    cp_async_t(L.s_dzy + e, g.dzph_y + o);
    cp_async_t(L.s_ddx + e, g.d_dx + o);
  }
}

// State-independent data of a tile held in registers from the prologue to the
// main part.  With one region point per thread (TileShape::kHeld) its metric,
// and one halo value's constants: those of the thread's region point if that
// lies in the halo, else -- float32 -- those of the line point it gathers.
// float64 has the registers for that line point's sources only (C96, 8 x 16:
// 13.97 us per substep; 14.54 with all its constants held and 11 registers
// spilled; float32 10.66 with all held against 11.56).  With more points per
// thread only the points' halo sources are held.
template <typename T, int TI, int TJ>
struct HPre {
  using S = TileShape<TI, TJ>;
  HaloRef<T> ref[S::kHeld ? 1 : S::KP];
  static constexpr bool kLineHeld = sizeof(T) == 4;
  HaloWork<T> halo;
  HaloRef<T> lref;
  T g[4], sn;
  int slot;  // the line halo point whose constants (kLineHeld) or sources are held, -1: none
  EdgeCnt cnt;
  int P;  // edge positions of the tile (0 for tiles that touch no face edge)
};

// Line points of a tile (3 per edge position) go to the threads from
// line_thread0 on, whose region points lie on the tile's own rows: interior
// points, except in tiles thinner than TI next to an N edge.
template <int TI, int TJ>
__device__ __forceinline__ int line_first() {
  constexpr int line_thread0 = kHalo * TJ;
  const int t = (int)threadIdx.x - line_thread0;
  return t >= 0 ? t : t + TileShape<TI, TJ>::kT;
}

// Metric, halo sources and line constants of the tile.
template <typename T, int TI, int TJ, bool FULL>
__device__ __forceinline__ void tile_h_points(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                              HPre<T, TI, TJ>& pre) {
  using S = TileShape<TI, TJ>;
  const int m = g.m;
  const LayoutH<T, TI, TJ> L(sm);
  pre.P = FULL ? 0 : edge_count(b, m, g.route, pre.cnt);
  pre.slot = -1;
  bool halo = false;
#pragma unroll
  for (int k = 0; k < S::KP; ++k) {
    const int p = k * S::kT + (int)threadIdx.x;
    if (p >= S::NP) continue;
    const RegionPoint<TI, TJ, FULL> pt(b, p);
    if (!pt.on) continue;
    const int i = b.i0 - kHalo + pt.r, j = b.j0 - kHalo + pt.c, o = cell32(b.f, i, j, m);
    if (!FULL && !io.stored_halo) {
      const PointKind pk(i, j, m);
      if (pk.side >= 0) {
        halo = true;
        if (S::kHeld) {
          pre.halo.ref.load(g, b.f, pk.side, pk.c, pk.k);
          ld_quad(g.l2c + 4 * (long)o, pre.halo.l2);
        } else {
          pre.ref[k].load(g, b.f, pk.side, pk.c, pk.k);
        }
      }
    }
    if constexpr (S::kHeld) {
      ld_quad(g.gct + 4 * (long)o, pre.g);
      pre.sn = g.sina[o];
    } else {
      cp_async_mat(L.s_g + 4 * p, g.gct + 4 * (long)o);
      cp_async_t(L.s_sn + p, g.sina + o);
    }
  }
  if (!FULL && pre.P > 0) {
#pragma unroll 1
    for (int t = line_first<TI, TJ>(); t < 3 * pre.P; t += S::kT) {
      const LinePoint lp(b, pre.cnt, pre.P, t, g.n, S::EW);
      if (io.last) line_depth<T, TI, TJ>(g, lp, L);
      if (S::kHeld && !io.stored_halo && t < S::kT) {
        if (!HPre<T, TI, TJ>::kLineHeld) {
          pre.slot = lp.slot_out;
          pre.lref.load(g, lp.nb, lp.ns, lp.d, lp.kk);
        } else if (!halo) {
          pre.slot = lp.slot_out;
          pre.halo.ref.load(g, lp.nb, lp.ns, lp.d, lp.kk);
          pre.halo.line_constants(g, lp);
        }
      }
    }
  }
}

// Phase H prologue: constants of the tile, metric, halo sources.  Independent
// of the state, so it may run before the previous phase has finished
// (programmatic launch, or before a grid barrier).
template <typename T, int TI, int TJ, bool FULL>
__device__ __forceinline__ void tile_h_pro_t(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                             HPre<T, TI, TJ>& pre) {
  tile_consts<T, TI, TJ>(g, b, LayoutH<T, TI, TJ>(sm));
  tile_h_points<T, TI, TJ, FULL>(g, io, b, sm, pre);
}

// The faces of a tile whose region is staged: x faces, then y faces.  When all
// of them fit one pass they run one copy of the face code with run-time strides
// (a warp may hold both kinds, and the code is fetched once); else each kind
// starts at a warp boundary.  hx0 / hy0: the first of the six h values of x face
// (0, 0) / y face (0, 0), rows HP apart; L: the tile's arrays (LayoutH or alike).
template <typename T, int TI, int TJ, bool FULL, int HP, typename LAY>
__device__ __forceinline__ void tile_faces(const StageIO<T>& io, const TileBox& b, int m, int ni, int nj, const T* hx0,
                                           const T* hy0, const LAY& L) {
  using S = TileShape<TI, TJ>;
  constexpr int RJ = S::RJ;
  auto x_face = [&](int e) {
    const int a = e / TJ, q = e % TJ;
    if (!FULL && (a > ni || q >= nj)) return;
    const int side =
        FULL ? -1 : ((a == 0 && b.i0 == kHalo) ? kS : ((a == ni && b.i0 + ni == m - kHalo) ? kN : -1));
    face_h<T>(io, hx0 + a * HP + q, HP, L.s_uc + e, L.s_v + e, TJ, side, (side == kS ? LAY::kSlotS : LAY::kSlotN) + q,
              L.s_dzx[e], L.s_cdy[e], L.s_np, L.s_nh, L.s_ndz, L.s_fx + e, S::FXP);
  };
  auto y_face = [&](int e) {
    const int r = e / (TJ + 1), q = e - r * (TJ + 1);
    if (!FULL && (r >= ni || q > nj)) return;
    const int side =
        FULL ? -1 : ((q == 0 && b.j0 == kHalo) ? kW : ((q == nj && b.j0 + nj == m - kHalo) ? kE : -1));
    face_h<T>(io, hy0 + r * HP + q, 1, L.s_vc + r * RJ + q, L.s_u + r * RJ + q, 1, side,
              (side == kW ? LAY::kSlotW : LAY::kSlotE) + r, L.s_dzy[e], L.s_ddx[e], L.s_np, L.s_nh, L.s_ndz, L.s_fy + e, S::FYP);
  };
  if constexpr (S::FX + S::FY <= S::kT) {
    const int t = threadIdx.x;
    if (t < S::FX + S::FY) {
      const bool y = t >= S::FX;
      const int e = y ? t - S::FX : t;
      const int a = y ? e / (TJ + 1) : e / TJ, q = y ? e - a * (TJ + 1) : e % TJ;
      const bool on = y ? (a < ni && q <= nj) : (a <= ni && q < nj);
      if (FULL || on) {
        int side = -1;
        if (!FULL) {
          const int z = y ? q : a, w = y ? nj : ni, i0 = y ? b.j0 : b.i0;
          if (z == 0 && i0 == kHalo) side = y ? kW : kS;
          if (z == w && i0 + w == m - kHalo) side = y ? kE : kN;
        }
        const int slot = y ? (side == kW ? LAY::kSlotW : LAY::kSlotE) + a : (side == kS ? LAY::kSlotS : LAY::kSlotN) + q;
        const int at = y ? a * RJ + q : e;
        face_h<T>(io, (y ? hy0 : hx0) + a * HP + q, y ? 1 : HP,
                  (y ? L.s_vc : L.s_uc) + at, (y ? L.s_u : L.s_v) + at, y ? 1 : TJ, side, slot,
                  (y ? L.s_dzy : L.s_dzx)[e], (y ? L.s_ddx : L.s_cdy)[e], L.s_np, L.s_nh, L.s_ndz,
                  (y ? L.s_fy : L.s_fx) + e, y ? S::FYP : S::FXP);
      }
    }
  } else {
    constexpr int XS = (S::FX + 31) & ~31;  // y faces start here
#pragma unroll
    for (int z = 0; z < XS + S::FY; z += S::kT) {
      const int t = z + (int)threadIdx.x;
      if (z < S::FX && t < S::FX)
        x_face(t);
      else if (z + S::kT > XS && t >= XS && t < XS + S::FY)
        y_face(t - XS);
    }
  }
}

// The cells of a tile whose faces are computed: divergence (agrid.py:43-53) and
// the h update (barotr_pure.py:119-120), vorticity (agrid.py:31-41), advection
// (barotr_pure.py:78-97), Coriolis, celerity viscosity (barotr_pure.py:63-75).
// hpc: the base h of the thread's cells.
template <typename T, int TI, int TJ, bool FULL, typename LAY, typename TERMS>
__device__ __forceinline__ void tile_cells(const StageIO<T>& io, const TileBox& b, int n, int m, int ni, int nj,
                                           const T* hpc, const TERMS& ta, const LAY& L) {
  using S = TileShape<TI, TJ>;
  constexpr int RJ = S::RJ;
  const int f = b.f, o0 = cell32(f, b.i0, b.j0, m);
#pragma unroll
  for (int k = 0; k < S::KC; ++k) {
    const int e = k * S::kT + (int)threadIdx.x, a = e / TJ, q = e % TJ;
    if (a < ni && q < nj) {
      const T* X = L.s_fx + e;
      const T* Y = L.s_fy + a * (TJ + 1) + q;
      const T* c = L.s_cell + e;
      const T rda = c[0], rdx = c[S::C], rdy = c[2 * S::C], af = c[3 * S::C];
      const T div = rda * (X[TJ] - X[0] + Y[1] - Y[0]);
      const T hn = mad(-div, io.dt, hpc[k]);
      io.h_out[o0 + a * m + q] = hn;
      if (!FULL) for_bands(f, b.i0 + a, b.j0 + q, n, [&](int, int z) { io.band_hn[z] = hn; });
      const T uct = L.s_uc[(a + kHalo) * TJ + q], vct = L.s_vc[a * RJ + q + kHalo];
      const T* kx = X + S::FXP;
      const T* ky = Y + S::FYP;
      const T* tx = X + 2 * S::FXP;
      const T* ty = Y + 2 * S::FYP;
      const T* vx = X + 3 * S::FXP;
      const T* vy = Y + 3 * S::FYP;
      const T vort = rda * (ty[0] + tx[TJ] - ty[1] - tx[0]);
      const T advx = lin2(vort, vct, -(kx[TJ] - kx[0]), rdx);
      const T advy = lin2(-vort, uct, -(ky[1] - ky[0]), rdy);
      if constexpr (kTerms<T> == 6) {
        const T visx = -(rdx * (vx[TJ] - vx[0]));
        const T visy = -(rdy * (vy[1] - vy[0]));
        ta.at(0, a, q) = advx;
        ta.at(1, a, q) = af * vct;
        ta.at(2, a, q) = visx;
        ta.at(3, a, q) = advy;
        ta.at(4, a, q) = af * uct;
        ta.at(5, a, q) = visy;
      } else {
        ta.at(0, a, q) = mad(-rdx, vx[TJ] - vx[0], mad(af, vct, advx));
        ta.at(1, a, q) = mad(-rdy, vy[1] - vy[0], mad(-af, uct, advy));
      }
    }
  }
}

// Phase H of one tile: writes the new h and the momentum terms of the tile's
// interior cells, and the new h of its cells in the face's bands.  RES
// (tile-resident round): the terms stay on chip.
template <typename T, int TI, int TJ, bool FULL, bool LOOP, bool RES = false>
__device__ __forceinline__ void tile_h_main_t(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                              const HPre<T, TI, TJ>& pre, const ResSm<T>& rs = ResSm<T>{}) {
  using S = TileShape<TI, TJ>;
  constexpr int RJ = S::RJ;
  const int m = g.m, n = g.n, f = b.f;
  const int ni = FULL ? TI : b.ni, nj = FULL ? TJ : b.nj;
  const LayoutH<T, TI, TJ> L(sm);
  const int o0 = cell32(f, b.i0, b.j0, m);

  // region: state of the thread's points (halo points from the bands) and base h of its cells
  T hv[S::KP], uv[S::KP], vv[S::KP], hpc[S::KC];
  begin_items<LOOP>(hv);
  begin_items<LOOP>(uv);
  begin_items<LOOP>(vv);
  begin_items<LOOP>(hpc);
#pragma unroll
  for (int k = 0; k < S::KP; ++k) {
    const int p = k * S::kT + (int)threadIdx.x;
    if (p >= S::NP) continue;
    const RegionPoint<TI, TJ, FULL> pt(b, p);
    if (!pt.on) continue;
    const int o = o0 + (pt.r - kHalo) * m + pt.c - kHalo;
    if (!FULL && !io.stored_halo) {
      const int i = b.i0 - kHalo + pt.r, j = b.j0 - kHalo + pt.c;
      const PointKind pk(i, j, m);
      if (pk.side >= 0) {
        T l2[4];
        if (!S::kHeld) ld_quad(g.l2c + 4 * (long)o, l2);
        const HaloRef<T>& ref = S::kHeld ? pre.halo.ref : pre.ref[k];
        halo_uv(io, ref, band_plane(n), S::kHeld ? pre.halo.l2 : l2, uv[k], vv[k]);
        hv[k] = ref.lerp(io.band_h);
        continue;
      }
    }
    hv[k] = io.h[o];
    uv[k] = io.u[o];
    vv[k] = io.v[o];
  }
#pragma unroll
  for (int k = 0; k < S::KC; ++k) {
    const int c = k * S::kT + (int)threadIdx.x, a = c / TJ, q = c % TJ;
    if (a < ni && q < nj) hpc[k] = io.hp[o0 + a * m + q];
  }
  if (!FULL && pre.P > 0) {
#pragma unroll 1
    for (int t = line_first<TI, TJ>(); t < 3 * pre.P; t += S::kT) {
      const LinePoint lp(b, pre.cnt, pre.P, t, n, S::EW);
      if (io.stored_halo) {
        line_stored<T, TI, TJ>(g, io, lp, L);
      } else {
        line_inside<T, TI, TJ>(g, io, lp, L);
        const bool held = S::kHeld && lp.slot_out == pre.slot;
        if (!(HPre<T, TI, TJ>::kLineHeld && held)) {
          HaloWork<T> w;
          if (held)
            w.ref = pre.lref;
          else
            w.ref.load(g, lp.nb, lp.ns, lp.d, lp.kk);
          w.line_constants(g, lp);
          line_outside<T, TI, TJ>(io, lp.slot_out, w, band_plane(n), L);
        }
      }
    }
    if (S::kHeld && HPre<T, TI, TJ>::kLineHeld && pre.slot >= 0)
      line_outside<T, TI, TJ>(io, pre.slot, pre.halo, band_plane(n), L);
  }
  if (!S::kHeld) {
    cp_async_wait_all();
    __syncthreads();
  }
  // h, raw and contravariant velocities (remap.py:34-39)
#pragma unroll
  for (int k = 0; k < S::KP; ++k) {
    const int p = k * S::kT + (int)threadIdx.x;
    if (p >= S::NP) continue;
    const RegionPoint<TI, TJ, FULL> pt(b, p);
    if (!pt.on) continue;
    const T* G = S::kHeld ? pre.g : L.s_g + 4 * p;
    const T sn = S::kHeld ? pre.sn : L.s_sn[p];
    const T u = uv[k], v = vv[k];
    L.s_h[pt.r * RJ + pt.c] = hv[k];
    if (pt.vbar) {
      L.s_uc[pt.r * TJ + pt.c - kHalo] = lin2(G[0], u, G[1], v) * sn;
      L.s_v[pt.r * TJ + pt.c - kHalo] = v;
    }
    if (pt.hbar) {
      L.s_vc[(pt.r - kHalo) * RJ + pt.c] = lin2(G[2], u, G[3], v) * sn;
      L.s_u[(pt.r - kHalo) * RJ + pt.c] = u;
    }
  }
  if (S::kHeld) {
    cp_async_wait_all();
    __syncthreads();
  }
  const bool lines = !FULL && pre.P > 0 && io.last;
  if (lines) edge_lines<T, S::EW>(b, pre.cnt, pre.P, L.s_np, L.s_nh, L.s_ndz);
  if (!S::kHeld || lines) __syncthreads();

  tile_faces<T, TI, TJ, FULL, RJ>(io, b, m, ni, nj, L.s_h + kHalo, L.s_h + kHalo * RJ, L);
  __syncthreads();
  if constexpr (RES)
    tile_cells<T, TI, TJ, FULL>(io, b, n, m, ni, nj, hpc, TermsAt<T, TI, TJ, false>(rs.terms), L);
  else
    tile_cells<T, TI, TJ, FULL>(io, b, n, m, ni, nj, hpc, TermsAt<T, TI, TJ, kPlanarTerms<TI, TJ>>(io.fx, b, n), L);
}

// ---- phase UV -----------------------------------------------------------------
// State-independent data of phase UV held in registers from the prologue: the
// thread's cell constants (with the metric of cells in the bands) and, with one
// region point per thread, its halo sources.
template <typename T, int TI, int TJ>
struct UvPre {
  using S = TileShape<TI, TJ>;
  T rdx[S::KC], rdy[S::KC];
  HaloRef<T> ref[S::KP];
  static constexpr bool kBandHeld = S::KC == 1;
  T c2[4], g[4], sn;  // of a cell in the bands (kBandHeld; else loaded at use)
};

template <typename T, int TI, int TJ, bool FULL>
__device__ __forceinline__ void tile_uv_pro_t(const Geo<T>& g, const TileBox& b, UvPre<T, TI, TJ>& pre) {
  using S = TileShape<TI, TJ>;
  const int m = g.m, o0 = cell32(b.f, b.i0, b.j0, m);
  const int ni = FULL ? TI : b.ni, nj = FULL ? TJ : b.nj;
#pragma unroll
  for (int k = 0; k < S::KC; ++k) {
    const int c = k * S::kT + (int)threadIdx.x, a = c / TJ, q = c % TJ;
    if (a < ni && q < nj) {
      pre.rdx[k] = g.rdx[o0 + a * m + q];
      pre.rdy[k] = g.rdy[o0 + a * m + q];
      if (!FULL && UvPre<T, TI, TJ>::kBandHeld && in_bands(b.i0 + a, b.j0 + q, g.n)) {
        const long o = o0 + a * m + q;
        ld_quad(g.c2l + 4 * o, pre.c2);
        ld_quad(g.gct + 4 * o, pre.g);
        pre.sn = g.sina[o];
      }
    }
  }
  if (!FULL) {
#pragma unroll
    for (int k = 0; k < S::KP; ++k) {
      const int p = k * S::kT + (int)threadIdx.x;
      if (p >= S::NP) continue;
      const RegionPoint<TI, TJ, FULL> pt(b, p);
      if (!pt.on) continue;
      const PointKind pk(b.i0 - kHalo + pt.r, b.j0 - kHalo + pt.c, m);
      if (pk.side >= 0) pre.ref[k].load(g, b.f, pk.side, pk.c, pk.k);
    }
  }
}

// Phase UV of one tile: pressure gradient of the new h (agrid.py:55-69,
// barotr_pure.py:57-60) and the momentum update (barotr_pure.py:149-150) with
// phase H's terms; the lon/lat and normal contravariant velocity of the tile's
// cells in the face's bands.  RES (tile-resident round): the terms are in
// shared memory.
template <typename T, int TI, int TJ, bool FULL, bool LOOP, bool RES = false>
__device__ __forceinline__ void tile_uv_main_t(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                               const UvPre<T, TI, TJ>& pre, const ResSm<T>& rs = ResSm<T>{}) {
  using S = TileShape<TI, TJ>;
  constexpr int RJ = S::RJ;
  const int m = g.m, n = g.n, f = b.f;
  const int ni = FULL ? TI : b.ni, nj = FULL ? TJ : b.nj;
  const bool blend = io.beta != T(0.0);  // fb_scheme needs the stage h only when beta_d != 0
  const T* hn_src = (const T*)io.h_out;
  const T* hn_band = (const T*)io.band_hn;
  const int o0 = cell32(f, b.i0, b.j0, m);

  // new h of the region, blended with the stage h (fb_scheme, barotr_pure.py:52-54)
  T hn[S::KP], hs[S::KP];
  begin_items<LOOP>(hn);
  begin_items<LOOP>(hs);
#pragma unroll
  for (int k = 0; k < S::KP; ++k) {
    const int p = k * S::kT + (int)threadIdx.x;
    if (p >= S::NP) continue;
    const RegionPoint<TI, TJ, FULL> pt(b, p);
    if (!pt.on) continue;
    const int o = o0 + (pt.r - kHalo) * m + pt.c - kHalo;
    if (!FULL) {
      const PointKind pk(b.i0 - kHalo + pt.r, b.j0 - kHalo + pt.c, m);
      if (pk.side >= 0) {  // the new h never has a stored halo
        hn[k] = pre.ref[k].lerp(hn_band);
        if (blend) hs[k] = io.stored_halo ? io.h[o] : pre.ref[k].lerp(io.band_h);
        continue;
      }
    }
    hn[k] = hn_src[o];
    if (blend) hs[k] = io.h[o];
  }
  // base velocities and terms of the thread's cells
  T upc[S::KC], vpc[S::KC], tm[S::KC][kTerms<T>];
  begin_items<LOOP>(upc);
  begin_items<LOOP>(vpc);
  begin_items<LOOP>(tm);
  const auto ta = [&] {
    if constexpr (RES)
      return TermsAt<T, TI, TJ, false>(rs.terms);
    else
      return TermsAt<T, TI, TJ, kPlanarTerms<TI, TJ>>(io.fx, b, n);
  }();
#pragma unroll
  for (int k = 0; k < S::KC; ++k) {
    const int c = k * S::kT + (int)threadIdx.x, a = c / TJ, q = c % TJ;
    if (a < ni && q < nj) {
      upc[k] = io.up[o0 + a * m + q];
      vpc[k] = io.vp[o0 + a * m + q];
#pragma unroll
      for (int z = 0; z < kTerms<T>; ++z) tm[k][z] = ta.at(z, a, q);
    }
  }
#pragma unroll
  for (int k = 0; k < S::KP; ++k) {
    const int p = k * S::kT + (int)threadIdx.x;
    if (p >= S::NP) continue;
    const RegionPoint<TI, TJ, FULL> pt(b, p);
    if (!pt.on) continue;
    sm[pt.r * RJ + pt.c] = blend ? lin2(T(1.0) - io.beta, hn[k], io.beta, hs[k]) : hn[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < S::KC; ++k) {
    const int c = k * S::kT + (int)threadIdx.x, a = c / TJ, q = c % TJ;
    if (a < ni && q < nj) {
      T hx[7], hy[7];
#pragma unroll
      for (int z = 0; z < 7; ++z) {
        hx[z] = sm[(a + z) * RJ + q + kHalo];
        hy[z] = sm[(a + kHalo) * RJ + q + z];
      }
      const T gx = gradient(pre.rdx[k], hx), gy = gradient(pre.rdy[k], hy);
      const int o = o0 + a * m + q;
      const T u = momentum<T, false>(upc[k], gx, tm[k], io.dt);
      const T v = momentum<T, true>(vpc[k], gy, tm[k], io.dt);
      io.u_out[o] = u;
      io.v_out[o] = v;
      if (!FULL && in_bands(b.i0 + a, b.j0 + q, n)) {
        // the bands: lon/lat velocity (cube.py:137-145) and normal contravariant component (remap.py:34-39)
        T c2[4], G[4], sn;
        if constexpr (UvPre<T, TI, TJ>::kBandHeld) {
#pragma unroll
          for (int z = 0; z < 4; ++z) {
            c2[z] = pre.c2[z];
            G[z] = pre.g[z];
          }
          sn = pre.sn;
        } else {
          ld_quad(g.c2l + 4 * (long)o, c2);
          ld_quad(g.gct + 4 * (long)o, G);
          sn = g.sina[o];
        }
        const T ull = lin2(c2[0], u, c2[1], v), vll = lin2(c2[2], u, c2[3], v);
        const T uct = lin2(G[0], u, G[1], v) * sn, vct = lin2(G[2], u, G[3], v) * sn;
        T* const bu = io.band_uv;
        const int plane = band_plane(n);
        for_bands(f, b.i0 + a, b.j0 + q, n, [&](int side, int z) {
          bu[z] = ull;
          bu[plane + z] = vll;
          bu[2 * plane + z] = side == kE || side == kW ? vct : uct;
        });
      }
    }
  }
}

// Tile phases dispatched on the tile's kind: with FP (the full-tile path
// compiled in), full interior tiles run the FULL = true instantiation and the
// others the edge instantiation; without it every tile runs the edge
// instantiation, which handles full tiles too.  The kernel without the full
// path is about half the code: at one-wave sizes (every CTA runs the code
// once, and instruction fetch is the largest stall) it is the faster one.
// Prologue and main part of one tile take the same branch, since both test
// the same tile box.
template <typename T, int TI, int TJ, bool FP = true>
__device__ __forceinline__ void tile_h_pro(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                           HPre<T, TI, TJ>& pre) {
  if (FP && tile_full(b, g.m, TI, TJ))
    tile_h_pro_t<T, TI, TJ, true>(g, io, b, sm, pre);
  else
    tile_h_pro_t<T, TI, TJ, false>(g, io, b, sm, pre);
}
template <typename T, int TI, int TJ, bool FP, bool LOOP>
__device__ __forceinline__ void tile_h_main(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                            const HPre<T, TI, TJ>& pre) {
  if (FP && tile_full(b, g.m, TI, TJ))
    tile_h_main_t<T, TI, TJ, true, LOOP>(g, io, b, sm, pre);
  else
    tile_h_main_t<T, TI, TJ, false, LOOP>(g, io, b, sm, pre);
}
template <typename T, int TI, int TJ, bool FP = true>
__device__ __forceinline__ void tile_uv_pro(const Geo<T>& g, const TileBox& b, UvPre<T, TI, TJ>& pre) {
  if (FP && tile_full(b, g.m, TI, TJ))
    tile_uv_pro_t<T, TI, TJ, true>(g, b, pre);
  else
    tile_uv_pro_t<T, TI, TJ, false>(g, b, pre);
}
template <typename T, int TI, int TJ, bool FP, bool LOOP>
__device__ __forceinline__ void tile_uv_main(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                             const UvPre<T, TI, TJ>& pre) {
  if (FP && tile_full(b, g.m, TI, TJ))
    tile_uv_main_t<T, TI, TJ, true, LOOP>(g, io, b, sm, pre);
  else
    tile_uv_main_t<T, TI, TJ, false, LOOP>(g, io, b, sm, pre);
}

// One tile phase with the prologue issued first (the stream/graph kernels).
template <typename T, int TI, int TJ, bool FP = true>
__device__ __forceinline__ void tile_h(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                       int late = 0) {
  HPre<T, TI, TJ> pre;
  tile_h_pro<T, TI, TJ, FP>(g, io, b, sm, pre);
  wait_prior_grid();
  if (late) release_dependents();
  tile_h_main<T, TI, TJ, FP, false>(g, io, b, sm, pre);
}
template <typename T, int TI, int TJ, bool FP = true>
__device__ __forceinline__ void tile_uv(const Geo<T>& g, const StageIO<T>& io, const TileBox& b, T* sm,
                                       int late = 0) {
  UvPre<T, TI, TJ> pre;
  tile_uv_pro<T, TI, TJ, FP>(g, b, pre);
  wait_prior_grid();
  if (late) release_dependents();
  tile_uv_main<T, TI, TJ, FP, false>(g, io, b, sm, pre);
}


// ---------------------------------------------------------------------------
// Grid-wide barrier of the persistent round kernel
// ---------------------------------------------------------------------------
// Monotone arrival counter: the k-th barrier completes when the low 31 bits
// of the counter reach k * gridDim.x.  Thread 0 of each CTA arrives with a
// release reduction (publishing the CTA's writes, ordered by the preceding
// __syncthreads) and polls with acquire loads, at most ``limit`` times.  A CTA
// that gives up raises kErrBarrierTimeout and sets the counter's top bit, which
// every other CTA sees at its next poll: all CTAs then leave the round.
// Returns false when the round must stop.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned& gen, int* err, long long limit) {
  __shared__ int s_ok;
  constexpr unsigned kAbort = 0x80000000u;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++gen;
    const unsigned target = gen * gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    long long polls = 0;
    int ok = 1;
    while (true) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (seen & kAbort) {
        ok = 0;
        break;
      }
      if ((int)((seen & ~kAbort) - target) >= 0) break;
      if (++polls > limit) {
        atomicOr(err, kErrBarrierTimeout);
        atomicOr(bar, kAbort);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Stage pointers of (substep, stage) of a round, ``step`` counted from the
// round's first substep; mirrors the host schedule.
// Fields are picked with constant indexes only, so the kernel arguments are
// never addressed (which would copy them to local memory).
template <typename T>
__device__ __forceinline__ StageIO<T> round_stage(const RoundArgs<T>& a, int step, int st) {
  StageIO<T> io;
  const int nst = a.rk == 2 ? 2 : 3;
  const bool first = step == 0, last = st == nst - 1;
  // stage input: the round input (first substep) or the running state, then Y, then Z
  io.h = st == 0 ? (first ? a.x0[0] : a.x[0]) : (st == 1 ? a.y[0] : a.z[0]);
  io.u = st == 0 ? (first ? a.x0[1] : a.x[1]) : (st == 1 ? a.y[1] : a.z[1]);
  io.v = st == 0 ? (first ? a.x0[2] : a.x[2]) : (st == 1 ? a.y[2] : a.z[2]);
  io.hp = first ? a.b0[0] : a.x[0];
  io.up = first ? a.b0[1] : a.x[1];
  io.vp = first ? a.b0[2] : a.x[2];
  io.h_out = last ? a.x[0] : (st == 0 ? a.y[0] : a.z[0]);
  io.u_out = last ? a.x[1] : (st == 0 ? a.y[1] : a.z[1]);
  io.v_out = last ? a.x[2] : (st == 0 ? a.y[2] : a.z[2]);
  io.fx = a.fx;
  const int sg = step * nst + st;  // the new-h bands alternate between consecutive stages
  io.band_uv = a.band;
  io.band_h = a.band + (3 + (sg & 1)) * band_plane(a.g.n);
  io.band_hn = a.band + (4 - (sg & 1)) * band_plane(a.g.n);
  double dt;
  if (a.rk == 2) {
    dt = st == 0 ? a.dtb / 2.0 : a.dtb;      // barotr.py:50-56
    io.beta = T(0.0);
  } else {
    dt = st == 0 ? a.dtb / 3.0 : (st == 1 ? a.dtb / 2.0 : a.dtb);  // barotr.py:73-83
    io.beta = T(1.0);
  }
  io.dt = (T)dt;
  io.stored_halo = (first && st == 0) ? 1 : 0;
  io.last = last ? 1 : 0;
  return io;
}

// ---------------------------------------------------------------------------
// Materialised halos (end of a round) and diagnostics
// ---------------------------------------------------------------------------
// Write every halo cell of face-major field(s) from their own interior.
template <typename T>
__device__ void fill_halo_cell(const Geo<T>& g, T* H, T* U, T* V, int k) {
  const int f = k / g.nh, id = k - f * g.nh;
  const int m = g.m, n = g.n;
  int i, j;
  if (id < 3 * m) {
    i = id / m;
    j = id - i * m;
  } else if (id < 6 * m) {
    i = m - kHalo + (id - 3 * m) / m;
    j = (id - 3 * m) % m;
  } else if (id < 6 * m + 3 * n) {
    i = kHalo + (id - 6 * m) / 3;
    j = (id - 6 * m) % 3;
  } else {
    i = kHalo + (id - 6 * m - 3 * n) / 3;
    j = m - kHalo + (id - 6 * m - 3 * n) % 3;
  }
  const long o = cell(f, i, j, m);
  if (H) H[o] = fetch_s(H, g, f, i, j, 0);
  if (U) {
    T u, v;
    fetch_v(U, V, g, f, i, j, 0, u, v);
    U[o] = u;
    V[o] = v;
  }
}

template <typename T>
struct DiagOut {
  T* cx;
  T* cy;
  T* uct;
  T* vct;
  T* ucx;
  T* ucy;
  T* vcx;
  T* vcy;
  T* advx;
  T* advy;
};

// C-grid quantities at x face i (y face when y = 1) of column j (row i) with
// the reference's full-array pad semantics; the inputs have materialised halos.
template <typename T>
struct FaceQ {
  T bc, vis, tang;
};

template <typename T>
__device__ FaceQ<T> face_full(const Geo<T>& g, const T* H, const T* U, const T* V, int f, int i, int j,
                              int y) {
  FaceQ<T> r{T(0.0), T(0.0), T(0.0)};
  const int m = g.m;
  const int fidx = y ? j : i;
  if (fidx < kHalo || fidx > m - kHalo) return r;
  T ph[6], pc[6], pt[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const int ii = y ? i : i - kHalo + q, jj = y ? j - kHalo + q : j;
    const long o = cell(f, ii, jj, m);
    ph[q] = H[o];
    pc[q] = contra(g, o, U[o], V[o], y);
    pt[q] = y ? U[o] : V[o];
  }
  T bc = T(0.5) * (rplus(pc, 1) + rminus(pc + 1, 1));
  const int other = y ? i : j;
  const int side = y ? yface_side(j, m) : xface_side(i, m);
  if (side >= 0 && other >= kHalo && other < m - kHalo)
    bc = (bc + nb_normal_raw(g, U, V, 1, f, side, other - kHalo)) / T(2.0);
  r.bc = bc;
  r.tang = bc > T(0.0) ? rplus(pt, 1) : rminus(pt + 1, 1);
  const long o = cell(f, i, j, m);
  const T dz = y ? g.dzph_y[o] : g.dzph_x[o];
  const bool valid_mid = other >= kHalo && other <= m - kHalo;  // Poly.scalar_* core range
  const T c = celerity(valid_mid ? mid6(ph, 1) : T(0.0), dz);
  r.vis = bc + (T(4.9) / c) * (rplus(ph, 1) - rminus(ph + 1, 1));
  return r;
}

template <typename T>
__device__ T kin_full(const Geo<T>& g, const T* H, const T* U, const T* V, int f, int i, int j, int y) {
  FaceQ<T> q = face_full(g, H, U, V, f, i, j, y);
  return T(0.5) * (q.vis * q.vis + q.tang * q.tang);
}

template <typename T>
__device__ T vort_full(const Geo<T>& g, const T* H, const T* U, const T* V, int f, int i, int j) {
  const int m = g.m;
  if (i > m - 2 || j > m - 2) return T(0.0);
  const long o = cell(f, i, j, m);
  const T uy0 = face_full(g, H, U, V, f, i, j, 1).tang, uy1 = face_full(g, H, U, V, f, i, j + 1, 1).tang;
  const T vx0 = face_full(g, H, U, V, f, i, j, 0).tang, vx1 = face_full(g, H, U, V, f, i + 1, j, 0).tang;
  return g.rda[o] * (uy0 * g.d_dx[o] + vx1 * g.c_dy[o + m] - uy1 * g.d_dx[o + 1] - vx0 * g.c_dy[o]);
}

// The ten diagnostic state fields of the last stage (barotr_pure.py:158-168)
// at cell (f, i, j), over the whole padded array.
template <typename T>
__device__ void diag_cell(const Geo<T>& g, const T* H, const T* U, const T* V, const DiagOut<T>& d, int f,
                          int i, int j) {
  const int m = g.m;
  const long o = cell(f, i, j, m);
  const bool mid_ok = i >= kHalo && i <= m - kHalo && j >= kHalo && j <= m - kHalo;
  T hx = T(0.0), hy = T(0.0);
  if (mid_ok) {
    T px[6], py[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      px[q] = H[cell(f, i - kHalo + q, j, m)];
      py[q] = H[cell(f, i, j - kHalo + q, m)];
    }
    hx = mid6(px, 1);
    hy = mid6(py, 1);
  }
  d.cx[o] = celerity(hx, g.dzph_x[o]);
  d.cy[o] = celerity(hy, g.dzph_y[o]);
  const T uct = contra(g, o, U[o], V[o], 0), vct = contra(g, o, U[o], V[o], 1);
  d.uct[o] = uct;
  d.vct[o] = vct;
  const FaceQ<T> xq = face_full(g, H, U, V, f, i, j, 0);
  const FaceQ<T> yq = face_full(g, H, U, V, f, i, j, 1);
  d.ucx[o] = xq.vis;
  d.vcx[o] = xq.tang;
  d.vcy[o] = yq.vis;
  d.ucy[o] = yq.tang;
  const T vort = vort_full(g, H, U, V, f, i, j);
  if (i <= m - 2) {
    const T k0 = T(0.5) * (xq.vis * xq.vis + xq.tang * xq.tang);
    d.advx[o] = vort * vct - (kin_full(g, H, U, V, f, i + 1, j, 0) - k0) * g.rdx[o];
  } else {
    d.advx[o] = T(0.0);
  }
  if (j <= m - 2) {
    const T k0 = T(0.5) * (yq.vis * yq.vis + yq.tang * yq.tang);
    d.advy[o] = -vort * uct - (kin_full(g, H, U, V, f, i, j + 1, 1) - k0) * g.rdy[o];
  } else {
    d.advy[o] = T(0.0);
  }
}

}  // namespace bt
