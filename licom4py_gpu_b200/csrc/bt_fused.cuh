// bt_fused.cuh - the fused stage kernel: phase UV of one RK stage and phase H of
// the next in one launch.
//
// A stage's two phases meet at global dependencies (the new h, then the new
// velocity, of neighbouring tiles), so the phase kernels need two launches per
// stage.  At one-wave sizes each launch costs about 0.8 us besides its own
// load latency.  The velocity, however, is pointwise in what earlier launches
// have written -- the base, the momentum terms and the 13-point cross of h --
// so a tile can form it itself wherever phase H reads it: on its own region and
// on the three lines of the neighbouring face behind each face edge it
// touches.  k_stage does that: it
//
//   1. loads h on the tile and 6 cells around it (the crosses of the region's
//      points) and, behind a touched face edge, on a patch of the neighbouring
//      face: 3 lines in its halo, 6 inside; halo cells come from the h bands;
//   2. forms the velocity of every region point inside the face and of the
//      neighbour's three lines ("evaluations", one per thread);
//   3. interpolates the region's halo points and the halo points of the
//      neighbour's lines from those;
//   4. runs phase H's faces and cells.
//
// One global dependency per stage is left.  A round of S stages is phase H of
// the first, S - 1 fused kernels, and phase UV of the last (RK3 runs the first
// stage's two phases apart: its blend reads the round's stored halo cells); only the velocity of
// a substep's start is stored (the base of its stages).  What the phases updated
// in place is double-buffered: terms and base velocity alternate between two
// buffers, the h bands between three, because neighbouring tiles read them
// while this tile writes.
//
// Which points, evaluations and interpolations a thread does depends on the tile
// alone, so that decoding -- some 300 instructions per thread, which at C96 no
// earlier kernel's tail would hide, the SMs being full -- is done once per plan
// (k_stage_tables) and the kernel reads the result: 12 packed ints and two
// weights per thread, of which tiles away from the face edges need four ints.
//
// The arithmetic of each value is the phase kernels' own, so the results are
// bitwise the same.

#pragma once

#include "bt_stencil.cuh"

namespace bt {

// Pointers of one fused kernel: ``io`` are those of the stage whose phase H runs
// (u, v, up, vp, u_out, v_out and band_uv unused), the others finish the stage before it.
template <typename T>
struct FusedIO {
  StageIO<T> io;
  const T* h_prev;       // that stage's input h and its bands (fb blend, beta != 0)
  const T* band_hprev;
  const T* terms_prev;   // its momentum terms
  const T* u_base;       // its base velocity
  const T* v_base;
  T* u_keep;             // where the velocity it gives is kept (nullptr: nowhere)
  T* v_keep;
  T dt_prev, beta_prev;
};

template <int TI, int TJ>
struct FusedShape {
  using S = TileShape<TI, TJ>;
  static constexpr int kT = S::kT;
  static constexpr int PW = TJ + 12, HR = TI + 12;  // own h: rows i0 - 6 .., columns j0 - 6 ..
  static constexpr int XA = TJ + 12, XB = TI + 12;  // h patch behind an S/N and a W/E edge: 9 lines each
  static constexpr int OA = TJ + 6, OB = TI + 6;    // evaluated lines, 3 each
  static constexpr int NH = HR * PW + 9 * (XA + XB);
  static constexpr int kJobs = 6 * (TI + TJ), kJobWords = 10;
  // halo points of h and patch points beside the evaluated ones: one per thread
  static constexpr int kHaloA = 3 * S::RJ, kPatchA = 3 * (TJ + 3), kHaloB = 3 * S::RI, kPatchB = 3 * (TI + 3);
  static_assert(kHaloA + kPatchA + kHaloB + kPatchB + 36 <= kT, "one halo point per thread");
  // evaluations of an interior, S/N-edge, W/E-edge and corner tile: one per thread
  static_assert(S::NP <= kT && (TI + 3) * TJ + 6 * TI + 3 * TJ + 6 <= kT &&
                    S::VB + 6 * TI + 6 <= kT && (TI + 3) * TJ + 3 * TI + 3 * TJ + 3 * TI + 12 <= kT,
                "one evaluation per thread");
  static_assert(kJobs <= kT && S::C <= kT, "one pass");
  static constexpr int NE = 2 * S::EW;  // line slots: patch A, patch B
  // evaluation constants per thread: pairs gct, c2l (4), then rdx, rdy, sina
  static constexpr int kEvalWords = 11 * kT;
  static constexpr int kFaces = 4 * (S::FXP + S::FYP);
  // shared memory (words): h_s, contravariant and raw velocities, evaluation constants (the face
  // results share their memory: evaluated by then), interpolation constants, constant block, lines,
  // evaluated lon/lat velocity of the patches and of our own lines, and last the blend's h of the
  // stage before, for beta != 0 only
  static constexpr int kH = 0, kUC = up4(NH), kVC = up4(kUC + S::VB), kV = up4(kVC + TI * S::RJ), kU = up4(kV + S::VB),
                       kEC = up4(kU + TI * S::RJ), kFX = kEC, kFY = kFX + 4 * S::FXP,
                       kJ = up4(kEC + (kEvalWords > kFaces ? kEvalWords : kFaces)), kC = up4(kJ + kJobs * kJobWords),
                       kNP = up4(kC + S::cW), kNH = kNP + 6 * NE, kNDZ = kNH + 6 * NE, kPU = up4(kNDZ + NE),
                       kOU = kPU + 6 * (OA + OB), kHP = up4(kOU + 6 * (OA + OB)), kWords = kHP + up4(NH);
};

// The arrays phase H's faces and cells read (as LayoutH).
template <typename T, int TI, int TJ>
struct LayoutF {
  using S = TileShape<TI, TJ>;
  using F = FusedShape<TI, TJ>;
  static constexpr int kSlotS = 0, kSlotN = 0, kSlotW = S::EW, kSlotE = S::EW;  // lines of an S, N, W, E edge
  T *s_uc, *s_vc, *s_v, *s_u, *s_fx, *s_fy, *s_cell, *s_cdy, *s_ddx, *s_dzx, *s_dzy, *s_np, *s_nh, *s_ndz;
  __device__ __forceinline__ explicit LayoutF(T* sm) {
    s_uc = sm + F::kUC;
    s_vc = sm + F::kVC;
    s_v = sm + F::kV;
    s_u = sm + F::kU;
    s_fx = sm + F::kFX;
    s_fy = sm + F::kFY;
    s_cell = sm + F::kC;
    s_cdy = s_cell + S::bCDY;
    s_ddx = s_cell + S::bDDX;
    s_dzx = s_cell + S::bDZX;
    s_dzy = s_cell + S::bDZY;
    s_np = sm + F::kNP;
    s_nh = sm + F::kNH;
    s_ndz = sm + F::kNDZ;
  }
};

// What lies behind a face edge the tile touches: positions k0..k1 along our
// side; the neighbour nb, its side ns, whether its positions run the other way.
struct EdgePatch {
  int side, nb, ns, k0, k1;
  bool rev;
  __device__ __forceinline__ void set(int s, int route, int first, int count) {
    side = s;
    nb = route_nb(route);
    ns = route_side(route);
    rev = route_rev(route) != 0;
    k0 = first;
    k1 = first + count - 1;
  }
  // Positions of the neighbour's line d (0..2 cells from the edge) that the tile
  // needs: its own and the sources of its halo points, which lie at most d + 1
  // positions towards the middle of the edge (bt_plan checks the tables).
  __device__ __forceinline__ int lo(int d, int n) const {
    const int h = (n + 1) / 2;
    return k1 >= h ? min(k0, max(k0, h) - 1 - d) : k0;
  }
  __device__ __forceinline__ int hi(int d, int n) const {
    const int h = (n + 1) / 2;
    return k0 < h ? max(k1, min(k1, h - 1) + 1 + d) : k1;
  }
  // cell of the neighbour at distance dd from the edge (negative: in its halo), our position pos
  __device__ __forceinline__ void cell_at(int dd, int pos, int n, int& i, int& j) const {
    const int kk = kHalo + (rev ? n - 1 - pos : pos), in = kHalo + dd, out = n + kHalo - 1 - dd;
    i = ns == kS ? in : ns == kN ? out : kk;
    j = ns == kW ? in : ns == kE ? out : kk;
  }
};

// Line number (0..2, increasing i or j) of the halo cells d + 1 outside side s.
__device__ __forceinline__ int outer_line(int s, int d) { return s == kS || s == kW ? 2 - d : d; }

// A thread's decoded work (three int4 per thread, planes of S::kT):
//   0: evaluation: cell offset, position in a terms plane, pack_eval, destination
//      (region point: row | column << 8; patch: lon/lat word | (line slot + 1) << 9 | y << 20)
//   1: halo point of h: cell offset, or band number for an interpolated one; its
//      shared word | kind << 12 (0 none, 1 read, 2 / 3 interpolated, second source
//      after / before the first); directly read patch point: cell offset, shared word (-1: none)
//   2: interpolation: pack_job, cell offset, weight number; depth of a line:
//      cell offset | slot << 24, -1: none
struct StageRec {
  static constexpr int kInts = 12;
  // type 0 none, 1 region point, 2 patch; at: word of the cell's h; si, sj: steps of i and j
  __device__ __forceinline__ static int pack_eval(int type, int at, int si, int sj) {
    return type | (at << 2) | ((si + 64) << 14) | ((sj + 64) << 21);
  }
  // dst 1: uc and v, 2: vc and u, 3: a line; src: word past the patches' lon/lat velocity
  __device__ __forceinline__ static int pack_job(int dst, int src, int step, int at, int y) {
    return dst | (src << 2) | ((step < 0 ? 1 : 0) << 14) | (at << 15) | (y << 30);
  }
};

// Builds the tables of the fused kernel: one CTA per tile.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(TileShape<TI, TJ>::kT) k_stage_tables(Geo<T> g, Tiling t, int4* rec, T* weights) {
  using S = TileShape<TI, TJ>;
  using F = FusedShape<TI, TJ>;
  constexpr int RJ = S::RJ, PW = F::PW;
  const int tid = threadIdx.x, n = g.n, m = g.m;
  const TileBox b = tile_box(t, n, blockIdx.x);
  const int f = b.f, ni = b.ni, nj = b.nj;
  EdgeCnt cnt;
  const int P = edge_count(b, m, g.route, cnt);
  // the tile touches at most one of S / N (patch A) and one of W / E (patch B)
  const int sa = cnt.s ? kS : cnt.n ? kN : -1, sb = cnt.w ? kW : cnt.e ? kE : -1;
  EdgePatch pa, pb;
  pa.set(sa, g.route[f * 4 + max(sa, 0)], b.j0 - kHalo, nj);
  pb.set(sb, g.route[f * 4 + max(sb, 0)], b.i0 - kHalo, ni);
  constexpr int kPA = F::HR * PW, kPB = kPA + 9 * F::XA;  // the patches' h after the tile's own

  // the thread's halo (or patch side) point of h
  int hdst = -1, ho = 0, hb = 0;
  bool hlerp = false;
  int hd = 1;
  T w0 = T(0.0), w1 = T(0.0);
  if (P > 0) {
    int q = tid, hf = f, i = 0, j = 0, dst = -1;
    if (q < F::kHaloA) {
      const int d = q / RJ, c = q - d * RJ;
      if (sa >= 0 && c < nj + 6) {
        const int r = sa == kS ? d : ni + kHalo + d;
        i = b.i0 - kHalo + r;
        j = b.j0 - kHalo + c;
        dst = (r + 3) * PW + c + 3;
      }
    } else if ((q -= F::kHaloA) < F::kHaloB) {
      const int r = q / 3, d = q - 3 * r;
      if (sb >= 0 && r < ni + 6) {
        const int c = sb == kW ? d : nj + kHalo + d;
        i = b.i0 - kHalo + r;
        j = b.j0 - kHalo + c;
        dst = (r + 3) * PW + c + 3;
      }
    } else {
      q -= F::kHaloB;
      const bool isa = q < F::kPatchA + 18;
      if (!isa) q -= F::kPatchA + 18;
      const EdgePatch e = isa ? pa : pb;
      const int w = isa ? TJ + 3 : TI + 3, lo = e.lo(2, n), hi = e.hi(2, n);
      int dd, pos;
      bool on = e.side >= 0 && q < 3 * w + 18;
      if (q < 3 * w) {  // the neighbour's halo lines
        const int l = isa ? q / (TJ + 3) : q / (TI + 3);
        dd = -1 - l;
        pos = lo + q - l * w;
        on = on && pos <= hi;
      } else {  // three positions beyond each end of its three evaluated lines
        q -= 3 * w;
        dd = q / 6;
        const int s = q - 6 * dd;
        pos = s < 3 ? lo - 3 + s : hi - 2 + s;
      }
      if (on) {
        hf = e.nb;
        e.cell_at(dd, pos, n, i, j);
        dst = (isa ? kPA + (dd + 3) * F::XA : kPB + (dd + 3) * F::XB) + pos - e.k0 + 6;
      }
    }
    if (dst >= 0) {
      const bool oi = i < kHalo || i >= m - kHalo, oj = j < kHalo || j >= m - kHalo;
      if (!(oi && oj)) {
        hdst = dst;
        ho = cell32(hf, i, j, m);
        if (oi || oj) {
          const PointKind pk(i, j, m);
          hlerp = true;
          HaloRef<T> ref;
          ref.load(g, hf, pk.side, pk.c, pk.k);
          hb = ref.b0;
          hd = ref.d;
          w0 = ref.w0;
          w1 = ref.w1;
        }
      }
    }
  }

  // the thread's directly read patch point: lines 0..5 cells inside the neighbour
  int pdst = -1, po = 0;
  {
    int q = tid;
    const bool isa = q < 6 * (TJ + 3);
    if (!isa) q -= 6 * (TJ + 3);
    const EdgePatch e = isa ? pa : pb;
    const int w = isa ? TJ + 3 : TI + 3;
    if (e.side >= 0 && q < 6 * w) {
      const int dd = q / w, pos = e.lo(2, n) + q - dd * w;
      if (pos <= e.hi(2, n)) {
        int i, j;
        e.cell_at(dd, pos, n, i, j);
        po = cell32(e.nb, i, j, m);
        pdst = (isa ? kPA + (dd + 3) * F::XA : kPB + (dd + 3) * F::XB) + pos - e.k0 + 6;
      }
    }
  }

  // the thread's evaluation: a region point inside the face (ev = 1: region row er, column ec) or
  // cell (er from the edge, position ec) of a patch (ev = 2: A, 3: B)
  int ev = 0, er = 0, ec = 0, eo = 0, et = 0;
  {
    const int rlo = sa == kS ? kHalo : 0, nr = ni + 6 - (sa >= 0 ? kHalo : 0);
    const int nc = sb >= 0 ? 3 : 6;
    int q = tid;
    if (q < nr * TJ) {
      er = rlo + q / TJ;
      ec = q % TJ + kHalo;
      if (ec < nj + kHalo) ev = 1;
    } else if ((q -= nr * TJ) < ni * nc) {
      const int a = nc == 6 ? q / 6 : q / 3, d = q - a * nc;
      er = a + kHalo;
      ec = (sb == kW || (nc == 6 && d >= 3)) ? nj + kHalo + (nc == 6 ? d - 3 : d) : d;
      ev = 1;
    } else {
      q -= ni * nc;
      if (sa >= 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int w = pa.hi(d, n) - pa.lo(d, n) + 1;
          if (ev == 0 && q >= 0 && q < w) {
            ev = 2;
            er = d;
            ec = pa.lo(d, n) + q;
          }
          q -= w;
        }
      }
      if (sb >= 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int w = pb.hi(d, n) - pb.lo(d, n) + 1;
          if (ev == 0 && q >= 0 && q < w) {
            ev = 3;
            er = d;
            ec = pb.lo(d, n) + q;
          }
          q -= w;
        }
      }
    }
    if (ev) {
      int i, j, ef = f;
      if (ev == 1) {
        i = b.i0 - kHalo + er;
        j = b.j0 - kHalo + ec;
      } else {
        const EdgePatch e = ev == 2 ? pa : pb;
        e.cell_at(er, ec, n, i, j);
        ef = e.nb;
      }
      eo = cell32(ef, i, j, m);
      et = (ef * n + i - kHalo) * n + j - kHalo;
    }
  }

  // h position and the steps of its face's i and j; where the result goes
  int pack1 = 0, pack2 = 0;
  if (ev == 1) {
    pack1 = StageRec::pack_eval(1, (er + 3) * PW + ec + 3, PW, 1);
    pack2 = er | (ec << 8);
  } else if (ev) {
    const EdgePatch e = ev == 2 ? pa : pb;
    const int X = ev == 2 ? F::XA : F::XB;
    const int along = e.rev ? -1 : 1, in = e.ns == kS || e.ns == kW ? X : -X;
    const bool i_in = e.ns == kS || e.ns == kN;  // the neighbour's i runs away from the edge
    pack1 = StageRec::pack_eval(2, (ev == 2 ? kPA : kPB) + (er + 3) * X + ec - e.k0 + 6, i_in ? in : along,
                                i_in ? along : in);
    const int x = (ev == 2 ? er * F::OA : 3 * F::OA + er * F::OB) + ec - e.k0 + 3;
    int slot = 0;  // the line's inside point, + 1
    if (ec >= e.k0 && ec <= e.k1)
      slot = 1 + ((ev == 2 ? 0 : S::EW) + ec - e.k0) * 6 + (e.ns == kS || e.ns == kW ? 3 + er : 2 - er);
    pack2 = x | (slot << 9) | ((e.ns == kE || e.ns == kW ? 1 : 0) << 20);
  }

  // the thread's interpolation: halo point of the region (jb = 1) or of a neighbour's line (jb = 2),
  // jd cells outside
  int jb = 0, jd = 0, jx = 0, jstep = 1, jdst = 0, jside = 0, jo = 0, jw = 0, jy = 0, jz = -1, jslot = 0;
  if (tid < 6 * P) {
    jb = tid < 3 * P ? 1 : 2;
    const int q = jb == 1 ? tid : tid - 3 * P;
    jd = div24(q, P);
    const EdgeItem e = edge_item(b, cnt, q - jd * P);
    const EdgePatch pt = e.kind < 2 ? pa : pb;
    const int hf = jb == 1 ? f : pt.nb, side = jb == 1 ? e.side : pt.ns, c = outer_line(side, jd);
    const int k = jb == 1 ? e.k : (pt.rev ? n - 1 - e.k : e.k);
    jside = e.kind;
    // sources, as positions along our edge
    const int b0 = g.bsrc[band_no(hf, side, c, k, n)];
    if (jb == 1) {
      const int pos = b0 - band_no(pt.nb, pt.ns, c, 0, n);
      jx = pt.rev ? n - 1 - pos : pos;
      jstep = 1;
      const int r = e.kind < 2 ? (e.side == kS ? c : ni + kHalo + c) : e.pos + kHalo;
      const int cc = e.kind < 2 ? e.pos + kHalo : (e.side == kW ? c : nj + kHalo + c);
      jdst = e.kind < 2 ? r * TJ + cc - kHalo : (r - kHalo) * RJ + cc;
    } else {
      jx = b0 - band_no(f, e.side, c, 0, n);
      jstep = route_rev(g.route[hf * 4 + side]) ? -1 : 1;
      jdst = ((e.kind < 2 ? 0 : S::EW) + e.pos) * 6 + (side == kS || side == kW ? 2 - jd : 3 + jd);
    }
    jx -= pt.k0 - 3;
    const int i = side == kS ? c : side == kN ? m - kHalo + c : k + kHalo;
    const int j = side == kW ? c : side == kE ? m - kHalo + c : k + kHalo;
    const int o = cell32(hf, i, j, m);
    jo = o;
    jw = hf * g.nh + HaloRef<T>::halo_word(g, side, c, k);
    jy = side == kE || side == kW ? 1 : 0;
    if (jb == 2 && jd == 0) {  // depth at the edge face: the line's fourth point
      int di, dj;
      edge_point(side, k, 3, m, di, dj);
      jz = cell32(hf, di, dj, m);
      jslot = (e.kind < 2 ? 0 : S::EW) + e.pos;
    }
  }
  int jpack = 0;
  if (jb) {
    const int src = (jb == 1 ? F::kPU : F::kOU) + (jside < 2 ? jd * F::OA : 3 * F::OA + jd * F::OB) + jx - F::kPU;
    jpack = StageRec::pack_job(jb == 2 ? 3 : jside < 2 ? 1 : 2, src, jstep, jdst, jy);
  }

  int4* const r = rec + (long)b.idx * 3 * S::kT + tid;
  r[0] = make_int4(ev ? eo : 0, et, pack1, pack2);
  r[S::kT] = make_int4(hlerp ? hb : ho, hdst < 0 ? 0 : hdst | ((hlerp ? (hd < 0 ? 3 : 2) : 1) << 12), po, pdst);
  r[2 * S::kT] = make_int4(jpack, jo, jw, jz < 0 ? -1 : jz | (jslot << 24));
  T* const w = weights + ((long)b.idx * S::kT + tid) * 2;
  w[0] = w0;
  w[1] = w1;
}

// One RK stage's phase UV and the next one's phase H (file comment).  Bound by
// latency while a tile has an SM to itself (the loads' round trip, four barriers,
// the evaluation and face chains: 5000-6600 cycles from the wait on at C48 of
// float64), by issue slots and the shared-memory pipe with two 12 x 16 tiles per
// SM, and there by the SMs that hold two edge tiles.  us per substep, two phase
// kernels per stage / fused: C48 float64 12.3 / 8.8, float32 9.3 / 6.0; C96
// float64 14.2 / 13.2, float32 11.0 / 8.2; C90 RK3 float32 18.0 / 14.3.
template <typename T, int TI, int TJ>
__global__ void __launch_bounds__(TileShape<TI, TJ>::kT, TI == 8 ? 3 : 2)
    k_stage(Geo<T> g, FusedIO<T> p, Tiling t, const int4* rec, const T* weights) {
  using S = TileShape<TI, TJ>;
  using F = FusedShape<TI, TJ>;
  constexpr int RJ = S::RJ, PW = F::PW;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* const sm = reinterpret_cast<T*>(smraw);
  const LayoutF<T, TI, TJ> L(sm);
  const StageIO<T>& io = p.io;
  const int tid = threadIdx.x, n = g.n, m = g.m;
  const TileBox b = tile_box(t, n, blockIdx.x);
  const int f = b.f, ni = b.ni, nj = b.nj, o0 = cell32(f, b.i0, b.j0, m);
  const bool blend = p.beta_prev != T(0.0);

  // ---- ahead of the previous kernel: the thread's work and constants -------------
  const int4* const r = rec + (long)b.idx * 3 * S::kT + tid;
  const int4 re = __ldg(r);
  EdgeCnt cnt;
  const int P = edge_count(b, m, g.route, cnt);
  // only tiles at a face edge have halo points, patches and lines: the others need a quarter of the record
  int4 rj = make_int4(0, 0, 0, -1), rh = make_int4(0, 0, 0, -1);
  T w0 = T(0.0), w1 = T(0.0);
  if (P > 0) {
    rj = __ldg(r + 2 * S::kT);
    rh = __ldg(r + S::kT);
    ld_pair(weights + ((long)b.idx * S::kT + tid) * 2, w0, w1);
  }
  tile_consts<T, TI, TJ>(g, b, L);
  const int ev = re.z & 3, eo = re.x;
  T* const s_ec = sm + F::kEC;
  if (ev) {
    cp_async_pairs<2>(s_ec + 2 * tid, g.gct + 4 * (long)eo);
    cp_async_pairs<2>(s_ec + 2 * (tid + S::kT), g.gct + 4 * (long)eo + 2);
    if (P > 0) {
      cp_async_pairs<2>(s_ec + 2 * (tid + 2 * S::kT), g.c2l + 4 * (long)eo);
      cp_async_pairs<2>(s_ec + 2 * (tid + 3 * S::kT), g.c2l + 4 * (long)eo + 2);
    }
    cp_async_t(s_ec + 8 * S::kT + tid, g.rdx + eo);
    cp_async_t(s_ec + 9 * S::kT + tid, g.rdy + eo);
    cp_async_t(s_ec + 10 * S::kT + tid, g.sina + eo);
  }
  const int jb = rj.x & 3;
  if (jb) {
    const int o = rj.y;
    T* const s = sm + F::kJ + tid * F::kJobWords;
    cp_async_pairs<4>(s, g.l2c + 4 * (long)o);
    cp_async_pairs<2>(s + 4, g.gct + 4 * (long)o + ((rj.x >> 30) & 1 ? 2 : 0));
    cp_async_pairs<2>(s + 6, g.hw + 2 * (long)rj.z);
    cp_async_t(s + 8, g.sina + o);
    if (io.last && rj.w >= 0)
      cp_async_t(L.s_ndz + (rj.w >> 24), ((rj.x >> 30) & 1 ? g.dzph_y : g.dzph_x) + (rj.w & 0xffffff));
  }

  wait_prior_grid();
  // Only now may the next kernel start: at small sizes it would otherwise start at once, and so would the ones
  // after it as long as SMs have room, and the CTAs of the running kernel would share SMs while others idle
  // (C48 float64, before launches were spread evenly: 14.67 us per substep with the release at the top, 8.79 here).
  release_dependents();

  // ---- 1. h, and what the evaluations read -------------------------------------
#pragma unroll
  for (int k = 0; k < F::HR * PW; k += S::kT) {
    const int q = k + tid, row = q / PW, col = q - row * PW, i = b.i0 - 6 + row, j = b.j0 - 6 + col;
    if (q < F::HR * PW && row < ni + 12 && col < nj + 12 && is_interior(i, j, m)) {
      const int o = cell32(f, i, j, m);
      cp_async_t(sm + F::kH + q, io.h + o);
      if (blend) cp_async_t(sm + F::kHP + q, p.h_prev + o);
    }
  }
  if (rh.w >= 0) {
    cp_async_t(sm + F::kH + rh.w, io.h + rh.z);
    if (blend) cp_async_t(sm + F::kHP + rh.w, p.h_prev + rh.z);
  }
  T upc, vpc, tm[kTerms<T>];
  if (ev) {
    upc = p.u_base[eo];
    vpc = p.v_base[eo];
#pragma unroll
    for (int z = 0; z < kTerms<T>; ++z) tm[z] = p.terms_prev[z * (6 * n * n) + re.y];
  }
  T hpc = T(0.0);
  if (tid < S::C && tid / TJ < ni && tid % TJ < nj) hpc = io.hp[o0 + tid / TJ * m + tid % TJ];
  const int hk = rh.y >> 12;
  if (hk) {
    const int at = rh.y & 0xfff, e2 = rh.x + (hk == 2 ? 1 : -1);
    sm[F::kH + at] = hk == 1 ? io.h[rh.x] : lin2(w0, io.band_h[rh.x], w1, io.band_h[e2]);
    if (blend) sm[F::kHP + at] = hk == 1 ? p.h_prev[rh.x] : lin2(w0, p.band_hprev[rh.x], w1, p.band_hprev[e2]);
  }
  cp_async_wait_all();
  __syncthreads();

  // ---- 2. evaluations: the velocity the stage before gives -----------------------
  if (ev) {
    const int at = (re.z >> 2) & 0xfff, si = ((re.z >> 14) & 127) - 64, sj = ((re.z >> 21) & 127) - 64;
    T hx[7], hy[7];
    const T* const H = sm + F::kH + at;
#pragma unroll
    for (int z = 0; z < 7; ++z) {
      hx[z] = H[(z - 3) * si];
      hy[z] = H[(z - 3) * sj];
    }
    if (blend) {  // fb_scheme, barotr_pure.py:52-54
      const T* const B = sm + F::kHP + at;
#pragma unroll
      for (int z = 0; z < 7; ++z) {
        hx[z] = lin2(T(1.0) - p.beta_prev, hx[z], p.beta_prev, B[(z - 3) * si]);
        hy[z] = lin2(T(1.0) - p.beta_prev, hy[z], p.beta_prev, B[(z - 3) * sj]);
      }
    }
    const T gx = gradient(s_ec[8 * S::kT + tid], hx), gy = gradient(s_ec[9 * S::kT + tid], hy);
    const T u = momentum<T, false>(upc, gx, tm, p.dt_prev);
    const T v = momentum<T, true>(vpc, gy, tm, p.dt_prev);
    T G[4];
    ld_pair(s_ec + 2 * tid, G[0], G[1]);
    ld_pair(s_ec + 2 * (tid + S::kT), G[2], G[3]);
    const T sn = s_ec[10 * S::kT + tid];
    const T uct = lin2(G[0], u, G[1], v) * sn, vct = lin2(G[2], u, G[3], v) * sn;  // remap.py:34-39
    T ull = T(0.0), vll = T(0.0);
    if (P > 0) {  // cube.py:137-145
      T c2[4];
      ld_pair(s_ec + 2 * (tid + 2 * S::kT), c2[0], c2[1]);
      ld_pair(s_ec + 2 * (tid + 3 * S::kT), c2[2], c2[3]);
      ull = lin2(c2[0], u, c2[1], v);
      vll = lin2(c2[2], u, c2[3], v);
    }
    constexpr int WA = 3 * F::OA, WP = 3 * (F::OA + F::OB);  // words of patch A, of both
    if (ev == 1) {
      const int er = re.w & 0xff, ec = re.w >> 8;
      const bool row = er >= kHalo && er < ni + kHalo, col = ec >= kHalo && ec < nj + kHalo;
      if (col) {
        L.s_uc[er * TJ + ec - kHalo] = uct;
        L.s_v[er * TJ + ec - kHalo] = v;
      }
      if (row) {
        L.s_vc[(er - kHalo) * RJ + ec] = vct;
        L.s_u[(er - kHalo) * RJ + ec] = u;
      }
      if (row && col && p.u_keep) {
        p.u_keep[eo] = u;
        p.v_keep[eo] = v;
      }
      if (P > 0) {  // our own three lines: the sources of the neighbours' halo points
        const int da = cnt.s ? er - kHalo : ni + kHalo - 1 - er, db = cnt.w ? ec - kHalo : nj + kHalo - 1 - ec;
        T* const s_ou = sm + F::kOU;
        if (cnt.s + cnt.n > 0 && da >= 0 && da < 3) {
          s_ou[da * F::OA + ec] = ull;
          s_ou[WP + da * F::OA + ec] = vll;
        }
        if (cnt.w + cnt.e > 0 && db >= 0 && db < 3) {
          s_ou[WA + db * F::OB + er] = ull;
          s_ou[WP + WA + db * F::OB + er] = vll;
        }
      }
    } else {
      const int x = re.w & 0x1ff, slot = ((re.w >> 9) & 0x7ff) - 1;
      sm[F::kPU + x] = ull;
      sm[F::kPU + WP + x] = vll;
      if (slot >= 0) L.s_np[slot] = re.w >> 20 ? vct : uct;
    }
  }
  __syncthreads();

  // ---- 3. halo points of the region and of the neighbours' lines ------------------
  if (P > 0) {
    if (jb) {
      constexpr int WP = 3 * (F::OA + F::OB);
      const T* const s = sm + F::kJ + tid * F::kJobWords;
      const T* const src = sm + F::kPU + ((rj.x >> 2) & 0xfff);
      const int step = (rj.x >> 14) & 1 ? -1 : 1, at = (rj.x >> 15) & 0x7fff;
      const T ull = lin2(s[6], src[0], s[7], src[step]), vll = lin2(s[6], src[WP], s[7], src[WP + step]);
      const T u = lin2(s[0], ull, s[1], vll), v = lin2(s[2], ull, s[3], vll);  // cube.py:137-153
      const T ct = lin2(s[4], u, s[5], v) * s[8];
      if (jb == 3) {
        L.s_np[at] = ct;
      } else if (jb == 1) {
        L.s_uc[at] = ct;
        L.s_v[at] = v;
      } else {
        L.s_vc[at] = ct;
        L.s_u[at] = u;
      }
    }
    __syncthreads();
    if (io.last) {  // the neighbour's side of the edge faces' mass flux (edge_lines)
      if (tid < P) {
        const EdgeItem e = edge_item(b, cnt, tid);
        const int X = e.kind < 2 ? F::XA : F::XB, slot = (e.kind < 2 ? 0 : S::EW) + e.pos;
        const int ns = route_side((cnt.routes >> (8 * e.kind)) & 0xff);
        const bool low = ns == kS || ns == kW;
        const T* const h0 = sm + F::kH + (e.kind < 2 ? F::HR * PW : F::HR * PW + 9 * F::XA) + (low ? 0 : 5 * X) + e.pos + 6;
        T hh[6];
#pragma unroll
        for (int z = 0; z < 6; ++z) hh[z] = h0[low ? z * X : -z * X];
        T* const np = L.s_np + 6 * slot;
        T* const nh = L.s_nh + 6 * slot;
        const T lr = line_raw(np);
        const T nhe = rplus(hh, 1), nhw = rminus(hh + 1, 1);
        T nc, ncoef;
        celerity_coef(mid6(hh, 1), L.s_ndz[slot], nc, ncoef);
        nh[0] = nhe;
        nh[1] = nhw;
        nh[2] = ncoef;
        np[0] = lr;
      }
      __syncthreads();
    }
  }

  // ---- 4. phase H ------------------------------------------------------------------
  tile_faces<T, TI, TJ, false, PW>(io, b, m, ni, nj, sm + F::kH + 3 * PW + 6, sm + F::kH + 6 * PW + 3, L);
  __syncthreads();
  tile_cells<T, TI, TJ, false>(io, b, n, m, ni, nj, &hpc, TermsAt<T, TI, TJ, true>(io.fx, b, n), L);
}

}  // namespace bt
