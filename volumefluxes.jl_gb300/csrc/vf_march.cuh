// vf_march.cuh -- column-marching step kernels.
//
// Each warp owns a strip of 32 consecutive columns: lanes 2..29 produce the 28
// output columns, lanes 0-1 and 30-31 are the 2-cell halo. The warp marches up
// a segment of SEG rows keeping a 3-row register window of (w, hu, hv); the
// y-direction reconstruction, central-upwind face flux and bottom source are
// carried from row to row in registers, and x-neighbours come from warp
// shuffles. No shared memory and no block-wide barrier: every face flux of the
// strip is computed once (plus the halo faces), which is what matters on
// GB300 where the Float64 pipe is 1/64 of the Float32 rate and Float32 is
// instruction-issue bound.
//
// flux pass  (k_flux_march):  L(U0) of src/system.jl:62-75, S(U0) of
//            src/friction.jl:62-78, CFL maxima (src/numericalflux/numericalflux.jl:32).
// stage pass (k_stage_march): U1 = clamp((U0 + dt*L) ./ (1 .- dt*[0,S,S])) with its
//            wall ghosts, formed on the fly for every loaded row; then stage 2 on U1,
//            the RK2 average, friction, dry clamp and U2's wall ghosts
//            (src/timestepper/rungekutta.jl:26-52, src/simulator.jl:145-177).
#pragma once
#include <type_traits>
#include "vf_kernels.cuh"

namespace vf {

constexpr int MW = 32;        // lanes per strip
constexpr int MOUT = 28;      // output columns per strip
constexpr int MWPB = 4;       // warps (strips) per block

template <typename T>
__device__ __forceinline__ T shfl_up1(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }
template <typename T>
__device__ __forceinline__ T shfl_dn1(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <typename T>
__device__ __forceinline__ T shfl_idx(T v, int src) { return __shfl_sync(0xffffffffu, v, src); }

struct StripGeom {
  int lane, x, xs;     // lane, its column, first output column
  int ys, ye;          // output rows [ys, ye)
  int xl;              // column the lane loads from: its own, or the last one (such a lane feeds no output)
  bool out_col;        // lane holds an output column inside the domain
  bool xedge;          // some lane of the strip is a ghost column or one of the two columns next to one
};

// Strip `strip`, row segment `seg` (of seg_rows rows) for the calling warp.
template <typename T>
__device__ __forceinline__ bool strip_setup_at(const Geom<T>& g, int seg_rows, int strip, int seg, StripGeom& s) {
  s.lane = threadIdx.x & (MW - 1);
  const int nstrips = (g.nx + MOUT - 1) / MOUT;
  if (strip >= nstrips) return false;
  s.xs = g.gc + strip * MOUT;
  s.x = s.xs - 2 + s.lane;
  s.ys = g.gc + seg * seg_rows;
  s.ye = min(s.ys + seg_rows, g.gc + g.ny);
  s.out_col = s.lane >= 2 && s.lane < 2 + MOUT && s.x < g.gc + g.nx;
  s.xl = min(s.x, g.N1 - 1);
  // Lanes span columns xs-2 .. xs+29; ghost columns are < gc and >= gc+nx,
  // and the two interior columns beside each side write wall ghosts.
  s.xedge = s.xs - 2 <= g.gc + 1 || s.xs + (MW - 3) >= g.gc + g.nx - 2;
  return true;
}

// The calling warp's unit of a whole-grid launch: units count through the
// strips of one segment before the next segment, so a grid of few strips fills
// its blocks too.
template <typename T>
__device__ __forceinline__ bool strip_setup(const Geom<T>& g, int seg_rows, StripGeom& s) {
  const int unit = (int)(blockIdx.x * MWPB + (threadIdx.x >> 5));
  const int nstrips = (g.nx + MOUT - 1) / MOUT;
  const int seg = unit / nstrips;
  if (seg * seg_rows >= g.ny) return false;
  return strip_setup_at(g, seg_rows, unit - seg * nstrips, seg, s);
}

// Loads and stores of the marching kernels. A cell's byte offset from the start
// of its plane is the same in the state, derivative and friction arrays, so one
// running offset per lane (O: 32 bits where a plane is smaller than 4 GB)
// addresses all of them, and every row and column a warp visits exists: rows
// are never checked, columns are clamped once (StripGeom::xl). With a 64-bit
// index per array and checks on every row, 241 of the 618 instructions per cell
// of the Float32 flux pass and 389 of the 821 of the stage pass were addresses,
// predicates, constant loads and branches.
template <bool CG, typename T, typename O>
__device__ __forceinline__ T ldo(const T* base, O off) {
  return gld<CG>(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off));
}
template <typename T, typename O>
__device__ __forceinline__ void sto(T* base, O off, T v) {
  *reinterpret_cast<T*>(reinterpret_cast<char*>(base) + off) = v;
}
// Byte offset of column x of row r of an array whose rows are `pitch` elements apart.
template <typename T, typename O>
__device__ __forceinline__ O row_off(long long pitch, int x, int r) {
  return (O)(((O)r * (O)pitch + (O)(x + XOFF)) * (O)sizeof(T));
}

// Bottom corners (x, r) and (x+1, r) of one corner row.
template <typename T>
struct CornerRow {
  T a, b;
};

// CB 0: corner array, 1: constant bottom, 2: as g says.
template <int CB, typename T>
__device__ __forceinline__ bool flat(const Geom<T>& g) {
  return CB == 1 || (CB == 2 && g.bottom_const);
}
template <int CB, typename T, typename O>
__device__ __forceinline__ CornerRow<T> load_corner_row(const Geom<T>& g, const T* __restrict__ B, O off) {
  if (flat<CB>(g)) return CornerRow<T>{g.bconst, g.bconst};
  return CornerRow<T>{ldo<false>(B, off), ldo<false>(B + 1, off)};
}

// Lookups of src/bottom_topography.jl:97-101 from two corner rows (lo = row of
// the cell, hi = the row above).
template <int CB, typename T>
__device__ __forceinline__ T b_cell(const Geom<T>& g, const CornerRow<T>& lo, const CornerRow<T>& hi) {
  if (flat<CB>(g)) return g.bconst;
  return (T)0.25 * (((lo.a + lo.b) + hi.a) + hi.b);
}
template <int CB, typename T>
__device__ __forceinline__ T b_xface_l(const Geom<T>& g, const CornerRow<T>& lo, const CornerRow<T>& hi) {
  if (flat<CB>(g)) return g.bconst;
  return (T)0.5 * (lo.a + hi.a);
}
template <int CB, typename T>
__device__ __forceinline__ T b_yface(const Geom<T>& g, const CornerRow<T>& r) {
  if (flat<CB>(g)) return g.bconst;
  return (T)0.5 * (r.a + r.b);
}

template <typename T>
struct Cell3 {
  T w, hu, hv;
};

template <bool CG, typename T, typename O>
__device__ __forceinline__ Cell3<T> load_cell(const Geom<T>& g, const T* U, O off) {
  return Cell3<T>{ldo<CG>(U, off), ldo<CG>(U + g.PS, off), ldo<CG>(U + 2 * g.PS, off)};
}

// Reconstruction of this lane's cell along y (DIR 1) or x (DIR 0); lo and hi are
// the cell's corner rows.
template <int CB, bool GEN, typename T>
__device__ __forceinline__ void recon(const Geom<T>& g, const Phys<T>& p, const Cell3<T>& l, const Cell3<T>& c,
                                      const Cell3<T>& r, T Bl, T Br, const CornerRow<T>& lo, const CornerRow<T>& hi,
                                      Cell3<T>& L, Cell3<T>& R) {
  const T lv[3] = {l.w, l.hu, l.hv}, cv[3] = {c.w, c.hu, c.hv}, rv[3] = {r.w, r.hu, r.hv};
  T Lv[3], Rv[3];
  if (GEN && p.rec_none) no_reconstruction<T>(cv, b_cell<CB>(g, lo, hi), Lv, Rv);
  else reconstruct_cell<T>(p, lv, cv, rv, Bl, Br, Lv, Rv);
  L = Cell3<T>{Lv[0], Lv[1], Lv[2]};
  R = Cell3<T>{Rv[0], Rv[1], Rv[2]};
}

template <typename T, int DIR, bool SPEED>
__device__ __forceinline__ Cell3<T> face(const Phys<T>& p, const Cell3<T>& m, const Cell3<T>& q, T& speed) {
  Cell3<T> F;
  cu_face<T, DIR, SPEED>(p, m.w, m.hu, m.hv, q.w, q.hu, q.hv, F.w, F.hu, F.hv, speed);
  return F;
}

// Bottom source of one direction added to acc (src/sourceterms/source_term_bottom.jl:34-40):
// once per SourceTermBottom entry in order; Float32 adds n_bottom * (-g) times
// the term at once (no loop; the same value for the usual single entry up to
// where multiply-add contraction falls).
template <typename T>
__device__ __forceinline__ T add_bottom(const Phys<T>& p, T acc, T slope, T hmean) {
  if constexpr (sizeof(T) == 4) {
    return acc + p.bottom_g * slope * hmean;
  } else {
    for (int b = 0; b < p.n_bottom; ++b) acc = acc + p.neg_g * slope * hmean;
    return acc;
  }
}

// x-direction contribution of row j for this lane: -(1/Δx)(F_{x+1/2} - F_{x-1/2})
// plus the bottom source along x (src/numericalflux/numericalflux.jl:24-30,
// src/sourceterms/source_term_bottom.jl:34-40). Every lane participates in the
// shuffles; lanes 2..30 compute valid faces x-1/2.
template <int CB, bool SPEED, bool GEN, typename T>
__device__ __forceinline__ Cell3<T> x_derivative(const Geom<T>& g, const Phys<T>& p, const Cell3<T>& u,
                                                 const CornerRow<T>& clo, const CornerRow<T>& chi, T& sx) {
  Cell3<T> ul{shfl_up1(u.w), shfl_up1(u.hu), shfl_up1(u.hv)};
  Cell3<T> ur{shfl_dn1(u.w), shfl_dn1(u.hu), shfl_dn1(u.hv)};
  const T bl = b_xface_l<CB>(g, clo, chi);
  const T br = shfl_dn1(bl);  // right x-face of x == left x-face of x+1
  Cell3<T> L, R;
  recon<CB, GEN>(g, p, ul, u, ur, bl, br, clo, chi, L, R);
  const Cell3<T> Rm{shfl_up1(R.w), shfl_up1(R.hu), shfl_up1(R.hv)};
  T sp = (T)0;
  const Cell3<T> Fl = face<T, 0, SPEED>(p, Rm, L, sp);  // face x-1/2
  if (SPEED) sx = sp;
  const Cell3<T> Fr{shfl_dn1(Fl.w), shfl_dn1(Fl.hu), shfl_dn1(Fl.hv)};
  Cell3<T> acc;
  acc.w = (T)0 - p.inv_dx * (Fr.w - Fl.w);
  acc.hu = (T)0 - p.inv_dx * (Fr.hu - Fl.hu);
  acc.hv = (T)0 - p.inv_dx * (Fr.hv - Fl.hv);
  acc.hu = add_bottom<T>(p, acc.hu, slope_over<T>(br - bl, p.dx, p.inv_dx, p.dx_pow2), (R.w + L.w) * (T)0.5);
  return acc;
}

// March state of the y direction: reconstruction of row j and flux of face j-1/2.
template <typename T>
struct YCarry {
  Cell3<T> R;     // right (upper) face value of row j
  T Lh;           // left (lower) face depth of row j
  T Bl, Br;       // y-face bottoms of row j
  Cell3<T> Gm;    // flux through face j-1/2
};

__device__ __forceinline__ void warp_speed_max(unsigned long long& k) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
}

// Block reduction of the per-warp CFL maxima, one atomicMax per direction.
__device__ __forceinline__ void block_speed_commit(StepRecord* rec, int parity, unsigned long long kx,
                                                   unsigned long long ky) {
  __shared__ unsigned long long red[2][MWPB];
  warp_speed_max(kx);
  warp_speed_max(ky);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = kx;
    red[1][threadIdx.x >> 5] = ky;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long m = 0;
#pragma unroll
    for (int w = 0; w < MWPB; ++w) m = max(m, red[threadIdx.x][w]);
    if (m) atomicMax(&rec->speed_bits[parity][threadIdx.x], m);
  }
}

// ---------------------------------------------------------------------------
// Rain and infiltration of an output cell (GEN: the time- and cell-dependent ones too).
template <typename T, bool GEN>
__device__ __forceinline__ T march_sources(const Geom<T>& g, const Phys<T>& p, T acc, const T* scal, const StripGeom& s,
                                           int j) {
  if constexpr (GEN) {
    if (p.any_dynamic) return s.out_col ? add_point_sources<T>(p, acc, scal, sidx(g, s.x, j)) : acc;
  }
  return add_point_sources<T>(p, acc);
}

// Flux pass of one strip segment (warp-collective): L(U0), S(U0); mx, my
// collect the warp's CFL maxima as bit-pattern keys. scal holds point_scalars().
template <typename T, bool CG, typename O, bool GEN = false, int CB = 2>
__device__ __forceinline__ void flux_march_unit(const Geom<T>& g, const Phys<T>& p, const T* U,
                                                const T* __restrict__ B, T* Lout, T* Sout, const StripGeom& s,
                                                unsigned long long& mx_out, unsigned long long& my_out,
                                                const T* scal = nullptr) {
  // Float32 speed keys fit 32 bits: one 32-bit max per face instead of a
  // 64-bit one (the flux pass measured 0.367 instead of 0.385 ms at 4096^2).
  using Key = typename std::conditional<sizeof(T) == 4, unsigned, unsigned long long>::type;
  Key mx = 0, my = 0;
  const O P = (O)(g.P * (long long)sizeof(T)), PB = (O)(g.PB * (long long)sizeof(T));
  // prologue: rows ys-2..ys+1, corner rows ys-1..ys+2
  O o = row_off<T, O>(g.P, s.xl, s.ys - 2), ob = row_off<T, O>(g.PB, s.xl, s.ys - 1);
  const Cell3<T> um2 = load_cell<CG>(g, U, o);
  const Cell3<T> um1 = load_cell<CG>(g, U, o += P);
  Cell3<T> uc = load_cell<CG>(g, U, o += P);
  Cell3<T> un = load_cell<CG>(g, U, o += P);
  const CornerRow<T> cm1 = load_corner_row<CB>(g, B, ob);
  CornerRow<T> c0 = load_corner_row<CB>(g, B, ob += PB);
  CornerRow<T> c1 = load_corner_row<CB>(g, B, ob += PB);
  YCarry<T> y;
  {
    Cell3<T> Lm, Rm, L0, R0;
    const T blm = b_yface<CB>(g, cm1), b0 = b_yface<CB>(g, c0), b1 = b_yface<CB>(g, c1);
    recon<CB, GEN>(g, p, um2, um1, uc, blm, b0, cm1, c0, Lm, Rm);  // row ys-1
    recon<CB, GEN>(g, p, um1, uc, un, b0, b1, c0, c1, L0, R0);     // row ys
    T sp = (T)0;
    y.Gm = face<T, 1, true>(p, Rm, L0, sp);
    if (s.out_col) my = max(my, (Key)speed_key<T>(sp));
    y.R = R0;
    y.Lh = L0.w;
    y.Bl = b0;
    y.Br = b1;
  }
  const bool face_col = s.lane >= 2 && s.lane <= 2 + MOUT && s.x <= g.gc + g.nx;
  for (int j = s.ys; j < s.ye; ++j) {
    const Cell3<T> u2 = load_cell<CG>(g, U, o += P);
    const CornerRow<T> c2 = load_corner_row<CB>(g, B, ob += PB);
    T sx = (T)0;
    Cell3<T> acc = x_derivative<CB, true, GEN>(g, p, uc, c0, c1, sx);
    if (face_col) mx = max(mx, (Key)speed_key<T>(sx));
    // y: reconstruct row j+1, flux through face j+1/2
    Cell3<T> Ln, Rn;
    const T b2 = b_yface<CB>(g, c2);
    recon<CB, GEN>(g, p, uc, un, u2, y.Br, b2, c1, c2, Ln, Rn);
    T sp = (T)0;
    const Cell3<T> Gp = face<T, 1, true>(p, y.R, Ln, sp);
    if (s.out_col) my = max(my, (Key)speed_key<T>(sp));
    acc.w = acc.w - p.inv_dy * (Gp.w - y.Gm.w);
    acc.hu = acc.hu - p.inv_dy * (Gp.hu - y.Gm.hu);
    acc.hv = acc.hv - p.inv_dy * (Gp.hv - y.Gm.hv);
    acc.hv = add_bottom<T>(p, acc.hv, slope_over<T>(y.Br - y.Bl, p.dy, p.inv_dy, p.dy_pow2), (y.R.w + y.Lh) * (T)0.5);
    acc.w = march_sources<T, GEN>(g, p, acc.w, scal, s, j);
    if (s.out_col) {
      const O oj = o - 2 * P;  // row j
      sto(Lout, oj, acc.w);
      sto(Lout + g.PS, oj, acc.hu);
      sto(Lout + 2 * g.PS, oj, acc.hv);
      if (p.friction) {
        T S = (T)0;
        if (friction_active<T>(uc.hu, uc.hv)) S = friction_factor<T>(p, uc.w, uc.hu, uc.hv, b_cell<CB>(g, c0, c1));
        sto(Sout, oj, S);
      }
    }
    // shift the window
    uc = un;
    un = u2;
    c0 = c1;
    c1 = c2;
    y.R = Rn;
    y.Lh = Ln.w;
    y.Bl = y.Br;
    y.Br = b2;
    y.Gm = Gp;
  }
  mx_out = max(mx_out, (unsigned long long)mx);
  my_out = max(my_out, (unsigned long long)my);
}

// Resident blocks per SM the Float32 kernels are compiled for. The flux pass
// fits eight (64 registers, no spill); the stage pass runs best at seven (72
// registers, 100 bytes of spill): 4096^2 wet/dry, four steps, 2.62 ms at 8 / 7
// blocks, 2.67 at 8 / 6, 2.71 at 8 / 8 (3.15 before the offsets, the branch-free
// faces and the shared Float32 dt; 2.59 at 8 / 7 with the faces' selects). Float64 (190 registers) is bound by the FP64
// pipe and is left alone.
#ifndef VF_MARCH_STAGE_BLOCKS_F32
#define VF_MARCH_STAGE_BLOCKS_F32 7
#endif
#ifndef VF_MARCH_FLUX_BLOCKS_F32
#define VF_MARCH_FLUX_BLOCKS_F32 8
#endif
template <typename T> struct MarchStageBlocks {
  static constexpr int value = sizeof(T) == 4 ? VF_MARCH_STAGE_BLOCKS_F32 : 1;
  static constexpr int general = sizeof(T) == 4 ? 6 : 1;
  static constexpr int resident = sizeof(T) == 4 ? value : 4, resident_general = sizeof(T) == 4 ? general : 4;
};
template <typename T> struct MarchFluxBlocks {
  static constexpr int value = sizeof(T) == 4 ? VF_MARCH_FLUX_BLOCKS_F32 : 1;
  static constexpr int resident = sizeof(T) == 4 ? value : 4;
};

// GEN: NoReconstruction and time- or cell-dependent sources as well (the ghost
// cells come from memory, so the boundary kind does not matter here).
template <typename T, typename O, bool GEN, int CB>
__global__ void __launch_bounds__(MW * MWPB, MarchFluxBlocks<T>::value) k_flux_march(Geom<T> g, Phys<T> p, const T* __restrict__ U,
                                                          const T* __restrict__ B, T* __restrict__ Lout,
                                                          T* __restrict__ Sout, StepRecord* rec, int parity, int seg_rows) {
  if (!rec->active[parity]) return;
  __shared__ T scal[kScalars];
  if (GEN && p.any_dynamic) {
    if (threadIdx.x == 0) point_scalars<T>(p, rec->t[parity], scal);
    __syncthreads();
  }
  StripGeom s;
  unsigned long long mx = 0ull, my = 0ull;  // CFL maxima as bit patterns (speeds are >= 0)
  if (strip_setup(g, seg_rows, s)) flux_march_unit<T, false, O, GEN, CB>(g, p, U, B, Lout, Sout, s, mx, my, scal);
  block_speed_commit(rec, parity, mx, my);
}

// What U1 of one cell is made from: U0, L(U0) and S(U0).
template <typename T>
struct Stage1Cell {
  Cell3<T> u0, l;
  T S;
};
template <bool CG, typename T, typename O>
__device__ __forceinline__ Stage1Cell<T> load_stage1(const Geom<T>& g, const Phys<T>& p, const T* U0, const T* Lin,
                                                     const T* Sin, O off) {
  return Stage1Cell<T>{load_cell<CG>(g, U0, off), load_cell<CG>(g, Lin, off), p.friction ? ldo<CG>(Sin, off) : (T)0};
}
// U1 of one interior row for this lane (stage-1 update + dry clamp), before ghost
// mirroring. Ghost lanes compute on what their column holds and are overwritten
// by their mirror cell's value.
template <int CB, typename T>
__device__ __forceinline__ Cell3<T> stage1_row(const Geom<T>& g, const Phys<T>& p, T tdt, const Stage1Cell<T>& c,
                                               const CornerRow<T>& clo, const CornerRow<T>& chi) {
  Cell3<T> u1;
  stage1_point<T>(p, tdt, c.u0.w, c.u0.hu, c.u0.hv, c.l.w, c.l.hu, c.l.hv, c.S, b_cell<CB>(g, clo, chi), u1.w, u1.hu,
                  u1.hv);
  return u1;
}

// The same for any cell of the volume (GEN): ghost cells take U1 of their boundary
// source cell, computed the same pointwise way from global memory, or for
// NeumannBC's right and top ghosts their own isolated update; corner ghosts are
// zero.
template <bool CG, int CB, typename T>
__device__ __forceinline__ Cell3<T> stage1_any(const Geom<T>& g, const Phys<T>& p, T tdt, const T* U0, const T* Lin,
                                               const T* Sin, const T* __restrict__ B, const T* scal, int x, int r,
                                               const Stage1Cell<T>& c, bool xin, const CornerRow<T>& clo,
                                               const CornerRow<T>& chi) {
  const bool yin = r >= g.gc && r < g.gc + g.ny;
  if (xin && yin) return stage1_row<CB>(g, p, tdt, c, clo, chi);
  Cell3<T> u{(T)0, (T)0, (T)0};
  if (yin == xin || x >= g.N1) return u;
  const int axis = yin ? 0 : 1, v = yin ? x : r, n = yin ? g.nx : g.ny;
  if (g.bc == 3 && v >= g.gc + n) {
    T a0, a1, a2, lpt, Bg;
    neumann_u1<T, CG>(g, p, tdt, U0, B, scal, yin ? g.N1 - 1 : x, yin ? r : g.N2 - 1, u.w, u.hu, u.hv, a0, a1, a2, lpt, Bg);
    return u;
  }
  const int q = bc_source(v, g.gc, n, g.bc, axis);
  u1_global<T, CG>(g, p, tdt, U0, Lin, Sin, B, yin ? q : x, yin ? r : q, u.w, u.hu, u.hv);
  if (g.bc == 1) {
    if (yin) u.hu = -u.hu;
    else u.hv = -u.hv;
  }
  return u;
}

// Wall ghost columns of a U1 row (src/bc.jl:92-100): ghost lanes read their
// mirror source lane, hu negated. Every lane takes part in the shuffles.
template <typename T>
__device__ __forceinline__ Cell3<T> mirror_columns(const Geom<T>& g, const StripGeom& s, const Cell3<T>& u, bool yin) {
  if (!s.xedge) return u;  // warp-uniform: no ghost column in this strip
  int src = s.lane;
  bool ghost = false;
  if (yin && s.x < g.gc) {
    src = s.lane + (2 * g.gc - 1 - 2 * s.x);
    ghost = true;
  } else if (yin && s.x >= g.gc + g.nx && s.x < g.N1) {
    src = s.lane + (2 * (g.gc + g.nx) - 1 - 2 * s.x);
    ghost = true;
  }
  src = min(max(src, 0), MW - 1);
  Cell3<T> m{shfl_idx(u.w, src), shfl_idx(u.hu, src), shfl_idx(u.hv, src)};
  if (!ghost) return u;
  m.hu = -m.hu;
  return m;
}

template <typename T>
__device__ __forceinline__ Cell3<T> mirror_row(const Cell3<T>& src) {  // src/bc.jl:101-109, hv negated
  return Cell3<T>{src.w, src.hu, -src.hv};
}

// U2 of cell (x, j) and the wall ghosts it is the mirror source of
// (src/bc.jl:81-110): what store_with_ghosts writes for a wall boundary, with
// the ghost logic skipped in warp-uniform branches for strips without ghost
// columns and rows away from the bottom and top. With mirror_columns' early
// return for such strips, the Float32 stage pass at 4096^2 measured 0.503
// instead of 0.543 ms (the same bits).
template <typename T, typename O>
__device__ __forceinline__ void store_march(const Geom<T>& g, const StripGeom& s, T* __restrict__ Uo, O off, int x,
                                            int j, T w, T hu, T hv) {
  if (s.xedge || j < g.gc + 2 || j >= g.gc + g.ny - 2) {
    store_with_ghosts<T>(g, Uo, x, j, w, hu, hv);
    return;
  }
  sto(Uo, off, w);
  sto(Uo + g.PS, off, hu);
  sto(Uo + 2 * g.PS, off, hv);
}

// RK2 stage pass of one strip segment (warp-collective): U2 with its ghosts into
// Uo. GEN: every boundary kind, reconstruction and source; otherwise walls,
// whose ghosts come from the window by shuffles and row mirrors.
template <typename T, bool CG, typename O, bool GEN = false, int CB = 2>
__device__ __forceinline__ void stage_march_unit(const Geom<T>& g, const Phys<T>& p, const T* U0,
                                                 const T* __restrict__ B, const T* Lin, const T* Sin, T* Uo,
                                                 const StripGeom& s, T tdt, const T* scal = nullptr) {
  const int x = s.x;
  const bool xin = x >= g.gc && x < g.gc + g.nx;
  const int top = g.gc + g.ny;  // first top ghost row
  const O P = (O)(g.P * (long long)sizeof(T)), PB = (O)(g.PB * (long long)sizeof(T));
  O o = row_off<T, O>(g.P, s.xl, s.ys), ob = row_off<T, O>(g.PB, s.xl, s.ys - 2);
  // U1 of row r from its cells c, between the corner rows lo and hi
  auto u1_of = [&](int r, const Stage1Cell<T>& c, const CornerRow<T>& lo, const CornerRow<T>& hi) -> Cell3<T> {
    if constexpr (GEN) return stage1_any<CG, CB>(g, p, tdt, U0, Lin, Sin, B, scal, x, r, c, xin, lo, hi);
    else return mirror_columns(g, s, stage1_row<CB>(g, p, tdt, c, lo, hi), true);
  };
  auto u1_row = [&](int r, O off, const CornerRow<T>& lo, const CornerRow<T>& hi, Cell3<T>& u0) -> Cell3<T> {
    const Stage1Cell<T> c = load_stage1<CG>(g, p, U0, Lin, Sin, off);
    u0 = c.u0;
    return u1_of(r, c, lo, hi);
  };
  // prologue: corner rows ys-2..ys+2, U1 rows ys-2..ys+1
  const CornerRow<T> cm2 = load_corner_row<CB>(g, B, ob);
  const CornerRow<T> cm1 = load_corner_row<CB>(g, B, ob += PB);
  CornerRow<T> c0 = load_corner_row<CB>(g, B, ob += PB);
  CornerRow<T> c1 = load_corner_row<CB>(g, B, ob += PB);
  CornerRow<T> c2 = load_corner_row<CB>(g, B, ob += PB);
  Cell3<T> u0c{(T)0, (T)0, (T)0}, u0n{(T)0, (T)0, (T)0}, dummy;
  Cell3<T> uc = u1_row(s.ys, o, c0, c1, u0c);
  Cell3<T> un;
  if (!GEN && s.ys + 1 >= top) {
    un = mirror_row(uc);  // top ghost above a one-row segment
  } else {
    un = u1_row(s.ys + 1, o + P, c1, c2, u0n);
  }
  Cell3<T> um1, um2;
  if (!GEN && s.ys == g.gc) {  // bottom ghosts mirror rows gc, gc+1
    um1 = mirror_row(uc);
    um2 = mirror_row(un);
  } else {
    um1 = u1_row(s.ys - 1, o - P, cm1, c0, dummy);
    if (!GEN && s.ys == g.gc + 1) um2 = mirror_row(um1);  // one-row segments: the ghost below row gc
    else um2 = u1_row(s.ys - 2, o - 2 * P, cm2, cm1, dummy);
  }
  // Ghost row top+1 mirrors row top-2, which leaves the window before it is needed.
  Cell3<T> stash{(T)0, (T)0, (T)0};
  if (!GEN && s.ys + 1 == top) stash = mirror_row(um1);
  YCarry<T> y;
  {
    Cell3<T> Lm, Rm, L0, R0;
    const T blm = b_yface<CB>(g, cm1), b0 = b_yface<CB>(g, c0), b1 = b_yface<CB>(g, c1);
    recon<CB, GEN>(g, p, um2, um1, uc, blm, b0, cm1, c0, Lm, Rm);
    recon<CB, GEN>(g, p, um1, uc, un, b0, b1, c0, c1, L0, R0);
    T sp;
    y.Gm = face<T, 1, false>(p, Rm, L0, sp);
    y.R = R0;
    y.Lh = L0.w;
    y.Bl = b0;
    y.Br = b1;
  }
  for (int j = s.ys; j < s.ye; ++j) {
    // The cells of row j+2 are asked for before the x direction of row j, which
    // does not need them, and used after it.
    const CornerRow<T> c3 = load_corner_row<CB>(g, B, ob += PB);
    Stage1Cell<T> next{};
    const bool inner = GEN || j + 2 < top;
    if (inner) next = load_stage1<CG>(g, p, U0, Lin, Sin, o + 2 * P);
    T sx;
    Cell3<T> acc = x_derivative<CB, false, GEN>(g, p, uc, c0, c1, sx);
    // U1 of row j+2 (needs corner rows j+2, j+3)
    Cell3<T> u2;
    if (inner) {
      u2 = u1_of(j + 2, next, c2, c3);
    } else if (j + 2 == top) {
      u2 = mirror_row(un);     // row top mirrors top-1
      stash = mirror_row(uc);  // row top+1 mirrors top-2
    } else {
      u2 = stash;
    }
    Cell3<T> Ln, Rn;
    const T b2 = b_yface<CB>(g, c2);
    recon<CB, GEN>(g, p, uc, un, u2, y.Br, b2, c1, c2, Ln, Rn);
    T sp;
    const Cell3<T> Gp = face<T, 1, false>(p, y.R, Ln, sp);
    acc.w = acc.w - p.inv_dy * (Gp.w - y.Gm.w);
    acc.hu = acc.hu - p.inv_dy * (Gp.hu - y.Gm.hu);
    acc.hv = acc.hv - p.inv_dy * (Gp.hv - y.Gm.hv);
    acc.hv = add_bottom<T>(p, acc.hv, slope_over<T>(y.Br - y.Bl, p.dy, p.inv_dy, p.dy_pow2), (y.R.w + y.Lh) * (T)0.5);
    acc.w = march_sources<T, GEN>(g, p, acc.w, scal, s, j);
    if (s.out_col) {
      T w = uc.w + tdt * acc.w;
      T hu = uc.hu + tdt * acc.hu;
      T hv = uc.hv + tdt * acc.hv;
      w = (T)0.5 * (u0c.w + w);
      hu = (T)0.5 * (u0c.hu + hu);
      hv = (T)0.5 * (u0c.hv + hv);
      const T Bc = b_cell<CB>(g, c0, c1);
      if (p.friction && friction_active<T>(uc.hu, uc.hv))
        apply_friction<T>(tdt, friction_factor<T>(p, uc.w, uc.hu, uc.hv, Bc), hu, hv);
      dry_clamp<T>(p, w, hu, hv, Bc);
      store_march<T>(g, s, Uo, o, x, j, w, hu, hv);
      if (GEN && g.bc == 3) {
        if (x == g.gc + g.nx - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, scal, g.N1 - 1, j, 0, true, Uo);
        if (j == g.gc + g.ny - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, scal, x, g.N2 - 1, 1, true, Uo);
      }
    }
    o += P;
    uc = un;
    un = u2;
    u0c = u0n;
    u0n = next.u0;
    c0 = c1;
    c1 = c2;
    c2 = c3;
    y.R = Rn;
    y.Lh = Ln.w;
    y.Bl = y.Br;
    y.Br = b2;
    y.Gm = Gp;
  }
}

template <typename T, typename O, bool GEN, int CB>
__global__ void __launch_bounds__(MW * MWPB, GEN ? MarchStageBlocks<T>::general : MarchStageBlocks<T>::value) k_stage_march(Geom<T> g, Phys<T> p, const T* __restrict__ U0,
                                                           const T* __restrict__ B, const T* __restrict__ Lin,
                                                           const T* __restrict__ Sin, T* __restrict__ Uo,
                                                           StepRecord* rec, int parity, int seg_rows) {
  const bool root = blockIdx.x == 0 && threadIdx.x == 0;
  if (!rec->active[parity]) {
    if (root) carry_record(rec, parity);
    return;
  }
  // dt in the state's type, shared: left to every thread, the conversion from
  // double was redone three times a row, on the FP64 pipe.
  __shared__ T s_dt;
  __shared__ T scal[kScalars];
  double dt = 0.0;
  if (threadIdx.x == 0) {
    dt = step_dt<T>(g, rec, parity);
    s_dt = (T)dt;
    if (GEN && p.any_dynamic) point_scalars<T>(p, rec->t[parity], scal);
  }
  __syncthreads();
  StripGeom s;
  if (strip_setup(g, seg_rows, s)) stage_march_unit<T, false, O, GEN, CB>(g, p, U0, B, Lin, Sin, Uo, s, s_dt, scal);
  if (root) advance_record<T>(rec, parity, dt);
}

}  // namespace vf
