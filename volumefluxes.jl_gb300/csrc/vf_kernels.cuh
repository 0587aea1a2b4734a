// vf_kernels.cuh -- the fused tile kernels of one RK2 / forward-Euler step.
//
// A step is two launches (three for nothing else):
//   flux pass   reads U0 (+2-cell halo) and B, computes the time derivative
//               L(U0) of src/system.jl:62-75 (x then y: reconstruction, central-
//               upwind fluxes, bottom source; then rain/infiltration), the
//               friction factor S(U0) of src/friction.jl:62-78, and the CFL
//               maxima (warp shuffles + one atomicMax per block per direction).
//   stage pass  (RK2) reads U0, L, S on the tile + halo, forms the stage-1
//               result U1 = clamp((U0 + dt*L) ./ (1 .- dt*[0,S,S])) pointwise in
//               shared memory with its wall ghosts, runs the whole stage-2
//               derivative on U1, then the Euler update, RK2 average, friction,
//               dry clamp and wall ghosts of U2 (src/timestepper/rungekutta.jl:26-52,
//               src/simulator.jl:145-177). dt comes from the flux pass's maxima
//               (src/simulator.jl:147-150) and is computed on the device.
//   apply pass  (forward Euler) the pointwise stage-1 update alone.
//
// Tiles are TX x TY interior cells (TileShape); each block stages its tile with a 2-cell
// halo of (w, hu, hv) and a 2..3-cell halo of bottom corners in shared memory.
// The Float64 kernels of the per-step path (k_flux_tma, k_stage2_tma) stage
// them with TMA copies, and the stage pass writes its output tile with a TMA
// tensor store (vf_tma.cuh); the ensemble and Float32 tiles load and store
// the plain way.
#pragma once
#include "vf_math.cuh"
#include "vf_tma.cuh"

namespace vf {

// Tile of X x Y interior cells worked on by N threads, of which B blocks are to
// fit on an SM (launch bounds). D: the x and the y direction at the same time,
// half of the warps each, instead of one after the other.
template <int X, int Y, int N, int B, bool D>
struct TileShape {
  static constexpr int TX = X, TY = Y, NT = N, MINB = B;
  static constexpr bool SPLIT = D;
  static constexpr int DIRS = D ? 2 : 1;               // buffers of face values and fluxes
  static constexpr int CPT = (TX * TY + NT - 1) / NT;  // cells per thread
  static constexpr int HX = TX + 4, HY = TY + 4;
  static constexpr int BHX = TX + 6;  // TX + 5 corner columns are read; one more keeps Float64 rows 16-byte multiples
  static constexpr int BHY = TY + 5;
  static constexpr int LRN = (TX + 2) * TY > TX * (TY + 2) ? (TX + 2) * TY : TX * (TY + 2);
  static constexpr int FN = (TX + 1) * TY > TX * (TY + 1) ? (TX + 1) * TY : TX * (TY + 1);
};
using BigTile = TileShape<32, 16, 256, 1, false>;  // Float32, and the ensemble in both precisions
// Float64: 288 threads hold every phase of a 16x16 tile in one pass (18 x 16
// cells reconstructed), in 72 registers and 40 KB, so 27 warps of three blocks
// share an SM and wait at one another's barriers less than 24 warps of 32x16
// tiles: 2.36 instead of 2.41 ms per step at 2048^2, 0.68 / 0.73 at 1024^2,
// 0.241 / 0.292 at 512^2, 0.084 / 0.115 at 256^2 (two blocks of 112 registers:
// 2.49 ms at 2048^2). 8x8 tiles with the directions side by side halve the
// chain of phases that bounds a grid of few tiles: 37 instead of 62 us per step
// up to 96^2, 47 / 59 at 160x128, 59 / 59 at 192^2, 105 / 84 at 256^2 (32x16
// tiles: 117 us up to 256^2, 8 tiles for 64^2).
using SmallTile = TileShape<16, 16, 288, 3, false>;
using TinyTile = TileShape<8, 8, 192, 4, true>;
constexpr int TX = BigTile::TX, TY = BigTile::TY, NT = BigTile::NT;
constexpr int HX = BigTile::HX, HY = BigTile::HY, BHX = BigTile::BHX, BHY = BigTile::BHY;
constexpr int XOFF = 2;  // leading pad columns in device rows

// Device-resident step record. Slots indexed by step parity let every kernel
// of step n read slot n&1 while the stage pass prepares slot (n+1)&1.
struct StepRecord {
  unsigned long long speed_bits[2][2];  // CFL maxima (ax, ay) as IEEE bit patterns, >= 0
  double t[2];
  int active[2];
  int match_endtime;
  int has_max_ts;
  double endtime;
  double max_ts;
  double stop_time;
  double last_dt;
  long long n_done;
  long long max_steps;  // device loop: stop after this many steps (0: no limit)
  double explicit_max_dt;
  int explicit_mode;
  int force_dt;        // 1: every step uses forced_dt (a frozen dt sequence)
  int wait_fault;      // set when a bounded wait for a tile copy gave up
  int stop_stalled;    // device loop: stop after a step that leaves t unchanged (batch members)
  int stalled;         // set when it did
  double forced_dt;
};

template <typename T>
struct Geom {
  int nx, ny, gc, N1, N2;
  long long P, PS, PB;  // state row pitch, plane stride, corner row pitch (elements)
  int bottom_const;
  T bconst;
  double dx, dy, cfl;
  int bc;  // 1 wall (src/bc.jl:81-110), 2 periodic (src/bc.jl:29-40)
};

// Interior source cell of ghost coordinate v (0 <= v < n + 2gc) along axis 0
// (x) or 1 (y): the mirror for walls (src/bc.jl:81-110), the opposite side for
// periodic boundaries (src/bc.jl:29-40). NeumannBC as src/bc.jl:49-60 writes
// it: the left columns mirror the interior, the bottom rows copy the top
// interior rows; its right and top ghosts have no source (neumann_outer).
__device__ __forceinline__ int bc_source(int v, int gc, int n, int bc, int axis) {
  if (bc == 2 || (bc == 3 && axis == 1 && v < gc)) return v < gc ? v + n : v - n;
  return v < gc ? 2 * gc - 1 - v : 2 * (gc + n) - 1 - v;
}

// Byte offsets within one state plane, and within the corner array, fit 32 bits.
template <typename T>
__host__ __device__ inline bool plane_fits_u32(const Geom<T>& g) {
  return g.PB * (long long)(g.N2 + 1) * (long long)sizeof(T) < (1ll << 32);
}

template <typename T>
__device__ __forceinline__ long long sidx(const Geom<T>& g, int x, int y) {
  return (long long)y * g.P + x + XOFF;
}

// Global load of step data. CG = true reads through L2 only (ld.global.cg): the
// ensemble kernel reads fields that other CTAs of its cluster wrote earlier in
// the same launch, which the read-only and L1 paths may not see.
template <bool CG, typename T>
__device__ __forceinline__ T gld(const T* ptr) {
  if constexpr (CG) {
    return __ldcg(ptr);
  } else {
    return *ptr;
  }
}

// Bottom topography seen from a tile; (lx, ly) are tile-local cell coordinates,
// corner (x0+lx, y0+ly) lives at sB[(ly+2)*BHX + lx+2]. Lookups follow
// src/bottom_topography.jl:97-101.
template <typename T, typename S = BigTile>
struct BTile {
  const T* sB;
  int is_const;
  T c;
  __device__ __forceinline__ T cn(int lx, int ly) const { return sB[(ly + 2) * S::BHX + lx + 2]; }
  __device__ __forceinline__ T cell(int lx, int ly) const {
    if (is_const) return c;
    return quarter<T>(((cn(lx, ly) + cn(lx + 1, ly)) + cn(lx, ly + 1)) + cn(lx + 1, ly + 1));
  }
  template <int DIR>
  __device__ __forceinline__ T face_l(int lx, int ly) const {
    if (is_const) return c;
    return halve<T>(DIR == 0 ? cn(lx, ly) + cn(lx, ly + 1) : cn(lx, ly) + cn(lx + 1, ly));
  }
  template <int DIR>
  __device__ __forceinline__ T face_r(int lx, int ly) const {
    if (is_const) return c;
    return halve<T>(DIR == 0 ? cn(lx + 1, ly) + cn(lx + 1, ly + 1) : cn(lx, ly + 1) + cn(lx + 1, ly + 1));
  }
};

template <typename S, typename T>
__device__ __forceinline__ void load_corners(const Geom<T>& g, const T* __restrict__ B, T* sB, int x0, int y0) {
  constexpr int BHX = S::BHX, BHY = S::BHY, NT = S::NT;
  for (int idx = threadIdx.x; idx < BHX * BHY; idx += NT) {
    const int bx = idx % BHX, by = idx / BHX;
    const int cx = x0 - 2 + bx, cy = y0 - 2 + by;
    T v = (T)0;
    if (cx <= g.N1 && cy <= g.N2) v = B[(long long)cy * g.PB + cx + XOFF];
    sB[idx] = v;
  }
}

// NoReconstruction for practical SWE, src/reconstruction/noreconstruction.jl:30-46:
// both face values are (w - B_cell, hu, hv).
template <typename T>
__device__ __forceinline__ void no_reconstruction(const T c[3], T Bc, T L[3], T R[3]) {
  L[0] = R[0] = c[0] - Bc;
  L[1] = R[1] = c[1];
  L[2] = R[2] = c[2];
}

// Stage-1 result U1 of one interior cell read straight from global memory
// (used for ghost cells, whose source may lie outside the tile).
template <typename T>
__device__ __forceinline__ void stage1_point(const Phys<T>& p, T tdt, T u0, T u1, T u2, T l0, T l1, T l2, T S, T Bc,
                                             T& w, T& hu, T& hv);
template <typename T, bool CG>
__device__ __forceinline__ void u1_global(const Geom<T>& g, const Phys<T>& p, T tdt, const T* U0, const T* Lin,
                                          const T* Sin, const T* __restrict__ B, int x, int y, T& w, T& hu, T& hv) {
  const long long o = sidx(g, x, y);
  T Bc = g.bconst;
  if (!g.bottom_const) {
    const long long b = (long long)y * g.PB + x + XOFF;
    Bc = (T)0.25 * (((B[b] + B[b + 1]) + B[b + g.PB]) + B[b + g.PB + 1]);
  }
  const T S = p.friction ? gld<CG>(Sin + o) : (T)0;
  stage1_point<T>(p, tdt, gld<CG>(U0 + o), gld<CG>(U0 + g.PS + o), gld<CG>(U0 + 2 * g.PS + o), gld<CG>(Lin + o),
                  gld<CG>(Lin + g.PS + o), gld<CG>(Lin + 2 * g.PS + o), S, Bc, w, hu, hv);
}

// Time derivative of one stage on the tile held in sU (3 planes of HY x HX),
// direction by direction in three phases: reconstruct the tile's cells and one
// layer on either side along DIR, the faces between them, the flux differences
// and the bottom source. src/system.jl:64-70 (directions in order),
// numericalflux.jl:21-33, linearreconstruction.jl:58-102,
// source_term_bottom.jl:24-41. tid of nt threads take part.
//
// x: cells lx in [-1, TX], ly in [0, TY); y: cells lx in [0, TX), ly in [-1, TY].
template <typename S, typename T, int DIR>
__device__ __forceinline__ void tile_recon(const Phys<T>& p, const T* sU, const BTile<T, S>& bt, T* sL, T* sR, int tid,
                                           int nt) {
  constexpr int TX = S::TX, TY = S::TY, HX = S::HX, HY = S::HY, LRN = S::LRN;
  constexpr int W = DIR == 0 ? TX + 2 : TX, N = W * (DIR == 0 ? TY : TY + 2), STEP = DIR == 0 ? 1 : HX;
  for (int idx = tid; idx < N; idx += nt) {
    const int lx = DIR == 0 ? idx % W - 1 : idx % W, ly = DIR == 0 ? idx / W : idx / W - 1;
    const int c = (ly + 2) * HX + lx + 2;
    T l[3], m[3], r[3], L[3], R[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      l[k] = sU[k * HX * HY + c - STEP];
      m[k] = sU[k * HX * HY + c];
      r[k] = sU[k * HX * HY + c + STEP];
    }
    if (p.rec_none) {
      no_reconstruction<T>(m, bt.cell(lx, ly), L, R);
    } else {
      reconstruct_cell<T>(p, l, m, r, bt.template face_l<DIR>(lx, ly), bt.template face_r<DIR>(lx, ly), L, R);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      sL[k * LRN + idx] = L[k];
      sR[k * LRN + idx] = R[k];
    }
  }
}

// Faces f between cells f-1 and f: x: f in [0, TX]; y: f in [0, TY].
template <typename S, typename T, int DIR, bool SPEED>
__device__ __forceinline__ void tile_faces(const Phys<T>& p, const T* sL, const T* sR, T* sF, T& mx, int nvx, int nvy,
                                           int tid, int nt) {
  constexpr int TX = S::TX, TY = S::TY, LRN = S::LRN, FN = S::FN;
  constexpr int W = DIR == 0 ? TX + 1 : TX, N = W * (DIR == 0 ? TY : TY + 1);
  for (int idx = tid; idx < N; idx += nt) {
    const int fx = idx % W, fy = idx / W;
    const int im = DIR == 0 ? fy * (TX + 2) + fx : idx, ip = im + (DIR == 0 ? 1 : TX);
    T F0, F1, F2, sp = (T)0;
    cu_face<T, DIR, SPEED>(p, sR[im], sR[LRN + im], sR[2 * LRN + im], sL[ip], sL[LRN + ip], sL[2 * LRN + ip], F0, F1,
                           F2, sp);
    sF[idx] = F0;
    sF[FN + idx] = F1;
    sF[2 * FN + idx] = F2;
    if (SPEED && (DIR == 0 ? fy < nvy && fx <= nvx : fx < nvx && fy <= nvy)) mx = speed_max<T>(mx, sp);
  }
}

// acc[k][*] receives -(1/Δx)(F_r-F_l) [+ bottom x], then -(1/Δy)(G_r-G_l)
// [+ bottom y] for the cells this thread owns (cell tid + k*NT, x fastest).
template <typename S, typename T, int DIR>
__device__ __forceinline__ void tile_accumulate(const Phys<T>& p, const BTile<T, S>& bt, const T* sL, const T* sR,
                                                const T* sF, T (&acc)[S::CPT][3]) {
  constexpr int TX = S::TX, TY = S::TY, NT = S::NT, CPT = S::CPT, FN = S::FN;
  constexpr int STEP = DIR == 0 ? 1 : TX, M = DIR == 0 ? 1 : 2;
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int c = threadIdx.x + k * NT;
    if (CPT * NT > TX * TY && c >= TX * TY) break;
    const int lx = c % TX, ly = c / TX;
    const int fl = DIR == 0 ? ly * (TX + 1) + lx : c;
    if constexpr (std::is_same<T, double>::value) {
      T v[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) v[j] = sF[j * FN + fl + STEP] - sF[j * FN + fl];
      over_delta<DIR>(p, v);
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[k][j] = DIR == 0 ? exact::zero_minus(v[j]) : acc[k][j] - v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j)
        acc[k][j] = (DIR == 0 ? (T)0 : acc[k][j]) -
                    (DIR == 0 ? p.inv_dx : p.inv_dy) * (sF[j * FN + fl + STEP] - sF[j * FN + fl]);
    }
    const int rc = DIR == 0 ? ly * (TX + 2) + lx + 1 : c + TX;
    for (int b = 0; b < p.n_bottom; ++b) {
      const T Bl = bt.template face_l<DIR>(lx, ly), Br = bt.template face_r<DIR>(lx, ly);
      acc[k][M] = acc[k][M] + p.neg_g * bottom_slope<T, DIR>(p, Br - Bl) * halve<T>(sR[rc] + sL[rc]);
    }
  }
}

template <typename S, typename T, bool SPEED>
__device__ __forceinline__ void tile_derivative(const Phys<T>& p, const T* sU, const BTile<T, S>& bt, T* sL, T* sR,
                                                T* sF, T (&acc)[S::CPT][3], T& mx, T& my, int nvx, int nvy) {
  constexpr int NT = S::NT;
  const int tid = threadIdx.x;
  if constexpr (S::SPLIT) {
    // x and y side by side, half of the warps each, with buffers of their own
    constexpr int H = NT / 2;
    T *yL = sL + 3 * S::LRN, *yR = sR + 3 * S::LRN, *yF = sF + 3 * S::FN;
    if (tid < H) tile_recon<S, T, 0>(p, sU, bt, sL, sR, tid, H);
    else tile_recon<S, T, 1>(p, sU, bt, yL, yR, tid - H, H);
    __syncthreads();
    if (tid < H) tile_faces<S, T, 0, SPEED>(p, sL, sR, sF, mx, nvx, nvy, tid, H);
    else tile_faces<S, T, 1, SPEED>(p, yL, yR, yF, my, nvx, nvy, tid - H, H);
    __syncthreads();
    tile_accumulate<S, T, 0>(p, bt, sL, sR, sF, acc);
    tile_accumulate<S, T, 1>(p, bt, yL, yR, yF, acc);
  } else {
    tile_recon<S, T, 0>(p, sU, bt, sL, sR, tid, NT);
    __syncthreads();
    tile_faces<S, T, 0, SPEED>(p, sL, sR, sF, mx, nvx, nvy, tid, NT);
    __syncthreads();
    tile_accumulate<S, T, 0>(p, bt, sL, sR, sF, acc);
    __syncthreads();
    tile_recon<S, T, 1>(p, sU, bt, sL, sR, tid, NT);
    __syncthreads();
    tile_faces<S, T, 1, SPEED>(p, sL, sR, sF, my, nvx, nvy, tid, NT);
    __syncthreads();
    tile_accumulate<S, T, 1>(p, bt, sL, sR, sF, acc);
  }
}

template <typename T>
__device__ __forceinline__ unsigned long long speed_key(T v);
template <>
__device__ __forceinline__ unsigned long long speed_key<double>(double v) {
  return (unsigned long long)__double_as_longlong(v);
}
template <>
__device__ __forceinline__ unsigned long long speed_key<float>(float v) {
  return (unsigned long long)(unsigned)__float_as_uint(v);
}
template <typename T>
__device__ __forceinline__ double speed_from_key(unsigned long long k);
template <>
__device__ __forceinline__ double speed_from_key<double>(unsigned long long k) {
  return __longlong_as_double((long long)k);
}
template <>
__device__ __forceinline__ double speed_from_key<float>(unsigned long long k) {
  return (double)__uint_as_float((unsigned)k);
}

// ---------------------------------------------------------------------------
// Flux pass: L(U0), S(U0) and the CFL maxima.
// U and B come first: for Float64 both start 128-byte aligned (TMA destinations).
template <typename T, typename S = BigTile>
struct SmemFlux {
  T U[3 * S::HX * S::HY];
  T B[S::BHX * S::BHY];
  T L[S::DIRS * 3 * S::LRN];
  T R[S::DIRS * 3 * S::LRN];
  T F[S::DIRS * 3 * S::FN];
  unsigned long long red[2][S::NT / 32];
  T scal[kScalars];
  unsigned long long bar;  // mbarrier of the tile copies
  int plain;               // 0: staged by TMA; 1: not staged (alignment); 2: the wait gave up
};

// Flux pass over one tile at (x0, y0) (block-collective): L(U0) and S(U0) to
// global memory; mx, my accumulate this thread's share of the CFL maxima.
// t is the step's start time (time-dependent sources).
// STAGED: s.U and s.B already hold the tile (TMA).
template <typename T, bool CG, bool STAGED = false, typename S = BigTile>
__device__ __forceinline__ void flux_tile(const Geom<T>& g, const Phys<T>& p, const T* U, const T* __restrict__ B,
                                          T* Lout, T* Sout, int x0, int y0, SmemFlux<T, S>& s, double t, T& mx, T& my) {
  constexpr int TX = S::TX, TY = S::TY, NT = S::NT, CPT = S::CPT, HX = S::HX, HY = S::HY;
  const int tid = threadIdx.x;
  const int nvx = min(TX, g.gc + g.nx - x0), nvy = min(TY, g.gc + g.ny - y0);

  if constexpr (!STAGED) {
    for (int idx = tid; idx < HX * HY; idx += NT) {
      const int lx = idx % HX, ly = idx / HX;
      const int gx = x0 - 2 + lx, gy = y0 - 2 + ly;
      const bool ok = gx < g.N1 && gy < g.N2;
      const long long o = sidx(g, gx, gy);
#pragma unroll
      for (int k = 0; k < 3; ++k) s.U[k * HX * HY + idx] = ok ? gld<CG>(U + k * g.PS + o) : (T)0;
    }
    if (!g.bottom_const) load_corners<S>(g, B, s.B, x0, y0);
  }
  if (p.any_dynamic && tid == 0) point_scalars<T>(p, t, s.scal);
  __syncthreads();

  BTile<T, S> bt{s.B, g.bottom_const, g.bconst};
  T acc[CPT][3];
  tile_derivative<S, T, true>(p, s.U, bt, s.L, s.R, s.F, acc, mx, my, nvx, nvy);

#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int c = tid + k * NT;
    const int lx = c % TX, ly = c / TX;
    if (lx >= nvx || ly >= nvy) continue;  // also the threads past the tile (ly >= TY >= nvy)
    const long long o = sidx(g, x0 + lx, y0 + ly);
    acc[k][0] = p.any_dynamic ? add_point_sources<T>(p, acc[k][0], s.scal, o) : add_point_sources<T>(p, acc[k][0]);
#pragma unroll
    for (int j = 0; j < 3; ++j) Lout[j * g.PS + o] = acc[k][j];
    if (p.friction) {
      const int ci = (ly + 2) * HX + lx + 2;
      const T q0 = s.U[ci], q1 = s.U[HX * HY + ci], q2 = s.U[2 * HX * HY + ci];
      // at rest the factor is a zero whatever the depth, and every reader skips
      // zeros (Float32, bound by its registers here, computes it all the same)
      Sout[o] = sizeof(T) == 4 || friction_active<T>(q1, q2) ? friction_factor<T>(p, q0, q1, q2, bt.cell(lx, ly)) : (T)0;
    }
  }
}

// Block maximum of per-thread CFL speed keys (IEEE bit patterns of speeds
// >= 0): warp shuffles, then one shared-memory pass; valid in thread 0.
template <int NT>
__device__ __forceinline__ void block_key_max(unsigned long long kx, unsigned long long ky,
                                              unsigned long long (*red)[NT / 32], unsigned long long& kx_out,
                                              unsigned long long& ky_out) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    kx = max(kx, __shfl_xor_sync(0xffffffffu, kx, o));
    ky = max(ky, __shfl_xor_sync(0xffffffffu, ky, o));
  }
  if ((tid & 31) == 0) {
    red[0][tid >> 5] = kx;
    red[1][tid >> 5] = ky;
  }
  __syncthreads();
  if (tid == 0) {
    kx = 0;
    ky = 0;
    for (int w = 0; w < NT / 32; ++w) {
      kx = max(kx, red[0][w]);
      ky = max(ky, red[1][w]);
    }
    kx_out = kx;
    ky_out = ky;
  }
}

template <typename T, int NT>
__device__ __forceinline__ void block_speed_keys(T mx, T my, unsigned long long (*red)[NT / 32],
                                                 unsigned long long& kx_out, unsigned long long& ky_out) {
  block_key_max<NT>(speed_key<T>(mx), speed_key<T>(my), red, kx_out, ky_out);
}

template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB) k_flux(Geom<T> g, Phys<T> p, const T* __restrict__ U, const T* __restrict__ B,
                                             T* __restrict__ Lout, T* __restrict__ Sout, StepRecord* rec, int parity) {
  if (!rec->active[parity]) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemFlux<T, S>& s = *reinterpret_cast<SmemFlux<T, S>*>(smem_raw);
  const int x0 = g.gc + blockIdx.x * S::TX, y0 = g.gc + blockIdx.y * S::TY;
  const double t = p.any_dynamic ? rec->t[parity] : 0.0;
  T mx = (T)0, my = (T)0;
  flux_tile<T, false, false, S>(g, p, U, B, Lout, Sout, x0, y0, s, t, mx, my);

  // CFL maxima: warp shuffle, then one atomic per block and direction.
  unsigned long long kx = 0, ky = 0;
  block_speed_keys<T, S::NT>(mx, my, s.red, kx, ky);
  if (threadIdx.x == 0) {
    atomicMax(&rec->speed_bits[parity][0], kx);
    atomicMax(&rec->speed_bits[parity][1], ky);
  }
}

// Bytes of one staged tile of n planes, and of the corner tile.
template <typename T, typename S>
__host__ __device__ constexpr unsigned tile_bytes(int planes) { return (unsigned)(planes * S::HX * S::HY * sizeof(T)); }
template <typename T, typename S>
__host__ __device__ constexpr unsigned corner_bytes() { return (unsigned)(S::BHX * S::BHY * sizeof(T)); }

// k_flux with the tile staged by TMA (Float64). Thread 0 issues one 3D copy of
// the three state planes and one 2D copy of the corners; everyone waits on the
// mbarrier, then the flux pass runs as in k_flux.
template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB)
    k_flux_tma(Geom<T> g, Phys<T> p, const __grid_constant__ CUtensorMap mU, const __grid_constant__ CUtensorMap mB,
               const T* __restrict__ U, const T* __restrict__ B, T* __restrict__ Lout, T* __restrict__ Sout,
               StepRecord* rec, int parity) {
  static_assert(sizeof(T) == 8, "TMA tiles are Float64 (the tile origin is 16-byte aligned only for 8-byte cells)");
  if (!rec->active[parity]) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemFlux<T, S>& s = *reinterpret_cast<SmemFlux<T, S>*>(smem_raw);
  const int x0 = g.gc + blockIdx.x * S::TX, y0 = g.gc + blockIdx.y * S::TY;
  const int cx = x0 - 2 + XOFF, cy = y0 - 2;
  if (threadIdx.x == 0) {
    const bool ok = tma_ok(cx, (int)sizeof(T), s.U) && (g.bottom_const || tma_ok(cx, (int)sizeof(T), s.B));
    s.plain = ok ? 0 : 1;
    if (ok) {
      mbar_init(&s.bar, 1);
      mbar_expect_tx(&s.bar, tile_bytes<T, S>(3) + (g.bottom_const ? 0u : corner_bytes<T, S>()));
      tma_load_3d(s.U, &mU, cx, cy, 0, &s.bar);
      if (!g.bottom_const) tma_load_2d(s.B, &mB, cx, cy, &s.bar);
    }
  }
  __syncthreads();
  if (!s.plain && !mbar_wait_bounded(&s.bar, 0)) {
    rec->wait_fault = 1;
    s.plain = 2;  // gave up; every thread that gives up sets it, the barrier below makes it uniform
  }
  __syncthreads();
  const double t = p.any_dynamic ? rec->t[parity] : 0.0;
  T mx = (T)0, my = (T)0;
  if (s.plain)
    flux_tile<T, false, false, S>(g, p, U, B, Lout, Sout, x0, y0, s, t, mx, my);
  else
    flux_tile<T, false, true, S>(g, p, U, B, Lout, Sout, x0, y0, s, t, mx, my);

  unsigned long long kx = 0, ky = 0;
  block_speed_keys<T, S::NT>(mx, my, s.red, kx, ky);
  if (threadIdx.x == 0) {
    atomicMax(&rec->speed_bits[parity][0], kx);
    atomicMax(&rec->speed_bits[parity][1], ky);
  }
  // After a give-up, wait once more (bounded) so a late copy does not land
  // after the block has released its shared memory.
  if (s.plain == 2 && threadIdx.x == 0) mbar_wait_bounded(&s.bar, 0);
}

// dt of stage 1 from the CFL maxima, src/simulator.jl:147-150.
template <typename T>
__device__ __forceinline__ double cfl_dt(const Geom<T>& g, double ax, double ay, double max_dt) {
  double dt = jmin<double>(g.cfl * jmin<double>(g.dx / ax, g.dy / ay), max_dt);
  if (sizeof(T) == 4) dt = (double)(float)dt;  // current_timestep is a MVector{1,Float32}
  return dt;
}

// The simulated time after a step (t += dt, src/simulator.jl:205, in the
// backend's real type).
template <typename T>
__device__ __forceinline__ double next_time(double t, double dt) {
  return sizeof(T) == 4 ? (double)((float)t + (float)dt) : t + dt;
}

// max_dt of simulate_to_time (src/simulator.jl:199-203).
__device__ __forceinline__ double loop_max_dt(int match_endtime, double endtime, double t, int has_max_ts,
                                              double max_ts) {
  double max_dt = match_endtime ? endtime - t : __longlong_as_double(0x7ff0000000000000ll);
  if (has_max_ts) max_dt = jmin<double>(max_dt, max_ts);
  return max_dt;
}

// dt and time bookkeeping of the step of this parity.
template <typename T>
__device__ __forceinline__ double step_dt(const Geom<T>& g, const StepRecord* rec, int parity) {
  if (rec->force_dt) return rec->forced_dt;
  const double ax = speed_from_key<T>(rec->speed_bits[parity][0]);
  const double ay = speed_from_key<T>(rec->speed_bits[parity][1]);
  const double max_dt = rec->explicit_mode
                            ? rec->explicit_max_dt
                            : loop_max_dt(rec->match_endtime, rec->endtime, rec->t[parity], rec->has_max_ts,
                                          rec->max_ts);
  return cfl_dt<T>(g, ax, ay, max_dt);
}

template <typename T>
__device__ __forceinline__ void advance_record(StepRecord* rec, int parity, double dt) {
  const double tn = next_time<T>(rec->t[parity], dt);
  rec->last_dt = dt;
  rec->t[parity ^ 1] = tn;
  const long long done = rec->n_done + 1;
  rec->n_done = done;
  const bool still = rec->stop_stalled && tn == rec->t[parity];
  if (still) rec->stalled = 1;
  const bool more = !rec->explicit_mode && (tn < rec->endtime) && !(tn + dt >= rec->stop_time) &&
                    !(rec->max_steps > 0 && done >= rec->max_steps) && !still;
  rec->active[parity ^ 1] = more ? 1 : 0;
  rec->speed_bits[parity ^ 1][0] = 0ull;
  rec->speed_bits[parity ^ 1][1] = 0ull;
}

__device__ __forceinline__ void carry_record(StepRecord* rec, int parity) {
  rec->t[parity ^ 1] = rec->t[parity];
  rec->active[parity ^ 1] = 0;
}

// Ghosts written by the owner of each boundary source cell: wall mirrors
// (src/bc.jl:81-110; x ghosts negate hu, y ghosts hv) or periodic copies
// (src/bc.jl:29-40). Corner ghosts are never written, as in the reference.
// INTERIOR = false: the ghost copies only (the cell itself is stored elsewhere).
template <typename T, bool INTERIOR = true>
__device__ __forceinline__ void store_with_ghosts(const Geom<T>& g, T* __restrict__ Uo, int gx, int gy, T w, T hu,
                                                  T hv) {
  if constexpr (INTERIOR) {
    const long long o = sidx(g, gx, gy);
    Uo[o] = w;
    Uo[g.PS + o] = hu;
    Uo[2 * g.PS + o] = hv;
  }
  int gxs[2] = {-1, -1}, gys[2] = {-1, -1};
  const T sx = g.bc == 1 ? (T)-1 : (T)1;  // normal momentum sign across a ghost
  if (g.bc == 2) {
    if (gx < 2 * g.gc) gxs[0] = gx + g.nx;
    if (gx >= g.nx) gxs[1] = gx - g.nx;
    if (gy < 2 * g.gc) gys[0] = gy + g.ny;
    if (gy >= g.ny) gys[1] = gy - g.ny;
  } else if (g.bc == 3) {  // Neumann: left mirror, bottom from the top rows
    const int lo = g.gc;
    if (gx == lo) gxs[0] = lo - 1;
    if (gx == lo + 1) gxs[0] = lo - 2;
    if (gy >= g.ny) gys[1] = gy - g.ny;
  } else {
    const int lo = g.gc, hi = g.gc + g.nx - 1;
    if (gx == lo) gxs[0] = lo - 1;
    if (gx == lo + 1) gxs[0] = lo - 2;
    if (gx == hi) gxs[1] = hi + 1;
    if (gx == hi - 1) gxs[1] = hi + 2;
    const int ylo = g.gc, yhi = g.gc + g.ny - 1;
    if (gy == ylo) gys[0] = ylo - 1;
    if (gy == ylo + 1) gys[0] = ylo - 2;
    if (gy == yhi) gys[1] = yhi + 1;
    if (gy == yhi - 1) gys[1] = yhi + 2;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (gxs[i] >= 0) {
      const long long q = sidx(g, gxs[i], gy);
      Uo[q] = w;
      Uo[g.PS + q] = sx * hu;
      Uo[2 * g.PS + q] = hv;
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (gys[i] >= 0) {
      const long long q = sidx(g, gx, gys[i]);
      Uo[q] = w;
      Uo[g.PS + q] = hu;
      Uo[2 * g.PS + q] = sx * hv;
    }
  }
}

// Stage-1 pointwise update of one cell: Euler, friction, dry clamp.
// src/timestepper/rungekutta.jl:39-41, src/friction.jl:77,80-84,
// src/timestepper/timestepper.jl:41-51.
template <typename T>
__device__ __forceinline__ void stage1_point(const Phys<T>& p, T tdt, T u0, T u1, T u2, T l0, T l1, T l2, T S, T Bc,
                                             T& w, T& hu, T& hv) {
  w = u0 + tdt * l0;
  hu = u1 + tdt * l1;
  hv = u2 + tdt * l2;
  if (p.friction) apply_friction<T>(tdt, S, hu, hv);
  dry_clamp<T>(p, w, hu, hv, Bc);
}

// NeumannBC's right and top ghosts (src/bc.jl:53,58 copy ghost onto ghost):
// the outer ghost of a row or column evolves by the all-cell passes alone --
// no flux, its rain and infiltration, its own friction and dry clamp -- and
// the boundary update copies it onto the inner ghost. (x, y) is the outer
// ghost; its stage-1 value, and with rk2 its stage-2 value, is written to it
// and to the inner ghost (x-1, y) or (x, y-1). scal holds point_scalars().
template <typename T, bool CG>
__device__ __forceinline__ void neumann_u1(const Geom<T>& g, const Phys<T>& p, T tdt, const T* U0,
                                           const T* __restrict__ B, const T* scal, int x, int y, T& w, T& hu, T& hv,
                                           T& a0, T& a1, T& a2, T& lpt, T& Bc) {
  const long long o = sidx(g, x, y);
  Bc = g.bconst;
  if (!g.bottom_const) {
    const long long b = (long long)y * g.PB + x + XOFF;
    Bc = (T)0.25 * (((B[b] + B[b + 1]) + B[b + g.PB]) + B[b + g.PB + 1]);
  }
  a0 = gld<CG>(U0 + o);
  a1 = gld<CG>(U0 + g.PS + o);
  a2 = gld<CG>(U0 + 2 * g.PS + o);
  lpt = p.any_dynamic ? add_point_sources<T>(p, (T)0, scal, o) : add_point_sources<T>(p, (T)0);
  T S = (T)0;
  if (p.friction && friction_active<T>(a1, a2)) S = friction_factor<T>(p, a0, a1, a2, Bc);
  stage1_point<T>(p, tdt, a0, a1, a2, lpt, (T)0, (T)0, S, Bc, w, hu, hv);
}

template <typename T, bool CG>
__device__ __forceinline__ void neumann_outer(const Geom<T>& g, const Phys<T>& p, T tdt, const T* U0,
                                              const T* __restrict__ B, const T* scal, int x, int y, int axis, bool rk2,
                                              T* Uo) {
  T w, hu, hv, a0, a1, a2, lpt, Bc;
  neumann_u1<T, CG>(g, p, tdt, U0, B, scal, x, y, w, hu, hv, a0, a1, a2, lpt, Bc);
  if (rk2) {  // src/timestepper/rungekutta.jl:42-50 on the ghost
    const T v0 = w, v1 = hu, v2 = hv;
    w = v0 + tdt * lpt;
    hu = v1 + tdt * (T)0;
    hv = v2 + tdt * (T)0;
    w = (T)0.5 * (a0 + w);
    hu = (T)0.5 * (a1 + hu);
    hv = (T)0.5 * (a2 + hv);
    if (p.friction && friction_active<T>(v1, v2)) apply_friction<T>(tdt, friction_factor<T>(p, v0, v1, v2, Bc), hu, hv);
    dry_clamp<T>(p, w, hu, hv, Bc);
  }
  const long long q0 = sidx(g, x, y);
  const long long q1 = axis == 0 ? sidx(g, x - 1, y) : sidx(g, x, y - 1);
  Uo[q0] = w;
  Uo[g.PS + q0] = hu;
  Uo[2 * g.PS + q0] = hv;
  Uo[q1] = w;
  Uo[g.PS + q1] = hu;
  Uo[2 * g.PS + q1] = hv;
}

// ---------------------------------------------------------------------------
// RK2 stage pass.
// L, R and F come first and are contiguous: before the stage-2 derivative
// overwrites them they hold the TMA-staged halo tiles of U0 (3 planes) and L
// (3), planes of HX x HY from offset 0; S is staged in the first plane of U1
// (k_stage2_tma). For Float64 every TMA destination starts 128-byte aligned.
template <typename T, typename S = BigTile>
struct SmemStage {
  T L[S::DIRS * 3 * S::LRN];
  T R[S::DIRS * 3 * S::LRN];
  T F[S::DIRS * 3 * S::FN];
  T U1[3 * S::HX * S::HY];
  T U0[3 * S::TX * S::TY];
  T B[S::BHX * S::BHY];
  double dt;
  T scal[kScalars];
  unsigned long long bar;  // mbarrier of the tile copies
  int plain;               // 0: staged by TMA; 1: not staged (alignment); 2: the wait gave up
};
using TmaTile = SmallTile;
static_assert(6 * TmaTile::LRN + 3 * TmaTile::FN >= 6 * TmaTile::HX * TmaTile::HY,
              "the staged planes of U0 and L must fit in L, R, F");

// RK2 stage pass over one tile at (x0, y0) (block-collective): U2 with its
// ghosts into Uo. dt is the step's dt, t its start time.
// STAGED: the halo tiles of U0 and L sit at the start of s (planes of HX x HY:
// U0 0..2, L 3..5), that of S in s.U1, and s.B holds the corners (TMA); the interior of U2
// goes to s.U0 (in place: each thread overwrites the cells it read) for a
// tensor store by the caller, its ghost copies straight to Uo.
template <typename T, bool CG, bool STAGED = false, typename S = BigTile>
__device__ __forceinline__ void stage2_tile(const Geom<T>& g, const Phys<T>& p, const T* U0, const T* __restrict__ B,
                                            const T* Lin, const T* Sin, T* Uo, int x0, int y0, SmemStage<T, S>& s,
                                            double dt, double t) {
  constexpr int TX = S::TX, TY = S::TY, NT = S::NT, CPT = S::CPT, HX = S::HX, HY = S::HY;
  const int tid = threadIdx.x;
  const int nvx = min(TX, g.gc + g.nx - x0), nvy = min(TY, g.gc + g.ny - y0);
  if (p.any_dynamic && tid == 1) point_scalars<T>(p, t, s.scal);
  if (!STAGED && !g.bottom_const) load_corners<S>(g, B, s.B, x0, y0);
  __syncthreads();
  const T* stg = s.L;  // staged planes (STAGED only)
  const T tdt = (T)dt;
  BTile<T, S> bt{s.B, g.bottom_const, g.bconst};

  // U1 on tile + halo, from U0, L, S. Ghost cells take U1 of their boundary
  // source cell (src/bc.jl:29-40, 81-110), computed the same pointwise way;
  // corner ghosts are never read and stay zero.
  for (int idx = tid; idx < HX * HY; idx += NT) {
    const int lx = idx % HX - 2, ly = idx / HX - 2;
    const int gx = x0 + lx, gy = y0 + ly;
    const bool xin = gx >= g.gc && gx < g.gc + g.nx;
    const bool yin = gy >= g.gc && gy < g.gc + g.ny;
    T w = (T)0, hu = (T)0, hv = (T)0;
    if (xin && yin) {
      T a0, a1, a2, l0, l1, l2, fr;
      if constexpr (STAGED) {
        constexpr int A = HX * HY;
        a0 = stg[idx];
        a1 = stg[A + idx];
        a2 = stg[2 * A + idx];
        l0 = stg[3 * A + idx];
        l1 = stg[4 * A + idx];
        l2 = stg[5 * A + idx];
        fr = p.friction ? s.U1[idx] : (T)0;  // this thread writes U1[idx] below
      } else {
        const long long o = sidx(g, gx, gy);
        a0 = gld<CG>(U0 + o);
        a1 = gld<CG>(U0 + g.PS + o);
        a2 = gld<CG>(U0 + 2 * g.PS + o);
        l0 = gld<CG>(Lin + o);
        l1 = gld<CG>(Lin + g.PS + o);
        l2 = gld<CG>(Lin + 2 * g.PS + o);
        fr = p.friction ? gld<CG>(Sin + o) : (T)0;
      }
      stage1_point<T>(p, tdt, a0, a1, a2, l0, l1, l2, fr, bt.cell(lx, ly), w, hu, hv);
      if (lx >= 0 && lx < TX && ly >= 0 && ly < TY) {
        const int t = ly * TX + lx;
        s.U0[t] = a0;
        s.U0[TX * TY + t] = a1;
        s.U0[2 * TX * TY + t] = a2;
      }
    } else if (yin && gx < g.N1) {
      if (g.bc == 3 && gx >= g.gc + g.nx) {
        T a0, a1, a2, lpt, Bg;
        neumann_u1<T, CG>(g, p, tdt, U0, B, s.scal, g.N1 - 1, gy, w, hu, hv, a0, a1, a2, lpt, Bg);
      } else {
        u1_global<T, CG>(g, p, tdt, U0, Lin, Sin, B, bc_source(gx, g.gc, g.nx, g.bc, 0), gy, w, hu, hv);
        if (g.bc == 1) hu = -hu;
      }
    } else if (xin && gy < g.N2) {
      if (g.bc == 3 && gy >= g.gc + g.ny) {
        T a0, a1, a2, lpt, Bg;
        neumann_u1<T, CG>(g, p, tdt, U0, B, s.scal, gx, g.N2 - 1, w, hu, hv, a0, a1, a2, lpt, Bg);
      } else {
        u1_global<T, CG>(g, p, tdt, U0, Lin, Sin, B, gx, bc_source(gy, g.gc, g.ny, g.bc, 1), w, hu, hv);
        if (g.bc == 1) hv = -hv;
      }
    }
    s.U1[idx] = w;
    s.U1[HX * HY + idx] = hu;
    s.U1[2 * HX * HY + idx] = hv;
  }
  __syncthreads();

  T acc[CPT][3];
  T mx = (T)0, my = (T)0;
  tile_derivative<S, T, false>(p, s.U1, bt, s.L, s.R, s.F, acc, mx, my, nvx, nvy);

#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const int c = tid + k * NT;
    const int lx = c % TX, ly = c / TX;
    if (lx >= nvx || ly >= nvy) continue;
    const long long o = sidx(g, x0 + lx, y0 + ly);
    acc[k][0] = p.any_dynamic ? add_point_sources<T>(p, acc[k][0], s.scal, o) : add_point_sources<T>(p, acc[k][0]);
    const int ci = (ly + 2) * HX + lx + 2;
    const T v0 = s.U1[ci], v1 = s.U1[HX * HY + ci], v2 = s.U1[2 * HX * HY + ci];
    T w = v0 + tdt * acc[k][0];
    T hu = v1 + tdt * acc[k][1];
    T hv = v2 + tdt * acc[k][2];
    w = halve<T>(s.U0[c] + w);
    hu = halve<T>(s.U0[TX * TY + c] + hu);
    hv = halve<T>(s.U0[2 * TX * TY + c] + hv);
    const T Bc = bt.cell(lx, ly);
    if (p.friction && friction_active<T>(v1, v2)) apply_friction<T>(tdt, friction_factor<T>(p, v0, v1, v2, Bc), hu, hv);
    dry_clamp<T>(p, w, hu, hv, Bc);
    if (STAGED && x0 + lx + XOFF < tma_store_cols(XOFF + g.gc + g.nx)) {
      s.U0[c] = w;  // stored by the tile's tensor store
      s.U0[TX * TY + c] = hu;
      s.U0[2 * TX * TY + c] = hv;
      store_with_ghosts<T, false>(g, Uo, x0 + lx, y0 + ly, w, hu, hv);
    } else {
      store_with_ghosts<T>(g, Uo, x0 + lx, y0 + ly, w, hu, hv);
    }
    if (g.bc == 3) {
      if (x0 + lx == g.gc + g.nx - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, s.scal, g.N1 - 1, y0 + ly, 0, true, Uo);
      if (y0 + ly == g.gc + g.ny - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, s.scal, x0 + lx, g.N2 - 1, 1, true, Uo);
    }
  }
}

template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB) k_stage2(Geom<T> g, Phys<T> p, const T* __restrict__ U0, const T* __restrict__ B,
                                               const T* __restrict__ Lin, const T* __restrict__ Sin, T* __restrict__ Uo,
                                               StepRecord* rec, int parity) {
  const bool root = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
  if (!rec->active[parity]) {
    if (root) carry_record(rec, parity);
    return;
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemStage<T, S>& s = *reinterpret_cast<SmemStage<T, S>*>(smem_raw);
  const int x0 = g.gc + blockIdx.x * S::TX, y0 = g.gc + blockIdx.y * S::TY;
  if (threadIdx.x == 0) s.dt = step_dt<T>(g, rec, parity);
  __syncthreads();
  const double dt = s.dt;
  stage2_tile<T, false, false, S>(g, p, U0, B, Lin, Sin, Uo, x0, y0, s, dt, rec->t[parity]);
  if (root) advance_record<T>(rec, parity, dt);
}

// k_stage2 with the halo tiles of U0, L, S and the corners staged by TMA
// (Float64): three or four copies on one mbarrier, issued by thread 0.
template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB)
    k_stage2_tma(Geom<T> g, Phys<T> p, const __grid_constant__ CUtensorMap mU, const __grid_constant__ CUtensorMap mL,
                 const __grid_constant__ CUtensorMap mS, const __grid_constant__ CUtensorMap mB,
                 const __grid_constant__ CUtensorMap mUo,
                 const T* __restrict__ U0, const T* __restrict__ B, const T* __restrict__ Lin,
                 const T* __restrict__ Sin, T* __restrict__ Uo, StepRecord* rec, int parity) {
  static_assert(sizeof(T) == 8, "TMA tiles are Float64 (the tile origin is 16-byte aligned only for 8-byte cells)");
  const bool root = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
  if (!rec->active[parity]) {
    if (root) carry_record(rec, parity);
    return;
  }
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemStage<T, S>& s = *reinterpret_cast<SmemStage<T, S>*>(smem_raw);
  const int x0 = g.gc + blockIdx.x * S::TX, y0 = g.gc + blockIdx.y * S::TY;
  const int cx = x0 - 2 + XOFF, cy = y0 - 2;
  if (threadIdx.x == 0) {
    constexpr int A = S::HX * S::HY;
    T* stg = s.L;
    const bool ok = tma_ok(cx, (int)sizeof(T), stg) && tma_ok(cx, (int)sizeof(T), stg + 3 * A) &&
                    tma_ok(cx, (int)sizeof(T), s.U1) && (g.bottom_const || tma_ok(cx, (int)sizeof(T), s.B)) &&
                    tma_ok(x0 + XOFF, (int)sizeof(T), s.U0);
    s.plain = ok ? 0 : 1;
    if (ok) {
      mbar_init(&s.bar, 1);
      mbar_expect_tx(&s.bar, tile_bytes<T, S>(6) + (p.friction ? tile_bytes<T, S>(1) : 0u) +
                                 (g.bottom_const ? 0u : corner_bytes<T, S>()));
      tma_load_3d(stg, &mU, cx, cy, 0, &s.bar);
      tma_load_3d(stg + 3 * A, &mL, cx, cy, 0, &s.bar);
      if (p.friction) tma_load_2d(s.U1, &mS, cx, cy, &s.bar);
      if (!g.bottom_const) tma_load_2d(s.B, &mB, cx, cy, &s.bar);
    }
    s.dt = step_dt<T>(g, rec, parity);
  }
  __syncthreads();
  if (!s.plain && !mbar_wait_bounded(&s.bar, 0)) {
    rec->wait_fault = 1;
    s.plain = 2;  // gave up
  }
  __syncthreads();
  const double dt = s.dt;
  if (s.plain) {
    stage2_tile<T, false, false, S>(g, p, U0, B, Lin, Sin, Uo, x0, y0, s, dt, rec->t[parity]);
  } else {
    stage2_tile<T, false, true, S>(g, p, U0, B, Lin, Sin, Uo, x0, y0, s, dt, rec->t[parity]);
    // The interior tile from s.U0 (128-byte aligned, x0 + XOFF even) in one tensor store.
    fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      tma_store_3d(&mUo, s.U0, x0 + XOFF, y0, 0);
      bulk_commit();
      bulk_wait_all();
    }
  }
  if (root) advance_record<T>(rec, parity, dt);
  if (s.plain == 2 && threadIdx.x == 0) mbar_wait_bounded(&s.bar, 0);  // a late copy lands before exit
}

// ---------------------------------------------------------------------------
// Forward-Euler apply pass: U1 = clamp((U0 + dt*L) ./ (1 .- dt*[0,S,S])).
// Forward-Euler apply over one tile at (x0, y0): the pointwise stage-1 update.
// NEU: NeumannBC as well, whose isolated ghosts (friction included) would hold
// every other kernel to a third of its threads: 154 instead of 40 registers.
template <typename T, bool CG, bool NEU = true>
__device__ __forceinline__ void apply_fe_tile(const Geom<T>& g, const Phys<T>& p, const T* U0,
                                              const T* __restrict__ B, const T* Lin, const T* Sin, T* Uo, int x0,
                                              int y0, double dt, double t) {
  const T tdt = (T)dt;
  const int lx = threadIdx.x % TX, ly0 = threadIdx.x / TX;
  for (int ly = ly0; ly < TY; ly += NT / TX) {
    const int gx = x0 + lx, gy = y0 + ly;
    if (gx >= g.gc + g.nx || gy >= g.gc + g.ny) continue;
    const long long o = sidx(g, gx, gy);
    T Bc = g.bconst;
    if (!g.bottom_const) {
      const long long b = (long long)gy * g.PB + gx + XOFF;
      Bc = (T)0.25 * (((B[b] + B[b + 1]) + B[b + g.PB]) + B[b + g.PB + 1]);
    }
    const T S = p.friction ? gld<CG>(Sin + o) : (T)0;
    T w, hu, hv;
    stage1_point<T>(p, tdt, gld<CG>(U0 + o), gld<CG>(U0 + g.PS + o), gld<CG>(U0 + 2 * g.PS + o), gld<CG>(Lin + o),
                    gld<CG>(Lin + g.PS + o), gld<CG>(Lin + 2 * g.PS + o), S, Bc, w, hu, hv);
    store_with_ghosts<T>(g, Uo, gx, gy, w, hu, hv);
    if (NEU && g.bc == 3 && (gx == g.gc + g.nx - 1 || gy == g.gc + g.ny - 1)) {
      T scal[kScalars];
      if (p.any_dynamic) point_scalars<T>(p, t, scal);
      if (gx == g.gc + g.nx - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, scal, g.N1 - 1, gy, 0, false, Uo);
      if (gy == g.gc + g.ny - 1) neumann_outer<T, CG>(g, p, tdt, U0, B, scal, gx, g.N2 - 1, 1, false, Uo);
    }
  }
}

template <typename T, bool NEU>
__global__ void __launch_bounds__(NT) k_apply_fe(Geom<T> g, Phys<T> p, const T* __restrict__ U0,
                                                 const T* __restrict__ B, const T* __restrict__ Lin,
                                                 const T* __restrict__ Sin, T* __restrict__ Uo, StepRecord* rec,
                                                 int parity) {
  const bool root = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
  if (!rec->active[parity]) {
    if (root) carry_record(rec, parity);
    return;
  }
  __shared__ double sdt;
  if (threadIdx.x == 0) sdt = step_dt<T>(g, rec, parity);
  __syncthreads();
  const double dt = sdt;
  apply_fe_tile<T, false, NEU>(g, p, U0, B, Lin, Sin, Uo, g.gc + blockIdx.x * TX, g.gc + blockIdx.y * TY, dt,
                          rec->t[parity]);
  if (root) advance_record<T>(rec, parity, dt);
}

// Boundary update of a whole volume (after uploads): wall, src/bc.jl:81-110,
// periodic, src/bc.jl:29-40, or Neumann, src/bc.jl:49-60 (right and top: the
// inner ghost takes the outer ghost's value). Ghost columns at interior rows,
// ghost rows at interior columns; corners untouched.
template <typename T>
__global__ void k_bc(Geom<T> g, T* __restrict__ U) {
  const int n_x = g.ny * 2 * g.gc;
  const int n_y = g.nx * 2 * g.gc;
  const T sgn = g.bc == 1 ? (T)-1 : (T)1;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n_x + n_y; idx += gridDim.x * blockDim.x) {
    if (idx < n_x) {
      const int j = g.gc + idx / (2 * g.gc), r = idx % (2 * g.gc);
      const int gx = r < g.gc ? r : g.gc + g.nx + (r - g.gc);
      if (g.bc == 3 && gx >= g.gc + g.nx) {
        if (gx == g.N1 - 2) {
          const long long d = sidx(g, gx, j), sI = sidx(g, g.N1 - 1, j);
          U[d] = U[sI];
          U[g.PS + d] = U[g.PS + sI];
          U[2 * g.PS + d] = U[2 * g.PS + sI];
        }
        continue;
      }
      const int sx = bc_source(gx, g.gc, g.nx, g.bc, 0);
      const long long d = sidx(g, gx, j), sI = sidx(g, sx, j);
      U[d] = U[sI];
      U[g.PS + d] = sgn * U[g.PS + sI];
      U[2 * g.PS + d] = U[2 * g.PS + sI];
    } else {
      const int q = idx - n_x;
      const int i = g.gc + q / (2 * g.gc), r = q % (2 * g.gc);
      const int gy = r < g.gc ? r : g.gc + g.ny + (r - g.gc);
      if (g.bc == 3 && gy >= g.gc + g.ny) {
        if (gy == g.N2 - 2) {
          const long long d = sidx(g, i, gy), sI = sidx(g, i, g.N2 - 1);
          U[d] = U[sI];
          U[g.PS + d] = U[g.PS + sI];
          U[2 * g.PS + d] = U[2 * g.PS + sI];
        }
        continue;
      }
      const int sy = bc_source(gy, g.gc, g.ny, g.bc, 1);
      const long long d = sidx(g, i, gy), sI = sidx(g, i, sy);
      U[d] = U[sI];
      U[g.PS + d] = U[g.PS + sI];
      U[2 * g.PS + d] = sgn * U[2 * g.PS + sI];
    }
  }
}

// State of n interior cells (0-based (i, j) pairs) gathered into out[3][n].
template <typename T>
__global__ void k_sample(Geom<T> g, const T* __restrict__ U, const int* __restrict__ ij, int n, T* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const long long o = sidx(g, g.gc + ij[k], g.gc + ij[n + k]);
  out[k] = U[o];
  out[n + k] = U[g.PS + o];
  out[2 * n + k] = U[2 * g.PS + o];
}

// Water volume sum((w - B_cell) * dx * dy) over the interior, in Float64:
// per-block partial sums in a fixed order, then one block sums the partials.
template <typename T>
__global__ void k_volume_partial(Geom<T> g, const T* __restrict__ U, const T* __restrict__ B, double* partial) {
  __shared__ double red[NT];
  double acc = 0.0;
  const long long n = (long long)g.nx * g.ny;
  for (long long c = (long long)blockIdx.x * NT + threadIdx.x; c < n; c += (long long)gridDim.x * NT) {
    const int i = g.gc + (int)(c % g.nx), j = g.gc + (int)(c / g.nx);
    double Bc = (double)g.bconst;
    if (!g.bottom_const) {
      const long long b = (long long)j * g.PB + i + XOFF;
      Bc = (double)((T)0.25 * (((B[b] + B[b + 1]) + B[b + g.PB]) + B[b + g.PB + 1]));
    }
    acc += ((double)U[sidx(g, i, j)] - Bc) * g.dx * g.dy;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}



}  // namespace vf
