// vf_adjoint.cuh -- reverse (adjoint) kernels of one RK2 step with a frozen dt.
//
// For a loss of the final state, the reverse sweep carries lambda = dLoss/dU
// backwards through every step and accumulates dLoss/dB (bottom corners) and
// dLoss/dCz (friction coefficient). One step is reversed stage by stage, each
// stage in four launches that read the recomputed forward data:
//   k_adj_point   the stage's pointwise part in reverse: dry clamp, implicit
//                 friction, RK2 average, Euler update; gives lambda of L (the
//                 stage's time derivative) and the direct lambda of the stage
//                 input;
//   k_adj_face    per face of both directions: lambda of the two face values
//                 from the lambda of the central-upwind flux through it;
//   k_adj_recon   per cell of both directions: the bottom source and the minmod
//                 reconstruction in reverse, split into contributions to the
//                 cell and its two neighbours;
//   k_adj_gather  lambda of the stage input per interior cell: the direct part
//                 plus the neighbour contributions, with the lambda of wall
//                 ghost cells folded onto the interior cells they mirror; and,
//                 in the same launch, dLoss/dB per corner from the B_cell and
//                 face-bottom parts.
// The flux and the friction law are reversed by hand, statement by statement:
// values come from the forward kernels' own expressions (vf_math.cuh), so every
// branch is the forward pass's, and the derivatives follow the branch taken
// (the subgradient at kinks: minmod switches, dry faces, the dry clamp). A face
// costs one forward evaluation and about as many FP64 instructions again for
// its six derivatives; evaluating it on dual numbers took six forward
// evaluations per cell and direction, each about twice a plain one (160x128
// cells, Float64: 113 + 119 us per stage for the two directions, 59 us for the
// pointwise part with its five dual friction factors, all at ~87% of the FP64
// pipe). Gathers instead of atomics keep the sums in a fixed order: the
// gradient is deterministic.
// A face or cell none of whose incoming lambda is nonzero passes on zeros
// without evaluating anything: a gauge loss reaches two cells further per stage.
#pragma once
#include "vf_kernels.cuh"

namespace vf {

// Which operand the forward kernels' max/min returned (also for equal values),
// so the derivative follows the same operand.
template <typename T>
__device__ __forceinline__ bool picks_second_max(T x, T y) {
  if constexpr (sizeof(T) == 8) return !(Arith<double>::key(x) > Arith<double>::key(y));
  return !(x >= y);
}
template <typename T>
__device__ __forceinline__ bool picks_second_min(T x, T y) {
  if constexpr (sizeof(T) == 8) return !(Arith<double>::key(x) < Arith<double>::key(y));
  return !(x <= y);
}
template <typename T>
__device__ __forceinline__ T inverse(T x) {
  return Arith<T>::inv(Arith<T>::recip(x));
}
template <typename T>
__device__ __forceinline__ bool all_zero(const T (&v)[3]) {
  return Arith<T>::is_zero(v[0]) && Arith<T>::is_zero(v[1]) && Arith<T>::is_zero(v[2]);
}
// d desingularize(h) / dh: |h| / kappa below kappa, where h* = sign(h) (h^2/(2 kappa) + kappa/2).
template <typename T>
__device__ __forceinline__ T desing_slope(T h, T kappa) {
  return Arith<T>::abs_lt(h, kappa) ? Arith<T>::div(fabs(h), kappa) : (T)1;
}

// ---------------------------------------------------------------------------
template <typename T>
struct AdjArgs {
  Geom<T> g;
  Phys<T> p;
  const T* B;
  double dt;
  int stage2;           // 1: the RK2 second stage (RK2 average with Ubase)
  const T* Uprev;       // the stage's input (friction and Euler update)
  const T* Ubase;       // stage 2: U^n of the RK2 average
  const T* L;           // the stage's time derivative (forward)
  const T* lam_out;     // lambda of the stage's output (interior cells)
  T* lamL;              // lambda of L (interior cells)
  T* lam_direct;        // lambda of Uprev through the pointwise part
  T* lam_base;          // lambda of U^n through the stage-2 average (written by stage 2, read by stage 1)
  T* gBc;               // dLoss/dB_cell per interior cell
  double* gCz_part;     // one running sum per block of k_adj_point
  T* C[2];              // per direction: 9 planes = (to c-1, to c, to c+1) x (w, hu, hv); before that, planes
                        // 0..2 hold lambda of the cell's right face value, 3..5 of its left one
  T* gBf[2];            // per direction: 2 planes (left face bottom, right face bottom) per cell
  T* lam_in;            // gather output: lambda of the stage input
  double* gB;           // dLoss/dB per corner, accumulated
};

template <typename T>
__device__ __forceinline__ T cell_bottom(const Geom<T>& g, const T* __restrict__ B, int x, int y) {
  if (g.bottom_const) return g.bconst;
  const long long b = (long long)y * g.PB + x + XOFF;
  return (T)0.25 * (((B[b] + B[b + 1]) + B[b + g.PB]) + B[b + g.PB + 1]);
}

// Stage pointwise part in reverse (one interior cell per thread). Bound by one
// cell's chain of FP64 operations on small grids and by the FP64 pipe on large
// ones; blocks of 32 x kPointRows cells reach all SMs early (160x128 cells: 17.5 us
// a launch in 80 blocks of 32 x 8, 14.6 us in 320).
constexpr int kPointRows = 2;
__host__ __device__ inline int adj_point_blocks(int nx, int ny) {
  return ((nx + 31) / 32) * ((ny + kPointRows - 1) / kPointRows);
}
template <typename T>
__global__ void __launch_bounds__(32 * kPointRows) k_adj_point(AdjArgs<T> a) {
  using A = Arith<T>;
  __shared__ double red[32 * kPointRows];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int columns = (a.g.nx + 31) / 32;  // of blocks; the grid is one-dimensional
  const int x = a.g.gc + (int)(blockIdx.x % columns) * 32 + threadIdx.x;
  const int y = a.g.gc + (int)(blockIdx.x / columns) * kPointRows + threadIdx.y;
  double gcz = 0.0;
  if (x < a.g.gc + a.g.nx && y < a.g.gc + a.g.ny) {
    const Geom<T>& g = a.g;
    const Phys<T>& p = a.p;
    const long long o = sidx(g, x, y);
    const T tdt = (T)a.dt;
    const T Bc = cell_bottom(g, a.B, x, y);
    const T q0 = a.Uprev[o], q1 = a.Uprev[g.PS + o], q2 = a.Uprev[2 * g.PS + o];
    const T l0 = a.L[o], l1 = a.L[g.PS + o], l2 = a.L[2 * g.PS + o];
    // forward, as stage1_point / the stage-2 epilogue compute it
    T w = q0 + tdt * l0, hu = q1 + tdt * l1, hv = q2 + tdt * l2;
    T b0 = 0, b1 = 0, b2 = 0;
    if (a.stage2) {
      b0 = a.Ubase[o];
      b1 = a.Ubase[g.PS + o];
      b2 = a.Ubase[2 * g.PS + o];
      w = (T)0.5 * (b0 + w);
      hu = (T)0.5 * (b1 + hu);
      hv = (T)0.5 * (b2 + hv);
    }
    T S = (T)0;
    if (p.friction && friction_active<T>(q1, q2)) S = friction_factor<T>(p, q0, q1, q2, Bc);
    const bool fric = p.friction && !A::is_zero(S);
    T den = (T)1;
    if (fric) {
      den = (T)1 - tdt * S;
      apply_friction<T>(tdt, S, hu, hv);
    }
    // reverse
    T lw = a.lam_out[o], lhu = a.lam_out[g.PS + o], lhv = a.lam_out[2 * g.PS + o];
    T gbc = (T)0;
    if (A::lt(w - Bc, p.cutoff)) {  // dry clamp: (max(w, Bc), 0, 0)
      if (picks_second_max<T>(w, Bc)) {  // Bc kept
        gbc = gbc + lw;
        lw = (T)0;
      }
      lhu = (T)0;
      lhv = (T)0;
    }
    T lq0 = 0, lq1 = 0, lq2 = 0;
    if (fric) {
      // hu_out = huA / den, den = 1 - dt*S(Uprev, Bc, Cz)
      const T lden = -(lhu * hu + lhv * hv) / den;
      lhu = lhu / den;
      lhv = lhv / den;
      const T lS = -tdt * lden;
      // S = -Cz |u| / den_s(h*) with u = (q1, q2) / h*, h* = desingularize(q0 - Bc)
      // (src/friction.jl:30-43,62-78), statement by statement in reverse
      const T h = q0 - Bc;
      const T hs = desing<T>(h, p.kappa);
      T u, v;
      velocities<T>(p, h, hs, q1, q2, u, v);
      const T speed = A::sqrt_(u * u + v * v);
      T ds, dds;  // den_s and its derivative
      if (p.friction == 3) {
        ds = hs * hs;
        dds = (T)2 * hs;
      } else {
        const T cb = vcbrt<T>(hs);
        ds = p.friction == 1 ? cb * hs : cb * hs * hs;
        dds = p.friction == 1 ? cb * (T)(4.0 / 3.0) : cb * hs * (T)(7.0 / 3.0);
      }
      const T lSd = lS * inverse<T>(ds);
      gcz = (double)(-lSd * speed);
      const T lspeed = A::is_zero(speed) ? (T)0 : -lSd * p.Cz * inverse<T>(speed);
      const T lu = lspeed * u, lv = lspeed * v;
      const T ihs = inverse<T>(hs);
      lq1 = lu * ihs;
      lq2 = lv * ihs;
      lq0 = (-(lSd * S) * dds - fma(lq1, u, lq2 * v)) * desing_slope<T>(h, p.kappa);
      gbc = gbc - lq0;
    }
    T lW0 = lw, lW1 = lhu, lW2 = lhv;
    T lb0 = 0, lb1 = 0, lb2 = 0;
    if (a.stage2) {  // out = 0.5*(Ubase + W): half to each
      lW0 = (T)0.5 * lw;
      lW1 = (T)0.5 * lhu;
      lW2 = (T)0.5 * lhv;
      a.lam_base[o] = lW0;
      a.lam_base[g.PS + o] = lW1;
      a.lam_base[2 * g.PS + o] = lW2;
    } else {  // stage 1: its input is U^n, which the stage-2 average saw too
      lb0 = a.lam_base[o];
      lb1 = a.lam_base[g.PS + o];
      lb2 = a.lam_base[2 * g.PS + o];
    }
    a.lamL[o] = tdt * lW0;
    a.lamL[g.PS + o] = tdt * lW1;
    a.lamL[2 * g.PS + o] = tdt * lW2;
    a.lam_direct[o] = (lq0 + lW0) + lb0;
    a.lam_direct[g.PS + o] = (lq1 + lW1) + lb1;
    a.lam_direct[2 * g.PS + o] = (lq2 + lW2) + lb2;
    a.gBc[o] = gbc;
  }
  red[tid] = gcz;
  __syncthreads();
  for (int s = 16 * kPointRows; s > 0; s >>= 1) {
    if (tid < s) red[tid] += red[tid + s];
    __syncthreads();
  }
  if (tid == 0) a.gCz_part[blockIdx.x] += red[0];
}

// Reverse of minmod_slope (src/reconstruction/linearreconstruction.jl:28-43):
// adds d(slope)/d(l, c, r) * ls to (ll, lc, lr), following the operand the
// forward minmod returned.
template <typename T>
__device__ __forceinline__ void minmod_slope_rev(T l, T c, T r, T theta, T ls, T& ll, T& lc, T& lr) {
  using A = Arith<T>;
  const T fwd = r - c, bwd = c - l;
  const T ma = theta * fwd, mb = (fwd + bwd) * (T)0.5, mc = theta * bwd;
  int pick = -1;
  if (A::gt0(ma) && A::gt0(mb) && A::gt0(mc)) {
    const T m1 = A::min(ma, mb);
    const int p1 = (m1 == ma && !picks_second_min<T>(ma, mb)) ? 0 : 1;
    const T m2 = A::min(m1, mc);
    pick = (m2 == m1 && !picks_second_min<T>(m1, mc)) ? p1 : 2;
  } else if (A::lt0(ma) && A::lt0(mb) && A::lt0(mc)) {
    const T m1 = A::max(ma, mb);
    const int p1 = (m1 == ma && !picks_second_max<T>(ma, mb)) ? 0 : 1;
    const T m2 = A::max(m1, mc);
    pick = (m2 == m1 && !picks_second_max<T>(m1, mc)) ? p1 : 2;
  }
  T lf = 0, lb = 0;
  if (pick == 0) lf = theta * ls;
  if (pick == 1) {
    lf = (T)0.5 * ls;
    lb = (T)0.5 * ls;
  }
  if (pick == 2) lb = theta * ls;
  lr = lr + lf;
  lc = lc - lf + lb;
  ll = ll - lb;
}

// One side of a face as side_flux computes it (n: normal, t: transverse).
template <typename T>
struct AdjSide {
  bool wet;
  T h, hs, un, ut, f0, fn, ft, c, e1, e2;
};
template <typename T, int DIR>
__device__ __forceinline__ AdjSide<T> adj_side(const Phys<T>& p, const T (&q)[3]) {
  using A = Arith<T>;
  AdjSide<T> s{};
  s.h = q[0];
  s.wet = A::gt(s.h, p.cutoff);
  if (!s.wet) return s;
  s.hs = desing<T>(s.h, p.kappa);
  T u, v;
  velocities<T>(p, s.h, s.hs, q[1], q[2], u, v);
  s.un = DIR == 0 ? u : v;
  s.ut = DIR == 0 ? v : u;
  s.f0 = (p.rho * s.h) * s.un;
  s.fn = s.f0 * s.un + p.c2 * (s.h * s.h);
  s.ft = s.f0 * s.ut;
  s.c = A::sqrt_(p.g * s.h);
  s.e1 = s.un + s.c;
  s.e2 = s.un - s.c;
  return s;
}
// Adds d(f0, fn, ft, e1, e2)/d(h, hu_n, hu_t) times their lambda to (lh, ln, lt).
template <typename T>
__device__ __forceinline__ void adj_side_rev(const Phys<T>& p, const AdjSide<T>& s, T lf0, T lfn, T lft, T le1, T le2,
                                             T& lh, T& ln, T& lt) {
  if (!s.wet) return;
  const T l0 = fma(lft, s.ut, fma(lfn, s.un, lf0));          // of f0, which fn and ft use
  const T lun = fma(lfn, s.f0, fma(l0, p.rho * s.h, le1 + le2));
  const T lut = lft * s.f0;
  const T ihs = inverse<T>(s.hs);
  const T an = lun * ihs, at = lut * ihs;
  const T lhs = fma(an, s.un, at * s.ut);
  T dh = fma(lfn, (T)2 * p.c2 * s.h, l0 * (p.rho * s.un));
  if (!Arith<T>::is_zero(s.c)) dh = fma(le1 - le2, p.g * ((T)0.5 * inverse<T>(s.c)), dh);
  lh = lh + fma(-lhs, desing_slope<T>(s.h, p.kappa), dh);
  ln = ln + an;
  lt = lt + at;
}

// cu_face in reverse: lambda of the face values m (minus side) and q (plus side)
// from lambda of the flux, all in the order (h, hu, hv). With a+, a- the
// one-sided speeds, d = a+ - a-, N = a+ f(m) - a- f(q):
// F = N/d + (a+ a-)/d (q - m).
template <typename T, int DIR>
__device__ __forceinline__ void face_rev(const Phys<T>& p, const T (&m)[3], const T (&q)[3], const T (&lF)[3],
                                         T (&lm)[3], T (&lq)[3]) {
  using A = Arith<T>;
  constexpr int n = DIR == 0 ? 1 : 2, t = 3 - n;
  const AdjSide<T> M = adj_side<T, DIR>(p, m), Q = adj_side<T, DIR>(p, q);
  const bool ap_m = picks_second_max<T>(Q.e1, M.e1), am_m = picks_second_min<T>(Q.e2, M.e2);
  const T ap1 = ap_m ? M.e1 : Q.e1, am1 = am_m ? M.e2 : Q.e2;
  const bool ap_0 = picks_second_max<T>(ap1, (T)0), am_0 = picks_second_min<T>(am1, (T)0);
  const T ap = ap_0 ? (T)0 : ap1, am = am_0 ? (T)0 : am1;
  const T d = ap - am;
#pragma unroll
  for (int k = 0; k < 3; ++k) lm[k] = lq[k] = (T)0;
  if (A::abs_lt(d, p.kappa)) return;
  const T id = inverse<T>(d);
  const T l0 = lF[0] * id, ln = lF[n] * id, lt = lF[t] * id;  // of N
  const T N0 = fma(ap, M.f0, -(am * Q.f0)), Nn = fma(ap, M.fn, -(am * Q.fn)), Nt = fma(ap, M.ft, -(am * Q.ft));
  const T qa = ap * am * id;
  // of the product a+ a-, and of d through both quotients
  const T lp = fma(l0, q[0] - m[0], fma(ln, q[n] - m[n], lt * (q[t] - m[t])));
  const T ld = -(fma(l0, N0, fma(ln, Nn, lt * Nt)) * id + lp * qa);
  const T lap = fma(l0, M.f0, fma(ln, M.fn, fma(lt, M.ft, fma(lp, am, ld))));
  const T lam = fma(-l0, Q.f0, fma(-ln, Q.fn, fma(-lt, Q.ft, fma(lp, ap, -ld))));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lm[k] = -(lF[k] * qa);
    lq[k] = lF[k] * qa;
  }
  const T z = (T)0;
  adj_side_rev<T>(p, M, ap * l0, ap * ln, ap * lt, !ap_0 && ap_m ? lap : z, !am_0 && am_m ? lam : z, lm[0], lm[n], lm[t]);
  adj_side_rev<T>(p, Q, -(am * l0), -(am * ln), -(am * lt), !ap_0 && !ap_m ? lap : z, !am_0 && !am_m ? lam : z, lq[0],
                  lq[n], lq[t]);
}

// Access along DIR at (al + s, ac): al along, ac across.
template <typename T, int DIR>
struct AdjLine {
  const AdjArgs<T>& a;
  int al, ac, n_al;
  __device__ __forceinline__ int x(int s) const { return DIR == 0 ? al + s : ac; }
  __device__ __forceinline__ int y(int s) const { return DIR == 0 ? ac : al + s; }
  __device__ __forceinline__ void state(int s, T (&u)[3]) const {
    const Geom<T>& g = a.g;
    const bool in = x(s) >= 0 && y(s) >= 0 && x(s) < g.N1 && y(s) < g.N2;
    const long long o = sidx(g, x(s), y(s));
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = in ? a.Uprev[k * g.PS + o] : (T)0;
  }
  __device__ __forceinline__ void lamL(int s, T (&l)[3]) const {  // of L at an interior cell, else 0
    const Geom<T>& g = a.g;
    const bool in = al + s >= g.gc && al + s < g.gc + n_al;
    const long long o = sidx(g, x(s), y(s));
#pragma unroll
    for (int k = 0; k < 3; ++k) l[k] = in ? a.lamL[k * g.PS + o] : (T)0;
  }
  // bottom of the face left of the cell at offset s
  __device__ __forceinline__ T bface(int s) const {
    if (a.g.bottom_const) return a.g.bconst;
    const long long b = (long long)y(s) * a.g.PB + x(s) + XOFF;
    return halve<T>(a.B[b] + (DIR == 0 ? a.B[b + a.g.PB] : a.B[b + 1]));
  }
  __device__ __forceinline__ T bcell(int s) const { return cell_bottom(a.g, a.B, x(s), y(s)); }
  // face values of the cell at offset s, as the forward pass reconstructs them
  __device__ __forceinline__ void faces(int s, const T (&l)[3], const T (&c)[3], const T (&r)[3], T (&L)[3],
                                        T (&R)[3]) const {
    if (a.p.rec_none) no_reconstruction<T>(c, bcell(s), L, R);
    else reconstruct_cell<T>(a.p, l, c, r, bface(s), bface(s + 1), L, R);
  }
};

// Faces along DIR: face f lies between the cells gc-1+f and gc+f, f = 0..n.
template <typename T, int DIR>
__device__ __forceinline__ void adj_face(const AdjArgs<T>& a, int ix, int iy) {
  const Geom<T>& g = a.g;
  const int f = DIR == 0 ? ix : iy, n_al = DIR == 0 ? g.nx : g.ny;
  if (ix >= g.nx + (DIR == 0) || iy >= g.ny + (DIR == 1)) return;
  const AdjLine<T, DIR> c{a, g.gc - 1 + f, g.gc + (DIR == 0 ? iy : ix), n_al};
  T lmc[3], lpc[3], lF[3], lm[3] = {0, 0, 0}, lq[3] = {0, 0, 0};
  c.lamL(0, lmc);
  c.lamL(1, lpc);
  const T inv = DIR == 0 ? a.p.inv_dx : a.p.inv_dy;
#pragma unroll
  for (int k = 0; k < 3; ++k) lF[k] = inv * (lpc[k] - lmc[k]);
  if (!all_zero(lF)) {
    T u0[3], u1[3], u2[3], u3[3], t[3], m[3], q[3];
    c.state(-1, u0);
    c.state(0, u1);
    c.state(1, u2);
    c.state(2, u3);
    c.faces(0, u0, u1, u2, t, m);
    c.faces(1, u1, u2, u3, q, t);
    face_rev<T, DIR>(a.p, m, q, lF, lm, lq);
  }
  const long long om = sidx(g, c.x(0), c.y(0)), oq = sidx(g, c.x(1), c.y(1));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.C[DIR][k * g.PS + om] = lm[k];
    a.C[DIR][(3 + k) * g.PS + oq] = lq[k];
  }
}
// blockIdx.z: direction; threadIdx.x runs along x in both, so loads coalesce.
template <typename T>
__global__ void __launch_bounds__(128) k_adj_face(AdjArgs<T> a) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y * blockDim.y + threadIdx.y;
  if (blockIdx.z == 0) adj_face<T, 0>(a, ix, iy);
  else adj_face<T, 1>(a, ix, iy);
}

// Per cell of the reconstruction range along DIR (the first ghost layer
// included, src/reconstruction/linearreconstruction.jl:60-68), interior across.
template <typename T, int DIR>
__device__ __forceinline__ void adj_recon(const AdjArgs<T>& a, int ix, int iy) {
  using A = Arith<T>;
  const Geom<T>& g = a.g;
  const Phys<T>& p = a.p;
  const int n_al = DIR == 0 ? g.nx : g.ny;
  if (ix >= g.nx + 2 * (DIR == 0) || iy >= g.ny + 2 * (DIR == 1)) return;
  const AdjLine<T, DIR> c{a, g.gc - 1 + (DIR == 0 ? ix : iy), g.gc + (DIR == 0 ? iy : ix), n_al};
  const bool face_r = c.al <= g.gc + n_al - 1;  // face c+1/2 is used
  const bool face_l = c.al >= g.gc;             // face c-1/2 is used
  const long long o = sidx(g, c.x(0), c.y(0));
  T lR[3], lL[3], lam[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lR[k] = face_r ? a.C[DIR][k * g.PS + o] : (T)0;
    lL[k] = face_l ? a.C[DIR][(3 + k) * g.PS + o] : (T)0;
  }
  c.lamL(0, lam);
  T gBl = 0, gBr = 0;
  T lu[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};  // [neighbour -1, 0, +1][component]
  if (!(all_zero(lR) && all_zero(lL) && all_zero(lam))) {
    const T inv = DIR == 0 ? p.inv_dx : p.inv_dy;
    const T Blc = c.bface(0), Brc = c.bface(1);
    T ul[3], uc[3], ur[3], Lc[3], Rc[3];
    c.state(-1, ul);
    c.state(0, uc);
    c.state(1, ur);
    // bottom source of interior cells (src/sourceterms/source_term_bottom.jl:24-41)
    if (face_l && face_r && p.n_bottom > 0) {
      c.faces(0, ul, uc, ur, Lc, Rc);
      const T lk = lam[DIR == 0 ? 1 : 2] * (T)p.n_bottom;
      const T slope = slope_over<T>(Brc - Blc, DIR == 0 ? p.dx : p.dy, inv, DIR == 0 ? p.dx_pow2 : p.dy_pow2);
      const T hmean = (Rc[0] + Lc[0]) * (T)0.5;
      lR[0] = lR[0] + lk * p.neg_g * slope * (T)0.5;
      lL[0] = lL[0] + lk * p.neg_g * slope * (T)0.5;
      const T ldb = lk * p.neg_g * hmean * inv;  // d(dB/Δ)/d(dB) = 1/Δ
      gBr = gBr + ldb;
      gBl = gBl - ldb;
    }
    // reconstruction of cell c in reverse
    if (p.rec_none) {
      // L = R = (w - B_cell, hu, hv): the cell takes both faces' lambda, and
      // d/dB_cell = -(lambda_L.h + lambda_R.h) goes to the corners a quarter
      // each, i.e. half to each face bottom of this direction (whose corners
      // are the cell's, a half each)
#pragma unroll
      for (int k = 0; k < 3; ++k) lu[1][k] = lL[k] + lR[k];
      const T dBc = (T)0 - (lL[0] + lR[0]);
      gBl = gBl + (T)0.5 * dBc;
      gBr = gBr + (T)0.5 * dBc;
    } else {
#pragma unroll
      for (int k = 1; k < 3; ++k) {  // hu, hv: L = c - s/2, R = c + s/2
        lu[1][k] = lL[k] + lR[k];
        const T ls = (T)0.5 * (lR[k] - lL[k]);
        minmod_slope_rev<T>(ul[k], uc[k], ur[k], p.theta, ls, lu[0][k], lu[1][k], lu[2][k]);
      }
      // w with the bottom-limited slope: L0 = (w - s/2) - Bl, R0 = (w + s/2) - Br
      const T w = uc[0];
      const T s0 = minmod_slope<T>(ul[0], uc[0], ur[0], p.theta);
      lu[1][0] = lL[0] + lR[0];
      gBl = gBl - lL[0];
      gBr = gBr - lR[0];
      const T ls = (T)0.5 * (lR[0] - lL[0]);
      if (A::lt(w - (T)0.5 * s0, Blc)) {          // s = 2(w - Bl)
        lu[1][0] = lu[1][0] + (T)2 * ls;
        gBl = gBl - (T)2 * ls;
      } else if (A::lt(w + (T)0.5 * s0, Brc)) {   // s = 2(Br - w)
        lu[1][0] = lu[1][0] - (T)2 * ls;
        gBr = gBr + (T)2 * ls;
      } else {
        minmod_slope_rev<T>(ul[0], uc[0], ur[0], p.theta, ls, lu[0][0], lu[1][0], lu[2][0]);
      }
    }
  }
  T* C = a.C[DIR];
#pragma unroll
  for (int nb = 0; nb < 3; ++nb)
#pragma unroll
    for (int k = 0; k < 3; ++k) C[(nb * 3 + k) * g.PS + o] = lu[nb][k];
  a.gBf[DIR][o] = gBl;
  a.gBf[DIR][g.PS + o] = gBr;
}
template <typename T>
__global__ void __launch_bounds__(128) k_adj_recon(AdjArgs<T> a) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y * blockDim.y + threadIdx.y;
  if (blockIdx.z == 0) adj_recon<T, 0>(a, ix, iy);
  else adj_recon<T, 1>(a, ix, iy);
}

// lambda of the stage input per interior cell: direct part + neighbour
// contributions, with the lambda of wall ghost cells folded onto the interior
// cells they mirror (src/bc.jl:81-110; x ghosts negate hu, y ghosts hv).
template <typename T>
__device__ __forceinline__ void adj_gather(const AdjArgs<T>& a, int x, int y) {
  const Geom<T>& g = a.g;
  if (x >= g.gc + g.nx || y >= g.gc + g.ny) return;
  // contributions landing on cell (xx, yy) from the reconstructions along DIR
  auto land = [&](int dir, int xx, int yy, int k) -> T {
    const int al = dir == 0 ? xx : yy;
    const int n = dir == 0 ? g.nx : g.ny;
    const T* C = a.C[dir];
    T s = 0;
    // from the cell itself (to c), from c-1 (to c+1), from c+1 (to c-1)
    auto in_range = [&](int c) { return c >= g.gc - 1 && c <= g.gc + n; };
    if (in_range(al)) s = s + C[(3 + k) * g.PS + sidx(g, xx, yy)];
    if (in_range(al - 1)) {
      const int px = dir == 0 ? xx - 1 : xx, py = dir == 0 ? yy : yy - 1;
      s = s + C[(6 + k) * g.PS + sidx(g, px, py)];
    }
    if (in_range(al + 1)) {
      const int px = dir == 0 ? xx + 1 : xx, py = dir == 0 ? yy : yy + 1;
      s = s + C[(0 + k) * g.PS + sidx(g, px, py)];
    }
    return s;
  };
  const long long o = sidx(g, x, y);
  T lam[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) lam[k] = a.lam_direct[k * g.PS + o] + land(0, x, y, k) + land(1, x, y, k);
  // ghosts copying this cell: wall ghosts mirror it, x' = 2gc-1-x (left) or
  // 2(gc+nx)-1-x (right), with the normal momentum negated; periodic ghosts
  // repeat it a period away, x' = x + n (right) or x - n (left)
  // (src/bc.jl:29-40, 81-110)
#pragma unroll
  for (int dir = 0; dir < 2; ++dir) {
    const int v = dir == 0 ? x : y;
    const int n = dir == 0 ? g.nx : g.ny;
    int gh[2] = {-1, -1};
    if (g.bc == 2) {
      if (v - n >= 0 && v - n < g.gc) gh[0] = v - n;            // left/bottom ghost
      if (v + n >= g.gc + n && v + n < 2 * g.gc + n) gh[1] = v + n;  // right/top ghost
    } else {
      if (v < 2 * g.gc) gh[0] = 2 * g.gc - 1 - v;                  // left/bottom ghost
      if (v >= g.gc + n - g.gc) gh[1] = 2 * (g.gc + n) - 1 - v;    // right/top ghost
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int q = gh[s];
      if (q < 0 || (q >= g.gc && q < g.gc + n)) continue;
      const int gx = dir == 0 ? q : x, gy = dir == 0 ? y : q;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const T l = land(dir, gx, gy, k);
        const bool normal = g.bc == 1 && ((dir == 0 && k == 1) || (dir == 1 && k == 2));
        lam[k] = lam[k] + (normal ? -l : l);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) a.lam_in[k * g.PS + o] = lam[k];
}

// dLoss/dB per corner (I, J) of the (N1+1) x (N2+1) corner grid.
template <typename T>
__device__ __forceinline__ void adj_corner(const AdjArgs<T>& a, int I, int J) {
  const Geom<T>& g = a.g;
  if (I > g.N1 || J > g.N2) return;
  auto cellv = [&](const T* arr, int cx, int cy) -> double {
    if (cx < 0 || cy < 0 || cx >= g.N1 || cy >= g.N2) return 0.0;
    return (double)arr[sidx(g, cx, cy)];
  };
  auto interior = [&](int cx, int cy) {
    return cx >= g.gc && cx < g.gc + g.nx && cy >= g.gc && cy < g.gc + g.ny;
  };
  double s = 0.0;
  // B_cell of the four cells sharing the corner
  double sc = 0.0;
  for (int dy = -1; dy <= 0; ++dy)
    for (int dx = -1; dx <= 0; ++dx)
      if (interior(I + dx, J + dy)) sc += cellv(a.gBc, I + dx, J + dy);
  s += 0.25 * sc;
  // face bottoms: x faces (left of cell (I, J) and (I, J-1); right of (I-1, J), (I-1, J-1))
  const T* fx = a.gBf[0];
  const T* fy = a.gBf[1];
  double sf = 0.0;
  sf += cellv(fx, I, J) + cellv(fx, I, J - 1);
  sf += cellv(fx + g.PS, I - 1, J) + cellv(fx + g.PS, I - 1, J - 1);
  // y faces (bottom of (I, J), (I-1, J); top of (I, J-1), (I-1, J-1))
  sf += cellv(fy, I, J) + cellv(fy, I - 1, J);
  sf += cellv(fy + g.PS, I, J - 1) + cellv(fy + g.PS, I - 1, J - 1);
  s += 0.5 * sf;
  a.gB[(long long)J * (g.N1 + 1) + I] += s;
}

// blockIdx.z 0: lambda of the stage input; 1: dLoss/dB. Both read what the
// earlier launches of the stage wrote and neither what the other writes.
template <typename T>
__global__ void __launch_bounds__(256) k_adj_gather(AdjArgs<T> a) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y * blockDim.y + threadIdx.y;
  if (blockIdx.z == 0) adj_gather<T>(a, a.g.gc + ix, a.g.gc + iy);
  else adj_corner<T>(a, ix, iy);
}

// The step record of a reversed or recomputed step: dt forced, start time t.
static __global__ void k_adj_record(StepRecord* rec, double dt, double t) {
  StepRecord r = {};
  r.active[0] = 1;
  r.t[0] = t;
  r.explicit_mode = 1;
  r.force_dt = 1;
  r.forced_dt = dt;
  r.wait_fault = rec->wait_fault;  // kept until the host reads the record
  *rec = r;
}

// lambda of the final state from the gauge loss sum_g (w[g] - target[g])^2,
// and the loss, in gauge order (one thread).
template <typename T>
__global__ void k_adj_seed(Geom<T> g, const T* U, T* lam, const int* gi, const int* gj, const double* target, int n,
                           double* loss) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double L = 0.0;
  for (int k = 0; k < n; ++k) {
    const long long o = sidx(g, g.gc + gi[k], g.gc + gj[k]);
    const double d = (double)U[o] - target[k];
    L += d * d;
    lam[o] = (T)((double)lam[o] + 2.0 * d);
  }
  *loss = L;
}

// Sum of the per-block dLoss/dCz sums into *acc, in a fixed order (one block).
static __global__ void k_adj_sum(const double* part, int n, double* acc) {
  __shared__ double red[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) s += part[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *acc = red[0];
}

}  // namespace vf
