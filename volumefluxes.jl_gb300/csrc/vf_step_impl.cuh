// vf_step_impl.cuh -- launcher bodies shared by the per-precision units.
#pragma once
#include "vf_launch.cuh"

namespace vf {

static __global__ void k_volume_final_impl(const double* partial, int n, double* out) {
  __shared__ double red[NT];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += NT) acc += partial[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// Rows per marching segment of the flux and of the stage pass, at most. Shorter
// segments recompute more halo rows (4 per segment) but give the block
// scheduler more, smaller units: measured on the Float32 4096^2 step (ms per
// launch), flux 0.351 / 0.334 / 0.326 / 0.323 / 0.327 at 96 / 64 / 48 / 40 /
// 32 rows, stage 0.534 / 0.474 / 0.460 / 0.454 / 0.449 / 0.451 at 96 / 64 /
// 48 / 32 / 24 / 16 rows (the same bits at every length).
template <typename T> struct MarchSeg {
  static constexpr int flux = 40;
  static constexpr int stage = 24;
};
template <typename T>
cudaError_t configure_impl() {
  cudaError_t e = cudaSuccess;
  if constexpr (sizeof(T) == 4) {  // the Float64 tiles stay within the 48 KB that need no opt-in
    e = cudaFuncSetAttribute(k_flux<T, BigTile>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemFlux<T>));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_stage2<T, BigTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SmemStage<T>));
    if (e != cudaSuccess) return e;
  } else {
    static_assert(sizeof(SmemStage<T, SmallTile>) <= 48 * 1024 && sizeof(SmemStage<T, TinyTile>) <= 48 * 1024, "");
  }
  e = cudaFuncSetAttribute(k_ensemble<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemEns<T>));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_ensemble<T, 1>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if constexpr (sizeof(T) == 4) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ensemble<T, 0>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_ensemble<T, 2>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }
  return e;
}

// Column marching (variants 0 and 2) exists for Float32 only: the Float64
// members run on tiles, where full warps keep the 1/64-rate FP64 pipe busy.
template <typename T, int VAR>
cudaLaunchConfig_t ensemble_config(int n, int csize, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n * csize), 1, 1);
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = VAR == 1 ? sizeof(SmemEns<T>) : 0;  // marching needs none
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <typename T>
cudaError_t launch_ensemble_impl(const EnsItem<T>* items, const int* order, int n, int csize, int variant,
                                 unsigned long long time_limit_ns, cudaStream_t st) {
  cudaLaunchAttribute attr[1];
  if (variant == 0 || variant == 2) {
    if constexpr (sizeof(T) == 8) {
      return cudaErrorInvalidValue;
    } else {
      cudaLaunchConfig_t cfg = ensemble_config<T, 0>(n, csize, st, attr);
      if (variant == 2) return cudaLaunchKernelEx(&cfg, k_ensemble<T, 2>, items, order, csize, time_limit_ns);
      return cudaLaunchKernelEx(&cfg, k_ensemble<T, 0>, items, order, csize, time_limit_ns);
    }
  }
  cudaLaunchConfig_t cfg = ensemble_config<T, 1>(n, csize, st, attr);
  return cudaLaunchKernelEx(&cfg, k_ensemble<T, 1>, items, order, csize, time_limit_ns);
}

template <typename T>
cudaError_t ensemble_max_clusters_impl(int csize, int variant, int* out) {
  cudaLaunchAttribute attr[1];
  if (variant == 0 || variant == 2) {
    if constexpr (sizeof(T) == 8) {
      return cudaErrorInvalidValue;
    } else {
      cudaLaunchConfig_t cfg = ensemble_config<T, 0>(1, csize, nullptr, attr);
      if (variant == 2) return cudaOccupancyMaxActiveClusters(out, k_ensemble<T, 2>, &cfg);
      return cudaOccupancyMaxActiveClusters(out, k_ensemble<T, 0>, &cfg);
    }
  }
  cudaLaunchConfig_t cfg = ensemble_config<T, 1>(1, csize, nullptr, attr);
  return cudaOccupancyMaxActiveClusters(out, k_ensemble<T, 1>, &cfg);
}

// Segment length of one launch: the shortest whose blocks are resident all at
// once, blocks_per_sm on each of the 152 SMs, and at most `longest`. A launch of
// fewer warps is bound by the latency of one warp's rows (1.2 us a row in the flux
// pass, 2 us in the stage pass), one of a second wave by that wave. With 40 and 24
// rows at every size, a 200x120 grid had 24 and 40 warps on the whole GPU: 51 and
// 57 us a pass, 5.6 ms for a request of 40 steps instead of 1.7. us per step with
// segments for 8 / 16 / 28 / 40 warps per SM, the lean form (28 to 32 are resident):
// 997x753 77 / 53 / 49 / 51, 1021x511 - / 48 / 43 / 45, 1500x1100 107 / 91 / 81 / 83,
// 2048^2 193 / 195 / 184 / 186; the general form at 8 / 16 / 24 / 40 (24 are
// resident): 997x753 82 / 58 / 54 / 55, 1500x1100 120 / 105 / 95 / 92. From about
// 2400^2 cells on nothing changes. Launches of `share` simulations at once fill the
// GPU together: each takes its part of the wave, in longer segments that recompute
// fewer halo rows.
template <typename T>
int march_seg(const StepArgs<T>& a, int longest, int blocks_per_sm) {
  const Geom<T>& g = a.g;
  const long long nstrips = (g.nx + MOUT - 1) / MOUT;
  const long long units = 152LL * MWPB * blocks_per_sm / (a.share > 1 ? a.share : 1);
  long long rows = (nstrips * g.ny + units - 1) / units;
  while (rows < longest && nstrips * ((g.ny + rows - 1) / rows) > units) ++rows;
  return (int)(rows < longest ? rows : longest);
}
template <typename T>
int march_blocks(const Geom<T>& g, int seg) {
  const long long units = (long long)((g.nx + MOUT - 1) / MOUT) * ((g.ny + seg - 1) / seg);
  return (int)((units + MWPB - 1) / MWPB);
}

// Index of the handle volume Uin is (0 or 1) when the launch can stage its
// tiles with the handle's tensor maps, else -1.
template <typename T>
int tma_volume(const StepArgs<T>& a, const T* Uin) {
  if constexpr (sizeof(T) != 8) {
    return -1;
  } else {
    if (!a.tma.ok || a.variant != 1 || a.L != a.tma.Lb || a.S != a.tma.Sb || a.B != a.tma.Bb) return -1;
    if (Uin == a.tma.Ub[0]) return 0;
    if (Uin == a.tma.Ub[1]) return 1;
    return -1;
  }
}

template <typename S, typename T>
dim3 tile_grid(const Geom<T>& g) {
  return dim3((g.nx + S::TX - 1) / S::TX, (g.ny + S::TY - 1) / S::TY);
}
// Float64 grids small enough that TinyTile leaves at most kTinyTilesPerSM
// blocks to an SM: measured even with SmallTile at 3.8 (192^2), ahead at 2.1
// (160x128: 47 against 59 us per step), behind at 6.7 (256^2).
constexpr int kTinyTilesPerSM = 3;
template <typename T>
bool tiny_tiles(const Geom<T>& g) {
  const dim3 t = tile_grid<TinyTile>(g);
  return (long long)t.x * t.y <= 152LL * kTinyTilesPerSM;
}
template <typename S, typename T>
cudaError_t launch_flux_tiles(const StepArgs<T>& a, const T* Uin, int parity, cudaStream_t st) {
  k_flux<T, S><<<tile_grid<S>(a.g), S::NT, sizeof(SmemFlux<T, S>), st>>>(a.g, a.p, Uin, a.B, a.L, a.S, a.rec, parity);
  return cudaGetLastError();
}
template <typename S, typename T>
cudaError_t launch_stage_tiles(const StepArgs<T>& a, const T* Uin, T* Uout, int parity, cudaStream_t st) {
  k_stage2<T, S><<<tile_grid<S>(a.g), S::NT, sizeof(SmemStage<T, S>), st>>>(a.g, a.p, Uin, a.B, a.L, a.S, Uout, a.rec,
                                                                            parity);
  return cudaGetLastError();
}

// Calls f(offset type, general form?, bottom kind) with the marching kernels'
// compile-time form of a handle. 32-bit offsets reach 4 GB of one plane (2^30
// Float32 cells); larger grids, and Float64, take 64-bit ones.
template <typename T, typename F>
void with_march_form(const StepArgs<T>& a, F f) {
  using u32 = unsigned;
  using u64 = unsigned long long;
  const bool small = plane_fits_u32<T>(a.g) && !a.far;
  if constexpr (sizeof(T) == 8) {
    if (a.general) f(u64{}, std::true_type{}, std::integral_constant<int, 2>{});
    else f(u64{}, std::false_type{}, std::integral_constant<int, 2>{});
  } else {
    if (!small) f(u64{}, std::true_type{}, std::integral_constant<int, 2>{});
    else if (a.general) f(u32{}, std::true_type{}, std::integral_constant<int, 2>{});
    else if (a.g.bottom_const) f(u32{}, std::false_type{}, std::integral_constant<int, 1>{});
    else f(u32{}, std::false_type{}, std::integral_constant<int, 0>{});
  }
}

template <typename T>
cudaError_t launch_flux_impl(const StepArgs<T>& a, const T* Uin, int parity, cudaStream_t st) {
  if (a.variant == 0) {
    const int seg = march_seg(a, MarchSeg<T>::flux, MarchFluxBlocks<T>::resident);
    with_march_form(a, [&](auto o, auto gen, auto cb) {
      k_flux_march<T, decltype(o), decltype(gen)::value, decltype(cb)::value>
          <<<march_blocks(a.g, seg), MW * MWPB, 0, st>>>(a.g, a.p, Uin, a.B, a.L, a.S, a.rec, parity, seg);
    });
    return cudaGetLastError();
  }
  if constexpr (sizeof(T) == 8) {
    if (tiny_tiles(a.g)) return launch_flux_tiles<TinyTile>(a, Uin, parity, st);
    const int v = tma_volume<T>(a, Uin);
    if (v < 0) return launch_flux_tiles<SmallTile>(a, Uin, parity, st);
    k_flux_tma<T, TmaTile><<<tile_grid<TmaTile>(a.g), TmaTile::NT, sizeof(SmemFlux<T, TmaTile>), st>>>(
        a.g, a.p, a.tma.U[v], a.tma.B, Uin, a.B, a.L, a.S, a.rec, parity);
    return cudaGetLastError();
  } else {
    return launch_flux_tiles<BigTile>(a, Uin, parity, st);
  }
}

template <typename T>
cudaError_t launch_stage_impl(const StepArgs<T>& a, const T* Uin, T* Uout, int parity, cudaStream_t st) {
  if (!a.rk2) {
    if (a.g.bc == 3)
      k_apply_fe<T, true><<<tile_grid<BigTile>(a.g), NT, 0, st>>>(a.g, a.p, Uin, a.B, a.L, a.S, Uout, a.rec, parity);
    else
      k_apply_fe<T, false><<<tile_grid<BigTile>(a.g), NT, 0, st>>>(a.g, a.p, Uin, a.B, a.L, a.S, Uout, a.rec, parity);
    return cudaGetLastError();
  }
  if (a.variant == 0) {
    const int seg = march_seg(a, MarchSeg<T>::stage,
                              a.general ? MarchStageBlocks<T>::resident_general : MarchStageBlocks<T>::resident);
    with_march_form(a, [&](auto o, auto gen, auto cb) {
      k_stage_march<T, decltype(o), decltype(gen)::value, decltype(cb)::value>
          <<<march_blocks(a.g, seg), MW * MWPB, 0, st>>>(a.g, a.p, Uin, a.B, a.L, a.S, Uout, a.rec, parity, seg);
    });
    return cudaGetLastError();
  }
  if constexpr (sizeof(T) == 8) {
    if (tiny_tiles(a.g)) return launch_stage_tiles<TinyTile>(a, Uin, Uout, parity, st);
    const int v = tma_volume<T>(a, Uin);
    if (v < 0 || Uout != a.tma.Ub[v ^ 1]) return launch_stage_tiles<SmallTile>(a, Uin, Uout, parity, st);
    k_stage2_tma<T, TmaTile><<<tile_grid<TmaTile>(a.g), TmaTile::NT, sizeof(SmemStage<T, TmaTile>), st>>>(
        a.g, a.p, a.tma.U[v], a.tma.L, a.tma.S, a.tma.B, a.tma.Ust[v ^ 1], Uin, a.B, a.L, a.S, Uout, a.rec, parity);
    return cudaGetLastError();
  } else {
    return launch_stage_tiles<BigTile>(a, Uin, Uout, parity, st);
  }
}

template <typename T>
cudaError_t launch_step_impl(const StepArgs<T>& a, const T* Uin, T* Uout, int parity, cudaStream_t st) {
  cudaError_t e = launch_flux_impl<T>(a, Uin, parity, st);
  if (e != cudaSuccess) return e;
  return launch_stage_impl<T>(a, Uin, Uout, parity, st);
}

template <typename T>
cudaError_t launch_bc_impl(const Geom<T>& g, T* U, cudaStream_t st) {
  const int n = 2 * g.gc * (g.nx + g.ny);
  int blocks = (n + NT - 1) / NT;
  if (blocks > 4096) blocks = 4096;
  k_bc<T><<<blocks, NT, 0, st>>>(g, U);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_volume_impl(const Geom<T>& g, const T* U, const T* B, double* partial, int nblocks, double* out,
                               cudaStream_t st) {
  k_volume_partial<T><<<nblocks, NT, 0, st>>>(g, U, B, partial);
  k_volume_final_impl<<<1, NT, 0, st>>>(partial, nblocks, out);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_point_impl(const AdjArgs<T>& a, int* nblocks_out, cudaStream_t st) {
  const int blocks = adj_point_blocks(a.g.nx, a.g.ny);
  k_adj_point<T><<<blocks, dim3(32, kPointRows), 0, st>>>(a);
  if (nblocks_out) *nblocks_out = blocks;
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_face_impl(const AdjArgs<T>& a, cudaStream_t st) {
  const dim3 blk(32, 4);
  k_adj_face<T><<<dim3((a.g.nx + 1 + 31) / 32, (a.g.ny + 1 + 3) / 4, 2), blk, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_recon_impl(const AdjArgs<T>& a, cudaStream_t st) {
  const dim3 blk(32, 4);
  k_adj_recon<T><<<dim3((a.g.nx + 2 + 31) / 32, (a.g.ny + 2 + 3) / 4, 2), blk, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_gather_impl(const AdjArgs<T>& a, cudaStream_t st) {
  const dim3 blk(32, 8);
  k_adj_gather<T><<<dim3((a.g.N1 + 1 + 31) / 32, (a.g.N2 + 1 + 7) / 8, 2), blk, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adj_seed_impl(const Geom<T>& g, const T* U, T* lam, const int* gi, const int* gj,
                                 const double* target, int n, double* loss, cudaStream_t st) {
  k_adj_seed<T><<<1, 32, 0, st>>>(g, U, lam, gi, gj, target, n, loss);
  return cudaGetLastError();
}

}  // namespace vf
