// vf_pack.cuh -- many simulations stepped together by whole-grid launches.
//
// A pack is a list of Float64 RK2 simulations. Every step is two launches for all
// of them: the grid is the union of the members' tiles (map: block -> member and
// its tile), and each member keeps its own step record, dt and end time as in
// vf_simulate. A batch of small grids so fills the GPU as one large grid does,
// where launches of their own would pay two launches per member and step, and a
// cluster leaves a member 16 SMs at most. The tiles are the plain kernels' and
// give the same bits. Bound by the FP64 pipe where there are enough members, by
// launches and tails with few: 20 members of 64-224^2 cells, at most 8 steps, took
// 4.15 ms as clusters and launches of their own, 1.84 ms packed, while they took four
// steps on average (4.0 ms packed when all take eight); 200 of 64-80^2, 40 steps,
// 40.6 and 27.8 ms (vf_batch.cu has where the line lies).
// A member that has ended costs its blocks' empty turns until the host drops it
// from the map.
#pragma once
#include "vf_kernels.cuh"

namespace vf {

template <typename T>
struct PackItem {
  Geom<T> g;
  Phys<T> p;
  const T* B;
  T* U[2];  // step n reads U[n & 1] and writes U[(n & 1) ^ 1]
  T* L;
  T* S;
  StepRecord* rec;
  StepRecord* report[3];  // device addresses of the host's copies, one per chunk in flight
};

struct PackBlock {
  int member, block;  // block: the member's own block number
};

// The block's member, copied to shared memory; false when the member has ended
// (then its block 0 hands the record on after a stage pass).
template <typename T>
__device__ __forceinline__ bool pack_enter(const PackItem<T>* __restrict__ items, const PackBlock& b, int parity,
                                           PackItem<T>& it) {
  static_assert(sizeof(PackItem<T>) % 8 == 0, "items copy in 8-byte words");
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(items + b.member);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(&it);
  for (int i = threadIdx.x; i < (int)(sizeof(PackItem<T>) / 8); i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  return it.rec->active[parity] != 0;
}

template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB)
    k_pack_flux(const PackItem<T>* __restrict__ items, const PackBlock* __restrict__ map, int parity) {
  __shared__ PackItem<T> it;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemFlux<T, S>& s = *reinterpret_cast<SmemFlux<T, S>*>(smem_raw);
  const PackBlock b = map[blockIdx.x];
  if (!pack_enter<T>(items, b, parity, it)) return;
  const int tx = (it.g.nx + S::TX - 1) / S::TX;
  const double t = it.p.any_dynamic ? it.rec->t[parity] : 0.0;
  T mx = (T)0, my = (T)0;
  flux_tile<T, false, false, S>(it.g, it.p, it.U[parity], it.B, it.L, it.S, it.g.gc + (b.block % tx) * S::TX,
                                it.g.gc + (b.block / tx) * S::TY, s, t, mx, my);
  unsigned long long kx = 0, ky = 0;
  block_speed_keys<T, S::NT>(mx, my, s.red, kx, ky);
  if (threadIdx.x == 0) {
    atomicMax(&it.rec->speed_bits[parity][0], kx);
    atomicMax(&it.rec->speed_bits[parity][1], ky);
  }
}

template <typename T, typename S>
__global__ void __launch_bounds__(S::NT, S::MINB)
    k_pack_stage(const PackItem<T>* __restrict__ items, const PackBlock* __restrict__ map, int parity) {
  __shared__ PackItem<T> it;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemStage<T, S>& s = *reinterpret_cast<SmemStage<T, S>*>(smem_raw);
  const PackBlock b = map[blockIdx.x];
  const bool root = b.block == 0 && threadIdx.x == 0;
  if (!pack_enter<T>(items, b, parity, it)) {
    if (root) carry_record(it.rec, parity);
    return;
  }
  if (threadIdx.x == 0) s.dt = step_dt<T>(it.g, it.rec, parity);
  __syncthreads();
  const double dt = s.dt;
  const int tx = (it.g.nx + S::TX - 1) / S::TX;
  stage2_tile<T, false, false, S>(it.g, it.p, it.U[parity], it.B, it.L, it.S, it.U[parity ^ 1],
                                  it.g.gc + (b.block % tx) * S::TX, it.g.gc + (b.block / tx) * S::TY, s, dt,
                                  it.rec->t[parity]);
  if (root) advance_record<T>(it.rec, parity, dt);
}

// Every member's record to the host's copy `slot` (pinned, mapped memory).
template <typename T>
__global__ void k_pack_report(const PackItem<T>* __restrict__ items, int n, int slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) *items[i].report[slot] = *items[i].rec;
}

}  // namespace vf
