// check_warp.cuh -- the checking warps' view of a plant: which check runs
// (mode), the per-warp shared memory, FK and check of a few configurations,
// launch sizes.
#pragma once
#include <type_traits>

#include "check_field.cuh"

namespace csd {

// How a configuration is checked. kModeField (spheres and capsules against
// the statics' grid, check_field.cuh) wherever the plant has the tables and
// the broad phase is on: a free configuration of the 7-DOF arm in 200
// primitives costs 1.6 ns there against 9.5 ns with the link-sphere
// broad phase. The other two are the pair sweep of check_core.cuh, for plants
// with moving boxes, more than 1,024 statics, geometry that build_field leaves
// out, or the broad phase switched off (every pair tested): statics staged in shared memory, or read from global
// memory when they do not fit.
enum : int { kModeGlobal = 0, kModeStaged = 1, kModeField = 2 };

template <int M>
struct WarpCtx {
  const float4* stat;
  const float4* aabb;
  float* X;
  float* qs;   // [warp_batch][kMaxDim]
  float* q1;
  float* q2;
  float* pose;
  bool ok;
};

template <int M>
static __host__ __device__ __forceinline__ int mode_warp_floats(const DevPlant& p) {
  return M == kModeField ? field_warp_floats(p) : warp_floats(p);
}

// Configurations a warp takes at once: fk_configs runs their FK together where
// the mode can, and their slot transforms and coordinates are kept apart.
template <int M>
static __host__ __device__ __forceinline__ int warp_batch(const DevPlant& p) {
  return M == kModeField ? fk_batch(p) : 1;
}

template <int M>
static __device__ __forceinline__ void warp_buffers(const DevPlant& p, float* wbase, WarpCtx<M>& w) {
  w.X = wbase + (threadIdx.x >> 5) * mode_warp_floats<M>(p);
  w.qs = w.X + warp_batch<M>(p) * p.num_slots * 12;
  w.q1 = w.qs + warp_batch<M>(p) * kMaxDim;
  w.q2 = w.q1 + kMaxDim;
  w.pose = w.q2 + kMaxDim;
}

template <int M>
static __device__ __forceinline__ WarpCtx<M> warp_setup(const DevPlant& p, float4* smem4, uint64_t* bar) {
  WarpCtx<M> w;
  float* wbase = reinterpret_cast<float*>(smem4);
  w.ok = true;
  w.stat = p.statics;
  w.aabb = p.aabb;
  if (M == kModeStaged) {
    w.ok = stage_statics(p, smem4, bar);
    w.stat = smem4;
    w.aabb = smem4 + 4 * p.num_static;
    wbase += p.static_bytes / 4;
  }
  warp_buffers<M>(p, wbase, w);
  return w;
}

// FK of the configurations w.qs[0 .. m), m <= warp_batch.
template <int M>
static __device__ __forceinline__ void fk_configs(const DevPlant& p, const WarpCtx<M>& w, int m, int lane) {
  if (M == kModeField)
    fk_rows(p, w.qs, m, w.X, w.pose, lane);
  else
    fk_warp(p, w.qs, w.X, lane);
}

// Whether configuration g of the last fk_configs collides (warp-uniform).
template <int M>
static __device__ __forceinline__ bool check_nth(const DevPlant& p, const WarpCtx<M>& w, int g, int lane,
                                                 const VoxArgs& va) {
  if (M == kModeField) return check_field(p, w.X + g * p.num_slots * 12, w.pose, lane, va);
  return check_config(p, w.stat, w.aabb, w.X, w.pose, lane, va);
}

// Configurations q[i0 .. i1) by one warp: verdict(i, collides) in order.
template <int M, typename F>
static __device__ __forceinline__ void check_range(const DevPlant& p, const WarpCtx<M>& w, const float* __restrict__ q,
                                                   int64_t i0, int64_t i1, int lane, const VoxArgs& va, F verdict) {
  if constexpr (M != kModeField) {
    for (int64_t i = i0; i < i1; ++i) {
      __syncwarp();
      if (lane < p.dim) w.qs[lane] = q[i * p.dim + lane];
      __syncwarp();
      fk_warp(p, w.qs, w.X, lane);
      const bool hit = check_config(p, w.stat, w.aabb, w.X, w.pose, lane, va);
      if (lane == 0) verdict(i, hit);
    }
    return;
  }
  const int B = warp_batch<M>(p);
  for (int64_t i = i0; i < i1; i += B) {
    const int m = (int)(i1 - i < B ? i1 - i : B);
    __syncwarp();
    for (int e = lane; e < m * p.dim; e += kWarp) {
      const int g = e / p.dim;
      w.qs[g * kMaxDim + e - g * p.dim] = q[i * p.dim + e];
    }
    __syncwarp();
    fk_configs<M>(p, w, m, lane);
    for (int g = 0; g < m; ++g) {
      const bool hit = check_nth<M>(p, w, g, lane, va);
      if (lane == 0) verdict(i + g, hit);
    }
  }
}

// Blocks per SM the check kernels are compiled for.
template <int M>
struct ModeBlocks {
  static constexpr int n = M == kModeField ? 4 : 3;
};

// ---- host helpers shared by the launchers
static inline int plant_mode(const csd_plant_s* p) {
  if (p->dp.cull && p->dp.has_field) return kModeField;
  return p->dp.static_bytes <= kStaticSmemLimit ? kModeStaged : kModeGlobal;
}

static inline size_t smem_bytes(const csd_plant_s* p, int wpb) {
  const int mode = plant_mode(p);
  const size_t per = (size_t)(mode == kModeField ? field_warp_floats(p->dp) : warp_floats(p->dp)) * sizeof(float) * wpb;
  return per + (mode == kModeStaged ? (size_t)p->dp.static_bytes : 0);
}

// Calls f with the mode as a compile-time constant.
template <typename F>
static inline csd_status_t with_mode(int mode, F f) {
  switch (mode) {
    case kModeField: return f(std::integral_constant<int, kModeField>());
    case kModeStaged: return f(std::integral_constant<int, kModeStaged>());
    default: return f(std::integral_constant<int, kModeGlobal>());
  }
}

// Blocks of a launch. The blocks per SM of a kernel, device and size are asked
// for once per thread (a few entries, replaced in turn): the queries of
// attributes and occupancy, with the read of the staging status, cost a small
// call 12 us of 52. Shared-memory limits only ever rise, so one seen raised
// stays raised.
template <typename K>
static csd_status_t grid_for(K kernel, size_t smem, int64_t work_warps, int* grid, int wpb) {
  struct Seen {
    K kernel = nullptr;
    int dev = -1, wpb = 0, per_sm = 0;
    size_t smem = 0;
  };
  static thread_local Seen seen[8];
  static thread_local int next = 0;
  int per_sm = 0, dev = 0;
  CSD_CUDA_TRY(cudaGetDevice(&dev));
  for (const Seen& e : seen)
    if (e.kernel == kernel && e.dev == dev && e.wpb == wpb && e.smem == smem) per_sm = e.per_sm;
  if (per_sm <= 0) {
    CSD_CUDA_TRY(raise_smem_limit(kernel, (int)smem));
    CSD_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * wpb, smem));
    if (per_sm <= 0) {
      set_error("plant tables do not fit in shared memory");
      return CSD_ERR_CAPACITY;
    }
    seen[next] = Seen{kernel, dev, wpb, per_sm, smem};
    next = (next + 1) % 8;
  }
  int64_t need = (work_warps + wpb - 1) / wpb;
  int64_t full = (int64_t)per_sm * device_sm_count();
  *grid = (int)std::max<int64_t>(1, std::min(need, full));
  return CSD_OK;
}

}  // namespace csd
