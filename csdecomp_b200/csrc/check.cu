// check.cu -- fused forward kinematics + collision checks on sm_100a.
//
// Reference pipeline (per call): executeForwardKinematicsKernel writes every
// link transform of every configuration to HBM (cuda_forward_kinematics.cu:59-90),
// pairCollisionFreeKernel runs one thread per (configuration, pair) and
// re-multiplies two 4x4 transforms per pair (cuda_collision_checker.cu:16-64),
// and poolPairCollisionFreeResultsKernel ANDs the N*P byte flags (:66-85).
//
// Here one warp checks up to eight configurations end to end: FK of all of
// them side by side, then each one's placement and tests, in registers and
// shared memory; a warp vote stops at the first colliding pair. The statics
// are found through a grid (check_field.cuh) or, in the pair sweep
// (check_core.cuh), staged into shared memory once per block. Only the
// configurations and the verdict bytes touch HBM.
#include <algorithm>

#include "check_warp.cuh"

namespace csd {

// VOX: with voxels (their test costs registers that a check without them would spill).
template <int M, bool VOX>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, ModeBlocks<M>::n)
    check_points_kernel(DevPlant p, const float* __restrict__ q, int64_t n, VoxArgs vox, uint8_t* __restrict__ out) {
  const VoxArgs va = VOX ? vox : VoxArgs{};
  extern __shared__ float4 smem4[];
  __shared__ uint64_t bar;
  const WarpCtx<M> w = warp_setup<M>(p, smem4, &bar);
  if (!w.ok) return;
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  if constexpr (M != kModeField) {
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw) {
      if (lane < p.dim) w.qs[lane] = q[i * p.dim + lane];
      __syncwarp();
      fk_warp(p, w.qs, w.X, lane);
      const bool hit = check_config(p, w.stat, w.aabb, w.X, w.pose, lane, va);
      if (lane == 0) out[i] = hit ? 0 : 1;
    }
    return;
  }
  // runs of a warp's batch, shorter when there are not enough configurations for every warp
  const int64_t per = (n + nw - 1) / nw;
  const int64_t B = per < warp_batch<M>(p) ? per : warp_batch<M>(p);
  for (int64_t i = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * B; i < n; i += nw * B)
    check_range<M>(p, w, q, i, i + B < n ? i + B : n, lane, va, [&](int64_t k, bool hit) { out[k] = hit ? 0 : 1; });
}

// ------------------------------------------------------------------ edges
__device__ __forceinline__ int64_t edge_points(const float* q1, const float* q2, int d, float step, int mode) {
  if (mode == CSD_EDGE_LINF) {
    float m = 0.f;
    for (int k = 0; k < d; ++k) m = fmaxf(m, fabsf(__fsub_rn(q2[k], q1[k])));
    return (int64_t)ceilf(__fdiv_rn(m, step)) + 1;
  }
  float s = 0.f;
  for (int k = 0; k < d; ++k) {
    float x = __fsub_rn(q2[k], q1[k]);
    s = __fadd_rn(s, __fmul_rn(x, x));
  }
  float nrm = __fsqrt_rn(s);
  if (mode == CSD_EDGE_L2_REF) return (int64_t)ceilf(__fdiv_rn(nrm, step));
  float x = __fadd_rn(__fdiv_rn(nrm, step), 2.0f);
  return (int64_t)(uint32_t)x;
}

// Coordinate of point k of an edge from its endpoint coordinates (a1, a2),
// under a discretisation rule (see csd_capi.h).
__device__ __forceinline__ float edge_coord(float a1, float a2, int64_t np, int mode, int64_t k) {
  float t;
  if (mode == CSD_EDGE_L2_REF) {
    t = __double2float_rn(__ddiv_rn((double)k, (double)np));
  } else if (mode == CSD_EDGE_LINF) {
    if (np - 1 == 0) return a1;
    t = __double2float_rn(__ddiv_rn((double)k, (double)(np - 1)));
  } else {
    if (k == 0) return a1;
    if (k == 1) return a2;
    t = __fmul_rn(__double2float_rn(__ddiv_rn(1.0, (double)(np - 1))), (float)(k - 1));
  }
  return __fadd_rn(__fmul_rn(t, a2), __fmul_rn(__fsub_rn(1.0f, t), a1));
}

// Pair index e of the upper triangle (i < j, row-major) of n nodes -> (i, j):
// e = i n - i (i + 1) / 2 + (j - i - 1). The double-precision estimate of i
// is corrected with exact integer row starts.
static __device__ __forceinline__ void edge_pair(int64_t e, int64_t n, int64_t* i, int64_t* j) {
  auto row_start = [n](int64_t r) { return r * n - r * (r + 1) / 2; };
  const double b = 2.0 * (double)n - 1.0;
  int64_t r = (int64_t)floor((b - sqrt(b * b - 8.0 * (double)e)) * 0.5);
  r = r < 0 ? 0 : r > n - 2 ? n - 2 : r;
  while (r > 0 && row_start(r) > e) --r;
  while (r < n - 2 && row_start(r + 1) <= e) ++r;
  *i = r;
  *j = e - row_start(r) + r + 1;
}

// One warp per edge, edges taken from a work counter. Points are visited
// coarse to fine: with G = ceil(n/32), the visit order is g, G+g, 2G+g, ...
// for g = 0, 1, ..., so the first 32 visits sample the whole edge evenly.
// nodes > 0: the edges are every pair i < j of the `nodes` configurations in
// `starts` (ends unused), in upper-triangle row-major order.
template <int M>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, ModeBlocks<M>::n) check_edges_kernel(DevPlant p, const float* __restrict__ starts,
                                                                         const float* __restrict__ ends, int64_t n,
                                                                         float step, int mode,
                                                                         uint8_t* __restrict__ out,
                                                                         int64_t* __restrict__ pts,
                                                                         unsigned long long* counter, int64_t nodes) {
  extern __shared__ float4 smem4[];
  __shared__ uint64_t bar;
  const WarpCtx<M> w = warp_setup<M>(p, smem4, &bar);
  if (!w.ok) return;
  const int lane = threadIdx.x & 31;
  const int d = p.dim;
  VoxArgs none{nullptr, 0, 0.f, nullptr, nullptr, 0};
  while (true) {
    unsigned long long e = 0;
    if (lane == 0) e = atomicAdd(counter, 1ull);
    e = __shfl_sync(kFull, e, 0);
    if (e >= (unsigned long long)n) break;
    __syncwarp();
    if (nodes > 0) {
      int64_t i = 0, j = 0;
      edge_pair((int64_t)e, nodes, &i, &j);
      if (lane < d) {
        w.q1[lane] = starts[i * d + lane];
        w.q2[lane] = starts[j * d + lane];
      }
    } else if (lane < d) {
      w.q1[lane] = starts[e * d + lane];
      w.q2[lane] = ends[e * d + lane];
    }
    __syncwarp();
    const int64_t np = edge_points(w.q1, w.q2, d, step, mode);
    const int64_t G = (np + 31) / 32;
    bool collided = false;
    int64_t checked = 0;
    if constexpr (M != kModeField) {
      const float a1 = lane < d ? w.q1[lane] : 0.f, a2 = lane < d ? w.q2[lane] : 0.f;
      for (int64_t v = 0; v < 32 * G && !collided; ++v) {
        const int64_t k = (v % 32) * G + v / 32;
        if (k >= np) continue;
        const float x = edge_coord(a1, a2, np, mode, k);
        __syncwarp();
        if (lane < d) w.qs[lane] = x;
        __syncwarp();
        fk_warp(p, w.qs, w.X, lane);
        ++checked;
        collided = check_config(p, w.stat, w.aabb, w.X, w.pose, lane, none);
      }
      if (lane == 0) {
        out[e] = collided ? 0 : 1;
        if (pts) pts[e] = checked;
      }
      continue;
    }
    // batches of visits share their FK; a visit past the edge's points repeats the last point and is not checked
    const int B = warp_batch<M>(p);
    for (int64_t v0 = 0; v0 < 32 * G && !collided; v0 += B) {
      __syncwarp();
      for (int c = lane; c < B * d; c += kWarp) {
        const int g = c / d, k = c - g * d;
        const int64_t v = v0 + g, pt = (v % 32) * G + v / 32;
        w.qs[g * kMaxDim + k] = edge_coord(w.q1[k], w.q2[k], np, mode, pt < np ? pt : np - 1);
      }
      __syncwarp();
      fk_configs<M>(p, w, B, lane);
      for (int g = 0; g < B && !collided; ++g) {
        const int64_t v = v0 + g;
        if ((v % 32) * G + v / 32 >= np) continue;
        ++checked;
        collided = check_nth<M>(p, w, g, lane, none);
      }
    }
    if (lane == 0) {
      out[e] = collided ? 0 : 1;
      if (pts) pts[e] = checked;
    }
  }
}

// ------------------------------------------------- surrogate-ranked edge checks
// Points per edge (thread per edge).
__global__ void edge_count_kernel(const float* __restrict__ s, const float* __restrict__ e, int64_t n, int d,
                                  float step, int mode, int64_t* __restrict__ counts) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    counts[i] = edge_points(s + i * d, e + i * d, d, step, mode);
}

// The points of edges [e0, e1) as rows of x (edge i's points from row
// off[i] - off[e0]); warp per edge, lane per point.
__global__ void edge_materialize_kernel(const float* __restrict__ s, const float* __restrict__ e, int64_t e0,
                                        int64_t e1, const int64_t* __restrict__ off, int d, int mode,
                                        float* __restrict__ x) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = e0 + blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < e1; i += nw) {
    const int64_t np = off[i + 1] - off[i];
    float* xi = x + (off[i] - off[e0]) * d;
    for (int64_t k = lane; k < np; k += 32)
      for (int c = 0; c < d; ++c) xi[k * d + c] = edge_coord(s[i * d + c], e[i * d + c], np, mode, k);
  }
}

// Warp per edge of [e0, e1): if logits are given, the point with the highest
// logit in each residue class k mod 32 is a candidate, the candidates are
// checked in decreasing logit (at most `top`), then every other point
// coarse-to-fine as check_edges_kernel visits them. The verdict is the AND
// over all points either way; only the order (and so the early exit) depends
// on the logits.
template <int M>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, ModeBlocks<M>::n)
    check_edges_ranked_kernel(DevPlant p, const float* __restrict__ starts, const float* __restrict__ ends, int64_t e0,
                              int64_t e1, const int64_t* __restrict__ off, const float* __restrict__ logits, int top,
                              int mode, uint8_t* __restrict__ out, int64_t* __restrict__ pts,
                              unsigned long long* counter) {
  extern __shared__ float4 smem4[];
  __shared__ uint64_t bar;
  const WarpCtx<M> w = warp_setup<M>(p, smem4, &bar);
  if (!w.ok) return;
  const int lane = threadIdx.x & 31;
  const int d = p.dim;
  VoxArgs none{};
  while (true) {
    unsigned long long c = 0;
    if (lane == 0) c = atomicAdd(counter, 1ull);
    c = __shfl_sync(kFull, c, 0);
    const int64_t e = e0 + (int64_t)c;
    if (e >= e1) break;
    const int64_t np = off[e + 1] - off[e];
    const float a1 = lane < d ? starts[e * d + lane] : 0.f, a2 = lane < d ? ends[e * d + lane] : 0.f;
    bool collided = false;
    int64_t checked = 0;
    // candidates: best logit of each residue class, sorted descending across the warp
    float bv = -FLT_MAX;
    int64_t bk = -1;
    if (logits) {
      const float* lg = logits + (off[e] - off[e0]);
      for (int64_t k = lane; k < np; k += 32) {
        const float v = lg[k];
        if (v > bv || bk < 0) {
          bv = v;
          bk = k;
        }
      }
    }
    // bitonic sort of (bv, bk) over the 32 lanes: lane r ends with the r-th
    // candidate by decreasing logit (lower index on ties; empty classes last)
    auto before = [](float va, int64_t ka, float vb, int64_t kb) {
      return ka >= 0 && (kb < 0 || va > vb || (va == vb && ka < kb));
    };
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        const float ov = __shfl_xor_sync(kFull, bv, stride);
        const int64_t ok = __shfl_xor_sync(kFull, bk, stride);
        const bool descending = (lane & size) == 0;
        const bool lower = (lane & stride) == 0;
        const bool take = (lower == descending) ? before(ov, ok, bv, bk) : before(bv, bk, ov, ok);
        if (take) {
          bv = ov;
          bk = ok;
        }
      }
    }
    int ncand = logits ? min(top, np < 32 ? (int)np : 32) : 0;
    const int64_t G = (np + 31) / 32;
    // one visiting loop (one inlined check): candidates r < ncand first, then coarse-to-fine
    int r = 0;
    int64_t v = 0;
    while (!collided) {
      int64_t k;
      if (r < ncand) {
        k = __shfl_sync(kFull, bk, r);
        ++r;
        if (k < 0) {  // fewer candidates than `top`: the rest are empty classes
          ncand = r - 1;
          continue;
        }
      } else {
        if (v >= 32 * G) break;
        k = (v % 32) * G + v / 32;
        ++v;
        if (k >= np) continue;
        if (__any_sync(kFull, lane < ncand && bk == k)) continue;  // checked as a candidate
      }
      const float x = edge_coord(a1, a2, np, mode, k);
      __syncwarp();
      if (lane < d) w.qs[lane] = x;
      __syncwarp();
      ++checked;
      fk_configs<M>(p, w, 1, lane);
      collided = check_nth<M>(p, w, 0, lane, none);
    }
    if (lane == 0) {
      out[e] = collided ? 0 : 1;
      if (pts) pts[e] = checked;
    }
  }
}

// ---------------------------------------------------------------- FK output
// All link transforms as column-major 4x4, by one of two kernels (launch_fk).

// Warp per configuration: FK as the checks run it, then lane l composes and
// writes links l, l + 32, ... Its latency is one configuration's, so it serves
// small batches, and it stages nothing per link, so it serves any tree.
__global__ void __launch_bounds__(32 * kWarpsPerBlock) fk_warp_kernel(DevPlant p, const float* __restrict__ q, int64_t n,
                                                                     float* __restrict__ tf_out) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31;
  float* X = reinterpret_cast<float*>(smem4) + (threadIdx.x >> 5) * (p.num_slots * 12 + kMaxDim);
  float* qs = X + p.num_slots * 12;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += nw) {
    if (lane < p.dim) qs[lane] = q[i * p.dim + lane];
    __syncwarp();
    fk_warp(p, qs, X, lane);
    __syncwarp();
    for (int l = lane; l < p.num_links; l += kWarp) {
      const int s = __ldg(p.link_slot + l);
      const float4* F = reinterpret_cast<const float4*>(p.link_fixed + 12 * l);
      const float4 a = __ldg(F), b = __ldg(F + 1), c = __ldg(F + 2);
      const float Rf[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x}, tf[3] = {c.y, c.z, c.w};
      float R[9], t[3];
      if (s < 0) {  // welded to the world, or unreachable (zeros)
#pragma unroll
        for (int k = 0; k < 9; ++k) R[k] = s == -1 ? Rf[k] : 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = s == -1 ? tf[k] : 0.f;
      } else {
        compose(X + s * 12, X + s * 12 + 9, Rf, tf, R, t);
      }
      float4* dst = reinterpret_cast<float4*>(tf_out + (i * p.num_links + l) * 16);
      dst[0] = make_float4(R[0], R[1], R[2], 0.f);
      dst[1] = make_float4(R[3], R[4], R[5], 0.f);
      dst[2] = make_float4(R[6], R[7], R[8], 0.f);
      dst[3] = make_float4(t[0], t[1], t[2], s == -2 ? 0.f : 1.f);
    }
    __syncwarp();
  }
}

// Lane per configuration: a lane walks the tree with one slot transform in
// registers (those that joints branch off from later are kept in the warp's
// shared memory), so every lane works and no value crosses lanes. After each
// joint the links on its slot (link_order lists them by slot) are composed and
// written through a shared tile, four lanes per matrix, whole 32-byte sectors.
// The output is the work: 64 bytes per link. fk_warp_kernel (12 of 32 lanes
// composing by shuffles, each matrix stored as four 16-byte pieces per lane)
// reaches 0.7 TB/s: 87 us for 100,003 configurations of 9 links, 16 us here
// (3.7 TB/s).
constexpr int kFkWarps = 4;
constexpr int kFkTile = kWarp * 20;  // floats: 32 matrices, rows padded against bank conflicts

// Shared floats of the tables (joints, link transforms, slots and order) and of one warp (kept transforms,
// configurations, tile).
static __host__ __device__ __forceinline__ int fk_table_words(const DevPlant& p) {
  return p.num_fk * (int)(sizeof(FkJoint) / 4) + ((14 * p.num_links + 3) & ~3);
}
static __host__ __device__ __forceinline__ int fk_warp_words(const DevPlant& p) {
  return p.num_saved * 12 * kWarp + kMaxDim * kWarp + kFkTile;
}

__global__ void __launch_bounds__(kFkWarps * 32) fk_kernel(DevPlant p, const float* __restrict__ q, int64_t n,
                                                           float* __restrict__ tf_out) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, L = p.num_links;
  float* tab = reinterpret_cast<float*>(smem4);
  const FkJoint* fk = reinterpret_cast<const FkJoint*>(tab);
  float* fixed = tab + p.num_fk * (int)(sizeof(FkJoint) / 4);
  int* lslot = reinterpret_cast<int*>(fixed + 12 * L);
  int* order = lslot + L;
  float* keep = tab + fk_table_words(p) + warp * fk_warp_words(p);
  float* qs = keep + p.num_saved * 12 * kWarp;
  float* tile = qs + kMaxDim * kWarp;
  for (int i = threadIdx.x; i < p.num_fk * (int)(sizeof(FkJoint) / 4); i += blockDim.x)
    tab[i] = __ldg(reinterpret_cast<const float*>(p.fk) + i);
  for (int i = threadIdx.x; i < 12 * L; i += blockDim.x) fixed[i] = __ldg(p.link_fixed + i);
  for (int i = threadIdx.x; i < L; i += blockDim.x) {
    lslot[i] = __ldg(p.link_slot + i);
    order[i] = __ldg(p.link_order + i);
  }
  __syncthreads();
  const int64_t nw = (int64_t)gridDim.x * kFkWarps;
  for (int64_t i0 = ((int64_t)blockIdx.x * kFkWarps + warp) * kWarp; i0 < n; i0 += nw * kWarp) {
    const int cnt = (int)(n - i0 < kWarp ? n - i0 : kWarp);
    for (int i = lane; i < cnt * p.dim; i += kWarp) qs[i] = __ldg(q + i0 * p.dim + i);
    __syncwarp();
    const float* ql = qs + min(lane, cnt - 1) * p.dim;
    float R[9], t[3];
    int at = 0;
    for (int j = -1; j < p.num_fk; ++j) {
      if (j >= 0) {
        const FkJoint& J = fk[j];
        float Rl[9], tl[3];
        joint_local(J, ql[J.qidx], Rl, tl);
        if (J.parent < 0) {
#pragma unroll
          for (int k = 0; k < 9; ++k) R[k] = Rl[k];
#pragma unroll
          for (int k = 0; k < 3; ++k) t[k] = tl[k];
        } else {
          if (J.from >= 0) {
            const float* src = keep + J.from * 12 * kWarp + lane;
#pragma unroll
            for (int k = 0; k < 9; ++k) R[k] = src[k * kWarp];
#pragma unroll
            for (int k = 0; k < 3; ++k) t[k] = src[(9 + k) * kWarp];
          }
          float Ro[9], to[3];
          compose(R, t, Rl, tl, Ro, to);
#pragma unroll
          for (int k = 0; k < 9; ++k) R[k] = Ro[k];
#pragma unroll
          for (int k = 0; k < 3; ++k) t[k] = to[k];
        }
        if (J.save >= 0) {
          float* dst = keep + J.save * 12 * kWarp + lane;
#pragma unroll
          for (int k = 0; k < 9; ++k) dst[k * kWarp] = R[k];
#pragma unroll
          for (int k = 0; k < 3; ++k) dst[(9 + k) * kWarp] = t[k];
        }
      }
      for (; at < L; ++at) {
        const int l = order[at], s = lslot[l];
        if (s > j) break;
        const float4* F = reinterpret_cast<const float4*>(fixed + 12 * l);
        const float4 a = F[0], b = F[1], c = F[2];
        const float Rf[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x}, tfx[3] = {c.y, c.z, c.w};
        float Ro[9], to[3];
        if (s < 0) {
#pragma unroll
          for (int k = 0; k < 9; ++k) Ro[k] = s == -1 ? Rf[k] : 0.f;
#pragma unroll
          for (int k = 0; k < 3; ++k) to[k] = s == -1 ? tfx[k] : 0.f;
        } else {
          compose(R, t, Rf, tfx, Ro, to);
        }
        float4* w = reinterpret_cast<float4*>(tile + 20 * lane);
        __syncwarp();
        w[0] = make_float4(Ro[0], Ro[1], Ro[2], 0.f);
        w[1] = make_float4(Ro[3], Ro[4], Ro[5], 0.f);
        w[2] = make_float4(Ro[6], Ro[7], Ro[8], 0.f);
        w[3] = make_float4(to[0], to[1], to[2], s == -2 ? 0.f : 1.f);
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int c = 8 * h + (lane >> 2);
          if (c < cnt)
            *reinterpret_cast<float4*>(tf_out + ((i0 + c) * L + l) * 16 + 4 * (lane & 3)) =
                *reinterpret_cast<const float4*>(tile + 20 * c + 4 * (lane & 3));
        }
      }
    }
    __syncwarp();
  }
}

// Single pair on the device (one thread), GPU contact rule.
__global__ void pair_kernel(int ta, const float* g, int tb, uint8_t* out) {
  // g: [2][16] world-format poses computed on the host from FP32 inputs
  *out = pair_hit(ta, g, tb, g + 16) ? 0 : 1;
}

// ----------------------------------------------------------------- launchers
csd_status_t launch_check_points(const csd_plant_s* p, const float* q, int64_t n, const VoxelTables& vt,
                                 uint8_t* out, cudaStream_t st) {
  if (n <= 0) return CSD_OK;
  const VoxArgs va = vox_args(vt);
  return with_mode(plant_mode(p), [&](auto m) -> csd_status_t {
    auto kernel = va.nv > 0 ? check_points_kernel<decltype(m)::value, true> : check_points_kernel<decltype(m)::value, false>;
    const size_t smem = smem_bytes(p, kWarpsPerBlock);
    int grid = 0;
    if (csd_status_t s = grid_for(kernel, smem, n, &grid, kWarpsPerBlock)) return s;
    kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(p->dp, q, n, va, out);
    CSD_CUDA_TRY(cudaGetLastError());
    return CSD_OK;
  });
}

// The lane kernel once it has the warps to cover its latency, a walk over the
// whole tree: from 6,144 configurations and 64 per link on, 16,384 at most, and
// where its tables fit a block. Warp kernel against lane kernel: 8 links 10.2 /
// 12.3 us at 512 configurations, 12.3 / 12.3 at 6,144, 31.6 / 13.1 at 32,768;
// 57 links 12.3 / 24.6 at 512, 23.2 / 23.3 at 8,192, 57 / 33 at 32,768; 2,101
// links 33 / 465 at one, 516 / 586 at 12,288, 705 / 586 at 16,384.
constexpr int64_t kFkLaneMin = 6144, kFkLanePerLink = 64, kFkLaneMost = 16384;
constexpr size_t kFkLaneShared = 220 * 1024;

csd_status_t launch_fk(const csd_plant_s* p, const float* q, int64_t n, float* tf, cudaStream_t st) {
  if (n <= 0) return CSD_OK;
  size_t smem = ((size_t)fk_table_words(p->dp) + (size_t)fk_warp_words(p->dp) * kFkWarps) * sizeof(float);
  int grid = 0;
  if (n < std::min(kFkLaneMost, kFkLaneMin + kFkLanePerLink * p->dp.num_links) || smem > kFkLaneShared) {
    smem = (size_t)(p->dp.num_slots * 12 + kMaxDim) * kWarpsPerBlock * sizeof(float);
    if (csd_status_t s = grid_for(fk_warp_kernel, smem, n, &grid, kWarpsPerBlock)) return s;
    fk_warp_kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(p->dp, q, n, tf);
    CSD_CUDA_TRY(cudaGetLastError());
    return CSD_OK;
  }
  if (csd_status_t s = grid_for(fk_kernel, smem, (n + kWarp - 1) / kWarp, &grid, kFkWarps)) return s;
  fk_kernel<<<grid, 32 * kFkWarps, smem, st>>>(p->dp, q, n, tf);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

csd_status_t launch_edge_count(const float* s, const float* e, int64_t n, int d, float step, int mode,
                               int64_t* counts, cudaStream_t st) {
  if (n <= 0) return CSD_OK;
  const int grid = (int)std::min<int64_t>((n + 255) / 256, 8 * device_sm_count());
  edge_count_kernel<<<grid, 256, 0, st>>>(s, e, n, d, step, mode, counts);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

csd_status_t launch_edge_materialize(const float* s, const float* e, int64_t e0, int64_t e1, const int64_t* off, int d,
                                     int mode, float* x, cudaStream_t st) {
  if (e1 <= e0) return CSD_OK;
  const int grid = (int)std::min<int64_t>((e1 - e0 + 7) / 8, 8 * device_sm_count());
  edge_materialize_kernel<<<grid, 256, 0, st>>>(s, e, e0, e1, off, d, mode, x);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

csd_status_t launch_check_edges_ranked(const csd_plant_s* p, const float* s0, const float* e0p, int64_t e0, int64_t e1,
                                       const int64_t* off, const float* logits, int top, int mode, uint8_t* out,
                                       int64_t* pts, unsigned int* counter, cudaStream_t st) {
  if (e1 <= e0) return CSD_OK;
  CSD_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
  unsigned long long* ctr = reinterpret_cast<unsigned long long*>(counter);
  return with_mode(plant_mode(p), [&](auto m) -> csd_status_t {
    auto kernel = check_edges_ranked_kernel<decltype(m)::value>;
    const size_t smem = smem_bytes(p, kWarpsPerBlock);
    int grid = 0;
    if (csd_status_t s = grid_for(kernel, smem, e1 - e0, &grid, kWarpsPerBlock)) return s;
    kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(p->dp, s0, e0p, e0, e1, off, logits, top, mode, out, pts, ctr);
    CSD_CUDA_TRY(cudaGetLastError());
    return CSD_OK;
  });
}

csd_status_t launch_check_edges(const csd_plant_s* p, const float* s0, const float* e0, int64_t n, float step,
                                int mode, uint8_t* out, int64_t* pts, unsigned int* counter, cudaStream_t st,
                                int64_t nodes) {
  if (n <= 0) return CSD_OK;
  CSD_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
  unsigned long long* ctr = reinterpret_cast<unsigned long long*>(counter);
  return with_mode(plant_mode(p), [&](auto m) -> csd_status_t {
    auto kernel = check_edges_kernel<decltype(m)::value>;
    const size_t smem = smem_bytes(p, kWarpsPerBlock);
    int grid = 0;
    if (csd_status_t s = grid_for(kernel, smem, n, &grid, kWarpsPerBlock)) return s;
    kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(p->dp, s0, e0, n, step, mode, out, pts, ctr, nodes);
    CSD_CUDA_TRY(cudaGetLastError());
    return CSD_OK;
  });
}

csd_status_t launch_pair(int ta, const float* g_dev, int tb, uint8_t* out, cudaStream_t st) {
  pair_kernel<<<1, 1, 0, st>>>(ta, g_dev, tb, out);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

}  // namespace csd
