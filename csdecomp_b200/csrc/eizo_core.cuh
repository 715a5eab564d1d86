// eizo_core.cuh -- EI-ZO stage bodies shared by the single-inflation kernels
// (eizo.cu) and the batched kernels (batch.cu): ordered compaction, the
// per-particle bisection and the greedy face placement.
#pragma once
#include <cfloat>

#include "check_warp.cuh"
#include "sampler_core.cuh"

namespace csd {

struct EizoCounters {
  uint32_t total;     // colliding samples
  uint32_t first_m;   // colliding samples among the first M
  uint32_t placed;    // faces placed by the last faces_kernel
  int32_t status;     // 0 ok, 2 face capacity exceeded
};

// Ordered compaction of the colliding samples (first max_keep kept, in index
// order) and the first-M collision count; one block.
static __device__ __forceinline__ void compact_block(const uint8_t* __restrict__ flags,
                                                     const float* __restrict__ samples, int N, int M, int max_keep,
                                                     int dim, float* __restrict__ cols, EizoCounters* cnt) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t running;
  __shared__ uint32_t first_m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  if (tid == 0) {
    running = 0;
    first_m = 0;
  }
  __syncthreads();
  for (int base = 0; base < N; base += blockDim.x) {
    int i = base + tid;
    uint32_t f = (i < N && !flags[i]) ? 1u : 0u;
    uint32_t ballot = __ballot_sync(0xffffffffu, f);
    uint32_t pre = __popc(ballot & ((1u << lane) - 1u));
    uint32_t fm = __popc(__ballot_sync(0xffffffffu, f && i < M));
    if (lane == 0) warp_sums[warp] = __popc(ballot);
    if (lane == 0 && fm) atomicAdd(&first_m, fm);
    __syncthreads();
    uint32_t off = 0;
    for (int w = 0; w < warp; ++w) off += warp_sums[w];
    uint32_t pos = running + off + pre;
    if (f && pos < (uint32_t)max_keep)
      for (int k = 0; k < dim; ++k) cols[(size_t)pos * dim + k] = samples[(size_t)i * dim + k];
    __syncthreads();
    if (tid == 0) {
      uint32_t tot = 0;
      for (int w = 0; w < nw; ++w) tot += warp_sums[w];
      running += tot;
    }
    __syncthreads();
  }
  if (tid == 0) {
    cnt->total = running;
    cnt->first_m = first_m;
  }
}


// Particles i0 .. i0 + m of one warp (m <= warp_batch), bisected side by side:
// a step's midpoints share their FK, then each is checked. Lane k holds
// coordinate k of a particle's bounds (m pairs of registers). starts(i) and ends(i) give particle i's segment. Dot products
// are accumulated in coordinate order with fused multiply-adds (the order the
// CPU restatement uses).
template <int M, typename S0, typename S1>
static __device__ __forceinline__ void bisect_particles(const DevPlant& p, const WarpCtx<M>& w, int i0, int m, int dim,
                                                        int steps, S0 starts, S1 ends, const VoxArgs& va,
                                                        float* __restrict__ cols, float* __restrict__ proj,
                                                        float* __restrict__ dist, int lane) {
  if constexpr (M != kModeField) {  // one particle (m is 1)
    const float* ci = cols + (size_t)i0 * dim;
    const float *ls = starts(i0), *le = ends(i0);
    float seg2 = 0.f, a = 0.f;
    for (int k = 0; k < dim; ++k) {
      float dk = __fsub_rn(le[k], ls[k]);
      seg2 = __fmaf_rn(dk, dk, seg2);
      a = __fmaf_rn(__fsub_rn(ci[k], ls[k]), dk, a);
    }
    const float t = fminf(fmaxf(__fdiv_rn(a, seg2), 0.0f), 1.0f);
    const float omt = __fsub_rn(1.0f, t);
    float pr = 0.f, lo = 0.f, hi = 0.f;
    if (lane < dim) {
      pr = __fmaf_rn(t, le[lane], __fmul_rn(omt, ls[lane]));
      lo = pr;
      hi = ci[lane];
    }
    for (int s = 0; s < steps; ++s) {
      const float mid = __fmul_rn(0.5f, __fadd_rn(lo, hi));
      __syncwarp();
      if (lane < dim) w.qs[lane] = mid;
      __syncwarp();
      fk_warp(p, w.qs, w.X, lane);
      if (check_config(p, w.stat, w.aabb, w.X, w.pose, lane, va))
        hi = mid;
      else
        lo = mid;
    }
    __syncwarp();
    if (lane < dim) w.qs[lane] = __fsub_rn(hi, pr);
    __syncwarp();
    float s2 = 0.f;
    for (int k = 0; k < dim; ++k) s2 = __fmaf_rn(w.qs[k], w.qs[k], s2);
    if (lane < dim) {
      cols[(size_t)i0 * dim + lane] = hi;
      proj[(size_t)i0 * dim + lane] = pr;
    }
    if (lane == 0) dist[i0] = __fsqrt_rn(s2);
    __syncwarp();
    return;
  }
  constexpr int MB = M == kModeField ? kFkBatch : 1;
  float lo[MB], hi[MB];  // hi: the collision point so far
#pragma unroll
  for (int g = 0; g < MB; ++g) {
    lo[g] = hi[g] = 0.f;
    if (g >= m) break;
    const float* ci = cols + (size_t)(i0 + g) * dim;
    const float *ls = starts(i0 + g), *le = ends(i0 + g);
    // projection onto the segment (every lane evaluates the same serial sums)
    float seg2 = 0.f, a = 0.f;
    for (int k = 0; k < dim; ++k) {
      float dk = __fsub_rn(le[k], ls[k]);
      seg2 = __fmaf_rn(dk, dk, seg2);
      a = __fmaf_rn(__fsub_rn(ci[k], ls[k]), dk, a);
    }
    const float t = fminf(fmaxf(__fdiv_rn(a, seg2), 0.0f), 1.0f);
    const float omt = __fsub_rn(1.0f, t);
    if (lane < dim) {
      hi[g] = ci[lane];
      lo[g] = __fmaf_rn(t, le[lane], __fmul_rn(omt, ls[lane]));
      proj[(size_t)(i0 + g) * dim + lane] = lo[g];
    }
  }
  for (int s = 0; s < steps; ++s) {
    __syncwarp();
#pragma unroll
    for (int g = 0; g < MB; ++g)
      if (g < m && lane < dim) w.qs[g * kMaxDim + lane] = __fmul_rn(0.5f, __fadd_rn(lo[g], hi[g]));
    __syncwarp();
    fk_configs<M>(p, w, m, lane);
    uint32_t hits = 0;
    for (int g = 0; g < m; ++g) hits |= check_nth<M>(p, w, g, lane, va) ? 1u << g : 0u;
#pragma unroll
    for (int g = 0; g < MB; ++g) {
      const float mid = __fmul_rn(0.5f, __fadd_rn(lo[g], hi[g]));
      if ((hits >> g) & 1u)
        hi[g] = mid;
      else
        lo[g] = mid;
    }
  }
  // distance to the projection, coordinates in order
#pragma unroll
  for (int g = 0; g < MB; ++g) {
    if (g >= m) break;
    const size_t at = (size_t)(i0 + g) * dim + lane;
    __syncwarp();
    if (lane < dim) w.qs[lane] = __fsub_rn(hi[g], proj[at]);
    __syncwarp();
    float s2 = 0.f;
    for (int k = 0; k < dim; ++k) s2 = __fmaf_rn(w.qs[k], w.qs[k], s2);
    if (lane < dim) cols[at] = hi[g];
    if (lane == 0) dist[i0 + g] = __fsqrt_rn(s2);
  }
  __syncwarp();
}

// Particles per warp at once for K particles over `warps` warps: one each
// until every warp has some (the particles of a warp are checked one after
// the other).
template <int M>
static __device__ __forceinline__ int bisect_batch(const DevPlant& p, int K, int warps) {
  return min(warp_batch<M>(p), max(1, K / warps));
}

// Greedy face placement by one block (256 to 1,024 threads): the nearest live
// candidate (lower index on ties) gets a face, which drops every candidate it
// cuts off; up to max_faces faces. EDIT: region editing's rule (a zero normal
// stays zero, relaxation + 2e-6 in double, a candidate on the face is cut
// off) and, before the first face, candidates outside the region's nf faces
// are dropped. rows (optional) receives each face as a face-pair row with its
// start slack at ls, the layout the EI-ZO sampler reads (put_face). Returns
// the faces placed; *status = 2 when capacity (faces of A in all) ran out.
//
// A thread keeps kFaceRegs candidates' coordinates and distances in registers
// (the rest, beyond kFaceRegs x threads, stays in global memory), the minimum
// is two integer warp reductions (distances are not negative, so their bits
// order as they do), and one warp works out the face with a coordinate per
// lane. Bound by the two block barriers and the face's serial dot products per
// placed face: 46 us for ten faces of 2,000 candidates when one thread loaded
// and summed everything, 24 us now.
constexpr int kFaceRegs = 2;
template <bool EDIT>
static __device__ int place_faces(int K, int dim, int max_faces, int nf, int capacity, float margin,
                                  const float* __restrict__ ls, const float* __restrict__ le,
                                  const float* __restrict__ cols, const float* __restrict__ proj,
                                  float* __restrict__ dist, float* __restrict__ A, float* __restrict__ b,
                                  float* __restrict__ rows, int* status) {
  __shared__ uint32_t red_v[32], red_i[32];
  __shared__ float face[kMaxDim + 1], vec[3][kMaxDim];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, nt = blockDim.x;
  const uint32_t none = __float_as_uint(FLT_MAX);
  float x[kFaceRegs][kMaxDim];
  uint32_t d[kFaceRegs];  // bits of the distance; `none` or above: not a candidate (any more)
#pragma unroll
  for (int r = 0; r < kFaceRegs; ++r) {
    const int i = tid + r * nt;
    d[r] = i < K ? __float_as_uint(dist[i]) : none;
#pragma unroll
    for (int k = 0; k < kMaxDim; ++k) x[r][k] = i < K && k < dim ? cols[(size_t)i * dim + k] : 0.f;
  }
  if (EDIT) {
    for (int f = 0; f < nf; ++f) {
      const float* a = A + (size_t)f * dim;
#pragma unroll
      for (int r = 0; r < kFaceRegs; ++r) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < kMaxDim; ++k)
          if (k < dim) v = __fmaf_rn(a[k], x[r][k], v);
        if (!(__fsub_rn(v, b[f]) < 0.f)) d[r] = none;
      }
    }
    for (int i = tid + kFaceRegs * nt; i < K; i += nt) {
      bool inside = true;
      for (int f = 0; f < nf && inside; ++f) {
        float v = 0.f;
        for (int k = 0; k < dim; ++k) v = __fmaf_rn(A[(size_t)f * dim + k], cols[(size_t)i * dim + k], v);
        inside = __fsub_rn(v, b[f]) < 0.f;
      }
      if (!inside) dist[i] = FLT_MAX;
    }
  }
  *status = 0;
  int placed = 0;
  for (; placed < max_faces; ++placed) {
    uint32_t bv = none, bi = ~0u;
#pragma unroll
    for (int r = 0; r < kFaceRegs; ++r)
      if (d[r] < bv) {  // ascending index: the first of equal values is kept
        bv = d[r];
        bi = (uint32_t)(tid + r * nt);
      }
    for (int i = tid + kFaceRegs * nt; i < K; i += nt) {
      const uint32_t v = __float_as_uint(dist[i]);
      if (v < bv) {
        bv = v;
        bi = (uint32_t)i;
      }
    }
    uint32_t wv = __reduce_min_sync(0xffffffffu, bv), wi = __reduce_min_sync(0xffffffffu, bv == wv ? bi : ~0u);
    if (lane == 0) {
      red_v[warp] = wv;
      red_i[warp] = wi;
    }
    __syncthreads();
    bv = lane < nw ? red_v[lane] : none;
    bi = lane < nw ? red_i[lane] : ~0u;
    wv = __reduce_min_sync(0xffffffffu, bv);
    wi = __reduce_min_sync(0xffffffffu, bv == wv ? bi : ~0u);
    if (wv >= none) break;  // the same in every warp
    if (nf >= capacity) {
      *status = 2;
      break;
    }
#pragma unroll
    for (int r = 0; r < kFaceRegs; ++r)
      if (wi == (uint32_t)(tid + r * nt)) d[r] = none;
    if (tid == 0 && wi >= (uint32_t)(kFaceRegs * nt)) dist[wi] = FLT_MAX;
    if (warp == 0) {
      float a = 0.f;
      if (lane < dim) {
        const float c = cols[(size_t)wi * dim + lane];
        a = __fsub_rn(c, proj[(size_t)wi * dim + lane]);
        face[lane] = a;
        vec[0][lane] = c;
        vec[1][lane] = ls[lane];
        vec[2][lane] = le[lane];
      }
      __syncwarp();
      float n2 = 0.f;
      for (int k = 0; k < dim; ++k) n2 = __fmaf_rn(face[k], face[k], n2);
      if (!EDIT || n2 > 0.f) a = __fdiv_rn(a, __fsqrt_rn(n2));
      __syncwarp();
      if (lane < dim) face[lane] = a;
      __syncwarp();
      // lane 0: a . collision, lane 1: a . start, lane 2: a . end, each in coordinate order
      float s = 0.f;
      const float* w = vec[lane < 3 ? lane : 0];
      for (int k = 0; k < dim; ++k) s = __fmaf_rn(face[k], w[k], s);
      const float v0 = __shfl_sync(0xffffffffu, s, 1), v2 = __shfl_sync(0xffffffffu, s, 2);
      float bb = __fsub_rn(__shfl_sync(0xffffffffu, s, 0), margin);
      const float r1 = __fsub_rn(v0, bb), r2 = __fsub_rn(v2, bb);
      const float relax = r2 > r1 ? r2 : r1;
      if (EDIT) {
        if (relax > 0.f) bb = __double2float_rn(__dadd_rn((double)bb, __dadd_rn((double)relax, 2e-6)));
      } else {
        bb = __fadd_rn(bb, relax > 0 ? relax : 0.f);
      }
      if (lane < dim) A[(size_t)nf * dim + lane] = a;
      if (lane == 0) {
        b[nf] = bb;
        face[dim] = bb;
      }
      if (rows) {  // put_face, a coordinate per lane
        const int md = pair_maxd(dim), h = nf & 1;
        float* r = rows + (size_t)(nf >> 1) * pair_stride(dim);
        const float slack = __fsub_rn(bb, v0);
        const float big = __any_sync(0xffffffffu, lane < dim && !(fabsf(a) <= kMaxCoeff)) ? 1.f : 0.f;
        if (lane < md) {
          r[2 * lane + h] = lane < dim ? a : 0.f;
          if (!h) r[2 * lane + 1] = lane < dim ? a : 0.f;
        }
        if (lane == 0) {
          r[2 * md + h] = slack;
          r[2 * md + 2 + h] = big;
          if (!h) {
            r[2 * md + 1] = slack;
            r[2 * md + 3] = big;
          }
        }
      }
    }
    __syncthreads();
    const float bb = face[dim];
    float fk[kMaxDim];
#pragma unroll
    for (int k = 0; k < kMaxDim; ++k) fk[k] = k < dim ? face[k] : 0.f;
#pragma unroll
    for (int r = 0; r < kFaceRegs; ++r) {
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < kMaxDim; ++k)
        if (k < dim) v = __fmaf_rn(fk[k], x[r][k], v);
      v = __fsub_rn(v, bb);
      if (EDIT ? !(v < 0.f) : v > 0.f) d[r] = none;
    }
    for (int i = tid + kFaceRegs * nt; i < K; i += nt) {
      if (!(dist[i] < FLT_MAX)) continue;
      float v = 0.f;
      for (int k = 0; k < dim; ++k) v = __fmaf_rn(face[k], cols[(size_t)i * dim + k], v);
      v = __fsub_rn(v, bb);
      if (EDIT ? !(v < 0.f) : v > 0.f) dist[i] = FLT_MAX;
    }
    ++nf;
  }
  return placed;
}

// EI-ZO's iteration: places the faces and updates the region's count and the counters.
static __device__ __forceinline__ void faces_block(int K, int dim, int max_faces, int capacity, float margin,
                                                   const float* __restrict__ ls, const float* __restrict__ le,
                                                   const float* __restrict__ cols, const float* __restrict__ proj,
                                                   float* __restrict__ dist, float* __restrict__ A,
                                                   float* __restrict__ b, int* __restrict__ num_faces,
                                                   EizoCounters* cnt, float* __restrict__ rows) {
  const int nf = *num_faces;
  int status = 0;
  const int placed =
      place_faces<false>(K, dim, max_faces, nf, capacity, margin, ls, le, cols, proj, dist, A, b, rows, &status);
  if (threadIdx.x == 0) {
    *num_faces = nf + placed;
    cnt->placed = (uint32_t)placed;
    cnt->status = status;
  }
}

}  // namespace csd
