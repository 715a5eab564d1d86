// edit.cu -- region editing (EditRegionsCuda) on the device.
//
// Reference: EditRegionsCuda (csdecomp/src/planning/cuda_edit_regions.cu:44-301)
// groups the collisions by segment on the host, then launches a projection
// kernel and 9 x (midpoint, FK, voxel check, bounds, store) plus a distance
// kernel, each step through global-memory transform and per-pair buffers, and
// places the faces on the host: per region an argsort of the distances and an
// Eigen loop that tests every candidate against all faces so far.
//
// Here the editing is two launches after one upload:
//   1. edit_bisect_kernel   one warp per collision (or a few collisions, where
//                            there are more than warps): projection onto its own
//                            segment, every bisection step a fused FK +
//                            collision check of the midpoint, distance to the
//                            projection (the EI-ZO bisection body,
//                            bisect_particles)
//   2. edit_faces_kernel    one block per region: copies the region, drops the
//                            candidates outside it, then repeatedly takes the
//                            nearest live candidate (lower index on ties),
//                            places its face with the segment relaxation of
//                            cuda_edit_regions.cu:262-272 and drops every
//                            candidate the new face cuts off. A candidate is
//                            placed exactly when the reference's ascending
//                            loop finds it strictly inside the region edited
//                            so far (:253-259): faces only accumulate, so
//                            "inside all faces so far" is "not cut off by the
//                            original region nor by a face placed before it".
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <vector>

#include "eizo_core.cuh"

namespace csd {

constexpr int kEditFaceThreads = 256;
constexpr int kEditMaxVoxels = 10000;  // MAX_NUM_VOXELS, cuda_edge_inflation_zero_order.h:13

template <int M, bool VOX>  // VOX: with voxels
__global__ void __launch_bounds__(32 * kWarpsPerBlock, ModeBlocks<M>::n)
    edit_bisect_kernel(DevPlant p, int K, int dim, int steps, const float* __restrict__ starts,
                       const float* __restrict__ ends, const uint32_t* __restrict__ seg, VoxArgs vox,
                       float* __restrict__ cols, float* __restrict__ proj, float* __restrict__ dist) {
  const VoxArgs va = VOX ? vox : VoxArgs{};
  extern __shared__ float4 smem4[];
  __shared__ uint64_t bar;
  const WarpCtx<M> w = warp_setup<M>(p, smem4, &bar);
  if (!w.ok) return;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (blockDim.x >> 5);
  const int B = bisect_batch<M>(p, K, nw);
  for (int i = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * B; i < K; i += nw * B)
    bisect_particles<M>(p, w, i, min(B, K - i), dim, steps, [&](int k) { return starts + (size_t)seg[k] * dim; },
                        [&](int k) { return ends + (size_t)seg[k] * dim; }, va, cols, proj, dist, lane);
}

// Region r: faces [face_off[r], face_off[r+1]) of A/b, candidates
// [coll_off[r], coll_off[r+1]) of cols/proj/dist; written at row
// face_off[r] + coll_off[r] of A_out/b_out. One block per region: copy, then
// place_faces. dist is consumed. (A warp per region left 64 regions of 512
// candidates to 64 warps: 519 us, 116 us with a block each.)
__global__ void __launch_bounds__(kEditFaceThreads)
    edit_faces_kernel(int m, int dim, float margin, const float* __restrict__ starts, const float* __restrict__ ends,
                      const float* __restrict__ A, const float* __restrict__ b, const int* __restrict__ face_off,
                      const int* __restrict__ coll_off, const float* __restrict__ cols,
                      const float* __restrict__ proj, float* __restrict__ dist, float* __restrict__ A_out,
                      float* __restrict__ b_out, int* __restrict__ num_faces) {
  for (int r = blockIdx.x; r < m; r += gridDim.x) {
    const int f0 = face_off[r], F0 = face_off[r + 1] - f0;
    const int c0 = coll_off[r], K = coll_off[r + 1] - c0;
    const int64_t row0 = (int64_t)f0 + c0;
    float* Ao = A_out + row0 * dim;
    float* bo = b_out + row0;
    for (int i = threadIdx.x; i < F0 * dim; i += blockDim.x) Ao[i] = A[(int64_t)f0 * dim + i];
    for (int i = threadIdx.x; i < F0; i += blockDim.x) bo[i] = b[f0 + i];
    __syncthreads();
    int status = 0;
    const int placed = place_faces<true>(K, dim, K, F0, F0 + K, margin, starts + (int64_t)r * dim,
                                         ends + (int64_t)r * dim, cols + (int64_t)c0 * dim, proj + (int64_t)c0 * dim,
                                         dist + c0, Ao, bo, nullptr, &status);
    if (threadIdx.x == 0) num_faces[r] = F0 + placed;
    __syncthreads();
  }
}

static bool point_in_region(const float* A, const float* b, int F, int d, const float* x) {
  // HPolyhedron::PointInSet (hpolyhedron.cpp:265-274), tolerance 1e-9 in FP32
  for (int f = 0; f < F; ++f) {
    float ax = 0.f;
    for (int k = 0; k < d; ++k) ax += A[(size_t)f * d + k] * x[k];
    if (!(ax <= b[f] + 1e-9f)) return false;
  }
  return true;
}

}  // namespace csd

using namespace csd;

extern "C" {

csd_status_t csd_edit_regions(csd_plant_t plant, const float* collisions, const uint32_t* line_segment_idxs,
                              int64_t n, const float* line_starts, const float* line_ends, int32_t m,
                              const float* A, const float* b, const int32_t* face_offsets, const float* voxels,
                              int32_t nv, float voxel_radius, const int32_t* robot_geometry_ids, int32_t nr,
                              const csd_edit_regions_options_t* options, float* A_out, float* b_out,
                              int32_t* num_faces, float* projections, float* optimized_collisions) {
  CSD_CHECK(plant && options && line_starts && line_ends && face_offsets && A && b && A_out && b_out && num_faces,
            CSD_ERR_INVALID, "null argument");
  CSD_CHECK(m >= 1, CSD_ERR_INVALID, "Regions vector cannot be empty");
  CSD_CHECK(n >= 0 && nv >= 0 && nr >= 0, CSD_ERR_INVALID, "negative size");
  // cuda_edit_regions.cu:55-83
  CSD_CHECK(nr >= 1 && robot_geometry_ids, CSD_ERR_INVALID, "Robot geometry IDs cannot be empty");
  CSD_CHECK(voxel_radius > 0.f, CSD_ERR_INVALID, "Voxel radius must be positive");
  CSD_CHECK(nv <= kEditMaxVoxels, CSD_ERR_CAPACITY, "Voxel buffer size insufficient");
  CSD_CHECK(nv == 0 || voxels, CSD_ERR_INVALID, "null voxels");
  const int d = plant->dp.dim;
  CSD_CHECK(d >= 1 && d <= kMaxDim, CSD_ERR_DIMENSION, "plant dimension must be in [1, 16]");
  CSD_CHECK(face_offsets[0] == 0, CSD_ERR_INVALID, "face_offsets[0] must be 0");
  for (int r = 0; r < m; ++r) {
    const int F = face_offsets[r + 1] - face_offsets[r];
    CSD_CHECK(F >= 0, CSD_ERR_INVALID, "face offsets must not decrease");
    const float* Ar = A + (size_t)face_offsets[r] * d;
    const float* br = b + face_offsets[r];
    CSD_CHECK(point_in_region(Ar, br, F, d, line_starts + (size_t)r * d), CSD_ERR_NOT_CONTAINED,
              "line start is not contained in region " + std::to_string(r));
    CSD_CHECK(point_in_region(Ar, br, F, d, line_ends + (size_t)r * d), CSD_ERR_NOT_CONTAINED,
              "line end is not contained in region " + std::to_string(r));
  }
  CSD_CHECK(n >= 1, CSD_ERR_INVALID,
            "[EditRegionsCuda] No collisions are contained in the regions, this is not supported.");
  CSD_CHECK(collisions && line_segment_idxs && projections && optimized_collisions, CSD_ERR_INVALID,
            "null argument");
  CSD_CHECK(n <= 0x7fffffff, CSD_ERR_CAPACITY, "too many collisions");
  // stable grouping by segment (cuda_edit_regions.cu:85-107)
  std::vector<int> coff(m + 1, 0);
  for (int64_t i = 0; i < n; ++i) {
    CSD_CHECK(line_segment_idxs[i] < (uint32_t)m, CSD_ERR_INVALID, "line segment index out of range");
    ++coff[line_segment_idxs[i] + 1];
  }
  for (int r = 0; r < m; ++r) coff[r + 1] += coff[r];
  const int F_total = face_offsets[m];
  std::vector<int> fill(coff.begin(), coff.end() - 1);
  std::vector<float> grouped((size_t)n * d);
  std::vector<uint32_t> gseg(n);
  for (int64_t i = 0; i < n; ++i) {
    const uint32_t s = line_segment_idxs[i];
    const int j = fill[s]++;
    std::memcpy(&grouped[(size_t)j * d], collisions + (size_t)i * d, sizeof(float) * d);
    gseg[j] = s;
  }
  std::vector<uint32_t> vtab;
  int num_other = 0;
  csd_status_t s;
  if ((s = build_voxel_tables(plant, robot_geometry_ids, nr, &vtab, &num_other))) return s;

  int cur = 0;
  cudaGetDevice(&cur);
  if (cur != plant->device) cudaSetDevice(plant->device);
  struct Restore {
    int cur, dev;
    ~Restore() {
      if (cur != dev) cudaSetDevice(cur);
    }
  } restore{cur, plant->device};

  // one device allocation for the call
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t sz_cols = al((size_t)n * d * 4), sz_dist = al((size_t)n * 4), sz_seg = al((size_t)n * 4);
  const size_t sz_ends = al((size_t)m * d * 4), sz_A = al((size_t)std::max(F_total, 1) * d * 4);
  const size_t sz_b = al((size_t)std::max(F_total, 1) * 4), sz_off = al((size_t)(m + 1) * 4);
  const size_t cap = (size_t)F_total + n;
  const size_t sz_Ao = al(cap * d * 4), sz_bo = al(cap * 4), sz_nf = al((size_t)m * 4);
  const size_t sz_vox = al((size_t)std::max(nv, 1) * 12), sz_vt = al((vtab.size() + 1) * 4);
  const size_t total = 2 * sz_cols + sz_dist + sz_seg + 2 * sz_ends + sz_A + sz_b + 2 * sz_off + sz_Ao + sz_bo +
                       sz_nf + sz_vox + sz_vt;
  const cudaStream_t st = 0;
  CallScratch buf(st);
  DevBuf grid_buf;
  if ((s = buf.reserve(total))) return s;
  char* base = buf.as<char>();
  size_t off = 0;
  auto take = [&](size_t x) {
    char* p = base + off;
    off += x;
    return p;
  };
  float* cols = (float*)take(sz_cols);
  float* proj = (float*)take(sz_cols);
  float* dist = (float*)take(sz_dist);
  uint32_t* seg = (uint32_t*)take(sz_seg);
  float* ls = (float*)take(sz_ends);
  float* le = (float*)take(sz_ends);
  float* Ad = (float*)take(sz_A);
  float* bd = (float*)take(sz_b);
  int* foff = (int*)take(sz_off);
  int* coffd = (int*)take(sz_off);
  float* Ao = (float*)take(sz_Ao);
  float* bo = (float*)take(sz_bo);
  int* nfd = (int*)take(sz_nf);
  float* vox = (float*)take(sz_vox);
  uint32_t* vt = (uint32_t*)take(sz_vt);
  CSD_CUDA_TRY(cudaMemcpyAsync(cols, grouped.data(), (size_t)n * d * 4, cudaMemcpyHostToDevice, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(seg, gseg.data(), (size_t)n * 4, cudaMemcpyHostToDevice, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(ls, line_starts, (size_t)m * d * 4, cudaMemcpyHostToDevice, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(le, line_ends, (size_t)m * d * 4, cudaMemcpyHostToDevice, st));
  if (F_total) {
    CSD_CUDA_TRY(cudaMemcpyAsync(Ad, A, (size_t)F_total * d * 4, cudaMemcpyHostToDevice, st));
    CSD_CUDA_TRY(cudaMemcpyAsync(bd, b, (size_t)F_total * 4, cudaMemcpyHostToDevice, st));
  }
  CSD_CUDA_TRY(cudaMemcpyAsync(foff, face_offsets, (size_t)(m + 1) * 4, cudaMemcpyHostToDevice, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(coffd, coff.data(), (size_t)(m + 1) * 4, cudaMemcpyHostToDevice, st));
  if (nv) CSD_CUDA_TRY(cudaMemcpyAsync(vox, voxels, (size_t)nv * 12, cudaMemcpyHostToDevice, st));
  if (!vtab.empty()) CSD_CUDA_TRY(cudaMemcpyAsync(vt, vtab.data(), vtab.size() * 4, cudaMemcpyHostToDevice, st));
  const bool staged = plant_mode(plant) != kModeField;  // only the pair sweep's staging wait can give up
  if (staged) CSD_CUDA_TRY(cudaMemsetAsync(plant->dp.status, 0, 4, st));
  VoxelTables vtab_dev;
  if (nv > 0) {
    vtab_dev.vox = vox;
    vtab_dev.nv = nv;
    vtab_dev.vr = voxel_radius;
    vtab_dev.tile_mask = vt;
    vtab_dev.other = vt + plant->dp.num_tiles;
    vtab_dev.num_other = num_other;
    if ((s = build_voxel_grid(plant, voxel_reach(plant, vtab, voxel_radius), n * (options->bisection_steps + 1),
                              &grid_buf, &vtab_dev, st)))
      return s;
  }
  const VoxArgs va = vox_args(vtab_dev);

  // 1. bisection
  const int K = (int)n, steps = (int)options->bisection_steps;
  s = with_mode(plant_mode(plant), [&](auto md) -> csd_status_t {
    constexpr int M = decltype(md)::value;
    auto kernel = va.nv > 0 ? edit_bisect_kernel<M, true> : edit_bisect_kernel<M, false>;
    const size_t smem = smem_bytes(plant, kWarpsPerBlock);
    int grid = 0;
    if (csd_status_t e = grid_for(kernel, smem, K, &grid, kWarpsPerBlock)) return e;
    kernel<<<grid, 32 * kWarpsPerBlock, smem, st>>>(plant->dp, K, d, steps, ls, le, seg, va, cols, proj, dist);
    return CSD_OK;
  });
  if (s) return s;
  CSD_CUDA_TRY(cudaGetLastError());
  // 2. faces, one block per region
  const int fgrid = std::min(m, 8 * device_sm_count());
  edit_faces_kernel<<<fgrid, kEditFaceThreads, 0, st>>>(m, d, options->configuration_margin, ls, le, Ad, bd, foff,
                                                        coffd, cols, proj, dist, Ao, bo, nfd);
  CSD_CUDA_TRY(cudaGetLastError());
  int kstat = 0;
  CSD_CUDA_TRY(cudaMemcpyAsync(num_faces, nfd, (size_t)m * 4, cudaMemcpyDeviceToHost, st));
  if (staged) CSD_CUDA_TRY(cudaMemcpyAsync(&kstat, plant->dp.status, 4, cudaMemcpyDeviceToHost, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(A_out, Ao, cap * d * 4, cudaMemcpyDeviceToHost, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(b_out, bo, cap * 4, cudaMemcpyDeviceToHost, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(projections, proj, (size_t)n * d * 4, cudaMemcpyDeviceToHost, st));
  CSD_CUDA_TRY(cudaMemcpyAsync(optimized_collisions, cols, (size_t)n * d * 4, cudaMemcpyDeviceToHost, st));
  CSD_CUDA_TRY(cudaStreamSynchronize(st));
  buf.settled();
  CSD_CHECK(kstat == 0, CSD_ERR_CUDA, "static geometry staging timed out in the bisection kernel");
  return CSD_OK;
}

}  // extern "C"
