// voxgrid.cu -- per-call spatial hash grid over the voxels of a voxel check.
//
// Reference: checkCollisionFreeVoxelsCuda (cuda_collision_checker.cu:374-435)
// tests every robot geometry against every voxel (a pair buffer of
// geometries x MAX_NUM_VOXELS per configuration). Here the voxels of a call
// are bucketed once on the device (count, sums, scan, scatter: four launches,
// O(voxels)), and each robot geometry tests only the voxels in the cells its
// bounding sphere touches (check_core.cuh::grid_geom_hit) or, a capsule, its
// probe spheres touch (check_field.cuh::field_voxels). The cell edge is about
// a robot sphere's diameter plus the voxel diameter, so a sphere visits at
// most 8 cells, in 4 columns; for many configurations the cells are half that
// wide and list the voxels around them too, so that it visits one
// (build_voxel_grid).
#include <algorithm>
#include <vector>

#include "check_core.cuh"

namespace csd {

constexpr int kScanBlock = 1024;  // buckets one block of the scan covers
constexpr int kVoxSpan = 3;       // cells per axis that list one voxel, at most

// Buckets of the cells that list voxel (x, y, z): f(bucket). With rins > 0 these
// are the cells within rins of it, at most kVoxSpan per axis: the cell edge
// exceeds 1.01 rins. Every operation rounds by itself: the count and the
// scatter have to name the same buckets.
template <typename F>
__device__ __forceinline__ void voxel_cells(float x, float y, float z, float inv_h, float rins, int mask, F f) {
  if (!(rins > 0.f)) {
    f(vox_bucket(vox_cell(x, inv_h), vox_cell(y, inv_h), vox_cell(z, inv_h), mask));
    return;
  }
  const float v[3] = {x, y, z}, h = 1.f / inv_h;
  float d2[3][kVoxSpan];  // squared distance to the cells of each axis
  int lo[3], n[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    lo[i] = vox_cell(__fsub_rn(v[i], rins), inv_h);
    n[i] = min(vox_cell(__fadd_rn(v[i], rins), inv_h) - lo[i] + 1, kVoxSpan);
#pragma unroll
    for (int j = 0; j < kVoxSpan; ++j) {
      const float a = __fmul_rn((float)(lo[i] + j), h);
      const float e = fmaxf(fmaxf(__fsub_rn(a, v[i]), __fsub_rn(v[i], __fadd_rn(a, h))), 0.f);
      d2[i][j] = __fmul_rn(e, e);
    }
  }
  const float far2 = __fmul_rn(__fmul_rn(rins, rins), 1.001f);
#pragma unroll
  for (int i = 0; i < kVoxSpan; ++i)
#pragma unroll
    for (int j = 0; j < kVoxSpan; ++j)
#pragma unroll
      for (int k = 0; k < kVoxSpan; ++k)
        if (i < n[0] && j < n[1] && k < n[2] && !(__fadd_rn(__fadd_rn(d2[0][i], d2[1][j]), d2[2][k]) > far2))
          f(vox_bucket(lo[0] + i, lo[1] + j, lo[2] + k, mask));
}

__global__ void vox_count_kernel(const float* __restrict__ vox, int nv, float inv_h, float rins, int mask,
                                 int* __restrict__ cnt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x)
    voxel_cells(vox[3 * i], vox[3 * i + 1], vox[3 * i + 2], inv_h, rins, mask,
                [&](uint32_t b) { atomicAdd(cnt + b, 1); });
}

// Counts of each run of 1,024 buckets.
__global__ void __launch_bounds__(kScanBlock / 4) vox_sum_kernel(const int* __restrict__ cnt, int* __restrict__ block_cnt,
                                                                 int B) {
  __shared__ int part[kScanBlock / 128];
  const int t = threadIdx.x, b = blockIdx.x * kScanBlock + 4 * t;
  int4 c = make_int4(0, 0, 0, 0);
  if (b < B) c = *reinterpret_cast<const int4*>(cnt + b);  // B is a multiple of 256
  const int s = __reduce_add_sync(0xffffffffu, c.x + c.y + c.z + c.w);
  if ((t & 31) == 0) part[t >> 5] = s;
  __syncthreads();
  if (t == 0) {
    int sum = 0;
    for (int w = 0; w < kScanBlock / 128; ++w) sum += part[w];
    block_cnt[blockIdx.x] = sum;
  }
}

// Exclusive scan of the bucket counts in place (start[B] = total), copied to
// the scatter cursors. A block takes 1,024 buckets, four per thread, and sums
// the counts of the blocks before it itself (vox_sum_kernel), so no block waits
// on another. One block over everything was bound by its threads' serial,
// uncoalesced loads: 81 us for 32,768 buckets, 2.3 us with a block each 1,024.
__global__ void __launch_bounds__(kScanBlock / 4) vox_scan_kernel(int* __restrict__ start, int* __restrict__ cursor,
                                                                  const int* __restrict__ block_cnt, int B) {
  __shared__ int part[kScanBlock / 128], before[kScanBlock / 128];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, b = blockIdx.x * kScanBlock + 4 * t;
  int prev = 0;
  for (int i = t; i < (int)blockIdx.x; i += kScanBlock / 4) prev += block_cnt[i];
  prev = __reduce_add_sync(0xffffffffu, prev);
  int4 c = make_int4(0, 0, 0, 0);
  if (b < B) c = *reinterpret_cast<const int4*>(start + b);  // B is a multiple of 256
  int s = c.x + c.y + c.z + c.w;
  const int mine = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += v;
  }
  if (lane == 31) part[warp] = s;
  if (lane == 0) before[warp] = prev;
  __syncthreads();
  int run = s - mine;
#pragma unroll
  for (int w = 0; w < kScanBlock / 128; ++w) run += before[w] + (w < warp ? part[w] : 0);
  if (b < B) {
    const int4 v = make_int4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
    *reinterpret_cast<int4*>(start + b) = v;
    *reinterpret_cast<int4*>(cursor + b) = v;
  }
  if (b < B && b + 4 >= B) start[B] = run + mine;
}

__global__ void vox_fill_kernel(const float* __restrict__ vox, int nv, float inv_h, float rins, int mask,
                                int* __restrict__ cursor, float4* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
    const float x = vox[3 * i], y = vox[3 * i + 1], z = vox[3 * i + 2];
    voxel_cells(x, y, z, inv_h, rins, mask,
                [&](uint32_t b) { out[atomicAdd(cursor + b, 1)] = make_float4(x, y, z, 0.f); });
  }
}

VoxelReach voxel_reach(const csd_plant_s* p, const std::vector<uint32_t>& tab, float vr) {
  std::vector<float> r;
  const int T = p->dp.num_tiles;
  for (int t = 0; t < T && t < (int)tab.size(); ++t)
    for (int l = 0; l < kWarp; ++l)
      if ((tab[t] >> l) & 1u) r.push_back(p->host.moving[t * kWarp + l].r);
  if (r.empty()) r.push_back(0.05f);
  std::nth_element(r.begin(), r.begin() + r.size() / 2, r.end());
  const float med = r[r.size() / 2], top = *std::max_element(r.begin(), r.end());
  return {med + std::max(vr, 0.f), top + std::max(vr, 0.f)};
}

// Cells that list voxels from around them, or only their own? Around: a robot
// sphere looks up one cell and tests the voxels within reach of that cell (21
// cell volumes' worth, edge = reach), in place of the 8 cells of twice the edge
// that its box touches (64 of those volumes). Measured at 262,147
// configurations, 10,000 voxels: 1.08 -> 0.55 ms for the check kernel. A voxel is then written up to
// 27 times (23 us of building at 10,000 voxels against 8), which a few configurations do
// not repay, and takes up to 27 entries, so the lists of more than
// kVoxAroundMax voxels (28 MB) stay cells' own.
constexpr int64_t kVoxAroundChecks = 4096;
constexpr int kVoxAroundMax = 1 << 16;

csd_status_t build_voxel_grid(const csd_plant_s* p, VoxelReach reach, int64_t checks, DevBuf* buf, VoxelTables* vt,
                              cudaStream_t st) {
  vt->gvox = nullptr;
  vt->gstart = nullptr;
  if (!p->vox_grid || vt->nv < kVoxGridMinVoxels || !(reach.med > 0.f)) return CSD_OK;
  const int nv = vt->nv;
  const bool around = checks >= kVoxAroundChecks && nv <= kVoxAroundMax;
  // the spheres' padded reach (check_field.cuh), the larger ones' up to half as much again as the median's
  const float rins = around ? std::min(reach.max, 1.5f * reach.med) * 1.001f + 1e-4f : 0.f;
  const float cell = std::max(around ? 1.02f * rins : 2.f * reach.med, 1e-3f);
  const int64_t entries = around ? (int64_t)nv * kVoxSpan * kVoxSpan * kVoxSpan : nv;
  int B = 256;
  while (B < (around ? entries : 2 * entries) && B < (1 << 24)) B <<= 1;
  const int nb = (B + kScanBlock - 1) / kScanBlock;
  const size_t o_blk = ((size_t)(B + 1) * 4 + 15) & ~size_t(15);  // [start | block counts | cursors | voxels]
  const size_t o_cur = (o_blk + (size_t)nb * 4 + 15) & ~size_t(15);
  const size_t o_vox = o_cur + (size_t)B * 4;
  csd_status_t s;
  if ((s = buf->reserve(o_vox + (size_t)entries * 16))) return s;
  char* base = buf->as<char>();
  int* start = reinterpret_cast<int*>(base);
  int* block_cnt = reinterpret_cast<int*>(base + o_blk);
  int* cursor = reinterpret_cast<int*>(base + o_cur);
  float4* gvox = reinterpret_cast<float4*>(base + o_vox);
  const float inv_h = 1.f / cell;
  CSD_CUDA_TRY(cudaMemsetAsync(start, 0, o_cur, st));
  const int grid = std::max(1, std::min((nv + 63) / 64, 8 * device_sm_count()));
  vox_count_kernel<<<grid, 64, 0, st>>>(vt->vox, nv, inv_h, rins, B - 1, start);
  vox_sum_kernel<<<nb, kScanBlock / 4, 0, st>>>(start, block_cnt, B);
  vox_scan_kernel<<<nb, kScanBlock / 4, 0, st>>>(start, cursor, block_cnt, B);
  vox_fill_kernel<<<grid, 64, 0, st>>>(vt->vox, nv, inv_h, rins, B - 1, cursor, gvox);
  CSD_CUDA_TRY(cudaGetLastError());
  vt->gvox = gvox;
  vt->gstart = start;
  vt->gmask = B - 1;
  vt->ginv_h = inv_h;
  vt->grins = rins;
  return CSD_OK;
}

}  // namespace csd

using namespace csd;

extern "C" {

csd_status_t csd_plant_set_voxel_grid(csd_plant_t plant, int32_t enable) {
  CSD_CHECK(plant, CSD_ERR_INVALID, "null argument");
  plant->vox_grid = enable != 0;
  return CSD_OK;
}

}  // extern "C"
