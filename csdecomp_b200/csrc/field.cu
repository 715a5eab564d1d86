// field.cu -- tables of the field path (check_field.cuh), built once per plant:
// the grid of cells over the world statics (on the device), the probes of the
// moving capsules, the link capsules and the moving-moving pairs by link pair.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "check_field.cuh"

namespace csd {

namespace {

constexpr int kFieldCells = 1 << 18;     // most cells of a grid (16 bytes each)
constexpr int kFieldMaxStatics = 1024;   // as the broad phase (cull_eligible)
constexpr size_t kFieldMinList = 1 << 16; // entries of the cells' lists, at least (one cell can list kFieldMaxStatics)
constexpr double kFieldMinEdge = 0.02;   // finer cells list the same statics
constexpr double kProbeGrowth = 1.2;     // a probe's radius over its capsule's, at most (more probes below it)
constexpr int kMaxProbes = 12;           // probes of one capsule
constexpr size_t kFieldStaticShared = 2048;  // static shared memory of a checking kernel, at most (a plant, work items)
// Largest coordinates (metres from the world's origin) of a grid's box and of a
// static's extents, and longest side of the box: up to there the FP32 rounding
// of a cell's centre (1 ulp of 128 m on each axis), of a probe's place in its
// cell (4 ulp of 64 m) and of a distance to a static (3 ulp of 128 m) stay below
// kFieldMargin together. On a rail (no bound on the reach) the box ends kFieldRail
// from the origin.
constexpr double kFieldGridLimit = 128, kFieldGridSide = 128, kFieldRail = 64, kFieldStaticLimit = 256;

struct FieldBuild {
  const float4* statics;  // WG poses
  const int* type;
  int S;
  float ox, oy, oz, h;
  int nx, ny, nz;
  float reach;            // statics farther from a cell's centre cannot be touched from the cell
  float cap;              // distance stored where nothing is nearer
  uint4* cells;
  uint16_t* list;
  unsigned list_cap;
  unsigned* used;         // entries of `list` in use
};

__device__ float static_distance(const FieldBuild& b, int s, const float* c) {
  const float4 a = b.statics[4 * s];
  const int ty = b.type[s];
  if (ty == G_SPHERE) {
    const float dx = c[0] - a.x, dy = c[1] - a.y, dz = c[2] - a.z;
    return sqrtf(dx * dx + dy * dy + dz * dz) - a.w;
  }
  if (ty == G_CAPSULE) {
    float C[8];
    load4f(b.statics + 4 * s, 2, C);
    return sqrtf(pt_seg_d2(c, C)) - C[3];
  }
  float B[16], e2 = 0.f;
  load4f(b.statics + 4 * s, 4, B);
  for (int i = 0; i < 3; ++i) {
    const float l = B[4 * i + 2] * c[2] + B[4 * i + 1] * c[1] + B[4 * i] * c[0] + B[4 * i + 3];
    const float e = fmaxf(fabsf(l) - B[12 + i], 0.f);
    e2 += e * e;
  }
  return sqrtf(e2);
}

// Block = 8 x 8 x 4 cells, thread per cell. The block first collects the
// statics that some cell of it can list (most blocks keep a few of hundreds),
// then each cell measures only those: 2^18 cells against 200 statics in 40 us,
// launched once per plant.
__global__ void __launch_bounds__(256) field_cells_kernel(FieldBuild b) {
  __shared__ uint16_t near[kFieldMaxStatics];
  __shared__ int num_near;
  const int t = threadIdx.x;
  const int bx = blockIdx.x * 8, by = blockIdx.y * 8, bz = blockIdx.z * 4;
  if (t == 0) num_near = 0;
  __syncthreads();
  const float bc[3] = {b.ox + (bx + 4.f) * b.h, b.oy + (by + 4.f) * b.h, b.oz + (bz + 2.f) * b.h};
  // centres of the block's cells lie within (3.5, 3.5, 1.5) edges of its centre
  const float half = sqrtf(2.f * 3.5f * 3.5f + 1.5f * 1.5f) * b.h * 1.001f + 1e-4f;
  for (int s = t; s < b.S; s += 256)
    if (!(static_distance(b, s, bc) > b.reach + half)) near[atomicAdd(&num_near, 1)] = (uint16_t)s;
  __syncthreads();
  const int ix = bx + (t & 7), iy = by + ((t >> 3) & 7), iz = bz + (t >> 6);
  if (ix >= b.nx || iy >= b.ny || iz >= b.nz) return;
  const float c[3] = {b.ox + (ix + 0.5f) * b.h, b.oy + (iy + 0.5f) * b.h, b.oz + (iz + 0.5f) * b.h};
  float dmin = b.cap;
  int cnt = 0;
  uint32_t w[3] = {0u, 0u, 0u};
  for (int k = 0; k < num_near; ++k) {
    const int s = near[k];
    const float d = static_distance(b, s, c);
    if (d > b.reach) continue;
    dmin = fminf(dmin, d);
    if (cnt < 6) w[cnt >> 1] |= (uint32_t)s << ((cnt & 1) * 16);
    ++cnt;
  }
  if (cnt > 6) {
    const unsigned at = atomicAdd(b.used, (unsigned)cnt);
    if (at + (unsigned)cnt <= b.list_cap) {  // (otherwise the host builds again with fewer cells)
      unsigned j = at;
      for (int k = 0; k < num_near; ++k)
        if (!(static_distance(b, near[k], c) > b.reach)) b.list[j++] = near[k];
      w[0] = at;
    }
  }
  // padded (the FP32 distances are off by far less) and rounded down
  const unsigned short dh = __half_as_ushort(__float2half_rd(fmaxf(dmin - 1e-5f, 0.f)));
  b.cells[((size_t)iz * b.ny + iy) * b.nx + ix] = make_uint4((unsigned)dh | (unsigned)cnt << 16, w[0], w[1], w[2]);
}

struct Ball {
  double c[3], r;
};

double seg_dist(const double* p, const double* a, const double* u, double hl) {
  double d[3], t = 0;
  for (int k = 0; k < 3; ++k) {
    d[k] = p[k] - a[k];
    t += d[k] * u[k];
  }
  t = std::max(-hl, std::min(hl, t));
  double s = 0;
  for (int k = 0; k < 3; ++k) s += (d[k] - t * u[k]) * (d[k] - t * u[k]);
  return std::sqrt(s);
}

// Capsule around balls: the axis along the farthest pair of centres, radius
// the largest distance to it, padded as the broad phase's spheres.
void fit_capsule(const std::vector<Ball>& balls, float* out) {
  size_t bi = 0, bj = 0;
  double best = 0;
  for (size_t i = 0; i < balls.size(); ++i)
    for (size_t j = i + 1; j < balls.size(); ++j) {
      double s = 0;
      for (int k = 0; k < 3; ++k) s += (balls[i].c[k] - balls[j].c[k]) * (balls[i].c[k] - balls[j].c[k]);
      if (s > best) {
        best = s;
        bi = i;
        bj = j;
      }
    }
  const double len = std::sqrt(best);
  double a[3], u[3] = {1, 0, 0}, r = 0;
  for (int k = 0; k < 3; ++k) {
    a[k] = 0.5 * (balls[bi].c[k] + balls[bj].c[k]);
    if (len > 1e-9) u[k] = (balls[bj].c[k] - balls[bi].c[k]) / len;
  }
  const double hl = len > 1e-9 ? 0.5 * len : 0.0;
  for (const Ball& q : balls) r = std::max(r, seg_dist(q.c, a, u, hl) + q.r);
  for (int k = 0; k < 3; ++k) {
    out[k] = (float)a[k];
    out[4 + k] = (float)u[k];
  }
  out[3] = (float)(r * (1 + 1e-6) + 1e-4);
  out[7] = (float)hl;
}

}  // namespace

// Whether every number of the plant's geometry is one the tables are made for:
// finite, radii and half extents not negative, statics within
// kFieldStaticLimit. Other plants keep the pair sweep.
static bool ordinary_geometry(const HostPlant& hp, const std::vector<FkJoint>& fk) {
  auto within = [](const float* v, int n, float lo, float hi) {
    bool ok = true;
    for (int i = 0; i < n; ++i) ok = ok && v[i] >= lo && v[i] <= hi;
    return ok;
  };
  constexpr float kLim = (float)kFieldStaticLimit;
  bool ok = true;
  for (const FkJoint& j : fk)
    ok = ok && within(j.P, 9, -4.f, 4.f) && within(j.S, 9, -4.f, 4.f) && within(j.T, 9, -4.f, 4.f) &&
         within(j.t, 3, -kLim, kLim) && within(j.v, 3, -4.f, 4.f);
  for (const MovingGeom& g : hp.moving)
    ok = ok && within(g.p, 3, -kLim, kLim) && within(&g.r, 1, 0.f, kLim) &&
         (g.type == G_SPHERE || (within(&g.hl, 1, 0.f, kLim) && within(g.z, 3, -2.f, 2.f)));
  for (size_t s = 0; s < hp.static_type.size(); ++s) {
    const float* W = hp.statics.data() + 16 * s;
    if (hp.static_type[s] == G_SPHERE)
      ok = ok && within(W, 3, -kLim, kLim) && within(W + 3, 1, 0.f, kLim);
    else if (hp.static_type[s] == G_CAPSULE)
      ok = ok && within(W, 3, -kLim, kLim) && within(W + 3, 1, 0.f, kLim) && within(W + 4, 3, -2.f, 2.f) &&
           within(W + 7, 1, 0.f, kLim);
    else
      ok = ok && within(W, 12, -kLim, kLim) && within(W + 12, 3, 0.f, kLim);
  }
  return ok;
}

csd_status_t build_field(csd_plant_s* h, const std::vector<FkJoint>& fk, const std::vector<uint32_t>& moving_pairs,
                         const std::vector<uint32_t>& world_bits, const std::vector<float>& rounded,
                         const std::vector<double>& static_box, const std::vector<double>& reach_box) {
  DevPlant& dp = h->dp;
  const HostPlant& hp = h->host;
  const int S = dp.num_static, M = dp.num_moving, NS = dp.num_slots;
  dp.has_field = 0;
  if (!h->cull_eligible || M == 0 || M > 0xffff || S > kFieldMaxStatics || dp.num_msph + dp.num_mcap != M ||
      !ordinary_geometry(hp, fk))
    return CSD_OK;
  FieldTables f{};
  // ---- geometries, probes, link capsules
  std::vector<float> geom((size_t)M * 4), axis, probes, link((size_t)NS * 8, 0.f);
  std::vector<std::vector<Ball>> balls(NS);
  double max_r = 0;
  for (int m = 0; m < M; ++m) {
    const MovingGeom& g = hp.moving[m];
    for (int k = 0; k < 3; ++k) geom[4 * m + k] = g.p[k];
    geom[4 * m + 3] = g.r;
    if (g.type == G_SPHERE) {
      max_r = std::max(max_r, (double)g.r);
      balls[g.slot].push_back({{g.p[0], g.p[1], g.p[2]}, g.r});
      continue;
    }
    for (int k = 0; k < 3; ++k) axis.push_back(g.z[k]);
    axis.push_back(g.hl);
    for (int sg = -1; sg <= 1; sg += 2)
      balls[g.slot].push_back({{g.p[0] + (double)sg * g.hl * g.z[0], g.p[1] + (double)sg * g.hl * g.z[1],
                                g.p[2] + (double)sg * g.hl * g.z[2]}, g.r});
    // n centres from end to end: every point of the capsule is within sqrt(r^2 + (spacing / 2)^2) of one
    int n = g.hl > 0.f ? 2 : 1;
    auto radius = [&](int k) {
      const double half = k > 1 ? g.hl / (k - 1.0) : 0.0;
      return std::sqrt((double)g.r * g.r + half * half);
    };
    while (n > 1 && n < kMaxProbes && radius(n) > kProbeGrowth * g.r) ++n;
    const double rad = radius(n) * (1 + 1e-6) + 1e-5;
    max_r = std::max(max_r, rad);
    const int q = m - dp.num_msph;
    float qf;
    std::memcpy(&qf, &q, 4);
    for (int k = 0; k < n; ++k) {
      probes.push_back(n > 1 ? (float)(-g.hl + 2.0 * g.hl * k / (n - 1.0)) : 0.f);
      probes.push_back((float)rad);
      probes.push_back(qf);
      probes.push_back(0.f);
    }
  }
  for (int k = 0; k < NS; ++k) {
    if (balls[k].empty())
      link[8 * k + 3] = -1.f;
    else
      fit_capsule(balls[k], &link[8 * k]);
  }
  // ---- moving-moving pairs by link pair, then by type, in the order given (a counting sort: a tree of vectors cost
  // plant creation 0.2 to 0.4 ms for some 3,000 pairs)
  auto bucket = [&](uint32_t w) {
    const MovingGeom &a = hp.moving[w & 0xffffu], &b = hp.moving[w >> 16];
    const int ty = (a.type == G_CAPSULE) + (b.type == G_CAPSULE);
    return (std::min(a.slot, b.slot) * NS + std::max(a.slot, b.slot)) * 3 + ty;
  };
  std::vector<int> begin((size_t)NS * NS * 3 + 1, 0);
  for (uint32_t w : moving_pairs) ++begin[bucket(w) + 1];
  for (size_t k = 1; k < begin.size(); ++k) begin[k] += begin[k - 1];
  std::vector<LinkPair> lps;
  for (int k = 0; k < NS * NS; ++k) {
    const int* o = &begin[3 * k];
    if (o[3] > o[0]) lps.push_back({k / NS, k % NS, o[0], o[1] - o[0], o[2] - o[1], o[3] - o[2]});
  }
  std::vector<uint32_t> pairs(moving_pairs.size());
  for (uint32_t w : moving_pairs) pairs[begin[bucket(w)]++] = w;
  // ---- FK table
  std::vector<float> entry((size_t)dp.num_fk * 36, 0.f);
  for (int j = 0; j < dp.num_fk; ++j)
    for (int i = 0; i < 9; ++i) {
      float* e = &entry[(size_t)(9 * j + i) * 4];
      e[0] = fk[j].P[i];
      e[1] = fk[j].S[i];
      e[2] = fk[j].T[i];
      e[3] = i < 3 ? fk[j].t[i] : i < 6 ? fk[j].v[i - 3] : 0.f;
    }
  // FK schedule of `width` lane groups per configuration: the joints whose
  // parents are done, a joint staying with the group that holds its parent's row
  auto schedule = [&](int width) {
    std::vector<uint32_t> steps;
    std::vector<int> step_of(dp.num_fk, -1), group_of(dp.num_fk, -1);
    std::vector<int> last(width, -1);
    for (int done = 0, s = 0; done < dp.num_fk; ++s) {
      std::vector<int> job(width, -1);
      for (int pass = 0; pass < 2; ++pass)
        for (int j = 0; j < dp.num_fk; ++j) {
          const int par = fk[j].parent;
          if (step_of[j] >= 0 || (par >= 0 && (step_of[par] < 0 || step_of[par] == s))) continue;
          int g = -1;
          if (pass == 0) {
            if (par >= 0 && last[group_of[par]] == par && job[group_of[par]] < 0) g = group_of[par];
          } else {
            for (int k = 0; k < width && g < 0; ++k)
              if (job[k] < 0) g = k;
          }
          if (g < 0) continue;
          job[g] = j;
          step_of[j] = s;
          group_of[j] = g;
          ++done;
        }
      uint32_t sync = 0;
      std::vector<uint32_t> w(width);
      for (int g = 0; g < width; ++g) {
        const int j = job[g];
        uint32_t par = 253;
        if (j >= 0 && fk[j].parent >= 0) par = last[g] == fk[j].parent ? 254u : (uint32_t)fk[j].parent;
        if (j >= 0 && par < 253) sync = 1u << 31;
        w[g] = (j < 0 ? 255u : (uint32_t)j) | par << 8 | (j >= 0 && fk[j].type == J_REVOLUTE ? 1u << 16 : 0u);
      }
      for (int g = 0; g < width; ++g) {
        steps.push_back(w[g] | sync);
        if (job[g] >= 0) last[g] = job[g];
      }
    }
    return steps;
  };
  // more groups per configuration while they nearly halve its steps
  std::vector<uint32_t> steps = schedule(1);
  f.fk_branches = 1;
  for (int width = 2; width <= 4; width *= 2) {
    std::vector<uint32_t> wider = schedule(width);
    if (10 * (wider.size() / width) > 6 * (steps.size() / f.fk_branches)) break;
    steps = wider;
    f.fk_branches = width;
  }
  f.fk_steps = (int)steps.size() / f.fk_branches;
  f.fk_batch = std::min(kFkBatch / f.fk_branches, dp.num_slots <= 8 ? 8 : dp.num_slots <= 16 ? 4 : 2);
  // a block's warps have to fit: fewer configurations at once (their slot transforms are most of what the pair
  // sweep does not need), or the pair sweep
  int shared = 0;
  CSD_CUDA_TRY(cudaDeviceGetAttribute(&shared, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device));
  auto fits = [&] {
    DevPlant t = dp;
    t.field = f;
    return (size_t)field_warp_floats(t) * sizeof(float) * kWarpsPerBlock + kFieldStaticShared <= (size_t)shared;
  };
  while (f.fk_batch > 1 && !fits()) f.fk_batch /= 2;
  if (!fits()) return CSD_OK;
  // ---- grid over the part of the padded statics' box that the robot reaches
  double lo[3], hi[3], edge = 0;
  auto set_grid = [&](double e) {  // cells of edge e or the least larger one that keeps their number
    int n[3];
    for (edge = e;; edge *= 1.01) {
      for (int k = 0; k < 3; ++k) n[k] = (int)std::min(1e6, std::ceil((hi[k] - lo[k]) / edge));
      if ((double)n[0] * n[1] * n[2] <= kFieldCells) break;
    }
    f.h = (float)edge;
    f.inv_h = (float)(1.0 / edge);
    f.ox = (float)lo[0];
    f.oy = (float)lo[1];
    f.oz = (float)lo[2];
    f.nx = n[0];
    f.ny = n[1];
    f.nz = n[2];
  };
  if (S > 0) {
    double vol = 1;
    for (int k = 0; k < 3; ++k) {
      const double pad = max_r * (1 + 1e-6) + 1e-3;
      f.far_lo[k] = (float)(static_box[k] - pad);
      f.far_hi[k] = (float)(static_box[3 + k] + pad);
      const bool rail = reach_box[k] < -1e299;  // a prismatic joint: probes beyond the grid test every static
      lo[k] = std::max((double)f.far_lo[k], rail ? -kFieldRail : reach_box[k]);
      hi[k] = std::min((double)f.far_hi[k], rail ? kFieldRail : reach_box[3 + k]);
      if (rail && hi[k] <= lo[k]) return CSD_OK;
      hi[k] = std::max(lo[k] + 1e-3, hi[k]);
      if (lo[k] < -kFieldGridLimit || hi[k] > kFieldGridLimit || hi[k] - lo[k] > kFieldGridSide) return CSD_OK;
      vol *= hi[k] - lo[k];
    }
    set_grid(std::max(std::cbrt(vol / kFieldCells), kFieldMinEdge));
  }
  bool all = true;
  f.pair_words = (S + 31) / 32;
  for (int m = 0; m < M && all; ++m)
    for (int s = 0; s < S; ++s) all = all && ((world_bits[(size_t)m * f.pair_words + (s >> 5)] >> (s & 31)) & 1u);
  // ---- upload
  const size_t cells = (size_t)f.nx * f.ny * f.nz, list_cap = std::max<size_t>(8 * cells, kFieldMinList);
  size_t off = 0;
  auto section = [&](size_t bytes) {
    const size_t o = off;
    off = (off + std::max<size_t>(bytes, 16) + 255) & ~size_t(255);
    return o;
  };
  const size_t o_geom = section(geom.size() * 4), o_axis = section(axis.size() * 4),
               o_probe = section(probes.size() * 4), o_link = section(link.size() * 4),
               o_lp = section(lps.size() * sizeof(LinkPair)), o_pairs = section(pairs.size() * 4),
               o_entry = section(entry.size() * 4), o_step = section(steps.size() * 4),
               o_round = section(rounded.size() * 4), o_bits = section(all ? 0 : world_bits.size() * 4),
               o_used = section(16), host_bytes = off, o_cells = section(cells * 16), o_list = section(list_cap * 2);
  std::vector<char> blob(host_bytes, 0);
  auto put = [&](size_t o, const void* src, size_t n) {
    if (n) std::memcpy(blob.data() + o, src, n);
  };
  put(o_geom, geom.data(), geom.size() * 4);
  put(o_axis, axis.data(), axis.size() * 4);
  put(o_probe, probes.data(), probes.size() * 4);
  put(o_link, link.data(), link.size() * 4);
  put(o_lp, lps.data(), lps.size() * sizeof(LinkPair));
  put(o_pairs, pairs.data(), pairs.size() * 4);
  put(o_entry, entry.data(), entry.size() * 4);
  put(o_step, steps.data(), steps.size() * 4);
  put(o_round, rounded.data(), rounded.size() * 4);
  if (!all) put(o_bits, world_bits.data(), world_bits.size() * 4);
  CSD_CUDA_TRY(cudaMalloc(&h->field_blob, off));
  CSD_CUDA_TRY(cudaMemcpy(h->field_blob, blob.data(), host_bytes, cudaMemcpyHostToDevice));
  char* base = (char*)h->field_blob;
  f.cells = (const uint4*)(base + o_cells);
  f.list = (const uint16_t*)(base + o_list);
  f.rounded = (const float4*)(base + o_round);
  f.pair_bits = all ? nullptr : (const uint32_t*)(base + o_bits);
  f.geom = (const float4*)(base + o_geom);
  f.cap_axis = (const float4*)(base + o_axis);
  f.probes = (const float4*)(base + o_probe);
  f.num_probes = (int)probes.size() / 4;
  f.link_cap = (const float4*)(base + o_link);
  f.link_pairs = (const LinkPair*)(base + o_lp);
  f.num_link_pairs = (int)lps.size();
  f.pairs = (const uint32_t*)(base + o_pairs);
  f.fk_entry = (const float4*)(base + o_entry);
  f.fk_step = (const uint32_t*)(base + o_step);
  if (S > 0) {
    FieldBuild b{};
    b.statics = dp.statics;
    b.type = dp.static_type;
    b.S = S;
    b.cells = (uint4*)(base + o_cells);
    b.list = (uint16_t*)(base + o_list);
    b.list_cap = (unsigned)list_cap;
    b.used = (unsigned*)(base + o_used);
    auto keep_sweep = [&] {
      cudaFree(h->field_blob);
      h->field_blob = nullptr;
      return CSD_OK;
    };
    for (bool first = true;; first = false) {
      b.ox = f.ox;
      b.oy = f.oy;
      b.oz = f.oz;
      b.h = f.h;
      b.nx = f.nx;
      b.ny = f.ny;
      b.nz = f.nz;
      const double half = 0.5 * std::sqrt(3.0) * f.h;
      b.reach = (float)((max_r + half) * (1 + 1e-5) + 3e-4);
      b.cap = (float)(max_r + half + 2.5e-4);
      const dim3 grid((f.nx + 7) / 8, (f.ny + 7) / 8, (f.nz + 3) / 4);
      if (grid.y > 65535u || grid.z > 65535u) return keep_sweep();  // a sliver of a box: not worth a grid
      field_cells_kernel<<<grid, 256>>>(b);
      CSD_CUDA_TRY(cudaGetLastError());
      // (the copy waits for the kernel: the tables are read from any stream after this)
      unsigned used = 0;
      CSD_CUDA_TRY(cudaMemcpy(&used, b.used, sizeof(used), cudaMemcpyDeviceToHost));
      // One probe much larger than the others makes every list long. Up to about S / 25 entries a cell the field path
      // is the faster (131,072 configurations of an arm with one sphere of 0.3 to 1 m among 900, 300 and 100 small
      // statics: 1.0 -> 0.4 ms against the pair sweep with 26 entries, 1.0 -> 1.2 with 50; 0.54 -> 0.26 with 8,
      // 0.54 -> 0.61 with 16; 0.34 -> 0.25 with 4, 0.35 -> 0.46 with 7).
      if (first && used > (2.0 + S / 25.0) * cells) return keep_sweep();
      if (used <= list_cap) break;
      // The lists do not fit. Wider cells list little more each (the large probe's radius decides), so fewer of them
      // do; with cells without room testing every static those arms took 3.7 to 5.5 ms.
      set_grid(1.03 * edge * std::cbrt((double)used / list_cap));
      CSD_CUDA_TRY(cudaMemset(b.used, 0, sizeof(used)));
    }
  }
  dp.field = f;
  dp.has_field = 1;
  return CSD_OK;
}

}  // namespace csd
