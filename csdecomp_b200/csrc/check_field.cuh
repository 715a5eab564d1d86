// check_field.cuh -- collision check of one configuration by one warp for
// plants whose moving geometries are spheres and capsules.
//
// World pairs. The statics never move, so csd_plant_create lays a grid of
// cells over them (field.cu): each cell lists the statics that a sphere of at
// most the plant's largest probe radius centred in the cell can touch, with
// the distance from the cell's centre to the nearest of them. A lane places
// one moving sphere, reads its cell (one 16-byte load), and is done unless
// the distance, less the centre's offset in the cell, is below the radius;
// then it tests the listed statics (a handful) with the pair test of the full
// sweep. A moving capsule is covered by probe spheres along its axis; a static
// that meets one of them is tested against the capsule. A static missing from
// a cell's list is at least 1e-4 m clear of the probe, far above the rounding
// of the FP32 tests, so the verdict is the full sweep's.
//
// Self pairs. The geometry of each link lies in a capsule (host fit); one lane
// per link pair measures the distance of two link capsules, and only the pairs
// of links that overlap are swept, one geometry pair per lane.
//
// Why: with the link-sphere broad phase (check_core.cuh) 2^20 free
// configurations of the 7-DOF arm in 200 primitives took 9.9 ms, most of it
// in the group and static sphere tests and in the capsule-static and self
// pairs: they visit every static or most link pairs whatever the clearance.
// Work here is per moving geometry, about one cell read each: 1.65 ms (10^6
// uniform configurations 5.6 -> 1.1 ms, 40,009 edges 18.2 -> 2.9 ms). Still
// bound by instruction issue and by the latency of dependent loads, not by
// bandwidth. Cells of at most 2^18 per plant (4 MB, and as much for their
// lists): the radius plus half a cell diagonal bounds a list, so finer cells
// list little less.
#pragma once
#include <cuda_fp16.h>

#include "check_core.cuh"

namespace csd {

// Most configurations whose FK a warp runs at once (fk_rows).
constexpr int kFkBatch = 8;
static __host__ __device__ __forceinline__ int fk_batch(const DevPlant& p) { return p.field.fk_batch; }

// Per-warp shared memory (floats): slot transforms as rows
// [batch][slots][3][4], configurations [batch][kMaxDim], two spare ones
// [2][kMaxDim], world poses (first the sines and cosines of fk_rows), link
// capsules [slots][8].
static __host__ __device__ __forceinline__ int field_scratch_floats(const DevPlant& p) {
  const int a = (p.pose_words + 3) & ~3, b = (2 * fk_batch(p) * p.num_fk + 3) & ~3;
  return a > b ? a : b;
}
static __host__ __device__ __forceinline__ int field_warp_floats(const DevPlant& p) {
  return fk_batch(p) * (p.num_slots * 12 + kMaxDim) + 2 * kMaxDim + field_scratch_floats(p) + 8 * p.num_slots;
}

// FK of the m <= fk_batch configurations in qs [m][kMaxDim] into X
// [m][slots][3][4], rows (R[r][0..2], t[r]); sc: scratch.
//
// Sines and cosines first, one joint of one configuration per lane. Then the
// warp's eight groups of four lanes share out the configurations and, on
// trees with arms side by side, their branches: group h follows branch
// h % fk_branches of configuration h / fk_branches, and its lane r < 3 carries
// row r of the branch: per joint the nine local rotation entries, then twelve
// FMAs on the parent's row, which it still holds unless the joint branches
// off, each in the order of check_core.cuh::fk_warp. fk_step: joint (255:
// none), parent slot << 8 (254: the row in registers, 253: the world), bit 31:
// a parent row of this step comes from another group. Twelve lanes exchanging
// one configuration's entries took 0.6 of the 2.1 ms of 2^20 free
// configurations of the 7-DOF arm, eight configurations at once 0.2.
static __device__ __forceinline__ void fk_rows(const DevPlant& p, const float* qs, int m, float* X, float* sc,
                                               int lane) {
  const FieldTables& f = p.field;
  float2* sc2 = reinterpret_cast<float2*>(sc);
  const int nf = p.num_fk, ne = m * nf, nb = f.fk_branches;
  for (int e = lane; e < ne; e += kWarp) {
    const int g = e / nf;
    const FkJoint* J = p.fk + (e - g * nf);
    const float q = qs[g * kMaxDim + __ldg(&J->qidx)];
    float s = q, c = 0.f;  // prismatic: the joint value itself
    if (__ldg(&J->type) == J_REVOLUTE) sincosf(q, &s, &c);
    sc2[e] = make_float2(s, c);
  }
  __syncwarp();
  const int h = lane >> 2, r = lane & 3, g = h / nb;
  const bool mine = g < m && r < 3;
  const uint32_t* step = f.fk_step + (h - g * nb);
  float4* Xg = reinterpret_cast<float4*>(X + g * p.num_slots * 12) + r;
  float4 row = make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t next = __ldg(step);
  for (int s = 0; s < f.fk_steps; ++s) {
    const uint32_t w = next;
    if (s + 1 < f.fk_steps) next = __ldg(step + (s + 1) * nb);
    if (w >> 31) __syncwarp();  // set for the whole step
    const int j = w & 255, par = (w >> 8) & 255;
    if (!mine || j == 255) continue;
    const float4* E = f.fk_entry + 9 * j;
    const float2 v = sc2[g * nf + j];
    const bool rev = (w >> 16) & 1u;
    float L[9], t[3];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float4 e = __ldg(E + i);
      L[i] = rev ? fmaf(v.y, e.x, fmaf(v.x, e.y, e.z)) : e.x;
      if (i < 3) t[i] = e.w;
      if (i >= 3 && i < 6 && !rev) t[i - 3] = fmaf(e.w, v.x, t[i - 3]);
    }
    if (par == 253) {
      row = r == 0 ? make_float4(L[0], L[3], L[6], t[0]) : r == 1 ? make_float4(L[1], L[4], L[7], t[1])
                                                                  : make_float4(L[2], L[5], L[8], t[2]);
    } else {
      if (par != 254) row = Xg[3 * par];
      row = make_float4(fmaf(row.z, L[2], fmaf(row.y, L[1], row.x * L[0])),
                        fmaf(row.z, L[5], fmaf(row.y, L[4], row.x * L[3])),
                        fmaf(row.z, L[8], fmaf(row.y, L[7], row.x * L[6])),
                        fmaf(row.z, t[2], fmaf(row.y, t[1], fmaf(row.x, t[0], row.w))));
    }
    Xg[3 * j] = row;
  }
  __syncwarp();
}

// ------------------------------------------------------------------- world
constexpr float kFieldMargin = 1e-4f;  // metres by which an untested pair is clear, at least

// Cell of a probe (centre c, radius r): true if listed statics may touch it.
// cnt: how many (kFieldAll: test every static).
constexpr int kFieldAll = 0xffff;
static __device__ __forceinline__ bool probe_near(const FieldTables& f, float cx, float cy, float cz, float r,
                                                  uint4& cell, int& cnt) {
  const float fx = (cx - f.ox) * f.inv_h, fy = (cy - f.oy) * f.inv_h, fz = (cz - f.oz) * f.inv_h;
  cnt = 0;
  if (fx >= 0.f && fy >= 0.f && fz >= 0.f && fx < (float)f.nx && fy < (float)f.ny && fz < (float)f.nz) {
    const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
    cell = __ldg(f.cells + ((iz * f.ny + iy) * f.nx + ix));
    const float t = __half2float(__ushort_as_half((unsigned short)(cell.x & 0xffffu))) - r - kFieldMargin;
    const float dx = fx - (float)ix - 0.5f, dy = fy - (float)iy - 0.5f, dz = fz - (float)iz - 0.5f;
    const float off2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) * (f.h * f.h);
    if (t > 0.f && t * t >= off2 * 1.0001f) return false;
    cnt = (int)(cell.x >> 16);
    return cnt > 0;
  }
  // outside the grid: clear of every static outside the padded box of the statics; otherwise (NaN, or
  // outside the part of it the robot can reach) every static is tested
  const float sum = cx + cy + cz;
  const bool far = sum == sum && (cx < f.far_lo[0] || cx > f.far_hi[0] || cy < f.far_lo[1] || cy > f.far_hi[1] ||
                                  cz < f.far_lo[2] || cz > f.far_hi[2]);
  if (far || f.nx == 0) return false;
  cnt = kFieldAll;
  return true;
}

// k-th static of a cell.
static __device__ __forceinline__ int cell_static(const FieldTables& f, const uint4& cell, int cnt, int k) {
  if (cnt == kFieldAll) return k;
  if (cnt > 6) return (int)__ldg(f.list + cell.y + k);
  const uint32_t w = k < 2 ? cell.y : k < 4 ? cell.z : cell.w;
  return (int)((w >> ((k & 1) * 16)) & 0xffffu);
}

static __device__ __forceinline__ bool pair_exists(const FieldTables& f, int m, int s) {
  return !f.pair_bits || ((__ldg(f.pair_bits + m * f.pair_words + (s >> 5)) >> (s & 31)) & 1u);
}

// Sphere (c, r) against static s by the full sweep's tests: spheres and
// aligned boxes as one rounded box (a sphere's half extents are zero, a box's
// radius is zero, so each term rounds as in sph_sph_hit and sph_abox_hit), in
// the dense sweep's form (one FMA) or the tile sweep's (compare of squares).
static __device__ __forceinline__ bool sphere_static_hit(const DevPlant& p, const float* c, int s, bool dense) {
  const float4 P = __ldg(p.field.rounded + 2 * s), H = __ldg(p.field.rounded + 2 * s + 1);
  if (H.w == 0.f) {
    const float d0 = c[0] - P.x, d1 = c[1] - P.y, d2 = c[2] - P.z;
    const float e0 = fmaxf(fabsf(d0) - H.x, 0.f), e1 = fmaxf(fabsf(d1) - H.y, 0.f), e2 = fmaxf(fabsf(d2) - H.z, 0.f);
    const float ee = fmaf(e2, e2, fmaf(e1, e1, e0 * e0));
    const float rr = c[3] + P.w;
    // a NaN centre collides (fmaxf drops the NaN, so it is asked for here)
    const bool nan = !(d0 + d1 + d2 == d0 + d1 + d2);
    return nan || (dense ? !(fmaf(-rr, rr, ee) >= 0.f) : !(ee >= rr * rr));
  }
  if (H.w == 1.f) {
    float B[16];
    load4f(p.statics + 4 * s, 4, B);
    return sph_box_hit(c, c[3], B);
  }
  float C[8];
  load4f(p.statics + 4 * s, 2, C);
  return sph_cap_hit(c, C);
}

// Moving capsule A (WG) against static s by the full sweep's tests.
static __device__ __forceinline__ bool capsule_static_hit(const DevPlant& p, const float* A, int s) {
  const float4 P = __ldg(p.field.rounded + 2 * s);
  const int ty = __ldg(p.static_type + s);
  if (ty == G_SPHERE) {
    const float S[4] = {P.x, P.y, P.z, P.w};
    return sph_cap_hit(S, A);
  }
  float B[16];
  if (ty == G_CAPSULE) {
    load4f(p.statics + 4 * s, 2, B);
    return cap_cap_hit(A, B);
  }
  load4f(p.statics + 4 * s, 4, B);
  return sph_box_hit(A, A[3] + A[7], B) && cap_box_hit(A, B);
}

// Places the moving geometries and tests them against the statics (true: some
// pair collides; warp-uniform). Poses go to `pose` for the self pairs.
static __device__ __forceinline__ bool field_world(const DevPlant& p, const float* X, float* pose, int lane) {
  const FieldTables& f = p.field;
  const float4* X4 = reinterpret_cast<const float4*>(X);
  const bool dense = p.dense_spheres && p.num_tiles >= 1 && p.num_tiles <= 4;
  for (int m0 = 0; m0 < p.num_msph; m0 += kWarp) {
    const int m = m0 + lane;
    bool near = false, hit = false;
    float c[4];
    uint4 cell = make_uint4(0u, 0u, 0u, 0u);
    int cnt = 0;
    if (m < p.num_msph) {
      const float4 g = __ldg(f.geom + m);
      const int sl = 3 * (int)__ldg(p.moving_slot + m);
      const float4 r0 = X4[sl], r1 = X4[sl + 1], r2 = X4[sl + 2];
      c[0] = fmaf(r0.z, g.z, fmaf(r0.y, g.y, fmaf(r0.x, g.x, r0.w)));
      c[1] = fmaf(r1.z, g.z, fmaf(r1.y, g.y, fmaf(r1.x, g.x, r1.w)));
      c[2] = fmaf(r2.z, g.z, fmaf(r2.y, g.y, fmaf(r2.x, g.x, r2.w)));
      c[3] = g.w;
      *reinterpret_cast<float4*>(pose + 4 * m) = make_float4(c[0], c[1], c[2], c[3]);
      near = probe_near(f, c[0], c[1], c[2], c[3], cell, cnt);
    }
    if (!near) cnt = 0;
    const int todo = cnt == kFieldAll ? p.num_static : cnt;
    for (int k = 0; __any_sync(kFull, k < todo); ++k) {
      if (k < todo) {
        const int s = cell_static(f, cell, cnt, k);
        hit = sphere_static_hit(p, c, s, dense) && pair_exists(f, m, s);
      }
      if (__any_sync(kFull, hit)) return true;
    }
  }
  if (p.num_mcap == 0) return false;
  for (int q0 = 0; q0 < p.num_mcap; q0 += kWarp) {
    const int q = q0 + lane, m = p.num_msph + q;
    if (q < p.num_mcap) {
      const float4 g = __ldg(f.geom + m), z = __ldg(f.cap_axis + q);
      const int sl = 3 * (int)__ldg(p.moving_slot + m);
      const float4 r0 = X4[sl], r1 = X4[sl + 1], r2 = X4[sl + 2];
      float4* dst = reinterpret_cast<float4*>(pose + 4 * p.num_msph + 8 * q);
      dst[0] = make_float4(fmaf(r0.z, g.z, fmaf(r0.y, g.y, fmaf(r0.x, g.x, r0.w))),
                           fmaf(r1.z, g.z, fmaf(r1.y, g.y, fmaf(r1.x, g.x, r1.w))),
                           fmaf(r2.z, g.z, fmaf(r2.y, g.y, fmaf(r2.x, g.x, r2.w))), g.w);
      dst[1] = make_float4(fmaf(r0.z, z.z, fmaf(r0.y, z.y, r0.x * z.x)), fmaf(r1.z, z.z, fmaf(r1.y, z.y, r1.x * z.x)),
                           fmaf(r2.z, z.z, fmaf(r2.y, z.y, r2.x * z.x)), z.w);
    }
  }
  __syncwarp();
  for (int b0 = 0; b0 < f.num_probes; b0 += kWarp) {
    const int b = b0 + lane;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), u = a, pr = a;
    float cx = 0.f, cy = 0.f, cz = 0.f;
    uint4 cell = make_uint4(0u, 0u, 0u, 0u);
    int cnt = 0, q = 0;
    bool near = false;
    if (b < f.num_probes) {
      pr = __ldg(f.probes + b);
      q = __float_as_int(pr.z);
      const float4* src = reinterpret_cast<const float4*>(pose + 4 * p.num_msph + 8 * q);
      a = src[0];
      u = src[1];
      cx = fmaf(pr.x, u.x, a.x);
      cy = fmaf(pr.x, u.y, a.y);
      cz = fmaf(pr.x, u.z, a.z);
      near = probe_near(f, cx, cy, cz, pr.y, cell, cnt);
    }
    if (!near) cnt = 0;
    const int todo = cnt == kFieldAll ? p.num_static : cnt;
    int k = 0;
    while (__any_sync(kFull, k < todo)) {
      // the next static of this lane's list that its probe sphere may meet (padded), then the exact test
      int s = -1;
      while (k < todo && s < 0) {
        const int cand = cell_static(f, cell, cnt, k++);
        const float4 P = __ldg(f.rounded + 2 * cand), H = __ldg(f.rounded + 2 * cand + 1);
        const float e0 = fmaxf(fabsf(cx - P.x) - H.x, 0.f), e1 = fmaxf(fabsf(cy - P.y) - H.y, 0.f),
                    e2 = fmaxf(fabsf(cz - P.z) - H.z, 0.f);
        const float rr = pr.y + P.w + kFieldMargin;
        if (H.w != 0.f || !(fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) >= rr * rr)) s = cand;
      }
      bool hit = false;
      if (s >= 0) {
        const float A[8] = {a.x, a.y, a.z, a.w, u.x, u.y, u.z, u.w};
        hit = capsule_static_hit(p, A, s) && pair_exists(f, p.num_msph + q, s);
      }
      if (__any_sync(kFull, hit)) return true;
    }
  }
  return false;
}

// -------------------------------------------------------------------- self
// Moving-moving pairs [b0, b1) of FieldTables::pairs, one per lane.
template <int TA, int TB>
static __device__ __forceinline__ bool field_pairs(const DevPlant& p, const float* pose, int b0, int b1, int lane) {
  const float* cap = pose - 4 * p.num_msph;  // capsule m at 4 num_msph + 8 (m - num_msph)
  for (int base = b0; base < b1; base += kWarp) {
    bool hit = false;
    if (base + lane < b1) {
      const uint32_t w = __ldg(p.field.pairs + base + lane);
      const int a = (int)(w & 0xffffu), b = (int)(w >> 16);
      float A[Words<TA>::n], B[Words<TB>::n];
      const float4* pa = reinterpret_cast<const float4*>(TA == G_SPHERE ? pose + 4 * a : cap + 8 * a);
      const float4* pb = reinterpret_cast<const float4*>(TB == G_SPHERE ? pose + 4 * b : cap + 8 * b);
#pragma unroll
      for (int i = 0; i < Words<TA>::n / 4; ++i) {
        const float4 v = pa[i];
        A[4 * i] = v.x; A[4 * i + 1] = v.y; A[4 * i + 2] = v.z; A[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < Words<TB>::n / 4; ++i) {
        const float4 v = pb[i];
        B[4 * i] = v.x; B[4 * i + 1] = v.y; B[4 * i + 2] = v.z; B[4 * i + 3] = v.w;
      }
      hit = pair_hit(TA, A, TB, B);
    }
    if (__any_sync(kFull, hit)) return true;
  }
  return false;
}

static __device__ __forceinline__ bool field_self(const DevPlant& p, const float* X, const float* pose, float* lc,
                                                  int lane) {
  const FieldTables& f = p.field;
  if (f.num_link_pairs == 0) return false;
  float4* lc4 = reinterpret_cast<float4*>(lc);
  if (lane < p.num_slots) {
    const float4* X4 = reinterpret_cast<const float4*>(X) + 3 * lane;
    const float4 r0 = X4[0], r1 = X4[1], r2 = X4[2];
    const float4 a = __ldg(f.link_cap + 2 * lane), u = __ldg(f.link_cap + 2 * lane + 1);
    lc4[2 * lane] = make_float4(fmaf(r0.z, a.z, fmaf(r0.y, a.y, fmaf(r0.x, a.x, r0.w))),
                                fmaf(r1.z, a.z, fmaf(r1.y, a.y, fmaf(r1.x, a.x, r1.w))),
                                fmaf(r2.z, a.z, fmaf(r2.y, a.y, fmaf(r2.x, a.x, r2.w))), a.w);
    lc4[2 * lane + 1] = make_float4(fmaf(r0.z, u.z, fmaf(r0.y, u.y, r0.x * u.x)),
                                    fmaf(r1.z, u.z, fmaf(r1.y, u.y, r1.x * u.x)),
                                    fmaf(r2.z, u.z, fmaf(r2.y, u.y, r2.x * u.x)), u.w);
  }
  __syncwarp();
  for (int l0 = 0; l0 < f.num_link_pairs; l0 += kWarp) {
    bool near = false;
    int begin = 0, nss = 0, nsc = 0, ncc = 0;
    if (l0 + lane < f.num_link_pairs) {
      const int2* L = reinterpret_cast<const int2*>(f.link_pairs + l0 + lane);
      const int2 ab = __ldg(L), bs = __ldg(L + 1), sc = __ldg(L + 2);
      begin = bs.x;
      nss = bs.y;
      nsc = sc.x;
      ncc = sc.y;
      float A[8], B[8];
      load4f(lc4 + 2 * ab.x, 2, A);
      load4f(lc4 + 2 * ab.y, 2, B);
      const float rr = A[3] + B[3];
      near = !(seg_seg_d2(A, B) > rr * rr);  // a NaN pose counts as near, so its pairs are tested (and collide)
    }
    uint32_t km = __ballot_sync(kFull, near);
    while (km) {
      const int j = __ffs(km) - 1;
      km &= km - 1u;
      const int b0 = __shfl_sync(kFull, begin, j), b1 = b0 + __shfl_sync(kFull, nss, j),
                b2 = b1 + __shfl_sync(kFull, nsc, j), b3 = b2 + __shfl_sync(kFull, ncc, j);
      if (field_pairs<G_SPHERE, G_SPHERE>(p, pose, b0, b1, lane)) return true;
      if (b2 > b1 && field_pairs<G_SPHERE, G_CAPSULE>(p, pose, b1, b2, lane)) return true;
      if (b3 > b2 && field_pairs<G_CAPSULE, G_CAPSULE>(p, pose, b2, b3, lane)) return true;
    }
  }
  return false;
}

// ------------------------------------------------------------------ voxels
// Voxels through their hash grid (voxgrid.cu): a lane per probe, the moving
// spheres and then the capsules' probe spheres, each reading the voxels of the
// columns that its sphere grown by the voxel radius touches (the bound of
// check_core.cuh::grid_geom_hit). A voxel within that bound gets the full
// sweep's exact test against the sphere or capsule, so the verdict is the full
// sweep's. Bound by the scattered 16-byte voxel loads (a line each) and the
// spread of the lanes' list lengths: 2^18 uniform configurations, of which a
// quarter come here, against 10,000 voxels took 1.05 ms in all when a lane
// walked every cell of a capsule's bounding sphere and eight cells a sphere,
// 0.55 ms now. Votes inside the loops, to leave at the first hit, cost more
// than they saved (1.35 ms against 1.08 ms with the older lists).
static __device__ __forceinline__ bool field_voxels(const DevPlant& p, const float* pose, const VoxArgs& va, int lane) {
  const FieldTables& f = p.field;
  const int np = p.num_msph + f.num_probes;
  for (int i0 = 0; i0 < np; i0 += kWarp) {
    const int i = i0 + lane;
    float c[3] = {0.f, 0.f, 0.f}, r = 0.f;
    const float4* G4 = nullptr;
    bool cap = false;
    if (i < p.num_msph) {
      if ((__ldg(va.tile_mask + i / kWarp) >> (i % kWarp)) & 1u) {
        G4 = reinterpret_cast<const float4*>(pose + 4 * i);
        const float4 g = *G4;
        c[0] = g.x;
        c[1] = g.y;
        c[2] = g.z;
        r = g.w;
      }
    } else if (i < np) {
      const float4 pr = __ldg(f.probes + (i - p.num_msph));
      const int q = __float_as_int(pr.z);
      if ((__ldg(va.other + va.num_other + q / kWarp) >> (q % kWarp)) & 1u) {
        G4 = reinterpret_cast<const float4*>(pose + 4 * p.num_msph + 8 * q);
        const float4 a = G4[0], u = G4[1];
        c[0] = fmaf(pr.x, u.x, a.x);
        c[1] = fmaf(pr.x, u.y, a.y);
        c[2] = fmaf(pr.x, u.z, a.z);
        r = pr.y;
        cap = true;
      }
    }
    const float R = fmaf(r + va.vr, 1.001f, 1e-4f), R2 = R * R;
    auto exact = [&](float x, float y, float z) {
      const float4 g = G4[0];
      const float S[4] = {x, y, z, va.vr};
      if (!cap) {
        const float A[4] = {g.x, g.y, g.z, g.w};
        return sph_sph_hit(A, S);
      }
      const float4 u = G4[1];
      const float A[8] = {g.x, g.y, g.z, g.w, u.x, u.y, u.z, u.w};
      return pair_hit(G_SPHERE, S, G_CAPSULE, A);
    };
    bool hit = false;
    int lo[3], n[3], cols = 0;
    if (G4) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lo[k] = vox_cell(c[k] - fmaxf(R - va.grins, 0.f), va.ginv_h);
        n[k] = vox_cell(c[k] + fmaxf(R - va.grins, 0.f), va.ginv_h) - lo[k] + 1;
      }
      const bool finite = isfinite(c[0]) && isfinite(c[1]) && isfinite(c[2]) && isfinite(R);
      if (!finite || vox_sweep((long long)n[0] * n[1], n[2], va.nv)) {  // (a NaN pose collides with every voxel)
        if (!cap) {  // four at a time, their loads together
          const float A[4] = {c[0], c[1], c[2], r};
          for (int v0 = 0; v0 < va.nv && !hit; v0 += 4) {
            float S[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float* v = va.vox + 3 * min(v0 + j, va.nv - 1);
              S[j][0] = __ldg(v);
              S[j][1] = __ldg(v + 1);
              S[j][2] = __ldg(v + 2);
              S[j][3] = va.vr;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) hit = sph_sph_hit(A, S[j]) || hit;
          }
        } else {
          for (int v = 0; v < va.nv && !hit; ++v)
            hit = exact(__ldg(va.vox + 3 * v), __ldg(va.vox + 3 * v + 1), __ldg(va.vox + 3 * v + 2));
        }
      } else {
        cols = n[0] * n[1];
      }
    }
    // four columns at a time, their runs looked up together; a column that wraps has a second run
    const int nz = cols ? min(n[2], va.gmask + 1) : 0;
    for (int j0 = 0; j0 < cols && !hit; j0 += 4) {
      int k0[4], k1[4], wrap = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        k0[j] = k1[j] = 0;
        if (j0 + j < cols) {
          const int ix = (j0 + j) / n[1], iy = j0 + j - ix * n[1];
          const int b = (int)vox_bucket(lo[0] + ix, lo[1] + iy, lo[2], va.gmask);
          const int e = min(b + nz, va.gmask + 1);
          k0[j] = __ldg(va.gstart + b);
          k1[j] = __ldg(va.gstart + e);
          wrap = max(wrap, b + nz - e);
        }
      }
      if (wrap)  // the first `wrap` buckets
        for (int k = 0, e = __ldg(va.gstart + wrap); k < e; ++k) {
          const float4 v = __ldg(va.gvox + k);
          hit |= exact(v.x, v.y, v.z);
        }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        for (int k = k0[j]; k < k1[j] && !hit; k += 2) {
          const float4 v = __ldg(va.gvox + k), w = __ldg(va.gvox + min(k + 1, k1[j] - 1));
          const float v0 = v.x - c[0], v1 = v.y - c[1], v2 = v.z - c[2];
          const float w0 = w.x - c[0], w1 = w.y - c[1], w2 = w.z - c[2];
          if (!(fmaf(v2, v2, fmaf(v1, v1, v0 * v0)) > R2)) hit |= exact(v.x, v.y, v.z);
          if (!(fmaf(w2, w2, fmaf(w1, w1, w0 * w0)) > R2)) hit |= exact(w.x, w.y, w.z);
        }
    }
    if (__any_sync(kFull, hit)) return true;
  }
  // robot geometries fixed to the world
  for (int o0 = 0; o0 < va.num_other; o0 += kWarp) {
    const int o = o0 + lane;
    const uint32_t ref = o < va.num_other ? __ldg(va.other + o) : 0u;
    bool hit = false;
    if (ref & 0x80000000u) {
      const int s = (int)(ref & 0x7fffffffu), tg = __ldg(p.static_type + s);
      float G[16], bc[3];
      load4f(p.statics + 4 * s, tg == G_SPHERE ? 1 : tg == G_CAPSULE ? 2 : 4, G);
      const float br = geom_bound(tg, G, bc);
      hit = grid_geom_hit<false>(va, tg, G, bc, br);
    }
    if (__any_sync(kFull, hit)) return true;
  }
  return false;
}

// Full check of the configuration whose slot transforms are in X (rows).
static __device__ bool check_field(const DevPlant& p, const float* X, float* pose, int lane, const VoxArgs& va) {
  if (p.always_colliding) return true;
  if (field_world(p, X, pose, lane)) return true;
  __syncwarp();
  if (field_self(p, X, pose, pose + field_scratch_floats(p), lane)) return true;
  return va.nv > 0 && (va.gstart ? field_voxels(p, pose, va, lane) : sweep_voxels(p, p.statics, pose, va, lane));
}

}  // namespace csd
