// sampler_core.cuh -- one hit-and-run chain, shared by the sampler and the
// batched EI-ZO kernels.
#pragma once
#include <cfloat>

#include "csd_rng.cuh"

namespace csd {

// ---- packed FP32 pairs (sm_100 f32x2): each half is an IEEE round-to-nearest
// operation, so a packed result is bit for bit the two scalar results.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float* lo, float* hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*lo), "=f"(*hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// ---------------------------------------------------------------------------
// EI-ZO sampling: hit-and-run with carried slacks over face pairs.
//
// Every chain of an EI-ZO iteration starts at the segment's start point x0,
// so the slack b_f - a_f . x0 of a face at the start of a chain is common to
// all chains. It is computed once, when the face is written (put_face), in the
// serial chain's order (product of coordinate 0, fused multiply-adds in
// coordinate order, then b minus that). A chain carries its slacks: after a
// step of length theta along dir it updates s_f = fma(-theta, a_f . dir, s_f),
// so a mixing step costs one dim-long dot product per face instead of two
// (the reference recomputes b - A x every step,
// csdecomp/src/planning/cuda_hit_and_run_sampling.cu:83-104). The theta
// bounds, the theta draw (0.999999 scales theta_max only, :106-107) and the
// position update are the serial chain's.
//
// Face-pair rows: row p holds faces 2p and 2p + 1 interleaved, coordinate k of
// face 2p + h at float 2k + h (k < MAXD, zero past dim), the two start slacks
// at 2 MAXD and 2 MAXD + 1, then a mark per face (1: a coefficient is beyond
// kMaxCoeff, else 0): 2 MAXD + 4 floats, a multiple of 16 bytes. A face that does not exist yet (the partner of the
// last face of an odd count) holds a copy of that face: it bounds theta
// exactly as the face does, so it changes no bound. One 16-byte load brings two
// coordinates of both faces, and one packed FMA (fma.rn.f32x2, each half an
// IEEE round-to-nearest FMA) advances both faces' dot products.
__host__ __device__ constexpr int pair_maxd(int dim) { return dim <= 8 ? 8 : 16; }
__host__ __device__ constexpr int pair_stride(int dim) { return 2 * pair_maxd(dim) + 4; }

// Coefficients up to here leave a . dir finite (a direction's coordinates stay
// below 8); a face with one beyond, or a NaN, is marked for one division per
// face, because the packed quotient of an infinite a . dir is NaN, not 0.
constexpr float kMaxCoeff = 1.2676506002282294e30f;  // 2^100

// Writes face f (coordinates a[0..dim), offset b) of a region whose chains
// start at x0. An even f also fills its partner half with a copy of itself.
__device__ __forceinline__ void put_face(float* __restrict__ rows, int dim, int f, const float* a, float b,
                                         const float* __restrict__ x0) {
  const int md = pair_maxd(dim), h = f & 1;
  float* r = rows + (size_t)(f >> 1) * pair_stride(dim);
  float ax = __fmul_rn(a[0], x0[0]);
  for (int k = 1; k < dim; ++k) ax = __fmaf_rn(a[k], x0[k], ax);
  bool big = false;
  for (int k = 0; k < md; ++k) {
    r[2 * k + h] = k < dim ? a[k] : 0.f;
    big = big || (k < dim && !(fabsf(a[k]) <= kMaxCoeff));
  }
  r[2 * md + h] = __fsub_rn(b, ax);
  r[2 * md + 2 + h] = big ? 1.f : 0.f;
  if (!h) {  // until face f + 1 is written, its half repeats face f (a face seen twice bounds nothing new)
    for (int k = 0; k < md; ++k) r[2 * k + 1] = r[2 * k];
    r[2 * md + 1] = r[2 * md];
    r[2 * md + 3] = r[2 * md + 2];
  }
}

// Pair rows of faces [0, F) of a row-major A (F x dim) and b; thread t of
// nthreads writes whole pairs t, t + nthreads, ...
__device__ __forceinline__ void put_faces(const float* __restrict__ A, const float* __restrict__ b, int F, int dim,
                                          const float* __restrict__ x0, float* __restrict__ rows, int t,
                                          int nthreads) {
  for (int p = t; p < (F + 1) / 2; p += nthreads) {
    put_face(rows, dim, 2 * p, A + (size_t)(2 * p) * dim, b[2 * p], x0);
    if (2 * p + 1 < F) put_face(rows, dim, 2 * p + 1, A + (size_t)(2 * p + 1) * dim, b[2 * p + 1], x0);
  }
}

// theta bounds of one face (slack s, a . dir = ad): the reference's rule
// (ad < 0 raises theta_min to s / ad, ad > 0 lowers theta_max to s / ad, ad = 0
// bounds nothing), as one IEEE division and two selects, so that lanes whose
// faces point either way do not split into two division paths. For ad = 0
// (either sign) the quotient is infinite or NaN and neither select takes it;
// the rows hold no zero faces (an unpaired face is repeated), so that case,
// which takes the division's slow path, only arises when a . dir is exactly 0.
__device__ __forceinline__ void theta_bound(float s, float ad, float& tmin, float& tmax) {
  const float q = __fdiv_rn(s, ad);
  tmin = ad < 0.0f ? fmaxf(tmin, q) : tmin;
  tmax = ad > 0.0f ? fminf(tmax, q) : tmax;
}

// ---- theta bounds of a face pair without a division per face.
//
// Two correctly rounded quotients at once: reciprocal estimates (at most 1 ulp
// off) and packed fused steps. y1 = y0 + y0 (1 - a y0) is the correctly
// rounded reciprocal, q1 is within one ulp of s / a, and q1 + y1 (s - a q1)
// then rounds as the quotient does (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1),
// 1990, theorems 4 and 7), as long as nothing overflows or leaves the normal
// range. na holds -a. tests/test_gpu_sampler_bounds.py compares it with the
// IEEE division, the one significand that the theorem leaves out included.
__device__ __forceinline__ float rcp_estimate(float a) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
  return y;
}
__device__ __forceinline__ uint64_t f2_quotient(uint64_t s, uint64_t na) {
  float a0, a1;
  f2_unpack(na, &a0, &a1);
  const uint64_t y0 = f2_pack(rcp_estimate(-a0), rcp_estimate(-a1));
  const uint64_t y1 = f2_fma(f2_fma(na, y0, f2_pack(1.f, 1.f)), y0, y0);
  const uint64_t q0 = f2_mul(s, y0);
  const uint64_t q1 = f2_fma(f2_fma(na, q0, s), y0, q0);
  return f2_fma(f2_fma(na, q1, s), y1, q1);
}

// Running bounds as the bits of the quotients. While every slack is positive
// a quotient has the sign of a . dir, and then theta_max, the least positive
// quotient, is the least of the bit patterns as unsigned integers, and
// theta_min, the negative quotient nearest to zero, the least as signed
// integers: one three-way integer minimum each per face pair. (NaN and
// infinite quotients, from a . dir = 0, lose against the initial
// +-FLT_MAX as they do in theta_bound.) `slack` tracks the least slack the
// same way.
struct ThetaBits {
  uint32_t hi;   // theta_max
  int32_t lo;    // theta_min
  int32_t slack;
};
__device__ __forceinline__ ThetaBits theta_bits_start() {
  return {__float_as_uint(FLT_MAX), __float_as_int(-FLT_MAX), __float_as_int(FLT_MAX)};
}
__device__ __forceinline__ void theta_bits(ThetaBits& t, uint64_t s, uint64_t na) {
  const uint64_t q = f2_quotient(s, na);
  const int q0 = (int)(uint32_t)q, q1 = (int)(q >> 32);
  t.hi = __vimin3_u32(t.hi, (uint32_t)q0, (uint32_t)q1);
  t.lo = __vimin3_s32(t.lo, q0, q1);
  t.slack = __vimin3_s32(t.slack, (int)(uint32_t)s, (int)(s >> 32));
}
// Where that holds: every slack at least kMinSlack (a start on a face has none:
// such a lane takes theta_bound over its faces), and both bounds of the group
// within [kMinTheta, kMaxTheta), so that the binding a . dir lies in
// [2^-59, 2^126) and its quotient is exact (otherwise the group takes
// theta_bound). A face whose finite a . dir is too small or too large for the
// packed steps has a quotient outside that range, so it cannot bind unseen; a
// lane holding a marked face (kMaxCoeff) takes theta_bound whatever its slacks:
// its least slack is compared with kNoSlack, which every slack is below.
//
// The slow path over n face pairs copied to local memory, in a loop that is
// not unrolled: the branch is next to never taken, and with the quotients of
// every register-held pair written out there the fast path lost 40% to the
// registers they took (42 -> 25 cycles per 32 pairs, register rows at 14
// dimensions).
__device__ __forceinline__ void theta_bounds_slow(const uint64_t* s, const uint64_t* na, int n, float& tmin,
                                                  float& tmax) {
#pragma unroll 1
  for (int j = 0; j < n; ++j) {
    float sa, sb, aa, ab;
    f2_unpack(s[j], &sa, &sb);
    f2_unpack(na[j], &aa, &ab);
    theta_bound(sa, -aa, tmin, tmax);
    theta_bound(sb, -ab, tmin, tmax);
  }
}
constexpr float kMinSlack = 9.313225746154785e-10f;   // 2^-30
constexpr int kNoSlack = 0x7fffffff;
constexpr float kMinTheta = 7.888609052210118e-31f;   // 2^-100
constexpr float kMaxTheta = 536870912.f;              // 2^29

// Steps whose draws a group computes at once (when its drawing lanes hold
// that many steps' jobs).
constexpr int kDrawSteps = 8;

// Shared scratch of a group wider than a warp (G = 64, 128, 256 lanes): the
// directions and theta uniforms of a batch of drawn steps (coordinates 0..15,
// the uniform at 16), double buffered by batch parity, and each warp's
// partial theta bounds, double buffered by step parity (a warp cannot
// run two steps, or two batches, ahead of the group's barriers). The
// directions are stored negated (see run_chain_pairs).
struct GroupScratch {
  float dir[2][kDrawSteps][17];
  float red[3][8][2];  // by step parity; [2]: a step's second reduction
};
constexpr int kMaxWideGroups = 4;  // 256 threads / 64 lanes

__device__ __forceinline__ void group_bar(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Lanes per chain: at least `g` (set by the chain count) and enough that
// each lane holds at most KP face pairs; 0 if even 256 lanes do not.
__host__ __device__ __forceinline__ int pair_group_width(int g, int P, int KP) {
  while (g <= 256 && (long long)g * KP < P) g <<= 1;
  return g <= 256 ? g : 0;
}

// One chain run by a group of G lanes over a region of P face pairs (staged in
// shared memory or read from global memory). Lane gl holds pairs gl + G j
// (j < KP) and their slacks and a . dir values in registers, and coordinates
// gl + G r of the position (xl). The draws are the serial chain's: step s
// reads words 0 .. 2 ceil(dim/2) of its stream (Gaussian pair j from words 2j
// and 2j + 1, the theta uniform from word 2 ceil(dim/2)), four words per
// Philox block. A drawing slot is one block: both its Box-Muller pairs (or a
// pair and the theta uniform). A step has JB = ceil(dim/2) / 2 + 1 blocks; the
// group's drawing lanes (all of a group of up to 32, the first warp of a wider
// one) draw S = min(kDrawSteps, lanes / JB) steps at once, slot q = gl holding
// block q % JB of step offset q / JB, so Gaussian pair p of offset t lies on
// lane t JB + p / 2. The direction reaches the group by shuffles (G <= 32) or
// through GroupScratch (wider groups, named barrier bar_id). The theta bounds
// are max/min reductions, which do not depend on the order, so every chain
// ends bit for bit where the oracle's serial chain ends whatever G. Directions
// are drawn negated, so that the dot products are the -(a . dir) that the
// quotients' residuals and (with the sign taken into theta) the slack and
// position updates want; negation is exact. A chain whose line search fails keeps stepping without moving (the group's lanes
// stay convergent) and returns false.
//
// MAXD: coordinates of a row (8 or 16); NQ: coordinate pairs the dot products
// run over, at least dim / 2. Coefficients past dim are zero, so they change
// no dot product, and a count known at compile time spares a test of dim per
// coordinate.
template <int MAXD, int NQ, int G, int KP>
__device__ __forceinline__ bool run_chain_pairs(const float* __restrict__ rows, int P, int dim, int mixing,
                                                uint32_t k0, uint32_t k1, uint32_t chain, uint32_t stream,
                                                float* xl, int gl, GroupScratch* gs, int bar_id) {
  constexpr int RS = 2 * MAXD + 4;
  constexpr int GD = G < 32 ? G : 32;    // drawing lanes
  constexpr int XL = (MAXD + G - 1) / G;  // position coordinates per lane
  static_assert(MAXD / 4 + 1 <= GD, "one step's blocks fit the drawing lanes");
  const int npairs = (dim + 1) >> 1, JB = (npairs >> 1) + 1;
  const int S = min(kDrawSteps, GD / JB);  // steps drawn at once (uniform)
  const int tq = gl / JB, bq = gl - tq * JB;  // this lane's slot: step offset, block
  // a lane past the last pair in round j holds a copy of pair P - 1 there: its work is the same
  // as that pair's owner's (so the group's lanes never diverge in the face loop) and a face seen
  // twice changes no theta bound
  uint64_t s2[KP], na2[KP];  // na2: -(a . dir)
  int min_slack = __float_as_int(kMinSlack);
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    const int p = min(gl + G * j, P - 1);
    ulonglong2 sm = make_ulonglong2(0ull, 0ull);  // slacks, marks
    if (P > 0) sm = *reinterpret_cast<const ulonglong2*>(rows + (size_t)p * RS + 2 * MAXD);
    s2[j] = sm.x;
    if (sm.y) min_slack = kNoSlack;
    na2[j] = 0ull;  // with th = -0 the first update leaves every slack as it is
  }
  float th = -0.0f;
  bool ok = true;
  // this lane's block: pair 2 bq (c0a, c1a) and pair 2 bq + 1 (c0b, c1b); where a pair index
  // reaches npairs its c0 holds the theta uniform instead
  float c0a = 0.f, c1a = 0.f, c0b = 0.f, c1b = 0.f;
  int t = 0, batch = -1;  // step offset within the drawn batch, batch parity
  for (int step = 0; step < mixing; ++step) {
    if (t == 0) {
      ++batch;
      // wide groups draw in their first warp (uniform across a warp); every drawing lane
      // evaluates its slot without branching (lanes past the batch's last slot compute values
      // nobody reads), so the group's lanes stay convergent through the draws
      if (G <= 32 || gl < 32) {
        uint32_t w[4];
        philox4x32_10((uint32_t)(step + tq), chain, stream, (uint32_t)bq, k0, k1, w);
        const float ua = u01_open0(w[0]), ub = u01_open0(w[2]);
        const float rada = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ua)));
        const float radb = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ub)));
        float sna, csa, snb, csb;
        sincos_2pi(u01_open1(w[1]), &sna, &csa);
        sincos_2pi(u01_open1(w[3]), &snb, &csb);
        const bool ga = 2 * bq < npairs, gb = 2 * bq + 1 < npairs;
        c0a = ga ? -__fmul_rn(rada, csa) : ua;
        c1a = -__fmul_rn(rada, sna);
        c0b = gb ? -__fmul_rn(radb, csb) : ub;
        c1b = -__fmul_rn(radb, snb);
      }
      if constexpr (G > 32) {
        if (gl < S * JB) {  // the first warp's lanes (S JB <= 32)
          float* db = gs->dir[batch & 1][tq];
          if (2 * bq < npairs) {
            db[4 * bq] = c0a;
            db[4 * bq + 1] = c1a;
          } else {
            db[16] = c0a;
          }
          if (2 * bq + 1 < npairs) {
            db[4 * bq + 2] = c0b;
            db[4 * bq + 3] = c1b;
          } else if (2 * bq + 1 == npairs) {
            db[16] = c0b;
          }
        }
      }
    }
    const int base = t * JB;  // lane of this step's block 0
    uint64_t dd[2 * NQ];      // (-dir_k, -dir_k); past dim: any finite number
    float ut;
    if constexpr (G <= 32) {
#pragma unroll
      for (int k = 0; k < 2 * NQ; ++k) {
        // coordinate k: pair k >> 1 = block k >> 2, half (k >> 1) & 1, cosine or sine k & 1
        const float v = ((k >> 1) & 1) ? ((k & 1) ? c1b : c0b) : ((k & 1) ? c1a : c0a);
        const float dk = __shfl_sync(0xffffffffu, v, base + (k >> 2), G);
        dd[k] = f2_pack(dk, dk);
      }
      const float utv = (npairs & 1) ? c0b : c0a;  // the theta uniform: block npairs / 2, half npairs & 1
      ut = __shfl_sync(0xffffffffu, utv, base + (npairs >> 1), G);
    } else {
      const float* db = gs->dir[batch & 1][t];
      if (t == 0) group_bar(bar_id, G);  // the batch's draws are in scratch
#pragma unroll
      for (int k = 0; k < 2 * NQ; ++k) {
        const float dk = db[k];
        dd[k] = f2_pack(dk, dk);
      }
      ut = db[16];
    }
    ThetaBits tb = theta_bits_start();
    const uint64_t th2 = f2_pack(th, th);
#pragma unroll
    for (int j = 0; j < KP; ++j) {
      if (G * j >= P) break;  // no lane of the group holds pair j (uniform across the group)
      const int p = min(gl + G * j, P - 1);
      const uint64_t s = f2_fma(th2, na2[j], s2[j]);  // the previous step's slack update
      s2[j] = s;
      const ulonglong2* row = reinterpret_cast<const ulonglong2*>(rows + (size_t)p * RS);
      uint64_t acc = 0ull;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const ulonglong2 v = row[q];  // coordinates 2q and 2q + 1 of both faces
        acc = q == 0 ? f2_mul(v.x, dd[0]) : f2_fma(v.x, dd[2 * q], acc);
        acc = f2_fma(v.y, dd[2 * q + 1], acc);
      }
      na2[j] = acc;
      theta_bits(tb, s, acc);
    }
    float tmax, tmin;
    for (int pass = 0;; ++pass) {
      if (pass || tb.slack < min_slack) {  // this lane's faces one division each
        tmax = FLT_MAX;
        tmin = -FLT_MAX;
        uint64_t ls[KP], ln[KP];
#pragma unroll
        for (int j = 0; j < KP; ++j) {
          ls[j] = s2[j];
          ln[j] = na2[j];
        }
        theta_bounds_slow(ls, ln, min(KP, (P + G - 1) / G), tmin, tmax);
      } else {
        tmax = __uint_as_float(tb.hi);
        tmin = __int_as_float(tb.lo);
      }
      if constexpr (G <= 32) {
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
          tmin = fmaxf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o, G));
          tmax = fminf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o, G));
        }
      } else {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          tmin = fmaxf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
          tmax = fminf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        }
        float(*red)[2] = gs->red[pass ? 2 : step & 1];
        if ((gl & 31) == 0) {
          red[gl >> 5][0] = tmin;
          red[gl >> 5][1] = tmax;
        }
        group_bar(bar_id, G);
        tmin = red[0][0];
        tmax = red[0][1];
#pragma unroll
        for (int w = 1; w < G / 32; ++w) {
          tmin = fmaxf(tmin, red[w][0]);
          tmax = fminf(tmax, red[w][1]);
        }
      }
      if (pass) break;
      const bool in_range = tmax >= kMinTheta && tmax < kMaxTheta && -tmin >= kMinTheta && -tmin < kMaxTheta;
      // uniform across the warp (G <= 32: its groups share the shuffles) or the group
      if (G <= 32 ? __all_sync(0xffffffffu, in_range) : in_range) break;
    }
    if (isinf(tmax) || isinf(tmin) || tmax < tmin) ok = false;
    // this step's direction at the position coordinates the lane holds (coordinate k: block
    // k >> 2 on lane base + (k >> 2), half (k >> 1) & 1, cosine or sine k & 1)
    float dkl[XL];
#pragma unroll
    for (int r = 0; r < XL; ++r) {
      const int k = min(gl + G * r, MAXD - 1);
      if constexpr (G <= 32) {
        const int src = base + (k >> 2);
        const float va0 = __shfl_sync(0xffffffffu, c0a, src, G), va1 = __shfl_sync(0xffffffffu, c1a, src, G);
        const float vb0 = __shfl_sync(0xffffffffu, c0b, src, G), vb1 = __shfl_sync(0xffffffffu, c1b, src, G);
        dkl[r] = ((k >> 1) & 1) ? ((k & 1) ? vb1 : vb0) : ((k & 1) ? va1 : va0);
      } else {
        dkl[r] = gs->dir[batch & 1][t][k];
      }
    }
    th = -0.0f;
    if (ok) {
      const double td = __dadd_rn(__dmul_rn((double)ut, __dsub_rn(__dmul_rn(0.999999, (double)tmax), (double)tmin)),
                            (double)tmin);
      const float theta = __double2float_rn(td);
#pragma unroll
      for (int r = 0; r < XL; ++r)
        if (gl + G * r < dim) xl[r] = __fmaf_rn(-theta, dkl[r], xl[r]);
      th = theta;
    }
    t = t + 1 == S ? 0 : t + 1;
  }
  return ok;
}

// Chains [first, last) of one region by the whole block (256 threads), G
// lanes per chain; groups past `last` repeat the last chain and store
// nothing, so every group takes the same number of trips (wide groups meet
// at named barriers 1 + group index). A failed chain stores `start`.
template <int MAXD, int NQ, int G, int KP>
__device__ __forceinline__ void sample_chains_pairs(const float* __restrict__ rows, int P, int dim,
                                                    const float* __restrict__ start, int first, int last, int mixing,
                                                    uint32_t k0, uint32_t k1, uint32_t stream,
                                                    float* __restrict__ out, GroupScratch* gsa) {
  constexpr int XL = (MAXD + G - 1) / G;
  const int gl = threadIdx.x & (G - 1), gid = threadIdx.x / G, ngroups = blockDim.x / G;
  GroupScratch* gs = G > 32 ? gsa + gid : nullptr;
  if constexpr (G > 32) {  // directions past dim stay zero (they meet zero coefficients and must be finite)
    float* d = &gs->dir[0][0][0];
    for (int i = gl; i < 2 * kDrawSteps * 17; i += G) d[i] = 0.f;
    group_bar(1 + gid, G);
  }
  for (int c0 = first; c0 < last; c0 += ngroups) {
    const int chain = c0 + gid;
    const int cc = chain < last ? chain : last - 1;
    float xl[XL];
#pragma unroll
    for (int r = 0; r < XL; ++r) {
      const int k = gl + G * r;
      xl[r] = k < dim ? start[k] : 0.f;
    }
    const bool ok = run_chain_pairs<MAXD, NQ, G, KP>(rows, P, dim, mixing, k0, k1, (uint32_t)cc, stream, xl, gl, gs,
                                                 1 + gid);
    if (chain < last) {
#pragma unroll
      for (int r = 0; r < XL; ++r) {
        const int k = gl + G * r;
        if (k < dim) out[(int64_t)chain * dim + k] = ok ? xl[r] : start[k];
      }
    }
  }
}

// The chains of one region with G lanes each (G from pair_group_width, one of
// 8 .. 256).
template <int MAXD, int NQ, int KP>
__device__ __forceinline__ void sample_region_q(int G, const float* __restrict__ rows, int P, int dim,
                                              const float* __restrict__ start, int first, int last, int mixing,
                                              uint32_t k0, uint32_t k1, uint32_t stream, float* __restrict__ out,
                                              GroupScratch* gsa) {
  switch (G) {
    case 8:
      sample_chains_pairs<MAXD, NQ, 8, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
    case 16:
      sample_chains_pairs<MAXD, NQ, 16, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
    case 32:
      sample_chains_pairs<MAXD, NQ, 32, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
    case 64:
      sample_chains_pairs<MAXD, NQ, 64, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
    case 128:
      sample_chains_pairs<MAXD, NQ, 128, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
    default:
      sample_chains_pairs<MAXD, NQ, 256, KP>(rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
      break;
  }
}

template <int MAXD, int KP>
__device__ __forceinline__ void sample_region(int G, const float* __restrict__ rows, int P, int dim,
                                              const float* __restrict__ start, int first, int last, int mixing,
                                              uint32_t k0, uint32_t k1, uint32_t stream, float* __restrict__ out,
                                              GroupScratch* gsa) {
  if constexpr (MAXD == 16) {
    if (dim <= 14)
      sample_region_q<16, 7, KP>(G, rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
    else
      sample_region_q<16, 8, KP>(G, rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
  } else {
    sample_region_q<8, 4, KP>(G, rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
  }
}

// ---------------------------------------------------------------------------
// Large regions above 8 dimensions: the face pairs stay in registers.
//
// run_chain_pairs reads every pair's coefficients from shared memory for every
// chain and step: 7 16-byte loads per pair at 14 dimensions, 4 cycles of the
// SM's shared-memory port each when 32 lanes read 32 rows. On regions of a few
// hundred faces that port was 84% busy and the issue slots 47%: nothing else
// could make it faster. Here a lane holds KR pairs' coefficients in registers
// for all chains of a work item, and a group of W warps runs C chains side by
// side; a step reads only the C directions (stored twice per coordinate, the
// packed FMA's operand), the same address for all lanes. Per pair and chain
// that is 7 / KR broadcast loads instead of 7 distinct ones.
//
// Per step: dot products, slack updates and quotient bounds (theta_bits) of
// the lane's KR x C pairs; one integer warp minimum per bound and chain;
// partials of the W warps through shared memory behind the group's barrier;
// then every warp works out theta of the C chains (8 lanes each, which also
// hold the chain's position). Same draws, same operations per face, order-free
// minima: bit for bit the chains of run_chain_pairs.
constexpr int kRegChains = 4;  // C: 8 lanes each in the theta phase
constexpr int kRegSteps = 8;   // steps drawn at once
// Row of the warp `wig` of group `gid`: rotated by group, so that the warps
// with one row more than the others sit on different schedulers.
__device__ __forceinline__ int reg_row(int wig, int gid, int W) { return (wig + gid) & (W - 1); }
struct RegScratch {            // per group
  float dir[2][kRegChains][kRegSteps][32];  // (-dir_k, -dir_k), by batch parity
  float ut[2][kRegChains][kRegSteps];
  float red[3][kRegChains][8][2];           // (theta_min, theta_max) per warp, by step parity; [2]: second pass
};

//
// KR is the calling warp's own count: a region of R = ceil(P / 32) rows of 32
// pairs gives warp r of the group rows r, r + W, ..., so the group's warps may
// run different instantiations, which meet at the same barriers.
template <int NQ, int KR>
__device__ __forceinline__ void sample_chains_regs(const float* __restrict__ rows, int P, int dim,
                                                   const float* __restrict__ start, int first, int last, int mixing,
                                                   uint32_t k0, uint32_t k1, uint32_t stream, int W,
                                                   float* __restrict__ out, RegScratch* scratch) {
  constexpr int C = kRegChains, S = kRegSteps, RS = 2 * 16 + 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gid = warp / W, wig = warp - gid * W, ngroups = (int)(blockDim.x >> 5) / W;
  const int gl = wig * 32 + lane, GL = 32 * W, bar_id = 1 + gid;
  RegScratch& sc = scratch[gid];
  const int npairs = (dim + 1) >> 1, JB = (npairs >> 1) + 1;
  // this lane's pairs; past the last pair: copies of it (they bound what it bounds)
  uint64_t a[KR][2 * NQ], s0[KR];
  int min_slack = __float_as_int(kMinSlack);
  const int row0 = reg_row(wig, gid, W);
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const float* r = rows + (size_t)min(32 * (row0 + W * j) + lane, P - 1) * RS;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(r + 4 * q);
      a[j][2 * q] = v.x;
      a[j][2 * q + 1] = v.y;
    }
    const ulonglong2 sm = *reinterpret_cast<const ulonglong2*>(r + 32);  // slacks, marks
    s0[j] = sm.x;
    if (sm.y) min_slack = kNoSlack;
  }
  // coordinates past dim have zero coefficients; their direction must only be finite
  for (int i = gl; i < 2 * C * S * 32; i += GL) (&sc.dir[0][0][0][0])[i] = 0.f;
  const int tc = lane >> 3, ti = lane & 7;  // theta phase: chain and coordinates ti, ti + 8
  group_bar(bar_id, GL);
  for (int c0 = first + gid * C; c0 < last; c0 += ngroups * C) {
    uint64_t s2[C][KR], na2[C][KR];
    float th[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      th[c] = -0.0f;
#pragma unroll
      for (int j = 0; j < KR; ++j) {
        s2[c][j] = s0[j];
        na2[c][j] = 0ull;
      }
    }
    float x0 = ti < dim ? start[ti] : 0.f, x1 = ti + 8 < dim ? start[ti + 8] : 0.f;
    bool ok = true;
    int t = 0, par = 1;
    for (int step = 0; step < mixing; ++step) {
      if (t == 0) {
        par ^= 1;
        for (int job = gl; job < C * S * JB; job += GL) {
          const int bq = job % JB, ct = job / JB, c = ct % C, tq = ct / C;
          uint32_t w[4];
          philox4x32_10((uint32_t)(step + tq), (uint32_t)min(c0 + c, last - 1), stream, (uint32_t)bq, k0, k1, w);
          const float ua = u01_open0(w[0]), ub = u01_open0(w[2]);
          const float rada = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ua)));
          const float radb = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ub)));
          float sna, csa, snb, csb;
          sincos_2pi(u01_open1(w[1]), &sna, &csa);
          sincos_2pi(u01_open1(w[3]), &snb, &csb);
          float4* d = reinterpret_cast<float4*>(&sc.dir[par][c][tq][8 * bq]);
          if (2 * bq < npairs) {
            const float g0 = -__fmul_rn(rada, csa), g1 = -__fmul_rn(rada, sna);
            d[0] = make_float4(g0, g0, g1, g1);
          } else {
            sc.ut[par][c][tq] = ua;
          }
          if (2 * bq + 1 < npairs) {
            const float g0 = -__fmul_rn(radb, csb), g1 = -__fmul_rn(radb, snb);
            d[1] = make_float4(g0, g0, g1, g1);
          } else if (2 * bq + 1 == npairs) {
            sc.ut[par][c][tq] = ub;
          }
        }
        group_bar(bar_id, GL);
      }
      float(*red)[8][2] = sc.red[step & 1];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const uint64_t th2 = f2_pack(th[c], th[c]);
#pragma unroll
        for (int j = 0; j < KR; ++j) s2[c][j] = f2_fma(th2, na2[c][j], s2[c][j]);
      }
      // coordinates outermost: C x KR independent dot products hide each other's latency
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const ulonglong2 dd = *reinterpret_cast<const ulonglong2*>(&sc.dir[par][c][t][4 * q]);
#pragma unroll
          for (int j = 0; j < KR; ++j) {
            na2[c][j] = q == 0 ? f2_mul(a[j][0], dd.x) : f2_fma(a[j][2 * q], dd.x, na2[c][j]);
            na2[c][j] = f2_fma(a[j][2 * q + 1], dd.y, na2[c][j]);
          }
        }
      }
      ThetaBits tb[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        tb[c] = theta_bits_start();
#pragma unroll
        for (int j = 0; j < KR; ++j) theta_bits(tb[c], s2[c][j], na2[c][j]);
      }
      // a slack too small for the packed quotients: theta_max = 0 sends the group to the second pass
#pragma unroll
      for (int c = 0; c < C; ++c) {
        tb[c].hi = tb[c].slack < min_slack ? 0u : tb[c].hi;
        tb[c].hi = __reduce_min_sync(0xffffffffu, tb[c].hi);
        tb[c].lo = __reduce_min_sync(0xffffffffu, tb[c].lo);
      }
      if (lane == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          *reinterpret_cast<float2*>(red[c][wig]) = make_float2(__int_as_float(tb[c].lo), __uint_as_float(tb[c].hi));
      }
      float tmin, tmax;
      for (int pass = 0;; ++pass) {
        group_bar(bar_id, GL);
        const float2 v = *reinterpret_cast<const float2*>(red[tc][min(ti, W - 1)]);
        tmin = v.x;
        tmax = v.y;
#pragma unroll
        for (int o = 4; o; o >>= 1) {
          tmin = fmaxf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
          tmax = fminf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        }
        const bool in_range = tmax >= kMinTheta && tmax < kMaxTheta && -tmin >= kMinTheta && -tmin < kMaxTheta;
        if (pass || __all_sync(0xffffffffu, in_range)) break;  // the same in every warp of the group
        red = sc.red[2];
        uint64_t ls[C * KR], ln[C * KR];
#pragma unroll
        for (int i = 0; i < C * KR; ++i) {
          ls[i] = s2[i / KR][i % KR];
          ln[i] = na2[i / KR][i % KR];
        }
#pragma unroll 1
        for (int c = 0; c < C; ++c) {
          float lmax = FLT_MAX, lmin = -FLT_MAX;
          theta_bounds_slow(ls + c * KR, ln + c * KR, KR, lmin, lmax);
#pragma unroll
          for (int o = 16; o; o >>= 1) {
            lmin = fmaxf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
            lmax = fminf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
          }
          if (lane == 0) *reinterpret_cast<float2*>(red[c][wig]) = make_float2(lmin, lmax);
        }
      }
      if (isinf(tmax) || isinf(tmin) || tmax < tmin) ok = false;
      float theta = -0.0f;
      if (ok) {
        const double ut = (double)sc.ut[par][tc][t];
        theta = __double2float_rn(__dadd_rn(
            __dmul_rn(ut, __dsub_rn(__dmul_rn(0.999999, (double)tmax), (double)tmin)), (double)tmin));
        const float* d = sc.dir[par][tc][t];
        x0 = ti < dim ? __fmaf_rn(-theta, d[2 * ti], x0) : x0;
        x1 = ti + 8 < dim ? __fmaf_rn(-theta, d[2 * ti + 16], x1) : x1;
      }
#pragma unroll
      for (int c = 0; c < C; ++c) th[c] = __shfl_sync(0xffffffffu, theta, 8 * c);
      t = t + 1 == S ? 0 : t + 1;
    }
    const int chain = c0 + tc;
    if (wig == 0 && chain < last) {
      if (ti < dim) out[(int64_t)chain * dim + ti] = ok ? x0 : start[ti];
      if (ti + 8 < dim) out[(int64_t)chain * dim + ti + 8] = ok ? x1 : start[ti + 8];
    }
    // the next chains' draws overwrite what this warp may be ahead of: dir[par] (read by slower warps)
    group_bar(bar_id, GL);
  }
}

// Regions sampled from registers: more than 8 dimensions and 65 to 1,024 face
// pairs, two to four of them per lane. SM cycles per chain and step at 14
// dimensions, from registers against run_chain_pairs' best (16 pairs per lane,
// 2 blocks per SM): 93 / 119 with 75 pairs, 112 / 175 with 125, 204 / 340 with
// 250, 391 / 674 with 500. Up to 64 pairs run_chain_pairs splits a warp over
// four chains and wins; beyond 1,024 the pairs do not fit a block's registers.
constexpr int kRegMinPairs = 65, kRegMaxPairs = 1024;
__host__ __device__ __forceinline__ bool region_in_regs(int dim, int faces) {
  const int P = (faces + 1) >> 1;
  return dim > 8 && P >= kRegMinPairs && P <= kRegMaxPairs;
}
template <int NQ>
__device__ __forceinline__ void sample_region_regs(const float* __restrict__ rows, int P, int dim,
                                                   const float* __restrict__ start, int first, int last, int mixing,
                                                   uint32_t k0, uint32_t k1, uint32_t stream,
                                                   float* __restrict__ out, RegScratch* scratch) {
  const int R = (P + 31) >> 5, W = R <= 4 ? 1 : R <= 8 ? 2 : R <= 16 ? 4 : 8;
  const int warp = threadIdx.x >> 5, gid = warp / W;
  switch ((R - reg_row(warp - gid * W, gid, W) + W - 1) / W) {  // this warp's rows
    case 2:
      sample_chains_regs<NQ, 2>(rows, P, dim, start, first, last, mixing, k0, k1, stream, W, out, scratch);
      break;
    case 3:
      sample_chains_regs<NQ, 3>(rows, P, dim, start, first, last, mixing, k0, k1, stream, W, out, scratch);
      break;
    default:
      sample_chains_regs<NQ, 4>(rows, P, dim, start, first, last, mixing, k0, k1, stream, W, out, scratch);
      break;
  }
}

// Copies P pair rows (stride floats each, 16-byte multiples) to shared memory.
__device__ __forceinline__ void stage_pairs(const float* __restrict__ rows, int P, int stride, float* sm) {
  const float4* src = reinterpret_cast<const float4*>(rows);
  float4* dst = reinterpret_cast<float4*>(sm);
  const int n = P * stride / 4;
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

// Group width for `total` chains over `grid_warps` resident warps: 8 lanes
// per chain when there are enough chains to fill the grid that way, wider
// groups when there are few (the tail of an inflation).
__host__ __device__ __forceinline__ int group_width(int64_t total, int64_t grid_warps) {
  return total >= 8 * grid_warps ? 8 : total >= 4 * grid_warps ? 16 : 32;
}

}  // namespace csd
