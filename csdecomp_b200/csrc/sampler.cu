// sampler.cu -- hit-and-run sampling in H-polytopes.
//
// Reference: uniformSampleInHPolyhedronKernel, one thread per sample chain,
// cuda_hit_and_run_sampling.cu:18-119: a Gaussian direction per mixing step,
// slack b - A x and A dir per face, theta interval from the sign of (A dir)_i,
// theta = u * (0.999999 * theta_max - theta_min) + theta_min (:106-107).
// Same chain here with the draws of csd_rng.cuh, by 8 to 32 lanes or, where
// there are chains enough to fill the GPU that way, by one thread
// (chain_faces).
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <type_traits>

#include "csd_internal.h"
#include "csd_rng.cuh"
#include "sampler_core.cuh"

namespace csd {

constexpr size_t kUniformStageBytes = 48 * 1024 - 64;  // with the flag, what a block has without being asked for more
// Floats of a row: coefficients, offsets, padded so that 8 consecutive rows fall on different banks.
__host__ __device__ constexpr int uniform_stride(int nq) { return nq == 7 ? 36 : 4 * nq + 4; }
// Coordinate pairs that the packed rows of a dimension hold.
__host__ __device__ constexpr int uniform_pairs(int dim) { return dim <= 4 ? 2 : dim <= 8 ? 4 : dim <= 14 ? 7 : 8; }

// Face counts of the polytopes sampled by a thread per chain (up to `few`, from
// `many` on) in a call of `total` chains; both kernels look, each leaves the
// other its polytopes. A thread per chain fills the GPU from some 12,000 chains
// on, later the more faces it walks; then its draws and position cost one lane
// instead of eight, and up to 44 faces (58 above 8 dimensions) that outweighs
// sharing the faces out. Thread against group, us: 7 dimensions, 28 faces 71 /
// 32 with 16,000 chains, 128 / 160 with 100,000, 1,416 / 1,918 with 1.6 million;
// 114 faces 4,783 / 3,963; 2 dimensions, 12 faces 419 / 992. Rows beyond the
// staging buffer are read from global memory, by all threads alike (a thread
// per chain) or by each lane of a group elsewhere: 1,514 faces at 7 dimensions
// 2,880 / 828 with 16,000 chains, 19,100 / 25,100 with 480,000; 828 faces at 14
// dimensions 14,500 / 14,000, 2,028 faces 42,300 / 55,600.
struct ChainFaces {
  int few, many;
  __host__ __device__ bool thread(int F) const { return F <= few || F >= many; }
};
static ChainFaces chain_faces(int dim, int64_t total) {
  const int staged = 2 * (int)(kUniformStageBytes / (uniform_stride(uniform_pairs(dim)) * sizeof(float)));
  const int64_t least = total < 12000 ? -1 : total >= 60000 ? 58 : (total - 12000) / 1500;
  return {(int)std::min<int64_t>(least, dim <= 8 ? 44 : 58),
          total >= 80000 ? std::max(staged + 1, dim <= 8 ? 0 : 1001) : INT32_MAX};
}
// Where only the device has the face counts, calls of fewer chains are all left to the groups (a launch that finds
// nothing to do costs 2 us).
constexpr int64_t kChainThreadMinUnseen = 24000;

// Direction (dim Gaussians) and the theta uniform of one mixing step.
// Gaussian pair g uses words 2g (radius) and 2g+1 (angle); the theta uniform
// is word 2*ceil(dim/2). Words 4k..4k+3 come from Philox block k.
template <int MAXD>
__device__ __forceinline__ void step_draws(uint32_t k0, uint32_t k1, uint32_t chain, uint32_t stream, uint32_t step,
                                           int dim, float* dir, float* u_theta) {
  const int npairs = (dim + 1) >> 1;
  uint32_t w[4];
  int have_block = -1;
#pragma unroll
  for (int g = 0; g < (MAXD + 1) / 2; ++g) {
    if (g < npairs) {
      int blk = (2 * g) >> 2;
      if (blk != have_block) {
        philox4x32_10(step, chain, stream, (uint32_t)blk, k0, k1, w);
        have_block = blk;
      }
      float u = u01_open0(w[(2 * g) & 3]);
      float v = u01_open1(w[(2 * g + 1) & 3]);
      float rad = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(u)));
      float sn, cs;
      sincos_2pi(v, &sn, &cs);
      dir[2 * g] = __fmul_rn(rad, cs);
      if (2 * g + 1 < MAXD) dir[2 * g + 1] = __fmul_rn(rad, sn);
    }
  }
  int tw = 2 * npairs;
  int blk = tw >> 2;
  if (blk != have_block) philox4x32_10(step, chain, stream, (uint32_t)blk, k0, k1, w);
  *u_theta = u01_open0(w[tw & 3]);
}

// One hit-and-run chain (cuda_hit_and_run_sampling.cu:57-118): returns false
// if a line search found an empty theta interval. x holds the start on entry.
template <int MAXD>
__device__ __forceinline__ bool run_chain(const float* __restrict__ Ap, const float* __restrict__ bp, int F, int dim,
                                          int mixing, uint32_t k0, uint32_t k1, uint32_t chain, uint32_t stream,
                                          float* x) {
  float dir[MAXD];
#pragma unroll
  for (int k = 0; k < MAXD; ++k) dir[k] = 0.f;
  for (int step = 0; step < mixing; ++step) {
    float ut;
    step_draws<MAXD>(k0, k1, chain, stream, (uint32_t)step, dim, dir, &ut);
    float tmax = FLT_MAX, tmin = -FLT_MAX;
    for (int f = 0; f < F; ++f) {
      const float* a = Ap + (int64_t)f * dim;
      float ax = __fmul_rn(a[0], x[0]);
      float ad = __fmul_rn(a[0], dir[0]);
#pragma unroll
      for (int k = 1; k < MAXD; ++k) {
        if (k < dim) {
          float ak = a[k];
          ax = __fmaf_rn(ak, x[k], ax);
          ad = __fmaf_rn(ak, dir[k], ad);
        }
      }
      float lb = __fsub_rn(bp[f], ax);
      if (ad < 0.0f)
        tmin = fmaxf(tmin, __fdiv_rn(lb, ad));
      else if (ad > 0.0f)
        tmax = fminf(tmax, __fdiv_rn(lb, ad));
    }
    if (isinf(tmax) || isinf(tmin) || tmax < tmin) return false;
    double th = __dadd_rn(__dmul_rn((double)ut, __dsub_rn(__dmul_rn(0.999999, (double)tmax), (double)tmin)),
                          (double)tmin);
    float theta = __double2float_rn(th);
#pragma unroll
    for (int k = 0; k < MAXD; ++k)
      if (k < dim) x[k] = __fmaf_rn(theta, dir[k], x[k]);
  }
  return true;
}

// Blocks per SM: one wave of chains more or less is the whole difference at 100,000 chains (up to 4 dimensions the
// compiler finds more by itself).
template <int MAXD>
__global__ void __launch_bounds__(128, MAXD > 8 ? 7 : MAXD > 4 ? 9 : 0)
    chain_kernel(const float* __restrict__ A, const float* __restrict__ b, const int32_t* __restrict__ face_off,
                 int num_poly, int dim, const float* __restrict__ starts, int S, int mixing, uint32_t k0, uint32_t k1,
                 float* __restrict__ out, int* num_failed, ChainFaces faces) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, total = (int64_t)num_poly * S;
  if (i >= total) return;
  const int poly = (int)(i / S), s = (int)(i % S);
  const int f0 = face_off[poly], F = face_off[poly + 1] - f0;
  if (!faces.thread(F)) return;
  float x[MAXD];
#pragma unroll
  for (int k = 0; k < MAXD; ++k) x[k] = k < dim ? starts[(int64_t)poly * dim + k] : 0.f;
  const bool ok = run_chain<MAXD>(A + (int64_t)f0 * dim, b + f0, F, dim, mixing, k0, k1, (uint32_t)s, (uint32_t)poly, x);
  if (!ok && num_failed) atomicAdd(num_failed, 1);
  // a chain whose line search fails writes NaN
  float* dst = out + i * dim;
#pragma unroll
  for (int k = 0; k < MAXD; ++k)
    if (k < dim) dst[k] = ok ? x[k] : __int_as_float(0x7fc00000);
}

// Chains of num_poly polytopes, G lanes each; block = `chunk` chains of one
// polytope (cpp chunks per polytope), whose faces it stages as face-pair rows
// with the offsets b where the EI-ZO rows have start slacks. A lane walks
// pairs gl, gl + G, ...: both dot products (b - A x and A dir are recomputed
// every step) as packed FMAs in the serial chain's order, the quotients packed
// (theta_bits); every lane carries the whole position. Polytopes whose rows do
// not fit the staging buffer are read face by face from global memory. Same
// draws and operations per face as run_chain, and order-free bounds: the
// chain is the serial chain's bit for bit.
template <int NQ, int G>  // NQ coordinate pairs (dim rounded up)
__global__ void __launch_bounds__(256, NQ <= 4 ? 4 : 2)
    hit_and_run_kernel(const float* __restrict__ A, const float* __restrict__ b, const int32_t* __restrict__ face_off,
                       int dim, const float* __restrict__ starts, int S, int mixing, uint32_t k0, uint32_t k1,
                       float* __restrict__ out, int* num_failed, int chunk, int cpp, ChainFaces faces) {
  extern __shared__ __align__(16) float sm[];
  constexpr int MAXD = 2 * NQ, RS = uniform_stride(NQ);
  const int poly = blockIdx.x / cpp, first = (blockIdx.x % cpp) * chunk, last = min(S, first + chunk);
  const int f0 = face_off[poly], F = face_off[poly + 1] - f0, P = (F + 1) >> 1;
  if (faces.thread(F)) return;  // chain_kernel's (uniform across the block)
  const float* Ap = A + (int64_t)f0 * dim;
  const float* bp = b + f0;
  const bool staged = (size_t)P * RS * sizeof(float) <= kUniformStageBytes;
  // coefficients beyond kMaxCoeff: one division per face. (A flag in shared memory is known to be uniform; with the
  // result of a block vote the compiler keeps the step loop ready for divergence, 4% of it.)
  __shared__ int big;
  if (threadIdx.x == 0) big = 0;
  if (staged) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * P * MAXD; i += blockDim.x) {
      const int p = i / (2 * MAXD), k = (i >> 1) % MAXD, f = min(2 * p + (i & 1), F - 1);  // an odd count repeats its last face
      const float v = k < dim ? Ap[(int64_t)f * dim + k] : 0.f;
      sm[p * RS + 2 * k + (i & 1)] = v;
      if (!(fabsf(v) <= kMaxCoeff)) big = 1;
    }
    for (int i = threadIdx.x; i < 2 * P; i += blockDim.x) sm[(i >> 1) * RS + 2 * MAXD + (i & 1)] = bp[min(i, F - 1)];
    __syncthreads();
  }
  const int gl = threadIdx.x & (G - 1), ngroups = blockDim.x / G;
  const int npairs = (dim + 1) >> 1, JB = (npairs >> 1) + 1;
  const int steps = min(kDrawSteps, G / JB), tq = gl / JB, bq = gl - tq * JB;  // draws as run_chain_pairs
  const uint32_t stream = (uint32_t)poly;
  for (int c0 = first; c0 < last; c0 += ngroups) {
    const int mine = c0 + threadIdx.x / G, chain = min(mine, last - 1);
    uint64_t xx[MAXD], dd[MAXD];  // (x_k, x_k), (-dir_k, -dir_k)
#pragma unroll
    for (int k = 0; k < MAXD; ++k) {
      const float x = k < dim ? starts[(int64_t)poly * dim + k] : 0.f;
      xx[k] = f2_pack(x, x);
    }
    bool ok = true;
    float c0a = 0.f, c1a = 0.f, c0b = 0.f, c1b = 0.f;
    int t = 0;
    for (int step = 0; step < mixing; ++step) {
      if (t == 0) {
        uint32_t w[4];
        philox4x32_10((uint32_t)(step + tq), (uint32_t)chain, stream, (uint32_t)bq, k0, k1, w);
        const float ua = u01_open0(w[0]), ub = u01_open0(w[2]);
        const float rada = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ua)));
        const float radb = __fsqrt_rn(__fmul_rn(-2.0f, log_unit(ub)));
        float sna, csa, snb, csb;
        sincos_2pi(u01_open1(w[1]), &sna, &csa);
        sincos_2pi(u01_open1(w[3]), &snb, &csb);
        c0a = 2 * bq < npairs ? -__fmul_rn(rada, csa) : ua;
        c1a = -__fmul_rn(rada, sna);
        c0b = 2 * bq + 1 < npairs ? -__fmul_rn(radb, csb) : ub;
        c1b = -__fmul_rn(radb, snb);
      }
      const int base = t * JB;
#pragma unroll
      for (int k = 0; k < MAXD; ++k) {
        const float v = ((k >> 1) & 1) ? ((k & 1) ? c1b : c0b) : ((k & 1) ? c1a : c0a);
        const float dk = __shfl_sync(0xffffffffu, v, base + (k >> 2), G);
        dd[k] = f2_pack(dk, dk);
      }
      const float ut = __shfl_sync(0xffffffffu, (npairs & 1) ? c0b : c0a, base + (npairs >> 1), G);
      // pairs gl, gl + G, ... (staged): slacks and -(a . dir) of pair p
      auto pair = [&](int p, uint64_t& s, uint64_t& na) {
        const ulonglong2* row = reinterpret_cast<const ulonglong2*>(sm + p * RS);
        uint64_t ax = 0ull;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {  // coefficients past dim are zero
          const ulonglong2 v = row[q];
          ax = q == 0 ? f2_mul(v.x, xx[0]) : f2_fma(v.x, xx[2 * q], ax);
          na = q == 0 ? f2_mul(v.x, dd[0]) : f2_fma(v.x, dd[2 * q], na);
          ax = f2_fma(v.y, xx[2 * q + 1], ax);
          na = f2_fma(v.y, dd[2 * q + 1], na);
        }
        s = f2_sub(*reinterpret_cast<const uint64_t*>(sm + p * RS + 2 * MAXD), ax);
      };
      float tmax = FLT_MAX, tmin = -FLT_MAX;
      for (int pass = staged && !big ? 0 : 1;; ++pass) {
        if (pass == 0) {
          ThetaBits tb = theta_bits_start();
          for (int p = gl; p < P; p += G) {
            uint64_t s, na;
            pair(p, s, na);
            theta_bits(tb, s, na);
          }
          // a slack too small for the packed quotients: theta_max = 0 asks for the second pass
          tmax = tb.slack < __float_as_int(kMinSlack) ? 0.f : __uint_as_float(tb.hi);
          tmin = __int_as_float(tb.lo);
        } else if (staged) {
          tmax = FLT_MAX;
          tmin = -FLT_MAX;
          for (int p = gl; p < P; p += G) {
            uint64_t s, na;
            pair(p, s, na);
            theta_bounds_slow(&s, &na, 1, tmin, tmax);
          }
        } else {
          const float* a = Ap + (int64_t)gl * dim;
          for (int f = gl; f < F; f += G, a += G * dim) {
            float x0, d0, hi;
            f2_unpack(xx[0], &x0, &hi);
            f2_unpack(dd[0], &d0, &hi);
            float ax = __fmul_rn(a[0], x0), na = __fmul_rn(a[0], d0);
#pragma unroll
            for (int k = 1; k < MAXD; ++k)
              if (k < dim) {
                f2_unpack(xx[k], &x0, &hi);
                f2_unpack(dd[k], &d0, &hi);
                ax = __fmaf_rn(a[k], x0, ax);
                na = __fmaf_rn(a[k], d0, na);
              }
            theta_bound(__fsub_rn(bp[f], ax), -na, tmin, tmax);
          }
        }
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
          tmin = fmaxf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o, G));
          tmax = fminf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o, G));
        }
        const bool in_range = tmax >= kMinTheta && tmax < kMaxTheta && -tmin >= kMinTheta && -tmin < kMaxTheta;
        if (pass || __all_sync(0xffffffffu, in_range)) break;  // uniform: the warp's groups share the shuffles
      }
      if (isinf(tmax) || isinf(tmin) || tmax < tmin) ok = false;
      if (ok) {
        const double th = __dadd_rn(__dmul_rn((double)ut, __dsub_rn(__dmul_rn(0.999999, (double)tmax), (double)tmin)),
                                    (double)tmin);
        const float nth = -__double2float_rn(th);
        const uint64_t nth2 = f2_pack(nth, nth);
#pragma unroll
        for (int k = 0; k < MAXD; ++k)
          if (k < dim) xx[k] = f2_fma(nth2, dd[k], xx[k]);
      }
      t = t + 1 == steps ? 0 : t + 1;
    }
    if (mine < last && gl == 0) {
      if (!ok && num_failed) atomicAdd(num_failed, 1);
      // a chain whose line search fails writes NaN
      float* dst = out + ((int64_t)poly * S + chain) * dim;
#pragma unroll
      for (int k = 0; k < MAXD; ++k)
        if (k < dim) dst[k] = ok ? __uint_as_float((uint32_t)xx[k]) : __int_as_float(0x7fc00000);
    }
  }
}

// EI-ZO sampler over one region (the single inflation and the
// allocation-free inflation), whose face count is read on the device: the
// region's face-pair rows are staged in shared memory once per block when
// they fit (else the chains read them from global memory, through L1), and
// the block's chains run with G lanes each (sampler_core.cuh; G from the
// chain count, widened so that a lane holds at most kRegionKP face pairs).
constexpr int kRegionKP = 8;
constexpr size_t kRegionStageBytes = 104 * 1024;  // two blocks per SM
static_assert(kMaxRegionFaces <= 2 * 256 * kRegionKP, "the widest group samples the largest region");

__global__ void __launch_bounds__(256, 2) sample_region_kernel(const float* __restrict__ rows,
                                                              const int* __restrict__ num_faces_dev, int dim,
                                                              const float* __restrict__ start, int S, int mixing,
                                                              uint32_t k0, uint32_t k1, uint32_t stream,
                                                              float* __restrict__ out) {
  extern __shared__ __align__(16) float smf[];  // the face loop reads 16-byte vectors
  __shared__ GroupScratch gsa[kMaxWideGroups];
  const int F = *num_faces_dev;
  const int P = (F + 1) >> 1, rs = pair_stride(dim);
  const int G = pair_group_width(group_width(S, (int64_t)gridDim.x * (blockDim.x >> 5)), P, kRegionKP);
  const int per = (S + gridDim.x - 1) / gridDim.x;
  const int first = blockIdx.x * per, last = min(S, first + per);
  if (first >= last || G == 0) return;  // uniform across the block (the host bounds F)
  const bool fits = (size_t)P * rs * sizeof(float) <= kRegionStageBytes;
  if (fits) {
    stage_pairs(rows, P, rs, smf);
    __syncthreads();
  }
  // separate calls for staged and global rows (shared-memory loads in the staged face loop)
  if (fits) {
    if (dim <= 8)
      sample_region<8, kRegionKP>(G, smf, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
    else
      sample_region<16, kRegionKP>(G, smf, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
  } else {
    if (dim <= 8)
      sample_region<8, kRegionKP>(G, rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
    else
      sample_region<16, kRegionKP>(G, rows, P, dim, start, first, last, mixing, k0, k1, stream, out, gsa);
  }
}

csd_status_t launch_sample_region(const float* rows, const int* num_faces_dev, int dim, const float* start, int S,
                                  int mixing, uint64_t seed, uint32_t stream, float* out, cudaStream_t st) {
  if (S <= 0) return CSD_OK;
  CSD_CHECK(dim >= 1 && dim <= kMaxDim, CSD_ERR_DIMENSION, "dimension must be in [1, 16]");
  static std::atomic<bool> attr_set[64] = {};  // per device: limit raised (any thread)
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !attr_set[dev]) {
    CSD_CUDA_TRY(raise_smem_limit(sample_region_kernel, (int)kRegionStageBytes));
    if (dev < 64) attr_set[dev] = true;
  }
  const int sms = device_sm_count();
  const int blocks = (int)std::min<int64_t>(((int64_t)S + 7) / 8, (int64_t)sms * 2);
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  sample_region_kernel<<<blocks, 256, kRegionStageBytes, st>>>(rows, num_faces_dev, dim, start, S, mixing, k0, k1,
                                                                stream, out);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

__global__ void put_faces_kernel(const float* __restrict__ A, const float* __restrict__ b, int F, int dim,
                                 const float* __restrict__ x0, float* __restrict__ rows) {
  put_faces(A, b, F, dim, x0, rows, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

csd_status_t launch_put_faces(const float* A, const float* b, int F, int dim, const float* x0, float* rows,
                              cudaStream_t st) {
  if (F <= 0) return CSD_OK;
  const int pairs = (F + 1) / 2;
  put_faces_kernel<<<(pairs + 127) / 128, 128, 0, st>>>(A, b, F, dim, x0, rows);
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

csd_status_t launch_hit_and_run(const float* A, const float* b, const int32_t* face_off, int num_poly, int dim,
                                const float* starts, int S, int mixing, uint64_t seed, float* out, int* num_failed,
                                cudaStream_t st, const int32_t* face_off_host) {
  const int64_t total = (int64_t)num_poly * S;
  if (total <= 0) return CSD_OK;
  CSD_CHECK(dim >= 1 && dim <= kMaxDim, CSD_ERR_DIMENSION, "dimension must be in [1, 16]");
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  // polytopes for a thread per chain and for groups: known where the host has the face counts, else each kernel looks
  ChainFaces faces = chain_faces(dim, total);
  if (!face_off_host && total < kChainThreadMinUnseen) faces = {-1, INT32_MAX};
  bool threads = faces.few >= 0 || faces.many < INT32_MAX, grouped = true;
  if (threads && face_off_host) {
    threads = grouped = false;
    for (int p = 0; p < num_poly; ++p) (faces.thread(face_off_host[p + 1] - face_off_host[p]) ? threads : grouped) = true;
  }
  if (threads) {
    const int64_t blocks = (total + 127) / 128;
    CSD_CHECK(blocks < (1ll << 31), CSD_ERR_CAPACITY, "too many samples");
    auto launch = [&](auto kernel) {
      kernel<<<(unsigned)blocks, 128, 0, st>>>(A, b, face_off, num_poly, dim, starts, S, mixing, k0, k1, out, num_failed, faces);
    };
    dim <= 2 ? launch(chain_kernel<2>) : dim <= 4 ? launch(chain_kernel<4>) : dim <= 8 ? launch(chain_kernel<8>)
                                                                                       : launch(chain_kernel<16>);
    CSD_CUDA_TRY(cudaGetLastError());
  }
  if (!grouped) return CSD_OK;
  // 8 lanes per chain once that gives every SM 16 warps, wider groups for fewer chains
  const int64_t warps = (int64_t)device_sm_count() * 16;
  const int G = total * 8 / 32 >= warps ? 8 : total * 16 / 32 >= warps ? 16 : 32;
  const int groups = 256 / G;
  // a block runs several rounds of chains only when there are blocks to spare (its staging is then shared)
  const int64_t rounds = std::max<int64_t>(1, std::min<int64_t>(16, total / (groups * 4 * (int64_t)device_sm_count())));
  const int chunk = (int)std::min<int64_t>(groups * rounds, ((int64_t)S + groups - 1) / groups * groups);
  const int cpp = (S + chunk - 1) / chunk;
  const int64_t blocks = (int64_t)num_poly * cpp;
  CSD_CHECK(blocks < (1ll << 31), CSD_ERR_CAPACITY, "too many samples");
  auto launch = [&](auto kernel) {
    kernel<<<(unsigned)blocks, 256, kUniformStageBytes, st>>>(A, b, face_off, dim, starts, S, mixing, k0, k1, out,
                                                              num_failed, chunk, cpp, faces);
  };
  auto by_width = [&](auto nq) {
    constexpr int NQ = decltype(nq)::value;
    G == 8 ? launch(hit_and_run_kernel<NQ, 8>) : G == 16 ? launch(hit_and_run_kernel<NQ, 16>)
                                                         : launch(hit_and_run_kernel<NQ, 32>);
  };
  switch (uniform_pairs(dim)) {
    case 2: by_width(std::integral_constant<int, 2>()); break;
    case 4: by_width(std::integral_constant<int, 4>()); break;
    case 7: by_width(std::integral_constant<int, 7>()); break;
    default: by_width(std::integral_constant<int, 8>());
  }
  CSD_CUDA_TRY(cudaGetLastError());
  return CSD_OK;
}

}  // namespace csd
