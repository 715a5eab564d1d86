// probe.cu -- diagnostics on the device: the FP32 FMA throughput probe (the
// denominator of the collision kernels' FP32 roofline; the measured peaks cover
// HBM and BF16 only) and the comparison of the samplers' packed quotient with
// the IEEE division.
#include <cstring>

#include "csd_internal.h"
#include "sampler_core.cuh"

namespace csd {

// 8 independent FMA chains per thread; the result is written so the chains stay live.
__global__ void __launch_bounds__(256) fma_probe_kernel(int64_t iters, float* out) {
  float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
  float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
  const float m = 0.9999999f, c = 1e-7f;
  for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
      a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
    }
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
}

// f2_quotient against __fdiv_rn: numerator s[i] by every divisor a[j], or by
// a[i] alone (paired); each half of the packed pair gets the operands in turn.
// res: mismatches, then the bits of the operands of one of them.
__global__ void __launch_bounds__(256) quotient_probe_kernel(const float* __restrict__ s, int64_t ns,
                                                             const float* __restrict__ a, int64_t na, int paired,
                                                             unsigned long long* res) {
  const int64_t total = paired ? ns : ns * na;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const float x = s[paired ? t : t % ns], y = a[paired ? t : t / ns];
    const float other = __int_as_float(0x3f800000 | (int)(t & 0x7fffff));
    float lo, hi, unused;
    f2_unpack(f2_quotient(f2_pack(x, other), f2_pack(-y, other)), &lo, &unused);
    f2_unpack(f2_quotient(f2_pack(other, x), f2_pack(other, -y)), &unused, &hi);
    const uint32_t ref = __float_as_uint(__fdiv_rn(x, y));
    if (__float_as_uint(lo) != ref || __float_as_uint(hi) != ref) {
      atomicAdd(res, 1ull);
      res[1] = (unsigned long long)__float_as_uint(x) << 32 | __float_as_uint(y);
    }
  }
}

}  // namespace csd

extern "C" csd_status_t csd_quotient_probe(const float* s, int64_t ns, const float* a, int64_t na, int32_t paired,
                                           int64_t* mismatches, float* example) {
  using namespace csd;
  CSD_CHECK(s && a && mismatches && ns > 0 && na > 0 && ns <= (1 << 24) && na <= (1 << 24) && (!paired || ns == na),
            CSD_ERR_INVALID, "the quotient probe takes 1 to 2^24 numerators and divisors, as many of each when paired");
  DevBuf buf;
  const size_t os = 256, oa = os + (((size_t)ns * 4 + 255) & ~size_t(255));
  if (csd_status_t e = buf.reserve(oa + (size_t)na * 4)) return e;
  char* base = buf.as<char>();
  CSD_CUDA_TRY(cudaMemset(base, 0, 256));
  CSD_CUDA_TRY(cudaMemcpy(base + os, s, (size_t)ns * 4, cudaMemcpyHostToDevice));
  CSD_CUDA_TRY(cudaMemcpy(base + oa, a, (size_t)na * 4, cudaMemcpyHostToDevice));
  unsigned long long* res = (unsigned long long*)base;
  quotient_probe_kernel<<<device_sm_count() * 8, 256>>>((const float*)(base + os), ns, (const float*)(base + oa), na,
                                                        paired, res);
  CSD_CUDA_TRY(cudaGetLastError());
  unsigned long long h[2];
  CSD_CUDA_TRY(cudaMemcpy(h, res, sizeof(h), cudaMemcpyDeviceToHost));
  *mismatches = (int64_t)h[0];
  if (example) {
    const uint32_t x = (uint32_t)(h[1] >> 32), y = (uint32_t)h[1];
    memcpy(example, &x, 4);
    memcpy(example + 1, &y, 4);
  }
  return CSD_OK;
}

extern "C" csd_status_t csd_fp32_fma_probe(int64_t iters, double* flops, double* seconds) {
  using namespace csd;
  CSD_CHECK(flops && seconds && iters > 0, CSD_ERR_INVALID, "null argument");
  const int sms = device_sm_count();
  const int blocks = sms * 8, threads = 256;
  float* out = nullptr;
  CSD_CUDA_TRY(cudaMalloc(&out, sizeof(float) * blocks * threads));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  fma_probe_kernel<<<blocks, threads>>>(iters / 8 + 1, out);  // warm-up
  cudaEventRecord(e0);
  fma_probe_kernel<<<blocks, threads>>>(iters, out);
  cudaEventRecord(e1);
  cudaError_t err = cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (err != cudaSuccess) {
    set_error(cudaGetErrorString(err));
    return CSD_ERR_CUDA;
  }
  *seconds = ms * 1e-3;
  *flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
  return CSD_OK;
}
