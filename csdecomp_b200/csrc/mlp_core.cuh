// mlp_core.cuh -- device code of the surrogate MLP shared by the bank's own
// kernels (mlp.cu) and the batched EI-ZO scoring stage (batch.cu): operand
// tile loads and the fused three-layer forward of one 128-row tile.
#pragma once
#include <cuda_bf16.h>

#include "umma.cuh"

namespace csd {
namespace mlp {

using bf16 = __nv_bfloat16;
constexpr int kH = 256;     // hidden width
constexpr int kIn = 16;     // padded input width
constexpr int kKC = 32;     // K chunk of a streamed operand
constexpr int kStages = 4;  // chunks in flight or in use
constexpr int kThreads = 256;

// parameter offsets within one net (floats)
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH,
              oB3 = oW3 + kH * kH, oW4 = oB3 + kH, oB4 = oW4 + kH, kParams = oB4 + 1;
// bf16 weight copies within one net: W1 [256][16], W2, W3 [out][in], W2t, W3t [in][out]
constexpr int qW1 = 0, qW2 = qW1 + kH * kIn, qW3 = qW2 + kH * kH, qW2t = qW3 + kH * kH, qW3t = qW2t + kH * kH,
              kBf = qW3t + kH * kH;

// Starts the copy of rows [r0, r0 + R) x k [k0, k0 + KC) of a K-major bf16
// matrix (row stride ld elements, `rows` x `K` valid) into an R x KC K-major
// tile; zero outside. ld, K and k0 are multiples of 8 and the base 16-byte
// aligned. (Loads through registers left every chunk waiting for its own
// loads: 25 of 30 stalled cycles per issue.)
template <int R, int KC>
__device__ __forceinline__ void load_tile(const bf16* __restrict__ src, int ld, int rows, int K, int r0, int k0,
                                          char* tile) {
  const uint32_t base = umma::smem_u32(tile);
#pragma unroll
  for (int idx0 = 0; idx0 < R * (KC >> 3); idx0 += kThreads) {
    const int idx = idx0 + threadIdx.x;
    if (R * (KC >> 3) % kThreads != 0 && idx >= R * (KC >> 3)) break;
    const int r8 = idx & 7, chunk = (idx >> 3) % (KC >> 3), rg = idx / KC;
    const int row = rg * 8 + r8, k = chunk * 8;
    const bool ok = r0 + row < rows && k0 + k < K;
    umma::copy16(base + umma::tile_offset(row, k, KC), ok ? src + (size_t)(r0 + row) * ld + k0 + k : src, ok);
  }
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// --------------------------------------------------------- fused forward
// One group = rows of one net's input. Inputs are f32 rows of `dim`
// coordinates (scaled by in_scale, zero padded to 16) or, for training, bf16
// rows already padded (xb).
struct FwdGroup {
  const float* x;   // [rows][dim] f32, read where xb is null (training groups: what xb was converted from)
  const bf16* xb;   // [rows][16] bf16, or null
  int rows, dim, net;
  float* logits;    // [rows]
  // training outputs (optional): transposed bf16 copies, leading dimension ld_t
  bf16 *xt, *h1t, *h2t, *h3t;
  int ld_t;
};

struct FwdArgs {
  const FwdGroup* groups;
  int row0;            // first row of xb in each group (training batches)
  const bf16* wb;      // bf16 weights, kBf per net
  const float* params; // f32 parameters, kParams per net (biases, w4, b4)
  float in_scale;
  int* status;
};

constexpr size_t kFwdX = 128 * kIn * 2;           // 4 KB
constexpr size_t kFwdH = 128 * kH * 2;            // 64 KB; first W1 (8 KB), read before the first epilogue writes
constexpr size_t kFwdStage = (size_t)kH * kKC * 2;  // 16 KB
constexpr size_t kFwdBias = (4 * kH + 32) * sizeof(float);  // b1, b2, b3, w4, b4
constexpr size_t kFwdSmem = kFwdX + kFwdH + kStages * kFwdStage + kFwdBias + 1024;
constexpr int kFwdBars = kStages + 1;

// Epilogue of a hidden layer: relu(acc + b) -> bf16 into the next layer's
// operand tile (and the transposed copy when training).
__device__ __forceinline__ void hidden_epilogue(uint32_t tmem, const float* bias, char* hs, bf16* ht, int ld_t,
                                                int row0, int rows) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = 32 * (warp & 3) + lane;
  const int c0 = (warp >> 2) * (kH / 2);
  for (int j = c0; j < c0 + kH / 2; j += 16) {
    float v[16];
    umma::tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)j, v);
    uint32_t p[8];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const float a = fmaxf(v[i] + bias[j + i], 0.f), b = fmaxf(v[i + 1] + bias[j + i + 1], 0.f);
      p[i >> 1] = pack2(a, b);
      v[i] = a;
      v[i + 1] = b;
    }
    *reinterpret_cast<uint4*>(hs + umma::tile_offset(r, j, kH)) = make_uint4(p[0], p[1], p[2], p[3]);
    *reinterpret_cast<uint4*>(hs + umma::tile_offset(r, j + 8, kH)) = make_uint4(p[4], p[5], p[6], p[7]);
    if (ht && row0 + r < rows) {
#pragma unroll
      for (int i = 0; i < 16; ++i) ht[(size_t)(j + i) * ld_t + row0 + r] = __float2bfloat16_rn(v[i]);
    }
  }
}

// Chunk g of the weight stream: chunks 0 .. 7 of W2, then of W3. The copies run
// three chunks ahead, across the layers' epilogues.
constexpr int kLayerChunks = kH / kKC;
__device__ __forceinline__ void load_weights(const bf16* wb, int g, char* stages) {
  if (g < 2 * kLayerChunks)
    load_tile<kH, kKC>(wb + (g < kLayerChunks ? qW2 : qW3), kH, kH, kH, 0, (g % kLayerChunks) * kKC,
                       stages + (g % kStages) * kFwdStage);
  umma::copy_commit();  // (an empty group past the end keeps the count)
}

// MMAs of one hidden layer (K = 256, chunks g0 .. g0 + 7 of the stream).
// Returns false on a barrier timeout.
__device__ __forceinline__ bool hidden_layer(uint32_t tmem, const bf16* wb, int g0, char* hs, char* stages,
                                             uint64_t* bars) {
  const uint32_t idesc = umma::instr_desc_bf16(128, kH);
  bool ok = true;
  for (int c = 0; c < kLayerChunks; ++c) {
    const int g = g0 + c, st = g % kStages;
    umma::copy_wait<kStages - 2>();  // chunk g has arrived
    umma::fence_smem_async();
    if (!__syncthreads_and(ok)) return false;
    if (threadIdx.x == 0) {
      umma::fence_after_sync();
      for (int s = 0; s < kKC / 16; ++s)
        umma::mma_bf16(tmem, umma::tile_desc(umma::smem_u32(hs), c * (kKC / 16) + s, kH),
                       umma::tile_desc(umma::smem_u32(stages + st * kFwdStage), s, kKC), idesc,
                       (c > 0 || s > 0) ? 1u : 0u);
      umma::commit(&bars[st]);
    }
    // chunk g + 3 goes where chunk g - 1 was: once its MMAs are done
    if (g > 0) ok = umma::bar_wait(&bars[(g - 1) % kStages], ((g - 1) / kStages) & 1);
    load_weights(wb, g + kStages - 1, stages);
  }
  // the last commit covers every MMA of the layer
  const int g = g0 + kLayerChunks - 1;
  ok = umma::bar_wait(&bars[g % kStages], (g / kStages) & 1) && ok;
  ok = __syncthreads_and(ok);
  umma::fence_after_sync();
  return ok;
}

static __device__ void forward_tile(const FwdArgs& a, const FwdGroup& G, int row0, char* smem, uint64_t* bars,
                             uint32_t tmem) {
  char* xs = smem;
  char* hs = xs + kFwdX;
  char* stages = hs + kFwdH;
  float* bias = reinterpret_cast<float*>(stages + kStages * kFwdStage);  // b1, b2, b3, w4, b4
  const bf16* wb = a.wb + (size_t)G.net * kBf;
  const float* pr = a.params + (size_t)G.net * kParams;
  load_tile<kH, kIn>(wb + qW1, kIn, kH, kIn, 0, 0, hs);
  umma::copy_commit();
  for (int g = 0; g < kStages - 1; ++g) load_weights(wb, g, stages);
  for (int i = threadIdx.x; i < kH; i += blockDim.x) {
    bias[i] = pr[oB1 + i];
    bias[kH + i] = pr[oB2 + i];
    bias[2 * kH + i] = pr[oB3 + i];
    bias[3 * kH + i] = pr[oW4 + i];
  }
  if (threadIdx.x == 0) bias[4 * kH] = pr[oB4];
  // input tile (128 x 16) and W1 (256 x 16), K-major, KC = 16
  for (int idx = threadIdx.x; idx < 128 * 2; idx += blockDim.x) {
    const int r = idx >> 1, half = idx & 1, row = row0 + r;
    uint32_t p[4] = {0, 0, 0, 0};
    if (row < G.rows) {
      if (G.xb) {
        uint4 v = *reinterpret_cast<const uint4*>(G.xb + (size_t)(a.row0 + row) * kIn + half * 8);
        p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
      } else {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int k = half * 8 + i;
          f[i] = k < G.dim ? G.x[(size_t)row * G.dim + k] * a.in_scale : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = pack2(f[2 * i], f[2 * i + 1]);
      }
    }
    *reinterpret_cast<uint4*>(xs + umma::tile_offset(r, half * 8, kIn)) = make_uint4(p[0], p[1], p[2], p[3]);
    if (G.xt && row < G.rows) {
      const bf16* hv = reinterpret_cast<const bf16*>(p);
#pragma unroll
      for (int i = 0; i < 8; ++i) G.xt[(size_t)(half * 8 + i) * G.ld_t + row] = hv[i];
    }
  }
  umma::copy_wait<kStages - 1>();  // W1 has arrived
  umma::fence_smem_async();
  __syncthreads();
  // layer 1: one K step
  if (threadIdx.x == 0) {
    umma::fence_after_sync();
    umma::mma_bf16(tmem, umma::tile_desc(umma::smem_u32(xs), 0, kIn), umma::tile_desc(umma::smem_u32(hs), 0, kIn),
                   umma::instr_desc_bf16(128, kH), 0u);
    umma::commit(&bars[kStages]);
  }
  bool ok = __syncthreads_and(umma::bar_wait(&bars[kStages], 0));
  umma::fence_after_sync();
  if (ok) hidden_epilogue(tmem, bias, hs, G.h1t, G.ld_t, row0, G.rows);
  umma::fence_before_sync();
  umma::fence_smem_async();
  __syncthreads();
  // layers 2 and 3
  ok = ok && hidden_layer(tmem, wb, 0, hs, stages, bars);
  if (ok) hidden_epilogue(tmem, bias + kH, hs, G.h2t, G.ld_t, row0, G.rows);
  umma::fence_before_sync();
  umma::fence_smem_async();
  __syncthreads();
  ok = ok && hidden_layer(tmem, wb, kLayerChunks, hs, stages, bars);
  umma::copy_wait<0>();
  if (!ok) {
    if (threadIdx.x == 0 && a.status) atomicExch(a.status, 1);
    return;
  }
  // layer 3 epilogue: h3 = relu(acc + b3); logit = h3 . w4 + b4 (the two warps of a lane quadrant add halves)
  __shared__ float part[128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = 32 * (warp & 3) + lane;
  const int c0 = (warp >> 2) * (kH / 2);
  float acc = 0.f;
  for (int j = c0; j < c0 + kH / 2; j += 16) {
    float v[16];
    umma::tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)j, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float h = fmaxf(v[i] + bias[2 * kH + j + i], 0.f);
      const float hb = __bfloat162float(__float2bfloat16_rn(h));
      acc = fmaf(hb, bias[3 * kH + j + i], acc);
      if (G.h3t && row0 + r < G.rows) G.h3t[(size_t)(j + i) * G.ld_t + row0 + r] = __float2bfloat16_rn(h);
    }
  }
  if (warp >= 4) part[r] = acc;
  __syncthreads();
  if (warp < 4 && row0 + r < G.rows) G.logits[row0 + r] = acc + part[r] + bias[4 * kH];
  umma::fence_before_sync();
  __syncthreads();
}

}  // namespace mlp
}  // namespace csd
