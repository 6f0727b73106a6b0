// Forward and backward pass of the surrogate's network (16 -> 4 x 256 GELU ->
// 16, padded) and its Adam step, as tcgen05 kernels with fused epilogues.
//
// Every BF16 matrix lives in device memory as the shared-memory image its
// MMA operand needs: 64-column chunks of 128-byte rows in 8-row atoms with the
// 128-byte swizzle (tc::sw128_offset).  A batch matrix is cut into tiles of 128
// rows first.  The same image is a K-major operand over its columns and an
// MN-major operand over its rows, so one copy of the activations, of the
// output gradients and of the weights serves the forward products (A W^T), the
// input gradients (dZ W) and the weight gradients (dZ^T A): nothing is
// transposed, and every operand arrives by linear bulk copies.
//
// What a step moves through memory bounds it: per hidden layer the FP32
// pre-activations (67 MB at a batch of 65536) are written and read once and
// the BF16 activations and gradients (33 MB each) written once and read twice.
// Bias, GELU, its derivative, the loss and the bias gradients run in the
// epilogues on the accumulators.  A step at a batch of 65536 on one B200 takes
// 0.45 ms (12 steps with the final read of the losses and weights); as separate
// GEMM, activation, transpose and reduction passes over FP32 results it took
// 3.67 ms.
#pragma once

#include <cuda_bf16.h>

#include "stage_ring.hpp"
#include "surrogate.hpp"
#include "tc_mma.cuh"

namespace ostc {
namespace mlp {

constexpr int kTile = 128;                           // rows of a tile
constexpr int kH = kSurHidden;                       // width of a hidden layer
constexpr uint32_t kChunk = kTile * 128;             // bytes of a 64-column chunk of a batch tile
constexpr uint32_t kTileBytes = kH / 64 * kChunk;    // a tile of a hidden layer's image
constexpr uint32_t kStage = kChunk + kH * 128;       // one 64-wide K chunk of both operands
constexpr int kThreads = 256;                        // 4 TMEM lane quarters x 2 column halves
constexpr uint32_t kLayerSmem = 2 * kStage + 1024 + 128;
constexpr uint32_t kOutSmem = kTileBytes + kH / 64 * 2048 + 1024 + 128;
constexpr uint32_t kHalf = kTile / 2 * 128;          // 64 rows of a chunk
constexpr uint32_t kDwStage = 8 * kHalf;             // 64 batch rows of two hidden layers
constexpr int kDwStages = 3;
constexpr uint32_t kDwSmem = kDwStages * kDwStage + 1024 + 128;
// CTAs of the weight-gradient launch: a share of the 148 SMs by the bytes a
// layer's gradient reads (512 B + 512 B per row for the three hidden ones,
// 512 B + 128 B for the first and the last)
constexpr int kSplitHidden = 36, kSplitThin = 20;

static_assert(kH == 256 && kSurInPad == 16 && kSurOutPad == 16, "the kernels are laid out for these widths");

__device__ __forceinline__ void expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_in(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void copy_out(void *dst, const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(tc::smem_u32(src)),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// What a CTA does before it exits when one of its waits ran out: the loader
// waits for the copies it started (`issued` chunks through the ring), the MMA
// thread, whose last commit goes to acc, for the MMAs it issued, so that neither
// can still reach this CTA's shared or tensor memory.
constexpr uint32_t kDrainPolls = 1u << 20;
template <int N>
__device__ __forceinline__ void drain(uint64_t *full, int issued) {
  for (int c = tc::StageRing<N>::first_open(issued); c < issued; ++c)
    tc::mbar_wait(&full[tc::StageRing<N>::slot(c)], tc::StageRing<N>::parity(c), kDrainPolls);
}

// MN-major SWIZZLE_128B operand: 8 K rows of 64 MN elements per 1024-byte
// atom; lbo: bytes to the next 64 MN elements (the next K atom follows at
// 1024 bytes).
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t lbo) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor bits of MN-major operands
constexpr uint32_t kAMn = 1u << 15, kBMn = 1u << 16;

__device__ __forceinline__ float gelu(float x) {
  const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x));
  return 0.5f * x * (1.f + t);
}
__device__ __forceinline__ float gelu_grad(float x) {
  const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x));
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// Byte offset of (r, c) in the image of a matrix of `rows` rows.
__host__ __device__ constexpr uint32_t image_offset(int rows, int r, int c) {
  return static_cast<uint32_t>(c >> 6) * static_cast<uint32_t>(rows) * 128u + tc::sw128_offset(r, c & 63);
}

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) { return p + ((1024 - (tc::smem_u32(p) & 1023)) & 1023); }

// 32 columns of this thread's row into the output tile's image in shared memory
__device__ __forceinline__ void stage_row(uint8_t *img, int row, int col0, const float *v) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float *u = v + 8 * p;
    *reinterpret_cast<uint4 *>(img + image_offset(kTile, row, col0 + 8 * p)) =
        make_uint4(pack2(u[0], u[1]), pack2(u[2], u[3]), pack2(u[4], u[5]), pack2(u[6], u[7]));
  }
}

// v[c] of 32 lanes summed over the lanes: lane c returns column c's sum.
__device__ __forceinline__ float column_sums(float *v, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float send = up ? v[j] : v[j + o], keep = up ? v[j + o] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// One hidden layer's product for a tile of 128 rows, 256 output columns, and
// its epilogue.  A CTA has two 48 KB stages and 256 TMEM columns, so two are
// resident per SM and one's epilogue overlaps the other's copies and MMAs.
//   BWD = false: z = in W^T + b (FP32, kept if z is given), out = GELU(z)
//   BWD = true:  out = (in W) * GELU'(z), and per-tile column sums of the FP32
//                values (the bias gradient)
// z is column-major within a tile ([tile][column][row]) so that a warp's
// accesses, one row per lane, are contiguous.
//   THIN: the contracted width is 16 (the first layer forward, the last one
//         backward) instead of 256.
template <bool BWD, bool THIN>
__global__ void __launch_bounds__(kThreads, 2) k_layer(const uint8_t *__restrict__ in, const uint8_t *__restrict__ w,
                                                       const float *__restrict__ bias, float *z, uint8_t *out,
                                                       float *colsum, int *err) {
  constexpr int NCH = THIN ? 1 : kH / 64, KSTEPS = THIN ? 1 : 4;
  using Ring = tc::StageRing<2>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align1024(smem_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + 2 * kStage), *done = full + 2, *acc = full + 4;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(full + 5);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tile = blockIdx.x;
  if (warp == 0) tc::tmem_alloc(tslot, kH);
  if (tid == 0) {
    for (int q = 0; q < 5; ++q) tc::mbar_init(&full[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  bool ok = true;
  int issued = 0;
  // BWD B operand: W as [K = its rows][N = its columns], column chunk j of
  // the image at j * rows * 128; the K chunk's rows of each
  constexpr uint32_t w_rows = THIN ? 16 : 64, w_piece = w_rows * 128;
  if (tid == 32) {  // copies
    const uint8_t *a = in + tile * NCH * kChunk;
    for (int c = 0; c < NCH; ++c) {
      const int s = Ring::slot(c);
      if (c >= 2) ok = tc::mbar_wait(&done[s], Ring::parity(c - 2));
      if (!ok) break;
      issued = c + 1;
      uint8_t *dst = smem + s * kStage;
      expect_tx(&full[s], kChunk + (BWD ? 4 * w_piece : kH * 128));
      copy_in(dst, a + c * kChunk, kChunk, &full[s]);
      if constexpr (BWD) {
        for (int j = 0; j < 4; ++j)
          copy_in(dst + kChunk + j * w_piece, w + (j * (THIN ? 16u : kH) + c * 64u) * 128u, w_piece, &full[s]);
      } else {
        copy_in(dst + kChunk, w + c * (kH * 128), kH * 128, &full[s]);
      }
    }
  } else if (tid == 0) {  // MMAs
    constexpr uint32_t idesc = tc::idesc_bf16(kTile, kH) | (BWD ? kBMn : 0u);
    for (int c = 0; c < NCH; ++c) {
      const int s = Ring::slot(c);
      ok = tc::mbar_wait(&full[s], Ring::parity(c));
      if (!ok) break;
      tc::fence_after_sync();
      const uint32_t ab = tc::smem_u32(smem + s * kStage), bb = ab + kChunk;
      for (int q = 0; q < KSTEPS; ++q)
        tc::mma_bf16(tmem, tc::desc_sw128(ab + q * 32), BWD ? desc_mn(bb + q * 2048, w_piece) : tc::desc_sw128(bb + q * 32),
                     idesc, (c > 0 || q > 0) ? 1u : 0u);
      if (c + 2 < NCH) tc::commit(&done[s]);
    }
    tc::commit(acc);  // whether or not all of them were issued
  }
  __syncwarp();
  const int row = (warp & 3) * 32 + lane, half = warp >> 2;
  float *zt = z ? z + tile * (kTile * kH) + row : nullptr;
  float zv[32];
  if constexpr (BWD) {  // the first pre-activations while the product runs
#pragma unroll
    for (int e = 0; e < 32; ++e) zv[e] = zt[(half * 128 + e) * kTile];
  }
  ok = tc::mbar_wait(acc, 0) && ok;
  ok = __syncthreads_and(ok);
  tc::fence_after_sync();
  float *red = reinterpret_cast<float *>(smem + kTileBytes);  // [4][256], past the output image
  if (ok) {
#pragma unroll 1
    for (int cc = 0; cc < 4; ++cc) {
      const int col0 = half * 128 + cc * 32;
      float v[32];
      tc::tmem_ld32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + col0, v);
      if constexpr (BWD) {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] *= gelu_grad(zv[e]);
        if (cc < 3) {
#pragma unroll
          for (int e = 0; e < 32; ++e) zv[e] = zt[(col0 + 32 + e) * kTile];
        }
        stage_row(smem, row, col0, v);
        const float s = column_sums(v, lane);
        red[(warp & 3) * kH + col0 + lane] = s;
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] += __ldg(bias + col0 + e);
        if (zt) {
#pragma unroll
          for (int e = 0; e < 32; ++e) zt[(col0 + e) * kTile] = v[e];
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = gelu(v[e]);
        stage_row(smem, row, col0, v);
      }
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) copy_out(out + tile * kTileBytes, smem, kTileBytes);
    if constexpr (BWD) colsum[tile * kH + tid] = (red[tid] + red[kH + tid]) + (red[2 * kH + tid] + red[3 * kH + tid]);
  } else {
    if (tid == 0) {
      atomicExch(err, 1);
      tc::mbar_wait(acc, 0, kDrainPolls);
    }
    if (tid == 32) drain<2>(full, issued);
    tc::fence_before_sync();
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kH);
}

// The output layer of a tile, pred = in W^T + b (16 columns, 9 used), and
// TRAIN: the loss of the tile's rows, dZ = 2 (pred - t) / (batch * 9) as BF16
// image and its column sums; otherwise pred itself (row-major).
template <bool TRAIN>
__global__ void __launch_bounds__(kTile) k_out(const uint8_t *__restrict__ in, const uint8_t *__restrict__ w,
                                               const float *__restrict__ bias, const float *__restrict__ t, int batch,
                                               float *pred, uint8_t *dz, float *colsum, double *loss, int *err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align1024(smem_raw);
  constexpr uint32_t wbytes = kH / 64 * 2048;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTileBytes + wbytes), *acc = full + 1;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(full + 2);
  __shared__ double sl[kTile / 32];
  __shared__ float sb[kTile / 32][kSurOutPad];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tile = blockIdx.x;
  if (warp == 0) tc::tmem_alloc(tslot, 32);
  if (tid == 0) {
    tc::mbar_init(full, 1);
    tc::mbar_init(acc, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  bool ok = true;
  if (tid == 0) {
    expect_tx(full, kTileBytes + wbytes);
    copy_in(smem, in + tile * kTileBytes, kTileBytes, full);
    copy_in(smem + kTileBytes, w, wbytes, full);
    ok = tc::mbar_wait(full, 0);
    if (ok) {
      tc::fence_after_sync();
      const uint32_t ab = tc::smem_u32(smem), bb = ab + kTileBytes;
      for (int q = 0; q < kH / 16; ++q)
        tc::mma_bf16(tmem, tc::desc_sw128(ab + (q >> 2) * kChunk + (q & 3) * 32),
                     tc::desc_sw128(bb + (q >> 2) * 2048 + (q & 3) * 32), tc::idesc_bf16(kTile, kSurOutPad), q > 0 ? 1u : 0u);
    }
    tc::commit(acc);
  }
  __syncwarp();
  const int64_t row = tile * kTile + tid;
  float tv[kSurOut];
  if constexpr (TRAIN) {
#pragma unroll
    for (int q = 0; q < kSurOut; ++q) tv[q] = __ldg(t + row * kSurOutPad + q);
  }
  ok = tc::mbar_wait(acc, 0) && ok;
  ok = __syncthreads_and(ok);
  tc::fence_after_sync();
  if (ok) {
    float v[kSurOutPad];
    tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16), v);
    if constexpr (TRAIN) {
      double l = 0;
      const float scale = static_cast<float>(batch) * kSurOut;
#pragma unroll
      for (int q = 0; q < kSurOutPad; ++q) {
        if (q < kSurOut) {
          const float e = v[q] + __ldg(bias + q) - tv[q];
          l += static_cast<double>(e) * e;
          v[q] = 2.f * e / scale;
        } else {
          v[q] = 0.f;
        }
      }
      uint8_t *img = dz + tile * kChunk;
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const float *u = v + 8 * p;
        *reinterpret_cast<uint4 *>(img + image_offset(kTile, tid, 8 * p)) =
            make_uint4(pack2(u[0], u[1]), pack2(u[2], u[3]), pack2(u[4], u[5]), pack2(u[6], u[7]));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
        for (int q = 0; q < kSurOut; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
      }
      if (lane == 0) {
        sl[warp] = l;
#pragma unroll
        for (int q = 0; q < kSurOutPad; ++q) sb[warp][q] = v[q];
      }
      __syncthreads();
      if (tid < kSurOutPad) colsum[tile * kSurOutPad + tid] = (sb[0][tid] + sb[1][tid]) + (sb[2][tid] + sb[3][tid]);
      if (tid == 0) loss[tile] = (sl[0] + sl[1]) + (sl[2] + sl[3]);
    } else {
#pragma unroll
      for (int q = 0; q < kSurOutPad; ++q) pred[row * kSurOutPad + q] = v[q] + __ldg(bias + q);
    }
  } else if (tid == 0) {
    atomicExch(err, 1);
    tc::mbar_wait(full, 0, kDrainPolls);
    tc::mbar_wait(acc, 0, kDrainPolls);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 32);
}

// The weight gradients of every layer in one launch, out[m][n] = sum over the
// batch of P[b][m] Q[b][n] with P 256 wide and Q 256 or 16 wide, both MN-major
// from their images: layer 0 P = dZ, Q = features; hidden layers P = dZ,
// Q = activations; the last one P = activations, Q = dZ (its transpose).  A
// CTA takes a range of 64-row half tiles through three stages into 2 x 256
// TMEM columns and writes its partial sum, column-major (out[n][m]).
struct DwArgs {
  const uint8_t *p[kSurLayers], *q[kSurLayers];
  float *part[kSurLayers];  // [split][n][256]
  int splits[kSurLayers];
  int halves;  // 64-row half tiles of the batch
};

__global__ void __launch_bounds__(kThreads, 1) k_dw(DwArgs a, int *err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align1024(smem_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + kDwStages * kDwStage), *done = full + kDwStages,
           *acc = done + kDwStages;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(acc + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int layer = 0, split = blockIdx.x;
  while (split >= a.splits[layer]) split -= a.splits[layer++];
  const bool thin = layer == 0 || layer == kSurLayers - 1;
  const int per = (a.halves + a.splits[layer] - 1) / a.splits[layer];
  const int h0 = split * per, h1 = min(a.halves, h0 + per), nh = max(0, h1 - h0);
  if (warp == 0) tc::tmem_alloc(tslot, 512);
  if (tid == 0) {
    for (int q = 0; q < 2 * kDwStages + 1; ++q) tc::mbar_init(&full[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  bool ok = true;
  const int nq = thin ? 1 : 4;  // 64-column chunks of Q
  using Ring = tc::StageRing<kDwStages>;
  int issued = 0;
  if (tid == 32) {
    for (int c = 0; c < nh; ++c) {
      const int s = Ring::slot(c), h = h0 + c;
      if (c >= kDwStages) ok = tc::mbar_wait(&done[s], Ring::parity(c - kDwStages));
      if (!ok) break;
      issued = c + 1;
      uint8_t *dst = smem + s * kDwStage;
      expect_tx(&full[s], (4 + nq) * kHalf);
      const size_t t = h >> 1, r = (h & 1) * kHalf;
      for (int j = 0; j < 4; ++j) copy_in(dst + j * kHalf, a.p[layer] + t * kTileBytes + j * kChunk + r, kHalf, &full[s]);
      for (int j = 0; j < nq; ++j)
        copy_in(dst + (4 + j) * kHalf, a.q[layer] + t * (nq * kChunk) + j * kChunk + r, kHalf, &full[s]);
    }
  } else if (tid == 0) {
    const uint32_t idesc = tc::idesc_bf16(128, thin ? 16 : kH) | kAMn | kBMn;
    for (int c = 0; c < nh; ++c) {
      const int s = Ring::slot(c);
      ok = tc::mbar_wait(&full[s], Ring::parity(c));
      if (!ok) break;
      tc::fence_after_sync();
      const uint32_t pb = tc::smem_u32(smem + s * kDwStage), qb = pb + 4 * kHalf;
      for (int q = 0; q < 4; ++q)
        for (int m = 0; m < 2; ++m)
          tc::mma_bf16(tmem + m * 256, desc_mn(pb + 2 * m * kHalf + q * 2048, kHalf), desc_mn(qb + q * 2048, kHalf),
                       idesc, (c > 0 || q > 0) ? 1u : 0u);
      tc::commit(&done[s]);
    }
    tc::commit(acc);
  }
  __syncwarp();
  ok = tc::mbar_wait(acc, 0, 1u << 26) && ok;
  ok = __syncthreads_and(ok);
  tc::fence_after_sync();
  if (ok) {
    const int n_cols = thin ? 16 : kH, m = (warp >> 2) * 128 + (warp & 3) * 32 + lane;
    float *o = a.part[layer] + static_cast<size_t>(split) * n_cols * kH + m;
    const uint32_t ta = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * 256;
#pragma unroll 1
    for (int c0 = 0; c0 < n_cols; c0 += 16) {
      float v[16];
      if (nh > 0) {
        tc::tmem_ld16(ta + c0, v);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0.f;
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) o[(c0 + e) * kH] = v[e];
    }
  } else {
    if (tid == 0) {
      atomicExch(err, 1);
      tc::mbar_wait(acc, 0, kDrainPolls);
    }
    if (tid == 32) drain<kDwStages>(full, issued);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// Sums the partial gradients and takes the Adam step (grad null), or stores
// the gradient in the flat parameter order (per layer W, then b); nothing after
// a wait that ran out, so that the weights stay those of the last whole step.  Blocks of
// 32 x 8 threads: kWeightBlocks tiles of 32 x 32 weights, then 32 bias columns
// each, then the loss.
struct StepArgs {
  float *w[kSurLayers], *b[kSurLayers], *mw[kSurLayers], *vw[kSurLayers], *mb[kSurLayers], *vb[kSurLayers];
  uint8_t *img[kSurLayers];
  const float *part[kSurLayers], *colsum[kSurLayers];
  int splits[kSurLayers], tiles, batch;
  const double *loss_part;
  double *loss;
  float *grad;
  const int *err;  // not 0: a wait of an earlier kernel ran out, its results are not there
  float lr, b1, b2, eps, bc1, bc2;
};
constexpr int kThinBlocks = kH / 32, kHiddenBlocks = kThinBlocks * kThinBlocks;
constexpr int kWeightBlocks = 2 * kThinBlocks + 3 * kHiddenBlocks;
constexpr int kBiasBlocks = 4 * kThinBlocks + 1;
constexpr int kStepBlocks = kWeightBlocks + kBiasBlocks + 1;

__device__ __forceinline__ float adam(const StepArgs &a, float *p, float *m, float *v, float g) {
  const float mi = a.b1 * *m + (1 - a.b1) * g, vi = a.b2 * *v + (1 - a.b2) * g * g;
  *m = mi;
  *v = vi;
  return *p -= a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
}

__device__ __forceinline__ int flat_offset(int layer, bool bias) {
  constexpr int thin = 16 * kH, wide = kH * kH;
  int off = 0;
  for (int l = 0; l < layer; ++l) off += (l == 0 || l == kSurLayers - 1 ? thin : wide) + (l == kSurLayers - 1 ? 16 : kH);
  return bias ? off + (layer == 0 || layer == kSurLayers - 1 ? thin : wide) : off;
}

__global__ void __launch_bounds__(256) k_step(StepArgs a) {
  if (*a.err) return;
  __shared__ float tile[32][33];
  const int x = threadIdx.x, y = threadIdx.y;
  int blk = blockIdx.x;
  if (blk < kWeightBlocks) {
    int layer = 0;
    if (blk >= kThinBlocks) {
      blk -= kThinBlocks;
      layer = 1 + min(blk / kHiddenBlocks, 3);
      blk -= (layer - 1) * kHiddenBlocks;
    }
    const bool thin = layer == 0 || layer == kSurLayers - 1, last = layer == kSurLayers - 1;
    const int n_cols = thin ? 16 : kH, m0 = (blk % kThinBlocks) * 32, n0 = blk / kThinBlocks * 32;
    const float *p = a.part[layer] + static_cast<size_t>(n0 + y) * kH + m0 + x;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const int rows = thin ? 2 : 4;
#pragma unroll 4
    for (int q = 0; q < a.splits[layer]; ++q) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < rows) s[e] += __ldg(p + (static_cast<size_t>(q) * n_cols + 8 * e) * kH);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) tile[y + 8 * e][x] = s[e];
    __syncthreads();
    const int din = layer == 0 ? 16 : kH, dout = last ? 16 : kH;
    for (int e = 0; e < 4; ++e) {
      // the last layer's partials are its transpose: m is the input column
      const int yy = y + 8 * e, r = last ? n0 + yy : m0 + yy, k = last ? m0 + x : n0 + x;
      if (r >= dout || k >= din) continue;
      const float g = last ? tile[yy][x] : tile[x][yy];
      const int idx = r * din + k;
      if (a.grad) {
        a.grad[flat_offset(layer, false) + idx] = g;
      } else {
        const float v = adam(a, a.w[layer] + idx, a.mw[layer] + idx, a.vw[layer] + idx, g);
        *reinterpret_cast<__nv_bfloat16 *>(a.img[layer] + image_offset(dout, r, k)) = __float2bfloat16_rn(v);
      }
    }
    return;
  }
  blk -= kWeightBlocks;
  if (blk < kBiasBlocks) {
    const int layer = blk / kThinBlocks, width = layer == kSurLayers - 1 ? 16 : kH;
    const int c = blk % kThinBlocks * 32 + x;
    float s = 0.f;
    if (c < width)
      for (int t = y; t < a.tiles; t += 8) s += __ldg(a.colsum[layer] + static_cast<size_t>(t) * width + c);
    tile[y][x] = s;
    __syncthreads();
    if (y == 0 && c < width) {
      float g = 0.f;
      for (int q = 0; q < 8; ++q) g += tile[q][x];
      if (a.grad)
        a.grad[flat_offset(layer, true) + c] = g;
      else
        adam(a, a.b[layer] + c, a.mb[layer] + c, a.vb[layer] + c, g);
    }
    return;
  }
  // the mean loss of the batch
  __shared__ double sl[256];
  const int id = y * 32 + x;
  double l = 0;
  for (int t = id; t < a.tiles; t += 256) l += a.loss_part[t];
  sl[id] = l;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (id < o) sl[id] += sl[id + o];
    __syncthreads();
  }
  if (id == 0) *a.loss = sl[0] / (static_cast<double>(a.batch) * kSurOut);
}

}  // namespace mlp
}  // namespace ostc
