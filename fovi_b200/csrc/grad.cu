// Passes around the backward contractions of KNNConv: ReLU mask with bias sums (where no input gradient kernel has done it: knnconv_tc2.cu), column sums, and a layout change that makes the batch index the
// innermost (contiguous) one, so that it can play the role of the channels in the tensor-core kernel (fovi_knnconv_forward_scatter_add).
#include <algorithm>

#include <cuda_bf16.h>

#include "common.cuh"

namespace {

// src: logical [B, I, J], element (b,i,j) at b*sb + i*si + j*sj, with si == 1 (FAST_I) or sj == 1 (!FAST_I).
// dst: [I, Jp, Bp] bf16, zero where j >= J or b >= B.  32x32 tiles of (batch, fast index) go through shared memory:
// reads run along the source's contiguous index, writes along the batch.
template <typename T, bool FAST_I>
__global__ void batch_to_inner_kernel(const T* __restrict__ src, __nv_bfloat16* __restrict__ dst, int B, int I, int J, int Jp, int Bp,
                                      long long sb, long long si, long long sj) {
  __shared__ float tile[32][33];
  const int b0 = blockIdx.x * 32, f0 = blockIdx.y * 32, slow = blockIdx.z;
  const int F = FAST_I ? I : J;   // extent of the fast index in the source
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int b = b0 + r, f = f0 + threadIdx.x;
    const int i = FAST_I ? f : slow, j = FAST_I ? slow : f;
    tile[r][threadIdx.x] = (b < B && f < F && j < J) ? ld_as_float(src + b * sb + i * si + j * sj) : 0.f;
  }
  __syncthreads();
  const int Fd = FAST_I ? I : Jp;  // extent of the fast index in the destination
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int f = f0 + r, b = b0 + threadIdx.x;
    if (f < Fd && b < Bp) {
      const int i = FAST_I ? f : slow, j = FAST_I ? slow : f;
      dst[((long long)i * Jp + j) * Bp + b] = __float2bfloat16_rn(tile[threadIdx.x][r]);
    }
  }
}

// Same, 64x64 tiles with two elements per access: a warp reads 64 consecutive source elements per row and writes 64 consecutive
// batch entries (128 bytes) per row.  Needs an even fast extent and even strides (so that pairs are aligned).
constexpr int X2_SLOW = 4;   // consecutive values of the slow index one block works through

template <typename T, bool FAST_I>
__global__ void __launch_bounds__(256) batch_to_inner_x2_kernel(const T* __restrict__ src, __nv_bfloat16* __restrict__ dst, int B, int I, int J,
                                                               int Jp, int Bp, long long sb, long long si, long long sj) {
  __shared__ __nv_bfloat16 tile[64][66];
  const int b0 = blockIdx.x * 64, f0 = blockIdx.y * 64;
  const int F = FAST_I ? I : J, n_slow = FAST_I ? Jp : I;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int sl = 0; sl < X2_SLOW; ++sl) {
    const int slow = blockIdx.z * X2_SLOW + sl;
    if (slow >= n_slow) break;           // uniform over the block
    if (sl) __syncthreads();             // the tile is free again
    for (int r = ty; r < 64; r += 8) {
      const int b = b0 + r, f = f0 + 2 * tx;
      const int i = FAST_I ? f : slow, j = FAST_I ? slow : f;
      float v0 = 0.f, v1 = 0.f;
      if (b < B && f < F && j < J) {   // F is even: f + 1 < F as well
        const long long off = b * sb + i * si + j * sj;
        const T* p = src + off;
        if (sizeof(T) == 2) {
          const __nv_bfloat162 q = *reinterpret_cast<const __nv_bfloat162*>(p);
          v0 = __bfloat162float(q.x); v1 = __bfloat162float(q.y);
        } else {
          const float2 q = *reinterpret_cast<const float2*>(p);
          v0 = q.x; v1 = q.y;
        }
      }
      __nv_bfloat162 t2;
      t2.x = __float2bfloat16_rn(v0); t2.y = __float2bfloat16_rn(v1);
      *reinterpret_cast<__nv_bfloat162*>(&tile[r][2 * tx]) = t2;
    }
    __syncthreads();
    const int Fd = FAST_I ? I : Jp;
    for (int r = ty; r < 64; r += 8) {
      const int f = f0 + r, b = b0 + 2 * tx;
      if (f < Fd && b < Bp) {          // Bp is even
        const int i = FAST_I ? f : slow, j = FAST_I ? slow : f;
        __nv_bfloat162 q;
        q.x = tile[2 * tx][r]; q.y = tile[2 * tx + 1][r];
        *reinterpret_cast<__nv_bfloat162*>(dst + ((long long)i * Jp + j) * Bp + b) = q;
      }
    }
  }
}

// Start of the backward pass of a layer with a fused ReLU, on channels-last bf16: the gradient is masked where the layer's output is not
// positive and summed over everything but the channel, in one pass (reads gradient and output, writes the masked gradient: bound by
// memory).  One thread per 8 channels (16-byte accesses) of every step-th row; sums in registers, one shared-memory round per block.
__global__ void relu_mask_colsum_kernel(const uint4* __restrict__ grad, const uint4* __restrict__ act, uint4* __restrict__ masked,
                                        float* __restrict__ colsum, long long R, int c8) {
  extern __shared__ float rm_part[];               // [rows per block][8 * c8]
  const int cg = threadIdx.x % c8, r0 = threadIdx.x / c8, rows = blockDim.x / c8;
  const long long step = (long long)gridDim.x * rows;
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (long long r = (long long)blockIdx.x * rows + r0; r < R; r += step) {
    const uint4 g = __ldg(grad + r * c8 + cg), y = __ldg(act + r * c8 + cg);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, yw[4] = {y.x, y.y, y.z, y.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float y0 = __uint_as_float(yw[i] << 16), y1 = __uint_as_float(yw[i] & 0xFFFF0000u);     // bf16 -> float32, exact
      const uint32_t lo = y0 > 0.f ? gw[i] & 0xFFFFu : 0u, hi = y1 > 0.f ? gw[i] & 0xFFFF0000u : 0u;
      o[i] = lo | hi;
      sum[2 * i] += __uint_as_float(lo << 16); sum[2 * i + 1] += __uint_as_float(hi);
    }
    masked[r * c8 + cg] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (!colsum) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) rm_part[(size_t)r0 * 8 * c8 + cg * 8 + i] = sum[i];
  __syncthreads();
  for (int c = threadIdx.x; c < 8 * c8; c += blockDim.x) {
    float t = 0.f;
    for (int r = 0; r < rows; ++r) t += rm_part[(size_t)r * 8 * c8 + c];
    atomicAdd(colsum + c, t);
  }
}

// Column sums of a row-major [R, C] matrix (C even) into float32 dst[C] (zeroed by the caller's launch order: see the entry
// point).  A warp reads 64 consecutive columns of a row (128 bytes of bf16); rows are strided over the 8 warps of a block
// and over grid.y; partial sums meet in shared memory and leave with one atomic per column and block.
template <typename T>
__global__ void __launch_bounds__(256) column_sum_kernel(const T* __restrict__ src, float* __restrict__ dst, long long R, int C,
                                                        long long rows_per_block) {
  __shared__ float part[8][64];
  const int c = blockIdx.x * 64 + 2 * threadIdx.x;
  const long long r0 = blockIdx.y * rows_per_block, r1 = min(R, r0 + rows_per_block);
  float s0 = 0.f, s1 = 0.f;
  if (c < C) {
    for (long long r = r0 + threadIdx.y; r < r1; r += 8) {
      const T* p = src + r * C + c;
      if (sizeof(T) == 2) {
        const __nv_bfloat162 q = *reinterpret_cast<const __nv_bfloat162*>(p);
        s0 += __bfloat162float(q.x); s1 += __bfloat162float(q.y);
      } else {
        const float2 q = *reinterpret_cast<const float2*>(p);
        s0 += q.x; s1 += q.y;
      }
    }
  }
  part[threadIdx.y][2 * threadIdx.x] = s0;
  part[threadIdx.y][2 * threadIdx.x + 1] = s1;
  __syncthreads();
  if (threadIdx.y == 0) {
    for (int e = 0; e < 2; ++e) {
      float t = 0.f;
      for (int w = 0; w < 8; ++w) t += part[w][2 * threadIdx.x + e];
      if (c + e < C) atomicAdd(dst + c + e, t);
    }
  }
}

}  // namespace

extern "C" int fovi_relu_mask_colsum(const void* grad, const void* act, void* masked, float* colsum, long long R, int C, void* stream) {
  if (R < 0 || C <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (C % 8 || C > 2048) return FOVI_ERR_UNSUPPORTED;
  if (R > 0 && (!grad || !act || !masked)) return FOVI_ERR_INVALID_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(act) | reinterpret_cast<uintptr_t>(masked)) & 15) return FOVI_ERR_UNSUPPORTED;
  if (colsum) FOVI_CUDA(cudaMemsetAsync(colsum, 0, sizeof(float) * (size_t)C, st));
  if (R == 0) return FOVI_OK;
  const int c8 = C / 8, rows = std::max(1, 256 / c8);
  const int grid = (int)std::min<long long>((R + rows - 1) / rows, (long long)fovi::sm_count() * 8);
  relu_mask_colsum_kernel<<<grid, rows * c8, colsum ? sizeof(float) * rows * C : 0, st>>>((const uint4*)grad, (const uint4*)act, (uint4*)masked, colsum, R, c8);
  return fovi::after_launch("relu_mask_colsum_kernel");
}

extern "C" int fovi_column_sum(const void* src, int dtype, long long R, int C, float* dst, void* stream) {
  if (!fovi::valid_dtype(dtype) || R < 0 || C <= 0 || !dst) return FOVI_ERR_INVALID_ARGUMENT;
  if (C % 2 || (R > 0 && (!src || reinterpret_cast<uintptr_t>(src) % (2 * fovi::dtype_size(dtype))))) return FOVI_ERR_UNSUPPORTED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  FOVI_CUDA(cudaMemsetAsync(dst, 0, sizeof(float) * (size_t)C, st));
  if (R == 0) return FOVI_OK;
  const long long rows_per_block = std::max<long long>(256, (R + 4095) / 4096);
  dim3 grid((C + 63) / 64, (unsigned)((R + rows_per_block - 1) / rows_per_block)), block(32, 8);
  if (dtype == FOVI_F32) column_sum_kernel<float><<<grid, block, 0, st>>>((const float*)src, dst, R, C, rows_per_block);
  else column_sum_kernel<__nv_bfloat16><<<grid, block, 0, st>>>((const __nv_bfloat16*)src, dst, R, C, rows_per_block);
  return fovi::after_launch("column_sum_kernel");
}

extern "C" int fovi_batch_to_inner(const void* src, int dtype, int B, int I, int J, long long sb, long long si, long long sj, void* dst,
                                   int Jp, int Bp, void* stream) {
  if (!fovi::valid_dtype(dtype) || B < 0 || I <= 0 || J <= 0 || Jp < J || Bp < B || Bp <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (!src || !dst) return FOVI_ERR_INVALID_ARGUMENT;
  if (si != 1 && sj != 1) return FOVI_ERR_UNSUPPORTED;
  const bool fast_i = si == 1 && !(sj == 1 && J >= I);
  const int fast = fast_i ? I : Jp, slow = fast_i ? Jp : I;
  if (slow > 65535 || (fast + 31) / 32 > 65535) return FOVI_ERR_UNSUPPORTED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int F = fast_i ? I : J;
  const size_t esz = fovi::dtype_size(dtype);
  const bool x2 = F % 2 == 0 && Bp % 2 == 0 && sb % 2 == 0 && (fast_i ? sj : si) % 2 == 0 &&
                  reinterpret_cast<uintptr_t>(src) % (2 * esz) == 0 && reinterpret_cast<uintptr_t>(dst) % 4 == 0 && (fast + 63) / 64 <= 65535;
  if (x2) {
    dim3 grid2((Bp + 63) / 64, (fast + 63) / 64, (slow + X2_SLOW - 1) / X2_SLOW), block2(32, 8);
#define RUN2(T, FI) batch_to_inner_x2_kernel<T, FI><<<grid2, block2, 0, st>>>((const T*)src, (__nv_bfloat16*)dst, B, I, J, Jp, Bp, sb, si, sj)
    if (dtype == FOVI_F32) { if (fast_i) RUN2(float, true); else RUN2(float, false); }
    else { if (fast_i) RUN2(__nv_bfloat16, true); else RUN2(__nv_bfloat16, false); }
#undef RUN2
    return fovi::after_launch("batch_to_inner_x2_kernel");
  }
  dim3 grid((Bp + 31) / 32, (fast + 31) / 32, slow), block(32, 8);
#define RUN(T, FI) batch_to_inner_kernel<T, FI><<<grid, block, 0, st>>>((const T*)src, (__nv_bfloat16*)dst, B, I, J, Jp, Bp, sb, si, sj)
  if (dtype == FOVI_F32) { if (fast_i) RUN(float, true); else RUN(float, false); }
  else { if (fast_i) RUN(__nv_bfloat16, true); else RUN(__nv_bfloat16, false); }
#undef RUN
  return fovi::after_launch("batch_to_inner_kernel");
}
