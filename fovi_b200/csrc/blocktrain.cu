// What stands between the batch norm of a training step and the next convolution, on the kernels' channels-last activations, with the gradients of all
// of it and of the norm itself.  The norm's forward pass is the library's, on [B,C,N] (its sums are part of what a step's numbers are: another order of
// them would move roundings, and with them the masks and maxima of every later layer); everything here is either exact or behind all masks.
//
//   forward    conv result y [B,N,C] -> [B,C,N] for the norm (tile transpose); the norm's result -> relu -> maximum over each output point's neighbours ->
//              [B,n_out,C], through a slab of channels in shared memory: the three passes and two layout changes of the separate modules in one.
//              The list position of each maximum is kept in a byte (255: none, or nothing passes the ReLU).
//   backward   the upstream gradient is taken back through the pooling by GATHER (every input knows the places that read it: no atomics, no zero-filled
//              buffer), masked and summed (dbeta = sum dy, dgamma = sum dy * xhat), then dx = gamma / std * (dy - mean(dy) - xhat * mean(dy * xhat)) is
//              written once, in bf16 and channels last: what the convolution's two gradient contractions read.  Sums in a fixed order.
//
// Bound by the stream of y, h and the gradients through L2 and memory (47 MB each for the 96-channel, 960-point block at 128 rows: transpose 20 us, relu and pool
// 33, gradient sums 32, input gradient 29).  Five blocks of the shipped backbone at 128 rows, device time of a step's kernels with separate modules -> with
// these: 1827 -> 1315 us (the library's norm gradients 320, layout copies 150, packing 55, mask, ReLU and pools 225 -> transposes 50, relu and pool 87, gradients 165).
#include <algorithm>
#include <initializer_list>

#include "knnpool_plan.cuh"

namespace {

struct BlockGeom {
  long long R;                            // rows of y: batch x points
  int C, N;                               // channels, points
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float relu_keep_nan(float v) { return v > 0.f ? v : (v != v ? v : 0.f); }

// src [B][N][C] -> dst [B][C][N], float32, 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) points_to_channels_kernel(const float* __restrict__ src, float* __restrict__ dst, int N, int C) {
  __shared__ float tile[32][33];
  const int n0 = blockIdx.x * 32, c0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const float* s = src + (size_t)blockIdx.z * N * C;
  float* d = dst + (size_t)blockIdx.z * N * C;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = n0 + ty + 8 * i;
    if (n < N && c0 + tx < C) tile[ty + 8 * i][tx] = __ldg(s + (size_t)n * C + c0 + tx);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = c0 + ty + 8 * i;
    if (c < C && n0 + tx < N) d[(size_t)c * N + n0 + tx] = tile[tx][ty + 8 * i];
  }
}

// One CTA: one sample x CH channels, staged in shared memory with an odd pitch (lanes of one warp hold different channels of the same point: no bank
// conflicts).  Without a pool the output points are the inputs (K = 0).  CH: as many channels as leave three CTAs' slabs room on an SM.  gridDim.z CTAs share the
// output points of a slab where samples and channels do not fill the chip (one sample of 5602 points, 96 channels, 81 neighbours: 12 CTAs, the training step
// 580 us, with the separate modules 511; with twelve CTAs a slab 460).
constexpr int SLAB_THREADS = 512;

template <int CH>
__global__ void __launch_bounds__(SLAB_THREADS) relu_pool_kernel(const float* __restrict__ h, const int* __restrict__ idx, int n_out, int K, int relu,
                                                                 float* __restrict__ out, unsigned char* __restrict__ arg, const BlockGeom q) {
  extern __shared__ float slab[];
  const int pitch = q.N | 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = blockIdx.y * CH;
  const size_t b = blockIdx.x;
  for (int r = warp; r < CH && c0 + r < q.C; r += SLAB_THREADS / 32) {
    const float* src = h + (b * q.C + c0 + r) * q.N;
#pragma unroll 8
    for (int n = lane; n < q.N; n += 32) slab[r * pitch + n] = __ldg(src + n);
  }
  __syncthreads();
  const int cl = lane % CH, c = c0 + cl;
  if (c >= q.C) return;
  const float* mine = slab + cl * pitch;
  constexpr int PER_PASS = SLAB_THREADS / CH;
  for (int n = blockIdx.z * PER_PASS + threadIdx.x / CH; n < n_out; n += PER_PASS * gridDim.z) {
    const size_t at = (b * n_out + n) * q.C + c;
    if (K == 0) {
      const float v = mine[n];
      out[at] = relu ? relu_keep_nan(v) : v;
      continue;
    }
    float best = -INFINITY;
    int who = 255;
#pragma unroll 3
    for (int k = 0; k < K; ++k) {
      const int j = __ldg(idx + (size_t)n * K + k);
      float v = mine[min(j, q.N - 1)];
      if (relu) v = relu_keep_nan(v);
      if (j < q.N && v == v && (who == 255 || v > best)) { best = v; who = k; }      // pads and NaN are ignored, the first maximum wins
    }
    out[at] = best;
    arg[at] = (unsigned char)(relu && !(best > 0.f) ? 255 : who);                     // what the ReLU stops hands nothing back
  }
}

// The channel's normalisation: (x - mean) / std = xhat.
struct Chan4 {
  float m[4], r[4], g[4];
  __device__ __forceinline__ Chan4(const float* mean, const float* rstd, const float* gamma, int c) {
    const float4 a0 = ld4(mean + c), a1 = ld4(rstd + c), a2 = ld4(gamma + c);
    m[0] = a0.x; m[1] = a0.y; m[2] = a0.z; m[3] = a0.w;
    r[0] = a1.x; r[1] = a1.y; r[2] = a1.z; r[3] = a1.w;
    g[0] = a2.x; g[1] = a2.y; g[2] = a2.z; g[3] = a2.w;
  }
};

// What the places that read input m of sample b hand back, channels cg * 4 ..: two places' reads are in flight at a time.
struct PoolGrad { const float* g; const uchar4* arg; const int* t_start; const int* t_entry; int n_out; };

__device__ __forceinline__ void pool_grad(const PoolGrad& a, uint32_t b, uint32_t m, uint32_t c4, uint32_t cg, float (&up)[4]) {
  const int e0 = __ldg(a.t_start + m), e1 = __ldg(a.t_start + m + 1);
  const long long row0 = (long long)b * a.n_out;
  for (int i = e0; i < e1; i += 2) {
    const int p0 = __ldg(a.t_entry + i), p1 = i + 1 < e1 ? __ldg(a.t_entry + i + 1) : p0;
    const long long a0 = (row0 + (p0 >> 8)) * c4 + cg, a1 = (row0 + (p1 >> 8)) * c4 + cg;
    const uchar4 k0 = __ldg(a.arg + a0), k1 = __ldg(a.arg + a1);
    const float4 g0 = __ldg(reinterpret_cast<const float4*>(a.g) + a0), g1 = __ldg(reinterpret_cast<const float4*>(a.g) + a1);
    const int q0 = p0 & 255, q1 = i + 1 < e1 ? p1 & 255 : 256;
    if (k0.x == q0) up[0] += g0.x;
    if (k0.y == q0) up[1] += g0.y;
    if (k0.z == q0) up[2] += g0.z;
    if (k0.w == q0) up[3] += g0.w;
    if (k1.x == q1) up[0] += g1.x;
    if (k1.y == q1) up[1] += g1.y;
    if (k1.z == q1) up[2] += g1.z;
    if (k1.w == q1) up[3] += g1.w;
  }
}

// Gradient at the normalised activations of a row (before gamma), channels cg * 4 .., and their normalised values.  act: the ReLU's result [B,N,C] where it is
// not followed by a pool (whose bytes hold the mask), else null.
struct RowGrad {
  float dy[4], xh[4];
  template <bool POOL>
  __device__ __forceinline__ void read(const float* y, const PoolGrad& a, const Chan4& ch, const float* act, uint32_t r, uint32_t N, uint32_t c4, uint32_t cg) {
    const size_t at = (size_t)r * c4 + cg;
    const float4 x = __ldg(reinterpret_cast<const float4*>(y) + at);
    float up[4] = {0.f, 0.f, 0.f, 0.f};
    if (POOL) {
      const uint32_t b = r / N;
      pool_grad(a, b, r - b * N, c4, cg, up);
    } else {
      const float4 u = __ldg(reinterpret_cast<const float4*>(a.g) + at);
      up[0] = u.x; up[1] = u.y; up[2] = u.z; up[3] = u.w;
      if (act) {
        const float4 o = __ldg(reinterpret_cast<const float4*>(act) + at);
        up[0] = o.x <= 0.f ? 0.f : up[0]; up[1] = o.y <= 0.f ? 0.f : up[1]; up[2] = o.z <= 0.f ? 0.f : up[2]; up[3] = o.w <= 0.f ? 0.f : up[3];
      }
    }
    const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { xh[i] = (xv[i] - ch.m[i]) * ch.r[i]; dy[i] = up[i]; }
  }
};

// Both backward kernels: a thread keeps its four channels (CTA: `quads` channel quads x `rows` rows) and walks the rows.  They gather the pooled gradient anew
// rather than pass it through memory (47 MB each way for the largest block).
struct QuadTile { int quads, rows; };

template <bool POOL>
__global__ void __launch_bounds__(256, 4) bn_grad_sums_kernel(const float* __restrict__ y, const float* __restrict__ mean, const float* __restrict__ rstd,
                                                              const float* __restrict__ gamma, const PoolGrad a, const float* __restrict__ act,
                                                              float2* __restrict__ part, const BlockGeom q, const QuadTile t) {
  extern __shared__ float4 bn_sm[];                               // [2][rows][quads]
  const uint32_t c4 = (uint32_t)q.C / 4u;
  const int ql = threadIdx.x % t.quads, r0 = threadIdx.x / t.quads;
  const uint32_t cg = blockIdx.y * t.quads + ql;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
  if (cg < c4) {
    const Chan4 ch(mean, rstd, gamma, (int)cg * 4);
    const uint32_t step = gridDim.x * t.rows, R = (uint32_t)q.R;
#pragma unroll POOL ? 1 : 4
    for (uint32_t r = blockIdx.x * t.rows + r0; r < R; r += step) {
      RowGrad w;
      w.read<POOL>(y, a, ch, act, r, (uint32_t)q.N, c4, cg);
#pragma unroll
      for (int i = 0; i < 4; ++i) { s[i] += w.dy[i]; u[i] = fmaf(w.dy[i], w.xh[i], u[i]); }
    }
  }
  float4* s1 = bn_sm + r0 * t.quads + ql;
  float4* s2 = s1 + t.rows * t.quads;
  *s1 = make_float4(s[0], s[1], s[2], s[3]); *s2 = make_float4(u[0], u[1], u[2], u[3]);
  __syncthreads();
  if (r0 || cg >= c4) return;
  for (int w = 1; w < t.rows; ++w) {
    const float4 v = s1[w * t.quads], x = s2[w * t.quads];
    s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
    u[0] += x.x; u[1] += x.y; u[2] += x.z; u[3] += x.w;
  }
  float4* d = reinterpret_cast<float4*>(part + (size_t)blockIdx.x * q.C + cg * 4);
  d[0] = make_float4(s[0], u[0], s[1], u[1]);
  d[1] = make_float4(s[2], u[2], s[3], u[3]);
}

// Eight channels per CTA, 64 threads share a channel's partial sums; added in double, in a fixed order.
constexpr int FIN_CH = 8, FIN_T = 64;

// Sum over the FIN_T threads of a channel (threadIdx.x = thread * FIN_CH + channel), valid in its first thread.
__device__ __forceinline__ double finish_sum(double v, double (&sm)[FIN_T * FIN_CH / 32][FIN_CH]) {
  v += __shfl_down_sync(0xffffffffu, v, 16);
  v += __shfl_down_sync(0xffffffffu, v, 8);
  if ((threadIdx.x & 31) < FIN_CH) sm[threadIdx.x >> 5][threadIdx.x & 31] = v;
  __syncthreads();
  if (threadIdx.x < FIN_CH)
    for (int w = 1; w < FIN_T * FIN_CH / 32; ++w) v += sm[w][threadIdx.x];
  __syncthreads();
  return v;
}

__global__ void __launch_bounds__(FIN_T * FIN_CH) bn_grad_finish_kernel(const float2* __restrict__ part, int chunks, int C, float* __restrict__ dgamma,
                                                                        float* __restrict__ dbeta) {
  __shared__ double sm[FIN_T * FIN_CH / 32][FIN_CH];
  const int j = threadIdx.x / FIN_CH, c = blockIdx.x * FIN_CH + threadIdx.x % FIN_CH;
  double s = 0., t = 0.;
  if (c < C) {
#pragma unroll 4
    for (int p = j; p < chunks; p += FIN_T) {
      const float2 v = __ldg(part + (long long)p * C + c);
      s += (double)v.x; t += (double)v.y;
    }
  }
  s = finish_sum(s, sm); t = finish_sum(t, sm);
  if (j || c >= C) return;
  dbeta[c] = (float)s;
  dgamma[c] = (float)t;
}

template <bool POOL>
__global__ void __launch_bounds__(256, 4) bn_grad_input_kernel(const float* __restrict__ y, const float* __restrict__ mean, const float* __restrict__ rstd,
                                                               const float* __restrict__ gamma, const PoolGrad a, const float* __restrict__ act,
                                                               const float* __restrict__ dgamma, const float* __restrict__ dbeta,
                                                               __nv_bfloat16* __restrict__ dx, const BlockGeom q, const QuadTile t) {
  const uint32_t c4 = (uint32_t)q.C / 4u;
  const int ql = threadIdx.x % t.quads, r0 = threadIdx.x / t.quads;
  const uint32_t cg = blockIdx.y * t.quads + ql;
  if (cg >= c4) return;
  const int c = (int)cg * 4;
  const Chan4 ch(mean, rstd, gamma, c);
  const float inv = 1.f / (float)q.R;
  const float4 sg = ld4(dgamma + c), sb = ld4(dbeta + c);
  const float mg[4] = {sg.x * inv, sg.y * inv, sg.z * inv, sg.w * inv}, mb[4] = {sb.x * inv, sb.y * inv, sb.z * inv, sb.w * inv};
  const uint32_t step = gridDim.x * t.rows, R = (uint32_t)q.R;
#pragma unroll POOL ? 1 : 4
  for (uint32_t r = blockIdx.x * t.rows + r0; r < R; r += step) {
    RowGrad w;
    w.read<POOL>(y, a, ch, act, r, (uint32_t)q.N, c4, cg);
    float d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] = ch.g[i] * ch.r[i] * (w.dy[i] - mb[i] - w.xh[i] * mg[i]);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(d[0], d[1]), hi = __floats2bfloat162_rn(d[2], d[3]);
    uint2 o;
    o.x = *reinterpret_cast<const uint32_t*>(&lo); o.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(dx + ((size_t)r * c4 + cg) * 4) = o;
  }
}

// CTAs of up to 256 threads: all of a row's channel quads when that many fit, else equal tiles of them.
QuadTile quad_tile(int C, int& tiles) {
  const int c4 = C / 4;
  tiles = (c4 + 255) / 256;
  const int quads = (c4 + tiles - 1) / tiles;
  return {quads, std::max(1, 256 / quads)};
}
int sums_ctas(long long R, int C) {      // four per SM, or as many as give every thread two rows
  int tiles;
  const QuadTile t = quad_tile(C, tiles);
  return (int)std::max<long long>(1, std::min<long long>((R + 2 * t.rows - 1) / (2 * t.rows), 4ll * fovi::sm_count() / tiles));
}
bool misaligned(std::initializer_list<const void*> ps) {
  uintptr_t u = 0;
  for (const void* p : ps) u |= reinterpret_cast<uintptr_t>(p);
  return (u & 15) != 0;
}

// Channels per slab of the forward kernel, 0: not even eight fit.
int slab_channels(int N) {
  for (int ch = 32; ch >= 8; ch /= 2)
    if ((long long)ch * (N | 1) * 4 <= 72 * 1024) return ch;
  return 8ll * (N | 1) * 4 <= 200 * 1024 ? 8 : 0;
}

}  // namespace

extern "C" int fovi_points_to_channels(const float* src, float* dst, int B, int N, int C, void* stream) {
  if (B < 0 || N <= 0 || C <= 0 || (B > 0 && (!src || !dst))) return FOVI_ERR_INVALID_ARGUMENT;
  if (B > 65535 || (C + 31) / 32 > 65535) return FOVI_ERR_UNSUPPORTED;
  if (B == 0) return FOVI_OK;
  points_to_channels_kernel<<<dim3((N + 31) / 32, (C + 31) / 32, B), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(src, dst, N, C);
  return fovi::after_launch("points_to_channels_kernel");
}

extern "C" int fovi_relu_pool_supported(int N, const fovi_knnpool_plan* pool) { return N > 0 && slab_channels(N) > 0 && (!pool || pool->t_start) ? 1 : 0; }

extern "C" int fovi_relu_pool_forward(const float* h, int B, int N, int C, int relu, const fovi_knnpool_plan* pool, float* out, unsigned char* arg, void* stream) {
  if (B < 0 || N <= 0 || C <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  const int ch = slab_channels(N);
  if (!ch || (C + ch - 1) / ch > 65535 || (pool && (pool->n_in != N || !pool->t_start))) return FOVI_ERR_UNSUPPORTED;
  if (B == 0) return FOVI_OK;
  if (!h || !out || (pool && !arg)) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  BlockGeom q;
  q.R = (long long)B * N; q.C = C; q.N = N;
  const int slabs = (C + ch - 1) / ch, passes = ((pool ? pool->n_out : N) * ch + SLAB_THREADS - 1) / SLAB_THREADS;
  const dim3 grid(B, slabs, (unsigned)std::max<long long>(1, std::min<long long>(passes, fovi::sm_count() / ((long long)B * slabs))));
  const size_t smem = (size_t)ch * (N | 1) * sizeof(float);
  auto k = ch == 32 ? relu_pool_kernel<32> : ch == 16 ? relu_pool_kernel<16> : relu_pool_kernel<8>;
  if (smem > 48 * 1024) FOVI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k<<<grid, SLAB_THREADS, smem, st>>>(h, pool ? pool->idx : nullptr, pool ? pool->n_out : N, pool ? pool->K : 0, relu, out, arg, q);
  return fovi::after_launch("relu_pool_kernel");
}

extern "C" int64_t fovi_norm_block_workspace_bytes(int B, int N, int C) {
  return B > 0 && N > 0 && C >= 4 ? (int64_t)sums_ctas((long long)B * N, C) * C * (int64_t)sizeof(float2) : 0;
}

extern "C" int fovi_norm_block_backward(const float* y, int B, int N, int C, const float* mean, const float* rstd, const float* gamma, const float* act,
                                        const fovi_knnpool_plan* pool, const unsigned char* arg, const float* g, float* dgamma, float* dbeta, void* dx,
                                        void* work, int64_t work_bytes, void* stream) {
  if (B <= 0 || N <= 0 || C <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (C % 4 || (pool && (pool->n_in != N || !pool->t_start))) return FOVI_ERR_UNSUPPORTED;
  const long long limit = (1ll << 31) / (C / 4);            // quads of channels are counted in 32 bits
  if ((long long)B * N >= limit || (pool && (long long)B * pool->n_out >= limit)) return FOVI_ERR_UNSUPPORTED;
  if (!y || !mean || !rstd || !gamma || !g || !dgamma || !dbeta || !dx || !work || (pool && !arg)) return FOVI_ERR_INVALID_ARGUMENT;
  if (misaligned({y, mean, rstd, gamma, act, arg, g, dgamma, dbeta, dx, work})) return FOVI_ERR_ALIGNMENT;
  if (work_bytes < fovi_norm_block_workspace_bytes(B, N, C)) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  BlockGeom q;
  q.R = (long long)B * N; q.C = C; q.N = N;
  const PoolGrad a = {g, reinterpret_cast<const uchar4*>(arg), pool ? pool->t_start : nullptr, pool ? pool->t_entry : nullptr, pool ? pool->n_out : N};
  int tiles;
  const QuadTile t = quad_tile(C, tiles);
  const int ctas = sums_ctas(q.R, C), threads = t.quads * t.rows;
  const size_t smem = 2 * sizeof(float4) * threads;
  float2* part = static_cast<float2*>(work);
  if (pool) bn_grad_sums_kernel<true><<<dim3(ctas, tiles), threads, smem, st>>>(y, mean, rstd, gamma, a, act, part, q, t);
  else bn_grad_sums_kernel<false><<<dim3(ctas, tiles), threads, smem, st>>>(y, mean, rstd, gamma, a, act, part, q, t);
  int rc = fovi::after_launch("bn_grad_sums_kernel");
  if (rc) return rc;
  bn_grad_finish_kernel<<<(C + FIN_CH - 1) / FIN_CH, FIN_T * FIN_CH, 0, st>>>(part, ctas, C, dgamma, dbeta);
  rc = fovi::after_launch("bn_grad_finish_kernel");
  if (rc) return rc;
  const dim3 grid((unsigned)std::min<long long>((q.R + t.rows - 1) / t.rows, std::max(1, 8 * fovi::sm_count() / tiles)), tiles);
  if (pool) bn_grad_input_kernel<true><<<grid, threads, 0, st>>>(y, mean, rstd, gamma, a, act, dgamma, dbeta, static_cast<__nv_bfloat16*>(dx), q, t);
  else bn_grad_input_kernel<false><<<grid, threads, 0, st>>>(y, mean, rstd, gamma, a, act, dgamma, dbeta, static_cast<__nv_bfloat16*>(dx), q, t);
  return fovi::after_launch("bn_grad_input_kernel");
}
