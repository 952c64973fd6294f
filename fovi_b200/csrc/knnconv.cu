// KNNConv: plan construction, operand packing and the exact float32 (CUDA-core) forward.
#include <algorithm>
#include <vector>

#include "knnconv_plan.cuh"

namespace {

// Changes between the reference's filter layout, W [c_out][c_in][V] (taps innermost), and tap-major slabs: transposes of [r][v] planes, one per
// `outer` index, where r is the slabs' innermost index (an input channel, or an output channel for the transposed layer and for gradients).
// What bounds them is memory, so a 64 x 64 tile of (r, v) goes through shared memory and both sides move in whole runs: taps on the filter's side
// (its rows are V long), channels on the slabs' side.  384 -> 256 channels, 36 taps (14 MB in, 7 out): 22 -> 11 us against one thread per
// slab element, whose reads were V apart.
//   to slabs   dst[v * d_v + outer * d_o + r] = r < R ? W[outer * w_o + r * w_r + v] : 0   for r < Rp
//   to filter  dst[outer * w_o + r * w_r + v] = src[v * d_v + outer * d_o + r]             for r < R
constexpr int TAP_T = 64;

template <typename TS, typename TD, bool TO_SLABS>
__global__ void __launch_bounds__(256) tap_transpose_kernel(const TS* __restrict__ src, TD* __restrict__ dst, int R, int Rp, int V, long long w_o,
                                                            long long w_r, long long d_v, long long d_o) {
  __shared__ float tile[TAP_T][TAP_T + 1];
  const int r0 = blockIdx.y * TAP_T, v0 = blockIdx.z * TAP_T;
  const long long outer = blockIdx.x;
  const int nv = min(TAP_T, V - v0), nr = min(TAP_T, (TO_SLABS ? Rp : R) - r0);
  const uint32_t inv = (0xFFFFFFFFu / (uint32_t)nv) + 1u;      // i / nv == umulhi(i, inv) for the i < 4096 here (nv == 1: inv wraps to 0)
  auto row_of = [&](int i) { return nv == 1 ? i : (int)__umulhi((uint32_t)i, inv); };
  if (TO_SLABS) {
#pragma unroll 4
    for (int i = threadIdx.x; i < nr * nv; i += 256) {
      const int r = row_of(i), v = i - r * nv;
      tile[r][v] = r0 + r < R ? ld_as_float(src + outer * w_o + (r0 + r) * w_r + v0 + v) : 0.f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nv * TAP_T; i += 256) {
      const int v = i / TAP_T, r = i % TAP_T;
      if (r < nr) dst[(v0 + v) * d_v + outer * d_o + r0 + r] = from_float<TD>(tile[r][v]);
    }
  } else {
    for (int i = threadIdx.x; i < nv * TAP_T; i += 256) {
      const int v = i / TAP_T, r = i % TAP_T;
      if (r < nr) tile[r][v] = ld_as_float(src + (v0 + v) * d_v + outer * d_o + r0 + r);
    }
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < nr * nv; i += 256) {
      const int r = row_of(i), v = i - r * nv;
      dst[outer * w_o + (r0 + r) * w_r + v0 + v] = from_float<TD>(tile[r][v]);
    }
  }
}

template <bool TO_SLABS>
int tap_transpose(const void* src, int s_dtype, void* dst, int d_dtype, int n_outer, int R, int Rp, int V, long long w_o, long long w_r, long long d_v,
                  long long d_o, cudaStream_t st) {
  const dim3 grid(n_outer, (Rp + TAP_T - 1) / TAP_T, (V + TAP_T - 1) / TAP_T);
  if (grid.y > 65535 || grid.z > 65535) return FOVI_ERR_UNSUPPORTED;
#define GO(TS, TD) tap_transpose_kernel<TS, TD, TO_SLABS><<<grid, 256, 0, st>>>((const TS*)src, (TD*)dst, R, Rp, V, w_o, w_r, d_v, d_o)
  if (s_dtype == FOVI_F32) { if (d_dtype == FOVI_F32) GO(float, float); else GO(float, __nv_bfloat16); }
  else { if (d_dtype == FOVI_F32) GO(__nv_bfloat16, float); else GO(__nv_bfloat16, __nv_bfloat16); }
#undef GO
  return fovi::after_launch("tap_transpose_kernel");
}

// Pair mode: W [c_out, c_in*V] -> per-output-point slabs [n_out, c_out/ct, sp, ct, 8] (so the eight
// slots of one stage of one c_out tile are contiguous); element (h, c) of a slot row is the weight
// of channel c (< 4) for the even (h = 0) or odd (h = 1) point of the pair.
template <typename TW>
__global__ void pack_weights_pairs_kernel(const TW* __restrict__ W, __nv_bfloat16* __restrict__ dst,
                                          const uint16_t* __restrict__ pair_tap, int n_out, int sp, int V, int c_out, int c_in, int ct) {
  const long long total = (long long)n_out * sp * c_out * 8;
  const int n_ct = c_out / ct;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(i & 7);
    long long r = i >> 3;
    const int oc = (int)(r % ct); r /= ct;
    const int sl = (int)(r % sp); r /= sp;
    const int tile = (int)(r % n_ct);
    const long long n = r / n_ct;
    const int o = tile * ct + oc;
    const long long slot = n * sp + sl;
    const int h = e >> 2, c = e & 3;
    const int t = pair_tap[slot * 2 + h];
    const float w = (c < c_in && t != 0xFFFF) ? ld_as_float(W + ((long long)o * c_in + c) * V + t) : 0.f;
    dst[i] = __float2bfloat16_rn(w);
  }
}

// Packed weights of a GROUPED pair-mode plan: the plan's "output points" are groups of G consecutive output points of the
// layer and its "output channels" are the G members' channels side by side (c_out = G * co), so the group's one
// neighbour list is the union of its members' lists.  The plan was created with tap[g][k] = k, i.e. pair_tap holds each
// slot's position in the union list; member_tap[g][k][j] is the filter tap member j gives that neighbour (0xFFFF: it
// is not a neighbour of member j, the weight is zero).  Same destination layout as pack_weights_pairs_kernel.
template <typename TW>
__global__ void pack_weights_grouped_kernel(const TW* __restrict__ W, __nv_bfloat16* __restrict__ dst,
                                            const uint16_t* __restrict__ pair_tap, const uint16_t* __restrict__ member_tap, int n_groups,
                                            int sp, int K, int G, int V, int co, int c_in, int ct) {
  // (any V; filters of up to GROUPED_TAPS taps take the kernel below)
  // one thread per 16-byte row of the destination (a pair slot of one output channel: 2 points x 4 channels), so the
  // index arithmetic and the two table look-ups are paid once per eight values and the store is a whole 16-byte piece
  const int c_out = G * co;
  const long long total = (long long)n_groups * sp * c_out;
  const int n_ct = c_out / ct;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    long long r = i;
    const int oc = (int)(r % ct); r /= ct;
    const int sl = (int)(r % sp); r /= sp;
    const int tile = (int)(r % n_ct);
    const long long g = r / n_ct;
    const int op = tile * ct + oc;          // channel of the group: member j, its channel o
    const int j = op / co, o = op - j * co;
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = pair_tap[(g * sp + sl) * 2 + h];
      int t = 0xFFFF;
      if (k != 0xFFFF) t = member_tap[(g * K + k) * G + j];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        v[h * 4 + c] = __float2bfloat16_rn((c < c_in && t != 0xFFFF) ? ld_as_float(W + ((long long)o * c_in + c) * V + t) : 0.f);
    }
    *reinterpret_cast<uint4*>(dst + i * 8) = *reinterpret_cast<const uint4*>(v);
  }
}

// Same result for filters whose 32-channel slice fits shared memory.  The rows are two 8-byte pieces of the filter each, and what bounds the kernel
// above is fetching them: six 4-byte loads a thread, V * c_in apart between neighbouring lanes.  Here a CTA holds 32 channels of one member in shared
// memory, tap-major and in bf16 (lanes read consecutive 8-byte pieces), and writes their rows for its share of the groups: a warp looks up the taps of
// 32 slots at a time, a lane per slot, and stores 32 rows of 16 bytes per slot.  3 -> 64 channels, 484 taps, 341 groups of 3 (92 MB): 80 -> 39 us.
constexpr int GROUPED_TAPS = 800;      // 211 KB

template <typename TW>
__global__ void __launch_bounds__(512) pack_weights_grouped_smem_kernel(const TW* __restrict__ W, __nv_bfloat16* __restrict__ dst,
                                                                        const uint16_t* __restrict__ pair_tap, const uint16_t* __restrict__ member_tap,
                                                                        int n_groups, int sp, int K, int G, int V, int co, int c_in, int ct) {
  extern __shared__ __align__(16) unsigned char pg_smem[];
  __nv_bfloat16* ws = reinterpret_cast<__nv_bfloat16*>(pg_smem);          // [V][33][4]
  const int o0 = blockIdx.x * 32, j = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int no = min(32, co - o0);
  for (int i = threadIdx.x; i < V * 33 * 2; i += blockDim.x) reinterpret_cast<uint32_t*>(pg_smem)[i] = 0u;
  __syncthreads();
  for (int r = warp; r < no * c_in; r += blockDim.x >> 5) {               // a warp per filter row
    const int o = r / c_in, c = r - o * c_in;
    const TW* row = W + ((long long)(o0 + o) * c_in + c) * V;
#pragma unroll 8
    for (int t = lane; t < V; t += 32) ws[((size_t)t * 33 + o) * 4 + c] = __float2bfloat16_rn(ld_as_float(row + t));
  }
  __syncthreads();
  const int op = j * co + o0 + lane, tile = op / ct, oc = op - tile * ct, n_ct = G * co / ct;
  const int chunks = (sp + 31) / 32;
  const long long units = (long long)n_groups * chunks;
  const int n_warps = (blockDim.x >> 5) * gridDim.z;
  for (long long u = (long long)blockIdx.z * (blockDim.x >> 5) + warp; u < units; u += n_warps) {
    const long long g = u / chunks;
    const int s0 = (int)(u - g * chunks) * 32, m = min(32, sp - s0);
    uint32_t taps = 0xFFFFFFFFu;                                            // this lane's slot: the two halves' taps
    if (lane < m) {
      const uint32_t ks = *reinterpret_cast<const uint32_t*>(pair_tap + (g * sp + s0 + lane) * 2);
      const uint32_t k0 = ks & 0xFFFFu, k1 = ks >> 16;
      const uint32_t t0 = k0 != 0xFFFFu ? __ldg(member_tap + (g * K + k0) * G + j) : 0xFFFFu;
      const uint32_t t1 = k1 != 0xFFFFu ? __ldg(member_tap + (g * K + k1) * G + j) : 0xFFFFu;
      taps = t0 | (t1 << 16);
    }
    uint4* out = reinterpret_cast<uint4*>(dst) + ((g * n_ct + tile) * sp + s0) * ct + oc;
#pragma unroll 4
    for (int s = 0; s < m; ++s) {
      const uint32_t tt = __shfl_sync(0xffffffffu, taps, s), t0 = tt & 0xFFFFu, t1 = tt >> 16;
      uint2 a = make_uint2(0u, 0u), b = make_uint2(0u, 0u);
      if (t0 != 0xFFFFu) a = *reinterpret_cast<const uint2*>(ws + ((size_t)t0 * 33 + lane) * 4);
      if (t1 != 0xFFFFu) b = *reinterpret_cast<const uint2*>(ws + ((size_t)t1 * 33 + lane) * 4);
      if (lane < no) out[(size_t)s * ct] = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
}

// X [B,C,N] -> [ceil(B/128), ceil(N/2), 128, 2, 4] bf16 (pair layout), one thread per (pair, row); the last tile's rows past the batch are zeros.
template <typename TX>
__global__ void pack_points_pairs_kernel(const TX* __restrict__ x, __nv_bfloat16* __restrict__ dst, int B, int C, int N) {
  const int n_pairs = (N + 1) / 2;
  const long long total = (long long)n_pairs * ((B + 127) / 128 * 128);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int pr = (int)(i % n_pairs), b = (int)(i / n_pairs);
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int n = 2 * pr + h;
        v[h * 4 + c] = __float2bfloat16_rn((c < C && n < N && b < B) ? ld_as_float(x + ((long long)b * C + c) * N + n) : 0.f);
      }
    *reinterpret_cast<uint4*>(dst + (((long long)(b >> 7) * n_pairs + pr) * 128 + (b & 127)) * 8) = *reinterpret_cast<const uint4*>(v);
  }
}

// X [B,C,N] -> [B,N,cp] bf16, transposing 32x32 tiles through shared memory.
template <typename TX>
__global__ void pack_points_kernel(const TX* __restrict__ x, __nv_bfloat16* __restrict__ dst, int C, int N, int cp) {
  __shared__ float tile[32][33];
  const int b = blockIdx.z;
  const int n0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const TX* xb = x + (long long)b * C * N;
  __nv_bfloat16* db = dst + (long long)b * N * cp;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int c = c0 + r, n = n0 + threadIdx.x;
    tile[r][threadIdx.x] = (c < C && n < N) ? ld_as_float(xb + (long long)c * N + n) : 0.f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int n = n0 + r, c = c0 + threadIdx.x;
    if (n < N && c < cp) db[(long long)n * cp + c] = __float2bfloat16_rn(tile[threadIdx.x][r]);
  }
}

// Exact float32 forward of a layer with at most 4 input channels (fed by the sensor).
//
// The contraction is short (K * c_in = 27..147 products) and every output point has its own taps, so what bounds a plain
// kernel is not arithmetic (8 us of FMAs at 8 images, 3 -> 64 channels, 49 neighbours, 3976 points) but two loads per FMA and
// 4-byte stores a point apart.  Here one warp owns an output point: a lane holds NO output channels x BT images in registers, the
// neighbours' inputs are gathered once per point into shared memory (two lanes per neighbour, half of the images each; read back as broadcasts), and the
// filter is held in shared memory tap-major / channel-minor, so that a tap costs NO conflict-free loads for BT * NO FMAs.
// A CTA's eight points leave through shared memory as runs of eight points (one 32-byte sector) per channel.
// Persistent CTAs, so that the filter is staged once.  One accumulator per output, neighbours in list order, channels inside: the
// sums are those of the general kernel below, bit for bit.
// CTAs per SM (register limit): up to 64 registers hold the accumulators of 32 or 64 channels, so four CTAs hide the gathers of each other's passes;
// 96 channels x 8 images take up to 127 registers, two CTAs.  Serves tiles of one or two images, filters that do not fit shared memory, and grids too small for
// the kernel below (see quad_pays).
constexpr int F32_POINTS = 8;     // output points (warps) per CTA
constexpr int F32_NB = 16;        // neighbours staged per pass: two lanes each

__host__ __device__ constexpr int f32_union_floats(int C, int BT, int OT) {
  const int in = F32_POINTS * F32_NB * C * BT, out = BT * OT * (F32_POINTS + 1);
  return ((in > out ? in : out) + 3) / 4 * 4;
}

template <typename TX, int BT, int NO, int CT, bool WS>
__global__ void __launch_bounds__(F32_POINTS * 32, NO == 3 ? 2 : 4) knnconv_f32_few_kernel(const TX* __restrict__ X, const float* __restrict__ Wt,
                                                                          const float* __restrict__ bias, float* __restrict__ Y,
                                                                          const int* __restrict__ nbr_idx, const uint16_t* __restrict__ nbr_tap,
                                                                          const int* __restrict__ nbr_cnt, int kp, int B, int n_in, int n_out,
                                                                          int c_in, int c_out, int cp, int V, int relu, int x_bnc, int y_bnc,
                                                                          int n_ot, int n_bt, int total) {
  extern __shared__ __align__(16) float f32_smem[];
  constexpr int OT = NO * 32;
  const int C = CT ? CT : c_in;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = f32_smem + warp * (F32_NB * C * BT);                        // [neighbour][channel][BT images]
  float* ys = f32_smem;                                                   // [BT][OT][F32_POINTS], rows of F32_POINTS + 1: over the inputs, once used
  float* ws = f32_smem + f32_union_floats(C, BT, OT);                     // [V][C][OT] (WS)
  int staged = -1;
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    const int ot = item % n_ot, t = item / n_ot;                          // grid is a multiple of n_ot: a CTA keeps its channel tile
    const int bt = t % n_bt, n0 = (t / n_bt) * F32_POINTS;
    const int o0 = ot * OT, b0 = bt * BT, nb = min(BT, B - b0), n = n0 + warp;
    if (WS && staged != ot) {
      __syncthreads();
      // a warp per (tap, 32 channels): consecutive lanes read consecutive rows of the tap's slab
#pragma unroll 4
      for (int r = warp; r < V * NO; r += F32_POINTS) {
        const int v = r / NO, o = (r - v * NO) * 32 + lane;
        const float* src = Wt + ((long long)v * c_out + o0 + o) * cp;
#pragma unroll
        for (int c = 0; c < (CT ? CT : 4); ++c)
          if (CT || c < C) ws[(v * C + c) * OT + o] = o0 + o < c_out ? __ldg(src + c) : 0.f;
      }
      staged = ot;
      __syncthreads();
    }
    float acc[NO][BT];
#pragma unroll
    for (int i = 0; i < NO; ++i)
#pragma unroll
      for (int b = 0; b < BT; ++b) acc[i][b] = 0.f;
    const int cnt = n < n_out ? __ldg(nbr_cnt + n) : 0;
    for (int k0 = 0; k0 < cnt; k0 += F32_NB) {
      const int m = min(F32_NB, cnt - k0);
      int tap = 0;
      __syncwarp();      // the previous pass has been read
      const int nk = lane & (F32_NB - 1), bh = (lane / F32_NB) * (BT / 2);      // this lane's neighbour and its half of the images
      if (nk < m) {
        const int j = __ldg(nbr_idx + (long long)n * kp + k0 + nk);
        tap = __ldg(nbr_tap + (long long)n * kp + k0 + nk);
#pragma unroll
        for (int c = 0; c < (CT ? CT : 4); ++c) {
          if (CT == 0 && c >= C) break;
          float v[BT / 2];
#pragma unroll
          for (int b = 0; b < BT / 2; ++b) {
            const long long bb = b0 + bh + b;
            v[b] = bh + b < nb ? ld_as_float(x_bnc ? X + (bb * n_in + j) * c_in + c : X + (bb * c_in + c) * n_in + j) : 0.f;
          }
          float* d = xs + (nk * C + c) * BT + bh;
          if constexpr (BT == 8) *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
          else if constexpr (BT == 4) *reinterpret_cast<float2*>(d) = make_float2(v[0], v[1]);
          else *d = v[0];
        }
      }
      __syncwarp();
#pragma unroll 2
      for (int k = 0; k < m; ++k) {
        const int tp = __shfl_sync(0xffffffffu, tap, k);
#pragma unroll
        for (int c = 0; c < (CT ? CT : 4); ++c) {
          if (CT == 0 && c >= C) break;
          float w[NO], x[BT];
#pragma unroll
          for (int i = 0; i < NO; ++i) {
            const int o = lane + 32 * i;
            if (WS) w[i] = ws[(tp * C + c) * OT + o];
            else w[i] = o0 + o < c_out ? __ldg(Wt + ((long long)tp * c_out + o0 + o) * cp + c) : 0.f;
          }
          const float* xr = xs + (k * C + c) * BT;
          if constexpr (BT % 4 == 0) {
#pragma unroll
            for (int b = 0; b < BT; b += 4) {
              const float4 q = *reinterpret_cast<const float4*>(xr + b);
              x[b] = q.x; x[b + 1] = q.y; x[b + 2] = q.z; x[b + 3] = q.w;
            }
          } else {
            const float2 q = *reinterpret_cast<const float2*>(xr);
            x[0] = q.x; x[1] = q.y;
          }
#pragma unroll
          for (int i = 0; i < NO; ++i)
#pragma unroll
            for (int b = 0; b < BT; ++b) acc[i][b] = fmaf(x[b], w[i], acc[i][b]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NO; ++i) {
      const int o = o0 + lane + 32 * i;
      const float bo = bias && o < c_out ? __ldg(bias + o) : 0.f;
#pragma unroll
      for (int b = 0; b < BT; ++b) {
        if (bias) acc[i][b] += bo;
        if (relu) acc[i][b] = fmaxf(acc[i][b], 0.f);
      }
    }
    if (y_bnc) {
      if (n < n_out) {
#pragma unroll
        for (int i = 0; i < NO; ++i) {
          const int o = o0 + lane + 32 * i;
#pragma unroll
          for (int b = 0; b < BT; ++b)
            if (o < c_out && b < nb) Y[((long long)(b0 + b) * n_out + n) * c_out + o] = acc[i][b];
        }
      }
      continue;
    }
    __syncthreads();     // every warp has used its inputs
#pragma unroll
    for (int i = 0; i < NO; ++i)
#pragma unroll
      for (int b = 0; b < BT; ++b) ys[(b * OT + lane + 32 * i) * (F32_POINTS + 1) + warp] = acc[i][b];
    __syncthreads();
    for (int i = threadIdx.x; i < nb * OT * F32_POINTS; i += blockDim.x) {
      const int p = i % F32_POINTS, o = (i / F32_POINTS) % OT, b = i / (F32_POINTS * OT);
      if (n0 + p < n_out && o0 + o < c_out)
        Y[((long long)(b0 + b) * c_out + o0 + o) * n_out + n0 + p] = ys[(b * OT + o) * (F32_POINTS + 1) + p];
    }
    __syncthreads();     // the tile has left: the next item's inputs go there
  }
}

// The same for more than two images, a filter that fits shared memory and enough points (quad_pays): four points per warp, eight lanes each.
//
// What bounds the kernel above is the load/store pipe (72 % while an SM is busy), not the FMAs: a warp-wide broadcast of 16 bytes costs as long as 32 lanes'
// worth of data, so a (neighbour, channel) step of 64 channels x 8 images takes 10 clocks of shared-memory reads for 4 of FMAs; and 497 CTAs of eight points
// leave a quarter of the SMs' time empty, each with its own copy of the filter.  Here a lane holds CPL channels x BT images of one point, so that a step reads
// 16 clocks' worth for FOUR points; a CTA per SM holds the filter once, and its warps walk the quads of points of its share, which differ by one at most.  The
// eight lanes of a point gather eight neighbours at a time into registers, while the eight before are multiplied; the lanes of a warp then fetch the same
// image and channel of four neighbouring points' neighbours, which share lines.  Sums as above, in the same order, bit for bit.
// 3975 points, 49 neighbours, float32, us before -> here: 3 -> 64 channels 3 images 25 -> 17, 8 38 -> 25, 16 64 -> 49, 64 217 -> 145; 3 -> 32, 8 images 27 -> 18;
// 3 -> 96 50 -> 34; 9 neighbours, 3 -> 64, 8 images 13 -> 10.  (Sixteen warps and 128 registers, 64 channels x 8 images: 29, 88 bytes spilled; neighbours staged by
// 4-byte asynchronous copies, which conflict in shared memory, in CTAs of four warps: 37.)
constexpr int QUAD_NB = 8;                   // neighbours per pass
template <int BT, int CPL> struct QuadShape { static constexpr int WARPS = BT * CPL >= 64 ? 12 : 16; };

__host__ __device__ constexpr int quad_stride(int C, int BT) { return C * BT + (C * BT / 4 % 2 ? 0 : 4); }     // floats of a staged neighbour: an odd number of 16-byte pieces

template <typename TX, int BT, int CPL, int CT>
__global__ void __launch_bounds__(QuadShape<BT, CPL>::WARPS * 32, 1) knnconv_f32_quad_kernel(const TX* __restrict__ X, const float* __restrict__ Wt, const float* __restrict__ bias,
                                                                                           float* __restrict__ Y, const int* __restrict__ nbr_idx,
                                                                                           const uint16_t* __restrict__ nbr_tap, const int* __restrict__ nbr_cnt, int kp,
                                                                                           int B, int n_in, int n_out, int c_in, int c_out, int cp, int V, int relu,
                                                                                           int x_bnc, int y_bnc, int n_ot, int n_bt, int total) {
  extern __shared__ __align__(16) float f32_smem[];
  constexpr int OT = CPL * 8, WARPS = QuadShape<BT, CPL>::WARPS, CMAX = CT ? CT : 4;
  const int C = CT ? CT : c_in;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane >> 3, i = lane & 7;
  const int stride = quad_stride(C, BT);
  float* ws = f32_smem;                                                   // [V][C][OT]
  float* xs = f32_smem + V * C * OT + (warp * 4 + q) * QUAD_NB * stride;  // [neighbour][channel][BT images] of this lane's point
  const int ot = blockIdx.x % n_ot, o0 = ot * OT, share = blockIdx.x / n_ot, shares = gridDim.x / n_ot;      // the grid is a multiple of n_ot
  // a warp per (tap, 32 channels): consecutive lanes read consecutive rows of the tap's slab
#pragma unroll 4
  for (int r = warp; r < V * (OT / 32); r += WARPS) {
    const int v = r / (OT / 32), o = (r - v * (OT / 32)) * 32 + lane;
    const float* src = Wt + ((long long)v * c_out + o0 + o) * cp;
#pragma unroll
    for (int c = 0; c < CMAX; ++c)
      if (CT || c < C) ws[(v * C + c) * OT + o] = o0 + o < c_out ? __ldg(src + c) : 0.f;
  }
  __syncthreads();
  const int last = (int)((long long)total * (share + 1) / shares);
  for (int t = (int)((long long)total * share / shares) + warp; t < last; t += WARPS) {
    const int bt = t % n_bt, n = t / n_bt * 4 + q, b0 = bt * BT, nb = min(BT, B - b0);
    const int cnt = n < n_out ? __ldg(nbr_cnt + n) : 0;
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    const long long row = (long long)n * kp;
    int j_next = 0, tap_next = 0, tap = 0;
    float g[CMAX][BT];
    auto fetch = [&](int k0) {                                            // this lane's neighbour of the pass at k0
      if (k0 + i < cnt) { j_next = __ldg(nbr_idx + row + k0 + i); tap_next = __ldg(nbr_tap + row + k0 + i); }
    };
    auto gather = [&](int k0) {
      if (k0 + i < cnt) {
        const TX* src = X + (x_bnc ? ((long long)b0 * n_in + j_next) * c_in : (long long)b0 * c_in * n_in + j_next);
        const long long per_c = x_bnc ? 1 : n_in, per_b = (long long)c_in * n_in;
#pragma unroll
        for (int b = 0; b < BT; ++b) {
#pragma unroll
          for (int c = 0; c < CMAX; ++c)
            if (CT || c < C) g[c][b] = b < nb ? ld_as_float(src + c * per_c) : 0.f;
          src += per_b;                                                   // (not read past the batch)
        }
      }
    };
    auto put = [&]() {
#pragma unroll
      for (int c = 0; c < CMAX; ++c)
        if (CT || c < C) {
#pragma unroll
          for (int b = 0; b < BT; b += 4)
            *reinterpret_cast<float4*>(xs + i * stride + c * BT + b) = make_float4(g[c][b], g[c][b + 1], g[c][b + 2], g[c][b + 3]);
        }
    };
    float acc[CPL][BT];
#pragma unroll
    for (int o = 0; o < CPL; ++o)
#pragma unroll
      for (int b = 0; b < BT; ++b) acc[o][b] = 0.f;
#pragma unroll
    for (int c = 0; c < CMAX; ++c)
#pragma unroll
      for (int b = 0; b < BT; ++b) g[c][b] = 0.f;
    fetch(0);
    gather(0);
    tap = tap_next;
    fetch(QUAD_NB);
    put();
    __syncwarp();
    for (int k0 = 0; k0 < most; k0 += QUAD_NB) {
      const bool more = k0 + QUAD_NB < most;
      const int tap_here = tap;
      if (more) {
        gather(k0 + QUAD_NB);
        tap = tap_next;
        fetch(k0 + 2 * QUAD_NB);
      }
#pragma unroll 1
      for (int k = 0; k < min(QUAD_NB, most - k0); ++k) {
        const int tp = __shfl_sync(0xffffffffu, tap_here, (lane & 24) + k);
        if (k0 + k >= cnt) continue;                                      // this point's list is shorter than a neighbour's
        const float* wr = ws + tp * C * OT + 4 * i;
        const float* xr = xs + k * stride;
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (CT == 0 && c >= C) break;
          float w[CPL], x[BT];
#pragma unroll
          for (int u = 0; u < CPL / 4; ++u) {
            const float4 v = *reinterpret_cast<const float4*>(wr + c * OT + u * 32);
            w[4 * u] = v.x; w[4 * u + 1] = v.y; w[4 * u + 2] = v.z; w[4 * u + 3] = v.w;
          }
#pragma unroll
          for (int b = 0; b < BT; b += 4) {
            const float4 v = *reinterpret_cast<const float4*>(xr + c * BT + b);
            x[b] = v.x; x[b + 1] = v.y; x[b + 2] = v.z; x[b + 3] = v.w;
          }
#pragma unroll
          for (int o = 0; o < CPL; ++o)
#pragma unroll
            for (int b = 0; b < BT; ++b) acc[o][b] = fmaf(x[b], w[o], acc[o][b]);
        }
      }
      __syncwarp();                                                       // the pass has been read
      if (more) {
        put();
        __syncwarp();
      }
    }
    if (n < n_out) {
#pragma unroll
      for (int o = 0; o < CPL; ++o) {
        const int oc = o0 + (o >> 2) * 32 + 4 * i + (o & 3);
        if (oc < c_out) {
          const float bo = bias ? __ldg(bias + oc) : 0.f;
          float* d = Y + (y_bnc ? ((long long)b0 * n_out + n) * c_out + oc : ((long long)b0 * c_out + oc) * n_out + n);   // (planar: four points' results side by side)
#pragma unroll
          for (int b = 0; b < BT; ++b) {
            float v = acc[o][b];
            if (bias) v += bo;
            if (relu) v = fmaxf(v, 0.f);
            if (b < nb) d[(long long)b * c_out * n_out] = v;
          }
        }
      }
    }
    __syncwarp();                                                         // (the next quad's neighbours go where this one's were)
  }
}

template <typename TX, int BT, int CPL, int CT>
int launch_f32_quad_t(const fovi_knnconv_plan* p, const void* X, int x_bnc, const float* Wt, const float* bias, float* Y, int y_bnc, int B, int relu,
                      cudaStream_t st) {
  auto k = knnconv_f32_quad_kernel<TX, BT, CPL, CT>;
  constexpr int WARPS = QuadShape<BT, CPL>::WARPS;
  const int n_ot = (p->c_out + CPL * 8 - 1) / (CPL * 8), n_bt = (B + BT - 1) / BT;
  const long long total = (long long)((p->n_out + 3) / 4) * n_bt;
  if (total >= (1ll << 31)) return FOVI_ERR_UNSUPPORTED;
  const size_t smem = sizeof(float) * ((size_t)p->V * p->c_in * CPL * 8 + (size_t)WARPS * 4 * QUAD_NB * quad_stride(p->c_in, BT));
  if (smem > 48 * 1024) FOVI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = n_ot * (int)std::min<long long>(total, std::max(1, fovi::sm_count() / n_ot));
  k<<<grid, WARPS * 32, smem, st>>>((const TX*)X, Wt, bias, Y, p->nbr_idx, p->nbr_tap, p->nbr_cnt, p->kp, B, p->n_in, p->n_out, p->c_in, p->c_out,
                                    p->cin_packed, p->V, relu, x_bnc, y_bnc, n_ot, n_bt, (int)total);
  return fovi::after_launch("knnconv_f32_quad_kernel");
}

template <typename TX, int BT, int NO, int CT, bool WS>
int launch_f32_few_t(const fovi_knnconv_plan* p, const void* X, int x_bnc, const float* Wt, const float* bias, float* Y, int y_bnc, int B,
                     int relu, size_t smem, cudaStream_t st) {
  auto k = knnconv_f32_few_kernel<TX, BT, NO, CT, WS>;
  const int n_ot = (p->c_out + NO * 32 - 1) / (NO * 32), n_bt = (B + BT - 1) / BT;
  const long long total = (long long)((p->n_out + F32_POINTS - 1) / F32_POINTS) * n_bt * n_ot;
  if (total >= (1ll << 31)) return FOVI_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) FOVI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  FOVI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, F32_POINTS * 32, smem));
  const long long slots = std::max<long long>(n_ot, (long long)std::max(per_sm, 1) * fovi::sm_count() / n_ot * n_ot);
  const int grid = (int)std::min<long long>(total, slots);       // both are multiples of n_ot
  k<<<grid, F32_POINTS * 32, smem, st>>>((const TX*)X, Wt, bias, Y, p->nbr_idx, p->nbr_tap, p->nbr_cnt, p->kp, B, p->n_in, p->n_out, p->c_in,
                                         p->c_out, p->cin_packed, p->V, relu, x_bnc, y_bnc, n_ot, n_bt, (int)total);
  return fovi::after_launch("knnconv_f32_few_kernel");
}

// Which of the two kernels above serves a layer whose filter is in shared memory and whose tiles hold more than two images.  A warp of the quad kernel does four
// times the work, on one CTA per SM: a small grid leaves it with a long chain in few warps, where the eight-point kernel spreads the same points over every
// SM.  As more of that kernel's tiles share an SM its load/store pipe saturates (sooner the more values a point gathers), while the quad kernel's time stands
// still until its warps take a second quad.  Time of the quad kernel / the eight-point kernel by tiles per SM, over 1 to 4 -> 32 to 160 channels, 9, 25 and 49
// neighbours, 7 to 3975 points, 3 to 64 images:
//   up to 1    0.94 to 1.39 (8 images of 964 points, 3 -> 96, 9 neighbours: 8.4 -> 11.0 us); 4 channels, 192 values and more, 8 images in a tile of 32 channels: 0.89 to 0.95
//   1 to 2     4 channels, or 96 values gathered and more, or 48 and more for a tile of 32 channels: 0.79 to 1.03; other 0.92 to 1.19
//   2 to 3     also 3 channels, tiles of 96 (two CTAs of the eight-point kernel per SM, not four), 2 -> 32: 0.67 to 0.97; the rest (1 and 2 channels) 0.95 to 1.10
//   above      0.49 to 0.96; for that rest up to 1.09 where the quad kernel's warps have just begun another round
bool quad_pays(const fovi_knnconv_plan* p, int B, int bt, int no) {
  const int n_ot = (p->c_out + no * 32 - 1) / (no * 32), n_bt = (B + bt - 1) / bt, gathered = p->c_in * p->kp;
  const long long sms = fovi::sm_count(), tiles = (long long)((p->n_out + F32_POINTS - 1) / F32_POINTS) * n_bt * n_ot;        // of the eight-point kernel
  if (p->c_in == 4 && gathered >= 192 && no == 1 && bt == 8) return true;
  if (p->c_in >= 2 && (p->c_in == 4 || gathered >= 96 || (no == 1 && gathered >= 48))) return tiles > sms;
  if (p->c_in == 3 || no == 3 || (p->c_in == 2 && no == 1)) return tiles > 2 * sms;
  const long long warps = sms * (bt * no * 4 >= 64 ? QuadShape<8, 8>::WARPS : QuadShape<4, 4>::WARPS);
  const long long rounds = ((long long)((p->n_out + 3) / 4) * n_bt * n_ot + warps - 1) / warps;
  return rounds == 1 ? tiles > 3 * sms : 2 * tiles > 7 * rounds * sms;
}

// The exact layer of at most 4 input channels.  Images per tile: the tiles of at most eight images are made equal and rounded up to 2, 4 or 8; channels per CTA:
// 32, 64 or 96, whichever wastes the fewest lanes (the wider one on a tie).  The filter goes to shared memory when a channel tile of it is at most 64 KB (two
// CTAs of the eight-point kernel per SM then, with the inputs; a 7 x 7 filter of 3 -> 64 channels is 37 KB), else that kernel reads it through L1.  (The quad
// kernel, with one CTA per SM, would hold a larger one; it has not been measured there.)
template <typename TX>
int launch_f32_few(const fovi_knnconv_plan* p, const void* X, int x_bnc, const float* Wt, const float* bias, float* Y, int y_bnc, int B, int relu,
                   cudaStream_t st) {
  const int tiles = (B + 7) / 8, per = (B + tiles - 1) / tiles, bt = per <= 2 ? 2 : per <= 4 ? 4 : 8;
  int no = 1, best = 1 << 30;
  for (int i = 1; i <= 3; ++i) {
    const int lanes = (p->c_out + 32 * i - 1) / (32 * i) * 32 * i;
    if (lanes <= best) { best = lanes; no = i; }
  }
  const size_t base = sizeof(float) * (size_t)f32_union_floats(p->c_in, bt, no * 32);
  const size_t wbytes = sizeof(float) * (size_t)p->V * p->c_in * no * 32;
  const bool ws = wbytes <= 64 * 1024;
  const size_t smem = base + (ws ? wbytes : 0);
#define QUAD(BT_, CPL_) do { if (p->c_in == 3) return launch_f32_quad_t<TX, BT_, CPL_, 3>(p, X, x_bnc, Wt, bias, Y, y_bnc, B, relu, st);    \
                             return launch_f32_quad_t<TX, BT_, CPL_, 0>(p, X, x_bnc, Wt, bias, Y, y_bnc, B, relu, st); } while (0)
#define QUAD_NO(BT_) do { if (no == 1) QUAD(BT_, 4); else if (no == 2) QUAD(BT_, 8); else QUAD(BT_, 12); } while (0)
  if (ws && bt > 2 && quad_pays(p, B, bt, no)) {
    if (bt == 4) QUAD_NO(4);
    QUAD_NO(8);
  }
#undef QUAD_NO
#undef QUAD
#define GO(BT_, NO_, CT_, WS_) return launch_f32_few_t<TX, BT_, NO_, CT_, WS_>(p, X, x_bnc, Wt, bias, Y, y_bnc, B, relu, smem, st)
#define GO_WS(BT_, NO_, CT_) do { if (ws) GO(BT_, NO_, CT_, true); else GO(BT_, NO_, CT_, false); } while (0)
#define GO_CT(BT_, NO_) do { if (p->c_in == 3) GO_WS(BT_, NO_, 3); else GO_WS(BT_, NO_, 0); } while (0)
#define GO_NO(BT_) do { if (no == 1) GO_CT(BT_, 1); else if (no == 2) GO_CT(BT_, 2); else GO_CT(BT_, 3); } while (0)
  if (bt == 2) GO_NO(2);
  if (bt == 4) GO_NO(4);
  GO_NO(8);
#undef GO_NO
#undef GO_CT
#undef GO_WS
#undef GO
}

// Exact float32 forward of any layer.  One CTA: one output point, BT batch rows, all output channels.  Serves the layers of more
// than 4 input channels (parity runs and their gradients); the others take the kernel above.
template <typename TX, bool X_BNC, bool Y_BNC>
__global__ void __launch_bounds__(128) knnconv_f32_kernel(const TX* __restrict__ X, const float* __restrict__ Wt,
                                                          const float* __restrict__ bias, float* __restrict__ Y,
                                                          const int* __restrict__ nbr_idx, const uint16_t* __restrict__ nbr_tap,
                                                          const int* __restrict__ nbr_cnt, int kp, int B, int n_in, int n_out,
                                                          int c_in, int c_out, int cp, int relu, int BT) {
  const int n = blockIdx.x;
  const int b0 = blockIdx.y * BT;
  const int cnt = nbr_cnt[n];
  const int* idx = nbr_idx + (long long)n * kp;
  const uint16_t* tp = nbr_tap + (long long)n * kp;
  const int bt = min(BT, B - b0);
  for (int p = threadIdx.x; p < bt * c_out; p += blockDim.x) {
    const int o = p % c_out, b = b0 + p / c_out;
    float acc = 0.f;
    for (int k = 0; k < cnt; ++k) {
      const int j = idx[k];
      const float* w = Wt + ((long long)tp[k] * c_out + o) * cp;
      for (int c = 0; c < c_in; ++c) {
        const float xv = X_BNC ? ld_as_float(X + ((long long)b * n_in + j) * c_in + c)
                               : ld_as_float(X + ((long long)b * c_in + c) * n_in + j);
        acc = fmaf(xv, __ldg(w + c), acc);
      }
    }
    if (bias) acc += __ldg(bias + o);
    if (relu) acc = fmaxf(acc, 0.f);
    if (Y_BNC) Y[((long long)b * n_out + n) * c_out + o] = acc;
    else Y[((long long)b * c_out + o) * n_out + n] = acc;
  }
}

}  // namespace

extern "C" int fovi_knnconv_plan_create(const int32_t* knn_idx_pad, const uint16_t* tap, int n_in, int n_out, int K, int V,
                                        int c_in, int c_out, fovi_knnconv_plan** out) {
  if (!knn_idx_pad || !tap || !out) return FOVI_ERR_INVALID_ARGUMENT;
  if (n_in <= 0 || n_out <= 0 || K <= 0 || V <= 0 || c_in <= 0 || c_out <= 0 || V > 65535) return FOVI_ERR_INVALID_ARGUMENT;
  const int kp = (K + 7) / 8 * 8;
  std::vector<int> idx((size_t)n_out * kp, n_in), cnt(n_out, 0);
  std::vector<uint16_t> tp((size_t)n_out * kp, 0);
  int64_t nnz = 0;
  for (int n = 0; n < n_out; ++n) {
    int m = 0;
    for (int k = 0; k < K; ++k) {
      const int j = knn_idx_pad[(size_t)k * n_out + n];
      const int t = tap[(size_t)n * K + k];
      if (j < 0 || j > n_in || t >= V) return FOVI_ERR_TABLE_RANGE;
      if (j == n_in) continue;  // pad neighbour: contributes nothing
      idx[(size_t)n * kp + m] = j;
      tp[(size_t)n * kp + m] = (uint16_t)t;
      ++m;
    }
    cnt[n] = m;
    nnz += m;
  }
  auto* p = new fovi_knnconv_plan();
  p->n_in = n_in; p->n_out = n_out; p->K = K; p->V = V; p->c_in = c_in; p->c_out = c_out; p->kp = kp; p->nnz = nnz; p->bias_period = c_out;
  p->cin_packed = (c_in % 64 == 0) ? c_in : (c_in + 7) / 8 * 8;
  p->ct = (c_out % 16 == 0) ? fovi::pick_cout_tile(c_out) : 0;
  // Pair mode for tiny channel counts: group each point's neighbours into aligned input pairs
  // (2p, 2p+1).  A neighbour takes the free half of a slot of its pair, or opens a new slot (so a
  // table that lists the same input point twice still adds both taps).
  std::vector<int> pidx, pcnt;
  std::vector<uint16_t> ptap, prun, pbox;
  if (c_in <= 4) {
    p->x_layout = FOVI_X_PAIRS;
    p->n_pairs = (n_in + 1) / 2;
    std::vector<std::vector<int>> slots_idx(n_out);
    std::vector<std::vector<uint16_t>> slots_tap(n_out);
    int max_slots = 0;
    for (int n = 0; n < n_out; ++n) {
      auto& si = slots_idx[n];
      auto& st = slots_tap[n];
      for (int m = 0; m < cnt[n]; ++m) {
        const int j = idx[(size_t)n * kp + m], pr = j >> 1, h = j & 1;
        size_t s = 0;
        for (; s < si.size(); ++s)
          if (si[s] == pr && st[2 * s + h] == 0xFFFF) break;
        if (s == si.size()) { si.push_back(pr); st.push_back(0xFFFF); st.push_back(0xFFFF); }
        st[2 * s + h] = tp[(size_t)n * kp + m];
      }
      max_slots = std::max<int>(max_slots, (int)si.size());
    }
    p->sp = std::max(8, (max_slots + 7) / 8 * 8);
    pidx.assign((size_t)n_out * p->sp, p->n_pairs);
    ptap.assign((size_t)n_out * p->sp * 2, 0xFFFF);
    pcnt.assign(n_out, 0);
    for (int n = 0; n < n_out; ++n) {
      // visit pairs in ascending order: neighbouring slots then read neighbouring memory
      std::vector<int> order(slots_idx[n].size());
      for (size_t s = 0; s < order.size(); ++s) order[s] = (int)s;
      std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return slots_idx[n][a] < slots_idx[n][b]; });
      for (size_t s = 0; s < order.size(); ++s) {
        pidx[(size_t)n * p->sp + s] = slots_idx[n][order[s]];
        ptap[((size_t)n * p->sp + s) * 2] = slots_tap[n][2 * order[s]];
        ptap[((size_t)n * p->sp + s) * 2 + 1] = slots_tap[n][2 * order[s] + 1];
      }
      pcnt[n] = (int)order.size();
    }
    // Copy plan: inside every 8-slot stage, consecutive pair indices are consecutive 2 KB blocks of the
    // activations, so each run moves with one copy; the unused tail of the last stage is one run of zeros.
    prun.assign((size_t)n_out * p->sp, 0);
    pbox.assign((size_t)n_out * p->sp, 0);
    for (int n = 0; n < n_out; ++n) {
      const int* row = &pidx[(size_t)n * p->sp];
      for (int s0 = 0; s0 < p->sp; s0 += 8) {
        int j = 0;
        while (j < 8) {
          int len = 1;
          if (row[s0 + j] >= p->n_pairs) len = 8 - j;
          else while (j + len < 8 && row[s0 + j + len] == row[s0 + j] + len && row[s0 + j + len] < p->n_pairs) ++len;
          prun[(size_t)n * p->sp + s0 + j] = (uint16_t)len;
          for (int at = j, left = len; left > 0;) {
            int lg = 3;
            while ((1 << lg) > left) --lg;
            pbox[(size_t)n * p->sp + s0 + at] = (uint16_t)(lg + 1);
            at += 1 << lg; left -= 1 << lg;
          }
          j += len;
        }
      }
    }
  }
  cudaError_t e = cudaGetDevice(&p->device);
  if (e == cudaSuccess && p->x_layout == FOVI_X_PAIRS) {
    e = cudaMalloc(&p->pair_idx, sizeof(int) * pidx.size());
    if (e == cudaSuccess) e = cudaMalloc(&p->pair_cnt, sizeof(int) * n_out);
    if (e == cudaSuccess) e = cudaMalloc(&p->pair_tap, sizeof(uint16_t) * ptap.size());
    if (e == cudaSuccess) e = cudaMalloc(&p->pair_run, sizeof(uint16_t) * prun.size());
    if (e == cudaSuccess) e = cudaMemcpy(p->pair_run, prun.data(), sizeof(uint16_t) * prun.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&p->pair_box, sizeof(uint16_t) * pbox.size());
    if (e == cudaSuccess) e = cudaMemcpy(p->pair_box, pbox.data(), sizeof(uint16_t) * pbox.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&p->zero_block, 16384);
    if (e == cudaSuccess) e = cudaMemset(p->zero_block, 0, 16384);
    if (e == cudaSuccess) e = cudaMemcpy(p->pair_idx, pidx.data(), sizeof(int) * pidx.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->pair_cnt, pcnt.data(), sizeof(int) * n_out, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->pair_tap, ptap.data(), sizeof(uint16_t) * ptap.size(), cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) e = cudaMalloc(&p->nbr_idx, sizeof(int) * idx.size());
  if (e == cudaSuccess) e = cudaMalloc(&p->nbr_tap, sizeof(uint16_t) * tp.size());
  if (e == cudaSuccess) e = cudaMalloc(&p->nbr_cnt, sizeof(int) * n_out);
  if (e == cudaSuccess) e = cudaMalloc(&p->status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(p->nbr_idx, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p->nbr_tap, tp.data(), sizeof(uint16_t) * tp.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p->nbr_cnt, cnt.data(), sizeof(int) * n_out, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(p->status, 0, sizeof(int));
  if (e != cudaSuccess) {
    fovi_knnconv_plan_destroy(p);
    return fovi::cuda_fail(e, "fovi_knnconv_plan_create");
  }
  *out = p;
  return FOVI_OK;
}

extern "C" void fovi_knnconv_plan_destroy(fovi_knnconv_plan* p) {
  if (!p) return;
  if (p->nbr_idx) cudaFree(p->nbr_idx);
  if (p->nbr_tap) cudaFree(p->nbr_tap);
  if (p->nbr_cnt) cudaFree(p->nbr_cnt);
  if (p->status) cudaFree(p->status);
  if (p->pair_idx) cudaFree(p->pair_idx);
  if (p->pair_cnt) cudaFree(p->pair_cnt);
  if (p->pair_tap) cudaFree(p->pair_tap);
  if (p->zero_block) cudaFree(p->zero_block);
  if (p->pair_run) cudaFree(p->pair_run);
  if (p->pair_box) cudaFree(p->pair_box);
  if (p->seg_start) cudaFree(p->seg_start);
  if (p->seg_place) cudaFree(p->seg_place);
  delete p;
}

extern "C" int fovi_knnconv_plan_set_bias_period(fovi_knnconv_plan* p, int period) {
  if (!p || period <= 0 || p->c_out % period) return FOVI_ERR_INVALID_ARGUMENT;
  if (p->x_layout != FOVI_X_PAIRS) return FOVI_ERR_UNSUPPORTED;   // only the pair-layout kernel reads the period
  p->bias_period = period;
  return FOVI_OK;
}

extern "C" int fovi_knnconv_cin_packed(const fovi_knnconv_plan* p) { return p ? p->cin_packed : -1; }
extern "C" int64_t fovi_knnconv_nnz(const fovi_knnconv_plan* p) { return p ? p->nnz : -1; }
extern "C" int fovi_knnconv_x_layout(const fovi_knnconv_plan* p) { return p ? p->x_layout : -1; }
extern "C" int fovi_knnconv_tc_supported(const fovi_knnconv_plan* p) {
  if (!p || !p->ct) return 0;
  return (p->x_layout == FOVI_X_PAIRS ? p->sp : p->kp) <= 256 ? 1 : 0;
}

extern "C" int64_t fovi_knnconv_packed_weight_bytes(const fovi_knnconv_plan* p, int dst_dtype) {
  if (!p || !fovi::valid_dtype(dst_dtype)) return -1;
  if (p->x_layout == FOVI_X_PAIRS && dst_dtype == FOVI_BF16) return (int64_t)p->n_out * p->sp * p->c_out * 8 * 2;
  return (int64_t)p->V * p->c_out * p->cin_packed * (int64_t)fovi::dtype_size(dst_dtype);
}

extern "C" int fovi_knnconv_pack_weights(const fovi_knnconv_plan* p, const void* W, int w_dtype, void* dst, int dst_dtype,
                                         void* stream) {
  if (!p || !W || !dst || !fovi::valid_dtype(w_dtype) || !fovi::valid_dtype(dst_dtype)) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (p->x_layout == FOVI_X_PAIRS && dst_dtype == FOVI_BF16) {
    if (!p->ct) return FOVI_ERR_UNSUPPORTED;
    const long long tot = (long long)p->n_out * p->sp * p->c_out * 8;
    const int g = (int)std::min<long long>((tot + 255) / 256, 148 * 32);
    if (w_dtype == FOVI_F32)
      pack_weights_pairs_kernel<float><<<g, 256, 0, st>>>((const float*)W, (__nv_bfloat16*)dst, p->pair_tap, p->n_out, p->sp, p->V, p->c_out, p->c_in, p->ct);
    else
      pack_weights_pairs_kernel<__nv_bfloat16><<<g, 256, 0, st>>>((const __nv_bfloat16*)W, (__nv_bfloat16*)dst, p->pair_tap, p->n_out, p->sp, p->V, p->c_out, p->c_in, p->ct);
    return fovi::after_launch("pack_weights_pairs_kernel");
  }
  // slabs [V][c_out][cin_packed]
  return tap_transpose<true>(W, w_dtype, dst, dst_dtype, p->c_out, p->c_in, p->cin_packed, p->V, (long long)p->c_in * p->V, p->V,
                             (long long)p->c_out * p->cin_packed, p->cin_packed, st);
}

extern "C" int fovi_knnconv_pack_weights_transposed(const fovi_knnconv_plan* p, const void* W, int w_dtype, void* dst, int dst_dtype, void* stream) {
  if (!p || !W || !dst || !fovi::valid_dtype(w_dtype) || !fovi::valid_dtype(dst_dtype)) return FOVI_ERR_INVALID_ARGUMENT;
  if (p->x_layout == FOVI_X_PAIRS) return FOVI_ERR_UNSUPPORTED;
  return tap_transpose<true>(W, w_dtype, dst, dst_dtype, p->c_out, p->c_in, p->cin_packed, p->V, p->V, (long long)p->c_out * p->V,
                             (long long)p->c_out * p->cin_packed, p->cin_packed, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int fovi_weight_grad_unpack(const float* src, int V, int n_i, int n_j, int swapped, int c_out, int c_in, void* dst, int dst_dtype, void* stream) {
  if (!src || !dst || V <= 0 || c_out <= 0 || c_in <= 0 || !fovi::valid_dtype(dst_dtype)) return FOVI_ERR_INVALID_ARGUMENT;
  if ((swapped ? n_j : n_i) < c_out || (swapped ? n_i : n_j) < c_in) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long plane = (long long)n_i * n_j;
  return swapped ? tap_transpose<false>(src, FOVI_F32, dst, dst_dtype, c_in, c_out, c_out, V, V, (long long)c_in * V, plane, n_j, st)
                 : tap_transpose<false>(src, FOVI_F32, dst, dst_dtype, c_out, c_in, c_in, V, (long long)c_in * V, V, plane, n_j, st);
}

extern "C" int fovi_knnconv_pack_weights_grouped(const fovi_knnconv_plan* p, const void* W, int w_dtype, const uint16_t* member_tap, int G,
                                                 int V, void* dst, void* stream) {
  if (!p || !W || !member_tap || !dst || !fovi::valid_dtype(w_dtype) || G <= 0 || V <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (p->x_layout != FOVI_X_PAIRS || !p->ct || p->c_out % G) return FOVI_ERR_UNSUPPORTED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (V <= GROUPED_TAPS && p->c_in <= 4) {
    const size_t smem = (size_t)V * 33 * 8;
    const int co = p->c_out / G;
    const int nx = (co + 31) / 32, split = std::max(1, fovi::sm_count() / (nx * G));
    const dim3 grid3(nx, G, split);
#define GO(TW)                                                                                                                                   \
  do {                                                                                                                                           \
    if (smem > 48 * 1024)                                                                                                                        \
      FOVI_CUDA(cudaFuncSetAttribute(pack_weights_grouped_smem_kernel<TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));             \
    pack_weights_grouped_smem_kernel<TW><<<grid3, 512, smem, st>>>((const TW*)W, (__nv_bfloat16*)dst, p->pair_tap, member_tap, p->n_out, p->sp, p->K, \
                                                                   G, V, co, p->c_in, p->ct);                                                    \
  } while (0)
    if (w_dtype == FOVI_F32) GO(float); else GO(__nv_bfloat16);
#undef GO
    return fovi::after_launch("pack_weights_grouped_smem_kernel");
  }
  const long long tot = (long long)p->n_out * p->sp * p->c_out;   // 16-byte rows
  const int grid = (int)std::min<long long>((tot + 255) / 256, 148 * 32);
  if (w_dtype == FOVI_F32)
    pack_weights_grouped_kernel<float><<<grid, 256, 0, st>>>((const float*)W, (__nv_bfloat16*)dst, p->pair_tap, member_tap, p->n_out, p->sp, p->K,
                                                             G, V, p->c_out / G, p->c_in, p->ct);
  else
    pack_weights_grouped_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)W, (__nv_bfloat16*)dst, p->pair_tap, member_tap, p->n_out,
                                                                     p->sp, p->K, G, V, p->c_out / G, p->c_in, p->ct);
  return fovi::after_launch("pack_weights_grouped_kernel");
}

extern "C" int fovi_pack_points(const void* x, int x_dtype, int B, int C, int N, void* dst, int cp, int x_layout, void* stream) {
  if (!fovi::valid_dtype(x_dtype) || B < 0 || C <= 0 || N <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (x_layout != FOVI_X_BNC && x_layout != FOVI_X_PAIRS) return FOVI_ERR_INVALID_ARGUMENT;
  if (x_layout == FOVI_X_BNC && (cp < C || cp % 8)) return FOVI_ERR_INVALID_ARGUMENT;
  if (x_layout == FOVI_X_PAIRS && C > 4) return FOVI_ERR_INVALID_ARGUMENT;
  if (B == 0) return FOVI_OK;
  if (!x || !dst) return FOVI_ERR_INVALID_ARGUMENT;
  if (B > 65535) return FOVI_ERR_UNSUPPORTED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (x_layout == FOVI_X_PAIRS) {
    const long long tot = (long long)((N + 1) / 2) * ((B + 127) / 128 * 128);
    const int g = (int)std::min<long long>((tot + 255) / 256, 148 * 32);
    if (x_dtype == FOVI_F32) pack_points_pairs_kernel<float><<<g, 256, 0, st>>>((const float*)x, (__nv_bfloat16*)dst, B, C, N);
    else pack_points_pairs_kernel<__nv_bfloat16><<<g, 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)dst, B, C, N);
    return fovi::after_launch("pack_points_pairs_kernel");
  }
  dim3 grid((N + 31) / 32, (cp + 31) / 32, B), block(32, 8);
  if (x_dtype == FOVI_F32) pack_points_kernel<float><<<grid, block, 0, st>>>((const float*)x, (__nv_bfloat16*)dst, C, N, cp);
  else pack_points_kernel<__nv_bfloat16><<<grid, block, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)dst, C, N, cp);
  return fovi::after_launch("pack_points_kernel");
}

extern "C" int fovi_knnconv_forward_f32(const fovi_knnconv_plan* p, const void* X, int x_dtype, int x_layout, const float* Wt,
                                        const float* bias, float* Y, int y_layout, int B, int relu, void* stream) {
  if (!p || !fovi::valid_dtype(x_dtype) || B < 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (B > 0 && (!X || !Wt || !Y)) return FOVI_ERR_INVALID_ARGUMENT;
  if ((x_layout != FOVI_ACT_BCN && x_layout != FOVI_ACT_BNC) || (y_layout != FOVI_ACT_BCN && y_layout != FOVI_ACT_BNC))
    return FOVI_ERR_INVALID_ARGUMENT;
  if (B == 0) return FOVI_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int BT = 4;
  if ((B + BT - 1) / BT > 65535) return FOVI_ERR_UNSUPPORTED;
  if (p->c_in <= 4) {
    const int xb_ = x_layout == FOVI_ACT_BNC, yb_ = y_layout == FOVI_ACT_BNC;
    return x_dtype == FOVI_F32 ? launch_f32_few<float>(p, X, xb_, Wt, bias, Y, yb_, B, relu, st)
                               : launch_f32_few<__nv_bfloat16>(p, X, xb_, Wt, bias, Y, yb_, B, relu, st);
  }
  dim3 grid(p->n_out, (B + BT - 1) / BT);
#define RUN(TX, XL, YL)                                                                                                   \
  knnconv_f32_kernel<TX, XL, YL><<<grid, 128, 0, st>>>((const TX*)X, Wt, bias, Y, p->nbr_idx, p->nbr_tap, p->nbr_cnt, p->kp, B, \
                                                       p->n_in, p->n_out, p->c_in, p->c_out, p->cin_packed, relu, BT)
  const bool xb = x_layout == FOVI_ACT_BNC, yb = y_layout == FOVI_ACT_BNC;
  if (x_dtype == FOVI_F32) {
    if (xb && yb) RUN(float, true, true); else if (xb) RUN(float, true, false);
    else if (yb) RUN(float, false, true); else RUN(float, false, false);
  } else {
    if (xb && yb) RUN(__nv_bfloat16, true, true); else if (xb) RUN(__nv_bfloat16, true, false);
    else if (yb) RUN(__nv_bfloat16, false, true); else RUN(__nv_bfloat16, false, false);
  }
#undef RUN
  return fovi::after_launch("knnconv_f32_kernel");
}

// ------------------------------------------------------------------------------------------------
// Allocation-free forward from the reference's [B, c_in, n_in] layout.
//
// Some hosts may not allocate device memory at the point where they run a layer: code inside a
// real-time loop or a serving thread that was handed a fixed memory budget at start-up, or a
// plug-in whose host application owns the allocator and forbids allocation calls from callbacks
// (cudaMalloc also synchronises the whole device, which such hosts cannot afford).  For them the
// repacked copy of the activations that the tensor-core kernel reads lives in the fixed array
// below instead of a caller-provided or freshly allocated buffer.
//
// The array is part of the library image: every GPU that loads the library holds these bytes
// until the process exits.  All calls on a device share it and it keeps the last call's contents,
// so two calls that overlap on the GPU (different streams) race; issue them on one stream.
#define FOVI_STATIC_SCRATCH_BYTES (32u << 20)
static __device__ __align__(256) unsigned char g_static_scratch[FOVI_STATIC_SCRATCH_BYTES];

namespace {
// Device address of g_static_scratch on each device.  In host code the array's name is only a
// handle for the runtime, not an address a kernel could use, so it is resolved once per device.
int static_scratch_address(unsigned char** out) {
  static unsigned char* addr[64] = {nullptr};
  int dev = -1;
  FOVI_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return FOVI_ERR_UNSUPPORTED;
  if (!addr[dev]) {
    void* p = nullptr;
    FOVI_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));  // the current device is `dev`
    addr[dev] = static_cast<unsigned char*>(p);
  }
  *out = addr[dev];
  return FOVI_OK;
}
}  // namespace

extern "C" int64_t fovi_static_scratch_bytes(void) { return (int64_t)FOVI_STATIC_SCRATCH_BYTES; }

extern "C" int fovi_knnconv_forward_bcn_static(fovi_knnconv_plan* p, const void* X, int x_dtype, const void* Wt,
                                               const float* bias, void* Y, int y_dtype, int B, int relu, void* stream) {
  if (!p || !fovi::valid_dtype(x_dtype) || !fovi::valid_dtype(y_dtype) || B < 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (B == 0) return FOVI_OK;
  if (!X || !Wt || !Y) return FOVI_ERR_INVALID_ARGUMENT;
  const bool pairs = p->x_layout == FOVI_X_PAIRS;
  const long long need = pairs ? (long long)((B + 127) / 128) * p->n_pairs * 2048
                               : (long long)B * p->n_in * p->cin_packed * 2;
  if (need > (long long)FOVI_STATIC_SCRATCH_BYTES) {
    fovi::g_last_cuda_error = "fovi_knnconv_forward_bcn_static: the packed activations need " + std::to_string(need) +
                              " bytes, the static scratch holds " + std::to_string(FOVI_STATIC_SCRATCH_BYTES) +
                              "; use a smaller batch or fovi_pack_points + fovi_knnconv_forward";
    return FOVI_ERR_UNSUPPORTED;
  }
  unsigned char* scratch = nullptr;
  int rc = static_scratch_address(&scratch);
  if (rc) return rc;
  rc = fovi_pack_points(X, x_dtype, B, p->c_in, p->n_in, scratch, p->cin_packed, p->x_layout, stream);
  if (rc) return rc;
  return fovi_knnconv_forward(p, scratch, Wt, bias, Y, y_dtype, B, relu, stream);
}
