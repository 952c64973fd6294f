// KNNConv, 64-channel mode, for small batches (at most 16 rows): several output points share an MMA tile.
//
// The other tensor-core kernels fill a tile's rows with the batch, one output point at a time; with 4 rows, 128-row tiles are 97 % idle and, worse, every
// point streams its own weight slabs (5 layers, 4 rows: 1 GB from L2 to shared memory, which is what bounds them).  Here a CTA pair's 256 rows are
// 256 / Bp output points x Bp rows (Bp: the batch rounded up to 8 or 16), consecutive points, which mostly use the same filter taps: the
// contraction runs over the union of the group's (tap, multiplicity) entries, a tap's weight slab is loaded once for all of the group's points, and a
// point without a neighbour at that tap reads an out-of-range box, which the tensor copy fills with zeros.  The few tiles this leaves are split along
// the contraction: every split writes its float32 partial tile to a workspace and a second launch adds them in order (deterministic), with bias, ReLU and
// conversion.  4 rows, one point per tile -> this kernel: 64->192 (25 neighbours, 225 points) 21.7 -> 14.7 us, 192->384 (9) 38.5 -> 16.5, 384->256 40.7 -> 21.0,
// 256->256 30.0 -> 18.6.
//
// Roles, barriers and bounded waits as in knnconv_tc2.cu.
#include "tc_common.cuh"

namespace {

struct SmArgs {
  const uint16_t* ent_tap; const int* ent_idx; const int* ent_cnt;   // [groups][u_max], [groups][u_max][points], [groups]
  const float* bias; void* Y; float* ws; int* status;
  int u_max, points, bp_log2, B, n_in, n_out, c_out, cp, ct, n_ct, splits, nstage, relu, y_f32, total;
  uint32_t stage_bytes, wait_limit;
};

__device__ __forceinline__ uint32_t sm_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t sm_map(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void sm_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void sm_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void sm_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void sm_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// stages [lo, hi) of a unit: its share of the group's entries x 64-channel chunks
__device__ __forceinline__ void sm_range(const SmArgs& a, int chunks, int group, int split, int& lo, int& hi) {
  const int all = __ldg(a.ent_cnt + group) * chunks;
  lo = (int)((long long)all * split / a.splits); hi = (int)((long long)all * (split + 1) / a.splits);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
fovi_knnconv_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SmArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  SmemHeader* hdr = reinterpret_cast<SmemHeader*>(smem_raw + (base - raw));
  const uint32_t stages0 = base + 1024u;
  volatile int* abort_flag = &hdr->abort_flag;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = (int)sm_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int chunks = (a.cp + 63) / 64, half = a.ct / 2, per_cta = a.points / 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.nstage; ++s) { mbar_init(smem_u32(&hdr->full[s]), 1); mbar_init(smem_u32(&hdr->empty[s]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&hdr->acc_full[i]), 1); mbar_init(smem_u32(&hdr->acc_empty[i]), 8); }
    mbar_init(smem_u32(&hdr->drain), 1);
    hdr->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&hdr->tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // see fovi_knnconv_tc_kernel
  asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before();
  sm_cluster_sync();
  tc_fence_after();
  const uint32_t tmem = hdr->tmem_base;
  const ItemWalk start(pair, n_pairs, a.splits, a.n_ct);            // d0 split, d1 c_out tile, d2 group

  if (warp >= 5) {
    // ------------------------------------------------------------ producers: warp w fills every W-th stage; lanes 0 .. per_cta - 1 copy a point's rows, lane 31 the weights
    constexpr int W = PRODUCER_WARPS;
    int pos = warp - 5, lo = 0, hi = 0, sel = 0;
    uint32_t s = (uint32_t)pos, ph = 0;
    while (s >= (uint32_t)a.nstage) { s -= (uint32_t)a.nstage; ph ^= 1u; }
    ItemWalk it = start;
    int unit = pair;
    if (unit < a.total) sm_range(a, chunks, it.d2, it.d0, lo, hi);
    auto settle = [&]() {   // moves on to an existing stage and requests its point (or tap)
      while (pos >= hi - lo) {
        pos -= hi - lo;
        unit += n_pairs;
        if (unit >= a.total) return;
        it.next();
        sm_range(a, chunks, it.d2, it.d0, lo, hi);
      }
      const size_t e = (size_t)it.d2 * a.u_max + (lo + pos) / chunks;
      if (lane < per_cta) sel = __ldg(a.ent_idx + e * a.points + rank * per_cta + lane);
      if (lane == 31) sel = __ldg(a.ent_tap + e);
    };
    if (unit < a.total) settle();
    while (unit < a.total) {
      const uint32_t full_leader = sm_map(smem_u32(&hdr->full[s]), 0);
      const uint32_t sa = stages0 + s * a.stage_bytes;
      const int c0 = (lo + pos) % chunks * 64;
      bool mine = true;
      if (lane == 0) {
        mine = mbar_wait(smem_u32(&hdr->empty[s]), ph ^ 1u, abort_flag, a.status, 41, a.wait_limit);
        if (mine && rank == 0) mbar_expect_tx(smem_u32(&hdr->full[s]), 2u * a.stage_bytes);   // both CTAs' bytes
      }
      if (!__all_sync(0xffffffffu, mine)) break;
      if (lane == 31) sm_load(sa + A_STAGE_BYTES, &tmB, full_leader, c0, it.d1 * a.ct + rank * half, sel);
      if (lane < per_cta) sm_load(sa + ((uint32_t)lane << (a.bp_log2 + 7)), &tmA, full_leader, c0, sel, 0);   // no neighbour at this tap: point n_in reads as zeros
      pos += W;
      settle();
      for (s += W; s >= (uint32_t)a.nstage; s -= (uint32_t)a.nstage) ph ^= 1u;
    }
    if (lane == 0 && *abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies in flight land before this CTA's shared memory goes away
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------ MMA issuer (leader; see elect_one)
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.ct >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint64_t desc0 = smem_desc(0, 16u, 1024u, 2u);
      const uint32_t u_stages0 = warp_uniform(stages0), u_tmem = warp_uniform(tmem);
      uint32_t s = 0, ph = 0, acc = 0, aph = 0;
      bool ok = true;
      ItemWalk it = start;
      for (int unit = pair; unit < a.total && ok; unit += n_pairs, it.next()) {
        int lo, hi;
        sm_range(a, chunks, it.d2, it.d0, lo, hi);
        const int steps = warp_uniform(hi - lo);
        ok = mbar_wait_warp(smem_u32(&hdr->acc_empty[acc]), aph ^ 1u, abort_flag, a.status, 42, a.wait_limit);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = u_tmem + acc * 256u;
        for (int st = 0; st < steps; ++st) {
          ok = mbar_wait_warp(smem_u32(&hdr->full[s]), ph, abort_flag, a.status, 43, a.wait_limit);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = u_stages0 + s * a.stage_bytes;
          const uint64_t da = desc0 + (sa >> 4), db = desc0 + ((sa + A_STAGE_BYTES) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) sm_mma(d_tmem, da + kk * 2u, db + kk * 2u, idesc, (st | kk) ? 1u : 0u);
            sm_commit(smem_u32(&hdr->empty[s]));
            if (st == steps - 1) sm_commit(smem_u32(&hdr->acc_full[acc]));
          }
          __syncwarp();
          if (++s == (uint32_t)a.nstage) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        if (steps == 0) {
          if (elect_one()) sm_commit(smem_u32(&hdr->acc_full[acc]));
          __syncwarp();
        }
        if (++acc == 2) { acc = 0; aph ^= 1u; }
      }
      if (*abort_flag && elect_one()) {
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&hdr->drain)) : "memory");
        for (uint32_t i = 0; i < (1u << 20); ++i)
          if (mbar_try_wait(smem_u32(&hdr->drain), 0)) break;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;
    uint32_t acc = 0, aph = 0;
    ItemWalk it = start;
    for (int unit = pair; unit < a.total; unit += n_pairs, it.next()) {
      int lo, hi;
      sm_range(a, chunks, it.d2, it.d0, lo, hi);
      if (!mbar_wait_warp(smem_u32(&hdr->acc_full[acc]), aph, abort_flag, a.status, 44, a.wait_limit)) break;
      tc_fence_after();
      const int tile_row = q * 32 + lane;
      const int n = it.d2 * a.points + rank * per_cta + (tile_row >> a.bp_log2), b = tile_row & ((1 << a.bp_log2) - 1);
      const bool live = b < a.B && n < a.n_out;
      const int o0 = it.d1 * a.ct;
      float* part = a.ws + (((size_t)it.d0 * a.n_out + n) * a.B + b) * a.c_out + o0;          // splits > 1
      const size_t y_off = ((size_t)b * a.n_out + n) * a.c_out + o0;
      const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + acc * 256u;
      for (int c0 = 0; c0 < a.ct; c0 += 32) {
        uint32_t r[32];
        tc_ld32(t_base + c0, r);
        tc_ld_wait();
        if (hi == lo) {     // nothing was accumulated, the columns hold an earlier unit's values
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (!live) continue;
        if (a.splits > 1) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t w8[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w8[e] = r[8 * g + e];
            st_global_32(part + c0 + 8 * g, w8);
          }
        } else {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v[i] = __uint_as_float(r[i]) + (a.bias ? __ldg(a.bias + o0 + c0 + i) : 0.f);
            if (a.relu) v[i] = fmaxf(v[i], 0.f);
          }
          if (a.y_f32) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint32_t w8[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) w8[e] = __float_as_uint(v[8 * g + e]);
              st_global_32(reinterpret_cast<float*>(a.Y) + y_off + c0 + 8 * g, w8);
            }
          } else {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              uint32_t pk[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                __nv_bfloat162 h = __floats2bfloat162_rn(v[16 * g + 2 * e], v[16 * g + 2 * e + 1]);
                pk[e] = *reinterpret_cast<uint32_t*>(&h);
              }
              st_global_32(reinterpret_cast<__nv_bfloat16*>(a.Y) + y_off + c0 + 16 * g, pk);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(sm_map(smem_u32(&hdr->acc_empty[acc]), 0)) : "memory");
      if (++acc == 2) { acc = 0; aph ^= 1u; }
    }
  }

  tc_fence_before();
  sm_cluster_sync();   // nobody frees tensor memory or leaves while the other CTA may still signal or read
  if (warp == 4) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// Y[b][n][o] = act(bias[o] + sum over the splits, in order, of ws[s][n][b][o]); one thread per 8 channels.
__global__ void __launch_bounds__(128) knnconv_small_finish_kernel(const float* __restrict__ ws, const float* __restrict__ bias, void* __restrict__ Y, int B, int n_out,
                                                                  int c_out, int splits, int relu, int y_f32) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int c8 = c_out / 8;
  const long long total = (long long)n_out * B * c8, plane = (long long)n_out * B * c_out;
  const long long i = blockIdx.x * 128ll + threadIdx.x;
  if (i >= total) return;
  const int o = (int)(i % c8) * 8;
  const long long nb = i / c8;
  const int b = (int)(nb % B), n = (int)(nb / B);
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float4* src = reinterpret_cast<const float4*>(ws + nb * c_out + o);
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float4 p = src[0], q = src[1];
    v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w; v[4] += q.x; v[5] += q.y; v[6] += q.z; v[7] += q.w;
    src += plane / 4;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (bias) v[e] += __ldg(bias + o + e);
    if (relu) v[e] = fmaxf(v[e], 0.f);
  }
  const size_t off = ((size_t)b * n_out + n) * c_out + o;
  if (y_f32) {
    float4* d = reinterpret_cast<float4*>(reinterpret_cast<float*>(Y) + off);
    d[0] = make_float4(v[0], v[1], v[2], v[3]); d[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint32_t pk[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      pk[e] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(Y) + off) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  }
}

}  // namespace

// Batch -> log2 of the rows a point takes (8 or 16), or -1 when the kernel does not apply.  The line lies where four layers of the benchmark's stack
// take the same time either way: 16 rows 99 us here and 132 with one point per tile, 24 rows 129 / 132, 48 rows 163 / 135 (a group of eight points
// or less shares too few taps).
constexpr int SMALL_ROWS = 16;
static int small_bp_log2(const fovi_knnconv_plan* p, int B) {
  if (!p->small_ok || B <= 0 || B > SMALL_ROWS || fovi::sm_count() < 2) return -1;
  return B <= 8 ? 3 : 4;
}

// Splits of the contraction: as many as give every CTA pair at most one unit, but at least eight stages each.
static int small_splits(const fovi_knnconv_plan* p, int lg) {
  const auto& t = p->small[lg - 3];
  const int units = t.n_groups * (p->c_out / p->ct), chunks = (p->cin_packed + 63) / 64;
  return std::max(1, std::min({fovi::sm_count() / 2 / units, t.u_max * chunks / 8, 16}));
}

extern "C" int64_t fovi_knnconv_workspace_bytes(const fovi_knnconv_plan* p, int B) {
  if (!p || B < 0) return -1;
  const int lg = small_bp_log2(p, B);
  if (lg < 0) return 0;
  const int s = small_splits(p, lg);
  return s > 1 ? (int64_t)s * p->n_out * B * p->c_out * 4 : 0;
}

int fovi::launch_knnconv_small(const fovi_knnconv_plan* p, const void* X, const void* Wt, const float* bias, void* Y, int y_dtype, int B, int relu, void* ws,
                               int64_t ws_bytes, cudaStream_t st, int skip_loads, uint32_t wait_limit) {
  const int lg = small_bp_log2(p, B);
  if (lg < 0 || skip_loads) return FOVI_ERR_UNSUPPORTED;
  SmArgs a;
  const auto& t = p->small[lg - 3];
  a.splits = small_splits(p, lg);
  if (a.splits > 1 && (!ws || ws_bytes < fovi_knnconv_workspace_bytes(p, B) || (reinterpret_cast<uintptr_t>(ws) & 31))) return FOVI_ERR_UNSUPPORTED;
  a.ent_tap = t.tap; a.ent_idx = t.idx; a.ent_cnt = t.cnt;
  a.bias = bias; a.Y = Y; a.ws = static_cast<float*>(ws); a.status = p->status;
  a.u_max = t.u_max; a.points = 256 >> lg; a.bp_log2 = lg; a.B = B; a.n_in = p->n_in; a.n_out = p->n_out; a.c_out = p->c_out; a.cp = p->cin_packed;
  a.ct = p->ct; a.n_ct = p->c_out / p->ct; a.relu = relu; a.y_f32 = y_dtype == FOVI_F32; a.wait_limit = wait_limit;
  const long long units = (long long)t.n_groups * a.n_ct * a.splits;
  if (units >= (1ll << 30)) return FOVI_ERR_UNSUPPORTED;
  a.total = (int)units;
  a.stage_bytes = A_STAGE_BYTES + (uint32_t)(a.ct / 2) * 128u;
  a.nstage = (int)std::min<uint32_t>(MAX_STAGES, (224u * 1024u - 2048u) / a.stage_bytes);
  const size_t smem = 2048 + (size_t)a.nstage * a.stage_bytes;
  CUtensorMap tmA, tmB;
  const uint64_t cp = (uint64_t)a.cp;
  int rc = fovi::encode_3d(&tmA, X, cp, (uint64_t)p->n_in, (uint64_t)B, cp * 2, (uint64_t)p->n_in * cp * 2, 64, 1, 1u << lg, true);
  if (rc) return rc;
  rc = fovi::encode_3d(&tmB, Wt, cp, (uint64_t)p->c_out, (uint64_t)p->V, cp * 2, (uint64_t)p->c_out * cp * 2, 64, (uint32_t)(a.ct / 2), 1, true);
  if (rc) return rc;
  FOVI_CUDA(cudaFuncSetAttribute(fovi_knnconv_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int pairs = (int)std::min<long long>(units, fovi::sm_count() / 2);
  FOVI_CUDA(fovi::launch_pdl(fovi_knnconv_small_kernel, 2 * pairs, TC_THREADS, smem, st, tmA, tmB, a));
  rc = fovi::after_launch("fovi_knnconv_small_kernel");
  if (rc || a.splits == 1) return rc;
  const long long threads = (long long)p->n_out * B * (p->c_out / 8);
  FOVI_CUDA(fovi::launch_pdl(knnconv_small_finish_kernel, (int)((threads + 127) / 128), 128, 0, st, (const float*)ws, bias, Y, B, p->n_out, p->c_out, a.splits, relu,
                             a.y_f32));
  return fovi::after_launch("knnconv_small_finish_kernel");
}

// Tables of the small-batch kernel: for groups of 32 and 16 consecutive points, the union of their (tap, multiplicity) entries and each point's
// input at every entry (n_in: none).  Built with the plan for layers the kernel takes.
int fovi::build_small_tables(fovi_knnconv_plan* p, const std::vector<int>& idx, const std::vector<uint16_t>& tap, const std::vector<int>& cnt) {
  const int n_out = p->n_out, kp = p->kp;
  if (p->x_layout != FOVI_X_BNC || p->cin_packed < 16 || !p->ct || p->ct % 32 || (long long)n_out * kp > (4ll << 20)) return FOVI_OK;
  for (int lg = 3; lg <= 4; ++lg) {
    const int points = 256 >> lg, n_groups = (n_out + points - 1) / points;
    std::vector<std::vector<uint16_t>> taps(n_groups);
    std::vector<std::vector<int>> cells(n_groups);
    int u_max = 1;
    for (int g = 0; g < n_groups; ++g) {
      std::vector<std::vector<std::pair<uint16_t, int>>> lists(points);       // per point: (tap, input), sorted by tap (stable: list order inside a tap)
      for (int i = 0; i < points && g * points + i < n_out; ++i) {
        const int n = g * points + i;
        for (int k = 0; k < cnt[n]; ++k) lists[i].push_back({tap[(size_t)n * kp + k], idx[(size_t)n * kp + k]});
        std::stable_sort(lists[i].begin(), lists[i].end(), [](const auto& u, const auto& v) { return u.first < v.first; });
      }
      std::vector<size_t> at(points, 0);
      for (;;) {                                                              // the smallest tap any point still holds makes the next entry
        int t = -1;
        for (int i = 0; i < points; ++i)
          if (at[i] < lists[i].size() && (t < 0 || lists[i][at[i]].first < t)) t = lists[i][at[i]].first;
        if (t < 0) break;
        taps[g].push_back((uint16_t)t);
        for (int i = 0; i < points; ++i) {
          const bool has = at[i] < lists[i].size() && lists[i][at[i]].first == t;
          cells[g].push_back(has ? lists[i][at[i]].second : p->n_in);
          if (has) ++at[i];
        }
      }
      u_max = std::max<int>(u_max, (int)taps[g].size());
    }
    auto& s = p->small[lg - 3];
    s.n_groups = n_groups; s.u_max = u_max;
    std::vector<uint16_t> ht((size_t)n_groups * u_max, 0);
    std::vector<int> hi((size_t)n_groups * u_max * points, p->n_in), hc(n_groups);
    for (int g = 0; g < n_groups; ++g) {
      hc[g] = (int)taps[g].size();
      std::copy(taps[g].begin(), taps[g].end(), ht.begin() + (size_t)g * u_max);
      std::copy(cells[g].begin(), cells[g].end(), hi.begin() + (size_t)g * u_max * points);
    }
    FOVI_CUDA(cudaMalloc(&s.tap, sizeof(uint16_t) * ht.size()));
    FOVI_CUDA(cudaMalloc(&s.idx, sizeof(int) * hi.size()));
    FOVI_CUDA(cudaMalloc(&s.cnt, sizeof(int) * hc.size()));
    FOVI_CUDA(cudaMemcpy(s.tap, ht.data(), sizeof(uint16_t) * ht.size(), cudaMemcpyHostToDevice));
    FOVI_CUDA(cudaMemcpy(s.idx, hi.data(), sizeof(int) * hi.size(), cudaMemcpyHostToDevice));
    FOVI_CUDA(cudaMemcpy(s.cnt, hc.data(), sizeof(int) * hc.size(), cudaMemcpyHostToDevice));
  }
  p->small_ok = 1;
  return FOVI_OK;
}
