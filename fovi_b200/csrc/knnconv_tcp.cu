// KNNConv, pair layout (c_in <= 4: RGB first layers, patch embeddings), on CTA PAIRS (tcgen05 cta_group::2).
//
// Same contraction and operand layouts as the PAIRS mode of knnconv_tc.cu (activations [row tile][point pair][128 rows][2 x 4]
// bf16, weights pre-gathered per output point and c_out tile), for batches of more than one row tile.  The single-CTA kernel is
// bound by the L2 -> shared-memory stream: every stage brings 16 KB of activations and 24-32 KB of weights for 4 MMAs of 128 rows.
// Here a cluster of two CTAs computes 256 rows x one c_out tile with M = 256 MMAs; each CTA stages its own 128 rows of A and half of
// the c_out tile of B, which halves the weight bytes per SM and keeps more stages in flight.
//
// Roles per CTA: warps 0-7 epilogue; warp 8 MMA issuer (leader); four producer warps (both CTAs; copies land in the CTA's own shared memory
// and complete on the leader's full[s]), taking turns on the stages: issuing a stage's three to nine copies and waiting for its
// slot takes one warp longer than the MMAs of the stage last.  The copies are tensor copies, because a plain bulk copy can only signal a barrier
// of the CTA it writes to: a (pair, 128 rows) block is 2 KB and consecutive pairs follow each other, so a run of consecutive pairs
// of the list moves as boxes of 8, 4, 2 and 1 blocks (the plan lists them, one tensor map per size), and a stage's weights are one box.
// Slots past the list read pair n_pairs, which the copy fills with zeros.
// Barriers: full[s] and acc_empty[i] are the leader's; empty[s] and acc_full[i] exist in both CTAs and are signalled by the leader's
// multicast commits.  All waits are bounded.
// Measured, single-CTA kernel -> this one: 3 -> 1280 onto 63 tokens, 8192 rows 681 -> 565 us; 3 -> 384, 1024 rows 38 -> 33, 256 rows 21 -> 13;
// 3 -> 1280 onto 231 tokens, 2048 rows 464 -> 342; 3 -> 64 grouped by 3 onto 1023 points, 1024 rows 118 -> 87.  Of 565 us the 1.3 GB of results
// need 200 at the copy rate and the MMAs 320.  (With plain bulk copies and a relay warp in the peer, whose arrival has to be a
// cluster-scope release, a stage took 850 ns whatever the ring's depth and the bytes per stage.)
#include "tc_common.cuh"

namespace {

constexpr int PS_EPI_WARPS = 8;                                     // two sets of four, one per accumulator
constexpr int PS_THREADS = (PS_EPI_WARPS + 1 + PRODUCER_WARPS) * 32;

struct PsArgs {
  const int* slot_pair; const uint16_t* slot_box; const int* slot_cnt;
  const float* bias; void* Y; int* status;
  int kp, B, n_out, c_out, ct, n_ct, n_mt2, nstage, relu, y_f32, y_tma, bias_period, total;
  uint32_t bias_bytes, stage_bytes, wait_limit;
  int skip_loads;
};

struct PsHeader {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t ps_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t ps_map(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void ps_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void ps_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// Tensor copy whose completion is counted on a barrier that may live in the peer CTA of the pair.
__device__ __forceinline__ void ps_load(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void ps_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void ps_commit(uint32_t bar) {   // arrives on this barrier of BOTH CTAs when the MMAs so far have completed
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}

struct PsMaps { CUtensorMap x[4], w, y; };   // x[i]: boxes of 2^i pair blocks; w: one stage's half of a c_out tile; y: 32 rows x 64 columns of bf16 results

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PS_THREADS, 1)
fovi_knnconv_tc_pairs2_kernel(const __grid_constant__ PsMaps maps, const PsArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* basep = smem_raw + (base - raw);
  PsHeader* hdr = reinterpret_cast<PsHeader*>(basep);
  float* bias_s = reinterpret_cast<float*>(basep + 1024);
  const uint32_t stages0 = base + 1024u + a.bias_bytes;
  const int half = a.ct / 2;                                                         // c_out rows of B this CTA stages
  volatile int* abort_flag = &hdr->abort_flag;

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t rank = ps_ctarank();
  const int pair = blockIdx.x >> 1, n_cta_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.nstage; ++s) { mbar_init(smem_u32(&hdr->full[s]), 1); mbar_init(smem_u32(&hdr->empty[s]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&hdr->acc_full[i]), 1); mbar_init(smem_u32(&hdr->acc_empty[i]), 8); }
    mbar_init(smem_u32(&hdr->drain), 1);
    hdr->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == PS_EPI_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&hdr->tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // see fovi_knnconv_tc_kernel
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int i = threadIdx.x; i < a.c_out; i += blockDim.x) bias_s[i] = a.bias ? __ldg(a.bias + i % a.bias_period) : 0.f;
  tc_fence_before();
  ps_cluster_sync();
  tc_fence_after();
  const uint32_t tmem = hdr->tmem_base;

  if (warp > PS_EPI_WARPS) {
    // ------------------------------------------------------------ producers (both CTAs): the warps take turns on the stages (see ring.cuh), nine lanes
    // Unit order: the row tile varies fastest, so that the pairs that run at the same time share a point's weights, which are the larger operand, and
    // the c_out tiles of a point follow each other while its activations are in L2.
    int st = warp - PS_EPI_WARPS - 1;
    RingTurn ring(st, a.nstage);
    int unit = a.skip_loads || ring.idle ? a.total : pair;
    ItemWalk it(pair, n_cta_pairs, a.n_mt2, a.n_ct), ahead = it;             // d0 row tile, d1 c_out tile, d2 output point
    int steps = unit < a.total ? (__ldg(a.slot_cnt + it.d2) + 7) / 8 : 0, cnt_ahead = 0;
    auto look_ahead = [&]() {
      ahead.next();
      if (unit + n_cta_pairs < a.total) cnt_ahead = __ldg(a.slot_cnt + ahead.d2);
    };
    look_ahead();
    int pr = 0;
    uint32_t box = 0;                          // the slot this lane serves in the warp's next stage
    auto settle = [&]() {                      // moves on to an existing stage and requests its slots
      while (st >= steps) {
        st -= steps;
        unit += n_cta_pairs;
        if (unit >= a.total) return;
        it = ahead; steps = (cnt_ahead + 7) / 8;
        look_ahead();
      }
      if (lane < 8) {
        const size_t at = (size_t)it.d2 * a.kp + st * 8 + lane;
        pr = __ldg(a.slot_pair + at);
        box = __ldg(a.slot_box + at);          // 1 + log2(blocks) at the first slot of a box, else 0
      }
    };
    if (unit < a.total) settle();
    while (unit < a.total) {
      const uint32_t full_leader = ps_map(smem_u32(&hdr->full[ring.s]), 0);
      const uint32_t sa = stages0 + ring.s * a.stage_bytes;
      bool mine = true;
      if (lane == 0) {
        mine = mbar_wait(smem_u32(&hdr->empty[ring.s]), ring.ph ^ 1u, abort_flag, a.status, 21, a.wait_limit);
        if (mine && rank == 0) mbar_expect_tx(smem_u32(&hdr->full[ring.s]), 2u * a.stage_bytes);   // both CTAs' bytes
      }
      if (!__all_sync(0xffffffffu, mine)) break;   // nobody copies into a stage before lane 0 saw it free
      if (lane < 8) {                          // a row tile past an odd last one reads as zeros; nothing of it is stored
        if (box) ps_load(sa + lane * 2048u, &maps.x[box - 1], full_leader, 0, 0, pr, it.d0 * 2 + (int)rank);
      } else if (lane == 8) {
        ps_load(sa + A_STAGE_BYTES, &maps.w, full_leader, 0, (int)rank * (half >> 4), st * 8, it.d2 * a.n_ct + it.d1);
      }
      st += (int)ring.step;
      settle();
      ring.next();
    }
    if (lane == 0 && *abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies in flight land before this CTA's shared memory goes away
    }
  } else if (warp == PS_EPI_WARPS) {
    // ------------------------------------------------------------ MMA issuer (leader; see elect_one)
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.ct >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint32_t lbo_b = (uint32_t)half * 16u;
      const uint64_t desc_a = smem_desc(0, 2048u, 128u, 0u), desc_b = smem_desc(0, lbo_b, 128u, 0u);
      const uint32_t u_stages0 = warp_uniform(stages0), u_tmem = warp_uniform(tmem);
      uint32_t s = 0, ph = 0, acc = 0, aph = 0;
      bool ok = true;
      int cnt = pair < a.total ? __ldg(a.slot_cnt + pair / a.n_mt2 / a.n_ct) : 0;
      for (int unit = pair; unit < a.total && ok; unit += n_cta_pairs) {
        const int cnt_next = unit + n_cta_pairs < a.total ? __ldg(a.slot_cnt + (unit + n_cta_pairs) / a.n_mt2 / a.n_ct) : 0;
        const int steps = (warp_uniform(cnt) + 7) / 8;
        ok = mbar_wait_warp(smem_u32(&hdr->acc_empty[acc]), aph ^ 1u, abort_flag, a.status, 24, a.wait_limit);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = u_tmem + acc * 256u;
        for (int st = 0; st < steps; ++st) {
          ok = mbar_wait_warp(smem_u32(&hdr->full[s]), ph, abort_flag, a.status, 25, a.wait_limit);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = u_stages0 + s * a.stage_bytes;
          const uint64_t da = desc_a + (sa >> 4), db = desc_b + ((sa + A_STAGE_BYTES) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) ps_mma(d_tmem, da + kk * 256u, db + kk * (lbo_b >> 3), idesc, (st | kk) ? 1u : 0u);
            ps_commit(smem_u32(&hdr->empty[s]));
            if (st == steps - 1) ps_commit(smem_u32(&hdr->acc_full[acc]));
          }
          __syncwarp();
          if (++s == (uint32_t)a.nstage) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        if (steps == 0) {                                  // a point without neighbours: nothing to wait for
          if (elect_one()) ps_commit(smem_u32(&hdr->acc_full[acc]));
          __syncwarp();
        }
        if (++acc == 2) { acc = 0; aph ^= 1u; }
        cnt = cnt_next;
      }
      if (*abort_flag && elect_one()) {
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&hdr->drain)) : "memory");
        for (uint32_t i = 0; i < (1u << 20); ++i)
          if (mbar_try_wait(smem_u32(&hdr->drain), 0)) break;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    // Four warps take longer over 256 columns (2.8 us, 3.8 us with the stores) than the MMAs of a short list do (8 stages: 2.2 us): two sets of
    // four take turns (63 tokens, 1280 channels, 8192 rows: 632 -> 590 us; 231 tokens, 2048 rows: 452 -> 401).
    const int q = warp & 3, acc = warp >> 2;
    unsigned char* tile_s = basep + 1024 + a.bias_bytes + (size_t)a.nstage * a.stage_bytes + warp * 4096;   // 32 rows x 64 columns (y_tma)
    bool ok = true;
    uint32_t aph = 0;
    const int step = 2 * n_cta_pairs;
    ItemWalk it(pair + acc * n_cta_pairs, step, a.n_mt2, a.n_ct);             // d0 row tile, d1 c_out tile, d2 output point
    for (int unit = pair + acc * n_cta_pairs; unit < a.total; unit += step, it.next()) {
      const int cnt = __ldg(a.slot_cnt + it.d2);
      ok = mbar_wait(smem_u32(&hdr->acc_full[acc]), aph, abort_flag, a.status, 26, a.wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int n = it.d2, o0 = it.d1 * a.ct;
      const int row = (it.d0 * 2 + (int)rank) * BM + q * 32 + lane;
      const size_t y_off = ((size_t)row * a.n_out + n) * a.c_out + o0;
      const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + acc * 256u;
      for (int c0 = 0; c0 < a.ct; c0 += 64) {
        uint32_t r[64];
        const int w = min(64, a.ct - c0);   // 32 or 64 (ct is a multiple of 32 here)
        tc_ld32(t_base + c0, r);
        if (w == 64) tc_ld32(t_base + c0 + 32, r + 32);
        tc_ld_wait();
        if (cnt <= 0) {   // a point without neighbours: nothing was accumulated, the columns hold an earlier unit's values
#pragma unroll
          for (int i = 0; i < 64; ++i) r[i] = 0u;
        }
        if (a.y_tma) {    // the staging tile's last copy has been read
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (g * 16 < w) {
            float v[16];
            const float4* b4 = reinterpret_cast<const float4*>(bias_s + o0 + c0 + g * 16);   // 64-byte aligned
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 bb = b4[i];
              v[4 * i] = __uint_as_float(r[g * 16 + 4 * i]) + bb.x;
              v[4 * i + 1] = __uint_as_float(r[g * 16 + 4 * i + 1]) + bb.y;
              v[4 * i + 2] = __uint_as_float(r[g * 16 + 4 * i + 2]) + bb.z;
              v[4 * i + 3] = __uint_as_float(r[g * 16 + 4 * i + 3]) + bb.w;
            }
            if (a.relu) {
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
            }
            if (a.y_f32) {
              if (row < a.B) {
                float* dst = reinterpret_cast<float*>(a.Y) + y_off + c0 + g * 16;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  uint32_t w8[8];
#pragma unroll
                  for (int e = 0; e < 8; ++e) w8[e] = __float_as_uint(v[8 * i + e]);
                  st_global_32(dst + 8 * i, w8);
                }
              }
            } else {
              uint32_t pk[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                pk[i] = *reinterpret_cast<uint32_t*>(&h);
              }
              if (a.y_tma) {      // 16-byte pieces of the row's 128 bytes, in the tensor copy's 128-byte swizzle: no bank conflicts
                uint4* row_s = reinterpret_cast<uint4*>(tile_s + lane * 128);
                row_s[(2 * g) ^ (lane & 7)] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                row_s[(2 * g + 1) ^ (lane & 7)] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
              } else if (row < a.B) {
                st_global_32(reinterpret_cast<__nv_bfloat16*>(a.Y) + y_off + c0 + g * 16, pk);
              }
            }
          }
        }
        if (a.y_tma) {            // rows past the batch are outside the tensor and are not written
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                         ::"l"(&maps.y), "r"(smem_u32(tile_s)), "r"(o0 + c0), "r"(n), "r"(row - lane) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) ps_arrive_cluster(ps_map(smem_u32(&hdr->acc_empty[acc]), 0));   // the leader's MMA thread waits for all 8 warps
      aph ^= 1u;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  ps_cluster_sync();   // nobody frees tensor memory or leaves while the other CTA may still signal or read
  if (warp == PS_EPI_WARPS) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace

// Returns FOVI_ERR_UNSUPPORTED when the kernel does not apply: one row tile only (half of every MMA would be idle), or a c_out tile
// that does not split into two halves of whole 16-row groups.
int fovi::launch_knnconv_tc_pairs2(const fovi_knnconv_plan* p, const void* X, const void* Wt, const float* bias, void* Y, int y_dtype, int B,
                                 int relu, cudaStream_t st, int skip_loads, uint32_t wait_limit) {
  const int ct = p->ct;
  if (p->x_layout != FOVI_X_PAIRS || !ct || ct % 32 || B <= BM) return FOVI_ERR_UNSUPPORTED;
  const int sms = fovi::sm_count();
  if (sms < 2) return FOVI_ERR_UNSUPPORTED;
  PsArgs a;
  a.slot_pair = p->pair_idx; a.slot_box = p->pair_box; a.slot_cnt = p->pair_cnt;
  a.bias = bias; a.Y = Y; a.status = p->status;
  a.kp = p->sp; a.B = B; a.n_out = p->n_out; a.c_out = p->c_out; a.ct = ct; a.n_ct = p->c_out / ct;
  a.n_mt2 = (B + 2 * BM - 1) / (2 * BM);
  a.relu = relu; a.y_f32 = y_dtype == FOVI_F32; a.bias_period = p->bias_period;
  a.wait_limit = wait_limit; a.skip_loads = skip_loads;
  const long long units = (long long)p->n_out * a.n_ct * a.n_mt2;
  if (units >= (1ll << 30)) return FOVI_ERR_UNSUPPORTED;
  a.total = (int)units;
  a.bias_bytes = ((uint32_t)p->c_out * 4u + 1023u) & ~1023u;
  a.stage_bytes = A_STAGE_BYTES + 8u * (uint32_t)(ct / 2) * 16u;
  const uint32_t budget = 224u * 1024u - 2048u - a.bias_bytes;
  // bf16 results leave as tensor copies of 32 rows x 64 columns, through 4 KB of shared memory per epilogue warp, where the stores
  // bound the kernel: short lists (231 tokens of 28 points, 1280 channels, 2048 rows: 407 us with 32-byte stores, 342 with the
  // copies; 192 channels: 72 / 68) and results far larger than the L2 cache (63 tokens, 8192 rows, 1.3 GB: 595 / 568).  Elsewhere the
  // 32 KB are worth more as a ring stage (63 tokens, 384 channels, 1024 rows: 31.8 / 33.2; grouped 3 -> 64: 86.8 / 89.2).
  const long long y_bytes = (long long)B * p->n_out * p->c_out * 2;
  a.y_tma = !a.y_f32 && ct % 64 == 0 && (a.kp <= 32 || y_bytes > (256ll << 20));
  const uint32_t tiles = a.y_tma ? PS_EPI_WARPS * 4096u : 0u;
  a.nstage = (int)std::min<uint32_t>(MAX_STAGES, (budget - tiles) / a.stage_bytes);
  if (a.nstage < 3) return FOVI_ERR_UNSUPPORTED;
  const size_t smem = 1024 + 1024 + a.bias_bytes + (size_t)a.nstage * a.stage_bytes + tiles;
  PsMaps maps;
  const uint64_t n_mt = (uint64_t)(B + BM - 1) / BM, n_pairs = (uint64_t)p->n_pairs, slot = (uint64_t)ct * 16, kp = (uint64_t)a.kp;
  for (int i = 0; i < 4; ++i) {      // X: [row tile][pair][4][256] elements
    const uint64_t dims[4] = {256, 4, n_pairs, n_mt}, strides[3] = {512, 2048, n_pairs * 2048};
    const uint32_t box[4] = {256, 4, 1u << i, 1};
    const int rc = fovi::encode_4d(&maps.x[i], X, dims, strides, box);
    if (rc) return rc;
  }
  {                                  // weights: [slab][slot][ct / 16][128] elements
    const uint64_t dims[4] = {128, (uint64_t)ct / 16, kp, (uint64_t)p->n_out * a.n_ct}, strides[3] = {256, slot, slot * kp};
    const uint32_t box[4] = {128, (uint32_t)ct / 32, 8, 1};
    const int rc = fovi::encode_4d(&maps.w, Wt, dims, strides, box);
    if (rc) return rc;
  }
  memset(&maps.y, 0, sizeof(maps.y));
  if (a.y_tma) {
    const uint64_t row = (uint64_t)p->c_out * 2;
    const int rc = fovi::encode_3d(&maps.y, Y, (uint64_t)p->c_out, (uint64_t)p->n_out, (uint64_t)B, row, row * p->n_out, 64, 1, 32, true);
    if (rc) return rc;
  }
  FOVI_CUDA(cudaFuncSetAttribute(fovi_knnconv_tc_pairs2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int pairs = (int)std::min<long long>(units, sms / 2);
  FOVI_CUDA(fovi::launch_pdl(fovi_knnconv_tc_pairs2_kernel, 2 * pairs, PS_THREADS, smem, st, maps, a));
  return fovi::after_launch("fovi_knnconv_tc_pairs2_kernel");
}
