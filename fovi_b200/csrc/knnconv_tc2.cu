// KNNConv, 64-channel mode, on CTA PAIRS (tcgen05 cta_group::2).
//
// Same table-driven gather-GEMM as knnconv_tc.cu, but one work item is 256 batch rows x one c_out tile,
// computed by a cluster of two CTAs on neighbouring SMs with a single M=256 MMA: each CTA stages its own
// 128 batch rows of the activations (A) and only HALF of the weight slab (B: c_out tile / 2 rows), and the
// tensor cores of both SMs read both halves.  Halving B per SM cuts the L2 -> shared-memory
// stream (16 KB of A + 24-32 KB of B per 64-channel chunk in the single-CTA kernel) by 30-33 % for the same MMA work.
//
// Roles per CTA: warps 0-3 epilogue (both CTAs, each for its own 128 rows), warp 4 MMA issuer (leader CTA only; both
// CTAs allocate and free tensor memory), four producer warps (both CTAs; loads land in the CTA's own shared memory
// but complete on the LEADER's "full" barrier), taking turns on the stages.  One producer thread takes 518 clocks to wait for a
// free slot and issue a stage's two copies (a stage's MMAs: 384 at N = 192) and 2500 to change to the next item's list, and the copies land
// 430 clocks later: the ring never held more than a stage.  Four warps with their entries requested a turn ahead keep it full.
// 1024 rows, 225 points, one producer -> four: layer 64->192 (25 neighbours) 120 -> 106 us, 192->384 240 -> 211, 384->256 273 -> 266,
// 256->256 188 -> 181 (with the MMA loop of a single thread before it: 126, 252, 282, 194).  A stage now takes 520 clocks at N = 256,
// where the MMAs need 512, at the 1.41 GHz that the power limit leaves; what is left is the last round of items (12.2 per pair: 13).
// Barriers: full[s] and acc_empty[a] are used in the leader's shared memory only (the peer's copies and
// epilogue threads signal them through cluster addresses); empty[s] and acc_full[a] exist in both CTAs and
// are signalled by the leader's tcgen05.commit, multicast to both.  No TMA load here is multicast.
// All waits are bounded; both CTAs always reach the closing cluster barrier.
// MASK: an input gradient that leaves behind the ReLU mask of the layer below, with its sums per channel (that layer's bias gradient).  The epilogue has
// the time (54 stages of MMAs per item), where a pass of its own reads the gradient and the activations and writes the gradient again: 280 us for four layers of the
// benchmark's stack at 1024 rows, against 30 more in these launches; the training step under the power limit 3714 -> 3609.  With few stages per item the epilogue is
// what bounds the kernel: the activations of the next 64 columns are read ahead, while the accumulator fills or the columns before are worked on (each read where it
// is used: 2.9 us per 64 columns; ahead: 2.0; 512 <- 64 channels, one neighbour, 1000 points, 256 rows 318 -> 224, where the separate pass takes 233).
#include "tc_common.cuh"

namespace {

struct Tc2Args {
  const int* nbr_idx; const uint16_t* nbr_tap; const int* nbr_cnt;
  const float* bias; void* Y; int* status;
  int kp, B, n_in, n_out, c_out, cp;
  int ct, n_ct, n_mt2, nstage, relu, y_f32, total_items;
  uint32_t stage_bytes, bias_bytes;
  uint32_t wait_limit; int skip_loads;   // as in TcArgs
  const int* out_map; int n_out_y; int accumulate;   // see OutMode
  const __nv_bfloat16* act; float* colsum;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// TMA load whose completion is counted on a barrier that may live in the peer CTA of the pair.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on the barrier at this shared-memory offset in BOTH CTAs once the MMAs issued so far have completed.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// Sums over the warp's 32 lanes (rows) of 64 columns, by halving exchanges: lane l ends with columns l and 32 + l.  62 exchanges, where a tree per column takes 320.
__device__ __forceinline__ float2 column_sums(float (&v)[64], int lane) {
  const bool up16 = lane & 16, up8 = lane & 8, up4 = lane & 4, up2 = lane & 2, up1 = lane & 1;
#pragma unroll
  for (int h = 0; h < 2; ++h) {                                             // columns 32h .. 32h + 31
    float* c = v + 32 * h;
#pragma unroll
    for (int i = 0; i < 16; ++i) c[i] = (up16 ? c[i + 16] : c[i]) + __shfl_xor_sync(0xffffffffu, up16 ? c[i] : c[i + 16], 16);
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = (up8 ? c[i + 8] : c[i]) + __shfl_xor_sync(0xffffffffu, up8 ? c[i] : c[i + 8], 8);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = (up4 ? c[i + 4] : c[i]) + __shfl_xor_sync(0xffffffffu, up4 ? c[i] : c[i + 4], 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) c[i] = (up2 ? c[i + 2] : c[i]) + __shfl_xor_sync(0xffffffffu, up2 ? c[i] : c[i + 2], 2);
    c[0] = (up1 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, up1 ? c[0] : c[1], 1);
  }
  return make_float2(v[0], v[32]);
}

__device__ __forceinline__ void decode_item2(const Tc2Args& a, int item, int& n, int& mt2, int& ctile) {
  ctile = item % a.n_ct;
  const int t = item / a.n_ct;
  n = t % a.n_out;
  mt2 = t / a.n_out;
}

template <bool MASK>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
fovi_knnconv_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Tc2Args a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* basep = smem_raw + (base - raw);
  SmemHeader* hdr = reinterpret_cast<SmemHeader*>(basep);
  float* bias_s = reinterpret_cast<float*>(basep + 1024);
  const uint32_t stages0 = base + 1024u + a.bias_bytes;
  volatile int* abort_flag = &hdr->abort_flag;

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();      // 0 = leader (issues the MMAs), 1 = peer
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int chunks = (a.cp + 63) / 64;   // a last box reaching past cp is zero-filled by the tensor copy
  const int half = a.ct / 2;                    // rows of B this CTA stages

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.nstage; ++s) { mbar_init(smem_u32(&hdr->full[s]), 1); mbar_init(smem_u32(&hdr->empty[s]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&hdr->acc_full[i]), 1); mbar_init(smem_u32(&hdr->acc_empty[i]), 8); }
    mbar_init(smem_u32(&hdr->drain), 1);
    hdr->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {  // both CTAs of the pair allocate together: 512 columns = two accumulators of up to 256
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&hdr->tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  // Programmatic dependent launch: let the next kernel of the stream be scheduled onto SMs as they free up (its
  // prologue then overlaps this kernel's tail), and hold this kernel's own first read of global data until the
  // kernel before it has completed.  Everything above (barriers, tensor memory) needed no global data.  Both are
  // no-ops when the kernel was launched without the attribute.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int i = threadIdx.x; i < a.c_out; i += blockDim.x) bias_s[i] = a.bias ? __ldg(a.bias + i) : 0.f;
  float* sums_s = bias_s + a.bias_bytes / 4 / (MASK ? 5 : 1);               // MASK: [4 epilogue warps][c_out] behind the bias
  if (MASK)
    for (int i = threadIdx.x; i < 4 * a.c_out; i += blockDim.x) sums_s[i] = 0.f;
  tc_fence_before();
  cluster_sync_all();   // barriers of both CTAs are initialised before anyone signals across
  tc_fence_after();
  const uint32_t tmem = hdr->tmem_base;

  if (warp >= 5) {
    // ------------------------------------------------------------ producers (both CTAs): the warps take turns on the stages (see ring.cuh); lane 0
    // copies the activations, lane 1 the weights
    RingTurn ring(warp - 5, a.nstage);
    int item = a.skip_loads || ring.idle ? a.total_items : pair, k = 0, cc = warp - 5, sel = 0;   // this warp's stage: chunk cc of neighbour k
    ItemWalk it(pair, n_pairs, a.n_ct, a.n_out), ahead = it;                        // d0 c_out tile, d1 output point, d2 row tile
    int cnt = item < a.total_items ? __ldg(a.nbr_cnt + it.d1) : 0, cnt_ahead = 0;
    auto look_ahead = [&]() {
      ahead.next();
      if (item + n_pairs < a.total_items) cnt_ahead = __ldg(a.nbr_cnt + ahead.d1);
    };
    look_ahead();
    auto settle = [&]() {   // moves on to an existing stage and requests its neighbour (lane 0) and tap (lane 1)
      while (cc >= chunks) { cc -= chunks; ++k; }
      while (k >= cnt) {
        k -= cnt;
        item += n_pairs;
        if (item >= a.total_items) return;
        it = ahead; cnt = cnt_ahead;
        look_ahead();
      }
      const size_t at = (size_t)it.d1 * a.kp + k;
      if (lane == 0) sel = __ldg(a.nbr_idx + at);
      if (lane == 1) sel = __ldg(a.nbr_tap + at);
    };
    if (item < a.total_items) settle();
    while (item < a.total_items) {
      const uint32_t full_leader = map_to_cta(smem_u32(&hdr->full[ring.s]), 0);
      const uint32_t sa = stages0 + ring.s * a.stage_bytes;
      bool mine = true;
      if (lane == 0) {
        mine = mbar_wait(smem_u32(&hdr->empty[ring.s]), ring.ph ^ 1u, abort_flag, a.status, 11, a.wait_limit);
        if (mine && rank == 0) mbar_expect_tx(smem_u32(&hdr->full[ring.s]), 2u * a.stage_bytes);   // both CTAs' bytes
      }
      if (!__all_sync(0xffffffffu, mine)) break;
      if (lane == 0) tma_load_3d_pair(sa, &tmA, full_leader, cc * 64, sel, (it.d2 * 2 + (int)rank) * BM);            // this CTA's 128 batch rows
      if (lane == 1) tma_load_3d_pair(sa + A_STAGE_BYTES, &tmB, full_leader, cc * 64, it.d0 * a.ct + (int)rank * half, sel);   // half of the c_out tile
      cc += (int)ring.step;
      settle();
      ring.next();
    }
    if (lane == 0 && *abort_flag) {
      // Give copies that are still in flight time to land before this CTA's shared memory goes away.
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only; see elect_one)
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.ct >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint64_t desc0 = smem_desc(0, 16u, 1024u, 2u);
      const uint32_t u_stages0 = warp_uniform(stages0), u_tmem = warp_uniform(tmem);
      uint32_t s = 0, ph = 0, acc = 0, aph = 0;
      bool ok = true;
      int cnt = pair < a.total_items ? __ldg(a.nbr_cnt + (pair / a.n_ct) % a.n_out) : 0;
      for (int item = pair; item < a.total_items && ok; item += n_pairs) {
        const int next = item + n_pairs;
        const int cnt_next = next < a.total_items ? __ldg(a.nbr_cnt + (next / a.n_ct) % a.n_out) : 0;
        const int steps = warp_uniform(cnt) * chunks;
        ok = mbar_wait_warp(smem_u32(&hdr->acc_empty[acc]), aph ^ 1u, abort_flag, a.status, 12, a.wait_limit);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = u_tmem + acc * 256u;
        for (int st = 0; st < steps; ++st) {
          ok = mbar_wait_warp(smem_u32(&hdr->full[s]), ph, abort_flag, a.status, 13, a.wait_limit);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = u_stages0 + s * a.stage_bytes;
          const uint64_t da = desc0 + (sa >> 4), db = desc0 + ((sa + A_STAGE_BYTES) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) tc_mma_bf16_pair(d_tmem, da + kk * 2u, db + kk * 2u, idesc, (st | kk) ? 1u : 0u);
            tc_commit_pair(smem_u32(&hdr->empty[s]));      // frees the stage in both CTAs
            if (st == steps - 1) tc_commit_pair(smem_u32(&hdr->acc_full[acc]));   // accumulator halves complete in both CTAs
          }
          __syncwarp();
          if (++s == (uint32_t)a.nstage) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        if (steps == 0) {                                  // a point without neighbours: nothing to wait for
          if (elect_one()) tc_commit_pair(smem_u32(&hdr->acc_full[acc]));
          __syncwarp();
        }
        if (++acc == 2) { acc = 0; aph ^= 1u; }
        cnt = cnt_next;
      }
      if (*abort_flag && elect_one()) {
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&hdr->drain)) : "memory");
        for (uint32_t it = 0; it < (1u << 20); ++it)
          if (mbar_try_wait(smem_u32(&hdr->drain), 0)) break;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int q = warp & 3;
    uint32_t acc = 0, aph = 0;
    bool ok = true;
    int cnt = pair < a.total_items ? __ldg(a.nbr_cnt + (pair / a.n_ct) % a.n_out) : 0;
    for (int item = pair; item < a.total_items && ok; item += n_pairs) {
      int n, mt2, ctile;
      decode_item2(a, item, n, mt2, ctile);
      const int next = item + n_pairs;
      const int cnt_next = next < a.total_items ? __ldg(a.nbr_cnt + (next / a.n_ct) % a.n_out) : 0;
      const int row = (mt2 * 2 + (int)rank) * BM + q * 32 + lane;
      const int o0 = ctile * a.ct;
      const int n_y = a.out_map ? __ldg(a.out_map + n) : n;
      const size_t y_off = ((size_t)row * a.n_out_y + n_y) * a.c_out + o0;
      uint4 m[8];                           // MASK: activations of the next 64 columns, read while the accumulator fills or the columns before are worked on
      auto fetch = [&](int c0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (row < a.B && c0 + i * 8 < a.ct) m[i] = __ldg(reinterpret_cast<const uint4*>(a.act + y_off + c0) + i);
      };
      if (MASK) fetch(0);
      ok = mbar_wait(smem_u32(&hdr->acc_full[acc]), aph, abort_flag, a.status, 14, a.wait_limit);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + acc * 256u;
      for (int c0 = 0; c0 < a.ct; c0 += 64) {
        uint32_t r[64];
        const int w = min(64, a.ct - c0);   // 32 or 64 (ct is a multiple of 32 here)
        tc_ld32(t_base + c0, r);
        if (w == 64) tc_ld32(t_base + c0 + 32, r + 32);
        tc_ld_wait();
        if (cnt <= 0) {   // a point without neighbours: nothing was accumulated, the columns hold an earlier item's values
#pragma unroll
          for (int i = 0; i < 64; ++i) r[i] = 0u;
        }
        if (MASK) {               // (bf16 results, no bias, no ReLU)
          float v[64];
          uint4 here[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) here[i] = m[i];
          if (c0 + 64 < a.ct) fetch(c0 + 64);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t pk[8];
            if (g * 16 < w && row < a.B) {
              const uint4 m0 = here[2 * g], m1 = here[2 * g + 1];
              const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[g * 16 + 2 * i]), __uint_as_float(r[g * 16 + 2 * i + 1]));
                const uint32_t b = *reinterpret_cast<const uint32_t*>(&h);
                const float y0 = __uint_as_float(mw[i] << 16), y1 = __uint_as_float(mw[i] & 0xFFFF0000u);     // bf16 -> float32, exact
                pk[i] = (y0 > 0.f ? b & 0xFFFFu : 0u) | (y1 > 0.f ? b & 0xFFFF0000u : 0u);
              }
              st_global_32(reinterpret_cast<__nv_bfloat16*>(a.Y) + y_off + c0 + g * 16, pk);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) pk[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) { v[g * 16 + 2 * i] = __uint_as_float(pk[i] << 16); v[g * 16 + 2 * i + 1] = __uint_as_float(pk[i] & 0xFFFF0000u); }
          }
          const float2 s = column_sums(v, lane);
          float* d = sums_s + q * a.c_out + o0 + c0 + lane;                 // this warp's own
          d[0] += s.x;
          if (w == 64) d[32] += s.y;
          continue;
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
            if (row < a.B) {
              if (a.accumulate) {
                float* dst = reinterpret_cast<float*>(a.Y) + y_off + c0 + g * 16;
                if (cnt > 0) {
#pragma unroll
                  for (int i = 0; i < 4; ++i) red_add_f32x4(dst + 4 * i, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
              } else if (a.y_f32) {
                float* dst = reinterpret_cast<float*>(a.Y) + y_off + c0 + g * 16;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  uint32_t w8[8];
#pragma unroll
                  for (int e = 0; e < 8; ++e) w8[e] = __float_as_uint(v[8 * i + e]);
                  st_global_32(dst + 8 * i, w8);
                }
              } else {
                uint32_t pk[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                  pk[i] = *reinterpret_cast<uint32_t*>(&h);
                }
                st_global_32(reinterpret_cast<__nv_bfloat16*>(a.Y) + y_off + c0 + g * 16, pk);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();   // every lane has finished reading the accumulator; one arrival per warp (8 in the pair)
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&hdr->acc_empty[acc]), 0));   // the leader's MMA thread waits for all 8
      if (++acc == 2) { acc = 0; aph ^= 1u; }
      cnt = cnt_next;
    }
    if (MASK) {
      asm volatile("bar.sync 1, 128;" ::: "memory");                        // the four epilogue warps
      for (int c = threadIdx.x; c < a.c_out; c += 128) {
        const float s = sums_s[c] + sums_s[a.c_out + c] + sums_s[2 * a.c_out + c] + sums_s[3 * a.c_out + c];
        if (s != 0.f) atomicAdd(a.colsum + c, s);
      }
    }
  }

  tc_fence_before();
  cluster_sync_all();   // nobody frees tensor memory or leaves while the other CTA may still signal or read
  if (warp == 4) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace

namespace {
// Shared memory of the bias table (and, with a mask, of the warps' channel sums), and how many stages fit beside it.
uint32_t pair_bias_bytes(const fovi_knnconv_plan* p, bool mask) { return (((uint32_t)p->c_out * 4u + 1023u) & ~1023u) * (mask ? 5u : 1u); }
uint32_t pair_stages(const fovi_knnconv_plan* p, bool mask) {
  const uint32_t taken = 2048u + pair_bias_bytes(p, mask), all = 220u * 1024u;
  return taken >= all ? 0u : std::min<uint32_t>(MAX_STAGES, (all - taken) / (A_STAGE_BYTES + (uint32_t)(p->ct / 2) * 128u));
}
bool pair_applies(const fovi_knnconv_plan* p, int B, bool mask) {
  return p->x_layout == FOVI_X_BNC && p->cin_packed >= 16 && p->ct >= 32 && p->ct % 32 == 0 && B > BM && p->kp <= 32 * TBQ && fovi::sm_count() >= 2 &&
         (long long)((B + 2 * BM - 1) / (2 * BM)) * p->n_out * (p->c_out / p->ct) < (1ll << 31) && pair_stages(p, mask) >= 2;
}
}  // namespace

bool fovi::knnconv_tc_pair_masks(const fovi_knnconv_plan* p, int B) { return pair_applies(p, B, true); }

int fovi::launch_knnconv_tc_pair(const fovi_knnconv_plan* p, const void* X, const void* Wt, const float* bias, void* Y, int y_dtype,
                                 int B, int relu, cudaStream_t st, int skip_loads, uint32_t wait_limit, const OutMode& om) {
  const int ct = p->ct, cp = p->cin_packed;
  const bool mask = om.act != nullptr;
  if (!pair_applies(p, B, mask) || (mask && (bias || relu || om.out_map || y_dtype != FOVI_BF16))) return FOVI_ERR_UNSUPPORTED;
  const int sms = fovi::sm_count();
  Tc2Args a;
  a.nbr_idx = p->nbr_idx; a.nbr_tap = p->nbr_tap; a.nbr_cnt = p->nbr_cnt;
  a.bias = bias; a.Y = Y; a.status = p->status;
  a.kp = p->kp; a.B = B; a.n_in = p->n_in; a.n_out = p->n_out; a.c_out = p->c_out; a.cp = cp;
  a.ct = ct; a.n_ct = p->c_out / ct; a.n_mt2 = (B + 2 * BM - 1) / (2 * BM);
  a.relu = relu; a.y_f32 = y_dtype == FOVI_F32;
  a.wait_limit = wait_limit; a.skip_loads = skip_loads;
  a.out_map = om.out_map; a.n_out_y = om.out_map ? om.n_out_y : p->n_out; a.accumulate = om.accumulate;
  a.act = static_cast<const __nv_bfloat16*>(om.act); a.colsum = om.colsum;
  const long long items = (long long)a.n_mt2 * p->n_out * a.n_ct;
  a.total_items = (int)items;
  a.stage_bytes = A_STAGE_BYTES + (uint32_t)(ct / 2) * 128u;
  a.bias_bytes = pair_bias_bytes(p, mask);
  a.nstage = (int)pair_stages(p, mask);
  const size_t smem = 1024 + 1024 + a.bias_bytes + (size_t)a.nstage * a.stage_bytes;

  CUtensorMap tmA, tmB;
  int rc = fovi::encode_3d(&tmA, X, (uint64_t)cp, (uint64_t)p->n_in, (uint64_t)B, (uint64_t)cp * 2, (uint64_t)p->n_in * cp * 2, 64, 1, BM, true);
  if (rc) return rc;
  rc = fovi::encode_3d(&tmB, Wt, (uint64_t)cp, (uint64_t)p->c_out, (uint64_t)p->V, (uint64_t)cp * 2, (uint64_t)p->c_out * cp * 2, 64, (uint32_t)(ct / 2), 1, true);
  if (rc) return rc;

  auto k = mask ? fovi_knnconv_tc_pair_kernel<true> : fovi_knnconv_tc_pair_kernel<false>;
  FOVI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int pairs = (int)std::min<long long>(items, sms / 2);
  FOVI_CUDA(fovi::launch_pdl(k, 2 * pairs, TC_THREADS, smem, st, tmA, tmB, a));   // cluster size 2 comes from __cluster_dims__
  return fovi::after_launch("fovi_knnconv_tc_pair_kernel");
}
