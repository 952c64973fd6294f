// Weight gradient of KNNConv on the tensor cores, read straight from the activations' own layouts.
//
//   dW[v][o][c] = sum over the pairs (n, m) that use filter tap v, sum over the batch b of  gY[b, n, o] * X[b, m, c]
//
// The contraction runs over the batch, so both operands have their OUTER index contiguous (channels-last activations [b][point][channel]):
// MN-major operands in the tensor core's terms.  A tensor-copy box of 64 channels x one point x 64 batch rows lands as 64 rows of 128 bytes,
// which with the 128-byte swizzle is exactly the MN-major layout (64-channel blocks 8 KB apart, groups of 8 batch rows 1 KB apart), so no operand
// is transposed, packed or gathered in memory first (the K-major formulation had to write batch-innermost copies of every activation and
// gradient: 933 of 5280 us of the 5-layer training step at 1024 rows, and a gathered copy of the input plus per-point products for the first layer: 640 us).
//
// Two modes share the kernel:
//   channels   a work item is one part of a tap's pair list x one tile of P's channels x one tile of Q's channels; P and Q are gY and X in either
//              role.  A stage is 64 batch rows of one pair.  Result tiles are ADDED into out[v][p channel][q channel] (float32 reductions in L2).
//   pair       (c_in <= 4) X is in the pair layout of knnconv_tc.cu: a (pair, 64 rows) block is 64 x 16 bytes = MN-major core matrices of 8 columns
//              (2 points x 4 channels).  A work item is one output point x 128 channels of gY x up to 32 slots of the point's list (256 columns);
//              a stage is 64 batch rows; the four channel sums of a listed point leave as one 16-byte store per lane, 512 contiguous bytes per warp,
//              into a workspace with a place for every (output point, listed point).  A second kernel adds each tap's places in the order of the output
//              points: the result is the same bits every time (sums of the channels mode are float32 reductions in no fixed order).
// CG = 2: cluster of two CTAs, M = 256 (P channels), each CTA stages its half of Q's tile.  CG = 1: M = 128.
// Roles: warps 0-3 epilogue, warp 4 MMA issuer, the rest producers (see knnconv_tc2.cu).  All waits are bounded.
#include "tc_common.cuh"

#include <mutex>
#include <vector>

struct fovi_knndw_plan {
  int n_groups = 0, kp = 0, V = 0, n_p = 0, n_q = 0;
  int* p_pt = nullptr;    // [n_groups, kp] points of operand P
  int* q_pt = nullptr;    // [n_groups, kp] points of operand Q
  int* cnt = nullptr;     // [n_groups]
  int* tap = nullptr;     // [n_groups] result row
  int* status = nullptr;
};

namespace {

constexpr int DW_ROWS = 64;                 // batch rows per stage (K)
constexpr uint32_t DW_BOX = 8192;           // 64 channels x 64 rows

struct DwArgs {
  const int* p_pt; const int* q_pt; const int* cnt; const int* tap;                     // channels mode
  const int* slot_pair; const uint16_t* slot_box; const uint16_t* slot_tap;             // pair mode (cnt: slots per point)
  float* out; int* status;                                                              // pair mode: out is the workspace
  int n0;                                                                               // pair mode: first output point of this launch
  int kp, chunks, cp, cq, ct, n_mt, n_nt, total, nstage;   // ct: columns of a Q tile (pair mode: 8 per slot)
  uint32_t stage_bytes, wait_limit;
  int skip_loads;   // self-test: the producers withhold every copy, so the first consumer wait must give up
};

struct DwMaps { CUtensorMap p, q[4]; };     // q[0] in channels mode; boxes of 2^i pairs in pair mode

struct DwHeader {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t dw_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t dw_map(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
template <int CG> __device__ __forceinline__ void dw_sync_all() {
  if (CG == 2) asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
  else __syncthreads();
}
template <int CG> __device__ __forceinline__ void dw_load3(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  if (CG == 2)
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
  else
    tma_load_3d(dst, map, bar, c0, c1, c2);
}
__device__ __forceinline__ void dw_load4(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
template <int CG> __device__ __forceinline__ void dw_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  if (CG == 2)
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
  else
    tc_mma_bf16(d, a, b, idesc, accumulate);
}
template <int CG> __device__ __forceinline__ void dw_commit(uint32_t bar) {
  if (CG == 2)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
  else
    tc_commit(bar);
}

template <int CG, bool PAIRS>
__device__ __forceinline__ void dw_body(const DwMaps& maps, const DwArgs& a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  DwHeader* hdr = reinterpret_cast<DwHeader*>(smem_raw + (base - raw));
  const uint32_t stages0 = base + 1024u;                                 // per stage: P [2][64 rows][128 B], then Q
  volatile int* abort_flag = &hdr->abort_flag;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = CG == 2 ? (int)dw_rank() : 0;
  const int worker = blockIdx.x / CG, workers = gridDim.x / CG;
  const int half = a.ct / CG;                                            // columns of Q's tile this CTA stages (channels mode)

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.nstage; ++s) { mbar_init(smem_u32(&hdr->full[s]), 1); mbar_init(smem_u32(&hdr->empty[s]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&hdr->acc_full[i]), 1); mbar_init(smem_u32(&hdr->acc_empty[i]), 4 * CG); }
    mbar_init(smem_u32(&hdr->drain), 1);
    hdr->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    if (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&hdr->tmem_base)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&hdr->tmem_base)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // see fovi_knnconv_tc_kernel
  asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before();
  dw_sync_all<CG>();
  tc_fence_after();
  const uint32_t tmem = hdr->tmem_base;
  const ItemWalk start(worker, workers, a.n_nt, a.n_mt);            // d0 tile of Q, d1 tile of P, d2 group (channels) / output point (pair)

  if (warp >= 5) {
    // ------------------------------------------------------------ producers: the warps take turns on the stages (see ring.cuh)
    RingTurn ring(warp - 5, a.nstage);
    int item = a.skip_loads || ring.idle ? a.total : worker, cc = warp - 5, k = 0;   // this warp's stage: row chunk cc of pair k (pair mode: k stays 0)
    ItemWalk it = start, ahead = start;
    int cnt = item < a.total ? (PAIRS ? 1 : __ldg(a.cnt + it.d2)) : 0, cnt_ahead = 0;
    auto look_ahead = [&]() {
      ahead.next();
      if (item + workers < a.total) cnt_ahead = PAIRS ? 1 : __ldg(a.cnt + ahead.d2);
    };
    look_ahead();
    int sel = 0, slots = 0, seen = -1;
    uint32_t box = 0;
    // moves on to an existing stage and requests what it needs: the pair's points (lanes 0-1: P, others: Q), or this lane's slot of the list
    auto settle = [&]() {
      while (cc >= a.chunks) { cc -= a.chunks; ++k; }
      while (k >= cnt) {
        k -= cnt;
        item += workers;
        if (item >= a.total) return;
        it = ahead; cnt = cnt_ahead;
        look_ahead();
      }
      if (PAIRS) {
        if (seen != item) {
          seen = item;
          const int ts = a.ct / 8, s0 = it.d0 * ts + lane;
          slots = min(ts, (__ldg(a.cnt + it.d2) + 7) / 8 * 8 - it.d0 * ts);      // <= 0: nothing of the list in this tile
          box = 0;
          if (lane < slots) {
            sel = __ldg(a.slot_pair + (size_t)it.d2 * a.kp + s0);
            box = __ldg(a.slot_box + (size_t)it.d2 * a.kp + s0);
          }
        }
      } else {
        sel = __ldg((lane < 2 ? a.p_pt : a.q_pt) + (size_t)it.d2 * a.kp + k);
      }
    };
    if (item < a.total) settle();
    while (item < a.total) {
      const uint32_t full = CG == 2 ? dw_map(smem_u32(&hdr->full[ring.s]), 0) : smem_u32(&hdr->full[ring.s]);
      const uint32_t sa = stages0 + ring.s * a.stage_bytes, sb = sa + 2u * DW_BOX;
      const int m0 = it.d1 * (128 * CG) + rank * 128;                                     // first P channel of this CTA
      // boxes wholly past the channels are not loaded: their rows / columns are never stored
      const int pb = min(2, max(0, (a.cp - m0 + 63) / 64));
      const int q0 = PAIRS ? 0 : it.d0 * a.ct + rank * half;
      const int qb = PAIRS ? 0 : min((half + 63) / 64, max(0, (a.cq - q0 + 63) / 64));
      bool mine = true;
      if (lane == 0) {
        mine = mbar_wait(smem_u32(&hdr->empty[ring.s]), ring.ph ^ 1u, abort_flag, a.status, 31, a.wait_limit);
        if (mine) {
          uint32_t bytes = (uint32_t)pb * DW_BOX + (PAIRS ? (uint32_t)max(slots, 0) * 1024u : (uint32_t)qb * DW_BOX);
          if (CG == 2) {                     // the leader arms for both CTAs
            const int m1 = it.d1 * 256 + 128, q1 = it.d0 * a.ct + half;
            bytes += (uint32_t)min(2, max(0, (a.cp - m1 + 63) / 64)) * DW_BOX + (uint32_t)min((half + 63) / 64, max(0, (a.cq - q1 + 63) / 64)) * DW_BOX;
          }
          if (rank == 0) mbar_expect_tx(smem_u32(&hdr->full[ring.s]), bytes);
        }
      }
      if (!__all_sync(0xffffffffu, mine)) break;
      if (PAIRS) {
        if (box) dw_load4(sb + lane * 1024u, &maps.q[box - 1], full, 0, (cc & 1) * 2, sel, cc >> 1);
        if (lane < pb) dw_load3<CG>(sa + lane * DW_BOX, &maps.p, full, m0 + lane * 64, a.n0 + it.d2, cc * DW_ROWS);
      } else {
        if (lane < pb) dw_load3<CG>(sa + lane * DW_BOX, &maps.p, full, m0 + lane * 64, sel, cc * DW_ROWS);
        else if (lane >= 2 && lane - 2 < qb) dw_load3<CG>(sb + (lane - 2) * DW_BOX, &maps.q[0], full, q0 + (lane - 2) * 64, sel, cc * DW_ROWS);
      }
      cc += (int)ring.step;
      settle();
      ring.next();
    }
    if (lane == 0 && *abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(1000);    // copies in flight land before this CTA's shared memory goes away
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------ MMA issuer (see elect_one)
    if (rank == 0) {
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(128 * CG >> 4) << 24);   // both operands MN-major
      const uint64_t desc_p = smem_desc(0, DW_BOX, 1024u, 2u), desc_q = PAIRS ? smem_desc(0, 128u, 1024u, 0u) : desc_p;
      const uint32_t step_q = PAIRS ? 16u : 128u;                    // 16 batch rows further, in 16-byte units
      const uint32_t u_stages0 = warp_uniform(stages0), u_tmem = warp_uniform(tmem);
      uint32_t s = 0, ph = 0, acc = 0, aph = 0;
      bool ok = true;
      ItemWalk it = start;
      for (int item = worker; item < a.total && ok; item += workers, it.next()) {
        const int cnt = warp_uniform(__ldg(a.cnt + it.d2));
        const int steps = PAIRS ? a.chunks : cnt * a.chunks;
        const int cols = PAIRS ? min(a.ct, max((cnt + 7) / 8 * 64 - it.d0 * a.ct, 64)) : a.ct;
        const uint32_t idesc = idesc0 | ((uint32_t)(cols >> 3) << 17);
        ok = mbar_wait_warp(smem_u32(&hdr->acc_empty[acc]), aph ^ 1u, abort_flag, a.status, 32, a.wait_limit);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = u_tmem + acc * 256u;
        for (int st = 0; st < steps; ++st) {
          ok = mbar_wait_warp(smem_u32(&hdr->full[s]), ph, abort_flag, a.status, 33, a.wait_limit);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = u_stages0 + s * a.stage_bytes;
          const uint64_t dp = desc_p + (sa >> 4), dq = desc_q + ((sa + 2u * DW_BOX) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) dw_mma<CG>(d_tmem, dp + kk * 128u, dq + kk * step_q, idesc, (st | kk) ? 1u : 0u);
            dw_commit<CG>(smem_u32(&hdr->empty[s]));
            if (st == steps - 1) dw_commit<CG>(smem_u32(&hdr->acc_full[acc]));
          }
          __syncwarp();
          if (++s == (uint32_t)a.nstage) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        if (steps == 0) {
          if (elect_one()) dw_commit<CG>(smem_u32(&hdr->acc_full[acc]));
          __syncwarp();
        }
        if (++acc == 2) { acc = 0; aph ^= 1u; }
      }
      if (*abort_flag && elect_one()) {
        if (CG == 2) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&hdr->drain)) : "memory");
        else tc_commit(smem_u32(&hdr->drain));
        for (uint32_t i = 0; i < (1u << 20); ++i)
          if (mbar_try_wait(smem_u32(&hdr->drain), 0)) break;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: add the tile into the result (pair mode: store it)
    const int q = warp & 3;
    uint32_t acc = 0, aph = 0;
    ItemWalk it = start;
    for (int item = worker; item < a.total; item += workers, it.next()) {
      const int cnt = __ldg(a.cnt + it.d2);
      const bool ok = mbar_wait_warp(smem_u32(&hdr->acc_full[acc]), aph, abort_flag, a.status, 34, a.wait_limit);
      if (!ok) break;
      tc_fence_after();
      const int row = it.d1 * (128 * CG) + rank * 128 + q * 32 + lane;                    // P channel
      const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + acc * 256u;
      if (PAIRS) {
        const int ts = a.ct / 8, slots = min(ts, cnt - it.d0 * ts);
        const size_t place = ((size_t)it.d2 * a.kp + it.d0 * ts) * 2;                      // of the tile's first slot
        const uint16_t* taps = a.slot_tap + place;
        for (int s0 = 0; s0 < slots; s0 += 4) {                                           // four slots = 32 columns
          uint32_t r[32];
          tc_ld32(t_base + s0 * 8, r);
          tc_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (s0 + (j >> 1) < slots) {
              const uint32_t t = __ldg(taps + s0 * 2 + j);
              if (t != 0xFFFFu && row < a.cp)
                reinterpret_cast<uint4*>(a.out)[(place + s0 * 2 + j) * a.cp + row] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
          }
        }
      } else if (cnt > 0) {
        const int c_base = it.d0 * a.ct;
        float* dst = a.out + ((size_t)__ldg(a.tap + it.d2) * a.cp + row) * a.cq + c_base;
        const int cols = min(a.ct, a.cq - c_base);                                        // a multiple of 8
        for (int c0 = 0; c0 < cols; c0 += 32) {
          uint32_t r[32];
          tc_ld32(t_base + c0, r);
          tc_ld_wait();
          if (row < a.cp) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (c0 + 4 * j < cols)
                red_add_f32x4(dst + c0 + 4 * j, __uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) {
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(dw_map(smem_u32(&hdr->acc_empty[acc]), 0)) : "memory");
        } else {
          mbar_arrive(smem_u32(&hdr->acc_empty[acc]));
        }
      }
      if (++acc == 2) { acc = 0; aph ^= 1u; }
    }
  }

  tc_fence_before();
  dw_sync_all<CG>();
  if (warp == 4) {
    __syncwarp();
    tc_fence_after();
    if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
fovi_knnconv_dw2_kernel(const __grid_constant__ DwMaps maps, const DwArgs a) { dw_body<2, false>(maps, a); }
__global__ void __launch_bounds__(TC_THREADS, 1)
fovi_knnconv_dw1_kernel(const __grid_constant__ DwMaps maps, const DwArgs a) { dw_body<1, false>(maps, a); }
__global__ void __launch_bounds__(TC_THREADS, 1)
fovi_knnconv_dw_pairs_kernel(const __grid_constant__ DwMaps maps, const DwArgs a) { dw_body<1, true>(maps, a); }

// out[v][o] += the places of tap v between `lo` and `hi` (of the whole layer's (output point, slot, half) places; the workspace starts at `lo`), in
// ascending order: warp w adds every W-th place, the warps' sums are added in the order of the warps.  Bound by writing and reading the workspace.  Both
// kernels, 1024 rows, against float32 reductions in no order: 3 -> 64 onto 1023 points 165 us / 132, 3 -> 384 onto 63 tokens 54 / 44, 3 -> 1280 128 / 95.
template <int TS_WARPS>
__global__ void __launch_bounds__(TS_WARPS * 32) fovi_tap_sum_kernel(const float4* __restrict__ work, const int* __restrict__ seg_start,
                                                                     const int* __restrict__ seg_place, int lo, int hi, int c_out, float4* __restrict__ out) {
  __shared__ float4 part[TS_WARPS][32];
  const int v = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, o = blockIdx.y * 32 + lane;
  const int i0 = __ldg(seg_start + v), i1 = __ldg(seg_start + v + 1);
  auto first_from = [&](int place) {      // first index in [i0, i1) whose place is not below `place`
    int a = i0, b = i1;
    while (a < b) {
      const int m = (a + b) >> 1;
      if (__ldg(seg_place + m) < place) a = m + 1; else b = m;
    }
    return a;
  };
  // (the whole list unless the layer is done in parts)
  const int from = i0 < i1 && __ldg(seg_place + i0) < lo ? first_from(lo) : i0, to = i0 < i1 && __ldg(seg_place + i1 - 1) >= hi ? first_from(hi) : i1;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (o < c_out) {
#pragma unroll 8
    for (int i = from + warp; i < to; i += TS_WARPS) {
      const float4 x = __ldg(work + (size_t)(__ldg(seg_place + i) - lo) * c_out + o);
      s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
    }
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && o < c_out) {
    float4* d = out + (size_t)v * c_out + o;
    float4 t = *d;
#pragma unroll
    for (int w = 0; w < TS_WARPS; ++w) { t.x += part[w][lane].x; t.y += part[w][lane].y; t.z += part[w][lane].z; t.w += part[w][lane].w; }
    *d = t;
  }
}

// The places of every tap, ascending: built from the plan's slot table by the first weight gradient (inference never needs them).
int tap_places(fovi_knnconv_plan* p) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (p->seg_start) return FOVI_OK;
  const size_t n = (size_t)p->n_out * p->sp * 2;
  if (n >= (1ull << 31)) return FOVI_ERR_UNSUPPORTED;
  std::vector<uint16_t> tap(n);
  FOVI_CUDA(cudaMemcpy(tap.data(), p->pair_tap, n * sizeof(uint16_t), cudaMemcpyDeviceToHost));
  std::vector<int> start((size_t)p->V + 1, 0), place;
  for (size_t i = 0; i < n; ++i)
    if (tap[i] != 0xFFFF) ++start[(size_t)tap[i] + 1];
  for (int v = 0; v < p->V; ++v) start[v + 1] += start[v];
  place.resize(std::max<size_t>(1, start[p->V]));
  std::vector<int> at(start.begin(), start.end() - 1);
  for (size_t i = 0; i < n; ++i)
    if (tap[i] != 0xFFFF) place[at[tap[i]]++] = (int)i;
  int *d_start = nullptr, *d_place = nullptr;
  cudaError_t e = cudaMalloc(&d_start, start.size() * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&d_place, place.size() * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(d_place, place.data(), place.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d_start, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    if (d_start) cudaFree(d_start);
    if (d_place) cudaFree(d_place);
    return fovi::cuda_fail(e, "fovi_knnconv_weight_grad_pairs");
  }
  p->seg_place = d_place;
  p->seg_start = d_start;
  return FOVI_OK;
}

int64_t place_bytes(const fovi_knnconv_plan* p) { return (int64_t)p->sp * 2 * p->c_out * 16; }    // workspace of one output point

int dw_launch(int cg, bool pairs, DwMaps& maps, DwArgs& a, cudaStream_t st) {
  const uint32_t budget = 224u * 1024u - 2048u;
  a.nstage = (int)std::min<uint32_t>(MAX_STAGES, budget / a.stage_bytes);
  const size_t smem = 2048 + (size_t)a.nstage * a.stage_bytes;
  const int grid = cg * (int)std::min<long long>(a.total, fovi::sm_count() / cg);
  if (pairs) {
    FOVI_CUDA(cudaFuncSetAttribute(fovi_knnconv_dw_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    FOVI_CUDA(fovi::launch_pdl(fovi_knnconv_dw_pairs_kernel, grid, TC_THREADS, smem, st, maps, a));
  } else if (cg == 2) {
    FOVI_CUDA(cudaFuncSetAttribute(fovi_knnconv_dw2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    FOVI_CUDA(fovi::launch_pdl(fovi_knnconv_dw2_kernel, grid, TC_THREADS, smem, st, maps, a));
  } else {
    FOVI_CUDA(cudaFuncSetAttribute(fovi_knnconv_dw1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    FOVI_CUDA(fovi::launch_pdl(fovi_knnconv_dw1_kernel, grid, TC_THREADS, smem, st, maps, a));
  }
  return fovi::after_launch("fovi_knnconv_dw_kernel");
}

}  // namespace

extern "C" int fovi_knndw_plan_create(const int32_t* p_pt, const int32_t* q_pt, const int32_t* cnt, const int32_t* tap, int n_groups, int kp, int V,
                                      int n_p, int n_q, fovi_knndw_plan** out) {
  if (!p_pt || !q_pt || !cnt || !tap || !out || n_groups <= 0 || kp <= 0 || V <= 0 || n_p <= 0 || n_q <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  for (int g = 0; g < n_groups; ++g) {
    if (cnt[g] < 0 || cnt[g] > kp || tap[g] < 0 || tap[g] >= V) return FOVI_ERR_TABLE_RANGE;
    for (int k = 0; k < cnt[g]; ++k) {
      const int p = p_pt[(size_t)g * kp + k], q = q_pt[(size_t)g * kp + k];
      if (p < 0 || p >= n_p || q < 0 || q >= n_q) return FOVI_ERR_TABLE_RANGE;
    }
  }
  auto* d = new fovi_knndw_plan();
  d->n_groups = n_groups; d->kp = kp; d->V = V; d->n_p = n_p; d->n_q = n_q;
  const size_t lists = sizeof(int) * (size_t)n_groups * kp, words = sizeof(int) * (size_t)n_groups;
  cudaError_t e = cudaMalloc(&d->p_pt, lists);
  if (e == cudaSuccess) e = cudaMalloc(&d->q_pt, lists);
  if (e == cudaSuccess) e = cudaMalloc(&d->cnt, words);
  if (e == cudaSuccess) e = cudaMalloc(&d->tap, words);
  if (e == cudaSuccess) e = cudaMalloc(&d->status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(d->p_pt, p_pt, lists, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d->q_pt, q_pt, lists, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d->cnt, cnt, words, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d->tap, tap, words, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(d->status, 0, sizeof(int));
  if (e != cudaSuccess) {
    fovi_knndw_plan_destroy(d);
    return fovi::cuda_fail(e, "fovi_knndw_plan_create");
  }
  *out = d;
  return FOVI_OK;
}

extern "C" void fovi_knndw_plan_destroy(fovi_knndw_plan* d) {
  if (!d) return;
  if (d->p_pt) cudaFree(d->p_pt);
  if (d->q_pt) cudaFree(d->q_pt);
  if (d->cnt) cudaFree(d->cnt);
  if (d->tap) cudaFree(d->tap);
  if (d->status) cudaFree(d->status);
  delete d;
}

extern "C" int fovi_knndw_check(fovi_knndw_plan* d, void* stream) {
  if (!d) return FOVI_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int h = 0;
  FOVI_CUDA(cudaMemcpyAsync(&h, d->status, sizeof(int), cudaMemcpyDeviceToHost, st));
  FOVI_CUDA(cudaStreamSynchronize(st));
  if (h != 0) {
    FOVI_CUDA(cudaMemsetAsync(d->status, 0, sizeof(int), st));
    FOVI_CUDA(cudaStreamSynchronize(st));
    fovi::g_last_cuda_error = "weight-gradient kernel gave up on wait site " + std::to_string(h);
    return FOVI_ERR_DEVICE_TIMEOUT;
  }
  return FOVI_OK;
}

static int knndw_run_impl(fovi_knndw_plan* d, const void* P, int cp, const void* Q, int cq, int B, float* out, void* stream, int skip_loads,
                          uint32_t wait_limit) {
  if (!d || B < 0 || cp <= 0 || cq <= 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (B == 0) return FOVI_OK;
  if (!P || !Q || !out) return FOVI_ERR_INVALID_ARGUMENT;
  if (cp % 8 || cq % 8) return FOVI_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(P) | reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(out)) & 15) return FOVI_ERR_ALIGNMENT;
  DwArgs a;
  memset(&a, 0, sizeof(a));
  a.p_pt = d->p_pt; a.q_pt = d->q_pt; a.cnt = d->cnt; a.tap = d->tap; a.out = out; a.status = d->status;
  a.kp = d->kp; a.chunks = (B + DW_ROWS - 1) / DW_ROWS; a.cp = cp; a.cq = cq; a.wait_limit = wait_limit; a.skip_loads = skip_loads;
  // CTA pairs (half of Q's bytes per SM) unless one 128-channel tile covers P, where half of every M = 256 MMA would be idle.
  const int cg = cp > 128 ? 2 : 1;
  // Q's tile: the fewest tiles of at most 256 columns, equal, in whole 32s (a load brings 64 channels: what it brings past a tile is not used)
  const int n_nt = (cq + 255) / 256;
  a.ct = ((cq + n_nt - 1) / n_nt + 31) / 32 * 32;
  a.n_nt = (cq + a.ct - 1) / a.ct; a.n_mt = (cp + 128 * cg - 1) / (128 * cg);
  const long long total = (long long)d->n_groups * a.n_nt * a.n_mt;
  if (total >= (1ll << 30)) return FOVI_ERR_UNSUPPORTED;
  a.total = (int)total;
  a.stage_bytes = 2u * DW_BOX + (uint32_t)((a.ct / cg + 63) / 64) * DW_BOX;
  DwMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc = fovi::encode_3d(&maps.p, P, (uint64_t)cp, (uint64_t)d->n_p, (uint64_t)B, (uint64_t)cp * 2, (uint64_t)d->n_p * cp * 2, 64, 1, DW_ROWS, true);
  if (rc) return rc;
  rc = fovi::encode_3d(&maps.q[0], Q, (uint64_t)cq, (uint64_t)d->n_q, (uint64_t)B, (uint64_t)cq * 2, (uint64_t)d->n_q * cq * 2, 64, 1, DW_ROWS, true);
  if (rc) return rc;
  return dw_launch(cg, false, maps, a, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int fovi_knndw_run(fovi_knndw_plan* d, const void* P, int cp, const void* Q, int cq, int B, float* out, void* stream) {
  return knndw_run_impl(d, P, cp, Q, cq, B, out, stream, 0, WAIT_LIMIT);
}

extern "C" int fovi_knndw_selftest_wait_timeout(fovi_knndw_plan* d, const void* P, int cp, const void* Q, int cq, int B, float* out, void* stream) {
  return knndw_run_impl(d, P, cp, Q, cq, B, out, stream, 1, 4096u);     // as fovi_knnconv_selftest_wait_timeout
}

extern "C" int64_t fovi_knnconv_weight_grad_workspace_bytes(const fovi_knnconv_plan* p) {
  if (!p || p->x_layout != FOVI_X_PAIRS) return -1;
  const int64_t one = place_bytes(p);      // (in two parts of 128 MB the first of those layers takes 185 us)
  return std::min<int64_t>(one * p->n_out, std::max<int64_t>(one, 256ll << 20));
}

static int weight_grad_pairs_impl(fovi_knnconv_plan* p, const void* gY, const void* X, int B, void* work, int64_t work_bytes, float* out, void* stream,
                                  int skip_loads, uint32_t wait_limit) {
  if (!p || B < 0) return FOVI_ERR_INVALID_ARGUMENT;
  if (B == 0) return FOVI_OK;
  if (!gY || !X || !work || !out) return FOVI_ERR_INVALID_ARGUMENT;
  if (p->x_layout != FOVI_X_PAIRS || p->c_out % 8) return FOVI_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(gY) | reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(work) | reinterpret_cast<uintptr_t>(out)) & 15)
    return FOVI_ERR_ALIGNMENT;
  const int64_t fit = std::min<int64_t>(p->n_out, work_bytes / place_bytes(p));              // output points
  if (fit < 1) return FOVI_ERR_INVALID_ARGUMENT;
  const int64_t launches = (p->n_out + fit - 1) / fit;
  const int per_launch = (int)((p->n_out + launches - 1) / launches);                         // in equal parts
  int rc = tap_places(p);
  if (rc) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  DwArgs a;
  memset(&a, 0, sizeof(a));
  a.out = static_cast<float*>(work); a.status = p->status;
  a.kp = p->sp; a.chunks = (B + DW_ROWS - 1) / DW_ROWS; a.cp = p->c_out; a.cq = 0; a.wait_limit = wait_limit; a.skip_loads = skip_loads;
  a.n_mt = (p->c_out + 127) / 128; a.n_nt = (p->sp + 31) / 32;
  a.ct = (p->sp / 8 + a.n_nt - 1) / a.n_nt * 64;           // equal tiles of at most 32 slots, in whole 8s
  if ((long long)per_launch * a.n_nt * a.n_mt >= (1ll << 30)) return FOVI_ERR_UNSUPPORTED;
  a.stage_bytes = 2u * DW_BOX + (uint32_t)a.ct * 128u;
  DwMaps maps;
  memset(&maps, 0, sizeof(maps));
  const uint64_t c = (uint64_t)p->c_out, n = (uint64_t)p->n_out, n_pairs = (uint64_t)p->n_pairs;
  rc = fovi::encode_3d(&maps.p, gY, c, n, (uint64_t)B, c * 2, n * c * 2, 64, 1, DW_ROWS, true);
  if (rc) return rc;
  for (int i = 0; i < 4; ++i) {
    const uint64_t dims[4] = {256, 4, n_pairs, (uint64_t)(B + BM - 1) / BM}, strides[3] = {512, 2048, n_pairs * 2048};
    const uint32_t box[4] = {256, 2, 1u << i, 1};
    rc = fovi::encode_4d(&maps.q[i], X, dims, strides, box);
    if (rc) return rc;
  }
  for (a.n0 = 0; a.n0 < p->n_out; a.n0 += per_launch) {
    const int points = std::min(per_launch, p->n_out - a.n0);
    const size_t first = (size_t)a.n0 * p->sp;
    a.slot_pair = p->pair_idx + first; a.slot_box = p->pair_box + first; a.slot_tap = p->pair_tap + 2 * first; a.cnt = p->pair_cnt + a.n0;
    a.total = points * a.n_nt * a.n_mt;
    rc = dw_launch(1, true, maps, a, st);
    if (rc) return rc;
    const dim3 grid(p->V, (p->c_out + 31) / 32);
    const int lo = (int)(2 * first), hi = lo + points * p->sp * 2;
    // about eight places per warp (26 per tap, 1280 channels: sixteen warps 148 us in all, four 128; 243 per tap, 64 channels: sixteen)
    const int64_t per_tap = p->nnz / p->V;
    auto k = per_tap >= 128 ? fovi_tap_sum_kernel<16> : per_tap >= 32 ? fovi_tap_sum_kernel<8> : fovi_tap_sum_kernel<4>;
    k<<<grid, (per_tap >= 128 ? 16 : per_tap >= 32 ? 8 : 4) * 32, 0, st>>>(static_cast<const float4*>(work), p->seg_start, p->seg_place, lo, hi, p->c_out,
                                                                           reinterpret_cast<float4*>(out));
    rc = fovi::after_launch("fovi_tap_sum_kernel");
    if (rc) return rc;
  }
  return FOVI_OK;
}

extern "C" int fovi_knnconv_weight_grad_pairs(fovi_knnconv_plan* p, const void* gY, const void* X, int B, void* work, int64_t work_bytes, float* out,
                                              void* stream) {
  return weight_grad_pairs_impl(p, gY, X, B, work, work_bytes, out, stream, 0, WAIT_LIMIT);
}

extern "C" int fovi_knnconv_weight_grad_pairs_selftest_wait_timeout(fovi_knnconv_plan* p, const void* gY, const void* X, int B, void* work,
                                                                    int64_t work_bytes, float* out, void* stream) {
  return weight_grad_pairs_impl(p, gY, X, B, work, work_bytes, out, stream, 1, 4096u);
}
