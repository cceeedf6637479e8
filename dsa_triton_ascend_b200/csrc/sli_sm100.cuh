// Indexer KL losses on tcgen05 tensor cores: the scoring passes and the gradient pass of sli_grad.cuh
// (same math, same buffers) for the shapes that training uses.
//
//   sli_score_sm100_kernel   p[k] (attention heads that share one key head) or I[k] (index heads) of a
//                            query row's gathered keys: KEYS on the 128 lanes, heads on the columns, so
//                            that the sum over heads is a thread's own.
//   sli_mha_sm100_kernel     p of the dense operator when every query head has its own key head: plain
//                            128 rows x 128 keys tiles, the heads walked over with p in registers.
//   sli_grad_sm100_kernel    dW, dQI and the scattered dKI of a query row (D_idx = 128).
//
// All waits are bounded; one that gives up sets the status word.
#pragma once

#include "sfa_bwd_sm100.cuh"
#include "sli_grad.cuh"

namespace dsa {

constexpr int kSlKeys = 128;                       // keys per tile (the lanes)
constexpr uint32_t kSlKBlk = kSlKeys * 128;        // 128 keys x 64 features
constexpr uint32_t kSlSmemMax = 232448;

// ---- scores --------------------------------------------------------------------------------------
// What bounds it: the hand-overs between gather, issuers and epilogue (512 rows x 2048 keys x 64 heads: 150 us; with a
// quarter of the products and no global reads still 117).  A row's selected keys are its own, so each (row, key) pair
// is a gather of 2 (D + Dr) bytes; cp.async copies of 8 warps bring 58 B/clk of them to an SM that does nothing else,
// TMA gather4 31 (one 512-byte load per 16.5 cycles).  A block takes up to 128 heads of the row (every gathered byte serves all of them), Q stays
// in shared memory and the keys stream through a ring of 64-feature blocks (16 KB each: a whole tile of 147 KB would
// not fit beside 128 heads of Q).  Rows are cut into parts when there are few of them.
// With gather4 and one issuer, and with the copies and two (attention / index side): 512 rows x 64 heads 191 / 67 us
// -> 150 / 56.  2048 rows x 128 heads, fp16, in calls back to back: 838 / 252 of a call of 1721 -> 705 / 209 of 1605;
// the gradient kernel behind them, the same code, takes 590 -> 629 there, at the lower clock that the power cap leaves
// (602 and 603 in single calls).  Rows of one tile gain nothing: 1234 rows of 64 keys 58.4 / 19.3 -> 59.8 / 19.9.
// Warps: 0..7 epilogue (two groups on alternate accumulators), 8..15 gather, 16, 17 MMA issuers, 18 Q and head
// parameters.
constexpr int kScThreads = 608, kScGatherWarp0 = 8, kScGatherWarps = 8, kScIssuer = 16, kScLoader = 18;
constexpr int kScMaxStages = 12;

struct SliScoreArgs {
  SliGradDev p;
  int32_t* status;
  const void *ka, *kb;       // the keys' first tensor, and the rope's
  float* out;                // [rows, topk]
  int32_t heads;             // of this side
  int32_t nblk, nblk_a;      // 64-feature blocks in all / of the first tensor (the others: rope)
  int32_t hp;                // heads per item, padded to 16
  int32_t hchunks, parts, items, stages;
  uint32_t idesc, off_k, off_prm, off_bar;
};

struct SliItem { int32_t row, b, h0, n, t0, t1; };
__device__ __forceinline__ SliItem sli_score_item(const SliScoreArgs& a, int32_t item) {
  SliItem it;
  const int32_t per_row = a.hchunks * a.parts;
  it.row = item / per_row;
  const int32_t rem = item - it.row * per_row;
  const int32_t hc = rem / a.parts, part = rem - hc * a.parts;
  it.h0 = hc * a.hp;
  it.n = sli_row_slots(a.p, it.row, &it.b);
  const int32_t nt = (it.n + kSlKeys - 1) / kSlKeys, per = (nt + a.parts - 1) / a.parts;
  it.t0 = part * per;
  it.t1 = min(nt, it.t0 + per);
  return it;
}

// PAD: the last chunk of attention heads is not full.  Q of the missing ones is zero, their scores are NaN beside an
// infinite key; compiled apart because the test costs the others 1 % (2048 rows x 128 heads: 1658 -> 1674 us).
template <bool ATT, bool PAD>
__global__ void __launch_bounds__(kScThreads, 1)
sli_score_sm100_kernel(const __grid_constant__ CUtensorMap tmap_qa, const __grid_constant__ CUtensorMap tmap_qb,
                       const SliScoreArgs a) {
  extern __shared__ __align__(1024) unsigned char slsm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(slsm + a.off_bar);
  uint64_t* full = bars;                       // [stages] gather -> its issuer    (64 lanes' copies)
  uint64_t* empty = bars + kScMaxStages;       // [stages] products done -> gather (commit)
  uint64_t* s_full = bars + 2 * kScMaxStages;  // [2] scores -> epilogue           (both issuers' commits)
  uint64_t* s_empty = s_full + 2;              // [2] scores read                  (4 warps)
  uint64_t* q_full = s_full + 4;               // Q landed                         (tx bytes)
  uint64_t* q_empty = s_full + 5;              // last products of the item        (both issuers' commits)
  uint64_t* m_full = s_full + 6;               // [2] head parameters stored       (loader)
  uint64_t* m_empty = s_full + 8;              // [2] head parameters read         (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(s_full + 11);
  float2* prm = reinterpret_cast<float2*>(slsm + a.off_prm);    // [2][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool misaligned = (ptx::smem_u32(slsm) & 1023u) != 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kScMaxStages; ++i) { ptx::mbar_init(&full[i], 64); ptx::mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&s_full[i], 2);
      ptx::mbar_init(&s_empty[i], 4);
      ptx::mbar_init(&m_full[i], 1);
      ptx::mbar_init(&m_empty[i], 8);
    }
    ptx::mbar_init(q_full, 1);
    ptx::mbar_init(q_empty, 2);
    *abort_flag = misaligned ? 1 : 0;
    ptx::mbar_fence_init();
  }
  if (warp == kScIssuer) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sm0 = ptx::smem_u32(slsm);
  const uint32_t qblk = (uint32_t)a.hp * 128;
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::mbar_wait_warp(bar, parity, abort_flag); };
  auto spin = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::mbar_spin(bar, parity, abort_flag); };

  if (*abort_flag) {
    // nothing started
  } else if (warp < kScGatherWarp0) {
    const int wg = warp >> 2, quarter = warp & 3;
    const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + wg * 256;
    uint32_t n_tile = 0, n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliItem it = sli_score_item(a, item);
      if (it.t1 <= it.t0) continue;
      const int mb = n_item & 1;
      const float2* pm = prm + mb * 128;
      ok = wait(&m_full[mb], (n_item >> 1) & 1);
      float* out_row = a.out + (int64_t)it.row * a.p.topk;
      const int32_t hn = PAD ? min(a.hp, a.heads - it.h0) : a.hp;
      for (int32_t t = it.t0; t < it.t1 && ok; ++t, ++n_tile) {
        if ((int)(n_tile & 1) != wg) continue;
        ok = wait(&s_full[wg], (n_tile >> 1) & 1);
        if (!ok) break;
        ptx::tc_fence_after();
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 1
        for (int c = 0; c < a.hp; c += 32) {
          const bool two = c + 16 < a.hp;
          float v[32], u[32];
          ptx::tmem_ld_x16(base + c, reinterpret_cast<uint32_t*>(v));
          ptx::tmem_ld_x16(base + 128 + c, reinterpret_cast<uint32_t*>(u));
          if (two) {
            ptx::tmem_ld_x16(base + c + 16, reinterpret_cast<uint32_t*>(v + 16));
            ptx::tmem_ld_x16(base + 128 + c + 16, reinterpret_cast<uint32_t*>(u + 16));
          }
          ptx::tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 32; ++h) v[h] += u[h];
          if (c + 32 >= a.hp) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s_empty[wg]);
          }
          if (PAD && c + 32 > hn) {
#pragma unroll
            for (int h = 0; h < 32; ++h) v[h] = c + h < hn ? v[h] : 0.f;
          }
#pragma unroll
          for (int h = 0; h < 32; h += 2) {
            if (h < 16 || two) {
              const float4 m = *reinterpret_cast<const float4*>(pm + c + h);
              if (ATT) {   // m: max, 1 / sum of head h, then of head h + 1
                s0 = fmaf(expf(fmaf(v[h], a.p.scale, -m.x)), m.y, s0);
                s1 = fmaf(expf(fmaf(v[h + 1], a.p.scale, -m.z)), m.w, s1);
              } else {     // m: weight, unused
                s0 = fmaf(fmaxf(v[h], 0.f), m.x, s0);
                s1 = fmaf(fmaxf(v[h + 1], 0.f), m.z, s1);
              }
            }
          }
        }
        const int32_t j = t * kSlKeys + quarter * 32 + lane;
        if (j < it.n) {
          if (a.hchunks > 1) atomicAdd(&out_row[j], s0 + s1);
          else out_row[j] = s0 + s1;
        }
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&m_empty[mb]);
      ++n_item;
    }
  } else if (warp < kScIssuer) {
    // gather: pairs of warps take the 64-feature blocks in turn, a warp half of a block's keys (16 copies per lane, an
    // instruction is 4 keys x 128 bytes).  Pairs <= stages: a warp that waited for a ring slot one round ahead of
    // another would take the round before for its own (the wait tells odd from even rounds only).
    const int pair = (warp - kScGatherWarp0) >> 1, key_w = ((warp - kScGatherWarp0) & 1) * 64 + (lane >> 3), ch = lane & 7;
    const uint32_t dst0 = sm0 + a.off_k + key_w * 128 + ((ch ^ (key_w & 7)) << 4);
    const uint32_t dst1 = sm0 + a.off_k + (key_w + 4) * 128 + ((ch ^ ((key_w + 4) & 7)) << 4);
    const unsigned char *ka = (const unsigned char*)a.ka + ch * 16, *kb = (const unsigned char*)a.kb + ch * 16;
    // (the pair's block of the ring: `blk` of the current tile; it and `stage` move on by kPairs.  The wait suspends:
    // eight polling warps take the issuers' issue slots, 150 -> 155 us)
    constexpr int kPairs = kScGatherWarps / 2;
    uint32_t ph = 1;
    int stage = pair, blk = pair;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliItem it = sli_score_item(a, item);
      if (it.t1 <= it.t0) continue;
      const int32_t* idx_row = a.p.sparse_indices ? a.p.sparse_indices + (int64_t)it.row * a.p.topk : nullptr;
      int32_t rn[16];
      auto load = [&](int32_t t) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {        // (no branch, or each load would wait for the one before it)
          const int32_t j = min(t * kSlKeys + key_w + 4 * i, it.n - 1);
          rn[i] = idx_row ? idx_row[j] : j;
        }
      };
      load(it.t0);
      for (int32_t t = it.t0; t < it.t1 && ok; ++t) {
        int32_t r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)          // (slots past the row's last: -1)
          r[i] = t * kSlKeys + key_w + 4 * i < it.n ? it.b * a.p.s2 + min(max(rn[i], 0), a.p.s2 - 1) : -1;
        if (t + 1 < it.t1) load(t + 1);
        for (; blk < a.nblk; blk += kPairs) {
          ok = wait(&empty[stage], ph);
          if (!ok) break;
          const unsigned char* src = blk < a.nblk_a ? ka + blk * 128 : kb + (blk - a.nblk_a) * 128;
          const uint32_t pitch = (uint32_t)(blk < a.nblk_a ? a.nblk_a : a.nblk - a.nblk_a) * 128;
          const uint32_t off = stage * kSlKBlk;
#pragma unroll
          for (int i = 0; i < 16; ++i)        // (slots past the row's last load zeros)
            ptx::cp_async_16(((i & 1) ? dst1 : dst0) + off + (i >> 1) * 1024, src + (uint64_t)max(r[i], 0) * pitch,
                             r[i] >= 0 ? 16u : 0u);
          ptx::cp_async_mbar_arrive(&full[stage]);
          stage += kPairs;
          if (stage >= a.stages) { stage -= a.stages; ph ^= 1; }
        }
        blk -= a.nblk;
      }
    }
  } else if (warp < kScLoader) {
    // Two issuers, one thread each, take the ring's even and odd blocks into accumulators of their own (the epilogue
    // adds them): one thread needs about 560 cycles for a block's four products, twice what the tensor core does.
    // The number of stages is even, so that a stage has one reader: one that waited for a stage whose block before
    // belongs to the other would take the round before for its own.
    if (lane == 0) {
      const uint64_t q_d = ptx::desc_kmajor_sw128(sm0), k_d = ptx::desc_kmajor_sw128(sm0 + a.off_k);
      const int me = warp - kScIssuer;
      uint32_t n_tile = 0, n_item = 0, ph = 0;
      int stage = me, first = me;              // first: my first block of the tile
      bool ok = true;
      for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
        const SliItem it = sli_score_item(a, item);
        if (it.t1 <= it.t0) continue;
        ok = spin(q_full, n_item & 1);
        for (int32_t t = it.t0; t < it.t1 && ok; ++t, ++n_tile) {
          const int buf = n_tile & 1;
          ok = spin(&s_empty[buf], ((n_tile >> 1) & 1) ^ 1);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint32_t acc = tmem + buf * 256 + me * 128;
          for (int blk = first; blk < a.nblk; blk += 2) {
            ok = spin(&full[stage], ph);
            if (!ok) break;
            ptx::fence_proxy_async_smem();     // (the copies went through the generic proxy)
            const uint64_t kd = k_d + ((stage * kSlKBlk) >> 4), qd = q_d + ((blk * qblk) >> 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) ptx::mma_ss(acc, kd + i * 2, qd + i * 2, a.idesc, (blk > first || i > 0) ? 1u : 0u);
            ptx::mma_commit(&empty[stage]);
            stage += 2;
            if (stage >= a.stages) { stage = me; ph ^= 1; }
          }
          if (!ok) break;
          first ^= a.nblk & 1;
          ptx::mma_commit(&s_full[buf]);
          if (t == it.t1 - 1) ptx::mma_commit(q_empty);
        }
        ++n_item;
      }
    }
    __syncwarp();
  } else if (warp == kScLoader) {
    if (lane == 0) { ptx::prefetch_tmap(&tmap_qa); ptx::prefetch_tmap(&tmap_qb); }
    uint32_t n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliItem it = sli_score_item(a, item);
      if (it.t1 <= it.t0) continue;
      const int mb = n_item & 1;
      ok = wait(&m_empty[mb], ((n_item >> 1) & 1) ^ 1);
      if (!ok) break;
      for (int h = lane; h < a.hp; h += 32) {
        const int32_t hh = it.h0 + h;
        float2 m = make_float2(0.f, 0.f);          // (heads past the last one add nothing)
        if (hh < a.heads) {
          if (ATT) {
            const int64_t si = (int64_t)it.row * a.p.n1 + hh;      // [batch, 1, s1, n1]
            m = make_float2(a.p.softmax_max[si], 1.f / (a.p.softmax_sum[si] + kSliEps));
          } else {
            m.x = load_weight(a.p.weights, a.p.dtype_w, (int64_t)it.row * a.p.g + hh);
          }
        }
        prm[mb * 128 + h] = m;
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&m_full[mb]);
      ok = wait(q_empty, (n_item & 1) ^ 1);
      if (!ok) break;
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(q_full, (uint32_t)a.nblk * qblk);
        for (int blk = 0; blk < a.nblk; ++blk) {
          if (blk < a.nblk_a) ptx::tma_load_3d(slsm + blk * qblk, &tmap_qa, q_full, blk * 64, it.h0, it.row);
          else ptx::tma_load_3d(slsm + blk * qblk, &tmap_qb, q_full, (blk - a.nblk_a) * 64, it.h0, it.row);
        }
      }
      __syncwarp();
      ++n_item;
    }
  }

  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies / MMAs in flight land
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kScIssuer) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.status, misaligned ? 2 : 1);
}

// ---- dense attention probabilities, one key head per query head -------------------------------------
// What bounds it: a (row, key) pair is one exponential per head, 16 a cycle and SM (1024 cycles for a 128 x
// 128 tile and head, against 770 of tensor pipe at D = 192), and each head brings 96 KB of its own Q and K
// through the ring.  p of the tile stays in registers while the heads go by, so it is stored once.  The heads
// are cut into parts (added with reductions into a zeroed buffer) only when the tiles alone would leave more
// than half of the SMs idle.
// Warps: 0..7 epilogue (lane quarter x column half), 8 TMA, 9 MMA issuer.
constexpr int kMhThreads = 320, kMhStages = 6;
constexpr uint32_t kMhStage = 2 * kSlKBlk;                        // [Q block | K block]
constexpr uint32_t kMhSmemBytes = kMhStages * kMhStage + 256;

struct SliMhaArgs {
  SliGradDev p;
  int32_t* status;
  int32_t nblk, nblk_a, rtiles, ktiles, parts, items;
  uint32_t idesc;
};
struct SliMhaItem { int32_t b, pos0, key0, h0, h1; bool live; };
__device__ __forceinline__ SliMhaItem sli_mha_item(const SliMhaArgs& a, int32_t item) {
  SliMhaItem it;
  const int32_t tile = item / a.parts, part = item - tile * a.parts;
  const int32_t rt = tile / a.ktiles;
  it.key0 = (tile - rt * a.ktiles) * kSlKeys;
  it.b = rt / a.rtiles;
  it.pos0 = (rt - it.b * a.rtiles) * 128;
  const int32_t per = (a.p.n1 + a.parts - 1) / a.parts;
  it.h0 = part * per;
  it.h1 = min(a.p.n1, it.h0 + per);
  const int32_t aq = a.p.act_q ? min(a.p.act_q[it.b], a.p.s1) : a.p.s1;
  const int32_t last = min(it.pos0 + 127, aq - 1);                // (the last valid row sees most)
  int32_t bb, n = 0;
  if (last >= it.pos0) n = sli_row_slots(a.p, it.b * a.p.s1 + last, &bb);
  it.live = it.key0 < n && it.h0 < it.h1;
  return it;
}

__global__ void __launch_bounds__(kMhThreads, 1)
sli_mha_sm100_kernel(const __grid_constant__ CUtensorMap tmap_ka, const __grid_constant__ CUtensorMap tmap_kb,
                     const __grid_constant__ CUtensorMap tmap_qa, const __grid_constant__ CUtensorMap tmap_qb,
                     const SliMhaArgs a) {
  extern __shared__ __align__(1024) unsigned char mhsm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(mhsm + kMhStages * kMhStage);
  uint64_t* full = bars;                    // [6]
  uint64_t* empty = bars + kMhStages;       // [6]
  uint64_t* s_full = bars + 2 * kMhStages;  // [2]
  uint64_t* s_empty = s_full + 2;           // [2] (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(s_full + 5);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool misaligned = (ptx::smem_u32(mhsm) & 1023u) != 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMhStages; ++i) { ptx::mbar_init(&full[i], 1); ptx::mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { ptx::mbar_init(&s_full[i], 1); ptx::mbar_init(&s_empty[i], 8); }
    *abort_flag = misaligned ? 1 : 0;
    ptx::mbar_fence_init();
  }
  if (warp == 9) {
    ptx::tmem_alloc(tmem_slot, 256);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sm0 = ptx::smem_u32(mhsm);
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::mbar_wait_warp(bar, parity, abort_flag); };

  if (*abort_flag) {
    // nothing started
  } else if (warp < 8) {
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + half * 64;
    uint32_t n_s = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliMhaItem it = sli_mha_item(a, item);
      if (!it.live) continue;
      const int32_t pos = it.pos0 + quarter * 32 + lane;
      int32_t bb, n = 0;
      if (pos < a.p.s1) n = sli_row_slots(a.p, it.b * a.p.s1 + pos, &bb);
      const int64_t st0 = (int64_t)it.b * a.p.n1 * a.p.s1 + min(pos, a.p.s1 - 1);      // [batch, n1, s1, 1]
      float acc[64];
#pragma unroll
      for (int k = 0; k < 64; ++k) acc[k] = 0.f;
      float mx = a.p.softmax_max[st0 + (int64_t)it.h0 * a.p.s1], sm = a.p.softmax_sum[st0 + (int64_t)it.h0 * a.p.s1];
      for (int32_t h = it.h0; h < it.h1; ++h, ++n_s) {
        const int buf = n_s & 1;
        const float m = mx, inv = 1.f / (sm + kSliEps);
        if (h + 1 < it.h1) {
          mx = a.p.softmax_max[st0 + (int64_t)(h + 1) * a.p.s1];
          sm = a.p.softmax_sum[st0 + (int64_t)(h + 1) * a.p.s1];
        }
        ok = wait(&s_full[buf], (n_s >> 1) & 1);
        if (!ok) break;
        ptx::tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          float v[32];
          ptx::tmem_ld_x32(base + buf * 128 + c, reinterpret_cast<uint32_t*>(v));
          ptx::tmem_ld_wait();
          if (c == 32) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s_empty[buf]);
          }
#pragma unroll
          for (int k = 0; k < 32; ++k)
            acc[c + k] = fmaf(expf(fmaf(v[k], a.p.scale, -m)), inv, acc[c + k]);
        }
      }
      if (!ok) break;
      float* out = a.p.p_buf + ((int64_t)it.b * a.p.s1 + pos) * a.p.topk + it.key0 + half * 64;
      const int32_t left = n - it.key0 - half * 64;
      if (a.parts > 1) {
#pragma unroll
        for (int k = 0; k < 64; ++k)
          if (k < left) atomicAdd(&out[k], acc[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 64; ++k)
          if (k < left) out[k] = acc[k];
      }
    }
  } else if (warp == 8) {
    uint32_t ph = 1;
    int stage = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliMhaItem it = sli_mha_item(a, item);
      if (!it.live) continue;
      const int32_t qrow = it.b * a.p.s1 + it.pos0, krow = it.b * a.p.s2 + it.key0;
      for (int32_t h = it.h0; h < it.h1 && ok; ++h)
        for (int blk = 0; blk < a.nblk && ok; ++blk) {
          ok = wait(&empty[stage], ph);
          if (!ok) break;
          if (lane == 0) {
            unsigned char* dst = mhsm + stage * kMhStage;
            ptx::mbar_arrive_expect_tx(&full[stage], kMhStage);
            if (blk < a.nblk_a) {
              ptx::tma_load_3d(dst, &tmap_qa, &full[stage], blk * 64, qrow, h);
              ptx::tma_load_3d(dst + kSlKBlk, &tmap_ka, &full[stage], blk * 64, krow, h);
            } else {
              ptx::tma_load_3d(dst, &tmap_qb, &full[stage], (blk - a.nblk_a) * 64, qrow, h);
              ptx::tma_load_3d(dst + kSlKBlk, &tmap_kb, &full[stage], (blk - a.nblk_a) * 64, krow, h);
            }
          }
          __syncwarp();
          if (++stage == kMhStages) { stage = 0; ph ^= 1; }
        }
    }
  } else {
    const uint64_t q_d = ptx::desc_kmajor_sw128(sm0), k_d = ptx::desc_kmajor_sw128(sm0 + kSlKBlk);
    uint32_t n_s = 0, ph = 0;
    int stage = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliMhaItem it = sli_mha_item(a, item);
      if (!it.live) continue;
      for (int32_t h = it.h0; h < it.h1 && ok; ++h, ++n_s) {
        const int buf = n_s & 1;
        ok = wait(&s_empty[buf], ((n_s >> 1) & 1) ^ 1);
        for (int blk = 0; blk < a.nblk && ok; ++blk) {
          ok = wait(&full[stage], ph);
          if (!ok) break;
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              ptx::mma_ss(tmem + buf * 128, q_d + ((stage * kMhStage) >> 4) + i * 2, k_d + ((stage * kMhStage) >> 4) + i * 2,
                          a.idesc, (blk > 0 || i > 0) ? 1u : 0u);
            ptx::mma_commit(&empty[stage]);
            if (blk == a.nblk - 1) ptx::mma_commit(&s_full[buf]);
          }
          __syncwarp();
          if (++stage == kMhStages) { stage = 0; ph ^= 1; }
        }
      }
    }
  }

  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies / MMAs in flight land
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 256);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.status, misaligned ? 2 : 1);
}

// ---- gradients -----------------------------------------------------------------------------------
// What it is built around: the scatter-adds of dKI (512 B per (row, key): 2300 cycles of the load / store unit
// per 128 keys, 4.5 per line; all SMs together 6.2 TB/s), against 1300 cycles of tensor pipe and 1170 of
// gather.  ncu, 512 rows x 2048 keys, 64 heads: 174 us, 3.1 TB/s of reductions, load / store data pipe 41 %, tensor
// pipe 29 % (dense over 3840 keys a row: 286 us, 3.5 TB/s, 44 %, 33 %).  So a work item is (query row, 64 index heads),
// which makes every reduction carry all heads of up to 64, and as in sfa_bwd_sm100.cuh the gradient products run with
// FEATURES on the lanes, so that a reduction instruction is one full line.  Per tile of 128 gathered keys (M = the first named):
//     S   [keys, heads]     = K . QI^T                              E = S > 0
//     dKI^T [features, keys]  = (w QI)^T . E^T, times dI of the key   when it is drained
//     dQI^T [features, heads] += K^T . (dI E), times w of the head      at the end of the row
// E is exact in 16 bits.  w QI (once per row) and dI (once per key) enter as a high and a low io-dtype part
// (x = hi + lo up to 2^-16 relative for bf16, 2^-22 for fp16), dI E is then two masked copies of the parts
// without a conversion per element.  fp16: both are scaled by a power of two per row taken from the
// row's largest magnitude (sli_grad_kernel scales dI per 64 keys; all terms meet in one sum, whose error the row's largest
// decides either way).  dW = sum_k dI relu(S) is summed in fp32 registers.
// Tensor memory: S 2 x 64 columns | dKI^T 2 x 128 | dQI^T 64.
// Warps: 0..7 epilogue (lane quarter x 32 heads), 8..15 drain (lane quarter x 64 keys), 16..23 gather, 24
// issuer of S / dKI, 25 issuer of dQI, 26..27 QI and w QI.  (A thread issues a product of 64 columns only every
// 60-90 cycles, and a gather warp its lanes' loads one by one, ~180 cycles each: one issuer and four gather
// warps took 3300 and 3000 cycles a tile.)
constexpr int kSgThreads = 896, kSgDrainWarp0 = 8, kSgGatherWarp0 = 16, kSgGatherWarps = 8, kSgIssueA = 24, kSgIssueB = 25;
constexpr int kSgStager0 = 26;
// the epilogue and drain warps take the registers that the others give back
constexpr int kSgLaunchRegs = 72, kSgRegsLow = 48, kSgRegsDrain = 80, kSgRegsEpi = 96;
static_assert((kSgRegsEpi - kSgLaunchRegs) * kSgDrainWarp0 + (kSgRegsDrain - kSgLaunchRegs) * (kSgGatherWarp0 - kSgDrainWarp0) <=
                  (kSgLaunchRegs - kSgRegsLow) * (kSgThreads / 32 - kSgGatherWarp0),
              "setmaxnreg: more registers requested than released");
static_assert(kSgLaunchRegs * kSgThreads <= 65536, "register file");
constexpr int kSgStages = 3;
constexpr uint32_t kSgHBlk = 64 * 128;                             // 64 heads x 64 features
constexpr uint32_t kSgOffQ = 0;                                    // 2 blocks
constexpr uint32_t kSgOffW = kSgOffQ + 2 * kSgHBlk;                // w QI hi: 2 blocks, lo: 2 blocks
constexpr uint32_t kSgOffK = kSgOffW + 4 * kSgHBlk;                // stages x 2 blocks
constexpr uint32_t kSgOffE = kSgOffK + kSgStages * 2 * kSlKBlk;    // E, dI E hi, dI E lo: [128 keys][64 heads]
constexpr uint32_t kSgOffRows = kSgOffE + 3 * kSlKBlk;             // int32 [4][128] key rows
constexpr uint32_t kSgOffDi = kSgOffRows + 4 * kSlKeys * 4;        // float [4][128]
constexpr uint32_t kSgOffDw = kSgOffDi + 4 * kSlKeys * 4;          // float [2][4][64]
constexpr uint32_t kSgOffBar = kSgOffDw + 2 * 4 * 64 * 4;
constexpr uint32_t kSgSmemBytes = kSgOffBar + 256;
static_assert(kSgSmemBytes <= kSlSmemMax, "shared memory");
constexpr uint32_t kSgTmS = 0, kSgTmK = 128, kSgTmQ = 384;

constexpr int kSgPart = 64 * 128 + 64;
constexpr int kSgMaxParts = 4;

struct SliGradArgs {
  SliGradDev p;
  int32_t* status;
  const float* di_max;       // [rows] largest |dI| of the row (fp16)
  int32_t hchunks, items, key_rows;
  int32_t full, parts;
  float* part;               // [items - full][kSgPart]: dQI of 64 heads x 128 features (before w), dW of 64 heads
  uint32_t idesc_s, idesc_k, idesc_q;
};

// Parts that a row with `tiles` tiles is cut into, at most `parts`: of 3 tiles or more, and all of them with slots
// ((n - 1)^2 < tiles).  Whole calls, 2048 selected slots, rows whole / cut, us: 20 rows of 700 keys (6 tiles) 59 / 54, 222
// rows of up to 700 101 / 97; cut by slots alone, as if every row had 2048 keys, 20 rows of 100 keys 60 for 46, 222 of
// 300 85 for 78 (with a kernel of its own for the sums).
__device__ __forceinline__ int32_t sli_row_parts(int32_t tiles, int32_t parts) { return max(1, min(parts, tiles / 3)); }
// Work item: (row, 64 heads) or, in the last round, a part of its slots (SliGradSplit): slots off .. off + n - 1.  Its
// place in `part`, -1: the whole row.  n = -1: nothing to do, the row has fewer parts.
struct SliGradItem { int32_t row, h0, n, off, key0, slot; };      // key0: key row that dense slots and indices count from
template <bool kCut>
__device__ __forceinline__ SliGradItem sli_grad_item(const SliGradArgs& a, int32_t i) {
  SliGradItem it;
  it.slot = -1;
  it.off = 0;
  int32_t base = i, part = 0;
  if (kCut && i >= a.full) {
    it.slot = i - a.full;
    const int32_t r = it.slot / a.parts;
    part = it.slot - r * a.parts;
    base = a.full + r;
  }
  it.row = base / a.hchunks;
  it.h0 = (base - it.row * a.hchunks) * 64;
  int32_t b;
  it.n = sli_row_slots(a.p, it.row, &b);
  it.key0 = b * a.p.s2;
  if (kCut && it.slot >= 0) {
    const int32_t tiles = (it.n + kSlKeys - 1) / kSlKeys, n = sli_row_parts(tiles, a.parts);
    if (n == 1) it.slot = -1;
    if (part >= n) {
      it.n = -1;
    } else if (n > 1) {
      const int32_t per = (tiles + n - 1) / n * kSlKeys;
      it.off = part * per;
      it.n = min(per, it.n - it.off);
      if (a.p.sparse_indices == nullptr) it.key0 += it.off;
    }
  }
  return it;
}
// Key row of the item's j-th slot; past its n slots `none` (a row that does not exist: TMA fills zeros).
__device__ __forceinline__ int32_t sli_key_row(const SliGradDev& p, const int32_t* idx_row, const SliGradItem& it, int32_t j,
                                               int32_t none) {
  return j < it.n ? it.key0 + sli_slot_key(p, idx_row, j) : none;
}

// Exponent of the power of two that brings magnitudes up to `m` below 2^14.
__device__ __forceinline__ int sli_exponent(float m) {
  return (m > 0.f && m < INFINITY) ? max(-100, min(100, 13 - ilogbf(m))) : 0;
}

template <typename T>
__device__ __forceinline__ uint32_t sli_bits(T v) { return (uint32_t)*reinterpret_cast<const uint16_t*>(&v); }

// kCut: items of the last round may be parts of rows.  Compiled apart because the other calls pay for it otherwise (this
// kernel, 625 dense rows of 202 to 826 keys: 72.7 us apart, 74.3 together, 75.9 with the choice between part and row
// inside the loop that stores dQI; 678 rows, fp16: 88.8, 89.2, 91.9).
template <typename T, bool kCut>
__global__ void __launch_bounds__(kSgThreads, 1)
sli_grad_sm100_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_q,
                      const SliGradArgs a) {
  constexpr bool kScaled = !kIsBf16<T>;
  extern __shared__ __align__(1024) unsigned char sgsm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(sgsm + kSgOffBar);
  uint64_t* k_full = bars;          // [3] gather -> issuer                               (tx bytes)
  uint64_t* k_empty = bars + 3;     // [3] dQI of the tile done                           (commit)
  uint64_t* s_full = bars + 6;      // [2] scores -> epilogue                             (commit)
  uint64_t* s_empty = bars + 8;     // [2] scores read                                    (8 warps)
  uint64_t* e_full = bars + 10;     // E, dI E, rows and dI of the tile stored            (8 warps)
  uint64_t* e_empty = bars + 11;    // gradient products of the tile done                 (commits A, B)
  uint64_t* d_full = bars + 12;     // [2] dKI^T -> drain                                 (commit)
  uint64_t* d_empty = bars + 14;    // [2] dKI^T read                                     (8 warps)
  uint64_t* q_full = bars + 16;     // QI landed                                          (tx bytes)
  uint64_t* q_empty = bars + 17;    // last scores of the item done, w QI taken           (commit, 2 warps)
  uint64_t* w_full = bars + 18;     // w QI stored                                        (2 warps)
  uint64_t* w_empty = bars + 19;    // last gradient products of the item done            (commit)
  uint64_t* dq_full = bars + 20;    // dQI^T complete                                     (commit)
  uint64_t* dq_empty = bars + 21;   // dQI^T read                                         (8 warps)
  uint64_t* dw_full = bars + 22;    // dW parts of the quarters stored                    (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 24);
  int32_t* w_exp = reinterpret_cast<int32_t*>(bars + 25);          // [2] exponent of w QI of the item
  int32_t* rows_s = reinterpret_cast<int32_t*>(sgsm + kSgOffRows);
  float* di_s = reinterpret_cast<float*>(sgsm + kSgOffDi);
  float* dw_s = reinterpret_cast<float*>(sgsm + kSgOffDw);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool misaligned = (ptx::smem_u32(sgsm) & 1023u) != 0;
  if (threadIdx.x == 0) {
    const int counts[23] = {1, 1, 1, 1, 1, 1, 1, 1, 8, 8, 8, 2, 1, 1, 8, 8, 1, 3, 2, 1, 1, 8, 8};
#pragma unroll
    for (int i = 0; i < 23; ++i) ptx::mbar_init(&bars[i], counts[i]);
    *abort_flag = misaligned ? 1 : 0;
    ptx::mbar_fence_init();
  }
  if (warp == kSgIssueA) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sm0 = ptx::smem_u32(sgsm);
  const int32_t g = a.p.g;
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::mbar_wait_warp(bar, parity, abort_flag); };
  auto tiles_of = [&](int32_t n) -> int32_t { return (n + kSlKeys - 1) / kSlKeys; };

  // Each class of roles sits in its own branch, right under its setmaxnreg: the compiler budgets a
  // branch by the setmaxnreg that dominates it.
  if (warp < kSgDrainWarp0) {
   asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSgRegsEpi));
   if (!*abort_flag) {
    // -------------------------------------------------------------------- E and dI E, dW; then dQI
    const int quarter = warp & 3, half = warp >> 2;
    const int key = quarter * 32 + lane;                  // within the tile
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    unsigned char* e_row = sgsm + kSgOffE + key * 128;
    uint32_t n_tile = 0, n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliGradItem it = sli_grad_item<kCut>(a, item);
      if (kCut && it.n < 0) continue;
      const int32_t row = it.row, h0 = it.h0, n = it.n, ntiles = tiles_of(n);
      const int32_t hn = min(32, g - h0 - half * 32);     // this warp's heads that exist
      float* part = kCut && it.slot >= 0 ? a.part + (int64_t)it.slot * kSgPart : nullptr;
      T* dq = (T*)a.p.d_query_index + ((int64_t)row * g + h0 + half * 32) * 128 + key;
      if (ntiles == 0) {
        for (int h = 0; h < hn; ++h) dq[h * 128] = from_f32<T>(0.f);
        if (quarter == 0 && lane < hn)
          store_weight(a.p.d_weights, a.p.dtype_w, (int64_t)row * g + h0 + half * 32 + lane, 0.f);
        continue;
      }
      const int32_t* idx_row = a.p.sparse_indices ? a.p.sparse_indices + (int64_t)row * a.p.topk + it.off : nullptr;
      const float* di_row = a.p.di + (int64_t)row * a.p.topk + it.off;
      float up = 1.f, down = 1.f, w_down = 1.f;
      if constexpr (kScaled) {
        const int e = sli_exponent(a.di_max[row]);
        up = scalbnf(1.f, e);
        down = scalbnf(1.f, -e);
        ok = wait(w_full, n_item & 1);
        if (!ok) break;
        w_down = scalbnf(1.f, -w_exp[n_item & 1]);
      }
      float dw[32];
#pragma unroll
      for (int h = 0; h < 32; ++h) dw[h] = 0.f;
      float d_next = key < n ? di_row[key] : 0.f;
      int32_t r_next = sli_key_row(a.p, idx_row, it, key, -1);
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        const int buf = n_tile & 1;
        const float d = d_next;
        const int32_t r = r_next;
        {
          const int32_t j = (t + 1) * kSlKeys + key;
          d_next = j < n ? di_row[j] : 0.f;
          r_next = sli_key_row(a.p, idx_row, it, j, -1);
        }
        const float du = kScaled ? d * up : d;
        const T hi = from_f32<T>(du), lo = from_f32<T>(du - to_f32<T>(hi));
        const uint32_t hi2 = sli_bits<T>(hi) * 0x10001u, lo2 = sli_bits<T>(lo) * 0x10001u;
        const uint32_t one2 = kScaled ? 0x3C003C00u : 0x3F803F80u;
        ok = wait(&s_full[buf], (n_tile >> 1) & 1);
        if (!ok) break;
        ptx::tc_fence_after();
        uint32_t m[16];                                   // masks of the head pairs
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
          float v[16];
          ptx::tmem_ld_x16(lane_addr + kSgTmS + buf * 64 + half * 32 + c, reinterpret_cast<uint32_t*>(v));
          ptx::tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 16; h += 2) {
            dw[c + h] = fmaf(d, fmaxf(v[h], 0.f), dw[c + h]);
            dw[c + h + 1] = fmaf(d, fmaxf(v[h + 1], 0.f), dw[c + h + 1]);
            m[(c + h) / 2] = (v[h] > 0.f ? 0x0000FFFFu : 0u) | (v[h + 1] > 0.f ? 0xFFFF0000u : 0u);
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&s_empty[buf]);
        ok = wait(e_empty, (n_tile & 1) ^ 1);
        if (!ok) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          unsigned char* dst = e_row + (((half * 4 + q) ^ (key & 7)) << 4);
          const uint32_t* mq = m + q * 4;
          *reinterpret_cast<uint4*>(dst) = make_uint4(mq[0] & one2, mq[1] & one2, mq[2] & one2, mq[3] & one2);
          *reinterpret_cast<uint4*>(dst + kSlKBlk) = make_uint4(mq[0] & hi2, mq[1] & hi2, mq[2] & hi2, mq[3] & hi2);
          *reinterpret_cast<uint4*>(dst + 2 * kSlKBlk) = make_uint4(mq[0] & lo2, mq[1] & lo2, mq[2] & lo2, mq[3] & lo2);
        }
        // The drain warps' rows and dI, four buffers: e_empty of the last tile means that its dKI^T tile was
        // started, so that the drain warps have read the one of two tiles before and left all earlier ones.
        if (half == 0) {
          rows_s[(n_tile & 3) * kSlKeys + key] = r;
          di_s[(n_tile & 3) * kSlKeys + key] = kScaled ? d * w_down : d;
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(e_full);
      }
      if (!ok) break;
      // dW: lane h ends up with the warp's sum of head h
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const bool up_half = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float keep = up_half ? dw[i + o] : dw[i], send = up_half ? dw[i] : dw[i + o];
          dw[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      float* dwb = dw_s + (n_item & 1) * 256;
      dwb[quarter * 64 + half * 32 + lane] = dw[0];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(dw_full);
      ok = wait(dw_full, n_item & 1);
      if (!ok) break;
      if (quarter == 0 && lane < hn) {
        const int h = half * 32 + lane;
        const float sum = (dwb[h] + dwb[64 + h]) + (dwb[128 + h] + dwb[192 + h]);
        if (part) part[64 * 128 + h] = sum;
        else store_weight(a.p.d_weights, a.p.dtype_w, (int64_t)row * g + h0 + h, sum);
      }
      ok = wait(dq_full, n_item & 1);
      if (!ok) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int c = 0; c < 32; c += 16) {
        float v[16];
        ptx::tmem_ld_x16(lane_addr + kSgTmQ + half * 32 + c, reinterpret_cast<uint32_t*>(v));
        ptx::tmem_ld_wait();
        if (c == 16) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(dq_empty);
        }
        if (part) {
#pragma unroll
          for (int h = 0; h < 16; ++h)
            if (c + h < hn) part[(half * 32 + c + h) * 128 + key] = kScaled ? v[h] * down : v[h];
        } else {
#pragma unroll
          for (int h = 0; h < 16; ++h)
            if (c + h < hn) {
              const float w = load_weight(a.p.weights, a.p.dtype_w, (int64_t)row * g + h0 + half * 32 + c + h);
              dq[(c + h) * 128] = from_f32<T>((kScaled ? v[h] * down : v[h]) * w);
            }
        }
      }
      ++n_item;
    }
   }
  } else if (warp < kSgGatherWarp0) {
   asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSgRegsDrain));
   if (!*abort_flag) {
    // -------------------------------------------------------------------- drain: reductions of dKI^T
    const int quarter = warp & 3, k0 = ((warp - kSgDrainWarp0) >> 2) * 64;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + kSgTmK + k0;
    float* base = a.p.dki_acc + quarter * 32 + lane;
    uint32_t n_tile = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const int32_t n = sli_grad_item<kCut>(a, item).n, ntiles = tiles_of(n);
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        const int buf = n_tile & 1;
        const int4* rows4 = reinterpret_cast<const int4*>(rows_s + (n_tile & 3) * kSlKeys + k0);
        const float4* di4 = reinterpret_cast<const float4*>(di_s + (n_tile & 3) * kSlKeys + k0);
        ok = wait(&d_full[buf], (n_tile >> 1) & 1);
        if (!ok) break;
        ptx::tc_fence_after();
        const bool whole = n - t * kSlKeys >= kSlKeys;
#pragma unroll 1
        for (int c = 0; c < 64; c += 16) {
          float v[16];
          int4 r[4];
          ptx::tmem_ld_x16(lane_addr + buf * kSlKeys + c, reinterpret_cast<uint32_t*>(v));
#pragma unroll
          for (int k = 0; k < 4; ++k) r[k] = rows4[c / 4 + k];
          float4 d[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) d[k] = di4[c / 4 + k];
          ptx::tmem_ld_wait();
          if (c == 48) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&d_empty[buf]);
          }
          if (whole) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              red_add(base + (int64_t)r[k].x * 128, v[4 * k] * d[k].x);
              red_add(base + (int64_t)r[k].y * 128, v[4 * k + 1] * d[k].y);
              red_add(base + (int64_t)r[k].z * 128, v[4 * k + 2] * d[k].z);
              red_add(base + (int64_t)r[k].w * 128, v[4 * k + 3] * d[k].w);
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              red_add_if(r[k].x >= 0, base + (int64_t)r[k].x * 128, v[4 * k] * d[k].x);
              red_add_if(r[k].y >= 0, base + (int64_t)r[k].y * 128, v[4 * k + 1] * d[k].y);
              red_add_if(r[k].z >= 0, base + (int64_t)r[k].z * 128, v[4 * k + 2] * d[k].z);
              red_add_if(r[k].w >= 0, base + (int64_t)r[k].w * 128, v[4 * k + 3] * d[k].w);
            }
          }
        }
      }
    }
   }
  } else {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSgRegsLow));
   if (*abort_flag) {
    // nothing started
   } else if (warp < kSgIssueA) {
    // -------------------------------------------------------------------- gather: 32 groups of 4 keys x 2 blocks
    const int o = (warp - kSgGatherWarp0) + kSgGatherWarps * lane;
    const bool active = o < 64;
    const int grp = o >> 1, blk = o & 1;
    if (lane == 0) ptx::prefetch_tmap(&tmap_k);
    uint32_t ph = 1;
    int stage = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliGradItem it = sli_grad_item<kCut>(a, item);
      const int32_t ntiles = tiles_of(it.n);
      const int32_t* idx_row = a.p.sparse_indices ? a.p.sparse_indices + (int64_t)it.row * a.p.topk + it.off : nullptr;
      int32_t rn[4];
      auto load = [&](int32_t t) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          rn[i] = active ? sli_key_row(a.p, idx_row, it, t * kSlKeys + grp * 4 + i, a.key_rows) : a.key_rows;
      };
      load(0);
      for (int32_t t = 0; t < ntiles && ok; ++t) {
        int32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = rn[i];
        load(t + 1);
        ok = wait(&k_empty[stage], ph);
        if (!ok) break;
        if (warp == kSgGatherWarp0 && lane == 0) ptx::mbar_arrive_expect_tx(&k_full[stage], 2 * kSlKBlk);
        __syncwarp();
        if (active)
          ptx::tma_gather4_2d(sgsm + kSgOffK + (stage * 2 + blk) * kSlKBlk + grp * 512, &tmap_k, &k_full[stage], blk * 64,
                              r[0], r[1], r[2], r[3]);
        __syncwarp();
        if (++stage == kSgStages) { stage = 0; ph ^= 1; }
      }
    }
   } else if (warp == kSgIssueA) {
    // -------------------------------------------------------------------- issuer A: scores one tile ahead, then dKI
    const uint64_t q_k = ptx::desc_kmajor_sw128(sm0 + kSgOffQ), k_k = ptx::desc_kmajor_sw128(sm0 + kSgOffK);
    const uint64_t w_m = ptx::desc_mnmajor_sw128(sm0 + kSgOffW, kSgHBlk, 1024);
    const uint64_t e_k = ptx::desc_kmajor_sw128(sm0 + kSgOffE);
    uint32_t n_s = 0, n_g = 0, n_item = 0, ph_s = 0;
    int st_s = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliGradItem it = sli_grad_item<kCut>(a, item);
      const int32_t ntiles = tiles_of(it.n);
      if (ntiles == 0) continue;
      const int steps = (min(64, g - it.h0) + 15) / 16;
      ok = wait(q_full, n_item & 1);
      for (int32_t t = 0; t <= ntiles && ok; ++t) {
        if (t < ntiles) {
          const int buf = n_s & 1;
          ok = wait(&k_full[st_s], ph_s) && wait(&s_empty[buf], ((n_s >> 1) & 1) ^ 1);
          if (!ok) break;
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              ptx::mma_ss(tmem + kSgTmS + buf * 64, k_k + (((st_s * 2 + (i >> 2)) * kSlKBlk) >> 4) + (i & 3) * 2,
                          q_k + (((i >> 2) * kSgHBlk) >> 4) + (i & 3) * 2, a.idesc_s, i ? 1u : 0u);
            ptx::mma_commit(&s_full[buf]);
            if (t == ntiles - 1) ptx::mma_commit(q_empty);
          }
          __syncwarp();
          ++n_s;
          if (++st_s == kSgStages) { st_s = 0; ph_s ^= 1; }
        }
        if (t > 0) {
          const int buf = n_g & 1;
          if (t == 1) ok = wait(w_full, n_item & 1);
          ok = ok && wait(e_full, n_g & 1) && wait(&d_empty[buf], ((n_g >> 1) & 1) ^ 1);
          if (!ok) break;
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
            ptx::fence_proxy_async_smem();
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              if (s < steps) {
                ptx::mma_ss(tmem + kSgTmK + buf * kSlKeys, w_m + ((s * 2048) >> 4), e_k + s * 2, a.idesc_k, s ? 1u : 0u);
                ptx::mma_ss(tmem + kSgTmK + buf * kSlKeys, w_m + ((2 * kSgHBlk + s * 2048) >> 4), e_k + s * 2, a.idesc_k, 1u);
              }
            }
            ptx::mma_commit(&d_full[buf]);
            ptx::mma_commit(e_empty);
            if (t == ntiles) ptx::mma_commit(w_empty);
          }
          __syncwarp();
          ++n_g;
        }
      }
      ++n_item;
    }
   } else if (warp == kSgIssueB) {
    // -------------------------------------------------------------------- issuer B: dQI
    const uint64_t k_m = ptx::desc_mnmajor_sw128(sm0 + kSgOffK, kSlKBlk, 1024);
    const uint64_t de_m = ptx::desc_mnmajor_sw128(sm0 + kSgOffE + kSlKBlk, 0, 1024);
    uint32_t n_tile = 0, n_item = 0;
    int stage = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const int32_t ntiles = tiles_of(sli_grad_item<kCut>(a, item).n);
      if (ntiles == 0) continue;
      ok = wait(dq_empty, (n_item & 1) ^ 1);
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        // (E is there, so the scores of its keys are: the tile has landed)
        ok = wait(e_full, n_tile & 1);
        if (!ok) break;
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          ptx::fence_proxy_async_smem();
#pragma unroll
          for (int s = 0; s < 8; ++s)
#pragma unroll
            for (int lo = 0; lo < 2; ++lo)
              ptx::mma_ss(tmem + kSgTmQ, k_m + ((stage * 2 * kSlKBlk + s * 2048) >> 4),
                          de_m + ((lo * kSlKBlk + s * 2048) >> 4), a.idesc_q, (t > 0 || s > 0 || lo > 0) ? 1u : 0u);
          ptx::mma_commit(&k_empty[stage]);
          ptx::mma_commit(e_empty);
          if (t == ntiles - 1) ptx::mma_commit(dq_full);
        }
        __syncwarp();
        if (++stage == kSgStages) stage = 0;
      }
      ++n_item;
    }
   } else {
    // -------------------------------------------------------------------- QI (heads past the last: zeros), then
    // w QI, high and low part (same place in its block as QI: the operand's layout is QI's)
    if (warp == kSgStager0 && lane == 0) ptx::prefetch_tmap(&tmap_q);
    const int th = threadIdx.x - kSgStager0 * 32;         // 0..63
    uint32_t n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const SliGradItem it = sli_grad_item<kCut>(a, item);
      const int32_t row = it.row, h0 = it.h0;
      if (it.n <= 0) continue;
      const int32_t hn = min(64, g - h0);
      if (warp == kSgStager0) {
        ok = wait(q_empty, (n_item & 1) ^ 1);
        if (!ok) break;
        if (lane == 0) {
          ptx::mbar_arrive_expect_tx(q_full, 2 * kSgHBlk);
          ptx::tma_load_3d(sgsm + kSgOffQ, &tmap_q, q_full, 0, h0, row);
          ptx::tma_load_3d(sgsm + kSgOffQ + kSgHBlk, &tmap_q, q_full, 64, h0, row);
        }
        __syncwarp();
      }
      ok = wait(q_full, n_item & 1);
      if (!ok) break;
      int e = 0;
      if constexpr (kScaled) {
        // every warp takes the maximum over the whole item (so that no warp waits for another)
        float mx = 0.f;
#pragma unroll 2
        for (int i = lane; i < 1024; i += 32) {           // 16-byte chunk of head (i / 8) % 64
          const uint4 x = reinterpret_cast<const uint4*>(sgsm + kSgOffQ)[i];
          const int h = (i >> 3) & 63;
          const T* xv = reinterpret_cast<const T*>(&x);
          float q = 0.f;
#pragma unroll
          for (int u = 0; u < 8; ++u) q = fmaxf(q, fabsf(to_f32<T>(xv[u])));
          if (h < hn) mx = fmaxf(mx, q * fabsf(load_weight(a.p.weights, a.p.dtype_w, (int64_t)row * g + h0 + h)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        e = sli_exponent(mx);
      }
      const float up = kScaled ? scalbnf(1.f, e) : 1.f;
      ok = wait(w_empty, (n_item & 1) ^ 1);
      if (!ok) break;
#pragma unroll 2
      for (int i = 0; i < 16; ++i) {
        const int c = th + 64 * i, h = (c >> 3) & 63;     // 16-byte chunk c: of head h
        const float w = h < hn ? load_weight(a.p.weights, a.p.dtype_w, (int64_t)row * g + h0 + h) * up : 0.f;
        const uint4 x = reinterpret_cast<const uint4*>(sgsm + kSgOffQ)[c];
        const T* xv = reinterpret_cast<const T*>(&x);
        uint32_t hw[4], lw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float v0 = to_f32<T>(xv[2 * u]) * w, v1 = to_f32<T>(xv[2 * u + 1]) * w;
          const T a0 = from_f32<T>(v0), a1 = from_f32<T>(v1);
          hw[u] = sli_bits<T>(a0) | (sli_bits<T>(a1) << 16);
          lw[u] = sli_bits<T>(from_f32<T>(v0 - to_f32<T>(a0))) | (sli_bits<T>(from_f32<T>(v1 - to_f32<T>(a1))) << 16);
        }
        uint4* dst = reinterpret_cast<uint4*>(sgsm + kSgOffW) + c;
        dst[0] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        dst[2 * kSgHBlk / 16] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
      }
      if (kScaled && th == 0) w_exp[n_item & 1] = e;
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(w_full);
        ptx::mbar_arrive(q_empty);
      }
      ++n_item;
    }
   }
  }

  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies / MMAs in flight land
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kSgIssueA) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.status, misaligned ? 2 : 1);
}

// dQI and dW of the items that were cut into parts: the parts' sums in their order.  A block per item and 8 heads, before
// the `blocks` blocks of the same kernel that round dKI (a kernel of its own costs a call of short rows, in which there
// is nothing to add, 4 to 6 us).
struct SliGradParts {
  const float* part;
  int32_t full, parts, items, hchunks;    // items: of 64 heads, that may be cut
};
template <typename T>
__global__ void __launch_bounds__(256) sli_finalize_parts_kernel(SliGradDev p, int64_t total, int32_t rows, SliGradParts s,
                                                                 int32_t blocks) {
  if ((int32_t)blockIdx.x >= s.items * 8) {
    sli_finalize<T>(p, total, rows, (int32_t)blockIdx.x - s.items * 8, blocks);
    return;
  }
  const int32_t item = (int32_t)blockIdx.x >> 3, base = s.full + item, row = base / s.hchunks;
  const int32_t hl0 = ((int32_t)blockIdx.x & 7) * 8, h0 = (base - row * s.hchunks) * 64 + hl0;
  int32_t b;
  const int32_t n = sli_row_parts((sli_row_slots(p, row, &b) + kSlKeys - 1) / kSlKeys, s.parts), heads = min(8, p.g - h0);
  if (n == 1) return;
  const float* src = s.part + (int64_t)item * s.parts * kSgPart;
  const int64_t o = (int64_t)row * p.g + h0;
#pragma unroll 4
  for (int32_t i = threadIdx.x; i < heads * 128; i += 256) {
    float x[kSgMaxParts];
#pragma unroll
    for (int32_t q = 0; q < kSgMaxParts; ++q) x[q] = q < n ? src[(int64_t)q * kSgPart + hl0 * 128 + i] : 0.f;
    float v = x[0];
#pragma unroll
    for (int32_t q = 1; q < kSgMaxParts; ++q)
      if (q < n) v += x[q];
    ((T*)p.d_query_index)[o * 128 + i] = from_f32<T>(v * load_weight(p.weights, p.dtype_w, o + (i >> 7)));
  }
  if ((int32_t)threadIdx.x < heads) {
    const int32_t i = 64 * 128 + hl0 + threadIdx.x;
    float v = src[i];
    for (int32_t q = 1; q < n; ++q) v += src[(int64_t)q * kSgPart + i];
    store_weight(p.d_weights, p.dtype_w, o + threadIdx.x, v);
  }
}

// ---- host side -----------------------------------------------------------------------------------
// Gradient items of a last round that would leave half of the SMs idle or more: cut into 2 to 4 parts, by the slots (4
// tiles of them a part, or more; as sfa_bwd_split, a row with fewer keys has fewer: sli_row_parts).  Whole calls of
// 64 index heads, rows of the last round whole / cut, us, 2048 selected of 4096 keys | dense over 4096:
//   first round   1 row 77 / 54 | 115 / 69,  37 rows (four parts) 86 / 62 | 137 / 95,  38 (three) 88 / 68 | 138 / 100,
//                 49 92 / 72 | 141 / 104,  50 (two) 92 / 75 | 140 / 112,  74 97 / 82 | 147 / 122
//   second        149 156 / 133 | 231 / 187,  222 162 / 147 | 244 / 214      fourth  512 284 / 269 | 427 / 402
//   fourteenth    1925 925 / 906 | 1137 / 1113,  1998 945 / 932 | 1161 / 1140
// and 222 rows of 1024 slots, the fewest that two parts are made of, 110 / 101.
struct SliGradSplit { int32_t full, parts, items; };
inline SliGradSplit sli_grad_split(int64_t items, int64_t slots) {
  const int64_t sms = 148, rest = items % sms;
  const int64_t parts = rest == 0 ? 1 : std::min<int64_t>(std::min<int64_t>(kSgMaxParts, sms / rest), slots / (4 * kSlKeys));
  if (parts < 2) return SliGradSplit{(int32_t)items, 1, (int32_t)items};
  return SliGradSplit{(int32_t)(items - rest), (int32_t)parts, (int32_t)(items - rest + rest * parts)};
}
// Bytes that the parts leave their sums in, at the end of the workspace: without room for them the rows stay whole, so
// that a workspace made for a larger call is enough for a smaller one with a thinner last round.
inline size_t sli_grad_part_bytes(const DsaSliGradParams* p) {
  if (p->d_idx != 128) return 0;
  const SliGradSplit sp = sli_grad_split((int64_t)p->batch * p->s1 * ((p->g + 63) / 64), p->dense ? p->s2 : p->topk);
  return (size_t)(sp.items - sp.full) * kSgPart * sizeof(float);
}

// Workspaces of the operator reach these kernels with 16-byte aligned rows; what is asked for here is what
// TMA wants of the caller's tensors.
inline bool sli_sm100_aligned(const DsaSliGradParams* p) {
  return (((uintptr_t)p->query | (uintptr_t)p->query_rope | (uintptr_t)p->key | (uintptr_t)p->key_rope |
           (uintptr_t)p->query_index | (uintptr_t)p->key_index) & 15u) == 0 &&
         p->kernel != DSA_KERNEL_PORTABLE && (int64_t)p->batch * p->s2 < (1ll << 31) - 1 &&
         (int64_t)p->batch * p->s1 < (1ll << 24);
}

inline int sli_sm100_prepare(int* sms_out) {
  static std::atomic<int> sm_count[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return DSA_ERR_CUDA;
  int sms = sm_count[dev].load(std::memory_order_acquire);
  if (sms == 0) {
    // (idempotent: two threads that get here together do the same thing)
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1 ||
        cudaFuncSetAttribute(sli_score_sm100_kernel<true, false>, attr, (int)kSlSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(sli_score_sm100_kernel<true, true>, attr, (int)kSlSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(sli_score_sm100_kernel<false, false>, attr, (int)kSlSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(sli_mha_sm100_kernel, attr, (int)kMhSmemBytes) != cudaSuccess)
      return DSA_ERR_CUDA;
    const void* grads[] = {(const void*)sli_grad_sm100_kernel<__nv_bfloat16, false>,
                           (const void*)sli_grad_sm100_kernel<__nv_bfloat16, true>,
                           (const void*)sli_grad_sm100_kernel<__half, false>,
                           (const void*)sli_grad_sm100_kernel<__half, true>};
    for (const void* f : grads) {
      // (a build with another register count must not run: setmaxnreg.inc could block for good)
      cudaFuncAttributes fa;
      if (cudaFuncSetAttribute(f, attr, (int)kSgSmemBytes) != cudaSuccess || cudaFuncGetAttributes(&fa, f) != cudaSuccess ||
          fa.numRegs != kSgLaunchRegs)
        return DSA_ERR_CUDA;
    }
    sm_count[dev].store(sms, std::memory_order_release);
  }
  *sms_out = sms;
  return DSA_OK;
}

// One side's scores into d.p_buf (attention, one key head) or d.di (index).  More than 128 heads are added
// chunk by chunk: the buffer must then be zero.
inline bool sli_score_needs_zero(int heads) { return heads > 128; }
inline int sli_score_sm100_launch(const DsaSliGradParams* p, const SliGradDev& d, bool att, int32_t* status, int sms,
                                  cudaStream_t st) {
  const bool bf16 = p->dtype == DSA_DTYPE_BF16;
  const int64_t rows = (int64_t)p->batch * p->s1;
  SliScoreArgs a;
  a.p = d;
  a.status = status;
  a.out = att ? d.p_buf : d.di;
  a.heads = att ? p->n1 : p->g;
  const int wa = att ? p->d : p->d_idx, wb = att ? p->d_rope : 0;
  a.nblk_a = wa / 64;
  a.nblk = a.nblk_a + wb / 64;
  a.hp = std::min(128, (a.heads + 15) / 16 * 16);
  a.hchunks = (a.heads + a.hp - 1) / a.hp;
  // about six items per SM keep the last wave short (512 rows: 7 rounds of half rows instead of 4 of whole
  // ones); a part still walks over two tiles or more, or loading Q would weigh
  const int64_t most = std::max<int64_t>(1, d.topk / (2 * kSlKeys));
  a.parts = (int32_t)std::max<int64_t>(1, std::min<int64_t>(most, (6 * sms + rows * a.hchunks - 1) / (rows * a.hchunks)));
  if (rows * a.hchunks * a.parts >= (1ll << 31)) return DSA_ERR_TOO_LARGE;
  a.items = (int32_t)(rows * a.hchunks * a.parts);
  a.idesc = ptx::idesc_f16(bf16 ? 1u : 0u, 128, (uint32_t)a.hp, 0, 0);
  const uint32_t qbytes = (uint32_t)a.nblk * a.hp * 128, tail = 2 * 128 * 8 + 512;
  // (the ring starts on a 1024-byte boundary: hp * 128 is a multiple of 2048)
  a.off_k = qbytes;
  a.stages = (int32_t)std::min<uint32_t>(kScMaxStages, (kSlSmemMax - tail - qbytes) / kSlKBlk) & ~1;
  if (a.stages < kScGatherWarps / 2 || a.nblk < 2) return DSA_ERR_TOO_LARGE;   // (nblk: 2 to 9, nine leave four)
  a.off_prm = a.off_k + a.stages * kSlKBlk;
  a.off_bar = a.off_prm + 2 * 128 * 8;
  const uint32_t smem = a.off_bar + 512;
  const void *ka = att ? p->key : p->key_index, *kb = wb ? p->key_rope : ka;
  const void *qa = att ? p->query : p->query_index, *qb = wb ? p->query_rope : qa;
  const int wkb = wb ? wb : wa;
  a.ka = ka; a.kb = kb;
  CUtensorMap tqa, tqb;
  if (!make_tmap_3d_16bit(&tqa, qa, (uint64_t)rows, (uint64_t)a.heads, wa, wa * 2, (uint64_t)a.heads * wa * 2, a.hp, 64,
                          bf16) ||
      !make_tmap_3d_16bit(&tqb, qb, (uint64_t)rows, (uint64_t)a.heads, wkb, wkb * 2, (uint64_t)a.heads * wkb * 2, a.hp, 64,
                          bf16))
    return DSA_ERR_CUDA;
  const int grid = std::min(a.items, sms);
  if (!att) sli_score_sm100_kernel<false, false><<<grid, kScThreads, smem, st>>>(tqa, tqb, a);
  else if (a.heads % a.hp) sli_score_sm100_kernel<true, true><<<grid, kScThreads, smem, st>>>(tqa, tqb, a);
  else sli_score_sm100_kernel<true, false><<<grid, kScThreads, smem, st>>>(tqa, tqb, a);
  if (cudaGetLastError() != cudaSuccess) return DSA_ERR_CUDA;
  count_launch();
  return DSA_OK;
}

// Dense, as many key heads as query heads.  Parts of the heads add into the (zeroed) buffer.
inline SliMhaArgs sli_mha_args(const DsaSliGradParams* p, const SliGradDev& d, int sms) {
  SliMhaArgs a;
  a.p = d;
  a.status = nullptr;
  a.nblk_a = p->d / 64;
  a.nblk = a.nblk_a + p->d_rope / 64;
  a.rtiles = (p->s1 + 127) / 128;
  a.ktiles = (p->s2 + kSlKeys - 1) / kSlKeys;
  const int64_t tiles = (int64_t)p->batch * a.rtiles * a.ktiles;
  a.parts = tiles * 2 > sms ? 1 : (int32_t)std::min<int64_t>(p->n1, sms / tiles);
  a.items = (int32_t)std::min<int64_t>(tiles * a.parts, 0x7FFFFFFF);
  a.idesc = ptx::idesc_f16(p->dtype == DSA_DTYPE_BF16 ? 1u : 0u, 128, kSlKeys, 0, 0);
  return a;
}
inline int sli_mha_sm100_launch(const DsaSliGradParams* p, SliMhaArgs a, int32_t* status, int sms, cudaStream_t st) {
  const bool bf16 = p->dtype == DSA_DTYPE_BF16;
  a.status = status;
  const void *kb = p->d_rope ? p->key_rope : p->key, *qb = p->d_rope ? p->query_rope : p->query;
  const int wa = p->d, wb = p->d_rope ? p->d_rope : p->d;
  const uint64_t qrows = (uint64_t)p->batch * p->s1, krows = (uint64_t)p->batch * p->s2, n = (uint64_t)p->n1;
  CUtensorMap tka, tkb, tqa, tqb;
  if (!make_tmap_3d_16bit(&tka, p->key, n, krows, wa, n * wa * 2, wa * 2, kSlKeys, 64, bf16) ||
      !make_tmap_3d_16bit(&tkb, kb, n, krows, wb, n * wb * 2, wb * 2, kSlKeys, 64, bf16) ||
      !make_tmap_3d_16bit(&tqa, p->query, n, qrows, wa, n * wa * 2, wa * 2, 128, 64, bf16) ||
      !make_tmap_3d_16bit(&tqb, qb, n, qrows, wb, n * wb * 2, wb * 2, 128, 64, bf16))
    return DSA_ERR_CUDA;
  sli_mha_sm100_kernel<<<std::min(a.items, sms), kMhThreads, kMhSmemBytes, st>>>(tka, tkb, tqa, tqb, a);
  if (cudaGetLastError() != cudaSuccess) return DSA_ERR_CUDA;
  count_launch();
  return DSA_OK;
}

template <typename T>
inline int sli_grad_sm100_launch(const DsaSliGradParams* p, const SliGradDev& d, float* part, SliGradParts* parts,
                                 int32_t* status, int sms, cudaStream_t st) {
  const bool bf16 = p->dtype == DSA_DTYPE_BF16;
  const int64_t rows = (int64_t)p->batch * p->s1;
  SliGradArgs a;
  a.p = d;
  a.status = status;
  a.di_max = d.di_max;
  a.hchunks = (p->g + 63) / 64;
  if (rows * a.hchunks >= (1ll << 31)) return DSA_ERR_TOO_LARGE;
  const int64_t whole = rows * a.hchunks;
  const SliGradSplit sp = part ? sli_grad_split(whole, p->dense ? p->s2 : p->topk)
                               : SliGradSplit{(int32_t)whole, 1, (int32_t)whole};
  a.items = sp.items; a.full = sp.full; a.parts = sp.parts;
  a.part = part;
  a.key_rows = (int32_t)((int64_t)p->batch * p->s2);
  const uint32_t fmt = bf16 ? 1u : 0u;
  a.idesc_s = ptx::idesc_f16(fmt, 128, 64, 0, 0);
  a.idesc_k = ptx::idesc_f16(fmt, 128, kSlKeys, 1, 0);
  a.idesc_q = ptx::idesc_f16(fmt, 128, 64, 1, 1);
  CUtensorMap tk, tq;
  if (!make_tmap_gather4_16bit(&tk, p->key_index, (uint64_t)a.key_rows, 128, 256, 64, bf16) ||
      !make_tmap_3d_16bit(&tq, p->query_index, (uint64_t)rows, (uint64_t)p->g, 128, 256, (uint64_t)p->g * 256, 64, 64, bf16))
    return DSA_ERR_CUDA;
  const int grid = std::min(a.items, sms);
  if (sp.parts > 1) sli_grad_sm100_kernel<T, true><<<grid, kSgThreads, kSgSmemBytes, st>>>(tk, tq, a);
  else sli_grad_sm100_kernel<T, false><<<grid, kSgThreads, kSgSmemBytes, st>>>(tk, tq, a);
  if (cudaGetLastError() != cudaSuccess) return DSA_ERR_CUDA;
  count_launch();
  if (sp.parts > 1) *parts = SliGradParts{part, sp.full, sp.parts, (sp.items - sp.full) / sp.parts, a.hchunks};
  return DSA_OK;
}

}  // namespace dsa
