// Sparse flash attention backward on tcgen05 tensor cores for D = 512 (+ 64 rope), one KV head, 16
// heads or more, BSND / TND, token- or block-wise indices.  Same math as sfa_bwd_mma_kernel
// (sparse_flash_attention_grad_triton.py:100-470, golden sparse_flash_attention_grad_numpy.py:96-135):
//     S  = q . k^T          dP = dO . k_nope^T
//     P  = exp(S * scale - max) / sum       dS = P * (dP - delta) * scale
//     dQ += dS . k          dK += dS^T . q  dV += P^T . dO
//
// What it is built around: the scatter-adds.  A selected (row, key) pair adds 1088 fp32 values to d_key /
// d_value, 4.56 GB for 512 rows x 2048 keys x 64 heads, and the L2 takes whole-line fp32 reductions at
// 6.2 TB/s (lanes that cover 32-byte sectors only: 3.7 TB/s) whichever instruction brings them (scalar,
// 16-byte or bulk).  So a block covers 64 heads - every reduction then carries 64 heads - and everything
// else is arranged to run beside the stream of reductions:
//
//   * A work item is (query row, 64 heads).  Q and dO stay in shared memory for the whole row (136 KB),
//     keys come 48 at a time (cp.async, 54 KB, one buffer: 1.26 -> 1.22 ms and 7.54 -> 7.37 ms for the calls below
//     against TMA gather4, which takes 3700 cycles from a free buffer to a full one, the copies 1700).
//   * Q and dO are stacked: feature block f of both forms one 128-row A operand, so that ONE product
//     with the key tile yields S (lanes 0..63) and dP (lanes 64..127).  The rope part of S goes to
//     columns of its own (its lower 64 rows are whatever follows in shared memory; nobody reads them).
//   * The three gradient products run transposed, FEATURES on the 128 lanes: dV^T and dK^T tiles of
//     128 features x 48 keys, dQ^T tiles of 128 features x 64 heads.  A warp that drains a dV^T / dK^T
//     tile holds 32 consecutive features of one key per register: its reduction instruction is one full
//     128-byte line.  Q, dO and K serve these products as transposed (MN-major) operands straight from
//     the layout the score product uses.
//   * P and dS are fp32 values that enter their products as a high and a low io-dtype part
//     (x = hi + lo up to 2^-16 relative for bf16, 2^-22 for fp16), as in sfa_bwd_mma_kernel.  fp16: P is
//     scaled by 2^13, dS by a power of two per item that keeps |dS| <= scale * (|dO| |v| + |delta|)
//     (Cauchy-Schwarz over the item's heads and selected keys, taken by small kernels in front) below 2^13.
//
// Measured, whole operator call: B1 S1 512 S2 4096 N1 64 k 2048 in bf16 1.14 ms (sfa_bwd_mma_kernel: 4.63 ms); 4092
// rows x 128 heads in bf16 7.3-7.4 ms back to back under the power cap (32.2 ms), 7.1 as single calls a second apart.
// A tile of 48 keys takes 12 400 cycles: its reductions alone would take 8400, its products 8000.  What is left is
// the chain of a tile (keys 1700, S 2200, P and dS 5500, of which 1600 wait for dK of the tile before, dQ 2100) beside
// the chain of the dV / dK tiles (issue 6400, ring slots 3100), and the reload of Q / dO between items.
// ptxas spills 0 bytes (bf16) and 32 bytes (fp16) of a thread's 72 registers.
//
// Tensor memory: dQ^T 5 x 64 columns | S, dP 48 | rope part of S 48 | drain ring 2 x 48.
// Warps (896 threads): 0..7 softmax (lane quarter = warp & 3: quarters 0, 1 hold S of heads 0..63,
// quarters 2, 3 hold dP; warps 0..3 take keys 0..23, warps 4..7 keys 24..47), 8..19 drain (three groups
// take the tiles in turn: a group empties its ring slot into registers at once, so that three tiles are
// being added while two are being computed), 20..24 K gather, 25 issuer of S / dP / dQ, 26 issuer of
// dV / dK, 27 Q / dO loader.  Waits suspend (try_wait): polling warps take the load / store unit's issue
// slots from the reductions (1.47 -> 1.36 ms).
// All waits are bounded; one that gives up sets the status word.
#pragma once

#include "sfa_bwd_simt.cuh"
#include "sfa_fwd_sm100.cuh"

namespace dsa {

constexpr int kBwdHeads = 64;        // heads per item
constexpr int kBwdBK = 48;           // keys per tile
constexpr int kBwdThreads = 896;
constexpr int kBwdDrainWarp0 = 8, kBwdDrainGroups = 3, kBwdGatherWarp0 = 20, kBwdGatherWarps = 5;
constexpr int kBwdIssueA = 25, kBwdIssueB = 26, kBwdLoader = 27;
constexpr uint32_t kBwdHBlk = kBwdHeads * 128;                    // 64 heads x 64 features
constexpr uint32_t kBwdQdBlk = 2 * kBwdHBlk;                      // [Q block | dO block]
constexpr uint32_t kBwdKBlk = kBwdBK * 128;                       // 48 keys x 64 features
constexpr uint32_t kBwdPMat = kBwdBK * 128;                       // 48 keys x 64 heads, 16 bit
constexpr uint32_t kBwdOffQd = 0;                                 // 8 x [Q | dO]
constexpr uint32_t kBwdOffQr = kBwdOffQd + 8 * kBwdQdBlk;
constexpr uint32_t kBwdOffK = kBwdOffQr + kBwdHBlk;               // 9 blocks
constexpr uint32_t kBwdOffP = kBwdOffK + 9 * kBwdKBlk;            // P hi, P lo, dS hi, dS lo
constexpr uint32_t kBwdOffX = kBwdOffP + 4 * kBwdPMat;            // P as fp32 [48 keys][64 heads]
constexpr uint32_t kBwdOffBar = kBwdOffX + kBwdBK * kBwdHeads * 4;
constexpr uint32_t kBwdOffRows = kBwdOffBar + 256;               // int32 [3][48]: key rows of the last tiles
constexpr uint32_t kBwdSmemBytes = kBwdOffRows + 3 * kBwdBK * 4;
constexpr uint32_t kBwdQBytes = 8 * kBwdQdBlk + kBwdHBlk;
static_assert(kBwdOffK % 1024 == 0 && kBwdOffP % 1024 == 0, "operand alignment");
static_assert(kBwdSmemBytes <= 232448, "shared memory");
// the drain warps take the registers that the gather, issuer and loader warps give back
constexpr int kBwdLaunchRegs = 72, kBwdRegsLow = 56, kBwdRegsHigh = 80;
static_assert((kBwdRegsHigh - kBwdLaunchRegs) * (kBwdGatherWarp0 - kBwdDrainWarp0) <=
                  (kBwdLaunchRegs - kBwdRegsLow) * (kBwdThreads / 32 - kBwdGatherWarp0),
              "setmaxnreg: more registers requested than released");
static_assert(kBwdLaunchRegs * kBwdThreads <= 65536, "register file");
constexpr uint32_t kBwdTmQ = 0, kBwdTmS = 320, kBwdTmR = 368, kBwdTmD = 416;
constexpr int kBwdTiles = 9;         // dV^T tiles 0..3, dK^T tiles 4..8 (8: rope)

struct SfaBwdArgs {
  SfaGradDev p;
  int32_t* status;
  const int2* nvalid;        // [rows] .x slots that take part, .y first entry in key_list
  const int32_t* key_list;   // [rows, slots] their key rows, front-packed, all in [0, key_rows)
  const float* delta;        // [rows, n1]
  const int32_t* exps;       // fp16: [items] exponent of the power of two that the item's dS is scaled by
  uint32_t idesc_s, idesc_q, idesc_d;
  int32_t items, hblocks;    // rows * hblocks, the last ones cut into parts (SfaBwdSplit)
  int32_t full, parts;
  float* dq_part;            // [items - full][64 heads][576]
  int32_t key_rows;
};
// Parts that a row with `tiles` tiles is cut into, at most `parts`, all of them with keys: of 2 tiles or more when rows
// are cut in two, of a tile in three or four.  A part loads Q and dO again (136 KB), which costs less the fewer blocks do
// it.  Whole calls, rows whole / parts of a tile / of two (a kernel of its own for the sums would add 3 to 7), us:
//    45 rows, in three  16 heads: 90 keys 38 / 39 / 38,    140 43 / 38 / 45, 240 53 / 41 / 45;  64 heads: 140 45 / 39 / 47
//   222, 74 of them in two  16 heads: 90 keys 58 / 55 / 58, 190 83 / 73 / 73; 64 heads: 90 62 / 64 / 64, 190 89 / 84 / 84
//   500, 56 of them in two  64 heads: 90 keys 115 / 119 / 116, 190 168 / 165 / 164; with parts of three tiles 169
__device__ __forceinline__ int32_t bwd_row_parts(int32_t tiles, int32_t parts) {
  if (parts == 1) return 1;
  const int32_t n = max(1, min(parts, tiles / (parts == 2 ? 2 : 1))), per = max(1, (tiles + n - 1) / n);
  return max(1, (tiles + per - 1) / per);
}
struct BwdItem { int32_t base, row, h0, slot; int2 nv; };
// Work item `i`: its (row, 64 heads), its share of the row's list, and its place in dq_part (-1: the whole row, -2:
// nothing to do, the row has fewer parts).
__device__ __forceinline__ BwdItem bwd_item(const SfaBwdArgs& a, int32_t i) {
  BwdItem it;
  it.base = i;
  it.slot = i - a.full;
  int32_t part = 0;
  if (it.slot >= 0) {
    const int32_t r = it.slot / a.parts;
    part = it.slot - r * a.parts;
    it.base = a.full + r;
  } else {
    it.slot = -1;
  }
  it.row = it.base / a.hblocks;
  it.h0 = (it.base - it.row * a.hblocks) * kBwdHeads;
  it.nv = a.nvalid[it.row];
  if (it.slot >= 0) {
    const int32_t tiles = (it.nv.x + kBwdBK - 1) / kBwdBK, n = bwd_row_parts(tiles, a.parts);
    if (part >= n) {
      it.slot = -2;
      it.nv.x = 0;
    } else if (n == 1) {
      it.slot = -1;
    } else {
      const int32_t per = (tiles + n - 1) / n * kBwdBK;
      it.nv.x = min(per, it.nv.x - part * per);
      it.nv.y += part * per;
    }
  }
  return it;
}

__device__ __forceinline__ void red_add(float* addr, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void red_add_if(bool on, float* addr, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}\n" ::"l"(addr),
               "f"(v), "r"((int)on)
               : "memory");
}

// delta = dO . O per (row, head), one warp each; for fp16 also the item's largest |dO| and |delta|, and, by the
// warps past the last pair, the norm of the value part of each key.  A head with an Inf or NaN in either is left
// out of the bounds (its own gradients are lost, those of the other heads keep their scale), and the norm of a
// key that is not finite is 0.
template <typename T>
__global__ void __launch_bounds__(256) sfa_bwd_delta_kernel(const T* __restrict__ d_out, const T* __restrict__ out,
                                                            float* __restrict__ delta, float* __restrict__ bound,
                                                            int64_t total, int32_t n1, int32_t hblocks,
                                                            const T* __restrict__ key, float* __restrict__ norms,
                                                            int64_t key_rows) {
  const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const bool pair = i < total;
  if (!pair && i - total >= key_rows) return;
  const T* x_row = pair ? d_out + i * 512 : key + (i - total) * 512;
  const T* y_row = pair ? out + i * 512 : x_row;
  float s = 0.f, n = 0.f;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint4 a = reinterpret_cast<const uint4*>(x_row)[lane + 32 * u];
    const uint4 b = reinterpret_cast<const uint4*>(y_row)[lane + 32 * u];
    const T* av = reinterpret_cast<const T*>(&a);
    const T* bv = reinterpret_cast<const T*>(&b);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float x = to_f32<T>(av[e]);
      s = fmaf(x, to_f32<T>(bv[e]), s);
      n = fmaf(x, x, n);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if (lane != 0) return;
  if (!pair) {
    norms[i - total] = n < INFINITY ? sqrtf(n) : 0.f;
    return;
  }
  delta[i] = s;
  if (bound != nullptr && n < INFINITY && fabsf(s) < INFINITY) {
    // (non-negative floats order like their bit patterns)
    const int64_t row = i / n1, item = row * hblocks + (i - row * n1) / kBwdHeads;
    atomicMax(reinterpret_cast<int*>(bound + 2 * item), __float_as_int(sqrtf(n)));
    atomicMax(reinterpret_cast<int*>(bound + 2 * item + 1), __float_as_int(fabsf(s)));
  }
}

// fp16: the exponents of a row's items, a block per row.  Only the keys that the row selected count: what a key tensor
// holds elsewhere (padding past the valid lengths, keys of other sequences) may be anything.
__global__ void __launch_bounds__(256) sfa_bwd_exponent_kernel(const int2* __restrict__ nvalid,
                                                               const int32_t* __restrict__ key_list,
                                                               const float* __restrict__ norms,
                                                               const float* __restrict__ bound,
                                                               int32_t* __restrict__ exps, int32_t hblocks, float scale) {
  __shared__ float red[8];
  const int32_t row = blockIdx.x;
  const int2 nv = nvalid[row];
  const int32_t* list = key_list + nv.y;
  float m = 0.f;
#pragma unroll 8
  for (int32_t j = threadIdx.x; j < nv.x; j += 256) m = fmaxf(m, norms[list[j]]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
  for (int32_t h = threadIdx.x; h < hblocks; h += 256) {
    const int64_t item = (int64_t)row * hblocks + h;
    const float b = fabsf(scale) * fmaf(bound[2 * item], m, bound[2 * item + 1]);
    exps[item] = b > 0.f && b < INFINITY ? max(-100, min(100, 12 - ilogbf(b))) : 0;
  }
}

template <typename T>
__global__ void __launch_bounds__(kBwdThreads, 1)
sfa_bwd_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_qr,
                     const __grid_constant__ CUtensorMap tmap_do, const SfaBwdArgs a) {
  constexpr bool kScaled = !kIsBf16<T>;
  extern __shared__ __align__(1024) unsigned char bwd_sm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(bwd_sm + kBwdOffBar);
  uint64_t* k_full = bars;          // gather -> issuer A                                 (128 lanes' copies, rows_s)
  uint64_t* k_empty = bars + 1;     // dQ of the tile done -> gather                      (commit A)
  uint64_t* q_full = bars + 2;      // Q, dO landed -> issuer A (issuer B follows it)     (tx bytes)
  uint64_t* q_empty = bars + 3;     // both issuers through with the item -> loader       (commits A, B)
  uint64_t* s_full = bars + 4;      // S, dP -> softmax                                   (commit A)
  uint64_t* s_empty = bars + 5;     // softmax holds them in registers                    (8 warps)
  uint64_t* p_full = bars + 6;      // P hi / lo stored                                   (4 warps)
  uint64_t* p_empty = bars + 7;     // dV of the tile done                                (commit B)
  uint64_t* ds_full = bars + 8;     // dS hi / lo stored                                  (4 warps)
  uint64_t* ds_empty = bars + 9;    // dK and dQ of the tile done                         (commits A, B)
  uint64_t* x_full = bars + 10;     // [4] fp32 P handed from an S warp to its dP warp
  uint64_t* x_empty = bars + 14;    // [4]
  uint64_t* d_full = bars + 18;     // [3] the drain group's next dV^T / dK^T tile is there (commit B)
  uint64_t* d_empty = bars + 21;    // [2] ring slot read                                 (4 warps)
  uint64_t* dq_full = bars + 23;    // dQ^T of the item complete                          (commit A)
  uint64_t* dq_empty = bars + 24;   // dQ^T read                                          (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 25);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 26);
  int32_t* rows_s = reinterpret_cast<int32_t*>(bwd_sm + kBwdOffRows);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t n1 = a.p.n1;
  const bool misaligned = (ptx::smem_u32(bwd_sm) & 1023u) != 0;
  if (threadIdx.x == 0) {
    const int counts[25] = {4 * 32 + 1, 1, 1, 2, 1, 8, 4, 1, 4, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 4, 4, 1, 8};
#pragma unroll
    for (int i = 0; i < 25; ++i) ptx::mbar_init(&bars[i], counts[i]);
    *abort_flag = misaligned ? 1 : 0;
    ptx::mbar_fence_init();
  }
  // (the operands' padding is read by products whose results nobody uses, and by those of the heads past
  // n1, which have to be zero: start from zeros)
  for (uint32_t i = threadIdx.x; i < (kBwdOffBar - kBwdOffK) / 16; i += kBwdThreads)
    reinterpret_cast<uint4*>(bwd_sm + kBwdOffK)[i] = make_uint4(0, 0, 0, 0);
  ptx::fence_proxy_async_smem();
  if (warp == kBwdIssueA) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sm0 = ptx::smem_u32(bwd_sm);

  auto tiles_of = [&](int32_t n) -> int32_t { return (n + kBwdBK - 1) / kBwdBK; };
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::mbar_wait_warp(bar, parity, abort_flag); };

  // Each class of roles sits in its own branch, right under its setmaxnreg: the compiler budgets a
  // branch by the setmaxnreg that dominates it.
  if (warp < kBwdDrainWarp0) {
   if (!*abort_flag) {
    // -------------------------------------------------------------------- softmax, then dQ^T
    const int quarter = warp & 3, half = warp >> 2;
    const bool is_s = quarter < 2;
    const int hl = (quarter & 1) * 32 + lane;               // head within the item
    const int pair = (quarter & 1) * 2 + half;
    const int kk0 = half * 24;                              // this warp's keys of a tile
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    unsigned char* mat_hi = bwd_sm + kBwdOffP + (is_s ? 0u : 2u * kBwdPMat) + (hl & 7) * 2;
    float* xbuf = reinterpret_cast<float*>(bwd_sm + kBwdOffX) + hl;
    uint32_t n_tile = 0, n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const BwdItem it = bwd_item(a, item);
      if (it.slot == -2) continue;
      const int32_t row = it.row, h0 = it.h0, nvalid = it.nv.x, ntiles = tiles_of(nvalid);
      const bool head = h0 + hl < n1;
      const int64_t hi_ = (int64_t)row * n1 + h0 + hl;
      if (ntiles > 0) {
        float c0 = 0.f, c1 = 0.f, up = 1.f;                 // S: max, 1 / sum; dP: delta
        if (head) {
          if (is_s) {
            c0 = a.p.softmax_max[hi_];
            const float l = a.p.softmax_sum[hi_];
            c1 = l > 0.f ? 1.f / l : 0.f;
          } else {
            c0 = a.delta[hi_];
          }
        }
        // (a head without a sum, or past the last one, has P = 0 whatever its scores are)
        const int32_t nlive = !is_s || c1 > 0.f ? nvalid : 0;
        if constexpr (kScaled) up = is_s ? 8192.f : scalbnf(1.f, a.exps[it.base]);
        for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
          const uint32_t ph = n_tile & 1;
          ok = wait(s_full, ph);
          if (!ok) break;
          ptx::tc_fence_after();
          float v[24];
          ptx::tmem_ld_x16(lane_addr + kBwdTmS + kk0, reinterpret_cast<uint32_t*>(v));
          ptx::tmem_ld_x8(lane_addr + kBwdTmS + kk0 + 16, reinterpret_cast<uint32_t*>(v + 16));
          if (is_s) {
            float r[24];
            ptx::tmem_ld_x16(lane_addr + kBwdTmR + kk0, reinterpret_cast<uint32_t*>(r));
            ptx::tmem_ld_x8(lane_addr + kBwdTmR + kk0 + 16, reinterpret_cast<uint32_t*>(r + 16));
            ptx::tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 24; ++k) v[k] += r[k];
          } else {
            ptx::tmem_ld_wait();
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(s_empty);
          const int32_t cnt = nlive - t * kBwdBK - kk0;     // keys among this warp's 24 that take part
          if (is_s) {
            // (exp of a sum beside 1 / sum: against 64 bits P is off by 1.7e-7 (rms), expf(..) / sum by 1.1e-7.  Its
            // share shows in neither the fp32 sums of d_key - fp16, 64 heads, k 1024: 8.1e-7 and 7.8e-7, most of
            // it from the 512-feature score products - nor in the results, 2.0692e-4 and 2.0692e-4 from their one
            // rounding; four S warps have this tile's exponentials to themselves, and expf takes 1262 us to 1584.)
#pragma unroll
            for (int k = 0; k < 24; ++k)
              v[k] = k < cnt ? ex2(fmaf(v[k], a.p.scale, -c0) * 1.4426950408889634f) * c1 : 0.f;
            ok = wait(&x_empty[pair], ph ^ 1);
            if (!ok) break;
#pragma unroll
            for (int k = 0; k < 24; ++k) xbuf[(kk0 + k) * kBwdHeads] = v[k];
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&x_full[pair]);
            ok = wait(p_empty, ph ^ 1);
          } else {
            ok = wait(&x_full[pair], ph);
            if (!ok) break;
#pragma unroll
            for (int k = 0; k < 24; ++k) v[k] = xbuf[(kk0 + k) * kBwdHeads] * (v[k] - c0) * a.p.scale;
            if (cnt < 24) {
#pragma unroll
              for (int k = 0; k < 24; ++k) v[k] = k < cnt ? v[k] : 0.f;
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&x_empty[pair]);
            ok = wait(ds_empty, ph ^ 1);
          }
          if (!ok) break;
#pragma unroll
          for (int k = 0; k < 24; ++k) {
            const float x = kScaled ? v[k] * up : v[k];
            const T hi = from_f32<T>(x);
            unsigned char* dst = mat_hi + (kk0 + k) * 128 + (((hl >> 3) ^ (k & 7)) << 4);   // (24 is a multiple of 8)
            *reinterpret_cast<T*>(dst) = hi;
            *reinterpret_cast<T*>(dst + kBwdPMat) = from_f32<T>(x - to_f32<T>(hi));
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(is_s ? p_full : ds_full);
        }
        if (!ok) break;
        ok = wait(dq_full, n_item & 1);
        if (!ok) break;
        ptx::tc_fence_after();
      }
      // dQ^T tile m: this thread's feature is m * 128 + quarter * 32 + lane, a column is a head
      float down = 1.f;
      if constexpr (kScaled) { if (ntiles > 0) down = scalbnf(1.f, -a.exps[it.base]); }
      const int32_t hn = min(kBwdHeads, n1 - h0);
#pragma unroll 1
      for (int m = half; m < 5; m += 2) {
        const int f = quarter * 32 + lane;
        if (m == 4 && quarter >= 2) continue;
        T* dst = m < 4 ? (T*)a.p.d_query + ((int64_t)row * n1 + h0) * 512 + m * 128 + f
                       : (T*)a.p.d_query_rope + ((int64_t)row * n1 + h0) * 64 + f;
        const int step = m < 4 ? 512 : 64;
#pragma unroll 1
        for (int c = 0; c < kBwdHeads; c += 16) {
          if (c >= hn) break;
          float o[16];
          if (ntiles > 0) {
            ptx::tmem_ld_x16(lane_addr + kBwdTmQ + m * 64 + c, reinterpret_cast<uint32_t*>(o));
            ptx::tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = 0.f;
          }
          if (it.slot < 0) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c + i < hn) dst[(int64_t)(c + i) * step] = from_f32<T>(o[i] * down);
          } else {
            float* part = a.dq_part + ((int64_t)it.slot * kBwdHeads + c) * 576 + m * 128 + f;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c + i < hn) part[i * 576] = o[i] * down;
          }
        }
      }
      if (ntiles > 0) {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(dq_empty);
        ++n_item;
      }
    }
   }
  } else if (warp < kBwdGatherWarp0) {
   asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kBwdRegsHigh));
   if (!*abort_flag) {
    // -------------------------------------------------------------------- drain: reductions of dV^T / dK^T
    const int quarter = warp & 3, group = (warp - kBwdDrainWarp0) >> 2;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16) + kBwdTmD;
    const int f = quarter * 32 + lane;
    uint32_t n_drain = 0, n_mine = 0;
    int turn = 0, rbuf = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const BwdItem it = bwd_item(a, item);
      const int2 nv = it.nv;
      const int32_t ntiles = tiles_of(nv.x);
      float dk_down = 1.f;
      if constexpr (kScaled) { if (ntiles > 0) dk_down = scalbnf(1.f, -a.exps[it.base]); }
      for (int32_t t = 0; t < ntiles && ok; ++t) {
        const int4* rows4 = reinterpret_cast<const int4*>(rows_s + rbuf * kBwdBK);
        rbuf = rbuf == 2 ? 0 : rbuf + 1;
#pragma unroll 1
        for (int m = 0; m < kBwdTiles; ++m, ++n_drain) {
          const bool mine = turn == group;
          turn = turn == kBwdDrainGroups - 1 ? 0 : turn + 1;
          if (!mine) continue;
          const uint32_t slot = n_drain & 1;
          ok = wait(&d_full[group], n_mine++ & 1);
          if (!ok) break;
          ptx::tc_fence_after();
          float v[48];
          ptx::tmem_ld_x16(lane_addr + slot * kBwdBK, reinterpret_cast<uint32_t*>(v));
          ptx::tmem_ld_x16(lane_addr + slot * kBwdBK + 16, reinterpret_cast<uint32_t*>(v + 16));
          ptx::tmem_ld_x16(lane_addr + slot * kBwdBK + 32, reinterpret_cast<uint32_t*>(v + 32));
          ptx::tmem_ld_wait();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&d_empty[slot]);
          if (m == 8 && quarter >= 2) continue;              // the rope tile has 64 features
          const bool is_v = m < 4;
          const int32_t width = is_v ? 512 : 576;
          float* base = is_v ? a.p.dv_acc + m * 128 + f : a.p.dk_acc + (m - 4) * 128 + f;
          const float down = kScaled ? (is_v ? 1.f / 8192.f : dk_down) : 1.f;
          // one instruction = 32 features of one key = one full line
          if (nv.x - t * kBwdBK >= kBwdBK) {                 // whole tile of existing rows: no predicates
#pragma unroll
            for (int kb = 0; kb < kBwdBK; kb += 4) {
              const int4 kr = rows4[kb / 4];
              const int32_t r[4] = {kr.x, kr.y, kr.z, kr.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) red_add(base + (int64_t)r[i] * width, kScaled ? v[kb + i] * down : v[kb + i]);
            }
          } else {
#pragma unroll
            for (int kb = 0; kb < kBwdBK; kb += 4) {
              const int4 kr = rows4[kb / 4];
              const int32_t r[4] = {kr.x, kr.y, kr.z, kr.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                red_add_if(r[i] < a.key_rows, base + (int64_t)r[i] * width, kScaled ? v[kb + i] * down : v[kb + i]);
            }
          }
        }
      }
    }
   }
  } else {
   asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kBwdRegsLow));
   if (*abort_flag) {
    // nothing started
   } else if (warp < kBwdIssueA) {
    // -------------------------------------------------------------------- K gather: four warps take 12 keys each, 9
    // blocks (27 copies per lane, an instruction is 4 keys x 128 bytes); the fifth writes the drain warps' row numbers
    const int gw = warp - kBwdGatherWarp0;
    const int ch = lane & 7, key_w = gw * 12 + (lane >> 3);          // this lane's keys: key_w + 4 j
    const unsigned char* kn = (const unsigned char*)a.p.key + ch * 16;
    const unsigned char* kr = (const unsigned char*)a.p.key_rope + ch * 16;
    uint32_t n_tile = 0;
    int rbuf = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const int2 nv = bwd_item(a, item).nv;
      const int32_t ntiles = tiles_of(nv.x);
      const int32_t* list = a.key_list + nv.y;
      int32_t rn[3] = {0, 0, 0};
      auto load = [&](int32_t t) {
        const int32_t left = nv.x - t * kBwdBK;
        if (left <= 0) return;
        if (gw < 4) {
#pragma unroll
          for (int j = 0; j < 3; ++j) rn[j] = list[t * kBwdBK + (key_w + 4 * j < left ? key_w + 4 * j : 0)];
        } else {
          rn[0] = lane < left ? list[t * kBwdBK + lane] : a.key_rows;
          rn[1] = lane < 16 && 32 + lane < left ? list[t * kBwdBK + 32 + lane] : a.key_rows;
        }
      };
      load(0);
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        int32_t r[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) r[j] = rn[j];
        load(t + 1);
        ok = wait(k_empty, (n_tile & 1) ^ 1);
        if (!ok) break;
        if (gw < 4) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int key = key_w + 4 * j;
            const uint32_t dst = sm0 + kBwdOffK + key * 128 + ((ch ^ (key & 7)) << 4);
            const unsigned char* src = kn + (int64_t)r[j] * 1024;
#pragma unroll
            for (int b = 0; b < 8; ++b) ptx::cp_async_16(dst + b * kBwdKBlk, src + b * 128, 16u);
            ptx::cp_async_16(dst + 8 * kBwdKBlk, kr + (int64_t)r[j] * 128, 16u);
          }
          ptx::cp_async_mbar_arrive(k_full);
        } else {
          // The drain warps' row numbers (past the keys: no such key).  Three buffers: tile t + 3 is gathered
          // after dQ of tile t + 2, i.e. after every dK^T tile of t + 1 was issued and so after every drain
          // group has left tile t behind.
          rows_s[rbuf * kBwdBK + lane] = r[0];
          if (lane < 16) rows_s[rbuf * kBwdBK + 32 + lane] = r[1];
          rbuf = rbuf == 2 ? 0 : rbuf + 1;
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(k_full);
        }
      }
    }
   } else if (warp == kBwdIssueA) {
    // -------------------------------------------------------------------- issuer A: S / dP, then dQ^T
    const uint64_t qd_k = ptx::desc_kmajor_sw128(sm0 + kBwdOffQd), qr_k = ptx::desc_kmajor_sw128(sm0 + kBwdOffQr);
    const uint64_t k_k = ptx::desc_kmajor_sw128(sm0 + kBwdOffK);
    const uint64_t k_m = ptx::desc_mnmajor_sw128(sm0 + kBwdOffK, kBwdKBlk, 1024);
    const uint64_t ds_m = ptx::desc_mnmajor_sw128(sm0 + kBwdOffP + 2 * kBwdPMat, 0, 1024);
    uint32_t n_tile = 0, n_item = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const int32_t ntiles = tiles_of(bwd_item(a, item).nv.x);
      if (ntiles == 0) continue;
      ok = wait(q_full, n_item & 1);
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        const uint32_t ph = n_tile & 1;
        ok = wait(k_full, ph) && wait(s_empty, ph ^ 1);
        if (!ok) break;
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          ptx::fence_proxy_async_smem();   // (the copies went through the generic proxy)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            ptx::mma_ss(tmem + kBwdTmR, qr_k + i * 2, k_k + ((8 * kBwdKBlk) >> 4) + i * 2, a.idesc_s, i ? 1u : 0u);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            ptx::mma_ss(tmem + kBwdTmS, qd_k + (((i >> 2) * kBwdQdBlk) >> 4) + (i & 3) * 2,
                        k_k + (((i >> 2) * kBwdKBlk) >> 4) + (i & 3) * 2, a.idesc_s, i ? 1u : 0u);
          ptx::mma_commit(s_full);
        }
        __syncwarp();
        ok = wait(ds_full, ph) && (t > 0 || wait(dq_empty, (n_item & 1) ^ 1));
        if (!ok) break;
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          ptx::fence_proxy_async_smem();
#pragma unroll
          for (int m = 0; m < 5; ++m)
#pragma unroll
            for (int ks = 0; ks < 3; ++ks)
#pragma unroll
              for (int lo = 0; lo < 2; ++lo)
                ptx::mma_ss(tmem + kBwdTmQ + m * 64, k_m + ((m * 2 * kBwdKBlk + ks * 2048) >> 4),
                            ds_m + ((lo * kBwdPMat + ks * 2048) >> 4), a.idesc_q, (t > 0 || ks > 0 || lo > 0) ? 1u : 0u);
          ptx::mma_commit(k_empty);
          ptx::mma_commit(ds_empty);
          if (t == ntiles - 1) {
            ptx::mma_commit(dq_full);
            ptx::mma_commit(q_empty);
          }
        }
        __syncwarp();
      }
      ++n_item;
    }
   } else if (warp == kBwdIssueB) {
    // -------------------------------------------------------------------- issuer B: dV^T, dK^T
    const uint64_t q_m = ptx::desc_mnmajor_sw128(sm0 + kBwdOffQd, kBwdQdBlk, 1024);
    const uint64_t do_m = ptx::desc_mnmajor_sw128(sm0 + kBwdOffQd + kBwdHBlk, kBwdQdBlk, 1024);
    const uint64_t p_k = ptx::desc_kmajor_sw128(sm0 + kBwdOffP);
    uint32_t n_tile = 0, n_drain = 0;
    int turn = 0;
    bool ok = true;
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const BwdItem it = bwd_item(a, item);
      const int32_t ntiles = tiles_of(it.nv.x);
      if (ntiles == 0) continue;
      const int steps = (min(kBwdHeads, n1 - it.h0) + 15) / 16;       // 16-head steps with real heads
      for (int32_t t = 0; t < ntiles && ok; ++t, ++n_tile) {
        const uint32_t ph = n_tile & 1;
#pragma unroll 1
        for (int m = 0; m < kBwdTiles; ++m, ++n_drain) {
          if (m == 0) ok = wait(p_full, ph);
          if (m == 4) ok = wait(ds_full, ph);
          const uint32_t slot = n_drain & 1;
          ok = ok && wait(&d_empty[slot], ((n_drain >> 1) & 1) ^ 1);
          if (!ok) break;
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
            ptx::fence_proxy_async_smem();
            const uint64_t ad = m < 4 ? do_m + ((m * 2 * kBwdQdBlk) >> 4) : q_m + (((m - 4) * 2 * kBwdQdBlk) >> 4);
            const uint64_t bd = p_k + (m < 4 ? 0 : (2 * kBwdPMat) >> 4);
            const uint32_t dst = tmem + kBwdTmD + slot * kBwdBK;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              if (s < steps) {
                ptx::mma_ss(dst, ad + ((s * 2048) >> 4), bd + s * 2, a.idesc_d, s ? 1u : 0u);
                ptx::mma_ss(dst, ad + ((s * 2048) >> 4), bd + (kBwdPMat >> 4) + s * 2, a.idesc_d, 1u);
              }
            }
            ptx::mma_commit(&d_full[turn]);
            if (m == 3) ptx::mma_commit(p_empty);
            if (m == kBwdTiles - 1) {
              ptx::mma_commit(ds_empty);
              if (t == ntiles - 1) ptx::mma_commit(q_empty);
            }
          }
          turn = turn == kBwdDrainGroups - 1 ? 0 : turn + 1;
          __syncwarp();
        }
      }
    }
   } else if (warp == kBwdLoader) {
    // -------------------------------------------------------------------- Q / dO loader
    uint32_t n_item = 0;
    bool ok = true;
    if (lane == 0) { ptx::prefetch_tmap(&tmap_q); ptx::prefetch_tmap(&tmap_qr); ptx::prefetch_tmap(&tmap_do); }
    for (int32_t item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const BwdItem it = bwd_item(a, item);
      const int32_t row = it.row, h0 = it.h0;
      if (it.nv.x == 0) continue;
      if (lane == 0) {
        ok = ptx::mbar_wait(q_empty, (n_item & 1) ^ 1, abort_flag);
        if (ok) {
          ptx::mbar_arrive_expect_tx(q_full, kBwdQBytes);
#pragma unroll 1
          for (int b = 0; b < 8; ++b) {
            ptx::tma_load_3d(bwd_sm + kBwdOffQd + b * kBwdQdBlk, &tmap_q, q_full, b * 64, h0, row);
            ptx::tma_load_3d(bwd_sm + kBwdOffQd + b * kBwdQdBlk + kBwdHBlk, &tmap_do, q_full, b * 64, h0, row);
          }
          ptx::tma_load_3d(bwd_sm + kBwdOffQr, &tmap_qr, q_full, 0, h0, row);
        }
      } else {
        // the other lanes pull the next item's rows into L2
        const int32_t next = item + gridDim.x;
        if (next < a.items) {
          const BwdItem nx = bwd_item(a, next);
          const int32_t nrow = nx.row, nh0 = nx.h0;
          const int64_t off = ((int64_t)nrow * n1 + nh0) * 1024;
          for (int32_t i = lane - 1; i < min(kBwdHeads, n1 - nh0) * 8; i += 31) {
            ptx::prefetch_l2((const unsigned char*)a.p.query + off + (int64_t)i * 128);
            ptx::prefetch_l2((const unsigned char*)a.p.d_out + off + (int64_t)i * 128);
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      ++n_item;
    }
   }
  }

  // ---------------------------------------------------------------------- teardown
  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies / MMAs in flight land
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kBwdIssueA) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(a.status, misaligned ? 2 : 1);
}

// d_query of the rows that were cut into parts: the parts' sums in their order, rounded once.  A block per item and 8
// heads, in front of the `blocks` blocks of the same kernel that round d_key and d_value (a kernel of its own costs a
// call of short rows, in which there is nothing to add, 3 to 7 us).
constexpr int kBwdMaxParts = 4;
struct SfaBwdParts {
  const int2* nvalid;
  const float* dq_part;
  void *d_query, *d_query_rope;
  int32_t full, parts, items, hblocks, n1;    // items: of 64 heads, that may be cut
};
template <typename T>
__global__ void __launch_bounds__(256) sfa_bwd_finalize_parts_kernel(SfaBwdRounding<T> r, SfaBwdParts s, int32_t blocks) {
  if ((int32_t)blockIdx.x >= s.items * 8) {
    sfa_bwd_finalize(r, (int32_t)blockIdx.x - s.items * 8, blocks);
    return;
  }
  const int32_t item = (int32_t)blockIdx.x >> 3, base = s.full + item, row = base / s.hblocks;
  const int32_t hl0 = ((int32_t)blockIdx.x & 7) * 8, h0 = (base - row * s.hblocks) * kBwdHeads + hl0;
  const int32_t n = bwd_row_parts((s.nvalid[row].x + kBwdBK - 1) / kBwdBK, s.parts), heads = min(8, s.n1 - h0);
  if (n == 1) return;
  const float* src = s.dq_part + ((int64_t)item * s.parts * kBwdHeads + hl0) * 576;
#pragma unroll 5
  for (int32_t i = threadIdx.x; i < heads * 144; i += 256) {
    float4 x[kBwdMaxParts];
#pragma unroll
    for (int32_t q = 0; q < kBwdMaxParts; ++q)
      x[q] = q < n ? reinterpret_cast<const float4*>(src + (int64_t)q * kBwdHeads * 576)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    float v[4] = {x[0].x, x[0].y, x[0].z, x[0].w};
#pragma unroll
    for (int32_t q = 1; q < kBwdMaxParts; ++q) {
      if (q < n) { v[0] += x[q].x; v[1] += x[q].y; v[2] += x[q].z; v[3] += x[q].w; }
    }
    const int32_t h = i / 144, f = (i - h * 144) * 4;
    const int64_t o = (int64_t)row * s.n1 + h0 + h;
    T* dst = f < 512 ? (T*)s.d_query + o * 512 + f : (T*)s.d_query_rope + o * 64 + f - 512;
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = from_f32<T>(v[e]);
  }
}

// ---- host side ---------------------------------------------------------------------------------
// Items of the last round: a round lasts as long as its longest item, so where half of the SMs or more would idle in
// it, its items are cut into 2 to 4 parts, whose d_query is added up afterwards.  This rule goes by the slots, all
// that the host knows (8 tiles of them a part, or more); a row with fewer keys has fewer parts (bwd_row_parts).
// Whole calls of 64 heads, 2048 of 4096 keys, rows of the last round whole / cut, us:
//   first round   1 row 315 / 110,   20 rows 313 / 112,  37 (four parts) 316 / 118,  38 (three) 316 / 140,
//                 49 316 / 144,      50 (two) 316 / 186, 74 316 / 190
//   second        149 rows 609 / 400,  222 615 / 482     third 300 905 / 693     fourth 512 1206 / 1066
//   fourteenth    1925 rows 4139 / 3957, 1998 4266 / 4111 (under the power cap)
// and 222 rows of 768 slots, the fewest that two parts are made of, 261 / 218.  148 SMs are assumed (the workspace is
// sized from it); any other number is still correct.
struct SfaBwdSplit { int32_t full, parts, items; };
inline SfaBwdSplit sfa_bwd_split(int64_t items, int64_t slots) {
  const int64_t sms = 148, rest = items % sms;
  const int64_t parts = rest == 0 ? 1 : std::min<int64_t>(std::min<int64_t>(kBwdMaxParts, sms / rest), slots / (8 * kBwdBK));
  if (parts < 2) return SfaBwdSplit{(int32_t)items, 1, (int32_t)items};
  return SfaBwdSplit{(int32_t)(items - rest), (int32_t)parts, (int32_t)(items - rest + rest * parts)};
}
inline int64_t sfa_bwd_rows(const DsaSfaGradParams* p) {
  return p->layout_q == DSA_LAYOUT_TND ? (int64_t)p->s1 : (int64_t)p->batch * p->s1;
}
// The shapes this kernel takes, given the larger workspace and 16-byte aligned tensors.
inline bool sfa_bwd_sm100_shape(const DsaSfaGradParams* p) {
  if (p->d != 512 || p->d_rope != 64 || p->kernel == DSA_KERNEL_PORTABLE) return false;
  // Fewer than 16 heads: the workspace that dsa_sfa_grad_workspace_bytes names for them is the accumulators alone,
  // a documented figure that callers size from, and this kernel does not fit in it.  Time is not the reason: 512
  // rows x 2048 of 4096 keys, 1 / 8 / 15 heads: mma.sync 1814 / 1818 / 1838 us, this kernel 1185 / 1185 / 1187; at 16
  // and 32 heads 1838 and 2655 us against 1187 and 1220.
  if (p->n1 < 16) return false;
  if (p->key_rows < 1 || p->key_rows >= (1ll << 31) - 1) return false;
  const int64_t rows = sfa_bwd_rows(p);
  if (rows < 1 || rows * ((p->n1 + kBwdHeads - 1) / kBwdHeads) >= (1ll << 31)) return false;
  return rows * p->sparse_count * p->sparse_block_size < (1ll << 31);    // key_list offsets are int32
}
inline bool sfa_bwd_sm100_aligned(const DsaSfaGradParams* p) {
  return (((uintptr_t)p->query | (uintptr_t)p->query_rope | (uintptr_t)p->key | (uintptr_t)p->key_rope |
           (uintptr_t)p->d_out | (uintptr_t)p->out) & 15u) == 0;
}
// Workspace: header | dk / dv accumulators | fp16: bounds of the items - zeroed before the call - | fp16: exponents
// of the items, norms of the keys | nvalid | delta | redo flags and count of the pre-pass (unused) | key_list | d_query
// of parts of rows.  What lies before the parts (`uncut` bytes) grows with every size of the call, the parts come and
// go with its last round: without room for them the rows stay whole, so that a workspace made for a larger call is
// enough for a smaller one.
struct SfaBwdWs { size_t acc, bound, zeroed, exps, norms, nvalid, delta, redo, key_list, uncut, dq_part, total; };
inline SfaBwdWs sfa_bwd_ws_layout(const DsaSfaGradParams* p, size_t header) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  const size_t rows = (size_t)sfa_bwd_rows(p);
  SfaBwdWs w;
  w.acc = header;
  w.bound = w.acc + up((size_t)p->key_rows * (size_t)(2 * p->d + p->d_rope) * sizeof(float));
  const bool fp16 = p->dtype == DSA_DTYPE_FP16;
  const size_t items = rows * ((p->n1 + kBwdHeads - 1) / kBwdHeads);
  w.zeroed = w.bound + (fp16 ? up(items * 2 * 4) : 0);
  w.exps = w.zeroed;
  w.norms = w.exps + (fp16 ? up(items * 4) : 0);
  w.nvalid = w.norms + (fp16 ? up((size_t)p->key_rows * 4) : 0);
  w.delta = w.nvalid + up(rows * 8);
  w.redo = w.delta + up(rows * p->n1 * 4);
  w.key_list = w.redo + up(rows * 4) + 256;
  w.uncut = w.key_list + rows * p->sparse_count * p->sparse_block_size * 4;
  w.dq_part = up(w.uncut);
  const SfaBwdSplit sp = sfa_bwd_split((int64_t)items, (int64_t)p->sparse_count * p->sparse_block_size);
  w.total = sp.parts > 1 ? w.dq_part + (size_t)(sp.items - sp.full) * kBwdHeads * 576 * 4 : w.uncut;
  return w;
}

template <typename T>
inline int sfa_bwd_sm100_launch(const DsaSfaGradParams* p, const SfaGradDev& d, char* ws, size_t ws_bytes,
                                const SfaBwdWs& w, SfaBwdParts* parts, cudaStream_t st) {
  static std::atomic<int> sm_count[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return DSA_ERR_CUDA;
  int sms = sm_count[dev].load(std::memory_order_acquire);
  if (sms == 0) {
    // (idempotent: two threads that get here together do the same thing)
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return DSA_ERR_CUDA;
    if (cudaFuncSetAttribute(sfa_bwd_sm100_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBwdSmemBytes) != cudaSuccess ||
        cudaFuncSetAttribute(sfa_bwd_sm100_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBwdSmemBytes) != cudaSuccess)
      return DSA_ERR_CUDA;
    // (a build with another register count must not run: setmaxnreg.inc could block for good)
    cudaFuncAttributes fa0, fa1;
    if (cudaFuncGetAttributes(&fa0, sfa_bwd_sm100_kernel<__nv_bfloat16>) != cudaSuccess ||
        cudaFuncGetAttributes(&fa1, sfa_bwd_sm100_kernel<__half>) != cudaSuccess || fa0.numRegs != kBwdLaunchRegs ||
        fa1.numRegs != kBwdLaunchRegs)
      return DSA_ERR_CUDA;
    sm_count[dev].store(sms, std::memory_order_release);
  }
  const bool bf16 = p->dtype == DSA_DTYPE_BF16;
  int32_t* status = (int32_t*)ws;
  int2* nvalid = (int2*)(ws + w.nvalid);
  int32_t* key_list = (int32_t*)(ws + w.key_list);
  float* delta = (float*)(ws + w.delta);
  float* bound = bf16 ? nullptr : (float*)(ws + w.bound);
  int32_t* exps = (int32_t*)(ws + w.exps);
  float* norms = (float*)(ws + w.norms);
  int32_t* redo = (int32_t*)(ws + w.redo);
  SfaDev f = {};
  f.seq = d.seq;
  f.sparse_indices = d.sparse_indices;
  f.rows = d.rows;
  f.sparse_count = d.sparse_count; f.sparse_block_size = d.sparse_block_size;
  const int64_t slots = (int64_t)p->sparse_count * p->sparse_block_size;
  // (slots without a row are left out: the reductions of a whole tile go to every listed row unchecked)
  sfa_compact_launch(f, nvalid, key_list, 1, (int32_t)slots, (int32_t)p->key_rows, -1, redo, redo + d.rows, status, st);
  const int64_t pairs = (int64_t)d.rows * p->n1;
  const int32_t hblocks = (p->n1 + kBwdHeads - 1) / kBwdHeads;
  const int64_t norm_rows = bf16 ? 0 : p->key_rows;
  sfa_bwd_delta_kernel<T><<<(unsigned)((pairs + norm_rows + 7) / 8), 256, 0, st>>>(
      (const T*)p->d_out, (const T*)p->out, delta, bound, pairs, p->n1, hblocks, (const T*)p->key, norms, norm_rows);
  if (!bf16)
    sfa_bwd_exponent_kernel<<<d.rows, 256, 0, st>>>(nvalid, key_list, norms, bound, exps, hblocks, p->scale);
  if (cudaGetLastError() != cudaSuccess) return DSA_ERR_CUDA;
  count_launch(bf16 ? 2 : 3);
  SfaBwdArgs a;
  a.p = d;
  a.status = status;
  a.nvalid = nvalid; a.key_list = key_list; a.delta = delta; a.exps = exps;
  const uint32_t fmt = bf16 ? 1u : 0u;
  a.idesc_s = ptx::idesc_f16(fmt, 128, kBwdBK, 0, 0);
  a.idesc_q = ptx::idesc_f16(fmt, 128, kBwdHeads, 1, 1);
  a.idesc_d = ptx::idesc_f16(fmt, 128, kBwdBK, 1, 0);
  a.hblocks = hblocks;
  const int64_t whole = (int64_t)d.rows * hblocks;
  const SfaBwdSplit sp = ws_bytes >= w.total ? sfa_bwd_split(whole, slots)
                                             : SfaBwdSplit{(int32_t)whole, 1, (int32_t)whole};
  a.items = sp.items; a.full = sp.full; a.parts = sp.parts;
  a.dq_part = (float*)(ws + w.dq_part);
  a.key_rows = (int32_t)p->key_rows;
  CUtensorMap tq, tqr, tdo;
  if (!make_tmap_3d_16bit(&tq, p->query, (uint64_t)d.rows, (uint64_t)p->n1, 512, 1024, (uint64_t)p->n1 * 1024, kBwdHeads,
                          64, bf16) ||
      !make_tmap_3d_16bit(&tqr, p->query_rope, (uint64_t)d.rows, (uint64_t)p->n1, 64, 128, (uint64_t)p->n1 * 128,
                          kBwdHeads, 64, bf16) ||
      !make_tmap_3d_16bit(&tdo, p->d_out, (uint64_t)d.rows, (uint64_t)p->n1, 512, 1024, (uint64_t)p->n1 * 1024,
                          kBwdHeads, 64, bf16))
    return DSA_ERR_CUDA;
  const int grid = std::min(a.items, sms);
  sfa_bwd_sm100_kernel<T><<<grid, kBwdThreads, kBwdSmemBytes, st>>>(tq, tqr, tdo, a);
  if (cudaGetLastError() != cudaSuccess) return DSA_ERR_CUDA;
  count_launch();
  if (sp.parts > 1)
    *parts = SfaBwdParts{nvalid, a.dq_part, p->d_query, p->d_query_rope, sp.full, sp.parts, (sp.items - sp.full) / sp.parts,
                         hblocks, p->n1};
  return DSA_OK;
}

}  // namespace dsa
