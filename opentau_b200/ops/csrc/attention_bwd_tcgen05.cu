// Block-causal flash attention backward for sm_100a (tcgen05 + TMEM + TMA) without scratch memory for P and dS: for many samples of one
// tile each, where nothing is recomputed, and for calls of which not even one sample's P and dS find room
// (attention_bwd_stored_tcgen05.cu keeps them and elsewhere takes about half the time).
//
// Three launches of one templated kernel, each an "inner products -> elementwise -> accumulate" pipeline
// with the same warp roles as the forward kernel (warp 0 TMA, warp 1 MMA, warps 2..9 elementwise: two warps per
// TMEM lane quadrant split the columns of a block; groups of 32 columns that are fully visible or fully hidden for a
// row skip the per-element mask test):
//
//   MODE_DQ  tile = 128 query rows (position x head-of-group); stream key blocks j:
//              S = Q K_j^T, dP = dO V_j^T  ->  dS = P o (dP - delta) * scale  ->  dQ += dS K_j
//   MODE_DK  tile = 128 keys of one kv head; stream query-row blocks i (all heads of the group, so
//            the GQA sum happens inside the accumulator, without atomics):
//              S^T = K Q_i^T, dP^T = V dO_i^T  ->  dS^T  ->  dK += dS^T Q_i
//   MODE_DV  tile = 128 keys; stream query-row blocks:
//              S^T = K Q_i^T  ->  P^T  ->  dV += P^T dO_i
//
// P is recomputed from the saved log-sum-exp (no running maximum needed); delta = rowsum(O o dO) comes
// from a small pre-kernel.  Splitting dK and dV keeps each accumulator (128 x D fp32 = up to 256 TMEM
// columns) beside the first fixed tile and the scores inside the 512-column tensor memory at D = 256.
// Results are deterministic: no atomics, fixed accumulation order.
//
// Order of a block j in the MMA warp: S of block j + 1 (its columns are free once S of j has been read, so it runs under the
// elementwise work), the accumulation of j, dP of j + 1 (over the columns that held dS of j, once the accumulation has retired:
// at width 256 the wait costs 0.06 us a block, and the first k-steps of S of j + 2 put into it cost more).  Measured against
// 32-wide blocks with all operands in shared memory, backward alone: 4096 positions, 8 heads on 1, width 256, 1024 of them
// causal: 1041 -> 568 us; 8 x 1227 positions (a pi0.5 training step's layer) 913 -> 583; 32 heads of 128 on 8, 2 x 2048: 1121 -> 737;
// 16 heads of 72, 24 x 256: 225 -> 202.
#include "common.cuh"
#include <limits.h>

namespace otb {

constexpr unsigned KID_ATTN_BWD = 3;
constexpr int BW_M = 128;
enum { MODE_DQ = 0, MODE_DK = 1, MODE_DV = 2 };

struct BwdParams {
  int B, Sq, Sk, H, Hkv, D, Dmma, g;
  float scale, scale_log2;
  const int* q_blk;
  const int* k_blk;
  const unsigned char* q_valid;
  const unsigned char* k_valid;
  const float* lse;     // (B, H, Sq), natural log
  const float* delta;   // (B, H, Sq)
  const __nv_bfloat16 *f1, *f2;   // tensors of the fixed tiles that go to tensor memory, and their strides in elements
  long long f1_sb, f1_ss, f1_sh, f2_sb, f2_ss, f2_sh;
  __nv_bfloat16* out;   // dq (B,Sq,H,D) | dk, dv (B,Sk,Hkv,D), contiguous
  float* parts;         // splits > 1: fp32 sums of each part instead, (splits, ...) of the same layout
  int splits;           // blocks that share a tile's streamed blocks
  KernelStatus* status;
};

// Tensor memory (512 columns of 32 bits) and shared memory of one CTA.
//
// The product that every block pays twice is the score product, and its A operand, the fixed tile, is what it used to
// spend its time on: with both operands in shared memory an M = 128 instruction of width N reads 4096 + 32 N bytes for N / 2
// clocks of arithmetic (shared memory: 128 bytes a clock), so 32-wide blocks kept the pipe at most 40 % busy.  A fixed tile is
// therefore moved into tensor memory once (two bf16 to a column), where an instruction reads only its 32 N bytes of B from
// shared memory; P and dS take the place of the scores they were made from and are the A operand of the accumulation from
// there.  At width 256 that is columns 128 (first fixed tile) + 64 + 64 (S, dP) + 256 (accumulator); the second fixed tile
// stays in shared memory.  Without the first tile and the dS tiles there, blocks are 64 wide in five 32 KB slots.
// Clocks of tensor pipe a 64-wide block at width 256: S 512, dP 768 (bound by operand reads), accumulation 512, by that
// arithmetic.  Counted (ncu, 8 x 1227 positions, 8 heads on 1): the pipe is busy 39 / 41 / 50 % of the cycles in dQ / dK / dV, issue
// slots 21 - 23 %, DRAM 6 - 8 %: the rest is the chain from the scores through the eight elementwise warps to the next product.
// By -Xptxas -v at most 168 registers, no spills but 4 bytes in dK up to width 128.
template <int MODE, int DPAD, int BN>
struct BwdSmem {
  static constexpr bool TWO = MODE != MODE_DV;                // second score product (dP)
  static constexpr bool F2_TMEM = TWO && DPAD <= 128;         // second fixed tile in tensor memory too
  static constexpr bool F2_SMEM = TWO && !F2_TMEM;
  static constexpr int NCHUNK = DPAD / 64;
  static constexpr int F_BYTES = BW_M * DPAD * 2;
  static constexpr int Y_BYTES = BN * DPAD * 2;
  static constexpr int NY1 = 3;                               // ring of the operand that S and (not in DV) the accumulation read
  static constexpr int NY2 = F2_SMEM ? 2 : 3;                 // ring of the other one
  static constexpr int OFF_F = 0;
  static constexpr int OFF_Y1 = F2_SMEM ? F_BYTES : 0;
  static constexpr int OFF_Y2 = OFF_Y1 + NY1 * Y_BYTES;
  static constexpr int OFF_META = OFF_Y2 + NY2 * Y_BYTES;     // per slot: int blk[BN], float lse2[BN], float delta[BN]
  static constexpr int OFF_KMM = OFF_META + 2 * BN * 12;      // int kmm[2][BN/32][2]: min / max block id per 32 columns
  static constexpr int OFF_BAR = OFF_KMM + 2 * (BN / 32) * 2 * 4;
  static constexpr int NBAR = 22;
  static constexpr int USED = OFF_BAR + NBAR * 8 + 32;
  static constexpr int TOTAL = USED + 1024;
  static_assert(TOTAL <= 232448, "shared memory budget");
  static constexpr int NS = TWO ? 1 : 2;                      // S tiles in flight
  static constexpr int TM_F1 = 0;
  static constexpr int TM_F2 = DPAD / 2;
  static constexpr int TM_S = TM_F2 + (F2_TMEM ? DPAD / 2 : 0);
  static constexpr int TM_DP = TM_S + NS * BN;
  static constexpr int TM_ACC = TM_DP + (TWO ? BN : 0);
  static_assert(TM_ACC + DPAD <= 512, "tensor memory budget");
};

__device__ __forceinline__ float bw_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int MODE, int DPAD, int BN>
__global__ void __launch_bounds__(320, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_f2, const __grid_constant__ CUtensorMap tm_y1,
                const __grid_constant__ CUtensorMap tm_y2, BwdParams p) {
  using L = BwdSmem<MODE, DPAD, BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sF = smem + L::OFF_F;
  uint8_t* sY1 = smem + L::OFF_Y1;
  uint8_t* sY2 = smem + L::OFF_Y2;
  int* meta_blk = reinterpret_cast<int*>(smem + L::OFF_META);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* f_full = bars + 0;     // the fixed tile in shared memory has landed
  uint64_t* a_full = bars + 1;     // the fixed tiles are in tensor memory
  uint64_t* y1_full = bars + 2;    // [3]
  uint64_t* y1_empty = bars + 5;   // [3]
  uint64_t* y2_full = bars + 8;    // [3]
  uint64_t* y2_empty = bars + 11;  // [3]
  uint64_t* s_full = bars + 14;    // [2]
  uint64_t* s_free = bars + 16;    // S has been read (TWO)
  uint64_t* dp_full = bars + 17;
  uint64_t* t_full = bars + 18;    // [2] P or dS is in tensor memory
  uint64_t* acc_full = bars + 20;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* range_smem = reinterpret_cast<int*>(tmem_slot + 2);   // [0] = first block, [1] = end (exclusive, in elements)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z % p.B, split = blockIdx.z / p.B;
  const int g = p.g;
  const int pos_per_tile = BW_M / g;   // MODE_DQ: positions per row tile
  const int pos_per_blk = BN / g;      // MODE_DK/DV: positions per streamed query block

  if (threadIdx.x == 0) {
    mbar_init(f_full, 1);
    mbar_init(a_full, 256);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&y1_full[i], 1);
      mbar_init(&y1_empty[i], 1);
      mbar_init(&y2_full[i], 1);
      mbar_init(&y2_empty[i], 1);
    }
    mbar_init(s_free, 256);
    mbar_init(dp_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&t_full[i], 256);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    range_smem[0] = INT_MAX;
    range_smem[1] = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_y1);
    tma_prefetch_desc(&tm_y2);
    if (L::F2_SMEM) tma_prefetch_desc(&tm_f2);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_acc = tmem_base + L::TM_ACC;

  // ---- range of streamed blocks that can contain a visible (query, key) pair
  __shared__ int s_ext, s_any;
  if (threadIdx.x == 0) {
    s_ext = (MODE == MODE_DQ) ? INT_MIN : INT_MAX;
    s_any = 0;
  }
  __syncthreads();
  if (MODE == MODE_DQ) {
    const int p0 = tile * pos_per_tile;
    int qmax = INT_MIN;
    bool any = false;
    for (int i = threadIdx.x; i < pos_per_tile; i += blockDim.x) {
      const int pos = p0 + i;
      if (pos < p.Sq && p.q_valid[(long long)b * p.Sq + pos]) {
        qmax = max(qmax, p.q_blk[(long long)b * p.Sq + pos]);
        any = true;
      }
    }
    if (any) {
      atomicMax(&s_ext, qmax);
      atomicOr(&s_any, 1);
    }
    __syncthreads();
    int last = -1;
    if (s_any) {
      const int qm = s_ext;
#pragma unroll 8
      for (int j = threadIdx.x; j < p.Sk; j += blockDim.x) {
        const int kbj = p.k_blk[(long long)b * p.Sk + j];
        const int kvj = p.k_valid[(long long)b * p.Sk + j];
        if (kvj && kbj <= qm) last = max(last, j);
      }
    }
    if (last >= 0) atomicMax(&range_smem[1], last + 1);
    if (threadIdx.x == 0) range_smem[0] = 0;
  } else {
    const int k0 = tile * BW_M;
    int kmin = INT_MAX;
    bool any = false;
    for (int i = threadIdx.x; i < BW_M; i += blockDim.x) {
      const int key = k0 + i;
      if (key < p.Sk && p.k_valid[(long long)b * p.Sk + key]) {
        kmin = min(kmin, p.k_blk[(long long)b * p.Sk + key]);
        any = true;
      }
    }
    if (any) {
      atomicMin(&s_ext, kmin);
      atomicOr(&s_any, 1);
    }
    __syncthreads();
    int first = INT_MAX, last = -1;
    if (s_any) {
      const int km = s_ext;
#pragma unroll 8
      for (int i = threadIdx.x; i < p.Sq; i += blockDim.x) {
        const int qbi = p.q_blk[(long long)b * p.Sq + i];
        const int qvi = p.q_valid[(long long)b * p.Sq + i];
        if (qvi && qbi >= km) {
          first = min(first, i);
          last = max(last, i);
        }
      }
    }
    if (last >= 0) {
      atomicMin(&range_smem[0], first);
      atomicMax(&range_smem[1], last + 1);
    }
  }
  __syncthreads();
  int blk0, nblk;
  if (MODE == MODE_DQ) {
    blk0 = 0;
    nblk = max(1, (range_smem[1] + BN - 1) / BN);
  } else {
    const int first = range_smem[0] == INT_MAX ? 0 : range_smem[0];
    blk0 = first / pos_per_blk;
    const int endb = (range_smem[1] + pos_per_blk - 1) / pos_per_blk;
    nblk = max(1, endb - blk0);
  }
  bool none = false;                     // my part has no block: its sum is zero (one block is run all the same)
  if (p.splits > 1) {
    const int lo = (int)((long long)nblk * split / p.splits), hi = (int)((long long)nblk * (split + 1) / p.splits);
    none = lo == hi;
    blk0 += lo;
    nblk = max(1, hi - lo);
  }

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      if (L::F2_SMEM) {
        mbar_expect_tx(f_full, L::F_BYTES);
#pragma unroll
        for (int c = 0; c < L::NCHUNK; ++c) {
          if (MODE == MODE_DQ) tma_load_4d(sF + c * (BW_M * 128), &tm_f2, f_full, c * 64, kvh * g, tile * pos_per_tile, b);
          else tma_load_4d(sF + c * (BW_M * 128), &tm_f2, f_full, c * 64, kvh, tile * BW_M, b);
        }
      }
      int s1 = 0, s2 = 0;
      uint32_t ph1 = 1, ph2 = 1;                     // a ring's first round does not wait
      for (int j = 0; j < nblk; ++j) {
        const int blk = blk0 + j;
        mbar_wait(&y1_empty[s1], ph1, abort_flag, p.status, KID_ATTN_BWD, 1, j);
        mbar_expect_tx(&y1_full[s1], L::Y_BYTES);
#pragma unroll
        for (int c = 0; c < L::NCHUNK; ++c) {
          uint8_t* y = sY1 + s1 * L::Y_BYTES + c * (BN * 128);
          if (MODE == MODE_DQ) tma_load_4d(y, &tm_y1, &y1_full[s1], c * 64, kvh, blk * BN, b);
          else tma_load_4d(y, &tm_y1, &y1_full[s1], c * 64, kvh * g, blk * pos_per_blk, b);
        }
        if (++s1 == L::NY1) { s1 = 0; ph1 ^= 1; }
        mbar_wait(&y2_empty[s2], ph2, abort_flag, p.status, KID_ATTN_BWD, 8, j);
        mbar_expect_tx(&y2_full[s2], L::Y_BYTES);
#pragma unroll
        for (int c = 0; c < L::NCHUNK; ++c) {
          uint8_t* y = sY2 + s2 * L::Y_BYTES + c * (BN * 128);
          if (MODE == MODE_DQ) tma_load_4d(y, &tm_y2, &y2_full[s2], c * 64, kvh, blk * BN, b);
          else tma_load_4d(y, &tm_y2, &y2_full[s2], c * 64, kvh * g, blk * pos_per_blk, b);
        }
        if (++s2 == L::NY2) { s2 = 0; ph2 ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // dP of block j + 1 (with two S tiles: S of block j + 1) goes over the columns that held dS of block j (P of j - 1).
    // Only instructions with one accumulator and shape are promised to run in the order they are issued (PTX ISA, pipelined
    // tcgen05 instructions), so it waits for the commit of the accumulation that reads them.
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(BW_M, BN, 0, 0);
      const uint32_t idesc_acc = make_idesc_bf16(BW_M, p.Dmma, 0, 1);
      const int ksteps = p.Dmma / 16;
      // scores of block j against a fixed tile in tensor memory
      auto scores_tmem = [&](uint32_t d, uint32_t f, uint32_t y) {
        for (int kk = 0; kk < ksteps; ++kk) {
          uint64_t bd = make_smem_desc(y + (kk >> 2) * (BN * 128) + (kk & 3) * 32, 16, 1024);
          umma_ts(d, f + kk * 8, bd, idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      int s1 = 0, s2 = 0;                            // ring slots of the next S and of the next dP (DV: accumulation)
      uint32_t ph1 = 0, ph2 = 0;
      auto issue_s = [&](int j) {
        mbar_wait(&y1_full[s1], ph1, abort_flag, p.status, KID_ATTN_BWD, 2, j);
        if (L::TWO) {
          if (j > 0) mbar_wait(s_free, (j - 1) & 1, abort_flag, p.status, KID_ATTN_BWD, 3, j);
        } else if (j > 1) {
          mbar_wait(&y2_empty[(j - 2) % L::NY2], ((j - 2) / L::NY2) & 1, abort_flag, p.status, KID_ATTN_BWD, 12, j);
        }
        tc_fence_after();
        const int buf = L::TWO ? 0 : (j & 1);
        scores_tmem(tmem_base + L::TM_S + buf * BN, tmem_base + L::TM_F1, smem_u32(sY1 + s1 * L::Y_BYTES));
        umma_commit(&s_full[buf]);
        if (!L::TWO) umma_commit(&y1_empty[s1]);     // DV reads this operand nowhere else
        if (++s1 == L::NY1) { s1 = 0; ph1 ^= 1; }
      };
      auto issue_dp = [&](int j) {
        mbar_wait(&y2_full[s2], ph2, abort_flag, p.status, KID_ATTN_BWD, 10, j);
        if (j > 0) mbar_wait(&y1_empty[(j - 1) % L::NY1], ((j - 1) / L::NY1) & 1, abort_flag, p.status, KID_ATTN_BWD, 13, j);
        tc_fence_after();
        const uint32_t y = smem_u32(sY2 + s2 * L::Y_BYTES), d = tmem_base + L::TM_DP;
        if (L::F2_TMEM) {
          scores_tmem(d, tmem_base + L::TM_F2, y);
        } else {
          const uint32_t fa = smem_u32(sF);
          for (int kk = 0; kk < ksteps; ++kk) {
            const int c = kk >> 2, w = kk & 3;
            uint64_t ad = make_smem_desc(fa + c * (BW_M * 128) + w * 32, 16, 1024);
            uint64_t bd = make_smem_desc(y + c * (BN * 128) + w * 32, 16, 1024);
            umma_ss(d, ad, bd, idesc_s, kk != 0 ? 1u : 0u);
          }
        }
        umma_commit(dp_full);
        umma_commit(&y2_empty[s2]);
        if (++s2 == L::NY2) { s2 = 0; ph2 ^= 1; }
      };
      mbar_wait(a_full, 0, abort_flag, p.status, KID_ATTN_BWD, 4, 0);
      if (L::F2_SMEM) mbar_wait(f_full, 0, abort_flag, p.status, KID_ATTN_BWD, 11, 0);
      tc_fence_after();
      issue_s(0);
      if (L::TWO) issue_dp(0);
      int sa = 0;                                    // ring slot of the accumulation's operand
      for (int j = 0; j < nblk; ++j) {
        if (j + 1 < nblk) issue_s(j + 1);
        const int buf = L::TWO ? 0 : (j & 1);
        if (!L::TWO) mbar_wait(&y2_full[s2], ph2, abort_flag, p.status, KID_ATTN_BWD, 10, j);
        mbar_wait(&t_full[buf], (L::TWO ? j : (j >> 1)) & 1, abort_flag, p.status, KID_ATTN_BWD, 5, j);
        tc_fence_after();
        const uint32_t t = tmem_base + (L::TWO ? L::TM_DP : L::TM_S + buf * BN);
        const uint32_t yb = smem_u32(L::TWO ? sY1 + sa * L::Y_BYTES : sY2 + s2 * L::Y_BYTES);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          // each half of a block's columns was written over the first columns of its own scores
          const uint32_t at = t + (kk / (BN / 32)) * (BN / 2) + (kk % (BN / 32)) * 8;
          uint64_t bd = make_smem_desc(yb + kk * 2048, BN * 128, 1024);
          umma_ts(tmem_acc, at, bd, idesc_acc, (j | kk) != 0 ? 1u : 0u);
        }
        if (L::TWO) {
          umma_commit(&y1_empty[sa]);
          if (++sa == L::NY1) sa = 0;
          if (j + 1 < nblk) issue_dp(j + 1);
        } else {
          umma_commit(&y2_empty[s2]);
          if (++s2 == L::NY2) { s2 = 0; ph2 ^= 1; }
        }
      }
      umma_commit(acc_full);
    }
  } else {
    // ------------------------------------------------------------------ elementwise + epilogue
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;            // which half of a block's columns this thread handles
    const int row = quad * 32 + lane;
    const int st = threadIdx.x - 64;             // 0..255
    int* kmm = reinterpret_cast<int*>(smem + L::OFF_KMM);
    constexpr int HB = BN / 2;                   // columns per thread per block
    static_assert(HB % 32 == 0, "TMEM reads are 32 columns wide");
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    float* meta_lse = reinterpret_cast<float*>(meta_blk + 2 * BN);
    float* meta_delta = meta_lse + 2 * BN;
    const float LOG2E = 1.4426950408889634f;

    // per-row constants
    bool row_ok;
    int row_blk = 0;
    float row_lse2 = 0.f, row_delta = 0.f;
    long long out_off;
    bool row_in;
    const __nv_bfloat16 *f1_row, *f2_row;
    if (MODE == MODE_DQ) {
      const int pos = tile * pos_per_tile + row / g;
      const int head = kvh * g + row % g;
      row_in = pos < p.Sq;
      row_ok = row_in && p.q_valid[(long long)b * p.Sq + pos] != 0;
      if (row_ok) {
        row_blk = p.q_blk[(long long)b * p.Sq + pos];
        row_lse2 = p.lse[((long long)b * p.H + head) * p.Sq + pos] * LOG2E;
        row_delta = p.delta[((long long)b * p.H + head) * p.Sq + pos];
      }
      out_off = (((long long)b * p.Sq + pos) * p.H + head) * p.D;
      f1_row = p.f1 + b * p.f1_sb + pos * p.f1_ss + head * p.f1_sh;
      f2_row = p.f2 + out_off;                   // dO is laid out like dQ
    } else {
      const int key = tile * BW_M + row;
      row_in = key < p.Sk;
      row_ok = row_in && p.k_valid[(long long)b * p.Sk + key] != 0;
      if (row_ok) row_blk = p.k_blk[(long long)b * p.Sk + key];
      out_off = (((long long)b * p.Sk + key) * p.Hkv + kvh) * p.D;
      f1_row = p.f1 + b * p.f1_sb + key * p.f1_ss + kvh * p.f1_sh;
      f2_row = p.f2 + b * p.f2_sb + key * p.f2_ss + kvh * p.f2_sh;
    }

    // ---- fixed tiles -> tensor memory: this thread's row, its half of the head width
    auto fixed_tile = [&](const __nv_bfloat16* src, int col) {
      constexpr int CW = DPAD / 4 < 32 ? DPAD / 4 : 32;      // 32-bit columns a piece: the half row is one or two pieces
#pragma unroll
      for (int c = 0; c < DPAD / 4; c += CW) {
        uint32_t r[CW];
#pragma unroll
        for (int e = 0; e < CW; e += 4) {
          const int d = 2 * (half * (DPAD / 4) + c + e);
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (row_in && d < p.D) v = *reinterpret_cast<const uint4*>(src + d);
          r[e] = v.x; r[e + 1] = v.y; r[e + 2] = v.z; r[e + 3] = v.w;
        }
        __syncwarp();
        const uint32_t dst = tmem_base + col + lane_off + half * (DPAD / 4) + c;
        if (CW == 32) tmem_st_x32(dst, r);
        else tmem_st_x16(dst, r);
      }
    };
    fixed_tile(f1_row, L::TM_F1);
    if (L::F2_TMEM) fixed_tile(f2_row, L::TM_F2);
    tmem_wait_st();
    tc_fence_before();
    mbar_arrive(a_full);

    // ---- what a block's columns carry (thread st < BN: one column), fetched one block ahead
    int nx_blk = 0;
    float nx_lse = 0.f, nx_delta = 0.f;
    auto fetch_meta = [&](int j) {
      if (st >= BN) return;
      if (MODE == MODE_DQ) {
        const int key = (blk0 + j) * BN + st;
        nx_blk = INT_MAX;
        if (key < p.Sk) {
          const int kbv = p.k_blk[(long long)b * p.Sk + key];
          const int kvv = p.k_valid[(long long)b * p.Sk + key];
          nx_blk = kvv ? kbv : INT_MAX;
        }
      } else {
        const int pos = (blk0 + j) * pos_per_blk + st / g;
        const int head = kvh * g + st % g;
        nx_blk = INT_MIN;
        nx_lse = INFINITY;
        nx_delta = 0.f;
        if (pos < p.Sq) {
          // four independent loads; the validity only selects afterwards
          const int qvv = p.q_valid[(long long)b * p.Sq + pos];
          const int qbv = p.q_blk[(long long)b * p.Sq + pos];
          const float lv = p.lse[((long long)b * p.H + head) * p.Sq + pos];
          const float dv2 = p.delta[((long long)b * p.H + head) * p.Sq + pos];
          if (qvv) {
            nx_blk = qbv;
            nx_lse = lv * LOG2E;
            nx_delta = dv2;
          }
        }
      }
    };
    fetch_meta(0);
    for (int j = 0; j < nblk; ++j) {
      const int slot = j & 1;
      if (st < BN) {                             // whole warps
        meta_blk[slot * BN + st] = nx_blk;
        if (MODE != MODE_DQ) {
          meta_lse[slot * BN + st] = nx_lse;
          meta_delta[slot * BN + st] = nx_delta;
        }
        const int mn = __reduce_min_sync(0xffffffffu, nx_blk), mxk = __reduce_max_sync(0xffffffffu, nx_blk);
        if (lane == 0) {
          kmm[(slot * (BN / 32) + st / 32) * 2 + 0] = mn;
          kmm[(slot * (BN / 32) + st / 32) * 2 + 1] = mxk;
        }
      }
      if (j + 1 < nblk) fetch_meta(j + 1);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const int* mb = meta_blk + slot * BN + half * HB;
      const float* ml = meta_lse + slot * BN + half * HB;
      const float* md = meta_delta + slot * BN + half * HB;
      const int buf = L::TWO ? 0 : slot;
      const uint32_t s_addr = tmem_base + L::TM_S + buf * BN + half * HB + lane_off;
      const uint32_t d_addr = tmem_base + L::TM_DP + half * HB + lane_off;
      const uint32_t t_addr = L::TWO ? d_addr : s_addr;
      mbar_wait(&s_full[buf], (L::TWO ? j : (j >> 1)) & 1, abort_flag, p.status, KID_ATTN_BWD, 6, j);
      tc_fence_after();
      uint32_t rs[HB];
#pragma unroll
      for (int c = 0; c < HB; c += 32) {
        __syncwarp();
        tmem_ld_x32(s_addr + c, rs + c);
      }
      tmem_wait_ld();
      if (L::TWO) {
        tc_fence_before();
        mbar_arrive(s_free);
      }
      // ---- P, over the scores; visibility per group of 32 columns for this row: 2 = all, 0 = none, 1 = test each
      int cls[HB / 32];
#pragma unroll
      for (int c = 0; c < HB / 32; ++c) {
        const int gi = (slot * (BN / 32) + half * (HB / 32) + c) * 2;
        const int gmin = kmm[gi], gmax = kmm[gi + 1];
        if (MODE == MODE_DQ) cls[c] = (!row_ok || gmin > row_blk) ? 0 : (gmax <= row_blk ? 2 : 1);
        else cls[c] = (!row_ok || gmax < row_blk) ? 0 : (gmin >= row_blk ? 2 : 1);
        if (cls[c] != 0) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int col = c * 32 + e;
            const float l2 = MODE == MODE_DQ ? row_lse2 : ml[col];
            rs[col] = __float_as_uint(bw_exp2(fmaf(__uint_as_float(rs[col]), p.scale_log2, -l2)));
          }
          if (cls[c] == 1) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const int col = c * 32 + e;
              if (!(MODE == MODE_DQ ? mb[col] <= row_blk : row_blk <= mb[col])) rs[col] = 0u;
            }
          }
        }
      }
      if (L::TWO) {
        mbar_wait(dp_full, j & 1, abort_flag, p.status, KID_ATTN_BWD, 7, j);
        tc_fence_after();
      }
      // every score of mine has to be read before its columns are written
      uint32_t packed[HB / 2];
#pragma unroll
      for (int c = 0; c < HB / 32; ++c) {
        uint32_t rd[32];
        if (L::TWO) {
          __syncwarp();
          tmem_ld_x32(d_addr + c * 32, rd);
          tmem_wait_ld();
        }
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const int col = c * 32 + e;
          float v[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float pr = __uint_as_float(rs[col + h]);
            if (!L::TWO) v[h] = pr;
            else v[h] = pr * (__uint_as_float(rd[e + h]) - (MODE == MODE_DQ ? row_delta : md[col + h])) * p.scale;
          }
          packed[col >> 1] = cls[c] == 0 ? 0u : pack_bf16(v[0], v[1]);
        }
      }
      __syncwarp();
      if (HB == 64) tmem_st_x32(t_addr, packed);
      else tmem_st_x16(t_addr, packed);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&t_full[buf]);
    }

    mbar_wait(acc_full, 0, abort_flag, p.status, KID_ATTN_BWD, 9, 0);
    tc_fence_after();
    __nv_bfloat16* orow = p.out + out_off;
    float* prow = nullptr;
    if (p.splits > 1)
      prow = p.parts + (long long)split * p.B * (MODE == MODE_DQ ? (long long)p.Sq * p.H : (long long)p.Sk * p.Hkv) * p.D +
             out_off;
    const int n16 = p.Dmma / 16;
    const int a_lo = half ? (n16 + 1) / 2 : 0, a_hi = half ? n16 : (n16 + 1) / 2;
#pragma unroll 1
    for (int c = a_lo; c < a_hi; ++c) {
      uint32_t r[16];
      __syncwarp();
      tmem_ld_x16(tmem_acc + lane_off + c * 16, r);
      tmem_wait_ld();
      if (row_in) {
#pragma unroll
        for (int h8 = 0; h8 < 2; ++h8) {
          const int col = c * 16 + h8 * 8;
          if (col < p.D && prow != nullptr) {
#pragma unroll
            for (int e = 0; e < 8; e += 4)
              *reinterpret_cast<float4*>(prow + col + e) =
                  none ? make_float4(0.f, 0.f, 0.f, 0.f)
                       : make_float4(__uint_as_float(r[h8 * 8 + e]), __uint_as_float(r[h8 * 8 + e + 1]),
                                     __uint_as_float(r[h8 * 8 + e + 2]), __uint_as_float(r[h8 * 8 + e + 3]));
          } else if (col < p.D) {
            uint4 o;
            o.x = pack_bf16(__uint_as_float(r[h8 * 8 + 0]), __uint_as_float(r[h8 * 8 + 1]));
            o.y = pack_bf16(__uint_as_float(r[h8 * 8 + 2]), __uint_as_float(r[h8 * 8 + 3]));
            o.z = pack_bf16(__uint_as_float(r[h8 * 8 + 4]), __uint_as_float(r[h8 * 8 + 5]));
            o.w = pack_bf16(__uint_as_float(r[h8 * 8 + 6]), __uint_as_float(r[h8 * 8 + 7]));
            *reinterpret_cast<uint4*>(orow + col) = o;
          }
        }
      }
    }
    tc_fence_before();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[b,h,s] = sum_d O[b,s,h,d] * dO[b,s,h,d]; one warp per (b,s,h) row.
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                  float* __restrict__ delta, int B, int S, int H, int D) {
  const long long rowi = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (rowi >= (long long)B * S * H) return;
  const __nv_bfloat16* a = o + rowi * D;
  const __nv_bfloat16* c = d_o + rowi * D;
  float acc = 0.f;
  for (int i = lane * 8; i < D; i += 256) {
    uint4 ua = *reinterpret_cast<const uint4*>(a + i);
    uint4 uc = *reinterpret_cast<const uint4*>(c + i);
    float2 x, y;
    x = unpack_bf16(ua.x); y = unpack_bf16(uc.x); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16(ua.y); y = unpack_bf16(uc.y); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16(ua.z); y = unpack_bf16(uc.z); acc += x.x * y.x + x.y * y.y;
    x = unpack_bf16(ua.w); y = unpack_bf16(uc.w); acc += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) {
    const int h = int(rowi % H);
    const long long bs = rowi / H;
    const int s = int(bs % S);
    const int b = int(bs / S);
    delta[((long long)b * H + h) * S + s] = acc;
  }
}

static int make_map4b(CUtensorMap* m, const void* base, int D, int Hx, int S, int B, long long sh, long long ss,
                      long long sb, int box_h, int box_s) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)Hx, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)sh * 2, (uint64_t)ss * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {64, (uint32_t)box_h, (uint32_t)box_s, 1};
  return make_tmap_bf16(m, base, 4, dims, strides, box);
}

struct Strides {
  long long sb, ss, sh;
};

// out[i] = bf16(sum over `splits` parts of 8 n8 floats each, in order)
__global__ void attn_bwd_sum_kernel(const float* __restrict__ parts, __nv_bfloat16* __restrict__ out, long long n8,
                                    int splits) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n8) return;
  float a[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float4* src = reinterpret_cast<const float4*>(parts + (s * n8 + i) * 8);
    const float4 u = src[0], w = src[1];
    a[0] += u.x; a[1] += u.y; a[2] += u.z; a[3] += u.w;
    a[4] += w.x; a[5] += w.y; a[6] += w.z; a[7] += w.w;
  }
  *reinterpret_cast<uint4*>(out + i * 8) =
      make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
}

template <int MODE>
static long long bwd_tiles(int Sq, int Sk, int g) {
  return MODE == MODE_DQ ? (Sq + BW_M / g - 1) / (BW_M / g) : (Sk + BW_M - 1) / BW_M;
}

template <int MODE, int DPAD, int BN>
static int launch_bwd(const void* q, Strides qs, const void* k, Strides ks, const void* v, Strides vs, const void* d_o,
                      BwdParams p, cudaStream_t stream) {
  using L = BwdSmem<MODE, DPAD, BN>;
  static bool configured = false;
  auto kern = attn_bwd_kernel<MODE, DPAD, BN>;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int g = p.g;
  if (MODE != MODE_DQ && (BN % g)) return -20;
  CUtensorMap f2, y1, y2;
  const Strides dos = {(long long)p.Sq * p.H * p.D, (long long)p.H * p.D, (long long)p.D};
  const Strides f1s = MODE == MODE_DQ ? qs : ks, f2s = MODE == MODE_DQ ? dos : vs;
  p.f1 = static_cast<const __nv_bfloat16*>(MODE == MODE_DQ ? q : k);
  p.f2 = static_cast<const __nv_bfloat16*>(MODE == MODE_DQ ? d_o : v);
  p.f1_sb = f1s.sb; p.f1_ss = f1s.ss; p.f1_sh = f1s.sh;
  p.f2_sb = f2s.sb; p.f2_ss = f2s.ss; p.f2_sh = f2s.sh;
  int r;
  if (MODE == MODE_DQ) {
    r = make_map4b(&f2, d_o, p.D, p.H, p.Sq, p.B, dos.sh, dos.ss, dos.sb, g, BW_M / g);
    if (r) return 2000 + r;
    r = make_map4b(&y1, k, p.D, p.Hkv, p.Sk, p.B, ks.sh, ks.ss, ks.sb, 1, BN);
    if (r) return 3000 + r;
    r = make_map4b(&y2, v, p.D, p.Hkv, p.Sk, p.B, vs.sh, vs.ss, vs.sb, 1, BN);
    if (r) return 4000 + r;
  } else {
    r = make_map4b(&f2, v, p.D, p.Hkv, p.Sk, p.B, vs.sh, vs.ss, vs.sb, 1, BW_M);
    if (r) return 2000 + r;
    r = make_map4b(&y1, q, p.D, p.H, p.Sq, p.B, qs.sh, qs.ss, qs.sb, g, BN / g);
    if (r) return 3000 + r;
    r = make_map4b(&y2, d_o, p.D, p.H, p.Sq, p.B, dos.sh, dos.ss, dos.sb, g, BN / g);
    if (r) return 4000 + r;
  }
  const dim3 grid((unsigned)bwd_tiles<MODE>(p.Sq, p.Sk, g), p.Hkv, p.B * p.splits);
  kern<<<grid, 320, L::TOTAL, stream>>>(f2, y1, y2, p);
  if (p.splits > 1) {
    const long long n8 = (long long)p.B * (MODE == MODE_DQ ? (long long)p.Sq * p.H : (long long)p.Sk * p.Hkv) * p.D / 8;
    attn_bwd_sum_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(p.parts, p.out, n8, p.splits);
  }
  return (int)cudaGetLastError();
}

constexpr int BWD_MAX_SPLITS = 16;
constexpr double BWD_MAX_SCRATCH = 256.0 * (1 << 20);   // bytes of one output's parts; past it a tile's share is small anyway

// Into how many parts a tile's streamed blocks are dealt.  One block fills an SM, so the time is rounds x the blocks a part
// streams, plus what every part does once (fixed tiles, first scores, epilogue: PER_PART blocks' worth) and the
// sums that are written and read in fp32 (charged to the parts of the whole launch) by one more launch, `extra` blocks' worth:
// short sequences are bound by what the host issues, so parts must win a twentieth as well.  One sample of 4096 keys under one
// kv head is 32 dK and 32 dV tiles, which leaves 116 of 148 SMs idle: backward 1.48 ms without parts, 0.57 ms with (8 heads on 1,
// width 256, 1024 causal positions).  Against the best number of parts for each product, over 615 sizes (1 - 16 samples, 200 -
// 4096 positions, five head layouts of width 64 - 256, no, a fifth and half of the positions causal), the rule costs 1.9 % in the
// mean with any PER_PART from 2 to 16, and one part always 5.3 %; what is left are masks, which sizes do not show.
static int pick_bwd_splits(long long tiles, int blocks, int B, double out_bytes, double sum_cost, double extra) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) return 1;
  }
  constexpr double PER_PART = 4.0, MUST_WIN = 0.95;
  int best = 1;
  double best_cost = 0;
  for (int s = 1; s <= BWD_MAX_SPLITS && s * 4 <= (blocks > 4 ? blocks : 4) && (long long)B * s <= 65535 &&
                  (s == 1 || s * out_bytes <= BWD_MAX_SCRATCH); ++s) {
    const double cost = (double)((tiles * s + sms - 1) / sms) * ((double)((blocks + s - 1) / s) + PER_PART) +
                        (s > 1 ? sum_cost * (s + 1) + extra : 0.0);
    if (s == 1 || cost < best_cost) {
      best = s;
      best_cost = s == 1 ? MUST_WIN * cost : cost;
    }
  }
  return best;
}

}  // namespace otb

using namespace otb;

// columns of a streamed block by padded head width
static constexpr int bwd_bn(int dpad) { return dpad == 256 ? 64 : 128; }

// Parts of the three products; `dq`, `dk`, `dv` above 1 want fp32 scratch of that many outputs each.  Sk must be the
// streamed length of dQ.
extern "C" void otb_attn_bwd_splits(int B, int Sq, int Sk, int H, int Hkv, int D, int* dq, int* dk, int* dv) {
  const int g = H / Hkv, dpad = D <= 64 ? 64 : (D <= 128 ? 128 : 256);
  const int bn = bwd_bn(dpad);
  const long long kv = (long long)Hkv * B;
  // a block of 64 x 256 takes about 1.1 us (dV: 0.65), others in proportion; fp32 sums move at about 4 TB/s
  const double us = 1.1 * bn * dpad / (64 * 256), us_v = 0.65 * bn * dpad / (64 * 256);
  const double q_out = 4.0 * B * Sq * H * D, k_out = 4.0 * B * Sk * Hkv * D, q_sum = q_out / 4e6, k_sum = k_out / 4e6;
  *dq = pick_bwd_splits(bwd_tiles<MODE_DQ>(Sq, Sk, g) * kv, (Sk + bn - 1) / bn, B, q_out, q_sum / us, 15.0 / us);
  *dk = pick_bwd_splits(bwd_tiles<MODE_DK>(Sq, Sk, g) * kv, (int)(((long long)Sq * g + bn - 1) / bn), B, k_out, k_sum / us,
                        15.0 / us);
  *dv = pick_bwd_splits(bwd_tiles<MODE_DV>(Sq, Sk, g) * kv, (int)(((long long)Sq * g + bn - 1) / bn), B, k_out, k_sum / us_v,
                        15.0 / us_v);
}

// q (B,Sq,H,D), k/v (B,Sk,Hkv,D) with element strides; o, do: (B,Sq,H,D) contiguous; lse (B,H,Sq);
// delta: scratch (B,H,Sq) fp32; dq (B,Sq,H,D), dk/dv (B,Sk,Hkv,D) contiguous outputs; *_parts: the scratch that
// otb_attn_bwd_splits asks for (null where the parts are 1).
extern "C" int otb_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                            const float* lse, float* delta, void* dq, void* dk, void* dv, float* dq_parts,
                            float* dk_parts, float* dv_parts, int dq_splits, int dk_splits, int dv_splits,
                            const int* q_blk, const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid, int B,
                            int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh,
                            long long k_sb, long long k_ss, long long k_sh, long long v_sb, long long v_ss,
                            long long v_sh, float scale, void* status, cudaStream_t stream) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || H <= 0 || Hkv <= 0 || H % Hkv) return -2;
  const int g = H / Hkv;
  if (g > 32 || (32 % g)) return -3;
  if (D % 8 || D > 256 || D < 16) return -4;
  const long long strides[9] = {q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh};
  for (int i = 0; i < 9; ++i)
    if (strides[i] % 8) return -5;
  // rows are read and written in 128-bit pieces by the kernels themselves, not only through tensor maps
  const void* const bases[8] = {q, k, v, o, d_o, dq, dk, dv};
  for (int i = 0; i < 8; ++i)
    if (reinterpret_cast<uintptr_t>(bases[i]) & 15) return -6;
  const int splits[3] = {dq_splits, dk_splits, dv_splits};
  float* const parts[3] = {dq_parts, dk_parts, dv_parts};
  for (int i = 0; i < 3; ++i)
    if (splits[i] < 1 || splits[i] > BWD_MAX_SPLITS || (splits[i] > 1 && parts[i] == nullptr) ||
        (reinterpret_cast<uintptr_t>(parts[i]) & 15))
      return -7;
  {
    const long long rows = (long long)B * Sq * H;
    const int threads = 256;
    const long long blocks = (rows * 32 + threads - 1) / threads;
    attn_delta_kernel<<<(unsigned)blocks, threads, 0, stream>>>(static_cast<const __nv_bfloat16*>(o),
                                                               static_cast<const __nv_bfloat16*>(d_o), delta, B, Sq,
                                                               H, D);
  }
  BwdParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.D = D; p.g = g;
  p.Dmma = (D + 15) / 16 * 16;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.q_blk = q_blk; p.k_blk = k_blk; p.q_valid = q_valid; p.k_valid = k_valid;
  p.lse = lse; p.delta = delta;
  p.status = static_cast<KernelStatus*>(status);
  const Strides qs = {q_sb, q_ss, q_sh}, ks = {k_sb, k_ss, k_sh}, vs = {v_sb, v_ss, v_sh};
  const int dpad = D <= 64 ? 64 : (D <= 128 ? 128 : 256);
  int r = 0;
#define RUN3(DP)                                                                       \
  p.out = static_cast<__nv_bfloat16*>(dq);                                             \
  p.parts = dq_parts;                                                                  \
  p.splits = dq_splits;                                                                \
  r = launch_bwd<MODE_DQ, DP, bwd_bn(DP)>(q, qs, k, ks, v, vs, d_o, p, stream);         \
  if (r) return r;                                                                     \
  p.out = static_cast<__nv_bfloat16*>(dk);                                             \
  p.parts = dk_parts;                                                                  \
  p.splits = dk_splits;                                                                \
  r = launch_bwd<MODE_DK, DP, bwd_bn(DP)>(q, qs, k, ks, v, vs, d_o, p, stream);         \
  if (r) return 100000 + r;                                                            \
  p.out = static_cast<__nv_bfloat16*>(dv);                                             \
  p.parts = dv_parts;                                                                  \
  p.splits = dv_splits;                                                                \
  r = launch_bwd<MODE_DV, DP, bwd_bn(DP)>(q, qs, k, ks, v, vs, d_o, p, stream);       \
  if (r) return 200000 + r;
  if (dpad == 64) { RUN3(64) }
  else if (dpad == 128) { RUN3(128) }
  else { RUN3(256) }
#undef RUN3
  return 0;
}
