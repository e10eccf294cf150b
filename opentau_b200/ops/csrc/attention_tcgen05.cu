// Block-causal flash attention forward for sm_100a: TMA-fed, S = Q K^T and O += P V on tcgen05 with
// both accumulators in tensor memory, online softmax by 256 threads, two to a TMEM lane.
//
// Mask rule (same as the dense reference): query i sees key j iff q_valid[i] && k_valid[j] &&
// k_blk[j] <= q_blk[i].  Cached cross-attention keys carry k_blk = INT_MIN.  Rows that see no key
// produce O = 0 and LSE = 0.
//
// Work decomposition: one CTA per (batch, kv head, tile of 128 "rows"), where a row is a
// (query position, query head of the GQA group) pair: 128 rows = (128/g) positions x g heads, so one
// K/V tile load serves every head of the group (MQA: g = 8 -> K/V traffic / 8).
//
// Warps: 0 = TMA producer, 1 = MMA issuer (owns TMEM), 2..9 = softmax / correction / epilogue.
// Per KV block j:  MMA issues S[j+1] = Q K_{j+1}^T early, softmax turns S[j] into bf16 P, in shared memory
// (128B-swizzled, K-major) or, with two CTAs to an SM (SPLIT_TWO), over the scores in tensor memory, MMA issues
// O += P V_j.  O is rescaled lazily: only when the running row maximum grew by more than 2^8 since the maximum
// in use, so the common case touches O never.
//
// Few query tiles against many keys (a denoising step or a decoded token against a cached prefix) share the key blocks of
// a tile among `nsplit` CTAs.  Where the tiles are few enough (SPLIT_CLUSTER) those CTAs are one cluster and the partials
// never leave the chip's shared memory: a tile holds 64 or 32 rows, every CTA leaves its fp32 partial (with the row's maximum
// and sum behind it) in its own shared memory, sends each peer the rows that peer owns with one bulk copy, and merges its
// own rows.  Otherwise (SPLIT_GLOBAL) the partials go to global memory and attn_combine_kernel merges them.
#include "common.cuh"
#include <limits.h>

namespace otb {

constexpr unsigned KID_ATTN = 2;
constexpr int ATT_M = 128;
constexpr int CL_ROWS = 64;        // rows, at most, of a tile whose key blocks a cluster shares
enum { SPLIT_GLOBAL = 0, SPLIT_CLUSTER = 1, SPLIT_TWO = 2 };     // SPLIT_TWO: no split, two CTAs per SM

struct AttnParams {
  int B, Sq, Sk, H, Hkv, D, Dmma, g;
  float scale_log2;                 // scale * log2(e)
  const int* q_blk;                 // (B, Sq)
  const int* k_blk;                 // (B, Sk)
  const unsigned char* q_valid;     // (B, Sq)
  const unsigned char* k_valid;     // (B, Sk)
  __nv_bfloat16* o;                 // (B, Sq, H, D) contiguous
  float* lse;                       // (B, H, Sq)
  // split-KV (few query tiles, many keys: a denoising step against a cached prefix): CTA (tile, split) covers its
  // share of the key blocks and leaves an unnormalised partial; attn_combine_kernel merges the partials
  int skip_reach;                   // visit every key block: skip the prologue scan for the last reachable key
  int nsplit;                       // 1: write o / lse directly
  int cl_rows;                      // SPLIT_CLUSTER: rows of a tile (32 or 64)
  int ahead;                        // SPLIT_CLUSTER: key blocks, at most, that a CTA of the first tile requests into L2
  float* part_o;                    // (nsplit, B, Sq, H, D) fp32, accumulators expressed against part m
  float2* part_ml;                  // (nsplit, B, H, Sq): (running maximum in log2 units, row sum)
  KernelStatus* status;
};

// TSP: P is written over the scores in tensor memory and is the A operand of the PV product from there.  Without P in shared
// memory and with 64-wide blocks a CTA is 99 KB and 256 columns, so two share an SM: the softmax of one block is a chain of
// tensor-memory reads, an exchange and exponentials that one CTA's eight warps leave three quarters open (ncu: issue slots 25 %
// busy, tensor pipe 14 %, at 16 heads of 72).
constexpr bool attn_tsp(int split) { return split == SPLIT_TWO; }

template <int DPAD, int BN, int SPLIT>
struct AttnSmem {
  static constexpr bool TSP = attn_tsp(SPLIT);
  static constexpr int NCHUNK = DPAD / 64;
  static constexpr int Q_BYTES = ATT_M * DPAD * 2;
  static constexpr int KV_TILE = BN * DPAD * 2;        // one K or V tile
  static constexpr int STAGE_BYTES = 2 * KV_TILE;      // K and V of one block
  static constexpr int P_BYTES = TSP ? 0 : ATT_M * BN * 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_KV = Q_BYTES;
  static constexpr int OFF_P = OFF_KV + 2 * STAGE_BYTES;
  static constexpr int OFF_META = OFF_P + 2 * P_BYTES;  // int kmeta[2][BN]
  static constexpr int OFF_RED = OFF_META + 2 * BN * 4;  // float red[2][128]: row max / row sum exchange
  static constexpr int OFF_KMM = OFF_RED + 2 * ATT_M * 4;  // int kmm[2][BN/32][2]: min / max block id per 32 keys
  static constexpr int OFF_BAR = OFF_KMM + 2 * (BN / 32) * 2 * 4;
  static constexpr int NBAR = 17;
  // a cluster's partials: [row][DPAD + 4] floats (the pad spreads the banks and carries the row's maximum and sum).  Mine of all
  // rows and the peers' of the rows I own lie over the operand tiles; in a tile of DIRECT_ROWS the latter fit behind its query rows
  static constexpr int DIRECT_ROWS = 32;
  static constexpr int PART_LD = DPAD + 4;
  static constexpr int OFF_PEER = CL_ROWS * PART_LD * 4;
  static_assert(SPLIT != SPLIT_CLUSTER || OFF_PEER + (CL_ROWS + 8) * PART_LD * 4 <= OFF_META, "the partials must fit over the operand tiles");
  static_assert(SPLIT != SPLIT_CLUSTER || DIRECT_ROWS * DPAD * 2 + (DIRECT_ROWS + 8) * PART_LD * 4 <= OFF_KV, "and behind the query rows");
  static_assert(SPLIT != SPLIT_CLUSTER || DIRECT_ROWS * PART_LD * 4 <= 2 * STAGE_BYTES, "mine over the keys and values");
  static constexpr int USED = OFF_BAR + NBAR * 8 + 32;
  // room for rounding the base up to 1024 bytes (the kernel has no static shared memory, so the base normally is
  // aligned already); capped at the 227 KB a CTA may own, and checked at run time
  static constexpr int TOTAL = USED + 1024 <= 232448 ? USED + 1024 : 232448;
  static_assert(USED <= 232448, "shared memory budget");
  static constexpr int TMEM_COLS = TSP ? 256 : 512;    // two S tiles, O
  static_assert(2 * BN + DPAD <= TMEM_COLS, "tensor memory budget");
};

__device__ __forceinline__ void l2_prefetch_4d(const CUtensorMap* m, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The rows a CTA of a cluster owns, from the partials of all (mine and the peers', rows of DPAD + 4 floats): M = max m_s,
// O = sum O_s 2^(m_s - M) / sum l_s 2^(m_s - M).  A warp to a row; every lane weighs the splits by itself and their loads are independent
// of one another.  (Walking through it once ahead of the dependency wait, against its cold instruction cache, loses where a launch is
// not resident before its predecessor ends: 8.9 -> 9.8 us in a row of these kernels.)
template <int DPAD, int N>
__device__ __forceinline__ void merge_rows(const AttnParams& p, const float* mine, const float* peers, int split, int rpr, int own, int t0,
                                           int p0, int kvh, int b, int w, int lane) {
  constexpr int LD = DPAD + 4, NV = DPAD / 128 < 1 ? 1 : DPAD / 128;       // four columns a lane, NV times
#pragma unroll 1
  for (int t = w; t < own; t += 8) {
    float m_s[N], l_s[N], M = -INFINITY;
    float4 v[N][NV];
#pragma unroll
    for (int sp = 0; sp < N; ++sp) {
      m_s[sp] = -INFINITY;
      l_s[sp] = 0.f;
#pragma unroll
      for (int c = 0; c < NV; ++c) v[sp][c] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (sp < p.nsplit) {
        const float* src = sp == split ? mine + t * LD : peers + ((sp < split ? sp : sp - 1) * rpr + t) * LD;
        const float2 ml = *reinterpret_cast<const float2*>(src + DPAD);
        if (DPAD >= 128 || lane < DPAD / 4) {
#pragma unroll
          for (int c = 0; c < NV; ++c) v[sp][c] = *reinterpret_cast<const float4*>(src + c * 128 + lane * 4);
        }
        l_s[sp] = ml.y;
        if (ml.y > 0.f) m_s[sp] = ml.x;
      }
      M = fmaxf(M, m_s[sp]);
    }
    float sum = 0.f;
#pragma unroll
    for (int sp = 0; sp < N; ++sp) {
      m_s[sp] = m_s[sp] == -INFINITY ? 0.f : fast_exp2(m_s[sp] - M);       // its weight
      sum += l_s[sp] * m_s[sp];
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    const int r = t0 + t, g = p.g, rpos = p0 + r / g, rhead = kvh * g + r % g;
    __nv_bfloat16* orow = p.o + (((long long)b * p.Sq + rpos) * p.H + rhead) * p.D;
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int sp = 0; sp < N; ++sp) {
        const float wt = m_s[sp] * inv;              // 0 where nothing is visible; a NaN there stays one
        acc.x += v[sp][c].x * wt;
        acc.y += v[sp][c].y * wt;
        acc.z += v[sp][c].z * wt;
        acc.w += v[sp][c].w * wt;
      }
      const int col = c * 128 + lane * 4;
      if (col < p.D)
        *reinterpret_cast<uint2*>(orow + col) = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
    }
    if (lane == 0)
      p.lse[((long long)b * p.H + rhead) * p.Sq + rpos] = sum > 0.f ? (M + log2f(sum)) * 0.6931471805599453f : 0.f;
  }
}
template <int DPAD, int BN, int SPLIT>
__global__ void __launch_bounds__(320, attn_tsp(SPLIT) ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, AttnParams p) {
  using L = AttnSmem<DPAD, BN, SPLIT>;
  constexpr bool TSP = L::TSP;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sKV = smem + L::OFF_KV;
  uint8_t* sP = smem + L::OFF_P;
  int* kmeta = reinterpret_cast<int*>(smem + L::OFF_META);
  float* red = reinterpret_cast<float*>(smem + L::OFF_RED);
  int* kmm = reinterpret_cast<int*>(smem + L::OFF_KMM);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;     // [2]
  uint64_t* kv_empty = bars + 3;   // [2]
  uint64_t* s_full = bars + 5;     // [2]
  uint64_t* s_free = bars + 7;     // [2]
  uint64_t* p_full = bars + 9;     // [2]
  uint64_t* p_free = bars + 11;    // [2]
  uint64_t* o_full = bars + 13;
  uint64_t* recv_bar = bars + 14;  // the peers' partials of my rows have landed (SPLIT_CLUSTER)
  uint64_t* v_full = bars + 15;    // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* kv_end_smem = reinterpret_cast<int*>(tmem_slot + 2);
  int& s_qmax = *reinterpret_cast<int*>(tmem_slot + 3);
  int& s_any = *reinterpret_cast<int*>(tmem_slot + 4);
  if ((int)(smem - smem_raw) + L::USED > L::TOTAL) {   // base less aligned than assumed: refuse instead of overrunning
    if (threadIdx.x == 0) report_timeout(p.status, KID_ATTN, 99, (unsigned)(smem - smem_raw));
    return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr bool CL = SPLIT == SPLIT_CLUSTER;        // the cluster lies along y
  const int tile = CL ? blockIdx.x : blockIdx.x / p.nsplit, split = CL ? (int)cluster_ctarank() : blockIdx.x % p.nsplit;
  const int kvh = CL ? blockIdx.y / p.nsplit : blockIdx.y, b = blockIdx.z;
  const int g = p.g;
  const int ROWS = CL ? p.cl_rows : ATT_M;
  const int q_chunk = ROWS * 128;                    // bytes of the query tile's 64-column chunks
  const bool direct = CL && ROWS == L::DIRECT_ROWS;  // peers send into room that no operand lies in
  const int pos_per_tile = ROWS / g;
  const int p0 = tile * pos_per_tile;
  // SPLIT_CLUSTER: the tile's valid rows, dealt to the CTAs in order; mine are [t0, t0 + own)
  const int rows_valid = min(pos_per_tile, p.Sq - p0) * g;
  const int rpr = (rows_valid + p.nsplit - 1) / p.nsplit;
  const int t0 = split * rpr, own = max(0, min(rpr, rows_valid - t0));

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&kv_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 256);
      mbar_init(&p_full[i], 256);
      mbar_init(&p_free[i], 1);
    }
    mbar_init(o_full, 1);
    if (CL) mbar_init(recv_bar, 1);
    *abort_flag = 0;
    *kv_end_smem = 0;
    mbar_fence_init();
    if (CL) mbar_expect_tx(recv_bar, (uint32_t)((p.nsplit - 1) * own * L::PART_LD * 4));
    tma_prefetch_desc(&tma_q);
    tma_prefetch_desc(&tma_k);
    tma_prefetch_desc(&tma_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;            // two buffers of BN columns
  const uint32_t tmem_O = tmem_base + 2 * BN;   // Dmma columns
  pdl_launch_dependents();                      // after the TMEM allocation (see common.cuh)
  if (direct) cluster_arrive();                 // waited for in front of the first copy to a peer: all have started
  if (CL && threadIdx.x == 0 && tile == 0) {
    // The cached keys and values have left L2 since the last pass: on their way while the preceding kernel finishes, requested
    // by the first tile of a kv head alone.  us with a norm in front, no requests / by every tile / by the first: 50 queries of 8
    // heads on 1 of 256 against 1018 keys 10.3 / 10.2 / 10.0, 4096 21.2 / 20.7 / 20.3, 32768 122.9 / 130.7 / 119.5; on 4, 4096 keys
    // 24.2 / 22.8 / 22.8; one query: within 0.2 of none
    const int all = (p.Sk + BN - 1) / BN, per = (all + p.nsplit - 1) / p.nsplit;
    for (int j = split * per; j < min(all, split * per + min(per, p.ahead)); ++j)
      for (int c = 0; c < L::NCHUNK; ++c) {
        l2_prefetch_4d(&tma_k, c * 64, kvh, j * BN, b);
        l2_prefetch_4d(&tma_v, c * 64, kvh, j * BN, b);
      }
  }
  pdl_wait();                                   // q / k / v and the masks come from the preceding kernels

  // ---- how many keys can this tile reach?  1 + the last key index j that is valid and has
  //      k_blk[j] <= the largest valid q_blk in the tile (no monotonicity assumed).  With split keys the scan is
  //      skipped: the few tiles of such a launch reach (almost) every key, blocks without a visible key cost one
  //      masked pass, and the scan itself is a serial prologue of two dependent global reads per key.  The same holds
  //      for a launch with ONE query tile per (batch, kv head): a short suffix attending to a cached prefix.
  if (p.skip_reach) {
    if (threadIdx.x == 0) *kv_end_smem = p.Sk;
    __syncthreads();
  } else {
    int qmax = INT_MIN;
    bool any_q = false;
    for (int i = threadIdx.x; i < pos_per_tile; i += blockDim.x) {
      int pos = p0 + i;
      if (pos < p.Sq && p.q_valid[(long long)b * p.Sq + pos]) {
        qmax = max(qmax, p.q_blk[(long long)b * p.Sq + pos]);
        any_q = true;
      }
    }
    // block-wide max of qmax (values) through shared atomics on a small scratch word
    if (threadIdx.x == 0) {
      s_qmax = INT_MIN;
      s_any = 0;
    }
    __syncthreads();
    if (any_q) {
      atomicMax(&s_qmax, qmax);
      atomicOr(&s_any, 1);
    }
    __syncthreads();
    int last = -1;
    if (s_any) {
      const int qm = s_qmax;
      // both loads are unconditional and the loop is unrolled, so several keys are in flight per thread
#pragma unroll 8
      for (int j = threadIdx.x; j < p.Sk; j += blockDim.x) {
        const int kbj = p.k_blk[(long long)b * p.Sk + j];
        const int kvj = p.k_valid[(long long)b * p.Sk + j];
        if (kvj && kbj <= qm) last = max(last, j);
      }
    }
    if (last >= 0) atomicMax(kv_end_smem, last + 1);
    __syncthreads();
  }
  const int kv_end = *kv_end_smem;
  const int nblk_all = max(1, (kv_end + BN - 1) / BN);
  // this CTA's key blocks [jb0, jb0 + nblk).  A split beyond the reachable keys still runs one block: every key in
  // it is invisible to the tile, so it contributes a zero row sum that the combine step ignores.
  const int per_split = (nblk_all + p.nsplit - 1) / p.nsplit;
  const int jb0 = split * per_split;
  const int nblk = max(1, min(nblk_all, jb0 + per_split) - jb0);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(q_full, L::Q_BYTES * ROWS / ATT_M);        // the rows past a smaller tile are never looked at
#pragma unroll
      for (int c = 0; c < L::NCHUNK; ++c)
        tma_load_4d(sQ + c * q_chunk, &tma_q, q_full, c * 64, kvh * g, p0, b);
      for (int j = 0; j < nblk; ++j) {
        const int slot = j & 1, u = j >> 1;
        mbar_wait(&kv_empty[slot], (u & 1) ^ 1, abort_flag, p.status, KID_ATTN, 1, j);
        uint8_t* sk = sKV + slot * L::STAGE_BYTES;
        uint8_t* sv = sk + L::KV_TILE;
        mbar_expect_tx(&k_full[slot], L::KV_TILE);
#pragma unroll
        for (int c = 0; c < L::NCHUNK; ++c) tma_load_4d(sk + c * (BN * 128), &tma_k, &k_full[slot], c * 64, kvh, (jb0 + j) * BN, b);
        mbar_expect_tx(&v_full[slot], L::KV_TILE);
#pragma unroll
        for (int c = 0; c < L::NCHUNK; ++c) tma_load_4d(sv + c * (BN * 128), &tma_v, &v_full[slot], c * 64, kvh, (jb0 + j) * BN, b);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_qk = make_idesc_bf16(ATT_M, BN, 0, 0);
      const uint32_t idesc_pv = make_idesc_bf16(ATT_M, p.Dmma, 0, 1);
      const int ksteps_qk = p.Dmma / 16;
      const uint32_t q_addr = smem_u32(sQ);
      auto issue_qk = [&](int j) {
        const int slot = j & 1, u = j >> 1;
        mbar_wait(&k_full[slot], u & 1, abort_flag, p.status, KID_ATTN, 2, j);
        // TSP: the scores of block j - 2 gave way to their P.  Block j's keys are in the slot of block j - 2, which the
        // producer filled behind the commit of the PV product that read that P: k_full stands for both
        if (!TSP) mbar_wait(&s_free[slot], (u & 1) ^ 1, abort_flag, p.status, KID_ATTN, 3, j);
        tc_fence_after();
        const uint32_t k_addr = smem_u32(sKV + slot * L::STAGE_BYTES);
        for (int kk = 0; kk < ksteps_qk; ++kk) {
          const int c = kk >> 2, w = kk & 3;
          uint64_t ad = make_smem_desc(q_addr + c * q_chunk + w * 32, 16, 1024);
          uint64_t bd = make_smem_desc(k_addr + c * (BN * 128) + w * 32, 16, 1024);
          umma_ss(tmem_S + slot * BN, ad, bd, idesc_qk, kk != 0 ? 1u : 0u);
        }
        umma_commit(&s_full[slot]);
      };
      mbar_wait(q_full, 0, abort_flag, p.status, KID_ATTN, 4, 0);
      issue_qk(0);
      for (int j = 0; j < nblk; ++j) {
        const int slot = j & 1, u = j >> 1;
        if (j + 1 < nblk) issue_qk(j + 1);
        mbar_wait(&p_full[slot], u & 1, abort_flag, p.status, KID_ATTN, 5, j);
        mbar_wait(&v_full[slot], u & 1, abort_flag, p.status, KID_ATTN, 11, j);
        tc_fence_after();
        const uint32_t p_addr = smem_u32(sP + slot * L::P_BYTES);
        const uint32_t v_addr = smem_u32(sKV + slot * L::STAGE_BYTES + L::KV_TILE);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          uint64_t bd = make_smem_desc(v_addr + kk * 2048, BN * 128, 1024);
          if (TSP) {
            // each half of the columns was written over the first columns of its own scores
            umma_ts(tmem_O, tmem_S + slot * BN + (kk / (BN / 32)) * (BN / 2) + (kk % (BN / 32)) * 8, bd, idesc_pv,
                    (j | kk) != 0 ? 1u : 0u);
          } else {
            uint64_t ad = make_smem_desc(p_addr + (kk >> 2) * (ATT_M * 128) + (kk & 3) * 32, 16, 1024);
            umma_ss(tmem_O, ad, bd, idesc_pv, (j | kk) != 0 ? 1u : 0u);
          }
        }
        umma_commit(&kv_empty[slot]);
        umma_commit(&p_free[slot]);
      }
      umma_commit(o_full);
    }
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    // Eight warps: two per TMEM lane quadrant.  Both threads of a pair own the same row (TMEM lane) and split the
    // columns of S, of P and of O between them; the row maximum (per block) and the row sum (once, at the end) are
    // exchanged through shared memory.  The scores of a block are read from TMEM once and stay in registers.
    // Masking is decided per 32 keys from the min / max block id of those keys: fully visible and fully hidden
    // groups take paths without per-element tests.
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;            // 0: first half of the columns, 1: second half
    const int row = quad * 32 + lane;            // TMEM lane owned by this thread
    const int st = threadIdx.x - 64;             // 0..255 index among softmax threads
    const int pos = p0 + row / g;
    const int head = kvh * g + row % g;
    const bool row_in = pos < p.Sq && row < ROWS;
    const bool q_ok = row_in && p.q_valid[(long long)b * p.Sq + pos] != 0;
    const int qb = q_ok ? p.q_blk[(long long)b * p.Sq + pos] : INT_MIN;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    constexpr int HB = BN / 2;                   // columns per thread
    constexpr int NCH = HB / 32;                 // 32-column groups per thread
    const int c0 = half * HB;
    float m_used = -INFINITY;   // maximum the accumulators are currently expressed against
    float l = 0.f;              // this thread's part of the row sum
    const float scale = p.scale_log2;
    const int n16 = p.Dmma / 16;
    const int o_lo = half ? (n16 + 1) / 2 : 0, o_hi = half ? n16 : (n16 + 1) / 2;   // this thread's O column groups

    auto load_meta = [&](int jj) -> int {
      const int key = (jb0 + jj) * BN + st;
      if (st >= BN || key >= p.Sk) return INT_MAX;
      const int kbv = p.k_blk[(long long)b * p.Sk + key];
      const int kvv = p.k_valid[(long long)b * p.Sk + key];
      return kvv ? kbv : INT_MAX;
    };
    int kb_next = load_meta(0);
    for (int j = 0; j < nblk; ++j) {
      const int slot = j & 1, u = j >> 1;
      if (st < BN) {                              // whole warps: st < BN covers warps 0 .. BN/32-1 of the group
        kmeta[slot * BN + st] = kb_next;
        const int mn = __reduce_min_sync(0xffffffffu, kb_next);
        const int mxk = __reduce_max_sync(0xffffffffu, kb_next);
        if (lane == 0) {
          kmm[(slot * (BN / 32) + st / 32) * 2 + 0] = mn;
          kmm[(slot * (BN / 32) + st / 32) * 2 + 1] = mxk;
        }
      }
      kb_next = (j + 1 < nblk) ? load_meta(j + 1) : INT_MAX;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const int* km = kmeta + slot * BN + c0;
      mbar_wait(&s_full[slot], u & 1, abort_flag, p.status, KID_ATTN, 6, j);
      tc_fence_after();
      const uint32_t s_addr = tmem_S + slot * BN + c0 + lane_off;
      // ---- read this thread's scores once; visibility class per 32 keys: 2 = all, 0 = none, 1 = test each
      uint32_t r[NCH][32];
      int cls[NCH];
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        __syncwarp();
        tmem_ld_x32(s_addr + c * 32, r[c]);
        const int gi = (slot * (BN / 32) + (c0 / 32) + c) * 2;
        const int gmin = kmm[gi], gmax = kmm[gi + 1];
        cls[c] = (!q_ok || gmin > qb) ? 0 : (gmax <= qb ? 2 : 1);
      }
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains instead of one
        if (cls[c] == 2) {
#pragma unroll
          for (int e = 0; e < 32; ++e) m4[e & 3] = fmaxf(m4[e & 3], __uint_as_float(r[c][e]));
        } else if (cls[c] == 1) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (km[c * 32 + e] <= qb) m4[e & 3] = fmaxf(m4[e & 3], __uint_as_float(r[c][e]));
        }
        mx = fmaxf(mx, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
      }
      mx *= scale;                                // scale > 0: max commutes with it
      red[half * ATT_M + row] = mx;
      asm volatile("bar.sync 2, 256;" ::: "memory");
      mx = fmaxf(mx, red[(half ^ 1) * ATT_M + row]);
      const float m_new = fmaxf(m_used, mx);
      // lazy rescale decision (warp-uniform because tcgen05.ld/st are warp-collective; both warps of a pair hold
      // the same rows and the same maxima, so they decide alike)
      const bool want = (m_new > m_used + 8.0f) || (m_used == -INFINITY && m_new != -INFINITY);
      const bool any_want = __any_sync(0xffffffffu, want);
      float alpha = 1.f;
      if (want) {
        alpha = (m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new);
        m_used = m_new;
      }
      // P buffer `slot` was last read by PV(j-2)
      if (!TSP && j >= 2) mbar_wait(&p_free[slot], ((u - 1) & 1), abort_flag, p.status, KID_ATTN, 7, j);
      if (any_want && j > 0) {
        // O may only be touched once PV(j-1) has retired
        const int ps = (j - 1) & 1, pu = (j - 1) >> 1;
        mbar_wait(&p_free[ps], pu & 1, abort_flag, p.status, KID_ATTN, 8, j);
        tc_fence_after();
        const uint32_t o_addr = tmem_O + lane_off;
#pragma unroll 1
        for (int c = o_lo; c < o_hi; ++c) {
          uint32_t ro[16];
          __syncwarp();
          tmem_ld_x16(o_addr + c * 16, ro);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) ro[e] = __float_as_uint(__uint_as_float(ro[e]) * alpha);
          tmem_st_x16(o_addr + c * 16, ro);
        }
        tmem_wait_st();
      }
      l *= alpha;
      // ---- probabilities -> bf16 -> swizzled shared memory or tensor memory (A operand of the PV product)
      uint8_t* prow = sP + slot * L::P_BYTES + row * 128;
      float lsum = 0.f;
      const float m_safe = (m_used == -INFINITY) ? 0.f : m_used;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        uint32_t packed[16];
        if (cls[c] == 2) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float p0f = fast_exp2(fmaf(__uint_as_float(r[c][e]), scale, -m_safe));
            const float p1f = fast_exp2(fmaf(__uint_as_float(r[c][e + 1]), scale, -m_safe));
            lsum += p0f + p1f;
            packed[e >> 1] = pack_bf16(p0f, p1f);
          }
        } else if (cls[c] == 1) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float p0f = km[c * 32 + e] <= qb ? fast_exp2(fmaf(__uint_as_float(r[c][e]), scale, -m_safe)) : 0.f;
            const float p1f =
                km[c * 32 + e + 1] <= qb ? fast_exp2(fmaf(__uint_as_float(r[c][e + 1]), scale, -m_safe)) : 0.f;
            lsum += p0f + p1f;
            packed[e >> 1] = pack_bf16(p0f, p1f);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) packed[e] = 0u;
        }
        if constexpr (TSP) {
          static_assert(NCH == 1, "a thread's scores are one piece");
          __syncwarp();
          tmem_st_x16(s_addr, packed);
          continue;
        }
        // 32 keys = 64 bytes = four 16-byte units; unit index within the 128-byte row is XOR-swizzled
        const int col = c0 + c * 32;
        const int chunk = col / 64;                // 64-key chunk (16 KB apart)
        const int unit0 = (col % 64) / 8;          // first 16-byte unit inside the row
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const int unit = (unit0 + q4) ^ (row & 7);
          uint4 val = make_uint4(packed[q4 * 4 + 0], packed[q4 * 4 + 1], packed[q4 * 4 + 2], packed[q4 * 4 + 3]);
          *reinterpret_cast<uint4*>(prow + chunk * (ATT_M * 128) + unit * 16) = val;
        }
      }
      l += lsum;
      // S buffer is free for QK(j+2); P is visible to the tensor core (async proxy)
      if constexpr (TSP) {
        tmem_wait_st();
        tc_fence_before();
      } else {
        tc_fence_before();
        mbar_arrive(&s_free[slot]);
        fence_async_smem();
      }
      mbar_arrive(&p_full[slot]);
    }

    // ---- epilogue: O / l -> bf16 -> global, LSE.  The two threads of a row add their partial sums first.
    asm volatile("bar.sync 1, 256;" ::: "memory");   // every read of `red` from the last block is done
    red[half * ATT_M + row] = l;
    asm volatile("bar.sync 2, 256;" ::: "memory");
    l += red[(half ^ 1) * ATT_M + row];
    mbar_wait(o_full, 0, abort_flag, p.status, KID_ATTN, 9, 0);
    tc_fence_after();
    const uint32_t o_addr = tmem_O + lane_off;
    if constexpr (CL) {
      // mine of all rows over operand tiles, which my own MMAs have left; the peers' of my rows in room of their own (32 rows), or
      // over operand tiles as well once all have left them
      float* part = reinterpret_cast<float*>(smem + (direct ? L::OFF_KV : 0));
      float* peers = reinterpret_cast<float*>(smem + (direct ? L::NCHUNK * q_chunk : L::OFF_PEER));
      if (quad * 32 < rows_valid) {                  // warp-uniform; every MMA of mine has retired: the tiles are free
        float* dst = part + row * L::PART_LD;
#pragma unroll 1
        for (int c = o_lo; c < o_hi; c += 2) {
          uint32_t ro[32];
          __syncwarp();
          tmem_ld_x16(o_addr + c * 16, ro);
          if (c + 1 < o_hi) tmem_ld_x16(o_addr + c * 16 + 16, ro + 16);
          tmem_wait_ld();
          const int n = c + 1 < o_hi ? 8 : 4;
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            if (q4 < n)
              *reinterpret_cast<uint4*>(dst + c * 16 + q4 * 4) =
                  make_uint4(ro[q4 * 4 + 0], ro[q4 * 4 + 1], ro[q4 * 4 + 2], ro[q4 * 4 + 3]);
        }
        if (half == 0) *reinterpret_cast<float2*>(dst + DPAD) = make_float2(m_used, l);
      }
      fence_async_smem();                            // the bulk copies read what was just written
      if (!direct) cluster_arrive();                 // after my last MMA: peers may write over my tiles
      cluster_wait();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      {
        const int owner = warp - 2;                  // a warp sends to one peer: lanes of one would go one after the other
        const int cnt = owner < p.nsplit ? min(rpr, rows_valid - owner * rpr) : 0;
        if (lane == 0 && owner != split && cnt > 0)
          bulk_to_peer(map_rank(smem_u32(peers) + (uint32_t)((split < owner ? split : split - 1) * rpr) * (L::PART_LD * 4u),
                                (uint32_t)owner),
                       smem_u32(part + owner * rpr * L::PART_LD), (uint32_t)cnt * (L::PART_LD * 4u),
                       map_rank(smem_u32(recv_bar), (uint32_t)owner));
        __syncwarp();
      }
      if (own > 0) mbar_wait(recv_bar, 0, abort_flag, p.status, KID_ATTN, 10, 0);
      __syncwarp();
      cluster_arrive();                              // my rows have all arrived; waited for before leaving
      const int rows = *abort_flag ? 0 : own;
      if (p.nsplit <= 4) merge_rows<DPAD, 4>(p, part + t0 * L::PART_LD, peers, split, rpr, rows, t0, p0, kvh, b, warp - 2, lane);
      else merge_rows<DPAD, 8>(p, part + t0 * L::PART_LD, peers, split, rpr, rows, t0, p0, kvh, b, warp - 2, lane);
    } else {
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* orow = p.o + (((long long)b * p.Sq + pos) * p.H + head) * p.D;
      float* prow_o = p.nsplit > 1
                          ? p.part_o + ((((long long)split * p.B + b) * p.Sq + pos) * p.H + head) * (long long)p.D
                          : nullptr;
#pragma unroll 1
      for (int c = o_lo; c < o_hi; ++c) {
        uint32_t ro[16];
        __syncwarp();
        tmem_ld_x16(o_addr + c * 16, ro);
        tmem_wait_ld();
        if (row_in && prow_o != nullptr) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            const int col = c * 16 + q4 * 4;
            if (col < p.D)
              *reinterpret_cast<float4*>(prow_o + col) =
                  make_float4(__uint_as_float(ro[q4 * 4 + 0]), __uint_as_float(ro[q4 * 4 + 1]),
                              __uint_as_float(ro[q4 * 4 + 2]), __uint_as_float(ro[q4 * 4 + 3]));
          }
        } else if (row_in) {
#pragma unroll
          for (int h8 = 0; h8 < 2; ++h8) {
            const int col = c * 16 + h8 * 8;
            if (col < p.D) {
              uint4 o;
              o.x = pack_bf16(__uint_as_float(ro[h8 * 8 + 0]) * inv_l, __uint_as_float(ro[h8 * 8 + 1]) * inv_l);
              o.y = pack_bf16(__uint_as_float(ro[h8 * 8 + 2]) * inv_l, __uint_as_float(ro[h8 * 8 + 3]) * inv_l);
              o.z = pack_bf16(__uint_as_float(ro[h8 * 8 + 4]) * inv_l, __uint_as_float(ro[h8 * 8 + 5]) * inv_l);
              o.w = pack_bf16(__uint_as_float(ro[h8 * 8 + 6]) * inv_l, __uint_as_float(ro[h8 * 8 + 7]) * inv_l);
              *reinterpret_cast<uint4*>(orow + col) = o;
            }
          }
        }
      }
      if (row_in && half == 0) {
        if (p.nsplit > 1) {
          p.part_ml[(((long long)split * p.B + b) * p.H + head) * p.Sq + pos] = make_float2(m_used, l);
        } else {
          const float lse = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : 0.f;
          p.lse[((long long)b * p.H + head) * p.Sq + pos] = lse;
        }
      }
    }
    tc_fence_before();
  }

  if (CL && warp < 2) {
    __syncwarp();
    if (!direct) cluster_arrive();
    cluster_wait();
    cluster_arrive();
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (CL) cluster_wait();                            // every copy out of my shared memory has arrived at its owner
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------ head widths above 128, keys unsplit
// At width 256 the kernel above keeps one tile of scores ahead, but all its softmax warps work on one block: 64 keys took 2970 clocks
// for 1024 of arithmetic (4096 positions, 8 heads on 1: 200 us).  Here the query tile lies in tensor memory (128 columns) beside
// two tiles of scores (64 each) and O (256), so a score product reads only keys from shared memory, and two groups of four warps take
// the blocks in turn, a thread a whole row.  What one group needs of the other is the row's maximum in use, which it publishes
// before its exponentials, and behind them the row's sums, which are so added in the order of the kernel above, to the same bits.
// P goes over the scores it was made from; scores of block j + 2 wait for the commit of the product that reads P of j.
// us, before / now: 4096 positions, 8 heads on 1, 1024 of them causal 191 / 104; 16 x 1227 (259 causal) 337 / 193; 2 x 1500, 8 on 4 80 /
// 55; 4 x 589 23 / 18; 5000, 4 heads of 160 236 / 135.  At 4096 a block takes 1700 clocks: the chain from scores to P and the products
// of two blocks that take turns.
template <int DPAD>
struct WideSmem {
  static constexpr int BN = 64, NCHUNK = DPAD / 64;
  static constexpr int Y_BYTES = BN * DPAD * 2;        // an item of the ring: 64 rows of Q, K or V
  static constexpr int NY = 7;
  static constexpr int OFF_M = NY * Y_BYTES;           // float [2 groups][128]: maxima in use
  static constexpr int OFF_L = OFF_M + 2 * ATT_M * 4;  // float2 [128]: row sums, handed from group to group
  static constexpr int OFF_BAR = OFF_L + ATT_M * 8;
  static constexpr int NBAR = 1 + 2 * NY + 6 + 16;
  static constexpr int USED = OFF_BAR + NBAR * 8 + 16;
  static constexpr int TOTAL = USED + 1024 <= 232448 ? USED + 1024 : 232448;
  static_assert(USED <= 232448, "shared memory budget");
  static constexpr int TM_Q = 0, TM_S = DPAD / 2, TM_O = DPAD / 2 + 2 * BN;
  static_assert(TM_O + DPAD <= 512, "tensor memory budget");
};

template <int DPAD>
__global__ void __launch_bounds__(320, 1)
attn_fwd_wide_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                     const __grid_constant__ CUtensorMap tma_v, AttnParams p) {
  using L = WideSmem<DPAD>;
  constexpr int BN = L::BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* m_pub = reinterpret_cast<float*>(smem + L::OFF_M);
  float2* l_pub = reinterpret_cast<float2*>(smem + L::OFF_L);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars;                       // the query tile is in tensor memory
  uint64_t* y_full = bars + 1;                   // [NY]
  uint64_t* y_empty = y_full + L::NY;            // [NY]
  uint64_t* s_full = y_empty + L::NY;            // [2]
  uint64_t* p_full = s_full + 2;                 // [2] P is in tensor memory
  uint64_t* pv_done = s_full + 4;                // [2] the product that reads it has retired
  uint64_t* m_ready = s_full + 6;                // [2][4 quadrants] a group's maxima are published
  uint64_t* l_ready = s_full + 14;               // [2][4 quadrants] and its row sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* reach = reinterpret_cast<int*>(tmem_slot + 2);
  if ((int)(smem - smem_raw) + L::USED > L::TOTAL) {   // base less aligned than assumed: refuse instead of overrunning
    if (threadIdx.x == 0) report_timeout(p.status, KID_ATTN, 99, (unsigned)(smem - smem_raw));
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // late tiles see the most keys where the text behind a prefix is causal: they go first
  const int tile = gridDim.x - 1 - blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int g = p.g, pos_per_tile = ATT_M / g, p0 = tile * pos_per_tile;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 256);
    for (int i = 0; i < L::NY; ++i) {
      mbar_init(&y_full[i], 1);
      mbar_init(&y_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&pv_done[i], 1);
    }
    for (int i = 0; i < 16; ++i) mbar_init(&m_ready[i], 32);               // and l_ready behind them
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_q);
    tma_prefetch_desc(&tma_k);
    tma_prefetch_desc(&tma_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                       // after the TMEM allocation (see common.cuh)
  pdl_wait();

  // ---- 1 + the last valid key with k_blk <= the tile's largest valid q_blk (no order assumed), searched from the end; the loads
  // of Q and of the first keys are on their way meanwhile (a tile that sees nothing runs one block).  All reads that the last 512 keys
  // take are in flight together, those of the queries beside them
  if (warp == 1) {
    int kb[16], kv[16];
    auto fetch_keys = [&](int end) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int j = end - 512 + i * 32 + lane;
        kb[i] = j >= 0 ? p.k_blk[(long long)b * p.Sk + j] : 0;
        kv[i] = j >= 0 ? p.k_valid[(long long)b * p.Sk + j] : 0;
      }
    };
    fetch_keys(p.Sk);
    int qb[4], qv[4];                            // pos_per_tile <= 128
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ps = p0 + i * 32 + lane;
      const bool in = i * 32 + lane < pos_per_tile && ps < p.Sq;
      qb[i] = in ? p.q_blk[(long long)b * p.Sq + ps] : 0;
      qv[i] = in ? p.q_valid[(long long)b * p.Sq + ps] : 0;
    }
    int qmax = INT_MIN, any = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (qv[i]) qmax = max(qmax, qb[i]);
      any |= qv[i];
    }
    qmax = __reduce_max_sync(0xffffffffu, qmax);
    any = __any_sync(0xffffffffu, any);
    int last = -1;
    for (int end = p.Sk; any && end > 0 && last < 0; end -= 512) {
      if (end < p.Sk) fetch_keys(end);
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (kv[i] && kb[i] <= qmax) last = max(last, end - 512 + i * 32 + lane);
      last = __reduce_max_sync(0xffffffffu, last);
    }
    if (lane == 0) *reach = last + 1;
  }
  auto load_item = [&](int s, const CUtensorMap* m, int head, int row) {
    mbar_expect_tx(&y_full[s], L::Y_BYTES);
#pragma unroll
    for (int c = 0; c < L::NCHUNK; ++c) tma_load_4d(smem + s * L::Y_BYTES + c * (BN * 128), m, &y_full[s], c * 64, head, row, b);
  };
  if (threadIdx.x == 0) {
    load_item(0, &tma_q, kvh * g, p0);
    load_item(1, &tma_q, kvh * g, p0 + 64 / g);
    load_item(2, &tma_k, kvh, 0);
  }
  __syncthreads();
  const int nblk = max(1, (*reach + BN - 1) / BN);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, in the order of use: K0 K1 V0 K2 V1 K3 ...
    if (elect_one()) {
      int s = 3;
      uint32_t ph = 1;                           // the ring's first round does not wait
      for (int i = 1; i < 2 * nblk; ++i) {
        // items: K0, then K_(i+1)/2 for odd i, V_(i/2 - 1) for even i; the last item is the last V
        const bool key = (i & 1) && (i + 1) / 2 < nblk;
        const int j = key ? (i + 1) / 2 : ((i & 1) ? nblk - 1 : i / 2 - 1);
        mbar_wait(&y_empty[s], ph, abort_flag, p.status, KID_ATTN, 1, i);
        load_item(s, key ? &tma_k : &tma_v, kvh, j * BN);
        if (++s == L::NY) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_qk = make_idesc_bf16(ATT_M, BN, 0, 0), idesc_pv = make_idesc_bf16(ATT_M, p.Dmma, 0, 1);
      const int ksteps = p.Dmma / 16;
      int s = 2;
      uint32_t ph = 0;
      auto next = [&]() {
        if (++s == L::NY) { s = 0; ph ^= 1; }
      };
      auto scores = [&](int j) {
        mbar_wait(&y_full[s], ph, abort_flag, p.status, KID_ATTN, 2, j);
        tc_fence_after();
        // 16-byte units: a chunk of 64 columns is 8 KB, a step in it 32 bytes
        const uint64_t bd = make_smem_desc(smem_u32(smem + s * L::Y_BYTES), 16, 1024);
        const uint32_t d = tmem_base + L::TM_S + (j & 1) * BN, a = tmem_base + L::TM_Q;
#pragma unroll
        for (int kk = 0; kk < DPAD / 16; ++kk)
          if (kk < ksteps) umma_ts(d, a + kk * 8, bd + (kk >> 2) * 512 + (kk & 3) * 2, idesc_qk, kk != 0 ? 1u : 0u);
        umma_commit(&y_empty[s]);
        umma_commit(&s_full[j & 1]);
        next();
      };
      mbar_wait(q_full, 0, abort_flag, p.status, KID_ATTN, 4, 0);
      tc_fence_after();
      mbar_arrive(&y_empty[0]);                  // the query tile has been copied out of the ring
      mbar_arrive(&y_empty[1]);
      scores(0);
      if (nblk > 1) scores(1);
      for (int j = 0; j < nblk; ++j) {
        const int buf = j & 1;
        mbar_wait(&p_full[buf], (j >> 1) & 1, abort_flag, p.status, KID_ATTN, 5, j);
        mbar_wait(&y_full[s], ph, abort_flag, p.status, KID_ATTN, 3, j);
        tc_fence_after();
        const uint64_t bd = make_smem_desc(smem_u32(smem + s * L::Y_BYTES), BN * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
          umma_ts(tmem_base + L::TM_O, tmem_base + L::TM_S + buf * BN + kk * 8, bd + kk * 128, idesc_pv, (j | kk) != 0 ? 1u : 0u);
        umma_commit(&y_empty[s]);
        umma_commit(&pv_done[buf]);
        next();
        if (j + 2 < nblk) {
          mbar_wait(&pv_done[buf], (j >> 1) & 1, abort_flag, p.status, KID_ATTN, 11, j);
          scores(j + 2);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: group `grp` takes every second block, a thread a row
    const int quad = warp & 3, grp = (warp - 2) >> 2, row = quad * 32 + lane;
    const int pos = p0 + row / g, head = kvh * g + row % g;
    const bool row_in = pos < p.Sq;
    const bool q_ok = row_in && p.q_valid[(long long)b * p.Sq + pos] != 0;
    const int qb = q_ok ? p.q_blk[(long long)b * p.Sq + pos] : INT_MIN;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const float scale = p.scale_log2;
    {
      // ---- the query tile into tensor memory: this thread's row, half of it
      const uint8_t* y = smem + (row >> 6) * L::Y_BYTES + (row & 63) * 128;
      mbar_wait(&y_full[row >> 6], 0, abort_flag, p.status, KID_ATTN, 12, 0);
#pragma unroll
      for (int c = 0; c < DPAD / 4; c += 32) {
        uint32_t r[32];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const int u8 = (grp * (DPAD / 4) + c + e) / 4;
          const uint4 v = *reinterpret_cast<const uint4*>(y + (u8 >> 3) * (BN * 128) + ((u8 & 7) ^ (row & 7)) * 16);
          r[e] = v.x; r[e + 1] = v.y; r[e + 2] = v.z; r[e + 3] = v.w;
        }
        __syncwarp();
        tmem_st_x32(tmem_base + L::TM_Q + lane_off + grp * (DPAD / 4) + c, r);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(q_full);
    }
    float m_used = -INFINITY;                    // maximum that O and the sums are expressed against
    auto key_id = [&](int j, int h) {            // of this lane's key of the block's half h
      const int key = j * BN + h * 32 + lane;
      if (j >= nblk || key >= p.Sk) return INT_MAX;
      const int kbv = p.k_blk[(long long)b * p.Sk + key];
      const int kvv = p.k_valid[(long long)b * p.Sk + key];
      return kvv ? kbv : INT_MAX;
    };
    // the maximum in use after block j, from the group that had it
    auto follow = [&](int j) {
      const int from = j & 1;
      mbar_wait(&m_ready[from * 4 + quad], (j >> 1) & 1, abort_flag, p.status, KID_ATTN, 13, j);
      m_used = m_pub[from * ATT_M + row];
    };
    // the row's sums up to block j: of the first and of the second 32 keys of every block, in the order of the blocks
    auto sums_of = [&](int j) {
      const int from = j & 1;
      mbar_wait(&l_ready[from * 4 + quad], (j >> 1) & 1, abort_flag, p.status, KID_ATTN, 14, j);
      return l_pub[row];
    };
    int nx0 = key_id(grp, 0), nx1 = key_id(grp, 1);
    for (int j = grp; j < nblk; j += 2) {
      const int kid[2] = {nx0, nx1};
      // visibility of 32 keys: to every row, to no row, or a test each; `hidden` has a bit for each key this row does not see
      bool all[2];
      unsigned hidden[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gmax = __reduce_max_sync(0xffffffffu, kid[h]);
        all[h] = __all_sync(0xffffffffu, q_ok && gmax <= qb);
        hidden[h] = 0;
        if (!all[h]) {
#pragma unroll
          for (int e = 0; e < 32; ++e) hidden[h] |= (__shfl_sync(0xffffffffu, kid[h], e) <= qb ? 0u : 1u) << e;
          if (!q_ok) hidden[h] = ~0u;
        }
      }
      nx0 = key_id(j + 2, 0);
      nx1 = key_id(j + 2, 1);
      mbar_wait(&s_full[grp], (j >> 1) & 1, abort_flag, p.status, KID_ATTN, 6, j);
      tc_fence_after();
      const uint32_t s_addr = tmem_base + L::TM_S + grp * BN + lane_off;
      uint32_t r[BN];
      __syncwarp();
      tmem_ld_x32(s_addr, r);
      tmem_ld_x32(s_addr + 32, r + 32);
      tmem_wait_ld();
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};          // four chains instead of one
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (all[h]) {
#pragma unroll
          for (int e = 0; e < 32; ++e) m4[e & 3] = fmaxf(m4[e & 3], __uint_as_float(r[h * 32 + e]));
        } else if (hidden[h] != ~0u) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (!(hidden[h] >> e & 1)) m4[e & 3] = fmaxf(m4[e & 3], __uint_as_float(r[h * 32 + e]));
        }
      }
      const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * scale;      // scale > 0: max commutes with it
      if (j > 0) follow(j - 1);
      // lazy rescale: only where the maximum grew by more than 2^8 (warp-uniform: tensor memory is accessed by whole warps)
      const float m_new = fmaxf(m_used, mx);
      const bool want = (m_new > m_used + 8.0f) || (m_used == -INFINITY && m_new != -INFINITY);
      float alpha = 1.f;
      if (want) {
        alpha = (m_used == -INFINITY) ? 0.f : fast_exp2(m_used - m_new);
        m_used = m_new;
      }
      m_pub[grp * ATT_M + row] = m_used;
      mbar_arrive(&m_ready[grp * 4 + quad]);
      if (__any_sync(0xffffffffu, want) && j > 0) {
        // O may only be touched once PV(j-1) has retired; PV(j) waits for this thread's P
        mbar_wait(&pv_done[grp ^ 1], ((j - 1) >> 1) & 1, abort_flag, p.status, KID_ATTN, 8, j);
        tc_fence_after();
        const uint32_t o_addr = tmem_base + L::TM_O + lane_off;
#pragma unroll 1
        for (int c = 0; c < p.Dmma; c += 16) {
          uint32_t ro[16];
          __syncwarp();
          tmem_ld_x16(o_addr + c, ro);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) ro[e] = __float_as_uint(__uint_as_float(ro[e]) * alpha);
          tmem_st_x16(o_addr + c, ro);
        }
        tmem_wait_st();
      }
      const float m_safe = (m_used == -INFINITY) ? 0.f : m_used;
      float lsum[2] = {0.f, 0.f};
      uint32_t packed[BN / 2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float a = fast_exp2(fmaf(__uint_as_float(r[h * 32 + e]), scale, -m_safe));
          float z = fast_exp2(fmaf(__uint_as_float(r[h * 32 + e + 1]), scale, -m_safe));
          if (!all[h]) {
            if (hidden[h] >> e & 1) a = 0.f;
            if (hidden[h] >> (e + 1) & 1) z = 0.f;
          }
          lsum[h] += a + z;
          packed[h * 16 + (e >> 1)] = pack_bf16(a, z);
        }
      }
      __syncwarp();
      tmem_st_x32(s_addr, packed);               // over the scores of my own row, which are all in registers
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&p_full[grp]);
      const float2 before = j > 0 ? sums_of(j - 1) : make_float2(0.f, 0.f);
      l_pub[row] = make_float2(fmaf(before.x, alpha, lsum[0]), fmaf(before.y, alpha, lsum[1]));
      mbar_arrive(&l_ready[grp * 4 + quad]);
    }

    // ---- epilogue: O / l -> bf16 -> global, LSE
    const int lastj = nblk - 1;
    if ((lastj & 1) != grp) follow(lastj);
    const float2 sums = sums_of(lastj);
    const float l = sums.x + sums.y;
    mbar_wait(&pv_done[lastj & 1], (lastj >> 1) & 1, abort_flag, p.status, KID_ATTN, 9, 0);
    tc_fence_after();
    const float inv_l = l > 0.f ? 1.f / l : 0.f;
    // a warp's 32 rows x half the width go through the ring, which nothing uses any more, and leave in whole pieces of a row:
    // a thread's own row in 16-byte pieces takes twice the time of the rest of the epilogue
    constexpr int LD = DPAD * 2 + 16;                    // bytes; the pad spreads the banks
    uint8_t* orow = smem + row * LD + grp * DPAD;
    const int cols = min(p.Dmma - grp * (DPAD / 2), DPAD / 2);
#pragma unroll 1
    for (int c = 0; c < cols; c += 16) {
      uint32_t ro[16];
      __syncwarp();
      tmem_ld_x16(tmem_base + L::TM_O + lane_off + grp * (DPAD / 2) + c, ro);
      tmem_wait_ld();
#pragma unroll
      for (int h8 = 0; h8 < 2; ++h8) {
        uint4 o;
        o.x = pack_bf16(__uint_as_float(ro[h8 * 8 + 0]) * inv_l, __uint_as_float(ro[h8 * 8 + 1]) * inv_l);
        o.y = pack_bf16(__uint_as_float(ro[h8 * 8 + 2]) * inv_l, __uint_as_float(ro[h8 * 8 + 3]) * inv_l);
        o.z = pack_bf16(__uint_as_float(ro[h8 * 8 + 4]) * inv_l, __uint_as_float(ro[h8 * 8 + 5]) * inv_l);
        o.w = pack_bf16(__uint_as_float(ro[h8 * 8 + 6]) * inv_l, __uint_as_float(ro[h8 * 8 + 7]) * inv_l);
        *reinterpret_cast<uint4*>(orow + c * 2 + h8 * 16) = o;
      }
    }
    __syncwarp();
    constexpr int LANES = DPAD / 16;                     // that write half a row
    const int col = grp * (DPAD / 2) + lane % LANES * 8;
#pragma unroll 4
    for (int i = lane / LANES; i < 32; i += 32 / LANES) {
      const int r = quad * 32 + i, rpos = p0 + r / g;
      if (rpos < p.Sq && col < p.D)
        *reinterpret_cast<uint4*>(p.o + (((long long)b * p.Sq + rpos) * p.H + kvh * g + r % g) * p.D + col) =
            *reinterpret_cast<const uint4*>(smem + r * LD + col * 2);
    }
    if (row_in && grp == 0)
      p.lse[((long long)b * p.H + head) * p.Sq + pos] = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : 0.f;
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

// Merge of the split-KV partials: one warp per (batch, position, head) row.
//   M = max_s m_s over splits with l_s > 0,  L = sum_s l_s 2^(m_s - M),  O = sum_s O_s 2^(m_s - M) / L
__global__ void attn_combine_kernel(const float* __restrict__ part_o, const float2* __restrict__ part_ml,
                                    __nv_bfloat16* __restrict__ o, float* __restrict__ lse, int nsplit, int B, int Sq,
                                    int H, int D) {
  pdl_launch_dependents();
  pdl_wait();
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long rows = (long long)B * Sq * H;
  if (row >= rows) return;
  const int head = int(row % H);
  const long long bp = row / H;                    // b * Sq + pos
  const int pos = int(bp % Sq), b = int(bp / Sq);
  // lane s < nsplit owns split s: (maximum, row sum); the weights travel by shuffle
  float m_s = -INFINITY, l_s = 0.f;
  if (lane < nsplit) {
    const float2 ml = part_ml[(((long long)lane * B + b) * H + head) * Sq + pos];
    l_s = ml.y;
    m_s = ml.y > 0.f ? ml.x : -INFINITY;
  }
  float M = m_s;
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));   // nsplit <= 8
  const float w_s = (m_s == -INFINITY) ? 0.f : fast_exp2(m_s - M);
  float L = l_s * w_s;
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
  M = __shfl_sync(0xffffffffu, M, 0);
  L = __shfl_sync(0xffffffffu, L, 0);
  const float inv = L > 0.f ? 1.f / L : 0.f;
  float w[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) w[s] = __shfl_sync(0xffffffffu, w_s, s) * inv;   // zero for s >= nsplit
  const long long split_stride = (long long)B * Sq * H * D;
  const float* src = part_o + (bp * H + head) * (long long)D;
  for (int c = lane; c < D / 4; c += 32) {
    float4 v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      v[s] = s < nsplit ? *reinterpret_cast<const float4*>(src + s * split_stride + c * 4) : make_float4(0, 0, 0, 0);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      acc.x += v[s].x * w[s]; acc.y += v[s].y * w[s]; acc.z += v[s].z * w[s]; acc.w += v[s].w * w[s];
    }
    uint2 packed = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
    *reinterpret_cast<uint2*>(o + row * D + c * 4) = packed;
  }
  if (lane == 0) lse[((long long)b * H + head) * Sq + pos] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : 0.f;
}

// rank-4 bf16 map over a (B, S, Hx, D) tensor with element strides (sb, ss, sh, 1); dims innermost first
static int make_map4(CUtensorMap* m, const void* base, int D, int Hx, int S, int B, long long sh, long long ss,
                     long long sb, int box_h, int box_s) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)Hx, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)sh * 2, (uint64_t)ss * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {64, (uint32_t)box_h, (uint32_t)box_s, 1};
  return make_tmap_bf16(m, base, 4, dims, strides, box);
}

template <int DPAD, int BN, int SPLIT>
static int launch_attn(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p,
                       cudaStream_t stream) {
  using L = AttnSmem<DPAD, BN, SPLIT>;
  static bool configured = false;
  auto kern = attn_fwd_kernel<DPAD, BN, SPLIT>;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int pos_per_tile = (SPLIT == SPLIT_CLUSTER ? p.cl_rows : ATT_M) / p.g;
  dim3 grid((p.Sq + pos_per_tile - 1) / pos_per_tile, p.Hkv, p.B);
  (SPLIT == SPLIT_CLUSTER ? grid.y : grid.x) *= p.nsplit;
  cudaError_t e = launch_pdl(kern, grid, dim3(320), (size_t)L::TOTAL, stream,
                             SPLIT == SPLIT_CLUSTER ? (unsigned)p.nsplit : 0u, tq, tk, tv, p);
  if (e != cudaSuccess || p.nsplit == 1 || SPLIT == SPLIT_CLUSTER) return (int)e;
  const long long rows = (long long)p.B * p.Sq * p.H;
  e = launch_pdl(attn_combine_kernel, dim3((unsigned)((rows * 32 + 255) / 256)), dim3(256), 0, stream, 0u,
                 (const float*)p.part_o, (const float2*)p.part_ml, p.o, p.lse, p.nsplit, p.B, p.Sq, p.H, p.D);
  return (int)e;
}

template <int DPAD>
static int launch_wide(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p, cudaStream_t stream) {
  using L = WideSmem<DPAD>;
  static bool configured = false;
  auto kern = attn_fwd_wide_kernel<DPAD>;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int pos_per_tile = ATT_M / p.g;
  return (int)launch_pdl(kern, dim3((p.Sq + pos_per_tile - 1) / pos_per_tile, p.Hkv, p.B), dim3(320), (size_t)L::TOTAL, stream, 0u,
                         tq, tk, tv, p);
}

}  // namespace otb

using namespace otb;

static int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}

template <int DPAD, int BN>
static int max_clusters(int n) {
  using L = AttnSmem<DPAD, BN, SPLIT_CLUSTER>;
  auto kern = attn_fwd_kernel<DPAD, BN, SPLIT_CLUSTER>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(1, (unsigned)n, 1);
  cfg.blockDim = dim3(320);
  cfg.dynamicSmemBytes = L::TOTAL;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = (unsigned)n;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  return cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess ? clusters : 0;
}

// whether `tiles` clusters of `n` CTAs are resident at once
static bool cluster_fits(int D, int n, long long tiles) {
  static int cap[3][9] = {};                         // -1: none
  if (n < 1 || n > 8) return false;
  const int which = D <= 64 ? 0 : (D <= 128 ? 1 : 2);
  int c = cap[which][n];
  if (c == 0) {
    c = which == 0 ? max_clusters<64, 128>(n) : which == 1 ? max_clusters<128, 128>(n) : max_clusters<256, 64>(n);
    cap[which][n] = c = c > 0 ? c : -1;
  }
  return tiles <= c;
}

// q: (B,Sq,H,D) strides (q_sb,q_ss,q_sh,1); k,v: (B,Sk,Hkv,D); o: (B,Sq,H,D) contiguous; lse: (B,H,Sq).
static int attn_fwd_impl(const void* q, const void* k, const void* v, void* o, float* lse, const int* q_blk,
                         const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid, int B, int Sq,
                         int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh, long long k_sb,
                         long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh, float scale,
                         int nsplit, float* part_o, float* part_ml, void* status, cudaStream_t stream) {
  if (nsplit < 1 || nsplit > 8) return -7;
  // split without scratch: one cluster per tile of 64 or 32 rows merges on chip
  const bool cluster = nsplit > 1 && part_o == nullptr;
  if (nsplit > 1 && !cluster && (part_ml == nullptr || D % 4)) return -7;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || H <= 0 || Hkv <= 0 || H % Hkv) return -2;
  const int g = H / Hkv;
  if (g > 128 || (128 % g) || (cluster && g > CL_ROWS)) return -3;
  if (D % 8 || D > 256 || D < 16) return -4;
  const long long strides[9] = {q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh};
  for (int i = 0; i < 9; ++i)
    if (strides[i] % 8) return -5;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o)) & 15)
    return -6;
  AttnParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.D = D; p.g = g;
  p.Dmma = (D + 15) / 16 * 16;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.q_blk = q_blk; p.k_blk = k_blk; p.q_valid = q_valid; p.k_valid = k_valid;
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.nsplit = nsplit;
  p.skip_reach = (nsplit > 1 || Sq <= ATT_M / g) ? 1 : 0;
  p.part_o = part_o;
  p.part_ml = reinterpret_cast<float2*>(part_ml);
  p.status = static_cast<KernelStatus*>(status);
  const int dpad = D <= 64 ? 64 : (D <= 128 ? 128 : 256);
  // Head widths up to 128, more tiles than SMs: two CTAs per SM.  us inside a replayed graph, one CTA per SM against two: 16 heads
  // of 72, 24 x 256 positions 52.3 / 34.4 (768 tiles), 3 x 1024 61.6 / 53.1, 8 x 256 18.6 / 13.2; 32 heads of 128 on 8, 2 x 2048
  // 228.6 / 178.7, 700 31.2 / 23.1 (176 tiles); with a tile per SM there is nothing to share it with: 3 x 256 of 72 9.7 / 11.1 (96
  // tiles), 300 of 128 11.0 / 13.3 (80)
  const bool two = dpad <= 128 && nsplit == 1 && (long long)((Sq + ATT_M / g - 1) / (ATT_M / g)) * Hkv * B > sm_count();
  const int bn = dpad == 256 || two ? 64 : 128;
  CUtensorMap tq, tk, tv;
  // 32-row tiles halve what a cluster's CTAs send one another, where twice the clusters are still resident at once.  Every tile
  // streams all keys, so the gain fades with their number: us with a norm in front, 64 / 32 rows, 50 queries of 8 heads on 1 of 256
  // (13 clusters): 384 keys 10.7 / 9.1, 1018 11.7 / 10.0, 4096 21.8 / 20.3, 16384 62.3 / 62.6, 32768 123.2 / 119.5; 20 of 4 heads on
  // 1 of 64, 4096 keys 12.0 / 11.9.  Clusters in two rounds lose: 50 queries of 8 heads on 4, 1074 keys 13.8 / 18.8
  p.cl_rows = CL_ROWS;
  if (cluster && g <= 32 && cluster_fits(D, nsplit, ((long long)Sq * g + 31) / 32 * Hkv * B)) p.cl_rows = 32;
  // what a launch requests ahead stays a quarter of L2
  const long long block_bytes = 4LL * bn * dpad * Hkv * B * nsplit;
  p.ahead = (int)((32LL << 20) / block_bytes);
  // unsplit, head width above 128 (64 rows of a query tile at a time: groups up to 64).  Where a kv head has one query tile the other
  // kernel does not look for the last visible key, and of a few blocks that and the query tile's way into tensor memory are the larger
  // part: us, 8 heads on 1 of 256, wide / other, 148 tiles of 96 rows against 20, 100, 192 and 256 keys 8.9 / 7.2, 9.5 / 8.8, 10.9 / 10.3 and
  // 11.9 / 11.6; 600 tiles 36.6 / 31.5, 42.9 / 42.0, 48.5 / 55.0 and 53.1 / 64.6.  With more tiles to a kv head both look, and wide wins
  // (tiles of 248 rows against 20 and 128 keys 8.2 / 9.0 and 8.7 / 10.1)
  const bool brief = p.skip_reach && (Sk <= 64 || (Sk <= 192 && (long long)Hkv * B <= 2 * sm_count()));
  const bool wide = dpad == 256 && nsplit == 1 && g <= 64 && !brief;
  int r = make_map4(&tq, q, D, H, Sq, B, q_sh, q_ss, q_sb, g, (cluster ? p.cl_rows : (wide ? 64 : ATT_M)) / g);
  if (r) return 1000 + r;
  r = make_map4(&tk, k, D, Hkv, Sk, B, k_sh, k_ss, k_sb, 1, bn);
  if (r) return 2000 + r;
  r = make_map4(&tv, v, D, Hkv, Sk, B, v_sh, v_ss, v_sb, 1, bn);
  if (r) return 3000 + r;
#define RUN(DP, BLK) (cluster ? launch_attn<DP, BLK, SPLIT_CLUSTER>(tq, tk, tv, p, stream) \
                              : launch_attn<DP, BLK, SPLIT_GLOBAL>(tq, tk, tv, p, stream))
  switch (dpad) {
    case 64: return two ? launch_attn<64, 64, SPLIT_TWO>(tq, tk, tv, p, stream) : RUN(64, 128);
    case 128: return two ? launch_attn<128, 64, SPLIT_TWO>(tq, tk, tv, p, stream) : RUN(128, 128);
    default: return wide ? launch_wide<256>(tq, tk, tv, p, stream) : RUN(256, 64);
  }
#undef RUN
}

extern "C" int otb_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int* q_blk,
                            const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid, int B,
                            int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh,
                            long long k_sb, long long k_ss, long long k_sh, long long v_sb, long long v_ss,
                            long long v_sh, float scale, void* status, cudaStream_t stream) {
  return attn_fwd_impl(q, k, v, o, lse, q_blk, k_blk, q_valid, k_valid, B, Sq, Sk, H, Hkv, D, q_sb, q_ss, q_sh, k_sb,
                       k_ss, k_sh, v_sb, v_ss, v_sh, scale, 1, nullptr, nullptr, status, stream);
}

// Split-KV form: `nsplit` (2..8) CTAs per query tile share the key blocks; part_o holds nsplit*B*Sq*H*D floats and
// part_ml 2*nsplit*B*H*Sq floats of scratch, or both are null and a cluster merges on chip.  Same result as otb_attn_fwd up to fp32 rounding of the merge.
extern "C" int otb_attn_fwd_splitkv(const void* q, const void* k, const void* v, void* o, float* lse, const int* q_blk,
                                    const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid,
                                    int B, int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss,
                                    long long q_sh, long long k_sb, long long k_ss, long long k_sh, long long v_sb,
                                    long long v_ss, long long v_sh, float scale, int nsplit, float* part_o,
                                    float* part_ml, void* status, cudaStream_t stream) {
  return attn_fwd_impl(q, k, v, o, lse, q_blk, k_blk, q_valid, k_valid, B, Sq, Sk, H, Hkv, D, q_sb, q_ss, q_sh, k_sb,
                       k_ss, k_sh, v_sb, v_ss, v_sh, scale, nsplit, part_o, part_ml, status, stream);
}

// CTAs per cluster for `tiles` tiles of 64 rows (the launch may then halve the tiles): the most (up to 8) whose clusters are all
// resident at once, since a second round costs more than anything a larger cluster saves; 1 if not even pairs are.  Measured at 50
// queries of 8 heads on 1, width 256, against the best of one pass and a merge through global memory, us: 7 tiles, 1018 keys, 8 CTAs
// 8.1 / 17; 28 tiles, 639 keys, 4 11.7 / 17.1; 42 tiles, 900 keys, 3 15.6 / 20.1; pairs, 70 tiles of 560 and 1018 keys 15.2 / 16.3 and
// 20.1 / 23.2 (the caller says where pairs lose).  Clusters that do not fit lose (28 tiles with 8: 20.5).
extern "C" int otb_attn_cluster_fit(int D, long long tiles) {
  for (int n = 8; n >= 2; --n)
    if (cluster_fits(D, n, tiles)) return n;
  return 1;
}

// key-block width the forward kernel uses for this head dimension (callers size split-KV from it)
extern "C" int otb_attn_block(int D) { return D > 128 ? 64 : 128; }
