// Block-causal flash attention backward for sm_100a with the bf16 operands P and dS kept in global memory.
//
// dQ = dS K, dK = dS^T Q and dV = P^T dO contract over P and dS as bf16 tensor-core operands.  Recomputing them for each output
// (attention_bwd_tcgen05.cu, three kernels) takes eight products where five are needed, and at head width 256 one accumulator
// fills half of the tensor memory, so that scores have no second buffer and every block waits for the elementwise work.
// Here the operands are made once and stored:
//
//   attn_bwd_cover_kernel    how many blocks of 64 keys each pair of query tiles has to visit, and which 64 rows of it see any
//   attn_bwd_scores_kernel   tile = 128 query rows (position x head of the group), streams blocks of 64 keys:
//                              S = Q K_j^T, dP = dO V_j^T -> P, dS = P o (dP - delta) * scale -> bf16 -> global
//                            No accumulator: both fixed tiles lie in tensor memory beside two pairs of (S, dP), so the products of
//                            one block run under the elementwise work of the other.  One block an SM; the visited (tile, key
//                            block) pairs are dealt to them in equal runs.
//   attn_bwd_products_kernel CTA pairs, one to two SMs, take jobs of one output tile: 256 rows of dQ over the key blocks, or 256 keys
//                            of dK / dV over the query rows or a part of them.  Two accumulators: a job's end runs under the next.
//
// A stored block is the 16 KB image that its 128 rows x 64 keys have in shared memory under the 128-byte swizzle.  As it is, it is
// a K-major A operand (dQ); rows 64 h .. 64 h + 63 of it are 8 contiguous KB and a 64-key chunk of an MN-major A operand (dK, dV).  So
// it is written by bulk copies of contiguous memory and read without another swizzle.
//
// Hidden blocks are neither computed nor stored: the first cover[b][t] key blocks of query tiles 2 t and 2 t + 1 are, in whole tiles
// of dK and dV (four blocks) or up to the last key.  The products multiply P and dS, zeros included, by what stands in K, Q and dO, where
// padding may hold anything: dQ ends with the pair's last visible block, and dK and dV leave out every 64 rows that see nothing.
// Results are deterministic: no atomics, fixed order of accumulation.
//
// us for the whole backward, recomputing / stored: 4096 positions, 8 heads on 1 of 256, 1024 of them causal 556 / 306; 8 x 1227 and
// 16 x 1227 (259 causal; a training step's layer) 577 / 274 and 938 / 508; 2 x 700, 8 on 4 115 / 45; 2 x 2048, 32 on 8 of 128 744 / 488;
// 24 x 256 and 3 x 1024, 16 of 72 211 / 124 and 196 / 146; 2 x 3000, 16 of 64 783 / 558; 2 x 566, 16 of 72 94 / 60, 200 of 256 76 / 27; up to
// about 300 positions of few samples a call is the host's time either way (33 us of launches, 37 recomputing).  Many samples of
// one tile lose (2048 x 6 3534 / 5337) and stay with the recomputing kernels (stored_bwd_samples).
// What bounds it: at 16 x 1227 the scores take 248 us, 1.5 us a block of 128 x 64, with DRAM at 48 % of its peak (0.63 GB written, 0.37 read
// of q, o, dO and what other tiles' writes push out of L2), the tensor pipe at 34 % and issue slots at 47 %: the chain of a block from its
// products through tensor memory and the elementwise warps to the staged images, and the start of every query tile (fixed tiles, delta)
// that nothing runs under.  4096 positions, longer runs of one tile, 1.2 us a block.  The products read P and dS three times, 240 us for 1.2 GB;
// with their A operands in L2 they would take 183.  Tried
// and slower: S and dP of 128 keys without a second buffer (scores 117 -> 138 us at 4096 positions), eight elementwise warps (160),
// all scores of a thread in registers at once (168: spills), storing warps of their own (127), products cut into runs
// of equal length with fp32 sums at the cuts (289 -> 315 us in all: the streams of the pairs drift apart in memory).
#include "common.cuh"
#include <limits.h>

namespace otb {

constexpr unsigned KID_BWD_SCORES = 8;
constexpr unsigned KID_BWD_PRODUCTS = 9;
constexpr int ST_M = 128;                      // query rows of a tile
constexpr int ST_BN = 64;                      // keys of a stored block
constexpr int ST_IMAGE = ST_M * ST_BN;         // elements of a stored block

struct StoredParams {
  int B, Sq, Sk, H, Hkv, D, g;
  int ptiles, kblks, key_tiles;                // pairs of query tiles; key blocks of the scratch; tiles of 256 keys
  int splits;                                  // parts of a dK / dV tile's query rows
  int dq_more;                                 // dQ jobs of the CTA pairs that have one dK / dV job more than others, all together
  float scale, scale_log2;
  const int* q_blk;
  const int* k_blk;
  const unsigned char* q_valid;
  const unsigned char* k_valid;
  const float* lse;                            // (B, H, Sq), natural log
  const __nv_bfloat16* o;                      // (B, Sq, H, D) contiguous
  __nv_bfloat16 *P, *dS;                       // (B, Hkv, 2 ptiles, kblks, ST_IMAGE)
  int* cover;                                  // (B, ptiles): key blocks of a pair, whole tiles of dK and dV
  unsigned* reach;                             // (B, ptiles): blocks up to the last visible key; bit 28 + i: rows 64 i .. see any
  __nv_bfloat16 *dq, *dk, *dv;                 // contiguous
  float *dk_parts, *dv_parts;                  // splits > 1: (splits, B, Sk, Hkv, D) fp32
  KernelStatus* status;
};

__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar) & PEER_BIT_MASK), "r"(x), "r"(y), "r"(z),
      "r"(w)
      : "memory");
}
__device__ __forceinline__ float st_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ------------------------------------------------------------------------------------------ cover
constexpr unsigned REACH_MASK = (1u << 28) - 1;   // blocks; above it the four bits
// One block per pair of query tiles: 1 + the last valid key with k_blk <= the pair's largest valid q_blk (no order assumed), searched
// from the end a thousand keys at a time until every 64 rows with a valid one have found a key.
__global__ void __launch_bounds__(256) attn_bwd_cover_kernel(StoredParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, b = blockIdx.y, pos_per = 2 * ST_M / p.g;
  __shared__ int s_qmax[4], s_last;
  __shared__ unsigned s_any, s_found;
  if (threadIdx.x < 4) s_qmax[threadIdx.x] = INT_MIN;
  if (threadIdx.x == 0) {
    s_last = -1;
    s_any = s_found = 0;
  }
  // the queries and the last thousand keys in one round trip
  int kb[4], kv[4];
  auto fetch_keys = [&](int end) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = end - 1024 + i * 256 + (int)threadIdx.x;
      kb[i] = j >= 0 ? p.k_blk[(long long)b * p.Sk + j] : 0;
      kv[i] = j >= 0 ? p.k_valid[(long long)b * p.Sk + j] : 0;
    }
  };
  fetch_keys(p.Sk);
  const int ps = t * pos_per + threadIdx.x, quarter = threadIdx.x * p.g / 64;
  const bool in = (int)threadIdx.x < pos_per && ps < p.Sq;                                   // pos_per <= 256
  const int qblk = in ? p.q_blk[(long long)b * p.Sq + ps] : INT_MIN;
  const bool any = in && p.q_valid[(long long)b * p.Sq + ps] != 0;
  const int some = __syncthreads_or(any);
  if (any) {
    atomicMax(&s_qmax[quarter], qblk);
    atomicOr(&s_any, 1u << quarter);
  }
  __syncthreads();
  int qmax[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) qmax[i] = s_qmax[i];
  const unsigned asked = s_any;
  for (int end = p.Sk; some && end > 0; end -= 1024) {
    if (end < p.Sk) fetch_keys(end);
    int last = -1;
    unsigned found = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned sees = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) sees |= (kv[i] && kb[i] <= qmax[q] ? 1u : 0u) << q;
      if (sees & asked) last = max(last, end - 1024 + i * 256 + (int)threadIdx.x);
      found |= sees & asked;
    }
    last = __reduce_max_sync(0xffffffffu, last);
    found = __reduce_or_sync(0xffffffffu, found);
    if (found && (threadIdx.x & 31) == 0) {
      atomicMax(&s_last, last);
      atomicOr(&s_found, found);
    }
    __syncthreads();
    if (__syncthreads_and(s_found == asked)) break;
  }
  if (threadIdx.x == 0) {
    const int blocks = (s_last + ST_BN) / ST_BN;
    p.reach[(long long)b * p.ptiles + t] = (unsigned)blocks | s_found << 28;
    p.cover[(long long)b * p.ptiles + t] = min((blocks + 3) / 4 * 4, p.kblks);
  }
}

// ------------------------------------------------------------------------------------------ P and dS
constexpr int SC_WARPS = 16;                   // elementwise warps
constexpr int SC_THREADS = 64 + SC_WARPS * 32;

template <int DPAD>
struct ScoreSmem {
  static constexpr int NCHUNK = DPAD / 64;
  static constexpr int Y_BYTES = ST_BN * DPAD * 2;                // an item of the ring: 64 rows of Q, dO, K or V
  static constexpr int NY = DPAD == 256 ? 5 : 8;
  static constexpr int OFF_ST = NY * Y_BYTES;                     // [2 groups][4 quadrants]: 32 rows of P, 32 rows of dS
  static constexpr int OFF_DELTA = OFF_ST + 8 * 8192;             // float [2][128]
  static constexpr int OFF_BAR = OFF_DELTA + 2 * ST_M * 4;
  static constexpr int NBAR = 1 + 2 * NY + 4;
  static constexpr int USED = OFF_BAR + NBAR * 8 + 16;
  static constexpr int TOTAL = USED + 1024 <= 232448 ? USED + 1024 : 232448;
  static_assert(USED <= 232448, "shared memory budget");
  static constexpr int TM_F1 = 0, TM_F2 = DPAD / 2, TM_S = DPAD, TM_DP = DPAD + 2 * ST_BN;
  static_assert(TM_DP + 2 * ST_BN <= 512, "tensor memory budget");
};

// A run of key blocks of one query tile.
struct Segment {
  int b, kvh, tile, blk0, nblk;
};
// The visited (sample, pair of tiles, kv head, tile of the pair, key block) in this order, cut into gridDim.x runs of equal length;
// every role of a block walks through its run by itself.
struct SegmentWalk {
  const int* cover;
  int Hkv, ptiles, e, c;
  long long off, left;
  __device__ SegmentWalk(const StoredParams& p, int lane) : cover(p.cover), Hkv(p.Hkv), ptiles(p.ptiles), e(0), c(0) {
    const int n = p.B * p.ptiles;
    long long total = 0;
    for (int i = lane; i < n; i += 32) total += cover[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    total *= 2 * Hkv;
    const long long start = total * blockIdx.x / gridDim.x;
    left = total * (blockIdx.x + 1) / gridDim.x - start;
    off = start;
    for (int base = 0; base < n && left > 0; base += 32) {
      const long long w = base + lane < n ? 2ll * Hkv * cover[base + lane] : 0;
      long long incl = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const unsigned here = __ballot_sync(0xffffffffu, incl > off);
      if (here != 0) {
        const int l = __ffs(here) - 1;
        e = base + l;
        off -= __shfl_sync(0xffffffffu, incl - w, l);
        break;
      }
      off -= __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __device__ bool next(Segment& s) {
    if (left <= 0) return false;
    while ((c = cover[e]) == 0) ++e;
    const int r = (int)off;
    s.b = e / ptiles;
    s.kvh = r / (2 * c);
    const int rem = r - s.kvh * 2 * c, sub = rem >= c;
    s.tile = 2 * (e - s.b * ptiles) + sub;
    s.blk0 = rem - sub * c;
    s.nblk = (int)min((long long)(c - s.blk0), left);
    left -= s.nblk;
    off += s.nblk;
    if (off == 2ll * c * Hkv) {
      off = 0;
      ++e;
    }
    return true;
  }
};

template <int DPAD>
__global__ void __launch_bounds__(SC_THREADS, 1)
attn_bwd_scores_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, StoredParams p) {
  using L = ScoreSmem<DPAD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* f_full = bars;                       // a run's fixed tiles are in tensor memory, its delta in shared memory
  uint64_t* y_full = bars + 1;                   // [NY]
  uint64_t* y_empty = y_full + L::NY;            // [NY]
  uint64_t* sd_full = y_empty + L::NY;           // [2] S and dP of a block
  uint64_t* sd_free = sd_full + 2;               // [2] they have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if ((int)(smem - smem_raw) + L::USED > L::TOTAL) {              // base less aligned than assumed: refuse instead of overrunning
    if (threadIdx.x == 0) report_timeout(p.status, KID_BWD_SCORES, 99, (unsigned)(smem - smem_raw));
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = p.g;

  if (threadIdx.x == 0) {
    mbar_init(f_full, SC_WARPS * 32);
    for (int i = 0; i < L::NY; ++i) {
      mbar_init(&y_full[i], 1);
      mbar_init(&y_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sd_full[i], 1);
      mbar_init(&sd_free[i], SC_WARPS * 16);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
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

  SegmentWalk walk(p, lane);
  Segment sg;
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: Q, Q, dO, dO, then K_j, V_j of a run's blocks
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 1;                           // the ring's first round does not wait
      auto slot = [&](int what) {
        mbar_wait(&y_empty[s], ph, abort_flag, p.status, KID_BWD_SCORES, 1, what);
        mbar_expect_tx(&y_full[s], L::Y_BYTES);
        return smem + s * L::Y_BYTES;
      };
      auto advance = [&]() {
        if (++s == L::NY) { s = 0; ph ^= 1; }
      };
      while (walk.next(sg)) {
        for (int i = 0; i < 4; ++i) {
          uint8_t* y = slot(i);
          const int pos = (sg.tile * ST_M + (i & 1) * 64) / g;
#pragma unroll
          for (int c = 0; c < L::NCHUNK; ++c)
            tma_load_4d(y + c * 8192, i < 2 ? &tm_q : &tm_do, &y_full[s], c * 64, sg.kvh * g, pos, sg.b);
          advance();
        }
        for (int i = 0; i < 2 * sg.nblk; ++i) {
          uint8_t* y = slot(4 + i);
          const int key = (sg.blk0 + (i >> 1)) * ST_BN;
#pragma unroll
          for (int c = 0; c < L::NCHUNK; ++c)
            tma_load_4d(y + c * 8192, (i & 1) ? &tm_v : &tm_k, &y_full[s], c * 64, sg.kvh, key, sg.b);
          advance();
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(ST_M, ST_BN, 0, 0);
      const int ksteps = (p.D + 15) / 16;
      int s = 0, n = 0;
      uint32_t ph = 0, fph = 0;
      auto advance = [&]() {
        if (++s == L::NY) { s = 0; ph ^= 1; }
      };
      while (walk.next(sg)) {
        mbar_wait(f_full, fph, abort_flag, p.status, KID_BWD_SCORES, 2, n);
        fph ^= 1;
        for (int i = 0; i < 4; ++i) {            // the fixed tiles have been copied out of the ring
          mbar_arrive(&y_empty[s]);
          advance();
        }
        for (int j = 0; j < sg.nblk; ++j, ++n) {
          const int buf = n & 1;
          if (n > 1) mbar_wait(&sd_free[buf], ((n >> 1) - 1) & 1, abort_flag, p.status, KID_BWD_SCORES, 3, n);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mbar_wait(&y_full[s], ph, abort_flag, p.status, KID_BWD_SCORES, 4, n);
            tc_fence_after();
            const uint32_t y = smem_u32(smem + s * L::Y_BYTES);
            const uint32_t d = tmem_base + (h ? L::TM_DP : L::TM_S) + buf * ST_BN, f = tmem_base + (h ? L::TM_F2 : L::TM_F1);
            for (int kk = 0; kk < ksteps; ++kk) {
              uint64_t bd = make_smem_desc(y + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024);
              umma_ts(d, f + kk * 8, bd, idesc, kk != 0 ? 1u : 0u);
            }
            umma_commit(&y_empty[s]);
            advance();
          }
          umma_commit(&sd_full[buf]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ elementwise: 32 rows x 32 keys of every second block a warp
    const int ew = warp - 2, quad = warp & 3, grp = ew >> 3, half = (ew >> 2) & 1, row = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    float* delta = reinterpret_cast<float*>(smem + L::OFF_DELTA);
    uint8_t* stage = smem + L::OFF_ST + (grp * 4 + quad) * 8192;
    const uint32_t out_u = smem_u32(stage) + half * 4096;         // what this warp sends off: the pair's P or its dS
    uint8_t* prow = stage + lane * 128;
    const int pair_bar = 1 + grp * 4 + quad;
    constexpr int PARTS = DPAD >= 128 ? 4 : 2, CW = DPAD / 2 / PARTS;      // 32-bit columns of a fixed row that a thread copies
    const int part = grp * 2 + half;
    int n = 0, items = 0, seg = 0;
    while (walk.next(sg)) {
      const int p0 = sg.tile * (ST_M / g);
      const int pos = p0 + row / g, head = sg.kvh * g + row % g;
      // rows of O for delta: eight a warp, a row in one access
      uint4 orow[ST_M / SC_WARPS];
#pragma unroll
      for (int i = 0; i < ST_M / SC_WARPS; ++i) {
        const int r = ew * (ST_M / SC_WARPS) + i, rp = p0 + r / g;
        orow[i] = make_uint4(0u, 0u, 0u, 0u);
        if (rp < p.Sq && lane * 8 < p.D)
          orow[i] = *reinterpret_cast<const uint4*>(p.o + (((long long)sg.b * p.Sq + rp) * p.H + sg.kvh * g + r % g) * p.D + lane * 8);
      }
      const bool row_ok = pos < p.Sq && p.q_valid[(long long)sg.b * p.Sq + pos] != 0;
      int row_blk = 0;
      float row_lse2 = 0.f;
      if (row_ok) {
        row_blk = p.q_blk[(long long)sg.b * p.Sq + pos];
        row_lse2 = p.lse[((long long)sg.b * p.H + head) * p.Sq + pos] * 1.4426950408889634f;
      }
      // every product of the last run has read its fixed tiles
      if (n > 0) mbar_wait(&sd_full[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, p.status, KID_BWD_SCORES, 5, n);
      auto item = [&](int i) {                   // waits for the run's i-th item
        const int at = items + i, s = at % L::NY;
        mbar_wait(&y_full[s], (at / L::NY) & 1, abort_flag, p.status, KID_BWD_SCORES, 6, i);
        return smem + s * L::Y_BYTES;
      };
      tc_fence_after();
#pragma unroll
      for (int w = 0; w < 2; ++w) {              // Q, then dO
        const uint8_t* y = item(2 * w + (row >> 6));
        if (part < PARTS) {
          uint32_t r[CW];
#pragma unroll
          for (int e = 0; e < CW; e += 4) {
            const int u8 = (part * CW + e) / 4;                   // 16-byte unit of the row
            const uint4 v = *reinterpret_cast<const uint4*>(y + (u8 >> 3) * 8192 + (row & 63) * 128 + ((u8 & 7) ^ (row & 7)) * 16);
            r[e] = v.x; r[e + 1] = v.y; r[e + 2] = v.z; r[e + 3] = v.w;
          }
          __syncwarp();
          const uint32_t dst = tmem_base + lane_off + (w ? L::TM_F2 : L::TM_F1) + part * CW;
          if (CW == 32) tmem_st_x32(dst, r);
          else tmem_st_x16(dst, r);
        }
      }
#pragma unroll
      for (int i = 0; i < ST_M / SC_WARPS; ++i) {
        const int r = ew * (ST_M / SC_WARPS) + i;
        const uint8_t* y = item(2 + (r >> 6));
        float acc = 0.f;
        if (lane * 8 < p.D) {
          const uint4 x = *reinterpret_cast<const uint4*>(y + (lane >> 3) * 8192 + (r & 63) * 128 + ((lane & 7) ^ (r & 7)) * 16);
          const uint32_t a[4] = {orow[i].x, orow[i].y, orow[i].z, orow[i].w}, z[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 u = unpack_bf16(a[k]), v = unpack_bf16(z[k]);
            acc += u.x * v.x + u.y * v.y;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) delta[(seg & 1) * ST_M + r] = acc;
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(f_full);
      mbar_wait(f_full, seg & 1, abort_flag, p.status, KID_BWD_SCORES, 7, seg);
      const float row_ds = delta[(seg & 1) * ST_M + row] * p.scale;
      items += 4 + 2 * sg.nblk;
      ++seg;

      const long long image0 = (((long long)sg.b * p.Hkv + sg.kvh) * (2 * p.ptiles) + sg.tile) * p.kblks + sg.blk0;
      __nv_bfloat16* out = (half ? p.dS : p.P) + image0 * ST_IMAGE + quad * (32 * ST_BN);
      auto key_id = [&](int j) {                 // of this lane's key of the warp's 32
        const int key = (sg.blk0 + j) * ST_BN + half * 32 + lane;
        if (j >= sg.nblk || key >= p.Sk) return INT_MAX;
        const int kbv = p.k_blk[(long long)sg.b * p.Sk + key];
        const int kvv = p.k_valid[(long long)sg.b * p.Sk + key];
        return kvv ? kbv : INT_MAX;
      };
      const int j0 = (n & 1) == grp ? 0 : 1;
      int nx = key_id(j0);
      for (int j = j0; j < sg.nblk; j += 2) {
        const int kid = nx;
        nx = key_id(j + 2);
        const int gmin = __reduce_min_sync(0xffffffffu, kid), gmax = __reduce_max_sync(0xffffffffu, kid);
        // visibility of the 32 keys: to every row, to no row, or a test each
        const bool all = __all_sync(0xffffffffu, row_ok && gmax <= row_blk), none = __all_sync(0xffffffffu, !row_ok || gmin > row_blk);
        mbar_wait(&sd_full[grp], ((n + j) >> 1) & 1, abort_flag, p.status, KID_BWD_SCORES, 8, n + j);
        tc_fence_after();
        const uint32_t s_addr = tmem_base + L::TM_S + grp * ST_BN + half * 32 + lane_off;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t rs[16], rd[16], pk[8], dk[8];
          __syncwarp();
          tmem_ld_x16(s_addr + c * 16, rs);
          tmem_ld_x16(s_addr + (L::TM_DP - L::TM_S) + c * 16, rd);
          tmem_wait_ld();
          if (c == 1) {
            tc_fence_before();
            mbar_arrive(&sd_free[grp]);
          }
          if (none) {
#pragma unroll
            for (int e = 0; e < 8; ++e) pk[e] = dk[e] = 0u;
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              rs[e] = __float_as_uint(st_exp2(fmaf(__uint_as_float(rs[e]), p.scale_log2, -row_lse2)));
              rd[e] = __float_as_uint(__uint_as_float(rs[e]) * fmaf(__uint_as_float(rd[e]), p.scale, -row_ds));
            }
            if (!all) {
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const int id = __shfl_sync(0xffffffffu, kid, c * 16 + e);          // by the whole warp
                const bool see = row_ok && id <= row_blk;
                rs[e] = see ? rs[e] : 0u;
                rd[e] = see ? rd[e] : 0u;
              }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              pk[e] = pack_bf16(__uint_as_float(rs[2 * e]), __uint_as_float(rs[2 * e + 1]));
              dk[e] = pack_bf16(__uint_as_float(rd[2 * e]), __uint_as_float(rd[2 * e + 1]));
            }
          }
          if (c == 0) {                          // the pair's last block has left the staging tile
            if (lane == 0) bulk_wait_read();
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
          }
#pragma unroll
          for (int q2 = 0; q2 < 2; ++q2) {
            const int unit = ((half * 4 + c * 2 + q2) ^ (lane & 7)) * 16;
            *reinterpret_cast<uint4*>(prow + unit) = make_uint4(pk[q2 * 4], pk[q2 * 4 + 1], pk[q2 * 4 + 2], pk[q2 * 4 + 3]);
            *reinterpret_cast<uint4*>(prow + 4096 + unit) = make_uint4(dk[q2 * 4], dk[q2 * 4 + 1], dk[q2 * 4 + 2], dk[q2 * 4 + 3]);
          }
        }
        fence_async_smem();
        asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
        if (lane == 0) {
          bulk_store(out + (long long)j * ST_IMAGE, out_u, 4096);
          bulk_commit();
        }
      }
      n += sg.nblk;
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
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

// ------------------------------------------------------------------------------------------ dQ, dK, dV
// Two CTAs (two SMs) hold one 256-row tile: `tcgen05.mma.cta_group::2`, each with its own 128 rows of A and accumulator and half of
// the columns of B.  Barriers as in the CTA-pair GEMM: full[s] and tempty[b] are the leader's (rank 0), empty[s] and tfull[b] are
// committed to both.  One CTA fills an SM's shared memory on purpose: pairs that share SMs could wait for each other's tensor memory.
template <int DPAD>
struct ProductSmem {
  static constexpr int NCH = DPAD == 256 ? 2 : 1;                 // 64-column chunks of this CTA's half of B
  static constexpr int A_BYTES = ST_M * 64 * 2, B_BYTES = NCH * 8192, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = DPAD == 256 ? 6 : 8;
  static constexpr int OFF_BAR = STAGES * STAGE_BYTES;
  static constexpr int TOTAL = OFF_BAR + (2 * STAGES + 4) * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 2 * DPAD;
};
constexpr int PR_THREADS = 192;                  // warp 0 copies, warp 1 MMA, warps 2..5 epilogue

// A job: 0 dQ of a query pair, 1 dK or 2 dV of a key tile and a part of its query pairs; steps of 64 along the contraction.
struct Job {
  int which, b, kvh, tile, split, lo, nsteps;
};
// Pair i takes the dK / dV jobs i, i + pairs, ...: long ones, all of one length; then a run of dQ jobs: an equal share of the first
// `dq_more` where it has one of the former more than others, of the rest where it has not.  Every role walks through the jobs by itself.
struct JobWalk {
  const StoredParams& p;
  int lane, pair, pairs, kv, next_kv, n_kv, next_q, end_q;
  __device__ JobWalk(const StoredParams& q, int l) : p(q), lane(l), pair(blockIdx.x >> 1), pairs(gridDim.x >> 1) {
    kv = p.B * p.Hkv;
    n_kv = kv * 2 * p.key_tiles * p.splits;
    next_kv = pair;
    const int n_q = kv * p.ptiles, more = n_kv % pairs;
    const bool has_more = pair < more;
    const int first = has_more ? 0 : p.dq_more, jobs = has_more ? p.dq_more : n_q - p.dq_more;
    const int i = has_more ? pair : pair - more, of = has_more ? more : pairs - more;
    next_q = first + (int)((long long)jobs * i / of);
    end_q = first + (int)((long long)jobs * (i + 1) / of);
  }
  __device__ bool next(Job& j) {                 // by whole warps
    int sample_head;
    if (next_kv < n_kv) {
      int r = next_kv;
      j.which = 1 + r % 2;
      r /= 2;
      j.split = r % p.splits;
      r /= p.splits;
      j.tile = r % p.key_tiles;
      sample_head = r / p.key_tiles;
      next_kv += pairs;
    } else if (next_q < end_q) {
      j.which = j.split = 0;
      j.tile = next_q % p.ptiles;
      sample_head = next_q / p.ptiles;
      ++next_q;
    } else {
      return false;
    }
    j.b = sample_head / p.Hkv;
    j.kvh = sample_head - j.b * p.Hkv;
    const unsigned* reach = p.reach + (long long)j.b * p.ptiles;
    j.lo = 0;
    if (j.which == 0) {
      j.nsteps = reach[j.tile] & REACH_MASK;
    } else {                                     // a part takes pairs in equal numbers, of each pair the 64 rows that see any key
      auto steps_of = [&](int t) {
        const unsigned r = t < p.ptiles ? reach[t] : 0u;
        return (r & REACH_MASK) > 4u * j.tile ? __popc(r >> 28) : 0;
      };
      int n = 0, steps = 0;
      for (int t0 = 0; t0 < p.ptiles; t0 += 32) {
        const int mine = steps_of(t0 + lane);
        n += __popc(__ballot_sync(0xffffffffu, mine > 0));
        steps += mine;
      }
      steps = __reduce_add_sync(0xffffffffu, steps);
      if (p.splits > 1) {
        j.lo = (int)((long long)n * j.split / p.splits);
        const int hi = (int)((long long)n * (j.split + 1) / p.splits);
        if (steps == 4 * n) {                    // all rows of all pairs
          j.nsteps = 4 * (hi - j.lo);
          return true;
        }
        steps = 0;
        for (int t0 = 0, seen = 0; t0 < p.ptiles && seen < hi; t0 += 32) {
          const int mine = steps_of(t0 + lane);
          const unsigned in = __ballot_sync(0xffffffffu, mine > 0);
          const int at = seen + __popc(in & ((1u << lane) - 1));
          if (at >= j.lo && at < hi) steps += mine;
          seen += __popc(in);
        }
        steps = __reduce_add_sync(0xffffffffu, steps);
      }
      j.nsteps = steps;
    }
    return true;
  }
};

template <int DPAD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PR_THREADS, 1)
attn_bwd_products_kernel(const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_ds,
                         const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                         const __grid_constant__ CUtensorMap tm_k, StoredParams p) {
  using L = ProductSmem<DPAD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* empty_bar = full_bar + L::STAGES;
  uint64_t* tfull_bar = empty_bar + L::STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int n2 = (p.D + 31) / 32 * 32;           // columns of the product: a multiple of 32 for pairs

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull_bar[i], 1);
      mbar_init(&tempty_bar[i], 256);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, L::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                            // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                       // after the TMEM allocation (see common.cuh)
  pdl_wait();

  JobWalk walk(p, lane);
  Job j;
  if (warp == 0) {
    // ------------------------------------------------------------------ producer (both CTAs)
    int s0 = 0;
    uint32_t ph0 = 1;
    const int x0 = rank * (n2 >> 1);
    while (walk.next(j)) {
      const long long images = ((long long)j.b * p.Hkv + j.kvh) * (2 * p.ptiles) * p.kblks;
      const unsigned* reach = p.reach + (long long)j.b * p.ptiles;
      int s = s0;                                // the elected lane's position in the ring
      uint32_t ph = ph0;
      auto slot = [&](int what) {
        mbar_wait(&empty_bar[s], ph, abort_flag, p.status, KID_BWD_PRODUCTS, 1, what);
        if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * L::STAGE_BYTES);
        return smem + s * L::STAGE_BYTES;
      };
      auto advance = [&]() {
        if (++s == L::STAGES) { s = 0; ph ^= 1; }
      };
      if (elect_one()) {
        if (j.which == 0) {
          const int row0 = (int)(images + (long long)(2 * j.tile + rank) * p.kblks) * ST_M;
          for (int i = 0; i < j.nsteps; ++i) {
            uint8_t* sa = slot(i);
#pragma unroll
            for (int h = 0; h < 2; ++h) tma_load_2d_pair(sa + h * 8192, &tm_ds, &full_bar[s], 0, row0 + i * ST_M + h * 64);
#pragma unroll
            for (int c = 0; c < L::NCH; ++c)
              tma_load_4d_pair(sa + L::A_BYTES + c * 8192, &tm_k, &full_bar[s], x0 + c * 64, j.kvh, i * 64, j.b);
            advance();
          }
        } else {
          const CUtensorMap* ta = j.which == 1 ? &tm_ds : &tm_p;
          const CUtensorMap* tb = j.which == 1 ? &tm_q : &tm_do;
          for (int t = 0, seen = 0, left = j.nsteps; left > 0 && t < p.ptiles; ++t) {
            const unsigned r = reach[t];
            if ((r & REACH_MASK) <= 4u * j.tile || seen++ < j.lo) continue;
#pragma unroll 1
            for (unsigned rows = r >> 28; rows != 0; rows &= rows - 1) {        // 64 rows: half a tile of the pair
              const int q = __ffs(rows) - 1;
              --left;
              const int tq = 2 * t + (q >> 1);
              const int row0 = (int)(images + (long long)tq * p.kblks + 4 * j.tile + 2 * rank) * ST_M + (q & 1) * 64;
              uint8_t* sa = slot(t);
#pragma unroll
              for (int h = 0; h < 2; ++h) tma_load_2d_pair(sa + h * 8192, ta, &full_bar[s], 0, row0 + h * ST_M);
#pragma unroll
              for (int c = 0; c < L::NCH; ++c)
                tma_load_4d_pair(sa + L::A_BYTES + c * 8192, tb, &full_bar[s], x0 + c * 64, j.kvh * p.g,
                                 (tq * ST_M + (q & 1) * 64) / p.g, j.b);
              advance();
            }
          }
        }
      }
      __syncwarp();
      s0 += j.nsteps;
      ph0 ^= (s0 / L::STAGES) & 1;
      s0 %= L::STAGES;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    int s = 0, acc = 0;
    uint32_t ph = 0, acc_ph = 0;
    while (rank == 0 && walk.next(j)) {
      if (elect_one()) {
        const bool mn = j.which != 0;            // dK, dV: the stored rows are the contraction
        const uint32_t idesc = make_idesc_bf16(2 * ST_M, n2, mn ? 1 : 0, 1);
        const uint32_t a_lbo = mn ? 8192u : 16u, a_step = mn ? 2048u : 32u;
        const uint32_t d = tmem_base + acc * DPAD;
        mbar_wait(&tempty_bar[acc], acc_ph ^ 1, abort_flag, p.status, KID_BWD_PRODUCTS, 2, acc);
        tc_fence_after();
        int s1 = s;
        uint32_t ph1 = ph;
        for (int i = 0; i < j.nsteps; ++i) {
          mbar_wait(&full_bar[s1], ph1, abort_flag, p.status, KID_BWD_PRODUCTS, 3, i);
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s1 * L::STAGE_BYTES), sb = sa + L::A_BYTES;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint64_t ad = make_smem_desc(sa + k * a_step, a_lbo, 1024);
            uint64_t bd = make_smem_desc(sb + k * 2048, 8192, 1024);
            umma_ss_pair(d, ad, bd, idesc, (i | k) != 0 ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s1]);
          if (++s1 == L::STAGES) { s1 = 0; ph1 ^= 1; }
        }
        umma_commit_pair(&tfull_bar[acc]);
      }
      __syncwarp();
      s += j.nsteps;
      ph ^= (s / L::STAGES) & 1;
      s %= L::STAGES;
      acc ^= 1;
      if (acc == 0) acc_ph ^= 1;
    }
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs)
    const int quad = warp & 3, row = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_ph = 0;
    while (walk.next(j)) {
      bool in;
      long long off;
      __nv_bfloat16* out;
      float* part = nullptr;
      if (j.which == 0) {
        const int pos = (2 * j.tile + rank) * (ST_M / p.g) + row / p.g, head = j.kvh * p.g + row % p.g;
        in = pos < p.Sq;
        off = (((long long)j.b * p.Sq + pos) * p.H + head) * p.D;
        out = p.dq;
      } else {
        const int key = (2 * j.tile + rank) * ST_M + row;
        in = key < p.Sk;
        off = (((long long)j.b * p.Sk + key) * p.Hkv + j.kvh) * p.D;
        out = j.which == 1 ? p.dk : p.dv;
        if (p.splits > 1)
          part = (j.which == 1 ? p.dk_parts : p.dv_parts) + (long long)j.split * p.B * p.Sk * p.Hkv * p.D;
      }
      mbar_wait(&tfull_bar[acc], acc_ph, abort_flag, p.status, KID_BWD_PRODUCTS, 4, acc);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < n2; c += 32) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld_x32(tmem_base + acc * DPAD + (uint32_t(quad * 32) << 16) + c, r);
        tmem_wait_ld();
        if (j.nsteps == 0) {                     // nothing sees these rows
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
        if (in) {
#pragma unroll
          for (int h8 = 0; h8 < 4; ++h8) {
            const int col = c + h8 * 8;
            if (col >= p.D) break;
            const uint32_t* v = r + h8 * 8;
            if (part != nullptr) {
              *reinterpret_cast<uint4*>(part + off + col) = make_uint4(v[0], v[1], v[2], v[3]);
              *reinterpret_cast<uint4*>(part + off + col + 4) = make_uint4(v[4], v[5], v[6], v[7]);
            } else {
              uint4 o;
              o.x = pack_bf16(__uint_as_float(v[0]), __uint_as_float(v[1]));
              o.y = pack_bf16(__uint_as_float(v[2]), __uint_as_float(v[3]));
              o.z = pack_bf16(__uint_as_float(v[4]), __uint_as_float(v[5]));
              o.w = pack_bf16(__uint_as_float(v[6]), __uint_as_float(v[7]));
              *reinterpret_cast<uint4*>(out + off + col) = o;
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive_leader(&tempty_bar[acc]);
      acc ^= 1;
      if (acc == 0) acc_ph ^= 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                            // nobody leaves while its peer may still signal its barriers or read its tiles
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, L::TMEM_COLS);
  }
}

// out[i] = bf16(sum over `splits` parts of 8 n8 floats each, in order); y: dK, dV
__global__ void attn_bwd_parts_kernel(const float* __restrict__ dk_parts, const float* __restrict__ dv_parts,
                                      __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, long long n8, int splits) {
  pdl_launch_dependents();
  pdl_wait();
  const float* parts = blockIdx.y ? dv_parts : dk_parts;
  __nv_bfloat16* out = blockIdx.y ? dv : dk;
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

static int st_map(CUtensorMap* m, const void* base, int D, int Hx, int S, int B, long long sh, long long ss, long long sb,
                  int box_h, int box_s) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)Hx, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)sh * 2, (uint64_t)ss * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {64, (uint32_t)box_h, (uint32_t)box_s, 1};
  return make_tmap_bf16(m, base, 4, dims, strides, box);
}
// the stored blocks as rows of 64 elements, 64 rows at a time, copied as they lie (they are swizzled already)
static int image_map(CUtensorMap* m, const void* base, long long rows) {
  PFN_encodeTiled enc = get_encode_fn();
  if (!enc) return -1;
  cuuint64_t dims[2] = {64, (cuuint64_t)rows}, strides[1] = {128};
  cuuint32_t box[2] = {64, 64}, es[2] = {1, 1};
  return (int)enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// How the jobs of dQ, dK and dV are dealt to CTA pairs: the pairs with one dK / dV job more than others take `more_q` dQ jobs together,
// the others the rest, so that the longest share is shortest; returns its steps (an end of a job counts as four).  With 36 (sample, kv
// head)s of one tile each 72 of 74 pairs have a dK / dV job: left to the other two, the 36 dQ jobs take 54 us (one query of 32 heads,
// width 256), one to every second of the 72 25.
static double deal_jobs(long long kv, long long pt, long long kb, long long kt, int splits, int pairs, int* more_q) {
  const long long n_kv = kv * 2 * kt * splits, n_q = kv * pt, base = n_kv / pairs, more = n_kv % pairs;
  const double len_kv = 4.0 * ((pt + splits - 1) / splits) + 4.0, len_q = kb + 4.0;
  const double mean = (n_kv * len_kv + n_q * len_q) / pairs;
  // as many to each pair of `more` as end by the mean, or one more
  long long q = more ? (long long)((mean - (base + 1) * len_kv) / len_q) : 0;
  if (q < 0) q = 0;
  double best = 0.0;
  for (int i = 0; i < (more ? 2 : 1); ++i, ++q) {
    const long long jobs = q * more < n_q ? q * more : n_q, rest = n_q - jobs;
    const double first = more ? (base + 1) * len_kv + (jobs + more - 1) / more * len_q : 0.0;
    const double second = base * len_kv + (rest + pairs - more - 1) / (pairs - more) * len_q;
    const double longest = first > second ? first : second;
    if (i == 0 || longest < best) {
      best = longest;
      *more_q = (int)jobs;
    }
  }
  return best;
}

static int st_sms() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms > 0 ? sms : 148;
}

struct StoredMaps {
  CUtensorMap q, d_o, k, v, p, ds;
};

template <int DPAD>
static int launch_stored(const StoredMaps& m, const StoredParams& p, int pairs, cudaStream_t stream) {
  auto ks = attn_bwd_scores_kernel<DPAD>;
  auto kp = attn_bwd_products_kernel<DPAD>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(ks, cudaFuncAttributeMaxDynamicSharedMemorySize, ScoreSmem<DPAD>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, ProductSmem<DPAD>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  cudaError_t e = launch_pdl(attn_bwd_cover_kernel, dim3((unsigned)p.ptiles, (unsigned)p.B), dim3(256), 0, stream, 0u, p);
  if (e != cudaSuccess) return (int)e;
  const long long blocks = 2ll * p.ptiles * p.kblks * p.Hkv * p.B;
  const int sms = st_sms();
  e = launch_pdl(ks, dim3((unsigned)(blocks < sms ? blocks : sms)), dim3(SC_THREADS), ScoreSmem<DPAD>::TOTAL, stream, 0u, m.q, m.d_o,
                 m.k, m.v, p);
  if (e != cudaSuccess) return (int)e;
  e = launch_pdl(kp, dim3((unsigned)(2 * pairs)), dim3(PR_THREADS), ProductSmem<DPAD>::TOTAL, stream, 0u, m.p, m.ds, m.q, m.d_o, m.k, p);
  if (e != cudaSuccess || p.splits == 1) return (int)e;
  const long long n8 = (long long)p.B * p.Sk * p.Hkv * p.D / 8;
  return (int)launch_pdl(attn_bwd_parts_kernel, dim3((unsigned)((n8 + 255) / 256), 2), dim3(256), 0, stream, 0u,
                         (const float*)p.dk_parts, (const float*)p.dv_parts, p.dk, p.dv, n8, p.splits);
}

}  // namespace otb

using namespace otb;

constexpr int ST_MAX_SPLITS = 16;

// Sizes of a call: bytes of P (dS takes the same), ints of cover, parts of a dK / dV tile's rows (above 1 they want that many fp32
// copies of dK and of dV).
extern "C" void otb_attn_bwd_stored_plan(int B, int Sq, int Sk, int H, int Hkv, int D, long long* operand_bytes, int* cover_ints,
                                         int* kv_splits) {
  const int g = H / Hkv, pairs = st_sms() / 2;
  const long long pt = (Sq + 2 * ST_M / g - 1) / (2 * ST_M / g), kb = (Sk + ST_BN - 1) / ST_BN, kt = (kb + 3) / 4, kv = (long long)Hkv * B;
  *operand_bytes = kv * 2 * pt * kb * ST_IMAGE * 2;
  *cover_ints = (int)(2 * B * pt);               // and, behind it, reach
  // the longest share of a CTA pair, and the parts' sums
  *kv_splits = 1;
  const double dpad = D <= 64 ? 64 : (D <= 128 ? 128 : 256), step_us = 0.3 * (0.4 + 0.6 * dpad / 256);
  const double out_bytes = 4.0 * B * Sk * Hkv * D;
  double best = 0;
  for (int s = 1; s <= ST_MAX_SPLITS && s <= pt && (s == 1 || s * out_bytes <= 256.0 * (1 << 20)); ++s) {
    int more_q;
    const double cost = deal_jobs(kv, pt, kb, kt, s, pairs, &more_q) * step_us + (s > 1 ? 5.0 + 2 * out_bytes * (2 * s + 0.5) / 5e6 : 0.0);
    if (s == 1 || cost < best) {
      best = cost;
      *kv_splits = s;
    }
  }
}

// dQ jobs that the pairs with one dK / dV job more than others take together (deal_jobs), for tests on the host.
extern "C" int otb_attn_bwd_stored_deal(int kv, int ptiles, int kblks, int key_tiles, int splits, int pairs) {
  int more_q = 0;
  deal_jobs(kv, ptiles, kblks, key_tiles, splits, pairs, &more_q);
  return more_q;
}

// Arguments of one call (mirrored field by field by the ctypes structure of the Python launcher).  q (B,Sq,H,D), k / v (B,Sk,Hkv,D)
// with element strides; o, do (B,Sq,H,D) contiguous; lse (B,H,Sq); dq, dk, dv contiguous outputs; P, dS, cover, *_parts: scratch.
struct OtbAttnBwdStored {
  const void *q, *k, *v, *o, *d_o;
  const float* lse;
  void *dq, *dk, *dv;
  void *P, *dS;
  int* cover;
  float *dk_parts, *dv_parts;
  const int *q_blk, *k_blk;
  const unsigned char *q_valid, *k_valid;
  void* status;
  long long strides[9];                          // q, k, v: sample, position, head
  int B, Sq, Sk, H, Hkv, D;
  int kv_splits;
  float scale;
};

extern "C" int otb_attn_bwd_stored(const OtbAttnBwdStored* a, cudaStream_t stream) {
  const int B = a->B, Sq = a->Sq, Sk = a->Sk, H = a->H, Hkv = a->Hkv, D = a->D;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || H <= 0 || Hkv <= 0 || H % Hkv || B > 65535 || Hkv > 65535) return -2;
  const int g = H / Hkv;
  if (g > 32 || (32 % g)) return -3;
  if (D % 8 || D > 256 || D < 16) return -4;
  for (int i = 0; i < 9; ++i)
    if (a->strides[i] % 8) return -5;
  // rows are read and written in 128-bit pieces and bulk copies by the kernels themselves, not only through tensor maps
  const void* const bases[10] = {a->q, a->k, a->v, a->o, a->d_o, a->dq, a->dk, a->dv, a->P, a->dS};
  for (int i = 0; i < 10; ++i)
    if (bases[i] == nullptr || (reinterpret_cast<uintptr_t>(bases[i]) & 15)) return -6;
  if (a->kv_splits < 1 || a->kv_splits > ST_MAX_SPLITS || a->cover == nullptr) return -7;
  if (a->kv_splits > 1 && (a->dk_parts == nullptr || a->dv_parts == nullptr ||
                           ((reinterpret_cast<uintptr_t>(a->dk_parts) | reinterpret_cast<uintptr_t>(a->dv_parts)) & 15)))
    return -7;
  StoredParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.D = D; p.g = g;
  p.ptiles = (Sq + 2 * ST_M / g - 1) / (2 * ST_M / g);
  p.kblks = (Sk + ST_BN - 1) / ST_BN;
  p.key_tiles = (p.kblks + 3) / 4;
  p.splits = a->kv_splits;
  p.scale = a->scale;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.q_blk = a->q_blk; p.k_blk = a->k_blk; p.q_valid = a->q_valid; p.k_valid = a->k_valid;
  p.lse = a->lse;
  p.o = static_cast<const __nv_bfloat16*>(a->o);
  p.P = static_cast<__nv_bfloat16*>(a->P);
  p.dS = static_cast<__nv_bfloat16*>(a->dS);
  p.cover = a->cover;
  p.reach = reinterpret_cast<unsigned*>(a->cover + (long long)B * p.ptiles);
  p.dq = static_cast<__nv_bfloat16*>(a->dq);
  p.dk = static_cast<__nv_bfloat16*>(a->dk);
  p.dv = static_cast<__nv_bfloat16*>(a->dv);
  p.dk_parts = a->dk_parts; p.dv_parts = a->dv_parts;
  p.status = static_cast<KernelStatus*>(a->status);
  const long long rows = 2ll * p.ptiles * p.kblks * Hkv * B * ST_M;
  if (rows > INT_MAX) return -8;
  const long long jobs = (long long)Hkv * B * (p.ptiles + 2 * p.key_tiles * p.splits);
  const int pairs = (int)(jobs < st_sms() / 2 ? jobs : st_sms() / 2);
  deal_jobs((long long)Hkv * B, p.ptiles, p.kblks, p.key_tiles, p.splits, pairs, &p.dq_more);
  StoredMaps m;
  const long long* t = a->strides;
  int r = st_map(&m.q, a->q, D, H, Sq, B, t[2], t[1], t[0], g, 64 / g);
  if (r) return 1000 + r;
  r = st_map(&m.d_o, a->d_o, D, H, Sq, B, D, (long long)H * D, (long long)Sq * H * D, g, 64 / g);
  if (r) return 2000 + r;
  r = st_map(&m.k, a->k, D, Hkv, Sk, B, t[5], t[4], t[3], 1, 64);
  if (r) return 3000 + r;
  r = st_map(&m.v, a->v, D, Hkv, Sk, B, t[8], t[7], t[6], 1, 64);
  if (r) return 4000 + r;
  r = image_map(&m.p, a->P, rows);
  if (r) return 5000 + r;
  r = image_map(&m.ds, a->dS, rows);
  if (r) return 6000 + r;
  if (D <= 64) return launch_stored<64>(m, p, pairs, stream);
  if (D <= 128) return launch_stored<128>(m, p, pairs, stream);
  return launch_stored<256>(m, p, pairs, stream);
}
