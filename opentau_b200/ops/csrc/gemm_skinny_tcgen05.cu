// Weight-streaming bf16 GEMM for few rows (inference: one decoded token, a 50-token action suffix, a few hundred
// candidate rows) on sm_100a:   out[M,N] = X[M,K] * W[N,K]^T.
//
// What bounds it: a 4 - 17 MB weight matrix is 1 - 3 us of HBM time, so a launch of this kernel is a chain of latencies
// (dependency wait, first load, MMA, cross-CTA reduction, store) and everything below is about keeping that chain short:
//
//   * operands are swapped: the WEIGHT rows are the 128-row M operand of tcgen05.mma, the tokens are the N operand
//     (any multiple of 16 up to 256), so every weight element crosses shared memory once per 256 tokens and the
//     accumulator D^T[128 weight rows, tokens] sits in TMEM with one weight row per lane;
//   * K is split over the CTAs of a thread-block cluster (1 to 8), grid = (N/128, splits, token chunks).  Tokens are
//     dealt to the ranks; every CTA drains its fp32 partial tile into its own shared memory and sends each owner its
//     tokens with ONE bulk copy that completes on the owner's mbarrier, so no cluster barrier stands between the last
//     MMA and the epilogue and the sum reads local shared memory.  (Element-wise remote stores move about 12 bytes a
//     clock: 1.5 us for 50 tokens, measured; remote loads between two cluster barriers were slower still.)  The sum
//     runs in rank order: deterministic, no atomics, no workspace;
//   * the first ring of weight tiles is requested before the dependency wait (weights do not depend on the preceding
//     kernel), so under programmatic dependent launch its HBM latency overlaps the predecessor's tail;
//   * ring depth follows from the shared memory that lets two CTAs share an SM: the next kernel of the chain can then
//     become resident (and prefetch) while this one drains.
//
// Warp roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 TMEM readers and epilogue.  Every
// wait is bounded; a CTA whose wait gave up still sends its peers their (zero) partials and arrives at the barriers.
#include "common.cuh"

namespace otb {

constexpr unsigned KID_SKINNY = 4;
constexpr int SK_BW = 128;  // weight rows per CTA (UMMA M)
constexpr int SK_BK = 64;
constexpr int SK_UMMA_K = 16;
constexpr int SK_THREADS = 320;
constexpr int SK_WORKERS = 256;
constexpr int SK_MAX_STAGES = 12;
constexpr int SK_TAIL = 1024 /* barriers */ + 1024 /* alignment */;

enum SkinnyFlags {  // same values as the big GEMM's epilogue flags
  SK_BIAS = 1,
  SK_RESIDUAL = 2,
  SK_OUT_F32 = 8,
  SK_GLU_GELU = 16,
  SK_GLU_SILU = 32,
  SK_BIAS_F32 = 64,
  SK_NO_OUT = 128,
  SK_ACT_GELU = 256,
  SK_GATE = 512,       // with SK_RESIDUAL: out = residual + gate * result (adaptive-norm gate of the residual branch)
};

struct SkinnyParams {
  int M, N, K;
  void* out;
  long long ldo;
  const void* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  __nv_bfloat16* out2;
  long long ldo2;
  const __nv_bfloat16* gate;      // rows of N gates; row (gate_idx ? gate_idx[m] : m / rows_per_gate), stride gate_stride
  long long gate_stride;
  int rows_per_gate;
  const int* mod_idx;             // per output row: row of `gate` (null: m / rows_per_gate)
  int flags;
  int splits;
  int stages;
  int nt;
  int stage_bytes;
  int tmem_cols;
  int buf_offset;                 // byte offset of the peers' partial tiles
  int bar_offset;
  KernelStatus* status;
};

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// MAXT: tokens per CTA at most (64: two CTAs may share an SM; 256: one).
// EPI >= 0: the epilogue flags are known at compile time (the products of a decoder layer); -1: any flags.
template <int MAXT, int EPI>
__global__ void __launch_bounds__(SK_THREADS, MAXT <= 64 ? 2 : 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                   SkinnyParams p) {
  constexpr int W_BYTES = SK_BW * SK_BK * 2;
  const int NT = p.nt;                               // tokens per CTA, a multiple of 16
  const int STAGE_BYTES = p.stage_bytes;             // weight tile + token tile, rounded up to the swizzle atom
  const int X_LOAD = NT * SK_BK * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.bar_offset);
  uint64_t* empty_bar = full_bar + SK_MAX_STAGES;
  uint64_t* tfull_bar = empty_bar + SK_MAX_STAGES;
  uint64_t* recv_bar = tfull_bar + 1;                // the peers' partials of my tokens have landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // partial tiles, [token][128 weight rows]: mine of all tokens goes over the ring (my MMAs have retired by then), the
  // other ranks' partials of MY tokens into buffers of their own (they may arrive while my MMAs still read the ring)
  float* own_part = reinterpret_cast<float*>(smem);
  float* peer_part = reinterpret_cast<float*>(smem + p.buf_offset);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int S = p.splits;
  const int split = (int)cluster_ctarank();          // the cluster spans gridDim.y == S
  const int n0 = blockIdx.x * SK_BW;
  const int m_base = blockIdx.z * NT;
  const int m_valid = min(NT, p.M - m_base);
  const int tpr = (m_valid + S - 1) / S;             // tokens a rank owns
  const int t0 = split * tpr, own = max(0, min(tpr, m_valid - t0));      // my tokens: [t0, t0 + own)
  const int num_kb = (p.K + SK_BK - 1) / SK_BK;
  const int per = (num_kb + S - 1) / S;
  const int kb0 = split * per;
  const int nkb = max(min(num_kb, kb0 + per) - kb0, 0);
  const int stages = p.stages;
  const int early = min(stages, nkb);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tfull_bar, 1);
    mbar_init(recv_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < early; ++i) {
      mbar_expect_tx(&full_bar[i], W_BYTES + X_LOAD);
      tma_load_2d(smem + i * STAGE_BYTES, &tma_w, &full_bar[i], (kb0 + i) * SK_BK, n0);
    }
    tma_prefetch_desc(&tma_x);
    if (S > 1) mbar_expect_tx(recv_bar, (uint32_t)((S - 1) * own * SK_BW * 4));
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();                 // after the TMEM allocation (see common.cuh)
  if (S > 1) cluster_arrive();             // waited for in front of the first copy to a peer: all have started

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    pdl_wait();
    if (elect_one()) {
      for (int i = 0; i < early; ++i)
        tma_load_2d(smem + i * STAGE_BYTES + W_BYTES, &tma_x, &full_bar[i], (kb0 + i) * SK_BK, m_base);
      int stage = early == stages ? 0 : early;
      uint32_t phase = early == stages ? 1 : 0;
      for (int i = early; i < nkb; ++i) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, KID_SKINNY, 1, stage)) break;
        uint8_t* sw = smem + stage * STAGE_BYTES;
        mbar_expect_tx(&full_bar[stage], W_BYTES + X_LOAD);
        tma_load_2d(sw, &tma_w, &full_bar[stage], (kb0 + i) * SK_BK, n0);
        tma_load_2d(sw + W_BYTES, &tma_x, &full_bar[stage], (kb0 + i) * SK_BK, m_base);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
    if (S > 1) {
      cluster_wait();
      cluster_arrive();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(SK_BW, NT, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, KID_SKINNY, 2, stage)) break;
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * STAGE_BYTES);
        const uint32_t sx = sw + W_BYTES;
#pragma unroll
        for (int k = 0; k < SK_BK / SK_UMMA_K; ++k) {
          uint64_t wd = make_smem_desc(sw + k * 32u, 16u, 1024);
          uint64_t xd = make_smem_desc(sx + k * 32u, 16u, 1024);
          umma_ss(tmem_base, wd, xd, idesc, (i | k) != 0 ? 1u : 0u);
        }
        umma_commit(&empty_bar[stage]);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      umma_commit(tfull_bar);   // fires when every MMA above has retired (at once if there was none)
    }
    __syncwarp();
    if (S > 1) {
      cluster_wait();
      cluster_arrive();
    }
  } else {
    const int ww = warp - 2;
    const int flags = EPI >= 0 ? EPI : p.flags;
    const bool glu = (flags & (SK_GLU_GELU | SK_GLU_SILU)) != 0;
    const int n = n0 + lane * 4;
    uint2 res_v = make_uint2(0u, 0u), gate_v = make_uint2(0u, 0u);
    auto fetch_epi = [&](int t) {
      if (t < own && (flags & SK_RESIDUAL) && n < p.N) {
        const int m = m_base + t0 + t;
        if (flags & SK_GATE)
          gate_v = *reinterpret_cast<const uint2*>(
              p.gate + (long long)(p.mod_idx ? __ldg(p.mod_idx + m) : m / p.rows_per_gate) * p.gate_stride + n);
        res_v = *reinterpret_cast<const uint2*>(p.residual + (long long)m * p.ldr + n);
      }
    };
    float bias_v[4] = {0.f, 0.f, 0.f, 0.f};
    const int quad = warp & 3;                        // TMEM lane quadrant this warp may read
    bool ok = true;
    // Everything from the accumulator to the output runs twice: a launch meets its code in a cold instruction cache (about nine
    // cycles an instruction), so a first pass walks through it in front of the dependency wait, where these warps are idle. It
    // reads tensor and shared memory whatever they hold, nothing of the predecessor's, and stores nothing.
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      asm volatile("" : "+r"(pass));                  // one body for both passes
      const bool live = pass != 0;
      if (live) {
        pdl_wait();                                   // X, residual, gates and outputs belong to the predecessor
        // ---------------------------------------------------------------- epilogue operands of my first token
        fetch_epi(ww);
        if ((flags & SK_BIAS) && n < p.N) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            bias_v[e] = (flags & SK_BIAS_F32) ? __ldg(static_cast<const float*>(p.bias) + n + e)
                                              : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[n + e]);
        }
        if (S > 1) cluster_wait();                    // all have started: their buffers are there before the first copy
        ok = mbar_wait(tfull_bar, 0, abort_flag, p.status, KID_SKINNY, 3, 0);
        tc_fence_after();
      }
      // ------------------------------------------------------------------ TMEM -> my partial tile -> the tokens' owners
      {
        const uint32_t taddr = tmem_base + (uint32_t(quad * 32) << 16);
        float* col = own_part + quad * 32 + lane;     // weight row inside the tile
        constexpr int CHUNK = MAXT > 64 ? 32 : 16;    // a chunk's tail past the last token is never looked at
        const bool have = nkb > 0 && ok;              // a split without k-blocks (or one that gave up) sends zeros
        const int c_end = live ? m_valid : 1;
#pragma unroll 1
        for (int c0 = live ? (ww >> 2) * CHUNK : 0; c0 < c_end; c0 += 2 * CHUNK) {
          uint32_t r[32];
          __syncwarp();
          if (CHUNK == 32) tmem_ld_x32(taddr + c0, r); else tmem_ld_x16(taddr + c0, r);
          tmem_wait_ld();
          if (!have) {
#pragma unroll
            for (int j = 0; j < CHUNK; ++j) r[j] = 0u;
          }
          float* dst = col + c0 * SK_BW;
#pragma unroll
          for (int j = 0; j < CHUNK; ++j)
            if (live) dst[j * SK_BW] = __uint_as_float(r[j]);
        }
      }
      if (live) {
        tc_fence_before();
        if (S > 1) fence_async_smem();                // the bulk copies read what the workers have just written
        workers_sync();
        if (S > 1) {
          const int owner = ww;                       // a warp sends to one peer: a lane after the other would take 0.3 us
          if (lane == 0 && owner < S && owner != split) {
            const int cnt = min(tpr, m_valid - owner * tpr);
            if (cnt > 0)
              bulk_to_peer(map_rank(smem_u32(peer_part) + (uint32_t)(split < owner ? split : split - 1) * (uint32_t)tpr * (SK_BW * 4u),
                                    (uint32_t)owner),
                           smem_u32(own_part) + (uint32_t)(owner * tpr) * (SK_BW * 4u), (uint32_t)cnt * (SK_BW * 4u),
                           map_rank(smem_u32(recv_bar), (uint32_t)owner));
          }
          __syncwarp();
          if (own > 0) mbar_wait(recv_bar, 0, abort_flag, p.status, KID_SKINNY, 5, 0);
          __syncwarp();
          cluster_arrive();                           // my tokens have all arrived; waited for before leaving
        }
      }
      // ------------------------------------------------------------------ reduction + epilogue of my tokens
      const int t_end = live ? (*abort_flag ? 0 : own) : 1;
#pragma unroll 1
      for (int t = live ? ww : 0; t < t_end; t += SK_WORKERS / 32) {
        const int m = m_base + t0 + t;
        const uint2 rv = res_v, gv = gate_v;
        if (live) fetch_epi(t + SK_WORKERS / 32);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int s0 = 0; s0 < S; s0 += 4) {           // four partials in flight, added in rank order
          float4 u[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int s = s0 + i;
            const float* part = s == split ? own_part + t0 * SK_BW : peer_part + (s < split ? s : s - 1) * tpr * SK_BW;
            if (s < S) u[i] = reinterpret_cast<const float4*>(part + t * SK_BW)[lane];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (s0 + i < S) {
              v.x += u[i].x;
              v.y += u[i].y;
              v.z += u[i].z;
              v.w += u[i].w;
            }
          }
        }
        const float f[4] = {v.x, v.y, v.z, v.w};
        if (!(flags & SK_NO_OUT)) {
          if (n < p.N) {
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = f[e] + bias_v[e];
            if (flags & SK_ACT_GELU) {
#pragma unroll
              for (int e = 0; e < 4; ++e) o[e] = gelu_tanh_f(o[e]);
            }
            if (flags & SK_RESIDUAL) {
              if (flags & SK_GATE) {
                const float2 g0 = unpack_bf16(gv.x), g1 = unpack_bf16(gv.y);
                o[0] *= g0.x; o[1] *= g0.y; o[2] *= g1.x; o[3] *= g1.y;
              }
              const float2 q0 = unpack_bf16(rv.x), q1 = unpack_bf16(rv.y);
              o[0] += q0.x; o[1] += q0.y; o[2] += q1.x; o[3] += q1.y;
            }
            if (flags & SK_OUT_F32) {
              if (live)
                *reinterpret_cast<float4*>(static_cast<float*>(p.out) + (long long)m * p.ldo + n) =
                    make_float4(o[0], o[1], o[2], o[3]);
            } else {
              if (live)
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + (long long)m * p.ldo + n) =
                    make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
            }
          }
        }
        if (glu) {
          // rows come in blocks of 32: [gate | up | gate | up]; a gate lane takes its up values from 8 lanes further
          float o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // match the unfused path: gate / up are rounded to bf16 before the activation
            const float up = __bfloat162float(__float2bfloat16(__shfl_down_sync(0xffffffffu, f[e], 8)));
            const float g = __bfloat162float(__float2bfloat16(f[e]));
            o[e] = ((flags & SK_GLU_GELU) ? gelu_tanh_f(g) : silu_f(g)) * up;
          }
          if (live && !(lane & 8) && n < p.N)
            *reinterpret_cast<uint2*>(p.out2 + (long long)m * p.ldo2 + (n0 >> 1) + (lane >> 4) * 32 + (lane & 7) * 4) =
                make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
        }
      }
    }
  }

  // ---------------------------------------------------------------------- teardown
  __syncthreads();
  if (S > 1) cluster_wait();                         // every copy out of my shared memory has arrived at its owner
  if (warp == 1) {
    if (*abort_flag) {
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let TMA copies / MMAs in flight finish
    }
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

static int g_sk_sms = 0;

// Clusters of `n` CTAs that are resident at once with one CTA to an SM (a GPC's SMs do not divide by every size: 15 of eight
// on a B200, not 18).  Token tiles of at most 64 put two to an SM, which the query does not count.
static int resident_clusters(int n) {
  static int cap[9] = {};                            // -1: none
  int& c = cap[n];
  if (c == 0) {
    auto kern = gemm_skinny_kernel<256, -1>;
    int got = 0;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(1, (unsigned)n, 1);
    cfg.blockDim = dim3(SK_THREADS);
    cfg.dynamicSmemBytes = 224 * 1024;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1;
    attr.val.clusterDim.y = (unsigned)n;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&got, kern, &cfg) != cudaSuccess)
      got = 0;
    c = got > 0 ? got : -1;
  }
  return c > 0 ? c : 0;
}

// How a product is dealt out: token chunks of `nt` (a multiple of the MMA's 16) and the CTAs that share a sum over K.
struct SkinnyPlan {
  int chunks, nt, splits, stages;
  int stage_bytes, ring, buf_bytes;    // shared memory: a stage; ring or my partial tile, whichever is larger; the peers' partials
};

// Fills in chunks, token tile and shared memory for `chunks` and `splits`; false where they do not fit.  The ring is as deep as
// the CTA's k-blocks need or the budget gives (my own partial overlays it), the peers' partials lie behind it, then barriers.
// 111 KB keeps two CTAs on an SM while there are at most 64 tokens; wider tiles take the SM alone.
static bool layout_plan(int M, int K, int chunks, int splits, SkinnyPlan* p) {
  const int nt = ((M + chunks - 1) / chunks + 15) / 16 * 16;
  const int num_kb = (K + SK_BK - 1) / SK_BK, per = (num_kb + splits - 1) / splits;
  p->chunks = (M + nt - 1) / nt;
  p->nt = nt;
  p->splits = splits;
  p->stage_bytes = (SK_BW * SK_BK * 2 + nt * SK_BK * 2 + 1023) / 1024 * 1024;
  const int tile_bytes = (nt <= 64 ? nt : (nt + 31) / 32 * 32) * SK_BW * 4;
  p->buf_bytes = (nt + splits - 1) / splits * SK_BW * 4 * (splits - 1);
  const int room = (nt > 64 ? 224 : 111) * 1024 - SK_TAIL - p->buf_bytes;
  int stages = room / p->stage_bytes;
  if (stages > per) stages = per;
  if (stages > SK_MAX_STAGES) stages = SK_MAX_STAGES;
  p->stages = stages;
  p->ring = stages * p->stage_bytes > tile_bytes ? stages * p->stage_bytes : tile_bytes;
  return nt <= 256 && stages >= 1 && tile_bytes <= room;
}

// The plan of an M x N x K product on `sms` SMs; clusters(n): clusters of n CTAs resident at once, one CTA to an SM.
//
// Up to 64 rows: one token tile, and the largest cluster size whose grid is resident at once and leaves every CTA two k-blocks;
// going beyond ONE CTA per SM only pays while each CTA still streams four k-blocks (a launch of two-k-block CTAs that fills every
// SM twice keeps the next kernel of the chain from becoming resident early).
//
// More rows: of the token tiles from 32 to 256 and 1 to 8 CTAs to a sum, the cheapest that is resident at once.  A CTA
// pays for its k-blocks, for every round of the ring behind the first, for the partials it sends, for its own tokens' epilogue,
// and the launch for its CTAs: microseconds fitted to 3400 resident plans at 65 - 640 rows, 128 - 2048 columns, K 256 - 8192 inside a
// replayed graph with cold weights (rms error 6 %; the plan taken costs 1.5 % more than the best one in the mean, 10 % at most; where
// rows of K are no multiple of 128 bytes, reading the weights once per chunk costs up to a tenth that this does not charge).
// The weights are read once per chunk, from L2.  With the norm behind them, us, against one tile of up to 256 rows and
// against chunks of 64 that two to four CTAs share (what ran before): 100 x 1024 x 4096 9.4 / 11.2 -> 8.7, 200 x 1024 x 4096 14.8 /
// 12.2 -> 9.5, 256 x 1280 x 5120 31.8 / 16.5 -> 13.0, 200 x 128 x 256 13.8 / 13.8 -> 4.7.
template <typename F>
static bool choose_plan(int M, int N, int K, int sms, F clusters, SkinnyPlan* best) {
  const int n_tiles = (N + SK_BW - 1) / SK_BW, num_kb = (K + SK_BK - 1) / SK_BK;
  const int one = (M + 255) / 256;
  if (M <= 64) {
    int splits = 1;
    for (int s = 2; s <= 8; ++s) {
      const long long ctas = (long long)n_tiles * s;
      if (ctas <= 2LL * sms && num_kb / s >= 2 && (ctas <= sms || num_kb / s >= 4)) splits = s;
    }
    return layout_plan(M, K, one, splits, best);
  }
  bool found = false;
  double best_cost = 0.0;
  for (int nt = 256, last = 0; nt >= 32; nt -= 16) {
    const int chunks = (M + nt - 1) / nt;
    if (chunks == last) continue;
    last = chunks;
    for (int s = 1; s <= 8; ++s) {
      SkinnyPlan c;
      const int per = (num_kb + s - 1) / s;
      if ((s - 1) * per >= num_kb || !layout_plan(M, K, chunks, s, &c)) continue;
      const long long units = (long long)n_tiles * c.chunks;
      // the last places do not fill: 26 clusters of five of 80 tokens, or 90 of three of 48, took a second round
      if (units > (c.nt <= 64 ? 2LL * clusters(s) - 2 : clusters(s) - (s > 2 ? 1LL : 0LL))) continue;
      const double cost = per * (0.05 + 0.0004 * c.nt) + 0.8 * (per > c.stages ? (double)(per - c.stages) / c.stages : 0.0) +
                          0.03 * c.nt * (s - 1) / s + 0.075 * ((c.nt + s - 1) / s) + 1.25 * (double)(units * s) / sms;
      if (!found || cost < best_cost) {
        found = true;
        best_cost = cost;
        *best = c;
      }
    }
  }
  // more CTAs than the chip holds whatever the tile: the widest tiles
  return found || layout_plan(M, K, one, 1, best);
}

template <int MAXT, int EPI>
static int launch_skinny_epi(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int n_tiles, int chunks,
                         int smem_bytes, cudaStream_t stream) {
  static bool configured = false;
  auto kern = gemm_skinny_kernel<MAXT, EPI>;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  cudaError_t e = launch_pdl(kern, dim3((unsigned)n_tiles, (unsigned)p.splits, (unsigned)chunks),
                             dim3(SK_THREADS, 1, 1), (size_t)smem_bytes, stream, (unsigned)p.splits, tw, tx, p);
  return (int)e;
}

// A launch runs its code once, from a cold instruction cache: at about nine cycles an instruction, code that is only
// branched over costs as much as the loads it hides.  The flag sets of the decoder layers get code of their own.
template <int MAXT>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int n_tiles, int chunks,
                         int smem_bytes, cudaStream_t stream) {
  switch (p.flags) {
    case 0: return launch_skinny_epi<MAXT, 0>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
    case SK_RESIDUAL: return launch_skinny_epi<MAXT, SK_RESIDUAL>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
    case SK_RESIDUAL | SK_GATE:
      return launch_skinny_epi<MAXT, SK_RESIDUAL | SK_GATE>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
    case SK_NO_OUT | SK_GLU_GELU:
      return launch_skinny_epi<MAXT, SK_NO_OUT | SK_GLU_GELU>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
    default: return launch_skinny_epi<MAXT, -1>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
  }
}

}  // namespace otb

using namespace otb;

// Arguments of one launch (mirrored field by field by the ctypes structure of the Python launcher).
struct OtbSkinnyArgs {
  const void* x;
  const void* w;
  void* out;
  const void* bias;
  const void* residual;
  void* out2;
  const void* gate;
  const int* mod_idx;
  void* status;
  long long ldx, ldw, ldo, ldr, ldo2, gate_stride;
  int M, N, K;
  int rows_per_gate, flags, splits;
};

// The plan that a launch with `splits` 0 takes, for `sms` SMs that hold clusters[n] clusters of n CTAs (null: of this device).
// plan: token chunks, tokens per CTA, CTAs to a sum, stages of the ring, bytes of shared memory.
extern "C" int otb_gemm_skinny_plan(int M, int N, int K, int sms, const int* clusters, int* plan) {
  if (M <= 0 || N <= 0 || K <= 0 || sms <= 0) return -2;
  SkinnyPlan p;
  if (!choose_plan(M, N, K, sms, [&](int n) { return clusters != nullptr ? clusters[n] : resident_clusters(n); }, &p)) return -13;
  plan[0] = p.chunks;
  plan[1] = p.nt;
  plan[2] = p.splits;
  plan[3] = p.stages;
  plan[4] = p.ring + p.buf_bytes + SK_TAIL;
  return 0;
}

// out[M,N] = X[M,K] W[N,K]^T (+ epilogue).  Returns 0, a CUDA / driver error code, or a negative argument-check
// code.  `splits`: 0 = choose (choose_plan).
extern "C" int otb_gemm_skinny_bf16(const OtbSkinnyArgs* a, cudaStream_t stream) {
  const int M = a->M, N = a->N, K = a->K, flags = a->flags;
  if (M <= 0 || N <= 0 || K <= 0 || (N % 8)) return -2;
  if ((a->ldx % 8) || (a->ldw % 8)) return -3;
  if ((reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->w)) & 15) return -4;
  if (flags & 4) return -9;                                  // accumulate-into-output is the big GEMM's job
  if ((flags & SK_RESIDUAL) && ((a->ldr % 4) || (reinterpret_cast<uintptr_t>(a->residual) & 7))) return -11;
  if ((flags & SK_GATE) && (!(flags & SK_RESIDUAL) || a->gate == nullptr || (a->gate_stride % 4) ||
                            (reinterpret_cast<uintptr_t>(a->gate) & 7)))
    return -10;
  if (a->rows_per_gate < 1) return -10;
  const bool glu = (flags & (SK_GLU_GELU | SK_GLU_SILU)) != 0;
  if (glu && ((N % 64) || a->out2 == nullptr || (a->ldo2 % 4) || (reinterpret_cast<uintptr_t>(a->out2) & 7))) return -6;
  if (!(flags & SK_NO_OUT) &&
      (a->out == nullptr || (a->ldo % 4) || (reinterpret_cast<uintptr_t>(a->out) & ((flags & SK_OUT_F32) ? 15 : 7))))
    return -6;
  if (g_sk_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sk_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sk_sms <= 0) return -7;
  }
  SkinnyPlan plan;
  if (a->splits < 0 || a->splits > 8) return -8;
  bool ok;
  if (a->splits == 0) {
    ok = choose_plan(M, N, K, g_sk_sms, resident_clusters, &plan);
  } else {
    // a forced split: as few chunks of at most 256 as cover M, narrower where the partials do not fit side by side
    ok = layout_plan(M, K, (M + 255) / 256, a->splits, &plan) || layout_plan(M, K, (M + 127) / 128, a->splits, &plan);
  }
  if (!ok) return -13;
  const int n_tiles = (N + SK_BW - 1) / SK_BW;
  const int chunks = plan.chunks, nt = plan.nt, splits = plan.splits;
  SkinnyParams p;
  p.buf_offset = plan.ring;
  p.bar_offset = plan.ring + plan.buf_bytes;
  const int smem_bytes = p.bar_offset + SK_TAIL;
  CUtensorMap tw, tx;
  {
    uint64_t dims[2], strides[1];
    uint32_t box[2];
    dims[0] = (uint64_t)K; dims[1] = (uint64_t)N; box[0] = 64; box[1] = SK_BW;
    strides[0] = (uint64_t)a->ldw * 2;
    int r = make_tmap_bf16(&tw, a->w, 2, dims, strides, box);
    if (r) return 1000 + r;
    dims[0] = (uint64_t)K; dims[1] = (uint64_t)M; box[0] = 64; box[1] = (uint32_t)nt;
    strides[0] = (uint64_t)a->ldx * 2;
    r = make_tmap_bf16(&tx, a->x, 2, dims, strides, box);
    if (r) return 2000 + r;
  }
  p.M = M; p.N = N; p.K = K;
  p.out = a->out; p.ldo = a->ldo;
  p.bias = a->bias;
  p.residual = static_cast<const __nv_bfloat16*>(a->residual); p.ldr = a->ldr;
  p.out2 = static_cast<__nv_bfloat16*>(a->out2); p.ldo2 = a->ldo2;
  p.gate = static_cast<const __nv_bfloat16*>(a->gate); p.gate_stride = a->gate_stride;
  p.rows_per_gate = a->rows_per_gate;
  p.mod_idx = a->mod_idx;
  p.flags = flags;
  p.splits = splits;
  p.stages = plan.stages;
  p.nt = nt;
  p.stage_bytes = plan.stage_bytes;
  p.tmem_cols = nt <= 32 ? 32 : (nt <= 64 ? 64 : (nt <= 128 ? 128 : 256));
  p.status = static_cast<KernelStatus*>(a->status);
  if (nt <= 64) return launch_skinny<64>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
  return launch_skinny<256>(tw, tx, p, n_tiles, chunks, smem_bytes, stream);
}
