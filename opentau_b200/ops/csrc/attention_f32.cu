// Exact fp32 block-causal attention, forward and backward, on the CUDA cores (no tensor-core rounding): the path that
// fp32 policies and fp32 validation runs take.
//
// What bounds it: fp32 multiply-adds against shared-memory reads.  A 128-bit shared load takes four cycles of the SM
// whatever it broadcasts, a multiply-add one cycle of one of its four schedulers, so a register tile of a x b outputs
// runs at most a * b / (4 (a + b)) of the arithmetic peak: 8 x 8 tiles throughout (one owner row times one streamed row
// per lane, as an earlier version had it, stops at a fifth of the peak).
//
// Decomposition (all kernels): a 256-thread block owns 32 rows -- query rows of one head (forward, dQ) or keys of one
// kv head (dK / dV) -- and streams tiles of 64 rows of the other side through shared memory with asynchronous copies.
//   inner products   a warp computes a 32 x 16 (backward) or 32 x 8 (forward) piece of the 32 x 64 product in 8 x 8 register
//                    tiles; its lanes split the head width four (eight) ways and add their tiles by shuffles, halving
//                    what a lane keeps at every exchange, so that a tile that is small against 256 threads still
//                    gives every lane an 8 x 8.  The two products of the backward take four warps each.
//   accumulation     a lane owns 8 owner rows x 4 (8) columns; the two groups of four warps take halves of the streamed
//                    rows (forward, dQ; their sums are added at the end) or one of dK / dV each.
// Rows are Dp + 4 floats apart (Dp: head width rounded up to 16, zero-filled): any eight lanes of a 128-bit access fall
// into different bank groups.  One block per SM (170 - 218 KB at head width 256; the forward up to width 128 has two: 731
// -> 669 us for 2 x 700 positions, 32 heads of 128, where the backward's spills lose more than that wins), so loads hide behind arithmetic of the
// same block: the next K behind softmax and accumulation, V behind the scores, the next V of dQ behind its accumulation.
//
// dS that the dK / dV kernel has at hand is kept where it fits (fp32 scratch, a row per key), and dQ is then one
// product of it instead of three (forward + backward of 2 x 601 positions, 8 heads on 1 of width 256: 984 -> 800 us);
// longer sequences recompute it.
//
// Sums over the streamed rows of dQ and dK / dV may be dealt to several blocks (`splits`), whose partial sums one more
// kernel adds in a fixed order: with one kv head, 38 key blocks would leave three quarters of the chip idle.
//
//   forward : online softmax; writes O (B,Sq,H*D) and the natural-log LSE (B,H,Sq); a row that sees no key gets
//             O = 0 and LSE = 0, one with a NaN among its visible scores NaN in both, as the dense evaluation does
//   dQ      : P is recomputed from LSE; dS = P * (dP - delta) * scale; dQ += dS K
//   dK / dV : the heads of the GQA group are one stream, so the sum over the group happens in registers (no atomics)
//   delta   : rowsum(O * dO), one warp per row
//
// Visibility of (query i, key j): q_valid[i] && k_valid[j] && k_blk[j] <= q_blk[i].  A streamed tile none of whose rows
// sees (or is seen by) any owner row is skipped; single rows of that kind are read as zeros.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>

namespace otb {

constexpr int F32_OWN = 32;       // owner rows per block
constexpr int F32_STR = 64;       // streamed rows per tile
constexpr int F32_THREADS = 256;
constexpr int F32_PLD = F32_STR + 4;
constexpr int F32_MAX_SPLITS = 8;
constexpr long long F32_MAX_SCRATCH = 256ll << 20;      // bytes of one output's parts
// Bytes of dS.  The dense evaluation holds five tensors of that size; without it the backward computes seven products
// instead of five (forward + backward with nothing hidden: 8 x 1227 positions, 8 heads on 1 of 256, 15.9 ms against 12.5;
// 16 x 601, 16 heads of 72, 8.1 against 6.2).
constexpr long long F32_MAX_DS = 2ll << 30;

struct F32Params {
  const float* q;
  const float* k;
  const float* v;
  long long q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh;
  const int* q_blk;
  const int* k_blk;
  const unsigned char* q_valid;
  const unsigned char* k_valid;
  int B, Sq, Sk, H, Hkv, D;
  float scale;
};

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// The larger of two numbers, NaN if either is (fmaxf would drop it).
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool read) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(read ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ROWS rows from `src` on (row stride rs) into a shared tile (row stride ld); row r is read if bit r of `rows` is set and
// zero-filled otherwise.  128-bit copies: D is a multiple of 4, bases and strides are 16-byte aligned.
template <int ROWS>
__device__ __forceinline__ void load_rows(float* dst, const float* src, long long rs, unsigned long long rows, int D,
                                          int ld) {
  const int vec = D >> 2;
  for (int i = threadIdx.x; i < ROWS * vec; i += F32_THREADS) {
    const int r = i / vec, c = (i - r * vec) << 2;
    const bool read = (rows >> r) & 1ull;
    cp_async16(dst + r * ld + c, read ? src + r * rs + c : src, read);
  }
}

__device__ __forceinline__ void fma4(float& a, const float4& x, const float4& y) {
  a = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, a))));
}

// One exchange of the lane-split inner products: lanes that differ in bit MASK hold partial sums of the same n values; each
// keeps one half (the upper one if its bit is set) and adds the other lane's part of it.
template <int N, int MASK>
__device__ __forceinline__ void halve(float (&a)[N], int lane) {
  const bool up = (lane & MASK) != 0;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float send = up ? a[i] : a[i + N / 2];
    const float keep = up ? a[i + N / 2] : a[i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
  }
}

// out[32][64] (row stride F32_PLD) = own . str^T by four warps (wg: 0..3), a 32 x 16 piece each; lanes split the width
// four ways.
__device__ __forceinline__ void product_by_4_warps(const float* own, const float* str, float* out, int Dp, int ld, int wg,
                                                   int lane) {
  const int q = lane & 3, ty = (lane >> 2) & 3, tx = lane >> 4;
  const float* po = own + (4 * ty) * ld + 4 * q;
  const float* ps = str + (16 * wg + 4 * tx) * ld + 4 * q;
  float acc[64];                                   // [i][j], i: owner row 4 ty + (i & 3) + 16 (i >> 2)
#pragma unroll
  for (int i = 0; i < 64; ++i) acc[i] = 0.f;
  for (int c = 0; c < Dp; c += 16) {
    float4 y[8];                                   // j: streamed row 16 wg + 4 tx + (j & 3) + 8 (j >> 2)
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = *reinterpret_cast<const float4*>(ps + ((j & 3) + 8 * (j >> 2)) * ld + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(po + ((i & 3) + 16 * (i >> 2)) * ld + c);
#pragma unroll
      for (int j = 0; j < 8; ++j) fma4(acc[i * 8 + j], x, y[j]);
    }
  }
  halve<64, 1>(acc, lane);                         // bit 0: i >> 2
  float h[32];
#pragma unroll
  for (int i = 0; i < 4; ++i)                      // j halves to the front: [j >> 2][i][j & 3]
#pragma unroll
    for (int j = 0; j < 8; ++j) h[(j >> 2) * 16 + i * 4 + (j & 3)] = acc[i * 8 + j];
  halve<32, 2>(h, lane);                           // bit 1: j >> 2
  float* po_ = out + (4 * ty + 16 * (lane & 1)) * F32_PLD + 16 * wg + 4 * tx + 8 * ((lane >> 1) & 1);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(po_ + i * F32_PLD) = make_float4(h[i * 4], h[i * 4 + 1], h[i * 4 + 2], h[i * 4 + 3]);
}

// The same product by eight warps (w: 0..7), a 32 x 8 piece each; lanes split the width eight ways.
__device__ __forceinline__ void product_by_8_warps(const float* own, const float* str, float* out, int Dp, int ld, int w,
                                                   int lane) {
  const int q = lane & 7, ty = lane >> 3;
  const float* po = own + (8 * ty) * ld + 4 * q;
  const float* ps = str + (8 * w) * ld + 4 * q;
  float acc[64];                                   // [i][j]: owner row 8 ty + i, streamed row 8 w + j
#pragma unroll
  for (int i = 0; i < 64; ++i) acc[i] = 0.f;
  for (int c = 0; c < Dp; c += 32) {
    if (c + 4 * q >= Dp) break;                    // the width is a multiple of 16: half the lanes may end earlier
    float4 y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = *reinterpret_cast<const float4*>(ps + j * ld + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(po + i * ld + c);
#pragma unroll
      for (int j = 0; j < 8; ++j) fma4(acc[i * 8 + j], x, y[j]);
    }
  }
  __syncwarp();
  halve<64, 1>(acc, lane);                         // bit 0: i >> 2
  float h[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) h[i] = acc[i];
  halve<32, 2>(h, lane);                           // bit 1: (i >> 1) & 1
  float g[16];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) g[(j >> 2) * 8 + i * 4 + (j & 3)] = h[i * 8 + j];
  halve<16, 4>(g, lane);                           // bit 2: j >> 2
  float* po_ = out + (8 * ty + 4 * (lane & 1) + 2 * ((lane >> 1) & 1)) * F32_PLD + 8 * w + 4 * ((lane >> 2) & 1);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    *reinterpret_cast<float4*>(po_ + i * F32_PLD) = make_float4(g[i * 4], g[i * 4 + 1], g[i * 4 + 2], g[i * 4 + 3]);
}

// acc[8 rows][G x 4 columns] += P[8 rows][j0 .. j1) * X[j0 .. j1)[columns]: `pr` the first of the eight rows, `xc` the
// lane's first column; the second group of columns is 128 further.
template <int G>
__device__ __forceinline__ void accumulate(float (&acc)[8][4 * G], const float* pr, const float* xc, int ld, int j0, int j1) {
  for (int j = j0; j < j1; j += 4) {
    float4 pv[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) pv[r] = *reinterpret_cast<const float4*>(pr + r * F32_PLD + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 x = *reinterpret_cast<const float4*>(xc + (j + jj) * ld + 128 * g);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float pw = jj == 0 ? pv[r].x : jj == 1 ? pv[r].y : jj == 2 ? pv[r].z : pv[r].w;
          acc[r][4 * g + 0] = fmaf(pw, x.x, acc[r][4 * g + 0]);
          acc[r][4 * g + 1] = fmaf(pw, x.y, acc[r][4 * g + 1]);
          acc[r][4 * g + 2] = fmaf(pw, x.z, acc[r][4 * g + 2]);
          acc[r][4 * g + 3] = fmaf(pw, x.w, acc[r][4 * g + 3]);
        }
      }
    }
  }
}

// Owner rows of a block as every warp sees them: which of its 32 rows are valid, and the extreme block id among those.
struct Owners {
  unsigned ok;
  int bound;
};
__device__ __forceinline__ Owners owner_rows(const unsigned char* valid, const int* blk, int r0, int n, int lane, bool want_max) {
  const bool ok = r0 + lane < n && valid[r0 + lane] != 0;
  int v = ok ? blk[r0 + lane] : (want_max ? INT_MIN : INT_MAX);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int u = __shfl_xor_sync(0xffffffffu, v, o);
    v = want_max ? max(v, u) : min(v, u);
  }
  Owners r;
  r.ok = __ballot_sync(0xffffffffu, ok);
  r.bound = v;
  return r;
}

// Bit r: row r0 + r of the streamed side can meet an owner row (keys: block id at most the owners' largest; queries: at
// least the owners' smallest).  The same in every warp.
__device__ __forceinline__ unsigned long long tile_rows(const unsigned char* valid, const int* blk, int r0, int n, int lane,
                                                        const Owners& own, bool keys) {
  unsigned long long m = 0;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = r0 + 32 * half + lane;
    bool ok = r < n && valid[r] != 0;
    if (ok) ok = keys ? blk[r] <= own.bound : blk[r] >= own.bound;
    m |= (unsigned long long)__ballot_sync(0xffffffffu, ok) << (32 * half);
  }
  return own.ok ? m : 0ull;
}

// zero-fills the columns [D, Dp) of `rows` consecutive tile rows (read by the inner products, never loaded)
__device__ __forceinline__ void clear_tail(float* tile, int rows, int D, int Dp, int ld) {
  const int t = Dp - D;
  for (int i = threadIdx.x; i < rows * t; i += F32_THREADS) tile[(i / t) * ld + D + i % t] = 0.f;
}

// ---------------------------------------------------------------------------------------------------------- forward
template <int G>  // groups of 128 head-dim columns
__global__ void __launch_bounds__(F32_THREADS, G == 1 ? 2 : 1) attn_f32_fwd_kernel(F32Params p, float* __restrict__ o,
                                                                      float* __restrict__ lse) {
  extern __shared__ __align__(16) float smem[];
  const int D = p.D, Dp = (D + 15) & ~15, ld = Dp + 4;
  float* sQ = smem;                         // [32][ld]
  float* sK = sQ + F32_OWN * ld;            // [64][ld]
  float* sV = sK + F32_STR * ld;            // [64][ld]
  float* sP = sV + F32_STR * ld;            // [32][F32_PLD] scores, then probabilities
  float* sC = sP + F32_OWN * F32_PLD;       // [32] rescale factors
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = blockIdx.x * F32_OWN, h = blockIdx.y, b = blockIdx.z;
  const int kvh = h / (p.H / p.Hkv);
  const float* kb = p.k + (long long)b * p.k_sb + (long long)kvh * p.k_sh;
  const float* vb = p.v + (long long)b * p.v_sb + (long long)kvh * p.v_sh;
  const unsigned char* kval = p.k_valid + (long long)b * p.Sk;
  const int* kblk = p.k_blk + (long long)b * p.Sk;
  const Owners own = owner_rows(p.q_valid + (long long)b * p.Sq, p.q_blk + (long long)b * p.Sq, q0, p.Sq, lane, true);
  const auto next_tile = [&](int k0, unsigned long long& rows) {
    for (; k0 < p.Sk; k0 += F32_STR) {
      rows = tile_rows(kval, kblk, k0, p.Sk, lane, own, true);
      if (rows) break;
    }
    return k0;
  };
  if (Dp != D) clear_tail(sQ, F32_OWN + 2 * F32_STR, D, Dp, ld);
  unsigned long long rows = 0;
  int k0 = next_tile(0, rows);
  {
    const int n = min(F32_OWN, p.Sq - q0);
    load_rows<F32_OWN>(sQ, p.q + (long long)b * p.q_sb + (long long)h * p.q_sh + (long long)q0 * p.q_ss, p.q_ss,
                       n >= 32 ? 0xffffffffull : (1ull << n) - 1, D, ld);
    if (k0 < p.Sk) load_rows<F32_STR>(sK, kb + (long long)k0 * p.k_ss, p.k_ss, rows, D, ld);
    cp_async_commit();
  }
  // softmax: eight threads per row, thread part x columns 4 part .. and 32 + 4 part ..
  const int row = threadIdx.x >> 3, part = threadIdx.x & 7;
  const bool row_ok = (own.ok >> row) & 1;
  const int row_blk = row_ok ? p.q_blk[(long long)b * p.Sq + q0 + row] : INT_MIN;
  float m = -INFINITY, l = 0.f;
  unsigned seen = 0;                                 // visible keys met so far by this thread
  const int grp = warp >> 2, r0 = 8 * (warp & 3), col = lane * 4 < Dp ? lane * 4 : 0;
  float acc[8][4 * G];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4 * G; ++c) acc[r][c] = 0.f;

  while (k0 < p.Sk) {
    load_rows<F32_STR>(sV, vb + (long long)k0 * p.v_ss, p.v_ss, rows, D, ld);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();                                 // Q and K are here
    product_by_8_warps(sQ, sK, sP, Dp, ld, warp, lane);
    __syncthreads();                                 // scores complete, K free
    const unsigned long long cur = rows;
    const int cur0 = k0;
    k0 = next_tile(k0 + F32_STR, rows);
    if (k0 < p.Sk) load_rows<F32_STR>(sK, kb + (long long)k0 * p.k_ss, p.k_ss, rows, D, ld);
    cp_async_commit();
    {
      float* sr = sP + row * F32_PLD + 4 * part;
      float s[8];
      *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(sr);
      *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(sr + 32);
      unsigned vis = 0;
      float mt = -INFINITY;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int j = 4 * part + (e & 3) + 32 * (e >> 2);
        if (row_ok && ((cur >> j) & 1ull) && kblk[cur0 + j] <= row_blk) {
          vis |= 1u << e;
          s[e] *= p.scale;
          mt = max_nan(mt, s[e]);
        }
      }
      seen |= vis;
#pragma unroll
      for (int x = 4; x > 0; x >>= 1) mt = max_nan(mt, __shfl_xor_sync(0xffffffffu, mt, x));
      const float mn = max_nan(m, mt);
      float corr = 1.f, sum = 0.f;
      if (mn != -INFINITY) corr = m == -INFINITY ? 0.f : expf(m - mn);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        s[e] = (vis >> e) & 1 && mn != -INFINITY ? expf(s[e] - mn) : 0.f;
        sum += s[e];
      }
#pragma unroll
      for (int x = 4; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      l = l * corr + sum;
      m = mn;
      *reinterpret_cast<float4*>(sr) = *reinterpret_cast<const float4*>(s);
      *reinterpret_cast<float4*>(sr + 32) = *reinterpret_cast<const float4*>(s + 4);
      if (part == 0) sC[row] = corr;
    }
    cp_async_wait<1>();
    __syncthreads();                                 // probabilities, factors and V are here
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float corr = sC[r0 + r];
#pragma unroll
      for (int c = 0; c < 4 * G; ++c) acc[r][c] *= corr;
    }
    accumulate<G>(acc, sP + r0 * F32_PLD, sV + col, ld, 32 * grp, 32 * grp + 32);
    __syncthreads();                                 // V, probabilities and factors free
  }
  cp_async_wait<0>();
  __syncthreads();
  // the second group's sums go through shared memory (over K); 1 / l through the factors
#pragma unroll
  for (int x = 4; x > 0; x >>= 1) seen |= __shfl_xor_sync(0xffffffffu, seen, x);
  if (part == 0) {
    // a maximum that is no finite number is the LSE, and no probability is one: 1 / l is NaN (of l = 0: all scores -inf)
    const bool finite = fabsf(m) < INFINITY;
    sC[row] = !seen ? 0.f : finite ? 1.f / l : NAN;
    if (q0 + row < p.Sq) lse[((long long)b * p.H + h) * p.Sq + q0 + row] = !seen ? 0.f : finite ? m + logf(l) : m;
  }
  if (grp == 1 && lane * 4 < Dp) {
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (lane * 4 + 128 * g < Dp)
          *reinterpret_cast<float4*>(sK + (r0 + r) * ld + col + 128 * g) = *reinterpret_cast<const float4*>(&acc[r][4 * g]);
  }
  __syncthreads();
  if (grp == 0) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = q0 + r0 + r;
      const float inv = sC[r0 + r];
      float* orow = o + ((long long)b * p.Sq + i) * p.H * D + (long long)h * D;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int c = lane * 4 + 128 * g;
        if (i < p.Sq && c < D) {
          const float4 u = *reinterpret_cast<const float4*>(sK + (r0 + r) * ld + c);
          *reinterpret_cast<float4*>(orow + c) =
              make_float4((acc[r][4 * g] + u.x) * inv, (acc[r][4 * g + 1] + u.y) * inv, (acc[r][4 * g + 2] + u.z) * inv,
                          (acc[r][4 * g + 3] + u.w) * inv);
        }
      }
    }
  }
}

// delta[b,h,i] = sum_d O[b,i,h,d] * dO[b,i,h,d]; one warp per row
__global__ void attn_f32_delta_kernel(const float* __restrict__ o, const float* __restrict__ d_o,
                                      float* __restrict__ delta, int B, int S, int H, int D) {
  const long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= (long long)B * S * H) return;
  float a = 0.f;
  for (int d = lane; d < D; d += 32) a = fmaf(o[row * D + d], d_o[row * D + d], a);
  a = warp_sum(a);
  if (lane == 0) {
    const int h = int(row % H);
    const long long bs = row / H;
    delta[((bs / S) * H + h) * S + bs % S] = a;
  }
}

// -------------------------------------------------------------------------------------------------------- dQ, dK, dV
// DQ: owners are query rows (A = Q, B = dO), K and V are streamed; otherwise owners are keys (A = K, B = V) and the query
// rows of every head of the group are streamed.  The streamed tiles (head by head, tile by tile) are one list, of which
// the block takes the `split`-th of `splits` parts; its sums go to `out0` (dQ or dK) and `out1` (dV), part by part.  dK / dV
// leaves dS in `ds_keep` (B, H, Sk, Sq rounded up to the tile) unless that is null; tiles it skips stay unwritten.
template <bool DQ, int G>
__global__ void __launch_bounds__(F32_THREADS, 1) attn_f32_bwd_kernel(F32Params p, const float* __restrict__ d_o,
                                                                      const float* __restrict__ lse,
                                                                      const float* __restrict__ delta,
                                                                      float* __restrict__ out0, float* __restrict__ out1,
                                                                      float* __restrict__ ds_keep, int splits) {
  extern __shared__ __align__(16) float smem[];
  const int D = p.D, Dp = (D + 15) & ~15, ld = Dp + 4;
  float* sOA = smem;                        // [32][ld] Q | K
  float* sOB = sOA + F32_OWN * ld;          // [32][ld] dO | V
  float* sSA = sOB + F32_OWN * ld;          // [64][ld] K | Q
  float* sSB = sSA + F32_STR * ld;          // [64][ld] V | dO
  float* sP = sSB + F32_STR * ld;           // [32][F32_PLD] scores; then dS | P
  float* sS = sP + F32_OWN * F32_PLD;       // [32][F32_PLD] dP; then dS
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int o0 = blockIdx.x * F32_OWN, head = blockIdx.y, b = blockIdx.z / splits, split = blockIdx.z % splits;
  const int group = p.H / p.Hkv;
  const int n_own = DQ ? p.Sq : p.Sk, n_str = DQ ? p.Sk : p.Sq;
  const int tiles = (n_str + F32_STR - 1) / F32_STR;
  const long long steps = DQ ? tiles : (long long)tiles * group;
  const int end = (int)(steps * (split + 1) / splits);
  const unsigned char* oval = (DQ ? p.q_valid : p.k_valid) + (long long)b * n_own;
  const int* oblk = (DQ ? p.q_blk : p.k_blk) + (long long)b * n_own;
  const unsigned char* sval = (DQ ? p.k_valid : p.q_valid) + (long long)b * n_str;
  const int* sblk = (DQ ? p.k_blk : p.q_blk) + (long long)b * n_str;
  const Owners own = owner_rows(oval, oblk, o0, n_own, lane, DQ);
  const auto next_step = [&](int st, unsigned long long& rows) {
    for (; st < end; ++st) {
      rows = tile_rows(sval, sblk, st % tiles * F32_STR, n_str, lane, own, DQ);
      if (rows) break;
    }
    return st;
  };
  const int kvh = DQ ? head / group : head;
  const float* kb = p.k + (long long)b * p.k_sb + (long long)kvh * p.k_sh;
  const float* vb = p.v + (long long)b * p.v_sb + (long long)kvh * p.v_sh;
  const float* qb = p.q + (long long)b * p.q_sb;
  const float* dob = d_o + (long long)b * p.Sq * p.H * D;                    // contiguous (B,Sq,H,D)
  const long long do_ss = (long long)p.H * D;
  const auto load_a = [&](int st, unsigned long long rows) {
    const long long r = (long long)(st % tiles) * F32_STR;
    if (DQ) load_rows<F32_STR>(sSA, kb + r * p.k_ss, p.k_ss, rows, D, ld);
    else load_rows<F32_STR>(sSA, qb + (long long)(head * group + st / tiles) * p.q_sh + r * p.q_ss, p.q_ss, rows, D, ld);
  };
  const auto load_b = [&](int st, unsigned long long rows) {
    const long long r = (long long)(st % tiles) * F32_STR;
    if (DQ) load_rows<F32_STR>(sSB, vb + r * p.v_ss, p.v_ss, rows, D, ld);
    else load_rows<F32_STR>(sSB, dob + (long long)(head * group + st / tiles) * D + r * do_ss, do_ss, rows, D, ld);
  };
  if (Dp != D) clear_tail(sOA, 2 * F32_OWN + 2 * F32_STR, D, Dp, ld);
  unsigned long long rows = 0;
  int st = next_step((int)(steps * split / splits), rows);
  {
    const int n = min(F32_OWN, n_own - o0);
    const unsigned long long mine = n >= 32 ? 0xffffffffull : (1ull << n) - 1;
    if (DQ) {
      load_rows<F32_OWN>(sOA, qb + (long long)head * p.q_sh + (long long)o0 * p.q_ss, p.q_ss, mine, D, ld);
      load_rows<F32_OWN>(sOB, dob + (long long)head * D + (long long)o0 * do_ss, do_ss, mine, D, ld);
    } else {
      load_rows<F32_OWN>(sOA, kb + (long long)o0 * p.k_ss, p.k_ss, mine, D, ld);
      load_rows<F32_OWN>(sOB, vb + (long long)o0 * p.v_ss, p.v_ss, mine, D, ld);
    }
    if (st < end) {
      load_a(st, rows);
      load_b(st, rows);
    }
    cp_async_commit();
  }
  const int row = threadIdx.x >> 3, part = threadIdx.x & 7;                  // as in the forward's softmax
  const bool row_ok = (own.ok >> row) & 1;
  const int row_blk = row_ok ? oblk[o0 + row] : 0;
  float row_lse = 0.f, row_delta = 0.f;
  if (DQ && row_ok) {
    row_lse = lse[((long long)b * p.H + head) * p.Sq + o0 + row];
    row_delta = delta[((long long)b * p.H + head) * p.Sq + o0 + row];
  }
  const int grp = warp >> 2, r0 = 8 * (warp & 3), col = lane * 4 < Dp ? lane * 4 : 0;
  float acc[8][4 * G];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4 * G; ++c) acc[r][c] = 0.f;

  while (st < end) {
    cp_async_wait<0>();
    __syncthreads();                                 // owners and both streamed tiles are here
    if (grp == 0) product_by_4_warps(sOA, sSA, sP, Dp, ld, warp & 3, lane);
    else product_by_4_warps(sOB, sSB, sS, Dp, ld, warp & 3, lane);
    __syncthreads();
    const unsigned long long cur = rows;
    const int cur0 = st % tiles * F32_STR;
    const int cur_head = head * group + st / tiles;                                              // dK / dV only
    const long long stat0 = ((long long)b * p.H + cur_head) * p.Sq + cur0;
    st = next_step(st + 1, rows);
    if (DQ && st < end) load_b(st, rows);            // V is not read again for this tile
    {
      float* pp = sP + row * F32_PLD + 4 * part;
      float* ps = sS + row * F32_PLD + 4 * part;
      float s[8], d[8];
      *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(pp);
      *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(pp + 32);
      *reinterpret_cast<float4*>(d) = *reinterpret_cast<const float4*>(ps);
      *reinterpret_cast<float4*>(d + 4) = *reinterpret_cast<const float4*>(ps + 32);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int j = 4 * part + (e & 3) + 32 * (e >> 2);
        float pr = 0.f, ds = 0.f;
        if (row_ok && ((cur >> j) & 1ull)) {
          const int jb = sblk[cur0 + j];
          if (DQ ? jb <= row_blk : row_blk <= jb) {
            pr = expf(s[e] * p.scale - (DQ ? row_lse : lse[stat0 + j]));
            ds = pr * (d[e] - (DQ ? row_delta : delta[stat0 + j])) * p.scale;
          }
        }
        s[e] = pr;
        d[e] = ds;
      }
      if (!DQ) {
        *reinterpret_cast<float4*>(pp) = *reinterpret_cast<const float4*>(s);
        *reinterpret_cast<float4*>(pp + 32) = *reinterpret_cast<const float4*>(s + 4);
      }
      *reinterpret_cast<float4*>(ps) = *reinterpret_cast<const float4*>(d);
      *reinterpret_cast<float4*>(ps + 32) = *reinterpret_cast<const float4*>(d + 4);
      if (!DQ && ds_keep != nullptr && o0 + row < n_own) {
        float* keep = ds_keep + (((long long)b * p.H + cur_head) * p.Sk + o0 + row) * ((long long)tiles * F32_STR) + cur0 + 4 * part;
        *reinterpret_cast<float4*>(keep) = *reinterpret_cast<const float4*>(d);
        *reinterpret_cast<float4*>(keep + 32) = *reinterpret_cast<const float4*>(d + 4);
      }
    }
    __syncthreads();
    if (DQ) accumulate<G>(acc, sS + r0 * F32_PLD, sSA + col, ld, 32 * grp, 32 * grp + 32);
    else if (grp == 0) accumulate<G>(acc, sS + r0 * F32_PLD, sSA + col, ld, 0, F32_STR);        // dK += dS Q
    else accumulate<G>(acc, sP + r0 * F32_PLD, sSB + col, ld, 0, F32_STR);                      // dV += P dO
    __syncthreads();
    if (st < end) {
      load_a(st, rows);
      if (!DQ) load_b(st, rows);
    }
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncthreads();
  const int n_heads = DQ ? p.H : p.Hkv;
  const long long part0 = ((long long)split * p.B + b) * n_own;
  if (DQ && grp == 1 && lane * 4 < Dp) {             // the second group's sums go through shared memory (over K)
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (lane * 4 + 128 * g < Dp)
          *reinterpret_cast<float4*>(sSA + (r0 + r) * ld + col + 128 * g) = *reinterpret_cast<const float4*>(&acc[r][4 * g]);
  }
  if (DQ) __syncthreads();
  if (DQ && grp == 1) return;
  float* out = !DQ && grp == 1 ? out1 : out0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = o0 + r0 + r;
    float* orow = out + ((part0 + i) * n_heads + head) * D;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int c = lane * 4 + 128 * g;
      if (i < n_own && c < D) {
        float4 u = *reinterpret_cast<const float4*>(&acc[r][4 * g]);
        if (DQ) {
          const float4 w = *reinterpret_cast<const float4*>(sSA + (r0 + r) * ld + c);
          u = make_float4(u.x + w.x, u.y + w.y, u.z + w.z, u.w + w.w);
        }
        *reinterpret_cast<float4*>(orow + c) = u;
      }
    }
  }
}

// dQ from the kept dS (`ds`: B, H, Sk, sq_ld): one product per streamed tile of keys, both operands double-buffered.
template <int G>
__global__ void __launch_bounds__(F32_THREADS, 1) attn_f32_dq_kernel(F32Params p, const float* __restrict__ ds, int sq_ld,
                                                                     float* __restrict__ out, int splits) {
  extern __shared__ __align__(16) float smem[];
  constexpr int TLD = F32_OWN + 4;
  const int D = p.D, Dp = (D + 15) & ~15, ld = Dp + 4;
  float* sK = smem;                         // [2][64][ld]
  float* sT = sK + 2 * F32_STR * ld;        // [2][64][TLD] dS, a row per key
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int o0 = blockIdx.x * F32_OWN, h = blockIdx.y, b = blockIdx.z / splits, split = blockIdx.z % splits;
  const int tiles = (p.Sk + F32_STR - 1) / F32_STR, end = (int)((long long)tiles * (split + 1) / splits);
  const float* kb = p.k + (long long)b * p.k_sb + (long long)(h / (p.H / p.Hkv)) * p.k_sh;
  const float* tb = ds + ((long long)b * p.H + h) * p.Sk * (long long)sq_ld + o0;
  const unsigned char* kval = p.k_valid + (long long)b * p.Sk;
  const int* kblk = p.k_blk + (long long)b * p.Sk;
  const Owners own = owner_rows(p.q_valid + (long long)b * p.Sq, p.q_blk + (long long)b * p.Sq, o0, p.Sq, lane, true);
  const auto next_load = [&](int st, int buf) {      // the next tile that meets an owner row, on its way into `buf`
    unsigned long long rows = 0;
    for (; st < end; ++st) {
      rows = tile_rows(kval, kblk, st * F32_STR, p.Sk, lane, own, true);
      if (rows) break;
    }
    if (st < end) {
      load_rows<F32_STR>(sK + buf * F32_STR * ld, kb + (long long)st * F32_STR * p.k_ss, p.k_ss, rows, D, ld);
      load_rows<F32_STR>(sT + buf * F32_STR * TLD, tb + (long long)st * F32_STR * sq_ld, sq_ld, rows, F32_OWN, TLD);
    }
    cp_async_commit();
    return st;
  };
  const int grp = warp >> 2, r0 = 8 * (warp & 3), col = lane * 4 < Dp ? lane * 4 : 0;
  float acc[8][4 * G];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4 * G; ++c) acc[r][c] = 0.f;
  int buf = 0;
  for (int st = next_load((int)((long long)tiles * split / splits), 0); st < end; buf ^= 1) {
    st = next_load(st + 1, buf ^ 1);
    cp_async_wait<1>();
    __syncthreads();
    const float* x = sK + (buf * F32_STR + 32 * grp) * ld + col;
    const float* t = sT + (buf * F32_STR + 32 * grp) * TLD + r0;
#pragma unroll 4
    for (int j = 0; j < 32; ++j) {
      float pv[8];
      *reinterpret_cast<float4*>(pv) = *reinterpret_cast<const float4*>(t + j * TLD);
      *reinterpret_cast<float4*>(pv + 4) = *reinterpret_cast<const float4*>(t + j * TLD + 4);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 y = *reinterpret_cast<const float4*>(x + j * ld + 128 * g);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          acc[r][4 * g + 0] = fmaf(pv[r], y.x, acc[r][4 * g + 0]);
          acc[r][4 * g + 1] = fmaf(pv[r], y.y, acc[r][4 * g + 1]);
          acc[r][4 * g + 2] = fmaf(pv[r], y.z, acc[r][4 * g + 2]);
          acc[r][4 * g + 3] = fmaf(pv[r], y.w, acc[r][4 * g + 3]);
        }
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  __syncthreads();
  if (grp == 1) {                                    // the second group's sums go through shared memory
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (lane * 4 + 128 * g < Dp)
          *reinterpret_cast<float4*>(sK + (r0 + r) * ld + lane * 4 + 128 * g) = *reinterpret_cast<const float4*>(&acc[r][4 * g]);
  }
  __syncthreads();
  if (grp == 1) return;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int i = o0 + r0 + r;
    float* orow = out + ((((long long)split * p.B + b) * p.Sq + i) * p.H + h) * D;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int c = lane * 4 + 128 * g;
      if (i < p.Sq && c < D) {
        const float4 u = *reinterpret_cast<const float4*>(&acc[r][4 * g]);
        const float4 w = *reinterpret_cast<const float4*>(sK + (r0 + r) * ld + c);
        *reinterpret_cast<float4*>(orow + c) = make_float4(u.x + w.x, u.y + w.y, u.z + w.z, u.w + w.w);
      }
    }
  }
}

// out[i] = sum over `splits` parts of n4 float4 each, in order
__global__ void attn_f32_sum_kernel(const float4* __restrict__ parts, float4* __restrict__ out, long long n4, int splits) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n4) return;
  float4 a = parts[i];
  for (int s = 1; s < splits; ++s) {
    const float4 u = parts[s * n4 + i];
    a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
  }
  out[i] = a;
}

static int check(const F32Params& p) {
  if (p.B <= 0 || p.Sq <= 0 || p.Sk <= 0 || p.H <= 0 || p.Hkv <= 0 || p.H % p.Hkv) return -2;
  if (p.D % 4 || p.D < 4 || p.D > 256) return -4;
  const long long st[9] = {p.q_sb, p.q_ss, p.q_sh, p.k_sb, p.k_ss, p.k_sh, p.v_sb, p.v_ss, p.v_sh};
  for (int i = 0; i < 9; ++i)
    if (st[i] % 4) return -5;
  if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15)
    return -6;
  return 0;
}

template <typename K>
static int set_smem(K kern, size_t bytes) {
  return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Into how many parts the streamed tiles are dealt: the fewest rounds of one block per SM for the work there is, and a
// hundredth of it charged per part (its partial sums are written and read once more).
static int pick_splits(long long blocks, long long steps, int B, long long out_bytes) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) return 1;
  }
  int best = 1;
  double best_cost = 0;
  for (int s = 1; s <= F32_MAX_SPLITS && s <= steps && (long long)B * s <= 65535 && (s == 1 || s * out_bytes <= F32_MAX_SCRATCH);
       ++s) {
    const long long per = (steps + s - 1) / s;
    const double cost = (double)((blocks * s + sms - 1) / sms) * per * (1.0 + 0.01 * (s - 1));
    if (s == 1 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace otb

using namespace otb;

static F32Params make_params(const float* q, const float* k, const float* v, const int* q_blk, const int* k_blk,
                             const unsigned char* q_valid, const unsigned char* k_valid, int B, int Sq, int Sk, int H,
                             int Hkv, int D, long long q_sb, long long q_ss, long long q_sh, long long k_sb,
                             long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh,
                             float scale) {
  F32Params p;
  p.q = q; p.k = k; p.v = v;
  p.q_sb = q_sb; p.q_ss = q_ss; p.q_sh = q_sh; p.k_sb = k_sb; p.k_ss = k_ss; p.k_sh = k_sh;
  p.v_sb = v_sb; p.v_ss = v_ss; p.v_sh = v_sh;
  p.q_blk = q_blk; p.k_blk = k_blk; p.q_valid = q_valid; p.k_valid = k_valid;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.D = D; p.scale = scale;
  return p;
}

// q (B,Sq,H,D), k / v (B,Sk,Hkv,D) fp32 with element strides (innermost 1); o (B,Sq,H*D) and lse (B,H,Sq) contiguous.
extern "C" int otb_attn_f32_fwd(const float* q, const float* k, const float* v, float* o, float* lse, const int* q_blk,
                                const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid, int B,
                                int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh,
                                long long k_sb, long long k_ss, long long k_sh, long long v_sb, long long v_ss,
                                long long v_sh, float scale, cudaStream_t stream) {
  const F32Params p = make_params(q, k, v, q_blk, k_blk, q_valid, k_valid, B, Sq, Sk, H, Hkv, D, q_sb, q_ss, q_sh, k_sb,
                                  k_ss, k_sh, v_sb, v_ss, v_sh, scale);
  int r = check(p);
  if (r) return r;
  const int ld = (D + 15) / 16 * 16 + 4;
  const size_t smem = (size_t)((F32_OWN + 2 * F32_STR) * ld + F32_OWN * F32_PLD + F32_OWN) * 4;
  const dim3 grid((Sq + F32_OWN - 1) / F32_OWN, H, B);
  auto kern = D > 128 ? attn_f32_fwd_kernel<2> : attn_f32_fwd_kernel<1>;
  r = set_smem(kern, smem);
  if (r) return r;
  kern<<<grid, F32_THREADS, smem, stream>>>(p, o, lse);
  return (int)cudaGetLastError();
}

// Scratch of the backward: `dq` and `dkv` above 1 want that many outputs each (the parts that the streamed tiles are dealt
// to); `ds` floats for dS, 0 where it would pass F32_MAX_DS and is recomputed instead.
extern "C" void otb_attn_f32_bwd_plan(int B, int Sq, int Sk, int H, int Hkv, int D, int* dq, int* dkv, long long* ds) {
  const long long qt = (Sq + F32_STR - 1) / F32_STR, kt = (Sk + F32_STR - 1) / F32_STR;
  *dq = pick_splits((long long)((Sq + F32_OWN - 1) / F32_OWN) * H * B, kt, B, 4ll * B * Sq * H * D);
  *dkv = pick_splits((long long)((Sk + F32_OWN - 1) / F32_OWN) * Hkv * B, qt * (H / Hkv), B,
                     4ll * B * Sk * Hkv * D);
  const long long n = (long long)B * H * Sk * qt * F32_STR;
  *ds = n * 4 <= F32_MAX_DS ? n : 0;
}

// o, d_o (B,Sq,H,D) contiguous; delta: scratch (B,H,Sq); dq (B,Sq,H,D), dk / dv (B,Sk,Hkv,D) contiguous outputs; dq_parts:
// scratch of dq_splits outputs where that is above 1, dk_parts / dv_parts likewise; ds: scratch for dS, null to recompute it.
extern "C" int otb_attn_f32_bwd(const float* q, const float* k, const float* v, const float* o, const float* d_o,
                                const float* lse, float* delta, float* dq, float* dk, float* dv, float* dq_parts,
                                float* dk_parts, float* dv_parts, float* ds, int dq_splits, int dkv_splits, const int* q_blk,
                                const int* k_blk, const unsigned char* q_valid, const unsigned char* k_valid, int B,
                                int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh,
                                long long k_sb, long long k_ss, long long k_sh, long long v_sb, long long v_ss,
                                long long v_sh, float scale, cudaStream_t stream) {
  const F32Params p = make_params(q, k, v, q_blk, k_blk, q_valid, k_valid, B, Sq, Sk, H, Hkv, D, q_sb, q_ss, q_sh, k_sb,
                                  k_ss, k_sh, v_sb, v_ss, v_sh, scale);
  int r = check(p);
  if (r) return r;
  if (dq_splits < 1 || dkv_splits < 1 || dq_splits > F32_MAX_SPLITS || dkv_splits > F32_MAX_SPLITS ||
      (dq_splits > 1 && !dq_parts) || (dkv_splits > 1 && (!dk_parts || !dv_parts)))
    return -7;
  if ((reinterpret_cast<uintptr_t>(d_o) | reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
       reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(dq_parts) | reinterpret_cast<uintptr_t>(dk_parts) |
       reinterpret_cast<uintptr_t>(dv_parts) | reinterpret_cast<uintptr_t>(ds)) & 15)
    return -6;
  {
    const long long rows = (long long)B * Sq * H;
    const long long blocks = (rows * 32 + 255) / 256;
    attn_f32_delta_kernel<<<(unsigned)blocks, 256, 0, stream>>>(o, d_o, delta, B, Sq, H, D);
  }
  const int ld = (D + 15) / 16 * 16 + 4;
  const size_t smem = (size_t)((2 * F32_OWN + 2 * F32_STR) * ld + 2 * F32_OWN * F32_PLD) * 4;
  const dim3 grid_q((Sq + F32_OWN - 1) / F32_OWN, H, B * dq_splits);
  const dim3 grid_kv((Sk + F32_OWN - 1) / F32_OWN, Hkv, B * dkv_splits);
  auto kern_kv = D > 128 ? attn_f32_bwd_kernel<false, 2> : attn_f32_bwd_kernel<false, 1>;
  r = set_smem(kern_kv, smem);
  if (r) return 100000 + r;
  kern_kv<<<grid_kv, F32_THREADS, smem, stream>>>(p, d_o, lse, delta, dkv_splits > 1 ? dk_parts : dk,
                                                  dkv_splits > 1 ? dv_parts : dv, ds, dkv_splits);
  float* dq_out = dq_splits > 1 ? dq_parts : dq;
  if (ds != nullptr) {
    const size_t smem_q = (size_t)(2 * F32_STR * (ld + F32_OWN + 4)) * 4;
    auto kern_q = D > 128 ? attn_f32_dq_kernel<2> : attn_f32_dq_kernel<1>;
    r = set_smem(kern_q, smem_q);
    if (r) return r;
    kern_q<<<grid_q, F32_THREADS, smem_q, stream>>>(p, ds, (Sq + F32_STR - 1) / F32_STR * F32_STR, dq_out, dq_splits);
  } else {
    auto kern_q = D > 128 ? attn_f32_bwd_kernel<true, 2> : attn_f32_bwd_kernel<true, 1>;
    r = set_smem(kern_q, smem);
    if (r) return r;
    kern_q<<<grid_q, F32_THREADS, smem, stream>>>(p, d_o, lse, delta, dq_out, nullptr, nullptr, dq_splits);
  }
  const auto add = [&](const float* parts, float* out, long long n, int splits) {
    if (splits > 1)
      attn_f32_sum_kernel<<<(unsigned)((n / 4 + 255) / 256), 256, 0, stream>>>(
          reinterpret_cast<const float4*>(parts), reinterpret_cast<float4*>(out), n / 4, splits);
  };
  add(dq_parts, dq, (long long)B * Sq * H * D, dq_splits);
  add(dk_parts, dk, (long long)B * Sk * Hkv * D, dkv_splits);
  add(dv_parts, dv, (long long)B * Sk * Hkv * D, dkv_splits);
  return (int)cudaGetLastError();
}
