// Exact f32 attention forward on the FFMA pipe.
//
// Replaces autorust's `ar_flash_f32` (src/runtime/cuda_flash.rs:48-142): same math --
// s = (q.k) * 1/sqrt(D) (+ mask), key >= S or (causal and key > row) -> -1e30, online softmax
// with expf, O = acc * (l > 0 ? 1/l : 0) -- but tiled for registers instead of one thread
// per query row.  No tensor cores and no reduced precision anywhere: this is the mode that must agree with the graph
// SDPA to 1e-5.
//
// A CTA owns RQ * TY query rows.  Its GROUPS groups of TX * TY threads take the key tiles of 64 in turn, each with an
// online softmax of its own, and one combination at the end adds the groups' sums.  A thread keeps RQ x 64/TX scores
// and RQ x D/TX outputs in registers.  K and V tiles arrive by cp.async under the other half of the group's step.
// Bound: the FFMA pipe and the shared-memory reads.  Four d of an RQ x JK block cost RQ + JK 16-byte reads per thread (4
// cycles per warp and SM each) for 4 * RQ * JK FFMA (1 cycle per warp and scheduler): 4 x 4 reads 32 cycles for 16 of
// math, 8 x 8 breaks even at 64.
#include "ar_ptx.cuh"
#include "cta_order.cuh"

#include <cmath>
#include "ar_kernels.h"

namespace ar {
namespace {

using namespace arptx;

constexpr int BK = 64;  // keys per tile
constexpr float NEG = -1e30f;

template <int D, int RQ, int TX, int TY, int GROUPS>
struct ExactCfg {
  static constexpr int BQ = RQ * TY;           // query rows of a CTA
  static constexpr int GT = TX * TY;           // threads of a group
  static constexpr int THREADS = GT * GROUPS;
  static constexpr int JK = BK / TX;           // scores per row and thread
  static constexpr int OD = D / (4 * TX);      // float4 output columns per row and thread
  static constexpr int LDQ = D + 4;            // padded rows (floats): 16-byte aligned, conflict-free float4 reads
  static constexpr int LDP = BK + (TX == 8 ? 8 : 16);  // the rows of a warp's lanes fall into different banks
  static constexpr int GROUP_FLOATS = BK * LDQ + BK * D + BQ * LDP;  // K, V, P
  static constexpr int SMEM_BYTES = (BQ * LDQ + GROUPS * GROUP_FLOATS) * 4;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static_assert(GT * (RQ * OD * 4 + 2 * RQ) <= GROUP_FLOATS, "a group's result passes through its own tiles");
};

// CAUSAL: the mask is known when the kernel is compiled (NO, YES) for the forms whose tiles reach over the end of a row's 64
// keys (see `past`): what that takes cost the 128-row form 2 to 5 % without a mask.  The others are told at run time, and so
// is the 12-row form without a mask, which is 2 to 4 % faster that way.
enum { CAUSAL_NO, CAUSAL_YES, CAUSAL_ARG };
template <int D, int RQ, int TX, int TY, int GROUPS, int CAUSAL>
__global__ void __launch_bounds__(TX* TY* GROUPS, 1)
    attn_fwd_exact_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                          float* __restrict__ O, const float* __restrict__ M, float* __restrict__ LSE, int N, int Hq,
                          int Hkv, int grouped, int causal_arg) {
  using C = ExactCfg<D, RQ, TX, TY, GROUPS>;
  constexpr int JK = C::JK, OD = C::OD, D4 = D / 4;
  extern __shared__ __align__(16) float smem_f[];
  const int tid = threadIdx.x, grp = tid / C::GT, gt = tid % C::GT;
  const int tx = gt % TX, ty = gt / TX;  // rows ty + TY * i, keys tx + TX * jj, columns (tx + TX * dd) * 4 ..
  float* sQ = smem_f;
  float* sK = sQ + C::BQ * C::LDQ + grp * C::GROUP_FLOATS;
  float* sV = sK + BK * C::LDQ;
  float* sP = sV + BK * D;
  const int bh = cta_head(grouped);
  int tile = cta_tile(grouped);
  const bool causal = CAUSAL == CAUSAL_ARG ? causal_arg != 0 : CAUSAL == CAUSAL_YES;
  if (causal) tile = cta_tiles(grouped) - 1 - tile;  // the last query tile sees the most keys
  const int b = bh / Hq, h = bh - b * Hq;
  const int kvbh = b * Hkv + h / (Hq / Hkv);
  const int q0 = tile * C::BQ;
  const float* qb = Q + (size_t)bh * N * D;
  const float* kb = K + (size_t)kvbh * N * D;
  const float* vb = V + (size_t)kvbh * N * D;
  const float scale = 1.0f / sqrtf((float)D);

  auto load_rows = [&](float* dst, int ld, const float* src, int row0) {  // 64 rows; past the end: zeros
#pragma unroll 4
    for (int i = gt; i < BK * D4; i += C::GT) {
      const int r = i / D4, c = i % D4;
      const bool in = row0 + r < N;
      cp_async16(smem_u32(dst + r * ld + c * 4), in ? src + (size_t)(row0 + r) * D + c * 4 : src, in);
    }
    cp_async_commit();
  };
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(C::GT) : "memory"); };

  const int kend = causal ? min(N, q0 + C::BQ) : N;
  const int tiles = (kend + BK - 1) / BK;
  for (int i = tid; i < C::BQ * D4; i += C::THREADS) {
    const int r = i / D4, c = i % D4;
    const bool in = q0 + r < N;
    cp_async16(smem_u32(sQ + r * C::LDQ + c * 4), in ? qb + (size_t)(q0 + r) * D + c * 4 : qb, in);
  }
  cp_async_commit();
  load_rows(sK, C::LDQ, kb, grp * BK);
  load_rows(sV, D, vb, grp * BK);
  cp_async_wait<2>();
  __syncthreads();  // Q is visible to every group

  float m[RQ], l[RQ];
  float4 o[RQ][OD];
#pragma unroll
  for (int i = 0; i < RQ; i++) {
    m[i] = NEG;
    l[i] = 0.f;
#pragma unroll
    for (int dd = 0; dd < OD; dd++) o[i][dd] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int kt = grp; kt < tiles; kt += GROUPS) {
    const int k0 = kt * BK;
    cp_async_wait<1>();  // K of this tile (V still in flight)
    group_sync();
    float s[RQ][JK];
#pragma unroll
    for (int i = 0; i < RQ; i++)
#pragma unroll
      for (int jj = 0; jj < JK; jj++) s[i][jj] = 0.f;
#pragma unroll 2
    for (int d4 = 0; d4 < D4; d4++) {
      float4 kv[JK];
#pragma unroll
      for (int jj = 0; jj < JK; jj++) kv[jj] = *(const float4*)(sK + (tx + TX * jj) * C::LDQ + d4 * 4);
#pragma unroll
      for (int i = 0; i < RQ; i++) {
        const float4 qv = *(const float4*)(sQ + (ty + TY * i) * C::LDQ + d4 * 4);
#pragma unroll
        for (int jj = 0; jj < JK; jj++) {
          s[i][jj] = fmaf(qv.x, kv[jj].x, s[i][jj]);
          s[i][jj] = fmaf(qv.y, kv[jj].y, s[i][jj]);
          s[i][jj] = fmaf(qv.z, kv[jj].z, s[i][jj]);
          s[i][jj] = fmaf(qv.w, kv[jj].w, s[i][jj]);
        }
      }
    }
    group_sync();  // the group is done with this K tile
    load_rows(sK, C::LDQ, kb, min(k0 + GROUPS * BK, N));  // (past the last tile: zeros, nothing is read)
    // Excluded keys get the finite sentinel, which a row whose visible keys all carry -1e30 counts along.  Under a causal
    // mask a row counts them up to the end of the 64 keys its diagonal lies in; a CTA whose rows reach over that end gives
    // them no weight, so that such a row has the same value whatever tile height its call takes.
    const bool past = CAUSAL == CAUSAL_YES && k0 > q0;
    const bool bounds = k0 + BK > N || (causal && k0 + BK - 1 > q0);
#pragma unroll
    for (int i = 0; i < RQ; i++) {
      const int row = q0 + ty + TY * i;
      // (tiles of 128 rows reach over the end by whole halves of their rows)
      const float out = past && (C::BQ == 2 * BK ? TY * i < BK : row < k0) ? -INFINITY : NEG;
      float mx = m[i];
#pragma unroll
      for (int jj = 0; jj < JK; jj++) {
        const int key = k0 + tx + TX * jj;
        float x = s[i][jj] * scale;
        if (M != nullptr && row < N && key < N) x += M[(size_t)row * N + key];
        if (bounds && (key >= N || (causal && key > row))) x = out;
        s[i][jj] = x;
        mx = fmaxf(mx, x);
      }
#pragma unroll
      for (int sh = 1; sh < TX; sh <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
      const float alpha = expf(m[i] - mx);
      float sum = 0.f;
#pragma unroll
      for (int jj = 0; jj < JK; jj++) {
        const float p = expf(s[i][jj] - mx);
        sum += p;
        sP[(ty + TY * i) * C::LDP + tx + TX * jj] = p;
      }
#pragma unroll
      for (int sh = 1; sh < TX; sh <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
      l[i] = l[i] * alpha + sum;
      m[i] = mx;
#pragma unroll
      for (int dd = 0; dd < OD; dd++) {
        o[i][dd].x *= alpha;
        o[i][dd].y *= alpha;
        o[i][dd].z *= alpha;
        o[i][dd].w *= alpha;
      }
    }
    cp_async_wait<1>();  // V of this tile
    group_sync();        // ... of every thread, and P
#pragma unroll 2
    for (int k4 = 0; k4 < BK / 4; k4++) {
      float4 v4[4][OD];
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
#pragma unroll
        for (int dd = 0; dd < OD; dd++) v4[kk][dd] = *(const float4*)(sV + (k4 * 4 + kk) * D + (tx + TX * dd) * 4);
#pragma unroll
      for (int i = 0; i < RQ; i++) {
        const float4 pv = *(const float4*)(sP + (ty + TY * i) * C::LDP + k4 * 4);
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
          const float p = kk == 0 ? pv.x : kk == 1 ? pv.y : kk == 2 ? pv.z : pv.w;
#pragma unroll
          for (int dd = 0; dd < OD; dd++) {
            o[i][dd].x = fmaf(p, v4[kk][dd].x, o[i][dd].x);
            o[i][dd].y = fmaf(p, v4[kk][dd].y, o[i][dd].y);
            o[i][dd].z = fmaf(p, v4[kk][dd].z, o[i][dd].z);
            o[i][dd].w = fmaf(p, v4[kk][dd].w, o[i][dd].w);
          }
        }
      }
    }
    group_sync();  // the group is done with V and P
    load_rows(sV, D, vb, min(k0 + GROUPS * BK, N));
  }
  cp_async_wait<0>();
  if constexpr (GROUPS > 1) {
    // groups 1 .. leave (m, l, o) in their own tiles, laid out so that group 0's thread of the same place reads its
    // counterparts' values side by side with its neighbours
    float* mine = sK + gt;
    __syncthreads();
    if (grp > 0) {
#pragma unroll
      for (int i = 0; i < RQ; i++) {
        mine[(2 * i) * C::GT] = m[i];
        mine[(2 * i + 1) * C::GT] = l[i];
#pragma unroll
        for (int dd = 0; dd < OD; dd++) {
          float* at = mine + (2 * RQ + (i * OD + dd) * 4) * C::GT;
          at[0] = o[i][dd].x;
          at[C::GT] = o[i][dd].y;
          at[2 * C::GT] = o[i][dd].z;
          at[3 * C::GT] = o[i][dd].w;
        }
      }
    }
    __syncthreads();
    if (grp > 0) return;
#pragma unroll 1
    for (int g = 1; g < GROUPS; g++) {
      const float* theirs = mine + g * C::GROUP_FLOATS;
#pragma unroll
      for (int i = 0; i < RQ; i++) {
        const float mg = theirs[(2 * i) * C::GT], mx = fmaxf(m[i], mg);
        const float a0 = expf(m[i] - mx), a1 = expf(mg - mx);
        l[i] = l[i] * a0 + theirs[(2 * i + 1) * C::GT] * a1;
        m[i] = mx;
#pragma unroll
        for (int dd = 0; dd < OD; dd++) {
          const float* at = theirs + (2 * RQ + (i * OD + dd) * 4) * C::GT;
          o[i][dd].x = o[i][dd].x * a0 + at[0] * a1;
          o[i][dd].y = o[i][dd].y * a0 + at[C::GT] * a1;
          o[i][dd].z = o[i][dd].z * a0 + at[2 * C::GT] * a1;
          o[i][dd].w = o[i][dd].w * a0 + at[3 * C::GT] * a1;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RQ; i++) {
    const int row = q0 + ty + TY * i;
    if (row >= N) continue;
    const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
    // training forward: the row's log-sum-exp, LSE = m + log(l) (src/runtime/cuda_flash_train.rs:8-11)
    if (LSE != nullptr && tx == 0) LSE[(size_t)bh * N + row] = m[i] + logf(l[i]);
    float* dst = O + ((size_t)bh * N + row) * D;
#pragma unroll
    for (int dd = 0; dd < OD; dd++)
      *(float4*)(dst + (tx + TX * dd) * 4) =
          make_float4(o[i][dd].x * inv, o[i][dd].y * inv, o[i][dd].z * inv, o[i][dd].w * inv);
  }
}

template <int D, int RQ, int TX, int TY, int GROUPS>
cudaError_t launch_exact(const ExactArgs& a, cudaStream_t stream) {
  using C = ExactCfg<D, RQ, TX, TY, GROUPS>;
  constexpr bool ENDS_WITH_KEYS = BK % C::BQ == 0;
  auto kern = attn_fwd_exact_kernel<D, RQ, TX, TY, GROUPS, ENDS_WITH_KEYS || C::BQ == 12 ? CAUSAL_ARG : CAUSAL_NO>;
  if (!ENDS_WITH_KEYS && a.causal) kern = attn_fwd_exact_kernel<D, RQ, TX, TY, GROUPS, ENDS_WITH_KEYS ? CAUSAL_ARG : CAUSAL_YES>;
  static bool configured[2][64] = {};
  const int form = a.causal ? 1 : 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[form][dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured[form][dev] = true;
  }
  const CtaGrid g = cta_grid((size_t)a.S * D * 8 / (size_t)(a.Hq / a.Hkv), a.B * a.Hq, (a.S + C::BQ - 1) / C::BQ,
                             a.causal ? CAUSAL_TILES : a.S % C::BQ != 0);
  kern<<<g.grid, C::THREADS, C::SMEM_BYTES, stream>>>(a.q, a.k, a.v, a.out, a.mask, a.lse, a.S, a.Hq, a.Hkv, g.grouped,
                                                     a.causal);
  return cudaGetLastError();
}

// The plain form: 4 x 4 scores per thread on 64 rows, one group, plain loads; at D = 64 three CTAs of an SM fill each other's
// waits.  It needs no key tiles to deal out, so it ends first for short sequences of many heads, and where larger tiles
// would leave a last round half empty.
constexpr int PLAIN_BQ = 64;
template <int D>
constexpr int PLAIN_SMEM = (PLAIN_BQ * (D + 4) + BK * (D + 4) + BK * D + PLAIN_BQ * (BK + 4)) * 4;
template <int D>
__global__ void __launch_bounds__(256) attn_fwd_exact_plain_kernel(const float* __restrict__ Q, const float* __restrict__ K,
                                                             const float* __restrict__ V, float* __restrict__ O,
                                                             const float* __restrict__ M, float* __restrict__ LSE,
                                                             int N, int Hq, int Hkv, int causal) {
  constexpr int LDQ = D + 4, LDP = BK + 4;  // padded rows (floats)
  extern __shared__ __align__(16) float smem_f[];
  float* sQ = smem_f;
  float* sK = sQ + PLAIN_BQ * LDQ;
  float* sV = sK + BK * LDQ;
  float* sP = sV + BK * D;
  const int tid = threadIdx.x;
  const int tx = tid & 15;
  const int ty = tid >> 4;
  const int bh = blockIdx.y;
  const int b = bh / Hq;
  const int h = bh - b * Hq;
  const int kvbh = b * Hkv + h / (Hq / Hkv);
  const int q0 = blockIdx.x * PLAIN_BQ;
  const float* qb = Q + (size_t)bh * N * D;
  const float* kb = K + (size_t)kvbh * N * D;
  const float* vb = V + (size_t)kvbh * N * D;
  const float scale = 1.0f / sqrtf((float)D);
  constexpr int D4 = D / 4;
  constexpr int OD = D / 64;  // float4 output groups per thread

  for (int i = tid; i < PLAIN_BQ * D4; i += 256) {
    const int r = i / D4, c = i - r * D4;
    float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q0 + r < N) v4 = *(const float4*)(qb + (size_t)(q0 + r) * D + c * 4);
    *(float4*)(sQ + r * LDQ + c * 4) = v4;
  }
  float m[4], l[4];
  float4 o[4][OD];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    m[i] = NEG;
    l[i] = 0.f;
#pragma unroll
    for (int dd = 0; dd < OD; dd++) o[i][dd] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int kend = causal ? min(N, q0 + PLAIN_BQ) : N;
  for (int k0 = 0; k0 < kend; k0 += BK) {
    __syncthreads();  // previous tile fully consumed (and sQ visible on the first pass)
    for (int i = tid; i < BK * D4; i += 256) {
      const int r = i / D4, c = i - r * D4;
      float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f), v4 = k4;
      if (k0 + r < N) {
        k4 = *(const float4*)(kb + (size_t)(k0 + r) * D + c * 4);
        v4 = *(const float4*)(vb + (size_t)(k0 + r) * D + c * 4);
      }
      *(float4*)(sK + r * LDQ + c * 4) = k4;
      *(float4*)(sV + r * D + c * 4) = v4;
    }
    __syncthreads();
    // S block: rows ty*4+i, keys tx+16*jj
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int jj = 0; jj < 4; jj++) s[i][jj] = 0.f;
#pragma unroll 4
    for (int d4 = 0; d4 < D4; d4++) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) qv[i] = *(const float4*)(sQ + (ty * 4 + i) * LDQ + d4 * 4);
#pragma unroll
      for (int jj = 0; jj < 4; jj++) kv[jj] = *(const float4*)(sK + (tx + 16 * jj) * LDQ + d4 * 4);
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
          s[i][jj] = fmaf(qv[i].x, kv[jj].x, s[i][jj]);
          s[i][jj] = fmaf(qv[i].y, kv[jj].y, s[i][jj]);
          s[i][jj] = fmaf(qv[i].z, kv[jj].z, s[i][jj]);
          s[i][jj] = fmaf(qv[i].w, kv[jj].w, s[i][jj]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int row = q0 + ty * 4 + i;
      float mx = m[i];
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const int key = k0 + tx + 16 * jj;
        float x = s[i][jj] * scale;
        if (M != nullptr && row < N && key < N) x += M[(size_t)row * N + key];
        if (key >= N || (causal && key > row)) x = NEG;
        s[i][jj] = x;
        mx = fmaxf(mx, x);
      }
#pragma unroll
      for (int sh = 1; sh < 16; sh <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
      const float alpha = expf(m[i] - mx);
      float sum = 0.f;
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const float p = expf(s[i][jj] - mx);
        sum += p;
        sP[(ty * 4 + i) * LDP + tx + 16 * jj] = p;
      }
#pragma unroll
      for (int sh = 1; sh < 16; sh <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, sh);
      l[i] = l[i] * alpha + sum;
      m[i] = mx;
#pragma unroll
      for (int dd = 0; dd < OD; dd++) {
        o[i][dd].x *= alpha;
        o[i][dd].y *= alpha;
        o[i][dd].z *= alpha;
        o[i][dd].w *= alpha;
      }
    }
    __syncthreads();
    // O block: rows ty*4+i, columns tx*4 + 64*dd
#pragma unroll 4
    for (int k4 = 0; k4 < BK / 4; k4++) {
      float4 pv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) pv[i] = *(const float4*)(sP + (ty * 4 + i) * LDP + k4 * 4);
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
#pragma unroll
        for (int dd = 0; dd < OD; dd++) {
          const float4 v4 = *(const float4*)(sV + (k4 * 4 + kk) * D + tx * 4 + 64 * dd);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float p = kk == 0 ? pv[i].x : kk == 1 ? pv[i].y : kk == 2 ? pv[i].z : pv[i].w;
            o[i][dd].x = fmaf(p, v4.x, o[i][dd].x);
            o[i][dd].y = fmaf(p, v4.y, o[i][dd].y);
            o[i][dd].z = fmaf(p, v4.z, o[i][dd].z);
            o[i][dd].w = fmaf(p, v4.w, o[i][dd].w);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = q0 + ty * 4 + i;
    if (row >= N) continue;
    const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
    // training forward: the row's log-sum-exp, LSE = m + log(l) (src/runtime/cuda_flash_train.rs:8-11)
    if (LSE != nullptr && tx == 0) LSE[(size_t)bh * N + row] = m[i] + logf(l[i]);
    float* dst = O + ((size_t)bh * N + row) * D;
#pragma unroll
    for (int dd = 0; dd < OD; dd++)
      *(float4*)(dst + tx * 4 + 64 * dd) =
          make_float4(o[i][dd].x * inv, o[i][dd].y * inv, o[i][dd].z * inv, o[i][dd].w * inv);
  }
}

template <int D>
cudaError_t launch_exact_plain(const ExactArgs& a, cudaStream_t stream) {
  auto kern = attn_fwd_exact_plain_kernel<D>;
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PLAIN_SMEM<D>);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  kern<<<dim3((a.S + PLAIN_BQ - 1) / PLAIN_BQ, a.B * a.Hq, 1), 256, PLAIN_SMEM<D>, stream>>>(
      a.q, a.k, a.v, a.out, a.mask, a.lse, a.S, a.Hq, a.Hkv, a.causal);
  return cudaGetLastError();
}

// What a CTA of each form costs, in microseconds: cta + step * (its groups' turns) + tile * (its key tiles of 64), and
// `launch` once per launch.  Fitted to the device times of every form at 302 shapes (D = 64 and 128, S = 50 to 2048, 2 to
// 200 heads, causal and not); without a causal mask the fits are within 3 % in the mean, 11 % at worst.
struct Form {
  int rows, groups;
  double launch, cta, step, tile;
};
constexpr Form FORMS_64[] = {{8, 4, 1.2, 1.9, 1.45, 0.77}, {12, 4, 1.2, 2.4, 1.8, 0.88}, {16, 4, 1.2, 2.5, 2.5, 0.92},
                             {20, 4, 1.2, 2.8, 3.05, 1.0}, {24, 4, 1.5, 3.2, 3.5, 1.1},  {32, 4, 1.7, 3.6, 4.35, 1.25},
                             {64, 2, 1.5, 2.1, 3.0, 3.1},  {128, 2, 2.3, 2.2, 5.4, 5.3}};
constexpr Form FORMS_128[] = {{8, 2, 1.2, 2.3, 3.3, 0.6},   {12, 2, 1.2, 2.5, 4.45, 0.42}, {16, 2, 1.3, 2.6, 5.5, 0.36},
                              {20, 2, 1.7, 3.05, 6.9, 0.2}, {24, 2, 1.9, 3.5, 7.1, 0.37},  {32, 2, 2.3, 3.6, 9.4, 0.2},
                              {64, 2, 1.6, 3.1, 4.3, 5.8}};

// Launch time of `ctas` CTAs of a form on 148 SMs.  Without a causal mask (or with one key tile) all CTAs weigh the same:
// rounds.  Under a causal mask, heaviest first: no launch ends before its heaviest CTA, nor before the work is done, plus
// a part of a mean CTA for the uneven end.
double form_time(const Form& f, double tiles, double heads, int key_tiles, bool uneven) {
  const double ctas = tiles * heads;
  const int turns = (key_tiles + f.groups - 1) / f.groups;
  const double heaviest = f.cta + f.step * turns + f.tile * key_tiles;
  if (!uneven) return f.launch + ceil(ctas / 148.0) * heaviest;
  const double full = key_tiles / f.groups, part = key_tiles % f.groups;  // mean turns of 1 .. key_tiles tiles
  const double mean_turns = (f.groups * full * (full + 1) / 2 + part * (full + 1)) / key_tiles;
  const double mean = f.cta + f.step * mean_turns + f.tile * 0.5 * (key_tiles + (f.rows > BK ? f.rows / BK : 1));
  const double first = heaviest + (ctas > 148.0 ? f.cta : 0.0), work = ctas / 148.0 * mean + 0.3 * mean;
  return f.launch + (first > work ? first : work);
}
// The same for the plain form; at D = 64 an SM holds three of its CTAs (5.9 us per key tile for one, 9.2 for two, 13 for
// three).  Its tiles run in the order of their index, a causal launch ends on heavy ones.
double plain_time(double tiles, double heads, int key_tiles, bool uneven, int D) {
  const double ctas = tiles * heads;
  auto together = [D](double k, int n) {
    return D == 128 ? 2.2 + 9.0 * k : n == 1 ? 2.7 + 5.9 * k : n == 2 ? 3.2 + 9.2 * k : 4.0 + 13.0 * k;
  };
  if (D == 128 && !uneven) {  // (from the fifth round on a round takes a fifth longer: 200 heads of S=256 278 us, S=500 945)
    const double rounds = ceil(ctas / 148.0);
    return 1.0 + rounds * (rounds > 4.0 ? 1.2 : 1.0) * together(key_tiles, 1);
  }
  if (!uneven) {
    const double full = floor(ctas / 444.0);
    const int rest = (int)ceil((ctas - 444.0 * full) / 148.0);
    return 0.3 + full * together(key_tiles, 3) + (rest ? together(key_tiles, rest) : 0.0);
  }
  const int n = D == 128 || ctas <= 148.0 ? 1 : ctas <= 296.0 ? 2 : 3;
  const double heaviest = together(key_tiles, n), work = ctas / 148.0 * together(0.5 * (key_tiles + 1), n) / n + 0.75 * heaviest / n;
  return 0.3 + (ctas <= 148.0 || heaviest > work ? heaviest : work);  // (up to 148 all start at once)
}

}  // namespace

// The form that ends first by these estimates.  Over the measured shapes the choice lies 0.3 % on average above the best
// form and at most 2 % above the plain one, which used to serve every call.
ExactPlan exact_forward_plan(int B, int Hq, int S, int D, int causal) {
  const double heads = (double)B * Hq;
  const int key_tiles = (S + BK - 1) / BK;
  const bool uneven = causal && key_tiles > 1;
  ExactPlan p{PLAIN_BQ, 1};
  double least = plain_time((S + PLAIN_BQ - 1) / PLAIN_BQ, heads, key_tiles, uneven, D);
  auto offer = [&](const Form& f) {
    const double t = form_time(f, (S + f.rows - 1) / f.rows, heads, key_tiles, uneven);
    if (t < least) {
      least = t;
      p = ExactPlan{f.rows, 0};
    }
  };
  if (D == 64)
    for (const Form& f : FORMS_64) offer(f);
  else
    for (const Form& f : FORMS_128) offer(f);
  return p;
}

cudaError_t launch_attn_exact(const ExactArgs& a, cudaStream_t stream) {
  if (a.D != 64 && a.D != 128) return cudaErrorInvalidValue;
  const ExactPlan p = exact_forward_plan(a.B, a.Hq, a.S, a.D, a.causal);
  if (p.plain) return a.D == 64 ? launch_exact_plain<64>(a, stream) : launch_exact_plain<128>(a, stream);
#define AR_EXACT(D_, G_)                                         \
  if (a.D == D_) {                                               \
    switch (p.rows) {                                            \
      case 8: return launch_exact<D_, 2, 16, 4, G_>(a, stream);  \
      case 12: return launch_exact<D_, 3, 16, 4, G_>(a, stream); \
      case 16: return launch_exact<D_, 4, 16, 4, G_>(a, stream); \
      case 20: return launch_exact<D_, 5, 16, 4, G_>(a, stream); \
      case 24: return launch_exact<D_, 6, 16, 4, G_>(a, stream); \
      case 32: return launch_exact<D_, 8, 16, 4, G_>(a, stream); \
      case 64: return launch_exact<D_, 4, 8, 16, 2>(a, stream);  \
      default: return launch_exact<64, 8, 8, 16, 2>(a, stream);  \
    }                                                            \
  }
  AR_EXACT(64, 4)
  AR_EXACT(128, 2)
#undef AR_EXACT
  return cudaErrorInvalidValue;
}

}  // namespace ar
