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

template <int D, int RQ, int TX, int TY, int GROUPS>
__global__ void __launch_bounds__(TX* TY* GROUPS, 1)
    attn_fwd_exact_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                          float* __restrict__ O, const float* __restrict__ M, float* __restrict__ LSE, int N, int Hq,
                          int Hkv, int grouped, int causal) {
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
    // mask a row counts them up to the end of the 64 keys its diagonal lies in; a tile that reaches further gives them
    // no weight, so that such a row has the same value whatever tile height its call takes.
    const bool bounds = k0 + BK > N || (causal && k0 + BK - 1 > q0);
#pragma unroll
    for (int i = 0; i < RQ; i++) {
      const int row = q0 + ty + TY * i;
      float mx = m[i];
#pragma unroll
      for (int jj = 0; jj < JK; jj++) {
        const int key = k0 + tx + TX * jj;
        float x = s[i][jj] * scale;
        if (M != nullptr && row < N && key < N) x += M[(size_t)row * N + key];
        if (bounds && (key >= N || (causal && key > row))) x = causal && k0 > row ? -INFINITY : NEG;
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
  auto kern = attn_fwd_exact_kernel<D, RQ, TX, TY, GROUPS>;
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const CtaGrid g = cta_grid((size_t)a.S * D * 8 / (size_t)(a.Hq / a.Hkv), a.B * a.Hq, (a.S + C::BQ - 1) / C::BQ,
                             a.causal ? CAUSAL_TILES : a.S % C::BQ != 0);
  kern<<<g.grid, C::THREADS, C::SMEM_BYTES, stream>>>(a.q, a.k, a.v, a.out, a.mask, a.lse, a.S, a.Hq, a.Hkv, g.grouped,
                                                     a.causal);
  return cudaGetLastError();
}

// D = 64 without a causal mask, for calls whose tiles of 128 rows would leave a last round half empty: 4 x 4 scores per
// thread on 64 rows, plain loads, two CTAs per SM that fill each other's waits.
constexpr int PAIR_BQ = 64;
constexpr int PAIR_SMEM = (PAIR_BQ * 68 + BK * 68 + BK * 64 + PAIR_BQ * (BK + 4)) * 4;
__global__ void __launch_bounds__(256) attn_fwd_exact_pair_kernel(const float* __restrict__ Q, const float* __restrict__ K,
                                                             const float* __restrict__ V, float* __restrict__ O,
                                                             const float* __restrict__ M, float* __restrict__ LSE,
                                                             int N, int Hq, int Hkv, int causal) {
  constexpr int D = 64, LDQ = D + 4, LDP = BK + 4;  // padded rows (floats)
  extern __shared__ __align__(16) float smem_f[];
  float* sQ = smem_f;
  float* sK = sQ + PAIR_BQ * LDQ;
  float* sV = sK + BK * LDQ;
  float* sP = sV + BK * D;
  const int tid = threadIdx.x;
  const int tx = tid & 15;
  const int ty = tid >> 4;
  const int bh = blockIdx.y;
  const int b = bh / Hq;
  const int h = bh - b * Hq;
  const int kvbh = b * Hkv + h / (Hq / Hkv);
  const int q0 = blockIdx.x * PAIR_BQ;
  const float* qb = Q + (size_t)bh * N * D;
  const float* kb = K + (size_t)kvbh * N * D;
  const float* vb = V + (size_t)kvbh * N * D;
  const float scale = 1.0f / sqrtf((float)D);
  constexpr int D4 = D / 4;
  constexpr int OD = D / 64;  // float4 output groups per thread

  for (int i = tid; i < PAIR_BQ * D4; i += 256) {
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
  const int kend = causal ? min(N, q0 + PAIR_BQ) : N;
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

cudaError_t launch_exact_pair(const ExactArgs& a, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(attn_fwd_exact_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  attn_fwd_exact_pair_kernel<<<dim3((a.S + PAIR_BQ - 1) / PAIR_BQ, a.B * a.Hq, 1), 256, PAIR_SMEM, stream>>>(
      a.q, a.k, a.v, a.out, a.mask, a.lse, a.S, a.Hq, a.Hkv, a.causal);
  return cudaGetLastError();
}

// What a launch with tiles of `rows` rows costs, in rows of the large form: rounds of one CTA per SM -- under a causal
// mask the average tile sees half of the keys and the rounds overlap, but none ends before its heaviest tile -- each as
// long as its rows plus the part of a CTA that does not depend on them (loads, softmax, combination: about 8 rows).
double launch_cost(const ExactArgs& a, int rows) {
  const double ctas = (double)((a.S + rows - 1) / rows) * a.B * a.Hq;
  const double rounds = a.causal ? fmax(1.0, 0.55 * ctas / 148.0) : ceil(ctas / 148.0);
  return rounds * (rows + 8);
}

}  // namespace

cudaError_t launch_attn_exact(const ExactArgs& a, cudaStream_t stream) {
  // The form that ends first.  Weights per row of a round, measured at S = 197 to 1024: 1 for the large form, 1.6 for the
  // tiles of 8 to 32 rows that spread a small call over the chip, at D = 64 also 1.11 for 4 x 8 blocks on 64 rows, and
  // for the 64-row form with two CTAs per SM 105 rows alone, 150 in pairs, 45.5 per half round beyond, the last one included
  // (B=6 Hq=4 S=848: 189 us against 199 with 4 x 8 blocks; B=2 H=8 S=1024: 152 against 135 in the large form).
  const int large = a.D == 64 ? 128 : 64;
  int rows = large;
  double cost = launch_cost(a, large);
  auto offer = [&](int r, double c) {
    if (c < cost) {
      rows = r;
      cost = c;
    }
  };
  for (int r : {8, 12, 16, 20, 24, 32}) offer(r, 1.6 * launch_cost(a, r));
  if (a.D == 64) offer(64, 1.11 * launch_cost(a, 64));
  if (a.D == 64 && !a.causal) {
    const double ctas = (double)((a.S + 63) / 64) * a.B * a.Hq;
    offer(-64, ctas <= 148 ? 105.0 : ctas <= 296 ? 150.0 : 45.5 * 2.0 * ctas / 148.0);
  }
  if (rows == -64) return launch_exact_pair(a, stream);
#define AR_EXACT(D_, G_)                                         \
  if (a.D == D_) {                                               \
    switch (rows) {                                              \
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
