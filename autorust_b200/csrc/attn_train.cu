// Backward of the exact f32 attention: dQ, dK, dV from the saved log-sum-exp.
//
// Replaces autorust's `ar_fl_prep`, `ar_fl_bwd_dq` and `ar_fl_bwd_dkv`
// (src/runtime/cuda_flash_train.rs:118-309; the forward with LSE, `ar_fl_fwd` :49-117, is the exact forward kernel of
// attn_fwd_exact.cu with its LSE output on).  Same math, no atomics, deterministic order:
//   s = (q.k) / sqrt(D) (+ mask), key >= S or (causal and key > row) excluded, p = exp(s - LSE),
//   D_i = O_i . dO_i,  dS = p (dO.v - D_i),  dQ_i = sum_j dS_ij k_j / sqrt(D),
//   dK_j = sum_i dS_ij q_i / sqrt(D),  dV_j = sum_i p_ij dO_i, the last two summed over the query heads of a GQA group.
// The reference runs one thread per row with 32-wide tiles; here a CTA of 256 threads owns a 64 x 64 tile of the score
// matrix, every thread a 4 x 4 block of it (rows ty*4+i, keys tx+16*jj, as in the forward) for the two products that
// rebuild p and dS, and a 4 x D/16 block of the gradient tile for the product that accumulates it.  f32 on the FFMA
// pipe throughout: this is the path held to the graph's autograd, not a tensor-core path.
// At D = 64, where the tiles of 128 rows fit, calls with enough rows take the kernels with 8 x 8 blocks per thread (the
// _wide ones): four d of a 4 x 4 block read 8 x 16 bytes of shared memory per thread (32 cycles per warp and SM) for 16
// cycles of FFMA, an 8 x 8 block 64 for 64.
#include "ar_kernels.h"
#include "ar_ptx.cuh"
#include "cta_order.cuh"

namespace ar {
namespace {

constexpr int BT = 64;  // tile edge: queries and keys

// delta[bh, i] = O_i . dO_i: one warp per row
__global__ void __launch_bounds__(256) train_prep_kernel(const float* __restrict__ O, const float* __restrict__ dO,
                                                         float* __restrict__ delta, long long rows, int D) {
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
  for (int d = lane * 4; d < D; d += 128) {
    const float4 a = *(const float4*)(O + row * D + d);
    const float4 b = *(const float4*)(dO + row * D + d);
    acc = fmaf(a.x, b.x, acc);
    acc = fmaf(a.y, b.y, acc);
    acc = fmaf(a.z, b.z, acc);
    acc = fmaf(a.w, b.w, acc);
  }
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
  if (lane == 0) delta[row] = acc;
}

template <int D>
struct BwdCfg {
  static constexpr int LD = D + 4;   // padded row (floats): 16-byte aligned, conflict-free float4 reads
  static constexpr int LDP = BT + 4;
  static constexpr int DQ_SMEM = (4 * BT * LD + BT * LDP + 2 * BT) * 4;            // Q, dO, K, V, dS, lse, delta
  static constexpr int DKV_SMEM = (4 * BT * LD + 2 * BT * LDP + 2 * BT) * 4;      // K, V, Q, dO, P, dS, lse, delta
};

// Loads `rows` x D floats (rows past N zero-filled) into a padded shared tile.
template <int D>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int row0, int N, int tid) {
  constexpr int D4 = D / 4;
  for (int i = tid; i < BT * D4; i += 256) {
    const int r = i / D4, c = i - r * D4;
    float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row0 + r < N) v4 = *(const float4*)(src + (size_t)(row0 + r) * D + c * 4);
    *(float4*)(dst + r * BwdCfg<D>::LD + c * 4) = v4;
  }
}

// The 4 x 4 block of two products over d at once: s = A.B^T (rows of sA against rows of sB) and t = C.E^T.
template <int D>
__device__ __forceinline__ void two_products(const float* sA, const float* sB, const float* sC, const float* sE, int ty,
                                             int tx, float (&s)[4][4], float (&t)[4][4]) {
  constexpr int LD = BwdCfg<D>::LD;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int jj = 0; jj < 4; jj++) s[i][jj] = t[i][jj] = 0.f;
#pragma unroll 2
  for (int d4 = 0; d4 < D / 4; d4++) {
    float4 a[4], b[4], c[4], e[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      a[i] = *(const float4*)(sA + (ty * 4 + i) * LD + d4 * 4);
      c[i] = *(const float4*)(sC + (ty * 4 + i) * LD + d4 * 4);
    }
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      b[jj] = *(const float4*)(sB + (tx + 16 * jj) * LD + d4 * 4);
      e[jj] = *(const float4*)(sE + (tx + 16 * jj) * LD + d4 * 4);
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        s[i][jj] = fmaf(a[i].x, b[jj].x, s[i][jj]);
        s[i][jj] = fmaf(a[i].y, b[jj].y, s[i][jj]);
        s[i][jj] = fmaf(a[i].z, b[jj].z, s[i][jj]);
        s[i][jj] = fmaf(a[i].w, b[jj].w, s[i][jj]);
        t[i][jj] = fmaf(c[i].x, e[jj].x, t[i][jj]);
        t[i][jj] = fmaf(c[i].y, e[jj].y, t[i][jj]);
        t[i][jj] = fmaf(c[i].z, e[jj].z, t[i][jj]);
        t[i][jj] = fmaf(c[i].w, e[jj].w, t[i][jj]);
      }
  }
}

// p and dS of one element from its raw products (s = q.k, t = dO.v).
__device__ __forceinline__ void p_and_ds(float s, float t, float scale, const float* __restrict__ M, int row, int key, int N,
                                         int causal, float lse, float delta, float& p, float& ds) {
  float x = s * scale;
  if (M != nullptr && row < N && key < N) x += M[(size_t)row * N + key];
  const bool out = key >= N || row >= N || (causal && key > row);
  p = out ? 0.f : expf(x - lse);
  ds = p * (t - delta);
}

// dQ: one CTA per (64 queries, batch x head); walks the keys 64 at a time.  (GROUPED: cta_order.cuh; known at compile time,
// as the plain form spills with the choice in it, 2 % at D = 128.)
template <int D, bool GROUPED>
__global__ void __launch_bounds__(256) train_dq_kernel(const float* __restrict__ Q, const float* __restrict__ K,
                                                       const float* __restrict__ V, const float* __restrict__ dO,
                                                       const float* __restrict__ LSE, const float* __restrict__ delta,
                                                       const float* __restrict__ M, float* __restrict__ dQ, int N, int Hq,
                                                       int Hkv, int causal) {
  using C = BwdCfg<D>;
  extern __shared__ __align__(16) float smem_t[];
  float* sQ = smem_t;
  float* sdO = sQ + BT * C::LD;
  float* sK = sdO + BT * C::LD;
  float* sV = sK + BT * C::LD;
  float* sDS = sV + BT * C::LD;
  float* sL = sDS + BT * C::LDP;
  float* sDl = sL + BT;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int bh = cta_head(GROUPED);
  int tile = cta_tile(GROUPED);
  if (GROUPED && causal) tile = cta_tiles(GROUPED) - 1 - tile;  // the last query tile sees the most keys
  const int b = bh / Hq, h = bh - b * Hq;
  const int kvbh = b * Hkv + h / (Hq / Hkv);
  const int q0 = tile * BT;
  const float scale = 1.0f / sqrtf((float)D);
  constexpr int OD = D / 64;
  load_tile<D>(sQ, Q + (size_t)bh * N * D, q0, N, tid);
  load_tile<D>(sdO, dO + (size_t)bh * N * D, q0, N, tid);
  if (tid < BT) {
    sL[tid] = q0 + tid < N ? LSE[(size_t)bh * N + q0 + tid] : 0.f;
    sDl[tid] = q0 + tid < N ? delta[(size_t)bh * N + q0 + tid] : 0.f;
  }
  float4 acc[4][OD];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int dd = 0; dd < OD; dd++) acc[i][dd] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int kend = causal ? min(N, q0 + BT) : N;
  for (int k0 = 0; k0 < kend; k0 += BT) {
    __syncthreads();  // the previous tile is consumed (and Q, dO, lse, delta are visible on the first pass)
    load_tile<D>(sK, K + (size_t)kvbh * N * D, k0, N, tid);
    load_tile<D>(sV, V + (size_t)kvbh * N * D, k0, N, tid);
    __syncthreads();
    float s[4][4], t[4][4];
    two_products<D>(sQ, sK, sdO, sV, ty, tx, s, t);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        float p, ds;
        p_and_ds(s[i][jj], t[i][jj], scale, M, q0 + ty * 4 + i, k0 + tx + 16 * jj, N, causal, sL[ty * 4 + i],
                 sDl[ty * 4 + i], p, ds);
        sDS[(ty * 4 + i) * C::LDP + tx + 16 * jj] = ds;
      }
    __syncthreads();
    // dQ block: rows ty*4+i, columns tx*4 + 64*dd:  dQ += dS . K
#pragma unroll 4
    for (int k4 = 0; k4 < BT / 4; k4++) {
      float4 dsv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) dsv[i] = *(const float4*)(sDS + (ty * 4 + i) * C::LDP + k4 * 4);
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
#pragma unroll
        for (int dd = 0; dd < OD; dd++) {
          const float4 k4v = *(const float4*)(sK + (k4 * 4 + kk) * C::LD + tx * 4 + 64 * dd);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float w = kk == 0 ? dsv[i].x : kk == 1 ? dsv[i].y : kk == 2 ? dsv[i].z : dsv[i].w;
            acc[i][dd].x = fmaf(w, k4v.x, acc[i][dd].x);
            acc[i][dd].y = fmaf(w, k4v.y, acc[i][dd].y);
            acc[i][dd].z = fmaf(w, k4v.z, acc[i][dd].z);
            acc[i][dd].w = fmaf(w, k4v.w, acc[i][dd].w);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = q0 + ty * 4 + i;
    if (row >= N) continue;
    float* dst = dQ + ((size_t)bh * N + row) * D;
#pragma unroll
    for (int dd = 0; dd < OD; dd++)
      *(float4*)(dst + tx * 4 + 64 * dd) =
          make_float4(acc[i][dd].x * scale, acc[i][dd].y * scale, acc[i][dd].z * scale, acc[i][dd].w * scale);
  }
}

// dK, dV: one CTA per (64 keys, batch x kv head); walks the query heads of the group and their query tiles in a
// fixed order, so the sums have one writer and one order.
template <int D, bool GROUPED>
__global__ void __launch_bounds__(256) train_dkv_kernel(const float* __restrict__ Q, const float* __restrict__ K,
                                                        const float* __restrict__ V, const float* __restrict__ dO,
                                                        const float* __restrict__ LSE, const float* __restrict__ delta,
                                                        const float* __restrict__ M, float* __restrict__ dK,
                                                        float* __restrict__ dV, int N, int Hq, int Hkv, int causal) {
  using C = BwdCfg<D>;
  extern __shared__ __align__(16) float smem_t[];
  float* sK = smem_t;
  float* sV = sK + BT * C::LD;
  float* sQ = sV + BT * C::LD;
  float* sdO = sQ + BT * C::LD;
  float* sP = sdO + BT * C::LD;
  float* sDS = sP + BT * C::LDP;
  float* sL = sDS + BT * C::LDP;
  float* sDl = sL + BT;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kvbh = GROUPED ? cta_head(1) : blockIdx.y;
  const int b = kvbh / Hkv, hk = kvbh - b * Hkv;
  const int group = Hq / Hkv;
  const int k0 = (GROUPED ? blockIdx.y : blockIdx.x) * BT;  // (under a causal mask the first key tile sees the most queries)
  const float scale = 1.0f / sqrtf((float)D);
  constexpr int OD = D / 64;
  load_tile<D>(sK, K + (size_t)kvbh * N * D, k0, N, tid);
  load_tile<D>(sV, V + (size_t)kvbh * N * D, k0, N, tid);
  float4 ak[4][OD], av[4][OD];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int dd = 0; dd < OD; dd++) ak[i][dd] = av[i][dd] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int q_first = causal ? k0 : 0;  // under a causal mask the queries before this key tile see none of it
  for (int g = 0; g < group; g++) {
    const int bh = b * Hq + hk * group + g;
    for (int q0 = q_first; q0 < N; q0 += BT) {
      __syncthreads();  // the previous query tile is consumed (and K, V are visible on the first pass)
      load_tile<D>(sQ, Q + (size_t)bh * N * D, q0, N, tid);
      load_tile<D>(sdO, dO + (size_t)bh * N * D, q0, N, tid);
      if (tid < BT) {
        sL[tid] = q0 + tid < N ? LSE[(size_t)bh * N + q0 + tid] : 0.f;
        sDl[tid] = q0 + tid < N ? delta[(size_t)bh * N + q0 + tid] : 0.f;
      }
      __syncthreads();
      float s[4][4], t[4][4];
      two_products<D>(sQ, sK, sdO, sV, ty, tx, s, t);  // rows: queries ty*4+i, columns: keys tx+16*jj
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
          float p, ds;
          p_and_ds(s[i][jj], t[i][jj], scale, M, q0 + ty * 4 + i, k0 + tx + 16 * jj, N, causal, sL[ty * 4 + i],
                   sDl[ty * 4 + i], p, ds);
          sP[(ty * 4 + i) * C::LDP + tx + 16 * jj] = p;
          sDS[(ty * 4 + i) * C::LDP + tx + 16 * jj] = ds;
        }
      __syncthreads();
      // gradient blocks: keys ty*4+i, columns tx*4 + 64*dd:  dV += P^T . dO,  dK += dS^T . Q
#pragma unroll 4
      for (int qi = 0; qi < BT; qi++) {
        const float4 pv = *(const float4*)(sP + qi * C::LDP + ty * 4);
        const float4 dsv = *(const float4*)(sDS + qi * C::LDP + ty * 4);
#pragma unroll
        for (int dd = 0; dd < OD; dd++) {
          const float4 do4 = *(const float4*)(sdO + qi * C::LD + tx * 4 + 64 * dd);
          const float4 q4 = *(const float4*)(sQ + qi * C::LD + tx * 4 + 64 * dd);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float wp = i == 0 ? pv.x : i == 1 ? pv.y : i == 2 ? pv.z : pv.w;
            const float wd = i == 0 ? dsv.x : i == 1 ? dsv.y : i == 2 ? dsv.z : dsv.w;
            av[i][dd].x = fmaf(wp, do4.x, av[i][dd].x);
            av[i][dd].y = fmaf(wp, do4.y, av[i][dd].y);
            av[i][dd].z = fmaf(wp, do4.z, av[i][dd].z);
            av[i][dd].w = fmaf(wp, do4.w, av[i][dd].w);
            ak[i][dd].x = fmaf(wd, q4.x, ak[i][dd].x);
            ak[i][dd].y = fmaf(wd, q4.y, ak[i][dd].y);
            ak[i][dd].z = fmaf(wd, q4.z, ak[i][dd].z);
            ak[i][dd].w = fmaf(wd, q4.w, ak[i][dd].w);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int key = k0 + ty * 4 + i;
    if (key >= N) continue;
    float* dk = dK + ((size_t)kvbh * N + key) * D;
    float* dv = dV + ((size_t)kvbh * N + key) * D;
#pragma unroll
    for (int dd = 0; dd < OD; dd++) {
      *(float4*)(dk + tx * 4 + 64 * dd) =
          make_float4(ak[i][dd].x * scale, ak[i][dd].y * scale, ak[i][dd].z * scale, ak[i][dd].w * scale);
      *(float4*)(dv + tx * 4 + 64 * dd) = av[i][dd];
    }
  }
}

// ---------------------------------------------------------------- D = 64, 8 x 8 blocks
namespace wide {
using namespace arptx;
constexpr int D = 64, LD = D + 4;  // padded row (floats): 16-byte aligned, conflict-free float4 reads
constexpr int OWN = 128;           // rows a CTA owns
constexpr int STREAM = 64;         // rows of a streamed tile
constexpr int LDS_DQ = STREAM + 8;    // dS row of the dQ kernel: a warp's 4 rows x 8 keys fall into different banks
constexpr int LDS_DKV = OWN + 16;     // P and dS rows of the dK/dV kernel: 2 rows x 16 keys
constexpr int DQ_GROUP = 2 * STREAM * LD + OWN * LDS_DQ;  // floats: K, V, dS of one group
constexpr int DQ_SMEM = (2 * OWN * LD + 2 * DQ_GROUP) * 4;
constexpr int DKV_STAGE = 2 * STREAM * LD + 2 * STREAM;   // Q, dO, LSE, D_i of one query tile
constexpr int DKV_SMEM = (2 * OWN * LD + 2 * DKV_STAGE + 2 * STREAM * LDS_DKV) * 4;
static_assert(DQ_SMEM <= 227 * 1024 && DKV_SMEM <= 227 * 1024, "shared memory budget");
static_assert(128 * 64 <= DQ_GROUP, "a group's dQ passes through its own tiles");

// `rows` rows of a [.., N, D] tensor into a padded tile by `threads` threads; rows past the end become zeros
__device__ __forceinline__ void load_async(float* dst, const float* src, int rows, int row0, int N, int t, int threads) {
#pragma unroll 4
  for (int i = t; i < rows * (D / 4); i += threads) {
    const int r = i / (D / 4), c = i % (D / 4);
    const bool in = row0 + r < N;
    cp_async16(smem_u32(dst + r * LD + c * 4), in ? src + (size_t)(row0 + r) * D + c * 4 : src, in);
  }
}

// s[i][jj] = A[(ra + RA * i)] . B[(rb + RB * jj)] over d
template <int RA, int RB>
__device__ __forceinline__ void product(const float* sA, const float* sB, int ra, int rb, float (&s)[8][8]) {
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int jj = 0; jj < 8; jj++) s[i][jj] = 0.f;
#pragma unroll 1
  for (int d4 = 0; d4 < D / 4; d4++) {
    float4 bv[8];
#pragma unroll
    for (int jj = 0; jj < 8; jj++) bv[jj] = *(const float4*)(sB + (rb + RB * jj) * LD + d4 * 4);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float4 av = *(const float4*)(sA + (ra + RA * i) * LD + d4 * 4);
#pragma unroll
      for (int jj = 0; jj < 8; jj++) {
        s[i][jj] = fmaf(av.x, bv[jj].x, s[i][jj]);
        s[i][jj] = fmaf(av.y, bv[jj].y, s[i][jj]);
        s[i][jj] = fmaf(av.z, bv[jj].z, s[i][jj]);
        s[i][jj] = fmaf(av.w, bv[jj].w, s[i][jj]);
      }
    }
  }
}

// p of one element from its raw product
__device__ __forceinline__ float prob(float s, float scale, const float* __restrict__ M, int row, int key, int N, int causal,
                                      float lse) {
  float x = s * scale;
  if (M != nullptr && row < N && key < N) x += M[(size_t)row * N + key];
  return key >= N || row >= N || (causal && key > row) ? 0.f : expf(x - lse);
}

// dQ: one CTA per (128 queries, batch x head); two groups of 128 threads take the key tiles of 64 in turn, each with a
// dQ of its own (8 rows x 8 columns per thread); group 0 adds the two.
__global__ void __launch_bounds__(256, 1)
    train_dq_wide_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                         const float* __restrict__ dO, const float* __restrict__ LSE, const float* __restrict__ delta,
                         const float* __restrict__ M, float* __restrict__ dQ, int N, int Hq, int Hkv, int grouped,
                         int causal) {
  extern __shared__ __align__(16) float smem_t[];
  const int tid = threadIdx.x, grp = tid >> 7, gt = tid & 127;
  const int tx = gt & 7, ty = gt >> 3;  // rows ty + 16 * i, keys tx + 8 * jj, columns (tx + 8 * dd) * 4 ..
  float* sQ = smem_t;
  float* sdO = sQ + OWN * LD;
  float* sK = sdO + OWN * LD + grp * DQ_GROUP;
  float* sV = sK + STREAM * LD;
  float* sDS = sV + STREAM * LD;
  const int bh = cta_head(grouped);
  int tile = cta_tile(grouped);
  if (causal) tile = cta_tiles(grouped) - 1 - tile;  // the last query tile sees the most keys
  const int b = bh / Hq, h = bh - b * Hq;
  const size_t kv = (size_t)(b * Hkv + h / (Hq / Hkv)) * N * D;
  const int q0 = tile * OWN;
  const float scale = 1.0f / sqrtf((float)D);
  const int tiles = ((causal ? min(N, q0 + OWN) : N) + STREAM - 1) / STREAM;
  load_async(sQ, Q + (size_t)bh * N * D, OWN, q0, N, tid, 256);
  load_async(sdO, dO + (size_t)bh * N * D, OWN, q0, N, tid, 256);
  load_async(sK, K + kv, STREAM, grp * STREAM, N, gt, 128);
  load_async(sV, V + kv, STREAM, grp * STREAM, N, gt, 128);
  cp_async_commit();
  float lse[8], dl[8], acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int row = q0 + ty + 16 * i;
    lse[i] = row < N ? LSE[(size_t)bh * N + row] : 0.f;
    dl[i] = row < N ? delta[(size_t)bh * N + row] : 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) acc[i][c] = 0.f;
  }
  auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
  cp_async_wait<0>();
  __syncthreads();
  for (int kt = grp; kt < tiles; kt += 2) {
    const int k0 = kt * STREAM;
    cp_async_wait<0>();
    group_sync();
    float p[8][8], t[8][8];
    product<16, 8>(sQ, sK, ty, tx, p);
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int jj = 0; jj < 8; jj++)
        p[i][jj] = prob(p[i][jj], scale, M, q0 + ty + 16 * i, k0 + tx + 8 * jj, N, causal, lse[i]);
    product<16, 8>(sdO, sV, ty, tx, t);
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int jj = 0; jj < 8; jj++) sDS[(ty + 16 * i) * LDS_DQ + tx + 8 * jj] = p[i][jj] * (t[i][jj] - dl[i]);
    group_sync();  // dS is complete and V consumed
    load_async(sV, V + kv, STREAM, min(k0 + 2 * STREAM, N), N, gt, 128);
    cp_async_commit();
    // dQ += dS . K
#pragma unroll 2
    for (int k4 = 0; k4 < STREAM / 4; k4++) {
      float4 kr[4][2];
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
#pragma unroll
        for (int dd = 0; dd < 2; dd++) kr[kk][dd] = *(const float4*)(sK + (k4 * 4 + kk) * LD + (tx + 8 * dd) * 4);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float4 ds = *(const float4*)(sDS + (ty + 16 * i) * LDS_DQ + k4 * 4);
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
          const float w = kk == 0 ? ds.x : kk == 1 ? ds.y : kk == 2 ? ds.z : ds.w;
#pragma unroll
          for (int dd = 0; dd < 2; dd++) {
            acc[i][dd * 4 + 0] = fmaf(w, kr[kk][dd].x, acc[i][dd * 4 + 0]);
            acc[i][dd * 4 + 1] = fmaf(w, kr[kk][dd].y, acc[i][dd * 4 + 1]);
            acc[i][dd * 4 + 2] = fmaf(w, kr[kk][dd].z, acc[i][dd * 4 + 2]);
            acc[i][dd * 4 + 3] = fmaf(w, kr[kk][dd].w, acc[i][dd * 4 + 3]);
          }
        }
      }
    }
    group_sync();  // K and dS are consumed
    load_async(sK, K + kv, STREAM, min(k0 + 2 * STREAM, N), N, gt, 128);
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncthreads();
  float* mine = sK + gt;
  if (grp == 1) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int c = 0; c < 8; c++) mine[(i * 8 + c) * 128] = acc[i][c];
  }
  __syncthreads();
  if (grp == 1) return;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int row = q0 + ty + 16 * i;
    if (row >= N) continue;
    const float* other = mine + DQ_GROUP + i * 8 * 128;
#pragma unroll
    for (int dd = 0; dd < 2; dd++)
      *(float4*)(dQ + ((size_t)bh * N + row) * D + (tx + 8 * dd) * 4) =
          make_float4((acc[i][dd * 4 + 0] + other[(dd * 4 + 0) * 128]) * scale, (acc[i][dd * 4 + 1] + other[(dd * 4 + 1) * 128]) * scale,
                      (acc[i][dd * 4 + 2] + other[(dd * 4 + 2) * 128]) * scale, (acc[i][dd * 4 + 3] + other[(dd * 4 + 3) * 128]) * scale);
  }
}

// dK, dV: one CTA per (128 keys, batch x kv head), walking the query tiles of 64 of every query head of the group in a
// fixed order.  Threads 0-127 rebuild p and accumulate dV = P^T dO, threads 128-255 form dS from their dO.V and that p
// and accumulate dK = dS^T Q, so that each holds one 8 x 8 block of scores and one of gradients.  The next query tile
// arrives under this one's products.
__global__ void __launch_bounds__(256, 1)
    train_dkv_wide_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                          const float* __restrict__ dO, const float* __restrict__ LSE, const float* __restrict__ delta,
                          const float* __restrict__ M, float* __restrict__ dK, float* __restrict__ dV, int N, int Hq, int Hkv,
                          int grouped, int causal) {
  extern __shared__ __align__(16) float smem_t[];
  const int tid = threadIdx.x, half = tid >> 7, ht = tid & 127;
  const int tx = ht & 15, ty = ht >> 4;  // scores: queries ty + 8 * i, keys tx + 16 * jj
  const int cx = ht & 7, ky = ht >> 3;   // gradients: keys ky * 8 + i, columns (cx + 8 * dd) * 4 ..
  float* sK = smem_t;
  float* sV = sK + OWN * LD;
  float* stages = sV + OWN * LD;
  float* sP = stages + 2 * DKV_STAGE;
  float* sDS = sP + STREAM * LDS_DKV;
  const int kvbh = cta_head(grouped);
  const int tile = cta_tile(grouped);  // (under a causal mask the first key tile sees the most queries)
  const int b = kvbh / Hkv, hk = kvbh - b * Hkv, group = Hq / Hkv;
  const int k0 = tile * OWN;
  const float scale = 1.0f / sqrtf((float)D);
  const int first = causal ? k0 / STREAM : 0;  // queries before the key tile see none of it
  const int per_head = (N + STREAM - 1) / STREAM - first;
  const int steps = group * per_head;
  auto load_step = [&](int n) {
    if (n < steps) {
      const int g = n / per_head, r0 = (first + n - g * per_head) * STREAM;
      const size_t bh = (size_t)(b * Hq + hk * group + g);
      float* st = stages + (n & 1) * DKV_STAGE;
      load_async(st, Q + bh * N * D, STREAM, r0, N, tid, 256);
      load_async(st + STREAM * LD, dO + bh * N * D, STREAM, r0, N, tid, 256);
      if (tid < 2 * STREAM) {
        const int r = r0 + (tid & (STREAM - 1));
        const float* src = tid < STREAM ? LSE : delta;
        cp_async4(smem_u32(st + 2 * STREAM * LD + tid), r < N ? src + bh * N + r : src, r < N);
      }
    }
    cp_async_commit();
  };
  load_async(sK, K + (size_t)kvbh * N * D, OWN, k0, N, tid, 256);
  load_async(sV, V + (size_t)kvbh * N * D, OWN, k0, N, tid, 256);
  load_step(0);
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int c = 0; c < 8; c++) acc[i][c] = 0.f;
  for (int n = 0; n < steps; n++) {
    load_step(n + 1);
    cp_async_wait<1>();
    __syncthreads();  // this step's tiles (and K, V) are in place
    const int g = n / per_head, q0 = (first + n - g * per_head) * STREAM;
    const float* sQ = stages + (n & 1) * DKV_STAGE;
    const float* sdO = sQ + STREAM * LD;
    const float* sL = sdO + STREAM * LD;
    float s[8][8];
    product<8, 16>(half ? sdO : sQ, half ? sV : sK, ty, tx, s);
    if (half == 0) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int jj = 0; jj < 8; jj++)
          sP[(ty + 8 * i) * LDS_DKV + tx + 16 * jj] =
              prob(s[i][jj], scale, M, q0 + ty + 8 * i, k0 + tx + 16 * jj, N, causal, sL[ty + 8 * i]);
    }
    __syncthreads();  // P is in place
    if (half == 1) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int jj = 0; jj < 8; jj++) {
          const int at = (ty + 8 * i) * LDS_DKV + tx + 16 * jj;
          sDS[at] = sP[at] * (s[i][jj] - sL[STREAM + ty + 8 * i]);
        }
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    const float* sW = half ? sDS : sP;
    const float* sX = half ? sQ : sdO;
#pragma unroll 4
    for (int q = 0; q < STREAM; q++) {
      const float4 w0 = *(const float4*)(sW + q * LDS_DKV + ky * 8), w1 = *(const float4*)(sW + q * LDS_DKV + ky * 8 + 4);
      const float4 x0 = *(const float4*)(sX + q * LD + cx * 4), x1 = *(const float4*)(sX + q * LD + (cx + 8) * 4);
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int c = 0; c < 8; c++) acc[i][c] = fmaf(w[i], x[c], acc[i][c]);
    }
    __syncthreads();  // this step's tiles, P and dS are consumed
  }
  cp_async_wait<0>();
  float* out = half ? dK : dV;
  const float f = half ? scale : 1.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int key = k0 + ky * 8 + i;
    if (key >= N) continue;
#pragma unroll
    for (int dd = 0; dd < 2; dd++)
      *(float4*)(out + ((size_t)kvbh * N + key) * D + (cx + 8 * dd) * 4) =
          make_float4(acc[i][dd * 4] * f, acc[i][dd * 4 + 1] * f, acc[i][dd * 4 + 2] * f, acc[i][dd * 4 + 3] * f);
  }
}

cudaError_t configure() {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || (dev < 64 && configured[dev])) return e;
  e = cudaFuncSetAttribute(train_dq_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(train_dkv_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DKV_SMEM);
  if (e == cudaSuccess && dev < 64) configured[dev] = true;
  return e;
}

// The 128-row tiles do their rows about 5 % faster than the 64-row ones, of which an SM holds two: the form whose
// rounds come to fewer rows per SM (B=6 Hq=4 S=848: dQ 2 x 128 against 3 x 64, a step 7 % slower in the wide form).
// Under a causal mask, where rounds overlap, it is the rows altogether that count (352 heads of S=405, of which 128-row tiles
// walk 512: 1700 us the training step, 1625 with 64 rows), and they want more than four rounds: their heaviest tiles, twice as long, end the launch (96 heads of
// S=700: 764 us against 702 with 64 rows; 96 of S=848, 4.5 rounds: 1110 against 1230).
bool worth_it(int S, int heads, int causal) {
  const long long w = (long long)((S + 127) / 128) * heads, n = (long long)((S + 63) / 64) * heads;
  if (causal) return w > 4 * 148 + 74 && w * 128 * 20 <= n * 64 * 21;
  return ((w + 147) / 148) * 128 * 20 <= ((n + 147) / 148) * 64 * 21;
}
}  // namespace wide

template <int D>
cudaError_t launch_bwd(const TrainBwdArgs& a, cudaStream_t stream, int* launches) {
  using C = BwdCfg<D>;
  const TrainExactPlan p = train_exact_plan(a.B, a.Hq, a.Hkv, a.S, a.D, a.causal);
  const bool wide_dq = p.dq_rows == wide::OWN, wide_dkv = p.dkv_rows == wide::OWN;
  auto dq_kern = p.dq.grouped ? train_dq_kernel<D, true> : train_dq_kernel<D, false>;
  auto dkv_kern = p.dkv.grouped ? train_dkv_kernel<D, true> : train_dkv_kernel<D, false>;
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    for (auto k : {train_dq_kernel<D, false>, train_dq_kernel<D, true>}) {
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::DQ_SMEM);
      if (e != cudaSuccess) return e;
    }
    for (auto k : {train_dkv_kernel<D, false>, train_dkv_kernel<D, true>}) {
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::DKV_SMEM);
      if (e != cudaSuccess) return e;
    }
    configured[dev] = true;
  }
  *launches = 0;
  const long long rows = (long long)a.B * a.Hq * a.S;
  train_prep_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>(a.o, a.d_o, a.delta, rows, D);
  (*launches)++;
  if (wide_dq || wide_dkv) {
    e = wide::configure();
    if (e != cudaSuccess) return e;
  }
  if (wide_dq)
    wide::train_dq_wide_kernel<<<p.dq.grid, 256, wide::DQ_SMEM, stream>>>(a.q, a.k, a.v, a.d_o, a.lse, a.delta, a.mask, a.dq,
                                                                         a.S, a.Hq, a.Hkv, p.dq.grouped, a.causal);
  else
    dq_kern<<<p.dq.grid, 256, C::DQ_SMEM, stream>>>(a.q, a.k, a.v, a.d_o, a.lse, a.delta, a.mask, a.dq, a.S, a.Hq, a.Hkv,
                                                  a.causal);
  (*launches)++;
  if (wide_dkv)
    wide::train_dkv_wide_kernel<<<p.dkv.grid, 256, wide::DKV_SMEM, stream>>>(a.q, a.k, a.v, a.d_o, a.lse, a.delta, a.mask, a.dk,
                                                                            a.dv, a.S, a.Hq, a.Hkv, p.dkv.grouped, a.causal);
  else
    dkv_kern<<<p.dkv.grid, 256, C::DKV_SMEM, stream>>>(a.q, a.k, a.v, a.d_o, a.lse, a.delta, a.mask, a.dk, a.dv, a.S, a.Hq, a.Hkv,
                                                   a.causal);
  (*launches)++;
  return cudaGetLastError();
}

}  // namespace

TrainExactPlan train_exact_plan(int B, int Hq, int Hkv, int S, int D, int causal) {
  const int group = Hq / Hkv;
  TrainExactPlan p;
  p.dq_rows = D == 64 && wide::worth_it(S, B * Hq, causal) ? wide::OWN : BT;
  p.dkv_rows = D == 64 && wide::worth_it(S, B * Hkv, causal) ? wide::OWN : BT;
  // The 64-row kernels take a grouped grid under a causal mask, of one head per group where cta_grid gives a plain one;
  // that grid has the tiles in y, and a sequence with more than y holds stays plain.
  auto grid_of = [&](int rows, size_t bytes, int heads) {
    const int tiles = (S + rows - 1) / rows;
    const CtaGrid plain{dim3((unsigned)tiles, (unsigned)heads, 1), 0};
    if (rows == BT && !causal) return plain;
    const CtaGrid g = cta_grid(bytes, heads, tiles, causal ? CAUSAL_TILES : S % rows != 0);
    if (rows != BT || g.grouped) return g;
    return tiles <= 65535 ? CtaGrid{dim3(1, (unsigned)tiles, (unsigned)heads), 1} : plain;
  };
  // f32 bytes that stream past a tile: the shared K and V, or Q and dO of the group's heads
  p.dq = grid_of(p.dq_rows, (size_t)S * D * 8 / (size_t)group, B * Hq);
  p.dkv = grid_of(p.dkv_rows, (size_t)S * D * 8 * (size_t)group, B * Hkv);
  return p;
}

cudaError_t launch_attn_train_backward(const TrainBwdArgs& a, cudaStream_t stream, int* launches) {
  if (a.D == 64) return launch_bwd<64>(a, stream, launches);
  if (a.D == 128) return launch_bwd<128>(a, stream, launches);
  return cudaErrorInvalidValue;
}

}  // namespace ar
