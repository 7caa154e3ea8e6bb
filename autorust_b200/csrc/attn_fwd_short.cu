// Fused bf16 attention forward for short sequences (S <= 256, D = 64, no additive mask), e.g. a vision transformer's 197
// tokens: the semantics of attn_fwd_tc.cu's bf16 mode with the whole key range in one pass.
//
// All scores of a query tile fit the TMEM columns of half an SM: S = Q K^T is one MMA chain of N = S columns (rounded up
// to 16), the softmax has seen all of a row's scores before its first exponential, and P V is one chain of K = S.  There
// is no rescaling of O, no key loop and no padding to 128 keys.  The arithmetic is that of the two 128-key steps of
// attn_fwd_tc.cu, so that a row's bits do not depend on which of the kernels served it: the maximum of the first 128 keys
// is the reference unless a later score exceeds it by RESCALE_THRESHOLD (only then do the roundings of P differ), a
// step's row sum is kept in two accumulators, and only a step of 128 visible keys has a quarter of its exponentials on
// the FMA pipe (1.1e-4; the row sum and the log-sum-exp of shorter sequences keep the accuracy of the MUFU unit).
//
//   persistent CTA, two per SM, 192 threads; its items are (batch x head, tile of 128 queries)
//     warps 0-3  softmax and epilogue (thread r owns row r = TMEM lane r)
//     warp  4    TMA producer: Q and K of the next item as soon as this item's Q K^T has read them, V likewise
//     warp  5    MMA issuer
//   TMEM (256 columns): S [0, 256); P (bf16, two per column) overwrites [0, 128) as S is read; O takes [128, 192) once
//   all of S has been read.
//
// Bound: latency.  Measured, B=64 H=12 S=197 on strided views: 42.5 us in the key loop's one-tile form, 31.4 us here against
// 11.8 us for its 77 MB (29.4 with the cubic in every whole chunk: what the accuracy costs); the MUFU unit and the issue
// slots are about a third busy.  An item's chain is about 8000 cycles: maximum 1070, exponentials 3100, P V with its
// hand-overs 1350, from O read to the next scores 2300, and two CTAs per SM are what TMEM holds.
#include "ar_kernels.h"
#include "ar_ptx.cuh"
#include "softmax_math.cuh"

namespace ar {
namespace {
using namespace arptx;

#ifdef AR_WAIT_TEST
__device__ int g_test_skip_item = -1;  // test builds only: the item whose V tiles are never requested
#endif

constexpr int BM = 128, D = 64, KEYS = 256;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float NEG = -1e30f * LOG2E;  // the reference's finite sentinel in the log2 domain
constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units, as in attn_fwd_tc.cu
constexpr int NUM_THREADS = 192;
constexpr int W_PROD = 4, W_MMA = 5;
constexpr int Q_BYTES = BM * D * 2, KV_BYTES = KEYS * D * 2;
constexpr int STAGE_BYTES = BM * D * 2;  // output rows on their way to whole 128-byte stores
constexpr int NUM_BARS = 8;
constexpr int SMEM_BYTES = Q_BYTES + 2 * KV_BYTES + STAGE_BYTES + NUM_BARS * 8 + 16 + 1024;
static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");

// Exponentials of 32 columns of a row: P (bf16 pairs) into pk, the unrounded values added to the two sums.  POLY: a
// quarter on the FMA pipe (columns that may be -inf take the MUFU path, whose 2^-inf is exactly 0).
template <bool POLY>
__device__ __forceinline__ void exp_chunk(const uint32_t* sv, uint64_t c2, uint64_t negm2, uint32_t (&pk)[16],
                                          uint64_t (&sum)[2]) {
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), c2, negm2);
    float p0, p1;
    if (POLY && (i & 3) == 3)
      exp2_poly_x2(x2, p0, p1);
    else
      exp2_mufu_x2(x2, p0, p1);
    sum[i & 1] = add_f32x2(sum[i & 1], pack_f32x2(p0, p1));
    pk[i] = pack_bf16x2(p0, p1);
  }
}
__device__ __forceinline__ float max_chunk(const uint32_t* sv, float m) {
  float m0 = m, m1 = __uint_as_float(sv[31]);
#pragma unroll
  for (int i = 0; i < 28; i += 4) {
    m0 = fmax3(m0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
    m1 = fmax3(m1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
  }
  return fmax3(fmaxf(m0, m1), __uint_as_float(sv[28]), fmaxf(__uint_as_float(sv[29]), __uint_as_float(sv[30])));
}
// columns from the first excluded one on become -inf
__device__ __forceinline__ void exclude(uint32_t* sv, int first_out) {
  if (first_out >= 32) return;
#pragma unroll
  for (int i = 0; i < 32; i++)
    if (i >= first_out) sv[i] = 0xff800000u;
}

// EXTRA: further output buffers or completion reports, an instantiation of its own (with both in the plain one: 29.5 ->
// 37.9 us for the shape above).
template <bool EXTRA>
__global__ void __launch_bounds__(NUM_THREADS, 2)
    attn_fwd_short_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                          const __grid_constant__ CUtensorMap tm_v, void* __restrict__ out, int N, int Hq, int Hkv, int items,
                          int causal, int out_f32, int token_major, long long o_sb, long long o_sh, long long o_ss,
                          const OutReplicas reps, const OutProgress progress, float* __restrict__ lse_out, uint32_t* status,
                          uint32_t* sticky, uint32_t ticket) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + Q_BYTES;
  uint8_t* sV = sK + KV_BYTES;
  uint8_t* stage = sV + KV_BYTES;
  uint64_t* bars = (uint64_t*)(stage + STAGE_BYTES);
  uint64_t* qk_full = bars;        // every barrier completes once per item
  uint64_t* qk_empty = bars + 1;   // Q K^T has read Q and K
  uint64_t* v_full = bars + 2;
  uint64_t* v_empty = bars + 3;    // P V has read V
  uint64_t* s_full = bars + 4;
  uint64_t* p_full = bars + 5;     // P written, S read
  uint64_t* o_full = bars + 6;
  uint64_t* o_empty = bars + 7;    // O read: the columns may take the next S
  uint32_t* tmem_slot = (uint32_t*)(bars + NUM_BARS);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const WaitCtx wctx{abort_flag, status, sticky, ticket};

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int qtiles = (N + BM - 1) / BM;
  const int group = Hq / Hkv;
  struct Item {
    int b, h, q0, keys;  // keys: how many of them the tile's rows can see
  };
  auto item_at = [&](int i) {
    const int bh = i / qtiles, qt = i - bh * qtiles;
    const int b = bh / Hq;
    return Item{b, bh - b * Hq, qt * BM, causal ? min(N, (qt + 1) * BM) : N};
  };
  auto load_tile = [&](uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int tok, int head, int b, int tensor) {
    if ((token_major >> tensor) & 1)
      tma_load_4d(dst, m, bar, 0, head, tok, b);
    else
      tma_load_4d(dst, m, bar, 0, tok, head, b);
  };
  auto issue_qk = [&](const Item& it) {
    const int boxes = (it.keys + BM - 1) / BM;
    mbar_arrive_expect_tx(qk_full, Q_BYTES + boxes * (BM * D * 2));
    load_tile(sQ, &tm_q, qk_full, it.q0, it.h, it.b, 0);
    for (int x = 0; x < boxes; x++) load_tile(sK + x * (BM * D * 2), &tm_k, qk_full, x * BM, it.h / group, it.b, 1);
  };
  auto issue_v = [&](const Item& it, int item) {
#ifdef AR_WAIT_TEST
    if (item == g_test_skip_item) return;
#endif
    const int boxes = (it.keys + BM - 1) / BM;
    mbar_arrive_expect_tx(v_full, boxes * (BM * D * 2));
    for (int x = 0; x < boxes; x++) load_tile(sV + x * (BM * D * 2), &tm_v, v_full, x * BM, it.h / group, it.b, 2);
  };

  bool lost = false;  // (meaningful in the producer thread only)
  if (warp == W_PROD && lane == 0) {
    // a launch whose status word is already set is lost: this CTA only allocates and frees its TMEM
    lost = launch_lost(status, ticket);
    *abort_flag = lost ? 1u : 0u;
    for (int i = 0; i < NUM_BARS; i++) mbar_init(&bars[i], &bars[i] == p_full || &bars[i] == o_empty ? 128 : 1);
    fence_mbar_init();
    if (!lost) {
      const Item it = item_at(blockIdx.x);
      issue_qk(it);
      issue_v(it, blockIdx.x);
    }
  }
  if (warp == W_MMA) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = *tmem_slot;

  if (warp == W_PROD) {
    if (lane == 0 && !lost) {
      int qk_issued = 1, v_issued = 1;
      for (int i = blockIdx.x + gridDim.x; i < items; i += gridDim.x) {
        const Item it = item_at(i);
        if (!mbar_wait(qk_empty, (qk_issued - 1) & 1, wctx, 0x60)) break;
        issue_qk(it);
        qk_issued++;
        if (!mbar_wait(v_empty, (v_issued - 1) & 1, wctx, 0x61)) break;
        issue_v(it, i);
        v_issued++;
      }
      if (*abort_flag) {  // let what was started land before the shared memory goes back
        mbar_wait_quiet(qk_full, (qk_issued - 1) & 1);
        mbar_wait_quiet(v_full, (v_issued - 1) & 1);
      }
    }
  } else if (warp == W_MMA) {
    const uint64_t k_proto = make_sdesc_sw128(0, 16, 1024), v_proto = make_sdesc_sw128(0, KEYS * 128, 1024);
    const uint32_t k_hi = (uint32_t)(k_proto >> 32), v_hi = (uint32_t)(v_proto >> 32);
    const uint32_t qa = (uint32_t)k_proto | (smem_u32(sQ) >> 4), ka = (uint32_t)k_proto | (smem_u32(sK) >> 4);
    const uint32_t va = (uint32_t)v_proto | (smem_u32(sV) >> 4);
    constexpr uint32_t IDESC_PV = make_idesc(1, 1, 1, 0, 1, BM, D);
    bool ok = true;
    int n = 0;
    for (int i = blockIdx.x; i < items && ok; i += gridDim.x, n++) {
      const int ksteps = (item_at(i).keys + 15) >> 4;
      const uint32_t idesc_qk = make_idesc(1, 1, 1, 0, 0, BM, ksteps * 16);
      ok = __all_sync(0xffffffffu, mbar_wait(qk_full, n & 1, wctx, 0x62));
      if (!ok) break;
      if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(o_empty, (n - 1) & 1, wctx, 0x63));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int s = 0; s < D / 16; s++)
          mma_ss_lohi<KIND_F16>(tb, qa + (s * 32 >> 4), k_hi, ka + (s * 32 >> 4), k_hi, idesc_qk, s > 0);
      }
      commit_one(s_full);
      commit_one(qk_empty);
      ok = __all_sync(0xffffffffu, mbar_wait(v_full, n & 1, wctx, 0x64));
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(p_full, n & 1, wctx, 0x65));
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll 1
        for (int s = 0; s < ksteps; s++)
          mma_ts_lohi<KIND_F16>(tb + 128, tb + s * 8, va + s * (2048 >> 4), v_hi, IDESC_PV, s > 0 ? 1u : 0u);
      }
      commit_one(o_full);
      commit_one(v_empty);
    }
  } else {
    const int r = tid;
    const uint32_t lane_base = (uint32_t)warp * 32;
    const uint32_t tS = tmem_addr(tb, lane_base, 0), tO = tmem_addr(tb, lane_base, 128);
    const float c = (1.0f / sqrtf((float)D)) * LOG2E;
    const uint64_t c2 = pack_f32x2(c, c);
    bool ok = true;
    int n = 0;
    for (int i = blockIdx.x; i < items && ok; i += gridDim.x, n++) {
      const Item it = item_at(i);
      const int row = it.q0 + r;
      const bool rows_in = it.q0 + warp * 32 < N;       // the warp has rows inside the sequence
      const int visible = causal ? min(N, row + 1) : N;  // keys this row sees
      const int chunks = (it.keys + 31) >> 5;            // columns past the last key may hold anything: excluded below
      // (uniform) no lane of the CTA excludes a column before chunk `whole`; the 128-key steps before chunk `poly` are
      // whole ones
      const int whole = causal ? it.q0 >> 5 : N >> 5, poly = whole & ~3;
      float m = NEG, l = 0.f;
      do {  // (left early by a warp whose wait ran out or whose rows lie past the sequence end)
      ok = __all_sync(0xffffffffu, mbar_wait(s_full, n & 1, wctx, 0x66));
      if (!ok) break;
      tc_fence_after();
      if (rows_in) {
        // the row's maximum over the first 128 keys, and over the others
        uint32_t sa[32], sb[32];
        float mx = __uint_as_float(0xff800000u), first = mx;
#pragma unroll 1
        for (int q = 0; q < chunks; q += 2) {
          tmem_ld32(tS + q * 32, sa);
          tmem_ld32(tS + q * 32 + 32, sb);  // (chunk 7 at most; past the last one everything is excluded)
          tmem_wait_ld32(sa);
          tmem_wait_ld32(sb);
          if (q + 1 >= whole) {
            exclude(sa, visible - q * 32);
            exclude(sb, visible - q * 32 - 32);
          }
          mx = max_chunk(sb, max_chunk(sa, mx));
          if (q < 4) {
            first = mx;
            if (q == 2) mx = __uint_as_float(0xff800000u);
          }
        }
        m = fmaxf(m, first * c);
        if (chunks > 4 && mx * c > m + RESCALE_THRESHOLD) m = mx * c;
        const uint64_t negm2 = pack_f32x2(-m, -m);
        uint64_t sum[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
        auto end_step = [&]() {
          float lo, hi;
          unpack_f32x2(add_f32x2(sum[0], sum[1]), lo, hi);
          l += lo + hi;
          sum[0] = sum[1] = pack_f32x2(0.f, 0.f);
        };
        // P of chunk q goes to columns [16 q, 16 q + 16): the scores there have been read.  The next chunk's scores are
        // on their way during this one's exponentials.
        auto chunk = [&](uint32_t(&sv)[32], int q) {
          uint32_t pk[16];
          if (q < poly) {
            exp_chunk<true>(sv, c2, negm2, pk, sum);
          } else {
            exclude(sv, visible - q * 32);
            exp_chunk<false>(sv, c2, negm2, pk, sum);
          }
          tmem_st16(tS + q * 16, pk);
        };
        tmem_ld32(tS, sa);
        tmem_wait_ld32(sa);
#pragma unroll 1
        for (int q = 0; q < chunks; q += 2) {
          if (q + 1 < chunks) tmem_ld32(tS + q * 32 + 32, sb);
          chunk(sa, q);
          if (q + 1 < chunks) {
            tmem_wait_ld32(sb);
            if (q + 2 < chunks) tmem_ld32(tS + q * 32 + 64, sa);
            chunk(sb, q + 1);
            if (q + 2 < chunks) tmem_wait_ld32(sa);
          }
          if (q == 2) end_step();
        }
        tmem_wait_st();
        end_step();
      }
      tc_fence_before();
      mbar_arrive(p_full);
      ok = __all_sync(0xffffffffu, mbar_wait(o_full, n & 1, wctx, 0x67));
      if (!ok) break;
      tc_fence_after();
      uint32_t ov[D];
      tmem_ld32(tO, ov);
      tmem_ld32(tO + 32, ov + 32);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive(o_empty);  // the next item's Q K^T may start under this item's stores
      if (!rows_in) break;
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      const long long base = (long long)it.b * o_sb + (long long)it.h * o_sh;
      if (lse_out != nullptr && row < N)
        lse_out[(size_t)(it.b * Hq + it.h) * N + row] = (m + log2f(l)) * (1.0f / LOG2E);
      if (out_f32) {
        if (row < N) {
          float4* dst = (float4*)((float*)out + base + (long long)row * o_ss);
#pragma unroll
          for (int x = 0; x < D / 4; x++)
            dst[x] = make_float4(__uint_as_float(ov[4 * x]) * inv, __uint_as_float(ov[4 * x + 1]) * inv,
                                 __uint_as_float(ov[4 * x + 2]) * inv, __uint_as_float(ov[4 * x + 3]) * inv);
        }
      } else {
        // whole 128-byte rows per store: through shared memory, 16-byte piece x of row r at x ^ (r & 7); a warp reads
        // back only the rows it wrote
#pragma unroll
        for (int x = 0; x < 8; x++) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(ov[8 * x]) * inv, __uint_as_float(ov[8 * x + 1]) * inv);
          w.y = pack_bf16x2(__uint_as_float(ov[8 * x + 2]) * inv, __uint_as_float(ov[8 * x + 3]) * inv);
          w.z = pack_bf16x2(__uint_as_float(ov[8 * x + 4]) * inv, __uint_as_float(ov[8 * x + 5]) * inv);
          w.w = pack_bf16x2(__uint_as_float(ov[8 * x + 6]) * inv, __uint_as_float(ov[8 * x + 7]) * inv);
          *(uint4*)(stage + r * 128 + ((x ^ (r & 7)) * 16)) = w;
        }
        __syncwarp();
#pragma unroll
        for (int x = 0; x < 8; x++) {
          const int rr = warp * 32 + 4 * x + (lane >> 3), ch = lane & 7;
          const uint4 w = *(const uint4*)(stage + rr * 128 + ((ch ^ (rr & 7)) * 16));
          if (it.q0 + rr < N) {
            const size_t off = (size_t)(base + (long long)(it.q0 + rr) * o_ss + ch * 8) * 2;
            if (EXTRA && reps.multicast) {
              multimem_st16((uint8_t*)reps.p[0] + off, w);  // one store, delivered to every GPU by the switch
            } else {
              *(uint4*)((uint8_t*)out + off) = w;
              if constexpr (EXTRA) {
                for (int e = 0; e < reps.n; e++) *(uint4*)((uint8_t*)reps.p[e] + off) = w;
              }
            }
          }
        }
        __syncwarp();
      }
      } while (false);
      if (EXTRA && progress.count != nullptr) {
        // Completion report, as in the long kernel: the barrier orders the item's rows before this thread, the count
        // releases them device-wide, and the pair's last item releases the flag to the host.
        ok = bar_all(1, 128, ok);
        if (ok && tid == 0) {
          const int pair = it.b * Hq + it.h;
          uint32_t before;
          asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(progress.count + pair) : "memory");
          if (before + 1u == (uint32_t)qtiles)
            asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(progress.flag + pair), "r"(progress.epoch) : "memory");
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W_MMA) tmem_dealloc(tb, 256);
}

}  // namespace

// Up to one item per SM a launch is one chain of latencies, which the key loop's one-tile form gets through sooner: it reads
// the scores once, into 128 registers, and hands P over in halves (12 heads of S=128: 5.3 us against 5.7, causal 5.8 and
// 6.3, S=256 6.4 and 6.9).  With more, items under way side by side count.
bool attn_short_takes(const TcArgs& a) {
  return a.mode == TC_BF16 && a.D == D && a.S <= KEYS && a.mask == nullptr &&
         (long long)((a.S + BM - 1) / BM) * a.B * a.Hq > 148;
}

template <bool EXTRA>
cudaError_t launch_short(const TcArgs& a, cudaStream_t stream) {
  auto kern = attn_fwd_short_kernel<EXTRA>;
  static bool configured[64] = {};
  static int sm_count[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int items = ((a.S + BM - 1) / BM) * a.B * a.Hq;
  const int resident = 2 * (dev < 64 ? sm_count[dev] : 148);
  kern<<<items < resident ? items : resident, NUM_THREADS, SMEM_BYTES, stream>>>(
      a.tm_q, a.tm_k, a.tm_v, a.out, a.S, a.Hq, a.Hkv, items, a.causal, a.out_f32, a.token_major, a.o_sb, a.o_sh, a.o_ss,
      a.replicas, a.progress, a.lse_out, a.status, a.sticky, a.ticket);
  return cudaGetLastError();
}

cudaError_t launch_attn_short(const TcArgs& a, cudaStream_t stream) {
  return a.replicas.n > 0 || a.progress.count != nullptr ? launch_short<true>(a, stream) : launch_short<false>(a, stream);
}

}  // namespace ar

#ifdef AR_WAIT_TEST
extern "C" int ar_test_skip_short_item(int item) {
  return cudaMemcpyToSymbol(ar::g_test_skip_item, &item, sizeof(int)) == cudaSuccess ? 0 : -1;
}
#endif
