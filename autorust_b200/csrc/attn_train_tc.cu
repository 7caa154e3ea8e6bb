// Backward of the attention path on the sm_100a tensor cores: dQ, dK, dV from the saved log-sum-exp, with bf16
// operands and f32 accumulation.
//
// The same mathematics as the f32 kernels of attn_train.cu (which replace autorust's `ar_fl_bwd_dq` / `ar_fl_bwd_dkv`,
// src/runtime/cuda_flash_train.rs:118-309) -- p = exp(s - LSE) rebuilt tile by tile, dS = p (dO.v - D_i),
// dQ = dS K / sqrt(D), dK = dS^T Q / sqrt(D), dV = P^T dO -- but every product is a tcgen05.mma:
//
//   dQ kernel   one CTA per (128 queries, batch x head); per step of 64 keys
//                 S = Q K^T, dP = dO V^T           (both operands K-major in shared memory, accumulators in TMEM)
//                 dS = p (dP - D) -> bf16 in TMEM over S
//                 dQ += dS K                       (A from TMEM, K consumed MN-major from the tile it was loaded as)
//   dK/dV kernel one CTA per (128 keys, batch x kv head); per step of 64 queries of every query head of the GQA group
//                 S^T = K Q^T, dP^T = V dO^T       (TMEM lanes are KEYS here, so that P^T and dS^T can be A operands)
//                 P^T, dS^T -> bf16 in TMEM
//                 dV += P^T dO, dK += dS^T Q       (dO and Q consumed MN-major from the tiles S^T and dP^T read K-major)
//
// A step's scores and dP take 128 TMEM columns, and the columns that the accumulators leave hold STAGES = 3 steps (2 for
// dK/dV at D = 128), each with an element-wise warpgroup of its own (thread = TMEM lane); one CTA per SM.  SMALL (D = 64):
// 256 columns, one step and one element-wise warpgroup, two CTAs per SM, for short walks in several rounds.  The MMA warp keeps STAGES steps of S and dP issued ahead, so that the tensor pipe works on later steps while the
// warpgroups are on theirs:  ... dQ(n), S/dP(n + STAGES), dQ(n + 1), S/dP(n + 1 + STAGES) ...  MMAs of one thread
// execute in issue order, which is what lets S(n + STAGES) overwrite the columns dQ(n) has read.
// Floor of a step per SM at D = 64: S and dP 384 cycles of the tensor pipe (N = 64 with both operands from shared memory
// reads 6 KB for 32 cycles of math), dK and dV 256, and 512 cycles for 8192 exponentials.  Measured, B=4 H=16 S=2048
// D=64: dQ 163 -> 158 us (1030 cycles per step), dK/dV 254 -> 205 us (1250) against two CTAs per SM that each ran S/dP ->
// element-wise -> dQ with nothing issued ahead.  What bounds it now is the MMA warp: of a step's 1030 cycles it spends
// 760 issuing into a full tensor queue and 270 on its waits, its instructions queueing behind the element-wise warps';
// the element-wise part takes a warpgroup 1050 of the 3060 cycles it has (2000 of 3750 in dK/dV).
//
// No atomics: a CTA owns its output tile and walks its reduction in a fixed order, so two launches give the same
// bits.  Operands are bf16 copies of the f32 tensors (made by the caller of these kernels); P and dS are rounded to
// bf16 like P in the forward kernels.  On the reference test's inputs (tests/flash_train_cuda.rs:18-22) that keeps
// every gradient within about 2e-3 of its largest entry: inside the test's absolute 2e-3 for its plain and masked
// cases (1.6e-3 at most), above it where a causal mask or GQA makes the gradients larger (up to 8.8e-3 on a dV whose
// largest entry is 5.7).  A fast mode with a stated accuracy, like the bf16 forward; the f32 kernels remain the
// exact path.
#include "ar_kernels.h"
#include "ar_ptx.cuh"
#include "cta_order.cuh"

#include <cmath>
#include <cooperative_groups.h>

namespace ar {
namespace {
using namespace arptx;

#ifdef AR_WAIT_TEST
__device__ int g_test_skip_step = -1;  // test builds only: the step whose streamed tiles CTA 0 never requests
#endif

constexpr int T = 128;  // rows a CTA owns: queries (dQ) or keys (dK/dV)
constexpr int NH = 64;  // rows streamed per step: keys (dQ) or queries (dK/dV)
constexpr float LOG2E = 1.4426950408889634f;

template <int D, bool DKV, bool SMALL>
struct TcBwd {
  static constexpr int ROW_BYTES = D * 2;
  static constexpr int OWN_BYTES = T * ROW_BYTES;     // one tile of the CTA's own rows (two: Q and dO, or K and V)
  static constexpr int STREAM_BYTES = NH * ROW_BYTES; // one streamed tile (two per step)
  static constexpr int ACC_COLS = DKV ? 2 * D : D;    // TMEM columns of the gradient accumulators
  static constexpr int TMEM_COLS = SMALL ? 256 : 512;
  static constexpr int MIN_CTAS = SMALL ? 2 : 1;
  static constexpr int STAGES = (TMEM_COLS - ACC_COLS) / (2 * NH) < 3 ? (TMEM_COLS - ACC_COLS) / (2 * NH) : 3;
  static constexpr int SLOTS = D == 64 && !SMALL ? 6 : 4;  // streamed steps in shared memory; STAGES + 1 keep the MMAs fed
  static_assert(SLOTS > STAGES, "a slot beyond the steps in flight");
  static constexpr int ROWVALS_BYTES = STAGES * 2 * 2 * NH * 4;  // dK/dV: LSE and D_i of a step's queries, double-buffered
  static constexpr int NUM_BARS = 2 + 2 * SLOTS + 2 * STAGES;
  static constexpr int SMEM_BYTES = 2 * OWN_BYTES + SLOTS * 2 * STREAM_BYTES + ROWVALS_BYTES + NUM_BARS * 8 + 16 + 1024;
  static_assert(MIN_CTAS * (SMEM_BYTES + 1024) <= 228 * 1024, "shared memory budget");
  static_assert(ACC_COLS * T * 4 <= 2 * OWN_BYTES + SLOTS * 2 * STREAM_BYTES, "accumulators pass through the tiles");
  static constexpr int KSTEPS_D = D / 16;             // k-steps of a product over d
  static constexpr int KSTEPS_NH = NH / 16;           // k-steps of a product over one step's rows
  static constexpr uint32_t IDESC_SS = make_idesc(1, 1, 1, 0, 0, T, NH);  // bf16 x bf16 -> f32, both K-major, N = NH
  static constexpr uint32_t IDESC_TS = make_idesc(1, 1, 1, 0, 1, T, D);   // A from TMEM, B MN-major, N = D
  static constexpr int W_PROD = 4 * STAGES, W_MMA = W_PROD + 1;
  static constexpr int NUM_THREADS = 128 * STAGES + (SMALL ? 64 : 128);   // (two more warps complete the last warpgroup)
  // registers per thread: launched with LAUNCH_REGS, then (two stages) moved from the last warpgroup to the others
  static constexpr bool MOVE_REGS = STAGES == 2;
  static constexpr int LAUNCH_REGS = STAGES == 3 ? 128 : 168;
  static constexpr int EW_REGS = 192, SERVICE_REGS = 120;
  static_assert(!MOVE_REGS || 128 * STAGES * EW_REGS + 128 * SERVICE_REGS <= LAUNCH_REGS * NUM_THREADS, "register pool of the CTA");
  static_assert(MIN_CTAS * LAUNCH_REGS * NUM_THREADS <= 65536, "register file of the SM");
};

// D[tmem, 128 x NH] = A[128 x D] B[NH x D]^T, both tiles K-major (rows of 128-byte boxes, 128-byte swizzle)
template <int D, bool DKV, bool SMALL>
__device__ __forceinline__ void mma_abt(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi) {
  if (!elect_one()) return;
#pragma unroll
  for (int s = 0; s < TcBwd<D, DKV, SMALL>::KSTEPS_D; s++) {
    const uint32_t a = a_lo + (((s >> 2) * (T * 128) + (s & 3) * 32) >> 4);
    const uint32_t b = b_lo + (((s >> 2) * (NH * 128) + (s & 3) * 32) >> 4);
    mma_ss_lohi<KIND_F16>(d_tmem, a, hi, b, hi, TcBwd<D, DKV, SMALL>::IDESC_SS, s > 0);
  }
}
// D[tmem, 128 x D] (+)= A[tmem, 128 x NH bf16] B[NH x D], B consumed MN-major from a row-major tile
template <int D, bool DKV, bool SMALL>
__device__ __forceinline__ void mma_tb(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, bool acc) {
  if (!elect_one()) return;
#pragma unroll
  for (int s = 0; s < TcBwd<D, DKV, SMALL>::KSTEPS_NH; s++)
    mma_ts_lohi<KIND_F16>(d_tmem, a_tmem + s * 8, b_lo + s * (2048 >> 4), b_hi, TcBwd<D, DKV, SMALL>::IDESC_TS,
                          (acc || s > 0) ? 1u : 0u);
}

// `rows` (64 or 128) rows of D bf16 from a [B, H, S, D] tensor into a tile of boxes of 64 columns; the maps' boxes are
// 64 rows high.
template <int D>
__device__ __forceinline__ void load_rows(uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int rows, int row0, int head,
                                          int b) {
  for (int bx = 0; bx < D / 64; bx++)
    for (int r = 0; r < rows; r += NH) tma_load_4d(dst + (bx * rows + r) * 128, m, bar, bx * 64, row0 + r, head, b);
}

// dQ (DKV = false): own rows are queries (A tiles Q, dO), K and V stream.  dK/dV (DKV = true): own rows are keys (A
// tiles K, V), Q and dO of the group's query heads stream.
// dK/dV with split > 1: a cluster of `split` CTAs shares a key tile, each walks its part of the group's query heads, and
// the CTAs add their accumulators through distributed shared memory, column by column in rank order.
template <int D, bool DKV, bool SMALL>
__global__ void __launch_bounds__(TcBwd<D, DKV, SMALL>::NUM_THREADS, TcBwd<D, DKV, SMALL>::MIN_CTAS)
train_bwd_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                    const float* __restrict__ LSE, const float* __restrict__ delta, const float* __restrict__ mask,
                    float* __restrict__ out0, float* __restrict__ out1, int N, int Hq, int Hkv, int grouped, int split,
                    int causal, uint32_t* status, uint32_t* sticky) {
  using C = TcBwd<D, DKV, SMALL>;
  constexpr int ST = C::STAGES, SL = C::SLOTS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* own0 = smem;                               // Q | K
  uint8_t* own1 = own0 + C::OWN_BYTES;                // dO | V
  uint8_t* ring = own1 + C::OWN_BYTES;                // per slot: K, V | Q, dO
  float* rowvals = (float*)(ring + SL * 2 * C::STREAM_BYTES);
  uint64_t* bars = (uint64_t*)((uint8_t*)rowvals + C::ROWVALS_BYTES);
  uint64_t* own_full = bars;
  uint64_t* acc_full = own_full + 1;                  // every MMA complete
  uint64_t* slot_full = acc_full + 1;                 // [SL]
  uint64_t* slot_empty = slot_full + SL;              // [SL]
  uint64_t* s_full = slot_empty + SL;                 // [ST] S and dP of a step complete
  uint64_t* p_full = s_full + ST;                     // [ST] dS (and P) written by the stage's 128 threads
  uint32_t* tmem_slot = (uint32_t*)(p_full + ST);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const WaitCtx wctx{abort_flag, status, sticky};

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  if (!DKV) split = 1;
  const int bh = cta_head(grouped, split);
  int tile = cta_tile(grouped, split);
  const int rank = DKV && split > 1 ? (int)(blockIdx.x % (uint32_t)split) : 0;
  // dQ under a causal mask: the last query tile sees the most keys; dK/dV: the first key tile sees the most queries
  if (!DKV && causal) tile = cta_tiles(grouped) - 1 - tile;
  const int H = DKV ? Hkv : Hq, G = Hq / Hkv;
  const int heads = DKV ? G / split : 1;              // query heads this CTA walks, from g0 on
  const int g0 = rank * heads;
  const int b = bh / H, h = bh - b * H;               // DKV: h is a kv head
  const int row0 = tile * T;
  // the steps this tile walks: dQ -- blocks of 64 keys; dK/dV -- blocks of 64 queries, head by head of the group
  const int first = DKV && causal ? row0 / NH : 0;    // queries before the key tile see none of it
  const int last = !DKV && causal ? (min(N, row0 + T) + NH - 1) / NH : (N + NH - 1) / NH;
  const int per_head = last - first;
  const int steps = heads * per_head;

  if (warp == C::W_PROD && lane == 0) {
    *abort_flag = 0;
    mbar_init(own_full, 1);
    mbar_init(acc_full, 1);
    for (int i = 0; i < SL; i++) {
      mbar_init(&slot_full[i], 1);
      mbar_init(&slot_empty[i], 1);
    }
    for (int i = 0; i < ST; i++) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
    }
    fence_mbar_init();
  }
  if (warp == C::W_MMA) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = *tmem_slot;
  const uint32_t col_acc = ST * 2 * NH;               // accumulators: dQ | dV, dK

  bool finished = false;  // (element-wise warps)
  // 32 accumulator columns of one of the CTA's rows to the output they belong to
  auto store_chunk = [&](const uint32_t(&ov)[32], int c, int row) {
    const bool second = DKV && c >= D / 32;  // dV first, then dK
    const int cd = second ? c - D / 32 : c;
    const float f = DKV && !second ? 1.0f : 1.0f / sqrtf((float)D);
    if (row < N) {
      float4* dst = (float4*)((second ? out1 : out0) + ((size_t)bh * N + row) * D + cd * 32);
#pragma unroll
      for (int i = 0; i < 8; i++)
        dst[i] = make_float4(__uint_as_float(ov[4 * i]) * f, __uint_as_float(ov[4 * i + 1]) * f,
                             __uint_as_float(ov[4 * i + 2]) * f, __uint_as_float(ov[4 * i + 3]) * f);
    }
  };

  if constexpr (C::MOVE_REGS) {
    if (warp >= C::W_PROD) setmaxnreg_dec<C::SERVICE_REGS>();
  }
  if (warp == C::W_PROD) {
    if (lane == 0) {
      const int own_h = h;
      mbar_arrive_expect_tx(own_full, 2 * C::OWN_BYTES);
      load_rows<D>(own0, DKV ? &tm_k : &tm_q, own_full, T, row0, own_h, b);
      load_rows<D>(own1, DKV ? &tm_v : &tm_do, own_full, T, row0, own_h, b);
      int issued = 0;
      for (int n = 0; n < steps; n++) {
        const int sl = n % SL;
        const int g = DKV ? n / per_head : 0;
        const int r = (first + n - g * per_head) * NH;
        const int sh = DKV ? h * G + g0 + g : h / G;       // head of the streamed tensors
        if (n >= SL && !mbar_wait(&slot_empty[sl], ((n / SL) - 1) & 1, wctx, 0x50)) break;
#ifdef AR_WAIT_TEST
        if (n == g_test_skip_step && blockIdx.x + blockIdx.y + blockIdx.z == 0) continue;
#endif
        uint8_t* dst = ring + sl * 2 * C::STREAM_BYTES;
        mbar_arrive_expect_tx(&slot_full[sl], 2 * C::STREAM_BYTES);
        load_rows<D>(dst, DKV ? &tm_q : &tm_k, &slot_full[sl], NH, r, sh, b);
        load_rows<D>(dst + C::STREAM_BYTES, DKV ? &tm_do : &tm_v, &slot_full[sl], NH, r, sh, b);
        issued = n + 1;
      }
      if (*abort_flag) {  // let what was started land before the shared memory goes back
        mbar_wait_quiet(own_full, 0);
        for (int n = max(0, issued - SL); n < issued; n++) mbar_wait_quiet(&slot_full[n % SL], (n / SL) & 1);
      }
    }
  } else if (warp == C::W_MMA) {
    const uint64_t k_proto = make_sdesc_sw128(0, 16, 1024);         // K-major
    const uint64_t mn_proto = make_sdesc_sw128(0, NH * 128, 1024);  // MN-major: 64-column boxes NH * 128 bytes apart
    const uint32_t k_hi = (uint32_t)(k_proto >> 32), mn_hi = (uint32_t)(mn_proto >> 32);
    // a descriptor holds 18 bits of an address; in a cluster the rank lies above them, which would fall into the offsets
    auto desc_addr = [](const void* p) { return (smem_u32(p) & 0x3ffffu) >> 4; };
    const uint32_t a0 = (uint32_t)k_proto | desc_addr(own0), a1 = (uint32_t)k_proto | desc_addr(own1);
    const uint32_t ring0 = desc_addr(ring);
    bool ok = __all_sync(0xffffffffu, mbar_wait(own_full, 0, wctx, 0x51));
    auto scores = [&](int n) {  // S and dP of step n into its stage
      const int st = n % ST;
      if (!__all_sync(0xffffffffu, mbar_wait(&slot_full[n % SL], (n / SL) & 1, wctx, 0x52))) return false;
      tc_fence_after();
      const uint32_t x = ring0 + (n % SL) * (2 * C::STREAM_BYTES >> 4), y = x + (C::STREAM_BYTES >> 4);
      mma_abt<D, DKV, SMALL>(tb + st * 2 * NH, a0, (uint32_t)k_proto | x, k_hi);       // S = Q K^T     | S^T = K Q^T
      mma_abt<D, DKV, SMALL>(tb + st * 2 * NH + NH, a1, (uint32_t)k_proto | y, k_hi);  // dP = dO V^T   | dP^T = V dO^T
      commit_one(&s_full[st]);
      return true;
    };
    for (int n = 0; n < min(ST, steps) && ok; n++) ok = scores(n);
    for (int n = 0; n < steps && ok; n++) {
      const int st = n % ST;
      ok = __all_sync(0xffffffffu, mbar_wait(&p_full[st], (n / ST) & 1, wctx, 0x53));
      if (!ok) break;
      tc_fence_after();
      const uint32_t x = ring0 + (n % SL) * (2 * C::STREAM_BYTES >> 4), y = x + (C::STREAM_BYTES >> 4);
      const uint32_t s_cols = tb + st * 2 * NH, p_cols = s_cols + NH;
      if constexpr (DKV) {
        mma_tb<D, DKV, SMALL>(tb + col_acc, s_cols, (uint32_t)mn_proto | y, mn_hi, n > 0);      // dV += P^T dO
        mma_tb<D, DKV, SMALL>(tb + col_acc + D, p_cols, (uint32_t)mn_proto | x, mn_hi, n > 0);  // dK += dS^T Q
      } else {
        mma_tb<D, DKV, SMALL>(tb + col_acc, s_cols, (uint32_t)mn_proto | x, mn_hi, n > 0);      // dQ += dS K
      }
      commit_one(&slot_empty[n % SL]);
      if (n + ST < steps) ok = scores(n + ST);
    }
    if (ok) commit_one(acc_full);
  } else if (warp < C::W_PROD) {
    // element-wise: warpgroup wg takes steps wg, wg + STAGES, ...; thread r owns the CTA's row row0 + r
    if constexpr (C::MOVE_REGS) setmaxnreg_inc<C::EW_REGS>();
    const int wg = warp >> 2;
    const int r = tid & 127;
    const int row = row0 + r;
    const uint32_t lane_base = (uint32_t)(warp & 3) * 32;
    const uint32_t tS = tmem_addr(tb, lane_base, wg * 2 * NH), tdP = tS + NH;
    const float scale_log2 = (1.0f / sqrtf((float)D)) * LOG2E;
    const uint64_t sc2 = pack_f32x2(scale_log2, scale_log2);
    // dQ: this query's -LSE (log2 domain) and -D_i
    float nlse = 0.f, ndl = 0.f;
    if (!DKV && row < N) {
      nlse = -LSE[(size_t)bh * N + row] * LOG2E;
      ndl = -delta[(size_t)bh * N + row];
    }
    // dK/dV: the same of the step's 64 queries, through shared memory; threads 0-63 bring LSE, 64-127 D_i, one step of
    // this warpgroup ahead
    float* vals = rowvals + wg * (2 * 2 * NH);
    auto fetch = [&](int n) {
      const int g = n / per_head, qrow = (first + n - g * per_head) * NH + (r & (NH - 1));
      if (n >= steps || qrow >= N) return 0.f;
      const size_t at = (size_t)(b * Hq + h * G + g0 + g) * N + qrow;
      return r < NH ? -LSE[at] * LOG2E : -delta[at];
    };
    float next_val = 0.f;
    if constexpr (DKV) next_val = fetch(wg);
    bool ok = true;
    int it = 0;
    for (int n = wg; n < steps; n += ST, it++) {
      const float* lv = vals + (it & 1) * (2 * NH);  // [NH] -LSE, [NH] -D_i
      if constexpr (DKV) {
        vals[(it & 1) * (2 * NH) + r] = next_val;
        next_val = fetch(n + ST);
        ok = bar_all(1 + wg, 128, ok);  // (a warp whose wait ran out takes the others with it)
        if (!ok) break;
      }
      const int g = DKV ? n / per_head : 0;
      const int c0 = (first + n - g * per_head) * NH;  // first streamed row: key (dQ) or query (dK/dV)
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[wg], it & 1, wctx, 0x54));
      if (!ok) {
        if constexpr (DKV) continue;
        break;
      }
      tc_fence_after();
      // a step whose 64 streamed rows lie inside the sequence, on the visible side of the causal diagonal and under no
      // additive mask needs none of the per-element tests: two lanes per instruction.  (The CTA's own rows past the end
      // may hold anything: a row of P or dS reaches its own row of the accumulators only, and that one is not stored.)
      const bool interior = mask == nullptr && c0 + NH <= N &&
                            (!causal || (DKV ? row0 + T - 1 <= c0 : c0 + NH - 1 <= row0));
      // 16 columns at a time, the next 16 on their way meanwhile: [0, 16) of a buffer are scores, [16, 32) dP
      uint32_t buf[2][32];
      tmem_ld16(tS, buf[0]);
      tmem_ld16(tdP, buf[0] + 16);
#pragma unroll 2
      for (int c = 0; c < NH / 16; c++) {
        uint32_t* sv = buf[c & 1];
        uint32_t* pv = sv + 16;
        tmem_wait_ld32(sv);
        if (c + 1 < NH / 16) {
          tmem_ld16(tS + (c + 1) * 16, buf[(c + 1) & 1]);
          tmem_ld16(tdP + (c + 1) * 16, buf[(c + 1) & 1] + 16);
        }
        uint32_t pk[8], dk[8];
        if (interior) {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            float4 l = make_float4(nlse, nlse, nlse, nlse), d = make_float4(ndl, ndl, ndl, ndl);
            if constexpr (DKV) {
              l = *(const float4*)(lv + c * 16 + i);
              d = *(const float4*)(lv + NH + c * 16 + i);
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              float x0, x1, d0, d1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i + e]), __uint_as_float(sv[i + e + 1])), sc2,
                                     e ? pack_f32x2(l.z, l.w) : pack_f32x2(l.x, l.y)), x0, x1);
              const float p0 = ex2f(x0), p1 = ex2f(x1);
              const uint64_t t2 = add_f32x2(pack_f32x2(__uint_as_float(pv[i + e]), __uint_as_float(pv[i + e + 1])),
                                            e ? pack_f32x2(d.z, d.w) : pack_f32x2(d.x, d.y));
              unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), t2), d0, d1);
              if constexpr (DKV) pk[(i + e) >> 1] = pack_bf16x2(p0, p1);
              dk[(i + e) >> 1] = pack_bf16x2(d0, d1);
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float p[2], ds[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const int cc = c * 16 + i + e;
              const int key = DKV ? row : c0 + cc, qrow = DKV ? c0 + cc : row;
              const float l = DKV ? lv[cc] : nlse, d = DKV ? lv[NH + cc] : ndl;
              float x = __uint_as_float(sv[i + e]) * scale_log2;
              if (mask != nullptr && qrow < N && key < N) x = fmaf(mask[(size_t)qrow * N + key], LOG2E, x);
              const bool out = key >= N || qrow >= N || (causal && key > qrow);
              p[e] = out ? 0.f : ex2f(x + l);
              ds[e] = p[e] * (__uint_as_float(pv[i + e]) + d);
            }
            if constexpr (DKV) pk[i >> 1] = pack_bf16x2(p[0], p[1]);
            dk[i >> 1] = pack_bf16x2(ds[0], ds[1]);
          }
        }
        // over the columns that have been read: dS | P^T over S^T, dS^T over dP^T
        if constexpr (DKV) {
          tmem_st8(tS + c * 8, pk);
          tmem_st8(tdP + c * 8, dk);
        } else {
          tmem_st8(tS + c * 8, dk);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&p_full[wg]);
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, wctx, 0x55));
    if (ok) {
      tc_fence_after();
      // the accumulators' 32-column chunks, shared out over the warpgroups
#pragma unroll 1
      for (int c = wg; c < C::ACC_COLS / 32; c += ST) {
        uint32_t ov[32];
        tmem_ld32(tmem_addr(tb, lane_base, col_acc + c * 32), ov);
        tmem_wait_ld();
        if (DKV && split > 1) {  // every MMA and copy is done: the tiles' memory takes the accumulators, [column][row]
          float* buf = (float*)smem + (c * 32) * T + r;
#pragma unroll
          for (int i = 0; i < 32; i++) buf[i * T] = __uint_as_float(ov[i]);
        } else {
          store_chunk(ov, c, row);
        }
      }
    }
    finished = ok;
  }
  if constexpr (DKV) {
    if (split > 1) {  // (every thread of the cluster comes by here, whatever its waits returned)
      namespace cg = cooperative_groups;
      cg::cluster_group cluster = cg::this_cluster();
      __syncwarp();  // the cluster barrier counts whole warps: the producer's lanes meet again first
      cluster.sync();
      if (finished && warp < C::W_PROD) {
        const int r = tid & 127;
        const int chunks = C::ACC_COLS / 32, mine = (rank * chunks) / split, end = ((rank + 1) * chunks) / split;
#pragma unroll 1
        for (int c = mine + (warp >> 2); c < end; c += ST) {
          uint32_t ov[32];
#pragma unroll
          for (int i = 0; i < 32; i++) ov[i] = 0u;
#pragma unroll 1
          for (int k = 0; k < split; k++) {
            const float* buf = cluster.map_shared_rank((float*)smem, k) + (c * 32) * T + r;
#pragma unroll
            for (int i = 0; i < 32; i++) ov[i] = __float_as_uint(__uint_as_float(ov[i]) + buf[i * T]);
          }
          store_chunk(ov, c, row0 + r);
        }
      }
      __syncwarp();
      cluster.sync();  // nobody's shared memory goes away while another CTA reads it
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == C::W_MMA) tmem_dealloc(tb, C::TMEM_COLS);
}

// delta[row] = O_row . dO_row and the bf16 copy of dO in one pass over both: D / 4 lanes per row.
template <int D>
__global__ void __launch_bounds__(256) train_prep_tc_kernel(const float* __restrict__ O, const float* __restrict__ dO,
                                                            float* __restrict__ delta, uint2* __restrict__ dO16,
                                                            long long rows) {
  constexpr int LPR = D / 4;
  const long long at = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long row = at / LPR;
  float acc = 0.f;
  if (row < rows) {
    const float4 a = ((const float4*)O)[at], g = ((const float4*)dO)[at];
    acc = fmaf(a.w, g.w, fmaf(a.z, g.z, fmaf(a.y, g.y, a.x * g.x)));
    dO16[at] = make_uint2(pack_bf16x2(g.x, g.y), pack_bf16x2(g.z, g.w));
  }
#pragma unroll
  for (int sh = LPR / 2; sh > 0; sh >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
  if (row < rows && threadIdx.x % LPR == 0) delta[row] = acc;
}

// bf16 copies of q, k and v in one launch, and the launch's status word cleared on the way (the attention kernels that
// follow on the stream want it zero).
__global__ void __launch_bounds__(256) train_convert_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                            const float* __restrict__ v, uint4* __restrict__ q16,
                                                            uint4* __restrict__ k16, uint4* __restrict__ v16,
                                                            long long nq8, long long nk8, uint32_t* status) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0u;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < nq8 + 2 * nk8; i += (long long)gridDim.x * 256) {
    const float* src = i < nq8 ? q : i < nq8 + nk8 ? k : v;
    uint4* dst = i < nq8 ? q16 : i < nq8 + nk8 ? k16 : v16;
    const long long at = i < nq8 ? i : i < nq8 + nk8 ? i - nq8 : i - nq8 - nk8;
    const float4 a = *(const float4*)(src + at * 8), c = *(const float4*)(src + at * 8 + 4);
    dst[at] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(c.x, c.y), pack_bf16x2(c.z, c.w));
  }
}

template <int D, bool DKV, bool SMALL>
cudaError_t launch_bwd_tc(const TrainBwdTcArgs& a, int split, cudaStream_t stream) {
  using C = TcBwd<D, DKV, SMALL>;
  auto kern = train_bwd_tc_kernel<D, DKV, SMALL>;
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && !configured[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int heads = a.B * (DKV ? a.Hkv : a.Hq), group = a.Hq / a.Hkv, tiles = (a.S + T - 1) / T;
  // bf16 bytes that stream past a tile: Q and dO of the group's heads, or the shared K and V
  const size_t head_bytes = (size_t)a.S * D * 4 * (DKV ? group : 1) / (DKV ? 1 : group);
  cudaLaunchConfig_t cfg = {};
  const CtaGrid g = cta_grid(head_bytes, heads, tiles, a.causal ? CAUSAL_TILES : a.S % T != 0, split);
  cfg.gridDim = g.grid;
  cfg.blockDim = dim3(C::NUM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, a.tm_q, a.tm_k, a.tm_v, a.tm_do, a.lse, a.delta, a.mask, DKV ? a.dv : a.dq,
                            DKV ? a.dk : (float*)nullptr, a.S, a.Hq, a.Hkv, g.grouped, split, a.causal,
                            a.status, a.sticky);
}

}  // namespace

// The forms that end first by estimate, in microseconds, from measurements of every form at 536 shapes (S = 64 to 8192, 12
// to 1500 heads, groups of 1 to 16).  Over those shapes the choice lies 0.3 % on average above the best of the forms, and
// none is slower than two CTAs per SM without steps issued ahead, which used to serve every D = 64 call.
TrainTcPlan train_tc_plan(int B, int Hq, int Hkv, int S, int D, int causal) {
  TrainTcPlan p{0, 0, 1};
  const int group = Hq / Hkv, tiles = (S + T - 1) / T, steps = (S + NH - 1) / NH;
  // steps of the average tile and, under a causal mask, of the heaviest one, before which no launch ends
  const double mean = causal ? 0.5 * (steps + 2 < 2 * steps ? steps + 2 : 2 * steps) : steps;
  const double most = causal ? steps : 0.0;
  // D = 64, two CTAs per SM: one CTA's set-up and hand-overs run under the other's, which is worth 2 to 3 us per pair; a
  // CTA that is alone on its SM takes nearly twice as long per step.  So: short walks in more than one round of CTAs
  // (768 heads of S=197: 254 us with one CTA per SM, 216 with two; 24 heads of S=768: 33 and 47).
  struct Form {
    double set_up, step;              // one CTA per SM
    double pair_set_up, pair_step;    // two: both CTAs
    double alone_set_up, alone_step;  // ... and one that has its SM to itself
  };
  auto two_per_sm = [&](const Form& f, long long ctas, int heads) {
    if (D != 64 || ctas <= 148) return 0;
    const double one = (double)((ctas + 147) / 148) * (f.set_up + f.step * mean * heads);
    const long long rest = ctas % 296;
    double two = (double)(ctas / 296) * (f.pair_set_up + f.pair_step * mean * heads);
    if (rest > 148)
      two += f.pair_set_up + f.pair_step * mean * heads;
    else if (rest > 0)
      two += f.alone_set_up + f.alone_step * mean * heads;
    const double one_least = f.set_up + f.step * most * heads, two_least = f.pair_set_up + f.pair_step * most * heads;
    return (two > two_least ? two : two_least) < (one > one_least ? one : one_least) ? 1 : 0;
  };
  p.small_dq = two_per_sm({3.5, 0.54, 5.0, 1.08, 2.9, 1.06}, (long long)tiles * B * Hq, 1);
  // dK/dV of a GQA group: few CTAs with `group` times a head's steps each.  The query heads of the group may be dealt out
  // over a cluster, so that the last CTA to end has a `split`-th of the work; each CTA then pays its own set-up, two
  // cluster barriers and the sum over the ranks, and clusters of some sizes leave SMs of an 18-SM group idle.  It pays
  // where less than a round of CTAs has long walks (B=1 Hq=16 Hkv=2 S=1531 D=64: 193 us, 87 over four) and costs where
  // there are several rounds (B=36 Hq=64 Hkv=8 S=256: 406 us, 841 over eight).
  const long long ctas = (long long)tiles * B * Hkv;
  double least = 0.0;
  for (int split = 1; split <= 8; split++) {
    if (group % split != 0) continue;
    const double set_up = split == 1 ? 4.0 : 4.0 + 2.0 * sqrt((double)split), step = D == 64 ? 0.78 : 1.08;
    const int resident = split == 1 ? 148 : 8 * (18 / split) * split, heads = group / split;
    const double rounds = (double)(ctas * split) / resident, heaviest = set_up + step * heads * steps;
    double t = ceil(rounds) * heaviest;
    if (causal) {
      t = 1.15 * rounds * (set_up + step * heads * 0.5 * (steps + 2));
      if (t < heaviest) t = heaviest;
    }
    if (split == 1 || t < least * (p.split == 1 ? 0.97 : 1.0)) {
      least = t;
      p.split = split;
    }
  }
  if (p.split == 1) p.small_dkv = two_per_sm({4.0, 0.66, 4.8, 1.72, 3.1, 1.5}, ctas, group);
  return p;
}

cudaError_t launch_attn_train_backward_tc(const TrainBwdTcArgs& a, cudaStream_t stream, int* launches) {
  if (a.D != 64 && a.D != 128) return cudaErrorInvalidValue;
  const TrainTcPlan p = train_tc_plan(a.B, a.Hq, a.Hkv, a.S, a.D, a.causal);
  cudaError_t e = a.D == 128   ? launch_bwd_tc<128, false, false>(a, 1, stream)
                  : p.small_dq ? launch_bwd_tc<64, false, true>(a, 1, stream)
                               : launch_bwd_tc<64, false, false>(a, 1, stream);
  if (e != cudaSuccess) return e;
  (*launches)++;
  e = a.D == 128    ? launch_bwd_tc<128, true, false>(a, p.split, stream)
      : p.small_dkv ? launch_bwd_tc<64, true, true>(a, p.split, stream)
                    : launch_bwd_tc<64, true, false>(a, p.split, stream);
  if (e != cudaSuccess) return e;
  (*launches)++;
  return cudaSuccess;
}

cudaError_t launch_train_prep_tc(const float* o, const float* d_o, float* delta, void* do16, long long rows, int D,
                                 cudaStream_t stream) {
  const unsigned blocks = (unsigned)((rows * (D / 4) + 255) / 256);
  if (D == 64)
    train_prep_tc_kernel<64><<<blocks, 256, 0, stream>>>(o, d_o, delta, (uint2*)do16, rows);
  else
    train_prep_tc_kernel<128><<<blocks, 256, 0, stream>>>(o, d_o, delta, (uint2*)do16, rows);
  return cudaGetLastError();
}

cudaError_t launch_train_convert(const float* q, const float* k, const float* v, void* q16, void* k16, void* v16,
                                 long long nq, long long nk, uint32_t* status, cudaStream_t stream) {
  const long long n8 = nq / 8 + 2 * (nk / 8);
  const long long blocks = (n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16;
  train_convert_kernel<<<(unsigned)blocks, 256, 0, stream>>>(q, k, v, (uint4*)q16, (uint4*)k16, (uint4*)v16, nq / 8, nk / 8,
                                                             status);
  return cudaGetLastError();
}

}  // namespace ar

#ifdef AR_WAIT_TEST
extern "C" int ar_test_skip_backward_step(int step) {
  return cudaMemcpyToSymbol(ar::g_test_skip_step, &step, sizeof(int)) == cudaSuccess ? 0 : -1;
}
#endif
