// Shared-MLP GEMMs for few tokens on the 5th-generation tensor cores (sm_100a).
//
// With few tokens the weights are the traffic and there are not enough 256 x 256 tiles to keep the SMs busy.  Here the
// WEIGHT rows are the 128 rows of the MMA and the tokens its columns,
//   D[128 weight rows, bn tokens] = W[128, K] * x[bn, K]^T          (bn: any multiple of 16 up to 256)
// so a tile carries no padding beyond 15 tokens and every weight byte is read once per token tile.
//
// 320 threads, one tile per CTA: warp 0 (one lane) TMA producer, warp 1 (one lane) MMA issuer, warps 2..9 epilogue with one
// weight row per thread: a warp's load of one token's float32 addend or residual covers 32 consecutive columns (the
// transposed tile makes the down GEMM's addend coalesced without staging), and the finished tile, [token][weight row] in
// shared memory, leaves in one tiled store.
// Epilogues: SWIGLU (two weight tiles per stage, gate and up rows of the same outputs), ADD (+ addend, + residual) and RAW
// (the float32 sums, where a later kernel adds).  Every mbarrier wait is bounded.
//
// Bound by the weight bytes, and with the narrowest tiles by the MMAs that follow one another on the same sums: 1 token, hidden
// 1024, intermediate 4096 (25 MB of weights, both GEMMs inside a forward, us): 33 -> 17; 64 tokens, 2048 x 5632 (69 MB): 48 ->
// 29; 777 tokens, 1000 x 2728: 43 -> 35 (128-row token tiles in one or two CTAs per row of tiles before).  The set-up runs
// ahead of the predecessor's end: barriers and the first ring of weight tiles need nothing from it.
#include <algorithm>

#include "gemm_epilogue.cuh"

namespace fmoe {
namespace {

constexpr int BLOCK_K = 64;
constexpr int UMMA_K = 16;
constexpr int kEpiWarps = 8;  // two per TMEM lane quarter, on alternate batches of token columns
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kMaxStages = 20;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kBarBytes = 512;

enum { NARROW_ADD = 0, NARROW_SWIGLU = 1, NARROW_RAW = 2 };  // RAW: the float32 sums

struct NarrowEpi {
  void* out;
  const float* addend;   // ADD, nullable: float32 [M, N]
  const void* residual;  // ADD, nullable: [M, N] in the module dtype
  void* pre_gate;        // SWIGLU, nullable (both or neither): the two products rounded to T
  void* pre_up;
  int n_valid;
};

struct NarrowShape {
  int M;            // tokens
  int bn;           // tokens per tile
  int num_kb;       // 64-column blocks of K
  int stages;
  int acc_cols;     // TMEM columns per accumulator (power of two)
  int early;        // kEarlyWeights | kEarlyTokens
};

// BLOCK_R weight rows per tile: 128, or 64 where that gives more CTAs.  With 64 the accumulator's row i sits in TMEM lane
// 32 * (i / 16) + i % 16: each epilogue warp finds 16 rows in the first 16 lanes of its lane quarter.
template <int BLOCK_R, int EPI, typename T>
__global__ void __launch_bounds__(kThreads, 1)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                   const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmOut, NarrowEpi ep,
                   NarrowShape sh, int32_t* status) {
  constexpr int NB = EPI == NARROW_SWIGLU ? 2 : 1;
  constexpr int W_BYTES = BLOCK_R * BLOCK_K * 2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw_u32 + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw_u32);
  const int stage_bytes = NB * W_BYTES + sh.bn * BLOCK_K * 2;
  const int ring_bytes = sh.stages * stage_bytes;
  const uint32_t bar_base = base + ring_bytes;
  auto stage_smem = [&](int s) { return base + s * stage_bytes; };
  auto full_bar = [&](int s) { return bar_base + s * 8; };
  auto empty_bar = [&](int s) { return bar_base + (kMaxStages + s) * 8; };
  const uint32_t tfull_bar = bar_base + 2 * kMaxStages * 8;
  uint8_t* gen_bar = gen + ring_bytes;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen_bar + (2 * kMaxStages + 1) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_bar + (2 * kMaxStages + 1) * 8 + 8);

  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0);  // known to be warp-uniform
  const int lane = threadIdx.x & 31;
  const bool late = (sh.early & kEarlyTokens) != 0;
  const int r0 = blockIdx.x * BLOCK_R;
  const int t0 = blockIdx.y * sh.bn;
  const int nkb = sh.num_kb;
  const uint32_t tmem_cols = NB * sh.acc_cols < 32 ? 32 : NB * sh.acc_cols;

  if (warp == 0) {
    // ------------------------------------------------------------ set-up and TMA producer
    auto load_weights = [&](int s, int i) {
      ptx::tma_load_2d(stage_smem(s), &tmW0, full_bar(s), i * BLOCK_K, r0);
      if (NB == 2) ptx::tma_load_2d(stage_smem(s) + W_BYTES, &tmW1, full_bar(s), i * BLOCK_K, r0);
    };
    auto load_tokens = [&](int s, int i) {
      ptx::tma_load_2d(stage_smem(s) + NB * W_BYTES, &tmX, full_bar(s), i * BLOCK_K, t0);
    };
    if (ptx::elect_one()) {
      for (int s = 0; s < sh.stages; ++s) {
        ptx::mbar_init(full_bar(s), 1);
        ptx::mbar_init(empty_bar(s), 1);
      }
      ptx::mbar_init(tfull_bar, 1);
      *abort_flag = 0;
      ptx::mbar_fence_init();
    }
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");  // the others may use the barriers; no wait here
    if (ptx::elect_one()) {
      ptx::prefetch_tensormap(&tmW0);
      ptx::prefetch_tensormap(&tmX);
      ptx::prefetch_tensormap(&tmOut);
      if (NB == 2) ptx::prefetch_tensormap(&tmW1);
    }
    const int first = nkb < sh.stages ? nkb : sh.stages;
    if (sh.early & kEarlyWeights) {
      for (int i = 0; i < first; ++i)
        if (ptx::elect_one()) {
          ptx::mbar_arrive_expect_tx(full_bar(i), stage_bytes);
          load_weights(i, i);
        }
    }
    __syncwarp();
    if (!late) {
      pdl_wait();  // the tokens come from the kernel before this one
      pdl_launch_dependents();
    }
    for (int i = 0; i < first; ++i)
      if (ptx::elect_one()) {
        if (!(sh.early & kEarlyWeights)) {
          ptx::mbar_arrive_expect_tx(full_bar(i), stage_bytes);
          load_weights(i, i);
        }
        load_tokens(i, i);
      }
    __syncwarp();
    bool ok = true;
    int i = first, s = 0;
    uint32_t ph = 0;
    for (; i < nkb; ++i) {
      if (!ptx::mbar_wait_bounded(empty_bar(s), ph, abort_flag)) { ok = false; break; }
      if (ptx::elect_one()) {
        ptx::mbar_arrive_expect_tx(full_bar(s), stage_bytes);
        load_weights(s, i);
        load_tokens(s, i);
      }
      if (++s == sh.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (!ok)  // let the copies already issued land before the CTA goes away (bounded)
      for (int j = i > sh.stages ? i - sh.stages : 0; j < i; ++j)
        ptx::mbar_wait_drain(full_bar(j % sh.stages), (j / sh.stages) & 1u);
    __syncwarp();
  } else {
    if (warp == 1) {
      ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
      ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
    ptx::tc_fence_after();
    // late: only the epilogue waits.  The first thread of a CTA that gets here lets the next kernel start, so with `late` that
    // is one of those that have waited.
    if (!late || warp >= 2) {
      pdl_wait();
      pdl_launch_dependents();  // this CTA holds its tensor memory: once all do, the next kernel may set up
    }
  }
  const uint32_t tmem_base = warp == 0 ? 0u : __shfl_sync(kFull, *tmem_slot, 0);

  if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = (1u << 4) | (epi::UmmaFmt<T>::v << 7) | (epi::UmmaFmt<T>::v << 10) |
                           (static_cast<uint32_t>(sh.bn >> 3) << 17) | (static_cast<uint32_t>(BLOCK_R >> 4) << 24);
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < nkb; ++i) {
      if (!ptx::mbar_wait_bounded(full_bar(s), ph, abort_flag)) { ok = false; break; }
      ptx::tc_fence_after();
      const uint64_t dw = ptx::umma_desc_kmajor_sw128(stage_smem(s));
      const uint64_t dx = ptx::umma_desc_kmajor_sw128(stage_smem(s) + NB * W_BYTES);
      if (ptx::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BLOCK_K / UMMA_K; ++kk)  // the two accumulators in turn: an MMA waits for the sums it adds to
#pragma unroll
          for (int b = 0; b < NB; ++b)
            ptx::umma_bf16_ss(tmem_base + b * sh.acc_cols, dw + (b * W_BYTES >> 4) + 2 * kk, dx + 2 * kk, idesc,
                              (i | kk) != 0 ? 1u : 0u);
        ptx::umma_commit(empty_bar(s));
      }
      if (++s == sh.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (ok && ptx::elect_one()) ptx::umma_commit(tfull_bar);
    __syncwarp();
  }

  // ---------------------------------------------------------------- epilogue
  const bool epilogue_warp = warp >= 2;
  const int q = warp & 3;            // TMEM lane quarter this warp may read
  const int turn = (warp - 2) >> 2;  // which of the quarter's two warps
  const int row = BLOCK_R == 128 ? q * 32 + lane : q * 16 + (lane & 15);
  const bool lane_ok = BLOCK_R == 128 || lane < 16;
  const int n = r0 + row;
  const bool n_ok = n < ep.n_valid && lane_ok;
  const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
  T* otile = reinterpret_cast<T*>(gen);   // [sh.bn][BLOCK_R]: the ring is free once the accumulator is complete
  // 16 token columns at a time: the sums of the next batch and their addends are requested before this batch is worked on
  // (777 tokens, 1000 x 2728 and back: layer 65.5 -> 59.4 us), the first batch's addends while the MMAs still run
  constexpr int CH = 16;
  struct Batch {
    uint32_t a[CH], b[CH];
    float ad[CH];
    uint16_t rs[CH];
  };
  auto request_addends = [&](int c0, Batch& t) {
    if (EPI == NARROW_ADD) {
      const int lim = sh.M - (t0 + c0);
      const int64_t o = static_cast<int64_t>(t0 + c0) * ep.n_valid + n;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const bool in = n_ok && i < lim;
        t.ad[i] = (in && ep.addend != nullptr) ? ld_after_wait(ep.addend + o + static_cast<int64_t>(i) * ep.n_valid) : 0.f;
        t.rs[i] = (in && ep.residual != nullptr)
                      ? ld_after_wait(static_cast<const uint16_t*>(ep.residual) + o + static_cast<int64_t>(i) * ep.n_valid) : 0;
      }
    }
  };
  auto request_sums = [&](int c0, Batch& t) {
    ptx::tmem_ld_32x16(taddr + c0, t.a);
    if (NB == 2) ptx::tmem_ld_32x16(taddr + sh.acc_cols + c0, t.b);
  };
  auto wait_sums = [&](Batch& t) {
    ptx::tmem_ld_wait(t.a);
    if (NB == 2) ptx::tmem_ld_wait(t.b);
  };
  auto finish = [&](int c0, const Batch& t) {
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const float v = __uint_as_float(t.a[i]);
      float r = v;
      if (EPI == NARROW_SWIGLU) r = silu_f32(v) * __uint_as_float(t.b[i]);
      if (EPI == NARROW_ADD) r = v + t.ad[i] + to_f32<T>(*reinterpret_cast<const T*>(&t.rs[i]));
      if (lane_ok) {
        if (EPI == NARROW_RAW) reinterpret_cast<float*>(gen)[(c0 + i) * BLOCK_R + row] = v;
        else otile[(c0 + i) * BLOCK_R + row] = from_f32<T>(r);
      }
    }
    if (EPI == NARROW_SWIGLU && ep.pre_gate != nullptr) {
      const int64_t o = static_cast<int64_t>(t0 + c0) * ep.n_valid + n;
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if (n_ok && t0 + c0 + i < sh.M) {
          static_cast<T*>(ep.pre_gate)[o + static_cast<int64_t>(i) * ep.n_valid] = from_f32<T>(__uint_as_float(t.a[i]));
          static_cast<T*>(ep.pre_up)[o + static_cast<int64_t>(i) * ep.n_valid] = from_f32<T>(__uint_as_float(t.b[i]));
        }
    }
  };
  bool done = true;
  if (epilogue_warp) {
    Batch even, odd;
    const int first = turn * CH;
    if (first < sh.bn) request_addends(first, even);
    done = ptx::mbar_wait_bounded(tfull_bar, 0u, abort_flag);
    done = __all_sync(kFull, done);
    ptx::tc_fence_after();
    // gave up: let the copies in flight land before the ring is reused or goes away (bounded)
    if (!done && threadIdx.x == 64)
      for (int j = nkb > sh.stages ? nkb - sh.stages : 0; j < nkb; ++j)
        ptx::mbar_wait_drain(full_bar(j % sh.stages), (j / sh.stages) & 1u);
    if (done && first < sh.bn) {
      // sums are requested and waited for in straight-line code, after the last batch those of that batch again
      const int last = sh.bn - CH - (sh.bn - CH - first) % (2 * CH);  // sh.bn is a multiple of CH
      request_sums(first, even);
      wait_sums(even);
#pragma unroll 1
      for (int c0 = first;; c0 += 4 * CH) {
        request_sums(min(c0 + 2 * CH, last), odd);
        if (c0 < last) request_addends(c0 + 2 * CH, odd);
        finish(c0, even);
        wait_sums(odd);
        if (c0 >= last) break;
        request_sums(min(c0 + 4 * CH, last), even);
        if (c0 + 2 * CH < last) request_addends(c0 + 4 * CH, even);
        finish(c0 + 2 * CH, odd);
        wait_sums(even);
        if (c0 + 2 * CH >= last) break;
      }
    }
  }

  // ---------------------------------------------------------------- the finished tile leaves; teardown
  ptx::fence_async_smem();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2 && done && ptx::elect_one()) {
    ptx::tma_store_2d(&tmOut, base, r0, t0);
    ptx::tma_store_commit();
    ptx::tma_store_wait();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, tmem_cols);
  }
  if (threadIdx.x == 0 && *abort_flag != 0 && status != nullptr) atomicOr(status, FMOE_STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ host side
struct NarrowPlan {
  int rows = 128, tiles_t = 0, bn = 0, stages = 0;
  double cost = 1e30;  // estimated SM cycles
};

int narrow_stages(int rows, int nb, int bn) {
  const int stages = (kSmemLimit - 1024 - kBarBytes) / (nb * rows * BLOCK_K * 2 + bn * BLOCK_K * 2);
  return stages > kMaxStages ? kMaxStages : stages;
}

// Tile with the least estimated time, in SM clocks.  Per k-block an SM is limited by the bytes it pulls from L2 (about 62 per
// clock) or by the MMAs, of which the narrowest take 65 clocks each, one after the other (they add to the same sums); on top
// come the fixed start (first operands from memory) and the epilogue.  The constants are a fit to timed tiles at 12 shapes
// from 1 to 2048 tokens.  K is not split: over a cluster it was faster by 5 us at 64 tokens x 5632, but the sums then depend on
// the split, and in a stack of layers the last bit of an output decides a later layer's selection.
NarrowPlan plan_narrow(int64_t M, int N, int K, int nb) {
  NarrowPlan best;
  const int sms = device_sm_count();
  const int num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  const int64_t t_min = (M + 255) / 256;
  for (int rows = 64; rows <= 128; rows *= 2) {
    const int row_tiles = (N + rows - 1) / rows;
    for (int64_t tt = t_min; tt <= t_min + 12 && tt * 16 < M + 16; ++tt) {
      const int bn = static_cast<int>(((M + tt - 1) / tt + 15) / 16 * 16);
      const int64_t tiles_t = (M + bn - 1) / bn;
      const int stages = bn <= 256 ? narrow_stages(rows, nb, bn) : 0;
      if (stages < 3) continue;
      const double bytes = (nb * rows * BLOCK_K * 2 + bn * BLOCK_K * 2) / 62.0;
      const double mma = nb * std::max((rows == 64 ? 1.65 : 2.2) * bn, 260.0);
      const double waves = static_cast<double>((row_tiles * tiles_t + sms - 1) / sms);
      const double cost = waves * (3000.0 + num_kb * std::max(bytes, mma) + 39.0 * bn * nb);
      if (cost < best.cost) best = {rows, static_cast<int>(tiles_t), bn, stages, cost};
    }
  }
  return best;
}

// the same estimate for the 256 x 256 pair tiles of gemm_sm100_pair.cu (about 620 clocks per k-block of a pair)
double pair_cost(int64_t M, int N, int K, int nb) {
  const int64_t tiles = ((M + 255) / 256) * ((N * nb + 255) / 256);
  const int64_t pairs = device_sm_count() / 2;
  const double waves = static_cast<double>((tiles + pairs - 1) / pairs);
  const int num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  return 4500.0 + waves * num_kb * 620.0 + (nb == 2 ? 5000.0 : 12000.0);
}

template <int BLOCK_R, int EPI, typename T>
int launch_plan(const NarrowPlan& p, const void* w0, const void* w1, const void* x, const NarrowEpi& ep, int dtype, int64_t M,
                int N, int K, int early, int32_t* status, cudaStream_t stream) {
  constexpr int NB = EPI == NARROW_SWIGLU ? 2 : 1;
  CUtensorMap tW0, tW1, tX;
  int rc;
  if ((rc = epi::make_tensor_map(&tW0, w0, dtype, K, N, K, BLOCK_R)) != FMOE_OK) return rc;
  tW1 = tW0;
  if (NB == 2 && (rc = epi::make_tensor_map(&tW1, w1, dtype, K, N, K, BLOCK_R)) != FMOE_OK) return rc;
  if ((rc = epi::make_tensor_map(&tX, x, dtype, K, M, K, p.bn)) != FMOE_OK) return rc;
  CUtensorMap tOut;
  if ((rc = epi::make_tensor_map_out(&tOut, ep.out, EPI == NARROW_RAW ? FMOE_DTYPE_F32 : dtype, N, M, BLOCK_R, p.bn)) != FMOE_OK) return rc;
  NarrowShape sh;
  sh.M = static_cast<int>(M);
  sh.bn = p.bn;
  sh.num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  sh.stages = p.stages;
  sh.acc_cols = next_pow2(p.bn);
  sh.early = early;
  const int smem = p.stages * (NB * BLOCK_R * BLOCK_K * 2 + p.bn * BLOCK_K * 2) + kBarBytes + 1024;
  auto kern = gemm_narrow_kernel<BLOCK_R, EPI, T>;
  FMOE_CUDA_TRY(allow_smem(kern, kSmemLimit));
  FMOE_CUDA_TRY(launch_pdl(16, kern, dim3((N + BLOCK_R - 1) / BLOCK_R, p.tiles_t), dim3(kThreads), smem, stream,
                           1, tW0, tW1, tX, tOut, ep, sh, status));
  return FMOE_OK;
}

// Token tiles are the grid's second dimension (at most 65535 of them): more tokens than this go in several launches.  Each
// stands to the one in front of it as that one to its predecessor, so `early` holds for all of them.
constexpr int64_t kMaxTokens = int64_t{1} << 23;

template <int EPI, typename T>
int launch_narrow(const void* w0, const void* w1, const void* x, const NarrowEpi& ep, int dtype, int64_t M, int N, int K,
                  int early, int32_t* status, cudaStream_t stream) {
  auto from = [](auto* p, int64_t row, int64_t row_bytes) {
    using P = decltype(p);
    using Byte = std::conditional_t<std::is_const_v<std::remove_pointer_t<P>>, const char, char>;
    return p == nullptr ? p : reinterpret_cast<P>(reinterpret_cast<Byte*>(p) + row * row_bytes);
  };
  for (int64_t m0 = 0; m0 < M; m0 += kMaxTokens) {
    const int64_t rows = std::min(M - m0, kMaxTokens);
    const int64_t pitch = static_cast<int64_t>(N) * sizeof(T);
    const NarrowEpi part{from(ep.out, m0, EPI == NARROW_RAW ? N * int64_t{4} : pitch), from(ep.addend, m0, N * int64_t{4}),
                         from(ep.residual, m0, pitch), from(ep.pre_gate, m0, pitch), from(ep.pre_up, m0, pitch), ep.n_valid};
    const void* xp = from(x, m0, static_cast<int64_t>(K) * sizeof(T));
    const NarrowPlan p = plan_narrow(rows, N, K, EPI == NARROW_SWIGLU ? 2 : 1);
    const int rc = p.rows == 64 ? launch_plan<64, EPI, T>(p, w0, w1, xp, part, dtype, rows, N, K, early, status, stream)
                                : launch_plan<128, EPI, T>(p, w0, w1, xp, part, dtype, rows, N, K, early, status, stream);
    if (rc != FMOE_OK) return rc;
  }
  return FMOE_OK;
}

}  // namespace

// CTAs of the gate/up GEMM
int narrow_swiglu_ctas(int64_t M, int I, int K) {
  const NarrowPlan p = plan_narrow(M, I, K, 2);
  return ((I + p.rows - 1) / p.rows) * p.tiles_t;
}

// 16-bit operands with 16-byte aligned rows (K % 8 == 0), where the estimate is below that of the pair tiles
bool gemm_narrow_preferred(int64_t M, int N, int K, bool swiglu) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 8 != 0) return false;
  if (!gemm_pair_supported(M, N, K)) return true;
  if (M > 8192) return false;
  return plan_narrow(M, N, K, swiglu ? 2 : 1).cost < pair_cost(M, N, K, swiglu ? 2 : 1);
}

int launch_gemm_swiglu_narrow(const void* x, const void* gate_w, const void* up_w, void* h, int dtype, int64_t M, int I,
                              int K, int early, int32_t* status, cudaStream_t stream, void* pre_gate,
                              void* pre_up) {
  if ((pre_gate == nullptr) != (pre_up == nullptr)) return FMOE_ERR_BAD_ARG;
  const NarrowEpi ep{h, nullptr, nullptr, pre_gate, pre_up, I};
  if (dtype == FMOE_DTYPE_BF16)
    return launch_narrow<NARROW_SWIGLU, __nv_bfloat16>(gate_w, up_w, x, ep, dtype, M, I, K, early, status, stream);
  return launch_narrow<NARROW_SWIGLU, __half>(gate_w, up_w, x, ep, dtype, M, I, K, early, status, stream);
}

int launch_gemm_add_narrow(const void* a, const void* b, const float* addend, void* out, int dtype, int64_t M, int N,
                           int K, int early, int32_t* status, cudaStream_t stream, const void* residual, bool raw) {
  const NarrowEpi ep{out, addend, residual, nullptr, nullptr, N};
  if (raw) {
    if (dtype == FMOE_DTYPE_BF16)
      return launch_narrow<NARROW_RAW, __nv_bfloat16>(b, b, a, ep, dtype, M, N, K, early, status, stream);
    return launch_narrow<NARROW_RAW, __half>(b, b, a, ep, dtype, M, N, K, early, status, stream);
  }
  if (dtype == FMOE_DTYPE_BF16)
    return launch_narrow<NARROW_ADD, __nv_bfloat16>(b, b, a, ep, dtype, M, N, K, early, status, stream);
  return launch_narrow<NARROW_ADD, __half>(b, b, a, ep, dtype, M, N, K, early, status, stream);
}

}  // namespace fmoe
