// Shared-MLP GEMMs for few tokens on the 5th-generation tensor cores (sm_100a).
//
// With few tokens the weights are the traffic and there are not enough 256 x 256 tiles to keep the SMs busy.  Here the
// WEIGHT rows are the 128 rows of the MMA and the tokens its columns,
//   D[128 weight rows, bn tokens] = W[128, K] * x[bn, K]^T          (bn: any multiple of 16 up to 256)
// so a tile carries no padding beyond 15 tokens, every weight byte is read once per token tile, and K is split over the
// 1, 2, 4 or 8 CTAs of a cluster.  The partial sums of a cluster meet in distributed shared memory: each CTA owns bn / S
// of the token columns, adds the S partial columns in rank order (so results do not depend on timing) and finishes them.
//
// 320 threads, one tile per CTA: warp 0 (one lane) TMA producer, warp 1 (one lane) MMA issuer, warps 2..9 epilogue with one
// weight row per thread: a warp's load of one token's float32 addend or residual covers 32 consecutive columns (the
// transposed tile makes the down GEMM's addend coalesced without staging), and the finished tile, [token][weight row] in
// shared memory, leaves in one tiled store.
// Epilogues: SWIGLU (two weight tiles per stage, gate and up rows of the same outputs) and ADD (+ addend, + residual).
// Every mbarrier wait is bounded; a CTA that gives up still meets its cluster at both barriers.
//
// Bound by the weight bytes: 1 token, hidden 1024, intermediate 4096 (25 MB of weights, both GEMMs, us): 33 -> 10; 64
// tokens, 2048 x 5632 (69 MB): 48 -> 22, 3.1 TB/s; 777 tokens, 1000 x 2728: 43 -> 33 (128-row token tiles in one or two
// CTAs per row of tiles before).  The set-up runs ahead of the predecessor's end: barriers and the first ring of weight
// tiles need nothing from it.
#include "gemm_epilogue.cuh"

namespace fmoe {
namespace {

constexpr int BLOCK_K = 64;
constexpr int UMMA_K = 16;
constexpr int kEpiWarps = 8;  // two per TMEM lane quarter, on alternate batches of token columns
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int kMaxStages = 8;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kBarBytes = 256;

enum { NARROW_ADD = 0, NARROW_SWIGLU = 1 };

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
  int xchg_bytes;   // buffer of the partial sums (0 without a split)
  int acc_cols;     // TMEM columns per accumulator (power of two)
  int early;        // kEarlyWeights | kEarlyTokens
};

__device__ __forceinline__ void st_cluster_v4(uint32_t cluster_addr, const uint32_t (&v)[4]) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}

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
  const uint32_t bar_base = base + ring_bytes + sh.xchg_bytes;
  auto stage_smem = [&](int s) { return base + s * stage_bytes; };
  auto full_bar = [&](int s) { return bar_base + s * 8; };
  auto empty_bar = [&](int s) { return bar_base + (kMaxStages + s) * 8; };
  const uint32_t tfull_bar = bar_base + 2 * kMaxStages * 8;
  uint8_t* gen_bar = gen + ring_bytes + sh.xchg_bytes;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen_bar + (2 * kMaxStages + 1) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_bar + (2 * kMaxStages + 1) * 8 + 8);

  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0);  // known to be warp-uniform
  const int lane = threadIdx.x & 31;
  const int S = gridDim.x;  // = cluster size
  const bool late = (sh.early & kEarlyTokens) != 0;
  const int rank = blockIdx.x;
  const int r0 = blockIdx.y * BLOCK_R;
  const int t0 = blockIdx.z * sh.bn;
  const int kb0 = rank * sh.num_kb / S;
  const int nkb = (rank + 1) * sh.num_kb / S - kb0;
  const uint32_t tmem_cols = NB * sh.acc_cols < 32 ? 32 : NB * sh.acc_cols;

  if (warp == 0) {
    // ------------------------------------------------------------ set-up and TMA producer
    auto load_weights = [&](int s, int i) {
      ptx::tma_load_2d(stage_smem(s), &tmW0, full_bar(s), (kb0 + i) * BLOCK_K, r0);
      if (NB == 2) ptx::tma_load_2d(stage_smem(s) + W_BYTES, &tmW1, full_bar(s), (kb0 + i) * BLOCK_K, r0);
    };
    auto load_tokens = [&](int s, int i) {
      ptx::tma_load_2d(stage_smem(s) + NB * W_BYTES, &tmX, full_bar(s), (kb0 + i) * BLOCK_K, t0);
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
    if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
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
    // a CTA's shared memory may be written by its peers once all have arrived here; the wait is in front of the exchange
    if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    // late: only the epilogue waits.  The first thread of a CTA that gets here lets the next kernel start, so with `late` that
    // is one of those that have waited.
    if (!late || (warp >= 2 && !(sh.early & kWaitAtEnd))) {
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
        for (int b = 0; b < NB; ++b)
#pragma unroll
          for (int kk = 0; kk < BLOCK_K / UMMA_K; ++kk)
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
  const int cols = sh.bn / S;             // token columns this CTA finishes
  const int tc0 = t0 + rank * cols;       // the first of them
  T* otile = reinterpret_cast<T*>(gen);   // [cols][BLOCK_R]: the ring is free once the accumulator is complete
  bool done = true;
  if (epilogue_warp) {
    done = ptx::mbar_wait_bounded(tfull_bar, 0u, abort_flag);
    done = __all_sync(kFull, done);
    ptx::tc_fence_after();
    // gave up: let the copies in flight land before the ring is reused or goes away (bounded)
    if (!done && threadIdx.x == 64)
      for (int j = nkb > sh.stages ? nkb - sh.stages : 0; j < nkb; ++j)
        ptx::mbar_wait_drain(full_bar(j % sh.stages), (j / sh.stages) & 1u);
  }
  // COUNT token columns from c0 (of this CTA's `cols`) from their float32 sums.  ad / rs: addend and residual.
  auto fetch_addends = [&](int c0, auto& ad, auto& rs) {
    constexpr int COUNT = sizeof(ad) / sizeof(float);
    if (EPI == NARROW_ADD) {
      const int lim = min(cols - c0, sh.M - (tc0 + c0));
      const int64_t o = static_cast<int64_t>(tc0 + c0) * ep.n_valid + n;
#pragma unroll
      for (int i = 0; i < COUNT; ++i) {
        const bool in = n_ok && i < lim;
        ad[i] = (in && ep.addend != nullptr) ? ld_after_wait(ep.addend + o + static_cast<int64_t>(i) * ep.n_valid) : 0.f;
        rs[i] = 0.f;
        if (in && ep.residual != nullptr) {
          const uint16_t raw = ld_after_wait(static_cast<const uint16_t*>(ep.residual) + o + static_cast<int64_t>(i) * ep.n_valid);
          rs[i] = to_f32<T>(*reinterpret_cast<const T*>(&raw));
        }
      }
    }
  };
  auto finish = [&](int c0, const auto& v, const auto& u, const auto& ad, const auto& rs) {
    constexpr int COUNT = sizeof(ad) / sizeof(float);
    const int lim = cols - c0;
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
      const float r = EPI == NARROW_SWIGLU ? silu_f32(v[i]) * u[i] : v[i] + ad[i] + rs[i];
      if (lane_ok && i < lim) otile[(c0 + i) * BLOCK_R + row] = from_f32<T>(r);
    }
    if (EPI == NARROW_SWIGLU && ep.pre_gate != nullptr) {
      const int64_t o = static_cast<int64_t>(tc0 + c0) * ep.n_valid + n;
#pragma unroll
      for (int i = 0; i < COUNT; ++i)
        if (n_ok && i < lim && tc0 + c0 + i < sh.M) {
          static_cast<T*>(ep.pre_gate)[o + static_cast<int64_t>(i) * ep.n_valid] = from_f32<T>(v[i]);
          static_cast<T*>(ep.pre_up)[o + static_cast<int64_t>(i) * ep.n_valid] = from_f32<T>(u[i]);
        }
    }
  };
  constexpr int CH = 16;  // token columns per batch
  if (S == 1) {
    if (epilogue_warp && done) {
#pragma unroll 1
      for (int c0 = turn * CH; c0 < sh.bn; c0 += 2 * CH) {
        float ad[CH], rs[CH];
        fetch_addends(c0, ad, rs);
        uint32_t a[CH], b[CH];
        ptx::tmem_ld_32x16(taddr + c0, a);
        if (NB == 2) ptx::tmem_ld_32x16(taddr + sh.acc_cols + c0, b);
        ptx::tmem_ld_wait();
        float v[CH], u[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
          v[i] = __uint_as_float(a[i]);
          u[i] = NB == 2 ? __uint_as_float(b[i]) : 0.f;
        }
        finish(c0, v, u, ad, rs);
      }
    }
  } else {
    // partial sums to their owners: token column c belongs to CTA c / cols; slot [source][b][c % cols / 4][row][c % 4]
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (epilogue_warp && done) {
#pragma unroll 1
      for (int b = 0; b < NB; ++b) {
        const uint32_t slot = base + ring_bytes + ((rank * NB + b) * cols * BLOCK_R + row * 4) * 4;
#pragma unroll 1
        for (int c0 = turn * CH; c0 < sh.bn; c0 += 2 * CH) {
          int owner = c0 / cols, left = cols - (c0 - owner * cols);
          uint32_t dst = ptx::map_to_cta(slot, owner) + (cols - left) * BLOCK_R * 4;
          uint32_t a[CH];
          ptx::tmem_ld_32x16(taddr + b * sh.acc_cols + c0, a);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < CH; i += 4) {
            if (left == 0) {
              left = cols;
              dst = ptx::map_to_cta(slot, ++owner);
            }
            const uint32_t v[4] = {a[i], a[i + 1], a[i + 2], a[i + 3]};
            if (lane_ok) st_cluster_v4(dst, v);
            dst += BLOCK_R * 16;
            left -= 4;
          }
        }
      }
    }
    ptx::cluster_sync();  // the partial sums have arrived (release / acquire)
    if (epilogue_warp && done) {
      constexpr int OC = 4;  // a CTA owns few columns behind a split
      const float4* part = reinterpret_cast<const float4*>(gen + ring_bytes);
      for (int c0 = turn * OC; c0 < cols; c0 += 2 * OC) {
        float ad[OC], rs[OC], v[2][OC];
        fetch_addends(c0, ad, rs);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const float4* p = part + (b * (cols / 4) + c0 / 4) * BLOCK_R + row;
          const int step = NB * (cols / 4) * BLOCK_R;
          float4 w[8];
#pragma unroll
          for (int s = 0; s < 8; ++s) w[s] = s < S ? p[s * step] : make_float4(0.f, 0.f, 0.f, 0.f);
          float4 sum = w[0];
#pragma unroll
          for (int s = 1; s < 8; ++s) {
            sum.x += w[s].x;
            sum.y += w[s].y;
            sum.z += w[s].z;
            sum.w += w[s].w;
          }
          v[b][0] = sum.x;
          v[b][1] = sum.y;
          v[b][2] = sum.z;
          v[b][3] = sum.w;
        }
        finish(c0, v[0], v[NB - 1], ad, rs);
      }
    }
  }

  // ---------------------------------------------------------------- the finished tile leaves; teardown
  ptx::fence_async_smem();
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 2 && done && tc0 < sh.M && ptx::elect_one()) {
    ptx::tma_store_2d(&tmOut, base, r0, tc0);
    ptx::tma_store_commit();
    ptx::tma_store_wait();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, tmem_cols);
  }
  if (sh.early & kWaitAtEnd) pdl_wait();
  if (threadIdx.x == 0 && *abort_flag != 0 && status != nullptr) atomicOr(status, FMOE_STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ host side
struct NarrowPlan {
  int rows = 128, tiles_t = 0, bn = 0, split = 0, stages = 0;
  double cost = 1e30;  // estimated SM cycles
};

// ring depth beside the exchange buffer; 0: it does not fit
int narrow_stages(int rows, int nb, int bn, int split) {
  if (split > 1 && bn % (4 * split) != 0) return 0;
  const int xchg = split > 1 ? nb * bn * rows * 4 : 0;
  const int stages = (kSmemLimit - 1024 - kBarBytes - xchg) / (nb * rows * BLOCK_K * 2 + bn * BLOCK_K * 2);
  return stages > kMaxStages ? kMaxStages : stages;
}

// Tile and K split with the least estimated time, in SM clocks.  Per k-block an SM is limited by the bytes it pulls from L2
// (about 62 per clock) or by the MMAs; on top come the fixed start (first operands from memory), the epilogue and, with
// a split, the exchange of the partial sums.  The constants are a fit to 600 timed combinations of tile and split at 12
// shapes from 1 to 2048 tokens; the tile it picks is within 6 % of the best of them on average.
// Up to kSameSplit tokens the split is the one that suits 64 tokens: it decides the order of the sums, and a row's result then
// does not depend on how many other rows the call has (token shards equal the unsharded batch bit for bit).
constexpr int kSameSplit = 512;
NarrowPlan plan_narrow(int64_t M, int N, int K, int nb, int fixed_split = 0) {
  if (fixed_split == 0 && M <= kSameSplit) return plan_narrow(M, N, K, nb, plan_narrow(64, N, K, nb, -1).split);
  NarrowPlan best;
  const int sms = device_sm_count();
  const int num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  const int64_t t_min = (M + 255) / 256;
  for (int rows = 64; rows <= 128; rows *= 2) {
    const int row_tiles = (N + rows - 1) / rows;
    for (int64_t tt = t_min; tt <= t_min + 12 && tt * 16 < M + 16; ++tt) {
      for (int split = 1; split <= 8 && split <= num_kb; split *= 2) {
        if (fixed_split > 0 && split != fixed_split) continue;
        const int unit = split == 8 ? 32 : 16;
        const int bn = static_cast<int>(((M + tt - 1) / tt + unit - 1) / unit * unit);
        const int64_t tiles_t = (M + bn - 1) / bn;
        const int stages = bn <= 256 ? narrow_stages(rows, nb, bn, split) : 0;
        if (stages < 3) continue;
        const int stage = nb * rows * BLOCK_K * 2 + bn * BLOCK_K * 2;
        const int64_t ctas = static_cast<int64_t>(split) * row_tiles * tiles_t;
        // clusters are placed within a GPC: 74 of 2, 33 of 4 and 15 of 8 CTAs of this size fit at once
        const int per_wave = split <= 2 ? sms / split * split : split == 4 ? sms * 33 / 148 * 4 : sms * 15 / 148 * 8;
        const double waves = static_cast<double>((ctas + per_wave - 1) / per_wave);
        const int kb = (num_kb + split - 1) / split;
        const double bytes = stage / 62.0, mma = (rows == 64 ? 1.65 : 2.2) * bn * nb;
        const double per_kb = bytes > mma ? bytes : mma;
        const double out = split > 1 ? 400.0 + 40.0 * bn * nb + 18.0 * bn / split : 39.0 * bn * nb;
        const double cost = waves * (3000.0 + kb * per_kb + out);
        if (cost < best.cost) {
          best.cost = cost;
          best.rows = rows;
          best.tiles_t = static_cast<int>(tiles_t);
          best.bn = bn;
          best.split = split;
          best.stages = stages;
        }
      }
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
  if ((rc = epi::make_tensor_map_out(&tOut, ep.out, dtype, N, M, BLOCK_R, p.bn / p.split)) != FMOE_OK) return rc;
  NarrowShape sh;
  sh.M = static_cast<int>(M);
  sh.bn = p.bn;
  sh.num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  sh.stages = p.stages;
  sh.xchg_bytes = p.split > 1 ? NB * p.bn * BLOCK_R * 4 : 0;
  sh.acc_cols = next_pow2(p.bn);
  sh.early = early;
  const int smem = p.stages * (NB * BLOCK_R * BLOCK_K * 2 + p.bn * BLOCK_K * 2) + sh.xchg_bytes + kBarBytes + 1024;
  auto kern = gemm_narrow_kernel<BLOCK_R, EPI, T>;
  FMOE_CUDA_TRY(allow_smem(kern, kSmemLimit));
  FMOE_CUDA_TRY(launch_pdl(16, kern, dim3(p.split, (N + BLOCK_R - 1) / BLOCK_R, p.tiles_t), dim3(kThreads), smem, stream,
                           p.split, tW0, tW1, tX, tOut, ep, sh, status));
  return FMOE_OK;
}

template <int EPI, typename T>
int launch_narrow(const void* w0, const void* w1, const void* x, const NarrowEpi& ep, int dtype, int64_t M, int N, int K,
                  int early, int32_t* status, cudaStream_t stream) {
  const NarrowPlan p = plan_narrow(M, N, K, EPI == NARROW_SWIGLU ? 2 : 1);
  if (p.rows == 64) return launch_plan<64, EPI, T>(p, w0, w1, x, ep, dtype, M, N, K, early, status, stream);
  return launch_plan<128, EPI, T>(p, w0, w1, x, ep, dtype, M, N, K, early, status, stream);
}

}  // namespace

// CTAs of the gate/up GEMM
int narrow_swiglu_ctas(int64_t M, int I, int K) {
  const NarrowPlan p = plan_narrow(M, I, K, 2);
  return p.split * ((I + p.rows - 1) / p.rows) * p.tiles_t;
}

// 16-bit operands with 16-byte aligned rows (K % 8 == 0), where the estimate is below that of the pair tiles
bool gemm_narrow_preferred(int64_t M, int N, int K, bool swiglu) {
  if (M <= 0 || M > (int64_t{1} << 23) || N <= 0 || K <= 0 || K % 8 != 0) return false;
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
                           int K, int early, int32_t* status, cudaStream_t stream, const void* residual) {
  const NarrowEpi ep{out, addend, residual, nullptr, nullptr, N};
  if (dtype == FMOE_DTYPE_BF16)
    return launch_narrow<NARROW_ADD, __nv_bfloat16>(b, b, a, ep, dtype, M, N, K, early, status, stream);
  return launch_narrow<NARROW_ADD, __half>(b, b, a, ep, dtype, M, N, K, early, status, stream);
}

}  // namespace fmoe
