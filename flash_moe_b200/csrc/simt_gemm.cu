// C[M, N] = A[M, K] * B[N, K]^T with fp32 FMA accumulation on the CUDA cores.
// Used where the tensor-core path does not apply: float32 modules (tcgen05 has no fp32-exact
// mode) and operand shapes TMA cannot address (K not a multiple of 8 elements).  Same fused
// epilogues as the tcgen05 kernels: plain store (+ optional fp32 addend) and SwiGLU.
//
//   sgemm_kernel      float32 rows of whole 16-byte pieces: cp.async ring, register tiles, optional split of K over
//                     the warps of a CTA
//   simt_gemm_kernel  everything else (16-bit operands, rows that are not whole 16-byte pieces)
#include "common.cuh"

namespace fmoe {
namespace {

// ---------------------------------------------------------------- float32, 16-byte aligned rows
// Bound by the FMA pipe when large (8 x 8 outputs per thread need 16 LDS.128 for 256 FFMA; 37 TF/s measured, packed f32x2
// FMAs gave the same) and by one CTA's chain of k-steps when small, hence the cp.async ring (operands of STAGES - 1 steps in
// flight), KG thread groups that take alternate 16-column slices of every step (KSL of them each) and a cluster of S CTAs
// that share the k-steps of a tile; the partial sums meet in (distributed) shared memory at the end.  CTAS bounds the
// registers so that so many fit an SM: 16 warps instead of 8 hide the reads of the operands.
// With KG = S = 1 an output is one fmaf chain over ascending k, whatever the tile: the router's logits do not depend on the
// tile chosen.  Rows are kept as they lie in memory, padded by 4 floats (16-byte reads of 8 consecutive rows then cover
// all banks), so a thread reads 4 k of each of its rows at once.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, int rank) {  // the word at `addr` of this CTA, in CTA `rank`
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU, int KSL, int S, int CTAS>
struct SgemmCfg {
  static constexpr int TX = BN / TN, TY = BM / TM;
  static constexpr int GROUP = TX * TY;
  static constexpr int THREADS = GROUP * KG;
  static constexpr int NB = SWIGLU ? 2 : 1;
  static constexpr int KSTEP = 16 * KG * KSL;
  static constexpr int LD = KSTEP + 4;
  static constexpr int ROWS = BM + NB * BN;
  static constexpr int STAGE_FLOATS = ROWS * LD;
  static constexpr int RED_FLOATS = KG * S > 1 ? KG * GROUP * TM * TN * NB : 0;
  static constexpr int SMEM = (STAGES * STAGE_FLOATS > RED_FLOATS ? STAGES * STAGE_FLOATS : RED_FLOATS) * 4;
};

template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU, int KSL, int S, int CTAS>
__global__ void __launch_bounds__(SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU, KSL, S, CTAS>::THREADS, CTAS)
sgemm_kernel(const float* A, int64_t lda, const float* __restrict__ B0, const float* __restrict__ B1,
             const float* addend, const float* residual, float* __restrict__ out, int64_t ldo,
             int M, int N, int K, float* __restrict__ pre_gate, float* __restrict__ pre_up) {
  using C = SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU, KSL, S, CTAS>;
  extern __shared__ float4 sg_smem[];
  float* sm = reinterpret_cast<float*>(sg_smem);
  const int tid = threadIdx.x;
  const int group = tid / C::GROUP, gt = tid % C::GROUP;
  // a warp covers 8 columns x 4 rows of threads where the group has them: its reads of both operands are then at most 128
  // different bytes
  constexpr bool BLOCKED = C::TX % 8 == 0 && C::TY % 4 == 0;
  const int tx = BLOCKED ? (gt / 32) % (C::TX / 8) * 8 + gt % 8 : gt % C::TX;
  const int ty = BLOCKED ? (gt / 32) / (C::TX / 8) * 4 + gt % 32 / 8 : gt / C::TX;
  const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / S) * BN;
  // S > 1: the cluster's CTAs share a tile, each with a run of the k-steps
  const int all_steps = (K + C::KSTEP - 1) / C::KSTEP;
  const int per_cta = (all_steps + S - 1) / S;
  const int rank = S > 1 ? static_cast<int>(blockIdx.x) % S : 0;
  const int step0 = rank * per_cta;
  const int nsteps = max(0, min(per_cta, all_steps - step0));

  auto fetch = [&](int step) {
    float* st = sm + (step % STAGES) * C::STAGE_FLOATS;
    const int k0 = (step0 + step) * C::KSTEP;
    constexpr int PIECES = C::KSTEP / 4;
    for (int c = tid; c < C::ROWS * PIECES; c += C::THREADS) {
      const int r = c / PIECES, kc = k0 + (c % PIECES) * 4;
      const float* src;
      bool in = kc < K;
      if (r < BM) {
        in = in && m0 + r < M;
        src = A + static_cast<int64_t>(m0 + r) * lda + kc;
      } else {
        const int br = (r - BM) % BN;
        in = in && n0 + br < N;
        src = (SWIGLU && r - BM >= BN ? B1 : B0) + static_cast<int64_t>(n0 + br) * K + kc;
      }
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(st + r * C::LD + (c % PIECES) * 4));
      const int bytes = in ? 16 : 0;  // the rest of the piece is filled with zeros
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? src : A), "r"(bytes) : "memory");
    }
  };

  float acc[C::NB][TM][TN];
#pragma unroll
  for (int b = 0; b < C::NB; ++b)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[b][i][j] = 0.f;

  pdl_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nsteps) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int step = 0; step < nsteps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // the step's rows have landed; the stage read one step ago is free
    if (step + STAGES - 1 < nsteps) fetch(step + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* st = sm + (step % STAGES) * C::STAGE_FLOATS;
    const float* as = st + ty * C::LD;
    const float* bs = st + (BM + tx) * C::LD;
#pragma unroll
    for (int p = 0; p < 4 * KSL; ++p) {
      const int k4 = ((p / 4) * KG + group) * 4 + p % 4;
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * C::TY * C::LD + k4 * 4);
#pragma unroll
      for (int b = 0; b < C::NB; ++b)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(bs + (b * BN + j * C::TX) * C::LD + k4 * 4);
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            float& c = acc[b][i][j];
            c = fmaf(a[i].x, v.x, c);
            c = fmaf(a[i].y, v.y, c);
            c = fmaf(a[i].z, v.z, c);
            c = fmaf(a[i].w, v.w, c);
          }
        }
    }
  }

  pdl_launch_dependents();
  auto store = [&](int i, int j, float v, float u) {
    const int m = m0 + ty + i * C::TY, n = n0 + tx + j * C::TX;
    if (m >= M || n >= N) return;
    const int64_t o = static_cast<int64_t>(m) * ldo + n;
    if (SWIGLU) {
      if (pre_gate != nullptr) {
        pre_gate[o] = v;
        pre_up[o] = u;
      }
      v = (v / (1.0f + expf(-v))) * u;
    } else {
      if (addend != nullptr) v += addend[o];
      if (residual != nullptr) v += residual[o];
    }
    out[o] = v;
  };
  if constexpr (KG * S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) store(i, j, acc[0][i][j], acc[C::NB - 1][i][j]);
  } else {
    // every group leaves its sums in shared memory; output (i, j) of a thread position is finished by group i % KG of the
    // CTA with rank j % S, over the ranks and groups in order
    static_assert(TM % KG == 0 && TN % S == 0, "outputs are dealt to the groups and the CTAs of the cluster");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int b = 0; b < C::NB; ++b)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sm[(((b * TM + i) * TN + j) * KG + group) * C::GROUP + gt] = acc[b][i][j];
    if constexpr (S > 1) {
      cluster_barrier();
    } else {
      __syncthreads();
    }
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
#pragma unroll
    for (int ii = 0; ii < TM / KG; ++ii) {
      const int i = group + ii * KG;
#pragma unroll
      for (int jj = 0; jj < TN / S; ++jj) {
        const int j = rank + jj * S;
        float v[2] = {0.f, 0.f};
#pragma unroll
        for (int b = 0; b < C::NB; ++b) {
          float part[S][KG];
#pragma unroll
          for (int r = 0; r < S; ++r)
#pragma unroll
            for (int g = 0; g < KG; ++g) {
              const int at = (((b * TM + i) * TN + j) * KG + g) * C::GROUP + gt;
              if constexpr (S > 1)
                part[r][g] = ld_cluster(base + at * 4, r);
              else
                part[r][g] = sm[at];
            }
#pragma unroll
          for (int r = 0; r < S; ++r)
#pragma unroll
            for (int g = 0; g < KG; ++g) v[b] += part[r][g];
        }
        store(i, j, v[0], v[1]);
      }
    }
    if constexpr (S > 1) cluster_barrier();  // the other CTAs have read this one's sums
  }
}

template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU, int KSL, int S, int CTAS>
int run_sgemm(const float* a, int64_t lda, const float* b0, const float* b1, const float* addend, float* out, int64_t ldo,
              int64_t M, int N, int K, cudaStream_t stream, const float* residual, float* pre_gate, float* pre_up) {
  using C = SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU, KSL, S, CTAS>;
  auto kern = sgemm_kernel<BM, BN, TM, TN, KG, STAGES, SWIGLU, KSL, S, CTAS>;
  FMOE_CUDA_TRY(allow_smem(kern, C::SMEM));
  FMOE_CUDA_TRY(launch_pdl(16, kern, dim3(static_cast<unsigned>((N + BN - 1) / BN) * S, static_cast<unsigned>((M + BM - 1) / BM)),
                           dim3(C::THREADS), C::SMEM, stream, S, a, lda, b0, b1, addend, residual, out, ldo,
                           static_cast<int>(M), N, K, pre_gate, pre_up));
  return FMOE_OK;
}

// Tile and split by what the busiest SM has to do: multiply-adds of its share of the CTAs (k rounded to whole steps), over
// the rate that a tile reaches of the 64 a clock of plain FMAs (1.1, 0.98 and 0.8 of that at 128, 64 and 32 rows - the small
// tiles read more operands per FMA - and a quarter less while the SM has one CTA), plus each CTA's start and the exchange of a split.
// `ordered` (the router's logits) keeps K unsplit.
// Measured (us, tile by the number of tiles alone, K split inside a CTA only -> now): 256 tokens, hidden 256, 1024 columns:
// logits 10 -> 5, down 18 -> 10; 200 x 800 x 5000: gate/up 200 -> 131; 1000 x 512 x 2000: down 99 -> 78.
template <bool SWIGLU>
int pick_sgemm(const float* a, int64_t lda, const float* b0, const float* b1, const float* addend, float* out,
               int64_t ldo, bool ordered, int64_t M, int N, int K, cudaStream_t stream, const float* residual,
               float* pre_gate, float* pre_up) {
  constexpr int NB = SWIGLU ? 2 : 1;  // both operands of the SwiGLU count as columns
  const int64_t sms = device_sm_count();
  auto tiles = [&](int bm, int bn) { return ((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
#define FMOE_SGEMM(...) \
  run_sgemm<__VA_ARGS__>(a, lda, b0, b1, addend, out, ldo, M, N, K, stream, residual, pre_gate, pre_up)
  if (ordered) {
    if (tiles(128, 128 / NB) >= sms) return FMOE_SGEMM(128, 128 / NB, 8, 8 / NB, 1, 4, SWIGLU, 1, 1, 2);
    if (tiles(32, 32) * 2 <= sms) return FMOE_SGEMM(16, 16, 1, 1, 1, 4, SWIGLU, 4, 1, 1);
    return FMOE_SGEMM(32, 32, 2, 4, 1, 6, SWIGLU, 1, 1, 1);
  }
  auto cost = [&](int bm, int bn, int kstep, int split, double rate) {
    if ((M + bm - 1) / bm > 65535) return 1e30;  // rows of tiles are the grid's second dimension
    const int64_t ctas = (tiles(bm, bn) * split + sms - 1) / sms;
    const int64_t steps = (K + kstep - 1) / kstep;
    const double macs = static_cast<double>(ctas) * bm * bn * NB * ((steps + split - 1) / split * kstep);
    return macs / (64.0 * rate * (ctas == 1 ? 0.75 : 1.0)) + (split > 1 ? 3000.0 + 1200.0 * ctas : 600.0 * ctas);
  };
  const double c[5] = {cost(128, 128 / NB, 16, 1, 1.1), cost(64, 64 / NB, 64, 2, 0.98), cost(32, 32, 64, 1, 0.8),
                       cost(32, 32, 64, 2, 0.8), cost(32, 32, 64, 4, 0.8)};
  int best = 0;
  for (int i = 1; i < 5; ++i)
    if (c[i] < c[best]) best = i;
  switch (best) {
    case 0: return FMOE_SGEMM(128, 128 / NB, 8, 8 / NB, 1, 4, SWIGLU, 1, 1, 2);
    case 1: return FMOE_SGEMM(64, 64 / NB, 8, 8 / NB, 4, 3, SWIGLU, 1, 2, 2);
    case 2: return FMOE_SGEMM(32, 32, 4, 4, 4, 4, SWIGLU, 1, 1, 1);
    case 3: return FMOE_SGEMM(32, 32, 4, 4, 4, 4, SWIGLU, 1, 2, 1);
    default: return FMOE_SGEMM(32, 32, 4, 4, 4, 4, SWIGLU, 1, 4, 1);
  }
#undef FMOE_SGEMM
}

// ---------------------------------------------------------------- any type, any alignment

constexpr int TM = 64, TN = 64, TK = 16;

template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(256) simt_gemm_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ B0,
                                                       const T* __restrict__ B1, int64_t ldb,
                                                       const float* __restrict__ addend,
                                                       const T* __restrict__ residual, T* __restrict__ out,
                                                       int64_t ldo, int M, int N, int K) {
  __shared__ float As[TK][TM + 4];
  __shared__ float Bs0[TK][TN + 4];
  __shared__ float Bs1[SWIGLU ? TK : 1][TN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  float acc0[4][4] = {}, acc1[4][4] = {};
  const int lr = tid >> 2;        // 0..63: row of the tile this thread stages
  const int lk = (tid & 3) * 4;   // 0,4,8,12
  for (int k0 = 0; k0 < K; k0 += TK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int kk = k0 + lk + j;
      const int am = m0 + lr, bn = n0 + lr;
      As[lk + j][lr] = (am < M && kk < K) ? to_f32<T>(A[static_cast<int64_t>(am) * lda + kk]) : 0.f;
      Bs0[lk + j][lr] = (bn < N && kk < K) ? to_f32<T>(B0[static_cast<int64_t>(bn) * ldb + kk]) : 0.f;
      if (SWIGLU) Bs1[lk + j][lr] = (bn < N && kk < K) ? to_f32<T>(B1[static_cast<int64_t>(bn) * ldb + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      float a[4], b[4], c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs0[k][tx * 4 + j];
      if (SWIGLU) {
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = Bs1[k][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc0[i][j] = fmaf(a[i], b[j], acc0[i][j]);
          if (SWIGLU) acc1[i][j] = fmaf(a[i], c[j], acc1[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc0[i][j];
      if (SWIGLU) {
        v = (v / (1.0f + expf(-v))) * acc1[i][j];
      } else {
        if (addend != nullptr) v += addend[static_cast<int64_t>(m) * ldo + n];
        if (residual != nullptr) v += to_f32<T>(residual[static_cast<int64_t>(m) * ldo + n]);
      }
      out[static_cast<int64_t>(m) * ldo + n] = from_f32<T>(v);
    }
  }
}

template <typename T>
int run(const void* a, int64_t lda, const void* b0, const void* b1, const float* addend, void* out, int64_t ldo,
        int swiglu, int64_t M, int N, int K, cudaStream_t stream, const void* residual) {
  dim3 grid((N + TN - 1) / TN, static_cast<unsigned>((M + TM - 1) / TM));
  if (swiglu)
    simt_gemm_kernel<T, true><<<grid, 256, 0, stream>>>(static_cast<const T*>(a), lda, static_cast<const T*>(b0),
                                                        static_cast<const T*>(b1), K, nullptr, nullptr,
                                                        static_cast<T*>(out), ldo, static_cast<int>(M), N, K);
  else
    simt_gemm_kernel<T, false><<<grid, 256, 0, stream>>>(static_cast<const T*>(a), lda, static_cast<const T*>(b0),
                                                         nullptr, K, addend, static_cast<const T*>(residual),
                                                         static_cast<T*>(out), ldo, static_cast<int>(M), N, K);
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}

}  // namespace

int launch_simt_gemm(const void* a, int64_t lda, const void* b0, const void* b1, const float* addend, void* out,
                     int64_t ldo, int dtype, int swiglu, int64_t M, int N, int K, cudaStream_t stream,
                     const void* residual, bool ordered, void* pre_gate, void* pre_up) {
  if (a == nullptr || b0 == nullptr || out == nullptr || (swiglu && b1 == nullptr)) return FMOE_ERR_BAD_ARG;
  if (M <= 0 || N <= 0 || K <= 0 || M > 0x7FFFFFFFll - TM || (M + TM - 1) / TM > 65535) return FMOE_ERR_UNSUPPORTED;
  const bool rows16 = dtype == FMOE_DTYPE_F32 && K % 4 == 0 && lda % 4 == 0 && aligned16(a) && aligned16(b0) &&
                      (b1 == nullptr || aligned16(b1));
  if (rows16) {
    const float *af = static_cast<const float*>(a), *bf = static_cast<const float*>(b0), *cf = static_cast<const float*>(b1);
    const float* rf = static_cast<const float*>(residual);
    float* of = static_cast<float*>(out);
    return swiglu ? pick_sgemm<true>(af, lda, bf, cf, nullptr, of, ldo, ordered, M, N, K, stream, nullptr,
                                     static_cast<float*>(pre_gate), static_cast<float*>(pre_up))
                  : pick_sgemm<false>(af, lda, bf, nullptr, addend, of, ldo, ordered, M, N, K, stream, rf, nullptr, nullptr);
  }
  if (pre_gate != nullptr || pre_up != nullptr) return FMOE_ERR_UNSUPPORTED;  // only the kernel above keeps them
  switch (dtype) {
    case FMOE_DTYPE_F32: return run<float>(a, lda, b0, b1, addend, out, ldo, swiglu, M, N, K, stream, residual);
    case FMOE_DTYPE_BF16: return run<__nv_bfloat16>(a, lda, b0, b1, addend, out, ldo, swiglu, M, N, K, stream, residual);
    case FMOE_DTYPE_F16: return run<__half>(a, lda, b0, b1, addend, out, ldo, swiglu, M, N, K, stream, residual);
    default: return FMOE_ERR_BAD_ARG;
  }
}

}  // namespace fmoe
