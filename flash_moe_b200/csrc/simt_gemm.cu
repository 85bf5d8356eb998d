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
// Bound by the FMA pipe when large (one FFMA per issue slot; 8 x 8 outputs per thread need 16 LDS.128 for 256 FFMA) and
// by one CTA's chain of k-steps when small, hence the cp.async ring (operands of STAGES - 1 steps in flight) and KG
// thread groups that take alternate 16-column slices of every step and add their sums in shared memory at the end.
// With KG = 1 an output is one fmaf chain over ascending k, whatever the tile: the router's logits do not depend on the
// tile chosen.  Rows are kept as they lie in memory, padded by 4 floats (16-byte reads of 8 consecutive rows then cover
// all banks), so a thread reads 4 k of each of its rows at once.
// Measured at 256 tokens, hidden 256 (us, scalar-load 64 x 64 x 16 tiles before -> now): router logits 47 -> 10, gate/up +
// SwiGLU 29 -> 13, down 47 -> 18.
template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU>
struct SgemmCfg {
  static constexpr int TX = BN / TN, TY = BM / TM;
  static constexpr int GROUP = TX * TY;
  static constexpr int THREADS = GROUP * KG;
  static constexpr int NB = SWIGLU ? 2 : 1;
  static constexpr int KSTEP = 16 * KG;
  static constexpr int LD = KSTEP + 4;
  static constexpr int ROWS = BM + NB * BN;
  static constexpr int STAGE_FLOATS = ROWS * LD;
  static constexpr int RED_FLOATS = KG > 1 ? KG * GROUP * TM * TN * NB : 0;
  static constexpr int SMEM = (STAGES * STAGE_FLOATS > RED_FLOATS ? STAGES * STAGE_FLOATS : RED_FLOATS) * 4;
};

template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU>
__global__ void __launch_bounds__(SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU>::THREADS)
sgemm_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ B0, const float* __restrict__ B1,
             const float* __restrict__ addend, const float* __restrict__ residual, float* __restrict__ out, int64_t ldo,
             int M, int N, int K, float* __restrict__ pre_gate, float* __restrict__ pre_up) {
  using C = SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU>;
  extern __shared__ float4 sg_smem[];
  float* sm = reinterpret_cast<float*>(sg_smem);
  const int tid = threadIdx.x;
  const int group = tid / C::GROUP, gt = tid % C::GROUP;
  const int tx = gt % C::TX, ty = gt / C::TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int nsteps = (K + C::KSTEP - 1) / C::KSTEP;

  auto fetch = [&](int step) {
    float* st = sm + (step % STAGES) * C::STAGE_FLOATS;
    const int k0 = step * C::KSTEP;
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
    const float* st = sm + (step % STAGES) * C::STAGE_FLOATS + group * 16;
    const float* as = st + ty * C::LD;
    const float* bs = st + (BM + tx) * C::LD;
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
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
  if constexpr (KG == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) store(i, j, acc[0][i][j], acc[C::NB - 1][i][j]);
  } else {
    // every group leaves its sums in shared memory and finishes the rows i = group, group + KG, ...
    static_assert(TM % KG == 0, "rows are dealt to the groups");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int b = 0; b < C::NB; ++b)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sm[(((b * TM + i) * TN + j) * KG + group) * C::GROUP + gt] = acc[b][i][j];
    __syncthreads();
#pragma unroll
    for (int ii = 0; ii < TM / KG; ++ii) {
      const int i = group + ii * KG;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        float v[2] = {0.f, 0.f};
#pragma unroll
        for (int b = 0; b < C::NB; ++b)
#pragma unroll
          for (int g = 0; g < KG; ++g) v[b] += sm[(((b * TM + i) * TN + j) * KG + g) * C::GROUP + gt];
        store(i, j, v[0], v[1]);
      }
    }
  }
}

template <int BM, int BN, int TM, int TN, int KG, int STAGES, bool SWIGLU>
int run_sgemm(const float* a, int64_t lda, const float* b0, const float* b1, const float* addend, float* out, int64_t ldo,
              int64_t M, int N, int K, cudaStream_t stream, const float* residual, float* pre_gate, float* pre_up) {
  using C = SgemmCfg<BM, BN, TM, TN, KG, STAGES, SWIGLU>;
  auto kern = sgemm_kernel<BM, BN, TM, TN, KG, STAGES, SWIGLU>;
  FMOE_CUDA_TRY(allow_smem(kern, C::SMEM));
  kern<<<dim3((N + BN - 1) / BN, static_cast<unsigned>((M + BM - 1) / BM)), C::THREADS, C::SMEM, stream>>>(
      a, lda, b0, b1, addend, residual, out, ldo, static_cast<int>(M), N, K, pre_gate, pre_up);
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}

// Tile by the number of tiles: the largest whose grid still covers the SMs.  `ordered` (the router's logits) keeps K
// unsplit.
template <bool SWIGLU>
int pick_sgemm(const float* a, int64_t lda, const float* b0, const float* b1, const float* addend, float* out,
               int64_t ldo, bool ordered, int64_t M, int N, int K, cudaStream_t stream, const float* residual,
               float* pre_gate, float* pre_up) {
  const int64_t sms = device_sm_count();
  auto tiles = [&](int bm, int bn) { return ((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  constexpr int WIDE = SWIGLU ? 64 : 128;  // both operands of the SwiGLU count as columns
  if (tiles(128, WIDE) >= sms)
    return run_sgemm<128, WIDE, 8, WIDE / 16, 1, 4, SWIGLU>(a, lda, b0, b1, addend, out, ldo, M, N, K, stream, residual, pre_gate,
                                                      pre_up);
  if (ordered) return run_sgemm<32, 32, 2, 4, 1, 6, SWIGLU>(a, lda, b0, b1, addend, out, ldo, M, N, K, stream, residual,
                                                            pre_gate, pre_up);
  if (tiles(64, 64) >= sms)
    return run_sgemm<64, 64, 4, SWIGLU ? 4 : 8, 2, 4, SWIGLU>(a, lda, b0, b1, addend, out, ldo, M, N, K, stream, residual,
                                                              pre_gate, pre_up);
  return run_sgemm<32, 32, 4, 4, 4, 4, SWIGLU>(a, lda, b0, b1, addend, out, ldo, M, N, K, stream, residual, pre_gate, pre_up);
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
