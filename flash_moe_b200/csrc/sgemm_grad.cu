// Float32 gradients of the dense weights of a layer, on the CUDA cores: the six products behind the experts' and the router's
// backward in two launches.
//   1. dh = dy Wd, and from it and the kept products a = x Wg^T, b = x Wu^T in the epilogue
//        d[a | b] = [dh b silu'(a) | dh silu(a)],  h = silu(a) b              (flash_moe/ops/triton/flash_mlp.py:52-102)
//   2. dx += da Wg + db Wu,  d[Wg; Wu] = d[a | b]^T x,  dWd = dy^T h,  dxn = dlogits Wr,  dWr = dlogits^T xn, side by side
// As library calls (and a kernel for the activation between them) they were eight launches, and for a small step the host sets
// the pace: 500 tokens x 512 x 768, the host's part of the step 613 -> 508 us, the step 634 -> 545, the kernels 110 and 116.
//
// All have a B operand of rows of k, so one kernel takes them: 64 x 64 outputs per CTA, two groups of 64 threads on alternate
// halves of each 32-row step of k, 8 x 8 outputs per thread, cp.async ring of three steps.  The A operand lies k-major (rows of
// dab, dlogits) or m-major (columns of dab, dy, dlogits).  The longest products come first in the grid.  Bound by the reads of
// shared memory (16 floats for 64 FMAs take the 128 bytes a clock that it gives for as long as the FMAs take): 41 TF/s at
// 2048 tokens x 1024 x 4096, where the library reaches 52 with larger tiles.  Three CTAs per SM; four spill (130 us, 116).
#include "common.cuh"

namespace fmoe {
namespace {

constexpr int kTile = 64, kStep = 32, kRing = 3;
constexpr int kLdK = kStep + 4;  // k-major rows of A, padded
constexpr int kFloatsA = kTile * kLdK, kFloatsB = kStep * kTile;
constexpr int kSmemBytes = kRing * (kFloatsA + kFloatsB) * 4;
constexpr int kMaxProducts = 5;

struct GradProduct {  // C[M, N] (+)= A B, B = rows k < split of b0, then rows of b1
  const float *a, *b0, *b1;
  float* c;
  int M, N, K, split, lda, ldb, ldc;
  int a_kmajor;    // A[m][k] at m * lda + k, else at k * lda + m
  int accumulate;  // add to C
  int tiles_n, first_tile;
};
struct GradGroup {
  GradProduct p[kMaxProducts];
  int count;
};
struct SwigluGrad {
  const float *a, *b;  // [T, I]
  float *dab, *h;      // [T, 2 I], [T, I]
};

template <bool SWIGLU>
__global__ void __launch_bounds__(128, 3) grad_gemm_kernel(const __grid_constant__ GradGroup group, SwigluGrad sw) {
  extern __shared__ __align__(16) float grad_smem[];
  const int tid = threadIdx.x, half = tid >> 6, gt = tid & 63, ty = gt >> 3, tx = gt & 7;
  int which = 0;
  while (which + 1 < group.count && static_cast<int>(blockIdx.x) >= group.p[which + 1].first_tile) ++which;
  const GradProduct& g = group.p[which];
  const int tile = blockIdx.x - g.first_tile;
  const int m0 = tile / g.tiles_n * kTile, n0 = tile % g.tiles_n * kTile;
  const int steps = (g.K + kStep - 1) / kStep;
  const bool kmajor = g.a_kmajor != 0;

  auto copy = [](float* dst, const float* src, bool in, const float* any) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(in ? src : any), "r"(in ? 16 : 0)  // outside: zeros
                 : "memory");
  };
  auto fetch = [&](int step) {
    float* sa = grad_smem + step % kRing * (kFloatsA + kFloatsB);
    float* sb = sa + kFloatsA;
    const int k0 = step * kStep;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = tid + 128 * i;
      if (kmajor) {
        const int r = c >> 3, k = (c & 7) * 4;
        copy(sa + r * kLdK + k, g.a + static_cast<int64_t>(m0 + r) * g.lda + k0 + k, m0 + r < g.M && k0 + k < g.K, g.a);
      } else {
        const int k = c >> 4, m = (c & 15) * 4;
        copy(sa + k * kTile + m, g.a + static_cast<int64_t>(k0 + k) * g.lda + m0 + m, m0 + m < g.M && k0 + k < g.K, g.a);
      }
      const int k = c >> 4, n = (c & 15) * 4, row = k0 + k;
      const float* b = row < g.split ? g.b0 + static_cast<int64_t>(row) * g.ldb : g.b1 + static_cast<int64_t>(row - g.split) * g.ldb;
      copy(sb + k * kTile + n, b + n0 + n, n0 + n < g.N && row < g.K, g.b0);
    }
  };

  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  auto rank1 = [&](const float (&a)[8], const float* brow) {  // one k
    const float4 lo = *reinterpret_cast<const float4*>(brow + 4 * tx), hi = *reinterpret_cast<const float4*>(brow + 32 + 4 * tx);
    const float b[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  };
#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) {
    if (s < steps) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
    __syncthreads();  // the step has landed; the stage read one step ago is free
    if (step + kRing - 1 < steps) fetch(step + kRing - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* sa = grad_smem + step % kRing * (kFloatsA + kFloatsB);
    const float* sb = sa + kFloatsA + half * (kStep / 2) * kTile;
    if (kmajor) {
#pragma unroll
      for (int k4 = 0; k4 < kStep / 8; ++k4) {
        float4 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(sa + (ty + 8 * i) * kLdK + half * (kStep / 2) + 4 * k4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
          rank1(f, sb + (4 * k4 + kk) * kTile);
        }
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < kStep / 2; ++k) {
        const float* arow = sa + (half * (kStep / 2) + k) * kTile;
        const float4 lo = *reinterpret_cast<const float4*>(arow + 4 * ty), hi = *reinterpret_cast<const float4*>(arow + 32 + 4 * ty);
        const float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        rank1(f, sb + k * kTile);
      }
    }
  }

  // the two groups' sums meet in shared memory: group 0 finishes the rows i < 4 of each thread position, group 1 the others
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i >= 4) == (half == 0)) {
#pragma unroll
      for (int j = 0; j < 8; ++j) grad_smem[(i * 8 + j) * 64 + gt] = acc[i][j];
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if ((i >= 4) == (half == 0)) continue;
    const int m = m0 + (kmajor ? ty + 8 * i : (i >> 2) * 32 + 4 * ty + (i & 3));
    if (m >= g.M) continue;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int n = n0 + 32 * q + 4 * tx;
      if (n >= g.N) continue;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = acc[i][4 * q + j] + grad_smem[(i * 8 + 4 * q + j) * 64 + gt];
      if constexpr (SWIGLU) {
        const int64_t o = static_cast<int64_t>(m) * g.N + n;
        const float4 a4 = *reinterpret_cast<const float4*>(sw.a + o), b4 = *reinterpret_cast<const float4*>(sw.b + o);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
        float da[4], db[4], h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float sig = __fdividef(1.0f, 1.0f + __expf(-a[j]));
          const float act = a[j] * sig;
          da[j] = v[j] * b[j] * (sig * (1.0f + a[j] * (1.0f - sig)));
          db[j] = v[j] * act;
          h[j] = act * b[j];
        }
        float* row = sw.dab + static_cast<int64_t>(m) * 2 * g.N + n;
        *reinterpret_cast<float4*>(row) = make_float4(da[0], da[1], da[2], da[3]);
        *reinterpret_cast<float4*>(row + g.N) = make_float4(db[0], db[1], db[2], db[3]);
        *reinterpret_cast<float4*>(sw.h + o) = make_float4(h[0], h[1], h[2], h[3]);
      } else {
        float4* c = reinterpret_cast<float4*>(g.c + static_cast<int64_t>(m) * g.ldc + n);
        if (g.accumulate) {
          const float4 old = *c;
          v[0] += old.x;
          v[1] += old.y;
          v[2] += old.z;
          v[3] += old.w;
        }
        *c = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

}  // namespace

int launch_dense_backward_f32(const fmoe_dense_backward_args& q) {
  const int64_t T64 = q.num_tokens;
  const int H = q.hidden, I = q.intermediate, R = q.router_rows;
  if (T64 <= 0 || H <= 0 || I <= 0 || R < 0) return FMOE_ERR_BAD_ARG;
  const bool router = q.dxn != nullptr || q.drouter_w != nullptr;
  if (H % 4 != 0 || I % 4 != 0 || (router && R % 4 != 0) || T64 > (1 << 24)) return FMOE_ERR_UNSUPPORTED;
  const void* all[] = {q.dy, q.x, q.gate_pre, q.up_pre, q.gate_w, q.up_w, q.down_w, q.dab, q.h};
  for (const void* p : all)
    if (p == nullptr) return FMOE_ERR_BAD_ARG;
  if (router && (q.dlogits == nullptr || q.xn == nullptr || q.router_w == nullptr)) return FMOE_ERR_BAD_ARG;
  for (const void* p : all)
    if (!aligned16(p)) return FMOE_ERR_ALIGNMENT;
  const void* some[] = {q.dlogits, q.xn, q.router_w, q.dx, q.dxn, q.dgate_up_w, q.ddown_w, q.drouter_w};
  for (const void* p : some)
    if (!aligned16(p)) return FMOE_ERR_ALIGNMENT;
  const int T = static_cast<int>(T64);
  cudaStream_t stream = static_cast<cudaStream_t>(q.stream);
  auto f = [](const void* p) { return static_cast<const float*>(p); };
  GradGroup group{};
  int64_t tiles = 0;
  auto add = [&](const void* a, bool kmajor, int lda, const void* b0, const void* b1, int split, int ldb, void* c, bool accumulate,
                 int M, int N, int K) {
    if (c == nullptr) return;
    GradProduct& p = group.p[group.count++];
    p = GradProduct{f(a), f(b0), f(b1), static_cast<float*>(c), M, N, K, split, lda, ldb, N, kmajor, accumulate,
                    (N + kTile - 1) / kTile, static_cast<int>(tiles)};
    tiles += static_cast<int64_t>((M + kTile - 1) / kTile) * p.tiles_n;
  };
  auto go = [&](auto kern, const SwigluGrad& sw) -> int {
    if (tiles > 0x7FFFFFFF) return FMOE_ERR_UNSUPPORTED;
    FMOE_CUDA_TRY(allow_smem(kern, kSmemBytes));
    if (tiles > 0) kern<<<static_cast<unsigned>(tiles), 128, kSmemBytes, stream>>>(group, sw);
    FMOE_LAUNCH_CHECK();
    group = GradGroup{};
    tiles = 0;
    return FMOE_OK;
  };
  add(q.dy, true, H, q.down_w, q.down_w, H, I, q.h, false, T, I, H);
  int rc = go(grad_gemm_kernel<true>, SwigluGrad{f(q.gate_pre), f(q.up_pre), static_cast<float*>(q.dab), static_cast<float*>(q.h)});
  if (rc != FMOE_OK) return rc;
  add(q.dab, true, 2 * I, q.gate_w, q.up_w, I, H, q.dx, true, T, H, 2 * I);
  add(q.dab, false, 2 * I, q.x, q.x, T, H, q.dgate_up_w, false, 2 * I, H, T);
  add(q.dy, false, H, q.h, q.h, T, I, q.ddown_w, false, H, I, T);
  add(q.dlogits, true, R, q.router_w, q.router_w, R, H, q.dxn, false, T, H, R);
  add(q.dlogits, false, R, q.xn, q.xn, T, H, q.drouter_w, false, R, H, T);
  return go(grad_gemm_kernel<false>, SwigluGrad{});
}

}  // namespace fmoe
