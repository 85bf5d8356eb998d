// Backward kernels of the router op and of the SwiGLU activation (sm_100a).  The expert op's backward lives
// with its forward in expert.cu.
#include <type_traits>

#include "common.cuh"

namespace fmoe {
namespace {

// d log_probs[h, t, c] = sum over the token's selected slots j whose sub-key of half h is c of dscores[t, j]
// (flash_moe/ops/triton/flash_router.py:197-249 scatters with atomics in the gradient's dtype; here every
// output element is a float32 sum over the slots in ascending j, rounded once).
template <typename T>
__global__ void __launch_bounds__(128) router_bwd_kernel(const T* __restrict__ dscores, const int64_t* __restrict__ idx,
                                                         T* __restrict__ dlogp, int64_t ntok, int nk, int k) {
  extern __shared__ unsigned char smem_raw[];
  float* ds = reinterpret_cast<float*>(smem_raw);  // [k]
  int* ix = reinterpret_cast<int*>(ds + k);        // [k]
  int* iy = ix + k;                                // [k]
  for (int64_t t = blockIdx.x; t < ntok; t += gridDim.x) {
    __syncthreads();
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
      const int64_t e = idx[t * k + j];
      const bool ok = e >= 0 && e < static_cast<int64_t>(nk) * nk;
      ds[j] = ok ? to_f32<T>(dscores[t * k + j]) : 0.f;
      ix[j] = ok ? static_cast<int>(e / nk) : -1;
      iy[j] = ok ? static_cast<int>(e % nk) : -1;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * nk; c += blockDim.x) {
      const int half = c >= nk ? 1 : 0;
      const int key = c - half * nk;
      const int* sel = half ? iy : ix;
      float acc = 0.f;
      for (int j = 0; j < k; ++j)
        if (sel[j] == key) acc += ds[j];
      dlogp[(static_cast<int64_t>(half) * ntok + t) * nk + key] = from_f32<T>(acc);
    }
  }
}

// One warp per token: the whole chain from the gradients of the gates back to the router logits.
//   gates g = exp(s):                    ds_j = dg_j g_j
//   gates G = g / sum(g) (renormalised): ds_j = G_j (dG_j - sum_i dG_i G_i)
//   top-k: d lp[h, c] = sum of ds_j over the slots whose sub-key of half h is c (float32, ascending j)
//   log-softmax: dl[h, c] = d lp[h, c] - exp(lp[h, c]) sum_c d lp[h, c], and that sum is the sum of all ds_j
// (flash_moe/ops/triton/flash_router.py:197-249 and torch's exp / div / log_softmax nodes around it: nine kernels, one of
// which walked all slots for each of the 2 nk sums, 20 us at 4096 tokens x 128 keys, top-64).
template <typename T>
__global__ void __launch_bounds__(128) router_chain_bwd_kernel(const T* __restrict__ dgates, const T* __restrict__ gates,
                                                               const int64_t* __restrict__ idx, const T* __restrict__ logp,
                                                               T* __restrict__ dlogits, int64_t ntok, int nk, int k, int norm) {
  extern __shared__ float chain_smem[];
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  float* acc = chain_smem + (threadIdx.x >> 5) * 2 * nk;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < ntok; t += warps_total) {
    for (int c = lane; c < 2 * nk; c += 32) acc[c] = 0.f;
    float dot = 0.f;
    if (norm) {
      for (int j = lane; j < k; j += 32) dot = fmaf(to_f32<T>(dgates[t * k + j]), to_f32<T>(gates[t * k + j]), dot);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(kAll, dot, d);
    }
    float total = 0.f;
    __syncwarp();
    for (int j0 = 0; j0 < k; j0 += 32) {
      const int j = j0 + lane;
      float ds = 0.f;
      int key = 0;  // first sub-key | second sub-key << 16
      if (j < k) {
        const int64_t e = idx[t * k + j];
        if (e >= 0 && e < static_cast<int64_t>(nk) * nk) {
          const int first = static_cast<int>(static_cast<uint32_t>(e) / static_cast<uint32_t>(nk));
          key = first | ((static_cast<int>(e) - first * nk) << 16);
          ds = to_f32<T>(gates[t * k + j]) * (to_f32<T>(dgates[t * k + j]) - dot);
        }
      }
      total += ds;
      const int n = min(32, k - j0);
      for (int i = 0; i < n; ++i) {  // one slot at a time: lane 0 its first sub-key, lane 1 its second
        const float v = __shfl_sync(kAll, ds, i);
        const int kk = __shfl_sync(kAll, key, i);
        if (lane < 2) acc[lane == 0 ? kk & 0xFFFF : nk + (kk >> 16)] += v;
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(kAll, total, d);
    __syncwarp();
    for (int c = lane; c < 2 * nk; c += 32)
      dlogits[t * 2 * nk + c] = from_f32<T>(acc[c] - expf(to_f32<T>(logp[t * 2 * nk + c])) * total);
    __syncwarp();
  }
}

// h = silu(a) * b;  da = dh * b * silu'(a);  db = dh * silu(a)   (flash_moe/ops/triton/flash_mlp.py:52-102)
template <typename T>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const T* __restrict__ dh, const T* __restrict__ a,
                                                         const T* __restrict__ b, T* __restrict__ da,
                                                         T* __restrict__ db, T* __restrict__ h, int64_t nvec, int row_vecs) {
  constexpr int VEC = Vec16<T>::N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    // row_vecs > 0: da and db are the two halves of rows twice as long (one weight-gradient GEMM reads both)
    const int64_t o = row_vecs > 0 ? i + i / row_vecs * row_vecs : i;
    float fd[VEC], fa[VEC], fb[VEC], oa[VEC], ob[VEC], oh[VEC];
    unpack16<T>(ldg16(dh + i * VEC), fd);
    unpack16<T>(ldg16(a + i * VEC), fa);
    unpack16<T>(ldg16(b + i * VEC), fb);
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const float sig = __fdividef(1.0f, 1.0f + __expf(-fa[j]));
      const float act = fa[j] * sig;
      oa[j] = fd[j] * fb[j] * (sig * (1.0f + fa[j] * (1.0f - sig)));
      ob[j] = fd[j] * act;
      oh[j] = act * fb[j];
    }
    *reinterpret_cast<uint4*>(da + o * VEC) = pack16<T>(oa);
    *reinterpret_cast<uint4*>(db + o * VEC) = pack16<T>(ob);
    if (h != nullptr) *reinterpret_cast<uint4*>(h + i * VEC) = pack16<T>(oh);
  }
}

template <typename T>
int router_bwd_typed(const void* dscores, const int64_t* idx, void* dlogp, int64_t ntok, int nk, int k,
                     cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(k) * 12;
  auto kern = router_bwd_kernel<T>;
  FMOE_CUDA_TRY(allow_smem(kern, static_cast<int>(smem)));
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 16;
  const int grid = static_cast<int>(ntok < cap ? ntok : cap);
  kern<<<grid, 128, smem, stream>>>(static_cast<const T*>(dscores), idx, static_cast<T*>(dlogp), ntok, nk, k);
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}

template <typename T>
int swiglu_bwd_typed(const void* dh, const void* a, const void* b, void* da, void* db, void* h, int64_t n, int64_t row,
                     cudaStream_t stream) {
  constexpr int VEC = Vec16<T>::N;
  const int64_t nvec = n / VEC;
  const int64_t want = (nvec + 255) / 256;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 16;
  const int grid = static_cast<int>(want < cap ? want : cap);
  swiglu_bwd_kernel<T><<<grid, 256, 0, stream>>>(static_cast<const T*>(dh), static_cast<const T*>(a),
                                                 static_cast<const T*>(b), static_cast<T*>(da), static_cast<T*>(db),
                                                 static_cast<T*>(h), nvec, static_cast<int>(row / VEC));
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}

}  // namespace

int launch_router_topk_backward(const void* dscores, const int64_t* indices, int dtype, int64_t T, int nk, int k,
                                void* dlog_probs, cudaStream_t stream) {
  if (T < 0 || nk <= 0 || k < 0 || k > nk) return FMOE_ERR_BAD_ARG;
  if (T == 0) return FMOE_OK;
  if (dlog_probs == nullptr || (k > 0 && (dscores == nullptr || indices == nullptr))) return FMOE_ERR_BAD_ARG;
  if (static_cast<size_t>(k) * 12 > 200 * 1024) return FMOE_ERR_UNSUPPORTED;
  switch (dtype) {
    case FMOE_DTYPE_F32: return router_bwd_typed<float>(dscores, indices, dlog_probs, T, nk, k, stream);
    case FMOE_DTYPE_BF16: return router_bwd_typed<__nv_bfloat16>(dscores, indices, dlog_probs, T, nk, k, stream);
    case FMOE_DTYPE_F16: return router_bwd_typed<__half>(dscores, indices, dlog_probs, T, nk, k, stream);
    default: return FMOE_ERR_BAD_ARG;
  }
}

int launch_router_chain_backward(const void* dgates, const void* gates, const int64_t* indices, const void* log_probs,
                                 void* dlogits, int dtype, int64_t T, int nk, int k, int norm, cudaStream_t stream) {
  if (T <= 0) return FMOE_OK;
  // The float32 sums of a CTA's tokens, one per warp, sit in shared memory: four tokens up to 6144 keys, fewer above.  One
  // fits up to 28672 keys, far beyond the 8192 or so that the forward's top-k takes.
  constexpr int kMaxSmem = 224 * 1024;
  int warps = 4;
  while (warps > 1 && static_cast<int64_t>(warps) * 8 * nk > (192 << 10)) warps >>= 1;
  if (static_cast<int64_t>(warps) * 8 * nk > kMaxSmem) return FMOE_ERR_UNSUPPORTED;
  const int smem = warps * 8 * nk;
  const int64_t want = (T + warps - 1) / warps;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 16;
  const int grid = static_cast<int>(want < cap ? want : cap);
  auto go = [&](auto kern, auto* tag) -> int {
    using P = decltype(tag);
    FMOE_CUDA_TRY(allow_smem(kern, smem));
    kern<<<grid, warps * 32, smem, stream>>>(static_cast<P>(dgates), static_cast<P>(gates), indices,
                                             static_cast<P>(log_probs),
                                             static_cast<std::remove_const_t<std::remove_pointer_t<P>>*>(dlogits), T, nk, k,
                                             norm);
    FMOE_LAUNCH_CHECK();
    return FMOE_OK;
  };
  switch (dtype) {
    case FMOE_DTYPE_F32: return go(router_chain_bwd_kernel<float>, static_cast<const float*>(nullptr));
    case FMOE_DTYPE_BF16: return go(router_chain_bwd_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(nullptr));
    case FMOE_DTYPE_F16: return go(router_chain_bwd_kernel<__half>, static_cast<const __half*>(nullptr));
    default: return FMOE_ERR_BAD_ARG;
  }
}

int launch_swiglu_backward(const void* dh, const void* a, const void* b, void* da, void* db, void* h, int dtype,
                           int64_t n, int64_t row, cudaStream_t stream) {
  if (dtype != FMOE_DTYPE_F32 && dtype != FMOE_DTYPE_BF16 && dtype != FMOE_DTYPE_F16) return FMOE_ERR_BAD_ARG;
  if (n < 0) return FMOE_ERR_BAD_ARG;
  if (n == 0) return FMOE_OK;
  if (dh == nullptr || a == nullptr || b == nullptr || da == nullptr || db == nullptr) return FMOE_ERR_BAD_ARG;
  if (n % (16 / dtype_size(dtype)) != 0 || row < 0 || row % (16 / dtype_size(dtype)) != 0) return FMOE_ERR_ALIGNMENT;
  if (!aligned16(dh) || !aligned16(a) || !aligned16(b) || !aligned16(da) || !aligned16(db) || !aligned16(h))
    return FMOE_ERR_ALIGNMENT;
  switch (dtype) {
    case FMOE_DTYPE_F32: return swiglu_bwd_typed<float>(dh, a, b, da, db, h, n, row, stream);
    case FMOE_DTYPE_BF16: return swiglu_bwd_typed<__nv_bfloat16>(dh, a, b, da, db, h, n, row, stream);
    case FMOE_DTYPE_F16: return swiglu_bwd_typed<__half>(dh, a, b, da, db, h, n, row, stream);
    default: return FMOE_ERR_BAD_ARG;
  }
}

}  // namespace fmoe
