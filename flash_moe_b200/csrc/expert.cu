// Fine-grained expert forward for sm_100a:
//   out[t] = sum_j silu(<x[t], D[e_tj]>) * g[t,j] * U[e_tj]
// (flash_moe/ops/triton/flash_expert.py:13-211, preprocessing :528-577).
//
// Per token, no sort, in two passes:
//   2. scores: gs = silu(<x[t], D[e]>) * gate per (token, slot) - 16-bit tables on the tensor cores (mma.sync, groups of 16
//      gathered down rows against the token's x row), float32 with FMAs - stored at the pair's position (4 bytes a pair);
//   3. accumulate: out[t] = sum_j gs[t,j] * U[e_tj] in fp32 (packed f32x2 FMAs), fixed slot order, one rounding on
//      store - no atomics, run-to-run deterministic.
// Both have a form for few tokens that spreads one task over the warps of a CTA.  Ids outside [0, N) are skipped and
// flagged.  (A single kernel that streamed the rows of both steps through shared memory was the faster one for tables of
// 1 GiB and more until the scores pass read whole lines: 32768 tokens x 2048, 2^20 experts, Zipf 1.1 ids 562 us against 391
// now, uniform ids 675 against 683.)

#include "common.cuh"
#include "warp_sort.cuh"

namespace fmoe {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// ---------------------------------------------------------------- 1. segment offsets (backward)
__device__ __forceinline__ int block_reduce_sum(int v, int* sh) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  int tot = 0;
  for (int w = 0; w < (blockDim.x >> 5); ++w) tot += sh[w];
  __syncthreads();
  return tot;
}

__global__ void __launch_bounds__(kScanThreads) scan_tile_sums_kernel(const int* __restrict__ counts, int64_t N,
                                                                     int* __restrict__ tile_sums) {
  __shared__ int sh[kScanThreads / 32];
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile;
  int v = 0;
  for (int i = threadIdx.x; i < kScanTile; i += kScanThreads)
    if (base + i < N) v += counts[base + i];
  const int tot = block_reduce_sum(v, sh);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

// offsets[i] = sum(counts[0..i)), offsets[N] = total.  tile_sums == nullptr: the prefix of the
// preceding tiles is recomputed from counts (cheap when there are only a few tiles).
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const int* __restrict__ counts, int64_t N,
                                                                  const int* __restrict__ tile_sums,
                                                                  int* __restrict__ offsets) {
  __shared__ int sh[kScanThreads / 32];
  __shared__ int warp_pref[kScanThreads / 32];
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile;
  int v = 0;
  if (tile_sums != nullptr) {
    for (int i = threadIdx.x; i < static_cast<int>(blockIdx.x); i += kScanThreads) v += tile_sums[i];
  } else {
    for (int64_t i = threadIdx.x; i < base; i += kScanThreads) v += counts[i];
  }
  const int prefix = block_reduce_sum(v, sh);

  int item[kScanItems];
  int tsum = 0;
  const int64_t first = base + static_cast<int64_t>(threadIdx.x) * kScanItems;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    item[i] = (first + i < N) ? counts[first + i] : 0;
    tsum += item[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = tsum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) warp_pref[warp] = incl;
  __syncthreads();
  int wbase = 0;
  for (int w = 0; w < warp; ++w) wbase += warp_pref[w];
  int run = prefix + wbase + incl - tsum;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (first + i < N) offsets[first + i] = run;
    run += item[i];
    if (first + i == N - 1) offsets[N] = run;
  }
}

// ---------------------------------------------------------------- 2b. scores per token on mma.sync
// Token-centric scores for 16-bit dtypes, no sort.  Groups of 16 of a token's experts form the A operand (their down rows,
// gathered with 128-bit loads), the token's x row is every column of B, so each accumulator
// column holds <x, D[e]> for the 16 rows (fp32 accumulate).  The k index inside a 32-column
// block is permuted identically for A and B so that every thread's 16-byte load feeds two MMAs.
template <typename T> struct Mma16816;
template <> struct Mma16816<__nv_bfloat16> {
  static __device__ __forceinline__ void run(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <> struct Mma16816<__half> {
  static __device__ __forceinline__ void run(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

// Row e of a table that is either one array or, PEER, sharded over the GPUs of a node by e % world (shard r holds
// expert e at row e / world; shards[r] may point into a peer GPU's memory, read with plain loads over NVLink).
// In the sharded form ids at or above `sharded` address a small table replicated on every GPU (the hottest
// experts, copied once): row e - sharded of `table`, which is local memory.
template <typename T, bool PEER>
__device__ __forceinline__ const T* table_row(const T* table, const T* const* shards, int world, int64_t e, int H,
                                              int64_t sharded = 0) {
  if constexpr (PEER) {
    if (e >= sharded) return table + (e - sharded) * H;
    const int64_t local = e / world;
    return shards[e - local * world] + local * H;
  } else {
    return table + e * H;
  }
}

// One warp per (token, group of 16 of its experts).  The token's x row is parked in the warp's slice of shared memory (read back
// as B fragments right before each MMA; fetched with cp.async one task ahead, together with the next task's expert ids), so
// every register that waits for data waits for a gathered down row: batches of 128 columns (8 x 16 B per lane) in two register
// buffers keep gathers in flight across batches to cover the L2 latency.
//
// SLABS: the table is walked in slabs of columns (slab_columns), every task of a slab before the next slab; the sums so far
// wait in gs, where the thread that stored them takes them up again (same order of columns, same bits).  Gathers from a slab that
// fits L2 run at up to 17 TB/s, from 256 MiB at 9.7 (loads alone).  Without, slab is H, in a kernel of its own: 381 -> 373 us for
// both passes over 32768 tokens x 1024 float16, top-32 of 2^18 experts by Zipf's law.
//
// Bound by the L1's data path: a load takes 64 bytes of each of eight rows, eight of its cycles for 512 bytes, and the x
// fragments as much again for each fourth load.  Measured and not kept at 4096 x 1024, top-64 (52 us): whole lines per load and
// an exchange between lanes (56), whole lines and sums handed from lane to lane between the halves of a line (twice the MMAs:
// 56; rows as B: 71), rows as B and the token as A (twice the MMAs for no register moves: 53.7), 32 rows per fragment (54).
template <typename T, bool PEER, int COLS, bool LOAD32 = false, bool SLABS = false>
__global__ void __launch_bounds__(128, 4) expert_scores_mma_kernel(const T* x, const T* __restrict__ down, const int64_t* idx,
                                                                  const T* gates, float* gs, int64_t ntok, int H, int64_t N,
                                                                  int k, int slab, int32_t* status, int act,
                                                                  const T* const* __restrict__ shards, int world,
                                                                  float* __restrict__ raw_out, int64_t sharded) {
  extern __shared__ uint4 xs_all[];
  pdl_wait();  // ids and gates come from the kernel before this one
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;
  if (!SLABS) slab = H;
  const int xs_stride = (slab + 255) / 256 * 32;  // 16-byte pieces of an x row buffer, two per warp
  uint4* xs_buf = xs_all + (threadIdx.x >> 5) * 2 * xs_stride;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t warp_global = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  // the next task's first batch is requested before this task's last one is consumed (52.5 -> 51.5 us at 4096 tokens x 1024,
  // top-64); with the wider loads or several tables that takes more registers than it gives
  constexpr bool kCross = COLS == 8 && !PEER;
  constexpr int UNROLL = 4, STEP = 32 * UNROLL;
  const int groups = (k + 15) >> 4;
  const int64_t tasks = ntok * groups;
  if (warp_global >= tasks) return;
  const bool lone = warp_global + warps_total >= tasks;  // one task: its partial sums stay in registers
  // the slot whose sum this lane finishes
  const int own = g + 8 * tq;  // tq < 2
  bool bad = false;
  int64_t e[2];
  auto fetch_ids = [&](int64_t t_, int G_) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j_ = G_ * 16 + g + 8 * i;
      e[i] = j_ < k ? idx[t_ * k + j_] : -1;
    }
  };
  auto fetch_x = [&](int64_t t_, int col_, uint4* dst) {
    const T* xr = x + t_ * H + col_;
    const int pieces = min(slab, H - col_) >> 3;
    for (int c = lane; c < xs_stride; c += 32) {
      if (c < pieces) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst + c))),
                     "l"(reinterpret_cast<uint64_t>(xr + c * 8))
                     : "memory");
      } else {
        dst[c] = make_uint4(0, 0, 0, 0);
      }
    }
  };
  const T* row[2];
  auto rows_of = [&](int col_) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      row[i] = table_row<T, PEER>(down, shards, world, e[i] >= 0 && e[i] < N ? e[i] : 0, H, sharded) + col_ + COLS * tq;
  };
  struct Batch {
    uint4 q[2][UNROLL];
  };
  // COLS = 8: lane tq has columns 8 tq .. 8 tq + 7 of each 32-column block u.  COLS = 16: columns 16 tq .. 16 tq + 15 of each
  // 64-column block, so that the four lanes of a row cover a whole 128-byte line, in one 32-byte load (LOAD32) or, for tables
  // that are only 16-byte aligned or whose alignment the host does not know (PEER), in two.
  auto load = [&](Batch& b, int c0, int cols) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if constexpr (COLS == 8) {
        const bool in = c0 + 32 * u + 8 * tq < cols;
#pragma unroll
        for (int i = 0; i < 2; ++i) b.q[i][u] = in ? ldg16(row[i] + c0 + 32 * u) : zero;
      } else if ((u & 1) == 0) {
        if (c0 + 32 * u + 16 * tq < cols) {  // H % 16 == 0
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if constexpr (LOAD32) {
              ldg32(row[i] + c0 + 32 * u, b.q[i][u], b.q[i][u + 1]);
            } else {
              b.q[i][u] = ldg16(row[i] + c0 + 32 * u);
              b.q[i][u + 1] = ldg16(row[i] + c0 + 32 * u + 8);
            }
          }
        } else {
          b.q[0][u] = b.q[0][u + 1] = b.q[1][u] = b.q[1][u + 1] = zero;
        }
      }
    }
  };
  float c[4] = {};
  int cur = 0;
  auto consume = [&](const Batch& b, int c0) {
    const uint4* xs = xs_buf + cur * xs_stride + (c0 >> 3);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const uint4 xq = xs[COLS == 16 ? 4 * (u & ~1) + 2 * tq + (u & 1) : 4 * u + tq];
      const uint4 &qa = b.q[0][u], &qb = b.q[1][u];
      Mma16816<T>::run(c, qa.x, qb.x, qa.y, qb.y, xq.x, xq.y);
      Mma16816<T>::run(c, qa.z, qb.z, qa.w, qb.w, xq.z, xq.w);
    }
  };

  // (token, group) of tasks, stepped without divisions
  const int64_t dt = warps_total / groups, t_first = warp_global / groups;
  const int dG = static_cast<int>(warps_total - dt * groups), G_first = static_cast<int>(warp_global - t_first * groups);
  int64_t t_next = t_first;
  int G_next = G_first;
  Batch b0, b1;
  fetch_ids(t_first, G_first);
  float part_next = 0.f;
  fetch_x(t_first, 0, xs_buf);
  rows_of(0);
  load(b0, 0, min(slab, H));
  int col = 0;
  do {
    const int cols = SLABS ? min(slab, H - col) : H;
    const bool last_slab = !SLABS || col + slab >= H;
    for (int64_t task = warp_global; task < tasks; task += warps_total) {
      const bool last_task = task + warps_total >= tasks;
      const bool more = !(last_slab && last_task);
      if (!more) pdl_launch_dependents();  // the next kernel may set up
      const int next_col = SLABS ? (last_task ? col + slab : col) : 0;
      const int64_t t = t_next;
      const int j = G_next * 16;
      if (SLABS && last_task) {
        t_next = t_first;
        G_next = G_first;
      } else {
        t_next += dt;
        if ((G_next += dG) >= groups) {
          G_next -= groups;
          ++t_next;
        }
      }
      bool present = false;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const bool ok = e[i] >= 0 && e[i] < N;
        bad |= !ok && e[i] != -1;  // -1: empty slot, no flag
        if (tq == i) present = ok;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();  // this task's x row has landed; the other buffer is free (its task is finished)
      c[0] = c[2] = part_next;  // of this lane's sums that of its own slot counts
      if (more) {
        fetch_ids(t_next, G_next);
        fetch_x(t_next, next_col, xs_buf + (cur ^ 1) * xs_stride);
        part_next = 0.f;
        if (SLABS && next_col > 0 && !lone && tq < 2 && G_next * 16 + own < k) part_next = gs[t_next * k + G_next * 16 + own];
      }
      for (int c0 = 0; c0 < cols; c0 += 2 * STEP) {
        const bool two = c0 + STEP < cols;
        if (two) load(b1, c0 + STEP, cols);
        consume(b0, c0);
        if (c0 + 2 * STEP < cols) {
          load(b0, c0 + 2 * STEP, cols);
        } else if (kCross && more) {
          rows_of(next_col);
          load(b0, 0, SLABS ? min(slab, H - next_col) : H);
        }
        if (two) consume(b1, c0 + STEP);
      }
      if (!kCross && more) {
        rows_of(next_col);
        load(b0, 0, SLABS ? min(slab, H - next_col) : H);
      }
      cur ^= 1;
      if (tq < 2 && j + own < k) {
        const int64_t p = t * k + j + own;
        const float v = tq == 0 ? c[0] : c[2];
        if (!last_slab) {
          if (lone) part_next = v;
          else gs[p] = v;
        } else {
          const float s = present ? v : 0.f;
          gs[p] = gates != nullptr && present ? expert_act(v, act) * to_f32<T>(gates[p]) : s;
          if (raw_out != nullptr) raw_out[p] = s;
        }
      }
    }
  } while (SLABS && (col += slab) < H);
  if (bad && status != nullptr) atomicOr(status, FMOE_STATUS_BAD_EXPERT_ID);
}

// ---------------------------------------------------------------- 2c. scores, few tokens
// One CTA of W warps per (token, group of 16 of its experts), each warp on its own 128-column chunks of the 16 gathered
// rows; the sums pass through the warps in column order, so they are those of the kernel above with the same COLS bit for
// bit, whatever the number of tokens.  With few tasks that kernel leaves most of the chip idle while a warp pulls 16 whole
// rows: 64 tokens x 2048 columns, top-32 (128 tasks) took 11.2 us there.
template <typename T, int W, bool PEER, int COLS>
__global__ void __launch_bounds__(32 * W) expert_scores_split_kernel(const T* x, const T* __restrict__ down,
                                                                    const int64_t* idx, const T* gates, float* __restrict__ gs,
                                                                    int64_t tasks, int groups, int H, int64_t N, int k,
                                                                    int32_t* status, int act, float* __restrict__ raw_out,
                                                                    const T* const* __restrict__ shards, int world,
                                                                    int64_t sharded) {
  __shared__ float2 chain[32];
  pdl_wait();  // ids and gates come from the kernel before this one
  pdl_launch_dependents();  // the accumulate pass may start gathering: it needs the ids, and only later the scores
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, tq = lane & 3;
  for (int64_t task = blockIdx.x; task < tasks; task += gridDim.x) {
    const int64_t t = task / groups;
    const int j0 = static_cast<int>(task - t * groups) * 16;
    const int ja = j0 + g, jb = ja + 8;
    const int64_t ea = ja < k ? idx[t * k + ja] : 0, eb = jb < k ? idx[t * k + jb] : 0;
    const bool oka = (ja < k) && ea >= 0 && ea < N;
    const bool okb = (jb < k) && eb >= 0 && eb < N;
    if (((ja < k && !oka && ea != -1) || (jb < k && !okb && eb != -1)) && status != nullptr)
      atomicOr(status, FMOE_STATUS_BAD_EXPERT_ID);  // -1: empty slot, no flag
    const T* ra = table_row<T, PEER>(down, shards, world, oka ? ea : 0, H, sharded) + COLS * tq;
    const T* rb = table_row<T, PEER>(down, shards, world, okb ? eb : 0, H, sharded) + COLS * tq;
    const T* rx = x + t * H + COLS * tq;
    // the thread that finishes a slot fetches its id and gate now, beside the rows
    const int64_t p = t * k + j0 + threadIdx.x;
    const bool mine = threadIdx.x < 16 && j0 + static_cast<int>(threadIdx.x) < k;
    const int64_t e = mine ? idx[p] : -1;
    const float gate = mine && gates != nullptr ? to_f32<T>(gates[p]) : 0.f;
    // warp w loads the 128-column blocks w, w + W, ...; the sums go from warp to warp in column order (every column of B is
    // the token's row, so c[0] = c[1] and c[2] = c[3])
    for (int base = 0; base < H; base += W * 128) {
      const int c0 = base + warp * 128;
      uint4 qa[4], qb[4], qx[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        // COLS = 16: lane tq has the columns 16 tq .. 16 tq + 15 of a 64-column block, the first eight of them in step u = 0, 2
        const int col = COLS == 16 ? c0 + 64 * (u >> 1) + 8 * (u & 1) : c0 + 32 * u;
        const bool in = col + COLS * tq < H;
        qa[u] = in ? ldg16(ra + col) : make_uint4(0, 0, 0, 0);
        qb[u] = in ? ldg16(rb + col) : make_uint4(0, 0, 0, 0);
        qx[u] = in ? ld16(rx + col) : make_uint4(0, 0, 0, 0);
      }
      for (int w = 0; w < W; ++w) {
        if (warp == w && c0 < H) {
          const float2 sum = c0 == 0 ? make_float2(0.f, 0.f) : chain[lane];
          float c[4] = {sum.x, sum.x, sum.y, sum.y};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            Mma16816<T>::run(c, qa[u].x, qb[u].x, qa[u].y, qb[u].y, qx[u].x, qx[u].y);
            Mma16816<T>::run(c, qa[u].z, qb[u].z, qa[u].w, qb[u].w, qx[u].z, qx[u].w);
          }
          chain[lane] = make_float2(c[0], c[2]);
        }
        __syncthreads();
      }
    }
    if (mine) {
      const bool ok = e >= 0 && e < N;
      const float2 both = chain[(threadIdx.x & 7) * 4];
      const float s = !ok ? 0.f : threadIdx.x < 8 ? both.x : both.y;
      gs[p] = gates != nullptr && ok ? expert_act(s, act) * gate : s;  // no gates: the raw dot product
      if (raw_out != nullptr) raw_out[p] = s;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- 2d. scores, float32
// One warp per (token, 4 of its experts): 16-byte pieces of the four gathered rows and of the token's row, fp32 FMAs, one
// shuffle reduction.  No sort in front of it (histogram, scan, scatter and a pass over the sorted pairs took 5 launches and
// 22 us at 256 tokens x 256 columns, top-8; this takes one and 9).
__global__ void __launch_bounds__(128) expert_scores_f32_kernel(const float* x, const float* __restrict__ down,
                                                               const int64_t* idx, const float* gates, float* __restrict__ gs,
                                                               int64_t ntok, int H, int64_t N, int k, int32_t* status,
                                                               int act, float* __restrict__ raw_out) {
  constexpr int G = 4;
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t warp_global = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int groups = (k + G - 1) / G;
  bool bad = false;
  for (int64_t task = warp_global; task < ntok * groups; task += warps_total) {
    if (task + warps_total >= ntok * groups) pdl_launch_dependents();
    const int64_t t = task / groups;
    const int j0 = static_cast<int>(task - t * groups) * G;
    const float4* rx = reinterpret_cast<const float4*>(x + t * H);
    const float4* row[G];
    bool ok[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int64_t e = j0 + i < k ? idx[t * k + j0 + i] : -1;
      ok[i] = e >= 0 && e < N;
      bad |= !ok[i] && e != -1;
      row[i] = reinterpret_cast<const float4*>(down + (ok[i] ? e : 0) * H);
    }
    float acc[G] = {0.f, 0.f, 0.f, 0.f};
    const int hv = H >> 2;
#pragma unroll 2
    for (int c = lane; c < hv; c += 32) {
      const float4 v = rx[c];
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const float4 d = __ldg(row[i] + c);
        acc[i] = fmaf(v.x, d.x, acc[i]);
        acc[i] = fmaf(v.y, d.y, acc[i]);
        acc[i] = fmaf(v.z, d.z, acc[i]);
        acc[i] = fmaf(v.w, d.w, acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < G; ++i)
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc[i] += __shfl_xor_sync(kFull, acc[i], d);
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if (lane == i && j0 + i < k) {
        const int64_t p = t * k + j0 + i;
        const float s = ok[i] ? acc[i] : 0.f;
        gs[p] = gates != nullptr && ok[i] ? expert_act(s, act) * gates[p] : s;
        if (raw_out != nullptr) raw_out[p] = s;
      }
    }
  }
  if (bad && status != nullptr) atomicOr(status, FMOE_STATUS_BAD_EXPERT_ID);
}

// ---------------------------------------------------------------- 3. per-token accumulate
// One warp per (token, column block of 32*VEC*NCH elements); 16 x 16 B of gathered rows in flight
// per lane, packed f32x2 FMAs (two accumulators per instruction).  The launch bound keeps the kernel at 120
// registers so that four CTAs (not three) fit an SM: a third more gathers in flight, 52 -> 48 us at the benchmark
// shape (a fifth CTA would need spills and is slower: 120 vs 105 us for both passes).
// The column blocks are the outer loop: all tokens gather from the same 512 columns of the table before the next ones, which
// stay in L2 where the whole table does not (131072 tokens x 2048, 65536 experts top-32: 1960 -> 1400 us with the CTAs in
// step).  Bound by the gathers in flight: loads alone reach 11 TB/s with as many as four such CTAs hold, 17 with eight.  Half of
// the batches through shared memory by cp.async put more of them in flight and took longer all the same (48 -> 50 us).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void ffma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// The columns from col0 of one token, slot by slot and without the absent ones: the rare case of the kernel below, apart so
// that its registers and loads do not weigh on that one's loop.  Same sums in the same order.
template <typename T, typename OutT, int NCH, bool PEER>
__device__ __noinline__ void accum_present_slots(const T* up, const int64_t* idx, const float* gs, OutT* out, int64_t t, int col0,
                                                 int H, int64_t N, int k, const T* const* shards, int world, int64_t sharded) {
  constexpr int VEC = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c = 0; c < NCH; ++c) {
    const int col = col0 + (c * 32 + lane) * VEC;
    if (col >= H) continue;
    float acc[VEC] = {};
#pragma unroll 1
    for (int j = 0; j < k; ++j) {
      const int64_t e = idx[t * k + j];
      if (e < 0 || e >= N) continue;
      const float w = gs[t * k + j];
      float f[VEC];
      unpack16<T>(ldg16(table_row<T, PEER>(up, shards, world, e, H, sharded) + col), f);
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[i] = fmaf(f[i], w, acc[i]);
    }
    OutT* o = out + t * H + col;
#pragma unroll
    for (int i = 0; i < VEC; ++i) o[i] = from_f32<OutT>(acc[i]);
  }
}

template <typename T, typename OutT, int NCH, bool PEER = false>
__global__ void __launch_bounds__(128, 4) expert_accum_kernel(const T* __restrict__ up, const int64_t* idx,
                                                          const float* gs, OutT* __restrict__ out,
                                                          int64_t ntok, int H, int64_t N, int k, int colblocks,
                                                          const T* const* __restrict__ shards = nullptr,
                                                          int world = 1, int64_t sharded = 0) {
  constexpr int VEC = Vec16<T>::N;
  constexpr int SLOTS = 8;
  pdl_wait();  // the weights gs come from the scores pass
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t warp_global = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t tasks = ntok * colblocks;
  // each lane fetches one slot's (expert id, weight) - one batch of 32 slots AHEAD of the batch being gathered,
  // also across tasks, so that the gathers of a batch never wait for their own ids; invalid or absent slots get
  // weight -0, which adds nothing and marks them
  auto fetch_slot = [&](int64_t t_, int j0_, int& e_, float& w_) {
    e_ = 0;
    w_ = -0.f;
    const int j = j0_ + lane;
    if (j < k) {
      const int64_t e = idx[t_ * k + j];
      if (e >= 0 && e < N) {
        e_ = static_cast<int>(e);
        w_ = gs[t_ * k + j];
      }
    }
  };
  int e_next = 0;
  float w_next = 0.f;
  int64_t t_next = warp_global;
  int col_next = 0;
  auto wrap = [&]() {
    while (t_next >= ntok) {
      t_next -= ntok;
      col_next += 32 * VEC * NCH;
    }
  };
  auto step = [&]() {
    t_next += warps_total;
    wrap();
  };
  wrap();
  if (warp_global < tasks) fetch_slot(t_next, 0, e_next, w_next);
  for (int64_t task = warp_global; task < tasks; task += warps_total) {
    if (task + warps_total >= tasks) pdl_launch_dependents();  // last task of this warp: the next kernel may set up
    const int64_t t = t_next;
    const int col0 = col_next;
    step();
    bool in[NCH];
#pragma unroll
    for (int c = 0; c < NCH; ++c) in[c] = col0 + (c * 32 + lane) * VEC < H;
    uint64_t acc[NCH][VEC / 2];
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) acc[c][i] = 0ull;

    bool some_absent = false;
    for (int j0 = 0; j0 < k; j0 += 32) {
      const int e_l = e_next;
      const float w_l = w_next;
      if (j0 + 32 < k) fetch_slot(t, j0 + 32, e_next, w_next);
      else if (task + warps_total < tasks) fetch_slot(t_next, 0, e_next, w_next);
      const int nslots = min(32, k - j0);
      some_absent |= __any_sync(kFull, lane < (nslots + SLOTS - 1) / SLOTS * SLOTS && __float_as_uint(w_l) == 0x80000000u);
      auto load = [&](uint4 (&q)[SLOTS][NCH], uint64_t (&ww)[SLOTS], int s) {
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {
          const int e = __shfl_sync(kFull, e_l, s + u);
          const float w = __shfl_sync(kFull, w_l, s + u);
          ww[u] = pack_f32x2(w, w);
          const T* row = table_row<T, PEER>(up, shards, world, e, H, sharded) + col0 + lane * VEC;
#pragma unroll
          for (int c = 0; c < NCH; ++c) q[u][c] = in[c] ? ldg16(row + c * 32 * VEC) : make_uint4(0, 0, 0, 0);
        }
      };
      auto consume = [&](const uint4 (&q)[SLOTS][NCH], const uint64_t (&ww)[SLOTS]) {
#pragma unroll
        for (int u = 0; u < SLOTS; ++u)
#pragma unroll
          for (int c = 0; c < NCH; ++c) {
            float f[VEC];
            unpack16<T>(q[u][c], f);
#pragma unroll
            for (int i = 0; i < VEC / 2; ++i) ffma2(acc[c][i], pack_f32x2(f[2 * i], f[2 * i + 1]), ww[u]);
          }
      };
      // one batch of SLOTS gathered rows at a time (a second register buffer was measured slower: 64 vs 52 us)
      for (int s = 0; s < nslots; s += SLOTS) {
        uint4 q[SLOTS][NCH];
        uint64_t ww[SLOTS];
        load(q, ww, s);
        consume(q, ww);
      }
    }
    // Absent slots above read row 0 with weight 0, and that product is not 0 where the row is not finite: a sum that is not
    // finite is then formed again from the present slots alone.  (Leaving the loads out above makes the sums wait for all of them:
    // both passes of 32768 tokens x 2048, top-16, 392 -> 450 us.)
    if (some_absent) {
      uint64_t check = 0ull;
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int i = 0; i < VEC / 2; ++i) ffma2(check, acc[c][i], 0ull);
      float lo, hi;
      unpack_f32x2(check, lo, hi);
      if (__any_sync(kFull, !(lo + hi == 0.f))) {
        accum_present_slots<T, OutT, NCH, PEER>(up, idx, gs, out, t, col0, H, N, k, shards, world, sharded);
        continue;
      }
    }
    OutT* orow = out + t * H + col0;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int col = (c * 32 + lane) * VEC;
      if (in[c]) {
        float f[VEC];
#pragma unroll
        for (int i = 0; i < VEC / 2; ++i) unpack_f32x2(acc[c][i], f[2 * i], f[2 * i + 1]);
        if constexpr (sizeof(OutT) == 4) {
#pragma unroll
          for (int i = 0; i < VEC; i += 4)
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(orow) + col + i) =
                make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
        } else {
          *reinterpret_cast<uint4*>(orow + col) = pack16<OutT>(f);
        }
      }
    }
  }
}

// The same sum for few tokens: a CTA of W warps per (token, block of 32 * VEC columns), each warp on its own batches of 8
// slots; the sums pass through the warps in slot order (bit for bit those of the kernel above).  The kernel is made resident
// beside the scores pass (which has itself waited for the ids) and gathers its first batch of rows before it waits for the
// weights.
template <typename T, typename OutT, int W, bool PEER>
__global__ void __launch_bounds__(32 * W) expert_accum_split_kernel(const T* __restrict__ up, const int64_t* idx,
                                                                   const float* gs, OutT* __restrict__ out,
                                                                   int64_t tasks, int H, int64_t N, int k, int colblocks,
                                                                   int early, const T* const* __restrict__ shards,
                                                                   int world, int64_t sharded,
                                                                   const float* addend, const OutT* residual) {
  constexpr int VEC = Vec16<T>::N;
  constexpr int SLOTS = 8;
  constexpr int COLS = 32 * VEC;
  __shared__ float part[COLS];  // the sums on their way from warp to warp
  pdl_launch_dependents();  // all CTAs are resident once the last of them is here: the next kernel may start beside them
  if (!early) pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool waited = !early;
  for (int64_t task = blockIdx.x; task < tasks; task += gridDim.x) {
    const int64_t t = task / colblocks;
    const int col0 = static_cast<int>(task - t * colblocks) * COLS;
    static_assert(COLS <= 32 * W * 4, "every thread finishes at most one group of four columns");
    const bool mine = threadIdx.x * 4 < COLS && col0 + static_cast<int>(threadIdx.x) * 4 < H;
    const int64_t at = t * H + col0 + threadIdx.x * 4;
    float ad[4] = {}, rs[4] = {};
    const bool in = col0 + lane * VEC < H;
    for (int base = 0; base < k; base += W * SLOTS) {
      const int j0 = base + warp * SLOTS;
      const int j = j0 + (lane & (SLOTS - 1));
      // ids and rows are read past the L1 cache: an early CTA may find lines of an earlier forward there
      const int64_t e = j < k ? __ldcg(reinterpret_cast<const long long*>(idx) + t * k + j) : -1;
      const bool ok = e >= 0 && e < N;
      const int row = ok ? static_cast<int>(e) : -1;  // -1: nothing is read
      uint4 q[SLOTS];
#pragma unroll
      for (int u = 0; u < SLOTS; ++u) {
        const int r = __shfl_sync(kFull, row, u);
        q[u] = in && r >= 0 ? __ldcg(reinterpret_cast<const uint4*>(table_row<T, PEER>(up, shards, world, r, H, sharded) + col0 + lane * VEC))
                            : make_uint4(0, 0, 0, 0);
      }
      if (!waited) {
        pdl_wait();
        waited = true;
      }
      if (base == 0 && mine) {  // addend: the shared MLP's output, residual: the skip connection
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (addend != nullptr) ad[i] = ld_after_wait(addend + at + i);
          if (sizeof(OutT) == 2 && residual != nullptr) {
            const uint16_t raw = ld_after_wait(reinterpret_cast<const uint16_t*>(residual) + at + i);
            rs[i] = to_f32<OutT>(*reinterpret_cast<const OutT*>(&raw));
          }
        }
      }
      const float w = ok ? ld_after_wait(gs + t * k + j) : 0.f;
      for (int turn = 0; turn < W; ++turn) {  // slots in ascending order, as the one-warp-per-task kernel adds them
        if (warp == turn && j0 < k) {
          float2* p = reinterpret_cast<float2*>(&part[lane * VEC]);
          uint64_t acc[VEC / 2];
#pragma unroll
          for (int i = 0; i < VEC / 2; ++i) {
            const float2 v = j0 == 0 ? make_float2(0.f, 0.f) : p[i];
            acc[i] = pack_f32x2(v.x, v.y);
          }
#pragma unroll
          for (int u = 0; u < SLOTS; ++u) {
            const float wu = __shfl_sync(kFull, w, u);
            const uint64_t w2 = pack_f32x2(wu, wu);
            float f[VEC];
            unpack16<T>(q[u], f);
#pragma unroll
            for (int i = 0; i < VEC / 2; ++i) ffma2(acc[i], pack_f32x2(f[2 * i], f[2 * i + 1]), w2);
          }
#pragma unroll
          for (int i = 0; i < VEC / 2; ++i) {
            float lo, hi;
            unpack_f32x2(acc[i], lo, hi);
            p[i] = make_float2(lo, hi);
          }
        }
        __syncthreads();
      }
    }
    if (mine) {
      const float4 s = *reinterpret_cast<const float4*>(&part[threadIdx.x * 4]);
      OutT* o = out + at;
      if constexpr (sizeof(OutT) == 4) {
        *reinterpret_cast<float4*>(o) = s;
      } else {
        // in the order of the down GEMM's epilogue
        const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float r = addend != nullptr ? ad[i] + v[i] : v[i];
          o[i] = from_f32<OutT>(residual != nullptr ? r + rs[i] : r);
        }
      }
    }
    __syncthreads();
  }
}

struct Carver {
  char* base;
  size_t off = 0;
  template <typename E> E* take(size_t count) {
    E* p = base ? reinterpret_cast<E*>(base + off) : nullptr;
    off += align_up(count * sizeof(E), 256);
    return p;
  }
};

// forward: the weights of the pairs, between the two passes
struct ExpertWs {
  float* gs;
  size_t bytes;
};

ExpertWs carve(void* ws, int64_t T, int k) {
  Carver c{static_cast<char*>(ws)};
  ExpertWs w;
  w.gs = c.take<float>(static_cast<size_t>(T) * k);
  w.bytes = c.off;
  return w;
}

// Few tokens: warps per task, by the pieces it can be cut into; 0 selects the one-warp-per-task kernels.  `limit` is where
// those take over (measured over 1 to 1000 tokens): the scores pass at 5 1/3 tasks per SM, the accumulate pass at 8 - or at
// one, where a task has only 16 slots and two of its four warps would find none (500 tokens x 512, top-16: 9.6 -> 6.3 us).
int split_warps(int64_t tasks, int pieces, int64_t limit) {
  if (tasks > limit) return 0;
  return pieces >= 8 ? 8 : pieces >= 2 ? 4 : 0;
}

struct PeerTable {  // a table sharded over the GPUs of a node (table_row); no shards: one array
  const void* const* shards = nullptr;
  int world = 1;
  int64_t sharded = 0;
};

int scores_split_warps(int64_t T, int H, int k) {
  return split_warps(T * ((k + 15) / 16), (H + 127) / 128, static_cast<int64_t>(device_sm_count()) * 16 / 3);
}
int accum_split_warps(int64_t T, int H, int k, int cols) {
  const int pieces = (k + 7) / 8;
  return split_warps(T * ((H + 2 * cols - 1) / (2 * cols)), pieces, static_cast<int64_t>(device_sm_count()) * (pieces >= 3 ? 8 : 1));
}

// Scores pass with one thread's share of a row in 16 columns at a time, for tables of more than 384 MiB: rows taken 64 bytes
// at a time cost twice the time there (16384 tokens x 2048 columns, top-16, table of 512 MiB 283 -> 153 us, 4 GiB with Zipf
// 1.1 ids 519 -> 185 at 32768 tokens), and make no difference at 256 MiB (253 and 246).  It also groups the columns of a
// sum differently, so the smaller tables of a stack of layers, where the last bit of a score can decide a later layer's
// selection, keep the order that they have; tables in L2 give 16% for that (51 and 43 us at 4096 x 1024, top-64).  The rule
// looks at the table alone and holds for every scores kernel: a token has the same bits alone and in a batch.
template <typename T>
bool whole_lines(int64_t N, int H) {
  return H % 16 == 0 && N * H * static_cast<int64_t>(sizeof(T)) > (384ll << 20);
}

// Whether the table does not stay in L2 (126 MB).
template <typename T>
bool beyond_l2(int64_t N, int H) {
  return N * H * static_cast<int64_t>(sizeof(T)) > (144ll << 20);
}

// Columns that the scores pass walks the table in: slabs of 512 for the ids of the layer's own router, which spread over the
// experts, where the table does not stay in L2, a slab nearly does and its rows come more than once.  Both passes then run with
// exactly the CTAs that are resident at once, so that all of them are at the same slab.  Layer of 131072 tokens, 2048 x 5632,
// 65536 experts top-32, whole rows and slabs: 11.6 and 11.1 ms, 16384 tokens 1.40 and 1.37 ms; with a router that sends
// everything to 5 % of the experts 10.15 and 10.2, 1.32 and 1.32.  Other ids may be skewed, and where the wanted rows stay in L2
// anyway a slab only costs every task a start and a partial sum: the scores and accumulate passes on ids by Zipf's law (1.1),
// 32768 tokens x 2048 top-16 of 2^18 experts, 370 us whole and 399 in slabs, 2000 tokens top-33 of 2^17 70 and 80 (uniform ids
// 621 and 600, 93 and 98).  Up to 128 MiB slabs give nothing (65536 x 1024: 112.3 and 112.7 us).
template <typename T>
int slab_columns(int64_t T_, int H, int64_t N, int k, bool router_ids) {
  constexpr int kSlab = 512;
  const bool slabs = router_ids && beyond_l2<T>(N, H) && N * kSlab * static_cast<int64_t>(sizeof(T)) <= (256ll << 20) && T_ * k >= N;
  return slabs && H > kSlab ? kSlab : H;
}

// the scores pass / accumulate pass for few tokens; false: not the shape for it (or, with `rc`, a launch error)
template <typename T, bool PEER>
bool try_scores_split(const void* rows, const void* table, const int64_t* idx, const void* gates, float* out, int64_t T_, int H,
                      int64_t N, int k, int32_t* status, cudaStream_t stream, int act, float* raw_out, const PeerTable& pt,
                      cudaError_t* rc) {
  const bool lines = whole_lines<T>(PEER ? pt.sharded : N, H);
  const int groups = (k + 15) / 16;
  const int64_t tasks = T_ * groups;
  const int split = scores_split_warps(T_, H, k);
  if (split == 0) return false;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * (64 / split);
  auto kern = split == 8 ? (lines ? expert_scores_split_kernel<T, 8, PEER, 16> : expert_scores_split_kernel<T, 8, PEER, 8>)
                         : (lines ? expert_scores_split_kernel<T, 4, PEER, 16> : expert_scores_split_kernel<T, 4, PEER, 8>);
  *rc = launch_pdl(PEER ? 0 : 8, kern, dim3(static_cast<unsigned>(tasks < cap ? tasks : cap)), dim3(32 * split), 0, stream, 1,
                   static_cast<const T*>(rows), static_cast<const T*>(table), idx, static_cast<const T*>(gates), out, tasks,
                   groups, H, N, k, status, act, raw_out, reinterpret_cast<const T* const*>(pt.shards), pt.world, pt.sharded);
  return true;
}

template <typename T, bool PEER>
bool try_accum_split(const void* table, const int64_t* idx, const float* coef, void* out, int out_f32, int64_t T_, int H,
                     int64_t N, int k, bool early, cudaStream_t stream, const PeerTable& pt, cudaError_t* rc, const float* addend = nullptr, const void* residual = nullptr) {
  constexpr int COLS = 32 * Vec16<T>::N;
  const int split = accum_split_warps(T_, H, k, COLS);
  if (split == 0) return false;
  const int colblocks = (H + COLS - 1) / COLS;
  const int64_t tasks = T_ * colblocks;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * (64 / split);
  auto go = [&](auto kern, auto* o) {
    using OutT = std::remove_pointer_t<decltype(o)>;
    *rc = launch_pdl(PEER ? 0 : 8, kern, dim3(static_cast<unsigned>(tasks < cap ? tasks : cap)), dim3(32 * split), 0, stream, 1,
                     static_cast<const T*>(table), idx, coef, o, tasks, H, N, k, colblocks, early && !PEER ? 1 : 0,
                     reinterpret_cast<const T* const*>(pt.shards), pt.world, pt.sharded, addend, static_cast<const OutT*>(residual));
  };
  if (out_f32) {
    if (split == 8) go(expert_accum_split_kernel<T, float, 8, PEER>, static_cast<float*>(out));
    else go(expert_accum_split_kernel<T, float, 4, PEER>, static_cast<float*>(out));
  } else {
    if (split == 8) go(expert_accum_split_kernel<T, T, 8, PEER>, static_cast<T*>(out));
    else go(expert_accum_split_kernel<T, T, 4, PEER>, static_cast<T*>(out));
  }
  return true;
}

template <typename T, typename OutT, int NCH>
void launch_accum(const void* up, const int64_t* idx, const float* gs, void* out, int64_t T_, int H, int64_t N, int k,
                  cudaStream_t stream) {
  constexpr int VEC = Vec16<T>::N;
  const int colblocks = (H + 32 * VEC * NCH - 1) / (32 * VEC * NCH);
  const int64_t tasks = T_ * colblocks;
  const int64_t want = (tasks + 3) / 4;
  // a table beyond L2: the CTAs that are resident at once, all of them at the same columns (32768 tokens x 2048 top-16 of 2^18
  // experts, both passes: uniform ids 637 -> 620 us, Zipf 1.1 379 -> 373; top-64 of 2^18 x 1024 by Zipf's law 672 -> 681)
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * (beyond_l2<T>(N, H) ? 4 : 16);
  const int grid = static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
  auto kern = expert_accum_kernel<T, OutT, NCH>;
  (void)launch_pdl(8, kern, dim3(grid), dim3(128), 0, stream, 1, static_cast<const T*>(up), idx, gs, static_cast<OutT*>(out), T_,
                   H, N, k, colblocks, nullptr, 1, 0);  // launch errors surface through the caller's launch check
}

// per-pair dot products <rows[t], table[e]>: gates != nullptr stores silu(dot) * gate (forward), nullptr the
// raw dot product
template <typename T>
int run_scores(const void* rows, const void* table, const int64_t* idx, const void* gates, float* out, int64_t T_, int H,
               int64_t N, int k, int32_t* status, cudaStream_t stream, int act = 0, float* raw_out = nullptr,
               bool router_ids = false) {
  const int sms = device_sm_count();
  if constexpr (sizeof(T) == 2) {
    cudaError_t rc = cudaSuccess;
    if (try_scores_split<T, false>(rows, table, idx, gates, out, T_, H, N, k, status, stream, act, raw_out, PeerTable{}, &rc)) {
      FMOE_CUDA_TRY(rc);
      return FMOE_OK;
    }
    const int64_t want = (T_ * ((k + 15) / 16) + 3) / 4;
    // exactly the CTAs that are resident at once (four per SM at 121 registers): every warp walks its tasks with
    // the next one's ids and x row already in flight, and the work ends evenly (53.7 vs 55.7 us with 16 per SM)
    const int64_t cap = static_cast<int64_t>(sms) * 4;
    const int grid = static_cast<int>(want < cap ? want : cap);
    const int slab = slab_columns<T>(T_, H, N, k, router_ids);
    const int smem = 4 * 2 * ((slab + 255) / 256 * 32) * 16;  // two x-row buffers per warp
    const bool aligned32 = (reinterpret_cast<uintptr_t>(table) & 31u) == 0;
    auto kernel = [&](auto slabs) {
      constexpr bool S = decltype(slabs)::value;
      return !whole_lines<T>(N, H) ? expert_scores_mma_kernel<T, false, 8, false, S>
             : aligned32 ? expert_scores_mma_kernel<T, false, 16, true, S> : expert_scores_mma_kernel<T, false, 16, false, S>;
    };
    auto kern = slab < H ? kernel(std::true_type{}) : kernel(std::false_type{});
    FMOE_CUDA_TRY(allow_smem(kern, smem));
    FMOE_CUDA_TRY(launch_pdl(4, kern, dim3(grid), dim3(128), smem, stream, 1, static_cast<const T*>(rows),
                             static_cast<const T*>(table), idx, static_cast<const T*>(gates), out, T_, H, N, k, slab,
                             status, act, nullptr, 1, raw_out, 0));
  } else {
    const int64_t want = (T_ * ((k + 3) / 4) + 3) / 4;
    const int64_t cap = static_cast<int64_t>(sms) * 16;
    FMOE_CUDA_TRY(launch_pdl(8, expert_scores_f32_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(128), 0,
                             stream, 1, static_cast<const float*>(rows), static_cast<const float*>(table), idx,
                             static_cast<const float*>(gates), out, T_, H, N, k, status, act, raw_out));
  }
  return FMOE_OK;
}

// out[t] = sum_j coef[t,j] * table[idx[t,j]] (float32 accumulation, one rounding)
template <typename T>
int run_accum(const void* table, const int64_t* idx, const float* coef, void* out, int out_f32, int64_t T_, int H,
              int64_t N, int k, cudaStream_t stream, bool early = false) {
  constexpr int VEC = Vec16<T>::N;
  cudaError_t split_rc = cudaSuccess;
  if (try_accum_split<T, false>(table, idx, coef, out, out_f32, T_, H, N, k, early, stream, PeerTable{}, &split_rc)) {
    FMOE_CUDA_TRY(split_rc);
    return FMOE_OK;
  }
  const int need = (H + 32 * VEC - 1) / (32 * VEC);
#define FMOE_ACCUM(NCH_)                                                                       \
  do {                                                                                         \
    if (out_f32) launch_accum<T, float, NCH_>(table, idx, coef, out, T_, H, N, k, stream);     \
    else launch_accum<T, T, NCH_>(table, idx, coef, out, T_, H, N, k, stream);                 \
  } while (0)
  // narrow column blocks: more warps per token, i.e. more gathers in flight
  if (need <= 1) FMOE_ACCUM(1);
  else FMOE_ACCUM(2);
#undef FMOE_ACCUM
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}

template <typename T>
int run_typed(const void* x, const void* down, const void* up, const int64_t* idx, const void* gates, void* out,
              int out_f32, int64_t T_, int H, int64_t N, int k, const ExpertWs& w, int32_t* status,
              cudaStream_t stream, void* const* between_passes, int act, float* raw_scores, bool router_ids) {
  auto mark_between = [&]() -> int {
    if (between_passes != nullptr)
      for (int i = 0; i < 2; ++i)
        if (between_passes[i] != nullptr)
          FMOE_CUDA_TRY(cudaEventRecord(static_cast<cudaEvent_t>(between_passes[i]), stream));
    return FMOE_OK;
  };
  int rc = run_scores<T>(x, down, idx, gates, w.gs, T_, H, N, k, status, stream, act, raw_scores, router_ids);
  if (rc != FMOE_OK) return rc;
  if ((rc = mark_between()) != FMOE_OK) return rc;
  // the accumulate pass may gather rows while the scores pass runs: that pass has waited for the ids (only the kernels
  // for few tokens, which are launched with programmatic serialisation, let it in early)
  return run_accum<T>(up, idx, w.gs, out, out_f32, T_, H, N, k, stream, true);
}

// ---------------------------------------------------------------- backward
// Gradients of out[t] = sum_j silu(s_tj) * g_tj * U[e_tj], s_tj = <x[t], D[e_tj]>
// (flash_moe/ops/triton/flash_expert.py:214-525, host side :653-745):
//   q_tj  = <dout[t], U[e]>                      dg_tj = q * silu(s)
//   ds_tj = q * g * silu'(s)                     dx[t] = sum_j ds_tj * D[e]
//   dD[e] = sum_{pairs of e} ds * x[t]           dU[e] = sum_{pairs of e} silu(s) * g * dout[t]
// s is recomputed (nothing but the forward's inputs is saved).  All sums are float32 in a fixed order with one
// rounding on store: no atomics (the reference scatters with atomics), run-to-run deterministic.
// sorted pairs per warp task of the table-gradient pass: fewer when there are few pairs, so that every SM has warps at work
// (500 tokens float32 x 512 columns, top-16: 41 us with 64, 8 with 16)
int bwd_chunk(int64_t P) { return P >= (int64_t{1} << 18) ? 64 : P >= (int64_t{1} << 15) ? 32 : 16; }

// Pairs in the order of their experts, pairs of one expert in ascending pair id, so that the sums do not depend on timing:
//   histogram   counts per expert and each pair's arrival rank (an atomic per group of equal ids in a warp);
//   scan, scatter to offset + rank: segments per expert, in arrival order inside a segment;
//   sort of each segment by pair id: segments of up to 256 pairs in a warp's registers, longer ones (listed by the first
//   kernel, handled by the second) by setting their bits in a bitmap over the pair ids and reading it out in order.
// Skipped ids take no part.  262144 pairs over 16384 experts: 25 us; a stable radix sort of (expert, pair) took 47.
constexpr int kWarpSegment = 256;

__global__ void expert_hist_kernel(const int64_t* __restrict__ idx, int64_t P, int64_t N, int* __restrict__ counts,
                                   int* __restrict__ rank, int32_t* status) {
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t warp_global = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  bool bad = false;
  for (int64_t base = warp_global * 32; base < P; base += warps_total * 32) {
    const int64_t p = base + lane;
    const int64_t e = p < P ? idx[p] : -1;
    const bool valid = e >= 0 && e < N;
    bad |= p < P && !valid && e != -1;  // -1 is the empty-slot value: skipped without a flag
    const unsigned key = valid ? static_cast<unsigned>(e) : (0x80000000u | lane);
    const unsigned peers = __match_any_sync(kFull, key);
    const int leader = __ffs(peers) - 1;
    int first = 0;
    if (valid && lane == leader) first = atomicAdd(&counts[e], __popc(peers));
    first = __shfl_sync(kFull, first, leader);
    if (p < P) rank[p] = valid ? first + __popc(peers & ((1u << lane) - 1u)) : -1;
  }
  if (bad && status != nullptr) atomicOr(status, FMOE_STATUS_BAD_EXPERT_ID);
}

__global__ void expert_scatter_kernel(const int64_t* __restrict__ idx, const int* __restrict__ rank,
                                      const int* __restrict__ offsets, int64_t P, int* __restrict__ sorted_pair,
                                      int* __restrict__ sorted_expert) {
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int r = rank[p];
    if (r < 0) continue;
    const int e = static_cast<int>(idx[p]);
    const int pos = offsets[e] + r;
    sorted_pair[pos] = static_cast<int>(p);
    sorted_expert[pos] = e;
  }
}

template <int R>
__device__ __forceinline__ void sort_segment(int* seg, int n, int lane) {
  uint32_t a[R];  // descending keys of inverted ids: ascending ids; 0 pads
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = lane * R + r < n ? 0xFFFFFFFFu - static_cast<uint32_t>(seg[lane * R + r]) : 0u;
  sort_desc<R, false>(a, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane * R + r < n) seg[lane * R + r] = static_cast<int>(0xFFFFFFFFu - a[r]);
}

__global__ void __launch_bounds__(256) expert_segment_sort_kernel(const int* __restrict__ offsets, int64_t N,
                                                                  int* __restrict__ sorted_pair, int* __restrict__ num_long,
                                                                  int* __restrict__ long_experts) {
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t e = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; e < N; e += warps_total) {
    const int b = offsets[e], n = offsets[e + 1] - b;
    if (n < 2) continue;
    if (n <= 32) sort_segment<1>(sorted_pair + b, n, lane);
    else if (n <= 64) sort_segment<2>(sorted_pair + b, n, lane);
    else if (n <= kWarpSegment) sort_segment<8>(sorted_pair + b, n, lane);
    else if (lane == 0) long_experts[atomicAdd(num_long, 1)] = static_cast<int>(e);
  }
}

constexpr int kBitmapWords = 16384;  // pair ids per pass: 32 times as many
__global__ void __launch_bounds__(512) expert_long_sort_kernel(const int* __restrict__ offsets, const int* __restrict__ num_long,
                                                               const int* __restrict__ long_experts, int64_t P,
                                                               int* __restrict__ sorted_pair, int* __restrict__ temp) {
  extern __shared__ unsigned bitmap[];
  __shared__ int warp_sum[16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPer = kBitmapWords / 512;
  for (int l = blockIdx.x; l < *num_long; l += gridDim.x) {
    const int e = long_experts[l];
    const int b = offsets[e], en = offsets[e + 1];
    int done = b;
    for (int64_t r0 = 0; r0 < P; r0 += static_cast<int64_t>(kBitmapWords) * 32) {
      for (int i = threadIdx.x; i < kBitmapWords; i += 512) bitmap[i] = 0;
      __syncthreads();
      for (int i = b + threadIdx.x; i < en; i += 512) {
        const int64_t rel = sorted_pair[i] - r0;
        if (rel >= 0 && rel < static_cast<int64_t>(kBitmapWords) * 32) atomicOr(&bitmap[rel >> 5], 1u << (rel & 31));
      }
      __syncthreads();
      int mine = 0;
      for (int i = 0; i < kPer; ++i) mine += __popc(bitmap[threadIdx.x * kPer + i]);
      int incl = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += up;
      }
      if (lane == 31) warp_sum[warp] = incl;
      __syncthreads();
      int pos = done + incl - mine, all = 0;
      for (int w = 0; w < 16; ++w) {
        if (w < warp) pos += warp_sum[w];
        all += warp_sum[w];
      }
      for (int i = 0; i < kPer; ++i) {
        unsigned word = bitmap[threadIdx.x * kPer + i];
        while (word != 0) {
          const int bit = __ffs(word) - 1;
          word &= word - 1;
          temp[pos++] = static_cast<int>(r0 + (threadIdx.x * kPer + i) * 32 + bit);
        }
      }
      done += all;
      __syncthreads();
    }
    for (int i = b + threadIdx.x; i < en; i += 512) sorted_pair[i] = temp[i];
    __syncthreads();
  }
}

// in: s_in (raw <x, D>; may alias s_ds), q (raw <dout, U>), gates.  out: s_ds = ds, gs = silu(s) * g (over q), dgates.
template <typename T>
__global__ void expert_bwd_pairs_kernel(const float* s_in, float* s_ds, float* __restrict__ q_gs,
                                        const T* __restrict__ gates, const int64_t* __restrict__ idx, int64_t N,
                                        T* __restrict__ dgates, int64_t P) {
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t e = idx[p];
    if (e < 0 || e >= N) {  // a skipped pair contributes nothing and receives no gradient
      s_ds[p] = 0.f;
      q_gs[p] = 0.f;
      dgates[p] = from_f32<T>(0.f);
      continue;
    }
    const float s = s_in[p], q = q_gs[p], g = to_f32<T>(gates[p]);
    const float sig = __fdividef(1.0f, 1.0f + __expf(-s));
    const float act = s * sig;
    s_ds[p] = q * g * (sig * (1.0f + s * (1.0f - sig)));
    q_gs[p] = act * g;
    dgates[p] = from_f32<T>(q * act);
  }
}

// One warp per (chunk of sorted pairs, block of 32*VEC*NCH columns).  The warp walks its pairs in sorted
// order with the running sums of the current expert's two gradient rows in registers.  An expert of up to kWholeExpert
// pairs belongs whole to the chunk in which it begins and its rows are stored directly; a longer one is split at the chunk
// boundaries, its partial sums go to `partial` (slot 0: the expert began in an earlier chunk, slot 1: it began here and
// continues) and expert_bwd_finish_kernel adds the pieces in chunk order.  (With every expert split at the boundaries the
// partial rows were 134 MB written and read at the benchmark shape.)
// Bound by the gather of one x and one dout row per pair (1.07 GB at 4096 tokens x 1024 columns, top-64): 9.9 TB/s.
constexpr int kWholeExpert = 256;
// first sorted position of chunk c
__device__ __forceinline__ int chunk_begin(int64_t c, int chunk_pairs, int total, const int* __restrict__ sorted_expert,
                                           const int* __restrict__ offsets) {
  if (c * chunk_pairs >= total) return total;
  const int pos = static_cast<int>(c * chunk_pairs);
  const int e = sorted_expert[pos];
  const int b = offsets[e], en = offsets[e + 1];
  return b == pos || en - b > kWholeExpert ? pos : en;
}
template <typename T, int NCH, int DEPTH>
__global__ void __launch_bounds__(128) expert_bwd_tables_kernel(
    const T* __restrict__ x, const T* __restrict__ dout, const float* __restrict__ ds, const float* __restrict__ gs,
    const int* __restrict__ sorted_pair, const int* __restrict__ sorted_expert, const int* __restrict__ offsets,
    int64_t N, T* __restrict__ ddown, T* __restrict__ dup, float* __restrict__ partial_d, float* __restrict__ partial_u,
    int H, int k, int colblocks, int chunk_pairs) {
  constexpr int VEC = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t warp_global = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int total = offsets[N];
  const int64_t nchunks = (total + chunk_pairs - 1) / chunk_pairs;
  for (int64_t task = warp_global; task < nchunks * colblocks; task += warps_total) {
    const int64_t chunk = task / colblocks;
    const int cb = static_cast<int>(task - chunk * colblocks);
    const int col0 = cb * (32 * VEC * NCH);
    const int pos0 = chunk_begin(chunk, chunk_pairs, total, sorted_expert, offsets);
    const int pos1 = chunk_begin(chunk + 1, chunk_pairs, total, sorted_expert, offsets);
    if (pos0 >= pos1) continue;
    bool in[NCH];
#pragma unroll
    for (int c = 0; c < NCH; ++c) in[c] = col0 + (c * 32 + lane) * VEC < H;
    uint64_t ad[NCH][VEC / 2], au[NCH][VEC / 2];  // packed pairs of float32 sums (fma.rn.f32x2)
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) ad[c][i] = au[c][i] = 0ull;

    int cur_e = sorted_expert[pos0];
    bool began_earlier = offsets[cur_e] < pos0;
    // flush the running sums of expert e: final row, or a partial sum for the finishing pass
    auto flush = [&](int e, bool partial, int slot) {
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int col = col0 + (c * 32 + lane) * VEC;
        if (!in[c]) continue;
        float fd[VEC], fu[VEC];
#pragma unroll
        for (int i = 0; i < VEC / 2; ++i) {
          unpack_f32x2(ad[c][i], fd[2 * i], fd[2 * i + 1]);
          unpack_f32x2(au[c][i], fu[2 * i], fu[2 * i + 1]);
          ad[c][i] = au[c][i] = 0ull;
        }
        if (partial) {
          float* pd = partial_d + (chunk * 2 + slot) * H + col;
          float* pu = partial_u + (chunk * 2 + slot) * H + col;
#pragma unroll
          for (int i = 0; i < VEC; i += 4) {
            *reinterpret_cast<float4*>(pd + i) = make_float4(fd[i], fd[i + 1], fd[i + 2], fd[i + 3]);
            *reinterpret_cast<float4*>(pu + i) = make_float4(fu[i], fu[i + 1], fu[i + 2], fu[i + 3]);
          }
        } else {
          *reinterpret_cast<uint4*>(ddown + static_cast<int64_t>(e) * H + col) = pack16<T>(fd);
          *reinterpret_cast<uint4*>(dup + static_cast<int64_t>(e) * H + col) = pack16<T>(fu);
        }
      }
    };

    // 32 pairs at a time: each lane fetches one pair's token, expert and weights, a batch ahead of their use; the rows of
    // DEPTH pairs are in flight together
    int t_next = 0, e_next = 0;
    float wd_next = 0.f, wu_next = 0.f;
    auto fetch_pairs = [&](int base) {
      if (base + lane < pos1) {
        const int p = sorted_pair[base + lane];
        e_next = sorted_expert[base + lane];
        t_next = p / k;
        wd_next = ds[p];
        wu_next = gs[p];
      }
    };
    fetch_pairs(pos0);
    for (int base = pos0; base < pos1; base += 32) {
      const int t_l = t_next, e_l = e_next;
      const float wd_l = wd_next, wu_l = wu_next;
      if (base + 32 < pos1) fetch_pairs(base + 32);
      const int n = min(32, pos1 - base);
      for (int s0 = 0; s0 < n; s0 += DEPTH) {
        uint4 xq[DEPTH][NCH], oq[DEPTH][NCH];
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
          const int64_t t = __shfl_sync(kFull, t_l, s0 + u);
          const bool have = s0 + u < n;
#pragma unroll
          for (int c = 0; c < NCH; ++c) {
            const int col = col0 + (c * 32 + lane) * VEC;
            xq[u][c] = have && in[c] ? ldg16(x + t * H + col) : make_uint4(0, 0, 0, 0);
            oq[u][c] = have && in[c] ? ldg16(dout + t * H + col) : make_uint4(0, 0, 0, 0);
          }
        }
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
          const int e = __shfl_sync(kFull, e_l, s0 + u);
          const float wd = __shfl_sync(kFull, wd_l, s0 + u), wu = __shfl_sync(kFull, wu_l, s0 + u);
          if (s0 + u >= n) break;
          if (e != cur_e) {  // warp-uniform: cur_e ends inside this chunk
            flush(cur_e, began_earlier, 0);
            cur_e = e;
            began_earlier = false;
          }
          const uint64_t wd2 = pack_f32x2(wd, wd), wu2 = pack_f32x2(wu, wu);
#pragma unroll
          for (int c = 0; c < NCH; ++c) {
            float xf[VEC], of[VEC];
            unpack16<T>(xq[u][c], xf);
            unpack16<T>(oq[u][c], of);
#pragma unroll
            for (int i = 0; i < VEC / 2; ++i) {
              ffma2(ad[c][i], pack_f32x2(xf[2 * i], xf[2 * i + 1]), wd2);
              ffma2(au[c][i], pack_f32x2(of[2 * i], of[2 * i + 1]), wu2);
            }
          }
        }
      }
    }
    const bool continues = offsets[cur_e + 1] > pos1;
    flush(cur_e, began_earlier || continues, began_earlier ? 0 : 1);
  }
}

// One warp per expert: rows of experts without pairs are zeroed, rows of experts split over several chunks are the sum of
// their partial rows in chunk order; rows stored by the pass above are left alone.
template <typename T>
__global__ void __launch_bounds__(256) expert_bwd_finish_kernel(const int* __restrict__ offsets, int64_t N,
                                                                const float* __restrict__ partial_d,
                                                                const float* __restrict__ partial_u,
                                                                T* __restrict__ ddown, T* __restrict__ dup, int H,
                                                                int chunk_pairs) {
  constexpr int VEC = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
  const int64_t warps_total = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t e = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; e < N; e += warps_total) {
    const int b = offsets[e], en = offsets[e + 1];
    if (b != en && en - b <= kWholeExpert) continue;
    T* rd = ddown + e * H;
    T* ru = dup + e * H;
    const int c0 = b / chunk_pairs, c1 = b == en ? c0 - 1 : (en - 1) / chunk_pairs;  // no pairs: the empty sum
    for (int col = lane * VEC; col < H; col += 32 * VEC) {
      float sd[VEC], su[VEC];
#pragma unroll
      for (int i = 0; i < VEC; ++i) sd[i] = su[i] = 0.f;
      for (int c = c0; c <= c1; ++c) {
        const int64_t row = static_cast<int64_t>(c) * 2 + (c == c0 ? 1 : 0);
        const float* pd = partial_d + row * H + col;
        const float* pu = partial_u + row * H + col;
#pragma unroll
        for (int i = 0; i < VEC; i += 4) {
          const float4 a = *reinterpret_cast<const float4*>(pd + i);
          const float4 u = *reinterpret_cast<const float4*>(pu + i);
          sd[i] += a.x; sd[i + 1] += a.y; sd[i + 2] += a.z; sd[i + 3] += a.w;
          su[i] += u.x; su[i + 1] += u.y; su[i + 2] += u.z; su[i + 3] += u.w;
        }
      }
      *reinterpret_cast<uint4*>(rd + col) = pack16<T>(sd);
      *reinterpret_cast<uint4*>(ru + col) = pack16<T>(su);
    }
  }
}

// Tables sharded over the GPUs of one node, rows of the other GPUs read through peer pointers: the two gather
// kernels with the row address computed from (e % world, e / world).
// hot_down / hot_up (nullable, hot_rows rows): tables replicated on every GPU, addressed by the ids N .. N + hot_rows - 1
template <typename T>
int run_typed_peer(const void* x, const void* const* down_shards, const void* const* up_shards, int world,
                   const int64_t* idx, const void* gates, void* out, int out_f32, int64_t T_, int H, int64_t N, int k,
                   const ExpertWs& w, int32_t* status, cudaStream_t stream, const void* hot_down, const void* hot_up,
                   int64_t hot_rows) {
  if constexpr (sizeof(T) != 2) {
    return FMOE_ERR_UNSUPPORTED;
  } else {
    constexpr int VEC = Vec16<T>::N;
    const int sms = device_sm_count();
    // the same kernels, at the same sizes, as the unsharded forward: the results are bit-equal
    const PeerTable pd{down_shards, world, N}, pu{up_shards, world, N};
    cudaError_t split_rc = cudaSuccess;
    if (try_scores_split<T, true>(x, hot_down, idx, gates, w.gs, T_, H, N + hot_rows, k, status, stream, kActSilu, nullptr, pd,
                                  &split_rc)) {
      FMOE_CUDA_TRY(split_rc);
    } else {
      const int64_t want = (T_ * ((k + 15) / 16) + 3) / 4;
      const int64_t cap = static_cast<int64_t>(sms) * 16;
      const int grid = static_cast<int>(want < cap ? want : cap);
      const int smem = 4 * 2 * ((H + 255) / 256 * 32) * 16;  // two x-row buffers per warp
      auto kern = whole_lines<T>(N, H) ? expert_scores_mma_kernel<T, true, 16> : expert_scores_mma_kernel<T, true, 8>;
      FMOE_CUDA_TRY(allow_smem(kern, smem));
      kern<<<grid, 128, smem, stream>>>(static_cast<const T*>(x), static_cast<const T*>(hot_down), idx,
                                        static_cast<const T*>(gates), w.gs, T_, H, N + hot_rows, k, H, status,
                                        kActSilu, reinterpret_cast<const T* const*>(down_shards), world, nullptr, N);
      FMOE_LAUNCH_CHECK();
    }
    if (try_accum_split<T, true>(hot_up, idx, w.gs, out, out_f32, T_, H, N + hot_rows, k, false, stream, pu, &split_rc)) {
      FMOE_CUDA_TRY(split_rc);
      return FMOE_OK;
    }
    const int need = (H + 32 * VEC - 1) / (32 * VEC);
    const int nch = need <= 1 ? 1 : 2;
    const int colblocks = (H + 32 * VEC * nch - 1) / (32 * VEC * nch);
    const int64_t want = (T_ * colblocks + 3) / 4;
    const int64_t cap = static_cast<int64_t>(sms) * 16;
    const int grid = static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
    const T* const* us = reinterpret_cast<const T* const*>(up_shards);
#define FMOE_PEER_ACCUM(OUT_, NCH_)                                                                            \
  expert_accum_kernel<T, OUT_, NCH_, true><<<grid, 128, 0, stream>>>(static_cast<const T*>(hot_up), idx, w.gs,    \
                                                                     static_cast<OUT_*>(out), T_, H, N + hot_rows, k, \
                                                                     colblocks, us, world, N)
    if (out_f32) {
      if (nch == 1) FMOE_PEER_ACCUM(float, 1);
      else FMOE_PEER_ACCUM(float, 2);
    } else {
      if (nch == 1) FMOE_PEER_ACCUM(T, 1);
      else FMOE_PEER_ACCUM(T, 2);
    }
#undef FMOE_PEER_ACCUM
    FMOE_LAUNCH_CHECK();
    return FMOE_OK;
  }
}

template <typename T>
__global__ void weights_to_f32_kernel(const T* __restrict__ w, float* __restrict__ out, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = to_f32<T>(w[i]);
}

template <typename T>
int run_weighted_rows(const void* values, const void* weights, const int64_t* idx, void* out, int64_t T_, int H,
                      int64_t N, int k, float* coef, cudaStream_t stream) {
  const int64_t P = T_ * k;
  const int64_t want = (P + 255) / 256;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 8;
  weights_to_f32_kernel<T><<<static_cast<int>(want < cap ? want : cap), 256, 0, stream>>>(static_cast<const T*>(weights),
                                                                                          coef, P);
  FMOE_LAUNCH_CHECK();
  return run_accum<T>(values, idx, coef, out, sizeof(T) == 4 ? 1 : 0, T_, H, N, k, stream);
}

struct ExpertBwdWs {
  float* ds;          // s, then ds
  float* q;           // <dout, U>, then silu(s) * g
  int* counts;        // [N + 1]: per expert, then the number of long segments
  int* offsets;       // [N + 1]
  int* tile_sums;
  int* rank;
  int* sorted_pair;
  int* sorted_expert;
  int* long_experts;  // experts of more than kWarpSegment pairs
  int* temp;          // [P]
  float* partial_d;
  float* partial_u;
  size_t bytes;
};

ExpertBwdWs carve_bwd(void* ws, int64_t T, int H, int64_t N, int k) {
  Carver c{static_cast<char*>(ws)};
  ExpertBwdWs w;
  const int64_t P = T * k;
  const int64_t nchunks = (P + bwd_chunk(P) - 1) / bwd_chunk(P);
  w.ds = c.take<float>(P);
  w.q = c.take<float>(P);
  w.counts = c.take<int>(N + 1);
  w.offsets = c.take<int>(N + 1);
  w.tile_sums = c.take<int>((N + kScanTile - 1) / kScanTile);
  w.rank = c.take<int>(P);
  w.sorted_pair = c.take<int>(P);
  w.sorted_expert = c.take<int>(P);
  w.long_experts = c.take<int>(P / kWarpSegment + 1);
  w.temp = c.take<int>(P);
  w.partial_d = c.take<float>(static_cast<size_t>(nchunks) * 2 * H);
  w.partial_u = c.take<float>(static_cast<size_t>(nchunks) * 2 * H);
  w.bytes = c.off;
  return w;
}

template <typename T, int NCH, int DEPTH>
void launch_bwd_tables(const void* x, const void* dout, const ExpertBwdWs& w, int64_t N, void* ddown, void* dup, int H,
                       int k, int64_t P, cudaStream_t stream) {
  constexpr int VEC = Vec16<T>::N;
  const int colblocks = (H + 32 * VEC * NCH - 1) / (32 * VEC * NCH);
  const int64_t tasks = ((P + bwd_chunk(P) - 1) / bwd_chunk(P)) * colblocks;
  const int64_t want = (tasks + 3) / 4;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 16;
  const int grid = static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
  expert_bwd_tables_kernel<T, NCH, DEPTH><<<grid, 128, 0, stream>>>(
      static_cast<const T*>(x), static_cast<const T*>(dout), w.ds, w.q, w.sorted_pair, w.sorted_expert,
      w.offsets, N, static_cast<T*>(ddown), static_cast<T*>(dup), w.partial_d, w.partial_u, H, k, colblocks, bwd_chunk(P));
}

template <typename T>
int run_backward(const void* dout, const void* x, const void* down, const void* up, const int64_t* idx,
                 const void* gates, void* dx, void* ddown, void* dup, void* dgates, int64_t T_, int H, int64_t N, int k,
                 const ExpertBwdWs& w, int32_t* status, cudaStream_t stream, const float* saved_scores) {
  constexpr int VEC = Vec16<T>::N;
  const int64_t P = T_ * k;
  const int sms = device_sm_count();
  int rc;
  {  // the pairs in the order of their experts + segment offsets
    FMOE_CUDA_TRY(cudaMemsetAsync(w.counts, 0, static_cast<size_t>(N + 1) * 4, stream));
    const int64_t want = (P + 255) / 256;
    const int grid = static_cast<int>(want < sms * 8 ? want : sms * 8);
    expert_hist_kernel<<<grid, 256, 0, stream>>>(idx, P, N, w.counts, w.rank, status);
    FMOE_LAUNCH_CHECK();
    const int ntiles = static_cast<int>((N + kScanTile - 1) / kScanTile);
    if (ntiles > 16) {
      scan_tile_sums_kernel<<<ntiles, kScanThreads, 0, stream>>>(w.counts, N, w.tile_sums);
      FMOE_LAUNCH_CHECK();
      scan_apply_kernel<<<ntiles, kScanThreads, 0, stream>>>(w.counts, N, w.tile_sums, w.offsets);
    } else {
      scan_apply_kernel<<<ntiles, kScanThreads, 0, stream>>>(w.counts, N, nullptr, w.offsets);
    }
    FMOE_LAUNCH_CHECK();
    expert_scatter_kernel<<<grid, 256, 0, stream>>>(idx, w.rank, w.offsets, P, w.sorted_pair, w.sorted_expert);
    FMOE_LAUNCH_CHECK();
    const int64_t seg_want = (N + 7) / 8;
    const int seg_grid = static_cast<int>(seg_want < sms * 8 ? seg_want : sms * 8);
    expert_segment_sort_kernel<<<seg_grid, 256, 0, stream>>>(w.offsets, N, w.sorted_pair, w.counts + N, w.long_experts);
    FMOE_LAUNCH_CHECK();
    if (P > kWarpSegment) {
      FMOE_CUDA_TRY(allow_smem(expert_long_sort_kernel, kBitmapWords * 4));
      expert_long_sort_kernel<<<sms, 512, kBitmapWords * 4, stream>>>(w.offsets, w.counts + N, w.long_experts, P,
                                                                     w.sorted_pair, w.temp);
      FMOE_LAUNCH_CHECK();
    }
  }
  if (saved_scores == nullptr) {  // s = <x, D[e]> was not kept by the forward: recompute it
    rc = run_scores<T>(x, down, idx, nullptr, w.ds, T_, H, N, k, status, stream);
    if (rc != FMOE_OK) return rc;
  }
  rc = run_scores<T>(dout, up, idx, nullptr, w.q, T_, H, N, k, status, stream);
  if (rc != FMOE_OK) return rc;
  {
    const int64_t want = (P + 255) / 256;
    const int grid = static_cast<int>(want < sms * 8 ? want : sms * 8);
    expert_bwd_pairs_kernel<T><<<grid, 256, 0, stream>>>(saved_scores != nullptr ? saved_scores : w.ds, w.ds, w.q,
                                                        static_cast<const T*>(gates), idx, N, static_cast<T*>(dgates), P);
    FMOE_LAUNCH_CHECK();
  }
  rc = run_accum<T>(down, idx, w.ds, dx, sizeof(T) == 4 ? 1 : 0, T_, H, N, k, stream);
  if (rc != FMOE_OK) return rc;
  const int need = (H + 32 * VEC - 1) / (32 * VEC);
  // two 16-byte pieces of a row per lane and two pairs in flight measured best (4096 tokens x 1024 columns, top-64: 109 us;
  // four pieces and the weights of one pair at a time 152, four pieces and two pairs 194, two and four 132, one and four
  // 138); narrower column blocks where the tasks would not fill the SMs
  const int64_t tasks = (P + bwd_chunk(P) - 1) / bwd_chunk(P) * ((need + 1) / 2);
  if (need <= 1 || tasks < static_cast<int64_t>(sms) * 16)
    launch_bwd_tables<T, 1, 4>(x, dout, w, N, ddown, dup, H, k, P, stream);
  else
    launch_bwd_tables<T, 2, 2>(x, dout, w, N, ddown, dup, H, k, P, stream);
  FMOE_LAUNCH_CHECK();
  {
    const int64_t want = (N + 7) / 8, cap = static_cast<int64_t>(sms) * 8;
    const int grid = static_cast<int>(want < cap ? want : cap);
    expert_bwd_finish_kernel<T><<<grid, 256, 0, stream>>>(w.offsets, N, w.partial_d, w.partial_u,
                                                          static_cast<T*>(ddown), static_cast<T*>(dup), H, bwd_chunk(P));
    FMOE_LAUNCH_CHECK();
  }
  return FMOE_OK;
}

}  // namespace

size_t expert_forward_bytes(int64_t T, int k) { return carve(nullptr, T, k).bytes; }

// What the entry points of the op ask their callers for.  The forward needs expert_forward_bytes(); the rest, room for an
// order of the pairs by expert, is kept: callers hold buffers of this size, and the limit of fmoe_expert_forward_static is
// stated in it.
size_t expert_workspace_bytes(int64_t T, int H, int64_t N, int k) {
  (void)H;
  if (T < 0 || N < 0 || k < 0) return 0;
  Carver c{nullptr};
  c.take<int>(N);
  c.take<int>(N + 1);
  c.take<int>((N + kScanTile - 1) / kScanTile);
  for (int i = 0; i < 4; ++i) c.take<int>(T * k);
  return c.off;
}

// Few tokens, 16-bit: both passes in their few-token forms, the second of which also adds the shared MLP's output (and the
// residual) and rounds once.  `addend` is complete when the scores pass starts.
bool expert_forward_adding_supported(int dtype, int64_t T, int H, int64_t N, int k) {
  return dtype != FMOE_DTYPE_F32 && T > 0 && H % 8 == 0 && N <= 0x7FFFFFFFll && k > 0 && scores_split_warps(T, H, k) != 0 &&
         accum_split_warps(T, H, k, 256) != 0;
}

namespace {
template <typename T>
int run_adding(const void* x, const void* down, const void* up, const int64_t* idx, const void* gates, const float* addend,
               const void* residual, void* y, int64_t T_, int H, int64_t N, int k, const ExpertWs& w, int32_t* status,
               cudaStream_t stream) {
  cudaError_t rc = cudaSuccess;
  if (!try_scores_split<T, false>(x, down, idx, gates, w.gs, T_, H, N, k, status, stream, kActSilu, nullptr, PeerTable{}, &rc))
    return FMOE_ERR_UNSUPPORTED;
  FMOE_CUDA_TRY(rc);
  if (!try_accum_split<T, false>(up, idx, w.gs, y, 0, T_, H, N, k, true, stream, PeerTable{}, &rc, addend, residual))
    return FMOE_ERR_UNSUPPORTED;
  FMOE_CUDA_TRY(rc);
  return FMOE_OK;
}
}  // namespace

int launch_expert_forward_adding(const void* x, const void* down, const void* up, const int64_t* indices, const void* gates,
                                 const float* addend, const void* residual, void* y, int dtype, int64_t T, int H, int64_t N,
                                 int k, void* ws, size_t ws_bytes, int32_t* status, cudaStream_t stream) {
  if (!expert_forward_adding_supported(dtype, T, H, N, k)) return FMOE_ERR_UNSUPPORTED;
  if (!aligned16(x) || !aligned16(down) || !aligned16(up) || !aligned16(y)) return FMOE_ERR_ALIGNMENT;
  const ExpertWs w = carve(ws, T, k);
  if (ws == nullptr || ws_bytes < w.bytes) return FMOE_ERR_WORKSPACE;
  if (dtype == FMOE_DTYPE_BF16)
    return run_adding<__nv_bfloat16>(x, down, up, indices, gates, addend, residual, y, T, H, N, k, w, status, stream);
  return run_adding<__half>(x, down, up, indices, gates, addend, residual, y, T, H, N, k, w, status, stream);
}

int launch_expert_forward(const void* x, const void* down, const void* up, const int64_t* indices, const void* gates,
                          void* out, int dtype, int out_dtype, int64_t T, int H, int64_t N, int k, void* ws,
                          size_t ws_bytes, int32_t* status, cudaStream_t stream, void* const* between_passes, int act,
                          float* raw_scores, bool router_ids) {
  if (T < 0 || H <= 0 || N <= 0 || k < 0) return FMOE_ERR_BAD_ARG;
  if (act != kActSilu && act != kActGelu) return FMOE_ERR_BAD_ARG;
  if (out_dtype != dtype && out_dtype != FMOE_DTYPE_F32) return FMOE_ERR_BAD_ARG;
  if (T == 0) return FMOE_OK;
  if (x == nullptr || down == nullptr || up == nullptr || out == nullptr) return FMOE_ERR_BAD_ARG;
  if (k > 0 && (indices == nullptr || gates == nullptr)) return FMOE_ERR_BAD_ARG;
  if (N > 0x7FFFFFFFll || T * static_cast<int64_t>(k) > 0x7FFFFFFFll) return FMOE_ERR_UNSUPPORTED;
  const int vec = 16 / dtype_size(dtype);
  if (H % vec != 0) return FMOE_ERR_ALIGNMENT;
  if (!aligned16(x) || !aligned16(down) || !aligned16(up) || !aligned16(out)) return FMOE_ERR_ALIGNMENT;
  if (k == 0) {
    FMOE_CUDA_TRY(cudaMemsetAsync(out, 0, static_cast<size_t>(T) * H * dtype_size(out_dtype), stream));
    return FMOE_OK;
  }
  const ExpertWs w = carve(ws, T, k);
  if (ws == nullptr || ws_bytes < w.bytes) return FMOE_ERR_WORKSPACE;
  const int out_f32 = (out_dtype == FMOE_DTYPE_F32) ? 1 : 0;
  switch (dtype) {
    case FMOE_DTYPE_F32:
      return run_typed<float>(x, down, up, indices, gates, out, 1, T, H, N, k, w, status, stream, between_passes, act,
                              raw_scores, router_ids);
    case FMOE_DTYPE_BF16:
      return run_typed<__nv_bfloat16>(x, down, up, indices, gates, out, out_f32, T, H, N, k, w, status, stream,
                                      between_passes, act, raw_scores, router_ids);
    case FMOE_DTYPE_F16:
      return run_typed<__half>(x, down, up, indices, gates, out, out_f32, T, H, N, k, w, status, stream, between_passes,
                               act, raw_scores, router_ids);
    default:
      return FMOE_ERR_BAD_ARG;
  }
}

size_t expert_backward_workspace_bytes(int64_t T, int H, int64_t N, int k) {
  if (T < 0 || N < 0 || k < 0 || H <= 0) return 0;
  return carve_bwd(nullptr, T, H, N, k).bytes;
}

int launch_expert_backward(const void* dout, const void* x, const void* down, const void* up, const int64_t* indices,
                           const void* gates, void* dx, void* ddown, void* dup, void* dgates, int dtype, int64_t T,
                           int H, int64_t N, int k, void* ws, size_t ws_bytes, int32_t* status, cudaStream_t stream,
                           const float* saved_scores) {
  if (T < 0 || H <= 0 || N <= 0 || k < 0) return FMOE_ERR_BAD_ARG;
  if (dx == nullptr || ddown == nullptr || dup == nullptr) return FMOE_ERR_BAD_ARG;
  if (N > 0x7FFFFFFFll || T * static_cast<int64_t>(k) > 0x7FFFFFFFll) return FMOE_ERR_UNSUPPORTED;
  const int vec = 16 / dtype_size(dtype);
  if (H % vec != 0) return FMOE_ERR_ALIGNMENT;
  if (!aligned16(dx) || !aligned16(ddown) || !aligned16(dup)) return FMOE_ERR_ALIGNMENT;
  const size_t table_bytes = static_cast<size_t>(N) * H * dtype_size(dtype);
  if (T == 0 || k == 0) {  // no pairs: every gradient is zero
    FMOE_CUDA_TRY(cudaMemsetAsync(ddown, 0, table_bytes, stream));
    FMOE_CUDA_TRY(cudaMemsetAsync(dup, 0, table_bytes, stream));
    if (T > 0) FMOE_CUDA_TRY(cudaMemsetAsync(dx, 0, static_cast<size_t>(T) * H * dtype_size(dtype), stream));
    return FMOE_OK;
  }
  if (dout == nullptr || x == nullptr || down == nullptr || up == nullptr || indices == nullptr || gates == nullptr ||
      dgates == nullptr)
    return FMOE_ERR_BAD_ARG;
  if (!aligned16(dout) || !aligned16(x) || !aligned16(down) || !aligned16(up)) return FMOE_ERR_ALIGNMENT;
  const ExpertBwdWs w = carve_bwd(ws, T, H, N, k);
  if (ws == nullptr || ws_bytes < w.bytes) return FMOE_ERR_WORKSPACE;
  switch (dtype) {
    case FMOE_DTYPE_F32:
      return run_backward<float>(dout, x, down, up, indices, gates, dx, ddown, dup, dgates, T, H, N, k, w, status, stream,
                                 saved_scores);
    case FMOE_DTYPE_BF16:
      return run_backward<__nv_bfloat16>(dout, x, down, up, indices, gates, dx, ddown, dup, dgates, T, H, N, k, w, status,
                                         stream, saved_scores);
    case FMOE_DTYPE_F16:
      return run_backward<__half>(dout, x, down, up, indices, gates, dx, ddown, dup, dgates, T, H, N, k, w, status, stream,
                                  saved_scores);
    default:
      return FMOE_ERR_BAD_ARG;
  }
}

int launch_weighted_rows(const void* values, const void* weights, const int64_t* indices, void* out, int dtype,
                         int64_t T, int H, int64_t N, int k, void* ws, size_t ws_bytes, int32_t* status,
                         cudaStream_t stream) {
  (void)status;  // ids outside [0, N) contribute nothing (the accumulate pass skips them)
  if (T < 0 || H <= 0 || N <= 0 || k < 0) return FMOE_ERR_BAD_ARG;
  if (T == 0) return FMOE_OK;
  if (values == nullptr || out == nullptr) return FMOE_ERR_BAD_ARG;
  if (T * static_cast<int64_t>(k) > 0x7FFFFFFFll) return FMOE_ERR_UNSUPPORTED;
  if (H % (16 / dtype_size(dtype)) != 0 || !aligned16(values) || !aligned16(out)) return FMOE_ERR_ALIGNMENT;
  if (k == 0) {
    FMOE_CUDA_TRY(cudaMemsetAsync(out, 0, static_cast<size_t>(T) * H * dtype_size(dtype), stream));
    return FMOE_OK;
  }
  if (weights == nullptr || indices == nullptr) return FMOE_ERR_BAD_ARG;
  const size_t need = static_cast<size_t>(T) * k * 4;
  if (ws == nullptr || ws_bytes < need) return FMOE_ERR_WORKSPACE;
  float* coef = static_cast<float*>(ws);
  switch (dtype) {
    case FMOE_DTYPE_F32: return run_weighted_rows<float>(values, weights, indices, out, T, H, N, k, coef, stream);
    case FMOE_DTYPE_BF16: return run_weighted_rows<__nv_bfloat16>(values, weights, indices, out, T, H, N, k, coef, stream);
    case FMOE_DTYPE_F16: return run_weighted_rows<__half>(values, weights, indices, out, T, H, N, k, coef, stream);
    default: return FMOE_ERR_BAD_ARG;
  }
}

int launch_expert_forward_peer(const void* x, const void* const* down_shards, const void* const* up_shards, int world,
                               const int64_t* indices, const void* gates, void* out, int dtype, int out_dtype, int64_t T,
                               int H, int64_t N, int k, void* ws, size_t ws_bytes, int32_t* status, cudaStream_t stream,
                               const void* hot_down, const void* hot_up, int64_t hot_rows) {
  if (T < 0 || H <= 0 || N <= 0 || k < 0 || world < 1 || hot_rows < 0) return FMOE_ERR_BAD_ARG;
  if (hot_rows > 0 && (hot_down == nullptr || hot_up == nullptr || !aligned16(hot_down) || !aligned16(hot_up)))
    return FMOE_ERR_BAD_ARG;
  if (out_dtype != dtype && out_dtype != FMOE_DTYPE_F32) return FMOE_ERR_BAD_ARG;
  if (dtype == FMOE_DTYPE_F32) return FMOE_ERR_UNSUPPORTED;
  if (T == 0) return FMOE_OK;
  if (x == nullptr || down_shards == nullptr || up_shards == nullptr || out == nullptr) return FMOE_ERR_BAD_ARG;
  if (k > 0 && (indices == nullptr || gates == nullptr)) return FMOE_ERR_BAD_ARG;
  if (N + hot_rows > 0x7FFFFFFFll || T * static_cast<int64_t>(k) > 0x7FFFFFFFll) return FMOE_ERR_UNSUPPORTED;
  if (H % 8 != 0 || !aligned16(x) || !aligned16(out)) return FMOE_ERR_ALIGNMENT;
  if (k == 0) {
    FMOE_CUDA_TRY(cudaMemsetAsync(out, 0, static_cast<size_t>(T) * H * dtype_size(out_dtype), stream));
    return FMOE_OK;
  }
  const ExpertWs w = carve(ws, T, k);
  if (ws == nullptr || ws_bytes < w.bytes) return FMOE_ERR_WORKSPACE;
  const int out_f32 = (out_dtype == FMOE_DTYPE_F32) ? 1 : 0;
  if (dtype == FMOE_DTYPE_BF16)
    return run_typed_peer<__nv_bfloat16>(x, down_shards, up_shards, world, indices, gates, out, out_f32, T, H, N, k, w,
                                         status, stream, hot_down, hot_up, hot_rows);
  if (dtype == FMOE_DTYPE_F16)
    return run_typed_peer<__half>(x, down_shards, up_shards, world, indices, gates, out, out_f32, T, H, N, k, w, status,
                                  stream, hot_down, hot_up, hot_rows);
  return FMOE_ERR_BAD_ARG;
}

}  // namespace fmoe
