// SIMT kernels for what the tensor-core path does not take: f32 chains (tcgen05
// has no f32 MMA), f16 chains too small or too unaligned for it, and the
// unfused five-kernel pipeline the A/B harness compares the fused kernel with.
// k is accumulated in ascending order in f32, like a scalar loop nest.
#include "wtc_kernels.h"
#include "wtc_ptx.cuh"

#include <cuda_fp16.h>

namespace wtc {
namespace {

constexpr int kSimtThreads = 256;
constexpr int kKChunk = 64;
constexpr size_t kRowLimit = 200 * 1024;   // shared memory of the row kernel: bounds the rows the SIMT path takes

template <bool F16>
__device__ __forceinline__ float ld_elem(const void *p, int64_t i) {
  if (F16) return __half2float(static_cast<const __half *>(p)[i]);
  return static_cast<const float *>(p)[i];
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// logits tile of R rows x N columns: thread t owns columns t, t+256, ...
// shared: As[R][kKChunk] then S[R][N]
template <int R, bool F16>
__device__ __forceinline__ void matmul_rows(const void *A, const void *B, const SimtParams &p, int64_t a_off,
                                            int64_t b_off, int row0, int rows, float *As, float *S) {
  for (int j0 = 0; j0 < p.N; j0 += kSimtThreads) {
    const int j = j0 + threadIdx.x;
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    for (int k0 = 0; k0 < p.K; k0 += kKChunk) {
      const int kc = min(kKChunk, p.K - k0);
      __syncthreads();
      for (int i = threadIdx.x; i < R * kKChunk; i += kSimtThreads) {
        const int r = i / kKChunk, k = i - r * kKChunk;
        As[i] = (r < rows && k < kc) ? ld_elem<F16>(A, a_off + static_cast<int64_t>(row0 + r) * p.lda + k0 + k) : 0.f;
      }
      __syncthreads();
      if (j < p.N) {
        // sixteen independent loads of B's column are in flight before the first is used (a thread
        // walks down one column: without this the loop is a chain of L2 round trips); k stays ascending
        int k = 0;
        for (; k + 16 <= kc; k += 16) {
          float bv[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) bv[u] = ld_elem<F16>(B, b_off + static_cast<int64_t>(k0 + k + u) * p.ldb + j);
#pragma unroll
          for (int u = 0; u < 16; ++u) {
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fmaf(As[r * kKChunk + k + u], bv[u], acc[r]);
          }
        }
        for (; k < kc; ++k) {
          const float bv = ld_elem<F16>(B, b_off + static_cast<int64_t>(k0 + k) * p.ldb + j);
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] = fmaf(As[r * kKChunk + k], bv, acc[r]);
        }
      }
    }
    if (j < p.N) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float s = acc[r];
        if (p.acc_mode == 1) s = __half2float(__float2half_rn(s));
        S[static_cast<int64_t>(r) * p.N + j] = s * p.scale;
      }
    }
  }
  __syncthreads();
}

template <int R, bool F16>
__global__ void __launch_bounds__(kSimtThreads)
simt_fused_kernel(const void *__restrict__ A, const void *__restrict__ B, void *__restrict__ Out, const SimtParams p) {
  extern __shared__ float sm[];
  float *As = sm;
  float *S = sm + R * kKChunk;
  const int blocks_per_batch = (p.M + R - 1) / R;
  const int b = blockIdx.x / blocks_per_batch;
  const int row0 = (blockIdx.x - b * blocks_per_batch) * R;
  const int rows = min(R, p.M - row0);
  matmul_rows<R, F16>(A, B, p, b * p.a_batch_stride, b * p.b_batch_stride, row0, rows, As, S);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < rows; r += kSimtThreads / 32) {
    float *s = S + static_cast<int64_t>(r) * p.N;
    float mx = -3.4028235e38f;
    for (int j = lane; j < p.N; j += 32) mx = fmaxf(mx, s[j]);
    mx = warp_max(mx);
    float sum = 0.f;
    for (int j = lane; j < p.N; j += 32) { const float e = expf(s[j] - mx); s[j] = e; sum += e; }
    sum = warp_sum(sum);
    const int64_t o = b * p.o_batch_stride + static_cast<int64_t>(row0 + r) * p.ldo;
    if (p.out_f16) {
      __half *out = static_cast<__half *>(Out) + o;
      for (int j = lane; j < p.N; j += 32) out[j] = __float2half_rn(s[j] / sum);
    } else {
      float *out = static_cast<float *>(Out) + o;
      for (int j = lane; j < p.N; j += 32) out[j] = s[j] / sum;
    }
  }
}

// ---- f32 operands, register-tiled ------------------------------------------------------------
// A CTA of WR x WC warps owns a BM x BN tile (BM = WR * 4 * TM, BN = WC * 64); a thread TM rows x 8
// columns of it, accumulated as row pairs with two-wide f32 FMAs (fma.rn.f32x2: each half rounds
// like fmaf, and k ascends, so the sums are those of a scalar loop nest).  Operands come through a
// ring of 16-deep stages filled with cp.async: A element-wise, transposed on the way ([k][row], so
// that a thread reads four rows at once), B sixteen bytes at a time where its rows allow it; what
// lies outside the matrices is zero-filled.
//
// The CTAs of a cluster hold the column tiles of the same rows: the logits stay in registers, the
// row maximum and then the row sum go round the cluster through distributed shared memory, and the
// probabilities are written once.  Rows of more than eight column tiles (f32 output): the tiles store
// logits, and a row-softmax pass follows in place.
// Bound by the FMA pipes: 4096 x 1024 x 1024 takes 186 us (46 TFLOP/s; the 128 tiles of this shape can reach
// 64 of the chip's 74) where the row kernel, one column a thread, took 564 (every FMA there reads A from
// shared memory, and each row block reads B alone).  16 x 8 results a thread need six 16-byte reads of
// shared memory for 64 two-wide FMAs.
constexpr int kTileK = 16;
template <int TM, int WR, int WC> struct TileShape {
  static constexpr int BM = WR * 4 * TM, BN = WC * 64, kThreads = WR * WC * 32;
  static constexpr int kStages = TM == 16 ? 4 : 3;
  static constexpr int kAPitch = BM + 4;
  static constexpr int kAStage = kTileK * kAPitch, kBStage = kTileK * BN;       // floats
  static constexpr int kStatsOff = kStages * (kAStage + kBStage);
  static constexpr int kFloats = kStatsOff + (WC + 2 * 8 + 2) * BM;     // [WC] partial, 2 x [8] from the cluster, 2 x combined
  static constexpr size_t kSmem = kFloats * sizeof(float);
};

__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void fma_pair(uint64_t &acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 halves_of(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

template <int TM, int WR, int WC, bool VECB>
__global__ void __launch_bounds__(WR *WC * 32, TM == 16 ? 1 : 2)
simt_tile_kernel(const float *__restrict__ A, const float *__restrict__ B, void *__restrict__ Out, const SimtParams p, int num_rb, int num_nb,
                 int logits_only) {
  using T = TileShape<TM, WR, WC>;
  constexpr int BM = T::BM, BN = T::BN, NT = T::kThreads, ST = T::kStages;
  constexpr int A_PER = BM * kTileK / NT, B_PER = kTileK * BN / (VECB ? 4 : 1) / NT;
  static_assert(NT % kTileK == 0 && BM * kTileK % NT == 0 && kTileK * BN / (VECB ? 4 : 1) % NT == 0, "whole rounds of copies");
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = warp / WC, wc = warp - wr * WC;
  const int rg = lane >> 3, cg = lane & 7;
  const int nb = blockIdx.x % num_nb;
  const int unit = blockIdx.x / num_nb;
  const int b = unit / num_rb, rb = unit - b * num_rb;
  const int row0 = rb * BM, col0 = nb * BN;
  if (!logits_only) cluster_arrive_release();          // my shared memory exists; completed before the first remote store

  // ---- copies: element e of A's share is row tid / 16 + e * (NT / 16), k = tid % 16 ----
  const int ak = tid % kTileK, am = tid / kTileK;
  const float *a_src = A + b * p.a_batch_stride + static_cast<int64_t>(row0 + am) * p.lda + ak;
  const uint32_t sm_base = smem_u32(sm);
  const uint32_t a_dst = sm_base + (ak * T::kAPitch + am) * 4;
  const float *b_base = B + b * p.b_batch_stride + col0;
  constexpr int CW = VECB ? BN / 4 : BN;               // copies per k-row of B
  auto load_stage = [&](int kb) {
    const int st = kb % ST, k0 = kb * kTileK;
    const uint32_t as = a_dst + st * T::kAStage * 4;
    const bool a_k = k0 + ak < p.K;
#pragma unroll
    for (int e = 0; e < A_PER; ++e) {
      const bool live = a_k && row0 + am + e * (NT / kTileK) < p.M;
      cp_async4(as + e * (NT / kTileK) * 4, live ? a_src + static_cast<int64_t>(e * (NT / kTileK)) * p.lda + k0 : A, live);
    }
    const uint32_t bs = sm_base + (ST * T::kAStage + st * T::kBStage) * 4;
#pragma unroll
    for (int e = 0; e < B_PER; ++e) {
      const int i = tid + e * NT, k = i / CW, c = i - k * CW;
      if (VECB) {
        const bool live = k0 + k < p.K && col0 + c * 4 < p.N;
        cp_async16(bs + (k * BN + c * 4) * 4, live ? b_base + static_cast<int64_t>(k0 + k) * p.ldb + c * 4 : B, live);
      } else {
        const bool live = k0 + k < p.K && col0 + c < p.N;
        cp_async4(bs + (k * BN + c) * 4, live ? b_base + static_cast<int64_t>(k0 + k) * p.ldb + c : B, live);
      }
    }
  };

  uint64_t acc[TM / 2][8];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;

  const int num_kb = (p.K + kTileK - 1) / kTileK;
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (s < num_kb) load_stage(s);
    cp_async_commit();
  }
  for (int kb = 0; kb < num_kb; ++kb) {
    cp_async_wait<ST - 2>();
    __syncthreads();                                    // stage kb has landed for everyone; stage kb - 1 has been read by everyone
    if (kb + ST - 1 < num_kb) load_stage(kb + ST - 1);
    cp_async_commit();
    const float *as = sm + (kb % ST) * T::kAStage + wr * 4 * TM + rg * 4;
    const float *bs = sm + ST * T::kAStage + (kb % ST) * T::kBStage + wc * 64 + cg * 4;
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      // a thread's pairs are rows: its eight values of B are the ones doubled, fewer moves than its TM of A
      const float4 b0 = *reinterpret_cast<const float4 *>(bs + k * BN), b1 = *reinterpret_cast<const float4 *>(bs + k * BN + 32);
      const uint64_t bb[8] = {pair_of(b0.x, b0.x), pair_of(b0.y, b0.y), pair_of(b0.z, b0.z), pair_of(b0.w, b0.w),
                              pair_of(b1.x, b1.x), pair_of(b1.y, b1.y), pair_of(b1.z, b1.z), pair_of(b1.w, b1.w)};
#pragma unroll
      for (int q = 0; q < TM / 4; ++q) {
        const ulonglong2 aa = *reinterpret_cast<const ulonglong2 *>(as + k * T::kAPitch + q * 16);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          fma_pair(acc[q * 2][j], aa.x, bb[j]);
          fma_pair(acc[q * 2 + 1][j], aa.y, bb[j]);
        }
      }
    }
  }

  // ---- logits ----
  float v[TM][8];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float2 s = halves_of(acc[i][j]);
      if (p.acc_mode == 1) { s.x = __half2float(__float2half_rn(s.x)); s.y = __half2float(__float2half_rn(s.y)); }
      v[2 * i][j] = s.x * p.scale;
      v[2 * i + 1][j] = s.y * p.scale;
    }
  const int trow = wr * 4 * TM + rg * 4;                 // row i of mine is trow + (i / 4) * 16 + i % 4 of the tile
  const int tcol = wc * 64 + cg * 4;                     // column j of mine is tcol + (j / 4) * 32 + j % 4
  const int cols = p.N - col0 - tcol;                    // columns from my first to the row's end
  auto tile_row = [&](int i) { return trow + (i / 4) * 16 + i % 4; };
  auto col_live = [&](int j) { return (j / 4) * 32 + j % 4 < cols; };

  if (!logits_only) {
    const uint32_t rank = cluster_ctarank(), cluster = cluster_nctarank();
    float *part = sm + T::kStatsOff;                     // [WC][BM]
    float *from = part + WC * BM;                        // [2][8][BM]: maxima, sums of the cluster's CTAs
    float *comb = from + 2 * 8 * BM;                     // [2][BM]
    // reduces one value per (thread, row) over the row: the eight lanes that share it, the WC warps, the cluster
    auto reduce_rows = [&](float (&x)[TM], bool is_max, int round) {
#pragma unroll
      for (int i = 0; i < TM; ++i) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          const float y = __shfl_xor_sync(0xffffffffu, x[i], o);
          x[i] = is_max ? fmaxf(x[i], y) : x[i] + y;
        }
        if (cg == 0) part[wc * BM + tile_row(i)] = x[i];
      }
      __syncthreads();
      if (round == 0) cluster_wait_acquire();            // every CTA of the cluster is running
      for (int r = tid; r < BM; r += NT) {
        float t = part[r];
#pragma unroll
        for (int w = 1; w < WC; ++w) t = is_max ? fmaxf(t, part[w * BM + r]) : t + part[w * BM + r];
        const uint32_t slot = smem_u32(from + (round * 8 + rank) * BM + r);
        for (uint32_t peer = 0; peer < cluster; ++peer) st_cluster_f32(map_to_cta(slot, peer), t);
      }
      __syncwarp();
      cluster_sync_all();
      for (int r = tid; r < BM; r += NT) {
        float t = from[round * 8 * BM + r];
        for (uint32_t c = 1; c < cluster; ++c) {
          const float y = from[(round * 8 + c) * BM + r];
          t = is_max ? fmaxf(t, y) : t + y;
        }
        comb[round * BM + r] = t;
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < TM; ++i) x[i] = comb[round * BM + tile_row(i)];
    };
    float x[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      x[i] = -3.4028235e38f;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col_live(j)) x[i] = fmaxf(x[i], v[i][j]);
    }
    reduce_rows(x, true, 0);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[i][j] = expf(v[i][j] - x[i]);
        if (col_live(j)) s += v[i][j];
      }
      x[i] = s;
    }
    reduce_rows(x, false, 1);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = v[i][j] / x[i];
  }

  const int es = p.out_f16 ? 2 : 4;
  const bool vec = p.ldo % 4 == 0 && p.o_batch_stride % 4 == 0 && reinterpret_cast<uintptr_t>(Out) % (4 * es) == 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = row0 + tile_row(i);
    if (r >= p.M) continue;
    const int64_t o = b * p.o_batch_stride + static_cast<int64_t>(r) * p.ldo + col0 + tcol;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = h * 32;
      if (vec && c + 4 <= cols) {
        if (p.out_f16) *reinterpret_cast<uint2 *>(static_cast<__half *>(Out) + o + c) = make_uint2(pack_f16x2(v[i][4 * h], v[i][4 * h + 1]), pack_f16x2(v[i][4 * h + 2], v[i][4 * h + 3]));
        else *reinterpret_cast<float4 *>(static_cast<float *>(Out) + o + c) = make_float4(v[i][4 * h], v[i][4 * h + 1], v[i][4 * h + 2], v[i][4 * h + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < cols) {
            if (p.out_f16) static_cast<__half *>(Out)[o + c + j] = __float2half_rn(v[i][4 * h + j]);
            else static_cast<float *>(Out)[o + c + j] = v[i][4 * h + j];
          }
      }
    }
  }
}

// ---- the unfused pipeline ----------------------------------------------------
template <int R, bool F16>
__global__ void __launch_bounds__(kSimtThreads)
unfused_matmul_kernel(const void *__restrict__ A, const void *__restrict__ B, float *__restrict__ C32, const SimtParams p) {
  extern __shared__ float sm[];
  float *As = sm;
  const int blocks_per_batch = (p.M + R - 1) / R;
  const int b = blockIdx.x / blocks_per_batch;
  const int row0 = (blockIdx.x - b * blocks_per_batch) * R;
  const int rows = min(R, p.M - row0);
  // write straight to global: S points at this block's rows of C32 (row stride N)
  float *S = C32 + (static_cast<int64_t>(b) * p.M + row0) * p.N;
  // rows beyond `rows` must not be written: matmul_rows writes R rows, so guard here
  if (rows == R) {
    matmul_rows<R, F16>(A, B, p, b * p.a_batch_stride, b * p.b_batch_stride, row0, rows, As, S);
  } else {
    for (int r = 0; r < rows; ++r) {
      SimtParams q = p;
      matmul_rows<1, F16>(A, B, q, b * p.a_batch_stride, b * p.b_batch_stride, row0 + r, 1, As, S + static_cast<int64_t>(r) * p.N);
    }
  }
}

__global__ void rowmax_kernel(const float *__restrict__ C32, float *__restrict__ mx, int64_t rows, int N) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float m = -3.4028235e38f;
  for (int j = lane; j < N; j += 32) m = fmaxf(m, C32[row * N + j]);
  m = warp_max(m);
  if (lane == 0) mx[row] = m;
}
__global__ void exp_kernel(const float *__restrict__ C32, const float *__restrict__ mx, float *__restrict__ E, int64_t total, int N) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    E[i] = expf(C32[i] - mx[i / N]);
}
__global__ void rowsum_kernel(const float *__restrict__ E, float *__restrict__ sum, int64_t rows, int N) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float s = 0.f;
  for (int j = lane; j < N; j += 32) s += E[row * N + j];
  s = warp_sum(s);
  if (lane == 0) sum[row] = s;
}
__global__ void div_kernel(const float *__restrict__ E, const float *__restrict__ sum, void *__restrict__ Out, int64_t rows_per_batch,
                           int64_t total, int N, int64_t ldo, int64_t o_batch_stride, int out_f16) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / N; const int j = static_cast<int>(i - row * N);
    const int64_t b = row / rows_per_batch, r = row - b * rows_per_batch;
    const float v = E[i] / sum[row];
    const int64_t o = b * o_batch_stride + r * ldo + j;
    if (out_f16) static_cast<__half *>(Out)[o] = __float2half_rn(v);
    else static_cast<float *>(Out)[o] = v;
  }
}

int pick_rows(const SimtParams &p, size_t smem_limit) {
  // largest R in {16,8,4,2,1} whose logits tile fits shared memory; small problems trade rows
  // per CTA for more CTAs (latency-bound: fill the 148 SMs before deepening the per-CTA work)
  int best = 0;
  for (int R = 16; R >= 1; R >>= 1) {
    const size_t need = (static_cast<size_t>(R) * kKChunk + static_cast<size_t>(R) * p.N) * sizeof(float);
    if (need > smem_limit) continue;
    if (!best) best = R;
    const int64_t blocks = static_cast<int64_t>(p.batch) * ((p.M + R - 1) / R);
    if (blocks >= 148) return R;
    best = R;
  }
  return best;
}

// The opt-in to more than 48 KB of dynamic shared memory is per kernel instance and per device:
// it is raised once to the largest window this instance has been asked for there, not on every call.
template <int R, bool IN16>
cudaError_t fused_r_window(size_t smem) {
  static size_t granted[64] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (smem > granted[dev]) {
    e = cudaFuncSetAttribute(simt_fused_kernel<R, IN16>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    granted[dev] = smem;
  }
  return cudaSuccess;
}

template <int R>
cudaError_t launch_fused_r(const void *A, const void *B, void *Out, const SimtParams &p, cudaStream_t s) {
  const size_t smem = (static_cast<size_t>(R) * kKChunk + static_cast<size_t>(R) * p.N) * sizeof(float);
  const int64_t blocks = static_cast<int64_t>(p.batch) * ((p.M + R - 1) / R);
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  cudaError_t e;
  if (p.in_f16) {
    e = fused_r_window<R, true>(smem);
    if (e != cudaSuccess) return e;
    simt_fused_kernel<R, true><<<static_cast<unsigned>(blocks), kSimtThreads, smem, s>>>(A, B, Out, p);
  } else {
    e = fused_r_window<R, false>(smem);
    if (e != cudaSuccess) return e;
    simt_fused_kernel<R, false><<<static_cast<unsigned>(blocks), kSimtThreads, smem, s>>>(A, B, Out, p);
  }
  return cudaGetLastError();
}

// The f32 tile shapes, largest first, and the one for a problem: the cheapest by (rounds of tiles) x (tile) / (how near to
// the FMA rate an SM full of such tiles gets).  A round is what is resident at once: tiles one by one where the logits go to
// the output, else whole clusters (of n CTAs at one a SM: 15 of eight on a 148-SM part, one short of 148 / n otherwise).
struct TileChoice { int bm, bn, per_sm; double rate; };
constexpr TileChoice kTileChoices[] = {{128, 256, 1, 1.0}, {64, 256, 2, 1.0}, {64, 128, 3, 0.9}, {32, 128, 4, 0.7}};

int pick_tile(const SimtParams &p) {
  static const int kResident[9] = {0, 148, 72, 47, 35, 27, 22, 18, 15};
  int best = 0;
  double cost = 0;
  for (int i = 0; i < 4; ++i) {
    const TileChoice &c = kTileChoices[i];
    const int64_t units = static_cast<int64_t>(p.batch) * ((p.M + c.bm - 1) / c.bm), nb = (p.N + c.bn - 1) / c.bn;
    // full rounds at the rate of a full SM; in the last one an SM holds fewer tiles
    const int64_t per_round = nb > 8 ? 148 : kResident[nb];
    const int64_t items = nb > 8 ? units * nb : units;
    const int64_t deep = (items + per_round - 1) / per_round;             // tiles on the busiest SM
    const double t = static_cast<double>(deep) * c.bm * c.bn / (deep >= c.per_sm ? c.rate : c.rate * (0.5 + 0.5 * deep / c.per_sm));
    if (i == 0 || t < cost) { best = i; cost = t; }
  }
  return best;
}

// f32 operands take the tiles from 2^23 multiply-adds on: below that the row kernel's one row per CTA
// spreads the little work over more SMs (256 x 256 x 64: 6.3 against 8.3 us; 128 x 1024 x 64: 12.4 against 9.7;
// 1024 x 1024 x 128: 35 against 14.5).  (R = 0: refused, rows longer than the row kernel takes.)  A row of
// more than eight column tiles keeps its logits in the output, so that has to be f32.
bool use_tiles(const SimtParams &p, int R) {
  if (p.in_f16 || R == 0 || p.M > 0x7fffffff - kTileChoices[0].bm) return false;      // (a tile's rows are counted in 32 bits)
  if (static_cast<double>(p.batch) * p.M * p.N * (p.K > 0 ? p.K : 1) < (1 << 23)) return false;
  return !p.out_f16 || p.N <= 8 * kTileChoices[pick_tile(p)].bn;
}

template <int TM, int WR, int WC, bool VECB>
cudaError_t launch_tile_v(const float *A, const float *B, void *Out, const SimtParams &p, bool logits_only, cudaStream_t s) {
  using T = TileShape<TM, WR, WC>;
  auto kern = simt_tile_kernel<TM, WR, WC, VECB>;
  static bool granted[64] = {false};           // the opt-in to more than 48 KB of shared memory, per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!granted[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(T::kSmem));
    if (e != cudaSuccess) return e;
    granted[dev] = true;
  }
  const int num_rb = (p.M + T::BM - 1) / T::BM, num_nb = (p.N + T::BN - 1) / T::BN;
  const int64_t blocks = static_cast<int64_t>(p.batch) * num_rb * num_nb;
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks), 1, 1);
  cfg.blockDim = dim3(T::kThreads, 1, 1);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = logits_only ? 1 : num_nb;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, A, B, Out, p, num_rb, num_nb, logits_only ? 1 : 0);
}

template <int TM, int WR, int WC>
cudaError_t launch_tile(const float *A, const float *B, void *Out, const SimtParams &p, bool logits_only, cudaStream_t s) {
  const bool vecb = p.N % 4 == 0 && p.ldb % 4 == 0 && p.b_batch_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0;
  return vecb ? launch_tile_v<TM, WR, WC, true>(A, B, Out, p, logits_only, s) : launch_tile_v<TM, WR, WC, false>(A, B, Out, p, logits_only, s);
}

template <int TM, int WR, int WC> SimtPlan tile_plan() {
  using T = TileShape<TM, WR, WC>;
  return SimtPlan{T::BM, T::BN, kTileK, 1, T::kThreads, static_cast<int>(T::kSmem), T::kStages, 1};
}

bool stacked_densely(const SimtParams &p) { return p.batch == 1 || p.o_batch_stride == static_cast<int64_t>(p.M) * p.ldo; }

cudaError_t launch_tiles(const void *A, const void *B, void *Out, const SimtParams &p, cudaStream_t s) {
  const float *a = static_cast<const float *>(A), *b = static_cast<const float *>(B);
  const int c = pick_tile(p);
  const bool logits_only = p.N > 8 * kTileChoices[c].bn;
  cudaError_t e;
  if (c == 0) e = launch_tile<16, 2, 4>(a, b, Out, p, logits_only, s);
  else if (c == 1) e = launch_tile<8, 2, 4>(a, b, Out, p, logits_only, s);
  else if (c == 2) e = launch_tile<8, 2, 2>(a, b, Out, p, logits_only, s);
  else e = launch_tile<4, 2, 2>(a, b, Out, p, logits_only, s);
  if (e != cudaSuccess || !logits_only) return e;
  const bool dense = stacked_densely(p);
  const int64_t rows = dense ? static_cast<int64_t>(p.batch) * p.M : p.M;
  for (int i = 0; i < (dense ? 1 : p.batch) && e == cudaSuccess; ++i) {
    float *o = static_cast<float *>(Out) + i * p.o_batch_stride;
    e = launch_row_chain(2, o, o, rows, p.N, p.ldo, p.ldo, 0, 0, 0.f, 0.f, s);
  }
  return e;
}

} // namespace

bool simt_fused_takes(const SimtParams &p) { return pick_rows(p, kRowLimit) != 0; }

SimtPlan simt_fused_plan(const SimtParams &p) {
  if (!use_tiles(p, pick_rows(p, kRowLimit))) return SimtPlan{16, p.N, kKChunk, 1, kSimtThreads, 0, 0, 1};
  const int c = pick_tile(p);
  const int nb = (p.N + kTileChoices[c].bn - 1) / kTileChoices[c].bn;
  SimtPlan r = c == 0 ? tile_plan<16, 2, 4>() : c == 1 ? tile_plan<8, 2, 4>() : c == 2 ? tile_plan<8, 2, 2>() : tile_plan<4, 2, 2>();
  r.cluster_n = nb > 8 ? 1 : nb;
  r.launches = nb > 8 ? 1 + (stacked_densely(p) ? 1 : p.batch) : 1;
  return r;
}

cudaError_t launch_simt_fused(const void *A, const void *B, void *Out, const SimtParams &p, cudaStream_t s) {
  if (p.batch <= 0 || p.M <= 0 || p.N <= 0) return cudaSuccess;
  const int R = pick_rows(p, kRowLimit);
  if (use_tiles(p, R)) return launch_tiles(A, B, Out, p, s);
  switch (R) {
    case 16: return launch_fused_r<16>(A, B, Out, p, s);
    case 8: return launch_fused_r<8>(A, B, Out, p, s);
    case 4: return launch_fused_r<4>(A, B, Out, p, s);
    case 2: return launch_fused_r<2>(A, B, Out, p, s);
    case 1: return launch_fused_r<1>(A, B, Out, p, s);
    default: return cudaErrorInvalidValue;  // one row of logits does not fit shared memory
  }
}

size_t simt_unfused_workspace_bytes(const SimtParams &p) {
  const size_t rows = static_cast<size_t>(p.batch) * p.M;
  // C32[rows,N], E[rows,N], max[rows], sum[rows]
  return (2 * rows * p.N + 2 * rows) * sizeof(float);
}

cudaError_t launch_simt_unfused(const void *A, const void *B, void *Out, void *workspace, const SimtParams &p,
                                cudaStream_t s) {
  if (p.batch <= 0 || p.M <= 0 || p.N <= 0) return cudaSuccess;
  const int64_t rows = static_cast<int64_t>(p.batch) * p.M;
  const int64_t total = rows * p.N;
  float *C32 = static_cast<float *>(workspace);
  float *E = C32 + total;
  float *mx = E + total;
  float *sum = mx + rows;
  constexpr int R = 8;
  const size_t smem = static_cast<size_t>(R) * kKChunk * sizeof(float);
  const int64_t blocks = static_cast<int64_t>(p.batch) * ((p.M + R - 1) / R);
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  if (p.in_f16) unfused_matmul_kernel<R, true><<<static_cast<unsigned>(blocks), kSimtThreads, smem, s>>>(A, B, C32, p);
  else unfused_matmul_kernel<R, false><<<static_cast<unsigned>(blocks), kSimtThreads, smem, s>>>(A, B, C32, p);
  return launch_softmax_passes(C32, E, mx, sum, Out, rows, p.M, p.N, p.ldo, p.o_batch_stride, p.out_f16, s);
}

cudaError_t launch_softmax_passes(const float *C32, float *E, float *mx, float *sum, void *Out, int64_t rows, int64_t rows_per_batch,
                                  int N, int64_t ldo, int64_t o_batch_stride, int out_f16, cudaStream_t s) {
  const int64_t total = rows * N;
  const unsigned row_grid = static_cast<unsigned>((rows + 7) / 8);
  const unsigned ew_grid = static_cast<unsigned>(total / 256 + 1 < 148 * 16 ? total / 256 + 1 : 148 * 16);
  rowmax_kernel<<<row_grid, 256, 0, s>>>(C32, mx, rows, N);
  exp_kernel<<<ew_grid, 256, 0, s>>>(C32, mx, E, total, N);
  rowsum_kernel<<<row_grid, 256, 0, s>>>(E, sum, rows, N);
  div_kernel<<<ew_grid, 256, 0, s>>>(E, sum, Out, rows_per_batch, total, N, ldo, o_batch_stride, out_f16);
  return cudaGetLastError();
}

} // namespace wtc
