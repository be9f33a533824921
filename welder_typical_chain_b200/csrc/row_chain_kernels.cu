// The two row-only chains of the reference's backend inputs, as single fused kernels:
//
//   row softmax       Out[i,:] = softmax(X[i,:])                      (max -> exp(x - max) -> sum -> divide;
//                     backend/welder/mlir_pipeline/softmax_row_chain.mlir:10-75)
//   row variance      Out[i,j] = c2 * sum_j (A[i,j] - c1 * sum_j A[i,j])^2 for every j
//                     (sum -> mean -> squared differences -> sum -> variance -> broadcast;
//                     backend/welder/mlir_pipeline/layernorm_variance_chain.mlir:12-104)
//
// Both are bandwidth-bound: every element is read once and written once, with 16-byte loads and
// stores (8 f16 or 4 f32 a lane), whatever the rows' starts and lengths: the few elements in front of
// a row's first 16-byte boundary and behind its last whole vector go one by one.  A row is owned by
// 8 or 16 lanes (rows of at most that many vectors), a warp (N <= 2048: 64 values a lane), one CTA of
// up to 512 threads (1024 for one form; up to 32768 f32 or 65536 f16 elements; f16 rows beyond 12288
// stay packed as loaded) or a cluster of up to eight such CTAs (131072 f32, 262144 f16); in all of them the row lives in registers between the
// passes.  Longer rows, and rows whose input and output lie differently to a 16-byte boundary, take
// a CTA per row that re-reads the row (from L2) for the second and third pass.  f32 or f16 elements
// (input and output of the same type); the arithmetic is f32.
#include "wtc_kernels.h"
#include "wtc_ptx.cuh"

namespace wtc {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kWarpRowMax = 2048;            // longest row a warp keeps in registers (64 values a lane)

__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <bool F16> __device__ __forceinline__ float load_elem(const void *p, int64_t i) {
  return F16 ? __half2float(static_cast<const __half *>(p)[i]) : static_cast<const float *>(p)[i];
}
template <bool F16> __device__ __forceinline__ void store_elem(void *p, int64_t i, float v) {
  if (F16) static_cast<__half *>(p)[i] = __float2half_rn(v);
  else static_cast<float *>(p)[i] = v;
}

// ---- block-wide reductions for the long-row kernels -------------------------------------------
__device__ __forceinline__ float block_reduce(float v, bool is_max, float *scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = is_max ? warp_max_f(v) : warp_sum_f(v);
  __syncthreads();                       // scratch may still be read from the previous reduction
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = lane < (blockDim.x >> 5) ? scratch[lane] : (is_max ? -INFINITY : 0.f);
  t = is_max ? warp_max_f(t) : warp_sum_f(t);
  return t;
}

// ---- 16-byte vectors: 8 f16 or 4 f32 ----------------------------------------------------------
template <bool F16> struct VecOf { static constexpr int N = F16 ? 8 : 4; };

template <bool F16> __device__ __forceinline__ void store_vec(void *base, int64_t elem, const float (&v)[VecOf<F16>::N]) {
  if (F16) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pack_f16x2(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4 *>(static_cast<__half *>(base) + elem) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    *reinterpret_cast<float4 *>(static_cast<float *>(base) + elem) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// ---- a vector as it was loaded: 8 halves or 4 floats in four registers -------------------------
template <bool F16> __device__ __forceinline__ void unpack_vec(const uint4 &q, float (&v)[VecOf<F16>::N]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  if (F16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(w[i]);
  }
}
template <bool F16> __device__ __forceinline__ uint4 load_raw(const void *base, int64_t elem) {
  return *reinterpret_cast<const uint4 *>(static_cast<const char *>(base) + elem * (F16 ? 2 : 4));
}

// The chain on a row that is spread over a group of threads (part of a warp, a warp, a CTA or a
// cluster of CTAs), NV vectors a thread: vector t of thread `tid` is vector number t * group + tid
// of the row, so that the group's loads are contiguous.  `reduce(x, is_max)` reduces over the group.
//
// RAGGED: the row may start anywhere and have any length.  The elements in front of its first
// 16-byte boundary and behind its last whole vector (at most V - 1 each) are spread over the
// group's first threads, one of each a thread; everything between goes in whole vectors.
//
// PACKED (f16): the row stays as it was loaded (half the registers, so that two 512-thread CTAs
// share an SM and the phases of different rows overlap); the exponentials are taken twice, once
// for the sum, once for the result: the special-function unit has the headroom, the memory system
// does not.
//
// The exponent is fma(x, log2 e, -max * log2 e) of f16 rows, (x - max) * log2 e of f32 ones: there the
// product's rounding alone passes an f32's exponent range from |max| = 2^31 on.  KIND 2 is the
// softmax of the f32 chain's logits (X and Out the same buffer): expf and a division, as the fused
// f32 kernel computes them.
template <int KIND, bool F16, int NV, bool RAGGED, bool PACKED, typename Reduce>
__device__ __forceinline__ void chain_on_row(const void *X, void *Out, int64_t in0, int64_t out0, int N, int tid, int group, float c1, float c2,
                                             Reduce reduce) {
  static_assert(!PACKED || F16, "packed rows: f16");
  constexpr int V = VecOf<F16>::N;
  constexpr float kFill = KIND != 1 ? -INFINITY : 0.f;
  constexpr uint32_t kRawFill = KIND != 1 ? (F16 ? 0xFC00FC00u : 0xFF800000u) : 0u;      // the same as loaded bits
  int head = 0, end = N;                        // whole vectors cover [head, end)
  if (RAGGED) {
    const int sh = static_cast<int>((reinterpret_cast<uintptr_t>(X) / (F16 ? 2 : 4) + static_cast<uint64_t>(in0)) & (V - 1));
    head = min((V - sh) & (V - 1), N);
    end = head + ((N - head) & ~(V - 1));
  }
  // vector t of this thread: where it starts behind a row's base, and whether it exists.  (Two spellings of the same that lead to
  // different registers: of the long f32 rows the softmax runs at 187 us with the one and at 196 with the other (4096 x 32000),
  // the variance at 149 and 120 (4096 x 24000).)
  constexpr bool kFromRow = !F16 && KIND != 1;
  const int first = head + tid * V, step = group * V;
  auto from = [&](int64_t base, int t) { return kFromRow ? base + (head + (t * group + tid) * V) : base + first + t * step; };
  auto have = [&](int t) { return kFromRow ? (t * group + tid) * V < end - head : first + t * step < end; };
  // all loads first: NV independent 16-byte requests a thread
  uint4 raw[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    raw[t] = make_uint4(kRawFill, kRawFill, kRawFill, kRawFill);
    if (have(t)) raw[t] = load_raw<F16>(X, from(in0, t));
  }
  const bool has_head = RAGGED && tid < head, has_tail = RAGGED && tid < N - end;
  float xh = kFill, xt = kFill;
  if (has_head) xh = load_elem<F16>(X, in0 + tid);
  if (has_tail) xt = load_elem<F16>(X, in0 + end + tid);
  float v[PACKED ? 1 : NV][V];
  if (!PACKED) {
#pragma unroll
    for (int t = 0; t < NV; ++t) unpack_vec<F16>(raw[t], v[PACKED ? 0 : t]);
  }
  auto vec = [&](int t) -> float (&)[V] {
    if (PACKED) unpack_vec<F16>(raw[t], v[0]);
    return v[PACKED ? 0 : t];
  };
  if (KIND != 1) {
    float m = RAGGED ? fmaxf(xh, xt) : -INFINITY;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      if (PACKED && !have(t)) continue;
      float(&x)[V] = vec(t);
#pragma unroll
      for (int e = 0; e < V; ++e) m = fmaxf(m, x[e]);
    }
    m = reduce(m, true);
    const float mb = m * kLog2e;
    auto ex = [&](float x) { return KIND == 2 ? expf(x - m) : !F16 ? ex2_approx((x - m) * kLog2e) : ex2_approx(fmaf(x, kLog2e, -mb)); };   // exp(x - max); -inf padding gives 0
    float s = 0.f;
    if (RAGGED) {
      xh = ex(xh); xt = ex(xt);
      s = xh + xt;
    }
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      if (PACKED && !have(t)) continue;
      float(&x)[V] = vec(t);
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float y = ex(x[e]);
        if (!PACKED) x[e] = y;
        s += y;
      }
    }
    s = reduce(s, false);
    const float inv = 1.0f / s;
    auto norm = [&](float x) { return KIND == 2 ? x / s : x * inv; };
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      if (have(t)) {
        float(&x)[V] = vec(t);
#pragma unroll
        for (int e = 0; e < V; ++e) x[e] = norm(PACKED ? ex(x[e]) : x[e]);
        store_vec<F16>(Out, from(out0, t), x);
      }
    }
    if (has_head) store_elem<F16>(Out, out0 + tid, norm(xh));
    if (has_tail) store_elem<F16>(Out, out0 + end + tid, norm(xt));
  } else {
    float s = RAGGED ? xh + xt : 0.f;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      float(&x)[V] = vec(t);                       // (padding is zeros)
#pragma unroll
      for (int e = 0; e < V; ++e) s += x[e];
    }
    const float mean = reduce(s, false) * c1;
    float q = 0.f;
    if (has_head) q += (xh - mean) * (xh - mean);
    if (has_tail) q += (xt - mean) * (xt - mean);
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      if (have(t)) {
        float(&x)[V] = vec(t);
#pragma unroll
        for (int e = 0; e < V; ++e) { const float d = x[e] - mean; q += d * d; }
      }
    }
    const float var = reduce(q, false) * c2;
    float o[V];
#pragma unroll
    for (int e = 0; e < V; ++e) o[e] = var;
#pragma unroll
    for (int t = 0; t < NV; ++t)
      if (have(t)) store_vec<F16>(Out, from(out0, t), o);
    if (has_head) store_elem<F16>(Out, out0 + tid, var);
    if (has_tail) store_elem<F16>(Out, out0 + end + tid, var);
  }
}

// G lanes per row (32 / G rows a warp, eight warps a CTA), the row in the lanes' registers.
template <int KIND, bool F16, int NV, bool RAGGED, int G>
__global__ void __launch_bounds__(256) row_chain_warp_kernel(const void *X, void *Out, int64_t rows, int N, int64_t ld_in, int64_t ld_out,
                                                             float c1, float c2) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / G) + threadIdx.x / G;
  const bool live = row < rows;                // (the shuffles take whole warps: rows that do not exist run along empty)
  chain_on_row<KIND, F16, NV, RAGGED, false>(X, Out, live ? row * ld_in : 0, row * ld_out, live ? N : 0, threadIdx.x & (G - 1), G, c1, c2,
                                             [](float x, bool is_max) {
#pragma unroll
                                               for (int o = G / 2; o > 0; o >>= 1) {
                                                 const float y = __shfl_xor_sync(0xffffffffu, x, o);
                                                 x = is_max ? fmaxf(x, y) : x + y;
                                               }
                                               return x;
                                             });
}

// One CTA of up to 512 threads per row, the row in the CTA's registers (NV vectors a thread).
template <int KIND, bool F16, int NV, bool RAGGED, bool PACKED>
__global__ void __launch_bounds__(512, PACKED ? 2 : 1)
row_chain_cta_kernel(const void *X, void *Out, int N, int64_t ld_in, int64_t ld_out, float c1, float c2) {
  __shared__ float scratch[32];
  chain_on_row<KIND, F16, NV, RAGGED, PACKED>(X, Out, static_cast<int64_t>(blockIdx.x) * ld_in, static_cast<int64_t>(blockIdx.x) * ld_out, N,
                                              threadIdx.x, blockDim.x, c1, c2,
                                              [&](float x, bool is_max) { return block_reduce(x, is_max, scratch); });
}

template <int KIND, bool RAGGED>
__global__ void __launch_bounds__(1024, 1)
row_chain_wide_cta_kernel(const void *X, void *Out, int N, int64_t ld_in, int64_t ld_out, float c1, float c2) {
  __shared__ float scratch[32];
  chain_on_row<KIND, true, 8, RAGGED, true>(X, Out, static_cast<int64_t>(blockIdx.x) * ld_in, static_cast<int64_t>(blockIdx.x) * ld_out, N,
                                          threadIdx.x, blockDim.x, c1, c2,
                                          [&](float x, bool is_max) { return block_reduce(x, is_max, scratch); });
}

// Softmax of long aligned f16 rows, sixteen packed vectors a thread: the packed form above with every
// step of a vector behind one check, which is what fits 64 registers almost without spills.
template <int NV>
__global__ void __launch_bounds__(512, 2) row_softmax_cta_packed_kernel(const void *X, void *Out, int N, int64_t ld_in, int64_t ld_out) {
  __shared__ float scratch[32];
  const int64_t in0 = static_cast<int64_t>(blockIdx.x) * ld_in, out0 = static_cast<int64_t>(blockIdx.x) * ld_out;
  const int tid = threadIdx.x, group = blockDim.x;
  const auto reduce = [&](float x, bool is_max) { return block_reduce(x, is_max, scratch); };
  const __half *x = static_cast<const __half *>(X);
  uint4 raw[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    const int j = (t * group + tid) * 8;
    raw[t] = j < N ? *reinterpret_cast<const uint4 *>(x + in0 + j) : make_uint4(0u, 0u, 0u, 0u);
  }
  float m = -INFINITY;
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    if ((t * group + tid) * 8 < N) {
      float v[8]; unpack_vec<true>(raw[t], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) m = fmaxf(m, v[e]);
    }
  }
  m = reduce(m, true);
  const float mb = m * kLog2e;
  float s = 0.f;
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    if ((t * group + tid) * 8 < N) {
      float v[8]; unpack_vec<true>(raw[t], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) s += ex2_approx(fmaf(v[e], kLog2e, -mb));
    }
  }
  s = reduce(s, false);
  const float inv = 1.0f / s;
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    const int j = (t * group + tid) * 8;
    if (j < N) {
      float v[8]; unpack_vec<true>(raw[t], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = ex2_approx(fmaf(v[e], kLog2e, -mb)) * inv;
      store_vec<true>(Out, out0 + j, v);
    }
  }
}

// A cluster of CTAs of 512 threads per row: rows that do not fit one CTA's registers.  The CTAs
// exchange their two partial reductions through distributed shared memory.  (Aligned rows too take
// the ragged form here: with no ends it costs nothing.)
template <int KIND, bool F16, int NV, bool PACKED>
__global__ void __launch_bounds__(512, 2)
row_chain_cluster_kernel(const void *X, void *Out, int N, int64_t ld_in, int64_t ld_out, float c1, float c2) {
  __shared__ float scratch[32];
  __shared__ float peers[2][8];
  const uint32_t rank = cluster_ctarank(), cluster = cluster_nctarank();
  const int64_t row = blockIdx.x / cluster;
  cluster_arrive_release();                    // my shared memory exists ...
  int round = 0;
  chain_on_row<KIND, F16, NV, true, PACKED>(X, Out, row * ld_in, row * ld_out, N, rank * blockDim.x + threadIdx.x, cluster * blockDim.x, c1, c2,
                                            [&](float x, bool is_max) {
    x = block_reduce(x, is_max, scratch);
    if (round == 0) cluster_wait_acquire();    // ... and so does everyone's
    if (threadIdx.x < cluster) st_cluster_f32(map_to_cta(smem_u32(&peers[round][rank]), threadIdx.x), x);
    __syncwarp();
    cluster_sync_all();
    float t = is_max ? -INFINITY : 0.f;
    for (uint32_t i = 0; i < cluster; ++i) t = is_max ? fmaxf(t, peers[round][i]) : t + peers[round][i];
    ++round;
    return t;
  });
}

// One CTA per row, any length and alignment: three passes over the row (the second and third come from L2).
template <int KIND, bool IN16, bool OUT16>
__global__ void __launch_bounds__(256) row_chain_block_kernel(const void *X, void *Out, int N, int64_t ld_in,
                                                              int64_t ld_out, float c1, float c2) {
  __shared__ float scratch[32];
  const int64_t in0 = static_cast<int64_t>(blockIdx.x) * ld_in, out0 = static_cast<int64_t>(blockIdx.x) * ld_out;
  if (KIND != 1) {
    float m = -INFINITY;
    for (int j = threadIdx.x; j < N; j += blockDim.x) m = fmaxf(m, load_elem<IN16>(X, in0 + j));
    m = block_reduce(m, true, scratch);
    auto ex = [&](float x) { return KIND == 2 ? expf(x - m) : ex2_approx((x - m) * kLog2e); };
    float s = 0.f;
    for (int j = threadIdx.x; j < N; j += blockDim.x) s += ex(load_elem<IN16>(X, in0 + j));
    s = block_reduce(s, false, scratch);
    const float inv = 1.0f / s;
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      const float y = ex(load_elem<IN16>(X, in0 + j));
      store_elem<OUT16>(Out, out0 + j, KIND == 2 ? y / s : y * inv);
    }
  } else {
    float s = 0.f;
    for (int j = threadIdx.x; j < N; j += blockDim.x) s += load_elem<IN16>(X, in0 + j);
    const float mean = block_reduce(s, false, scratch) * c1;
    float q = 0.f;
    for (int j = threadIdx.x; j < N; j += blockDim.x) { const float d = load_elem<IN16>(X, in0 + j) - mean; q += d * d; }
    const float var = block_reduce(q, false, scratch) * c2;
    for (int j = threadIdx.x; j < N; j += blockDim.x) store_elem<OUT16>(Out, out0 + j, var);
  }
}

// Aligned rows (16-byte starts, N a multiple of the vector) and ragged ones (any start and length,
// input and output equally far from a 16-byte boundary) take the same kernels; the ragged instances
// carry the element-wise ends.
template <int KIND, bool F16, bool RAGGED>
cudaError_t launch_rows(const void *X, void *Out, int64_t rows, int N, int64_t ld_in, int64_t ld_out, float c1, float c2, cudaStream_t s) {
  constexpr int V = VecOf<F16>::N;
  if (N <= kWarpRowMax) {
    const int nv = (N + 32 * V - 1) / (32 * V);            // vectors a lane
    constexpr int kMaxNv = 64 / V;                          // 64 values a lane at most
    const auto grid = [&](int g) { return static_cast<unsigned>((rows + 256 / g - 1) / (256 / g)); };
    // short rows: with a warp per row most lanes would hold no vector at all
    if (N <= 8 * V) row_chain_warp_kernel<KIND, F16, 1, RAGGED, 8><<<grid(8), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else if (N <= 16 * V) row_chain_warp_kernel<KIND, F16, 1, RAGGED, 16><<<grid(16), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else if (nv <= 1) row_chain_warp_kernel<KIND, F16, 1, RAGGED, 32><<<grid(32), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else if (nv <= 2) row_chain_warp_kernel<KIND, F16, 2, RAGGED, 32><<<grid(32), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else if (nv <= 4) row_chain_warp_kernel<KIND, F16, 4, RAGGED, 32><<<grid(32), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else if (nv <= 8 || kMaxNv == 8) row_chain_warp_kernel<KIND, F16, 8, RAGGED, 32><<<grid(32), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    else row_chain_warp_kernel<KIND, F16, kMaxNv, RAGGED, 32><<<grid(32), 256, 0, s>>>(X, Out, rows, N, ld_in, ld_out, c1, c2);
    return cudaGetLastError();
  }
  const unsigned g = static_cast<unsigned>(rows);
  // as many threads as the row needs with 4, 8 or (f32) 16 vectors a thread, in whole warps, 512 at most
  auto threads_for = [&](int n, int nv) { return (((n + nv * V - 1) / (nv * V)) + 31) & ~31; };
  const int t4 = threads_for(N, 4), t8 = threads_for(N, 8), t16 = threads_for(N, 16);
  if (t4 <= 512) {
    // f16 rows beyond 12288: packed, three CTAs an SM instead of two (8192 x 16384: 88 against 99 us; 8192 x 10000: 61 against 55)
    if (F16 && N > 12288) row_chain_cta_kernel<KIND, F16, 4, RAGGED, F16><<<g, t4, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    else row_chain_cta_kernel<KIND, F16, 4, RAGGED, false><<<g, t4, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    return cudaGetLastError();
  }
  if (t8 <= 512) {
    row_chain_cta_kernel<KIND, F16, 8, RAGGED, F16><<<g, t8, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    return cudaGetLastError();
  }
  if (t16 <= 512) {
    // f32 up to 32768, f16 up to 65536 elements.  Of the f16 forms (4096 x 40000): softmax 137 us with sixteen vectors a thread in the
    // aligned kernel below, 146 in the general one, 156 in a cluster; variance 130 us with eight vectors and up to 1024 threads, 146, 202
    if constexpr (!F16) row_chain_cta_kernel<KIND, F16, 16, RAGGED, false><<<g, t16, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    else if constexpr (KIND == 1) row_chain_wide_cta_kernel<KIND, RAGGED><<<g, t8, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    else if constexpr (RAGGED) row_chain_cta_kernel<KIND, F16, 16, true, true><<<g, t16, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
    else row_softmax_cta_packed_kernel<16><<<g, t16, 0, s>>>(X, Out, N, ld_in, ld_out);
    return cudaGetLastError();
  }
  constexpr int kNv = 8, one = 512 * kNv * V;           // vectors a thread and elements a CTA of a cluster
  const int cluster = N <= 4 * one ? 4 : 8;              // (rows of up to two CTAs' worth went above)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g * cluster, 1, 1);
  cfg.blockDim = dim3(threads_for((N + cluster - 1) / cluster, kNv), 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, row_chain_cluster_kernel<KIND, F16, kNv, F16>, X, Out, N, ld_in, ld_out, c1, c2);
}

template <int KIND, bool F16>
cudaError_t launch_typed(const void *X, void *Out, int64_t rows, int N, int64_t ld_in, int64_t ld_out, float c1, float c2, cudaStream_t s) {
  constexpr int V = VecOf<F16>::N;
  constexpr int ES = F16 ? 2 : 4;
  if (rows > 0x7fffffff) return cudaErrorInvalidConfiguration;
  const uintptr_t x = reinterpret_cast<uintptr_t>(X), o = reinterpret_cast<uintptr_t>(Out);
  const bool vec = N % V == 0 && (ld_in * ES) % 16 == 0 && (ld_out * ES) % 16 == 0 && (x & 15) == 0 && (o & 15) == 0;
  // every row's input and output lie equally far from a 16-byte boundary: whole vectors on both sides
  const bool together = x % ES == 0 && (x & 15) == (o & 15) && ((ld_in - ld_out) * ES) % 16 == 0;
  // a CTA holds the row, or a cluster of eight (whose grid is eight times the rows)
  const bool fits = N <= 512 * 16 * V || (N <= 8 * 512 * 8 * V && rows <= 0x7fffffff / 8);
  if (fits && vec) return launch_rows<KIND, F16, false>(X, Out, rows, N, ld_in, ld_out, c1, c2, s);
  if (fits && together) return launch_rows<KIND, F16, true>(X, Out, rows, N, ld_in, ld_out, c1, c2, s);
  row_chain_block_kernel<KIND, F16, F16><<<static_cast<unsigned>(rows), 256, 0, s>>>(X, Out, N, ld_in, ld_out, c1, c2);
  return cudaGetLastError();
}

} // namespace

cudaError_t launch_row_chain(int kind, const void *X, void *Out, int64_t rows, int64_t N, int64_t ld_in, int64_t ld_out, int in_f16,
                             int out_f16, float c1, float c2, cudaStream_t s) {
  if (rows <= 0 || N <= 0) return cudaSuccess;
  if (N > 0x7fffffff) return cudaErrorInvalidValue;
  if ((in_f16 != 0) != (out_f16 != 0)) return cudaErrorInvalidValue;
  const int n = static_cast<int>(N);
  if (kind == 2 && !in_f16) return launch_typed<2, false>(X, Out, rows, n, ld_in, ld_out, c1, c2, s);
  if (kind == 0) return in_f16 ? launch_typed<0, true>(X, Out, rows, n, ld_in, ld_out, c1, c2, s) : launch_typed<0, false>(X, Out, rows, n, ld_in, ld_out, c1, c2, s);
  if (kind == 1) return in_f16 ? launch_typed<1, true>(X, Out, rows, n, ld_in, ld_out, c1, c2, s) : launch_typed<1, false>(X, Out, rows, n, ld_in, ld_out, c1, c2, s);
  return cudaErrorInvalidValue;
}

} // namespace wtc
