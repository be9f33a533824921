// Bandwidth-bound companions of the tiled kernel: combine per-tile (max, sum)
// pairs into per-row statistics and rescale the stored exp(v - tile max) values
// into probabilities.  All maxima are in the log2 domain (v = scale*log2(e)*s).
#include "wtc_kernels.h"
#include "wtc_ptx.cuh"

namespace wtc {
namespace {

__device__ __forceinline__ float2 lse_combine(float2 a, float2 b) {
  // (max, sum) pairs of disjoint column sets -> pair of their union
  const float m = fmaxf(a.x, b.x);
  if (m == -INFINITY) return make_float2(m, 0.f);
  return make_float2(m, a.y * ex2_approx(a.x - m) + b.y * ex2_approx(b.x - m));
}

__device__ __forceinline__ float2 warp_lse(float2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float2 other = make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    v = lse_combine(v, other);
  }
  return v;
}

// one warp per row
__global__ void row_stats_kernel(const float2 *__restrict__ tile_stats, float2 *__restrict__ row_stats,
                                 int64_t rows, int num_nb) {
  grid_dependency_wait();
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float2 v = make_float2(-INFINITY, 0.f);
  for (int t = lane; t < num_nb; t += 32) v = lse_combine(v, tile_stats[row * num_nb + t]);
  v = warp_lse(v);
  if (lane == 0) row_stats[row] = v;
}

// One CTA per row, or -- when there are few rows -- gridDim.y CTAs per row, each taking `chunk`
// columns (a multiple of 256) after working out the row's total for itself.
//
// Pure traffic: the output read and written once more.  Rows go from the last to the first, because
// the tiled kernel in front wrote the last ones last: up to an L2 of them need no read from memory;
// and what is written is not kept from the rows still to come.  Whole chain, f16: 8192 x 8192 x 256
// 110 us from the first row on, 97 so; 4096 x 12000 x 64 79 and 67.  (Ordinary stores in place of the
// streaming ones are slower or the same from 4 MB of output on: 8192 x 8192 x 256 100.7 and 99.5 us,
// 2048 x 4096 x 128 19.6 and 19.4, f32 2048 x 4096 x 128 23.7 and 23.2.)
//
// VECS vectors a thread are in flight: with many CTAs one, since 32 registers let eight of them share an
// SM (four take 40: six), four where all are resident at once anyway.  One and four, f16: 512 x 8192 x
// 256 14.5 and 13.8 us, 700 x 2568 x 128 12.6 and 11.8, 1000 x 3000 x 128 12.9 and 13.2, 4096 x 4096 x
// 128 30.3 and 31.8, 16384 x 4096 x 64 100 and 106; f32 600 x 30000 x 128 47.6 and 42.5, 4096 x 4096 x
// 128 37.0 and 38.4.
template <int VECS>
__global__ void __launch_bounds__(256)
rescale_rows_kernel(void *__restrict__ out_v, int out_f32, int N, int64_t ld_out, int BN, int num_nb,
                    const float2 *__restrict__ tile_stats, const float2 *__restrict__ global_stats,
                    int num_parts, int64_t rows, int chunk) {
  extern __shared__ float factor[];          // [num_nb]
  __shared__ float2 warp_part[8];
  __shared__ float2 row_total;
  grid_dependency_wait();                    // launched behind the tiled kernel with programmatic serialisation
  const int64_t row = gridDim.x - 1 - blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  float2 v = make_float2(-INFINITY, 0.f);
  if (global_stats) {
    for (int t = threadIdx.x; t < num_parts; t += blockDim.x) v = lse_combine(v, global_stats[static_cast<int64_t>(t) * rows + row]);
  } else {
    for (int t = threadIdx.x; t < num_nb; t += blockDim.x) v = lse_combine(v, tile_stats[row * num_nb + t]);
  }
  v = warp_lse(v);
  if (lane == 0) warp_part[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float2 t = lane < (blockDim.x >> 5) ? warp_part[lane] : make_float2(-INFINITY, 0.f);
    t = warp_lse(t);
    if (lane == 0) row_total = t;
  }
  __syncthreads();
  const float gm = row_total.x;
  const float inv = 1.0f / row_total.y;
  for (int t = threadIdx.x; t < num_nb; t += blockDim.x)
    factor[t] = ex2_approx(tile_stats[row * num_nb + t].x - gm) * inv;
  __syncthreads();
  const int c0 = blockIdx.y * chunk;                       // my columns: [c0, c1)
  const int c1 = min(N, c0 + chunk);

  if (out_f32) {
    float *frow = static_cast<float *>(out_v) + row * ld_out;
    if ((N % 4 == 0) && (ld_out % 4 == 0) && ((reinterpret_cast<uintptr_t>(out_v) & 15) == 0) && (BN % 4 == 0)) {
      float4 *o4 = reinterpret_cast<float4 *>(frow);
      for (int j0 = c0 / 4 + threadIdx.x; j0 < c1 / 4; j0 += VECS * blockDim.x) {
        float4 x[VECS];
#pragma unroll
        for (int u = 0; u < VECS; ++u) {
          const int j = j0 + u * blockDim.x;
          if (j < c1 / 4) x[u] = o4[j];
        }
#pragma unroll
        for (int u = 0; u < VECS; ++u) {
          const int j = j0 + u * blockDim.x;
          if (j < c1 / 4) {
            const float fct = factor[(j * 4) / BN];
            __stcs(&o4[j], make_float4(x[u].x * fct, x[u].y * fct, x[u].z * fct, x[u].w * fct));
          }
        }
      }
    } else {
      for (int j = c0 + threadIdx.x; j < c1; j += blockDim.x) frow[j] *= factor[j / BN];
    }
    return;
  }
  __half *out = static_cast<__half *>(out_v);
  __half *orow = out + row * ld_out;
  const bool vec_ok = (N % 8 == 0) && (ld_out % 8 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) && (BN % 8 == 0);
  if (vec_ok) {
    uint4 *o4 = reinterpret_cast<uint4 *>(orow);
    for (int j0 = c0 / 8 + threadIdx.x; j0 < c1 / 8; j0 += VECS * blockDim.x) {
      uint4 x[VECS];
#pragma unroll
      for (int u = 0; u < VECS; ++u) {
        const int j = j0 + u * blockDim.x;
        if (j < c1 / 8) x[u] = o4[j];
      }
#pragma unroll
      for (int u = 0; u < VECS; ++u) {
        const int j = j0 + u * blockDim.x;
        if (j < c1 / 8) {
          const float f = factor[(j * 8) / BN];
          __half2 *h = reinterpret_cast<__half2 *>(&x[u]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 t = __half22float2(h[i]);
            h[i] = __floats2half2_rn(t.x * f, t.y * f);
          }
          __stcs(&o4[j], x[u]);
        }
      }
    }
  } else {
    // rows that start or end anywhere: element by element up to the first 16-byte boundary and behind
    // the last whole vector; a vector may lie across two tiles
    const int head = min(static_cast<int>((8 - ((reinterpret_cast<uintptr_t>(orow + c0) >> 1) & 7)) & 7), c1 - c0);
    const int v0 = c0 + head, v1 = v0 + ((c1 - v0) & ~7);
    for (int j = v0 + threadIdx.x * 8; j < v1; j += blockDim.x * 8) {
      const int t0 = j / BN, split = (t0 + 1) * BN - j;      // elements from `split` on belong to the next tile
      const float f0 = factor[t0], f1 = split < 8 ? factor[t0 + 1] : f0;
      uint4 x = *reinterpret_cast<uint4 *>(orow + j);
      __half2 *h = reinterpret_cast<__half2 *>(&x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 t = __half22float2(h[i]);
        h[i] = __floats2half2_rn(t.x * (2 * i < split ? f0 : f1), t.y * (2 * i + 1 < split ? f0 : f1));
      }
      *reinterpret_cast<uint4 *>(orow + j) = x;
    }
    const int ends = head + (c1 - v1);
    if (static_cast<int>(threadIdx.x) < ends) {
      const int j = static_cast<int>(threadIdx.x) < head ? c0 + static_cast<int>(threadIdx.x) : v1 + static_cast<int>(threadIdx.x) - head;
      orow[j] = __float2half_rn(__half2float(orow[j]) * factor[j / BN]);
    }
  }
}

} // namespace

cudaError_t launch_row_stats(const float2 *tile_stats, float2 *row_stats_out, int64_t rows, int num_nb,
                             cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  const int warps = 8;
  const unsigned grid = static_cast<unsigned>((rows + warps - 1) / warps);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(warps * 32, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, row_stats_kernel, tile_stats, row_stats_out, rows, num_nb);
}

cudaError_t launch_rescale_rows(void *out, int out_f32, int64_t rows, int N, int64_t ld_out, int BN, int num_nb,
                                const float2 *tile_stats, const float2 *global_stats, int num_parts,
                                cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  // few rows (skinny problems): several CTAs per row so that the pass still fills the chip
  // (16 rows x 32000 columns: one CTA per row takes 12 us, sixteen per row 3 us)
  int splits = 1, chunk = N;
  if (rows < 2 * 148 && N > 4096) {
    const int want = static_cast<int>((2 * 148 + rows - 1) / rows);
    const int by_size = (N + 2047) / 2048;
    splits = want < by_size ? want : by_size;
    chunk = ((N + splits - 1) / splits + 255) / 256 * 256;
    splits = (N + chunk - 1) / chunk;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows), static_cast<unsigned>(splits), 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = num_nb * sizeof(float);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  constexpr int64_t kResident = 148 * 6;       // CTAs of the four-vector form that the chip holds at once
  return cudaLaunchKernelEx(&cfg, rows * splits <= kResident ? rescale_rows_kernel<4> : rescale_rows_kernel<1>, out, out_f32, N, ld_out, BN,
                            num_nb, tile_stats, global_stats, num_parts, rows, chunk);
}

// ---- operand copies -----------------------------------------------------------------------------
// For the chain that truncates its f32 arguments to f16, and for f16 operands whose rows TMA cannot
// read (strides that are no multiple of 16 bytes).
namespace {
struct CopyJob {
  const void *src; __half *dst;
  int64_t ld, batch_stride;
  int64_t rows, cols, per_row, work;     // rows of one batch; work = units of eight destination columns, per_row of them a row
  int vec;                               // whole units can be read with 16-byte loads
};

// I: what units are counted in (32 bits unless there are more than 2^32 of them: its divisions are several times shorter)
template <bool F32, typename I>
__device__ __forceinline__ void copy_unit(const CopyJob &j, I u) {
  const I row = u / static_cast<I>(j.per_row);
  const int64_t c = static_cast<int64_t>(u - row * static_cast<I>(j.per_row)) * 8;
  const I b = row / static_cast<I>(j.rows), r = row - b * static_cast<I>(j.rows);
  const int64_t at = static_cast<int64_t>(b) * j.batch_stride + static_cast<int64_t>(r) * j.ld + c;
  uint32_t w[4];
  if (F32) {
    const float *src = static_cast<const float *>(j.src) + at;
    float v[8];
    if (j.vec && c + 8 <= j.cols) {
      const float4 lo = *reinterpret_cast<const float4 *>(src), hi = *reinterpret_cast<const float4 *>(src + 4);
      v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
      v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = c + e < j.cols ? src[e] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = pack_f16x2(v[2 * e], v[2 * e + 1]);
  } else {
    const uint16_t *src = static_cast<const uint16_t *>(j.src) + at;
    if (j.vec && c + 8 <= j.cols) {
      const uint4 o = *reinterpret_cast<const uint4 *>(src);
      w[0] = o.x; w[1] = o.y; w[2] = o.z; w[3] = o.w;
    } else {
      uint32_t h[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) h[e] = c + e < j.cols ? src[e] : 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = h[2 * e] | h[2 * e + 1] << 16;
    }
  }
  *reinterpret_cast<uint4 *>(j.dst + static_cast<int64_t>(u) * 8) = make_uint4(w[0], w[1], w[2], w[3]);
}

// One launch copies A and B: one thread per eight destination columns, A's units first, then B's.
// Launched with programmatic stream serialisation: the chain's kernel behind it starts its set-up
// as soon as these CTAs are resident, and waits for them to finish before its first load.
template <bool F32, typename I>
__global__ void __launch_bounds__(256) copy_operands_kernel(const CopyJob a, const CopyJob b) {
  grid_dependency_wait();                    // the operands may be the previous kernel's output
  grid_launch_dependents();
  const int64_t u = blockIdx.x * int64_t{256} + threadIdx.x;
  if (u < a.work) copy_unit<F32, I>(a, static_cast<I>(u));
  else if (u < a.work + b.work) copy_unit<F32, I>(b, static_cast<I>(u - a.work));
}

CopyJob make_job(const OperandCopy &c, bool f32) {
  CopyJob j{};
  if (!c.dst) return j;
  j.src = c.src; j.dst = static_cast<__half *>(c.dst);
  j.ld = c.ld; j.batch_stride = c.batch_stride;
  j.rows = c.rows; j.cols = c.cols; j.per_row = c.ld_dst / 8;
  j.work = c.batch * c.rows * j.per_row;
  const int per16 = f32 ? 4 : 8;
  j.vec = c.ld % per16 == 0 && (c.batch == 1 || c.batch_stride % per16 == 0) && (reinterpret_cast<uintptr_t>(c.src) & 15) == 0;
  return j;
}
} // namespace

cudaError_t launch_copy_operands(const OperandCopy &a, const OperandCopy &b, bool src_f32, cudaStream_t s) {
  const CopyJob ja = make_job(a, src_f32), jb = make_job(b, src_f32);
  const int64_t work = ja.work + jb.work;
  if (work == 0) return cudaSuccess;
  if ((work + 255) / 256 > 0x7fffffff) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((work + 255) / 256), 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool wide = ja.work >= (int64_t{1} << 32) || jb.work >= (int64_t{1} << 32);
  if (src_f32) return wide ? cudaLaunchKernelEx(&cfg, copy_operands_kernel<true, uint64_t>, ja, jb) : cudaLaunchKernelEx(&cfg, copy_operands_kernel<true, uint32_t>, ja, jb);
  return wide ? cudaLaunchKernelEx(&cfg, copy_operands_kernel<false, uint64_t>, ja, jb) : cudaLaunchKernelEx(&cfg, copy_operands_kernel<false, uint32_t>, ja, jb);
}

} // namespace wtc
