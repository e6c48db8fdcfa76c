// RMSNorm / LayerNorm forward + backward with the residual add fused in (sm_100a, HBM-bound).
//
//   forward :  h = x (+ res);  y = norm(h) * w (+ b);   writes y, (h if res given), per-row stats
//   backward:  dx = dnorm(dy) (+ dres);  dw/db partials per CTA, reduced by a second kernel
//
// One CTA handles rows in a grid-stride loop with the row held in registers (H <= 8192), 16-byte
// vector loads, fp32 math.  Replaces apex FusedRMSNorm/FusedLayerNorm reached through
// cornstarch/shardformer/policies/llama.py:252-275 and the eager HF norms.
#include "host.h"
#include "ptx.cuh"

namespace csb {

constexpr int NORM_MAX_H = 8192;  // the backward's largest block: 512 threads with two 16-byte vectors each (norm_bwd_shape)

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the threads that share a row: a warp (ONE_WARP) or the whole block.  One barrier per sum: the warp sums of
// consecutive calls go to alternating halves of `sh`, and whoever writes a half again has passed the barrier of the call in
// between, which every reader of that half's old contents reached after reading.
template <bool ONE_WARP>
__device__ __forceinline__ float row_sum(float v, float* sh, uint32_t& n_calls) {
  v = warp_sum(v);
  if constexpr (ONE_WARP) return v;
  float* buf = sh + (n_calls++ & 1) * 32;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) buf[w] = v;
  __syncthreads();
  return warp_sum(l < (int)(blockDim.x >> 5) ? buf[l] : 0.f);
}

// Two such sums with the barrier of one; `sh` holds 128 floats on an 8-byte boundary.
template <bool ONE_WARP>
__device__ __forceinline__ void row_sum2(float& a, float& b, float* sh, uint32_t& n_calls) {
  a = warp_sum(a);
  b = warp_sum(b);
  if constexpr (ONE_WARP) return;
  float* buf = sh + (n_calls++ & 1) * 64;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, n = blockDim.x >> 5;
  if (l == 0) *reinterpret_cast<float2*>(buf + 2 * w) = make_float2(a, b);
  __syncthreads();
  const float2 v = l < n ? *reinterpret_cast<const float2*>(buf + 2 * l) : make_float2(0.f, 0.f);
  a = warp_sum(v.x);
  b = warp_sum(v.y);
}

// Eight bf16 values as four packed pairs of fp32: half the issue slots of an element-wise loop.
struct Pair4 {
  uint64_t p[4];
};
__device__ __forceinline__ Pair4 unpack_pairs(const uint4& u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  Pair4 r;
#pragma unroll
  for (int i = 0; i < 4; ++i) r.p[i] = pack_u32x2(w[i] << 16, w[i] & 0xffff0000u);
  return r;
}

struct Vec8 {
  float f[8];
};
__device__ __forceinline__ Vec8 load8(const __nv_bfloat16* p) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
  Vec8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    v.f[2 * i] = t.x;
    v.f[2 * i + 1] = t.y;
  }
  return v;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const Vec8& v) {
  uint4 u;
  u.x = pack_bf16x2(v.f[0], v.f[1]);
  u.y = pack_bf16x2(v.f[2], v.f[3]);
  u.z = pack_bf16x2(v.f[4], v.f[5]);
  u.w = pack_bf16x2(v.f[6], v.f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

__device__ __forceinline__ Vec8 unpack8(const uint4& u) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
  Vec8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    v.f[2 * i] = t.x;
    v.f[2 * i + 1] = t.y;
  }
  return v;
}

// Where the forward kernel has the weight (and bias) of its columns while it walks the rows: in registers as fp32, in registers
// as they were loaded (a quarter of them), or read again for every row (they stay in the L1 cache).
enum NormWeights : int { W_FP32, W_RAW, W_RELOAD };

// IS_LN: LayerNorm (mean subtraction + bias) else RMSNorm.  w_offset: Gemma-style (1 + w).
// Every thread holds NV 16-byte vectors of the row (ONE_WARP: H <= 256, a warp per row and eight rows per block; else a
// block per row, rounded up to whole warps).  HBM bounds this kernel; what kept it from that were the dependent phases of a
// row (load, reduce, store), so the next row of the block is loaded before the current one is reduced and several small
// blocks per SM are in different phases.  MIN_BLOCKS and NormWeights are chosen so that they fit the registers without spills
// (norm_fwd_launch).
// 8192 x 4096 with the residual, in a CUDA graph: RMSNorm 50.9 -> 44.9 us (6.0 TB/s), LayerNorm 59 -> 45.6 us (blocks of 256 threads
// with up to four vectors each and nothing in flight across rows before); 262144 x 128: 517 -> 57 us.
template <bool IS_LN, bool ONE_WARP, int NV, NormWeights WM, int MAX_THREADS, int MIN_BLOCKS>
__global__ void __launch_bounds__(MAX_THREADS, MIN_BLOCKS)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out, float* __restrict__ mean_out,
                float* __restrict__ rstd_out, int rows, int H, float eps, float w_offset) {
  __shared__ float sh[64];
  uint32_t n_sums = 0;
  const int lanes = ONE_WARP ? 32 : blockDim.x;               // threads of a row
  const int c = ONE_WARP ? (threadIdx.x & 31) : threadIdx.x;  // this thread's vectors of the row: c, c + lanes, ...
  const int nvec = H / 8;
  const int first = ONE_WARP ? blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  const int step = ONE_WARP ? gridDim.x * (blockDim.x >> 5) : gridDim.x;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  Vec8 w_f[WM == W_FP32 ? NV : 1], b_f[WM == W_FP32 ? NV : 1];
  uint4 w_raw[NV], b_raw[NV];
  auto fetch_weights = [&]() {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      w_raw[i] = b_raw[i] = zero;
      if (c + i * lanes < nvec) {
        w_raw[i] = *reinterpret_cast<const uint4*>(w + (c + i * lanes) * 8);
        if (IS_LN && b) b_raw[i] = *reinterpret_cast<const uint4*>(b + (c + i * lanes) * 8);
      }
    }
  };
  if constexpr (WM != W_RELOAD) fetch_weights();
  if constexpr (WM == W_FP32) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      w_f[i] = unpack8(w_raw[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) w_f[i].f[j] += w_offset;
      b_f[i] = unpack8(b_raw[i]);
    }
  }
  uint4 n_x[NV], n_r[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) n_x[i] = n_r[i] = zero;
  auto fetch = [&](int row) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const size_t at = static_cast<size_t>(row) * H + (c + i * lanes) * 8;
      if (c + i * lanes < nvec) {
        n_x[i] = *reinterpret_cast<const uint4*>(x + at);
        if (res) n_r[i] = *reinterpret_cast<const uint4*>(res + at);
      }
    }
  };
  if (first < rows) fetch(first);
  for (int row = first; row < rows; row += step) {
    const size_t at = static_cast<size_t>(row) * H;
    Vec8 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i] = unpack8(n_x[i]);
      if (res) {
        const Vec8 r = unpack8(n_r[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i].f[j] += r.f[j];
      }
    }
    if (row + step < rows) fetch(row + step);
    if (h_out) {
      // the residual stream is stored in bf16; normalise the rounded value so that the
      // backward (which re-reads h) sees exactly what the forward normalised
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (c + i * lanes < nvec) store8(h_out + at + (c + i * lanes) * 8, v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i].f[j] = __bfloat162float(__float2bfloat16(v[i].f[j]));
      }
    }
    float mean = 0.f, ss = 0.f;
    if (IS_LN) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[i].f[j];
      mean = row_sum<ONE_WARP>(s, sh, n_sums) / H;
      // two-pass variance on the register-resident row
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (c + i * lanes < nvec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float d = v[i].f[j] - mean;
            ss += d * d;
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[i].f[j] * v[i].f[j];
    }
    const float var = row_sum<ONE_WARP>(ss, sh, n_sums) / H;
    const float rstd = rsqrtf(var + eps);
    if (c == 0) {
      if (IS_LN && mean_out) mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (c + i * lanes < nvec) {
        Vec8 o;
        if constexpr (WM == W_FP32) {
#pragma unroll
          for (int j = 0; j < 8; ++j) o.f[j] = (v[i].f[j] - mean) * rstd * w_f[i].f[j] + (IS_LN ? b_f[i].f[j] : 0.f);
        } else {
          const Vec8 wv = WM == W_RAW ? unpack8(w_raw[i]) : load8(w + (c + i * lanes) * 8);
          Vec8 bv = unpack8(zero);
          if (IS_LN) bv = WM == W_RAW ? unpack8(b_raw[i]) : (b ? load8(b + (c + i * lanes) * 8) : bv);
#pragma unroll
          for (int j = 0; j < 8; ++j) o.f[j] = (v[i].f[j] - mean) * rstd * (wv.f[j] + w_offset) + (IS_LN ? bv.f[j] : 0.f);
        }
        store8(y + at + (c + i * lanes) * 8, o);
      }
    }
  }
}

// dx = rstd * (g - xhat * mean(g*xhat) [- mean(g)])  with g = dy * w;  dw += dy * xhat;  db += dy
// NV 16-byte vectors per thread, with the next row's inputs and statistics in flight while the current row is reduced.
// The arithmetic of a row, not HBM, took the time (three unpackings and a conversion of the weight per element and pass, 19
// instructions; LayerNorm's two sums behind two barriers): products and sums go in packed pairs of fp32 now, dy * w and xhat stay in
// registers between the passes (6 instructions), and one barrier serves both sums.  NV and MIN_BLOCKS: see norm_bwd_shape.
// With the sums below and the residual's gradient, inputs from HBM, before -> now: 8192 x 4096 RMSNorm 56.5 -> 53.1 us (5.0 TB/s),
// LayerNorm 77 -> 60.4; 16384 x 1152 LayerNorm 48.6 -> 38.2; 16384 x 5120 RMSNorm 162 -> 118; 1531 x 4096 17.6 -> 14.9; 262144 x
// 128 LayerNorm 108 -> 83.  (Rows in shared memory by bulk copies, up to eight ahead: 0.81 at 8192 elements, but 1.02 to 1.14 up
// to 4096, and 1.2 to 1.6 for the forward kernel.)
template <bool IS_LN, bool ONE_WARP, int NV, int MAX_THREADS, int MIN_BLOCKS>
__global__ void __launch_bounds__(MAX_THREADS, MIN_BLOCKS)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean_in,
                const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_partial, float* __restrict__ db_partial,
                int rows, int H, float w_offset) {
  __shared__ __align__(16) float sh[128];
  uint32_t n_sums = 0;
  const int lanes = ONE_WARP ? 32 : blockDim.x;
  const int c = ONE_WARP ? (threadIdx.x & 31) : threadIdx.x;  // this thread's vectors of the row: c, c + lanes, ...
  const int nvec = H / 8;
  const int first = ONE_WARP ? blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  const int step = ONE_WARP ? gridDim.x * (blockDim.x >> 5) : gridDim.x;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  Pair4 dw_acc[NV], db_acc[IS_LN ? NV : 1], w2[NV];
  uint4 n_dy[NV], n_h[NV], n_dr[NV], w_raw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    n_dy[i] = n_h[i] = n_dr[i] = zero;
    w_raw[i] = c + i * lanes < nvec ? *reinterpret_cast<const uint4*>(w + (c + i * lanes) * 8) : zero;
  }
  float n_mean = 0.f, n_rstd = 0.f;
  auto fetch = [&](int row) {
    n_rstd = rstd_in[row];
    if (IS_LN) n_mean = mean_in[row];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const size_t at = static_cast<size_t>(row) * H + (c + i * lanes) * 8;
      if (c + i * lanes < nvec) {
        n_dy[i] = __ldcs(reinterpret_cast<const uint4*>(dy + at));
        n_h[i] = __ldcs(reinterpret_cast<const uint4*>(h + at));
        if (dres) n_dr[i] = __ldcs(reinterpret_cast<const uint4*>(dres + at));
      }
    }
  };
  if (first < rows) fetch(first);
#pragma unroll
  for (int i = 0; i < NV; ++i) {  // (not before the first row is on its way: few rows are bound by these latencies)
    w2[i] = unpack_pairs(w_raw[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w2[i].p[j] = add_f32x2(w2[i].p[j], pack_f32x2(w_offset, w_offset));
      dw_acc[i].p[j] = 0ull;
      if (IS_LN) db_acc[i].p[j] = 0ull;
    }
  }
  for (int row = first; row < rows; row += step) {
    const float rstd = n_rstd;
    const uint64_t rstd2 = pack_f32x2(rstd, rstd), neg_mean2 = pack_f32x2(-n_mean, -n_mean);
    uint4 c_dr[NV];
    Pair4 g[NV], xh[NV];
    uint64_t s1 = 0ull, s2 = 0ull;
#pragma unroll
    for (int i = 0; i < NV; ++i) {  // vectors beyond the row are zeros: dy = 0, nothing is added
      const Pair4 d = unpack_pairs(n_dy[i]), hv = unpack_pairs(n_h[i]);
      c_dr[i] = n_dr[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        xh[i].p[j] = mul_f32x2(IS_LN ? add_f32x2(hv.p[j], neg_mean2) : hv.p[j], rstd2);
        g[i].p[j] = mul_f32x2(d.p[j], w2[i].p[j]);
        s1 = fma_f32x2(g[i].p[j], xh[i].p[j], s1);
        dw_acc[i].p[j] = fma_f32x2(d.p[j], xh[i].p[j], dw_acc[i].p[j]);
        if (IS_LN) {
          s2 = add_f32x2(s2, g[i].p[j]);
          db_acc[i].p[j] = add_f32x2(db_acc[i].p[j], d.p[j]);
        }
      }
    }
    if (row + step < rows) fetch(row + step);
    float s1a, s1b, m1, m2 = 0.f;
    unpack_f32x2(s1, s1a, s1b);
    m1 = s1a + s1b;
    if (IS_LN) {
      float s2a, s2b;
      unpack_f32x2(s2, s2a, s2b);
      m2 = s2a + s2b;
      row_sum2<ONE_WARP>(m1, m2, sh, n_sums);
      m2 /= H;
    } else {
      m1 = row_sum<ONE_WARP>(m1, sh, n_sums);
    }
    m1 /= H;
    const uint64_t neg_m1 = pack_f32x2(-m1, -m1), neg_m2 = pack_f32x2(-m2, -m2);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (c + i * lanes < nvec) {
        const Pair4 r = unpack_pairs(c_dr[i]);  // zeros without a second gradient
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint64_t t = fma_f32x2(xh[i].p[j], neg_m1, g[i].p[j]);
          if (IS_LN) t = add_f32x2(t, neg_m2);
          float lo, hi;
          unpack_f32x2(fma_f32x2(t, rstd2, r.p[j]), lo, hi);
          o[j] = pack_bf16x2(lo, hi);
        }
        *reinterpret_cast<uint4*>(dx + static_cast<size_t>(row) * H + (c + i * lanes) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
  if constexpr (ONE_WARP) {
    // the warps of a block add up their sums: one partial row per block
    __shared__ __align__(16) float part[8][2][256];  // written in pairs
    const int wi = threadIdx.x >> 5;
    if (c < nvec) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        *reinterpret_cast<uint64_t*>(&part[wi][0][c * 8 + 2 * j]) = dw_acc[0].p[j];
        if (IS_LN) *reinterpret_cast<uint64_t*>(&part[wi][1][c * 8 + 2 * j]) = db_acc[0].p[j];
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
      float sw = 0.f, sb = 0.f;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
        sw += part[k][0][i];
        if (IS_LN) sb += part[k][1][i];
      }
      dw_partial[static_cast<size_t>(blockIdx.x) * H + i] = sw;
      if (IS_LN && db_partial) db_partial[static_cast<size_t>(blockIdx.x) * H + i] = sb;
    }
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (c + i * lanes < nvec) {
        const size_t at = static_cast<size_t>(blockIdx.x) * H + (c + i * lanes) * 8;
        ulonglong2* pw = reinterpret_cast<ulonglong2*>(dw_partial + at);
        pw[0] = make_ulonglong2(dw_acc[i].p[0], dw_acc[i].p[1]);
        pw[1] = make_ulonglong2(dw_acc[i].p[2], dw_acc[i].p[3]);
        if constexpr (IS_LN) {
          if (db_partial) {
            ulonglong2* pb = reinterpret_cast<ulonglong2*>(db_partial + at);
            pb[0] = make_ulonglong2(db_acc[i].p[0], db_acc[i].p[1]);
            pb[1] = make_ulonglong2(db_acc[i].p[2], db_acc[i].p[3]);
          }
        }
      }
    }
  }
}

// out[c] (+)= sum_r partial[r][c]; out is fp32 (main-grad accumulation) or bf16.  blockIdx.y = 1: the second pair of arrays.
// One CTA = 32 columns x 32 row groups: every warp reads 128 contiguous bytes of a row, the groups are summed in shared
// memory.  The loads of a thread are what takes the time (592 rows of partial sums: 74 in a row with 8 groups, 5.9 us).
struct PartialSums {
  const float* partial[2];
  void* out[2];
};
constexpr int REDUCE_GROUPS = 32;  // 8 where there are no more partial rows than that gives work to (reduce_threads)
__global__ void __launch_bounds__(32 * REDUCE_GROUPS) reduce_partials_kernel(const PartialSums p, int nparts, int H, int out_fp32,
                                                                             int accumulate) {
  __shared__ float sh[REDUCE_GROUPS][33];
  const float* __restrict__ partial = blockIdx.y == 0 ? p.partial[0] : p.partial[1];
  void* __restrict__ out = blockIdx.y == 0 ? p.out[0] : p.out[1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, groups = blockDim.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int r = ty; r < nparts; r += groups) s += partial[static_cast<size_t>(r) * H + c];
  }
  sh[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < H) {
#pragma unroll 8
    for (int k = 1; k < groups; ++k) s += sh[k][tx];
    if (out_fp32) {
      float* o = reinterpret_cast<float*>(out);
      o[c] = accumulate ? o[c] + s : s;
    } else {
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
      o[c] = __float2bfloat16(accumulate ? __bfloat162float(o[c]) + s : s);
    }
  }
}

// Column sum of a bf16 matrix [rows][H] (bias gradients): partial sums per row slice, then reduce_partials.
// A block owns 256 columns (a warp reads 512 contiguous bytes of a row) and one slice of the rows, which its eight warps
// share; columns x slices fill the GPU.  (One block for all columns walked its few rows once per 2048 columns with a single
// load in flight per thread.)
constexpr int COLSUM_COLS = 256;
__global__ void __launch_bounds__(256) colsum_partial_kernel(const __nv_bfloat16* __restrict__ x,
                                                            float* __restrict__ partial, int rows, int H) {
  __shared__ float part[8][COLSUM_COLS];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int col = blockIdx.x * COLSUM_COLS + lane * 8;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col < H) {
#pragma unroll 4
    for (int r = blockIdx.y * 8 + wi; r < rows; r += gridDim.y * 8) {
      const Vec8 v = load8(x + static_cast<size_t>(r) * H + col);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v.f[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) part[wi][lane * 8 + j] = acc[j];
  __syncthreads();
  const int c = blockIdx.x * COLSUM_COLS + threadIdx.x;
  if (c < H) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += part[k][threadIdx.x];
    partial[static_cast<size_t>(blockIdx.y) * H + c] = s;
  }
}

}  // namespace csb

using namespace csb;

static int reduce_threads(int nparts) { return 32 * (nparts <= 32 ? 8 : REDUCE_GROUPS); }

// Upper bound of the partial rows of a launch (what csb_norm_bwd_parts promises the caller).
static int norm_grid(int rows) {
  int g = sm_count() * 4;
  return rows < g ? rows : g;
}
// Threads, vectors per thread and blocks of a backward launch for rows of H elements: up to 256 elements a warp per row and eight
// rows per block, above that one block per row.
// - Two vectors per thread above 2048 elements, two blocks of up to 320 threads per SM: with one vector, blocks of 512 threads at 64
//   registers take 1.03 to 1.2 times as long (1000 x 4096 RMSNorm with residual 14.8 / 12.7 us, 8192 rows 55.1 / 53.1, LayerNorm
//   65.0 / 60.4), at 640 to 1024 threads only one fits (16384 x 5120: 157 / 118).  Three blocks at 80 registers spill (8192 x 4096:
//   61 us).  One vector with no more rows than SMs, where a row's latency counts (77 x 4096 LayerNorm: 7.5 / 8.0 us).
// - Four blocks up to 1280 elements at up to 102 registers, three of those with a warp per row: at 64 LayerNorm spills (4096 x 768:
//   15.3 / 13.3 us; 262144 x 128: 84 / 83 but 700 x 256 RMSNorm 4.9 / 5.0).
struct NormBwdShape {
  int threads, nv, blocks, grid;  // blocks per SM
};
static NormBwdShape norm_bwd_shape(int rows, int H) {
  NormBwdShape r;
  const int nvec = H / 8;
  r.nv = nvec > 512 || (nvec > 256 && rows > sm_count()) ? 2 : 1;
  r.threads = nvec <= 32 ? 256 : ((nvec + r.nv - 1) / r.nv + 31) / 32 * 32;
  const long units = nvec <= 32 ? (rows + 7) / 8 : rows;
  r.blocks = r.threads > 320 && r.nv == 2 ? 1 : (r.nv == 2 || r.threads > 256 ? 2 : 4);
  if (nvec <= 32) r.blocks = 3;
  const long g = (long)sm_count() * r.blocks;
  r.grid = (int)(units < g ? units : g);
  return r;
}

// Number of fp32 rows the caller must provide in the dw/db partial buffers for a given row count.
CSB_API int csb_norm_bwd_parts(int rows) { return norm_grid(rows); }

// Vectors per thread, threads per block and blocks per SM of the forward kernel, four blocks per SM at most in the grid.  Times are
// of a CUDA graph, both sides of a line.
// - Two vectors per thread above 2048 elements: blocks of half the threads, so that two to four fit the registers of an SM (one
//   block of 640 threads does).  One vector against two, RMSNorm with residual: 4096 x 2560 14.7 / 11.2 us, 1000 x 4096 6.5 / 5.7,
//   1000 x 5120 8.6 / 6.7, 16384 x 5120 129 / 111, 16384 x 6144 144 / 129, 8192 x 8192 89 / 89; LayerNorm with residual: 4096 x
//   2560 18.1 / 15.2, 8192 x 4096 47.3 / 45.6, 16384 x 5120 136 / 107.
// - One vector with no more rows than SMs, where a row's latency counts (77 x 4096 LayerNorm: 2.86 / 3.07 us), and for the
//   RMSNorm with residual of many rows of 3080 to 4096 elements (8192 x 4096: 44.9 / 46.2 us, 16384 rows: 86.5 / 91.7; but 4096
//   rows: 24.1 / 20.5).
// - The weights stay in registers as loaded where that costs no spills; LayerNorm reads weight and bias again for every row in
//   the blocks of 256 and 512 threads (8192 x 4096: 45.6 us, 50.6 with spills), and takes two blocks of up to 320 threads instead
//   of three (16384 x 5120: 107 us, 136 with three).
template <bool LN>
static void norm_fwd_launch(const __nv_bfloat16* x, const __nv_bfloat16* r, const __nv_bfloat16* w, const __nv_bfloat16* b,
                            __nv_bfloat16* y, __nv_bfloat16* h, float* mean, float* rstd, int rows, int H, float eps, float w_offset,
                            cudaStream_t s) {
  const bool stream = !LN && r != nullptr && H > 3072 && H <= 4096 && rows >= 8192;
  const bool wide = H > 2048 && rows > sm_count() && !stream;
  const int nvec = H / 8, per_thread = wide ? 2 : 1;
  const int threads = H <= 256 ? 256 : ((nvec + per_thread - 1) / per_thread + 31) / 32 * 32;
  const long units = H <= 256 ? (rows + 7) / 8 : rows;
  const int grid = (int)(units < 4L * sm_count() ? units : 4L * sm_count());
#define CSB_NORM_FWD(OW, NV, WM, MT, MB) \
  norm_fwd_kernel<LN, OW, NV, WM, MT, MB><<<grid, threads, 0, s>>>(x, r, w, b, y, h, mean, rstd, rows, H, eps, w_offset)
  if (H <= 256) CSB_NORM_FWD(true, 1, W_FP32, 256, 4);
  else if (!wide) CSB_NORM_FWD(false, 1, W_FP32, 1024, 1);
  else if (threads <= 256) CSB_NORM_FWD(false, 2, LN ? W_RELOAD : W_RAW, 256, 4);
  else if (threads <= 320) CSB_NORM_FWD(false, 2, W_RAW, 320, LN ? 2 : 3);
  else if (threads <= 384) CSB_NORM_FWD(false, 2, W_RAW, 384, 2);
  else CSB_NORM_FWD(false, 2, LN ? W_RELOAD : W_RAW, 512, 2);
#undef CSB_NORM_FWD
}

CSB_API int csb_norm_fwd(int is_layernorm, const void* x, const void* res, const void* w, const void* b, void* y,
                         void* h_out, float* mean, float* rstd, int rows, int H, float eps, float w_offset,
                         void* stream) {
  if (H % 8 != 0 || H > NORM_MAX_H || rows <= 0) return CSB_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto R = reinterpret_cast<const __nv_bfloat16*>(res);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto B = reinterpret_cast<const __nv_bfloat16*>(b);
  auto Y = reinterpret_cast<__nv_bfloat16*>(y);
  auto Ho = reinterpret_cast<__nv_bfloat16*>(h_out);
  if (is_layernorm) norm_fwd_launch<true>(X, R, W, B, Y, Ho, mean, rstd, rows, H, eps, w_offset, s);
  else norm_fwd_launch<false>(X, R, W, B, Y, Ho, mean, rstd, rows, H, eps, w_offset, s);
  return launch_result();
}

// dw_out/db_out: final gradient tensors (fp32 or bf16 by *_fp32 flag), accumulated into when accumulate=1.
CSB_API int csb_norm_bwd(int is_layernorm, const void* dy, const void* h, const void* w, const float* mean,
                         const float* rstd, const void* dres, void* dx, float* dw_partial, float* db_partial,
                         void* dw_out, void* db_out, int grads_fp32, int accumulate, int rows, int H,
                         float w_offset, void* stream) {
  if (H % 8 != 0 || H > NORM_MAX_H || rows <= 0) return CSB_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const NormBwdShape shape = norm_bwd_shape(rows, H);
  const int grid = shape.grid;
  auto DY = reinterpret_cast<const __nv_bfloat16*>(dy);
  auto Hh = reinterpret_cast<const __nv_bfloat16*>(h);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto DR = reinterpret_cast<const __nv_bfloat16*>(dres);
  auto DX = reinterpret_cast<__nv_bfloat16*>(dx);
  constexpr int LARGEST_NV = 2, LARGEST_THREADS = 512;
  static_assert(LARGEST_NV * LARGEST_THREADS * 8 == NORM_MAX_H, "every admitted row has its threads");
#define CSB_NORM_BWD(LN, OW, NV, MT, MB)                                                                                     \
  norm_bwd_kernel<LN, OW, NV, MT, MB><<<grid, shape.threads, 0, s>>>(DY, Hh, W, mean, rstd, DR, DX, dw_partial, db_partial, rows, H, w_offset)
#define CSB_NORM_BWD_LN(OW, NV, MT, MB) \
  if (is_layernorm) CSB_NORM_BWD(true, OW, NV, MT, MB); else CSB_NORM_BWD(false, OW, NV, MT, MB)
  if (H <= 256) { CSB_NORM_BWD_LN(true, 1, 256, 3); }
  else if (shape.nv == 1 && shape.threads <= 160) { CSB_NORM_BWD_LN(false, 1, 160, 4); }
  else if (shape.nv == 1) { CSB_NORM_BWD_LN(false, 1, 512, 2); }
  else if (shape.threads <= 256) { CSB_NORM_BWD_LN(false, 2, 256, 2); }
  else if (shape.threads <= 320) { CSB_NORM_BWD_LN(false, 2, 320, 2); }
  else { CSB_NORM_BWD_LN(false, LARGEST_NV, LARGEST_THREADS, 1); }
#undef CSB_NORM_BWD_LN
#undef CSB_NORM_BWD
  int r = launch_result();
  if (r) return r;
  PartialSums ps = {};
  int n = 0;
  if (dw_out) {
    ps.partial[n] = dw_partial;
    ps.out[n++] = dw_out;
  }
  if (is_layernorm && db_out && db_partial) {
    ps.partial[n] = db_partial;
    ps.out[n++] = db_out;
  }
  if (n > 0) reduce_partials_kernel<<<dim3((H + 31) / 32, n), reduce_threads(grid), 0, s>>>(ps, grid, H, grads_fp32, accumulate);
  return launch_result();
}

// Bias gradient: out[H] (+)= column sums of dy[rows][H].  `partial` needs csb_colsum_parts() * H floats.
CSB_API int csb_colsum_parts(int rows) {
  int g = sm_count() * 2;
  return rows < g ? rows : g;
}
CSB_API int csb_colsum(const void* x, float* partial, void* out, int out_fp32, int accumulate, int rows, int H,
                       void* stream) {
  if (H % 8 != 0 || H <= 0 || rows <= 0) return CSB_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return CSB_ERR_BAD_ARG;  // 16-byte loads
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // row slices: enough blocks to fill the GPU four times, at least 8 rows (one per warp) in each, never more than promised
  const int col_blocks = (H + COLSUM_COLS - 1) / COLSUM_COLS;
  int slices = (sm_count() * 4 + col_blocks - 1) / col_blocks;
  if (slices > (rows + 7) / 8) slices = (rows + 7) / 8;
  if (slices > csb_colsum_parts(rows)) slices = csb_colsum_parts(rows);
  colsum_partial_kernel<<<dim3(col_blocks, slices), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), partial, rows, H);
  if (int e = launch_result()) return e;
  PartialSums ps = {{partial, nullptr}, {out, nullptr}};
  reduce_partials_kernel<<<(H + 31) / 32, reduce_threads(slices), 0, s>>>(ps, slices, H, out_fp32, accumulate);
  return launch_result();
}
