// Memory-bound ops of the decoder, each a single pass with 16-byte accesses and fp32 math:
// RMSNorm fwd/bwd, rotary embedding on a fused qkv activation, SwiGLU fwd/bwd, softmax
// cross-entropy that turns logits into their gradient in place, AdamW on flat shards (also
// refreshing the low-precision copy that peers gather), casts and a sum-of-squares reduction.
// The reference runs these as eager PyTorch ops inside Hugging Face modules
// (examples/llm_training/torch_fsdp2.py:164, lm_head.py:7-59) and torch.optim.AdamW (:322).
#include <cuda_bf16.h>

#include "api.h"
#include "launch.cuh"
#include "odc_device.cuh"

namespace odc {
namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  f[0] = lo(u.x); f[1] = hi(u.x); f[2] = lo(u.y); f[3] = hi(u.y);
  f[4] = lo(u.z); f[5] = hi(u.z); f[6] = lo(u.w); f[7] = hi(u.w);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7]));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// block-wide sum, result in every thread; `red` holds 32 floats
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -INFINITY;
  return warp_max(t);
}

// ------------------------------------------------------------------------- RMSNorm ----------
// A row is handled by R warps (R = 1 up to 2048 columns, 2 up to 4096, 4 up to 8192); a lane keeps up to 8
// 16-byte pieces of the row in registers with all loads in flight at once.  With R = 1 the row statistics
// need only warp shuffles and no block-wide barrier sits on the critical path.
constexpr int kNormThreads = 256;
constexpr int kNormWarps = kNormThreads / 32;
constexpr int kNormVec = 8;

// sum over the R warps that share a row (R > 1 only); every thread of the CTA must call it, with another `red` than in
// the call before (one barrier per call keeps two calls on the same slots apart, not two in a row)
template <int R>
__device__ __forceinline__ float row_sum(float v, float* red, int warp, int lane) {
  v = warp_sum(v);
  if constexpr (R == 1) return v;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const int first = warp - warp % R;
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i) t += red[first + i];
  return t;
}

template <int R>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int cols, float eps) {
  __shared__ float red[2][kNormWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = warp % R;                       // which part of the row this warp covers
  constexpr int kRowsPerIter = kNormWarps / R;
  const int nvec = cols / 8;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const int iters = (rows + gridDim.x * kRowsPerIter - 1) / (gridDim.x * kRowsPerIter);
  for (int it = 0; it < iters; ++it) {
    const int row = (it * gridDim.x + blockIdx.x) * kRowsPerIter + warp / R;
    const bool live = row < rows;
    const uint4* xr = reinterpret_cast<const uint4*>(x + size_t(live ? row : 0) * cols);
    uint4 xv[kNormVec];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < kNormVec; ++k) {
      const int v = (sub * kNormVec + k) * 32 + lane;
      if (live && v < nvec) xv[k] = xr[v];
    }
#pragma unroll
    for (int k = 0; k < kNormVec; ++k) {
      const int v = (sub * kNormVec + k) * 32 + lane;
      if (live && v < nvec) {
        float f[8];
        unpack8(xv[k], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
      }
    }
    ss = row_sum<R>(ss, red[it & 1], warp, lane);
    if (!live) continue;
    const float rstd = rsqrtf(ss / cols + eps);
    if (lane == 0 && sub == 0) rstd_out[row] = rstd;
    uint4* yr = reinterpret_cast<uint4*>(y + size_t(row) * cols);
#pragma unroll
    for (int k = 0; k < kNormVec; ++k) {
      const int v = (sub * kNormVec + k) * 32 + lane;
      if (v < nvec) {
        float f[8], g[8];
        unpack8(xv[k], f);
        unpack8(wr[v], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * g[i];
        yr[v] = pack8(f);
      }
    }
  }
}

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x)).  A row is handled by R warps and a lane keeps V 16-byte pieces of
// x and dy in registers (V <= 4, so the kernel fits two CTAs per SM and both keep loads in flight); each lane
// accumulates dw for its own columns over all rows it handles, the warps of a CTA combine through shared memory,
// and the CTA then either adds its sums into dw (kAtomic: dw zeroed before the launch, one launch in total) or
// writes one row of partial sums for a second, fixed-order pass.  Bound by HBM on many rows and by the chain of one row on
// few: everything a row reads (the residual gradient included) is requested at its start, and the warps of a row meet once.
// With the residual gradient read after the row's sum and two barriers: 16321 x 2048 71 us, 765 x 1536 14.2 us; without 51 us
// (5.2 TB/s) and 10.4 us.  The warps' column sums then met in shared memory by atomics; with rows of their own 16321 x 2048
// 62 -> 57 us, 765 x 1536 12.7 -> 8.2, 2000 x 512 7.9 -> 4.6 (profiler, one run).
template <int R, int V, bool kAtomic>
__global__ void __launch_bounds__(kNormThreads, 2)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                   const float* __restrict__ rstd_in, bf16* __restrict__ dx, float* __restrict__ partial,
                   float* __restrict__ dw_out, int rows, int cols, const bf16* __restrict__ dres) {
  extern __shared__ float dw_smem[];  // [kRowsPerIter][cols]
  __shared__ float red[2][kNormWarps];  // alternating, so that a row's sums outlive the next row's first writer
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = warp % R;
  constexpr int kRowsPerIter = kNormWarps / R;
  const int nvec = cols / 8;
  float dw[V][8];
#pragma unroll
  for (int k = 0; k < V; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) dw[k][i] = 0.f;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const int iters = (rows + gridDim.x * kRowsPerIter - 1) / (gridDim.x * kRowsPerIter);
  for (int it = 0; it < iters; ++it) {
    const int row = (it * gridDim.x + blockIdx.x) * kRowsPerIter + warp / R;
    const bool live = row < rows;
    const uint4* xr = reinterpret_cast<const uint4*>(x + size_t(live ? row : 0) * cols);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + size_t(live ? row : 0) * cols);
    const float rstd = live ? rstd_in[row] : 0.f;
    const uint4* rr = reinterpret_cast<const uint4*>(dres + size_t(live ? row : 0) * cols);
    uint4 xv[V], gv[V], rv[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = (sub * V + k) * 32 + lane;
      if (live && v < nvec) {
        xv[k] = xr[v];
        gv[k] = gr[v];
        if (dres != nullptr) rv[k] = rr[v];
      }
    }
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = (sub * V + k) * 32 + lane;
      if (live && v < nvec) {
        float xf[8], gf[8], wf[8];
        unpack8(xv[k], xf);
        unpack8(gv[k], gf);
        unpack8(wr[v], wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          dot += gf[i] * wf[i] * xf[i];
          dw[k][i] += gf[i] * xf[i] * rstd;
        }
      }
    }
    dot = row_sum<R>(dot, red[it & 1], warp, lane);
    if (!live) continue;
    const float c = dot * rstd * rstd / cols;
    uint4* dr = reinterpret_cast<uint4*>(dx + size_t(row) * cols);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = (sub * V + k) * 32 + lane;
      if (v < nvec) {
        float xf[8], gf[8], wf[8], o[8];
        unpack8(xv[k], xf);
        unpack8(gv[k], gf);
        unpack8(wr[v], wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rstd * (gf[i] * wf[i] - xf[i] * c);
        if (dres != nullptr) {  // gradient that reached x through the residual path: one pass instead of a separate add
          float rf[8];
          unpack8(rv[k], rf);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += rf[i];
        }
        dr[v] = pack8(o);
      }
    }
  }
  // every group of warps writes its sums to a row of its own: floating-point atomics in shared memory are loops of
  // compare-and-swap, which the eight warps of a short kernel spent on one another
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = (sub * V + k) * 32 + lane;
    if (v < nvec) {
      float4* to = reinterpret_cast<float4*>(dw_smem + (warp / R) * cols + v * 8);
      to[0] = make_float4(dw[k][0], dw[k][1], dw[k][2], dw[k][3]);
      to[1] = make_float4(dw[k][4], dw[k][5], dw[k][6], dw[k][7]);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    float sum = dw_smem[c];
#pragma unroll
    for (int g = 1; g < kRowsPerIter; ++g) sum += dw_smem[g * cols + c];
    if constexpr (kAtomic) atomicAdd(dw_out + c, sum);
    else partial[size_t(blockIdx.x) * cols + c] = sum;
  }
}

__global__ void colsum_kernel(const float* __restrict__ partial, float* __restrict__ out, int parts, int cols) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  float s = 0.f;
  for (int p = 0; p < parts; ++p) s += partial[size_t(p) * cols + c];
  out[c] = s;
}

// Column sums of a bf16 matrix (bias gradients): a CTA owns 64 columns and walks all rows, so there is one launch, no
// zeroed scratch and a fixed order of additions.  Bound by the load latency of the walk: 1024 threads with four 16-byte
// loads each keep 64 KiB in flight per CTA.
constexpr int kColSumThreads = 1024;
__global__ void __launch_bounds__(kColSumThreads)
column_sum_kernel(const bf16* __restrict__ x, bf16* __restrict__ out, float* __restrict__ sink, long long rows, int cols) {
  __shared__ float part[kColSumThreads / 32][64];
  const int vec = threadIdx.x & 7, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 64 + vec * 8;
  constexpr int kRows = kColSumThreads / 8;
  float s[8] = {};
  if (col < cols) {
    const bf16* p = x + col;
#pragma unroll 4
    for (long long r = threadIdx.x >> 3; r < rows; r += kRows) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(p + r * cols), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] += f[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s[i] += __shfl_xor_sync(0xffffffffu, s[i], 8);
    s[i] += __shfl_xor_sync(0xffffffffu, s[i], 16);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) part[warp][vec * 8 + i] = s[i];
  }
  __syncthreads();
  const int c = blockIdx.x * 64 + threadIdx.x;
  if (threadIdx.x < 64 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kColSumThreads / 32; ++w) t += part[w][threadIdx.x];
    if (sink != nullptr) sink[c] += t; else out[c] = __float2bfloat16(t);
  }
}

// ------------------------------------------------------------------------- RoPE -------------
// one CTA per token; cos/sin of the head_dim/2 angles computed once and reused by all heads
__global__ void __launch_bounds__(128)
rope_qkv_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, const long long* __restrict__ pos, int n_q,
                int n_kv, int head_dim, float log2_theta, float sign) {
  extern __shared__ float cs[];  // [head_dim/2] cos, [head_dim/2] sin
  const int t = blockIdx.x;
  const int half = head_dim / 2;
  const float p = static_cast<float>(pos[t]);
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float inv = exp2f(-log2_theta * (2.0f * i) / head_dim);
    float s, c;
    sincosf(p * inv, &s, &c);
    cs[i] = c;
    cs[half + i] = s * sign;
  }
  __syncthreads();
  const int width = (n_q + 2 * n_kv) * head_dim;
  const bf16* row = in + size_t(t) * width;
  bf16* orow = out + size_t(t) * width;
  const int rot_heads = n_q + n_kv;
  const int vec_per_half = half / 8;
  const int rot_items = rot_heads * vec_per_half;
  for (int it = threadIdx.x; it < rot_items; it += blockDim.x) {
    const int h = it / vec_per_half, j = (it % vec_per_half) * 8;
    const uint4 a = *reinterpret_cast<const uint4*>(row + h * head_dim + j);
    const uint4 b = *reinterpret_cast<const uint4*>(row + h * head_dim + half + j);
    float x1[8], x2[8], o1[8], o2[8];
    unpack8(a, x1);
    unpack8(b, x2);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      rotate_pair(x1[i], x2[i], cs[j + i], cs[half + j + i], &o1[i], &o2[i]);
    }
    *reinterpret_cast<uint4*>(orow + h * head_dim + j) = pack8(o1);
    *reinterpret_cast<uint4*>(orow + h * head_dim + half + j) = pack8(o2);
  }
  const int v_off = rot_heads * head_dim;
  const int v_vecs = n_kv * head_dim / 8;
  for (int it = threadIdx.x; it < v_vecs; it += blockDim.x)
    *reinterpret_cast<uint4*>(orow + v_off + it * 8) = *reinterpret_cast<const uint4*>(row + v_off + it * 8);
}

// ------------------------------------------------------------------------- SwiGLU -----------
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ out, long long rows, int f) {
  const int vec_per_row = f / 8;
  const long long total = rows * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = static_cast<int>(i % vec_per_row) * 8;
    const uint4 g = *reinterpret_cast<const uint4*>(gu + r * 2 * f + c);
    const uint4 u = *reinterpret_cast<const uint4*>(gu + r * 2 * f + f + c);
    float gf[8], uf[8], o[8];
    unpack8(g, gf);
    unpack8(u, uf);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = gf[k] / (1.f + __expf(-gf[k])) * uf[k];
    *reinterpret_cast<uint4*>(out + r * f + c) = pack8(o);
  }
}

__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ gu, bf16* __restrict__ dgu, long long rows,
                  int f) {
  const int vec_per_row = f / 8;
  const long long total = rows * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = static_cast<int>(i % vec_per_row) * 8;
    const uint4 g = *reinterpret_cast<const uint4*>(gu + r * 2 * f + c);
    const uint4 u = *reinterpret_cast<const uint4*>(gu + r * 2 * f + f + c);
    const uint4 d = *reinterpret_cast<const uint4*>(dy + r * f + c);
    float gf[8], uf[8], df[8], dg[8], du[8];
    unpack8(g, gf);
    unpack8(u, uf);
    unpack8(d, df);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sig = 1.f / (1.f + __expf(-gf[k]));
      const float silu = gf[k] * sig;
      du[k] = df[k] * silu;
      dg[k] = df[k] * uf[k] * (sig + silu * (1.f - sig));
    }
    *reinterpret_cast<uint4*>(dgu + r * 2 * f + c) = pack8(dg);
    *reinterpret_cast<uint4*>(dgu + r * 2 * f + f + c) = pack8(du);
  }
}

// ------------------------------------------------------------------------- cross-entropy ----
// one CTA per row; pass 1: online max / sum-exp; pass 2: logits <- scale * (softmax - onehot)
// kForwardOnly: pass 1 only, the logits stay as they are and the row's log-probability of its label
// (0 for an ignored row) goes to per_token[row]; the scale and the summed loss are not used.
// inv_temp multiplies every logit on the way in (fp32): dividing the stored logits by a temperature would be one more
// pass over them and a second rounding to bf16.
constexpr int kCeThreads = 1024;
template <bool kForwardOnly>
__global__ void __launch_bounds__(kCeThreads)
ce_fwd_bwd_kernel(bf16* __restrict__ logits, const long long* __restrict__ labels, const float* __restrict__ loss_scale,
                  float* __restrict__ loss, int vocab, long long ignore_index, float* __restrict__ per_token,
                  float inv_temp) {
  __shared__ float red[32];
  const int row = blockIdx.x;
  bf16* lr = logits + size_t(row) * vocab;
  const long long label = labels[row];
  const float scale = (!kForwardOnly && loss_scale) ? loss_scale[row] : 1.f;
  const bool ignored = (label == ignore_index) || scale == 0.f;
  const int nvec = vocab / 8;
  uint4* lv = reinterpret_cast<uint4*>(lr);
  if (ignored) {
    if constexpr (kForwardOnly) {
      if (threadIdx.x == 0) per_token[row] = 0.f;
    } else {
      for (int v = threadIdx.x; v < nvec; v += blockDim.x) lv[v] = make_uint4(0, 0, 0, 0);
      for (int j = nvec * 8 + threadIdx.x; j < vocab; j += blockDim.x) lr[j] = __float2bfloat16(0.f);
    }
    return;
  }
  float m = -INFINITY, s = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(lv[v], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] *= inv_temp;
    float mx = f[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, f[i]);
    if (mx > m) {
      s *= __expf(m - mx);
      m = mx;
    }
    const float m_sub = m == -INFINITY ? 0.f : m;   // nothing but -inf so far has no weight
#pragma unroll
    for (int i = 0; i < 8; ++i) s += __expf(f[i] - m_sub);
  }
  for (int j = nvec * 8 + threadIdx.x; j < vocab; j += blockDim.x) {
    const float f = __bfloat162float(lr[j]) * inv_temp;
    if (f > m) {
      s *= __expf(m - f);
      m = f;
    }
    s += __expf(f - (m == -INFINITY ? 0.f : m));
  }
  const float gm = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + logf(gs);
  if constexpr (kForwardOnly) {
    if (threadIdx.x == 0) per_token[row] = __bfloat162float(lr[label]) * inv_temp - lse;
    return;
  }
  if (threadIdx.x == 0) atomicAdd(loss, scale * (lse - __bfloat162float(lr[label]) * inv_temp));
  __syncthreads();  // the label logit is read above before anyone overwrites it
  const float inv = 1.f / gs;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(lv[v], f);
    const int base = v * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float p = __expf(f[i] * inv_temp - gm) * inv;
      if (base + i == label) p -= 1.f;
      f[i] = p * scale;
    }
    lv[v] = pack8(f);
  }
  for (int j = nvec * 8 + threadIdx.x; j < vocab; j += blockDim.x) {
    float p = __expf(__bfloat162float(lr[j]) * inv_temp - gm) * inv;
    if (j == label) p -= 1.f;
    lr[j] = __float2bfloat16(p * scale);
  }
}

// The same from the statistics that the head's product left per row and tile of 256 columns (logits / temperature in units of
// log2(e)): one pass over the logits, bound by HBM, four 16-byte loads in flight per thread.  (From the logits
// alone, 4096 x 128256: two passes, 0.49 ms.)
constexpr float kLn2 = 0.6931471805599453f, kLog2e = 1.4426950408889634f;
// log2 of the sum of 2^x over a row, from its tiles' (maximum, sum); `red`: by the whole CTA, else by one warp
__device__ __forceinline__ float row_lse2(const float2* stats, int tiles, long long rows, int first, int step, float* red) {
  float m = -INFINITY, s = 0.f;
  for (int t = first; t < tiles; t += step) {
    const float2 x = stats[t * rows];
    const float m_new = fmaxf(m, x.x), m_sub = m_new == -INFINITY ? 0.f : m_new;
    s = s * exp2f(m - m_sub) + x.y * exp2f(x.x - m_sub);
    m = m_new;
  }
  const float gm = red ? block_max(m, red) : warp_max(m), m_sub = gm == -INFINITY ? 0.f : gm;
  s *= exp2f(m - m_sub);
  return gm + log2f(red ? block_sum(s, red) : warp_sum(s));
}

__global__ void __launch_bounds__(256)
ce_from_stats_kernel(bf16* __restrict__ logits, const long long* __restrict__ labels, const float* __restrict__ loss_scale,
                     const float2* __restrict__ stats, const float* __restrict__ label_logits, float* __restrict__ loss,
                     int rows, int vocab, int tiles, long long ignore_index, float inv_temp) {
  __shared__ float red[32];
  const int row = blockIdx.x, threads = blockDim.x;
  const long long label = labels[row];
  const float scale = loss_scale ? loss_scale[row] : 1.f;
  const int nvec = vocab / 8;
  uint4* lv = reinterpret_cast<uint4*>(logits + size_t(row) * vocab);
  if (label == ignore_index || scale == 0.f) {
    for (int v = threadIdx.x; v < nvec; v += threads) lv[v] = make_uint4(0, 0, 0, 0);
    return;
  }
  // few tiles: every warp sums them up by itself, without a barrier
  const float lse2 = tiles <= 64 ? row_lse2(stats + row, tiles, rows, threadIdx.x & 31, 32, nullptr)
                                 : row_lse2(stats + row, tiles, rows, threadIdx.x, threads, red);
  if (threadIdx.x == 0) atomicAdd(loss, scale * (lse2 * kLn2 - label_logits[row] * inv_temp));
  const float t2 = inv_temp * kLog2e;
  constexpr int kU = 4;
  for (int v0 = threadIdx.x; v0 < nvec; v0 += kU * threads) {
    uint4 u[kU];
#pragma unroll
    for (int k = 0; k < kU; ++k)
      if (v0 + k * threads < nvec) u[k] = lv[v0 + k * threads];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      const int v = v0 + k * threads;
      if (v < nvec) {
        float f[8];
        unpack8(u[k], f);
        const long long at = label - 8ll * v;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float p = exp2f(fmaf(f[i], t2, -lse2));
          if (at == i) p -= 1.f;
          f[i] = p * scale;
        }
        lv[v] = pack8(f);
      }
    }
  }
}

__global__ void __launch_bounds__(256)
logprobs_from_stats_kernel(const long long* __restrict__ labels, const float2* __restrict__ stats,
                           const float* __restrict__ label_logits, float* __restrict__ per_token, int rows, int tiles,
                           long long ignore_index, float inv_temp) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float lse2 = row_lse2(stats + row, tiles, rows, lane, 32, nullptr);
  if (lane == 0) per_token[row] = labels[row] == ignore_index ? 0.f : label_logits[row] * inv_temp - lse2 * kLn2;
}

// ------------------------------------------------------------------------- AdamW ------------
struct AdamWArgs {
  float lr, beta1, beta2, eps, wd, inv_bc1, inv_sqrt_bc2, grad_scale;
};
__device__ __forceinline__ void adamw_element(float& p, float g, float& m, float& v, const AdamWArgs& a) {
  g *= a.grad_scale;
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  const float denom = sqrtf(v) * a.inv_sqrt_bc2 + a.eps;
  p = p * (1.f - a.lr * a.wd) - a.lr * a.inv_bc1 * m / denom;
}

// Bound by HBM (30 bytes per element; 154 M elements: 768 us with 4-byte accesses in a grid-stride loop, 679 us, 6.8 TB/s,
// with V = 4).  V = 4: a thread moves 16 bytes of every fp32 array, once, so a resident SM has 128 KiB of loads in flight;
// the thread behind the last whole four takes the n % 4 elements that are left, in the same launch (in one of their own:
// 2097153 elements 10.3 us instead of 8.2).  V = 1 is for arrays that do not start on those boundaries.
template <typename GT, int V>
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ p, const GT* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
             bf16* __restrict__ p_lowp, size_t n, const AdamWArgs a) {
  size_t i = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * V;
  if (V == 1 || i + V > n) {
    for (const size_t end = V == 1 && i < n ? i + 1 : n; i < end; ++i) {
      float pi = p[i], mi = m[i], vi = v[i];
      adamw_element(pi, float(g[i]), mi, vi, a);
      p[i] = pi; m[i] = mi; v[i] = vi;
      if (p_lowp) p_lowp[i] = __float2bfloat16(pi);
    }
    return;
  }
  float4 p4 = *reinterpret_cast<const float4*>(p + i), m4 = *reinterpret_cast<const float4*>(m + i);
  float4 v4 = *reinterpret_cast<const float4*>(v + i), g4;
  if constexpr (sizeof(GT) == 4) {
    g4 = *reinterpret_cast<const float4*>(g + i);
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(g + i);
    g4 = make_float4(lo(u.x), hi(u.x), lo(u.y), hi(u.y));
  }
  adamw_element(p4.x, g4.x, m4.x, v4.x, a);
  adamw_element(p4.y, g4.y, m4.y, v4.y, a);
  adamw_element(p4.z, g4.z, m4.z, v4.z, a);
  adamw_element(p4.w, g4.w, m4.w, v4.w, a);
  *reinterpret_cast<float4*>(p + i) = p4;
  *reinterpret_cast<float4*>(m + i) = m4;
  *reinterpret_cast<float4*>(v + i) = v4;
  if (p_lowp) *reinterpret_cast<uint2*>(p_lowp + i) = make_uint2(pack(p4.x, p4.y), pack(p4.z, p4.w));
}

template <typename GT>
cudaError_t adamw_t(float* p, const GT* g, float* m, float* v, bf16* p_lowp, size_t n, const AdamWArgs& a, cudaStream_t stream) {
  const uintptr_t wide = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v);
  const bool aligned = wide % 16 == 0 && reinterpret_cast<uintptr_t>(g) % (4 * sizeof(GT)) == 0 &&
                       reinterpret_cast<uintptr_t>(p_lowp) % 8 == 0;
  const size_t threads = aligned ? (n + 3) / 4 : n;
  const unsigned int grid = static_cast<unsigned int>((threads + 255) / 256);
  if (aligned)
    adamw_kernel<GT, 4><<<grid, 256, 0, stream>>>(p, g, m, v, p_lowp, n, a);
  else
    adamw_kernel<GT, 1><<<grid, 256, 0, stream>>>(p, g, m, v, p_lowp, n, a);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
cast_f32_bf16_kernel(const float* __restrict__ in, bf16* __restrict__ out, size_t n) {
  const size_t nvec = n / 8;
  for (size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x; v < nvec; v += size_t(gridDim.x) * blockDim.x) {
    const float4 a = *reinterpret_cast<const float4*>(in + v * 8);
    const float4 b = *reinterpret_cast<const float4*>(in + v * 8 + 4);
    *reinterpret_cast<uint4*>(out + v * 8) = make_uint4(pack(a.x, a.y), pack(a.z, a.w), pack(b.x, b.y), pack(b.z, b.w));
  }
  if (blockIdx.x == 0)
    for (size_t j = nvec * 8 + threadIdx.x; j < n; j += blockDim.x) out[j] = __float2bfloat16(in[j]);
}

// out = in * *scale, one pass from fp32 or bf16 (gradients that were formed for a loss gradient of one)
template <typename T>
__global__ void __launch_bounds__(256)
scale_to_bf16_kernel(const T* __restrict__ in, bf16* __restrict__ out, const float* __restrict__ scale, size_t n) {
  const float s = *scale;
  const size_t nvec = n / 8;
  for (size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x; v < nvec; v += size_t(gridDim.x) * blockDim.x) {
    float f[8];
    if constexpr (sizeof(T) == 4) {
      const float4 a = *reinterpret_cast<const float4*>(in + v * 8), b = *reinterpret_cast<const float4*>(in + v * 8 + 4);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
      unpack8(*reinterpret_cast<const uint4*>(in + v * 8), f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] *= s;
    *reinterpret_cast<uint4*>(out + v * 8) = pack8(f);
  }
  if (blockIdx.x == 0)
    for (size_t j = nvec * 8 + threadIdx.x; j < n; j += blockDim.x) out[j] = __float2bfloat16(float(in[j]) * s);
}

template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(const T* __restrict__ x, size_t n, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    float f;
    if constexpr (sizeof(T) == 4) f = x[i]; else f = __bfloat162float(x[i]);
    s += f * f;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

int cap_grid(long long work_items, int threads, int sm_count, int per_sm) {
  long long g = (work_items + threads - 1) / threads;
  const long long cap = (long long)sm_count * per_sm;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

template <int R>
cudaError_t rmsnorm_fwd_t(const void* x, const void* w, void* y, float* rstd, int rows, int cols, float eps, int sm_count,
                          cudaStream_t stream) {
  const int want = (rows + kNormWarps / R - 1) / (kNormWarps / R);
  const int grid = want < sm_count * 8 ? want : sm_count * 8;
  launch(rmsnorm_fwd_kernel<R>, grid, kNormThreads, 0, stream,
      static_cast<const bf16*>(x), static_cast<const bf16*>(w), static_cast<bf16*>(y), rstd, rows, cols, eps);
  return cudaGetLastError();
}

template <int R, int V>
cudaError_t rmsnorm_bwd_t(const void* dy, const void* x, const void* w, const float* rstd, void* dx, float* partial,
                          float* dw, int rows, int cols, int grid, cudaStream_t stream, const void* dres) {
  if (partial == nullptr) {
    launch(rmsnorm_bwd_kernel<R, V, true>, grid, kNormThreads, kNormWarps / R * cols * sizeof(float), stream,
        static_cast<const bf16*>(dy), static_cast<const bf16*>(x), static_cast<const bf16*>(w), rstd,
        static_cast<bf16*>(dx), nullptr, dw, rows, cols, static_cast<const bf16*>(dres));
  } else {
    launch(rmsnorm_bwd_kernel<R, V, false>, grid, kNormThreads, kNormWarps / R * cols * sizeof(float), stream,
        static_cast<const bf16*>(dy), static_cast<const bf16*>(x), static_cast<const bf16*>(w), rstd,
        static_cast<bf16*>(dx), partial, dw, rows, cols, static_cast<const bf16*>(dres));
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows, int cols, float eps,
                               int sm_count, cudaStream_t stream) {
  if (cols % 8 != 0 || cols > 8192) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  if (cols <= 2048) return rmsnorm_fwd_t<1>(x, w, y, rstd, rows, cols, eps, sm_count, stream);
  if (cols <= 4096) return rmsnorm_fwd_t<2>(x, w, y, rstd, rows, cols, eps, sm_count, stream);
  return rmsnorm_fwd_t<4>(x, w, y, rstd, rows, cols, eps, sm_count, stream);
}

int rmsnorm_bwd_grid(int rows, int sm_count) {
  const int want = (rows + kNormWarps - 1) / kNormWarps;
  const int g = sm_count * 2;
  return want < g ? (want < 1 ? 1 : want) : g;
}

// partial == nullptr: single launch, the CTAs add their column sums into dw (zeroed here first unless `add`; the order
// of the additions varies from run to run).  partial = [grid, cols] scratch: per-CTA sums, then a fixed-order column pass.
cudaError_t launch_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                               float* partial, float* dw, int rows, int cols, int grid, cudaStream_t stream,
                               const void* dres, bool add) {
  if (cols % 8 != 0 || cols > 8192 || (add && partial != nullptr)) return cudaErrorInvalidValue;
  cudaError_t e;
  if (add) {
    if (rows == 0) return cudaSuccess;
  } else if (partial == nullptr) {
    e = cudaMemsetAsync(dw, 0, sizeof(float) * cols, stream);
    if (e != cudaSuccess) return e;
    if (rows == 0) return cudaSuccess;
  }
  if (cols <= 1024) e = rmsnorm_bwd_t<1, 4>(dy, x, w, rstd, dx, partial, dw, rows, cols, grid, stream, dres);
  else if (cols <= 2048) e = rmsnorm_bwd_t<2, 4>(dy, x, w, rstd, dx, partial, dw, rows, cols, grid, stream, dres);
  else if (cols <= 4096) e = rmsnorm_bwd_t<4, 4>(dy, x, w, rstd, dx, partial, dw, rows, cols, grid, stream, dres);
  else e = rmsnorm_bwd_t<8, 4>(dy, x, w, rstd, dx, partial, dw, rows, cols, grid, stream, dres);
  if (e != cudaSuccess) return e;
  if (partial != nullptr) {
    colsum_kernel<<<(cols + 255) / 256, 256, 0, stream>>>(partial, dw, grid, cols);
    e = cudaGetLastError();
  }
  return e;
}

// Two fp32 vectors next to one another, in bf16, each into a tensor of its own: what a layer's norms sum up in its backward.  Cleared
// and narrowed together they take two launches of the layer's backward instead of four, 8 us of 331 over 1000 tokens (narrowing them in
// the CTA that adds last instead lengthened that kernel by 5 us each).
__global__ void __launch_bounds__(256) narrow_pair_kernel(const float* __restrict__ in, bf16* __restrict__ a, bf16* __restrict__ b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 2 * n) (i < n ? a[i] : b[i - n]) = __float2bfloat16(in[i]);
}
cudaError_t launch_narrow_pair(const float* in, void* a, void* b, int n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  launch(narrow_pair_kernel, (2 * n + 255) / 256, 256, 0, stream, in, static_cast<bf16*>(a), static_cast<bf16*>(b), n);
  return cudaGetLastError();
}

cudaError_t launch_column_sum(const void* x, void* out, float* sink, long long rows, int cols, cudaStream_t stream) {
  if (cols % 8 != 0 || (out == nullptr) == (sink == nullptr)) return cudaErrorInvalidValue;
  if (cols == 0) return cudaSuccess;
  launch(column_sum_kernel, (cols + 63) / 64, kColSumThreads, 0, stream,
      static_cast<const bf16*>(x), static_cast<bf16*>(out), sink, rows, cols);
  return cudaGetLastError();
}

cudaError_t launch_rope_qkv(const void* in, void* out, const long long* pos, int tokens, int n_q, int n_kv,
                            int head_dim, float theta, bool inverse, cudaStream_t stream) {
  if (head_dim % 16 != 0) return cudaErrorInvalidValue;
  if (tokens == 0) return cudaSuccess;
  launch(rope_qkv_kernel, tokens, 128, head_dim * sizeof(float), stream,
      static_cast<const bf16*>(in), static_cast<bf16*>(out), pos, n_q, n_kv, head_dim, log2f(theta),
      inverse ? -1.f : 1.f);
  return cudaGetLastError();
}

cudaError_t launch_swiglu_fwd(const void* gate_up, void* out, long long rows, int f, int sm_count,
                              cudaStream_t stream) {
  if (f % 8 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  launch(swiglu_fwd_kernel, cap_grid(rows * (f / 8), 256, sm_count, 16), 256, 0, stream,
      static_cast<const bf16*>(gate_up), static_cast<bf16*>(out), rows, f);
  return cudaGetLastError();
}

cudaError_t launch_swiglu_bwd(const void* dy, const void* gate_up, void* dgate_up, long long rows, int f,
                              int sm_count, cudaStream_t stream) {
  if (f % 8 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  launch(swiglu_bwd_kernel, cap_grid(rows * (f / 8), 256, sm_count, 16), 256, 0, stream,
      static_cast<const bf16*>(dy), static_cast<const bf16*>(gate_up), static_cast<bf16*>(dgate_up), rows, f);
  return cudaGetLastError();
}

cudaError_t launch_ce_fwd_bwd(void* logits, const long long* labels, const float* loss_scale, float* loss,
                              int rows, int vocab, long long ignore_index, cudaStream_t stream, float inv_temp) {
  if (rows == 0) return cudaSuccess;
  if (vocab % 8 != 0) return cudaErrorInvalidValue;  // rows must stay 16-byte aligned
  launch(ce_fwd_bwd_kernel<false>, rows, kCeThreads, 0, stream,
      static_cast<bf16*>(logits), labels, loss_scale, loss, vocab, ignore_index, nullptr, inv_temp);
  return cudaGetLastError();
}

cudaError_t launch_token_logprobs(const void* logits, const long long* labels, float* per_token, int rows, int vocab,
                                  long long ignore_index, cudaStream_t stream, float inv_temp) {
  if (rows == 0) return cudaSuccess;
  if (vocab % 8 != 0 || per_token == nullptr) return cudaErrorInvalidValue;
  // the forward-only instantiation never writes through the logits pointer
  launch(ce_fwd_bwd_kernel<true>, rows, kCeThreads, 0, stream,
      static_cast<bf16*>(const_cast<void*>(logits)), labels, nullptr, nullptr, vocab, ignore_index, per_token, inv_temp);
  return cudaGetLastError();
}

cudaError_t launch_ce_from_stats(void* logits, const long long* labels, const float* loss_scale, const float* row_stats,
                                 const float* label_logits, float* loss, int rows, int vocab, int tiles, long long ignore_index,
                                 cudaStream_t stream, float inv_temp) {
  if (rows == 0) return cudaSuccess;
  if (vocab % 8 != 0) return cudaErrorInvalidValue;
  // 256 threads a row at every length: more of them wait for one another over the tiles' statistics.  Head product of width 64
  // and this pass, 4096 rows: 4096 words 49 us (512 threads 63, 1024 92), 32000 247 (262, 304), 128256 941 (944, 982), 151936
  // 1109 (1122, 1155)
  launch(ce_from_stats_kernel, rows, 256, 0, stream, static_cast<bf16*>(logits), labels, loss_scale,
      reinterpret_cast<const float2*>(row_stats), label_logits, loss, rows, vocab, tiles, ignore_index, inv_temp);
  return cudaGetLastError();
}

cudaError_t launch_logprobs_from_stats(const long long* labels, const float* row_stats, const float* label_logits, float* per_token,
                                       int rows, int tiles, long long ignore_index, cudaStream_t stream, float inv_temp) {
  if (rows == 0) return cudaSuccess;
  launch(logprobs_from_stats_kernel, (rows + 7) / 8, 256, 0, stream, labels, reinterpret_cast<const float2*>(row_stats),
      label_logits, per_token, rows, tiles, ignore_index, inv_temp);
  return cudaGetLastError();
}

cudaError_t launch_adamw(float* p, const void* g, int g_kind, float* m, float* v, void* p_lowp, size_t n, float lr,
                         float beta1, float beta2, float eps, float wd, float bc1, float bc2, float grad_scale,
                         cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const AdamWArgs a{lr, beta1, beta2, eps, wd, 1.f / bc1, 1.f / sqrtf(bc2), grad_scale};
  if (g_kind == kF32) return adamw_t(p, static_cast<const float*>(g), m, v, static_cast<bf16*>(p_lowp), n, a, stream);
  if (g_kind == kBF16) return adamw_t(p, static_cast<const bf16*>(g), m, v, static_cast<bf16*>(p_lowp), n, a, stream);
  return cudaErrorInvalidValue;
}

cudaError_t launch_cast_f32_to_bf16(const float* in, void* out, size_t n, int sm_count, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  cast_f32_bf16_kernel<<<cap_grid(static_cast<long long>(n / 8 + 1), 256, sm_count, 16), 256, 0, stream>>>(
      in, static_cast<bf16*>(out), n);
  return cudaGetLastError();
}

cudaError_t launch_scale_to_bf16(const void* in, int in_kind, void* out, const float* scale, size_t n, int sm_count,
                                 cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const int grid = cap_grid(static_cast<long long>(n / 8 + 1), 256, sm_count, 16);
  if (in_kind == kF32)
    scale_to_bf16_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(in), static_cast<bf16*>(out), scale, n);
  else if (in_kind == kBF16)
    scale_to_bf16_kernel<bf16><<<grid, 256, 0, stream>>>(static_cast<const bf16*>(in), static_cast<bf16*>(out), scale, n);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_sumsq(const void* x, int kind, size_t n, float* out, int sm_count, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const int grid = cap_grid(static_cast<long long>(n), 256, sm_count, 8);
  if (kind == kF32)
    sumsq_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(x), n, out);
  else
    sumsq_kernel<bf16><<<grid, 256, 0, stream>>>(static_cast<const bf16*>(x), n, out);
  return cudaGetLastError();
}

}  // namespace odc
