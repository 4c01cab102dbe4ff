// Memory-bound fused ops for sm_100a. Each kernel moves 16-byte vectors, touches
// every activation byte once, and can emit the next GEMM's FP8 operand
// (e4m3 values + one fp32 scale per 128 consecutive elements) directly, so that
// no stand-alone quantisation pass reads the activation again.
//
// Covers the reference kernels
//   layernorm  : 3rdparty/LLM_kernels/csrc/kernels/nvidia/layernorm/layernorm.cu:378-587
//   add        : .../add/add.cu:55-90
//   activation : .../activation/activation.cu:205-232,497-507
//   embedding  : .../embedding/embedding.cu:20-75
//   assemble   : .../assemble_last_token/assemble_last_token.cu:14-42
//   rotary     : .../rotary_embedding/rotary_embedding.cu:70-197
//   cache copy : .../paged_attention/cache_copy.cu:21-254
//   fp8 quant  : 3rdparty/LLM_kernels/csrc/utils/nvidia/cuda_fp8_utils.cu:27-140
#include "guards.cuh"
#include "pdl.cuh"
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_fp4.h>
#include <stdint.h>
#include "fp8_scale.cuh"
#include "fast_div.cuh"
#define KSANA_F32X2_FLUSH          // as this file's arithmetic on single floats: a row's bits do not depend on the kernel that a launch takes
#include "f32x2.cuh"
#include "vec8.cuh"

namespace ksana {

typedef __nv_bfloat16 bf16;

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
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = l < nw ? red[l] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(p[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}
// 8 floats -> 8 e4m3 bytes (two 32-bit words)
__device__ __forceinline__ uint2 pack8_e4m3(const float (&f)[8], float inv_scale) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(
        make_float2(f[4 * h] * inv_scale, f[4 * h + 1] * inv_scale), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(
        make_float2(f[4 * h + 2] * inv_scale, f[4 * h + 3] * inv_scale), __NV_SATFINITE, __NV_E4M3);
    w[h] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  return make_uint2(w[0], w[1]);
}
// 1 / scale for a scale of fp8_group_scale, exactly: a power of two up to 2^120, or infinite (a group that holds an infinity), whose
// inverse is 0: finite values become 0 and infinite ones NaN
__device__ __forceinline__ float pow2_inverse(float s) {
  const uint32_t b = __float_as_uint(s);
  return __uint_as_float(b < 0x7F000000u ? 0x7F000000u - b : 0u);
}
// largest magnitude of eight bf16 values over the 16 lanes that share one 128-element group, on packed pairs
__device__ __forceinline__ float group16_absmax(const uint4& v) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
  __nv_bfloat162 m = __hmax2(__hmax2(__habs2(p[0]), __habs2(p[1])), __hmax2(__habs2(p[2]), __habs2(p[3])));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const uint32_t x = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&m), o);
    m = __hmax2(m, *reinterpret_cast<const __nv_bfloat162*>(&x));
  }
  const float2 f = __bfloat1622float2(m);
  return fmaxf(f.x, f.y);
}

// ----------------------------------------------------------------------------
// (residual +=) x ; y = norm(residual or x) * w (+ beta) ; optional fp8 copy of y.
// mode 0 = RMSNorm, 1 = LayerNorm. One CTA per row; up to kMaxVec vectors per thread.
constexpr int kMaxVec = 4;

// QUANT: with the fp8 copy. What a launch does not need is left out of its instance. Layer norms, norms that update a residual and rows that
// norm_rows_kernel does not take.
template <int MODE, bool RES, bool QUANT>
__global__ void norm_kernel(const bf16* __restrict__ x, bf16* __restrict__ residual, const bf16* __restrict__ w,
                            const bf16* __restrict__ beta, bf16* __restrict__ y, uint8_t* __restrict__ yq,
                            float* __restrict__ yscale, int scale_ld, int H, float eps) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int row = blockIdx.x;
  const int nvec = H >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * H);
  uint4* rr = RES ? reinterpret_cast<uint4*>(residual + static_cast<size_t>(row) * H) : nullptr;
  float v[kMaxVec][8];
  float s = 0.f, s2 = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * blockDim.x;
    if (i < nvec) {
      unpack8(xr[i], v[j]);
      if (RES) {
        float r[8];
        unpack8(rr[i], r);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[j][e] += r[e];
        const uint4 packed = pack8(v[j]);
        rr[i] = packed;
        unpack8(packed, v[j]);   // normalise exactly what the residual stream now holds
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) { if (MODE == 1) s += v[j][e]; else s2 += v[j][e] * v[j][e]; }
    }
  }
  float mean = 0.f, rstd;
  if (MODE == 1) {
    mean = block_sum(s, red) / H;
    float var = 0.f;
#pragma unroll
    for (int j = 0; j < kMaxVec; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if (i < nvec) {
#pragma unroll
        for (int e = 0; e < 8; ++e) { const float d = v[j][e] - mean; var += d * d; }
      }
    }
    rstd = rsqrtf(block_sum(var, red) / H + eps);
  } else {
    rstd = rsqrtf(block_sum(s2, red) / H + eps);
  }
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const uint4* br = beta ? reinterpret_cast<const uint4*>(beta) : nullptr;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * blockDim.x;   // blockDim is a multiple of 32, so groups of 16 lanes stay aligned
    const bool on = i < nvec;
    uint4 packed = make_uint4(0, 0, 0, 0);
    if (on) {
      float wf[8], o[8];
      unpack8(wr[i], wf);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = (MODE == 1 ? v[j][e] - mean : v[j][e]) * rstd * wf[e];
      if (br) {
        float bfv[8];
        unpack8(br[i], bfv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += bfv[e];
      }
      // round to bf16 first so that the fp8 copy quantises the same values y holds
      packed = pack8(o);
      if (y) reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * H)[i] = packed;
    }
    if (QUANT) {
      const float scale = fp8_group_scale(group16_absmax(packed));
      if (on) {
        float o[8];
        unpack8(packed, o);
        reinterpret_cast<uint2*>(yq + static_cast<size_t>(row) * H)[i] = pack8_e4m3(o, pow2_inverse(scale));
        if ((i & 15) == 0) yscale[static_cast<size_t>(i >> 4) * scale_ld + row] = scale;
      }
    }
  }
}

// ----------------------------------------------------------------------------
// Chunks of 16 elements (32 bytes of bf16) per thread, for launches of many rows: eight lanes share a 128-element group instead of sixteen, so
// that the group's maximum takes three exchanges per 16 elements instead of eight, and arithmetic runs on packed pairs of floats. After GEMMs
// that bring the card to its power limit the SM clock is a third lower while memory is not: these kernels are paced by their instructions then.
struct Chunk16 { uint32_t w[8]; };
__device__ __forceinline__ Chunk16 ld_chunk(const bf16* p) {
  Chunk16 c;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(c.w[0]), "=r"(c.w[1]), "=r"(c.w[2]), "=r"(c.w[3]), "=r"(c.w[4]), "=r"(c.w[5]), "=r"(c.w[6]), "=r"(c.w[7]) : "l"(p) : "memory");
  return c;
}
__device__ __forceinline__ F2 unpack2(uint32_t w) { return f2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ uint32_t pack2(F2 p) {
  float x, y;
  split(p, x, y);
  const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&b);
}
// largest magnitude of a chunk and those of the lanes that share its 128-element group (eight in a row)
__device__ __forceinline__ float group8_absmax(const Chunk16& c) {
  auto b2 = [](uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); };
  __nv_bfloat162 m = __habs2(b2(c.w[0]));
#pragma unroll
  for (int k = 1; k < 8; ++k) m = __hmax2(m, __habs2(b2(c.w[k])));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    const uint32_t x = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&m), o);
    m = __hmax2(m, b2(x));
  }
  const float2 f = __bfloat1622float2(m);
  return fmaxf(f.x, f.y);
}
// Largest of the threads' magnitudes m (up to 8 warps), at the CTA's place of `parts`; NaN do not count.
__device__ __forceinline__ void publish_absmax(float m, float* parts) {
  __shared__ float red[8];
  const float w = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x == 0) {
    float all = red[0];
    for (int k = 1; k < static_cast<int>(blockDim.x >> 5); ++k) all = fmaxf(all, red[k]);
    parts[blockIdx.x] = all;
  }
}
__device__ __forceinline__ float larger(__nv_bfloat162 m) {
  const float2 f = __bfloat1622float2(m);
  return fmaxf(f.x, f.y);
}
__device__ __forceinline__ __nv_bfloat162 chunk_absmax(const Chunk16& c, __nv_bfloat162 m) {
#pragma unroll
  for (int e = 0; e < 8; ++e) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&c.w[e])));
  return m;
}
// a chunk times `inv` as 16 e4m3 values
__device__ __forceinline__ uint4 chunk_e4m3(const Chunk16& c, float inv) {
  uint32_t o[4];
  const F2 inv2 = f2(inv);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float x0, x1, y0, y1;
    split(unpack2(c.w[2 * k]) * inv2, x0, x1);
    split(unpack2(c.w[2 * k + 1]) * inv2, y0, y1);
    const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(x0, x1), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(y0, y1), __NV_SATFINITE, __NV_E4M3);
    o[k] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Root-mean-square norm: CTAs stay and take row after row, the next row's loads in flight under the work on this one. One CTA per row
// (norm_kernel) spent its time waiting and on 21.6 instructions an element. us, there / here: with fp8 copy 16384 x 8192 122 / 74 (5.5 TB/s),
// 8000 x 7168 60 / 39, 300 x 7168 5.7 / 4.2; 16384 x 4096 56 / 43, 64 x 4096 3.9 / 2.6. V chunks per thread.
// AMAX: parts[CTA] takes the largest magnitude of its results (the tensor scale of an NVFP4 operand without a pass of its own).
template <bool QUANT, int V, bool AMAX>
__global__ void __launch_bounds__(256, V == 1 ? 4 : V == 2 ? 3 : 2)
norm_rows_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y, uint8_t* __restrict__ yq,
                 float* __restrict__ yscale, int scale_ld, int M, int H, float eps, float* parts) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[2][8];
  const int chunks = H >> 4, warps = blockDim.x >> 5;
  Chunk16 next[V];
  auto fetch = [&](int row) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = threadIdx.x + k * blockDim.x;
      if (c < chunks) next[k] = ld_chunk(x + static_cast<size_t>(row) * H + c * 16);
    }
  };
  int row = blockIdx.x, turn = 0;
  __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
  if (row < M) fetch(row);
  for (; row < M; row += gridDim.x, turn ^= 1) {
    Chunk16 v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = next[k];
    if (row + static_cast<int>(gridDim.x) < M) fetch(row + gridDim.x);
    F2 s2[2] = {f2(0.f), f2(0.f)};
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (static_cast<int>(threadIdx.x + k * blockDim.x) < chunks) {
#pragma unroll
        for (int e = 0; e < 8; ++e) { const F2 t = unpack2(v[k].w[e]); s2[e & 1] = fma2(t, t, s2[e & 1]); }
      }
    const float s = warp_sum(sum2(s2[0] + s2[1]));
    if ((threadIdx.x & 31) == 0) red[turn][threadIdx.x >> 5] = s;
    __syncthreads();                               // (the other set of sums is written only after the next row's)
    float all = 0.f;
    for (int i = 0; i < warps; ++i) all += red[turn][i];
    const F2 rstd = f2(rsqrtf(all / H + eps));
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = threadIdx.x + k * blockDim.x;
      const bool on = c < chunks;                  // (whole groups of eight lanes where QUANT: H is a multiple of 128)
      Chunk16 o = {};
      if (on) {
        const Chunk16 wc = ld_chunk(w + c * 16);
#pragma unroll
        for (int e = 0; e < 8; ++e) o.w[e] = pack2(unpack2(v[k].w[e]) * rstd * unpack2(wc.w[e]));
      }
      if constexpr (AMAX) top = chunk_absmax(o, top);
      if constexpr (QUANT) {
        const float scale = fp8_group_scale(group8_absmax(o));
        if (on) {
          *reinterpret_cast<uint4*>(yq + static_cast<size_t>(row) * H + c * 16) = chunk_e4m3(o, pow2_inverse(scale));
          if ((c & 7) == 0) yscale[static_cast<size_t>(c >> 3) * scale_ld + row] = scale;
        }
      }
      if (on && (!QUANT || y)) {
        st_global_32(y + static_cast<size_t>(row) * H + c * 16, make_uint4(o.w[0], o.w[1], o.w[2], o.w[3]),
                     make_uint4(o.w[4], o.w[5], o.w[6], o.w[7]));
      }
    }
  }
  if constexpr (AMAX) publish_absmax(larger(top), parts);
}

// ----------------------------------------------------------------------------
// out[m, i] = act(gate_up[m, i]) * gate_up[m, I + i] ; optional fp8 copy. act: 0 silu 1 gelu(tanh) 2 relu
// When `gated` is 0 the input is [M, I] and out = act(in). tile_rows (may be null): of every 128 rows only so many hold
// anything, the others are skipped.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 0.5 x (1 + tanh(c)) = x / (1 + exp(-2 c)) with c = sqrt(2 / pi) (x + 0.044715 x^3): no cancellation where tanh is near -1
__device__ __forceinline__ float gelu_tanh(float x) {
  return x / (1.f + __expf(-1.5957691216f * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float act_fn(float x, int act) {
  // silu(x) = x * sigmoid(x) = 0.5 x (1 + tanh(x / 2)): one special-function op per element instead of an
  // exponential and a division (the special-function unit, not memory, paced this kernel); the approximation's
  // error (about 2^-11) is below the bf16 rounding of the result
  if (act == 0) { const float hx = 0.5f * x; return fmaf(hx, tanh_fast(hx), hx); }
  if (act == 1) return gelu_tanh(x);
  return fmaxf(x, 0.f);
}

// Memory is the bound it nears: gated and quantised, an element reads 4 bytes and writes 1. Row and column come from a multiplication (the
// 64-bit division of a flat index was half of the kernel's instructions: 16384 x 28672 gated, quantised: 733 us with it, 566 us without,
// 532 us with maxima on packed pairs: 4.4 TB/s). V vectors of a thread are in flight together; see launch_vectors for how many.
template <int ACT, bool GATED, bool QUANT, int V>
__global__ void __launch_bounds__(256)
act_mul_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, uint8_t* __restrict__ outq, float* __restrict__ oscale,
               int scale_ld, uint32_t total, FastDiv nvec, int in_ld, const int* __restrict__ tile_rows) {
  pdl_trigger();
  pdl_wait();
  const uint32_t step = gridDim.x * blockDim.x;
  // whole warps stay in the loop for the shuffles; nvec is a multiple of 16 with QUANT, so 16 consecutive lanes share (m, group)
  for (uint32_t base = blockIdx.x * blockDim.x + threadIdx.x; (base & ~31u) < total; base += V * step) {
    uint4 g[V], u[V];
    uint32_t m[V], i[V];
    bool on[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint32_t idx = base + k * step;
      on[k] = idx < total;
      m[k] = on[k] ? nvec.div(idx) : 0u;
      i[k] = on[k] ? idx - m[k] * nvec.d : 0u;
      if (tile_rows) on[k] = on[k] && static_cast<int>(m[k] & 127) < tile_rows[m[k] >> 7];
      if (on[k]) {
        const uint4* row = reinterpret_cast<const uint4*>(in + static_cast<size_t>(m[k]) * in_ld);
        g[k] = __ldcs(row + i[k]);
        if (GATED) u[k] = __ldcs(row + nvec.d + i[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      uint4 packed = make_uint4(0, 0, 0, 0);
      if (on[k]) {
        float gf[8], uf[8], o[8];
        unpack8(g[k], gf);
        if (GATED) unpack8(u[k], uf);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = GATED ? act_fn(gf[e], ACT) * uf[e] : act_fn(gf[e], ACT);
        packed = pack8(o);
        if (out) reinterpret_cast<uint4*>(out + static_cast<size_t>(m[k]) * nvec.d * 8)[i[k]] = packed;
      }
      if (QUANT) {
        const float scale = fp8_group_scale(group16_absmax(packed));
        if (on[k]) {
          float o[8];
          unpack8(packed, o);
          reinterpret_cast<uint2*>(outq + static_cast<size_t>(m[k]) * nvec.d * 8)[i[k]] = pack8_e4m3(o, pow2_inverse(scale));
          if ((i[k] & 15) == 0) oscale[static_cast<size_t>(i[k] >> 4) * scale_ld + m[k]] = scale;
        }
      }
    }
  }
}

// Gated rows in chunks of 16 elements (see there); arguments as act_mul_kernel, nchunk counts a row's chunks. At full clocks 16384 x 28672
// quantised 405 -> 379 us (6.2 TB/s), without fp8 16384 x 14336 226 -> 224; quantisation alone of 16384 x 8192 74 -> 67.
template <int ACT, bool QUANT, bool AMAX>
__global__ void __launch_bounds__(256)
act_chunks_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, uint8_t* __restrict__ outq, float* __restrict__ oscale, int scale_ld,
                  uint32_t total, FastDiv nchunk, int in_ld, const int* __restrict__ tile_rows, float* parts) {
  pdl_trigger();
  pdl_wait();
  const uint32_t step = gridDim.x * blockDim.x, I = nchunk.d * 16;
  __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; (idx & ~31u) < total; idx += step) {
    bool on = idx < total;                         // whole warps stay in the loop for the exchanges
    const uint32_t m = on ? nchunk.div(idx) : 0u, i = on ? idx - m * nchunk.d : 0u;
    if (tile_rows) on = on && static_cast<int>(m & 127) < tile_rows[m >> 7];
    Chunk16 o = {};
    if (on) {
      const bf16* row = in + static_cast<size_t>(m) * in_ld + i * 16;
      const Chunk16 g = ld_chunk(row), u = ld_chunk(row + I);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        F2 a;
        if constexpr (ACT == 0) {                  // act_fn on pairs
          const F2 hx = unpack2(g.w[e]) * f2(0.5f);
          float x, y;
          split(hx, x, y);
          a = fma2(hx, f2(tanh_fast(x), tanh_fast(y)), hx);
        } else {
          float x, y;
          split(unpack2(g.w[e]), x, y);
          a = f2(act_fn(x, ACT), act_fn(y, ACT));
        }
        o.w[e] = pack2(a * unpack2(u.w[e]));
      }
    }
    if constexpr (AMAX) top = chunk_absmax(o, top);
    if constexpr (QUANT) {
      const float scale = fp8_group_scale(group8_absmax(o));
      if (on) {
        *reinterpret_cast<uint4*>(outq + static_cast<size_t>(m) * I + i * 16) = chunk_e4m3(o, pow2_inverse(scale));
        if ((i & 7) == 0) oscale[static_cast<size_t>(i >> 3) * scale_ld + m] = scale;
      }
    }
    if (on && (!QUANT || out)) {
      st_global_32(out + static_cast<size_t>(m) * I + i * 16, make_uint4(o.w[0], o.w[1], o.w[2], o.w[3]), make_uint4(o.w[4], o.w[5], o.w[6], o.w[7]));
    }
  }
  if constexpr (AMAX) publish_absmax(larger(top), parts);
}

// The same on fp32 rows, with the exponential instead of the approximate tanh.
__global__ void act_mul_f32_kernel(const float* __restrict__ in, float* __restrict__ out, int M, int I, int in_ld, int act, int gated) {
  pdl_trigger();
  pdl_wait();
  const long long total = static_cast<long long>(M) * I;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long m = idx / I, i = idx - m * I;
    const float* row = in + m * in_ld;
    const float g = row[i];
    const float a = act == 0 ? g / (1.f + __expf(-g)) : act == 1 ? gelu_tanh(g) : fmaxf(g, 0.f);
    out[idx] = gated ? a * row[I + i] : a;
  }
}

// x[M,K] bf16 -> e4m3 + one scale per (row, 128 columns); scales stored [K/128][scale_ld]. Index arithmetic and loads in flight as in
// act_mul_kernel.
template <int V>
__global__ void __launch_bounds__(256)
quant_fp8_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, int scale_ld, uint32_t total,
                 FastDiv nvec, int x_ld) {
  pdl_trigger();
  pdl_wait();
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + threadIdx.x; (base & ~31u) < total; base += V * step) {
    uint4 v[V];
    uint32_t m[V], i[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const uint32_t idx = base + k * step;
      m[k] = idx < total ? nvec.div(idx) : 0u;
      i[k] = idx < total ? idx - m[k] * nvec.d : 0u;
      v[k] = idx < total ? __ldcs(reinterpret_cast<const uint4*>(x + static_cast<size_t>(m[k]) * x_ld) + i[k]) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float sc = fp8_group_scale(group16_absmax(v[k]));
      if (base + k * step < total) {
        float f[8];
        unpack8(v[k], f);
        reinterpret_cast<uint2*>(q + static_cast<size_t>(m[k]) * nvec.d * 8)[i[k]] = pack8_e4m3(f, pow2_inverse(sc));
        if ((i[k] & 15) == 0) scale[static_cast<size_t>(i[k] >> 4) * scale_ld + m[k]] = sc;
      }
    }
  }
}

__global__ void __launch_bounds__(256)
quant_chunks_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, int scale_ld, uint32_t total,
                    FastDiv nchunk, int x_ld) {
  pdl_trigger();
  pdl_wait();
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; (idx & ~31u) < total; idx += step) {
    const bool on = idx < total;
    const uint32_t m = on ? nchunk.div(idx) : 0u, i = on ? idx - m * nchunk.d : 0u;
    Chunk16 v = {};
    if (on) v = ld_chunk(x + static_cast<size_t>(m) * x_ld + i * 16);
    const float sc = fp8_group_scale(group8_absmax(v));
    if (on) {
      *reinterpret_cast<uint4*>(q + static_cast<size_t>(m) * nchunk.d * 16 + i * 16) = chunk_e4m3(v, pow2_inverse(sc));
      if ((i & 7) == 0) scale[static_cast<size_t>(i >> 3) * scale_ld + m] = sc;
    }
  }
}

// ----------------------------------------------------------------------------
// Embedding gather with vocabulary-shard awareness; rows whose id falls outside
// [vocab_lo, vocab_hi) are zero-filled (the TP all-reduce then completes them).
// Optional learned position table add and scale (GPT-style models).
__global__ void embedding_kernel(const int* __restrict__ ids, const bf16* __restrict__ table,
                                 const int* __restrict__ positions, const bf16* __restrict__ pos_table,
                                 bf16* __restrict__ out, int H, int vocab_lo, int vocab_hi, float scale) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const int id = ids[t];
  const bool mine = id >= vocab_lo && id < vocab_hi;
  const uint4* src = reinterpret_cast<const uint4*>(table + static_cast<size_t>(mine ? id - vocab_lo : 0) * H);
  const uint4* psrc = pos_table ? reinterpret_cast<const uint4*>(pos_table + static_cast<size_t>(positions[t]) * H)
                                : nullptr;
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) {
    float f[8];
    if (mine) {
      unpack8(src[i], f);
      if (scale != 1.f) {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= scale;
      }
      if (psrc) {
        float pf[8];
        unpack8(psrc[i], pf);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += pf[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = 0.f;
    }
    dst[i] = pack8(f);
  }
}

// out[r, :] = in[idx[r], :]  (last-token assembly, logits gather)
__global__ void gather_rows_kernel(const bf16* __restrict__ in, const int* __restrict__ idx, bf16* __restrict__ out,
                                   int H, int in_rows, int* err) {
  pdl_trigger();
  pdl_wait();
  int r = idx[blockIdx.x];
  if (r < 0 || r >= in_rows) { if (threadIdx.x == 0) guard_report(err, kGuardGatherRow, r); r = 0; }
  const uint4* src = reinterpret_cast<const uint4*>(in + static_cast<size_t>(r) * H);
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(blockIdx.x) * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) dst[i] = src[i];
}

// rows[pos[r], :] = emb[r, :] (fp32 source): input-refit embeddings from plugins.
__global__ void refit_rows_kernel(bf16* __restrict__ hidden, const int* __restrict__ pos, const float* __restrict__ emb,
                                  int H) {
  const float* src = emb + static_cast<size_t>(blockIdx.x) * H;
  bf16* dst = hidden + static_cast<size_t>(pos[blockIdx.x]) * H;
  for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] = __float2bfloat16(src[i]);
}

// ----------------------------------------------------------------------------
// RoPE on q and k of the packed qkv activations + append of k, v to the paged
// cache (optionally as fp8 with per-layer scales), one CTA per token.
// qkv row layout: [Hq*D | Hkv*D | Hkv*D]. cos_sin: [max_pos][rot_dim] = cos(rot/2) | sin(rot/2).
// Cache layout per layer: [block][2][Hkv][block_tokens][D] with `block_stride` elements between blocks.
// slot < 0 skips the cache write (padding rows). neox: rotate halves; otherwise rotate pairs.
// positions may carry 3 rows ([3][T]) for multimodal rotary sections (mrope_s0/s1 = section ends in pairs).
template <typename CacheT>
__global__ void rope_kv_append_kernel(bf16* __restrict__ qkv, const int* __restrict__ positions, int pos_stride,
                                      const int* __restrict__ slots, const float* __restrict__ cos_sin,
                                      CacheT* __restrict__ cache, long long block_stride, int block_tokens, int Hq,
                                      int Hkv, int D, int rot_dim, int neox, int mrope_s0, int mrope_s1,
                                      float k_scale_inv, float v_scale_inv, int apply_rope) {
  const int t = blockIdx.x;
  bf16* row = qkv + static_cast<size_t>(t) * (Hq + 2 * Hkv) * D;
  const int half = rot_dim >> 1;
  if (apply_rope) {
    const int nrot = (Hq + Hkv) * half;
    for (int i = threadIdx.x; i < nrot; i += blockDim.x) {
      const int h = i / half, j = i % half;
      int pos = positions[t];
      if (pos_stride) {   // multimodal: pair index selects the temporal / height / width position row
        const int sec = j < mrope_s0 ? 0 : (j < mrope_s1 ? 1 : 2);
        pos = positions[sec * pos_stride + t];
      }
      const float* cs = cos_sin + static_cast<size_t>(pos) * rot_dim;
      const float c = cs[j], s = cs[half + j];
      bf16* hp = row + static_cast<size_t>(h) * D;
      const int i0 = neox ? j : 2 * j, i1 = neox ? j + half : 2 * j + 1;
      const float x0 = __bfloat162float(hp[i0]), x1 = __bfloat162float(hp[i1]);
      hp[i0] = __float2bfloat16(x0 * c - x1 * s);
      hp[i1] = __float2bfloat16(x1 * c + x0 * s);
    }
    __syncthreads();
  }
  const int slot = slots[t];
  if (slot < 0 || cache == nullptr) return;
  const int blk = slot / block_tokens, off = slot % block_tokens;
  CacheT* kbase = cache + static_cast<size_t>(blk) * block_stride;
  const bf16* ksrc = row + static_cast<size_t>(Hq) * D;
  const int n = Hkv * D;
  for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) {
    const int kv = i / n, r = i % n;
    const int h = r / D, d = r % D;
    const float val = __bfloat162float(ksrc[i]);
    const size_t dst = ((static_cast<size_t>(kv) * Hkv + h) * block_tokens + off) * D + d;
    if constexpr (sizeof(CacheT) == 1) {
      kbase[dst] = static_cast<CacheT>(
          __nv_cvt_float_to_fp8(val * (kv ? v_scale_inv : k_scale_inv), __NV_SATFINITE, __NV_E4M3));
    } else {
      kbase[dst] = ksrc[i];
    }
  }
}

// Vector form of the kernel above for the common case (rotate halves over the whole head, one position row):
// a thread rotates 8 pairs with two 16-byte loads / stores, and what it holds of a key goes on to the cache; values are copied the same way.
// (Keys written back, waited for and read again: 8000 rows of 80 heads 67.6 us, now 64.8.)
template <typename CacheT>
__global__ void rope_kv_append_vec_kernel(bf16* __restrict__ qkv, const int* __restrict__ positions,
                                          const int* __restrict__ slots, const float* __restrict__ cos_sin,
                                          CacheT* __restrict__ cache, long long block_stride, int block_tokens, int Hq,
                                          int Hkv, int D, float k_scale_inv, float v_scale_inv, int apply_rope) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  bf16* row = qkv + static_cast<size_t>(t) * (Hq + 2 * Hkv) * D;
  const int half = D >> 1, hv = half >> 3;                   // 16-byte vectors per half head
  const int slot = slots[t];
  const bool keep = slot >= 0 && cache != nullptr;
  const int blk = keep ? slot / block_tokens : 0, off = keep ? slot - blk * block_tokens : 0;
  CacheT* kbase = cache + static_cast<size_t>(blk) * block_stride;
  auto to_cache = [&](int kv, int h, int d, const uint4& v) {
    const size_t dst = ((static_cast<size_t>(kv) * Hkv + h) * block_tokens + off) * D + d;
    if constexpr (sizeof(CacheT) == 1) {
      float f[8];
      unpack8(v, f);
      *reinterpret_cast<uint2*>(kbase + dst) = pack8_e4m3(f, kv ? v_scale_inv : k_scale_inv);
    } else {
      *reinterpret_cast<uint4*>(kbase + dst) = v;
    }
  };
  // queries and keys: two halves of a head at a time, keys on to the cache from registers; then the values, copied
  const float* cs = apply_rope ? cos_sin + static_cast<size_t>(positions[t]) * D : nullptr;
  const int first = apply_rope ? 0 : Hq * hv, turned = (Hq + Hkv) * hv, items = turned + Hkv * hv;
  for (int i = first + threadIdx.x; i < items; i += blockDim.x) {
    const int h = i / hv, j0 = (i - h * hv) << 3;
    if (h >= Hq && !keep && (h >= Hq + Hkv || !apply_rope)) continue;
    bf16* hp = row + static_cast<size_t>(h) * D;
    uint4 a = *reinterpret_cast<const uint4*>(hp + j0), b = *reinterpret_cast<const uint4*>(hp + half + j0);
    if (apply_rope && i < turned) {
      float x0[8], x1[8], c[8], sn[8], y0[8], y1[8];
      unpack8(a, x0);
      unpack8(b, x1);
      *reinterpret_cast<float4*>(&c[0]) = *reinterpret_cast<const float4*>(cs + j0);
      *reinterpret_cast<float4*>(&c[4]) = *reinterpret_cast<const float4*>(cs + j0 + 4);
      *reinterpret_cast<float4*>(&sn[0]) = *reinterpret_cast<const float4*>(cs + half + j0);
      *reinterpret_cast<float4*>(&sn[4]) = *reinterpret_cast<const float4*>(cs + half + j0 + 4);
#pragma unroll
      for (int e = 0; e < 8; ++e) { y0[e] = x0[e] * c[e] - x1[e] * sn[e]; y1[e] = x1[e] * c[e] + x0[e] * sn[e]; }
      a = pack8(y0);
      b = pack8(y1);
      *reinterpret_cast<uint4*>(hp + j0) = a;
      *reinterpret_cast<uint4*>(hp + half + j0) = b;
    }
    if (h >= Hq && keep) {
      const int kv = h >= Hq + Hkv;
      to_cache(kv, h - Hq - (kv ? Hkv : 0), j0, a);
      to_cache(kv, h - Hq - (kv ? Hkv : 0), half + j0, b);
    }
  }
}

// Block-to-block copy inside the paged cache (beam fork, flexible cache, swap staging):
// pairs[2*i] = source block, pairs[2*i+1] = destination block; copies all layers of a block.
// A block id outside [0, num_blocks) is recorded in the error word and its copy is skipped.
__global__ void copy_blocks_kernel(uint4* __restrict__ cache, const int* __restrict__ pairs, long long block_vec,
                                   int num_blocks, int* err) {
  const int sb = pairs[2 * blockIdx.x], db = pairs[2 * blockIdx.x + 1];
  if (sb < 0 || sb >= num_blocks || db < 0 || db >= num_blocks) {
    if (threadIdx.x == 0 && blockIdx.y == 0) guard_report(err, kGuardBlockId, (sb < 0 || sb >= num_blocks) ? sb : db);
    return;
  }
  const uint4* src = cache + static_cast<size_t>(sb) * block_vec;
  uint4* dst = cache + static_cast<size_t>(db) * block_vec;
  for (long long i = blockIdx.y * static_cast<long long>(blockDim.x) + threadIdx.x; i < block_vec;
       i += static_cast<long long>(gridDim.y) * blockDim.x)
    dst[i] = src[i];
}

// Whole cache blocks between the device cache and a pool of host blocks in pinned (device-visible) host memory:
// pairs[2*i] = device block, pairs[2*i+1] = host block; dir 0: cache -> host pool, 1: host pool -> cache. One launch
// per swap list; the kernel moves the bytes over PCIe itself, so no staging copy and no host synchronisation is
// needed. Ids outside their pools are recorded in the error word and skipped.
__global__ void swap_blocks_kernel(uint4* __restrict__ cache, uint4* __restrict__ pool, const int* __restrict__ pairs,
                                   long long block_vec, int dir, int num_blocks, int num_pool_blocks, int* err) {
  const int b = pairs[2 * blockIdx.x], hb = pairs[2 * blockIdx.x + 1];
  if (b < 0 || b >= num_blocks || hb < 0 || hb >= num_pool_blocks) {
    if (threadIdx.x == 0 && blockIdx.y == 0) guard_report(err, kGuardBlockId, (b < 0 || b >= num_blocks) ? b : hb);
    return;
  }
  uint4* c = cache + static_cast<size_t>(b) * block_vec;
  uint4* s = pool + static_cast<size_t>(hb) * block_vec;
  for (long long i = blockIdx.y * static_cast<long long>(blockDim.x) + threadIdx.x; i < block_vec;
       i += static_cast<long long>(gridDim.y) * blockDim.x) {
    if (dir == 0) s[i] = c[i]; else c[i] = s[i];
  }
}

// Flexible-cache copies land at another position of the sequence: the K rows of the destination block are rotated by
// the position delta (rotary rotations add, so one rotation by |delta| with the sign on the sine does it), in place,
// for every layer and KV head of the block. triples[3*i] = source block (unused here), [3*i+1] = destination block,
// [3*i+2] = position delta. Cache layout [blocks][layers][2][kv heads][block tokens][head dim], K panel first;
// cos_sin [max_pos][rot_dim] = cos | sin (fp32). FP8 caches are rotated on their raw values (the tensor scale is
// a common factor). Bad block ids and deltas beyond the table are recorded in the error word and skipped.
template <typename T>
__device__ __forceinline__ float kv_to_float(T v);
template <> __device__ __forceinline__ float kv_to_float<bf16>(bf16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float kv_to_float<uint8_t>(uint8_t v) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw(v, __NV_E4M3)));
}
template <typename T>
__device__ __forceinline__ T kv_from_float(float v);
template <> __device__ __forceinline__ bf16 kv_from_float<bf16>(float v) { return __float2bfloat16(v); }
template <> __device__ __forceinline__ uint8_t kv_from_float<uint8_t>(float v) {
  return __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

template <typename T>
__global__ void rerotate_blocks_kernel(T* __restrict__ cache, const int* __restrict__ triples, const float* __restrict__ cos_sin,
                                       int max_pos, int layers, int hkv, int bt, int D, int rot_dim, int neox,
                                       int num_blocks, long long rec_stride, int* err) {
  const int db = triples[3 * blockIdx.x + 1], delta = triples[3 * blockIdx.x + 2];
  if (delta == 0) return;
  const int ad = delta < 0 ? -delta : delta;
  if (db < 0 || db >= num_blocks || ad >= max_pos) {
    if (threadIdx.x == 0 && blockIdx.y == 0) guard_report(err, db < 0 || db >= num_blocks ? kGuardBlockId : kGuardPosition,
                                                          db < 0 || db >= num_blocks ? db : ad);
    return;
  }
  const int half = rot_dim >> 1;
  const float* cs = cos_sin + static_cast<size_t>(ad) * rot_dim;
  const float sgn = delta > 0 ? 1.f : -1.f;
  const long long panel = static_cast<long long>(bt) * D;                 // one head's K panel
  const long long layer_stride = 2LL * hkv * panel, block_stride = rec_stride > 0 ? rec_stride : layers * layer_stride;
  T* blk = cache + static_cast<size_t>(db) * block_stride;
  const long long pairs = static_cast<long long>(layers) * hkv * bt * half;
  for (long long i = blockIdx.y * static_cast<long long>(blockDim.x) + threadIdx.x; i < pairs;
       i += static_cast<long long>(gridDim.y) * blockDim.x) {
    const int j = static_cast<int>(i % half);
    long long t = i / half;
    const int tok = static_cast<int>(t % bt); t /= bt;
    const int head = static_cast<int>(t % hkv);
    const int layer = static_cast<int>(t / hkv);
    T* row = blk + layer * layer_stride + head * panel + static_cast<long long>(tok) * D;
    const int i0 = neox ? j : 2 * j, i1 = neox ? j + half : 2 * j + 1;
    const float c = cs[j], sn = cs[half + j] * sgn;
    const float x0 = kv_to_float<T>(row[i0]), x1 = kv_to_float<T>(row[i1]);
    row[i0] = kv_from_float<T>(x0 * c - x1 * sn);
    row[i1] = kv_from_float<T>(x1 * c + x0 * sn);
  }
}

// Largest magnitude of a bf16 matrix as a quantisation scale on the device: scale = max(|x|) / divisor (at least
// `floor`), without a host round trip and without a widened copy of x. Every CTA leaves its own maximum in `parts`, which the
// finishing kernel reads: scratch of one call, so that calls on several streams have nothing in common.
__global__ void __launch_bounds__(256) absmax_kernel(const bf16* __restrict__ x, int rows, int cols, long long ldx, float* parts) {
  const int vec_per_row = cols >> 3;
  const long long nvec = static_cast<long long>(rows) * vec_per_row;
  float m = 0.f;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = static_cast<int>(i - r * vec_per_row);
    const uint4 v = *reinterpret_cast<const uint4*>(x + r * ldx + c * 8);
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(p[k]);
      m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  publish_absmax(m, parts);
}
// The same in chunks of 16 elements, four in flight a thread, maxima on packed pairs (by: chunks of a row): 9753 x 14336 53 -> 44 us, x 4096 19.8 -> 16.5.
__global__ void __launch_bounds__(256) absmax_chunks_kernel(const bf16* __restrict__ x, uint32_t total, FastDiv by, long long ldx, float* parts) {
  const uint32_t step = gridDim.x * blockDim.x;
  __nv_bfloat162 m = __floats2bfloat162_rn(0.f, 0.f);
  for (uint32_t base = blockIdx.x * blockDim.x + threadIdx.x; base < total; base += 4 * step) {
    Chunk16 c[4] = {};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t i = base + k * step;
      if (i < total) {
        const uint32_t r = by.div(i);
        c[k] = ld_chunk(x + r * ldx + (i - r * by.d) * 16);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) m = chunk_absmax(c[k], m);
  }
  publish_absmax(larger(m), parts);
}
// One CTA: n maxima to the scale. (One thread that read one word took as long as the 1184 values of a full launch do here, about 2 us.)
__global__ void absmax_finish_kernel(const float* __restrict__ parts, int n, float* scale, float inv_divisor, float floor_value) {
  __shared__ float red[32];
  float m = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, parts[i]);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = warp_max(threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f);
    if (threadIdx.x == 0) *scale = fmaxf(m * inv_divisor, floor_value);
  }
}

// ids[rows[i]] = prev_tokens[src[i]]: a pipelined step takes the input ids of its decode rows straight from the
// previous step's sampler output on the device (the host has not read those tokens yet).
__global__ void patch_ids_kernel(int* __restrict__ ids, const int* __restrict__ rows, const int* __restrict__ src,
                                 const int* __restrict__ prev_tokens, int n, int n_ids, int n_prev, int* err) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], sidx = src[i];
  if (r < 0 || r >= n_ids || sidx < 0 || sidx >= n_prev) { guard_report(err, kGuardGatherRow, r < 0 || r >= n_ids ? r : sidx); return; }
  ids[r] = prev_tokens[sidx];
}

// out = a + b (+ bias), bf16 (used for unfused residual paths and the baseline backend)
__global__ void add_kernel(const bf16* __restrict__ a, const bf16* __restrict__ b, const bf16* __restrict__ bias,
                           bf16* __restrict__ out, long long nvec_total, int nvec_row) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nvec_total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8], y[8];
    unpack8(reinterpret_cast<const uint4*>(a)[i], x);
    if (b) {
      unpack8(reinterpret_cast<const uint4*>(b)[i], y);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] += y[e];
    }
    if (bias) {
      unpack8(reinterpret_cast<const uint4*>(bias)[i % nvec_row], y);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] += y[e];
    }
    reinterpret_cast<uint4*>(out)[i] = pack8(x);
  }
}

// bf16 -> fp32 cast of selected rows (logits for the sampler when the GEMM wrote bf16)
__global__ void cast_f32_kernel(const bf16* __restrict__ in, float* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    out[i] = __bfloat162float(in[i]);
}

static inline int grid_for(long long work, int threads, int cap = 148 * 8) {
  long long g = (work + threads - 1) / threads;
  if (g < 1) g = 1;
  return static_cast<int>(g > cap ? cap : g);
}
// 16-byte vectors per thread of the activation and quantisation kernels: one while all threads are resident at once (300 x 7168 quantised: 2.5
// us with one, 3.2 with two, 4.0 with four) and for gated inputs, which have two loads in flight anyway (9000 x 14336 gated and quantised
// 112 / 123 / 114 us); else two (9000 x 14336 quantised 73 / 70 / 81 us, activation without a gate 95.7 / 94 / 97).
static inline int launch_vectors(long long total, bool gated) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return gated || total <= sms * 2048LL ? 1 : 2;
}
// launches of more 16-byte vectors than threads fit the machine at once (or than `per_sm` for every SM)
static inline bool chunks_pay(long long total, int per_sm = 2048) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return total > static_cast<long long>(sms) * per_sm;
}
static inline int norm_threads(int H) {
  int t = ((H >> 3) + kMaxVec - 1) / kMaxVec;
  t = ((t + 31) / 32) * 32;
  if (t < 32) t = 32;
  return t > 1024 ? 1024 : t;
}

// ----------------------------------------------------------------------------
// NVFP4 quantisation of GEMM inputs: 16-element blocks along K, e2m1 values (two per byte, even element in the
// low nibble), one e4m3 scale per block, one fp32 scale per tensor (given): x ~= e2m1 * block_scale * tensor_scale.
// (row and block by multiplication: the two 64-bit divisions a block took a few percent: 9753 x 14336 73 -> 71.7 us)
__global__ void quant_nvfp4_kernel(const bf16* __restrict__ x, int ldx, uint8_t* __restrict__ q, int ldq,
                                   uint8_t* __restrict__ bs, int ldbs, const float* __restrict__ ts, uint32_t total, FastDiv by) {
  const float inv_ts = 1.f / (ts ? *ts : 1.f);
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t row = by.div(idx), b = idx - row * by.d;
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * ldx + b * 16);
    float f[16];
    unpack8(src[0], *reinterpret_cast<float(*)[8]>(&f[0]));
    unpack8(src[1], *reinterpret_cast<float(*)[8]>(&f[8]));
    float am = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) { f[i] *= inv_ts; am = fmaxf(am, fabsf(f[i])); }
    const __nv_fp8_storage_t sc8 = __nv_cvt_float_to_fp8(fminf(am / 6.f, 448.f), __NV_SATFINITE, __NV_E4M3);
    const float scf = fmaxf(__half2float(__half(__nv_cvt_fp8_to_halfraw(sc8, __NV_E4M3))), 1.f / 512.f);
    uint32_t w[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_fp4x2_storage_t v = __nv_cvt_float2_to_fp4x2(make_float2(f[2 * i] / scf, f[2 * i + 1] / scf), __NV_E2M1,
                                                              cudaRoundNearest);
      w[i >> 2] |= static_cast<uint32_t>(v) << (8 * (i & 3));
    }
    *reinterpret_cast<uint2*>(q + static_cast<size_t>(row) * ldq + b * 8) = make_uint2(w[0], w[1]);
    bs[static_cast<size_t>(row) * ldbs + b] = sc8;
  }
}

}  // namespace ksana

using namespace ksana;

// parts (may be null, nparts places): also the largest magnitude of y by CTA, nparts becoming their number; -100 where the kernel that does
// that does not take the call.
static int norm_impl(const void* x, void* residual, const void* w, const void* beta, void* y, void* yq,
                     float* yscale, int scale_ld, int M, int H, float eps, int layernorm, float* parts, int* nparts, cudaStream_t st) {
  if (M <= 0 || H == 0) return 0;
  if (H < 0 || H % 8 || H > 8 * kMaxVec * 1024) return -10;
  if (yq && (H % 128)) return -11;
  // plain root-mean-square norm of aligned rows: the kernel whose CTAs stay (one row has half the barriers and wider loads: 1 x 4096 3.6 -> 2.4 us)
  if (!layernorm && !residual && !beta && H % 16 == 0 && H <= 16384 &&
      !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(yq)) & 31)) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int chunks = H / 16, v = chunks <= 256 ? 1 : chunks <= 512 ? 2 : 4;
    const int threads = ((chunks + v - 1) / v + 31) / 32 * 32, per_sm = (v == 1 ? 4 : v == 2 ? 3 : 2) * (256 / threads > 1 ? 256 / threads : 1);
    int ctas = M < sms * per_sm ? M : sms * per_sm;
    if (parts) *nparts = ctas = ctas < *nparts ? ctas : *nparts;
    const dim3 grid(ctas);
#define KSANA_NORM_ROWS(Q, V, A) launch_early(norm_rows_kernel<Q, V, A>, grid, dim3(threads), 0, st, (const bf16*)x, (const bf16*)w, (bf16*)y, \
                                              (uint8_t*)yq, yscale, scale_ld, M, H, eps, parts)
    if (parts) v == 1 ? KSANA_NORM_ROWS(false, 1, true) : v == 2 ? KSANA_NORM_ROWS(false, 2, true) : KSANA_NORM_ROWS(false, 4, true);
    else if (yq) v == 1 ? KSANA_NORM_ROWS(true, 1, false) : v == 2 ? KSANA_NORM_ROWS(true, 2, false) : KSANA_NORM_ROWS(true, 4, false);
    else v == 1 ? KSANA_NORM_ROWS(false, 1, false) : v == 2 ? KSANA_NORM_ROWS(false, 2, false) : KSANA_NORM_ROWS(false, 4, false);
#undef KSANA_NORM_ROWS
    return cudaGetLastError() == cudaSuccess ? 0 : -4;
  }
  if (parts) return -100;
  const int threads = norm_threads(H);
#define KSANA_NORM(MODE, RES, Q) launch_early(norm_kernel<MODE, RES, Q>, dim3(M), dim3(threads), 0, st, (const bf16*)x, (bf16*)residual, \
                                              (const bf16*)w, (const bf16*)beta, (bf16*)y, (uint8_t*)yq, yscale, scale_ld, H, eps)
#define KSANA_NORM_Q(MODE, RES) (yq ? KSANA_NORM(MODE, RES, true) : KSANA_NORM(MODE, RES, false))
  if (layernorm) residual ? KSANA_NORM_Q(1, true) : KSANA_NORM_Q(1, false);
  else residual ? KSANA_NORM_Q(0, true) : KSANA_NORM_Q(0, false);
#undef KSANA_NORM_Q
#undef KSANA_NORM
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_norm(const void* x, void* residual, const void* w, const void* beta, void* y, void* yq,
                          float* yscale, int scale_ld, int M, int H, float eps, int layernorm, cudaStream_t st) {
  return norm_impl(x, residual, w, beta, y, yq, yscale, scale_ld, M, H, eps, layernorm, nullptr, nullptr, st);
}

static int finish_absmax(const float* parts, int n, float* scale, float divisor, float floor_value, cudaStream_t st) {
  absmax_finish_kernel<<<1, n > 512 ? 1024 : (n + 31) / 32 * 32, 0, st>>>(parts, n, scale, 1.f / divisor, floor_value);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// y = the root-mean-square norm of x times w, and *scale = max(largest |y| / divisor, floor_value); parts: scratch of this call, nparts > 0
// places. Read again for that, 9753 x 4096 cost 16.5 us and x 14336 44 us; a 4096-wide NVFP4 layer's prefill of 9753 rows with head 2276 ->
// 2231 us. -100: not covered (rows off 32-byte boundaries, H no multiple of 16 or above 16384): norm and largest magnitude one after the
// other do it.
extern "C" int ksana_norm_absmax(const void* x, const void* w, void* y, int M, int H, float eps, float divisor, float floor_value, float* parts,
                                 int nparts, float* scale, cudaStream_t st) {
  if (M <= 0 || divisor <= 0.f || !parts || nparts <= 0 || !scale) return -10;
  if (H <= 0) return -100;
  const int rc = norm_impl(x, nullptr, w, nullptr, y, nullptr, nullptr, 0, M, H, eps, 0, parts, &nparts, st);
  return rc ? rc : finish_absmax(parts, nparts, scale, divisor, floor_value, st);
}

// out = act(gate) * up of packed rows and the scale of its largest magnitude, as above. -100: not covered (small launches, no whole chunks).
extern "C" int ksana_act_mul_absmax(const void* in, void* out, int M, int I, int in_ld, int act, float divisor, float floor_value, float* parts,
                                    int nparts, float* scale, cudaStream_t st) {
  if (M <= 0 || divisor <= 0.f || !parts || nparts <= 0 || !scale) return -10;
  const long long total = static_cast<long long>(M) * (I >> 3);
  if (I % 16 || in_ld % 16 || !chunks_pay(total) || total >= (1LL << 31) || ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 31))
    return -100;
  const FastDiv by = make_fast_div(I / 16);
  const dim3 grid(grid_for(total / 2, 256, nparts < 148 * 8 ? nparts : 148 * 8));
#define KSANA_ACT_AMAX(A) launch_early(act_chunks_kernel<A, false, true>, grid, dim3(256), 0, st, (const bf16*)in, (bf16*)out, \
                                       static_cast<uint8_t*>(nullptr), static_cast<float*>(nullptr), 0, static_cast<uint32_t>(total / 2), by, in_ld, \
                                       static_cast<const int*>(nullptr), parts)
  if (act == 0) KSANA_ACT_AMAX(0);
  else if (act == 1) KSANA_ACT_AMAX(1);
  else KSANA_ACT_AMAX(2);
#undef KSANA_ACT_AMAX
  return finish_absmax(parts, grid.x, scale, divisor, floor_value, st);
}

extern "C" int ksana_act_mul(const void* in, void* out, void* outq, float* oscale, int scale_ld, int M, int I,
                             int in_ld, int act, int gated, const int* tile_rows, cudaStream_t st) {
  if (M <= 0 || I == 0) return 0;
  if (I < 0 || I % 8 || in_ld % 8) return -10;
  if (outq && (I % 128)) return -11;
  if (act < 0 || act > 2) act = 2;
  // flat indices stay below 2^31: larger inputs go in row ranges (multiples of 128 rows, as tile_rows counts them)
  const int nvec = I >> 3;
  const FastDiv div = make_fast_div(nvec);
  int most = static_cast<int>(((1LL << 31) - 1) / nvec);
  if (most > 128) most -= most % 128;
  for (int m0 = 0; m0 < M; m0 += most) {
    const int rows = M - m0 < most ? M - m0 : most;
    const uint32_t total = static_cast<uint32_t>(rows) * nvec;
    const bf16* src = (const bf16*)in + static_cast<size_t>(m0) * in_ld;
    bf16* dst = out ? (bf16*)out + static_cast<size_t>(m0) * I : nullptr;
    uint8_t* dq = outq ? (uint8_t*)outq + static_cast<size_t>(m0) * I : nullptr;
    float* ds = oscale ? oscale + m0 : nullptr;
    const int* tr = tile_rows ? tile_rows + m0 / 128 : nullptr;
    // Half as many threads with twice the work each gain where there are enough of them. us, vectors / chunks, on 148 SMs: not quantised
    // 307200 vectors 2.4 / 2.8 (gelu 2.9 / 3.6), 409600 2.9 / 3.0 (3.7 / 3.9), 465920 3.1 / 3.0 (4.0 / 3.9), 537600 3.5 / 3.0; quantised
    // 307200 3.2 / 3.2 (gelu 3.75 / 4.2), 332800 3.5 / 3.3 (4.1 / 4.3), 358400 3.8 / 3.3 (4.5 / 4.4).
    if (chunks_pay(total, !dq ? 3200 : act == 1 ? 2368 : 2048) && gated && I % 16 == 0 && in_ld % 16 == 0 &&
        !((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(dq)) & 31)) {
      const FastDiv by = make_fast_div(I / 16);
      const dim3 chunk_grid(grid_for(total / 2, 256));
#define KSANA_ACT16(A, Q) launch_early(act_chunks_kernel<A, Q, false>, chunk_grid, dim3(256), 0, st, src, dst, dq, ds, scale_ld, total / 2, by, in_ld, tr, \
                                          static_cast<float*>(nullptr))
      if (act == 0) dq ? KSANA_ACT16(0, true) : KSANA_ACT16(0, false);
      else if (act == 1) dq ? KSANA_ACT16(1, true) : KSANA_ACT16(1, false);
      else dq ? KSANA_ACT16(2, true) : KSANA_ACT16(2, false);
#undef KSANA_ACT16
      continue;
    }
    const int v = launch_vectors(total, gated);
    const dim3 grid(grid_for((static_cast<long long>(total) + v - 1) / v, 256));
#define KSANA_ACT(A, G, Q, V) launch_early(act_mul_kernel<A, G, Q, V>, grid, dim3(256), 0, st, src, dst, dq, ds, scale_ld, total, div, in_ld, tr)
#define KSANA_ACT_V(A, Q) (v == 1 ? KSANA_ACT(A, false, Q, 1) : KSANA_ACT(A, false, Q, 2))
#define KSANA_ACT_G(A) (gated ? (outq ? KSANA_ACT(A, true, true, 1) : KSANA_ACT(A, true, false, 1)) \
                              : (outq ? KSANA_ACT_V(A, true) : KSANA_ACT_V(A, false)))
    if (act == 0) KSANA_ACT_G(0);
    else if (act == 1) KSANA_ACT_G(1);
    else KSANA_ACT_G(2);
#undef KSANA_ACT_G
#undef KSANA_ACT_V
#undef KSANA_ACT
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_act_mul_f32(const float* in, float* out, int M, int I, int in_ld, int act, int gated, cudaStream_t st) {
  if (M <= 0 || I <= 0) return 0;
  if (in_ld < I * (gated ? 2 : 1) || act < 0 || act > 2) return -10;
  return launch_pdl(act_mul_f32_kernel, dim3(grid_for(static_cast<long long>(M) * I, 256)), dim3(256), 0, st, in, out, M, I, in_ld, act,
                    gated) == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_quant_fp8(const void* x, void* q, float* scale, int scale_ld, int M, int K, int x_ld,
                               cudaStream_t st) {
  if (M <= 0 || K == 0) return 0;
  if (K < 0 || K % 128 || x_ld % 8) return -10;
  const int nvec = K >> 3;
  const FastDiv div = make_fast_div(nvec);
  const int most = static_cast<int>(((1LL << 31) - 1) / nvec);
  for (int m0 = 0; m0 < M; m0 += most) {
    const int rows = M - m0 < most ? M - m0 : most;
    const uint32_t total = static_cast<uint32_t>(rows) * nvec;
    const bf16* src = (const bf16*)x + static_cast<size_t>(m0) * x_ld;
    uint8_t* dst = (uint8_t*)q + static_cast<size_t>(m0) * K;
    if (chunks_pay(total) && x_ld % 16 == 0 && !((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 31)) {
      launch_early(quant_chunks_kernel, dim3(grid_for(total / 2, 256)), dim3(256), 0, st, src, dst, scale + m0, scale_ld, total / 2,
                   make_fast_div(K / 16), x_ld);
      continue;
    }
    const int v = launch_vectors(total, false);
    launch_early(v == 1 ? quant_fp8_kernel<1> : quant_fp8_kernel<2>, dim3(grid_for((static_cast<long long>(total) + v - 1) / v, 256)), dim3(256), 0,
                 st, (const bf16*)x + static_cast<size_t>(m0) * x_ld, (uint8_t*)q + static_cast<size_t>(m0) * K, scale + m0, scale_ld, total, div,
                 x_ld);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// x [M, K] bf16 -> q [M, K/2] packed e2m1, bs [M, K/16] e4m3 block scales; ts: device fp32 tensor scale (null = 1).
extern "C" int ksana_quant_nvfp4(const void* x, int x_ld, void* q, int q_ld, void* bs, int bs_ld, const float* ts, int M,
                                 int K, cudaStream_t st) {
  if (M <= 0 || K == 0) return 0;
  if (K < 0 || K % 16 || x_ld % 8 || q_ld % 8) return -10;
  const int nb = K >> 4, most = static_cast<int>((1LL << 30) / nb);       // (flat indices stay below 2^31, a step beyond the end included)
  for (int m0 = 0; m0 < M; m0 += most) {
    const uint32_t total = static_cast<uint32_t>(M - m0 < most ? M - m0 : most) * nb;
    quant_nvfp4_kernel<<<grid_for(total, 256), 256, 0, st>>>((const bf16*)x + static_cast<size_t>(m0) * x_ld, x_ld,
                                                             (uint8_t*)q + static_cast<size_t>(m0) * q_ld, q_ld,
                                                             (uint8_t*)bs + static_cast<size_t>(m0) * bs_ld, bs_ld, ts, total,
                                                             make_fast_div(nb));
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_embedding(const int* ids, const void* table, const int* positions, const void* pos_table,
                               void* out, int T, int H, int vocab_lo, int vocab_hi, float scale, cudaStream_t st) {
  if (T <= 0) return 0;
  if (H % 8) return -10;
  launch_early(embedding_kernel, dim3(T), dim3(256), 0, st, ids, (const bf16*)table, positions, (const bf16*)pos_table, (bf16*)out, H,
                                      vocab_lo, vocab_hi, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_gather_rows(const void* in, const int* idx, void* out, int R, int H, int in_rows, int* err,
                                 cudaStream_t st) {
  if (R <= 0) return 0;
  if (H % 8 || in_rows <= 0) return -10;
  launch_pdl(gather_rows_kernel, dim3(R), dim3(256), 0, st, (const bf16*)in, idx, (bf16*)out, H, in_rows, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_refit_rows(void* hidden, const int* pos, const float* emb, int R, int H, cudaStream_t st) {
  if (R <= 0) return 0;
  refit_rows_kernel<<<R, 256, 0, st>>>((bf16*)hidden, pos, emb, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_rope_kv_append(void* qkv, const int* positions, int pos_stride, const int* slots,
                                    const float* cos_sin, void* cache, long long block_stride, int block_tokens, int T,
                                    int Hq, int Hkv, int D, int rot_dim, int neox, int mrope_s0, int mrope_s1,
                                    int cache_fp8, float k_scale, float v_scale, int apply_rope, cudaStream_t st) {
  if (T <= 0 || D == 0 || Hq + 2 * Hkv == 0) return 0;
  if (neox && rot_dim == D && (D % 16) == 0 && pos_stride == 0 && (block_stride % 16) == 0 &&
      (reinterpret_cast<uintptr_t>(qkv) % 16) == 0 && (reinterpret_cast<uintptr_t>(cache) % 16) == 0 &&
      (reinterpret_cast<uintptr_t>(cos_sin) % 16) == 0) {
    // as many threads as leave none idle in the last turn: 48 heads of 128 are 384 items, two turns of 192. Few rows spare themselves a turn
    // that would hold a quarter of the threads: 36 heads, 64 rows 2.5 us in two turns of 160, 2.2 in one of 288 (1000 rows 4.7 / 4.6, but
    // 4000 11.3 / 12.8)
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int items = (Hq + 2 * Hkv) * (D >> 4), full = (items + (T <= 8 * sms ? 191 : 255)) / 256, turns = full > 1 ? full : 1;
    const int threads = ((items + turns - 1) / turns + 31) / 32 * 32;
    if (cache_fp8)
      launch_early(rope_kv_append_vec_kernel<uint8_t>, dim3(T), dim3(threads), 0, st, (bf16*)qkv, positions, slots, cos_sin, (uint8_t*)cache,
                                                            block_stride, block_tokens, Hq, Hkv, D, 1.f / k_scale,
                                                            1.f / v_scale, apply_rope);
    else
      launch_early(rope_kv_append_vec_kernel<bf16>, dim3(T), dim3(threads), 0, st, (bf16*)qkv, positions, slots, cos_sin, (bf16*)cache,
                                                         block_stride, block_tokens, Hq, Hkv, D, 1.f, 1.f, apply_rope);
    return cudaGetLastError() == cudaSuccess ? 0 : -4;
  }
  if (cache_fp8)
    rope_kv_append_kernel<uint8_t><<<T, 256, 0, st>>>((bf16*)qkv, positions, pos_stride, slots, cos_sin,
                                                      (uint8_t*)cache, block_stride, block_tokens, Hq, Hkv, D, rot_dim,
                                                      neox, mrope_s0, mrope_s1, 1.f / k_scale, 1.f / v_scale,
                                                      apply_rope);
  else
    rope_kv_append_kernel<bf16><<<T, 256, 0, st>>>((bf16*)qkv, positions, pos_stride, slots, cos_sin, (bf16*)cache,
                                                   block_stride, block_tokens, Hq, Hkv, D, rot_dim, neox, mrope_s0,
                                                   mrope_s1, 1.f, 1.f, apply_rope);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_copy_blocks(void* cache, const int* pairs, int npairs, long long block_bytes, int num_blocks,
                                 int* err, cudaStream_t st) {
  if (npairs <= 0) return 0;
  if (block_bytes % 16) return -10;
  copy_blocks_kernel<<<dim3(npairs, 16), 256, 0, st>>>((uint4*)cache, pairs, block_bytes / 16, num_blocks, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_swap_blocks(void* cache, void* pool, const int* pairs, int n, long long block_bytes, int dir,
                                 int num_blocks, int num_pool_blocks, int* err, cudaStream_t st) {
  if (n <= 0) return 0;
  if (block_bytes % 16) return -10;
  swap_blocks_kernel<<<dim3(n, 16), 256, 0, st>>>((uint4*)cache, (uint4*)pool, pairs, block_bytes / 16, dir, num_blocks,
                                                  num_pool_blocks, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// kv_bytes: 2 (bf16 cache) or 1 (e4m3 cache). rec_stride: elements between blocks, 0 = a dense
// [blocks][layers][2][kv heads][block tokens][head dim] cache.
extern "C" int ksana_rerotate_blocks(void* cache, const int* triples, int n, const float* cos_sin, int max_pos, int layers,
                                     int hkv, int bt, int D, int rot_dim, int neox, int kv_bytes, int num_blocks,
                                     long long rec_stride, int* err, cudaStream_t st) {
  if (n <= 0) return 0;
  if (rot_dim <= 0 || rot_dim > D || (rot_dim & 1) || (kv_bytes != 1 && kv_bytes != 2)) return -10;
  if (kv_bytes == 2)
    rerotate_blocks_kernel<bf16><<<dim3(n, 8), 256, 0, st>>>((bf16*)cache, triples, cos_sin, max_pos, layers, hkv, bt, D,
                                                            rot_dim, neox, num_blocks, rec_stride, err);
  else
    rerotate_blocks_kernel<uint8_t><<<dim3(n, 8), 256, 0, st>>>((uint8_t*)cache, triples, cos_sin, max_pos, layers, hkv,
                                                                bt, D, rot_dim, neox, num_blocks, rec_stride, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// scale[0] = max(max |x| / divisor, floor) for x [rows, cols] bf16 (row stride ldx, cols a multiple of 8); parts:
// scratch of this call, nparts > 0 places.
extern "C" int ksana_absmax_scale(const void* x, int rows, int cols, long long ldx, float divisor, float floor_value,
                                  float* parts, int nparts, float* scale, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return 0;
  if ((cols % 8) || (ldx % 8) || divisor <= 0.f || !parts || nparts <= 0 || (reinterpret_cast<uintptr_t>(x) & 15)) return -10;
  const long long nvec = static_cast<long long>(rows) * (cols >> 3);
  const int cap = nparts < 148 * 8 ? nparts : 148 * 8;
  int ctas;
  if (cols % 16 == 0 && ldx % 16 == 0 && !(reinterpret_cast<uintptr_t>(x) & 31) && nvec / 2 < (1LL << 30)) {
    ctas = grid_for(nvec / 2, 256, cap);
    absmax_chunks_kernel<<<ctas, 256, 0, st>>>((const bf16*)x, static_cast<uint32_t>(nvec / 2), make_fast_div(cols / 16), ldx, parts);
  } else {
    ctas = grid_for(nvec, 256, cap);
    absmax_kernel<<<ctas, 256, 0, st>>>((const bf16*)x, rows, cols, ldx, parts);
  }
  return finish_absmax(parts, ctas, scale, divisor, floor_value, st);
}

extern "C" int ksana_patch_ids(int* ids, const int* rows, const int* src, const int* prev_tokens, int n, int n_ids,
                               int n_prev, int* err, cudaStream_t st) {
  if (n <= 0) return 0;
  return launch_pdl(patch_ids_kernel, dim3((n + 127) / 128), dim3(128), 0, st, ids, rows, src, prev_tokens, n, n_ids,
                    n_prev, err) == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_add(const void* a, const void* b, const void* bias, void* out, long long M, int H,
                         cudaStream_t st) {
  if (M <= 0) return 0;
  if (H % 8) return -10;
  const long long nvec = M * (H >> 3);
  add_kernel<<<grid_for(nvec, 256), 256, 0, st>>>((const bf16*)a, (const bf16*)b, (const bf16*)bias, (bf16*)out, nvec,
                                                  H >> 3);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int ksana_cast_f32(const void* in, float* out, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  cast_f32_kernel<<<grid_for(n, 256), 256, 0, st>>>((const bf16*)in, out, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
