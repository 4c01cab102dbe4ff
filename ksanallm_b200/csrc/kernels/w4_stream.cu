// Weight-only 4-bit linear layers for decode-sized batches (storage as in w4a16.cu): a weight stream whose packed levels go from
// global memory to the tensor cores through registers alone.
//
//   D[M,N] = X[M,K] * (level * scale - zs)[N,K]^T (+bias)(+residual),  M <= 64, groups of a multiple of 128 along K
//
// Bound by HBM at half a byte per weight once the expansion is cheap. The form before it (gemm_smallm.cu, kind 3) wrote expanded tiles
// to shared memory for tcgen05.mma, and the hand-offs between its expansion warps and the MMA thread set the pace: 65 us for
// 16 x 28672 x 4096 (59 MB), 41 us for 16 x 4096 x 14336. This one takes 34 and 22 us (in CUDA graphs, weights from HBM): a fifth
// of HBM's rate; what is left is the instructions of the expansion and mma.sync's own rate (an eighth of tcgen05's), which is why
// wide layers at more than 32 rows stay with the other kernel (ksana_w4_stream_wins). Here a warp owns 16 features and multiplies with mma.sync:
//   * one 16-byte load per lane and row gives 32 levels; two instructions turn a pair of levels into bf16(128 + level), exactly.
//     mma.sync takes the pairs as they fall out of the packed word, because the activations are staged in the same order;
//   * the sums of a group are scaled in fp32: sum(w x) = scale * sum((128 + level) x) - (zs + 128 scale) * sum(x), with the group's sums of
//     the activations taken when they are staged. The offset of 128 costs the fp32 sums up to 2^-12 of a group's scale * sum|x| (eight
//     steps, sums up to 143 of them); no weight is rounded to bf16, which could cost 2^-6. (An infinite activation makes its row NaN.)
//   * tiles of 128 features are cut along K over the CTAs of a cluster, which add their sums through distributed shared memory.
#include "pdl.cuh"
#include "cluster.cuh"
#include <atomic>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksana {

typedef __nv_bfloat16 bf16;
constexpr int kW4sThreads = 256;
constexpr int kW4sPanelBytes = 32 * 1024;       // activations staged at a time
constexpr int kW4sRedPitch = 132;               // floats between the tokens of the sums in shared memory

struct W4StreamParams {
  const bf16* x; long long ldx;
  const uint8_t* qw; const __half* scale; const __half* zs;
  int ngroups, group_chunks;                    // groups per row, 128-deep chunks per group
  const bf16* bias; const bf16* residual; long long ldr;
  bf16* out; long long ldo;
  int M, N, K, splits, panel_chunks, vec_scales;
};

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_stream16(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// levels q and q + 4 of a packed word as bf16(128 + level): 0x4300 | level
__device__ __forceinline__ uint32_t level_pair(uint32_t w, int q) { return ((w >> (4 * q)) & 0x000f000fu) | 0x43004300u; }

template <int NT>                               // 8-token column tiles per CTA
__global__ void __launch_bounds__(kW4sThreads, NT <= 2 ? 4 : NT == 4 ? 3 : 2)
w4_stream_kernel(const W4StreamParams p) {
  constexpr int MP = NT * 8;
  constexpr int kW4sDepth = 2;    // 128-deep chunks of weights in flight per warp (registers)
  extern __shared__ __align__(16) uint8_t smem_w4[];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int split = static_cast<int>(blockIdx.x) % p.splits, tile = static_cast<int>(blockIdx.x) / p.splits;
  const int m0 = blockIdx.y * MP, rows = min(MP, p.M - m0);
  const int chunks = p.K / 128;
  const int c0 = static_cast<int>(static_cast<long long>(split) * chunks / p.splits);
  const int c1 = static_cast<int>(static_cast<long long>(split + 1) * chunks / p.splits);
  const int pitch = p.panel_chunks * 256 + 64;  // bytes between tokens: eight lanes' 16-byte reads fall on different banks
  uint8_t* xs = smem_w4;
  float* sx = reinterpret_cast<float*>(smem_w4 + MP * pitch);              // [panel chunk][MP] sums of the activations
  float2* sz = reinterpret_cast<float2*>(sx + p.panel_chunks * MP);        // [panel chunk][128 rows] scale, zs + 128 scale

  const int n_lo = min(tile * 128 + warp * 16 + g, p.N - 1), n_hi = min(tile * 128 + warp * 16 + g + 8, p.N - 1);
  const uint8_t* w_lo = p.qw + static_cast<size_t>(n_lo) * (p.K / 2) + t * 16;
  const uint8_t* w_hi = p.qw + static_cast<size_t>(n_hi) * (p.K / 2) + t * 16;
  uint4 lo[kW4sDepth], hi[kW4sDepth];
  auto fetch = [&](int d, int c) {
    if (c < c1) { lo[d] = ld_stream16(w_lo + static_cast<size_t>(c) * 64); hi[d] = ld_stream16(w_hi + static_cast<size_t>(c) * 64); }
  };
#pragma unroll
  for (int d = 0; d < kW4sDepth; ++d) fetch(d, c0 + d);
  pdl_wait();                                   // the weights are never written while the engine runs; the activations are

  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  for (int cp = c0; cp < c1; cp += p.panel_chunks) {
    const int np = min(p.panel_chunks, c1 - cp);
    if (cp != c0) __syncthreads();              // the previous panel is no longer read
    // All loads of a panel are in flight together: taken one by one (each waited for before the next), they took longer than the
    // weights of the whole tile.
    constexpr int kSets = NT <= 2 ? 4 : 8;
    if (p.vec_scales) {                           // eight groups of a row per load, from the octet that holds the panel's first on
      const int o0 = cp >> 3, octets = ((cp + np - 1) >> 3) - o0 + 1;
      for (int i = threadIdx.x; i < octets * 128; i += kW4sThreads) {
        const int row = i & 127, o = o0 + (i >> 7);
        const size_t at = static_cast<size_t>(min(tile * 128 + row, p.N - 1)) * p.ngroups + o * 8;
        const uint4 s4 = __ldg(reinterpret_cast<const uint4*>(p.scale + at)), z4 = __ldg(reinterpret_cast<const uint4*>(p.zs + at));
        const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w}, zw[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float sc = __half2float(__ushort_as_half(static_cast<unsigned short>(sw[e >> 1] >> (16 * (e & 1)))));
          const float zz = __half2float(__ushort_as_half(static_cast<unsigned short>(zw[e >> 1] >> (16 * (e & 1)))));
          const int q = o * 8 + e - cp;
          if (q >= 0 && q < np) sz[q * 128 + row] = make_float2(sc, fmaf(128.f, sc, zz));
        }
      }
    } else {
      for (int i0 = threadIdx.x; i0 < np * 128; i0 += kW4sThreads * kSets) {
        __half sh[kSets], zh[kSets];
#pragma unroll
        for (int k = 0; k < kSets; ++k) {
          const int i = i0 + k * kW4sThreads;
          if (i < np * 128) {
            const size_t at = static_cast<size_t>(min(tile * 128 + (i & 127), p.N - 1)) * p.ngroups + (cp + (i >> 7)) / p.group_chunks;
            sh[k] = p.scale[at];
            zh[k] = p.zs[at];
          }
        }
#pragma unroll
        for (int k = 0; k < kSets; ++k) {
          const int i = i0 + k * kW4sThreads;
          if (i < np * 128) sz[i] = make_float2(__half2float(sh[k]), fmaf(128.f, __half2float(sh[k]), __half2float(zh[k])));
        }
      }
    }
    // 16 lanes take a token's chunk: piece c = 4 t' + j of its 128 activations goes to 4 j + t', its values in the order 0 4 1 5 2 6 3 7
    const int c = threadIdx.x & 15, place = ((c & 3) * 4 + (c >> 2)) * 16;
    for (int i0 = threadIdx.x >> 4; i0 < MP * np; i0 += 16 * kSets) {
      uint4 v[kSets];
#pragma unroll
      for (int k = 0; k < kSets; ++k) {
        const int i = i0 + k * 16, q = i / MP, row = i % MP;                  // MP is a power of two
        v[k] = make_uint4(0, 0, 0, 0);
        if (i < MP * np && row < rows)
          v[k] = *reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(m0 + row) * p.ldx + static_cast<size_t>(cp + q) * 128 + c * 8);
      }
#pragma unroll
      for (int k = 0; k < kSets; ++k) {
        const int i = i0 + k * 16, q = i / MP, row = i % MP;
        const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) s += __uint_as_float(w[e] << 16) + __uint_as_float(w[e] & 0xffff0000u);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (i < MP * np) {
          *reinterpret_cast<uint4*>(xs + row * pitch + q * 256 + place) =
              make_uint4(__byte_perm(w[0], w[2], 0x5410), __byte_perm(w[0], w[2], 0x7632), __byte_perm(w[1], w[3], 0x5410),
                         __byte_perm(w[1], w[3], 0x7632));
          if (c == 0) sx[q * MP + row] = s;
        }
      }
    }
    __syncthreads();
    for (int q0 = 0; q0 < np; q0 += kW4sDepth) {
#pragma unroll
      for (int d = 0; d < kW4sDepth; ++d) {
        const int q = q0 + d;
        if (q >= np) break;
        float sum[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0.f;
        const uint32_t wl[4] = {lo[d].x, lo[d].y, lo[d].z, lo[d].w}, wh[4] = {hi[d].x, hi[d].y, hi[d].z, hi[d].w};
        const uint8_t* xq = xs + g * pitch + q * 256 + t * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t pl[4], ph[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) { pl[e] = level_pair(wl[j], e); ph[e] = level_pair(wh[j], e); }
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint4 v = *reinterpret_cast<const uint4*>(xq + n * 8 * pitch + j * 64);
            mma_bf16_16816(sum[n], pl[0], ph[0], pl[1], ph[1], v.x, v.y);
            mma_bf16_16816(sum[n], pl[2], ph[2], pl[3], ph[3], v.z, v.w);
          }
        }
        fetch(d, cp + q + kW4sDepth);
        const float2 a = sz[q * 128 + warp * 16 + g], b = sz[q * 128 + warp * 16 + g + 8];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float2 s = *reinterpret_cast<const float2*>(sx + q * MP + n * 8 + 2 * t);
          acc[n][0] += a.x * sum[n][0] - a.y * s.x;
          acc[n][1] += a.x * sum[n][1] - a.y * s.y;
          acc[n][2] += b.x * sum[n][2] - b.y * s.x;
          acc[n][3] += b.x * sum[n][3] - b.y * s.y;
        }
      }
    }
  }
  // ---- sums of the cluster's CTAs, in rank order: each CTA finishes its share of the tokens
  __syncthreads();
  float* red = reinterpret_cast<float*>(smem_w4);
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    float* dst = red + (n * 8 + 2 * t) * kW4sRedPitch + warp * 16 + g;
    dst[0] = acc[n][0];
    dst[kW4sRedPitch] = acc[n][1];
    dst[8] = acc[n][2];
    dst[kW4sRedPitch + 8] = acc[n][3];
  }
  if (p.splits > 1) cluster_sync_all(); else __syncthreads();
  const int f = threadIdx.x & 127, n = tile * 128 + f;
  const int tok0 = split * MP / p.splits, tok1 = (split + 1) * MP / p.splits;
  const float bias = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
  for (int k = tok0 + (threadIdx.x >> 7); k < tok1; k += 2) {
    const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(red + k * kW4sRedPitch + f));
    float v = bias;
    if (p.splits > 1) {
      for (int r = 0; r < p.splits; ++r) v += ld_cluster_f32(at, r);
    } else {
      v += red[k * kW4sRedPitch + f];
    }
    if (k < rows && n < p.N) {
      if (p.residual) v += __bfloat162float(p.residual[static_cast<size_t>(m0 + k) * p.ldr + n]);
      p.out[static_cast<size_t>(m0 + k) * p.ldo + n] = __float2bfloat16(v);
    }
  }
  if (p.splits > 1) cluster_sync_all();         // a peer may still read this CTA's sums
}

// Activations staged at a time when a CTA has `per` chunks: its whole share where that fits, else whole turns of the ring of weights in
// registers (multiples of kW4sDepth, four at least).
template <int NT>
static int w4_panel(int per) {
  int fit = kW4sPanelBytes / (NT * 8 * 256);
  fit = fit > 16 ? 16 : fit < 4 ? 4 : fit & ~3;
  return per < fit ? per : fit;
}
template <int NT>
static int w4_smem(int panel) {
  constexpr int MP = NT * 8;
  const int most = MP * (panel * 256 + 64) + panel * (MP * 4 + 128 * 8), red = MP * kW4sRedPitch * 4;
  return most > red ? most : red;
}

constexpr int kW4sSmemLimit = 100 * 1024;
template <int NT>
static bool w4_prepare(int dev) {
  static std::atomic<bool> set[64];
  if (set[dev].load(std::memory_order_acquire)) return true;
  if (cudaFuncSetAttribute(w4_stream_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kW4sSmemLimit) != cudaSuccess) return false;
  set[dev].store(true, std::memory_order_release);
  return true;
}

// Clusters of s CTAs that run at once (they do not fill every group of SMs: 296 CTAs of 64 rows, but 33 clusters of 8).
template <int NT>
static int w4_at_once(int dev, int sms, int s) {
  static std::atomic<int> known[64][9];
  int n = known[dev][s].load(std::memory_order_relaxed);
  if (n) return n;
  if (!w4_prepare<NT>(dev)) return sms / s;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = s; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(s); cfg.blockDim = dim3(kW4sThreads);
  cfg.dynamicSmemBytes = w4_smem<NT>(w4_panel<NT>(16));
  cfg.attrs = &attr; cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, w4_stream_kernel<NT>, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    n = sms / s;
  }
  known[dev][s].store(n, std::memory_order_relaxed);
  return n;
}

// Cuts along K, by powers of two (other clusters leave more SMs empty). Up to 16 rows a CTA is short of work in flight more than of SMs:
// cuts go on while a CTA keeps 2 / 4 / 8 chunks where all CTAs make two per SM / fit at once / do not (us for 1 / 2 / 4 / 8 cuts, 1 row:
// 1024 x 2048 10.3 / 7.2 / 5.8 / 5.1, 15360 x 5120 28.7 / 24.2 / 21.4 / 23.1, 28672 x 4096 32.1 / 31.8 / 27.8 / 33.3, 21912 x 14208 156 /
// 115 / 107 / 72). With more rows the multiplications fill an SM: cuts go on while all CTAs fit at once (32 rows: 8192 x 4096 43.9 / 25.7 /
// 20.0 / 25.6, 27648 x 5120 77 / 57 / 76 / 88; 64 rows: 4096 x 4096 65 / 38 / 21 / 18, 6144 x 4096 65 / 38 / 29 / 32); tiles that do not fit
// uncut are cut to fill the last wave (32 rows, 57344 x 8192: 239 / 205 / 195 / 219).
template <int NT>
static int w4_cuts(int dev, int sms, int tiles, int chunks) {
  int s = 1;
  if (NT <= 2) {
    const int at_once = w4_at_once<NT>(dev, sms, 1);
    for (; s < 8; s *= 2) {
      const int t = 2 * s, ctas = tiles * t;
      if (chunks < (ctas <= 2 * sms ? 2 : ctas <= at_once ? 4 : 8) * t) break;
    }
  } else if (tiles > w4_at_once<NT>(dev, sms, 1)) {
    while (s < 4 && chunks >= 32 * s) s *= 2;
  } else {
    while (s < 8 && tiles <= w4_at_once<NT>(dev, sms, 2 * s) && chunks >= 3 * s) s *= 2;
  }
  return s;
}

template <int NT>
static int launch_w4_stream(W4StreamParams p, int blocks_y, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !w4_prepare<NT>(dev)) return -3;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (p.N + 127) / 128, chunks = p.K / 128;
  p.splits = w4_cuts<NT>(dev, sms, tiles * blocks_y, chunks);
  p.panel_chunks = w4_panel<NT>((chunks + p.splits - 1) / p.splits);
  return launch_cluster(pdl_enabled(), w4_stream_kernel<NT>, dim3(tiles * p.splits, blocks_y), dim3(kW4sThreads), p.splits,
                        w4_smem<NT>(p.panel_chunks), st, p) == cudaSuccess ? 0 : -4;
}

}  // namespace ksana

using namespace ksana;

// Whether this kernel is the faster one for a shape it takes. One or two rows: the CUDA-core kernel needs no staging, which decides
// where there are few short rows (1 row here / there, us: 1024 x 2048 5.1 / 4.0, 4864 x 896 5.4 / 3.9; but 512 x 3584 6.0 / 6.2, 2640 x 5120
// 8.4 / 9.8), and for one row where the scales' rows are no multiple of 4 bytes (8192 x 29568 84 / 71). 33 to 64 rows: a CTA takes 2.05 us a chunk by itself and 3.3 beside
// another on its SM; the stream-K tensor-core kernel about 14 us and 1.6 per chunk and SM, however they are cut (64 rows, us here / there:
// 4096 x 4096 18 / 32, 7168 x 5120 35.5 / 40.5, 4096 x 14336 47 / 53, 8192 x 8192 52.5 / 55.6; 5168 x 11136 73 / 56, 12288 x 4096 48 / 46.5,
// 28672 x 4096 98 / 80).
extern "C" int ksana_w4_stream_wins(int M, int N, int K, int group) {
  const int tiles = (N + 127) / 128, chunks = K / 128;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long all = static_cast<long long>(tiles) * chunks;
  if (M <= 2 && ((K <= 2048 && all <= 2 * sms) || (M == 1 && (K / group) % 2))) return 0;
  if (M <= 32) return 1;
  if (M > 64) return 0;
  const int s = w4_cuts<8>(dev, sms, tiles, chunks), per = (chunks + s - 1) / s, waves = (tiles * s + 2 * sms - 1) / (2 * sms);
  const float here = 4.f + per * (tiles * s <= sms ? 2.05f : 3.3f) * waves, there = 14.f + 1.6f * static_cast<float>(all) / sms;
  return here <= there;
}

// qw [N, K/2] packed levels, scale / zs [N, K/group] fp16; x, out, bias, residual bf16 (out may alias residual). K and group multiples of
// 128, x rows and qw on 16-byte boundaries; returns -10 otherwise. More than 64 rows take several passes over the weights.
extern "C" int ksana_w4_stream(const void* x, long long ldx, const void* qw, const void* scale, const void* zs, const void* bias,
                               const void* residual, long long ldr, void* out, long long ldo, int M, int N, int K, int group,
                               cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 128 || group <= 0 || group % 128 || K % group || ldx % 8) return -10;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(qw)) & 15) return -10;
  W4StreamParams p{};
  p.x = (const bf16*)x; p.ldx = ldx; p.qw = (const uint8_t*)qw; p.scale = (const __half*)scale; p.zs = (const __half*)zs;
  p.ngroups = K / group; p.group_chunks = group / 128;
  p.bias = (const bf16*)bias; p.residual = (const bf16*)residual; p.ldr = ldr; p.out = (bf16*)out; p.ldo = ldo;
  p.M = M; p.N = N; p.K = K;
  const int nt = M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 8;
  p.vec_scales = p.group_chunks == 1 && p.ngroups % 8 == 0 &&
                 !((reinterpret_cast<uintptr_t>(scale) | reinterpret_cast<uintptr_t>(zs)) & 15);
  const int y = (M + nt * 8 - 1) / (nt * 8);
  switch (nt) {
    case 1: return launch_w4_stream<1>(p, y, st);
    case 2: return launch_w4_stream<2>(p, y, st);
    case 4: return launch_w4_stream<4>(p, y, st);
    default: return launch_w4_stream<8>(p, y, st);
  }
}
