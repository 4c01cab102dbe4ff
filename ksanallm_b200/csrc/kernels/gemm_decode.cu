// GEMM of decode steps (up to 64 tokens) on tcgen05 tensor cores, for weights that are read once:
//
//   D[M,N] = X[M,K] * W[N,K]^T (+bias)(+residual)
//
// Operands are swapped as in gemm_smallm.cu: the 128-row MMA dimension carries weight rows, the MMA N dimension the padded tokens.
// Bound by HBM; what a launch costs beside its bytes decides how near it comes. gemm_smallm.cu cuts the (tile, K block) units evenly
// over one persistent CTA per SM and completes cut tiles through global memory: scratch, fences, counters and the wait for all pieces
// took about 7 us of every launch, and its 226 KB of shared memory keep any other kernel off the SM. Here:
//   * a CTA owns one 128-feature tile, or one of S equal shares of its K range; the S CTAs of a tile are a cluster and add their fp32
//     sums through distributed shared memory (one cluster barrier instead of the exchange);
//   * half an SM's shared memory per CTA (up to 165 KB for e4m3 with K in the tens of thousands, whose token exponents are kept there):
//     two share an SM, so that one streams while the other starts or ends, and under
//     programmatic dependent launch the weights of this kernel are on their way while the kernel before it finishes (where the
//     caller says that nothing in flight writes them).
// Against gemm_smallm.cu (us, in graphs): bf16, 1 row, 6144 x 4096 21 -> 12, 4096 x 4096 18 -> 9, 28672 x 4096 50 -> 37, 4096 x 14336
// 30 -> 20; e4m3, 64 rows, 8192 x 8192 29 -> 18, 8192 x 28672 61 -> 52. Wide e4m3 layers at more than 32 rows stay with the tiled
// kernel (57344 x 8192, 64 rows: 86 against 102 us here, where every weight tile is followed by its 8 KB of activations).
// The producer and the MMA warp run their loops as a whole and issue by predicate (a lane behind a branch takes 100 clocks for a copy or an
// MMA, which shows where a share is few K blocks long: bf16, 1 row, 4096 x 4096 9.2 -> 8.45, 6144 x 4096 12.4 -> 11.7; e4m3, 64 rows, 10240 x
// 8192 28.0 -> 26.6).
// Kinds: 0 bf16; 2 e4m3 with power-of-two scales (1 x 128 activations, 128 x 128 weights) applied by the tensor cores. No multicast.
// Every wait is bounded.
#include "sm100_ptx.cuh"
#include "pdl.cuh"
#include "cluster.cuh"
#include <atomic>
#include <cuda_bf16.h>

namespace ksana {

constexpr int kGdSfStages = 4;
constexpr int kGdRedPitch = 132;              // floats between tokens of the sums in shared memory

struct GemmDecodeParams {
  int M, N, K, splits;
  __nv_bfloat16* D; float* out_f32; int ldd;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual; int ldr;
  const float* a_scale; int a_scale_ld;       // [K/128][ld]
  const float* w_scale;                       // [ceil(N/128)][K/128]
  int* err;
};

template <int MP, int KIND>
struct GemmDecodeCfg {
  static constexpr int kThreads = KIND == 2 ? 224 : 192;
  static constexpr int kWBytes = 128 * 128, kXBytes = MP * 128, kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = MP <= 32 ? 5 : 4;
  static constexpr int kElems = KIND == 0 ? 64 : 128;
  static constexpr int kSfBytes = KIND == 2 ? kGdSfStages * 1024 : 0;
  static constexpr int kSfBase = MP;          // TMEM: two sets of 8 scale columns behind the accumulator
  static constexpr int kTmemCols = MP + (KIND == 2 ? 16 : 0) <= 32 ? 32 : MP + (KIND == 2 ? 16 : 0) <= 64 ? 64 : 128;
  static constexpr int kFixedBytes = kStages * kStageBytes + kSfBytes + 1024 + 256;      // + exponents [K blocks][MP] (kind 2)
  static_assert(MP * kGdRedPitch * 4 <= kStages * kStageBytes, "the sums lie over the operand ring");
};

// feature n of B consecutive tokens from m0 on (those below m1): bias and residual added, rounded once
template <int B>
__device__ __forceinline__ void gd_store(const GemmDecodeParams& p, int n, int m0, int m1, float bias, const float (&v)[B]) {
  if (n >= p.N) return;
  float r[B];
#pragma unroll
  for (int i = 0; i < B; ++i)
    r[i] = p.residual && m0 + i < m1 ? __bfloat162float(p.residual[static_cast<size_t>(m0 + i) * p.ldr + n]) : 0.f;
#pragma unroll
  for (int i = 0; i < B; ++i) {
    if (m0 + i >= m1) continue;
    const float o = v[i] + bias + r[i];
    if (p.out_f32) p.out_f32[static_cast<size_t>(m0 + i) * p.ldd + n] = o;
    else p.D[static_cast<size_t>(m0 + i) * p.ldd + n] = __float2bfloat16(o);
  }
}

template <int MP, int KIND>
__global__ void __launch_bounds__(GemmDecodeCfg<MP, KIND>::kThreads, 2)
gemm_decode_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, const GemmDecodeParams p) {
  using Cfg = GemmDecodeCfg<MP, KIND>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sf_smem = smem + Cfg::kStages * Cfg::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_smem + Cfg::kSfBytes);
  uint64_t* empty_bar = full_bar + Cfg::kStages;
  uint64_t* sf_full = empty_bar + Cfg::kStages;
  uint64_t* sf_empty = sf_full + kGdSfStages;
  uint64_t* done_bar = sf_empty + kGdSfStages;
  uint64_t* xs_ready = done_bar + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xs_ready + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  uint8_t* xs_tab = reinterpret_cast<uint8_t*>(full_bar) + 256;              // kind 2: exponents of the tokens, [K block][MP]

  pdl_trigger();
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int S = p.splits, rank = static_cast<int>(blockIdx.x) % S, tile = static_cast<int>(blockIdx.x) / S;
  const int num_kb = (p.K + Cfg::kElems - 1) / Cfg::kElems;
  const int kb0 = rank * num_kb / S, kb1 = (rank + 1) * num_kb / S;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    for (int i = 0; i < kGdSfStages; ++i) { mbar_init(&sf_full[i], 1); mbar_init(&sf_empty[i], 1); }
    mbar_init(done_bar, 1);
    mbar_init(xs_ready, 128);
    *abort_flag = 0;
    mbar_fence_init();
    // the first weight tiles need nothing that an earlier kernel writes: they are requested before anything else happens
    tma_prefetch_desc(&tma_w);
    for (int i = 0; i < Cfg::kStages && kb0 + i < kb1; ++i) {
      mbar_expect_tx(&full_bar[i], Cfg::kStageBytes);
      tma_load_2d(smem + i * Cfg::kStageBytes, &tma_w, &full_bar[i], (kb0 + i) * Cfg::kElems, tile * 128);
    }
  }
  if (warp == 1) { tmem_alloc(tmem_slot, Cfg::kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t lead = elect_one();             // one lane of every warp: it polls and issues for the warp
  pdl_wait();

  float accv[MP];
  bool ok = true;
  if (warp == 0) {
    {
      if (lane == 0) tma_prefetch_desc(&tma_x);
      __syncwarp();
      int stage = 0; uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        uint8_t* sw = smem + stage * Cfg::kStageBytes;
        if (kb - kb0 >= Cfg::kStages) {
          if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, lead, abort_flag)) break;
          mbar_expect_tx_lead(lead, &full_bar[stage], Cfg::kStageBytes);
          tma_load_2d_lead(lead, sw, &tma_w, &full_bar[stage], kb * Cfg::kElems, tile * 128);
        }
        tma_load_2d_lead(lead, sw + Cfg::kWBytes, &tma_x, &full_bar[stage], kb * Cfg::kElems, 0);
        if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    {
      int stage = 0; uint32_t phase = 0;
      if constexpr (KIND == 0) {
        constexpr uint32_t idesc = make_idesc(128, MP, 1, 1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, lead, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + stage * Cfg::kStageBytes);
          const uint64_t wdesc = make_smem_desc_sw128(sw), xdesc = make_smem_desc_sw128(sw + Cfg::kWBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_lead(lead, tmem_base, wdesc + 2 * k, xdesc + 2 * k, idesc, (kb != kb0) || k != 0);
          tc_commit_lead(lead, &empty_bar[stage]);
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
      } else {
        // groups of up to four K blocks share one pair of scale chunks (byte j of a chunk = block g0 + j)
        int sfs = 0; uint32_t sf_phase = 0, set = 0;
        for (int g0 = kb0; g0 < kb1 && ok; g0 += 4) {
          if (!mbar_wait_warp(&sf_full[sfs], sf_phase, lead, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tsfa = tmem_base + Cfg::kSfBase + set * 8, tsfb = tsfa + 4;
          const uint32_t sf_addr = smem_u32(sf_smem + sfs * 1024);
          tmem_cp_sf_lead(lead, tsfa, make_sf_desc(sf_addr));
          tmem_cp_sf_lead(lead, tsfb, make_sf_desc(sf_addr + 512));
          for (int j = 0; j < 4 && g0 + j < kb1; ++j) {
            if (!mbar_wait_warp(&full_bar[stage], phase, lead, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sw = smem_u32(smem + stage * Cfg::kStageBytes);
            const uint64_t wdesc = make_smem_desc_sw128(sw), xdesc = make_smem_desc_sw128(sw + Cfg::kWBytes);
            const uint32_t idesc = make_idesc_mx(128, MP, static_cast<uint32_t>(j));
#pragma unroll
            for (int k = 0; k < 4; ++k)
              mma_mxf8_lead(lead, tmem_base, wdesc + 2 * k, xdesc + 2 * k, idesc, (g0 + j != kb0) || k != 0, tsfa, tsfb);
            tc_commit_lead(lead, &empty_bar[stage]);
            if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
          }
          tc_commit_lead(lead, &sf_empty[sfs]);
          if (++sfs == kGdSfStages) { sfs = 0; sf_phase ^= 1; }
          set ^= 1;
        }
      }
      if (ok) tc_commit_lead(lead, done_bar);
    }
    __syncwarp();
  } else if (warp < 6) {
    // ---- epilogue warps
    const int q = warp & 3;
    if constexpr (KIND == 2) {
      // exponents of the tokens' scales for the K blocks of this share; tokens past M get the neutral one
      const int t = threadIdx.x - 64;
#pragma unroll 4
      for (int i = t; i < (kb1 - kb0) * MP; i += 128) {
        const int kb = i / MP, tok = i % MP;
        xs_tab[i] = tok < p.M ? static_cast<uint8_t>(ue8m0_of(p.a_scale[static_cast<size_t>(kb0 + kb) * p.a_scale_ld + tok])) : 127;
      }
      mbar_arrive(xs_ready);
    }
    ok = mbar_wait_all(done_bar, 0, abort_flag);
    if (ok) {
      tc_fence_after();
      const uint32_t at = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (MP >= 32) {
#pragma unroll
        for (int c = 0; c < MP; c += 32) {
          uint32_t r[32];
          tmem_ld32(at + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) accv[c + i] = __uint_as_float(r[i]);
        }
      } else {
        uint32_t r[16];
        tmem_ld16(at, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) accv[i] = __uint_as_float(r[i]);
      }
      tc_fence_before();
      const int f = q * 32 + lane, n = tile * 128 + f;
      if (S == 1) {
        const float bias = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
#pragma unroll
        for (int m = 0; m < MP; m += 8) {
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = accv[m + i];
          if (m < p.M) gd_store<8>(p, n, m, p.M, bias, v);
        }
      } else {
        // all MMAs have completed and with them all loads: the ring is free
        float* red = reinterpret_cast<float*>(smem);
#pragma unroll
        for (int m = 0; m < MP; ++m) red[m * kGdRedPitch + f] = accv[m];
      }
    }
  } else {
    // ---- scale packer (kind 2)
    if constexpr (KIND == 2) {
      const float* ws = p.w_scale + static_cast<size_t>(tile) * num_kb;
      uint32_t wexp = 127u;                   // exponent of block (wbase + lane)
      int wbase = -1000000, sfs = 0; uint32_t sf_phase = 0;
      wbase = kb0;
      wexp = kb0 + lane < kb1 ? ue8m0_of(ws[kb0 + lane]) : 127u;
      ok = mbar_wait_all(xs_ready, 0, abort_flag);
      for (int g0 = kb0; g0 < kb1 && ok; g0 += 4) {
        if (g0 + 4 > wbase + 32) {
          wbase = g0;
          wexp = g0 + lane < kb1 ? ue8m0_of(ws[g0 + lane]) : 127u;
        }
        uint32_t w0 = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) w0 |= __shfl_sync(0xffffffffu, wexp, g0 - wbase + j) << (8 * j);
        uint32_t w[4];
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          const int tok = r4 * 32 + lane;
          uint32_t word = 0;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            word |= static_cast<uint32_t>(tok < MP && g0 + j < kb1 ? xs_tab[(g0 + j - kb0) * MP + tok] : 127) << (8 * j);
          w[r4] = word;
        }
        if (!mbar_wait_all(&sf_empty[sfs], sf_phase ^ 1, abort_flag)) { ok = false; break; }
        uint8_t* buf = sf_smem + sfs * 1024;
        *reinterpret_cast<uint4*>(buf + lane * 16) = make_uint4(w0, w0, w0, w0);
        *reinterpret_cast<uint4*>(buf + 512 + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sf_full[sfs]);
        if (++sfs == kGdSfStages) { sfs = 0; sf_phase ^= 1; }
      }
    }
  }
  if (S > 1) {
    __syncwarp();
    cluster_sync_all();                        // every share's sums are in its CTA's shared memory
    if (warp >= 2 && warp < 6 && !*abort_flag) {
      const int f = (warp & 3) * 32 + lane, n = tile * 128 + f;
      const int m0 = rank * p.M / S, m1 = (rank + 1) * p.M / S;               // the tokens this CTA finishes
      const float bias = p.bias && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
      const uint32_t base = smem_u32(smem) + f * 4;
      for (int m = m0; m < m1; m += 4) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < S; r += 2) {      // in rank order
          float x[2][4];
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) x[k][i] = r + k < S ? ld_cluster_f32(base + min(m + i, MP - 1) * (kGdRedPitch * 4), r + k) : 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = (v[i] + x[0][i]) + x[1][i];
        }
        gd_store<4>(p, n, m, m1, bias, v);
      }
    }
    __syncwarp();
    cluster_sync_all();                        // a peer may still read this CTA's sums
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 2);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::kTmemCols); }
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*GdEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static GdEncodeFn gd_encode_fn() {
  static GdEncodeFn fn = []() -> GdEncodeFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<GdEncodeFn>(ptr);
  }();
  return fn;
}
static bool gd_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int esz, int box_rows) {
  GdEncodeFn enc = gd_encode_fn();
  if (!enc) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * esz};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / esz), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  return enc(map, esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides,
             box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MP, int KIND>
static int launch_gemm_decode(const CUtensorMap& mw, const CUtensorMap& mx, const GemmDecodeParams& p, bool early, cudaStream_t st) {
  using Cfg = GemmDecodeCfg<MP, KIND>;
  const int num_kb = (p.K + Cfg::kElems - 1) / Cfg::kElems;
  const int smem = Cfg::kFixedBytes + (KIND == 2 ? ((num_kb + p.splits - 1) / p.splits) * MP : 0);
  if (smem > 226 * 1024) return -22;
  static std::atomic<bool> set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -3;
  if (!set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(gemm_decode_kernel<MP, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) return -3;
    set[dev].store(true, std::memory_order_release);
  }
  return launch_cluster(early && pdl_early_enabled(), gemm_decode_kernel<MP, KIND>, dim3(((p.N + 127) / 128) * p.splits),
                        dim3(Cfg::kThreads), p.splits, smem, st, mw, mx, p) == cudaSuccess ? 0 : -4;
}

}  // namespace ksana

using namespace ksana;

// kind 0: X [M,K], W [N,K] bf16, K a multiple of 8. kind 2: e4m3 with power-of-two scales, K a multiple of 128. Output bf16 (D) or fp32
// (out_f32); residual may alias D. fixed_w: no work in flight writes W. The first weight tiles are requested before the kernel ahead has
// been waited for, so only then may this one be launched early; W made by an earlier kernel of the stream takes an ordinary launch.
// -20: more than 64 rows; -22: K too long for one launch (kind 2).
extern "C" int ksana_gemm_decode(int kind, const void* X, int ldx, const float* a_scale, int a_scale_ld, const void* W, int ldw,
                                 const float* w_scale, void* D, void* out_f32, int ldd, const void* bias, const void* residual, int ldr,
                                 int M, int N, int K, int fixed_w, int* err_flag, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 64) return -20;
  if (kind != 0 && kind != 2) return -10;
  const int esz = kind == 0 ? 2 : 1;
  if ((K % (kind == 0 ? 8 : 128)) || (ldx % (16 / esz)) || (ldw % (16 / esz))) return -10;
  const int MP = M <= 16 ? 16 : M <= 32 ? 32 : 64;
  const int tiles = (N + 127) / 128, num_kb = (K + (esz == 2 ? 64 : 128) - 1) / (esz == 2 ? 64 : 128);
  CUtensorMap mw, mx;
  if (!gd_map(&mx, X, M, K, ldx, esz, MP)) return -13;
  if (!gd_map(&mw, W, N, K, ldw, esz, 128)) return -12;
  GemmDecodeParams p{};
  p.M = M; p.N = N; p.K = K;
  p.D = static_cast<__nv_bfloat16*>(D); p.out_f32 = static_cast<float*>(out_f32); p.ldd = ldd;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual); p.ldr = ldr;
  p.a_scale = a_scale; p.a_scale_ld = a_scale_ld; p.w_scale = w_scale;
  p.err = err_flag;
  // fewest shares that give every SM a CTA, four K blocks each at least. Measured (us for 1 / 2 / 4 / 8 shares, cold weights): e4m3, 32
  // rows, N x K = 10240 x 8192 32 / 21 / 27 / 27, 8192 x 8192 31 / 20 / 16 / 21, 4096 x 7168 26 / 17 / 11 / 10, 57344 x 8192 82 / 102 /
  // 100 / 129; bf16, 16 rows, 6144 x 4096 21 / 14 / 12 / 16, 4096 x 14336 67 / 37 / 23 / 22, 28672 x 4096 38 / 44 / 49 / 58.
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  p.splits = 1;
  while (p.splits < 8 && tiles * p.splits < sms && num_kb >= p.splits * 8) p.splits *= 2;
  // Three for two and six for four where all of them run at once with room to spare (a CTA alone on its SM has half the loads in flight; clusters
  // do not fill every group of SMs, and one that has to wait costs a whole round). us, before / after: e4m3 10240 x 8192, 64 rows 26.9 / 24.1,
  // 32 rows 21.6 / 20.2; bf16 10240 x 8192, 1 row 31.5 / 28.9, 5120 x 13824, 4 rows 26.8 / 26.2; but 288 CTAs: 6144 x 4096 11.6 / 15.8,
  // e4m3 12288 x 7168 26.5 / 34.4.
  const int more = p.splits + p.splits / 2;
  if ((p.splits == 2 || p.splits == 4) && 20 * tiles * more <= 33 * sms && num_kb >= 8 * more) p.splits = more;
  const bool early = fixed_w != 0;
  if (kind == 0)
    return MP == 16 ? launch_gemm_decode<16, 0>(mw, mx, p, early, st) : MP == 32 ? launch_gemm_decode<32, 0>(mw, mx, p, early, st)
                                                                                 : launch_gemm_decode<64, 0>(mw, mx, p, early, st);
  return MP == 16 ? launch_gemm_decode<16, 2>(mw, mx, p, early, st) : MP == 32 ? launch_gemm_decode<32, 2>(mw, mx, p, early, st)
                                                                               : launch_gemm_decode<64, 2>(mw, mx, p, early, st);
}
