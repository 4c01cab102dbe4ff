// NVFP4 GEMM on the block-scaled tensor-core path (tcgen05.mma kind::mxf4nvf4, 16-element blocks).
//
//   D[M,N] = alpha * (A_q * a_bs)[M,K] * (W_q * w_bs)[N,K]^T (+bias)(+residual),   alpha = a_ts * w_ts
//
// Both operands are e2m1 values, two per byte (even element in the low nibble), with one e4m3 scale per 16
// elements along K ([rows, K/16] bytes) and one fp32 scale per tensor. A 128-byte swizzled shared-memory row
// holds 256 elements = four MMAs of K = 64; each MMA consumes four scales per row, i.e. exactly one 32-bit
// TMEM word: the scales of 128 rows are four columns, row r in lane r % 32 of column r / 32, the same in all four quarters.
// Warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 scales, warps 6..13 epilogue; single 256-column accumulator and bounded waits as in
// the FP8 hardware-scaled kernel. The scales of a K block travel by TMA with its operands (16 bytes a row); four warps, one per quarter
// of TMEM, write them there from registers. (tcgen05.cp of 512-byte chunks, twelve a block, took about 80 clocks each between the MMAs of two
// blocks, 1500 clocks a block with 512 of MMAs; now about 1050;
// a tile of 256 x 192 with them was slower by its work: 1002 us.) The epilogue stores whole sectors, 32 bytes a lane (with 16 a sector
// reaches the L2 in two halves). 9753 x 28672 x 4096: 1094 us with scales loaded by a packer warp on demand, 832 by TMA and tcgen05.cp, 695
// from registers, 627 with the wider stores (3.65 PFLOP/s); 9753 x 4096 x 14336: 612, 432, 319, 282.
//
// No counterpart in the reference (its low-bit paths are GPTQ/AWQ W4A16 through Marlin/Machete,
// 3rdparty/LLM_kernels/csrc/kernels/nvidia/mixture_of_experts and .../machete); the operator is specified by
// the fp32 statement in ops/reference.py (gemm_nvfp4).
#include "sm100_ptx.cuh"
#include "vec8.cuh"
#include <cuda_bf16.h>
#include <stdio.h>

namespace ksana {

constexpr int kF4BM = 128;
constexpr int kF4RowBytes = 128;
constexpr int kF4Threads = 192 + 256;

template <int BN>
struct F4Cfg {
  static constexpr int kABytes = kF4BM * kF4RowBytes;
  static constexpr int kBBytes = BN * kF4RowBytes;
  static constexpr int kSfOff = kABytes + kBBytes;                 // scales of the stage: rows of 16 bytes
  static constexpr int kSfBytes = (kF4BM + BN) * 16;
  static constexpr int kStageBytes = kSfOff + kSfBytes;
  static constexpr int kStages = BN == 256 ? 4 : 6;
  static constexpr int kAccStages = BN == 256 ? 1 : 2;
  static constexpr int kBChunks = BN / 128;
  static constexpr int kSfCols = 4 * 4 * (1 + kBChunks);           // TMEM columns of one scale set (4 MMAs), a set per stage
  static constexpr int kSfBase = kAccStages * BN;             // first scale column
  static constexpr int kTmemCols = 512;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 512;
  static constexpr int kEpiCols = BN / 2;
  static_assert(kSfBase + kStages * kSfCols <= kTmemCols && kStageBytes % 1024 == 0 && kSmemBytes <= 227 * 1024, "tile does not fit");
};

struct F4Params {
  int M, N, K;
  __nv_bfloat16* D; float* out_f32; int ldd;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual; int ldr;
  const float* a_ts; const float* w_ts;    // per-tensor scales (device scalars)
  int* err;
  int wide;                                  // rows of D start on 32-byte boundaries
  // grouped (mixture-of-experts) mode: row tile i multiplies with expert tile_expert[i] (< 0: tile unused); W, w_bs
  // are the experts' matrices stacked along N (expert_rows rows each) and w_ts holds one tensor scale per expert
  const int* tile_expert; int expert_rows;
};

constexpr int kF4GroupM = 16;
__device__ __forceinline__ void f4_tile_coords(int tile, int m_tiles, int n_tiles, int& m_blk, int& n_blk) {
  const int per_group = kF4GroupM * n_tiles;
  const int group = tile / per_group;
  const int first_m = group * kF4GroupM;
  const int gsz = min(m_tiles - first_m, kF4GroupM);
  const int in_group = tile - group * per_group;
  m_blk = first_m + in_group % gsz;
  n_blk = in_group / gsz;
}

template <int BN>
__global__ void __launch_bounds__(kF4Threads, 1)
gemm_nvfp4_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                  const __grid_constant__ CUtensorMap tma_sa, const __grid_constant__ CUtensorMap tma_sb, const F4Params p) {
  using Cfg = F4Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kStages * Cfg::kStageBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = full_bar + Cfg::kStages;
  uint64_t* sf_full = empty_bar + Cfg::kStages;             // the stage's scales are in TMEM
  uint64_t* tfull_bar = sf_full + Cfg::kStages;
  uint64_t* tempty_bar = tfull_bar + Cfg::kAccStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + Cfg::kAccStages);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int m_tiles = (p.M + kF4BM - 1) / kF4BM;
  const int n_tiles = (p.N + BN - 1) / BN;
  const int num_tiles = m_tiles * n_tiles;
  const int num_kb = p.K / 256;            // 256 elements = one 128-byte row per stage

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); mbar_init(&sf_full[i], 4); }
    for (int i = 0; i < Cfg::kAccStages; ++i) { mbar_init(&tfull_bar[i], 1); mbar_init(&tempty_bar[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, Cfg::kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t lead = elect_one();             // one lane of every warp: it polls and issues for the warp

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tma_a);
      tma_prefetch_desc(&tma_b);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int m_blk, n_blk;
        f4_tile_coords(tile, m_tiles, n_tiles, m_blk, n_blk);
        int b_row = n_blk * BN;
        if (p.tile_expert) {
          const int e = p.tile_expert[m_blk];
          if (e < 0) continue;                 // every role skips the tiles of unused row blocks
          b_row += e * p.expert_rows;
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + stage * Cfg::kStageBytes;
          mbar_expect_tx(&full_bar[stage], Cfg::kStageBytes);
          tma_load_2d(sa, &tma_a, &full_bar[stage], kb * 128, m_blk * kF4BM);
          tma_load_2d(sa + Cfg::kABytes, &tma_b, &full_bar[stage], kb * 128, b_row);
          tma_load_2d(sa + Cfg::kSfOff, &tma_sa, &full_bar[stage], kb * 16, m_blk * kF4BM);
          tma_load_2d(sa + Cfg::kSfOff + kF4BM * 16, &tma_sb, &full_bar[stage], kb * 16, b_row);
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    {
      int stage = 0; uint32_t phase = 0;
      int acc = 0; uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        if (p.tile_expert) {
          int m_blk, n_blk;
          f4_tile_coords(tile, m_tiles, n_tiles, m_blk, n_blk);
          if (__any_sync(0xffffffffu, p.tile_expert[m_blk] < 0)) continue;
        }
        if (!mbar_wait_warp(&tempty_bar[acc], acc_phase ^ 1, lead, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb && ok; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, lead, abort_flag)) { ok = false; break; }
          if (!mbar_wait_warp(&sf_full[stage], phase, lead, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tsf = tmem_base + Cfg::kSfBase + stage * Cfg::kSfCols;
          const uint32_t sa = smem_u32(smem + stage * Cfg::kStageBytes);
          constexpr int kPerMma = 1 + Cfg::kBChunks;          // groups of 128 scale rows: A, then the B halves
          const uint64_t adesc = make_smem_desc_sw128(sa);
          const uint64_t bdesc = make_smem_desc_sw128(sa + Cfg::kABytes);
          constexpr uint32_t idesc = make_idesc_nvf4(kF4BM, BN);
#pragma unroll
          for (int k = 0; k < 4; ++k)      // 64 elements (32 bytes) per MMA, four e4m3 scales per row and MMA
            mma_nvf4_lead(lead, d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0, tsf + 4 * kPerMma * k,
                     tsf + 4 * kPerMma * k + 4);
          tc_commit_lead(lead, &empty_bar[stage]);
          if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) {
          tc_commit_lead(lead, &tfull_bar[acc]);
          if (++acc == Cfg::kAccStages) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp < 6) {
    // ------------------------------------------------------------ scale warps, one per TMEM quarter (the scales are in all four)
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      if (p.tile_expert) {
        int m_blk, n_blk;
        f4_tile_coords(tile, m_tiles, n_tiles, m_blk, n_blk);
        if (p.tile_expert[m_blk] < 0) continue;
      }
      for (int kb = 0; kb < num_kb; ++kb) {
        // the stage was loaded after its MMAs had ended, so that its scale columns are free too
        if (!mbar_wait_warp(&full_bar[stage], phase, lead, abort_flag)) { ok = false; break; }
        tc_fence_after();
        constexpr int kPerMma = 1 + Cfg::kBChunks;
        const uint4* rows = reinterpret_cast<const uint4*>(smem + stage * Cfg::kStageBytes + Cfg::kSfOff);
        // 16 bytes a row are one word per MMA; a group of 128 rows takes four columns per MMA: row r in lane r % 32 of column r / 32
        uint32_t v[Cfg::kSfCols];
#pragma unroll
        for (int c = 0; c < kPerMma; ++c)
#pragma unroll
          for (int r4 = 0; r4 < 4; ++r4) {
            const uint4 x = rows[c * 128 + r4 * 32 + lane];
            v[4 * c + r4] = x.x;
            v[4 * (kPerMma + c) + r4] = x.y;
            v[4 * (2 * kPerMma + c) + r4] = x.z;
            v[4 * (3 * kPerMma + c) + r4] = x.w;
          }
        const uint32_t dst = tmem_base + lane_base + Cfg::kSfBase + stage * Cfg::kSfCols;
        tmem_st32(dst, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        if constexpr (Cfg::kSfCols > 32) tmem_st16(dst + 32, *reinterpret_cast<uint32_t(*)[16]>(&v[32]));
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_lead(lead, &sf_full[stage]);
        if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int q = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    const int wg = (warp - 6) >> 2;
    constexpr int EC = Cfg::kEpiCols;
    const int col_off = wg * EC;
    int acc = 0; uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      int m_blk, n_blk;
      f4_tile_coords(tile, m_tiles, n_tiles, m_blk, n_blk);
      const int row = m_blk * kF4BM + q * 32 + lane;
      const int n0 = n_blk * BN + col_off;
      const bool row_ok = row < p.M;
      int expert = 0;
      if (p.tile_expert) {
        expert = p.tile_expert[m_blk];
        if (expert < 0) continue;
      }
      __syncwarp();                             // lanes without a row come from the tile before by another path
      if (!mbar_wait_warp(&tfull_bar[acc], acc_phase, lead, abort_flag)) { ok = false; break; }
      tc_fence_after();
      uint32_t r[EC];
#pragma unroll
      for (int c0 = 0; c0 < EC; c0 += 32) tmem_ld32(tmem_base + lane_base + acc * BN + col_off + c0, *reinterpret_cast<uint32_t(*)[32]>(&r[c0]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_lead(lead, &tempty_bar[acc]);     // the accumulator is in registers: the next tile may start
      if (++acc == Cfg::kAccStages) { acc = 0; acc_phase ^= 1; }
      if (!row_ok) continue;
      const float alpha = (p.a_ts ? *p.a_ts : 1.f) * (p.w_ts ? p.w_ts[expert] : 1.f);
#pragma unroll
      for (int c0 = 0; c0 < EC; c0 += 16) {
        uint4 ov[2];
        const int col0 = n0 + c0;
#pragma unroll
        for (int h8 = 0; h8 < 2; ++h8) {
          const int col = col0 + h8 * 8;
          if (col >= p.N) continue;
          float o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(r[c0 + h8 * 8 + i]) * alpha;
          if (p.bias) {
            const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);
            const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&bv);
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(b2[i]); o[2 * i] += f.x; o[2 * i + 1] += f.y; }
          }
          if (p.residual) {
            const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + static_cast<size_t>(row) * p.ldr + col);
            const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(r2[i]); o[2 * i] += f.x; o[2 * i + 1] += f.y; }
          }
          if (p.out_f32) {
            float4* dst = reinterpret_cast<float4*>(p.out_f32 + static_cast<size_t>(row) * p.ldd + col);
            dst[0] = make_float4(o[0], o[1], o[2], o[3]);
            dst[1] = make_float4(o[4], o[5], o[6], o[7]);
          }
          __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov[h8]);
#pragma unroll
          for (int i = 0; i < 4; ++i) o2[i] = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
        }
        if (p.out_f32 || col0 >= p.N) continue;
        __nv_bfloat16* dst = p.D + static_cast<size_t>(row) * p.ldd + col0;
        if (p.wide && col0 + 16 <= p.N) {
          st_global_32(dst, ov[0], ov[1]);
        } else {
          *reinterpret_cast<uint4*>(dst) = ov[0];
          if (col0 + 8 < p.N) *reinterpret_cast<uint4*>(dst + 8) = ov[1];
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 8);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::kTmemCols); }
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*F4EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static F4EncodeFn f4_encode_fn() {
  static F4EncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) return nullptr;
    fn = reinterpret_cast<F4EncodeFn>(ptr);
  }
  return fn;
}
static int f4_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows, int box_cols = 128) {
  F4EncodeFn enc = f4_encode_fn();
  if (!enc) return -1;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld)};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

template <int BN>
static int launch_f4(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& sa, const CUtensorMap& sb, const F4Params& p, int max_ctas, cudaStream_t st) {
  using Cfg = F4Cfg<BN>;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(gemm_nvfp4_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) !=
        cudaSuccess) return -3;
    set = true;
  }
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  const int tiles = ((p.M + kF4BM - 1) / kF4BM) * ((p.N + BN - 1) / BN);
  int grid = tiles < sms ? tiles : sms;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  gemm_nvfp4_kernel<BN><<<grid, kF4Threads, Cfg::kSmemBytes, st>>>(ma, mb, sa, sb, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace ksana

using namespace ksana;

// A_q [M, K/2] packed e2m1 (row stride lda bytes), a_bs [M, K/16] e4m3 bytes (row stride a_bs_ld), a_ts device fp32
// scalar (null = 1); W likewise with N rows. K must be a multiple of 256, N of 8; strides multiples of 16 bytes.
// Output bf16 (D) or fp32 (out_f32). bn_hint: 128, 256 or 0 (automatic).
extern "C" int ksana_gemm_nvfp4(const void* Aq, int lda, const void* a_bs, int a_bs_ld, const float* a_ts, const void* Wq,
                                int ldw, const void* w_bs, int w_bs_ld, const float* w_ts, void* D, void* out_f32, int ldd,
                                const void* bias, const void* residual, int ldr, int M, int N, int K, int bn_hint,
                                int max_ctas, int* err_flag, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N % 8) || (K % 256) || (lda % 16) || (ldw % 16) || (a_bs_ld % 16) || (w_bs_ld % 16) || (ldd % 8) ||
      (residual && (ldr % 8))) return -10;
  if ((reinterpret_cast<uintptr_t>(Aq) | reinterpret_cast<uintptr_t>(Wq) | reinterpret_cast<uintptr_t>(a_bs) |
       reinterpret_cast<uintptr_t>(w_bs)) & 15) return -11;
  int bn = bn_hint;
  if (bn != 128 && bn != 256) {
    const int m_tiles = (M + kF4BM - 1) / kF4BM;
    bn = (m_tiles * ((N + 255) / 256) >= 100) ? 256 : 128;
  }
  CUtensorMap ma, mb, sa, sb;
  if (f4_map(&ma, Aq, M, K / 2, lda, kF4BM)) return -12;
  if (f4_map(&mb, Wq, N, K / 2, ldw, bn)) return -13;
  if (f4_map(&sa, a_bs, M, K / 16, a_bs_ld, kF4BM, 16) || f4_map(&sb, w_bs, N, K / 16, w_bs_ld, bn, 16)) return -14;
  F4Params p{};
  p.M = M; p.N = N; p.K = K;
  p.D = static_cast<__nv_bfloat16*>(D); p.out_f32 = static_cast<float*>(out_f32); p.ldd = ldd;
  p.wide = D && ldd % 16 == 0 && (reinterpret_cast<uintptr_t>(D) & 31) == 0;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual); p.ldr = ldr;
  p.a_ts = a_ts; p.w_ts = w_ts;
  p.err = err_flag;
  return bn == 256 ? launch_f4<256>(ma, mb, sa, sb, p, max_ctas, st) : launch_f4<128>(ma, mb, sa, sb, p, max_ctas, st);
}

// Grouped (mixture-of-experts) form: A_q [cap, K/2] holds expert-major rows in 128-row tiles, tile_expert[cap / 128]
// names the expert of every tile (-1: unused, nothing is computed or stored for it). W_q [E * N, K/2], w_bs
// [E * N, K/16] are the experts' matrices stacked along N, w_ts [E] their tensor scales. N must be a multiple of 128.
extern "C" int ksana_gemm_grouped_nvfp4(const void* Aq, int lda, const void* a_bs, int a_bs_ld, const float* a_ts,
                                        const void* Wq, int ldw, const void* w_bs, int w_bs_ld, const float* w_ts,
                                        void* D, int ldd, int cap, int N, int K, int num_experts, const int* tile_expert,
                                        int bn_hint, int* err_flag, cudaStream_t st) {
  if (cap <= 0 || N <= 0 || K <= 0 || num_experts <= 0) return 0;
  if ((cap % 128) || (N % 128) || (K % 256) || (lda % 16) || (ldw % 16) || (a_bs_ld % 16) || (w_bs_ld % 16) || (ldd % 8) ||
      tile_expert == nullptr || w_ts == nullptr) return -10;
  if ((reinterpret_cast<uintptr_t>(Aq) | reinterpret_cast<uintptr_t>(Wq) | reinterpret_cast<uintptr_t>(a_bs) |
       reinterpret_cast<uintptr_t>(w_bs)) & 15) return -11;
  // a weight tile must not reach into the next expert's rows
  int bn = (bn_hint == 128 || (N % 256)) ? 128 : 256;
  CUtensorMap ma, mb, sa, sb;
  if (f4_map(&ma, Aq, cap, K / 2, lda, kF4BM)) return -12;
  if (f4_map(&mb, Wq, num_experts * N, K / 2, ldw, bn)) return -13;
  if (f4_map(&sa, a_bs, cap, K / 16, a_bs_ld, kF4BM, 16) || f4_map(&sb, w_bs, num_experts * N, K / 16, w_bs_ld, bn, 16)) return -14;
  F4Params p{};
  p.M = cap; p.N = N; p.K = K;
  p.D = static_cast<__nv_bfloat16*>(D); p.ldd = ldd;
  p.wide = D && ldd % 16 == 0 && (reinterpret_cast<uintptr_t>(D) & 31) == 0;
  p.a_ts = a_ts; p.w_ts = w_ts;
  p.err = err_flag;
  p.tile_expert = tile_expert; p.expert_rows = N;
  return bn == 256 ? launch_f4<256>(ma, mb, sa, sb, p, 0, st) : launch_f4<128>(ma, mb, sa, sb, p, 0, st);
}
