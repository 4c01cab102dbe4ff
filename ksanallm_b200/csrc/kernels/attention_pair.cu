// Prefill attention with two query tiles per CTA on the tcgen05 tensor cores: causal attention of new query rows, from the paged
// cache (grouped queries, head sizes up to 128) or against expanded latents (192 columns of keys, 128 of values, one key/value head
// per query head).
//
// A CTA owns two groups of up to 128 packed rows (token, head inside the kv group) of one kv head, which share every staged K/V tile.
// Per tile and group S = Q K^T and O += P V as in attention_tc.cu (S and O in TMEM, P read from TMEM); one group's products run while
// the other's softmax does. A row's columns are split between two threads (8 softmax warps per group), which exchange their maxima
// through shared memory. The exponentials (32768 of them, 16 a clock) and the products take about 2000 clocks each for a tile of 256 x
// 128; what remains is the chain S -> softmax -> P V of a group. Against attention_tc.cu (one group per CTA, two CTAs per SM, which
// loads, multiplies and takes exponentials in turn), per layer: one prompt of 16384 tokens (32/8 heads) 3692 -> 2839 us, 775 TFLOP/s
// of the pairs below the diagonal; 8 of 2048 (64/8) 1489 -> 1241; 32 turns of 60-250 tokens on 1000-3500 cached ones 831 -> 633.
// Warp roles: 0 TMA producer (one or two tiles ahead), 1 and 2 MMA issuers of the groups (1 owns the TMEM), 3..10 and 11..18 the groups'
// softmax and epilogue. (One issuing thread for both groups kept the tensor pipe at a quarter: it builds and issues 32 MMAs a tile.)
// No multicast. Every wait is bounded.
#include "sm100_ptx.cuh"
#include <atomic>
#include <cuda_bf16.h>
#include <math_constants.h>

namespace ksana {

typedef __nv_bfloat16 bf16;
constexpr int kPaThreads = 96 + 512;
constexpr int kPaQPanel = 128 * 128;            // bytes of a 64-column panel of 128 query rows
constexpr float kPaRescaleLog2 = 8.f;           // O is rescaled only when a row maximum grew by more than this

template <int KP>
struct PairCfg {                                // KP: 64-column panels of queries and keys
  // Keys per tile: what a tile costs beside its keys (two TMEM round trips, the exchange of the maxima, the hand-offs to and from the
  // MMA thread) counts half as much with 128; three panels leave room for tiles of 64 only.
  static constexpr int kTok = KP == 3 ? 64 : 128;
  static constexpr int kStages = KP == 3 ? 3 : 2;
  static constexpr int kKvPanel = kTok * 128;   // bytes of a 64-column panel of a key or value tile
  static constexpr int kQBytes = 2 * KP * kPaQPanel;
  static constexpr int kStageBytes = (KP + 2) * kKvPanel;
  static constexpr int kSmemBytes = kQBytes + kStages * kStageBytes + 2 * 2 * 128 * 4 + 256 + 1024;
};

struct PairParams {
  bf16* out; long long out_stride;              // [T][out_stride], head h at column h * Dv
  const int* block_table; int table_stride;     // paged keys and values
  const int* cu_k;                              // contiguous ones: first row of every sequence
  const int* cu_q; const int* kv_lens;
  const float* alibi; const float* sinks;       // [Hq] or null
  int G, rows, block_tokens;                    // heads per kv head, query rows of a group (a multiple of G), tokens per cache block
  int kpanels, vpanels, Dv;
  float scale_log2;
  int* err;
};

__device__ __forceinline__ float pa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// PAGED: k_map, v_map are the panels of the cache [block][head x token][column]. Otherwise k_map holds rows [token][head][128 keys |
// 128 values] and v_map the 64 key columns that all heads share [token][64].
template <int KP, bool PAGED>
__global__ void __launch_bounds__(kPaThreads, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                    const __grid_constant__ CUtensorMap v_map, const PairParams p) {
  using Cfg = PairCfg<KP>;
  constexpr int kPaTok = Cfg::kTok, kPaKvPanel = Cfg::kKvPanel, HC = kPaTok / 2;      // HC: columns of S per softmax thread
  extern __shared__ uint8_t pa_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pa_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* kv_s = smem + Cfg::kQBytes;
  float* row_s = reinterpret_cast<float*>(kv_s + Cfg::kStages * Cfg::kStageBytes);     // [group][half][row] maxima, at the end sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_s + 2 * 2 * 128);
  uint64_t* q_full = bars;
  uint64_t* full = bars + 1;                    // [stages]
  uint64_t* empty = full + Cfg::kStages;
  uint64_t* s_full = empty + Cfg::kStages;      // [group]
  uint64_t* p_full = s_full + 2;
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = blockIdx.z, g = blockIdx.y, G = p.G;
  const int q0 = p.cu_q[s], q_len = p.cu_q[s + 1] - q0, kv_len = p.kv_lens[s];
  const int qtile = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);   // longest rows first
  const int row0 = qtile * 2 * p.rows, all_rows = q_len * G;
  if (row0 >= all_rows) return;
  const int past = kv_len - q_len;
  int nt[2];                                    // tiles that each group's rows see
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r0 = row0 + i * p.rows, last = min(r0 + p.rows, all_rows) - 1;
    nt[i] = r0 < all_rows ? (min(kv_len, past + last / G + 1) + kPaTok - 1) / kPaTok : 0;
  }
  const int ntiles = max(nt[0], nt[1]);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(full + i, 1); mbar_init(empty + i, 2); }
    for (int i = 0; i < 2; ++i) { mbar_init(s_full + i, 1); mbar_init(p_full + i, 8); mbar_init(o_full + i, 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;             // S of the groups at columns 0 and kPaTok, O behind

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&q_map);
      tma_prefetch_desc(&k_map);
      tma_prefetch_desc(&v_map);
      const int groups = nt[1] > 0 ? 2 : 1;
      mbar_expect_tx(q_full, groups * p.kpanels * p.rows * 128);
      for (int i = 0; i < groups; ++i)
        for (int h = 0; h < p.kpanels; ++h)
          tma_load_3d(q_s + (i * KP + h) * kPaQPanel, &q_map, q_full, h * 64, g * G, q0 + (row0 + i * p.rows) / G);
    }
    __syncwarp();
    const int* table = PAGED ? p.block_table + static_cast<size_t>(s) * p.table_stride : nullptr;
    const int bt = PAGED ? p.block_tokens : kPaTok, per = p.kpanels + p.vpanels;
    const int k0 = PAGED ? 0 : p.cu_k[s];
    bool ok = true;
    int stage = 0; uint32_t phase = 0;
    for (int j = 0; j < ntiles; ++j) {
      const int t0 = j * kPaTok;
      const int boxes = (PAGED ? min(kPaTok / bt, (kv_len - t0 + bt - 1) / bt) : 1) * per;
      int blk = 0;
      if (PAGED && lane < boxes) blk = table[t0 / bt + lane / per];         // in flight while the stage is waited for
      ok = mbar_wait(empty + stage, phase ^ 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (lane == 0) mbar_expect_tx(full + stage, static_cast<uint32_t>(boxes) * bt * 128);
      __syncwarp();
      uint8_t* st = kv_s + stage * Cfg::kStageBytes;
      for (int i = lane; i < boxes; i += 32) {
        const int b = i / per, h = i - b * per;
        const bool v = h >= p.kpanels;
        const int pn = v ? h - p.kpanels : h;
        uint8_t* dst = st + (v ? KP + pn : pn) * kPaKvPanel + b * bt * 128;
        if constexpr (PAGED) {
          if (i >= 32) blk = table[t0 / bt + b];
          tma_load_3d(dst, v ? &v_map : &k_map, full + stage, pn * 64, g * bt, blk);
        } else {
          if (!v && pn == 2) tma_load_2d(dst, &v_map, full + stage, 0, k0 + t0);
          else tma_load_3d(dst, &k_map, full + stage, (v ? 128 : 0) + pn * 64, g, k0 + t0);
        }
      }
      if (++stage == Cfg::kStages) { stage = 0; phase ^= 1; }
    }
  } else if (warp < 3) {
    // ------------------------------------------------------------------ MMA issuers, one per group
    if (lane == 0) {
      const int i = warp - 1, n = nt[i];
      constexpr uint32_t idesc_qk = make_idesc(128, kPaTok, 1, 1);
      const uint32_t idesc_pv = make_idesc(128, p.vpanels * 64, 1, 1) | (1u << 16);     // B (= V) is MN-major
      // descriptors differ in their start address alone: constants are added to three of them
      const uint64_t q_desc = make_smem_desc_sw128(smem_u32(q_s + i * KP * kPaQPanel));
      const uint64_t k_desc = make_smem_desc_sw128(smem_u32(kv_s));
      const uint64_t v_desc = make_smem_desc_mn_sw128(smem_u32(kv_s + KP * kPaKvPanel), kPaKvPanel);
      const uint32_t s_at = tmem + i * kPaTok, o_at = tmem + 2 * kPaTok + i * 128;
      auto qk = [&](int st) {
        const uint64_t kd = k_desc + static_cast<uint32_t>(st) * (Cfg::kStageBytes >> 4);
#pragma unroll
        for (int pn = 0; pn < KP; ++pn) {
          if (pn >= p.kpanels) break;                 // (columns of the last panel past the row's end are zeros)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f16(s_at, q_desc + (pn * (kPaQPanel >> 4) + 2 * k), kd + (pn * (kPaKvPanel >> 4) + 2 * k), idesc_qk, (pn | k) != 0);
        }
        tc_commit(s_full + i);
      };
      bool ok = mbar_wait(q_full, 0, abort_flag);
      if (n > 0) {
        ok = ok && mbar_wait(full, 0, abort_flag);
        tc_fence_after();
        if (ok) qk(0);
      }
      int st = 0; uint32_t phase = 0;                 // stage of tile j
      for (int j = 0; j < ntiles && ok; ++j) {
        const int st1 = st + 1 == Cfg::kStages ? 0 : st + 1;
        const uint32_t phase1 = st1 ? phase : phase ^ 1;
        if (j < n) {
          if (!mbar_wait(p_full + i, j & 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t vd = v_desc + static_cast<uint32_t>(st) * (Cfg::kStageBytes >> 4);
#pragma unroll
          for (int k = 0; k < kPaTok / 16; ++k)       // 16 tokens per MMA: 8 TMEM columns of P, 16 rows (2 KB) of the V tile
            mma_f16_ts(o_at, s_at + 8 * k, vd + k * (2048 >> 4), idesc_pv, (j | k) != 0);
          tc_commit(empty + st);
          if (j == n - 1) tc_commit(o_full + i);
          if (j + 1 < n) {
            // S over the P that the products just issued read: the tensor pipe takes one thread's MMAs in order
            if (!mbar_wait(full + st1, phase1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            qk(st1);
          }
        } else {
          // a tile that only the other group's rows see
          if (!mbar_wait(full + st, phase, abort_flag)) { ok = false; break; }
          mbar_arrive(empty + st);
        }
        st = st1; phase = phase1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (two threads per row)
    const int i = (warp - 3) >> 3, half = ((warp - 3) >> 2) & 1, qd = warp & 3;
    const int rl = qd * 32 + lane, cb = half * HC;
    const uint32_t lane_off = static_cast<uint32_t>(qd * 32) << 16;
    const uint32_t tmem_s = tmem + i * kPaTok + lane_off, tmem_o = tmem + 2 * kPaTok + i * 128 + lane_off;
    const int vr = row0 + i * p.rows + rl;                 // packed row index inside the sequence
    const bool active = rl < p.rows && vr < all_rows;
    const int tok = vr / G, head = g * G + vr % G;
    const int limit = active ? past + tok : -1;            // last visible position
    const float slope2 = p.alibi && active ? p.alibi[head] * 1.44269504f : 0.f;
    float* mine = row_s + (i * 2 + half) * 128 + rl;
    const float* other = row_s + (i * 2 + (half ^ 1)) * 128 + rl;
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + i * 4 + qd) : "memory"); };   // the two warps of these rows
    float m_used = -CUDART_INF_F, l = 0.f;
    bool ok = true;
    const int n = nt[i];
    for (int j = 0; j < n; ++j) {
      const int t0 = j * kPaTok, c0 = t0 + cb;
      if (ok) ok = mbar_wait(s_full + i, j & 1, abort_flag);
      tc_fence_after();
      uint32_t r[HC];
#pragma unroll
      for (int c = 0; c < HC; c += 32) tmem_ld32(tmem_s + cb + c, *reinterpret_cast<uint32_t(*)[32]>(&r[c]));
      tmem_ld_wait();
      const bool biased = __any_sync(0xffffffffu, slope2 != 0.f || p.scale_log2 <= 0.f);
      if (biased) {                                        // ALiBi (or a scale that is not positive): the finished logits
#pragma unroll
        for (int k = 0; k < HC; ++k)
          r[k] = __float_as_uint(__uint_as_float(r[k]) * p.scale_log2 + slope2 * static_cast<float>(c0 + k - limit));
      }
      if (__any_sync(0xffffffffu, c0 + HC - 1 > limit)) {
        const int last = limit - c0;
#pragma unroll
        for (int k = 0; k < HC; ++k)
          if (k > last) r[k] = 0xff800000u;
      }
      float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int k = 0; k < HC; ++k) mx4[k & 3] = fmaxf(mx4[k & 3], __uint_as_float(r[k]));
      const float factor = biased ? 1.f : p.scale_log2;
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * factor;
      *mine = mx;
      pair_sync();                                         // ... and both halves of S are in registers: P may be written over it
      mx = fmaxf(mx, *other);
      // lazy rescale of O: keep the old reference maximum unless the row's maximum grew by more than 2^8
      float m_new = m_used;
      if (mx > m_used + kPaRescaleLog2 || m_used == -CUDART_INF_F) m_new = mx == -CUDART_INF_F ? m_used : mx;
      const bool grow = j > 0 && m_new != m_used && m_used != -CUDART_INF_F;
      if (__any_sync(0xffffffffu, grow)) {
        const float f = grow ? exp2f(m_used - m_new) : 1.f;
        l *= f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[16];
          tmem_ld16(tmem_o + half * 64 + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * f);
          tmem_st16(tmem_o + half * 64 + c * 16, o);
        }
      }
      m_used = m_new;
      const float mref = m_used == -CUDART_INF_F ? 0.f : m_used;
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < HC; k += 2) {
        const float p0 = pa_exp2(fmaf(__uint_as_float(r[k]), factor, -mref));
        const float p1 = pa_exp2(fmaf(__uint_as_float(r[k + 1]), factor, -mref));
        l4[(k >> 1) & 3] += p0 + p1;
        const __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);
        r[k >> 1] = *reinterpret_cast<const uint32_t*>(&pb);      // in place: slot k / 2 has been consumed
      }
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
#pragma unroll
      for (int c = 0; c < HC / 2; c += 16) tmem_st16(tmem_s + cb / 2 + c, *reinterpret_cast<uint32_t(*)[16]>(&r[c]));
      tmem_st_wait();
      if (t0 + kPaTok > kv_len && ok) {
        // V rows past the sequence's end: stale shared memory or another sequence's rows; their probabilities are 0, but
        // 0 x NaN would poison O. (S is complete, so the tile has landed; both groups write the same zeros.)
        uint8_t* vt = kv_s + (j % Cfg::kStages) * Cfg::kStageBytes + KP * kPaKvPanel;
        const int bad = kv_len - t0;
        for (int k = (threadIdx.x - 96) & 255; k < (kPaTok - bad) * 16; k += 256) {
          const int r_ = bad + (k >> 4), ch = k & 15;
          *reinterpret_cast<uint4*>(vt + (ch >> 3) * kPaKvPanel + r_ * 128 + (((ch & 7) ^ (r_ & 7)) << 4)) = make_uint4(0, 0, 0, 0);
        }
        fence_async_smem();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + i);
    }
    if (n > 0) {
      pair_sync();                                         // the last tile's maxima have been read
      *mine = l;
      pair_sync();
      if (ok && mbar_wait(o_full + i, 0, abort_flag)) {
        tc_fence_after();
        float lt = half ? *other + l : l + *other;
        if (p.sinks && active) lt += exp2f(p.sinks[head] * 1.44269504f - m_used);
        const float inv = lt > 0.f ? 1.f / lt : 0.f;
        bf16* dst = p.out + static_cast<size_t>(q0 + tok) * p.out_stride + static_cast<size_t>(head) * p.Dv;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = half * 64 + c * 32;
          if (col >= p.Dv) break;
          uint32_t o[32];
          tmem_ld32(tmem_o + col, o);
          tmem_ld_wait();
          if (active) {
#pragma unroll
            for (int k = 0; k < 32; k += 8) {
              if (col + k >= p.Dv) break;
              uint4 ov;
              __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
              for (int e = 0; e < 4; ++e)
                o2[e] = __floats2bfloat162_rn(__uint_as_float(o[k + 2 * e]) * inv, __uint_as_float(o[k + 2 * e + 1]) * inv);
              *reinterpret_cast<uint4*>(dst + col + k) = ov;
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 4);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// Latents of whole sequences, one after the other: out[cu_k[s] + i] = the cached row of token i of sequence s (row_vec 16-byte words).
__global__ void gather_latents_kernel(const uint4* __restrict__ cache, long long block_vec, int block_tokens, int row_vec,
                                      const int* __restrict__ table, int table_stride, const int* __restrict__ kv_lens,
                                      const int* __restrict__ cu_k, uint4* __restrict__ out, int num_blocks) {
  const int s = blockIdx.y, n = kv_lens[s], t0 = blockIdx.x * 32;
  if (t0 >= n) return;
  uint4* dst = out + static_cast<size_t>(cu_k[s] + t0) * row_vec;
  const int work = min(32, n - t0) * row_vec;
  for (int i = threadIdx.x; i < work; i += blockDim.x) {
    const int r = i / row_vec, t = t0 + r;
    const int blk = table[static_cast<size_t>(s) * table_stride + t / block_tokens];
    if (blk < 0 || blk >= num_blocks) { dst[i] = make_uint4(0, 0, 0, 0); continue; }
    dst[i] = cache[blk * block_vec + static_cast<long long>(t % block_tokens) * row_vec + (i - r * row_vec)];
  }
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*PaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static PaEncodeFn pa_encode_fn() {
  static PaEncodeFn fn = []() -> PaEncodeFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<PaEncodeFn>(ptr);
  }();
  return fn;
}
// bf16 map of `rank` dimensions (innermost first), strides in elements, box of 64 columns
static bool pa_map(CUtensorMap* map, const void* base, int rank, const long long* dims, const long long* strides, int box1, int box2) {
  PaEncodeFn enc = pa_encode_fn();
  if (!enc) return false;
  cuuint64_t d[3], st[2];
  for (int i = 0; i < rank; ++i) d[i] = static_cast<cuuint64_t>(dims[i]);
  for (int i = 0; i + 1 < rank; ++i) st[i] = static_cast<cuuint64_t>(strides[i]) * 2;
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box1), static_cast<cuuint32_t>(box2)};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), d, st, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int KP, bool PAGED>
static int launch_pair(const CUtensorMap& qm, const CUtensorMap& km, const CUtensorMap& vm, const PairParams& p, dim3 grid, cudaStream_t st) {
  static std::atomic<bool> set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -3;
  if (!set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(prefill_pair_kernel<KP, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<KP>::kSmemBytes) !=
        cudaSuccess) return -3;
    set[dev].store(true, std::memory_order_release);
  }
  prefill_pair_kernel<KP, PAGED><<<grid, kPaThreads, PairCfg<KP>::kSmemBytes, st>>>(qm, km, vm, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace ksana

using namespace ksana;

// Arguments as ksana_paged_prefill_tc (attention_tc.cu) without window, sigmoid weights and gate; separate K and V panels. -100: not
// covered, the caller takes that kernel.
extern "C" int ksana_paged_prefill_pair(const void* q, long long q_stride, long long q_rows, void* out, long long out_stride,
                                        const void* kc, const void* vc, long long block_stride, int block_tokens,
                                        const int* block_table, int table_stride, const int* cu_q, const int* kv_lens,
                                        const float* alibi, const float* sinks, int B, int max_q_len, int Hq, int Hkv, int D, int Dv,
                                        float scale, int num_blocks, int* err, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0) return 0;
  if (D <= 0 || Dv <= 0 || D > 128 || Dv > 128 || D % 8 || Dv % 8 || Hkv <= 0 || Hq % Hkv || kc == vc) return -100;
  const int G = Hq / Hkv, bt = block_tokens;
  if (G > 128 || !(bt == 8 || bt == 16 || bt == 32 || bt == 64 || bt == 128) || B > 65535 || Hkv > 65535) return -100;
  if (block_stride % 8 || num_blocks <= 0 || q_rows <= 0 || out_stride % 8 || q_stride % 8) return -100;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) |
       reinterpret_cast<uintptr_t>(out)) & 15) return -100;
  CUtensorMap qm, km, vm;
  const long long qd[3] = {D, Hq, q_rows}, qs[2] = {D, q_stride};
  const long long kd[3] = {D, static_cast<long long>(Hkv) * bt, num_blocks}, ks[2] = {D, block_stride};
  const long long vd[3] = {Dv, static_cast<long long>(Hkv) * bt, num_blocks}, vs[2] = {Dv, block_stride};
  if (!pa_map(&qm, q, 3, qd, qs, G, 128 / G) || !pa_map(&km, kc, 3, kd, ks, bt, 1) || !pa_map(&vm, vc, 3, vd, vs, bt, 1)) return -100;
  PairParams p{};
  p.out = static_cast<bf16*>(out); p.out_stride = out_stride;
  p.block_table = block_table; p.table_stride = table_stride; p.cu_q = cu_q; p.kv_lens = kv_lens; p.alibi = alibi; p.sinks = sinks;
  p.G = G; p.rows = 128 / G * G; p.block_tokens = bt;
  p.kpanels = (D + 63) / 64; p.vpanels = (Dv + 63) / 64; p.Dv = Dv;
  p.scale_log2 = scale * 1.44269504f; p.err = err;
  const long long rows = static_cast<long long>(max_q_len) * G;
  return launch_pair<2, true>(qm, km, vm, p, dim3(static_cast<unsigned>((rows + 2 * p.rows - 1) / (2 * p.rows)), Hkv, B), st);
}

// Attention of rows q [T][heads][192] against expanded latents: kx [tokens][heads][128 keys | 128 values], the last 64 key columns of
// every head in pe [tokens][pe_ld]; sequence s owns rows cu_k[s] .. cu_k[s] + kv_lens[s]. out [T][heads][128].
extern "C" int ksana_mha_prefill(const void* q, long long T, const void* kx, const void* pe, long long pe_ld, long long tokens,
                                 const int* cu_q, const int* cu_k, const int* kv_lens, int B, int max_q_len, int heads, void* out,
                                 float scale, int* err, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0 || T <= 0 || tokens <= 0) return 0;
  if (heads <= 0 || heads > 65535 || B > 65535 || pe_ld % 8) return -10;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kx) | reinterpret_cast<uintptr_t>(pe) |
       reinterpret_cast<uintptr_t>(out)) & 15) return -11;
  CUtensorMap qm, km, pm;
  const long long qd[3] = {192, heads, T}, qs[2] = {192, heads * 192LL};
  const long long kd[3] = {256, heads, tokens}, ks[2] = {256, heads * 256LL};
  const int kPaTok = PairCfg<3>::kTok;
  const long long pd[2] = {64, tokens}, ps[1] = {pe_ld};
  if (!pa_map(&qm, q, 3, qd, qs, 1, 128) || !pa_map(&km, kx, 3, kd, ks, 1, kPaTok) || !pa_map(&pm, pe, 2, pd, ps, kPaTok, 1)) return -12;
  PairParams p{};
  p.out = static_cast<bf16*>(out); p.out_stride = heads * 128LL;
  p.cu_k = cu_k; p.cu_q = cu_q; p.kv_lens = kv_lens;
  p.G = 1; p.rows = 128; p.kpanels = 3; p.vpanels = 2; p.Dv = 128;
  p.scale_log2 = scale * 1.44269504f; p.err = err;
  return launch_pair<3, false>(qm, km, pm, p, dim3((max_q_len + 255) / 256, heads, B), st);
}

extern "C" int ksana_gather_latents(const void* cache, long long block_stride, int block_tokens, int row, const int* table,
                                    int table_stride, const int* kv_lens, const int* cu_k, void* out, int B, int max_kv_len,
                                    int num_blocks, cudaStream_t st) {
  if (B <= 0 || max_kv_len <= 0) return 0;
  if (row % 8 || block_stride % 8 || block_tokens <= 0 || B > 65535 ||
      ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15)) return -10;
  gather_latents_kernel<<<dim3((max_kv_len + 31) / 32, B), 256, 0, st>>>(
      static_cast<const uint4*>(cache), block_stride / 8, block_tokens, row / 8, table, table_stride, kv_lens, cu_k,
      static_cast<uint4*>(out), num_blocks);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
