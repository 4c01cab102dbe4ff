// Prefill attention with two query tiles per CTA on the tcgen05 tensor cores: causal attention of new query rows, from the paged
// cache (grouped queries, head sizes up to 128) or against expanded latents (192 columns of keys, 128 of values, one key/value head
// per query head).
//
// A CTA owns two groups of up to 128 packed rows (token, head inside the kv group) of one kv head, which share every staged K/V tile.
// Per tile and group S = Q K^T and O += P V as in attention_tc.cu (S and O in TMEM, P read from TMEM). A row's columns are split between
// two threads (8 softmax warps per group), which exchange their maxima through shared memory. The products and the exponentials (32768 of
// them, 16 a clock) take about 2000 clocks each for a tile of 256 x 128, so one group's products have to run under the other's softmax:
//   * one warp issues both groups' products in turn. (With an issuer for each, the two groups' MMAs interleaved, both got their scores at
//     the same time and softmax and products took turns: 6200 clocks a tile. Now 3200.) It runs its loop as a whole warp;
//   * a group's chain S -> softmax -> P V -> next S bounds what is left. P is handed over in two parts, so that P V starts under the
//     second part's exponentials; the exponentials start against the reference maximum before the tile's own is known; with tiles of 64
//     keys a second tile of S is multiplied ahead;
//   * keys and values have rings of their own: a tile of keys is free before its values are needed.
// us a layer against the form before (two issuers) and attention_tc.cu (one group per CTA): one prompt of 16384 tokens (32/8 heads) 1740,
// 2780, 3690 (1265, 790, 595 TFLOP/s of the pairs below the diagonal; 1.63 GHz under the power cap against 1.95); 8 of 2048 (64/8) 651, 996;
// 32 turns of 60-250 tokens on 1000-3500 cached ones 423, 637; latents of 8 prompts of 650-1500 tokens, 128 heads of 192 584, 828.
// Warp roles: 0 TMA producer (one or two tiles ahead), 1 MMA issuer and owner of the TMEM, 2..9 and 10..17 the groups' softmax and
// epilogue. No multicast. Every wait is bounded.
#include "sm100_ptx.cuh"
#include "f32x2.cuh"
#include <atomic>
#include <cuda_bf16.h>
#include <math_constants.h>

namespace ksana {

typedef __nv_bfloat16 bf16;
constexpr int kPaThreads = 64 + 512;
constexpr int kPaQPanel = 128 * 128;            // bytes of a 64-column panel of 128 query rows
constexpr float kPaRescaleLog2 = 8.f;           // O is rescaled only when a row maximum grew by more than this

template <int KP>
struct PairCfg {                                // KP: 64-column panels of queries and keys
  // Keys per tile: what a tile costs beside its keys (two TMEM round trips, the exchange of the maxima, the hand-offs to and from the
  // MMA warp) counts half as much with 128; three panels leave room for tiles of 64 only.
  static constexpr int kTok = KP == 3 ? 64 : 128;
  static constexpr int kStages = KP == 3 ? 3 : 2;             // of keys and of values
  static constexpr int kBufs = KP == 3 ? 2 : 1;               // tiles of S per group: tiles of 64 keys leave room for a second one
  static constexpr int kParts = KP == 3 ? 1 : 2;              // pieces in which a tile's P is handed over
  static constexpr int kKvPanel = kTok * 128;   // bytes of a 64-column panel of a key or value tile
  static constexpr int kQBytes = 2 * KP * kPaQPanel;
  static constexpr int kKBytes = KP * kKvPanel, kVBytes = 2 * kKvPanel;
  static constexpr int kSmemBytes = kQBytes + kStages * (kKBytes + kVBytes) + kBufs * 2 * 2 * 128 * 4 + 256 + 1024;
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
__device__ __forceinline__ float pa_max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
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
  constexpr int ST = Cfg::kStages, SB = Cfg::kBufs, PARTS = Cfg::kParts;
  extern __shared__ uint8_t pa_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pa_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + Cfg::kQBytes;
  uint8_t* v_s = k_s + ST * Cfg::kKBytes;
  float* row_s = reinterpret_cast<float*>(v_s + ST * Cfg::kVBytes);     // [buffer][group][half][row] maxima, at the end sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_s + SB * 2 * 2 * 128);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;                  // [stages]
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* s_full = v_empty + ST;              // [group][buffer]
  uint64_t* p_full = s_full + 2 * SB;           // [group][buffer][part]
  uint64_t* o_done = p_full + 2 * SB * PARTS;   // [group] one tile of S: O is complete; two: the products of a tile are
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  static_assert((1 + 4 * ST + 2 * SB * (1 + PARTS) + 2) * 8 + 8 <= 256, "barriers");

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int s = blockIdx.z, g = blockIdx.y, G = p.G;
  const int q0 = p.cu_q[s], q_len = p.cu_q[s + 1] - q0, kv_len = p.kv_lens[s];
  const int qtile = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);   // longest rows first
  const int row0 = qtile * 2 * p.rows, all_rows = q_len * G;
  if (row0 >= all_rows) return;
  const int past = kv_len - q_len;
  auto tiles_of = [&](int i) {                  // tiles that a group's rows see
    const int r0 = row0 + i * p.rows, last = min(r0 + p.rows, all_rows) - 1;
    return r0 < all_rows ? (min(kv_len, past + last / G + 1) + kPaTok - 1) / kPaTok : 0;
  };
  const int nt0 = tiles_of(0), nt1 = tiles_of(1);
  const int ntiles = max(nt0, nt1);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 4 * ST; ++i) mbar_init(k_full + i, 1);
    for (int i = 0; i < 2 * SB; ++i) mbar_init(s_full + i, 1);
    for (int i = 0; i < 2 * SB * PARTS; ++i) mbar_init(p_full + i, 8);
    for (int i = 0; i < 2; ++i) mbar_init(o_done + i, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);        // S tiles [group][buffer] of kPaTok columns, O behind

  const uint32_t lead = elect_one();            // set in one lane of every warp: it polls, arrives and issues for the warp

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&q_map);
      tma_prefetch_desc(&k_map);
      tma_prefetch_desc(&v_map);
      const int groups = nt1 > 0 ? 2 : 1;
      mbar_expect_tx(q_full, groups * p.kpanels * p.rows * 128);
      for (int i = 0; i < groups; ++i)
        for (int h = 0; h < p.kpanels; ++h)
          tma_load_3d(q_s + (i * KP + h) * kPaQPanel, &q_map, q_full, h * 64, g * G, q0 + (row0 + i * p.rows) / G);
    }
    __syncwarp();
    const int* table = PAGED ? p.block_table + static_cast<size_t>(s) * p.table_stride : nullptr;
    const int bt = PAGED ? p.block_tokens : kPaTok;
    const int k0 = PAGED ? 0 : p.cu_k[s];
    int stage = 0; uint32_t phase = 0;
    for (int j = 0; j < ntiles; ++j) {
      const int t0 = j * kPaTok;
      const int blocks = PAGED ? min(kPaTok / bt, (kv_len - t0 + bt - 1) / bt) : 1;
      int blk = 0;
      if (PAGED && lane < blocks) blk = table[t0 / bt + lane];              // in flight while the stage is waited for
      if (!mbar_wait_warp(k_empty + stage, phase ^ 1, lead, abort_flag)) break;
      if (lane == 0) mbar_expect_tx(k_full + stage, static_cast<uint32_t>(blocks * p.kpanels) * bt * 128);
      __syncwarp();
      uint8_t* ks = k_s + stage * Cfg::kKBytes;
      uint8_t* vs = v_s + stage * Cfg::kVBytes;
      if constexpr (PAGED) {
        if (lane < blocks)
          for (int pn = 0; pn < p.kpanels; ++pn) tma_load_3d(ks + pn * kPaKvPanel + lane * bt * 128, &k_map, k_full + stage, pn * 64, g * bt, blk);
      } else {
        if (lane < 2) tma_load_3d(ks + lane * kPaKvPanel, &k_map, k_full + stage, lane * 64, g, k0 + t0);
        else if (lane == 2) tma_load_2d(ks + 2 * kPaKvPanel, &v_map, k_full + stage, 0, k0 + t0);
      }
      __syncwarp();
      if (!mbar_wait_warp(v_empty + stage, phase ^ 1, lead, abort_flag)) break;
      if (lane == 0) mbar_expect_tx(v_full + stage, static_cast<uint32_t>(blocks * p.vpanels) * bt * 128);
      __syncwarp();
      if constexpr (PAGED) {
        if (lane < blocks)
          for (int pn = 0; pn < p.vpanels; ++pn) tma_load_3d(vs + pn * kPaKvPanel + lane * bt * 128, &v_map, v_full + stage, pn * 64, g * bt, blk);
      } else {
        if (lane < 2) tma_load_3d(vs + lane * kPaKvPanel, &k_map, v_full + stage, 128 + lane * 64, g, k0 + t0);
      }
      __syncwarp();
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of both groups, in turn
    {
      constexpr uint32_t idesc_qk = make_idesc(128, kPaTok, 1, 1);
      const uint32_t idesc_pv = make_idesc(128, p.vpanels * 64, 1, 1) | (1u << 16);     // B (= V) is MN-major
      // descriptors differ in their start address alone: constants are added to three of them
      const uint64_t q_desc = make_smem_desc_sw128(smem_u32(q_s));
      const uint64_t k_desc = make_smem_desc_sw128(smem_u32(k_s));
      const uint64_t v_desc = make_smem_desc_mn_sw128(smem_u32(v_s), kPaKvPanel);
      bool ok = mbar_wait_warp(q_full, 0, lead, abort_flag);
      int ks = 0; uint32_t kphase = 0;                // stage of the next tile of keys
      auto qk = [&](int i, int buf) {
        const uint64_t qd = q_desc + static_cast<uint32_t>(i) * (KP * kPaQPanel >> 4), kd = k_desc + static_cast<uint32_t>(ks) * (Cfg::kKBytes >> 4);
        const uint32_t s_at = tmem + (i * SB + buf) * kPaTok;
#pragma unroll
        for (int pn = 0; pn < KP; ++pn) {
          if (pn >= p.kpanels) break;                 // (columns of the last panel past the row's end are zeros)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f16_lead(lead, s_at, qd + (pn * (kPaQPanel >> 4) + 2 * k), kd + (pn * (kPaKvPanel >> 4) + 2 * k), idesc_qk, (pn | k) != 0);
        }
        tc_commit_lead(lead, s_full + i * SB + buf);
      };
      auto next_k = [&](int t) {                      // all products that read this tile of keys have been issued
        if (t + ST < ntiles) tc_commit_lead(lead, k_empty + ks);
        if (++ks == ST) { ks = 0; kphase ^= 1; }
      };
      for (int t = 0; t < SB && t < ntiles && ok; ++t) {
        ok = mbar_wait_warp(k_full + ks, kphase, lead, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (t < nt0) qk(0, t);
        if (t < nt1) qk(1, t);
        next_k(t);
      }
      int vs = 0; uint32_t vphase = 0;
      for (int j = 0; j < ntiles && ok; ++j) {
        const int buf = j % SB; const uint32_t par = (j / SB) & 1;
        const int t = j + SB;                         // the tile of keys whose scores take the place of this tile's P
        if (!mbar_wait_warp(v_full + vs, vphase, lead, abort_flag)) { ok = false; break; }
        bool keys = false;                            // tile t has landed
#pragma unroll 1
        for (int i = 0; i < 2 && ok; ++i) {
          const int n = i ? nt1 : nt0;
          if (j >= n) continue;
          const uint64_t vd = v_desc + static_cast<uint32_t>(vs) * (Cfg::kVBytes >> 4);
          const uint32_t p_at = tmem + (i * SB + buf) * kPaTok, o_at = tmem + 2 * SB * kPaTok + i * 128;
#pragma unroll
          for (int part = 0; part < PARTS; ++part) {
            if (!mbar_wait_warp(p_full + (i * SB + buf) * PARTS + part, par, lead, abort_flag)) { ok = false; break; }
            tc_fence_after();
            constexpr int PK = kPaTok / 32 / PARTS;   // MMAs (16 tokens: 8 TMEM columns of P, 2 KB of the V tile) per half and part
#pragma unroll
            for (int m = 0; m < 2 * PK; ++m) {
              const int k = (m / PK) * (kPaTok / 32) + part * PK + m % PK;
              mma_f16_ts_lead(lead, o_at, p_at + 8 * k, vd + k * (2048 >> 4), idesc_pv, (j | part | m) != 0);
            }
          }
          if (!ok) break;
          if (SB > 1 || j == n - 1) tc_commit_lead(lead, o_done + i);
          if (t < n) {
            // S over the P that the products just issued read: the tensor pipe takes one thread's MMAs in order
            if (!keys) {
              if (!mbar_wait_warp(k_full + ks, kphase, lead, abort_flag)) { ok = false; break; }
              tc_fence_after();
              keys = true;
            }
            qk(i, buf);
          }
        }
        if (!ok) break;
        if (t < ntiles) next_k(t);
        if (j + ST < ntiles) tc_commit_lead(lead, v_empty + vs);
        if (++vs == ST) { vs = 0; vphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (two threads per row)
    const int i = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1, qd = warp & 3;
    const int rl = qd * 32 + lane, cb = half * HC;
    const uint32_t lane_off = static_cast<uint32_t>(qd * 32) << 16;
    const uint32_t tmem_o = tmem + 2 * SB * kPaTok + i * 128 + lane_off;
    const int vr = row0 + i * p.rows + rl;                 // packed row index inside the sequence
    const bool active = rl < p.rows && vr < all_rows;
    const int tok = vr / G, head = g * G + vr % G;
    const int limit = active ? past + tok : -1;            // last visible position
    const float slope2 = p.alibi && active ? p.alibi[head] * 1.44269504f : 0.f;
    const bool biased = __any_sync(0xffffffffu, slope2 != 0.f || p.scale_log2 <= 0.f);
    const float factor = biased ? 1.f : p.scale_log2;
    float* mine = row_s + (i * 2 + half) * 128 + rl;
    const float* other = row_s + (i * 2 + (half ^ 1)) * 128 + rl;
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + i * 4 + qd) : "memory"); };   // the two warps of these rows
    float m_used = -CUDART_INF_F, l = 0.f;
    bool ok = true;
    const int n = i ? nt1 : nt0;
    for (int j = 0; j < n; ++j) {
      const int t0 = j * kPaTok, c0 = t0 + cb, buf = j % SB;
      const uint32_t tmem_s = tmem + (i * SB + buf) * kPaTok + lane_off;
      uint64_t* p_bar = p_full + (i * SB + buf) * PARTS;
      if (ok) ok = mbar_wait_warp(s_full + i * SB + buf, (j / SB) & 1, lead, abort_flag);
      tc_fence_after();
      // Two tiles of S: every phase of o_done is waited for in turn, before this tile's P is handed over (the next phase cannot end earlier)
      bool waited = SB == 1 || j == 0;
      uint32_t r[HC];
      constexpr int PC = HC / PARTS;                       // columns of a part
      const bool masked = __any_sync(0xffffffffu, t0 + kPaTok - 1 > limit);      // (the same for both warps of these rows)
      // Exponentials of a part against mref; P is packed in place (slots k / 2 have been consumed)
      F2 l2[2] = {f2(0.f), f2(0.f)};
      auto weights = [&](int part, float mref) {
        const F2 factor2 = f2(factor), mref2 = f2(-mref);
#pragma unroll
        for (int k = part * PC; k < (part + 1) * PC; k += 2) {
          float y0, y1;
          split(fma2(f2(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), factor2, mref2), y0, y1);
          const float p0 = pa_exp2(y0), p1 = pa_exp2(y1);
          l2[(k >> 1) & 1] = l2[(k >> 1) & 1] + f2(p0, p1);
          const __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);
          r[k >> 1] = *reinterpret_cast<const uint32_t*>(&pb);
        }
      };
      auto hand_over = [&](int part) {
#pragma unroll
        for (int c = part * PC / 2; c < (part + 1) * PC / 2; c += 16)
          tmem_st16(tmem_s + cb / 2 + c, *reinterpret_cast<uint32_t(*)[16]>(&r[c]));
        tmem_st_wait();
        if constexpr (SB > 1) {
          if (!waited && ok) ok = mbar_wait_warp(o_done + i, (j - 1) & 1, lead, abort_flag);
        }
        tc_fence_before();
        __syncwarp();
        mbar_arrive_lead(lead, p_bar + part);
      };
      auto clear_values = [&]() {
        if (t0 + kPaTok > kv_len && ok) {
          // V rows past the sequence's end: stale shared memory or another sequence's rows; their probabilities are 0, but
          // 0 x NaN would poison O. (Both groups write the same zeros.)
          ok = mbar_wait_warp(v_full + j % ST, (j / ST) & 1, lead, abort_flag);
          uint8_t* vt = v_s + (j % ST) * Cfg::kVBytes;
          const int bad = kv_len - t0;
          for (int k = (threadIdx.x - 64) & 255; k < (kPaTok - bad) * 16; k += 256) {
            const int r_ = bad + (k >> 4), ch = k & 15;
            *reinterpret_cast<uint4*>(vt + (ch >> 3) * kPaKvPanel + r_ * 128 + (((ch & 7) ^ (r_ & 7)) << 4)) = make_uint4(0, 0, 0, 0);
          }
          fence_async_smem();
          __syncwarp();
        }
      };
      auto largest = [&]() {
        float mx4[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
        for (int k = 0; k < HC; k += 2) mx4[(k >> 1) & 3] = pa_max3(mx4[(k >> 1) & 3], __uint_as_float(r[k]), __uint_as_float(r[k + 1]));
        return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      };
      // Most tiles: no column is masked and the row's reference maximum stays. The first part's exponentials are taken against it while
      // the maxima are still being formed; where one outgrew it, they are taken again.
      if (j > 0 && !masked && !biased) {
        const float mref = m_used == -CUDART_INF_F ? 0.f : m_used;
#pragma unroll
        for (int c = 0; c < HC; c += 32) tmem_ld32(tmem_s + cb + c, *reinterpret_cast<uint32_t(*)[32]>(&r[c]));
        tmem_ld_wait();
        float mx = largest();
        weights(0, mref);
        mx *= factor;
        mine[buf * 512] = mx;
        pair_sync();                                       // ... and both halves of S are in registers: P may be written over it
        mx = fmaxf(mx, other[buf * 512]);
        if (!__any_sync(0xffffffffu, mx > m_used + kPaRescaleLog2)) {
          hand_over(0);                                      // (no key past kv_len: such a tile is masked)
          if constexpr (PARTS > 1) {
            weights(1, mref);
            hand_over(1);
          }
          l += sum2(l2[0] + l2[1]);
          continue;
        }
        l2[0] = l2[1] = f2(0.f);
      }
#pragma unroll
      for (int c = 0; c < HC; c += 32) tmem_ld32(tmem_s + cb + c, *reinterpret_cast<uint32_t(*)[32]>(&r[c]));
      tmem_ld_wait();
      if (biased) {                                        // ALiBi (or a scale that is not positive): the finished logits
#pragma unroll
        for (int k = 0; k < HC; ++k)
          r[k] = __float_as_uint(__uint_as_float(r[k]) * p.scale_log2 + slope2 * static_cast<float>(c0 + k - limit));
      }
      if (masked) {
        const int last = limit - c0;
#pragma unroll
        for (int k = 0; k < HC; ++k)
          if (k > last) r[k] = 0xff800000u;
      }
      float mx = largest() * factor;
      mine[buf * 512] = mx;
      pair_sync();
      mx = fmaxf(mx, other[buf * 512]);
      // lazy rescale of O: keep the old reference maximum unless the row's maximum grew by more than 2^8
      float m_new = m_used;
      if (mx > m_used + kPaRescaleLog2 || m_used == -CUDART_INF_F) m_new = mx == -CUDART_INF_F ? m_used : mx;
      const bool grow = j > 0 && m_new != m_used && m_used != -CUDART_INF_F;
      if (__any_sync(0xffffffffu, grow)) {
        if constexpr (SB > 1) {                            // (one tile of S: its products came after those of the tile before)
          if (ok) ok = mbar_wait_warp(o_done + i, (j - 1) & 1, lead, abort_flag);
          tc_fence_after();
          waited = true;
        }
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
      clear_values();
#pragma unroll
      for (int part = 0; part < PARTS; ++part) {
        weights(part, m_used == -CUDART_INF_F ? 0.f : m_used);
        hand_over(part);
      }
      l += sum2(l2[0] + l2[1]);
    }
    if (n > 0) {
      pair_sync();                                         // the last tile's maxima have been read
      *mine = l;
      pair_sync();
      if (ok && mbar_wait_warp(o_done + i, SB > 1 ? (n - 1) & 1 : 0, lead, abort_flag)) {
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
          __syncwarp();
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
