// Paged attention for sm_100a: causal prefill (chunked-prefill and prefix-cache
// aware) and split-KV decode, both reading K/V in place from the paged cache
// through a block table.
//
// Grouped-query packing: the query heads that share one KV head are packed into
// the M dimension of the tensor-core tiles together with the query tokens, so a
// K/V tile staged in shared memory is used by the whole head group (8 heads for
// Llama-3 / Qwen2 70B) instead of being re-read per query head.
//
//   virtual row r of (sequence s, kv head g):  token = r / G,  head = g*G + r % G
//
// Prefill: 64 rows per CTA (4 warps x 16), K/V tiles of 64 tokens, online
// softmax in fp32 (exp2), only the NEW query rows are computed: the causal
// offset is kv_len - q_len, so cached prefixes cost no attention work.
// Decode: all (sequence, kv head, tile) units of a launch lie in one line that is shared out over the resident CTAs, in equal
// ranges or by items, whichever is cheaper (paged_decode_stream_kernel); 4 warps walk disjoint 16-token slices of each tile, a fifth keeps the
// tile ring full by TMA. Caches that TMA cannot read (other block sizes or strides) take paged_decode_kernel: one
// CTA per (kv head, sequence, split), all threads copying, and a small reduce kernel.
//
// FP8 (e4m3) caches: the decode kernel multiplies the stored values in f16 (exact) and applies the per-layer scales
// to scores and outputs; the other kernels dequantise while staging tiles.
//
// Head sizes: a kernel is compiled for a padded head size DP (64, 128, 192, 256); the real query/key size D and value
// size Dv are run-time values up to DP (multiples of 8), padded with zeros in shared memory only (TMA fills the
// columns past the row's end). K and V lie in panels of their own: [block][Hkv][block_tokens][D] and [...][Dv].
// Sliding window: position i sees j <= i with i - j < window or j < keep; tiles between the kept tokens and the
// window are not visited. Sink: an extra logit per head in the softmax denominator, without a value.
// Panels that coincide (the values are the keys) are staged once.
// Sigmoid weights (SIG): every visible key has the weight sigmoid(score + bias[head][distance]), nothing is normalised over
// keys. Gate: outputs are multiplied by the sigmoid of a gate element and by one factor.
//
// Functional counterpart of the reference's decode kernels
// (3rdparty/LLM_kernels/csrc/kernels/nvidia/paged_attention/paged_attention.cu:81-640)
// and of its FlashAttention-2 call (src/ksana_llm/kernels/nvidia/kernel_wrapper.cpp:437-588),
// without the reverse cache copy the latter needs.
#include "sm100_ptx.cuh"
#include "pdl.cuh"
#include "fp8_scale.cuh"
#include <atomic>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace ksana {

// K/V staging modes: plain cp.async (any block size), FP8 cache with conversion, or TMA: one elected thread
// issues a 2-D bulk tensor copy per (cache block, 64-column half) - the per-16-byte address arithmetic of
// the cp.async path made the decode kernel instruction-bound at a third of HBM bandwidth.
enum KvMode { kKvCpAsync = 0, kKvFp8 = 1, kKvTma = 2, kKvTmaFp8 = 3 };

typedef __nv_bfloat16 bf16;
constexpr int kTileTok = 64;     // KV tokens per shared-memory tile
constexpr int kAttnThreads = 128;
constexpr int kBiasSmem = 2048;  // floats of bias rows that a decode CTA stages
__host__ __device__ constexpr int kv_stages(int dp) { return dp <= 192 ? 3 : 2; }    // K/V tile ring: all but one tile in flight while one is consumed

// elements of a decode CTA's K and V rings (one ring where they are the same); the fp32 merge area lies over them
__host__ __device__ constexpr int decode_ring(int dp, bool shared) {
  const int rings = (shared ? 1 : 2) * kv_stages(dp) * kTileTok * dp, merge = 4 * 16 * (dp + 2) * 2;
  return rings > merge ? rings : merge;
}

struct AttnParams {
  const bf16* q; long long q_stride;     // [T, q_stride] ; head h at column h*D
  bf16* out; long long out_stride;       // [T, out_stride]
  const void* kc; const void* vc;        // panels of block 0: K [Hkv][block_tokens][D], V [Hkv][block_tokens][Dv]
  long long block_stride;                // elements between blocks
  int block_tokens;
  int D, Dv;                             // real head sizes
  int window, keep;                      // sliding window in tokens (0: none) and first tokens every row sees
  const float* sinks;                    // [Hq] logits added to the softmax denominator, or null
  const int* block_table; int table_stride;   // [B][table_stride]
  const int* cu_q;                       // [B+1] query row offsets (prefill) or null (decode: row = s)
  const int* kv_lens;                    // [B]
  const float* alibi;                    // [Hq] slopes or null
  const float* bias; int bias_len;       // sigmoid weights: [Hq][bias_len] added by distance (the last entry holds beyond)
  int bias_smem;                         // decode: the rows of a CTA's heads are staged in shared memory (floats; 0: not)
  const bf16* gate; long long gate_stride;   // optional, same layout as out
  float out_factor;                      // of gated outputs
  int Hq, Hkv;
  float scale_log2;                      // softmax scale * log2(e)
  float k_scale, v_scale;                // fp8 cache dequant scales
  // decode split workspace
  float* part_o; float* part_ml; int num_splits;
  // stream decode: tile ring, partial results of cut (sequence, head) items [2 * CTAs][rows][Dv] and [2 * CTAs][rows][2],
  // arrival counters [B * heads] (zero before and after every launch)
  int B, stages, stage_bytes, rows, vec_out;
  float* cut_o; float* cut_ml; unsigned int* counters;
  int* err;                              // device word set when a bounded wait gave up
  // decode, head dim 128: also emit the output as the FP8 operand of the next GEMM (e4m3 values [T][Hq*D] and one
  // power-of-two scale per row and head, [Hq][oscale_ld]), quantised from the bf16-rounded values exactly as the
  // stand-alone quantiser would
  uint8_t* outq; float* oscale; int oscale_ld;
};

// One head row of D = 128 outputs held one per thread of a 128-thread block: rounds to bf16, stores it (if `out`),
// and stores the row's e4m3 values and scale. Every thread of the block must call it.
__device__ __forceinline__ void store_head_row_q(const AttnParams& p, int s, int head, int d, float v, float* red4) {
  const __nv_bfloat16 b = __float2bfloat16(v);
  const float fb = __bfloat162float(b);
  if (p.out) p.out[static_cast<size_t>(s) * p.out_stride + head * 128 + d] = b;
  float am = fabsf(fb);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
  __syncthreads();                                   // red4 may still be read from the previous row
  if ((threadIdx.x & 31) == 0) red4[threadIdx.x >> 5] = am;
  __syncthreads();
  am = fmaxf(fmaxf(red4[0], red4[1]), fmaxf(red4[2], red4[3]));
  const float sc = fp8_group_scale(am);
  const __nv_fp8_storage_t q = __nv_cvt_float_to_fp8(fb * (1.f / sc), __NV_SATFINITE, __NV_E4M3);
  p.outq[(static_cast<size_t>(s) * p.Hq + head) * 128 + d] = q;
  if (d == 0) p.oscale[static_cast<size_t>(head) * p.oscale_ld + s] = sc;
}

// Tiles of `tile` tokens a range of rows visits, in order: those that hold kept first tokens, then the window's. `lo` is
// the first position inside the window of the range's first row, `total` the tile count up to the last visible token.
struct TileRange { int nkeep, first, count; };
__device__ __forceinline__ TileRange visited_tiles(int lo, int keep, int total, int tile) {
  TileRange r;
  r.first = lo > 0 ? lo / tile : 0;
  r.nkeep = min((keep + tile - 1) / tile, r.first);
  r.count = r.nkeep + total - r.first;
  return r;
}
__device__ __forceinline__ int tile_at(const TileRange& r, int i) { return i < r.nkeep ? i : r.first + i - r.nkeep; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Shared tile of ROWS rows x D bf16, stored as D/64 panels of [ROWS][64] (128-byte rows); inside a panel the
// 16-byte chunk cc of row r lives at chunk (cc ^ (r & 7)): exactly what a TMA copy with the 128-byte swizzle
// writes, and conflict-free for ldmatrix.
template <int D, int ROWS>
__device__ __forceinline__ bf16* tile_ptr(bf16* base, int r, int chunk) {
  return base + (chunk >> 3) * (ROWS * 64) + r * 64 + (((chunk & 7) ^ (r & 7)) << 3);
}

// Stage one K or V tile (kTileTok tokens x D) of kv head g into shared memory.
template <int D, bool FP8>
__device__ __forceinline__ void load_kv_tile(bf16* dst, const AttnParams& p, const int* table, int g, int which,
                                             int tok0, int kv_len, float dq) {
  constexpr int CH = D / 8;
  const int rd = which ? p.Dv : p.D;
  const void* base = which ? p.vc : p.kc;
  for (int i = threadIdx.x; i < kTileTok * CH; i += kAttnThreads) {
    const int r = i / CH, c = i % CH;
    const int tok = tok0 + r;
    bf16* d = tile_ptr<D, kTileTok>(dst, r, c);
    if (tok < kv_len && c * 8 < rd) {
      const int blk = table[tok / p.block_tokens];
      const size_t off = static_cast<size_t>(blk) * p.block_stride +
                         (static_cast<size_t>(g) * p.block_tokens + tok % p.block_tokens) * rd + c * 8;
      if (FP8) {
        const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const uint8_t*>(base) + off);
        const uint8_t* b = reinterpret_cast<const uint8_t*>(&raw);
        uint4 o;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __half_raw h0 = __nv_cvt_fp8_to_halfraw(b[2 * e], __NV_E4M3);
          const __half_raw h1 = __nv_cvt_fp8_to_halfraw(b[2 * e + 1], __NV_E4M3);
          ow[e] = pack_bf16(__half2float(__half(h0)) * dq, __half2float(__half(h1)) * dq);
        }
        *reinterpret_cast<uint4*>(d) = o;
      } else {
        cp_async16(d, static_cast<const bf16*>(base) + off);
      }
    } else {
      *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
    }
  }
}

// TMA staging of one K + V tile (one thread; `shared`: the keys are the values, one tile): a box of [block_tokens rows x 64
// columns] per cache block and 64-column panel. Tokens past kv_len inside the last block are loaded as they are (finite cache contents)
// and masked by the softmax; blocks past the sequence are not loaded at all.
template <int D>
__device__ __forceinline__ void tma_issue_kv(bf16* ks, bf16* vs, bool shared, uint64_t* bar, const CUtensorMap* kmap, const CUtensorMap* vmap,
                                             const AttnParams& p, const int* table, int g, int tok0, int kv_len) {
  const int bt = p.block_tokens;
  const int nblk = min(kTileTok / bt, (kv_len - tok0 + bt - 1) / bt);
  constexpr int PANELS = D / 64;
  mbar_expect_tx(bar, static_cast<uint32_t>(nblk) * (shared ? 1 : 2) * PANELS * bt * 128);
  for (int b = 0; b < nblk; ++b) {
    const int blk = table[tok0 / bt + b];
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      if (which && shared) break;
      bf16* dst = which ? vs : ks;
#pragma unroll
      for (int h = 0; h < PANELS; ++h)      // columns past the row's end arrive as zeros
        tma_load_3d(dst + h * (kTileTok * 64) + b * bt * 64, which ? vmap : kmap, bar, h * 64, g * bt, blk);
    }
  }
}

// After a TMA-staged tile has landed: zero the V rows of tokens past the sequence end (rows of blocks that were
// not loaded hold stale shared memory, rows past kv_len inside the last block hold whatever the cache has there);
// their probabilities are exactly 0, but 0 x NaN would poison the output. K needs nothing: its scores are masked.
template <int D>
__device__ __forceinline__ void zero_v_tail(bf16* vs, int valid_rows) {
  if (valid_rows >= kTileTok) return;
  constexpr int CH = D / 8;
  const int n = (kTileTok - valid_rows) * CH;
  for (int i = threadIdx.x; i < n; i += kAttnThreads) {
    const int r = valid_rows + i / CH, c = i % CH;
    *reinterpret_cast<uint4*>(tile_ptr<D, kTileTok>(vs, r, c)) = make_uint4(0, 0, 0, 0);
  }
}

// One warp: S(16 x NT*8 tokens) = Q(16 x D) K^T over tokens [t0, t0 + NT*8) of the staged tile.
template <int D, int NT>
__device__ __forceinline__ void warp_qk(float (&s)[NT][4], const uint32_t (&qf)[D / 16][4], bf16* ks, int t0, int lane) {
#pragma unroll
  for (int j = 0; j < NT; ++j) { s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f; }
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
    for (int jp = 0; jp < NT / 2; ++jp) {
      uint32_t b[4];
      const int r = t0 + jp * 16 + (lane & 7) + ((lane >> 4) << 3);
      const int c = kk * 2 + ((lane >> 3) & 1);
      ldsm_x4(b, smem_addr(tile_ptr<D, kTileTok>(ks, r, c)));
      mma16816(s[2 * jp], qf[kk], b[0], b[1]);
      mma16816(s[2 * jp + 1], qf[kk], b[2], b[3]);
    }
  }
}

// One warp: O(16 x D) += P(16 x NT*8) V over tokens [t0, t0 + NT*8).
template <int D, int NT>
__device__ __forceinline__ void warp_pv(float (&o)[D / 8][4], const float (&s)[NT][4], bf16* vs, int t0, int lane) {
#pragma unroll
  for (int kk = 0; kk < NT / 2; ++kk) {
    uint32_t a[4];
    a[0] = pack_bf16(s[2 * kk][0], s[2 * kk][1]);
    a[1] = pack_bf16(s[2 * kk][2], s[2 * kk][3]);
    a[2] = pack_bf16(s[2 * kk + 1][0], s[2 * kk + 1][1]);
    a[3] = pack_bf16(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      uint32_t b[4];
      const int r = t0 + kk * 16 + (lane & 7) + (((lane >> 3) & 1) << 3);
      const int c = np * 2 + (lane >> 4);
      ldsm_x4_t(b, smem_addr(tile_ptr<D, kTileTok>(vs, r, c)));
      mma16816(o[2 * np], a, b[0], b[1]);
      mma16816(o[2 * np + 1], a, b[2], b[3]);
    }
  }
}

// Mask + online-softmax update for one warp's 16 x (NT*8) score tile.
// Rows lane/4 and lane/4+8; limit[i] = last visible kv position of that row (-1 = row inactive), lo[i] = first position
// inside its window (tokens below `keep` are seen as well).
// PERM: column 2t + e of an 8-token group is token t + 4e (the FP8 form's order).
template <int D, int NT, bool PERM = false>
__device__ __forceinline__ void softmax_update(float (&s)[NT][4], float (&o)[D / 8][4], float (&m)[2], float (&l)[2],
                                               const int (&limit)[2], const int (&lo)[2], int keep, const float (&slope)[2],
                                               int tok0, int lane, const float (&scale_log2)[2]) {
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < NT; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = e >> 1;
      const int tok = tok0 + j * 8 + (PERM ? (lane & 3) + (e & 1) * 4 : (lane & 3) * 2 + (e & 1));
      float v = s[j][e] * scale_log2[i];
      if (slope[i] != 0.f) v += slope[i] * 1.44269504f * static_cast<float>(tok - limit[i]);
      v = (tok <= limit[i] && (tok >= lo[i] || tok < keep)) ? v : -INFINITY;
      s[j][e] = v;
      mx[i] = fmaxf(mx[i], v);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
  }
  float corr[2], mnew[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    mnew[i] = fmaxf(m[i], mx[i]);
    corr[i] = (mnew[i] == -INFINITY) ? 1.f : exp2f(m[i] - mnew[i]);
    m[i] = mnew[i];
    l[i] *= corr[i];
  }
  if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {      // most tiles leave every row's maximum as it was
#pragma unroll
    for (int n = 0; n < D / 8; ++n) { o[n][0] *= corr[0]; o[n][1] *= corr[0]; o[n][2] *= corr[1]; o[n][3] *= corr[1]; }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = e >> 1;
      const float pv = (mnew[i] == -INFINITY) ? 0.f : exp2f(s[j][e] - mnew[i]);
      s[j][e] = pv;
      l[i] += pv;   // per-thread partial; reduced over the 4 lanes of a row at the end
    }
  }
}

// Independent weights for one warp's 16 x (NT*8) score tile; bias[i]: the bias row of row i's head.
template <int NT>
__device__ __forceinline__ void sigmoid_weights(float (&s)[NT][4], const int (&limit)[2], const int (&lo)[2], int keep,
                                                const float* const (&bias)[2], int bias_last, int tok0, int lane, float scale_log2) {
#pragma unroll
  for (int j = 0; j < NT; ++j) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = e >> 1;
      const int tok = tok0 + j * 8 + (lane & 3) * 2 + (e & 1);
      const bool seen = tok <= limit[i] && (tok >= lo[i] || tok < keep);
      const float b = seen ? bias[i][min(limit[i] - tok, bias_last)] : 0.f;
      s[j][e] = seen ? 1.f / (1.f + exp2f(-fmaf(s[j][e], scale_log2, b * 1.44269504f))) : 0.f;
    }
  }
}

// factor of an output element: sigmoid of its gate
__device__ __forceinline__ float gate_of(const AttnParams& p, long long row, int col) {
  return p.gate ? p.out_factor / (1.f + exp2f(-1.44269504f * __bfloat162float(p.gate[row * p.gate_stride + col]))) : 1.f;
}

// exp(sink - m) of the softmax denominator; m is the row's reference maximum in the log2 domain
__device__ __forceinline__ float sink_term(const AttnParams& p, int head, float m) {
  return (p.sinks && m != -INFINITY) ? exp2f(p.sinks[head] * 1.44269504f - m) : 0.f;
}

// ----------------------------------------------------------------------------- prefill
template <int D, int MODE, bool SIG>
__global__ void __launch_bounds__(kAttnThreads)
paged_prefill_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, const AttnParams p) {
  constexpr bool FP8 = MODE == kKvFp8;
  constexpr int kKvStages = kv_stages(D);
  extern __shared__ uint8_t smem_attn_raw[];
  uint8_t* smem_attn = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_attn_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kKvStages];
  __shared__ uint32_t abort_word;
  bf16* qs = reinterpret_cast<bf16*>(smem_attn);            // 64 x D
  bf16* ks = qs + 64 * D;                                   // kKvStages x (64 x D)
  const bool shared = p.kc == p.vc;
  bf16* vs = shared ? ks : ks + kKvStages * kTileTok * D;   // kKvStages x (64 x D)

  const int s = blockIdx.z, g = blockIdx.y;
  const int G = p.Hq / p.Hkv;
  const int q0 = p.cu_q[s], q_len = p.cu_q[s + 1] - q0;
  const int kv_len = p.kv_lens[s];
  const int row0 = blockIdx.x * 64;
  if (row0 >= q_len * G) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* table = p.block_table + static_cast<size_t>(s) * p.table_stride;
  const int past = kv_len - q_len;   // tokens already in the cache before this chunk

  // stage Q rows (zero for rows beyond the sequence)
  constexpr int CH = D / 8;
  for (int i = threadIdx.x; i < 64 * CH; i += kAttnThreads) {
    const int r = i / CH, c = i % CH;
    const int vr = row0 + r;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (vr < q_len * G && c * 8 < p.D) {
      const int tok = vr / G, head = g * G + vr % G;
      v = *reinterpret_cast<const uint4*>(p.q + static_cast<size_t>(q0 + tok) * p.q_stride + head * p.D + c * 8);
    }
    *reinterpret_cast<uint4*>(tile_ptr<D, 64>(qs, r, c)) = v;
  }
  // causal bound of this CTA's rows
  const int last_row = min(row0 + 63, q_len * G - 1);
  const int kv_end = min(kv_len, past + last_row / G + 1);
  const TileRange tiles = visited_tiles(p.window > 0 ? past + row0 / G - p.window + 1 : 0, p.keep, (kv_end + kTileTok - 1) / kTileTok,
                                        kTileTok);
  const int ntiles = tiles.count;

  if (MODE == kKvTma && threadIdx.x == 0) {
    for (int i = 0; i < kKvStages; ++i) mbar_init(&full_bar[i], 1);
    abort_word = 0;
    mbar_fence_init();
  }
  __syncthreads();
  auto issue = [&](int t) {      // cp.async modes always commit a group so that the wait counts stay uniform
    const int st = t % kKvStages, tok0 = tile_at(tiles, t) * kTileTok;
    if (MODE == kKvTma) {
      if (threadIdx.x == 0 && t < ntiles)
        tma_issue_kv<D>(ks + st * kTileTok * D, vs + st * kTileTok * D, shared, &full_bar[st], &k_map, &v_map, p, table, g, tok0, kv_len);
      return;
    }
    if (t < ntiles) {
      load_kv_tile<D, FP8>(ks + st * kTileTok * D, p, table, g, 0, tok0, kv_len, p.k_scale);
      if (!shared) load_kv_tile<D, FP8>(vs + st * kTileTok * D, p, table, g, 1, tok0, kv_len, p.v_scale);
    }
    cp_commit();
  };
#pragma unroll
  for (int i = 0; i < kKvStages - 1; ++i) issue(i);
  __syncthreads();

  uint32_t qf[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const int r = warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3);
    const int c = kk * 2 + (lane >> 4);
    ldsm_x4(qf[kk], smem_addr(tile_ptr<D, 64>(qs, r, c)));
  }
  int limit[2], lo[2]; float slope[2];
  const float* bias[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int vr = row0 + warp * 16 + (lane >> 2) + i * 8;
    limit[i] = vr < q_len * G ? past + vr / G : -1;
    lo[i] = p.window > 0 ? limit[i] - p.window + 1 : 0;
    slope[i] = (p.alibi && vr < q_len * G) ? p.alibi[g * G + vr % G] : 0.f;
    bias[i] = SIG ? p.bias + static_cast<size_t>(g * G + vr % G) * p.bias_len : nullptr;
  }
  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  const float sl2[2] = {p.scale_log2, p.scale_log2};

  bool ok = true;
  for (int t = 0; t < ntiles; ++t) {
    const int buf = t % kKvStages, tok0 = tile_at(tiles, t) * kTileTok;
    if (MODE == kKvTma) {
      if (!mbar_wait(&full_bar[buf], (t / kKvStages) & 1, &abort_word)) { ok = false; break; }
      zero_v_tail<D>(vs + buf * kTileTok * D, kv_len - tok0);
    } else {
      cp_wait<kKvStages - 2>();   // tile t has landed (only newer groups may still be in flight)
    }
    __syncthreads();              // ... for every thread, and everyone is done with tile t-1
    issue(t + kKvStages - 1);     // refill the stage tile t-1 used
    float sc[8][4];
    warp_qk<D, 8>(sc, qf, ks + buf * kTileTok * D, 0, lane);
    if constexpr (SIG) sigmoid_weights<8>(sc, limit, lo, p.keep, bias, p.bias_len - 1, tok0, lane, p.scale_log2);
    else softmax_update<D, 8>(sc, o, m, l, limit, lo, p.keep, slope, tok0, lane, sl2);
    warp_pv<D, 8>(o, sc, vs + buf * kTileTok * D, 0, lane);
  }
  if (!ok) {                      // a bounded wait gave up: leave the output untouched, report through the error word
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 4);
    return;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int vr = row0 + warp * 16 + (lane >> 2) + i * 8;
    if (vr >= q_len * G) continue;
    const int tok = vr / G, head = g * G + vr % G;
    l[i] += sink_term(p, head, m[i]);
    const float inv = SIG ? 1.f : l[i] > 0.f ? 1.f / l[i] : 0.f;
    bf16* dst = p.out + static_cast<size_t>(q0 + tok) * p.out_stride + head * p.Dv + (lane & 3) * 2;
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      if (n * 8 < p.Dv) {
        float a = o[n][2 * i] * inv, b = o[n][2 * i + 1] * inv;
        if (SIG && p.gate) {
          const int col = head * p.Dv + (lane & 3) * 2 + n * 8;
          a *= gate_of(p, q0 + tok, col);
          b *= gate_of(p, q0 + tok, col + 1);
        }
        *reinterpret_cast<uint32_t*>(dst + n * 8) = pack_bf16(a, b);
      }
    }
  }
}

// ------------------------------------------------------------------------------ decode, caches that TMA cannot read
// grid (Hkv x row groups, B, splits). Rows = up to 16 of the G query heads of kv head g, one new token each.
template <int D, int MODE, bool SIG>
__global__ void __launch_bounds__(kAttnThreads)
paged_decode_kernel(const AttnParams p) {
  constexpr bool FP8 = MODE == kKvFp8;
  constexpr int kKvStages = kv_stages(D);
  extern __shared__ uint8_t smem_attn_raw[];
  uint8_t* smem_attn = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_attn_raw) + 1023) & ~uintptr_t(1023));
  __shared__ float red4[4];
  bf16* qs = reinterpret_cast<bf16*>(smem_attn);            // 16 x D
  bf16* ks = qs + 16 * D;                                   // kKvStages x (64 x D)
  const bool shared = p.kc == p.vc;
  bf16* vs = shared ? ks : ks + kKvStages * kTileTok * D;
  float* merge = reinterpret_cast<float*>(ks);              // 4 warps x 16 rows x (D + 2), reuses the K ring after the loop

  pdl_trigger();
  pdl_wait();
  const int GA = p.Hq / p.Hkv, groups = (GA + 15) / 16;
  const int g = blockIdx.x / groups, head0 = g * GA + (blockIdx.x % groups) * 16;
  const int G = min(16, (g + 1) * GA - head0);               // query heads of this CTA: head0 .. head0 + G
  const int s = blockIdx.y, split = blockIdx.z;
  const int kv_len = p.kv_lens[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int* table = p.block_table + static_cast<size_t>(s) * p.table_stride;
  const int win_lo = p.window > 0 ? kv_len - p.window : 0;
  const TileRange tiles = visited_tiles(win_lo, p.keep, (kv_len + kTileTok - 1) / kTileTok, kTileTok);
  const int total_tiles = tiles.count;
  const int tiles_per = (total_tiles + p.num_splits - 1) / p.num_splits;
  const int t_begin = split * tiles_per, t_end = min(total_tiles, t_begin + tiles_per);

  constexpr int CH = D / 8;
  for (int i = threadIdx.x; i < 16 * CH; i += kAttnThreads) {
    const int r = i / CH, c = i % CH;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < G && c * 8 < p.D)
      v = *reinterpret_cast<const uint4*>(p.q + static_cast<size_t>(s) * p.q_stride + (head0 + r) * p.D + c * 8);
    *reinterpret_cast<uint4*>(tile_ptr<D, 16>(qs, r, c)) = v;
  }
  float* bias_s = reinterpret_cast<float*>(ks + decode_ring(D, shared));
  if (SIG && p.bias_smem)
    for (int i = threadIdx.x; i < G * p.bias_len; i += kAttnThreads) bias_s[i] = p.bias[static_cast<size_t>(head0) * p.bias_len + i];
  __syncthreads();
  auto issue = [&](int t) {
    const int st = (t - t_begin) % kKvStages, tok0 = tile_at(tiles, t) * kTileTok;
    if (t < t_end) {
      load_kv_tile<D, FP8>(ks + st * kTileTok * D, p, table, g, 0, tok0, kv_len, p.k_scale);
      if (!shared) load_kv_tile<D, FP8>(vs + st * kTileTok * D, p, table, g, 1, tok0, kv_len, p.v_scale);
    }
    cp_commit();
  };
#pragma unroll
  for (int i = 0; i < kKvStages - 1; ++i) issue(t_begin + i);
  __syncthreads();
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const int r = (lane & 7) + (((lane >> 3) & 1) << 3);
    const int c = kk * 2 + (lane >> 4);
    ldsm_x4(qf[kk], smem_addr(tile_ptr<D, 16>(qs, r, c)));
  }
  int limit[2], lo[2]; float slope[2];
  const float* bias[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = (lane >> 2) + i * 8;
    limit[i] = r < G ? kv_len - 1 : -1;
    lo[i] = win_lo;
    slope[i] = (p.alibi && r < G) ? p.alibi[head0 + r] : 0.f;
    bias[i] = !SIG ? nullptr : (p.bias_smem ? bias_s : p.bias + static_cast<size_t>(head0) * p.bias_len) + (r < G ? r : 0) * p.bias_len;
  }
  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  if (SIG) { m[0] = m[1] = 0.f; }            // nothing is rescaled when partial sums are merged

  const float sl2[2] = {p.scale_log2, p.scale_log2};
  for (int t = t_begin; t < t_end; ++t) {
    const int buf = (t - t_begin) % kKvStages, tok0 = tile_at(tiles, t) * kTileTok;
    cp_wait<kKvStages - 2>();
    __syncthreads();
    issue(t + kKvStages - 1);
    float sc[2][4];
    warp_qk<D, 2>(sc, qf, ks + buf * kTileTok * D, warp * 16, lane);
    if constexpr (SIG) sigmoid_weights<2>(sc, limit, lo, p.keep, bias, p.bias_len - 1, tok0 + warp * 16, lane, p.scale_log2);
    else softmax_update<D, 2>(sc, o, m, l, limit, lo, p.keep, slope, tok0 + warp * 16, lane, sl2);
    warp_pv<D, 2>(o, sc, vs + buf * kTileTok * D, warp * 16, lane);
  }
  cp_wait<0>();
  __syncthreads();                // the merge area aliases the K ring: every warp must be out of the loop
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  // merge the 4 warps' streams: stage (m, l, O) per warp, then every thread combines a slice
  constexpr int MS = D + 2;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = (lane >> 2) + i * 8;
    float* dst = merge + (warp * 16 + r) * MS;
    if ((lane & 3) == 0) { dst[D] = m[i]; dst[D + 1] = l[i]; }
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      dst[n * 8 + (lane & 3) * 2] = o[n][2 * i];
      dst[n * 8 + (lane & 3) * 2 + 1] = o[n][2 * i + 1];
    }
  }
  __syncthreads();
  const int Dv = p.Dv;
  for (int i = threadIdx.x; i < G * Dv; i += kAttnThreads) {
    const int r = i / Dv, d = i % Dv;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, merge[(w * 16 + r) * MS + D]);
    float acc = 0.f, ll = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float* src = merge + (w * 16 + r) * MS;
      const float f = (src[D] == -INFINITY) ? 0.f : exp2f(src[D] - mm);
      acc += src[d] * f;
      ll += src[D + 1] * f;
    }
    const int head = head0 + r;
    if (p.num_splits == 1) {
      ll += sink_term(p, head, mm);
      const float v = SIG ? acc * gate_of(p, s, head * Dv + d) : ll > 0.f ? acc / ll : 0.f;
      if constexpr (D == 128) {
        if (p.outq) { store_head_row_q(p, s, head, d, v, red4); continue; }   // (Dv == blockDim: r is uniform per pass)
      }
      p.out[static_cast<size_t>(s) * p.out_stride + head * Dv + d] = __float2bfloat16(v);
    } else {
      const size_t base = (static_cast<size_t>(s) * p.Hq + head) * p.num_splits + split;
      p.part_o[base * Dv + d] = acc;
      if (d == 0) { p.part_ml[base * 2] = mm; p.part_ml[base * 2 + 1] = ll; }
    }
  }
}

// ------------------------------------------------------------------------------ decode, stream form
// Bound by HBM (every K/V byte is read once). A grid of one CTA per (head, sequence, split) of equal split counts left
// the longest sequences of a ragged batch and a nearly empty last wave to a few CTAs; here the units are cut evenly, whatever the
// lengths, and an item (sequence, kv head row group) that lies in several CTAs' ranges is summed by the CTA that delivers
// its last piece, so there is no second launch either. A warp of its own issues the TMA boxes (block table entries
// read by its lanes in parallel), which took the table's latency out of the compute warps' path. Per layer: 64 ragged sequences of
// 100-3000 tokens (32/8 heads) 76 -> 46 us; 64 sequences, 64/8 heads 130 -> 102; e4m3 cache, 12 sequences 603 -> 58, which came
// through registers before.
constexpr int kStreamThreads = 160;      // 4 warps that compute, 1 that loads
constexpr int kStreamMaxStages = 8;
// What an item costs beside its tiles (its query rows, the merge of the warps, the piece that is handed over), in tiles: the line that
// is cut has so many empty units behind every item.
constexpr int kStreamItemUnits = 2;
// What a piece of a cut item costs beyond that, in tiles (its sums out and in again, a fence, the arrival); and what the even cut costs,
// whose CTAs have a second, shorter piece before or behind the first and some more to compute.
constexpr int kStreamPieceUnits = 3;
constexpr int kStreamCutUnits = 10;

__device__ __forceinline__ void stream_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

struct StreamItem { int s, h, t0, t1, n, units; };     // tiles [t0, t1) of the n tiles of sequence s, row group h; units taken of the line

// the item of unit u (t0 = t1: only the empty units behind its tiles); `s` only ever moves forward
__device__ __forceinline__ void stream_item(const int* first, int heads, long long u, long long end, int& s, StreamItem& it) {
  while (static_cast<long long>(first[s + 1]) * heads <= u) ++s;
  const int n = first[s + 1] - first[s];
  const long long r = u - static_cast<long long>(first[s]) * heads;
  it.s = s; it.n = n - kStreamItemUnits;
  it.h = r < (1LL << 31) ? static_cast<int>(r) / n : static_cast<int>(r / n);
  const int at = static_cast<int>(r - static_cast<long long>(it.h) * n);
  const long long room = end - u;
  it.units = room < n - at ? static_cast<int>(room) : n - at;
  it.t0 = min(at, it.n);
  it.t1 = min(at + it.units, it.n);
}

__device__ __forceinline__ TileRange decode_tiles(const AttnParams& p, int kv_len) {
  return visited_tiles(p.window > 0 ? kv_len - p.window : 0, p.keep, (kv_len + kTileTok - 1) / kTileTok, kTileTok);
}

__device__ __forceinline__ void mma16816_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// four e4m3 values as two f16 pairs, exactly
__device__ __forceinline__ void f16_of_e4m3(uint32_t w, uint32_t& low, uint32_t& high) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, h;\n\t}"
      : "=r"(low), "=r"(high) : "r"(w));
}
// token of column i of an 8-token group: neighbours lie four rows apart, so that the 16-byte reads of eight lanes (two
// tokens, four chunks each) fall on different banks of the 128-byte-swizzled tile
__device__ __forceinline__ int perm8(int i) { return (i >> 1) | ((i & 1) << 2); }

// One warp, FP8 tile (rows of 128 bytes): S(16 x 16 tokens) = Q K^T. The dimensions are taken in an order of their own: lane t of a
// row holds dimensions 16 (4 h + t) + 4 w .. + 3 of step (h, w), which is what one 16-byte read of a key row gives.
__device__ __forceinline__ void warp_qk_fp8(float (&s)[2][4], const uint32_t (&qf)[8][4], const uint8_t* ks, int t0, int lane) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    const int r7 = perm8(lane >> 2);
    const uint8_t* row = ks + (t0 + j * 8 + r7) * 128;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + (((h * 4 + (lane & 3)) ^ r7) << 4));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t b0, b1;
        f16_of_e4m3(w[k], b0, b1);
        mma16816_f16(s[j], qf[h * 4 + k], b0, b1);
      }
    }
  }
}

// One warp, FP8 tile: O(16 x 128) += P(16 x 16 tokens) V. Pairs of dimensions travel as one 16-bit element through the transposing
// load; o[2 c] holds the even and o[2 c + 1] the odd dimensions of chunk c: columns 4t, 4t + 2 and 4t + 1, 4t + 3.
__device__ __forceinline__ void warp_pv_fp8(float (&o)[16][4], const float (&s)[2][4], const uint8_t* vs, int t0, int lane) {
  const uint32_t a[4] = {pack_f16(s[0][0], s[0][1]), pack_f16(s[0][2], s[0][3]), pack_f16(s[1][0], s[1][1]), pack_f16(s[1][2], s[1][3])};
  const int r7 = perm8(lane & 7);
  const uint8_t* row = vs + (t0 + ((lane >> 3) & 1) * 8 + r7) * 128;
#pragma unroll
  for (int c2 = 0; c2 < 4; ++c2) {
    uint32_t b[4];
    ldsm_x4_t(b, smem_addr(row + (((c2 * 2 + (lane >> 4)) ^ r7) << 4)));
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t e0, o0, e1, o1;
      f16_of_e4m3(__byte_perm(b[2 * c], 0, 0x3120), e0, o0);
      f16_of_e4m3(__byte_perm(b[2 * c + 1], 0, 0x3120), e1, o1);
      mma16816_f16(o[(c2 * 2 + c) * 2], a, e0, e1);
      mma16816_f16(o[(c2 * 2 + c) * 2 + 1], a, o0, o1);
    }
  }
}

// Four consecutive outputs of one head row (a warp per row, lane's columns d .. d + 3 of Dv); `q`: D = 128 as the next GEMM's FP8
// operand, quantised from the bf16-rounded values exactly as the stand-alone quantiser would.
template <int D, bool SIG>
__device__ __forceinline__ void store_head_row4(const AttnParams& p, int s, int head, int d, float4 v) {
  const bool on = d < p.Dv;
  if (SIG && p.gate && on) {
    const int col = head * p.Dv + d;
    v.x *= gate_of(p, s, col); v.y *= gate_of(p, s, col + 1); v.z *= gate_of(p, s, col + 2); v.w *= gate_of(p, s, col + 3);
  }
  const uint2 w = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  if (p.out && on) {
    bf16* dst = p.out + static_cast<size_t>(s) * p.out_stride + head * p.Dv + d;
    if (p.vec_out) {
      *reinterpret_cast<uint2*>(dst) = w;
    } else {
      dst[0] = __float2bfloat16(v.x); dst[1] = __float2bfloat16(v.y); dst[2] = __float2bfloat16(v.z); dst[3] = __float2bfloat16(v.w);
    }
  }
  if constexpr (D == 128) {
    if (p.outq) {                                                     // Dv = 128: every lane of the warp holds four columns
      const float f[4] = {__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                          __uint_as_float(w.y & 0xffff0000u)};
      float am = fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fmaxf(fabsf(f[2]), fabsf(f[3])));
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, x));
      const float sc = fp8_group_scale(am), inv = 1.f / sc;
      uint32_t q = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        q |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(f[e] * inv, __NV_SATFINITE, __NV_E4M3)) << (8 * e);
      uint8_t* dst = p.outq + (static_cast<size_t>(s) * p.Hq + head) * 128 + d;
      if (p.vec_out) {
        *reinterpret_cast<uint32_t*>(dst) = q;
      } else {
        for (int e = 0; e < 4; ++e) dst[e] = static_cast<uint8_t>(q >> (8 * e));
      }
      if (d == 0) p.oscale[static_cast<size_t>(head) * p.oscale_ld + s] = sc;
    }
  }
}

template <int D, int MODE, bool SIG>
__global__ void __launch_bounds__(kStreamThreads, D <= 64 ? 3 : D <= 128 ? 2 : 1)
paged_decode_stream_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, const AttnParams p) {
  constexpr bool FP8 = MODE == kKvTmaFp8;
  static_assert(!FP8 || (D == 128 && !SIG), "FP8 tiles have rows of 128 bytes");
  constexpr int kTileBytes = kTileTok * D * (FP8 ? 1 : 2);
  extern __shared__ uint8_t smem_attn_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_attn_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kStreamMaxStages], empty_bar[kStreamMaxStages];
  __shared__ uint32_t abort_word, last_piece;
  __shared__ float ml_s[4][16][2];
  __shared__ long long line_s[2];                 // units and CTAs of an even cut: read where a cut item is summed, not held in registers
  __shared__ int piece_s[2];                      // this CTA's piece of its item and the tiles of a piece (0: the even cut)
  const bool shared = p.kc == p.vc;
  // the merge area is the consumed last stage of an item where that is large enough, else one of its own behind the ring
  const bool own_merge = FP8 || shared;
  uint8_t* behind = ring + p.stages * p.stage_bytes;
  float* merge_own = reinterpret_cast<float*>(behind);
  float* bias_s = reinterpret_cast<float*>(behind + (own_merge ? 4 * p.rows * D * 4 : 0));
  int* first = reinterpret_cast<int*>(bias_s + p.bias_smem);            // [B + 1] tiles before each sequence

  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int GA = p.Hq / p.Hkv, groups = (GA + 15) / 16, heads = p.Hkv * groups;
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 4); }
    abort_word = 0;
    mbar_fence_init();
    first[0] = 0;
  }
  // tiles of every sequence (at least one: an empty sequence's rows are written too), prefix sums; every warp computes them for
  // itself, so that one barrier is all the set-up waits for
  int before = 0, longest = 0;
#pragma unroll 4
  for (int s0 = 0; s0 < p.B; s0 += 32) {
    const int s = s0 + lane;
    int x = s < p.B ? max(1, decode_tiles(p, p.kv_lens[s]).count) + kStreamItemUnits : 0;
    longest = max(longest, x);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (s < p.B) first[s + 1] = before + x;                              // the same value from every warp
    before += __shfl_sync(0xffffffffu, x, 31);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  __syncthreads();
  // How the line is shared out: cut evenly, or by items. By items, a CTA takes a run of whole ones, or where there are CTAs enough one of
  // the `m` pieces of `per` tiles of one. The model counts units on the longest path. Even cut / by items (us): 1 sequence of 517 tokens
  // 10.1 / 9.3, 25 of 194 (40/8 heads) 16.8 / 10.8, 34 of 51-103 (20/4 heads of 192) 18.2 / 9.1, 18 of 3079 50.3 / 44.5, 9 of 9558 66.5 /
  // 62; ragged or uneven: 64 of 100-3000 47.5 / 100, 41 of 600 (20/4 heads of 192) 30.8 / 36.1, 128 of 100-400 38.0 / 43.7.
  const long long U = static_cast<long long>(before) * heads;
  const long long I = static_cast<long long>(p.B) * heads, grid = gridDim.x;
  const long long p_cut = U < grid ? U : grid;
  const bool can_cut = p.counters != nullptr, few = I <= grid;
  const int most = longest - kStreamItemUnits;
  int per = most, m = 1;
  if (few && can_cut) {
    const int share = static_cast<uint32_t>(grid) / static_cast<uint32_t>(I);
    const int part = max(2, (most + share - 1) / share);
    if (part + kStreamPieceUnits < most) { per = part; m = (most + per - 1) / per; }
  }
  const long long item_units = few ? per + kStreamItemUnits + (m > 1 ? kStreamPieceUnits : 0) : (I + grid - 1) / grid * longest;
  const bool cuts = can_cut && item_units * p_cut > U + kStreamCutUnits * p_cut;
  const bool by_piece = !cuts && few;
  const long long P = cuts ? p_cut : by_piece ? I * m : grid;
  const long long c = blockIdx.x;
  if (c >= P) return;
  const bool narrow = U * grid < (1LL << 32);                          // 64-bit divisions cost a tenth of a short launch
  auto mul_div = [](long long x, long long y, long long z, bool narrow) -> long long {
    return narrow ? static_cast<uint32_t>(x * y) / static_cast<uint32_t>(z) : x * y / z;
  };
  auto item_start = [&](long long i) -> long long {
    const int s = narrow ? static_cast<int>(static_cast<uint32_t>(i) / static_cast<uint32_t>(heads)) : static_cast<int>(i / heads);
    return static_cast<long long>(first[s]) * heads + (i - static_cast<long long>(s) * heads) * (first[s + 1] - first[s]);
  };
  auto begin_of = [&](long long k) -> long long {
    if (cuts) return mul_div(k, U, P, narrow);
    const long long i = mul_div(k, I, P, narrow);                      // (I <= U)
    return i >= I ? U : item_start(i);
  };
  long long u_begin, u_end;
  int piece = 0, s_at = 0;                                               // sequence of u_begin
  if (by_piece) {
    const int i = static_cast<uint32_t>(c) / static_cast<uint32_t>(m);
    piece = static_cast<int>(c) - i * m;
    s_at = static_cast<uint32_t>(i) / static_cast<uint32_t>(heads);
    const int n = first[s_at + 1] - first[s_at];
    const int t0 = piece * per, t1 = min(t0 + per, n - kStreamItemUnits);
    if (t0 >= t1) return;                                              // (an item shorter than the longest)
    u_begin = item_start(i) + t0;
    u_end = u_begin + (t1 - t0);
  } else {
    u_begin = begin_of(c);
    u_end = begin_of(c + 1);
    for (int lo = 0, hi = p.B - 1; lo <= hi;) {
      const int mid = (lo + hi) / 2;
      if (static_cast<long long>(first[mid]) * heads <= u_begin) { s_at = mid; lo = mid + 1; } else hi = mid - 1;
    }
  }

  if (threadIdx.x == 0) {
    line_s[0] = U; line_s[1] = P;
    piece_s[0] = piece; piece_s[1] = by_piece ? per : 0;
  }

  if (warp == 4) {
    // ---- loads: a box of [block tokens x 64 columns] (FP8: x 128) per cache block and panel, spread over the lanes
    constexpr int PANELS = FP8 ? 1 : D / 64;
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    const int bt = p.block_tokens;
    StreamItem it;
    for (long long u = u_begin; u < u_end && ok; u += it.units) {
      stream_item(first, heads, u, u_end, s_at, it);
      if (it.t0 == it.t1) continue;
      const int kv_len = p.kv_lens[it.s], g = it.h / groups;
      const int* table = p.block_table + static_cast<size_t>(it.s) * p.table_stride;
      const TileRange tiles = decode_tiles(p, kv_len);
      for (int t = it.t0; t < it.t1 && ok; ++t) {
        const int tok0 = tile_at(tiles, t) * kTileTok;
        const int nblk = max(0, min(kTileTok / bt, (kv_len - tok0 + bt - 1) / bt));
        const int per_blk = (shared ? 1 : 2) * PANELS, boxes = nblk * per_blk;
        int blk = 0;
        if (lane < boxes) blk = table[tok0 / bt + lane / per_blk];
        ok = mbar_wait(&empty_bar[stage], phase ^ 1, &abort_word);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&full_bar[stage], static_cast<uint32_t>(boxes) * bt * 128);
        __syncwarp();
        for (int i = lane; i < boxes; i += 32) {
          if (i >= 32) blk = table[tok0 / bt + i / per_blk];
          const int j = i % per_blk, which = j / PANELS, h = j % PANELS;
          uint8_t* dst = ring + stage * p.stage_bytes + which * kTileBytes + h * (kTileTok * 128) + (i / per_blk) * bt * 128;
          tma_load_3d(dst, which ? &v_map : &k_map, &full_bar[stage], h * 64, g * bt, blk);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else {
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    StreamItem it;
    for (long long u = u_begin; u < u_end; u += it.units) {
      stream_item(first, heads, u, u_end, s_at, it);
      if (it.t0 == it.t1) continue;
      const int kv_len = p.kv_lens[it.s], s = it.s;
      const int g = it.h / groups, head0 = g * GA + (it.h % groups) * 16;
      const int G = min(16, (g + 1) * GA - head0);             // query heads of this item: head0 .. head0 + G
      const TileRange tiles = decode_tiles(p, kv_len);
      const int win_lo = p.window > 0 ? kv_len - p.window : 0;
      if (SIG && p.bias_smem) {
        stream_bar();                                          // the previous item's rows are no longer read
        for (int i = threadIdx.x; i < G * p.bias_len; i += 128) bias_s[i] = p.bias[static_cast<size_t>(head0) * p.bias_len + i];
        stream_bar();
      }
      // Q fragments straight from global memory (the loads of the item's first tiles are in flight meanwhile)
      uint32_t qf[D / 16][4];
      float sl2[2] = {p.scale_log2, p.scale_log2};
      int limit[2], lo[2]; float slope[2];
      const float* bias[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = (lane >> 2) + i * 8;
        limit[i] = r < G ? kv_len - 1 : -1;
        lo[i] = win_lo;
        slope[i] = (p.alibi && r < G) ? p.alibi[head0 + r] : 0.f;
        bias[i] = !SIG ? nullptr : (p.bias_smem ? bias_s : p.bias + static_cast<size_t>(head0) * p.bias_len) + (r < G ? r : 0) * p.bias_len;
        const bf16* src = p.q + static_cast<size_t>(s) * p.q_stride + static_cast<size_t>(head0 + r) * p.D;
        if constexpr (!FP8) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int col = kk * 16 + x * 8 + (lane & 3) * 2;
              qf[kk][x * 2 + i] = (r < G && col < p.D) ? *reinterpret_cast<const uint32_t*>(src + col) : 0u;
            }
        } else {
          // f16 rows scaled by a power of two to a largest magnitude in [1, 2): exact but for elements 2^14 below it, whose
          // rounding is smaller than that of the fp32 sums
          uint32_t w[2][8];
          float am = 0.f;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = (h * 4 + (lane & 3)) * 16;
            const bool on = r < G && col < p.D;
            const uint4 a = on ? *reinterpret_cast<const uint4*>(src + col) : make_uint4(0, 0, 0, 0);
            const uint4 b = on ? *reinterpret_cast<const uint4*>(src + col + 8) : make_uint4(0, 0, 0, 0);
            w[h][0] = a.x; w[h][1] = a.y; w[h][2] = a.z; w[h][3] = a.w; w[h][4] = b.x; w[h][5] = b.y; w[h][6] = b.z; w[h][7] = b.w;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              am = fmaxf(am, fmaxf(fabsf(__uint_as_float(w[h][k] << 16)), fabsf(__uint_as_float(w[h][k] & 0xffff0000u))));
          }
          am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
          am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
          const uint32_t e = min(max(__float_as_uint(am) >> 23, 1u), 250u);
          const float up = __uint_as_float((254u - e) << 23);
          sl2[i] = p.scale_log2 * p.k_scale * __uint_as_float(e << 23);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 8; ++k)
              qf[h * 4 + k / 2][(k & 1) * 2 + i] =
                  pack_f16(__uint_as_float(w[h][k] << 16) * up, __uint_as_float(w[h][k] & 0xffff0000u) * up);
        }
      }
      float o[D / 8][4];
#pragma unroll
      for (int n = 0; n < D / 8; ++n) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
      float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
      if (SIG) { m[0] = m[1] = 0.f; }                          // nothing is rescaled when partial sums are merged
      uint8_t* held = nullptr;                                 // stage of the item's last tile
      uint64_t* held_bar = nullptr;
      for (int t = it.t0; t < it.t1; ++t) {
        if (ok) ok = mbar_wait(&full_bar[stage], phase, &abort_word);
        uint8_t* kt = ring + stage * p.stage_bytes;
        uint8_t* vt = shared ? kt : kt + kTileBytes;
        const int tok0 = tile_at(tiles, t) * kTileTok, w0 = warp * 16;
        if (ok) {
          // V rows past the sequence's end (this warp's own): stale shared memory or whatever the cache holds there; their weights
          // are exactly 0, but 0 x NaN would poison the output. K needs nothing: its scores are masked.
          const int valid = kv_len - tok0 - w0;
          if (valid < 16) {
            for (int i = lane; i < 16 * (FP8 ? 8 : D / 8); i += 32) {
              const int r = i / (FP8 ? 8 : D / 8), ch = i % (FP8 ? 8 : D / 8);
              if (r < valid) continue;
              if constexpr (FP8) *reinterpret_cast<uint4*>(vt + (w0 + r) * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
              else *reinterpret_cast<uint4*>(tile_ptr<D, kTileTok>(reinterpret_cast<bf16*>(vt), w0 + r, ch)) = make_uint4(0, 0, 0, 0);
            }
            fence_async_smem();
            __syncwarp();
          }
          float sc[2][4];
          if constexpr (FP8) {
            warp_qk_fp8(sc, qf, kt, w0, lane);
            softmax_update<D, 2, true>(sc, o, m, l, limit, lo, p.keep, slope, tok0 + w0, lane, sl2);
            warp_pv_fp8(o, sc, vt, w0, lane);
          } else {
            warp_qk<D, 2>(sc, qf, reinterpret_cast<bf16*>(kt), w0, lane);
            if constexpr (SIG) sigmoid_weights<2>(sc, limit, lo, p.keep, bias, p.bias_len - 1, tok0 + w0, lane, p.scale_log2);
            else softmax_update<D, 2>(sc, o, m, l, limit, lo, p.keep, slope, tok0 + w0, lane, sl2);
            warp_pv<D, 2>(o, sc, reinterpret_cast<bf16*>(vt), w0, lane);
          }
        }
        if (t + 1 == it.t1 && !own_merge) {
          held = kt; held_bar = &empty_bar[stage];             // released after the merge
        } else {
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty_bar[stage]);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      // ---- the warps' sums: [4 warps][rows][D] floats, columns swizzled by row so that neither side conflicts
      float* merge = own_merge ? merge_own : reinterpret_cast<float*>(held);
      const int R = p.rows;
      stream_bar();                                            // every warp is done with the last tile
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        const int r = (lane >> 2) + i * 8;
        if (r < R) {
          if ((lane & 3) == 0) { ml_s[warp][r][0] = m[i]; ml_s[warp][r][1] = l[i]; }
          float* dst = merge + (warp * R + r) * D;
          const int x = (r & 7) << 3;
          if constexpr (FP8) {
#pragma unroll
            for (int ch = 0; ch < 8; ++ch)
              *reinterpret_cast<float4*>(dst + ((ch * 16 + (lane & 3) * 4) ^ x)) =
                  make_float4(o[2 * ch][2 * i] * p.v_scale, o[2 * ch + 1][2 * i] * p.v_scale, o[2 * ch][2 * i + 1] * p.v_scale,
                              o[2 * ch + 1][2 * i + 1] * p.v_scale);
          } else {
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
              *reinterpret_cast<float2*>(dst + ((n * 8 + (lane & 3) * 2) ^ x)) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
          }
        }
      }
      stream_bar();
      const bool whole = it.t1 - it.t0 == it.n;
      const long long slot = 2 * c + (u == u_begin ? 0 : 1);
      for (int r = warp; r < G; r += 4) {
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w) mm = fmaxf(mm, ml_s[w][r][0]);
        float f[4], ll = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          f[w] = ml_s[w][r][0] == -INFINITY ? 0.f : exp2f(ml_s[w][r][0] - mm);
          ll += ml_s[w][r][1] * f[w];
        }
        if (whole) ll += sink_term(p, head0 + r, mm);
        const float inv = SIG ? 1.f : ll > 0.f ? 1.f / ll : 0.f;
#pragma unroll
        for (int d0 = 0; d0 < D; d0 += 128) {
          const int d = d0 + lane * 4;
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
          if (d < D) {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const float4 v = *reinterpret_cast<const float4*>(merge + (w * R + r) * D + (d ^ ((r & 7) << 3)));
              acc.x += v.x * f[w]; acc.y += v.y * f[w]; acc.z += v.z * f[w]; acc.w += v.w * f[w];
            }
          }
          if (whole) {
            store_head_row4<D, SIG>(p, s, head0 + r, d, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
          } else if (d < p.Dv) {
            __stcg(reinterpret_cast<float4*>(p.cut_o + (slot * R + r) * p.Dv + d), acc);
          }
        }
        if (!whole && lane == 0) __stcg(reinterpret_cast<float2*>(p.cut_ml + (slot * R + r) * 2), make_float2(mm, ll));
      }
      if (!own_merge) {
        fence_async_smem();                                    // the stage goes back to the TMA ring
        __syncwarp();
        if (lane == 0) mbar_arrive(held_bar);
      }
      if (whole) continue;
      // ---- a cut item: whoever delivers the last piece adds them up, in their order along the line
      const int part = piece_s[1];
      long long cf, slot0;                                     // CTA and slot of its first piece
      int pieces;
      if (part) {
        cf = c - piece_s[0];
        slot0 = 2 * cf;
        pieces = (it.n + part - 1) / part;
      } else {
        const long long units = line_s[0], ctas = line_s[1], a = u - it.t0;        // a: the item's first unit
        const bool small = units * ctas < (1LL << 32);
        auto begin = [&](long long k) { return mul_div(k, units, ctas, small); };
        auto owner = [&](long long x) {
          long long k = mul_div(x, ctas, units, small);
          while (k + 1 < ctas && begin(k + 1) <= x) ++k;
          while (k > 0 && begin(k) > x) --k;
          return k;
        };
        cf = owner(a);
        slot0 = 2 * cf + (begin(cf) < a ? 1 : 0);
        pieces = static_cast<int>(owner(a + it.n - 1) - cf) + 1;
      }
      __threadfence();
      stream_bar();
      if (threadIdx.x == 0) {
        unsigned int* cnt = p.counters + static_cast<size_t>(s) * heads + it.h;
        const bool last = atomicAdd(cnt, 1u) + 1u == static_cast<unsigned int>(pieces);
        if (last) *cnt = 0;
        last_piece = last;
        __threadfence();
      }
      stream_bar();
      if (last_piece) {
        for (int r = warp; r < G; r += 4) {
          float mm = -INFINITY;
          for (int k = lane; k < pieces; k += 32) mm = fmaxf(mm, __ldcg(p.cut_ml + ((k ? 2 * (cf + k) : slot0) * R + r) * 2));
#pragma unroll
          for (int x = 16; x > 0; x >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, x));
          float ll = 0.f;
          constexpr int ND = (D + 127) / 128, NK = ND == 1 ? 8 : 4;      // pieces whose loads are in flight together
          float4 acc[ND];
#pragma unroll
          for (int j = 0; j < ND; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int k0 = 0; k0 < pieces; k0 += NK) {
            float2 ml[NK];
            float4 v[NK][ND];
#pragma unroll
            for (int k = 0; k < NK; ++k) {
              const long long sl = k0 + k ? 2 * (cf + k0 + k) : slot0;
              ml[k] = make_float2(-INFINITY, 0.f);
              if (k0 + k < pieces) ml[k] = __ldcg(reinterpret_cast<const float2*>(p.cut_ml + (sl * R + r) * 2));
#pragma unroll
              for (int j = 0; j < ND; ++j) {
                const int d = j * 128 + lane * 4;
                v[k][j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + k < pieces && d < p.Dv) v[k][j] = __ldcg(reinterpret_cast<const float4*>(p.cut_o + (sl * R + r) * p.Dv + d));
              }
            }
#pragma unroll
            for (int k = 0; k < NK; ++k) {
              const float f = ml[k].x == -INFINITY ? 0.f : exp2f(ml[k].x - mm);
              ll += ml[k].y * f;
#pragma unroll
              for (int j = 0; j < ND; ++j) {
                acc[j].x += v[k][j].x * f; acc[j].y += v[k][j].y * f; acc[j].z += v[k][j].z * f; acc[j].w += v[k][j].w * f;
              }
            }
          }
          ll += sink_term(p, head0 + r, mm);
          const float inv = SIG ? 1.f : ll > 0.f ? 1.f / ll : 0.f;
#pragma unroll
          for (int j = 0; j < (D + 127) / 128; ++j)
            store_head_row4<D, SIG>(p, s, head0 + r, j * 128 + lane * 4,
                                    make_float4(acc[j].x * inv, acc[j].y * inv, acc[j].z * inv, acc[j].w * inv));
        }
      }
    }
  }
  __syncthreads();
  if (abort_word) {                        // a bounded wait gave up: copies in flight land before the CTA's memory is reused
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 4);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
}

// grid (Hq, B): combine the per-split partials.
template <int D>
__global__ void decode_reduce_kernel(const AttnParams p) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red4[4];
  const int head = blockIdx.x, s = blockIdx.y;
  const size_t base = (static_cast<size_t>(s) * p.Hq + head) * p.num_splits;
  float mm = -INFINITY;
  for (int k = 0; k < p.num_splits; ++k) mm = fmaxf(mm, p.part_ml[(base + k) * 2]);
  const float sink = sink_term(p, head, mm);
  const int Dv = p.Dv;
  for (int d = threadIdx.x; d < Dv; d += blockDim.x) {
    float acc = 0.f, ll = 0.f;
    for (int k = 0; k < p.num_splits; ++k) {
      const float mk = p.part_ml[(base + k) * 2];
      const float f = (mk == -INFINITY) ? 0.f : exp2f(mk - mm);
      acc += p.part_o[(base + k) * Dv + d] * f;
      ll += p.part_ml[(base + k) * 2 + 1] * f;
    }
    ll += sink;
    const float v = p.bias ? acc * gate_of(p, s, head * Dv + d) : ll > 0.f ? acc / ll : 0.f;
    if constexpr (D == 128) {
      if (p.outq) { store_head_row_q(p, s, head, d, v, red4); continue; }     // 128 threads: one pass, every thread in it
    }
    p.out[static_cast<size_t>(s) * p.out_stride + head * Dv + d] = __float2bfloat16(v);
  }
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*AttnEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static AttnEncodeFn attn_encode_fn() {
  static AttnEncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) return nullptr;
    fn = reinterpret_cast<AttnEncodeFn>(ptr);
  }
  return fn;
}

// A K or V panel of every block seen as [block][row = head x token][D] bf16; box = one cache block's tokens x 64 columns,
// 128-byte swizzle. Columns past D arrive as zeros.
static bool make_kv_map(CUtensorMap* map, const void* panel, long long block_stride, int num_blocks, int Hkv, int D, int block_tokens) {
  AttnEncodeFn enc = attn_encode_fn();
  if (!enc) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(Hkv) * block_tokens, static_cast<cuuint64_t>(num_blocks)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(D) * 2, static_cast<cuuint64_t>(block_stride) * 2};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(block_tokens), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(panel), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same panel of e4m3 values: box = one cache block's tokens x 128 columns.
static bool make_kv_map_fp8(CUtensorMap* map, const void* panel, long long block_stride, int num_blocks, int Hkv, int D, int block_tokens) {
  AttnEncodeFn enc = attn_encode_fn();
  if (!enc) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(Hkv) * block_tokens, static_cast<cuuint64_t>(num_blocks)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(block_stride)};
  cuuint32_t box[3] = {128, static_cast<cuuint32_t>(block_tokens), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(panel), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether TMA reads the cache: block sizes that divide a tile, panels and strides on 16-byte boundaries.
static bool tma_covers(const AttnParams& p, int num_blocks, bool fp8) {
  const int bt = p.block_tokens, unit = fp8 ? 16 : 8;
  return (bt == 8 || bt == 16 || bt == 32 || bt == 64) && p.block_stride % unit == 0 && p.D % unit == 0 && p.Dv % unit == 0 &&
         num_blocks > 0 && !((reinterpret_cast<uintptr_t>(p.kc) | reinterpret_cast<uintptr_t>(p.vc)) & 15);
}

// The maps of both panels of such a cache.
static bool tma_maps(const AttnParams& p, int num_blocks, CUtensorMap* km, CUtensorMap* vm) {
  const int bt = p.block_tokens;
  if (!tma_covers(p, num_blocks, false)) return false;
  return make_kv_map(km, p.kc, p.block_stride, num_blocks, p.Hkv, p.D, bt) &&
         make_kv_map(vm, p.vc, p.block_stride, num_blocks, p.Hkv, p.Dv, bt);
}

static bool tma_maps_fp8(const AttnParams& p, int num_blocks, CUtensorMap* km, CUtensorMap* vm) {
  const int bt = p.block_tokens;
  if (!tma_covers(p, num_blocks, true)) return false;
  return make_kv_map_fp8(km, p.kc, p.block_stride, num_blocks, p.Hkv, p.D, bt) &&
         make_kv_map_fp8(vm, p.vc, p.block_stride, num_blocks, p.Hkv, p.Dv, bt);
}

template <int D, int MODE, bool SIG = false>
static int launch_prefill(const AttnParams& p, const CUtensorMap& km, const CUtensorMap& vm, int B, int max_q_len, cudaStream_t st) {
  const int smem = (64 + 2 * kv_stages(D) * kTileTok) * D * 2 + 1024;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(paged_prefill_kernel<D, MODE, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess) return -3;
    set = true;
  }
  const int G = p.Hq / p.Hkv;
  dim3 grid((max_q_len * G + 63) / 64, p.Hkv, B);
  paged_prefill_kernel<D, MODE, SIG><<<grid, kAttnThreads, smem, st>>>(km, vm, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// Partial results of the cut items (two per CTA) and the counters of a stream launch.
struct StreamWork { float* scratch; long long scratch_bytes; unsigned int* counters; long long counters_len; };

constexpr int kStreamLimit = 226 * 1024;
// Shared memory of a stream launch (padded head size d, cache values of `esz` bytes) beside its stages, and of a stage.
static long long stream_extra(const AttnParams& p, int d, int esz, int B) {
  const int GA = p.Hq / p.Hkv, rows = GA < 16 ? GA : 16;
  return 1024 + (esz == 1 || p.kc == p.vc ? 4LL * rows * d * 4 : 0) + p.bias_smem * 4LL + (B + 1) * 4LL;
}
static int stream_stage(const AttnParams& p, int d, int esz) { return (p.kc == p.vc ? 1 : 2) * kTileTok * d * esz; }
static bool stream_fits(const AttnParams& p, int d, int esz, int B) {
  return stream_extra(p, d, esz, B) + 2 * stream_stage(p, d, esz) <= kStreamLimit;
}

// Returns 1 when the launch does not fit (the caller takes the other kernel).
template <int D, int MODE, bool SIG>
static int launch_stream(AttnParams p, const CUtensorMap& km, const CUtensorMap& vm, int B, const StreamWork& w, cudaStream_t st) {
  constexpr int ESZ = MODE == kKvTmaFp8 ? 1 : 2;
  if (!stream_fits(p, D, ESZ, B)) return 1;
  const int GA = p.Hq / p.Hkv, heads = p.Hkv * ((GA + 15) / 16);
  p.B = B;
  p.rows = GA < 16 ? GA : 16;
  p.vec_out = !(reinterpret_cast<uintptr_t>(p.out) & 7) && p.out_stride % 4 == 0 && !(reinterpret_cast<uintptr_t>(p.outq) & 3);
  p.stage_bytes = stream_stage(p, D, ESZ);
  const long long extra = stream_extra(p, D, ESZ, B);
  static std::atomic<bool> set[64];
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -3;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Two CTAs per SM, each with as many stages as that leaves room for, three at least where they fit. Three where heads are small and two
  // CTAs per SM would have several items each: an item's fixed parts are most of its time then (158 sequences of 3-191 tokens, 64/8 heads
  // of 64: 25.9 -> 20.4 us; but 3 of 2299-4598 14.9 -> 17.3, which are cut into more pieces).
  const int want = D <= 64 && static_cast<long long>(B) * heads > 2LL * sms ? 3 : 2, share = (want == 3 ? 74 : 112) * 1024;
  long long stages = (share - extra) / p.stage_bytes;
  if (stages < 3) stages = (kStreamLimit - extra) / p.stage_bytes < 3 ? 2 : 3;
  p.stages = static_cast<int>(stages < kStreamMaxStages ? stages : kStreamMaxStages);
  const int smem = static_cast<int>(extra) + p.stages * p.stage_bytes;
  if (!set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(paged_decode_stream_kernel<D, MODE, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamLimit) !=
        cudaSuccess) return -3;
    set[dev].store(true, std::memory_order_release);
  }
  const int per_sm = smem <= share ? want : 1;
  const long long grid = static_cast<long long>(sms) * per_sm;
  const long long need = 2 * grid * p.rows * (p.Dv + 2) * 4;
  if (w.scratch && need <= w.scratch_bytes && w.counters && static_cast<long long>(B) * heads <= w.counters_len) {
    p.cut_o = w.scratch;
    p.cut_ml = w.scratch + 2 * grid * p.rows * p.Dv;
    p.counters = w.counters;
  }
  return launch_early(paged_decode_stream_kernel<D, MODE, SIG>, dim3(static_cast<unsigned>(grid)), dim3(kStreamThreads), smem, st, km, vm,
                    p) == cudaSuccess ? 0 : -4;
}

template <int D, int MODE, bool SIG>
static int launch_decode(const AttnParams& p, int B, cudaStream_t st) {
  constexpr int most = (16 * D + decode_ring(D, false)) * 2 + 1024 + (SIG ? kBiasSmem * 4 : 0);
  const int smem = (16 * D + decode_ring(D, p.kc == p.vc)) * 2 + 1024 + (SIG ? p.bias_smem * 4 : 0);
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(paged_decode_kernel<D, MODE, SIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) !=
        cudaSuccess) return -3;
    set = true;
  }
  dim3 grid(p.Hkv * ((p.Hq / p.Hkv + 15) / 16), B, p.num_splits);
  if (launch_pdl(paged_decode_kernel<D, MODE, SIG>, grid, dim3(kAttnThreads), smem, st, p) != cudaSuccess)
    return -4;
  if (p.num_splits > 1) {
    if (launch_pdl(decode_reduce_kernel<D>, dim3(p.Hq, B), dim3(D < 128 ? 64 : 128), 0, st, p) != cudaSuccess) return -5;
  }
  return 0;
}

template <int D>
static int dispatch_prefill(const AttnParams& p, int cache_fp8, int num_blocks, int B, int max_q_len, cudaStream_t st) {
  CUtensorMap km{}, vm{};
  if (p.bias) {
    if (cache_fp8) return -11;
    if (tma_maps(p, num_blocks, &km, &vm)) return launch_prefill<D, kKvTma, true>(p, km, vm, B, max_q_len, st);
    return launch_prefill<D, kKvCpAsync, true>(p, km, vm, B, max_q_len, st);
  }
  if constexpr (D <= 128) {
    if (cache_fp8) return launch_prefill<D, kKvFp8>(p, km, vm, B, max_q_len, st);
  } else if (cache_fp8) {
    return -11;
  }
  if (tma_maps(p, num_blocks, &km, &vm)) return launch_prefill<D, kKvTma>(p, km, vm, B, max_q_len, st);
  return launch_prefill<D, kKvCpAsync>(p, km, vm, B, max_q_len, st);
}

template <int D>
static int dispatch_decode(const AttnParams& p, int cache_fp8, int num_blocks, int B, const StreamWork& w, cudaStream_t st) {
  CUtensorMap km{}, vm{};
  int rc = 1;
  if (p.bias) {
    if (cache_fp8) return -11;
    if (tma_maps(p, num_blocks, &km, &vm)) rc = launch_stream<D, kKvTma, true>(p, km, vm, B, w, st);
    return rc <= 0 ? rc : launch_decode<D, kKvCpAsync, true>(p, B, st);
  }
  if (cache_fp8) {
    if constexpr (D <= 128) {
      if (tma_maps_fp8(p, num_blocks, &km, &vm)) rc = launch_stream<128, kKvTmaFp8, false>(p, km, vm, B, w, st);
      return rc <= 0 ? rc : launch_decode<D, kKvFp8, false>(p, B, st);
    } else {
      return -11;
    }
  }
  if (tma_maps(p, num_blocks, &km, &vm)) rc = launch_stream<D, kKvTma, false>(p, km, vm, B, w, st);
  return rc <= 0 ? rc : launch_decode<D, kKvCpAsync, false>(p, B, st);
}

// The padded head size that serves (D, Dv), 0 when none does.
static int padded_head(int D, int Dv) {
  const int m = D > Dv ? D : Dv;
  if (D <= 0 || Dv <= 0 || D % 8 || Dv % 8 || m > 256) return 0;
  return (m + 63) / 64 * 64;
}

}  // namespace ksana

using namespace ksana;

// Causal attention of new query rows against the paged cache (which already holds their K/V). kc / vc: the layer's K and
// V panels of block 0; block_stride: elements between blocks; num_blocks: blocks addressable (0 disables the TMA path).
// window 0: no sliding window. sinks: [Hq] fp32 or null. D, Dv: query/key and value head size (out rows: Hq * Dv).
// bias [Hq][bias_len] fp32 switches to sigmoid weights; gate: optional rows like out's, with a common factor (sigmoid weights
// only).
extern "C" int ksana_paged_prefill(const void* q, long long q_stride, void* out, long long out_stride,
                                   const void* kc, const void* vc, long long block_stride, int block_tokens,
                                   const int* block_table, int table_stride, const int* cu_q, const int* kv_lens,
                                   const float* alibi, const float* sinks, int B, int max_q_len, int Hq, int Hkv, int D, int Dv,
                                   int window, int keep, float scale, int cache_fp8, float k_scale, float v_scale,
                                   int num_blocks, const float* bias, int bias_len, const void* gate, long long gate_stride,
                                   float out_factor, int* err, cudaStream_t st) {
  if (B <= 0 || max_q_len <= 0) return 0;
  if (bias ? (bias_len <= 0 || sinks || alibi) : gate != nullptr) return -14;
  if (Hkv <= 0 || Hq % Hkv || q_stride % 8 || (reinterpret_cast<uintptr_t>(q) & 15)) return -10;
  AttnParams p{};
  p.q = (const bf16*)q; p.q_stride = q_stride; p.out = (bf16*)out; p.out_stride = out_stride;
  p.kc = kc; p.vc = vc; p.block_stride = block_stride; p.block_tokens = block_tokens; p.D = D; p.Dv = Dv;
  p.window = window; p.keep = window > 0 ? keep : 0; p.sinks = sinks;
  p.block_table = block_table; p.table_stride = table_stride; p.cu_q = cu_q; p.kv_lens = kv_lens; p.alibi = alibi;
  p.Hq = Hq; p.Hkv = Hkv; p.scale_log2 = scale * 1.44269504f; p.k_scale = k_scale; p.v_scale = v_scale;
  p.num_splits = 1; p.err = err;
  p.bias = bias; p.bias_len = bias_len; p.gate = (const bf16*)gate; p.gate_stride = gate_stride; p.out_factor = out_factor;
  switch (padded_head(D, Dv)) {
    case 64: return dispatch_prefill<64>(p, cache_fp8, num_blocks, B, max_q_len, st);
    case 128: return dispatch_prefill<128>(p, cache_fp8, num_blocks, B, max_q_len, st);
    case 192: return dispatch_prefill<192>(p, cache_fp8, num_blocks, B, max_q_len, st);
    case 256: return dispatch_prefill<256>(p, cache_fp8, num_blocks, B, max_q_len, st);
  }
  return -11;
}

// Rows of distance biases of one head group, where they are staged in shared memory (0: read from global memory).
static int bias_staged(int Hq, int Hkv, int bias_len) {
  const int table = (Hq / Hkv < 16 ? Hq / Hkv : 16) * bias_len;
  return table <= kBiasSmem ? table : 0;
}

// 1: ksana_paged_decode shares such a batch out by itself (the stream form). 0: it runs the number of splits it is given.
extern "C" int ksana_decode_streams(const void* kc, const void* vc, long long block_stride, int block_tokens, int B, int Hq, int Hkv, int D,
                                    int Dv, int cache_fp8, int num_blocks, int bias_len) {
  const int d = padded_head(D, Dv);
  if (!d || Hkv <= 0 || Hq < Hkv || Hq % Hkv || (cache_fp8 && d > 128)) return 0;
  AttnParams p{};
  p.kc = kc; p.vc = vc; p.block_stride = block_stride; p.block_tokens = block_tokens; p.D = D; p.Dv = Dv; p.Hq = Hq; p.Hkv = Hkv;
  p.bias_smem = bias_len > 0 ? bias_staged(Hq, Hkv, bias_len) : 0;
  return tma_covers(p, num_blocks, cache_fp8 != 0) && stream_fits(p, cache_fp8 ? 128 : d, cache_fp8 ? 1 : 2, B);
}

// One new token per sequence. scratch, counters (zero before the first launch): place for the pieces of items that the stream form
// cuts; without enough of it nothing is cut. num_splits and part_o [B*Hq*splits*Dv], part_ml [B*Hq*splits*2] fp32 (splits > 1)
// serve caches that TMA cannot read.
extern "C" int ksana_paged_decode(const void* q, long long q_stride, void* out, long long out_stride,
                                  const void* kc, const void* vc, long long block_stride, int block_tokens,
                                  const int* block_table, int table_stride, const int* kv_lens, const float* alibi,
                                  const float* sinks, int B, int Hq, int Hkv, int D, int Dv, int window, int keep, float scale,
                                  int cache_fp8, float k_scale, float v_scale, int num_splits, float* part_o, float* part_ml,
                                  int num_blocks, void* outq, float* oscale, int oscale_ld, const float* bias, int bias_len,
                                  const void* gate, long long gate_stride, float out_factor, float* scratch, long long scratch_bytes,
                                  unsigned int* counters, long long counters_len, int* err, cudaStream_t st) {
  if (B <= 0) return 0;
  if (bias ? (bias_len <= 0 || sinks || alibi || outq) : gate != nullptr) return -14;
  if (outq && (D != 128 || Dv != 128 || !oscale)) return -13;
  if (Hkv <= 0 || Hq % Hkv || q_stride % 8 || (reinterpret_cast<uintptr_t>(q) & 15)) return -10;
  if (num_splits < 1) num_splits = 1;
  if (num_splits > 1 && (!part_o || !part_ml)) return -12;
  const StreamWork w{scratch, scratch_bytes, counters, counters_len};
  AttnParams p{};
  p.q = (const bf16*)q; p.q_stride = q_stride; p.out = (bf16*)out; p.out_stride = out_stride;
  p.kc = kc; p.vc = vc; p.block_stride = block_stride; p.block_tokens = block_tokens; p.D = D; p.Dv = Dv;
  p.window = window; p.keep = window > 0 ? keep : 0; p.sinks = sinks;
  p.block_table = block_table; p.table_stride = table_stride; p.cu_q = nullptr; p.kv_lens = kv_lens; p.alibi = alibi;
  p.Hq = Hq; p.Hkv = Hkv; p.scale_log2 = scale * 1.44269504f; p.k_scale = k_scale; p.v_scale = v_scale;
  p.num_splits = num_splits; p.part_o = part_o; p.part_ml = part_ml; p.err = err;
  p.outq = static_cast<uint8_t*>(outq); p.oscale = oscale; p.oscale_ld = oscale_ld;
  p.bias = bias; p.bias_len = bias_len; p.gate = (const bf16*)gate; p.gate_stride = gate_stride; p.out_factor = out_factor;
  p.bias_smem = bias ? bias_staged(Hq, Hkv, bias_len) : 0;
  switch (padded_head(D, Dv)) {
    case 64: return dispatch_decode<64>(p, cache_fp8, num_blocks, B, w, st);
    case 128: return dispatch_decode<128>(p, cache_fp8, num_blocks, B, w, st);
    case 192: return dispatch_decode<192>(p, cache_fp8, num_blocks, B, w, st);
    case 256: return dispatch_decode<256>(p, cache_fp8, num_blocks, B, w, st);
  }
  return -11;
}
