// bfloat16 matrix product out[t, f] = sum_k act[t, k] * w[f, k] on the Blackwell tensor cores:
// TMA loads into 128-byte-swizzled shared memory, tcgen05.mma with the accumulator in tensor
// memory, tcgen05.ld for the epilogue.  This replaces the SIMT matmuls of cuongvng/bare-cuda-4gib
// (engine/kernels/gemm_tiled.cuh:36-96 for m > 16, engine/kernels/gemv_fp16.cu:21-101 for
// m <= 16) with one kernel for prefill and decode.
//
// Two orientations of the same kernel.
// ORIENT 0 (few tokens): the weight matrix is the 128-row MMA operand (A) and the activations are
// the N operand (B): one thread block computes 128 output features for BN tokens, BN in
// {16, 32, 64, 128, 256}.  A decode step therefore still fills the 128 MMA rows with weights,
// which is what has to be streamed from memory.  In tensor memory lane = feature and column =
// token, so an epilogue warp stores 32 consecutive features of one token with one store.
// ORIENT 1 (many tokens): 128 tokens are the MMA rows and BN (128 or 256) output features the
// N operand; lane = token, column = feature, so an epilogue thread stores 16 consecutive
// features of its token with vector stores.
//
// Split K.  gridDim.z thread blocks share the K range of a tile; each writes its float32 partial
// result to out + z * partial_stride.  The consumer kernels (residual add + norm, rotation,
// SwiGLU) add the partials in index order, so no atomics and no reduction pass are needed and
// the result does not depend on timing.
//
// MODE 1 (SwiGLU): w is [gate rows; up rows] and the block stores silu(gate) * up.  ORIENT 0
// makes its 128 MMA rows of 64 gate rows and the matching 64 up rows, so the accumulator holds
// gate in lanes 0..63 and up in lanes 64..127; the two epilogue warps that own the up lanes hand
// their values over through shared memory.  ORIENT 1 loads BN/2 gate rows and the matching BN/2
// up rows as one N operand, so a thread finds gate in column c and up in column BN/2 + c.
// MODE 2 (ORIENT 1): w is [Wq; Wk; Wv] and the epilogue turns heads and writes the cache (see HeadsExtra).
//
// Warps: 0 = TMA producer, 1 = tensor memory allocation + MMA issue, 2..5 = epilogue.
// Every wait on an mbarrier is bounded: after about a second without progress the thread sets
// the error word, every role leaves its loop, tensor memory is released and the block returns.

#include "common.cuh"

#include <cuda.h>
#include <string.h>

namespace {

constexpr int BM = 128;      // features per block (MMA M)
constexpr int BK = 64;       // k elements per stage (one 128-byte swizzle row)
constexpr int UMMA_K = 16;
constexpr int NUM_THREADS = 192;
// The gated end of tokens on the MMA rows, one block to an SM, is arithmetic (an exponential and a division an output) that nothing
// hides: eight warps share it instead of four, half of the tile's columns each (300 tokens x 11,264 x 2,048: 23.4 -> 19.8 us; 150 cases of 256 to
// 5,632 outputs and 65 to 300 tokens: tiles of 64 rows 0.96 of the time, 128 0.90, 256 0.86, silu and gelu alike; experts' products 0.88).  The
// adding end, which memory bounds, gets slower with eight (2,048 x 2,048 x 5,632: 44.4 -> 47.9).
constexpr int epilogue_warps(int mode, int orient, int blocks_per_sm) { return mode == 1 && orient == 1 && blocks_per_sm == 1 ? 8 : 4; }
constexpr int threads_of(int mode, int orient, int blocks_per_sm) { return 64 + 32 * epilogue_warps(mode, orient, blocks_per_sm); }
constexpr unsigned long long WAIT_LIMIT_NS = 1000000000ull;

constexpr int ERR_TIMEOUT_PRODUCER = 1;
constexpr int ERR_TIMEOUT_MMA = 2;
constexpr int ERR_TIMEOUT_EPILOGUE = 3;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity; gives up after limit_ns or when another role
// has already given up.  Returns false on giving up.  The time of the kernels before does not count: a role comes here behind
// pdl_wait(), or names a flag of the block that a role sets which did.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long limit_ns, const volatile int* past_wait = nullptr) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long start = global_timer();
  for (unsigned spins = 0;; ++spins) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spins & 63u) == 63u) {
      if (*abort_flag) return false;
      if (past_wait && !*past_wait) start = global_timer();
      else if (global_timer() - start > limit_ns) return false;
    }
  }
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// Shared-memory matrix descriptor for a K-major tile whose rows are 128 bytes, swizzled in
// 1024-byte groups of 8 rows (start address and offsets in 16-byte units, Blackwell version 1,
// layout type 2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);  // start address
  d |= (uint64_t)1 << 16;                  // leading byte offset (unused with swizzle)
  d |= (uint64_t)(1024 >> 4) << 32;        // stride byte offset: 8 rows of 128 bytes
  d |= (uint64_t)1 << 46;                  // descriptor version
  d |= (uint64_t)2 << 61;                  // 128-byte swizzle
  return d;
}

// Instruction descriptor: float32 accumulator, bfloat16 A and B, both K-major, M x N tile.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// What the epilogue of the tokens-on-rows orientation may do beyond storing the product.
struct RowsExtra {
  // The input was prepared for a norm whose factor is one number per row (see AddTo / Prenormed in
  // the launcher): it is bfloat16(residual * norm weight), and the factor rsqrt(mean of squares +
  // eps) is applied here to the float32 sums.  `sq_in` [sq_items][sq_stride]: parts of every
  // input row's sum of squares, added in index order.  Null: the input is what it is.
  const float* sq_in;
  int sq_items;
  long long sq_stride;
  float norm_width, eps;
  // With `out` the float32 residual stream (accumulate): besides residual += product the epilogue
  // leaves what the next norm's product needs: pre_x = bfloat16(new residual * pre_w) and this
  // tile's part of every row's sum of squares in pre_sq[feature tile][row].  Null: neither.
  __nv_bfloat16* pre_x;
  long long pre_x_stride;
  const void* pre_w;
  int pre_w_dtype;
  float* pre_sq;
  long long pre_sq_stride;
  // Grouped products (a mixture of experts): `group_tiles` lists (group, first row, rows) per token
  // tile, `*group_n_tiles` of them; a tile's 128 rows start at its first row (of which `rows` count) and
  // its weight rows at group * group_w_rows.  Null: one weight matrix for all rows.
  const int32_t* group_tiles;
  const int32_t* group_n_tiles;
  int group_w_rows;
  // Row t of the product is stored at row row_map[t] of `out`, times row_weight[row_map[t]].  Null: neither.
  const int32_t* row_map;
  const float* row_weight;
};

// What the epilogue of a [q; k; v] product needs (MODE 2; `out` is q, bfloat16): q and k heads turned by `turn`
// [dim / 2][stride] (cosine, sine) pairs, k and v into the paged cache.  Tiles hold whole heads, and a half head is a
// multiple of 16.  `turn` null: q and k are not turned.
struct HeadsExtra {
  int dim, q_heads, write_cache;
  const float2* turn;
  long long stride;             // tokens lie next to one another: a warp's lanes are tokens
  PagedCache cache;
  const int32_t* positions;
  const int32_t* row_seq;
};

constexpr int STAGING_BYTES = 4 * 32 * 32 * 4;   // per epilogue warp 32 rows of 32 float32, for the adding epilogue

// The factor of the norm that the input rows were prepared for (1 without one).
__device__ __forceinline__ float row_scale(const RowsExtra& ex, int t, int n_tokens) {
  if (!ex.sq_in || t >= n_tokens) return 1.0f;
  float sq = 0.0f;
  for (int i = 0; i < ex.sq_items; ++i) sq += ex.sq_in[(long long)i * ex.sq_stride + t];
  return 1.0f / sqrtf(sq / ex.norm_width + ex.eps);
}

// Epilogue of one warp for a tile with tokens on the tensor-memory lanes (lane = token, column =
// feature): the warp's 32 tokens start at `t_first`, the tile's features at f0.  `lane_base` is
// the tensor-memory address of the warp's lanes at the accumulator's first column; `have_acc`
// false means an empty K range (zeros).  MODE 1: gate in column c, up in column BN/2 + c.
// `wait_acc()` waits until the accumulator is complete (false: the block has given up, nothing is
// stored); what does not depend on the accumulator is requested from memory before it is called.  Modes 0 (but for the adding end)
// and 1 take the columns [c_begin, c_end) of the tile's F_TILE (multiples of 16).
template <int MODE, int DEPTH, typename Wait>
__device__ __forceinline__ void epilogue_tokens_on_rows(uint32_t lane_base, int BN, int F_TILE, int f0, int f_tile_index,
                                                        int t_first, int lane, bool have_acc, void* out, int out_is_f32,
                                                        long long ld_out, int n_tokens, int n_features,
                                                        const RowsExtra& ex, const HeadsExtra& hx, float* staging, int c_begin, int c_end,
                                                        Wait&& wait_acc) {
  float* out_f32 = reinterpret_cast<float*>(out);
  __nv_bfloat16* out_bf16 = reinterpret_cast<__nv_bfloat16*>(out);
  if (MODE == 0 && out_is_f32 == 2 && ex.pre_x) {
    // ---- residual += product, with the next norm prepared.  A thread owns a token's row of the
    // accumulator, but rows of the residual stream lie far apart in memory, so the warp passes 32
    // columns at a time through shared memory (16-byte chunks swizzled by row, free of bank
    // conflicts both ways) and then walks over them four rows per instruction, each row's 128
    // bytes read and written by eight neighbouring lanes.  The old residual values and the norm's
    // weights of DEPTH such chunks are in registers at any time: the first ones are requested
    // while the tensor core still works on the tile, and a chunk's registers are refilled for
    // the chunk DEPTH further on as soon as it is done, so the memory's latency is not waited for.
    const int sub = lane >> 3, ch = lane & 7;
    float sq_acc[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) sq_acc[it] = 0.0f;
    float4 old[DEPTH][8], w[DEPTH];
    bool f_ok[DEPTH];
    auto fetch = [&](int d, int cc) {     // (d is a constant wherever this is called)
      const int f = f0 + cc + ch * 4;
      f_ok[d] = cc < F_TILE && f + 4 <= n_features && cc + ch * 4 < F_TILE;   // (a tile's width is a multiple of 16)
      w[d] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (f_ok[d]) {
        if (ex.pre_w_dtype == DT_BF16) {
          const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(ex.pre_w) + f);
          const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
          const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
          w[d] = make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
        } else {
          w[d] = *reinterpret_cast<const float4*>(static_cast<const float*>(ex.pre_w) + f);
        }
      }
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int t = t_first + it * 4 + sub;
        old[d][it] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (f_ok[d] && t < n_tokens) old[d][it] = *reinterpret_cast<const float4*>(out_f32 + (long long)t * ld_out + f);
      }
    };
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) fetch(d, 32 * d);
    if (!wait_acc()) return;
#pragma unroll 1
    for (int c0 = 0; c0 < F_TILE; c0 += 32 * DEPTH) {
      if (f0 + c0 >= n_features) break;   // uniform across the block
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        const int cc = c0 + 32 * d, f = f0 + cc + ch * 4;
        if (cc < F_TILE && f0 + cc < n_features) {   // uniform across the warp
          uint32_t v[32];
          if (have_acc) {
            tmem_load16(lane_base + cc, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
            tmem_load16(lane_base + cc + 16, *reinterpret_cast<uint32_t(*)[16]>(&v[16]));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0u;
          }
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(staging + lane * 32 + ((c ^ (lane & 7)) << 2)) =
                make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + sub, t = t_first + row;
            if (!f_ok[d] || t >= n_tokens) continue;
            const float4 a = *reinterpret_cast<const float4*>(staging + row * 32 + ((ch ^ (row & 7)) << 2));
            const float4 o4 = old[d][it];
            const float4 now = make_float4(o4.x + a.x, o4.y + a.y, o4.z + a.z, o4.w + a.w);
            *reinterpret_cast<float4*>(out_f32 + (long long)t * ld_out + f) = now;
            const __nv_bfloat162 p01 = __floats2bfloat162_rn(now.x * w[d].x, now.y * w[d].y);
            const __nv_bfloat162 p23 = __floats2bfloat162_rn(now.z * w[d].z, now.w * w[d].w);
            uint2 packed;
            packed.x = *reinterpret_cast<const uint32_t*>(&p01);
            packed.y = *reinterpret_cast<const uint32_t*>(&p23);
            *reinterpret_cast<uint2*>(ex.pre_x + (long long)t * ex.pre_x_stride + f) = packed;
            sq_acc[it] += now.x * now.x;
            sq_acc[it] += now.y * now.y;
            sq_acc[it] += now.z * now.z;
            sq_acc[it] += now.w * now.w;
          }
          __syncwarp();   // the staging rows are about to be overwritten
          fetch(d, cc + 32 * DEPTH);
        }
      }
    }
    // a row's eight lanes add up (in a fixed order), the first of them writes this tile's part
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      float part = sq_acc[it];
      part += __shfl_xor_sync(0xffffffffu, part, 1);
      part += __shfl_xor_sync(0xffffffffu, part, 2);
      part += __shfl_xor_sync(0xffffffffu, part, 4);
      const int t = t_first + it * 4 + sub;
      if (ch == 0 && t < n_tokens) ex.pre_sq[(long long)f_tile_index * ex.pre_sq_stride + t] = part;
    }
    return;
  }
  const int t = t_first + lane;
  float rs = row_scale(ex, t, n_tokens);
  int t_out = t;
  if (ex.row_map && t < n_tokens) {
    t_out = ex.row_map[t];
    if (ex.row_weight) rs *= ex.row_weight[t_out];
  }
  if (!wait_acc()) return;
  if (MODE == 2) {
    // ---- heads turned and put where attention reads them: a thread has a token's whole heads in its row of the
    // accumulator, so both halves of a pair meet here.  The angles' cosines and sines come from a table that the step
    // makes once for all its layers (precise sincosf: too much to repeat for every head).
    const int half = hx.dim / 2;
    const bool live = t < n_tokens;
    const int seq = live ? hx.row_seq[t] : 0, pos = live ? hx.positions[t] : 0;
#pragma unroll 1
    for (int h0 = 0; h0 < F_TILE; h0 += hx.dim) {
      if (f0 + h0 >= n_features) break;   // uniform across the block
      const int head = (f0 + h0) / hx.dim;
      const bool is_q = head < hx.q_heads, is_v = head >= hx.q_heads + hx.cache.kv_heads;
      __nv_bfloat16* dst = nullptr;
      if (live && is_q) {
        dst = out_bf16 + (long long)t * ld_out + (long long)head * hx.dim;
      } else if (live && hx.write_cache) {
        const long long at = cache_offset(hx.cache, seq, pos, head - hx.q_heads - (is_v ? hx.cache.kv_heads : 0));
        if (at >= 0) dst = static_cast<__nv_bfloat16*>(is_v ? hx.cache.v : hx.cache.k) + at;
      }
#pragma unroll 1
      for (int p0 = 0; p0 < half; p0 += 16) {
        float2 cs[16];
        const bool turned = dst && !is_v && hx.turn;
        if (turned)
#pragma unroll
          for (int j = 0; j < 16; ++j) cs[j] = hx.turn[(p0 + j) * hx.stride + t];
        uint32_t g[16], u[16];
        if (have_acc) {
          tmem_load16(lane_base + h0 + p0, g);
          tmem_load16(lane_base + h0 + half + p0, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) g[j] = u[j] = 0u;
        }
        if (!dst) continue;
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          float a0 = __uint_as_float(g[j]) * rs, b0 = __uint_as_float(u[j]) * rs;
          float a1 = __uint_as_float(g[j + 1]) * rs, b1 = __uint_as_float(u[j + 1]) * rs;
          if (turned) {
            const float x0 = a0, y0 = b0, x1 = a1, y1 = b1;
            a0 = x0 * cs[j].x - y0 * cs[j].y, b0 = y0 * cs[j].x + x0 * cs[j].y;
            a1 = x1 * cs[j + 1].x - y1 * cs[j + 1].y, b1 = y1 * cs[j + 1].x + x1 * cs[j + 1].y;
          }
          const __nv_bfloat162 l2 = __floats2bfloat162_rn(a0, a1), h2 = __floats2bfloat162_rn(b0, b1);
          lo[j / 2] = *reinterpret_cast<const uint32_t*>(&l2);
          hi[j / 2] = *reinterpret_cast<const uint32_t*>(&h2);
        }
        uint4* to = reinterpret_cast<uint4*>(dst + p0);
        to[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        to[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        to = reinterpret_cast<uint4*>(dst + half + p0);
        to[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        to[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
      }
    }
    return;
  }
  const bool vec_ok = out_is_f32 ? (ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out_f32) & 15) == 0)
                                 : (ld_out % 8 == 0 && (reinterpret_cast<uintptr_t>(out_bf16) & 15) == 0);
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_end; c0 += 16) {
    if (f0 + c0 >= n_features) break;  // uniform across the warp
    uint32_t g[16], u[16];
    if (have_acc) {
      tmem_load16(lane_base + c0, g);
      if (MODE == 1) tmem_load16(lane_base + BN / 2 + c0, u);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = u[j] = 0u;
    }
    // (rows past the step's last token hold whatever the activation buffer held before: nothing is
    // computed from them, least of all a division, whose slow path such values would take)
    if (t >= n_tokens) continue;
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = __uint_as_float(g[j]) * rs;
      if (MODE == 1) v[j] = glu_pair(v[j], __uint_as_float(u[j]) * rs);
#ifdef GROUPED_UP_RELU2
      // a library built with -DGROUPED_UP_RELU2: a grouped product that keeps its rows in place (the up
      // product of ungated experts) stores relu(x)^2
      if (MODE == 0 && ex.group_tiles && !ex.row_map) {
        const float r = fmaxf(v[j], 0.0f);
        v[j] = r * r;
      }
#endif
    }
    const int f = f0 + c0;
    const long long at = (long long)t_out * ld_out + f;
    if (vec_ok && f + 16 <= n_features) {
      if (out_is_f32) {
        float4* dst = reinterpret_cast<float4*>(out_f32 + at);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          float4 w4 = make_float4(v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
          if (out_is_f32 == 2) {   // accumulate: the output is the float32 residual stream
            const float4 old = dst[q4];
            w4.x += old.x, w4.y += old.y, w4.z += old.z, w4.w += old.w;
          }
          dst[q4] = w4;
        }
      } else {
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          pk[j] = *reinterpret_cast<uint32_t*>(&b);
        }
        uint4* dst = reinterpret_cast<uint4*>(out_bf16 + at);
        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (f + j < n_features) {
          if (out_is_f32) out_f32[at + j] = out_is_f32 == 2 ? out_f32[at + j] + v[j] : v[j];
          else out_bf16[at + j] = __float2bfloat16_rn(v[j]);
        }
      }
    }
  }
}

// Sizes of a launch that depend on the N tile `bn` (a run-time value: any multiple of 16 up to
// 256, so that the number of tiles can be matched to the number of SMs).
struct Geometry {
  int bn;           // MMA N: tokens (ORIENT 0) or weight rows (ORIENT 1) per tile
  int a_tiles;      // 128-row operand tiles per stage
  int b_bytes;      // bytes of the N operand tile
  int stage_bytes;
  int stages;
  int tmem_cols;    // power of two >= bn * a_tiles, at least 32
  uint32_t idesc;
  unsigned long long wait_ns;   // how long a role waits on an mbarrier before it gives up
  int drop_k_block;             // tests only (llm_gemm_test_hooks): this k block's barrier is armed, its copies are left out
};

constexpr int A_BYTES = BM * BK * 2;
constexpr int MAX_STAGES = 8;

// Set by llm_gemm_test_hooks: the wait limit of the launches that follow, and a k block whose copies
// the producer of the non-persistent kernel leaves out (in the cluster kernel, whose barrier waits for more than
// they bring), so that a test can watch a bounded wait run out.
static unsigned long long g_wait_ns = WAIT_LIMIT_NS;
static int g_drop_k_block = -1;

static Geometry make_geometry(int bn, int mode, int orient, int blocks_per_sm) {
  Geometry g;
  g.wait_ns = g_wait_ns;
  g.drop_k_block = g_drop_k_block;
  g.bn = bn;
  g.a_tiles = 1;
  g.b_bytes = bn * BK * 2;
  g.stage_bytes = g.a_tiles * A_BYTES + g.b_bytes;
  const int budget = (blocks_per_sm == 2 ? 110 : 200) * 1024;
  g.stages = budget / g.stage_bytes;
  if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
  int cols = 32;
  while (cols < bn * g.a_tiles) cols *= 2;
  g.tmem_cols = cols;
  g.idesc = instr_desc_bf16(BM, bn);
  return g;
}

// Streaming multiprocessors of the current device, asked once.
static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n < 1)
      n = 148;   // a B200
  }
  return n;
}

static size_t smem_bytes(const Geometry& g) { return (size_t)g.stages * g.stage_bytes + 1024 + 256; }

template <int MODE, int ORIENT, int BLOCKS_PER_SM>
__global__ void __launch_bounds__(threads_of(MODE, ORIENT, BLOCKS_PER_SM), BLOCKS_PER_SM)
gemm_tcgen05_kernel(const Geometry geo, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                    void* __restrict__ out, int out_is_f32, int n_tokens, int n_features, int k_blocks,
                    int k_blocks_per_split, long long ld_out, long long partial_stride, int up_row_offset,
                    const RowsExtra ex, const HeadsExtra hx, int* __restrict__ error_word) {
  const int BN = geo.bn;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + geo.stages * geo.stage_bytes);
  uint64_t* empty_bar = full_bar + geo.stages;
  uint64_t* tmem_full_bar = empty_bar + geo.stages;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(tmem_full_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // ORIENT 0: 128 features (MODE 1: 64 outputs) x BN tokens.  ORIENT 1: 128 tokens x BN features
  // (MODE 1: BN/2 outputs).
  const int F_TILE = ORIENT == 0 ? (MODE == 1 ? BM / 2 : BM) : (MODE == 1 ? BN / 2 : BN);
  const int f0 = blockIdx.x * F_TILE;
  int t0 = blockIdx.y * (ORIENT == 0 ? BN : BM);
  int w_row0 = 0;   // a grouped product: the first weight row of this tile's group
  if (ORIENT == 1 && ex.group_tiles) {
    pdl_wait();     // the list of tiles is another kernel's result
    if ((int)blockIdx.y >= *ex.group_n_tiles) return;   // (the whole block, before it holds anything)
    const int32_t* tile = ex.group_tiles + 3 * blockIdx.y;
    w_row0 = tile[0] * ex.group_w_rows;
    t0 = tile[1];
    n_tokens = t0 + tile[2];   // rows behind the tile's own are another group's: computed, never stored
  }
  const int kb_begin = blockIdx.z * k_blocks_per_split;
  const int kb_end = min(k_blocks, kb_begin + k_blocks_per_split);
  const int n_kb = max(0, kb_end - kb_begin);

  // One stage's loads, in two halves: the weight tiles depend on no other kernel and may be
  // fetched before pdl_wait(); the activation tile is another kernel's output and may not.
  // The first half arms the stage's barrier with the bytes of both.
  auto issue_weights = [&](int i, int s) {
    uint8_t* stage = smem + s * geo.stage_bytes;
    mbar_expect_tx(&full_bar[s], geo.stage_bytes);
    if (i == geo.drop_k_block) return;   // a test's way to leave a barrier waiting (never set otherwise)
    const int k0 = (kb_begin + i) * BK;
    if (ORIENT == 0) {
      tma_load_2d(stage, &map_w, &full_bar[s], k0, f0);   // MODE 1: map_w's box has 64 rows
      if (MODE == 1) tma_load_2d(stage + A_BYTES / 2, &map_w, &full_bar[s], k0, up_row_offset + f0);
    } else {
      uint8_t* b_tile = stage + A_BYTES;
      tma_load_2d(b_tile, &map_w, &full_bar[s], k0, w_row0 + f0);
      // MODE 1: map_w's box has BN/2 rows: gate rows above, the matching up rows below
      if (MODE == 1)
        tma_load_2d(b_tile + geo.b_bytes / 2, &map_w, &full_bar[s], k0, w_row0 + up_row_offset + f0);
    }
  };
  auto issue_activations = [&](int i, int s) {
    if (i == geo.drop_k_block) return;
    uint8_t* stage = smem + s * geo.stage_bytes;
    const int k0 = (kb_begin + i) * BK;
    if (ORIENT == 0) tma_load_2d(stage + geo.a_tiles * A_BYTES, &map_a, &full_bar[s], k0, t0);
    else tma_load_2d(stage, &map_a, &full_bar[s], k0, t0);
  };
  const int n_early = min(n_kb, geo.stages);  // stages that are free from the start

  pdl_launch_dependents();
  if (warp == 0 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    for (int s = 0; s < geo.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int i = 0; i < n_early; ++i) issue_weights(i, i);   // overlaps the tail of the kernel before
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                 "r"(geo.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_base_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      pdl_wait();
      for (int i = 0; i < n_early; ++i) issue_activations(i, i);
      int armed = n_early;
      // stage and phase advance by counting: a division per k block would slow the issue down
      int s = n_early == geo.stages ? 0 : n_early;
      uint32_t phase = n_early == geo.stages ? 1 : 0;
      for (int i = n_early; i < n_kb; ++i) {
        if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_flag, geo.wait_ns)) {
          *abort_flag = 1;
          atomicCAS(error_word, 0, ERR_TIMEOUT_PRODUCER);
          break;
        }
        issue_weights(i, s);
        issue_activations(i, s);
        armed = i + 1;
        if (++s == geo.stages) { s = 0; phase ^= 1; }
      }
      if (*abort_flag) {
        // copies already issued still land in shared memory: wait for them (bounded) before leaving
        for (int i = max(0, armed - geo.stages); i < armed; ++i) {
          const unsigned long long start = global_timer();
          while (!mbar_try_wait(&full_bar[i % geo.stages], (i / geo.stages) & 1) &&  // rare path
                 global_timer() - start < geo.wait_ns / 10) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      pdl_wait();      // the limit of its waits counts from here: the kernels before have their own time
      const uint32_t idesc = geo.idesc;
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      const uint32_t smem_base = smem_u32(smem);
      for (int i = 0; i < n_kb && ok; ++i) {
        if (!mbar_wait(&full_bar[s], phase, abort_flag, geo.wait_ns)) {
          *abort_flag = 1;
          atomicCAS(error_word, 0, ERR_TIMEOUT_MMA);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_addr = smem_base + s * geo.stage_bytes;
        const uint32_t b_addr = a_addr + geo.a_tiles * A_BYTES;
        const uint64_t desc_a = smem_desc_sw128(a_addr);
        const uint64_t desc_b = smem_desc_sw128(b_addr);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint32_t acc = (i > 0 || k > 0) ? 1u : 0u;
          const uint64_t koff = (uint64_t)((k * UMMA_K * 2) >> 4);
          umma_bf16(tmem_base, desc_a + koff, desc_b + koff, idesc, acc);
        }
        umma_commit(&empty_bar[s]);  // frees the stage once these MMAs have read it
        if (++s == geo.stages) { s = 0; phase ^= 1; }
      }
      umma_commit(tmem_full_bar);    // accumulator complete (or, after giving up, releases the epilogue)
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2..5, or 2..9)
    constexpr int EPI = epilogue_warps(MODE, ORIENT, BLOCKS_PER_SM);
    pdl_wait();
    const int quad = warp & 3;  // tensor-memory lanes 32 * quad .. + 31 belong to this warp
    auto wait_acc = [&]() -> bool {
      bool ok = mbar_wait(tmem_full_bar, 0, abort_flag, geo.wait_ns);
      if (!ok) {
        *abort_flag = 1;
        atomicCAS(error_word, 0, ERR_TIMEOUT_EPILOGUE);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI) : "memory");   // the epilogue warps agree on whether to go on
      ok = !*abort_flag;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    float* out_f32 = reinterpret_cast<float*>(out) + (long long)blockIdx.z * partial_stride;
    __nv_bfloat16* out_bf16 = reinterpret_cast<__nv_bfloat16*>(out) + (long long)blockIdx.z * partial_stride;
    if (ORIENT == 1) {
      const int first_half = EPI == 8 ? (F_TILE + 31) / 32 * 16 : F_TILE, part = (warp - 2) / 4;
      // (the pipeline's stages are idle once the accumulator is complete: the adding epilogue passes its tiles through them)
      epilogue_tokens_on_rows<MODE, BLOCKS_PER_SM == 1 ? 4 : 1>(
          lane_base, BN, F_TILE, f0, blockIdx.x, t0 + quad * 32, lane, n_kb > 0,
          out_is_f32 ? static_cast<void*>(out_f32) : static_cast<void*>(out_bf16), out_is_f32, ld_out, n_tokens, n_features,
          ex, hx, reinterpret_cast<float*>(smem) + quad * (32 * 32), part ? first_half : 0, part ? F_TILE : first_half, wait_acc);
    } else if (wait_acc()) {
      if (ORIENT == 0 && MODE == 1) {
        // lanes 0..63 hold gate, lanes 64..127 up, for the block's 64 output features: the up warps
        // park their values in shared memory (the pipeline stages are idle by now), [token][feature]
        float* handover = reinterpret_cast<float*>(smem);
        const int l64 = (quad & 1) * 32 + lane;
        if (quad >= 2) {
#pragma unroll 1
          for (int c0 = 0; c0 < BN; c0 += 16) {
            if (t0 + c0 >= n_tokens) break;
            uint32_t u[16];
            if (n_kb > 0) {
              tmem_load16(lane_base + c0, u);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) u[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) handover[(c0 + j) * 64 + l64] = __uint_as_float(u[j]);
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");   // the four epilogue warps
        if (quad < 2) {
          const int f = f0 + l64;
#pragma unroll 1
          for (int c0 = 0; c0 < BN; c0 += 16) {
            if (t0 + c0 >= n_tokens) break;
            uint32_t g[16];
            if (n_kb > 0) {
              tmem_load16(lane_base + c0, g);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) g[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int t = t0 + c0 + j;
              if (t < n_tokens && f < n_features) {
                const float gate = __uint_as_float(g[j]);
                const float v = glu_pair(gate, handover[(c0 + j) * 64 + l64]);
                if (out_is_f32) out_f32[(long long)t * ld_out + f] = v;
                else out_bf16[(long long)t * ld_out + f] = __float2bfloat16_rn(v);
              }
            }
          }
        }
      } else if (ORIENT == 0) {
        const int f = f0 + quad * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
          if (t0 + c0 >= n_tokens) break;  // uniform across the warp
          uint32_t g[16];
          if (n_kb > 0) {
            tmem_load16(lane_base + c0, g);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) g[j] = 0u;
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int t = t0 + c0 + j;
            if (t < n_tokens && f < n_features) {
              const float v = __uint_as_float(g[j]);
              if (out_is_f32) out_f32[(long long)t * ld_out + f] = v;
              else out_bf16[(long long)t * ld_out + f] = __float2bfloat16_rn(v);
            }
          }
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(geo.tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// The same product for many tokens (ORIENT 1, no K split) as a persistent kernel: one block per SM
// walks over output tiles, the stage ring runs on across tile boundaries (no pipeline drain and
// refill per tile, all of shared memory for one ring), and the accumulator alternates between two
// halves of tensor memory, so that the epilogue warps drain tile j while the MMA warp already
// works on tile j + 1.  Consecutive tiles of a block's neighbours share activation rows and weight
// rows (tile index -> token tile fastest), which keeps both operands in L2.
constexpr int ACC_COLS = 256;   // tensor-memory columns per accumulator half

template <int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_persistent_kernel(const Geometry geo, const __grid_constant__ CUtensorMap map_w,
                               const __grid_constant__ CUtensorMap map_a, void* __restrict__ out, int out_is_f32,
                               int n_tokens, int n_features, int n_kb, long long ld_out, int up_row_offset,
                               int f_tiles, int t_tiles, const RowsExtra ex, const HeadsExtra hx, int* __restrict__ error_word) {
  const int BN = geo.bn;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + geo.stages * geo.stage_bytes);
  uint64_t* empty_bar = full_bar + geo.stages;
  uint64_t* acc_full = empty_bar + geo.stages;      // [2]: the accumulator half holds a finished tile
  uint64_t* acc_empty = acc_full + 2;               // [2]: the epilogue has read it out
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int F_TILE = MODE == 1 ? BN / 2 : BN;
  const int n_tiles = f_tiles * t_tiles;

  pdl_launch_dependents();
  if (warp == 0 && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    for (int s = 0; s < geo.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);   // the four epilogue warps
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                 "r"(2 * ACC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_base_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      pdl_wait();
      int s = 0, armed = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        const int f0 = (tile / t_tiles) * F_TILE, t0 = (tile % t_tiles) * BM;
        for (int i = 0; i < n_kb; ++i) {
          if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_flag, geo.wait_ns)) {
            *abort_flag = 1;
            atomicCAS(error_word, 0, ERR_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          uint8_t* stage = smem + s * geo.stage_bytes;
          uint8_t* b_tile = stage + A_BYTES;
          const int k0 = i * BK;
          mbar_expect_tx(&full_bar[s], geo.stage_bytes);
          tma_load_2d(b_tile, &map_w, &full_bar[s], k0, f0);
          if (MODE == 1) tma_load_2d(b_tile + geo.b_bytes / 2, &map_w, &full_bar[s], k0, up_row_offset + f0);
          tma_load_2d(stage, &map_a, &full_bar[s], k0, t0);
          ++armed;
          if (++s == geo.stages) { s = 0; phase ^= 1; }
        }
      }
      if (*abort_flag) {
        // copies already issued still land in shared memory: wait for them (bounded) before leaving
        for (int i = max(0, armed - geo.stages); i < armed; ++i) {
          const unsigned long long start = global_timer();
          while (!mbar_try_wait(&full_bar[i % geo.stages], (i / geo.stages) & 1) &&
                 global_timer() - start < geo.wait_ns / 10) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      pdl_wait();      // (the limit of its waits counts from here)
      const uint32_t idesc = geo.idesc, smem_base = smem_u32(smem);
      int s = 0, j = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++j) {
        const int buf = j & 1;
        if (!mbar_wait(&acc_empty[buf], ((j >> 1) & 1) ^ 1, abort_flag, geo.wait_ns)) {
          *abort_flag = 1;
          atomicCAS(error_word, 0, ERR_TIMEOUT_MMA);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc_addr = tmem_base + buf * ACC_COLS;
        for (int i = 0; i < n_kb; ++i) {
          if (!mbar_wait(&full_bar[s], phase, abort_flag, geo.wait_ns)) {
            *abort_flag = 1;
            atomicCAS(error_word, 0, ERR_TIMEOUT_MMA);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = smem_base + s * geo.stage_bytes;
          const uint64_t desc_a = smem_desc_sw128(a_addr), desc_b = smem_desc_sw128(a_addr + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t koff = (uint64_t)((k * UMMA_K * 2) >> 4);
            umma_bf16(acc_addr, desc_a + koff, desc_b + koff, idesc, (i > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(&empty_bar[s]);
          if (++s == geo.stages) { s = 0; phase ^= 1; }
        }
        umma_commit(&acc_full[buf]);   // (after giving up this still releases the epilogue)
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2..5)
    pdl_wait();
    const int quad = warp & 3;
    int j = 0;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++j) {
      const int buf = j & 1;
      const int f0 = (tile / t_tiles) * F_TILE, t0 = (tile % t_tiles) * BM;
      bool ok = true;
      auto wait_acc = [&]() -> bool {
        if (!mbar_wait(&acc_full[buf], (j >> 1) & 1, abort_flag, geo.wait_ns) || *abort_flag) {
          *abort_flag = 1;
          atomicCAS(error_word, 0, ERR_TIMEOUT_EPILOGUE);
          ok = false;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return ok;
      };
      const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * ACC_COLS;
      epilogue_tokens_on_rows<MODE, 2>(lane_base, BN, F_TILE, f0, tile / t_tiles, t0 + quad * 32, lane, n_kb > 0, out, out_is_f32,
                                       ld_out, n_tokens, n_features, ex, hx,
                                       reinterpret_cast<float*>(smem + geo.stages * geo.stage_bytes + 256) + quad * (32 * 32),
                                       0, F_TILE, wait_acc);
      if (!ok) break;
      // this warp has read its lanes of the half out: the MMA warp may overwrite it
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * ACC_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// The product for a few dozen tokens with the work around it fused in (the counterpart of gemv_fused.cu,
// whose input no longer fits in shared memory there).  With weights on the MMA rows a product of
// a layer has 16 to 90 tiles, too few to draw HBM's bandwidth, so K has to be split; and split over
// independent blocks it leaves partial sums that further kernels add up (norm, rotation: three more launches a
// layer, 4 to 6 us each).  Here the blocks that share a tile's K range are a cluster: each turns its
// accumulator over to the others in slices (bulk copies through distributed shared memory), so block r
// ends up with all parts of slice r, adds them in the order of the blocks and finishes the outputs:
//   CL_ADD     residual[t, f] += result, and what the next norm's product needs (see RowsExtra)
//   CL_SWIGLU  w = [gate; up]: act(gate) * up
//   CL_ROPE    w = [Wq; Wk; Wv]: q and k rotated by position, q to `out`, k and v into the paged cache
// Rows of a tile go by pairs (a feature and its rotation partner, a gate row and its up row): a slice is
// half = 64 / cluster pairs, first all their first members, then the second ones.  Without pairs the two
// members are simply neighbouring runs.
// Two blocks share an SM (112 KB of shared memory each), so that a kernel's weights are on their way while
// the kernel before it still runs on the other half.  What bounds it: the chain wait for the input - first tile - last
// product - exchange - stores, which is why eight warps share the epilogue, why every role waits for the kernel before by itself,
// and why metadata, angles and the next norm's weights are read before that wait (a step of 22 layers of TinyLlama's sizes, with elected
// issuers: 61 rows 1,094 -> 934 us, 128 rows 1,289 -> 1,089, 240 rows 1,587 -> 1,349).  An arrival at the cluster's barrier that
// releases costs about 0.5 us each time, waiting for the thread's own accesses.  (Storing the slices straight from registers into
// the other blocks' shared memory, 16 bytes a lane, measured slower: 9.5 against 8.0 us for 64 tokens x 2,048 x 2,048.)
enum { CL_ADD = 1, CL_SWIGLU = 2, CL_ROPE = 3 };
constexpr int CL_MAX_TOKENS = 64;         // of a tile; more tokens are more tiles, which read the weights again, from L2
constexpr int CL_EPI_WARPS = 8, CL_EPI = CL_EPI_WARPS * 32, CL_THREADS = 64 + CL_EPI;
constexpr int ERR_TIMEOUT_CLUSTER = 4;

struct ClusterArgs {
  int bn, stages, stage_bytes, tmem_cols;
  uint32_t idesc;
  unsigned long long wait_ns;
  int drop_k_block;             // tests only (llm_gemm_test_hooks): this k block's barrier waits for 16 bytes more than its copies bring
  int pair_span;                // a row's partner lies this far behind it, rows come in groups of twice this many
  int n_tokens, n_features, k_blocks, k_per_block, up_row_offset;
  const float* sq_in;           // parts of the input rows' sums of squares (null: the input is what it is)
  int sq_items;
  long long sq_stride;
  float norm_width, eps;
  void* out;                    // CL_ADD: the float32 residual stream; CL_ROPE: q
  int out_is_f32;
  long long ld_out;
  __nv_bfloat16* pre_x;
  long long pre_x_stride;
  const void* pre_w;
  int pre_w_dtype;
  float* pre_sq;                // [slice][pre_sq_stride]
  long long pre_sq_stride;
  PagedCache cache;
  const int32_t* positions;
  const int32_t* row_seq;
  const float* inv_freq;
  int q_heads, write_cache;
  int* error_word;
};

// The cluster's barrier in two halves: a thread arrives, later waits, then may arrive again.  An arrival says only that this block
// has its barriers (which fence.mbarrier_init has made visible) or has received its slices; data go by the copies' own barriers.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

__device__ __forceinline__ uint32_t peer_address(uint32_t smem_addr, int rank) {
  uint32_t at;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr), "r"(rank));
  return at;
}

template <int N>
__device__ __forceinline__ void load_run(const float* from, float (&v)[N]) {
  if (N == 4) {
    const float4 x = *reinterpret_cast<const float4*>(from);
    v[0] = x.x, v[1] = x.y, v[N - 2] = x.z, v[N - 1] = x.w;
  } else {
    const float2 x = *reinterpret_cast<const float2*>(from);
    v[0] = x.x, v[1] = x.y;
  }
}

// 4 or 2 neighbouring values.
template <int N>
__device__ __forceinline__ void store_run(float* to, const float (&v)[N]) {
  if (N == 4) *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<float2*>(to) = make_float2(v[0], v[1]);
}
template <int N>
__device__ __forceinline__ void store_run(__nv_bfloat16* to, const float (&v)[N]) {
  __nv_bfloat162 b[N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) b[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  if (N == 4) *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<uint32_t*>(&b[0]), *reinterpret_cast<uint32_t*>(&b[N / 2 - 1]));
  else *reinterpret_cast<uint32_t*>(to) = *reinterpret_cast<uint32_t*>(&b[0]);
}

template <int EPI, int C>
__global__ void __launch_bounds__(CL_THREADS, 2)
gemm_cluster_kernel(const ClusterArgs a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a) {
  constexpr int HALF = 64 / C, ROWS = 2 * HALF;       // pairs and rows of a slice
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int slot = a.bn * ROWS + 8;                                                 // floats of a slice (8 more keep slices on other banks)
  float* received = reinterpret_cast<float*>(smem + a.stages * a.stage_bytes);      // [C][bn][ROWS], a slice `slot` apart
  float* sq_part = received + C * slot;                                             // [CL_EPI_WARPS][bn]
  float* scale_s = sq_part + CL_EPI_WARPS * a.bn;                                   // [bn]
  long long* place = reinterpret_cast<long long*>(scale_s + a.bn);                  // CL_ROPE: [bn], where a token's first key head goes in the cache
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(place + a.bn);
  uint64_t* empty_bar = full_bar + a.stages;
  uint64_t* acc_bar = empty_bar + a.stages;
  uint64_t* received_bar = acc_bar + 1;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(received_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
  volatile int* past_wait = reinterpret_cast<volatile int*>(tmem_base_slot + 2);   // the producer is behind its pdl_wait()

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % C, tile = blockIdx.x / C;
  constexpr int TILE_OUT = EPI == CL_SWIGLU ? BM / 2 : BM;
  const int f0 = tile * TILE_OUT;
  const int t0 = blockIdx.y * a.bn, n_tokens = min(a.bn, a.n_tokens - t0);      // this block's tokens: rows t0 .. of everything
  const int kb_begin = rank * a.k_per_block, n_kb = max(0, min(a.k_blocks, kb_begin + a.k_per_block) - kb_begin);

  auto issue_weights = [&](int i, int s) {
    uint8_t* stage = smem + s * a.stage_bytes;
    mbar_expect_tx(&full_bar[s], a.stage_bytes + (kb_begin + i == a.drop_k_block ? 16 : 0));
    const int k0 = (kb_begin + i) * BK;
    tma_load_2d(stage, &map_w, &full_bar[s], k0, f0);      // CL_SWIGLU: the box has 64 rows
    if (EPI == CL_SWIGLU) tma_load_2d(stage + A_BYTES / 2, &map_w, &full_bar[s], k0, a.up_row_offset + f0);
  };
  auto issue_activations = [&](int i, int s) {
    tma_load_2d(smem + s * a.stage_bytes + A_BYTES, &map_a, &full_bar[s], (kb_begin + i) * BK, t0);
  };
  const int n_early = min(n_kb, a.stages);

  pdl_launch_dependents();
  if (warp == 0 && elect_one()) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_bar, 1);
    mbar_init(received_bar, 1);
    *abort_flag = 0;
    *past_wait = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(received_bar, (uint32_t)(C * n_tokens * ROWS * 4));
    for (int i = 0; i < n_early; ++i) issue_weights(i, i);   // overlaps the tail of the kernel before
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_slot)),
                 "r"(a.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  cluster_arrive();        // this block has its barriers
  const uint32_t tmem_base = *tmem_base_slot;
  // Every role that reads what other kernels write waits for them by itself: with a barrier of the block behind one thread's wait and
  // copies the others began 0.9 us later.  The MMA issuer goes by the producer's wait.

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      pdl_wait();
      *past_wait = 1;
      for (int i = 0; i < n_early; ++i) issue_activations(i, i);
      int armed = n_early;
      int s = n_early == a.stages ? 0 : n_early;
      uint32_t phase = n_early == a.stages ? 1 : 0;
      for (int i = n_early; i < n_kb; ++i) {
        if (!mbar_wait(&empty_bar[s], phase ^ 1, abort_flag, a.wait_ns)) {
          *abort_flag = 1;
          atomicCAS(a.error_word, 0, ERR_TIMEOUT_PRODUCER);
          break;
        }
        issue_weights(i, s);
        issue_activations(i, s);
        armed = i + 1;
        if (++s == a.stages) { s = 0; phase ^= 1; }
      }
      if (*abort_flag) {
        // copies already issued still land in shared memory: wait for them (bounded) before leaving
        for (int i = max(0, armed - a.stages); i < armed; ++i) {
          const unsigned long long start = global_timer();
          while (!mbar_try_wait(&full_bar[i % a.stages], (i / a.stages) & 1) && global_timer() - start < a.wait_ns / 10) {
          }
        }
      }
    }
    __syncwarp();
    cluster_wait();
    cluster_arrive();
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      const uint32_t smem_base = smem_u32(smem);
      for (int i = 0; i < n_kb; ++i) {
        if (!mbar_wait(&full_bar[s], phase, abort_flag, a.wait_ns, past_wait)) {
          *abort_flag = 1;
          atomicCAS(a.error_word, 0, ERR_TIMEOUT_MMA);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t desc_a = smem_desc_sw128(smem_base + s * a.stage_bytes);
        const uint64_t desc_b = smem_desc_sw128(smem_base + s * a.stage_bytes + A_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t koff = (uint64_t)((k * UMMA_K * 2) >> 4);
          umma_bf16(tmem_base, desc_a + koff, desc_b + koff, a.idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&empty_bar[s]);
        if (++s == a.stages) { s = 0; phase ^= 1; }
      }
      umma_commit(acc_bar);
    }
    __syncwarp();
    cluster_wait();
    cluster_arrive();
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2..9)
    const int e = threadIdx.x - 64, ew = warp - 2, quad = warp & 3;   // quad: the tensor-memory lanes 32 quad .. of this warp
    // What does not depend on the accumulator comes first, before the wait what no kernel of the step writes: the next norm's
    // weights; a token's place in the cache and its angles.  A thread owns RUN neighbouring features of a token, with pairs
    // their partners too; a token's threads are neighbouring lanes.
    constexpr bool PAIRED = EPI == CL_SWIGLU || EPI == CL_ROPE;
    constexpr int RUN = EPI == CL_ROPE ? 2 : 4, PER_TOKEN = (PAIRED ? HALF : ROWS) / RUN, TOKEN_STEP = CL_EPI / PER_TOKEN;
    static_assert(PER_TOKEN <= 32, "a token's threads lie in one warp");
    const int at = e % PER_TOKEN * RUN, first_token = e / PER_TOKEN;     // first row of the slice that the thread owns
    const int f_plain = f0 + rank * ROWS + at;                           // CL_ADD: its feature
    // The residual values and angles of the thread's next two tokens.
    float old[2][4], pre_w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    float rot_c[2][2], rot_s[2][2];
    const int dim = a.cache.head_dim, span = max(dim / 2, 1), first_pair = tile * 64 + rank * HALF + at;
    const int head = first_pair / span, entry = first_pair % span;       // CL_ROPE: of [q; k; v]
    const bool turned = EPI == CL_ROPE && a.inv_freq && head < a.q_heads + a.cache.kv_heads;
    auto fetch_old = [&](int round, float (&o)[4]) {
      const int mine = first_token + round * TOKEN_STEP;
      if (mine < n_tokens && f_plain + 4 <= a.n_features) {
        const float4 x = *reinterpret_cast<const float4*>(static_cast<const float*>(a.out) + (long long)(t0 + mine) * a.ld_out + f_plain);
        o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w;
      }
    };
    auto fetch_angles = [&](int round, float (&c)[2], float (&s)[2]) {
      const int mine = first_token + round * TOKEN_STEP;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        c[j] = 1.0f, s[j] = 0.0f;
        if (turned && mine < n_tokens) sincosf((float)a.positions[t0 + mine] * a.inv_freq[entry + j], &s[j], &c[j]);
      }
    };
    if (EPI == CL_ADD && a.pre_x && f_plain + 4 <= a.n_features) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        pre_w[j] = a.pre_w_dtype == DT_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(a.pre_w)[f_plain + j])
                                            : static_cast<const float*>(a.pre_w)[f_plain + j];
    }
    if (EPI == CL_ROPE) {
      if (e < n_tokens) place[e] = a.write_cache ? cache_offset(a.cache, a.row_seq[t0 + e], a.positions[t0 + e], 0) : -1;
      fetch_angles(0, rot_c[0], rot_s[0]);
      fetch_angles(1, rot_c[1], rot_s[1]);
      asm volatile("bar.sync 1, %0;" ::"n"(CL_EPI) : "memory");
    }
    pdl_wait();
    if (EPI == CL_ADD) {
      fetch_old(0, old[0]);
      fetch_old(1, old[1]);
    }
    // The norm's factor per token.
    if (a.sq_in) {
      float sq[2] = {0.0f, 0.0f};
#pragma unroll 16
      for (int i = ew; i < a.sq_items; i += CL_EPI_WARPS)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (lane + 32 * j < n_tokens) sq[j] += a.sq_in[(long long)i * a.sq_stride + t0 + lane + 32 * j];
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (lane + 32 * j < n_tokens) sq_part[ew * a.bn + lane + 32 * j] = sq[j];
      asm volatile("bar.sync 1, %0;" ::"n"(CL_EPI) : "memory");
      if (e < n_tokens) {
        float total = 0.0f;
#pragma unroll
        for (int i = 0; i < CL_EPI_WARPS; ++i) total += sq_part[i * a.bn + e];
        scale_s[e] = 1.0f / sqrtf(total / a.norm_width + a.eps);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(CL_EPI) : "memory");
    }

    bool ok = mbar_wait(acc_bar, 0, abort_flag, a.wait_ns);
    if (!ok) {
      *abort_flag = 1;
      atomicCAS(a.error_word, 0, ERR_TIMEOUT_EPILOGUE);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // Two groups of four warps take half of the tokens each: the accumulator, cut into slices, into the pipeline's
    // stages (idle by now), then one bulk copy to every block of the cluster.
    const int part = ew / 4, part_tokens = (a.bn / 2 + 15) / 16 * 16, t_begin = part * part_tokens;
    const int t_end = min(n_tokens, t_begin + part_tokens);
    float* outgoing = reinterpret_cast<float*>(smem);
    if (ok) {
      const int row = quad * 32 + lane, in_group = row % (2 * a.pair_span);
      const int pair = row / (2 * a.pair_span) * a.pair_span + in_group % a.pair_span;
      float* mine = outgoing + pair / HALF * slot + pair % HALF + (in_group >= a.pair_span ? HALF : 0);
      const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
      uint32_t v[2][16];       // at most 32 tokens
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (n_kb > 0 && t_begin + 16 * c < t_end) {
          tmem_load16(lane_base + t_begin + 16 * c, v[c]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[c][j] = 0u;
        }
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (t_begin + 16 * c < t_end)
#pragma unroll
          for (int j = 0; j < 16; ++j) mine[(t_begin + 16 * c + j) * ROWS] = __uint_as_float(v[c][j]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    cluster_wait();          // the others have their barriers
    asm volatile("bar.sync %0, 128;" ::"r"(2 + part) : "memory");
    // A role that gave up leaves an accumulator that is complete by its barrier and wrong: the flag, which every warp of this
    // group has set by now if it did, says so.  Nothing is sent then, and the others' waits for it run out.
    ok = ok && !*abort_flag;
    if (ok && t_end > t_begin && ew % 4 == 0 && lane < C) {      // a lane per receiver
      const uint32_t bytes = (uint32_t)(t_end - t_begin) * ROWS * 4;
      const uint32_t to = peer_address(smem_u32(received + rank * slot + t_begin * ROWS), lane);
      asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(to), "r"(smem_u32(outgoing + lane * slot + t_begin * ROWS)), "r"(bytes),
                     "r"(peer_address(smem_u32(received_bar), lane)) : "memory");
    }
    if (ok) {
      ok = mbar_wait(received_bar, 0, abort_flag, a.wait_ns);
      if (!ok) atomicCAS(a.error_word, 0, ERR_TIMEOUT_CLUSTER);
    }
    ok = __all_sync(0xffffffffu, ok);
    cluster_arrive();        // what was sent here has come (or this thread has given up)
    if (ok) {
      auto summed = [&](int t, int r, float (&v)[RUN]) {      // rows r .. of the slice, the parts added in the order of the blocks
        float part_of[C][RUN];
#pragma unroll
        for (int q = 0; q < C; ++q) load_run(received + q * slot + t * ROWS + r, part_of[q]);
#pragma unroll
        for (int j = 0; j < RUN; ++j) v[j] = part_of[0][j];
#pragma unroll
        for (int q = 1; q < C; ++q)
#pragma unroll
          for (int j = 0; j < RUN; ++j) v[j] += part_of[q][j];
        if (a.sq_in) {
          const float f = scale_s[t];
#pragma unroll
          for (int j = 0; j < RUN; ++j) v[j] *= f;
        }
      };
      const int rounds = (n_tokens + TOKEN_STEP - 1) / TOKEN_STEP;
#pragma unroll 1
      for (int i = 0; i < rounds; ++i) {
        const int mine = first_token + i * TOKEN_STEP, t = t0 + mine;
        const bool there = mine < n_tokens;
        float v[RUN];
        if (EPI == CL_ADD) {
          float sq = 0.0f;
          if (there && f_plain + 4 <= a.n_features) {         // (the width is a multiple of four)
            summed(mine, at, v);
            const long long where = (long long)t * a.ld_out + f_plain;
            float* res = static_cast<float*>(a.out) + where;
#pragma unroll
            for (int j = 0; j < RUN; ++j) v[j] += old[0][j];
            store_run(res, v);
            if (a.pre_x) {
              float w[RUN];
#pragma unroll
              for (int j = 0; j < RUN; ++j) w[j] = v[j] * pre_w[j], sq += v[j] * v[j];
              store_run(a.pre_x + (long long)t * a.pre_x_stride + f_plain, w);
            }
          }
          if (a.pre_x) {
#pragma unroll
            for (int o = 1; o < PER_TOKEN; o <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if (at == 0 && there) a.pre_sq[(long long)(tile * C + rank) * a.pre_sq_stride + t] = sq;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) old[0][j] = old[1][j];
          fetch_old(i + 2, old[1]);
        } else if (there) {
          float u[RUN];
          summed(mine, at, v);
          summed(mine, HALF + at, u);
          if (EPI == CL_SWIGLU) {
            const int f = f0 + rank * HALF + at;
            if (f + RUN > a.n_features) continue;
#pragma unroll
            for (int j = 0; j < RUN; ++j) v[j] = glu_pair(v[j], u[j]);
            if (a.out_is_f32) store_run(static_cast<float*>(a.out) + (long long)t * a.ld_out + f, v);
            else store_run(static_cast<__nv_bfloat16*>(a.out) + (long long)t * a.ld_out + f, v);
          } else if (head < a.q_heads + 2 * a.cache.kv_heads) {     // CL_ROPE: RUN pairs of one head
            if (turned) {
#pragma unroll
              for (int j = 0; j < RUN; ++j) {
                const float lo = v[j], hi = u[j];
                v[j] = lo * rot_c[0][j] - hi * rot_s[0][j];
                u[j] = hi * rot_c[0][j] + lo * rot_s[0][j];
              }
            }
            __nv_bfloat16* to = nullptr;
            if (head < a.q_heads) {
              to = static_cast<__nv_bfloat16*>(a.out) + (long long)t * a.ld_out + (long long)head * dim;
            } else if (place[mine] >= 0) {
              const bool is_v = head >= a.q_heads + a.cache.kv_heads;
              const long long kvh = head - a.q_heads - (is_v ? a.cache.kv_heads : 0);
              to = static_cast<__nv_bfloat16*>(is_v ? a.cache.v : a.cache.k) + place[mine] + kvh * a.cache.page_tokens * dim;
            }
            if (to) {
              store_run(to + entry, v);
              store_run(to + entry + span, u);
            }
#pragma unroll
            for (int j = 0; j < RUN; ++j) rot_c[0][j] = rot_c[1][j], rot_s[0][j] = rot_s[1][j];
            if (i + 2 < rounds) fetch_angles(i + 2, rot_c[1], rot_s[1]);
          }
        }
      }
    }
    __syncwarp();
  }

  cluster_wait();          // no block leaves while slices of it are on their way
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols)
                 : "memory");
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

template <int MODE, int ORIENT, int BLOCKS_PER_SM>
int launch(int bn, const CUtensorMap* map_w, const CUtensorMap* map_a, void* out, int out_is_f32, int n_tokens,
           int n_features, int K, long long ld_out, long long partial_stride, int splits, int up_row_offset,
           const RowsExtra& ex, const HeadsExtra& hx, int* error_word, cudaStream_t stream) {
  const Geometry g = make_geometry(bn, MODE, ORIENT, BLOCKS_PER_SM);
  if (g.stages < 1 || g.tmem_cols * BLOCKS_PER_SM > 512) return ERR_BAD_SIZE;
  auto kern = gemm_tcgen05_kernel<MODE, ORIENT, BLOCKS_PER_SM>;
  static size_t configured = 0;
  const size_t smem = smem_bytes(g);
  if (smem > configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return launch_status();
    configured = smem;
  }
  const int k_blocks = (K + BK - 1) / BK;
  const int per_split = (k_blocks + splits - 1) / splits;
  const int f_tile = ORIENT == 0 ? (MODE == 1 ? BM / 2 : BM) : (MODE == 1 ? bn / 2 : bn);
  const int t_tile = ORIENT == 0 ? bn : BM;
  dim3 grid((n_features + f_tile - 1) / f_tile, (n_tokens + t_tile - 1) / t_tile, splits);
  if (grid.y > 65535 || grid.z > 65535) return ERR_BAD_SIZE;
  launch_kernel(kern, grid, threads_of(MODE, ORIENT, BLOCKS_PER_SM), smem, stream, g, *map_w, *map_a, out, out_is_f32, n_tokens, n_features,
                k_blocks, per_split, ld_out, partial_stride, up_row_offset, ex, hx, error_word);
  return launch_status();
}

template <int MODE>
int launch_persistent(int bn, const CUtensorMap* map_w, const CUtensorMap* map_a, void* out, int out_is_f32, int n_tokens,
                      int n_features, int K, long long ld_out, int up_row_offset, const RowsExtra& ex, const HeadsExtra& hx, int* error_word,
                      cudaStream_t stream) {
  const Geometry g = make_geometry(bn, MODE, 1, 1);
  if (g.stages < 2 || g.tmem_cols > ACC_COLS) return ERR_BAD_SIZE;
  auto kern = gemm_tcgen05_persistent_kernel<MODE>;
  static size_t configured = 0;
  const size_t smem = smem_bytes(g) + STAGING_BYTES;   // the adding epilogue's staging rows lie behind the barriers
  if (smem > configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return launch_status();
    configured = smem;
  }
  const int f_tile = MODE == 1 ? bn / 2 : bn;
  const int f_tiles = (n_features + f_tile - 1) / f_tile, t_tiles = (n_tokens + BM - 1) / BM;
  const long long tiles = (long long)f_tiles * t_tiles;
  const int grid = tiles < sm_count() ? (int)tiles : sm_count();
  launch_kernel(kern, grid, NUM_THREADS, smem, stream, g, *map_w, *map_a, out, out_is_f32, n_tokens, n_features,
                (K + BK - 1) / BK, ld_out, up_row_offset, f_tiles, t_tiles, ex, hx, error_word);
  return launch_status();
}

// How a cluster product lays out a block: as many stages as let two blocks share an SM.
static bool cluster_layout(int bn, int k_per_block, int& stages, size_t& smem) {
  const size_t fixed = (size_t)(128 * bn + 8 * 8) * 4 + (size_t)(CL_EPI_WARPS + 1) * bn * 4 + (size_t)bn * 8 + (2 * MAX_STAGES + 2) * 8 + 16 + 1024;
  const size_t stage = A_BYTES + (size_t)bn * BK * 2, budget = 112 * 1024;
  stages = (int)((budget - fixed) / stage);
  if (stages > k_per_block) stages = k_per_block;
  if (stages > MAX_STAGES) stages = MAX_STAGES;
  smem = fixed + stages * stage;
  const size_t outgoing = (size_t)(128 * bn + 8 * 8) * 4;        // the outgoing slices lie in the stages
  while (stages * stage < outgoing) ++stages;
  smem = fixed + stages * stage;
  return smem <= budget && (stages >= 2 || stages >= k_per_block);
}

template <int EPI, int C>
int launch_cluster(const ClusterArgs& a, size_t smem, int tiles, const CUtensorMap& map_w, const CUtensorMap& map_a, cudaStream_t stream) {
  auto kern = gemm_cluster_kernel<EPI, C>;
  static size_t configured = 0;
  if (smem > configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return launch_status();
    configured = smem;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * C, (a.n_tokens + a.bn - 1) / a.bn);
  cfg.blockDim = dim3(CL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kern, a, map_w, map_a);
  return launch_status();
}

template <int EPI>
int launch_cluster_of(int cluster, const ClusterArgs& a, size_t smem, int tiles, const CUtensorMap& mw, const CUtensorMap& ma, cudaStream_t stream) {
  switch (cluster) {
    case 1: return launch_cluster<EPI, 1>(a, smem, tiles, mw, ma, stream);
    case 2: return launch_cluster<EPI, 2>(a, smem, tiles, mw, ma, stream);
    case 4: return launch_cluster<EPI, 4>(a, smem, tiles, mw, ma, stream);
    case 8: return launch_cluster<EPI, 8>(a, smem, tiles, mw, ma, stream);
  }
  return ERR_BAD_SIZE;
}

}  // namespace

// Writes a 128-byte CUtensorMap for a row-major bfloat16 matrix [rows, cols] (row stride in
// elements) with a box of box_rows x 64 columns and the 128-byte swizzle.  Out-of-range parts of
// a box read as zero.  The base must be 16-byte aligned and the row stride a multiple of 8.
extern "C" int llm_gemm_tensor_map(void* map_out, const void* base, long long rows, long long cols,
                                   long long row_stride, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return 1000 + (int)cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (row_stride % 8) || rows <= 0 || cols <= 0) return ERR_BAD_ALIGN;
  if (box_rows <= 0 || box_rows > 256) return ERR_BAD_SIZE;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = fn(reinterpret_cast<CUtensorMap*>(map_out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 2000 + (int)r;
}

// A grouped product for a mixture of experts (tokens on the MMA rows): `tiles` lists (group, first
// row, rows) for `*n_tiles` <= max_tiles tiles of at most 128 rows of `map_a`'s matrix, whose rows are
// grouped; a tile's weights are rows group * group_w_rows .. of `map_w`'s matrix (all groups stacked).
// mode 1: a group's rows are [gate; up] with the up rows `up_row_offset` behind, and n_features counts the
// outputs silu(gate) * up.  `row_map` (or null): row t goes to row row_map[t] of out, times
// row_weight[row_map[t]] (or null).  map_a's box has 128 rows, map_w's bn (bn / 2 in mode 1).
extern "C" int llm_gemm_grouped_bf16(const void* map_w, const void* map_a, void* out, int out_dtype, int max_tiles,
                                     int n_features, int K, long long ld_out, int bn, int mode, int up_row_offset,
                                     int group_w_rows, const int32_t* tiles, const int32_t* n_tiles,
                                     const int32_t* row_map, const float* row_weight, int* error_word,
                                     cudaStream_t stream) {
  if (max_tiles <= 0 || n_features <= 0) return 0;
  if (K <= 0 || !tiles || !n_tiles || group_w_rows <= 0) return ERR_BAD_SIZE;
  if (out_dtype != DT_F32 && out_dtype != DT_BF16) return ERR_BAD_DTYPE;
  if (bn < 16 || bn > 256 || bn % 16 || (mode == 1 && bn % 32) || (mode != 0 && mode != 1)) return ERR_BAD_SIZE;
  CUtensorMap mw, ma;
  memcpy(&mw, map_w, sizeof(CUtensorMap));
  memcpy(&ma, map_a, sizeof(CUtensorMap));
  RowsExtra ex = {};
  const HeadsExtra hx = {};
  ex.group_tiles = tiles, ex.group_n_tiles = n_tiles, ex.group_w_rows = group_w_rows;
  ex.row_map = row_map, ex.row_weight = row_weight;
  const int f32 = out_dtype == DT_F32 ? 1 : 0;
  const Geometry two = make_geometry(bn, mode, 1, 2);
  const long long f_tile = mode == 1 ? bn / 2 : bn;
  const long long blocks = ((n_features + f_tile - 1) / f_tile) * max_tiles;
  const bool pair = blocks > sm_count() && two.tmem_cols <= 256 && two.stages >= (mode == 1 ? 2 : 3);
  const int rows_bound = max_tiles * BM;   // sizes the grid only: every tile brings its own rows
#define GROUPED_CASE(MODE_)                                                                                           \
  if (mode == MODE_)                                                                                                  \
    return pair ? launch<MODE_, 1, 2>(bn, &mw, &ma, out, f32, rows_bound, n_features, K, ld_out, 0, 1, up_row_offset, \
                                      ex, hx, error_word, stream)                                                         \
                : launch<MODE_, 1, 1>(bn, &mw, &ma, out, f32, rows_bound, n_features, K, ld_out, 0, 1, up_row_offset, \
                                      ex, hx, error_word, stream)
  GROUPED_CASE(0);
  GROUPED_CASE(1);
  return ERR_BAD_SIZE;
#undef GROUPED_CASE
}

// For tests of the bounded waits: the launches that follow give up on an mbarrier after `wait_ns`
// nanoseconds (0: the default of one second), and the producer of the non-persistent kernel arms
// the barrier of k block `drop_k_block` of every tile without issuing its copies (the cluster kernel's, for 16 bytes more than
// its copies bring; -1: none), so the MMA issuer's wait for it runs out: the kernel reports "MMA issuer" in the error
// word (a cluster's other blocks, which wait for the slices, may come first), releases its tensor memory and returns.  Call with (0, -1) to put things back.
extern "C" void llm_gemm_test_hooks(long long wait_ns, int drop_k_block) {
  g_wait_ns = wait_ns > 0 ? (unsigned long long)wait_ns : WAIT_LIMIT_NS;
  g_drop_k_block = drop_k_block;
}

// out[z][t, f] (z < splits) = partial sums of act[t, :] . w[f, :]; mode 1: silu(gate) * up with
// w = [gate; up], the up rows starting at `up_row_offset` (splits must be 1 then).
// `bn` is the N tile, a multiple of 16 up to 256 (of 32 for orient 1 with mode 1).
// `accumulate` (orient 1, mode 0, float32 out, no split): out[t, f] += the product, which is how a
// projection adds itself into the residual stream.
// orient 0: bn tokens per tile; map_a's box must have bn rows, map_w's 128 (64 in mode 1).
// orient 1: bn weight rows per tile; map_a's box must have 128 rows, map_w's bn rows (bn / 2 in mode 1).
// Orient 1 only, both optional (see RowsExtra):
// `sq_in` [sq_items][sq_stride]: the activations are bfloat16(residual * norm weight) and the norm's
// factor per row, 1 / sqrt(sum of the parts / norm_width + eps), is applied to the sums;
// `pre_x` (with accumulate): the kernel also writes pre_x[t, f] = bfloat16(out[t, f] * pre_w[f]) and
// pre_sq[feature tile][t] = that tile's part of the row's sum of squares (ceil(n_features / bn) tiles).
static int gemm_bf16(const void* map_w, const void* map_a, void* out, int out_dtype, int n_tokens,
                     int n_features, int K, long long ld_out, long long partial_stride, int splits,
                     int bn, int mode, int orient, int up_row_offset, int accumulate, const float* sq_in,
                     int sq_items, long long sq_stride, float norm_width, float eps, void* pre_x,
                     long long pre_x_stride, const void* pre_w, int pre_w_dtype, float* pre_sq,
                     long long pre_sq_stride, const HeadsExtra& hx, int* error_word, cudaStream_t stream) {
  if (n_tokens <= 0 || n_features <= 0) return 0;
  if (K <= 0 || splits <= 0 || (mode == 1 && splits != 1)) return ERR_BAD_SIZE;
  if (splits > 1 && out_dtype != DT_F32) return ERR_BAD_DTYPE;
  if (out_dtype != DT_F32 && out_dtype != DT_BF16) return ERR_BAD_DTYPE;
  CUtensorMap mw_copy, ma_copy;  // the caller's buffers need not be 64-byte aligned
  memcpy(&mw_copy, map_w, sizeof(CUtensorMap));
  memcpy(&ma_copy, map_a, sizeof(CUtensorMap));
  const CUtensorMap* mw = &mw_copy;
  const CUtensorMap* ma = &ma_copy;
  if (accumulate && (orient != 1 || mode != 0 || splits != 1 || out_dtype != DT_F32)) return ERR_BAD_SIZE;
  const int f32 = out_dtype == DT_F32 ? (accumulate ? 2 : 1) : 0;   // 2: out[t, f] += result
  if (bn < 16 || bn > 256 || bn % 16 || (mode == 1 && orient == 1 && bn % 32)) return ERR_BAD_SIZE;
  RowsExtra ex = {};
  if (sq_in) {
    if (orient != 1 || sq_items < 1 || sq_stride < n_tokens || !(norm_width > 0.0f)) return ERR_BAD_SIZE;
    ex.sq_in = sq_in, ex.sq_items = sq_items, ex.sq_stride = sq_stride, ex.norm_width = norm_width, ex.eps = eps;
  }
  if (pre_x) {
    if (!accumulate || !pre_w || !pre_sq || pre_sq_stride < n_tokens || n_features % 4 || ld_out % 4 || pre_x_stride % 4)
      return ERR_BAD_SIZE;
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(pre_w)) & 15 || reinterpret_cast<uintptr_t>(pre_x) & 7)
      return ERR_BAD_ALIGN;
    if (pre_w_dtype != DT_F32 && pre_w_dtype != DT_BF16) return ERR_BAD_DTYPE;
    ex.pre_x = static_cast<__nv_bfloat16*>(pre_x), ex.pre_x_stride = pre_x_stride, ex.pre_w = pre_w;
    ex.pre_w_dtype = pre_w_dtype, ex.pre_sq = pre_sq, ex.pre_sq_stride = pre_sq_stride;
  }
  // Two thread blocks per SM let one block's epilogue overlap the other's main loop, at the price
  // of half the pipeline depth each: worth it only when there are more tiles than SMs and at
  // least three stages still fit (two for the SwiGLU tiles, whose long epilogue gains most).
  const Geometry two = make_geometry(bn, mode, orient, 2);
  const long long f_tile = orient == 0 ? (mode == 1 ? BM / 2 : BM) : (mode == 1 ? bn / 2 : bn), t_tile = orient == 0 ? bn : BM;
  const long long tiles = ((n_features + f_tile - 1) / f_tile) * ((n_tokens + t_tile - 1) / t_tile) * splits;
  const bool pair = tiles > sm_count() && two.tmem_cols <= 256 && two.stages >= ((orient == 1 && mode == 1) ? 2 : 3);
  if (orient == 1 && splits == 1 && tiles > sm_count() && bn >= 192) {
    // More tiles than SMs: one block per SM walks over them (see the persistent kernel).  Only for
    // wide tiles, which do not fit twice on an SM.  Narrower ones, adding end, 2,048 rows, two blocks an SM / persistent: tiles of 128,
    // 2,048 x 2,048 24.0 / 25.4 us, 2,048 x 5,632 47.9 / 48.4, 4,096 x 4,096 74.4 / 70.0; of 160, 27.1 / 29.5, 52.7 / 54.6, 79.9 /
    // 66.1: only products for which tiles of 256 are the choice anyway (67.3) would gain by it.
    if (hx.dim) return launch_persistent<2>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out, up_row_offset, ex, hx, error_word, stream);
    if (mode == 0) return launch_persistent<0>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out, up_row_offset, ex, hx, error_word, stream);
    return launch_persistent<1>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out, up_row_offset, ex, hx, error_word, stream);
  }
#define GEMM_CASE(MODE_, ORIENT_)                                                                            \
  if (mode == MODE_ && orient == ORIENT_)                                                                    \
    return pair ? launch<MODE_, ORIENT_, 2>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out,           \
                                            partial_stride, splits, up_row_offset, ex, hx, error_word, stream)  \
                : launch<MODE_, ORIENT_, 1>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out,           \
                                            partial_stride, splits, up_row_offset, ex, hx, error_word, stream)
  if (hx.dim)
    return pair ? launch<2, 1, 2>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out, 0, 1, 0, ex, hx, error_word, stream)
                : launch<2, 1, 1>(bn, mw, ma, out, f32, n_tokens, n_features, K, ld_out, 0, 1, 0, ex, hx, error_word, stream);
  GEMM_CASE(0, 0);
  GEMM_CASE(1, 0);
  GEMM_CASE(0, 1);
  GEMM_CASE(1, 1);
  return ERR_BAD_SIZE;
#undef GEMM_CASE
}

extern "C" int llm_gemm_bf16(const void* map_w, const void* map_a, void* out, int out_dtype, int n_tokens,
                             int n_features, int K, long long ld_out, long long partial_stride, int splits,
                             int bn, int mode, int orient, int up_row_offset, int accumulate, const float* sq_in,
                             int sq_items, long long sq_stride, float norm_width, float eps, void* pre_x,
                             long long pre_x_stride, const void* pre_w, int pre_w_dtype, float* pre_sq,
                             long long pre_sq_stride, int* error_word, cudaStream_t stream) {
  return gemm_bf16(map_w, map_a, out, out_dtype, n_tokens, n_features, K, ld_out, partial_stride, splits, bn, mode, orient,
                   up_row_offset, accumulate, sq_in, sq_items, sq_stride, norm_width, eps, pre_x, pre_x_stride, pre_w,
                   pre_w_dtype, pre_sq, pre_sq_stride, HeadsExtra{}, error_word, stream);
}

// The [q; k; v] product of many tokens (orient 1, no split) whose epilogue turns q and k heads by `turn`
// [head_dim / 2][turn_stride] (cosine, sine; null: not at all), writes q to `q_out` [token][q_stride] and k and v into the paged
// cache.  bn is a multiple of head_dim, head_dim of 32.
extern "C" int llm_gemm_qkv(const void* map_w, const void* map_a, void* q_out, int n_tokens, int K, long long q_stride, int bn,
                            const float* sq_in, int sq_items, long long sq_stride, float norm_width, float eps, const float* turn,
                            long long turn_stride, void* k_base, void* v_base, const int32_t* block_table, long long page_stride, int table_stride,
                            int page_tokens, int kv_heads, int head_dim, const int32_t* positions, const int32_t* row_seq,
                            int q_heads, int write_cache, int* error_word, cudaStream_t stream) {
  if (head_dim < 32 || head_dim % 32 || bn % head_dim || (turn && turn_stride < n_tokens) || q_stride % 8 || page_stride % 8) return ERR_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_base) | reinterpret_cast<uintptr_t>(v_base) |
       reinterpret_cast<uintptr_t>(turn)) & 15)
    return ERR_BAD_ALIGN;
  HeadsExtra hx = {};
  hx.dim = head_dim, hx.q_heads = q_heads, hx.write_cache = write_cache, hx.turn = reinterpret_cast<const float2*>(turn);
  hx.stride = turn_stride;
  hx.cache = PagedCache{k_base, v_base, block_table, page_stride, table_stride, page_tokens, kv_heads, head_dim};
  hx.positions = positions, hx.row_seq = row_seq;
  return gemm_bf16(map_w, map_a, q_out, DT_BF16, n_tokens, (q_heads + 2 * kv_heads) * head_dim, K, q_stride, 0, 1, bn, 0, 1, 0, 0,
                   sq_in, sq_items, sq_stride, norm_width, eps, nullptr, 0, nullptr, DT_F32, nullptr, 0, hx, error_word, stream);
}

// turn[p][t] = (cosine, sine) of positions[t] * inv_freq[p], a float32 product and the precise functions.
__global__ void turn_table_kernel(const int32_t* __restrict__ positions, const float* __restrict__ inv_freq, float2* __restrict__ turn,
                                  long long stride, int n_tokens) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
  if (t >= n_tokens) return;
  float2 v;
  sincosf((float)positions[t] * inv_freq[p], &v.y, &v.x);
  turn[p * stride + t] = v;
}

extern "C" int llm_turn_table(const int32_t* positions, const float* inv_freq, float* turn, long long stride, int n_tokens, int half,
                              cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (half <= 0 || half > 65535 || stride < n_tokens) return ERR_BAD_SIZE;
  launch_kernel(turn_table_kernel, dim3((n_tokens + 255) / 256, half), 256, 0, stream, positions, inv_freq,
                reinterpret_cast<float2*>(turn), stride, n_tokens);
  return launch_status();
}

// The product of a few dozen tokens with its ends fused in (see gemm_cluster_kernel): `cluster` (1, 2, 4 or 8)
// blocks share a tile of 128 weight rows and bn tokens (a multiple of 16, at most 64).  map_w's box has 128 rows (64 for
// CL_SWIGLU), map_a's bn rows.  `pair_span` (CL_ROPE: head_dim / 2).  CL_ADD: out is the float32 residual
// stream; pre_x, pre_w, pre_sq as for llm_gemm_bf16, with one row of parts per slice of 128 / cluster rows.
extern "C" int llm_gemm_cluster(const void* map_w, const void* map_a, int epi, int cluster, int bn, int n_tokens, int n_features,
                                int K, void* out, int out_dtype, long long ld_out, int up_row_offset, const float* sq_in,
                                int sq_items, long long sq_stride, float norm_width, float eps, void* pre_x, long long pre_x_stride,
                                const void* pre_w, int pre_w_dtype, float* pre_sq, long long pre_sq_stride, void* k_base,
                                void* v_base, const int32_t* block_table, long long page_stride, int table_stride,
                                int page_tokens, int kv_heads, int head_dim, const int32_t* positions, const int32_t* row_seq,
                                const float* inv_freq, int q_heads, int write_cache, int* error_word, cudaStream_t stream) {
  if (n_tokens <= 0 || n_features <= 0) return 0;
  if (bn < 16 || bn > CL_MAX_TOKENS || bn % 16 || (n_tokens + bn - 1) / bn > 65535 || K <= 0 || n_features % 4) return ERR_BAD_SIZE;
  if (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8) return ERR_BAD_SIZE;
  if (out_dtype != DT_F32 && out_dtype != DT_BF16) return ERR_BAD_DTYPE;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || ld_out % 4) return ERR_BAD_ALIGN;
  ClusterArgs a = {};
  a.bn = bn, a.pair_span = 64 / cluster;
  a.stage_bytes = A_BYTES + bn * BK * 2;
  a.tmem_cols = 32;
  while (a.tmem_cols < bn) a.tmem_cols *= 2;
  a.idesc = instr_desc_bf16(BM, bn);
  a.wait_ns = g_wait_ns;
  a.drop_k_block = g_drop_k_block;
  a.k_blocks = (K + BK - 1) / BK;
  a.k_per_block = (a.k_blocks + cluster - 1) / cluster;
  size_t smem = 0;
  if (!cluster_layout(bn, a.k_per_block, a.stages, smem)) return ERR_BAD_SIZE;
  a.n_tokens = n_tokens, a.n_features = n_features, a.up_row_offset = up_row_offset;
  if (sq_in) {
    if (sq_items < 1 || sq_stride < n_tokens || !(norm_width > 0.0f)) return ERR_BAD_SIZE;
    a.sq_in = sq_in, a.sq_items = sq_items, a.sq_stride = sq_stride, a.norm_width = norm_width, a.eps = eps;
  }
  a.out = out, a.out_is_f32 = out_dtype == DT_F32 ? 1 : 0, a.ld_out = ld_out;
  a.error_word = error_word;
  CUtensorMap mw, ma;
  memcpy(&mw, map_w, sizeof(CUtensorMap));
  memcpy(&ma, map_a, sizeof(CUtensorMap));
  int rows = n_features;
  switch (epi) {
    case CL_ADD:
      if (out_dtype != DT_F32) return ERR_BAD_DTYPE;
      if (pre_x) {
        if (!pre_w || !pre_sq || pre_sq_stride < n_tokens || pre_x_stride % 4) return ERR_BAD_SIZE;
        if ((reinterpret_cast<uintptr_t>(pre_w) & 15) || (reinterpret_cast<uintptr_t>(pre_x) & 7)) return ERR_BAD_ALIGN;
        if (pre_w_dtype != DT_F32 && pre_w_dtype != DT_BF16) return ERR_BAD_DTYPE;
        a.pre_x = static_cast<__nv_bfloat16*>(pre_x), a.pre_x_stride = pre_x_stride, a.pre_w = pre_w;
        a.pre_w_dtype = pre_w_dtype, a.pre_sq = pre_sq, a.pre_sq_stride = pre_sq_stride;
      }
      return launch_cluster_of<CL_ADD>(cluster, a, smem, (rows + BM - 1) / BM, mw, ma, stream);
    case CL_SWIGLU:
      if (up_row_offset < n_features) return ERR_BAD_SIZE;
      a.pair_span = 64;
      return launch_cluster_of<CL_SWIGLU>(cluster, a, smem, (rows + 63) / 64, mw, ma, stream);
    case CL_ROPE:
      if (out_dtype != DT_BF16 || head_dim < 8 || head_dim % 8 || 128 % head_dim || (q_heads + 2 * kv_heads) * head_dim != n_features)
        return ERR_BAD_SIZE;
      if ((reinterpret_cast<uintptr_t>(k_base) | reinterpret_cast<uintptr_t>(v_base)) & 7 || page_stride % 4) return ERR_BAD_ALIGN;
      a.pair_span = head_dim / 2;
      a.cache = PagedCache{k_base, v_base, block_table, page_stride, table_stride, page_tokens, kv_heads, head_dim};
      a.positions = positions, a.row_seq = row_seq, a.inv_freq = inv_freq, a.q_heads = q_heads, a.write_cache = write_cache;
      return launch_cluster_of<CL_ROPE>(cluster, a, smem, (rows + BM - 1) / BM, mw, ma, stream);
  }
  return ERR_BAD_SIZE;
}
