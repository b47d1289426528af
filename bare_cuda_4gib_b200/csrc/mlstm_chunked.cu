// The matrix memory of xLSTM over a step's portions in chunks, on the tensor cores, for bfloat16 steps.  Per head, with a = exp(la)
// the decay of a token, b the weight its input gate gives it, cum_i the sum of la over a chunk's tokens up to i, S
// the memory at the chunk's start and v extended by a column of ones (so that S^T q has n . q behind it):
//
//   y_i = sum_{j <= i} (q_i . k_j) exp(cum_i - cum_j) b_j v_j  +  exp(cum_i) S^T q_i
//   S  <- exp(cum_last) S + sum_j k_j (exp(cum_last - cum_j) b_j v_j)^T
//
// which is S_t = a_t S_(t-1) + b_t k_t v_t^T, y_t = S_t^T q_t written out over a chunk of 128 (64) tokens.  A block owns one
// request, one head and 16 value columns (one block more per head has the ones) and walks the request's chunks in
// order, so blocks never wait on one another.  A chunk's tiles arrive by cp.async while the chunk before them is multiplied.
//
// The design wants weights, decays and memory in 32 bits, and the walk stands in for one in float32 products: it must not be
// further from the recurrence in 64 bits.  Only q . k, whose operands are bfloat16 as they are, runs on mma.sync m16n8k16 (every 16
// products by themselves, those sums added pairwise in float32); exponentials, weights, sums and the memory between chunks are 64-bit numbers, the sums on mma.sync
// m16n8k4.  (Three bfloat16 numbers for each 32-bit factor came out up to 1.07 times further away than the float32 scan:
// the tensor core cuts off what it adds up where float32 rounds.)
//
// 16 heads of 128 x 128, 2,048 tokens: 217 us, where operands, scan in stretches, carry and correction take 491 + 36 and the
// walk with three bfloat16 numbers a factor took 177.  Relative distance from 64 bits, scan -> here (open gates, half open): results 1.5e-7 ->
// 5.9e-8 and 9.4e-8 -> 6.2e-8, worst element 1.3e-7 -> 6.3e-8 and 1.7e-7 -> 7.6e-8 of the sum of its terms' sizes, memory 1.2e-7 ->
// 2.5e-8 and 4.8e-8 -> 2.5e-8.  (q . k in 64 bits as well: 3.1e-8, 415 us.)  What bounds it: 64-bit products, and the longest warp's share
// of a chunk's causal triangle.
//
// Built per model with -DML_DK (key size, a multiple of 16 up to 256) and -DML_DV (value size, a multiple of 16).

#include "common.cuh"

#include <math.h>

#ifndef ML_DK
#define ML_DK 128
#endif
#ifndef ML_DV
#define ML_DV 128
#endif

namespace {

constexpr int N = ML_DK, P = ML_DV;
static_assert(N % 16 == 0 && N >= 16 && N <= 256, "ML_DK must be a multiple of 16 up to 256");
static_assert(P % 16 == 0 && P >= 16, "ML_DV must be a multiple of 16");
constexpr int L = N <= 128 ? 128 : 64;        // tokens of a chunk, 16 to a warp: what shared memory holds
constexpr int PC = 16;                        // value columns of a block: 16 heads of 128 values are 144 blocks
constexpr int SP = P + 4;                     // columns of the state and of the result: values, row sum, three of padding
constexpr int LDN = N + 8, LDP = PC + 8;      // padded rows (conflict-free ldmatrix)
constexpr int LDW = PC + 2;                   // ... of 64-bit numbers (four rows and four columns at once on all banks)
constexpr int WARPS = L / 16, THREADS = WARPS * 32;
constexpr int MT_N = N / 16;                  // row tiles of the state
constexpr int MTW = (MT_N + WARPS - 1) / WARPS;   // of which a warp owns at most this many
constexpr int NT = PC / 8;                    // column tiles of a block's columns

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// 16 (or 4) bytes from global to shared memory without passing through registers; `valid` false fills zeros
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A warp's 16 x 8 sums += 16 x 4 factors (a0: row gq, a1: row gq + 8, column tq) times 4 x 8 (row tq, column gq).  Which four of
// the places summed over go together is free as long as both factors agree: below, a thread's column pair (2 tq, 2 tq + 1) of
// a bfloat16 fragment becomes column tq of two such products.
__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// the lower (e 0) or upper (e 1) of two packed bfloat16 numbers
__device__ __forceinline__ double unpacked(uint32_t pair, int e) {
  return (double)__uint_as_float(e ? pair & 0xffff0000u : pair << 16);
}

struct Args {
  const __nv_bfloat16* q;      // rows `in_stride` apart, like k and v
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  long long in_stride;
  const float* weight;         // [rows, heads]   b
  const float* log_decay;      // [rows, heads]   la
  float* state;                // [slots][heads][N][SP]
  float* out;                  // [rows, heads * SP]   S_t^T q_t * out_scale
  float out_scale;
  const int32_t* seq_slot;
  const int32_t* seq_q_start;
  const int32_t* seq_q_len;
  int heads;
};

struct Shared {
  __nv_bfloat16 k[2][L][LDN], q[2][L][LDN], v[2][L][LDP];   // two sets of a chunk's tiles
  double vt[L][LDW];            // v times its weight and its decay to the chunk's end
  double s[N][LDW];             // the memory at the chunk's start
  double cum[L];
  double to_tile[L];            // exp(cum of the last of the token's 16 - cum) times the token's weight
  double to_chunk[L];           // exp(cum of the chunk's last - cum) times the token's weight
  double from_start[L];         // exp(cum)
  float weight[2][L], log_decay[2][L];
};
static_assert(sizeof(Shared) <= 227 * 1024, "a block's tiles fit in shared memory");

__global__ void __launch_bounds__(THREADS) mlstm_chunked_kernel(Args a) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);

  pdl_launch_dependents();
  pdl_wait();
  const int col0 = blockIdx.x * PC, h = blockIdx.y, seq = blockIdx.z;
  const int q_len = a.seq_q_len[seq];
  if (q_len <= 0) return;
  const int q_start = a.seq_q_start[seq], slot = a.seq_slot[seq], H = a.heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;      // a thread's row within eight and its column pair
  const int mid = lane >> 3;
  const long long out_stride = (long long)H * SP;
  float* S_g = a.state + (((long long)slot * H + h) * N) * SP + col0;
  const bool ones = col0 == P;                  // this block walks the column whose v is 1
  const int cols = min(PC, SP - col0);

  // the state's tiles this warp owns, for the whole walk
  double sreg[MTW][NT][4];
#pragma unroll
  for (int i = 0; i < MTW; ++i) {
    const int mt = warp + i * WARPS;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = mt * 16 + gq + (e >> 1) * 8, col = nt * 8 + tq * 2 + (e & 1);
        sreg[i][nt][e] = mt < MT_N && col < cols ? S_g[(long long)n * SP + col] : 0.0f;
        if (mt < MT_N) sh.s[n][col] = sreg[i][nt][e];
      }
  }

  const int n_chunks = (q_len + L - 1) / L;
  constexpr int CN = N / 8, CP = PC / 8;
  // requests chunk `ch`'s k, q, v (rows past the portion's end are zero), weights and decays, and closes one group
  auto load_chunk = [&](int ch) {
    if (ch < n_chunks) {
      const int st = ch & 1, count = min(L, q_len - ch * L);
      const long long row0 = q_start + (long long)ch * L;
      for (int i = threadIdx.x; i < L * CN; i += THREADS) {
        const int r = i / CN, c8 = i % CN;
        const bool valid = r < count;
        const long long src = valid ? (row0 + r) * a.in_stride + h * N + c8 * 8 : 0;
        cp_async16(&sh.k[st][r][c8 * 8], a.k + src, valid);
        cp_async16(&sh.q[st][r][c8 * 8], a.q + src, valid);
      }
      for (int i = threadIdx.x; i < L * CP; i += THREADS) {
        const int r = i / CP, c8 = i % CP;
        const bool valid = r < count;
        if (ones) {
          *reinterpret_cast<uint4*>(&sh.v[st][r][c8 * 8]) = make_uint4(valid && c8 == 0 ? 0x3f80u : 0u, 0u, 0u, 0u);
          continue;
        }
        cp_async16(&sh.v[st][r][c8 * 8], a.v + (valid ? (row0 + r) * a.in_stride + h * P + col0 + c8 * 8 : 0), valid);
      }
      if (threadIdx.x < L) {
        const int r = threadIdx.x;
        const bool valid = r < count;
        const long long src = valid ? (row0 + r) * H + h : 0;
        cp_async4(&sh.weight[st][r], a.weight + src, valid);
        cp_async4(&sh.log_decay[st][r], a.log_decay + src, valid);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_chunk(0);
  for (int ch = 0; ch < n_chunks; ++ch) {
    const int st = ch & 1, t0 = ch * L, count = min(L, q_len - t0);
    const long long row0 = q_start + t0;
    load_chunk(ch + 1);      // into the other set, which every warp left at the last chunk's end
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();         // chunk `ch` has landed
    if (warp == 0) {         // the running sum over the chunk's tokens: a lane takes L / 32 neighbours
      constexpr int EACH = L / 32;
      double v[EACH], run = 0.0;
#pragma unroll
      for (int j = 0; j < EACH; ++j) v[j] = sh.log_decay[st][EACH * lane + j], run += v[j];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
      }
#pragma unroll
      for (int j = EACH - 1; j >= 0; --j) {
        sh.cum[EACH * lane + j] = run;
        run -= v[j];
      }
    }
    __syncthreads();
    if (threadIdx.x < L) {
      const int r = threadIdx.x;
      const double cum = sh.cum[r], weight = sh.weight[st][r];
      sh.to_tile[r] = exp(sh.cum[r | 15] - cum) * weight;
      sh.to_chunk[r] = exp(sh.cum[L - 1] - cum) * weight;
      sh.from_start[r] = exp(cum);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < L * PC; i += THREADS) {
      const int r = i / PC, c = i % PC;
      sh.vt[r][c] = (double)__bfloat162float(sh.v[st][r][c]) * sh.to_chunk[r];
    }

    // ---- this warp's 16 tokens i against the tokens j <= i, 16 at a time: q . k, the weights (q_i . k_j) exp(cum_i - cum_j) b_j, and
    // their product with v
    uint32_t qf[N / 16][4];
#pragma unroll
    for (int ks = 0; ks < N / 16; ++ks)
      ldmatrix_x4(qf[ks], &sh.q[st][warp * 16 + (lane & 15)][ks * 16 + (lane >> 4) * 8]);
    const int i0 = warp * 16 + gq, i1 = i0 + 8;
    const double ci0 = sh.cum[i0], ci1 = sh.cum[i1];
    double y[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) y[nt][0] = y[nt][1] = y[nt][2] = y[nt][3] = 0.0;
#pragma unroll
    for (int ks = 0; ks < N / 16; ++ks)
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double a0 = unpacked(qf[ks][2 * half], e), a1 = unpacked(qf[ks][2 * half + 1], e);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_f64(y[nt], a0, a1, sh.s[ks * 16 + half * 8 + tq * 2 + e][nt * 8 + gq]);
        }
    {
      const double f0 = sh.from_start[i0], f1 = sh.from_start[i1];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) y[nt][0] *= f0, y[nt][1] *= f0, y[nt][2] *= f1, y[nt][3] *= f1;
    }
#pragma unroll 1
    for (int kk = 0; kk <= warp; ++kk) {
      float s[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
      constexpr int GROUP = N % 64 == 0 ? 4 : N % 32 == 0 ? 2 : 1;      // sums of 16 products that are added to one another first
#pragma unroll
      for (int k0 = 0; k0 < N / 16; k0 += GROUP) {
        float now[GROUP][2][4];
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
          uint32_t kf[4];
          ldmatrix_x4(kf, &sh.k[st][kk * 16 + (mid >> 1) * 8 + (lane & 7)][(k0 + u) * 16 + (mid & 1) * 8]);
#pragma unroll
          for (int e = 0; e < 4; ++e) now[u][0][e] = now[u][1][e] = 0.0f;
          mma_bf16(now[u][0], qf[k0 + u], kf[0], kf[1]);
          mma_bf16(now[u][1], qf[k0 + u], kf[2], kf[3]);
        }
#pragma unroll
        for (int step = 1; step < GROUP; step *= 2)
#pragma unroll
          for (int u = 0; u < GROUP; u += 2 * step)
#pragma unroll
            for (int e = 0; e < 8; ++e) now[u][e >> 2][e & 3] += now[u + step][e >> 2][e & 3];
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e >> 2][e & 3] += now[0][e >> 2][e & 3];
      }
      double w[2][4];
      if (kk < warp) {         // exp(cum_i - cum_j) as two factors of at most 1, through the last of the 16 tokens j
        const double end = sh.cum[kk * 16 + 15], f0 = exp(ci0 - end), f1 = exp(ci1 - end);
#pragma unroll
        for (int jt = 0; jt < 2; ++jt)
#pragma unroll
          for (int e = 0; e < 4; ++e) w[jt][e] = (double)s[jt][e] * ((e >> 1 ? f1 : f0) * sh.to_tile[kk * 16 + jt * 8 + tq * 2 + (e & 1)]);
      } else {
#pragma unroll
        for (int jt = 0; jt < 2; ++jt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = e >> 1 ? i1 : i0, j = kk * 16 + jt * 8 + tq * 2 + (e & 1);
            w[jt][e] = j <= i ? (double)s[jt][e] * (exp((e >> 1 ? ci1 : ci0) - sh.cum[j]) * (double)sh.weight[st][j]) : 0.0;
          }
      }
      double x[2][2][NT];
      bool finite = true;
#pragma unroll
      for (int jt = 0; jt < 2; ++jt)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const float v = __bfloat162float(sh.v[st][kk * 16 + jt * 8 + tq * 2 + e][nt * 8 + gq]);
            finite = finite && isfinite(v);
            x[jt][e][nt] = v;
          }
      if (kk < warp || __all_sync(0xffffffffu, finite)) {
#pragma unroll
        for (int jt = 0; jt < 2; ++jt)
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_f64(y[nt], w[jt][e], w[jt][2 + e], x[jt][e][nt]);
      } else {                 // a weight of zero does not stop infinity or NaN: tokens leave out what comes after them
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int from = (lane & ~3) | ((j & 7) >> 1);
          const double w0 = __shfl_sync(0xffffffffu, w[j >> 3][j & 1], from), w1 = __shfl_sync(0xffffffffu, w[j >> 3][2 + (j & 1)], from);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const double v = (double)__bfloat162float(sh.v[st][kk * 16 + j][nt * 8 + tq * 2 + c]);
              if (j <= gq) y[nt][c] += w0 * v;
              if (j <= gq + 8) y[nt][2 + c] += w1 * v;
            }
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (nt * 8 + tq * 2 >= cols) continue;
      const int col = h * SP + col0 + nt * 8 + tq * 2;
      const double scale = a.out_scale;
      if (i0 < count)
        *reinterpret_cast<float2*>(a.out + (row0 + i0) * out_stride + col) = make_float2((float)(y[nt][0] * scale), (float)(y[nt][1] * scale));
      if (i1 < count)
        *reinterpret_cast<float2*>(a.out + (row0 + i1) * out_stride + col) = make_float2((float)(y[nt][2] * scale), (float)(y[nt][3] * scale));
    }
    __syncthreads();           // vt is complete, and every warp has read the old memory
    // ---- the memory: S <- exp(cum_last) S + k^T vt, this warp's row tiles
    const double keep = sh.from_start[L - 1];
#pragma unroll
    for (int i = 0; i < MTW; ++i)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sreg[i][nt][e] *= keep;
#pragma unroll 2
    for (int kk = 0; kk < L / 16; ++kk) {
      uint32_t kt[MTW][4];     // k^T as the row operand: the stored [token][n] tile, transposed on the way in
#pragma unroll
      for (int i = 0; i < MTW; ++i)
        if (warp + i * WARPS < MT_N)
          ldmatrix_x4_trans(kt[i], &sh.k[st][kk * 16 + (mid >> 1) * 8 + (lane & 7)][(warp + i * WARPS) * 16 + (mid & 1) * 8]);
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double x[NT];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) x[nt] = sh.vt[kk * 16 + half * 8 + tq * 2 + e][nt * 8 + gq];
#pragma unroll
          for (int i = 0; i < MTW; ++i) {
            if (warp + i * WARPS >= MT_N) break;
            const double a0 = unpacked(kt[i][2 * half], e), a1 = unpacked(kt[i][2 * half + 1], e);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_f64(sreg[i][nt], a0, a1, x[nt]);
          }
        }
    }
#pragma unroll
    for (int i = 0; i < MTW; ++i) {
      const int mt = warp + i * WARPS;
      if (mt >= MT_N) break;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) sh.s[mt * 16 + gq + (e >> 1) * 8][nt * 8 + tq * 2 + (e & 1)] = sreg[i][nt][e];
    }
    __syncthreads();           // every warp has read this chunk's tiles (and the next chunk's barriers come before the memory is read)
  }
#pragma unroll
  for (int i = 0; i < MTW; ++i) {
    const int mt = warp + i * WARPS;
    if (mt >= MT_N) break;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int n = mt * 16 + gq + (e >> 1) * 8, col = nt * 8 + tq * 2;
        if (col < cols) *reinterpret_cast<float2*>(S_g + (long long)n * SP + col) = make_float2((float)sreg[i][nt][e], (float)sreg[i][nt][e + 1]);
      }
  }
}

}  // namespace

extern "C" int llm_mlstm_chunked(const void* q, const void* k, const void* v, long long in_stride, const float* weight,
                                 const float* log_decay, float* state, float* out, float out_scale, const int32_t* seq_slot,
                                 const int32_t* seq_q_start, const int32_t* seq_q_len, int n_seqs, int heads, int dk, int dv,
                                 cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  LLM_HOST_CHECK(dk == N && dv == P && heads >= 1 && heads <= 65535 && n_seqs <= 65535 && in_stride % 8 == 0, ERR_BAD_SIZE);
  LLM_HOST_CHECK(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15) == 0 &&
                     ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(state)) & 7) == 0,
                 ERR_BAD_ALIGN);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(mlstm_chunked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared)) != cudaSuccess)
      return launch_status();
    configured = true;
  }
  Args a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, in_stride, weight, log_decay, state, out, out_scale,
         seq_slot, seq_q_start, seq_q_len, heads};
  launch_kernel(mlstm_chunked_kernel, dim3(P / PC + 1, heads, n_seqs), THREADS, sizeof(Shared), stream, a);
  return launch_status();
}
