// The float32 matrix product of the 32-bit run: out[m, n] = sum_k a[m, k] * w[n, k], all float32, on
// the ordinary arithmetic units (no tensor cores).
//
// What bounds it: few rows read every weight once (HBM), many rows are bound by the FMA units, which
// take two products at once as packed pairs (fma.rn.f32x2, the same rounding as two single ones).
//
// The order of a sum depends on k alone, never on the number of rows or on the grid, so any cutting of
// the same tokens into steps gives the same bits: k is cut into 8 equal segments (multiples of 32, the
// last ones possibly short or empty); in a segment the even and the odd k's each form one chain of
// FMAs, which are the two halves of a packed pair, so that operands come as they lie in memory; a
// segment's sum is even + odd, and the segments are added in order.  The longest chain of roundings is
// segment / 2 + 1 + 8 with segment = k / 8 rounded up to a multiple of 32: k / 16 + 9 for multiples of 256 (the plain kernel's, which
// adds slices of 16: k / 16 + 16), and 25 for every k up to 256.
//
// Layout of the work.  A block takes BM rows x BN weight rows; k goes by in stages of 32 (128 bytes a
// row), brought by 16-byte cp.async into a ring, the 16-byte pieces of a row exchanged by the row's
// number (piece ^ (row & 7)) so that the 8 weight rows that a warp reads at once lie on all 32 banks.
// A warp reads 32 weight rows at once, one a lane, and a row of `a` as one broadcast; a thread owns TM rows x
// TN weight rows (of 32 lanes x TN), and a warp's stores are runs of 128 bytes.
//
// SPLIT: the 8 segments go to the 8 blocks of a cluster, each leaves its sums in its shared memory
// and every block adds an eighth of the tile over the 8 in order, through distributed shared memory.
// Without it a block walks through all segments.  The launcher splits where the tiles alone would leave
// SMs idle.
//
// Measured on one B200 (microseconds a launch; the plain kernel's 64 x 64 tiles before, this now):
//   weights 11,264 x 2,048 (92 MB): 4 rows 1,010 -> 19.2 (4.8 TB/s); 257 rows 1,380 -> 303; 2,048 rows 2,106 (44.9 TFLOP/s)
//   weights 2,048 x 2,048 (17 MB):  4 rows 450 -> 6.0 (2.8 TB/s); 257 rows 69; 2,048 rows 436
// The FMA units' peak is 74.4 TFLOP/s (148 SMs x 128 FMAs x 1.965 GHz); with eight rows x four weight rows a thread the shared-memory wavefronts
// (32 for 64 packed FMAs) take as long as the arithmetic.  Tiles of 8 x 8 or 16 x 4 a thread (one block an SM) gained 4 % at
// 2,048 rows and lose it at 257.
#include "common.cuh"

namespace {

constexpr int BK = 32;            // k values per stage: 8 pieces of 16 bytes a row
constexpr int SEGMENTS = 8;       // of k; with SPLIT the blocks of a cluster (8 is the portable limit)

typedef unsigned long long pair32;   // two packed float32

__device__ __forceinline__ void fma_pair(pair32& acc, pair32 a, pair32 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ float pair_sum(pair32 v) {
  float even, odd;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(v));
  return even + odd;
}

// 16 bytes of global into shared memory; `bytes` 0 reads nothing and writes zeros.
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The cluster's barrier: what a thread has written is seen, and what it has read may be written again or go, behind everyone's wait.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ float4 peer_load(uint32_t smem_addr, uint32_t rank) {
  uint32_t at;
  float4 v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}

// Two packed pairs from shared memory.
__device__ __forceinline__ void pairs_load(pair32& x, pair32& y, uint32_t at) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(at));
}

struct Args {
  const float* a;
  const float* w;
  float* out;
  int M, N, K;
  long long lda, ldo;
  int segment;       // k values of a segment, a multiple of BK
  int tile_rows;     // rows that a tile advances by (at most BM: the rows are dealt out evenly)
};

template <int TM, int TN, int WM, int WN, int STAGES, bool SPLIT>
struct Shape {
  static constexpr int BM = TM * WM, BN = 32 * TN * WN, THREADS = 32 * WM * WN;
  static constexpr int STAGE_FLOATS = (BM + BN) * BK;
  static constexpr int RING = STAGES * STAGE_FLOATS * 4, SUMS = SPLIT ? BM * BN * 4 : 0;
  static constexpr int TOTALS = SPLIT ? 0 : TM * TN * THREADS * 4;     // the sums of the segments behind
  static constexpr int SMEM = (RING > SUMS ? RING : SUMS) + TOTALS;
};

template <int TM, int TN, int WM, int WN, int STAGES, bool SPLIT>
__global__ void __launch_bounds__(32 * WM * WN, 2)
matmul_f32_kernel(const Args p) {
  using S = Shape<TM, TN, WM, WN, STAGES, SPLIT>;
  extern __shared__ __align__(128) float smem[];
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp / WN, wn = warp % WN, low = lane & 7;
  const int rank = SPLIT ? (int)(blockIdx.x % SEGMENTS) : 0;
  // neighbouring blocks share weight rows
  const int n0 = (SPLIT ? blockIdx.z : blockIdx.y) * S::BN, m0 = (SPLIT ? blockIdx.y : blockIdx.x) * p.tile_rows;
  const int m_end = min(p.M, m0 + p.tile_rows);
  const int k_begin = SPLIT ? min(p.K, rank * p.segment) : 0;
  const int k_end = SPLIT ? min(p.K, k_begin + p.segment) : p.K;
  const int n_stages = (k_end - k_begin + BK - 1) / BK;

  // A thread copies piece `ch` of rows r0, r0 + STEP, ...; rows beyond the tile's last and k's beyond the segment
  // become zeros.
  constexpr int STEP = S::THREADS / 8;
  const int ch = tid & 7, r0 = tid >> 3;
  const uint32_t to_a = base + r0 * 128 + (ch << 4), to_w = base + S::BM * 128 + r0 * 128 + ((ch ^ (r0 & 7)) << 4);
  const float* from_a = p.a + (long long)min(m0 + r0, p.M - 1) * p.lda + k_begin + ch * 4;
  const float* from_w = p.w + (long long)min(n0 + r0, p.N - 1) * p.K + k_begin + ch * 4;
  const long long next_a = (long long)STEP * p.lda, next_w = (long long)STEP * p.K;
  const int rows_a = m_end - m0 - r0, rows_w = p.N - n0 - r0, pieces = k_end - k_begin - ch * 4;
  auto load_w = [&](int s, uint32_t slot) {
    const float* from = from_w + s * BK;
    const bool in_k = s * BK < pieces;
#pragma unroll
    for (int i = 0; i * STEP < S::BN; ++i) {
      const bool in = in_k && i * STEP < rows_w;
      if (S::BN % STEP == 0 || i * STEP + r0 < S::BN)
        copy16(to_w + slot * (S::STAGE_FLOATS * 4) + i * STEP * 128, in ? from + i * next_w : p.w, in ? 16 : 0);
    }
  };
  auto load_a = [&](int s, uint32_t slot) {
    const float* from = from_a + s * BK;
    const bool in_k = s * BK < pieces;
#pragma unroll
    for (int i = 0; i * STEP < S::BM; ++i) {
      const bool in = in_k && i * STEP < rows_a;
      if (S::BM % STEP == 0 || i * STEP + r0 < S::BM)
        copy16(to_a + slot * (S::STAGE_FLOATS * 4) + i * STEP * 128, in ? from + i * next_a : p.a, in ? 16 : 0);
    }
  };

  // weights are no kernel's output: the ring's share of them is asked for before the wait
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < n_stages) load_w(s, s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_stages) load_a(s, s);
    copies_commit();
  }

  pair32 part[TM][TN];
  float* totals = smem + S::RING / 4 + tid;     // [TM * TN][THREADS], a thread's own
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) part[i][j] = 0ull;
  bool first = true;

  // byte offsets of a thread's rows in a stage, and its row numbers' low bits for the exchange
  const uint32_t a_at = (uint32_t)(wm * TM) * 128, w_at = (uint32_t)(S::BM + wn * TN * 32 + lane) * 128;
  int left = p.segment / BK;         // stages until the segment ends
  uint32_t slot = 0;
  for (int s = 0; s < n_stages; ++s) {
    copies_wait<STAGES - 2>();
    __syncthreads();
    if (s + STAGES - 1 < n_stages) {
      const uint32_t free_slot = slot == 0 ? STAGES - 1 : slot - 1;     // what the stage before this one held
      load_w(s + STAGES - 1, free_slot);
      load_a(s + STAGES - 1, free_slot);
    }
    copies_commit();
    const uint32_t stage = base + slot * (S::STAGE_FLOATS * 4);
    const uint32_t a_row = stage + a_at, w_row = (stage + w_at) | (low << 4);
    if (++slot == STAGES) slot = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      pair32 wx[TN], wy[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) pairs_load(wx[j], wy[j], (w_row ^ (c << 4)) + j * 4096);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        pair32 ax, ay;
        pairs_load(ax, ay, a_row + i * 128 + (c << 4));
#pragma unroll
        for (int j = 0; j < TN; ++j) fma_pair(part[i][j], ax, wx[j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma_pair(part[i][j], ay, wy[j]);
      }
    }
    if (!SPLIT && --left == 0) {
      left = p.segment / BK;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          float* mine = totals + (i * TN + j) * S::THREADS;
          *mine = (first ? 0.0f : *mine) + pair_sum(part[i][j]);
          part[i][j] = 0ull;
        }
      first = false;
    }
  }

  if (!SPLIT) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + wm * TM + i;
      if (m >= m_end) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + (wn * TN + j) * 32 + lane;
        if (n < p.N) p.out[(long long)m * p.ldo + n] = (first ? 0.0f : totals[(i * TN + j) * S::THREADS]) + pair_sum(part[i][j]);
      }
    }
    return;
  }

  copies_wait<0>();
  __syncthreads();                   // the ring becomes the block's table of sums
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      smem[(wm * TM + i) * S::BN + (wn * TN + j) * 32 + lane] = pair_sum(part[i][j]);
  cluster_arrive();
  cluster_wait();
  constexpr int PIECES = S::BM * S::BN / 4, EACH = PIECES / SEGMENTS, ROW_PIECES = S::BN / 4;
  static_assert(PIECES % SEGMENTS == 0, "every block of a cluster adds up the same number of pieces");
  static_assert(EACH <= S::THREADS, "a thread adds up one piece at most");
  const int piece = rank * EACH + tid, r = piece / ROW_PIECES, c = (piece % ROW_PIECES) * 4;
  const int m = m0 + r, n = n0 + c;
  const bool mine = tid < EACH && m < m_end && n < p.N;
  float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (mine) {
    const uint32_t at = base + (uint32_t)(r * S::BN + c) * 4;
    float4 v[SEGMENTS];
#pragma unroll
    for (int q = 0; q < SEGMENTS; ++q) v[q] = peer_load(at, q);
#pragma unroll
    for (int q = 0; q < SEGMENTS; ++q) sum.x += v[q].x, sum.y += v[q].y, sum.z += v[q].z, sum.w += v[q].w;
  }
  __syncwarp();
  cluster_arrive();                  // this block's reads are done (ahead of the results' stores, which the arrival would wait for: 0.5 us)
  if (mine) {
    float* to = p.out + (long long)m * p.ldo + n;
    to[0] = sum.x;
    if (n + 1 < p.N) to[1] = sum.y;
    if (n + 2 < p.N) to[2] = sum.z;
    if (n + 3 < p.N) to[3] = sum.w;
  }
  __syncwarp();
  cluster_wait();                    // no block leaves while another reads its sums
}

template <int TM, int TN, int WM, int WN, int STAGES, bool SPLIT>
int launch(const Args& p, cudaStream_t stream) {
  using S = Shape<TM, TN, WM, WN, STAGES, SPLIT>;
  auto kern = matmul_f32_kernel<TM, TN, WM, WN, STAGES, SPLIT>;
  static bool raised = false;   // one instantiation, one attribute (per process; one device per process)
  if (!raised) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM) != cudaSuccess) return launch_status();
    raised = true;
  }
  const unsigned n_tiles = (p.N + S::BN - 1) / S::BN, m_tiles = (p.M + p.tile_rows - 1) / p.tile_rows;
  if (n_tiles > 65535 || (SPLIT && m_tiles > 65535)) return ERR_BAD_SIZE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = SPLIT ? dim3(SEGMENTS, m_tiles, n_tiles) : dim3(m_tiles, n_tiles);
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (SPLIT) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = SEGMENTS;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (pdl_enabled()) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  cudaLaunchKernelEx(&cfg, kern, p);
  return launch_status();
}

template <int TM>
int launch_few(const Args& p, bool many, cudaStream_t stream) {
  return many ? launch<TM, 1, 1, 2, 4, true>(p, stream) : launch<TM, 2, 1, 2, 6, true>(p, stream);
}

template <int TM>
int launch_many(const Args& p, bool split, cudaStream_t stream) {
  return split ? launch<TM, 4, 8, 1, 4, true>(p, stream) : launch<TM, 4, 8, 1, 3, false>(p, stream);
}

}  // namespace

extern "C" int llm_matmul_f32(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldo,
                              int sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 4 || lda % 4 || sms < 1) return ERR_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) return ERR_BAD_ALIGN;
  Args p{a, w, out, M, N, K, lda, ldo, 0, M};
  p.segment = ((K + SEGMENTS - 1) / SEGMENTS + BK - 1) / BK * BK;
  if (M <= 16) {
    // Up to 16 rows the weights' bytes bound the product.  With at least four blocks of 64 weight rows an SM, many small
    // blocks (four an SM, 38 KB each) keep the most reads in flight; with fewer, blocks of 128 weight rows and a deeper
    // ring, whose segments are over sooner (4 rows, 11,264 x 2,048: 17.9 us against 20.9; 2,048 x 2,048: 6.8 against 5.4).
    const bool many = (long long)((N + 63) / 64) * SEGMENTS >= 4ll * sms;
    if (M <= 2) return launch_few<2>(p, many, stream);
    if (M <= 4) return launch_few<4>(p, many, stream);
    if (M <= 8) return launch_few<8>(p, many, stream);
    return launch_few<16>(p, many, stream);
  }
  // Tiles of at most 64 rows, the rows dealt out evenly.  (More and smaller tiles, where their number would fill the last
  // wave of blocks better, measured slower: 257 rows in 6 tiles of 43 instead of 5 of 52, 128 us against 110 a split launch.)
  const int m_tiles = (M + 63) / 64;
  p.tile_rows = (M + m_tiles - 1) / m_tiles;
  const int tm = (p.tile_rows + 7) / 8;
  const bool split = (long long)m_tiles * ((N + 127) / 128) < 2ll * sms;
  switch (tm) {
    case 3: return launch_many<3>(p, split, stream);
    case 4: return launch_many<4>(p, split, stream);
    case 5: return launch_many<5>(p, split, stream);
    case 6: return launch_many<6>(p, split, stream);
    case 7: return launch_many<7>(p, split, stream);
    case 8: return launch_many<8>(p, split, stream);
  }
  return ERR_BAD_SIZE;
}
