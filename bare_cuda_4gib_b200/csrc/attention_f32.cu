// Softmax attention of the 32-bit run: float32 queries against the paged float32 cache, head sizes 64
// and 128 (-DHEAD_DIM), grouped queries, an optional window.  Ordinary arithmetic units, packed pairs
// (fma.rn.f32x2), precise expf.
//
// The order of every sum is fixed by absolute positions, so any cutting of the same tokens into steps gives
// the same bits.  Keys are taken in spans of 64 from position 0.  One warp makes a span's state for eight
// rows (a row = a token and one query head of the key head's group): scores as two chains over the
// head's even and odd entries; the largest visible score m; weights exp(s - m); their sum l; and the weighted
// values o, one chain over the span's keys.  States are joined in the order of the spans.  `span_state` and
// `join` are the only code that does this arithmetic, and both ways of dealing out the work call them:
//   walk   (more than eight rows of a request): a block takes 64 rows, eight a warp; spans come through
//          shared memory two at a time, once for all warps, and every warp joins as it goes.
//   few    (a decoding request): the spans are dealt out to the eight blocks of a cluster, warp r makes the states of
//          row r, they stay in shared memory, and block r joins them for row r through distributed shared memory.
//          (One warp for all eight rows of a span: 19.3 us a layer for 4 requests of up to 300 keys, a warp a row 13.7.)
// What bounds it: shared-memory wavefronts in the walk (24 of them for 32 packed FMAs), latency with few rows.
//
// A key that no row of a tile sees, or whose page is not held, is zero in shared memory.  A weight of zero (the key is not
// seen, or its weight underflows beside the span's largest) skips the value, which may be anything, infinity or NaN
// too; so does a span that underflows beside the rest of a row.
#include "common.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 64
#endif

namespace {

constexpr int D = HEAD_DIM;
static_assert(D == 64 || D == 128, "a lane owns one or two pairs of output columns");
constexpr int SPAN = 64, ROWS = 8, WARPS = 8, THREADS = WARPS * 32, TILE_ROWS = WARPS * ROWS;
constexpr int CLUSTER = 8;                       // blocks that share a decoding request's keys
constexpr int SLOTS = D == 64 ? 4 : 2;           // spans a block holds at once with few rows
constexpr int PAIRS = D / 64;                    // pairs of output columns a lane owns
constexpr int SPAN_BYTES = SPAN * D * 4;         // keys or values of a span
constexpr int GRID_MAX = 65535;                  // of a grid's second and third axis
constexpr int STATE_FLOATS = ROWS * (D + 2);     // m [ROWS], l [ROWS], o [ROWS][D]

typedef unsigned long long pair32;

__device__ __forceinline__ void fma_pair(pair32& acc, pair32 a, pair32 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ pair32 pack(float x, float y) {
  pair32 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ float2 unpack(pair32 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ void pairs_load(pair32& x, pair32& y, uint32_t at) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(at));
}
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float peer_float(uint32_t smem_addr, uint32_t rank) {
  uint32_t at;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

struct Args {
  const float* q;
  float* out;
  PagedCache cache;
  const int32_t* q_start;
  const int32_t* q_len;
  const int32_t* kv_len;
  int q_heads, group, window;
  float scale;
};

struct Shared {                       // byte offsets in dynamic shared memory
  static constexpr int Q = 0;                                         // [TILE_ROWS][D]
  static constexpr int P = Q + TILE_ROWS * D * 4;                     // [WARPS][ROWS][SPAN]
  static constexpr int STATES = P + WARPS * ROWS * SPAN * 4;          // [SLOTS][STATE_FLOATS]
  static constexpr int HELD = STATES + SLOTS * STATE_FLOATS * 4;      // [4][SPAN] a key is there
  static constexpr int SPANS = (HELD + 4 * SPAN * 4 + 127) / 128 * 128;   // [2 or SLOTS][keys | values]
  static constexpr int TOTAL_WALK = SPANS + 2 * 2 * SPAN_BYTES, TOTAL_FEW = SPANS + SLOTS * 2 * SPAN_BYTES;
};

// What joins one more span's state of a row (m, l, one value of o) to the state of the spans before it.
struct Join {
  float before, now, m;
  __device__ __forceinline__ Join(float m_before, float m_span) {
    m = fmaxf(m_before, m_span);
    before = m_before == -INFINITY ? 0.0f : expf(m_before - m);
    now = m_span == -INFINITY ? 0.0f : expf(m_span - m);
  }
  __device__ __forceinline__ bool underflows(float m_span) const { return now == 0.0f && m_span != -INFINITY; }
  __device__ __forceinline__ float operator()(float x_before, float x_span) const {
    return __fmaf_rn(x_before, before, __fmul_rn(x_span, now));
  }
};

// One warp: the state of keys [64 span, 64 span + 64) for NR rows.  Row i sees keys first[i] .. last[i].
template <int NR>
__device__ __forceinline__ void span_state(uint32_t q, uint32_t keys, uint32_t values, uint32_t p, const int* held, int span,
                                           const int (&first)[NR], const int (&last)[NR], float scale, int lane,
                                           float (&m)[NR], float (&l)[NR], pair32 (&o)[NR][PAIRS]) {
  pair32 dot[NR][2];
#pragma unroll
  for (int i = 0; i < NR; ++i) dot[i][0] = dot[i][1] = 0ull;
  const uint32_t low = lane & 7, key = keys + lane * D * 4;
#pragma unroll 4
  for (uint32_t c = 0; c < D / 4; ++c) {
    pair32 ax, ay, bx, by;
    pairs_load(ax, ay, key + ((c ^ low) << 4));
    pairs_load(bx, by, key + 32 * D * 4 + ((c ^ low) << 4));
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      pair32 qx, qy;
      pairs_load(qx, qy, q + i * D * 4 + (c << 4));
      fma_pair(dot[i][0], qx, ax);
      fma_pair(dot[i][1], qx, bx);
      fma_pair(dot[i][0], qy, ay);
      fma_pair(dot[i][1], qy, by);
    }
  }
  const int j0 = span * SPAN + lane, j1 = j0 + 32;
  const bool held0 = held[lane] != 0, held1 = held[lane + 32] != 0;
  bool none_zero = true;
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const float2 d0 = unpack(dot[i][0]), d1 = unpack(dot[i][1]);
    const float s0 = held0 && j0 >= first[i] && j0 <= last[i] ? __fmul_rn(__fadd_rn(d0.x, d0.y), scale) : -INFINITY;
    const float s1 = held1 && j1 >= first[i] && j1 <= last[i] ? __fmul_rn(__fadd_rn(d1.x, d1.y), scale) : -INFINITY;
    m[i] = warp_max(fmaxf(s0, s1));
    const float p0 = s0 == -INFINITY ? 0.0f : expf(s0 - m[i]);
    const float p1 = s1 == -INFINITY ? 0.0f : expf(s1 - m[i]);
    none_zero = none_zero && p0 != 0.0f && p1 != 0.0f;
    l[i] = warp_sum(__fadd_rn(p0, p1));
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(p + (i * SPAN + lane) * 4), "f"(p0));
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(p + (i * SPAN + lane + 32) * 4), "f"(p1));
  }
  none_zero = __all_sync(0xffffffffu, none_zero);       // then no weight has to be looked at below
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int c = 0; c < PAIRS; ++c) o[i][c] = 0ull;
  const uint32_t value = values + lane * (PAIRS * 8);
#pragma unroll 2
  for (int j = 0; j < SPAN; j += 4) {
    pair32 v[4][PAIRS];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < PAIRS; ++c)
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v[u][c]) : "r"(value + (j + u) * D * 4 + c * 8));
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      float w[4];
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]) : "r"(p + (i * SPAN + j) * 4));
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (none_zero || w[u] != 0.0f)
#pragma unroll
          for (int c = 0; c < PAIRS; ++c) fma_pair(o[i][c], pack(w[u], w[u]), v[u][c]);
    }
  }
  __syncwarp();          // the weights' place may be written again
}

// All threads: asks for the keys and values of a span; keys outside [first, last] and those without a page become zero.
__device__ __forceinline__ void stage_span(const Args& a, int seq, int kvh, int span, int first, int last, uint32_t to, int* held) {
  constexpr int PIECES = D / 4, STEP = THREADS / PIECES;
  const int piece = threadIdx.x % PIECES;
  for (int r = threadIdx.x / PIECES; r < SPAN; r += STEP) {
    const int j = span * SPAN + r;
    const long long off = j >= first && j <= last ? cache_offset(a.cache, seq, j, kvh) : -1;
    const float* k = static_cast<const float*>(a.cache.k);
    const float* v = static_cast<const float*>(a.cache.v);
    copy16(to + r * D * 4 + ((piece ^ (r & 7)) << 4), off >= 0 ? k + off + piece * 4 : k, off >= 0 ? 16 : 0);
    copy16(to + SPAN_BYTES + r * D * 4 + (piece << 4), off >= 0 ? v + off + piece * 4 : v, off >= 0 ? 16 : 0);
    if (piece == 0) held[r] = off >= 0;
  }
}

__global__ void __launch_bounds__(THREADS) attention_f32_kernel(const Args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.y, seq = blockIdx.z, G = a.group;
  int* held = reinterpret_cast<int*>(smem + Shared::HELD);
  pdl_launch_dependents();
  // the step's metadata is written by the host before the step's first kernel and by no kernel: it is read ahead of the wait
  const int q_len = a.q_len[seq], q_start = a.q_start[seq];
  const int rows = q_len * G, base_pos = a.kv_len[seq] - q_len;
  const bool few = rows <= ROWS;
  const int tiles = (rows + TILE_ROWS - 1) / TILE_ROWS;
  if (rows == 0 || (!few && (int)blockIdx.x >= tiles) || (few && blockIdx.x >= CLUSTER)) {         // whole clusters, or blocks of a walk
    pdl_wait();
    return;
  }
  // the last tile sees the most keys: it starts first
  const int r0 = few ? 0 : (tiles - 1 - (int)blockIdx.x) * TILE_ROWS;
  const int tile_last = base_pos + (min(r0 + TILE_ROWS, rows) - 1) / G;
  const int tile_first = a.window > 0 ? max(0, base_pos + r0 / G - a.window + 1) : 0;
  const int span_first = tile_first / SPAN, n_spans = tile_last / SPAN - span_first + 1;
  const uint32_t spans = base + Shared::SPANS, p = base + Shared::P + warp * (ROWS * SPAN * 4);
  // A few rows' first spans that lie below the step's first new position hold what earlier steps wrote: they too are asked for
  // ahead of the wait.
  auto early = [&](int s) { return s < n_spans && (span_first + s + 1) * SPAN <= base_pos; };
  if (few) {
#pragma unroll
    for (int slot = 0; slot < SLOTS; ++slot) {
      const int s = slot * CLUSTER + (int)blockIdx.x;
      if (early(s)) stage_span(a, seq, kvh, span_first + s, tile_first, tile_last, spans + slot * 2 * SPAN_BYTES, held + slot * SPAN);
    }
  }
  pdl_wait();
  for (int e = threadIdx.x; e < (few ? ROWS : TILE_ROWS) * (D / 4); e += THREADS) {
    const int r = r0 + e / (D / 4), c = (e % (D / 4)) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (r < rows) v = *reinterpret_cast<const float4*>(a.q + ((long long)(q_start + r / G) * a.q_heads + kvh * G + r % G) * D + c);
    reinterpret_cast<float4*>(smem + Shared::Q)[e] = v;
  }
  if (!few) {
    int first[ROWS], last[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int r = r0 + warp * ROWS + i, pos = base_pos + r / G;
      last[i] = r < rows ? pos : -1;                                   // a row that does not exist sees nothing
      first[i] = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    }
    float M[ROWS], L[ROWS];
    float2 O[ROWS][PAIRS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      M[i] = -INFINITY, L[i] = 0.0f;
#pragma unroll
      for (int c = 0; c < PAIRS; ++c) O[i][c] = make_float2(0.0f, 0.0f);
    }
    stage_span(a, seq, kvh, span_first, tile_first, tile_last, spans, held);
    copies_commit();
    for (int s = 0; s < n_spans; ++s) {
      const int slot = s & 1;
      copies_wait_all();
      __syncthreads();                // the span has come, and every warp is done with the one before
      if (s + 1 < n_spans) {
        stage_span(a, seq, kvh, span_first + s + 1, tile_first, tile_last, spans + (slot ^ 1) * 2 * SPAN_BYTES, held + (slot ^ 1) * SPAN);
        copies_commit();
      }
      const int span = span_first + s;
      bool seen = false;
#pragma unroll
      for (int i = 0; i < ROWS; ++i) seen = seen || (last[i] >= span * SPAN && first[i] < span * SPAN + SPAN);
      if (!seen) continue;
      float m[ROWS], l[ROWS];
      pair32 o[ROWS][PAIRS];
      const uint32_t at = spans + slot * 2 * SPAN_BYTES;
      span_state<ROWS>(base + Shared::Q + warp * ROWS * D * 4, at, at + SPAN_BYTES, p, held + slot * SPAN, span, first, last, a.scale, lane, m, l, o);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        if (l[i] == 0.0f) continue;          // nothing seen (a score of NaN is seen: it makes l NaN, whatever m is)
        const Join join(M[i], m[i]);
        if (join.underflows(m[i])) continue;
        M[i] = join.m;
        L[i] = join(L[i], l[i]);
#pragma unroll
        for (int c = 0; c < PAIRS; ++c) {
          const float2 now = unpack(o[i][c]);
          O[i][c] = make_float2(join(O[i][c].x, now.x), join(O[i][c].y, now.y));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int r = r0 + warp * ROWS + i;
      if (r >= rows) continue;
      const float inv = L[i] > 0.0f ? 1.0f / L[i] : 0.0f;
      float* to = a.out + ((long long)(q_start + r / G) * a.q_heads + kvh * G + r % G) * D + lane * (PAIRS * 2);
#pragma unroll
      for (int c = 0; c < PAIRS; ++c)
        *reinterpret_cast<float2*>(to + 2 * c) = make_float2(__fmul_rn(O[i][c].x, inv), __fmul_rn(O[i][c].y, inv));
    }
    return;
  }

  const int few_pos = base_pos + warp / G, few_last = warp < rows ? few_pos : -1;
  const int few_first = a.window > 0 ? max(0, few_pos - a.window + 1) : 0;
  const int rank = blockIdx.x;          // grid.x is a multiple of the cluster, and only its first one has few rows
  float M = -INFINITY, L = 0.0f, O = 0.0f;     // row `rank`, output column threadIdx.x
  for (int s0 = 0; s0 < n_spans; s0 += CLUSTER * SLOTS) {
#pragma unroll
    for (int slot = 0; slot < SLOTS; ++slot) {
      const int s = s0 + slot * CLUSTER + rank;
      if (s < n_spans && !(s0 == 0 && early(s)))
        stage_span(a, seq, kvh, span_first + s, tile_first, tile_last, spans + slot * 2 * SPAN_BYTES, held + slot * SPAN);
    }
    copies_commit();
    copies_wait_all();
    __syncthreads();
    if (warp < rows) {                // row `warp` of every span that is here
      const int row_first[1] = {few_first}, row_last[1] = {few_last};
#pragma unroll 1
      for (int slot = 0; slot < SLOTS && s0 + slot * CLUSTER + rank < n_spans; ++slot) {
        float m[1], l[1];
        pair32 o[1][PAIRS];
        const uint32_t at = spans + slot * 2 * SPAN_BYTES;
        span_state<1>(base + Shared::Q + warp * D * 4, at, at + SPAN_BYTES, p, held + slot * SPAN, span_first + s0 + slot * CLUSTER + rank,
                      row_first, row_last, a.scale, lane, m, l, o);
        float* state = reinterpret_cast<float*>(smem + Shared::STATES) + slot * STATE_FLOATS;
        if (lane == 0) state[warp] = m[0], state[ROWS + warp] = l[0];
#pragma unroll
        for (int c = 0; c < PAIRS; ++c)
          *reinterpret_cast<float2*>(state + 2 * ROWS + warp * D + lane * (PAIRS * 2) + 2 * c) = unpack(o[0][c]);
      }
    }
    cluster_sync();
    if (rank < rows && threadIdx.x < D) {
      const int n = min(CLUSTER * SLOTS, n_spans - s0);
#pragma unroll 8
      for (int s = 0; s < n; ++s) {
        const uint32_t at = base + Shared::STATES + (s / CLUSTER) * (STATE_FLOATS * 4);
        const float m = peer_float(at + rank * 4, s % CLUSTER), l = peer_float(at + (ROWS + rank) * 4, s % CLUSTER);
        const float o = peer_float(at + (2 * ROWS + rank * D + threadIdx.x) * 4, s % CLUSTER);
        if (l == 0.0f) continue;
        const Join join(M, m);
        if (join.underflows(m)) continue;
        M = join.m;
        L = join(L, l);
        O = join(O, o);
      }
    }
    // The states may be written again, and no block leaves while they are read.  The arrival has to release: a relaxed one would not
    // order the reads of other blocks' states before their next writes.  No store to global memory lies ahead of it to wait for.
    cluster_sync();
  }
  if (rank < rows && threadIdx.x < D) {
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
    a.out[((long long)(q_start + rank / G) * a.q_heads + kvh * G + rank % G) * D + threadIdx.x] = __fmul_rn(O, inv);
  }
}

}  // namespace

// `max_q_len`: the most tokens a request of the step brings; `any_few`: some request has at most 8 rows.
extern "C" int llm_attention_f32(const float* q, float* out, float* k_base, float* v_base, const int32_t* block_table,
                                 long long page_stride, int table_stride, int page_tokens, int kv_heads, int head_dim,
                                 const int32_t* q_start, const int32_t* q_len, const int32_t* kv_len, int n_seqs, int max_q_len,
                                 int any_few, int q_heads, float scale, int window, cudaStream_t stream) {
  if (n_seqs <= 0 || max_q_len <= 0) return 0;
  if (head_dim != D || kv_heads < 1 || q_heads % kv_heads || kv_heads > GRID_MAX) return ERR_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(k_base) |
       reinterpret_cast<uintptr_t>(v_base)) & 15 || page_stride % 4)
    return ERR_BAD_ALIGN;
  Args a;
  a.q = q, a.out = out;
  a.q_heads = q_heads, a.group = q_heads / kv_heads, a.window = window, a.scale = scale;
  const int smem = any_few ? Shared::TOTAL_FEW : Shared::TOTAL_WALK;
  static bool raised = false;
  if (!raised) {
    constexpr int most = Shared::TOTAL_FEW > Shared::TOTAL_WALK ? Shared::TOTAL_FEW : Shared::TOTAL_WALK;
    if (cudaFuncSetAttribute(attention_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return launch_status();
    raised = true;
  }
  const long long tiles = ((long long)max_q_len * a.group + TILE_ROWS - 1) / TILE_ROWS;
  cudaLaunchConfig_t cfg = {};
  // clusters only where some request needs one: they leave a few SMs of each group idle
  cfg.gridDim = dim3((unsigned)(any_few ? (tiles + CLUSTER - 1) / CLUSTER * CLUSTER : tiles), kv_heads);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (any_few) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = CLUSTER;
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
  for (int s = 0; s < n_seqs; s += GRID_MAX) {        // (one launch unless a step has more requests than a grid has layers)
    a.cache = PagedCache{k_base, v_base, block_table + (long long)s * table_stride, page_stride, table_stride, page_tokens, kv_heads, head_dim};
    a.q_start = q_start + s, a.q_len = q_len + s, a.kv_len = kv_len + s;
    cfg.gridDim.z = n_seqs - s < GRID_MAX ? n_seqs - s : GRID_MAX;
    if (cudaLaunchKernelEx(&cfg, attention_f32_kernel, a) != cudaSuccess) break;
  }
  return launch_status();
}
