// Linear recurrences of portions of prompts in chunks of 64 tokens: the rules of recurrent.cu without the walk token by
// token.  Per head, with g_t the decay and u_t what is written at token t,
//
//   S_t = g_t S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t (+ skip v_t)
//
// Inside a chunk everything is a product; only the state's way from chunk to chunk is a chain.  With G(i, j) the product of
// the decays behind token j up to token i and G(i) that from the chunk's start:
//
//   chunk_write  N_c = sum_j G(end, j) u_j k_j^T                                           (a block per chunk and head)
//   chunk_chain  the state before every chunk, in place of its N; S <- G(end) S + N_c      (a thread per few elements)
//   chunk_read   O = ((Q K^T) * G(i, j), j <= i) U + G(i) Q S                              (a block per chunk and head)
//
// Under the delta rule u_t = b_t (v_t - g_t S_(t-1)^T k_t) reads the state.  With A(i, j) = b_i G(i, j) k_i . k_j below the
// diagonal and T the inverse of 1 + A, a chunk's writes are U = T (b V) - T (b G K) S, of which all but S is made ahead:
//
//   chunk_solve  T by blocks of 16, W = T (b G K), U_0 = T (b V), K' = G(end, .) K         (a block per chunk and head)
//   chunk_walk   U = U_0 - W S, S <- G(end) S + K'^T U, chunk after chunk                  (a block per head and 16 values)
//   chunk_read   as above
//
// The steps are the published ones: chunks of state-space duality after Dao and Gu, "Transformers are SSMs" (2024), the delta
// rule's inverse and its W and U after Yang et al., "Parallelizing Linear Transformers with the Delta Rule over Sequence
// Length" and "Gated Delta Networks" (both 2024).
//
// Precision.  The state and everything around it is float32, so the products have to be as good as float32: each operand
// enters the tensor cores (mma.sync.m16n8k16, float32 accumulators) as three bfloat16 parts whose sum is the float32 value,
// in the six products of weight 2^-16 and more.  The largest one (high x high) has accumulators of its own: the tensor
// core truncates when it accumulates, and so truncates 4 or 8 times into a sum at full size instead of 24 or 48 times.
// Decays are products of the g, as in the walk, never differences of logarithms, so a decay of 0 is a 0.
// A number that is not finite spoils what the walk lets it spoil, its own token and those behind it: chunk_read takes a chunk
// whose sums are not all finite token by token (walk_chunk).  (The state behind it may hold NaN where the walk's holds an infinity.)
//
// Why chunks: the walk is a chain of about 110 dependent instructions a token and head column, 0.15 to 0.25 us a token
// whatever the machine could do beside it.  Single tokens, short portions and many portions of small states, which fill the
// machine, stay on it (chunks_pay in kernels/device.py).
// 2,048 tokens of 12 heads of 128: 372 us in the walk, 92 in chunks (state-space duality); 507 and 169 (delta rule).
//
// What bounds the kernels: mma.sync (1,024 multiply-adds a cycle and SM; 12 for a 16 x 16 x 16 step) and the reads of shared
// memory that feed it, each about a third of a block's time, behind loads that a block makes once and the splitting of
// operands into parts; chunk_walk the chain itself, 2.4 us a chunk.
#include "recurrent.cuh"
#include "tcgen05.cuh"

namespace distie {

constexpr int kChunkThreads = 256;  // write, solve: two blocks an SM
constexpr int kWideThreads = 512;   // read: one
constexpr int kChunkWarps = kChunkThreads / 32;
constexpr int kKeyPitch = 128;      // elements a row of a matrix over the key's elements
constexpr int kBlocks = kChunk / 16;
constexpr int kImage = 3 * kChunk * kKeyPitch;  // elements of one image

struct ChunkArgs {
  const float *q, *k, *v;
  int q_stride, k_stride, v_stride;
  Sliced decay, write;               // p null: not given
  const float *rate, *bias, *skip;
  float* state;                      // [seats, heads, value_dim, key_dim]
  float* chunks;                     // [2 tiles, heads, value_dim, key_dim]: N, then the state before the chunk
  float* whole;                      // [2 tiles, heads]: G(end)
  __nv_bfloat16* images;             // delta rule, [2 tiles, heads, 2]: W and K' of the chunk as chunk_walk's shared memory holds them
  float* writes;                     // delta rule, [2 tiles, heads, value slices of 16, 64, 16]: U_0, then U
  float* out;
  int out_stride;
  const int *q_tiles, *token_seq, *seq_seat;
  int tiles, heads, groups, key_dim, value_dim, v_dim;
  int* error;
  float q_scale;      // gated rule: q is multiplied by it
  const float* floor; // gated rule with a unit column, [tokens, heads], or null.  Given: what leaves are the v_dim read-outs of
};                    // a head divided by max(|the unit column's|, floor) + 1e-6, without the unit column's own

constexpr int kRuleDelta = 0, kRuleSsd = 1, kRuleGated = 2;

// x as three parts of eight bits each, the low halves of the words; y in the high halves.
__device__ __forceinline__ void three_parts(float x, float y, uint32_t (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    out[i] = *reinterpret_cast<const uint32_t*>(&h);
    x -= __uint_as_float(out[i] << 16);
    y -= __uint_as_float(out[i] & 0xffff0000u);
  }
}

// A matrix as three bfloat16 parts, in shared memory or as an image of it.  Pieces of eight columns are swapped by the
// row's last three bits, so that the eight rows of an ldmatrix lie in different banks.  PITCH: elements of a row, a multiple
// of 64; ROWS: of a part, in elements PITCH * ROWS.  A step of 16 columns is a flip of address bits (stepped) where the
// columns start at 0 and the pitch is a power of two.
template <int PITCH, int ROWS>
struct Triple {
  __nv_bfloat16* p;
  static constexpr int kPitch = PITCH, kPart = PITCH * ROWS;
  static constexpr size_t kBytes = 3 * (size_t)kPart * 2;
  static __device__ __forceinline__ int at(int row, int col) { return row * PITCH + ((((col >> 3) ^ (row & 7)) << 3) | (col & 7)); }
};
// The same with 16 columns: rows lie 48 bytes apart, which keeps an ldmatrix's rows in different banks by itself.
template <int ROWS>
struct NarrowTriple {
  __nv_bfloat16* p;
  static constexpr int kPitch = 24, kPart = kPitch * ROWS;
  static constexpr size_t kBytes = 3 * (size_t)kPart * 2;
  static __device__ __forceinline__ int at(int row, int col) { return row * kPitch + col; }
};
using KeyTriple = Triple<kKeyPitch, kChunk>;  // 64 tokens by the key's elements
using SquareTriple = Triple<kChunk, kChunk>;
template <class M>
__device__ __forceinline__ void put4(const M& m, int row, int col, float4 x) {  // col a multiple of 4
  uint32_t a[3], b[3];
  three_parts(x.x, x.y, a);
  three_parts(x.z, x.w, b);
  __nv_bfloat16* to = m.p + m.at(row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(to + i * M::kPart) = make_uint2(a[i], b[i]);
}
template <class M>
__device__ __forceinline__ void put2(const M& m, int row, int col, float x, float y) {  // col even
  uint32_t a[3];
  three_parts(x, y, a);
  __nv_bfloat16* to = m.p + m.at(row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(to + i * M::kPart) = a[i];
}

// Fragments of m16n8k16 in three parts.  rows: stored [m][k] (first operand) or [n][k] (second), walked along k by
// 16-column steps; turned: [k][m] or [k][n], walked by rows.  A second operand's fragment covers 16 columns: words 0, 1 are
// the first eight, 2, 3 the others.
using Fragment = uint32_t[3][4];
template <class M>
struct AlongRows {  // the lane's place in rows row0 .. row0 + 15, column 0
  const __nv_bfloat16* p;
  int at;
  __device__ __forceinline__ void load(Fragment& f, int step) const {
    const __nv_bfloat16* q = p + (at ^ (16 * step));
#pragma unroll
    for (int i = 0; i < 3; ++i) load_matrices(f[i], q + i * M::kPart);
  }
};
template <class M>
__device__ __forceinline__ AlongRows<M> first_rows(const M& m, int row0, int lane) { return {m.p, M::at(row0 + (lane & 15), (lane >> 4) * 8)}; }
template <class M>
__device__ __forceinline__ AlongRows<M> second_rows(const M& m, int col0, int lane) {
  return {m.p, M::at(col0 + (lane & 7) + (lane >> 4) * 8, ((lane >> 3) & 1) * 8)};
}
template <class M>
struct DownRows {  // the lane's place in rows 0 .. 15
  const __nv_bfloat16* p;
  __device__ __forceinline__ void load(Fragment& f, int step) const {
#pragma unroll
    for (int i = 0; i < 3; ++i) load_matrices_turned(f[i], p + 16 * step * M::kPitch + i * M::kPart);
  }
};
template <class M>
__device__ __forceinline__ DownRows<M> first_turned(const M& m, int row0, int lane) {
  return {m.p + M::at((lane & 7) + (lane >> 4) * 8, row0 + ((lane >> 3) & 1) * 8)};
}
template <class M>
__device__ __forceinline__ DownRows<M> second_turned(const M& m, int col0, int lane) { return {m.p + M::at(lane & 15, col0 + (lane >> 4) * 8)}; }

// 16 x 16 results: the high x high products and the five smaller ones apart.
struct Tile {
  float high[2][4] = {}, rest[2][4] = {};
  __device__ __forceinline__ void add(const Fragment& a, const Fragment& b) {
    constexpr int kFirst[5] = {2, 0, 1, 1, 0}, kSecond[5] = {0, 2, 1, 0, 1};
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int n = 0; n < 2; ++n) mma_16bit(rest[n], a[kFirst[i]], b[kSecond[i]][2 * n], b[kSecond[i]][2 * n + 1]);
#pragma unroll
    for (int n = 0; n < 2; ++n) mma_16bit(high[n], a[0], b[0][2 * n], b[0][2 * n + 1]);
  }
  __device__ __forceinline__ float of(int n, int r) const { return high[n][r] + rest[n][r]; }
};

// The decays of a chunk and what its tokens' writes are multiplied by.  Tokens past the chunk's end: decay 1, factor 0.
struct alignas(16) Decays {
  float g[kChunk], factor[kChunk];
  float pre[kChunk], suf[kChunk];      // within the token's block of 16: the product up to it, and behind it
  float from_start[kChunk], to_end[kChunk];
  float inside[kBlocks][16][17];       // G(i, j) of two tokens of one block
  // The product of all decays of the blocks between bi and bj < bi: G(i, j) = suf[j] * blocks(bi, bj) * pre[i].
  __device__ __forceinline__ float blocks(int bi, int bj) const {
    float x = 1.f;
    for (int b = bj + 1; b < bi; ++b) x *= pre[16 * b + 15];
    return x;
  }
};

// The elements of a 16 x 16 result (rows of block bi, columns of block bj, bi >= bj) times G(i, j); zeros above the diagonal.
__device__ __forceinline__ void times_decays(float (&x)[2][4], const Tile& t, const Decays& d, int bi, int bj, int lane) {
  const int g = lane >> 2, c = lane & 3;
  if (bi == bj) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 4; ++r) x[n][r] = t.of(n, r) * d.inside[bi][g + 8 * (r >> 1)][8 * n + 2 * c + (r & 1)];
  } else {
    const float mid = d.blocks(bi, bj), up[2] = {d.pre[16 * bi + g] * mid, d.pre[16 * bi + g + 8] * mid};
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const float2 down = *reinterpret_cast<const float2*>(&d.suf[16 * bj + 8 * n + 2 * c]);
#pragma unroll
      for (int r = 0; r < 4; ++r) x[n][r] = t.of(n, r) * (up[r >> 1] * (r & 1 ? down.y : down.x));
    }
  }
}

// Every thread of the block calls it; it ends with a barrier.
__device__ __forceinline__ void make_decays(Decays& d, const ChunkArgs& a, int rule, int head, int t0, int rows) {
  const int t = threadIdx.x;
  if (t < kChunk) {
    float g = 1.f, factor = 0.f;
    if (t < rows) {
      const size_t token = t0 + t;
      if (rule == kRuleGated) {
        g = a.decay.p ? a.decay.at(token, head) : a.rate[head];
        factor = a.write.p ? a.write.at(token, head) : 1.f;
      } else {
        const float rate = expf(a.rate[head]), bias = a.bias ? a.bias[head] : 0.f, w = a.write.at(token, head);
        factor = rule == kRuleDelta ? sigmoid_f(w) : softplus_f(w + bias);
        g = expf(-rate * (rule == kRuleDelta ? softplus_f(a.decay.at(token, head) + bias) : factor));
      }
    }
    d.g[t] = g;
    d.factor[t] = factor;
  }
  __syncthreads();
  if (t < kChunk) {
    const int b = t >> 4, j = t & 15;
    float down = 1.f, up = 1.f;
    for (int i = 0; i < 16; ++i) {
      const float g = d.g[16 * b + i];
      if (i > j) down *= g;
      if (i <= j) up *= g;
      d.inside[b][i][j] = i >= j ? down : 0.f;
    }
    d.pre[t] = up;
    d.suf[t] = down;
  }
  __syncthreads();
  if (t < kChunk) {
    const int b = t >> 4;
    float start = d.pre[t], end = d.suf[t];
    for (int i = 0; i < b; ++i) start *= d.pre[16 * i + 15];
    for (int i = b + 1; i < kBlocks; ++i) end *= d.pre[16 * i + 15];
    d.from_start[t] = start;
    d.to_end[t] = end;
  }
  __syncthreads();
}

// Whether rows of `dim` floats can be read four at a time.
__device__ __forceinline__ bool by_fours(const float* p, int stride, int dim) {
  return (dim & 3) == 0 && (stride & 3) == 0 && ((uintptr_t)p & 15) == 0;
}
__device__ __forceinline__ float4 four_at(const float* p, int col, int dim, bool fours) {
  if (fours) return *reinterpret_cast<const float4*>(p + col);
  return make_float4(p[col], col + 1 < dim ? p[col + 1] : 0.f, col + 2 < dim ? p[col + 2] : 0.f, col + 3 < dim ? p[col + 3] : 0.f);
}

// COUNT rows of a matrix, a warp a row and four elements a lane (from column 4 lane + offset on): fetched first, stored
// as parts later, so that the loads of several matrices are in flight together.  Rows from `live` on and elements from
// `dim` on are zeros, except that with `unit` element `dim` of a live row is 1.
template <int COUNT, int THREADS>
struct Rows {
  static constexpr int LANES = 32, kStep = THREADS / LANES, kMine = (COUNT + kStep - 1) / kStep;
  float4 x[kMine];
  static __device__ __forceinline__ int row(int i) { return (int)threadIdx.x / LANES + i * kStep; }
  static __device__ __forceinline__ int column(int offset) { return 4 * ((int)threadIdx.x % LANES) + offset; }
  __device__ __forceinline__ void fetch(const float* src, int stride, int live, int dim, int offset = 0) {
    const int c = column(offset);
    const bool fours = by_fours(src, stride, dim);
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row(i) < live && c < dim) x[i] = four_at(src + (size_t)row(i) * stride, c, dim, fours);
    }
  }
  // From the slices of 16 columns that chunk_walk leaves.
  __device__ __forceinline__ void fetch_slices(const float* src, int padded, int offset = 0) {
    const int c = column(offset);
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < padded) x[i] = *reinterpret_cast<const float4*>(src + ((size_t)(c >> 4) * kChunk + row(i)) * 16 + (c & 15));
    }
  }
  __device__ __forceinline__ void scale(float s) {
#pragma unroll
    for (int i = 0; i < kMine; ++i) x[i] = make_float4(x[i].x * s, x[i].y * s, x[i].z * s, x[i].w * s);
  }
  // Rows of at most 128 elements made unit vectors, times `scale`.
  __device__ __forceinline__ void make_unit(float scale) {
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const float s = scale / sqrtf(warp_sum(x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w) + 1e-6f);
      x[i] = make_float4(x[i].x * s, x[i].y * s, x[i].z * s, x[i].w * s);
    }
  }
  // weight: per row, or null
  template <class M>
  __device__ __forceinline__ void store(const M& m, int count, int live, int dim, int padded, const float* weight, bool unit,
                                        int offset = 0) {
    const int c = column(offset);
    if (c >= padded) return;
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int r = row(i);
      if (r >= count) break;
      if (unit && r < live) {
        if (c == dim) x[i].x = 1.f;
        if (c + 1 == dim) x[i].y = 1.f;
        if (c + 2 == dim) x[i].z = 1.f;
        if (c + 3 == dim) x[i].w = 1.f;
      }
      const float w = weight ? weight[r] : 1.f;
      put4(m, r, c, make_float4(x[i].x * w, x[i].y * w, x[i].z * w, x[i].w * w));
    }
  }
};

// N^T [value_dim, key_dim] of a chunk: rows are value elements (U^T is the first operand), columns key elements.  VALUES:
// columns of U in shared memory (value_dim up to 128, or to 144).
template <int RULE, int VALUES>
__global__ void __launch_bounds__(kChunkThreads, VALUES > 128 ? 1 : 2) chunk_write_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  using ValueTriple = Triple<VALUES, kChunk>;
  const KeyTriple k{reinterpret_cast<__nv_bfloat16*>(chunk_s)};
  const ValueTriple u{reinterpret_cast<__nv_bfloat16*>(chunk_s + KeyTriple::kBytes)};
  const int group = head / (a.heads / a.groups);
  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  Rows<kChunk, kChunkThreads> fetched_k, fetched_u;
  fetched_k.fetch(a.k + (size_t)t0 * a.k_stride + group * a.key_dim, a.k_stride, rows, a.key_dim);
  fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim);
  make_decays(d, a, RULE, head, t0, rows);
  if (threadIdx.x < kChunk) d.factor[threadIdx.x] *= d.to_end[threadIdx.x];
  if (threadIdx.x == 0) a.whole[(size_t)blockIdx.y * a.heads + head] = d.from_start[kChunk - 1];
  __syncthreads();
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim);
  const bool unit_column = a.v_dim < a.value_dim;
  fetched_k.store(k, kChunk, rows, a.key_dim, key_padded, nullptr, false);
  fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, d.factor, unit_column);
  if (VALUES > 128) {
    fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, d.factor, unit_column, 128);
  }
  __syncthreads();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int m_tiles = value_padded / 16, n_pairs = (key_padded + 31) / 32, steps = (rows + 15) / 16;
  float* dst = a.chunks + ((size_t)blockIdx.y * a.heads + head) * a.value_dim * a.key_dim;
  const bool pairs = (a.key_dim & 1) == 0;
  for (int unit = warp; unit < m_tiles * n_pairs; unit += kChunkWarps) {  // 16 value by 32 key elements
    const int m0 = unit % m_tiles * 16, n0 = unit / m_tiles * 32;
    const bool both = n0 + 16 < key_padded;
    const auto u_at = first_turned(u, m0, lane);
    const auto k_at = second_turned(k, n0, lane), k_next = second_turned(k, n0 + 16, lane);
    Tile acc[2];
    for (int s = 0; s < steps; ++s) {
      Fragment x, y;
      u_at.load(x, s);
      k_at.load(y, s);
      acc[0].add(x, y);
      if (both) {
        k_next.load(y, s);
        acc[1].add(x, y);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = m0 + g + 8 * h, col = n0 + 8 * j + 2 * c;
        if (row >= a.value_dim || col >= a.key_dim) continue;
        const float x = acc[j >> 1].of(j & 1, 2 * h), y = acc[j >> 1].of(j & 1, 2 * h + 1);
        float* to = dst + (size_t)row * a.key_dim + col;
        if (pairs) *reinterpret_cast<float2*>(to) = make_float2(x, y);
        else {
          to[0] = x;
          if (col + 1 < a.key_dim) to[1] = y;
        }
      }
  }
}

// The chain of the rules whose write does not read the state: a thread owns W neighbouring elements of one head's state.
// A block whose tile is not the first of its request has nothing to do.
constexpr int kChainThreads = 256;
template <int W>
__global__ void __launch_bounds__(kChainThreads) chunk_chain_kernel(ChunkArgs a) {
  const int tile0 = blockIdx.z, head = blockIdx.y;
  const int seq = a.token_seq[a.q_tiles[2 * tile0]];
  if (tile0 > 0 && a.token_seq[a.q_tiles[2 * (tile0 - 1)]] == seq) return;
  const size_t size = (size_t)a.value_dim * a.key_dim, at = ((size_t)blockIdx.x * kChainThreads + threadIdx.x) * W;
  if (at >= size) return;
  struct alignas(4 * W) Piece { float v[W]; };
  Piece* slot = reinterpret_cast<Piece*>(a.state + ((size_t)a.seq_seat[seq] * a.heads + head) * size + at);
  Piece S = *slot;
  float* mine = a.chunks + (size_t)head * size + at;
  const size_t stride = (size_t)a.heads * size;
  constexpr int kAhead = 4;  // tiles whose chunks are in flight together
  for (int tile = tile0; tile < a.tiles; tile += kAhead) {
    int rows[kAhead];
    bool more = true;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      more = more && tile + j < a.tiles && a.token_seq[a.q_tiles[2 * (tile + j)]] == seq;
      rows[j] = more ? a.q_tiles[2 * (tile + j) + 1] : 0;
    }
    Piece n[2 * kAhead];
    float whole[2 * kAhead];
#pragma unroll
    for (int j = 0; j < 2 * kAhead; ++j)
      if (rows[j >> 1] > (j & 1) * kChunk) {
        n[j] = *reinterpret_cast<const Piece*>(mine + (size_t)(2 * tile + j) * stride);
        whole[j] = a.whole[(size_t)(2 * tile + j) * a.heads + head];
      }
#pragma unroll
    for (int j = 0; j < 2 * kAhead; ++j)
      if (rows[j >> 1] > (j & 1) * kChunk) {
        *reinterpret_cast<Piece*>(mine + (size_t)(2 * tile + j) * stride) = S;
#pragma unroll
        for (int e = 0; e < W; ++e) S.v[e] = fmaf(whole[j], S.v[e], n[j].v[e]);
      }
    if (!more) break;
  }
  *slot = S;
}

// The inverse T of 1 + A, A [64, 64] strictly below the diagonal, both with rows of kSolvePitch floats; T arrives as zeros.
// Blocks of 16 by substitution, a thread a column; then pairs of blocks, then the pair of pairs:
// [1 + A11, 0; A21, 1 + A22] has the inverse [T11, 0; -T22 A21 T11, T22].  m_s: 32 x 33 floats.
constexpr int kSolvePitch = 68;
__device__ __forceinline__ void invert(const float* A, float* T, float* m_s) {
  const int tid = threadIdx.x;
  static_assert(kChunkThreads == 256, "threads are shared out by hand");
  if (tid < kChunk) {
    const int b0 = tid & ~15, j = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float sum = 0.f;
#pragma unroll
      for (int l = 0; l < i; ++l) sum += A[(b0 + i) * kSolvePitch + b0 + l] * x[l];
      x[i] = i == j ? 1.f : (i > j ? -sum : 0.f);
      T[(b0 + i) * kSolvePitch + tid] = x[i];
    }
  }
  __syncthreads();
  {  // rows 16 + i of both pairs
    const int i = tid >> 4, l = tid & 15;
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int m = 0; m < 16; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p) sum[p] += A[(32 * p + 16 + i) * kSolvePitch + 32 * p + m] * T[(32 * p + m) * kSolvePitch + 32 * p + l];
#pragma unroll
    for (int p = 0; p < 2; ++p) m_s[(16 * p + i) * 16 + l] = sum[p];
    __syncthreads();
    sum[0] = sum[1] = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p) sum[p] += T[(32 * p + 16 + i) * kSolvePitch + 32 * p + 16 + m] * m_s[(16 * p + m) * 16 + l];
#pragma unroll
    for (int p = 0; p < 2; ++p) T[(32 * p + 16 + i) * kSolvePitch + 32 * p + l] = -sum[p];
  }
  __syncthreads();
  const int i = tid >> 5, l = tid & 31;  // rows i, i + 8, i + 16, i + 24
  float sum[4] = {};
#pragma unroll 8
  for (int m = 0; m < 32; ++m) {
    const float t = T[m * kSolvePitch + l];
#pragma unroll
    for (int h = 0; h < 4; ++h) sum[h] += A[(32 + i + 8 * h) * kSolvePitch + m] * t;
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) m_s[(i + 8 * h) * 33 + l] = sum[h];
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 4; ++h) sum[h] = 0.f;
#pragma unroll 8
  for (int m = 0; m < 32; ++m) {
    const float x = m_s[m * 33 + l];
#pragma unroll
    for (int h = 0; h < 4; ++h) sum[h] += T[(32 + i + 8 * h) * kSolvePitch + 32 + m] * x;
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) T[(32 + i + 8 * h) * kSolvePitch + l] = -sum[h];
  __syncthreads();
}

// What the delta rule's chunk needs besides the state: T, W and K' (images), U_0.  Shared memory: K as parts (then, with
// the place of A and T, b V), A and T as floats, T as parts.
constexpr size_t kSolveShared = KeyTriple::kBytes + 2 * (size_t)kChunk * kSolvePitch * 4 + SquareTriple::kBytes;
static_assert(Triple<192, kChunk>::kBytes <= KeyTriple::kBytes + 2 * (size_t)kChunk * kSolvePitch * 4, "V in the place of K, A and T");
__global__ void __launch_bounds__(kChunkThreads, 2) chunk_solve_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), group = head / (a.heads / a.groups);
  unsigned char* at = chunk_s;
  const KeyTriple k{reinterpret_cast<__nv_bfloat16*>(at)};
  const Triple<192, kChunk> v{k.p};
  at += KeyTriple::kBytes;
  float* A = reinterpret_cast<float*>(at);
  float* T = A + kChunk * kSolvePitch;
  at += 2 * kChunk * kSolvePitch * sizeof(float);
  float* m_s = reinterpret_cast<float*>(at);
  const SquareTriple t_s{reinterpret_cast<__nv_bfloat16*>(at)};
  const size_t chunk_head = (size_t)blockIdx.y * a.heads + head;
  const KeyTriple w_image{a.images + 2 * chunk_head * kImage};
  const KeyTriple k_image{a.images + (2 * chunk_head + 1) * kImage};
  float* writes = a.writes + chunk_head * value_padded * kChunk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;

  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  Rows<kChunk, kChunkThreads> fetched;
  fetched.fetch(a.k + (size_t)t0 * a.k_stride + group * a.key_dim, a.k_stride, rows, a.key_dim);
  for (int i = threadIdx.x; i < 2 * kChunk * kSolvePitch; i += kChunkThreads) A[i] = 0.f;
  make_decays(d, a, kRuleDelta, head, t0, rows);
  if (threadIdx.x == 0) a.whole[chunk_head] = d.from_start[kChunk - 1];
  fetched.make_unit(1.f);
  fetched.store(k, kChunk, rows, a.key_dim, key_padded, nullptr, false);
  fetched.store(k_image, kChunk, rows, a.key_dim, key_padded, d.to_end, false);
  __syncthreads();

  for (int block = warp; block < 10; block += kChunkWarps) {  // the blocks of 16 x 16 on and below the diagonal
    const int bi = block < 1 ? 0 : block < 3 ? 1 : block < 6 ? 2 : 3, bj = block - bi * (bi + 1) / 2;
    const auto x_at = first_rows(k, bi * 16, lane), y_at = second_rows(k, bj * 16, lane);
    Tile acc;
    for (int s = 0; s < key_padded / 16; ++s) {
      Fragment x, y;
      x_at.load(x, s);
      y_at.load(y, s);
      acc.add(x, y);
    }
    float made[2][4];
    times_decays(made, acc, d, bi, bj, lane);
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = bi * 16 + g + 8 * (r >> 1), j = bj * 16 + 8 * n + 2 * c + (r & 1);
        if (j < i) A[i * kSolvePitch + j] = d.factor[i] * made[n][r];
      }
  }
  __syncthreads();
  invert(A, T, m_s);
  // Rows of 16 tokens see up to 16 (row + 1) of them: a warp takes all four, for the columns of its units.
  auto times = [&](const auto& m, int unit, Tile (&acc)[4]) {
    const auto y_at = second_turned(m, unit * 16, lane);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      Fragment x, y;
      y_at.load(y, s);
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        if (mt < s) continue;
        first_rows(t_s, mt * 16, lane).load(x, s);
        acc[mt].add(x, y);
      }
    }
  };
  auto weigh = [&](bool from_start) {
    for (int idx = threadIdx.x; idx < kChunk * kChunk / 2; idx += kChunkThreads) {
      const int i = idx / (kChunk / 2), j = 2 * (idx % (kChunk / 2));
      const float x = T[i * kSolvePitch + j] * d.factor[j], y = T[i * kSolvePitch + j + 1] * d.factor[j + 1];
      put2(t_s, i, j, from_start ? x * d.from_start[j] : x, from_start ? y * d.from_start[j + 1] : y);
    }
  };
  weigh(true);
  __syncthreads();
  fetched.fetch(v_rows, a.v_stride, rows, a.v_dim);
  for (int unit = warp; unit < key_padded / 16; unit += kChunkWarps) {
    Tile acc[4];
    times(k, unit, acc);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          put2(w_image, mt * 16 + g + 8 * h, unit * 16 + 8 * n + 2 * c, acc[mt].of(n, 2 * h), acc[mt].of(n, 2 * h + 1));
  }
  __syncthreads();
  weigh(false);
  __syncthreads();  // T is in parts, K done with
  fetched.store(v, kChunk, rows, a.v_dim, value_padded, nullptr, false);
  if (value_padded > 128) {
    fetched.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched.store(v, kChunk, rows, a.v_dim, value_padded, nullptr, false, 128);
  }
  __syncthreads();
  for (int unit = warp; unit < value_padded / 16; unit += kChunkWarps) {
    Tile acc[4];
    times(v, unit, acc);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(writes + ((size_t)unit * kChunk + mt * 16 + g + 8 * h) * 16 + 8 * n + 2 * c) =
              make_float2(acc[mt].of(n, 2 * h), acc[mt].of(n, 2 * h + 1));
  }
}

// The chain of the delta rule: 16 value elements of one head's state, chunk after chunk.  What it reads of a chunk (W and
// K', 96 KB) is copied a chunk ahead.  Sixteen warps: in the first product four share the 16 tokens of a row of tiles, each
// a quarter of the keys, and finish a quarter of the result each; in the second one each owns eight keys of the state.  A
// block whose tile is not the first of its request has nothing to do.  STEPS: key_dim / 16 rounded up, 0: any.
constexpr int kWalkThreads = 512;
constexpr size_t kWalkStage = 2 * (size_t)kImage * 2;
constexpr size_t kWalkShared = 2 * kWalkStage + 16 + Triple<kKeyPitch, 16>::kBytes + NarrowTriple<kChunk>::kBytes + 16 * 3 * 32 * 8;
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
template <int STEPS>
__global__ void __launch_bounds__(kWalkThreads, 1) chunk_walk_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  const int slice = blockIdx.x, head = blockIdx.y, tile0 = blockIdx.z, tid = threadIdx.x;
  const int seq = a.token_seq[a.q_tiles[2 * tile0]];
  if (tile0 > 0 && a.token_seq[a.q_tiles[2 * (tile0 - 1)]] == seq) return;
  uint64_t* full = reinterpret_cast<uint64_t*>(chunk_s + 2 * kWalkStage);  // one a stage
  unsigned char* at = chunk_s + 2 * kWalkStage + 16;
  const Triple<kKeyPitch, 16> S_s{reinterpret_cast<__nv_bfloat16*>(at)};
  const NarrowTriple<kChunk> u_s{reinterpret_cast<__nv_bfloat16*>(at + S_s.kBytes)};
  float2* quarter_s = reinterpret_cast<float2*>(at + S_s.kBytes + u_s.kBytes);  // [4 to][3 from][4 mt][32]
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), steps = STEPS ? STEPS : key_padded / 16;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  const int mt = warp & 3, kq = warp >> 2;
  const bool owner = warp * 8 < key_padded;  // of keys of the state

  auto copy_chunk = [&](int chunk, int stage) {  // one thread; W and K' lie side by side
    mbar_expect_tx(&full[stage], (uint32_t)kWalkStage);
    bulk_load(chunk_s + stage * kWalkStage, a.images + 2 * ((size_t)chunk * a.heads + head) * kImage, (uint32_t)kWalkStage, &full[stage]);
  };
  // The request's tiles follow one another, all but the last of them full: its chunks are a range.
  int tiles = 0;
  for (int ahead = 0; tile0 + ahead < a.tiles; ahead += kWalkThreads) {
    const int tile = tile0 + ahead + tid;
    const int mine = __syncthreads_count(tile < a.tiles && a.token_seq[a.q_tiles[2 * min(tile, a.tiles - 1)]] == seq);
    tiles += mine;
    if (mine < kWalkThreads) break;
  }
  const int end = 2 * (tile0 + tiles) - (a.q_tiles[2 * (tile0 + tiles) - 1] <= kChunk);
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    copy_chunk(2 * tile0, 0);
  }
  // the warp's part of S^T: 16 values by the 8 keys from 8 warp on
  float S[4];
  const size_t size = (size_t)a.value_dim * a.key_dim;
  float* slot = a.state + ((size_t)a.seq_seat[seq] * a.heads + head) * size;
  const bool pairs = (a.key_dim & 1) == 0 && ((uintptr_t)a.state & 7) == 0;
  const int col0 = warp * 8 + 2 * c, row0 = slice * 16 + g;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int row = row0 + 8 * (r >> 1), col = col0 + (r & 1);
    S[r] = row < a.value_dim && col < a.key_dim ? slot[(size_t)row * a.key_dim + col] : 0.f;
  }
  auto store_state = [&](float* to) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = row0 + 8 * h;
      if (row >= a.value_dim || col0 >= a.key_dim) continue;
      float* p = to + (size_t)row * a.key_dim + col0;
      if (pairs) *reinterpret_cast<float2*>(p) = make_float2(S[2 * h], S[2 * h + 1]);
      else {
        p[0] = S[2 * h];
        if (col0 + 1 < a.key_dim) p[1] = S[2 * h + 1];
      }
    }
  };
  auto share_state = [&]() {
    if (owner) {
#pragma unroll
      for (int h = 0; h < 2; ++h) put2(S_s, g + 8 * h, col0, S[2 * h], S[2 * h + 1]);
    }
  };
  share_state();
  __syncthreads();  // the barriers are there

  // quarter kq of a 16 x 16 tile: its eight columns from 8 (kq & 1), rows g or g + 8
  float2* out = reinterpret_cast<float2*>(a.writes + (((size_t)2 * tile0 * a.heads + head) * value_padded + (size_t)slice * 16) * kChunk +
                                          (mt * 16 + g + 8 * (kq >> 1)) * 16 + 8 * (kq & 1) + 2 * c);
  const size_t out_step = (size_t)a.heads * value_padded * kChunk / 2, chunk_step = (size_t)a.heads * size;
  float* before = a.chunks + ((size_t)2 * tile0 * a.heads + head) * size;
  const float* whole_at = a.whole + (size_t)2 * tile0 * a.heads + head;
  float2 ahead = *out;  // U_0 of the coming chunk
  float whole = *whole_at;
  for (int chunk = 2 * tile0, round = 0; chunk < end; ++chunk, ++round) {
    const int stage = round & 1;
    const bool more = chunk + 1 < end;
    if (more && tid == 0) copy_chunk(chunk + 1, stage ^ 1);  // its last readers passed a barrier behind their last product
    const float2 u0 = ahead;
    const float decay = whole;
    if (more) {
      ahead = out[out_step];
      whole = *(whole_at += a.heads);
    }
    const bool here = mbar_wait(&full[stage], (round >> 1) & 1);
    if (__syncthreads_or(!here)) {  // (given up: the copies in flight get the same time to land)
      if (tid == 0) {
        atomicExch(a.error, 6);
        if (more) mbar_wait(&full[stage ^ 1], ((round + 1) >> 1) & 1);
      }
      return;
    }
    const KeyTriple w{reinterpret_cast<__nv_bfloat16*>(chunk_s + stage * kWalkStage)}, k{w.p + kImage};
    const auto w_at = first_rows(w, mt * 16, lane);
    const auto S_at = second_rows(S_s, 0, lane);
    store_state(before);
    before += chunk_step;

    {
      Tile sum;
      if (STEPS) {
#pragma unroll
        for (int i = 0; i < (STEPS + 3) / 4; ++i) {
          const int s = kq + 4 * i;
          if (STEPS % 4 && s >= STEPS) break;
          Fragment x, y;
          w_at.load(x, s);
          S_at.load(y, s);
          sum.add(x, y);
        }
      } else {
        for (int s = kq; s < steps; s += 4) {
          Fragment x, y;
          w_at.load(x, s);
          S_at.load(y, s);
          sum.add(x, y);
        }
      }
      float2 own = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 part = make_float2(sum.of(i & 1, 2 * (i >> 1)), sum.of(i & 1, 2 * (i >> 1) + 1));
        if (i == kq) own = part;
        else quarter_s[((i * 3 + (kq > i ? kq - 1 : kq)) * 4 + mt) * 32 + lane] = part;
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float2 part = quarter_s[((kq * 3 + i) * 4 + mt) * 32 + lane];
        own.x += part.x;
        own.y += part.y;
      }
      const float2 u = make_float2(u0.x - own.x, u0.y - own.y);
      put2(u_s, mt * 16 + g + 8 * (kq >> 1), 8 * (kq & 1) + 2 * c, u.x, u.y);
      *out = u;
      out += out_step;
    }
    __syncthreads();
    if (owner) {
      const auto u_at = first_turned(u_s, 0, lane);
      float high[4] = {}, rest[2][4] = {};
#pragma unroll
      for (int s = 0; s < kChunk / 16; s += 2) {
        Fragment x0, x1, y;  // y: eight keys, both steps
        u_at.load(x0, s);
        u_at.load(x1, s + 1);
        const __nv_bfloat16* p = k.p + k.at(16 * s + lane, warp * 8);
#pragma unroll
        for (int i = 0; i < 3; ++i) load_matrices_turned(y[i], p + i * k.kPart);
        constexpr int kFirst[5] = {2, 0, 1, 1, 0}, kSecond[5] = {0, 2, 1, 0, 1};
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          mma_16bit(rest[0], x0[kFirst[i]], y[kSecond[i]][0], y[kSecond[i]][1]);
          mma_16bit(rest[1], x1[kFirst[i]], y[kSecond[i]][2], y[kSecond[i]][3]);
        }
        mma_16bit(high, x0[0], y[0][0], y[0][1]);
        mma_16bit(high, x1[0], y[0][2], y[0][3]);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) S[r] = fmaf(decay, S[r], high[r] + (rest[0][r] + rest[1][r]));
    }
    share_state();  // (every warp has read the old one: two barriers ago)
    if (more) __syncthreads();  // this stage's copies may be overwritten from here on
  }
  store_state(slot);
}

// The read-outs of a chunk token by token, as the walk of recurrent.cu takes them, from the state before the chunk: what
// chunk_read does when a sum of its products is not finite.  A product with a weight of 0 for a token that a row does not see is NaN
// when that token's numbers are not finite; here a row meets nothing behind it.  A warp a value element, the state's column
// over its lanes.  Every thread of the block calls it; reads_s: rows * value_dim floats.
template <int RULE>
__device__ __noinline__ void walk_chunk(const ChunkArgs& a, const Decays& d, float* reads_s, int chunk, int head, int t0, int rows) {
  const int lane = threadIdx.x & 31, group = head / (a.heads / a.groups);
  const float skip = RULE == kRuleSsd && a.skip ? a.skip[head] : 0.f;
  for (int j = threadIdx.x >> 5; j < a.value_dim; j += kWideThreads / 32) {
    const float* column = a.chunks + (((size_t)chunk * a.heads + head) * a.value_dim + j) * a.key_dim;
    float S[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) S[r] = lane + 32 * r < a.key_dim ? column[lane + 32 * r] : 0.f;
    for (int t = 0; t < rows; ++t) {
      const float* q_row = a.q + (size_t)(t0 + t) * a.q_stride + group * a.key_dim;
      const float* k_row = a.k + (size_t)(t0 + t) * a.k_stride + group * a.key_dim;
      float q[4], k[4], qq = 0.f, kk = 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool live = lane + 32 * r < a.key_dim;
        q[r] = live ? q_row[lane + 32 * r] : 0.f;
        k[r] = live ? k_row[lane + 32 * r] : 0.f;
        qq += q[r] * q[r];
        kk += k[r] * k[r];
      }
      if (RULE == kRuleDelta) {
        qq = rsqrtf((float)a.key_dim) / sqrtf(warp_sum(qq) + 1e-6f);
        kk = 1.f / sqrtf(warp_sum(kk) + 1e-6f);
      }
      float kq = 0.f, sum_k = 0.f, sum_q = 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (RULE == kRuleDelta) q[r] *= qq, k[r] *= kk;
        if (RULE == kRuleGated) q[r] *= a.q_scale;
        kq += k[r] * q[r];
        sum_k += S[r] * k[r];
        sum_q += S[r] * q[r];
      }
      const float g = d.g[t], factor = d.factor[t], v = j < a.v_dim ? a.v[(size_t)(t0 + t) * a.v_stride + (size_t)head * a.v_dim + j] : 1.f;
      const float u = RULE == kRuleDelta ? factor * (v - g * warp_sum(sum_k)) : factor * v;
#pragma unroll
      for (int r = 0; r < 4; ++r) S[r] = g * S[r] + k[r] * u;
      const float read = g * warp_sum(sum_q) + u * warp_sum(kq);
      if (lane == 0) reads_s[t * a.value_dim + j] = RULE == kRuleSsd ? read + skip * v : read;
    }
  }
  __syncthreads();
  const bool divided = RULE == kRuleGated && a.floor;
  const int columns = divided ? a.v_dim : a.value_dim;
  for (int idx = threadIdx.x; idx < rows * columns; idx += kWideThreads) {
    const int t = idx / columns, j = idx % columns;
    float x = reads_s[t * a.value_dim + j];
    if (divided) x /= fmaxf(fabsf(reads_s[t * a.value_dim + a.v_dim]), a.floor[(size_t)(t0 + t) * a.heads + head]) + 1e-6f;
    a.out[(size_t)(t0 + t) * a.out_stride + (size_t)head * columns + j] = x;
  }
}

// O of a chunk from its own tokens and the state before it.  Shared memory: Q | K | S, then Q | the scores | U.
using StateTriple = Triple<kKeyPitch, 144>;
constexpr size_t read_shared(int value_dim) {  // (parts of S and U lie as for 144 values where there are more than 128)
  return 2 * KeyTriple::kBytes + (value_dim > 128 ? StateTriple::kBytes : Triple<kKeyPitch, 128>::kBytes);
}
template <int RULE, int VALUES>
__global__ void __launch_bounds__(kWideThreads, 1) chunk_read_kernel(const __grid_constant__ ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), group = head / (a.heads / a.groups);
  constexpr int kStateRows = VALUES > 128 ? 144 : 128;
  using ValueTriple = Triple<VALUES, kChunk>;
  static_assert(ValueTriple::kBytes <= Triple<kKeyPitch, kStateRows>::kBytes, "U in the place of S");
  const KeyTriple q{reinterpret_cast<__nv_bfloat16*>(chunk_s)}, k{reinterpret_cast<__nv_bfloat16*>(chunk_s + KeyTriple::kBytes)};
  const Triple<kKeyPitch, kStateRows> S{reinterpret_cast<__nv_bfloat16*>(chunk_s + 2 * KeyTriple::kBytes)};
  const SquareTriple p{k.p};
  const ValueTriple u{S.p};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  // 16 rows of the chunk; a quarter of the columns.  Later rows see more keys: each scheduler gets warps of all four.
  const int cq = warp >> 2, rg = (warp + cq) & 3;
  const int row0 = rg * 16 + g;
  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  const bool unit_column = a.v_dim < a.value_dim;
  Rows<kChunk, kWideThreads> fetched_u;
  {
    Rows<kChunk, kWideThreads> fetched_q, fetched_k;
    Rows<kStateRows, kWideThreads> fetched_S;
    fetched_q.fetch(a.q + (size_t)t0 * a.q_stride + group * a.key_dim, a.q_stride, rows, a.key_dim);
    fetched_k.fetch(a.k + (size_t)t0 * a.k_stride + group * a.key_dim, a.k_stride, rows, a.key_dim);
    fetched_S.fetch(a.chunks + ((size_t)blockIdx.y * a.heads + head) * a.value_dim * a.key_dim, a.key_dim, a.value_dim, a.key_dim);
    make_decays(d, a, RULE, head, t0, rows);
    if (RULE == kRuleDelta) {
      fetched_q.make_unit(rsqrtf((float)a.key_dim));
      fetched_k.make_unit(1.f);
    }
    if (RULE == kRuleGated) fetched_q.scale(a.q_scale);
    fetched_q.store(q, kChunk, rows, a.key_dim, key_padded, nullptr, false);
    fetched_k.store(k, kChunk, rows, a.key_dim, key_padded, nullptr, false);
    fetched_S.store(S, value_padded, a.value_dim, a.key_dim, key_padded, nullptr, false);
  }
  __syncthreads();

  const int steps = key_padded / 16, units = value_padded / 16;  // 16 values a unit
  constexpr int kUnits = VALUES > 128 ? 3 : 2;                    // at most, a warp
  const auto q_at = first_rows(q, rg * 16, lane);
  float o[kUnits][2][4], score[2][4] = {};
  if (cq <= rg) {  // the warp's keys are not all behind its rows
    const auto k_at = second_rows(k, cq * 16, lane);
    Tile acc;
#pragma unroll 2
    for (int s = 0; s < steps; ++s) {
      Fragment x, y;
      q_at.load(x, s);
      k_at.load(y, s);
      acc.add(x, y);
    }
    times_decays(score, acc, d, rg, cq, lane);
  }
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int unit = cq + 4 * i;
    if (unit < units) {
      const auto S_at = second_rows(S, unit * 16, lane);
      Tile acc;
#pragma unroll 2
      for (int s = 0; s < steps; ++s) {
        Fragment x, y;
        q_at.load(x, s);
        S_at.load(y, s);
        acc.add(x, y);
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) o[i][n][r] = acc.of(n, r) * d.from_start[row0 + (r >> 1) * 8];
    }
  }
  const float* writes = a.writes + ((size_t)blockIdx.y * a.heads + head) * value_padded * kChunk;
  const float* factor = RULE == kRuleDelta ? nullptr : d.factor;
  if (RULE == kRuleDelta) fetched_u.fetch_slices(writes, value_padded);
  else fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim);
  __syncthreads();  // K and S are done with
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) put2(p, row0 + 8 * h, cq * 16 + 8 * n + 2 * c, score[n][2 * h], score[n][2 * h + 1]);
  fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, factor, unit_column);
  if (VALUES > 128) {
    if (RULE == kRuleDelta) fetched_u.fetch_slices(writes, value_padded, 128);
    else fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, factor, unit_column, 128);
  }
  __syncthreads();

  const float skip = (RULE == kRuleSsd && a.skip) ? a.skip[head] : 0.f;
  const bool divided = RULE == kRuleGated && a.floor;
  const int columns = divided ? a.v_dim : a.value_dim;
  float* out = a.out + (size_t)t0 * a.out_stride + (size_t)head * columns;
  const bool pairs = (columns & 1) == 0 && (a.out_stride & 1) == 0 && ((uintptr_t)a.out & 7) == 0;
  const auto p_at = first_rows(p, rg * 16, lane);
  float odd = 0.f;  // NaN when a sum is not finite
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int unit = cq + 4 * i;
    if (unit >= units) break;
    const auto u_at = second_turned(u, unit * 16, lane);
    Tile acc;
    for (int s = 0; s <= rg; ++s) {  // keys up to the warp's last row
      Fragment x, y;
      p_at.load(x, s);
      u_at.load(y, s);
      acc.add(x, y);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        o[i][n][r] += acc.of(n, r);
        odd += 0.f * o[i][n][r];
        if (divided && unit * 16 + 8 * n + 2 * c + (r & 1) == a.v_dim) d.suf[row0 + 8 * (r >> 1)] = o[i][n][r];  // (done with)
      }
  }
  if (__syncthreads_or(odd != 0.f)) {
    walk_chunk<RULE>(a, d, reinterpret_cast<float*>(chunk_s), blockIdx.y, head, t0, rows);
    return;
  }
  float over[2] = {1.f, 1.f};
  if (divided) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (row0 + 8 * h < rows)
        over[h] = fmaxf(fabsf(d.suf[row0 + 8 * h]), a.floor[(size_t)(t0 + row0 + 8 * h) * a.heads + head]) + 1e-6f;
  }
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int unit = cq + 4 * i;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = row0 + 8 * h, col = unit * 16 + 8 * n + 2 * c;
        if (unit >= units || row >= rows || col >= columns) continue;
        float x = o[i][n][2 * h], y = o[i][n][2 * h + 1];
        if (RULE == kRuleSsd) {
          const float* v = v_rows + (size_t)row * a.v_stride + col;
          x += skip * v[0];
          if (col + 1 < columns) y += skip * v[1];
        }
        if (divided) {
          x /= over[h];
          y /= over[h];
        }
        float* to = out + (size_t)row * a.out_stride + col;
        if (pairs) *reinterpret_cast<float2*>(to) = make_float2(x, y);
        else {
          to[0] = x;
          if (col + 1 < columns) to[1] = y;
        }
      }
  }
}

}  // namespace distie

using namespace distie;

// Floats of scratch that distie_recurrence_chunks takes for `tiles` tiles.
extern "C" long long distie_recurrence_chunks_scratch_floats(int rule, int tiles, int heads, int key_dim, int value_dim) {
  const long long own = rule == kRuleDelta ? kImage + (long long)up16(value_dim) * kChunk : 0;  // (two images of two bytes an element)
  return 2LL * tiles * heads * ((long long)key_dim * value_dim + 4 + own);
}

// The tokens of `q_tiles` ([tiles, 2] int32: first token, rows <= 128; the tiles of a request follow one another) under a
// rule of distie_linear_recurrence, whose arguments these are, except that q and k stay as they are.  scratch: 16-byte
// aligned.  q_scale and floor: gated rule (see ChunkArgs; floor null and q_scale 1 otherwise; with a floor `out` holds the
// divided read-outs, heads * (value_dim - 1) columns).  -2: sizes that the kernels do not take (key_dim up to 128, value_dim up to 144).
extern "C" int distie_recurrence_chunks(int rule, const float* q, int q_stride, const float* k, int k_stride, const float* v,
                                        int v_stride, const float* decay, int decay_stride, const float* write, int write_stride,
                                        int splits, long long split_stride, const float* rate, const float* bias, const float* skip,
                                        float* state, float* out, int out_stride, float* scratch, const int* q_tiles, int tiles,
                                        const int* token_seq, const int* seq_seat, int heads, int groups, int key_dim, int value_dim,
                                        int unit_column, float q_scale, const float* floor, int* error, cudaStream_t stream) {
  if (tiles <= 0) return 0;
  if (!error || heads < 1 || groups < 1 || heads % groups || key_dim < 1 || value_dim < 1 || splits < 1 || !q_tiles || !scratch || !state ||
      rule < kRuleDelta || rule > kRuleGated || (rule == kRuleDelta && !decay) ||
      (rule != kRuleGated && (!rate || !write || unit_column)) || (rule == kRuleGated && !rate && !decay) ||
      (unit_column && value_dim < 2) || (floor && !unit_column))
    return DISTIE_ERR_ARG;
  if (key_dim > 128 || value_dim > 144 || tiles > 32767 || heads > 65535) return DISTIE_ERR_UNSUPPORTED;
  if ((uintptr_t)scratch & 15) return DISTIE_ERR_ARG;
  ChunkArgs a;
  a.q = q; a.k = k; a.v = v;
  a.q_stride = q_stride; a.k_stride = k_stride; a.v_stride = v_stride;
  a.decay = Sliced{decay, decay_stride, splits, split_stride};
  a.write = Sliced{write, write_stride, splits, split_stride};
  a.rate = rate; a.bias = bias; a.skip = skip; a.state = state;
  const long long chunk_heads = 2LL * tiles * heads;
  a.images = reinterpret_cast<__nv_bfloat16*>(scratch);
  a.writes = scratch + (rule == kRuleDelta ? chunk_heads * kImage : 0);
  a.chunks = a.writes + (rule == kRuleDelta ? chunk_heads * up16(value_dim) * kChunk : 0);
  a.whole = a.chunks + chunk_heads * key_dim * value_dim;
  a.out = out; a.out_stride = out_stride;
  a.q_tiles = q_tiles; a.token_seq = token_seq; a.seq_seat = seq_seat;
  a.tiles = tiles; a.heads = heads; a.groups = groups; a.key_dim = key_dim; a.value_dim = value_dim;
  a.v_dim = unit_column ? value_dim - 1 : value_dim;
  a.error = error;
  a.q_scale = q_scale;
  a.floor = floor;
  const dim3 grid(heads, 2 * tiles);
  const bool narrow = value_dim <= 128;
  auto launch = [&](auto kernel, dim3 blocks, int threads, size_t shared) -> int {
    if (shared > 48 * 1024) {
      cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
      if (err != cudaSuccess) return (int)err;
    }
    kernel<<<blocks, threads, shared, stream>>>(a);
    return (int)cudaGetLastError();
  };
#define DISTIE_READ(RULE)                                                                              \
  (narrow ? launch(chunk_read_kernel<RULE, 128>, grid, kWideThreads, read_shared(value_dim))           \
          : launch(chunk_read_kernel<RULE, 192>, grid, kWideThreads, read_shared(value_dim)))
  int status;
  if (rule == kRuleDelta) {
    status = launch(chunk_solve_kernel, grid, kChunkThreads, kSolveShared);
    const dim3 walk(up16(value_dim) / 16, heads, tiles);
    if (status == 0)
      status = up16(key_dim) == 128 ? launch(chunk_walk_kernel<8>, walk, kWalkThreads, kWalkShared)
                                    : launch(chunk_walk_kernel<0>, walk, kWalkThreads, kWalkShared);
    return status != 0 ? status : DISTIE_READ(kRuleDelta);
  }
  const size_t write_shared = KeyTriple::kBytes + (narrow ? Triple<128, kChunk>::kBytes : Triple<192, kChunk>::kBytes);
#define DISTIE_WRITE(RULE)                                                                       \
  (narrow ? launch(chunk_write_kernel<RULE, 128>, grid, kChunkThreads, write_shared)             \
          : launch(chunk_write_kernel<RULE, 192>, grid, kChunkThreads, write_shared))
  status = rule == kRuleSsd ? DISTIE_WRITE(kRuleSsd) : DISTIE_WRITE(kRuleGated);
#undef DISTIE_WRITE
  if (status != 0) return status;
  const int size = key_dim * value_dim;
  const bool fours = (size & 3) == 0 && ((uintptr_t)state & 15) == 0;
  const int width = fours ? 4 : 1;
  const dim3 chain((size / width + kChainThreads - 1) / kChainThreads, heads, tiles);
  status = fours ? launch(chunk_chain_kernel<4>, chain, kChainThreads, 0) : launch(chunk_chain_kernel<1>, chain, kChainThreads, 0);
  if (status != 0) return status;
  return rule == kRuleSsd ? DISTIE_READ(kRuleSsd)
                          : DISTIE_READ(kRuleGated);
#undef DISTIE_READ
}
