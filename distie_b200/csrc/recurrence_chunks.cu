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
// Precision.  The state and everything around it is float32, so the products have to be as good as float32: each operand
// enters the tensor cores (mma.sync.m16n8k16, float32 accumulators) as three bfloat16 parts whose sum is the float32 value,
// in the six products of weight 2^-16 and more.  The largest one (high x high) has accumulators of its own: the tensor
// core truncates when it accumulates, and so truncates 4 or 8 times into a sum at full size instead of 24 or 48 times.
// Decays are products of the g, as in the walk, never differences of logarithms, so a decay of 0 is a 0.
// (A value that is not finite spoils the whole chunk of its request, as it spoils all later tokens in the walk.)
//
// Why chunks: the walk is a chain of about 110 dependent instructions a token and head column, 0.15 to 0.25 us a token
// whatever the machine could do beside it.  Single tokens and short portions stay on it (the rule is in kernels/device.py).
#include "recurrent.cuh"

namespace distie {

constexpr int kWideThreads = 512;   // read: one block an SM, 16 warps
constexpr int kNarrowThreads = 256; // write: two blocks an SM
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
};

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
// row's last three bits, so that the eight rows of an ldmatrix lie in different banks; a row is a multiple of 64 elements.
struct Triple {
  __nv_bfloat16* p;
  int pitch, part;  // elements of a row, of a part
  __device__ __forceinline__ int at(int row, int col) const { return row * pitch + ((((col >> 3) ^ (row & 7)) << 3) | (col & 7)); }
};
// The same with 16 columns: rows lie 48 bytes apart, which keeps an ldmatrix's rows in different banks by itself.
struct NarrowTriple {
  __nv_bfloat16* p;
  int part;
  static constexpr int kPitch = 24;
  __device__ __forceinline__ int at(int row, int col) const { return row * kPitch + col; }
};
template <class M>
__device__ __forceinline__ void put4(const M& m, int row, int col, float4 x) {  // col a multiple of 4
  uint32_t a[3], b[3];
  three_parts(x.x, x.y, a);
  three_parts(x.z, x.w, b);
  __nv_bfloat16* to = m.p + m.at(row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(to + i * m.part) = make_uint2(a[i], b[i]);
}
template <class M>
__device__ __forceinline__ void put2(const M& m, int row, int col, float x, float y) {  // col even
  uint32_t a[3];
  three_parts(x, y, a);
  __nv_bfloat16* to = m.p + m.at(row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(to + i * m.part) = a[i];
}
__host__ __device__ constexpr int value_pitch(int value_dim) { return (value_dim + 63) / 64 * 64; }
__host__ __device__ constexpr size_t triple_bytes(int rows, int pitch) { return (size_t)3 * rows * pitch * 2; }
__device__ __forceinline__ Triple triple_at(unsigned char*& at, int rows, int pitch) {
  Triple t{reinterpret_cast<__nv_bfloat16*>(at), pitch, rows * pitch};
  at += triple_bytes(rows, pitch);
  return t;
}

// Fragments of m16n8k16 in three parts.  rows: stored [m][k] (first operand) or [n][k] (second); turned: [k][m] or [k][n].
// A second operand's fragment covers 16 columns: words 0, 1 are the first eight, 2, 3 the others.
using Fragment = uint32_t[3][4];
template <class M>
__device__ __forceinline__ void first_rows(Fragment& f, const M& m, int row0, int k0, int lane) {
  const __nv_bfloat16* p = m.p + m.at(row0 + (lane & 15), k0 + (lane >> 4) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) load_matrices(f[i], p + i * m.part);
}
template <class M>
__device__ __forceinline__ void first_turned(Fragment& f, const M& m, int row0, int k0, int lane) {
  const __nv_bfloat16* p = m.p + m.at(k0 + (lane & 7) + (lane >> 4) * 8, row0 + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) load_matrices_turned(f[i], p + i * m.part);
}
template <class M>
__device__ __forceinline__ void second_rows(Fragment& f, const M& m, int col0, int k0, int lane) {
  const __nv_bfloat16* p = m.p + m.at(col0 + (lane & 7) + (lane >> 4) * 8, k0 + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) load_matrices(f[i], p + i * m.part);
}
template <class M>
__device__ __forceinline__ void second_turned(Fragment& f, const M& m, int col0, int k0, int lane) {
  const __nv_bfloat16* p = m.p + m.at(k0 + (lane & 15), col0 + (lane >> 4) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) load_matrices_turned(f[i], p + i * m.part);
}

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
struct Decays {
  float g[kChunk], factor[kChunk];
  float pre[kChunk], suf[kChunk];      // within the token's block of 16: the product up to it, and behind it
  float from_start[kChunk], to_end[kChunk];
  float inside[kBlocks][16][17];       // G(i, j) of two tokens of one block
  __device__ __forceinline__ float between(int i, int j) const {  // G(i, j), i >= j
    const int bi = i >> 4, bj = j >> 4;
    if (bi == bj) return inside[bi][i & 15][j & 15];
    float d = suf[j];
    for (int b = bj + 1; b < bi; ++b) d *= pre[16 * b + 15];
    return d * pre[i];
  }
};

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

// N rows of a matrix a warp, four elements a lane (from column 4 lane + offset on): fetched first, stored as parts later, so
// that the loads of several matrices are in flight together.  Row i of warp w is w + i * WARPS; rows from `live` on and
// elements from `dim` on are zeros, except that with `unit` element `dim` of a live row is 1.
template <int N, int WARPS>
struct Rows {
  float4 x[N];
  __device__ __forceinline__ void fetch(const float* src, int stride, int live, int dim, int offset = 0) {
    const int c = 4 * (threadIdx.x & 31) + offset, warp = threadIdx.x >> 5;
    const bool fours = by_fours(src, stride, dim);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      const int r = warp + i * WARPS;
      if (r < live && c < dim) x[i] = four_at(src + (size_t)r * stride, c, dim, fours);
    }
  }
  // From the slices of 16 columns that chunk_walk leaves.
  __device__ __forceinline__ void fetch_slices(const float* src, int padded, int offset = 0) {
    const int c = 4 * (threadIdx.x & 31) + offset, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < padded) x[i] = *reinterpret_cast<const float4*>(src + ((size_t)(c >> 4) * kChunk + warp + i * WARPS) * 16 + (c & 15));
    }
  }
  // Rows of at most 128 elements made unit vectors, times `scale`.
  __device__ __forceinline__ void make_unit(float scale) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float s = scale / sqrtf(warp_sum(x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w) + 1e-6f);
      x[i] = make_float4(x[i].x * s, x[i].y * s, x[i].z * s, x[i].w * s);
    }
  }
  // weight: per row, or null
  __device__ __forceinline__ void store(const Triple& m, int count, int live, int dim, int padded, const float* weight, bool unit,
                                        int offset = 0) {
    const int c = 4 * (threadIdx.x & 31) + offset, warp = threadIdx.x >> 5;
    if (c >= padded) return;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = warp + i * WARPS;
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

// N^T [value_dim, key_dim] of a chunk: rows are value elements (U^T is the first operand), columns key elements.
template <int RULE>
__global__ void __launch_bounds__(kNarrowThreads, 2) chunk_write_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  unsigned char* at = chunk_s;
  const Triple k = triple_at(at, kChunk, kKeyPitch), u = triple_at(at, kChunk, value_pitch(a.value_dim));
  const int group = head / (a.heads / a.groups);
  constexpr int kWarps = kNarrowThreads / 32;
  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  Rows<kChunk / kWarps, kWarps> fetched_k, fetched_u;
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
  if (value_padded > 128) {
    fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, d.factor, unit_column, 128);
  }
  __syncthreads();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int m_tiles = value_padded / 16, n_pairs = (key_padded + 31) / 32, steps = (rows + 15) / 16;
  float* dst = a.chunks + ((size_t)blockIdx.y * a.heads + head) * a.value_dim * a.key_dim;
  const bool pairs = (a.key_dim & 1) == 0;
  for (int unit = warp; unit < m_tiles * n_pairs; unit += kWarps) {  // 16 value by 32 key elements
    const int m0 = unit % m_tiles * 16, n0 = unit / m_tiles * 32;
    const bool both = n0 + 16 < key_padded;
    Tile acc[2];
    for (int s = 0; s < steps; ++s) {
      Fragment x, y;
      first_turned(x, u, m0, 16 * s, lane);
      second_turned(y, k, n0, 16 * s, lane);
      acc[0].add(x, y);
      if (both) {
        second_turned(y, k, n0 + 16, 16 * s, lane);
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
// [1 + A11, 0; A21, 1 + A22] has the inverse [T11, 0; -T22 A21 T11, T22].  m_s: 32 x 33 floats.  512 threads.
constexpr int kSolvePitch = 68;
__device__ __forceinline__ void invert(const float* A, float* T, float* m_s) {
  const int tid = threadIdx.x;
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
  {
    const int r0 = (tid >> 8) * 32, i = (tid >> 4) & 15, l = tid & 15;
    float sum = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) sum += A[(r0 + 16 + i) * kSolvePitch + r0 + m] * T[(r0 + m) * kSolvePitch + r0 + l];
    m_s[tid] = sum;
    __syncthreads();
    sum = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) sum += T[(r0 + 16 + i) * kSolvePitch + r0 + 16 + m] * m_s[(tid & 256) + 16 * m + l];
    T[(r0 + 16 + i) * kSolvePitch + r0 + l] = -sum;
  }
  __syncthreads();
  const int i = tid >> 5, l = tid & 31;
  float sum[2] = {0.f, 0.f};
#pragma unroll 8
  for (int m = 0; m < 32; ++m) {
    const float t = T[m * kSolvePitch + l];
#pragma unroll
    for (int h = 0; h < 2; ++h) sum[h] += A[(32 + i + 16 * h) * kSolvePitch + m] * t;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) m_s[(i + 16 * h) * 33 + l] = sum[h];
  __syncthreads();
  sum[0] = sum[1] = 0.f;
#pragma unroll 8
  for (int m = 0; m < 32; ++m) {
    const float x = m_s[m * 33 + l];
#pragma unroll
    for (int h = 0; h < 2; ++h) sum[h] += T[(32 + i + 16 * h) * kSolvePitch + 32 + m] * x;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) T[(32 + i + 16 * h) * kSolvePitch + l] = -sum[h];
  __syncthreads();
}

// What the delta rule's chunk needs besides the state: T, W and K' (images), U_0.
__global__ void __launch_bounds__(kWideThreads, 1) chunk_solve_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), group = head / (a.heads / a.groups);
  unsigned char* at = chunk_s;
  const Triple k = triple_at(at, kChunk, kKeyPitch), v = triple_at(at, kChunk, value_pitch(a.value_dim));
  const Triple t_keys = triple_at(at, kChunk, kChunk), t_values = triple_at(at, kChunk, kChunk);
  float* A = reinterpret_cast<float*>(at);
  float *T = A + kChunk * kSolvePitch, *m_s = T + kChunk * kSolvePitch;
  const size_t chunk_head = (size_t)blockIdx.y * a.heads + head;
  const Triple w_image{a.images + 2 * chunk_head * kImage, kKeyPitch, kChunk * kKeyPitch};
  const Triple k_image{a.images + (2 * chunk_head + 1) * kImage, kKeyPitch, kChunk * kKeyPitch};
  float* writes = a.writes + chunk_head * value_padded * kChunk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;

  constexpr int kWarps = kWideThreads / 32;
  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  Rows<kChunk / kWarps, kWarps> fetched_k, fetched_v;
  fetched_k.fetch(a.k + (size_t)t0 * a.k_stride + group * a.key_dim, a.k_stride, rows, a.key_dim);
  fetched_v.fetch(v_rows, a.v_stride, rows, a.v_dim);
  for (int i = threadIdx.x; i < 2 * kChunk * kSolvePitch; i += kWideThreads) A[i] = 0.f;
  make_decays(d, a, kRuleDelta, head, t0, rows);
  if (threadIdx.x == 0) a.whole[chunk_head] = d.from_start[kChunk - 1];
  fetched_k.make_unit(1.f);
  fetched_k.store(k, kChunk, rows, a.key_dim, key_padded, nullptr, false);
  fetched_k.store(k_image, kChunk, rows, a.key_dim, key_padded, d.to_end, false);
  fetched_v.store(v, kChunk, rows, a.v_dim, value_padded, nullptr, false);
  if (value_padded > 128) {
    fetched_v.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched_v.store(v, kChunk, rows, a.v_dim, value_padded, nullptr, false, 128);
  }
  __syncthreads();

  if (warp < 10) {  // the blocks of 16 x 16 on and below the diagonal
    const int bi = warp < 1 ? 0 : warp < 3 ? 1 : warp < 6 ? 2 : 3, bj = warp - bi * (bi + 1) / 2;
    Tile acc;
    for (int s = 0; s < key_padded / 16; ++s) {
      Fragment x, y;
      first_rows(x, k, bi * 16, 16 * s, lane);
      second_rows(y, k, bj * 16, 16 * s, lane);
      acc.add(x, y);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = bi * 16 + g + 8 * (r >> 1), j = bj * 16 + 8 * n + 2 * c + (r & 1);
        if (j < i) A[i * kSolvePitch + j] = d.factor[i] * d.between(i, j) * acc.of(n, r);
      }
  }
  __syncthreads();
  invert(A, T, m_s);
  for (int idx = threadIdx.x; idx < kChunk * kChunk / 2; idx += kWideThreads) {
    const int i = idx / (kChunk / 2), j = 2 * (idx % (kChunk / 2));
    const float x = T[i * kSolvePitch + j] * d.factor[j], y = T[i * kSolvePitch + j + 1] * d.factor[j + 1];
    put2(t_values, i, j, x, y);
    put2(t_keys, i, j, x * d.from_start[j], y * d.from_start[j + 1]);
  }
  __syncthreads();

  // Rows of 16 tokens see up to 16 (row + 1) of them: a warp takes an early and a late one.
  for (int unit = warp & 7; unit < value_padded / 16 || unit < key_padded / 16; unit += 8) {
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const int mt = which ? 3 - (warp >> 3) : warp >> 3;
      Tile keys, values;
      for (int s = 0; s <= mt; ++s) {
        Fragment x, y;
        if (unit < key_padded / 16) {
          first_rows(x, t_keys, mt * 16, 16 * s, lane);
          second_turned(y, k, unit * 16, 16 * s, lane);
          keys.add(x, y);
        }
        if (unit < value_padded / 16) {
          first_rows(x, t_values, mt * 16, 16 * s, lane);
          second_turned(y, v, unit * 16, 16 * s, lane);
          values.add(x, y);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = mt * 16 + g + 8 * h, col = 8 * n + 2 * c;
          if (unit < key_padded / 16) put2(w_image, row, unit * 16 + col, keys.of(n, 2 * h), keys.of(n, 2 * h + 1));
          if (unit < value_padded / 16)
            *reinterpret_cast<float2*>(writes + ((size_t)unit * kChunk + row) * 16 + col) =
                make_float2(values.of(n, 2 * h), values.of(n, 2 * h + 1));
        }
    }
  }
}

// The chain of the delta rule: 16 value elements of one head's state, chunk after chunk.  What it reads of a chunk (W, K'
// and its slice of U_0: 100 KB) is copied a chunk ahead.  A block whose tile is not the first of its request has nothing
// to do.
constexpr int kWalkThreads = 256;
constexpr size_t kWalkStage = 2 * (size_t)kImage * 2 + kChunk * 16 * 4;
constexpr size_t kWalkShared = 2 * kWalkStage + triple_bytes(16, kKeyPitch) + (size_t)3 * kChunk * NarrowTriple::kPitch * 2 + 4096;
__device__ __forceinline__ void copy_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__global__ void __launch_bounds__(kWalkThreads, 1) chunk_walk_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  const int slice = blockIdx.x, head = blockIdx.y, tile0 = blockIdx.z, tid = threadIdx.x;
  const int seq = a.token_seq[a.q_tiles[2 * tile0]];
  if (tile0 > 0 && a.token_seq[a.q_tiles[2 * (tile0 - 1)]] == seq) return;
  unsigned char* at = chunk_s + 2 * kWalkStage;
  const Triple S_s = triple_at(at, 16, kKeyPitch);
  const NarrowTriple u_s{reinterpret_cast<__nv_bfloat16*>(at), kChunk * NarrowTriple::kPitch};
  float4* half_s = reinterpret_cast<float4*>(at + (size_t)3 * kChunk * NarrowTriple::kPitch * 2);  // [2][4][32]
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), steps = key_padded / 16;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  const int mt = warp & 3, kh = warp >> 2;  // first product: 16 tokens, every other step over the keys

  auto copy_chunk = [&](int chunk, int stage) {
    unsigned char* to = chunk_s + stage * kWalkStage;
    const size_t chunk_head = (size_t)chunk * a.heads + head;
    const unsigned char* from = reinterpret_cast<const unsigned char*>(a.images + 2 * chunk_head * kImage);
#pragma unroll 8
    for (int i = 0; i < 2 * kImage * 2 / 16 / kWalkThreads; ++i) copy_16(to + 16 * (i * kWalkThreads + tid), from + 16 * (i * kWalkThreads + tid));
    const float* u0 = a.writes + (chunk_head * value_padded + (size_t)slice * 16) * kChunk;
    copy_16(to + 2 * (size_t)kImage * 2 + 16 * tid, u0 + 4 * tid);
    cp_async_commit();
  };
  auto next_chunk = [&](int chunk) {  // -1: the request ends
    if (!(chunk & 1) && a.q_tiles[chunk + 1] > kChunk) return chunk + 1;
    const int tile = (chunk >> 1) + 1;
    return tile < a.tiles && a.token_seq[a.q_tiles[2 * tile]] == seq ? 2 * tile : -1;
  };

  copy_chunk(2 * tile0, 0);
  // the warp's part of S^T: 16 values by 16 keys from 16 warp on
  float S[2][4];
  const size_t size = (size_t)a.value_dim * a.key_dim;
  float* slot = a.state + ((size_t)a.seq_seat[seq] * a.heads + head) * size;
  const bool pairs = (a.key_dim & 1) == 0;
  const int col0 = warp * 16 + 2 * c, row0 = slice * 16 + g;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = row0 + 8 * (r >> 1), col = col0 + 8 * n + (r & 1);
      S[n][r] = row < a.value_dim && col < a.key_dim ? slot[(size_t)row * a.key_dim + col] : 0.f;
    }
  auto store_state = [&](float* to) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = row0 + 8 * h, col = col0 + 8 * n;
        if (row >= a.value_dim || col >= a.key_dim) continue;
        float* p = to + (size_t)row * a.key_dim + col;
        if (pairs) *reinterpret_cast<float2*>(p) = make_float2(S[n][2 * h], S[n][2 * h + 1]);
        else {
          p[0] = S[n][2 * h];
          if (col + 1 < a.key_dim) p[1] = S[n][2 * h + 1];
        }
      }
  };
  auto share_state = [&]() {
    if (warp * 16 < key_padded) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) put2(S_s, g + 8 * h, col0 + 8 * n, S[n][2 * h], S[n][2 * h + 1]);
    }
  };
  share_state();

  int stage = 0;
  for (int chunk = 2 * tile0; chunk >= 0; stage ^= 1) {
    const int next = next_chunk(chunk);
    const size_t chunk_head = (size_t)chunk * a.heads + head;
    const float whole = a.whole[chunk_head];
    if (next >= 0) {  // (the stage's last readers passed a barrier behind their last product)
      copy_chunk(next, stage ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    unsigned char* base = chunk_s + stage * kWalkStage;
    const Triple w{reinterpret_cast<__nv_bfloat16*>(base), kKeyPitch, kChunk * kKeyPitch};
    const Triple k{reinterpret_cast<__nv_bfloat16*>(base) + kImage, kKeyPitch, kChunk * kKeyPitch};
    const float* u0 = reinterpret_cast<const float*>(base + 2 * (size_t)kImage * 2);
    store_state(a.chunks + chunk_head * size);

    Tile sum;
    for (int s = kh; s < steps; s += 2) {
      Fragment x, y;
      first_rows(x, w, mt * 16, 16 * s, lane);
      second_rows(y, S_s, 0, 16 * s, lane);
      sum.add(x, y);
    }
    // each half of the warps finishes eight columns: the other eight go to its partner
    half_s[((kh ^ 1) * 4 + mt) * 32 + lane] = kh ? make_float4(sum.of(0, 0), sum.of(0, 1), sum.of(0, 2), sum.of(0, 3))
                                                : make_float4(sum.of(1, 0), sum.of(1, 1), sum.of(1, 2), sum.of(1, 3));
    __syncthreads();
    {
      const float4 other = half_s[(kh * 4 + mt) * 32 + lane];
      const int row = mt * 16 + g, col = 8 * kh + 2 * c;
      float* out = a.writes + (chunk_head * value_padded + (size_t)slice * 16) * kChunk;
      const float2 p = *reinterpret_cast<const float2*>(u0 + row * 16 + col), q = *reinterpret_cast<const float2*>(u0 + (row + 8) * 16 + col);
      const float2 x = make_float2(p.x - (kh ? sum.of(1, 0) : sum.of(0, 0)) - other.x, p.y - (kh ? sum.of(1, 1) : sum.of(0, 1)) - other.y);
      const float2 y = make_float2(q.x - (kh ? sum.of(1, 2) : sum.of(0, 2)) - other.z, q.y - (kh ? sum.of(1, 3) : sum.of(0, 3)) - other.w);
      put2(u_s, row, col, x.x, x.y);
      put2(u_s, row + 8, col, y.x, y.y);
      *reinterpret_cast<float2*>(out + row * 16 + col) = x;
      *reinterpret_cast<float2*>(out + (row + 8) * 16 + col) = y;
    }
    __syncthreads();
    if (warp * 16 < key_padded) {
      Tile moved;
#pragma unroll
      for (int s = 0; s < kChunk / 16; ++s) {
        Fragment x, y;
        first_turned(x, u_s, 0, 16 * s, lane);
        second_turned(y, k, warp * 16, 16 * s, lane);
        moved.add(x, y);
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) S[n][r] = fmaf(whole, S[n][r], moved.of(n, r));
    }
    share_state();  // (every warp has read the old one: two barriers ago)
    chunk = next;
    if (chunk >= 0) __syncthreads();  // this stage's copies may be overwritten from here on
  }
  store_state(slot);
}

// O of a chunk from its own tokens and the state before it.
template <int RULE>
__global__ void __launch_bounds__(kWideThreads, 1) chunk_read_kernel(ChunkArgs a) {
  extern __shared__ __align__(128) unsigned char chunk_s[];
  __shared__ Decays d;
  int t0;
  const int head = blockIdx.x, rows = chunk_rows(a.q_tiles, blockIdx.y, t0);
  if (rows <= 0) return;
  const int key_padded = up16(a.key_dim), value_padded = up16(a.value_dim), group = head / (a.heads / a.groups);
  unsigned char* at = chunk_s;
  const Triple q = triple_at(at, kChunk, kKeyPitch);
  unsigned char *behind_q = at;
  const Triple k = triple_at(at, kChunk, kKeyPitch);
  unsigned char *behind_k = at;
  const Triple S = triple_at(at, value_padded, kKeyPitch);
  // once the products with K and S are made, the scores and U lie in their place
  const Triple p = triple_at(behind_q, kChunk, kChunk), u = triple_at(behind_k, kChunk, value_pitch(a.value_dim));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  // 16 rows of the chunk; a quarter of the columns.  Later rows see more keys: each scheduler gets warps of all four.
  const int cq = warp >> 2, rg = (warp + cq) & 3;
  const int row0 = rg * 16 + g;

  constexpr int kWarps = kWideThreads / 32;
  const float* v_rows = a.v + (size_t)t0 * a.v_stride + (size_t)head * a.v_dim;
  const bool unit_column = a.v_dim < a.value_dim;
  Rows<kChunk / kWarps, kWarps> fetched_q, fetched_k, fetched_u;
  {
    Rows<9, kWarps> fetched_S;
    fetched_q.fetch(a.q + (size_t)t0 * a.q_stride + group * a.key_dim, a.q_stride, rows, a.key_dim);
    fetched_k.fetch(a.k + (size_t)t0 * a.k_stride + group * a.key_dim, a.k_stride, rows, a.key_dim);
    fetched_S.fetch(a.chunks + ((size_t)blockIdx.y * a.heads + head) * a.value_dim * a.key_dim, a.key_dim, a.value_dim, a.key_dim);
    if (RULE == kRuleDelta) {
      fetched_q.make_unit(rsqrtf((float)a.key_dim));
      fetched_k.make_unit(1.f);
    }
    fetched_q.store(q, kChunk, rows, a.key_dim, key_padded, nullptr, false);
    fetched_k.store(k, kChunk, rows, a.key_dim, key_padded, nullptr, false);
    fetched_S.store(S, value_padded, a.value_dim, a.key_dim, key_padded, nullptr, false);
  }
  make_decays(d, a, RULE, head, t0, rows);

  const int steps = key_padded / 16, units = value_padded / 16;  // 16 values a unit
  constexpr int kUnits = 3;                                       // at most, a warp
  float o[kUnits][2][4];
  Tile score;
  if (cq <= rg) {  // the warp's keys are not all behind its rows
    for (int s = 0; s < steps; ++s) {
      Fragment x, y;
      first_rows(x, q, rg * 16, 16 * s, lane);
      second_rows(y, k, cq * 16, 16 * s, lane);
      score.add(x, y);
    }
  }
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int unit = cq + 4 * i;
    if (unit < units) {
      Tile acc;
      for (int s = 0; s < steps; ++s) {
        Fragment x, y;
        first_rows(x, q, rg * 16, 16 * s, lane);
        second_rows(y, S, unit * 16, 16 * s, lane);
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
    for (int h = 0; h < 2; ++h) {
      const int row = row0 + 8 * h, key = cq * 16 + 8 * n + 2 * c;
      put2(p, row, key, key <= row ? score.of(n, 2 * h) * d.between(row, key) : 0.f,
           key + 1 <= row ? score.of(n, 2 * h + 1) * d.between(row, key + 1) : 0.f);
    }
  fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, factor, unit_column);
  if (value_padded > 128) {
    if (RULE == kRuleDelta) fetched_u.fetch_slices(writes, value_padded, 128);
    else fetched_u.fetch(v_rows, a.v_stride, rows, a.v_dim, 128);
    fetched_u.store(u, kChunk, rows, a.v_dim, value_padded, factor, unit_column, 128);
  }
  __syncthreads();

  const float skip = (RULE == kRuleSsd && a.skip) ? a.skip[head] : 0.f;
  float* out = a.out + (size_t)t0 * a.out_stride + (size_t)head * a.value_dim;
  const bool pairs = (a.value_dim & 1) == 0 && (a.out_stride & 1) == 0 && ((uintptr_t)a.out & 7) == 0;
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int unit = cq + 4 * i;
    if (unit >= units) break;
    Tile acc;
    for (int s = 0; s <= rg; ++s) {  // keys up to the warp's last row
      Fragment x, y;
      first_rows(x, p, rg * 16, 16 * s, lane);
      second_turned(y, u, unit * 16, 16 * s, lane);
      acc.add(x, y);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = row0 + 8 * h, col = unit * 16 + 8 * n + 2 * c;
        if (row >= rows || col >= a.value_dim) continue;
        float x = o[i][n][2 * h] + acc.of(n, 2 * h), y = o[i][n][2 * h + 1] + acc.of(n, 2 * h + 1);
        if (RULE == kRuleSsd) {
          const float* v = a.v + (size_t)(t0 + row) * a.v_stride + (size_t)head * a.v_dim + col;
          x += skip * v[0];
          if (col + 1 < a.value_dim) y += skip * v[1];
        }
        float* to = out + (size_t)row * a.out_stride + col;
        if (pairs) *reinterpret_cast<float2*>(to) = make_float2(x, y);
        else {
          to[0] = x;
          if (col + 1 < a.value_dim) to[1] = y;
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
// aligned.  -2: sizes that the kernels do not take (key_dim up to 128, value_dim up to 144).
extern "C" int distie_recurrence_chunks(int rule, const float* q, int q_stride, const float* k, int k_stride, const float* v,
                                        int v_stride, const float* decay, int decay_stride, const float* write, int write_stride,
                                        int splits, long long split_stride, const float* rate, const float* bias, const float* skip,
                                        float* state, float* out, int out_stride, float* scratch, const int* q_tiles, int tiles,
                                        const int* token_seq, const int* seq_seat, int heads, int groups, int key_dim, int value_dim,
                                        int unit_column, cudaStream_t stream) {
  if (tiles <= 0) return 0;
  if (heads < 1 || groups < 1 || heads % groups || key_dim < 1 || value_dim < 1 || splits < 1 || !q_tiles || !scratch || !state ||
      rule < kRuleDelta || rule > kRuleGated || (rule == kRuleDelta && !decay) ||
      (rule != kRuleGated && (!rate || !write || unit_column)) || (rule == kRuleGated && !rate && !decay) ||
      (unit_column && value_dim < 2))
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
  const dim3 grid(heads, 2 * tiles);
  const size_t key_bytes = triple_bytes(kChunk, kKeyPitch), value_bytes = triple_bytes(kChunk, value_pitch(value_dim));
  const size_t state_bytes = triple_bytes(up16(value_dim), kKeyPitch);
  auto launch = [&](auto kernel, dim3 blocks, int threads, size_t shared) -> int {
    if (shared > 48 * 1024) {
      cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
      if (err != cudaSuccess) return (int)err;
    }
    kernel<<<blocks, threads, shared, stream>>>(a);
    return (int)cudaGetLastError();
  };
  // in chunk_read the scores lie where K was, U where S was: each is taken at the larger of the two
  const size_t read_shared = 2 * key_bytes + (state_bytes > value_bytes ? state_bytes : value_bytes);
  int status;
  if (rule == kRuleDelta) {
    const size_t solve_shared = key_bytes + value_bytes + 2 * triple_bytes(kChunk, kChunk) + (2 * kChunk * kSolvePitch + 32 * 33) * sizeof(float);
    status = launch(chunk_solve_kernel, grid, kWideThreads, solve_shared);
    if (status == 0) status = launch(chunk_walk_kernel, dim3(up16(value_dim) / 16, heads, tiles), kWalkThreads, kWalkShared);
    return status != 0 ? status : launch(chunk_read_kernel<kRuleDelta>, grid, kWideThreads, read_shared);
  }
  const size_t write_shared = key_bytes + value_bytes;
  status = rule == kRuleSsd ? launch(chunk_write_kernel<kRuleSsd>, grid, kNarrowThreads, write_shared)
                            : launch(chunk_write_kernel<kRuleGated>, grid, kNarrowThreads, write_shared);
  if (status != 0) return status;
  const int size = key_dim * value_dim;
  const bool fours = (size & 3) == 0 && ((uintptr_t)state & 15) == 0;
  const int width = fours ? 4 : 1;
  const dim3 chain((size / width + kChainThreads - 1) / kChainThreads, heads, tiles);
  status = fours ? launch(chunk_chain_kernel<4>, chain, kChainThreads, 0) : launch(chunk_chain_kernel<1>, chain, kChainThreads, 0);
  if (status != 0) return status;
  return rule == kRuleSsd ? launch(chunk_read_kernel<kRuleSsd>, grid, kWideThreads, read_shared)
                          : launch(chunk_read_kernel<kRuleGated>, grid, kWideThreads, read_shared);
}
