// Float32 attention of prompt portions over the paged cache, a tile of 32 tokens and one head a block.
//
// The size-agnostic kernel (attention_generic.cu) takes a token and a head a block: every key and value is read for every
// token, and a key costs a warp a sum across its lanes.  Here a block keeps 32 queries in shared memory, takes the keys 64
// at a time and holds 4 x 4 scores and 4 x D/16 outputs a thread: eight reads of 16 bytes feed 64 multiply-adds of the
// scores, twelve (D = 128) feed 128 of the outputs.  The FMA pipe (74 TFLOP/s) is the ceiling, of which 38 % is reached (28 TFLOP/s
// of the visible half, 1,100 tokens); the reads of shared memory take 70 % of the pipe's time beside it, and the rest goes
// to four barriers a block of keys, the softmax between the two products and the hidden half of diagonal blocks.  The keys of
// the next block are copied while this one's values are multiplied, and the other way round (cp.async).  Tiles of 32 rows
// and not 64 or 128: prompts of a few hundred tokens would not fill the machine, and a causal tile's time grows with its
// last position.  Layer of two prompts of 339 and 438 tokens, 12 heads of 128: 449 -> 61 us; 1,100 tokens, 28 heads:
// 3,567 -> 308 us.  Which portions are worth a tile: tiles_pay in kernels/device.py.
//
// Arithmetic is the size-agnostic kernel's: float32 products and sums, scores scaled (and capped) after the product,
// accurate exponentials, the same visible keys (window, chunk, keep_first), the sink in the denominator, and a key whose
// page the block table does not hold is reported and skipped.  Sizes: multiples of four up to 128.
//
// A value that is not finite reaches the tokens that see it and no others: a tile whose sums are not all finite is gone
// through once more without the products of the keys that a row does not see (the check of the sums: nothing that shows).
#include <type_traits>

#include "common.cuh"

namespace distie {

constexpr int kTileRows = 32, kTileKeys = 64, kTileThreads = 128;

struct TileAttention {
  const float* q;
  int q_stride;
  float* out;
  int out_stride;
  const int *q_tiles, *positions, *token_seq, *seq_seat, *block_table;
  int table_width;
  const float *k, *v;
  int group, kv_heads, head_dim, value_dim, page_size, num_pages, window, chunk, keep_first;
  float scale, softcap;
  const float* sink;
  int* error;
};

template <int D>
struct TileShared {
  static constexpr int kKeyPitch = D + 4;  // rows four banks apart: eight rows of one column are a whole wavefront
  float q[kTileRows][kKeyPitch];
  float k[kTileKeys][kKeyPitch];
  float v[kTileKeys][D];
  float p[kTileRows][kTileKeys + 4];
  long long row[2][kTileKeys];  // of a key block, by parity: the row of each key in its head's cache, -1: none
};

__device__ __forceinline__ void copy_float4(float* dst, const float* src, bool live) {  // zeros when not live
  const int bytes = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// D: the larger of head_dim and value_dim rounded up to 32, 64 or 128.
template <int D>
__global__ void __launch_bounds__(kTileThreads, 2) attention_tiles_kernel(TileAttention a) {
  extern __shared__ __align__(16) unsigned char tile_smem[];
  TileShared<D>& sm = *reinterpret_cast<TileShared<D>*>(tile_smem);
  constexpr int kCols = D / 16;  // output columns a thread: four (two) neighbours, every 64 (32)
  constexpr int kVec = kCols < 4 ? kCols : 4;
  const int tid = threadIdx.x, rg = tid >> 4, c = tid & 15;
  const int head = blockIdx.x, kv_head = head / a.group;
  const int piece = gridDim.y - 1 - blockIdx.y;  // late tiles see the most keys: first
  const int tile = piece >> 2, skip = (piece & 3) * kTileRows;
  const int rows = min(kTileRows, a.q_tiles[2 * tile + 1] - skip);
  if (rows <= 0) return;
  const int t0 = a.q_tiles[2 * tile] + skip;
  const int pos0 = a.positions[t0], pos1 = pos0 + rows - 1;  // consecutive tokens of one request
  const int* table = a.block_table + (size_t)a.seq_seat[a.token_seq[t0]] * a.table_width;
  const int first0 = first_visible_key(pos0, a.window, a.chunk);
  const int kept = min(a.keep_first, first0);
  // key blocks: those of the keys kept for good, then those from the first row's oldest key on
  const int kept_blocks = (kept + kTileKeys - 1) / kTileKeys;
  const int main0 = max(kept_blocks, first0 / kTileKeys), blocks = kept_blocks + pos1 / kTileKeys - main0 + 1;
  auto block_start = [&](int b) { return (b < kept_blocks ? b : main0 + b - kept_blocks) * kTileKeys; };

  auto find_rows = [&](int b) {  // where the keys of block b lie
    if (tid < kTileKeys) {
      const int key = block_start(b) + tid;
      long long row = -1;
      if (key <= pos1 && (key >= first0 || key < kept)) {
        const int column = key / a.page_size;
        const int page = column < a.table_width ? table[column] : -1;
        if (page >= 0 && page < a.num_pages) row = ((long long)page * a.kv_heads + kv_head) * a.page_size + key % a.page_size;
        else if (a.error) atomicExch(a.error, 3);  // a table that does not cover the keys: report, skip
      }
      sm.row[b & 1][tid] = row;
    }
  };
  constexpr int kRowCopies = D / 4;  // of 16 bytes
  auto copy_block = [&](int b, const float* src, int dim, float* dst, int pitch) {
#pragma unroll
    for (int i = 0; i < kTileKeys * kRowCopies / kTileThreads; ++i) {
      const int idx = i * kTileThreads + tid, r = idx / kRowCopies, e = idx % kRowCopies * 4;
      const long long row = sm.row[b & 1][r];
      const bool live = row >= 0 && e < dim;
      copy_float4(dst + r * pitch + e, src + (live ? row * dim + e : 0), live);
    }
    copies_commit();
  };

#pragma unroll
  for (int i = 0; i < kTileRows * kRowCopies / kTileThreads; ++i) {
    const int idx = i * kTileThreads + tid, r = idx / kRowCopies, e = idx % kRowCopies * 4;
    const bool live = r < rows && e < a.head_dim;
    copy_float4(&sm.q[r][e], a.q + (live ? (size_t)(t0 + r) * a.q_stride + (size_t)head * a.head_dim + e : 0), live);
  }
  float o[4][kCols], m[4], l[4];
  int first[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) first[i] = first_visible_key(pos0 + rg * 4 + i, a.window, a.chunk);
  // All keys of the tile.  A key that a row does not see has weight 0 there, and 0 times a value that is not finite is NaN:
  // CAREFUL marks such weights as -0 and leaves the products out.
  auto walk_keys = [&](auto careful) {
    constexpr bool CAREFUL = decltype(careful)::value;
    find_rows(0);
    __syncthreads();
    copy_block(0, a.k, a.head_dim, sm.k[0], TileShared<D>::kKeyPitch);  // (and the queries)
    copy_block(0, a.v, a.value_dim, sm.v[0], D);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
#pragma unroll
      for (int e = 0; e < kCols; ++e) o[i][e] = 0.f;
    }
    for (int b = 0; b < blocks; ++b) {
      const bool more = b + 1 < blocks;
      if (more) find_rows(b + 1);
      copies_wait<1>();  // K is here (and the queries); V may be on its way
      __syncthreads();
      float s[4][4] = {};
#pragma unroll 4
      for (int e = 0; e < D; e += 4) {
        float4 q[4], k[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(&sm.q[rg * 4 + i][e]);
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(&sm.k[c + 16 * j][e]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            s[i][j] = fmaf(q[i].x, k[j].x, s[i][j]);
            s[i][j] = fmaf(q[i].y, k[j].y, s[i][j]);
            s[i][j] = fmaf(q[i].z, k[j].z, s[i][j]);
            s[i][j] = fmaf(q[i].w, k[j].w, s[i][j]);
          }
      }
      const int start = block_start(b);
      bool live[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) live[j] = sm.row[b & 1][c + 16 * j] >= 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pos = pos0 + rg * 4 + i;
        float top = m[i];
        bool hidden[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = start + c + 16 * j;
          const bool seen = live[j] && key <= pos && (key >= first[i] || key < a.keep_first);
          hidden[j] = !seen;
          s[i][j] = seen ? cap_score(s[i][j] * a.scale, a.softcap) : -INFINITY;  // scaled after the product
          top = fmaxf(top, s[i][j]);
        }
#pragma unroll
        for (int offset = 8; offset > 0; offset >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
        const float base = top == -INFINITY ? 0.f : top;  // nothing seen yet: every exponential is 0
        const float corr = expf(m[i] - base);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = expf(s[i][j] - base);
          sm.p[rg * 4 + i][c + 16 * j] = CAREFUL && hidden[j] ? -0.f : p;
          sum += p;
        }
        l[i] = l[i] * corr + sum;  // of this thread's keys: summed over the row's threads at the end
        m[i] = top;
#pragma unroll
        for (int e = 0; e < kCols; ++e) o[i][e] *= corr;
      }
      __syncthreads();  // K is done with
      if (more) {
        copy_block(b + 1, a.k, a.head_dim, sm.k[0], TileShared<D>::kKeyPitch);
        copies_wait<1>();
      } else {
        copies_wait<0>();
      }
      __syncthreads();  // V is here
#pragma unroll 4
      for (int j = 0; j < kTileKeys; j += 4) {
        float4 p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(&sm.p[rg * 4 + i][j]);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float v[kCols];
#pragma unroll
          for (int e = 0; e < kCols; e += kVec) {
            const float* src = &sm.v[j + jj][kVec * c + 16 * e];
            if (kVec == 4) {
              const float4 x = *reinterpret_cast<const float4*>(src);
              v[e] = x.x; v[e + 1] = x.y; v[e + (kVec > 2 ? 2 : 0)] = x.z; v[e + (kVec > 3 ? 3 : 0)] = x.w;
            } else {
              const float2 x = *reinterpret_cast<const float2*>(src);
              v[e] = x.x; v[e + 1] = x.y;
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float w = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
            if (CAREFUL && __float_as_uint(w) == 0x80000000u) continue;
#pragma unroll
            for (int e = 0; e < kCols; ++e) o[i][e] = fmaf(w, v[e], o[i][e]);
          }
        }
      }
      __syncthreads();
      if (more) copy_block(b + 1, a.v, a.value_dim, sm.v[0], D);
    }
  };
  walk_keys(std::false_type{});
  float odd = 0.f;  // NaN when a sum is not finite: then once more, row by row only what it sees
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < kCols; ++e) odd += 0.f * o[i][e];
  if (__syncthreads_or(odd != 0.f)) walk_keys(std::true_type{});
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int offset = 8; offset > 0; offset >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], offset);
    const int r = rg * 4 + i;
    if (r >= rows) continue;
    const float inv = a.sink ? sink_inverse(m[i], l[i], a.sink[head]) : (l[i] > 0.f ? 1.f / l[i] : 0.f);
    float* to = a.out + (size_t)(t0 + r) * a.out_stride + (size_t)head * a.value_dim;
#pragma unroll
    for (int e = 0; e < kCols; ++e) {
      const int col = kVec * c + 16 * (e / kVec * kVec) + e % kVec;
      if (col < a.value_dim) to[col] = o[i][e] * inv;
    }
  }
}

}  // namespace distie

using namespace distie;

// The tokens of `q_tiles` ([tiles, 2] int32: first token, rows <= 128, consecutive tokens of one request).
// -2: sizes, strides or addresses that the kernel does not take.
extern "C" int distie_attention_tiles(const float* q, int q_stride, float* out, int out_stride, const int* q_tiles, int tiles,
                                      const int* positions, const int* token_seq, const int* seq_seat, const int* block_table,
                                      int table_width, const float* k_cache, const float* v_cache, int num_heads, int num_kv_heads,
                                      int head_dim, int value_dim, int page_size, int num_pages, int window, int chunk,
                                      int keep_first, float scale, float softcap, const float* sink, int* error,
                                      cudaStream_t stream) {
  if (tiles <= 0) return 0;
  if (num_heads < 1 || num_kv_heads < 1 || num_heads % num_kv_heads || head_dim < 1 || value_dim < 1 || keep_first < 0 ||
      page_size < 1 || table_width < 1 || !q_tiles)
    return DISTIE_ERR_ARG;
  const int most = head_dim > value_dim ? head_dim : value_dim;
  if (most > 128 || ((head_dim | value_dim | q_stride) & 3) || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) ||
      tiles > 16383)
    return DISTIE_ERR_UNSUPPORTED;
  TileAttention a{q, q_stride, out, out_stride, q_tiles, positions, token_seq, seq_seat, block_table, table_width, k_cache,
                  v_cache, num_heads / num_kv_heads, num_kv_heads, head_dim, value_dim, page_size, num_pages, window, chunk,
                  keep_first, scale, softcap, sink, error};
  auto launch = [&](auto kernel, size_t shared) -> int {
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (err != cudaSuccess) return (int)err;
    kernel<<<dim3(num_heads, 4 * tiles), kTileThreads, shared, stream>>>(a);
    return (int)cudaGetLastError();
  };
  if (most <= 32) return launch(attention_tiles_kernel<32>, sizeof(TileShared<32>));
  if (most <= 64) return launch(attention_tiles_kernel<64>, sizeof(TileShared<64>));
  return launch(attention_tiles_kernel<128>, sizeof(TileShared<128>));
}
