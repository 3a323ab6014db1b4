// What the kernels of layers with a state per request share: elementwise functions, matrices that may still be the
// slices of a split product, asynchronous copies into shared memory, and the pieces of recurrences taken in chunks.
#pragma once

#include "common.cuh"

namespace distie {

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return log1pf(expf(-fabsf(z))) + fmaxf(z, 0.f); }
__device__ __forceinline__ float gate_f(int sigmoid, float z) { return sigmoid ? sigmoid_f(z) : silu_f(z); }

// A float32 matrix that may still be the slices of a split product: `splits` matrices `split_stride` floats apart
// whose sum it is (splits == 1: the matrix itself).  Loads add the slices up, in their order.
struct Sliced {
  const float* p;
  int stride;  // of a row
  int splits;
  long long split_stride;
  const float* bias = nullptr;  // per column, added to the sum of the slices (a projection's bias); null: none
  __device__ __forceinline__ float at(size_t row, int col) const {
    const float* q = p + row * stride + col;
    float v = q[0];
    for (int s = 1; s < splits; ++s) v += q[(size_t)s * split_stride];
    return bias ? v + bias[col] : v;
  }
  __device__ __forceinline__ float4 at4(size_t row, int col) const {
    const float* q = p + row * stride + col;
    float4 v = *reinterpret_cast<const float4*>(q);
    for (int s = 1; s < splits; ++s) {
      const float4 w = *reinterpret_cast<const float4*>(q + (size_t)s * split_stride);
      v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    if (bias) {
      const float4 b = *reinterpret_cast<const float4*>(bias + col);
      v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    return v;
  }
};

__device__ __forceinline__ void cp_async_f4(float* dst, const float* src, bool live) {
  const int bytes = live ? 16 : 0;  // zero-fills when not live
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_f1(float* dst, const float* src, bool live) {
  const int bytes = live ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// -- recurrences in chunks of a step's tiles ---------------------------------------------------------------------
constexpr int kChunk = 64;  // tokens; a chunk starts where a tile of the step (at most 128 tokens of one request) or its second half starts

__host__ __device__ constexpr int up16(int n) { return (n + 15) & ~15; }

// Where chunk `chunk` of the step lies: its first token and its number of tokens (0: the second half of a short tile).
__device__ __forceinline__ int chunk_rows(const int* q_tiles, int chunk, int& t0) {
  const int tile = chunk >> 1, half = chunk & 1;
  t0 = q_tiles[2 * tile] + half * kChunk;
  return min(kChunk, q_tiles[2 * tile + 1] - half * kChunk);
}

// D[16 x 8] += A[16 x 16] B[16 x 8]; with g = lane / 4, c = lane % 4: d = D[g][2c], D[g][2c+1], D[g+8][2c], D[g+8][2c+1].
__device__ __forceinline__ void mma_16bit(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void load_matrices_turned(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

}  // namespace distie
