// Float32 products of many rows on the 5th-generation tensor cores: out[M, N] = x[M, K] w[N, K]^T (+ bias), float32 in and out.
//
// A float32 number is the sum of three bfloat16 numbers (8 bits each of its 24): x = h + m + l, each the rounded rest of the
// ones before.  Of the nine products of two such sums the six largest are taken, h h, h m, m h, m m, h l, l h; what is left out
// is 2^-26 of a term.  Two kernels: split_planes_kernel writes the three planes of x and of w, gemm_float32_kernel multiplies.
//
// What bounds it: six MMAs where bfloat16 has one, 270 TFLOP/s at the measured peak (74 with FMA), and 96 KB from L2 for every
// 128 x 128 x 64 of them, about 39 bytes a clock and SM: 2,460 cycles against 1,536 of MMAs.  777 x 2,048 x 1,536: 39 us (125
// TFLOP/s), the planes 8 of them, where the library's FMA product takes 112; 2,048 x 18,944 x 3,584 1,570 against 4,322.  Relative
// error against 64 bits 1.4e-7 (K 1,536) and 1.9e-7 (K 8,960), of the library's 7.0e-7 and 1.7e-6.  The tensor core truncates when
// it adds to an accumulator, so accumulators live for 128 of K only, h h in one of its own (eight additions); they are
// double-buffered, and the epilogue warps add them up in registers, rounding to nearest, while the next ones fill.
//
//   warp 0      producer: TMA loads of a stage (three 128 x 64 tiles of x and three of w, 128-byte swizzle), two stages
//   warp 1      allocates tensor memory; one lane issues the MMAs
//   warps 2..9  sums: two warps per quarter of the rows, 64 columns each; at the end bias and stores
//
//   tensor memory   two buffers of [h h: 128 columns | the other five: 128 columns]
//
// bfloat16 numbers end at 2^-133, where the third plane of a number below 2^-110 would lie, and products of large ones overflow
// before their sum need do: a row whose largest number lies outside 2^-40 .. 2^40 is divided by the power of two that
// brings that number into [1, 2), and the outputs are multiplied again.  (What is lost below 2^-110 in other rows is less than 2^-93 of
// their largest number.)  A number that is not finite has itself as h and zeros behind it; infinity times a plane's zero is
// not a number, so where the five other products' sum is not finite, h h alone counts, which is infinite, and not a number,
// exactly where the product of the numbers is.  The search for a row's largest number costs 1 us of the 39 (5 with a whole row in one
// warp's registers); rows that are not finite, whose outputs were once computed again one by one, 5,200 us, cost nothing.  Every wait is bounded: when one runs out the error word becomes 6.
#include "tcgen05.cuh"

namespace distie {

constexpr int kWideTile = 128, kWideK = 64, kWideStages = 2, kWideThreads = 10 * 32;
constexpr int kWidePlane = kWideTile * kWideK * 2;  // bytes of a plane's tile
constexpr int kWideDrain = 2;                       // stages that an accumulator lives
constexpr int kWidePitch = 68;                      // floats of a row of 64 outputs in shared memory
constexpr int kWideHeld = 3;
constexpr float kWideMax = 3.402823466e38f;
constexpr float kWideLeast = 0x1p-133f;             // the smallest bfloat16 number
constexpr float kWideSmall = 0x1p-40f, kWideLarge = 0x1p40f;  // rows whose largest number lies outside are divided by a power of two

struct WideShared {
  alignas(1024) unsigned char a[kWideStages][3][kWidePlane];
  alignas(1024) unsigned char b[kWideStages][3][kWidePlane];
  uint64_t full[kWideStages], empty[kWideStages];
  uint64_t sum_full[2], sum_empty[2];
  uint32_t tmem_base;
  uint32_t failed;
};

// v 2^e, e in [-298, 254] (what lies below 2^-252 of a sum of products of numbers below 2 is zero).
__device__ __forceinline__ float times_power(float v, int e) {
  e = max(e, -252);
  return v * __int_as_float(((e >> 1) + 127) << 23) * __int_as_float((e - (e >> 1) + 127) << 23);
}

// Planes [3][rows][K] of rows of K numbers, and of each row a mark: the power of two that it was divided by, times two, and 1 more
// where a number of it is not finite.  WARPS warps take a row, eight numbers a thread at a time; the first kWideHeld of these
// stay in registers between the search for the largest and the split.
template <int WARPS>
__global__ void __launch_bounds__(256) split_planes_kernel(const float* __restrict__ x, int x_stride, int x_rows, __nv_bfloat16* __restrict__ xp,
                                                           const float* __restrict__ w, int w_rows, __nv_bfloat16* __restrict__ wp,
                                                           int* __restrict__ marks, int K) {
  constexpr int PER_ROW = WARPS * 32, STEP = PER_ROW * 8;
  __shared__ float largest[8];
  __shared__ bool with_odd[8];
  grid_dependency_release();
  const int row = blockIdx.x * (256 / PER_ROW) + threadIdx.x / PER_ROW, col0 = (threadIdx.x % PER_ROW) * 8;
  const int cols = row < x_rows + w_rows ? K : 0;
  const bool of_x = row < x_rows;
  const float* from = of_x ? x + (size_t)row * x_stride : w + (size_t)(row - x_rows) * K;
  float held[kWideHeld][8], most = 0.f;
  bool odd = false;  // a number that is not finite
  auto search = [&](const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool finite = fabsf(v[i]) <= kWideMax;
      most = fmaxf(most, finite ? fabsf(v[i]) : 0.f);
      odd = odd || !finite;
    }
  };
  grid_dependency_wait();
#pragma unroll
  for (int h = 0; h < kWideHeld; ++h)
    if (col0 + h * STEP < cols) load8_cg(from + col0 + h * STEP, held[h]);
#pragma unroll
  for (int h = 0; h < kWideHeld; ++h)
    if (col0 + h * STEP < cols) search(held[h]);
  for (int col = col0 + kWideHeld * STEP; col < cols; col += STEP) {
    float v[8];
    load8_cg(from + col, v);
    search(v);
  }
  most = warp_max(most);
  odd = __any_sync(0xffffffffu, odd);
  if (WARPS > 1) {
    if ((threadIdx.x & 31) == 0) {
      largest[threadIdx.x >> 5] = most;
      with_odd[threadIdx.x >> 5] = odd;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WARPS; ++i) {
      const int of = threadIdx.x / PER_ROW * WARPS + i;
      most = fmaxf(most, largest[of]);
      odd = odd || with_odd[of];
    }
  }
  int e = 0;
  if (most > 0.f && (most < kWideSmall || most >= kWideLarge))
    e = most < 1.17549435e-38f ? (__float_as_int(most * 16777216.f) >> 23) - 127 - 24 : (__float_as_int(most) >> 23) - 127;
  if (cols > 0 && col0 == 0) marks[row] = 2 * e + odd;
  const size_t plane = (size_t)(of_x ? x_rows : w_rows) * K;
  __nv_bfloat16* to = of_x ? xp + (size_t)row * K : wp + (size_t)(row - x_rows) * K;
  auto split = [&](int col, const float (&v)[8]) {
    float h[8], m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool finite = fabsf(v[i]) <= kWideMax;
      const float s = e == 0 ? v[i] : times_power(v[i], -e);
      float top = __bfloat162float(__float2bfloat16_rn(s));
      if (top == 0.f && v[i] != 0.f) top = copysignf(kWideLeast, v[i]);  // (infinity times it is not infinity times zero)
      h[i] = finite ? top : v[i];
      const float rest = finite ? s - top : 0.f;
      m[i] = __bfloat162float(__float2bfloat16_rn(rest));
      l[i] = rest - m[i];
    }
    store8(to + col, h);
    store8(to + col + plane, m);
    store8(to + col + 2 * plane, l);
  };
#pragma unroll
  for (int h = 0; h < kWideHeld; ++h)
    if (col0 + h * STEP < cols) split(col0 + h * STEP, held[h]);
  for (int col = col0 + kWideHeld * STEP; col < cols; col += STEP) {
    float v[8];
    load8_cg(from + col, v);
    split(col, v);
  }
}

__global__ void __launch_bounds__(kWideThreads, 1)
gemm_float32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const int* __restrict__ marks, const float* __restrict__ bias, float* __restrict__ out, int ldo, int M, int N, int K,
                    int* __restrict__ error) {
  extern __shared__ unsigned char raw[];
  auto& sm = *reinterpret_cast<WideShared*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t TMEM_COLS = 512;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kWideTile, n0 = blockIdx.y * kWideTile;
  const int blocks = (K + kWideK - 1) / kWideK, drains = (blocks + kWideDrain - 1) / kWideDrain;
  volatile uint32_t* failed = &sm.failed;
  if (threadIdx.x == 32) {
    prefetch_tensor_map(&map_a);
    prefetch_tensor_map(&map_b);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWideStages; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.sum_full[b], 1);
      mbar_init(&sm.sum_empty[b], 8);  // one arrival per warp
    }
    sm.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;
  grid_dependency_release();
  grid_dependency_wait();

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int issued = 0;
      for (int kb = 0; kb < blocks; ++kb) {
        const int s = kb % kWideStages;
        if (!mbar_wait_unless(&sm.empty[s], ((kb / kWideStages) & 1) ^ 1, failed)) { ok = false; break; }
        mbar_expect_tx(&sm.full[s], 6 * kWidePlane);
        for (int p = 0; p < 3; ++p) {  // (a box past K or past the last plane's rows is filled with zeros and still counted)
          tma_load_2d(sm.a[s][p], &map_a, &sm.full[s], kb * kWideK, p * M + m0);
          tma_load_2d(sm.b[s][p], &map_b, &sm.full[s], kb * kWideK, p * N + n0);
        }
        issued = kb + 1;
      }
      if (!ok) {
        atomicExch(&sm.failed, 1u);
        for (int kb = max(0, issued - kWideStages); kb < issued; ++kb) mbar_wait(&sm.full[kb % kWideStages], (kb / kWideStages) & 1);
      }
    }
  } else if (warp == 1) {
    // The warp walks together and an elected lane issues (see attention_prefill_pairs.cu).
    constexpr uint32_t idesc = instr_desc(kWideTile);
    bool ok = true;
    for (int kb = 0; kb < blocks && ok; ++kb) {
      const int s = kb % kWideStages, drain = kb / kWideDrain, buffer = drain & 1;
      const bool first = kb % kWideDrain == 0, last = kb + 1 == blocks || (kb + 1) % kWideDrain == 0;
      if (first) ok = __all_sync(0xffffffffu, mbar_wait_unless(&sm.sum_empty[buffer], ((drain >> 1) & 1) ^ 1, failed));
      ok = ok && __all_sync(0xffffffffu, mbar_wait_unless(&sm.full[s], (kb / kWideStages) & 1, failed));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t main = tmem + buffer * 256, rest = main + 128;
#pragma unroll
        for (int product = 0; product < 6; ++product) {
          constexpr int OF_A[6] = {2, 0, 1, 1, 0, 0}, OF_B[6] = {0, 2, 1, 0, 1, 0};  // l h, h l, m m, m h, h m, h h
          const uint64_t a_desc = smem_desc(sm.a[s][OF_A[product]]), b_desc = smem_desc(sm.b[s][OF_B[product]]);
#pragma unroll
          for (int k = 0; k < kWideK / 16; ++k)
            umma_bf16(product == 5 ? main : rest, a_desc + 2 * k, b_desc + 2 * k, idesc,
                      (!first || k > 0 || (product > 0 && product < 5)) ? 1u : 0u);
        }
        umma_commit(&sm.empty[s]);
        if (last) umma_commit(&sm.sum_full[buffer]);
      }
      __syncwarp();
    }
    if (!ok) atomicExch(&sm.failed, 1u);
  } else {
    const int quadrant = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)(quadrant * 32) << 16) + half * 64;
    const int row = m0 + quadrant * 32 + lane, col0 = n0 + half * 64;
    // Whether a row or a column of the warp's part was divided by a power of two or holds a number that is not finite.
    int marked = row < M ? __ldcg(marks + row) : 0;
    for (int c = col0 + lane; c < min(col0 + 64, N); c += 32) marked |= __ldcg(marks + M + c);
    const bool special = __any_sync(0xffffffffu, marked != 0);
    float sum[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) sum[i] = 0.f;
    bool ok = true;
    for (int drain = 0; drain < drains; ++drain) {
      const int buffer = drain & 1;
      ok = __all_sync(0xffffffffu, mbar_wait_unless(&sm.sum_full[buffer], (drain >> 1) & 1, failed));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        uint32_t rest[32], main[32];
        tmem_load_32(lane_base + buffer * 256 + 128 + c, rest);
        tmem_load_32(lane_base + buffer * 256 + c, main);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (special) {
#pragma unroll
          for (int i = 0; i < 32; ++i) rest[i] = fabsf(__uint_as_float(rest[i])) <= kWideMax ? rest[i] : 0u;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[c + i] += __uint_as_float(main[i]) + __uint_as_float(rest[i]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.sum_empty[buffer]);
    }
    if (!ok) {
      atomicExch(&sm.failed, 1u);
    } else {
      // Through shared memory (all products are done with it), so that a warp stores whole lines of two rows at a time.
      float* tile = reinterpret_cast<float*>(sm.a) + (warp - 2) * 32 * kWidePitch;
#pragma unroll
      for (int i = 0; i < 64; i += 4)
        *reinterpret_cast<float4*>(tile + lane * kWidePitch + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
      __syncwarp();
      const int col = col0 + (lane & 15) * 4;
      if (col < N) {  // (N is a multiple of 4)
        const float4 add = bias ? make_float4(bias[col], bias[col + 1], bias[col + 2], bias[col + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
        int4 by = make_int4(0, 0, 0, 0);
        if (special) by = make_int4(__ldcg(marks + M + col) >> 1, __ldcg(marks + M + col + 1) >> 1, __ldcg(marks + M + col + 2) >> 1,
                                    __ldcg(marks + M + col + 3) >> 1);
#pragma unroll 4
        for (int r = lane >> 4; r < 32; r += 2) {
          const int to = m0 + quadrant * 32 + r;
          if (to >= M) break;
          float4 v = *reinterpret_cast<const float4*>(tile + r * kWidePitch + (lane & 15) * 4);
          if (special) {
            const int e = __ldcg(marks + to) >> 1;
            v = make_float4(times_power(v.x, e + by.x), times_power(v.y, e + by.y), times_power(v.z, e + by.z), times_power(v.w, e + by.w));
          }
          if (bias) v = make_float4(v.x + add.x, v.y + add.y, v.z + add.z, v.w + add.w);
          *reinterpret_cast<float4*>(out + (size_t)to * ldo + col) = v;
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  if (threadIdx.x == 0 && sm.failed && error) atomicCAS(error, 0, 6);
}

}  // namespace distie

using namespace distie;

// Floats of scratch of the product below: the planes and the powers of two.
extern "C" long long distie_gemm_float32_scratch_floats(int M, int N, int K) {
  return ((long long)M + N) * K * 3 / 2 + M + N;
}

// out[M, N] (row stride ldo) = x[M, K] (row stride x_stride) w[N, K]^T + bias (or null), all float32.  Returns
// DISTIE_ERR_UNSUPPORTED for a K that is no multiple of 8, an N or a row of out that is none of 4, or an address off 16 bytes.
extern "C" int distie_gemm_float32(const float* x, int x_stride, const float* w, const float* bias, float* out, int ldo, int M, int N,
                                   int K, float* scratch, int* error, cudaStream_t stream) {
  if (M < 1 || N < 1 || K < 1 || !scratch) return DISTIE_ERR_ARG;
  if ((K & 7) || (N & 3) || (ldo & 3) || (x_stride & 3) ||
      (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out | (uintptr_t)scratch) & 15) || 3ll * M > 0x7fffffffLL || 3ll * N > 0x7fffffffLL ||
      (N + kWideTile - 1) / kWideTile > 65535)
    return DISTIE_ERR_UNSUPPORTED;
  __nv_bfloat16 *xp = (__nv_bfloat16*)scratch, *wp = xp + (size_t)3 * M * K;
  CUtensorMap map_a, map_b;
  int status = make_map(&map_a, xp, 3 * M, K, K, kWideTile);
  if (status == 0) status = make_map(&map_b, wp, 3 * N, K, K, kWideTile);
  if (status != 0) return status;
  int* marks = (int*)(wp + (size_t)3 * N * K);
  static bool configured = false;
  const size_t shared = sizeof(WideShared) + 1024;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(gemm_float32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (err != cudaSuccess) return (int)err;
    configured = true;
  }
  // As many warps a row as hold it in registers, at most eight: 6,144 numbers (longer rows are read twice).
  const int warps = K <= kWideHeld * 256 ? 1 : K <= kWideHeld * 512 ? 2 : 8;
  const auto split = warps == 1 ? split_planes_kernel<1> : warps == 2 ? split_planes_kernel<2> : split_planes_kernel<8>;
  const dim3 split_grid((unsigned)(((long long)M + N + 8 / warps - 1) / (8 / warps)));
  cudaError_t err = launch_dependent(split, split_grid, dim3(256), 0, stream, x, x_stride, M, xp, w, N, wp, marks, K);
  if (err == cudaSuccess)
    err = launch_dependent(gemm_float32_kernel, dim3((M + kWideTile - 1) / kWideTile, (N + kWideTile - 1) / kWideTile), dim3(kWideThreads), shared,
                           stream, map_a, map_b, marks, bias, out, ldo, M, N, K, error);
  return err == cudaSuccess ? 0 : (int)err;
}
