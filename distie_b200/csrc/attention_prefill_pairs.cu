// Attention of prompt portions over the paged cache on the 5th-generation tensor cores, bfloat16: two query tiles a CTA, for
// steps with work for the whole machine (attention_prefill_tcgen05.cu takes the others; pairs_pay in kernels/device.py).
//
// What bounds it: a block of 128 x 128 scores costs 1,024 cycles of exponentials (16 a clock and SM) and, with heads of 128,
// 1,024 cycles of MMAs.  A CTA takes two query tiles of 128 rows that walk the same keys (a "unit": two heads of one group
// over the same tokens or, in groups of odd size, two tiles of one head), each with its own softmax warps.  While one tile's
// warps take exponentials, the tensor core multiplies for the other one:
//
//   S_h = Q_h K^T    tcgen05.mma, M = 128 query rows, N = 128 keys, reduction over head_dim; Q and K are K-major tiles in
//                    shared memory (TMA, 128-byte swizzle); S_h in tensor memory, 128 columns a tile
//   P_h = softmax    four warps a tile, a thread per query row with 64 of its scores in registers at a time; P goes back over
//                    the first 64 of the tile's columns of S as bfloat16, two keys to a column, in two halves of 64 keys, each
//                    with an mbarrier of its own, so that the first half's products run beside the second one's exponentials
//   O_h += P_h V     tcgen05.mma with P as the A operand straight from tensor memory, N = head_dim; V stays as the cache
//                    holds it (a key per row, head_dim contiguous), an MN-major B operand
//
//   tensor memory    S0 | S1 | O0 | O1 (128 + 128 + head_dim + head_dim columns)
//   MMA order        PV0(j), S0(j + 1), PV1(j), S1(j + 1): the S that overwrites a block's P is issued behind the products
//                    that read it (MMAs of one thread execute in the order of issue)
//
// Measured (28 heads of 128 in groups of 7, 1,733 tokens of three requests behind 7,000): 231 us against 373 with a tile a CTA,
// 0.79 PFLOP/s.  A block of both tiles takes 3,600 cycles, and either tile's chain is what they are: 1,100 for each half of the
// exponentials (512 of the special-function unit; the scores, the sums and the way back into tensor memory are the rest), 250
// to wake the issuer, 900 for the products.  Measured while the sums were of unrounded weights, 3,430 cycles a block:
// sixteen softmax warps with half of a row each 4,150, a search for the maximum in every block 3,800, a rolled loop over the
// halves 4,300 (copies of the scores), polling without sleep 3,600.
//
// Work is shared out among at most one CTA an SM by key blocks, not by tiles.  Every CTA reads the step's tiles and finds its
// part itself (a warp, before the wait for the kernel ahead):
//   * fewer units than CTAs: every unit is cut into ceil(blocks / L) pieces, a piece a CTA, with the smallest L >= kMinPiece
//     that leaves no more pieces than CTAs;
//   * more units, or pieces that leave some CTAs with much less than others: the units' blocks in a row (with kUnitCost for the
//     start and the end of each) are cut into equal shares; a cut within kMinCut blocks of an end of its unit moves there.
// A piece that is not its whole unit leaves maximum, sum and O of its rows in scratch, float32, and merge_pairs_kernel adds
// the pieces up.  A CTA's pieces run through one pipeline: the next piece's keys are loaded beside the last one's end.
//
// Keys and values come straight from their pages: a page of the cache is page_size rows of head_dim, so one TMA box of
// [page_size x 64] per page and half of the head fills its rows of the 128-key tile.  The copy engine takes such a box of 16
// rows every 55 cycles, 1,770 cycles for K and V of a block, which two tiles share.  Pages past the last key the tiles need are
// not fetched.  The page ids of a block are read from the table one block ahead of their use, by two producer warps (K and V),
// so that neither the look-up nor the other operand's stage stands between a stage becoming free and its copies.
//
// The running maximum is not searched for in every block: P is taken with the one in use, and only where the sum of a row's 64
// exponentials leaves the range (2^30: floating-point numbers keep their precision up to there, and far beyond) are its
// scores read again for their maximum, O and the sum so far scaled, and P taken once more.  So is the first block of a row.
// Searched for in every block, the maximum cost 800 of the 3,700 cycles between two blocks of a tile.  Normalisation by the row
// sum happens once, at the end.  The sum is that of the weights as bfloat16, which the product takes: a key that outweighs the
// others lies above the maximum in use and is no power of two, and its rounding would scale the whole output (standard
// deviation of the scores 1 / 3 / 6, error along the output's own direction 3.1e-4 / 1.1e-3 / 1.4e-3 with sums of what was not
// rounded yet, 3.0e-4 / 7.4e-4 / 5.2e-4 so; 3.0e-4 / 9.5e-4 / 1.05e-3 where a maximum is searched for in every block).  The two
// instructions a pair of weights that it costs are 12 of 226 us; a new maximum from 2^7 on instead, as exact, is free
// at a deviation of 1 and costs 130 us at 3.
//
// Rows of V that belong to no key of the request (pages that were not fetched) are set to zero in shared memory before the
// product, since 0 * garbage need not be 0.
//
//   warp 0       shares the work out (a ring of pieces in shared memory), loads Q, then K through its stages (a lane per page)
//   warp 1       allocates tensor memory; one lane issues the MMAs and commits them to mbarriers
//   warp 2       producer of the V blocks
//   warps 4..11  softmax, correction of O, end of a piece (4..7 tile 0, 8..11 tile 1)
//
// Every wait on an mbarrier is bounded; when one runs out the CTA sets the error word to 6, every role stops at its next
// wait, the producers wait (bounded) for their copies in flight, and tensor memory is released.  Page sizes 8, 16, ..., 128.
//
// Sizes: keys of up to DK = 64 or 128 elements and values of up to DV = 64 or 128, multiples of 8 and of one another
// independent.  A head smaller than its tile is padded on the way in: the copies fill what lies past the end of a key's or
// value's row with zeros.  (The columns of Q past the head's end hold the next head's: they meet the zeros of K.)
#include "softmax_pairs.cuh"
#include "tcgen05.cuh"

namespace distie {

constexpr int kPairRows = 128;   // query rows of a tile = lanes of tensor memory
constexpr int kPairKeys = 128;   // keys per block
constexpr int kPairVWarp = 2;
constexpr int kPairSoftmaxWarp = 4;  // the first one
constexpr int kPairThreads = 12 * 32;
constexpr int kPairRing = 4;     // pieces that the sharing warp may be ahead
constexpr int kPairHalf = kPairRows * 128;  // bytes of one [128 rows x 64 elements] swizzled half tile
constexpr float kPairLimit = 1073741824.f;  // a row whose exponentials of 64 keys sum up to more gets a new maximum
constexpr int kMinPiece = 8;     // blocks of a piece, at least, where units are cut to fill the machine
constexpr int kMinCut = 4;       // and where shares are cut
constexpr int kUnitCost = 2;     // blocks that the start and the end of a unit cost
constexpr int kPlanTiles = 4096; // tiles of a launch (their plan lies in the V stages until those are needed)
constexpr int kPairHeader = 8;   // ints of a slot of scratch: state, halves, then first token, rows, head of both tiles

struct PairArgs {
  const int* q_tiles;
  int num_tiles;
  const int *positions, *token_seq, *seq_seat, *block_table;
  int table_width, num_heads, group_size, num_kv_heads, key_dim, value_dim, page_shift, num_pages, window, key_chunk, keep_first;
  float scale_log2, cap, cap_pre;  // cap > 0: a raw score s becomes tanh(s * cap_pre), and scale_log2 is cap * log2(e)
  const float* sink_logits;        // one float per head whose exponential joins the row's sum at the end (null: none)
  __nv_bfloat16* out;
  int out_row_stride;
  float* partial;  // [2 * CTAs][2 tiles][128 * (DV + 2)], null: no unit is cut
  int* headers;    // [2 * CTAs][kPairHeader]
  int* error;
};

// A part of a unit that one CTA computes.
struct PairPiece {
  int t0[2], rows[2], pos0[2], head[2];
  int kv_head, seat;
  int first, end;  // blocks of the unit
  int halves;      // tiles of it: 2, or 1 where no second one goes with the first
  int slot;        // of the scratch that takes it; -1: the whole unit
  int stop;        // no piece: the CTA's work is done
  // Blocks that hold keys for a tile, where two tiles share the unit: the first one sees those before `seen_end`, the second one
  // all but [gap_from, gap_to), between the kept keys and its window.  Products with the others are left out: 0 * (what is
  // not finite) is not 0.
  int seen_end, gap_from, gap_to;
};

template <int DK, int DV>
struct PairShared {
  static constexpr int K_STAGES = 2, V_STAGES = 3;
  alignas(1024) unsigned char q[2][kPairRows * (DK > DV ? DK : DV) * 2];  // at the end of a unit: the output tiles
  alignas(1024) unsigned char k[K_STAGES][kPairKeys * DK * 2];
  alignas(1024) unsigned char v[V_STAGES][kPairKeys * DV * 2];
  alignas(16) PairPiece ring[kPairRing];
  uint64_t ring_full[kPairRing], ring_empty[kPairRing];
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[K_STAGES], k_empty[K_STAGES];
  uint64_t v_full[V_STAGES], v_empty[V_STAGES];
  uint64_t s_full[2];
  uint64_t p_full[2][2];  // [tile][half of the block's keys]
  uint64_t pv_done[2][2];
  uint64_t store_ready[2];  // the four warps have put their part of an output tile into shared memory
  uint32_t tmem_base;
  uint32_t failed;
};

// The key blocks that tokens at positions [first_pos, last_pos] of a request walk.  With a window that keeps the request's
// first `keep_first` keys, the blocks that hold those keys and lie wholly before the window's first block come first.
struct PairWalk {
  int first_key, kept, block_first, sink_blocks, blocks, last_pos;
  __device__ __forceinline__ PairWalk(int first_pos, int last, int window, int key_chunk, int keep_first) {
    last_pos = last;
    first_key = first_visible_key(first_pos, window, key_chunk);
    kept = min(keep_first, first_key);
    block_first = first_key / kPairKeys;
    sink_blocks = min((kept + kPairKeys - 1) / kPairKeys, block_first);
    blocks = sink_blocks + last_pos / kPairKeys - block_first + 1;
  }
  __device__ __forceinline__ int key0(int j) const { return (j < sink_blocks ? j : block_first + j - sink_blocks) * kPairKeys; }
  __device__ __forceinline__ int last_key(int j) const { return j < sink_blocks ? kept - 1 : last_pos; }
  // The page of `page` keys from `key` on is fetched when it holds a key that some row sees: one up to the block's last
  // needed key that lies in the window of the first row or among the kept first keys.  A cache with a window may have given
  // the other pages back already, so they are neither looked up nor fetched.
  __device__ __forceinline__ bool needed(int j, int key, int page) const {
    return key <= last_key(j) && (key + page - 1 >= first_key || key < kept);
  }
  __device__ __forceinline__ bool all_needed(int j, int page) const {  // (a sufficient condition)
    const int key = key0(j);
    return key + kPairKeys - page <= last_key(j) && (key + page - 1 >= first_key || (j < sink_blocks && key + kPairKeys <= kept));
  }
};

// Units of one tile, or of two where a group's heads do not pair up and the next tile goes on where this one ends.
struct PairGroup {
  int t0, rows, rows1, pos0, seq, tiles, units, blocks;
};
__device__ __forceinline__ bool pair_link(const PairArgs& a, int t, int t0, int rows, int seq) {
  if (t + 1 >= a.num_tiles) return false;
  const int next = __ldg(a.q_tiles + 2 * t + 2);
  return next == t0 + rows && __ldg(a.token_seq + next) == seq;
}
// `pairs`: the tile may go with the one behind it (it is the first, third, ... of its request).
__device__ __forceinline__ PairGroup pair_group(const PairArgs& a, int t, bool linked) {
  PairGroup g;
  g.t0 = __ldg(a.q_tiles + 2 * t);
  g.rows = __ldg(a.q_tiles + 2 * t + 1);
  g.pos0 = __ldg(a.positions + g.t0);
  g.seq = __ldg(a.token_seq + g.t0);
  g.tiles = linked ? 2 : 1;
  g.rows1 = linked ? __ldg(a.q_tiles + 2 * t + 3) : 0;
  g.units = a.num_kv_heads * (linked ? a.group_size : (a.group_size + 1) / 2);
  g.blocks = PairWalk(g.pos0, g.pos0 + g.rows + g.rows1 - 1, a.window, a.key_chunk, a.keep_first).blocks;
  return g;
}

// Where a CTA's work begins or ends: a block of a unit of a group of tiles.
struct PairPlace {
  int tile, unit, block;
};

// One warp: the parts of the step that CTA `cta` of `ctas` computes, from `start` up to `end`.  `plan` takes two ints a tile.
__device__ __forceinline__ void share_out(const PairArgs& a, int2* plan, int cta, int ctas, PairPlace& start, PairPlace& end) {
  const int lane = threadIdx.x & 31;
  const bool odd = a.group_size & 1;
  long long units = 0, blocks = 0;
  int longest = 0, carry_start = 0;
  bool carry_link = false;
  for (int base = 0; base < a.num_tiles; base += 32) {
    const int t = base + lane;
    int2 mine = make_int2(0, 0);  // units, blocks of each
    bool link = false;
    int t0 = 0, rows = 0;
    if (t < a.num_tiles) {
      t0 = __ldg(a.q_tiles + 2 * t);
      rows = __ldg(a.q_tiles + 2 * t + 1);
      link = odd && pair_link(a, t, t0, rows, __ldg(a.token_seq + t0));
    }
    // The first tile of this one's run of linked tiles: every second one from there leads a pair.
    bool before = __shfl_up_sync(0xffffffffu, link, 1);
    if (lane == 0) before = carry_link;
    int run = before ? -1 : t;
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, run, d);
      if (lane >= d) run = max(run, other);
    }
    run = max(run, carry_start);
    carry_start = __shfl_sync(0xffffffffu, run, 31);
    carry_link = __shfl_sync(0xffffffffu, link, 31);
    if (t < a.num_tiles) {
      if (((t - run) & 1) == 0 || !odd) {
        const PairGroup g = pair_group(a, t, link);
        mine = make_int2(g.units, g.blocks);
      }
      plan[t] = mine;
      units += mine.x;
      blocks += (long long)mine.x * mine.y;
      longest = max(longest, mine.y);
    }
  }
#pragma unroll 1
  for (int d = 16; d > 0; d >>= 1) {
    units += __shfl_xor_sync(0xffffffffu, units, d);
    blocks += __shfl_xor_sync(0xffffffffu, blocks, d);
    longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, d));
  }
  __syncwarp();
  const long long all = blocks + units * kUnitCost;
  bool few = units <= ctas;
  int low = 0;
  if (few) {  // the smallest size of a piece with enough CTAs for all
    int high = max(longest, kMinPiece);
    low = a.partial == nullptr ? high : (int)max((long long)kMinPiece, (blocks + ctas - 1) / ctas);
    high = max(high, low);
#pragma unroll 1
    while (low < high) {
      const int middle = (low + high) / 2;
      int pieces = 0;
#pragma unroll 1
      for (int t = lane; t < a.num_tiles; t += 32) pieces += plan[t].x * ((plan[t].y + middle - 1) / middle);
#pragma unroll 1
      for (int d = 16; d > 0; d >>= 1) pieces += __shfl_xor_sync(0xffffffffu, pieces, d);
      if (pieces <= ctas) high = middle;
      else low = middle + 1;
    }
    // Equal shares where whole units leave CTAs with much less than others (112 units of up to 33 blocks: 24 against 15).
    if (a.partial != nullptr && low > kMinPiece && 4ll * (low + kUnitCost) * ctas > 5 * all + 8ll * ctas) few = false;
  }
  // What a unit of n blocks counts for: its pieces, or its blocks and kUnitCost.  (Tiles that lead no unit have none of 0 blocks.)
  auto weight = [&](int n) { return few ? max(1, (n + low - 1) / low) : n + kUnitCost; };
  start.tile = end.tile = a.num_tiles;
  start.unit = start.block = end.unit = end.block = 0;
#pragma unroll 1
  for (int edge = 0; edge < (few ? 1 : 2); ++edge) {
    const long long x = few ? cta : all * (cta + edge) / ctas;
    long long done = 0;
#pragma unroll 1
    for (int base = 0; base < a.num_tiles; base += 32) {  // the unit that x of the row of all units falls into
      const int t = base + lane;
      const int2 p = t < a.num_tiles ? plan[t] : make_int2(0, 1);
      const int each = weight(p.y);
      const long long own = (long long)p.x * each;
      long long upto = own;
#pragma unroll 1
      for (int d = 1; d < 32; d <<= 1) {
        const long long other = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += other;
      }
      const unsigned past = __ballot_sync(0xffffffffu, done + upto > x);
      if (past == 0) {
        done += __shfl_sync(0xffffffffu, upto, 31);
        continue;
      }
      const int who = __ffs(past) - 1;
      const int at = (int)max(0ll, min(x - (done + upto - own), own));  // (of lane `who`: less than own)
      const int unit = __shfl_sync(0xffffffffu, at / each, who), rest = __shfl_sync(0xffffffffu, at % each, who);
      const int size = __shfl_sync(0xffffffffu, p.y, who);
      PairPlace place = {base + who, unit, 0};
      if (few) {
        const int pieces = weight(size);
        place.block = (int)((long long)rest * size / pieces);
        start = end = place;
        end.block = (int)((long long)(rest + 1) * size / pieces);
      } else {
        const int block = max(0, rest - kUnitCost), least = a.partial == nullptr ? size : kMinCut;
        place.block = min(block, size - block) >= least ? block : (2 * block <= size ? 0 : size);
        if (edge == 0) start = place;
        else end = place;
      }
      break;
    }
  }
}

// A warp's bounded wait, given up when another role of the CTA has failed (small: it is written out at every place that
// waits, and the roles together have to fit the instruction cache).
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, const volatile uint32_t* failed) {
#pragma unroll 1
  for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, done)) return true;
    if ((spin & 1023u) == 1023u && __any_sync(0xffffffffu, *failed)) return false;
  }
  return false;
}

// Waits for the warp's loads from tensor memory; no use of what they fill moves ahead of the wait.
__device__ __forceinline__ void behind_wait(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]),
                 "+r"(r[i + 7]));
}
__device__ __forceinline__ void tmem_wait_loads(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  behind_wait(r);
}
__device__ __forceinline__ void tmem_wait_loads(uint32_t (&r)[32], uint32_t (&s)[32]) {
  tmem_wait_loads(r);
  behind_wait(s);
}

template <int DK, int DV>
__global__ void __launch_bounds__(kPairThreads, 1)
attention_prefill_pairs_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                               const __grid_constant__ PairArgs a) {
  extern __shared__ unsigned char raw[];
  using Shared = PairShared<DK, DV>;
  auto& sm = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  constexpr int K_HALVES = DK / 64, V_HALVES = DV / 64, K_STAGES = Shared::K_STAGES, V_STAGES = Shared::V_STAGES;
  constexpr uint32_t TMEM_COLS = 512, O_COL = 256;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile uint32_t* failed = &sm.failed;

  if (threadIdx.x == 64) {
    prefetch_tensor_map(&map_q);
    prefetch_tensor_map(&map_k);
    prefetch_tensor_map(&map_v);
    prefetch_tensor_map(&map_out);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairRing; ++s) {
      mbar_init(&sm.ring_full[s], 1);
      mbar_init(&sm.ring_empty[s], 10);  // the MMA warp, eight softmax warps, the V producer
    }
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(&sm.k_full[s], 1);
      mbar_init(&sm.k_empty[s], 1);
    }
    for (int s = 0; s < V_STAGES; ++s) {
      mbar_init(&sm.v_full[s], 1);
      mbar_init(&sm.v_empty[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&sm.q_full[h], 1);
      mbar_init(&sm.q_empty[h], 1);
      mbar_init(&sm.s_full[h], 1);
      mbar_init(&sm.p_full[h][0], 4);  // one arrival per warp of the tile
      mbar_init(&sm.p_full[h][1], 4);
      mbar_init(&sm.pv_done[h][0], 1);
      mbar_init(&sm.pv_done[h][1], 1);
      mbar_init(&sm.store_ready[h], 4);
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

  const int page_size = 1 << a.page_shift, pages_per_block = kPairKeys >> a.page_shift;  // at most 16 pages
  // The warp polls a barrier and continues as one (the tensor-memory instructions need all lanes).
  auto wait_all = [&](uint64_t* bar, uint32_t parity) { return pair_wait(smem_u32(bar), parity, failed); };
  // This lane's page of block j of a piece, -1 where it is not needed or not in the table.
  auto page_of = [&](const PairWalk& walk, int seat, int j, bool& mine) {
    const int key = walk.key0(j) + (lane << a.page_shift);
    mine = lane < pages_per_block && walk.needed(j, key, page_size);
    const int column = key >> a.page_shift;
    return mine && column < a.table_width ? __ldg(a.block_table + (size_t)seat * a.table_width + column) : -1;
  };
  // Blocks [first, end) of a piece through the stages of K (warp 0) or V.  `count`: blocks loaded before this piece.
  auto load_blocks = [&](bool for_k, const PairWalk& walk, int kv_head, int seat, int first, int end, int& count, int page, bool mine) {
    const int stages = for_k ? K_STAGES : V_STAGES, halves = for_k ? K_HALVES : V_HALVES;
    const CUtensorMap* map = for_k ? &map_k : &map_v;
    uint64_t* full = for_k ? sm.k_full : sm.v_full;
    uint64_t* empty = for_k ? sm.k_empty : sm.v_empty;
    int s = count % stages, parity = ((count / stages) & 1) ^ 1;
    for (int j = first; j < end; ++j) {
      const uint32_t need = __ballot_sync(0xffffffffu, mine);
      if (__any_sync(0xffffffffu, mine && (unsigned)page >= (unsigned)a.num_pages)) {
        if (lane == 0 && a.error) atomicExch(a.error, 5);
        return false;
      }
      const bool now = mine;
      const int row = (page * a.num_kv_heads + kv_head) * page_size;
      mine = false;
      page = j + 1 < end ? page_of(walk, seat, j + 1, mine) : -1;
      if (!wait_all(&empty[s], parity)) return false;
      if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)(__popc(need) * page_size * halves * 128));
      __syncwarp();
      if (now) {
        unsigned char* stage = (for_k ? sm.k[s] : sm.v[s]) + lane * page_size * 128;
#pragma unroll 1
        for (int h = 0; h < halves; ++h) tma_load_2d(stage + h * kPairHalf, map, &full[s], h * 64, row);
      }
      __syncwarp();
      ++count;
      if (++s == stages) {
        s = 0;
        parity ^= 1;
      }
    }
    return true;
  };
  // Copies already under way must land before the CTA may leave: wait (bounded) for the last few.
  auto drain = [&](int count, bool for_k) {
    const int stages = for_k ? K_STAGES : V_STAGES;
#pragma unroll 1
    for (int n = max(0, count - stages); n < count; ++n) mbar_wait(for_k ? &sm.k_full[n % stages] : &sm.v_full[n % stages], (n / stages) & 1);
  };

  if (warp < kPairSoftmaxWarp) {
    if (warp == 0) {
      // ---- shares the work out, loads Q and K -------------------------------------------------------------------
      // The tiles' places in the step (tiles, positions, seats and block tables are inputs of the step, written by no kernel)
      // are looked up before the wait for the kernel that makes q and the newest keys and values.
      PairPlace at, end;
      share_out(a, reinterpret_cast<int2*>(sm.v[0]), blockIdx.x, gridDim.x, at, end);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the plan's place is loaded over by copies
      bool ok = true, waited = false;
      int pieces = 0, blocks = 0, q_uses[2] = {0, 0};
      const bool odd = a.group_size & 1;
      while (ok) {
        PairPiece p;
        p.stop = 1;
        PairGroup g;
        bool ends = false;
        while (at.tile < a.num_tiles && (at.tile < end.tile || (at.tile == end.tile && at.unit <= end.unit))) {
          const int t0 = __ldg(a.q_tiles + 2 * at.tile), rows = __ldg(a.q_tiles + 2 * at.tile + 1);
          g = pair_group(a, at.tile, odd && pair_link(a, at.tile, t0, rows, __ldg(a.token_seq + t0)));
          const bool last = at.tile == end.tile && at.unit == end.unit;
          const int upto = last ? end.block : g.blocks;
          const bool some = at.block < upto;
          if (some) {
            const int per_kv = g.units / a.num_kv_heads, pair = at.unit % per_kv;
            p.kv_head = at.unit / per_kv;
            p.halves = 2;
            for (int h = 0; h < 2; ++h) {
              const bool next = g.tiles == 2 && h == 1;  // the second of two tiles
              p.t0[h] = g.t0 + (next ? g.rows : 0);
              p.rows[h] = next ? g.rows1 : g.rows;
              p.pos0[h] = g.pos0 + (next ? g.rows : 0);
              p.head[h] = p.kv_head * a.group_size + (g.tiles == 2 ? pair : 2 * pair + h);
            }
            if (g.tiles == 1 && 2 * pair + 1 >= a.group_size) {
              p.halves = 1;
              p.head[1] = p.head[0];
            }
            p.seat = __ldg(a.seq_seat + g.seq);
            p.first = at.block;
            p.end = upto;
            p.stop = 0;
            ends = upto == g.blocks;
            p.slot = at.block == 0 && ends ? -1 : 2 * (int)blockIdx.x + (at.block == 0 ? 1 : 0);
          }
          at.block = 0;
          if (++at.unit >= g.units) {
            at.unit = 0;
            at.tile += g.tiles;
          }
          if (some || last) break;
        }
        const PairWalk walk(p.stop ? 0 : p.pos0[0], p.stop ? 0 : p.pos0[1] + p.rows[1] - 1, a.window, a.key_chunk, a.keep_first);
        p.seen_end = 0x7fffffff;
        p.gap_from = p.gap_to = 0;
        if (!p.stop && g.tiles == 2) {
          const int at_first = walk.sink_blocks - walk.block_first;  // from a block of keys to its place in the walk
          p.seen_end = at_first + (g.pos0 + g.rows - 1) / kPairKeys + 1;
          p.gap_from = at_first + max(walk.block_first, (a.keep_first + kPairKeys - 1) / kPairKeys);
          p.gap_to = at_first + first_visible_key(g.pos0 + g.rows, a.window, a.key_chunk) / kPairKeys;
        }
        bool mine = false;
        const int page = p.stop ? -1 : page_of(walk, p.seat, p.first, mine);
        if (!waited) {
          grid_dependency_wait();  // q and the newest keys and values come from the kernel before this one
          waited = true;
          if (a.partial != nullptr && lane == 0) a.headers[2 * blockIdx.x * kPairHeader] = a.headers[(2 * blockIdx.x + 1) * kPairHeader] = 0;
        }
        if (!p.stop && p.slot >= 0 && lane == 0) {
          int* header = a.headers + p.slot * kPairHeader;
          header[1] = p.halves;
          for (int h = 0; h < 2; ++h) {
            header[2 + h] = p.t0[h];
            header[4 + h] = p.rows[h];
            header[6 + h] = p.head[h];
          }
          header[0] = ends ? 3 : 1;
        }
        const int r = pieces % kPairRing;
        if (!wait_all(&sm.ring_empty[r], ((pieces / kPairRing) & 1) ^ 1)) { ok = false; break; }
        if (lane == 0) {
          sm.ring[r] = p;
          mbar_arrive(&sm.ring_full[r]);
        }
        __syncwarp();
        ++pieces;
        if (p.stop) break;
        for (int h = 0; h < p.halves && ok; ++h) {
          ok = wait_all(&sm.q_empty[h], (q_uses[h] & 1) ^ 1);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&sm.q_full[h], kPairRows * DK * 2);
            for (int c = 0; c < K_HALVES; ++c)
              tma_load_2d(sm.q[h] + c * kPairHalf, &map_q, &sm.q_full[h], p.head[h] * a.key_dim + c * 64, p.t0[h]);
          }
          ++q_uses[h];
        }
        __syncwarp();
        ok = ok && load_blocks(true, walk, p.kv_head, p.seat, p.first, p.end, blocks, page, mine);
      }
      if (!ok) atomicExch(&sm.failed, 1u);
      if (*failed && lane == 0) {
        for (int h = 0; h < 2; ++h)
          if (q_uses[h] > 0) mbar_wait(&sm.q_full[h], (q_uses[h] - 1) & 1);
        drain(blocks, true);
      }
    } else if (warp == kPairVWarp) {
      // ---- loads V -------------------------------------------------------------------------------------------------
      grid_dependency_wait();
      bool ok = true;
      int blocks = 0;
      for (int pieces = 0; ok; ++pieces) {
        const int r = pieces % kPairRing;
        if (!wait_all(&sm.ring_full[r], (pieces / kPairRing) & 1)) { ok = false; break; }
        const int kv_head = sm.ring[r].kv_head, seat = sm.ring[r].seat, first = sm.ring[r].first, end = sm.ring[r].end;
        const int stop = sm.ring[r].stop, pos0 = sm.ring[r].pos0[0], last_pos = sm.ring[r].pos0[1] + sm.ring[r].rows[1] - 1;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.ring_empty[r]);
        if (stop) break;
        const PairWalk walk(pos0, last_pos, a.window, a.key_chunk, a.keep_first);
        bool mine;
        const int page = page_of(walk, seat, first, mine);
        ok = load_blocks(false, walk, kv_head, seat, first, end, blocks, page, mine);
      }
      if (!ok) atomicExch(&sm.failed, 1u);
      if (*failed && lane == 0) drain(blocks, false);
    } else if (warp == 1) {
      // ---- MMA issuer: the warp walks together and an elected lane issues a batch.  In a branch that one lane takes for itself
      // the compiler looks for more lanes with other operands at every MMA: 130 cycles to issue one of 64 -----------------
      constexpr uint32_t idesc_s = instr_desc(kPairKeys);
      constexpr uint32_t idesc_o = instr_desc(DV, true);
      bool ok = true;
      int blocks = 0, cnt[2] = {0, 0}, uses[2] = {0, 0};
      for (int pieces = 0; ok; ++pieces) {
        const int r = pieces % kPairRing;
        if (!wait_all(&sm.ring_full[r], (pieces / kPairRing) & 1)) { ok = false; break; }
        const int n = sm.ring[r].end - sm.ring[r].first, halves = sm.ring[r].halves, stop = sm.ring[r].stop;
        const int seen_end = sm.ring[r].seen_end - sm.ring[r].first, gap_from = sm.ring[r].gap_from - sm.ring[r].first;
        const int gap_to = sm.ring[r].gap_to - sm.ring[r].first, first1 = gap_from <= 0 ? max(0, gap_to) : 0;  // (the second tile's first)
        // Where the output tile goes through the place of Q, the store hands that back.
        const bool plain = sm.ring[r].slot >= 0 || a.value_dim != DV;
        const bool frees_q[2] = {plain || sm.ring[r].rows[0] != kPairRows, plain || sm.ring[r].rows[1] != kPairRows};
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.ring_empty[r]);
        if (stop) break;
        // One copy of the code for both tiles, and for the first S alone (j = -1): what is small stays in the cache.
#pragma unroll 1
        for (int j = -1; j < n && ok; ++j) {
          const bool more = j + 1 < n;
          const int next = blocks + (j >= 0), vs = blocks % V_STAGES, ks = next % K_STAGES;
          const uint64_t v_desc = smem_desc_mn(sm.v[0], kPairHalf, 1024) + (uint64_t)(vs * (kPairKeys * DV * 2 / 16));
          const uint64_t k_desc = smem_desc(sm.k[0]) + (uint64_t)(ks * (kPairKeys * DK * 2 / 16));
          if (j >= 0) ok = wait_all(&sm.v_full[vs], (blocks / V_STAGES) & 1);
          if (ok && more) ok = wait_all(&sm.k_full[ks], (next / K_STAGES) & 1);
#pragma unroll 1
          for (int h = 0; h < halves && ok; ++h) {
            const uint32_t s_cols = tmem + h * kPairKeys, o_cols = tmem + O_COL + h * DV;
            const uint32_t phase = (h == 0 ? cnt[0] : cnt[1]) & 1;
            if (j >= 0) {  // O of the tile += P V of block j of the piece
              const bool sees = h == 0 ? j < seen_end : j < gap_from || j >= gap_to;
              const uint32_t add = j > (h == 0 ? 0 : first1) ? 1u : 0u;
#pragma unroll
              for (int part = 0; part < 2; ++part) {
                if (!wait_all(&sm.p_full[h][part], phase)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                  if (sees) {
#pragma unroll
                    for (int kk = part * 4; kk < part * 4 + 4; ++kk)  // 16 keys: 8 columns of P, 16 rows of V
                      umma_bf16_ts(o_cols, s_cols + kk * 8, v_desc + (uint64_t)((kk * 16 * 128) >> 4), idesc_o, kk > 0 ? 1u : add);
                  }
                  umma_commit(&sm.pv_done[h][part]);
                  if (part == 1 && h == halves - 1) umma_commit(&sm.v_empty[vs]);
                }
                __syncwarp();
              }
              if (h == 0) ++cnt[0];
              else ++cnt[1];
            } else {
              ok = wait_all(&sm.q_full[h], (h == 0 ? uses[0]++ : uses[1]++) & 1);
            }
            if (ok && more && elect_one()) {  // S of the tile over the block behind
              const uint64_t q_desc = smem_desc(sm.q[0]) + (uint64_t)(h * (sizeof(sm.q[0]) / 16));
#pragma unroll
              for (int kk = 0; kk < DK / 16; ++kk) {
                const uint64_t step = (uint64_t)(((kk >> 2) * kPairHalf + (kk & 3) * 32) >> 4);
                umma_bf16(s_cols, q_desc + step, k_desc + step, idesc_s, kk > 0 ? 1u : 0u);
              }
              umma_commit(&sm.s_full[h]);
              if (h == halves - 1) umma_commit(&sm.k_empty[ks]);
              if (j + 2 == n && (h == 0 ? frees_q[0] : frees_q[1])) umma_commit(&sm.q_empty[h]);
            }
            __syncwarp();
          }
          blocks = next;
        }
      }
      if (!ok) atomicExch(&sm.failed, 1u);
    }
  } else {
    // ---- softmax, correction, end of a piece: thread = query row of tile h ---------------------------------------------
    const int quadrant = warp & 3, h = (warp - kPairSoftmaxWarp) >> 2;
    const int r = quadrant * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quadrant * 32) << 16);
    const uint32_t s_addr = lane_base + h * kPairKeys, o_addr = lane_base + O_COL + h * DV;
    bool ok = true;
    int cnt = 0, blocks = 0, stored = 0;  // blocks of this tile, blocks of the CTA, output tiles through shared memory
    grid_dependency_wait();
    for (int pieces = 0; ok; ++pieces) {
      const int ring = pieces % kPairRing;
      if (!wait_all(&sm.ring_full[ring], (pieces / kPairRing) & 1)) { ok = false; break; }
      const PairPiece& entry = sm.ring[ring];  // ours until the piece is done
      auto done_with = [&] {
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.ring_empty[ring]);
      };
      if (entry.stop || h >= entry.halves) {
        const bool stop = entry.stop;
        blocks += stop ? 0 : entry.end - entry.first;
        done_with();
        if (stop) break;
        continue;
      }
      const int first = entry.first, last = entry.end, pos0 = entry.pos0[h];
      const int open_from = first_visible_key(pos0 + entry.rows[h] - 1, a.window, a.key_chunk);
      const PairWalk walk(entry.pos0[0], entry.pos0[1] + entry.rows[1] - 1, a.window, a.key_chunk, a.keep_first);
      float m_used = -INFINITY, l = 0.f;
#pragma unroll 1
      for (int j = first; j < last; ++j, ++cnt, ++blocks) {
        float cap = a.cap;  // (hidden from the compiler, which would write the loop out for either case)
        asm volatile("" : "+f"(cap));
        const int key0 = walk.key0(j);
        // No row of the tile needs a mask when every key of the block is old enough and inside every window.
        const bool unmasked = j >= walk.sink_blocks && key0 + kPairKeys - 1 <= pos0 && key0 >= open_from;
        const bool plain = unmasked && !(cap > 0.f);
        auto special = [&](uint32_t (&sv)[32], int column) {
          if (cap > 0.f) {  // one more special-function instruction per score, and a multiplication per pair of scores
            const uint64_t pre2 = pair_of(a.cap_pre, a.cap_pre), zero2 = pair_of(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float x0, x1;
              halves_of(fma_pairs(pair_of(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), pre2, zero2), x0, x1);
              sv[i] = __float_as_uint(tanh_fast(x0));
              sv[i + 1] = __float_as_uint(tanh_fast(x1));
            }
          }
          const int limit = pos0 + min(r, entry.rows[h] - 1);                  // newest key this row may see
          const int oldest = first_visible_key(limit, a.window, a.key_chunk);  // oldest key inside its window or chunk
          const int key = key0 + column, upto = limit - key, from = oldest - key, kept = a.keep_first - key;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i > upto || (i < from && i >= kept)) sv[i] = 0xff800000u;  // -inf
        };
        if (!wait_all(&sm.s_full[h], cnt & 1)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // Rows of V in pages that were not fetched: zero, so that P = 0 gives 0.  Tile 0's warps clear them for both tiles:
        // its products with a block are issued ahead of the other one's.  (A block that needs no mask needs all its pages.)
        if (h == 0 && !unmasked && !walk.all_needed(j, page_size)) {
          const int vs = blocks % V_STAGES;
          if (!wait_all(&sm.v_full[vs], (blocks / V_STAGES) & 1)) { ok = false; break; }
          if (!walk.needed(j, key0 + (r >> a.page_shift << a.page_shift), page_size)) {
#pragma unroll 1
            for (int c = 0; c < V_HALVES * 8; ++c)
              *reinterpret_cast<uint4*>(sm.v[vs] + (c >> 3) * kPairHalf + r * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();  // (what follows a branch is not written out once more for either way)
        uint32_t s0[32], s1[32], s2[32], s3[32];
        tmem_load_32(s_addr, s0);
        tmem_load_32(s_addr + 32, s1);
        tmem_wait_loads(s0, s1);
#pragma unroll
        for (int part = 0; part < 2; ++part) {  // 64 keys
          auto& u = part == 0 ? s0 : s2;
          auto& v = part == 0 ? s1 : s3;
          const int column = part * 64;
          // The maximum of these scores becomes the one in use in the rows that ask for it; O and the sum follow.
          auto raise = [&](bool mine) {
            float mx = -INFINITY;
#pragma unroll 1
            for (int c = 0; c < 64; c += 16) {
              uint32_t t[16];
              tmem_load_16(s_addr + column + c, t);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              const int key = key0 + column + c, limit = pos0 + min(r, entry.rows[h] - 1);
              const int oldest = first_visible_key(limit, a.window, a.key_chunk);
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (key + i <= limit && (key + i >= oldest || key + i < a.keep_first)) mx = fmaxf(mx, __uint_as_float(t[i]));
            }
            if (cap > 0.f) mx = mx == -INFINITY ? mx : tanh_fast(mx * a.cap_pre);
            const float m_new = mine ? fmaxf(m_used, mx * a.scale_log2) : m_used;
            const float corr = m_used == -INFINITY ? 0.f : exp2_approx(m_used - m_new);
            m_used = m_new;
            l *= corr;
            // O holds the products of the piece's keys before these, of which the last may still run.
            if (part == 1 && !wait_all(&sm.pv_done[h][0], cnt & 1)) return false;
            if (part == 1 || j > first) {
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
              for (int c0 = 0; c0 < DV; c0 += 16) {
                uint32_t o[16];
                tmem_load_16(o_addr + c0, o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                tmem_store_16(o_addr + c0, o);
              }
            }
            return true;
          };
          if (!plain) {
            special(u, column);
            special(v, column + 32);
          }
          if (__any_sync(0xffffffffu, m_used == -INFINITY) && !raise(m_used == -INFINITY)) { ok = false; break; }
          __syncwarp();
          // P = exp2(S * scale - maximum in use), two keys to a register, and the sum of what they hold; a masked S is -inf and gives 0.
          uint32_t packed[32];
          auto take = [&] {
            const float shift = m_used == -INFINITY ? 0.f : m_used;
            const uint64_t scale2 = pair_of(a.scale_log2, a.scale_log2), shift2 = pair_of(-shift, -shift);
            uint64_t sum4[4] = {0ull, 0ull, 0ull, 0ull};  // four pairs of running sums
#pragma unroll
            for (int i = 0; i < 64; i += 2) {
              const uint32_t s0 = i < 32 ? u[i & 31] : v[i & 31], s1 = i < 32 ? u[(i + 1) & 31] : v[(i + 1) & 31];
              float x0, x1;
              halves_of(fma_pairs(pair_of(__uint_as_float(s0), __uint_as_float(s1)), scale2, shift2), x0, x1);
              const __nv_bfloat162 pair = __floats2bfloat162_rn(exp2_approx(x0), exp2_approx(x1));
              packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&pair);
              sum4[(i >> 1) & 3] = add_pairs(sum4[(i >> 1) & 3], pair_of(__uint_as_float(packed[i >> 1] << 16),
                                                                         __uint_as_float(packed[i >> 1] & 0xffff0000u)));
            }
            float even, uneven;
            halves_of(add_pairs(add_pairs(sum4[0], sum4[1]), add_pairs(sum4[2], sum4[3])), even, uneven);
            return even + uneven;
          };
          float sum = take();
          if (__any_sync(0xffffffffu, !(sum <= kPairLimit))) {
            if (!raise(!(sum <= kPairLimit))) { ok = false; break; }
            sum = take();
          }
          __syncwarp();
          l += sum;
          if (part == 0) {
            tmem_load_32(s_addr + 64, s2);
            tmem_load_32(s_addr + 96, s3);
          }
          // P of these keys over the first columns of S, whose scores have been read: two keys to a column.
          tmem_store_32(s_addr + part * 32, packed);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.p_full[h][part]);
          if (part == 0) tmem_wait_loads(s2, s3);
        }
        if (!ok) break;
      }
      if (!ok) break;
      // ---- end of the piece: the whole unit's rows to `out`, a part's to scratch ----------------------------------------
      if (!wait_all(&sm.pv_done[h][1], (cnt - 1) & 1)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int slot = entry.slot;
      if (slot >= 0) {
        float* dst = a.partial + (size_t)(2 * slot + h) * (kPairRows * (DV + 2));
#pragma unroll 1
        for (int c0 = 0; c0 < DV; c0 += 32) {
          uint32_t u[32];
          tmem_load_32(o_addr + c0, u);
          tmem_wait_loads(u);
#pragma unroll
          for (int i = 0; i < 32; i += 4)  // [4 columns][128 rows]: a warp's rows lie side by side
            reinterpret_cast<uint4*>(dst)[(c0 + i) / 4 * kPairRows + r] = make_uint4(u[i], u[i + 1], u[i + 2], u[i + 3]);
        }
        dst[kPairRows * DV + r] = m_used;
        dst[kPairRows * (DV + 1) + r] = l;
        done_with();
        continue;
      }
      const int t0 = entry.t0[h], rows = entry.rows[h], head = entry.head[h];
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (a.sink_logits) inv = sink_inverse_log2(m_used, l, a.sink_logits[head]);
      // A whole tile of 128 rows goes into the shared memory that held Q (all products with Q are done), in the layout of a
      // tile copy, and leaves as one: 128 rows of whole lines, where the threads' own stores are 16 bytes of 32 different
      // rows per instruction.  A partial tile (the end of a request) is stored by the threads, row by row; so is a tile of
      // heads that do not fill it: a copy would reach into the next head's columns.
      const bool whole = rows == kPairRows && a.value_dim == DV;
      __nv_bfloat16* dst = a.out + (size_t)(t0 + r) * a.out_row_stride + (size_t)head * a.value_dim;
#pragma unroll 1
      for (int c0 = 0; c0 < DV; c0 += 32) {
        uint32_t u[32];
        tmem_load_32(o_addr + c0, u);
        tmem_wait_loads(u);
        if (whole || r < rows) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            const int dim = c0 + i;  // 8 dims = one 16-byte piece of the row's 128-byte line
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(u[i + e]) * inv;
            if (whole) {
              const uint32_t to = smem_u32(sm.q[h]) + (dim >> 6) * kPairHalf + r * 128 + ((((dim & 63) >> 3) ^ (r & 7)) << 4);
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 pair = __floats2bfloat162_rn(y[2 * e], y[2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t*>(&pair);
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
            } else if (dim < a.value_dim) {
              store8(dst + dim, y);
            }
          }
        }
        __syncwarp();
      }
      done_with();
      if (whole) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stores above, before the copy reads them
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.store_ready[h]);
        if (quadrant == 0) {
          if (!wait_all(&sm.store_ready[h], stored & 1)) { ok = false; break; }
          if (lane == 0) {
#pragma unroll
            for (int c = 0; c < V_HALVES; ++c)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&map_out),
                           "r"(head * DV + c * 64), "r"(t0), "r"(smem_u32(sm.q[h] + c * kPairHalf)) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // read before Q is loaded over it or the CTA ends
            mbar_arrive(&sm.q_empty[h]);
          }
          __syncwarp();
        }
        ++stored;
      }
    }
    if (!ok) atomicExch(&sm.failed, 1u);
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  if (threadIdx.x == 0 && sm.failed && a.error) atomicCAS(a.error, 0, 6);
}

// Adds the parts of a cut unit up: block (x, y) takes 32 rows of a tile of the unit whose first part CTA x wrote (slot 2 x + 1);
// the next ones are slots 2 (x + 1), 2 (x + 2), ... up to the part that ends the unit.
template <int DV>
__global__ void __launch_bounds__(256) merge_pairs_kernel(const __grid_constant__ PairArgs a, int ctas) {
  __shared__ float tile[32][DV + 4];
  grid_dependency_release();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cta = blockIdx.x, half = blockIdx.y >> 2, row0 = (blockIdx.y & 3) * 32;
  const int* header = a.headers + (2 * cta + 1) * kPairHeader;
  if (__ldcg(header) == 0 || half >= __ldcg(header + 1)) return;
  const int t0 = __ldcg(header + 2 + half), rows = __ldcg(header + 4 + half), head = __ldcg(header + 6 + half);
  if (row0 >= rows) return;
  int parts = 0;
  for (int base = cta + 1; base < ctas && parts == 0; base += 32) {
    const unsigned ending = __ballot_sync(0xffffffffu, base + lane < ctas && __ldcg(a.headers + 2 * (base + lane) * kPairHeader) == 3);
    if (ending) parts = base - cta + __ffs(ending);
  }
  if (parts == 0) {  // (every unit that a CTA begins is ended by one behind it: a plan or a header went wrong)
    if (threadIdx.x == 0 && a.error) atomicCAS(a.error, 0, 6);
    return;
  }
  auto part_at = [&](int i) {
    return a.partial + (size_t)(2 * (i == 0 ? 2 * cta + 1 : 2 * (cta + i)) + half) * (kPairRows * (DV + 2));
  };
  const int row = row0 + lane;
  float top = -INFINITY;
  for (int i = 0; i < parts; ++i) top = fmaxf(top, __ldcg(part_at(i) + kPairRows * DV + row));
  float sum = 0.f;
  constexpr int OWN = DV / 32;  // groups of four columns a thread
  float4 acc[OWN];
#pragma unroll
  for (int c = 0; c < OWN; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int i = 0; i < parts; ++i) {
    const float* part = part_at(i);
    float4 v[OWN];
#pragma unroll
    for (int c = 0; c < OWN; ++c) v[c] = __ldcg(reinterpret_cast<const float4*>(part) + (warp * OWN + c) * kPairRows + row);
    const float m = __ldcg(part + kPairRows * DV + row);
    if (m == -INFINITY) continue;  // (a part without a key for this row: where its tile sees none at all, O was not written)
    const float w = exp2_approx(m - top);
    sum += w * __ldcg(part + kPairRows * (DV + 1) + row);
#pragma unroll
    for (int c = 0; c < OWN; ++c) {
      acc[c].x += w * v[c].x;
      acc[c].y += w * v[c].y;
      acc[c].z += w * v[c].z;
      acc[c].w += w * v[c].w;
    }
  }
  float inv = sum > 0.f ? 1.f / sum : 0.f;
  if (a.sink_logits) inv = sink_inverse_log2(top, sum, a.sink_logits[head]);
#pragma unroll
  for (int c = 0; c < OWN; ++c) {
    float* to = &tile[lane][(warp * OWN + c) * 4];
    *reinterpret_cast<float4*>(to) = make_float4(acc[c].x * inv, acc[c].y * inv, acc[c].z * inv, acc[c].w * inv);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp * 4 + i;
    if (row0 + r < rows && lane * 4 < a.value_dim && lane * 4 < DV)
      store4(a.out + (size_t)(t0 + row0 + r) * a.out_row_stride + (size_t)head * a.value_dim + lane * 4,
             *reinterpret_cast<const float4*>(&tile[r][lane * 4]));
  }
}

template <int DK, int DV>
static int launch_attention_pairs(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                                  const CUtensorMap& map_out, PairArgs args, int ctas, cudaStream_t stream) {
  const size_t shared = sizeof(PairShared<DK, DV>) + 1024;
  static_assert(sizeof(PairShared<DK, DV>) + 1024 <= 232448, "shared memory of a CTA");
  static_assert(kPlanTiles * 8 <= PairShared<DK, DV>::V_STAGES * kPairKeys * DV * 2, "the plan lies in the V stages");
  static bool configured = false;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(attention_prefill_pairs_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)shared);
    if (err != cudaSuccess) return (int)err;
    configured = true;
  }
  const int tiles = args.num_tiles;
  const int* q_tiles = args.q_tiles;
  for (int first = 0; first < tiles; first += kPlanTiles) {
    args.q_tiles = q_tiles + 2 * first;
    args.num_tiles = min(kPlanTiles, tiles - first);
    cudaError_t err = launch_dependent(attention_prefill_pairs_kernel<DK, DV>, dim3(ctas), dim3(kPairThreads), shared, stream, map_q,
                                       map_k, map_v, map_out, args);
    if (err == cudaSuccess && args.partial != nullptr)
      err = launch_dependent(merge_pairs_kernel<DV>, dim3(ctas, 8), dim3(256), 0, stream, args, ctas);
    if (err != cudaSuccess) return (int)err;
  }
  return 0;
}

}  // namespace distie

using namespace distie;

// Floats of scratch that distie_attention_prefill_pairs wants, 0 where no unit is cut: `max_keys` is the most keys that a
// request of the step has.
extern "C" long long distie_attention_prefill_pairs_scratch_floats(int max_keys, int value_dim, int sm_count) {
  if (max_keys <= kMinPiece * kPairKeys) return 0;
  const int dv = value_dim <= 64 ? 64 : 128;
  return (long long)sm_count * 2 * (2 * kPairRows * (dv + 2) + kPairHeader);
}

// q_tiles: [num_tiles, 2] int32, first token and number of rows (<= 128) of tiles whose tokens belong to one request.
// q is [tokens, >= num_heads * head_dim] bfloat16 with row stride q_row_stride; the caches are
// [num_pages, num_kv_heads, page_size, head_dim] (values: value_dim).  scratch: distie_attention_prefill_pairs_scratch_floats
// floats, 16-byte aligned, or null where that is 0.  Returns DISTIE_ERR_UNSUPPORTED for a head_dim or value_dim above 128 or
// no multiple of 8, or a page size that is not 8, 16, ..., 128.
extern "C" int distie_attention_prefill_pairs(const void* q, int q_row_stride, void* out, int out_row_stride,
                                              const int* q_tiles, int num_tiles, const int* positions,
                                              const int* token_seq, const int* seq_seat, const int* block_table,
                                              int table_width, const void* k_cache, const void* v_cache, int tokens,
                                              int num_heads, int num_kv_heads, int head_dim, int value_dim, int page_size,
                                              int num_pages, int window, int key_chunk, int keep_first, float scale,
                                              float softcap, const float* sink, float* scratch, int sm_count, int* error,
                                              cudaStream_t stream) {
  if (num_tiles <= 0) return 0;
  if (tokens < 1 || num_heads < 1 || num_kv_heads < 1 || num_heads % num_kv_heads != 0 || table_width < 1 ||
      num_pages < 1 || num_tiles > 65535 || keep_first < 0 || sm_count < 1)
    return DISTIE_ERR_ARG;
  if (head_dim < 8 || head_dim > 128 || (head_dim & 7) || value_dim < 8 || value_dim > 128 || (value_dim & 7) || page_size < 8 ||
      page_size > 128 || (page_size & (page_size - 1)) || (q_row_stride & 7) || (out_row_stride & 7) || ((uintptr_t)q & 15) ||
      ((uintptr_t)out & 15) || ((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15) || ((uintptr_t)scratch & 15))
    return DISTIE_ERR_UNSUPPORTED;
  PairArgs args = {};
  while ((1 << args.page_shift) < page_size) ++args.page_shift;
  CUtensorMap map_q, map_k, map_v, map_out;
  int status = make_map(&map_q, q, tokens, num_heads * head_dim, q_row_stride, kPairRows);
  if (status != 0) return status;
  if ((status = make_map(&map_out, out, tokens, num_heads * value_dim, out_row_stride, kPairRows)) != 0) return status;
  const long long cache_rows = (long long)num_pages * num_kv_heads * page_size;
  if (cache_rows > 0x7fffffffLL) return DISTIE_ERR_UNSUPPORTED;
  if ((status = make_map(&map_k, k_cache, (int)cache_rows, head_dim, head_dim, page_size)) != 0) return status;
  if ((status = make_map(&map_v, v_cache, (int)cache_rows, value_dim, value_dim, page_size)) != 0) return status;
  args.q_tiles = q_tiles;
  args.num_tiles = num_tiles;
  args.positions = positions;
  args.token_seq = token_seq;
  args.seq_seat = seq_seat;
  args.block_table = block_table;
  args.table_width = table_width;
  args.num_heads = num_heads;
  args.group_size = num_heads / num_kv_heads;
  args.num_kv_heads = num_kv_heads;
  args.key_dim = head_dim;
  args.value_dim = value_dim;
  args.num_pages = num_pages;
  args.window = window;
  args.key_chunk = key_chunk;
  args.keep_first = keep_first;
  args.cap = softcap > 0.f ? softcap : 0.f;
  args.cap_pre = args.cap > 0.f ? scale / args.cap : 0.f;
  args.scale_log2 = (args.cap > 0.f ? args.cap : scale) * 1.4426950408889634f;
  args.sink_logits = sink;
  args.out = (__nv_bfloat16*)out;
  args.out_row_stride = out_row_stride;
  args.error = error;
  if (scratch != nullptr) {
    const int dv = value_dim <= 64 ? 64 : 128;
    args.partial = scratch;
    args.headers = (int*)(scratch + (size_t)sm_count * 4 * kPairRows * (dv + 2));
  }
  if (head_dim <= 64) {
    if (value_dim <= 64) return launch_attention_pairs<64, 64>(map_q, map_k, map_v, map_out, args, sm_count, stream);
    return launch_attention_pairs<64, 128>(map_q, map_k, map_v, map_out, args, sm_count, stream);
  }
  if (value_dim <= 64) return launch_attention_pairs<128, 64>(map_q, map_k, map_v, map_out, args, sm_count, stream);
  return launch_attention_pairs<128, 128>(map_q, map_k, map_v, map_out, args, sm_count, stream);
}
