// Gate scorer on tcgen05 tensor cores (bf16/f16, head_dim 64/128): block_size 128 and at most 8 ranked
// blocks per query; EXACT (below) for the other block sizes and up to 16.
//
// Persistent CTAs (two per SM) walk units of two neighbouring 128-query tiles of one (sequence, query
// head), heaviest first, in alternating direction per round. With 128-token blocks a tile is exactly one
// block, so every row of a tile has the same candidates: the blocks before the tile's own. Roles:
//   loader (1 thread)  TMA: block means, 64 blocks a step; the unit's queries into the L2
//   mma    (1 warp)    S = Q Kbar^T (M128 N64 K=D) with Q as operand A from TMEM, tile by tile, for a
//                      few steps of the unit (bounding pass) and then for all (ranking pass)
//   select (4 warps per tile) bring the tile's queries into TMEM, then one row per thread; no two
//          threads share a word:
//          1. The bounding pass only keeps, per row, the maxima of sixteen interleaved subsets of
//             the scores (half an instruction per score): the L-th largest of them is a score that at
//             least L candidates reach, so nothing below it can be selected.
//          2. The ranking pass rounds the scores to the input dtype, two per instruction, takes the
//             signs of (bound - score) of four scores into a bit mask with four more, and leaves the row's
//             64 scores in shared memory.
//          3. What passed (some 18 of 1024 candidates) is popped from the mask and offered to the
//             row's sorted register list of L keys, all lanes of the warp in step, which raises the
//             bound to the score of the list's last entry (candidates arrive in ascending block order,
//             so an equal score never wins). A lane may lag a window behind: with two windows of 64
//             scores per thread the rounds are the most that any lane has left of the *older* one, 38 for
//             1024 candidates where windows popped on their own take 58.
//          A key is the score rounded to the input dtype and made monotone in the high half and
//          0xFFFF - block id in the low half, so "score descending, ties to the lower id" is plain
//          integer order.
// The ALU pipe bounds it (58 % of its peak): 2.5 of the 5.7 instructions that one more score costs run there, at
// half rate. An SM's tensor pipe takes
// 90 clocks for an M128 N64 K16 instruction with both operands in shared memory and half of that with A in
// TMEM, which at head_dim 128 would bound the kernel otherwise; and issued from a branch of one lane, where
// descriptors do not stay in uniform registers, one took 120. Before, each score that passed was appended to a
// buffer by predicated stores, five instructions a score whether it passed or not, and the two halves of a row's
// candidates had lists of their own. us, before and now:
//   131072 queries x 4 heads of 64, 1024 blocks       218    125       65536 x 4, 512 blocks, 12 each (exact)    319   137
//   131072 x 32 heads of 128                         2170   1070       2 x 8192 x 4 of 128, blocks of 64 (exact) 117    42
//   524288 x 32 heads of 128, skewed                27300  12500       16 sequences, 40000 x 32 heads of 128     271   144
//
// EXACT: the same kernel where the portable gate used to run (other block sizes that divide 128,
// more than eight ranked blocks): its selections are those of exact scores, bit for bit. The
// tensor-core sum is off by at most `err` (a bound from the lengths of the query and of the means of
// the unit's candidates), so the entry test is loosened by err, the windows keep all 32 bits of a score,
// and a candidate whose rounding to the input dtype depends on that error is scored again in float64
// before it is ranked, four by a warp at a time: about one in forty where scores are large against err,
// every one near zero. A row without a finite bound (infinities, NaN, squares outside float32) has every candidate
// scored in float64. With blocks finer than the tile a row's candidates end at its own block.
//
// Scores are float32 tensor-core sums rounded to the input dtype; the portable
// gate rounds the exact sum. The two differ only when a float32 partial sum
// straddles a rounding boundary of the input dtype.
//
// Stands in for gate_kernel of the reference (src/moba/kernels/gating.py:92-335).
#include "common.cuh"
#include "sm100.cuh"

#include <type_traits>

namespace moba {
using namespace sm100;

namespace {

constexpr int kTile = 128;
constexpr int kSub = kTile * 128;
constexpr int kStepBlocks = 64;            // blocks scored per step
constexpr int kMaxTake = 8;
constexpr int kSubsets = 16;               // column subsets of the bounding pass: at least L

// Two tiles to a CTA and two CTAs to an SM, so that one's hand-over between units falls into the other's work.
template <int D, bool EXACT> struct GateCfg {
  static constexpr int kTiles = 2, kCtas = 2;
  static constexpr int kSubs = D / 64;
  static constexpr int kKb = kSubs * kStepBlocks * 128, kStages = D == 64 ? 4 : 2;   // block means: bytes of a step, stages
  static constexpr int kSelect = kTiles * kTile, kThreads = kSelect + 64;
  static constexpr int kMmaWarp = kSelect / 32, kLoadWarp = kMmaWarp + 1;
  // A thread's window of scores: 64 columns of two bytes (exact: 32 of four), in eight pieces of 16 bytes.
  // The two windows of a warpgroup also take its Q tile on the way to TMEM.
  static constexpr int kPiece = kTile * 16, kWindow = 8 * kPiece, kQ = kSubs * kSub;
  static_assert(kQ <= 2 * kWindow, "a Q tile fits its warpgroup's windows");
  // Exact: ids of a row's candidates that are to be scored again.
  static constexpr int kPending = EXACT ? 16 : 0, kPendingBytes = kSelect * kPending * 2;
  static constexpr int kSmem = kTiles * 2 * kWindow + kStages * kKb + kPendingBytes + 1024 + 512;
  // TMEM columns of a tile: scores [0, 64), queries [64, 64 + D / 2)
  static constexpr int kTileCols = 128, kQCol = kStepBlocks;
};

struct Bars {
  uint64_t q_here[2], q_full[2], kb_full[4], kb_empty[4], s_full[2], s_free[2], drain;
  uint32_t tmem_base;
  int abort;
};

// Sorted (descending) register list of the L best keys seen so far, t[0, L).
template <int L, int N>
__device__ __forceinline__ void list_offer(uint32_t (&t)[N], uint32_t x) {
#pragma unroll
  for (int i = 0; i < L; ++i) {
    const uint32_t hi = max(t[i], x);
    x = min(t[i], x);
    t[i] = hi;
  }
}

// Batcher's odd-even merge sort, descending; N a power of two.
template <int N, typename V>
__device__ __forceinline__ void sort_descending(V (&a)[N]) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1)
#pragma unroll
    for (int k = p; k >= 1; k >>= 1)
#pragma unroll
      for (int j = k % p; j + k < N; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
            const V x = a[i + j], y = a[i + j + k];
            a[i + j] = max(x, y);
            a[i + j + k] = min(x, y);
          }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

template <typename T> __device__ __forceinline__ uint32_t round16(float a);
template <> __device__ __forceinline__ uint32_t round16<__nv_bfloat16>(float a) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a));
}
template <> __device__ __forceinline__ uint32_t round16<__half>(float a) {
  return (uint32_t)__half_as_ushort(__float2half_rn(a));
}
template <typename T> __device__ __forceinline__ float widen16(uint32_t bits);
template <> __device__ __forceinline__ float widen16<__nv_bfloat16>(uint32_t bits) { return __uint_as_float(bits << 16); }
template <> __device__ __forceinline__ float widen16<__half>(uint32_t bits) {
  return __half2float(__ushort_as_half((unsigned short)bits));
}

// Bits of a score rounded to T, sign-extended, and the low half -> sortable key; never 0 for a real
// candidate (the low half is 0xFFFF - id with id <= 0xFFFE). The high half counts the steps of T from
// zero, which both zeros are, with 0x8000 added.
__device__ __forceinline__ uint32_t make_key(int b, uint32_t low) {
  const uint32_t mono = b < 0 ? (uint32_t)-b : (uint32_t)b + 0x8000u;
  return (mono << 16) | low;
}
// The other way, from the high half of a key (at least that of -infinity) to the bits of T.
__device__ __forceinline__ uint32_t bits_of(uint32_t mono) { return mono & 0x8000u ? mono & 0x7FFFu : 0x10000u - mono; }
template <typename T> constexpr uint32_t kLowest = std::is_same<T, __nv_bfloat16>::value ? 0x80u : 0x400u;   // of -infinity

// What a score has to exceed to be ranked. The plain gate compares scores rounded to T, two at a time,
// with a number of T; the exact one float32 scores with a bar that err has been taken off.
template <typename T, bool EXACT> struct Bar;
template <typename T> struct Bar<T, false> {
  uint32_t mono = kLowest<T>, pair = 0x10001u * bits_of(kLowest<T>);
  __device__ __forceinline__ void raise(uint32_t m) { mono = max(mono, m); pair = 0x10001u * bits_of(mono); }
  // to a score that the list's last entry has, or to the step below one that L candidates reach
  __device__ __forceinline__ void raise_to_entry(uint32_t key, float) { raise(key >> 16); }
  __device__ __forceinline__ void raise_below(float reached, float) { raise((make_key((int)(short)round16<T>(reached), 0u) >> 16) - 1u); }
};
template <typename T> struct Bar<T, true> {
  float bar = -INFINITY;
  __device__ __forceinline__ void raise(uint32_t mono, float err) { bar = fmaxf(bar, widen16<T>(bits_of(max(mono, kLowest<T>))) - err); }
  __device__ __forceinline__ void raise_to_entry(uint32_t key, float err) { raise(key >> 16, err); }
  __device__ __forceinline__ void raise_below(float reached, float err) { raise((make_key((int)(short)round16<T>(reached - err), 0u) >> 16) - 1u, err); }
};

// Which unit a CTA takes in its `round`-th turn: heaviest units first, alternating
// direction, so that no CTA collects the heaviest unit of every round.
__device__ __forceinline__ int unit_of(int round) {
  const int g = (int)gridDim.x, c = (int)blockIdx.x;
  return round * g + ((round & 1) ? (g - 1 - c) : c);
}

// Blocks are 128 keys, or (exact) a power of two that divides 128.
template <bool EXACT> __device__ __forceinline__ int block_of(int row, const moba_b200_problem& p) {
  return EXACT ? row >> (31 - __clz(p.block_size)) : row / kTile;
}

// The bounding pass looks at 256 candidates only: they give a bar that few scores of another
// step pass, and scoring a long row of block means twice would cost more tensor-core time than the
// tighter bar saves: us for 1024 and 4096 blocks, head_dim 128: 2 steps 1070 and 337, 4 steps 1068 and 332, 6 1088
// and 342, 8 1141 and 383. Two steps are the first and two the last that a unit fills: scores that rise with
// the position pass a bar of the first blocks one and all. us with all four at the front, and so (the last step itself,
// half empty, makes a worse bar of independent scores), for scores of deviation 0.7 (1.4 in blocks of 32) that rise
// over the sequence by                                               0            6            32
//   131072 queries x 4 heads of 64, 1024 blocks                   125  126     250  122     425  136
//   262144 x 4 of 64, 2048 blocks                                 370  372     625  343    1938  359
//   65536 x 4 of 64, 512 blocks, 12 each (exact)                  132  133     213  144     272  154
//   16384 x 4 of 64, 512 blocks of 32 (exact)                      32   33      51   36     143   49
constexpr int kBoundSteps = 4;
// Neighbouring tiles of one (sequence, query head); warpgroup w has tile `tile0 + w`.
struct Unit {
  int tile0, tiles, seq, hq, n_steps, bos, len;   // (tile0 may be negative: tiles before the first do not exist)
  int own_hi;               // own block of the unit's last row
  int n_lo, s_hi0;          // steps [0, n_lo) and [s_hi0, ...) of the Kbar row are visited
  int n_first;              // steps the bounding pass scores before the ranking pass scores all
  // 64 blocks of the Kbar row: the s-th that the unit scores, and what its `step` scores. The bounding pass takes
  // two from the front, then the last two before the last. (From the sum `steps` alone: with n_steps beside it the
  // select warps spill up to 48 bytes more, 1 to 8 % of the exact gate.)
  __device__ __forceinline__ int blocks_at(int s) const { return (s < n_lo ? s : s_hi0 + (s - n_lo)) * kStepBlocks; }
  __device__ __forceinline__ int bound_step(int step, int steps) const {
    return step < kBoundSteps / 2 ? step : max(step, steps + step - (1 + kBoundSteps) - n_first);
  }
  __device__ __forceinline__ int blocks_of(int step) const {
    return blocks_at(step >= n_first ? step - n_first : bound_step(step, steps()));
  }
  // a unit takes n_first + n_steps steps: the bounding pass, then the ranking pass
  __device__ __forceinline__ int steps() const { return n_first + n_steps; }
  __device__ __forceinline__ bool has(int w) const { return w < tiles && tile0 + w >= 0; }
};
// So few candidates are ranked faster than a pass of their own takes: 8192 x 4, 64 blocks 12.8 us with the line at
// 32, 11.1 at 16, 10.9 at 8; 16 sequences of 300 to 9000 tokens 149, 144, 144.
constexpr int kUnboundedBlocks = 16;
template <bool EXACT>
__device__ __forceinline__ bool load_unit(Unit& u, int idx, const moba_b200_problem& p, const int32_t* cu, int tiles, int n_groups) {
  const int ny = p.n_seq * p.q_heads;
  const int y = idx % ny;
  u.seq = y / p.q_heads; u.hq = y % p.q_heads;
  const SeqSpan sp = seq_span(cu, p.packed, u.seq, p.tokens);
  u.bos = sp.bos; u.len = sp.len; u.tiles = tiles;
  // groups of tiles counted from the end of the sequence, long ones first
  const int nt = (sp.len + kTile - 1) / kTile, from_end = (nt + tiles - 1) / tiles - (n_groups - 1 - idx / ny);
  u.tile0 = nt - tiles * from_end;
  if (from_end <= 0) return false;
  u.own_hi = block_of<EXACT>(min((u.tile0 + tiles) * kTile, sp.len) - 1, p);
  // Candidates are blocks [0, own); with a candidate window only [0, sinks) and
  // [own - window, own), so only the steps that hold some of those are scored.
  const int total = (p.take > 0) ? (u.own_hi + kStepBlocks - 1) / kStepBlocks : 0;
  if (p.gate_window <= 0) {
    u.n_lo = total; u.s_hi0 = total;
  } else {
    const int recent0 = max(0, block_of<EXACT>(max(0, u.tile0) * kTile, p) - p.gate_window);   // first block of the recent window
    u.n_lo = min(total, (min(p.gate_sinks, recent0) + kStepBlocks - 1) / kStepBlocks);
    u.s_hi0 = max(u.n_lo, recent0 / kStepBlocks);
  }
  u.n_steps = u.n_lo + (total - u.s_hi0);
  u.n_first = u.own_hi > (EXACT ? p.take : kUnboundedBlocks) ? min(u.n_steps, kBoundSteps) : 0;
  return true;
}

// Exact scores of four (query, block) pairs by a warp, eight lanes a pair: the products of two 16-bit numbers
// and their float64 sum carry no error, the result is rounded to float32 as everywhere in the gate.
template <int D, typename T>
__device__ __forceinline__ float exact_score(const T* q_row, const T* kbar_row, int lane8) {
  double acc = 0.0;
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    const uint4 a = *(reinterpret_cast<const uint4*>(q_row) + i * 8 + lane8), b = __ldg(reinterpret_cast<const uint4*>(kbar_row) + i * 8 + lane8);
    const T *x = reinterpret_cast<const T*>(&a), *y = reinterpret_cast<const T*>(&b);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc = fma((double)Elem<T>::to_f(x[e]), (double)Elem<T>::to_f(y[e]), acc);
  }
#pragma unroll
  for (int o = 4; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return (float)acc;
}

// Bound of |tensor-core sum - exact score| for one query and the blocks [0, n_cand) of its KV row,
// whose lengths are `norms`; the warp's lanes share the blocks. D / 16 accumulation steps of 17
// addends, each cut at 2^-23 of the largest: D 17/16 2^-23 of a quantity that |q| |kbar| bounds;
// doubled, and the smallest normal number for what is lost below it. Infinite where that cannot be
// said: an infinity or NaN in the query, an infinity in a block mean, squares whose sum does not fit
// float32. A NaN in a block mean needs no bound, its score is NaN either way; nor does a query of zeros
// (`any`: the query's bits or-ed together; `square`: its squared length).
template <int D>
__device__ __forceinline__ float score_error(uint32_t any, float square, const float* norms, int n_cand, int lane) {
  float longest = 0.f;
#pragma unroll 4
  for (int i = lane; i < n_cand; i += 32) longest = fmaxf(longest, __ldg(norms + i));
#pragma unroll
  for (int o = 16; o; o >>= 1) longest = fmaxf(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  if ((any & 0x7fff7fffu) == 0u || longest == 0.f) return 0.f;
  if (!(square >= 1e-30f && square <= 1e30f)) return INFINITY;
  const float e = sqrtf(square) * longest * ((float)D * (17.f / 8.f) * 1.1920929e-7f);
  return e < INFINITY ? e + 1.17549435e-38f : INFINITY;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
template <typename T> __device__ __forceinline__ uint32_t pack2(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(uint32_t a, uint32_t b) {
  const __half2 v = __floats2half2_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <typename T> __device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t sub2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
template <> __device__ __forceinline__ uint32_t sub2<__half>(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// The signs of four 16-bit numbers, each over a byte.
__device__ __forceinline__ uint32_t signs4(uint32_t lo, uint32_t hi) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, 0xFDB9;" : "=r"(d) : "r"(lo), "r"(hi));
  return d;
}
// The wait for a load that was issued some time ago: the registers are not to be looked at before.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :: "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[32], uint32_t (&b)[32]) {
  tmem_ld_wait(a);
  tmem_ld_wait(b);
}
// Bit k: block g0 + k is a candidate of a query whose own block is `own` (gate_candidate).
__device__ __forceinline__ uint32_t below32(int n) { return n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u; }
__device__ __forceinline__ uint32_t candidates32(const moba_b200_problem& p, int g0, int own) {
  uint32_t open = below32(own - g0);
  if (p.gate_window > 0) open &= below32(p.gate_sinks - g0) | ~below32(own - p.gate_window - g0);
  return open;
}

template <int D, typename T, int L, bool EXACT>
__global__ void __launch_bounds__(GateCfg<D, EXACT>::kThreads, GateCfg<D, EXACT>::kCtas)
gate_sm100_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kb_map,
                  const int32_t* __restrict__ cu, int32_t* __restrict__ block_idx, float* __restrict__ lse_fill,
                  moba_b200_problem p, int tiles, int n_groups, int n_units, unsigned* error_word,
                  const T* __restrict__ q, const T* __restrict__ kbar, const float* __restrict__ norms) {
  using Cfg = GateCfg<D, EXACT>;
  constexpr int NT = Cfg::kTiles, NST = Cfg::kStages;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* sWin = smem;                                 // two windows of scores per thread, by warpgroups
  unsigned char* sKb = sWin + NT * 2 * Cfg::kWindow;
  Bars* bars = reinterpret_cast<Bars*>(sKb + NST * Cfg::kKb + Cfg::kPendingBytes);
  static_assert(sizeof(Bars) <= 512, "barrier block outgrew its reservation");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.q_heads / p.kv_heads;
  const int take = p.take;
#ifdef MOBA_WAIT_STATS
  __shared__ unsigned long long wait_stats[32];
  if (threadIdx.x < 32) wait_stats[threadIdx.x] = 0;
  const long long kernel_t0 = clock64();
  const WaitCtx wc{&bars->abort, error_word, wait_stats};
#else
  const WaitCtx wc{&bars->abort, error_word};
#endif

  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) { mbar_init(&bars->kb_full[i], 1); mbar_init(&bars->kb_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars->q_here[i], 1); mbar_init(&bars->q_full[i], 4); mbar_init(&bars->s_full[i], 1); mbar_init(&bars->s_free[i], 4); }
    mbar_init(&bars->drain, 1);
    bars->abort = 0;
    fence_barrier_init();
  }
  if (warp == Cfg::kMmaWarp) tmem_alloc(&bars->tmem_base, NT * Cfg::kTileCols);
  if (warp == Cfg::kLoadWarp && lane == 0) { tma_prefetch_desc(&q_map); tma_prefetch_desc(&kb_map); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem = bars->tmem_base;

  // Every role walks the same units and the same steps of each (Unit::steps). Kbar stages go round by
  // the steps of the CTA, a tile's score columns are used once a step of the units it has a tile in.
  if (warp < Cfg::kMmaWarp) {
    // ================================ select ================================
    const int wg = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t tbuf = tmem + ((uint32_t)((warp & 3) * 32) << 16) + wg * Cfg::kTileCols;
    // This thread's windows: piece j of window w at win0 + w * kWindow + j * kPiece.
    constexpr uint32_t kPiece = Cfg::kPiece;
    unsigned char* sQ = sWin + wg * 2 * Cfg::kWindow;
    const uint32_t win0 = smem_u32(sQ) + (uint32_t)r * 16u;
    uint32_t loads = 0;                                         // Q tiles of this warpgroup so far
    uint32_t gc = 0;                                            // steps of this warpgroup so far
    PHASE_CLOCK(ph);
    for (int round = 0; round * (int)gridDim.x < n_units; ++round) {
      const int ui = unit_of(round);
      if (ui >= n_units) continue;
      Unit u;
      if (!load_unit<EXACT>(u, ui, p, cu, tiles, n_groups) || !u.has(wg)) continue;
      const int row0 = (u.tile0 + wg) * kTile;
      const int own_lo = block_of<EXACT>(row0, p);              // own blocks of the tile's first and last row
      const int own_hi = block_of<EXACT>(min(row0 + kTile, u.len) - 1, p);
      const int own = EXACT ? block_of<EXACT>(min(row0 + r, u.len - 1), p) : own_lo;
      const T* q_row = q + ((size_t)(p.packed ? u.bos : (size_t)u.seq * p.tokens) + min(row0 + r, u.len - 1)) * ((size_t)p.q_heads * D) + (size_t)u.hq * D;
      const int steps = u.steps();
      float err = 0.f;                                          // EXACT: bound of |tensor-core sum - exact score|
      if (steps > 0) {
        // ---- the tile's queries, a row per thread, into TMEM: operand A of the scores. They come through
        // the windows, which every warp is done with. ----
        fence_proxy_async();
        __syncwarp();                                           // named barriers count whole warps
        asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");
        if (r == 0) {
          mbar_expect_tx(&bars->q_here[wg], Cfg::kQ);
          for (int s = 0; s < Cfg::kSubs; ++s)
            tma_load_3d(sQ + s * kSub, &q_map, &bars->q_here[wg], s * 64, u.hq, (p.packed ? u.bos : u.seq * p.tokens) + row0);
        }
        mbar_wait(&bars->q_here[wg], loads & 1u, wc, 8);
        ++loads;
        uint32_t any = 0u;
        float square = 0.f;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 x = *reinterpret_cast<const uint4*>(sQ + (c >> 1) * kSub + swz128(r, (c & 1) * 4 + i));
            w[i * 4] = x.x; w[i * 4 + 1] = x.y; w[i * 4 + 2] = x.z; w[i * 4 + 3] = x.w;
          }
          if constexpr (EXACT) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float lo = widen16<T>(w[i] & 0xffffu), hi = widen16<T>(w[i] >> 16);
              any |= w[i];
              square = fmaf(hi, hi, fmaf(lo, lo, square));
            }
          }
          tmem_st16(tbuf + Cfg::kQCol + c * 16, w);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(&bars->q_full[wg]);
        __syncwarp();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");   // the windows may be written
        if constexpr (EXACT) {
          err = score_error<D>(any, square, norms + ((size_t)u.seq * p.kv_heads + u.hq / group) * p.num_blocks, own_hi, lane);
          if (row0 + r >= u.len) err = 0.f;
        }
      }
      // Bounding pass: the maxima of the column subsets. Ranking pass: the row's list, best[0, L).
      uint32_t best[kSubsets];
#pragma unroll
      for (int e = 0; e < kSubsets; ++e) best[e] = u.n_first > 0 ? 0xff800000u : 0u;   // -inf; 0 sorts below every real key
      Bar<T, EXACT> bar;
      // Scores that passed and are not ranked yet, a bit per column of a window. `hi` and `lo` are of the
      // window at `at0`, whose first column has id 0xFFFF - id0; `hi1` and `lo1` of the newest.
      uint32_t hi = 0, lo = 0, at0 = win0, id0 = 0, hi1 = 0, lo1 = 0, at1 = win0, id1 = 0;
      // EXACT: candidates whose rounding depends on the sum's error wait here, by id, and are scored again in
      // float64 for the whole warp at once, at the end of the unit or when a lane has no room for another. (Scored
      // as they were popped they were most of the kernel, a memory latency each: 65536 x 4 heads, 12 of 512 blocks,
      // 163 us, 137 so; 2 x 8192 x 4 of 128, blocks of 64, 60 and 42. Telling those that are in or out whichever way
      // they round first, so that a sixth is left, costs what it saves: 142 and 40.) The order in which keys get
      // to the list does not matter.
      uint32_t pending = 0;
      const uint32_t pend0 = smem_u32(sKb + NST * Cfg::kKb) + threadIdx.x * 2u;
      auto resolve = [&]() {
        while (const unsigned all = __ballot_sync(0xffffffffu, pending != 0u)) {
          uint32_t id = 0;                                      // of this lane's last
          if (pending != 0u) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(id) : "r"(pend0 + (pending - 1u) * (Cfg::kSelect * 2u)));
          float exact = -INFINITY;
          const size_t kv_row = (size_t)u.seq * p.kv_heads + u.hq / group;
          for (unsigned open = all; open != 0u;) {              // eight lanes a candidate, two candidates each
            float got[2];
            unsigned mine[2] = {0u, 0u};                        // the lanes that the two rounds of four take
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              int who = -1;
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const int next = __ffs((int)open) - 1;
                if ((lane >> 3) == g) who = next;
                if (next >= 0) mine[j] |= 1u << next;
                open &= open - 1u;
              }
              const int from = max(who, 0);
              const uint32_t blk = __shfl_sync(0xffffffffu, id, from);
              const T* qr = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(q_row), from));
              got[j] = exact_score<D, T>(qr, kbar + (kv_row * p.num_blocks + blk) * (size_t)D, lane & 7);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {                       // the n-th lane taken finds its score in the n-th group
              const float x = __shfl_sync(0xffffffffu, got[j], (__popc(mine[j] & ((1u << lane) - 1u)) & 3) * 8);
              if (mine[j] >> lane & 1u) exact = x;
            }
          }
          // (a score taken again in float64 may be one that is never selected)
          list_offer<L>(best, pending != 0u && exact > -INFINITY ? make_key((int)(short)round16<T>(exact), 0xFFFFu - id) : 0u);
          if (pending != 0u) --pending;
        }
      };
      // Every lane offers one of its scores to its list, n times.
      auto pop = [&](uint32_t n) {
        PHASE_CLOCK(fl);
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i) {
          const bool top = !EXACT && hi != 0u;
          const uint32_t bits = top ? hi : lo;
          const bool some = bits != 0u;
          uint32_t k;                                           // a column (31 if there is none)
          asm("bfind.u32 %0, %1;" : "=r"(k) : "r"(bits));
          k &= 31u;
          const uint32_t rest = bits & ~(1u << k);
          uint32_t key;
          if constexpr (!EXACT) {
            if (top) hi = rest; else lo = rest;
            const uint32_t c = top ? k + 32u : k;
            int b;
            asm volatile("ld.shared.s16 %0, [%1];" : "=r"(b) : "r"(at0 + (k & 7u) * kPiece + (c >> 3) * 2u));
            key = some ? make_key(b, id0 - c) : 0u;
          } else {
            lo = rest;
            float s;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(s) : "r"(at0 + (k >> 2) * kPiece + (k & 3u) * 4u));
            const uint32_t pair = pack2<T>(__float_as_uint(s - err), __float_as_uint(s + err));
            const bool unsure = some && (pair >> 16) != (pair & 0xffffu);
            if (unsure) asm volatile("st.shared.u16 [%0], %1;" ::"r"(pend0 + pending * (Cfg::kSelect * 2u)), "h"((short)(0xFFFFu - (id0 - k))) : "memory");
            pending += unsure ? 1u : 0u;
            key = some && !unsure ? make_key((int)(short)round16<T>(s), id0 - k) : 0u;
          }
          list_offer<L>(best, key);
          if ((hi | lo) == 0u) { hi = hi1; lo = lo1; hi1 = 0u; lo1 = 0u; at0 = at1; id0 = id1; }
          if (EXACT && __any_sync(0xffffffffu, pending == Cfg::kPending)) resolve();
        }
        if (n != 0u) bar.raise_to_entry(best[L - 1], err);
        PHASE_ADD(wc, 4, fl);                                   // (also counted in its phase)
      };
      // Which of 32 scores pass; they go into the free window, at1, as its half `h`. The differences are
      // negative where the score exceeds the bar (also from -infinity), and a NaN has no sign.
      auto test = [&](const uint32_t* v, const uint32_t* w) -> uint2 {
        uint32_t part[4] = {0u, 0u, 0u, 0u};
        if constexpr (!EXACT) {
          // Columns i, i + 8, i + 16 and i + 24 of either half in a piece: their signs are bit i of the masks' bytes.
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t a = pack2<T>(v[i], v[8 + i]), b = pack2<T>(v[16 + i], v[24 + i]);
            const uint32_t c = pack2<T>(w[i], w[8 + i]), d = pack2<T>(w[16 + i], w[24 + i]);
            part[i & 1] |= signs4(sub2<T>(bar.pair, a), sub2<T>(bar.pair, b)) & (0x01010101u << i);
            part[2 + (i & 1)] |= signs4(sub2<T>(bar.pair, c), sub2<T>(bar.pair, d)) & (0x01010101u << i);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at1 + i * kPiece), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
          }
          return make_uint2(part[0] | part[1], part[2] | part[3]);
        } else {
          const float2 bar2 = {bar.bar, bar.bar}, minus = {-1.f, -1.f};
#pragma unroll
          for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int k = 6; k >= 0; k -= 2) {
              const float2 d = fma2(make_float2(__uint_as_float(v[h * 8 + k]), __uint_as_float(v[h * 8 + k + 1])), minus, bar2);
              part[h] = __funnelshift_l(__float_as_uint(d.y), part[h], 1);
              part[h] = __funnelshift_l(__float_as_uint(d.x), part[h], 1);
            }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at1 + j * kPiece), "r"(v[j * 4]), "r"(v[j * 4 + 1]),
                         "r"(v[j * 4 + 2]), "r"(v[j * 4 + 3]) : "memory");
          return make_uint2(part[0] | part[1] << 8 | part[2] << 16 | part[3] << 24, 0u);
        }
      };
      // After the scores of the window that begins with `block` have been tested: ranks what is left of the
      // window before, and more where lanes have time.
      auto rank = [&](uint32_t m_lo, uint32_t m_hi, int block) {
        const uint32_t left = __popc(hi) + __popc(lo);
        id1 = 0xFFFFu - (uint32_t)block;
        if (left == 0u) { hi = m_hi; lo = m_lo; at0 = at1; id0 = id1; } else { hi1 = m_hi; lo1 = m_lo; }
        pop(__reduce_max_sync(0xffffffffu, left));
        at1 = win0 + (win0 + Cfg::kWindow - at1);               // the other window
      };
      PHASE_ADD(wc, 1, ph);                                     // unit set-up
      bool run = true;                                          // a wait gave up: rank nothing unseen
      uint32_t v[32], w[32];
      // Candidates among the 32 blocks from g0 on. Most windows are candidates from end to end.
      auto open_of = [&](int g0) { return run ? (g0 + 32 <= own_lo && p.gate_window <= 0 ? 0xffffffffu : candidates32(p, g0, own)) : 0u; };
      auto wait_scores = [&]() {
        run = mbar_wait(&bars->s_full[wg], gc & 1u, wc, 9) && run;
        tc_fence_after();
      };
      auto free_scores = [&]() {                                // they are in registers
        tc_fence_before();
        mbar_arrive_warp(&bars->s_free[wg]);
        ++gc;
      };
      auto unbounded = [&]() {                                  // EXACT, no bound: every candidate is to be scored again
        if constexpr (EXACT) {
          if (__any_sync(0xffffffffu, err == INFINITY)) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (err == INFINITY) v[k] = 0x7f800000u;          // +inf passes the entry test
          }
        }
      };
      // ---- bounding pass ----
#pragma unroll 1
      for (int step = 0; step < u.n_first; ++step) {
        const int c0 = u.blocks_at(u.bound_step(step, steps));
        wait_scores();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_ld32(tbuf + h * 32, v);
          tmem_ld_wait(v);
          if (h == 1) free_scores();
          const uint32_t open = open_of(c0 + h * 32);
          unbounded();
          if (__any_sync(0xffffffffu, open != 0xffffffffu)) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (!(open >> k & 1u)) v[k] = 0xff800000u;        // -inf
          }
#pragma unroll
          for (int e = 0; e < kSubsets; ++e)
            best[e] = __float_as_uint(max3(__uint_as_float(best[e]), __uint_as_float(v[e]), __uint_as_float(v[kSubsets + e])));
        }
      }
      if (u.n_first > 0) {
        // The L-th largest of the subset maxima: at least L candidates reach it. Of two descending
        // lists a and b the L-th largest is the least of max(a[i], b[L - 1 - i]).
        float a[8], b[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) { a[e] = __uint_as_float(best[e]); b[e] = __uint_as_float(best[8 + e]); }
        sort_descending(a);
        sort_descending(b);
        float reached = INFINITY;
#pragma unroll
        for (int i = 0; i < L; ++i) {
          const int j = L - 1 - i;
          reached = fminf(reached, i >= 8 ? b[j & 7] : j >= 8 ? a[i & 7] : fmaxf(a[i & 7], b[j & 7]));
        }
        bar.raise_below(reached, err);
#pragma unroll
        for (int e = 0; e < kSubsets; ++e) best[e] = 0u;
      }
      PHASE_ADD(wc, 2, ph);
      // ---- ranking pass ----
#pragma unroll 1
      for (int step = u.n_first; step < steps; ++step) {
        const int g0 = u.blocks_at(step - u.n_first);
        wait_scores();
        tmem_ld32(tbuf, v);
        if constexpr (!EXACT) {
          tmem_ld32(tbuf + 32, w);
          tmem_ld_wait(v, w);
          free_scores();
          const uint2 m = test(v, w);
          rank(m.x & open_of(g0), m.y & open_of(g0 + 32), g0);
        } else {
          tmem_ld_wait(v);
          unbounded();
          const uint32_t m = test(v, v).x & open_of(g0);
          tmem_ld32(tbuf + 32, v);                              // on its way while the first half is ranked
          rank(m, 0u, g0);
          tmem_ld_wait(v);
          free_scores();
          unbounded();
          rank(test(v, v).x & open_of(g0 + 32), 0u, g0 + 32);
        }
        PHASE_ADD(wc, 3, ph);                                   // loads, masks, pops
      }
      pop(__reduce_max_sync(0xffffffffu, (uint32_t)(__popc(hi) + __popc(lo))));
      if constexpr (EXACT) resolve();
      if (row0 + r < u.len) {
        // ---- emit: the best `take` ids plus the own block, ascending, -1 padded ----
        constexpr int NS = L <= 8 ? 8 : 16;
        uint32_t low[NS];                                       // 0xFFFF - id, largest first; 0: none
        int ids[NS], kept = 0;
#pragma unroll
        for (int e = 0; e < NS; ++e) {
          low[e] = e < L && e < take ? best[e] & 0xFFFFu : 0u;
          kept += low[e] != 0u ? 1 : 0;
        }
        sort_descending(low);
#pragma unroll
        for (int e = 0; e < NS; ++e) ids[e] = (int)(0xFFFFu - low[e]);
        const size_t b = p.packed ? 0 : (size_t)u.seq;
        const size_t dst_at = ((b * p.q_heads + u.hq) * p.tokens + u.bos + row0 + r) * (size_t)p.slots;
        int32_t* dst = block_idx + dst_at;
        const int listed = kept + (p.always_current ? 1 : 0);
        if (p.slots == 8 && (reinterpret_cast<uintptr_t>(block_idx) & 15) == 0) {
          int4 o[2];
          int* oi = reinterpret_cast<int*>(o);
#pragma unroll
          for (int e = 0; e < 8; ++e) oi[e] = e < kept ? ids[e] : (e < listed ? own : -1);   // the own block is past every candidate
          reinterpret_cast<int4*>(dst)[0] = o[0];
          reinterpret_cast<int4*>(dst)[1] = o[1];
        } else {
#pragma unroll
          for (int e = 0; e < NS; ++e)
            if (e < kept) dst[e] = ids[e];
          if (p.always_current) dst[kept] = own;
          for (int e = listed; e < p.slots; ++e) dst[e] = -1;
        }
        if (lse_fill != nullptr)
          for (int e = listed; e < p.slots; ++e) lse_fill[dst_at + e] = -INFINITY;   // the slot's partial will not be written
      }
      PHASE_ADD(wc, 5, ph);                                     // last pops, emit
    }
    // No load may be in flight into this CTA's shared memory when it exits.
    if (loads >= 1) mbar_wait_quiet(&bars->q_here[wg], (loads - 1) & 1u);
  } else if (warp == Cfg::kMmaWarp) {
    // The whole warp walks the steps, so that descriptors stay in uniform registers, and one lane issues:
    // from a branch of one lane an MMA took some 120 clocks to issue, which bounded the kernel at head_dim 128.
    const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    const uint32_t idesc = make_idesc(0, 128, kStepBlocks, 0, 0) | (fmt << 7) | (fmt << 10);
    const uint64_t dKb = make_sdesc(smem_u32(sKb), 16, 1024);
    const bool issue = elect_one();
    uint32_t gc = 0, steps_of[NT] = {}, loads_of[NT] = {};      // steps of the CTA; steps and units of each tile
    for (int round = 0; round * (int)gridDim.x < n_units; ++round) {
      const int ui = unit_of(round);
      if (ui >= n_units) continue;
      Unit u;
      if (!load_unit<EXACT>(u, ui, p, cu, tiles, n_groups) || u.n_steps == 0) continue;
      for (int step = 0; step < u.steps(); ++step, ++gc) {
        const uint64_t dK = sdesc_at(dKb, (gc % NST) * Cfg::kKb);
        mbar_wait(&bars->kb_full[gc % NST], (gc / NST) & 1, wc, 10);
#pragma unroll
        for (int w = 0; w < NT; ++w) {
          if (!u.has(w)) continue;
          if (step == 0) { mbar_wait(&bars->q_full[w], loads_of[w] & 1, wc, 11); ++loads_of[w]; }
          if (steps_of[w] >= 1) mbar_wait(&bars->s_free[w], (steps_of[w] - 1) & 1, wc, 12);
          ++steps_of[w];
          tc_fence_after();
          __syncwarp();
          if (issue) {
            const uint32_t ts = tmem + w * Cfg::kTileCols;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
              umma_f16_ts(ts, ts + Cfg::kQCol + ks * 8, sdesc_at(dK, (ks >> 2) * (kStepBlocks * 128) + (ks & 3) * 32), idesc, ks > 0);
            umma_commit(&bars->s_full[w]);
          }
          __syncwarp();
        }
        if (issue) umma_commit(&bars->kb_empty[gc % NST]);
      }
    }
    // Every MMA has completed before the CTA lets go of its TMEM, also on the way out of
    // a run that gave up on a wait.
    if (issue) {
      umma_commit(&bars->drain);
      mbar_wait_quiet(&bars->drain, 0);
    }
    __syncwarp();
  } else {
    if (lane == 0) {
      uint32_t gc = 0;
      for (int round = 0; round * (int)gridDim.x < n_units && !*wc.abort; ++round) {   // no new loads once a wait gave up
        const int ui = unit_of(round);
        if (ui >= n_units) continue;
        Unit u;
        if (!load_unit<EXACT>(u, ui, p, cu, tiles, n_groups)) continue;
        const int kv_row = u.seq * p.kv_heads + u.hq / group;
        if (u.n_steps > 0) {                                    // its queries, as soon as the warpgroups have time, from the L2
          for (int w = 0; w < NT; ++w)
            for (int s = 0; u.has(w) && s < Cfg::kSubs; ++s)
              tma_prefetch_3d(&q_map, s * 64, u.hq, (p.packed ? u.bos : u.seq * p.tokens) + (u.tile0 + w) * kTile);
        }
        for (int step = 0; step < u.steps(); ++step, ++gc) {
          if (gc >= NST) mbar_wait(&bars->kb_empty[gc % NST], (gc / NST - 1) & 1, wc, 13);
          if (*wc.abort) break;
          mbar_expect_tx(&bars->kb_full[gc % NST], Cfg::kKb);
          for (int s = 0; s < Cfg::kSubs; ++s)
            tma_load_3d(sKb + (gc % NST) * Cfg::kKb + s * (kStepBlocks * 128), &kb_map, &bars->kb_full[gc % NST], s * 64, u.blocks_of(step), kv_row);
        }
      }
      // No load may be in flight into this CTA's shared memory when it exits.
      for (uint32_t k = 1; k <= NST && k <= gc; ++k) mbar_wait_quiet(&bars->kb_full[(gc - k) % NST], ((gc - k) / NST) & 1);
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kMmaWarp) tmem_dealloc(tmem, NT * Cfg::kTileCols);
#ifdef MOBA_WAIT_STATS
  if (threadIdx.x < 32 && blockIdx.x < 148) {
    unsigned long long* out = reinterpret_cast<unsigned long long*>(error_word + 64) + (size_t)blockIdx.x * 32;
    out[threadIdx.x] = threadIdx.x == 31 ? (unsigned long long)(clock64() - kernel_t0) : wait_stats[threadIdx.x];
  }
#endif
}


template <int D, typename T, int L, bool EXACT>
int launch_one(const moba_b200_problem& p, const CUtensorMap& qm, const CUtensorMap& km, const int32_t* cu,
               int32_t* block_idx, float* lse_fill, unsigned* err, const void* q, const void* kbar, const float* norms,
               cudaStream_t st) {
  using Cfg = GateCfg<D, EXACT>;
  auto kern = gate_sm100_kernel<D, T, L, EXACT>;
  static SmemLimit limit;
  if (int rc = raise_smem_limit(limit, (const void*)kern, Cfg::kSmem)) return rc;
  const int ctas = Cfg::kCtas * sm_count(), n_tiles = (p.max_seqlen + kTile - 1) / kTile;
  // Fewer tiles a unit where whole units would leave CTAs idle.
  int tiles = Cfg::kTiles;
  while (tiles > 1 && (long long)n_tiles * p.n_seq * p.q_heads <= (long long)ctas * (tiles / 2)) tiles /= 2;
  const int n_groups = (n_tiles + tiles - 1) / tiles;
  const long long n_units = (long long)n_groups * p.n_seq * p.q_heads;
  const int grid = (int)(n_units < ctas ? n_units : ctas);
  MOBA_CUDA_OK(launch_chained(kern, grid, Cfg::kThreads, Cfg::kSmem, st, qm, km, cu, block_idx, lse_fill, p, tiles, n_groups,
                              (int)n_units, err, (const T*)q, (const T*)kbar, norms));
  return MOBA_B200_OK;
}

}  // namespace

bool gate_sm100_supported(const moba_b200_problem& p) {
  return (p.dtype == MOBA_B200_BF16 || p.dtype == MOBA_B200_F16) && p.block_size == 128 &&
         (p.head_dim == 64 || p.head_dim == 128) && p.take <= kMaxTake && p.slots <= kMaxTake + 1 &&
         p.num_blocks <= 0xFFFF &&
         (long long)p.batch * p.tokens < 0x7fffffffLL &&
         (long long)((p.max_seqlen + 127) / 128) * p.n_seq * p.q_heads < 0x7fffffffLL;
}

int encode_kbar_map_impl(CUtensorMap* out, const void* base, uint64_t kv_rows, uint64_t nb, uint64_t dim);

int launch_gate_sm100(const moba_b200_problem& p, const void* q, const void* kbar, const int32_t* cu,
                      int32_t* block_idx, float* lse_fill, cudaStream_t st) {
  KernelTimer timer__("gate_sm100_kernel", st);
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("gate: no device error word"); return MOBA_B200_ECUDA; }
  CUtensorMap qm, km;
  int rc = encode_rows_map(&qm, q, (uint64_t)p.batch * p.tokens, p.q_heads, p.head_dim, 128);
  if (rc) return rc;
  rc = encode_kbar_map_impl(&km, kbar, (uint64_t)p.n_seq * p.kv_heads, p.num_blocks, p.head_dim);
  if (rc) return rc;
  const bool bf = p.dtype == MOBA_B200_BF16;
#define GO(D, T) return (p.take <= 7) ? launch_one<D, T, 7, false>(p, qm, km, cu, block_idx, lse_fill, err, q, kbar, nullptr, st) \
                                      : launch_one<D, T, 8, false>(p, qm, km, cu, block_idx, lse_fill, err, q, kbar, nullptr, st)
  if (p.head_dim == 64) { if (bf) GO(64, __nv_bfloat16); else GO(64, __half); }
  if (bf) GO(128, __nv_bfloat16); else GO(128, __half);
#undef GO
}

// Block sizes that divide the tile of 128 queries. The list of a row lies in registers: up to 16 ranked blocks at
// head_dim 64 (100 bytes of spills), 12 at 128 (116 in float16; a list of 16 spills some 210 there and is not built, 13
// to 16 ranked blocks keep the portable kernel). A candidate window keeps it too.
bool gate_exact_sm100_supported(const moba_b200_problem& p) {
  return (p.dtype == MOBA_B200_BF16 || p.dtype == MOBA_B200_F16) && p.block_size >= 16 && kTile % p.block_size == 0 &&
         (p.head_dim == 64 || p.head_dim == 128) && p.take <= (p.head_dim == 64 ? 16 : 12) && p.gate_window == 0 &&
         p.num_blocks <= 0xFFFF && (long long)p.batch * p.tokens < 0x7fffffffLL &&
         (long long)p.n_seq * p.kv_heads * p.num_blocks < 0x7fffffffLL &&
         (long long)((p.max_seqlen + 127) / 128) * p.n_seq * p.q_heads < 0x7fffffffLL;
}

int launch_gate_exact_sm100(const moba_b200_problem& p, const void* q, const void* kbar, const float* norms, const int32_t* cu,
                            int32_t* block_idx, float* lse_fill, cudaStream_t st) {
  KernelTimer timer__("gate_exact_sm100_kernel", st);
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("gate: no device error word"); return MOBA_B200_ECUDA; }
  CUtensorMap qm, km;
  int rc = encode_rows_map(&qm, q, (uint64_t)p.batch * p.tokens, p.q_heads, p.head_dim, 128);
  if (rc) return rc;
  rc = encode_kbar_map_impl(&km, kbar, (uint64_t)p.n_seq * p.kv_heads, p.num_blocks, p.head_dim);
  if (rc) return rc;
  const bool bf = p.dtype == MOBA_B200_BF16;
#define GO(D, T)                                                                                                      \
  return p.take <= 8    ? launch_one<D, T, 8, true>(p, qm, km, cu, block_idx, lse_fill, err, q, kbar, norms, st)     \
         : p.take <= 12 ? launch_one<D, T, 12, true>(p, qm, km, cu, block_idx, lse_fill, err, q, kbar, norms, st)    \
                        : launch_one<D, T, D == 64 ? 16 : 12, true>(p, qm, km, cu, block_idx, lse_fill, err, q, kbar, norms, st)
  if (p.head_dim == 64) { if (bf) GO(64, __nv_bfloat16); else GO(64, __half); }
  if (bf) GO(128, __nv_bfloat16); else GO(128, __half);
#undef GO
}

}  // namespace moba
