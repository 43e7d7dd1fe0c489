// Gate scorer on tcgen05 tensor cores (bf16/f16, block_size 128, head_dim
// 64/128, at most 8 ranked blocks per query).
//
// Persistent CTAs (two per SM) walk the (128-query tile, sequence, query head)
// units, heaviest first, in alternating direction per round. With 128-token
// blocks a tile is exactly one block, so every row of a tile has the same
// candidates: the blocks before the tile's own. Roles:
//   loader (1 thread)  TMA: the unit's Q tile, then block-mean chunks of 128 blocks
//   mma    (1 thread)  S = Q Kbar^T (M128 N128 K=D) into one of two TMEM buffers: the first
//                      two chunks of the unit (bounding pass), then every chunk (ranking pass)
//   select (2 x 4 warps; warpgroup w takes columns [64 w, 64 w + 64) of every chunk)
//          tcgen05.ld, one row per thread. The first two chunks of a unit are scored twice.
//          The first pass only keeps, per row, the maxima of eight interleaved subsets
//          of the scores (half an instruction per score): the L-th largest of the two
//          warpgroups' sixteen is a score that at least L candidates reach, so nothing
//          below it can be selected. The second
//          pass tests every score against that bound with one compare and appends the
//          few that pass, by predicated stores, to a small per-thread buffer in shared
//          memory; the buffer is emptied into the row's sorted register list of L keys
//          whenever some lane of the warp is about to run out of room, which also
//          raises the bound to the score of the list's last entry (candidates arrive
//          in ascending block order, so an equal score never wins), and a step under it
//          for the row's other half. (A bar from one half's maxima let one score in seven
//          through at first, and emptying the buffers took most of the time: 131072 queries
//          x 4 heads 0.244 ms, with the bar of both halves 0.215; exact, 12 of 512 blocks:
//          0.50 and 0.30.) A key is the score
//          rounded to the input dtype and made monotone in the high half and
//          0xFFFF - block id in the low half, so "score descending, ties to the lower
//          id" is plain integer order. Scoring two chunks twice costs tensor-core time the
//          gate has to spare; ranking every score would cost issue slots it has not.
// At the end of a unit the two warpgroups' lists are merged and each thread emits
// its ids plus the own block, ascending, -1 padded.
//
// EXACT: the same kernel where the portable gate used to run (other block sizes that divide 128,
// more than eight ranked blocks): its selections are those of exact scores, bit for bit. The
// tensor-core sum is off by at most `err` (a bound from the lengths of the query and of the means of
// the unit's candidates), so the entry test is loosened by err, and a candidate whose rounding to the
// input dtype depends on that error is scored again in float64 by its whole warp before it is ranked:
// about one buffered candidate in forty where scores are large against err, every one near zero. A
// row without a finite bound (infinities, NaN, squares outside float32) has every candidate scored in
// float64. With blocks finer than the tile a row's candidates end at its own block.
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
constexpr int kMmaWarp = 8, kLoadWarp = 9;
constexpr int kThreads = 10 * 32;
constexpr int kMaxTake = 8;
constexpr int kEmpty = 0x7fffffff;

template <int D> struct GateCfg {
  static constexpr int kSubs = D / 64;
  static constexpr int kOperand = kSubs * kSub;
  // Per-thread buffer of scores that passed the entry test, in slots of 8 bytes, and how
  // many columns are tested between two checks for room. Two CTAs share an SM, which at
  // head_dim 128 leaves room for 7 slots only.
  static constexpr int kCap = tensor_core_plan(D).gate_slots;
  static constexpr int kStep = tensor_core_plan(D).gate_step;
  static constexpr int kBufBytes = kCap * kTile * 8;                       // per warpgroup
  static constexpr int kSmem = 3 * kOperand + 2 * kBufBytes + 1024 + 512 + 2 * kTile * 4;  // Q + two Kbar stages + buffers, bars
};

struct Bars {
  uint64_t q_full, q_free, kb_full[2], kb_empty[2], s_full[2], s_free[2], drain;
  uint32_t tmem_base;
  int abort;
};

// Sorted (descending) register list of the L best keys seen so far.
template <int L>
__device__ __forceinline__ void list_offer(uint32_t (&t)[L], uint32_t x) {
#pragma unroll
  for (int i = 0; i < L; ++i) {
    const uint32_t hi = max(t[i], x);
    x = min(t[i], x);
    t[i] = hi;
  }
}

// Descending order by Batcher's odd-even merge sort; N a power of two.
template <int N>
__device__ __forceinline__ void sort_descending(float (&a)[N]) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1)
#pragma unroll
    for (int k = p; k >= 1; k >>= 1)
#pragma unroll
      for (int j = k % p; j + k < N; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
            const float x = a[i + j], y = a[i + j + k];
            a[i + j] = fmaxf(x, y);
            a[i + j + k] = fminf(x, y);
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

// Score (rounded to T) and block id -> sortable key; never 0 for a real candidate
// (the low half of a key is 0xFFFF - id with id <= 0xFFFE). The high half counts the steps of T from
// zero, which both zeros are, with 0x8000 added.
template <typename T>
__device__ __forceinline__ uint32_t make_key(float score, uint32_t block) {
  const uint32_t b = round16<T>(score);
  const uint32_t mono = (b & 0x8000u) ? 0x10000u - b : b + 0x8000u;
  return (mono << 16) | (0xFFFFu - block);
}
// The score a candidate has to exceed to get past `key` (the list's last entry):
// -inf while the list has room.
template <typename T>
__device__ __forceinline__ float entry_bar(uint32_t key) {
  if (key == 0u) return -INFINITY;
  const uint32_t mono = key >> 16;
  const uint32_t b = (mono & 0x8000u) ? (mono & 0x7FFFu) : 0x10000u - mono;
  return widen16<T>(b);
}

// The largest score that is certainly below every score whose rounding to T is at least
// that of `key`: one step of T under it, widened back to float.
template <typename T>
__device__ __forceinline__ float one_step_below_key(uint32_t key) {
  const uint32_t mono = key >> 16;
  if (mono == 0u) return -INFINITY;
  return entry_bar<T>(((mono - 1u) << 16) | 1u);
}
template <typename T>
__device__ __forceinline__ float one_step_below(float m) {
  if (!(m > -INFINITY)) return -INFINITY;
  return one_step_below_key<T>(make_key<T>(m, 0u));
}

// Which unit a CTA takes in its `round`-th turn: heaviest units first, alternating
// direction, so that no CTA collects the heaviest unit of every round.
__device__ __forceinline__ int unit_of(int round) {
  const int g = (int)gridDim.x, c = (int)blockIdx.x;
  return round * g + ((round & 1) ? (g - 1 - c) : c);
}

struct Unit {
  int tile, seq, hq, row0, n_chunks, bos, len;
  int own_lo, own_hi;       // own blocks of the tile's first and last row (equal when a block is a tile)
  int n_lo, c_hi0;          // chunks [0, n_lo) and [c_hi0, ...) of the Kbar row are visited
  int n_first;              // chunks the bounding pass scores before the ranking pass scores all
  // chunk of the Kbar row that step `s` of a pass scores
  __device__ __forceinline__ int chunk_of(int s) const { return s < n_lo ? s : c_hi0 + (s - n_lo); }
  // a unit takes n_first + n_chunks steps: the bounding pass, then the ranking pass
  __device__ __forceinline__ int steps() const { return n_first + n_chunks; }
  __device__ __forceinline__ int chunk_of_step(int step) const { return chunk_of(step < n_first ? step : step - n_first); }
};
// The bounding pass looks at the first two chunks only: 256 candidates give a bar that about
// one score in ten of a later chunk passes until the first flush raises it, and scoring a long
// row of block means twice would cost more tensor-core time than the tighter bar saves.
constexpr int kBoundChunks = 2;
// So few candidates go through the buffers faster than through a pass of their own (16 sequences
// of 300 to 9000 tokens, 32 heads: 0.31 ms with a bounding pass for every unit, 0.27 without). In the
// exact gate, where what passes the bar may be scored again in float64, the pass pays as soon as a
// row has more candidates than it ranks: against a line at 32 blocks 2 x 2048 queries x 4 heads, 32
// blocks of 64 46 -> 36 us, 2 x 8192 x 4 of 128 120 -> 113, 65536 x 4, 512 blocks 315 -> 309; with
// the line at 64 207 and 324.
constexpr int kUnboundedBlocks = 32;
template <bool EXACT>
__device__ __forceinline__ bool load_unit(Unit& u, int idx, const moba_b200_problem& p, const int32_t* cu,
                                          int n_tiles) {
  const int ny = p.n_seq * p.q_heads;
  u.tile = n_tiles - 1 - idx / ny;                              // long tiles first
  const int y = idx % ny;
  u.seq = y / p.q_heads; u.hq = y % p.q_heads;
  const SeqSpan sp = seq_span(cu, p.packed, u.seq, p.tokens);
  u.bos = sp.bos; u.len = sp.len;
  u.row0 = u.tile * kTile;
  u.own_lo = u.row0 / p.block_size;
  u.own_hi = min(u.row0 + kTile - 1, sp.len - 1) / p.block_size;
  // Candidates are blocks [0, tile); with a candidate window only [0, sinks) and
  // [tile - window, tile), so only the chunks that hold some of those are scored.
  const int total = (p.take > 0) ? (u.own_hi + kTile - 1) / kTile : 0;
  if (p.gate_window <= 0) {
    u.n_lo = total; u.c_hi0 = total;
  } else {
    const int recent0 = max(0, u.own_lo - p.gate_window);         // first block of the recent window
    u.n_lo = min(total, (min(p.gate_sinks, recent0) + kTile - 1) / kTile);
    u.c_hi0 = max(u.n_lo, recent0 / kTile);
  }
  u.n_chunks = u.n_lo + (total - u.c_hi0);
  u.n_first = u.own_hi > (EXACT ? p.take : kUnboundedBlocks) ? min(u.n_chunks, kBoundChunks) : 0;
  return u.row0 < sp.len;
}

// Exact score of one (query, block) pair by a whole warp: the products of two 16-bit numbers and
// their float64 sum carry no error, the result is rounded to float32 as everywhere in the gate.
template <int D, typename T>
__device__ __forceinline__ float exact_score(const T* q_row, const T* kbar_row, int lane) {
  double acc = 0.0;
#pragma unroll
  for (int i = 0; i < D / 32; ++i)
    acc = fma((double)Elem<T>::to_f(q_row[i * 32 + lane]), (double)Elem<T>::to_f(kbar_row[i * 32 + lane]), acc);
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return (float)acc;
}

// Bound of |tensor-core sum - exact score| for one query and the blocks [0, n_cand) of its KV row,
// whose lengths are `norms`; the warp's lanes share the blocks. D / 16 accumulation steps of 17
// addends, each cut at 2^-23 of the largest: D 17/16 2^-23 of a quantity that |q| |kbar| bounds;
// doubled, and the smallest normal number for what is lost below it. Infinite where that cannot be
// said: an infinity or NaN in the query, an infinity in a block mean, squares whose sum does not fit
// float32. A NaN in a block mean needs no bound, its score is NaN either way; nor does a query of zeros.
template <int D, typename T>
__device__ __forceinline__ float score_error(const T* q_row, const float* norms, int n_cand, int lane) {
  float longest = 0.f;
#pragma unroll 4
  for (int i = lane; i < n_cand; i += 32) longest = fmaxf(longest, __ldg(norms + i));
#pragma unroll
  for (int o = 16; o; o >>= 1) longest = fmaxf(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  float square = 0.f;
  uint32_t any = 0u;
#pragma unroll 4
  for (int i = 0; i < D / 8; ++i) {
    const uint4 raw = *reinterpret_cast<const uint4*>(q_row + i * 8);
    any |= raw.x | raw.y | raw.z | raw.w;
    const T* x = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int e = 0; e < 8; ++e) square = fmaf(Elem<T>::to_f(x[e]), Elem<T>::to_f(x[e]), square);
  }
  if ((any & 0x7fff7fffu) == 0u || longest == 0.f) return 0.f;
  if (!(square >= 1e-30f && square <= 1e30f)) return INFINITY;
  const float e = sqrtf(square) * longest * ((float)D * (17.f / 8.f) * 1.1920929e-7f);
  return e < INFINITY ? e + 1.17549435e-38f : INFINITY;
}

template <int D, typename T, int L, bool EXACT>
__global__ void __launch_bounds__(kThreads, 2)
gate_sm100_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kb_map,
                  const int32_t* __restrict__ cu, int32_t* __restrict__ block_idx, float* __restrict__ lse_fill,
                  moba_b200_problem p, int n_tiles, int n_units, unsigned* error_word,
                  const T* __restrict__ q, const T* __restrict__ kbar, const float* __restrict__ norms) {
  using Cfg = GateCfg<D>;
  constexpr int CAP = Cfg::kCap, STEP = Cfg::kStep;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* sQ = smem;
  unsigned char* sKb = sQ + Cfg::kOperand;                    // two stages
  unsigned char* sBuf = sKb + 2 * Cfg::kOperand;              // two warpgroups' buffers
  Bars* bars = reinterpret_cast<Bars*>(sBuf + 2 * Cfg::kBufBytes + 2 * kTile * 4);   // (bars of the rows' lists in between)

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
    mbar_init(&bars->q_full, 1); mbar_init(&bars->q_free, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->kb_full[i], 1); mbar_init(&bars->kb_empty[i], 1);
      mbar_init(&bars->s_full[i], 1); mbar_init(&bars->s_free[i], 8);
    }
    mbar_init(&bars->drain, 1);
    bars->abort = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) tmem_alloc(&bars->tmem_base, 256);
  if (warp == kLoadWarp && lane == 0) { tma_prefetch_desc(&q_map); tma_prefetch_desc(&kb_map); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem = bars->tmem_base;

  // Every role walks the same units and counts the same steps: a unit takes the steps of its
  // bounding pass and one per chunk (Unit::steps), `gc` is the number of steps of all earlier units
  // of this CTA, and a step uses Kbar stage and TMEM buffer (gc + step) & 1.
  if (warp < 8) {
    // ================================ select ================================
    const int wg = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    // This thread's buffer: slot s is the 8 bytes at buf0 + s * kSlot (shared-memory address).
    constexpr uint32_t kSlot = kTile * 8;
    const uint32_t buf0 = smem_u32(sBuf + wg * Cfg::kBufBytes) + (uint32_t)r * 8u;
    // List exchange at the end of a unit: thread r of warpgroup 1 leaves its list in the
    // (empty) buffer slots of thread r of warpgroup 0, two keys per slot, so a thread of
    // warpgroup 0 only ever reads and overwrites words of its own.
    const uint32_t xk0 = smem_u32(sBuf) + (uint32_t)r * 8u;
    static_assert((L + 1) / 2 <= CAP, "a list fits the slots of one thread");
    // The bar of this row's list in either warpgroup, for the other one.
    const uint32_t bar_mine = smem_u32(sBuf + 2 * Cfg::kBufBytes) + (uint32_t)(wg * kTile + r) * 4u, bar_other = bar_mine ^ (kTile * 4u);
    uint32_t gc = 0;
    PHASE_CLOCK(ph);
    for (int round = 0; round * (int)gridDim.x < n_units; ++round) {
      const int ui = unit_of(round);
      if (ui >= n_units) continue;
      Unit u;
      if (!load_unit<EXACT>(u, ui, p, cu, n_tiles)) continue;
      constexpr int NM = L <= 8 ? 8 : 16;                       // column subsets of the bounding pass: at least L
      const int own = EXACT ? min(u.row0 + r, u.len - 1) / p.block_size : u.tile;
      float err = 0.f;                                          // EXACT: bound of |tensor-core sum - exact score|
      const T* q_row = nullptr;
      if constexpr (EXACT) {
        q_row = q + ((size_t)(p.packed ? u.bos : (size_t)u.seq * p.tokens) + min(u.row0 + r, u.len - 1)) * ((size_t)p.q_heads * D) + (size_t)u.hq * D;
        err = score_error<D, T>(q_row, norms + ((size_t)u.seq * p.kv_heads + u.hq / group) * p.num_blocks, u.own_hi, lane);
        if (u.row0 + r >= u.len) err = 0.f;                     // past the end: nobody reads what it selects
      }
      uint32_t best[L];
#pragma unroll
      for (int e = 0; e < L; ++e) best[e] = 0u;                 // 0 sorts below every real key
      float mx[NM];                                             // first pass: maxima of 8 (16) column subsets
#pragma unroll
      for (int e = 0; e < NM; ++e) mx[e] = -INFINITY;
      float bar = -INFINITY;                                    // a score must exceed this to be appended
      uint32_t wa = buf0;                                       // address of the next free slot
      auto flush = [&]() {                                      // whole warp: empty the buffers into the lists
        PHASE_CLOCK(fl);
        while (__any_sync(0xffffffffu, wa != buf0)) {
          uint32_t key = 0u;
          uint32_t sx = 0, sy = 0;
          const bool popped = wa != buf0;
          if (popped) {
            wa -= kSlot;
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(sx), "=r"(sy) : "r"(wa));
          }
          if constexpr (EXACT) {                                // does the rounding depend on the sum's error?
            const float s = __uint_as_float(sx);
            unsigned unsure = __ballot_sync(0xffffffffu, popped && (err == INFINITY || round16<T>(s - err) != round16<T>(s + err)));
            while (unsure) {
              const int who = __ffs((int)unsure) - 1;
              unsure &= unsure - 1;
              const uint32_t blk = __shfl_sync(0xffffffffu, sy, who);
              const T* qr = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(q_row), who));
              const size_t kv_row = (size_t)u.seq * p.kv_heads + u.hq / group;
              const float exact = exact_score<D, T>(qr, kbar + (kv_row * p.num_blocks + blk) * (size_t)D, lane);
              if (lane == who) sx = __float_as_uint(exact);
            }
          }
          // (a score taken again in float64 may be one that is never selected)
          if (popped && (!EXACT || __uint_as_float(sx) > -INFINITY)) key = make_key<T>(__uint_as_float(sx), sy);
          list_offer<L>(best, key);
        }
        bar = fmaxf(bar, entry_bar<T>(best[L - 1]) - err);
        // to the other warpgroup, whose blocks may be the lower ones: a step less, so that it
        // does not drop an equal score
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(bar_mine), "f"(one_step_below_key<T>(best[L - 1]) - err) : "memory");
        PHASE_ADD(wc, 4, fl);                                   // flushes (also counted in their phase)
      };
      PHASE_ADD(wc, 1, ph);                                     // unit set-up
      for (int step = 0; step < u.steps(); ++step) {
        const uint32_t gidx = gc + (uint32_t)step, st = gidx & 1u;
        const bool second = step >= u.n_first;
        const int c = u.chunk_of_step(step);
        const bool halves = u.own_hi > kTile / 2;               // both warpgroups have candidates
        if (step == u.n_first && u.n_first > 0 && !halves) {
          // The L-th largest of the subset maxima: at least L candidates reach it.
          sort_descending<NM>(mx);
          bar = one_step_below<T>(mx[L - 1] - err) - err;
        } else if (step == u.n_first && u.n_first > 0) {
          // The L-th largest of both warpgroups' subset maxima.
          // Each leaves its maxima in the (empty) buffer of its thread, in descending order; of two
          // descending lists a and b the L-th largest is the least of max(a[i], b[L - 1 - i]).
          sort_descending<NM>(mx);
#pragma unroll
          for (int e = 0; e < L; ++e)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(buf0 + (uint32_t)(e >> 1) * kSlot + (uint32_t)(e & 1) * 4u), "f"(mx[e]) : "memory");
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(bar_mine), "f"(-INFINITY) : "memory");
          asm volatile("bar.sync 3, 256;" ::: "memory");
          const uint32_t other0 = smem_u32(sBuf + (wg ^ 1) * Cfg::kBufBytes) + (uint32_t)r * 8u;
          float reached = INFINITY;
#pragma unroll
          for (int e = 0; e < L; ++e) {
            float o;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(o) : "r"(other0 + (uint32_t)((L - 1 - e) >> 1) * kSlot + (uint32_t)((L - 1 - e) & 1) * 4u) : "memory");
            reached = fminf(reached, fmaxf(mx[e], o));
          }
          bar = one_step_below<T>(reached - err) - err;
          asm volatile("bar.sync 3, 256;" ::: "memory");        // both have read: the buffers may be filled
        }
        if (second && halves) {
          float o;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(o) : "r"(bar_other) : "memory");
          bar = fmaxf(bar, o);
        }
        const bool s_ok = mbar_wait(&bars->s_full[st], (gidx >> 1) & 1u, wc, 9);
        tc_fence_after();
        PHASE_ADD(wc, 2, ph);                                   // s_full wait
        const int c0 = c * kTile + wg * 64;                     // first column (block) of this warpgroup's half
        const bool run = __all_sync(0xffffffffu, s_ok);         // a wait gave up: rank nothing unseen
        uint32_t v[32];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          tmem_ld32(tmem + lane_off + st * 128 + wg * 64 + h * 32, v);
          tmem_ld_wait();
          if (h == 1) { tc_fence_before(); mbar_arrive_warp(&bars->s_free[st]); }   // the scores are in registers
          // which of these 32 blocks are candidates of the tile: all, none, or some
          const int g0 = c0 + h * 32;
          const bool none = g0 >= u.own_hi || (p.gate_window > 0 && g0 >= p.gate_sinks && g0 + 32 <= u.own_lo - p.gate_window);
          if (!run || none) continue;
          if constexpr (EXACT) {                                // no bound: every candidate is to be scored again
            if (__any_sync(0xffffffffu, err == INFINITY)) {
#pragma unroll
              for (int k = 0; k < 32; ++k)
                if (err == INFINITY) v[k] = 0x7f800000u;        // +inf passes the entry test
            }
          }
          const bool all = g0 + 32 <= u.own_lo &&
                           (p.gate_window <= 0 || g0 + 32 <= p.gate_sinks || g0 >= u.own_hi - p.gate_window);
          if (!all) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (!gate_candidate(p, g0 + k, own)) v[k] = 0xff800000u;   // -inf: never passes
          }
          if (!second) {
#pragma unroll
            for (int k = 0; k < 32; k += 2 * NM)
#pragma unroll
              for (int e = 0; e < NM; ++e) mx[e] = max3(mx[e], __uint_as_float(v[k + e]), __uint_as_float(v[k + NM + e]));
            continue;
          }
          const uint32_t col0 = (uint32_t)(c0 + h * 32);
#pragma unroll
          for (int k0 = 0; k0 < 32; k0 += STEP) {
            if (__any_sync(0xffffffffu, wa > buf0 + (CAP - STEP) * kSlot)) flush();   // room for STEP more
#pragma unroll
            for (int k = k0; k < k0 + STEP; ++k) {
              // if (score > bar) { slot <- (score, block id); next slot }, predicated: a branch
              // here would be taken by some lane of the warp at almost every score
              asm volatile(
                  "{\n\t.reg .pred p;\n\t"
                  "setp.gt.f32 p, %1, %2;\n\t"
                  "@p st.shared.v2.b32 [%0], {%3, %4};\n\t"
                  "@p add.u32 %0, %0, %5;\n\t}"
                  : "+r"(wa)
                  : "f"(__uint_as_float(v[k])), "f"(bar), "r"(v[k]), "r"(col0 + (uint32_t)k), "n"(kTile * 8)
                  : "memory");
            }
          }
        }
        PHASE_ADD(wc, 3, ph);                                   // loads, maxima / tests and appends, flushes
      }
      flush();
      gc += (uint32_t)u.steps();
      // ---- merge the two warpgroups' lists (warpgroup 1 -> warpgroup 0's empty buffer) ----
      asm volatile("bar.sync 2, 256;" ::: "memory");            // warpgroup 0 has emptied its buffer
      if (wg == 1) {
#pragma unroll
        for (int e = 0; e < L; ++e)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(xk0 + (uint32_t)(e >> 1) * kSlot + (uint32_t)(e & 1) * 4u), "r"(best[e]) : "memory");
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      if (wg == 0 && u.row0 + r < u.len) {
#pragma unroll
        for (int e = 0; e < L; ++e) {
          uint32_t other;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(other) : "r"(xk0 + (uint32_t)(e >> 1) * kSlot + (uint32_t)(e & 1) * 4u));
          list_offer<L>(best, other);
        }
        // ---- emit: the best `take` ids plus the own block, ascending, -1 padded ----
        int ids[L];
        int kept = 0;
#pragma unroll
        for (int e = 0; e < L; ++e) {
          const bool ok = e < take && best[e] != 0u;
          ids[e] = ok ? (int)(0xFFFFu - (best[e] & 0xFFFFu)) : kEmpty;
          kept += ok ? 1 : 0;
        }
        const size_t b = p.packed ? 0 : (size_t)u.seq;
        const size_t dst_at = ((b * p.q_heads + u.hq) * p.tokens + u.bos + u.row0 + r) * (size_t)p.slots;
        int32_t* dst = block_idx + dst_at;
#pragma unroll
        for (int e = 0; e < L; ++e) {                           // rank by id: position in the output
          if (ids[e] == kEmpty) continue;
          int rank = 0;
#pragma unroll
          for (int f = 0; f < L; ++f) rank += (ids[f] < ids[e]) ? 1 : 0;
          dst[rank] = ids[e];
        }
        if (p.always_current) dst[kept++] = own;                // the own block is past every candidate
        for (int e = kept; e < p.slots; ++e) {
          dst[e] = -1;
          if (lse_fill != nullptr) lse_fill[dst_at + e] = -INFINITY;   // the slot's partial will not be written
        }
      }
      // Warpgroup 0 reads the exchange area (its own buffer) before it appends to it again;
      // warpgroup 1 writes there only behind the first barrier of the next unit.
      PHASE_ADD(wc, 5, ph);                                     // last flush, merge, emit
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      const uint32_t idesc = make_idesc(0, 128, 128, 0, 0) | (fmt << 7) | (fmt << 10);
      const uint32_t aQ = smem_u32(sQ);
      uint32_t gc = 0, nq = 0;                                  // steps / Q tiles consumed so far
      for (int round = 0; round * (int)gridDim.x < n_units; ++round) {
        const int ui = unit_of(round);
        if (ui >= n_units) continue;
        Unit u;
        if (!load_unit<EXACT>(u, ui, p, cu, n_tiles) || u.n_chunks == 0) continue;
        mbar_wait(&bars->q_full, nq & 1, wc);
        for (int step = 0; step < u.steps(); ++step, ++gc) {
          const uint32_t st = gc & 1, use = gc >> 1;
          const uint32_t aK = smem_u32(sKb) + st * Cfg::kOperand;
          mbar_wait(&bars->kb_full[st], use & 1, wc);
          if (use >= 1) mbar_wait(&bars->s_free[st], (use - 1) & 1, wc);
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t o = (ks >> 2) * kSub + (ks & 3) * 32;
            umma_f16(tmem + st * 128, make_sdesc(aQ + o, 16, 1024), make_sdesc(aK + o, 16, 1024), idesc, ks > 0);
          }
          umma_commit(&bars->s_full[st]);
          umma_commit(&bars->kb_empty[st]);
        }
        umma_commit(&bars->q_free);                             // the Q tile may be replaced
        ++nq;
      }
      // Every MMA has completed before the CTA lets go of its TMEM, also on the way out of
      // a run that gave up on a wait.
      umma_commit(&bars->drain);
      mbar_wait_quiet(&bars->drain, 0);
    }
    __syncwarp();
  } else {
    if (lane == 0) {
      uint32_t gc = 0, nq = 0;
      for (int round = 0; round * (int)gridDim.x < n_units; ++round) {
        const int ui = unit_of(round);
        if (ui >= n_units) continue;
        Unit u;
        if (!load_unit<EXACT>(u, ui, p, cu, n_tiles) || u.n_chunks == 0) continue;
        if (*wc.abort) break;                                   // no new loads once a wait gave up
        const size_t b = p.packed ? 0 : (size_t)u.seq;
        const int kv_row = u.seq * p.kv_heads + u.hq / group;
        const int tok0 = (int)(b * p.tokens) + u.bos + u.row0;
        if (nq >= 1) mbar_wait(&bars->q_free, (nq - 1) & 1, wc);
        mbar_expect_tx(&bars->q_full, Cfg::kOperand);
        for (int s = 0; s < Cfg::kSubs; ++s) tma_load_3d(sQ + s * kSub, &q_map, &bars->q_full, s * 64, u.hq, tok0);
        ++nq;
        for (int step = 0; step < u.steps(); ++step, ++gc) {
          const uint32_t st = gc & 1, use = gc >> 1;
          const int c = u.chunk_of_step(step);
          if (use >= 1) mbar_wait(&bars->kb_empty[st], (use - 1) & 1, wc);
          if (*wc.abort) break;
          mbar_expect_tx(&bars->kb_full[st], Cfg::kOperand);
          for (int s = 0; s < Cfg::kSubs; ++s)
            tma_load_3d(sKb + st * Cfg::kOperand + s * kSub, &kb_map, &bars->kb_full[st], s * 64, c * kTile, kv_row);
        }
        if (*wc.abort) break;
      }
      // No load may be in flight into this CTA's shared memory when it exits.
      if (nq >= 1) mbar_wait_quiet(&bars->q_full, (nq - 1) & 1);
      for (uint32_t k = 1; k <= 2 && k <= gc; ++k) {
        const uint32_t c = gc - k;
        mbar_wait_quiet(&bars->kb_full[c & 1], (c >> 1) & 1);
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, 256);
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
  auto kern = gate_sm100_kernel<D, T, L, EXACT>;
  static SmemLimit limit;
  if (int rc = raise_smem_limit(limit, (const void*)kern, GateCfg<D>::kSmem)) return rc;
  const int n_tiles = (p.max_seqlen + kTile - 1) / kTile;
  const long long n_units = (long long)n_tiles * p.n_seq * p.q_heads;
  const int sms = sm_count();
  const int grid = (int)(n_units < 2LL * sms ? n_units : 2LL * sms);
  MOBA_CUDA_OK(launch_chained(kern, grid, kThreads, GateCfg<D>::kSmem, st, qm, km, cu, block_idx, lse_fill, p, n_tiles,
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

// Block sizes that divide the tile of 128 queries; as many ranked blocks as the per-thread buffers
// can exchange; a candidate window keeps the portable kernel.
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
