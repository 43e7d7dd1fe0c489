// Forward attention on tcgen05 tensor cores (bf16/f16, columns of 128 keys, head_dim 64 or 128).
//
// Persistent CTAs (one per SM) walk the work items (a column of 128 keys and a range of the list
// of queries that selected it) longest first, in alternating direction. An item is cut into tiles
// of 128 gathered queries; NB tiles (4 at head_dim 64, 2 at 128) are in flight per SM, each on
// its own TMEM buffer, Q stage, output staging tile and softmax warpgroup, because one tile is a
// long chain of short dependent steps (gather -> MMA -> softmax -> MMA -> epilogue) and only
// several chains side by side keep the SM busy.
//   loader   (1 warp)    walks the work list, publishes each item's descriptor in shared memory,
//                        TMA-loads its K block and V block (two buffers each at head_dim 64);
//                        zeroes the rows of a block that its sequence cuts short
//   gather   (4 warps)   one index entry per lane; TMA gathers of four query rows per request, a
//                        tile per buffer ahead of the softmax warps, and for each row of the tile
//                        where its output goes and which keys it attends. (The softmax warps used
//                        to copy the rows themselves, 16 bytes per lane: that took 1 700 of a
//                        tile's 9 000 clocks and blocked the load-store unit for all others.)
//   mma      (2 threads) one issues S = Q K^T (M128 N128 K=D) tile after tile, the other
//                        O = P V (M128 N=D K128) with P as operand A **from TMEM**; each
//                        blocks on what its next tile needs, so a tile that becomes ready
//                        is issued without a polling round
//   softmax  (NB x 4 warps; warpgroup w owns tiles t = w mod NB)
//            tcgen05.ld S, mask, exp2, row sum, P (16-bit pairs) -> tcgen05.st over the scores
//            already read (P never touches shared memory); then tcgen05.ld O, normalise, stage in
//            smem and store the partial output rows (eight or sixteen lanes per row) and their
//            log2-sum-exp at the (query, slot) addresses
//   storers  (head_dim 128 only: NB x 4 warps) take the staged output rows out beside the softmax
//            warps
// TMEM columns of a buffer: S [0,128), P over [0,64), O in [64,128) at head_dim 64 and in
// a second 128 columns at head_dim 128.
// Instruction issue and the hand-overs between the warps bound it, not memory (about half of the
// copy rate) and not the tensor cores (about a quarter). So the softmax works on two scores per
// instruction where it can, and compares keys only in the chunks of 32 that need it: on the
// diagonal and at the end of a sequence. At 131072 queries x 4 heads x 8 blocks, head_dim 64:
// 0.38 ms before these, 0.30 ms with them; 40000 x 32 heads, head_dim 128: 1.24 and 1.15 ms. Deeper
// staging, entries fetched further ahead and storers at head_dim 64 were slower or no faster.
// A (query, block) pair is complete inside one tile, so nothing is rescaled
// here; the merge kernel combines a query's slots.
//
// Stands in for moba_fwd_kernel of the reference (src/moba/kernels/moba_fwd.py:229-425).
#include "common.cuh"
#include "sm100.cuh"

#include <type_traits>

namespace moba {
using namespace sm100;

namespace {

constexpr int kTile = 128;                 // queries per tile == keys per column
constexpr int kSub = kTile * 128;          // bytes of one [128 rows][64 elems] swizzled sub-tile
constexpr int kGatherWarps = 4;

template <int D> struct FwdCfg {
  static constexpr int kSubs = D / 64;                 // sub-tiles per operand along the head dim
  static constexpr int kOperand = kSubs * kSub;        // bytes of K, V or one Q stage
  // Tiles in flight (TMEM buffers, Q stages, output staging tiles, softmax warpgroups).
  static constexpr int kBufs = tensor_core_plan(D).fwd_tiles_in_flight;
  static_assert(tensor_core_plan(D).fwd_q_stages == kBufs, "a tile's Q stage goes with its buffer");
  // K and V buffers: with two, the next item's blocks load while this item's last tiles run.
  static constexpr int kKvBufs = (D == 64) ? 2 : 1;
  static constexpr int kSmemData = 2 * kKvBufs * kOperand + 2 * kBufs * kOperand;      // K, V; Q stages, output staging
  static constexpr int kSmem = kSmemData + 1024 /*align*/ + 8192 /*barriers, row tables*/;
  static constexpr int kScoreWarp = 4 * kBufs, kPvWarp = kScoreWarp + 1, kLoadWarp = kScoreWarp + 2;
  static constexpr int kGatherWarp0 = kScoreWarp + 4;  // (the fourth warp of this warpgroup only completes it)
  static constexpr bool kStorers = (kBufs == 2);
  static constexpr int kStoreWarp0 = kGatherWarp0 + kGatherWarps;
  static constexpr int kThreads = (kStoreWarp0 + (kStorers ? 4 * kBufs : 0)) * 32;
  static_assert(kThreads == 768, "both plans fill six warpgroups");
  // Registers: launched with 80 each (61 440); the softmax warpgroups take more, the others give down.
  // At head_dim 64 with 96 and 48 the others spilled 76 bytes, with 88 and 64 nobody does: the forwards of
  // 65536 x 4, 12 blocks each, 493 -> 486 us; a step of 131072 x 4, 1447 -> 1432.
  static constexpr int kSoftmaxRegs = D == 64 ? 88 : 128, kOtherRegs = D == 64 ? 64 : 56;
  static_assert(4 * kBufs * 32 * kSoftmaxRegs + (kThreads - 4 * kBufs * 32) * kOtherRegs <= kThreads * 80, "register split");
};

struct Column {                            // one unit of work; n < 0 ends the stream
  int kv_row, blk, n, lo, key0, keys, bos, tok0;
};

struct RowMeta {                           // of a tile in flight, written by the gather warps
  int dest[kTile];                         // row of the partial buffers, -1 = none (2^31 rows would be 256 GB or more)
  uint16_t range[kTile];                   // first | last << 8 key of the column the query attends
};

struct Bars {
  uint64_t k_full[2], v_full[2], k_free[2], v_free[2];
  uint64_t k_fix[2], v_fix[2];             // per K / V buffer: the rows of a block cut short are zeroed (one for
                                           // both could complete twice before its first phase is looked at)
  uint64_t q_full[4];                      // per buffer: the tile's rows have landed and its row data is written
  uint64_t q_empty[4];                     // the S MMA that read the stage has retired
  uint64_t meta_free[4];                   // the softmax warps have read the row data
  uint64_t s_full[4], p_full[4], o_full[4], so_free[4];
  uint64_t o_staged[2], stage_free[2];     // storers: a tile's output rows are staged / have left the staging tile
  uint64_t sp_free[2];                     // head_dim 128: the S / P columns of a buffer are free (its P V has retired)
  uint64_t col_full[8], col_free[8];       // ring of item descriptors, published by the loader
  uint64_t drain[2];                       // all MMAs of an issuing thread have completed
  uint32_t tmem_base;
  int abort;
  int end[4];                              // per buffer: the stream has no further tile for it
  int stored_end[2];
  Column cols[8];
  RowMeta meta[4];
  int out_row[4][kTile];                   // rows of the partial buffer a warpgroup is storing, -1 = none
};

// AND of a predicate over the threads of a warpgroup (named barrier `id`). Every decision
// that steers a warpgroup past one of its own barriers is taken through this, so that a wait
// that gave up in some threads only can never leave the others alone at a barrier. The barrier
// counts warps, whole ones.
__device__ __forceinline__ bool group_all(bool pred, int id) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, %2, 128, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r) : "r"((uint32_t)pred), "r"(id) : "memory");
  return r != 0;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Work item `j` of a (sequence, kv head) row, in its dispatch order (heaviest first); false for padding.
__device__ __forceinline__ bool load_column(Column& c, int kv_row, int j, const moba_b200_index& ix,
                                            const moba_b200_problem& p, const int32_t* cu) {
  c.kv_row = kv_row;
  WorkItem w;
  if (!load_work_item(w, ix, ix.col_nnz + (size_t)c.kv_row * p.num_blocks, c.kv_row, j)) return false;
  c.blk = w.blk;
  c.n = w.n;
  c.lo = ix.col_offsets[(size_t)c.kv_row * (p.num_blocks + 1) + c.blk] + w.first;
  const int seq = c.kv_row / p.kv_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  c.tok0 = p.packed ? 0 : seq * p.tokens;
  c.bos = sp.bos;
  c.key0 = sp.bos + c.blk * kTile;
  c.keys = min(kTile, sp.bos + sp.len - c.key0);
  return c.n > 0 && c.keys > 0;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int D, typename T, typename TP, bool CLAIM>
__global__ void __launch_bounds__(FwdCfg<D>::kThreads, 1)
fwd_sm100_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                 const __grid_constant__ CUtensorMap q_map, moba_b200_index ix, const int32_t* __restrict__ cu,
                 TP* __restrict__ part_o, float* __restrict__ part_lse, moba_b200_problem p, int part_keys, int n_items,
                 ClaimOrder order, unsigned* error_word) {
  using Cfg = FwdCfg<D>;
  constexpr int NB = Cfg::kBufs, NKV = Cfg::kKvBufs;
  constexpr bool kStaged = sizeof(TP) == 2;
  // TMEM columns of a buffer: scores [0, 128); P, 16-bit pairs, over [0, 64); O in [128 - D, 128)
  // at head_dim 64 and in a second 128 columns at head_dim 128.
  constexpr uint32_t kOCol = (D == 64) ? 64 : 128, kBufCols = (D == 64) ? 128 : 256;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* sK = smem;                                     // NKV buffers
  unsigned char* sV = sK + NKV * Cfg::kOperand;
  unsigned char* sQ = sV + NKV * Cfg::kOperand;                 // NB stages
  unsigned char* sO = sQ + NB * Cfg::kOperand;                  // NB output staging tiles
  Bars* bars = reinterpret_cast<Bars*>(sO + NB * Cfg::kOperand);
  static_assert(sizeof(Bars) <= 8192, "barrier block outgrew its reservation");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_kv_rows = p.n_seq * p.kv_heads;
#ifdef MOBA_WAIT_STATS
  const WaitCtx wc{&bars->abort, error_word, nullptr};
#else
  const WaitCtx wc{&bars->abort, error_word};
#endif

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->k_full[i], 1); mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->k_free[i], 1); mbar_init(&bars->v_free[i], 1);
      mbar_init(&bars->o_staged[i], 4); mbar_init(&bars->stage_free[i], 4); mbar_init(&bars->sp_free[i], 1);
      mbar_init(&bars->drain[i], 1); mbar_init(&bars->k_fix[i], 1); mbar_init(&bars->v_fix[i], 1);
      bars->stored_end[i] = 0;
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&bars->q_full[i], kGatherWarps); mbar_init(&bars->q_empty[i], 1); mbar_init(&bars->meta_free[i], 4);
      mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_full[i], 4);
      mbar_init(&bars->o_full[i], 1); mbar_init(&bars->so_free[i], 4);
      bars->end[i] = 0;
    }
    for (int i = 0; i < 8; ++i) { mbar_init(&bars->col_full[i], 1); mbar_init(&bars->col_free[i], 2 + kGatherWarps); }
    bars->abort = 0;
    fence_barrier_init();
  }
  if (warp == Cfg::kScoreWarp) tmem_alloc(&bars->tmem_base, 512);
  if (warp == Cfg::kLoadWarp && lane == 0) { tma_prefetch_desc(&k_map); tma_prefetch_desc(&v_map); tma_prefetch_desc(&q_map); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem = bars->tmem_base;

  const float cs = rsqrtf((float)D) * kLog2e;
  const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;

  // The staged 16-bit output rows of buffer `wg` -> global memory, eight or sixteen lanes per row
  // (128 threads, `tid` of them).
  auto store_rows = [&](int wg, int tid) {
    constexpr int CPRO = D / 8;                      // 16-byte chunks per output row
    constexpr int RPPO = 128 / CPRO;                 // rows per pass
    const unsigned char* stage = sO + wg * Cfg::kOperand;
    const int cc = tid % CPRO;
#pragma unroll
    for (int pass = 0; pass < CPRO; ++pass) {
      const int rr = pass * RPPO + tid / CPRO;
      const int to = bars->out_row[wg][rr];
      const uint4 w = *reinterpret_cast<const uint4*>(stage + (cc >> 3) * kSub + swz128(rr, cc & 7));
      if (to >= 0) st_global_stream16(reinterpret_cast<unsigned char*>(part_o + (size_t)to * D) + cc * 16, w);
    }
  };

  if (warp < 4 * NB) {
    // ======================= softmax + epilogue warpgroups =======================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::kSoftmaxRegs));
    const int wg = warp >> 2;                         // owns tiles with t % NB == wg and buffer wg
    const int r = (warp & 3) * 32 + lane;             // row of the tile == TMEM lane
    const int bar_id = 1 + wg;                        // named barrier of this warpgroup
    const uint32_t tbuf = tmem + ((uint32_t)((warp & 3) * 32) << 16) + wg * kBufCols;
    unsigned char* myO = sO + wg * Cfg::kOperand;     // staging of this warpgroup's output rows
    uint32_t u = 0;                                   // how often this buffer has been used before
    for (;; ++u) {
      const bool q_ok = mbar_wait(&bars->q_full[wg], u & 1, wc, 1);
      if (!group_all(q_ok && bars->end[wg] == 0, bar_id)) break;
      const int dest = bars->meta[wg].dest[r];
      const uint32_t range = bars->meta[wg].range[r];
      mbar_arrive_warp(&bars->meta_free[wg]);
      const int jmin = (int)(range & 0xffu), jmax = (int)(range >> 8);
      // Which of the four chunks of 32 keys every row of the warp keeps whole (bits 0..3) and which
      // no row keeps any key of (bits 4..7): only the others need a comparison per score, a few on
      // the diagonal and where a sequence ends.
      uint32_t kind = 0;
      auto open_keys = [&](int ch) {                     // bit k: the row keeps key 32 ch + k
        const int lo = max(jmin - ch * 32, 0), hi = min(jmax - ch * 32, 31);
        return lo <= hi ? (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo) : 0u;
      };
      if (__all_sync(0xffffffffu, range == (uint32_t)(kTile - 1) << 8)) {
        kind = 15;
      } else {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          if (__all_sync(0xffffffffu, jmin <= ch * 32 && jmax >= ch * 32 + 31)) kind |= 1u << ch;
          if (__all_sync(0xffffffffu, jmax < ch * 32 || jmin > ch * 32 + 31)) kind |= 16u << ch;
        }
      }
      const bool s_ok = mbar_wait(&bars->s_full[wg], u & 1, wc, 2);
      tc_fence_after();

      uint32_t v[32];
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        if (kind >> ch & 16) continue;
        tmem_ld32(tbuf + ch * 32, v);
        tmem_ld_wait();
        if (kind >> ch & 1) {
#pragma unroll
          for (int k = 0; k < 32; k += 2)
            mx4[(k >> 1) & 3] = max3(mx4[(k >> 1) & 3], __uint_as_float(v[k]), __uint_as_float(v[k + 1]));
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k)
            mx4[k & 3] = fmaxf(mx4[k & 3], open_keys(ch) >> k & 1 ? __uint_as_float(v[k]) : -INFINITY);
        }
      }
      const float m2 = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * cs;

      // Two scores per instruction where the pipes allow it (fma, add, conversion).
      float2 l2[2] = {{0.f, 0.f}, {0.f, 0.f}};
      const float2 cs2 = {cs, cs}, neg_m2 = {-m2, -m2};
      auto exp_chunk = [&](int ch, auto masked) {
        tmem_ld32(tbuf + ch * 32, v);
        tmem_ld_wait();
        // P of these 32 keys goes back over scores that have been read: chunk ch's 16-bit
        // pairs land in columns [16 ch, 16 ch + 16), all of them below column 32 (ch + 1).
        uint32_t pk[16];
        const uint32_t open = decltype(masked)::value ? open_keys(ch) : 0u;
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          const float2 x = fma2(make_float2(__uint_as_float(v[k]), __uint_as_float(v[k + 1])), cs2, neg_m2);
          float2 e = make_float2(ex2(x.x), ex2(x.y));
          if constexpr (decltype(masked)::value) {
            if (!(open >> k & 1)) e.x = 0.f;
            if (!(open >> k & 2)) e.y = 0.f;
          }
          l2[(k >> 1) & 1] = add2(l2[(k >> 1) & 1], e);
          pk[k >> 1] = pack2<T>(e.x, e.y);
        }
        tmem_st16(tbuf + ch * 16, pk);
      };
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        if (kind >> ch & 1) {
          exp_chunk(ch, std::false_type{});
        } else if (kind >> ch & 16) {
          const uint32_t zero[16] = {0};
          tmem_st16(tbuf + ch * 16, zero);
        } else {
          exp_chunk(ch, std::true_type{});
        }
      }
      tmem_st_wait();
      const float l = (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
      tc_fence_before();
      mbar_arrive_warp(&bars->p_full[wg]);

      // ---- epilogue of the same tile ----
      const float inv = 1.f / l;
      // A wait that gave up leaves TMEM unspecified: the tile then stores nothing.
      const bool o_ok = mbar_wait(&bars->o_full[wg], u & 1, wc, 3) && s_ok;
      tc_fence_after();
      // the storers have taken the previous tile's rows out of the staging tile
      if (Cfg::kStorers && kStaged && u >= 1) mbar_wait(&bars->stage_free[wg], (u - 1) & 1, wc, 11);
      const bool live = dest >= 0 && o_ok;
#pragma unroll 1
      for (int ch = 0; ch < D / 32; ++ch) {
        tmem_ld32(tbuf + kOCol + ch * 32, v);
        tmem_ld_wait();
        if (kStaged) {
          // Stage the 16-bit tile in shared memory: one row per thread straight to global
          // memory would touch 32 lines per instruction.
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 w;
            w.x = pack2<T>(__uint_as_float(v[g * 8 + 0]) * inv, __uint_as_float(v[g * 8 + 1]) * inv);
            w.y = pack2<T>(__uint_as_float(v[g * 8 + 2]) * inv, __uint_as_float(v[g * 8 + 3]) * inv);
            w.z = pack2<T>(__uint_as_float(v[g * 8 + 4]) * inv, __uint_as_float(v[g * 8 + 5]) * inv);
            w.w = pack2<T>(__uint_as_float(v[g * 8 + 6]) * inv, __uint_as_float(v[g * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(myO + (ch >> 1) * kSub + swz128(r, (ch & 1) * 4 + g)) = w;
          }
        } else if (live) {
          float4* d4 = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(part_o + (size_t)dest * D) + ch * 128);
#pragma unroll
          for (int g = 0; g < 8; ++g)
            d4[g] = make_float4(__uint_as_float(v[g * 4 + 0]) * inv, __uint_as_float(v[g * 4 + 1]) * inv,
                                __uint_as_float(v[g * 4 + 2]) * inv, __uint_as_float(v[g * 4 + 3]) * inv);
        }
      }
      tc_fence_before();
      mbar_arrive_warp(&bars->so_free[wg]);               // the TMEM buffer may be overwritten
      if (live) st_global_stream_f32(part_lse + dest, m2 + log2f(l));
      if (kStaged) {
        bars->out_row[wg][r] = live ? dest : -1;
        if constexpr (Cfg::kStorers) {
          mbar_arrive_warp(&bars->o_staged[wg]);       // (releasing: the storers see the rows and the table)
        } else {
          asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
          store_rows(wg, r);
          asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");   // the staging tile may be written again
        }
      }
    }
    if (Cfg::kStorers && kStaged) {                    // no further tile of this buffer, once its last one has left
      if (u >= 1) mbar_wait(&bars->stage_free[wg], (u - 1) & 1, wc, 11);
      if (r == 0) bars->stored_end[wg] = 1;
      mbar_arrive_warp(&bars->o_staged[wg]);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kOtherRegs));
    if (Cfg::kStorers && warp >= Cfg::kStoreWarp0) {
      // ============================ storers ============================
      const int wg = (warp - Cfg::kStoreWarp0) >> 2, tid = ((warp - Cfg::kStoreWarp0) & 3) * 32 + lane;
      for (uint32_t u = 0; kStaged; ++u) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->o_staged[wg], u & 1, wc, 10))) break;
        if (bars->stored_end[wg]) break;
        store_rows(wg, tid);
        mbar_arrive_warp(&bars->stage_free[wg]);
      }
    } else if (warp >= Cfg::kGatherWarp0 && warp < Cfg::kGatherWarp0 + kGatherWarps) {
      // ============================ gather warps ============================
      // Warp g: rows [32 g, 32 g + 32) of every tile, one index entry per lane.
      const int gw = warp - Cfg::kGatherWarp0, pt = gw * 32 + lane;
      const int n_rows = p.batch * p.tokens * p.q_heads;
      uint32_t t = 0;
      bool stop = false;
      // the tile's row data and Q stage are free again
      auto wait_stage = [&](uint32_t b, uint32_t u) {
        if (u >= 1) {
          mbar_wait(&bars->q_empty[b], (u - 1) & 1, wc, 4);
          mbar_wait(&bars->meta_free[b], (u - 1) & 1, wc, 4);
        }
      };
      for (uint32_t it = 0;; ++it) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->col_full[it & 7], (it >> 3) & 1, wc, 5))) { stop = true; break; }
        const Column c = bars->cols[it & 7];
        mbar_arrive_warp(&bars->col_free[it & 7]);
        if (c.n < 0) break;
        const int nt = (c.n + kTile - 1) / kTile;
        const size_t list0 = (size_t)c.kv_row * ix.capacity + c.lo;
        const size_t b = p.packed ? 0 : (size_t)(c.kv_row / p.kv_heads);
        RawPair nx{0, 0, 0};                                 // index entry of the next tile, fetched ahead
        if (pt < c.n) nx = fetch_pair(ix, list0 + pt);
        for (int i = 0; i < nt; ++i, ++t) {
          const uint32_t buf = t % NB, u = t / NB;
          const int e = i * kTile + pt;
          const PairEntry me = pair_of(ix, nx);
          int row_id = n_rows, dest = -1;                    // a row past the end of the tensor: zeros
          int first = 0, last = kTile - 1;                   // (a dead row keeps no warp from the unmasked path)
          if (e < c.n) {
            row_id = (int)((b * p.tokens + me.row) * p.q_heads + me.head);
            dest = (int)(part_row(p, b, me.head, me.row) * (size_t)p.slots + me.slot);
            // keys of the column: those of the pair's block, up to the query itself
            first = me.part * part_keys;
            last = min(c.keys, first + part_keys) - 1;
            if (p.causal && (me.row - c.bos) / kTile == c.blk) last = min(last, me.row - c.key0);
          }
          if (e + kTile < c.n) nx = fetch_pair(ix, list0 + e + kTile);
          int rows[4];                                       // the four rows a lane gathers (lanes 0..7)
#pragma unroll
          for (int k = 0; k < 4; ++k) rows[k] = __shfl_sync(0xffffffffu, row_id, (lane * 4 + k) & 31);
          wait_stage(buf, u);
          if (__any_sync(0xffffffffu, *wc.abort)) { stop = true; break; }   // no new copies once a wait gave up
          bars->meta[buf].dest[pt] = dest;
          bars->meta[buf].range[pt] = (uint16_t)(first | (last << 8));
          __syncwarp();
          if (lane == 0) mbar_expect_tx(&bars->q_full[buf], 32 * D * 2);     // releases the row data, too
          __syncwarp();
          if (lane < 8) {
#pragma unroll
            for (int h = 0; h < Cfg::kSubs; ++h)
              tma_gather4(sQ + buf * Cfg::kOperand + h * kSub + (gw * 32 + lane * 4) * 128, &q_map, &bars->q_full[buf], h * 64,
                          rows[0], rows[1], rows[2], rows[3]);
          }
          __syncwarp();
        }
        if (stop) break;
      }
      // No copy may be in flight into this CTA's shared memory when it exits.
      for (uint32_t k = 1; k <= (uint32_t)NB && k <= t; ++k) mbar_wait_quiet(&bars->q_full[(t - k) % NB], ((t - k) / NB) & 1);
      // the end of the stream, to every softmax warpgroup
      for (uint32_t k = 0; k < (uint32_t)NB && !stop; ++k, ++t) {
        wait_stage(t % NB, t / NB);
        if (gw == 0 && lane == 0) bars->end[t % NB] = 1;
        mbar_arrive_warp(&bars->q_full[t % NB]);
      }
    } else if (warp == Cfg::kScoreWarp || warp == Cfg::kPvWarp) {
      // ============================== MMA issuers ==============================
      // Two threads feed the tensor core, each walking the CTA's tiles in order and blocking
      // on exactly what its next MMA needs: a tile is issued as soon as its inputs are there.
      if (lane == 0) {
        constexpr uint32_t idesc_s = make_idesc(0, 128, 128, 0, 0);
        constexpr uint32_t idesc_o = make_idesc(0, 128, D, 0, 1);
        const uint32_t fbits = (fmt << 7) | (fmt << 10);
        const uint32_t aQ = smem_u32(sQ);
        const bool is_s = warp == Cfg::kScoreWarp;
        uint32_t t = 0, fixes = 0;                                // tiles issued; bit b: parity of the cut-short columns seen in buffer b
        for (uint32_t it = 0;; ++it) {
          if (!mbar_wait(&bars->col_full[it & 7], (it >> 3) & 1, wc, 20)) break;
          const int n = bars->cols[it & 7].n;
          const bool partial = bars->cols[it & 7].keys < kTile;
          mbar_arrive(&bars->col_free[it & 7]);
          if (n < 0) break;
          const int nt = (n + kTile - 1) / kTile;
          const uint32_t kb = it % NKV, ku = it / NKV;             // K/V buffer of the item, its earlier uses
          const uint32_t aK = smem_u32(sK) + kb * Cfg::kOperand, aV = smem_u32(sV) + kb * Cfg::kOperand;
          for (int i = 0; i < nt; ++i, ++t) {
            const uint32_t b = t % NB, u = t / NB;
            if (is_s) {
              // ---- S = Q K^T of tile t ----
              mbar_wait(&bars->q_full[b], u & 1, wc, 21);
              // The buffer's columns: where O has columns of its own (head_dim 128) the scores of
              // the next tile only wait for P V of the previous one, not for its O to be read out.
              if (u >= 1) mbar_wait(D == 128 ? &bars->sp_free[b] : &bars->so_free[b], (u - 1) & 1, wc, 22);
              if (i == 0) {
                mbar_wait(&bars->k_full[kb], ku & 1, wc, 23);
                if (partial) mbar_wait(&bars->k_fix[kb], fixes >> kb & 1, wc, 23);
              }
              tc_fence_after();
              const uint32_t qb = aQ + b * Cfg::kOperand;
#pragma unroll
              for (int ks = 0; ks < D / 16; ++ks) {
                const uint32_t o = (ks >> 2) * kSub + (ks & 3) * 32;
                umma_f16(tmem + b * kBufCols, make_sdesc(qb + o, 16, 1024), make_sdesc(aK + o, 16, 1024),
                         idesc_s | fbits, ks > 0);
              }
              umma_commit(&bars->s_full[b]);
              umma_commit(&bars->q_empty[b]);
              if (i == nt - 1) umma_commit(&bars->k_free[kb]);
            } else {
              // ---- O = P V of tile t ----
              mbar_wait(&bars->p_full[b], u & 1, wc, 24);
              if (D == 128 && u >= 1) mbar_wait(&bars->so_free[b], (u - 1) & 1, wc, 24);   // the O columns have been read out
              if (i == 0) {
                mbar_wait(&bars->v_full[kb], ku & 1, wc, 25);
                if (partial) mbar_wait(&bars->v_fix[kb], fixes >> kb & 1, wc, 25);
              }
              tc_fence_after();
              // operand A: P from TMEM, 16 keys (eight columns of 16-bit pairs) per step
#pragma unroll
              for (int ks = 0; ks < 8; ++ks) {
                umma_f16_ts(tmem + b * kBufCols + kOCol, tmem + b * kBufCols + ks * 8,
                            make_sdesc(aV + ks * 2048, kSub, 1024), idesc_o | fbits, ks > 0);
              }
              umma_commit(&bars->o_full[b]);
              if (D == 128) umma_commit(&bars->sp_free[b]);
              if (i == nt - 1) umma_commit(&bars->v_free[kb]);
            }
          }
          if (partial) fixes ^= 1u << kb;
        }
        // Every MMA of this thread has completed before the CTA lets go of its TMEM, also on
        // the way out of a run that gave up on a wait.
        umma_commit(&bars->drain[is_s ? 0 : 1]);
        mbar_wait_quiet(&bars->drain[is_s ? 0 : 1], 0);
      }
      __syncwarp();
    } else if (warp == Cfg::kLoadWarp) {
      // ================== work-list walker and K/V TMA loader ==================
      // The only warp that resolves columns (three dependent global loads each); it runs
      // ahead of everybody and publishes the descriptors through a ring in shared memory.
      // All 32 lanes run the loop; lane 0 publishes and issues the loads, and the whole warp
      // zeroes the rows of a block that the end of its sequence cuts short (they belong to
      // the next sequence, or to the next batch row).
      uint32_t it_cnt = 0;
      const uint64_t keep = l2_policy_evict_last();
      // The list is sorted longest first; CTAs take it in alternating direction
      // (0..G-1, G-1..0, ...) so that no CTA collects the largest of every round.
      const int G = (int)gridDim.x;
      const size_t index_elems = (size_t)n_kv_rows * ix.capacity;
      // The index entries of a column are read by the gather warps a tile at a time, straight
      // from global memory; asking the L2 for them a column ahead turns a DRAM round trip per
      // tile into an L2 hit.
      auto prefetch_entries = [&](const Column& c) {
        if (packed_pairs(ix)) {
          if (lane == 0)
            l2_prefetch_i32(ix.row_indices, 2 * ((size_t)c.kv_row * ix.capacity + c.lo), 2 * c.n, 2 * index_elems);
        } else if (lane < 3) {
          const int32_t* arr = lane == 0 ? ix.row_indices : (lane == 1 ? ix.head_indices : ix.slot_of_pair);
          l2_prefetch_i32(arr, (size_t)c.kv_row * ix.capacity + c.lo, c.n, index_elems);
        }
      };
      // The next item with pairs; false at the end. The lanes look at 32 items at once: most of a
      // packed batch's list is padding (every row has room for the longest sequence's items), which
      // walked one by one took 0.15 of 1.13 ms (16 sequences of 300 to 9000 tokens, 32 heads) and
      // 0.85 of 4.9 ms (32 of 1024 to 32768, 16 heads). An item's row and place are divided out in 32 bits:
      // the division in 64 of 65536 x 4 heads of 64 took 4 of 152 us here, and 8 of 330 in the backward.
      Column mine;
      unsigned found = 0;
      int round0 = 0;
      auto take = [&](Column& c, int src) {
        c.kv_row = __shfl_sync(0xffffffffu, mine.kv_row, src); c.blk = __shfl_sync(0xffffffffu, mine.blk, src);
        c.n = __shfl_sync(0xffffffffu, mine.n, src); c.lo = __shfl_sync(0xffffffffu, mine.lo, src);
        c.key0 = __shfl_sync(0xffffffffu, mine.key0, src); c.keys = __shfl_sync(0xffffffffu, mine.keys, src);
        c.bos = __shfl_sync(0xffffffffu, mine.bos, src); c.tok0 = __shfl_sync(0xffffffffu, mine.tok0, src);
        return true;
      };
      auto dealt = [&](Column& c) {
        while (found == 0) {
          if ((long long)round0 * G >= n_items) return false;
          const int round = round0 + lane;
          const long long item = (long long)round * G + ((round & 1) ? (G - 1 - (int)blockIdx.x) : (int)blockIdx.x);
          found = __ballot_sync(0xffffffffu, item < n_items && load_column(mine, (int)item % n_kv_rows, (int)item / n_kv_rows, ix, p, cu));
          round0 += 32;
        }
        const int src = __ffs(found) - 1;
        found &= found - 1;
        return take(c, src);
      };
      ClaimWalk walk{0, 0};
      auto claimed = [&](Column& c) {
        int kv_row, j;
        do {                                                    // (an item without pairs is nothing to the forward)
          if (!claim_item(walk, order, ix, p, cu, n_kv_rows, kv_row, j)) return false;
        } while (!load_column(c, kv_row, j, ix, p, cu));
        return true;
      };
      auto next = [&](Column& c) { if constexpr (CLAIM) return claimed(c); else return dealt(c); };
      auto publish = [&](const Column& c, uint32_t n) {
        if (n >= 8) mbar_wait(&bars->col_free[n & 7], ((n >> 3) - 1) & 1, wc, 6);
        __syncwarp();
        if (lane == 0) {
          bars->cols[n & 7] = c;
          mbar_arrive(&bars->col_full[n & 7]);
        }
      };
      // One call of `next`: each turn takes an item and loads the one taken before.
      Column c, c_next;
      uint32_t published = 0;
      c.n = 0;
      for (;;) {
        // The gather warps run ahead of the MMAs: at the last tiles of an item they are at tiles of
        // the next one, so its descriptor (and, in the L2, its index entries) must be there before
        // this item's K and V are even loaded.
        const bool more = next(c_next);
        if (more) { prefetch_entries(c_next); publish(c_next, published++); }
        if (__any_sync(0xffffffffu, *wc.abort)) break;        // no new loads once a wait gave up
        if (c.n > 0) {
          const int kvh = c.kv_row % p.kv_heads, tok = c.tok0 + c.key0;
          const uint32_t kb = it_cnt % NKV, ku = it_cnt / NKV;     // buffer of this item, its earlier uses
          unsigned char* bK = sK + kb * Cfg::kOperand;
          unsigned char* bV = sV + kb * Cfg::kOperand;
          if (ku >= 1) mbar_wait(&bars->k_free[kb], (ku - 1) & 1, wc, 7);
          if (lane == 0) {
            mbar_expect_tx(&bars->k_full[kb], Cfg::kOperand);
            for (int s = 0; s < Cfg::kSubs; ++s) tma_load_3d_hint(bK + s * kSub, &k_map, &bars->k_full[kb], s * 64, kvh, tok, keep);
          }
          if (ku >= 1) mbar_wait(&bars->v_free[kb], (ku - 1) & 1, wc, 8);
          if (lane == 0) {
            mbar_expect_tx(&bars->v_full[kb], Cfg::kOperand);
            for (int s = 0; s < Cfg::kSubs; ++s) tma_load_3d_hint(bV + s * kSub, &v_map, &bars->v_full[kb], s * 64, kvh, tok, keep);
          }
          if (c.keys < kTile) {
            const int dead = kTile - c.keys;
            mbar_wait(&bars->k_full[kb], ku & 1, wc, 9);
            for (int i = lane; i < dead * 8 * Cfg::kSubs; i += 32) {
              const int s = i / (dead * 8), rr = c.keys + (i % (dead * 8)) / 8, ch = i % 8;
              *reinterpret_cast<uint4*>(bK + s * kSub + rr * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
            }
            fence_proxy_async();
            mbar_arrive_warp(&bars->k_fix[kb]);
            mbar_wait(&bars->v_full[kb], ku & 1, wc, 9);
            for (int i = lane; i < dead * 8 * Cfg::kSubs; i += 32) {
              const int s = i / (dead * 8), rr = c.keys + (i % (dead * 8)) / 8, ch = i % 8;
              *reinterpret_cast<uint4*>(bV + s * kSub + rr * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
            }
            fence_proxy_async();
            mbar_arrive_warp(&bars->v_fix[kb]);
          }
          ++it_cnt;
        }
        if (!more) break;
        c = c_next;
      }
      c.n = -1;                                                 // end of the stream
      publish(c, it_cnt);
      if (lane == 0) {
        // No load may be in flight into this CTA's shared memory when it exits.
        for (uint32_t back = 1; back <= (uint32_t)NKV && back <= it_cnt; ++back) {
          const uint32_t n = it_cnt - back;
          mbar_wait_quiet(&bars->k_full[n % NKV], (n / NKV) & 1);
          mbar_wait_quiet(&bars->v_full[n % NKV], (n / NKV) & 1);
        }
      }
      __syncwarp();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kScoreWarp) tmem_dealloc(tmem, 512);
}

template <int D, typename T, typename TP>
int launch_one(const moba_b200_problem& p, const CUtensorMap& km, const CUtensorMap& vm, const CUtensorMap& qm,
               const moba_b200_index& ix, const int32_t* cu, void* part_o, float* part_lse, int part_keys, int n_items,
               const ClaimOrder& order, unsigned* err, cudaStream_t st) {
  const bool claimed = order.next != nullptr;
  auto kern = claimed ? fwd_sm100_kernel<D, T, TP, true> : fwd_sm100_kernel<D, T, TP, false>;
  static SmemLimit limits[2];
  if (int rc = raise_smem_limit(limits[claimed], (const void*)kern, FwdCfg<D>::kSmem)) return rc;
  const int sms = sm_count();
  const int grid = n_items < sms ? n_items : sms;
  MOBA_CUDA_OK(launch_chained(kern, grid, FwdCfg<D>::kThreads, FwdCfg<D>::kSmem, st, km, vm, qm, ix, cu,
                              (TP*)part_o, part_lse, p, part_keys, n_items, order, err));
  return MOBA_B200_OK;
}

}  // namespace

bool fwd_sm100_supported(const moba_b200_problem& p) {
  return (p.dtype == MOBA_B200_BF16 || p.dtype == MOBA_B200_F16) && p.block_size == 128 &&
         (p.head_dim == 64 || p.head_dim == 128) &&
         (long long)p.batch * p.tokens * p.q_heads < 0x7fffffffLL;
}

int launch_fwd_sm100(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                     const moba_b200_index& ix, const int32_t* cu, void* part_o, float* part_lse,
                     int part_keys, int* claims, cudaStream_t st) {
  KernelTimer timer__("fwd_sm100_kernel", st);
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("forward: no device error word"); return MOBA_B200_ECUDA; }
  CUtensorMap km, vm;
  const uint64_t rows = (uint64_t)p.batch * p.tokens;
  int rc = encode_rows_map(&km, k, rows, p.kv_heads, p.head_dim, 128);
  if (rc) return rc;
  rc = encode_rows_map(&vm, v, rows, p.kv_heads, p.head_dim, 128);
  if (rc) return rc;
  CUtensorMap qm;
  rc = encode_2d_map(&qm, q, rows * p.q_heads, p.head_dim, 1);
  if (rc) return rc;
  if (ix.work_items == nullptr || ix.items_per_row <= 0) {
    set_error("forward: the index carries no work items (build it with moba_b200_transpose)");
    return MOBA_B200_EINVAL;
  }
  const long long n_items_ll = (long long)ix.items_per_row * p.n_seq * p.kv_heads;
  if (n_items_ll > 0x7fffffffLL) { set_error("forward: too many work items"); return MOBA_B200_EUNSUPPORTED; }
  const int n_items = (int)n_items_ll;
  const int rows_claimed = claims != nullptr ? claim_rows(p, p.head_dim == 64 ? 192 : 48) : 0;
  const ClaimOrder order{rows_claimed > 0 ? claims : nullptr, rows_claimed};
  const bool bf = p.dtype == MOBA_B200_BF16;
#define GO(D, T, TP) return launch_one<D, T, TP>(p, km, vm, qm, ix, cu, part_o, part_lse, part_keys, n_items, order, err, st)
  if (p.head_dim == 64) {
    if (bf) { if (p.part_f32) GO(64, __nv_bfloat16, float); else GO(64, __nv_bfloat16, __nv_bfloat16); }
    else { if (p.part_f32) GO(64, __half, float); else GO(64, __half, __half); }
  } else {
    if (bf) { if (p.part_f32) GO(128, __nv_bfloat16, float); else GO(128, __nv_bfloat16, __nv_bfloat16); }
    else { if (p.part_f32) GO(128, __half, float); else GO(128, __half, __half); }
  }
#undef GO
  return MOBA_B200_OK;
}

}  // namespace moba
