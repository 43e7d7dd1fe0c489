// Backward on tcgen05 tensor cores (bf16/f16, block_size 128, head_dim 64/128).
//
// Persistent CTAs walk the work items (a block and a range of the list of queries that selected
// it), largest first, in alternating direction. The CTA that takes an item accumulates its dK and
// dV in TMEM and stores them once.
//
// Everything is computed transposed: the 128 keys of the block are the rows (TMEM lanes) of S and
// dP, the 128 gathered queries of a tile their columns. P and dS then can be operand A *from TMEM*
// of the two long sums, P never touches shared memory, dS only once, and the freed shared memory
// holds a second gather stage at head_dim 128:
//   S  = K Q^T            A K  (K-major)   B Q  (K-major)   N 128
//   dP = V dO^T           A V  (K-major)   B dO (K-major)   N 128
//   P  = exp2(S c - lse) -> TMEM over S;  dS = P (dP - delta) -> shared memory (and TMEM over dP)
//   dV += P dO            A P  (TMEM)      B dO (N-major)   N D
//   dK += dS Q            A dS (TMEM / shared memory)   B Q  (N-major)   N D
//   dQ  = dS^T K          A dS (M-major)   B K  (N-major)   N D
// TMEM columns: head_dim 64: two S buffers (dQ of a tile lands on its own S buffer once dV has
// read P), dP, dV, dK = 512. head_dim 128: S, dP (dQ lands on it), dV, dK = 512.
//
// Roles: 16 elementwise warps (P and dS), two MMA issuers, four warps that gather Q and dO rows by
// TMA, four that take dQ out of TMEM and store its rows, one loader of K and V. Each tile's P runs
// under the dK / dQ of the tile before. What bounds it (clocks per tile, traces of a debug build):
// with every copy, store and exponential and seven eighths of every MMA left out, the hand-overs
// between the roles and the TMEM loads and stores still take 3 500 of 5 400 at head_dim 64 and
// 4 400 of 7 200 at 128; the tensor pipe needs 1 900 and 2 560. Measured against the untransposed
// version with copies through the load-store unit: 11.0 -> 7.4 ms on 262 144 packed tokens, 16
// heads of 128; 9.1 -> 6.9 ms on [1,131072,32,128] with 8 KV heads. At head_dim 64 it gained nothing
// that can be told from noise ([1,131072,4,64]: 0.667 ms before, 0.65 to 0.67 after); claimed items
// and the register split below make that 0.61.
//
// dQ rows go to the (query, slot) partial buffer; a later pass sums the slots.
//
// Stands in for moba_bwd_kernel of the reference (src/moba/kernels/moba_bwd.py:215-394),
// which splits a block into 64-key sub-tiles for lack of shared memory.
#include "common.cuh"
#include "sm100.cuh"

#include <type_traits>

namespace moba {
using namespace sm100;

namespace {

constexpr int kTile = 128;
constexpr int kSub = kTile * 128;
constexpr int kElemWarps = 16;                           // four query quarters x four key (lane) groups
constexpr int kScoreWarp = kElemWarps, kLoadWarp = kScoreWarp + 1, kGradWarp = kScoreWarp + 2;
constexpr int kGatherWarp0 = kElemWarps + 4, kGatherWarps = 4;
constexpr int kStoreWarp0 = kGatherWarp0 + kGatherWarps, kStoreWarps = 4;
constexpr int kThreads = (kStoreWarp0 + kStoreWarps) * 32;   // warp 19 only completes its warpgroup
// Registers: 896 threads are launched with 72 each (64 512). 512 elementwise threads take 80, 128
// storing threads what a dQ row needs, the other 256 give down to the rest: 64 512 again. At head_dim 64
// a dQ row needs 88; with 104 the other 256 had 40 and spilled 148 bytes (48 now): 624 -> 612 us at [1,131072,4,64].
// At 128 the other 256 spill 84 bytes (180 with a 64-bit division in the walk over the items, and the next item
// taken in two places of the code: the deal took 1 to 3 % longer). Splits that spill less cost more elsewhere: 72,
// 104 and 56 registers (56 bytes) 5 %, 80, 88 and 48 up to 13 %, on dealt and on claimed items.
constexpr int kLaunchRegs = 72, kElemRegs = 80;
template <int D> constexpr int kStoreRegs = D == 64 ? 88 : 104;
template <int D> constexpr int kOtherRegs = D == 64 ? 48 : 40;
template <int D> constexpr bool kRegsFit = kElemWarps * 32 * kElemRegs + kStoreWarps * 32 * kStoreRegs<D> + 256 * kOtherRegs<D> <= kThreads * kLaunchRegs;
static_assert(kRegsFit<64> && kRegsFit<128>, "register split");

template <int D> struct BwdCfg {
  static constexpr int kSubs = D / 64;
  static constexpr int kOperand = kSubs * kSub;          // K, V, one Q stage, one dO stage
  static constexpr int kStages = tensor_core_plan(D).bwd_gather_stages;   // Q / dO gather stages
  static constexpr int kKvBufs = tensor_core_plan(D).bwd_kv_buffers;
  static_assert(kStages <= 2 && kKvBufs <= 2, "barriers for two");
  static constexpr int kSBufs = D == 64 ? 2 : 1;         // S buffers in TMEM
  static constexpr int kDsBytes = 2 * kSub;              // dS tile [keys][queries]; dQ is staged in it too
  static constexpr int kSmemData = 2 * kKvBufs * kOperand + 2 * kStages * kOperand + kDsBytes;
  static constexpr int kBarBytes = D == 64 ? 5632 : 3072;   // barriers and per-stage row data; 227 KB in all at 128
  static constexpr int kSmem = kSmemData + kBarBytes;
  static_assert(kSmem <= 232448, "shared memory of an SM");
  static constexpr uint32_t cS = 0, cDP = 128 * kSBufs, cDV = cDP + 128, cDK = cDV + D;
  static_assert(cDK + D <= 512, "TMEM columns");
};

// dK takes dS from TMEM at head_dim 64 (N = 64: the operand read from shared memory would cost
// more than the MMA). At 128 it takes it from shared memory, which keeps up there, and the dP
// columns are free for dQ as soon as they have been read: dQ can go first.
template <int D> constexpr bool kDsInTmem = (D == 64);

struct Column {
  int kv_row, blk, n, lo, keys, key0, slot;              // slot: dK/dV partial slot, -1 = the item is the whole column
  int tok0;                                              // token axis position of the batch row (0 when packed)
};

struct Meta {                                            // of the queries of one gather stage
  float neg_lse[kTile], delta[kTile];                    // dead queries: -inf (then P = 0) and 0
  uint16_t last[kTile];                                  // last key of the block the query attends
};

template <int D> struct Bars {
  Meta meta[BwdCfg<D>::kStages];
  uint64_t k_full[2], v_full[2], k_free[2], v_free[2];
  uint64_t k_fix[BwdCfg<D>::kKvBufs], v_fix[BwdCfg<D>::kKvBufs];   // per K / V buffer: the rows of a block cut short are zeroed (one for
                                                         // both could complete twice before its first phase is looked at)
  uint64_t q_full[2], q_empty[2], g_full[2], g_empty[2]; // gather stages of Q (with the row data) and dO
  uint64_t s_full[2], dq_full[2], dq_read[2];   // per S buffer: at head_dim 64 two tiles' dQ can be waiting to be stored
  uint64_t p_full[2];                                    // by tiles in turn: with two S buffers P of the next tile may be complete before
                                                         // the issuer has looked at this one's, or while a slow warp still owes its part of it
  uint64_t dp_full, ds_full, p_used, acc_full, acc_read, drain[2];
  uint64_t col_full[4], col_free[4];
  Column cols[4];                                        // ring of item descriptors, published by the loader
  uint8_t masked[2][4];                                  // stage, gather warp: some query does not attend all 128 keys
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(Bars<64>) <= BwdCfg<64>::kBarBytes && sizeof(Bars<128>) <= BwdCfg<128>::kBarBytes, "barrier block outgrew its reservation");

// Work item `j` of a (sequence, kv head) row, in its dispatch order (heaviest first); false for padding.
__device__ __forceinline__ bool load_column(Column& c, int kv_row, int j, const moba_b200_index& ix,
                                            const moba_b200_problem& p, const int32_t* cu) {
  c.kv_row = kv_row;
  WorkItem w;
  if (!load_work_item(w, ix, ix.col_nnz + (size_t)c.kv_row * p.num_blocks, c.kv_row, j)) return false;
  const int seq = c.kv_row / p.kv_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  c.blk = w.blk;
  c.slot = w.slot;
  c.lo = ix.col_offsets[(size_t)c.kv_row * (p.num_blocks + 1) + c.blk] + w.first;
  c.tok0 = p.packed ? 0 : seq * p.tokens;
  c.key0 = sp.bos + c.blk * kTile;
  c.keys = min(kTile, sp.bos + sp.len - c.key0);
  if (c.keys <= 0) return false;                         // a block past the end of a short packed sequence
  c.n = w.n;
  return true;
}

// The work list is sorted longest first; CTAs take it in alternating direction
// (0..G-1, G-1..0, ...) so that no CTA collects the largest column of every round.
__device__ __forceinline__ long long snake_item(int round) {
  const int g = (int)gridDim.x, c = (int)blockIdx.x;
  return (long long)round * g + ((round & 1) ? (g - 1 - c) : c);
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

// 4 x 4 transposes of 16-byte pieces inside every four lanes: afterwards w[4 g + j] of lane l is
// piece 4 g + (l mod 4) of the row of lane (l - l mod 4 + j). Rows come out of TMEM one per lane;
// stored like that, an instruction touches 32 lines, and the stores of a finished column took
// 7 000 clocks. Exchanged, four lanes write 64 contiguous bytes of a row.
template <int N>
__device__ __forceinline__ void transpose_pieces(uint32_t (&w)[N][4], int lane) {
#pragma unroll
  for (int g = 0; g < N / 4; ++g) {
#pragma unroll
    for (int sft = 1; sft <= 2; sft <<= 1) {
      const bool up = (lane & sft) != 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j & sft) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t lo = w[g * 4 + j][k], hi = w[g * 4 + j + sft][k];
          const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, sft);
          w[g * 4 + j][k] = up ? got : lo;
          w[g * 4 + j + sft][k] = up ? hi : got;
        }
      }
    }
  }
}

// Two float32 operations in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "sub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// AND of a predicate over the threads of a role (named barrier `id`): whoever leaves a role's
// loop leaves it together, so that a wait that gave up in some threads cannot leave the others
// alone at a named barrier. The barrier counts warps, whole ones.
__device__ __forceinline__ bool group_all(bool pred, int id, int threads) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, %2, %3, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r) : "r"((uint32_t)pred), "r"(id), "r"(threads) : "memory");
  return r != 0;
}

template <int D, typename T>
__global__ void __launch_bounds__(kThreads, 1)
bwd_sm100_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                 const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap g_map, const float* __restrict__ lse,
                 const float* __restrict__ delta, moba_b200_index ix, const int32_t* __restrict__ cu,
                 T* __restrict__ dq_part, float* __restrict__ dkv_scratch, T* __restrict__ dk, T* __restrict__ dv,
                 moba_b200_problem p, int part_keys, int n_items, ClaimOrder order, unsigned* error_word) {
  using Cfg = BwdCfg<D>;
  constexpr int NST = Cfg::kStages, NKV = Cfg::kKvBufs, NS = Cfg::kSBufs;
  constexpr uint32_t cS = Cfg::cS, cDP = Cfg::cDP, cDV = Cfg::cDV, cDK = Cfg::cDK;
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sK = smem;                                  // NKV buffers
  unsigned char* sV = sK + NKV * Cfg::kOperand;
  unsigned char* sQ = sV + NKV * Cfg::kOperand;              // NST stages
  unsigned char* sG = sQ + NST * Cfg::kOperand;              // dO, NST stages
  unsigned char* sS = sG + NST * Cfg::kOperand;              // dS [keys][queries]; between tiles the 16-bit dQ rows
  Bars<D>* bars = reinterpret_cast<Bars<D>*>(sS + Cfg::kDsBytes);

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
      mbar_init(&bars->s_full[i], 1); mbar_init(&bars->dq_full[i], 1); mbar_init(&bars->dq_read[i], kStoreWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->p_full[i], kElemWarps);
      mbar_init(&bars->q_full[i], kGatherWarps); mbar_init(&bars->g_full[i], kGatherWarps);
      mbar_init(&bars->q_empty[i], 1); mbar_init(&bars->g_empty[i], 2);      // dK (after S); dP and dV, in either order
    }
    for (int i = 0; i < NKV; ++i) { mbar_init(&bars->k_fix[i], kGatherWarps); mbar_init(&bars->v_fix[i], kGatherWarps); }
    for (int i = 0; i < 4; ++i) { mbar_init(&bars->col_full[i], 1); mbar_init(&bars->col_free[i], kElemWarps + 2 + kGatherWarps + kStoreWarps); }
    mbar_init(&bars->dp_full, 1); mbar_init(&bars->ds_full, kElemWarps);
    mbar_init(&bars->acc_full, 1); mbar_init(&bars->acc_read, kElemWarps);
    mbar_init(&bars->p_used, 1); mbar_init(&bars->drain[0], 1); mbar_init(&bars->drain[1], 1);
    // The swizzled operands need a base on a 1024-byte boundary. It is one (there is no static
    // shared memory before it); should that change, nothing may run on it.
    bars->abort = (smem_u32(smem) & 1023u) ? 1 : 0;
    if (bars->abort) atomicOr(error_word, kErrWaitTimeout);
    fence_barrier_init();
  }
  if (warp == kScoreWarp) tmem_alloc(&bars->tmem_base, 512);
  if (warp == kLoadWarp && lane == 0) { tma_prefetch_desc(&k_map); tma_prefetch_desc(&v_map); tma_prefetch_desc(&q_map); tma_prefetch_desc(&g_map); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem = bars->tmem_base;
  const bool sound = bars->abort == 0;

  const float softmax_scale = rsqrtf((float)D);
  const float cs = softmax_scale * kLog2e;
  const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;

  if (warp < kElemWarps) {
    // =========================== elementwise warps ===========================
    // Warp w works on TMEM lanes (keys) [32 (w mod 4), +32) and on query quarter w / 4 of the
    // tile: 32 scores of a key row per thread.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kElemRegs));
    const int wq = warp >> 2, grp = warp & 3;
    const int r = grp * 32 + lane;                     // TMEM lane: key of the block
    const uint32_t lane_off = (uint32_t)(grp * 32) << 16;
    uint32_t t = 0, it = 0, items = 0;
    for (; sound; ++it) {
      const bool col_ok = mbar_wait(&bars->col_full[it & 3], (it >> 2) & 1, wc, 1);
      if (!group_all(col_ok, 1, 32 * kElemWarps)) break;
      const Column c = bars->cols[it & 3];
      mbar_arrive_warp(&bars->col_free[it & 3]);
      if (c.n < 0) break;                              // end of the stream
      const int kvh = c.kv_row % p.kv_heads;
      if (c.n == 0) {                                  // nobody selected this block: exact zeros
        if (r < c.keys && wq < 2) {
          T* base = (wq == 0 ? dv : dk) + ((size_t)(c.tok0 + c.key0 + r) * p.kv_heads + kvh) * (size_t)D;
          for (int i = 0; i < D / 8; ++i) reinterpret_cast<uint4*>(base)[i] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();                                  // a block cut short parts the warp, and a named barrier comes next
        continue;
      }
      const int nt = (c.n + kTile - 1) / kTile;
      for (int i = 0; i < nt; ++i, ++t) {
        const uint32_t st = t % NST;
        mbar_wait(&bars->s_full[t % NS], (t / NS) & 1, wc, 3);
        tc_fence_after();
        const Meta& mt = bars->meta[st];
        // Diagonal block or ragged end: the pairs (key, query) that do not attend are cleared in the
        // packed P and dS, two at a time. `last` and this thread's key are small positive integers,
        // and as such ordered alike when read as half-precision numbers.
        const bool masked = c.keys < kTile || bars->masked[st][wq] != 0;
        const uint32_t key2 = r < c.keys ? (uint32_t)r * 0x10001u : 0x7bff7bffu;   // past the end: after every `last`
        const uint32_t part_mask = (uint32_t)(~(part_keys - 1) & 0xffff) * 0x10001u;   // key -> first key of its block
        auto apply_mask = [&](uint32_t (&w)[8], const uint16_t* last) {
          const uint4 a = *reinterpret_cast<const uint4*>(last), b4 = *reinterpret_cast<const uint4*>(last + 8);
          const uint32_t l[8] = {a.x, a.y, a.z, a.w, b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint32_t m;
            asm("set.le.u32.f16x2 %0, %1, %2;" : "=r"(m) : "r"(key2), "r"(l[k]));
            w[k] &= m;
            if (part_keys < kTile) {                   // a finer block: not before its first key either
              const uint32_t first2 = l[k] & part_mask;
              asm("set.le.u32.f16x2 %0, %1, %2;" : "=r"(m) : "r"(first2), "r"(key2));
              w[k] &= m;
            }
          }
        };
        // ---- P = exp2(S c - lse), kept in registers for dS ----
        float pe[32];
        {
          uint32_t sv[32];
          tmem_ld32(tmem + lane_off + cS + (t % NS) * 128 + wq * 32, sv);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 l4 = *reinterpret_cast<const float4*>(&mt.neg_lse[wq * 32 + g * 4]);
            const float2 a = fma2(make_float2(__uint_as_float(sv[g * 4]), __uint_as_float(sv[g * 4 + 1])), make_float2(cs, cs), make_float2(l4.x, l4.y));
            const float2 e = fma2(make_float2(__uint_as_float(sv[g * 4 + 2]), __uint_as_float(sv[g * 4 + 3])), make_float2(cs, cs), make_float2(l4.z, l4.w));
            pe[g * 4] = ex2(a.x); pe[g * 4 + 1] = ex2(a.y); pe[g * 4 + 2] = ex2(e.x); pe[g * 4 + 3] = ex2(e.y);
          }
          // P of queries [16 k, +16) in the eight columns from 16 k: over scores this thread has read
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t pk[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) pk[k] = pack2<T>(pe[h * 16 + 2 * k], pe[h * 16 + 2 * k + 1]);
            if (masked) apply_mask(pk, mt.last + wq * 32 + h * 16);
            tmem_st8(tmem + lane_off + cS + (t % NS) * 128 + wq * 32 + h * 16, pk);
          }
          tmem_st_wait();
        }
        tc_fence_before();
        mbar_arrive_warp(&bars->p_full[t & 1]);
        // ---- dS = P (dP - delta) ----
        // The dS tile: dQ of the tile before has read it, and at head_dim 128 dK.
        if (t >= 1) {
          mbar_wait(&bars->dq_full[(t - 1) % NS], ((t - 1) / NS) & 1, wc, 5);
          if constexpr (!kDsInTmem<D>) mbar_wait(&bars->q_empty[(t - 1) % NST], ((t - 1) / NST) & 1, wc, 5);
        }
        mbar_wait(&bars->dp_full, t & 1, wc, 4);
        tc_fence_after();
        uint32_t pv[2][16];
        tmem_ld16(tmem + lane_off + cDP + wq * 32, pv[0]);
        tmem_ld16(tmem + lane_off + cDP + wq * 32 + 16, pv[1]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t dsk[8];
          const int col0 = wq * 32 + h * 16;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const float4 d4 = *reinterpret_cast<const float4*>(&mt.delta[col0 + g * 4]);
            const float2 x = mul2(make_float2(pe[h * 16 + g * 4], pe[h * 16 + g * 4 + 1]),
                                  sub2(make_float2(__uint_as_float(pv[h][g * 4]), __uint_as_float(pv[h][g * 4 + 1])), make_float2(d4.x, d4.y)));
            const float2 y = mul2(make_float2(pe[h * 16 + g * 4 + 2], pe[h * 16 + g * 4 + 3]),
                                  sub2(make_float2(__uint_as_float(pv[h][g * 4 + 2]), __uint_as_float(pv[h][g * 4 + 3])), make_float2(d4.z, d4.w)));
            dsk[g * 2] = pack2<T>(x.x, x.y);
            dsk[g * 2 + 1] = pack2<T>(y.x, y.y);
          }
          if (masked) apply_mask(dsk, mt.last + col0);
          unsigned char* s_sub = sS + (wq >> 1) * kSub;       // queries [64 h, 64 h + 64) live in sub-tile h
          const int ch = (wq & 1) * 4 + h * 2;
          *reinterpret_cast<uint4*>(s_sub + swz128(r, ch)) = make_uint4(dsk[0], dsk[1], dsk[2], dsk[3]);
          *reinterpret_cast<uint4*>(s_sub + swz128(r, ch + 1)) = make_uint4(dsk[4], dsk[5], dsk[6], dsk[7]);
          if constexpr (kDsInTmem<D>) tmem_st8(tmem + lane_off + cDP + col0, dsk);
        }
        if constexpr (kDsInTmem<D>) tmem_st_wait();
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive_warp(&bars->ds_full);
      }
      // ---- the item's dV (quarters 0, 1) and dK (quarters 2, 3): half of a key row per thread ----
      const bool acc_ok = mbar_wait(&bars->acc_full, items & 1, wc, 5);
      tc_fence_after();
      {
        constexpr int HC = D / 2;                        // columns of a half
        const uint32_t col = ((wq < 2) ? cDV : cDK) + (wq & 1) * HC;
        const float sc = (wq < 2) ? 1.f : softmax_scale;
        const int r4 = r & ~3;                           // first of the four rows this lane stores pieces of
#pragma unroll 1
        for (int ch = 0; ch < HC / 32; ++ch) {
          uint32_t av[32];
          tmem_ld32(tmem + lane_off + col + ch * 32, av);
          tmem_ld_wait();
          if (c.slot < 0) {                              // the item is the whole column: final values
            uint32_t w[4][4];
#pragma unroll
            for (int k = 0; k < 16; ++k)
              w[k / 4][k % 4] = pack2<T>(__uint_as_float(av[2 * k]) * sc, __uint_as_float(av[2 * k + 1]) * sc);
            transpose_pieces<4>(w, lane);
            T* base = (wq < 2 ? dv : dk) + ((size_t)(c.tok0 + c.key0) * p.kv_heads + kvh) * (size_t)D + (wq & 1) * HC + ch * 32 + (lane & 3) * 8;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (acc_ok && r4 + k < c.keys)
                *reinterpret_cast<uint4*>(base + (size_t)(r4 + k) * p.kv_heads * D) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
          } else {                                       // one of several items of the column: float32 partial
            uint32_t w[8][4];
#pragma unroll
            for (int k = 0; k < 32; ++k) w[k / 4][k % 4] = __float_as_uint(__uint_as_float(av[k]) * sc);
            transpose_pieces<8>(w, lane);
            float* base = dkv_scratch + ((size_t)c.slot * 2 + (wq < 2 ? 0 : 1)) * kTile * D + (wq & 1) * HC + ch * 32 + (lane & 3) * 4;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (acc_ok && r4 + (k & 3) < c.keys)
                *reinterpret_cast<uint4*>(base + (size_t)(r4 + (k & 3)) * D + (k >> 2) * 16) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
          }
        }
      }
      tc_fence_before();
      mbar_arrive_warp(&bars->acc_read);
      ++items;
    }
  } else {
    if (warp >= kStoreWarp0) {
      // ============================ dQ row storers ============================
      // Warp g reads rows [32 g, +32) of every tile's dQ out of TMEM, one row per lane, hands the
      // accumulator back at once and then writes the rows: lanes exchange 16-byte pieces four by
      // four so that four neighbouring lanes write 64 contiguous bytes of a row (one row per lane
      // would touch 32 lines per instruction). Kept off the elementwise warps, whose two phases
      // bound the tile, and off shared memory, which has no room for another tile at 128.
      asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kStoreRegs<D>));
      const int grp = warp & 3, r = grp * 32 + lane;
      const uint32_t lane_off = (uint32_t)(grp * 32) << 16;
      constexpr int CH = D / 8;                            // 16-byte pieces per row
      uint32_t t = 0;
      for (uint32_t it = 0; sound; ++it) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->col_full[it & 3], (it >> 2) & 1, wc, 6))) break;
        const Column c = bars->cols[it & 3];
        mbar_arrive_warp(&bars->col_free[it & 3]);
        if (c.n < 0) break;
        const int nt = (c.n + kTile - 1) / kTile;
        const size_t list0 = (size_t)c.kv_row * ix.capacity + c.lo;
        const size_t b = p.packed ? 0 : (size_t)(c.kv_row / p.kv_heads);
        RawPair nx{0, 0, 0};                               // index entry of the next tile's row, fetched ahead
        if (r < c.n) nx = fetch_pair(ix, list0 + r);
        for (int i = 0; i < nt; ++i, ++t) {
          const int e = i * kTile + r;
          const PairEntry me = pair_of(ix, nx);
          const int dest = e < c.n ? (int)(part_row(p, b, me.head, me.row) * p.slots + me.slot) : -1;
          if (e + kTile < c.n) nx = fetch_pair(ix, list0 + e + kTile);
          const bool dq_ok = __all_sync(0xffffffffu, mbar_wait(&bars->dq_full[t % NS], (t / NS) & 1, wc, 2));
          tc_fence_after();
          const uint32_t cDQ = (D == 64) ? cS + (t % NS) * 128 : cDP;
          uint32_t w[CH][4];
#pragma unroll
          for (int h = 0; h < D / 32; ++h) {
            uint32_t v[32];
            tmem_ld32(tmem + lane_off + cDQ + h * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k)
              w[h * 4 + k / 4][k % 4] = pack2<T>(__uint_as_float(v[2 * k]) * softmax_scale, __uint_as_float(v[2 * k + 1]) * softmax_scale);
          }
          tc_fence_before();
          mbar_arrive_warp(&bars->dq_read[t % NS]);                // the dQ columns may be overwritten
          transpose_pieces<CH>(w, lane);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int to = __shfl_sync(0xffffffffu, dest, (lane & ~3) + j);
            unsigned char* dst = reinterpret_cast<unsigned char*>(dq_part + (size_t)(to < 0 ? 0 : to) * D) + (lane & 3) * 16;
            if (to >= 0 && dq_ok) {
#pragma unroll
              for (int g = 0; g < CH / 4; ++g)
                st_global_stream16(dst + g * 64, make_uint4(w[g * 4 + j][0], w[g * 4 + j][1], w[g * 4 + j][2], w[g * 4 + j][3]));
            }
          }
        }
      }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs<D>));
    if (warp == kScoreWarp || warp == kGradWarp) {
      // ============================== MMA issuers ==============================
      // Two warps feed the tensor core, so that neither waits for what the other's next MMA
      // needs: one issues S and dP (what the elementwise warps read), the other dV, dK and dQ
      // (what they wrote). All 32 lanes run the loop, one issues.
      const bool leader = elect_one();
      const uint32_t fbits = (fmt << 7) | (fmt << 10);
      const uint32_t aS = smem_u32(sS);
      // The CTA's items that have tiles, in order; false at the end of the stream.
      struct Item { int nt; bool partial; uint32_t kb, ku, fix; };
      uint32_t it = 0, n_seen = 0, fixes = 0, t = 0;           // fixes, bit b: parity of the cut-short columns seen in buffer b
      auto next_item = [&](Item& c) -> bool {
        for (;;) {
          if (!sound || !mbar_wait(&bars->col_full[it & 3], (it >> 2) & 1, wc, 20)) return false;
          const int n = bars->cols[it & 3].n, keys = bars->cols[it & 3].keys;
          mbar_arrive_warp(&bars->col_free[it & 3]);
          ++it;
          if (n < 0) return false;
          if (n == 0) continue;
          c.nt = (n + kTile - 1) / kTile; c.partial = keys < kTile;
          c.kb = n_seen % NKV; c.ku = n_seen / NKV; c.fix = fixes >> c.kb & 1;
          ++n_seen;
          if (c.partial) fixes ^= 1u << c.kb;
          return true;
        }
      };
      Item c;
      if (warp == kScoreWarp) {
        const uint32_t id_s = make_idesc(0, 128, 128, 0, 0) | fbits;
        while (next_item(c)) {
          const uint32_t aK = smem_u32(sK) + c.kb * Cfg::kOperand, aV = smem_u32(sV) + c.kb * Cfg::kOperand;
          for (int i = 0; i < c.nt; ++i, ++t) {
            const uint32_t st = t % NST, us = t / NST;
            const uint32_t aQ = smem_u32(sQ) + st * Cfg::kOperand, aG = smem_u32(sG) + st * Cfg::kOperand;
            if (i == 0) {
              mbar_wait(&bars->k_full[c.kb], c.ku & 1, wc, 21);
              if (c.partial) mbar_wait(&bars->k_fix[c.kb], c.fix, wc, 21);
            }
            mbar_wait(&bars->q_full[st], us & 1, wc, 22);
            // the S buffer: two tiles ago its dQ sat there (64); dV of the tile before has read P (128)
            if (NS == 2) { if (t >= 2) mbar_wait(&bars->dq_read[t % NS], (t / NS - 1) & 1, wc, 23); }
            else if (t >= 1) mbar_wait(&bars->p_used, (t - 1) & 1, wc, 23);
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
              const uint32_t o = (ks >> 2) * kSub + (ks & 3) * 32;
              if (leader) umma_f16(tmem + cS + (t % NS) * 128, make_sdesc(aK + o, 16, 1024), make_sdesc(aQ + o, 16, 1024), id_s, ks > 0);
            }
            if (leader) umma_commit(&bars->s_full[t % NS]);
            if (i == 0) {
              mbar_wait(&bars->v_full[c.kb], c.ku & 1, wc, 24);
              if (c.partial) mbar_wait(&bars->v_fix[c.kb], c.fix, wc, 24);
            }
            mbar_wait(&bars->g_full[st], us & 1, wc, 24);
            // the dP columns: dK of the tile before has read dS there (64); its dQ has been read out (128)
            if (t >= 1) {
              if (NS == 2) mbar_wait(&bars->q_empty[(t - 1) % NST], ((t - 1) / NST) & 1, wc, 25);
              else mbar_wait(&bars->dq_read[0], (t - 1) & 1, wc, 25);
            }
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
              const uint32_t o = (ks >> 2) * kSub + (ks & 3) * 32;
              if (leader) umma_f16(tmem + cDP, make_sdesc(aV + o, 16, 1024), make_sdesc(aG + o, 16, 1024), id_s, ks > 0);
            }
            if (leader) { umma_commit(&bars->dp_full); umma_commit(&bars->g_empty[st]); }
            if (i == c.nt - 1 && leader) umma_commit(&bars->v_free[c.kb]);
          }
        }
      } else {
        const uint32_t id_acc = make_idesc(0, 128, D, 0, 1) | fbits;     // dV, dK
        const uint32_t id_dq = make_idesc(0, 128, D, 1, 1) | fbits;      // dQ: A M-major
        while (next_item(c)) {
          const uint32_t aK = smem_u32(sK) + c.kb * Cfg::kOperand;
          for (int i = 0; i < c.nt; ++i, ++t) {
            const uint32_t st = t % NST;
            const uint32_t aQ = smem_u32(sQ) + st * Cfg::kOperand, aG = smem_u32(sG) + st * Cfg::kOperand;
            const uint32_t cP = cS + (t % NS) * 128;
            mbar_wait(&bars->p_full[t & 1], (t >> 1) & 1, wc, 26);
            mbar_wait(&bars->g_full[st], (t / NST) & 1, wc, 26);
            if (i == 0 && n_seen >= 2) mbar_wait(&bars->acc_read, (n_seen - 2) & 1, wc, 27);   // the accumulators have been stored
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)             // 16 queries per step
              if (leader) umma_f16_ts(tmem + cDV, tmem + cP + 16 * ks, make_sdesc(aG + ks * 2048, kSub, 1024), id_acc, (i > 0 || ks > 0));
            if (leader) { umma_commit(&bars->g_empty[st]); if (NS == 1) umma_commit(&bars->p_used); }
            mbar_wait(&bars->ds_full, t & 1, wc, 28);
            tc_fence_after();
            auto issue_dk = [&]() {
#pragma unroll
              for (int ks = 0; ks < 8; ++ks) {         // 16 queries per step
                if (!leader) continue;
                const uint64_t b = make_sdesc(aQ + ks * 2048, kSub, 1024);
                if constexpr (kDsInTmem<D>) umma_f16_ts(tmem + cDK, tmem + cDP + 16 * ks, b, id_acc, (i > 0 || ks > 0));
                else umma_f16(tmem + cDK, make_sdesc(aS + (ks >> 2) * kSub + (ks & 3) * 32, 16, 1024), b, id_acc, (i > 0 || ks > 0));
              }
              if (leader) umma_commit(&bars->q_empty[st]);
            };
            const uint32_t cDQ = (D == 64) ? cP : cDP;
            if constexpr (kDsInTmem<D>) issue_dk();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)             // 16 keys per step
              if (leader) umma_f16(tmem + cDQ, make_sdesc(aS + ks * 2048, kSub, 1024), make_sdesc(aK + ks * 2048, kSub, 1024), id_dq, ks > 0);
            if (leader) umma_commit(&bars->dq_full[t % NS]);
            if constexpr (!kDsInTmem<D>) issue_dk();
            if (i == c.nt - 1 && leader) { umma_commit(&bars->acc_full); umma_commit(&bars->k_free[c.kb]); }
          }
        }
      }
      // Every MMA of this warp has completed before the CTA lets go of its TMEM, also on the way
      // out of a run that gave up on a wait.
      uint64_t* drain = &bars->drain[warp == kScoreWarp ? 0 : 1];
      if (leader) umma_commit(drain);
      mbar_wait_quiet(drain, 0);
      __syncwarp();
    } else if (warp == kLoadWarp) {
      // ================= work-list walker and K/V TMA loader =================
      // All 32 lanes walk the list, lane 0 publishes and issues the loads.
      if (sound) {
        uint32_t it = 0, n_seen = 0;
        const uint64_t keep = l2_policy_evict_last();
        const size_t index_elems = (size_t)n_kv_rows * ix.capacity;
        auto publish = [&](const Column& c) {
          if (it >= 4) mbar_wait(&bars->col_free[it & 3], ((it >> 2) - 1) & 1, wc, 10);
          __syncwarp();
          if (lane == 0) {
            bars->cols[it & 3] = c;
            mbar_arrive(&bars->col_full[it & 3]);
          }
          ++it;
        };
        // The next item that has something to do; false at the end. The lanes look at 32 items at
        // once: most of a packed batch's list is padding.
        Column mine;
        unsigned found = 0;
        int round0 = 0;
        auto take = [&](Column& c, int src) {
          c.kv_row = __shfl_sync(0xffffffffu, mine.kv_row, src); c.blk = __shfl_sync(0xffffffffu, mine.blk, src);
          c.n = __shfl_sync(0xffffffffu, mine.n, src); c.lo = __shfl_sync(0xffffffffu, mine.lo, src);
          c.keys = __shfl_sync(0xffffffffu, mine.keys, src); c.key0 = __shfl_sync(0xffffffffu, mine.key0, src);
          c.slot = __shfl_sync(0xffffffffu, mine.slot, src); c.tok0 = __shfl_sync(0xffffffffu, mine.tok0, src);
          return true;
        };
        auto dealt = [&](Column& c) {
          while (found == 0) {
            if ((long long)round0 * gridDim.x >= n_items) return false;
            const long long item = snake_item(round0 + lane);
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
          do {
            if (!claim_item(walk, order, ix, p, cu, n_kv_rows, kv_row, j)) return false;
          } while (!load_column(c, kv_row, j, ix, p, cu));
          return true;
        };
        auto next = [&](Column& c) { return order.next != nullptr ? claimed(c) : dealt(c); };
        // The index entries of a column are read a tile at a time; asking the L2 for them, and for
        // its K and V blocks, a column ahead saves a DRAM round trip per tile and item.
        auto prefetch = [&](const Column& c) {
          if (c.n <= 0 || lane != 0) return;
          const size_t lo = (size_t)c.kv_row * ix.capacity + c.lo;
          if (packed_pairs(ix)) {
            l2_prefetch_i32(ix.row_indices, 2 * lo, 2 * c.n, 2 * index_elems);
          } else {
            l2_prefetch_i32(ix.row_indices, lo, c.n, index_elems);
            l2_prefetch_i32(ix.head_indices, lo, c.n, index_elems);
            l2_prefetch_i32(ix.slot_of_pair, lo, c.n, index_elems);
          }
          for (int s = 0; s < Cfg::kSubs; ++s) {
            tma_prefetch_3d(&k_map, s * 64, c.kv_row % p.kv_heads, c.tok0 + c.key0);
            tma_prefetch_3d(&v_map, s * 64, c.kv_row % p.kv_heads, c.tok0 + c.key0);
          }
        };
        // One call of `next` (its code twice costs the other roles of this register share spills): each turn takes
        // an item and loads the one taken before.
        Column c, c_next;
        c.n = 0;
        for (;;) {
          const bool more = next(c_next);
          if (more) prefetch(c_next);
          if (__any_sync(0xffffffffu, *wc.abort)) break;   // no new loads once a wait gave up
          if (c.n > 0) {
            const int kvh = c.kv_row % p.kv_heads, tok = c.tok0 + c.key0;
            const uint32_t kb = n_seen % NKV, ku = n_seen / NKV;
            if (ku >= 1) mbar_wait(&bars->v_free[kb], (ku - 1) & 1, wc, 11);
            if (lane == 0) {
              mbar_expect_tx(&bars->v_full[kb], Cfg::kOperand);
              for (int s = 0; s < Cfg::kSubs; ++s)
                tma_load_3d_hint(sV + kb * Cfg::kOperand + s * kSub, &v_map, &bars->v_full[kb], s * 64, kvh, tok, keep);
            }
            if (ku >= 1) mbar_wait(&bars->k_free[kb], (ku - 1) & 1, wc, 12);
            if (lane == 0) {
              mbar_expect_tx(&bars->k_full[kb], Cfg::kOperand);
              for (int s = 0; s < Cfg::kSubs; ++s)
                tma_load_3d_hint(sK + kb * Cfg::kOperand + s * kSub, &k_map, &bars->k_full[kb], s * 64, kvh, tok, keep);
            }
            ++n_seen;
          }
          if (!more) break;
          c = c_next;
          publish(c);
        }
        c.n = -1;
        publish(c);
        // No load may be in flight into this CTA's shared memory when it exits.
        if (lane == 0) {
          for (uint32_t k = 1; k <= (uint32_t)NKV && k <= n_seen; ++k) {
            const uint32_t n = n_seen - k;
            mbar_wait_quiet(&bars->k_full[n % NKV], (n / NKV) & 1);
            mbar_wait_quiet(&bars->v_full[n % NKV], (n / NKV) & 1);
          }
        }
      }
      __syncwarp();
    } else if (warp >= kGatherWarp0) {
      // ========================= query / dO row gatherers =========================
      // Warp g brings in rows [32 g, 32 g + 32) of every tile: one index entry per lane, eight
      // lanes issuing TMA gathers of four rows each. The copies go past the load-store unit,
      // which with 16-byte asynchronous copies spent 2 500 (head_dim 64) to 6 000 clocks (128) of
      // every tile on them and held up every other load and store of the SM meanwhile (it keeps
      // about 24 KB outstanding; a gather of 32 or 64 KB fills that for a memory latency or two).
      const int gw = warp - kGatherWarp0, pt = gw * 32 + lane;
      const int n_rows = p.batch * p.tokens * p.q_heads;
      uint32_t t = 0, n_seen = 0;
      for (uint32_t it = 0; sound; ++it) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->col_full[it & 3], (it >> 2) & 1, wc, 13))) break;
        const Column c = bars->cols[it & 3];
        mbar_arrive_warp(&bars->col_free[it & 3]);
        if (c.n < 0) break;
        if (c.n == 0) continue;
        const int nt = (c.n + kTile - 1) / kTile;
        const uint32_t kb = n_seen % NKV, ku = n_seen / NKV;
        const size_t list0 = (size_t)c.kv_row * ix.capacity + c.lo;
        const size_t b = p.packed ? 0 : (size_t)(c.kv_row / p.kv_heads);
        RawPair nx{0, 0, 0};                                 // index entry of the next tile, fetched ahead
        if (pt < c.n) nx = fetch_pair(ix, list0 + pt);
        if (c.keys < kTile) {                                // zero the rows of a block its sequence cuts short
          const int dead = kTile - c.keys;
          mbar_wait(&bars->v_full[kb], ku & 1, wc, 14);
          for (int i = pt; i < dead * 8 * Cfg::kSubs; i += 32 * kGatherWarps) {
            const int s = i / (dead * 8), rr = c.keys + (i % (dead * 8)) / 8, ch = i % 8;
            *reinterpret_cast<uint4*>(sV + kb * Cfg::kOperand + s * kSub + rr * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async();
          mbar_arrive_warp(&bars->v_fix[kb]);
          mbar_wait(&bars->k_full[kb], ku & 1, wc, 14);
          for (int i = pt; i < dead * 8 * Cfg::kSubs; i += 32 * kGatherWarps) {
            const int s = i / (dead * 8), rr = c.keys + (i % (dead * 8)) / 8, ch = i % 8;
            *reinterpret_cast<uint4*>(sK + kb * Cfg::kOperand + s * kSub + rr * 128 + ch * 16) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async();
          mbar_arrive_warp(&bars->k_fix[kb]);
        }
        ++n_seen;
        int i = 0;
        for (; i < nt; ++i, ++t) {
          const uint32_t st = t % NST, us = t / NST;
          const int e = i * kTile + pt;
          const bool live = e < c.n;
          const PairEntry me = pair_of(ix, nx);
          int row_id = n_rows;                               // a row past the end of the tensor: zeros
          float l = INFINITY, dl = 0.f;                      // a dead query: P = exp2(0 - inf) = 0
          uint32_t last = kTile - 1;
          if (live) {
            row_id = (int)((b * p.tokens + me.row) * p.q_heads + me.head);
            const size_t qr = (b * p.q_heads + me.head) * p.tokens + me.row;
            l = ld_nc_pinned_f(lse + qr);
            dl = ld_nc_pinned_f(delta + qr);
            last = (uint32_t)((me.part + 1) * part_keys - 1);
            const int own = me.row - c.key0;                 // the query's own place, if it lies in the column
            if (p.causal && own >= 0 && own < (int)last) last = (uint32_t)own;
          }
          if (e + kTile < c.n) nx = fetch_pair(ix, list0 + e + kTile);
          int rows[4];                                       // the four rows lane gathers (lanes 0..7)
#pragma unroll
          for (int k = 0; k < 4; ++k) rows[k] = __shfl_sync(0xffffffffu, row_id, (lane * 4 + k) & 31);
          // dO before Q: its stage frees first (after dV), and its copies run while the tile that
          // still holds the Q stage finishes
          const uint32_t o = (gw * 32 + lane * 4) * 128;
          if (us >= 1) mbar_wait(&bars->g_empty[st], (us - 1) & 1, wc, 15);
          if (__any_sync(0xffffffffu, *wc.abort)) break;     // no new copies once a wait gave up
          if (lane == 0) mbar_expect_tx(&bars->g_full[st], 32 * D * 2);
          __syncwarp();
          if (lane < 8) {
#pragma unroll
            for (int h = 0; h < Cfg::kSubs; ++h)
              tma_gather4(sG + st * Cfg::kOperand + h * kSub + o, &g_map, &bars->g_full[st], h * 64, rows[0], rows[1], rows[2], rows[3]);
          }
          __syncwarp();
          if (us >= 1) mbar_wait(&bars->q_empty[st], (us - 1) & 1, wc, 16);
          Meta& mt = bars->meta[st];
          mt.neg_lse[pt] = -l;
          mt.delta[pt] = dl;
          mt.last[pt] = (uint16_t)last;
          const bool any = __any_sync(0xffffffffu, last != kTile - 1) || part_keys < kTile;
          if (lane == 0) bars->masked[st][gw] = any ? 1 : 0;
          __syncwarp();
          if (lane == 0) mbar_expect_tx(&bars->q_full[st], 32 * D * 2);     // releases the row data, too
          __syncwarp();
          if (lane < 8) {
#pragma unroll
            for (int h = 0; h < Cfg::kSubs; ++h)
              tma_gather4(sQ + st * Cfg::kOperand + h * kSub + o, &q_map, &bars->q_full[st], h * 64, rows[0], rows[1], rows[2], rows[3]);
          }
          __syncwarp();
        }
        if (i < nt) break;
      }
      // No copy may be in flight into this CTA's shared memory when it exits.
      for (uint32_t k = 1; k <= (uint32_t)NST && k <= t; ++k) {
        mbar_wait_quiet(&bars->g_full[(t - k) % NST], ((t - k) / NST) & 1);
        mbar_wait_quiet(&bars->q_full[(t - k) % NST], ((t - k) / NST) & 1);
      }
    }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kScoreWarp) tmem_dealloc(tmem, 512);
}

// dK / dV of the columns that were cut into several work items. CTA (x, y) looks at 256
// consecutive work items of one (sequence, kv head) row, one per thread, and of the first
// items of split columns it finds there takes every gridDim.y-th, starting at y, and of
// each such column the z-th part of its sums: it adds the column's float32 partials in item
// order and stores the result. Split columns are the heaviest ones and therefore neighbours in
// the dispatch order, hence the slicing; most CTAs find nothing and leave.
constexpr int kReduceSlices = 16;                       // at most; fewer when the rows give CTAs enough
template <int D, typename T>
__global__ void __launch_bounds__(256)
dkv_reduce_kernel(const float* __restrict__ dkv_scratch, moba_b200_index ix, const int32_t* __restrict__ cu,
                  T* __restrict__ dk, T* __restrict__ dv, moba_b200_problem p, int ctas_per_row) {
  __shared__ int4 found[256];
  __shared__ int n_found;
  pdl_wait();
  pdl_trigger();                                         // behind the wait: the dQ sums may start beside this kernel
  const int kv_row = blockIdx.x / ctas_per_row;
  const int j = (blockIdx.x % ctas_per_row) * 256 + threadIdx.x;
  if (threadIdx.x == 0) n_found = 0;
  __syncthreads();
  int4 it = make_int4(0, 0, 0, -2);
  if (j < ix.items_per_row)
    it = __ldg(reinterpret_cast<const int4*>(ix.work_items) + (size_t)kv_row * ix.items_per_row + j);
  const bool first = it.w >= 0 && it.y == 0;               // the first item of a split column
  // position among the CTA's finds, in item order (so that the slices are the same on every run)
  const unsigned ballot = __ballot_sync(0xffffffffu, first);
  __shared__ int warp_finds[8];
  if ((threadIdx.x & 31) == 0) warp_finds[threadIdx.x >> 5] = __popc(ballot);
  __syncthreads();
  int before = __popc(ballot & ((1u << (threadIdx.x & 31)) - 1u));
  for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) before += warp_finds[w];
  if (first) found[before] = it;
  if (threadIdx.x == 255) n_found = before + (first ? 1 : 0);
  __syncthreads();
  const int seq = kv_row / p.kv_heads, kvh = kv_row % p.kv_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const size_t b = p.packed ? 0 : (size_t)seq;
  for (int f = blockIdx.y; f < n_found; f += (int)gridDim.y) {
    const int4 col = found[f];
    const int nnz = ix.col_nnz[(size_t)kv_row * p.num_blocks + col.x];
    const int tiles = (nnz + kTile - 1) / kTile;
    const int n_chunks = (tiles + ix.chunk_tiles - 1) / ix.chunk_tiles;
    const int key0 = sp.bos + col.x * kTile;
    const int keys = min(kTile, sp.bos + sp.len - key0);
    constexpr int V4 = D / 4;                              // float4 per row
    constexpr int kAhead = 2, kDeep = 4;                   // elements per thread and partials of each in flight
    for (int i0 = (int)blockIdx.z * 256 * kAhead + threadIdx.x; i0 < 2 * kTile * V4; i0 += 256 * kAhead * (int)gridDim.z) {
      float4 acc[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int c0 = 0; c0 < n_chunks; c0 += kDeep) {       // loads first, then the sums in item order
        float4 x[kDeep][kAhead];
#pragma unroll
        for (int d = 0; d < kDeep; ++d) {
#pragma unroll
          for (int u = 0; u < kAhead; ++u) {
            const int i = i0 + u * 256;
            const int which = i / (kTile * V4), row = (i / V4) % kTile, c4 = i % V4;
            x[d][u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row >= keys || which > 1 || c0 + d >= n_chunks) continue;
            x[d][u] = __ldcs(reinterpret_cast<const float4*>(
                dkv_scratch + (((size_t)(col.w + c0 + d) * 2 + which) * kTile + row) * D) + c4);
          }
        }
#pragma unroll
        for (int d = 0; d < kDeep; ++d) {
#pragma unroll
          for (int u = 0; u < kAhead; ++u) {
            if (c0 + d >= n_chunks) continue;
            acc[u].x += x[d][u].x; acc[u].y += x[d][u].y; acc[u].z += x[d][u].z; acc[u].w += x[d][u].w;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = i0 + u * 256;
        const int which = i / (kTile * V4), row = (i / V4) % kTile, c4 = i % V4;
        if (row >= keys) continue;
        T* dst = (which == 0 ? dv : dk) + ((b * p.tokens + key0 + row) * p.kv_heads + kvh) * (size_t)D + c4 * 4;
        uint2 w;
        w.x = pack2<T>(acc[u].x, acc[u].y);
        w.y = pack2<T>(acc[u].z, acc[u].w);
        *reinterpret_cast<uint2*>(dst) = w;
      }
    }
  }
}

template <int D, typename T>
int launch_one(const moba_b200_problem& p, const CUtensorMap& km, const CUtensorMap& vm, const CUtensorMap& qm,
               const CUtensorMap& gm, const float* lse, const float* delta, const moba_b200_index& ix,
               const int32_t* cu, void* dq_part, float* dkv_scratch, void* dk, void* dv, int part_keys, bool* reduces, int n_items, const ClaimOrder& order, unsigned* err,
               cudaStream_t st) {
  const int sms = sm_count();
  const int grid = n_items < sms ? n_items : sms;
  {
    KernelTimer timer__("bwd_sm100_kernel", st);
    auto kern = bwd_sm100_kernel<D, T>;
    static SmemLimit limit;
    if (int rc = raise_smem_limit(limit, (const void*)kern, BwdCfg<D>::kSmem)) return rc;
    MOBA_CUDA_OK(launch_chained(kern, grid, kThreads, BwdCfg<D>::kSmem, st, km, vm, qm, gm, lse, delta,
                                ix, cu, (T*)dq_part, dkv_scratch, (T*)dk, (T*)dv, p, part_keys, n_items, order, err));
  }
  // No column can be long enough to be cut: nothing to sum.
  // (a query lists a column once per block in it)
  const long long longest = ((long long)(p.q_heads / p.kv_heads) * window_rows_of_seq(p) * (kTile / part_keys) + kTile - 1) / kTile;
  if (longest <= ix.chunk_tiles) return MOBA_B200_OK;
  *reduces = true;
  KernelTimer timer__("dkv_reduce_kernel", st);
  const int ctas_per_row = (ix.items_per_row + 255) / 256;
  // z: the 2 x 128 x D sums of a column in parts of at least 1024 float4; fewer parts when the
  // rows alone give CTAs enough (every CTA first looks through its 256 items)
  const int x_ctas = ctas_per_row * p.n_seq * p.kv_heads;
  int slices = 4096 / x_ctas;
  slices = slices < 1 ? 1 : (slices > kReduceSlices ? kReduceSlices : slices);
  int parts = 4096 / (x_ctas * slices);
  parts = parts < 1 ? 1 : (parts > D / 16 ? D / 16 : parts);
  MOBA_CUDA_OK(launch_chained(dkv_reduce_kernel<D, T>, dim3(x_ctas, slices, parts), 256, 0, st, (const float*)dkv_scratch, ix, cu,
                              (T*)dk, (T*)dv, p, ctas_per_row));
  return MOBA_B200_OK;
}

}  // namespace

bool bwd_sm100_supported(const moba_b200_problem& p) {
  return (p.dtype == MOBA_B200_BF16 || p.dtype == MOBA_B200_F16) && p.block_size == 128 &&
         (p.head_dim == 64 || p.head_dim == 128) && (long long)p.batch * p.tokens * p.q_heads < 0x7fffffffLL;
}

int launch_bwd_sm100(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                     const void* dout, const float* lse, const float* delta, const moba_b200_index& ix,
                     const int32_t* cu, void* dq_part, float* dkv_scratch, void* dk, void* dv, int part_keys, int* claims, bool* reduces,
                     cudaStream_t st) {
  *reduces = false;
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("backward: no device error word"); return MOBA_B200_ECUDA; }
  CUtensorMap km, vm;
  const uint64_t rows = (uint64_t)p.batch * p.tokens;
  int rc = encode_rows_map(&km, k, rows, p.kv_heads, p.head_dim, 128);
  if (rc) return rc;
  rc = encode_rows_map(&vm, v, rows, p.kv_heads, p.head_dim, 128);
  if (rc) return rc;
  CUtensorMap qm, gm;
  rc = encode_2d_map(&qm, q, rows * p.q_heads, p.head_dim, 1);
  if (rc) return rc;
  rc = encode_2d_map(&gm, dout, rows * p.q_heads, p.head_dim, 1);
  if (rc) return rc;
  if (ix.work_items == nullptr || ix.items_per_row <= 0 || ix.chunk_tiles <= 0) {
    set_error("backward: the index carries no work items (build it with moba_b200_transpose)");
    return MOBA_B200_EINVAL;
  }
  if (dkv_scratch == nullptr) { set_error("backward: dkv_scratch is NULL"); return MOBA_B200_EINVAL; }
  const long long n_items_ll = (long long)ix.items_per_row * p.n_seq * p.kv_heads;
  if (n_items_ll > 0x7fffffffLL) { set_error("backward: too many work items"); return MOBA_B200_EUNSUPPORTED; }
  const int n_items = (int)n_items_ll;
  const int rows_claimed = claims != nullptr ? claim_rows(p, p.head_dim == 64 ? 192 : 96) : 0;
  const ClaimOrder order{rows_claimed > 0 ? claims : nullptr, rows_claimed};
  const bool bf = p.dtype == MOBA_B200_BF16;
  if (p.head_dim == 64) {
    if (bf) return launch_one<64, __nv_bfloat16>(p, km, vm, qm, gm, lse, delta, ix, cu, dq_part, dkv_scratch, dk, dv, part_keys, reduces, n_items, order, err, st);
    return launch_one<64, __half>(p, km, vm, qm, gm, lse, delta, ix, cu, dq_part, dkv_scratch, dk, dv, part_keys, reduces, n_items, order, err, st);
  }
  if (bf) return launch_one<128, __nv_bfloat16>(p, km, vm, qm, gm, lse, delta, ix, cu, dq_part, dkv_scratch, dk, dv, part_keys, reduces, n_items, order, err, st);
  return launch_one<128, __half>(p, km, vm, qm, gm, lse, delta, ix, cu, dq_part, dkv_scratch, dk, dv, part_keys, reduces, n_items, order, err, st);
}

}  // namespace moba
