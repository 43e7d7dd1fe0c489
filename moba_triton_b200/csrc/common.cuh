// Shared declarations for the MoBA sm_100a engine: the problem record, dtype
// traits, error plumbing and the launch functions each translation unit exports
// to api.cu.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/moba_b200.h"

namespace moba {

constexpr float kLog2e = 1.4426950408889634f;

void set_error(const char* fmt, ...);

#define MOBA_CUDA_OK(expr)                                                        \
  do {                                                                            \
    cudaError_t e__ = (expr);                                                     \
    if (e__ != cudaSuccess) {                                                     \
      ::moba::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), \
                        __FILE__, __LINE__);                                      \
      return MOBA_B200_ECUDA;                                                     \
    }                                                                             \
  } while (0)

#define MOBA_TRY(expr) do { int rc__ = (expr); if (rc__ != MOBA_B200_OK) return rc__; } while (0)

// Counts every kernel launch of the library and, when profiling is switched on
// through moba_b200_profile_enable(), brackets it with CUDA events on its stream.
struct KernelTimer {
  KernelTimer(const char* name, cudaStream_t st);
  ~KernelTimer();
  const char* name_;
  cudaStream_t st_;
  cudaEvent_t start_;
  bool on_;
};

#define MOBA_LAUNCH_OK(what)                                                      \
  do {                                                                            \
    cudaError_t e__ = cudaGetLastError();                                         \
    if (e__ != cudaSuccess) {                                                     \
      ::moba::set_error("launch of %s failed: %s", what, cudaGetErrorString(e__));\
      return MOBA_B200_ECUDA;                                                     \
    }                                                                             \
  } while (0)

// ---- programmatic dependent launch ----------------------------------------
// The op is a chain of kernels, each reading what the one before wrote. Every kernel of the
// chain is launched with programmatic stream serialisation: it may be scheduled while its
// predecessor still runs, does its private set-up, and then waits (pdl_wait, executed by every
// thread before the first global access) until the predecessor has completed and its writes are
// visible. Completion of a kernel implies completion of everything before it, because it waited
// too. A launch then costs the chain about a microsecond instead of three, which is most of the
// time of a short sequence.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the stream be scheduled as soon as every CTA of this one got here.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static inline cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                         Args&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Raises a kernel's dynamic shared-memory limit once per device. `done` is the caller's static
// table (one entry per device), so that repeated launches cost a comparison.
struct SmemLimit { int bytes[64] = {0}; };
int raise_smem_limit(SmemLimit& done, const void* kernel, size_t bytes);
int sm_count();                              // SMs of the current device (cached)

// ---- element types -------------------------------------------------------
template <typename T> struct Elem;
template <> struct Elem<float> {
  static __device__ __forceinline__ float to_f(float x) { return x; }
  static __device__ __forceinline__ float from_f(float x) { return x; }
  static __device__ __forceinline__ float round_f(float x) { return x; }
};
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
  static __device__ __forceinline__ float round_f(float x) {
    return __bfloat162float(__float2bfloat16_rn(x));
  }
};
template <> struct Elem<__half> {
  static __device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f(float x) { return __float2half_rn(x); }
  static __device__ __forceinline__ float round_f(float x) {
    return __half2float(__float2half_rn(x));
  }
};

static inline size_t dtype_size(int dtype) { return dtype == MOBA_B200_F32 ? 4 : 2; }

// Sequence geometry shared by every kernel: where sequence `seq` starts on the
// token axis and how long it is. Padded batches have n_seq == batch and every
// sequence is `tokens` long; packed batches read cu_seqlens.
struct SeqSpan {
  int bos;   // first token (index on the token axis of its batch row)
  int len;   // tokens in the sequence
};
__device__ __forceinline__ SeqSpan seq_span(const int32_t* cu, int packed, int seq, int tokens) {
  SeqSpan s;
  if (packed) {
    s.bos = cu[seq];
    s.len = cu[seq + 1] - s.bos;
  } else {
    s.bos = 0;
    s.len = tokens;
  }
  return s;
}

// ---- gate candidates ----
// Block `blk` is a candidate of a query whose own block is `own`: strictly past, and, when a
// candidate window is set, among the first gate_sinks blocks or the last gate_window before
// the own block.
__host__ __device__ inline bool gate_candidate(const moba_b200_problem& p, int blk, int own) {
  return blk < own && (p.gate_window <= 0 || blk < p.gate_sinks || blk >= own - p.gate_window);
}

// ---- query window: rows of the partial buffers ----
// A call may cover only the query rows [win_begin, win_begin + win_rows) of every batch row
// (host-side chunking along the query axis: the partial buffers, slots times the size of the
// output, then exist for one window at a time). Row (b, head, row) of part_o / part_lse /
// dq_part:
__host__ __device__ inline int window_rows(const moba_b200_problem& p) { return p.win_rows > 0 ? p.win_rows : p.tokens; }
// rows of a sequence that a call can list: a bound of a column's pairs per query head
static inline int window_rows_of_seq(const moba_b200_problem& p) { return p.win_rows > 0 ? p.win_rows : p.max_seqlen; }
__device__ __forceinline__ size_t part_row(const moba_b200_problem& p, size_t b, int head, int row) {
  return (b * p.q_heads + head) * (size_t)window_rows(p) + (size_t)(row - p.win_begin);
}

// ---- launch table of the tensor-core kernels: one tile plan per head_dim ----
// The kernels take their compile-time constants from this table, and moba_b200_launch_plan
// reports it, so there is one place that says what runs. Shared memory decides the entries:
// at head_dim 64 four tiles, four Q stages and double-buffered K/V fit beside the output
// staging tiles; at 128 every operand is twice as large.
struct TensorCorePlan {
  int head_dim;
  int fwd_tiles_in_flight, fwd_q_stages;
  int bwd_kv_buffers, bwd_gather_stages;
};
constexpr TensorCorePlan kTensorCorePlans[2] = {
    {64, 4, 4, 2, 2},
    {128, 2, 2, 1, 2},
};
constexpr const TensorCorePlan& tensor_core_plan(int head_dim) { return kTensorCorePlans[head_dim == 64 ? 0 : 1]; }

void transpose_plan(const moba_b200_problem& p, int* chunk_rows, int* chunks, int* scatter_warps);

constexpr int kBlockKeys = 128;              // keys of a column of the tensor-core kernels

// ---- scheduling: columns are dispatched as work items of at most chunk_tiles tiles ----
// Sizes are fixed functions of the problem record, so that the caller can allocate the
// item table and the dK/dV partial slots without reading anything back from the device.
constexpr int kSchedSMs = 148;               // the part this engine is written for
constexpr int kSchedSplit = 4;               // a column above total / (kSchedSplit * SMs) tiles is cut
constexpr int kMinChunkTiles = 8;

static inline long long sched_pairs_bound(const moba_b200_problem& p) {
  return (long long)p.batch * (p.win_rows > 0 ? p.win_rows : p.tokens) * p.q_heads * p.slots;   // every (query head, slot) pair
}
static inline int sched_chunk_tiles(const moba_b200_problem& p) {
  if (p.chunk_tiles > 0) return p.chunk_tiles;
  const long long tiles = (sched_pairs_bound(p) + 127) / 128;
  const long long t = (tiles + kSchedSplit * kSchedSMs - 1) / (kSchedSplit * kSchedSMs);
  return t < kMinChunkTiles ? kMinChunkTiles : (int)(t > 0x3fffffff ? 0x3fffffff : t);
}
// Items beyond one per column: a column of n entries adds ceil(tiles / Tc) - 1 <= n / (128 Tc).
static inline long long sched_extra_items(const moba_b200_problem& p) {
  return sched_pairs_bound(p) / (128LL * sched_chunk_tiles(p)) + 1;
}
static inline long long sched_items_per_row(const moba_b200_problem& p) { return p.num_blocks + sched_extra_items(p); }
// dK/dV partial slots: a split column of c items uses c slots, and c <= 2 (c - 1).
static inline long long sched_part_slots(const moba_b200_problem& p) { return 2 * sched_extra_items(p) + 1; }
static inline size_t sched_dkv_scratch_bytes(const moba_b200_problem& p) {
  return (size_t)sched_part_slots(p) * 2 * 128 * p.head_dim * sizeof(float);
}

// One pair of a column's list. Inside the whole-op entry points, where no caller looks at the
// index, the pairs are packed into eight bytes {query position, query head << 12 | part << 8 |
// slot}, so that building and reading the list moves one word per pair: `row_indices` then points
// at those and `head_indices` is NULL.
// `part`: with blocks finer than 128 keys the tensor-core kernels work on columns of 128 keys,
// each of 128 / block_size blocks, and a pair names the block of its column it is for.
struct PairEntry { int row, head, slot, part; };
__host__ __device__ __forceinline__ int pack_pair(int head, int part, int slot) { return (head << 12) | (part << 8) | slot; }
__host__ __device__ __forceinline__ bool packed_pairs(const moba_b200_index& ix) { return ix.head_indices == nullptr; }
__device__ __forceinline__ PairEntry load_pair(const moba_b200_index& ix, size_t at) {
  PairEntry e;
  if (packed_pairs(ix)) {
    const int2 v = __ldg(reinterpret_cast<const int2*>(ix.row_indices) + at);
    e.row = v.x; e.head = v.y >> 12; e.part = (v.y >> 8) & 15; e.slot = v.y & 0xff;
  } else {
    e.part = 0;
    e.row = __ldg(ix.row_indices + at); e.head = __ldg(ix.head_indices + at); e.slot = __ldg(ix.slot_of_pair + at);
  }
  return e;
}
// Fetching an entry a tile ahead: the loads may not be moved (a plain load may be sunk to its
// first use), and nothing looks at the words before `pair_of` (unpacking them at once would wait
// for the load: a memory latency per tile, which had cost the attention kernels 3 to 8 %).
struct RawPair { int a, b, c; };
__device__ __forceinline__ RawPair fetch_pair(const moba_b200_index& ix, size_t at) {
  RawPair r{0, 0, 0};
  if (packed_pairs(ix)) {
    asm volatile("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(r.a), "=r"(r.b) : "l"(reinterpret_cast<const int2*>(ix.row_indices) + at));
  } else {
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(r.a) : "l"(ix.row_indices + at));
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(r.b) : "l"(ix.head_indices + at));
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(r.c) : "l"(ix.slot_of_pair + at));
  }
  return r;
}
__device__ __forceinline__ PairEntry pair_of(const moba_b200_index& ix, const RawPair& r) {
  return packed_pairs(ix) ? PairEntry{r.a, r.b >> 12, r.b & 0xff, (r.b >> 8) & 15} : PairEntry{r.a, r.b, r.c, 0};
}

// One work item as the kernels see it.
struct WorkItem {
  int blk;        // block (column) of the (sequence, kv head) row
  int first;      // first entry of the column's pair list this item covers
  int n;          // entries it covers (0: an empty column)
  int slot;       // dK/dV partial slot, -1: the item is the whole column
};
// Item `j` of row `kv_row`; false for padding. `col_nnz_row` is the row's col_nnz.
__device__ __forceinline__ bool load_work_item(WorkItem& w, const moba_b200_index& ix, const int32_t* col_nnz_row,
                                               int kv_row, int j) {
  const int4 it = __ldg(reinterpret_cast<const int4*>(ix.work_items) + (size_t)kv_row * ix.items_per_row + j);
  if (it.w == -2) return false;
  w.blk = it.x;
  w.first = it.y * 128;
  const int nnz = col_nnz_row[it.x];
  w.n = max(0, min(it.z * 128, nnz - w.first));
  w.slot = it.w;
  return true;
}

// ---- claimed items: which item a CTA takes next, by a counter instead of a fixed deal ----
// The items of `rows` neighbouring (sequence, kv head) rows are interleaved, each row's heaviest first, one
// group of rows after the other. What is claimed are items, not entries of the table: sequences of unequal
// lengths have several entries of padding to an item, and each that a claim met cost a round trip to the counter
// and to the table (4 heads of 64 over 4 sequences, forward dealt and claimed: 200 tiles per SM 1.13 -> 1.01,
// 300 1.11 -> 0.97; over one sequence nothing changed).
struct ClaimOrder {
  int* next;                 // counter of claims, zero before the launch; NULL: the fixed deal
  int rows;                  // of a group, at most 32
};
// The group of rows a warp claims from: its first row, and how many items the groups before it have.
struct ClaimWalk { int first, before; };
// Claims the next item for the warp: row and place of it in its row; false when there are no more.
__device__ __forceinline__ bool claim_item(ClaimWalk& w, const ClaimOrder& order, const moba_b200_index& ix,
                                           const moba_b200_problem& p, const int32_t* cu, int n_rows, int& kv_row, int& j) {
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(order.next, 1);
  // Items of the lane's row: its full pieces, which the padding at its end counts, and one for each block of its
  // sequence. (Read again with every claim, beside the counter: kept in registers they cost the backward spills.)
  int mine = 0, all;
  for (;;) {
    const int row = w.first + lane;
    if (lane < order.rows && row < n_rows) {
      const int pieces = __ldg(ix.work_items + ((size_t)(row + 1) * ix.items_per_row - 1) * 4 + 1);
      mine = pieces + (seq_span(cu, p.packed, row / p.kv_heads, p.tokens).len + kBlockKeys - 1) / kBlockKeys;
    }
    all = __reduce_add_sync(0xffffffffu, mine);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at < w.before + all) break;
    if (w.first + order.rows >= n_rows) return false;
    w.before += all;
    w.first += order.rows;
    mine = 0;
  }
  // The last place j with no more than `at` items before it: every row has min(mine, j) of those.
  at -= w.before;
  int hi = __reduce_max_sync(0xffffffffu, mine);
  j = 0;
  while (hi - j > 1) {
    const int mid = (j + hi) >> 1;
    if ((int)__reduce_add_sync(0xffffffffu, min(mine, mid)) <= at) j = mid; else hi = mid;
  }
  at -= __reduce_add_sync(0xffffffffu, min(mine, j));
  const unsigned there = __ballot_sync(0xffffffffu, mine > j);
  kv_row = w.first + __ffs((int)__ballot_sync(0xffffffffu, mine > j && __popc(there & ((1u << lane) - 1u)) == at)) - 1;
  return true;
}
// Rows of a group, 0 for the fixed deal.
// A CTA claims its next item when it begins one, and may then hold it while others have none. So a problem needs
// `tiles_per_sm` tiles per SM for claims to pay (192 at head_dim 64; 48 in the forward and 96 in the backward at
// 128), and six times those of a column, the size of the items that are left at the end. Kernel time, claimed over
// dealt, forward and backward, of one padded sequence by its tiles per SM (q heads on kv heads):
//                          60         75         110        160        220        300        440
//   head_dim 128   4 on 4  1.00 0.96  1.00 0.96  0.99 0.94  0.98 0.92  0.99 0.93  0.96 0.88  0.99 0.95
//                  4 on 1  1.13 1.07  1.09 1.03  1.04 1.01  1.00 1.00  1.01 1.00  0.99 0.94  0.99 0.96
//                 16 on 1  1.02 0.99  1.01 0.99  1.04 1.02  1.14 1.07  1.07 1.04  1.11 1.03  1.04 1.06
//   head_dim 64    4 on 4  1.03 1.01             1.03 0.96  1.00 0.96  0.98 0.95  0.96 0.95  0.99 0.96
//                  4 on 1  1.13 1.10             1.08 1.04  1.03 1.02  1.01 1.00  1.00 0.97  1.01 0.99
//                 16 on 1  0.99 1.01             1.05 1.04  1.09 1.07  1.08 1.09  1.05 1.06  1.06 1.05
// (524288 x 32 on 8 of 128, skewed, 7000 tiles per SM: 0.96 0.97.) The deal is even where all rows are equally
// long. Over a batch of unequal sequences it is off by a tenth to a half whatever the column, and the second
// condition does not apply: 16 on 1 of 128 over 8 sequences, 60 to 440 tiles per SM, 0.43 to 0.98; 8 on 2 of 64 over
// 4 or 8, 200 to 480, 0.56 to 1.05. Two sequences are nearer to one: 16 on 2, 110 to 300, 0.99 to 1.15.
// (Claiming one further ahead, to hide the claim's latency, was 2 to 10 % slower than that.)
// As a rule all rows are one group: its last items are its smallest. Where the queries of all rows are far more than
// the L2 and those of a few are not, groups of 48 MB keep them there while their columns gather them once per
// selected block: 262144 tokens in 32 sequences, 16 heads of 128, 4114 -> 3776, 7963 -> 7437 us. The items of the
// last group are then not small, and there have to be many more than they hold. Time in groups over that without
// (dealt, or claimed over all rows), least and most of packed batches of 12000 to 180000 tokens in 8, 16 and 32
// sequences, 16 to 64 heads, by tiles per SM over the tiles of a column:
//                      below 8      8 to 12     12 to 20    20 to 24    24 to 32    32 to 64    above
//   64   forward      0.92 1.23   0.86 1.16   0.96 1.12   0.81 0.99   0.91 0.97   0.90 0.96   0.83 0.89
//        backward     0.91 1.24   0.87 1.13   0.96 1.16   0.83 1.02   0.93 1.03   0.89 0.99   0.92 0.95
//   128  forward      0.81 1.14   0.84 1.12   0.88 1.14   0.73 0.98   0.78 1.00   0.78 0.96   0.90 0.92
//        backward     0.81 1.23   0.86 1.13   0.91 1.15   0.85 1.00   0.91 1.04   0.92 0.98   0.92 0.95
// The line is at 32, above which all of these 25 gained.
// A query window counts with its own rows, in tiles and in bytes.
static inline int claim_rows(const moba_b200_problem& p, int tiles_per_sm) {
  const long long tiles = (sched_pairs_bound(p) + 127) / 128, column = (long long)(p.q_heads / p.kv_heads) * p.slots;
  const bool even = !p.packed || p.n_seq <= 2;
  if (tiles < (even && 6 * column > tiles_per_sm ? 6 * column : (long long)tiles_per_sm) * kSchedSMs) return 0;
  const long long n_rows = (long long)p.n_seq * p.kv_heads;
  const double bytes = 2.0 * p.batch * window_rows(p) * p.q_heads * p.head_dim, row = bytes / (double)n_rows;
  if (bytes > 96e6 && 48e6 / row >= 2.0 && tiles >= 32LL * column * kSchedSMs) return (int)(48e6 / row < 32.0 ? 48e6 / row : 32.0);
  return n_rows <= 32 ? (int)n_rows : 0;                  // (a lane per row)
}

// ---- stage launchers (defined one per .cu file) -----------------------------
int launch_pool(const moba_b200_problem& p, const void* k, const int32_t* cu, void* kbar, int* zero_cell, float* norms,
                cudaStream_t st);
// `lse_fill` (may be NULL): the partial log-sum-exps, set to -inf where a slot names no block.
int launch_gate_portable(const moba_b200_problem& p, const void* q, const void* kbar,
                         const int32_t* cu, int32_t* block_idx, float* lse_fill, cudaStream_t st);
int launch_gate_sm100(const moba_b200_problem& p, const void* q, const void* kbar,
                      const int32_t* cu, int32_t* block_idx, float* lse_fill, cudaStream_t st);
bool gate_sm100_supported(const moba_b200_problem& p);
// The exact gate on tensor cores: selections of the portable (float64) gate, for 16-bit inputs.
int launch_gate_exact_sm100(const moba_b200_problem& p, const void* q, const void* kbar, const float* norms, const int32_t* cu,
                            int32_t* block_idx, float* lse_fill, cudaStream_t st);
bool gate_exact_sm100_supported(const moba_b200_problem& p);

size_t transpose_scratch_bytes(const moba_b200_problem& p);
int launch_transpose(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu,
                     int32_t* col_nnz, int32_t* col_offsets, int32_t* order, int32_t* rows,
                     int32_t* heads, int32_t* slots, int2* entries, int part_shift, int32_t* work_items, void* scratch,
                     size_t scratch_bytes, cudaStream_t st);
bool transpose_small_supported(const moba_b200_problem& p);
int launch_transpose_small(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu, int32_t* col_nnz,
                           int32_t* col_offsets, int32_t* order, int2* entries, int part_shift, int32_t* work_items,
                           int32_t* slot_counter, cudaStream_t st);

int launch_transpose_noalloc(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu,
                             int32_t* col_nnz, int32_t* col_offsets, int32_t* order, int32_t* rows,
                             int32_t* heads, int32_t* slots, int32_t* work_items, cudaStream_t st);

int launch_fill_lse(const moba_b200_problem& p, float* part_lse, cudaStream_t st);
int launch_fwd_portable(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                        const moba_b200_index& ix, const int32_t* cu, void* part_o,
                        float* part_lse, cudaStream_t st);
int launch_fwd_sm100(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                     const moba_b200_index& ix, const int32_t* cu, void* part_o,
                     float* part_lse, int part_keys, int* claims, cudaStream_t st);
bool fwd_sm100_supported(const moba_b200_problem& p);
int launch_merge(const moba_b200_problem& p, const void* part_o, const float* part_lse,
                 void* out, float* lse, cudaStream_t st);

int launch_delta(const moba_b200_problem& p, const void* out, const void* dout, float* delta, int* zero_cell,
                 cudaStream_t st);
int launch_bwd_portable(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                        const void* dout, const float* lse, const float* delta,
                        const moba_b200_index& ix, const int32_t* cu, void* dq_part, void* dk,
                        void* dv, cudaStream_t st);
int launch_bwd_sm100(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                     const void* dout, const float* lse, const float* delta,
                     const moba_b200_index& ix, const int32_t* cu, void* dq_part, float* dkv_scratch,
                     void* dk, void* dv, int part_keys, int* claims, bool* reduces, cudaStream_t st);
bool bwd_sm100_supported(const moba_b200_problem& p);
// `beside`: the kernel before is the dK/dV reduction, which this one does not depend on.
int launch_dq_reduce(const moba_b200_problem& p, const void* dq_part, const float* part_lse,
                     void* dq, bool beside, cudaStream_t st);

// ---- argument checks and kernel-family selection, shared by the entry points (api.cu) ----
int check_problem(const moba_b200_problem* p);
int need(const void* ptr, const char* name);
int pick(const moba_b200_problem& p, bool fast_ok, const char* stage);
// The launch table of a problem whose gate runs in family `gate_path` (an error code is passed on).
int fill_plan(const moba_b200_problem& p, int gate_path, moba_b200_plan* plan);

int launch_pack_index(const void* mask, int mask_bytes, int batch, int seq_len, int32_t* dest, int32_t* lengths,
                      int32_t* cu, int32_t* meta, cudaStream_t st);
int launch_seq_meta(const int32_t* cu, int n_seq, int32_t* meta, cudaStream_t st);
int launch_pack_rows(const void* x, const int32_t* dest, const int32_t* cu, void* packed, int batch, int seq_len,
                     size_t row_bytes, cudaStream_t st);
int launch_unpack_rows(const void* packed, const int32_t* cu, void* out, int batch, int seq_len, size_t row_bytes,
                       cudaStream_t st);

}  // namespace moba
