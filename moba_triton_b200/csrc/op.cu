// The whole op in two calls: moba_b200_op_forward (pool, gate, transpose, attention, merge) and
// moba_b200_op_backward (delta, dK/dV and dQ partials, reductions), each into one caller-owned
// workspace. They run the stages' kernels; what they save is what lies between the stages: a
// dozen allocations and as many foreign calls per pass on the host (300 of the 360 us of a
// thousand-token training step, 100 of the 150 us of an 8 192-token forward), the passes that
// only the separate entry points need (the fill of the partial log-sum-exps, the public form of
// the index) and, for short rows, four of the transpose's five launches.
//
// moba_b200_op_forward_window / _backward_window run the second half of each (from the block ids on)
// for a window of query rows, on the same kernels, so that a call run window by window gives the bits
// of the whole one whatever its block size.
#include "common.cuh"
#include "sm100.cuh"

namespace moba {
namespace {

constexpr size_t kAlign = 256;
inline size_t up(size_t x) { return (x + kAlign - 1) & ~(kAlign - 1); }

// The cut of the work items. The policy of the scheduler has a floor of eight tiles, which is
// right when the rows fill the GPU; a small problem is mostly tail, and finer items spread it over the
// SMs, at the price of more dK/dV partials to sum. Measured with items of 2, 4 and 8 tiles, us
// (head_dim 64 unless noted):          tiles per SM, per row   attention kernels of a step   whole forward call
//   [1,1000,4 heads on 2], top 4           0.8     63                 45   48   59
//   [1,2048,2]                             1.7    128                 45   46   57               29   30   33
//   [1,4096,2]                             3.5    256                 60   52   59               37.3 36.4 40.5
//   [1,8192,1]                             3.5    512                 66   55   61
//   [1,1024,16]                            6.9     64                 61   55   50               38.7 38.4 41.5
//   [1,2048,8 on 2], head_dim 128          6.9    512                 92   90   80               52.5 55.2 55.6
//   [1,8192,4]                            13.8    512                134  105   94               59.3 58.1 58.1
//   [1,8192,5]                            17.3    512                156  125  115               71.8 69.5 70.3
//   [1,4096,4] float32, whose kernel       6.9    256                                               -  185  198
//     starts a CTA for every tile that an item may have
// Between 24 and 64 tiles per SM the partials are what a finer cut costs: eight tiles on top of a quarter of an
// SM's share. Below 32 that makes about two items to an SM where columns are longer than the items, more than
// its share: with columns of more than 16 tiles six on top. Columns of four tiles or less are hardly cut, the longest
// of them alone, and begin at 27. Training step, its time over that with items of a quarter (at least 8), by tiles
// per SM (q heads on kv heads of selected blocks):
//                   quarter + 8:  24    27    30    32    40    50    58    64    72    84   100     + 6:  24    27    30    32
//   head_dim 64    4 on 4 of 8   0.96        0.96        0.96  0.98  0.97  0.98  0.98  0.99  1.01
//                  4 on 1 of 8   0.99        0.96        0.97  0.98  1.00  1.00  0.99  1.00  1.00
//                  8 on 2 of 8   0.99        0.92        0.95  0.95  0.97  0.96  0.97  0.96  0.99
//                  4 on 4 of 4   1.04  1.00  0.98  1.00                                                   1.03  0.99  0.98  0.99
//                  4 on 4 of 12  0.97  0.93  0.96  0.95                                                   0.98  0.97  0.98  0.96
//                  4 on 2 of 8   0.92  0.91  0.92  0.94                                                   0.94  0.94  0.94  0.95
//                 16 on 4 of 8   1.06  1.00  0.95  0.94                                                   0.95  0.94  0.91  0.94
//                 32 on 8 of 8   0.98  1.02  1.04  0.99                                                   1.00  0.98  0.98  0.94
//   head_dim 128   4 on 4 of 8   0.97  0.96  0.97  0.97  0.98  0.98  0.99  1.00  0.99  1.01  1.00         0.97  0.96  0.97  0.96
//                  4 on 1 of 8   1.04  0.96  0.96  0.97                                                   0.98  0.96  0.99  1.01
//                  8 on 2 of 8   1.04  0.95  0.94  0.94                                                   0.95  0.94  0.94  0.99
//                 16 on 4 of 8   1.05  1.00  0.97  0.94  0.96  0.98  0.99  0.99  0.99  0.98  0.99         0.96  0.94  0.93  0.96
//                 32 on 8 of 8   0.99  1.03  1.03  0.99                                                   0.99  0.98  0.97  0.94
//                  4 on 2 of 6   0.95  0.94  0.96  0.95                                                   0.97  0.98  0.97  0.96
//                 16 on 4 of 6   1.04  0.97  0.95  0.94                                                   0.98  0.94  0.95  0.96
//                  8 on 2 of 12  1.04  0.98  0.95  0.94                                                   0.97  0.95  0.91  0.94
//                 16 on 16 of 4  1.04  0.98  0.98  0.99                                                   1.04  0.98  0.99  1.00
//                  4 on 4 of 2   1.00  1.00  1.01  0.98                                                   1.00  1.00  1.01  0.98
// (Below, at 18 and 21, a longer item is 0.95 to 1.06 of the time. Passes of one KV head of such a call take the
// call's cut, for its bits; at head_dim 128 they were faster with items of 8: [1,16384,4] 884 us, 982 with 15.)
// A forward alone has no partials and keeps the finer items, the better spread (2 % of its kernel).
// The cut decides in which groups dK and dV are summed: who runs the KV heads of a problem in several
// passes and wants the bits of the whole gives every pass the whole's chunk_tiles
// (moba_b200_op_launch_plan).
moba_b200_problem with_cut(const moba_b200_problem& p0, bool training = true) {
  moba_b200_problem p = p0;
  if (p.chunk_tiles > 0) return p;
  p.chunk_tiles = sched_chunk_tiles(p);
  const long long tiles = (sched_pairs_bound(p) + 127) / 128;
  const long long row_tiles = ((long long)(p.q_heads / p.kv_heads) * p.max_seqlen * p.slots + 127) / 128;
  const int column = p.q_heads / p.kv_heads * p.slots;       // tiles, on average
  const bool short_rows = row_tiles <= 128;
  if (tiles <= 4LL * kSchedSMs) p.chunk_tiles = short_rows ? 2 : 4;
  else if (tiles <= 16LL * kSchedSMs && (short_rows || p.dtype == MOBA_B200_F32)) p.chunk_tiles = 4;
  else if (training && p.dtype != MOBA_B200_F32 && tiles >= (column <= 4 ? 27LL : 24LL) * kSchedSMs && tiles <= 64LL * kSchedSMs)
    p.chunk_tiles = (int)((tiles + kSchedSplit * kSchedSMs - 1) / (kSchedSplit * kSchedSMs)) +
                    (column > 16 && tiles < 32LL * kSchedSMs ? 6 : 8);
  return p;
}

// Blocks of 16, 32 or 64 keys on the tensor-core kernels, whose columns are 128 keys: a column
// then holds 128 / block_size blocks, its list the pairs of all of them, and the kernels mask a
// pair to its own block. Half of the scores of a tile (three quarters, ...) are computed for
// nothing, at many times the rate of the CUDA-core kernels that took these sizes before
// (2 x 8192 tokens, 4 heads of 128, blocks of 64: forward 2.2 ms, backward 6.1 ms there). Only
// where the library chooses the kernels: a caller who asks for a family gets it.
struct Columns {
  moba_b200_problem p;       // the problem in columns of the attention kernels
  int part_keys, part_shift; // keys per block, log2 of the blocks per column
};
Columns columns_of(const moba_b200_problem& p) {
  Columns c{p, kBlockKeys, 0};
  if (p.path != MOBA_B200_PATH_AUTO || p.block_size >= kBlockKeys || kBlockKeys % p.block_size || p.gate_window != 0) return c;
  moba_b200_problem w = p;
  w.block_size = kBlockKeys;
  w.num_blocks = (p.max_seqlen + kBlockKeys - 1) / kBlockKeys;
  if (!fwd_sm100_supported(w) || !bwd_sm100_supported(w)) return c;
  c.p = w;
  c.part_keys = p.block_size;
  while ((p.block_size << c.part_shift) < kBlockKeys) ++c.part_shift;
  return c;
}

// Byte offsets of the buffers inside the caller's workspaces. A window call gets block ids and the
// log-sum-exps from its caller and keeps nothing: its index is built again by the backward.
struct Layout {
  size_t col_nnz, col_offsets, order, items, entries, part_lse, lse, keep_bytes;      // kept for the backward
  size_t kbar, norms, block_idx, counter, transpose_scratch, part_o, fwd_bytes;              // forward only
  size_t delta, claims, dq_part, dkv, bwd_transpose_scratch, bwd_bytes;                       // backward only
};
inline long long row_capacity(const moba_b200_problem& p) {
  return (long long)(p.q_heads / p.kv_heads) * window_rows_of_seq(p) * p.slots;
}
Layout layout_of(const moba_b200_problem& gate, const moba_b200_problem& p) {
  Layout l;
  const size_t rows = (size_t)p.n_seq * p.kv_heads, nb = p.num_blocks;
  const size_t pairs = (size_t)p.batch * p.q_heads * window_rows(p) * p.slots;
  const size_t capacity = (size_t)row_capacity(p);
  const bool window = p.win_rows > 0;
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t o = at; at = up(at + bytes); return o; };
  l.col_nnz = take(rows * nb * 4);
  l.col_offsets = take(rows * (nb + 1) * 4);
  l.order = take(rows * nb * 4);
  moba_b200_problem alone = p;                               // a forward alone may have finer items, and more
  if (p.chunk_tiles > kMinChunkTiles) { alone.chunk_tiles = 0; alone.chunk_tiles = sched_chunk_tiles(alone); }
  l.items = take(rows * (size_t)(sched_items_per_row(alone) > sched_items_per_row(p) ? sched_items_per_row(alone) : sched_items_per_row(p)) * 16);
  l.entries = take(rows * capacity * 8);
  l.part_lse = take(pairs * 4);
  l.lse = take(window ? 0 : (size_t)p.batch * p.q_heads * p.tokens * 4);
  l.keep_bytes = at;
  at = 0;
  const size_t part_size = p.part_f32 ? 4 : dtype_size(p.dtype);
  const size_t scratch = transpose_small_supported(p) ? 16 : transpose_scratch_bytes(p);
  l.kbar = take(window ? 0 : rows * gate.num_blocks * p.head_dim * dtype_size(p.dtype));
  l.norms = take(window ? 0 : rows * gate.num_blocks * 4);
  l.block_idx = take(window ? 0 : pairs * 4);
  l.counter = take(16);
  l.transpose_scratch = take(scratch);
  l.part_o = take(pairs * p.head_dim * part_size);
  l.fwd_bytes = at;
  at = 0;
  l.delta = take((size_t)p.batch * p.q_heads * p.tokens * 4);
  l.claims = take(16);
  l.dq_part = take(pairs * p.head_dim * dtype_size(p.dtype));
  l.dkv = take(sched_dkv_scratch_bytes(p));
  l.bwd_transpose_scratch = take(window ? scratch : 0);
  l.bwd_bytes = at;
  return l;
}

moba_b200_index index_in(const moba_b200_problem& p, const Layout& l, unsigned char* keep) {
  moba_b200_index ix = {};
  ix.col_nnz = reinterpret_cast<int32_t*>(keep + l.col_nnz);
  ix.col_offsets = reinterpret_cast<int32_t*>(keep + l.col_offsets);
  ix.order = reinterpret_cast<int32_t*>(keep + l.order);
  ix.capacity = row_capacity(p);
  ix.work_items = reinterpret_cast<int32_t*>(keep + l.items);
  ix.items_per_row = (int)sched_items_per_row(p);
  ix.chunk_tiles = sched_chunk_tiles(p);
  ix.row_indices = reinterpret_cast<int32_t*>(keep + l.entries);   // packed pairs
  return ix;
}

// Which gate the op runs: where the portable one would by the library's choice, its selections come
// from the exact tensor-core gate if that covers the problem.
bool runs_exact_gate(const moba_b200_problem& gate, int gate_path) {
  return gate_path == MOBA_B200_PATH_PORTABLE && gate.path == MOBA_B200_PATH_AUTO && gate_exact_sm100_supported(gate);
}

int check_sizes(const moba_b200_problem* p) {
  MOBA_TRY(check_problem(p));
  if (p->q_heads >= 1 << 19) { set_error("%d query heads do not fit a packed index entry", p->q_heads); return MOBA_B200_EUNSUPPORTED; }
  if (sched_items_per_row(*p) > 0x7fffffffLL || sched_part_slots(*p) > 0x7fffffffLL) {
    set_error("chunk_tiles %d cuts the problem into too many work items", sched_chunk_tiles(*p));
    return MOBA_B200_EUNSUPPORTED;
  }
  return MOBA_B200_OK;
}
int check_op(const moba_b200_problem* p) {
  MOBA_TRY(check_sizes(p));
  if (p->win_rows > 0) { set_error("the whole-op entry points take no query window"); return MOBA_B200_EUNSUPPORTED; }
  return MOBA_B200_OK;
}
int check_window(const moba_b200_problem* p) {
  MOBA_TRY(check_sizes(p));
  if (p->win_rows == 0) { set_error("a window call needs a query window"); return MOBA_B200_EINVAL; }
  return MOBA_B200_OK;
}

int transpose_into(const Columns& c, const moba_b200_index& ix, const int32_t* block_idx, const int32_t* cu, void* scratch,
                   int32_t* counter, cudaStream_t st) {
  const moba_b200_problem& p = c.p;
  int32_t* col_nnz = const_cast<int32_t*>(ix.col_nnz);
  int32_t* col_offsets = const_cast<int32_t*>(ix.col_offsets);
  int32_t* order = const_cast<int32_t*>(ix.order);
  int32_t* items = const_cast<int32_t*>(ix.work_items);
  int2* entries = reinterpret_cast<int2*>(const_cast<int32_t*>(ix.row_indices));
  if (transpose_small_supported(p))
    return launch_transpose_small(p, block_idx, cu, col_nnz, col_offsets, order, entries, c.part_shift, items, counter, st);
  return launch_transpose(p, block_idx, cu, col_nnz, col_offsets, order, nullptr, nullptr, nullptr, entries, c.part_shift, items,
                          scratch, transpose_scratch_bytes(p), st);
}

// From block ids to the output: transpose, attention, merge. `claims`: a counter that is zero by then, or NULL.
int attend(const Columns& c, const Layout& l, int fwd_path, const void* q, const void* k, const void* v, const int32_t* block_idx,
           const int32_t* cu, unsigned char* keep, unsigned char* tmp, int* claims, void* out, float* lse, cudaStream_t st) {
  const moba_b200_problem& p = c.p;
  const moba_b200_index ix = index_in(p, l, keep);
  float* part_lse = reinterpret_cast<float*>(keep + l.part_lse);
  void* part_o = tmp + l.part_o;
  MOBA_TRY(transpose_into(c, ix, block_idx, cu, tmp + l.transpose_scratch, reinterpret_cast<int32_t*>(tmp + l.counter), st));
  if (fwd_path == MOBA_B200_PATH_TCGEN05) MOBA_TRY(launch_fwd_sm100(p, q, k, v, ix, cu, part_o, part_lse, c.part_keys, claims, st));
  else MOBA_TRY(launch_fwd_portable(p, q, k, v, ix, cu, part_o, part_lse, st));
  return launch_merge(p, part_o, part_lse, out, lse, st);
}

// The gradients from an index: delta, dK/dV and dQ partials, reductions.
int differentiate(const Columns& c, const Layout& l, int path, const void* q, const void* k, const void* v, const void* out,
                  const void* dout, const float* lse, const float* part_lse, const int32_t* cu, unsigned char* keep,
                  unsigned char* tmp, void* dq, void* dk, void* dv, cudaStream_t st) {
  const moba_b200_problem& p = c.p;
  const moba_b200_index ix = index_in(p, l, keep);
  float* delta = reinterpret_cast<float*>(tmp + l.delta);
  void* dq_part = tmp + l.dq_part;
  bool reduces = false;
  int* claims = reinterpret_cast<int*>(tmp + l.claims);
  MOBA_TRY(launch_delta(p, out, dout, delta, claims, st));
  if (path == MOBA_B200_PATH_TCGEN05)
    MOBA_TRY(launch_bwd_sm100(p, q, k, v, dout, lse, delta, ix, cu, dq_part, reinterpret_cast<float*>(tmp + l.dkv), dk, dv, c.part_keys, claims, &reduces, st));
  else
    MOBA_TRY(launch_bwd_portable(p, q, k, v, dout, lse, delta, ix, cu, dq_part, dk, dv, st));
  return launch_dq_reduce(p, dq_part, part_lse, dq, reduces, st);
}

// What a whole-op call runs; `training`: a forward that keeps its log-sum-exps, and its backward.
int op_plan(const moba_b200_problem* p0, bool training, moba_b200_plan* plan) {
  MOBA_TRY(check_sizes(p0));
  if (plan == nullptr) { set_error("plan is NULL"); return MOBA_B200_EINVAL; }
  const moba_b200_problem gate = with_cut(*p0);
  moba_b200_problem p = columns_of(gate).p;
  if (!training && p0->win_rows == 0) p.chunk_tiles = with_cut(*p0, false).chunk_tiles;   // (a window's forward takes the cut of its backward)
  const int gate_path = pick(gate, gate_sm100_supported(gate), "gate");
  MOBA_TRY(fill_plan(p, gate_path >= 0 && runs_exact_gate(gate, gate_path) ? MOBA_B200_PATH_TCGEN05 : gate_path, plan));
  if (transpose_small_supported(p)) plan->transpose_chunk_rows = plan->transpose_chunks = plan->scatter_warps = 0;
  return MOBA_B200_OK;
}

}  // namespace
}  // namespace moba

using namespace moba;

extern "C" {

int moba_b200_op_workspace(const moba_b200_problem* p0, size_t* keep_bytes, size_t* forward_bytes, size_t* backward_bytes) {
  MOBA_TRY(check_sizes(p0));
  const moba_b200_problem gate = with_cut(*p0);
  const Layout l = layout_of(gate, columns_of(gate).p);
  if (keep_bytes) *keep_bytes = l.keep_bytes;
  if (forward_bytes) *forward_bytes = l.fwd_bytes;
  if (backward_bytes) *backward_bytes = l.bwd_bytes;
  return MOBA_B200_OK;
}

int moba_b200_op_launch_plan(const moba_b200_problem* p0, moba_b200_plan* plan) { return op_plan(p0, true, plan); }
int moba_b200_op_forward_launch_plan(const moba_b200_problem* p0, moba_b200_plan* plan) { return op_plan(p0, false, plan); }

int moba_b200_op_forward(const moba_b200_problem* p0, const void* q, const void* k, const void* v,
                         const int32_t* cu_seqlens, void* keep_ws, void* forward_ws, void* out, int want_lse, void* stream) {
  MOBA_TRY(check_op(p0));
  MOBA_TRY(need(q, "q")); MOBA_TRY(need(k, "k")); MOBA_TRY(need(v, "v")); MOBA_TRY(need(out, "out"));
  MOBA_TRY(need(keep_ws, "keep_ws")); MOBA_TRY(need(forward_ws, "forward_ws"));
  if (p0->packed) MOBA_TRY(need(cu_seqlens, "cu_seqlens"));
  const moba_b200_problem gate = with_cut(*p0);
  const Columns columns = columns_of(gate);
  const moba_b200_problem& p = columns.p;
  const int gate_path = pick(gate, gate_sm100_supported(gate), "gate"), fwd_path = pick(p, fwd_sm100_supported(p), "forward");
  if (gate_path < 0) return gate_path;
  if (fwd_path < 0) return fwd_path;
  cudaStream_t st = (cudaStream_t)stream;
  const Layout l = layout_of(gate, p);
  unsigned char* keep = static_cast<unsigned char*>(keep_ws);
  unsigned char* tmp = static_cast<unsigned char*>(forward_ws);
  void* kbar = tmp + l.kbar;
  int32_t* block_idx = reinterpret_cast<int32_t*>(tmp + l.block_idx);
  float* part_lse = reinterpret_cast<float*>(keep + l.part_lse);
  int32_t* counter = reinterpret_cast<int32_t*>(tmp + l.counter);
  const bool exact_gate = runs_exact_gate(gate, gate_path);
  float* norms = reinterpret_cast<float*>(tmp + l.norms);
  Columns cut = columns;                                     // the layout holds either cut's table
  if (!want_lse) cut.p.chunk_tiles = with_cut(*p0, false).chunk_tiles;
  MOBA_TRY(launch_pool(gate, k, cu_seqlens, kbar, counter, exact_gate ? norms : nullptr, st));
  if (gate_path == MOBA_B200_PATH_TCGEN05) MOBA_TRY(launch_gate_sm100(gate, q, kbar, cu_seqlens, block_idx, part_lse, st));
  else if (exact_gate) MOBA_TRY(launch_gate_exact_sm100(gate, q, kbar, norms, cu_seqlens, block_idx, part_lse, st));
  else MOBA_TRY(launch_gate_portable(gate, q, kbar, cu_seqlens, block_idx, part_lse, st));
  return attend(cut, l, fwd_path, q, k, v, block_idx, cu_seqlens, keep, tmp, counter + 1, out,
                want_lse ? reinterpret_cast<float*>(keep + l.lse) : nullptr, st);
}

int moba_b200_op_backward(const moba_b200_problem* p0, const void* q, const void* k, const void* v, const void* out,
                          const void* dout, const int32_t* cu_seqlens, const void* keep_ws, void* backward_ws,
                          void* dq, void* dk, void* dv, void* stream) {
  MOBA_TRY(check_op(p0));
  MOBA_TRY(need(q, "q")); MOBA_TRY(need(k, "k")); MOBA_TRY(need(v, "v")); MOBA_TRY(need(out, "out"));
  MOBA_TRY(need(dout, "dout")); MOBA_TRY(need(dq, "dq")); MOBA_TRY(need(dk, "dk")); MOBA_TRY(need(dv, "dv"));
  MOBA_TRY(need(keep_ws, "keep_ws")); MOBA_TRY(need(backward_ws, "backward_ws"));
  if (p0->packed) MOBA_TRY(need(cu_seqlens, "cu_seqlens"));
  const moba_b200_problem gate = with_cut(*p0);
  const Columns columns = columns_of(gate);
  const moba_b200_problem& p = columns.p;
  const int path = pick(p, bwd_sm100_supported(p), "backward");
  if (path < 0) return path;
  cudaStream_t st = (cudaStream_t)stream;
  const Layout l = layout_of(gate, p);
  unsigned char* keep = const_cast<unsigned char*>(static_cast<const unsigned char*>(keep_ws));
  unsigned char* tmp = static_cast<unsigned char*>(backward_ws);
  return differentiate(columns, l, path, q, k, v, out, dout, reinterpret_cast<const float*>(keep + l.lse),
                       reinterpret_cast<const float*>(keep + l.part_lse), cu_seqlens, keep, tmp, dq, dk, dv, st);
}

int moba_b200_op_forward_window(const moba_b200_problem* p0, const void* q, const void* k, const void* v, const int32_t* block_idx,
                                void* keep_ws, void* forward_ws, void* out, float* lse, void* stream) {
  MOBA_TRY(check_window(p0));
  MOBA_TRY(need(q, "q")); MOBA_TRY(need(k, "k")); MOBA_TRY(need(v, "v")); MOBA_TRY(need(out, "out"));
  MOBA_TRY(need(block_idx, "block_idx")); MOBA_TRY(need(keep_ws, "keep_ws")); MOBA_TRY(need(forward_ws, "forward_ws"));
  const moba_b200_problem gate = with_cut(*p0);
  const Columns columns = columns_of(gate);
  const moba_b200_problem& p = columns.p;
  const int path = pick(p, fwd_sm100_supported(p), "forward");
  if (path < 0) return path;
  cudaStream_t st = (cudaStream_t)stream;
  const Layout l = layout_of(gate, p);
  unsigned char* keep = static_cast<unsigned char*>(keep_ws);
  MOBA_TRY(launch_fill_lse(p, reinterpret_cast<float*>(keep + l.part_lse), st));
  return attend(columns, l, path, q, k, v, block_idx, nullptr, keep, static_cast<unsigned char*>(forward_ws), nullptr, out, lse, st);
}

int moba_b200_op_backward_window(const moba_b200_problem* p0, const void* q, const void* k, const void* v, const void* out,
                                 const void* dout, const float* lse, const float* part_lse, const int32_t* block_idx, void* keep_ws,
                                 void* backward_ws, void* dq, void* dk, void* dv, void* stream) {
  MOBA_TRY(check_window(p0));
  MOBA_TRY(need(q, "q")); MOBA_TRY(need(k, "k")); MOBA_TRY(need(v, "v")); MOBA_TRY(need(out, "out"));
  MOBA_TRY(need(dout, "dout")); MOBA_TRY(need(lse, "lse")); MOBA_TRY(need(part_lse, "part_lse"));
  MOBA_TRY(need(dq, "dq")); MOBA_TRY(need(dk, "dk")); MOBA_TRY(need(dv, "dv"));
  MOBA_TRY(need(block_idx, "block_idx")); MOBA_TRY(need(keep_ws, "keep_ws")); MOBA_TRY(need(backward_ws, "backward_ws"));
  const moba_b200_problem gate = with_cut(*p0);
  const Columns columns = columns_of(gate);
  const moba_b200_problem& p = columns.p;
  const int path = pick(p, bwd_sm100_supported(p), "backward");
  if (path < 0) return path;
  cudaStream_t st = (cudaStream_t)stream;
  const Layout l = layout_of(gate, p);
  unsigned char* keep = static_cast<unsigned char*>(keep_ws);
  unsigned char* tmp = static_cast<unsigned char*>(backward_ws);
  MOBA_TRY(transpose_into(columns, index_in(p, l, keep), block_idx, nullptr, tmp + l.bwd_transpose_scratch, nullptr, st));
  return differentiate(columns, l, path, q, k, v, out, dout, lse, part_lse, nullptr, keep, tmp, dq, dk, dv, st);
}

}  // extern "C"
