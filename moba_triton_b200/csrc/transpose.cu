// Transpose: regroups per-query selections (CSR, block_idx) by key/value block
// (CSC) with a *stable* counting sort, so a column lists its queries ordered by
// (query head, row) on every run.
//
//   1. count    one CTA per (row chunk, sequence, query head): shared-memory
//               histogram over blocks -> tile_counts[seq,kvh][block][g*C + chunk]
//   2. colscan  one warp per (sequence, kv head, block): exclusive scan of that
//               block's tile counts in (g, chunk) order; total -> col_nnz
//   3. offsets  per (sequence, kv head): exclusive scan over blocks ->
//               col_offsets, and the longest-first dispatch order (stable
//               descending sort of col_nnz, by rank counting)
//   4. items    per (sequence, kv head): walks the columns in dispatch order and cuts
//               each into work items of at most chunk_tiles tiles; a split column's
//               items get consecutive dK/dV partial slots
//   5. scatter  one CTA per (row chunk, sequence, query head): its warps split the
//               chunk's rows into consecutive runs; a per-warp histogram and a scan
//               over the warps give each warp its own cursors, and every warp then
//               walks its run in order, ranks equal blocks inside the warp with
//               match.any and writes (row, head, slot) at cursor[block]++.
//
// Stands in for count_columns_kernel / offsets_and_order_kernel /
// scatter_pairs_kernel of the reference (src/moba/kernels/routing.py:138-301),
// which claim positions with an atomic cursor and therefore leave the order
// inside a column to the scheduler.
#include "common.cuh"
#include "sm100.cuh"

#include <mutex>

namespace moba {

struct TransposeGeom {
  int chunk_rows;   // R, a power of two
  int chunks;       // C = cdiv(max_seqlen, R)
};
static inline TransposeGeom transpose_geom(const moba_b200_problem& p) {
  int r = 256;
  while ((p.max_seqlen + r - 1) / r > 256) r <<= 1;
  return TransposeGeom{r, (p.max_seqlen + r - 1) / r};
}
static inline size_t tile_count_bytes(const moba_b200_problem& p) {
  const TransposeGeom g = transpose_geom(p);
  const size_t group = p.q_heads / p.kv_heads;
  return (size_t)p.n_seq * p.kv_heads * p.num_blocks * group * g.chunks * sizeof(int32_t);
}
// the per-chunk histograms, then one 16-byte cell holding the counter of dK/dV partial slots
size_t transpose_scratch_bytes(const moba_b200_problem& p) { return ((tile_count_bytes(p) + 15) & ~size_t(15)) + 16; }

__device__ __forceinline__ size_t block_idx_row(const moba_b200_problem& p, int seq, int hq,
                                                int bos, int row) {
  const size_t b = p.packed ? 0 : (size_t)seq;
  return ((b * p.q_heads + hq) * p.tokens + bos + row) * (size_t)p.slots;
}

__global__ void __launch_bounds__(256)
count_kernel(const int32_t* __restrict__ block_idx, const int32_t* __restrict__ cu,
             int32_t* __restrict__ tile_counts, int32_t* __restrict__ slot_counter, moba_b200_problem p, int part_shift, int R, int C) {
  extern __shared__ int hist[];
  pdl_trigger();
  pdl_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) *slot_counter = 0;     // claimed from by work_items_kernel, two launches on
  const int chunk = blockIdx.x % C, y = blockIdx.x / C;
  const int seq = y / p.q_heads, hq = y % p.q_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const int row0 = chunk * R;
  if (row0 >= sp.len) return;
  const int rows = min(R, sp.len - row0);
  const int nb_lim = (row0 + rows - 1) / p.block_size + 1;
  for (int i = threadIdx.x; i < nb_lim; i += 256) hist[i] = 0;
  __syncthreads();
  const int32_t* src = block_idx + block_idx_row(p, seq, hq, sp.bos, row0);
  // only the rows inside the query window are listed (all of them without a window)
  const int w_lo = max(0, p.win_begin - row0), w_hi = min(rows, (p.win_rows > 0 ? p.win_begin + p.win_rows : sp.len) - row0);
  const int n = max(w_lo, w_hi) * p.slots;
  for (int e = w_lo * p.slots + threadIdx.x; e < n; e += 256) {
    const int blk = src[e] >> part_shift;
    if (blk >= 0 && blk < nb_lim) atomicAdd(&hist[blk], 1);
  }
  __syncthreads();
  const int group = p.q_heads / p.kv_heads;
  const int kvh = hq / group, g = hq % group;
  int32_t* dst = tile_counts + ((size_t)(seq * p.kv_heads + kvh) * p.num_blocks) * (group * C) + g * C + chunk;
  for (int i = threadIdx.x; i < nb_lim; i += 256) dst[(size_t)i * (group * C)] = hist[i];
}

// One warp per column. Replaces the column's tile counts by their exclusive
// prefix (in (g, chunk) order) and writes the column total.
__global__ void __launch_bounds__(128)
colscan_kernel(const int32_t* __restrict__ cu, int32_t* __restrict__ tile_counts,
               int32_t* __restrict__ col_nnz, moba_b200_problem p, int R, int C, int ctas_per_row) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = (int)(blockIdx.x % ctas_per_row) * 4 + warp;
  const int kv_row = (int)(blockIdx.x / ctas_per_row);       // (sequence, kv head)
  if (col >= p.num_blocks) return;
  const int seq = kv_row / p.kv_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  int32_t* out_nnz = col_nnz + (size_t)kv_row * p.num_blocks + col;
  if ((size_t)col * p.block_size >= (size_t)sp.len) {
    if (lane == 0) *out_nnz = 0;
    return;
  }
  const int group = p.q_heads / p.kv_heads;
  const int c_lo = (int)(((size_t)col * p.block_size) / R);
  const int c_hi = (sp.len + R - 1) / R;                    // exclusive
  const int span = c_hi - c_lo;
  int32_t* base = tile_counts + ((size_t)kv_row * p.num_blocks + col) * (group * C);
  int running = 0;
  const int total = group * span;
  for (int i0 = 0; i0 < total; i0 += 32) {
    const int i = i0 + lane;
    int v = 0;
    int32_t* ptr = nullptr;
    if (i < total) {
      ptr = base + (i / span) * C + c_lo + (i % span);
      v = *ptr;
    }
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (ptr) *ptr = running + incl - v;
    running += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) *out_nnz = running;
}

// (sequence, kv head) x (128 columns): col_offsets (first CTA of the row) and the dispatch order.
__global__ void __launch_bounds__(1024)
offsets_order_kernel(const int32_t* __restrict__ col_nnz, int32_t* __restrict__ col_offsets,
                     int32_t* __restrict__ order, int nb) {
  extern __shared__ int cnt[];              // [nb]
  pdl_trigger();
  pdl_wait();
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  const int32_t* nnz = col_nnz + (size_t)blockIdx.x * nb;
  int32_t* off = col_offsets + (size_t)blockIdx.x * (nb + 1);
  int32_t* ord = order + (size_t)blockIdx.x * nb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int i0 = 0; i0 < nb; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const int v = (i < nb) ? nnz[i] : 0;
    if (i < nb) cnt[i] = v;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sums[lane];
      int wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      warp_sums[lane] = wi - w;             // exclusive over warps
    }
    __syncthreads();
    const int carry = carry_s;
    if (i < nb && blockIdx.y == 0) off[i] = carry + warp_sums[warp] + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = carry + warp_sums[warp] + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0 && blockIdx.y == 0) off[nb] = carry_s;
  // stable descending rank: position of column i = #{j : n_j > n_i or (n_j == n_i and j < i)}.
  // nb^2 comparisons in all: CTA y of the row ranks columns [128 y, 128 y + 128), eight
  // threads per column over interleaved j.
  const int i = (int)blockIdx.y * 128 + (int)(threadIdx.x >> 3), part = threadIdx.x & 7;
  int rank = 0;
  if (i < nb) {
    const int ni = cnt[i];
    for (int j = part; j < nb; j += 8) {
      const int nj = cnt[j];
      rank += (nj > ni || (nj == ni && j < i)) ? 1 : 0;
    }
  }
  rank += __shfl_xor_sync(0xffffffffu, rank, 1);
  rank += __shfl_xor_sync(0xffffffffu, rank, 2);
  rank += __shfl_xor_sync(0xffffffffu, rank, 4);
  if (i < nb && part == 0) ord[rank] = i;
}

// One CTA per (sequence, kv head) row: the row's work items, largest first. A column of more
// than `tc` tiles becomes ceil(tiles / tc) items, each with a dK/dV partial slot of its own:
// pieces of `tc` tiles and a last, shorter one. The kernels deal the list out to their CTAs in
// alternating direction, which balances a list that is sorted by size; so the full pieces come
// first and the last pieces of the cut columns are merged, by size, into the (already sorted)
// uncut columns: without that a CTA's share was off by up to 18 % when a CTA gets only some
// eight items. The slots of a row are consecutive and claimed from a counter, so rows may
// claim in any order: slot numbers name scratch memory, results do not depend on them, nor on
// the order of the list. A row with more than kMaxCut cut columns keeps its columns' pieces
// side by side, in column order (it has items enough for the order not to matter). Every row ends
// in at least one entry of padding (sched_extra_items); it says how many full pieces the row has
// (its items less one per block): who claims items, and not entries, reads it there.
constexpr int kMaxCut = 2048;
// The row's work items, by all 1024 threads of a CTA. `nnz` and `ord` are the row's column
// totals and dispatch order (global or shared memory), `out` its stretch of the item table.
__device__ void write_work_items(const int32_t* nnz, const int32_t* ord, int4* out, int32_t* slot_counter, int nb,
                                 int items_per_row, int tc, int slot_cap, unsigned* error_word) {
  __shared__ long long warp_sums[32];
  __shared__ long long carry_s;
  __shared__ int base_s;
  __shared__ int rem_s[kMaxCut], rank_s[kMaxCut], sorted_s[kMaxCut], slot_s[kMaxCut];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto tiles_of = [&](int r) { return (nnz[ord[r]] + 127) / 128; };
  auto chunks_of = [&](int r, int& blk, int& tiles) {
    blk = ord[r];
    tiles = (nnz[blk] + 127) / 128;
    return tiles <= tc ? 1 : (tiles + tc - 1) / tc;
  };
  // exclusive prefix of a 64-bit value over the CTA, and the CTA's total
  auto block_scan = [&](long long v, long long& total) {
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    long long before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      const long long s = warp_sums[w];
      before += (w < warp) ? s : 0;
      all += s;
    }
    total = all;
    return before + incl - v;
  };
  // pass 1: cut columns (a prefix of the dispatch order) and the partial slots the row needs
  long long mine = 0;
  for (int r = threadIdx.x; r < nb; r += 1024) {
    int blk, tiles;
    const int c = chunks_of(r, blk, tiles);
    if (c > 1) mine += 1LL | ((long long)c << 32);
  }
  long long row_total;
  block_scan(mine, row_total);
  const int n_cut = (int)(row_total & 0xffffffffLL);
  const int row_slots = (int)(row_total >> 32);
  if (threadIdx.x == 0) {
    base_s = row_slots > 0 ? atomicAdd(slot_counter, row_slots) : 0;
    carry_s = 0;
    if (row_slots > 0 && (long long)base_s + row_slots > slot_cap) atomicOr(error_word, 2u);   // sizes were promised by the host
  }
  __syncthreads();
  const int base = base_s;
  // beyond the promised capacity (flagged above) an item falls back to "whole column": wrong
  // sums, reported through the error word, but no access outside the scratch
  auto slot_or_none = [&](int s) { return s < slot_cap ? s : -1; };
  auto put = [&](int at, int4 it) {
    if (at >= 0 && at < items_per_row) out[at] = it;
    else atomicOr(error_word, 2u);
  };

  if (n_cut <= kMaxCut) {
    const int n_full = row_slots - n_cut;                   // pieces of exactly tc tiles: they lead the list
    // the cut columns: full pieces in column order, the last piece's size and slot for later
    for (int r0 = 0; r0 < n_cut; r0 += 1024) {
      const int r = r0 + threadIdx.x;
      int blk = 0, tiles = 0, c = 0;
      if (r < n_cut) c = chunks_of(r, blk, tiles);
      long long total;
      const long long carry = carry_s;
      const int slot0 = (int)(carry + block_scan((long long)c, total));   // pieces of the cut columns before this one
      if (r < n_cut) {
        const int full0 = slot0 - r;                        // each earlier cut column has one piece that is not full
        for (int i = 0; i + 1 < c; ++i) put(full0 + i, make_int4(blk, i * tc, tc, slot_or_none(base + slot0 + i)));
        rem_s[r] = tiles - (c - 1) * tc;
        slot_s[r] = slot0;
      }
      __syncthreads();
      if (threadIdx.x == 0) carry_s = carry + total;
      __syncthreads();
    }
    // rank of each last piece among the last pieces: larger first, ties in column order
    for (int r = threadIdx.x; r < n_cut; r += 1024) {
      const int mine_rem = rem_s[r];
      int rank = 0;
      for (int q = 0; q < n_cut; ++q) {
        const int o = rem_s[q];
        rank += (o > mine_rem || (o == mine_rem && q < r)) ? 1 : 0;
      }
      rank_s[r] = rank;
      sorted_s[rank] = mine_rem;
    }
    __syncthreads();
    // last pieces of the cut columns: behind the uncut columns that are larger
    for (int r = threadIdx.x; r < n_cut; r += 1024) {
      const int mine_rem = rem_s[r];
      int lo = n_cut, hi = nb;                              // first uncut column with tiles <= mine_rem
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tiles_of(mid) > mine_rem) lo = mid + 1; else hi = mid;
      }
      int blk, tiles;
      const int c = chunks_of(r, blk, tiles);
      put(n_full + rank_s[r] + (lo - n_cut), make_int4(blk, (c - 1) * tc, mine_rem, slot_or_none(base + slot_s[r] + c - 1)));
    }
    // uncut columns: behind the last pieces that are at least as large
    for (int r = n_cut + threadIdx.x; r < nb; r += 1024) {
      int blk, tiles;
      chunks_of(r, blk, tiles);
      int lo = 0, hi = n_cut;                               // first last piece smaller than this column
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sorted_s[mid] >= tiles) lo = mid + 1; else hi = mid;
      }
      put(n_full + (r - n_cut) + lo, make_int4(blk, 0, tiles, -1));
    }
    for (int j = n_full + nb + threadIdx.x; j < items_per_row; j += 1024) out[j] = make_int4(0, n_full, 0, -2);   // padding, which tells how many pieces lead the row
    return;
  }

  // more cut columns than the tables hold: each column's pieces side by side, in column order
  for (int r0 = 0; r0 < nb; r0 += 1024) {
    const int r = r0 + threadIdx.x;
    int blk = 0, tiles = 0, c = 0;
    if (r < nb) c = chunks_of(r, blk, tiles);
    const long long v = (long long)c | ((long long)(c > 1 ? c : 0) << 32);
    long long total;
    const long long carry = carry_s;
    const long long at = carry + block_scan(v, total);
    const int item0 = (int)(at & 0xffffffffLL), slot0 = (int)(at >> 32);
    for (int i = 0; i < c; ++i)
      put(item0 + i, make_int4(blk, i * tc, tiles == 0 ? 0 : min(tc, tiles - i * tc), c > 1 ? slot_or_none(base + slot0 + i) : -1));
    __syncthreads();
    if (threadIdx.x == 0) carry_s = carry + total;
    __syncthreads();
  }
  const int used = (int)(carry_s & 0xffffffffLL);
  for (int j = used + threadIdx.x; j < items_per_row; j += 1024) out[j] = make_int4(0, used - nb, 0, -2);   // padding, which tells how many pieces lead the row
}

__global__ void __launch_bounds__(1024)
work_items_kernel(const int32_t* __restrict__ col_nnz, const int32_t* __restrict__ order, int4* __restrict__ items,
                  int32_t* __restrict__ slot_counter, int nb, int items_per_row, int tc, int slot_cap,
                  unsigned* error_word) {
  pdl_trigger();
  pdl_wait();
  write_work_items(col_nnz + (size_t)blockIdx.x * nb, order + (size_t)blockIdx.x * nb,
                            items + (size_t)blockIdx.x * items_per_row, slot_counter, nb, items_per_row, tc, slot_cap,
                            error_word);
}

// One CTA of W warps per (row chunk, sequence, query head). The walk of a run is one
// dependent chain per warp (match, cursor, store), so the chunk is cut into W runs that are
// walked side by side: a histogram per run and a scan over the runs (both in shared memory)
// turn the chunk's cursors into cursors per run. The order inside a column stays
// (query head, row): runs are consecutive rows and keep the chunk's order.
// PACKED: one eight-byte entry per pair instead of three words in three arrays. The stores are
// scattered, so their number is what this kernel costs.
template <int W, bool PACKED>
__global__ void __launch_bounds__(32 * W)
scatter_kernel(const int32_t* __restrict__ block_idx, const int32_t* __restrict__ cu,
               const int32_t* __restrict__ tile_prefix, const int32_t* __restrict__ col_offsets,
               int32_t* __restrict__ rows_out, int32_t* __restrict__ heads_out,
               int32_t* __restrict__ slots_out, int2* __restrict__ entries_out, moba_b200_problem p, int part_shift, int R, int C,
               long long capacity) {
  extern __shared__ int cursor_all[];                        // [W][nb_lim]
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.x % C, y = blockIdx.x / C;
  const int seq = y / p.q_heads, hq = y % p.q_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const int row0 = chunk * R;
  if (row0 >= sp.len) return;                                // the whole CTA
  const int rows = min(R, sp.len - row0);
  const int nb_lim = (row0 + rows - 1) / p.block_size + 1;
  const int group = p.q_heads / p.kv_heads;
  const int kvh = hq / group, g = hq % group;
  const size_t kv_row = (size_t)seq * p.kv_heads + kvh;
  const int32_t* pre = tile_prefix + (kv_row * p.num_blocks) * (group * C) + g * C + chunk;
  const int32_t* off = col_offsets + kv_row * (p.num_blocks + 1);
  // this warp's run of rows
  // the chunk's rows inside the query window (all of them without a window), cut into W runs
  const int w_lo = max(0, p.win_begin - row0);
  const int w_hi = max(w_lo, min(rows, (p.win_rows > 0 ? p.win_begin + p.win_rows : sp.len) - row0));
  const int run = (w_hi - w_lo + W - 1) / W;
  const int r_lo = min(w_hi, w_lo + warp * run), r_hi = min(w_hi, r_lo + run);
  const int32_t* src = block_idx + block_idx_row(p, seq, hq, sp.bos, row0 + r_lo);
  const int n = (r_hi - r_lo) * p.slots;
  int* cursor = cursor_all + warp * nb_lim;

  for (int i = threadIdx.x; i < W * nb_lim; i += 32 * W) cursor_all[i] = 0;
  __syncthreads();
  for (int e = lane; e < n; e += 32) {
    const int blk = src[e] >> part_shift;
    if (blk >= 0 && blk < nb_lim) atomicAdd(&cursor[blk], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb_lim; i += 32 * W) {
    int at = off[i] + pre[(size_t)i * (group * C)];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const int t = cursor_all[w * nb_lim + i];
      cursor_all[w * nb_lim + i] = at;
      at += t;
    }
  }
  __syncthreads();

  int32_t* ro = rows_out + kv_row * capacity;
  int32_t* ho = heads_out + kv_row * capacity;
  int32_t* so = slots_out + kv_row * capacity;
  int2* eo = entries_out + kv_row * capacity;
  const unsigned lt = (1u << lane) - 1u;
  const int first_row = sp.bos + row0 + r_lo;
  // The entries are fetched a batch of kBatch steps ahead: one memory latency per batch
  // instead of one per step.
  constexpr int kBatch = 4;
  int nxt[kBatch];
#pragma unroll
  for (int j = 0; j < kBatch; ++j) {
    const int e = j * 32 + lane;
    nxt[j] = (e < n) ? src[e] : -1;
  }
  for (int e0 = 0; e0 < n; e0 += 32 * kBatch) {
    int cur[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      cur[j] = nxt[j];
      const int e = e0 + 32 * kBatch + j * 32 + lane;
      nxt[j] = (e < n) ? src[e] : -1;
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int e = e0 + j * 32 + lane;
      if (e0 + j * 32 >= n) break;                         // warp-uniform
      const int blk = cur[j] >> part_shift;
      const bool valid = blk >= 0 && blk < nb_lim;
      const int key = valid ? blk : (0x40000000 + lane);
      const unsigned same = __match_any_sync(0xffffffffu, key);
      int base = 0;
      if (valid) base = cursor[blk];
      __syncwarp();
      if (valid && (same & lt) == 0) cursor[blk] = base + __popc(same);
      __syncwarp();
      if (valid) {
        const long long dst = base + __popc(same & lt);
        if (dst < capacity) {
          const int row = (int)((unsigned)e / (unsigned)p.slots), slot = e - row * p.slots;
          if constexpr (PACKED) {
            eo[dst] = make_int2(first_row + row, pack_pair(hq, cur[j] & ((1 << part_shift) - 1), slot));
          } else {
            ro[dst] = first_row + row;
            ho[dst] = hq;
            so[dst] = slot;
          }
        }
      }
    }
  }
}

// warps per scatter CTA: as many runs side by side as their cursor arrays leave room for
static inline int scatter_warps_for(const moba_b200_problem& p) {
  const size_t hist_bytes = (size_t)p.num_blocks * sizeof(int);
  if (8 * hist_bytes <= 64 * 1024) return 8;
  if (4 * hist_bytes <= 200 * 1024) return 4;
  return 1;
}
void transpose_plan(const moba_b200_problem& p, int* chunk_rows, int* chunks, int* scatter_warps) {
  const TransposeGeom g = transpose_geom(p);
  *chunk_rows = g.chunk_rows; *chunks = g.chunks; *scatter_warps = scatter_warps_for(p);
}

template <int W, bool PACKED>
static int launch_scatter(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu,
                          const int32_t* tiles, const int32_t* col_offsets, int32_t* rows, int32_t* heads,
                          int32_t* slots, int2* entries, int part_shift, const TransposeGeom& g, long long capacity, cudaStream_t st) {
  const size_t smem = (size_t)W * p.num_blocks * sizeof(int);
  static SmemLimit limit;
  if (int rc = raise_smem_limit(limit, (const void*)scatter_kernel<W, PACKED>, smem)) return rc;
  const long long ctas = (long long)g.chunks * p.n_seq * p.q_heads;
  MOBA_CUDA_OK(launch_chained(scatter_kernel<W, PACKED>, (unsigned)ctas, 32 * W, smem, st, block_idx, cu, tiles, col_offsets,
                              rows, heads, slots, entries, p, part_shift, g.chunk_rows, g.chunks, capacity));
  return MOBA_B200_OK;
}

// `entries` non-null: packed pairs, and rows / heads / slots are not written. `part_shift`: the
// block ids are those of blocks 2^part_shift times finer than the columns of `p`.
int launch_transpose(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu,
                     int32_t* col_nnz, int32_t* col_offsets, int32_t* order, int32_t* rows,
                     int32_t* heads, int32_t* slots, int2* entries, int part_shift, int32_t* work_items, void* scratch,
                     size_t scratch_bytes, cudaStream_t st) {
  const TransposeGeom g = transpose_geom(p);
  if (scratch_bytes < transpose_scratch_bytes(p)) {
    set_error("transpose: scratch has %zu bytes, needs %zu", scratch_bytes,
              transpose_scratch_bytes(p));
    return MOBA_B200_ESCRATCH;
  }
  const size_t hist_bytes = (size_t)p.num_blocks * sizeof(int);
  if (hist_bytes > 200 * 1024) {
    set_error("transpose: %d blocks per sequence exceed the shared-memory histogram", p.num_blocks);
    return MOBA_B200_EUNSUPPORTED;
  }
  const long long row_ctas = (long long)g.chunks * p.n_seq * p.q_heads;
  if (row_ctas > 0x7fffffffLL) {
    set_error("transpose: %lld (row chunk, sequence, head) units exceed the grid limit", row_ctas);
    return MOBA_B200_EUNSUPPORTED;
  }
  int32_t* tiles = static_cast<int32_t*>(scratch);
  int32_t* slot_counter = reinterpret_cast<int32_t*>(static_cast<unsigned char*>(scratch) + ((tile_count_bytes(p) + 15) & ~size_t(15)));
  if (sched_items_per_row(p) > 0x7fffffffLL || sched_part_slots(p) > 0x7fffffffLL) {
    set_error("transpose: chunk_tiles %d cuts the problem into too many work items", sched_chunk_tiles(p));
    return MOBA_B200_EUNSUPPORTED;
  }
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("transpose: no device error word"); return MOBA_B200_ECUDA; }
  const int group = p.q_heads / p.kv_heads;
  const long long capacity = (long long)group * (p.win_rows > 0 ? p.win_rows : p.max_seqlen) * p.slots;
  static SmemLimit count_limit, order_limit;
  if (int rc = raise_smem_limit(count_limit, (const void*)count_kernel, hist_bytes)) return rc;
  if (int rc = raise_smem_limit(order_limit, (const void*)offsets_order_kernel, hist_bytes)) return rc;
  { KernelTimer t__("count_kernel", st);
  MOBA_CUDA_OK(launch_chained(count_kernel, (unsigned)row_ctas, 256, hist_bytes, st, block_idx, cu, tiles, slot_counter, p, part_shift,
                              g.chunk_rows, g.chunks)); }
  { KernelTimer t__("colscan_kernel", st);
  const unsigned per_row = (unsigned)((p.num_blocks + 3) / 4);
  MOBA_CUDA_OK(launch_chained(colscan_kernel, per_row * (unsigned)(p.n_seq * p.kv_heads), 128, 0, st, cu, tiles, col_nnz, p,
                              g.chunk_rows, g.chunks, (int)per_row)); }
  { KernelTimer t__("offsets_order_kernel", st);
  MOBA_CUDA_OK(launch_chained(offsets_order_kernel, dim3(p.n_seq * p.kv_heads, (p.num_blocks + 127) / 128), 1024, hist_bytes, st,
                              (const int32_t*)col_nnz, col_offsets, order, p.num_blocks)); }
  if (work_items != nullptr) {
    KernelTimer t__("work_items_kernel", st);
    MOBA_CUDA_OK(launch_chained(work_items_kernel, p.n_seq * p.kv_heads, 1024, 0, st, (const int32_t*)col_nnz, (const int32_t*)order,
                                reinterpret_cast<int4*>(work_items), slot_counter, p.num_blocks, (int)sched_items_per_row(p),
                                sched_chunk_tiles(p), (int)sched_part_slots(p), err));
  }
  KernelTimer t__("scatter_kernel", st);
  const int w = scatter_warps_for(p);
#define MOBA_SCATTER(W) \
  return entries != nullptr ? launch_scatter<W, true>(p, block_idx, cu, tiles, col_offsets, rows, heads, slots, entries, part_shift, g, capacity, st) \
                            : launch_scatter<W, false>(p, block_idx, cu, tiles, col_offsets, rows, heads, slots, entries, part_shift, g, capacity, st)
  if (w == 8) MOBA_SCATTER(8);
  if (w == 4) MOBA_SCATTER(4);
  MOBA_SCATTER(1);
#undef MOBA_SCATTER
}

// ---------------------------------------------------------------------------
// Short rows: the five passes in one launch, one cluster of CTAs per (sequence, kv head).
//
// The cluster's warps cut the row's queries, in (query head, position) order, into consecutive
// runs, and hold the block ids of their run in registers. A histogram per warp, a scan over the
// warps of a CTA and one exchange of column totals over distributed shared memory give every warp
// its own cursors; the walk that follows is the one of scatter_kernel, so the order inside a column
// is the same. The last CTA of the cluster also writes the work items: the pieces of `tc` tiles
// first, then the last piece of every column by size (the same balance as write_work_items, whose
// block-wide passes cost this kernel a quarter of its time). What bounds it is latency: one read
// of the selections, two cluster barriers and the walk.
// Lines: up to kSmallBlocks columns, because one CTA ranks them all against one another, and up
// to kSmallPairs pairs per row and cluster; a longer row leaves too much to one cluster.
// ---------------------------------------------------------------------------
constexpr int kSmallBlocks = 512;
constexpr int kSmallCluster = 8, kWideCluster = 16;
constexpr long long kSmallPairs = 1 << 17;
constexpr int kSmallThreads = 1024, kSmallWarps = kSmallThreads / 32;

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int ld_cluster_i32(const int* mine, uint32_t rank) {
  uint32_t local = sm100::smem_u32(mine), remote;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
  return v;
}

// K: block ids per lane, an upper bound of the run's entries / 32. C: CTAs of the cluster.
template <int K, int C>
__global__ void __launch_bounds__(kSmallThreads, 1)
transpose_small_kernel(const int32_t* __restrict__ block_idx, const int32_t* __restrict__ cu, int32_t* __restrict__ col_nnz,
                       int32_t* __restrict__ col_offsets, int32_t* __restrict__ order, int2* __restrict__ entries, int4* __restrict__ items,
                       int32_t* __restrict__ slot_counter, moba_b200_problem p, unsigned slots_recip, int part_shift, long long capacity,
                       int items_per_row, int tc, int slot_cap, unsigned* error_word) {
  extern __shared__ int cursor_all[];                        // [warps][nb]
  __shared__ int totals[kSmallBlocks];                       // this CTA's pairs per column (read by its peers)
  __shared__ int base_s[kSmallBlocks];
  __shared__ int2 size_s[kSmallBlocks];                      // pairs of a column, tiles of its last piece
  __shared__ int warp_sums[32], warp_pieces[32], slot_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = p.num_blocks;
  const uint32_t rank = cluster_rank();
  for (int i = threadIdx.x; i < kSmallWarps * nb; i += kSmallThreads) cursor_all[i] = 0;
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  const int kv_row = (int)(blockIdx.x / C);
  const int seq = kv_row / p.kv_heads, kvh = kv_row % p.kv_heads;
  const int group = p.q_heads / p.kv_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const unsigned slots = (unsigned)p.slots;
  // this warp's run of queries, in (head, position) order
  const unsigned total_q = (unsigned)group * (unsigned)sp.len;
  const unsigned per_warp = (total_q + C * kSmallWarps - 1) / (C * kSmallWarps);
  const unsigned q_lo = min(total_q, (rank * kSmallWarps + warp) * per_warp), q_hi = min(total_q, q_lo + per_warp);
  const int n = (int)((q_hi - q_lo) * slots);
  int g0 = 0, r0 = (int)q_lo;                                // head and position of the run's first query
  if (sp.len > 0) { g0 = (int)(q_lo / (unsigned)sp.len); r0 = (int)(q_lo - (unsigned)g0 * (unsigned)sp.len); }
  const size_t head0 = (p.packed ? 0 : (size_t)seq * p.q_heads) + (size_t)kvh * group;
  // entry e of the run: its query (head of the group, position) and slot; e < 2^16
  auto entry = [&](int e, int& g, int& row, int& slot) {
    const unsigned qi = slots == 1 ? (unsigned)e : __umulhi((unsigned)e, slots_recip);
    slot = e - (int)(qi * slots);
    row = r0 + (int)qi; g = g0;
    while (row >= sp.len) { row -= sp.len; ++g; }
  };
  int* cursor = cursor_all + warp * nb;
  int id[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int e = k * 32 + lane;
    id[k] = -1;
    if (e < n) {
      int g, row, slot;
      entry(e, g, row, slot);
      id[k] = __ldg(block_idx + ((head0 + g) * p.tokens + sp.bos + row) * (size_t)slots + slot);
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int blk = id[k] >> part_shift;
    if (blk >= 0 && blk < nb) atomicAdd(&cursor[blk], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += kSmallThreads) {
    int at = 0;
#pragma unroll 1
    for (int w0 = 0; w0 < kSmallWarps; w0 += 16) {
      int c[16];
#pragma unroll
      for (int w = 0; w < 16; ++w) c[w] = cursor_all[(w0 + w) * nb + i];
#pragma unroll
      for (int w = 0; w < 16; ++w) {
        cursor_all[(w0 + w) * nb + i] = at;
        at += c[w];
      }
    }
    totals[i] = at;
  }
  cluster_barrier();
  // column i: its pairs in the CTAs before this one, and in all of them
  int mine = 0, before = 0;
  const int col = threadIdx.x;                               // nb <= kSmallBlocks < threads
  if (col < nb) {
    int t[C];
#pragma unroll
    for (int c = 0; c < C; ++c) t[c] = ld_cluster_i32(&totals[col], (uint32_t)c);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      mine += t[c];
      before += c < (int)rank ? t[c] : 0;
    }
  }
  const int tiles = (mine + 127) / 128;
  const int pieces = tiles <= tc ? 1 : (tiles + tc - 1) / tc;   // of the column; all but the last have tc tiles
  const int last_tiles = tiles - (pieces - 1) * tc;
  if (col < nb) size_s[col] = make_int2(mine, last_tiles);
  // scans over the columns: pairs; full pieces (low half) and partial slots (high half)
  int incl = mine, cuts = col < nb ? (pieces - 1) | ((pieces > 1 ? pieces : 0) << 16) : 0, cuts_incl = cuts;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o), u = __shfl_up_sync(0xffffffffu, cuts_incl, o);
    if (lane >= o) { incl += t; cuts_incl += u; }
  }
  if (lane == 31) { warp_sums[warp] = incl; warp_pieces[warp] = cuts_incl; }
  __syncthreads();
  int off = incl - mine, cuts_before = cuts_incl - cuts, cuts_all = 0;
  for (int w = 0; w * 32 < nb; ++w) {
    if (w < warp) { off += warp_sums[w]; cuts_before += warp_pieces[w]; }
    cuts_all += warp_pieces[w];
  }
  if (col < nb) base_s[col] = off + before;
  const bool lister = rank == C - 1;
  if (lister && threadIdx.x == 0) {
    const int need = (int)((unsigned)cuts_all >> 16);
    const int base = need > 0 ? atomicAdd(slot_counter, need) : 0;
    slot_base = base;
    if (base + need > slot_cap || (cuts_all & 0xffff) + nb > items_per_row) atomicOr(error_word, 2u);   // sizes were promised by the host
  }
  cluster_barrier();                                         // totals have been read; base_s is complete

  int2* eo = entries + (size_t)kv_row * capacity;
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k * 32 >= n) break;                                  // warp-uniform
    const int blk = id[k] >> part_shift;
    const bool valid = blk >= 0 && blk < nb;
    const unsigned same = __match_any_sync(0xffffffffu, valid ? blk : (0x40000000 + lane));
    int base = 0;
    if (valid) base = cursor[blk];
    __syncwarp();
    if (valid && (same & lt) == 0) cursor[blk] = base + __popc(same);
    __syncwarp();
    if (valid) {
      int g, row, slot;
      entry(k * 32 + lane, g, row, slot);
      const long long dst = (long long)base_s[blk] + base + __popc(same & lt);
      if (dst < capacity) eo[dst] = make_int2(sp.bos + row, pack_pair(kvh * group + g, id[k] & ((1 << part_shift) - 1), slot));
    }
  }
  if (!lister) return;
  int4* out = items + (size_t)kv_row * items_per_row;
  const int n_full = cuts_all & 0xffff;
  if (col < nb) {
    col_nnz[(size_t)kv_row * nb + col] = mine;
    col_offsets[(size_t)kv_row * (nb + 1) + col] = off;
    if (col == nb - 1) col_offsets[(size_t)kv_row * (nb + 1) + nb] = off + mine;
    // stable descending ranks: of the column by pairs, of its last piece by tiles
    int by_pairs = 0, by_piece = 0;
    for (int j = 0; j < nb; ++j) {
      const int2 o = size_s[j];
      by_pairs += (o.x > mine || (o.x == mine && j < col)) ? 1 : 0;
      by_piece += (o.y > last_tiles || (o.y == last_tiles && j < col)) ? 1 : 0;
    }
    order[(size_t)kv_row * nb + by_pairs] = col;
    const int full0 = cuts_before & 0xffff, slot0 = slot_base + (int)((unsigned)cuts_before >> 16);
    auto slot_or_none = [&](int i) { return pieces > 1 && slot0 + i < slot_cap ? slot0 + i : -1; };
    for (int i = 0; i + 1 < pieces; ++i)
      if (full0 + i < items_per_row) out[full0 + i] = make_int4(col, i * tc, tc, slot_or_none(i));
    if (n_full + by_piece < items_per_row) out[n_full + by_piece] = make_int4(col, (pieces - 1) * tc, last_tiles, slot_or_none(pieces - 1));
  }
  for (int j = n_full + nb + threadIdx.x; j < items_per_row; j += kSmallThreads) out[j] = make_int4(0, n_full, 0, -2);   // padding, which tells how many pieces lead the row
}

// Entries of a warp's run: at most this many per lane.
static inline int small_ids_per_lane(const moba_b200_problem& p, int cluster = kSmallCluster) {
  const long long total_q = (long long)(p.q_heads / p.kv_heads) * p.max_seqlen;
  const long long per_warp = (total_q + cluster * kSmallWarps - 1) / (cluster * kSmallWarps);
  return (int)((per_warp * p.slots + 31) / 32);
}

bool transpose_small_supported(const moba_b200_problem& p) {
  const long long row_pairs = (long long)(p.q_heads / p.kv_heads) * p.max_seqlen * p.slots;
  return p.num_blocks <= kSmallBlocks && row_pairs <= kSmallPairs && p.win_rows == 0 && small_ids_per_lane(p) <= 20 &&
         row_pairs / (128LL * sched_chunk_tiles(p)) < 16384 &&        // two piece counts share a word
         (long long)p.n_seq * p.kv_heads * kSmallCluster < 0x7fffffffLL;
}

// Whether the current device can hold a cluster of kWideCluster CTAs with the largest shared memory
// they take here (more than eight is not portable). Asked once per device, which also allows it to
// the kernels.
static bool wide_clusters_fit() {
  static int known[64];                                      // 0 unknown, 1 yes, -1 no; written alike by whoever asks first
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (__atomic_load_n(&known[dev], __ATOMIC_ACQUIRE) == 0) {
    const auto kern = transpose_small_kernel<12, kWideCluster>;
    const size_t smem = (size_t)kSmallWarps * kSmallBlocks * sizeof(int);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kWideCluster; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kWideCluster); cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem; cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                    cudaFuncSetAttribute(transpose_small_kernel<4, kWideCluster>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaFuncSetAttribute(transpose_small_kernel<8, kWideCluster>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1;
    if (!ok) cudaGetLastError();
    __atomic_store_n(&known[dev], ok ? 1 : -1, __ATOMIC_RELEASE);
  }
  return __atomic_load_n(&known[dev], __ATOMIC_ACQUIRE) > 0;
}

// `slot_counter` must hold zero.
int launch_transpose_small(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu, int32_t* col_nnz,
                           int32_t* col_offsets, int32_t* order, int2* entries, int part_shift, int32_t* work_items,
                           int32_t* slot_counter, cudaStream_t st) {
  KernelTimer t__("transpose_small_kernel", st);
  unsigned* err = device_error_word();
  if (err == nullptr) { set_error("transpose: no device error word"); return MOBA_B200_ECUDA; }
  const size_t smem = (size_t)kSmallWarps * p.num_blocks * sizeof(int);
  // A few rows: clusters of sixteen, if the device has room for one. The scattered stores, a line per
  // entry, take about half of the kernel at 8192 keys a row: 4 rows 21.0 us with eight CTAs each, 16.8
  // with sixteen. Eight rows are slower (20.6 and 23.0): a part of the chip holds one such cluster.
  int cluster = kSmallCluster;
  if (p.n_seq * p.kv_heads <= 4 && small_ids_per_lane(p) > 2 && wide_clusters_fit()) cluster = kWideCluster;
  const bool wide = cluster == kWideCluster;
  const int k = small_ids_per_lane(p, cluster);
  const int which = (wide ? 3 : 0) + (k <= 4 ? 0 : (k <= 8 ? 1 : 2));
  const decltype(&transpose_small_kernel<4, kSmallCluster>) kernels[6] = {
      transpose_small_kernel<4, kSmallCluster>, transpose_small_kernel<8, kSmallCluster>, transpose_small_kernel<20, kSmallCluster>,
      transpose_small_kernel<4, kWideCluster>, transpose_small_kernel<8, kWideCluster>, transpose_small_kernel<12, kWideCluster>};
  auto kern = kernels[which];
  static SmemLimit limit[6];
  if (int rc = raise_smem_limit(limit[which], (const void*)kern, smem)) return rc;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.n_seq * p.kv_heads * cluster)); cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 2;
  const long long capacity = (long long)(p.q_heads / p.kv_heads) * p.max_seqlen * p.slots;
  const unsigned recip = (unsigned)(((1ull << 32) + p.slots - 1) / p.slots);    // e / slots for e < 2^16 and slots > 1
  MOBA_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, block_idx, cu, col_nnz, col_offsets, order, entries,
                                  reinterpret_cast<int4*>(work_items), slot_counter, p, recip, part_shift, capacity,
                                  (int)sched_items_per_row(p), sched_chunk_tiles(p), (int)sched_part_slots(p), err));
  return MOBA_B200_OK;
}

// ---------------------------------------------------------------------------
// Transpose for callers that cannot hand over scratch memory.
//
// Some hosts of this library may not allocate device memory at all: a serving
// process that lays out every byte of the GPU at start-up and forbids cudaMalloc
// afterwards (it synchronises the device and can fail once memory is
// fragmented), or a plugin that is handed nothing but its input and output
// buffers and has no allocator to ask. For them the per-chunk histogram of the
// transpose lives in this fixed array inside the library image. Every GPU that
// loads the library keeps these 8 MiB until the process exits.
//
// `g_transpose_scratch` names the array in device code. In host code the same
// name is only a handle for cudaGetSymbolAddress: passing it to a kernel as a
// pointer would hand the kernel a host address.
// ---------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = size_t(8) << 20;
static __device__ __align__(256) unsigned char g_transpose_scratch[kStaticScratchBytes];

// Device address of the array on the current device; looked up once per device,
// with that device current, and cached.
static int static_scratch_address(void** out) {
  static void* table[64] = {nullptr};
  static std::mutex mu;
  int dev = -1;
  MOBA_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_error("device ordinal %d out of range", dev); return MOBA_B200_EUNSUPPORTED; }
  std::lock_guard<std::mutex> lock(mu);
  if (table[dev] == nullptr) {
    void* ptr = nullptr;
    MOBA_CUDA_OK(cudaGetSymbolAddress(&ptr, g_transpose_scratch));
    table[dev] = ptr;
  }
  *out = table[dev];
  return MOBA_B200_OK;
}

int launch_transpose_noalloc(const moba_b200_problem& p, const int32_t* block_idx, const int32_t* cu,
                             int32_t* col_nnz, int32_t* col_offsets, int32_t* order, int32_t* rows,
                             int32_t* heads, int32_t* slots, int32_t* work_items, cudaStream_t st) {
  const size_t need = transpose_scratch_bytes(p);
  if (need > kStaticScratchBytes) {
    set_error("transpose without caller scratch: this problem needs %zu bytes of scratch, the built-in "
              "array holds %zu; use moba_b200_transpose with a caller buffer", need, kStaticScratchBytes);
    return MOBA_B200_EUNSUPPORTED;
  }
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != MOBA_B200_OK) return rc;
  // Nothing in the array has to be cleared by the caller: the count pass writes every entry
  // the scan pass reads and resets the slot counter, so the previous call's contents are
  // simply overwritten.
  return launch_transpose(p, block_idx, cu, col_nnz, col_offsets, order, rows, heads, slots, nullptr, 0, work_items, scratch,
                          kStaticScratchBytes, st);
}

}  // namespace moba
