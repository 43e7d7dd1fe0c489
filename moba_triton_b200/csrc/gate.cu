// Gate, portable kernels: block mean-pooling and the exact (float64) scorer with
// warp-level top-k selection. These run for every dtype / block size / head
// dim; the tcgen05 scorer in gate_sm100.cu replaces the second one for
// 16-bit inputs.
//
// Numerics contract (what makes selections comparable bit for bit):
//   block sum  = round_T(float(exact sum))      exact sum accumulated in float64
//   block mean = round_T(float(sum) / float(occupancy))
//   score      = round_T(float(exact dot))      unscaled
//   rank by (score desc, block id asc) over blocks strictly before the query's
//   own block; the own block is appended, never ranked.
// Reference behaviour being reproduced: src/moba/kernels/pooling.py:77-95 and
// src/moba/kernels/gating.py:183-335 (float32 accumulation there).
#include "common.cuh"

#include <float.h>

namespace moba {

// ---------------------------------------------------------------------------
// pool: grid (num_blocks, n_seq * Hkv), 128 or 256 threads
// ---------------------------------------------------------------------------
// NT threads of a block of keys, four rows in flight per thread. The conversions to float64 bound the 16-bit types (16
// a clock and SM), the memory latency float32, which takes 256 threads where a block has rows for them. us in
// float32, with 128 threads, 256, and 256 with eight rows in flight and sums over the lanes of a warp first:
//   8192 x 4 heads of 64       16.1  12.3  12.2         131072 x 4 of 64                     55  57   92
//   16384 x 2 of 128           24.4  16.2  16.3         16384 x 4 of 64, blocks of 16        14  20   35
// (The third kept so much in registers that a large call had too few CTAs on an SM.)
template <typename T, int NT>
__global__ void __launch_bounds__(NT)
pool_kernel(const T* __restrict__ k, const int32_t* __restrict__ cu, T* __restrict__ kbar,
            int packed, int tokens, int hkv, int d, int bs, int nb, int* __restrict__ zero_cell, float* __restrict__ norms) {
  pdl_trigger();
  pdl_wait();
  if (zero_cell != nullptr && blockIdx.x == 0 && threadIdx.x == 0) zero_cell[0] = zero_cell[1] = 0;
  constexpr int EPV = 16 / sizeof(T);            // elements per 16-byte vector
  const int blk = (int)(blockIdx.x % nb), kv_row = (int)(blockIdx.x / nb);
  const int seq = kv_row / hkv, h = kv_row % hkv;
  const SeqSpan sp = seq_span(cu, packed, seq, tokens);
  const int vpr = d / EPV;                       // vectors per row
  const int groups = NT / vpr;
  const int c = threadIdx.x % vpr, rg = threadIdx.x / vpr;

  T* dst = kbar + ((size_t)kv_row * nb + blk) * d;
  const int lo = blk * bs;
  if (lo >= sp.len) {                            // padded slot of a short packed sequence
    if (threadIdx.x < d) dst[threadIdx.x] = Elem<T>::from_f(0.f);
    for (int i = threadIdx.x + NT; i < d; i += NT) dst[i] = Elem<T>::from_f(0.f);
    if (norms != nullptr && threadIdx.x == 0) norms[(size_t)kv_row * nb + blk] = 0.f;
    return;
  }
  const int hi = min(lo + bs, sp.len);
  const size_t batch_base = packed ? 0 : (size_t)seq * tokens;
  const T* src = k + ((batch_base + sp.bos + lo) * hkv + h) * (size_t)d + c * EPV;
  const size_t row_stride = (size_t)hkv * d;

  double acc[EPV];
#pragma unroll
  for (int e = 0; e < EPV; ++e) acc[e] = 0.0;
  if (rg < groups) {
    constexpr int kAhead = 4;                                    // the loads do not depend on one another
    for (int r0 = rg; r0 < hi - lo; r0 += groups * kAhead) {
      uint4 raw[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int r = r0 + u * groups;
        raw[u] = (r < hi - lo) ? *reinterpret_cast<const uint4*>(src + r * row_stride) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (r0 + u * groups < hi - lo) {
          const T* vals = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
          for (int e = 0; e < EPV; ++e) acc[e] += (double)Elem<T>::to_f(vals[e]);
        }
      }
    }
  }
  // Sums over the row groups, one output element per thread (float64 sums of these values are
  // exact, so the order of the additions does not matter).
  __shared__ double red[NT * EPV];
#pragma unroll
  for (int e = 0; e < EPV; ++e) red[threadIdx.x * EPV + e] = acc[e];
  __syncthreads();
  const float occ = (float)(hi - lo);
  double square = 0.0;                                          // in float64: no square leaves its range
  for (int i = threadIdx.x; i < d; i += NT) {
    double s = 0.0;
    for (int g = 0; g < groups; ++g) s += red[g * d + i];       // thread g * vpr + i / EPV, element i % EPV
    const float total = Elem<T>::round_f((float)s);
    const T mean = Elem<T>::from_f(__fdiv_rn(total, occ));
    dst[i] = mean;
    square = fma((double)Elem<T>::to_f(mean), (double)Elem<T>::to_f(mean), square);
  }
  if (norms == nullptr) return;
  // the block mean's length, for the error bound of the exact gate
  __shared__ double squares[NT / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) square += __shfl_xor_sync(0xffffffffu, square, o);
  if ((threadIdx.x & 31) == 0) squares[threadIdx.x >> 5] = square;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < NT / 32; ++w) squares[0] += squares[w];
    norms[(size_t)kv_row * nb + blk] = (float)sqrt(squares[0]);
  }
}

// `zero_cell` (may be NULL): two counters that later kernels of the same op claim from; `norms`
// (may be NULL): the length of every block mean, [n_seq, Hkv, num_blocks].
int launch_pool(const moba_b200_problem& p, const void* k, const int32_t* cu, void* kbar, int* zero_cell, float* norms,
                cudaStream_t st) {
  KernelTimer timer__("pool_kernel", st);
  const int epv = 16 / (int)dtype_size(p.dtype);
  if (p.head_dim % epv || p.head_dim / epv > 128) {
    set_error("pool: head_dim %d unsupported", p.head_dim);
    return MOBA_B200_EUNSUPPORTED;
  }
  const long long ctas = (long long)p.num_blocks * p.n_seq * p.kv_heads;
  if (ctas > 0x7fffffffLL) { set_error("pool: %lld blocks exceed the grid limit", ctas); return MOBA_B200_EUNSUPPORTED; }
  const unsigned grid = (unsigned)ctas;
#define MOBA_POOL(T, NT)                                                                               \
  MOBA_CUDA_OK(launch_chained(pool_kernel<T, NT>, grid, NT, 0, st, (const T*)k, cu, (T*)kbar, p.packed, p.tokens, \
                              p.kv_heads, p.head_dim, p.block_size, p.num_blocks, zero_cell, norms))
  // (by the block size alone: the sums of a sequence do not depend on what else is in the call)
  if (p.dtype == MOBA_B200_F32 && p.block_size >= 64) MOBA_POOL(float, 256);
  else if (p.dtype == MOBA_B200_F32) MOBA_POOL(float, 128);
  else if (p.dtype == MOBA_B200_BF16) MOBA_POOL(__nv_bfloat16, 128);
  else MOBA_POOL(__half, 128);
#undef MOBA_POOL
  return MOBA_B200_OK;
}

// ---------------------------------------------------------------------------
// portable gate: grid (cdiv(max_seqlen, 32), n_seq * Hq), 128 threads.
// Each warp owns 8 query rows; a lane scores one candidate block of the
// current 32-block chunk for all 8 rows in float64, then the warp merges the
// chunk into each row's running list (over its lanes; past 32 entries in shared memory).
// ---------------------------------------------------------------------------
constexpr int kGateRows = 32;
constexpr int kGateChunk = 32;
constexpr int kRowsPerWarp = 8;
constexpr int kEmptyIdx = 0x7fffffff;

struct Cand {
  float v;
  int i;
};
// best = larger score, ties to the smaller id
__device__ __forceinline__ Cand warp_best(Cand c) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, c.v, o);
    int oi = __shfl_xor_sync(0xffffffffu, c.i, o);
    if (ov > c.v || (ov == c.v && oi < c.i)) { c.v = ov; c.i = oi; }
  }
  return c;
}
// weakest = smaller score, ties to the larger id (so the lower id survives)
__device__ __forceinline__ Cand warp_weakest(Cand c, int& slot) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, c.v, o);
    int oi = __shfl_xor_sync(0xffffffffu, c.i, o);
    int os = __shfl_xor_sync(0xffffffffu, slot, o);
    if (ov < c.v || (ov == c.v && (oi > c.i || (oi == c.i && os < slot)))) {
      c.v = ov; c.i = oi; slot = os;
    }
  }
  return c;
}

// Score (descending) and block id (ascending) as one number; 0 for what cannot be selected.
__device__ __forceinline__ unsigned long long rank_key(float s, int blk) {
  if (!(s > -INFINITY)) return 0ull;
  const unsigned u = __float_as_uint(s + 0.f);                   // one zero
  return (unsigned long long)(u & 0x80000000u ? ~u : u | 0x80000000u) << 32 | (0xffffffffu - (unsigned)blk);
}
__device__ __forceinline__ unsigned long long exchange(unsigned long long x, int j, bool keep_larger) {
  const unsigned long long o = __shfl_xor_sync(0xffffffffu, x, j);
  return (x > o) == keep_larger ? x : o;
}
// Bitonic: the warp's 32 keys of each row in descending order over the lanes. The rows go in step: an exchange
// waits for its shuffles, and N rows' wait together.
template <int N>
__device__ __forceinline__ void sort_lanes(unsigned long long (&x)[N], int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j >= 1; j >>= 1)
#pragma unroll
      for (int r = 0; r < N; ++r) x[r] = exchange(x[r], j, ((lane & j) == 0) == ((lane & k) == 0));
}
// a: the 32 largest of two descending sequences each, descending.
template <int N>
__device__ __forceinline__ void merge_sorted(unsigned long long (&a)[N], const unsigned long long (&b)[N], int lane) {
#pragma unroll
  for (int r = 0; r < N; ++r) {
    const unsigned long long o = __shfl_sync(0xffffffffu, b[r], 31 - lane);
    a[r] = a[r] > o ? a[r] : o;
  }
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1)
#pragma unroll
    for (int r = 0; r < N; ++r) a[r] = exchange(a[r], j, (lane & j) == 0);
}
// SORTED: up to 32 ranked blocks. The row's list lies sorted over the lanes of its warp, and a chunk
// of 32 candidates is sorted and merged into it in 21 exchanges; offering them one by one, a reduction
// over the warp and two over the list each, was two thirds of the kernel ([1,4096,4,64] float32,
// 7 of 32 blocks: 76 us, sorted 29, with the eight rows of a warp in step and two numbers a load 25).
// IN_STEP: the exchanges of the eight rows of a warp wait together, in every chunk that enters a list of theirs.
// That takes 128 registers, four CTAs an SM, where six fit the shared memory of head_dim 64, and the further a row
// goes the fewer of its chunks enter its list; the longer the list, the more do. Row by row, in 80 registers, the
// time is, of that in step (2 heads of 64 in float32, blocks of 16 unless noted, by ranked and all blocks):
//    1   500 1.06    700 0.98    850 0.98              9  1100 1.12   1500 1.01   2000 0.98
//    2   700 1.02    850 1.00   1024 0.97   4096 0.92  12  1500 1.03   2000 1.00   3000 0.96
//    4   800 1.10   1024 1.02                         16  1500 1.05   2000 1.03   3000 0.98   4096 0.95
//    7  1100 1.09   1500 0.99   2000 0.96             21  3000 1.04   4096 1.02
//    7 (of 128)  800 1.01   1000 0.98   1400 0.94     31  2500 1.12   4096 1.06   8000 0.97
// From head_dim 128 on the shared memory holds three CTAs whatever the registers (7 of 1024 blocks 1.20). (A minimum
// of 0 CTAs leaves the registers to the compiler, 128 and, without SORTED, 96; a minimum of one let it take 201,
// and [1,4096,4,64] 35 us.)
template <typename T, bool SORTED, bool IN_STEP>
__global__ void __launch_bounds__(128, SORTED && !IN_STEP ? 6 : 0)
gate_portable_kernel(const T* __restrict__ q, const T* __restrict__ kbar,
                     const int32_t* __restrict__ cu, int32_t* __restrict__ block_idx,
                     float* __restrict__ lse_fill, moba_b200_problem p) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int d = p.head_dim, take = p.take, slots = p.slots;
  const int qst = (d + 1) / 2 * 2;
  double* qs = reinterpret_cast<double*>(smem_raw);                       // [32][qst]
  const int kst = (d + 1) / 2 * 2 + 2;                                    // row stride of ks: lanes on different banks, 16-byte rows
  double* ks = qs + kGateRows * qst;                                      // [32][kst]
  float* lval = reinterpret_cast<float*>(ks + kGateChunk * kst);      // [32][take]
  int* lidx = reinterpret_cast<int*>(lval + kGateRows * max(take, 1));    // [32][take]

  const int group = p.q_heads / p.kv_heads;
  const int seq = blockIdx.y / p.q_heads, hq = blockIdx.y % p.q_heads;
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const int row0 = blockIdx.x * kGateRows;
  if (row0 >= sp.len) return;
  const int n_cand = (sp.len + p.block_size - 1) / p.block_size;
  const size_t batch_base = p.packed ? 0 : (size_t)seq * p.tokens;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // stage the 32 query rows as float64; dead rows are zero
  for (int i = threadIdx.x; i < kGateRows * qst; i += 128) {
    const int r = i / qst, c = i % qst;
    double v = 0.0;
    if (c < d && row0 + r < sp.len)
      v = (double)Elem<T>::to_f(q[((batch_base + sp.bos + row0 + r) * p.q_heads + hq) * (size_t)d + c]);
    qs[i] = v;
  }
  for (int i = threadIdx.x; i < kGateRows * take; i += 128) {
    lval[i] = -INFINITY;
    lidx[i] = kEmptyIdx;
  }
  __syncthreads();

  const int last_row = min(row0 + kGateRows, sp.len) - 1;
  const int horizon = min(last_row / p.block_size, n_cand);      // blocks < horizon can be candidates
  const T* kb = kbar + ((size_t)seq * p.kv_heads + hq / group) * p.num_blocks * (size_t)d;
  float thr[kRowsPerWarp];                                       // current entry bar per row
  unsigned long long best[kRowsPerWarp];                         // SORTED: lane e holds the row's e-th best key, 0 = none
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) { thr[r] = -INFINITY; best[r] = 0ull; }

  for (int c0 = 0; take > 0 && c0 < horizon; c0 += kGateChunk) {
    __syncthreads();
    for (int i = threadIdx.x; i < kGateChunk * qst; i += 128) {
      const int j = i / qst, c = i % qst;
      ks[j * kst + c] = (c < d && c0 + j < n_cand) ? (double)Elem<T>::to_f(kb[(size_t)(c0 + j) * d + c]) : 0.0;
    }
    __syncthreads();

    double acc[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) acc[r] = 0.0;
    const double* krow = ks + lane * kst;
    const double* qrow = qs + warp * kRowsPerWarp * qst;
    for (int c = 0; c < qst; c += 2) {                             // (past d: zeros)
      const double2 kv = *reinterpret_cast<const double2*>(krow + c);
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r) {
        const double2 qv = *reinterpret_cast<const double2*>(qrow + r * qst + c);
        acc[r] = fma(qv.y, kv.y, fma(qv.x, kv.x, acc[r]));
      }
    }
    const int blk = c0 + lane;
    if constexpr (SORTED) {
      if constexpr (IN_STEP) {
        unsigned long long key[kRowsPerWarp];
        bool enters = false;
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r) {
          const int row = row0 + warp * kRowsPerWarp + r;
          const bool candidate = gate_candidate(p, blk, row / p.block_size) && blk < n_cand && row < sp.len;
          key[r] = candidate ? rank_key(Elem<T>::round_f((float)acc[r]), blk) : 0ull;
          const unsigned long long bar = __shfl_sync(0xffffffffu, best[r], take - 1);   // (by all lanes)
          enters |= key[r] > bar;
        }
        if (__any_sync(0xffffffffu, enters)) {
          sort_lanes(key, lane);
          merge_sorted(best, key, lane);
        }
      } else {
#pragma unroll
        for (int r = 0; r < kRowsPerWarp; ++r) {
          const int row = row0 + warp * kRowsPerWarp + r;
          const bool candidate = gate_candidate(p, blk, row / p.block_size) && blk < n_cand && row < sp.len;
          unsigned long long key[1] = {candidate ? rank_key(Elem<T>::round_f((float)acc[r]), blk) : 0ull}, list[1] = {best[r]};
          if (!__any_sync(0xffffffffu, key[0] > __shfl_sync(0xffffffffu, best[r], take - 1))) continue;
          sort_lanes(key, lane);
          merge_sorted(list, key, lane);
          best[r] = list[0];
        }
      }
      continue;
    }
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      const int lrow = warp * kRowsPerWarp + r;
      const int row = row0 + lrow;
      const int own = row / p.block_size;
      float s = Elem<T>::round_f((float)acc[r]);
      if (!(gate_candidate(p, blk, own) && blk < n_cand && row < sp.len)) s = -INFINITY;
      float* lv = lval + lrow * take;
      int* li = lidx + lrow * take;
      // offer the chunk's candidates in (score desc, id asc) order while they clear the bar
      while (__any_sync(0xffffffffu, s > thr[r])) {
        Cand best = warp_best(Cand{s, blk});
        // weakest list entry (ties: highest id; empty entries carry the largest id)
        Cand weak{INFINITY, -1};
        int wslot = 0x7fffffff;
        for (int e = lane; e < take; e += 32) {
          const float ev = lv[e];
          const int ei = li[e];
          if (ev < weak.v || (ev == weak.v && (ei > weak.i || (ei == weak.i && e < wslot)))) {
            weak.v = ev; weak.i = ei; wslot = e;
          }
        }
        weak = warp_weakest(weak, wslot);
        if (!(best.v > weak.v)) break;           // cannot happen while thr is current; safety
        if (lane == 0) { lv[wslot] = best.v; li[wslot] = best.i; }
        if (blk == best.i) s = -INFINITY;
        __syncwarp();
        // new bar = weakest entry after the insert
        float m = INFINITY;
        for (int e = lane; e < take; e += 32) m = fminf(m, lv[e]);
#pragma unroll
        for (int o = 16; o; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
        thr[r] = m;
      }
    }
  }
  __syncwarp();

  // emit ascending ids: rank every kept entry (and the own block) by id
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) {
    const int lrow = warp * kRowsPerWarp + r;
    const int row = row0 + lrow;
    if (row >= sp.len) continue;
    const int own = row / p.block_size;
    const int* li = lidx + lrow * take;
    const size_t b = p.packed ? 0 : (size_t)seq;
    const size_t out_at = ((b * p.q_heads + hq) * p.tokens + sp.bos + row) * (size_t)slots;
    int32_t* out = block_idx + out_at;
    if constexpr (SORTED) {
      const unsigned long long key = best[r];
      const bool have = lane < take && key != 0ull;
      const int id = have ? (int)(0xffffffffu - (unsigned)key) : kEmptyIdx;
      int rank = 0;
      for (int f = 0; f < take; ++f) rank += __shfl_sync(0xffffffffu, id, f) < id ? 1 : 0;
      int kept = __popc(__ballot_sync(0xffffffffu, have));
      if (have) out[rank] = id;
      if (p.always_current) {                                    // the own block is past every candidate
        if (lane == 0) out[kept] = own;
        ++kept;
      }
      for (int e = kept + lane; e < slots; e += 32) {
        out[e] = -1;
        if (lse_fill != nullptr) lse_fill[out_at + e] = -INFINITY;
      }
      continue;
    }
    const int n_items = take + (p.always_current ? 1 : 0);
    int kept = 0;
    for (int e = lane; e < n_items; e += 32) {
      const int id = (e < take) ? li[e] : own;
      if (id == kEmptyIdx) continue;
      int rank = 0;
      for (int f = 0; f < n_items; ++f) {
        const int other = (f < take) ? li[f] : own;
        rank += (other < id) ? 1 : 0;
      }
      out[rank] = id;
      ++kept;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) kept += __shfl_xor_sync(0xffffffffu, kept, o);
    for (int e = kept + lane; e < slots; e += 32) {
      out[e] = -1;
      if (lse_fill != nullptr) lse_fill[out_at + e] = -INFINITY;
    }
  }
}

int launch_gate_portable(const moba_b200_problem& p, const void* q, const void* kbar,
                         const int32_t* cu, int32_t* block_idx, float* lse_fill, cudaStream_t st) {
  KernelTimer timer__("gate_portable_kernel", st);
  const int d = p.head_dim;
  const int qst = (d + 1) / 2 * 2;
  const size_t smem = sizeof(double) * (kGateRows * qst + kGateChunk * (qst + 2)) +
                      (size_t)kGateRows * (p.take > 0 ? p.take : 1) * 8;
  if (smem > 200 * 1024) {
    set_error("gate: head_dim %d / top_k %d need %zu bytes of shared memory", d, p.top_k, smem);
    return MOBA_B200_EUNSUPPORTED;
  }
  if ((long long)p.n_seq * p.q_heads > 65535) {
    set_error("portable gate: %d sequences x %d heads exceed 65535 grid rows", p.n_seq, p.q_heads);
    return MOBA_B200_EUNSUPPORTED;
  }
  dim3 grid((p.max_seqlen + kGateRows - 1) / kGateRows, p.n_seq * p.q_heads);
  const bool in_step = d >= 128 || p.take > 16 || p.num_blocks <= 768 + 128 * p.take;
#define MOBA_GATE(T, SORTED, IN_STEP)                                                         \
  do {                                                                                        \
    static SmemLimit limit;                                                                   \
    if (int rc = raise_smem_limit(limit, (const void*)gate_portable_kernel<T, SORTED, IN_STEP>, smem)) return rc; \
    MOBA_CUDA_OK(launch_chained(gate_portable_kernel<T, SORTED, IN_STEP>, grid, 128, smem, st, (const T*)q, (const T*)kbar, cu, block_idx, lse_fill, p)); \
  } while (0)
#define MOBA_GATE_T(T)                                                                        \
  do {                                                                                        \
    if (p.take > 32) MOBA_GATE(T, false, false);                                              \
    else if (in_step) MOBA_GATE(T, true, true);                                               \
    else MOBA_GATE(T, true, false);                                                           \
  } while (0)
  if (p.dtype == MOBA_B200_F32) MOBA_GATE_T(float);
  else if (p.dtype == MOBA_B200_BF16) MOBA_GATE_T(__nv_bfloat16);
  else MOBA_GATE_T(__half);
#undef MOBA_GATE_T
#undef MOBA_GATE
  return MOBA_B200_OK;
}

}  // namespace moba
