// Forward, portable kernels: marker fill, KV-block-major attention on CUDA
// cores (any dtype / block size / head dim that fits shared memory) and the
// log2-sum-exp merge. The merge is shared with the tcgen05 forward.
//
// Numerics contract of the attention (same as the tcgen05 kernel):
//   s = (q . k) * D^-1/2 * log2(e)  in float32, masked (tail keys, and keys
//   after the query inside the own block when causal); m = max s;
//   p = exp2(s - m); l = sum p (unrounded); p is rounded to the dtype of v
//   before p.v; the partial stores O_i = (p.v)/l and lse_i = m + log2 l.
// Reference: src/moba/kernels/moba_fwd.py:229-425 (it stores m, l and the
// unnormalised accumulator instead; the merged result is the same quantity).
#include "common.cuh"

#include <cuda_pipeline.h>

namespace moba {

__global__ void fill_kernel(float* __restrict__ dst, size_t n, float value) {
  pdl_trigger();
  pdl_wait();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = value;
}

int launch_fill_lse(const moba_b200_problem& p, float* part_lse, cudaStream_t st) {
  KernelTimer timer__("fill_kernel", st);
  const size_t n = (size_t)p.batch * p.q_heads * window_rows(p) * p.slots;
  const int blocks = (int)((n + 1023) / 1024 < 148 * 8 ? (n + 1023) / 1024 : 148 * 8);
  MOBA_CUDA_OK(launch_chained(fill_kernel, blocks > 0 ? blocks : 1, 256, 0, st, part_lse, n, -INFINITY));
  return MOBA_B200_OK;
}

// ---------------------------------------------------------------------------
// portable attention: grid (num_blocks, n_seq * Hkv), 256 threads. A warp
// handles four gathered query rows at a time; lanes run over keys for the
// scores and over the head dim for p.v.
// ---------------------------------------------------------------------------
constexpr int kFwdWarps = 8;
constexpr int kFwdRows = 4;       // rows per warp iteration

template <typename T, typename TP>
__global__ void __launch_bounds__(256)
fwd_portable_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                    moba_b200_index ix, const int32_t* __restrict__ cu, TP* __restrict__ part_o,
                    float* __restrict__ part_lse, moba_b200_problem p) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int d = p.head_dim, bs = p.block_size, nb = p.num_blocks;
  const int kstride = d + 1;
  float* Ks = reinterpret_cast<float*>(smem_raw);           // [bs][d+1]
  float* Vs = Ks + bs * kstride;                            // [bs][d]
  float* Qs = Vs + bs * d;                                  // [warps][rows][d]
  float* Ps = Qs + kFwdWarps * kFwdRows * d;                // [warps][rows][bs]

  const int kv_row = blockIdx.y;
  const int seq = kv_row / p.kv_heads, kvh = kv_row % p.kv_heads;
  const int blk = ix.order[(size_t)kv_row * nb + blockIdx.x];
  const int n = ix.col_nnz[(size_t)kv_row * nb + blk];
  if (n == 0) return;
  const int lo = ix.col_offsets[(size_t)kv_row * (nb + 1) + blk];
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const size_t b = p.packed ? 0 : (size_t)seq;
  const int key0 = sp.bos + blk * bs;                       // token index of the block's first key
  const int keys = min(bs, sp.bos + sp.len - key0);
  if (keys <= 0) return;

  for (int i = threadIdx.x; i < bs * d; i += 256) {
    const int j = i / d, c = i % d;
    float kv = 0.f, vv = 0.f;
    if (j < keys) {
      const size_t src = ((b * p.tokens + key0 + j) * p.kv_heads + kvh) * (size_t)d + c;
      kv = Elem<T>::to_f(k[src]);
      vv = Elem<T>::to_f(v[src]);
    }
    Ks[j * kstride + c] = kv;
    Vs[j * d + c] = vv;
  }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float scale = rsqrtf((float)d) * kLog2e;
  const size_t list0 = (size_t)kv_row * ix.capacity + lo;
  float* qw = Qs + warp * kFwdRows * d;
  float* pw = Ps + warp * kFwdRows * bs;
  const int key_iters = (bs + 31) / 32;

  for (int e0 = warp * kFwdRows; e0 < n; e0 += kFwdWarps * kFwdRows) {
    int row[kFwdRows], head[kFwdRows], slot[kFwdRows];
#pragma unroll
    for (int r = 0; r < kFwdRows; ++r) {
      const bool live = e0 + r < n;
      PairEntry pe{-1, 0, 0, 0};
      if (live) pe = load_pair(ix, list0 + e0 + r);
      row[r] = pe.row; head[r] = pe.head; slot[r] = pe.slot;
      for (int c = lane; c < d; c += 32)
        qw[r * d + c] = live ? Elem<T>::to_f(q[((b * p.tokens + row[r]) * p.q_heads + head[r]) * (size_t)d + c]) : 0.f;
    }
    __syncwarp();
    float m[kFwdRows], l[kFwdRows];
#pragma unroll
    for (int r = 0; r < kFwdRows; ++r) m[r] = -INFINITY;
    // scores -> Ps (raw), row maxima
    for (int it = 0; it < key_iters; ++it) {
      const int j = it * 32 + lane;
      float acc[kFwdRows];
#pragma unroll
      for (int r = 0; r < kFwdRows; ++r) acc[r] = 0.f;
      if (j < bs) {
        const float* kr = Ks + j * kstride;
        for (int c = 0; c < d; ++c) {
          const float kv = kr[c];
#pragma unroll
          for (int r = 0; r < kFwdRows; ++r) acc[r] = fmaf(qw[r * d + c], kv, acc[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < kFwdRows; ++r) {
        float s = acc[r] * scale;
        const bool ok = j < keys && row[r] >= 0 && (!p.causal || key0 + j <= row[r]);
        s = ok ? s : -INFINITY;
        if (j < bs) pw[r * bs + j] = s;
        m[r] = fmaxf(m[r], s);
      }
    }
#pragma unroll
    for (int r = 0; r < kFwdRows; ++r) {
#pragma unroll
      for (int o = 16; o; o >>= 1) m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], o));
      l[r] = 0.f;
    }
    __syncwarp();
    for (int it = 0; it < key_iters; ++it) {
      const int j = it * 32 + lane;
      if (j < bs) {
#pragma unroll
        for (int r = 0; r < kFwdRows; ++r) {
          const float s = pw[r * bs + j];
          const float pe = (s == -INFINITY) ? 0.f : exp2f(s - m[r]);
          l[r] += pe;
          pw[r * bs + j] = Elem<T>::round_f(pe);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kFwdRows; ++r) {
#pragma unroll
      for (int o = 16; o; o >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], o);
    }
    __syncwarp();
    // p.v, lanes over the head dim
    for (int c = lane; c < d; c += 32) {
      float o[kFwdRows];
#pragma unroll
      for (int r = 0; r < kFwdRows; ++r) o[r] = 0.f;
      for (int j = 0; j < keys; ++j) {
        const float vv = Vs[j * d + c];
#pragma unroll
        for (int r = 0; r < kFwdRows; ++r) o[r] = fmaf(pw[r * bs + j], vv, o[r]);
      }
#pragma unroll
      for (int r = 0; r < kFwdRows; ++r) {
        if (row[r] < 0) continue;
        const size_t dst = part_row(p, b, head[r], row[r]) * (size_t)p.slots + slot[r];
        part_o[dst * d + c] = Elem<TP>::from_f(o[r] / l[r]);
      }
    }
    // lane r publishes row r's log2-sum-exp
#pragma unroll
    for (int r = 0; r < kFwdRows; ++r) {
      if (lane == r && row[r] >= 0) {
        const size_t dst = part_row(p, b, head[r], row[r]) * (size_t)p.slots + slot[r];
        part_lse[dst] = m[r] + log2f(l[r]);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// float32 attention, blocks of 64 to 128 keys, head_dim 64 or 128. One CTA per tile of 128 pairs
// of a work item: S is a 128 x 128 x D product and O a 128 x D x 128 one, each thread holding 8 x 8
// (8 x D/16) of them in registers and reading operands as 16-byte pieces, so that an FMA costs a
// sixteenth of a shared-memory load; P takes the place of Q and K between the two. The sums run in
// the order of the portable kernel (over the head dim, over the keys), in float32 FMAs. A tile's FMAs
// are 16 400 clocks of the SM's pipe at head_dim 64. At [1,4096,4,64] (0.135 ms, about 980 tiles on 296
// resident CTAs: 3.3 rounds, paid as four) the pipe is half busy, the issue slots two thirds, shared-memory
// wavefronts 42 % of their peak: two CTAs of eight warps do not fill the gaps of each other's loads and
// barriers. The operands come by asynchronous copies, and V is not waited for before P is there: whole calls of
// [1,8192,4,128] 825 -> 738 us, of [1,4096,4,64] 180 -> 175. Two queries an FMA instruction (with Q, K and P
// transposed in shared memory) took 676 and 192: such an instruction takes as long as two, and at head_dim 64
// the copies it needs twice of an operand cost more than the issue slots it frees. The portable kernel, with one
// CTA per column, a load per FMA and as many as 32 tiles in one CTA, took 1.3 ms.
// ---------------------------------------------------------------------------
constexpr int kF32Tile = 128;
template <int D> struct F32Cfg {
  static constexpr int kRow = D + 4;                        // floats per row of Q, K, V: rows of 16 lanes on different banks
  static constexpr int kPRow = kF32Tile + 4;
  static constexpr int kQk = 2 * kF32Tile * kRow;           // Q and K, then P
  static constexpr int kFloats = (kQk > kF32Tile * kPRow ? kQk : kF32Tile * kPRow) + kF32Tile * kRow;
  static constexpr int kSmem = kFloats * 4;
};

template <int D>
__global__ void __launch_bounds__(256, D == 64 ? 2 : 1)
fwd_f32_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
               moba_b200_index ix, const int32_t* __restrict__ cu, float* __restrict__ part_o,
               float* __restrict__ part_lse, moba_b200_problem p, int n_kv_rows) {
  using Cfg = F32Cfg<D>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int row_s[kF32Tile], dst_s[kF32Tile];          // query position; row of the partial buffers (-1: none)
  float* Qs = reinterpret_cast<float*>(smem_raw);           // [128][D + 4]
  float* Ks = Qs + kF32Tile * Cfg::kRow;
  float* Ps = Qs;                                           // [128][128 + 4]
  float* Vs = Qs + Cfg::kFloats - kF32Tile * Cfg::kRow;
  pdl_wait();
  const int kv_row = (int)(blockIdx.x % n_kv_rows), seq = kv_row / p.kv_heads, kvh = kv_row % p.kv_heads;
  WorkItem w;
  if (!load_work_item(w, ix, ix.col_nnz + (size_t)kv_row * p.num_blocks, kv_row, (int)(blockIdx.x / n_kv_rows))) return;
  const int n = min(kF32Tile, w.n - (int)blockIdx.y * kF32Tile);
  const SeqSpan sp = seq_span(cu, p.packed, seq, p.tokens);
  const size_t b = p.packed ? 0 : (size_t)seq;
  const int key0 = sp.bos + w.blk * p.block_size;
  const int keys = min(p.block_size, sp.bos + sp.len - key0);
  if (n <= 0 || keys <= 0) return;
  const size_t list0 = (size_t)kv_row * ix.capacity + ix.col_offsets[(size_t)kv_row * (p.num_blocks + 1) + w.blk] + w.first +
                       (size_t)blockIdx.y * kF32Tile;
  // Everything by asynchronous copies, Q and K first; nobody waits for V before P is there.
  constexpr int CPR = D / 4;                                // 16-byte pieces per row
  auto put = [&](float* to, const float* from, bool there) {
    if (there) __pipeline_memcpy_async(to, from, 16);
    else *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
  };
#pragma unroll 4
  for (int i = threadIdx.x; i < kF32Tile * CPR; i += 256) {
    const int j = i / CPR, c = (i % CPR) * 4;
    put(Ks + j * Cfg::kRow + c, k + ((b * p.tokens + key0 + j) * p.kv_heads + kvh) * (size_t)D + c, j < keys);
  }
#pragma unroll 4
  for (int i = threadIdx.x; i < kF32Tile * CPR; i += 256) {
    const int j = i / CPR, c = (i % CPR) * 4;
    const float* from = q;
    int row = -1, dst = -1;
    if (j < n) {
      const PairEntry e = load_pair(ix, list0 + j);
      row = e.row;
      dst = (int)(part_row(p, b, e.head, e.row) * (size_t)p.slots + e.slot);
      from = q + ((b * p.tokens + e.row) * p.q_heads + e.head) * (size_t)D + c;
    }
    if (c == 0) { row_s[j] = row; dst_s[j] = dst; }
    put(Qs + j * Cfg::kRow + c, from, j < n);
  }
  __pipeline_commit();
#pragma unroll 4
  for (int i = threadIdx.x; i < kF32Tile * CPR; i += 256) {
    const int j = i / CPR, c = (i % CPR) * 4;
    put(Vs + j * Cfg::kRow + c, v + ((b * p.tokens + key0 + j) * p.kv_heads + kvh) * (size_t)D + c, j < keys);
  }
  __pipeline_commit();
  __pipeline_wait_prior(1);
  __syncthreads();

  // thread (ty, tx): queries ty + 16 i, keys tx + 16 j
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float s[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) s[i][j] = 0.f;
#pragma unroll 1
  for (int c = 0; c < D; c += 4) {
    float4 a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(Qs + (ty + 16 * i) * Cfg::kRow + c);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 bk = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * Cfg::kRow + c);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s[i][j] = fmaf(a[i].x, bk.x, s[i][j]);
        s[i][j] = fmaf(a[i].y, bk.y, s[i][j]);
        s[i][j] = fmaf(a[i].z, bk.z, s[i][j]);
        s[i][j] = fmaf(a[i].w, bk.w, s[i][j]);
      }
    }
  }
  __syncthreads();                                          // Q and K have been read
  const float scale = rsqrtf((float)D) * kLog2e;
  float l[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = row_s[ty + 16 * i];
    const int last = p.causal ? min(keys - 1, row - key0) : keys - 1;       // a dead query (row -1) keeps nothing
    float m = -INFINITY;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s[i][j] = (row >= 0 && tx + 16 * j <= last) ? s[i][j] * scale : -INFINITY;
      m = fmaxf(m, s[i][j]);
    }
#pragma unroll
    for (int o = 8; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float pe = s[i][j] == -INFINITY ? 0.f : exp2f(s[i][j] - m);
      sum += pe;
      Ps[(ty + 16 * i) * Cfg::kPRow + tx + 16 * j] = pe;
    }
#pragma unroll
    for (int o = 8; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    l[i] = sum;
    if (tx == 0 && row >= 0) part_lse[dst_s[ty + 16 * i]] = m + log2f(sum);
  }
  __pipeline_wait_prior(0);
  __syncthreads();

  // thread (ty, tx): queries ty + 16 i, head-dim columns 4 tx + 64 h
  constexpr int H = D / 64;
  float4 o[8][H];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int h = 0; h < H; ++h) o[i][h] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int j = 0; j < kF32Tile; j += 4) {
    float4 pr[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) pr[i] = *reinterpret_cast<const float4*>(Ps + (ty + 16 * i) * Cfg::kPRow + j);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float4 vv = *reinterpret_cast<const float4*>(Vs + (j + u) * Cfg::kRow + h * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float pe = u == 0 ? pr[i].x : u == 1 ? pr[i].y : u == 2 ? pr[i].z : pr[i].w;
          o[i][h].x = fmaf(pe, vv.x, o[i][h].x);
          o[i][h].y = fmaf(pe, vv.y, o[i][h].y);
          o[i][h].z = fmaf(pe, vv.z, o[i][h].z);
          o[i][h].w = fmaf(pe, vv.w, o[i][h].w);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int dst = dst_s[ty + 16 * i];
    if (dst < 0) continue;
#pragma unroll
    for (int h = 0; h < H; ++h)
      *reinterpret_cast<float4*>(part_o + (size_t)dst * D + h * 64 + tx * 4) =
          make_float4(o[i][h].x / l[i], o[i][h].y / l[i], o[i][h].z / l[i], o[i][h].w / l[i]);
  }
}

template <int D>
static int launch_fwd_f32(const moba_b200_problem& p, const void* q, const void* k, const void* v, const moba_b200_index& ix,
                          const int32_t* cu, void* part_o, float* part_lse, cudaStream_t st) {
  static SmemLimit limit;
  if (int rc = raise_smem_limit(limit, (const void*)fwd_f32_kernel<D>, F32Cfg<D>::kSmem)) return rc;
  const int n_kv_rows = p.n_seq * p.kv_heads;
  const long long items = (long long)ix.items_per_row * n_kv_rows;
  // no item has more tiles than the longest possible column
  const long long longest = ((long long)(p.q_heads / p.kv_heads) * window_rows_of_seq(p) + kF32Tile - 1) / kF32Tile;
  const long long tiles = longest < ix.chunk_tiles ? longest : ix.chunk_tiles;
  if (items > 0x7fffffffLL || tiles > 65535) { set_error("float32 forward: %lld items of %lld tiles exceed the grid", items, tiles); return MOBA_B200_EUNSUPPORTED; }
  MOBA_CUDA_OK(launch_chained(fwd_f32_kernel<D>, dim3((unsigned)items, (unsigned)tiles), 256, F32Cfg<D>::kSmem, st, (const float*)q,
                              (const float*)k, (const float*)v, ix, cu, (float*)part_o, part_lse, p, n_kv_rows));
  return MOBA_B200_OK;
}
// Pairs in one slot of the partial buffers are numbered in 31 bits; the index must carry work items.
static bool fwd_f32_supported(const moba_b200_problem& p, const moba_b200_index& ix) {
  return p.dtype == MOBA_B200_F32 && p.path == MOBA_B200_PATH_AUTO && p.block_size >= 64 && p.block_size <= kF32Tile &&
         (p.head_dim == 64 || p.head_dim == 128) && ix.work_items != nullptr && ix.chunk_tiles > 0 && ix.chunk_tiles <= 65535 &&
         (long long)p.batch * p.q_heads * window_rows(p) * p.slots < 0x7fffffffLL;
}

static size_t fwd_portable_smem(const moba_b200_problem& p) {
  const size_t d = p.head_dim, bs = p.block_size;
  return sizeof(float) * (bs * (d + 1) + bs * d + kFwdWarps * kFwdRows * (d + bs));
}

int launch_fwd_portable(const moba_b200_problem& p, const void* q, const void* k, const void* v,
                        const moba_b200_index& ix, const int32_t* cu, void* part_o,
                        float* part_lse, cudaStream_t st) {
  if (fwd_f32_supported(p, ix)) {
    KernelTimer timer__("fwd_f32_kernel", st);
    return p.head_dim == 64 ? launch_fwd_f32<64>(p, q, k, v, ix, cu, part_o, part_lse, st)
                            : launch_fwd_f32<128>(p, q, k, v, ix, cu, part_o, part_lse, st);
  }
  KernelTimer timer__("fwd_portable_kernel", st);
  const size_t smem = fwd_portable_smem(p);
  if (smem > 220 * 1024) {
    set_error("forward: block_size %d with head_dim %d needs %zu bytes of shared memory",
              p.block_size, p.head_dim, smem);
    return MOBA_B200_EUNSUPPORTED;
  }
  if ((long long)p.n_seq * p.kv_heads > 65535) {
    set_error("portable forward: %d sequences x %d heads exceed 65535 grid rows", p.n_seq, p.kv_heads);
    return MOBA_B200_EUNSUPPORTED;
  }
  dim3 grid(p.num_blocks, p.n_seq * p.kv_heads);
#define MOBA_FWD(T, TP)                                                                        \
  do {                                                                                         \
    static SmemLimit limit;                                                                    \
    if (int rc = raise_smem_limit(limit, (const void*)fwd_portable_kernel<T, TP>, smem)) return rc; \
    MOBA_CUDA_OK(launch_chained(fwd_portable_kernel<T, TP>, grid, 256, smem, st, (const T*)q, (const T*)k, (const T*)v, \
                                ix, cu, (TP*)part_o, part_lse, p));                           \
  } while (0)
  if (p.dtype == MOBA_B200_F32) MOBA_FWD(float, float);
  else if (p.dtype == MOBA_B200_BF16) { if (p.part_f32) MOBA_FWD(__nv_bfloat16, float); else MOBA_FWD(__nv_bfloat16, __nv_bfloat16); }
  else { if (p.part_f32) MOBA_FWD(__half, float); else MOBA_FWD(__half, __half); }
#undef MOBA_FWD
  return MOBA_B200_OK;
}

// ---------------------------------------------------------------------------
// merge: one thread per 16-byte vector of a partial row. Streams part_o once.
//   LSE = m + log2 sum_i 2^(lse_i - m),  O = sum_i 2^(lse_i - LSE) O_i
// Reference: src/moba/kernels/moba_fwd.py:428-521.
// ---------------------------------------------------------------------------
template <typename TP, typename TO>
__global__ void __launch_bounds__(256)
merge_kernel(const TP* __restrict__ part_o, const float* __restrict__ part_lse,
             TO* __restrict__ out, float* __restrict__ lse_out, int tokens,
             int q_heads, int d, int slots, int win_begin, int win_rows) {
  pdl_trigger();
  pdl_wait();
  // grid (row groups of one (batch entry, head), heads, batch): no division anywhere (generic
  // 64-bit divisions cost this streaming kernel more instructions than its sums)
  constexpr int EPV = 16 / sizeof(TP);
  const unsigned tpr = (unsigned)(d / EPV);                  // threads per row, a power of two
  const unsigned gid = blockIdx.x * 256u + threadIdx.x;
  const unsigned row = gid / tpr;                            // row of the window
  const int c = (int)(gid % tpr);
  if (row >= (unsigned)win_rows) return;
  const size_t h = blockIdx.y, b = blockIdx.z, bh = b * q_heads + h;
  const size_t r = bh * win_rows + row;                      // head-major row (b, h, s) of the partials
  const float* ls = part_lse + r * slots;
  float mg = -INFINITY;
  for (int i = 0; i < slots; ++i) {
    const float li = ls[i];
    if (li > -INFINITY) mg = fmaxf(mg, li);
  }
  float acc[EPV];
#pragma unroll
  for (int e = 0; e < EPV; ++e) acc[e] = 0.f;
  float wsum = 0.f;
  const TP* po = part_o + r * slots * (size_t)d + c * EPV;
  // One 16-byte load per thread at a time leaves the memory system short of requests, so
  // the slots are taken eight at a time: all loads first, then the sums in slot order.
  constexpr int kAhead = 8;
  for (int i0 = 0; i0 < slots; i0 += kAhead) {
    float li[kAhead];
    uint4 raw[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) li[u] = (i0 + u < slots) ? ls[i0 + u] : -INFINITY;
#pragma unroll
    for (int u = 0; u < kAhead; ++u)                           // unwritten: never touch its data
      raw[u] = (li[u] > -INFINITY) ? __ldcs(reinterpret_cast<const uint4*>(po + (size_t)(i0 + u) * d)) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (!(li[u] > -INFINITY)) continue;
      const float w = exp2f(li[u] - mg);
      wsum += w;
      const TP* vals = reinterpret_cast<const TP*>(&raw[u]);
#pragma unroll
      for (int e = 0; e < EPV; ++e) acc[e] = fmaf(w, Elem<TP>::to_f(vals[e]), acc[e]);
    }
  }
  const float inv = 1.f / wsum;                              // wsum == 0 -> NaN, as the reference
  const size_t s = (size_t)win_begin + row;
  TO* dst = out + ((b * tokens + s) * q_heads + h) * (size_t)d + c * EPV;
  __align__(16) TO packed_out[EPV];
#pragma unroll
  for (int e = 0; e < EPV; ++e) packed_out[e] = Elem<TO>::from_f(wsum > 0.f ? acc[e] * inv : NAN);
  if (sizeof(TO) * EPV == 16) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(packed_out);
  else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(packed_out);
  if (lse_out != nullptr && c == 0) lse_out[bh * tokens + s] = (wsum > 0.f) ? mg + log2f(wsum) : -INFINITY;
}

int launch_merge(const moba_b200_problem& p, const void* part_o, const float* part_lse,
                 void* out, float* lse, cudaStream_t st) {
  KernelTimer timer__("merge_kernel", st);
  const bool pf32 = p.part_f32 || p.dtype == MOBA_B200_F32;
  const int epv = pf32 ? 4 : 8;
  const int tpr = p.head_dim / epv;
  const long long threads = (long long)window_rows(p) * tpr;
  if (tpr < 1 || (tpr & (tpr - 1)) || threads >= (1ll << 31) || p.q_heads > 65535 || p.batch > 65535) {
    set_error("merge: head_dim %d, %d heads or batch %d outside the kernel's grid", p.head_dim, p.q_heads, p.batch);
    return MOBA_B200_EUNSUPPORTED;
  }
  if (threads == 0 || p.batch == 0) return MOBA_B200_OK;
  const dim3 blocks((unsigned)((threads + 255) / 256), (unsigned)p.q_heads, (unsigned)p.batch);
#define MOBA_MERGE(TP, TO)                                                                      \
  MOBA_CUDA_OK(launch_chained(merge_kernel<TP, TO>, blocks, 256, 0, st, (const TP*)part_o, part_lse, (TO*)out, lse, \
                              p.tokens, p.q_heads, p.head_dim, p.slots, p.win_begin, window_rows(p)))
  if (p.dtype == MOBA_B200_F32) MOBA_MERGE(float, float);
  else if (p.dtype == MOBA_B200_BF16) { if (pf32) MOBA_MERGE(float, __nv_bfloat16); else MOBA_MERGE(__nv_bfloat16, __nv_bfloat16); }
  else { if (pf32) MOBA_MERGE(float, __half); else MOBA_MERGE(__half, __half); }
#undef MOBA_MERGE
  return MOBA_B200_OK;
}

}  // namespace moba
