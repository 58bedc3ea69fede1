// Paged causal grouped-query attention in true 32-bit, for head sizes up to 128 in steps of four (others, and keys with
// factors of their own, take the plain kernel in attention_generic.cu).
//
// One order of arithmetic whatever the launch: keys in tiles of 32 absolute positions with an online softmax (a score's
// products in ascending order, a tile's weights added eight threads apart), tiles in chunks of 128 positions, each summed
// from nothing, and the chunks merged in ascending order. A tile or chunk without a key that a row sees changes nothing.
// So a row is the same bits in both forms, however a prompt is cut and whatever runs beside it:
//   rows_form   single tokens, short portions, and few rows: a block per (row, key head), its warps take the row's chunks
//               side by side
//   tile_form   longer portions: a block per (64 query vectors: consecutive rows times the heads of a group, key head); a run
//               of rows of one request shares its key and value tiles, and one run is walked after the other
// In both a thread holds 4 keys of one to four query vectors while it scores and every eighth run of four value columns
// while it weighs; the next key tile lands while this one's values are weighed, the next value tile while keys are scored.
// What bounds it: shared memory (128 bytes a clock feed 4 x 4 products a thread at half the multiply-adds' rate) over a
// prompt, latency over single tokens. Measured on 32 heads of 64 over 8 key heads: 700 rows 172 us, 4 rows of 516 keys
// 17 us; a warp per (row, head) whose lanes read a key each, before: 2,390 and 283 us.
#include "attention_options.cuh"
#include "common.cuh"
#include <math.h>

namespace {

constexpr int TILE = 32, CHUNK = 128;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;  // 0: nothing is read and the 16 bytes become zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Args {
  const float* q;
  float* out;
  const float* kpool;
  const float* vpool;
  const int* positions;
  const int* seq_of_row;
  const int* tables;
  int* err;
  int q_stride, out_stride, n_blocks, bs, table_stride, n_rows, nh, nkv, d, dv;
  int least;  // the tile form leaves runs of fewer rows (within a tile) to the rows form, and that one the others (0: neither does)
  CucaAttnOptions opt;
};

// The rows of a tile, and how many of them make up the run of one request around row `row` of the step: what both forms go
// by to tell whose it is. Every lane of a warp takes part.
__host__ __device__ __forceinline__ int tile_rows_of(int gq) { return 64 / gq; }
__device__ __forceinline__ int run_around(const Args& a, int row, int lane) {
  const int rt = tile_rows_of(a.nh / a.nkv), row0 = row / rt * rt, n = min(rt, a.n_rows - row0), seq = a.seq_of_row[row];
  const unsigned lo = __ballot_sync(0xffffffffu, lane < n && a.seq_of_row[row0 + lane] == seq);
  const unsigned hi = __ballot_sync(0xffffffffu, lane + 32 < n && a.seq_of_row[row0 + lane + 32] == seq);
  const unsigned long long same = (unsigned long long)hi << 32 | lo;
  const int b = row - row0;
  const unsigned long long above = ~(same >> b), below = ~(same << (63 - b));  // the first zero bit ends the run
  return (above ? __ffsll((long long)above) - 1 : 64) + (below ? __clzll((long long)below) : 64) - 1;
}

// the first key position in a row's window
__device__ __forceinline__ int window_start(const CucaAttnOptions& o, int P) {
  return o.window > 0 && P - (o.window - 1) > 0 ? P - (o.window - 1) : 0;
}
// The tiles a run of rows walks: those of the kept first keys (from 0, up to kept_end), then from `first` to `last`.
struct Walk {
  int first, kept_end, last;
  __device__ int start() const { return kept_end > 0 ? 0 : first; }
  __device__ int next(int t0) const { return t0 + TILE == kept_end ? first : t0 + TILE; }
};
__device__ __forceinline__ Walk walk_of(const CucaAttnOptions& o, int lo_min, int last) {
  Walk w;
  w.first = lo_min / TILE * TILE;
  const int keep = o.window > 0 ? o.keep : 0;
  w.kept_end = min((keep + TILE - 1) / TILE * TILE, w.first);
  w.last = last;
  return w;
}

// The pool row of key position kp (-1: none), for positions that some row of the run sees.
__device__ __forceinline__ long long pool_row(const Args& a, const int* table, int kvh, int kp, int lo_min, int last) {
  const int keep = a.opt.window > 0 ? a.opt.keep : 0;
  if (!((kp >= lo_min || kp < keep) && kp <= last)) return -1;
  const int blk = table[kp / a.bs];
  if (blk < 0 || blk >= a.n_blocks) {
    if (a.err) atomicExch(a.err, CUCA_ERR_BLOCK_RANGE);
    return -1;
  }
  return ((long long)blk * a.nkv + kvh) * a.bs + kp % a.bs;
}
// 32 rows of a pool (n floats each, `rows` in shared memory) into [32][pitch], zeros behind n and where there is no row.
template <int N, int PITCH, int THREADS>
__device__ __forceinline__ void load_tile(float* dst, const float* pool, const long long* rows, int n, int tid) {
#pragma unroll 4
  for (int e = tid; e < TILE * (N / 4); e += THREADS) {
    const int r = e / (N / 4), c = e % (N / 4) * 4;
    const long long row = rows[r];
    const bool ok = row >= 0 && c < n;
    copy16(dst + r * PITCH + c, pool + (ok ? row * n + c : 0), ok);
  }
}

// The scores of TM query vectors (rows of `qs`, pitch D + 4) and the keys tx, tx + 8, tx + 16, tx + 24 of a tile.
template <int D, int TM>
__device__ __forceinline__ void score(float (&s)[TM][4], const float* qs, const float* ks, int tx) {
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
  for (int c = 0; c < D; c += 4) {
    float4 q[TM], k[4];
#pragma unroll
    for (int i = 0; i < TM; ++i) q[i] = *reinterpret_cast<const float4*>(qs + i * (D + 4) + c);
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(ks + (tx + 8 * j) * (D + 4) + c);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = fmaf(q[i].x, k[j].x, s[i][j]);
        s[i][j] = fmaf(q[i].y, k[j].y, s[i][j]);
        s[i][j] = fmaf(q[i].z, k[j].z, s[i][j]);
        s[i][j] = fmaf(q[i].w, k[j].w, s[i][j]);
      }
  }
}

// One query vector's part of a chunk: maximum, denominator, weighed values (columns 4 tx + 32 c .. + 3).
template <int DV>
struct Part {
  float m, l, acc[DV / 8];
  __device__ void clear() {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) acc[i] = 0.f;
  }
  // this <- this and a later chunk. lost2: in that chunk a tile with scores that are no numbers came by before any that is
  // one. Such a tile counts for nothing at the start of a row, and from a row's first finite score on it makes the result no
  // number; where a row starts is known here only.
  __device__ void merge(float m2, float l2, const float (&acc2)[DV / 8], bool lost2) {
    if (lost2 && m != -INFINITY) {
      l = NAN;
#pragma unroll
      for (int i = 0; i < DV / 8; ++i) acc[i] = NAN;
    }
    if (m2 == -INFINITY) return;
    const float mn = fmaxf(m, m2), c1 = expf(m - mn), c2 = expf(m2 - mn);
    l = fmaf(l2, c2, l * c1);
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) acc[i] = fmaf(acc2[i], c2, acc[i] * c1);
    m = mn;
  }
};

// A tile's scores into weights, for one query vector at position P: raw products in, weights out; the chunk's maximum,
// denominator and values move with the maximum. `there`: which of the tile's 32 keys exist. Keys that the row does not see
// get a negative zero: unlike a weight that came out as zero, it keeps their values out of the sums whatever they are.
// FULL: the row sees all of them. Returns whether this thread has a score that is no number while no thread has one that is.
template <int DV, bool FULL>
__device__ __forceinline__ bool weigh(float (&s)[4], Part<DV>& p, const CucaAttnOptions& o, float slope, int t0, int tx, int P,
                                      int lo, bool row_live, unsigned there) {
  const int keep = o.window > 0 ? o.keep : 0;
  bool valid[4];
  float top = -INFINITY;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int kp = t0 + tx + 8 * j;
    valid[j] = FULL || (row_live && (there >> (tx + 8 * j) & 1u) && (kp >= lo || kp < keep) && kp <= P);
    float v = s[j] * o.scale;
    if (o.softcap > 0.f) v = o.softcap * tanhf(v / o.softcap);
    if (o.slopes) v -= slope * (float)(P - kp);
    s[j] = valid[j] ? v : -INFINITY;
    top = fmaxf(top, s[j]);  // (of those that are numbers)
  }
#pragma unroll
  for (int x = 4; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
  const float mn = fmaxf(p.m, top);
  const bool any = mn != -INFINITY;
  bool nan = false;
  if (!any)
#pragma unroll
    for (int j = 0; j < 4; ++j) nan |= s[j] != s[j];
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = any && valid[j] ? expf(s[j] - mn) : -0.f;
  float sum = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
  for (int x = 4; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
  if (!any) return nan;
  const float corr = expf(p.m - mn);
  p.l = fmaf(p.l, corr, sum);
#pragma unroll
  for (int i = 0; i < DV / 8; ++i) p.acc[i] *= corr;
  p.m = mn;
  return false;
}

// acc += weights (TM rows of `ps`, pitch TILE + 4) times the tile's values, keys in ascending order.
template <int DV, int TM, bool FULL>
__device__ __forceinline__ void add_values(Part<DV> (&p)[TM], const float* ps, const float* vs, int tx) {
#pragma unroll 2
  for (int j0 = 0; j0 < TILE; j0 += 4) {
    float4 w[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) w[i] = *reinterpret_cast<const float4*>(ps + i * (TILE + 4) + j0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 v[DV / 32];
#pragma unroll
      for (int c = 0; c < DV / 32; ++c) v[c] = *reinterpret_cast<const float4*>(vs + (j0 + j) * DV + 32 * c + 4 * tx);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float wj = j == 0 ? w[i].x : j == 1 ? w[i].y : j == 2 ? w[i].z : w[i].w;
        if (FULL || __float_as_uint(wj) != 0x80000000u) {  // (a negative zero: see `weigh`)
#pragma unroll
          for (int c = 0; c < DV / 32; ++c) {
            p[i].acc[4 * c] = fmaf(wj, v[c].x, p[i].acc[4 * c]);
            p[i].acc[4 * c + 1] = fmaf(wj, v[c].y, p[i].acc[4 * c + 1]);
            p[i].acc[4 * c + 2] = fmaf(wj, v[c].z, p[i].acc[4 * c + 2]);
            p[i].acc[4 * c + 3] = fmaf(wj, v[c].w, p[i].acc[4 * c + 3]);
          }
        }
      }
    }
  }
}

// A thread's TM query vectors through a tile: weights into its rows of `ps`. Returns which of the vectors (bit i) have
// scores and none that is a number. Every lane of a warp takes part.
template <int DV, int TM, bool FULL>
__device__ __forceinline__ unsigned weigh_all(float (&s)[TM][4], Part<DV> (&p)[TM], const CucaAttnOptions& o,
                                              const float (&slope)[TM], int t0, int tx, const int (&P)[TM], const int (&lo)[TM],
                                              const bool (&live)[TM], unsigned there, float* ps) {
  unsigned nans = 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    if (weigh<DV, FULL>(s[i], p[i], o, slope[i], t0, tx, P[i], lo[i], live[i], there)) nans |= 1u << i;
#pragma unroll
    for (int j = 0; j < 4; ++j) ps[i * (TILE + 4) + tx + 8 * j] = s[i][j];
  }
  if (__any_sync(0xffffffffu, nans != 0))  // (a vector's eight threads as one)
#pragma unroll
    for (int x = 4; x > 0; x >>= 1) nans |= __shfl_xor_sync(0xffffffffu, nans, x);
  return nans;
}

// Whether every vector of the warp that counts sees all keys of a tile (the others' results go nowhere).
template <int TM>
__device__ __forceinline__ bool all_seen(int t0, const int (&P)[TM], const int (&lo)[TM], const bool (&live)[TM], unsigned there) {
  bool full = there == 0xffffffffu;
#pragma unroll
  for (int i = 0; i < TM; ++i) full &= !live[i] || (t0 >= lo[i] && t0 + TILE - 1 <= P[i]);
  return __all_sync(0xffffffffu, full);
}

// N query vectors into [N][D + 4], zeros behind a.d and for those that `at` has no address for.
template <int D, int N, int THREADS, typename At>
__device__ __forceinline__ void load_queries(const Args& a, float* qs, int tid, At at) {
  if (a.q_stride % 4 == 0 && ((uintptr_t)a.q & 15) == 0) {
#pragma unroll 4
    for (int e = tid; e < N * D / 4; e += THREADS) {
      const int v = e / (D / 4), c = e % (D / 4) * 4;
      const float* src = at(v);
      *reinterpret_cast<float4*>(qs + v * (D + 4) + c) =
          src && c < a.d ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    for (int e = tid; e < N * D; e += THREADS) {
      const int v = e / D, c = e % D;
      const float* src = at(v);
      qs[v * (D + 4) + c] = src && c < a.d ? src[c] : 0.f;
    }
  }
}

// A query vector's result: sink, division, gate, store of the thread's columns.
template <int DV>
__device__ __forceinline__ void finish(const Args& a, Part<DV>& p, int row, int head, int tx) {
  if (a.opt.sink) {  // one more term in the denominator: a key of score 0 (or of the head's stored score) that has no value
    const float s0 = a.opt.sink_val ? a.opt.sink_val[head] : 0.f;
    const float mn = fmaxf(p.m, s0), corr = expf(p.m - mn);
    p.l = fmaf(p.l, corr, expf(s0 - mn));
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) p.acc[i] *= corr;
  }
  const float inv = p.l > 0.f ? 1.f / p.l : 0.f;
  float* o = a.out + (size_t)row * a.out_stride + (size_t)head * a.dv;
  const float* gate = a.opt.gate ? (const float*)a.opt.gate + (size_t)row * a.opt.gate_stride + (size_t)head * a.dv : nullptr;
#pragma unroll
  for (int c = 0; c < DV / 32; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int dim = 32 * c + 4 * tx + j;
      if (dim >= a.dv) continue;
      float r = p.acc[4 * c + j] * inv;
      if (gate) r /= 1.f + expf(-gate[dim]);
      o[dim] = r;
    }
}

template <int D>
struct TileForm {
  static constexpr int VECS = 64, TM = 4, THREADS = 128;
  static constexpr int SMEM = (VECS * (D + 4) + TILE * (D + 4) + TILE * D + VECS * (TILE + 4)) * 4;
};

template <int D>
__global__ void __launch_bounds__(128)
tile_form_kernel(const Args a) {
  using F = TileForm<D>;
  constexpr int VECS = F::VECS, TM = F::TM, THREADS = F::THREADS;
  extern __shared__ __align__(16) float sm[];
  __shared__ long long rows[2][TILE];
  __shared__ int s_pos[VECS], s_seq[VECS];
  float* qs = sm;                          // [VECS][D + 4]
  float* ks = qs + VECS * (D + 4);         // [TILE][D + 4]
  float* vs = ks + TILE * (D + 4);         // [TILE][D]
  float* ps = vs + TILE * D;               // [VECS][TILE + 4]
  pdl_trigger();
  pdl_wait();
  const int gq = a.nh / a.nkv, kvh = blockIdx.y, tid = threadIdx.x;
  const int rt = tile_rows_of(gq);                            // rows of a block
  const int row0 = (gridDim.x - 1 - blockIdx.x) * rt;         // later rows see more keys: first
  const int nr = min(rt, a.n_rows - row0);
  for (int r = tid; r < nr; r += THREADS) { s_pos[r] = a.positions[row0 + r]; s_seq[r] = a.seq_of_row[row0 + r]; }
  load_queries<D, VECS, THREADS>(a, qs, tid, [&](int v) {
    const int r = v / gq;
    return r < nr ? a.q + (size_t)(row0 + r) * a.q_stride + (size_t)(kvh * gq + v % gq) * a.d : nullptr;
  });
  __syncthreads();
  const int tx = tid % 8, v0 = tid / 8 * TM;  // this thread's query vectors v0 .. v0 + TM - 1
  float slope[TM];
#pragma unroll
  for (int i = 0; i < TM; ++i) slope[i] = a.opt.slopes && (v0 + i) / gq < nr ? a.opt.slopes[kvh * gq + (v0 + i) % gq] : 0.f;
  for (int b = 0; b < nr;) {  // runs of rows of one request
    const int seq = s_seq[b];
    int e = b + 1, last = s_pos[b];
    int lo_min = window_start(a.opt, last);
    for (; e < nr && s_seq[e] == seq; ++e) {
      last = max(last, s_pos[e]);
      lo_min = min(lo_min, window_start(a.opt, s_pos[e]));
    }
    const int rb = b, re = e;
    b = e;
    if (seq < 0 || re - rb < a.least) continue;
    const int* table = a.tables + (size_t)seq * a.table_stride;
    const Walk walk = walk_of(a.opt, lo_min, last);
    Part<D> total[TM], part[TM];
    int P[TM], lo[TM];
    bool live[TM];
    unsigned lost = 0;  // which vectors' parts of this chunk started with scores that are no numbers
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      total[i].clear();
      part[i].clear();
      const int r = (v0 + i) / gq;
      live[i] = r >= rb && r < re;
      P[i] = live[i] ? s_pos[r] : 0;
      lo[i] = window_start(a.opt, P[i]);
    }
    // pool rows of the first tile, its keys and values
    int t0 = walk.start(), buf = 0;
    if (tid < TILE) rows[0][tid] = pool_row(a, table, kvh, t0 + tid, lo_min, last);
    __syncthreads();
    load_tile<D, D + 4, THREADS>(ks, a.kpool, rows[0], a.d, tid);
    copy_commit();
    load_tile<D, D, THREADS>(vs, a.vpool, rows[0], a.dv, tid);
    copy_commit();
    for (; t0 <= last; buf ^= 1) {
      const int t1 = walk.next(t0);
      const bool more = t1 <= last;
      if (tid < TILE && more) rows[buf ^ 1][tid] = pool_row(a, table, kvh, t1 + tid, lo_min, last);
      const unsigned there = __ballot_sync(0xffffffffu, rows[buf][tid & 31] >= 0);
      copy_wait<1>();
      __syncthreads();  // the keys have landed
      float s[TM][4];
      score<D, TM>(s, qs + v0 * (D + 4), ks, tx);
      __syncthreads();  // the keys are read
      if (more) load_tile<D, D + 4, THREADS>(ks, a.kpool, rows[buf ^ 1], a.d, tid);
      copy_commit();
      const bool full = all_seen<TM>(t0, P, lo, live, there);
      float* mine = ps + v0 * (TILE + 4);
      lost |= full ? weigh_all<D, TM, true>(s, part, a.opt, slope, t0, tx, P, lo, live, there, mine)
                   : weigh_all<D, TM, false>(s, part, a.opt, slope, t0, tx, P, lo, live, there, mine);
      copy_wait<1>();
      __syncthreads();  // the values have landed, the weights are written
      if (full) add_values<D, TM, true>(part, mine, vs, tx);
      else add_values<D, TM, false>(part, mine, vs, tx);
      __syncthreads();  // the values are read
      if (more) load_tile<D, D, THREADS>(vs, a.vpool, rows[buf ^ 1], a.dv, tid);
      copy_commit();
      if (!more || t1 / CHUNK != t0 / CHUNK) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          total[i].merge(part[i].m, part[i].l, part[i].acc, lost >> i & 1u);
          part[i].clear();
        }
        lost = 0;
      }
      t0 = t1;
    }
    copy_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
      if (live[i]) finish<D>(a, total[i], row0 + (v0 + i) / gq, kvh * gq + (v0 + i) % gq, tx);
  }
}

template <int D, int TM, int WARPS_>
struct RowsForm {
  static constexpr int WARPS = WARPS_, VECS = 4 * TM;
  static constexpr int WARP_FLOATS = TILE * (D + 4) + TILE * D + VECS * (TILE + 4);
  static constexpr int PART = D + 3;  // a chunk's result of a query vector: values, maximum, denominator, lost or not
  static constexpr int SMEM = (VECS * (D + 4) + WARPS * WARP_FLOATS + WARPS * VECS * PART) * 4;
};

template <int D, int TM, int WARPS_>
__global__ void __launch_bounds__(32 * WARPS_)
rows_form_kernel(const Args a) {
  using F = RowsForm<D, TM, WARPS_>;
  constexpr int WARPS = F::WARPS, VECS = F::VECS, PART = F::PART;
  extern __shared__ __align__(16) float sm[];
  __shared__ long long rows[WARPS][2][TILE];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tx = lane % 8, v0 = lane / 8 * TM;
  float* qs = sm;  // [VECS][D + 4]
  float* ks = qs + VECS * (D + 4) + warp * F::WARP_FLOATS;
  float* vs = ks + TILE * (D + 4);
  float* ps = vs + TILE * D;
  float* parts = qs + VECS * (D + 4) + WARPS * F::WARP_FLOATS;  // [WARPS][VECS][PART]
  pdl_trigger();
  pdl_wait();
  const int gq = a.nh / a.nkv, kvh = blockIdx.x, row = blockIdx.y;
  const int seq = a.seq_of_row[row];
  if (seq < 0 || (a.least && run_around(a, row, lane) >= a.least)) return;
  const int P0 = a.positions[row], lo0 = window_start(a.opt, P0);
  load_queries<D, VECS, 32 * WARPS>(a, qs, threadIdx.x, [&](int v) {
    return v < gq ? a.q + (size_t)row * a.q_stride + (size_t)(kvh * gq + v) * a.d : nullptr;
  });
  __syncthreads();
  const int* table = a.tables + (size_t)seq * a.table_stride;
  const Walk walk = walk_of(a.opt, lo0, P0);
  float slope[TM];
#pragma unroll
  for (int i = 0; i < TM; ++i) slope[i] = a.opt.slopes && v0 + i < gq ? a.opt.slopes[kvh * gq + v0 + i] : 0.f;
  int P[TM], lo[TM];
  bool live[TM];
#pragma unroll
  for (int i = 0; i < TM; ++i) { P[i] = P0; lo[i] = lo0; live[i] = v0 + i < gq; }
  Part<D> total[TM];  // (of warp 0)
#pragma unroll
  for (int i = 0; i < TM; ++i) total[i].clear();
  // the chunks that have tiles to walk: of the kept first keys, then of the window; n of them, chunk_of(c) ascending
  const int kept = (walk.kept_end + CHUNK - 1) / CHUNK, first = walk.first / CHUNK;
  const int from = max(first, kept);  // (a chunk that holds both kinds counts as one of the kept ones)
  const int n = kept + max(0, P0 / CHUNK - from + 1);
  for (int c0 = 0; c0 < n; c0 += WARPS) {
    const int c = c0 + warp;
    Part<D> part[TM];
    unsigned lost = 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) part[i].clear();
    if (c < n) {
      const int chunk = c < kept ? c : from + c - kept;
      const int end = min(P0 + 1, (chunk + 1) * CHUNK);
      // the first tile of the chunk that the walk comes by
      int t0 = chunk * CHUNK;
      if (t0 >= walk.kept_end && t0 < walk.first) t0 = walk.first;
      int buf = 0;
      rows[warp][0][lane] = pool_row(a, table, kvh, t0 + lane, lo0, P0);
      __syncwarp();
      load_tile<D, D + 4, 32>(ks, a.kpool, rows[warp][0], a.d, lane);
      copy_commit();
      load_tile<D, D, 32>(vs, a.vpool, rows[warp][0], a.dv, lane);
      copy_commit();
      for (; t0 < end; buf ^= 1) {
        const int t1 = walk.next(t0);
        const bool more = t1 < end;
        const unsigned there = __ballot_sync(0xffffffffu, rows[warp][buf][lane] >= 0);
        if (more) rows[warp][buf ^ 1][lane] = pool_row(a, table, kvh, t1 + lane, lo0, P0);
        copy_wait<1>();
        __syncwarp();  // the keys have landed
        float s[TM][4];
        score<D, TM>(s, qs + v0 * (D + 4), ks, tx);
        __syncwarp();  // the keys are read
        if (more) load_tile<D, D + 4, 32>(ks, a.kpool, rows[warp][buf ^ 1], a.d, lane);
        copy_commit();
        const bool full = all_seen<TM>(t0, P, lo, live, there);
        float* mine = ps + v0 * (TILE + 4);
        lost |= full ? weigh_all<D, TM, true>(s, part, a.opt, slope, t0, tx, P, lo, live, there, mine)
                     : weigh_all<D, TM, false>(s, part, a.opt, slope, t0, tx, P, lo, live, there, mine);
        copy_wait<1>();
        __syncwarp();  // the values have landed, the weights are written
        if (full) add_values<D, TM, true>(part, mine, vs, tx);
        else add_values<D, TM, false>(part, mine, vs, tx);
        __syncwarp();  // the values are read
        if (more) load_tile<D, D, 32>(vs, a.vpool, rows[warp][buf ^ 1], a.dv, lane);
        copy_commit();
        t0 = t1;
      }
      copy_wait<0>();
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      float* to = parts + (warp * VECS + v0 + i) * PART;
#pragma unroll
      for (int e = 0; e < D / 8; ++e) to[tx * (D / 8) + e] = part[i].acc[e];
      if (tx == 0) { to[D] = part[i].m; to[D + 1] = part[i].l; to[D + 2] = lost >> i & 1u ? 1.f : 0.f; }
    }
    __syncthreads();
    if (warp == 0) {
      for (int w = 0; w < min(WARPS, n - c0); ++w)
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float* of = parts + (w * VECS + v0 + i) * PART;
          float acc[D / 8];
#pragma unroll
          for (int e = 0; e < D / 8; ++e) acc[e] = of[tx * (D / 8) + e];
          total[i].merge(of[D], of[D + 1], acc, of[D + 2] != 0.f);
        }
    }
    __syncthreads();
  }
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
      if (v0 + i < gq) finish<D>(a, total[i], row, kvh * gq + v0 + i, tx);
  }
}

template <typename F>
int launch(F* kernel, dim3 grid, int threads, int smem, cudaStream_t stream, const Args& a) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  CUCA_REQUIRE(e == cudaSuccess, "attention: %d bytes of shared memory were refused: %s", smem, cudaGetErrorString(e));
  cuca_launch(kernel, grid, dim3(threads), smem, stream, true, a);
  CUCA_CHECK_LAUNCH("attention_f32");
  return 0;
}

// How many chunks of keys a row may have to walk, at most.
int chunks_of(const Args& a) {
  const int keys = a.opt.keys > 0 ? a.opt.keys : a.table_stride * a.bs, w = a.opt.window;
  const int chunks = (keys + CHUNK - 1) / CHUNK;
  return w > 0 ? min(chunks, (a.opt.keep + CHUNK - 1) / CHUNK + (w + CHUNK - 1) / CHUNK + 1) : chunks;
}

template <int D, int TM>
int run_rows(const Args& a, cudaStream_t stream) {
  // A warp per chunk: a block of eight warps fills an SM's shared memory, and over short rows seven of them idle (single
  // tokens of up to 32 keys, 32 heads of 64 over 8: 65 rows 22 us with eight warps, 100 rows 9 with one).
  const int chunks = chunks_of(a);
  const dim3 grid(a.nkv, a.n_rows);
#define ROWS(W) return launch(rows_form_kernel<D, TM, W>, grid, 32 * W, RowsForm<D, TM, W>::SMEM, stream, a)
  if (chunks <= 1) ROWS(1);
  if (chunks <= 2) ROWS(2);
  if (D == 128 || chunks <= 4) ROWS(4);
  if constexpr (D == 64) ROWS(8);
#undef ROWS
  return 0;
}

template <int D>
int run(Args a, cudaStream_t stream) {
  const int gq = a.nh / a.nkv, rt = tile_rows_of(gq);
  // Runs of fewer rows than this go row by row. A tile's runs are walked one after the other, so a run of one row takes the
  // time of a whole tile (65 rows of 300 keys, 12 heads of 64: 3,524 us in tiles, 54 row by row). Both forms cost about the
  // same at some 32 query vectors a run (40 requests with 100 keys before, 32 heads of 64 over 8, us row by row, in tiles:
  // 8 rows 48, 75; 16 rows 91, 44; 12 heads of 64, 16 requests: 20 rows 69, 111; 32 rows 184, 78).
  const int least = max(4, 32 / gq + 1);
  a.least = 0;
  bool tiles = true, rows = false;
  if (gq <= 16) {
    // Few rows: blocks of 64 query vectors would leave most SMs idle. Where nothing is known of the runs, few rows of one
    // chunk of keys have little to share, and of others every row finds out for itself in both launches.
    const bool known = a.opt.run_max > 0;
    rows = a.n_rows <= 64 || !known || a.opt.run_min < least;
    tiles = a.n_rows > 64 && (known ? a.opt.run_max >= least : a.n_rows > 256 || chunks_of(a) > 1);
    if (rows && tiles) a.least = least;
  }
  if (tiles) {
    const int rc = launch(tile_form_kernel<D>, dim3((a.n_rows + rt - 1) / rt, a.nkv), TileForm<D>::THREADS, TileForm<D>::SMEM,
                          stream, a);
    if (rc) return rc;
  }
  if (!rows) return 0;
  return gq <= 4 ? run_rows<D, 1>(a, stream) : gq <= 8 ? run_rows<D, 2>(a, stream) : run_rows<D, 4>(a, stream);
}

}  // namespace

// Whether `cuca_attention_f32` takes these sizes and pools; a launch's rows have no say, so that all of a model's steps
// take one path.
bool cuca_attention_f32_takes(const void* kpool, const void* vpool, int nh, int nkv, int d, int dv, const CucaAttnOptions* opt) {
  return d <= 128 && d % 4 == 0 && dv % 4 == 0 && dv <= (d <= 64 ? 64 : 128) && nh / nkv <= 64 && nkv <= 65535 &&
         !opt->key_scale && (((uintptr_t)kpool | (uintptr_t)vpool) & 15) == 0;
}

int cuca_attention_f32(const float* q, int q_stride, float* out, int out_stride, const float* kpool, const float* vpool,
                       int n_blocks, int bs, const int* positions, const int* seq_of_row, const int* tables, int table_stride,
                       int n_rows, int nh, int nkv, int d, int dv, const CucaAttnOptions* opt, int* err, cudaStream_t stream) {
  const Args a{q, out, kpool, vpool, positions, seq_of_row, tables, err, q_stride, out_stride, n_blocks, bs, table_stride,
               n_rows, nh, nkv, d, dv, 0, *opt};
  return d <= 64 ? run<64>(a, stream) : run<128>(a, stream);
}
