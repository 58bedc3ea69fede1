// Mixers whose per-request state is a matrix per head, S [key channels, value columns], carried in 32-bit:
//   delta_scan      the delta rule with a decay per key channel:
//                     S <- g * S (rows);  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//   mlstm_scan      a matrix memory with exponential gates and a running maximum m (0 at the start):
//                     m' = max(f + m, i);  S <- e^(f + m - m') S + e^(i - m') k v^T;  n likewise from k alone;
//                     o = S^T q / (max(|n . q|, e^(-m')) + 1e-6)
//   forget_scan     linear attention whose forget gate f (per key channel) is also one minus its write strength:
//                     S <- f * S (rows) + (1 - f) v^T;  o = S^T q
//   retention_scan  linear attention with one fixed decay per head and no denominator:
//                     S <- decay S + k v^T;  o = S^T q
//   lightning_scan  the same recurrence on q = silu(.), k = silu(.), v = silu(.); lightning_step: for single tokens
//   head_norm_gate  out = o / rms(o) per head, times a weight (or none), times sigmoid(gate) or silu(gate)
// What does not depend on the state (unit vectors, decays, gates) is computed for all rows at once by a preparing
// kernel, in place. A scan block then takes one (head, request, run of value columns) and walks the request's rows of
// the step in order from the state its slot holds, leaving the new state there. A value column's state rows live in
// the registers of NS neighbouring threads (see Split); a token's vectors are copied to shared memory a few tokens
// ahead of their use. The arithmetic of a token depends neither on where the sequence was cut into steps or chunks
// nor on what else is in the launch (but for the delta rule four tokens at a time, which depends on the cuts, see there).
#include "common.cuh"
#include "state_rows.cuh"
#include <math.h>

namespace {

constexpr int MAX_DIM = 1024;  // key channels

__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + expf(-v)); }
__device__ __forceinline__ float softplusf_(float v) { return v > 20.f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float log_sigmoidf_(float v) { return v < 0.f ? v - log1pf(expf(v)) : -log1pf(expf(-v)); }

// Per row, in place: q and k heads (G heads of d at columns 0 and G d of qkv) become unit vectors, q times d^(-1/2);
// the decay pre-activations a_raw (rows of stride ld_a, H d values) become g = exp(-exp(A_log[h]) softplus(a + dt_bias)); the gate
// pre-activation of head h (column b_col + h of b_raw) becomes sigmoid. One block per row.
__global__ void __launch_bounds__(256)
delta_prepare_kernel(float* __restrict__ qkv, int ld, float* __restrict__ a_raw, int ld_a, const float* __restrict__ dt_bias,
                     const float* __restrict__ a_log, float* __restrict__ b_raw, int ld_b, int b_col,
                     const int* __restrict__ seq_of_row, int H, int G, int d) {
  pdl_trigger();
  pdl_wait();
  const size_t row = blockIdx.x;
  if (seq_of_row[row] < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float qscale = rsqrtf((float)d);
  for (int v = warp; v < 2 * G; v += 8) {  // q heads, then k heads
    float* x = qkv + row * ld + (size_t)v * d;
    float ss = 0.f;
    for (int i = lane; i < d; i += 32) ss = fmaf(x[i], x[i], ss);
    const float inv = (v < G ? qscale : 1.f) / sqrtf(warp_sum(ss) + 1e-6f);
    for (int i = lane; i < d; i += 32) x[i] *= inv;
  }
  float* ar = a_raw + row * ld_a;
  for (int i = threadIdx.x; i < H * d; i += 256)
    ar[i] = expf(-expf(a_log[i / d]) * softplusf_(ar[i] + dt_bias[i]));
  if (threadIdx.x < H) {
    float* b = b_raw + row * ld_b + b_col + threadIdx.x;
    *b = sigmoidf_(*b);
  }
}

// qkv: 32-bit rows of stride ld, prepared: unit q heads at column 0 (G heads of d), unit k heads at column G d, v
// heads at column 2 G d (H heads of dv). decay: rows of stride ld_g, H d decays; beta: rows of stride ld_b, head h at column
// b_col + h. state: [slots, H, dv, d]. out: [rows, H dv]. Two buffers of TC tokens: the next tokens' vectors are
// copied (cp.async) while these are worked through.
// What bounds it for one prompt: the chain of a token (state times decay, dot with k, four shuffles and one more to hand the
// sum round, correction), about 500 clocks at 128 channels; the outputs' dot products belong to the token before and run in
// the shadow of the shuffles.
// Requests that bring `below` tokens or more are the chunked form's.
template <typename C>
__global__ void __launch_bounds__(128)
delta_scan_kernel(const float* __restrict__ qkv, int ld, const float* __restrict__ decay, int ld_g,
                  const float* __restrict__ beta, int ld_b, int b_col, float* __restrict__ state,
                  float* __restrict__ out, const int* __restrict__ req_row0,
                  const int* __restrict__ req_count, const int* __restrict__ slots, int H, int G,
                  int d, int dv, int wide, int below) {
  constexpr int NS = C::NS, NC = C::NC, DP = C::DP, PB = C::PB, TC = C::TC, PAIRS = C::PAIRS;
  constexpr int PER = 3 * DP + ((PB + 1 + 3) & ~3);  // a token: q, k, g, the block's values, beta
  extern __shared__ __align__(16) float sm[];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq], n = req_count[rq], r0 = req_row0[rq];
  if (slot < 0 || n <= 0 || n >= below) return;
  const int kvh = h / (H / G);
  const int col_local = threadIdx.x / NS, s = threadIdx.x % NS;
  const int col0 = blockIdx.z * PB, at = col_local * NC;
  const int cols = min(NC, dv - col0 - at);               // columns of this thread that exist (none: 0 or less)
  float* st = state + (((size_t)slot * H + h) * dv + (cols > 0 ? col0 + at : 0)) * d;
  f32x2 S[NC][PAIRS];
  load_rows<C>(S, st, s, d, cols, wide);
  // what no copy writes: channels from d on (q = k = 0, g = 1) and the values of columns from dv on
  {
    const int spare = DP - d, there = min(PB, dv - col0), fill = 3 * spare + PB - there;
    for (int e = threadIdx.x; e < (n < TC ? n : 2 * TC) * fill; e += 128) {
      const int t = e / fill, w = e % fill;
      float* tok = sm + t * PER;
      if (w < 3 * spare) tok[(w / spare) * DP + d + w % spare] = w / spare == 2 ? 1.f : 0.f;
      else tok[3 * DP + there + (w - 3 * spare)] = 0.f;
    }
  }
  __syncthreads();
  auto stage = [&](int t0, int buf) {
    const int nt = n - t0 < TC ? n - t0 : TC;
    float* base = sm + buf * TC * PER;
    auto copy = [&](int t, int which, int r) {
      const size_t row = (size_t)(r0 + t0 + t);
      const float* src = which == 2 ? decay + row * ld_g + (size_t)h * d + r : qkv + row * ld + (size_t)(which * G + kvh) * d + r;
      if (r < d) cp_async_f(base + t * PER + which * DP + r, src, wide);
    };
    if (wide)
      for (int e = threadIdx.x; e < nt * 3 * (DP / 4); e += 128) copy(e / (3 * (DP / 4)), e / (DP / 4) % 3, e % (DP / 4) * 4);
    else
      for (int e = threadIdx.x; e < nt * 3 * DP; e += 128) copy(e / (3 * DP), e / DP % 3, e % DP);
    for (int e = threadIdx.x; e < nt * PB; e += 128) {
      const int t = e / PB, i = e % PB;
      if (col0 + i < dv)
        cp_async_f(base + t * PER + 3 * DP + i, qkv + (size_t)(r0 + t0 + t) * ld + (size_t)2 * G * d + (size_t)h * dv + col0 + i, false);
    }
    if (threadIdx.x < nt)
      cp_async_f(base + threadIdx.x * PER + 3 * DP + PB, beta + (size_t)(r0 + t0 + threadIdx.x) * ld_b + b_col + h, false);
    cp_async_commit();
  };
  const int n_chunks = (n + TC - 1) / TC;
  // A token's reductions over the channels (the corrections' of its own and the outputs' of the token before) go as one:
  // thread s ends up with value s / (NS / 2 NC) of [corrections | outputs].
  const int own = s / (NS / (2 * NC));
  const bool writes = s % (NS / (2 * NC)) == 0 && own >= NC && own - NC < cols;
  float* o_at = out + (size_t)r0 * H * dv + (size_t)h * dv + col0 + at + (own - NC);  // the output of the token before
  f32x2 q[PAIRS];
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) q[i] = 0;
  stage(0, 0);
  for (int c = 0; c < n_chunks; ++c) {
    if (c + 1 < n_chunks) { stage((c + 1) * TC, (c + 1) & 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int t0 = c * TC, nt = n - t0 < TC ? n - t0 : TC;
    // every thread of a warp takes part (the sums shuffle across whole warps); spare threads work on zeros
    const float* tok = sm + (c & 1) * TC * PER;
    f32x2 k[PAIRS], g[PAIRS];
    float v[NC], b = tok[3 * DP + PB];
    staged_rows<C>(k, tok + DP, s);
    staged_rows<C>(g, tok + 2 * DP, s);
    staged_values<NC>(v, tok + 3 * DP, at);
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      const float* next = t + 1 < nt ? tok + PER : tok;  // (read ahead of its use)
      f32x2 Sg[NC][PAIRS], k1[PAIRS];
      float v1[NC], sums[2 * NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) Sg[j][i] = f2_mul(S[j][i], g[i]);
        sums[j] = dot_rows(Sg[j], k);
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) sums[NC + j] = dot_rows(S[j], q);
      staged_rows<C>(k1, next + DP, s);
      staged_rows<C>(g, next + 2 * DP, s);
      staged_values<NC>(v1, next + 3 * DP, at);
      const float b1 = next[3 * DP + PB];
      const float o = spread_sum<NS, 2 * NC>(sums, s);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const float sum = __shfl_sync(0xffffffffu, o, j * (NS / (2 * NC)), NS);
        const f32x2 uu = f2_both(b * (v[j] - sum));
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) S[j][i] = f2_fma(k[i], uu, Sg[j][i]);
      }
      staged_rows<C>(q, tok, s);
      if (t0 + t > 0) {
        if (writes) *o_at = o;
        o_at += H * dv;
      }
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) k[i] = k1[i];
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] = v1[j];
      b = b1;
      tok = next;
    }
    __syncthreads();  // the buffer is free for the copies of the chunk after next
  }
  float sums[2 * NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) { sums[j] = 0.f; sums[NC + j] = dot_rows(S[j], q); }
  const float o = spread_sum<NS, 2 * NC>(sums, s);
  if (writes) *o_at = o;
  store_rows<C>(S, st, s, d, cols, wide);
}

// ---- the delta rule over long portions, four tokens at a time
// Token by token, every token's correction waits for a sum over the channels (four shuffles) of a state that the token
// before has just changed: about 500 clocks a token however the state is split. With P_t the product of the decays up to
// token t of a chunk, R_t of those behind it, G of all four, and S the state before the chunk, unrolled:
//   u_t = beta_t (v_t - S^T (P_t k_t) - sum_(s<t) c_ts u_s)   c_ts = k_s . (decays of s+1..t) k_t
//   o_t = S^T (P_t q_t) + sum_(s<=t) e_ts u_s                 e_ts = k_s . (decays of s+1..t) q_t
//   S  <- G S + sum_t (R_t k_t) u_t^T
// so eight sums over the channels go as one, and the scaled vectors and the numbers c and e, which do not depend on the
// state, are made by a kernel of their own over all chunks at once. All products of decays are at most 1. The rounding
// differs from token by token and depends on where a portion starts, so the 32-bit path does not come here; whether a
// request does depends on its own tokens and the sizes alone (`from` tokens or more), not on the step's other requests.
// Measured on 1,501 tokens, 16 heads of 128 x 128: 403 us token by token, 265 + 11 us
// this way (294 with a column a thread group, whose reads of the 13 vectors fill the shared memory's 128 bytes a clock).
constexpr int DC_T = 4, DC_D = 128;                          // tokens of a chunk; channels, zeros behind the last
constexpr int DC_COEF = 28;                                  // e [4][4], c_10, c_20, c_21, c_30, c_31, c_32, -, -, beta [4]
constexpr int DC_WORDS = (3 * DC_T + 1) * DC_D + DC_COEF;    // a (chunk, head): P k [4], P q [4], R k [4], G, coefficients

// Where a request's chunk c lies: portions are consecutive rows in the order of requests.
__device__ __forceinline__ size_t delta_chunk_slot(int r0, int c, int rq) { return (size_t)((r0 + DC_T * c) / DC_T + rq); }

// A warp per (chunk, head); a lane holds four channels.
__global__ void __launch_bounds__(256)
delta_chunk_prepare_kernel(const float* __restrict__ qkv, int ld, const float* __restrict__ decay, int ld_g,
                           const float* __restrict__ beta, int ld_b, int b_col, float* __restrict__ chunks,
                           const int* __restrict__ req_row0, const int* __restrict__ req_count,
                           const int* __restrict__ slots, int H, int G, int d, int from) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x, rq = blockIdx.y, h = blockIdx.z * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int n = req_count[rq], r0 = req_row0[rq];
  if (slots[rq] < 0 || n < from || c * DC_T >= n || h >= H) return;
  const int nt = min(DC_T, n - c * DC_T), kvh = h / (H / G), i = 4 * lane;
  float q[DC_T][4], k[DC_T][4], g[DC_T][4];
#pragma unroll
  for (int t = 0; t < DC_T; ++t) {
    float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), kv = qv, gv = make_float4(1.f, 1.f, 1.f, 1.f);  // no token: no change
    if (t < nt && i < d) {
      const size_t row = r0 + c * DC_T + t;
      qv = *reinterpret_cast<const float4*>(qkv + row * ld + (size_t)kvh * d + i);
      kv = *reinterpret_cast<const float4*>(qkv + row * ld + (size_t)(G + kvh) * d + i);
      gv = *reinterpret_cast<const float4*>(decay + row * ld_g + (size_t)h * d + i);
    }
    q[t][0] = qv.x; q[t][1] = qv.y; q[t][2] = qv.z; q[t][3] = qv.w;
    k[t][0] = kv.x; k[t][1] = kv.y; k[t][2] = kv.z; k[t][3] = kv.w;
    g[t][0] = gv.x; g[t][1] = gv.y; g[t][2] = gv.z; g[t][3] = gv.w;
  }
  float* to = chunks + (delta_chunk_slot(r0, c, rq) * H + h) * DC_WORDS;
  auto put = [&](int which, const float (&v)[4]) {
    *reinterpret_cast<float4*>(to + which * DC_D + i) = make_float4(v[0], v[1], v[2], v[3]);
  };
  float dots[16];  // e_00, e_10, e_11, e_20 .. e_33, then c_10, c_20, c_21, c_30, c_31, c_32
#pragma unroll
  for (int e = 0; e < 16; ++e) dots[e] = 0.f;
  {
    float P[4] = {1.f, 1.f, 1.f, 1.f}, v[4];
#pragma unroll
    for (int t = 0; t < DC_T; ++t) {
#pragma unroll
      for (int j = 0; j < 4; ++j) P[j] *= g[t][j];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = P[j] * k[t][j];
      put(t, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = P[j] * q[t][j];
      put(DC_T + t, v);
    }
    put(3 * DC_T, P);
  }
#pragma unroll
  for (int s = 0; s < DC_T; ++s) {  // token s's key, carried on through the decays behind it
    float w[4] = {k[s][0], k[s][1], k[s][2], k[s][3]};
#pragma unroll
    for (int t = s; t < DC_T; ++t) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (t > s) w[j] *= g[t][j];
        dots[t * (t + 1) / 2 + s] = fmaf(w[j], q[t][j], dots[t * (t + 1) / 2 + s]);
        if (t > s) dots[10 + t * (t - 1) / 2 + s] = fmaf(w[j], k[t][j], dots[10 + t * (t - 1) / 2 + s]);
      }
    }
    put(2 * DC_T + s, w);
  }
  const float mine = spread_sum<32, 16>(dots, lane);  // lane 2 e (and 2 e + 1): dot e
  float* coef = to + (3 * DC_T + 1) * DC_D;
  const int e = lane >> 1;
  if (lane & 1) {
    // the upper triangle of e and the spare numbers are zeros
    if (e < 6) coef[e < 3 ? e + 1 : e < 5 ? 6 + e - 3 : 11] = 0.f;
    else if (e < 8) coef[22 + e - 6] = 0.f;
    else if (e < 12) {
      const int t = e - 8;
      coef[24 + t] = t < nt ? beta[(size_t)(r0 + c * DC_T + t) * ld_b + b_col + h] : 0.f;
    }
  } else if (e < 10) {
    const int t = e < 1 ? 0 : e < 3 ? 1 : e < 6 ? 2 : 3;
    coef[t * 4 + e - t * (t + 1) / 2] = mine;
  } else {
    coef[16 + e - 10] = mine;
  }
}

// 256 threads: a warp per two value columns, four channels a lane. Two warps a scheduler over one prompt of 16 heads; the
// 13 vectors of a chunk are read from shared memory once for two columns (128 bytes a clock and SM: 416 clocks a chunk).
__global__ void __launch_bounds__(256)
delta_chunk_scan_kernel(const float* __restrict__ qkv, int ld, const float* __restrict__ chunks, float* __restrict__ state,
                        float* __restrict__ out, const int* __restrict__ req_row0, const int* __restrict__ req_count,
                        const int* __restrict__ slots, int H, int G, int d, int dv, int from) {
  using C = Split<32, 4, 2>;
  constexpr int NS = C::NS, NC = C::NC, PAIRS = C::PAIRS, PB = 16, RUN = 4;  // RUN: chunks staged at a time
  constexpr int PER = DC_WORDS + DC_T * PB;                      // a staged chunk, then the block's values [4][PB]
  extern __shared__ __align__(16) float sm[];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq], n = req_count[rq], r0 = req_row0[rq];
  if (slot < 0 || n < from) return;
  const int s = threadIdx.x % NS, col0 = blockIdx.z * PB, at = threadIdx.x / NS * NC;
  const int cols = min(NC, dv - col0 - at);  // columns of this warp that exist (none: 0 or less)
  float* st = state + (((size_t)slot * H + h) * dv + (cols > 0 ? col0 + at : 0)) * d;
  f32x2 S[NC][PAIRS];
  load_rows<C>(S, st, s, d, cols, 1);
  const int n_chunks = (n + DC_T - 1) / DC_T, runs = (n_chunks + RUN - 1) / RUN;
  // (values of columns from dv on: zeros, which no copy writes)
  for (int e = threadIdx.x; e < 2 * RUN * DC_T * PB; e += 256) sm[(e / (DC_T * PB)) * PER + DC_WORDS + e % (DC_T * PB)] = 0.f;
  __syncthreads();
  auto stage = [&](int run, int buf) {
    const int nc = min(RUN, n_chunks - run * RUN);
    float* base = sm + buf * RUN * PER;
    for (int e = threadIdx.x; e < nc * (DC_WORDS / 4); e += 256) {
      const int c = e / (DC_WORDS / 4), i = e % (DC_WORDS / 4) * 4;
      cp_async_f(base + c * PER + i, chunks + (delta_chunk_slot(r0, run * RUN + c, rq) * H + h) * DC_WORDS + i, true);
    }
    const int t = threadIdx.x / PB, i = threadIdx.x % PB, row = run * RUN * DC_T + t;  // 16 tokens, 16 columns
    if (row < n && col0 + i < dv)
      cp_async_f(base + (t / DC_T) * PER + DC_WORDS + (t % DC_T) * PB + i,
                 qkv + (size_t)(r0 + row) * ld + (size_t)2 * G * d + (size_t)h * dv + col0 + i, false);
    cp_async_commit();
  };
  // of the 16 sums, the one that this lane ends up with: [P k, P q][token][column]
  const int own = s / 2, own_t = own / NC % DC_T, own_c = own % NC;
  stage(0, 0);
  for (int run = 0; run < runs; ++run) {
    if (run + 1 < runs) { stage(run + 1, (run + 1) & 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int nc = min(RUN, n_chunks - run * RUN);
    const float* ch = sm + (run & 1) * RUN * PER;
    f32x2 w[2 * DC_T][PAIRS];  // P k, P q: read ahead of their use
#pragma unroll
    for (int t = 0; t < 2 * DC_T; ++t) staged_rows<C>(w[t], ch + t * DC_D, s);
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
      float sums[2 * DC_T * NC];
#pragma unroll
      for (int t = 0; t < 2 * DC_T; ++t)
#pragma unroll
        for (int j = 0; j < NC; ++j) sums[t * NC + j] = dot_rows(S[j], w[t]);
      const float* next = c + 1 < nc ? ch + PER : ch;
      const int there = n - (run * RUN + c) * DC_T;  // tokens of this chunk and behind it
#pragma unroll
      for (int t = 0; t < 2 * DC_T; ++t) staged_rows<C>(w[t], next + t * DC_D, s);
      f32x2 r[DC_T][PAIRS], g[PAIRS];
#pragma unroll
      for (int t = 0; t < DC_T; ++t) staged_rows<C>(r[t], ch + (2 * DC_T + t) * DC_D, s);
      staged_rows<C>(g, ch + 3 * DC_T * DC_D, s);
      const float* coef = ch + (3 * DC_T + 1) * DC_D;
      const float4 c4 = *reinterpret_cast<const float4*>(coef + 16);  // c_10, c_20, c_21, c_30
      const float2 c2 = *reinterpret_cast<const float2*>(coef + 20);  // c_31, c_32
      const float4 b = *reinterpret_cast<const float4*>(coef + 24);
      const float4 e4 = *reinterpret_cast<const float4*>(coef + own_t * 4);
      float v[DC_T][NC];
#pragma unroll
      for (int t = 0; t < DC_T; ++t) staged_values<NC>(v[t], ch + DC_WORDS + t * PB, at);
#pragma unroll
      for (int j = 0; j < NC; ++j)
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) S[j][i] = f2_mul(S[j][i], g[i]);
      const float mine = spread_sum<NS, 2 * DC_T * NC>(sums, s);
      float mine_u[DC_T];  // the corrections of this lane's own column
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        float a[DC_T];
#pragma unroll
        for (int t = 0; t < DC_T; ++t) a[t] = __shfl_sync(0xffffffffu, mine, 2 * (t * NC + j));
        if (there < DC_T) {  // tokens that do not exist (their write gates are zeros) correct nothing, whatever was found there
#pragma unroll
          for (int t = 1; t < DC_T; ++t)
            if (t >= there) a[t] = v[t][j] = 0.f;
        }
        const float u0 = b.x * (v[0][j] - a[0]);
        const float u1 = b.y * fmaf(-c4.x, u0, v[1][j] - a[1]);
        const float u2 = b.z * fmaf(-c4.z, u1, fmaf(-c4.y, u0, v[2][j] - a[2]));
        const float u3 = b.w * fmaf(-c2.y, u2, fmaf(-c2.x, u1, fmaf(-c4.w, u0, v[3][j] - a[3])));
        const float u[DC_T] = {u0, u1, u2, u3};
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
          if (j == 0 || own_c == j) mine_u[t] = u[t];
          const f32x2 uu = f2_both(u[t]);
#pragma unroll
          for (int i = 0; i < PAIRS; ++i) S[j][i] = f2_fma(r[t][i], uu, S[j][i]);
        }
      }
      // (tokens behind this lane's own are left out, not taken times zero: theirs may be no numbers)
      float o = fmaf(e4.x, mine_u[0], mine);
      if (own_t > 0) o = fmaf(e4.y, mine_u[1], o);
      if (own_t > 1) o = fmaf(e4.z, mine_u[2], o);
      if (own_t > 2) o = fmaf(e4.w, mine_u[3], o);
      if (own >= DC_T * NC && (s & 1) == 0 && own_c < cols && own_t < there)
        out[(size_t)(r0 + (run * RUN + c) * DC_T + own_t) * H * dv + (size_t)h * dv + col0 + at + own_c] = o;
      ch = next;
    }
    __syncthreads();  // the buffer is free again
  }
  store_rows<C>(S, st, s, d, cols, 1);
}

// Per row, in place, of a 32-bit projection [q | f | ...]: q (H d values at q_col) becomes silu(q); the forget gate's
// pre-activation (H d values at f_col) becomes f = l + (1 - l) sigmoid(x + bias) with a lower bound l per channel.
__global__ void forget_prepare_kernel(float* __restrict__ proj, int ld, int q_col, int f_col,
                                      const float* __restrict__ f_bias, const float* __restrict__ lower,
                                      const int* __restrict__ seq_of_row, int n_rows, int n) {
  pdl_trigger();
  pdl_wait();
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < (size_t)n_rows * n; e += (size_t)gridDim.x * blockDim.x) {
    const size_t row = e / n;
    const int i = (int)(e % n);
    if (seq_of_row[row] < 0) continue;
    float* r = proj + row * ld;
    const float q = r[q_col + i];
    r[q_col + i] = q * sigmoidf_(q);
    const float l = lower[i];
    r[f_col + i] = l + (1.f - l) * sigmoidf_(r[f_col + i] + (f_bias ? f_bias[i] : 0.f));
  }
}

// Per row, in place, of a 32-bit projection [q | k | ...] (H heads of d each): the first `rot` values of every q and k
// head turn by the row's position in pairs (i, i + rot/2) with the angle tables' row of that position; k is then
// multiplied by k_scale. One thread per (row, head, pair or unrotated value).
__global__ void retention_prepare_kernel(float* __restrict__ proj, int ld, int q_col, int k_col,
                                         const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                         int table_rows, int rot, float k_scale, const int* __restrict__ positions,
                                         const int* __restrict__ seq_of_row, int n_rows, int H, int d, int* err) {
  pdl_trigger();
  pdl_wait();
  const int half = rot / 2, per_head = half + (d - rot);
  const size_t per_row = (size_t)2 * H * per_head;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < (size_t)n_rows * per_row;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t row = e / per_row;
    const int w = (int)(e % per_row);
    if (seq_of_row[row] < 0) continue;
    const int which = w / (H * per_head), hh = (w / per_head) % H, i = w % per_head;
    float* head = proj + row * ld + (which ? k_col : q_col) + (size_t)hh * d;
    const float mul = which ? k_scale : 1.f;
    if (i < half) {
      const int pos = positions[row];
      if (pos < 0 || pos >= table_rows) {
        if (err) atomicExch(err, CUCA_ERR_TOKEN_RANGE);
        continue;
      }
      const float c = cos_t[(size_t)pos * half + i], sn = sin_t[(size_t)pos * half + i];
      const float a = head[i], b = head[i + half];
      head[i] = (a * c - b * sn) * mul;
      head[i + half] = (b * c + a * sn) * mul;
    } else if (which) {
      head[rot + (i - half)] *= mul;
    }
  }
}

// Per row, in place, of a 32-bit projection: `n` values from column col0 on become silu of themselves.
template <int V>
__global__ void __launch_bounds__(256)
silu_columns_kernel(float* __restrict__ proj, int ld, int col0, int n, const int* __restrict__ seq_of_row, int n_rows) {
  pdl_trigger();
  pdl_wait();
  const int per_row = n / V;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < (size_t)n_rows * per_row;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t row = e / per_row;
    if (seq_of_row[row] < 0) continue;
    float* at = proj + row * ld + col0 + (e % per_row) * V;
    if (V == 4) {
      float4 v = *reinterpret_cast<float4*>(at);
      v.x *= sigmoidf_(v.x); v.y *= sigmoidf_(v.y); v.z *= sigmoidf_(v.z); v.w *= sigmoidf_(v.w);
      *reinterpret_cast<float4*>(at) = v;
    } else {
      *at *= sigmoidf_(*at);
    }
  }
}

// A step in which every request brings one token: S <- decay[h] S + silu(k) silu(v)^T, o = S^T silu(q), with q, k, v the
// columns of the request's row from col0 on. A warp takes COLS value columns; a lane holds R packs of V consecutive key
// channels of each (32 V R >= d).
template <int V, int R, int COLS>
__global__ void __launch_bounds__(256)
lightning_step_kernel(const float* __restrict__ proj, int ld, int col0, const float* __restrict__ decay,
                      float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_row0,
                      const int* __restrict__ req_count, const int* __restrict__ slots, int H, int d, int dv) {
  struct alignas(4 * V) Pack { float v[V]; };
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq];
  if (slot < 0 || req_count[rq] <= 0) return;
  const size_t row = req_row0[rq];
  const int c0 = (blockIdx.z * 8 + (threadIdx.x >> 5)) * COLS, lane = threadIdx.x & 31;
  if (c0 >= dv) return;
  const float* pr = proj + row * ld + col0;
  const float* qp = pr + (size_t)h * d;
  const float* kp = qp + (size_t)H * d;
  const float* vp = pr + (size_t)2 * H * d + (size_t)h * dv;
  float* st = state + ((size_t)slot * H + h) * dv * d;
  const float dec = decay[h];
  Pack S[COLS][R], q[R], k[R];
#pragma unroll
  for (int c = 0; c < COLS; ++c)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = (lane + 32 * i) * V;
      if (c0 + c < dv && r < d) S[c][i] = *reinterpret_cast<const Pack*>(st + (size_t)(c0 + c) * d + r);
    }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = (lane + 32 * i) * V;
    if (r < d) { q[i] = *reinterpret_cast<const Pack*>(qp + r); k[i] = *reinterpret_cast<const Pack*>(kp + r); }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      q[i].v[j] = r < d ? q[i].v[j] * sigmoidf_(q[i].v[j]) : 0.f;
      k[i].v[j] = r < d ? k[i].v[j] * sigmoidf_(k[i].v[j]) : 0.f;
    }
  }
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    if (c0 + c >= dv) break;
    const float x = vp[c0 + c], v = x * sigmoidf_(x);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = (lane + 32 * i) * V;
      if (r < d) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
          S[c][i].v[j] = fmaf(dec, S[c][i].v[j], k[i].v[j] * v);
          sum = fmaf(S[c][i].v[j], q[i].v[j], sum);
        }
        *reinterpret_cast<Pack*>(st + (size_t)(c0 + c) * d + r) = S[c][i];
      }
    }
    sum = warp_sum(sum);
    if (lane == 0) out[row * H * dv + (size_t)h * dv + c0 + c] = sum;
  }
}

// proj: 32-bit rows of stride ld, prepared: q heads at q_col (H heads of d), forget gates at f_col (H heads of d),
// v heads at v_col (H heads of dv). state: [slots, H, dv, d]. out: [rows, H dv]. The delta scan's sibling without a
// correction: one shuffled sum per token and column.
// RET (retention): the second staged vector is the key k instead of the gate, and the state decays by one number per
// head: S <- decay[h] S + k v^T.
template <typename C, bool RET>
__global__ void __launch_bounds__(128)
forget_scan_kernel(const float* __restrict__ proj, int ld, int q_col, int f_col, int v_col,
                   const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ out,
                   const int* __restrict__ req_row0, const int* __restrict__ req_count,
                   const int* __restrict__ slots, int H, int d, int dv, int wide) {
  constexpr int NS = C::NS, NC = C::NC, DP = C::DP, PB = C::PB, TC = C::TC, PAIRS = C::PAIRS;
  constexpr int PER = 2 * DP + ((PB + 3) & ~3);  // a token: q, f, the block's values
  extern __shared__ __align__(16) float sm[];
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq], n = req_count[rq], r0 = req_row0[rq];
  if (slot < 0 || n <= 0) return;
  const int col_local = threadIdx.x / NS, s = threadIdx.x % NS;
  const int col0 = blockIdx.z * PB, at = col_local * NC;
  const int cols = min(NC, dv - col0 - at);               // columns of this thread that exist (none: 0 or less)
  float* st = state + (((size_t)slot * H + h) * dv + (cols > 0 ? col0 + at : 0)) * d;
  f32x2 S[NC][PAIRS];
  load_rows<C>(S, st, s, d, cols, wide);
  // what no copy writes: channels from d on (q = 0, f = 1, k = 0) and the values of columns from dv on
  {
    const int spare = DP - d, there = min(PB, dv - col0), fill = 2 * spare + PB - there;
    for (int e = threadIdx.x; e < (n < TC ? n : 2 * TC) * fill; e += 128) {
      const int t = e / fill, w = e % fill;
      float* tok = sm + t * PER;
      if (w < 2 * spare) tok[(w / spare) * DP + d + w % spare] = (w / spare == 1 && !RET) ? 1.f : 0.f;
      else tok[2 * DP + there + (w - 2 * spare)] = 0.f;
    }
  }
  __syncthreads();
  auto stage = [&](int t0, int buf) {
    const int nt = n - t0 < TC ? n - t0 : TC;
    float* base = sm + buf * TC * PER;
    auto copy = [&](int t, int which, int r) {
      const float* src = proj + (size_t)(r0 + t0 + t) * ld + (which ? f_col : q_col) + (size_t)h * d + r;
      if (r < d) cp_async_f(base + t * PER + which * DP + r, src, wide);
    };
    if (wide)
      for (int e = threadIdx.x; e < nt * 2 * (DP / 4); e += 128) copy(e / (2 * (DP / 4)), e / (DP / 4) % 2, e % (DP / 4) * 4);
    else
      for (int e = threadIdx.x; e < nt * 2 * DP; e += 128) copy(e / (2 * DP), e / DP % 2, e % DP);
    for (int e = threadIdx.x; e < nt * PB; e += 128) {
      const int t = e / PB, i = e % PB;
      if (col0 + i < dv)
        cp_async_f(base + t * PER + 2 * DP + i, proj + (size_t)(r0 + t0 + t) * ld + v_col + (size_t)h * dv + col0 + i, false);
    }
    cp_async_commit();
  };
  const int n_chunks = (n + TC - 1) / TC;
  const f32x2 dec = f2_both(RET ? decay[h] : 0.f), one = f2_both(1.f), minus = f2_both(-1.f);
  stage(0, 0);
  for (int c = 0; c < n_chunks; ++c) {
    if (c + 1 < n_chunks) { stage((c + 1) * TC, (c + 1) & 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int t0 = c * TC, nt = n - t0 < TC ? n - t0 : TC;
    const float* tok = sm + (c & 1) * TC * PER;
    float* o_at = out + (size_t)(r0 + t0) * H * dv + (size_t)h * dv + col0 + at;
    // Tokens depend on each other through the state's one multiply-add alone, so several are worked through at once and
    // their outputs summed together: thread s writes value s / (NS / (count NC)) of [tokens][columns].
    auto walk = [&](int t, auto count) {
      constexpr int U = decltype(count)::value;
      float o[U * NC];
#pragma unroll
      for (int i = 0; i < U; ++i, tok += PER) {
        f32x2 f[PAIRS], q[PAIRS], w[PAIRS];  // w: what is written, k or 1 - f
        float v[NC];
        staged_rows<C>(f, tok + DP, s);
        staged_rows<C>(q, tok, s);
        staged_values<NC>(v, tok + 2 * DP, at);
#pragma unroll
        for (int e = 0; e < PAIRS; ++e) w[e] = RET ? f[e] : f2_fma(f[e], minus, one);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const f32x2 vv = f2_both(v[j]);
          // decay S + k v or f S + (1 - f) v, each product rounded
#pragma unroll
          for (int e = 0; e < PAIRS; ++e) S[j][e] = f2_fma(RET ? dec : f[e], S[j][e], f2_mul(w[e], vv));
          o[i * NC + j] = dot_rows(S[j], q);
        }
      }
      constexpr int LANES = NS / (U * NC);
      const float sum = spread_sum<NS, U * NC>(o, s);
      const int own = s / LANES;
      if (s % LANES == 0 && own % NC < cols) o_at[(size_t)(t + own / NC) * H * dv + own % NC] = sum;
    };
    int t = 0;
    for (; t + C::U8 <= nt; t += C::U8) walk(t, Count<C::U8>());
    for (; t < nt; ++t) walk(t, Count<1>());
    __syncthreads();  // the buffer is free for the copies of the chunk after next
  }
  store_rows<C>(S, st, s, d, cols, wide);
}

// Per row, in place: the raw input gate of head h (column i_col + h of proj) becomes cap tanh((x + b_i) / cap), the
// raw forget gate (column f_col + h) becomes logsigmoid(cap tanh((x + b_f) / cap)).
__global__ void mlstm_prepare_kernel(float* __restrict__ proj, int ld, int i_col, int f_col,
                                     const float* __restrict__ i_bias, const float* __restrict__ f_bias, float cap,
                                     int n_rows, int H) {
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_rows * H) return;
  float* row = proj + (size_t)(e / H) * ld;
  const int h = e % H;
  row[i_col + h] = cap * tanhf((row[i_col + h] + (i_bias ? i_bias[h] : 0.f)) / cap);
  row[f_col + h] = log_sigmoidf_(cap * tanhf((row[f_col + h] + (f_bias ? f_bias[h] : 0.f)) / cap));
}

// proj: 32-bit rows of stride ld, prepared: q heads at q_col (H heads of d), k at k_col, v at v_col (H heads of dv),
// the log input gate of head h at i_col + h, the log forget gate at f_col + h.
// mem: [slots, H, dv, d]; nrm: [slots, H, d]; mx: [slots, H]. out: [rows, H dv].
// Every column's threads carry n too (three more multiply-adds a pair of channels, and no exchange between warps), and
// every warp works the running maximum of a run of tokens out for itself: a chain of one add and one max per token,
// after which a lane per token takes the exponentials. q enters unscaled: the sums are linear in it, so d^(-1/2)
// multiplies them afterwards. n and m are shared by all blocks of a (head, request): this launch only reads them and
// leaves the new ones aside (nm_new [requests, H, d + 1]); `mlstm_commit_kernel` moves them into the slots.
template <typename C>
__global__ void __launch_bounds__(128)
mlstm_scan_kernel(const float* __restrict__ proj, int ld, int q_col, int k_col, int v_col, int i_col,
                  int f_col, float* __restrict__ mem, const float* __restrict__ nrm, const float* __restrict__ mx,
                  float* __restrict__ out, const int* __restrict__ req_row0,
                  const int* __restrict__ req_count, const int* __restrict__ slots, int H, int d,
                  int dv, int wide, float* __restrict__ nm_new) {
  constexpr int NS = C::NS, NC = C::NC, DP = C::DP, PB = C::PB, TC = C::TC, PAIRS = C::PAIRS;
  constexpr int PER = 2 * DP + ((PB + 2 + 3) & ~3);  // a token: q, k, the block's values, the two gates
  static_assert(TC <= 32, "a lane a token");
  extern __shared__ __align__(16) float sm[];
  __shared__ float gates[4][TC][3];  // a warp's own: e^(f + m - m'), e^(i - m'), e^(-m')
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq], n = req_count[rq], r0 = req_row0[rq];
  if (slot < 0 || n <= 0) return;
  const int lane = threadIdx.x & 31;
  const int col_local = threadIdx.x / NS, s = threadIdx.x % NS;
  const int col0 = blockIdx.z * PB, at = col_local * NC;
  const int cols = min(NC, dv - col0 - at);               // columns of this thread that exist (none: 0 or less)
  float* st = mem + (((size_t)slot * H + h) * dv + (cols > 0 ? col0 + at : 0)) * d;
  using One = Split<C::NS, C::NR, 1>;
  f32x2 S[NC][PAIRS], Zs[1][PAIRS];
  load_rows<C>(S, st, s, d, cols, wide);
  load_rows<One>(Zs, nrm + ((size_t)slot * H + h) * d, s, d, 1, wide);
  f32x2(&Z)[PAIRS] = Zs[0];
  float m = mx[(size_t)slot * H + h];
  {
    const int spare = DP - d, there = min(PB, dv - col0), fill = 2 * spare + PB - there;
    for (int e = threadIdx.x; e < (n < TC ? n : 2 * TC) * fill; e += 128) {
      const int t = e / fill, w = e % fill;
      float* tok = sm + t * PER;
      if (w < 2 * spare) tok[(w / spare) * DP + d + w % spare] = 0.f;
      else tok[2 * DP + there + (w - 2 * spare)] = 0.f;
    }
  }
  __syncthreads();
  const float qscale = rsqrtf((float)d);
  auto stage = [&](int t0, int buf) {
    const int nt = n - t0 < TC ? n - t0 : TC;
    float* base = sm + buf * TC * PER;
    auto copy = [&](int t, int which, int r) {
      const float* src = proj + (size_t)(r0 + t0 + t) * ld + (which ? k_col : q_col) + (size_t)h * d + r;
      if (r < d) cp_async_f(base + t * PER + which * DP + r, src, wide);
    };
    if (wide)
      for (int e = threadIdx.x; e < nt * 2 * (DP / 4); e += 128) copy(e / (2 * (DP / 4)), e / (DP / 4) % 2, e % (DP / 4) * 4);
    else
      for (int e = threadIdx.x; e < nt * 2 * DP; e += 128) copy(e / (2 * DP), e / DP % 2, e % DP);
    for (int e = threadIdx.x; e < nt * PB; e += 128) {
      const int t = e / PB, i = e % PB;
      if (col0 + i < dv)
        cp_async_f(base + t * PER + 2 * DP + i, proj + (size_t)(r0 + t0 + t) * ld + v_col + (size_t)h * dv + col0 + i, false);
    }
    if (threadIdx.x < 2 * nt) {
      const int t = threadIdx.x >> 1, which = threadIdx.x & 1;
      cp_async_f(base + t * PER + 2 * DP + PB + which, proj + (size_t)(r0 + t0 + t) * ld + (which ? f_col : i_col) + h, false);
    }
    cp_async_commit();
  };
  const int n_chunks = (n + TC - 1) / TC;
  float(*mine)[3] = gates[threadIdx.x >> 5];
  stage(0, 0);
  for (int c = 0; c < n_chunks; ++c) {
    if (c + 1 < n_chunks) { stage((c + 1) * TC, (c + 1) & 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int t0 = c * TC, nt = n - t0 < TC ? n - t0 : TC;
    const float* tok = sm + (c & 1) * TC * PER;
    {
      float before = m, after = m;  // the maximum before and after this lane's token
#pragma unroll
      for (int t = 0; t < TC; ++t) {
        if (t < nt) {
          const float next = fmaxf(tok[t * PER + 2 * DP + PB + 1] + m, tok[t * PER + 2 * DP + PB]);
          if (t == lane) { before = m; after = next; }
          m = next;
        }
      }
      if (lane < nt) {
        const float* at = tok + lane * PER + 2 * DP + PB;
        mine[lane][0] = expf(at[1] + before - after);
        mine[lane][1] = expf(at[0] - after);
        mine[lane][2] = expf(-after);
      }
      __syncwarp();
    }
    float* o_at = out + (size_t)(r0 + t0) * H * dv + (size_t)h * dv + col0 + at;
    // (several tokens at once, as in the forget scan; a token's n . q ends up with the threads that write its outputs)
    auto walk = [&](int t, auto count) {
      constexpr int U = decltype(count)::value;
      float o[U * NC], z[U];
#pragma unroll
      for (int i = 0; i < U; ++i, tok += PER) {
        f32x2 k[PAIRS], q[PAIRS];
        float v[NC];
        staged_rows<C>(k, tok + DP, s);
        staged_rows<C>(q, tok, s);
        staged_values<NC>(v, tok + 2 * DP, at);
        const float take = mine[t + i][1];
        const f32x2 keep = f2_both(mine[t + i][0]), w1 = f2_both(take);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const f32x2 w = f2_both(take * v[j]);
#pragma unroll
          for (int e = 0; e < PAIRS; ++e) S[j][e] = f2_fma(keep, S[j][e], f2_mul(w, k[e]));
          o[i * NC + j] = dot_rows(S[j], q);
        }
#pragma unroll
        for (int e = 0; e < PAIRS; ++e) Z[e] = f2_fma(keep, Z[e], f2_mul(w1, k[e]));
        z[i] = dot_rows(Z, q);
      }
      constexpr int LANES = NS / (U * NC);
      const float num = spread_sum<NS, U * NC>(o, s) * qscale;
      const float den = spread_sum<NS, U>(z, s) * qscale;
      const int own = s / LANES;
      if (s % LANES == 0 && own % NC < cols)
        o_at[(size_t)(t + own / NC) * H * dv + own % NC] = num / (fmaxf(fabsf(den), mine[t + own / NC][2]) + 1e-6f);
    };
    int t = 0;
#pragma unroll 2
    for (; t + C::U8 <= nt; t += C::U8) walk(t, Count<C::U8>());
    for (; t < nt; ++t) walk(t, Count<1>());
    __syncthreads();  // the buffer is free again
  }
  // every block of a (head, request) starts from the same n and m, so no block of this launch may replace them: the
  // first column's threads of the first block leave the new ones aside
  store_rows<C>(S, st, s, d, cols, wide);
  if (blockIdx.z == 0 && col_local == 0) {
    float* nm = nm_new + ((size_t)rq * H + h) * (d + 1);
    store_column<C::NS, C::PAIRS>(Z, nm, s, d, 0);
    if (s == 0) nm[d] = m;
  }
}

__global__ void mlstm_commit_kernel(const float* __restrict__ nm_new, float* __restrict__ nrm, float* __restrict__ mx,
                                    const int* __restrict__ req_count, const int* __restrict__ slots, int H, int d) {
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, rq = blockIdx.y;
  const int slot = slots[rq];
  if (slot < 0 || req_count[rq] <= 0) return;
  const float* nm = nm_new + ((size_t)rq * H + h) * (d + 1);
  for (int i = threadIdx.x; i < d; i += blockDim.x) nrm[((size_t)slot * H + h) * d + i] = nm[i];
  if (threadIdx.x == 0) mx[(size_t)slot * H + h] = nm[d];
}

// o: [rows, H dv] 32-bit. out[r, h, j] = o / sqrt(mean_j o^2 + eps) * w[h * w_head + j] * sigmoid(gate[r, h dv + j]);
// w_head 0: one weight vector for every head; w null: no weight. gate: rows of stride ld_g (TG), null for none;
// SILU: the gate's factor is silu(gate) instead of sigmoid(gate).
template <typename TG, typename TO, bool SILU>
__global__ void __launch_bounds__(256)
head_norm_gate_kernel(const float* __restrict__ o, const float* __restrict__ w, int w_head,
                      const TG* __restrict__ gate, int ld_g, TO* __restrict__ out, int H, int dv, float eps,
                      long long n_items) {
  pdl_trigger();
  pdl_wait();
  // a warp per (row, head); 16 bytes of o a lane at a time where a head's values allow it
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= n_items) return;
  const size_t row = (size_t)(item / H);
  const int h = (int)(item % H);
  const float* orow = o + (size_t)item * dv;
  const float* wh = w ? w + (size_t)h * w_head : nullptr;
  auto gate_of = [](float g) { return SILU ? g * sigmoidf_(g) : sigmoidf_(g); };
  const TG* grow = gate ? gate + row * ld_g + (size_t)h * dv : nullptr;
  TO* dst = out + (size_t)item * dv;
  if ((dv & 3) == 0) {
    float ss = 0.f;
    for (int j = lane * 4; j < dv; j += 128) {
      const float4 v = *reinterpret_cast<const float4*>(orow + j);
      ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
    }
    const float inv = 1.f / sqrtf(warp_sum(ss) / (float)dv + eps);
    for (int j = lane * 4; j < dv; j += 128) {
      const float4 v = *reinterpret_cast<const float4*>(orow + j);
      float r[4] = {v.x * inv, v.y * inv, v.z * inv, v.w * inv};
      if (wh) {
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] *= wh[j + e];
      }
      if (grow) {
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] *= gate_of(to_f32(grow[j + e]));
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[j + e] = from_f32<TO>(r[e]);
    }
    return;
  }
  float ss = 0.f;
  for (int j = lane; j < dv; j += 32) ss = fmaf(orow[j], orow[j], ss);
  const float inv = 1.f / sqrtf(warp_sum(ss) / (float)dv + eps);
  for (int j = lane; j < dv; j += 32) {
    float v = orow[j] * inv * (wh ? wh[j] : 1.f);
    if (grow) v *= gate_of(to_f32(grow[j]));
    dst[j] = from_f32<TO>(v);
  }
}

// Runs `go` with the split of d key channels (at most MAX_DIM). A prompt of one request has few columns (16 heads of
// 128: 2,048) and a serial chain of one token after the other, so what counts is the time of one token in one warp: at
// 128 channels, eight channels of two columns a thread give each of the SM's four schedulers one warp.
template <typename F>
int with_split(int d, F go) {
  if (d <= 32) return go(Split<4, 8, 2>());
  if (d <= 64) return go(Split<8, 8, 2>());
  if (d <= 128) return go(Split<16, 8, 2>());
  if (d <= 256) return go(Split<32, 8, 2>());
  if (d <= 512) return go(Split<32, 16, 2>());
  return go(Split<32, 32, 2>());
}

// The same for the scans without a correction, which have less to do per channel: half as many channels a thread. (One
// prompt of 1,501 tokens, 16 heads of 128 x 128, eight tokens summed together: 208 us with eight channels, 165 with four;
// the matrix memory, which carries n too, 212 and 224. Eight requests of one token: 5 and 6 us.)
template <typename F>
int with_narrow_split(int d, F go) {
  if (d <= 32) return go(Split<8, 4, 2>());
  if (d <= 64) return go(Split<16, 4, 2>());
  if (d <= 128) return go(Split<32, 4, 2>());
  return with_split(d, go);
}

}  // namespace

CUCA_API int cuca_matrix_state_max_dim() { return MAX_DIM; }

// qkv, a_raw and the gate column of b_raw are rewritten in place by the preparing kernel (see there), then scanned.
CUCA_API int cuca_delta_scan(float* qkv, int ld, float* a_raw, int ld_a, const float* dt_bias, const float* a_log,
                             float* b_raw, int ld_b, int b_col, float* state, float* out, const int* seq_of_row,
                             const int* req_row0, const int* req_count, const int* slots, int n_rows, int n_seqs, int H,
                             int G, int d, int dv, cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && G > 0 && H % G == 0 && d > 0 && dv > 0, "delta_scan: bad sizes heads=%d key heads=%d dim=%d vdim=%d",
               H, G, d, dv);
  CUCA_REQUIRE(n_seqs <= 65535 && H <= 256, "delta_scan: %d requests or %d heads exceed the launch limits", n_seqs, H);
  CUCA_REQUIRE(d <= MAX_DIM, "delta_scan: %d key channels exceed %d", d, MAX_DIM);
  cuca_launch(delta_prepare_kernel, dim3(n_rows), dim3(256), 0, stream, true, qkv, ld, a_raw, ld_a, dt_bias, a_log, b_raw, ld_b,
              b_col, seq_of_row, H, G, d);
  CUCA_CHECK_LAUNCH("delta_prepare");
  // 16-byte copies where every source is aligned for them
  const int wide = d % 4 == 0 && ld % 4 == 0 && ld_a % 4 == 0 && ((uintptr_t)qkv & 15) == 0 && ((uintptr_t)a_raw & 15) == 0 &&
                   ((uintptr_t)state & 15) == 0;
  return with_split(d, [&](auto split) {
    using C = decltype(split);
    return launch_scan<C>("delta_scan", delta_scan_kernel<C>, 3 * C::DP + ((C::PB + 4) & ~3), H, n_seqs, dv, stream,
                          (const float*)qkv, ld, (const float*)a_raw, ld_a, (const float*)b_raw, ld_b, b_col, state, out,
                          req_row0, req_count, slots, H, G, d, dv, wide, 0x7fffffff);
  });
}

// Floats of the chunked form's scratch per (four tokens of a request, head); there are at most
// n_rows / 4 + n_seqs + 1 such fours in a step.
CUCA_API int cuca_delta_chunk_words() { return DC_WORDS; }

// The same, requests that bring `from` tokens or more in chunks of four tokens (see there), the others token by token; d a
// multiple of 4 up to 128, everything 16-byte aligned. min_count, max_count: the shortest and the longest portion (at least
// `from`). chunks: scratch.
CUCA_API int cuca_delta_scan_chunked(float* qkv, int ld, float* a_raw, int ld_a, const float* dt_bias, const float* a_log,
                                     float* b_raw, int ld_b, int b_col, float* state, float* out, float* chunks,
                                     const int* seq_of_row, const int* req_row0, const int* req_count, const int* slots,
                                     int n_rows, int n_seqs, int from, int min_count, int max_count, int H, int G, int d, int dv,
                                     cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && G > 0 && H % G == 0 && d > 0 && dv > 0, "delta_scan: bad sizes heads=%d key heads=%d dim=%d vdim=%d",
               H, G, d, dv);
  CUCA_REQUIRE(n_seqs <= 65535 && H <= 256, "delta_scan: %d requests or %d heads exceed the launch limits", n_seqs, H);
  CUCA_REQUIRE(from > 0 && max_count >= from, "delta_scan: no portion of %d tokens (the longest: %d)", from, max_count);
  CUCA_REQUIRE(d <= DC_D && d % 4 == 0 && ld % 4 == 0 && ld_a % 4 == 0 &&
                   (((uintptr_t)qkv | (uintptr_t)a_raw | (uintptr_t)state | (uintptr_t)chunks) & 15) == 0,
               "delta_scan: the chunked form does not take %d key channels, row strides %d and %d or an unaligned operand", d,
               ld, ld_a);
  cuca_launch(delta_prepare_kernel, dim3(n_rows), dim3(256), 0, stream, true, qkv, ld, a_raw, ld_a, dt_bias, a_log, b_raw, ld_b,
              b_col, seq_of_row, H, G, d);
  CUCA_CHECK_LAUNCH("delta_prepare");
  cuca_launch(delta_chunk_prepare_kernel, dim3((max_count + DC_T - 1) / DC_T, n_seqs, (H + 7) / 8), dim3(256), 0, stream, true,
              (const float*)qkv, ld, (const float*)a_raw, ld_a, (const float*)b_raw, ld_b, b_col, chunks, req_row0, req_count,
              slots, H, G, d, from);
  CUCA_CHECK_LAUNCH("delta_chunk_prepare");
  const int rc = launch_blocks("delta_chunk_scan", delta_chunk_scan_kernel, dim3(H, n_seqs, (dv + 15) / 16), 256,
                               2 * 4 * (DC_WORDS + DC_T * 16) * 4, stream, (const float*)qkv, ld, (const float*)chunks, state,
                               out, req_row0, req_count, slots, H, G, d, dv, from);
  if (rc || min_count >= from) return rc;
  return with_split(d, [&](auto split) {
    using C = decltype(split);
    return launch_scan<C>("delta_scan", delta_scan_kernel<C>, 3 * C::DP + ((C::PB + 4) & ~3), H, n_seqs, dv, stream,
                          (const float*)qkv, ld, (const float*)a_raw, ld_a, (const float*)b_raw, ld_b, b_col, state, out,
                          req_row0, req_count, slots, H, G, d, dv, 1, from);
  });
}

// The two gate columns of proj are rewritten in place by the preparing kernel (see there), then scanned.
// nm_new: scratch of n_seqs * H * (d + 1) floats.
CUCA_API int cuca_mlstm_scan(float* proj, int ld, int q_col, int k_col, int v_col, int i_col, int f_col,
                             const float* i_bias, const float* f_bias, float cap, float* mem, float* nrm, float* mx,
                             float* out, float* nm_new, const int* req_row0, const int* req_count, const int* slots,
                             int n_rows, int n_seqs, int H, int d, int dv, cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && d > 0 && dv > 0 && cap > 0.f, "mlstm_scan: bad sizes heads=%d dim=%d vdim=%d cap=%g", H, d, dv,
               (double)cap);
  CUCA_REQUIRE(n_seqs <= 65535, "mlstm_scan: %d requests exceed the launch limit", n_seqs);
  CUCA_REQUIRE(d <= MAX_DIM, "mlstm_scan: %d key channels exceed %d", d, MAX_DIM);
  cuca_launch(mlstm_prepare_kernel, dim3((n_rows * H + 127) / 128), dim3(128), 0, stream, true, proj, ld, i_col, f_col,
              i_bias, f_bias, cap, n_rows, H);
  CUCA_CHECK_LAUNCH("mlstm_prepare");
  const int wide = d % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && ((uintptr_t)proj & 15) == 0 &&
                   (((uintptr_t)mem | (uintptr_t)nrm) & 15) == 0;
  const int rc = with_split(d, [&](auto split) {
    using C = decltype(split);
    return launch_scan<C>("mlstm_scan", mlstm_scan_kernel<C>, 2 * C::DP + ((C::PB + 5) & ~3), H, n_seqs, dv, stream,
                          (const float*)proj, ld, q_col, k_col, v_col, i_col, f_col, mem, (const float*)nrm,
                          (const float*)mx, out, req_row0, req_count, slots, H, d, dv, wide, nm_new);
  });
  if (rc) return rc;
  cuca_launch(mlstm_commit_kernel, dim3(H, n_seqs), dim3(128), 0, stream, true, (const float*)nm_new, nrm, mx, req_count,
              slots, H, d);
  CUCA_CHECK_LAUNCH("mlstm_commit");
  return 0;
}

// The q and forget-gate columns of proj are rewritten in place by the preparing kernel (see there), then scanned.
CUCA_API int cuca_forget_scan(float* proj, int ld, int q_col, int f_col, int v_col, const float* f_bias,
                              const float* lower, float* state, float* out, const int* seq_of_row, const int* req_row0,
                              const int* req_count, const int* slots, int n_rows, int n_seqs, int H, int d, int dv,
                              cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && d > 0 && dv > 0, "forget_scan: bad sizes heads=%d dim=%d vdim=%d", H, d, dv);
  CUCA_REQUIRE(n_seqs <= 65535, "forget_scan: %d requests exceed the launch limit", n_seqs);
  CUCA_REQUIRE(d <= MAX_DIM, "forget_scan: %d key channels exceed %d", d, MAX_DIM);
  {
    size_t blocks = ((size_t)n_rows * H * d + 255) / 256;
    blocks = blocks > 8192 ? 8192 : blocks;
    cuca_launch(forget_prepare_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, true, proj, ld, q_col, f_col, f_bias,
                lower, seq_of_row, n_rows, H * d);
    CUCA_CHECK_LAUNCH("forget_prepare");
  }
  const int wide = d % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && f_col % 4 == 0 && ((uintptr_t)proj & 15) == 0 &&
                   ((uintptr_t)state & 15) == 0;
  return with_narrow_split(d, [&](auto split) {
    using C = decltype(split);
    return launch_scan<C>("forget_scan", forget_scan_kernel<C, false>, 2 * C::DP + ((C::PB + 3) & ~3), H, n_seqs, dv, stream,
                          (const float*)proj, ld, q_col, f_col, v_col, (const float*)nullptr, state, out, req_row0,
                          req_count, slots, H, d, dv, wide);
  });
}

// S <- decay[h] S + k v^T, o = S^T q along every request's rows of a prepared 32-bit projection
static int launch_decay_scan(const char* name, const float* proj, int ld, int q_col, int k_col, int v_col, const float* decay,
                             float* state, float* out, const int* req_row0, const int* req_count, const int* slots,
                             int n_seqs, int H, int d, int dv, cudaStream_t stream) {
  CUCA_REQUIRE(d <= MAX_DIM, "%s: %d key channels exceed %d", name, d, MAX_DIM);
  const int wide = d % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && ((uintptr_t)proj & 15) == 0 &&
                   ((uintptr_t)state & 15) == 0;
  return with_narrow_split(d, [&](auto split) {
    using C = decltype(split);
    return launch_scan<C>(name, forget_scan_kernel<C, true>, 2 * C::DP + ((C::PB + 3) & ~3), H, n_seqs, dv, stream, proj, ld,
                          q_col, k_col, v_col, decay, state, out, req_row0, req_count, slots, H, d, dv, wide);
  });
}

// Retention along every request's rows. proj: 32-bit rows of stride ld holding q heads at q_col, k heads at k_col (H
// heads of d each) and v heads at v_col (H heads of dv). The preparing kernel turns the first `rot` values of every q
// and k head by the row's position (pairs (i, i + rot/2); cos_t/sin_t: [table_rows, rot/2]) and multiplies k by
// k_scale, in place; the scan then runs S <- decay[h] S + k v^T, o = S^T q from the state in the request's slot
// (state: [slots, H, dv, d], out: [rows, H dv], both 32-bit).
CUCA_API int cuca_retention_scan(float* proj, int ld, int q_col, int k_col, int v_col, const float* decay,
                                 const float* cos_t, const float* sin_t, int table_rows, int rot, float k_scale,
                                 const int* positions, float* state, float* out, const int* seq_of_row,
                                 const int* req_row0, const int* req_count, const int* slots, int n_rows, int n_seqs,
                                 int H, int d, int dv, int* err, cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && d > 0 && dv > 0, "retention_scan: bad sizes heads=%d dim=%d vdim=%d", H, d, dv);
  CUCA_REQUIRE(rot >= 0 && rot <= d && rot % 2 == 0, "retention_scan: rotary size %d does not fit head size %d", rot, d);
  CUCA_REQUIRE(n_seqs <= 65535, "retention_scan: %d requests exceed the launch limit", n_seqs);
  {
    size_t blocks = ((size_t)n_rows * 2 * H * (d - rot / 2) + 255) / 256;
    blocks = blocks > 8192 ? 8192 : blocks;
    cuca_launch(retention_prepare_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, true, proj, ld, q_col, k_col,
                cos_t, sin_t, table_rows, rot, k_scale, positions, seq_of_row, n_rows, H, d, err);
    CUCA_CHECK_LAUNCH("retention_prepare");
  }
  return launch_decay_scan("retention_scan", proj, ld, q_col, k_col, v_col, decay, state, out, req_row0, req_count, slots,
                           n_seqs, H, d, dv, stream);
}

// Lightning attention along every request's rows. proj as for retention; q, k and v (contiguous from col0 on: H heads of
// d, H heads of d, H heads of dv) hold pre-activations and become silu of themselves in place; then retention's scan.
CUCA_API int cuca_lightning_scan(float* proj, int ld, int col0, const float* decay, float* state, float* out,
                                 const int* seq_of_row, const int* req_row0, const int* req_count, const int* slots,
                                 int n_rows, int n_seqs, int H, int d, int dv, cudaStream_t stream) {
  if (n_seqs == 0 || n_rows == 0) return 0;
  CUCA_REQUIRE(H > 0 && d > 0 && dv > 0, "lightning_scan: bad sizes heads=%d dim=%d vdim=%d", H, d, dv);
  CUCA_REQUIRE(n_seqs <= 65535, "lightning_scan: %d requests exceed the launch limit", n_seqs);
  const int n = H * (2 * d + dv);
  const bool wide = n % 4 == 0 && ld % 4 == 0 && col0 % 4 == 0 && ((uintptr_t)proj & 15) == 0;
  size_t blocks = ((size_t)n_rows * n / (wide ? 4 : 1) + 255) / 256;
  blocks = blocks > 8192 ? 8192 : blocks;
  if (wide)
    cuca_launch(silu_columns_kernel<4>, dim3((unsigned)blocks), dim3(256), 0, stream, true, proj, ld, col0, n, seq_of_row, n_rows);
  else
    cuca_launch(silu_columns_kernel<1>, dim3((unsigned)blocks), dim3(256), 0, stream, true, proj, ld, col0, n, seq_of_row, n_rows);
  CUCA_CHECK_LAUNCH("silu_columns");
  return launch_decay_scan("lightning_scan", proj, ld, col0, col0 + H * d, col0 + 2 * H * d, decay, state, out, req_row0,
                           req_count, slots, n_seqs, H, d, dv, stream);
}

// The same for a step in which every request brings one token, in one launch; proj is only read.
CUCA_API int cuca_lightning_step(const float* proj, int ld, int col0, const float* decay, float* state, float* out,
                                 const int* req_row0, const int* req_count, const int* slots, int n_seqs, int H, int d,
                                 int dv, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  CUCA_REQUIRE(H > 0 && d > 0 && dv > 0 && d <= MAX_DIM, "lightning_step: bad sizes heads=%d dim=%d vdim=%d", H, d, dv);
  CUCA_REQUIRE(n_seqs <= 65535, "lightning_step: %d requests exceed the launch limit", n_seqs);
  const bool wide = d % 4 == 0 && ld % 4 == 0 && col0 % 4 == 0 && ((uintptr_t)proj & 15) == 0 && ((uintptr_t)state & 15) == 0;
#define LS(V, R, COLS)                                                                                              \
  cuca_launch(lightning_step_kernel<V, R, COLS>, dim3(H, n_seqs, (dv + 8 * COLS - 1) / (8 * COLS)), dim3(256), 0,   \
              stream, true, proj, ld, col0, decay, state, out, req_row0, req_count, slots, H, d, dv)
  if (wide && d <= 128) LS(4, 1, 4);
  else if (wide && d <= 256) LS(4, 2, 4);
  else if (wide) LS(4, 8, 1);
  else if (d <= 128) LS(1, 4, 4);
  else LS(1, 32, 1);
#undef LS
  CUCA_CHECK_LAUNCH("lightning_step");
  return 0;
}

// gate_act 0: the gate's factor is sigmoid(gate); 1: silu(gate). w null: no weight.
CUCA_API int cuca_head_norm_gate_act(const float* o, const float* w, int w_head, const void* gate, int gate_dtype,
                                     int ld_g, int gate_act, void* out, int out_dtype, int n_rows, int H, int dv,
                                     float eps, cudaStream_t stream) {
  if (n_rows == 0) return 0;
  const long long n_items = (long long)n_rows * H;
  dim3 grid((unsigned)((n_items + 7) / 8));
#define HNG(TG, TO)                                                                                                 \
  do {                                                                                                              \
    if (gate_act)                                                                                                   \
      cuca_launch(head_norm_gate_kernel<TG, TO, true>, grid, dim3(256), 0, stream, true, o, w, w_head,              \
                  (const TG*)gate, ld_g, (TO*)out, H, dv, eps, n_items);                                            \
    else                                                                                                            \
      cuca_launch(head_norm_gate_kernel<TG, TO, false>, grid, dim3(256), 0, stream, true, o, w, w_head,             \
                  (const TG*)gate, ld_g, (TO*)out, H, dv, eps, n_items);                                            \
  } while (0)
  if (gate_dtype == CUCA_F32 && out_dtype == CUCA_F32) HNG(float, float);
  else if (gate_dtype == CUCA_F32 && out_dtype == CUCA_BF16) HNG(float, __nv_bfloat16);
  else if (gate_dtype == CUCA_BF16 && out_dtype == CUCA_BF16) HNG(__nv_bfloat16, __nv_bfloat16);
  else CUCA_REQUIRE(false, "head_norm_gate: unsupported dtypes %d/%d", gate_dtype, out_dtype);
#undef HNG
  CUCA_CHECK_LAUNCH("head_norm_gate");
  return 0;
}

CUCA_API int cuca_head_norm_gate(const float* o, const float* w, int w_head, const void* gate, int gate_dtype, int ld_g,
                                 void* out, int out_dtype, int n_rows, int H, int dv, float eps, cudaStream_t stream) {
  return cuca_head_norm_gate_act(o, w, w_head, gate, gate_dtype, ld_g, 0, out, out_dtype, n_rows, H, dv, eps, stream);
}
